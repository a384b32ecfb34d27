// C-ABI entry points over single stages, for callers that hold code-blocks rather than
// frames (and for the parity tests): a batch of quantised code-blocks through the
// Tier-1 encoder, and a batch of codewords through the Tier-1 decoder.
#include <cuda_runtime.h>

#include <cstring>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "capi_util.h"
#include "gail_b200.h"
#include "common.cuh"
#include "compact.cuh"
#include "pack_runs.h"
#include "t1_encode.cuh"

using namespace gb;

namespace {

// The memory of the call before, one block per device, kept for the next call up to kKeepBytes:
// taken by one call at a time (another allocates its own), replaced by a larger one, given back
// when an allocation of the library's fails for want of memory, by gb_t1_release_memory and when
// the library is unloaded. A call waits for its kernels before it returns, so the memory is idle
// in between.
constexpr size_t kKeepBytes = 64u << 20;
constexpr int kMaxDevices = 64;
struct Kept {
    std::mutex m;
    uint8_t* p = nullptr;
    size_t size = 0;
    bool taken = false;
    ~Kept() {
        if (p) cudaFree(p);
    }
};
Kept& keptOnThisDevice() {
    static Kept kept[kMaxDevices];
    int dev = 0;
    GB_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) throw std::runtime_error("device index out of range");
    return kept[dev];
}

// Gives back what is kept on this device, if no call is using it.
bool giveBack() {
    Kept& k = keptOnThisDevice();
    uint8_t* drop = nullptr;
    {
        std::lock_guard<std::mutex> lock(k.m);
        if (k.taken || !k.p) return false;
        drop = k.p;
        k.p = nullptr;
        k.size = 0;
    }
    GB_CHECK(cudaFree(drop));
    return true;
}

// Codewords come back packed, in runs of at most this many bytes: packed offsets are 32 bits, and a
// call's codewords may be more.
constexpr uint64_t kRunBytes = 64u << 20;

// One piece of device memory in parts, each 256-byte aligned: first the parts' offsets, then the
// memory.
class DeviceParts {
public:
    size_t add(size_t bytes) {
        const size_t at = size_;
        size_ += (bytes + 255) & ~(size_t)255;
        return at;
    }
    void make() {
        {
            std::lock_guard<std::mutex> lock(kept_.m);
            if (!kept_.taken && kept_.size >= size_) {
                kept_.taken = isKept_ = true;
                base_ = kept_.p;
                return;
            }
        }
        GB_CHECK(deviceAlloc((void**)&base_, size_));
    }
    template <class T>
    T* at(size_t offset) const {
        return reinterpret_cast<T*>(base_ + offset);
    }
    DeviceParts() : kept_(keptOnThisDevice()) {}
    ~DeviceParts() {
        uint8_t* drop = base_;
        {
            std::lock_guard<std::mutex> lock(kept_.m);
            if (isKept_) {
                kept_.taken = false;
                drop = nullptr;
            } else if (base_ && !kept_.taken && size_ <= kKeepBytes && size_ > kept_.size) {
                drop = kept_.p;
                kept_.p = base_;
                kept_.size = size_;
            }
        }
        if (drop) cudaFree(drop);
    }
    DeviceParts(const DeviceParts&) = delete;
    DeviceParts& operator=(const DeviceParts&) = delete;

private:
    Kept& kept_;
    uint8_t* base_ = nullptr;
    size_t size_ = 0;
    bool isKept_ = false;
};

}  // namespace

cudaError_t gb::deviceAlloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation && giveBack()) {
        cudaGetLastError();
        e = cudaMalloc(p, bytes);
    }
    return e;
}

extern "C" {

GB_API int gb_t1_release_memory(void) {
    return gbGuard([] { giveBack(); });
}

GB_API int gb_t1_encode_blocks(const uint32_t* coeffs, const int32_t* geom4, uint32_t n, float slope, const float* distScale,
                        uint32_t* info4, uint32_t* passLen, int32_t* passDist, uint8_t* data, uint32_t dataStride) {
    return gbGuard([&] {
        if (!coeffs || !geom4 || !info4 || !passLen || !passDist || !data) throw std::logic_error("null argument");
        if (n == 0) return;
        ensureDevice();
        std::vector<T1Job> jobs(n);
        std::vector<uint64_t> offset(n);
        uint64_t region = 0;
        for (uint32_t i = 0; i < n; ++i) {
            const int w = geom4[4 * i], h = geom4[4 * i + 1], orient = geom4[4 * i + 2], mp = geom4[4 * i + 3];
            if (w < 1 || w > 32 || h < 1 || h > 32 || orient < 0 || orient > 3 || mp < 0 || mp > 64)
                throw std::logic_error("code-block geometry out of range");
            offset[i] = region;
            region += t1SymbolBound(w, h, kMaxPlanes);
        }
        // one piece of memory for everything, kept between calls, and the codewords packed on the
        // device before they come back: their regions are sized for the worst case (56 KB a block),
        // and an allocation per table and a copy of the regions took most of a call's time (64
        // blocks on a B200: 6.0 ms, now 3.1)
        DeviceParts d;
        const size_t tables = (size_t)n * kMaxPasses * 4;
        const size_t oCoeffs = d.add((size_t)n * kCblkArea * 4), oJobs = d.add(n * sizeof(T1Job)), oInfo = d.add(16 * (size_t)n),
                     oEnd = d.add(tables), oLen = d.add(tables), oDist = d.add(tables), oCtl = d.add(64),
                     oSnaps = d.add(4 * tables), oPerm = d.add(4 * (size_t)n), oSlope = d.add(4), oOutInfo = d.add(20 * (size_t)n),
                     oOffsets = d.add(8 * (size_t)n), oSym = d.add(region), oCw = d.add(region);
        d.make();
        for (uint32_t i = 0; i < n; ++i) {
            const int w = geom4[4 * i], h = geom4[4 * i + 1], orient = geom4[4 * i + 2], mp = geom4[4 * i + 3];
            jobs[i] = {d.at<uint32_t>(oCoeffs) + (size_t)i * kCblkArea, d.at<uint8_t>(oSym) + offset[i],
                       d.at<uint8_t>(oCw) + offset[i], t1SymbolBound(w, h, kMaxPlanes), t1Geom(w, h, orient, mp),
                       distScale ? distScale[i] : 1.f, 0, {0, 0}};
        }
        GB_CHECK(cudaMemcpy(d.at<void>(oCoeffs), coeffs, (size_t)n * kCblkArea * 4, cudaMemcpyHostToDevice));
        GB_CHECK(cudaMemcpy(d.at<void>(oJobs), jobs.data(), n * sizeof(T1Job), cudaMemcpyHostToDevice));
        GB_CHECK(cudaMemcpy(d.at<void>(oSlope), &slope, 4, cudaMemcpyHostToDevice));
        // the control words, and before them the pass tables: the kernels write a block's passes alone,
        // and the rest of its rows is 0, not what a call before left
        GB_CHECK(cudaMemset(d.at<void>(oLen), 0, oCtl + 64 - oLen));
        uint32_t* const ctl = d.at<uint32_t>(oCtl);
        T1Launch L{d.at<T1Job>(oJobs), n, d.at<uint32_t>(oInfo), d.at<uint32_t>(oEnd), d.at<uint32_t>(oLen),
                   d.at<int32_t>(oDist), d.at<uint4>(oSnaps), d.at<uint32_t>(oPerm), ctl, d.at<float>(oSlope)};
        t1Encode(L, 0);
        // a run's packed codewords where the decisions were
        auto pack = [&](uint32_t first, uint32_t count) {
            CompactArgs ca{};
            ca.n = count;
            ca.info = d.at<uint32_t>(oInfo) + 4 * (size_t)first;
            ca.jobs = d.at<T1Job>(oJobs) + first;
            ca.outInfo = d.at<uint32_t>(oOutInfo);
            ca.outData = d.at<uint8_t>(oSym);
            ca.tot = ctl + 8;
            ca.dataCap = region;
            ca.scratch = d.at<uint32_t>(oPerm);
            ca.offsets = d.at<uint2>(oOffsets);
            compactTier1(ca, 0);
        };
        const bool whole = region <= kRunBytes;  // one run whatever the codewords' lengths
        if (whole) pack(0, n);
        uint32_t words[16];
        GB_CHECK(cudaMemcpy(words, ctl, 64, cudaMemcpyDeviceToHost));  // waits for the kernels
        if (words[1]) throw std::runtime_error("Tier-1 encoder status " + std::to_string(words[1]));
        GB_CHECK(cudaMemcpy(info4, d.at<void>(oInfo), 16 * (size_t)n, cudaMemcpyDeviceToHost));
        GB_CHECK(cudaMemcpy(passLen, d.at<void>(oLen), tables, cudaMemcpyDeviceToHost));
        GB_CHECK(cudaMemcpy(passDist, d.at<void>(oDist), tables, cudaMemcpyDeviceToHost));
        for (uint32_t first = 0, end; first < n; first = end) {
            uint64_t total = 0;
            end = packedRun(info4, first, n, kRunBytes, total);
            if (!whole) pack(first, end - first);
            const std::unique_ptr<uint8_t[]> cw(new uint8_t[total + 1]);
            if (total) GB_CHECK(cudaMemcpy(cw.get(), d.at<void>(oSym), total, cudaMemcpyDeviceToHost));
            size_t at = 0;  // block i's codeword, each on a 4-byte boundary
            for (uint32_t i = first; i < end; ++i) {
                const uint32_t len = info4[4 * (size_t)i + 3];
                if (len > dataStride) throw std::logic_error("dataStride too small for a codeword");
                std::memcpy(data + (size_t)i * dataStride, cw.get() + at, len);
                at += (len + 3u) & ~3u;
            }
        }
    });
}

GB_API int gb_t1_wait_selftest(uint32_t limitMs, uint32_t* status, float* elapsedMs) {
    return gbGuard([&] {
        if (!status) throw std::logic_error("null argument");
        if (limitMs < 1 || limitMs > 2000) throw std::logic_error("limitMs must be 1..2000");
        ensureDevice();
        *status = t1WaitSelftest(limitMs, elapsedMs);
    });
}

}  // extern "C"
