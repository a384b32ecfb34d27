// Sign-coding and probability tables of EBCOT Tier-1 (ISO/IEC 15444-1 Tables D.3 and C.2), built on
// the host in the packed forms the kernels index (zero-coding contexts, Table D.1, are boolean
// forms in t1_masks.cuh).
#pragma once
#include <cstdint>

namespace gb {

// Sign-coding context and XOR bit from the clamped horizontal and vertical sign
// contributions hc, vc in -1..1 (Table D.3).
inline void scContext(int hc, int vc, int& cx, int& xorbit) {
    if (hc == 0) {
        cx = vc == 0 ? 9 : 10;
        xorbit = vc < 0 ? 1 : 0;
        return;
    }
    const int v = hc > 0 ? vc : -vc;  // the table is symmetric under negating both
    cx = v > 0 ? 13 : (v == 0 ? 12 : 11);
    xorbit = hc < 0 ? 1 : 0;
}

// MQ probability states (Table C.2): Qe, next index after an MPS / LPS, and the switch.
struct MqState {
    uint16_t qe;
    uint8_t nmps, nlps, sw;
};
inline const MqState* mqStates() {
    static const MqState t[47] = {
        {0x5601, 1, 1, 1},   {0x3401, 2, 6, 0},   {0x1801, 3, 9, 0},   {0x0AC1, 4, 12, 0},  {0x0521, 5, 29, 0},
        {0x0221, 38, 33, 0}, {0x5601, 7, 6, 1},   {0x5401, 8, 14, 0},  {0x4801, 9, 14, 0},  {0x3801, 10, 14, 0},
        {0x3001, 11, 17, 0}, {0x2401, 12, 18, 0}, {0x1C01, 13, 20, 0}, {0x1601, 29, 21, 0}, {0x5601, 15, 14, 1},
        {0x5401, 16, 14, 0}, {0x5101, 17, 15, 0}, {0x4801, 18, 16, 0}, {0x3801, 19, 17, 0}, {0x3401, 20, 18, 0},
        {0x3001, 21, 19, 0}, {0x2801, 22, 19, 0}, {0x2401, 23, 20, 0}, {0x2201, 24, 21, 0}, {0x1C01, 25, 22, 0},
        {0x1801, 26, 23, 0}, {0x1601, 27, 24, 0}, {0x1401, 28, 25, 0}, {0x1201, 29, 26, 0}, {0x1101, 30, 27, 0},
        {0x0AC1, 31, 28, 0}, {0x09C1, 32, 29, 0}, {0x08A1, 33, 30, 0}, {0x0521, 34, 31, 0}, {0x0441, 35, 32, 0},
        {0x02A1, 36, 33, 0}, {0x0221, 37, 34, 0}, {0x0141, 38, 35, 0}, {0x0111, 39, 36, 0}, {0x0085, 40, 37, 0},
        {0x0049, 41, 38, 0}, {0x0025, 42, 39, 0}, {0x0015, 43, 40, 0}, {0x0009, 44, 41, 0}, {0x0005, 45, 42, 0},
        {0x0001, 45, 43, 0}, {0x5601, 46, 46, 0},
    };
    return t;
}

// 9 bytes indexed by (hc + 1) * 3 + (vc + 1): context | xor << 5.
inline void signTable(uint8_t* sc) {
    for (int hc = -1; hc <= 1; ++hc)
        for (int vc = -1; vc <= 1; ++vc) {
            int cx, x;
            scContext(hc, vc, cx, x);
            sc[(hc + 1) * 3 + (vc + 1)] = (uint8_t)(cx | (x << 5));
        }
}

// 47 words Qe | switch << 17 | NMPS << 18 | NLPS << 24.
inline void mqTable(uint32_t* mq) {
    const MqState* s = mqStates();
    for (int i = 0; i < 47; ++i)
        mq[i] = (uint32_t)s[i].qe | ((uint32_t)s[i].sw << 17) | ((uint32_t)s[i].nmps << 18) | ((uint32_t)s[i].nlps << 24);
}

}  // namespace gb
