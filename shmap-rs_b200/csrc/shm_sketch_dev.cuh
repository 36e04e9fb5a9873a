// Device pieces shared by the sketch kernels.
#pragma once
#include <stdint.h>

namespace shm {

struct SketchLuts {
    uint64_t fw[256], rc[256], fw_k[256], rc_r1[256], rc_k1[256];
};

// The tables of one k as create_device_luts makes them: the byte tables, and
// for the windows' full hashes a table per group of four bases (SKB kernels):
// wt[g][codes] is what bases 4g .. 4g + 3 of a window XOR into (F, R), as (F
// low, high, R low, high); bases past k contribute nothing.
struct SketchTabs {
    SketchLuts luts;
    uint4 wt[8][256];
};

__device__ __forceinline__ uint64_t u64_of(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }

// Code byte of four letters (the earliest in bits 0-1): the codes sit at
// bits 0-1 of each byte after the shift and mask; the multiply gathers byte
// i's code at bits 24 + 2i with no carry into them from the other products.
__device__ __forceinline__ uint32_t codes4(uint32_t w) { return (((w >> 1) & 0x03030303u) * 0x01041040u) >> 24; }

// Bit i set unless byte i of w is a letter A, C, G or T of either case: the
// byte that a letter of the same code would be (A, C, T, G = 0x41 + 2 code,
// plus 15 for T), against the byte with its case bit cleared.
__device__ __forceinline__ uint32_t bad4(uint32_t w) {
    const uint32_t d = w & 0x06060606u, t = (d >> 2) & ~(d >> 1) & 0x01010101u;
    const uint32_t x = (w & 0xdfdfdfdfu) ^ (0x41414141u + d + 15u * t);
    const uint32_t z = (((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x) & 0x80808080u;  // bit 7 of every byte but zero
    return ((z >> 7) * 0x01020408u) >> 24;
}

}  // namespace shm
