// The sketch on bit planes (SKB_KMIN <= k <= SKB_KMAX): reads' k-mers in any
// order (SK_APPEND), or all sequences' in sequence order (launch_sketch_ordered).
//
// Selection needs only the top bits of a window's hash h = F ^ R to reject
// all but about r of the windows, and each bit of F and R is an XOR of one
// function of each base's code. So a warp evaluates SKB_PL = 8 top bits of
// 32 windows at once, a 32-bit word a bit plane, and forms the full hash only
// of the windows whose top bits are not above the threshold's (1.2% of them
// at r = 0.01).
//
// Layout. A tile is 32 sub-runs of SKB_S = 120 consecutive bases; word j of a
// plane holds base (or window) j of every sub-run, sub-run i in bit i. The
// next base is therefore the next word, with no shifting: lane l holds the
// four words j = 4l - 8 .. 4l - 5 (the first eight words, the bases before
// the sub-runs, only carry the recurrences in; the words past the last
// sub-run position are the first words of the next sub-run, one shift each).
//
// With code(b) = (letter >> 1) & 3 (A, C, T, G = 0..3), code bits p0 and p1
// and w = fw of the letter (src/sketch.rs:50-97), window t's forward hash has
// bit b = XOR_i w(t + i)[b - (K - 1 - i)], its reverse hash bit b = XOR_i
// rc(t + i)[b - i] (bit numbers mod 64), every term a function of (p0, p1):
// one LOP3 with an immediate table. Those K terms are formed for one bit of F
// and one of R; the other planes follow from the rolling step, which moves
// bit b of window t - 1 to bit b + 1 (F) or b - 1 (R) of window t:
//   F_t[b + 1] = F_(t-1)[b] ^ w(t + K - 1)[b + 1] ^ w(t - 1)[b + 1 - K]
//   R_t[b - 1] = R_(t-1)[b] ^ rc(t + K - 1)[b - K] ^ rc(t - 1)[b]
// K is a template parameter because the tables are immediates.
//
// A tile with any byte that is no letter (or a masked base) rolls its
// sub-runs instead, a lane each, eight bases of it in registers at a time and
// the letters' words from five shared entries.
//
// Bound by integer issue, as the rolling kernels were, with a third of their
// instructions: 0.36 warp instructions a base against 1.09 (half of them the
// planes' LOP3s), 2.1 issued a clock of the ~2.4 this mix can reach. 0.46
// Gbases of letters at k = 25, r = 0.01: 0.32 ms, 0.75 ms rolled; the sketch
// of 150,000 hifi reads (3.45 Gbases) 2.3 ms, 5.3 ms rolled. 24 warps an SM
// (80 registers) against 16: 0.35 -> 0.32 ms with the next tile's bytes
// copied asynchronously while a tile is worked on.
#pragma once
#include <utility>

#include "shm_common.cuh"
#include "shm_sketch.cuh"
#include "shm_sketch_dev.cuh"

namespace shm {

constexpr int SKB_S = 120;                 // windows of a sub-run: 30 lanes x 4 words
constexpr int SKB_TILE = 32 * SKB_S;       // windows of a tile
constexpr int SKB_PL = 8;                  // top hash bits tested (the recurrences reach back SKB_PL - 1 = 7 words)
constexpr int SKB_WARPS = 8;
constexpr int SKB_LEAD = 8;                // words before the sub-runs (lanes 0 and 1)
constexpr int SKB_WORDS = 4 + 4 * 32 + 36; // a plane of a tile in shared memory: a pad, the lanes' words, the next sub-run's
constexpr int SKB_Q = 128;                 // queued candidates of a warp
constexpr uint32_t SKB_WAIT = 96;          // rolled windows selected and not yet listed
constexpr int SKB_SPAN = SKB_TILE + 128;   // bases a tile loads: the lead, 32 sub-runs, 120 past them
static_assert(SKB_S == 4 * 32 - SKB_LEAD && SKB_LEAD >= SKB_PL - 1, "lanes cover the lead and the sub-run");
static_assert(SKB_WAIT * 12 <= 2 * SKB_WORDS * 4, "they wait in the planes' place");

// Letter words by code, and their reverse complements' (the constants of src/sketch.rs:60-75).
__host__ __device__ constexpr uint64_t skb_fw(int code) {
    return code == 0 ? 0x3c8bfbb395c60474ULL : code == 1 ? 0x3193c18562a02b4cULL
           : code == 2 ? 0x295549f54be24456ULL : 0x20323ed082572324ULL;
}
__host__ __device__ constexpr uint64_t skb_word(bool rev, int code) { return skb_fw(rev ? code ^ 2 : code); }

// LOP3 table of acc ^ f(p0, p1), f = bit b (mod 64) of the letter's word.
__host__ __device__ constexpr int skb_imm(bool rev, int b) {
    int imm = 0;
    for (int i = 0; i < 8; i++) {
        const int acc = i >> 2, code = ((i >> 1) & 1) | ((i & 1) << 1);
        imm |= (acc ^ (int)((skb_word(rev, code) >> (((b % 64) + 64) % 64)) & 1)) << i;
    }
    return imm;
}
template <int IMM>
__device__ __forceinline__ uint32_t lop3(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(a), "r"(b), "r"(c), "n"(IMM));
    return d;
}
template <bool REV, int B>
__device__ __forceinline__ uint32_t skb_term(uint32_t acc, uint32_t p0, uint32_t p1) {
    return lop3<skb_imm(REV, B)>(acc, p0, p1);
}

template <int V>
struct Int {
    static constexpr int v = V;
};
template <int N, class F, int... I>
__device__ __forceinline__ void static_for_(F&& f, std::integer_sequence<int, I...>) {
    (f(Int<I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
    static_for_<N>(std::forward<F>(f), std::make_integer_sequence<int, N>{});
}

// Candidate masks of a lane's four words: bit i of le[q] is set unless the
// top SKB_PL hash bits of window (sub-run i, word q) are above thr's. pl0 and
// pl1 point at the lane's first word of the tile's planes (shared memory,
// 16-byte aligned).
template <int K>
__device__ __forceinline__ void skb_planes(const uint32_t* pl0, const uint32_t* pl1, uint32_t thr_hi,
                                           uint32_t (&le)[4]) {
    // words -1 .. K + 2 relative to the lane's first: P[x] is word x - 1
    constexpr int NP = K + 4;
    uint32_t P0[NP + 3], P1[NP + 3];
    P0[0] = pl0[-1];
    P1[0] = pl1[-1];
    static_for<(NP - 1 + 3) / 4>([&](auto g_) {
        constexpr int g = decltype(g_)::v;
        const uint4 a = *(const uint4*)(pl0 + 4 * g), b = *(const uint4*)(pl1 + 4 * g);
        constexpr int x = 1 + 4 * g;
        P0[x] = a.x, P1[x] = b.x;
        if constexpr (x + 1 < NP) P0[x + 1] = a.y, P1[x + 1] = b.y;
        if constexpr (x + 2 < NP) P0[x + 2] = a.z, P1[x + 2] = b.z;
        if constexpr (x + 3 < NP) P0[x + 3] = a.w, P1[x + 3] = b.w;
    });
    // bit 63 of R and bit 64 - SKB_PL of F: K terms each
    uint32_t R[SKB_PL][4], F[4];
#pragma unroll
    for (int q = 0; q < 4; q++) R[0][q] = F[q] = 0;
    static_for<K>([&](auto i_) {
        constexpr int i = decltype(i_)::v;
        static_for<4>([&](auto q_) {
            constexpr int q = decltype(q_)::v;
            constexpr int x = 1 + q + i;
            R[0][q] = skb_term<true, 63 - i>(R[0][q], P0[x], P1[x]);
            F[q] = skb_term<false, 64 - SKB_PL - (K - 1 - i)>(F[q], P0[x], P1[x]);
        });
    });
    // R downwards
    static_for<SKB_PL - 1>([&](auto pl_) {
        constexpr int pl = decltype(pl_)::v;
        constexpr int b = 63 - pl;  // from bit b to b - 1
        const uint32_t prev = __shfl_up_sync(0xffffffffu, R[pl][3], 1);
        static_for<4>([&](auto q_) {
            constexpr int q = decltype(q_)::v;
            uint32_t v = q == 0 ? prev : R[pl][q == 0 ? 0 : q - 1];
            v = skb_term<true, b - K>(v, P0[q + K], P1[q + K]);
            R[pl + 1][q] = skb_term<true, b>(v, P0[q], P1[q]);
        });
    });
    // F upwards, and the compare with thr from the lowest plane: a hash bit
    // below thr's makes the window a candidate, above it not, equal keeps
#pragma unroll
    for (int q = 0; q < 4; q++) le[q] = ~0u;
    static_for<SKB_PL>([&](auto pl_) {
        constexpr int pl = decltype(pl_)::v;
        constexpr int b = 64 - SKB_PL + pl;
        const uint32_t tm = 0u - ((thr_hi >> (b - 32)) & 1u);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint32_t h = F[q] ^ R[63 - b][q];
            le[q] = (~h & tm) | (~h & le[q]) | (tm & le[q]);
        }
        if constexpr (pl + 1 < SKB_PL) {
            const uint32_t prev = __shfl_up_sync(0xffffffffu, F[3], 1);
            uint32_t N[4];
            static_for<4>([&](auto q_) {
                constexpr int q = decltype(q_)::v;
                uint32_t v = q == 0 ? prev : F[q == 0 ? 0 : q - 1];
                v = skb_term<false, b + 1>(v, P0[q + K], P1[q + K]);
                N[q] = skb_term<false, b + 1 - K>(v, P0[q], P1[q]);
            });
#pragma unroll
            for (int q = 0; q < 4; q++) F[q] = N[q];
        }
    });
}

__host__ __device__ constexpr uint32_t rot32(uint32_t x, int n) {
    return (n & 31) ? (x << (n & 31)) | (x >> (32 - (n & 31))) : x;
}

// Four words of byte lanes: word G's byte q becomes byte G of out[q].
__device__ __forceinline__ void transpose4(const uint32_t (&y)[4], uint32_t (&out)[4]) {
    const uint32_t a = __byte_perm(y[0], y[1], 0x5140), b = __byte_perm(y[0], y[1], 0x7362);
    const uint32_t c = __byte_perm(y[2], y[3], 0x5140), d = __byte_perm(y[2], y[3], 0x7362);
    out[0] = __byte_perm(a, c, 0x5410);
    out[1] = __byte_perm(a, c, 0x7632);
    out[2] = __byte_perm(b, d, 0x5410);
    out[3] = __byte_perm(b, d, 0x7632);
}

// A lane's four words of windows (of lanes 2 up) that lie in [lo, hi), of a
// tile from t0 that reaches past them. The bases out there read as A, and k As
// can be selected (k = 20 from a ratio of 0.065 on, 26 from 0.022): the full
// hash of every window past the end, one round after another, made a call of
// 77 bases 0.23 ms, 0.06 where they are not. Out of line: most tiles reach
// past nothing.
template <int K>
__device__ __noinline__ uint4 skb_inside(int64_t t0, int64_t lo, int64_t hi) {
    const int at = 4 * ((int)(threadIdx.x & 31) - 2);
    const int from = (int)max(lo - t0, (int64_t)0);                                  // first position
    const int last = (int)min(max(hi - K - t0, (int64_t)-1), (int64_t)SKB_TILE - 1);  // and last one, -1: none
    uint32_t m[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int off = max(at + q, 0);
        const int i0 = off < from ? (from - off + SKB_S - 1) / SKB_S : 0;
        const int i1 = last < off ? 0 : min((last - off) / SKB_S + 1, 32);
        m[q] = i1 > i0 ? (0xffffffffu >> (32 - i1)) & (0xffffffffu << i0) : 0u;
    }
    return make_uint4(m[0], m[1], m[2], m[3]);
}

// The read source of one launch: positions are those of seq_off.
template <bool PK>
struct SkbSource {
    const uint8_t* seq;
    const uint32_t *codes, *mask;
    int64_t lo, hi;      // first base of the first read, end of the last
    int64_t code_bytes;  // readable bytes at codes (packed reads)

    // Where tile 0 starts: at most 63 bases before lo, so that the bytes from
    // SKB_LEAD bases before a tile start at a 16-byte boundary.
    __device__ __forceinline__ int64_t first_tile() const {
        if (PK) return lo - ((lo - SKB_LEAD + 4 * (int64_t)((uintptr_t)codes & 15)) & 63);
        return lo - (int64_t)(((uintptr_t)(seq + lo) - SKB_LEAD) & 15);
    }
    // A tile's bytes (letters, or bytes of four 2-bit codes) from position p =
    // its start - SKB_LEAD into shared memory, SKB_SPAN bases: asynchronous
    // 16-byte copies, or at the ends of the reads plain stores, with bases
    // outside [lo, hi) as A.
    __device__ __forceinline__ void fetch(uint8_t* buf, int64_t p, int lane) const {
        constexpr int BYTES = PK ? SKB_SPAN / 4 : SKB_SPAN;
        const uint8_t* from = PK ? (const uint8_t*)codes + (p >> 2) : seq + p;
        if (PK ? (p >= 0 && (p >> 2) + BYTES <= code_bytes) : (p >= lo && p + BYTES <= hi)) {
            const uint32_t to = (uint32_t)__cvta_generic_to_shared(buf);
            for (int x = 16 * lane; x < BYTES; x += 16 * 32)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + x), "l"(from + x) : "memory");
        } else {
            for (int x = lane; x < BYTES; x += 32) {
                if (PK) buf[x] = (p >> 2) + x >= 0 && (p >> 2) + x < code_bytes ? __ldg(from + x) : (uint8_t)0;
                else buf[x] = p + x >= lo && p + x < hi ? __ldg(from + x) : (uint8_t)0x41;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // Eight bases from p, which is a multiple of 8 from the fetched bytes' start
    // (so they share a word), as indices of the roll entries, four bits each:
    // the code, or 4 for a base that is no letter, masked or outside [lo, hi).
    // Reads only words that hold a base of [lo, hi).
    __device__ __forceinline__ uint32_t eight(int64_t p) const {
        if (p + 8 <= lo || p >= hi) return 0x44444444u;
        const uint32_t out = (p < lo ? 0xffu >> (8 - (int)(lo - p)) : 0u) | (p + 8 > hi ? 0xffu << (int)(hi - p) : 0u);
        uint32_t c, bad;  // two bits a base, one bit a base
        if (PK) {
            c = __ldg(codes + (p >> 4)) >> (2 * (p & 15)) & 0xffffu;
            bad = __ldg(mask + (p >> 5)) >> (p & 31);
        } else {
            uint2 w = make_uint2(0u, 0u);
            if (out == 0) {
                w = __ldg((const uint2*)(seq + p));
            } else {
#pragma unroll 1
                for (int i = (int)max(lo - p, (int64_t)0); i < (int)min(hi - p, (int64_t)8); i++) {
                    const uint32_t x = (uint32_t)__ldg(seq + p + i) << (8 * (i & 3));
                    if (i < 4) w.x |= x;
                    else w.y |= x;
                }
            }
            c = codes4(w.x) | codes4(w.y) << 8;
            bad = bad4(w.x) | bad4(w.y) << 4;
        }
        bad = (bad | out) & 0xffu;
        c = (c | c << 8) & 0x00ff00ffu;  // spread to four bits a base
        c = (c | c << 4) & 0x0f0f0f0fu;
        c = (c | c << 2) & 0x33333333u;
        bad = (bad | bad << 12) & 0x000f000fu;
        bad = (bad | bad << 6) & 0x03030303u;
        bad = (bad | bad << 3) & 0x11111111u;
        return (c & ~(3u * bad)) | bad << 2;
    }
    // Code byte (four bases, the earliest in bits 0-1) of bases p + 4g .. of a
    // window of K bases at p; bases past the window are any (their table
    // entries do not depend on them). Reads only words that hold a base of it.
    template <int K>
    __device__ __forceinline__ void codes_of(int64_t p, uint32_t (&c)[(K + 3) / 4]) const {
        if (PK) {
            const int64_t w0 = p >> 4, wl = (p + K - 1) >> 4;
            const uint32_t sh = 2 * (uint32_t)(p & 15);
            uint32_t w[(K + 15) / 16 + 1];
#pragma unroll
            for (int x = 0; x < (K + 15) / 16 + 1; x++) w[x] = __ldg(codes + min(w0 + x, wl));
#pragma unroll
            for (int g = 0; g < (K + 3) / 4; g++) {
                const uint32_t v = __funnelshift_r(w[g / 4], w[g / 4 + 1], sh);
                c[g] = (v >> (8 * (g & 3))) & 0xffu;
            }
        } else {
            const uintptr_t at = (uintptr_t)(seq + p);
            const uint32_t* w0 = (const uint32_t*)(at & ~(uintptr_t)3);
            const uint32_t sh = 8 * (uint32_t)(at & 3);
            const int wl = (int)((at & 3) + K - 1) >> 2;
            uint32_t lw = __ldg(w0);
#pragma unroll
            for (int g = 0; g < (K + 3) / 4; g++) {
                const uint32_t hw = __ldg(w0 + min(g + 1, wl));
                c[g] = codes4(__funnelshift_r(lw, hw, sh));
                lw = hw;
            }
        }
    }
};

// What a base contributes to a rolled window's hashes (F low, high, R low,
// high) as it enters (side 0) and as it leaves (side 1): entries by code, then
// the one of a base that hashes to 0.
template <int K>
__device__ __forceinline__ uint4 skb_roll_entry(int side, int code) {
    if (code > 3) return make_uint4(0u, 0u, 0u, 0u);
    const uint64_t f = rotl64(skb_fw(code), side ? K : 0), c = skb_fw(code ^ 2);
    const uint64_t r = side ? rotr64(c, 1) : rotl64(c, K - 1);
    return make_uint4((uint32_t)f, (uint32_t)(f >> 32), (uint32_t)r, (uint32_t)(r >> 32));
}

// Bit b of lane a's word to bit a of lane b's.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) {
        const uint32_t m = j == 16 ? 0x0000ffffu : j == 8 ? 0x00ff00ffu : j == 4 ? 0x0f0f0f0fu : j == 2 ? 0x33333333u
                                                                                                 : 0x55555555u;
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
        x = lane & j ? (x & ~m) | ((y & ~m) >> j) : (x & m) | ((y & m) << j);
    }
    return x;
}

template <int K, bool PK>
struct SkbShared {
    uint4 wt[(K + 3) / 4][256];
    uint32_t pl[SKB_WARPS][2][SKB_WORDS];
    uint32_t q[SKB_WARPS][SKB_Q];
    uint8_t tile[SKB_WARPS][PK ? SKB_SPAN / 4 : SKB_SPAN];
    uint4 roll[2][5];  // skb_roll_entry (before the planes: 8,000 ONT-like reads 0.140 ms, here 0.136)
};

// Resident CTAs an SM: three (80 registers a thread), two where the tables of
// more than 28 bases leave shared memory for no more.
template <int K, bool PK>
constexpr int skb_ctas() {
    return 3 * (sizeof(SkbShared<K, PK>) + 1024) <= 228 * 1024 ? 3 : 2;
}

// A tile whose bases are not all letters, by one warp: a lane rolls its
// sub-run of windows from t0 + SKB_S * lane, its bases read once, eight at a
// time as indices into the roll entries (skb_roll_entry, entering then
// leaving); those of the last K bases wait in registers, and the selected
// windows until the warp lists 32 at once. Out of line: its registers are not
// the other tiles'. Bound by integer issue, some 30 instructions a base and
// lane. 60 Mbases of letters with an N every 500, where every tile comes here:
// the sketch 0.19 ms (0.60 with a base read as it entered and again as it
// left, its words looked up in the byte tables, and a list counter's round
// trip for every selected window), 0.054 without the Ns.
// `wait`: the warp's planes, SKB_WAIT selected windows (not ORD). Returns
// ord_n and the tile's selected windows.
template <int K, bool PK, bool ORD>
__device__ __noinline__ uint32_t skb_roll_tile(const SketchArgs& a, SkbSource<PK> src, const uint4* entries,
                                               uint32_t* wait, int64_t t0, int64_t base, int32_t q_tile,
                                               uint64_t ord_base, uint32_t ord_cap, uint32_t ord_n) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint64_t thr = a.thr;
    const uint32_t thr_hi = (uint32_t)(thr >> 32);
    const int64_t s0 = t0 + SKB_S * lane;
    const int w0 = (int)min(max(src.lo - s0, (int64_t)0), (int64_t)SKB_S);
    const int w1 = (int)min(max(src.hi - s0, (int64_t)0), (int64_t)SKB_S);
    auto rs_of = [&](int64_t p, int32_t q, bool strand) {
        return ((uint32_t)((int32_t)(p - __ldg(a.seq_off + q)) + K - 1 + a.r_offset) << 1) | (strand ? 1u : 0u);
    };
    // each(window, selected, F, R) is called by all lanes together, for every
    // window of the sub-run that is selected in some lane
    auto roll = [&](auto&& each) {
        constexpr int BACK = (K + 7) / 8;  // words of eight bases to the first that leaves with this one's
        uint32_t W[BACK + 1];
#pragma unroll
        for (int x = 0; x <= BACK; x++) W[x] = 0x44444444u;  // (before the first base: none)
        uint32_t flo = 0, fhi = 0, rlo = 0, rhi = 0;
#pragma unroll 1
        for (int b0 = 0; b0 < SKB_S + K - 1; b0 += 8) {
#pragma unroll
            for (int x = 0; x < BACK; x++) W[x] = W[x + 1];
            W[BACK] = src.eight(s0 + b0);
            uint32_t in = W[BACK], out = K % 8 ? __funnelshift_r(W[0], W[1], 4 * (8 - K % 8)) : W[0];
#pragma unroll 1
            for (int b = b0; b < b0 + 8; b++) {
                const uint4 e = entries[in & 7u], l = entries[5 + (out & 7u)];
                in >>= 4;
                out >>= 4;
                const uint32_t f0 = __funnelshift_l(fhi, flo, 1), r0 = __funnelshift_r(rlo, rhi, 1);
                fhi = __funnelshift_l(flo, fhi, 1) ^ e.y ^ l.y;
                flo = f0 ^ e.x ^ l.x;
                rhi = __funnelshift_r(rhi, rlo, 1) ^ e.w ^ l.w;
                rlo = r0 ^ e.z ^ l.z;
                if (__ballot_sync(FULL, (fhi ^ rhi) <= thr_hi) == 0) continue;
                const uint64_t f = u64_of(flo, fhi), r = u64_of(rlo, rhi);
                const int w = b - (K - 1);
                each(w, (f ^ r) <= thr && w >= w0 && w < w1, f, r);
            }
        }
    };
    if (ORD) {
        // counted first, for the lanes' places, then written (a lane's windows ascend)
        int32_t q = q_tile;
        auto whole = [&](int w) {  // window w of the lane's sub-run lies in one sequence, q
            const int64_t p = s0 + w;
            while (__ldg(a.seq_off + q + 1) <= p) q++;  // ends: p < hi = seq_off[n_seq]
            return p + K <= __ldg(a.seq_off + q + 1);
        };
        uint32_t mine = 0;
        roll([&](int w, bool sel, uint64_t, uint64_t) {
            if (sel && whole(w)) {
                mine++;
                if (a.ord_seq_cnt) atomicAdd(a.ord_seq_cnt + q, 1u);
            }
        });
        __syncwarp();
        const uint32_t inc = warp_inclusive_scan(mine);
        uint32_t slot = ord_n + inc - mine;
        q = q_tile;
        if (ord_cap)
            roll([&](int w, bool sel, uint64_t f, uint64_t r) {
                if (sel && whole(w)) {
                    if (slot < ord_cap) {
                        a.out_h[ord_base + slot] = f ^ r;
                        a.out_rs[ord_base + slot] = rs_of(s0 + w, q, f > r);
                    }
                    slot++;
                }
            });
        return ord_n + __shfl_sync(FULL, inc, 31);
    }
    // the selected windows wait until there are enough for the whole warp
    // (their positions relative to base | strand << 31)
    uint64_t* const wh = (uint64_t*)wait;
    uint32_t* const wp = (uint32_t*)(wh + SKB_WAIT);
    uint32_t nw = 0;
    auto list = [&](uint32_t b, uint32_t n) {  // (as take of k_sketch_bits, from q_tile on, the hashes known)
        const bool act = (uint32_t)lane < n;
        const uint32_t e = act ? wp[b + lane] : 0u, rel = e & 0x7fffffffu;
        const int64_t p = base + rel, pmax = base + __reduce_max_sync(FULL, rel);
        int32_t q = q_tile;
        for (int32_t q1 = q_tile + 1;; q1 += 32) {
            const int64_t s = q1 + lane <= a.n_seq ? __ldg(a.seq_off + q1 + lane) : INT64_MAX;
            const int nle = __popc(__ballot_sync(FULL, s <= pmax));
            for (int x = 0; x < nle; x++) q += __shfl_sync(FULL, s, x) <= p ? 1 : 0;
            if (nle < 32) break;
        }
        const bool sel = act && p + K <= __ldg(a.seq_off + min(q, a.n_seq - 1) + 1);
        const unsigned peers = __match_any_sync(FULL, sel ? q : -1);
        const int leader = __ffs(peers) - 1;
        uint32_t at = 0;
        if (sel && lane == leader) at = atomicAdd(a.kmer_cnt + q, (uint32_t)__popc(peers));
        at = __shfl_sync(FULL, at, leader) + __popc(peers & ((1u << lane) - 1u));
        if (sel) {
            const uint64_t o = __ldg(a.kmer_off + q);
            if (at < (uint32_t)(__ldg(a.kmer_off + q + 1) - o)) {
                a.out_h[o + at] = wh[b + lane];
                a.out_rs[o + at] = rs_of(p, q, e >> 31);
            }
        }
    };
    roll([&](int w, bool sel, uint64_t f, uint64_t r) {
        const unsigned bal = __ballot_sync(FULL, sel);
        if (sel) {
            const uint32_t at = nw + __popc(bal & ((1u << lane) - 1u));
            wh[at] = f ^ r;
            wp[at] = (uint32_t)(s0 + w - base) + (f > r ? 1u << 31 : 0u);
        }
        nw += __popc(bal);
        if (nw > SKB_WAIT - 32) {
            __syncwarp();
            while (nw >= 32) list(nw -= 32, 32);
            __syncwarp();
        }
    });
    __syncwarp();
    for (uint32_t b = 0; b < nw; b += 32) list(b, min(32u, nw - b));
    return ord_n;
}

// ORD: the k-mers of a warp's tiles in sequence order, counted in
// a.ord_cnt[warp] and written (as many as there is room for) from
// a.ord_off[warp] to a.ord_off[warp + 1], or with no ord_off from warp *
// a.ord_stride; a.ord_seq_cnt[q] (unless null) counts those of sequence q. The
// candidate masks are transposed first, so that lane i holds sub-run i's and
// the queue fills in order.
template <int K, bool PK, bool ORD>
__global__ void __launch_bounds__(SKB_WARPS * 32, skb_ctas<K, PK>()) k_sketch_bits(const __grid_constant__ SketchArgs a,
                                                                          const SketchTabs* __restrict__ tabs) {
    constexpr int NG = (K + 3) / 4;
    extern __shared__ __align__(16) uint8_t skb_smem[];
    SkbShared<K, PK>& sm = *(SkbShared<K, PK>*)skb_smem;
    auto& s_wt = sm.wt;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned FULL = 0xffffffffu;
    uint32_t* const pl0 = sm.pl[wib][0];
    uint32_t* const pl1 = sm.pl[wib][1];
    uint32_t* const queue = sm.q[wib];
    uint8_t* const buf = sm.tile[wib];
    SkbSource<PK> src{a.seq, a.pk_codes, a.pk_mask, a.base0, a.base1, (int64_t)(4 * a.pk_words)};
    const int64_t lo = a.base0, hi = a.base1;
    const int64_t T0 = src.first_tile();
    const uint64_t thr = a.thr;
    const uint32_t thr_hi = (uint32_t)(thr >> 32);
    // a contiguous share of the tiles for every warp
    const int64_t n_tiles = (hi - T0 + SKB_TILE - 1) / SKB_TILE;
    const int64_t gw = (int64_t)blockIdx.x * SKB_WARPS + wib, nw = (int64_t)gridDim.x * SKB_WARPS;
    const int64_t t_first = gw * n_tiles / nw, t_end = (gw + 1) * n_tiles / nw;
    const bool any = t_first < t_end;
    const int64_t base = T0 + t_first * SKB_TILE;  // queue entries are positions relative to it
    // the tables and the first tile arrive while the warp looks its read up
    for (int i = threadIdx.x; i < NG * 256; i += SKB_WARPS * 32)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(&s_wt[0][0] + i)),
                     "l"(&tabs->wt[0][0] + i)
                     : "memory");
    if (threadIdx.x < 10) sm.roll[threadIdx.x / 5][threadIdx.x % 5] = skb_roll_entry<K>(threadIdx.x / 5, threadIdx.x % 5);
    if (any) src.fetch(buf, base - SKB_LEAD, lane);
    int32_t q_tile = warp_last_le((const uint64_t*)a.seq_off, a.n_seq, (uint64_t)min(max(base, lo), hi), lane);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (!any) {
        if (ORD && lane == 0) a.ord_cnt[gw] = 0;
        return;
    }
    // ORD: where the warp's k-mers go, and how many there were so far
    uint64_t ord_base = 0;
    uint32_t ord_cap = 0, ord_n = 0;
    if (ORD) {
        ord_base = a.ord_off ? (uint64_t)a.ord_off[gw] : (uint64_t)gw * a.ord_stride;
        ord_cap = a.ord_off ? a.ord_off[gw + 1] - a.ord_off[gw] : a.ord_stride;
    }
    int32_t q_queue = q_tile;  // no queued candidate's read comes before it
    uint32_t qn = 0;

    // The candidates queue[b + lane] (lane < n): their full hashes, and the
    // selected ones to their reads' lists.
    auto take = [&](uint32_t b, uint32_t n) {
        const bool act = (uint32_t)lane < n;
        const uint32_t rel = act ? queue[b + lane] : 0u;
        const int64_t p = base + rel;
        const int64_t pmax = base + __reduce_max_sync(FULL, rel);
        // its read: the starts after q_queue, 32 at a time, until past the last candidate
        int32_t q = q_queue;
        for (int32_t q1 = q_queue + 1;; q1 += 32) {
            const int64_t s = q1 + lane <= a.n_seq ? __ldg(a.seq_off + q1 + lane) : INT64_MAX;
            const int nle = __popc(__ballot_sync(FULL, s <= pmax));  // starts ascend
            for (int x = 0; x < nle; x++) q += __shfl_sync(FULL, s, x) <= p ? 1 : 0;
            if (nle < 32) break;
        }
        uint64_t h = 0;
        uint32_t rs = 0;
        bool sel = false;
        if (act && p >= lo && q < a.n_seq && p + K <= __ldg(a.seq_off + q + 1)) {
            uint32_t c[NG];
            src.template codes_of<K>(p, c);
            uint4 st = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int g = 0; g < NG; g++) {
                const uint4 t = s_wt[g][c[g]];
                st.x ^= t.x;
                st.y ^= t.y;
                st.z ^= t.z;
                st.w ^= t.w;
            }
            const uint64_t f = u64_of(st.x, st.y), r = u64_of(st.z, st.w);
            h = f ^ r;
            sel = h <= thr;
            rs = ((uint32_t)((int32_t)(p - __ldg(a.seq_off + q)) + K - 1 + a.r_offset) << 1) | (f > r ? 1u : 0u);
        }
        const unsigned peers = __match_any_sync(FULL, sel ? q : -1);
        const int leader = __ffs(peers) - 1;
        if (ORD) {
            const unsigned bal = __ballot_sync(FULL, sel);
            const uint32_t slot = ord_n + __popc(bal & ((1u << lane) - 1u));
            if (sel && slot < ord_cap) {
                a.out_h[ord_base + slot] = h;
                a.out_rs[ord_base + slot] = rs;
            }
            if (sel && lane == leader && a.ord_seq_cnt) atomicAdd(a.ord_seq_cnt + q, (uint32_t)__popc(peers));
            ord_n += __popc(bal);
            return;
        }
        uint32_t at = 0;
        if (sel && lane == leader) at = atomicAdd(a.kmer_cnt + q, (uint32_t)__popc(peers));
        at = __shfl_sync(FULL, at, leader) + __popc(peers & ((1u << lane) - 1u));
        if (sel) {
            const uint64_t o = __ldg(a.kmer_off + q);
            if (at < (uint32_t)(__ldg(a.kmer_off + q + 1) - o)) {
                a.out_h[o + at] = h;
                a.out_rs[o + at] = rs;
            }
        }
    };

    for (int64_t tl = t_first; tl < t_end; tl++) {
        const int64_t t0 = T0 + tl * SKB_TILE;
        for (;;) {  // the read of the tile's first base
            const int64_t s = q_tile + 1 + lane <= a.n_seq ? __ldg(a.seq_off + q_tile + 1 + lane) : INT64_MAX;
            const int nle = __popc(__ballot_sync(FULL, s <= t0));
            q_tile += nle;
            if (nle < 32) break;
        }
        if (qn == 0) q_queue = q_tile;
        // 33 sub-runs (the last for the words past the others' ends), a lane's
        // four words of each
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        auto four = [&](int i) {
            return PK ? (uint32_t)buf[SKB_S / 4 * i + lane] : *(const uint32_t*)(buf + SKB_S * i + 4 * lane);
        };
        uint32_t bad = 0;
        uint32_t y0[4], y1[4];
        if (PK) {
            // masked bases in the tile's reach
            const int64_t b = max(t0, lo), e = min(t0 + SKB_TILE + K, hi);
            for (int64_t m = (b >> 5) + lane; m <= (e - 1) >> 5; m += 32) {
                uint32_t v = __ldg(a.pk_mask + m);
                if (m == b >> 5) v &= ~0u << (b & 31);
                if (m == (e - 1) >> 5) v &= ~0u >> (31 - ((e - 1) & 31));
                bad |= v;
            }
            // a byte's four 2-bit codes to bits 0-1 of four bytes (two multiplies
            // by sums of powers of two, no copies meet), code bits of sub-run i to bit i
#pragma unroll
            for (int G = 0; G < 4; G++) {
                uint32_t lo0 = 0, hi1 = 0, top1 = 0;
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const uint32_t t = (four(8 * G + u) * 0x1001u) & 0x000f000fu, z = t * (0x41u << u);
                    lo0 |= z & (0x01010101u << u);
                    if (u < 7) hi1 |= z & (0x02020202u << u);
                    else top1 = (t * (0x41u << 6)) & 0x80808080u;
                }
                y0[G] = lo0;
                y1[G] = (hi1 >> 1) | top1;
            }
        } else {
            // code bits 1 and 2 of each letter to byte q, bit i, from one rotation
            // a word (bit 2 lands one place higher: turned back per group); bits
            // 0 and 4 too, for the check: a letter has bit 7 = 0, 6 = 1, 3 = 0,
            // bit 4 = bit 2 & ~bit 1 and bit 0 = ~bit 4 (A 41, C 43, T 54, G 47
            // hex, bit 5 is the case)
            uint32_t b1 = 0;
#pragma unroll
            for (int G = 0; G < 4; G++) {
                uint32_t c1 = 0, c2 = 0, c0 = 0, c4 = 0;
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const uint32_t x = four(8 * G + u), t = __funnelshift_l(x, x, (u + 31) & 31);
                    c1 |= t & rot32(0x01010101u, u);
                    c2 |= t & rot32(0x01010101u, u + 1);
                    c0 |= t & rot32(0x01010101u, u + 31);
                    c4 |= t & rot32(0x01010101u, u + 3);
                    b1 |= x ^ 0x40404040u;
                }
                y0[G] = c1;
                y1[G] = __funnelshift_r(c2, c2, 1);
                c0 = __funnelshift_l(c0, c0, 1);
                c4 = __funnelshift_r(c4, c4, 3);
                bad |= (c4 ^ (y1[G] & ~c1)) | ~(c0 ^ c4);
            }
            const uint32_t x = four(32);  // the last word's letters by themselves
            bad |= ((b1 | (x ^ 0x40404040u)) & 0xc8c8c8c8u) |
                   (((x ^ ((x << 2) & ~(x << 3))) | ~(x ^ (x << 4))) & 0x10101010u);
        }
        const uint32_t past = four(32);
        __syncwarp();  // the buffer is free: the next tile's bytes arrive while this one is worked on
        if (tl + 1 < t_end) src.fetch(buf, t0 + SKB_TILE - SKB_LEAD, lane);
        uint32_t le[4] = {0u, 0u, 0u, 0u};
        if (__builtin_expect(__any_sync(FULL, bad != 0), 0)) {
            if (ORD) {
                if (qn) take(0, qn);  // the tiles before come first
                qn = 0;
            }
            __syncwarp();
            ord_n = skb_roll_tile<K, PK, ORD>(a, src, sm.roll[0], pl0, t0, base, q_tile, ord_base, ord_cap, ord_n);
            __syncwarp();
        } else {
            uint32_t o0[4], o1[4];
            transpose4(y0, o0);
            transpose4(y1, o1);
            *(uint4*)(pl0 + 4 + 4 * lane) = make_uint4(o0[0], o0[1], o0[2], o0[3]);
            *(uint4*)(pl1 + 4 + 4 * lane) = make_uint4(o1[0], o1[1], o1[2], o1[3]);
            if (lane >= 2 && lane < 11) {  // words SKB_S + x of the sub-runs: words x of the next ones
                uint32_t e0[4], e1[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const uint32_t c = PK ? (past >> (2 * q)) & 3u : (past >> (8 * q + 1)) & 3u;
                    e0[q] = (o0[q] >> 1) | (c << 31);
                    e1[q] = (o1[q] >> 1) | ((c >> 1) << 31);
                }
                *(uint4*)(pl0 + 4 + SKB_S + 4 * lane) = make_uint4(e0[0], e0[1], e0[2], e0[3]);
                *(uint4*)(pl1 + 4 + SKB_S + 4 * lane) = make_uint4(e1[0], e1[1], e1[2], e1[3]);
            }
            __syncwarp();
            skb_planes<K>(pl0 + 4 + 4 * lane, pl1 + 4 + 4 * lane, thr_hi, le);
            if (lane < 2) le[0] = le[1] = le[2] = le[3] = 0;
            if (__builtin_expect(t0 < lo || t0 + SKB_TILE + K - 1 > hi, 0)) {
                const uint4 in = skb_inside<K>(t0, lo, hi);
                le[0] &= in.x, le[1] &= in.y, le[2] &= in.z, le[3] &= in.w;
            }
        }
        // the candidates to the queue; full rounds of 32 are taken at once, the
        // rest with the next tile's (or now, after the last tile)
        const uint32_t rel0 =
            (uint32_t)(t0 - base) - (uint32_t)SKB_LEAD + (ORD ? (uint32_t)SKB_S : 4u) * (uint32_t)lane;
        if (ORD) {
#pragma unroll
            for (int q = 0; q < 4; q++) le[q] = transpose32(le[q], lane);
        }
        for (bool more = true; more;) {
            const uint32_t cnt = __popc(le[0]) + __popc(le[1]) + __popc(le[2]) + __popc(le[3]);
            const uint32_t inc = warp_inclusive_scan(cnt), total = __shfl_sync(FULL, inc, 31);
            uint32_t at = qn + inc - cnt;
            if (ORD) {
                for (uint32_t l; (l = le[0] | le[1] | le[2] | le[3]) != 0 && at < (uint32_t)SKB_Q;) {
                    const uint32_t bit = l & (0u - l);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if ((le[q] & bit) && at < (uint32_t)SKB_Q) {
                            queue[at++] = rel0 + 4u * (uint32_t)(__ffs(bit) - 1) + (uint32_t)q;
                            le[q] &= ~bit;
                        }
                }
            }
            if (!ORD) {
#pragma unroll
                for (int q = 0; q < 4; q++)
                    while (le[q] != 0 && at < (uint32_t)SKB_Q) {
                        queue[at++] = rel0 + (uint32_t)q + (uint32_t)SKB_S * (uint32_t)(__ffs(le[q]) - 1);
                        le[q] &= le[q] - 1;
                    }
            }
            more = qn + total > (uint32_t)SKB_Q;
            const uint32_t have = min(qn + total, (uint32_t)SKB_Q);
            const uint32_t upto = !more && tl + 1 == t_end ? have : have & ~31u;
            __syncwarp();
#pragma unroll 1
            for (uint32_t b = 0; b < upto; b += 32) take(b, min(32u, have - b));
            qn = have - upto;
            if (upto && qn) {
                const uint32_t v = queue[upto + min((uint32_t)lane, qn - 1)];
                __syncwarp();
                if ((uint32_t)lane < qn) queue[lane] = v;
                q_queue = q_tile;
            }
            __syncwarp();
        }
    }
    if (ORD && lane == 0) a.ord_cnt[gw] = ord_n;
}

}  // namespace shm
