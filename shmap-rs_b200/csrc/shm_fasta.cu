// FASTA parsed on the device. The reference reads its inputs with needletail
// (src/io/mod.rs:383-427): a record per '>' header, the id cut at the first
// space or tab, the sequence the record's lines joined without their line
// ends. The command line's host reader (host/shmap_cli.cpp read_fastx) states
// those byte rules, and this parser keeps them exactly. Lines end at '\n'.
// One '\r' right before a line's end is dropped. A line whose first byte is
// '>' is a header, and every other line after the first header belongs to
// the current record, empty lines included. It declines a FASTA file that
// has a line starting with '@' or a non-empty line before the first header
// (which the host reader reports as an error), so such files go to the host
// reader. A file whose first byte is '@' is FASTQ: records of four lines
// (header, sequence, '+', quality), parsed by line index (see the FASTQ
// passes below).
//
// The file's bytes are processed in chunks of CHUNK bytes, one CTA per chunk,
// each thread taking 64 consecutive bytes as a mask of its line ends, so that
// the work goes by lines and not by bytes:
//  1. per chunk: the bytes kept, the headers and what else depends on how the
//     chunk's first line began, for every way it can have begun (FASTA: not in
//     a header, and how much less if it is one; FASTQ: the four line roles);
//  2. one block carries the state over the chunks, picks each chunk's counts
//     and scans them;
//  3. per chunk: the kept bytes compacted through shared memory and stored
//     coalesced at their place; each header's position and the number of
//     sequence bytes before it;
//  4. per header: its name's length, then (after a scan) the name itself.
// Not bound by memory: 125 MB of 100-base lines are counted in 0.061 ms and
// written in 0.129, at 2.1 and 1.9 TB/s of the 6.5 a copy reaches. Both passes
// issue in 61 to 71% of the cycles (0.31 and 0.75 warp instructions a byte:
// the masks and the per-line steps) and wait at the barriers of the chunk's
// scans; the carry between them, 0.037 ms, is one block's chain of loads over
// the chunks. (Byte by byte, in three passes over chunks staged by single
// bytes, 249 MB in two files took 6.5 ms; now 0.43.)
#include <cstring>
#include <string>
#include <vector>

#include "shm_common.cuh"
#include "shm_fasta.hpp"
#include "shm_internal.hpp"
#include "../host/utf8.hpp"
#include "shm_prims.cuh"

namespace shm {

namespace {

constexpr int FA_THREADS = 256;
constexpr int64_t CHUNK = (int64_t)FA_THREADS * 64;

enum : uint32_t { FA_FASTQ = 1u, FA_TEXT_BEFORE_HEADER = 2u, FQ_BAD = 4u };

struct FaView {
    const uint8_t* d;  // the file's bytes, 16-byte aligned, readable to the next multiple of 64
    int64_t len;
    int64_t n_chunks;
};

template <class T, class Op>
__device__ T block_scan_excl_op(T x, T ident, Op op, T* sh, T* total) {
    // exclusive scan with an associative op over the block's threads (in order)
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    T inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc = op(inc, y);
    }
    if (lane == 31) sh[w] = inc;
    __syncthreads();
    if (w == 0) {
        T t = lane < nw ? sh[lane] : ident;
        T ti = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, ti, o);
            if (lane >= o) ti = op(ti, y);
        }
        if (lane < nw) sh[lane] = ti;  // inclusive over warps
        if (lane == nw - 1) *total = ti;
    }
    __syncthreads();
    const T before_warp = w ? sh[w - 1] : ident;
    T excl = __shfl_up_sync(0xffffffffu, inc, 1);
    excl = lane ? op(before_warp, excl) : before_warp;
    __syncthreads();
    return excl;
}

struct MaxOp {
    template <class T>
    __device__ T operator()(T a, T b) const { return a > b ? a : b; }
};
struct SumOp {
    template <class T>
    __device__ T operator()(T a, T b) const { return a + b; }
};

// Bit j of the result for byte j of w equal to the byte repeated in pat.
__device__ __forceinline__ uint32_t eq4(uint32_t w, uint32_t pat) {
    const uint32_t x = w ^ pat;
    const uint32_t z = ~(((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x) & 0x80808080u;  // bit 7 of every zero byte
    return ((z >> 7) * 0x01020408u) >> 24 & 0xfu;
}

// A thread's 64 bytes from file position a: bit j is byte a + j.
struct Bytes64 {
    uint64_t valid;  // inside the file
    uint64_t nl;     // '\n'
    uint64_t start;  // first bytes of lines
    uint64_t cr;     // '\r' dropped before its line's end
};

// Every thread of the block calls this for its run of the chunk; the words go
// to `keep` too (16 of them) when it is not null.
__device__ __forceinline__ Bytes64 load64(const FaView& v, int64_t a, uint32_t* keep) {
    const int lane = threadIdx.x & 31;
    Bytes64 r;
    const int64_t left = v.len - a;
    r.valid = left >= 64 ? ~0ULL : left > 0 ? (1ULL << left) - 1 : 0ULL;
    uint32_t n0 = 0, n1 = 0, c0 = 0, c1 = 0;
    if (left > 0) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint4 u = __ldg((const uint4*)(v.d + a) + i);
            w[4 * i] = u.x, w[4 * i + 1] = u.y, w[4 * i + 2] = u.z, w[4 * i + 3] = u.w;
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            n0 |= eq4(w[i], 0x0a0a0a0au) << (4 * i);
            n1 |= eq4(w[8 + i], 0x0a0a0a0au) << (4 * i);
            c0 |= eq4(w[i], 0x0d0d0d0du) << (4 * i);
            c1 |= eq4(w[8 + i], 0x0d0d0d0du) << (4 * i);
        }
        if (keep)
#pragma unroll
            for (int i = 0; i < 16; i++) keep[i] = w[i];
    }
    r.nl = ((uint64_t)n1 << 32 | n0) & r.valid;
    const uint64_t cr = ((uint64_t)c1 << 32 | c0) & r.valid;
    // the byte before the run and the one after it
    uint32_t before = __shfl_up_sync(0xffffffffu, (uint32_t)(r.nl >> 63), 1);
    if (lane == 0) before = a == 0 ? 1u : a <= v.len ? (uint32_t)(v.d[a - 1] == '\n') : 0u;
    uint32_t after = __shfl_down_sync(0xffffffffu, (uint32_t)(r.nl & 1), 1);
    if (lane == 31) after = a + 64 < v.len ? (uint32_t)(v.d[a + 64] == '\n') : 0u;
    r.start = (r.nl << 1 | before) & r.valid;
    if (left == 64) after = 1u;  // a '\r' that ends the file is dropped too
    r.cr = cr & (r.nl >> 1 | (uint64_t)after << 63 | (left > 0 && left < 64 ? 1ULL << (left - 1) : 0ULL));
    return r;
}

// Calls f(segment mask, index in the run, whether it starts a line, its first
// position) for each part of a line in the run, in order (the part before the
// run's first line start, if any, has index 0).
template <class F>
__device__ __forceinline__ void each_line(const Bytes64& r, F&& f) {
    uint64_t rest = r.valid, st = r.start;
    int n = 0;
    if (!(st & 1) && rest) {
        const uint64_t seg = st ? rest & ((st & (0 - st)) - 1) : rest;
        f(seg, n++, false, 0);
        rest &= ~seg;
    }
    while (st) {
        const int at = __ffsll((long long)st) - 1;
        st &= st - 1;
        const uint64_t seg = st ? rest & ((st & (0 - st)) - 1) : rest;
        f(seg, n++, true, at);
        rest &= ~seg;
    }
}

// What a chunk counted, for every state its first line can be in.
struct ChunkSum {
    uint32_t kept[4], hdr[4];  // FASTQ: with its first line's role r; FASTA: kept[0] and hdr[0], no header coming in
    uint32_t prefix;           // FASTA: of kept[0], before the chunk's first line start
    uint32_t lines;            // FASTQ: line ends
    uint8_t last;              // FASTA: the last line start (0 none, 1 text, 2 header)
    uint8_t text;              // FASTA: bytes kept before the chunk's first header
    uint8_t not_at, not_plus;  // FASTQ: bit r: with role r of its first line, a line of role 0 / 2 begins otherwise
};

// Pass 1.
template <bool FQ>
__global__ void __launch_bounds__(FA_THREADS) k_fa_count(FaView v, ChunkSum* __restrict__ sums,
                                                       uint32_t* __restrict__ flags) {
    __shared__ int32_t sh[32];
    __shared__ int32_t tot;
    __shared__ uint32_t s_kept[4], s_hdr[4], s_prefix, s_not[2], s_text;
    for (int64_t c = blockIdx.x; c < v.n_chunks; c += gridDim.x) {
        const int64_t a = c * CHUNK + (int64_t)threadIdx.x * 64;
        if (threadIdx.x < 4) s_kept[threadIdx.x] = s_hdr[threadIdx.x] = 0;
        if (threadIdx.x == 4) s_prefix = s_not[0] = s_not[1] = s_text = 0;
        const Bytes64 r = load64(v, a, nullptr);
        const uint64_t text = r.valid & ~r.nl & ~r.cr;
        if (FQ) {
            // line ends before the run in the chunk: its first byte's line, counted from the chunk's first
            const int32_t l0 = block_scan_excl_op<int32_t>(__popcll(r.nl), 0, SumOp(), sh, &tot);
            uint32_t kept[4] = {0, 0, 0, 0}, hdr[4] = {0, 0, 0, 0}, na = 0, np = 0;
            int32_t line = l0;
            each_line(r, [&](uint64_t seg, int, bool starts, int at) {
                const uint32_t k = __popcll(seg & text);
                const int res = line & 3;  // role of this line = first line's role + res
#pragma unroll
                for (int ro = 0; ro < 4; ro++) {
                    const int role = (ro + res) & 3;
                    if (role == 1) kept[ro] += k;
                    if (starts && role == 0) {
                        const uint8_t ch = v.d[a + at];
                        if (ch != '\n') {
                            hdr[ro] += ch == '@';
                            if (ch != '@') na |= 1u << ro;
                        }
                    }
                    if (starts && role == 2) {
                        const uint8_t ch = v.d[a + at];
                        if (ch != '\n' && ch != '+') np |= 1u << ro;
                    }
                }
                line += (seg & r.nl) != 0;
            });
#pragma unroll
            for (int ro = 0; ro < 4; ro++) {
                const uint32_t k = __reduce_add_sync(0xffffffffu, kept[ro]), h = __reduce_add_sync(0xffffffffu, hdr[ro]);
                if ((threadIdx.x & 31) == 0) {
                    if (k) atomicAdd(&s_kept[ro], k);
                    if (h) atomicAdd(&s_hdr[ro], h);
                }
            }
            if (na) atomicOr(&s_not[0], na);
            if (np) atomicOr(&s_not[1], np);
            __syncthreads();
            if (threadIdx.x == 0) {
                ChunkSum o{};
                for (int ro = 0; ro < 4; ro++) {
                    o.kept[ro] = s_kept[ro];
                    o.hdr[ro] = s_hdr[ro];
                }
                o.lines = (uint32_t)tot;
                o.not_at = (uint8_t)s_not[0];
                o.not_plus = (uint8_t)s_not[1];
                sums[c] = o;
            }
        } else {
            // the run's last line start, as (thread + 1) * 4 + (1 text, 2 header)
            int32_t mine = 0;
            uint32_t hdrs = 0, fl = 0;
            for (uint64_t st = r.start; st; st &= st - 1) {
                const uint8_t ch = v.d[a + __ffsll((long long)st) - 1];
                mine = ((int32_t)threadIdx.x + 1) * 4 + (ch == '>' ? 2 : 1);
                hdrs += ch == '>';
                if (ch == '@') fl = FA_FASTQ;
            }
            if (fl) atomicOr(flags, fl);
            const int32_t in = block_scan_excl_op<int32_t>(mine, 0, MaxOp(), sh, &tot);
            const int32_t last = tot;
            const bool any_before = block_scan_excl_op<int32_t>(hdrs != 0 ? 1 : 0, 0, MaxOp(), sh, &tot) != 0;
            uint32_t kept = 0, prefix = 0, early = 0;
            bool hdr = (in & 3) == 2, open = any_before;
            each_line(r, [&](uint64_t seg, int, bool starts, int at) {
                if (starts) hdr = v.d[a + at] == '>';
                open = open || (starts && hdr);
                if (hdr) return;
                const uint32_t k = __popcll(seg & text);
                kept += k;
                if (!starts && in == 0) prefix += k;  // before the chunk's first line start
                if (!open) early += k;
            });
            kept = __reduce_add_sync(0xffffffffu, kept);
            prefix = __reduce_add_sync(0xffffffffu, prefix);
            hdrs = __reduce_add_sync(0xffffffffu, hdrs);
            if (early) s_text = 1;
            if ((threadIdx.x & 31) == 0) {
                if (kept) atomicAdd(&s_kept[0], kept);
                if (hdrs) atomicAdd(&s_hdr[0], hdrs);
                if (prefix) atomicAdd(&s_prefix, prefix);
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                ChunkSum o{};
                o.kept[0] = s_kept[0];
                o.hdr[0] = s_hdr[0];
                o.prefix = s_prefix;
                o.last = (uint8_t)(last & 3);
                o.text = (uint8_t)s_text;
                sums[c] = o;
            }
        }
        __syncthreads();
    }
}

// Pass 2 (one block): each chunk's incoming state (FASTA: 1 when its first
// bytes are a header's; FASTQ: its first line's role) and the kept bytes and
// headers before it; their totals and the flags to `out`.
struct FaTotals {
    unsigned long long kept, hdrs;
    uint32_t flags;
};
template <bool FQ>
__global__ void __launch_bounds__(1024) k_fa_carry(int64_t n_chunks, const ChunkSum* __restrict__ sums,
                                                   uint8_t* __restrict__ state, uint64_t* __restrict__ keep_off,
                                                   uint32_t* __restrict__ hdr_off, const uint32_t* __restrict__ flags,
                                                   FaTotals* __restrict__ out) {
    __shared__ int64_t sh[32];
    __shared__ int64_t tot;
    const int64_t per = (n_chunks + blockDim.x - 1) / blockDim.x;
    const int64_t a = min((int64_t)threadIdx.x * per, n_chunks), b = min(a + per, n_chunks);
    // the state coming into the thread's first chunk
    int64_t m = 0;
    int64_t any = 0;
    for (int64_t c = a; c < b; c++) {
        if (FQ) m += sums[c].lines;
        else if (sums[c].last) m = (c + 1) * 4 + sums[c].last;
        any |= sums[c].hdr[0] != 0;
    }
    int64_t in, open = 0;
    if (FQ) in = block_scan_excl_op<int64_t>(m, 0, SumOp(), sh, &tot);
    else in = block_scan_excl_op<int64_t>(m, 0, MaxOp(), sh, &tot) & 3;
    if (!FQ) open = block_scan_excl_op<int64_t>(any, 0, MaxOp(), sh, &tot);
    int64_t kept = 0, hdrs = 0;
    uint32_t bad = 0;
    const int64_t in0 = in;
    for (int64_t c = a; c < b; c++) {
        const ChunkSum& u = sums[c];
        if (FQ) {
            const int ro = (int)(in & 3);
            state[c] = (uint8_t)ro;
            kept += u.kept[ro];
            hdrs += u.hdr[ro];
            if (((u.not_at | u.not_plus) >> ro) & 1) bad |= FQ_BAD;
            in += u.lines;
        } else {
            state[c] = in == 2;
            kept += u.kept[0] - (in == 2 ? u.prefix : 0u);
            hdrs += u.hdr[0];
            if (!open && u.text) bad |= FA_TEXT_BEFORE_HEADER;
            open |= u.hdr[0] != 0;
            if (u.last) in = u.last;
        }
    }
    int64_t ko = block_scan_excl_op<int64_t>(kept, 0, SumOp(), sh, &tot);
    const int64_t ktot = tot;
    int64_t ho = block_scan_excl_op<int64_t>(hdrs, 0, SumOp(), sh, &tot);
    in = in0;
    for (int64_t c = a; c < b; c++) {
        const ChunkSum& u = sums[c];
        keep_off[c] = (uint64_t)ko;
        hdr_off[c] = (uint32_t)ho;
        const int st = state[c];
        ko += FQ ? (int64_t)u.kept[st] : (int64_t)u.kept[0] - (st ? (int64_t)u.prefix : 0);
        ho += FQ ? u.hdr[st] : u.hdr[0];
    }
    const int64_t htot = tot;
    if (bad) atomicOr(&out->flags, bad);
    if (threadIdx.x == 0) {
        out->kept = (unsigned long long)ktot;
        out->hdrs = (unsigned long long)htot;
        atomicOr(&out->flags, *flags);
        keep_off[n_chunks] = (uint64_t)ktot;
        hdr_off[n_chunks] = (uint32_t)htot;
    }
}

// Pass 3. The chunk's bytes are kept in shared memory with a pad word after
// every thread's 16 (threads' reads of their word i hit distinct banks), the
// output at its place modulo 16 in the file's sequence, so that whole 16-byte
// blocks are stored at once.
template <bool FQ>
__global__ void __launch_bounds__(FA_THREADS) k_fa_write(FaView v, const uint8_t* __restrict__ state,
                                                       const uint64_t* __restrict__ keep_off,
                                                       const uint32_t* __restrict__ hdr_off, uint8_t* __restrict__ out,
                                                       int64_t* __restrict__ hdr_pos, int64_t* __restrict__ hdr_seq) {
    __shared__ uint32_t s_in[FA_THREADS * 17 + 1];
    __shared__ __align__(16) uint8_t so[CHUNK + 32];
    __shared__ int32_t sh[32];
    __shared__ int32_t tot;
    for (int64_t c = blockIdx.x; c < v.n_chunks; c += gridDim.x) {
        const int64_t a = c * CHUNK + (int64_t)threadIdx.x * 64;
        uint32_t* const my = s_in + 17 * threadIdx.x;
        const Bytes64 r = load64(v, a, my);
        const uint64_t text = r.valid & ~r.nl & ~r.cr;
        uint64_t keep = 0, heads = 0;  // bytes kept, header lines' first bytes
        if (FQ) {
            int32_t line = (int32_t)state[c] + block_scan_excl_op<int32_t>(__popcll(r.nl), 0, SumOp(), sh, &tot);
            each_line(r, [&](uint64_t seg, int, bool starts, int at) {
                if ((line & 3) == 1) keep |= seg & text;
                if (starts && (line & 3) == 0 && v.d[a + at] == '@') heads |= 1ULL << at;
                line += (seg & r.nl) != 0;
            });
        } else {
            int32_t mine = 0;
            for (uint64_t st = r.start; st; st &= st - 1) {
                const int at = __ffsll((long long)st) - 1;
                const bool h = v.d[a + at] == '>';
                mine = ((int32_t)threadIdx.x + 1) * 4 + (h ? 2 : 1);
                if (h) heads |= 1ULL << at;
            }
            const int32_t in = block_scan_excl_op<int32_t>(mine, 0, MaxOp(), sh, &tot);
            bool hdr = in ? (in & 3) == 2 : state[c] != 0;
            each_line(r, [&](uint64_t seg, int, bool starts, int at) {
                if (starts) hdr = heads >> at & 1;
                if (!hdr) keep |= seg & text;
            });
        }
        const uint64_t ko = keep_off[c];
        const uint32_t shift = (uint32_t)(uintptr_t)(out + ko) & 15u;
        const int32_t kb = block_scan_excl_op<int32_t>(__popcll(keep), 0, SumOp(), sh, &tot);
        const int32_t ck = tot;
        const int32_t hb = block_scan_excl_op<int32_t>(__popcll(heads), 0, SumOp(), sh, &tot);
        int64_t hh = (int64_t)hdr_off[c] + hb;
        for (uint64_t h = heads; h; h &= h - 1) {
            const int at = __ffsll((long long)h) - 1;
            hdr_pos[hh] = a + at;
            hdr_seq[hh] = (int64_t)ko + kb + __popcll(keep & ((1ULL << at) - 1));
            hh++;
        }
        // the kept runs of the thread's bytes to their place
        uint32_t dst = shift + (uint32_t)kb;
        for (uint64_t k = keep; k;) {
            int at = __ffsll((long long)k) - 1;
            const uint64_t gap = ~(k >> at);
            int n = gap ? min(__ffsll((long long)gap) - 1, 64 - at) : 64 - at;
            k &= n + at >= 64 ? 0ULL : ~0ULL << (at + n);
            auto byte = [&](int i) { return (uint8_t)(my[i >> 2] >> (8 * (i & 3))); };
            for (; n && (dst & 3); n--) so[dst++] = byte(at++);
            for (; n >= 4; n -= 4, at += 4, dst += 4)
                *(uint32_t*)(so + dst) = __funnelshift_r(my[at >> 2], my[(at >> 2) + 1], 8 * (at & 3));
            for (; n; n--) so[dst++] = byte(at++);
        }
        __syncthreads();
        uint8_t* const base = out + ko - shift;  // 16-byte aligned
        const uint32_t end = shift + (uint32_t)ck;
        for (uint32_t x = 16 * threadIdx.x; x < end; x += 16 * FA_THREADS) {
            if (x >= shift && x + 16 <= end) {
                *(uint4*)(base + x) = *(const uint4*)(so + x);
            } else {
                for (uint32_t y = max(x, shift); y < min(x + 16, end); y++) base[y] = so[y];
            }
        }
        __syncthreads();
    }
}

// Pass 4: a header's name: after '>' up to the first space or tab, within
// the line without its dropped '\r'.
__device__ void name_span(const FaView& v, int64_t h, int64_t* s, int64_t* e) {
    int64_t i = h + 1;
    while (i < v.len && v.d[i] != '\n') i++;
    int64_t end = i;  // the line's end
    if (end > h + 1 && v.d[end - 1] == '\r') end--;
    int64_t j = h + 1;
    while (j < end && v.d[j] != ' ' && v.d[j] != '\t') j++;
    *s = h + 1;
    *e = j;
}

__global__ void k_fa_name_len(FaView v, const int64_t* __restrict__ hdr_pos, int64_t n, uint64_t* __restrict__ len) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
        int64_t s, e;
        name_span(v, hdr_pos[r], &s, &e);
        len[r] = (uint64_t)(e - s + 1);  // with its '\n' separator
    }
}

__global__ void k_fa_name_write(FaView v, const int64_t* __restrict__ hdr_pos, int64_t n,
                                const uint64_t* __restrict__ off, char* __restrict__ names) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
        int64_t s, e;
        name_span(v, hdr_pos[r], &s, &e);
        char* o = names + off[r];
        for (int64_t i = s; i < e; i++) *o++ = (char)v.d[i];
        *o = r + 1 < n ? '\n' : '\0';
    }
}

// FASTQ (needletail's, src/io/mod.rs:383-427): records of four lines, '@'
// header, sequence, '+' line, quality. A line's role is its index modulo 4. A
// line 4r must start with '@' and a line 4r + 2 with '+' (when not empty), else
// the file is refused and read on the host. Blank lines at the file's end are
// dropped first; a last record left without its quality (it was empty) or its
// '+' line reads as the host reader reads it: an empty or missing line.

}  // namespace

FastaDev* fasta_parse_device(int device, cudaStream_t s, UploadStage* up, const uint8_t* file, int64_t len,
                             std::string* why) {
    SHM_CUDA(cudaSetDevice(device));
    auto* F = new FastaDev();
    try {
        FaView v{};
        // FASTQ when the file starts with '@'; its blank lines at the end are
        // not part of any record
        const bool fastq = len > 0 && file[0] == '@';
        if (fastq)
            while (len > 0 && (file[len - 1] == '\n' || file[len - 1] == '\r')) len--;
        TmpBuf<uint8_t> raw;
        raw.reserve(((size_t)len + 64) / 64 * 64 + 64, s);
        upload(up, device, raw.p, file, (size_t)len, s);
        v.d = raw.p;
        v.len = len;
        v.n_chunks = (len + CHUNK - 1) / CHUNK;
        const int64_t nc = v.n_chunks;
        TmpBuf<ChunkSum> sums;
        TmpBuf<uint8_t> state;
        TmpBuf<uint64_t> keep_off;
        TmpBuf<uint32_t> hdr_off, flags;
        TmpBuf<FaTotals> totals;
        sums.reserve((size_t)nc + 1, s);
        state.reserve((size_t)nc + 1, s);
        keep_off.reserve((size_t)nc + 1, s);
        hdr_off.reserve((size_t)nc + 1, s);
        flags.reserve(1, s);
        totals.reserve(1, s);
        SHM_CUDA(cudaMemsetAsync(flags.p, 0, sizeof(uint32_t), s));
        SHM_CUDA(cudaMemsetAsync(totals.p, 0, sizeof(FaTotals), s));
        const int grid = grid_for((size_t)std::max<int64_t>(nc, 1), 1, 6);
        FaTotals T{};
        if (nc) {
            if (fastq) k_fa_count<true><<<grid, FA_THREADS, 0, s>>>(v, sums.p, flags.p);
            else k_fa_count<false><<<grid, FA_THREADS, 0, s>>>(v, sums.p, flags.p);
            SHM_CUDA(cudaGetLastError());
            if (fastq)
                k_fa_carry<true><<<1, 1024, 0, s>>>(nc, sums.p, state.p, keep_off.p, hdr_off.p, flags.p, totals.p);
            else
                k_fa_carry<false><<<1, 1024, 0, s>>>(nc, sums.p, state.p, keep_off.p, hdr_off.p, flags.p, totals.p);
            SHM_CUDA(cudaGetLastError());
            count_launch(2);
            SHM_CUDA(cudaMemcpyAsync(&T, totals.p, sizeof T, cudaMemcpyDeviceToHost, s));
            SHM_CUDA(cudaStreamSynchronize(s));
        }
        const uint64_t total = T.kept;
        const uint32_t n_rec = (uint32_t)T.hdrs, fl = T.flags;
        if (fl & FQ_BAD) {
            *why = "not FASTQ records of four lines";
            delete F;
            return nullptr;
        }
        if (fl & FA_FASTQ) {
            *why = "a line starts with '@' (FASTQ records are read on the host)";
            delete F;
            return nullptr;
        }
        if (fl & FA_TEXT_BEFORE_HEADER) {
            *why = "text before the first '>' header";
            delete F;
            return nullptr;
        }
        F->device = device;
        F->seq.reserve((size_t)total + 32, s);
        SHM_CUDA(cudaMemsetAsync(F->seq.p + total, 0, 32, s));
        F->offs.assign((size_t)n_rec + 1, (int64_t)total);
        if (n_rec) {
            TmpBuf<int64_t> hdr_pos, hdr_seq;
            hdr_pos.reserve(n_rec, s);
            hdr_seq.reserve(n_rec, s);
            if (fastq)
                k_fa_write<true><<<grid, FA_THREADS, 0, s>>>(v, state.p, keep_off.p, hdr_off.p, F->seq.p, hdr_pos.p,
                                                             hdr_seq.p);
            else
                k_fa_write<false><<<grid, FA_THREADS, 0, s>>>(v, state.p, keep_off.p, hdr_off.p, F->seq.p, hdr_pos.p,
                                                              hdr_seq.p);
            SHM_CUDA(cudaGetLastError());
            TmpBuf<uint64_t> nlen, noff;
            nlen.reserve(n_rec, s);
            noff.reserve((size_t)n_rec + 1, s);
            const int g2 = grid_for(n_rec, 128, 8);
            k_fa_name_len<<<g2, 128, 0, s>>>(v, hdr_pos.p, n_rec, nlen.p);
            SHM_CUDA(cudaGetLastError());
            exclusive_scan_u64(nlen.p, noff.p, n_rec, s);
            uint64_t nbytes = 0;
            SHM_CUDA(cudaMemcpyAsync(&nbytes, noff.p + n_rec, sizeof nbytes, cudaMemcpyDeviceToHost, s));
            SHM_CUDA(cudaStreamSynchronize(s));
            TmpBuf<char> names;
            names.reserve((size_t)nbytes + 1, s);
            k_fa_name_write<<<g2, 128, 0, s>>>(v, hdr_pos.p, n_rec, noff.p, names.p);
            SHM_CUDA(cudaGetLastError());
            count_launch(3);
            F->names.resize((size_t)nbytes);
            SHM_CUDA(cudaMemcpyAsync(&F->names[0], names.p, (size_t)nbytes, cudaMemcpyDeviceToHost, s));
            SHM_CUDA(cudaMemcpyAsync(F->offs.data(), hdr_seq.p, sizeof(int64_t) * n_rec, cudaMemcpyDeviceToHost, s));
            SHM_CUDA(cudaStreamSynchronize(s));
            if (!F->names.empty()) F->names.pop_back();  // the last name's terminator
            // names as String::from_utf8_lossy gives them (src/io/mod.rs:408-410)
            bool ascii = true;
            for (char ch : F->names) ascii = ascii && (unsigned char)ch < 0x80;
            if (!ascii) F->names = utf8_lossy(F->names);
        }
        F->n = (int32_t)n_rec;
        return F;
    } catch (...) {
        delete F;
        throw;
    }
}

}  // namespace shm
