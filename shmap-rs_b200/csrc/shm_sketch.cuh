// Device FracMinHash sketching (see shm_sketch.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace shm {

enum SketchMode { SK_APPEND = 0, SK_COUNT = 1, SK_WRITE = 2 };

// Sequences are concatenated in `seq` (device, padded by 16 bytes, 16-byte
// aligned base) with seq_off[n_seq+1]. chunk_off[n_seq+1] is the prefix of
// ceil(windows / SKETCH_WIN) per sequence.
//  - SK_APPEND: unordered output per sequence into [kmer_off[q], kmer_off[q+1]),
//    counted in kmer_cnt[q] (which may exceed the capacity: caller checks).
//  - SK_COUNT: chunk_cnt[c] = selected windows of chunk c.
//  - SK_WRITE: writes chunk c's selections in order from chunk_out[c].
struct SketchArgs {
    const uint8_t* seq;
    const int64_t* seq_off;
    const uint64_t* chunk_off;
    int32_t n_seq;
    uint64_t n_chunks;
    int32_t k;
    uint64_t thr;
    int32_t r_offset;  // added to every r (sketch_slice_into's `offset`)
    // SK_APPEND
    const uint64_t* kmer_off;
    uint32_t* kmer_cnt;
    // SK_COUNT / SK_WRITE
    uint32_t* chunk_cnt;
    const uint32_t* chunk_out;  // n_chunks+1 exclusive offsets (total < 2^32)
    // outputs
    uint64_t* out_h;
    uint32_t* out_rs;  // r << 1 | strand
    // SK_APPEND only: when set, the reads come as 2-bit codes and a non-ACGT
    // mask instead of `seq` (the layout of host/pack.hpp: base p, relative to
    // the batch, is bits 2(p & 15) of pk_codes[p >> 4], masked when bit p & 31
    // of pk_mask[p >> 5] is set; two spare groups of 32 past the end)
    const uint32_t* pk_codes;
    const uint32_t* pk_mask;
    uint64_t pk_words;  // code words readable at pk_codes (those past it read as 0)
    // SK_APPEND only: seq_off[0] and seq_off[n_seq] on the host, when the caller has
    // them and `luts` is of create_device_luts (the bit-plane kernels take the call then)
    int64_t base0, base1;
    // launch_sketch_ordered only (set by it)
    uint32_t *ord_cnt, *ord_seq_cnt;
    const uint32_t* ord_off;
    uint32_t ord_stride;
};

// The five lookup tables of src/sketch.rs:50-97 for one k, in device memory
// (owned by the caller, released with cudaFree).
struct SketchLuts;
SketchLuts* create_device_luts(int32_t k, cudaStream_t s);
// The bit-plane kernels (shm_sketch_bits.cuh) take sequences in order
// (launch_sketch_ordered) at this k and threshold, and n reads of `bases` bases
// in all (SK_APPEND).
bool sketch_bits_takes(int32_t k, uint64_t thr);
bool sketch_bits_reads(int32_t k, uint64_t thr, int64_t bases, int32_t n);
struct SketchTabs;
void launch_sketch_bits(const SketchArgs& a, const SketchTabs* tabs, cudaStream_t s);
// The selected windows of all sequences of a (seq, seq_off, n_seq, k, thr,
// r_offset, base0, base1; where sketch_bits_takes) in sequence order, by
// warps that each take a contiguous part: warp w's number goes to cnt[w], and
// from off[w] to off[w + 1] of a.out_h and a.out_rs (off null: from w * stride,
// at most stride) as many of them as there is room for; seq_cnt (may be null,
// n_seq zeroed words) counts each sequence's. ordered_warps: the number of
// warps, cnt's length (the same for the same a).
uint32_t ordered_warps(const SketchArgs& a);
void launch_sketch_ordered(SketchArgs a, const SketchLuts* luts, uint32_t* cnt, uint32_t* seq_cnt, const uint32_t* off,
                           uint32_t stride, cudaStream_t s);
void launch_sketch(int mode, const SketchArgs& a, const SketchLuts* luts, cudaStream_t s);

// Builds the tables on the device into caller-provided device memory of
// sketch_luts_bytes() bytes (8-byte aligned); no host copy, no allocation.
size_t sketch_luts_bytes();
void launch_fill_luts(SketchLuts* d, int32_t k, cudaStream_t s);

}  // namespace shm
