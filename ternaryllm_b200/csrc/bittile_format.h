// bittile_format.h -- the dense two-bit copy of W ("bit tiles") that the register-decode kernel (bits_kernel.cuh) and the
// batched tensor-core kernel (mma_kernel.cuh) read, shared by the host packer and the device code.
//
// A code is two bits, nz | neg << 1: 0 = zero, 1 = +1, 3 = -1.  Put into the top two bits of a 16-bit float -- sign and
// highest exponent bit -- it IS the number: 0, +2.0 or -2.0 in fp16 and in bf16 alike.  One word holds sixteen
// consecutive rows of one column; the pair of rows (2p, 2p+1) sits so that a left shift by 2p brings its two codes to the
// top of the word's two halves: one shift and one AND decode two entries (mm_code_bit below).
//
// Order: columns in groups of sixteen (N padded to 128), a group's slices of 64 rows one after the other along K, so a
// group is one contiguous stream of KB * 256 bytes (KB = ceil(K / 64)).  Slices come in pairs of 512 bytes = 32 chunks of 16
// bytes; chunk mm_chunk(g, t) holds { slice 0: column g, column g + 8; slice 1: column g, column g + 8 }, rows 16t .. 16t + 15
// of the slice.  A lane 4g + t of the register-decode kernel takes one chunk: the places that mma.sync.m16n8k16 wants it to
// fill.  A lane of the batched kernel takes the four chunks of one g, one t after the other: the exclusive or in mm_chunk
// spreads the eight values of g over all banks of shared memory.  An odd last slice is 256 bytes, 8 for each (g, t) in order.
#pragma once
#include <cstddef>
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define MM_FMT_HD __host__ __device__
#else
#define MM_FMT_HD
#endif
MM_FMT_HD inline int mm_code_bit(int kk) {            // kk = 0..15, row within the word
    return 14 - 2 * (kk >> 1) + 16 * (kk & 1);
}
MM_FMT_HD inline int mm_chunk(int g, int t) { return 4 * g + (t ^ ((g >> 1) & 3)); }
// index of the word that holds rows 16t .. 16t+15 of slice kb, column n
MM_FMT_HD inline size_t mm_word_index(int n, int kb, int t, int KB) {
    const size_t base = (size_t)(n >> 4) * KB * 64;
    const int g = n & 7, hi = (n >> 3) & 1;
    if ((kb | 1) < KB) return base + (size_t)(kb >> 1) * 128 + mm_chunk(g, t) * 4 + (kb & 1) * 2 + hi;
    return base + (size_t)kb * 64 + (4 * g + t) * 2 + hi;
}
void mm_pack_bits(const int8_t* w, int inners, int columns, std::vector<uint32_t>* bits, int* n_tiles, int* kb);
void mm_unpack_bits(const std::vector<uint32_t>& bits, int inners, int columns, int8_t* w);
