// Division of a codec block among threads.
//
// The encoder: one CTA of 128 threads per block; thread t owns the two neighbouring lanes 2t and 2t + 1.
// The lane mapping XORs a lane with an even mask, and rows 2k and 2k + 1 share their mask, so in
// every row a thread's two lanes are two neighbouring columns (in order), and a warp's 64 lanes
// are one aligned group of 64 columns.  A thread therefore handles whole 32-bit words of the
// dense tensor - two BF16 values - without exchanging anything with another thread: a warp reads
// or writes one full 128-byte line of the dense tensor and 64 bytes of the side bytes per row,
// and nothing but the codebook (and the encoder's payload image) goes through shared memory.
//
// Against the former split (one lane per thread for the streams, tiles of 32 rows transposed
// through shared memory to eight columns per thread for the dense side) this drops the tile's
// stores, loads, address arithmetic and barriers, gives every thread two independent stream
// chains, and halves the threads a block needs, so that more blocks are resident at once.
#pragma once

#include "common.cuh"

namespace lct {

constexpr int kPairThreads = kLanes / 2;
constexpr int kPairWarps = kPairThreads / 32;
// Rows per unrolled chunk: the mask's bits 1..2 are compile-time constants inside a chunk.
constexpr int kChunkPairs = 4;
constexpr int kChunkRows = 2 * kChunkPairs;

constexpr int kRowBytes = kLanes * 2;
// Byte offset inside the block's dense rows (512 bytes each) of this thread's word in the first
// row of the chunk that starts at `step0` (a multiple of kChunkRows); row pair k of the chunk is
// at chunk_word(offset, k), its second row 512 bytes further on.
template <int kLaneMask>
__device__ __forceinline__ uint32_t chunk_offset(int64_t row0, int step0, int lane_mask) {
  const int mask = kLaneMask >= 0 ? kLaneMask : lane_mask;
  const uint32_t moved = (2u * threadIdx.x) ^ (uint32_t)((row0 + step0) & mask);
  return (uint32_t)step0 * kRowBytes + moved * 2u;
}
// ... and of its word in row pair k of that chunk, less k * 1024 bytes (which callers add to the
// pointer, where it becomes part of the instruction).
template <int kLaneMask>
__device__ __forceinline__ uint32_t chunk_word(uint32_t offset, int k, int lane_mask) {
  const int mask = kLaneMask >= 0 ? kLaneMask : lane_mask;
  return offset ^ (uint32_t)(((2 * k) & mask) * 2);
}

// The other split, of the kernels that read bit streams: one CTA of 256 threads per block, one
// lane per thread (twice the warps to hide the walk's latency).  Two neighbouring threads' lanes
// are two neighbouring columns in every row, so the two exchange exponents with one shuffle per
// row pair, after which the even thread has both columns of the pair's first row and the odd one
// those of its second: whole 32-bit words of the dense tensor again, 64-byte segments per warp.

// Element offset inside the block of this thread's word in the chunk that starts at `step0`: the
// columns of its lane and its neighbour's, in the even or odd rows; see word_at.
__device__ __forceinline__ uint32_t word_offset(int64_t row0, int step0, int lane_mask) {
  const uint32_t moved = (threadIdx.x & 254u) ^ (uint32_t)((row0 + step0) & lane_mask);
  return (step0 + (threadIdx.x & 1u)) * kLanes + moved;
}
// ... in row pair k of that chunk.
template <int kLaneMask>
__device__ __forceinline__ uint32_t word_at(uint32_t offset, int k, int lane_mask) {
  const int mask = kLaneMask >= 0 ? kLaneMask : lane_mask;
  return (offset ^ (uint32_t)((2 * k) & mask)) + (uint32_t)(2 * k * kLanes);
}

// ---- shared memory by 32-bit address --------------------------------------
__device__ __forceinline__ uint32_t shared_address(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint32_t load_shared_u32(uint32_t address) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(address));
  return v;
}
__device__ __forceinline__ uint32_t load_shared_u16(uint32_t address) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(address));
  return v;
}
__device__ __forceinline__ uint32_t load_shared_u8(uint32_t address) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(address));
  return v;
}

// Streaming load that stays where it is written relative to other volatile assembly (the word
// stores of the encoder): requests are placed ahead of the work that hides their latency, and the
// compiler would otherwise move them behind it to save registers.
__device__ __forceinline__ uint32_t load_ahead_u32(const void* p) {
  uint32_t v;
  asm volatile("ld.global.cs.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t load_ahead_u16(const void* p) {
  uint16_t v;
  asm volatile("ld.global.cs.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}

// Bring `bytes` (a multiple of 16, at a 16-byte aligned address) from DRAM to L2: one instruction
// of one thread keeps several KB per CTA under way, far ahead of the loads that use them.
__device__ __forceinline__ void prefetch_l2(const void* address, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(address), "r"(bytes));
}

// a + sum over the four bytes of e (unsigned) * w (signed): with w = -1 in one byte this
// subtracts that byte of e from a.
__device__ __forceinline__ int dot_bytes(uint32_t e, int w, int a) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(e), "r"(w), "r"(a));
  return d;
}

// a where the mask is set, else b: one three-input logic operation.
__device__ __forceinline__ uint32_t select_bits(uint32_t a, uint32_t b, uint32_t mask) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xE4;" : "=r"(d) : "r"(a), "r"(b), "r"(mask));
  return d;
}

// ---- side bytes ------------------------------------------------------------
// Two BF16 words (rows 2k and 2k + 1, two columns each) -> side bytes and exponent bytes, in byte
// order [row 2k: column 0, 1 | row 2k + 1: column 0, 1].
__device__ __forceinline__ void split_words(uint32_t top, uint32_t bottom, uint32_t* sides,
                                            uint32_t* exponents) {
  const uint32_t low = prmt(top, bottom, 0x6420), high = prmt(top, bottom, 0x7531);
  *sides = select_bits(low, high, 0x7F7F7F7Fu);
  *exponents = select_bits(low >> 7, high << 1, 0x01010101u);
}
// Two side bytes (column 0 in byte 0) and two exponents in bits 7..14 / 23..30 -> two BF16 values.
__device__ __forceinline__ uint32_t join_word(uint32_t exponents, uint32_t sides) {
  return select_bits(exponents, prmt(sides, 0u, 0x1100), 0x7F807F80u);
}

}  // namespace lct
