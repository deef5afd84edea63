// Lane side of the encoder, shared by the encode kernels and the fused update: the bit stream
// under construction of one lane, and the epilogue that brings a block's payload to memory.
//
// Encode table (shared memory, one 32-bit entry per exponent byte): the code with its first bit
// in bit 31, the code length in bits 0..4, nothing in between.  One left funnel shift whose
// operand AND amount are the entry appends a code; adding the entry to the position counter adds
// its length (the counter's low 16 bits; the codes' bits only reach the upper half).  A lane's
// last 64 bits are kept, first bit highest.  A pair of symbols adds at most 32 bits, so at most
// one word is finished per pair, which shows as a flip of bit 5 of the position; it is stored to
// a shared image of the block's payload by predicated instructions, and bit-reversed into the
// format's first-bit-lowest order when the image is copied out (one reversal per word instead of
// one extra instruction per pair).
#pragma once

#include "lanes.cuh"

namespace lct {



// A code has at most 16 bits (a prefix of 8 and an 8-bit literal); the bounds that keep the word
// stores inside the image rest on this, so it is enforced here whatever the table holds.
__device__ __forceinline__ uint32_t encode_entry(uint32_t packed) {  // code | length << 20
  return (__brev(packed) & 0xFFFF0000u) | min(packed >> 20, 16u);
}
// Table entry of exponent byte k of `exponents`: one byte dot product with 4 in byte k gives the
// entry's address (multiplier pipe; the kernels are bound by the other integer pipe).  The load is
// not volatile: nothing writes the table between its barrier and the end of the kernel, and
// `table` (a shared address) comes out of after_barrier(), behind which it stays.
__device__ __forceinline__ uint32_t after_barrier(uint32_t address) {
  asm volatile("mov.u32 %0, %0;" : "+r"(address));
  return address;
}
template <int k>
__device__ __forceinline__ uint32_t encode_entry_of(uint32_t table, uint32_t exponents) {
  uint32_t entry;
  asm("{\n\t.reg .b32 a;\n\t"
      "dp4a.u32.u32 a, %1, %3, %2;\n\t"
      "ld.shared.u32 %0, [a];\n\t}"
      : "=r"(entry)
      : "r"(exponents), "r"(table), "r"(4u << (8 * k)));
  return entry;
}

struct LaneWriter {
  uint32_t low, high;  // the last 64 bits of the stream
  uint32_t pos;        // bits so far in the low 16 bits
  uint32_t at;         // shared address of the next image word of this lane
  int extra_start;     // first overflowing step, -1 = none

  __device__ __forceinline__ void open(uint32_t column) {
    low = high = pos = 0u;
    at = column;
    extra_start = -1;
  }
  __device__ __forceinline__ uint32_t bits() const { return pos & 0xFFFFu; }
  __device__ __forceinline__ void append(uint32_t first, uint32_t second) {
    high = __funnelshift_l(low, high, first);
    low = __funnelshift_l(first, low, first);
    high = __funnelshift_l(low, high, second);
    low = __funnelshift_l(second, low, second);
    const uint32_t next = pos + first + second;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b32 d, w;\n\t"
        "lop3.b32 d, %1, %2, 32, 0x28;\n\t"  // (pos ^ next) & 32
        "setp.ne.u32 p, d, 0;\n\t"
        "@p shf.r.wrap.b32 w, %3, %4, %2;\n\t"
        "@p st.shared.u32 [%0], w;\n\t"
        "@p add.u32 %0, %0, 1024;\n\t"
        "}"
        : "+r"(at)
        : "r"(pos), "r"(next), "r"(low), "r"(high));
    pos = next;
  }
  // The pair of rows at `step`, checked against the lane's budget: the first pair that does not
  // fit closes the lane.  No branches: a pair that is not taken is appended as two empty codes.
  __device__ __forceinline__ void append_checked(uint32_t first, uint32_t second, int step,
                                                 uint32_t budget_bits) {
    const bool fits = ((pos + first + second) & 0xFFFFu) <= budget_bits;
    const bool open = extra_start < 0;
    append(open && fits ? first : 0u, open && fits ? second : 0u);
    if (open && !fits) extra_start = step;
  }
  // The word under construction, after the last pair.
  __device__ __forceinline__ void close() {
    if (pos & 31u)
      asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(low << (32u - (pos & 31u))) : "memory");
  }
};
static_assert(kLanes * 4 == 1024, "LaneWriter steps from image row to image row");

// The same with finished words going straight to the payload in global memory, for kernels whose
// shared memory an image would cost resident CTAs (a warp's lanes write neighbouring words of the
// same payload rows; L2 merges them).
struct GlobalLaneWriter {
  uint32_t low, high;  // the last 64 bits of the stream
  uint32_t pos;        // bits so far in the low 16 bits
  uint32_t* at;        // next payload word of this lane
  int64_t row_bytes;   // from one payload word of a lane to the next
  int extra_start;     // first overflowing step, -1 = none

  __device__ __forceinline__ void open(uint32_t* column, int64_t streams) {
    low = high = pos = 0u;
    at = column;
    row_bytes = streams * 4;
    extra_start = -1;
  }
  __device__ __forceinline__ uint32_t bits() const { return pos & 0xFFFFu; }
  __device__ __forceinline__ void append(uint32_t first, uint32_t second) {
    high = __funnelshift_l(low, high, first);
    low = __funnelshift_l(first, low, first);
    high = __funnelshift_l(low, high, second);
    low = __funnelshift_l(second, low, second);
    const uint32_t next = pos + first + second;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b32 d, w;\n\t"
        "lop3.b32 d, %1, %2, 32, 0x28;\n\t"  // (pos ^ next) & 32
        "setp.ne.u32 p, d, 0;\n\t"
        "@p shf.r.wrap.b32 w, %3, %4, %2;\n\t"
        "@p brev.b32 w, w;\n\t"
        "@p st.global.u32 [%0], w;\n\t"
        "@p add.s64 %0, %0, %5;\n\t"
        "}"
        : "+l"(at)
        : "r"(pos), "r"(next), "r"(low), "r"(high), "l"(row_bytes)
        : "memory");
    pos = next;
  }
  __device__ __forceinline__ void append_checked(uint32_t first, uint32_t second, int step,
                                                 uint32_t budget_bits) {
    const bool fits = ((pos + first + second) & 0xFFFFu) <= budget_bits;
    const bool open = extra_start < 0;
    append(open && fits ? first : 0u, open && fits ? second : 0u);
    if (open && !fits) extra_start = step;
  }
  // The word under construction after the last pair, and zeros up to the budget.
  __device__ __forceinline__ void close(int fixed_words) {
    int word = bits() >> 5;
    char* to = reinterpret_cast<char*>(at);
    if (pos & 31u) {
      *reinterpret_cast<uint32_t*>(to) = __brev(low << (32u - (pos & 31u)));
      to += row_bytes;
      ++word;
    }
    for (; word < fixed_words; ++word, to += row_bytes) *reinterpret_cast<uint32_t*>(to) = 0u;
  }
};

// More bits than a chunk can add: lanes further than this from their budget need no check.
constexpr uint32_t kChunkBits = kChunkRows * 16;

// Fill the encode table from the tensor's shifted table (no barrier).
template <int kCtaThreads>
__device__ __forceinline__ void load_encode_table(uint32_t* table, const int32_t* shifted) {
#pragma unroll
  for (int i = threadIdx.x; i < 256; i += kCtaThreads)
    table[i] = encode_entry(load_dependent_u32(shifted + i));
}

// Clear the payload image of a block.
template <int kCtaThreads>
__device__ __forceinline__ void clear_image(uint32_t* image, int fixed_words) {
  uint4* rows = reinterpret_cast<uint4*>(image);
  for (int i = threadIdx.x; i < fixed_words * (kLanes / 4); i += kCtaThreads)
    rows[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Overflow starts of this thread's neighbouring lanes and the block's summary, with a block barrier
// between.  `writers`: kLanes / kCtaThreads of them.  `scan`: two shared ints per warp.
template <int kCtaThreads, typename Writer>
__device__ __forceinline__ void summarise_block(const Writer* writers, int* scan,
                                                uint8_t* __restrict__ extra_starts,
                                                int32_t* __restrict__ summaries, int64_t block,
                                                int64_t n_blocks, int steps) {
  constexpr int kOwn = kLanes / kCtaThreads, kCtaWarps = kCtaThreads / 32;
  const int tid = threadIdx.x;
  int bad = 0, bytes = 0;
#pragma unroll
  for (int i = 0; i < kOwn; ++i) {
    const int start = writers[i].extra_start;
    extra_starts[block * kLanes + kOwn * tid + i] = (uint8_t)start;  // none: 255
    bad += start >= 0 ? 1 : 0;
    bytes += start >= 0 ? steps - start : 0;
  }
  bad = __reduce_add_sync(0xFFFFFFFFu, bad);
  bytes = __reduce_add_sync(0xFFFFFFFFu, bytes);
  if ((tid & 31) == 0) { scan[tid >> 5] = bad; scan[kCtaWarps + (tid >> 5)] = bytes; }
  __syncthreads();
  if (tid == 0) {
    int total_bad = 0, total_bytes = 0;
#pragma unroll
    for (int w = 0; w < kCtaWarps; ++w) { total_bad += scan[w]; total_bytes += scan[kCtaWarps + w]; }
    summaries[block] = total_bad;
    summaries[n_blocks + block] = total_bytes;
  }
}

// Everything after the last pair of a block: last words, overflow starts, the block's summary,
// the payload image to global memory (word w of the block's 256 streams is one 1 KB row).
template <int kCtaThreads>
__device__ __forceinline__ void finish_block(LaneWriter* writers, const uint32_t* image, int* scan,
                                             uint32_t* __restrict__ encoded,
                                             uint8_t* __restrict__ extra_starts,
                                             int32_t* __restrict__ summaries, int64_t block,
                                             int64_t n_blocks, int64_t streams, int steps,
                                             int fixed_words) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int i = 0; i < kLanes / kCtaThreads; ++i) writers[i].close();
  // (Its barrier also publishes every lane's payload words.)
  summarise_block<kCtaThreads>(writers, scan, extra_starts, summaries, block, n_blocks, steps);
  uint32_t* out = encoded + block * kLanes + (tid & 63) * 4;
  for (int w = tid >> 6; w < fixed_words; w += kCtaThreads / 64) {
    const uint4 v = *reinterpret_cast<const uint4*>(&image[w * kLanes + (tid & 63) * 4]);
    __stcs(reinterpret_cast<uint4*>(out + (int64_t)w * streams),
           make_uint4(__brev(v.x), __brev(v.y), __brev(v.z), __brev(v.w)));
  }
}

}  // namespace lct
