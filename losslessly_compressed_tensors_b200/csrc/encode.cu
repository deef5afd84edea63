// Field split + fixed-budget Huffman encoder, and the overflow tail compaction.
//
// One CTA of 128 threads per codec block, thread = two neighbouring lanes (lanes.cuh).  Per row
// pair a thread has two 32-bit source words (requested a chunk of 8 rows ahead; a warp reads a
// full 128-byte line per row), splits off the side bytes and stores them (64 bytes per warp and
// row), looks the four exponents up in the shared encode table and appends two codes to each of
// its two bit streams (lane_writer.cuh).  Finished words are collected in a shared image of the
// block's payload (zero where nothing was written, so the output is deterministic), which is
// copied out at the end with 128-bit stores.
//
// A chunk in which some lane of the warp could run out of its bit budget (or already has) takes
// the checked form of the append; all others carry no per-pair conditions.  Once every lane of a
// warp has run out, only its side bytes are left to write, in a loop of their own (1 Mi elements
// that overflow everywhere, half-zero codebook: kernel 13.1 -> 10.4 us; as a third form inside the
// unrolled loop it costs all other tensors 2 %).
#include <type_traits>

#include "batch.cuh"
#include "common.cuh"
#include "lane_writer.cuh"
#include "lct_b200.h"

namespace lct {

// Resident CTAs per SM the encoder is compiled for, as many as its registers allow (96 x 128 threads).
constexpr int kEncodeMinCtas = 5;

struct EncodeShape {
  int64_t size;
  int64_t logical_numel;
  int64_t streams;
  int64_t n_blocks;
  int block_symbols;
  int steps;
  int fixed_words;
  int lane_mask;  // 254: lane ^ (row & 254) ("swizzle"); 0: "linear"
};

// How far ahead of the rows in work the source is brought to L2, and in what portions.
constexpr int kPrefetchRows = 32, kPrefetchPortion = 2 * kChunkRows;

// Shared memory: encode table | scratch | payload image.
struct __align__(16) EncodeSharedHead {
  uint32_t table[256];
  int scan[16];
};

// Exponent bytes of two columns, spread to where BF16 values hold them.
__device__ __forceinline__ uint32_t spread_exponents(uint32_t low, uint32_t high) {
  return (low << 7) | (high << 23);
}

// One codec block.  extra_starts and summaries are the tensor's own arrays
// (summaries holds g.n_blocks entries per row).
// kLaneMask: the lane mapping as a compile-time constant (254, the default mapping), or -1 to
// take it from the shape at run time.  kAligned: the source's words of two values are aligned.
template <bool kPrecomputed, int kLaneMask, bool kAligned>
struct BlockEncoder {
  const char* rows;  // the block's first source row
  uint8_t* side_rows;
  const EncodeShape& g;
  int64_t block;
  uint32_t table;
  int wide_rows;  // rows, in whole chunks, that may be read as two-value words
  LaneWriter lanes[2];

  // What the two lanes append for one row pair, and its side bytes.
  struct Pair {
    uint32_t sides, a0, a1, b0, b1;
  };

  __device__ __forceinline__ Pair look_up(uint32_t top, uint32_t bottom) const {
    Pair p;
    uint32_t exponents;
    split_words(top, bottom, &p.sides, &exponents);
    p.a0 = encode_entry_of<0>(table, exponents);
    p.b0 = encode_entry_of<1>(table, exponents);
    p.a1 = encode_entry_of<2>(table, exponents);
    p.b1 = encode_entry_of<3>(table, exponents);
    return p;
  }
  __device__ __forceinline__ void store_sides(const Pair& p, int k) const {
    if (kPrecomputed) return;
    uint8_t* s = side_rows + (2 * k) * kLanes;
    __stcs(reinterpret_cast<uint16_t*>(s), (uint16_t)p.sides);
    __stcs(reinterpret_cast<uint16_t*>(s + kLanes), (uint16_t)(p.sides >> 16));
  }
  template <bool kChecked>
  __device__ __forceinline__ void append(const Pair& p, int step, uint32_t budget_bits) {
    if (kChecked) {
      lanes[0].append_checked(p.a0, p.a1, step, budget_bits);
      lanes[1].append_checked(p.b0, p.b1, step, budget_bits);
    } else {
      lanes[0].append(p.a0, p.a1);
      lanes[1].append(p.b0, p.b1);
    }
  }
  // Bring rows of the source to L2, from the 16-byte granule on that holds the first one's start.
  __device__ __forceinline__ void prefetch(int first_row, int count) const {
    const uintptr_t at = reinterpret_cast<uintptr_t>(rows) + (uint32_t)(first_row * kRowBytes);
    prefetch_l2(reinterpret_cast<const void*>(at & ~(uintptr_t)15), count * kRowBytes);
  }
  // The words of the chunk at step0, all requested together: loads requested one by one between
  // other work would make every use wait for the latest of them.
  __device__ __forceinline__ void request(uint32_t (&words)[kChunkRows], int step0) const {
    if (step0 >= wide_rows) return;
    const uint32_t offset = chunk_offset<kLaneMask>(block * g.steps, step0, g.lane_mask);
#pragma unroll
    for (int row = 0; row < kChunkRows; ++row) {
      const uint32_t at = chunk_word<kLaneMask>(offset, row >> 1, g.lane_mask);
      if (kPrecomputed) {
        const uint32_t bytes = load_ahead_u16(rows + (at >> 1) + row * kLanes);
        words[row] = spread_exponents(bytes & 255u, bytes >> 8);
      } else {
        words[row] = load_ahead_u32(rows + at + row * kRowBytes);
      }
    }
  }
  // Rows of a source at an odd multiple of two bytes, up to `full_rows`: a word is two loads of two
  // bytes, requested a chunk ahead and joined when the chunk's turn comes.
  __device__ __forceinline__ void run_unaligned(int full_rows, uint32_t budget_bits) {
    uint32_t first[kChunkRows], second[kChunkRows];
    auto request_values = [&](int step0) {
      if (step0 >= full_rows) return;
      const uint32_t offset = chunk_offset<kLaneMask>(block * g.steps, step0, g.lane_mask);
#pragma unroll
      for (int row = 0; row < kChunkRows; ++row) {
        const char* p = rows + chunk_word<kLaneMask>(offset, row >> 1, g.lane_mask) + row * kRowBytes;
        first[row] = load_ahead_u16(p);
        second[row] = load_ahead_u16(p + 2);
      }
    };
    request_values(0);
#pragma unroll 1
    for (int step0 = 0; step0 < full_rows; step0 += kChunkRows) {
      Pair pairs[kChunkPairs];
#pragma unroll
      for (int k = 0; k < kChunkPairs; ++k)
        pairs[k] = look_up(first[2 * k] | (second[2 * k] << 16), first[2 * k + 1] | (second[2 * k + 1] << 16));
      request_values(step0 + kChunkRows);
#pragma unroll
      for (int k = 0; k < kChunkPairs; ++k) {
        store_sides(pairs[k], k);
        append<true>(pairs[k], step0 + 2 * k, budget_bits);
      }
      side_rows += kChunkRows * kLanes;
    }
  }

  // A word by guarded loads: a chunk that reaches past the end, exponent bytes of any alignment.
  __device__ __forceinline__ uint32_t guarded_word(int step0, int k, bool second) const {
    const int64_t left = g.logical_numel - block * (int64_t)g.block_symbols;
    const uint32_t offset = chunk_offset<kLaneMask>(block * g.steps, step0, g.lane_mask);
    const int64_t at = (chunk_word<kLaneMask>(offset, k, g.lane_mask) >> 1) + (2 * k + second) * kLanes;
    uint32_t low = 0u, high = 0u;
    if (kPrecomputed) {
      const uint8_t* p = reinterpret_cast<const uint8_t*>(rows) + at;
      if (at < left) low = p[0];
      if (at + 1 < left) high = p[1];
      return spread_exponents(low, high);
    }
    const uint16_t* p = reinterpret_cast<const uint16_t*>(rows) + at;
    if (at < left) low = p[0];
    if (at + 1 < left) high = p[1];
    return low | (high << 16);
  }

  // The software pipeline: `now` is the row pair to append; while it is appended, the next one's
  // entries are looked up.  Once a chunk's words (`words`) are looked up, their registers take the
  // words of the chunk after the next one (`ahead` holds the next one's).
  template <bool kChecked>
  __device__ __forceinline__ void step_chunk(int step0, Pair& now, uint32_t (&words)[kChunkRows],
                                             const uint32_t (&ahead)[kChunkRows], uint32_t budget_bits) {
#pragma unroll
    for (int k = 0; k < kChunkPairs; ++k) {
      const Pair next = k + 1 < kChunkPairs ? look_up(words[2 * k + 2], words[2 * k + 3])
                                            : look_up(ahead[0], ahead[1]);
      if (k + 2 == kChunkPairs) request(words, step0 + 2 * kChunkRows);
      store_sides(now, k);
      append<kChecked>(now, step0 + 2 * k, budget_bits);
      now = next;
    }
    side_rows += kChunkRows * kLanes;
  }

  // The rows that are read as words, up to the end or to where every lane of the warp has run out
  // of its budget; returns the row behind the last.
  __device__ __forceinline__ int run_open(bool prefetches, uint32_t budget_bits) {
    uint32_t even[kChunkRows], odd[kChunkRows];
    request(even, 0);
    request(odd, kChunkRows);
    Pair now = look_up(even[0], even[1]);
    auto near = [&] { return __any_sync(0xFFFFFFFFu, max(lanes[0].bits(), lanes[1].bits()) + kChunkBits > budget_bits); };
    int step0 = 0;
#pragma unroll 1
    do {
      if (prefetches && step0 + kPrefetchRows + kPrefetchPortion <= wide_rows)
        prefetch(step0 + kPrefetchRows, kPrefetchPortion);
      if (near())
        step_chunk<true>(step0, now, even, odd, budget_bits);
      else
        step_chunk<false>(step0, now, even, odd, budget_bits);
      step0 += kChunkRows;
      if (step0 >= wide_rows) break;
      bool closed = false;
      if (near()) {
        step_chunk<true>(step0, now, odd, even, budget_bits);
        closed = (lanes[0].extra_start | lanes[1].extra_start) >= 0;
      } else {
        step_chunk<false>(step0, now, odd, even, budget_bits);
      }
      step0 += kChunkRows;
      if (__all_sync(0xFFFFFFFFu, closed)) break;
    } while (step0 < wide_rows);
    return step0;
  }
  // ... and those behind, of which only the side bytes are left to write.
  __device__ __forceinline__ void run_closed(int step0) {
    uint32_t words[kChunkRows], ahead[kChunkRows];
    request(words, step0);
#pragma unroll 1
    for (; step0 < wide_rows; step0 += kChunkRows) {
      request(ahead, step0 + kChunkRows);
#pragma unroll
      for (int k = 0; k < kChunkPairs; ++k) {
        Pair p;
        uint32_t exponents;
        split_words(words[2 * k], words[2 * k + 1], &p.sides, &exponents);
        store_sides(p, k);
      }
#pragma unroll
      for (int row = 0; row < kChunkRows; ++row) words[row] = ahead[row];
      side_rows += kChunkRows * kLanes;
    }
  }

  // All rows up to `rows_used`: whole chunks as above, the rest by guarded loads.
  __device__ __forceinline__ void run(int rows_used, int full_rows, bool prefetches) {
    const uint32_t budget_bits = (uint32_t)g.fixed_words * 32u;
    if (kAligned && wide_rows > 0) {
      const int closed_from = run_open(prefetches, budget_bits);
      if (!kPrecomputed) run_closed(closed_from);
    }
    if (!kAligned && !kPrecomputed) run_unaligned(full_rows, budget_bits);
    const int lane = 2 * threadIdx.x;
    const int valid_a = valid_steps_of(block, lane, g.steps, g.block_symbols, g.logical_numel, g.lane_mask);
    const int valid_b = valid_steps_of(block, lane + 1, g.steps, g.block_symbols, g.logical_numel, g.lane_mask);
#pragma unroll 1
    for (int step0 = kPrecomputed ? wide_rows : full_rows; step0 < rows_used; step0 += kChunkRows) {
      Pair pairs[kChunkPairs];
#pragma unroll
      for (int k = 0; k < kChunkPairs; ++k) {
        Pair& p = pairs[k];
        p = look_up(guarded_word(step0, k, false), guarded_word(step0, k, true));
        const int step = step0 + 2 * k;  // padding carries no bits
        if (step >= valid_a) p.a0 = 0u;
        if (step + 1 >= valid_a) p.a1 = 0u;
        if (step >= valid_b) p.b0 = 0u;
        if (step + 1 >= valid_b) p.b1 = 0u;
      }
#pragma unroll
      for (int k = 0; k < kChunkPairs; ++k) {
        store_sides(pairs[k], k);
        append<true>(pairs[k], step0 + 2 * k, budget_bits);
      }
      side_rows += kChunkRows * kLanes;
    }
  }
};

template <bool kPrecomputed, int kLaneMask, bool kAligned>
__device__ __forceinline__ void encode_block(const void* __restrict__ src, uint8_t* __restrict__ side,
                                             uint32_t* __restrict__ encoded,
                                             const int32_t* shifted_encode,
                                             uint8_t* __restrict__ extra_starts,
                                             int32_t* __restrict__ summaries, const EncodeShape& g_in,
                                             int64_t block) {
  EncodeShape g = g_in;
  if (kLaneMask >= 0) g.lane_mask = kLaneMask;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  EncodeSharedHead& sh = *reinterpret_cast<EncodeSharedHead*>(smem_raw);
  uint32_t* image = reinterpret_cast<uint32_t*>(smem_raw + sizeof(EncodeSharedHead));

  const int tid = threadIdx.x;
  const int64_t block_base = block * (int64_t)g.block_symbols;
  // Rows of this block that hold elements, in whole chunks.  Rows of pure padding (the tail of a
  // ragged or tiny tensor) carry no bits; their side bytes are cleared in one sweep.
  const int64_t left = g.logical_numel - block_base;
  const int in_block = (int)max((int64_t)0, min((int64_t)g.block_symbols, left));
  const int full_rows = in_block / (kChunkRows * kLanes) * kChunkRows;
  const int rows_used = (in_block + kChunkRows * kLanes - 1) / (kChunkRows * kLanes) * kChunkRows;
  BlockEncoder<kPrecomputed, kLaneMask, kAligned> encoder{
      static_cast<const char*>(src) + block_base * (kPrecomputed ? 1 : 2),
      side + block_base + 2 * tid, g, block, 0u,
      kAligned ? full_rows : 0, {}};
  // A full block is fetched ahead; the first portions now, with everything up to the table still
  // to come.
  const bool prefetches = !kPrecomputed && tid == 0;
  if (prefetches && encoder.wide_rows >= kPrefetchRows) encoder.prefetch(0, kPrefetchRows);
  clear_image<kPairThreads>(image, g.fixed_words);
  if (block == 0 && tid < 4) encoded[g.streams * g.fixed_words + tid] = 0u;  // trailing pad words
  if (!kPrecomputed && rows_used < g.steps) {
    uint4* rest = reinterpret_cast<uint4*>(side + block_base + (int64_t)rows_used * kLanes);
    for (int i = tid; i < (g.steps - rows_used) * (kLanes / 16); i += kPairThreads)
      __stcs(rest + i, make_uint4(0u, 0u, 0u, 0u));
  }
  // Everything above is independent of the tensor's center.  The shifted table may come from a
  // kernel that is still running when this grid was launched with programmatic stream
  // serialisation (lct_compress): wait for it only now.
  cudaGridDependencySynchronize();
  load_encode_table<kPairThreads>(sh.table, shifted_encode);
  __syncthreads();

  encoder.lanes[0].open(shared_address(image + 2 * tid));
  encoder.lanes[1].open(shared_address(image + 2 * tid + 1));
  encoder.table = after_barrier(shared_address(sh.table));
  encoder.run(rows_used, full_rows, prefetches);
  finish_block<kPairThreads>(encoder.lanes, image, sh.scan, encoded, extra_starts, summaries, block,
               g.n_blocks, g.streams, g.steps, g.fixed_words);
}

// A closed lane must stay on the checked path: it closed within one pair (32 bits) of its budget.
static_assert(kChunkBits >= 32, "a closed lane is near its budget");

template <bool kPrecomputed, int kLaneMask, bool kAligned>
__global__ void __launch_bounds__(kPairThreads, kEncodeMinCtas)
encode_kernel(const void* __restrict__ src, uint8_t* __restrict__ side, uint32_t* __restrict__ encoded, const int32_t* shifted_encode,
              uint8_t* __restrict__ extra_starts, int32_t* __restrict__ summaries, EncodeShape g) {
  encode_block<kPrecomputed, kLaneMask, kAligned>(src, side, encoded, shifted_encode, extra_starts,
                                                  summaries, g, blockIdx.x);
}

// Shape of one job of a batch (all jobs share the geometry in `common`).
template <typename Job>
__device__ __forceinline__ EncodeShape shape_of_job(const Job& job, const EncodeShape& common) {
  EncodeShape g = common;
  g.size = job.size;
  g.logical_numel = job.logical_numel;
  g.n_blocks = job.size / common.block_symbols;
  g.streams = g.n_blocks * kLanes;
  return g;
}

template <typename Job>
__device__ __forceinline__ int find_encode_job(const Job* jobs, int n_jobs, int64_t block) {
  int lo = 0, hi = n_jobs - 1;
  while (lo < hi) {  // last job with first_block <= block
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].first_block <= block) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <int kLaneMask>
__global__ void __launch_bounds__(kPairThreads, kEncodeMinCtas)
encode_batch_kernel(const lct_encode_job* __restrict__ jobs, int n_jobs,
                    const int32_t* shifted_encode, uint8_t* __restrict__ extra_starts,
                    int32_t* __restrict__ summaries, EncodeShape common) {
  const int64_t block = blockIdx.x;
  const int j = find_encode_job(jobs, n_jobs, block);
  const lct_encode_job& job = jobs[j];
  const EncodeShape g = shape_of_job(job, common);
  const auto run = [&](auto aligned) {
    encode_block<false, kLaneMask, decltype(aligned)::value>(
        job.src, job.side, reinterpret_cast<uint32_t*>(job.encoded), shifted_encode + 256 * (int64_t)j,
        extra_starts + job.first_block * kLanes, summaries + 4 * job.first_block, g,
        block - job.first_block);
  };
  if ((reinterpret_cast<uintptr_t>(job.src) & 3u) == 0) run(std::true_type());
  else run(std::false_type());
}

// Compact overflow metadata and raw exponent tails of one block.  Lanes are
// listed in increasing order; a lane's tail holds exponent - 127 for every
// row from its overflow start to the end of the block (padding rows read as
// exponent byte 0).
template <bool kPrecomputed>
__device__ __forceinline__ void compact_block(const void* src, uint8_t* lanes,
                                              uint8_t* starts, uint8_t* tail,
                                              const int32_t* descriptor, const int32_t* counts,
                                              int32_t* blocks_out,
                                              const uint8_t* extra_starts,
                                              const int32_t* summaries,
                                              const EncodeShape& g, int64_t block) {
  __shared__ int scan[33];
  const int tid = threadIdx.x;
  const int count = summaries[block];
  const int first = summaries[2 * g.n_blocks + block];
  const int byte_base = summaries[3 * g.n_blocks + block];
  if (tid == 0) {
    blocks_out[block] = count;
    blocks_out[g.n_blocks + block] = first;
    blocks_out[2 * g.n_blocks + block] = byte_base;
  }
  if (count == 0) return;
  int64_t lane_off = 0, start_off = 0, tail_off = 0;
  if (descriptor != nullptr) {
    if (descriptor[2] != 0) return;  // no arena region: nothing may be written
    const int64_t total = counts[0];
    lane_off = descriptor[0];
    start_off = lane_off + total;
    tail_off = lane_off + 2 * total;
  }
  const int start = extra_starts[block * kLanes + tid];
  const bool bad = start != 255;
  int unused;
  const int rank = block_exclusive_scan(bad ? 1 : 0, scan, &unused);
  const int local = block_exclusive_scan(bad ? g.steps - start : 0, scan, &unused);
  if (bad) {
    lanes[lane_off + first + rank] = (uint8_t)tid;
    starts[start_off + first + rank] = (uint8_t)start;
  }
  // Each warp copies the tails of its own 32 lanes, one lane at a time, with
  // the 32 threads striding over that lane's rows.
  const int lane_in_warp = tid & 31;
  const int warp_first_lane = tid & ~31;
  unsigned pending = __ballot_sync(0xFFFFFFFFu, bad);
  const int64_t row0 = block * g.steps;
  while (pending) {
    const int owner = __ffs(pending) - 1;
    pending &= pending - 1;
    const int lane = warp_first_lane + owner;
    const int lane_start = __shfl_sync(0xFFFFFFFFu, start, owner);
    const int lane_local = __shfl_sync(0xFFFFFFFFu, local, owner);
    uint8_t* dst = tail + tail_off + byte_base + lane_local;
    for (int row = lane_start + lane_in_warp; row < g.steps; row += 32) {
      const int64_t n = row0 + row;
      const int64_t logical = n * kLanes + (lane ^ (int)(n & g.lane_mask));
      int byte = 0;
      if (logical < g.logical_numel) {
        byte = kPrecomputed ? (int)static_cast<const uint8_t*>(src)[logical]
                            : ((int)static_cast<const uint16_t*>(src)[logical] >> 7) & 255;
      }
      dst[row - lane_start] = (uint8_t)(byte - 127);
    }
  }
}

template <bool kPrecomputed>
__global__ void __launch_bounds__(kThreads)
compact_tails_kernel(const void* src, uint8_t* lanes, uint8_t* starts, uint8_t* tail,
                     const int32_t* descriptor, const int32_t* counts, int32_t* blocks_out,
                     const uint8_t* extra_starts, const int32_t* summaries,
                     EncodeShape g) {
  cudaGridDependencySynchronize();  // prefixes and the reservation come from the scan in front
  compact_block<kPrecomputed>(src, lanes, starts, tail, descriptor, counts, blocks_out,
                              extra_starts, summaries, g, blockIdx.x);
}

// Where the tail pass finds a job's exponents: the BF16 source of an encode job, the raw
// result exponents a fused update left for its overflowing lanes.
__device__ __forceinline__ const void* tail_source(const lct_encode_job& job) { return job.src; }
__device__ __forceinline__ const void* tail_source(const lct_update_job& job) { return job.spill; }

template <typename Job, bool kPrecomputed>
__global__ void __launch_bounds__(kThreads)
compact_batch_kernel(const Job* __restrict__ jobs, int n_jobs, uint8_t* arena_payload,
                     const uint8_t* extra_starts, const int32_t* summaries,
                     EncodeShape common) {
  cudaGridDependencySynchronize();  // prefixes and reservations come from the scan in front
  const int64_t block = blockIdx.x;
  const Job& job = jobs[find_encode_job(jobs, n_jobs, block)];
  const EncodeShape g = shape_of_job(job, common);
  compact_block<kPrecomputed>(tail_source(job), arena_payload, arena_payload, arena_payload,
                              job.descriptor, job.counts, job.blocks_out,
                              extra_starts + job.first_block * kLanes,
                              summaries + 4 * job.first_block, g, block - job.first_block);
}

static int check_encode_shape(int64_t size, int64_t logical_numel, int block_symbols, int steps,
                              int fixed_words, EncodeShape* g) {
  if (steps != 128 && steps != 256) return LCT_E_BAD_GEOMETRY;
  if (block_symbols != steps * kLanes) return LCT_E_BAD_GEOMETRY;
  if (fixed_words < 2 || fixed_words > 64) return LCT_E_BAD_GEOMETRY;
  if (size <= 0 || size % block_symbols != 0) return LCT_E_BAD_ARGUMENT;
  if (logical_numel <= 0 || logical_numel > size) return LCT_E_BAD_ARGUMENT;
  const int64_t blocks = size / block_symbols;
  if (blocks > 0x7FFFFFFFLL) return LCT_E_TOO_LARGE;
  g->size = size;
  g->logical_numel = logical_numel;
  g->n_blocks = blocks;
  g->streams = blocks * kLanes;
  g->block_symbols = block_symbols;
  g->steps = steps;
  g->fixed_words = fixed_words;
  g->lane_mask = lct::lane_mask_now();
  return 0;
}

}  // namespace lct

extern "C" {

// Argument checks and launch shared by lct_encode and lct_compress.
static int launch_encode(const void* src, uint8_t* side, int32_t* encoded,
                         const int32_t* shifted_encode, uint8_t* extra_starts, int32_t* summaries,
                         int64_t size, int64_t logical_numel, int block_symbols, int steps,
                         int fixed_words, int precomputed, bool overlapped, cudaStream_t st) {
  lct::EncodeShape g;
  int rc = lct::check_encode_shape(size, logical_numel, block_symbols, steps, fixed_words, &g);
  if (rc) return rc;
  if (src == nullptr || encoded == nullptr || shifted_encode == nullptr ||
      extra_starts == nullptr || summaries == nullptr)
    return LCT_E_NULL_POINTER;
  if (!precomputed && side == nullptr) return LCT_E_NULL_POINTER;
  const uintptr_t s = reinterpret_cast<uintptr_t>(src);
  if (!precomputed && (s & 1u)) return LCT_E_ALIGNMENT;
  if ((reinterpret_cast<uintptr_t>(encoded) & 15u) ||
      (!precomputed && (reinterpret_cast<uintptr_t>(side) & 15u)))
    return LCT_E_ALIGNMENT;
  const bool aligned = (s & (precomputed ? 1u : 3u)) == 0;
  const size_t shared = sizeof(lct::EncodeSharedHead) + (size_t)fixed_words * lct::kLanes * 4;
  uint32_t* words = reinterpret_cast<uint32_t*>(encoded);
  const bool swizzled = g.lane_mask == 254;
  // (Unaligned sources are rare: one kernel for both lane mappings serves them.)
  auto kernel = precomputed ? (!aligned    ? lct::encode_kernel<true, -1, false>
                               : swizzled  ? lct::encode_kernel<true, 254, true>
                                           : lct::encode_kernel<true, -1, true>)
                            : (!aligned    ? lct::encode_kernel<false, -1, false>
                               : swizzled  ? lct::encode_kernel<false, 254, true>
                                           : lct::encode_kernel<false, -1, true>);
  rc = (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
  if (rc) return rc;
  if (overlapped)
    return lct::launch_overlapped(kernel, (unsigned)g.n_blocks, lct::kPairThreads, shared, st, src,
                                  side, words, shifted_encode, extra_starts, summaries, g);
  kernel<<<(unsigned)g.n_blocks, lct::kPairThreads, shared, st>>>(src, side, words, shifted_encode,
                                                              extra_starts, summaries, g);
  return (int)cudaGetLastError();
}

}  // extern "C"

namespace lct {

int launch_compact_batch(const lct_update_job* jobs, int n_jobs, int64_t total_blocks,
                         uint8_t* arena_payload, const uint8_t* extra_starts,
                         const int32_t* summaries, int block_symbols, int steps, int fixed_words,
                         cudaStream_t stream) {
  EncodeShape g;
  const int rc = check_encode_shape(block_symbols, block_symbols, block_symbols, steps, fixed_words, &g);
  if (rc) return rc;
  return launch_overlapped(compact_batch_kernel<lct_update_job, true>, (unsigned)total_blocks,
                           kThreads, 0, stream, jobs, n_jobs, arena_payload, extra_starts,
                           summaries, g);
}

int launch_compact(const void* src, uint8_t* lanes, uint8_t* starts, uint8_t* tail,
                          const int32_t* descriptor, const int32_t* counts, int32_t* blocks_out,
                          const uint8_t* extra_starts, const int32_t* summaries, int64_t size,
                          int64_t logical_numel, int block_symbols, int steps, int precomputed,
                          bool overlapped, cudaStream_t st) {
  lct::EncodeShape g;
  int rc = lct::check_encode_shape(size, logical_numel, block_symbols, steps, 2, &g);
  if (rc) return rc;
  if (src == nullptr || counts == nullptr || blocks_out == nullptr || extra_starts == nullptr ||
      summaries == nullptr)
    return LCT_E_NULL_POINTER;
  // lanes/starts/tail may be NULL only when the tensor has no overflow at all
  // (zero-size private tensors); the kernel then never dereferences them.
  auto kernel = precomputed ? lct::compact_tails_kernel<true> : lct::compact_tails_kernel<false>;
  if (overlapped)
    return lct::launch_overlapped(kernel, (unsigned)g.n_blocks, lct::kThreads, 0, st, src, lanes,
                                  starts, tail, descriptor, counts, blocks_out, extra_starts,
                                  summaries, g);
  kernel<<<(unsigned)g.n_blocks, lct::kThreads, 0, st>>>(src, lanes, starts, tail, descriptor,
                                                         counts, blocks_out, extra_starts,
                                                         summaries, g);
  return (int)cudaGetLastError();
}

}  // namespace lct

extern "C" {

int lct_encode(const void* src, uint8_t* side, int32_t* encoded, const int32_t* shifted_encode,
               uint8_t* extra_starts, int32_t* summaries, int64_t size, int64_t logical_numel,
               int block_symbols, int steps, int fixed_words, int precomputed, void* stream) {
  return launch_encode(src, side, encoded, shifted_encode, extra_starts, summaries, size,
                       logical_numel, block_symbols, steps, fixed_words, precomputed, false,
                       static_cast<cudaStream_t>(stream));
}

int lct_compact_tails(const void* src, uint8_t* lanes, uint8_t* starts, uint8_t* tail,
                      const int32_t* descriptor, const int32_t* counts, int32_t* blocks_out,
                      const uint8_t* extra_starts, const int32_t* summaries, int64_t size,
                      int64_t logical_numel, int block_symbols, int steps, int precomputed,
                      void* stream) {
  return lct::launch_compact(src, lanes, starts, tail, descriptor, counts, blocks_out, extra_starts,
                        summaries, size, logical_numel, block_symbols, steps, precomputed, false,
                        static_cast<cudaStream_t>(stream));
}

int lct_compress(const void* src, int precomputed, uint8_t* side, int32_t* encoded,
                 const int32_t* encode_table, const int32_t* decode_table, int32_t* center,
                 int32_t* shifted_encode, int32_t* shifted_decode, uint8_t* extra_starts,
                 int32_t* summaries, int32_t* counts, int32_t* descriptor, int32_t* blocks_out,
                 void* arena_storage, int max_free_regions, int64_t size, int64_t logical_numel,
                 int block_symbols, int steps, int fixed_words, void* stream) {
  if (encode_table == nullptr || decode_table == nullptr || center == nullptr ||
      shifted_encode == nullptr || counts == nullptr || descriptor == nullptr ||
      arena_storage == nullptr || src == nullptr)
    return LCT_E_NULL_POINTER;
  if (max_free_regions <= 0 || (max_free_regions & (max_free_regions - 1))) return LCT_E_BAD_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // 1. center + tables: an ordinary launch, so everything queued before this call is complete
  //    and visible before any of the four kernels starts.
  int rc = lct::launch_center(src, logical_numel, precomputed != 0, encode_table, decode_table,
                              center, shifted_encode, shifted_decode, false, st);
  if (rc) return rc;
  // 2-4. each of these may be scheduled while its predecessor still runs and waits on the
  //    device for it where its first dependent read is.
  rc = launch_encode(src, side, encoded, shifted_encode, extra_starts, summaries, size,
                     logical_numel, block_symbols, steps, fixed_words, precomputed, true, st);
  if (rc) return rc;
  rc = lct::launch_scan_allocate(summaries, counts, descriptor, arena_storage, size / block_symbols,
                                 max_free_regions, true, st);
  if (rc) return rc;
  // The arena payload starts after the allocator words, padded to 16 bytes.
  const size_t metadata = ((size_t)8 * max_free_regions + 12 + 15) / 16 * 16;
  uint8_t* payload = static_cast<uint8_t*>(arena_storage) + metadata;
  return lct::launch_compact(src, payload, payload, payload, descriptor, counts, blocks_out,
                        extra_starts, summaries, size, logical_numel, block_symbols, steps,
                        precomputed, true, st);
}

}  // extern "C"

extern "C" {

int lct_compress_batch(const lct_encode_job* jobs, int n_jobs, int64_t total_blocks,
                       const int32_t* encode_table, const int32_t* decode_table,
                       void* arena_storage, int max_free_regions, uint8_t* extra_starts,
                       int32_t* summaries, int32_t* shifted_encode, int block_symbols, int steps,
                       int fixed_words, void* stream) {
  if (jobs == nullptr || encode_table == nullptr || decode_table == nullptr ||
      arena_storage == nullptr || extra_starts == nullptr || summaries == nullptr ||
      shifted_encode == nullptr)
    return LCT_E_NULL_POINTER;
  if (n_jobs <= 0 || total_blocks <= 0 || total_blocks > 0x7FFFFFFFLL) return LCT_E_BAD_ARGUMENT;
  if (max_free_regions <= 0 || (max_free_regions & (max_free_regions - 1))) return LCT_E_BAD_ARGUMENT;
  lct::EncodeShape g;
  int rc = lct::check_encode_shape(block_symbols, block_symbols, block_symbols, steps, fixed_words, &g);
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if ((rc = lct::launch_center_batch(jobs, n_jobs, encode_table, decode_table, shifted_encode, st)))
    return rc;
  const size_t shared = sizeof(lct::EncodeSharedHead) + (size_t)fixed_words * lct::kLanes * 4;
  auto encode_all = g.lane_mask == 254 ? lct::encode_batch_kernel<254> : lct::encode_batch_kernel<-1>;
  rc = (int)cudaFuncSetAttribute(encode_all, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
  if (rc) return rc;
  // Centers first (ordinary launch); the three kernels behind it may each be scheduled while
  // their predecessor still runs and wait for it on the device.
  if ((rc = lct::launch_overlapped(encode_all, (unsigned)total_blocks, lct::kPairThreads,
                                   shared, st, jobs, n_jobs, shifted_encode, extra_starts,
                                   summaries, g)))
    return rc;
  if ((rc = lct::launch_scan_batch(jobs, n_jobs, summaries, arena_storage, max_free_regions,
                                   block_symbols, st)))
    return rc;
  // The arena payload starts after the allocator words, padded to 16 bytes.
  const size_t metadata = ((size_t)8 * max_free_regions + 12 + 15) / 16 * 16;
  return lct::launch_overlapped(lct::compact_batch_kernel<lct_encode_job, false>,
                                (unsigned)total_blocks, lct::kThreads, 0, st, jobs, n_jobs,
                                static_cast<uint8_t*>(arena_storage) + metadata, extra_starts,
                                summaries, g);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Encode without any caller-side scratch: lct_encode_noalloc
// ---------------------------------------------------------------------------
//
// lct_encode needs two work buffers from its caller (one "first overflow step"
// byte per stream and four ints per block) that exist only to be handed to the
// summary scan.  Some callers cannot provide them: a serving loop that must
// not allocate once it has started, a host that gave all device memory to
// another allocator at start-up, or a C program that links this library and
// has no allocator at all.  For them the work buffers below live in the
// library image itself.  The first call on a GPU looks the array's address up
// and should come before any stream capture.

namespace lct {

// Largest tensor the built-in scratch serves: 1024 codec blocks (64 Mi
// elements in the 65536-element layouts, 32 Mi in the 32768-element ones).
constexpr int kNoAllocMaxBlocks = 1024;
constexpr size_t kNoAllocSummaryBytes = (size_t)kNoAllocMaxBlocks * 4 * sizeof(int32_t);
constexpr size_t kNoAllocBytes = kNoAllocSummaryBytes + (size_t)kNoAllocMaxBlocks * kLanes;

// 272 KiB per GPU that loads the library, held until the process exits.
// [0, 16 KiB): block summaries, int32[4 * blocks]; then one byte per stream.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

constexpr int kMaxDevices = 64;
static unsigned char* g_noalloc_address[kMaxDevices];  // device address of the array, per GPU

// In host code `g_noalloc_scratch` is only a handle for the runtime, not an
// address a kernel may use; the device address has to be asked for, once per
// GPU, while that GPU is current.  Returns 0 or a cudaError_t.
static int noalloc_scratch_address(unsigned char** out) {
  int device = -1;
  cudaError_t rc = cudaGetDevice(&device);
  if (rc != cudaSuccess) return (int)rc;
  if (device < 0 || device >= kMaxDevices) return LCT_E_BAD_ARGUMENT;
  unsigned char* known = __atomic_load_n(&g_noalloc_address[device], __ATOMIC_ACQUIRE);
  if (known == nullptr) {
    void* address = nullptr;
    rc = cudaGetSymbolAddress(&address, g_noalloc_scratch);
    if (rc != cudaSuccess) return (int)rc;
    if (address == nullptr) return (int)cudaErrorInvalidSymbol;
    known = static_cast<unsigned char*>(address);
    // Two threads racing here store the same value.
    __atomic_store_n(&g_noalloc_address[device], known, __ATOMIC_RELEASE);
  }
  *out = known;
  return 0;
}

}  // namespace lct

extern "C" {

int lct_scan_allocate(int32_t* summaries, int32_t* counts, int32_t* descriptor,
                      void* arena_storage, int64_t blocks, int max_free_regions, void* stream);

int lct_encode_noalloc(const void* src, uint8_t* side, int32_t* encoded,
                       const int32_t* shifted_encode, int32_t* counts, int64_t size,
                       int64_t logical_numel, int block_symbols, int steps, int fixed_words,
                       int precomputed, void* stream) {
  if (counts == nullptr) return LCT_E_NULL_POINTER;
  if (block_symbols <= 0 || size <= 0) return LCT_E_BAD_ARGUMENT;
  const int64_t blocks = (size + block_symbols - 1) / block_symbols;
  if (blocks > lct::kNoAllocMaxBlocks) return LCT_E_SCRATCH_LIMIT;
  unsigned char* scratch = nullptr;
  int rc = lct::noalloc_scratch_address(&scratch);
  if (rc) return rc;
  int32_t* summaries = reinterpret_cast<int32_t*>(scratch);
  uint8_t* extra_starts = scratch + lct::kNoAllocSummaryBytes;
  // Both kernels overwrite every scratch byte they later read (all streams of
  // the tensor, all four summary rows), so nothing left by an earlier call is
  // ever consumed and nothing has to be cleared first.
  rc = lct_encode(src, side, encoded, shifted_encode, extra_starts, summaries, size, logical_numel,
                  block_symbols, steps, fixed_words, precomputed, stream);
  if (rc) return rc;
  return lct_scan_allocate(summaries, counts, nullptr, nullptr, blocks, 256, stream);
}

}  // extern "C"
