// Table-driven decoder and the fused decode -> pointwise operation kernels.
//
// One CTA of 256 threads per codec block, thread = lane (lanes.cuh, lane_reader.cuh).
//
// Prologue: the block's payload and the 16 KB two-symbol table of this tensor's center are copied
// into shared memory with cp.async while the block's overflow map is expanded.
//
// Then, per row pair: one table lookup gives a lane's two exponents and the bits to consume (two
// funnel shifts by the table entry itself); one shuffle gives every thread both columns' exponents
// of one row; these are joined with two side bytes out of the warp's ring to one word of the dense
// tensor.  The stores of a pair are issued while the next pair's lookup is under way.  The only
// divergent path is the rare entry that is not a full pair.
//
// Bound by instruction issue (75 % of the issue slots, 45 instructions per warp and pair at 64 Mi
// weights, a quarter of them the not-a-full-pair path).  Against the former form (16-row tiles
// transposed through shared memory to eight columns per thread, 50 instructions), at 64 Mi
// elements: 69.0 -> 59.3 us (weights with outliers), 58.8 -> 52.1 (normal), 60.6 -> 52.8 (half
// zeros, overflow); 1 Mi: 11.3 -> 9.4.  Measured and left: two lanes per thread (96 us: half the
// warps, each with twice the serial chain), side bytes requested into registers (90 us: the loads'
// registers spill, which waits for every load at once), 3 instead of 4 CTAs per SM (61.0).
//
// Overflow lanes switch from the bit stream to their raw tail bytes at their recorded start step,
// inside the same launch.
#include "lane_reader.cuh"

namespace lct {

// ---------------------------------------------------------------------------
// Plain decode
// ---------------------------------------------------------------------------

// One codec block: 256 threads, thread = lane.  Per row pair a thread looks up one table entry of
// its lane - two symbols - exchanges exponents with its neighbour, joins those of its row with the
// side bytes of the two columns and stores one word.  Side bytes come through a ring in shared memory.
// kLaneMask: the lane mapping as a compile-time constant (254, the default mapping: the masked
// row addresses fold into constants), or -1 to take it from the shape at run time.
template <int kLaneMask>
struct BlockDecoder {
  const Shape& g;
  int64_t row0;
  DenseWords<uint16_t> out;
  RowExchange rows;
  SideRing sides;
  LaneWalk walk;

  __device__ __forceinline__ void chunk(int step0) {
    const uint32_t offset = word_offset(row0, step0, g.lane_mask);
    if (walk.whole_chunk(step0)) {
      uint32_t entry = 0u, neighbour = 0u, side = 0u;
      auto emit = [&](int k) {
        out.store(word_at<kLaneMask>(offset, k, g.lane_mask),
                  join_word(rows.exponents(entry, neighbour), side));
      };
#pragma unroll
      for (int k = 0; k < kWalkPairs; ++k) {
        entry = walk.read_pair(k, [&] { if (k > 0) emit(k - 1); });
        neighbour = rows.neighbours(entry);
        side = sides.pair(k);
      }
      emit(kWalkPairs - 1);
    } else {
      const bool full = out.holds_rows(step0 + kWalkRows);
      walk.read_chunk(step0, [&](int k, uint32_t entry) {
        const uint32_t at = word_at<kLaneMask>(offset, k, g.lane_mask);
        const uint32_t word = join_word(rows.exponents(entry, rows.neighbours(entry)), sides.pair(k));
        if (full) out.store(at, word);
        else out.store_guarded(at, word);
      });
    }
  }
};

template <int kLaneMask>
__device__ __forceinline__ void decode_block(const OperandView& a, const Shape& g_in,
                                             uint16_t* __restrict__ out, int64_t block) {
  Shape g = g_in;
  if (kLaneMask >= 0) g.lane_mask = kLaneMask;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int64_t block_base = block * (int64_t)g.block_symbols;
  const ReaderShared sh = carve_reader(smem_raw, 0, 1, g.fixed_words, kRingBytes);
  // Rows of pure padding (the tail of a ragged or tiny tensor) have nothing to decode or store.
  const int rows_used = rows_in_use(g, block);
  BlockDecoder<kLaneMask> decoder{g, block * g.steps, {out + block_base, elements_left(g, block)},
                                  {}, {}, {}};
  decoder.sides.open(smem_raw + kTableBytes, a.side + block_base, rows_used);
  stage_operand(sh, a, g, block);
  decoder.rows.open();
  cp_async_wait_all();
  __syncthreads();
  decoder.walk.open(sh, a, g, block);
#pragma unroll 1
  for (int step0 = 0; step0 < rows_used; step0 += kWalkRows) {
    decoder.sides.wait();
    decoder.chunk(step0);
    decoder.sides.advance();
  }
}

// Resident CTAs per SM the decoder is compiled for.
constexpr int kDecodeMinCtas = 4;
template <int kLaneMask>
__global__ void __launch_bounds__(kThreads, kDecodeMinCtas)
decode_kernel(OperandView a, Shape g, uint16_t* __restrict__ out) {
  decode_block<kLaneMask>(a, g, out, blockIdx.x);
}

// Many tensors of one geometry in one launch: CTA b serves the job whose block
// range contains b.  Jobs are sorted by first_block.
__device__ __forceinline__ OperandView view_of_job(const lct_operand& in) {
  OperandView v;
  v.encoded = reinterpret_cast<const uint32_t*>(in.encoded);
  v.side = in.side;
  v.center = in.center;
  v.pair_table = in.pair_table;
  v.lanes = in.overflow.lanes;
  v.starts = in.overflow.starts;
  v.tail = in.overflow.tail;
  v.descriptor = in.overflow.descriptor;
  v.count = in.overflow.count;
  v.blocks = in.overflow.blocks;
  v.base = in.overflow.base;
  v.mode = in.overflow.mode;
  return v;
}

template <typename Job>
__device__ __forceinline__ int find_job(const Job* jobs, int n_jobs, int64_t block) {
  int lo = 0, hi = n_jobs - 1;
  while (lo < hi) {  // last job with first_block <= block
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].first_block <= block) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Operand in a peer GPU's memory: bring one block's side bytes over in full 16-byte requests
// (four in flight per thread) so that the decoder reads a local copy.  `chunks` (2048 or 4096)
// is a multiple of 4 * kThreads.  Not inlined: its registers are dead before the decoder starts.
static __device__ __noinline__ void stage_side_bytes(const uint8_t* __restrict__ from_bytes,
                                                     uint8_t* __restrict__ to_bytes, int chunks) {
  const uint4* from = reinterpret_cast<const uint4*>(from_bytes);
  uint4* to = reinterpret_cast<uint4*>(to_bytes);
  for (int i = threadIdx.x; i < chunks; i += 4 * kThreads) {
    uint4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = __ldcs(from + i + k * kThreads);
#pragma unroll
    for (int k = 0; k < 4; ++k) to[i + k * kThreads] = v[k];
  }
  __syncthreads();  // the copy is read by other threads of this CTA only
}

template <int kLaneMask>
__global__ void __launch_bounds__(kThreads, kDecodeMinCtas)
decode_batch_kernel(const lct_decode_job* __restrict__ jobs, int n_jobs, Shape common) {
  const int64_t block = blockIdx.x;
  const lct_decode_job& job = jobs[find_job(jobs, n_jobs, block)];
  Shape g = common;
  g.size = job.size;
  g.logical_numel = job.logical_numel;
  g.n_blocks = job.size / common.block_symbols;
  g.streams = g.n_blocks * kLanes;
  OperandView view = view_of_job(job.operand);
  const int64_t local_block = block - job.first_block;
  if (job.side_stage != nullptr) {
    const int64_t base = local_block * (int64_t)g.block_symbols;
    stage_side_bytes(view.side + base, job.side_stage + base, g.block_symbols / 16);
    view.side = job.side_stage;
  }
  decode_block<kLaneMask>(view, g, reinterpret_cast<uint16_t*>(job.out), local_block);
}

// ---------------------------------------------------------------------------
// Fused pointwise operations
// ---------------------------------------------------------------------------

// One codec block, divided among threads as in the plain decoder.  The second operand is a dense
// tensor (its words are requested ahead, like the side bytes) or, kDual, another compressed one,
// whose lane the same thread walks.
// kForm: the operation's arithmetic, a constant of the kernel (see Operation).
// kCompressed: the result leaves as side bytes (storage order) and exponent bytes (`auxiliary`,
// element order) instead of dense values; padding counts as +0.0.
// Measured, a * A + B / A * B of one compressed operand, us (former tile form -> this): normal
// codebook 32768 elements 14.8 -> 9.6 / 10.3 -> 8.9, 16 Mi 26.1 -> 22.9 / 21.6 -> 20.8, 64 Mi 89.8 ->
// 72.5 / 74.9 -> 67.6; half-zero codebook 28 Mi 48.3 -> 41.4 / 40.6 -> 38.4; two compressed operands,
// 12 Mi 44.3 -> 38.7.
// kAligned: the dense operand's words of two values are aligned.  Where they are not, a word is
// two loads of two bytes, joined only when it is used (joined at once, the loads' latency would be
// waited for), and a chunk's registers are requested again as they become free, half a chunk
// ahead, in place of a second buffer.  a * A + B with B at an odd multiple of two bytes, normal
// codebook, us (tile form -> guarded loads of single values -> this): 32768 elements 18.7 -> 18.6 ->
// 11.8, 32 Mi 75 -> 87 -> 45, 64 Mi 140 -> 169 -> 87.
template <bool kDual, int kLaneMask, int kForm, bool kCompressed, bool kAligned>
struct BlockPointwise {
  const Shape& g;
  Operation<kForm> operation;
  int64_t row0;
  DenseWords<const uint16_t> other;
  int wide_rows;  // rows, in whole chunks, of `other` that are full
  DenseWords<uint16_t> out;  // dense result
  uint8_t* side_out;
  DenseWords<uint8_t> exponents_out;
  int rows_used;
  RowExchange rows;
  SideRing sides_a, sides_b;
  LaneWalk walk_a, walk_b;

  struct Buffer {
    uint32_t word[kWalkPairs];  // or its first value
    uint32_t second[kAligned ? 1 : kWalkPairs];

    __device__ __forceinline__ uint32_t operator[](int k) const {
      return kAligned ? word[k] : word[k] | (second[k] << 16);
    }
  };
  template <int kFrom = 0, int kTo = kWalkPairs>
  __device__ __forceinline__ void request(Buffer& words, int step0) const {
    if (kDual || step0 >= rows_used) return;
    const uint32_t offset = word_offset(row0, step0, g.lane_mask);
#pragma unroll
    for (int k = kFrom; k < kTo; ++k) {
      const uint32_t at = word_at<kLaneMask>(offset, k, g.lane_mask);
      if (kAligned) {
        words.word[k] = step0 < wide_rows ? other.load(at) : other.load_guarded(at);
      } else if (step0 < wide_rows) {
        words.word[k] = other.load_value(at);
        words.second[k] = other.load_value(at + 1);
      } else {
        words.word[k] = other.load_guarded(at);
        words.second[k] = 0u;
      }
    }
  }
  __device__ __forceinline__ void emit(int step, uint32_t at, bool guarded, uint32_t exponents_a,
                                       uint32_t exponents_b, uint32_t from_a, uint32_t from_b) const {
    const uint32_t left = join_word(exponents_a, from_a);
    const uint32_t right = kDual ? join_word(exponents_b, from_b) : from_b;
    uint32_t result = operation(left, right);
    if (!kCompressed) {
      if (guarded) out.store_guarded(at, result);
      else out.store(at, result);
      return;
    }
    if (guarded) {
      if ((int)at >= out.left) result = 0u;
      else if ((int)at + 1 >= out.left) result &= 0xFFFFu;
    }
    uint32_t sides, exponents;
    split_words(result, 0u, &sides, &exponents);
    *reinterpret_cast<uint16_t*>(side_out + step * kLanes) = (uint16_t)sides;
    if (guarded)
      exponents_out.store_guarded(at, (exponents & 255u) | ((exponents & 0xFF00u) << 8));
    else
      *reinterpret_cast<uint16_t*>(exponents_out.rows + at) = (uint16_t)exponents;
  }
  __device__ __forceinline__ void chunk(int step0, Buffer& words) {
    bool whole = walk_a.whole_chunk(step0);
    if constexpr (kDual) whole = walk_b.whole_chunk(step0) && whole;
    const uint32_t offset = word_offset(row0, step0, g.lane_mask);
    if (whole) {
      uint32_t entry_a = 0u, entry_b = 0u, neighbour_a = 0u, neighbour_b = 0u, side_a = 0u, side_b = 0u;
      auto emit_pair = [&](int k) {
        emit(step0 + 2 * k, word_at<kLaneMask>(offset, k, g.lane_mask), false,
             rows.exponents(entry_a, neighbour_a), rows.exponents(entry_b, neighbour_b), side_a,
             kDual ? side_b : words[k]);
      };
#pragma unroll
      for (int k = 0; k < kWalkPairs; ++k) {
        const uint32_t next_a = walk_a.read_pair(k, [&] { if (k > 0) emit_pair(k - 1); });
        if (!kAligned && k == kWalkPairs / 2)
          request<0, kWalkPairs / 2>(words, step0 + kWalkRows);
        entry_a = next_a;
        neighbour_a = rows.neighbours(entry_a);
        side_a = sides_a.pair(k);
        if constexpr (kDual) {
          entry_b = walk_b.read_pair(k, [] {});
          neighbour_b = rows.neighbours(entry_b);
          side_b = sides_b.pair(k);
        }
      }
      emit_pair(kWalkPairs - 1);
      if (!kAligned) request<kWalkPairs / 2>(words, step0 + kWalkRows);
    } else {
      const bool full = out.holds_rows(step0 + kWalkRows);
      int from_b = 0;
      uint32_t tail_b[kWalkPairs / 2] = {};
      if constexpr (kDual) {
        from_b = walk_b.head->overflow_start[threadIdx.x];
        walk_b.read_tail(tail_b, step0, from_b);
      }
      walk_a.read_chunk(step0, [&](int k, uint32_t entry_a) {
        const int step = step0 + 2 * k;
        uint32_t entry_b = 0u;
        if constexpr (kDual) {
          if ((k & 1) == 0) walk_b.cursor.clamp();
          entry_b = walk_b.read_any(step, from_b, (k & 1) ? tail_b[0] >> 8 : tail_b[0] << 8);
          if (k & 1) next_word(tail_b);
        }
        emit(step, word_at<kLaneMask>(offset, k, g.lane_mask), !full,
             rows.exponents(entry_a, rows.neighbours(entry_a)),
             kDual ? rows.exponents(entry_b, rows.neighbours(entry_b)) : 0u, sides_a.pair(k),
             kDual ? sides_b.pair(k) : words[0]);
        if (!kDual) next_word(words.word);
        if (!kAligned) next_word(words.second);
      });
      if (!kAligned) request(words, step0 + kWalkRows);
    }
  }
};

// Resident CTAs per SM.  Dense results: four, although three are up to 8 % faster below 10 Mi
// elements (no spills): with 444 slots a tensor of 448 to 592 blocks takes a second wave (28 Mi
// half zeros, A * B: 42.2 us with three, 38.4 with four; the tile form took 40.6).  Compressed
// results: three, 2 to 6 % faster than four throughout, the encoder behind included.
constexpr int pointwise_ctas(bool dual, bool compressed) { return dual ? 2 : compressed ? 3 : 4; }

template <bool kDual, int kLaneMask, int kForm, bool kCompressed, bool kAligned>
__global__ void __launch_bounds__(kThreads, pointwise_ctas(kDual, kCompressed))
pointwise_kernel(OperandView a, OperandView b, Shape g_in, const uint16_t* other, void* output,
                 uint8_t* auxiliary, OpSpec spec) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Shape g = g_in;
  if (kLaneMask >= 0) g.lane_mask = kLaneMask;  // see BlockDecoder
  constexpr int kOperands = kDual ? 2 : 1;
  const ReaderShared sh = carve_reader(smem_raw, 0, kOperands, g.fixed_words, kOperands * kRingBytes);
  const ReaderShared sh_b =
      carve_reader(smem_raw, kOperands - 1, kOperands, g.fixed_words, kOperands * kRingBytes);
  unsigned char* rings = smem_raw + kOperands * kTableBytes;
  const int64_t block = blockIdx.x;
  const int tid = threadIdx.x;
  const int64_t block_base = block * (int64_t)g.block_symbols;
  const int left = elements_left(g, block);
  const int rows_used = rows_in_use(g, block);
  uint8_t* side_out = static_cast<uint8_t*>(output) + block_base;
  using Block = BlockPointwise<kDual, kLaneMask, kForm, kCompressed, kAligned>;
  Block work{
      g, Operation<kForm>(spec), block * g.steps, {other + (kDual ? 0 : block_base), left},
      min(g.steps, left / kLanes) / kWalkRows * kWalkRows,
      {static_cast<uint16_t*>(output) + (kCompressed ? 0 : block_base), left},
      side_out + own_bytes(), {auxiliary + (kCompressed ? block_base : 0), left}, rows_used, {}, {}, {},
      {}, {}};
  typename Block::Buffer now, next;
  work.request(now, 0);
  if (kDual) work.sides_b.open(rings + kRingBytes, b.side + block_base, rows_used);
  work.sides_a.open(rings, a.side + block_base, rows_used);
  stage_operand(sh, a, g, block);
  if (kDual) stage_operand(sh_b, b, g, block);
  if (kCompressed)
    for (int row = rows_used + (tid >> 6); row < g.steps; row += 4)
      reinterpret_cast<uint32_t*>(side_out + row * kLanes)[tid & 63] = 0u;
  work.rows.open();
  cp_async_wait_all();
  __syncthreads();
  work.walk_a.open(sh, a, g, block);
  if (kDual) work.walk_b.open(sh_b, b, g, block);
#pragma unroll 1
  for (int step0 = 0; step0 < rows_used; step0 += kWalkRows) {
    if (kAligned) work.request(next, step0 + kWalkRows);
    if (kDual) work.sides_b.wait_both(work.sides_a);
    else work.sides_a.wait();
    work.chunk(step0, now);
    work.sides_a.advance();
    if (kDual) work.sides_b.advance();
    if (kAligned) now = next;
  }
}

using PointwiseKernel = void (*)(OperandView, OperandView, Shape, const uint16_t*, void*, uint8_t*,
                                OpSpec);
// (Unaligned dense operands are rare: one kernel for both lane mappings serves them.)
template <int kForm, bool kCompressed>
static PointwiseKernel pointwise_kernel_of(bool swizzled, bool aligned) {
  if (!aligned) return pointwise_kernel<false, -1, kForm, kCompressed, false>;
  return swizzled ? pointwise_kernel<false, 254, kForm, kCompressed, true>
                  : pointwise_kernel<false, -1, kForm, kCompressed, true>;
}
template <bool kCompressed>
static PointwiseKernel pointwise_kernel_of(int form, bool swizzled, bool aligned) {
  switch (form) {
    case kFormLerp: return pointwise_kernel_of<kFormLerp, kCompressed>(swizzled, aligned);
    case kFormRightScaled: return pointwise_kernel_of<kFormRightScaled, kCompressed>(swizzled, aligned);
    case kFormAdd: return pointwise_kernel_of<kFormAdd, kCompressed>(swizzled, aligned);
    case kFormMultiply: return pointwise_kernel_of<kFormMultiply, kCompressed>(swizzled, aligned);
    case kFormEmaSquare: return pointwise_kernel_of<kFormEmaSquare, kCompressed>(swizzled, aligned);
    default: return pointwise_kernel_of<kFormScaled, kCompressed>(swizzled, aligned);
  }
}

}  // namespace lct

extern "C" {

int lct_decode(const lct_operand* a, int16_t* out, int64_t size, int64_t logical_numel,
               int block_symbols, int steps, int fixed_words, int rare_length, void* stream) {
  lct::Shape g;
  lct::OperandView va;
  int rc = lct::check_shape(size, logical_numel, block_symbols, steps, fixed_words, rare_length, &g);
  if (rc) return rc;
  if ((rc = lct::view_of(a, &va)) != 0) return rc;
  if (out == nullptr) return LCT_E_NULL_POINTER;
  if (!lct::aligned16(out)) return LCT_E_ALIGNMENT;
  const size_t shared = lct::reader_shared_bytes(1, fixed_words, lct::kRingBytes);
  auto kernel = g.lane_mask == 254 ? lct::decode_kernel<254> : lct::decode_kernel<-1>;
  if ((rc = lct::opt_in_shared(kernel, shared)) != 0) return rc;
  kernel<<<(unsigned)g.n_blocks, lct::kThreads, shared, static_cast<cudaStream_t>(stream)>>>(
      va, g, reinterpret_cast<uint16_t*>(out));
  return (int)cudaGetLastError();
}

int lct_decode_batch(const lct_decode_job* jobs, int n_jobs, int64_t total_blocks,
                     int block_symbols, int steps, int fixed_words, int rare_length, void* stream) {
  if (jobs == nullptr) return LCT_E_NULL_POINTER;
  if (n_jobs <= 0 || total_blocks <= 0 || total_blocks > 0x7FFFFFFFLL) return LCT_E_BAD_ARGUMENT;
  lct::Shape g;
  int rc = lct::check_shape(block_symbols, block_symbols, block_symbols, steps, fixed_words,
                            rare_length, &g);
  if (rc) return rc;
  const size_t shared = lct::reader_shared_bytes(1, fixed_words, lct::kRingBytes);
  auto kernel = g.lane_mask == 254 ? lct::decode_batch_kernel<254> : lct::decode_batch_kernel<-1>;
  if ((rc = lct::opt_in_shared(kernel, shared)) != 0) return rc;
  kernel<<<(unsigned)total_blocks, lct::kThreads, shared, static_cast<cudaStream_t>(stream)>>>(
      jobs, n_jobs, g);
  return (int)cudaGetLastError();
}

int lct_pointwise(const lct_operand* a, const void* other, void* output, uint8_t* auxiliary,
                  const float* alpha, const float* beta, int op, int alpha_is_one,
                  int beta_is_one, int compressed_output, int64_t size, int64_t logical_numel,
                  int block_symbols, int steps, int fixed_words, int rare_length, void* stream) {
  lct::Shape g;
  lct::OperandView va;
  int rc = lct::check_shape(size, logical_numel, block_symbols, steps, fixed_words, rare_length, &g);
  if (rc) return rc;
  if ((rc = lct::view_of(a, &va)) != 0) return rc;
  if (other == nullptr || output == nullptr) return LCT_E_NULL_POINTER;
  if (compressed_output && auxiliary == nullptr) return LCT_E_NULL_POINTER;
  if ((rc = lct::check_op(op, alpha, beta, &alpha_is_one, &beta_is_one)) != 0) return rc;
  if (!lct::aligned16(output) || (compressed_output && !lct::aligned16(auxiliary)))
    return LCT_E_ALIGNMENT;
  if ((reinterpret_cast<uintptr_t>(other) & 1u) != 0) return LCT_E_ALIGNMENT;
  const lct::OpSpec spec{alpha, beta, op, alpha_is_one, beta_is_one};
  const size_t shared = lct::reader_shared_bytes(1, fixed_words, lct::kRingBytes);
  const int form = lct::form_of(op, alpha_is_one, beta_is_one);
  const bool swizzled = g.lane_mask == 254, aligned = (reinterpret_cast<uintptr_t>(other) & 3u) == 0;
  auto kernel = compressed_output ? lct::pointwise_kernel_of<true>(form, swizzled, aligned)
                                  : lct::pointwise_kernel_of<false>(form, swizzled, aligned);
  if ((rc = lct::opt_in_shared(kernel, shared)) != 0) return rc;
  kernel<<<(unsigned)g.n_blocks, lct::kThreads, shared, static_cast<cudaStream_t>(stream)>>>(
      va, va, g, static_cast<const uint16_t*>(other), output, auxiliary, spec);
  return (int)cudaGetLastError();
}

int lct_dual_scale_add(const lct_operand* a, const lct_operand* b, void* output,
                       uint8_t* auxiliary, const float* alpha, int compressed_output,
                       int64_t size, int64_t logical_numel, int block_symbols, int steps,
                       int fixed_words, int rare_length, void* stream) {
  lct::Shape g;
  lct::OperandView va, vb;
  int rc = lct::check_shape(size, logical_numel, block_symbols, steps, fixed_words, rare_length, &g);
  if (rc) return rc;
  if ((rc = lct::view_of(a, &va)) != 0) return rc;
  if ((rc = lct::view_of(b, &vb)) != 0) return rc;
  if (output == nullptr || alpha == nullptr) return LCT_E_NULL_POINTER;
  if (compressed_output && auxiliary == nullptr) return LCT_E_NULL_POINTER;
  if (!lct::aligned16(output) || (compressed_output && !lct::aligned16(auxiliary)))
    return LCT_E_ALIGNMENT;
  // fma(a, alpha, b): the scaled operation with beta == 1.
  const lct::OpSpec spec{alpha, nullptr, LCT_OP_SCALAR_MUL_ADD, 0, 1};
  const size_t shared = lct::reader_shared_bytes(2, fixed_words, 2 * lct::kRingBytes);
  constexpr int kForm = lct::kFormScaled;
  auto kernel = g.lane_mask == 254
                    ? (compressed_output ? lct::pointwise_kernel<true, 254, kForm, true, true>
                                         : lct::pointwise_kernel<true, 254, kForm, false, true>)
                    : (compressed_output ? lct::pointwise_kernel<true, -1, kForm, true, true>
                                         : lct::pointwise_kernel<true, -1, kForm, false, true>);
  if ((rc = lct::opt_in_shared(kernel, shared)) != 0) return rc;
  kernel<<<(unsigned)g.n_blocks, lct::kThreads, shared, static_cast<cudaStream_t>(stream)>>>(
      va, vb, g, nullptr, output, auxiliary, spec);
  return (int)cudaGetLastError();
}

}  // extern "C"
