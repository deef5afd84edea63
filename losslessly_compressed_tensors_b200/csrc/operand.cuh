// Compressed operands as the kernels see them, the arithmetic of the fused operations, and the
// host-side argument checks.
#pragma once

#include "common.cuh"
#include "lct_b200.h"

namespace lct {

struct OperandView {
  const uint32_t* encoded;
  const uint8_t* side;
  const int32_t* center;
  const uint32_t* pair_table;
  const uint8_t* lanes;
  const uint8_t* starts;
  const uint8_t* tail;
  const int32_t* descriptor;
  const int32_t* count;
  const int32_t* blocks;
  int64_t base;
  int mode;
};

constexpr size_t kTableBytes = (size_t)kPairEntries * 4;

struct Shape {
  int64_t size;
  int64_t logical_numel;
  int64_t streams;
  int64_t n_blocks;
  int block_symbols;
  int steps;
  int fixed_words;
  int rare_length;
  int lane_mask;  // 254: lane ^ (row & 254) ("swizzle"); 0: "linear"
};

__device__ __forceinline__ void cp_async_16(void* shared_dst, const void* global_src) {
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(shared_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(global_src) : "memory");
}
__device__ __forceinline__ void cp_async_16_to(uint32_t shared_dst, const void* global_src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(shared_dst), "l"(global_src) : "memory");
}
__device__ __forceinline__ void cp_async_4(void* shared_dst, const void* global_src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(shared_dst)),
               "l"(global_src));
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

__device__ __forceinline__ const uint8_t* tail_origin(const OperandView& a) {
  if (a.mode == 2) return a.tail + a.descriptor[0] + 2 * (int64_t)(*a.count);
  return a.tail + a.base;
}

struct OpSpec {
  const float* alpha;
  const float* beta;
  int op;
  int alpha_is_one;
  int beta_is_one;
};

// The arithmetic forms behind the operations.  fma(l, alpha, r * beta) serves every scaled sum
// but the one whose left operand is not scaled and whose right one is (it rounds once): a factor
// of one changes neither the product nor the sum.
enum OpForm { kFormScaled, kFormLerp, kFormRightScaled, kFormAdd, kFormMultiply, kFormEmaSquare };

__host__ __device__ __forceinline__ int form_of(int op, int alpha_is_one, int beta_is_one) {
  return op == LCT_OP_ADD          ? kFormAdd
         : op == LCT_OP_MULTIPLY   ? kFormMultiply
         : op == LCT_OP_LERP       ? kFormLerp
         : op == LCT_OP_EMA_SQUARE ? kFormEmaSquare
         : alpha_is_one && !beta_is_one ? kFormRightScaled
                                        : kFormScaled;
}

__device__ __forceinline__ float bf16_low(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_high(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

__device__ __forceinline__ uint32_t pack_rn(float low, float high) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(low, high);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// torch.lerp(start, end, weight) in float32, as PyTorch's CUDA kernel evaluates it.
__device__ __forceinline__ float lerp_f32(float start, float end, float weight) {
  const float d = __fsub_rn(end, start);
  return fabsf(weight) < 0.5f ? __fmaf_rn(weight, d, start)
                              : __fmaf_rn(-d, __fsub_rn(1.0f, weight), end);
}
// Two lanes of lerp(start, end, weight), rounded to BF16.
__device__ __forceinline__ uint32_t lerp_pair(uint32_t start, uint32_t end, float weight) {
  return pack_rn(lerp_f32(bf16_low(start), bf16_low(end), weight),
                 lerp_f32(bf16_high(start), bf16_high(end), weight));
}

// Two lanes of `left (op) right`, rounded once to BF16.
template <int kForm>
__device__ __forceinline__ uint32_t apply_form(uint32_t left, uint32_t right, float alpha, float beta) {
  if (kForm == kFormAdd) {
    const __nv_bfloat162 r = __hadd2(*reinterpret_cast<const __nv_bfloat162*>(&left),
                                     *reinterpret_cast<const __nv_bfloat162*>(&right));
    return *reinterpret_cast<const uint32_t*>(&r);
  }
  if (kForm == kFormMultiply) {
    const __nv_bfloat162 r = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&left),
                                     *reinterpret_cast<const __nv_bfloat162*>(&right));
    return *reinterpret_cast<const uint32_t*>(&r);
  }
  if (kForm == kFormLerp) return lerp_pair(left, right, alpha);
  const float l0 = bf16_low(left), l1 = bf16_high(left);
  const float r0 = bf16_low(right), r1 = bf16_high(right);
  if (kForm == kFormRightScaled) return pack_rn(__fmaf_rn(r0, beta, l0), __fmaf_rn(r1, beta, l1));
  if (kForm == kFormEmaSquare) {
    const uint32_t scaled = pack_rn(__fmul_rn(l0, alpha), __fmul_rn(l1, alpha));
    return pack_rn(__fmaf_rn(beta, __fmul_rn(r0, r0), bf16_low(scaled)),
                   __fmaf_rn(beta, __fmul_rn(r1, r1), bf16_high(scaled)));
  }
  return pack_rn(__fmaf_rn(l0, alpha, __fmul_rn(r0, beta)), __fmaf_rn(l1, alpha, __fmul_rn(r1, beta)));
}

// An operation with its scalars.  The form is a constant of the kernel: tested per word, it cuts
// the walk into pieces that no longer overlap (a product with a dense tensor took 15.0 instead of
// 10.3 us for one block, 98.6 instead of 74.9 for 64 Mi elements).
constexpr int kFormAtRunTime = -1;
template <int kForm>
struct Operation {
  int form;
  float alpha, beta;

  __device__ __forceinline__ explicit Operation(const OpSpec& spec)
      : form(form_of(spec.op, spec.alpha_is_one, spec.beta_is_one)),
        alpha(spec.alpha_is_one ? 1.0f : *spec.alpha), beta(spec.beta_is_one ? 1.0f : *spec.beta) {}
  __device__ __forceinline__ uint32_t operator()(uint32_t left, uint32_t right) const {
    const int f = kForm == kFormAtRunTime ? form : kForm;
    if (f == kFormScaled) return apply_form<kFormScaled>(left, right, alpha, beta);
    if (f == kFormLerp) return apply_form<kFormLerp>(left, right, alpha, beta);
    if (f == kFormRightScaled) return apply_form<kFormRightScaled>(left, right, alpha, beta);
    if (f == kFormAdd) return apply_form<kFormAdd>(left, right, alpha, beta);
    if (f == kFormMultiply) return apply_form<kFormMultiply>(left, right, alpha, beta);
    return apply_form<kFormEmaSquare>(left, right, alpha, beta);
  }
};

// ---------------------------------------------------------------------------
// Host-side launch helpers
// ---------------------------------------------------------------------------

static inline int check_shape(int64_t size, int64_t logical_numel, int block_symbols, int steps,
                       int fixed_words, int rare_length, Shape* g) {
  if (steps != 128 && steps != 256) return LCT_E_BAD_GEOMETRY;
  if (block_symbols != steps * kLanes) return LCT_E_BAD_GEOMETRY;
  if (fixed_words < 2 || fixed_words > 64) return LCT_E_BAD_GEOMETRY;
  if (rare_length < 0 || rare_length > 8) return LCT_E_BAD_ARGUMENT;
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
  g->rare_length = rare_length;
  g->lane_mask = lane_mask_now();
  return 0;
}

static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

static inline int view_of(const lct_operand* in, OperandView* v) {
  if (in == nullptr || in->encoded == nullptr || in->side == nullptr || in->center == nullptr ||
      in->pair_table == nullptr)
    return LCT_E_NULL_POINTER;
  if (!aligned16(in->side) || !aligned16(in->pair_table) || !aligned16(in->encoded))
    return LCT_E_ALIGNMENT;
  const lct_overflow& o = in->overflow;
  if (o.mode < 0 || o.mode > 2) return LCT_E_BAD_ARGUMENT;
  if (o.mode != 0 && (o.blocks == nullptr || o.tail == nullptr || o.lanes == nullptr ||
                      o.starts == nullptr))
    return LCT_E_NULL_POINTER;
  if (o.mode == 2 && (o.descriptor == nullptr || o.count == nullptr)) return LCT_E_NULL_POINTER;
  v->encoded = reinterpret_cast<const uint32_t*>(in->encoded);
  v->side = in->side;
  v->center = in->center;
  v->pair_table = in->pair_table;
  v->lanes = o.lanes;
  v->starts = o.starts;
  v->tail = o.tail;
  v->descriptor = o.descriptor;
  v->count = o.count;
  v->blocks = o.blocks;
  v->base = o.base;
  v->mode = o.mode;
  return 0;
}

// Operation code and its scalars: which of alpha / beta the kernels will read.
static inline int check_op(int op, const float* alpha, const float* beta, int* alpha_is_one,
                           int* beta_is_one) {
  if (op < LCT_OP_ADD || op > LCT_OP_EMA_SQUARE) return LCT_E_BAD_ARGUMENT;
  if (op == LCT_OP_SCALAR_MUL_ADD) {
    if (!*alpha_is_one && alpha == nullptr) return LCT_E_NULL_POINTER;
    if (!*beta_is_one && beta == nullptr) return LCT_E_NULL_POINTER;
  } else if (op == LCT_OP_LERP) {
    if (alpha == nullptr) return LCT_E_NULL_POINTER;
    *alpha_is_one = 0;
    *beta_is_one = beta == nullptr;  // beta: weight of the Nesterov direction, when one is emitted
  } else if (op == LCT_OP_EMA_SQUARE) {
    if (alpha == nullptr || beta == nullptr) return LCT_E_NULL_POINTER;
    *alpha_is_one = *beta_is_one = 0;
  } else {
    *alpha_is_one = *beta_is_one = 1;
  }
  return 0;
}

template <typename Kernel>
static inline int opt_in_shared(Kernel kernel, size_t bytes) {
  return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace lct
