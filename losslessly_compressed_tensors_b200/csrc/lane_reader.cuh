// Lane side of the decoder, shared by all kernels that read a compressed operand: the block's
// prologue, the read position of one lane, and the walk of a thread's lane through a block, chunk
// by chunk.  One CTA of 256 threads per block, one lane per thread (lanes.cuh).
#pragma once

#include "lanes.cuh"
#include "operand.cuh"

namespace lct {

// Rows per unrolled chunk of a walk.
constexpr int kWalkPairs = 8;
constexpr int kWalkRows = 2 * kWalkPairs;

// Shared memory of a reading CTA with n operands (n = 2 only for the fused operation on two
// compressed tensors):
//
//   table 0 .. n-1   the 4096-entry two-symbol table of each operand's center, 16 KB each, at
//                    fixed addresses: a lookup is one load at (window & 0x3FFC) + a constant
//   own              `own_bytes` for the caller
//   then per operand:
//   ReaderHead       byte table, overflow map, scan scratch
//   image            the block's payload, LAST word row first
//
// A lane therefore reads its column downwards, and what lies below the image's end is other
// shared memory of this CTA.  Bits past a lane's coded symbols never reach a result, so reading
// them is harmless; a lane's fetch address is pulled back to a row next to the image once per
// kClampPairs pairs and cannot leave the CTA's memory in between, whatever the stream holds.
struct __align__(16) ReaderHead {
  uint16_t overflow_offset[kLanes];  // from the block's first tail byte: below steps * kLanes
  uint16_t overflow_start[kLanes];
  uint8_t index_to_byte[256];
  const uint8_t* tail;               // the block's first tail byte
  int scan[36];
};
constexpr size_t kReaderHeadBytes = 1536;
static_assert(sizeof(ReaderHead) <= kReaderHeadBytes, "head must fit its slot");

constexpr uint32_t kWordRow = kLanes * 4;  // bytes of one word row of the image
// A lane's fetch address is never further below the image than this many rows when it is checked
// ...
constexpr uint32_t kRowsBelow = 3;
// ... and moves at most this much until the next check: a row per refill, at most two refills per
// pair.
constexpr int kClampPairs = 4;
static_assert((kRowsBelow + 2 * kClampPairs) * kWordRow <= kTableBytes + kReaderHeadBytes,
              "what a lane may read past its image is the head and the tables");

struct ReaderShared {
  ReaderHead* head;
  uint32_t* image;
  uint32_t* table;
};
static inline __host__ __device__ size_t reader_shared_bytes(int operands, int fixed_words,
                                                             size_t own_bytes = 0) {
  return operands * (kTableBytes + kReaderHeadBytes + (size_t)fixed_words * kWordRow) + own_bytes;
}
__device__ __forceinline__ ReaderShared carve_reader(unsigned char* base, int index, int operands,
                                                     int fixed_words, size_t own_bytes = 0) {
  unsigned char* rest = base + operands * kTableBytes + own_bytes +
                        index * (kReaderHeadBytes + (size_t)fixed_words * kWordRow);
  ReaderShared s;
  s.table = reinterpret_cast<uint32_t*>(base + index * kTableBytes);
  s.head = reinterpret_cast<ReaderHead*>(rest);
  s.image = reinterpret_cast<uint32_t*>(rest + kReaderHeadBytes);
  return s;
}

// CTA prologue (256 threads): stage the payload and the symbol table of the tensor's center,
// expand this block's overflow map.  The copies are still under way on return: the caller waits
// for them (cp_async_wait_all) and then for the other threads.
__device__ __forceinline__ void stage_operand(const ReaderShared& sh, const OperandView& a,
                                              const Shape& g, int64_t block) {
  const int tid = threadIdx.x;
  ReaderHead& head = *sh.head;
  const int center = *a.center;
  // Word w of the block's 256 streams is one contiguous, 1 KB aligned row.
  const uint32_t* rows = a.encoded + block * kLanes;
  for (int i = tid; i < g.fixed_words * (kLanes / 4); i += kThreads) {
    const int w = i >> 6, c = (i & 63) * 4;
    cp_async_16(&sh.image[(g.fixed_words - 1 - w) * kLanes + c], rows + (int64_t)w * g.streams + c);
  }
  // The overflow map's loads are requested before the table's copies have an address.
  int64_t lane_at = 0, start_at = 0;
  int count = 0, byte_base = 0;
  if (a.mode == 1 || (a.mode == 2 && a.descriptor[2] == 0)) {
    count = a.blocks[block];
    lane_at = start_at = a.blocks[g.n_blocks + block];
    byte_base = a.blocks[2 * g.n_blocks + block];
    if (a.mode == 2) {
      lane_at += a.descriptor[0];
      start_at += (int64_t)a.descriptor[0] + *a.count;
    }
  }
  // The codebook's table for this tensor's center, ready to use (symbols are exponent bytes).
  const uint32_t* source = a.pair_table + (size_t)((center + 128) & 255) * kPairEntries;
#pragma unroll
  for (int i = 0; i < kPairEntries / 4; i += kThreads)
    cp_async_16(&sh.table[4 * (tid + i)], source + 4 * (tid + i));
  head.index_to_byte[tid] = (uint8_t)index_to_exponent_byte((uint32_t)tid, center);
  head.overflow_start[tid] = (uint16_t)g.steps;
  if (count <= 0) return;  // uniform across the CTA
  if (tid == 0) head.tail = tail_origin(a) + byte_base;
  int lane = 0, length = 0;
  if (tid < count) {
    lane = a.lanes[lane_at + tid];
    length = g.steps - a.starts[start_at + tid];
  }
  int unused;
  // (Its barriers also put the defaults above before other threads' entries.)
  const int prefix = block_exclusive_scan(length, head.scan, &unused);
  if (tid < count) {
    head.overflow_start[lane] = (uint16_t)(g.steps - length);
    head.overflow_offset[lane] = (uint16_t)prefix;
  }
}

// Read position of one lane: up to 64 stream bits in two registers, already shifted so that the
// bit under the position is bit 2 of `lo` (bits 0..1 are the two bits before it), and the word
// that comes after them.  A lookup is  entry = table[lo & 0x3FFC]  and consuming n bits is two
// funnel shifts whose amount is the low five bits of a register, i.e. the table entry itself, so
// the dependent chain from one lookup to the next is  mask -> shared load -> shift.
// `valid` counts the loaded bits.  At least 32 at every refill() serve two lookups of full pairs
// (2 + 12 + 12 bits), after which at least 8 are left; the refill is a few predicated
// instructions off the lookup chain, its load is issued a refill ahead.
struct LaneCursor {
  uint32_t lo, hi, word;
  int valid;
  uint32_t next;    // shared address of the word behind `word`
  uint32_t lowest;  // where `next` is pulled back to

  __device__ __forceinline__ void open(const uint32_t* image, int lane, int fixed_words) {
    const uint32_t top = shared_address(image + (fixed_words - 1) * kLanes + lane);
    const uint32_t first = load_shared_u32(top);
    word = load_shared_u32(top - kWordRow);  // fixed_words >= 2
    lo = first << 2;
    hi = first >> 30;
    valid = 34;
    next = top - 2 * kWordRow;
    lowest = shared_address(image + lane) - kRowsBelow * kWordRow;
  }
  __device__ __forceinline__ void clamp() { next = max(next, lowest); }
  // `amount`: only its low five bits count.
  __device__ __forceinline__ void shift_out(uint32_t amount) {
    lo = __funnelshift_r(lo, hi, amount);
    hi = __funnelshift_r(hi, 0u, amount);
  }
  // Consume an entry: a full pair, or its first symbol.
  __device__ __forceinline__ void take(uint32_t entry) {
    shift_out(entry);
    valid = dot_bytes(entry, 0xFF, valid);
  }
  __device__ __forceinline__ void refill() {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b32 t;\n\t"
        "setp.lt.s32 p, %2, 32;\n\t"
        "@p shf.l.wrap.b32 t, 0, %3, %2;\n\t"   // word << valid
        "@p shf.l.wrap.b32 %1, %3, 0, %2;\n\t"  // the bits of word that did not fit
        "@p or.b32 %0, %0, t;\n\t"
        "@p ld.shared.u32 %3, [%4];\n\t"
        "@p add.s32 %2, %2, 32;\n\t"
        "@p sub.u32 %4, %4, 1024;\n\t"
        "}"
        : "+r"(lo), "+r"(hi), "+r"(valid), "+r"(word), "+r"(next));
  }
};
static_assert(kWordRow == 1024, "LaneCursor steps from image row to image row");

// Not volatile: the window comes out of the staged image, so the load cannot move ahead of the
// barrier that publishes image and table, and nothing writes the table afterwards.
__device__ __forceinline__ uint32_t look_up_entry(uint32_t table, uint32_t window) {
  uint32_t entry;
  asm("ld.shared.u32 %0, [%1];" : "=r"(entry) : "r"(table + (window & 0x3FFCu)));
  return entry;
}

// Move the word that was just used up out of a chunk's buffer.
template <int kWords>
__device__ __forceinline__ void next_word(uint32_t (&words)[kWords]) {
#pragma unroll
  for (int i = 0; i + 1 < kWords; ++i) words[i] = words[i + 1];
}

// The lane of one thread.  An entry that leaves this struct has the pair's exponent bytes in bytes
// 1 and 2, whatever else is in it.
struct LaneWalk {
  LaneCursor cursor;
  int coded;  // leading steps of this lane that are in the bit stream
  const ReaderHead* head;
  uint32_t table;       // shared address of the two-symbol table
  uint32_t byte_table;  // shared address of index_to_byte[256]
  int rare_shift;       // where an escape's literal is in the window it was looked up with

  // Behind the barrier that publishes the staged operand.
  __device__ __forceinline__ void open(const ReaderShared& sh, const OperandView& view,
                                       const Shape& g, int64_t block) {
    const int lane = threadIdx.x;
    table = shared_address(sh.table);
    byte_table = shared_address(sh.head->index_to_byte);
    rare_shift = g.rare_length + 2;
    cursor.open(sh.image, lane, g.fixed_words);
    head = sh.head;
    coded = min((int)head->overflow_start[lane],
                valid_steps_of(block, lane, g.steps, g.block_symbols, g.logical_numel, g.lane_mask));
  }
  // All rows of the chunk at step0 are in the streams of all lanes of the warp.
  __device__ __forceinline__ bool whole_chunk(int step0, int rows = kWalkRows) const {
    return __all_sync(0xFFFFFFFFu, step0 + rows <= coded);
  }
  __device__ __forceinline__ uint32_t literal(uint32_t window) const {
    return load_shared_u8(byte_table + ((window >> rare_shift) & 255u));
  }
  // The rest of a pair whose entry is not a full pair; its first symbol's bits have been taken,
  // `before` is the window it was looked up with.
  // `refills`: no refill follows before the next pair.
  __device__ __forceinline__ uint32_t finish_pair(uint32_t entry, uint32_t before, bool refills) {
    const uint32_t literal0 = literal(before);
    cursor.refill();
    const uint32_t second = look_up_entry(table, cursor.lo);
    const uint32_t literal1 = literal(cursor.lo);
    const uint32_t length = entry_first_length(second);
    cursor.shift_out(length);
    cursor.valid -= (int)length;
    if (refills) cursor.refill();
    if (entry & kEscape) entry = prmt(entry, literal0, 0x3240);
    return (second & kEscape) ? prmt(entry, literal1, 0x3410) : prmt(entry, second, 0x3510);
  }
  // Pair k of a whole chunk (k: a constant, in an unrolled loop).  `meanwhile` is issued between
  // the lookup and its first use.
  template <typename Meanwhile>
  __device__ __forceinline__ uint32_t read_pair(int k, Meanwhile meanwhile) {
    if (k % kClampPairs == 0) cursor.clamp();
    const uint32_t before = cursor.lo;
    uint32_t entry = look_up_entry(table, before);
    meanwhile();
    cursor.take(entry);
    // Rare: an escape, or two codes of more than 12 bits.
    if ((int32_t)entry < 0) entry = finish_pair(entry, before, (k & 1) == 0);
    if (k & 1) cursor.refill();  // two full pairs take at most 24 bits: one refill serves both
    return entry;
  }
  // Raw tail symbols of this lane in the rows from step0 on, four to a word, as exponent bytes
  // (rows before the tail: undefined).  The tail is a run of bytes of any alignment: it is read in
  // aligned words, each of which holds a byte of it, all of them requested together.
  template <int kWords>
  __device__ __forceinline__ void read_tail(uint32_t (&symbols)[kWords], int step0, int from) const {
    const int index = step0 - from;  // of the first row, in the tail
    uint32_t words[kWords + 1] = {};
    int misaligned = 0;
    if (index + 4 * kWords > 0) {
      const uint8_t* first = head->tail + (head->overflow_offset[threadIdx.x] + index);
      misaligned = (int)(reinterpret_cast<uintptr_t>(first) & 3u);
      const uint32_t* aligned = reinterpret_cast<const uint32_t*>(first - misaligned);
#pragma unroll
      for (int i = 0; i <= kWords; ++i)
        if (index + 4 * i + 3 >= misaligned && 4 * i < 4 * kWords + misaligned) words[i] = aligned[i];
    }
#pragma unroll
    for (int i = 0; i < kWords; ++i) {
      const uint32_t raw = __funnelshift_r(words[i], words[i + 1], 8 * misaligned);
      symbols[i] = ((raw & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) ^ (raw & 0x80808080u);  // + 127, bytewise
    }
  }
  // The pair at `step`, wherever its symbols are; `from`: where the lane's tail starts, `raw`: the
  // entry the pair has if it is in the tail.
  __device__ __forceinline__ uint32_t read_any(int step, int from, uint32_t raw) {
    if (step >= coded) return step < from ? 0u : raw;
    const uint32_t before = cursor.lo;
    uint32_t entry = look_up_entry(table, before);
    if (step + 2 <= coded) {
      cursor.take(entry);
      if ((int32_t)entry < 0) entry = finish_pair(entry, before, false);
    } else {  // the lane's last coded step is the first row of this pair
      entry = ((entry & kEscape) ? literal(before) : entry_first_symbol(entry)) << 8;
    }
    cursor.refill();
    return entry;
  }
  // The pairs of a chunk in which some lane's stream ends, or has ended.  `emit(k, entry)` gets
  // them one after the other.  Where the tail starts is read again each time: it would hold a
  // register throughout.  The tail's words are requested ahead of the loop; requested byte by byte
  // inside it, each pair waits for global memory.  Two pairs per turn: unrolled over the chunk it
  // saves 2 to 7 % here, and costs chunks of whole lanes as much or more (registers; decode.cu and
  // update.cu, all codebooks).  Against the former pair-by-pair loop, 32 Mi elements that overflow
  // in every lane: decoded in 176 -> 63 us (half-zero codebook), 99 -> 48 (normal codebook).
  template <int kPairs = kWalkPairs, typename Emit>
  __device__ __forceinline__ void read_chunk(int step0, Emit emit) {
    constexpr int kWords = kPairs / 2;
    const int from = head->overflow_start[threadIdx.x];
    uint32_t symbols[kWords];
    read_tail(symbols, step0, from);
#pragma unroll 1
    for (int k = 0; k < kPairs; k += 2) {
      cursor.clamp();
      emit(k, read_any(step0 + 2 * k, from, symbols[0] << 8));
      emit(k + 1, read_any(step0 + 2 * k + 2, from, symbols[0] >> 8));
      next_word(symbols);
    }
  }
};

// Both columns' exponents of this thread's row of a pair, in place for join_word(): the even
// thread of two gets the first row, the odd one the second.
struct RowExchange {
  // Of (own entry, neighbour's entry): byte 1 (first row) or 2 of both, the even lane's to byte 1
  // and the odd lane's to byte 3.
  uint32_t selector;
  __device__ __forceinline__ void open() { selector = (threadIdx.x & 1) ? 0x2060u : 0x5010u; }
  static __device__ __forceinline__ uint32_t neighbours(uint32_t own) {
    return __shfl_xor_sync(0xFFFFFFFFu, own, 1);
  }
  __device__ __forceinline__ uint32_t exponents(uint32_t entry, uint32_t neighbour) const {
    return prmt(entry, neighbour, selector) >> 1;
  }
};

constexpr int kMaxLeft = 1 << 20;  // more than a block has
// Elements from the block's first on, 0 to kMaxLeft.  Bounded on both sides: storage may hold any
// number of blocks of pure padding, and how far a block lies behind the end need not fit 32 bits.
__device__ __forceinline__ int elements_left(const Shape& g, int64_t block) {
  const int64_t left = g.logical_numel - block * (int64_t)g.block_symbols;
  return (int)max((int64_t)0, min((int64_t)kMaxLeft, left));
}

// Where a thread's words of a dense tensor are: rows of the block from `rows` on, a word of two
// neighbouring columns per row.  Offsets are in elements.
template <typename Element>
struct DenseWords {
  Element* rows;
  int left;  // elements_left()

  // The first `count` rows of the block are full.
  __device__ __forceinline__ bool holds_rows(int count) const { return count * kLanes <= left; }
  __device__ __forceinline__ void store(uint32_t at, uint32_t word) const {
    __stcs(reinterpret_cast<uint32_t*>(rows + at), word);
  }
  __device__ __forceinline__ void store_guarded(uint32_t at, uint32_t word) const {
    if ((int)at < left) rows[at] = (uint16_t)word;
    if ((int)at + 1 < left) rows[at + 1] = (uint16_t)(word >> 16);
  }
  __device__ __forceinline__ uint32_t load(uint32_t at) const { return load_ahead_u32(rows + at); }
  __device__ __forceinline__ uint32_t load_value(uint32_t at) const { return load_ahead_u16(rows + at); }
  __device__ __forceinline__ uint32_t load_guarded(uint32_t at) const {
    const uint32_t low = (int)at < left ? rows[at] : 0u;
    const uint32_t high = (int)at + 1 < left ? rows[at + 1] : 0u;
    return low | (high << 16);
  }
};

// Rows of a block that hold elements, in whole chunks.
__device__ __forceinline__ int rows_in_use(const Shape& g, int64_t block) {
  const int in_block = min(g.block_symbols, elements_left(g, block));
  return (in_block + kWalkRows * kLanes - 1) / (kWalkRows * kLanes) * kWalkRows;
}

// Side bytes of the chunks in work and ahead, in shared memory.  A warp's 32 lanes have 32 bytes in
// every row, so a chunk of 16 rows is one 16-byte asynchronous copy per thread into the warp's own
// part of the ring (nothing but a warp barrier orders copies and reads), two chunks ahead of its
// use.  Requested into registers instead, one load per thread and pair, they cost the decoder 33
// of 90 us (64 Mi elements): the walk leaves too few registers to hold them two chunks ahead.
constexpr int kRingStages = 3;
constexpr uint32_t kRingStage = kWalkRows * 32;  // bytes per warp
constexpr size_t kRingBytes = (size_t)kWarps * kRingStages * kRingStage;
static_assert(kRingStage == 32 * 16, "one 16-byte copy per thread");

struct SideRing {
  const uint8_t* from;  // what this thread copies of the next chunk to be requested
  uint32_t to, at;      // where it goes; this thread's bytes of the chunk in work
  uint32_t begin;       // the warp's part of the ring
  int rows_left;

  __device__ __forceinline__ void open(unsigned char* ring, const uint8_t* block_side, int rows_used) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    begin = shared_address(ring) + warp * kRingStages * kRingStage;
    from = block_side + (lane >> 1) * kLanes + warp * 32 + (lane & 1) * 16;
    to = begin + lane * 16;
    at = begin + (lane & 1) * 32 + (lane & 30);
    rows_left = rows_used;
    request();
    request();
  }
  __device__ __forceinline__ void request() {
    if (rows_left > 0) cp_async_16_to(to, from);
    asm volatile("cp.async.commit_group;" ::: "memory");
    rows_left -= kWalkRows;
    from += kWalkRows * kLanes;
    to += kRingStage;
    if (to >= begin + kRingStages * kRingStage) to -= kRingStages * kRingStage;
  }
  // The chunk at `at` is there; a further one is requested into the stage read before it.
  __device__ __forceinline__ void wait() {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    request();
  }
  // ... of two rings whose requests alternate.
  __device__ __forceinline__ void wait_both(SideRing& other) {
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    __syncwarp();
    request();
    other.request();
  }
  __device__ __forceinline__ uint32_t pair(int k) const { return load_shared_u16(at + k * 64); }
  __device__ __forceinline__ void advance() {
    at += kRingStage;
    if (at >= begin + kRingStages * kRingStage) at -= kRingStages * kRingStage;
  }
};

// This thread's two bytes, of its row, in a row pair's 512 side bytes.
__device__ __forceinline__ int own_bytes() {
  return (threadIdx.x & 1u) * kLanes + (threadIdx.x & 254u);
}

}  // namespace lct
