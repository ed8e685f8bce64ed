// Internal interface of the tensor-core decode path (moe_fast.cu), used by moe_layer.cu.
//
// The idea.  A 16-bit E8P codeword decodes to eight weights w = s*h/2 + p/4, with h an odd
// integer from the abs table (|h| in {1,3,5}), s the sign bit and p = +-1 by the parity of the
// sign byte.  Then 4w = 2q + 1 for the integer q = h ^ (neg ? 0xFE : 0) ^ parity, which is pure
// bit arithmetic on a byte.  So a row's dot product with integer activations x' is
//     4 * sum_k w_k x'_k = 2 * sum_k q_k x'_k + sum_k x'_k,
// an exact int8 tensor-core product plus one per-token constant.  Activations are quantised per
// row to 16-bit fixed point (power-of-two scale) and fed as two signed bytes (x' = 256 hi + lo).
// The only rounding in a projection is that fixed-point step.  The kernels hand the tensor cores
// u = q + 8 (a 4-bit unsigned value, two table words XORed) and take 8 * sum(x') off afterwards.
#pragma once

#include "common.cuh"

namespace keepvq {
namespace fast {

constexpr int MAX_GROUP_ROUTES = 8;     // routes of one expert that share an mma.sync tile (its 8 columns)
constexpr int FEW_TOKENS_ROUTES = 84;   // most routes of a layer call in one launch (few_tokens_pay)
constexpr int SMALL_CALL_ROUTES = 48;   // calls with fewer routes never run the plain slab kernel
constexpr int FEW_ROUTE_GROUPS = 96;    // below this many route groups a CTA's warps share rows AND inputs (sweep kernel, split slab kernel)
constexpr int PAIRED_GROUP_ROUTES = 4;  // ... when a route's two byte planes take a column each (one MMA per step)
constexpr int64_t MAX_GROUP_INPUTS = 65536;  // inputs of a scale group: sum(x') with |x'| <= 32639 fits the 32 bits it is kept in
static_assert(32639 * MAX_GROUP_INPUTS < (int64_t{1} << 31), "");
constexpr int PREFILL_GROUP_ROUTES = 96;   // routes of one expert per tcgen05 item (its accumulators and two operand stages fill tensor memory)
constexpr int PREFILL_GROUP_ROUTES_SMALL = 48;  // ... for calls with fewer routes per expert, and for rows with several scale groups
constexpr int PREFILL_FEW_ROUTES_MEAN = 32;     // routes per expert on average up to which a call counts as the former


// ------------------------------------------------------------------------------------------
// The codeword decoder shared by the decode kernels (projection_slab.cu, projection_sweep.cu) and
// the tcgen05 kernel (prefill_umma.cu), and the entries its tables are built from.
// Entry bytes: byte j of the low word is table nibble 3 - j, of the high word nibble 7 - j.
// ------------------------------------------------------------------------------------------
// The eight bytes q (4w = 2q + 1 for positive signs) of abs row `word` under one parity.
__device__ __forceinline__ uint2 abs_table_entry(uint32_t word, uint32_t par) {
  uint32_t lo = 0, hi = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int nl = 3 - j, nh = 7 - j;
    uint32_t hl = ((word >> (4 * nl)) & 0xFu) - 8u, hh = ((word >> (4 * nh)) & 0xFu) - 8u;
    if (par) { hl = nl == 0 ? ~hl : hl ^ 1u; hh ^= 1u; }
    lo |= (hl & 0xFFu) << (8 * j);
    hi |= (hh & 0xFFu) << (8 * j);
  }
  return make_uint2(lo, hi);
}
// The XOR masks of sign byte `sb`: 0xFE where the sign bit is set; ^1 everywhere (^0xFF on nibble 0) on odd parity.
__device__ __forceinline__ uint2 sign_table_entry(uint32_t sb) {
  const uint32_t par = __popc(sb) & 1u;
  uint32_t lo = 0, hi = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int nl = 3 - j, nh = 7 - j;
    uint32_t ml = ((sb >> nl) & 1u) ? 0xFEu : 0u, mh = ((sb >> nh) & 1u) ? 0xFEu : 0u;
    if (par) { ml ^= nl == 0 ? 0xFFu : 0x01u; mh ^= 0x01u; }
    lo |= ml << (8 * j);
    hi |= mh << (8 * j);
  }
  return make_uint2(lo, hi);
}

__device__ __forceinline__ uint2 table_entry(uint32_t addr) {  // tables never change after the set-up barrier: free to schedule
  uint2 v;
  asm("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}

// The nibble decoder.  Both tables hold an entry as eight 4-bit values in ONE word, u = q + 8 for the
// abs table (even parity) and the XOR masks of the sign byte for the other (4-bit XOR on q + 8 is
// the same as on q), 32 replicas each, interleaved in one 64 KB region on a 64 KB boundary:
//   abs entry  at region + abs byte * 256 + lane * 4,   sign entry at region + 128 + sign byte * 256 + lane * 4,
// so each address is one byte permute and each read one shared-memory wavefront (an 8-byte entry
// costs two).  The operand bytes are u (0..15, an UNSIGNED A operand); the caller
// takes 8 * sum(x') off the integer dot product to get back to sum(q x').
template <bool ODD>
__device__ __forceinline__ void decode_codeword_nibble(uint32_t word, uint32_t abs_lane, uint32_t sign_lane, uint32_t& lo, uint32_t& hi) {
  uint32_t e, m;
  asm("ld.shared.u32 %0, [%1];" : "=r"(e) : "r"(__byte_perm(word, abs_lane, ODD ? 0x7634 : 0x7614)));
  asm("ld.shared.u32 %0, [%1];" : "=r"(m) : "r"(__byte_perm(word, sign_lane, ODD ? 0x7624 : 0x7604)));
  // (e ^ m) & mask as ONE three-input logic operation each (written out: the compiler otherwise
  // turns the second into a shift and two operations), and one shift
  uint32_t top;
  asm("lop3.b32 %0, %1, %2, 0x0F0F0F0F, 0x28;" : "=r"(lo) : "r"(e), "r"(m));
  asm("lop3.b32 %0, %1, %2, 0xF0F0F0F0, 0x28;" : "=r"(top) : "r"(e), "r"(m));
  hi = top >> 4;
}
// The same without the shift: `odd` are the odd dims' bytes times 16, for kernels that give the odd dims
// MMAs and accumulators of their own (whose sums are then 16 times too large, exactly).
template <bool ODD>
__device__ __forceinline__ void decode_codeword_halves(uint32_t word, uint32_t abs_lane, uint32_t sign_lane, uint32_t& even, uint32_t& odd) {
  uint32_t e, m;
  asm("ld.shared.u32 %0, [%1];" : "=r"(e) : "r"(__byte_perm(word, abs_lane, ODD ? 0x7634 : 0x7614)));
  asm("ld.shared.u32 %0, [%1];" : "=r"(m) : "r"(__byte_perm(word, sign_lane, ODD ? 0x7624 : 0x7604)));
  asm("lop3.b32 %0, %1, %2, 0x0F0F0F0F, 0x28;" : "=r"(even) : "r"(e), "r"(m));
  asm("lop3.b32 %0, %1, %2, 0xF0F0F0F0, 0x28;" : "=r"(odd) : "r"(e), "r"(m));
}
__device__ __forceinline__ uint32_t pack_nibbles(uint2 v) { return (v.x & 0x0F0F0F0Fu) | ((v.y & 0x0F0F0F0Fu) << 4); }
// All `threads` threads of the CTA (whole warps) fill the 64 KB region at `region` (shared address on
// a 64 KB boundary): a thread works out one entry (one load of the codebook, all in flight together),
// then its warp writes its 32 entries one after the other, the 32 replicas of an entry side by side.
__device__ __forceinline__ void build_nibble_tables(uint32_t region, const uint32_t* __restrict__ codebook, int tid, int threads) {
  const int lane = tid & 31;
  for (int base = 0; base < 512; base += threads) {
    const int e = base + tid;
    uint32_t v = 0;
    if (e < 256) v = pack_nibbles(abs_table_entry(codebook[e], 0)) ^ 0x88888888u;
    else if (e < 512) v = pack_nibbles(sign_table_entry(e - 256));
    const int first = e - lane;  // the warp's first entry
#pragma unroll 8
    for (int i = 0; i < 32; ++i) {
      const uint32_t vi = __shfl_sync(0xFFFFFFFFu, v, i);
      const int ee = first + i;
      if (ee < 512) asm volatile("st.shared.u32 [%0], %1;" ::"r"(region + (ee & 255) * 256 + (ee >> 8) * 128 + lane * 4), "r"(vi) : "memory");
    }
  }
}
// 8-bit codes: a table word holds dim d in nibble d, and byte j of the operand's low word is dim
// 6 - 2j, of the high word dim 7 - 2j, so an entry is the word with its bytes reversed; 32 replicas at
// region + code * 256 + lane * 4.  The operand bytes are the nibbles themselves, u = q + 8.
__device__ __forceinline__ void build_byte_code_table(uint32_t region, const uint32_t* __restrict__ table, int tid, int threads) {
  const int lane = tid & 31;
  for (int first = tid - lane; first < 256; first += threads) {
    const uint32_t v = __byte_perm(table[first + lane], 0, 0x0123);
#pragma unroll 8
    for (int i = 0; i < 32; ++i) {
      const uint32_t vi = __shfl_sync(0xFFFFFFFFu, v, i);
      asm volatile("st.shared.u32 [%0], %1;" ::"r"(region + (first + i) * 256 + lane * 4), "r"(vi) : "memory");
    }
  }
}
__device__ __forceinline__ void decode_byte_code(uint32_t word, int byte, uint32_t table_lane, uint32_t& lo, uint32_t& hi) {
  uint32_t e;
  asm("ld.shared.u32 %0, [%1];" : "=r"(e) : "r"(__byte_perm(word, table_lane, 0x7604 | (byte << 4))));
  lo = e & 0x0F0F0F0Fu;
  hi = (e >> 4) & 0x0F0F0F0Fu;
}
// ------------------------------------------------------------------------------------------
// Activations -> 16-bit fixed point: the scale of a row from its largest magnitude (the bits of a
// float; not finite: 1), and eight values as the bytes of a codeword's operand words.
// ------------------------------------------------------------------------------------------
// Returns the scale, a power of two; `inv` = 1 / scale, exact (infinite for rows of the smallest subnormals).
static __device__ __noinline__ float quant_scale_small(uint32_t top_bits) {  // rows of zeros, of very small values, or without a finite maximum
  const float m = __uint_as_float(top_bits);
  float s = 1.0f;
  if (m > 0.0f && isfinite(m)) {
    s = ldexpf(1.0f, ilogbf(m) - 14);
    if (m / s > 32639.0f) s *= 2.0f;
  }
  return s;
}
__device__ __forceinline__ float quant_scale(uint32_t top_bits, float& inv) {
  if (top_bits >= (16u << 23) && top_bits < 0x7F800000u) {
    // |x| / s < 2^15 with s a power of two: the exponent of the maximum, less 14
    uint32_t bits = (top_bits & 0x7F800000u) - (14u << 23);
    if (__uint_as_float(top_bits) * __uint_as_float((254u << 23) - bits) > 32639.0f) bits += 1u << 23;  // 127 * 256 + 127: the largest value two signed bytes hold
    inv = __uint_as_float((254u << 23) - bits);
    return __uint_as_float(bits);
  }
  const float s = quant_scale_small(top_bits);
  inv = 1.0f / s;
  return s;
}
struct QuantWords { uint32_t hi0, hi1, lo0, lo1; int total; };
// `inv` = 1 / scale, exact.  plain: the values are finite and |v * inv| <= 32639.
__device__ __forceinline__ QuantWords quantize8(const float (&v)[8], float inv, bool plain) {
  QuantWords w;
  uint32_t t[8];  // the low 16 bits: x' in two's complement
  w.total = 0;
  if (plain) {    // 2^23 + 2^22 added to v * inv rounds it to nearest even, as a conversion would
#pragma unroll
    for (int d = 0; d < 8; ++d) {
      t[d] = __float_as_uint(fmaf(v[d], inv, 12582912.0f));
      w.total += static_cast<int>(t[d]);
    }
    w.total -= static_cast<int>(8u * 0x4B400000u);
  } else {
#pragma unroll
    for (int d = 0; d < 8; ++d) {
      const int q = max(-32639, min(32639, __float2int_rn(v[d] * inv)));
      t[d] = static_cast<uint32_t>(q);
      w.total += q;
    }
  }
  // x' = 256 * hi + lo with both bytes signed: lo is the low byte, hi the second byte of x' + 128.
  // byte j of word 0 pairs with table nibble 3-j = dim 6-2j; of word 1 with nibble 7-j = dim 7-2j
  w.lo0 = __byte_perm(__byte_perm(t[6], t[4], 0x0040), __byte_perm(t[2], t[0], 0x0040), 0x5410);
  w.lo1 = __byte_perm(__byte_perm(t[7], t[5], 0x0040), __byte_perm(t[3], t[1], 0x0040), 0x5410);
#pragma unroll
  for (int d = 0; d < 8; ++d) t[d] += 128u;
  w.hi0 = __byte_perm(__byte_perm(t[6], t[4], 0x0051), __byte_perm(t[2], t[0], 0x0051), 0x5410);
  w.hi1 = __byte_perm(__byte_perm(t[7], t[5], 0x0051), __byte_perm(t[3], t[1], 0x0051), 0x5410);
  return w;
}

// Quantised activation rows: the B operand of the projections.
struct QuantRows {
  uint8_t* q;       // [rows + 1, in_dim/8, 16] (last row all zero): per codeword 4 words: hi(dims 6,4,2,0) hi(7,5,3,1) lo(...) lo(...)
  float* scale;     // [rows + 1] power of two: x ~= scale * x'
  int32_t* sums;    // [rows + 1, groups] sum of x' over each scale group
  int32_t* chunk_sums;  // [rows + 1, in_dim / 256] sum of x' over every 256 inputs, or null: for kernels whose warps split a scale group
};

// Routes grouped by the slot they are served from.
struct RouteGroups {
  int32_t* count;        // [2] number of groups, number of routes in them (the live ones)
  int32_t* slot;         // [max_groups]
  int32_t* start;        // [max_groups] first entry in `routes`
  int32_t* size;         // [max_groups] 1..max_group
  int32_t* routes;       // [routes] route ids ordered by group
  int32_t* position = nullptr;  // [routes], may be null: where a route stands in `routes`, -1 for one without a slot
};

// ------------------------------------------------------------------------------------------
// Route grouping: routes that are served from the same slot share the code stream.  One block;
// counting sort by slot, then each slot's routes are cut into groups of at most max_group.
// ------------------------------------------------------------------------------------------
// One block of THREADS threads (a multiple of 32, at most 1024); `sm`: 3 * slots ints of shared memory.
template <int THREADS>
__device__ __forceinline__ void group_routes_block(const uint32_t* __restrict__ served_slot, int routes, int slots, int max_group, const RouteGroups& out, int32_t* clear, int32_t* sm) {
  constexpr int GR_THREADS = THREADS;
  if (clear && threadIdx.x == 0) *clear = 0;
  int32_t* count = sm;               // [slots] routes per slot, then running cursor
  int32_t* first = sm + slots;       // [slots] first position of the slot in `routes`
  int32_t* gfirst = sm + 2 * slots;  // [slots] first group index of the slot
  __shared__ int32_t warp_a[32], warp_b[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int s = tid; s < slots; s += GR_THREADS) count[s] = 0;
  __syncthreads();
  for (int r = tid; r < routes; r += GR_THREADS) {
    const uint32_t s = served_slot[r];
    if (s < static_cast<uint32_t>(slots)) atomicAdd(&count[s], 1);
  }
  __syncthreads();
  // exclusive scans of (routes, groups) per slot: each thread owns a contiguous run of slots
  const int per = (slots + GR_THREADS - 1) / GR_THREADS;
  const int lo = min(tid * per, slots), hi = min(lo + per, slots);
  int a = 0, b = 0;
  for (int s = lo; s < hi; ++s) { a += count[s]; b += (count[s] + max_group - 1) / max_group; }
  int ia = a, ib = b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int ta = __shfl_up_sync(0xFFFFFFFFu, ia, o), tb = __shfl_up_sync(0xFFFFFFFFu, ib, o);
    if (lane >= o) { ia += ta; ib += tb; }
  }
  if (lane == 31) { warp_a[warp] = ia; warp_b[warp] = ib; }
  __syncthreads();
  if (warp == 0) {
    int wa = lane < THREADS / 32 ? warp_a[lane] : 0, wb = lane < THREADS / 32 ? warp_b[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int ta = __shfl_up_sync(0xFFFFFFFFu, wa, o), tb = __shfl_up_sync(0xFFFFFFFFu, wb, o);
      if (lane >= o) { wa += ta; wb += tb; }
    }
    warp_a[lane] = wa; warp_b[lane] = wb;
  }
  __syncthreads();
  int base_a = ia - a + (warp ? warp_a[warp - 1] : 0), base_b = ib - b + (warp ? warp_b[warp - 1] : 0);
  for (int s = lo; s < hi; ++s) {
    first[s] = base_a; gfirst[s] = base_b;
    const int c = count[s], g = (c + max_group - 1) / max_group;
    for (int i = 0; i < g; ++i) {
      out.slot[base_b + i] = s;
      out.start[base_b + i] = base_a + i * max_group;
      out.size[base_b + i] = min(max_group, c - i * max_group);
    }
    base_a += c; base_b += g;
  }
  if (tid == GR_THREADS - 1) { out.count[0] = warp_b[31]; out.count[1] = warp_a[31]; }  // groups, grouped (live) routes
  __syncthreads();
  for (int s = tid; s < slots; s += GR_THREADS) count[s] = 0;  // reuse as cursors
  __syncthreads();
  for (int r = tid; r < routes; r += GR_THREADS) {
    const uint32_t s = served_slot[r];
    const int at = s < static_cast<uint32_t>(slots) ? first[s] + atomicAdd(&count[s], 1) : -1;
    if (at >= 0) out.routes[at] = r;
    if (out.position) out.position[r] = at;
  }
}

struct Projection {
  const uint16_t* codes;  // [slots, out_dim, in_dim/8]
  const void* scales;     // [slots, out_dim, groups]
  const uint8_t* res_codes;  // [hot rows, out_dim, in_dim/8] 8-bit residual codes, or nullptr
  const void* res_scales;    // [hot rows, out_dim, res_groups]
};

struct FastProjectionArgs {
  Projection a;           // gate (or down)
  Projection b;           // up, or {nullptr, nullptr} for a single projection
  int32_t scales_dtype;
  int64_t slots;          // rows of `codes` are slots * out_dim
  int64_t out_dim, in_dim, groups;
  const uint32_t* codebook;
  QuantRows x;            // activations
  int64_t x_zero_row;     // index of the all-zero row quantize_rows appends
  int32_t x_div;          // activation row of route r is r / x_div
  RouteGroups groups_of_routes;
  const float* route_weight;  // [routes] gate weight (gate/up only)
  float swiglu_limit;
  void* out;              // [routes, out_dim]
  int32_t out_dtype;
  int64_t max_routes;
  int32_t* status;        // device word a kernel sets when it gives up (bounded wait expired: 1; unexpected shared window: 2), or null
  int32_t group_cols;     // most routes a group holds: PAIRED_GROUP_ROUTES or MAX_GROUP_ROUTES (what group_routes was given)
  int32_t few_groups;     // what few_route_groups said of the call: 0 many route groups, 1 few, 2 a small call
  // nested residual tier (all null / 0 when the layer has none): slot s adds the 8-bit residual of
  // row hot_of_slot[s] unless that is 0xFFFFFFFF.  res_table is [256][4] fp16 pairs (dims 2k, 2k+1).
  int64_t res_groups;
  const uint32_t* hot_of_slot;
  const uint32_t* res_table;
};

// True when the shapes fit the tensor-core path (in_dim % 256 == 0, group size % 256 == 0, at most
// MAX_GROUP_INPUTS inputs in a scale group, ...).
bool shapes_supported(int64_t out_dim, int64_t in_dim, int64_t groups);
// True when gate_up / down can also add a nested residual with these scale groups to `routes` routes.
bool residual_supported(int64_t routes, int64_t in_dim, int64_t res_groups);

// Output rows of routes that name no expert: the projection kernels never touch them, so a caller
// that promises zeros there has the quantisation kernels write them.  slot == nullptr: no such promise.
struct DeadRows { const uint32_t* slot = nullptr; int32_t per_row = 1; int64_t slots = 0; void* out = nullptr; int64_t row_bytes = 0; };
// planes = false: 16 bytes per codeword (hi 8, lo 8), what the mma.sync kernels read;
// planes = true: all high bytes [rows + 1, in_dim] then all low bytes (quantize_rows_sorted writes that form).
// live_slot (may be null): [rows, per_row] slots of the routes that read the rows; rows whose routes are all dead (slot >= slots) are skipped.
int quantize_rows(const void* x, int32_t x_dtype, int64_t rows, int64_t in_dim, int64_t groups, const QuantRows& out, bool planes, cudaStream_t s,
                  const uint32_t* live_slot = nullptr, int32_t per_row = 1, int64_t slots = 0);
// What the tcgen05 kernels' TMA boxes copy: byte planes (all high bytes [rows + 1, in_dim], then all
// low bytes) with a row per route IN GROUPED ORDER: input row r is quantised once and written to the
// rows position[r * x_div ...] of its x_div routes (group_routes must have run); rows of routes
// without a slot are left alone; scale and sums are per output row.  rows = x_rows * x_div.
int quantize_rows_sorted(const void* x, int32_t x_dtype, int64_t x_rows, int64_t in_dim, int64_t groups, const QuantRows& out, const int32_t* position, int32_t x_div, cudaStream_t s,
                         const DeadRows& dead = {});
// `clear` (may be null): a status word the kernel zeroes for the projection kernels that follow it.
// The router's logits and quantize_rows (planes = false) of the same token rows in one launch, for
// calls of at most FRONT_MAX_TOKENS tokens with fp16 / bf16 activations.
constexpr int64_t FRONT_MAX_TOKENS = 23;  // from 24 tokens on the logits have a faster kernel of their own (router.cu)
bool logits_and_quantize_supported(const keepvq_router_logits_args& logits, int64_t groups);
int logits_and_quantize(const keepvq_router_logits_args& logits, int64_t groups, const QuantRows& out, cudaStream_t s);
// quantize_rows with one more block that groups the routes (group_routes): calls of at most 4096 routes.
bool group_with_quantize_supported(int64_t routes, int64_t slots);
int quantize_rows_and_group(const void* x, int32_t x_dtype, int64_t rows, int64_t in_dim, int64_t groups, const QuantRows& out, bool planes, cudaStream_t s,
                            const uint32_t* live_slot, int32_t per_row, int64_t slots,
                            const uint32_t* served_slot, int64_t routes, int max_group, const RouteGroups& route_groups, int32_t* clear, const DeadRows& dead = {});
// early = false: an ordinary launch, behind everything the stream's kernels before it wrote.
int group_routes(const uint32_t* served_slot, int64_t routes, int64_t slots, int max_group, const RouteGroups& out, int32_t* clear, cudaStream_t s, bool early = true);
// Routes per group for a decode call: four while experts rarely get more (the kernels then run one
// MMA per step for both byte planes), eight beyond.  `live` = routes expected to carry a slot.
int decode_group_routes(int64_t live, int64_t slots, int64_t widest_in_dim);
// Whether a decode call with `live` routes over `slots` experts forms few route groups: 0 no, 1 yes, 2 a small call.
inline int few_route_groups(int64_t live, int64_t slots) { return live < SMALL_CALL_ROUTES ? 2 : (live < slots ? live : slots) < FEW_ROUTE_GROUPS ? 1 : 0; }
int gate_up(const FastProjectionArgs& args, cudaStream_t s);   // h = round(silu(G) * U * weight)
int down(const FastProjectionArgs& args, cudaStream_t s);      // out = round(W2 h)

// The persistent slab kernels behind gate_up / down for calls with many route groups (projection_slab.cu).
int slab_max_in_dim(int cols);
int slab_gate_up(const FastProjectionArgs& args, int cols, cudaStream_t s);
int slab_down(const FastProjectionArgs& args, int cols, cudaStream_t s);
// ... and their split form for calls with few route groups (groups of at most four routes).
int slab_split_max_in_dim();
int slab_split_gate_up(const FastProjectionArgs& args, cudaStream_t s);
int slab_split_down(const FastProjectionArgs& args, cudaStream_t s);
// The sweep kernels for calls with few route groups and no residual tier (projection_sweep.cu):
// inputs of any width in multiples of 256.
bool sweep_supported(int64_t in_dim);
int sweep_gate_up(const FastProjectionArgs& args, cudaStream_t s);
int sweep_down(const FastProjectionArgs& args, cudaStream_t s);

// The few-token kernel (few_tokens.cu): a whole layer call, or part of one, in one launch, for calls of
// few routes; also a single routed projection (FT_DOWN alone).
constexpr int FT_MAX_ROUTES = 144;  // at most one per CTA
constexpr int FT_MAX_TOKENS = 23;   // from 24 tokens on the logits have a faster kernel of their own (router.cu)
constexpr int FT_MAX_CTAS = 160;
enum : uint32_t { FT_ROUTER = 1, FT_GATE_UP = 2, FT_DOWN = 4, FT_COMBINE = 8 };
struct FewTokensPhase {
  const uint16_t* codes[2];   // gate and up, or the one matrix and null
  const void* scales[2];
  const void* x;              // activation rows; route r reads row r / x_div
  void* out;                  // [routes, out_dim]
  int32_t out_dim, in_dim, groups, x_div, out_dtype;
  int32_t n_chunks, chunks_per_group, units_per_group;  // the rest is filled in by the launch
  uint64_t by_chunks, by_group_chunks, by_units;        // their divisors for ft_div
};
struct FewTokensArgs {
  uint32_t parts;             // FT_ROUTER only with FT_GATE_UP; FT_COMBINE only with FT_GATE_UP and FT_DOWN
  int32_t routes, tokens, top_k, scales_dtype;
  int64_t slots;
  const uint32_t* codebook;
  FewTokensPhase phase[2];    // gate/up, down
  keepvq_router_logits_args logits;  // FT_ROUTER
  keepvq_routed_topk_args topk;
  const uint32_t* slot;       // without FT_ROUTER: the routes' slots and gate weights (weight may be null: 1)
  const float* weight;
  float swiglu_limit;
  void* out;                  // FT_COMBINE: the pick sums, in the activation dtype, plus `shared` (may be null)
  const float* shared;
  void* dead_out;             // rows of routes without a slot are zeroed here (may be null)
  int64_t dead_row_bytes;
  int32_t* status;            // 1: a wait of the grid ran out, 2: unexpected shared window
  int32_t clear_status;       // ... set to 0 first
  uint64_t* barrier_words;    // filled in by the launch
  uint32_t* counters;
  uint64_t token, wait_ns;    // filled in by the launch where they are zero
  uint64_t by_grid;
  int32_t absent;             // self-test: a CTA comes to neither barrier (1), or to the first only (2)
  int32_t ctas;               // self-test: so many CTAs (0: one per SM)
  uint32_t act_bytes;
  int32_t group_shift;
};
// Which layer calls the few-token kernel is the faster one for (us a layer against the chain of kernels, B200): 12 and
// 14 tokens of top-6 of 384 experts 152 and 176 against 177 and 191, 16 tokens 192 against 178; 8, 12, 14 and 16
// tokens of 192 experts with scale groups 158, 214, 240 and 259 against 194, 240, 265 and 259.  Where experts get
// several routes each the chain's groups of them win earlier: of 16 experts 8 tokens 67 against 77, 10 tokens 78
// against 77, 12 tokens 84 against 77; 40 routes of four experts (10 tokens, top-4) 56.9 against 59.2, of 1024 x 512
// 28.9 against 29.7.
inline bool few_tokens_pay(int64_t routes, int64_t slots) { return routes < SMALL_CALL_ROUTES || (routes <= FEW_TOKENS_ROUTES && routes <= slots / 2); }
// ... and which of them have the router in the same launch.  There every CTA works out every token's picks, four tokens
// at a time, which ends the gain of two launches less: us a layer with the router in the launch / in front of it / the
// chain of kernels (B200; the latter two never differ by more than 1 % to the chain's side):
//   8 experts, top-2, 4096 x 2048    12 tokens 50.4 / 52.0 / 52.7, 14 tokens 55.3 / 55.4 / 57.1, 17 tokens 62.6 / 58.1 / 60.8, 23 tokens 72.7 / 64.8 / 66.7
//   8 experts, top-2, 1024 x 512     12 tokens 27.4 / 24.5 / 28.4, 14 tokens 29.6 / 24.7 / 29.5, 23 tokens 36.3 / 25.5 / 30.1
//   48 experts, top-2, 512 x 256     12 tokens 27.0 / 22.6 / 27.7, 14 tokens 29.0 / 22.8 / 28.2, 23 tokens 35.4 / 23.7 / 28.6
//   8 experts, top-2, 5120 x 2304 with scale groups  14 tokens 70.9 / 72.7 / 82.6, 16 tokens 72.2 / 73.8 / 83.1, 17 tokens 79.2 / 76.5 / 87.9
inline bool few_tokens_router_pays(int64_t tokens, int64_t hidden) { return tokens <= (hidden > 4096 ? 16 : 12); }
bool few_tokens_fits(int64_t routes, int64_t tokens, int64_t slots, int64_t out_dim, int64_t in_dim, int64_t groups);
bool few_tokens_router_fits(const keepvq_router_logits_args& logits, const keepvq_routed_topk_args& topk);
int64_t few_tokens_sync_bytes(int64_t tokens, int64_t out_dim);  // scratch of a call with gate/up and down, any contents
int few_tokens(const FewTokensArgs& a, int32_t x_dtype, void* sync, cudaStream_t s);  // KEEPVQ_ERR_UNSUPPORTED: nothing was launched, the other kernels take the call

// tcgen05 kernels for many routes per expert (prefill_umma.cu).  `status` is a device word that
// a CTA sets to 1 if one of its bounded waits expires.
bool prefill_supported(int64_t slots, int64_t out_dim, int64_t in_dim, int64_t groups);
// The tcgen05 kernels decode a code once per 48 or 96 routes of an expert and cost nearly the same for
// one route as for 48; the mma.sync kernels stream an expert's codes once per 4 or 8 routes.  Which
// one pays depends on routes per expert, and the host only knows their number over the call (reading
// the routing back would stall the stream).  Whole layers, mma.sync against tcgen05: 384 experts of
// 4096 x 2048, one scale group: 825 / 834 us at 4 routes an expert, 870 / 855 at 5, 1136 / 869 at 7.5;
// 192 experts of 5120 x 2304 in groups of 512 and 256: 713 / 971 us at 4, 961 / 962 at 8, 4459 / 1119 at 32.
constexpr int64_t PREFILL_MIN_ROUTES = 1024;
inline bool prefill_pays(int64_t live, int64_t slots, bool several_groups) { return live >= PREFILL_MIN_ROUTES && live >= (several_groups ? 8 : 5) * slots; }
// Routes per item (group_routes' max_group) of a call with `live` routes; a kernel takes p.group_cols.
int prefill_group_routes(int64_t live, int64_t slots, bool several_groups);
int prefill_gate_up(const FastProjectionArgs& args, int32_t* status, cudaStream_t s);
int prefill_down(const FastProjectionArgs& args, int32_t* status, cudaStream_t s);
int prefill_byte_codes(const FastProjectionArgs& args, int32_t* status, cudaStream_t s);
// One CTA one of whose loaders never publishes, with a deadline of wait_ns: the wait runs out, the CTA sets *status = 1 and returns.
int prefill_wait_selftest(int form, const FastProjectionArgs& args, int32_t* status, uint64_t wait_ns, cudaStream_t s);

}  // namespace fast
}  // namespace keepvq
