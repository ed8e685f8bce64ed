// Tensor-core decode path for the routed E8P experts: activation quantisation, route grouping
// and the choice of projection kernel.  See moe_fast.cuh for the arithmetic identity it rests on.
//
// The projection kernels themselves (HBM-bound by design: every code byte is read once per group
// of routes) live in their own files: projection_slab.cu (calls with many route groups, and their
// split form for a residual tier with few), projection_sweep.cu (few route groups),
// few_tokens.cu (a whole call of few routes in one launch) and prefill_umma.cu (many routes per expert, tcgen05).  They share:
//   - a codeword becomes the A fragment of an m16n8k32 int8 MMA through two 4-byte table reads
//     (abs byte, sign byte; 32 replicas each so lanes never share a bank) XORed and spread from
//     nibbles to bytes: the nibble decoder of moe_fast.cuh;
//   - the K order inside an MMA is permuted (byte j of the low word is table nibble 3-j, of the
//     high word nibble 7-j); the activations are stored in that same order by quantize_rows;
//   - accumulation is exact in int32; one conversion to fp32 per scale group.
#include <stdlib.h>

#include <algorithm>
#include <type_traits>

#include "moe_fast.cuh"
#include "router_logits.cuh"

namespace keepvq {
namespace fast {

// ------------------------------------------------------------------------------------------
// Activation quantisation: x -> 16-bit fixed point with a power-of-two scale per row.
// ------------------------------------------------------------------------------------------
// One row per team of THREADS threads, the whole block or (THREADS = 32) one warp of it.  What bounds it is bytes and, before that, instructions: an
// element costs about six (widen, one fused multiply-add whose magic addend leaves the rounded integer
// in the low bits, one add, one and a half byte permutes, half an add for the sums; the first form's
// conversions, clamps, shifts and shared-memory atomics took 138 us for the 4096 tokens of a 4096-wide
// call, written once per route).  The row stays in registers between the maximum and the conversion.
//
// Where a row's values go: `targets` rows of the output, target(j) its index or a negative value for
// none.  Inputs come in multiples of 256 (shapes_supported), so a warp's 32 codewords are one chunk of
// 256 inputs and a scale group is a whole number of chunks.  `sm`: in_dim / 256 ints.
template <typename XT, int THREADS, typename Target>
__device__ __forceinline__ void quantize_row(const XT* __restrict__ xr, int64_t rows, int64_t in_dim, int64_t groups, const QuantRows& out, int planes, int32_t* sm, int targets, Target target) {
  // Vectors of eight values a thread keeps.  Blocks of 256 serve calls of a few rows, where the code a
  // cold launch has to fetch counts (eight copies of the conversion cost such a call a microsecond).
  // They cover rows of 2560 inputs (a warp), 5120 (128 threads) and 4096 (256); wider rows read the rest
  // twice, and what that costs at the next widths (7168, 8192) has not been measured.
  constexpr int KEEP = THREADS == 32 ? 10 : THREADS == 128 ? 5 : 2;
  constexpr bool PAIRS = sizeof(XT) == 2;  // 16-bit values: kept as they are, maximum taken on pairs
  __shared__ uint32_t warp_max[THREADS / 32];  // (a warp on its own has none to share)
  auto team_sync = [] { if (THREADS > 32) __syncthreads(); else __syncwarp(); };
  const int cw = static_cast<int>(in_dim / 8), chunks = cw / 32, per_group = chunks / static_cast<int>(groups);
  const int tid = threadIdx.x % THREADS, lane = tid & 31, warp = tid >> 5;
  uint4 raw[KEEP];
  // largest magnitude, as the bits of a float (they order like the values): a NaN or an infinity
  // anywhere gives the bits of an infinity or more
  uint32_t top_bits = 0;
  if constexpr (PAIRS) {
    typedef typename std::conditional<std::is_same<XT, __half>::value, __half2, __nv_bfloat162>::type Pair;
    uint32_t top = 0;
    auto take = [&](const uint4& r) {
      const uint32_t word[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t magnitude = word[k] & 0x7FFF7FFFu;
        const Pair m = __hmax2_nan(*reinterpret_cast<const Pair*>(&top), *reinterpret_cast<const Pair*>(&magnitude));
        top = *reinterpret_cast<const uint32_t*>(&m);
      }
    };
#pragma unroll
    for (int i = 0; i < KEEP; ++i) {
      const int c = tid + i * THREADS;
      if (c < cw) raw[i] = *reinterpret_cast<const uint4*>(xr + c * 8);
    }
#pragma unroll
    for (int i = 0; i < KEEP; ++i)
      if (tid + i * THREADS < cw) take(raw[i]);
#pragma unroll 1
    for (int c = tid + KEEP * THREADS; c < cw; c += THREADS) take(*reinterpret_cast<const uint4*>(xr + c * 8));
    const Pair pair = *reinterpret_cast<const Pair*>(&top);
    const float a = std::is_same<XT, __half>::value ? __half2float(*reinterpret_cast<const __half*>(&pair.x)) : __uint_as_float(top << 16);
    const float b = std::is_same<XT, __half>::value ? __half2float(*reinterpret_cast<const __half*>(&pair.y)) : __uint_as_float(top & 0xFFFF0000u);
    top_bits = max(__float_as_uint(a) & 0x7FFFFFFFu, __float_as_uint(b) & 0x7FFFFFFFu);
  } else {
    for (int c = tid; c < cw; c += THREADS) {
      float v[8];
      load8_as_float<XT>(xr + c * 8, v);
#pragma unroll
      for (int d = 0; d < 8; ++d) top_bits = max(top_bits, __float_as_uint(v[d]) & 0x7FFFFFFFu);
    }
  }
  auto team_max = [&](uint32_t bits) {
    bits = __reduce_max_sync(0xFFFFFFFFu, bits);
    if (THREADS > 32) {
      if (lane == 0) warp_max[warp] = bits;
      __syncthreads();
#pragma unroll
      for (int w = 0; w < THREADS / 32; ++w) bits = max(bits, warp_max[w]);
    }
    return bits;
  };
  top_bits = team_max(top_bits);
  const bool odd = top_bits >= 0x7F800000u;
  if (odd) {  // rows with a NaN or an infinity: the maximum leaves the NaNs out
    float amax = 0.0f;
    for (int c = tid; c < cw; c += THREADS) {
      float v[8];
      load8_as_float<XT>(xr + c * 8, v);
#pragma unroll
      for (int d = 0; d < 8; ++d) amax = fmaxf(amax, fabsf(v[d]));
    }
    team_sync();  // everyone has read warp_max
    top_bits = team_max(__float_as_uint(amax));
  }
  float inv;
  const float s = quant_scale(top_bits, inv);
  const bool plain = !odd && isfinite(inv);

  auto convert = [&](const float (&v)[8], int c) {
    const QuantWords w = quantize8(v, inv, plain);
    const int chunk_total = __reduce_add_sync(0xFFFFFFFFu, w.total);
    if (lane == 0) sm[c >> 5] = chunk_total;
    for (int j = 0; j < targets; ++j) {
      const int64_t row = target(j);
      if (row < 0) continue;
      if (planes) {  // high bytes of every row first, then the low bytes: what the tcgen05 B tiles copy from
        reinterpret_cast<uint2*>(out.q)[row * cw + c] = make_uint2(w.hi0, w.hi1);
        reinterpret_cast<uint2*>(out.q + (rows + 1) * cw * 8)[row * cw + c] = make_uint2(w.lo0, w.lo1);
      } else {
        reinterpret_cast<uint4*>(out.q)[row * cw + c] = make_uint4(w.hi0, w.hi1, w.lo0, w.lo1);
      }
    }
  };
  if constexpr (PAIRS) {
#pragma unroll
    for (int i = 0; i < KEEP; ++i) {
      const int c = tid + i * THREADS;
      if (c < cw) {
        float v[8];
        load8_as_float<XT>(reinterpret_cast<const XT*>(&raw[i]), v);
        convert(v, c);
      }
    }
  }
#pragma unroll 1
  for (int c = tid + (PAIRS ? KEEP * THREADS : 0); c < cw; c += THREADS) {
    float v[8];
    load8_as_float<XT>(xr + c * 8, v);
    convert(v, c);
  }
  team_sync();
  for (int j = 0; j < targets; ++j) {
    const int64_t row = target(j);
    if (row < 0) continue;
    if (tid == 0) out.scale[row] = s;
    for (int g = warp; g < groups; g += THREADS / 32) {
      int total = 0;
      for (int c = lane; c < per_group; c += 32) total += sm[g * per_group + c];
      total = __reduce_add_sync(0xFFFFFFFFu, total);
      if (lane == 0) out.sums[row * groups + g] = total;
    }
    if (out.chunk_sums)
      for (int c = tid; c < chunks; c += THREADS) out.chunk_sums[row * chunks + c] = sm[c];
  }
}
// The extra all-zero row: the B operand of MMA columns that carry no route.
template <int THREADS>
__device__ __forceinline__ void zero_row(int64_t row, int64_t rows, int64_t in_dim, int64_t groups, const QuantRows& out, int planes) {
  const int64_t cw = in_dim / 8;
  // (both layouts: the buffer is (rows + 1) * cw * 16 bytes either way)
  for (int64_t c = threadIdx.x; c < cw; c += THREADS) {
    if (planes) {
      reinterpret_cast<uint2*>(out.q)[row * cw + c] = make_uint2(0, 0);
      reinterpret_cast<uint2*>(out.q + (rows + 1) * cw * 8)[row * cw + c] = make_uint2(0, 0);
    } else {
      reinterpret_cast<uint4*>(out.q)[row * cw + c] = make_uint4(0, 0, 0, 0);
    }
  }
  for (int64_t g = threadIdx.x; g < groups; g += THREADS) out.sums[row * groups + g] = 0;
  if (out.chunk_sums)
    for (int64_t c = threadIdx.x; c < cw / 32; c += THREADS) out.chunk_sums[row * (cw / 32) + c] = 0;
  if (threadIdx.x == 0) out.scale[row] = 1.0f;
}

// Zeroes the output rows of the dead routes that read activation row `row`.
template <int THREADS>
__device__ __forceinline__ void zero_dead_rows(const DeadRows& dead, int64_t row) {
  if (!dead.slot) return;
  for (int j = 0; j < dead.per_row; ++j) {
    const int64_t route = row * dead.per_row + j;
    if (dead.slot[route] < static_cast<uint64_t>(dead.slots)) continue;
    uint16_t* out = reinterpret_cast<uint16_t*>(static_cast<uint8_t*>(dead.out) + route * dead.row_bytes);
    for (int64_t i = threadIdx.x % THREADS; i < dead.row_bytes / 2; i += THREADS) out[i] = 0;
  }
}

// `live` (may be null): the slots of the routes that read the rows, `per_row` of them per row; a row
// none of whose routes has a slot below `slots` is skipped (no kernel reads it: projections only
// follow live routes).  An expert-parallel rank quantises 8 x capacity rows of which an eighth is live.
struct LiveRows { const uint32_t* slot; int32_t per_row; int64_t slots; };

// One more block (the last) may group the routes of the call, which needs nothing of the rows:
// one launch less in front of the projections.
struct GroupJob { const uint32_t* served_slot; int32_t routes, slots, max_group; RouteGroups out; int32_t* clear; };

template <typename XT>
__global__ void __launch_bounds__(256) quantize_rows_kernel(const XT* __restrict__ x, int64_t rows, int64_t in_dim, int64_t groups, QuantRows out, int planes, LiveRows live, GroupJob job, DeadRows dead) {
  grid_launch_dependents();
  grid_wait();
  extern __shared__ int32_t sm[];
  const int64_t row = blockIdx.x;
  if (row > rows) {  // only launched when there is a job
    group_routes_block<256>(job.served_slot, job.routes, job.slots, job.max_group, job.out, job.clear, sm);
    return;
  }
  if (row == rows) return zero_row<256>(row, rows, in_dim, groups, out, planes);
  zero_dead_rows<256>(dead, row);
  if (live.slot) {
    bool any = false;
    for (int j = 0; j < live.per_row; ++j) any = any || live.slot[row * live.per_row + j] < static_cast<uint64_t>(live.slots);
    if (!any) return;  // uniform over the block
  }
  quantize_row<XT, 256>(x + row * in_dim, rows, in_dim, groups, out, planes, sm, 1, [&](int) { return row; });
}

// Byte planes with a row per route in grouped order (what the tcgen05 kernels' TMA boxes copy).  Blocks
// of 128 threads; a row takes all of them or, up to QS_WARP_ROW inputs, one warp, which needs no block
// barrier.
constexpr int QS_THREADS = 128;
constexpr int64_t QS_WARP_ROW = 2560;
template <typename XT, int TEAM>
__global__ void __launch_bounds__(QS_THREADS) quantize_rows_sorted_kernel(const XT* __restrict__ x, int64_t x_rows, int64_t in_dim, int64_t groups, QuantRows out, const int32_t* __restrict__ position, int x_div, DeadRows dead) {
  grid_launch_dependents();
  grid_wait();
  extern __shared__ int32_t sm[];
  constexpr int TEAMS = QS_THREADS / TEAM;
  const int team = threadIdx.x / TEAM;
  const int64_t r = static_cast<int64_t>(blockIdx.x) * TEAMS + team, rows = x_rows * x_div;
  if (blockIdx.x == gridDim.x - 1) return zero_row<QS_THREADS>(rows, rows, in_dim, groups, out, 1);
  if (r >= x_rows) return;
  zero_dead_rows<TEAM>(dead, r);
  bool any = false;
  for (int j = 0; j < x_div; ++j) any = any || position[r * x_div + j] >= 0;
  if (!any) return;  // nothing reads the row (uniform over the team)
  quantize_row<XT, TEAM>(x + r * in_dim, rows, in_dim, groups, out, 1, sm + team * (in_dim / 256), x_div, [&](int j) { return static_cast<int64_t>(position[r * x_div + j]); });
}

// The front of a decode layer call in one launch: the router's logits (the few-token kernel's
// blocks, router_logits.cuh) and the quantisation of the same token rows for the projections
// (rows + 1 further blocks).  Neither needs the other's result, and at a handful of tokens a launch
// costs more than either does.
template <typename XT, typename WT>
__global__ void __launch_bounds__(256) logits_and_quantize_kernel(keepvq_router_logits_args a, int logit_blocks_x, int logit_blocks, int64_t groups, QuantRows out) {
  static_assert(RL_WARPS * 32 == 256, "both halves run on blocks of 256 threads");
  grid_launch_dependents();
  grid_wait();
  const int b = static_cast<int>(blockIdx.x);
  if (b < logit_blocks) router_logits_block<XT, WT>(a, b % logit_blocks_x, b / logit_blocks_x);
  else {
    extern __shared__ int32_t sm[];
    const int64_t row = b - logit_blocks;
    if (row == a.tokens) zero_row<256>(row, a.tokens, a.hidden, groups, out, 0);
    else quantize_row<XT, 256>(reinterpret_cast<const XT*>(a.x) + row * a.hidden, a.tokens, a.hidden, groups, out, 0, sm, 1, [&](int) { return row; });
  }
}

template <typename XT>
static cudaError_t launch_front(const keepvq_router_logits_args& a, int bx, int blocks, int64_t groups, const QuantRows& out, size_t smem, cudaStream_t s) {
  const unsigned grid = static_cast<unsigned>(blocks + a.tokens + 1);
  if (a.router_dtype == KEEPVQ_F32) return launch_after(true, logits_and_quantize_kernel<XT, float>, grid, 256, smem, s, a, bx, blocks, groups, out);
  if (a.router_dtype == KEEPVQ_F16) return launch_after(true, logits_and_quantize_kernel<XT, __half>, grid, 256, smem, s, a, bx, blocks, groups, out);
  return launch_after(true, logits_and_quantize_kernel<XT, __nv_bfloat16>, grid, 256, smem, s, a, bx, blocks, groups, out);
}

static size_t chunk_bytes(int64_t in_dim) { return static_cast<size_t>(in_dim / 256) * sizeof(int32_t); }  // quantize_row's shared memory

bool logits_and_quantize_supported(const keepvq_router_logits_args& a, int64_t groups) {
  return a.tokens > 0 && a.tokens <= FRONT_MAX_TOKENS && a.x_dtype != KEEPVQ_F32 && a.hidden % 256 == 0 && chunk_bytes(a.hidden) <= 40 * 1024 &&
         (a.pool + RL_ROWS - 1) / RL_ROWS * ((a.tokens + RL_TOKENS - 1) / RL_TOKENS) <= EARLY_LAUNCH_MAX_BLOCKS;
}

int logits_and_quantize(const keepvq_router_logits_args& a, int64_t groups, const QuantRows& out, cudaStream_t s) {
  const int bx = static_cast<int>((a.pool + RL_ROWS - 1) / RL_ROWS), by = static_cast<int>((a.tokens + RL_TOKENS - 1) / RL_TOKENS);
  const size_t smem = chunk_bytes(a.hidden);
  const cudaError_t err = a.x_dtype == KEEPVQ_F16 ? launch_front<__half>(a, bx, bx * by, groups, out, smem, s) : launch_front<__nv_bfloat16>(a, bx, bx * by, groups, out, smem, s);
  if (err != cudaSuccess) return note_cuda_error(err);
  return KEEPVQ_OK;
}

int quantize_rows(const void* x, int32_t x_dtype, int64_t rows, int64_t in_dim, int64_t groups, const QuantRows& out, bool planes, cudaStream_t s,
                  const uint32_t* live_slot, int32_t per_row, int64_t slots) {
  return quantize_rows_and_group(x, x_dtype, rows, in_dim, groups, out, planes, s, live_slot, per_row, slots, nullptr, 0, 0, RouteGroups{}, nullptr);
}

template <typename XT>
static cudaError_t launch_sorted(const void* x, int64_t x_rows, int64_t in_dim, int64_t groups, const QuantRows& out, const int32_t* position, int32_t x_div, cudaStream_t s, const DeadRows& dead) {
  const bool warps = in_dim <= QS_WARP_ROW;
  const int64_t teams = warps ? QS_THREADS / 32 : 1;
  const unsigned grid = static_cast<unsigned>((x_rows + teams - 1) / teams + 1);  // + the zero row
  return launch_after(grid < EARLY_LAUNCH_MAX_BLOCKS, warps ? quantize_rows_sorted_kernel<XT, 32> : quantize_rows_sorted_kernel<XT, QS_THREADS>, grid, QS_THREADS,
                      chunk_bytes(in_dim) * teams, s, static_cast<const XT*>(x), x_rows, in_dim, groups, out, position, x_div, dead);
}
int quantize_rows_sorted(const void* x, int32_t x_dtype, int64_t x_rows, int64_t in_dim, int64_t groups, const QuantRows& out, const int32_t* position, int32_t x_div, cudaStream_t s, const DeadRows& dead) {
  if (chunk_bytes(in_dim) > 40 * 1024) return KEEPVQ_ERR_CAPACITY;
  cudaError_t err;
  if (x_dtype == KEEPVQ_F32) err = launch_sorted<float>(x, x_rows, in_dim, groups, out, position, x_div, s, dead);
  else if (x_dtype == KEEPVQ_F16) err = launch_sorted<__half>(x, x_rows, in_dim, groups, out, position, x_div, s, dead);
  else err = launch_sorted<__nv_bfloat16>(x, x_rows, in_dim, groups, out, position, x_div, s, dead);
  if (err != cudaSuccess) return note_cuda_error(err);
  return KEEPVQ_OK;
}

bool group_with_quantize_supported(int64_t routes, int64_t slots) { return routes <= 4096 && slots * 3 * sizeof(int32_t) <= 40 * 1024; }

int quantize_rows_and_group(const void* x, int32_t x_dtype, int64_t rows, int64_t in_dim, int64_t groups, const QuantRows& out, bool planes, cudaStream_t s,
                            const uint32_t* live_slot, int32_t per_row, int64_t slots,
                            const uint32_t* served_slot, int64_t routes, int max_group, const RouteGroups& route_groups, int32_t* clear, const DeadRows& dead) {
  const LiveRows live = {live_slot, per_row, slots};
  const GroupJob job = {served_slot, static_cast<int32_t>(routes), static_cast<int32_t>(slots), max_group, route_groups, clear};
  size_t smem = chunk_bytes(in_dim);
  if (smem > 40 * 1024) return KEEPVQ_ERR_CAPACITY;
  if (served_slot) {
    if (!group_with_quantize_supported(routes, slots)) return KEEPVQ_ERR_UNSUPPORTED;
    smem = std::max(smem, static_cast<size_t>(slots) * 3 * sizeof(int32_t));
  }
  const unsigned grid = static_cast<unsigned>(rows + 1 + (served_slot ? 1 : 0));  // + the zero row (+ the grouping block)
  const bool early = rows < EARLY_LAUNCH_MAX_BLOCKS;
  cudaError_t err;
  if (x_dtype == KEEPVQ_F32) err = launch_after(early, quantize_rows_kernel<float>, grid, 256, smem, s, reinterpret_cast<const float*>(x), rows, in_dim, groups, out, planes ? 1 : 0, live, job, dead);
  else if (x_dtype == KEEPVQ_F16) err = launch_after(early, quantize_rows_kernel<__half>, grid, 256, smem, s, reinterpret_cast<const __half*>(x), rows, in_dim, groups, out, planes ? 1 : 0, live, job, dead);
  else err = launch_after(early, quantize_rows_kernel<__nv_bfloat16>, grid, 256, smem, s, reinterpret_cast<const __nv_bfloat16*>(x), rows, in_dim, groups, out, planes ? 1 : 0, live, job, dead);
  if (err != cudaSuccess) return note_cuda_error(err);
  return KEEPVQ_OK;
}

// ------------------------------------------------------------------------------------------
// Route grouping: routes that are served from the same slot share the code stream.  One block;
// counting sort by slot, then each slot's routes are cut into groups of at most max_group.
// ------------------------------------------------------------------------------------------
constexpr int GR_THREADS = 1024;

__global__ void __launch_bounds__(GR_THREADS) group_routes_kernel(const uint32_t* __restrict__ served_slot, int routes, int slots, int max_group, RouteGroups out, int32_t* clear) {
  grid_launch_dependents();
  grid_wait();
  extern __shared__ int32_t group_scratch[];
  group_routes_block<GR_THREADS>(served_slot, routes, slots, max_group, out, clear, group_scratch);
}

int group_routes(const uint32_t* served_slot, int64_t routes, int64_t slots, int max_group, const RouteGroups& out, int32_t* clear, cudaStream_t s, bool early) {
  if (routes > (1 << 20) || slots > 16384) return KEEPVQ_ERR_CAPACITY;
  const size_t smem = static_cast<size_t>(slots) * 3 * sizeof(int32_t);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(group_routes_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return note_cuda_error(e);
  }
  cudaError_t err = launch_after(early && routes <= 4 * EARLY_LAUNCH_MAX_BLOCKS, group_routes_kernel, 1, GR_THREADS, smem, s, served_slot, static_cast<int>(routes), static_cast<int>(slots), max_group, out, clear);
  if (err != cudaSuccess) return note_cuda_error(err);
  return KEEPVQ_OK;
}

// ------------------------------------------------------------------------------------------
// Which kernel runs a grouped projection.
// ------------------------------------------------------------------------------------------
constexpr int CHUNK_CODES = 32;               // codewords of a row a warp consumes per step: inputs come in multiples of 256

bool shapes_supported(int64_t out_dim, int64_t in_dim, int64_t groups) {
  if (in_dim % (8 * CHUNK_CODES) != 0 || groups <= 0) return false;
  const int64_t chunks = in_dim / (8 * CHUNK_CODES);
  return chunks % groups == 0 && in_dim / groups <= MAX_GROUP_INPUTS && out_dim > 0;
}

// Enough routes to give every CTA of the machine its own (group, slab) items, and activations
// that fit the shared-memory stage?
static bool many_items(const FastProjectionArgs& p) {
  return p.max_routes >= SMALL_CALL_ROUTES && p.in_dim <= slab_max_in_dim(p.group_cols > PAIRED_GROUP_ROUTES ? MAX_GROUP_ROUTES : PAIRED_GROUP_ROUTES);
}
// Few route groups of at most four routes (of the calls that the few-token kernel does not take).  Small calls run the sweep kernel (measured on a B200 at
// 4096 inputs: ahead of the split slab kernel up to four tokens of top-6, behind it at eight); the
// rest, and every layer with a residual tier (the slab kernels hold the residual pass), the split
// form of the slab kernel when the activations leave it room.  0 = neither, 1 = split slab, 2 = sweep.
static int few_items(const FastProjectionArgs& p) {
  if (!p.few_groups || p.group_cols > PAIRED_GROUP_ROUTES) return 0;
  const bool split_fits = p.in_dim <= slab_split_max_in_dim(), sweep_fits = !p.res_table && sweep_supported(p.in_dim);
  if (p.few_groups == 2 && sweep_fits) return 2;
  return split_fits ? 1 : sweep_fits ? 2 : 0;
}

int decode_group_routes(int64_t live, int64_t slots, int64_t widest_in_dim) {
  if (live < SMALL_CALL_ROUTES) return PAIRED_GROUP_ROUTES;  // the sweep kernel (the split slab kernel with a residual tier)
  if (widest_in_dim > slab_max_in_dim(MAX_GROUP_ROUTES)) return PAIRED_GROUP_ROUTES;
  return live <= 2 * slots ? PAIRED_GROUP_ROUTES : MAX_GROUP_ROUTES;
}

// The residual pass lives in the slab kernels only: a layer with a residual tier needs activations
// that fit their stage (three quarters of it for calls with few routes) and residual scale groups
// that close on chunk boundaries.
bool residual_supported(int64_t routes, int64_t in_dim, int64_t res_groups) {
  const int64_t widest = routes < SMALL_CALL_ROUTES ? slab_split_max_in_dim() : slab_max_in_dim(PAIRED_GROUP_ROUTES);
  if (in_dim > widest || in_dim % (8 * CHUNK_CODES) != 0 || res_groups <= 0) return false;
  return (in_dim / (8 * CHUNK_CODES)) % res_groups == 0;
}

int gate_up(const FastProjectionArgs& p, cudaStream_t s) {
  if (const int few = few_items(p)) return few == 2 ? sweep_gate_up(p, s) : slab_split_gate_up(p, s);
  if (!many_items(p)) return KEEPVQ_ERR_UNSUPPORTED;
  return slab_gate_up(p, p.group_cols > PAIRED_GROUP_ROUTES ? MAX_GROUP_ROUTES : PAIRED_GROUP_ROUTES, s);
}
int down(const FastProjectionArgs& p, cudaStream_t s) {
  if (const int few = few_items(p)) return few == 2 ? sweep_down(p, s) : slab_split_down(p, s);
  if (!many_items(p)) return KEEPVQ_ERR_UNSUPPORTED;
  return slab_down(p, p.group_cols > PAIRED_GROUP_ROUTES ? MAX_GROUP_ROUTES : PAIRED_GROUP_ROUTES, s);
}

}  // namespace fast
}  // namespace keepvq
