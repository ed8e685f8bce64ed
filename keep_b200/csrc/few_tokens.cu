// One routed layer for a handful of tokens as ONE launch, and the routed projections of calls with
// few routes: the few-token kernel.
//
// With a few tokens a layer call is some megabytes of codes and a chain of dependencies: logits,
// top-k, grouping, quantise, gate/up, quantise, down, pick sum.  As seven launches of one stream that
// chain cost a one-token layer (384 experts of 4096 x 2048) 47 us, 30 of them the two projections and
// the rest launches and their ramps, where the codes take 6 us to read.  Here one CTA per SM stays for
// the whole layer: 34 us (2 / 4 / 7 tokens: 62 -> 45, 92 -> 67, 132 -> 102; 192 experts of 5120 x 2304 with
// scale groups, 1 / 3 / 7 tokens: 62 -> 45, 115 -> 82, 195 -> 143).  What needs everybody's results waits at one of two grid barriers (the logits
// before the top-k, the hidden rows before the down projection); what is small is worked out by every
// CTA for itself (top-k, route grouping, the quantisation of the few activation rows its share of the
// work reads); the pick sum is done by whichever CTA brings a token's last row.
//
// The projections.  The unit of work is two MMA row tiles of one route group: 16 rows of gate and up,
// or 32 rows of a single matrix.  The CTAs get equal contiguous runs of units, and the 16 warps of a
// CTA equal contiguous runs of (unit, chunk of 256 inputs) pairs, whatever the number of chunks: a
// warp sweeps along the rows of a unit, then the next unit's, and only a unit that two or more
// warps share is added up through shared memory.  A CTA's units lie in at most two route groups, so
// the activations it needs are at most eight rows, quantised once into shared memory in the
// order the MMA fragments are read.  Codes come through a private cp.async ring per warp that runs
// ahead across units.
// Arithmetic as in the other decode kernels (moe_fast.cuh), int8 mma.sync with a route's two
// byte planes as neighbouring columns, except that the even and the odd dims of two codewords make an
// MMA each: the odd dims' nibbles then stay in the upper half of their bytes (their own accumulators
// come out 16 times too large, exactly), which saves the shift per codeword.
//
// What bounds it: from three tokens on the sweep, whose chunk of 32 x 32 codewords takes an SM some 135
// cycles where its table reads, codes and activations are 105 wavefronts of shared memory (the same
// with the codes brought by TMA: 150); with one or two tokens the chain of some twenty short steps between
// launch and last store, none of which keeps an SM busy.  Those run once, so what they cost is the code
// itself: at 230 KB of instructions (loops unrolled, score functions and slow paths inlined) the one-token
// layer took 38 us, at 97 KB 34.  Hence the loops kept rolled and the calls kept calls below.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <type_traits>
#include <utility>

#include "async_copy.cuh"
#include "moe_fast.cuh"
#include "router_topk.cuh"

namespace keepvq {
namespace fast {

constexpr int FT_WARPS = 16;
static_assert(FT_MAX_ROUTES % 4 == 0, "slots are looked at four at a time");
constexpr int FT_THREADS = FT_WARPS * 32;
constexpr int FT_CHUNK = 32;                  // codewords of a row per step of a warp
constexpr int FT_ROWS = 8;                    // activation rows a CTA stages: two groups of up to four routes, or all of up to eight tokens
constexpr int FT_MAX_IN = 5120;               // what the activation stage holds eight rows of
constexpr int FT_MAX_CHUNKS = FT_MAX_IN / 256;
constexpr int FT_CLOSE_CHUNKS = 16;           // 4 sum(w x') of 4096 inputs fits 32 bits
constexpr int FT_TOPK_NPL = 12;               // experts per lane: pools of up to 384 (16 tokens' scores lie in the low rings)
constexpr uint32_t FT_TABLE_BYTES = 64 * 1024;
constexpr uint32_t FT_STAGE_BYTES = 4 * 512;  // four 16-byte streams per lane
constexpr int FT_SMEM_BYTES = 217 * 1024;     // dynamic; the static arrays take 9 to 10 KB, and all of it is at most 227 KB
constexpr uint32_t FT_STATIC_MIN = 9 * 1024, FT_STATIC_MAX = 11 * 1024;  // where the dynamic part begins (the kernel checks what the launch makes of it)
constexpr int FT_BARRIER_WORDS = FT_MAX_CTAS + 16;  // a word per CTA, and on a line of its own the one all wait on
constexpr uint64_t FT_WAIT_NS = 2000000000ull;
constexpr int FT_ABSENT_CTA = 3;  // the one that does not come in the self-test
constexpr uint32_t FT_PREFETCH_BYTES = 96 * 1024;  // of a CTA's down codes, asked into L2 while gate/up runs
static_assert(FT_MAX_CHUNKS <= 32, "a warp looks at all chunks of a row at once");

template <int N, typename F, int... I>
__device__ __forceinline__ void ft_static_for_impl(F&& f, std::integer_sequence<int, I...>) { (f(std::integral_constant<int, I>{}), ...); }
template <int N, typename F>
__device__ __forceinline__ void ft_static_for(F&& f) { ft_static_for_impl<N>(static_cast<F&&>(f), std::make_integer_sequence<int, N>{}); }

__device__ __forceinline__ void ft_cp_async16(uint32_t dst, uint64_t src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ uint4 ft_lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
template <int OFF>
__device__ __forceinline__ uint2 ft_lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2+%3];" : "=r"(v.x), "=r"(v.y) : "r"(addr), "n"(OFF));
  return v;
}
__device__ __forceinline__ void ft_mma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t ft_word(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
// n / d for a divisor the launch has put as ceil(2^40 / d): exact while n * d < 2^40.
static uint64_t ft_divisor(int64_t d) { return ((uint64_t{1} << 40) + d - 1) / d; }
__device__ __forceinline__ int ft_div(uint32_t n, uint64_t divisor) { return static_cast<int>((n * divisor) >> 40); }
// All CTAs of the (cooperative) grid meet, in two halves.  Every CTA has a word of its own, which it
// sets to the launch's token.  A word left by another launch, or never written, does not match the
// token, so the words need no clearing before the launch.  A replay from a captured graph has the token
// of the launch before it, so none may be left set, however a launch ends: a CTA clears its own words on
// every way out, and the word that the others wait on is written by the first CTA alone, which clears
// it once every other CTA has taken its word back.  Nobody writes another's word, so this holds in
// whatever order CTAs give up.  A CTA may take its words back only when nobody still waits for them, so
// the last barrier of a launch is one that GATHERs, which the others pass only after the first CTA has
// seen every word (and by then everybody has passed the barrier before it, too).
__device__ __forceinline__ void ft_set(uint64_t* word, uint64_t value) { asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(word), "l"(value) : "memory"); }
__device__ __forceinline__ void ft_clear(uint64_t* word) { asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(word), "l"(uint64_t{0}) : "memory"); }
__device__ __forceinline__ uint64_t ft_get(const uint64_t* word) {
  uint64_t seen;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(word) : "memory");
  return seen;
}
__device__ __forceinline__ void ft_arrive(uint64_t* words, uint64_t token) {
  __syncthreads();
  if (threadIdx.x == 0) ft_set(words + blockIdx.x, token);
}
// Until the word holds the token (or, with `gone`, no longer does).
__device__ __forceinline__ int ft_poll(const uint64_t* word, uint64_t token, uint64_t deadline, bool gone = false) {
  for (uint32_t spin = 0;; ++spin) {
    if ((ft_get(word) == token) != gone) return 1;
    if ((spin & 63u) == 63u && global_timer_ns() > deadline) return 0;
  }
}
// False in every thread when the deadline passes.  Gathering, the first CTA looks at all words, then sets
// the one that the others wait on; without it every CTA looks at every word, which is sooner done
// where the words are mostly set already, and takes 4 to 6 us where they are not.
__device__ __forceinline__ bool ft_wait(uint64_t* words, uint64_t token, uint64_t deadline, bool gather) {
  uint64_t* go = words + FT_MAX_CTAS;
  int ok = 1;
  if (!gather || blockIdx.x == 0) {
    for (unsigned i = threadIdx.x; i < gridDim.x && ok; i += FT_THREADS) ok = ft_poll(words + i, token, deadline);
    ok = __syncthreads_and(ok);
    if (gather && threadIdx.x == 0 && ok) ft_set(go, token);
    return ok != 0;
  }
  if (threadIdx.x == 0) ok = ft_poll(go, token, deadline);
  return __syncthreads_and(ok) != 0;
}

template <typename XT>
__device__ __forceinline__ uint32_t ft_float_bits(uint32_t magnitude) {  // a 16-bit magnitude as the bits of a float
  if (std::is_same<XT, __half>::value) return __float_as_uint(__half2float(__ushort_as_half(static_cast<unsigned short>(magnitude))));
  return magnitude << 16;
}
__device__ __forceinline__ uint4 ft_load_row16(const void* p) {  // (not the read-only path: hidden rows were written by this kernel)
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

// The served picks of up to four tokens from t0 on, by four warps a token: each scores its share of the
// pool and picks from it, one of them picks from the shares' picks.  (A warp alone took 2650 cycles
// for twelve scores a lane and 3200 for six picks, and all warps reading all logits of one token 3600, from twelve
// lines of L2 that 148 CTAs want at once.)  The arithmetic and the order of additions of routed_topk_reg_kernel.
// `scratch`: FT_PICK_BYTES of shared memory.  own: the token whose outputs this CTA writes and whose scores it keeps.
constexpr int FT_PICK_PARTS = 4, FT_PICK_TOKENS = FT_WARPS / FT_PICK_PARTS;
constexpr uint32_t FT_PICK_ROW = 32 * FT_TOPK_NPL * 4, FT_PICK_BYTES = FT_PICK_TOKENS * (2 * FT_PICK_ROW + 64 * 8);
static __device__ __noinline__ float ft_sigmoid(float v) { return topk_sigmoid(v); }  // (calls: see the top on the size of the code)
static __device__ __noinline__ float ft_sqrt_softplus(float v) { return topk_sqrt_softplus(v); }
__device__ __forceinline__ void ft_pick(const keepvq_routed_topk_args& k, uint32_t scratch, int t0, int own, float* own_scores, uint32_t* route_slot, float* route_weight) {
  constexpr int NQ = FT_TOPK_NPL / FT_PICK_PARTS, PARTS = FT_PICK_PARTS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, local = warp / PARTS, part = warp % PARTS;
  const int tokens = static_cast<int>(k.tokens), pool = static_cast<int>(k.pool), tok = t0 + local;
  const bool here = tok < tokens;
  const uint32_t exps = scratch + local * FT_PICK_ROW, scores = exps + FT_PICK_TOKENS * FT_PICK_ROW, shares = scratch + 2 * FT_PICK_TOKENS * FT_PICK_ROW + local * (64 * 8);
  auto put = [](uint32_t at, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory"); };
  auto get = [](uint32_t at) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at));
    return v;
  };
  float sc[NQ];
  int id[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    id[q] = lane + 32 * (part + PARTS * q);
    sc[q] = here && id[q] < pool ? __ldcg(k.logits + static_cast<int64_t>(tok) * pool + id[q]) : -INFINITY;
  }
  if (k.score_func == KEEPVQ_SCORE_SOFTMAX) {
    float m = topk_max<NQ>(sc);
    if (lane == 0) put(shares + part * 4, __float_as_uint(m));
    __syncthreads();
#pragma unroll
    for (int q = 0; q < PARTS; ++q) m = fmaxf(m, __uint_as_float(get(shares + q * 4)));
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      sc[q] = id[q] < pool ? expf(sc[q] - m) : 0.0f;
      put(exps + id[q] * 4, __float_as_uint(sc[q]));
    }
    __syncthreads();
    float ex[FT_TOPK_NPL];
#pragma unroll
    for (int i = 0; i < FT_TOPK_NPL; ++i) ex[i] = __uint_as_float(get(exps + (lane + 32 * i) * 4));
    const float s = topk_sum<FT_TOPK_NPL>(ex, pool, lane);
#pragma unroll
    for (int q = 0; q < NQ; ++q) sc[q] = sc[q] / s;
  } else {
#pragma unroll
    for (int q = 0; q < NQ; ++q) sc[q] = k.score_func == KEEPVQ_SCORE_SIGMOID ? ft_sigmoid(sc[q]) : ft_sqrt_softplus(sc[q]);
  }
  uint32_t key[NQ], my_key;
  int my_e;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    put(scores + id[q] * 4, __float_as_uint(sc[q]));
    if (here && tok == own) own_scores[id[q]] = sc[q];
    key[q] = id[q] < pool ? topk_key(k.served_bias, id[q], sc[q]) : 0u;
  }
  topk_select<NQ>(key, id, k.top_k, lane, my_key, my_e);
  if (lane < 16) {
    put(shares + (part * 16 + lane) * 8, lane < k.top_k ? my_key : 0u);
    put(shares + (part * 16 + lane) * 8 + 4, static_cast<uint32_t>(my_e));
  }
  __syncthreads();
  if (part == 0 && here) {
    uint32_t share_key[2];  // 64 of them
    int share_id[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      share_key[q] = get(shares + (lane + 32 * q) * 8);
      share_id[q] = share_key[q] ? static_cast<int>(get(shares + (lane + 32 * q) * 8 + 4)) : 0x10000 + lane;  // (no key: no expert's id)
    }
    topk_select<2>(share_key, share_id, k.top_k, lane, my_key, my_e);
    uint32_t slot;
    float weight;
    topk_finish(k, tok, lane, 0, my_e, lane < k.top_k ? __uint_as_float(get(scores + my_e * 4)) : 0.0f, tok == own, slot, weight);
    if (lane < k.top_k) {
      route_slot[tok * k.top_k + lane] = slot;
      route_weight[tok * k.top_k + lane] = weight;
    }
  }
  __syncthreads();
}

// RAGGED: the output rows are not a multiple of a unit's rows, so the last unit of a group clamps its row indices.
// DEPTH: chunks of a warp in flight.
template <typename XT, bool RAGGED, int DEPTH>
__global__ void __launch_bounds__(FT_THREADS, 1) few_tokens_kernel(const __grid_constant__ FewTokensArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ __align__(16) uint32_t route_slot[FT_MAX_ROUTES];
  __shared__ float route_weight[FT_MAX_ROUTES];
  __shared__ int32_t grp_slot[FT_MAX_ROUTES], grp_size[FT_MAX_ROUTES], grp_route[FT_MAX_ROUTES][4];
  __shared__ int32_t grp_of_leader[FT_MAX_ROUTES], leaders_before[FT_MAX_ROUTES / 32 + 1];
  __shared__ float logit_part[2][8][2 * RL_TOKENS];
  __shared__ uint32_t piece_top[FT_ROWS * FT_MAX_CHUNKS];
  __shared__ float row_scale[FT_ROWS];
  __shared__ int32_t row_sums[FT_ROWS][FT_MAX_CHUNKS];
  __shared__ uint64_t deadline;
  __shared__ float own_scores[32 * FT_TOPK_NPL];
  __shared__ int32_t n_groups_s, n_due;
  constexpr uint32_t RING_BYTES = DEPTH * FT_STAGE_BYTES;  // of a warp; it also carries the warp's scores and its partial tile
  constexpr uint32_t INF16 = std::is_same<XT, __half>::value ? 0x7C00u : 0x7F80u;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int grid = static_cast<int>(gridDim.x), cta = static_cast<int>(blockIdx.x);
  grid_launch_dependents();
  if (warp == FT_WARPS - 1)  // the arguments' lines of constant memory, fetched together instead of one miss after the other
    asm volatile("" ::"l"(a.phase[0].codes[0]), "l"(a.phase[0].x), "l"(a.phase[0].by_units), "l"(a.phase[1].codes[0]), "l"(a.phase[1].x), "l"(a.phase[1].by_units),
                 "l"(a.topk.logits), "l"(a.topk.served_bias), "l"(a.topk.want), "l"(a.slot), "l"(a.shared), "l"(a.counters));

  // ---- the shared window: rings below the first 64 KB boundary as far as they fit, the two tables on
  // the boundary, the other rings, the activation rows
  const uint32_t base = smem_addr(smem);
  const uint32_t a0 = (base + 0xFFFFu) & ~0xFFFFu;
  const int low_rings = min(FT_WARPS, static_cast<int>((a0 - base) / RING_BYTES));
  const uint32_t high_rings = a0 + FT_TABLE_BYTES;
  const uint32_t acts = high_rings + (FT_WARPS - low_rings) * RING_BYTES;
  if (acts + a.act_bytes > base + FT_SMEM_BYTES || a0 - base < FT_PICK_BYTES) {  // uniform over the grid
    grid_wait();  // (an early launch that ended without it would let its successor overtake its predecessor)
    if (a.status && tid == 0) atomicExch(a.status, 2);
    return;
  }
  const uint32_t ring = (warp < low_rings ? base + warp * RING_BYTES : high_rings + (warp - low_rings) * RING_BYTES) + lane * 16;
  const uint32_t abs_lane = a0 + lane * 4u, sign_lane = a0 + 128u + lane * 4u;
  const bool with_router = a.parts & FT_ROUTER;
  const bool two_phases = (a.parts & FT_GATE_UP) && (a.parts & FT_DOWN);
  uint64_t* const words_a = a.barrier_words;
  uint64_t* const words_b = a.barrier_words + FT_BARRIER_WORDS;
  auto begin = [&]() {  // behind the wait on the previous kernel
    grid_wait();
    if (tid == 0) deadline = global_timer_ns() + a.wait_ns;  // (in shared memory: a pair of registers less in the sweep; read behind the barriers' own block barrier)
    if (cta == 0) {  // ordered before their first use by the barrier in front of the down projection
      if (a.parts & FT_COMBINE)  // the pick sum's counters
#pragma unroll 1
        for (int i = tid; i < a.tokens * (a.phase[1].out_dim / 32); i += FT_THREADS) a.counters[i] = 0;
      if (a.clear_status && a.status && tid == 0) *a.status = 0;
    }
  };
  auto take_words_back = [&]() {  // behind the last barrier, or on the way out
    if (tid == 0) {
      if (with_router) ft_clear(words_a + cta);
      if (two_phases) ft_clear(words_b + cta);
    }
  };
  auto give_up = [&]() {
    take_words_back();
    if (a.status && tid == 0) atomicExch(a.status, 1);
  };

  // ---- up to eight activation rows, quantised into fragment order in shared memory
  const int own_token = with_router ? grid - 1 - cta : -1;  // the token whose routing outputs this CTA writes (not the first CTA: it gathers a barrier)
  const int cap = 1 << a.group_shift;
  const bool by_token = with_router && a.tokens <= FT_ROWS;
  auto stage_rows = [&](const FewTokensPhase& P, int rows, int my_row) {  // lane r: the row of the phase's activations that is staged row r
    const int n_chunks = P.n_chunks, pieces = rows * n_chunks;  // (row, chunk) pairs, dealt round the warps
    const uint32_t row_stride = static_cast<uint32_t>(P.in_dim) * 2u + 64u;  // (64 bytes apart modulo 128: two rows of a group in one read do not meet in a bank)
    auto piece_from = [&](int piece) {  // the lane's eight values of it
      const int r = ft_div(piece, P.by_chunks);
      return static_cast<const uint8_t*>(P.x) + (static_cast<int64_t>(__shfl_sync(0xFFFFFFFFu, my_row, r)) * P.in_dim + (piece - r * n_chunks) * 256 + lane * 8) * 2;
    };
    uint4 kept = make_uint4(0, 0, 0, 0);  // of the warp's first piece, mostly its only one
#pragma unroll 1
    for (int p0 = warp; p0 < pieces; p0 += 4 * FT_WARPS) {  // four pieces of the warp at a time, their loads in flight together
      uint4 raw[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (p0 + i * FT_WARPS < pieces) raw[i] = ft_load_row16(piece_from(p0 + i * FT_WARPS));
      if (p0 == warp) kept = raw[0];
      uint32_t odd_pieces = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (p0 + i * FT_WARPS >= pieces) break;
        const uint32_t top = __vmaxu2(__vmaxu2(raw[i].x & 0x7FFF7FFFu, raw[i].y & 0x7FFF7FFFu), __vmaxu2(raw[i].z & 0x7FFF7FFFu, raw[i].w & 0x7FFF7FFFu));
        const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, max(top & 0xFFFFu, top >> 16));
        if (lane == 0) piece_top[p0 + i * FT_WARPS] = most << 16 | most;
        if (most >= INF16) odd_pieces |= 1u << i;
      }
#pragma unroll 1
      for (int i = 0; odd_pieces != 0; ++i, odd_pieces >>= 1) {  // a NaN or an infinity: the scale comes from a maximum that leaves the NaNs out
        if (!(odd_pieces & 1u)) continue;
        const uint4 again = ft_load_row16(piece_from(p0 + i * FT_WARPS));
        const uint32_t words[4] = {again.x, again.y, again.z, again.w};
        uint32_t finite = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t lo = words[q] & 0x7FFFu, hi = (words[q] >> 16) & 0x7FFFu;
          if (lo <= INF16) finite = max(finite, lo);
          if (hi <= INF16) finite = max(finite, hi);
        }
        finite = __reduce_max_sync(0xFFFFFFFFu, finite);
        if (lane == 0) piece_top[p0 + i * FT_WARPS] = 0xFFFF0000u | finite;
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int p = warp; p < pieces; p += FT_WARPS) {
      const uint4 raw = kept;
      if (p + FT_WARPS < pieces) kept = ft_load_row16(piece_from(p + FT_WARPS));  // the next piece's, under this one's arithmetic
      const int row = ft_div(p, P.by_chunks), chunk = p - row * n_chunks;
      const uint32_t tops = lane < n_chunks ? piece_top[row * n_chunks + lane] : 0u;
      const bool odd = __any_sync(0xFFFFFFFFu, (tops >> 16) >= INF16);
      float inv;
      const float s = quant_scale(ft_float_bits<XT>(__reduce_max_sync(0xFFFFFFFFu, tops & 0xFFFFu)), inv);
      float v[8];
      load8_as_float<XT>(reinterpret_cast<const XT*>(&raw), v);
      const QuantWords q = quantize8(v, inv, !odd && isfinite(inv));
      const int total = __reduce_add_sync(0xFFFFFFFFu, q.total);
      // codeword t * 8 + i of the chunk at [step i][t]: high plane's two words, low plane's two words
      asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(acts + row * row_stride + chunk * 512 + (lane & 7) * 64 + (lane >> 3) * 16), "r"(q.hi0), "r"(q.hi1), "r"(q.lo0), "r"(q.lo1) : "memory");
      if (lane == 0) { row_sums[row][chunk] = total; row_scale[row] = s; }
    }
    __syncthreads();
  };

  // ---- router: logits (the same order of additions as router_logits_block: eight warps split the
  // hidden dimension), then every CTA works out every token's picks
  if (with_router) {
    begin();
    const keepvq_router_logits_args& r = a.logits;
    const int pool = static_cast<int>(r.pool), first = pool * cta / grid, last = pool * (cta + 1) / grid;
    const int team = warp >> 3, part = warp & 7, chunks = static_cast<int>(r.hidden / 8);
    const __nv_bfloat16* w = static_cast<const __nv_bfloat16*>(r.router_w);
    const XT* x = static_cast<const XT*>(r.x);
#pragma unroll 1
    for (int e0 = first; e0 < last; e0 += 4)
#pragma unroll 1
      for (int t0 = 0; t0 < a.tokens; t0 += RL_TOKENS) {
        float acc[2][RL_TOKENS];
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int i = 0; i < RL_TOKENS; ++i) acc[q][i] = 0.0f;
        if (e0 + 2 * team < last) {
          const __nv_bfloat16* row0 = w + static_cast<int64_t>(e0 + 2 * team) * r.hidden;
          const __nv_bfloat16* row1 = w + static_cast<int64_t>(min(e0 + 2 * team + 1, last - 1)) * r.hidden;
#pragma unroll 1
          for (int c = part * 32 + lane; c < chunks; c += 256) {
            // all of a step's loads are in flight together (with a token's load in front of its sums, seven tokens took 9 us here)
            const uint4 raw0 = *reinterpret_cast<const uint4*>(row0 + c * 8), raw1 = *reinterpret_cast<const uint4*>(row1 + c * 8);
            uint4 raw[RL_TOKENS];
#pragma unroll
            for (int i = 0; i < RL_TOKENS; ++i)
              if (t0 + i < a.tokens) raw[i] = *reinterpret_cast<const uint4*>(x + static_cast<int64_t>(t0 + i) * r.hidden + c * 8);
            float w0[8], w1[8];
            load8_as_float<__nv_bfloat16>(reinterpret_cast<const __nv_bfloat16*>(&raw0), w0);
            load8_as_float<__nv_bfloat16>(reinterpret_cast<const __nv_bfloat16*>(&raw1), w1);
#pragma unroll
            for (int i = 0; i < RL_TOKENS; ++i)
              if (t0 + i < a.tokens) {
                float xv[8];
                load8_as_float<XT>(reinterpret_cast<const XT*>(&raw[i]), xv);
#pragma unroll
                for (int d = 0; d < 8; ++d) {
                  acc[0][i] = fmaf(xv[d], w0[d], acc[0][i]);
                  acc[1][i] = fmaf(xv[d], w1[d], acc[1][i]);
                }
              }
          }
        }
#pragma unroll
        for (int i = 0; i < RL_TOKENS; ++i) {
          if (t0 + i >= a.tokens) break;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            float v = acc[q][i];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
            if (lane == 0) logit_part[team][part][q * RL_TOKENS + i] = v;
          }
        }
        __syncthreads();
        if (tid < 4 * RL_TOKENS) {
          const int q = tid / RL_TOKENS, i = tid % RL_TOKENS;  // row e0 + q, token t0 + i
          if (e0 + q < last && t0 + i < a.tokens) {
            float v = 0.0f;
#pragma unroll
            for (int s = 0; s < 8; ++s) v += logit_part[q >> 1][s][(q & 1) * RL_TOKENS + i];
            r.logits[static_cast<int64_t>(t0 + i) * pool + e0 + q] = v / r.gate_temp;
          }
        }
        __syncthreads();
      }
    if (a.absent == 1 && cta == FT_ABSENT_CTA) return;
    ft_arrive(words_a, a.token);
  }
  // what needs no routing, while the others arrive (or, without a router, while the previous kernel
  // ends): the tables, from constants, and the rows of up to eight tokens
  build_nibble_tables(a0, a.codebook, tid, FT_THREADS);
  if (by_token) stage_rows(a.phase[0], a.tokens, lane);
  if (with_router) {
    if (!ft_wait(words_a, a.token, deadline, !two_phases)) return give_up();
    if (!two_phases) take_words_back();
    // ---- every CTA works out every token's picks (in the rings, which are still empty)
#pragma unroll 1
    for (int t0 = 0; t0 < a.tokens; t0 += FT_PICK_TOKENS) ft_pick(a.topk, base, t0, own_token, own_scores, route_slot, route_weight);
  } else {
    begin();
#pragma unroll 1
    for (int r = tid; r < a.routes; r += FT_THREADS) {
      route_slot[r] = a.slot[r];
      route_weight[r] = a.weight ? a.weight[r] : 1.0f;
    }
  }
  if (tid == 0) { n_groups_s = 0; n_due = 0; }
  __syncthreads();

  // ---- routes of one slot, at most `cap` (one, two or four) to a group, in order of the groups' first routes ----------
  {
    const bool mine = tid < a.routes && route_slot[tid] < static_cast<uint64_t>(a.slots);
    int seen = 0, total = 0, leader = 0;
    if (mine) {
      const uint32_t slot = route_slot[tid];
#pragma unroll 1
      for (int q = 0; q < a.routes; q += 4) {
        const uint4 four = *reinterpret_cast<const uint4*>(&route_slot[q]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool same = (i == 0 ? four.x : i == 1 ? four.y : i == 2 ? four.z : four.w) == slot && q + i < a.routes;
          if (same && q + i <= tid && (total & (cap - 1)) == 0) leader = q + i;
          seen += same && q + i < tid;
          total += same;
        }
      }
    }
    const bool leads = mine && leader == tid;
    const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, leads);
    if (lane == 0 && warp <= FT_MAX_ROUTES / 32) leaders_before[warp] = __popc(ballot);
    __syncthreads();
    int index = __popc(ballot & ((1u << lane) - 1u));
#pragma unroll 1
    for (int w = 0; w < warp && w <= FT_MAX_ROUTES / 32; ++w) index += leaders_before[w];
    if (leads) {
      grp_of_leader[tid] = index;
      grp_slot[index] = static_cast<int32_t>(route_slot[tid]);
      grp_size[index] = min(cap, total - seen);
      atomicAdd(&n_groups_s, 1);
    }
    __syncthreads();
    if (mine) grp_route[grp_of_leader[leader]][seen & (cap - 1)] = tid;
    __syncthreads();
  }
  // rows of routes without a slot, for the operators that promise zeros there
  if (a.dead_out)
#pragma unroll 1
    for (int r = cta; r < a.routes; r += grid)
      if (route_slot[r] >= static_cast<uint64_t>(a.slots)) {
        uint16_t* row = reinterpret_cast<uint16_t*>(static_cast<uint8_t*>(a.dead_out) + r * a.dead_row_bytes);
#pragma unroll 1
        for (int64_t i = tid; i < a.dead_row_bytes / 2; i += FT_THREADS) row[i] = 0;
      }

  // (what a phase derives from these is worked out again behind the sweep instead of kept through it: the
  // sweep needs all 128 registers, and a spilled one costs a trip to L2, shared memory taking all of L1)
  auto forgotten = [](int v) {
    asm volatile("" : "+r"(v));
    return v;
  };
#pragma unroll 1
  for (int ph = 0; ph < 2; ++ph) {
    if (!(a.parts & (ph == 0 ? FT_GATE_UP : FT_DOWN))) continue;
    const FewTokensPhase& P = a.phase[ph];
    const bool pair = ph == 0;
    const int unit_rows = pair ? 16 : 32;
    const int N = P.out_dim, n_chunks = P.n_chunks, chunks_per_group = P.chunks_per_group;
    const int units_per_group = P.units_per_group;
    const uint32_t units = static_cast<uint32_t>(n_groups_s * units_per_group);  // (times the grid: below 2^32, few_tokens_fits)
    const int u_begin = ft_div(units * cta, a.by_grid);
    const int n_units = ft_div(units * (cta + 1), a.by_grid) - u_begin;
    const int g0 = ft_div(u_begin, P.by_units), tile0 = u_begin - g0 * units_per_group;  // n_groups <= grid: the run spans at most two groups
    const int g_last = tile0 + n_units > units_per_group ? g0 + 1 : g0;
    const int tasks = n_units * n_chunks;
    const int task_first = tasks * warp / FT_WARPS, task_last = tasks * (warp + 1) / FT_WARPS;
    const int first_unit = ft_div(task_first, P.by_chunks), first_chunk = task_first - first_unit * n_chunks;

    // ---- the walk of the code fetches, ahead of the arithmetic -------------------------------------
    int f_left = task_last - task_first, f_chunk = first_chunk, f_group = g0, f_tile = tile0 + first_unit;
    if (f_tile >= units_per_group) { f_tile -= units_per_group; ++f_group; }
    const uint32_t row_bytes = static_cast<uint32_t>(n_chunks) * 64u;
    const uint64_t codes0 = reinterpret_cast<uint64_t>(P.codes[0]);
    const uint64_t sub_delta = pair ? reinterpret_cast<uint64_t>(P.codes[1]) - codes0 : 16u * row_bytes;  // (modulo 2^64)
    uint64_t f_ptr = 0;
    uint32_t f_off[RAGGED ? 4 : 1];  // to rows g + 8 s, where the last unit clamps them (a single matrix only)
    auto enter_unit = [&]() {
      int row = f_tile * unit_rows + g;
      if (RAGGED) {
        const int last_row = N - 1, row0 = min(row, last_row);
#pragma unroll
        for (int s = 1; s < 4; ++s) f_off[s] = static_cast<uint32_t>(min(row + 8 * s, last_row) - row0) * row_bytes;
        row = row0;
      }
      f_ptr = codes0 + (static_cast<uint64_t>(grp_slot[f_group]) * static_cast<uint64_t>(N) + static_cast<uint64_t>(row)) * row_bytes + static_cast<uint32_t>(t) * 16u;
    };
    if (f_left > 0) { enter_unit(); f_ptr += static_cast<uint32_t>(f_chunk) * 64u; }
    uint32_t stage = 0;  // of the ring: the next to be read, and then to be filled
    auto fetch = [&]() {
      if (f_left > 0) {
        const uint32_t dst = ring + stage;
#pragma unroll
        for (int s = 0; s < 4; ++s) ft_cp_async16(dst + s * 512, f_ptr + (s == 0 ? 0u : RAGGED ? f_off[s] : (s & 2 ? sub_delta : 0u) + (s & 1 ? 8u * row_bytes : 0u)));
        f_ptr += 64u;
        --f_left;
        if (++f_chunk == n_chunks) {
          f_chunk = 0;
          if (++f_tile == units_per_group) { f_tile = 0; ++f_group; }
          if (f_left > 0) enter_unit();
        }
      }
      stage = stage + FT_STAGE_BYTES == RING_BYTES ? 0u : stage + FT_STAGE_BYTES;
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll 1
    for (int i = 0; i < DEPTH; ++i) fetch();
    if (ph == 0 && (a.parts & FT_DOWN) && !RAGGED && warp == FT_WARPS - 1) {
      // the beginning of this CTA's share of the down codes, asked into L2: that phase starts with its reads under way
      const FewTokensPhase& D = a.phase[1];
      const uint32_t per_group = D.units_per_group, all = n_groups_s * per_group, unit_bytes = 32u * 64u * D.n_chunks;
      const uint32_t begin = ft_div(all * cta, a.by_grid), end = min(static_cast<uint32_t>(ft_div(all * (cta + 1), a.by_grid)), begin + FT_PREFETCH_BYTES / unit_bytes);
#pragma unroll 1
      for (uint32_t u = begin + lane; u < end; u += 32) {
        const uint32_t gi = ft_div(u, D.by_units);
        const uint64_t at = reinterpret_cast<uint64_t>(D.codes[0]) + (static_cast<uint64_t>(grp_slot[gi]) * per_group + (u - gi * per_group)) * unit_bytes;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(at), "r"(unit_bytes) : "memory");
      }
    }
    if (ph == 1 && (a.parts & FT_GATE_UP)) {
      const bool all_here = ft_wait(words_b, a.token, deadline, true);
      if (!all_here) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        return give_up();
      }
      take_words_back();
    }

    // ---- the activation rows of this CTA's (at most two) groups
    const bool staged = ph == 0 && by_token;
    auto row_of_route = [&](int route) { return P.x_div == 1 ? route : route / P.x_div; };
    const int first_rows = !staged && n_units > 0 ? grp_size[g0] : 0;  // staged rows of the first of them
    if (!staged) {
      const int group = lane < first_rows ? g0 : g_last, i = lane < first_rows ? lane : lane - first_rows;
      const int rows = g_last > g0 ? first_rows + grp_size[g_last] : first_rows;
      stage_rows(P, rows, lane < rows ? row_of_route(grp_route[group][i]) : 0);
    }
    const uint32_t row_stride = static_cast<uint32_t>(P.in_dim) * 2u + 64u;
    auto row_of = [&](int group, int i) { return staged ? row_of_route(grp_route[group][i]) : (group == g0 ? 0 : first_rows) + i; };

    // ---- the sweep ---------------------------------------------------------------------------------
    const void* const scales0 = P.scales[0];
    const void* const scales1 = pair ? P.scales[1] : P.scales[0];
    // y of one unit from its sums of 4 w x' times scale: lane (g, t) holds rows g and g + 8 of both tiles for route t of the group
    auto finish = [&](const float (&v)[4], int gi, int tile) {
      if (t >= grp_size[gi]) return;
      const int route = grp_route[gi][t];
      const float k = 0.25f * row_scale[row_of(gi, t)];
      const int64_t out_row = static_cast<int64_t>(route) * N;
      if (pair) {
        const float weight = route_weight[route];
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {  // round G and U to the activation dtype first, as the separate kernels of the reference do
          float gt = k * v[rr], up = k * v[2 + rr];
          if (std::is_same<XT, __half>::value) { gt = __half2float(__float2half_rn(gt)); up = __half2float(__float2half_rn(up)); }
          else { gt = __bfloat162float(__float2bfloat16_rn(gt)); up = __bfloat162float(__float2bfloat16_rn(up)); }
          if (a.swiglu_limit > 0.0f) { gt = fminf(gt, a.swiglu_limit); up = fminf(fmaxf(up, -a.swiglu_limit), a.swiglu_limit); }
          store_from_float(P.out, P.out_dtype, out_row + tile * 16 + g + 8 * rr, gt / (1.0f + expf(-gt)) * up * weight);
        }
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int row = tile * 32 + g + 8 * q;
          if (!RAGGED || row < N) store_from_float(P.out, P.out_dtype, out_row + row, k * v[q]);
        }
      }
    };
    float part[4] = {0.0f, 0.0f, 0.0f, 0.0f}, head[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    int even[2][4], odd[2][4], share = 0;  // [tile][row g | g + 8 x high | low plane of route t]
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int q = 0; q < 4; ++q) even[s][q] = odd[s][q] = 0;
    int unit = first_unit, chunk = first_chunk, gi = g0, tile = tile0 + first_unit;
    if (tile >= units_per_group) { tile -= units_per_group; ++gi; }
    int sg = ft_div(chunk, P.by_group_chunks), in_group = chunk - sg * chunks_per_group, open = 0;  // scale group, chunk within it, chunks since the sums were closed
    bool whole = first_chunk == 0, enter = true;
    uint32_t b_lane = 0;
    uint32_t sums = 0;
#pragma unroll 1
    for (int task = task_first; task < task_last; ++task) {
      if (enter) {  // a unit: its group's rows, and where its scales are
        enter = false;
        const int size = grp_size[gi];
        // column g of the MMA is (route g / 2, byte plane g % 2); a lane whose column carries no route
        // reads route 0's bytes (always there), and nothing ever looks at its column
        const int col = (g >> 1) < size ? (g >> 1) : 0;
        b_lane = acts + row_of(gi, col) * row_stride + t * 16 + (g & 1) * 8;
        sums = smem_addr(row_sums[row_of(gi, t < size ? t : 0)]);
      }
      asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");  // this chunk has landed
      uint4 cur[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) cur[s] = ft_lds128(ring + stage + s * 512);
      fetch();  // (a lane reads only what it fetched itself: the slot is free again)
      ++open;
      const bool close = in_group + 1 == chunks_per_group || open == FT_CLOSE_CHUNKS || task + 1 == task_last;
      float sc[4];  // rows g, g + 8 of the two tiles: asked for now, used behind the MMAs
      if (close) {
        const int64_t scale_row = static_cast<int64_t>(grp_slot[gi]) * N;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          int row = pair ? tile * 16 + g + 8 * (q & 1) : tile * 32 + g + 8 * q;
          if (RAGGED) row = min(row, N - 1);
          sc[q] = load_as_float(q < 2 ? scales0 : scales1, a.scales_dtype, (scale_row + row) * P.groups + sg);
        }
      }
      int chunk_sum;
      asm volatile("ld.shared.s32 %0, [%1];" : "=r"(chunk_sum) : "r"(sums + chunk * 4));
      share += chunk_sum;
      const uint32_t b_addr = b_lane + chunk * 512;
      ft_static_for<4>([&](auto index) {
        constexpr int I = decltype(index)::value;  // codewords 2 I and 2 I + 1 of the lane's eight
        const uint2 b0 = ft_lds64<2 * I * 64>(b_addr), b1 = ft_lds64<(2 * I + 1) * 64>(b_addr);
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const uint32_t lo = ft_word(cur[2 * s], I), hi = ft_word(cur[2 * s + 1], I);  // row g, row g + 8
          uint32_t e0, e1, e2, e3, o0, o1, o2, o3;
          decode_codeword_halves<false>(lo, abs_lane, sign_lane, e0, o0);
          decode_codeword_halves<false>(hi, abs_lane, sign_lane, e1, o1);
          decode_codeword_halves<true>(lo, abs_lane, sign_lane, e2, o2);
          decode_codeword_halves<true>(hi, abs_lane, sign_lane, e3, o3);
          ft_mma(even[s], e0, e1, e2, e3, b0.x, b1.x);
          ft_mma(odd[s], o0, o1, o2, o3, b0.y, b1.y);
        }
      });
      if (close) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          // 4 sum(w x') = 512 high + 2 low - 15 sum(x') of the operand u = q + 8, in wrapping 32-bit arithmetic, which the true value fits
          const int high = even[q >> 1][2 * (q & 1)] + (odd[q >> 1][2 * (q & 1)] >> 4), low = even[q >> 1][2 * (q & 1) + 1] + (odd[q >> 1][2 * (q & 1) + 1] >> 4);
          const int dot4 = static_cast<int>(static_cast<uint32_t>(high) * 512u + static_cast<uint32_t>(low) * 2u - 15u * static_cast<uint32_t>(share));
          part[q] = fmaf(sc[q], static_cast<float>(dot4), part[q]);
        }
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int q = 0; q < 4; ++q) even[s][q] = odd[s][q] = 0;
        share = 0;
        open = 0;
      }
      if (++in_group == chunks_per_group) { in_group = 0; ++sg; }
      if (++chunk == n_chunks) {
        if (whole) finish(part, gi, tile);
        else {
#pragma unroll
          for (int q = 0; q < 4; ++q) head[q] = part[q];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) part[q] = 0.0f;
        chunk = 0;
        sg = 0;
        whole = enter = true;
        ++unit;
        if (++tile == units_per_group) { tile = 0; ++gi; }
      }
    }
    // ---- units that several warps share: the partial sums meet in the (drained) ring of the warp they come
    // from, and the warp that ended the unit (each ends at most one that it did not begin) adds them up
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    if (task_first < task_last && chunk != 0) {  // the run ended inside a unit: in `part`
#pragma unroll
      for (int q = 0; q < 4; ++q) asm volatile("st.shared.f32 [%0], %1;" ::"r"(ring - lane * 12 + q * 128), "f"(part[q]) : "memory");
    }
    const bool ended = unit != first_unit;  // the unit the run began in
    __syncthreads();
    const int me = forgotten(warp), here = forgotten(cta);
    const uint32_t all_units = static_cast<uint32_t>(n_groups_s * units_per_group);
    const int run_first = ft_div(all_units * here, a.by_grid), run_tasks = (ft_div(all_units * (here + 1), a.by_grid) - run_first) * n_chunks;
    const int began = run_tasks * me / FT_WARPS, began_unit = ft_div(began, P.by_chunks);
    if (ended && began != began_unit * n_chunks) {  // ended a unit that it did not begin: in `head`
#pragma unroll 1
      for (int w = me - 1; w >= 0; --w) {
        const int begins = run_tasks * w / FT_WARPS;
        if (begins == run_tasks * (w + 1) / FT_WARPS) continue;  // fewer tasks than warps
        const uint32_t from = (w < low_rings ? base + w * RING_BYTES : high_rings + (w - low_rings) * RING_BYTES) + lane * 4;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float got;
          asm volatile("ld.shared.f32 %0, [%1];" : "=f"(got) : "r"(from + q * 128));
          head[q] += got;
        }
        if (begins <= began_unit * n_chunks) break;  // the one that began it
      }
      int gr = ft_div(run_first, P.by_units), tl = run_first - gr * units_per_group + began_unit;
      if (tl >= units_per_group) { tl -= units_per_group; ++gr; }
      finish(head, gr, tl);
    }
    if (ph == 0 && (a.parts & FT_DOWN)) {  // the hidden rows are written
      if (a.absent == 2 && cta == FT_ABSENT_CTA) return take_words_back();
      ft_arrive(words_b, a.token);
    } else __syncthreads();
    // the rings and the activation rows are free again
    if (ph == 0 && own_token >= 0 && own_token < a.tokens && warp == FT_WARPS - 1) {
      // the demanded picks of a token, which nothing here waits for
      uint32_t key[FT_TOPK_NPL], my_key, slot;
      int id[FT_TOPK_NPL], my_e;
      float weight;
#pragma unroll
      for (int i = 0; i < FT_TOPK_NPL; ++i) {
        id[i] = lane + 32 * i;
        key[i] = id[i] < a.topk.pool ? topk_key(a.topk.pool_bias, id[i], own_scores[id[i]]) : 0u;
      }
      topk_select<FT_TOPK_NPL>(key, id, a.top_k, lane, my_key, my_e);
      topk_finish(a.topk, own_token, lane, 1, my_e, lane < a.top_k ? own_scores[my_e] : 0.0f, true, slot, weight);
    }
  }

  // ---- the pick sum of a token's 32 columns, by the CTA that brought the last of its rows ------------
  if (a.parts & FT_COMBINE) {
    const FewTokensPhase& P = a.phase[1];
    auto store_out = [&](int64_t i, float v) {
      if (std::is_same<XT, __half>::value) static_cast<__half*>(a.out)[i] = __float2half_rn(v);
      else static_cast<__nv_bfloat16*>(a.out)[i] = __float2bfloat16_rn(v);
    };
    auto live_picks = [&](int tok) {
      int live = 0;
#pragma unroll 1
      for (int j = 0; j < a.top_k; ++j) live += route_slot[tok * a.top_k + j] < static_cast<uint64_t>(a.slots);
      return live;
    };
#pragma unroll 1
    for (int tok = cta; tok < a.tokens; tok += grid)
      if (live_picks(tok) == 0)  // nobody brings a row
#pragma unroll 1
        for (int d = tid; d < P.out_dim; d += FT_THREADS) {
          const int64_t i = static_cast<int64_t>(tok) * P.out_dim + d;
          store_out(i, a.shared ? a.shared[i] : 0.0f);
        }
    const int me = forgotten(cta), units_per_group = P.units_per_group;
    const uint32_t units = static_cast<uint32_t>(n_groups_s * units_per_group);
    const int u_begin = ft_div(units * me, a.by_grid), n_units = ft_div(units * (me + 1), a.by_grid) - u_begin;
    const int g0 = ft_div(u_begin, P.by_units), tile0 = u_begin - g0 * units_per_group;
#pragma unroll 1
    for (int i = tid; i < n_units * 4; i += FT_THREADS) {
      int tile = tile0 + (i >> 2), gi = g0;
      if (tile >= units_per_group) { tile -= units_per_group; ++gi; }
      if ((i & 3) >= grp_size[gi]) continue;
      const int tok = grp_route[gi][i & 3] / a.top_k;
      __threadfence();
      if (atomicAdd(&a.counters[tok * units_per_group + tile], 1u) + 1u == static_cast<uint32_t>(live_picks(tok))) {
        __threadfence();
        const int at = atomicAdd(&n_due, 1);
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(acts + at * 4), "r"(tok << 16 | tile) : "memory");
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int i = warp; i < n_due; i += FT_WARPS) {
      uint32_t due;
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(due) : "r"(acts + i * 4));
      const int tok = static_cast<int>(due >> 16), d = static_cast<int>(due & 0xFFFFu) * 32 + lane;
      float y = 0.0f;
      constexpr int AT_ONCE = 8;
#pragma unroll 1
      for (int j0 = 0; j0 < a.top_k; j0 += AT_ONCE) {  // a few rows in flight together, added in pick order
        uint16_t raw[AT_ONCE];
#pragma unroll
        for (int j = 0; j < AT_ONCE; ++j) {
          const int r = tok * a.top_k + j0 + j;
          if (j0 + j < a.top_k && route_slot[r] < static_cast<uint64_t>(a.slots))
            asm volatile("ld.global.cg.u16 %0, [%1];" : "=h"(raw[j]) : "l"(static_cast<const uint16_t*>(P.out) + static_cast<int64_t>(r) * P.out_dim + d) : "memory");
        }
#pragma unroll
        for (int j = 0; j < AT_ONCE; ++j) {
          const int r = tok * a.top_k + j0 + j;
          if (j0 + j < a.top_k && route_slot[r] < static_cast<uint64_t>(a.slots))
            y += std::is_same<XT, __half>::value ? __half2float(__ushort_as_half(raw[j])) : __uint_as_float(static_cast<uint32_t>(raw[j]) << 16);
        }
      }
      const int64_t o = static_cast<int64_t>(tok) * P.out_dim + d;
      if (a.shared) y += a.shared[o];
      store_out(o, y);
    }
  }
  // ---- the others' words are back: nobody waits on the first CTA's any more ----------------------------
  if (cta == 0 && (with_router || two_phases)) {
    uint64_t* const words = two_phases ? words_b : words_a;
    const uint64_t late = deadline + a.wait_ns;  // (a CTA that does not see the word gives up by its own deadline and takes its word back all the same)
    int ok = 1;
    for (int i = 1 + tid; i < grid && ok; i += FT_THREADS) ok = ft_poll(words + i, a.token, late, true);
    if (!__syncthreads_and(ok) && a.status && tid == 0) atomicExch(a.status, 1);
    if (tid == 0) ft_clear(words + FT_MAX_CTAS);
  }
}

// ---- launch -----------------------------------------------------------------------------------

// CTAs of a launch on the current device, one per SM; 0 where a grid of them cannot be launched cooperatively.
// (Of the device; a stream may have only part of its SMs, see stream_sms.)
static int few_tokens_grid() {
  static std::atomic<int> known[64];  // plus one; 0: not asked yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  if (dev < 0 || dev >= 64) return 0;
  int grid = known[dev].load() - 1;
  if (grid >= 0) return grid;
  int sms = 0, cooperative = 0, smem = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  grid = cooperative && smem >= static_cast<int>(FT_SMEM_BYTES + FT_STATIC_MAX - 1024) ? std::min(sms, FT_MAX_CTAS) : 0;  // (1 KB of that is the system's)
  known[dev].store(grid + 1);
  return grid;
}
// SMs that the stream's kernels may run on: a green context's are part of the device's.  Asked before a
// cooperative launch, because a launch refused as too large ends a capture under way.
static int stream_sms(cudaStream_t s, int device_sms) {
  struct Driver {
    CUresult(CUDAAPI* stream_green)(CUstream, CUgreenCtx*) = nullptr;
    CUresult(CUDAAPI* green_resource)(CUgreenCtx, CUdevResource*, CUdevResourceType) = nullptr;
    CUresult(CUDAAPI* current)(CUcontext*) = nullptr;
    CUresult(CUDAAPI* resource)(CUcontext, CUdevResource*, CUdevResourceType) = nullptr;
    bool known = false;
    Driver() {
      auto find = [](const char* name, auto& fn) {
        void* at = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint(name, &at, cudaEnableDefault, &found) != cudaSuccess) {
          cudaGetLastError();
          return false;
        }
        fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(at);
        return found == cudaDriverEntryPointSuccess && at;
      };
      known = find("cuStreamGetGreenCtx", stream_green) && find("cuGreenCtxGetDevResource", green_resource) && find("cuCtxGetCurrent", current) && find("cuCtxGetDevResource", resource);
    }
  };
  static const Driver driver;
  if (!driver.known) return device_sms;
  CUdevResource r = {};
  CUgreenCtx green = nullptr;
  CUcontext context = nullptr;
  const bool asked = driver.stream_green(s, &green) == CUDA_SUCCESS && green ? driver.green_resource(green, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS
                   : driver.current(&context) == CUDA_SUCCESS && context && driver.resource(context, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS;
  return asked && r.type == CU_DEV_RESOURCE_TYPE_SM ? static_cast<int>(r.sm.smCount) : device_sms;
}
bool few_tokens_fits(int64_t routes, int64_t tokens, int64_t slots, int64_t out_dim, int64_t in_dim, int64_t groups) {
  // (a CTA's share of the units must not span more than two route groups: no more routes than CTAs)
  return routes > 0 && slots * out_dim < (int64_t{1} << 31) - 64 && routes <= FT_MAX_ROUTES && tokens <= FT_MAX_TOKENS && in_dim <= FT_MAX_IN && out_dim > 0 && out_dim < (1 << 18) && shapes_supported(out_dim, in_dim, groups) &&
         routes <= few_tokens_grid();
}
int64_t few_tokens_sync_bytes(int64_t tokens, int64_t out_dim) { return 2 * 8 * FT_BARRIER_WORDS + tokens * (out_dim / 32) * 4; }
bool few_tokens_router_fits(const keepvq_router_logits_args& l, const keepvq_routed_topk_args& t) {
  return l.router_dtype == KEEPVQ_BF16 && l.pool <= 32 * FT_TOPK_NPL && l.hidden % 8 == 0 && t.top_k <= 16 && t.top_k <= l.pool && l.gate_temp > 0.0f &&
         t.score_func >= KEEPVQ_SCORE_SOFTMAX && t.score_func <= KEEPVQ_SCORE_SQRT_SOFTPLUS && aligned_to(l.x, 16) && aligned_to(l.router_w, 16);
}

// A token for the barrier words that no other launch of this or an earlier process is likely to have left
// behind: counted on from where and when the library came to be here (nothing that may throw: the callers are C).
static uint64_t next_token() noexcept {
  static char here;
  static std::atomic<uint64_t> next{(static_cast<uint64_t>(std::chrono::steady_clock::now().time_since_epoch().count()) * 0xD1342543DE82EF95ull) ^ reinterpret_cast<uintptr_t>(&here)};
  uint64_t z = next.fetch_add(0x9E3779B97F4A7C15ull, std::memory_order_relaxed);
  z ^= z >> 32;
  return z | 1u;  // (zero marks a clear word)
}

template <typename XT, bool RAGGED, int DEPTH>
static int launch_few_tokens(const FewTokensArgs& args, void* sync, cudaStream_t s) {
  auto kernel = few_tokens_kernel<XT, RAGGED, DEPTH>;
  static std::atomic<uint64_t> configured{0};  // one bit per device: the shared-memory opt-in is a per-device attribute of the function
  int dev = 0;
  cudaGetDevice(&dev);
  const int ctas = args.ctas ? args.ctas : few_tokens_grid();
  if (args.routes > ctas || dev < 0 || dev >= 64) return KEEPVQ_ERR_UNSUPPORTED;
  if (!((configured.load() >> dev) & 1ull)) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FT_SMEM_BYTES);
    if (e != cudaSuccess) return note_cuda_error(e);
    configured.fetch_or(1ull << dev);
  }
  FewTokensArgs a = args;
  for (FewTokensPhase& p : a.phase) {
    if (!p.out_dim) continue;
    const int unit_rows = p.codes[1] ? 16 : 32;
    p.n_chunks = p.in_dim / 256;
    p.chunks_per_group = p.n_chunks / p.groups;
    p.units_per_group = (p.out_dim + unit_rows - 1) / unit_rows;
    p.by_chunks = ft_divisor(p.n_chunks);
    p.by_units = ft_divisor(p.units_per_group);
    p.by_group_chunks = ft_divisor(p.chunks_per_group);
  }
  a.by_grid = ft_divisor(ctas);
  if (!a.token) a.token = next_token();
  if (!a.wait_ns) a.wait_ns = FT_WAIT_NS;
  a.barrier_words = static_cast<uint64_t*>(sync);
  a.counters = reinterpret_cast<uint32_t*>(static_cast<uint64_t*>(sync) + 2 * FT_BARRIER_WORDS);
  cudaLaunchConfig_t config = {};
  config.gridDim = static_cast<unsigned>(ctas);
  config.blockDim = FT_THREADS;
  config.dynamicSmemBytes = FT_SMEM_BYTES;
  config.stream = s;
  cudaLaunchAttribute attribute = {};
  if ((a.parts & FT_ROUTER) || ((a.parts & FT_GATE_UP) && (a.parts & FT_DOWN))) {  // its CTAs wait for one another: all of them resident
    if (stream_sms(s, ctas) < ctas) return KEEPVQ_ERR_UNSUPPORTED;
    attribute.id = cudaLaunchAttributeCooperative;
    attribute.val.cooperative = 1;
  } else {
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
  }
  config.attrs = &attribute;
  config.numAttrs = 1;
  const cudaError_t err = cudaLaunchKernelEx(&config, kernel, a);
  if (err == cudaErrorCooperativeLaunchTooLarge) {  // nothing was launched, and the caller has kernels whose blocks do not wait for one another
    cudaGetLastError();
    return KEEPVQ_ERR_UNSUPPORTED;
  }
  return err == cudaSuccess ? KEEPVQ_OK : note_cuda_error(err);
}

// Bytes of activation rows that fit beside rings of `depth` chunks.
static int64_t act_room(int depth) {
  const uint32_t ring = depth * FT_STAGE_BYTES;
  const int low = static_cast<int>((64 * 1024 - FT_STATIC_MAX) / ring);
  return static_cast<int64_t>(FT_SMEM_BYTES + FT_STATIC_MIN) - (64 * 1024 + FT_TABLE_BYTES + (FT_WARPS - low) * ring);
}
template <typename XT, bool RAGGED>
static int launch_depth(const FewTokensArgs& a, void* sync, cudaStream_t s) {
  // one or two tokens have few chunks a warp and wait for memory between them: the deeper ring that their
  // few activation rows leave room for; the more rows, the shallower
  if (a.act_bytes <= act_room(4)) return launch_few_tokens<XT, RAGGED, 4>(a, sync, s);
  if (a.act_bytes <= act_room(3)) return launch_few_tokens<XT, RAGGED, 3>(a, sync, s);
  if (a.act_bytes <= act_room(2)) return launch_few_tokens<XT, RAGGED, 2>(a, sync, s);
  return KEEPVQ_ERR_UNSUPPORTED;
}
int few_tokens(const FewTokensArgs& args, int32_t x_dtype, void* sync, cudaStream_t s) {
  const bool ragged = args.phase[1].out_dim % 32 != 0;
  if (ragged && (args.parts & (FT_GATE_UP | FT_COMBINE))) return KEEPVQ_ERR_UNSUPPORTED;
  FewTokensArgs a = args;
  // no more routes of an expert than tokens, but for a table that names a slot twice: those are groups of their own then
  a.group_shift = a.tokens <= 1 ? 0 : a.tokens == 2 ? 1 : 2;
  const int64_t by_group = 2ll << a.group_shift, by_token = (a.parts & FT_ROUTER) && a.tokens <= FT_ROWS ? a.tokens : by_group;
  int64_t bytes = 0;
  if (a.parts & FT_GATE_UP) bytes = by_token * (2 * a.phase[0].in_dim + 64);
  if (a.parts & FT_DOWN) bytes = std::max<int64_t>(bytes, by_group * (2 * a.phase[1].in_dim + 64));
  a.act_bytes = static_cast<uint32_t>(bytes);
  if (x_dtype == KEEPVQ_F16) return ragged ? launch_depth<__half, true>(a, sync, s) : launch_depth<__half, false>(a, sync, s);
  if (x_dtype == KEEPVQ_BF16) return ragged ? launch_depth<__nv_bfloat16, true>(a, sync, s) : launch_depth<__nv_bfloat16, false>(a, sync, s);
  return KEEPVQ_ERR_DTYPE;
}

}  // namespace fast
}  // namespace keepvq
