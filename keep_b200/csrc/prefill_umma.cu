// Expert-grouped projections for many tokens per expert (prefill) on the 5th-generation tensor
// cores: tcgen05.mma kind::i8 with both the A operand and the accumulators in tensor memory.
//
// Stands in for the reference's expert-block prefill kernels
// (native/vq_nax_ext/kernels/nax_fp16_matmul.metal:904-1062,11562-11674 and
// src/ramp/kernels/gather_vqmm.py:690-928): routes sorted by expert, codes decoded inside the
// kernel into operand tiles, a dense contraction per (expert, row tile).
//
// Arithmetic: the same exact-integer form as the decode kernels (moe_fast.cuh).  A codeword
// becomes eight int8 values q with 4w = 2q + 1; activations are 16-bit fixed point split in a
// signed high and a signed low byte.  Per (expert, 128 output rows, up to 48 or 96 routes):
//   [D_hi | D_lo][128 x 2N] += Q[128 x K] * [Xhi ; Xlo][2N x K]^T   (int32, exact, in TMEM)
//   y = scale_row * scale_x * (0.5 * (256 D_hi + D_lo) + 0.25 * sum(x'))
// The weights are the M operand (128 rows per tile) and the routes the N operand (their high-byte
// rows stacked on their low-byte rows, so one MMA reads the decoded tile once for both), so a
// ragged expert group costs at most 15 padded columns, and a code is decoded once per 48 or 96 routes.
//
// What bounds this kernel is turning codes into int8 operands: seven instructions and two 4-byte
// table reads per codeword and lane, 16 warps wide.  The roles are cut so that those warps do little
// else and rarely wait for one another:
//   warps 0-15   decode, and drain one segment behind.  A thread's row of the tile is its lane of
//                tensor memory (warp w reaches lanes 32 * (w % 4) ...).  Four warps decode one K block
//                (16 codewords per thread) of one tile; warps 0-3 take the even and 4-7 the odd K
//                blocks of an item's first tile, warps 8-11 and 12-15 those of the second, so a warp
//                pays its waits, its store to tensor memory and its arrivals once per 16 codewords
//                and has the time of two K blocks for them.  (All 16 warps on every K block, eight
//                codewords each behind private cp.async rings, took 1290 cycles per K block at 24
//                routes an expert; this form 740: a 1024-token product 302 -> 180 us, the two
//                projections of a 4096-token layer 1185 + 584 -> 715 + 367 us, 736 + 400 on another GPU.)  The bytes go straight into TENSOR MEMORY
//                (tcgen05.st), two stages of one or two K blocks deep, so the A operand never touches shared memory.
//                An item's accumulators are drained (tcgen05.ld: same lanes; each of the four warps
//                of a quadrant takes a quarter of the columns) behind the warp's first K block of the
//                NEXT item, so nobody waits for the tail of the MMAs.
//   warp  16     issues the MMAs: A from tensor memory, B from shared memory.
//   warp  17     one thread brings the routes' quantised activations into the B tiles with TMA: the
//                rows were quantised in grouped order, so a group's high bytes and its low bytes are
//                two runs of rows of one [2 x rows, K] byte matrix, and a K block of them is a handful
//                of cp.async.bulk.tensor.2d boxes of 16 rows x 128 bytes that land swizzled, ready
//                for the MMA; the boxes report to the stage's mbarrier (expect_tx / complete_tx).
//   warp  18     one thread brings the codes with TMA: boxes of 128 rows x 64 bytes (two K blocks of
//                a tile), 64-byte swizzle, so a thread reads its row's 32 bytes without bank conflicts.
//   warp  19     gathers what the drain needs per route (route id, activation scale and sums, gate weight).
// mbarrier full/empty pairs carry every dependency.  Every wait is bounded by a deadline on the
// global timer: on expiry the CTA raises a flag in `status`, stops issuing work, waits (bounded)
// for the MMAs and the copies in flight, frees its tensor memory and returns.
#include "async_copy.cuh"
#include "moe_fast.cuh"

namespace keepvq {
namespace fast {

constexpr int PF_DECODE_WARPS = 16;
constexpr int PF_MMA_WARP = PF_DECODE_WARPS;
constexpr int PF_B_WARP = PF_DECODE_WARPS + 1;     // activations by TMA
constexpr int PF_CODE_WARP = PF_DECODE_WARPS + 2;  // codes by TMA
constexpr int PF_INFO_WARP = PF_DECODE_WARPS + 3;  // per-route facts
constexpr int PF_THREADS = (PF_DECODE_WARPS + 4) * 32;  // 640
constexpr int PF_MAX_SEGMENTS = 32;             // most scale groups of a row
constexpr int64_t PF_MAX_SEGMENT_INPUTS = 4096; // ... and most inputs of one, where a row has several: sum(4w x') fits 32 bits
// One scale group per row, |u - 8| <= 8 for any table and |x'| <= 32639: sum(q x') fits 32 bits up to here ...
constexpr int64_t PF_EXACT32_INPUTS = 8192;
// ... and the two byte planes' sums and sum(x'), which meet in 64 bits beyond that, up to MAX_GROUP_INPUTS.
static_assert(8 * 32639 * PF_EXACT32_INPUTS < (int64_t{1} << 31) && 16 * 32639 * PF_MAX_SEGMENT_INPUTS < (int64_t{1} << 31), "");
static_assert(15 * 128 * MAX_GROUP_INPUTS < (int64_t{1} << 31), "");
constexpr int PF_ROWS = 128;                    // output rows per tile
constexpr int PF_KBLOCK_CODES = 16;             // codewords of a row per K block = 128 bytes of int8
constexpr int PF_A_TILE_COLS = PF_KBLOCK_CODES * 2;   // a decoded K block of one tile: 128 bytes per row = 32 columns
constexpr uint32_t PF_TMEM_COLS = 512;
constexpr uint32_t PF_TABLE_BYTES = 64 * 1024;  // the nibble decoder's two tables, interleaved (moe_fast.cuh)
// Shared window, absolute addresses (compile-time constants: the operands of the MMAs, copies and
// barriers are then immediates); a block whose window lies elsewhere reports and does nothing.
constexpr uint32_t PF_A0 = 64 * 1024;           // the 64 KB boundary the tables sit on
constexpr uint32_t PF_LOW_BYTES = 48 * 1024;    // what lies below the tables: B stages
constexpr uint32_t PF_BARS = PF_A0 - PF_LOW_BYTES - 1024;  // the mbarriers, below those
constexpr int PF_INFO_BUFFERS = 3;
constexpr int PF_SMEM_BYTES = 222 * 1024;       // dynamic request: reaches A0 + 160 KB behind the 3 to 5 KB of static and reserved shared memory
constexpr uint64_t PF_DEFAULT_WAIT_NS = 2000000000ull;

// What a kernel that takes up to N_MAX routes per item keeps in tensor memory and shared memory.
// Tensor memory (512 columns): per accumulator set 2 byte planes x M tiles x N_MAX columns, the rest
// decoded A stages of 32 columns per tile.  With several scale groups per row the accumulators are
// drained once per group, so there are two sets; with one, a single set leaves room for more A stages.
// Shared window: [A0 - 48 KB, A0) the first B stages | [A0, +64 KB) tables | code stages | the other B stages
template <int M, int N_MAX, bool GROUPED, int BITS>
struct PrefillPlan {
  static_assert(N_MAX % 16 == 0, "an item's routes pad to a multiple of sixteen columns");
  static constexpr uint32_t ACC_SET_COLS = 2 * M * N_MAX;
  static constexpr uint32_t ACC_SETS = GROUPED ? 2 : 1;
  // K blocks per stage: what the MMA warp pays once per stage (its wait, its commits, the instructions
  // around them: some 300 cycles alone, 550 to 700 beside the decode warps) is what a K block of few routes
  // takes, so where tensor memory has room for two stages of two K blocks they go in pairs (1000-token layer:
  // gate/up and down 534 + 297 -> 525 + 289 us; 24 tokens of 8-bit codes 91.7 -> 87.9)
  static constexpr uint32_t STAGE_BLOCKS = GROUPED || N_MAX > 48 ? 1 : 2;
  // The fp32 sums of the scale groups leave no registers for a K block's 32 operand columns at once: in halves, and
  // with the deadline in shared memory, nothing spills (layer of 1021 tokens: 631 + 448 -> 617 + 427 us)
  static constexpr bool HALVES = GROUPED;
  static constexpr uint32_t A_BLOCK_COLS = M * PF_A_TILE_COLS;
  static constexpr uint32_t A_STAGE_COLS = STAGE_BLOCKS * A_BLOCK_COLS;
  static constexpr uint32_t A_COL0 = ACC_SETS * ACC_SET_COLS;
  static constexpr uint32_t A_STAGES = 2;
  static_assert(A_COL0 + A_STAGES * A_STAGE_COLS <= PF_TMEM_COLS, "tensor memory holds the accumulators and the A stages");
  static constexpr uint32_t B_BLOCK_BYTES = 2 * N_MAX * 128;  // a K block: high-byte rows of the routes, then their low-byte rows
  static constexpr uint32_t B_STAGE_BYTES = STAGE_BLOCKS * B_BLOCK_BYTES;
  static constexpr uint32_t LOW_B_STAGES = PF_LOW_BYTES / B_STAGE_BYTES;
  static constexpr uint32_t B_STAGES = GROUPED ? 6 : 4;    // one ring of barriers for A and B: a stage's A columns are its index modulo A_STAGES
  static_assert(B_STAGES % A_STAGES == 0, "");
  static constexpr uint32_t CODE_ROW_BYTES = 2 * PF_KBLOCK_CODES * BITS / 8;  // two K blocks of a row's codes
  static constexpr uint32_t CODE_UNIT_BYTES = PF_ROWS * CODE_ROW_BYTES;       // ... of a tile's
  static constexpr uint32_t CODE_STAGE_BYTES = M * CODE_UNIT_BYTES;
  static constexpr uint32_t CODE_STAGES = BITS == 16 ? 3 : 6;
  static constexpr uint32_t SUMS_OFFSET = PF_TABLE_BYTES + CODE_STAGES * CODE_STAGE_BYTES + (B_STAGES - LOW_B_STAGES) * B_STAGE_BYTES;
  static constexpr uint32_t SUMS = PF_A0 + SUMS_OFFSET;  // [item buffers][segments][routes]: what comes off the segment's integer sums
  static constexpr uint32_t HIGH_BYTES = SUMS_OFFSET + (GROUPED ? PF_INFO_BUFFERS * PF_MAX_SEGMENTS * N_MAX * 4 : 0);
  static_assert(HIGH_BYTES <= 160 * 1024, "the window above A0");
  static constexpr uint32_t CODE_BASE = PF_A0 + PF_TABLE_BYTES;
  static constexpr __host__ __device__ uint32_t b_stage(uint32_t stage) {
    return stage < LOW_B_STAGES ? PF_A0 - PF_LOW_BYTES + stage * B_STAGE_BYTES : CODE_BASE + CODE_STAGES * CODE_STAGE_BYTES + (stage - LOW_B_STAGES) * B_STAGE_BYTES;
  }
};

__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// One arrival for the warp, predicated instead of a branch.
__device__ __forceinline__ void mbar_arrive_warp(uint32_t bar, int lane) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar), "r"(lane) : "memory");
}
// Wait of a whole warp, bounded by time.  Returns false (in every lane) when the deadline passes (the
// caller's CTA then gives up: the flag is raised for every role) or when another warp of the CTA
// already gave up.  RELAXED is for the loaders, which run stages ahead: their polls would take issue
// slots from the decode warps.
template <bool RELAXED = false, class Time>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const Time& deadline, volatile int* abort_flag) {
  for (uint32_t spin = 0;; ++spin) {
    if (__all_sync(0xFFFFFFFFu, mbar_complete(bar, parity))) return true;
    if (RELAXED) __nanosleep(160);
    if ((spin & 31u) == 31u) {
      if (__any_sync(0xFFFFFFFFu, *abort_flag)) return false;
      if (__any_sync(0xFFFFFFFFu, global_timer_ns() > deadline)) { *abort_flag = 1; return false; }
    }
  }
}
// A value that is the same in every lane, in a form the compiler knows to be (the result of a warp
// reduction): what depends on it (loop bounds, descriptors of MMAs and copies) then lives in uniform
// registers.
__device__ __forceinline__ uint32_t warp_uniform(uint32_t v) { return __reduce_or_sync(0xFFFFFFFFu, v); }
// The wait of a CTA that has given up, for what it still has in flight: bounded by 100 ms.
__device__ __forceinline__ void mbar_wait_grace(uint32_t bar, uint32_t parity) {
  const uint64_t grace = global_timer_ns() + 100000000ull;
  for (uint32_t spin = 0; spin < (1u << 22); ++spin) {
    if (mbar_complete(bar, parity) || ((spin & 31u) == 31u && global_timer_ns() > grace)) return;
  }
}
// A CTA that gives up waits for the copies of its code loader (`used` stage fills) before its shared memory goes.
template <uint32_t STAGES>
__device__ __forceinline__ void wait_codes_landed(uint32_t full_bars, uint32_t used) {
  for (uint32_t i = used > STAGES ? used - STAGES : 0; i < used; ++i) mbar_wait_grace(full_bars + 8u * (i % STAGES), (i / STAGES) & 1u);
}
// ... and for those of its activation loader (`used` stages).  A stage's barrier also counts the
// decode warps that fill its A columns (every other stage a warp's own with one K block a stage, all with
// two), so the arrivals they did not come to make are made for them:
// place[w] is where decode warp w stopped, its next stage modulo 2 STAGES.  A stage whose barrier
// is not complete has not been read, so no decode warp is as far as STAGES beyond it, none STAGES behind.
template <uint32_t STAGES, int STAGE_BLOCKS>
__device__ __forceinline__ void wait_activations_landed(uint32_t full_bars, uint32_t used, const uint32_t* place, int decode_warps) {
  for (uint32_t i = used > STAGES ? used - STAGES : 0; i < used; ++i) {
    const uint32_t bar = full_bars + 8u * (i % STAGES), phase = (i / STAGES) & 1u;
    if (mbar_complete(bar, phase)) continue;
    for (int w = 0; w < decode_warps; ++w) {
      const uint32_t ahead = (place[w] + 2 * STAGES - i % (2 * STAGES)) % (2 * STAGES);  // its next stage less this one
      if ((STAGE_BLOCKS == 2 || ((static_cast<uint32_t>(w) >> 2) & 1u) == (i & 1u)) && (ahead == 0 || ahead > STAGES)) mbar_arrive(bar);
    }
    mbar_wait_grace(bar, phase);
  }
}

// K-major SWIZZLE_128B operand tile: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc(uint32_t tile_addr) {
  return static_cast<uint64_t>((tile_addr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// A operand in tensor memory: row m of the tile in lane m, K packed along the columns (four int8 per column).  B: shared-memory descriptor.
__device__ __forceinline__ void umma_i8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
               ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// 32 consecutive columns of this thread's lane of tensor memory.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
               "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
                 "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]),
                 "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]) : "memory");
}
// ... and 16.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
                 "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr) : "memory");
}

__device__ __forceinline__ void tma_box_3d(uint32_t dst, const CUtensorMap* map, int32_t x, int32_t y, int32_t z, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
               ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
// Place in a ring of STAGES stages: every role walks its rings on its own, an index and a phase bit.
template <uint32_t STAGES>
struct RingPlace {
  uint32_t index = 0, phase = 0;
  __device__ __forceinline__ void advance(uint32_t by = 1) {
    index += by;
    if (index >= STAGES) { index -= STAGES; phase ^= 1u; }
  }
};

// GLU: the M = 2 A tiles are the gate and the up matrix over the same 128 rows, fused by SwiGLU.
// !GLU: the M tiles are consecutive 128-row tiles of one matrix, so an item covers 128 * M rows
// and its activation (B) stages serve all of them (the copies are what bounds a single projection).
// GROUPED: several scale groups per row.  The accumulators are drained once per group (a segment of
// the K blocks) into fp32 sums that the drain warps keep in registers.
// BITS: 16-bit E8P codes, or 8-bit codes of a table whose word holds dim d in nibble d, value
// (nibble - 8) / 2.  There a codeword is ONE table read, w = q / 2 without the quarter, and any table
// will do (the integer sums are bounded for |q| <= 8, not for the shipped table's codewords).
// `stall` != 0 is the wait self-test: a loader never publishes, or the per-route facts come only after
// somebody gave up, and a wait runs into the deadline.
enum { STALL_ACTIVATIONS = 1, STALL_CODES = 2, STALL_FACTS = 3 };
// Boxes over the activations, one map per padded number of routes: [2 planes][16 (i + 1) rows][128 bytes].
template <int N_MAX>
struct ActivationMaps { CUtensorMap rows[N_MAX / 16]; };

// WIDE: one scale group of more than PF_EXACT32_INPUTS inputs, whose sums meet in 64 bits (as a branch
// inside the drain that cost the other calls 1 to 2 %).
template <int M, bool GLU, int N_MAX, bool GROUPED, int BITS, bool WIDE>
__global__ void __launch_bounds__(PF_THREADS, 1) prefill_projection_kernel(FastProjectionArgs p, const __grid_constant__ ActivationMaps<N_MAX> x_maps, const __grid_constant__ CUtensorMap a_map,
                                                                           const __grid_constant__ CUtensorMap b_map, int32_t* status, int stall, uint64_t wait_ns) {
  using Plan = PrefillPlan<M, N_MAX, GROUPED, BITS>;
  constexpr int ITEM_ROWS = GLU ? PF_ROWS : PF_ROWS * M;
  constexpr int A_STAGES = Plan::A_STAGES, B_STAGES = Plan::B_STAGES, CODE_STAGES = Plan::CODE_STAGES, ACC_SETS = Plan::ACC_SETS;
  constexpr int SB = Plan::STAGE_BLOCKS;
  constexpr int TILE_STEP = GLU ? 0 : PF_ROWS;  // rows between the A tiles of an item
  extern __shared__ __align__(16) uint8_t smem_raw[];
  grid_launch_dependents();
  // STAGE_FULL: the decode warps' A tiles and the activations of a stage's K blocks are in place; STAGE_EMPTY: its MMAs have read them
  enum { STAGE_FULL = 0, STAGE_EMPTY = STAGE_FULL + B_STAGES, CODE_FULL = STAGE_EMPTY + B_STAGES, CODE_EMPTY = CODE_FULL + CODE_STAGES,
         ACC_FULL = CODE_EMPTY + CODE_STAGES, ACC_EMPTY = ACC_FULL + ACC_SETS, INFO_FULL = ACC_EMPTY + ACC_SETS, INFO_EMPTY = INFO_FULL + PF_INFO_BUFFERS, DRAINED = INFO_EMPTY + PF_INFO_BUFFERS, N_BARS = DRAINED + 1 };
  static_assert(N_BARS * 8 <= 1024, "");
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ volatile uint64_t shared_deadline;  // (in registers it and 64-bit row numbers made the scale-group form spill, 500 cycles of reloads from L2 per K block)
  __shared__ uint32_t decode_place[PF_DECODE_WARPS], codes_issued, activations_issued;  // where the roles stopped
  __shared__ int4 route_info[PF_INFO_BUFFERS][N_MAX];  // per item (three in flight): route, x scale, x sum (one scale group only), gate weight
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto bar = [](int which, uint32_t index) { return PF_BARS + 8u * (static_cast<uint32_t>(which) + index); };

  const uint32_t dyn_base = smem_addr(smem_raw);
  const bool window_ok = dyn_base <= PF_BARS && PF_A0 + Plan::HIGH_BYTES <= dyn_base + PF_SMEM_BYTES;  // uniform over the grid

  // ---- set-up: tables, barriers, tensor memory ------------------------------------------------
  if (window_ok) {
    if (BITS == 16) build_nibble_tables(PF_A0, p.codebook, tid, PF_THREADS);
    else build_byte_code_table(PF_A0, p.codebook, tid, PF_THREADS);
  }
  if (tid == 0) {
    abort_flag = window_ok ? 0 : 1;
    if (window_ok) {
      for (int s = 0; s < B_STAGES; ++s) { mbar_init(bar(STAGE_FULL, s), M * 4 * SB + 1); mbar_init(bar(STAGE_EMPTY, s), 1); }
      for (int s = 0; s < CODE_STAGES; ++s) { mbar_init(bar(CODE_FULL, s), 1); mbar_init(bar(CODE_EMPTY, s), M * 8); }
      for (int s = 0; s < ACC_SETS; ++s) { mbar_init(bar(ACC_FULL, s), 1); mbar_init(bar(ACC_EMPTY, s), PF_DECODE_WARPS); }
      for (int s = 0; s < PF_INFO_BUFFERS; ++s) { mbar_init(bar(INFO_FULL, s), 1); mbar_init(bar(INFO_EMPTY, s), PF_DECODE_WARPS); }
      mbar_init(bar(DRAINED, 0), 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == PF_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_slot)), "r"(PF_TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const bool set_up_ok = window_ok && tmem_base_slot == 0;  // uniform over the block
  if (!set_up_ok && tid == 0) abort_flag = 1;
  // an allocation of all 512 columns starts at column 0 of lane 0: a constant, which keeps the MMAs' operands in uniform registers
  constexpr uint32_t tmem = 0;
  grid_wait();  // the tables come from constants; everything below reads what the kernels before this one wrote
  const uint64_t own_deadline = global_timer_ns() + (wait_ns ? wait_ns : PF_DEFAULT_WAIT_NS);  // (the time spent waiting for those is not this kernel's)
  if constexpr (GROUPED) {
    if (tid == 0) shared_deadline = own_deadline;
    __syncthreads();
  }
  const auto& deadline = [&]() -> const auto& {
    if constexpr (GROUPED) return shared_deadline; else return own_deadline;
  }();

  const int N_out = static_cast<int>(p.out_dim);  // (slots * out_dim is below 2^31, prefill_supported)
  const int k_blocks = static_cast<int>(p.in_dim / (8 * PF_KBLOCK_CODES));
  const int code_units = k_blocks / 2;  // of two K blocks each (inputs come in multiples of 256)
  const int segments = GROUPED ? static_cast<int>(p.groups) : 1;  // drains per item
  const int segment_blocks = k_blocks / segments;
  const int row_tiles = (N_out + ITEM_ROWS - 1) / ITEM_ROWS;
  const int items = static_cast<int>(warp_uniform(p.groups_of_routes.count[0])) * row_tiles;
  volatile int* aborted = &abort_flag;
  const int items_here = set_up_ok ? items : 0;
  bool mma_issued = false;

  // Every role walks the same item list on its own clock; barriers carry the dependencies.
  if (warp < PF_DECODE_WARPS) {
    // ================= decode, and drain one segment behind =====================================
    const int quadrant = warp & 3, part = warp >> 2;    // part: which quarter of the columns this warp drains
    const int m = warp >> 3, parity = (warp >> 2) & 1;  // decodes every other K block of tile m
    const int row = quadrant * 32 + lane;
    const uint32_t abs_lane = PF_A0 + lane * 4u, sign_lane = PF_A0 + 128u + lane * 4u;
    const uint32_t lane_tmem = tmem + (static_cast<uint32_t>(quadrant * 32) << 16);
    // the rows of a code tile are swizzled in 16-byte chunks: 64-byte rows chunk ^ (row / 2) % 4, 32-byte rows chunk ^ (row / 4) % 2
    const uint32_t code_row = Plan::CODE_BASE + m * Plan::CODE_UNIT_BYTES + row * Plan::CODE_ROW_BYTES;
    const uint32_t code_chunk0 = BITS == 16 ? code_row + (((2u * parity) ^ ((row >> 1) & 3u)) << 4) : code_row + ((parity ^ ((row >> 2) & 1u)) << 4);
    const uint32_t code_chunk1 = code_row + (((2u * parity + 1u) ^ ((row >> 1) & 3u)) << 4);
    const Projection mats[2] = {p.a, GLU ? p.b : p.a};
    const bool scales32 = p.scales_dtype == KEEPVQ_F32;
    const float limit = p.swiglu_limit > 0.0f ? p.swiglu_limit : INFINITY;
    RingPlace<CODE_STAGES> code;
    // stage of this warp's K block, and the one A_STAGES before it: every other stage of one K block, every stage of two
    constexpr uint32_t OWN_STEP = SB == 2 ? 1 : 2;
    RingPlace<B_STAGES> stage, freed;
    if (SB == 1) { stage.advance(parity); freed.advance(parity); }
    int fresh = A_STAGES / OWN_STEP;   // this warp's first K blocks find their A stages free
    RingPlace<ACC_SETS> acc;
    RingPlace<PF_INFO_BUFFERS> info;
    bool ok = true;

    // the segment that waits for its drain
    bool pending = false;
    int pending_segment = 0;
    int quarter = 0;  // columns of the item, by four
    int erow = 0;
    uint32_t raw_scale[M];
    float sum[GROUPED ? M : 1][GROUPED ? N_MAX / 4 : 1];

    auto load_scale = [&](int64_t index, int mm) -> uint32_t {
      return scales32 ? static_cast<const uint32_t*>(mats[mm].scales)[index] : static_cast<const uint16_t*>(mats[mm].scales)[index];
    };
    auto as_scale = [&](uint32_t raw) {
      if (p.scales_dtype == KEEPVQ_F16) return __half2float(__ushort_as_half(static_cast<unsigned short>(raw)));
      return __uint_as_float(scales32 ? raw : raw << 16);
    };
    // accumulator columns c .. c + 3 of this thread's row
    auto load_columns = [&](uint32_t (&v)[M][2][4], int c) {
#pragma unroll
      for (int mm = 0; mm < M; ++mm)
#pragma unroll
        for (int piece = 0; piece < 2; ++piece) tmem_ld4(lane_tmem + acc.index * Plan::ACC_SET_COLS + mm * (2 * N_MAX) + piece * (quarter * 4) + c, v[mm][piece]);
    };
    // The accumulators are free again as soon as they are in registers: a warp gives its arrival when
    // the LAST of its columns has been read, before the arithmetic and the stores of those columns.
    auto release_accumulators = [&]() {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      mbar_arrive_warp(bar(ACC_EMPTY, acc.index), lane);
    };
    auto finish_column = [&](const int4& pr, const float (&y)[M], auto round_out, auto store_out) {
      if (GLU) {  // round G and U to the activation dtype first, as the separate kernels of the reference do
        const float gt = fminf(round_out(y[0]), limit);
        const float up = fminf(fmaxf(round_out(y[M - 1]), -limit), limit);
        const float result = gt / (1.0f + expf(-gt)) * up * __int_as_float(pr.w);
        if (pr.x >= 0 && erow < N_out) store_out(static_cast<int64_t>(pr.x) * N_out + erow, result);
      } else {
#pragma unroll
        for (int mm = 0; mm < M; ++mm)
          if (pr.x >= 0 && erow + mm * TILE_STEP < N_out) store_out(static_cast<int64_t>(pr.x) * N_out + erow + mm * TILE_STEP, y[mm]);
      }
    };
    // One instantiation per output dtype.
    auto drain_as = [&](auto round_out, auto store_out) {
      const int4* per_route = route_info[info.index];
      const int c_first = part * quarter;
      float scale[M];
#pragma unroll
      for (int mm = 0; mm < M; ++mm) scale[mm] = as_scale(raw_scale[mm]);
      if constexpr (GROUPED) {
#pragma unroll
        for (int c = 0; c < N_MAX / 4; c += 4) {  // (eight columns behind one wait have no registers: spills, 1086 -> 1160 us a layer of 1021 tokens)
          if (c >= quarter) break;
          uint32_t v[M][2][4], less[4];
          load_columns(v, c_first + c);
          asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(less[0]), "=r"(less[1]), "=r"(less[2]), "=r"(less[3])
                       : "r"(Plan::SUMS + ((info.index * PF_MAX_SEGMENTS + pending_segment) * N_MAX + c_first + c) * 4u));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (c + 4 >= quarter) release_accumulators();
#pragma unroll
          for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int mm = 0; mm < M; ++mm) {
              // 4 sum(w x') in wrapping 32-bit arithmetic, which the true value fits: four instructions a value and segment
              const int dot4 = static_cast<int>(v[mm][0][j] * 512u + (v[mm][1][j] * 2u + less[j]));
              sum[mm][c + j] += scale[mm] * static_cast<float>(dot4);
            }
          }
        }
        if (pending_segment == segments - 1) {
#pragma unroll
          for (int c = 0; c < N_MAX / 4; ++c) {
            if (c < quarter) {
              const int4 pr = per_route[c_first + c];
              float y[M];
#pragma unroll
              for (int mm = 0; mm < M; ++mm) y[mm] = 0.25f * __int_as_float(pr.y) * sum[mm][c];
              finish_column(pr, y, round_out, store_out);
            }
#pragma unroll
            for (int mm = 0; mm < M; ++mm) sum[mm][c] = 0.0f;
          }
        }
      } else {
        for (int c = 0; c < quarter; c += 4) {
          uint32_t v[M][2][4];
          load_columns(v, c_first + c);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (c + 4 >= quarter) release_accumulators();
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int4 pr = per_route[c_first + c + j];
            const float x_scale = __int_as_float(pr.y), x_sum4 = BITS == 16 ? 0.25f * static_cast<float>(pr.z) : 0.0f;
            const uint32_t offset = 8u * static_cast<uint32_t>(pr.z);  // the A operand was u = q + 8: 8 * sum(x') too much
            float y[M];
#pragma unroll
            for (int mm = 0; mm < M; ++mm) {
              // 256 high + low - 8 sum(x') = sum(q x'), in wrapping 32-bit arithmetic where the true value fits that
              const float dot = WIDE ? static_cast<float>(256 * static_cast<int64_t>(static_cast<int>(v[mm][0][j])) + static_cast<int>(v[mm][1][j]) - 8 * static_cast<int64_t>(pr.z))
                                     : static_cast<float>(static_cast<int>(v[mm][0][j] * 256u + v[mm][1][j] - offset));
              y[mm] = scale[mm] * x_scale * (0.5f * dot + x_sum4);
            }
            finish_column(pr, y, round_out, store_out);
          }
        }
      }
    };
    auto drain = [&]() {
      pending = false;
      if (!GROUPED || pending_segment == 0) ok = ok && mbar_wait(bar(INFO_FULL, info.index), info.phase, deadline, aborted);
      ok = ok && mbar_wait(bar(ACC_FULL, acc.index), acc.phase, deadline, aborted);
      if (!ok) return;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (p.out_dtype == KEEPVQ_BF16)
        drain_as([](float v) { return __bfloat162float(__float2bfloat16_rn(v)); },
                 [&](int64_t i, float v) { static_cast<__nv_bfloat16*>(p.out)[i] = __float2bfloat16_rn(v); });
      else if (p.out_dtype == KEEPVQ_F16)
        drain_as([](float v) { return __half2float(__float2half_rn(v)); },
                 [&](int64_t i, float v) { static_cast<__half*>(p.out)[i] = __float2half_rn(v); });
      else
        drain_as([](float v) { return v; }, [&](int64_t i, float v) { static_cast<float*>(p.out)[i] = v; });
      acc.advance();
      if (pending_segment == segments - 1) {
        __syncwarp();
        mbar_arrive_warp(bar(INFO_EMPTY, info.index), lane);
        info.advance();
      }
    };

    if constexpr (GROUPED) {
#pragma unroll
      for (int mm = 0; mm < M; ++mm)
#pragma unroll
        for (int c = 0; c < N_MAX / 4; ++c) sum[mm][c] = 0.0f;
    }
    for (int item = blockIdx.x; item < items_here && ok; item += gridDim.x) {
      const int gi = item / row_tiles, tile = item - gi * row_tiles;
      const int first_row = p.groups_of_routes.slot[gi] * N_out;
      const int gsize = p.groups_of_routes.size[gi];
      for (int segment = 0; segment < segments && ok; ++segment) {
        if (m < M) {
          for (int b = parity; b < segment_blocks; b += 2) {
            ok = mbar_wait(bar(CODE_FULL, code.index), code.phase, deadline, aborted);
            if (!ok) break;
            const uint32_t at = code.index * Plan::CODE_STAGE_BYTES;
            uint32_t w[8];
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(code_chunk0 + at));
            if constexpr (BITS == 16) asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "r"(code_chunk1 + at));
            const uint32_t to = lane_tmem + Plan::A_COL0 + (stage.index % A_STAGES) * Plan::A_STAGE_COLS + (SB == 2 ? parity * Plan::A_BLOCK_COLS : 0u) + m * PF_A_TILE_COLS;
            auto decode_words = [&](const uint32_t* words, uint32_t* q, int count) {  // the operand columns of `count` columns' codewords
              if constexpr (BITS == 16) {
#pragma unroll
                for (int i = 0; i < count / 4; ++i) {
                  decode_codeword_nibble<false>(words[i], abs_lane, sign_lane, q[4 * i], q[4 * i + 1]);
                  decode_codeword_nibble<true>(words[i], abs_lane, sign_lane, q[4 * i + 2], q[4 * i + 3]);
                }
              } else {
#pragma unroll
                for (int i = 0; i < count / 2; ++i) decode_byte_code(words[i >> 2], i & 3, abs_lane, q[2 * i], q[2 * i + 1]);
              }
            };
            auto codes_read = [&]() {
              __syncwarp();
              mbar_arrive_warp(bar(CODE_EMPTY, code.index), lane);
              code.advance();
            };
            if constexpr (Plan::HALVES) {
              // mostly the stage is free already: asked for under the reads of the codes
              const bool free = fresh > 0 || __all_sync(0xFFFFFFFFu, mbar_test(bar(STAGE_EMPTY, freed.index), freed.phase));
              uint32_t q[16];
              decode_words(w, q, 16);
              codes_read();
              if (!free) ok = mbar_wait(bar(STAGE_EMPTY, freed.index), freed.phase, deadline, aborted);
              if (!ok) break;
              if (fresh > 0) --fresh; else freed.advance(OWN_STEP);
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              tmem_st16(to, q);  // on its way to tensor memory under the decode of the other half
              uint32_t q2[16];
              decode_words(w + BITS / 4, q2, 16);
              tmem_st16(to + 16, q2);
            } else {
              uint32_t q[32];
              decode_words(w, q, 32);
              codes_read();
              if (fresh > 0) {
                --fresh;
              } else {
                ok = mbar_wait(bar(STAGE_EMPTY, freed.index), freed.phase, deadline, aborted);
                if (!ok) break;
                freed.advance(OWN_STEP);
              }
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              tmem_st32(to, q);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            mbar_arrive_warp(bar(STAGE_FULL, stage.index), lane);
            stage.advance(OWN_STEP);
            // the previous segment's MMAs have had this K block's decode to finish under
            if (pending) {
              drain();
              if (!ok) break;  // (the next wait would find its barrier complete and carry on)
            }
          }
        }
        if (pending) drain();  // a warp without K blocks
        // this segment is the next to be drained; what its drain needs from memory is asked for now
        pending = true;
        pending_segment = segment;
        if (segment == 0) {
          quarter = ((gsize + 15) & ~15) >> 2;
          erow = tile * ITEM_ROWS + row;
        }
#pragma unroll
        for (int mm = 0; mm < M; ++mm) raw_scale[mm] = load_scale(static_cast<int64_t>(first_row + min(erow + mm * TILE_STEP, N_out - 1)) * segments + segment, mm);
      }
    }
    if (pending && ok) drain();
    if (lane == 0) decode_place[warp] = (freed.phase * B_STAGES + freed.index + A_STAGES - OWN_STEP * fresh) % (2 * B_STAGES);  // its next stage
  } else if (warp == PF_MMA_WARP) {
    // ================= the MMAs ================================================================
    // One loop over all K blocks of the block's items, unrolled over the stage ring: this warp's own
    // instructions between two K blocks are on the critical path.  The whole warp walks and waits,
    // one elected lane issues, and the addresses are immediates: an MMA's descriptors live in uniform
    // registers, and code that moves them there for each MMA cost more than the MMAs themselves
    // (79 cycles each from a lane's branch; 610 cycles of issue per K block of eight MMAs with two
    // waits, two commits and addresses worked out inside the elected branch, where the tensor core
    // takes 128 to 256 at 16 to 32 routes).
    RingPlace<ACC_SETS> acc;
    uint32_t phase = 0, idesc = 0, d_cols = 0;
    bool ok = true, first_round = true;
    int item = static_cast<int>(blockIdx.x) - static_cast<int>(gridDim.x), segment = segments - 1, kb = segment_blocks - SB;
    // the next segment: its accumulators, and at the start of an item its width
    auto next_segment = [&]() {
      kb = 0;
      if (++segment == segments) {
        segment = 0;
        item += gridDim.x;
        if (item >= items_here) return false;
        const int gi = item / row_tiles;
        const int n_pad = (p.groups_of_routes.size[gi] + 15) & ~15;
        // N = 2 * n_pad: the high-byte rows and the low-byte rows of the routes are one B operand;
        // accumulator s32, A unsigned bytes (the nibble decoder's u = q + 8), B signed bytes
        idesc = warp_uniform((2u << 4) | (0u << 7) | (1u << 10) | (static_cast<uint32_t>(n_pad >> 2) << 17) | ((PF_ROWS >> 4) << 24));
      }
      if (!first_round && !mbar_wait(bar(ACC_EMPTY, acc.index), acc.phase ^ 1u, deadline, aborted)) return false;  // the set's last accumulators are in registers
      if (ACC_SETS > 1) d_cols = warp_uniform(acc.index * Plan::ACC_SET_COLS);
      return true;
    };
    while (ok) {
#pragma unroll
      for (uint32_t st = 0; st < B_STAGES; ++st) {
        if ((kb += SB) == segment_blocks) ok = ok && next_segment();
        ok = ok && mbar_wait(bar(STAGE_FULL, st), phase, deadline, aborted);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t accumulate = kb != 0;
        const bool last = kb == segment_blocks - SB;
        if (elect_one()) {
#pragma unroll
          for (int mj = 0; mj < M * SB; ++mj) {
            const int m = mj % M, j = mj / M;  // tile, K block of the stage
#pragma unroll
            for (int k = 0; k < 4; ++k)  // 32 bytes of K per instruction: 8 columns of A, 2 x 16 bytes of the B start address
              umma_i8_ts(d_cols + m * (2 * N_MAX), Plan::A_COL0 + (st % A_STAGES) * Plan::A_STAGE_COLS + j * Plan::A_BLOCK_COLS + m * PF_A_TILE_COLS + 8 * k,
                         umma_desc(Plan::b_stage(st) + j * Plan::B_BLOCK_BYTES) + 2 * k, idesc, accumulate | static_cast<uint32_t>(j | k));
          }
          umma_commit(bar(STAGE_EMPTY, st));  // the stage may be refilled once these MMAs have read it
          if (last) umma_commit(bar(ACC_FULL, acc.index));
        }
        __syncwarp();
        mma_issued = true;
        if (last) {
          acc.advance();
          if (acc.index == 0) first_round = false;
        }
      }
      phase ^= 1u;
    }
  } else if (warp == PF_B_WARP) {
    // ================= activation (B operand) loader: TMA ====================================
    // Rows gstart .. gstart + n_pad - 1 of the high-byte plane and of the low-byte plane in one box,
    // which lands swizzled as the operand tile it is; rows past the group's own belong to the next
    // group or to nobody, and nobody looks at their columns.  The whole warp walks and one elected
    // lane issues: from a branch of one lane a copy cost some 150 cycles of its issue.
    RingPlace<B_STAGES> b;
    uint32_t used = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < items_here && ok; item += gridDim.x) {
      const int gi = item / row_tiles;
      const int gsize = warp_uniform(p.groups_of_routes.size[gi]), gstart = warp_uniform(p.groups_of_routes.start[gi]);
      const int n_pad = (gsize + 15) & ~15;
      const CUtensorMap* map = &x_maps.rows[(n_pad >> 4) - 1];
      for (int kb = 0; kb < k_blocks; kb += SB) {
        ok = mbar_wait<true>(bar(STAGE_EMPTY, b.index), b.phase ^ 1u, deadline, aborted);
        if (!ok) break;
        if (stall != STALL_ACTIVATIONS) {
          if (elect_one()) {
            mbar_expect_tx(bar(STAGE_FULL, b.index), static_cast<uint32_t>(SB * 2 * n_pad * 128));
#pragma unroll
            for (int j = 0; j < SB; ++j)
              tma_box_3d(Plan::b_stage(b.index) + j * Plan::B_BLOCK_BYTES, map, (kb + j) * 128, gstart, 0, bar(STAGE_FULL, b.index));
          }
          ++used;
        }
        b.advance();
      }
    }
    if (lane == 0) activations_issued = used;
  } else if (warp == PF_CODE_WARP) {
    // ================= code loader: TMA ======================================================
    // Two K blocks of every tile per stage, straight from the caller's
    // layout seen as one byte matrix of slots * out_dim rows; rows past a slot's last tile are
    // the next slot's (or zeros past the end) and their outputs are never stored.
    RingPlace<CODE_STAGES> code;
    uint32_t used = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < items_here && ok; item += gridDim.x) {
      const int gi = item / row_tiles, tile = item - gi * row_tiles;
      const int row0 = static_cast<int>(warp_uniform(static_cast<uint32_t>(p.groups_of_routes.slot[gi] * N_out + tile * ITEM_ROWS)));
      for (int u = 0; u < code_units; ++u) {
        ok = mbar_wait<true>(bar(CODE_EMPTY, code.index), code.phase ^ 1u, deadline, aborted);
        if (!ok) break;
        if (stall == STALL_CODES) continue;
        if (elect_one()) {
          const uint32_t full = bar(CODE_FULL, code.index);
          mbar_expect_tx(full, Plan::CODE_STAGE_BYTES);
          tma_box_2d(Plan::CODE_BASE + code.index * Plan::CODE_STAGE_BYTES, &a_map, u * static_cast<int>(Plan::CODE_ROW_BYTES), row0, full);
          if (GLU) tma_box_2d(Plan::CODE_BASE + code.index * Plan::CODE_STAGE_BYTES + Plan::CODE_UNIT_BYTES, &b_map, u * static_cast<int>(Plan::CODE_ROW_BYTES), row0, full);
        }
        ++used;
        code.advance();
      }
    }
    if (lane == 0) codes_issued = used;
  }

  if (warp == PF_INFO_WARP) {
    // ================= what the drain needs per route, up to three items ahead ==================
    RingPlace<PF_INFO_BUFFERS> info;
    bool ok = true;
    for (int item = blockIdx.x; item < items_here && ok; item += gridDim.x) {
      const int gi = item / row_tiles;
      const int gsize = p.groups_of_routes.size[gi], gstart = p.groups_of_routes.start[gi];
      const int n_pad = (gsize + 15) & ~15;
      ok = mbar_wait<true>(bar(INFO_EMPTY, info.index), info.phase ^ 1u, deadline, aborted);
      if (!ok) break;
      for (int n = lane; n < n_pad; n += 32) {
        const int route = n < gsize ? p.groups_of_routes.routes[gstart + n] : -1;
        const int64_t xrow = route < 0 ? p.x_zero_row : static_cast<int64_t>(gstart + n);  // the activation rows were quantised in grouped order
        const float weight = (GLU && route >= 0) ? p.route_weight[route] : 1.0f;
        route_info[info.index][n] = make_int4(route, __float_as_int(p.x.scale[xrow]), GROUPED ? 0 : p.x.sums[xrow], __float_as_int(weight));
      }
      if constexpr (GROUPED) {
        // the A operand is u = q + 8 (4w = 2q + 1; 2q for 8-bit codes): 2 D - 15 sum(x') = sum(4w x'), or 2 D - 16 sum(x')
        const int step_n = 32 / segments, step_segment = 32 % segments;
        int n = lane / segments, segment = lane % segments;
        while (n < n_pad) {
          const int x_sum = n < gsize ? p.x.sums[static_cast<int64_t>(gstart + n) * segments + segment] : 0;
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(Plan::SUMS + ((info.index * PF_MAX_SEGMENTS + segment) * N_MAX + n) * 4u),
                       "r"((BITS == 16 ? 15u : 16u) * (0u - static_cast<uint32_t>(x_sum))) : "memory");
          n += step_n;
          segment += step_segment;
          if (segment >= segments) { segment -= segments; ++n; }
        }
      }
      while (stall == STALL_FACTS && !*aborted && global_timer_ns() <= deadline + 1000000) __nanosleep(1000);
      __syncwarp();
      mbar_arrive_warp(bar(INFO_FULL, info.index), lane);
      info.advance();
    }
  }

  // ---- teardown ------------------------------------------------------------------------------
  __syncthreads();  // every role has left its loop: nothing is issued any more, and the flag is what it will be
  if (*aborted) {
    if (tid == 0 && status) atomicExch(status, set_up_ok ? 1 : 2);
    // What may still be in flight is waited for, bounded as every wait: MMAs (one more commit arrives
    // when they are all done), codes, activations.
    if (warp == PF_MMA_WARP && mma_issued && elect_one()) {  // the lane that issued: a commit follows its own thread's MMAs
      umma_commit(bar(DRAINED, 0));
      mbar_wait_grace(bar(DRAINED, 0), 0u);
    }
    if (warp == PF_CODE_WARP && lane == 0) wait_codes_landed<CODE_STAGES>(bar(CODE_FULL, 0), codes_issued);
    if (warp == PF_B_WARP && lane == 0) wait_activations_landed<B_STAGES, SB>(bar(STAGE_FULL, 0), activations_issued, decode_place, M * 8);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == PF_MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base_slot), "r"(PF_TMEM_COLS) : "memory");
}

bool prefill_supported(int64_t slots, int64_t out_dim, int64_t in_dim, int64_t groups) {
  // code rows are addressed by a 32-bit box coordinate that may run past the last row by an item
  return shapes_supported(out_dim, in_dim, groups) && slots * out_dim < (int64_t{1} << 31) - 4 * PF_ROWS &&
         (groups == 1 || (groups <= PF_MAX_SEGMENTS && in_dim / groups <= PF_MAX_SEGMENT_INPUTS));
}

// Routes per item.  96 fill tensor memory (accumulators of two byte planes and two tiles, two A
// stages), 48 leave room for four K blocks' A tiles (two stages of two); rows with several scale groups take the second half of
// tensor memory for a second accumulator set instead.  An expert with more routes than that is
// decoded once per item, so 48 serve calls whose experts rarely get more: up to 32 on average
// (of a uniform router's experts 0.3 % then exceed 48).
int prefill_group_routes(int64_t live, int64_t slots, bool several_groups) {
  return several_groups || live <= PREFILL_FEW_ROUTES_MEAN * slots ? PREFILL_GROUP_ROUTES_SMALL : PREFILL_GROUP_ROUTES;
}

// A tensor map of bytes in this GPU's own memory: `planes` matrices of [rows, row_bytes] one after the
// other, boxes of planes x box_rows x box_bytes.
static int byte_map(CUtensorMap* map, const void* base, int64_t row_bytes, int64_t rows, uint32_t planes, uint32_t box_bytes, uint32_t box_rows, CUtensorMapSwizzle swizzle) {
  typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static EncodeTiled encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
    const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found);
    if (e != cudaSuccess) return note_cuda_error(e);
    if (found != cudaDriverEntryPointSuccess || !fn) return KEEPVQ_ERR_UNSUPPORTED;
    encode = reinterpret_cast<EncodeTiled>(fn);
  }
  if (row_bytes % 16 != 0 || (reinterpret_cast<uintptr_t>(base) & 15u) != 0) return KEEPVQ_ERR_ALIGN;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(row_bytes), static_cast<cuuint64_t>(rows), planes};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(row_bytes), static_cast<cuuint64_t>(row_bytes * rows)};
  const cuuint32_t box[3] = {box_bytes, box_rows, planes}, element_strides[3] = {1, 1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, planes > 1 ? 3 : 2, const_cast<void*>(base), dims, strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? KEEPVQ_OK : KEEPVQ_ERR_LAUNCH;
}
// A projection's codes: a byte matrix of slots * out_dim rows, two K blocks of a row's codes per box row.
static int code_map(const FastProjectionArgs& p, const void* codes, int bits, uint32_t box_rows, CUtensorMap* map) {
  return byte_map(map, codes, p.in_dim / 8 * (bits / 8), p.slots * p.out_dim, 1, 2 * PF_KBLOCK_CODES * bits / 8, box_rows, bits == 16 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

template <int M, bool GLU, int N_MAX, bool GROUPED, int BITS, bool WIDE>
static int launch_prefill_kernel(const FastProjectionArgs& p, int32_t* status, cudaStream_t s, int stall = 0, uint64_t wait_ns = 0, int ctas = 0) {
  ActivationMaps<N_MAX> x_maps;  // the quantised activations: the high-byte plane, then the low-byte plane, each [rows + 1, in_dim]
  for (int i = 0; i < N_MAX / 16; ++i)
    if (const int rc = byte_map(&x_maps.rows[i], p.x.q, p.in_dim, p.x_zero_row + 1, 2, 128, 16 * (i + 1), CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
  CUtensorMap a_map, b_map;
  if (const int rc = code_map(p, p.a.codes, BITS, GLU ? PF_ROWS : PF_ROWS * M, &a_map)) return rc;
  if (GLU) {
    if (const int rc = code_map(p, p.b.codes, BITS, PF_ROWS, &b_map)) return rc;
  } else b_map = a_map;
  auto kernel = prefill_projection_kernel<M, GLU, N_MAX, GROUPED, BITS, WIDE>;
  static uint64_t configured = 0;  // one bit per device: the shared-memory opt-in is a per-device attribute of the function
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !((configured >> dev) & 1ull)) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PF_SMEM_BYTES);
    if (e != cudaSuccess) return note_cuda_error(e);
    if (dev >= 0 && dev < 64) configured |= 1ull << dev;
  }
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const cudaError_t err = launch_after(true, kernel, ctas > 0 ? ctas : sms, PF_THREADS, PF_SMEM_BYTES, s, p, x_maps, a_map, b_map, status, stall, wait_ns);
  return err == cudaSuccess ? KEEPVQ_OK : note_cuda_error(err);
}

template <int M, bool GLU, int N_MAX, bool GROUPED, int BITS = 16>
static int launch_prefill(const FastProjectionArgs& p, int32_t* status, cudaStream_t s, int stall = 0, uint64_t wait_ns = 0, int ctas = 0) {
  if (!GROUPED && p.in_dim > PF_EXACT32_INPUTS) return launch_prefill_kernel<M, GLU, N_MAX, GROUPED, BITS, !GROUPED>(p, status, s, stall, wait_ns, ctas);
  return launch_prefill_kernel<M, GLU, N_MAX, GROUPED, BITS, false>(p, status, s, stall, wait_ns, ctas);
}

template <int M, bool GLU>
static int launch_prefill_any(const FastProjectionArgs& p, int32_t* status, cudaStream_t s) {
  if (p.groups > 1) return launch_prefill<M, GLU, PREFILL_GROUP_ROUTES_SMALL, true>(p, status, s);
  if (p.group_cols <= PREFILL_GROUP_ROUTES_SMALL) return launch_prefill<M, GLU, PREFILL_GROUP_ROUTES_SMALL, false>(p, status, s);
  return launch_prefill<M, GLU, PREFILL_GROUP_ROUTES, false>(p, status, s);
}
int prefill_gate_up(const FastProjectionArgs& p, int32_t* status, cudaStream_t s) { return launch_prefill_any<2, true>(p, status, s); }
// a single projection takes two row tiles per item when it has them (the activation copies serve both)
int prefill_down(const FastProjectionArgs& p, int32_t* status, cudaStream_t s) {
  return p.out_dim > PF_ROWS ? launch_prefill_any<2, false>(p, status, s) : launch_prefill_any<1, false>(p, status, s);
}
// 8-bit codes (p.a.codes holds bytes, p.codebook their table); p.group_cols is PREFILL_GROUP_ROUTES_SMALL.
int prefill_byte_codes(const FastProjectionArgs& p, int32_t* status, cudaStream_t s) {
  if (p.groups > 1) return launch_prefill<2, false, PREFILL_GROUP_ROUTES_SMALL, true, 8>(p, status, s);
  return launch_prefill<2, false, PREFILL_GROUP_ROUTES_SMALL, false, 8>(p, status, s);
}
// One CTA of a single-projection kernel, one of whose loaders never publishes, with a short deadline:
// a wait runs out, the CTA reports and returns.  `p` must describe a valid problem.
// 0: the 96-route form without activations; 1: the scale-group form without codes; 2: the 8-bit form without codes;
// 3: the 48-route form whose per-route facts come too late.
int prefill_wait_selftest(int form, const FastProjectionArgs& p, int32_t* status, uint64_t wait_ns, cudaStream_t s) {
  if (form == 1) return launch_prefill<2, false, PREFILL_GROUP_ROUTES_SMALL, true>(p, status, s, STALL_CODES, wait_ns, 1);
  if (form == 2) return launch_prefill<2, false, PREFILL_GROUP_ROUTES_SMALL, false, 8>(p, status, s, STALL_CODES, wait_ns, 1);
  if (form == 3) return launch_prefill<2, false, PREFILL_GROUP_ROUTES_SMALL, false>(p, status, s, STALL_FACTS, wait_ns, 1);
  return launch_prefill<1, false, PREFILL_GROUP_ROUTES, false>(p, status, s, STALL_ACTIVATIONS, wait_ns, 1);
}

}  // namespace fast
}  // namespace keepvq
