// One expert-grouped projection over routes, on the int8 tensor-core kernels: the operator-level
// counterpart of the reference's sorted-route prefill kernels
// (src/ramp/kernels/gather_vqmm.py:597-928, native/vq_nax_ext/kernels/nax_fp16_matmul.metal:904-1062).
//
// out[r] = W[rhs[r]] @ x[r] for r < routes; x holds one activation row per route (the caller
// gathers them, as the reference does before its kernels, src/ramp/ops/vq_switch.py:758-761).
// The sequence is the down projection of the layer call: quantise the rows, group the routes by
// expert on the device, then the tcgen05 kernel (5 or more routes per expert on average) or the
// mma.sync one; 8-bit codes run on the tcgen05 kernel alone.  Routes need not be sorted; a route with expert 0xFFFFFFFF gives a zero row.
#include <algorithm>

#include "moe_fast.cuh"

namespace keepvq {

// 8-bit codes: whether the grouped kernel is faster than the general one, which needs no grouping, no
// quantised rows and no 64 KB of tables in front of it, but reads an expert's codes once per four routes
// and a code tile with one output row a thread.  Device time with cold codes, general / grouped us, over
// matrices of 2^15 to 2^24 weights, 1 to 384 experts, 12 to 768 routes:
//   12 routes    25 / 32 at 1024 x 2048, 47 / 30 at 2048 x 4096 (384 experts)
//   24 routes    16 / 22 at 256 x 512, 27 / 26 at 512 x 1024, 37 / 32 at 1024 x 2048 (64 experts)
//   48 routes    16 / 20 at 128 x 256, 23 / 22 at 256 x 512 (64 experts)
//   96 routes    23 / 22 at 128 x 256 (384 experts), and 274 / 73 at 2048 x 4096
// With three routes an expert some expert has more than four, and the general kernel passes over its
// codes again: 39 / 20 for 12 routes of one 128 x 256 expert, 31 / 22 for 24 routes of eight 256 x 512.
static bool byte_codes_pay(int64_t routes, int64_t slots, int64_t weights) {
  if (routes < 12) return false;
  if (routes >= 96 || routes >= 3 * slots) return true;
  return weights >= (routes >= 48 ? int64_t{1} << 17 : routes >= 24 ? int64_t{1} << 19 : int64_t{1} << 22);
}

// ... and whether its limits hold the sizes.
static bool byte_codes_served(int64_t routes, int64_t slots, int64_t out_dim, int64_t in_dim, int64_t groups) {
  return routes <= (1 << 20) && slots <= 16384 && fast::prefill_supported(slots, out_dim, in_dim, groups) && byte_codes_pay(routes, slots, out_dim * in_dim);
}

struct GroupedScratch {
  int64_t xq, xscale, xsums, gcount, gslot, gstart, gsize, groutes, status, total;
};

static inline int64_t up256(int64_t v) { return (v + 255) / 256 * 256; }

static GroupedScratch plan_grouped(int64_t routes, int64_t in_dim) {
  GroupedScratch s;
  int64_t at = 0;
  s.xq = at;      at += up256((routes + 1) * in_dim * 2);
  s.xscale = at;  at += up256((routes + 1) * 4);
  s.xsums = at;   at += up256((routes + 1) * (in_dim / 8) * 4);
  s.gcount = at;  at += 256;
  s.gslot = at;   at += up256(routes * 4);
  s.gstart = at;  at += up256(routes * 4);
  s.gsize = at;   at += up256(routes * 4);
  s.groutes = at; at += up256(routes * 4);
  s.status = at;  at += 256;
  s.total = at;
  return s;
}

}  // namespace keepvq

namespace keepvq {
constexpr int64_t ZERO_ROUTES = 64;
static __device__ uint32_t g_zero_routes[ZERO_ROUTES];  // never written
}  // namespace keepvq

extern "C" int keepvq_zero_routes(const uint32_t** routes, int64_t* count) {
  if (!routes || !count) return KEEPVQ_ERR_NULL;
  void* address = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&address, keepvq::g_zero_routes);
  if (e != cudaSuccess) return keepvq::note_cuda_error(e);
  *routes = static_cast<const uint32_t*>(address);
  *count = keepvq::ZERO_ROUTES;
  return KEEPVQ_OK;
}

extern "C" int64_t keepvq_grouped_projection_workspace_bytes(int64_t routes, int64_t in_dim) {
  if (routes < 0 || in_dim <= 0 || in_dim % 8) return KEEPVQ_ERR_SHAPE;
  return keepvq::plan_grouped(routes, in_dim).total;
}

extern "C" int keepvq_grouped_projection_bytes_served(int64_t routes, int64_t slots, int64_t out_dim, int64_t in_dim, int64_t groups) {
  return routes > 0 && slots > 0 && out_dim > 0 && in_dim > 0 && groups > 0 && keepvq::byte_codes_served(routes, slots, out_dim, in_dim, groups) ? 1 : 0;
}

extern "C" int64_t keepvq_grouped_projection_status_offset(int64_t routes, int64_t in_dim) {
  if (routes < 0 || in_dim <= 0 || in_dim % 8) return KEEPVQ_ERR_SHAPE;
  return keepvq::plan_grouped(routes, in_dim).status;
}

namespace keepvq {

static int grouped_projection(const keepvq_grouped_projection_args* args, bool byte_codes, void* stream) {
  if (!args) return KEEPVQ_ERR_NULL;
  const keepvq_grouped_projection_args& a = *args;
  if (!valid_dtype(a.x_dtype) || !valid_dtype(a.scales_dtype)) return KEEPVQ_ERR_DTYPE;
  if (a.routes < 0 || a.slots <= 0 || a.out_dim <= 0 || a.in_dim <= 0 || a.in_dim % 8 || a.groups <= 0) return KEEPVQ_ERR_SHAPE;
  if (a.routes == 0) return KEEPVQ_OK;
  if (!a.x || !a.rhs || !a.codes || !a.scales || !a.codebook || !a.out || !a.workspace) return KEEPVQ_ERR_NULL;
  if (a.x_dtype == KEEPVQ_F32) return KEEPVQ_ERR_UNSUPPORTED;  // these kernels keep 16 bits of a row: not what an fp32 caller asked for
  if ((!byte_codes && !a.codebook_all_odd) || !fast::shapes_supported(a.out_dim, a.in_dim, a.groups)) return KEEPVQ_ERR_UNSUPPORTED;
  if (byte_codes && (a.res_codes || !aligned_to(a.codes, 16) || !byte_codes_served(a.routes, a.slots, a.out_dim, a.in_dim, a.groups))) return KEEPVQ_ERR_UNSUPPORTED;  // (the general kernel takes them)
  const int32_t x_div = a.x_div > 0 ? a.x_div : 1;
  if (a.routes % x_div) return KEEPVQ_ERR_SHAPE;
  const int64_t x_rows = a.routes / x_div;
  const bool residual = a.res_codes != nullptr;
  if (residual) {
    if (!a.res_scales || !a.res_table || !a.hot_of_slot) return KEEPVQ_ERR_NULL;
    if (a.res_rows <= 0 || a.res_groups <= 0) return KEEPVQ_ERR_SHAPE;
    if (!fast::residual_supported(a.routes, a.in_dim, a.res_groups)) return KEEPVQ_ERR_UNSUPPORTED;
    if (!aligned_to(a.res_codes, 8)) return KEEPVQ_ERR_ALIGN;
  }
  if (!aligned_to(a.x, 16) || !aligned_to(a.codes, 16) || !aligned_to(a.workspace, 256)) return KEEPVQ_ERR_ALIGN;
  const GroupedScratch sc = plan_grouped(a.routes, a.in_dim);
  if (a.workspace_bytes < sc.total) return KEEPVQ_ERR_CAPACITY;
  char* ws = reinterpret_cast<char*>(a.workspace);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  fast::RouteGroups groups = {reinterpret_cast<int32_t*>(ws + sc.gcount), reinterpret_cast<int32_t*>(ws + sc.gslot),
                              reinterpret_cast<int32_t*>(ws + sc.gstart), reinterpret_cast<int32_t*>(ws + sc.gsize),
                              reinterpret_cast<int32_t*>(ws + sc.groutes)};
  if (!byte_codes && !residual && a.routes < fast::SMALL_CALL_ROUTES && fast::few_tokens_fits(a.routes, 1, a.slots, a.out_dim, a.in_dim, a.groups)) {
    // Few routes: one launch that quantises and groups for itself, against two with the sweep kernel (us a captured call,
    // cold codes, B200; 3 / 24 / 47 routes): 2048 x 4096 of one matrix 10.0 / 13.5 / 17.4 against 11.4 / 14.6 / 18.7, of 192
    // 12.3 / 22.9 / 35.0 against 14.1 / 28.7 / 43.8; 5120 x 2304 with scale groups of one matrix 9.7 / 15.3 / 21.3 against
    // 15.4 / 20.8 / 28.8, of 192 13.6 / 35.8 / 58.0 against 17.9 / 43.1 / 71.8; 126 sizes timed, none the other way.
    fast::FewTokensArgs f = {};
    f.parts = fast::FT_DOWN;
    f.routes = static_cast<int32_t>(a.routes); f.tokens = static_cast<int32_t>(x_rows); f.top_k = x_div;
    f.scales_dtype = a.scales_dtype; f.slots = a.slots; f.codebook = a.codebook; f.slot = a.rhs;
    f.phase[1] = {{a.codes, nullptr}, {a.scales, nullptr}, a.x, a.out, static_cast<int32_t>(a.out_dim), static_cast<int32_t>(a.in_dim), static_cast<int32_t>(a.groups), x_div, a.out_dtype};
    f.dead_out = a.out; f.dead_row_bytes = a.out_dim * dtype_size(a.out_dtype);
    f.status = reinterpret_cast<int32_t*>(ws + sc.status); f.clear_status = 1;
    const int rc = fast::few_tokens(f, a.x_dtype, nullptr, s);
    if (rc != KEEPVQ_ERR_UNSUPPORTED) return rc;
  }
  const bool many = byte_codes || (!residual && fast::prefill_pays(a.routes, a.slots, a.groups > 1) && fast::prefill_supported(a.slots, a.out_dim, a.in_dim, a.groups));
  // (the sums region has room for a scale group per codeword; these kernels' rows have at most one
  // per 256 inputs, and their sums per 256 inputs go behind those)
  fast::QuantRows xq = {reinterpret_cast<uint8_t*>(ws + sc.xq), reinterpret_cast<float*>(ws + sc.xscale), reinterpret_cast<int32_t*>(ws + sc.xsums),
                        many ? nullptr : reinterpret_cast<int32_t*>(ws + sc.xsums) + (x_rows + 1) * a.groups};
  int32_t* wait_status = reinterpret_cast<int32_t*>(ws + sc.status);
  if (many) groups.position = reinterpret_cast<int32_t*>(ws + sc.xsums) + (a.routes + 1) * a.groups;  // behind the sums, as well
  int rc;
  const int group_cols = byte_codes ? fast::PREFILL_GROUP_ROUTES_SMALL : many ? fast::prefill_group_routes(a.routes, a.slots, a.groups > 1) : fast::decode_group_routes(a.routes, a.slots, a.in_dim);
  const fast::DeadRows dead = {a.rhs, x_div, a.slots, a.out, a.out_dim * dtype_size(a.out_dtype)};
  if (!many && fast::group_with_quantize_supported(a.routes, a.slots)) {  // one launch for both
    if ((rc = fast::quantize_rows_and_group(a.x, a.x_dtype, x_rows, a.in_dim, a.groups, xq, false, s, nullptr, 1, a.slots, a.rhs, a.routes, group_cols, groups, wait_status, dead))) return rc;
  } else {
    // The projection kernel reads its codebook before it waits for its predecessors.  8-bit calls take any
    // table, one that a kernel has just written too: their first launch is an ordinary one, and what it
    // waited for is in place for all that follow.  (A 16-bit table has been read back by its caller.)
    if ((rc = fast::group_routes(a.rhs, a.routes, a.slots, group_cols, groups, wait_status, s, !byte_codes))) return rc;
    if (many) rc = fast::quantize_rows_sorted(a.x, a.x_dtype, x_rows, a.in_dim, a.groups, xq, groups.position, x_div, s, dead);
    else rc = fast::quantize_rows_and_group(a.x, a.x_dtype, x_rows, a.in_dim, a.groups, xq, false, s, nullptr, 1, a.slots, nullptr, 0, 0, {}, nullptr, dead);
    if (rc) return rc;
  }
  fast::FastProjectionArgs p = {};
  p.slots = a.slots;
  p.a = {a.codes, a.scales, a.res_codes, a.res_scales}; p.b = {nullptr, nullptr, nullptr, nullptr};
  if (residual) { p.res_groups = a.res_groups; p.hot_of_slot = a.hot_of_slot; p.res_table = a.res_table; }
  p.scales_dtype = a.scales_dtype; p.codebook = a.codebook; p.groups_of_routes = groups; p.max_routes = a.routes; p.group_cols = group_cols; p.status = wait_status;
  p.few_groups = many ? 0 : fast::few_route_groups(a.routes, a.slots);
  p.out_dim = a.out_dim; p.in_dim = a.in_dim; p.groups = a.groups; p.x = xq; p.x_zero_row = many ? a.routes : x_rows; p.x_div = x_div;
  p.out = a.out; p.out_dtype = a.out_dtype; p.swiglu_limit = 0.0f; p.route_weight = nullptr;
  if (byte_codes) return fast::prefill_byte_codes(p, wait_status, s);
  return many ? fast::prefill_down(p, wait_status, s) : fast::down(p, s);
}

}  // namespace keepvq

extern "C" int keepvq_grouped_projection(const keepvq_grouped_projection_args* args, void* stream) { return keepvq::grouped_projection(args, false, stream); }
extern "C" int keepvq_grouped_projection_bytes(const keepvq_grouped_projection_args* args, void* stream) { return keepvq::grouped_projection(args, true, stream); }

// ------------------------------------------------------------------------------------------
// Self-test of the bounded waits of the tcgen05 kernel: runs of one CTA on a tiny problem laid out in
// the caller's scratch, one of whose loaders never publishes its tiles.  A wait then runs into its
// deadline (on the global timer); the CTA must set its status word to 1, wait for what the other
// loader still has in flight, free its tensor memory and return, and the context must stay usable.
// Nothing faults and nothing spins without a limit.  No counterpart in the reference.
// ------------------------------------------------------------------------------------------
namespace keepvq {
constexpr int64_t SELFTEST_BYTES = 192 * 1024;
constexpr int64_t SELFTEST_SHORT_NS = 5000000;  // the runs behind the first take no longer than this each
__global__ void selftest_init_kernel(int32_t* count, int32_t* size, int32_t* routes, float* x_scale) {
  if (threadIdx.x == 0) { count[0] = 1; size[0] = 16; }
  if (threadIdx.x < 16) routes[threadIdx.x] = threadIdx.x;
  if (threadIdx.x < 17) x_scale[threadIdx.x] = 1.0f;
}
// How many values of columns first .. 511 of 16 output rows are not `want`.
__global__ void selftest_check_kernel(const uint16_t* out, int first, uint32_t want, int32_t* wrong) {
  for (int i = threadIdx.x; i < 16 * (512 - first); i += 256)
    if (out[i / (512 - first) * 512 + first + i % (512 - first)] != want) atomicAdd(wrong, 1);
}
}  // namespace keepvq

extern "C" int64_t keepvq_wait_selftest_workspace_bytes(void) { return keepvq::SELFTEST_BYTES; }

extern "C" int keepvq_wait_selftest(void* workspace, int64_t workspace_bytes, int64_t wait_ns, void* stream) {
  using namespace keepvq;
  if (!workspace) return KEEPVQ_ERR_NULL;
  if (workspace_bytes < SELFTEST_BYTES) return KEEPVQ_ERR_CAPACITY;
  if (!aligned_to(workspace, 256)) return KEEPVQ_ERR_ALIGN;
  if (wait_ns <= 0 || wait_ns > 1000000000ll) return KEEPVQ_ERR_SHAPE;  // a self-test may hold the GPU for about a second at most
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  char* ws = reinterpret_cast<char*>(workspace);
  int32_t* status = reinterpret_cast<int32_t*>(ws);
  cudaError_t e = cudaMemsetAsync(ws, 0, SELFTEST_BYTES, s);
  if (e != cudaSuccess) return note_cuda_error(e);
  // status words 0 | groups 256.. | routes 1280 | table 2048 | x scale 3072 | x sums 4096 | scales 8192 | out 16384 | planes 32768 | codes 65536
  fast::RouteGroups groups = {reinterpret_cast<int32_t*>(ws + 256), reinterpret_cast<int32_t*>(ws + 512), reinterpret_cast<int32_t*>(ws + 768),
                              reinterpret_cast<int32_t*>(ws + 1024), reinterpret_cast<int32_t*>(ws + 1280)};
  fast::QuantRows xq = {reinterpret_cast<uint8_t*>(ws + 32768), reinterpret_cast<float*>(ws + 3072), reinterpret_cast<int32_t*>(ws + 4096), nullptr};
  selftest_init_kernel<<<1, 32, 0, s>>>(groups.count, groups.size, groups.routes, xq.scale);
  KEEPVQ_CHECK_LAUNCH();
  fast::FastProjectionArgs p = {};
  p.a = {reinterpret_cast<const uint16_t*>(ws + 65536), ws + 8192, nullptr, nullptr};
  p.scales_dtype = KEEPVQ_F16; p.slots = 1; p.in_dim = 512;  // two planes of 17 rows of 512 inputs
  p.codebook = reinterpret_cast<const uint32_t*>(ws + 2048);
  p.x = xq; p.x_zero_row = 16; p.x_div = 1; p.groups_of_routes = groups; p.max_routes = 16;
  p.out = ws + 16384; p.out_dtype = KEEPVQ_BF16;
  for (int form = 0; form < 4; ++form) {
    if (form == 3 && (e = cudaMemsetAsync(p.out, 0xFF, 16 * 512 * 2, s)) != cudaSuccess) return note_cuda_error(e);
    p.out_dim = form == 0 ? 128 : 512;  // (the other forms take 256 rows an item: two items)
    p.groups = form == 1 ? 2 : 1;
    p.group_cols = form == 0 ? fast::PREFILL_GROUP_ROUTES : fast::PREFILL_GROUP_ROUTES_SMALL;
    const int rc = fast::prefill_wait_selftest(form, p, status + form, static_cast<uint64_t>(form == 0 ? wait_ns : std::min(wait_ns, SELFTEST_SHORT_NS)), s);
    if (rc) return rc;
  }
  // nothing of the second item (rows 256 on) may have been stored: its drain had nothing to store
  selftest_check_kernel<<<1, 256, 0, s>>>(static_cast<const uint16_t*>(p.out), 256, 0xFFFFu, status + 4);
  KEEPVQ_CHECK_LAUNCH();
  return KEEPVQ_OK;
}
