"""The few-token kernel (csrc/few_tokens.cu): a layer call of few routes as one launch.

Against the CPU oracle at the sizes where its shares of the work change shape: one to seven tokens (one,
two and four routes to a group, rows staged by token and by group, deep and shallow code rings),
fewer chunks than warps, scale groups that close inside a warp's run, a second group that begins in
a block's run.  Bound of the outputs: the layer's own (three roundings to the activation dtype)."""

import numpy as np
import pytest
import torch

import synthetic
from test_gpu_moe_layer import TOLERANCE, build_layer, check_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,experts,top_k,hidden,inter,group_hidden,group_inter,score", [
    (1, 20, 2, 256, 256, None, None, "softmax"),      # one chunk of inputs a row: fewer chunks than warps
    (2, 384, 6, 512, 256, None, 256, "sigmoid"),      # the largest pool the kernel's own router takes
    (4, 6, 5, 768, 512, 256, 256, "softmax"),         # several groups of four on one expert
    (7, 33, 6, 4096, 512, None, None, "softmax"),     # a scale group of sixteen chunks; 42 routes
    (3, 12, 6, 5120, 768, 512, 256, "sqrtsoftplus"),  # the widest rows, scale groups of two chunks and of one
    (8, 12, 5, 2560, 256, None, None, "softmax"),     # eight tokens staged by token, two rounds of picks
    (9, 12, 5, 512, 2304, 256, 768, "softmax"),       # rows staged by group
    (23, 40, 2, 512, 256, None, None, "softmax"),     # the most tokens
    (2, 400, 3, 512, 256, None, None, "softmax"),     # a pool whose router runs in front
    (12, 40, 2, 4096, 256, None, None, "sigmoid"),    # the most tokens with the router in the launch
    (13, 40, 2, 4096, 256, None, None, "sigmoid"),
    (16, 20, 2, 4352, 256, None, None, "softmax"),    # ... of wider rows; four rounds of picks
    (17, 20, 2, 4352, 256, None, None, "softmax"),
])
def test_layer_calls_of_few_routes(cuda, tokens, experts, top_k, hidden, inter, group_hidden, group_inter, score):
    cfg = synthetic.layer(seed=71, experts=experts, hidden=hidden, inter=inter, group_hidden=group_hidden, group_inter=group_inter)
    x = synthetic.tokens(72 + tokens, tokens, hidden)
    layer = build_layer(cuda, cfg, top_k=top_k, score_func=score)
    assert layer.launches_per_call(tokens) == (1 if experts <= 384 and tokens <= (16 if hidden > 4096 else 12) else 3)
    layer.decode(x.to(cuda))
    for buf in layer._buffers.values():
        buf["workspace"].fill_(0x7F)  # whatever the scratch holds, the barrier words of an earlier call among it
    out, routing = layer.decode(x.to(cuda))
    assert not layer.wait_expired(tokens, x.dtype)
    check_layer(cfg, x, out, routing, top_k=top_k, score_func=score)


@pytest.mark.parametrize("tokens,experts,top_k,launches", [
    (8, 96, 6, 1),    # 48 routes, half as many as slots
    (14, 168, 6, 3),  # the most routes
    (8, 95, 6, 7),    # one expert fewer: the chain of kernels
    (17, 400, 5, 7),  # one route more
])
def test_layer_calls_of_48_routes_and_more(cuda, tokens, experts, top_k, launches):
    cfg = synthetic.layer(seed=79, experts=experts, hidden=512, inter=256, group_hidden=256)
    x = synthetic.tokens(80 + tokens, tokens, 512)
    layer = build_layer(cuda, cfg, top_k=top_k)
    assert layer.launches_per_call(tokens) == launches
    out, routing = layer.decode(x.to(cuda))
    assert not layer.wait_expired(tokens, x.dtype)
    check_layer(cfg, x, out, routing, top_k=top_k)


def test_stage_by_stage_and_replayed_from_a_graph(cuda):
    """The parts of a call one after the other, and a captured call replayed (which finds its own
    barrier words in the scratch), give what the whole call gives, to the bit."""
    from keep_b200 import _lib

    cfg = synthetic.layer(seed=73, experts=16, hidden=1024, inter=512, group_hidden=256, group_inter=256)
    layer = build_layer(cuda, cfg, top_k=5)
    xs = [synthetic.tokens(74 + i, 5, 1024).to(cuda) for i in range(3)]
    want = [layer.decode(x)[0].clone() for x in xs]
    for x, w in zip(xs, want):
        for stage in (_lib.STAGE_ROUTER, _lib.STAGE_PREPARE, _lib.STAGE_GATE_UP, _lib.STAGE_DOWN, _lib.STAGE_COMBINE):
            got, _ = layer.decode(x, stages=stage, state=1)
        assert torch.equal(got, w)
    x = xs[0].clone()
    layer.decode(x, state=2)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got, _ = layer.decode(x, state=2)
    for i in (1, 2, 0, 1):
        x.copy_(xs[i])
        graph.replay()
        assert torch.equal(got, want[i])


@pytest.mark.parametrize("stages,absent", [("all", 1), ("all", 2), ("no router", 2), ("router and gate/up", 1)])
def test_a_block_that_stays_away_from_a_grid_barrier(cuda, stages, absent):
    """The other blocks' waits run out after 3 ms, the status says so, and nothing of the failed call is
    left for the next: calls with the same token (what a captured call's replays have) over the same
    scratch, on tokens of their own, pass no barrier before everybody is there."""
    from keep_b200 import _lib

    cfg = synthetic.layer(seed=83, experts=16, hidden=1024, inter=512)
    layer = build_layer(cuda, cfg, top_k=5)
    mask = {"all": _lib.STAGE_ALL, "no router": _lib.STAGE_ALL & ~_lib.STAGE_ROUTER, "router and gate/up": _lib.STAGE_ROUTER | _lib.STAGE_PREPARE | _lib.STAGE_GATE_UP}[stages]
    lib, token = _lib.load(), 0x0123456789ABCDEF
    xs = [synthetic.tokens(84 + i, 5, 1024).to(cuda) for i in range(4)]
    want = []
    for x in xs:
        out, _ = layer.decode(x)
        want.append((out.clone(), layer.route_hidden(5, x.dtype).clone()))
    buf = layer._buffers_for(5, torch.bfloat16)

    def call(i, absent):
        if not mask & _lib.STAGE_ROUTER:
            layer.decode(xs[i], stages=_lib.STAGE_ROUTER)
        args = layer._layer_args(xs[i], buf["out"], buf["routing"], workspace=buf["workspace"], nbytes=buf["nbytes"])
        _lib.check(lib.keepvq_grid_wait_selftest(args, mask, absent, 0, 3_000_000 if absent else 1_000_000_000, token, _lib.stream_handle(cuda)), "keepvq_grid_wait_selftest")
        torch.cuda.synchronize()
        words = buf["workspace"][: buf["nbytes"] // 8 * 8].view(torch.int64)
        assert not (words == token).any()
        return layer.wait_expired(5, torch.bfloat16)

    for i, away in enumerate((0, absent, absent, 0)):
        assert call(i, away) == bool(away)
        if not away:
            assert torch.equal(layer.route_hidden(5, torch.bfloat16), want[i][1])
            if mask & _lib.STAGE_COMBINE:
                assert torch.equal(buf["out"], want[i][0])


def test_a_reported_wait_stays_reported_through_later_stages(cuda):
    """A wait that ran out in one stage of a call is still in the status word after the stages behind it;
    the next call's PREPARE clears it."""
    from keep_b200 import _lib

    layer = build_layer(cuda, synthetic.layer(seed=85, experts=16, hidden=512, inter=256), top_k=4)
    x = synthetic.tokens(86, 3, 512).to(cuda)
    layer.decode(x)
    buf = layer._buffers_for(3, x.dtype)
    args = layer._layer_args(x, buf["out"], buf["routing"], workspace=buf["workspace"], nbytes=buf["nbytes"])
    front = _lib.STAGE_ROUTER | _lib.STAGE_PREPARE | _lib.STAGE_GATE_UP
    _lib.check(_lib.load().keepvq_grid_wait_selftest(args, front, 1, 0, 3_000_000, 77, _lib.stream_handle(cuda)), "keepvq_grid_wait_selftest")
    assert layer.wait_expired(3, x.dtype)
    layer.decode(x, stages=_lib.STAGE_DOWN)
    layer.decode(x, stages=_lib.STAGE_COMBINE)
    assert layer.wait_expired(3, x.dtype)
    layer.decode(x, stages=_lib.STAGE_PREPARE)
    assert not layer.wait_expired(3, x.dtype)
    for clearing in (front, _lib.STAGE_ALL):
        buf["workspace"].fill_(0x7F)
        layer.decode(x, stages=clearing)
        assert not layer.wait_expired(3, x.dtype)


@pytest.mark.parametrize("top_k,experts", [(4, 12), (3, 400)])  # with the router in the launch, and in front of it
def test_a_grid_that_cannot_be_resident_leaves_the_call_to_the_other_kernels(cuda, top_k, experts):
    """One block more than there are SMs is refused by the cooperative launch, as the device's own number
    is in a context that has fewer of them.  The layer call is then served by the chain of kernels,
    whole and in parts, and the refusal is not left behind as an error of a later call."""
    from keep_b200 import _lib

    cfg = synthetic.layer(seed=87, experts=experts, hidden=512, inter=256, group_hidden=256)
    layer = build_layer(cuda, cfg, top_k=top_k)
    x = synthetic.tokens(88, 6, 512).to(cuda)
    layer.decode(x)
    buf = layer._buffers_for(6, x.dtype)
    args = layer._layer_args(x, buf["out"], buf["routing"], workspace=buf["workspace"], nbytes=buf["nbytes"])
    too_many = torch.cuda.get_device_properties(cuda).multi_processor_count + 1

    def call(stages):
        _lib.check(_lib.load().keepvq_grid_wait_selftest(args, stages, 0, too_many, 1_000_000, 1, _lib.stream_handle(cuda)), "keepvq_grid_wait_selftest")

    front = _lib.STAGE_ROUTER | _lib.STAGE_PREPARE
    for steps in ((_lib.STAGE_ALL,), (front | _lib.STAGE_GATE_UP, _lib.STAGE_DOWN | _lib.STAGE_COMBINE), (front, _lib.STAGE_GATE_UP | _lib.STAGE_DOWN, _lib.STAGE_COMBINE)):
        buf["workspace"].fill_(0x7F)
        buf["out"].zero_()
        for stages in steps:
            call(stages)
        torch.cuda.synchronize()
        assert not layer.wait_expired(6, x.dtype)
        check_layer(cfg, x.cpu(), buf["out"], buf["routing"], top_k=top_k)


def test_a_stream_with_part_of_the_SMs(cuda):
    """A green context's stream: the grid of one block per SM of the device cannot be resident there, so
    the call goes to the chain of kernels, captured as well as eager, before a launch is refused."""
    drv = pytest.importorskip("cuda.bindings.driver")

    def did(result):
        assert result[0] == drv.CUresult.CUDA_SUCCESS, result[0]
        return result[1] if len(result) == 2 else result[1:]

    cfg = synthetic.layer(seed=92, experts=12, hidden=512, inter=256)
    layer = build_layer(cuda, cfg, top_k=4)
    x = synthetic.tokens(93, 5, 512).to(cuda)
    layer.decode(x)
    torch.cuda.synchronize()
    device = did(drv.cuDeviceGet(cuda.index))
    every = did(drv.cuDeviceGetDevResource(device, drv.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    parts = did(drv.cuDevSmResourceSplitByCount(1, every, 0, every.sm.smCount // 2))[0]
    green = did(drv.cuGreenCtxCreate(did(drv.cuDevResourceGenerateDesc(parts, 1)), device, drv.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM.value))
    handle = did(drv.cuGreenCtxStreamCreate(green, drv.CUstream_flags.CU_STREAM_NON_BLOCKING.value, 0))
    stream = torch.cuda.ExternalStream(int(handle), device=cuda)
    with torch.cuda.stream(stream):
        out, routing = layer.decode(x)
    stream.synchronize()
    check_layer(cfg, x.cpu(), out, routing, top_k=4)
    want = out.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        layer.decode(x)
    out.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        graph.replay()
    stream.synchronize()
    assert torch.equal(out, want)
    # (the stream and its context stay until the process ends: the allocator may know the stream)


def test_calls_on_two_streams_at_once(cuda):
    cfg = synthetic.layer(seed=75, experts=16, hidden=1024, inter=512)
    layer = build_layer(cuda, cfg, top_k=4)
    xs = [synthetic.tokens(76 + i, 4, 1024).to(cuda) for i in range(2)]
    want = [layer.decode(x)[0].clone() for x in xs]
    for i, x in enumerate(xs):
        layer.decode(x, state=1 + i)
    streams = [torch.cuda.Stream(cuda) for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(20):
        outs = []
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                outs.append(layer.decode(xs[i], state=1 + i)[0])
    torch.cuda.synchronize()
    assert all(torch.equal(o, w) for o, w in zip(outs, want))


def test_two_experts_of_one_slot_and_a_token_without_any(cuda):
    """`slot_of` may name a slot twice (a token then has it twice), and every pick of a token may be absent."""
    from oracle import router as oracle_router

    pool, hidden, inter, k = 6, 512, 256, 2
    cfg = synthetic.layer(seed=77, experts=pool, hidden=hidden, inter=inter)
    x = synthetic.tokens(78, 1, hidden)
    slot_of = np.array([0, 0, 1, 1, 2, 2], dtype=np.uint32)
    slot_cfg = dict(cfg)
    for n in ("w1", "w3", "w2"):
        slot_cfg[n] = (cfg[n][0][:3], cfg[n][1][:3])
    bias = np.array([0, 0, -1e30, -1e30, -1e30, -1e30], dtype=np.float32)
    layer = build_layer(cuda, slot_cfg, top_k=k, served_bias=bias, slot_of=slot_of)
    out, routing = layer.decode(x.to(cuda))
    assert sorted(routing.served_slot.cpu().view(-1).tolist()) == [0, 0]
    check_layer(slot_cfg, x, out, routing, top_k=k, served_bias=bias, slot_of=slot_of)
    nothing = build_layer(cuda, slot_cfg, top_k=k, served_bias=np.full(pool, oracle_router.OFF, dtype=np.float32), slot_of=slot_of)
    shared = torch.arange(hidden, dtype=torch.float32, device=cuda)[None]
    out, _ = nothing.decode(x.to(cuda), shared=shared)
    assert torch.equal(out, shared.to(out.dtype))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("routes,out_dim,in_dim,group", [(1, 72, 256, 256), (5, 40, 1024, 256), (47, 8, 512, 512), (11, 2304, 5120, 512), (4, 1, 256, 256)])
def test_single_projections_with_ragged_rows(cuda, dtype, routes, out_dim, in_dim, group):
    """One routed product, output rows that are no multiple of a unit's, against decoded weights in fp64;
    dead routes give zeros.  Bound: the 16-bit steps of the activations (2^-15 of a row's largest
    magnitude each, so at most that times the sum of the weights' magnitudes) and the output's rounding."""
    from keep_b200 import prefill, vq

    rng = np.random.default_rng(79)
    experts = 9
    codes = torch.from_numpy(rng.integers(0, 65536, (experts, out_dim, in_dim // 8)).astype(np.uint16)).to(cuda)
    scales = torch.from_numpy((0.02 * (0.5 + rng.random((experts, out_dim, in_dim // group)))).astype(np.float16)).to(cuda)
    x = torch.from_numpy(rng.standard_normal((routes, in_dim)).astype(np.float32)).to(cuda).to(dtype)
    rhs = torch.from_numpy(rng.integers(0, experts, routes).astype(np.int32)).to(cuda)
    rhs[routes // 2] = -1 if routes > 1 else int(rhs[0])
    y = prefill.tensor_core_projection(x, codes, scales, vq.table_on(cuda, "e8p"), rhs)
    w = vq.decode_weight_matrix(codes, scales, code_bits=16).double()[rhs.long().clamp(min=0)]
    want = torch.einsum("rk,rnk->rn", x.double(), w) * (rhs >= 0).double()[:, None]
    bound = 2.0 ** -15 * x.double().abs().amax(1, keepdim=True) * w.abs().sum(2) + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * want.abs() + 1e-7
    assert ((y.double() - want).abs() <= bound).all()
    assert not y[rhs < 0].any()


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
def test_rows_that_are_not_finite_touch_no_other(cuda, bad):
    """A row with a NaN or an infinity beside ordinary ones: theirs are the same bits as without it, and
    every row goes through the same steps as in calls of many routes (the slab kernels): equal but for
    fp32 sums in another order, which may round to the neighbouring bf16: 2^-7 of the value."""
    from keep_b200 import prefill, vq

    rng = np.random.default_rng(80)
    codes = torch.from_numpy(rng.integers(0, 65536, (4, 64, 64)).astype(np.uint16)).to(cuda)
    scales = torch.full((4, 64, 1), 0.02, dtype=torch.float16, device=cuda)
    x = torch.randn((60, 512), generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(cuda)
    rhs = (torch.arange(60, device=cuda) % 4).to(torch.int32)
    table = vq.table_on(cuda, "e8p")
    before = prefill.tensor_core_projection(x[:8].contiguous(), codes, scales, table, rhs[:8].contiguous())
    x[2, 100] = bad
    many = prefill.tensor_core_projection(x, codes, scales, table, rhs)[:8].float()
    few = prefill.tensor_core_projection(x[:8].contiguous(), codes, scales, table, rhs[:8].contiguous())
    others = [0, 1, 3, 4, 5, 6, 7]
    assert torch.equal(few[others], before[others]) and not torch.equal(few[2], before[2])
    few = few.float()
    assert torch.isfinite(few).all()
    assert ((few - many).abs() <= 2.0 ** -7 * many.abs() + 1e-6 * many.abs().amax(1, keepdim=True)).all()


@pytest.mark.parametrize("dtype,tolerance", [(torch.bfloat16, TOLERANCE), (torch.float16, TOLERANCE / 8)])  # three roundings of 8 or of 11 bits
def test_masked_picks_of_the_largest_pool(cuda, dtype, tolerance):
    """384 experts of which a third is resident, the demanded picks by a bias of their own, admissions;
    and the output written over the tokens."""
    from oracle import router as oracle_router

    pool, hidden, inter, k, tokens = 384, 512, 256, 6, 7
    rng = np.random.default_rng(89)
    cfg = synthetic.layer(seed=90, experts=pool, hidden=hidden, inter=inter)
    resident = np.sort(rng.choice(pool, pool // 3, replace=False))
    slot_of = np.full(pool, 0xFFFFFFFF, dtype=np.uint32)
    slot_of[resident] = rng.permutation(pool // 3).astype(np.uint32)
    served_bias = np.full(pool, oracle_router.OFF, dtype=np.float32)
    served_bias[resident] = rng.normal(scale=1e-3, size=pool // 3)
    pool_bias = rng.normal(scale=1e-3, size=pool).astype(np.float32)
    expert_of_slot = np.empty(pool // 3, dtype=np.int64)
    expert_of_slot[slot_of[resident].astype(np.int64)] = resident
    slot_cfg = dict(cfg, **{n: (cfg[n][0][expert_of_slot], cfg[n][1][expert_of_slot]) for n in ("w1", "w3", "w2")})
    x = synthetic.tokens(91, tokens, hidden).to(dtype)
    layer = build_layer(cuda, slot_cfg, top_k=k, served_bias=served_bias, pool_bias=pool_bias, slot_of=slot_of, tau=0.2)
    assert layer.launches_per_call(tokens, dtype) == 1
    out, routing = layer.decode(x.to(cuda))
    assert out.dtype == dtype and (routing.admit.cpu().numpy() >= 0).any()
    check_layer(slot_cfg, x, out, routing, top_k=k, served_bias=served_bias, pool_bias=pool_bias, slot_of=slot_of, tau=0.2, dtype=dtype, tolerance=tolerance)
    want, over = out.clone(), x.to(cuda).clone()
    assert torch.equal(layer.decode(over, out=over)[0], want)
