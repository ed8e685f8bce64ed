"""The routed operators (gather_vqmm family) against the oracle and the golden fixtures.

Mirrors tests/test_gather_vqmm.py:40-337 of the reference: gather = per-route qmv; the sorted path
scatters back to the caller's order; explicit lhs; mixed-expert tile boundaries; traces."""

import numpy as np
import pytest
import torch

from oracle import ops

pytestmark = pytest.mark.gpu


def f32(t):
    return t.float().cpu().numpy()


def test_golden_reference_outputs(cuda, golden):
    from keep_b200 import vq_switch

    g = golden("operators")
    kw = dict(input_dims=128, output_dims=24, group_size=32, code_bits=16)
    x = torch.from_numpy(g["x"]).to(cuda)
    for impl in ("cuda", "reference"):
        got = vq_switch.gather_vqmm(x, g["codes"], g["scales"], None, g["rhs"], implementation=impl, **kw)
        np.testing.assert_allclose(f32(got), g["token"], rtol=1e-5, atol=1e-5)
        got = vq_switch.gather_vqmm(x, g["codes"], g["scales"], None, g["flat_rhs"], lhs_indices=g["lhs"], implementation=impl, **kw)
        np.testing.assert_allclose(f32(got), g["routed"], rtol=1e-5, atol=1e-5)
        got = vq_switch.vq_switch_qmv(torch.from_numpy(g["xr"]).to(cuda), g["codes"], g["scales"], None, g["rhs"], implementation=impl, **kw)
        np.testing.assert_allclose(f32(got), g["per_route"], rtol=1e-5, atol=1e-5)
    got = vq_switch.gather_vqmm(x, g["codes8"], g["scales"], None, g["rhs"], **{**kw, "code_bits": 8})
    np.testing.assert_allclose(f32(got), g["token8"], rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("strategy", ["direct", "sorted_tiled", "per_route_decoded", "auto"])
@pytest.mark.parametrize("tokens,top_k", [(4, 3), (50, 6)])
def test_every_strategy_returns_the_callers_order(cuda, strategy, tokens, top_k):
    from keep_b200 import vq_switch

    rng = np.random.default_rng(31)
    experts, out, inp, group = 7, 40, 256, 64
    codes = rng.integers(0, 1 << 16, (experts, out, inp // 8), dtype=np.uint16)
    scales = rng.uniform(0.01, 0.2, (experts, out, inp // group)).astype(np.float16)
    x = rng.normal(size=(tokens, inp)).astype(np.float32)
    rhs = np.stack([rng.choice(experts, top_k, replace=False) for _ in range(tokens)]).astype(np.int64)
    want = ops.gather_vqmm(x, codes, scales, None, rhs, code_bits=16)
    with vq_switch.trace_gather_vqmm_calls() as trace:
        got = vq_switch.gather_vqmm(torch.from_numpy(x).to(cuda), codes, scales, None, rhs, input_dims=inp, output_dims=out,
                                    group_size=group, code_bits=16, route_strategy=strategy)
    np.testing.assert_allclose(f32(got), want, rtol=1e-4, atol=1e-3)
    assert trace[0]["route_count"] == tokens * top_k
    if strategy == "auto":
        assert trace[0]["strategy"] == ("sorted_tiled" if tokens * top_k >= 128 else "direct")


def test_sorted_routes_with_explicit_descriptors_and_boundaries(cuda):
    from keep_b200 import vq_switch

    rng = np.random.default_rng(32)
    experts, out, inp, group = 5, 24, 128, 32
    codes = rng.integers(0, 1 << 16, (experts, out, inp // 8), dtype=np.uint16)
    scales = rng.uniform(0.01, 0.2, (experts, out, inp // group)).astype(np.float16)
    x = rng.normal(size=(9, inp)).astype(np.float32)
    sorted_rhs = np.array([0] * 3 + [2] * 37 + [4] * 2, dtype=np.int32)  # expert 1 and 3 unused; 2 spans tiles
    sorted_lhs = rng.integers(0, 9, sorted_rhs.shape[0]).astype(np.int32)
    want = ops.gather_vqmm(x, codes, scales, None, sorted_rhs, lhs_indices=sorted_lhs, code_bits=16)
    xt = torch.from_numpy(x).to(cuda)
    tiles = vq_switch.expert_block_tile_descriptors(torch.from_numpy(sorted_rhs).to(cuda), num_experts=experts, route_tile=32)
    te, to, tc = (t.cpu().numpy() for t in tiles)
    assert te.shape[0] == 2 + experts and tc.sum() == sorted_rhs.shape[0]
    assert [(int(e), int(o), int(c)) for e, o, c in zip(te, to, tc) if c] == [(0, 0, 3), (2, 3, 32), (2, 35, 5), (4, 40, 2)]
    got = vq_switch.gather_vqmm_sorted_routes(xt, codes, scales, None, sorted_rhs, sorted_lhs, input_dims=inp, output_dims=out,
                                              group_size=group, code_bits=16, validate_indices=True, tile_descriptors=tiles)
    np.testing.assert_allclose(f32(got), want, rtol=1e-4, atol=1e-3)
    with pytest.raises(ValueError, match="sorted nondecreasing"):
        vq_switch.gather_vqmm_sorted_routes(xt, codes, scales, None, sorted_rhs[::-1].copy(), sorted_lhs, input_dims=inp,
                                            output_dims=out, group_size=group, code_bits=16, validate_indices=True)
    empty = vq_switch.gather_vqmm_sorted_routes(xt, codes, scales, None, sorted_rhs[:0], sorted_lhs[:0], input_dims=inp,
                                                output_dims=out, group_size=group, code_bits=16)
    assert tuple(empty.shape) == (0, out)


def test_metadata_errors_match_the_reference_messages(cuda):
    from keep_b200 import vq_switch

    x = torch.zeros((2, 64), device=cuda)
    codes = torch.zeros((3, 8, 8), dtype=torch.uint16, device=cuda)
    scales = torch.ones((3, 8, 2), device=cuda)
    rhs = torch.zeros((2, 2), dtype=torch.int64, device=cuda)
    kw = dict(input_dims=64, output_dims=8, group_size=32, code_bits=16)
    with pytest.raises(ValueError, match="route_strategy must be"):
        vq_switch.gather_vqmm(x, codes, scales, None, rhs, route_strategy="tiled", **kw)
    with pytest.raises(ValueError, match="rhs_indices token dimension"):
        vq_switch.gather_vqmm(x, codes, scales, None, rhs[:1], **kw)
    with pytest.raises(ValueError, match="codes must have shape"):
        vq_switch.gather_vqmm(x, codes[:, :4], scales, None, rhs, **kw)
    with pytest.raises(ValueError, match="codes dtype must be uint16"):
        vq_switch.gather_vqmm(x, codes.to(torch.uint8), scales, None, rhs, **kw)
    with pytest.raises(ValueError, match=r"indices must be in \[0, 3\)"):
        vq_switch.gather_vqmm(x, codes, scales, None, rhs + 3, implementation="reference", **kw)
    with pytest.raises(ValueError, match="same flattened shape"):
        vq_switch.gather_vqmm(x, codes, scales, None, rhs.reshape(-1), lhs_indices=torch.zeros(3, dtype=torch.int32, device=cuda), **kw)


@pytest.mark.parametrize("routes,experts", [(300, 6), (1500, 6), (1200, 40)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sorted_routes_on_the_tensor_core_kernels(cuda, routes, experts, dtype):
    """Prefill-shaped sorted calls (16-bit codes, in_dim % 256 == 0, one scale group per row) with
    bf16 activations run keepvq_grouped_projection: the mma.sync kernel for 300 routes, the tcgen05
    kernel for 1500 routes over 6 experts, the mma.sync one again for 1200 routes spread over 40
    experts; the only rounding there is the 16-bit fixed-point step on the activations.  fp32
    activations are not narrowed: they take the general kernel (24-bit fixed point)."""
    from keep_b200 import prefill, vq, vq_switch

    rng = np.random.default_rng(90 + routes)
    out, inp, tokens = 136, 512, 64
    codes = rng.integers(0, 1 << 16, (experts, out, inp // 8), dtype=np.uint16)
    scales = (0.02 * rng.uniform(0.5, 1.5, (experts, out, 1))).astype(np.float16)
    x = torch.from_numpy(rng.normal(size=(tokens, inp)).astype(np.float32)).to(dtype)
    rhs = np.sort(rng.integers(0, experts - 1, routes)).astype(np.int64)  # the last expert gets no route
    lhs = rng.integers(0, tokens, routes).astype(np.int64)
    want = ops.gather_vqmm(x.float().numpy(), codes, scales, None, rhs, lhs_indices=lhs, code_bits=16)
    got = vq_switch.gather_vqmm_sorted_routes(x.to(cuda), codes, scales, None, rhs, lhs, input_dims=inp, output_dims=out,
                                              group_size=inp, code_bits=16, validate_indices=True)
    assert got.dtype == dtype and tuple(got.shape) == (routes, out)
    tol = dict(rtol=1e-4, atol=3e-4) if dtype == torch.float32 else dict(rtol=1e-2, atol=1e-2)
    np.testing.assert_allclose(f32(got), want, **tol)
    rows = x.to(cuda)[torch.from_numpy(lhs).to(cuda)]
    direct = prefill.tensor_core_projection(rows, torch.from_numpy(codes).to(cuda), torch.from_numpy(scales).to(cuda),
                                            vq.table_on(cuda, "e8p"), torch.from_numpy(rhs).to(cuda))
    if dtype == torch.float32:
        assert direct is None
    else:
        assert direct is not None and torch.equal(direct, got)  # the operator did take this entry point


@pytest.mark.parametrize("out,inp,group", [(100, 256, 256), (200, 512, 256), (300, 768, 256), (640, 512, 512)])
def test_sorted_routes_with_ragged_rows_and_scale_groups(cuda, out, inp, group):
    """Row counts that no tile divides (the tcgen05 kernels' code boxes then run into the next
    expert's rows, or past the last), one item tile and several, one scale group and several."""
    from keep_b200 import vq_switch

    rng = np.random.default_rng(23)
    experts, routes = 7, 1100
    codes = rng.integers(0, 1 << 16, (experts, out, inp // 8), dtype=np.uint16)
    scales = (0.02 * rng.uniform(0.5, 1.5, (experts, out, inp // group))).astype(np.float16)
    x = torch.from_numpy(rng.normal(size=(routes, inp)).astype(np.float32)).to(torch.bfloat16)
    rhs = np.sort(rng.integers(0, experts, routes)).astype(np.int64)
    lhs = np.arange(routes)
    want = ops.gather_vqmm(x.float().numpy(), codes, scales, None, rhs, lhs_indices=lhs, code_bits=16)
    got = vq_switch.gather_vqmm_sorted_routes(x.to(cuda), codes, scales, None, rhs, lhs, input_dims=inp, output_dims=out,
                                              group_size=group, code_bits=16, validate_indices=True)
    np.testing.assert_allclose(f32(got), want, rtol=1e-2, atol=1e-2)


def test_routes_without_an_expert_give_zero_rows_on_every_path(cuda):
    """A route whose index names no expert (0xFFFFFFFF, or any value past the last expert) returns
    a row of zeros from the tensor-core kernels and from the general kernel alike."""
    from keep_b200 import kernels, prefill, vq

    rng = np.random.default_rng(21)
    experts, out, inp = 4, 64, 256
    codes = rng.integers(0, 1 << 16, (experts, out, inp // 8), dtype=np.uint16)
    scales = (0.02 * rng.uniform(0.5, 1.5, (experts, out, 1))).astype(np.float16)
    table = vq.table_on(cuda, "e8p")
    for routes in (6, 64):  # the few-token kernel and the slab kernel
        rhs = rng.integers(0, experts, routes).astype(np.int64)
        rhs[1], rhs[routes - 2] = 0xFFFFFFFF, experts + 3
        x = torch.from_numpy(rng.normal(size=(routes, inp)).astype(np.float32)).to(cuda)
        dead = torch.tensor([1, routes - 2])
        rhs_t = torch.from_numpy(rhs.astype(np.uint32).view(np.int32)).to(cuda)
        fast = prefill.tensor_core_projection(x.to(torch.bfloat16), torch.from_numpy(codes).to(cuda), torch.from_numpy(scales).to(cuda), table, rhs_t)
        assert fast is not None and bool((fast[dead] == 0).all()) and bool((fast[0] != 0).any())
        general = kernels.e8p_m1_per_route(x, codes, scales, table, rhs.astype(np.uint32), output_dims=out)
        assert bool((general[dead] == 0).all()) and bool((general[0] != 0).any())


@pytest.mark.parametrize("routes,experts,out,inp,group", [
    (12, 3, 100, 256, 256),     # the fewest routes, one partial row tile
    (144, 96, 384, 1024, 1024),  # about a route per expert, a partial item
    (130, 2, 256, 512, 256),    # two 48-route items and a short one per expert, two scale groups of two K blocks
    (600, 40, 300, 768, 256),   # ragged rows, three scale groups
])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_8bit_codes_on_the_tcgen05_kernel(cuda, dtype, routes, experts, out, inp, group):
    """8-bit codes with enough routes for the grouped kernel, through both operators, and the same
    routes on the general kernel: two 16-bit fixed-point paths, apart by the output's rounding."""
    from keep_b200 import kernels, prefill, vq, vq_switch

    rng = np.random.default_rng(25)
    codes = rng.integers(0, 256, (experts, out, inp // 8), dtype=np.uint8)
    scales = (0.02 * rng.uniform(0.5, 1.5, (experts, out, inp // group))).astype(np.float16)
    table = vq.table_on(cuda, "e8_1bit")
    dev = lambda a: torch.from_numpy(a).to(cuda)  # noqa: E731
    rhs = rng.integers(0, experts, routes).astype(np.int32)
    x = torch.from_numpy(rng.normal(size=(routes, inp)).astype(np.float32)).to(dtype)
    want = ops.gather_vqmm(x.float().numpy(), codes, scales, None, rhs.astype(np.int64), lhs_indices=np.arange(routes), code_bits=8)
    named = dict(input_dims=inp, output_dims=out, group_size=group, code_bits=8)
    tokens = vq_switch.gather_vqmm(x.to(cuda), dev(codes), dev(scales), table, dev(rhs).reshape(routes, 1), **named)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10
    atol = 2.0 ** -14 * np.abs(want).max() * 8  # the fixed-point step of a row against its largest output
    np.testing.assert_allclose(f32(tokens).reshape(routes, out), want, rtol=eps, atol=atol)
    general = kernels.routed_matvec(x.to(cuda), dev(codes), dev(scales), table, dev(rhs), code_bits=8)
    np.testing.assert_allclose(f32(tokens).reshape(routes, out), f32(general), rtol=eps, atol=atol)
    direct = prefill.tensor_core_projection(x.to(cuda), dev(codes), dev(scales), table, dev(rhs), code_bits=8)
    assert direct is not None and torch.equal(direct, tokens.reshape(routes, out))
    dead = rhs.copy()
    dead[1] = experts + 2
    with_dead = prefill.tensor_core_projection(x.to(cuda), dev(codes), dev(scales), table, dev(dead), code_bits=8)
    assert bool((with_dead[1] == 0).all()) and torch.equal(with_dead[2:], direct[2:])


@pytest.mark.parametrize("routes,experts,out,inp,grouped", [
    (11, 1, 2048, 2048, False), (12, 64, 1024, 2048, False), (12, 64, 2048, 2048, True), (12, 4, 128, 256, True), (24, 9, 256, 512, False), (24, 8, 256, 512, True),
    (24, 64, 512, 1024, True), (47, 64, 256, 512, False), (48, 64, 256, 512, True), (95, 64, 128, 256, False), (96, 64, 128, 256, True),
])
def test_8bit_codes_take_the_kernel_that_is_faster_for_their_size(cuda, routes, experts, out, inp, grouped):
    """Both sides of every line of the rule for 8-bit codes, and the same outputs from the operator on either."""
    from keep_b200 import kernels, prefill, vq, vq_switch

    gen = torch.Generator(device=cuda).manual_seed(29)
    codes = torch.randint(0, 256, (experts, out, inp // 8), generator=gen, device=cuda, dtype=torch.uint8)
    scales = torch.full((experts, out, 1), 0.02, dtype=torch.float16, device=cuda)
    x = torch.randn((routes, inp), generator=gen, device=cuda).to(torch.bfloat16)
    rhs = torch.randint(0, experts, (routes, 1), generator=gen, device=cuda).to(torch.int32)
    table = vq.table_on(cuda, "e8_1bit")
    assert (prefill.tensor_core_projection(x, codes, scales, table, rhs.reshape(-1), code_bits=8) is not None) == grouped
    got = vq_switch.gather_vqmm(x, codes, scales, table, rhs, input_dims=inp, output_dims=out, group_size=inp, code_bits=8)
    want = kernels.routed_matvec(x, codes, scales, table, rhs.reshape(-1), code_bits=8)
    atol = 2.0 ** -11 * float(want.float().abs().max())  # the fixed-point step of a row against its largest output
    np.testing.assert_allclose(f32(got).reshape(routes, out), f32(want), rtol=2.0 ** -8, atol=atol)


@pytest.mark.parametrize("bits,inp,word,code", [
    (8, 8192, 0x00000000, 0), (8, 8704, 0x00000000, 0), (8, 66560, 0x00000000, 0),  # every weight -4
    (16, 8192, 0x11111111, 0), (16, 10240, 0x11111111, 0),  # an all-odd table: every weight -3.25
    (16, 66560, 0x11111111, 0),  # wider than the tcgen05 kernel's sums: another kernel takes it
])
def test_wide_rows_keep_their_integer_sums(cuda, bits, inp, word, code):
    """The largest sums a caller's own table allows: constant rows against constant weights.  From
    8257 inputs on 8 * 32,512 * inputs passes 32 bits, from 66,053 on sum(x') itself."""
    from keep_b200 import vq_switch

    routes, out = 1024, 32
    table = np.full(256, word, dtype=np.uint32)
    codes = np.full((1, out, inp // 8), code, dtype=np.uint8 if bits == 8 else np.uint16)
    scales = np.full((1, out, 1), 2.0 ** -12, dtype=np.float16)
    weight = ops.dense_experts(codes[:, :1], scales[:, :1], code_bits=bits, codebook=table, dtype=np.float64)[0, 0]
    value = 127 / 64  # 32,512 steps of 2^-14: a bf16 value near the top of the fixed-point range (32,639)
    x = torch.full((routes, inp), value, dtype=torch.bfloat16, device=cuda)
    got = vq_switch.gather_vqmm(x, torch.from_numpy(codes).to(cuda), torch.from_numpy(scales).to(cuda), torch.from_numpy(table.view(np.int32)).to(cuda),
                                torch.zeros((routes, 1), dtype=torch.int32, device=cuda), input_dims=inp, output_dims=out, group_size=inp, code_bits=bits)
    want = np.full((routes, 1, out), weight.sum() * value)
    np.testing.assert_allclose(f32(got), want, rtol=2.0 ** -8)  # exact sums, one rounding to bf16


def test_a_codebook_written_just_before_the_call(cuda):
    """A table that a kernel on the stream changes in place between calls: each call decodes the words it finds."""
    from keep_b200 import kernels, vq_switch

    gen = torch.Generator(device=cuda).manual_seed(29)
    codes = torch.randint(0, 256, (4, 256, 64), generator=gen, device=cuda, dtype=torch.uint8)
    scales = torch.full((4, 256, 1), 0.02, dtype=torch.float16, device=cuda)
    x = torch.randn((64, 512), generator=gen, device=cuda).to(torch.bfloat16)
    rhs = torch.randint(0, 4, (64, 2), generator=gen, device=cuda, dtype=torch.int32)
    tables = torch.randint(-2 ** 31, 2 ** 31 - 1, (8, 256), generator=gen, device=cuda, dtype=torch.int32)
    want = [kernels.routed_matvec(x, codes, scales, t, rhs.reshape(-1), x_div=2, code_bits=8).reshape(64, 2, 256) for t in tables]
    table = torch.empty(256, dtype=torch.int32, device=cuda)
    torch.cuda.synchronize()
    got = []
    for t in tables.repeat(8, 1):
        torch.add(t, 0, out=table)  # a kernel, not a copy
        got.append(vq_switch.gather_vqmm(x, codes, scales, table, rhs, input_dims=512, output_dims=256, group_size=512, code_bits=8))
    for i, y in enumerate(got):
        assert ((y.float() - want[i % 8].float()).norm() / want[i % 8].float().norm()).item() < 4e-3  # two roundings to bf16


def test_calls_on_two_streams_do_not_share_scratch(cuda):
    """The same shapes on two streams that may overlap, 8-bit and 16-bit codes: each call's own result."""
    from keep_b200 import vq, vq_switch

    rng = np.random.default_rng(27)
    named = dict(input_dims=512, output_dims=1024, group_size=512)
    streams = [torch.cuda.Stream(cuda) for _ in range(2)]
    for bits, table in ((8, vq.table_on(cuda, "e8_1bit")), (16, vq.table_on(cuda, "e8p"))):
        codes = torch.from_numpy(rng.integers(0, 1 << bits, (8, 1024, 64), dtype=np.uint8 if bits == 8 else np.uint16)).to(cuda)
        scales = torch.full((8, 1024, 1), 0.02, dtype=torch.float16, device=cuda)
        xs = [torch.from_numpy(rng.normal(size=(64, 512)).astype(np.float32)).to(cuda).to(torch.bfloat16) for _ in range(2)]
        rhs = [torch.from_numpy(rng.integers(0, 8, (64, 2)).astype(np.int32)).to(cuda) for _ in range(2)]
        want = [vq_switch.gather_vqmm(xs[i], codes, scales, table, rhs[i], code_bits=bits, **named) for i in range(2)]
        torch.cuda.synchronize()
        got = [[], []]
        for _ in range(20):
            for i, s in enumerate(streams):
                with torch.cuda.stream(s):
                    got[i].append(vq_switch.gather_vqmm(xs[i], codes, scales, table, rhs[i], code_bits=bits, **named))
        torch.cuda.synchronize()
        assert all(torch.equal(y, want[i]) for i in range(2) for y in got[i])


@pytest.mark.parametrize("bits", [8, 16])
@pytest.mark.parametrize("out,inp,role", [(512, 256, "down"), (256, 512, "gate_up")])
def test_the_trace_of_a_sorted_call_names_its_projection(cuda, bits, out, inp, role):
    """From 128 routes on (or when asked for) a call leaves the operator's record and the expert-grouped
    dispatch's, which names the projection; a direct call leaves one."""
    from keep_b200 import vq_switch

    codes = torch.zeros((4, out, inp // 8), dtype=torch.uint8 if bits == 8 else torch.uint16, device=cuda)
    scales = torch.ones((4, out, 1), dtype=torch.float16, device=cuda)
    named = dict(input_dims=inp, output_dims=out, group_size=inp, code_bits=bits)
    for tokens, strategy, records in ((64, "auto", 2), (10, "auto", 1), (10, "sorted_tiled", 2), (64, "direct", 1)):
        x, rhs = torch.ones((tokens, inp), dtype=torch.bfloat16, device=cuda), torch.zeros((tokens, 2), dtype=torch.int32, device=cuda)
        with vq_switch.trace_gather_vqmm_calls() as trace:
            vq_switch.gather_vqmm(x, codes, scales, None, rhs, route_strategy=strategy, **named)
        first = dict(token_rows=tokens, route_count=2 * tokens, input_dims=inp, output_dims=out, code_bits=bits, implementation="cuda",
                     strategy="sorted_tiled" if records == 2 else "direct")
        assert trace == [first, dict(first, projection=role)][:records]


def _calls_of_one_shape(cuda, count):
    """``count`` argument lists of one shape (100 tokens of top-2 over 8 experts) with inputs of their own, and their results."""
    from keep_b200 import vq, vq_switch

    rng = np.random.default_rng(28)
    table = vq.table_on(cuda, "e8p")
    codes = torch.from_numpy(rng.integers(0, 1 << 16, (8, 1024, 64), dtype=np.uint16)).to(cuda)
    scales = torch.full((8, 1024, 1), 0.02, dtype=torch.float16, device=cuda)
    named = dict(input_dims=512, output_dims=1024, group_size=512, code_bits=16)
    calls = []
    for _ in range(count):
        x = torch.from_numpy(rng.normal(size=(100, 512)).astype(np.float32)).to(cuda).to(torch.bfloat16)
        rhs = torch.from_numpy(rng.integers(0, 8, (100, 2)).astype(np.int32)).to(cuda)
        calls.append(lambda x=x, rhs=rhs: vq_switch.gather_vqmm(x, codes, scales, table, rhs, **named))
    want = [call() for call in calls]
    torch.cuda.synchronize()
    return calls, want


def test_two_host_threads_on_one_stream_do_not_share_scratch(cuda):
    """Threads start on the same (default) stream; each call's launches may fall between another's."""
    from concurrent.futures import ThreadPoolExecutor

    calls, want = _calls_of_one_shape(cuda, 2)
    with ThreadPoolExecutor(2) as pool:
        got = list(pool.map(lambda i: [calls[i]() for _ in range(200)], range(2)))
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i]) for i in range(2) for y in got[i])


def test_captured_graphs_of_one_shape_replay_side_by_side(cuda):
    """Two graphs captured one after the other (torch captures both on one stream), replayed on two
    streams with calls of many other shapes in between."""
    from keep_b200 import kernels

    calls, want = _calls_of_one_shape(cuda, 2)
    graphs, outs = [], []
    for call in calls:
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            outs.append([call() for _ in range(10)])
    codes, scales = torch.zeros((64, 32), dtype=torch.uint16, device=cuda), torch.ones((64, 1), dtype=torch.float16, device=cuda)
    for rows in range(50, 70):
        kernels.vq_qmm(torch.ones((rows, 256), dtype=torch.bfloat16, device=cuda), codes, scales, in_dim=256, out_dim=64, group_size=256, code_bits=16)
    streams = [torch.cuda.Stream(cuda) for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(10):
        for s, g in zip(streams, graphs):
            with torch.cuda.stream(s):
                g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i]) for i in range(2) for y in outs[i])


def test_rows_that_start_inside_an_allocation(cuda):
    """A view whose first row is not on a 16-byte boundary, few routes and many: the same outputs."""
    from keep_b200 import vq, vq_switch

    rng = np.random.default_rng(26)
    codes = torch.from_numpy(rng.integers(0, 1 << 16, (4, 128, 32), dtype=np.uint16)).to(cuda)
    scales = torch.full((4, 128, 1), 0.02, dtype=torch.float16, device=cuda)
    for tokens in (4, 100):
        base = torch.from_numpy(rng.normal(size=tokens * 256 + 1).astype(np.float32)).to(cuda).to(torch.bfloat16)
        view = base[1:].reshape(tokens, 256)
        rhs = torch.from_numpy(rng.integers(0, 4, (tokens, 2)).astype(np.int32)).to(cuda)
        named = dict(input_dims=256, output_dims=128, group_size=256, code_bits=16)
        table = vq.table_on(cuda, "e8p")
        assert torch.equal(vq_switch.gather_vqmm(view, codes, scales, table, rhs, **named), vq_switch.gather_vqmm(view.clone(), codes, scales, table, rhs, **named))


@pytest.mark.parametrize("routes,inp", [(6, 256), (64, 2560), (64, 8448), (1100, 2560), (1100, 2816)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_activation_rows_as_fixed_point(cuda, dtype, routes, inp):
    """The 16-bit fixed-point rows behind every tensor-core projection, through products whose sums
    are exact: codes that decode to one of two rows, inputs that are whole steps.  Widths at the
    edges of what a warp or a block keeps in registers; a row with an infinity (step 1, clamped to
    +-32639), a NaN (counts as zero), all zeros, and the largest value two signed bytes hold."""
    from keep_b200 import prefill, vq

    rng = np.random.default_rng(24)
    experts, out = 2, 64
    codes = rng.integers(0, 1 << 16, (experts, out, inp // 8), dtype=np.uint16)
    scales = np.full((experts, out, 1), 2.0 ** -6, dtype=np.float16)
    dense = ops.dense_experts(codes, scales, dtype=np.float64)
    x = rng.integers(-64, 65, (routes, inp)).astype(np.float32)
    x[0] = 0.0
    x[1, 5], x[1, 9] = np.inf, -np.inf
    x[2, 3] = np.nan
    x[3, 7] = 65280.0 if dtype == torch.bfloat16 else 65504.0  # in fixed point past 127 * 256 + 127: the step doubles
    fixed = np.nan_to_num(x.astype(np.float64), nan=0.0, posinf=32639.0, neginf=-32639.0)
    step = 4.0  # of the row with the large value: 65280 / 2 and 65504 / 2 exceed 32639
    fixed[3] = np.round(fixed[3] / step) * step
    rhs = (np.arange(routes) % experts).astype(np.int32)
    got = prefill.tensor_core_projection(torch.from_numpy(x).to(cuda).to(dtype), torch.from_numpy(codes).to(cuda), torch.from_numpy(scales).to(cuda),
                                         vq.table_on(cuda, "e8p"), torch.from_numpy(rhs).to(cuda)).double().cpu().numpy()
    want = np.stack([dense[rhs[r]] @ fixed[r] for r in range(routes)])
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10  # the output's own rounding; fp32 sums are far below it
    top = np.abs(want[np.isfinite(want)]).max() if dtype == torch.bfloat16 else 65504.0
    np.testing.assert_allclose(np.clip(got, -top, top), np.clip(want, -top, top), rtol=eps, atol=1e-3 * step)


@pytest.mark.parametrize("factor", [300.0, 3000.0])
def test_one_outlier_channel_costs_what_the_header_says(cuda, factor):
    """fp16 / bf16 rows are held as 16-bit fixed point with one power-of-two step per row, so a
    channel far above the rest takes precision from the small channels.  Bounds stated beside
    ``keepvq_grouped_projection``: against the true output the gap stays near 1e-3 of its largest
    magnitude; against the output the row would give without the outlier channel it is below 1 %
    at 300 times the row's RMS and below 5 % at 3000 times.  fp32 rows go to the general kernel,
    which keeps 24 bits of a row: 256 times tighter."""
    from keep_b200 import kernels, prefill, vq

    rng = np.random.default_rng(22)
    experts, out, inp, routes = 2, 256, 4096, 64
    codes = rng.integers(0, 1 << 16, (experts, out, inp // 8), dtype=np.uint16)
    scales = (0.02 * rng.uniform(0.5, 1.5, (experts, out, 1))).astype(np.float16)
    dense = ops.dense_experts(codes, scales, dtype=np.float64)
    rhs = rng.integers(0, experts, routes).astype(np.uint32)
    x = rng.normal(size=(routes, inp)).astype(np.float32)
    x[:, 7] = factor
    xb = torch.from_numpy(x).to(cuda).to(torch.bfloat16)
    xn = xb.float().cpu().numpy().astype(np.float64)
    want = np.stack([xn[r] @ dense[e].T for r, e in enumerate(rhs)])
    quiet = xn.copy()
    quiet[:, 7] = 0.0
    want_quiet = np.stack([quiet[r] @ dense[e].T for r, e in enumerate(rhs)])
    table = vq.table_on(cuda, "e8p")
    got = prefill.tensor_core_projection(xb, torch.from_numpy(codes).to(cuda), torch.from_numpy(scales).to(cuda), table,
                                         torch.from_numpy(rhs.view(np.int32)).to(cuda)).float().cpu().numpy()
    # bf16 output rounding alone is 2^-9 relative; the activation step adds the rest
    assert np.abs(got - want).max() <= 6e-3 * np.abs(want).max()
    noise = np.abs((got - want)).max() / np.abs(want_quiet).max()
    assert noise <= (0.01 if factor == 300.0 else 0.05) + 2 ** -8 * np.abs(want).max() / np.abs(want_quiet).max(), noise
    # fp32 rows: 24-bit fixed point in the general kernel
    got32 = kernels.e8p_m1_per_route(torch.from_numpy(xn.astype(np.float32)).to(cuda), codes, scales, table, rhs, output_dims=out).cpu().numpy()
    assert np.abs(got32 - want).max() <= (5e-5 if factor == 300.0 else 4e-4) * np.abs(want_quiet).max()
