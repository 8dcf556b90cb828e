"""The few-row FP4 linear (1 to 16 rows of W4A16) at the edges of its token tiles (8, 16),
of its 16-row units and of its chunks of K, and the first sizes of the bf16 route behind it, against the float32 oracles.  Tolerance: one bf16 rounding of the result
(2^-9) and the order of a float32 sum of at most 8192 exact products, the bar every other route is held to."""
import numpy as np
import pytest
import torch

import fp4_oracle as o
from gpu_util import REL_TOL_TIGHT, REL_TOL_VS_ORACLE, bits_of, to_dev_bf16, to_dev_u8

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from glm_asr_stack_b200 import ops as _ops
    yield _ops
    assert _ops.status() == 0


def dev(ops, w):
    return ops.Fp4Tensor(to_dev_u8(w[0]), to_dev_u8(w[1]), w[2])


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("N,K", [(16, 256), (272, 2048), (48, 8192), (4752, 512)])
def test_store_and_bias(ops, M, N, K):
    w, x = o.seeded_weight(N, K, N + K), o.seeded_activation(M, K, M)
    bias = o.seeded_activation(1, N, 3)[0]
    d = dev(ops, w)
    out = bits_of(ops.fp4_linear(to_dev_bf16(x), d.w_packed, d.w_scales, d.w_global_scale, None, to_dev_bf16(bias)))
    assert o.rel_err(out, o.fp4_linear(x, *w, None, bias)) <= REL_TOL_TIGHT
    if M <= 8:
        isc = o.default_input_scale(x)
        got = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
        assert ops.nvfp4_linear(got, to_dev_bf16(x), d.w_packed, d.w_scales, isc, d.w_global_scale) == 0
        assert o.rel_err(bits_of(got), o.nvfp4_linear(x, w[0], w[1], isc, w[2])) <= REL_TOL_TIGHT


@pytest.mark.parametrize("M", [1, 8, 13, 19])
def test_segments_gate_and_residual(ops, M):
    K = 512
    x = o.seeded_activation(M, K, M)
    ws = [o.seeded_weight(n, K, n) for n in (2384, 32, 80)]
    out = bits_of(ops.fp4_linear_fused(ops.MODE_W4A16, to_dev_bf16(x), [dev(ops, w) for w in ws]))
    for w, c in zip(ws, (0, 2384, 2416)):
        assert o.rel_err(out[:, c:c + w[0].shape[0]], o.linear_o1(x, *w)) <= REL_TOL_TIGHT
    g, u = o.seeded_weight(2416, K, 5), o.seeded_weight(2416, K, 6)
    act = bits_of(ops.fp4_linear_fused(ops.MODE_W4A16, to_dev_bf16(x), [dev(ops, g), dev(ops, u)], epilogue=ops.EPI_SILU_GATE))
    want = o.silu_mul_split_packed(np.concatenate([o.linear_o1(x, *g), o.linear_o1(x, *u)], axis=1))
    assert o.rel_err(act, want) <= REL_TOL_VS_ORACLE
    res = to_dev_bf16(o.seeded_activation(M, 2384, 9))
    want = o.residual_add(o.linear_o1(x, *ws[0]), bits_of(res))
    ops.fp4_linear_fused(ops.MODE_W4A16, to_dev_bf16(x), [dev(ops, ws[0])], epilogue=ops.EPI_RESIDUAL, residual=res, out=res)
    assert o.rel_err(bits_of(res), want) <= REL_TOL_TIGHT


def test_scale_codes(ops):
    """Every e4m3 scale byte, subnormal, 0x7F (480 here, not a NaN) and negative ones included, times every e2m1 code."""
    N, K = 256, 256
    packed = np.tile(np.arange(128, dtype=np.uint8) * 2 + 1, (N, 1))
    scales = np.repeat(np.arange(256, dtype=np.uint8)[:, None], K // 16, axis=1)
    for k0 in (0, 100):
        x = np.zeros((2, K), np.float32)
        x[0, k0:k0 + 16], x[1, k0 + 16:k0 + 32:2] = 1.0, -0.5
        xb = (x.view(np.uint32) >> 16).astype(np.uint16)
        out = ops.fp4_linear(to_dev_bf16(xb), to_dev_u8(packed), to_dev_u8(scales), 1.0)
        assert o.rel_err(bits_of(out), o.linear_o1(xb, packed, scales, 1.0)) <= REL_TOL_TIGHT


@pytest.mark.parametrize("M", [17, 64, 65, 173, 257, 512])
@pytest.mark.parametrize("N,K", [(136, 64), (1288, 5120), (2048, 1984)])
def test_cluster_split_k(ops, M, N, K):
    """bf16 linear of 17 to 512 rows (K cut over a cluster where that pays), ragged rows, columns and K shares: plain with
    bias, GELU, and the same sum against float32.  REL_TOL_TIGHT: one bf16 rounding and the order of the float32 sum."""
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    x, w = (torch.randn(s, generator=gen, device="cuda").to(torch.bfloat16) for s in ((M, K), (N, K)))
    b = torch.randn(N, generator=gen, device="cuda").to(torch.bfloat16)
    want = x.double() @ w.double().T + b.double()
    got = ops.bf16_linear(x, w, b).double()
    assert float((got - want).norm() / want.norm()) <= REL_TOL_TIGHT
    want = torch.nn.functional.gelu(want, approximate="tanh")
    got = ops.bf16_linear_gelu(x, w, b).double()
    assert float((got - want).norm() / want.norm()) <= REL_TOL_TIGHT


def rand_fp4(ops, N, K, seed):
    """A weight of any size quickly: random codes, scales around one; with it its values in float64."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    packed = torch.randint(0, 256, (N, K // 2), generator=gen, dtype=torch.uint8, device="cuda")
    scales = torch.randint(48, 64, (N, K // 16), generator=gen, dtype=torch.uint8, device="cuda")
    lut = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, 0, -.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64, device="cuda")
    v = torch.stack([lut[(packed & 15).long()], lut[(packed >> 4).long()]], -1).view(N, K // 16, 16)
    return ops.Fp4Tensor(packed, scales, 0.25), (v * scales.view(torch.float8_e4m3fn).double()[..., None] * 0.25).view(N, K)


@pytest.mark.parametrize("N,K,rounds", [(4752, 8192, 3), (20000, 2048, 2), (16 * 1333, 3072, 4)])
@pytest.mark.parametrize("M", [1, 7, 9, 15])
def test_weights_read_in_rounds(ops, N, K, rounds, M):
    """Weights too tall for one round: slots refilled, barrier phases, row sums kept, a last CTA with fewer units.  The shapes
    that take the other route by their size (128 KB of rows and more) are held to the same bar."""
    w, dense = rand_fp4(ops, N, K, N + M)
    x = to_dev_bf16(o.seeded_activation(M, K, M))
    got = ops.fp4_linear(x, w.w_packed, w.w_scales, w.w_global_scale)
    route = ops.last_gemm_route()
    if M * K < 65536:
        assert route[0] == "few_rows" and route[1] >= rounds, route
    else:
        assert route[0] != "few_rows", route
    want = x.double() @ dense.T
    assert float((got.double() - want).norm() / want.norm()) <= REL_TOL_TIGHT
    gate = ops.fp4_linear_fused(ops.MODE_W4A16, x, [w, w], epilogue=ops.EPI_SILU_GATE)
    want = want.to(torch.bfloat16).double()
    want = want * torch.sigmoid(want) * want
    assert float((gate.double() - want).norm() / want.norm()) <= REL_TOL_VS_ORACLE


@pytest.mark.parametrize("M,N,K,few", [(8, 2048, 6144, True), (16, 12288, 2048, True), (16, 4096, 8192, True), (8, 59264, 2048, True),
                                       (16, 59264, 2048, False), (8, 16384, 8192, False), (12, 8192, 6144, False), (16, 16384, 1024, False),
                                       (8, 16384, 512, False), (16, 4096, 256, False), (17, 2048, 2048, False)])
def test_route_is_the_faster_one(ops, M, N, K, few):
    """Sizes on both sides of the rule, each measured (skinny_pays); the result is the same up to the sum's order either way."""
    w, dense = rand_fp4(ops, N, K, 5)
    x = to_dev_bf16(o.seeded_activation(M, K, M))
    got = ops.fp4_linear(x, w.w_packed, w.w_scales, w.w_global_scale)
    assert (ops.last_gemm_route()[0] == "few_rows") == few
    want = x.double() @ dense.T
    assert float((got.double() - want).norm() / want.norm()) <= REL_TOL_TIGHT


@pytest.mark.parametrize("M,N,K,cluster", [(17, 2048, 6144, True), (173, 1280, 1280, True), (512, 512, 2048, True), (173, 2048, 2048, True),
                                           (384, 2048, 2048, False), (320, 1280, 1280, False), (128, 3840, 1280, False), (200, 1280, 384, False),
                                           (300, 8192, 512, False), (513, 512, 2048, False)])
def test_cluster_route_is_the_faster_one(ops, M, N, K, cluster):
    """Sizes on both sides of the estimates, each measured (run_cluster); the result holds either way."""
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    x, w = (torch.randn(s, generator=gen, device="cuda").to(torch.bfloat16) for s in ((M, K), (N, K)))
    got = ops.bf16_linear(x, w).double()
    assert (ops.last_gemm_route()[0] == "cluster") == cluster
    want = x.double() @ w.double().T
    assert float((got - want).norm() / want.norm()) <= REL_TOL_TIGHT


@pytest.mark.parametrize("M", [17, 19, 33, 65, 173])
def test_cluster_epilogues_with_k_split(ops, M):
    """W4A16 on the cluster GEMM with K really cut (asserted): three ragged segments, gate|up whose gate sums stay in a CTA's own
    partial tile while its peers read that tile, and a residual added in place.  Each runs twice: the second call finds the bf16
    copies and fetches them ahead of its dependency wait."""
    def check_split():
        assert ops.last_gemm_route()[0] == "cluster" and ops.last_gemm_route()[1] > 1, ops.last_gemm_route()

    for K, ns in ((2048, (2048, 512, 136)), (6144, (264, 40, 512))):
        x = to_dev_bf16(o.seeded_activation(M, K, M))
        ws = [rand_fp4(ops, n, K, n + M) for n in ns]
        wants = [x.double() @ d.to(torch.bfloat16).double().T for _, d in ws]
        for _ in range(2):
            out = ops.fp4_linear_fused(ops.MODE_W4A16, x, [w for w, _ in ws]).double()
            check_split()
            c = 0
            for n, want in zip(ns, wants):
                assert float((out[:, c:c + n] - want).norm() / want.norm()) <= REL_TOL_TIGHT
                c += n
        (g, gd), (u, ud) = rand_fp4(ops, 520, K, 1), rand_fp4(ops, 520, K, 2)
        gw, uw = (0.01 * (x.double() @ d.to(torch.bfloat16).double().T) for d in (gd, ud))
        g.w_global_scale = u.w_global_scale = 0.0025                    # gates where SiLU bends; the copies round bf16(v) * 0.01 alike
        want = gw * torch.sigmoid(gw) * uw
        for _ in range(2):
            act = ops.fp4_linear_fused(ops.MODE_W4A16, x, [g, u], epilogue=ops.EPI_SILU_GATE).double()
            check_split()
            assert float((act - want).norm() / want.norm()) <= REL_TOL_VS_ORACLE
        (w, _), want = ws[0], wants[0]
        res = to_dev_bf16(o.seeded_activation(M, ns[0], 9))
        want = want.to(torch.bfloat16).double() + res.double()
        for _ in range(2):
            h = res.clone()
            ops.fp4_linear_fused(ops.MODE_W4A16, x, [w], epilogue=ops.EPI_RESIDUAL, residual=h, out=h)
            check_split()
            assert float((h.double() - want).norm() / want.norm()) <= REL_TOL_TIGHT


def test_cluster_share_counts(ops):
    """K blocks that do not divide by the CTAs that share them (3, 5, 6 and 7 among them, asserted): bf16 weights, bias, GELU."""
    shares = set()
    for K, N in ((448, 128), (704, 128), (1984, 640), (3008, 1280), (5120, 1280), (64, 256)):
        for M in (17, 40, 100):
            gen = torch.Generator(device="cuda").manual_seed(K + M)
            x, w = (torch.randn(s, generator=gen, device="cuda").to(torch.bfloat16) for s in ((M, K), (N, K)))
            b = torch.randn(N, generator=gen, device="cuda").to(torch.bfloat16)
            want = x.double() @ w.double().T + b.double()
            got = ops.bf16_linear(x, w, b).double()
            assert float((got - want).norm() / want.norm()) <= REL_TOL_TIGHT, (M, N, K)
            name, n = ops.last_gemm_route()
            shares.add(n if name == "cluster" else 0)
            got = ops.bf16_linear_gelu(x, w, b).double()
            want = torch.nn.functional.gelu(want, approximate="tanh")
            assert float((got - want).norm() / want.norm()) <= REL_TOL_TIGHT, (M, N, K)
    assert {3, 5, 6, 7, 8} <= shares, shares
