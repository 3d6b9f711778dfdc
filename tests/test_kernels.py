"""Each CUDA kernel alone against a plain float64 torch reference, at sizes other than the engine's."""
import math

import pytest
import torch

from plain_minicpm import plain_attention, plain_rmsnorm, plain_rope, plain_sample

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
DTYPES = [torch.float32, torch.bfloat16]


def _tol(dtype):
    # float32: summation order only.  bfloat16: one rounding of the stored result (2^-9 relative).
    return dict(rtol=2e-5, atol=2e-6) if dtype == torch.float32 else dict(rtol=4e-3, atol=4e-3)


def _close(got, want, dtype, scale=1.0):
    t = _tol(dtype)
    torch.testing.assert_close(got.double().cpu(), want.double().cpu(), rtol=t["rtol"], atol=t["atol"] * scale)


@pytest.fixture(scope="module")
def K():
    from infinicore_infer_b200 import kernels
    return kernels


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("V,d,T", [(301, 80, 7), (1000, 2304, 3), (17, 6, 1)])
def test_embed(K, dtype, V, d, T):
    g = torch.Generator().manual_seed(V)
    table = torch.randn(V, d, generator=g).to(dtype)
    tok = torch.randint(0, V, (T,), generator=g, dtype=torch.int32)
    tok[0] = V - 1
    out = torch.empty(T, d, device=DEV)
    K.embed(tok.to(DEV), table.to(DEV), 2.5, out)
    assert torch.equal(out.cpu(), table.float()[tok.long()] * 2.5)


@pytest.mark.parametrize("out_dtype", DTYPES)
@pytest.mark.parametrize("delta_dtype", [None, torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,d,eps", [(5, 80, 1e-5), (3, 2304, 1e-6), (2, 5000, 3e-6), (1, 14336, 1e-5),
                                     (300, 2304, 1e-6), (261, 1000, 1e-5), (257, 3072, 1e-5), (256, 132, 1e-5), (400, 3076, 1e-5)])
def test_add_rmsnorm(K, out_dtype, delta_dtype, T, d, eps):
    g = torch.Generator().manual_seed(d)
    x = torch.randn(T, d, generator=g) * 3
    w = 1 + 0.1 * torch.randn(d, generator=g)
    delta = None if delta_dtype is None else torch.randn(T, d, generator=g).to(delta_dtype)
    xd = x.to(DEV).clone()
    out = torch.empty(T, d, dtype=out_dtype, device=DEV)
    K.add_rmsnorm(xd, None if delta is None else delta.to(DEV), 0.7, w.to(DEV), eps, out, out_scale=4.0)
    v = x.double() + (0 if delta is None else 0.7 * delta.double())
    _close(xd, v, torch.float32)                       # the sum is written back in float32
    _close(out, 4.0 * plain_rmsnorm(v, w.double(), eps), out_dtype, scale=4.0)


def test_add_rmsnorm_gathers_rows_without_touching_the_stream(K):
    g = torch.Generator().manual_seed(0)
    x = torch.randn(9, 96, generator=g)
    delta = torch.randn(9, 96, generator=g)
    w = torch.ones(96)
    rows = torch.tensor([8, 0, 3, 3], dtype=torch.int32)
    xd = x.to(DEV).clone()
    out = torch.empty(4, 96, device=DEV)
    K.add_rmsnorm(xd, delta.to(DEV), 2.0, w.to(DEV), 1e-6, out, rows=rows.to(DEV))
    assert torch.equal(xd.cpu(), x)
    _close(out, plain_rmsnorm((x + 2 * delta).double()[rows.long()], w.double(), 1e-6), torch.float32)
    # many gathered rows (a warp a row)
    x = torch.randn(400, 264, generator=g)
    delta = torch.randn(400, 264, generator=g)
    w = 1 + 0.1 * torch.randn(264, generator=g)
    rows = torch.randint(0, 400, (300,), generator=g).to(torch.int32)
    xd = x.to(DEV).clone()
    out = torch.empty(300, 264, device=DEV)
    K.add_rmsnorm(xd, delta.to(DEV), 2.0, w.to(DEV), 1e-6, out, rows=rows.to(DEV))
    assert torch.equal(xd.cpu(), x)
    _close(out, plain_rmsnorm((x + 2 * delta).double()[rows.long()], w.double(), 1e-6), torch.float32)


@pytest.mark.parametrize("in_dtype,out_dtype", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16),
                                                 (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("T,di", [(3, 136), (1, 5760), (17, 33)])
def test_swiglu(K, in_dtype, out_dtype, T, di):
    g = torch.Generator().manual_seed(di)
    gu = (torch.randn(T, 2 * di, generator=g) * 3).to(in_dtype)
    out = torch.empty(T, di, dtype=out_dtype, device=DEV)
    K.swiglu(gu.to(DEV), out)
    a, b = gu.double()[:, :di], gu.double()[:, di:]
    _close(out, a * torch.sigmoid(a) * b, out_dtype, scale=3.0)


@pytest.mark.parametrize("T,d", [(256, 1024), (257, 1028), (300, 2052), (2400, 3072)])
@pytest.mark.parametrize("delta", [False, True])
@pytest.mark.parametrize("wanted", [False, True])
def test_add_rmsnorm_of_many_rows(K, T, d, delta, wanted):
    """Widths at the edges of the kernel that walks over rows, one and several rows a block, all rows and picked ones."""
    g = torch.Generator().manual_seed(T + d)
    x, p, w = torch.randn(T, d, generator=g), torch.randn(T, d, generator=g), torch.randn(d, generator=g)
    rows = torch.randint(0, T, (T,), generator=g, dtype=torch.int32) if wanted else None
    xd, out = x.to(DEV), torch.full((T, d), 7.0, device=DEV)
    K.add_rmsnorm(xd, p.to(DEV) if delta else None, 0.25, w.to(DEV), 1e-5, out, 2.0, rows.to(DEV) if wanted else None)
    v = x.double() + (0.25 * p.double() if delta else 0.0)
    pick = v[rows.long()] if wanted else v
    want = pick * torch.rsqrt(pick.square().mean(-1, keepdim=True) + 1e-5) * w.double() * 2.0
    assert (out.cpu().double() - want).abs().max() <= 2e-6 * want.abs().max()
    assert torch.equal(xd.cpu(), x + 0.25 * p if delta and not wanted else x) or (delta and not wanted and (xd.cpu().double() - v).abs().max() <= 2e-7 * v.abs().max())


@pytest.mark.parametrize("in_dtype,out_dtype", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("T,di", [(96, 512), (13, 4100), (12, 4096)])
def test_swiglu_four_units_a_thread_in_the_types_of_the_models(K, in_dtype, out_dtype, T, di):
    """Sums in float32 or operands in bfloat16, rounded once: the bits of the form that rows off 16 bytes take, and 64 bits."""
    g = torch.Generator().manual_seed(di + T)
    gu = (torch.randn(T, 2 * di, generator=g) * 3).to(in_dtype)
    out, slow = torch.empty(T, di, dtype=out_dtype, device=DEV), torch.empty(T * di + 1, dtype=out_dtype, device=DEV)[1:].view(T, di)
    K.swiglu(gu.to(DEV), out)
    K.swiglu(gu.to(DEV), slow)
    a, b = gu.double().split(di, 1)
    _close(out, a * torch.sigmoid(a) * b, out_dtype, scale=3.0)
    assert torch.equal(out, slow)


@pytest.mark.parametrize("out_dtype", DTYPES)
@pytest.mark.parametrize("delta_dtype", [None, torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,d", [(1, 1536), (64, 2048), (255, 4096), (7, 1028), (200, 2052), (3, 132), (2, 6144)])
def test_add_rmsnorm_of_few_rows_in_registers(K, out_dtype, delta_dtype, T, d):
    """One, two and three vectors a thread, whole and in part, all rows and picked ones."""
    g = torch.Generator().manual_seed(T + d)
    x, w = torch.randn(T, d, generator=g) * 3, 1 + 0.1 * torch.randn(d, generator=g)
    delta = None if delta_dtype is None else torch.randn(T, d, generator=g).to(delta_dtype)
    v = x.double() + (0 if delta is None else 0.7 * delta.double())
    rows = torch.randint(0, T, (T,), generator=g, dtype=torch.int32)
    for pick in (None, rows):
        xd, out = x.to(DEV), torch.empty(T, d, dtype=out_dtype, device=DEV)
        K.add_rmsnorm(xd, None if delta is None else delta.to(DEV), 0.7, w.to(DEV), 1e-5, out, 4.0, None if pick is None else pick.to(DEV))
        _close(xd, x.double() if pick is not None else v, torch.float32)
        _close(out, 4.0 * plain_rmsnorm(v if pick is None else v[pick.long()], w.double(), 1e-5), out_dtype, scale=4.0)


def _norm_in_order(v, w, eps, threads):
    """The norm of float32 rows as a block of ``threads`` adds: four squares, a thread's vectors, a warp's tree, the warps' tree."""
    T, d = v.shape
    n = -(-d // (4 * threads))
    q = torch.zeros(T, n * threads * 4, dtype=torch.float64, device=DEV)
    q[:, :d] = v
    q, once, lanes = q.view(T, n, threads, 4), lambda x: x.float().double(), torch.arange(32, device=DEV)
    four = once(q[..., 3] ** 2 + once(q[..., 2] ** 2 + once(q[..., 0] ** 2 + once(q[..., 1] ** 2))))      # 64 bits hold a square, so each step rounds once
    total = torch.zeros(T, threads, device=DEV)
    for j in range(n):
        total = total + four[:, j].float()
    total = total.view(T, -1, 32)
    for o in (16, 8, 4, 2, 1):
        total = total + total[..., lanes ^ o]
    total = torch.nn.functional.pad(total[..., 0], (0, 32 - threads // 32))
    for o in (16, 8, 4, 2, 1):
        total = total + total[:, lanes ^ o]
    return v * torch.rsqrt(total[:, :1] / d + eps) * w


@pytest.mark.parametrize("T", [12, 300])
@pytest.mark.parametrize("delta_dtype", [None, torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d,threads", [(512, 128), (1024, 256), (4096, 512)])
def test_add_rmsnorm_adds_in_the_order_of_its_block(K, T, delta_dtype, d, threads):
    """One and two vectors a thread, in registers (few rows) and through shared memory: the same bits, which do not depend on how it was compiled.
    (Widths whose reciprocal is exact; many rows of up to 3,072 columns add a warp a row.)"""
    if T >= 256 and d <= 3072:
        pytest.skip("a warp a row")
    g = torch.Generator().manual_seed(T + d)
    x, w = torch.randn(T, d, generator=g).to(DEV), torch.randn(d, generator=g).to(DEV)
    delta = None if delta_dtype is None else torch.randn(T, d, generator=g).to(DEV).to(delta_dtype)
    v = x if delta is None else x + 0.5 * delta.float()         # a half is exact: one rounding, as in the kernel
    out = torch.empty(T, d, device=DEV)
    K.add_rmsnorm(x.clone(), delta, 0.5, w, 1e-5, out)
    assert torch.equal(out, _norm_in_order(v, w, 1e-5, threads))


@pytest.mark.parametrize("out_dtype", DTYPES)
@pytest.mark.parametrize("T,d", [(256, 1024), (257, 1028), (532, 1536), (512, 2304), (2400, 2052), (1300, 3072)])
@pytest.mark.parametrize("wanted", [False, True])
def test_add_rmsnorm_of_many_rows_adds_in_one_order(K, out_dtype, T, d, wanted):
    """The kernel that walks over rows with something to add, against the warp a row that takes the finished sum: the same bits."""
    g = torch.Generator().manual_seed(T + d)
    x, p, w = torch.randn(T, d, generator=g), torch.randn(T, d, generator=g), torch.randn(d, generator=g).to(DEV)
    rows = torch.randint(0, T, (T,), generator=g, dtype=torch.int32).to(DEV) if wanted else None
    added = (x + 0.25 * p).to(DEV)           # a quarter is exact: one rounding, as in the kernel
    out, want = (torch.full((T, d), 7.0, dtype=out_dtype, device=DEV) for _ in range(2))
    K.add_rmsnorm(x.to(DEV), p.to(DEV), 0.25, w, 1e-5, out, 2.0, rows)
    K.add_rmsnorm(added, None, 1.0, w, 1e-5, want, 2.0, rows)
    assert torch.equal(out, want)


@pytest.mark.parametrize("T,d", [(1, 4), (7, 1024), (7, 1540), (65, 4096), (64, 4100), (512, 4096), (513, 2052), (600, 1500), (600, 4096)])
def test_norm_add_with_the_row_in_registers(K, T, d):
    """Widths of one and two vectors a thread and a part of one, and the sizes next to them; one norm behind it, two, none."""
    g = torch.Generator().manual_seed(T + d)
    p, x = torch.randn(T, d, generator=g), torch.randn(T, d, generator=g)
    w, w1, w2 = (1 + 0.1 * torch.randn(d, generator=g) for _ in range(3))
    v = x.double() + plain_rmsnorm(p.double(), w.double(), 1e-5)
    for outs in range(3):
        got, h, h2 = x.to(DEV), torch.empty(T, d, device=DEV), torch.empty(T, d, device=DEV)
        more = dict(next_weight=w1.to(DEV), next_eps=1e-4, out=h) if outs else {}
        if outs == 2:
            K.norm_add(p.to(DEV), got, w.to(DEV), 1e-5, w1.to(DEV), 1e-4, h, w2.to(DEV), h2)
        else:
            K.norm_add(p.to(DEV), got, w.to(DEV), 1e-5, **more)
        # sums of d squares in a tree: a few roundings of 2^-24 each
        for have, want in ((got, v), (h, plain_rmsnorm(v, w1.double(), 1e-4)), (h2, plain_rmsnorm(v, w2.double(), 1e-4)))[: 1 + outs]:
            assert (have.cpu().double() - want).abs().max() <= 2e-6 * want.abs().max()


@pytest.mark.parametrize("T,di", [(96, 512), (100, 516), (13, 4100)])
def test_swiglu_four_units_a_thread_has_the_same_bits(K, T, di):
    """The vector form against the form that rows off 16 bytes take."""
    g = torch.Generator().manual_seed(di)
    gu = (torch.randn(T, 2 * di, generator=g) * 30).to(DEV)
    fast, slow = torch.empty(T, di, device=DEV), torch.empty(T * di + 1, device=DEV)[1:].view(T, di)
    K.swiglu(gu, fast)
    K.swiglu(gu, slow)
    assert torch.equal(fast, slow) and torch.isfinite(fast).all()


@pytest.mark.parametrize("M,N,K_", [(1, 1, 1), (7, 301, 80), (65, 129, 33), (130, 64, 2304), (3, 1000, 17)])
def test_gemm_f32_is_a_true_float32_product(K, M, N, K_):
    g = torch.Generator().manual_seed(M * N)
    a = torch.randn(M, K_, generator=g)
    w = torch.randn(N, K_, generator=g)
    bias = torch.randn(N, generator=g)
    out = torch.empty(M, N, device=DEV)
    K.gemm_f32(a.to(DEV), w.to(DEV), out, bias.to(DEV))
    want = a.double() @ w.double().T + bias.double()
    # TF32 would be wrong by 2^-11 of |a||w| ~ 5e-4 * sqrt(K); float32 stays below 1e-6 * sqrt(K)
    assert (out.cpu().double() - want).abs().max() <= 2e-6 * math.sqrt(K_) * 4
    # a row's result does not depend on the batch it is in
    if M > 1:
        one = torch.empty(1, N, device=DEV)
        K.gemm_f32(a[M - 1:].contiguous().to(DEV), w.to(DEV), one, bias.to(DEV))
        assert torch.equal(one[0], out[M - 1])


@pytest.mark.parametrize("M,N,K_", [(1, 1, 1), (8, 64, 16), (9, 65, 17), (16, 33, 63), (33, 2049, 64), (65, 130, 66), (301, 1536, 132), (129, 9601, 20)])
def test_gemm_f32_tiles_agree_bit_for_bit(K, M, N, K_):
    """Every tile size at its edges and with rows that do not start on 16 bytes: the sums' order depends on K alone."""
    g = torch.Generator().manual_seed(M + N + K_)
    a, w = torch.randn(M, K_, generator=g).to(DEV), torch.randn(N, K_, generator=g).to(DEV)
    out = torch.full((M, N), 7.0, device=DEV)
    K.gemm_f32(a, w, out)
    want = a.double() @ w.double().T
    # a product's rounding is below 2^-24 of |a||w| < 25 here, and K of them add up
    assert (out.double() - want).abs().max() <= 2.0 ** -24 * 25 * max(4, K_)
    for rows, cols in ((slice(0, 1), slice(None)), (slice(M // 2, None), slice(0, (N + 1) // 2))):
        part_a, part_w = a[rows].contiguous(), w[cols].contiguous()
        part = torch.full((part_a.shape[0], part_w.shape[0]), 7.0, device=DEV)
        K.gemm_f32(part_a, part_w, part)
        assert torch.equal(part, out[rows, cols])


@pytest.mark.parametrize("M,N,K_", [(1, 1, 4), (33, 130, 68), (97, 127, 1024), (161, 257, 640), (301, 129, 3840)])
@pytest.mark.parametrize("tile,cuts", [(32, 1), (32, 8), (64, 4), (96, 2), (128, 1), (160, 1), (160, 4)])
def test_gemm_f32_tcgen05_keeps_float32(K, M, N, K_, tile, cuts):
    """Tokens, features and K at the edges of their tiles, cuts of K with and without chunks of their own."""
    g = torch.Generator().manual_seed(M + N + K_)
    a, w, bias = torch.randn(M, K_, generator=g).to(DEV), torch.randn(N, K_, generator=g).to(DEV), torch.randn(N, generator=g).to(DEV)
    out, plain = torch.full((M, N), 7.0, device=DEV), torch.empty(M, N, device=DEV)
    K.gemm_f32_tcgen05(a, w, out, bias, tile=tile, cuts=cuts)
    K.check_gemm_status(DEV)
    want = a.double() @ w.double().T + bias.double()
    # a chunk's sum is cut off at most 24 times (a unit in the last place, 2^-23 of what is summed: below 25 x 64), then ceil(K / 64) sums round
    size = (a.double().abs() @ w.double().abs().T + bias.double().abs()).max().item()
    assert (out.double() - want).abs().max().item() <= 2.0 ** -23 * size
    K.gemm_f32(a, w, plain, bias)
    # no further off than the multiply-adds in float32, but for what three units in the last place of the few outputs' sizes make
    assert (out.double() - want).norm() <= (plain.double() - want).norm() + 3 * 2.0 ** -24 * want.norm()


@pytest.mark.parametrize("cuts", [1, 4])
def test_gemm_f32_tcgen05_what_the_split_does_not_carry(K, cuts):
    """Infinities, NaN and magnitudes that bfloat16 rounds to infinity: what float32 multiply-adds give."""
    g = torch.Generator().manual_seed(5)
    a, w = torch.randn(40, 512, generator=g), torch.randn(200, 512, generator=g)
    a[3, 5], a[7, 9], a[9, 1], w[11, 0], w[12, 4] = math.inf, math.nan, -math.inf, 3.4e38, 1e-42
    a, w = a.to(DEV), w.to(DEV)
    out, plain = torch.empty(40, 200, device=DEV), torch.empty(40, 200, device=DEV)
    K.gemm_f32_tcgen05(a, w, out, tile=32, cuts=cuts)
    K.gemm_f32(a, w, plain)
    assert torch.equal(out.isnan(), plain.isnan()) and torch.equal(out.isinf(), plain.isinf())
    assert torch.equal(out[out.isinf()], plain[plain.isinf()])
    ok = plain.isfinite()
    assert ((out - plain).abs()[ok] <= 1e-6 * plain.abs()[ok] + 2e-4).all()


@pytest.mark.parametrize("what", ["tiny and large", "below the normal numbers", "results below the normal numbers", "large", "one sign", "columns of uneven size", "rows of uneven size"])
@pytest.mark.parametrize("cuts", [1, 4])
def test_gemm_f32_tcgen05_of_operands_that_are_not_of_size_one(K, what, cuts):
    """Operands whose last bits lie below bfloat16's smallest number, large ones, sums that grow, terms of very unlike sizes: no further off than float32."""
    g = torch.Generator().manual_seed(8)
    M, N, K_ = 40, 136, 1536
    a, w = torch.randn(M, K_, generator=g), torch.randn(N, K_, generator=g)
    if what == "tiny and large": a, w = a * 1e-37, w * 1e30
    elif what == "below the normal numbers": a, w = a * 1e30, w * 1e-41
    elif what == "results below the normal numbers": a, w = a * 1e-20, w * 1e-20
    elif what == "large": a, w = a * 1e32, w * 1e-8
    elif what == "one sign": a, w = a.abs(), w.abs()
    elif what == "columns of uneven size": a, w = a * 2.0 ** torch.randint(-40, 40, (K_,), generator=g), w * 2.0 ** torch.randint(-8, 8, (K_,), generator=g)
    else: a, w = a * 2.0 ** torch.randint(-90, 60, (M, 1), generator=g), w * 2.0 ** torch.randint(-40, 20, (N, 1), generator=g)
    a, w = a.to(DEV), w.to(DEV)
    out, plain = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    K.gemm_f32_tcgen05(a, w, out, tile=64, cuts=cuts)
    K.gemm_f32(a, w, plain)
    want = a.double() @ w.double().T
    # each output by the sizes of its two operands, so that all of them count alike
    unit = a.double().norm(dim=1)[:, None] * w.double().norm(dim=1)[None] * K_ ** -0.5
    off = lambda x: ((x.double() - want) / unit).norm()
    # three units in the last place of the outputs' sizes beside what the multiply-adds are off by, and the spacing of the smallest numbers
    assert off(out) <= off(plain) + 3 * 2.0 ** -24 * (want / unit).norm() + (2.0 ** -149 / unit).norm()


@pytest.mark.parametrize("tile,cuts", [(32, 1), (32, 4), (160, 1)])
def test_gemm_f32_tcgen05_makes_what_is_not_finite_with_the_multiply_adds_bits(K, tile, cuts):
    """Rows with an infinity or a NaN, weights beyond what the split holds: what the product on the CUDA cores gives, and nothing else is touched."""
    g = torch.Generator().manual_seed(6)
    a, w, bias = torch.randn(70, 580, generator=g), torch.randn(200, 580, generator=g), torch.randn(200, generator=g)
    clean = torch.empty(70, 200, device=DEV)
    K.gemm_f32_tcgen05(a.to(DEV), w.to(DEV), clean, bias.to(DEV), tile=tile, cuts=cuts)
    a[3, 5], a[33, 579], a[34, 64], w[11, 7], w[130, 0] = math.inf, math.nan, -3e36, 2e37, -math.inf
    a, w, bias = a.to(DEV), w.to(DEV), bias.to(DEV)
    out, plain = torch.empty(70, 200, device=DEV), torch.empty(70, 200, device=DEV)
    K.gemm_f32_tcgen05(a, w, out, bias, tile=tile, cuts=cuts)
    K.gemm_f32(a, w, plain, bias)
    rows, cols = torch.ones(70, dtype=torch.bool, device=DEV), torch.ones(200, dtype=torch.bool, device=DEV)
    rows[[3, 33, 34]] = cols[[11, 130]] = False
    again = ~(rows[:, None] & cols[None])
    assert torch.equal(out[again].nan_to_num(7.0), plain[again].nan_to_num(7.0)) and torch.equal(out[again].isnan(), plain[again].isnan())
    assert torch.equal(out[~again], clean[~again])


@pytest.mark.parametrize("heads,n,k", [(3, 33, 16), (2, 100, 48), (5, 8, 512), (2, 32, 144)])
@pytest.mark.parametrize("gated", [False, True])
def test_head_linear_of_few_rows_has_the_tiles_bits(K, heads, n, k, gated):
    """Rows, features and K at the edges of the few-row kernel's blocks, against 64 bits and against the tiles that many rows take."""
    g = torch.Generator().manual_seed(n + k)
    x, w = torch.randn(70, heads * k, generator=g).bfloat16().to(DEV), (torch.randn(heads, n, k, generator=g) * k ** -0.5).bfloat16().to(DEV)
    gate = torch.randn(70, heads * n, generator=g).to(DEV) if gated else None
    many = torch.empty(70, heads * n, dtype=torch.bfloat16, device=DEV)
    K.head_linear(x, w, many, n, gate, heads * n)
    want = torch.einsum("thk,hnk->thn", x.view(70, heads, k).double(), w.double()).reshape(70, -1) * (torch.sigmoid(gate.double()) if gated else 1.0)
    assert ((many.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()
    for rows in (1, 15, 16, 17, 64):
        few = torch.full((rows, heads * n), 7.0, dtype=torch.bfloat16, device=DEV)
        K.head_linear(x[:rows], w, few, n, None if gate is None else gate[:rows], heads * n)
        assert torch.equal(few, many[:rows])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,d,ff,experts,top", [(1, 8, 8, 5, 1), (3, 2056, 40, 9, 2), (9, 72, 2064, 2, 1), (21, 64, 24, 3, 3), (2, 64, 16, 300, 8),
                                                  (32, 3000, 24, 100, 2), (32, 72, 1000, 100, 2)])
def test_routed_experts_of_few_rows(K, dtype, rows, d, ff, experts, top):
    """Rows of a matrix in one piece and in two, features at the edges of the blocks, more entries than run at a time, more experts than entries,
    several groups of short rows a block in either product."""
    g = torch.Generator().manual_seed(rows + d)
    h, router = torch.randn(rows, d, generator=g).to(dtype).to(DEV), (torch.randn(experts, d, generator=g) * 2 * d ** -0.5).to(DEV)
    up = (torch.randn(experts * 2 * ff, d, generator=g) * d ** -0.5).to(dtype).to(DEV)
    down = (torch.randn(experts * d, ff, generator=g) * ff ** -0.5).to(dtype).to(DEV)
    out = torch.full((rows, d), 7.0, device=DEV)
    K.routed_experts(h, router, up, down, out, False, experts, top, 1)
    K.check_gemm_status(DEV)
    score, chosen = torch.sigmoid(h.double() @ router.double().T).topk(top, -1)
    want = torch.zeros(rows, d, dtype=torch.float64, device=DEV)
    for t in range(rows):
        for s, e in zip(score[t], chosen[t].tolist()):
            gate, rest = (up[e * 2 * ff + i * ff: e * 2 * ff + (i + 1) * ff].double() @ (s * h[t].double()) for i in range(2))
            inner = (torch.nn.functional.silu(gate) * rest).to(dtype).double()      # rounded to the activation type, as it is stored
            want[t] += down[e * d: (e + 1) * d].double() @ inner
    # sums of ff terms below 1 in float32; in bfloat16 an inner activation may round the other way (2^-9 of it)
    assert (out.double() - want).abs().max() <= (2e-5 if dtype == torch.float32 else 2.0 ** -8 * want.abs().max().item())


@pytest.mark.parametrize("nh,nkvh,dh,page", [(6, 2, 64, 16), (3, 1, 128, 8), (400, 400, 64, 16), (40, 8, 128, 64)])
@pytest.mark.parametrize("reqs", [[(9, 0), (64, 3)], [(129, 60)], [(31, 200), (40, 0), (150, 129)]])
def test_attention_f32_in_tiles_of_rows(K, nh, nkvh, dh, page, reqs):
    """Both sizes of tiles (many heads take the large ones), rows and keys at their edges, histories, a value that is not finite behind some rows."""
    g = torch.Generator().manual_seed(nh + dh)
    T, blocks = sum(n for n, _ in reqs), max(-(-(n + h) // page) for n, h in reqs)
    q = torch.randn(T, nh, dh, generator=g).to(DEV)
    kp, vp = (torch.randn(blocks * len(reqs) + 1, nkvh, page, dh, generator=g).to(DEV) for _ in range(2))
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    table = ints([[1 + i * blocks + b for b in range(blocks)] for i in range(len(reqs))])
    start = [0]
    for n, _ in reqs:
        start.append(start[-1] + n)
    tiles = [[b, start[b] + t] for b, (n, _) in enumerate(reqs) for t in range(0, n, 128)]
    n, h = reqs[-1]
    last = (n + h - 1) // page
    vp[table[-1, last], :, (n + h - 1) % page] = math.nan          # the last position's value: its own row's result alone
    out = torch.full_like(q, 7.0)
    K.attention_f32(q, kp, vp, out, ints(tiles), len(tiles), ints(start), ints([h for _, h in reqs]), table, nh, dh ** -0.5)
    assert torch.isnan(out[-1]).all() and torch.isfinite(out[:-1]).all()
    for b, (n, h) in enumerate(reqs):
        flat = lambda p: p[table[b].long()].transpose(1, 2).reshape(-1, nkvh, dh)[: n + h].double().repeat_interleave(nh // nkvh, 1)
        v = flat(vp).nan_to_num(0.0)
        s = torch.einsum("thd,jhd->htj", q[start[b]: start[b + 1]].double(), flat(kp)) * dh ** -0.5
        s = s.masked_fill(torch.arange(n + h, device=DEV)[None] > torch.arange(h, n + h, device=DEV)[:, None], -math.inf)
        want = torch.einsum("htj,jhd->thd", s.softmax(-1), v)
        rows = slice(start[b], start[b + 1] - (1 if b == len(reqs) - 1 else 0))
        # scores of size 1 rounded 128 times, weights that sum to 1, values below 6
        assert (out[rows].double() - want[: rows.stop - rows.start]).abs().max() <= 1e-5


@pytest.mark.parametrize("nh,nkvh,dh,page", [(6, 2, 64, 16), (3, 1, 128, 8), (200, 200, 64, 16), (40, 8, 128, 64)])
@pytest.mark.parametrize("reqs", [[(9, 0), (64, 3)], [(129, 60)], [(31, 200), (40, 0), (150, 129)], [(63, 1), (1, 95)]])
def test_attention_f32_in_tiles_has_the_row_kernel_s_bits(K, nh, nkvh, dh, page, reqs):
    """Rows and chunks of 32 keys at the edges of the tiles, both tile sizes, a value that is not finite among the keys of some rows."""
    g = torch.Generator().manual_seed(nh + dh + len(reqs))
    T, blocks = sum(n for n, _ in reqs), max(-(-(n + h) // page) for n, h in reqs)
    q = (torch.randn(T, nh, dh, generator=g) * 2).to(DEV)
    kp, vp = (torch.randn(blocks * len(reqs) + 1, nkvh, page, dh, generator=g).to(DEV) for _ in range(2))
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    table = ints([[1 + i * blocks + b for b in range(blocks)] for i in range(len(reqs))])
    start = [0]
    for n, _ in reqs:
        start.append(start[-1] + n)
    tiles = [[b, start[b] + t] for b, (n, _) in enumerate(reqs) for t in range(0, n, 128)]
    n, h = reqs[0]
    vp[table[0, (n + h - 1) // page], :, (n + h - 1) % page] = math.inf
    out, rows = torch.full_like(q, 7.0), torch.full_like(q, 7.0)
    K.attention_f32(q, kp, vp, out, ints(tiles), len(tiles), ints(start), ints([h for _, h in reqs]), table, nh, dh ** -0.5)
    K.attention_rows(q, kp, vp, rows, ints([h + i for n, h in reqs for i in range(n)]), ints([r for r, (n, _) in enumerate(reqs) for _ in range(n)]), table, T, nh, dh ** -0.5)
    assert torch.equal(out.nan_to_num(5.0, 6.0, -6.0), rows.nan_to_num(5.0, 6.0, -6.0)) and torch.isfinite(out[start[1]:]).all()


@pytest.mark.parametrize("T,heads,dv", [(256, 64, 128), (1100, 32, 64), (2100, 16, 64)])
@pytest.mark.parametrize("per_head", [0, 1, 2])
def test_norm_gate_of_many_rows(K, T, heads, dv, per_head):
    g = torch.Generator().manual_seed(T)
    n = heads * dv
    o, u, w = (torch.randn(*s, generator=g).to(DEV) for s in ((T, n), (T, n + 8), (dv if per_head == 1 else n,)))
    out = torch.empty(T, n, device=DEV)
    K.norm_gate(o, u, 4, w, 1e-5, heads, dv, per_head, 1, out)
    x = o.double().view(T, heads, dv) if per_head else o.double()
    want = (x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5)).reshape(T, n) * (w.double().repeat(heads) if per_head == 1 else w.double())
    want = want * torch.nn.functional.silu(u[:, 4: 4 + n].double())
    assert ((out.double() - want).abs() <= 4e-6 * want.abs() + 1e-6).all()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,heads,dv", [(256, 64, 128), (300, 63, 128), (1100, 33, 64), (2100, 16, 64), (1100, 16, 128), (1400, 25, 64)])
@pytest.mark.parametrize("per_head,act", [(0, 1), (1, 0), (2, 1)])
def test_norm_gate_of_many_rows_has_the_bits_of_few(K, dtype, T, heads, dv, per_head, act):
    """Rows in registers against the form that steps of fewer than 256 rows take: heads in pairs and one over, one mean or many."""
    g = torch.Generator().manual_seed(T + heads)
    n = heads * dv
    o, u, w = (torch.randn(*s, generator=g).to(DEV) for s in ((T, n), (T, n + 8), (dv if per_head == 1 else n,)))
    out, want = (torch.full((T, n), 7.0, dtype=dtype, device=DEV) for _ in range(2))
    K.norm_gate(o, u, 4, w, 1e-5, heads, dv, per_head, act, out)
    for at in range(0, T, 200):
        rows = slice(at, min(T, at + 200))
        K.norm_gate(o[rows], u[rows], 4, w, 1e-5, heads, dv, per_head, act, want[rows])
    assert torch.equal(out, want)


def _off(t):
    """The same numbers four bytes off a 16-byte boundary: the element-by-element forms."""
    moved = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
    return moved.copy_(t)


@pytest.mark.parametrize("has_kv", [False, True])
def test_conv_qkv_four_channels_a_thread(K, has_kv):
    """Three requests of several hundred rows: rows that look into the tail, and rows that do not, against the form an element at a time."""
    g = torch.Generator().manual_seed(7)
    H, G, dk, page, lens = 4, 2, 64, 16, [1, 200, 130]
    T, nq, nk = sum(lens), H * dk, G * dk
    C = nq + (2 * nk if has_kv else 0)
    u, conv = torch.randn(T, nq + 2 * nk, generator=g).to(DEV), [torch.randn(c, 4, generator=g).to(DEV) for c in (nq, nk, nk)]
    norm, freq, tail = [torch.randn(c, generator=g).to(DEV) for c in (nq, nk)], torch.rand(16, generator=g).to(DEV), torch.randn(3, 3, C, generator=g).to(DEV)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pos, req, start = ints([i for n in lens for i in range(n)]), ints([r for r, n in enumerate(lens) for _ in range(n)]), ints([0, 1, 201, 331])
    table = ints([[1 + 13 * r + b for b in range(13)] for r in range(3)])
    got = []
    for move in (lambda t: t, _off):
        q, kp, vp, t = torch.zeros(T, nq, device=DEV), *(torch.zeros(40, G, page, dk, device=DEV) for _ in range(2)), tail.clone()
        K.conv_qkv(move(u), (0, nq, nq + nk), H, G, dk, dk, has_kv, conv, 4, norm, 1e-5, freq, 32, t, pos, req, start, ints([0, 1, 2]), table, page, q, kp, vp)
        got.append((q, kp, vp, t))
    for a, b in zip(*got):          # only the squares' sums may differ, by their order
        assert (a - b).abs().max() <= 2e-6 * b.abs().max()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,G,rot,half,temp,head_norm", [(4, 2, 32, False, False, 0), (16, 4, 64, True, True, 0), (5, 1, 16, True, False, 0), (16, 4, 32, False, True, 1),
                                                        (12, 12, 64, True, True, 2), (3, 1, 0, False, True, 0)])
def test_conv_qkv_four_channels_a_thread_has_the_same_bits(K, dtype, H, G, rot, half, temp, head_norm):
    """Each way of norm and rotation with and without what the heads are scaled by, in both types, against the form an element at a time."""
    g = torch.Generator().manual_seed(H + rot)
    dk, page, lens = 64, 16, [1, 200, 130]
    T, nq, nk = sum(lens), H * dk, G * dk
    C = nq + 2 * nk
    u, conv = torch.randn(T, C, generator=g).to(DEV), [torch.randn(c, 4, generator=g).to(DEV) for c in (nq, nk, nk)]
    norm, freq, tail = [torch.randn(dk if head_norm == 2 else c, generator=g).to(DEV) for c in (nq, nk)], torch.rand(32, generator=g).to(DEV), torch.randn(3, 3, C, generator=g).to(DEV)
    scale = torch.rand(H, generator=g).to(DEV) if temp else None
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pos, req, start = ints([i for n in lens for i in range(n)]), ints([r for r, n in enumerate(lens) for _ in range(n)]), ints([0, 1, 201, 331])
    table = ints([[1 + 13 * r + b for b in range(13)] for r in range(3)])
    got = []
    for move in (lambda t: t, _off):
        q, kp, vp, t = torch.zeros(T, nq, device=DEV).to(dtype), *(torch.zeros(40, G, page, dk, device=DEV).to(dtype) for _ in range(2)), tail.clone()
        K.conv_qkv(move(u), (0, nq, nq + nk), H, G, dk, dk, True, conv, 4, norm, 1e-5, freq if rot else None, rot, t, pos, req, start, ints([0, 1, 2]), table, page, q, kp, vp,
                   temp=scale, rot_half=half, head_norm=head_norm)
        got.append((q, kp, vp, t))
    assert all(torch.equal(a, b) for a, b in zip(*got)) and got[0][0].float().abs().max() > 0


@pytest.mark.parametrize("dr,dims,half", [(64, 64, False), (64, 32, True), (0, 0, False)])
def test_latent_qkv_four_elements_a_thread_has_the_same_bits(K, dr, dims, half):
    g = torch.Generator().manual_seed(dr + dims)
    T, H, dn, R, page = 37, 5, 24, 96, 8
    u, w, freq = torch.randn(T, H * (dn + dr) + R + dr, generator=g).to(DEV), torch.randn(R, generator=g).to(DEV), torch.rand(max(1, dims // 2), generator=g).to(DEV)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pos, req, table = ints(list(range(T))), ints([0] * T), ints([list(range(1, 6))])
    got = []
    for move in (lambda t: t, _off):
        plain, full, pages = torch.zeros(T, H * dn, device=DEV).bfloat16(), torch.zeros(T, H * (R + dr), device=DEV).bfloat16(), torch.zeros(6, page, R + dr, device=DEV).bfloat16()
        K.latent_qkv(move(u), 0, H * (dn + dr), H, dn, dr, R, dims, freq, 1.2, w, 1e-5, pos, req, table, page, plain, full, pages, rot_half=half)
        got.append((plain, full, pages))
    assert all(torch.equal(a, b) for a, b in zip(*got)) and got[0][0].abs().max() > 0


def _scatter_pages(k, v, tables, page, num_pages, dtype, junk=7.0):
    """Dense per-request keys/values [len, nkvh, dh] -> pages [num_pages, nkvh, page, dh]."""
    nkvh, dh = k[0].shape[1:]
    kp = torch.full((num_pages, nkvh, page, dh), junk).to(dtype)       # junk where nothing was written
    vp = torch.full((num_pages, nkvh, page, dh), -junk).to(dtype)
    for r, (kr, vr) in enumerate(zip(k, v)):
        for j in range(kr.shape[0]):
            p = tables[r][j // page]
            kp[p, :, j % page] = kr[j].to(dtype)
            vp[p, :, j % page] = vr[j].to(dtype)
    return kp, vp


@pytest.mark.parametrize("nh,nkvh,dh,page,with_rope", [(4, 2, 64, 16, True), (3, 1, 128, 8, True), (5, 5, 64, 32, False),
                                                        (9, 3, 64, 16, True)])
def test_qkv_product_rotates_and_writes_the_cache_in_its_epilogue(K, pairs, nh, nkvh, dh, page, with_rope):
    """The tcgen05 product of the fused [q | k | v] matrix, rotation and cache write included, against
    a plain product, a plain rotation and a plain scatter."""
    assert K.gemm_tcgen05_qkv_supports(dh) and not K.gemm_tcgen05_qkv_supports(48)
    g = torch.Generator().manual_seed(dh + nh)
    lens = [(37, 150), (0, 131), (200, 3)]              # (start position, rows): tiles of 128 rows straddle requests
    T = sum(n for _, n in lens)
    kdim = 200
    width = (nh + 2 * nkvh) * dh
    act = (torch.randn(T, kdim, generator=g) * 0.5).to(torch.bfloat16)
    w = (torch.randn(width, kdim, generator=g) * 0.1).to(torch.bfloat16)
    max_pos, theta = 384, 5000.0
    j = torch.arange(dh // 2, dtype=torch.float64)
    ang = torch.arange(max_pos, dtype=torch.float64)[:, None] / theta ** (j / (dh // 2))
    cos, sin = ang.cos().float(), ang.sin().float()
    max_blocks = max_pos // page
    table = (torch.randperm(3 * max_blocks, generator=g) + 1).view(3, max_blocks).to(torch.int32)
    positions = torch.cat([torch.arange(s, s + n) for s, n in lens]).to(torch.int32)
    row_req = torch.cat([torch.full((n,), i) for i, (_, n) in enumerate(lens)]).to(torch.int32)
    num_pages = 3 * max_blocks + 1
    kp = torch.zeros(num_pages, nkvh, page, dh, dtype=torch.bfloat16, device=DEV)
    vp = torch.zeros_like(kp)
    q_out = torch.full((T, nh * dh), 9.0, dtype=torch.bfloat16, device=DEV)
    K.gemm_tcgen05_qkv(act.to(DEV), w.to(DEV), q_out, kp, vp, cos.to(DEV) if with_rope else None,
                       sin.to(DEV) if with_rope else None, positions.to(DEV), row_req.to(DEV), table.to(DEV), nh)
    K.check_gemm_status(DEV)
    x = act.double() @ w.double().T
    q = x[:, :nh * dh].view(T, nh, dh)
    k = x[:, nh * dh:(nh + nkvh) * dh].view(T, nkvh, dh)
    v = x[:, (nh + nkvh) * dh:].view(T, nkvh, dh)
    rot = (lambda t: plain_rope(t, positions, theta)) if with_rope else (lambda t: t)
    _close(q_out.view(T, nh, dh), rot(q), torch.bfloat16, scale=2.0)
    want_k = torch.zeros(num_pages, nkvh, page, dh, dtype=torch.float64)
    want_v = torch.zeros_like(want_k)
    rk = rot(k)
    for t in range(T):
        p = int(table[row_req[t], positions[t] // page])
        want_k[p, :, positions[t] % page] = rk[t]
        want_v[p, :, positions[t] % page] = v[t]
    _close(kp, want_k, torch.bfloat16, scale=2.0)
    _close(vp, want_v, torch.bfloat16, scale=2.0)
    assert float(kp[0].abs().max()) == 0.0              # the null page was not written


@pytest.mark.parametrize("nh,nkvh,dh,page,with_rope,rows", [(4, 2, 64, 16, True, 8), (3, 1, 128, 8, True, 1), (5, 5, 48, 32, False, 16),
                                                             (9, 3, 16, 16, True, 11), (2, 2, 80, 4, True, 5)])
def test_small_row_qkv_product_rotates_and_writes_the_cache_in_its_epilogue(K, nh, nkvh, dh, page, with_rope, rows):
    """The same for at most 16 rows (decoded tokens of several requests): the small-row kernel."""
    kdim = 160
    assert K.linear_small_qkv_supports(rows, kdim, dh) and not K.linear_small_qkv_supports(17, kdim, dh)
    assert not K.linear_small_qkv_supports(rows, kdim, 24)
    g = torch.Generator().manual_seed(dh + nh + rows)
    width = (nh + 2 * nkvh) * dh
    act = (torch.randn(rows, kdim, generator=g) * 0.5).to(torch.bfloat16)
    w = (torch.randn(width, kdim, generator=g) * 0.1).to(torch.bfloat16)
    max_pos, theta = 96, 5000.0
    j = torch.arange(dh // 2, dtype=torch.float64)
    ang = torch.arange(max_pos, dtype=torch.float64)[:, None] / theta ** (j / (dh // 2))
    cos, sin = ang.cos().float(), ang.sin().float()
    max_blocks = max_pos // page
    table = (torch.randperm(rows * max_blocks, generator=g) + 1).view(rows, max_blocks).to(torch.int32)
    positions = torch.randint(0, max_pos, (rows,), generator=g).to(torch.int32)      # one decoded token per request
    row_req = torch.arange(rows, dtype=torch.int32)
    num_pages = rows * max_blocks + 1
    kp = torch.zeros(num_pages, nkvh, page, dh, dtype=torch.bfloat16, device=DEV)
    vp = torch.zeros_like(kp)
    q_out = torch.full((rows, nh * dh), 9.0, dtype=torch.bfloat16, device=DEV)
    K.linear_small_qkv(act.to(DEV), w.to(DEV), q_out, kp, vp, cos.to(DEV) if with_rope else None,
                       sin.to(DEV) if with_rope else None, positions.to(DEV), row_req.to(DEV), table.to(DEV), nh)
    x = act.double() @ w.double().T
    q = x[:, :nh * dh].view(rows, nh, dh)
    k = x[:, nh * dh:(nh + nkvh) * dh].view(rows, nkvh, dh)
    v = x[:, (nh + nkvh) * dh:].view(rows, nkvh, dh)
    rot = (lambda t: plain_rope(t, positions, theta)) if with_rope else (lambda t: t)
    _close(q_out.view(rows, nh, dh), rot(q), torch.bfloat16, scale=2.0)
    want_k = torch.zeros(num_pages, nkvh, page, dh, dtype=torch.float64)
    want_v = torch.zeros_like(want_k)
    rk = rot(k)
    for t in range(rows):
        p = int(table[row_req[t], positions[t] // page])
        want_k[p, :, positions[t] % page] = rk[t]
        want_v[p, :, positions[t] % page] = v[t]
    _close(kp, want_k, torch.bfloat16, scale=2.0)
    _close(vp, want_v, torch.bfloat16, scale=2.0)
    assert float(kp[0].abs().max()) == 0.0              # the null page was not written


@pytest.mark.parametrize("rows,width,kdim", [(8, 96, 160), (1, 40, 64), (16, 333, 2304), (11, 2304, 5760)])
def test_a_chain_of_few_row_products_carries_the_norm_between_them(K, rows, width, kdim):
    """The product before a norm adds itself into the residual stream, leaves bfloat16(x * norm weight) and the
    rows' sums of squares; the product after it scales its rows by 1 / rms: together they are product, residual
    add, RMSNorm and product, without a norm kernel."""
    assert K.linear_small_norm_supports(rows, width, kdim) and not K.linear_small_norm_supports(17, width, kdim)
    g = torch.Generator().manual_seed(rows + width + kdim)
    act = (torch.randn(rows, kdim, generator=g)).to(torch.bfloat16)
    w = (torch.randn(width, kdim, generator=g) / math.sqrt(kdim)).to(torch.bfloat16)
    x0 = torch.randn(rows, width, generator=g) * 3
    gain = 1 + 0.1 * torch.randn(width, generator=g)
    eps, scale = 1e-5, 0.7
    x = x0.to(DEV).clone()
    xb = torch.full((rows, width), 9.0, dtype=torch.bfloat16, device=DEV)
    sumsq = torch.zeros(16, dtype=torch.int64, device=DEV)
    K.linear_small_norm(act.to(DEV), w.to(DEV), x, K.EPI_RESIDUAL, xb=xb, next_w=gain.to(DEV), out_sumsq=sumsq, scale=scale)
    want_x = x0.double() + scale * (act.double() @ w.double().T)
    torch.testing.assert_close(x.double().cpu(), want_x, rtol=1e-5, atol=1e-5)
    _close(xb, want_x * gain.double(), torch.bfloat16, scale=2.0)
    got_ss = sumsq[:rows].cpu().double() / K.SUMSQ_FIXED
    torch.testing.assert_close(got_ss, (want_x ** 2).sum(-1), rtol=1e-5, atol=1e-5)
    assert int(sumsq[rows:].abs().max()) == 0 if rows < 16 else True
    # the same again gives the same counters to the last bit (integer additions, whatever the order of the tiles)
    x2, sumsq2 = x0.to(DEV).clone(), torch.zeros_like(sumsq)
    K.linear_small_norm(act.to(DEV), w.to(DEV), x2, K.EPI_RESIDUAL, xb=torch.empty_like(xb), next_w=gain.to(DEV), out_sumsq=sumsq2, scale=scale)
    assert torch.equal(sumsq, sumsq2) and torch.equal(x, x2)
    # without activations for a next product (the last layer): only the addition
    x3 = x0.to(DEV).clone()
    K.linear_small_norm(act.to(DEV), w.to(DEV), x3, K.EPI_RESIDUAL, scale=scale)
    assert torch.equal(x3, x)
    # the product after the norm: plain output and SwiGLU
    n2 = 72
    w2 = (torch.randn(2 * n2, width, generator=g) * 2 / math.sqrt(width)).to(torch.bfloat16)
    if K.linear_small_norm_supports(rows, n2, width):
        # the activations are what the first product left (rounded to bfloat16 before the 1 / rms)
        inv = 1 / torch.sqrt((want_x ** 2).mean(-1, keepdim=True) + eps)
        out = torch.full((rows, 2 * n2), 9.0, device=DEV)
        K.linear_small_norm(xb, w2.to(DEV), out, K.EPI_F32, in_sumsq=sumsq, in_eps=eps)
        ref = (xb.double().cpu() @ w2.double().T) * inv
        _close(out, ref, torch.bfloat16, scale=2.0)
        act2 = torch.full((rows, n2), 9.0, dtype=torch.bfloat16, device=DEV)
        K.linear_small_norm(xb, w2.to(DEV), act2, K.EPI_SWIGLU, in_sumsq=sumsq, in_eps=eps)
        _close(act2, ref[:, :n2] * torch.sigmoid(ref[:, :n2]) * ref[:, n2:], torch.bfloat16, scale=2.0)


def test_sums_of_squares_beyond_the_counters_are_reported(K):
    """The counters hold sums up to 2^38 a row; a tile whose share is beyond 2^27 says so in the status word that
    the engine checks, instead of wrapping around."""
    rows, width, kdim = 4, 64, 64
    act = torch.zeros(rows, kdim, dtype=torch.bfloat16, device=DEV)
    w = torch.zeros(width, kdim, dtype=torch.bfloat16, device=DEV)
    x = torch.full((rows, width), 1.0e4, device=DEV)          # 16 features x 1e8 = 1.6e9 a tile and row
    x[0] = 1.0
    sumsq = torch.zeros(16, dtype=torch.int64, device=DEV)
    K.check_gemm_status(DEV)
    K.linear_small_norm(act, w, x, K.EPI_RESIDUAL, xb=torch.empty(rows, width, dtype=torch.bfloat16, device=DEV),
                        next_w=torch.ones(width, device=DEV), out_sumsq=sumsq)
    with pytest.raises(K.KernelError, match="sum of squares"):
        K.check_gemm_status(DEV)
    K.check_gemm_status(DEV)                                   # the word was cleared
    assert int(sumsq[0]) == int(width * K.SUMSQ_FIXED)         # the row within range was counted as ever


def test_small_row_qkv_product_scales_its_rows_by_the_norm(K):
    nh, nkvh, dh, page, rows, kdim = 4, 2, 64, 16, 7, 192
    g = torch.Generator().manual_seed(3)
    width = (nh + 2 * nkvh) * dh
    x = torch.randn(rows, kdim, generator=g) * 4
    gain = 1 + 0.1 * torch.randn(kdim, generator=g)
    eps = 1e-6
    xb = (x * gain).to(torch.bfloat16)
    sumsq = torch.zeros(16, dtype=torch.int64)
    sumsq[:rows] = ((x.double() ** 2).sum(-1) * K.SUMSQ_FIXED).round().long()
    h = (x.double() * gain.double() / torch.sqrt((x.double() ** 2).mean(-1, keepdim=True) + eps)).float().to(torch.bfloat16)
    w = (torch.randn(width, kdim, generator=g) * 0.1).to(torch.bfloat16)
    max_pos, theta = 96, 5000.0
    j = torch.arange(dh // 2, dtype=torch.float64)
    ang = torch.arange(max_pos, dtype=torch.float64)[:, None] / theta ** (j / (dh // 2))
    cos, sin = ang.cos().float().to(DEV), ang.sin().float().to(DEV)
    max_blocks = max_pos // page
    table = (torch.randperm(rows * max_blocks, generator=g) + 1).view(rows, max_blocks).to(torch.int32).to(DEV)
    positions = torch.randint(0, max_pos, (rows,), generator=g).to(torch.int32).to(DEV)
    row_req = torch.arange(rows, dtype=torch.int32, device=DEV)
    num_pages = rows * max_blocks + 1
    kp = torch.zeros(num_pages, nkvh, page, dh, dtype=torch.bfloat16, device=DEV)
    vp = torch.zeros_like(kp)
    q_out = torch.full((rows, nh * dh), 9.0, dtype=torch.bfloat16, device=DEV)
    K.linear_small_qkv_norm(xb.to(DEV), w.to(DEV), q_out, kp, vp, cos, sin, positions, row_req, table, nh, sumsq.to(DEV), eps)
    # what it has to be: the product of the activations as they are (rounded before the 1 / rms), scaled, rotated
    inv = 1 / torch.sqrt((x.double() ** 2).mean(-1, keepdim=True) + eps)
    y = (xb.double() @ w.double().T) * inv
    q = y[:, :nh * dh].view(rows, nh, dh)
    k = y[:, nh * dh:(nh + nkvh) * dh].view(rows, nkvh, dh)
    v = y[:, (nh + nkvh) * dh:].view(rows, nkvh, dh)
    pos = positions.cpu()
    _close(q_out.view(rows, nh, dh), plain_rope(q, pos, theta), torch.bfloat16, scale=2.0)
    rk = plain_rope(k, pos, theta)
    for t in range(rows):
        p = int(table[t, pos[t] // page])
        _close(kp[p, :, pos[t] % page], rk[t], torch.bfloat16, scale=2.0)
        _close(vp[p, :, pos[t] % page], v[t], torch.bfloat16, scale=2.0)
    # and it is the plain kernel's result on normalised activations, up to where those were rounded
    kp2, vp2, q2 = torch.zeros_like(kp), torch.zeros_like(vp), torch.empty_like(q_out)
    K.linear_small_qkv(h.to(DEV), w.to(DEV), q2, kp2, vp2, cos, sin, positions, row_req, table, nh)
    assert float((q2.float() - q_out.float()).abs().max()) <= 0.05 * float(q2.float().abs().max())


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nh,nkvh,dh,page,interleaved", [(6, 2, 48, 8, False), (4, 4, 16, 16, True),
                                                          (3, 1, 128, 4, False), (8, 2, 256, 32, False)])
def test_rope_and_cache_write(K, dtype, nh, nkvh, dh, page, interleaved):
    g = torch.Generator().manual_seed(dh + nh)
    lens = [(5, 9), (0, 3), (20, 1)]                    # (start position, rows) of three requests
    T = sum(n for _, n in lens)
    width = (nh + 2 * nkvh) * dh
    qkv = torch.randn(T, width, generator=g)
    bias = torch.randn(width, generator=g) * 0.1
    max_pos, theta = 64, 5000.0
    j = torch.arange(dh // 2, dtype=torch.float64)
    ang = torch.arange(max_pos, dtype=torch.float64)[:, None] / theta ** (j / (dh // 2))
    cos, sin = ang.cos().float(), ang.sin().float()
    max_blocks = max_pos // page
    perm = torch.randperm(3 * max_blocks, generator=g) + 1
    table = perm.view(3, max_blocks).to(torch.int32)
    positions = torch.cat([torch.arange(s, s + n) for s, n in lens]).to(torch.int32)
    row_req = torch.cat([torch.full((n,), i) for i, (_, n) in enumerate(lens)]).to(torch.int32)
    num_pages = 3 * max_blocks + 1
    kp = torch.zeros(num_pages, nkvh, page, dh, dtype=dtype, device=DEV)
    vp = torch.zeros_like(kp)
    q_out = torch.empty(T, nh * dh, dtype=dtype, device=DEV)
    K.rope_kv(qkv.to(DEV), bias.to(DEV), positions.to(DEV), row_req.to(DEV), table.to(DEV), page,
              cos.to(DEV), sin.to(DEV), interleaved, q_out, kp, vp, T, nh, nkvh, dh)
    x = (qkv + bias).double()
    q = x[:, :nh * dh].view(T, nh, dh)
    k = x[:, nh * dh:(nh + nkvh) * dh].view(T, nkvh, dh)
    v = x[:, (nh + nkvh) * dh:].view(T, nkvh, dh)
    if interleaved:
        def rot(t):
            c, s = ang[positions.long()][:, None, :].cos(), ang[positions.long()][:, None, :].sin()
            o = torch.empty_like(t)
            o[..., 0::2] = t[..., 0::2] * c - t[..., 1::2] * s
            o[..., 1::2] = t[..., 0::2] * s + t[..., 1::2] * c
            return o
    else:
        rot = lambda t: plain_rope(t, positions, theta)
    _close(q_out.view(T, nh, dh), rot(q), dtype, scale=4.0)
    want_k = torch.zeros(num_pages, nkvh, page, dh, dtype=torch.float64)
    want_v = torch.zeros_like(want_k)
    rk = rot(k)
    for t in range(T):
        p = int(table[row_req[t], positions[t] // page])
        want_k[p, :, positions[t] % page] = rk[t]
        want_v[p, :, positions[t] % page] = v[t]
    _close(kp, want_k, dtype, scale=4.0)
    _close(vp, want_v, dtype, scale=4.0)
    assert float(kp[0].abs().max()) == 0.0              # the null page was not written


def _attention_case(K, dtype, nh, nkvh, dh, page, window, lens, queries, plant=None, seed=0, impl="rows", splits=1, junk=7.0, tile_keys=0):
    """lens: cached length of each request; queries: per request the positions that are rows.
    impl: "rows" (one warp per row and head), "decode" (split keys), "prefill" (tensor cores; the
    positions of a request must be consecutive)."""
    g = torch.Generator().manual_seed(seed)
    R = len(lens)
    k = [torch.randn(n, nkvh, dh, generator=g) for n in lens]
    v = [torch.randn(n, nkvh, dh, generator=g) for n in lens]
    qf = [torch.randn(n, nh, dh, generator=g) for n in lens]
    if plant:
        # one key far back gets a score that stands out: the row's output must be that key's value
        for (r, qpos, kpos, head) in plant:
            kk = k[r][kpos, head // (nh // nkvh)]
            qf[r][qpos, head] = kk * (40.0 / float(kk.norm()) ** 2) * math.sqrt(dh)
    qf = [t.to(dtype).float() for t in qf]; k = [t.to(dtype).float() for t in k]; v = [t.to(dtype).float() for t in v]
    max_blocks = (max(lens) + page - 1) // page + 1
    perm = (torch.randperm(R * max_blocks, generator=g) + 1).view(R, max_blocks)
    tables = perm.tolist()
    num_pages = R * max_blocks + 1
    kp, vp = _scatter_pages(k, v, tables, page, num_pages, dtype, junk)
    positions = torch.tensor([p for r in range(R) for p in queries[r]], dtype=torch.int32)
    row_req = torch.tensor([r for r in range(R) for _ in queries[r]], dtype=torch.int32)
    q = torch.stack([qf[r][p] for r in range(R) for p in queries[r]]).to(dtype)
    T = q.shape[0]
    out = torch.full((T, nh * dh), 55.0, dtype=dtype, device=DEV)
    scale = dh ** -0.5
    bt = perm.to(torch.int32).to(DEV)
    qd, kd, vd = q.view(T, nh * dh).to(DEV), kp.to(DEV), vp.to(DEV)
    if impl == "rows":
        K.attention_rows(qd, kd, vd, out, positions.to(DEV), row_req.to(DEV), bt, T, nh, scale, window or 0)
    elif impl == "decode":
        # work on a shuffled list of all rows, to show that the list is honoured
        rows = torch.randperm(T, generator=g).to(torch.int32).to(DEV)
        K.attention_decode(qd, kd, vd, out, rows, T, positions.to(DEV), row_req.to(DEV), bt, nh, scale,
                           window or 0, splits)
    else:                                                  # "prefill" (mma.sync) or "tcgen05"
        starts = [0]
        for r in range(R):
            assert list(queries[r]) == list(range(queries[r][0], queries[r][0] + len(queries[r]))) if len(queries[r]) else True
            starts.append(starts[-1] + len(queries[r]))
        tiles = [(r, t0) for r in range(R) for t0 in range(starts[r], starts[r + 1], K.TILE_ROWS)]
        req_pos = [queries[r][0] if len(queries[r]) else 0 for r in range(R)]
        i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
        if impl == "tcgen05":
            K.attention_tcgen05(qd, kd, vd, out, i32(tiles).flatten(), len(tiles), T, i32(starts), i32(req_pos), bt, nh,
                                scale, window or 0, tile_keys=tile_keys)
            K.check_gemm_status(DEV)
        else:
            K.attention_prefill(qd, kd, vd, out, i32(tiles).flatten(), len(tiles), i32(starts), i32(req_pos), bt, nh,
                                scale, window or 0)
    want = torch.cat([plain_attention(qf[r].double(), k[r].double(), v[r].double(), scale, window)[queries[r]]
                      for r in range(R) if len(queries[r])])
    return out.view(T, nh, dh), want, v


SHAPES = [(4, 4, 16, 16, None), (3, 1, 32, 8, None), (6, 2, 48, 4, None), (8, 2, 128, 16, None),
          (5, 5, 64, 16, 7), (2, 1, 80, 32, 33), (2, 2, 256, 16, None), (16, 1, 64, 16, None), (10, 2, 96, 5, 70)]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nh,nkvh,dh,page,window", SHAPES[:7])
def test_attention_rows_over_pages(K, dtype, nh, nkvh, dh, page, window):
    lens = [37, 1, 130, 64]
    # a portion at the end, a single first token, decoded tokens, a whole prompt cut at page edges
    queries = [list(range(30, 37)), [0], [129], list(range(0, 64))]
    got, want, _ = _attention_case(K, dtype, nh, nkvh, dh, page, window, lens, queries, seed=dh)
    _close(got, want, dtype, scale=2.0)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nh,nkvh,dh,page,window", [(1, 1, 4, 16, None), (40, 1, 20, 8, None), (6, 2, 6, 4, 50), (3, 3, 512, 16, 33), (16, 1, 130, 16, 31)])
def test_attention_rows_tiles(K, dtype, nh, nkvh, dh, page, window):
    """Tiles of rows at their edges (32, 16, 10 and 2 rows of a request a block, more heads than a block takes), the rest of the
    cache not a number, and every row alone: the same bits."""
    lens = [70, 33, 1, 65]
    queries = [list(range(3, 70)), [32], [0], list(range(31, 65))]
    got, want, _ = _attention_case(K, dtype, nh, nkvh, dh, page, window, lens, queries, seed=dh, junk=float("nan"))
    _close(got, want, dtype, scale=2.0)
    # the same rows as other tiles: one request less ahead of them
    less, _, _ = _attention_case(K, dtype, nh, nkvh, dh, page, window, lens, [list(range(5, 70)), [], [0], list(range(31, 65))], seed=dh, junk=float("nan"))
    assert torch.equal(torch.cat([got[2:67], got[68:]]), less)


@pytest.mark.parametrize("dtype,nh,nkvh,dh,dv,page,window,lens,rows", [
    # (dtype, heads, sizes, page, window (< 0: chunks), histories, rows of each request)
    (torch.float32, 4, 4, 16, 16, 8, 0, [1, 24, 17, 9], [1, 1, 2, 1]), (torch.float32, 2, 1, 256, 256, 8, 7, [24, 1, 23], [1, 1, 1]),
    (torch.bfloat16, 2, 2, 192, 160, 6, -10, [24, 11, 10, 1], [1, 1, 1, 1]), (torch.float32, 3, 3, 7, 30, 8, 9, [24, 24], [1, 1]),
    (torch.float32, 20, 20, 64, 48, 8, 5, [24, 19], [24, 1]), (torch.bfloat16, 40, 40, 40, 40, 8, 0, [24], [14]),
    (torch.bfloat16, 4, 2, 32, 32, 16, 50, [256, 100, 31, 33], [1, 1, 1, 1]), (torch.bfloat16, 4, 4, 16, 16, 16, -32, [256, 65, 64, 1], [1, 1, 1, 1])])
@pytest.mark.parametrize("extra", ["none", "sink and gate", "element gate, cap and kept keys"])
def test_attention_rows_by_warps_and_by_blocks(K, dtype, nh, nkvh, dh, dv, page, window, lens, rows, extra):
    """Not to know a bound on the histories moves a call from one kernel to the other: the same bits, whatever lies behind the histories."""
    from infinicore_infer_b200.kernels.host import attention_rows_walk
    g, R, T = torch.Generator().manual_seed(dh), len(lens), sum(rows)
    r = lambda *s: torch.randn(*s, generator=g)
    few = -(-max(lens) // page)
    kp, vp = r(R * few + 1, nkvh, page, dh), r(R * few + 1, nkvh, page, dv)
    table = (torch.randperm(R * few, generator=g) + 1).view(R, few)
    for i, n in enumerate(lens):
        if n % page:
            kp[table[i, n // page], :, n % page:], vp[table[i, n // page], :, n % page:] = float("nan"), float("nan")
    positions = torch.tensor([n - m + i for n, m in zip(lens, rows) for i in range(m)], dtype=torch.int32, device=DEV)
    row_req = torch.tensor([i for i, m in enumerate(rows) for _ in range(m)], dtype=torch.int32, device=DEV)
    q, kp, vp = (t.to(dtype).to(DEV) for t in (r(T, nh * dh), kp, vp))
    keep = 4 if window > 0 else 0
    options = {"none": {}, "sink and gate": dict(sink=True, sink_w=r(nh).to(DEV), gate=r(T, nh).to(DEV)),
               "element gate, cap and kept keys": dict(gate=r(T, nh * dv).to(DEV), gate_elem=True, cap=3.0, keep_first=keep)}[extra]
    for context, walks in ((max(lens), True), (0, False)):
        assert attention_rows_walk(T, R, min(context, window + keep) if window > 0 else context, nh, nkvh, max(dh, dv), 4 if dtype == torch.float32 else 2) == walks
    got = [K.attention_rows(q, kp, vp, torch.full((T, nh * dv), 55.0, dtype=dtype, device=DEV), positions, row_req, table.to(torch.int32).to(DEV), T, nh,
                            dh ** -0.5, window, context=context, **options) for context in (max(lens), 0)]
    assert torch.isfinite(got[0].float()).all() and torch.equal(*got)


# grouped heads of 64 or 128: the decode kernel that puts the group on the tensor cores (16 heads fill a tile;
# 20 need a second one; 2 to 7 leave most of it empty)
GROUPED = [(32, 2, 128, 16, None), (10, 2, 64, 16, 70), (40, 2, 128, 8, None), (6, 1, 64, 32, 33), (7, 1, 128, 5, None),
           (6, 3, 64, 16, None), (24, 8, 64, 16, 100)]


@pytest.mark.parametrize("splits", [1, 2, 5, 32])
@pytest.mark.parametrize("nh,nkvh,dh,page,window", SHAPES + GROUPED)
def test_attention_decode_kernel_with_split_keys(K, nh, nkvh, dh, page, window, splits):
    lens = [37, 1, 300, 64, 2]
    queries = [list(range(30, 37)), [0], [299], [62, 63], [0, 1]]
    got, want, _ = _attention_case(K, torch.bfloat16, nh, nkvh, dh, page, window, lens, queries, seed=dh,
                                   impl="decode", splits=splits)
    _close(got, want, torch.bfloat16, scale=2.0)


@pytest.mark.parametrize("nh,nkvh,dh,page,window", [s for s in SHAPES if s[2] != 256] + [(2, 2, 256, 16, None), (4, 2, 64, 16, 100)])
def test_attention_prefill_kernel_on_tensor_cores(K, nh, nkvh, dh, page, window):
    # a whole prompt of several tiles with a ragged end; a portion that starts mid-page far into the
    # context; a portion of exactly one tile; a short one
    lens = [150, 333, 64, 40]
    queries = [list(range(0, 150)), list(range(203, 333)), list(range(0, 64)), list(range(31, 40))]
    got, want, _ = _attention_case(K, torch.bfloat16, nh, nkvh, dh, page, window, lens, queries, seed=dh, impl="prefill")
    _close(got, want, torch.bfloat16, scale=2.0)


@pytest.mark.parametrize("dh", [64, 128])
@pytest.mark.parametrize("requests,splits", [(3, 4), (40, 2), (18, 8), (20, 8)])
def test_grouped_decode_attention_in_blocks_of_four_and_of_eight_warps(K, dh, requests, splits):
    """A launch of at most one block an SM (3 requests x 2 key/value heads x 4 cuts) runs blocks of eight warps on tiles
    of 128 keys, a larger one blocks of four on tiles of 64, whose cuts merge inside clusters (heads of 64: 40 x 2 x 2 and
    18 x 2 x 8) or through the merge kernel (20 x 2 x 8, and heads of 128); all against the plain attention, with a key
    far back that a row must find."""
    nh, nkvh, page = 32, 2, 16
    g = torch.Generator().manual_seed(requests)
    lens = [int(x) for x in torch.randint(130, 700, (requests,), generator=g)]
    queries = [[n - 1] for n in lens]
    plant = [(0, lens[0] - 1, 3, 17), (requests - 1, lens[-1] - 1, lens[-1] // 2, 5)]
    got, want, v = _attention_case(K, torch.bfloat16, nh, nkvh, dh, page, None, lens, queries, plant=plant, seed=7,
                                   impl="decode", splits=splits)
    _close(got, want, torch.bfloat16, scale=2.0)
    assert torch.allclose(got[0, 17].float().cpu(), v[0][3, 17 // 16], atol=2e-2)        # the row found the far key
    assert torch.allclose(got[requests - 1, 5].float().cpu(), v[-1][lens[-1] // 2, 0], atol=2e-2)


@pytest.mark.parametrize("nh,nkvh,dh,page,window", [(4, 4, 64, 16, None), (3, 1, 64, 8, None), (8, 2, 128, 16, None),
                                                     (6, 2, 64, 32, 100), (2, 1, 128, 64, 33), (4, 2, 64, 128, None),
                                                     (36, 36, 64, 16, None)])
def test_attention_prefill_kernel_on_tcgen05(K, nh, nkvh, dh, page, window):
    assert K.attention_tcgen05_supports(dh, page) and not K.attention_tcgen05_supports(48, 16)
    lens = [150, 460, 128, 40]
    queries = [list(range(0, 150)), list(range(203, 460)), list(range(0, 128)), list(range(31, 40))]
    got, want, _ = _attention_case(K, torch.bfloat16, nh, nkvh, dh, page, window, lens, queries, seed=dh + page, impl="tcgen05")
    _close(got, want, torch.bfloat16, scale=2.0)


@pytest.mark.parametrize("tile_keys", [64, 128])
@pytest.mark.parametrize("page,window", [(8, None), (64, None), (128, None), (16, 70), (32, 64)])
def test_attention_tcgen05_tiles_of_64_keys(K, page, window, tile_keys):
    """Heads of 128 walk 128 keys at a time, or 64 where a page fits into that (pages of 128: always 128): prompts and portions that end
    at, one before and one past the edges of key tiles and of query tiles; the operands and the bound of the cases above."""
    lens = [64, 65, 127, 193, 321]
    queries = [list(range(0, 64)), list(range(0, 65)), list(range(62, 127)), list(range(0, 193)), list(range(192, 321))]
    got, want, _ = _attention_case(K, torch.bfloat16, 6, 2, 128, page, window, lens, queries, seed=page, impl="tcgen05", tile_keys=tile_keys)
    _close(got, want, torch.bfloat16, scale=2.0)


@pytest.mark.parametrize("impl,dtype", [("rows", torch.float32), ("rows", torch.bfloat16), ("decode", torch.bfloat16),
                                         ("decode grouped", torch.bfloat16), ("prefill", torch.bfloat16),
                                         ("tcgen05", torch.bfloat16)])
@pytest.mark.parametrize("window", [None, 50])
def test_attention_finds_one_far_key_among_hundreds(K, impl, dtype, window):
    nh, nkvh, dh, page = 4, 2, 64, 16
    if impl == "decode grouped":                 # six query heads per key/value head instead of two
        nh, impl = 12, "decode"
    lens = [700]
    # the query at 699 must find key 3 (or, with a window, the key at the window's far edge); the query
    # at 320 the key at 319, across a page's edge
    far = 3 if window is None else 699 - window + 1
    plant = [(0, 699, far, 1), (0, 320, 319, 2)]
    if impl in ("prefill", "tcgen05"):
        queries, i699, i320 = [list(range(300, 700))], 399, 20
    else:
        queries, i699, i320 = [[320, 512, 699]], 2, 0
    kw = dict(impl=impl, splits=3) if impl != "rows" else {}
    got, want, v = _attention_case(K, dtype, nh, nkvh, dh, page, window, lens, queries, plant, seed=5, **kw)
    _close(got, want, dtype, scale=2.0)
    group = nh // nkvh
    assert torch.allclose(got[i699, 1].float().cpu(), v[0][far, 1 // group], atol=2e-2)
    assert torch.allclose(got[i320, 2].float().cpu(), v[0][319, 2 // group], atol=2e-2)
    if window:
        # one position beyond the window's edge must NOT be seen
        plant = [(0, 699, far - 1, 1)]
        got, want, v = _attention_case(K, dtype, nh, nkvh, dh, page, window, lens, queries, plant, seed=5, **kw)
        _close(got, want, dtype, scale=2.0)
        assert not torch.allclose(got[i699, 1].float().cpu(), v[0][far - 1, 1 // group], atol=0.2)


@pytest.mark.parametrize("junk", [float("nan"), float("inf")])
@pytest.mark.parametrize("impl,dtype,nh,nkvh,dh,page", [
    ("rows", torch.float32, 4, 2, 48, 8), ("rows", torch.bfloat16, 4, 4, 16, 16), ("decode", torch.bfloat16, 3, 3, 32, 8),
    ("decode", torch.bfloat16, 6, 2, 64, 16), ("decode", torch.bfloat16, 8, 2, 128, 16), ("prefill", torch.bfloat16, 4, 2, 64, 16),
    ("prefill", torch.bfloat16, 2, 1, 80, 32), ("tcgen05", torch.bfloat16, 4, 2, 64, 16), ("tcgen05", torch.bfloat16, 4, 2, 128, 64),
    ("tcgen05", torch.bfloat16, 2, 2, 64, 128)])
def test_attention_ignores_what_lies_beyond_a_request_s_length(K, impl, dtype, nh, nkvh, dh, page, junk):
    """The slots of a held page beyond the request's last position, and pages that were never written, may hold
    anything: what another request left there (a request whose activations overflowed leaves NaN or Inf) or what
    the allocator handed out.  No kernel may let it reach a result, not even multiplied by a weight of zero."""
    lens = [150, 333, 70, 41]
    if impl in ("prefill", "tcgen05"):
        queries = [list(range(0, 150)), list(range(203, 333)), list(range(6, 70)), list(range(31, 41))]
    else:
        queries = [[149], [331, 332], [69], list(range(36, 41))]
    kw = dict(impl=impl, splits=3) if impl == "decode" else dict(impl=impl)
    got, want, _ = _attention_case(K, dtype, nh, nkvh, dh, page, None, lens, queries, seed=dh + page, junk=junk, **kw)
    assert torch.isfinite(got.float()).all()
    _close(got, want, dtype, scale=2.0)


@pytest.mark.parametrize("V", [5, 301, 122753])
def test_argmax_takes_the_first_of_equal_maxima(K, V):
    g = torch.Generator().manual_seed(V)
    logits = torch.randn(3, V, generator=g)
    logits[1, V - 1] = 50.0
    logits[2, V // 2] = 60.0; logits[2, V // 3] = 60.0
    out = torch.empty(3, dtype=torch.int32, device=DEV)
    K.argmax(logits.to(DEV), out)
    assert out.tolist() == [int(logits[0].argmax()), V - 1, V // 3]
    # rows with a stride (a padded leading dimension)
    wide = torch.zeros(3, V + 3)
    wide[:, :V] = logits
    K.argmax(wide.to(DEV)[:, :V], out)
    assert out.tolist() == [int(logits[0].argmax()), V - 1, V // 3]


@pytest.mark.parametrize("V", [37, 1000, 122753])
def test_sample_matches_the_plain_rule(K, V):
    g = torch.Generator().manual_seed(V)
    cases = []
    for i, (temp, topk, topp) in enumerate([(0.0, 0, 1.0), (1.0, 1, 1.0), (1.0, 0, 1.0), (0.8, 0, 1.0), (2.5, 0, 1.0),
                                             (1.0, 5, 1.0), (0.7, 20, 1.0), (1.0, 0, 0.6), (1.3, 0, 0.9),
                                             (0.9, 8, 0.5), (1.0, V, 1.0), (1.0, 3, 0.999)]):
        for u in (0.0, 0.013, 0.31, 0.5, 0.77, 0.9991):
            cases.append((temp, topk, topp, u))
    n = len(cases)
    # logits on a grid of 1/64 with distinct values near the top: no ties at the cut, float32-exact
    base = (torch.randperm(V, generator=g).float() / 64.0)
    base = base - base.max() + 3.0
    logits = base.repeat(n, 1)
    out = torch.empty(n, dtype=torch.int32, device=DEV)
    f = lambda xs, dt: torch.tensor(xs, dtype=dt, device=DEV)
    K.sample(logits.to(DEV), f([c[0] for c in cases], torch.float32), f([c[1] for c in cases], torch.int32),
             f([c[2] for c in cases], torch.float32), f([c[3] for c in cases], torch.float32), out)
    got = out.tolist()
    miss = []
    for i, c in enumerate(cases):
        want = plain_sample(logits[i], *c)
        if got[i] != want:
            # a float32-vs-float64 difference may move the pick only to a neighbour in the running mass
            miss.append((c, got[i], want))
    assert not miss, miss[:5]


@pytest.mark.parametrize("V", [1, 384, 2048, 5000])
def test_sample_with_ties_and_long_candidate_lists(K, V):
    """Equal logits at the cut, more of them than the kernel's list holds, cuts at and beyond the threads of a block, masses that
    round to nothing.  Whole numbers: the running masses are far from any pick's edge."""
    g = torch.Generator().manual_seed(V)
    cases = [(t, k, p, u) for t in (0.5, 2.0) for k in (0, 2, 50, 1024, 1025, V) for p in (1.0, 0.7, 0.0) for u in (0.0, 0.4001, 0.9003)]
    rows = [torch.zeros(V), torch.randint(0, 4, (V,), generator=g).float(), torch.randint(-40, 4, (V,), generator=g).float()]
    for row in rows:
        f = lambda j, dt: torch.tensor([c[j] for c in cases], dtype=dt, device=DEV)
        out = torch.empty(len(cases), dtype=torch.int32, device=DEV)
        K.sample(row.repeat(len(cases), 1).to(DEV), f(0, torch.float32), f(1, torch.int32), f(2, torch.float32), f(3, torch.float32), out)
        want = [plain_sample(row, *c) for c in cases]
        assert out.tolist() == want, [(c, a, b) for c, a, b in zip(cases, out.tolist(), want) if a != b][:5]


def test_sample_is_reproducible_and_follows_the_distribution(K):
    V, n = 50, 4000
    g = torch.Generator().manual_seed(1)
    row = torch.randn(V, generator=g) * 2
    logits = row.repeat(n, 1).to(DEV)
    u = torch.rand(n, generator=g).to(DEV)
    ones = torch.full((n,), 1.0, device=DEV)
    zeros = torch.zeros(n, dtype=torch.int32, device=DEV)
    a = torch.empty(n, dtype=torch.int32, device=DEV)
    b = torch.empty_like(a)
    K.sample(logits, ones, zeros, ones, u, a)
    K.sample(logits, ones, zeros, ones, u, b)
    assert torch.equal(a, b)
    freq = torch.bincount(a.long().cpu(), minlength=V).double() / n
    p = torch.softmax(row.double(), 0)
    assert (freq - p).abs().max() < 4 * math.sqrt(0.25 / n)


@pytest.mark.parametrize("M", [1, 3, 8, 9, 16])
@pytest.mark.parametrize("N,K_", [(48, 64), (301, 96), (2304, 2304), (1000, 5760), (6912, 2304), (17, 32)])
def test_linear_small_streams_weights_for_few_rows(K, M, N, K_):
    g = torch.Generator().manual_seed(M * N + K_)
    act = torch.randn(M, K_, generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K_, generator=g) / math.sqrt(K_)).to(torch.bfloat16)
    # (16 rows of 5760 activations leave the ring kernel no room in shared memory; the tile kernel, which keeps a
    # tile of the weights there instead, takes them)
    assert K.linear_small_supports(M, N, K_)
    out = torch.full((M, N), 9.0, device=DEV)
    K.linear_small(act.to(DEV), w.to(DEV), out)
    want = act.double() @ w.double().T
    torch.testing.assert_close(out.double().cpu(), want, rtol=1e-4, atol=1e-4)      # float32 accumulation of bf16 products


def test_linear_small_with_copies_from_every_thread_instead_of_tma_boxes():
    """The tile kernel's other way to bring its tile (what runs where the weights are not 16-byte aligned for TMA or
    a tensor map cannot be had): a process of its own, because the switch is read once."""
    import os, subprocess, sys
    code = """
import math, os, sys, torch
sys.path.insert(0, os.getcwd())
from infinicore_infer_b200 import kernels as K
for M, N, K_ in ((1, 48, 64), (8, 301, 96), (13, 1000, 5760), (16, 2304, 2304)):
    g = torch.Generator().manual_seed(M * N + K_)
    act = torch.randn(M, K_, generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K_, generator=g) / math.sqrt(K_)).to(torch.bfloat16)
    out = torch.full((M, N), 9.0, device="cuda:0")
    K.linear_small(act.cuda(), w.cuda(), out)
    torch.testing.assert_close(out.double().cpu(), act.double() @ w.double().T, rtol=1e-4, atol=1e-4)
print("equal")
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, JK_SMALL_NO_TMA="1"),
                       capture_output=True, text=True, timeout=600)
    assert p.returncode == 0 and "equal" in p.stdout, p.stderr[-2000:]


@pytest.mark.parametrize("M", [1, 8, 13])
@pytest.mark.parametrize("N,K_", [(136, 96), (5760, 2304), (50, 64)])
def test_linear_small_with_swiglu_epilogue(K, M, N, K_):
    g = torch.Generator().manual_seed(M + N + K_)
    act = torch.randn(M, K_, generator=g).to(torch.bfloat16)
    w = (torch.randn(2 * N, K_, generator=g) * 2 / math.sqrt(K_)).to(torch.bfloat16)
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    K.linear_small(act.to(DEV), w.to(DEV), out, K.EPI_SWIGLU)
    gu = act.double() @ w.double().T
    want = gu[:, :N] * torch.sigmoid(gu[:, :N]) * gu[:, N:]
    _close(out, want, torch.bfloat16, scale=2.0)


def test_linear_small_refuses_what_it_cannot_take(K):
    assert not K.linear_small_supports(17, 64, 64)
    assert not K.linear_small_supports(4, 64, 80)       # K must be a multiple of 32
    assert not K.linear_small_supports(16, 64, 1 << 20)
    with pytest.raises(K.KernelError, match="outside what the kernel takes"):
        K.linear_small(torch.zeros(4, 80, dtype=torch.bfloat16, device=DEV), torch.zeros(8, 80, dtype=torch.bfloat16, device=DEV),
                       torch.zeros(4, 8, device=DEV))


@pytest.fixture(params=["rule", "pairs"])
def pairs(K, request):
    """The tcgen05 products under their own rule for pairs of blocks, and with every product of more than
    128 rows forced onto pairs (the rule sends only products of more than one wave there)."""
    before = K.gemm_tcgen05_pairs(2 if request.param == "pairs" else 1)
    yield request.param
    K.gemm_tcgen05_pairs(1 if before < 0 else before)


TG_SHAPES = [(128, 256, 64), (128, 128, 128), (1, 8, 8), (300, 520, 200), (257, 100, 2304), (512, 6912, 2304), (2048, 2304, 5760),
             # long K and few tiles: the residual epilogue cuts K into units that add themselves (four; two with a ragged end)
             (512, 512, 8192), (300, 520, 4104)]


@pytest.mark.parametrize("M,N,K_", TG_SHAPES)
@pytest.mark.parametrize("epi", ["f32", "bf16", "residual"])
def test_gemm_tcgen05_with_store_and_residual_epilogues(K, pairs, M, N, K_, epi):
    g = torch.Generator().manual_seed(M + N + K_)
    act = torch.randn(M, K_, generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K_, generator=g) / math.sqrt(K_)).to(torch.bfloat16)
    want = act.double() @ w.double().T
    assert K.gemm_tcgen05_supports(M, N, K_)
    if epi == "f32":
        out = torch.full((M, N), 9.0, device=DEV)
        K.gemm_tcgen05(act.to(DEV), w.to(DEV), out, K.TG_F32)
        K.check_gemm_status(DEV)
        torch.testing.assert_close(out.double().cpu(), want, rtol=1e-4, atol=1e-4)
    elif epi == "bf16":
        out = torch.full((M, N), 9.0, dtype=torch.bfloat16, device=DEV)
        K.gemm_tcgen05(act.to(DEV), w.to(DEV), out, K.TG_BF16)
        K.check_gemm_status(DEV)
        _close(out, want, torch.bfloat16, scale=2.0)
    else:
        x = torch.randn(M, N, generator=g)
        out = x.to(DEV).clone()
        K.gemm_tcgen05(act.to(DEV), w.to(DEV), out, K.TG_RESIDUAL, scale=0.7)
        K.check_gemm_status(DEV)
        torch.testing.assert_close(out.double().cpu(), x.double() + 0.7 * want, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("M,K_,widths", [(1, 64, (48, 48, 32, 32, 5)), (8, 2048, (256, 256, 256, 256, 64)), (13, 320, (192, 64, 7)), (16, 96, (16, 16))])
def test_few_row_products_of_different_activations_in_one_launch(K, M, K_, widths):
    """Each column range is the product of ITS activations (not of a neighbour's) with its rows of the matrix; columns
    beside the ranges stay as they were."""
    g = torch.Generator().manual_seed(M + K_ + len(widths))
    N = sum(widths)
    assert K.linear_small_parts_supports(M, N, K_)
    acts = torch.randn(len(widths), M, K_, generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K_, generator=g) / math.sqrt(K_)).to(torch.bfloat16)
    ends = [sum(widths[:i + 1]) for i in range(len(widths))]
    wide = torch.full((M, N + 3), 9.0, device=DEV)
    K.linear_small_parts(acts.to(DEV), w.to(DEV), ends, wide[:, 1: 1 + N])
    got = wide.double().cpu()
    lo = 0
    for p, hi in enumerate(ends):
        torch.testing.assert_close(got[:, 1 + lo: 1 + hi], acts[p].double() @ w[lo:hi].double().T, rtol=1e-4, atol=1e-4)
        lo = hi
    assert bool((got[:, 0] == 9.0).all()) and bool((got[:, 1 + N:] == 9.0).all())


@pytest.mark.parametrize("M,K_,widths", [(300, 256, (256, 256, 192, 192, 32)), (200, 96, (40, 24, 7)), (1024, 512, (512, 384, 64)),
                                         (64, 256, (256, 130, 30))])
def test_products_into_column_ranges_of_wider_rows(K, pairs, M, K_, widths):
    """Several products, each from activations of its own, into neighbouring column ranges of the same float32 rows (what a
    mixer whose projections read different mixtures asks for): every range holds its product, and nothing else is written.
    Row strides that are and are not multiples of 16 bytes."""
    g = torch.Generator().manual_seed(M + K_ + sum(widths))
    for pad in (0, 1):
        ld = sum(widths) + pad
        wide = torch.full((M, ld), 9.0, device=DEV)
        off, wants = 0, []
        for n in widths:
            act = torch.randn(M, K_, generator=g).to(torch.bfloat16)
            w = (torch.randn(n, K_, generator=g) / math.sqrt(K_)).to(torch.bfloat16)
            wants.append(act.double() @ w.double().T)
            out = wide[:, off: off + n]
            if M <= 128 and K.gemm_skinny_supports(M, n, K_):
                K.gemm_skinny(act.to(DEV), w.to(DEV), out, K.TG_F32)
            else:
                K.gemm_tcgen05(act.to(DEV), w.to(DEV), out, K.TG_F32)
            K.check_gemm_status(DEV)
            off += n
        got = wide.double().cpu()
        off = 0
        for n, want in zip(widths, wants):
            torch.testing.assert_close(got[:, off: off + n], want, rtol=1e-4, atol=1e-4)
            off += n
        assert bool((got[:, off:] == 9.0).all())


@pytest.mark.parametrize("M,N,K_", [(128, 128, 64), (300, 136, 96), (2048, 5760, 2304), (77, 520, 200)])
def test_gemm_tcgen05_with_swiglu_epilogue(K, pairs, M, N, K_):
    g = torch.Generator().manual_seed(M * 3 + N)
    act = torch.randn(M, K_, generator=g).to(torch.bfloat16)
    w = (torch.randn(2 * N, K_, generator=g) * 2 / math.sqrt(K_)).to(torch.bfloat16)
    out = torch.full((M, N), 9.0, dtype=torch.bfloat16, device=DEV)
    K.gemm_tcgen05(act.to(DEV), w.to(DEV), out, K.TG_SWIGLU)
    K.check_gemm_status(DEV)
    gu = act.double() @ w.double().T
    _close(out, gu[:, :N] * torch.sigmoid(gu[:, :N]) * gu[:, N:], torch.bfloat16, scale=2.0)


@pytest.mark.parametrize("gate", ["silu", "gelu_tanh"])
@pytest.mark.parametrize("impl,M", [("small", 7), ("small", 16), ("skinny", 100), ("tiled", 300)])
def test_gated_units_are_float32_accurate_over_the_gates_range(K, impl, M, gate):
    """Gates and ups that arrive exactly (rows of W pick one element each), from where the unit vanishes on: what is stored is the unit
    rounded to bfloat16.  A rounding is 2^-8 at most, and what float32 adds before it (e^-s to one unit in the last place, a sum,
    a quotient, a product: 2.5 x 2^-23; for gelu three roundings of s as well) seldom moves one: by at most twice that over the
    spacing 2^-8, 2^-12 for silu."""
    g, N = torch.Generator().manual_seed(M), 2048
    least = -88.5 if gate == "silu" else -9.9          # beyond, e^-s is no float32 any more and the unit is 0
    z = (least + (8.0 - least) * torch.rand(M, N, generator=g)).to(torch.bfloat16)
    z[:, :3] = torch.tensor([-88.5, -88.0, -87.5] if gate == "silu" else [-9.875, -9.75, -9.5])
    up = torch.randn(M, N, generator=g).abs().add(1.0).to(torch.bfloat16)
    act, w = torch.cat([z, up], 1).to(DEV), torch.eye(2 * N, dtype=torch.bfloat16, device=DEV)
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    module, entry = {"small": ("linear_small", "jk_linear_small"), "skinny": ("gemm_tcgen05", "jk_gemm_skinny"),
                     "tiled": ("gemm_tcgen05", "jk_gemm_tcgen05")}[impl]
    code = (K.EPI_SWIGLU if impl == "small" else K.TG_SWIGLU) | ({"silu": 0, "gelu_tanh": 2}[gate] << 8)
    extra = () if impl == "small" else (K._c_float(1.0), K._ptr(K.gemm_status(act.device)))
    K._check(module, getattr(K._build.load(module), entry)(K._ptr(act), K._ptr(w), K._ptr(out), *map(K._c_int, (M, N, 2 * N, N, code)), *extra,
                                                            K._c_int(148), K._stream()))
    K.check_gemm_status(DEV)
    z, up, got = z.double(), up.double(), out.double().cpu()
    s = z if gate == "silu" else 2 * math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)
    want = z * torch.sigmoid(s) * up
    before = 2.5 * 2.0 ** -23 + (0 if gate == "silu" else 3 * 2.0 ** -24 * s.abs())
    assert ((got - want).abs() <= (2.0 ** -8 + before) * want.abs() + 2.0 ** -133).all()
    if gate == "silu":
        assert (got != want.to(torch.bfloat16).double()).double().mean() <= 2.0 ** -12


@pytest.mark.parametrize("M,N,K_", [(32, 128, 64), (17, 256, 512), (64, 520, 200), (1, 100, 72), (100, 333, 4096), (128, 1200, 2304),
                                    (9, 77, 16384)])
@pytest.mark.parametrize("epi", ["f32", "residual", "swiglu"])
def test_gemm_of_few_rows_with_the_weights_on_the_m_side(K, M, N, K_, epi):
    """jk_gemm_skinny: up to 128 rows, any width (ragged tiles of 128 features, 64 for SwiGLU), K with a tail and
    long enough to be split among blocks whose partial sums meet in the output."""
    g = torch.Generator().manual_seed(M + N + K_)
    act = torch.randn(M, K_, generator=g).to(torch.bfloat16)
    rows = 2 * N if epi == "swiglu" else N
    w = (torch.randn(rows, K_, generator=g) * (2 if epi == "swiglu" else 1) / math.sqrt(K_)).to(torch.bfloat16)
    ref = act.double() @ w.double().T
    assert K.gemm_skinny_supports(M, N, K_) and not K.gemm_skinny_supports(129, N, K_) and not K.gemm_skinny_supports(M, N, 20)
    if epi == "f32":
        out = torch.full((M, N), 9.0, device=DEV)
        K.gemm_skinny(act.to(DEV), w.to(DEV), out, K.TG_F32)
        K.check_gemm_status(DEV)
        torch.testing.assert_close(out.double().cpu(), ref, rtol=1e-4, atol=1e-4)
    elif epi == "residual":
        x = torch.randn(M, N, generator=g)
        out = x.to(DEV).clone()
        K.gemm_skinny(act.to(DEV), w.to(DEV), out, K.TG_RESIDUAL, scale=0.7)
        K.check_gemm_status(DEV)
        torch.testing.assert_close(out.double().cpu(), x.double() + 0.7 * ref, rtol=1e-4, atol=1e-4)
    else:
        out = torch.full((M, N), 9.0, dtype=torch.bfloat16, device=DEV)
        K.gemm_skinny(act.to(DEV), w.to(DEV), out, K.TG_SWIGLU)
        K.check_gemm_status(DEV)
        _close(out, ref[:, :N] * torch.sigmoid(ref[:, :N]) * ref[:, N:], torch.bfloat16, scale=2.0)
    # an output with padded rows
    if epi == "f32":
        wide = torch.full((M, N + 5), 9.0, device=DEV)
        K.gemm_skinny(act.to(DEV), w.to(DEV), wide[:, :N], K.TG_F32)
        torch.testing.assert_close(wide[:, :N].double().cpu(), ref, rtol=1e-4, atol=1e-4)
        assert float(wide[:, N:].min()) == 9.0


def test_gemm_tcgen05_refuses_rows_that_tma_cannot_address(K):
    assert not K.gemm_tcgen05_supports(4, 4, 20)
    with pytest.raises(K.KernelError, match="multiple of 8"):
        K.gemm_tcgen05(torch.zeros(4, 20, dtype=torch.bfloat16, device=DEV), torch.zeros(4, 20, dtype=torch.bfloat16, device=DEV),
                       torch.zeros(4, 4, device=DEV))

