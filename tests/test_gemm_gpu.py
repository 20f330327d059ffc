"""tcgen05 GEMM against a plain PyTorch fp32 reference of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


PAIR = 512        # ab_gemm_route on CTA pairs, plus the kind of the epilogue (EpiKind in csrc/gemm_core.cuh)
ANY, BF16, GELU, GELU_GRAD, MUL, RESID, ACCUM, DOT = range(8)


@pytest.fixture
def routes(monkeypatch):
    """What each GEMM of a test was dispatched to: 32, 64, 128 or 256 (tile columns of the single-CTA kernel), or
    PAIR + kind."""
    from allie_b200.ops import _lib

    lib, seen = _lib.cuda(), []

    class Spy:
        def __getattr__(self, name):
            return getattr(lib, name)

        def ab_gemm_bf16(self, *args):
            seen.append(lib.ab_gemm_route(*args))
            return lib.ab_gemm_bf16(*args)

    monkeypatch.setattr(_lib, "_cuda_lib", Spy())
    return seen


def _ref(a, b, a_mn, b_mn):
    A = a.float().t() if a_mn else a.float()
    B = b.float() if b_mn else b.float().t()
    return A @ B


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 320), (384, 768, 1024), (200, 264, 136),
                                   (1000, 128, 512), (64, 64, 64),
                                   # CTA pairs where A is MN-major, else one wave of smaller tiles
                                   (1000, 264, 136), (640, 768, 320), (2304, 1024, 192),
                                   (512, 256, 64), (768, 512, 40),       # one K block; ragged K
                                   # beyond one wave: CTA pairs in every layout, with ragged edges
                                   (4744, 808, 136), (2440, 1032, 40)])
def test_gemm_layouts(routes, a_mn, b_mn, M, N, K):
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    torch.manual_seed(0)
    dev = "cuda"
    a = torch.randn((K, M) if a_mn else (M, K), device=dev).bfloat16()
    b = torch.randn((K, N) if b_mn else (N, K), device=dev).bfloat16()
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32)
    torch.cuda.synchronize()
    _lib.check_status()
    assert (routes == [PAIR + ANY]) == (M >= 2440 or (M >= 512 and N >= 256 and a_mn))
    ref = _ref(a, b, a_mn, b_mn)
    err = (out - ref).abs().max().item()
    assert err < 2e-2 * (K ** 0.5), (err, M, N, K)
    assert torch.allclose(out, ref, rtol=1e-3, atol=1e-2 * (K ** 0.5) * 0.1)


def test_gemm_epilogues():
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    torch.manual_seed(1)
    dev = "cuda"
    M, N, K = 512, 768, 256
    a = torch.randn(M, K, device=dev).bfloat16()
    w = (torch.randn(K, N, device=dev) * 0.05).bfloat16()
    bias = torch.randn(N, device=dev)
    ref = a.float() @ w.float() + bias
    # bias, bf16 out
    out = gemm(a, w, b_mn=True, bias=bias)
    assert torch.allclose(out.float(), ref, rtol=2e-2, atol=2e-2)
    # bias + gelu, preact saved
    pre = torch.empty(M, N, device=dev, dtype=torch.bfloat16)
    out = gemm(a, w, b_mn=True, bias=bias, act=1, aux=pre)
    assert torch.allclose(pre.float(), ref, rtol=2e-2, atol=2e-2)
    g = torch.nn.functional.gelu(ref, approximate="tanh")
    assert torch.allclose(out.float(), g, rtol=2e-2, atol=2e-2)
    # gelu backward multiply
    dy = torch.randn(M, K, device=dev).bfloat16()
    wt = (torch.randn(N, K, device=dev) * 0.05).bfloat16()  # dX[M,N] = dy[M,K] @ wt[N,K]^T
    o2 = gemm(dy, wt, act=2, aux=pre)
    x = pre.float().requires_grad_(True)
    torch.nn.functional.gelu(x, approximate="tanh").backward(dy.float() @ wt.float().t())
    assert torch.allclose(o2.float(), x.grad, rtol=3e-2, atol=3e-2)
    # residual (no dropout), fp32 out, in place
    resid = torch.randn(M, N, device=dev)
    r0 = resid.clone()
    gemm(a, w, b_mn=True, bias=bias, resid=resid, out=resid)
    assert torch.allclose(resid, r0 + ref, rtol=1e-2, atol=2e-2)
    # residual with dropout: kept fraction and scaling
    resid = torch.zeros(M, N, device=dev)
    gemm(a, w, b_mn=True, bias=bias, resid=resid, out=resid, drop_p=0.25, drop_seed=123, drop_stream=7)
    kept = resid != 0
    frac = kept.float().mean().item()
    assert abs(frac - 0.75) < 0.01, frac
    assert torch.allclose(resid[kept], (ref / 0.75)[kept], rtol=1e-2, atol=3e-2)
    # accumulate with split-K (wgrad shape): dW[K,N] += a^T @ dyy
    dyy = torch.randn(M, N, device=dev).bfloat16()
    dw = torch.ones(K, N, device=dev)
    gemm(a, dyy, a_mn=True, b_mn=True, out=dw, accumulate=True, k_splits=4)
    refw = 1.0 + a.float().t() @ dyy.float()
    assert torch.allclose(dw, refw, rtol=1e-3, atol=5e-2)
    torch.cuda.synchronize()
    _lib.check_status()


def test_gemm_big_and_timing():
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    dev = "cuda"
    torch.manual_seed(2)
    M, N, K = 16384, 4096, 1024
    a = torch.randn(M, K, device=dev).bfloat16()
    w = (torch.randn(K, N, device=dev) * 0.03).bfloat16()
    out = gemm(a, w, b_mn=True)
    ref = (a @ w).float()
    assert torch.allclose(out.float(), ref, rtol=3e-2, atol=3e-2)
    _lib.check_status()


def test_gemm_pair_split_k_accumulate():
    """Weight-gradient shape on the CTA-pair kernel: MN-major operands, split-K, TMA reduce-add."""
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    torch.manual_seed(3)
    dev = "cuda"
    T, I, O = 4096, 1024, 768
    x = torch.randn(T, I, device=dev).bfloat16()
    dy = torch.randn(T, O, device=dev).bfloat16()
    dw = torch.full((I, O), 2.0, device=dev)
    gemm(x, dy, a_mn=True, b_mn=True, out=dw, accumulate=True, k_splits=4)
    ref = 2.0 + x.float().t() @ dy.float()
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.allclose(dw, ref, rtol=1e-3, atol=0.2)


def test_gemm_skinny_residual_update_in_place():
    """Decode-sized x += a @ w + bias: few output tiles, long K (taken by the split-K route)."""
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    torch.manual_seed(4)
    dev = "cuda"
    for M, N, K in ((256, 1024, 4096), (192, 1024, 1024), (40, 768, 2048)):
        a = torch.randn(M, K, device=dev).bfloat16()
        w = (torch.randn(K, N, device=dev) * 0.03).bfloat16()
        bias = torch.randn(N, device=dev)
        x = torch.randn(M, N, device=dev)
        want = x + a.float() @ w.float() + bias
        gemm(a, w, b_mn=True, bias=bias, resid=x, out=x)
        torch.cuda.synchronize()
        _lib.check_status()
        assert torch.allclose(x, want, rtol=1e-3, atol=3e-2), (M, N, K, (x - want).abs().max().item())


@pytest.mark.parametrize("M,N,K,route", [(1000, 328, 192, 64), (2048, 1024, 256, 128), (640, 72, 128, 128),
                                         (4744, 808, 72, PAIR + ANY), (20000, 520, 128, PAIR + ANY)])
def test_gemm_gelu_backward_epilogue_ragged(routes, M, N, K, route):
    """out = (dy @ w^T) * gelu'(pre) on shapes with ragged row / column tiles (the CTA-pair kernel
    fetches the pre-activation tiles by TMA one tile ahead)."""
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    torch.manual_seed(5)
    dev = "cuda"
    dy = torch.randn(M, K, device=dev).bfloat16()
    wt = (torch.randn(N, K, device=dev) * 0.05).bfloat16()
    pre = torch.randn(M, N, device=dev).bfloat16()
    out = gemm(dy, wt, act=2, aux=pre)
    torch.cuda.synchronize()
    _lib.check_status()
    assert routes == [route]
    x = pre.float().requires_grad_(True)
    torch.nn.functional.gelu(x, approximate="tanh").backward(dy.float() @ wt.float().t())
    assert torch.allclose(out.float(), x.grad, rtol=3e-2, atol=3e-2), (out.float() - x.grad).abs().max().item()


def test_gemm_gelu_derivative_kept_in_aux():
    """act=1 / act=2 with aux_grad: the forward launch stores GELU'(pre-activation), the backward
    launch multiplies by it; same results as the pre-activation form."""
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    torch.manual_seed(6)
    dev = "cuda"
    M, N, K = 1000, 1152, 256
    x = torch.randn(M, K, device=dev).bfloat16()
    w = (torch.randn(K, N, device=dev) * 0.08).bfloat16()
    bias = torch.randn(N, device=dev)
    act = torch.empty(M, N, device=dev, dtype=torch.bfloat16)
    dact = torch.empty_like(act)
    gemm(x, w, b_mn=True, bias=bias, act=1, aux=dact, out=act, aux_grad=True)
    dy = torch.randn(M, 512, device=dev).bfloat16()
    w2 = (torch.randn(N, 512, device=dev) * 0.05).bfloat16()
    dpre = gemm(dy, w2, act=2, aux=dact, aux_grad=True)
    torch.cuda.synchronize()
    _lib.check_status()
    pre = (x.float() @ w.float() + bias).requires_grad_(True)
    ref = torch.nn.functional.gelu(pre, approximate="tanh")
    (want_d,) = torch.autograd.grad(ref.sum(), pre)
    assert torch.allclose(act.float(), ref.detach(), rtol=2e-2, atol=2e-2)
    assert torch.allclose(dact.float(), want_d, rtol=1e-2, atol=1e-2), (dact.float() - want_d).abs().max().item()
    want = (dy.float() @ w2.float().t()) * want_d
    assert torch.allclose(dpre.float(), want, rtol=3e-2, atol=3e-2), (dpre.float() - want).abs().max().item()


@pytest.mark.parametrize("drop_p", [0.0, 0.1])
@pytest.mark.parametrize("M,N,K,route", [
    (512, 256, 64, 32), (520, 264, 72, 32), (1100, 800, 256, 64),        # one wave of smaller tiles
    (2560, 1024, 64, PAIR + RESID),      # one tile per pair, both column groups of every warp
    (2440, 1032, 72, PAIR + RESID),      # rows past a tile, eight columns in the last tile
    (4744, 800, 256, PAIR + RESID),      # last column tile ends behind a warp's first group
    (4744, 808, 72, PAIR + RESID),       # and inside its second
    (20000, 512, 128, PAIR + RESID)])    # several units per pair: tiles fetched one unit ahead
def test_gemm_pair_residual_tiles(routes, M, N, K, route, drop_p):
    """A fp32 residual.  On CTA pairs its tiles travel by TMA through the output staging tile."""
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    torch.manual_seed(4)
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(K, N, device="cuda") * 0.05).bfloat16()
    bias, resid = torch.randn(N, device="cuda"), torch.randn(M, N, device="cuda")
    kw = dict(b_mn=True, bias=bias, drop_p=drop_p, drop_seed=11, drop_stream=3)
    out = torch.full((M, N), float("nan"), device="cuda")
    gemm(a, w, out=out, resid=resid, **kw)
    masked = gemm(a, w, out=torch.empty_like(out), resid=torch.zeros_like(resid), **kw)
    inplace = resid.clone()
    gemm(a, w, out=inplace, resid=inplace, **kw)
    torch.cuda.synchronize()
    _lib.check_status()
    assert routes == [route] * 3
    # the same accumulators and mask: only the last addition of the residual rounds differently (half
    # an ulp of values below 16)
    assert torch.equal(out, inplace)
    assert torch.allclose(out, masked + resid, rtol=0, atol=2e-6)
    if drop_p == 0:
        ref = a.float() @ w.float() + bias + resid
        assert torch.allclose(out, ref, rtol=1e-4, atol=1e-4 * K ** 0.5)


@pytest.mark.parametrize("M,N,K,pair", [(512, 256, 64, False), (520, 264, 72, False), (1100, 800, 256, False),
                                        (2440, 1032, 64, True), (4744, 800, 72, True), (20000, 512, 128, True),
                                        (4744, 1032, 136, True), (5000, 808, 72, True)])
def test_gemm_pair_specialised_epilogues(routes, M, N, K, pair):
    """The specialised drains of the CTA-pair kernel at tile edges (rows and columns past a tile, a last
    column tile that ends inside a warp's columns, several units per pair), and the same epilogues where one
    wave of smaller tiles takes them."""
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    torch.manual_seed(5)
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(K, N, device="cuda") * K ** -0.5).bfloat16()
    bias = torch.randn(N, device="cuda")
    ref = a.float() @ w.float() + bias
    # one bf16 rounding of a value of known size (2^-9 of it), plus the rounding of the fp32 sums and
    # of tanh.approx (2^-11)
    close = lambda x, y: torch.allclose(x.float(), y, rtol=2 ** -8, atol=2 ** -9)
    assert close(gemm(a, w, b_mn=True, bias=bias), ref)
    assert close(gemm(a, w, b_mn=True), ref - bias)
    gelu = torch.nn.functional.gelu(ref, approximate="tanh")
    assert close(gemm(a, w, b_mn=True, bias=bias, act=3), gelu)
    aux = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    assert close(gemm(a, w, b_mn=True, bias=bias, act=1, aux=aux, aux_grad=True), gelu)
    x = ref.clone().requires_grad_(True)
    torch.nn.functional.gelu(x, approximate="tanh").sum().backward()
    assert close(aux, x.grad)
    wt = w.t().contiguous()
    assert close(gemm(a, wt, act=2, aux=aux, aux_grad=True), (ref - bias) * aux.float())
    if pair:
        assert routes == [PAIR + kind for kind in (BF16, BF16, GELU, GELU_GRAD, MUL)]
    else:
        assert max(routes) < PAIR
    dy = torch.randn(M, N, device="cuda").bfloat16()
    dw = torch.full((K, N), 3.0, device="cuda")
    for splits in (1, 3):
        gemm(a, dy, a_mn=True, b_mn=True, out=dw, accumulate=True, k_splits=splits)
    # The tensor core adds 16 products at a time and cuts the fp32 sum off (no rounding to nearest): M / 16
    # additions lose up to 2^-23 of a partial sum, which stays below 6 sqrt(M) for these inputs, all with
    # the same sign; two launches.
    bound = 2 * (M / 16) * 2 ** -23 * 6 * M ** 0.5 + 1e-5
    assert ((dw.double() - 3.0 - 2 * (a.double().t() @ dy.double())).abs() <= bound).all()
    torch.cuda.synchronize()
    _lib.check_status()


@pytest.mark.parametrize("T", [650, 4096])
@pytest.mark.parametrize("I,O", [(1000, 808), (512, 256)])
def test_gemm_pair_accumulate_drain(routes, I, O, T):
    """Weight gradients on CTA pairs, whole and split contractions, rows and columns past a tile."""
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    torch.manual_seed(8)
    x, dy = torch.randn(T, I, device="cuda").bfloat16(), torch.randn(T, O, device="cuda").bfloat16()
    dw = torch.full((I, O), 3.0, device="cuda")
    for splits in (1, 3):
        gemm(x, dy, a_mn=True, b_mn=True, out=dw, accumulate=True, k_splits=splits)
    torch.cuda.synchronize()
    _lib.check_status()
    assert routes == [PAIR + ACCUM] * 2
    bound = 2 * (T / 16) * 2 ** -23 * 6 * T ** 0.5 + 1e-5      # as above
    assert ((dw.double() - 3.0 - 2 * (x.double().t() @ dy.double())).abs() <= bound).all()


def test_gemm_pair_general_drain(routes):
    """What no specialised drain of the CTA-pair kernel takes: a scaled product, a kept pre-activation, a
    residual with weights read K-major."""
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    torch.manual_seed(9)
    M, N, K = 4744, 808, 72
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(K, N, device="cuda") * K ** -0.5).bfloat16()
    bias, resid = torch.randn(N, device="cuda"), torch.randn(M, N, device="cuda")
    ref = a.float() @ w.float()
    close = lambda x, y: torch.allclose(x.float(), y, rtol=2 ** -8, atol=2 ** -9)     # as above
    assert close(gemm(a, w, b_mn=True, alpha=0.5), 0.5 * ref)
    pre = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    assert close(gemm(a, w, b_mn=True, bias=bias, act=1, aux=pre), torch.nn.functional.gelu(ref + bias, approximate="tanh"))
    assert close(pre, ref + bias)
    out = gemm(a, w.t().contiguous(), bias=bias, resid=resid, out=torch.empty_like(resid))
    assert torch.allclose(out, ref + bias + resid, rtol=1e-4, atol=1e-4 * K ** 0.5)
    torch.cuda.synchronize()
    _lib.check_status()
    assert routes == [PAIR + ANY] * 3


@pytest.mark.parametrize("M,N,K", [(512, 256, 64), (520, 264, 72), (1100, 832, 256), (20000, 512, 128), (96, 256, 128)])
def test_gemm_column_sums_and_head_products(routes, M, N, K):
    """The column sums that the derivative epilogue adds (and the pass that stands in below 512 rows) at
    tile edges, and the per-head products with a second tensor.  Both are fp32 sums of the bf16 values
    that were stored: any order is within terms * 2^-23 * sum|terms|."""
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    torch.manual_seed(6)
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16()
    aux = torch.randn(M, N, device="cuda").bfloat16()
    sums = torch.full((N,), 0.25, device="cuda")
    out = gemm(a, w, act=2, aux=aux, aux_grad=True, colsum=sums)
    plain = gemm(a, w, act=2, aux=aux, aux_grad=True)
    torch.cuda.synchronize()
    _lib.check_status()
    assert routes[0] == (PAIR + MUL if M >= 512 else 128)
    assert torch.equal(out, plain)
    terms = out.double()
    assert ((sums.double() - 0.25 - terms.sum(0)).abs() <= 1e-6 + M * 2.0 ** -23 * (terms.abs().sum(0) + 0.25)).all()
    if N % 64 == 0:
        T = 4 if M % 4 == 0 else 1
        dot = torch.full((M // T, N // 64, T), float("nan"), device="cuda")
        out = gemm(a, w, act=4, aux=aux, dot=(dot, T))
        torch.cuda.synchronize()
        _lib.check_status()
        assert routes[-1] == (PAIR + DOT if M >= 512 else 128)
        assert torch.equal(out, gemm(a, w))
        prod = (out.double() * aux.double()).view(M // T, T, N // 64, 64).permute(0, 2, 1, 3)
        assert ((dot.double() - prod.sum(-1)).abs() <= 1e-6 + 64 * 2.0 ** -23 * prod.abs().sum(-1)).all()


@pytest.mark.parametrize("M,N,K,route", [(4744, 808, 72, PAIR + RESID), (512, 256, 64, 32)])
def test_gemm_residual_drops_non_finite_values(routes, M, N, K, route):
    """A dropped element adds nothing to the residual, whatever it was: Inf and NaN of one row of the product
    stay out of its dropped columns."""
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    torch.manual_seed(7)
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = torch.rand(K, N, device="cuda").add_(1.0).bfloat16()
    resid = torch.randn(M, N, device="cuda")
    kw = dict(b_mn=True, drop_p=0.25, drop_seed=5, drop_stream=2)
    kept = gemm(torch.ones_like(a), w, out=torch.empty_like(resid), resid=torch.zeros_like(resid), **kw) != 0
    a[3] = float("inf")
    a[M - 1] = float("nan")
    out = gemm(a, w, out=torch.empty_like(resid), resid=resid, **kw)
    torch.cuda.synchronize()
    _lib.check_status()
    assert routes == [route] * 2
    assert 0.7 < float(kept.float().mean()) < 0.8
    assert torch.equal(out[~kept], resid[~kept])
    assert torch.isinf(out[3][kept[3]]).all() and torch.isnan(out[M - 1][kept[M - 1]]).all()
    keep = torch.ones(M, dtype=torch.bool, device="cuda")
    keep[[3, M - 1]] = False
    assert out[keep].isfinite().all()


@pytest.mark.parametrize("M", [1, 90, 256])
@pytest.mark.parametrize("nbytes", [0, 16, 40000, 16 * 100003])
def test_gemm_asks_for_the_next_weights(M, nbytes):
    """`then` changes no result, whatever its size (less than a CTA's share, no multiple of a copy)."""
    from allie_b200.ops.gemm import gemm

    N, K = 1024, 256
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(K, N, device="cuda") * 0.05).bfloat16()
    nxt = torch.zeros(max(8, nbytes // 2), device="cuda", dtype=torch.bfloat16)[:nbytes // 2]
    want = gemm(a, w, b_mn=True)
    got = gemm(a, w, b_mn=True, dependent=True, then=nxt)
    torch.cuda.synchronize()
    assert torch.equal(want, got)


@pytest.mark.parametrize("M,N,K,shares", [
    (1280, 3840, 16384, True),      # 75 tiles: a round of whole ones and one cut into 32 parts
    (1280, 1280, 16384, True),      # 25: two parts each, 24 pairs take what is left
    (1280, 5120, 4104, True),       # 100: a round, 26 in two parts and the rest; a last step of 8
    (1000, 1096, 8200, False), (2048, 1024, 12000, True), (520, 264, 40000, True), (1024, 4096, 8192, False),
    (1024, 4096, 32768, True),
])
def test_weight_gradients_in_equal_shares(routes, M, N, K, shares):
    """Shares of the contraction that are no equal parts, edges of tiles, and sums handed over every few steps.

    Every element: no accumulator sums up more than 32 steps of 64, of 16 products each addition, which are cut off at
    2^-23 of a partial sum below 6 sqrt(2048); each of the K / 2048 parts adds one such error at most, the fp32
    additions of the parts 2^-24 of 6 sqrt(K) each.  That would hold for longer chains, too; their error in the
    2-norm grows with the steps an accumulator sums up, 6.6e-8 each on the GPU (16 steps 9.9e-7, 32 2.1e-6, 64
    4.4e-6, whole contractions here 1.2e-6 to 3.1e-5), so 1e-7 for each of the steps that there should be
    tells a chain that was not cut, in all of these but the last but one, whose parts are shorter anyway."""
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm, num_sms, pick_k_splits

    torch.manual_seed(9)
    a, dy = torch.randn(K, M, device="cuda").bfloat16(), torch.randn(K, N, device="cuda").bfloat16()
    dw = torch.full((M, N), 3.0, device="cuda")
    gemm(a, dy, a_mn=True, b_mn=True, out=dw, accumulate=True)
    torch.cuda.synchronize()
    _lib.check_status()
    assert routes == [PAIR + ACCUM]
    steps = -(-K // 64)
    tiles = -(-M // 256) * -(-N // 256)
    assert (_lib.cuda().ab_gemm_even_units(tiles, steps, num_sms() // 2, None, 0) > 0) == shares
    want = a.double().t() @ dy.double()
    off = dw.double() - 3.0 - want
    parts = K / 2048 + 1
    bound = parts * (128 * 2 ** -23 * 6 * 2048 ** 0.5 + 2 ** -24 * 6 * K ** 0.5) + 1e-5
    assert (off.abs() <= bound).all()
    assert float(off.norm() / want.norm()) <= 1e-7 * min(32, -(-steps // pick_k_splits(M, N, K)))


@pytest.mark.parametrize("M", [1, 20, 64, 65, 90, 128, 200])
@pytest.mark.parametrize("N,K", [(1024, 1024), (1024, 72), (264, 520), (40, 4096), (1048, 200), (4096, 136), (4736, 64),
                                 (4744, 64)])
@pytest.mark.parametrize("b_mn", [True, False])
def test_gemm_small_tiles(routes, M, N, K, b_mn):
    """Tiles of 64 rows x 32 columns, wherever they are at most as many as the SMs: edges, a contraction that ends inside
    a stage, all epilogues; and the same bits as the tiles give that a larger batch of the same rows takes (contractions
    are not split)."""
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm, num_sms

    few = N >= 1024 and -(-M // 64) * -(-N // 32) <= num_sms()
    torch.manual_seed(10)
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(K, N, device="cuda") / K ** 0.5).bfloat16()
    b = w if b_mn else w.t().contiguous()
    bias, resid = torch.randn(N, device="cuda"), torch.randn(M, N, device="cuda")
    ref = a.double() @ w.double() + bias
    close = lambda x, y: torch.allclose(x.double(), y, rtol=1e-2, atol=1e-2)      # bf16 results: 2^-9 each
    plain = gemm(a, b, b_mn=b_mn, bias=bias)
    assert close(plain, ref)
    assert close(gemm(a, b, b_mn=b_mn, bias=bias, act=3), torch.nn.functional.gelu(ref, approximate="tanh"))
    aux = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    assert close(gemm(a, b, b_mn=b_mn, bias=bias, act=1, aux=aux), torch.nn.functional.gelu(ref, approximate="tanh"))
    assert close(aux, ref)
    out = torch.full((M + 1, N), 7.0, device="cuda")
    gemm(a, b, b_mn=b_mn, bias=bias, resid=resid, out=out[:M])
    assert ((out[:M].double() - ref - resid).abs() <= 1e-4).all() and (out[M] == 7.0).all()
    dropped = gemm(a, b, b_mn=b_mn, bias=bias, resid=resid, out_dtype=torch.float32, drop_p=0.25, drop_seed=5, drop_stream=3)
    kept = dropped != resid
    assert M * N < 1000 or abs(kept.double().mean() - 0.75) < 0.03
    assert ((dropped - resid).double()[kept] - (ref / 0.75)[kept]).abs().max() < 1e-3
    assert routes == [32 if few else 64 if N >= 1024 else 128] * 5
    more = torch.cat([a, torch.randn(3000, K, device="cuda").bfloat16()])
    assert torch.equal(gemm(more, b, b_mn=b_mn, bias=bias)[:M], plain)
    _lib.check_status()
