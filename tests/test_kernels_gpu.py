"""Non-GEMM sm_100a kernels against plain PyTorch fp32 references of the same ops."""
import ctypes

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _done():
    from allie_b200.ops import _lib

    torch.cuda.synchronize()
    _lib.check_status()


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("M,d", [(300, 256), (1024, 1024), (77, 2048)])
def test_layernorm_forward(M, d, rms):
    from allie_b200.ops import kernels as K

    torch.manual_seed(0)
    x = torch.randn(M, d, device=DEV) * 2 + 0.3
    g = torch.randn(d, device=DEV)
    b = torch.randn(d, device=DEV)
    y = torch.empty(M, d, device=DEV, dtype=torch.bfloat16)
    mean = torch.empty(M, device=DEV)
    rstd = torch.empty(M, device=DEV)
    K.layernorm_fwd(x, g, None if rms else b, y, mean, rstd, 1e-5, rms=rms)     # RMSNorm has no shift
    _done()
    if rms:
        ref = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5) * g
    else:
        ref = F.layer_norm(x, (d,), g, b, 1e-5)
        assert torch.allclose(mean, x.mean(-1), atol=1e-5)
    assert torch.allclose(y.float(), ref, rtol=1e-2, atol=2e-2)


@pytest.mark.parametrize("M,d,rms", [(520, 1024, False), (520, 1024, True), (77, 256, False), (131, 1280, False),
                                     (66, 2048, True), (3, 128, False)])
def test_layernorm_backward_with_residual_and_params(M, d, rms):
    from allie_b200.ops import kernels as K

    torch.manual_seed(1)
    x = (torch.randn(M, d, device=DEV) * 1.5).requires_grad_(True)
    g = torch.randn(d, device=DEV, requires_grad=True)
    b = torch.randn(d, device=DEV, requires_grad=True)
    dy = torch.randn(M, d, device=DEV).bfloat16()
    dres = torch.randn(M, d, device=DEV)
    if rms:
        yref = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5) * g
    else:
        yref = F.layer_norm(x, (d,), g, b, 1e-5)
    yref.backward(dy.float())
    y = torch.empty(M, d, device=DEV, dtype=torch.bfloat16)
    mean = torch.empty(M, device=DEV)
    rstd = torch.empty(M, device=DEV)
    K.layernorm_fwd(x.detach(), g.detach(), None if rms else b.detach(), y, mean, rstd, 1e-5, rms=rms)
    dx = torch.empty(M, d, device=DEV)
    dbranch = torch.empty(M, d, device=DEV, dtype=torch.bfloat16)
    dgamma = torch.zeros(d, device=DEV)
    dbeta = torch.zeros(d, device=DEV)
    K.layernorm_bwd(dy, x.detach(), mean, rstd, g.detach(), dres, dx, dbranch, dgamma,
                    None if rms else dbeta, rms=rms)
    _done()
    ref_dx = x.grad + dres
    assert torch.allclose(dx, ref_dx, rtol=1e-3, atol=2e-3)
    assert torch.allclose(dbranch.float(), ref_dx, rtol=1e-2, atol=3e-2)     # no dropout: a bf16 copy
    assert torch.allclose(dgamma, g.grad, rtol=1e-3, atol=5e-2)
    if not rms:
        assert torch.allclose(dbeta, b.grad, rtol=1e-3, atol=5e-2)


def test_layernorm_backward_dropout_copy_is_masked_and_scaled():
    from allie_b200.ops import kernels as K

    torch.manual_seed(2)
    M, d = 256, 1024
    x = torch.randn(M, d, device=DEV)
    g = torch.ones(d, device=DEV)
    b = torch.zeros(d, device=DEV)
    y = torch.empty(M, d, device=DEV, dtype=torch.bfloat16)
    mean = torch.empty(M, device=DEV)
    rstd = torch.empty(M, device=DEV)
    K.layernorm_fwd(x, g, b, y, mean, rstd, 1e-5)
    dy = torch.randn(M, d, device=DEV).bfloat16()
    dres = torch.randn(M, d, device=DEV) + 3.0     # keeps dx away from zero
    dx = torch.empty(M, d, device=DEV)
    dbranch = torch.empty(M, d, device=DEV, dtype=torch.bfloat16)
    dgamma = torch.zeros(d, device=DEV)
    dbeta = torch.zeros(d, device=DEV)
    dbias = torch.full((d,), 0.5, device=DEV)
    K.layernorm_bwd(dy, x, mean, rstd, g, dres, dx, dbranch, dgamma, dbeta, drop_seed=11, drop_stream=5,
                    drop_p=0.25, dbias=dbias)
    _done()
    # fused bias gradient of the projection below: column sums of the masked copy, accumulated
    assert torch.allclose(dbias, 0.5 + dbranch.float().sum(0), rtol=1e-2, atol=0.5)
    kept = dbranch != 0
    frac = kept.float().mean().item()
    assert abs(frac - 0.75) < 0.01, frac
    assert torch.allclose(dbranch.float()[kept], (dx / 0.75)[kept], rtol=1e-2, atol=3e-2)


@pytest.mark.parametrize("M,d,params", [(37, 1280, True), (21, 1024, True), (19, 2048, True), (37, 1280, False)])
def test_layernorm_backward_dropout_mask_is_the_element_indexed_one(M, d, params):
    """The masked copy keeps exactly the elements that the generator keeps for element index
    row * d + column (the mask the projection's forward epilogue applied), in both backward kernels
    (with and without parameter gradients) and at widths where a thread owns two column groups."""
    import ctypes

    import numpy as np

    from allie_b200.ops import _lib
    from allie_b200.ops import kernels as K

    torch.manual_seed(4)
    x = torch.randn(M, d, device=DEV)
    g = torch.ones(d, device=DEV)
    y = torch.empty(M, d, device=DEV, dtype=torch.bfloat16)
    mean = torch.empty(M, device=DEV)
    rstd = torch.empty(M, device=DEV)
    K.layernorm_fwd(x, g, torch.zeros(d, device=DEV), y, mean, rstd, 1e-5)
    dy = torch.randn(M, d, device=DEV).bfloat16()
    dres = torch.randn(M, d, device=DEV) + 5.0     # keeps dx away from zero
    dx = torch.empty(M, d, device=DEV)
    dbranch = torch.empty(M, d, device=DEV, dtype=torch.bfloat16)
    dgamma = torch.zeros(d, device=DEV) if params else None
    dbeta = torch.zeros(d, device=DEV) if params else None
    seed, stream, p = 1234567, 9, 0.3
    K.layernorm_bwd(dy, x, mean, rstd, g, dres, dx, dbranch, dgamma, dbeta, drop_seed=seed, drop_stream=stream,
                    drop_p=p)
    _done()
    host = np.empty(M * d, dtype=np.uint8)
    assert _lib.cuda().ab_dropout_mask_host(ctypes.c_ulonglong(seed), ctypes.c_uint(stream), ctypes.c_longlong(M * d),
                                            ctypes.c_uint(_lib.dropout_thr16(p)),
                                            host.ctypes.data_as(ctypes.c_void_p)) == 0
    want = torch.from_numpy(host).view(M, d).bool()
    assert torch.equal((dbranch != 0).cpu(), want)


@pytest.mark.parametrize("M,d", [(1, 128), (9, 256), (1001, 256), (13, 384), (6, 640), (2999, 768), (1201, 2048)])
def test_layernorm_backward_column_sums_and_mask_at_row_group_edges(M, d):
    """Widths that put several row groups into a block (d < 1024), leave lanes without columns
    (d = 128, 640) or use the widest group, with row counts that end inside a group's pair of rows.
    Sums of M fp32 terms: |error| <= M * 2^-24 * sum|terms| bounds any order; sqrt(M) of it is seen."""
    from allie_b200.ops import kernels as K

    torch.manual_seed(8)
    x = torch.randn(M, d, device=DEV)
    g = torch.randn(d, device=DEV)
    mean, rstd = x.mean(-1), (x.var(-1, unbiased=False) + 1e-5).rsqrt()
    dy = torch.randn(M, d, device=DEV).bfloat16()
    dres = torch.randn(M, d, device=DEV) + 4.0
    dx = torch.empty(M, d, device=DEV)
    dbranch = torch.empty(M, d, device=DEV, dtype=torch.bfloat16)
    sums = torch.zeros(3, d, device=DEV)
    K.layernorm_bwd(dy, x, mean, rstd, g, dres, dx, dbranch, sums[0], sums[1], dbias=sums[2], drop_seed=3,
                    drop_stream=2, drop_p=0.2)
    _done()
    xh = (x.double() - mean.double()[:, None]) * rstd.double()[:, None]
    gy = dy.double() * g.double()
    ref = (gy - gy.mean(-1, keepdim=True) - xh * (gy * xh).mean(-1, keepdim=True)) * rstd.double()[:, None] + dres.double()
    assert torch.allclose(dx.double(), ref, rtol=1e-5, atol=2e-5)
    keep = dbranch != 0
    scale = 65536.0 / (65536 - _thr16(0.2))
    assert torch.allclose(dbranch.float()[keep], dx[keep] * scale, rtol=2 ** -8, atol=1e-6)
    masked = torch.where(keep, dx.double() * scale, torch.zeros_like(ref))
    for got, terms in ((sums[0], dy.double() * xh), (sums[1], dy.double()), (sums[2], masked)):
        assert ((got.double() - terms.sum(0)).abs() <= 1e-6 + M * 2.0 ** -22 * terms.abs().sum(0)).all()


def test_layernorm_backward_without_bulk_copies():
    """A gradient at 8 bytes (bulk copies need 16) takes the form with plain loads: the same values."""
    from allie_b200.ops import kernels as K

    torch.manual_seed(9)
    M, d = 301, 768
    x, g, dres = torch.randn(M, d, device=DEV), torch.randn(d, device=DEV), torch.randn(M, d, device=DEV)
    mean, rstd = x.mean(-1), (x.var(-1, unbiased=False) + 1e-5).rsqrt()
    room = torch.randn(M * d + 4, device=DEV).bfloat16()
    results = []
    for dy in (room[4:].view(M, d), room[4:].view(M, d).clone()):
        dx, db = torch.empty(M, d, device=DEV), torch.empty(M, d, device=DEV, dtype=torch.bfloat16)
        K.layernorm_bwd(dy, x, mean, rstd, g, dres, dx, db, torch.zeros(d, device=DEV), torch.zeros(d, device=DEV))
        _done()
        results.append((dx, db))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


def _thr16(p):
    from allie_b200.ops import _lib

    return _lib.dropout_thr16(p)


def test_cross_entropy_loss_and_gradient():
    from allie_b200.ops import kernels as K

    torch.manual_seed(3)
    M, V = 700, 2048
    logits = (torch.randn(M, V, device=DEV) * 2).bfloat16()
    labels = torch.randint(0, V, (M,), device=DEV, dtype=torch.int32)
    labels[::7] = -100
    n_valid = (labels != -100).sum().to(torch.int32).reshape(1)
    ref_in = logits.float().requires_grad_(True)
    ref = F.cross_entropy(ref_in, labels.long(), ignore_index=-100)
    (ref * 0.5).backward()
    acc = torch.zeros(4, device=DEV)
    work = logits.clone()
    K.ce_fwd_bwd(work, labels, n_valid, 0.5, acc, write_grad=True)
    _done()
    assert abs(acc[0].item() / n_valid.item() - ref.item()) < 2e-3 * max(1.0, ref.item())
    assert torch.allclose(work.float(), ref_in.grad, rtol=2e-2, atol=2e-6)
    # loss only: logits stay untouched
    acc.zero_()
    work = logits.clone()
    K.ce_fwd_bwd(work, labels, n_valid, 0.5, acc, write_grad=False)
    _done()
    assert torch.equal(work, logits)


@pytest.mark.parametrize("M,N", [(32768, 1024), (1000, 3072), (129, 4096), (64, 8)])
def test_column_sums(M, N):
    from allie_b200.ops import kernels as K

    torch.manual_seed(4)
    x = torch.randn(M, N, device=DEV).bfloat16()
    out = torch.full((N,), 1.5, device=DEV)
    K.colsum_bf16(x, out)
    _done()
    assert torch.allclose(out, 1.5 + x.float().sum(0), rtol=1e-3, atol=2e-2)
    # device-side row limit
    lim = torch.tensor([M // 3], device=DEV, dtype=torch.int32)
    out.zero_()
    K.colsum_bf16(x, out, m_limit=lim)
    _done()
    assert torch.allclose(out, x[: M // 3].float().sum(0), rtol=1e-3, atol=2e-2)


def test_adamw_with_clipping_matches_torch():
    from allie_b200.ops import kernels as K

    torch.manual_seed(5)
    n = 1 << 20
    p = torch.randn(n, device=DEV)
    g = torch.randn(n, device=DEV) * 0.01
    ref_p = p.clone().requires_grad_(True)
    opt = torch.optim.AdamW([ref_p], lr=1e-3, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    m = torch.zeros(n, device=DEV)
    v = torch.zeros(n, device=DEV)
    shadow = torch.empty(n, device=DEV, dtype=torch.bfloat16)
    for step in (1, 2, 3):
        ref_p.grad = g.clone()
        torch.nn.utils.clip_grad_norm_([ref_p], 1.0)
        opt.step()
        nsq = torch.zeros(1, device=DEV)
        K.sumsq(g, nsq)
        K.adamw(p, g, m, v, shadow, 1e-3, 0.9, 0.95, 1e-8, 0.1, step, gnorm_sq=nsq, max_norm=1.0)
        _done()
        assert abs(nsq.item() - (g.double() ** 2).sum().item()) < 1e-3 * nsq.item()
        assert torch.allclose(p, ref_p.detach(), rtol=1e-5, atol=2e-6), step
        assert torch.allclose(shadow.float(), p, rtol=1e-2, atol=1e-3)
        g = g * 1.7 + 0.003


def test_cast_to_bf16():
    from allie_b200.ops import kernels as K

    src = torch.randn(100_003 * 8, device=DEV)
    dst = torch.empty_like(src, dtype=torch.bfloat16)
    K.cast_bf16(src, dst)
    _done()
    assert torch.equal(dst, src.bfloat16())


@pytest.mark.parametrize("M,V,K", [(1000, 2048, 256), (384, 1000, 128), (128 * 150 + 7, 2048, 1024),
                                   # one, two, four and eight CTAs of 512 columns, the last with few or none; 17 tiles
                                   # walked twice
                                   (130, 8, 64), (129, 512, 128), (1, 520, 64), (257, 1032, 128), (300, 2056, 192),
                                   (128, 4096, 64), (200, 4104, 128)])
def test_fused_lmhead_cross_entropy_matches_fp32(M, V, K):
    """Fused output-embedding GEMM + cross entropy: summed loss and d logits against plain PyTorch
    fp32 on the same bf16 operands; ragged row count, ignored rows, a vocabulary that is not a
    multiple of the 256-column tile, more row tiles than SMs (second unit per CTA)."""
    import torch.nn.functional as F

    from allie_b200.ops import _lib, kernels as K_

    torch.manual_seed(M + V)
    h = (torch.randn(M, K, device="cuda") * 1.0).bfloat16()
    wte = (torch.randn(V, K, device="cuda") * 0.08).bfloat16()
    labels = torch.randint(0, V, (M,), device="cuda", dtype=torch.int32)
    labels[torch.rand(M, device="cuda") < 0.2] = -100
    n_valid = (labels >= 0).sum().to(torch.int32).reshape(1)
    coef = 0.7
    dlogits = torch.full((M, V), 3.0, device="cuda", dtype=torch.bfloat16)
    loss = torch.zeros(1, device="cuda")
    K_.lmhead_ce(h, wte, labels, n_valid, coef, dlogits, loss)
    torch.cuda.synchronize()
    _lib.check_status()
    logits = (h.float() @ wte.float().t()).requires_grad_(True)
    ref = F.cross_entropy(logits, labels.long(), ignore_index=-100, reduction="sum")
    (ref * coef / int(n_valid)).backward()
    assert abs(loss.item() - ref.item()) < 2e-3 * ref.item()
    g = logits.grad
    err = (dlogits.float() - g).abs().max().item()
    assert err < 0.02 * g.abs().max().item() + 1e-7, (err, g.abs().max().item())
    assert (dlogits[labels < 0].float() == 0).all()


@pytest.mark.parametrize("dependent,ready", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("d", list(range(128, 2049, 128)))
def test_layernorm_forward_widths(d, rms, dependent, ready):
    """Every width, with and without the parameters fetched ahead; one row, more rows than SMs, two rows for a
    block's last warp and none.  bf16 results: half a unit in the last place of a value of up to 6."""
    from allie_b200.ops import kernels as K

    for M in (1, 147, 149, 1185):
        torch.manual_seed(M)
        x = torch.randn(M, d, device=DEV) * 2 + 1
        g, b = torch.randn(d, device=DEV), torch.randn(d, device=DEV)
        y = torch.empty(M, d, device=DEV, dtype=torch.bfloat16)
        mean, rstd = torch.empty(M, device=DEV), torch.empty(M, device=DEV)
        _done()                                  # with `ready`, no kernel in flight may be writing g and b
        K.layernorm_fwd(x, g, None if rms else b, y, mean, rstd, 1e-5, rms, dependent=dependent, weights_ready=ready)
        _done()
        x64 = x.double()
        mu = torch.zeros(M, 1, device=DEV, dtype=torch.float64) if rms else x64.mean(1, keepdim=True)
        r = ((x64 - mu).pow(2).mean(1, keepdim=True) + 1e-5).rsqrt()
        want = (x64 - mu) * r * g.double() + (0 if rms else b.double())
        assert ((y.double() - want).abs() <= want.abs() * 2 ** -8 + 1e-5).all()
        assert torch.allclose(rstd.double(), r[:, 0], rtol=1e-5) and torch.allclose(mean.double(), mu[:, 0], atol=1e-5)


@pytest.mark.parametrize("d", [128, 1024, 2048])
def test_dependent_layernorm_waits_for_its_weights(d):
    """Gamma and beta that the kernel before writes (a long contraction that lets its dependents start at once)
    are read when it has written them."""
    from allie_b200.ops import kernels as K
    from allie_b200.ops.gemm import gemm

    torch.manual_seed(d)
    a, w = torch.randn(2, 16384, device=DEV).bfloat16(), (torch.randn(16384, d, device=DEV) * 0.01).bfloat16()
    x = torch.randn(64, d, device=DEV)
    gb = torch.zeros(2, d, device=DEV)
    y, want = (torch.empty(64, d, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    mean, rstd = torch.empty(64, device=DEV), torch.empty(64, device=DEV)
    for _ in range(3):
        gb.zero_()
        gemm(a, w, b_mn=True, out=gb)
        K.layernorm_fwd(x, gb[0], gb[1], y, mean, rstd, 1e-5, dependent=True)
    _done()
    assert float(gb.abs().min(0).values.max()) > 0
    K.layernorm_fwd(x, gb[0], gb[1], want, mean, rstd, 1e-5)
    _done()
    assert torch.equal(y, want)


@pytest.mark.parametrize("M,d", [(1, 128), (5, 96), (7, 384), (3, 1024), (4, 1280), (300, 256), (9, 2048),
                                 (3072, 100), (3073, 100), (3077, 384), (3079, 1280)])
def test_embedding_rows_of_any_width(M, d):
    """Several rows to a block, one, and a row in two rounds, beyond 3072 rows a warp each: control token, dropped and
    kept elements."""
    from allie_b200.ops import _lib, kernels as K

    torch.manual_seed(11)
    V, P, p, seed, stream = 64, 32, 0.25, 5, 3
    wte, wpe, ctrl = (torch.randn(n, d, device="cuda") for n in (V, P, 2))
    ids = torch.randint(0, V, (M,), device="cuda", dtype=torch.int32)
    ids[0] = V + 1500
    pos = torch.randint(0, P, (M,), device="cuda", dtype=torch.int32)
    want = wte[ids.clamp(max=V - 1).long()] + wpe[pos.long()]
    e = (1500 - 500) / 2500
    want[0] = e * ctrl[0] + (1 - e) * ctrl[1] + wpe[pos[0].long()]
    x = torch.full((M + 1, d), 7.0, device="cuda")
    K.embed_fwd(ids, pos, wte, wpe, ctrl, x[:M], V, 0, 0, 0.0)
    assert torch.allclose(x[:M], want, rtol=1e-6, atol=1e-6) and (x[M] == 7.0).all()
    K.embed_fwd(ids, pos, wte, wpe, ctrl, x[:M], V, seed, stream, p)
    n = -(-M * d // 8) * 8
    keep = torch.empty(n, dtype=torch.uint8)
    thr = _lib.dropout_thr16(p)
    assert _lib.cuda().ab_dropout_mask_host(ctypes.c_ulonglong(seed), ctypes.c_uint(stream), ctypes.c_longlong(n),
                                            ctypes.c_uint(thr), ctypes.c_void_p(keep.data_ptr())) == 0
    keep = keep[:M * d].view(M, d).cuda()
    assert torch.allclose(x[:M], want * keep * (65536.0 / (65536 - thr)), rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("M,d", [(1, 128), (9, 1024), (3, 1280), (20, 2048), (5, 100)])
def test_scalar_heads_with_and_without_waiting(M, d):
    from allie_b200.ops import kernels as K

    torch.manual_seed(12)
    h = torch.randn(M, d, device="cuda").bfloat16()
    wv, wt = (torch.randn(d, device="cuda") * 0.05 for _ in range(2))
    bv, bt = torch.randn(1, device="cuda"), torch.randn(1, device="cuda")
    outs = [torch.full((M + 1,), 7.0, device="cuda") for _ in range(4)]
    K.heads_fwd(h, wv, bv, wt, bt, None, None, torch.zeros(4, dtype=torch.int32, device="cuda"), 0.0, 0.0, outs[0][:M],
                outs[1][:M], None, None, None)
    K.heads_fwd_ahead(h, wv, bv, wt, bt, outs[2][:M], outs[3][:M])
    want_v, want_t = torch.tanh(h.double() @ wv.double() + bv), h.double() @ wt.double() + bt
    # d products of fp32 rounding, summed to order 1
    assert torch.allclose(outs[0][:M].double(), want_v, atol=1e-5) and torch.allclose(outs[1][:M].double(), want_t, atol=1e-5)
    assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1], outs[3]) and outs[2][M] == 7.0


@pytest.mark.parametrize("M", [1, 8, 9, 2047, 2500, 20000])
def test_scalar_head_gradients_over_any_rows(M):
    from allie_b200.ops import kernels as K

    torch.manual_seed(13)
    d = 256
    h = torch.randn(M, d, device="cuda").bfloat16()
    dv, dt = torch.randn(M, device="cuda"), torch.randn(M, device="cuda")
    gv, gt = torch.ones(d, device="cuda"), torch.ones(d, device="cuda")
    bv, bt = torch.ones(1, device="cuda"), torch.ones(1, device="cuda")
    K.heads_bwd_w(h, dv, dt, gv, bv, gt, bt)
    tol = 1e-6 * M ** 0.5 * 6 + 1e-5          # sums of M terms of order one in fp32
    for g, b, x in ((gv, bv, dv), (gt, bt, dt)):
        assert (g.double() - 1 - x.double() @ h.double()).abs().max() < tol * 6
        assert abs(float(b) - 1 - float(x.double().sum())) < tol * 6


@pytest.mark.parametrize("dependent", [0, 1])
def test_policy_rows_of_any_number_of_moves(dependent):
    """None, a warp's worth, the 64 that stay in registers and more."""
    from allie_b200.ops import _lib

    torch.manual_seed(14)
    counts, width, V = [0, 1, 31, 32, 33, 63, 64, 65, 100, 224], 224, 2048
    n = len(counts)
    logits = torch.randn(n, V, device="cuda").bfloat16()
    active = torch.ones(n, dtype=torch.int32, device="cuda")
    active[3] = 0
    legal = torch.stack([torch.randperm(V, device="cuda")[:width] for _ in counts]).int()
    n_legal = torch.tensor(counts, dtype=torch.int32, device="cuda")
    value, time = torch.randn(n, device="cuda"), torch.randn(n, device="cuda")
    out = torch.full((n * (width + 4) + 1,), 7.0, device="cuda")
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    assert _lib.cuda().ab_policy_epilogue(P(logits), ctypes.c_longlong(V), P(active), P(legal), width, P(n_legal), P(value),
                                          P(time), 1992, ctypes.c_float(1.0), P(out), width + 4, n, P(_lib.status_word()),
                                          dependent, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    rows = out[:-1].view(n, width + 4)
    for t, c in enumerate(counts):
        if t == 3:
            assert (rows[t] == 7.0).all()
            continue
        x = logits[t, legal[t, :c].long()].float()
        assert torch.allclose(rows[t, :c], x.softmax(0), rtol=1e-5, atol=1e-6) and (rows[t, c:width] == 7.0).all()
        assert rows[t, width] == value[t] and rows[t, width + 1] == time[t] and rows[t, width + 2] == logits[t, 1992].float()
        assert c == 0 or rows[t, width + 3] == x.max()
