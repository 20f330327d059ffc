"""tcgen05 causal attention (forward and backward) against a plain PyTorch fp32 reference."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(qkv, B, T, H, hd, mask=None, scale_keep=1.0):
    q5 = qkv.float().view(B, T, 3, H, hd)
    q, k, v = (q5[:, :, i].transpose(1, 2) for i in range(3))
    s = (q @ k.transpose(-1, -2)) / math.sqrt(hd)
    causal = torch.ones(T, T, dtype=torch.bool, device=qkv.device).tril()
    s = s.masked_fill(~causal, float("-inf"))
    p = s.softmax(-1)
    lse = torch.logsumexp(s, -1)
    if mask is not None:
        p = p * mask * scale_keep
    o = (p @ v).transpose(1, 2).reshape(B * T, H * hd)
    return o, lse


@pytest.mark.parametrize("B,T,H,hd", [(2, 128, 2, 64), (2, 512, 3, 64), (1, 200, 2, 64), (2, 256, 2, 128),
                                      (1, 40, 1, 128), (20, 384, 16, 64)])
def test_attention_fwd_bwd_no_dropout(B, T, H, hd):
    from allie_b200.ops import _lib
    from allie_b200.ops.attention import attention_bwd, attention_fwd

    torch.manual_seed(0)
    dev = "cuda"
    d = H * hd
    qkv = (torch.randn(B * T, 3 * d, device=dev) * 0.7).bfloat16()
    out = torch.zeros(B * T, d, device=dev, dtype=torch.bfloat16)
    lse = torch.zeros(B, H, T, device=dev)
    attention_fwd(qkv, out, lse, B, T, H, hd, 0.0, 0, 0)
    torch.cuda.synchronize()
    _lib.check_status()
    leaf = qkv.float().requires_grad_(True)
    o_ref, lse_ref = _ref(leaf, B, T, H, hd)
    assert torch.allclose(out.float(), o_ref, rtol=2e-2, atol=2e-2), (out.float() - o_ref).abs().max()
    assert torch.allclose(lse, lse_ref, rtol=1e-3, atol=1e-2)
    dout = (torch.randn(B * T, d, device=dev) * 0.5).bfloat16()
    delta = torch.zeros(B, H, T, device=dev)
    o_ref.backward(dout.float())
    g = leaf.grad
    # two-kernel backward, and for head_dim 64 also the single-kernel one with its fp32 dQ
    # accumulator under both of its schedules (1 = one key tile per CTA, 2 = persistent walk)
    from allie_b200.ops.attention import set_backward_schedule

    variants = [(None, 0)] + ([(torch.zeros(B * T, d, device=dev), 1), (torch.zeros(B * T, d, device=dev), 2)]
                              if hd == 64 else [])
    for dq_acc, schedule in variants:
        set_backward_schedule(schedule)
        dqkv = torch.zeros(B * T, 3 * d, device=dev, dtype=torch.bfloat16)
        attention_bwd(qkv, out, lse, dout, dqkv, delta, B, T, H, hd, 0.0, 0, 0, None, dq_acc)
        torch.cuda.synchronize()
        _lib.check_status()
        err = (dqkv.float() - g).abs().max().item()
        assert err < 3e-2 * max(1.0, g.abs().max().item()), err
        for i, name in enumerate("qkv"):
            a, b_ = dqkv.float()[:, i * d:(i + 1) * d], g[:, i * d:(i + 1) * d]
            rel = (a - b_).norm() / (b_.norm() + 1e-9)
            assert rel < 2e-2, (name, rel.item(), dq_acc is not None)
        if dq_acc is not None:
            assert float(dq_acc.abs().max()) == 0.0     # handed back cleared
    set_backward_schedule(0)


def test_attention_dropout_mask_consistency():
    """Recover the dropped attention matrix through its linearity in V, check the keep rate and
    scaling, and check the backward pass against autograd with that same mask."""
    from allie_b200.ops import _lib
    from allie_b200.ops.attention import attention_bwd, attention_fwd

    torch.manual_seed(1)
    dev = "cuda"
    B, T, H, hd, p = 1, 256, 2, 64, 0.25
    d = H * hd
    seed, stream = 987654321, 5
    qkv = (torch.randn(B * T, 3 * d, device=dev) * 0.5).bfloat16()
    A = torch.zeros(B, H, T, T, device=dev)
    lse = torch.zeros(B, H, T, device=dev)
    for blk in range(T // hd):
        probe = qkv.clone()
        v = torch.zeros(B, T, H, hd, device=dev)
        for c in range(hd):
            v[:, blk * hd + c, :, c] = 1.0
        probe[:, 2 * d:] = v.view(B * T, d).bfloat16()
        out = torch.zeros(B * T, d, device=dev, dtype=torch.bfloat16)
        attention_fwd(probe, out, lse, B, T, H, hd, p, seed, stream)
        A[:, :, :, blk * hd:(blk + 1) * hd] = out.float().view(B, T, H, hd).permute(0, 2, 1, 3)
    torch.cuda.synchronize()
    _lib.check_status()
    causal = torch.ones(T, T, dtype=torch.bool, device=dev).tril()
    mask = (A != 0)
    keep_rate = mask[..., causal].float().mean().item()
    assert abs(keep_rate - (1 - p)) < 0.01, keep_rate
    assert not mask[..., ~causal].any()
    thr = _lib.dropout_thr16(p)
    scale_keep = 65536.0 / (65536 - thr)
    leaf = qkv.float().requires_grad_(True)
    o_ref, _ = _ref(leaf, B, T, H, hd, mask.float(), scale_keep)
    out = torch.zeros(B * T, d, device=dev, dtype=torch.bfloat16)
    bits = torch.zeros(B, H, T, T // 32, device=dev, dtype=torch.int32)
    attention_fwd(qkv, out, lse, B, T, H, hd, p, seed, stream, bits)
    assert torch.allclose(out.float(), o_ref, rtol=3e-2, atol=3e-2)
    # the stored keep bits are the mask recovered above
    unpacked = ((bits.unsqueeze(-1) >> torch.arange(32, device=dev)) & 1).view(B, H, T, T).bool()
    assert torch.equal(unpacked & causal, mask & causal)
    dout = (torch.randn(B * T, d, device=dev) * 0.5).bfloat16()
    delta = torch.zeros(B, H, T, device=dev)
    o_ref.backward(dout.float())
    # regenerate the mask / read the stored bits; two-kernel / single-kernel backward
    from allie_b200.ops.attention import set_backward_schedule

    for use_bits, fused in ((False, 0), (True, 0), (False, 1), (True, 1), (False, 2), (True, 2)):
        set_backward_schedule(fused)           # 0: two-kernel backward; 1, 2: the fused kernel's schedules
        dqkv = torch.zeros(B * T, 3 * d, device=dev, dtype=torch.bfloat16)
        dq_acc = torch.zeros(B * T, d, device=dev) if fused else None
        attention_bwd(qkv, out, lse, dout, dqkv, delta, B, T, H, hd, p, seed, stream,
                      bits if use_bits else None, dq_acc)
        torch.cuda.synchronize()
        _lib.check_status()
        rel = (dqkv.float() - leaf.grad).norm() / leaf.grad.norm()
        assert rel < 3e-2, (rel.item(), use_bits, fused)
    set_backward_schedule(0)


@pytest.mark.parametrize("B,T,H,hd", [(2, 128, 2, 64), (160, 256, 1, 64), (40, 512, 4, 64), (3, 200, 2, 64), (2, 256, 2, 128)])
def test_attention_bwd_bias_sums_and_accumulator(B, T, H, hd):
    """The column sums of dQKV that the backward adds, from its own tiles (persistent walk over whole
    tiles: one tile, a CTA with one slice and with two, the sums of a slice kept in place) and by the pass
    that stands in elsewhere; the accumulator comes back all zero; the schedules agree.  Sums of B*T fp32
    terms: any order is within B*T * 2^-23 * sum|terms|."""
    from allie_b200.ops import _lib
    from allie_b200.ops.attention import attention_bwd, attention_fwd, set_backward_schedule

    torch.manual_seed(3)
    d = H * hd
    dev = "cuda"
    qkv = (torch.randn(B * T, 3 * d, device=dev) * 0.7).bfloat16()
    out = torch.zeros(B * T, d, device=dev, dtype=torch.bfloat16)
    lse, delta = torch.zeros(B, H, T, device=dev), torch.zeros(B, H, T, device=dev)
    attention_fwd(qkv, out, lse, B, T, H, hd, 0.0, 0, 0)
    dout = torch.randn(B * T, d, device=dev).bfloat16()
    grads = []
    for schedule in (1, 2) if hd == 64 else (0,):
        set_backward_schedule(schedule)
        acc = torch.zeros(B * T, d, device=dev) if hd == 64 else None
        for _ in range(2):
            dqkv = torch.full((B * T, 3 * d), float("nan"), device=dev, dtype=torch.bfloat16)
            dbias = torch.full((3 * d,), 0.5, device=dev)
            attention_bwd(qkv, out, lse, dout, dqkv, delta, B, T, H, hd, 0.0, 0, 0, None, acc, dbias=dbias)
            torch.cuda.synchronize()
            _lib.check_status()
            terms = dqkv.double()
            bound = 1e-6 + B * T * 2.0 ** -23 * (terms.abs().sum(0) + 0.5)
            assert ((dbias.double() - 0.5 - terms.sum(0)).abs() <= bound).all()
            assert acc is None or not acc.any()
        grads.append(dqkv.float())
    set_backward_schedule(0)
    # the schedules add a query tile's parts in different orders: single bf16 roundings flip
    for g in grads[1:]:
        assert (g - grads[0]).norm() / grads[0].norm() < 1e-3


def _inputs(kind, B, T, H, hd):
    """plain; later keys score higher, so that the running maximum of a row grows in every key tile; values
    of one sign, whose sums lose most to rounding."""
    x = torch.randn(B, T, 3, H, hd, device="cuda") * 0.7
    if kind == "late":
        x[:, :, 0, :, :] = x[:, :, 0].abs()
        x[:, :, 1] = x[:, :, 1].abs() * torch.linspace(-3, 1, T, device="cuda").exp2()[None, :, None, None]
    elif kind == "mean":
        x[:, :, 2] += 1.0
    return x.reshape(B * T, 3 * H * hd).bfloat16()


@pytest.mark.parametrize("hd,T", [(64, 129), (64, 384), (64, 1000), (128, 129), (128, 384), (128, 520), (128, 1000)])
@pytest.mark.parametrize("kind", ["plain", "late", "mean"])
@pytest.mark.parametrize("p", [0.0, 0.1])
def test_attention_fwd_against_64_bits(hd, T, kind, p):
    """Two to eight key tiles (at heads of 128 every stage is used again, O is rescaled in place).  Bound,
    element by element: P and the stored result are rounded to bf16 (eight significant bits, so up to 2^-8 of
    each term, twice), exponentials and fp32 sums (the tensor core cuts them off) are good for 2^-13 together at
    these lengths."""
    from allie_b200.ops import _lib
    from allie_b200.ops.attention import attention_fwd

    if p and T % 32:
        T = T // 32 * 32                    # keep bits are kept for whole words
    torch.manual_seed(0)
    B, H = 2, 2
    d, dev = H * hd, "cuda"
    qkv = _inputs(kind, B, T, H, hd)
    out = torch.full((B * T, d), float("nan"), device=dev, dtype=torch.bfloat16)
    lse = torch.zeros(B, H, T, device=dev)
    bits = torch.zeros(B, H, T, T // 32, device=dev, dtype=torch.int32) if p else None
    attention_fwd(qkv, out, lse, B, T, H, hd, p, 77, 3, bits)
    torch.cuda.synchronize()
    _lib.check_status()
    q, k, v = (qkv.view(B, T, 3, H, hd)[:, :, i].transpose(1, 2).double() for i in range(3))
    s = (q @ k.transpose(-1, -2)) / math.sqrt(hd)
    s = s.masked_fill(~torch.ones(T, T, dtype=torch.bool, device=dev).tril(), float("-inf"))
    probs = s.softmax(-1)
    if kind == "late":                     # the maximum does grow, tile after tile
        tops = torch.stack([s[:, :, T - 1, j:j + 128].amax(-1) for j in range(0, T, 128)], -1)
        assert (tops[..., 1:-1] > tops[..., :-2]).all()
    assert torch.allclose(lse.double(), torch.logsumexp(s, -1), rtol=1e-5, atol=1e-4)
    if p:
        keep = ((bits.unsqueeze(-1) >> torch.arange(32, device=dev)) & 1).view(B, H, T, T)
        probs = probs * keep * (65536.0 / (65536 - _lib.dropout_thr16(p)))
    want = (probs @ v).transpose(1, 2).reshape(B * T, d)
    size = (probs @ v.abs()).transpose(1, 2).reshape(B * T, d)
    err = (out.double() - want).abs()
    assert (err <= (2 * 2 ** -8 + 2 ** -13) * size + 1e-7).all(), float((err / (size + 1e-9)).max())


@pytest.mark.parametrize("B,T,H,hd,p", [(2, 384, 2, 128, 0.1), (1, 520, 2, 128, 0.0), (2, 1000, 1, 128, 0.0), (2, 416, 2, 64, 0.1),
                                        # sequences that end inside a tile, enough slices for the persistent walk
                                        (20, 160, 16, 64, 0.1), (20, 330, 16, 64, 0.0), (20, 416, 16, 64, 0.1)])
def test_attention_bwd_over_several_key_tiles(B, T, H, hd, p):
    """Gradients against autograd in 64 bits with the stored mask, several key tiles, by all three
    schedules.  P, dS and the results are rounded to bf16: under 1 % in the 2-norm."""
    from allie_b200.ops import _lib
    from allie_b200.ops.attention import attention_bwd, attention_fwd

    torch.manual_seed(2)
    d, dev = H * hd, "cuda"
    qkv = (torch.randn(B * T, 3 * d, device=dev) * 0.7).bfloat16()
    out = torch.zeros(B * T, d, device=dev, dtype=torch.bfloat16)
    lse, delta = torch.zeros(B, H, T, device=dev), torch.zeros(B, H, T, device=dev)
    bits = torch.zeros(B, H, T, T // 32, device=dev, dtype=torch.int32) if p else None
    attention_fwd(qkv, out, lse, B, T, H, hd, p, 5, 1, bits)
    dout = torch.randn(B * T, d, device=dev).bfloat16()
    leaf = qkv.double().requires_grad_(True)
    q, k, v = (leaf.view(B, T, 3, H, hd)[:, :, i].transpose(1, 2) for i in range(3))
    s = (q @ k.transpose(-1, -2)) / math.sqrt(hd)
    probs = s.masked_fill(~torch.ones(T, T, dtype=torch.bool, device=dev).tril(), float("-inf")).softmax(-1)
    if p:
        keep = ((bits.unsqueeze(-1) >> torch.arange(32, device=dev)) & 1).view(B, H, T, T)
        probs = probs * keep * (65536.0 / (65536 - _lib.dropout_thr16(p)))
    (probs @ v).transpose(1, 2).reshape(B * T, d).backward(dout.double())
    dqkv = torch.full((B * T, 3 * d), float("nan"), device=dev, dtype=torch.bfloat16)
    acc = torch.zeros(B * T, d, device=dev) if hd == 64 else None
    launched = _lib.LAUNCHES
    attention_bwd(qkv, out, lse, dout, dqkv, delta, B, T, H, hd, p, 5, 1, bits, acc)
    torch.cuda.synchronize()
    _lib.check_status()
    # row sums of dO * O, and the walk; two kernels for heads of 128; a grid of key tiles and its conversion
    assert _lib.LAUNCHES - launched == (2 if B == 20 else 3)
    for i in range(3):
        a, b = dqkv[:, i * d:(i + 1) * d].double(), leaf.grad[:, i * d:(i + 1) * d]
        assert float((a - b).norm() / b.norm()) < 1e-2, "qkv"[i]


@pytest.mark.parametrize("B,H,T,p", [(40, 8, 200, 0.1), (20, 16, 328, 0.1), (20, 16, 330, 0.0), (160, 4, 72, 0.1),
                                     (38, 8, 160, 0.1), (38, 8, 129, 0.0)])
def test_persistent_backward_of_ragged_sequences(B, H, T, p):
    """Sequences that end inside a tile, walked by persistent CTAs, against one key tile per CTA: the sums over key
    tiles are added in another order, so single bf16 roundings flip (2^-8 of an element at most); the bias
    gradient is the column sums of what was stored."""
    from allie_b200.ops import _lib
    from allie_b200.ops.attention import attention_bwd, attention_fwd, set_backward_schedule

    torch.manual_seed(B + T)
    hd, d = 64, H * 64
    qkv = torch.randn(B * T, 3 * d, device="cuda").bfloat16()
    dout = torch.randn(B * T, d, device="cuda").bfloat16()
    out, lse, delta = torch.zeros_like(dout), torch.zeros(B, H, T, device="cuda"), torch.zeros(B, H, T, device="cuda")
    bits = torch.zeros(B, H, T, T // 32, device="cuda", dtype=torch.int32) if p and T % 32 == 0 else None
    attention_fwd(qkv, out, lse, B, T, H, hd, p, 5, 1, bits)
    got = {}
    for mode in (1, 2):
        set_backward_schedule(mode)
        dqkv, acc = torch.full_like(qkv, 7.0), torch.zeros(B * T, d, device="cuda")
        dbias = torch.zeros(3 * d, device="cuda")
        try:
            attention_bwd(qkv, out, lse, dout, dqkv, delta, B, T, H, hd, p, 5, 1, bits, acc, dbias=dbias)
        finally:
            set_backward_schedule(0)
        torch.cuda.synchronize()
        _lib.check_status()
        assert float(acc.abs().max()) == 0.0
        got[mode] = dqkv.float()
        sums = dqkv.double().sum(0)
        assert ((dbias.double() - sums).abs() <= 1e-5 * dqkv.double().abs().sum(0) + 1e-6).all()
    assert float((got[1] - got[2]).norm() / got[1].norm()) < 2e-3
    assert ((got[1] - got[2]).abs() <= 2 ** -7 * got[1].abs() + 1e-2 * got[1].pow(2).mean().sqrt()).all()


@pytest.mark.parametrize("T", [96, 160, 448])
@pytest.mark.parametrize("hd", [64, 128])
def test_two_kernel_backward_reads_no_keep_bits_past_a_sequence(T, hd):
    """The last key tile reaches past the sequence, where the mask's words are another row's or not the mask's at
    all.  Values that are not finite there (the next sequence's V) would reach dQ through such a bit: P is zero,
    but zero times infinity is not."""
    from allie_b200.ops import _lib
    from allie_b200.ops.attention import attention_bwd, attention_fwd

    torch.manual_seed(T)
    B, H = 2, 2
    d, dev = H * hd, "cuda"
    qkv = torch.randn(B * T, 3 * d, device=dev).bfloat16()
    dout = torch.randn(B * T, d, device=dev).bfloat16()
    out, lse, delta = torch.zeros_like(dout), torch.zeros(B, H, T, device=dev), torch.zeros(B, H, T, device=dev)
    words = B * H * T * (T // 32)
    store = torch.full((words + 64,), -1, device=dev, dtype=torch.int32)      # ones behind the mask
    bits = store[:words].view(B, H, T, T // 32)
    attention_fwd(qkv, out, lse, B, T, H, hd, 0.1, 5, 1, bits)
    got = []
    for last_v in (None, float("inf")):
        x = qkv.clone()
        if last_v is not None:
            x[T:, 2 * d:] = last_v
        dqkv = torch.zeros_like(qkv)
        attention_bwd(x, out, lse, dout, dqkv, delta, B, T, H, hd, 0.1, 5, 1, bits)
        got.append(dqkv[:T])
    torch.cuda.synchronize()
    _lib.check_status()
    assert got[0].isfinite().all() and torch.equal(got[0], got[1])


@pytest.mark.parametrize("hd,H,lens", [
    (64, 16, [300] * 20), (64, 8, [1, 128, 129, 300, 4, 257] * 14), (64, 3, [700, 1, 1, 1, 128] * 20 + [5]),
    (128, 8, [1, 128, 129, 300, 4, 257] * 14), (128, 5, [384] * 20), (64, 37, [16] * 8), (64, 37, [16] * 9),
])
def test_blocks_that_take_over_others(hd, H, lens):
    """More items than CTAs fit the GPU (and, last, just as many and some more than 296), with blocks in
    between that have no rows: packed sequences against a call of their own each, to the bit, and against fp32."""
    import ctypes

    import numpy as np

    from allie_b200.ops import _lib

    torch.manual_seed(3)
    lib, d = _lib.cuda(), H * hd
    row0 = torch.from_numpy(np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)).cuda()
    M = int(row0[-1])
    qkv = (torch.randn(M, 3 * d, device="cuda") * 0.7).bfloat16()
    P = lambda t: ctypes.c_void_p(t.data_ptr())

    def packed(rows, starts, n, longest):
        out = torch.full((rows.shape[0] + 128, d), 7.0, device="cuda", dtype=torch.bfloat16)
        assert lib.ab_attn_fwd_packed(P(rows), P(out), P(starts), n, longest, rows.shape[0], H, hd,
                                      ctypes.c_float(hd ** -0.5), 0, P(_lib.status_word()),
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        assert (out[rows.shape[0]:] == 7.0).all()
        return out[:rows.shape[0]]

    outs = [packed(qkv, row0, len(lens), max(lens)) for _ in range(3)]
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    starts = row0.tolist()
    for i in range(0, len(lens), 7):
        rows = qkv[starts[i]:starts[i + 1]].contiguous()
        alone = packed(rows, torch.tensor([0, len(rows)], dtype=torch.int32, device="cuda"), 1, len(rows))
        assert torch.equal(alone, outs[0][starts[i]:starts[i + 1]]), i
        ref, _ = _ref(rows, 1, len(rows), H, hd)
        assert torch.allclose(alone.float(), ref, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("B,T,H,hd", [(24, 296, 8, 64), (40, 512, 4, 64), (24, 384, 5, 128), (64, 384, 5, 128)])
def test_dropout_of_blocks_that_take_over_others(B, T, H, hd):
    """Keep bits of every item as the host draws them, and the outputs as fp32 gives them with these."""
    from allie_b200.ops import _lib
    from allie_b200.ops.attention import attention_fwd

    torch.manual_seed(4)
    d, p, seed, stream = H * hd, 0.1, 77, 9
    qkv = (torch.randn(B * T, 3 * d, device="cuda") * 0.5).bfloat16()
    out = torch.zeros(B * T, d, device="cuda", dtype=torch.bfloat16)
    lse = torch.zeros(B, H, T, device="cuda")
    bits = torch.zeros(B, H, T, T // 32, device="cuda", dtype=torch.int32) if T % 32 == 0 else None
    attention_fwd(qkv, out, lse, B, T, H, hd, p, seed, stream, bits)
    torch.cuda.synchronize()
    _lib.check_status()
    thr = _lib.dropout_thr16(p)
    keep = torch.empty(B * H * T * T, dtype=torch.uint8)
    import ctypes

    assert _lib.cuda().ab_dropout_mask_host(ctypes.c_ulonglong(seed), stream, ctypes.c_longlong(keep.numel()), thr,
                                            ctypes.c_void_p(keep.data_ptr())) == 0
    keep = keep.cuda().view(B, H, T, T).bool()
    if bits is not None:
        causal = torch.ones(T, T, dtype=torch.bool, device="cuda").tril()
        unpacked = ((bits.unsqueeze(-1) >> torch.arange(32, device="cuda")) & 1).view(B, H, T, T).bool()
        assert torch.equal(unpacked & causal, keep & causal)
    ref, lse_ref = _ref(qkv, B, T, H, hd, keep.float(), 65536.0 / (65536 - thr))
    assert torch.allclose(out.float(), ref, rtol=3e-2, atol=3e-2)
    assert torch.allclose(lse, lse_ref, rtol=1e-3, atol=1e-2)


@pytest.mark.parametrize("hd,H,lens", [
    (64, 16, [300] * 20), (64, 8, [1, 128, 129, 300, 4, 257, 31, 32, 33, 160] * 9), (64, 3, [700, 1, 1, 1, 128] * 20 + [5]),
    (128, 8, [1, 128, 129, 300, 4, 257, 31, 32, 33, 160] * 9), (128, 5, [384] * 20), (64, 2, [90]), (128, 2, [97, 40]),
])
def test_keys_and_values_of_a_packed_batch_in_a_cache(hd, H, lens):
    """Sequence ends inside and at blocks of 32 rows: the rows as they are, no slot behind a sequence touched."""
    import ctypes

    import numpy as np

    from allie_b200.ops import _lib

    torch.manual_seed(5)
    lib, d, S, n = _lib.cuda(), H * hd, max(lens) + 3, len(lens)
    starts = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    row0 = torch.from_numpy(starts).cuda()
    M = int(starts[-1])
    qkv = (torch.randn(M, 3 * d, device="cuda") * 0.7).bfloat16()
    P = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)

    def run(kc, vc):
        out = torch.empty(M, d, device="cuda", dtype=torch.bfloat16)
        assert lib.ab_attn_fwd_packed_kv(P(qkv), P(out), P(row0), n, max(lens), M, H, hd, ctypes.c_float(hd ** -0.5), P(kc),
                                         P(vc), S, 0, P(_lib.status_word()),
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        return out

    kc, vc = (torch.full((n, H, S, hd), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    out = run(kc, vc)
    assert torch.equal(out, run(None, None))
    torch.cuda.synchronize()
    _lib.check_status()
    for i, (a, b) in enumerate(zip(starts[:-1], starts[1:])):
        rows = qkv[a:b].view(b - a, 3, H, hd)
        for cache, part in ((kc, 1), (vc, 2)):
            assert torch.equal(cache[i, :, :b - a], rows[:, part].transpose(0, 1)), i
            assert (cache[i, :, b - a:] == 7.0).all(), i
    args = [P(qkv), P(out), P(row0), n, max(lens), M, H, hd, ctypes.c_float(0.1)]
    end = [0, P(_lib.status_word()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)]
    assert lib.ab_attn_fwd_packed_kv(*args, P(kc), P(vc), max(lens) - 1, *end) == -1      # a sequence that has no room
    assert lib.ab_attn_fwd_packed_kv(*args, P(kc), P(None), S, *end) == -1
