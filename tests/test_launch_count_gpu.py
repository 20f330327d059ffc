"""The launch counter against the kernel nodes of a captured graph, for operations whose number of kernels
depends on their sizes and options."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _kernels_and_count(call):
    """(kernel nodes that ``call`` adds to a graph, kernels it counted)."""
    from allie_b200.ops import _lib

    call()                                       # first-launch set-up happens outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    before = _lib.LAUNCHES
    with torch.cuda.graph(graph):
        call()
    counted = _lib.LAUNCHES - before
    cu, n = ctypes.CDLL("libcuda.so.1"), ctypes.c_size_t(0)
    raw = ctypes.c_void_p(graph.raw_cuda_graph())
    assert cu.cuGraphGetNodes(raw, None, ctypes.byref(n)) == 0
    nodes, kind = (ctypes.c_void_p * n.value)(), ctypes.c_int(-1)
    assert cu.cuGraphGetNodes(raw, nodes, ctypes.byref(n)) == 0
    kernels = 0
    for node in nodes:
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        kernels += kind.value == 0               # CU_GRAPH_NODE_TYPE_KERNEL
    return kernels, counted


# whole tiles under the persistent walk, the same ragged, one key tile per CTA, heads of 128 in two kernels
@pytest.mark.parametrize("B,T,H,hd", [(40, 128, 16, 64), (40, 72, 16, 64), (2, 256, 2, 64), (2, 128, 2, 128)])
@pytest.mark.parametrize("delta_ready", [False, True])
@pytest.mark.parametrize("bias", [False, True])
def test_attention_backward(B, T, H, hd, delta_ready, bias):
    from allie_b200.ops import _lib
    from allie_b200.ops.attention import attention_bwd, attention_fwd

    d, dev = H * hd, "cuda"
    qkv = torch.randn(B * T, 3 * d, device=dev).bfloat16()
    out, dout = torch.zeros(B * T, d, device=dev, dtype=torch.bfloat16), torch.randn(B * T, d, device=dev).bfloat16()
    lse, delta = torch.zeros(B, H, T, device=dev), torch.zeros(B, H, T, device=dev)
    attention_fwd(qkv, out, lse, B, T, H, hd, 0.0, 0, 0)
    acc = torch.zeros(B * T, d, device=dev) if hd == 64 else None
    dqkv, dbias = torch.zeros_like(qkv), torch.zeros(3 * d, device=dev) if bias else None
    kernels, counted = _kernels_and_count(lambda: attention_bwd(
        qkv, out, lse, dout, dqkv, delta, B, T, H, hd, 0.0, 0, 0, None, acc, delta_ready, dbias))
    _lib.check_status()
    assert kernels == counted > 0


@pytest.mark.parametrize("M,N", [(4736, 1024), (512, 256), (96, 256)])
def test_gemm_with_column_sums_and_head_products(M, N):
    from allie_b200.ops import _lib
    from allie_b200.ops.gemm import gemm

    a = torch.randn(M, 128, device="cuda").bfloat16()
    w = torch.randn(N, 128, device="cuda").bfloat16()
    aux, out = torch.randn(M, N, device="cuda").bfloat16(), torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    sums, dot = torch.zeros(N, device="cuda"), torch.zeros(M // 4, N // 64, 4, device="cuda")
    for kw in (dict(act=2, aux=aux, aux_grad=True, colsum=sums), dict(colsum=sums), dict(act=4, aux=aux, dot=(dot, 4)), {}):
        kernels, counted = _kernels_and_count(lambda: gemm(a, w, out=out, **kw))
        assert kernels == counted > 0, kw
    _lib.check_status()


@pytest.mark.parametrize("n", [2, 20])            # all layers in one kernel / the chain of kernels
def test_replayed_search_step(n):
    from allie_b200.data import UCITokenizer
    from allie_b200.models import initialize_model
    from allie_b200.models.engine import B200Engine
    from allie_b200.ops import _lib
    from allie_b200.search.evaluator import KVLeafEvaluator

    tok = UCITokenizer(max_length=64, vocab_size_multiple_of=128)
    eng = B200Engine(initialize_model(tok, "gpt2", use_control_token=True, use_regression_head=True, n_layer=2, n_embd=128,
                                      n_head=2, n_positions=64), "cuda")
    counts = []
    for use_graph in (False, True):
        ev = KVLeafEvaluator(eng, n, max_prefix=16, max_nodes=8, anc_max=4, legal_max=8, use_graph=use_graph)
        ev.step()
        before = _lib.LAUNCHES
        ev.step()
        counts.append(_lib.LAUNCHES - before)
    # embedding, layers, final norm, logits, heads, policy
    assert counts[0] == counts[1] == 5 + (1 if n == 2 else 7 * 2)
