"""Failure reporting of device-side waits: a wait on a peer flag that nothing ever sets runs out
after its clock limit (about a second), the kernel records the reason in the status word and
returns, the host turns that into an exception, and the CUDA context stays usable (GPU)."""
import time
from ctypes import c_int, c_uint

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_peer_wait_runs_out_with_a_status_and_the_context_survives():
    from allie_b200.ops import _lib
    from allie_b200.ops._lib import ptr, stream_ptr

    lib = _lib.cuda()
    flags = torch.zeros(4 * 32, dtype=torch.int32, device="cuda")       # phase slots no peer will write
    st = _lib.status_word()
    st.zero_()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    assert lib.ab_nvl_wait(ptr(flags), c_int(0), c_int(1), c_uint(1), ptr(st), stream_ptr()) == 0
    torch.cuda.synchronize()
    waited = time.perf_counter() - t0
    assert 0.2 < waited < 10, waited
    with pytest.raises(RuntimeError, match="peer"):
        _lib.check_status()
    assert int(st[0]) == 0                                               # reading the status clears it
    x = torch.ones(1024, device="cuda")
    assert float(x.sum()) == 1024.0                                      # the context still works
    flags[0] = 1                                                         # the "peer" has signalled epoch 1
    t0 = time.perf_counter()
    assert lib.ab_nvl_wait(ptr(flags), c_int(0), c_int(1), c_uint(1), ptr(st), stream_ptr()) == 0
    torch.cuda.synchronize()
    assert time.perf_counter() - t0 < 0.2
    _lib.check_status()


def _small_engine():
    from allie_b200.data import UCITokenizer
    from allie_b200.models import initialize_model
    from allie_b200.search.runner import EngineRunner

    torch.manual_seed(0)
    tok = UCITokenizer(max_length=64, vocab_size_multiple_of=128)
    model = initialize_model(tok, "gpt2", use_control_token=True, use_regression_head=True, n_layer=2, n_embd=256,
                             n_head=4, n_positions=64)
    return tok, EngineRunner(model, tok)


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("n", [3, 20])        # all layers in one kernel / the chain of kernels
def test_inference_raises_when_a_wait_ran_out(n, use_graph):
    """A kernel that gave up leaves a code in the status word and unfinished values behind it: whoever
    hands results to a program says so, and the next call works again."""
    import numpy as np

    from allie_b200.data import Game
    from allie_b200.ops import _lib
    from allie_b200.search.batched import KVStepEvaluator

    tok, runner = _small_engine()
    games = [Game("180+0", 1500, 1600, None, False, ["e2e4", "e7e5"][:i % 3], [1] * (i % 3)) for i in range(n)]
    ev = KVStepEvaluator(runner.engine, tok, n, anc_max=8, legal_max=8, max_prefix=32, max_nodes=8, use_graph=use_graph)
    slot = np.array([3 + i % 3 for i in range(n)], np.int32)
    anc = np.zeros((n, 8), np.int32)
    anc[:, 0] = slot
    req = dict(need_eval=np.ones(n, np.int32), tok=np.ones(n, np.int32), pos=slot, slot=slot, anc=anc,
               n_anc=np.ones(n, np.int32), n_legal=np.full(n, 8, np.int32), legal=np.tile(np.arange(8, dtype=np.int32), (n, 1)))
    calls = (lambda: ev.prefill(games), lambda: ev.step(req), lambda: runner.evaluate(games))
    for call in calls:
        call()
    for call in calls:
        _lib.status_word()[0] = 6                # as a kernel leaves it
        with pytest.raises(RuntimeError, match="timeout"):
            call()
        call()
        _lib.check_status()
