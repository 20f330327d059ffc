"""Packed inference (no padding rows, last positions only) against the plain PyTorch model."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,d,lens", [
    (4, 256, [1]), (4, 256, [90]), (4, 256, [3, 1, 128, 129, 127, 256]), (2, 256, [40, 200, 33, 128]),
    (4, 256, list(range(1, 180, 4))),
])
def test_packed_last_positions_and_cache(heads, d, lens):
    """Sequence ends on, before and after tile edges; few rows (programmatic launches) and many; head sizes 64 and 128.  Bound: bf16 operands give 2^-9 per product; three
    blocks deep the plain model differs by under 1 %."""
    from allie_b200.data import UCITokenizer
    from allie_b200.models import initialize_model
    from allie_b200.models.engine import B200Engine
    from allie_b200.ops import _lib

    torch.manual_seed(0)
    tok = UCITokenizer(max_length=256, vocab_size_multiple_of=128)
    model = initialize_model(tok, "gpt2", use_control_token=True, use_regression_head=True, n_layer=3, n_embd=d,
                             n_head=heads, n_positions=256)
    model.eval()
    eng = B200Engine(model, "cuda")
    rng = np.random.default_rng(1)
    rows = [rng.integers(0, 1968, size=n) for n in lens]
    for r in rows:
        r[0] = len(tok) + 1700
    S, L, n = 264, 3, len(rows)
    k = torch.zeros(L, n, heads, S, d // heads, dtype=torch.bfloat16, device="cuda")
    v = torch.zeros_like(k)
    logits, value, time = eng.infer_last(rows, (k, v))
    torch.cuda.synchronize()
    _lib.check_status()
    rel = lambda a, b: float((a.float() - b.float()).norm() / b.float().norm())
    grabbed = {}
    eng.load_batch({"input_ids": torch.from_numpy(np.stack([np.pad(r, (0, max(lens) - len(r)), constant_values=tok.pad_token_id) for r in rows]))}, False)
    eng.forward(n, max(lens), False, 0, False, False, kv_hook=lambda l, qkv: grabbed.update({l: qkv.clone()}))
    for i, r in enumerate(rows):
        ids = torch.from_numpy(r).cuda()[None]
        with torch.no_grad():
            out = model(input_ids=ids, position_ids=torch.arange(len(r), device="cuda")[None])
        assert rel(logits[i], out["logits"][0, -1]) < 2e-2, (i, lens[i])
        assert abs(float(value[i]) - float(out["value_logits"][0, -1])) < 2e-2
        assert abs(float(time[i]) - float(out["time_logits"][0, -1])) < 2e-2
        for l in range(L):
            q = grabbed[l].view(n, max(lens), 3, heads, d // heads)[i, :len(r)]
            for cache, want in ((k, q[:, 1]), (v, q[:, 2])):
                assert rel(cache[l, i, :, :len(r)], want.transpose(0, 1)) < 1e-2
                assert not cache[l, i, :, len(r):].any()        # slots of later nodes stay as they were


@pytest.mark.parametrize("heads,d", [(4, 256), (2, 256)])
def test_packed_sequences_of_several_key_tiles(heads, d):
    """Three to eight key tiles, heads of 64 and 128, beside short sequences; bound as above."""
    from allie_b200.data import UCITokenizer
    from allie_b200.models import initialize_model
    from allie_b200.models.engine import B200Engine
    from allie_b200.ops import _lib

    torch.manual_seed(0)
    tok = UCITokenizer(max_length=1000, vocab_size_multiple_of=128)
    model = initialize_model(tok, "gpt2", use_control_token=True, use_regression_head=True, n_layer=2, n_embd=d,
                             n_head=heads, n_positions=1000)
    model.eval()
    eng = B200Engine(model, "cuda")
    rng = np.random.default_rng(1)
    rows = [rng.integers(0, 1968, size=n) for n in (300, 5, 513, 1000, 385)]
    logits, value, _ = eng.infer_last(rows)
    torch.cuda.synchronize()
    _lib.check_status()
    for i, r in enumerate(rows):
        with torch.no_grad():
            out = model(input_ids=torch.from_numpy(r).cuda()[None], position_ids=torch.arange(len(r), device="cuda")[None])
        want = out["logits"][0, -1].float()
        assert float((logits[i].float() - want).norm() / want.norm()) < 2e-2, len(r)
        assert abs(float(value[i]) - float(out["value_logits"][0, -1])) < 2e-2


def test_evaluation_does_not_depend_on_the_games_beside_it():
    """Alone, among a few (programmatic launches, small tiles) and among many (CTA pairs): the same bits, in
    the results and in the cache."""
    from allie_b200.data import UCITokenizer
    from allie_b200.models import initialize_model
    from allie_b200.models.engine import B200Engine
    from allie_b200.ops import _lib

    torch.manual_seed(0)
    tok = UCITokenizer(max_length=400, vocab_size_multiple_of=128)
    eng = B200Engine(initialize_model(tok, "gpt2", use_control_token=True, use_regression_head=True, n_layer=4,
                                      n_embd=1024, n_head=16, n_positions=400), "cuda")
    rng = np.random.default_rng(2)
    picked = [rng.integers(0, 1968, size=n) for n in (1, 90, 130, 300)]
    others = [rng.integers(0, 1968, size=int(n)) for n in rng.integers(1, 400, size=120)]

    def run(rows):
        k = torch.zeros(4, len(rows), 16, 400, 64, dtype=torch.bfloat16, device="cuda")
        v = torch.zeros_like(k)
        return (*eng.infer_last(rows, (k, v)), k, v)

    alone = [run([r]) for r in picked]
    for n in (3, 12, 120):
        rows = [others[0], picked[0], picked[1], *others[1:n], picked[2], picked[3]]
        at = [next(i for i, r in enumerate(rows) if r is p) for p in picked]
        logits, value, time, k, v = run(rows)
        for i, (l1, v1, t1, k1, vc1) in zip(at, alone):
            assert torch.equal(logits[i], l1[0]) and torch.equal(value[i], v1[0]) and torch.equal(time[i], t1[0])
            assert torch.equal(k[:, i], k1[:, 0]) and torch.equal(v[:, i], vc1[:, 0])
    torch.cuda.synchronize()
    _lib.check_status()


def test_packed_inference_refuses_overlong_and_counts_launches():
    from allie_b200.data import UCITokenizer
    from allie_b200.models import initialize_model
    from allie_b200.models.engine import B200Engine
    from allie_b200.ops import _lib

    tok = UCITokenizer(max_length=256, vocab_size_multiple_of=128)
    eng = B200Engine(initialize_model(tok, "gpt2", use_control_token=True, use_regression_head=True, n_layer=2,
                                      n_embd=128, n_head=2, n_positions=64), "cuda")
    with pytest.raises(ValueError):
        eng.infer_last([np.arange(65)])
    before = _lib.LAUNCHES
    eng.infer_last([np.arange(64)])
    assert _lib.LAUNCHES - before == 1 + 2 * 7 + 1 + 3


def test_padding_token_inside_a_game():
    """A padding token among the moves takes no position and is not counted for the last index: such games
    go through the padded batch, with its results."""
    from allie_b200.data import Game, UCITokenizer
    from allie_b200.models import initialize_model
    from allie_b200.search.runner import EngineRunner

    torch.manual_seed(0)
    tok = UCITokenizer(max_length=64, vocab_size_multiple_of=128)
    model = initialize_model(tok, "gpt2", use_control_token=True, use_regression_head=True, n_layer=2, n_embd=128,
                             n_head=2, n_positions=64)
    game = lambda moves: Game("180+0", 1500, 1600, None, False, moves, [1] * len(moves))
    games = [game(["e2e4", tok.pad_token, "e7e5", "g1f3"]), game(["d2d4"]), game(["e2e4", "e7e5", tok.pad_token])]
    runner = EngineRunner(model, tok)
    got = runner.evaluate(games)
    batch = tok.pad_and_collate(games, return_labels=False)
    out = runner.engine.evaluate_batch(batch, with_loss=False)
    last = batch["attention_mask"].sum(-1).long() - 1
    assert last.tolist() == [5, 3, 4]
    for i, j in enumerate(last.tolist()):
        assert torch.equal(got.logits[i], out["logits"][i, j].float().cpu())
        assert float(got.value[i]) == float(out["value_logits"][i, j])


def test_many_short_games_in_dependent_launches():
    """240 rows (programmatic launches) of 120 games: more attention items than CTAs fit the GPU."""
    test_packed_last_positions_and_cache(4, 256, [2, 1, 3] * 40)


def test_buffers_of_many_rows_are_not_one_piece(monkeypatch):
    """One piece for a few rows only, and the same results either way."""
    from allie_b200.data import UCITokenizer
    from allie_b200.models import engine, initialize_model

    torch.manual_seed(0)
    tok = UCITokenizer(max_length=256, vocab_size_multiple_of=128)
    model = initialize_model(tok, "gpt2", use_control_token=True, use_regression_head=True, n_layer=2, n_embd=256,
                             n_head=4, n_positions=256)
    eng = engine.B200Engine(model, "cuda")
    rng = np.random.default_rng(2)
    empty, asked = torch.empty, []

    def counted(*shape, **kw):
        t = empty(*shape, **kw)
        if t.is_cuda:
            asked.append(t.nbytes)
        return t

    def run(games):
        asked.clear()
        with monkeypatch.context() as m:
            m.setattr(engine.torch, "empty", counted)
            return eng.infer_last(games), list(asked)

    few, many = ([rng.integers(0, 1968, size=n) for n in lens] for lens in ([90], [250] * 20))
    assert len(run(few)[1]) == 3                                   # the pass, logits, value and time
    want, sizes = run(many)
    assert max(sizes) <= 5000 * 8 * 256                            # the widest buffer of a row: 4 * 256 bf16
    monkeypatch.setattr(engine, "INFER_ONE_PIECE", 1 << 40)
    got, sizes = run(many)
    assert len(sizes) == 3 and all(torch.equal(a, b) for a, b in zip(want, got))
