"""KV-cached, batched leaf evaluator for MCTS on the sm_100a engine.

Every search tree owns a slice of a per-layer key/value cache: slots ``[0, prefix_len)`` hold the
game so far (filled once per move by a batched prefill), the following slots hold one entry per
evaluated tree node.  A search step evaluates one leaf per tree: the leaf's move token goes through
the network as a single new position whose attention reads the prefix slots plus the slots of the
leaf's ancestors (an index list produced by the C++ search), so a leaf costs one token of compute
instead of a re-encode of the whole game (the reference re-encodes, ``src/evaluation/decode.py:356-360``).
The step is a fixed sequence of kernels over static buffers and is replayed as a CUDA graph.
"""
from __future__ import annotations

import os
from ctypes import c_float, c_int, c_longlong

import numpy as np
import torch

from ..ops import _lib, kernels as K
from ..ops._lib import ptr, stream_ptr
from ..ops.gemm import gemm, num_sms
from ..ops.infer import results_to_host


class KVLeafEvaluator:
    FEW_TREES = 16

    def __init__(self, engine, n_trees: int, max_prefix: int = 320, max_nodes: int = 512,
                 anc_max: int = 128, legal_max: int = 224, use_graph: bool = True):
        self.eng = engine
        cfg = engine.cfg
        self.n, self.S = n_trees, max_prefix + max_nodes
        self.max_prefix, self.anc_max, self.legal_max = max_prefix, anc_max, legal_max
        dev, d, F, V, L = engine.device, cfg.n_embd, cfg.ffn_dim, cfg.vocab_size, cfg.n_layer
        bf, f32, i32 = torch.bfloat16, torch.float32, torch.int32
        self.kc = torch.zeros(L, n_trees, self.S, d, dtype=bf, device=dev)
        self.vc = torch.zeros(L, n_trees, self.S, d, dtype=bf, device=dev)
        n = n_trees
        # request block: one int32 buffer, one host->device copy per step
        self.off = {}
        o = 0
        for name, width in (("active", 1), ("tok", 1), ("pos", 1), ("slot", 1), ("prefix_len", 1),
                            ("n_anc", 1), ("n_legal", 1), ("anc", anc_max), ("legal", legal_max)):
            self.off[name] = (o, width)
            o += n * width
        self.req_host = torch.zeros(o, dtype=i32, pin_memory=True)
        self.req_dev = torch.zeros(o, dtype=i32, device=dev)
        self.out_stride = legal_max + 4
        # result rows, and the status word behind them (written by the step's last kernel)
        self.out_flat = torch.zeros(n * self.out_stride + 1, dtype=f32, device=dev)
        self.out_flat_host = torch.zeros(n * self.out_stride + 1, dtype=f32, pin_memory=True)
        self.out_host = self.out_flat_host[:-1].view(n, self.out_stride)
        self.status_host = self.out_flat_host[-1:].view(i32).numpy()
        e = lambda *s, dt=bf: torch.empty(*s, dtype=dt, device=dev)
        self.x = [e(n, d, dt=f32), e(n, d, dt=f32)]
        self.ln, self.qkv, self.att = e(n, d), e(n, 3 * d), e(n, d)
        self.act, self.h, self.logits = e(n, F), e(n, d), e(n, V)
        self.stat = [e(n, dt=f32) for _ in range(2)]
        self.value, self.time = e(n, dt=f32), e(n, dt=f32)
        self.resign_id = 1992
        # a handful of trees: all layers in one kernel (csrc/decode_few.cu), which reads the layers'
        # addresses from this table and keeps its accumulators in this scratch
        self.few = n_trees <= self.FEW_TREES and engine.dense
        self.few_max_wait = 0           # clock cycles at a meeting of that kernel's CTAs; 0: about a second
        if self.few:
            addr = lambda t: 0 if t is None else t.data_ptr()
            table = [[addr(Ly[k][0]) for k in ("ln1_w", "ln1_b", "ln2_w", "ln2_b", "qkv_b", "o_b", "fc_b", "pr_b")]
                     + [addr(Ly[k][1]) for k in ("qkv_w", "o_w", "fc_w", "pr_w")] + [addr(self.kc[l]), addr(self.vc[l])]
                     for l, Ly in enumerate(engine.layers)]
            self.layer_table = torch.tensor(table, dtype=torch.int64, device=dev)
            self.few_work = torch.zeros(256 + n * (3 * d + F), dtype=f32, device=dev)
        self.graph = None
        self.use_graph = use_graph
        self.steps = 0

    def view(self, t: torch.Tensor, name: str) -> torch.Tensor:
        o, w = self.off[name]
        v = t[o:o + self.n * w]
        return v.view(self.n, w) if w > 1 else v

    # ------------------------------------------------------------------ prefill
    @torch.no_grad()
    def prefill(self, token_rows: list[np.ndarray]):
        """Runs the prompts (one per tree, raw token ids incl. ELO pseudo-ids) through the network,
        fills cache slots [0, len) of every tree and returns host tensors
        (last-position logits [n, V] fp32, value [n], time [n])."""
        eng, n = self.eng, self.n
        assert len(token_rows) == n
        lens = [len(r) for r in token_rows]
        assert max(lens) <= self.max_prefix
        if eng.dense and min(lens) > 0:
            d = eng.cfg.head_dim
            shape = (eng.cfg.n_layer, n, eng.cfg.n_head, self.S, d)
            logits, value, time = eng.infer_last(token_rows, (self.kc.view(shape), self.vc.view(shape)))
        else:
            logits, value, time = self._prefill_padded(token_rows, lens)
        out = results_to_host(logits, value, time)
        self.view(self.req_host, "prefix_len").copy_(torch.tensor(lens, dtype=torch.int32))
        return out

    def _prefill_padded(self, token_rows, lens):
        """The same for models with experts, whose buffers are laid out for a fixed number of rows."""
        eng, n, Lp = self.eng, self.n, max(lens)
        pad = eng.cfg.pad_token_id if eng.cfg.pad_token_id is not None else 0
        ids = np.full((n, Lp), pad, dtype=np.int64)
        for i, r in enumerate(token_rows):
            ids[i, :len(r)] = r
        B, T = eng.load_batch({"input_ids": torch.from_numpy(ids)}, False)
        len_dev = torch.tensor(lens, dtype=torch.int32, device=eng.device)
        d = eng.cfg.n_embd

        def hook(l, qkv):
            rc = _lib.cuda().ab_kv_store(ptr(qkv), ptr(self.kc[l]), ptr(self.vc[l]), ptr(len_dev), c_int(n),
                                         c_int(Lp), c_int(self.S), c_int(d), c_int(eng.cfg.head_dim), stream_ptr())
            assert rc == 0
            _lib.count_launches(1)

        buf = eng.forward(B, T, False, 0, False, False, kv_hook=hook)
        rows = torch.arange(n, device=eng.device) * Lp + (len_dev.long() - 1)
        return (buf["logits"][rows], buf["value"][rows] if eng.reg is not None else None,
                buf["time"][rows] if eng.reg is not None else None)

    # --------------------------------------------------------------------- step
    def _launch_step(self) -> None:
        eng, cfg, n = self.eng, self.eng.cfg, self.n
        rd = self.req_dev
        V, eps = cfg.vocab_size, cfg.layer_norm_epsilon
        lib = _lib.cuda()
        K.embed_fwd(self.view(rd, "tok"), self.view(rd, "pos"), eng.wte[0], eng.wpe[0], eng.ctrl_w[0],
                    self.x[0], V, 0, 0, 0.0)
        x = self.x[0]
        scale = 1.0 / cfg.head_dim ** 0.5
        # the kernels of the step are programmatic dependents of the kernel before them: a GEMM's
        # set-up and first ring of weight tiles, the attention kernel's prompt-slot chunks and every
        # launch overlap the previous kernel (ALLIE_DECODE_PDL=0 turns it off)
        pdl = os.environ.get("ALLIE_DECODE_PDL", "1") != "0"
        few = self.few and self._launch_few(x)
        for l, Ly in enumerate(eng.layers if not few else ()):
            K.layernorm_fwd(x, Ly["ln1_w"][0], Ly["ln1_b"][0], self.ln, self.stat[0], self.stat[1], eps, eng.rms,
                            dependent=pdl, weights_ready=True)
            gemm(self.ln, Ly["qkv_w"][1], b_mn=True, out=self.qkv, bias=Ly["qkv_b"][0], dependent=pdl,
                 then=Ly["o_w"][1])
            rc = lib.ab_decode_attn(ptr(self.qkv), ptr(self.kc[l]), ptr(self.vc[l]), ptr(self.view(rd, "active")),
                                    ptr(self.view(rd, "slot")), ptr(self.view(rd, "prefix_len")),
                                    ptr(self.view(rd, "anc")), c_int(self.anc_max), ptr(self.view(rd, "n_anc")),
                                    ptr(self.att), c_int(n), c_int(cfg.n_head), c_int(cfg.head_dim),
                                    c_int(self.S), c_float(scale), c_int(int(pdl)), ptr(_lib.status_word()),
                                    stream_ptr())
            assert rc == 0
            _lib.count_launches(1)
            # residual updates in place: with a few hundred rows they run as split-K reduce-adds
            gemm(self.att, Ly["o_w"][1], b_mn=True, out=x, bias=Ly["o_b"][0], resid=x, dependent=pdl,
                 then=Ly["fc_w"][1])
            K.layernorm_fwd(x, Ly["ln2_w"][0], Ly["ln2_b"][0], self.ln, self.stat[0], self.stat[1], eps, eng.rms,
                            dependent=pdl, weights_ready=True)
            gemm(self.ln, Ly["fc_w"][1], b_mn=True, out=self.act, bias=Ly["fc_b"][0], act=3, dependent=pdl,
                 then=Ly["pr_w"][1])
            gemm(self.act, Ly["pr_w"][1], b_mn=True, out=x, bias=Ly["pr_b"][0], resid=x, dependent=pdl,
                 then=eng.layers[l + 1]["qkv_w"][1] if l + 1 < cfg.n_layer else eng.wte[1])
        K.layernorm_fwd(x, eng.lnf_w[0], eng.lnf_b[0], self.h, self.stat[0], self.stat[1], eps, eng.rms,
                        dependent=pdl, weights_ready=True)
        gemm(self.h, eng.wte[1], b_mn=False, out=self.logits, dependent=pdl)
        has_heads = eng.reg is not None
        if has_heads and pdl:
            K.heads_fwd_ahead(self.h, eng.wv[0], eng.bv[0], eng.wt[0], eng.bt[0], self.value, self.time)
        elif has_heads:
            K.heads_fwd(self.h, eng.wv[0], eng.bv[0], eng.wt[0], eng.bt[0], None, None, eng.counts, 0.0, 0.0,
                        self.value, self.time, None, None, None)
        rc = lib.ab_policy_epilogue(ptr(self.logits), c_longlong(self.logits.stride(0)),
                                    ptr(self.view(rd, "active")), ptr(self.view(rd, "legal")),
                                    c_int(self.legal_max), ptr(self.view(rd, "n_legal")),
                                    ptr(self.value if has_heads else None), ptr(self.time if has_heads else None),
                                    c_int(self.resign_id), c_float(1.0), ptr(self.out_flat),
                                    c_int(self.out_stride), c_int(n), ptr(_lib.status_word()), c_int(int(pdl)),
                                    stream_ptr())
        assert rc == 0
        _lib.count_launches(1)

    def _launch_few(self, x) -> bool:
        """All layers of the step as one kernel; False (nothing launched) for shapes it does not take and
        where its CTAs cannot all be resident."""
        cfg, rd = self.eng.cfg, self.req_dev
        rc = _lib.cuda().ab_decode_few(
            ptr(self.layer_table), c_int(cfg.n_layer), c_int(self.n), c_int(cfg.n_embd), c_int(cfg.n_head),
            c_int(cfg.ffn_dim), c_int(self.S), c_int(int(self.eng.rms)), c_float(cfg.layer_norm_epsilon), ptr(x),
            ptr(self.att), ptr(self.view(rd, "active")), ptr(self.view(rd, "slot")), ptr(self.view(rd, "prefix_len")),
            ptr(self.view(rd, "anc")), c_int(self.anc_max), ptr(self.view(rd, "n_anc")), ptr(self.few_work),
            c_int(num_sms()), c_longlong(self.few_max_wait), ptr(_lib.status_word()), stream_ptr())
        if rc < 0:
            raise RuntimeError(f"ab_decode_few failed with code {rc}")
        _lib.count_launches(int(rc == 0))
        return rc == 0

    @torch.no_grad()
    def step(self) -> np.ndarray:
        """Evaluates the requests currently in ``req_host``; returns the packed result rows
        (host, [n, legal_max + 4]: priors..., value, time, resign logit, best legal logit).  Raises if a
        wait of one of the step's kernels ran out."""
        self.req_dev.copy_(self.req_host, non_blocking=True)
        if self.use_graph:
            if self.graph is None:
                self._launch_step()                      # warm-up outside capture (first-launch set-up)
                torch.cuda.synchronize()
                g = torch.cuda.CUDAGraph()
                before = _lib.LAUNCHES
                with torch.cuda.graph(g):
                    self._launch_step()
                self.graph, self.graph_launches = g, _lib.LAUNCHES - before
                _lib.count_launches(-self.graph_launches)     # nothing ran yet: counted per replay
            self.graph.replay()
            _lib.count_launches(self.graph_launches)
        else:
            self._launch_step()
        self.out_flat_host.copy_(self.out_flat, non_blocking=True)
        torch.cuda.current_stream().synchronize()
        _lib.raise_on_status(int(self.status_host[0]))
        self.steps += 1
        return self.out_host.numpy()
