"""Autoregressive decoding with a per-layer KV cache for the decoder-only Transformer models.

The reference regenerates by re-running the whole context window for every token (greedy window generation,
Tutorial/Cpp/Ml/Nlp/TutorialNlpCommon.h:145-177; no KV cache anywhere in Source/).  Here the prompt is processed once with
the tiled attention kernel while its rotated keys and values go into the cache, and every further token costs one GEMV-
shaped pass over the weights plus one read of the cache (csrc/kernels/decode.cu).  `Generate` returns exactly what the
full-window recomputation returns (the tests compare the two).
"""
from __future__ import annotations

import math
from typing import Optional

import torch

from ..core import fn_matrix as F
from ..core.matrix import OaMatrix
from ..ml import autograd as AG
from ..ml import fn_fused as FF
from ..ml.nn.layers import OaRmsNorm
from ..models.gpt import OaGptModel
from ..ops import kernels as K


class OaKvCache:
    """Keys and values of every layer: [layers][batch, heads, max_seq, head_dim] in the model's dtype."""

    def __init__(self, layers: int, batch: int, heads: int, max_seq: int, head_dim: int, dtype, device):
        self.K = [torch.zeros((batch, heads, max_seq, head_dim), dtype=dtype, device=device) for _ in range(layers)]
        self.V = [torch.zeros((batch, heads, max_seq, head_dim), dtype=dtype, device=device) for _ in range(layers)]
        self.Length, self.MaxSeq, self.Batch = 0, max_seq, batch

    def Bytes(self) -> int:
        return sum(t.numel() * t.element_size() for t in self.K + self.V)

    def Reset(self) -> None:
        self.Length = 0


class _GraphedStep:
    """One decode step captured in a CUDA graph.  The position lives on the device (`pos`, int32 [1]): RoPE, the cache
    append and the attention length read it inside their kernels and the captured function or what runs before it adds one, so
    replaying needs no host-side parameter.  `ids` is the static input, the captured function's result the static output."""

    def __init__(self, device, batch: int):
        self.pos = torch.zeros(1, dtype=torch.int32, device=device)
        self.ids = torch.zeros((batch, 1), dtype=torch.int32, device=device)
        self.graph: Optional[torch.cuda.CUDAGraph] = None
        self.out = None

    def run(self, ids: torch.Tensor, fn, weights=lambda: (), begin=None):
        """`weights()`: tensors that the step reads and never writes.  `begin(ids)`: work on the caller's ids that runs before the
        graph, which then leaves the position alone."""
        if begin is None or ids.dtype != torch.int32 or ids.device != self.ids.device or not ids.is_contiguous():
            self.ids.copy_(ids.reshape(self.ids.shape))
            ids = self.ids
        if begin is not None:
            begin(ids)
        if self.graph is None:
            try:
                self._record(fn, weights, begin is None)
            except BaseException:
                if begin is not None:
                    self.pos.sub_(1)                  # no step was made: the next one begins where this one did
                raise
        self.graph.replay()
        return self.out

    def _record(self, fn, weights, counts: bool):
        fn(self.ids)                                  # eager once: lazily created buffers (workspaces) exist before the capture
        if counts:
            self.pos.sub_(1)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        # a replay begins after everything before it on the stream, so whatever changed the weights has finished by then
        with torch.cuda.graph(g, capture_error_mode="thread_local"), K.weights_at_rest(weights()):
            self.out = fn(self.ids)
        self.graph = g


class OaGptDecoder:
    def __init__(self, model: OaGptModel, batch: int, max_seq: int, use_graph: bool = True):
        self.Model, self.Cfg = model, model.Cfg
        c = self.Cfg
        w = model.Embed.Weight.Tensor()
        self.Cache = OaKvCache(c.NLayers, batch, c.NHeads, max_seq, c.DModel // c.NHeads, w.dtype, w.device)
        self._graphed = _GraphedStep(w.device, batch) if use_graph and w.is_cuda and w.dtype == torch.bfloat16 else None
        self._pos_dev: Optional[torch.Tensor] = None      # set while a graphed step records / replays
        if self._graphed is not None:
            self._graphed.pos.fill_(-1)                   # of the newest token: a step begins by adding one
            self._step_x = torch.zeros((batch, c.DModel), dtype=w.dtype, device=w.device)
            self._step_xw = torch.zeros_like(self._step_x)
            self._step_sq = torch.zeros((1, batch), dtype=torch.float32, device=w.device)
            # Products carry the norms around them up to 32 rows: beyond, the rows' work at the end of a product outweighs the launches
            # between (prompt of 100 and 24 steps of two 7B-class blocks, ms, without / with: 1 row 6.30 / 5.99, 8 6.64 / 6.32, 16 7.16 / 7.07,
            # 24 7.86 / 7.75, 32 8.50 / 8.42, 48 10.01 / 10.10, 64 11.55 / 11.78).
            self._fused = batch <= 32 and self._fusable()

    def _fusable(self) -> bool:
        """Whether every block is RMS norms, packed projections without biases and a gated feed-forward: the step then runs as products
        of a few rows that also do the norms' work (False once one of them has turned out not to fit)."""
        m = self.Model
        if not m.Blocks or not isinstance(m.LnFinal, OaRmsNorm) or m.PosEmbed is not None:
            return False                              # without blocks there is no norm for the rows to begin with
        for b in m.Blocks:
            a = b.Attention
            if b.Moe is not None or b.FfnKind == "gelu" or not isinstance(b.LnAttn, OaRmsNorm) or a.RopeTheta <= 0:
                return False
            if (a.Plan is not None and not a.Plan.PackedQkv) or (b.Ffn.Plan is not None and not b.Ffn.Plan.GatedFfn):
                return False
            if any(lin.Bias for lin in (a.QProj, a.KProj, a.VProj, a.OutProj, b.Ffn.Gate, b.Ffn.Up, b.Ffn.Down)):
                return False
        return True

    def _fused_step(self) -> Optional[torch.Tensor]:
        """The graphed step as products that carry the norms: the one in front of a norm leaves its rows times the norm's weight and their
        squares, the one behind scales by the factor.  None: some product does not fit the kernel, and the step is the general one."""
        m, pd = self.Model, self._pos_dev
        x, xw, sq = self._step_x, self._step_xw, self._step_sq
        for i, b in enumerate(m.Blocks):
            a, f = b.Attention, b.Ffn
            D = a.DModel
            wqkv = FF.packed_view([a.QProj.Weight.Tensor(), a.KProj.Weight.Tensor(), a.VProj.Weight.Tensor()])
            wgu = FF.packed_view([f.Gate.Weight.Tensor(), f.Up.Weight.Tensor()])
            if wqkv is None or wgu is None:
                return None
            t = K.few_rows_step(xw, wqkv, squares=sq, eps=b.LnAttn.Eps)
            if t is None:
                return None
            K.rope_kv_append(t, self.Cache.K[i], self.Cache.V[i], 0, a.RopeTheta, pos_dev=pd)
            attn = K.decode_attn(t[:, :D], self.Cache.K[i], self.Cache.V[i], 1, pos_dev=pd)
            o = K.few_rows_step(attn, a.OutProj.Weight.Tensor(), residual=x, norm_w=f.Norm.Weight.Tensor())
            if o is None:
                return None
            x, xw, sq = o
            h = K.few_rows_step(xw, wgu, squares=sq, eps=f.Norm.Eps, gated=True)
            norm = m.Blocks[i + 1].LnAttn if i + 1 < len(m.Blocks) else m.LnFinal
            o = K.few_rows_step(h, f.Down.Weight.Tensor(), residual=x, norm_w=norm.Weight.Tensor()) if h is not None else None
            if o is None:
                return None
            x, xw, sq = o
        return K.few_rows_step(xw, m.Head.Weight.Tensor(), squares=sq, eps=m.LnFinal.Eps, bias=m.Head.Bias.Tensor() if m.Head.Bias else None)

    # ---- one block on new tokens
    def _block(self, i: int, x: OaMatrix, batch: int, s_new: int) -> OaMatrix:
        b = self.Model.Blocks[i]
        a = b.Attention
        H, hd, D = a.NumHeads, a.HeadDim, a.DModel
        pos0, pd = self.Cache.Length, self._pos_dev
        if pd is not None:
            pos0 = 0                                  # the device-resident position carries the offset
        h = b.LnAttn.Forward(x)
        qkv = a.ProjectQkv(h)
        t = qkv.Tensor()
        if s_new > 1:
            # prompt: tiled attention over the new tokens (rotates q and k in place), then cache the rotated k and v
            assert pos0 == 0, "prefill starts an empty cache"
            attn = F.FlashAttentionPacked(qkv, batch, s_new, H, hd, causal=True, rope_theta=a.RopeTheta)
            K.kv_append(t[:, D:2 * D], t[:, 2 * D:], self.Cache.K[i], self.Cache.V[i], batch, s_new, 0)
        else:
            if a.RopeTheta > 0:
                K.rope_kv_append(t, self.Cache.K[i], self.Cache.V[i], pos0, a.RopeTheta, pos_dev=pd)
            else:
                K.kv_append(t[:, D:2 * D], t[:, 2 * D:], self.Cache.K[i], self.Cache.V[i], batch, 1, pos0, pos_dev=pd)
            attn = OaMatrix(K.decode_attn(t[:, :D], self.Cache.K[i], self.Cache.V[i], pos0 + 1, pos_dev=pd))
        o = a.OutProj
        x = F.Linear(attn, o.Weight.Data, o.Bias.Data if o.Bias else None, residual=x)
        if b.Moe is not None:
            return b.Moe.Forward(x)
        if b.FfnKind == "gelu":
            hh = b.LnFfn.Forward(x)
            return FF.FfnGelu(hh, b.Ffn1.Weight.Data, b.Ffn1.Bias.Data if b.Ffn1.Bias else None, b.Ffn2.Weight.Data,
                              b.Ffn2.Bias.Data if b.Ffn2.Bias else None, residual=x)
        f = b.Ffn
        if s_new == 1 and FF.packed_view([f.Gate.Weight.Tensor(), f.Up.Weight.Tensor()]) is None:
            hh = f.Norm.Forward(x)                    # weights that do not lie side by side: two products rather than a joined copy
            return F.Linear(F.SiluMul(F.Linear(hh, f.Gate.Weight.Data), F.Linear(hh, f.Up.Weight.Data)), f.Down.Weight.Data, None, residual=x)
        return f.Forward(x)

    def _forward(self, ids: torch.Tensor, x: Optional[torch.Tensor] = None) -> torch.Tensor:
        """ids [B, s_new] int32 -> logits of the last new position [B, vocab]; the cache grows by s_new.  `x`: the rows of the ids,
        fetched already."""
        m = self.Model
        batch, s_new = ids.shape
        if self.Cache.Length + s_new > self.Cache.MaxSeq:
            raise ValueError("KV cache is full")
        with AG.OaGradNo():
            if x is not None:
                x = OaMatrix(x)
            elif m.PosEmbed is not None:
                pos = m.PosEmbed.Weight.Tensor()[self.Cache.Length:self.Cache.Length + s_new]
                x = F.Embedding(m.Embed.Weight.Data, OaMatrix(ids.contiguous()), OaMatrix(pos.contiguous()), s_new)
            else:
                x = F.Embedding(m.Embed.Weight.Data, OaMatrix(ids.contiguous()), None, s_new)
            for i in range(len(m.Blocks)):
                x = self._block(i, x, batch, s_new)
            self.Cache.Length += s_new
            last = x.Tensor().reshape(batch, s_new, -1)[:, -1].contiguous() if s_new > 1 else x.Tensor()
            return m.Head.Forward(m.LnFinal.Forward(OaMatrix(last))).Tensor()

    def Prefill(self, prompt: torch.Tensor) -> torch.Tensor:
        self.Cache.Reset()
        out = self._forward(prompt)
        if self._graphed is not None:
            self._graphed.pos.fill_(self.Cache.Length - 1)
        return out

    def _graph_body(self, ids: torch.Tensor) -> torch.Tensor:
        self._pos_dev = self._graphed.pos
        try:
            if self._fused:
                out = self._fused_step()
                if out is not None:
                    return out
                self._fused = False                     # found in the eager pass, before the recording; what it cached is written again
            length = self.Cache.Length
            out = self._forward(ids, self._step_x)
            self.Cache.Length = length                  # the host-side length advances once per Step, not per recording
            return out
        finally:
            self._pos_dev = None

    def Step(self, ids: torch.Tensor) -> torch.Tensor:
        """One token per sequence.  On CUDA (bf16, learned-position-free models) the step replays a captured graph; the
        returned logits tensor is then the graph's static output and is overwritten by the next Step."""
        g = self._graphed
        if g is None or self.Model.PosEmbed is not None or ids.numel() != g.ids.numel():
            return self._forward(ids.reshape(-1, 1))
        if self.Cache.Length + 1 > self.Cache.MaxSeq:
            raise ValueError("KV cache is full")
        out = g.run(ids, self._graph_body, lambda: [p.Data.Tensor() for p in self.Model.AllParameterPtrs()],
                    lambda new: K.decode_begin(self.Model.Embed.Weight.Tensor(), new, self._step_x, self._graphed.pos,
                                               self.Model.Blocks[0].LnAttn.Weight.Tensor() if self._fused else None,
                                               self._step_xw if self._fused else None, self._step_sq if self._fused else None))
        self.Cache.Length += 1
        return out

    def Generate(self, prompt: torch.Tensor, new_tokens: int) -> torch.Tensor:
        """Greedy decoding: prompt [B, S] int32 -> [B, S + new_tokens]."""
        out = [prompt]
        logits = self.Prefill(prompt)
        for _ in range(new_tokens):
            nxt = logits.float().argmax(-1).to(torch.int32).reshape(-1, 1)
            out.append(nxt)
            if len(out) - 1 < new_tokens:
                logits = self.Step(nxt)
        return torch.cat(out, 1)
