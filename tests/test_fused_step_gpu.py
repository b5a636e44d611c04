"""A replayed decoding step whose products carry the RMS norms and the gate: against the general step and a model in 64 bits, and where it has to
give way to the general one."""
import pytest
import torch

from oa_b200.core import fn_matrix as F
from oa_b200.core.matrix import OaMatrix
from oa_b200.core.types import OaScalarType
from oa_b200.ml.nn.layers import OaLinear
from oa_b200.ml.optim import OaAdamW
from oa_b200.models.gpt import OaGptConfig, OaGptModel
from oa_b200.ops import kernels as K
from oa_b200.runtime.engine import OaInitComputeEngine
from oa_b200.serve.decoder import OaGptDecoder

pytestmark = pytest.mark.gpu
THETA = 10000.0


@pytest.fixture(autouse=True)
def _bf16():
    OaInitComputeEngine()
    prev = F.GetWeightDtype()
    F.SetWeightDtype(OaScalarType.BFloat16)
    yield
    F.SetWeightDtype(prev)


def _model(dim, heads, ff, vocab, layers=3, head_bias=False, seed=0):
    model = OaGptModel(OaGptConfig(vocab, dim, layers, heads, ff, 64, "rms", "swiglu", THETA, False, 1e-5, dim ** -0.5))
    if head_bias:
        model.Head = model.RegisterModule("head", OaLinear(dim, vocab, True, dim ** -0.5))
    model.opt = OaAdamW(model.AllParameterPtrs(), 1e-3)       # weights side by side, as a trained model has them
    model.opt.ZeroGrad()
    g = torch.Generator(device="cuda").manual_seed(seed)
    norms = [n for b in model.Blocks for n in (b.LnAttn, b.Ffn.Norm)] + [model.LnFinal]
    for i, n in enumerate(norms):                             # no two alike, neither in weight nor in eps
        n.Weight.Tensor().copy_(1 + 0.4 * torch.randn(dim, device="cuda", generator=g))
        n.Eps = 1e-3 * 3 ** (i % 5)
    if head_bias:
        model.Head.Bias.Tensor().copy_(torch.randn(vocab, device="cuda", generator=g))
    return model


def _reference(model, ids):
    """Logits of the last position in 64 bits, from the model's bf16 weights."""
    w = lambda p: p.Tensor().double()
    rms = lambda x, n: x * torch.rsqrt((x * x).mean(-1, keepdim=True) + n.Eps) * w(n.Weight)
    B, S = ids.shape
    x = w(model.Embed.Weight)[ids.long()]
    D, H = x.shape[-1], model.Cfg.NHeads
    hd = D // H
    ang = torch.arange(S, device="cuda").double()[:, None] * THETA ** (-torch.arange(hd // 2, device="cuda").double() * 2 / hd)
    cos, sin = ang.cos(), ang.sin()

    def rope(t):                                              # [B, H, S, hd]
        a, b = t[..., :hd // 2], t[..., hd // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    split = lambda t: t.reshape(B, S, H, hd).transpose(1, 2)
    mask = torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1)
    for b in model.Blocks:
        a, f = b.Attention, b.Ffn
        h = rms(x, b.LnAttn)
        q, k, v = (split(h @ w(lin.Weight).t()) for lin in (a.QProj, a.KProj, a.VProj))
        s = (rope(q) @ rope(k).transpose(-1, -2) / hd ** 0.5).masked_fill(mask, float("-inf"))
        x = x + (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(B, S, D) @ w(a.OutProj.Weight).t()
        h = rms(x, f.Norm)
        x = x + (torch.nn.functional.silu(h @ w(f.Gate.Weight).t()) * (h @ w(f.Up.Weight).t())) @ w(f.Down.Weight).t()
    out = rms(x[:, -1], model.LnFinal) @ w(model.Head.Weight).t()
    return out + w(model.Head.Bias) if model.Head.Bias else out


def _follow(model, batch, fused, prompt=9, steps=5):
    """Graphed, general and 64-bit logits step by step; `fused`: whether the products carry the norms once the graph is there."""
    ids = torch.randint(0, model.Cfg.Vocab, (batch, prompt + steps), device="cuda", dtype=torch.int32)
    graphed, general = OaGptDecoder(model, batch, 40), OaGptDecoder(model, batch, 40, use_graph=False)
    graphed.Prefill(ids[:, :prompt].contiguous())
    general.Prefill(ids[:, :prompt].contiguous())
    for i in range(prompt, prompt + steps):
        new = ids[:, i:i + 1].contiguous()
        got, plain, want = graphed.Step(new).double(), general.Step(new).double(), _reference(model, ids[:, :i + 1])
        e = lambda t: float((t - want).norm() / want.norm())
        # a dozen roundings to bf16 a layer either way, those between products and norms fewer in the joined step
        assert e(plain) <= 2e-2 and e(got) <= 1.2 * e(plain) + 1e-3, (i, e(got), e(plain))
    assert graphed._fused == fused
    for a, b in zip(graphed.Cache.K + graphed.Cache.V, general.Cache.K + general.Cache.V):
        assert float((a.double() - b.double()).norm() / b.double().norm()) <= 2e-2
    torch.cuda.synchronize()
    K.check_status()


@pytest.mark.parametrize("batch", [1, 3, 17, 32, 33])
@pytest.mark.parametrize("dim,heads,ff", [(512, 4, 1024), (1024, 16, 640)])
def test_joined_step(dim, heads, ff, batch):
    _follow(_model(dim, heads, ff, 1000, seed=batch), batch, fused=batch <= 32)


def test_head_with_a_bias():
    _follow(_model(512, 8, 512, 520, head_bias=True), 2, fused=True)


@pytest.mark.parametrize("dim,heads,ff,vocab", [(256, 4, 1024, 1000), (512, 8, 128, 1000), (512, 8, 512, 128)])
def test_gives_way(dim, heads, ff, vocab):
    """A product that the few-row kernel leaves to others, the first of a step, one inside a layer or the head alone: what the layers before it have
    written to the cache is written again."""
    _follow(_model(dim, heads, ff, vocab), 2, fused=False)


def test_weight_in_another_order():
    """A head whose weight is a transposed matrix: its product takes a copy, as in every other path."""
    model = _model(512, 8, 512, 1000)
    t = model.Head.Weight.Tensor()
    model.Head.Weight.Data = OaMatrix(t.t().contiguous().t())
    assert model.Head.Weight.Tensor().stride(1) != 1
    _follow(model, 2, fused=False)
