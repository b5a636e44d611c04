"""The work whose speed is watched: what programs written against this framework spend their time on.

Training of the language-model layers (attention, MLP, norm, loss head, sparse MoE, Mamba-3 mixer, GRU), one captured
training step of the small fp32 character model, prompt attention, and generation with a KV cache.  Each case goes through
the entry points a program calls; sizes are those of the configurations in oa_b200/models and of the benchmarks, with ragged
ones beside them.  `exact` states the same mathematics in 64 bits with plain torch.
"""
import math

import torch

from oa_b200.core import fn_matrix as F
from oa_b200.core.matrix import OaMatrix
from oa_b200.core.types import OaScalarType
from oa_b200.ml import fn_fused, fn_loss
from oa_b200.ml.autograd import OaGradientTape
from oa_b200.ml.nn.layers import OaMultiHeadAttention
from oa_b200.ml.nn.mamba3 import OaMamba3Module
from oa_b200.ml.nn.moe import OaMoE
from oa_b200.ml.nn.recurrent import OaGru
from oa_b200.ml.optim import OaAdamW
from oa_b200.ml.training import OaTrainingProgram
from oa_b200.models.gpt import OaGptConfig, OaGptModel
from oa_b200.runtime.engine import OaInitComputeEngine
from oa_b200.serve.decoder import OaGptDecoder

DEV = "cuda"
BF, F32, F64 = torch.bfloat16, torch.float32, torch.float64
ROPE_THETA = 10000.0


def listed():
    return [
        # one attention layer of the 24 x 1024 dense model in training: packed projection, RoPE, attention, output projection
        {"name": "attention_train_hd64", "kind": "attention", "batch": 8, "seq": 2048, "heads": 16, "hd": 64},
        # the attention operation alone, head dim 128, in training on a ragged sequence (fine-tuning batches end anywhere)
        {"name": "flash_train_hd128_ragged", "kind": "flash", "batch": 2, "seq": 3001, "heads": 16, "hd": 128, "train": True},
        # prompt attention of the 7B-class model
        {"name": "flash_prefill_hd128", "kind": "flash", "batch": 1, "seq": 4096, "heads": 32, "hd": 128, "train": False},
        # the GELU feed-forward of the dense model in training
        {"name": "mlp_train", "kind": "mlp", "rows": 16384, "dim": 1024, "ff": 4096},
        # its RMSNorm, forward and backward
        {"name": "norm_train", "kind": "norm", "rows": 16384, "dim": 1024},
        # its loss: mean cross-entropy of [tokens, vocabulary] logits and the gradient of the logits
        {"name": "loss_train", "kind": "loss", "rows": 16384, "vocab": 32000},
        # one sparse layer of the mixture-of-experts model in training, every expert on this GPU
        {"name": "moe_train", "kind": "moe", "tokens": 8192, "dim": 2048, "ff": 1408, "experts": 64, "topk": 2, "shared": 1},
        # one Mamba-3 mixer of the 32 x 1536 model in training, convolution and learned decay included
        {"name": "mamba3_train", "kind": "mamba3", "batch": 2, "seq": 4096, "dim": 1536},
        # batched generation with a KV cache at the 7B-class width (two blocks of it): prompt, then token by token
        {"name": "generate_b32", "kind": "generate", "batch": 32, "prompt": 256, "steps": 48},
        # the same for one conversation
        {"name": "generate_b1", "kind": "generate", "batch": 1, "prompt": 100, "steps": 32},
        # the character-level fp32 model: forward and backward of one micro-step, replayed as a captured program
        {"name": "char_lm_step", "kind": "char_lm", "batch": 16, "seq": 128},
        # a recurrent layer of the small fp32 language models in training
        {"name": "gru_train", "kind": "gru", "batch": 64, "seq": 128, "input": 64, "hidden": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "flash", "flash", "mlp", "norm", "loss", "moe", "mamba3", "generate", "char_lm", "gru"])
    if kind == "attention":
        hd = rng.choice([64, 128])
        batch, seq = rng.randint(1, 8), _log(rng, 64, 2048)
        return {"kind": kind, "batch": batch, "seq": max(8, seq // 8 * 8), "heads": rng.choice([4, 8, 16]) * 64 // hd, "hd": hd}
    if kind == "flash":
        hd, seq = rng.choice([64, 128]), _log(rng, 48, 6000)
        heads = rng.randint(2, 32)
        return {"kind": kind, "batch": max(1, min(8, int(2e5 / (heads * seq)))), "seq": seq, "heads": heads, "hd": hd,
                "train": rng.random() < 0.6}
    if kind == "mlp":
        dim = rng.choice([256, 512, 1024, 2048])
        return {"kind": kind, "rows": max(8, _log(rng, 64, 16384 * 1024 // dim) // 8 * 8), "dim": dim, "ff": 4 * dim}
    if kind == "norm":
        dim = rng.choice([128, 512, 1024, 1536, 2048, 4096])
        return {"kind": kind, "rows": _log(rng, 17, 32768 * 1024 // dim), "dim": dim}
    if kind == "loss":
        vocab = rng.choice([256, 4096, 32000, 50264])
        return {"kind": kind, "rows": _log(rng, 33, min(32768, 16384 * 32000 // vocab)), "vocab": vocab}
    if kind == "moe":
        return {"kind": kind, "tokens": max(64, _log(rng, 64, 8192) // 8 * 8), "dim": rng.choice([512, 1024, 2048]),
                "ff": rng.choice([512, 1408]), "experts": rng.choice([8, 16, 64]), "topk": 2, "shared": rng.randint(0, 1)}
    if kind == "mamba3":
        return {"kind": kind, "batch": rng.randint(1, 2), "seq": 128 * rng.randint(2, 32), "dim": rng.choice([512, 1024, 1536])}
    if kind == "generate":
        return {"kind": kind, "batch": rng.choice([1, 3, 8, 16, 32, 40]), "prompt": _log(rng, 16, 256), "steps": rng.randint(4, 24)}
    if kind == "char_lm":
        return {"kind": kind, "batch": rng.randint(1, 16), "seq": rng.randint(16, 128)}
    return {"kind": kind, "batch": rng.randint(1, 64), "seq": _log(rng, 8, 128), "input": 8 * rng.randint(2, 16),
            "hidden": 8 * rng.randint(4, 16)}


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 7919 + salt) & 0x7FFFFFFF)


def _randn(g, *shape, std=1.0, dtype=BF):
    return torch.randn(shape, generator=g, device=DEV, dtype=F32).mul_(std).to(dtype)


def _ints(g, hi, *shape):
    return torch.randint(0, hi, shape, generator=g, device=DEV, dtype=torch.int32)


def _engine(dtype):
    OaInitComputeEngine()
    F.SetWeightDtype(OaScalarType.Float32 if dtype == F32 else OaScalarType.BFloat16)


def _trainable(module):
    """The module's optimizer, whose arenas hold weights and gradients, as a training program keeps it."""
    for p in module.AllParameterPtrs():
        p.Data.SetRequiresGrad(True)
    opt = OaAdamW(module.AllParameterPtrs(), 1e-4)
    opt.ZeroGrad()
    return opt


def _leaf(t):
    m = OaMatrix(t)
    m.SetRequiresGrad(True)
    return m


def _inputs(case, seed):
    """The tensors a case starts from, by name, from the seed alone."""
    g = _gen(seed)
    k = case["kind"]
    if k == "attention":
        d, rows = case["heads"] * case["hd"], case["batch"] * case["seq"]
        return {"x": _randn(g, rows, d), "wqkv": _randn(g, 3 * d, d, std=1.0 / math.sqrt(d)), "wo": _randn(g, d, d, std=0.02),
                "dy": _randn(g, rows, d)}
    if k == "flash":
        d, rows = case["heads"] * case["hd"], case["batch"] * case["seq"]
        return {"qkv": _randn(g, rows, 3 * d), "do": _randn(g, rows, d)}
    if k == "mlp":
        r, d, f = case["rows"], case["dim"], case["ff"]
        return {"x": _randn(g, r, d), "w1": _randn(g, f, d, std=1.0 / math.sqrt(d)), "w2": _randn(g, d, f, std=1.0 / math.sqrt(f)),
                "dy": _randn(g, r, d)}
    if k == "norm":
        return {"x": _randn(g, case["rows"], case["dim"]), "w": 1.0 + _randn(g, case["dim"], std=0.1), "dy": _randn(g, case["rows"], case["dim"])}
    if k == "loss":
        return {"logits": _randn(g, case["rows"], case["vocab"], std=2.0), "target": _ints(g, case["vocab"], case["rows"])}
    if k == "moe":
        t, d, f, e = case["tokens"], case["dim"], case["ff"], case["experts"]
        router = _randn(g, e, d, std=0.02)
        # a trained router is sure of its choice: each token leans towards its experts, so that rounding decides no route
        pick = torch.argsort(torch.rand(t, e, generator=g, device=DEV), dim=1)[:, :case["topk"]]
        lean = torch.zeros(t, e, device=DEV)
        for j in range(case["topk"]):
            lean.scatter_(1, pick[:, j:j + 1], 10.0 - 1.5 * j)
        x = torch.randn(t, d, generator=g, device=DEV)
        rf = router.float()
        x = x + lean @ (rf / (rf * rf).sum(1, keepdim=True))
        out = {"x": x.to(BF), "router": router, "gu": _randn(g, e, 2 * f, d, std=0.02), "down": _randn(g, e, d, f, std=0.02), "dy": _randn(g, t, d)}
        if case["shared"]:
            out["sgu"], out["sdown"] = _randn(g, 2 * f, d, std=0.02), _randn(g, d, f, std=0.02)
        return out
    if k == "mamba3":
        d, rows = case["dim"], case["batch"] * case["seq"]
        di, n = 2 * d, 128
        h, a = di // 64, 32
        width = 2 * di + 2 * n + 3 * h + a
        u = torch.rand(h, generator=g, device=DEV)
        dt = torch.exp(torch.rand(h, generator=g, device=DEV) * math.log(100.0) + math.log(1e-3))
        taps = torch.zeros(4, di + 2 * n, device=DEV)
        taps[0] = 1.0
        return {"x": _randn(g, rows, d), "in": _randn(g, width, d, std=math.sqrt(2.0 / (width + d))), "out": _randn(g, d, di, std=math.sqrt(2.0 / (d + di))),
                "dt_bias": (dt + torch.log(-torch.expm1(-dt))).reshape(1, h), "bb": 1.0 + _randn(g, h, n, std=0.1, dtype=F32),
                "cb": 1.0 + _randn(g, h, n, std=0.1, dtype=F32), "skip": _randn(g, h, std=0.1, dtype=F32),
                "norm": 1.0 + _randn(g, h, 64, std=0.1, dtype=F32), "conv": taps + _randn(g, 4, di + 2 * n, std=0.1, dtype=F32),
                "a_log": torch.log(1.0 + 15.0 * u).reshape(1, h), "dy": _randn(g, rows, d)}
    if k == "generate":
        return {"ids": _ints(g, 32000, case["batch"], case["prompt"] + case["steps"])}
    if k == "char_lm":
        return {"ids": _ints(g, 256, case["batch"], case["seq"]), "target": _ints(g, 256, case["batch"] * case["seq"])}
    b, s, i, h = case["batch"], case["seq"], case["input"], case["hidden"]
    r = 1.0 / math.sqrt(h)
    return {"x": _randn(g, b, s, i, dtype=F32), "wih": _randn(g, 3 * h, i, std=r, dtype=F32), "whh": _randn(g, 3 * h, h, std=r, dtype=F32),
            "bih": _randn(g, 3 * h, std=0.1, dtype=F32), "bhh": _randn(g, 3 * h, std=0.1, dtype=F32), "dy": _randn(g, b, s, h, dtype=F32)}


def _fill(param, value):
    param.Data.Tensor().copy_(value.reshape(param.Data.Tensor().shape))


def _gpt_weights(cfg, seed):
    """Random weights of a model, block by block: {"embed", "head", "blocks": [{...}], ...}."""
    g = _gen(seed, 1)
    dt = F32 if cfg.Norm == "layer" else BF
    d, f, std = cfg.DModel, cfg.DFf, 1.0 / math.sqrt(cfg.DModel)
    w = {"embed": _randn(g, cfg.Vocab, d, dtype=dt), "head": _randn(g, cfg.Vocab, d, std=std, dtype=dt), "norm": 1.0 + _randn(g, d, std=0.1, dtype=dt)}
    if cfg.Norm == "layer":
        w["pos"], w["normb"], w["headb"] = _randn(g, cfg.SeqLen, d, std=0.1, dtype=dt), _randn(g, d, std=0.1, dtype=dt), _randn(g, cfg.Vocab, std=0.1, dtype=dt)
    w["blocks"] = []
    for _ in range(cfg.NLayers):
        b = {"qkv": _randn(g, 3 * d, d, std=std, dtype=dt), "o": _randn(g, d, d, std=0.5 * std, dtype=dt),
             "n1": 1.0 + _randn(g, d, std=0.1, dtype=dt), "n2": 1.0 + _randn(g, d, std=0.1, dtype=dt)}
        if cfg.Ffn == "gelu":
            b.update(f1=_randn(g, f, d, std=std, dtype=dt), f2=_randn(g, d, f, std=0.5 / math.sqrt(f), dtype=dt))
            for nm, n in (("qkvb", 3 * d), ("ob", d), ("n1b", d), ("n2b", d), ("f1b", f), ("f2b", d)):
                b[nm] = _randn(g, n, std=0.1, dtype=dt)
        else:
            b.update(gu=_randn(g, 2 * f, d, std=std, dtype=dt), down=_randn(g, d, f, std=0.5 / math.sqrt(f), dtype=dt))
        w["blocks"].append(b)
    return w


def _load_gpt(model, cfg, w):
    _fill(model.Embed.Weight, w["embed"])
    _fill(model.Head.Weight, w["head"])
    _fill(model.LnFinal.Weight, w["norm"])
    d, f = cfg.DModel, cfg.DFf
    if cfg.Norm == "layer":
        _fill(model.PosEmbed.Weight, w["pos"])
        _fill(model.LnFinal.Bias, w["normb"])
        _fill(model.Head.Bias, w["headb"])
    for blk, b in zip(model.Blocks, w["blocks"]):
        a = blk.Attention
        for i, lin in enumerate((a.QProj, a.KProj, a.VProj)):
            _fill(lin.Weight, b["qkv"][i * d:(i + 1) * d])
            if lin.Bias is not None:
                _fill(lin.Bias, b["qkvb"][i * d:(i + 1) * d])
        _fill(a.OutProj.Weight, b["o"])
        _fill(blk.LnAttn.Weight, b["n1"])
        if cfg.Ffn == "gelu":
            _fill(a.OutProj.Bias, b["ob"])
            _fill(blk.LnAttn.Bias, b["n1b"])
            _fill(blk.LnFfn.Weight, b["n2"])
            _fill(blk.LnFfn.Bias, b["n2b"])
            for lin, nm in ((blk.Ffn1, "f1"), (blk.Ffn2, "f2")):
                _fill(lin.Weight, b[nm])
                _fill(lin.Bias, b[nm + "b"])
        else:
            _fill(blk.Ffn.Norm.Weight, b["n2"])
            _fill(blk.Ffn.Gate.Weight, b["gu"][:f])
            _fill(blk.Ffn.Up.Weight, b["gu"][f:])
            _fill(blk.Ffn.Down.Weight, b["down"])


def _decode_config():
    cfg = OaGptConfig.Llama7B()
    cfg.NLayers = 2
    return cfg


def prepare(case, seed):
    k = case["kind"]
    t = _inputs(case, seed)
    s = {"case": case}
    if k == "attention":
        _engine(BF)
        d = case["heads"] * case["hd"]
        layer = OaMultiHeadAttention(d, case["heads"], case["seq"], bias=False, causal=True, rope_theta=ROPE_THETA, init_std=0.02)
        s["opt"] = _trainable(layer)
        for i, lin in enumerate((layer.QProj, layer.KProj, layer.VProj)):
            _fill(lin.Weight, t["wqkv"][i * d:(i + 1) * d])
        _fill(layer.OutProj.Weight, t["wo"])
        s.update(layer=layer, x=t["x"], dy=t["dy"])
    elif k == "flash":
        _engine(BF)
        s.update(t)
    elif k in ("mlp", "norm", "loss"):
        _engine(BF)
        s.update(t)
    elif k == "moe":
        _engine(BF)
        layer = OaMoE(case["dim"], case["ff"], case["experts"], case["topk"], 1e-5, case["shared"], 0.02, expert_bias=False)
        s["opt"] = _trainable(layer)
        _fill(layer.Router.Weight, t["router"])
        _fill(layer.GateUpW, t["gu"])
        _fill(layer.DownW, t["down"])
        if case["shared"]:
            _fill(layer.SharedExperts[0].GateUp.Weight, t["sgu"])
            _fill(layer.SharedExperts[0].Down.Weight, t["sdown"])
        s.update(layer=layer, x=t["x"], dy=t["dy"])
    elif k == "mamba3":
        _engine(BF)
        layer = OaMamba3Module(case["dim"], 128, 2, 64, is_outproj_norm=True, conv_width=4, a_log=True)
        s["opt"] = _trainable(layer)
        for p, nm in ((layer.InProj, "in"), (layer.OutProj, "out"), (layer.DtBias, "dt_bias"), (layer.BBias, "bb"), (layer.CBias, "cb"),
                      (layer.D, "skip"), (layer.NormWeight, "norm"), (layer.ConvWeight, "conv"), (layer.ALog, "a_log")):
            _fill(p, t[nm])
        s.update(layer=layer, x=t["x"].reshape(case["batch"], case["seq"], case["dim"]), dy=t["dy"].reshape(case["batch"], case["seq"], case["dim"]))
    elif k == "generate":
        _engine(BF)
        cfg = _decode_config()
        model = OaGptModel(cfg)
        _load_gpt(model, cfg, _gpt_weights(cfg, seed))
        s["dec"] = OaGptDecoder(model, case["batch"], case["prompt"] + case["steps"])
        s["prompt"] = t["ids"][:, :case["prompt"]].contiguous()
        s["next"] = [t["ids"][:, case["prompt"] + i:case["prompt"] + i + 1].contiguous() for i in range(case["steps"])]
        s["dec"].Prefill(s["prompt"])
        s["dec"].Step(s["next"][0])
    elif k == "char_lm":
        _engine(F32)
        cfg = OaGptConfig.CharLm()
        model = OaGptModel(cfg)
        opt = _trainable(model)
        _load_gpt(model, cfg, _gpt_weights(cfg, seed))
        s.update(ids=t["ids"], target=t["target"], x=F.FromTensor(t["ids"].clone()), y=F.FromTensor(t["target"].clone()), opt=opt)

        def micro_step():
            opt.ZeroGrad()
            with OaGradientTape() as tape:
                logits = model.Forward(s["x"])
                loss = fn_loss.CrossEntropy(logits, s["y"])
                tape.Backward(loss)
            return loss.Tensor(), logits.Tensor()

        micro_step()
        s["program"] = OaTrainingProgram()
        if not s["program"].Capture(micro_step).IsOk():
            raise RuntimeError("the training step could not be captured")
        out = list(s["program"].Outputs())
        for blk in model.Blocks:
            out += [p.Data.GradTensor() for p in blk.AllParameterPtrs() if p.Data.Tensor().dim() == 2]
        out += [m.Weight.Data.GradTensor() for m in (model.Embed, model.PosEmbed, model.LnFinal, model.Head)]
        out += [m.Bias.Data.GradTensor() for m in (model.LnFinal, model.Head)]
        s["out"] = out
    else:
        _engine(F32)
        layer = OaGru(case["input"], case["hidden"], 1)
        s["opt"] = _trainable(layer)
        c = layer.Layers[0]
        for p, nm in ((c.WeightIh, "wih"), (c.WeightHh, "whh"), (c.BiasIh, "bih"), (c.BiasHh, "bhh")):
            _fill(p, t[nm])
        s.update(layer=layer, x=t["x"], dy=t["dy"])
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k in ("attention", "moe", "mamba3", "gru"):
        s["opt"].ZeroGrad()
        x = _leaf(s["x"])
        with OaGradientTape() as tape:
            y = s["layer"].Forward(x, case["batch"], case["seq"]) if k == "attention" else s["layer"].Forward(x)
            tape.Backward(y, s["dy"])
        return [y.Tensor(), x.GradTensor()] + [p.Data.GradTensor() for p in s["layer"].AllParameterPtrs()]
    if k == "flash":
        shape = (case["batch"], case["seq"], case["heads"], case["hd"])
        if not case["train"]:
            return [F.FlashAttentionPacked(OaMatrix(s["qkv"]), *shape).Tensor()]
        qkv = _leaf(s["qkv"])
        with OaGradientTape() as tape:
            o = F.FlashAttentionPacked(qkv, *shape)
            tape.Backward(o, s["do"])
        return [o.Tensor(), qkv.GradTensor()]
    if k == "mlp":
        x, w1, w2 = _leaf(s["x"]), _leaf(s["w1"]), _leaf(s["w2"])
        with OaGradientTape() as tape:
            y = fn_fused.FfnGelu(x, w1, None, w2, None)
            tape.Backward(y, s["dy"])
        return [y.Tensor(), x.GradTensor(), w1.GradTensor(), w2.GradTensor()]
    if k == "norm":
        x, w = _leaf(s["x"]), _leaf(s["w"])
        with OaGradientTape() as tape:
            y = F.RmsNorm(x, w, 1e-5)
            tape.Backward(y, s["dy"])
        return [y.Tensor(), x.GradTensor(), w.GradTensor()]
    if k == "loss":
        logits = _leaf(s["logits"])
        with OaGradientTape() as tape:
            loss = fn_loss.CrossEntropy(logits, OaMatrix(s["target"]))
            tape.Backward(loss)
        return [loss.Tensor(), logits.GradTensor()]
    if k == "generate":
        out = [s["dec"].Prefill(s["prompt"])]
        for ids in s["next"]:
            out.append(s["dec"].Step(ids).clone())
        return [torch.stack(out)]
    s["x"].Tensor().copy_(s["ids"])
    s["y"].Tensor().copy_(s["target"])
    s["program"].Replay()
    return s["out"]


# ------------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    k = case["kind"]
    if k == "attention":
        d, r = case["heads"] * case["hd"], case["batch"] * case["seq"]
        att = 2 * case["batch"] * case["heads"] * case["hd"] * case["seq"] * (case["seq"] + 1)
        return {"bytes": 2 * (4 * r * d + 8 * d * d), "flops": 3 * 8 * r * d * d + 3.5 * att}
    if k == "flash":
        d, r = case["heads"] * case["hd"], case["batch"] * case["seq"]
        att = 2 * case["batch"] * case["heads"] * case["hd"] * case["seq"] * (case["seq"] + 1)
        return {"bytes": 2 * (8 if case["train"] else 4) * r * d, "flops": att * (3.5 if case["train"] else 1)}
    if k == "mlp":
        r, d, f = case["rows"], case["dim"], case["ff"]
        return {"bytes": 2 * (4 * r * d + 4 * d * f), "flops": 12 * r * d * f}
    if k == "norm":
        return {"bytes": 8 * case["rows"] * case["dim"] + 4 * case["dim"], "flops": 12 * case["rows"] * case["dim"]}
    if k == "loss":
        return {"bytes": 4 * case["rows"] * case["vocab"] + 4 * case["rows"] + 4, "flops": 6 * case["rows"] * case["vocab"]}
    if k == "moe":
        t, d, f, e = case["tokens"], case["dim"], case["ff"], case["experts"]
        n = (e + case["shared"]) * 3 * d * f + e * d
        return {"bytes": 2 * (4 * t * d + 2 * n), "flops": 6 * t * (3 * d * f * (case["topk"] + case["shared"]) + d * e)}
    if k == "mamba3":
        d, r = case["dim"], case["batch"] * case["seq"]
        di = 2 * d
        width = 2 * di + 2 * 128 + 3 * (di // 64) + 32
        return {"bytes": 2 * (4 * r * d + 2 * d * (width + di)), "flops": 3 * r * (2 * d * (width + di) + 6 * di * 128)}
    if k == "generate":
        c = _decode_config()
        per_layer = 4 * c.DModel ** 2 + 3 * c.DModel * c.DFf
        b, p, n = case["batch"], case["prompt"], case["steps"]
        kv = 4 * c.DModel * c.NLayers
        weights = 2 * (c.NLayers * per_layer + c.DModel * c.Vocab)
        flops = 2 * b * (p + n) * c.NLayers * per_layer + 2 * b * (n + 1) * c.DModel * c.Vocab
        return {"bytes": weights * (n + 1) + kv * b * (n * p + n * (n + 1) // 2) + 2 * b * (n + 1) * c.Vocab, "flops": flops}
    if k == "char_lm":
        c = OaGptConfig.CharLm()
        r = case["batch"] * case["seq"]
        mats = c.NLayers * 12 * c.DModel ** 2 + c.Vocab * c.DModel
        att = c.NLayers * 2 * r * (case["seq"] + 1) * c.DModel
        return {"bytes": 4 * (2 * mats + 2 * c.Vocab * c.DModel + r * c.Vocab + 2 * r), "flops": 6 * r * mats + 3.5 * att}
    b, t, i, h = case["batch"], case["seq"], case["input"], case["hidden"]
    return {"bytes": 4 * (2 * b * t * (i + h) + 6 * h * (i + h)), "flops": 6 * b * t * 3 * h * (i + h)}


def tolerance(case):
    """About four times the error of the paths against `exact`."""
    # mamba3: the gradient of the B bias, a sum over all tokens and rotations that nearly cancels, is 5.5e-2 off; the others 1e-2
    return {"rel": {"attention": 2e-2, "flash": 1e-2, "mlp": 1e-2, "norm": 7e-3, "loss": 1e-2, "moe": 2e-2, "mamba3": 2e-1, "generate": 2e-2,
                    "char_lm": 1e-5, "gru": 1e-5}[case["kind"]]}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rope64(x, theta=ROPE_THETA, back=False):
    """x [..., seq, heads, hd]: pairs (i, i + hd / 2) turned by position * theta^(-2 i / hd)."""
    s, hd = x.shape[-3], x.shape[-1]
    half = hd // 2
    freq = theta ** (-2.0 * torch.arange(half, device=x.device, dtype=F64) / hd)
    ang = torch.arange(s, device=x.device, dtype=F64)[:, None] * freq
    c, n = ang.cos()[:, None, :], ang.sin()[:, None, :]
    if back:
        n = -n
    a, b = x[..., :half], x[..., half:]
    return torch.cat((a * c - b * n, b * c + a * n), -1)


def _attention64(q, k, v, do=None):
    """Causal attention of [B, S, H, hd]: o, or (o, dq, dk, dv) for an upstream gradient; one sequence at a time."""
    outs = []
    for b in range(q.shape[0]):
        qb, kb, vb = (t[b].transpose(0, 1) for t in (q, k, v))
        scale = 1.0 / math.sqrt(q.shape[-1])
        sc = qb @ kb.transpose(1, 2) * scale
        sc.masked_fill_(torch.ones(sc.shape[1:], dtype=torch.bool, device=sc.device).triu_(1), float("-inf"))
        p = torch.softmax(sc, -1)
        del sc
        o = p @ vb
        if do is None:
            outs.append((o.transpose(0, 1),))
            continue
        g = do[b].transpose(0, 1)
        dv = p.transpose(1, 2) @ g
        ds = g @ vb.transpose(1, 2)
        ds = (ds - (g * o).sum(-1, keepdim=True)) * p
        outs.append(tuple(t.transpose(0, 1) for t in (o, ds @ kb * scale, ds.transpose(1, 2) @ qb * scale, dv)))
    outs = [torch.stack(t) for t in zip(*outs)]
    return outs[0] if do is None else outs


def _gelu64(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _rms64(x, w, eps=1e-5):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _grads(fn, tensors, dy):
    """[y] + gradients of the named tensors for y = fn(tensors) and the upstream gradient dy (None: y is a scalar)."""
    leaves = {n: t.double().requires_grad_(True) for n, t in tensors.items()}
    with torch.enable_grad():
        y = fn(leaves)
        g = torch.autograd.grad(y, list(leaves.values()), None if dy is None else dy.double().reshape(y.shape))
    return y.detach(), dict(zip(leaves, g))


def _moe64(case, t):
    d, f, k = case["dim"], case["ff"], case["topk"]
    zb = {"rb": torch.zeros(case["experts"], device=DEV)}
    if case["shared"]:
        zb.update(sgub=torch.zeros(2 * f, device=DEV), sdownb=torch.zeros(d, device=DEV))
    leaves = {n: t[n] for n in t if n not in ("gu", "down", "dy")}
    leaves.update(zb, nw=torch.ones(d, device=DEV))
    gu, down = t["gu"].double(), t["down"].double()
    dgu, ddown = torch.zeros_like(gu), torch.zeros_like(down)

    def swiglu(h):
        return torch.nn.functional.silu(h[:, :f]) * h[:, f:]

    class Expert(torch.autograd.Function):      # keeps the gradients of one expert's weights out of the graph: they are large
        @staticmethod
        def forward(ctx, x, e):
            ctx.e = e
            ctx.save_for_backward(x)
            return swiglu(x @ gu[e].t()) @ down[e].t()

        @staticmethod
        def backward(ctx, g):
            (x,) = ctx.saved_tensors
            with torch.enable_grad():
                x, a, b = (v.detach().requires_grad_(True) for v in (x, gu[ctx.e], down[ctx.e]))
                y = swiglu(x @ a.t()) @ b.t()
            dx, da, db = torch.autograd.grad(y, (x, a, b), g)
            dgu[ctx.e] += da
            ddown[ctx.e] += db
            return dx, None

    def fn(v):
        n = _rms64(v["x"], v["nw"])
        logits = n @ v["router"].t() + v["rb"]
        p = torch.softmax(logits, -1)
        idx = torch.topk(logits, k, dim=1).indices
        w = torch.gather(p, 1, idx)
        w = w / w.sum(1, keepdim=True)
        y = v["x"]
        for e in range(case["experts"]):
            rows, slot = (idx == e).nonzero(as_tuple=True)
            if rows.numel():
                y = y.index_add(0, rows, Expert.apply(n[rows], e) * w[rows, slot][:, None])
        if case["shared"]:
            y = y + swiglu(n @ v["sgu"].t() + v["sgub"]) @ v["sdown"].t() + v["sdownb"]
        return y

    y, g = _grads(fn, leaves, t["dy"])
    out = [y, g["x"], dgu, ddown, g["nw"], g["router"], g["rb"]]      # the layer's parameter order: its own, then its parts'
    if case["shared"]:
        out += [g["sgu"], g["sgub"], g["sdown"], g["sdownb"]]
    return out


def _mamba64(case, t):
    b, s, d = case["batch"], case["seq"], case["dim"]
    di, n, p, a = 2 * d, 128, 64, 32
    h = di // p
    names = ("in", "dt_bias", "bb", "cb", "skip", "out", "norm", "conv", "a_log")
    v = {k: t[k].double().requires_grad_(True) for k in names + ("x",)}

    def turn(m, cos, sin):
        r0, r1 = m[..., 0:2 * a:2], m[..., 1:2 * a:2]
        r = torch.stack((r0 * cos - r1 * sin, r0 * sin + r1 * cos), -1).flatten(-2)
        return torch.cat((r, m[..., 2 * a:]), -1)

    with torch.enable_grad():
        proj = (v["x"] @ v["in"].t()).reshape(b, s, -1)
        z, xbc, rest = proj[..., :di], proj[..., di:2 * di + 2 * n], proj[..., 2 * di + 2 * n:]
        pad = torch.nn.functional.pad(xbc, (0, 0, 3, 0))
        xbc = torch.nn.functional.silu(sum(pad[:, 3 - j:3 - j + s] * v["conv"][j] for j in range(4)))
        x, bm, cm = xbc[..., :di].reshape(b, s, h, p), xbc[..., di:di + n], xbc[..., di + n:]
        dd_dt, trap, angle = rest[..., :h], torch.sigmoid(rest[..., 2 * h:3 * h]), rest[..., 3 * h:]
        bm = bm * torch.rsqrt((bm * bm).mean(-1, keepdim=True) + 1e-5)
        cm = cm * torch.rsqrt((cm * cm).mean(-1, keepdim=True) + 1e-5)
        dt = torch.clamp(torch.nn.functional.softplus(dd_dt + v["dt_bias"]), 1e-3, 0.1)
        cum = torch.cumsum(-torch.exp(v["a_log"]) * dt, 1)
        gamma, late = dt * trap, dt * (1.0 - trap)
        scale = gamma + torch.cat((late[:, 1:], torch.zeros_like(late[:, :1])), 1)
        theta = torch.cumsum(angle[:, :, None, :] * dt[..., None], 1)
        cos, sin = theta.cos(), theta.sin()
        ct, bt = turn(cm[:, :, None] + v["cb"], cos, sin), turn(bm[:, :, None] + v["bb"], cos, sin)

        class Scan(torch.autograd.Function):     # all pairs of positions, four heads at a time, recomputed for the gradient
            @staticmethod
            def part(x, ct, bt, cum, scale, gamma, skip):
                q = ct.transpose(0, 1) @ bt.permute(1, 2, 0)
                dec = (cum.t()[:, :, None] - cum.t()[:, None, :])
                low = torch.ones(s, s, dtype=torch.bool, device=DEV).tril_(-1)
                m = q * torch.exp(dec.masked_fill(~low, float("-inf"))) * scale.t()[:, None, :]
                y = (m @ x.transpose(0, 1)).transpose(0, 1)
                return y + (skip + gamma * (ct * bt).sum(-1))[..., None] * x

            @staticmethod
            def pieces(args):
                for i in range(b):
                    for j in range(0, h, 4):
                        yield i, slice(j, j + 4), [t[i, :, j:j + 4] if t.dim() > 1 else t[j:j + 4] for t in args]

            @staticmethod
            def forward(ctx, *args):
                ctx.save_for_backward(*args)
                y = torch.empty_like(args[0])
                for i, j, piece in Scan.pieces(args):
                    y[i, :, j] = Scan.part(*piece)
                return y

            @staticmethod
            def backward(ctx, g):
                out = [torch.zeros_like(t) for t in ctx.saved_tensors]
                for i, j, piece in Scan.pieces(ctx.saved_tensors):
                    with torch.enable_grad():
                        piece = [t.detach().requires_grad_(True) for t in piece]
                        y = Scan.part(*piece)
                        gs = torch.autograd.grad(y, piece, g[i, :, j])
                    for o, gi in zip(out, gs):
                        if o.dim() > 1:
                            o[i, :, j] += gi
                        else:
                            o[j] += gi
                return tuple(out)

        y = Scan.apply(x, ct, bt, cum, scale, gamma, v["skip"])
        y = y * torch.rsqrt((y * y).mean(-1, keepdim=True) + 1e-5) * v["norm"] * torch.nn.functional.silu(z.reshape(b, s, h, p))
        y = y.reshape(b, s, di) @ v["out"].t()
        g = torch.autograd.grad(y, list(v.values()), t["dy"].double().reshape(y.shape))
    g = dict(zip(v, g))
    return [y.detach(), g["x"].reshape(b, s, d)] + [g[k] for k in names]


def _generate64(case, seed, ids):
    cfg = _decode_config()
    w = _gpt_weights(cfg, seed)
    h, d, f = cfg.NHeads, cfg.DModel, cfg.DFf
    x = w["embed"].double()[ids.long()]
    b, s = ids.shape
    for blk in w["blocks"]:
        wq = blk["qkv"].double()
        q, k, v = (_rms64(x, blk["n1"].double()) @ wq.t()).reshape(b, s, 3, h, d // h).unbind(2)
        o = _attention64(_rope64(q), _rope64(k), v).reshape(b, s, d)
        x = x + o @ blk["o"].double().t()
        gu = _rms64(x, blk["n2"].double()) @ blk["gu"].double().t()
        x = x + (torch.nn.functional.silu(gu[..., :f]) * gu[..., f:]) @ blk["down"].double().t()
    x = _rms64(x[:, case["prompt"] - 1:], w["norm"].double())
    return [(x @ w["head"].double().t()).transpose(0, 1).contiguous()]


def _char_lm64(case, seed, t):
    cfg = OaGptConfig.CharLm()
    w = _gpt_weights(cfg, seed)
    h, d = cfg.NHeads, cfg.DModel
    b, s = t["ids"].shape
    flat = {k: v for k, v in w.items() if k != "blocks"}
    for i, blk in enumerate(w["blocks"]):
        flat.update({f"{i}.{k}": v for k, v in blk.items()})
    leaves = {k: v.double().requires_grad_(True) for k, v in flat.items()}
    ln = torch.nn.functional.layer_norm
    with torch.enable_grad():
        x = leaves["embed"][t["ids"].long()] + leaves["pos"][:s]
        for i in range(cfg.NLayers):
            m = {k.split(".")[1]: v for k, v in leaves.items() if k.startswith(f"{i}.")}
            q, k, v = (ln(x, (d,), m["n1"], m["n1b"]) @ m["qkv"].t() + m["qkvb"]).reshape(b, s, 3, h, d // h).permute(2, 0, 3, 1, 4)
            o = torch.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True)
            x = x + o.transpose(1, 2).reshape(b, s, d) @ m["o"].t() + m["ob"]
            x = x + _gelu64(ln(x, (d,), m["n2"], m["n2b"]) @ m["f1"].t() + m["f1b"]) @ m["f2"].t() + m["f2b"]
        logits = (ln(x, (d,), leaves["norm"], leaves["normb"]) @ leaves["head"].t() + leaves["headb"]).reshape(b * s, -1)
        loss = torch.nn.functional.cross_entropy(logits, t["target"].long())
        g = dict(zip(leaves, torch.autograd.grad(loss, list(leaves.values()))))
    out = [loss.detach().reshape(1), logits.detach()]
    for i in range(cfg.NLayers):
        out += [g[f"{i}.f1"], g[f"{i}.f2"]] + [g[f"{i}.qkv"][j * d:(j + 1) * d] for j in range(3)] + [g[f"{i}.o"]]
    return out + [g["embed"], g["pos"], g["norm"], g["head"], g["normb"], g["headb"]]


def _gru64(t):
    def fn(v):
        hid = v["whh"].shape[1]
        gi = v["x"] @ v["wih"].t() + v["bih"]
        state, out = torch.zeros(v["x"].shape[0], hid, device=DEV, dtype=F64), []
        for i in range(v["x"].shape[1]):
            gh = state @ v["whh"].t() + v["bhh"]
            r, z = torch.sigmoid(gi[:, i, :hid] + gh[:, :hid]), torch.sigmoid(gi[:, i, hid:2 * hid] + gh[:, hid:2 * hid])
            new = torch.tanh(gi[:, i, 2 * hid:] + r * gh[:, 2 * hid:])
            state = (1 - z) * new + z * state
            out.append(state)
        return torch.stack(out, 1)

    y, g = _grads(fn, {n: t[n] for n in t if n != "dy"}, t["dy"])
    return [y] + [g[n] for n in ("x", "wih", "whh", "bih", "bhh")]


def exact(case, seed):
    k = case["kind"]
    t = _inputs(case, seed)
    if k in ("attention", "flash"):
        b, s, h, hd = case["batch"], case["seq"], case["heads"], case["hd"]
        d = h * hd
    if k == "flash":
        q, v, w = t["qkv"].double().reshape(b, s, 3, h, hd).unbind(2)
        if not case["train"]:
            return [_attention64(q, v, w).reshape(b * s, d)]
        o, *g = _attention64(q, v, w, t["do"].double().reshape(b, s, h, hd))
        return [o.reshape(b * s, d), torch.cat([x.reshape(b * s, d) for x in g], 1)]
    if k == "attention":
        x, wqkv, wo, dy = (t[n].double() for n in ("x", "wqkv", "wo", "dy"))
        q, v, w = (x @ wqkv.t()).reshape(b, s, 3, h, hd).unbind(2)
        o, dq, dk, dv = _attention64(_rope64(q), _rope64(v), w, (dy @ wo).reshape(b, s, h, hd))
        o = o.reshape(b * s, d)
        dqkv = torch.cat([g.reshape(b * s, d) for g in (_rope64(dq, back=True), _rope64(dk, back=True), dv)], 1)
        dw = dqkv.t() @ x
        return [o @ wo.t(), dqkv @ wqkv, dw[:d], dw[d:2 * d], dw[2 * d:], dy.t() @ o]
    if k == "mlp":
        y, g = _grads(lambda v: _gelu64(v["x"] @ v["w1"].t()) @ v["w2"].t(), {n: t[n] for n in ("x", "w1", "w2")}, t["dy"])
        return [y, g["x"], g["w1"], g["w2"]]
    if k == "norm":
        y, g = _grads(lambda v: _rms64(v["x"], v["w"]), {n: t[n] for n in ("x", "w")}, t["dy"])
        return [y, g["x"], g["w"]]
    if k == "loss":
        y, g = _grads(lambda v: torch.nn.functional.cross_entropy(v["logits"], t["target"].long()), {"logits": t["logits"]}, None)
        return [y.reshape(1), g["logits"]]
    if k == "moe":
        return _moe64(case, t)
    if k == "mamba3":
        return _mamba64(case, t)
    if k == "generate":
        return _generate64(case, seed, t["ids"])
    if k == "char_lm":
        return _char_lm64(case, seed, t)
    return _gru64(t)
