"""What a replayed decoding step begins with: the new tokens' rows and the position."""
import pytest
import torch

from oa_b200.core import fn_matrix as F
from oa_b200.core.types import OaScalarType
from oa_b200.models.gpt import OaGptConfig, OaGptModel
from oa_b200.ops import kernels as K
from oa_b200.runtime.engine import OaInitComputeEngine
from oa_b200.serve.decoder import OaGptDecoder

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,vocab", [(1, 8, 3), (1, 4096, 100), (3, 264, 50), (40, 1024, 7), (700, 2048, 31)])
def test_rows_and_position(n, dim, vocab):
    table = torch.randn(vocab, dim, device="cuda").bfloat16()
    ids = torch.randint(0, vocab, (n,), device="cuda", dtype=torch.int32)
    ids[n // 2] = vocab                                    # outside the table: a row of NaN, as the embedding gives it
    x, pos = torch.zeros(n, dim, device="cuda", dtype=torch.bfloat16), torch.tensor([41], dtype=torch.int32, device="cuda")
    K.decode_begin(table, ids, x, pos)
    ref = K.embedding_fwd(table, ids)
    assert torch.equal(x.view(torch.int16), ref.view(torch.int16)) and bool(x[n // 2].isnan().all())
    assert pos.item() == 42
    # with the norm behind it
    w, xw, sq = torch.randn(dim, device="cuda").bfloat16(), torch.zeros_like(x), torch.zeros(1, n, device="cuda")
    K.decode_begin(table, ids, x, pos, w, xw, sq)
    ok = ids < vocab
    assert torch.equal(xw[ok], (ref[ok].float() * w.float()).bfloat16()) and pos.item() == 43
    assert torch.allclose(sq[0][ok].double(), (ref[ok].double() ** 2).sum(1), rtol=1e-5) and bool(sq[0][~ok].isnan().all())


def test_ids_of_any_kind_continue_the_same_text():
    """A step takes ids of other integer types, from the host and from a larger tensor; without a prompt it starts at position 0."""
    OaInitComputeEngine()
    F.SetWeightDtype(OaScalarType.BFloat16)
    cfg = OaGptConfig(64, 128, 2, 2, 256, 64, "rms", "swiglu", 10000.0, False, 1e-5, 0.1)
    model = OaGptModel(cfg)
    eager, text = OaGptDecoder(model, 3, 32, use_graph=False), torch.randint(0, 64, (3, 12), device="cuda", dtype=torch.int32)
    for prompt in (0, 4):
        dec = OaGptDecoder(model, 3, 32)
        eager.Cache.Reset()
        if prompt:
            assert torch.equal(dec.Prefill(text[:, :prompt].contiguous()), eager.Prefill(text[:, :prompt].contiguous()))
        for i in range(prompt, 12):
            col = text[:, i:i + 1]
            ids = (col.contiguous(), col, col.long(), col.cpu())[i % 4]
            got, want = dec.Step(ids).float(), eager.Step(col.contiguous()).float()
            assert float((got - want).norm() / want.norm()) <= 1e-2, (prompt, i)     # a few bf16 roundings apart: other kernels for a graph's steps
        assert dec.Cache.Length == 12
