"""Few-row products that request their weights before the previous kernel has finished: every launch in a captured chain gives what
the same calls give one by one, weights changed between replays are the ones that count, and only resting storages are meant."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,dim,ff", [(1, 512, 512), (3, 1024, 2816), (33, 4096, 1024), (64, 512, 8200)])
def test_chain_in_a_graph(rows, dim, ff):
    g = torch.Generator(device="cuda").manual_seed(rows)
    rnd = lambda *s: (torch.randn(*s, device="cuda", generator=g) / s[-1] ** 0.5).bfloat16()
    x, w1, w2, gain = rnd(rows, dim) * 30, rnd(2 * ff, dim), rnd(dim, ff), 1.0 + rnd(dim)

    def chain():
        y = x
        for _ in range(3):
            h = K.rmsnorm_fwd(y, gain, 1e-5)[0]
            y = K.gemm(K.swiglu_fwd(K.gemm(h, w1)), w2, residual=y)
        return y

    chain()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph), K.weights_at_rest([w1, w2]):
        out = chain()
    for step in range(4):
        graph.replay()
        got = out.clone()
        torch.cuda.synchronize()
        assert torch.equal(got, chain()), step
        w1.mul_(-0.75)                                          # by a kernel right before the next replay
        w2.add_(w2, alpha=0.25)
    torch.cuda.synchronize()
    K.check_status()


def test_only_the_named_storages():
    w = torch.randn(1024, 512, device="cuda").bfloat16()
    x = torch.randn(2, 512, device="cuda").bfloat16()
    seen = []
    lib = K.N.require()
    few, tile = lib.oa_gemm_bf16_few_rows, lib.oa_gemm_bf16

    class Spy:
        def __getattr__(self, name):
            return getattr(lib, name)

        def oa_gemm_bf16_few_rows(self, *a):
            seen.append(("rest", a[1]))
            return few(*a)

        def oa_gemm_bf16(self, *a):
            seen.append(("any", a[1]))
            return tile(*a)

    require = K.N.require
    K.N.require = lambda: Spy()
    try:
        copy = w.clone()
        with K.weights_at_rest([w]):
            K.gemm(x, w)
            K.gemm(x, w[:512])                                  # a view of it
            K.gemm(x, copy)                                     # a copy may have been written just before
        K.gemm(x, w)
    finally:
        K.N.require = require
    torch.cuda.synchronize()
    assert seen == [("rest", w.data_ptr()), ("rest", w.data_ptr()), ("any", copy.data_ptr()), ("any", w.data_ptr())]
