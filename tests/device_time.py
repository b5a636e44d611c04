"""Device time of short calls for the tests that compare two routes through the kernels."""
import torch


def graph_us(*fns, replays=8):
    """Microseconds a call when `fns` run one after the other in a captured graph: the best of `replays`, so that a busy host or a
    clock ramp does not count."""
    for f in fns:
        f()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for f in fns:
            f()
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = float("inf")
    for _ in range(replays):
        t0.record()
        graph.replay()
        t1.record()
        torch.cuda.synchronize()
        best = min(best, t0.elapsed_time(t1) * 1e3 / len(fns))
    return best
