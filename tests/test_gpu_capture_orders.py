"""A translation recorded in a stream capture after calls of the same precision
mode at other order bounds: group sizes, and the tables that go with them,
differ with the bound, and inside a capture nothing can be uploaded."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,mode,op,P,warm,bound", [
    ("f64", "PLAIN", "m2l", 16, 12, 16),     # 4 threads, then 8
    ("f64", "PLAIN", "m2l", 16, 16, 12),
    ("f64", "PLAIN", "l2l", 40, 12, 40),     # one warp per translation
    ("f64", "PLAIN", "m2l", 40, 40, 12),
    ("f64", "PLAIN", "m2m", 40, 40, 20),
    ("f64", "SPLIT", "m2l", 16, 13, 14),
    ("f64", "SPLIT", "m2l", 20, 20, 10),
    ("f64", "SPLIT_FF", "m2l", 24, 8, 24),
    ("f64", "SPLIT", "m2m", 24, 16, 20),     # the FP64 kernel's tables
    ("f32", "PLAIN", "m2l", 16, 14, 15),
    ("f32", "PLAIN", "m2m", 24, 24, 6),
])
def test_capture_after_another_order(native, dtype, mode, op, P, warm, bound):
    import torch

    dev = "cuda:0"
    prec, n, S = getattr(native, mode), 40, P * (P + 1)
    rng = np.random.default_rng(P + bound)
    dt = torch.float64 if dtype == "f64" else torch.float32
    src = torch.as_tensor(rng.normal(size=(n, S)), dtype=dt, device=dev)
    sh = torch.as_tensor(rng.normal(size=(n, 3)) + 2, device=dev)
    orders = {p: torch.full((n,), p, dtype=torch.int32, device=dev) for p in (warm, bound)}
    ctx = native.Context(P, dtype)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)

    def call(p, dst):
        ctx.translate_device(op, prec, n, src, S, n, dst, S, n, orders[p], orders[p], sh, order_bound=p)

    dst = [torch.zeros(n, S, dtype=dt, device=dev) for _ in range(3)]
    torch.cuda.synchronize()
    call(warm, dst[0])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call(bound, dst[1])
    graph.replay()
    torch.cuda.synchronize()
    call(bound, dst[2])
    torch.cuda.synchronize()
    assert torch.isfinite(dst[1]).all() and dst[1].any()
    assert torch.equal(dst[1], dst[2])
