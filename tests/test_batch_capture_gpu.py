"""A batched advect captured into the caller's CUDA graph: the capture advances
nothing, every replay advances the fields as a call would, for odd and even
numbers of time blocks, among other calls, and with the settings of its capture
after the batch has gone on with others."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def _batch(fdb, specs, f, stream=None):
    b = fdb.Batch([(s["v"], s["L"], s["n"]) for s in specs])
    if stream is not None:
        b.set_stream(stream)
    b.set_tuning(depth=2)
    b.set_fields(f)
    return b


def _fields(b, like):
    import torch
    out = torch.empty_like(like)
    b.get_fields(out)
    return out


@pytest.mark.filterwarnings("ignore:The CUDA Graph is empty")
@pytest.mark.parametrize("steps", [6, 8, 1])  # 3, 4 and 1 time blocks
def test_replays_advance_like_calls(fdb, steps):
    import torch

    from fidibench_gb300.batch import random_instances
    specs = random_instances(12, 21, 9, 70)
    dts = [s["dt"] for s in specs]
    other = [0.7 * d for d in dts]
    stream = torch.cuda.Stream()
    total = sum(s["n"][0] * s["n"][1] * s["n"][2] for s in specs)
    f = torch.randn(total, dtype=torch.float64, device="cuda",
                    generator=torch.Generator("cuda").manual_seed(3))
    b = _batch(fdb, specs, f, stream)
    ref = _batch(fdb, specs, f)
    with pytest.raises(fdb.FdbError):  # no tables yet
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream, capture_error_mode="thread_local"):
            b.advect(steps, dts)
    assert torch.equal(_fields(b, f), f)

    def both(n, d):
        b.advect(n, d)
        ref.advect(n, d)
        assert torch.equal(_fields(b, f), _fields(ref, f))

    def replay(graph, d, times=1):
        for _ in range(times):
            with torch.cuda.stream(stream):
                graph.replay()
            ref.advect(steps, d)
        stream.synchronize()
        assert torch.equal(_fields(b, f), _fields(ref, f))

    both(steps, dts)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream, capture_error_mode="thread_local"):
        b.advect(steps, dts)
    assert torch.equal(_fields(b, f), _fields(ref, f))  # nothing ran
    replay(g, dts, 3)
    both(steps, dts)
    both(3, other)  # other tables
    b.set_tuning(tile_z=4)  # and larger ones
    both(5, other)
    replay(g, dts, 2)
    g2 = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g2, stream=stream, capture_error_mode="thread_local"):
        b.advect(steps, other)
    replay(g2, other)
    replay(g, dts)
    b.set_fields(f)
    ref.set_fields(f)
    replay(g2, other)
    # gradients run on buffers of their own
    assert torch.equal(b.advect_transposed(7, dts, f), ref.advect_transposed(7, dts, f))
    replay(g, dts)
    stream.synchronize()
    b.close()
    ref.close()


def test_looped_advect_under_capture(fdb):
    import torch

    from fidibench_gb300.batch import random_instances
    specs = random_instances(5, 22, 9, 70)
    dts = [s["dt"] for s in specs]
    stream = torch.cuda.Stream()
    total = sum(s["n"][0] * s["n"][1] * s["n"][2] for s in specs)
    f = torch.randn(total, dtype=torch.float64, device="cuda",
                    generator=torch.Generator("cuda").manual_seed(4))
    b = _batch(fdb, specs, f, stream)
    ref = _batch(fdb, specs, f)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream, capture_error_mode="thread_local"):
        b.advect_looped(6, dts)
    assert torch.equal(_fields(b, f), f)
    for _ in range(2):
        with torch.cuda.stream(stream):
            g.replay()
        ref.advect_looped(6, dts)
        stream.synchronize()
        assert torch.equal(_fields(b, f), _fields(ref, f))
    b.close()
    ref.close()
