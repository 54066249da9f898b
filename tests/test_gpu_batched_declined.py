"""Batched plans in which some segments are left to the digit passes, beside the
others: by a captured graph and without, run after run on a stream of the caller's,
and inside a capture of the caller's; many declined segments of few chunks, few of
many chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = {"many": [5_000 + 7 * i for i in range(300)], "mixed": [70_001, 5, 4097, 300_000, 3000, 0, 1_000_003, 20_000] * 3,
         "long": [2048 * 3072 + 1, 100, 2_000_000, 50_000]}


def batch(name):
    rng = np.random.default_rng(len(name))
    off = np.concatenate([[0], np.cumsum(SIZES[name])]).astype(np.uint64)
    keys = rng.integers(0, 1 << 32, int(off[-1]), dtype=np.uint32)
    for i, (a, b) in enumerate(zip(off[:-1].astype(int), off[1:].astype(int))):
        if i % 2 == 0:  # crowded: half of the keys in few values
            keys[a:b:2] = rng.integers(0, 9, keys[a:b:2].size, dtype=np.uint32) * np.uint32(123_456_789)
    want = keys.copy()
    for a, b in zip(off[:-1].astype(int), off[1:].astype(int)):
        want[a:b].sort()
    return off, keys, want


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("name", list(SIZES))
def test_runs_on_a_stream(pa, torch_cuda, name, graph):
    from parallelalgorithms_gb300.batched import SegmentedSortPlan
    torch = torch_cuda
    off, keys, want = batch(name)
    src = torch.from_numpy(keys.view(np.int32)).cuda()
    d, t = torch.empty_like(src), torch.empty_like(src)
    plan = SegmentedSortPlan(off, use_graph=graph)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    outs = []
    with torch.cuda.stream(stream):
        for _ in range(3):  # nothing waits between the runs but the stream
            d.copy_(src)
            plan.run(d, t, stream.cuda_stream, sync=False)
            outs.append(d.clone())
    plan.sync(stream.cuda_stream)
    for o in outs:
        assert np.array_equal(o.cpu().numpy().view(np.uint32), want)
    plan.close()


@pytest.mark.parametrize("name", ["mixed", "many"])
def test_inside_a_capture(pa, torch_cuda, name):
    from parallelalgorithms_gb300.batched import SegmentedSortPlan
    torch = torch_cuda
    off, keys, want = batch(name)
    src = torch.from_numpy(keys.view(np.int32)).cuda()
    d, t = torch.empty_like(src), torch.empty_like(src)
    plan = SegmentedSortPlan(off, use_graph=False)
    plan.run(d.copy_(src), t)  # (first use outside)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        d.copy_(src)
        plan.run(d, t, torch.cuda.current_stream().cuda_stream, sync=False)
    for _ in range(2):
        d.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(d.cpu().numpy().view(np.uint32), want)
    plan.close()


def test_declined_segments_are_not_walked_one_by_one(pa, torch_cuda):
    """2000 declined segments take at most three times what buckets take: 2.1 times
    by digit passes alone, 3.6 with a walk over all segments in every CTA."""
    import time

    from parallelalgorithms_gb300.batched import SegmentedSortPlan
    torch = torch_cuda
    off = np.arange(2001, dtype=np.uint64) * 20_000
    n = int(off[-1])
    even = torch.randint(-(1 << 31), 1 << 31, (n,), device="cuda", dtype=torch.int32)
    crowded = even.clone()
    crowded[::2] &= 3
    d, t = torch.empty_like(even), torch.empty_like(even)
    plan = SegmentedSortPlan(off)
    took = {}
    for name, src in (("even", even), ("crowded", crowded)):
        took[name] = 1e9
        for _ in range(5):
            d.copy_(src)
            torch.cuda.synchronize()
            start = time.perf_counter()
            plan.run(d, t)
            took[name] = min(took[name], time.perf_counter() - start)
        flip = -(1 << 31)
        assert torch.equal(d ^ flip, torch.sort((src ^ flip).view(2000, -1), dim=1)[0].view(-1))
    plan.close()
    assert took["crowded"] < 3 * took["even"], took
