"""A batched submission on a capturing stream is refused before it touches the
capture or the runner: the capture goes on and the runner's later submissions
(more than it has descriptor slots) work. Exact bytes."""
import pytest
import torch

from fgf_b200 import batch as fb
from fgf_b200 import ops
from fgf_b200.fields import Gf8D

pytestmark = pytest.mark.gpu

K, M, ROW = 20, 4, 4096


@pytest.mark.parametrize("graphs", [True, False], ids=["replayed", "launched"])
@pytest.mark.parametrize("before", [0, 1], ids=["fresh", "used"])
@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_a_capturing_stream_is_refused(cuda, mode, before, graphs):
    gen = torch.Generator(device="cuda").manual_seed(3)
    plan = ops.Plan.matrix(Gf8D, K, M, range(1, K * M + 1))
    srcs = [torch.randint(0, 256, (ROW,), dtype=torch.uint8, device="cuda", generator=gen) for _ in range(K)]
    dst = torch.zeros(M * ROW, dtype=torch.uint8, device="cuda")
    want = torch.zeros_like(dst)
    ops.dot_product_matrix_with(want, ROW, M, plan, srcs)
    runner = fb.Batch(graphs=graphs)
    jobs = runner.prepare([fb.Job(plan, srcs, dst, ROW, M)])
    for _ in range(before):
        runner.run_prepared(jobs)
    torch.cuda.synchronize()
    other = torch.zeros_like(dst)
    graph, side, refusal = torch.cuda.CUDAGraph(), torch.cuda.Stream(), None
    with torch.cuda.graph(graph, stream=side, capture_error_mode=mode):
        try:
            runner.run_prepared(jobs)
        except ops.FgfError as e:
            refusal = str(e)
        ops.dot_product_matrix_with(other, ROW, M, plan, srcs)  # single calls are recorded
    assert refusal is not None and "captured" in refusal
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(other, want)
    for _ in range(5):
        dst.zero_()
        runner.run_prepared(jobs)
        torch.cuda.synchronize()
        assert torch.equal(dst, want)


def test_zeroed_rows_are_recorded(cuda):
    """Jobs without sources only clear their rows, which a graph can repeat."""
    dst = torch.ones(3 * 64, dtype=torch.uint8, device="cuda")
    runner = fb.Batch()
    jobs = runner.prepare([fb.Job(ops.Plan.matrix(Gf8D, 0, 3, []), [], dst, 64, 3)])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        runner.run_prepared(jobs)
    dst.fill_(1)
    graph.replay()
    torch.cuda.synchronize()
    assert not dst.any()
