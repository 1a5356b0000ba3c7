"""Descriptors of a submission go up beside the caller's stream or as a node of the
replayed graph, by its size. Either way, two submissions of one shape that take
turns without waiting, each on its own buffers and more often than there are
descriptor slots, write what single calls write. Exact bytes."""
import pytest
import torch

from fgf_b200 import batch as fb
from fgf_b200 import ops
from fgf_b200.fields import Gf8D, Gf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [True, False], ids=["replayed", "launched"])
@pytest.mark.parametrize("n", [4096, 1 << 20], ids=["short", "long"])
def test_two_submissions_in_turn(cuda, n, graphs):
    gen = torch.Generator(device="cuda").manual_seed(n)
    runner, turns = fb.Batch(graphs=graphs), []
    for _ in range(2):
        jobs, wants = [], []
        for field, k, m in ((Gf8D, 20, 4), (Gf16, 12, 6), (Gf8D, 16, 3)):
            plan = ops.Plan.matrix(field, k, m, [(7 * i) % 251 + 1 for i in range(k * m)])
            srcs = [torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=gen) for _ in range(k)]
            want = torch.zeros(m * n, dtype=torch.uint8, device="cuda")
            ops.dot_product_matrix_with(want, n, m, plan, srcs)
            jobs.append(fb.Job(plan, srcs, torch.zeros_like(want), n, m))
            wants.append(want)
        turns.append((runner.prepare(jobs), jobs, wants))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for r in range(10):
        prepared, jobs, _ = turns[r % 2]
        with torch.cuda.stream(stream):
            for j in jobs:
                j.dst.zero_()
            runner.run_prepared(prepared)
    torch.cuda.synchronize()
    for _, jobs, wants in turns:
        for j, want in zip(jobs, wants):
            assert torch.equal(j.dst, want)
