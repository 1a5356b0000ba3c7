"""The batched byte-table kernels, which take classes of at least 8 MiB of row
length: numbers of sources around each change of layout and of pipelining,
stripes from a few bytes to megabytes (a CTA's range crosses several), rows at
the sources' offset within 16 bytes and off it, one plan and a plan per stripe.
Products from the CPU oracle; exact, tolerance 0. The counts of launches and
work items show which kernels ran."""
import numpy as np
import pytest
import torch

from fgf_b200 import batch as fb
from fgf_b200 import ops
from fgf_b200.fields import Gf8B, Gf8D
from oracle import orc

pytestmark = pytest.mark.gpu

LENGTHS = [3 << 20, 16, 70001, 5, (1 << 20) + 15, 16 * 1024 + 1, 33, (5 << 20) - 7, 4096, 99999]


def _products(field, coeffs):
    """The 256 products of each coefficient."""
    every, out = np.arange(256, dtype=np.uint8), []
    for c in coeffs:
        row = np.zeros(256, np.uint8)
        orc.dot_product_matrix(field.ID, row, 256, 1, [c], [every])
        out.append(row)
    return out


def _stripe(rng, k, m, n, offset, shifted):
    """Device sources and destination, their bytes, and the rows' starts."""
    srcs_h = [rng.integers(0, 256, size=n, dtype=np.uint8) for _ in range(k)]
    step = -(-(n + offset) // 16) * 16 + 16
    pool = torch.zeros(k * step + offset, dtype=torch.uint8, device="cuda")
    srcs = []
    for t, s in enumerate(srcs_h):
        at = pool[t * step + offset:t * step + offset + n]
        at.copy_(torch.from_numpy(s))
        srcs.append(at)
    starts = [j * step + (3 * j + 1 if shifted else 0) for j in range(m)]
    init = rng.integers(0, 256, size=m * step + 64, dtype=np.uint8)
    hold = torch.zeros(init.size + offset, dtype=torch.uint8, device="cuda")
    dst = hold[offset:]
    dst.copy_(torch.from_numpy(init))
    return srcs, dst, srcs_h, init, starts


@pytest.mark.parametrize("one_plan", [True, False], ids=["one plan", "own plans"])
@pytest.mark.parametrize("shifted", [False, True], ids=["aligned", "shifted"])
@pytest.mark.parametrize("k,m", [(1, 1), (2, 3), (3, 4), (4, 2), (5, 4), (6, 1), (10, 4), (11, 2), (14, 4)])
def test_stripes_of_all_lengths(cuda, k, m, shifted, one_plan):
    field = Gf8B if k % 2 else Gf8D
    rng = np.random.default_rng(100 * k + 10 * m + 2 * shifted + one_plan)
    base = [int(c) for c in rng.integers(0, 256, size=k * m)]
    plan, jobs, checks, vectors, edges = ops.Plan.matrix(field, k, m, base), [], [], 0, 0
    for i, n in enumerate(LENGTHS):
        coeffs = base if one_plan else [int(c) for c in rng.integers(0, 256, size=k * m)]
        if not one_plan:
            plan = ops.Plan.matrix(field, k, m, coeffs)
        offset = (0, 5, 0, 11)[i % 4]
        srcs, dst, srcs_h, want, starts = _stripe(rng, k, m, n, offset, shifted)
        jobs.append(fb.Job(plan, srcs, dst, n, m, bool(i % 3), starts))
        products = _products(field, coeffs)
        for j, s in enumerate(starts):
            row = np.zeros(n, np.uint8) if i % 3 else want[s:s + n].copy()
            for t in range(k):
                row ^= products[t * m + j][srcs_h[t]]
            want[s:s + n] = row
        checks.append((dst, want))
        head = min((16 - offset) % 16, n)
        vectors += n - head >= 16
        edges += (head or (n - head) % 16) != 0
    runner = fb.Batch()
    runner.run(jobs)
    torch.cuda.synchronize()
    for i, (dst, want) in enumerate(checks):
        got = dst.cpu().numpy()
        assert np.array_equal(got, want), (i, LENGTHS[i], np.nonzero(got != want)[0][:8])
    stats = runner.stats()
    if one_plan:
        assert stats["items"] == len(LENGTHS) and stats["launches"] == 1
    else:
        assert stats["items"] == vectors + edges and stats["launches"] == 2


@pytest.mark.parametrize("shifted", [False, True], ids=["aligned", "shifted"])
def test_more_stripes_than_one_parameter_block(cuda, shifted):
    """333 stripes of one plan above the byte tables' threshold: three launches,
    every stripe right."""
    k, m, n, count = 4, 2, 26000 + (4 if shifted else 0), 333
    rng = np.random.default_rng(9)
    coeffs = [int(c) for c in rng.integers(1, 256, size=k * m)]
    plan = ops.Plan.matrix(Gf8D, k, m, coeffs)
    step = -(-n // 16) * 16
    host = rng.integers(0, 256, size=(count, k, step), dtype=np.uint8)
    data = torch.from_numpy(host).cuda()
    out = torch.zeros(count * m * n, dtype=torch.uint8, device="cuda")
    runner = fb.Batch()
    runner.run([fb.Job(plan, [data[s, t, :n] for t in range(k)], out[s * m * n:(s + 1) * m * n], n, m)
                for s in range(count)])
    torch.cuda.synchronize()
    assert runner.stats()["launches"] == 3 and runner.stats()["items"] == count
    products = _products(Gf8D, coeffs)
    got = out.cpu().numpy().reshape(count, m, n)
    for j in range(m):
        want = np.zeros((count, n), np.uint8)
        for t in range(k):
            want ^= products[t * m + j][host[:, t, :n]]
        bad = np.nonzero((got[:, j] != want).any(axis=1))[0]
        assert bad.size == 0, (j, bad[:8])


@pytest.mark.parametrize("k,columns,lone", [(3, 26215, True), (10, 26215, True), (11, 26215, False), (10, 26215, False),
                                            (10, 26214, False)])
def test_short_stripes_of_own_plans(cuda, k, columns, lone):
    """A class far below the threshold, of at least 131072 columns, runs the byte
    tables where it is the submission's only one (up to 10 sources, rows at the
    sources' offset)."""
    m, n = 4, 16 * columns
    rng = np.random.default_rng(k + lone)
    jobs, checks = [], []
    for i in range(5):
        coeffs = [int(c) for c in rng.integers(0, 256, size=k * m)]
        plan = ops.Plan.matrix(Gf8D, k, m, coeffs)
        srcs, dst, srcs_h, want, starts = _stripe(rng, k, m, n, 0, False)
        jobs.append(fb.Job(plan, srcs, dst, n, m, True, starts))
        products = _products(Gf8D, coeffs)
        for j, s in enumerate(starts):
            want[s:s + n] = 0
            for t in range(k):
                want[s:s + n] ^= products[t * m + j][srcs_h[t]]
        checks.append((dst, want))
    if (k, columns, lone) == (10, 26215, False):  # another number of sources beside them
        srcs, dst, srcs_h, want, starts = _stripe(rng, 2, 1, n, 0, False)
        jobs.append(fb.Job(ops.Plan.matrix(Gf8D, 2, 1, [1, 1]), srcs, dst, n, 1, True, starts))
        want[starts[0]:starts[0] + n] = srcs_h[0] ^ srcs_h[1]
        checks.append((dst, want))
    runner = fb.Batch()
    runner.run(jobs)
    torch.cuda.synchronize()
    for i, (dst, want) in enumerate(checks):
        assert np.array_equal(dst.cpu().numpy(), want), i
    assert (runner.stats()["items"] == len(jobs)) == lone  # the table kernels take many items of a stripe
