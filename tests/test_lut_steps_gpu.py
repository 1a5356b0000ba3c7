"""Table kernels on calls and work items of several steps: a CTA's tiles and a
warp's blocks go round more than once, ending just around a step, with rows off
the sources' boundaries and with sources anywhere; shapes that fetch the next
column ahead and shapes that do not. Products from the CPU oracle; exact,
tolerance 0."""
import numpy as np
import pytest
import torch

from fgf_b200 import batch as fb
from fgf_b200 import ops, tune
from fgf_b200.fields import Gf8B, Gf8D, Gf16
from oracle import orc

pytestmark = pytest.mark.gpu

STEP = 256 // 32 * 31 * 16  # bytes that a CTA's warps write per tile, rows off the boundaries


@pytest.fixture(autouse=True)
def _tables_only(cuda):
    tune.force("nibble")
    yield
    tune.force("auto")
    tune.clear()


def _products(field, coeffs):
    """Products of every element by each coefficient (1- and 2-byte fields)."""
    dtype = np.uint8 if field.BYTES == 1 else np.uint16
    every = np.arange(1 << (8 * field.BYTES), dtype=dtype)
    out = []
    for c in coeffs:
        row = np.zeros(every.nbytes, np.uint8)
        orc.dot_product_matrix(field.ID, row, every.nbytes, 1, [c], [every.view(np.uint8)])
        out.append(row.view(dtype))
    return out


def _job(field, k, m, n, rows_off, srcs_off, rng):
    """A destination with guard bytes, sources, coefficients and the rows' sum."""
    b = field.BYTES
    coeffs = [int(c) for c in rng.integers(1, 1 << (8 * b), size=k * m)]
    products = _products(field, coeffs)
    srcs, host = [], []
    for t in range(k):
        h = rng.integers(0, 256, size=n, dtype=np.uint8)
        off = (3 * t + 1) % 16 if srcs_off else 0
        hold = torch.zeros(n + 32, dtype=torch.uint8, device="cuda")
        hold[off:off + n].copy_(torch.from_numpy(h))
        srcs.append(hold[off:off + n])
        host.append(h.view(np.uint8 if b == 1 else np.uint16))
    step = -(-n // 16) * 16 + 32
    starts = [j * step + ((5 * j + 3) * b % 16 if rows_off else 0) for j in range(m)]
    init = rng.integers(0, 256, size=m * step + 32, dtype=np.uint8)
    sums = []
    for j in range(m):
        s = products[j][host[0]].copy()
        for t in range(1, k):
            s ^= products[t * m + j][host[t]]
        sums.append(s.view(np.uint8))
    dst = torch.from_numpy(init).cuda()
    return ops.Plan.matrix(field, k, m, coeffs), srcs, dst, starts, init, sums


def _want(init, starts, sums, ovr):
    want = init.copy()
    for s, row in zip(starts, sums):
        want[s:s + row.size] = row if ovr else want[s:s + row.size] ^ row
    return want


@pytest.mark.parametrize("mode", ["aligned", "rows", "sources"])
@pytest.mark.parametrize("field,k,m", [(Gf8D, 4, 4), (Gf8B, 5, 13), (Gf16, 4, 8), (Gf16, 3, 2), (Gf16, 2, 5)],
                         ids=lambda x: getattr(x, "__name__", str(x)))
def test_calls_of_several_steps(field, k, m, mode):
    """More tiles than resident CTAs (444 or 592 of 4 KiB)."""
    rng = np.random.default_rng(100 * k + 10 * m + len(mode))
    b = field.BYTES
    for i, n in enumerate((600 * STEP - 16 + b, 600 * STEP + 17 * b, 1300 * STEP + 15 * b + 16)):
        n -= n % b
        plan, srcs, dst, starts, init, sums = _job(field, k, m, n, mode != "aligned", mode == "sources", rng)
        ovr = i != 1
        op = ops.dot_product_matrix_scattered_with if ovr else ops.mul_add_matrix_scattered_with
        op(dst, n, starts, plan, srcs)
        got = dst.cpu().numpy()
        want = _want(init, starts, sums, ovr)
        assert np.array_equal(got, want), (n, np.nonzero(got != want)[0][:8])


@pytest.mark.parametrize("mode", ["aligned", "rows", "sources"])
@pytest.mark.parametrize("cols", [1, 2, 4, 8, 16])
def test_items_of_every_tile(cols, mode):
    """Work items of as many tiles as the tile shape says, one each where it is 1."""
    rng = np.random.default_rng(cols + len(mode))
    jobs, checks, tiles = [], [], 0
    for field, k, m, n in ((Gf8D, 3, 8, (8 << 20) + 5), (Gf8B, 3, 7, (5 << 20) + 16 * 77 + 3), (Gf8D, 4, 6, 4 << 20)):
        plan, srcs, dst, starts, init, sums = _job(field, k, m, n, mode != "aligned", mode == "sources", rng)
        jobs.append(fb.Job(plan, srcs, dst, n, m, True, starts))
        checks.append((dst, _want(init, starts, sums, True)))
        tiles += n // 4096
    runner = fb.Batch()
    prepared = runner.prepare(jobs)
    tune.set_tile(1, 2, 1)
    runner.run_prepared(prepared)
    single = runner.stats()["items"]
    assert single >= tiles
    tune.set_tile(1, 2, cols)
    for dst, _ in checks:
        dst.zero_()
    runner.run_prepared(prepared)
    items = runner.stats()["items"]
    assert (items == single) == (cols == 1) and items >= single // (2 * cols)
    for i, (dst, want) in enumerate(checks):
        got = dst.cpu().numpy()
        for s in jobs[i].row_starts:  # the rows; the gaps were cleared
            n = jobs[i].row_len
            assert np.array_equal(got[s:s + n], want[s:s + n]), (i, s)
