"""Calls of the 8-byte fields on the kernel of short rows and few sources (wide.cu)
and around the lines where the table kernels take over: numbers of rows around
one launch's, of sources around one launch's tables, single elements, every kind
of offset, scatter and gather forms. Against the CPU oracle; exact, tolerance 0."""
import numpy as np
import pytest
import torch

from fgf_b200 import batch as fb
from fgf_b200 import ops
from fgf_b200.fields import FIELDS
from oracle import orc

pytestmark = pytest.mark.gpu

WIDE = [f for f in FIELDS.values() if f.BYTES == 8]


def _coeffs(n, rng):
    return [int.from_bytes(rng.bytes(8), "little") for _ in range(n)]


def _place(host, offset):
    hold = torch.zeros(host.size + 64, dtype=torch.uint8, device="cuda")
    hold[offset:offset + host.size] = torch.from_numpy(host).cuda()
    return hold[offset:offset + host.size]


def _check(field, k, m, n, src_off, dst_off, ovr, rng):
    srcs = [rng.integers(0, 256, size=n, dtype=np.uint8) for _ in range(k)]
    coeffs = _coeffs(k * m, rng)
    init = rng.integers(0, 256, size=m * n + 16, dtype=np.uint8)
    want = init.copy()
    (orc.dot_product_matrix if ovr else orc.mul_add_matrix)(field.ID, want[:m * n], n, m, coeffs, srcs)
    dst = _place(init, dst_off)
    op = ops.dot_product_matrix_with if ovr else ops.mul_add_matrix_with
    op(dst[:m * n], n, m, ops.Plan.matrix(field, k, m, coeffs), [_place(s, (src_off * (t + 1)) % 16) for t, s in enumerate(srcs)])
    got = dst.cpu().numpy()
    assert np.array_equal(got, want), (k, m, n, src_off, dst_off, ovr, np.nonzero(got != want)[0][:8])


@pytest.mark.parametrize("field", WIDE, ids=lambda f: f.__name__)
@pytest.mark.parametrize("k,m", [(1, 1), (1, 9), (2, 3), (3, 8), (4, 5), (13, 8), (14, 8), (27, 4), (64, 1), (65, 2)])
def test_rows_and_sources(cuda, field, k, m):
    rng = np.random.default_rng(k * 20 + m + field.ID)
    for i, elements in enumerate((1, 3, 255, 256, 257, 1000)):
        for src_off, dst_off in ((0, 0), (8, 0), (0, 8), (3, 5)):
            _check(field, k, m, 8 * elements, src_off, dst_off, (i + src_off) % 3 != 0, rng)


@pytest.mark.parametrize("field", WIDE, ids=lambda f: f.__name__)
@pytest.mark.parametrize("k,m", [(1, 1), (1, 2), (1, 3), (2, 2), (2, 3), (3, 2), (3, 6)])
def test_around_the_lines(cuda, field, k, m):
    rng = np.random.default_rng(k * 20 + m)
    for n in (512 * 1024 - 8, 512 * 1024, 768 * 1024 - 8, 768 * 1024):
        _check(field, k, m, n, 0, 0, True, rng)


@pytest.mark.parametrize("field", WIDE, ids=lambda f: f.__name__)
def test_scatter_and_gather(cuda, field):
    rng = np.random.default_rng(field.ID)
    n = 8 * 300
    coeffs = _coeffs(11, rng)
    plan = ops.Plan.new(field, coeffs)
    srcs = [rng.integers(0, 256, size=n, dtype=np.uint8) for _ in coeffs]
    want = rng.integers(0, 256, size=11 * n, dtype=np.uint8)
    rows = _place(want, 0)
    orc.mul_add_scatter(field.ID, want, n, coeffs, srcs[0])
    ops.mul_add_scatter_with(rows, n, plan, _place(srcs[0], 0))
    assert np.array_equal(rows.cpu().numpy(), want)
    want = rng.integers(0, 256, size=n, dtype=np.uint8)
    dst = _place(want, 0)
    orc.mul_add_gather(field.ID, want, coeffs, srcs)
    ops.mul_add_gather_with(dst, plan, [_place(s, 0) for s in srcs])
    assert np.array_equal(dst.cpu().numpy(), want)
    want = rng.integers(0, 256, size=n, dtype=np.uint8)
    for offset in (0, 3):
        mine, dst = want.copy(), _place(want, offset)
        orc.mul_assign(field.ID, mine, coeffs[0])
        ops.mul_assign(field, dst, coeffs[0])
        assert np.array_equal(dst.cpu().numpy(), mine)


@pytest.mark.parametrize("field", WIDE, ids=lambda f: f.__name__)
def test_long_stripes_in_a_batch(cuda, field):
    """Long stripes of few sources run as calls of their own; shorter and wider ones
    beside them on the work list."""
    rng = np.random.default_rng(field.ID + 5)
    jobs, checks = [], []
    for k, m, n in ((1, 3, 4 << 20), (1, 3, (4 << 20) - 8), (3, 2, 8000), (2, 3, (4 << 20) + 8), (1, 3, 8 << 20)):
        srcs = [rng.integers(0, 256, size=n, dtype=np.uint8) for _ in range(k)]
        coeffs = _coeffs(k * m, rng)
        ovr = k != 2
        want = rng.integers(0, 256, size=m * n, dtype=np.uint8)
        dst = _place(want, 0)
        (orc.dot_product_matrix if ovr else orc.mul_add_matrix)(field.ID, want, n, m, coeffs, srcs)
        jobs.append(fb.Job(ops.Plan.matrix(field, k, m, coeffs), [_place(s, 0) for s in srcs], dst, n, m, ovr))
        checks.append((dst, want))
    fb.Batch().run(jobs)
    torch.cuda.synchronize()
    for i, (dst, want) in enumerate(checks):
        assert np.array_equal(dst.cpu().numpy(), want), i
