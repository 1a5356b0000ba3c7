"""The table kernels of the matrix calls (lut.cuh) where they can go wrong:
numbers of sources around the groups of three and around one launch's limit,
numbers of rows around every change of tower split, lengths around whole
columns, around a warp's step and around its last blocks, and sources and rows
at every kind of offset. Against the CPU oracle; the arithmetic is exact, so
the tolerance is 0. Bytes around the rows must stay as they were."""
import numpy as np
import pytest
import torch

from fgf_b200 import batch as fb
from fgf_b200 import ops, tune
from fgf_b200.fields import FIELDS
from oracle import orc

pytestmark = pytest.mark.gpu

ALL = list(FIELDS.values())
ROWS = {1: (1, 4, 5, 8, 9, 12, 13, 16, 17), 2: (1, 2, 3, 4, 5, 8, 9), 4: (1, 2, 3, 4, 5), 8: (1, 2, 3, 4, 5)}
SOURCES = (1, 2, 3, 4, 6, 8, 19, 64, 65)
LENGTHS = (1, 2, 3, 4, 5, 30, 31, 32, 33, 62, 63, 64, 65, 66, 1000, 4096, 9001)  # elements


@pytest.fixture(autouse=True)
def _tables_only(cuda):
    tune.force("nibble")
    yield
    tune.force("auto")


def _buf(rng, n, off):
    """n bytes on the device, `off` past a 16-byte boundary."""
    host = rng.integers(0, 256, size=n, dtype=np.uint8)
    t = torch.empty(n + 64, dtype=torch.uint8, device="cuda")
    t[off:off + n] = torch.from_numpy(host).cuda()
    return host, t[off:off + n]


def _coeffs(field, n, rng):
    return [int.from_bytes(rng.bytes(field.BYTES), "little") for _ in range(n)]


def _run(field, k, m, rl, src_offs, base, row_offs, ovr, raw, batched, rng):
    srcs = [_buf(rng, rl, o) for o in src_offs]
    coeffs = _coeffs(field, k * m, rng)
    starts, at = [], 16
    for o in row_offs:
        starts.append(at + o)
        at += -(-(rl + o) // 16) * 16 + 16
    init, dst = _buf(rng, at + 16, base)
    want = init.copy()
    for s in starts:
        if ovr:
            want[s:s + rl] = 0
    orc.mul_add_matrix_scattered(field.ID, want, rl, starts, coeffs, [s for s, _ in srcs])
    if raw and not ovr:
        ops.mul_add_matrix_scattered(field, dst, rl, starts,
                                     [(coeffs[t * m:(t + 1) * m], srcs[t][1]) for t in range(k)])
    else:
        plan = ops.Plan.matrix(field, k, m, coeffs)
        if batched:
            fb.Batch().run([fb.Job(plan, [s for _, s in srcs], dst, rl, m, ovr, starts)])
        elif ovr:
            ops.dot_product_matrix_scattered_with(dst, rl, starts, plan, [s for _, s in srcs])
        else:
            ops.mul_add_matrix_scattered_with(dst, rl, starts, plan, [s for _, s in srcs])
    torch.cuda.synchronize()
    got = dst.cpu().numpy()
    bad = np.nonzero(got != want)[0]
    assert bad.size == 0, (field.__name__, k, m, rl, src_offs, base, row_offs, ovr, raw, batched, bad[:8], starts)


@pytest.mark.parametrize("batched", [False, True], ids=["single", "batch"])
@pytest.mark.parametrize("offsets", ["aligned", "common", "rows", "sources", "any"])
@pytest.mark.parametrize("field", ALL, ids=lambda f: f.__name__)
def test_matrix_shapes(cuda, field, offsets, batched):
    b = field.BYTES
    rng = np.random.default_rng(1000 * field.ID + len(offsets) + 7 * batched)
    shapes = [(k, m) for k in (3, 10) for m in ROWS[b]] + [(k, m) for k in SOURCES for m in (2, 4)]
    for i, (k, m) in enumerate(shapes):
        for rl in (LENGTHS[(3 * i) % len(LENGTHS)], LENGTHS[(5 * i + 1) % len(LENGTHS)], 2000 + i):
            rl *= b
            so, base, ro = [0] * k, 0, [0] * m
            if offsets == "common":
                base = (3 + i) % 16
                so = [base] * k
            if offsets in ("rows", "any"):  # row offsets are whole elements
                base = int(rng.integers(0, 16))
                ro = [int(x) * b for x in rng.integers(0, 16 // b, size=m)]
            if offsets in ("sources", "any"):
                so = [int(x) for x in rng.integers(0, 16, size=k)]
            _run(field, k, m, rl, so, base, ro, bool(i & 1), i % 3 == 0, batched, rng)


@pytest.mark.parametrize("field", ALL, ids=lambda f: f.__name__)
def test_in_place_at_any_offset(cuda, field):
    """mul_assign reads and writes the same bytes, also where elements
    straddle the 16-byte boundaries."""
    b = field.BYTES
    rng = np.random.default_rng(77 + field.ID)
    for off in (0, 1, 2, 4, 8, 15):
        for n in (1, 3, 31, 33, 500, 5000):
            host, t = _buf(rng, n * b, off)
            c = _coeffs(field, 1, rng)[0] | 2
            want = host.copy()
            orc.mul_assign(field.ID, want, c)
            ops.mul_assign(field, t, c)
            torch.cuda.synchronize()
            assert np.array_equal(t.cpu().numpy(), want), (field.__name__, off, n)


def test_graphs_of_submissions_with_equal_sizes(cuda):
    """One more descriptor and eight fewer pointers give a blob of the same size
    and the same items: a recorded graph must not serve both."""
    field = FIELDS[1]
    rng = np.random.default_rng(5)

    def jobs(shapes):
        out = []
        for k, n in shapes:
            plan = ops.Plan.matrix(field, k, 2, _coeffs(field, 2 * k, rng))
            out.append(fb.Job(plan, [_buf(rng, n, 0)[1] for _ in range(k)], _buf(rng, 2 * n, 0)[1], n, 2))
        return out

    first = jobs([(20, 4096), (5, 4096), (5, 4096)])
    second = jobs([(20, 8192), (20, 4096)])
    runner = fb.Batch()
    for submission in [first] * 4 + [second]:
        runner.run(submission)
    for j in first + second:
        want = torch.zeros_like(j.dst)
        ops.dot_product_matrix_with(want, j.row_len, 2, j.plan, j.srcs)
        assert torch.equal(j.dst, want)
