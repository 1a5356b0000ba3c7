"""One call on the byte-table kernel, which also takes the bytes before and after
the 16-byte columns: every head and tail around one and a few columns, and a last
warp with and without columns; rows at the sources' offset and off it, in place,
overwrite and accumulate. Against the CPU oracle; exact, tolerance 0."""
import numpy as np
import pytest
import torch

from fgf_b200 import ops, tune
from fgf_b200.fields import Gf8B, Gf8D
from oracle import orc

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _byte_tables(cuda):
    tune.force("byte")
    yield
    tune.force("auto")


def _place(host, offset):
    hold = torch.zeros(host.size + 64, dtype=torch.uint8, device="cuda")
    hold[offset:offset + host.size] = torch.from_numpy(host).cuda()
    return hold[offset:offset + host.size]


@pytest.mark.parametrize("k,m", [(1, 1), (2, 4), (4, 3), (5, 1), (7, 2), (10, 4), (12, 4), (14, 2)])
def test_heads_and_tails(cuda, k, m):
    field = Gf8D if k % 2 else Gf8B
    rng = np.random.default_rng(k * 10 + m)
    coeffs = [int(c) for c in rng.integers(0, 256, size=k * m)]
    plan = ops.Plan.matrix(field, k, m, coeffs)
    for offset in (0, 1, 4, 7, 13, 15):
        for n in (31, 32, 33, 47, 16 * 5 + 1, 16 * 512 + 7, 16 * 1024 + 30, 16 * 1600 + 3):
            for shift in (0, 3):
                for ovr in (True, False):
                    srcs = [rng.integers(0, 256, size=n, dtype=np.uint8) for _ in range(k)]
                    step = -(-n // 16) * 16 + 16
                    starts = [j * step + shift for j in range(m)]
                    want = rng.integers(0, 256, size=m * step, dtype=np.uint8)
                    dst = _place(want, offset)
                    if ovr:
                        for s in starts:
                            want[s:s + n] = 0
                    orc.mul_add_matrix_scattered(field.ID, want, n, starts, coeffs, srcs)
                    op = ops.dot_product_matrix_scattered_with if ovr else ops.mul_add_matrix_scattered_with
                    op(dst, n, starts, plan, [_place(s, offset) for s in srcs])
                    got = dst.cpu().numpy()
                    assert np.array_equal(got, want), (offset, n, shift, ovr, np.nonzero(got != want)[0][:8])


def test_in_place(cuda):
    rng = np.random.default_rng(1)
    for offset in (0, 5, 15):
        for n in (31, 48, 16 * 1024 + 30):
            want = rng.integers(0, 256, size=n, dtype=np.uint8)
            dst = _place(want, offset)
            orc.mul_assign(Gf8D.ID, want, 0x53)
            ops.mul_assign(Gf8D, dst, 0x53)
            assert np.array_equal(dst.cpu().numpy(), want), (offset, n)
