"""Fan-Paar arithmetic on the host, whose byte level goes by logarithms: every
inverse of the byte level and decode matrices of the wider ones, against the
oracle. No GPU needed."""
import numpy as np
import pytest

from fgf_b200 import codes
from fgf_b200.fields import FIELDS
from oracle import orc

FP8, FP16, FP32 = (FIELDS[i] for i in (orc.FP8, orc.FP16, orc.FP32))


def test_every_byte_inverse():
    k, m = 240, 16
    c = codes.cauchy_matrix(FP8, m, k, k)  # inverses of 1 .. 255
    for i in range(m):
        for j in range(k):
            assert c[i][j] == orc.inv(FP8.ID, (k + i) ^ j), (i, j)


@pytest.mark.parametrize("field,k,m", [(FP8, 20, 6), (FP16, 12, 5), (FP32, 9, 4)], ids=lambda x: getattr(x, "__name__", x))
def test_decode_matrices(field, k, m):
    c = codes.cauchy_matrix(field, m, k)
    rng = np.random.default_rng(field.ID)
    for _ in range(20):
        erased = sorted(int(x) for x in rng.choice(k + m, size=m, replace=False))
        survivors = [i for i in range(k + m) if i not in erased]
        got = codes.decode_matrix(field, c, survivors, erased)
        want = orc.decode_matrix(field.ID, np.array(c, dtype=np.uint32), survivors, erased)
        assert got == [int(want[e][t]) for t in range(k) for e in range(m)], erased
