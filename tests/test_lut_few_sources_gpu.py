"""Calls of one and two sources of the 2- and 4-byte fields, which take a table
word per 4 / E rows instead of a tower split: every number of rows of a launch
and one more, lengths around whole columns, a warp's step and several steps of
a CTA, every kind of offset, single and batched. Against the CPU oracle; exact,
tolerance 0."""
import numpy as np
import pytest

from fgf_b200 import tune
from fgf_b200.fields import FIELDS
from test_lut_gpu import _run

pytestmark = pytest.mark.gpu

LENGTHS = (1, 8, 31, 33, 62, 65, 1000, 9001)  # elements


@pytest.fixture(autouse=True)
def _tables_only(cuda):
    tune.force("nibble")
    yield
    tune.force("auto")


@pytest.mark.parametrize("batched", [False, True], ids=["single", "batch"])
@pytest.mark.parametrize("offsets", ["aligned", "rows", "any"])
@pytest.mark.parametrize("field", [f for f in FIELDS.values() if f.BYTES in (2, 4)], ids=lambda f: f.__name__)
def test_every_number_of_rows(field, offsets, batched):
    b = field.BYTES
    rng = np.random.default_rng(field.ID * 10 + len(offsets) + batched)
    for k in (1, 2):
        for m in range(1, 16 // b + 2):
            for i, n in enumerate((LENGTHS[(m + k) % 8], LENGTHS[(3 * m + 4 * k + 1) % 8])):
                so, base, ro = [0] * k, 0, [0] * m
                if offsets != "aligned":
                    base = int(rng.integers(0, 16))
                    ro = [int(x) * b for x in rng.integers(0, 16 // b, size=m)]
                if offsets == "any":
                    so = [int(x) for x in rng.integers(0, 16, size=k)]
                _run(field, k, m, n * b, so, base, ro, bool((m + i) & 1), i == 0, batched, rng)
