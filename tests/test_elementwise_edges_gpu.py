"""Products of vectors by bit planes: every length of head and of tail around no,
one, a warp's block of and a few more 16-byte vectors, and the shortest vectors
that take the planes. Against the CPU oracle; exact, tolerance 0."""
import numpy as np
import pytest
import torch

from fgf_b200 import ops
from fgf_b200.fields import FIELDS
from oracle import orc

pytestmark = pytest.mark.gpu

# shortest vectors of the planes kernel, by field name
FIRST = {"Gf16": 1 << 17, "Gf32": 1 << 19, "FanPaar32": 1 << 18, "Gf64": 5 << 18, "FanPaar64": 1 << 20}


@pytest.mark.parametrize("field", list(FIELDS.values()), ids=lambda f: f.__name__)
def test_every_head_and_tail(cuda, field):
    b, block = field.BYTES, 64 * field.BYTES  # vectors of a warp's block
    rng = np.random.default_rng(field.ID + 40)
    first = -(-FIRST.get(field.__name__, 0) // (16 * block)) * block  # whole blocks
    longest = 16 * (first + 2 * block + 3) + 48
    x_h, y_h = (rng.integers(0, 256, size=longest, dtype=np.uint8) for _ in range(2))
    want = np.zeros(longest, np.uint8)
    orc.mul_elementwise(field.ID, want, x_h, y_h)
    x, y, out = (torch.zeros(longest + 64, dtype=torch.uint8, device="cuda") for _ in range(3))
    for off in range(0, 16, b):
        x[off:off + longest].copy_(torch.from_numpy(x_h))
        y[off:off + longest].copy_(torch.from_numpy(y_h))
        for vectors in (first, first + 1, first + block, first + 2 * block + 3):
            for tail in range(0, 16, b):
                n = (16 - off) % 16 + 16 * vectors + tail
                if not n:
                    continue
                out.zero_()
                ops.mul_elementwise(field, out[off:off + n], x[off:off + n], y[off:off + n])
                got = out.cpu().numpy()
                assert np.array_equal(got[off:off + n], want[:n]), (field.__name__, off, vectors, tail)
                assert not got[:off].any() and not got[off + n:].any()
