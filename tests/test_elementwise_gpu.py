"""mul_elementwise by bit planes (elementwise.cu) at its edges: blocks of 64 E
16-byte vectors a warp, their remainders, heads and tails of vectors off the
16-byte boundaries, and the lengths where the wide fields change kernels.
Against the CPU oracle; exact, tolerance 0."""
import numpy as np
import pytest
import torch

from fgf_b200 import ops
from fgf_b200.fields import FIELDS
from oracle import orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 8, 3])
@pytest.mark.parametrize("field", list(FIELDS.values()), ids=lambda f: f.__name__)
def test_blocks_and_edges(cuda, field, offset):
    b = field.BYTES
    first = {4: 1 << 18, 8: 1 << 20}.get(b, 0)  # shortest vector of the planes kernel (the Fan-Paar fields')
    block = 1024 * b
    lengths = {first + n for n in (b, 16, block - 16, block, block + 16 + b, 5 * block + 3 * b, 700 * block + 48)}
    if b >= 4:
        lengths |= {first - b, (1 << 19) - b, 1 << 19, (5 << 18) - b, 5 << 18}
    rng = np.random.default_rng(field.ID * 10 + offset)
    for n in sorted(lengths):
        if n > 6 << 20:
            continue
        a_h, b_h = (rng.integers(0, 256, size=n, dtype=np.uint8) for _ in range(2))
        pool = [torch.zeros(n + 48, dtype=torch.uint8, device="cuda") for _ in range(3)]
        out, x, y = (p[offset:offset + n] for p in pool)
        x.copy_(torch.from_numpy(a_h))
        y.copy_(torch.from_numpy(b_h))
        ops.mul_elementwise(field, out, x, y)
        want = np.zeros(n, np.uint8)
        orc.mul_elementwise(field.ID, want, a_h, b_h)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), want), (field.__name__, offset, n)
        assert int(pool[0][:offset].count_nonzero()) == 0 and int(pool[0][offset + n:].count_nonzero()) == 0
