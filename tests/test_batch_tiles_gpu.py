"""Work-list tiles of batched stripes whose 4-byte output groups differ but
whose table kernel is one: 5 to 6 and 7 to 8 rows of 2 bytes (3 and 4 groups),
3 and 4 rows of 4 bytes. Each group count keeps a tile of its own, whatever the
order in which the plans were made. Counts of work items, so exact."""
import json

import pytest
import torch

from fgf_b200 import batch as fb
from fgf_b200 import ops, tune
from fgf_b200.fields import Gf16, Gf32

pytestmark = pytest.mark.gpu

# Three sources (one or two go without a split, a class per group count), long
# enough that the built-in split takes several columns per thread.
K, ROW = 3, 4 << 20


@pytest.fixture(autouse=True)
def _clear(cuda):
    tune.clear()
    yield
    tune.clear()


def _jobs(field, rows, order):
    plans = {m: ops.Plan.matrix(field, K, m, range(1, K * m + 1)) for m in order}
    srcs = [torch.zeros(ROW, dtype=torch.uint8, device="cuda") for _ in range(K)]
    return [fb.Job(plans[m], srcs, torch.empty(m * ROW, dtype=torch.uint8, device="cuda"), ROW, m) for m in rows]


def _items(runner, prepared):
    runner.run_prepared(prepared)
    return runner.stats()["items"]


@pytest.mark.parametrize("field,rows", [(Gf16, (6, 8)), (Gf32, (3, 4))], ids=["Gf16", "Gf32"])
@pytest.mark.parametrize("turn", [1, -1], ids=["fewer rows first", "more rows first"])
def test_each_group_count_has_its_own_tile(field, rows, turn):
    b = field.BYTES
    runner = fb.Batch()
    prepared = runner.prepare(_jobs(field, rows, rows[::turn]))
    built_in = _items(runner, prepared)
    grown = []
    for groups in (3, 4):
        tune.set_tile(b, groups, 1)
        grown.append(_items(runner, prepared) - built_in)
        tune.clear()
    for groups in (3, 4):
        tune.set_tile(b, groups, 1)
    assert grown[0] > 0 and grown[1] > 0, (built_in, grown)
    assert _items(runner, prepared) == built_in + sum(grown)


@pytest.mark.parametrize("turn", [1, -1], ids=["fewer rows first", "more rows first"])
def test_the_tuner_measures_every_group_count(tmp_path, turn):
    runner = fb.Batch()
    tune.tune_batch_tiles(runner, runner.prepare(_jobs(Gf16, (6, 8), (6, 8)[::turn])))
    path = tmp_path / "tune.json"
    tune.save(str(path))
    classes = {(t["elem_bytes"], t["groups"]) for t in json.loads(path.read_text())["tiles"]}
    assert classes == {(2, 3), (2, 4)}
