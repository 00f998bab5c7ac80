"""The launch-shape cache: an entry serves the kernel it was timed for and no
other, and an entry that names no launch shape is timed again."""
from __future__ import annotations

import json

import pytest

pytestmark = pytest.mark.gpu

SMALL, LARGE = [16, 20], [20] * 12   # one size class; nodes on both sides of the node update's two forms


def marked(pkg, cache, precision, sizes=SMALL, shape=(32, 1, 0)):
    """The cache of a tuned ensemble, every entry replaced by a shape that no tuning chooses."""
    with pkg.Batch(sizes, None, pkg.INIT_V2, precision) as b:
        b.autotune(str(cache))
    entries = {k: list(shape) for k in json.loads(cache.read_text())}
    cache.write_text(json.dumps(entries))
    return entries


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_node_update_forms_have_their_own_entries(pkg, tmp_path, precision):
    cache = tmp_path / "tuning.json"
    marked(pkg, cache, precision)
    with pkg.Batch(SMALL, None, pkg.INIT_V2, precision) as b:
        b.autotune(str(cache))
        assert all(b.tuning()[f"class0/{k}"]["block"] == 32 for k in pkg.BATCH_KERNELS)
    with pkg.Batch(LARGE, None, pkg.INIT_V2, precision) as b:
        b.autotune(str(cache))
        assert b.tuning()["class0/node_update"]["block"] in (64, 128, 256)


def test_entries_of_other_kernels_are_not_used(pkg, tmp_path):
    """Entries without the kernels' mark, as files had before it."""
    cache = tmp_path / "tuning.json"
    entries = marked(pkg, cache, 0)
    cache.write_text(json.dumps({k.split("|", 1)[1]: v for k, v in entries.items()}))
    with pkg.Batch(SMALL, None, pkg.INIT_V2, 0) as b:
        b.autotune(str(cache))
        assert all(b.tuning()[f"class0/{k}"]["block"] in (64, 128, 256) for k in pkg.BATCH_KERNELS)


@pytest.mark.parametrize("shape", [(0, 4, 0), (-64, 4, 0), (100, 4, 0), (512, 1, 0), (64, 0, 0), (64, -3, 0)])
def test_bad_entries_are_timed_again(pkg, tmp_path, shape):
    cache = tmp_path / "tuning.json"
    marked(pkg, cache, 0, shape=shape)
    with pkg.Batch(SMALL, None, pkg.INIT_V2, 0) as b:
        b.autotune(str(cache))
        assert all(b.tuning()[f"class0/{k}"]["block"] in (64, 128, 256) for k in pkg.BATCH_KERNELS)
        assert b.run(5) == 5
