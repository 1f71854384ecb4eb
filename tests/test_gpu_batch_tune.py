"""The autotuner of a Goldilocks batch plan times the default plan too, whose passes run on the tensor
cores and are about twice as fast here as the best explicit choice of columns."""
import json

import pytest

import ziros_b200 as Z
from conftest import rand_field

pytestmark = pytest.mark.gpu

SHAPES = [(1 << 16, 64), (1 << 12, 8)]


def _roots(plan):
    for i, s in enumerate(SHAPES):
        plan.copy_in(i, rand_field(Z.GOLDILOCKS, s, i))
    plan.run()
    return plan.roots()


def test_tuned_plan_keeps_the_tensor_core_passes():
    plan = Z.BatchCommit(SHAPES, field=Z.GOLDILOCKS, p2_width=12, autotune=True)
    assert plan.lde_tune(0) == (0, 0, 0)
    assert (_roots(plan) == _roots(Z.BatchCommit(SHAPES, field=Z.GOLDILOCKS, p2_width=12, autotune=False))).all()


def test_older_cache_entries_do_not_pin_the_butterflies(tmp_path):
    path = tmp_path / "tune.jsonl"
    old = {"key": "lde/1/16/64/1", "kmax": 7, "c_pass": 8, "c_fused": 8, "us": 500}
    path.write_text(json.dumps(old) + "\n")
    plan = Z.BatchCommit(SHAPES, field=Z.GOLDILOCKS, p2_width=12, autotune=True, tune_cache=str(path))
    assert plan.lde_tune(0) == (0, 0, 0)
    # what it chose is in the file, and the next plan takes it from there
    again = Z.BatchCommit(SHAPES, field=Z.GOLDILOCKS, p2_width=12, autotune=False, tune_cache=str(path))
    assert again.info()["tuned_from_cache"] == 1
    assert [again.lde_tune(i) for i in range(2)] == [plan.lde_tune(i) for i in range(2)]
