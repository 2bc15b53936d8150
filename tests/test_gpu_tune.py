"""Autotuner: candidates are timed on the caller's batch, the chosen launch
shapes are kept for later batches of the same precision class, and results do
not change beyond summation order.  Tolerances: E_RPA 1e-12 relative,
sigma_calc 1e-11 relative, QP energies 1e-8 eV (FP64); QP energies 1e-6 eV
(split precision)."""
import numpy as np
import pytest

from molgw_b200 import synth
from molgw_b200.rigw import RIGW_BF16X3, RIGW_FP64, RIGW_OZAKI, Engine
from tests.conftest import HA_EV

pytestmark = pytest.mark.gpu


def _batch():
    return [synth.make_instance(no, nv, na, nw, sd) for (no, nv, na, nw, sd) in
            [(4, 30, 70, 8, 71), (9, 80, 200, 16, 72), (6, 44, 300, 16, 73)]]


@pytest.mark.parametrize("precision", [RIGW_FP64, RIGW_BF16X3, RIGW_OZAKI(4)])
def test_autotune_keeps_results_and_reports_candidates(precision):
    eng = Engine(0)
    insts = _batch()
    before = eng.g0w0_batch(insts, precision)
    rep = eng.autotune(insts, precision)
    after = eng.g0w0_batch(insts, precision)
    eng.close()
    assert rep["chi0_rows"] in (64, 128) and rep["update_rows"] in (64, 128)
    # split classes also time an L2-resident frequency group and a group of 8
    assert rep["chains"] in (0, 1, 2, 4, 8)
    assert rep["split_group"] == 0 if precision == RIGW_FP64 else rep["split_group"] >= 0
    assert rep["precision_class"] == (0 if precision == RIGW_FP64 else (1 if precision == RIGW_BF16X3 else 2))
    assert len(rep["candidates"]) >= 3
    assert all(c["total_ms"] > 0 for c in rep["candidates"])
    chosen = [c for c in rep["candidates"]
              if (c["chi0_rows"], c["update_rows"], c["split_group"], c["chains"]) ==
              (rep["chi0_rows"], rep["update_rows"], rep["split_group"], rep["chains"])]
    assert chosen, "the chosen shapes are one of the timed candidates"
    for a, b in zip(before, after):
        assert np.abs(a.energy_qp_g - b.energy_qp_g).max() * HA_EV <= (1e-8 if precision == RIGW_FP64 else 1e-6)
        if precision == RIGW_FP64:
            assert abs(a.erpa - b.erpa) <= 1e-12 * abs(a.erpa)
            assert np.abs(a.sigma_calc - b.sigma_calc).max() <= 1e-11 * np.abs(a.sigma_calc).max()


def test_tuning_applies_to_other_batches_of_the_class():
    eng = Engine(0)
    sample = _batch()[:2]
    rep = eng.autotune(sample, RIGW_FP64)
    other = [synth.make_instance(5, 41, 130, 12, 74)]
    ref = Engine(0)
    a = eng.g0w0_batch(other, RIGW_FP64)[0]
    b = ref.g0w0_batch(other, RIGW_FP64)[0]
    eng.close()
    ref.close()
    assert rep["tuned_ms"] > 0
    assert abs(a.erpa - b.erpa) <= 1e-12 * abs(a.erpa)
    assert np.abs(a.energy_qp_g - b.energy_qp_g).max() * HA_EV <= 1e-8


@pytest.mark.parametrize("naux,nomega,fields", [
    (900, 16, set()),                          # digits in chi0 and in the factorization
    (500, 8, {"panel_group"}),                 # digits in chi0 only
    (200, 8, {"chi0_rows", "panel_group"}),    # DMMA
])
def test_fields_without_effect_are_not_tried(naux, nomega, fields):
    """Row heights of the DMMA chi0 and panel groups of the DMMA factorization are candidates only
    where the batch uses them, and stay at their defaults otherwise."""
    eng = Engine(0)
    rep = eng.autotune([synth.make_instance(8, 90, naux, nomega, 75)], RIGW_FP64)
    eng.close()
    for name in ("chi0_rows", "panel_group"):
        tried = {c[name] for c in rep["candidates"]}
        assert (len(tried) > 1) == (name in fields), (name, tried)
        if name not in fields:
            assert {rep[name]} == tried == {64 if name == "chi0_rows" else 2}


def test_autotune_without_room_for_the_digits():
    """A budget that holds the batch in one plan without its digit buffers only: tuned on DMMA."""
    insts = [synth.make_instance(9, 90, 400, 16, 76)]
    probe = Engine(0)
    probe.g0w0_batch(insts, RIGW_FP64)
    peak = probe.last_stats()["device_bytes_peak"]
    probe.close()
    eng = Engine(0, hbm_budget_bytes=peak - (4 << 20))
    rep = eng.autotune(insts, RIGW_FP64)
    eng.close()
    assert {c["chi0_rows"] for c in rep["candidates"]} == {64, 128}
