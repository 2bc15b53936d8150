"""Plans of the stand-alone calls that the context keeps between calls: a repeated sequence gives
the same bits, a W in use is never handed out twice, a failed W takes its Sigma plans with it,
and kept plans make room when an allocation needs it."""
from dataclasses import replace

import numpy as np
import pytest

from molgw_b200.rigw import Engine, RigwError, efermi_of
from molgw_b200.synth import make_instance, with_window

pytestmark = pytest.mark.gpu


def sequence(eng, inst):
    erpa, egw, w = eng.polarizability_grid_scalapack(inst)
    s = eng.gw_selfenergy_imag_scalapack(w, inst)
    q = eng.qp_solve(inst, s)
    w.release()
    return erpa, egw, s, q.energy_qp_g


def same(a, b):
    return a[0] == b[0] and a[1] == b[1] and np.array_equal(a[2], b[2]) and np.array_equal(a[3], b[3])


def test_repeated_sequences_and_other_inputs():
    a, b = make_instance(5, 40, 90, 8, seed=1), make_instance(5, 40, 90, 8, seed=2)   # same shapes
    c = make_instance(6, 44, 140, 8, seed=3)
    first = []
    for inst in (a, b, c):
        eng = Engine(0)
        first.append(sequence(eng, inst))
        eng.close()
    eng = Engine(0)
    for _ in range(3):                    # the third round replays captured graphs
        for inst, ref in zip((a, b, c), first):
            assert same(sequence(eng, inst), ref)
    eng.close()


def test_two_resident_w_of_one_shape():
    a, b = make_instance(5, 40, 90, 8, seed=1), make_instance(5, 40, 90, 8, seed=2)
    eng = Engine(0)
    ra, rb = sequence(eng, a), sequence(eng, b)
    _, _, wa = eng.polarizability_grid_scalapack(a)
    _, _, wb = eng.polarizability_grid_scalapack(b)
    for _ in range(2):
        assert np.array_equal(eng.gw_selfenergy_imag_scalapack(wa, a), ra[2])
        assert np.array_equal(eng.gw_selfenergy_imag_scalapack(wb, b), rb[2])
    wa.release()
    assert np.array_equal(eng.gw_selfenergy_imag_scalapack(wb, b), rb[2])
    wb.release()
    eng.close()


def test_sigma_on_the_w_of_another_context():
    """Sigma_c from a W that another context of the device made and gives up: the second context
    keeps no plan on its factors, whatever W comes to lie at their place."""
    a, b = make_instance(5, 40, 90, 8, seed=1), make_instance(5, 40, 90, 8, seed=2)
    big = make_instance(8, 60, 260, 16, seed=4)
    one, two = Engine(0), Engine(0)
    ref = {id(x): sequence(one, x)[2] for x in (a, b)}
    for x in (a, b, a):
        _, _, w = one.polarizability_grid_scalapack(x)
        held = two.last_stats()["device_bytes_in_use"]
        for _ in range(3):
            assert np.array_equal(two.gw_selfenergy_imag_scalapack(w, x), ref[id(x)])
            assert np.array_equal(one.gw_selfenergy_imag_scalapack(w, x), ref[id(x)])
        w.release()
        one.autotune([big])                    # drops every kept plan of the first context
    two.qp_solve(a, ref[id(a)])
    assert two.last_stats()["device_bytes_in_use"] <= held + (1 << 20)     # no Sigma plans kept
    one.close()
    assert np.array_equal(sequence(two, b)[2], ref[id(b)])
    two.close()


def test_a_w_outlives_its_context():
    """A context that ends takes the memory of the W it handed out; they can still be released, and
    calls with them are refused."""
    a = make_instance(5, 40, 90, 8, seed=1)
    other = Engine(0)
    ref = sequence(other, a)
    for _ in range(3):
        eng = Engine(0)
        _, _, w = eng.polarizability_grid_scalapack(a)
        _, _, v = eng.polarizability_grid_scalapack(a)
        v.release()
        eng.close()
        with pytest.raises(RigwError):
            other.gw_selfenergy_imag_scalapack(w, a)
        w.release()
        assert same(sequence(other, a), ref)
    other.close()


def test_failed_w_is_not_kept():
    good = make_instance(5, 40, 90, 8, seed=1)
    bad = replace(good, occupation=2.0 - good.occupation, m_ia=good.m_ia * 3.0)   # chi0 > 1: not positive definite
    eng = Engine(0)
    ref = sequence(eng, good)
    for _ in range(2):
        with pytest.raises(RigwError):
            eng.polarizability_grid_scalapack(bad)
        assert same(sequence(eng, good), ref)
    eng.close()


def test_kept_plans_give_way_to_an_allocation():
    small, large = make_instance(5, 40, 90, 8, seed=1), make_instance(8, 60, 260, 16, seed=4)
    probe = Engine(0)
    ref = sequence(probe, large)
    peak = probe.last_stats()["device_bytes_peak"]
    probe.close()
    eng = Engine(0, hbm_budget_bytes=int(peak * 1.02))
    sequence(eng, small)
    sequence(eng, replace(small, nomega=6))
    assert same(sequence(eng, large), ref)
    eng.close()


def vertex_call(eng, name, inst, mf):
    """One of the calls that check their workspace against the HBM budget, or chunk by it."""
    z = efermi_of(inst) + 1j * inst.step_sigma_calc * np.arange(inst.nomega_sigma_calc)
    if name == "density matrix":
        return eng.gw_density_matrix_imag(inst, mf, 8)[0]
    if name == "sox":
        return eng.sox_selfenergy_imag_grid(inst, z)
    _, _, w = eng.polarizability_grid_scalapack(inst)
    try:
        return (eng.g3w2_selfenergy_imag_grid if name == "g3w2" else eng.sosex_selfenergy_imag_grid)(w, inst, mf, z)
    finally:
        w.release()


@pytest.mark.parametrize("name", ["g3w2", "density matrix", "sosex", "sox"])
def test_kept_plans_do_not_count_against_the_budget(name):
    """In a context whose budget is full of kept plans (the W of the call among them) every call
    gives the bits that it gives without a budget."""
    inst, mf = with_window(make_instance(4, 25, 64, 6, seed=31), seed=32)
    inst.nomega_sigma_calc = 9
    other = make_instance(6, 40, 500, 8, seed=5)

    def fill(eng):
        eng.polarizability_grid_scalapack(inst)[2].release()
        sequence(eng, other)
        return eng.last_stats()["device_bytes_in_use"]

    probe = Engine(0)
    used = fill(probe)
    ref = vertex_call(probe, name, inst, mf)
    probe.close()
    eng = Engine(0, hbm_budget_bytes=used + (256 << 10))
    assert fill(eng) == used                   # nothing was dropped
    assert np.array_equal(vertex_call(eng, name, inst, mf), ref)
    eng.close()


def test_a_plan_without_room_for_digits_is_kept():
    """A W whose digit buffers the budget does not hold runs on DMMA, and its repetitions replay the
    kept plans of W and Sigma."""
    inst = make_instance(10, 100, 400, 8, seed=3)
    probe = Engine(0)
    ref = sequence(probe, inst)
    _, _, w = probe.polarizability_grid_scalapack(inst)
    digits = probe.last_stats()["device_bytes_in_use"]
    w.release()
    probe.close()
    eng = Engine(0, hbm_budget_bytes=digits - (12 << 20))
    replayed = []
    for _ in range(4):
        _, _, w = eng.polarizability_grid_scalapack(inst)
        st = eng.last_stats()
        replayed.append(st["graph_replayed"])
        assert st["device_bytes_in_use"] < digits - (12 << 20)
        s = eng.gw_selfenergy_imag_scalapack(w, inst)
        assert np.abs(s - ref[2]).max() <= 1e-12 * np.abs(ref[2]).max()
        replayed.append(eng.last_stats()["graph_replayed"])
        w.release()
    assert replayed == [False] * 2 + [True] * 6
    eng.close()


def test_the_digits_of_a_solved_w_give_way():
    """Three W in a budget that holds two with their digit buffers and one without, which is more
    than three without: all are accepted, and give what they give without a budget."""
    insts = [make_instance(10, 100, 400, 8, seed=s) for s in (3, 4, 5)]
    probe = Engine(0)
    ref = [sequence(probe, x)[2] for x in insts]
    probe.close()
    held = []
    for budget in (0, None):
        eng = Engine(0, hbm_budget_bytes=0 if budget == 0 else held[0] - (1 << 20))
        w = eng.polarizability_grid_scalapack(insts[0])[2]
        held.append(eng.last_stats()["device_bytes_in_use"])
        w.release()
        eng.close()
    assert held[0] - held[1] > (20 << 20)
    eng = Engine(0, hbm_budget_bytes=2 * held[0] + held[1] - (1 << 20))
    w = [eng.polarizability_grid_scalapack(x)[2] for x in insts]
    for x, v, r in zip(insts, w, ref):
        assert np.abs(eng.gw_selfenergy_imag_scalapack(v, x) - r).max() <= 1e-12 * np.abs(r).max()
    for v in w:
        v.release()
    assert np.array_equal(sequence(eng, insts[0])[2], ref[0])
    eng.close()
