"""FP64 chi0 from int8 digit products (molgw_b200/csrc/digit_gemm.cu) at the edges of its
tiles and chunks, against NumPy in FP64.

Tolerance: an FP64 sum of K products of entries with row norms |A_p|, |B_q| is off by at most
about K u |A_p| |B_q|, u = 2^-53; chi = eps^-1 - 1 is a contraction of that error (eps >= 1), so
|d chi| <= 2 K u max diag(eps) with both sides' errors, and ten times that is allowed.  The row
exponents and the layout of the digits would show as errors of 1e-2 and more."""
import ctypes as C

import numpy as np
import pytest

from molgw_b200.rigw import Engine, RigwError, WPol
from molgw_b200.synth import GWInstance, make_instance

pytestmark = pytest.mark.gpu


def molecule(nocc, nvirt, naux, nomega, seed=0, decades=0.0):
    rng = np.random.default_rng(seed)
    energy = np.concatenate([np.sort(rng.uniform(-1.1, -0.3, nocc)), np.sort(rng.uniform(0.02, 1.5, nvirt))])
    m = rng.standard_normal((nocc, nvirt, naux)) * (0.35 / np.sqrt(nocc * nvirt + naux))
    m *= 10.0 ** (-decades * rng.random(naux))[None, None, :]
    ms = rng.standard_normal((2, nocc + nvirt, naux)) * 0.01
    occ = np.concatenate([np.full(nocc, 2.0), np.zeros(nvirt)])
    return GWInstance(nocc=nocc, nvirt=nvirt, naux=naux, nomega=nomega, energy=energy, occupation=occ, m_ia=m,
                      m_sigma=ms, nsemin=nocc, nsemax=nocc + 1)


def reference(inst, omega):
    no, nv = inst.nocc, inst.nvirt
    de = (inst.energy[no:][None, :] - inst.energy[:no][:, None]).ravel()
    docc = (inst.occupation[:no][:, None] - inst.occupation[no:][None, :]).ravel()
    m = inst.m_ia.reshape(no * nv, -1)
    out, top = [], 0.0
    for w in omega:
        eps = np.eye(inst.naux) + m.T @ (m * (2.0 * docc * de / (w * w + de * de))[:, None])
        top = max(top, np.abs(np.diag(eps)).max())
        out.append(np.linalg.inv(eps) - np.eye(inst.naux))
    return np.array(out), top


def check(engine, inst):
    from molgw_b200.rigw import imag_grid
    erpa, egw, w = engine.polarizability_grid_scalapack(inst)
    chi = w.chi()
    w.release()
    ref, top = reference(inst, imag_grid(inst.nomega)[0])
    tol = 10 * 2 * inst.nocc * inst.nvirt * 2.0 ** -53 * top
    assert np.abs(chi - ref).max() <= tol, (np.abs(chi - ref).max(), tol)
    return erpa


@pytest.mark.parametrize("nocc,nvirt,naux,nomega", [
    (8, 64, 384, 3),       # whole tiles, K a multiple of the k-tile, smallest of the range
    (9, 57, 385, 2),       # one row beyond a 128-row block, one transition beyond a k-tile
    (7, 90, 511, 17),      # one row short of four blocks; more frequencies than one factor block
    (11, 61, 513, 2),      # an odd number of row blocks: the last pair has one
    (30, 547, 390, 2),     # 16410 transitions: two INT32 chunks, the second of one k-tile
])
def test_tile_and_chunk_edges(engine, nocc, nvirt, naux, nomega):
    check(engine, molecule(nocc, nvirt, naux, nomega, seed=naux))


def test_rows_of_very_different_size(engine):
    check(engine, molecule(10, 70, 400, 3, seed=5, decades=150.0))


OMEGA = (1.0e-4, 1.0e-2, 1.0)       # low frequencies, where D_w has the range of the gaps


def wide_gaps(nvirt, naux, decades, seed):
    """Two occupied states, gaps over ``decades`` decades, amplitudes that grow as their roots: what
    a small gap beside core states gives."""
    rng = np.random.default_rng(seed)
    inst = molecule(2, nvirt, naux, len(OMEGA), seed=seed)
    inst.energy[:] = np.concatenate([[-1.0e-5, 0.0], np.sort(10.0 ** (2.0 - decades * rng.random(nvirt)))])
    de = inst.energy[2:][None, :] - inst.energy[:2][:, None]
    inst.m_ia[:] = rng.standard_normal(inst.m_ia.shape) * np.sqrt(de / (4.0 * de.size))[:, :, None]
    return inst


def dominated(nvirt, naux, seed):
    """Three transitions carry every auxiliary function, the others 1e-4 of them."""
    rng = np.random.default_rng(seed)
    inst = molecule(2, nvirt, naux, len(OMEGA), seed=seed)
    m = 1.0e-4 * rng.standard_normal((2 * nvirt, naux))
    m[rng.integers(0, 2 * nvirt, (3, naux)), np.arange(naux)[None, :]] = 1.0
    inst.m_ia[:] = (0.3 * m).reshape(inst.m_ia.shape)
    return inst


def exact_chi(inst, omega):
    """eps^-1 - 1 in extended precision: the FP64 inverse and one Newton step."""
    no, nv, n = inst.nocc, inst.nvirt, inst.naux
    de = (inst.energy[no:][None, :] - inst.energy[:no][:, None]).ravel().astype(np.longdouble)
    docc = (inst.occupation[:no][:, None] - inst.occupation[no:][None, :]).ravel()
    m = inst.m_ia.reshape(no * nv, n).astype(np.longdouble)
    eye, out = np.eye(n, dtype=np.longdouble), []
    for w in omega:
        w = np.longdouble(w)
        eps = eye + m.T @ (m * (2.0 * docc * de / (w * w + de * de))[:, None])
        x = np.linalg.inv(eps.astype(float)).astype(np.longdouble)
        out.append(x + x @ (eye - eps @ x) - eye)
    return np.array(out)


def chi_and_bytes(eng, inst):
    """chi at OMEGA, and the device memory held with that W."""
    p, keep = eng.make_problem(inst, freq=(np.array(OMEGA), np.ones(len(OMEGA))))
    h = C.c_void_p()
    eng._check(eng._lib.rigw_polarizability_imag(eng._h, C.byref(p), None, None, C.byref(h)), "polarizability")
    w = WPol(eng, h, inst.naux, len(OMEGA))
    used = eng.last_stats()["device_bytes_in_use"]
    chi = w.chi()
    w.release()
    return chi, used


def chi_on_dmma(inst, bytes_with_digits):
    """The same W from a context without room for its digits."""
    eng = Engine(0, hbm_budget_bytes=bytes_with_digits - (1 << 20))
    chi, used = chi_and_bytes(eng, inst)
    eng.close()
    assert used < bytes_with_digits - (1 << 20)
    return chi


@pytest.mark.parametrize("nvirt", [300, 1100])
@pytest.mark.parametrize("kind", [1.0, 3.0, 5.0, "dominated"])
def test_no_further_from_64_bits_than_dmma(nvirt, kind):
    """The digits are no further from extended precision than the FP64 sums of the DMMA kernel,
    however wide the range of the gaps or of the entries: what both sides share (the rounding of
    eps and the factorization) is in both errors, and 10% covers that it is not the same rounding.
    M D_w and M as operands, whose scales are not bounded by sqrt(eps_pp eps_qq), give 2 times the
    error at three decades and 10 times at five; without the ninth level of digit products the
    dominated rows give 2 times the error."""
    inst = dominated(nvirt, 400, seed=11) if kind == "dominated" else wide_gaps(nvirt, 400, kind, seed=11)
    eng = Engine(0)
    chi, used = chi_and_bytes(eng, inst)
    eng.close()
    dmma = chi_on_dmma(inst, used)
    ref = exact_chi(inst, OMEGA)
    err = [float(np.sqrt(np.mean((c - ref) ** 2))) for c in (chi, dmma)]
    print(err)
    assert err[0] <= 1.1 * err[1], err


def test_negative_factors_are_left_to_dmma():
    """Some D_w < 0: bit for bit the result of the DMMA kernel, in a plan that ran with positive
    factors before and runs with them afterwards."""
    good, bad = molecule(10, 70, 400, 3, seed=6), molecule(10, 70, 400, 3, seed=6)
    bad.occupation[9], bad.occupation[10] = 0.5, 1.5
    eng = Engine(0)
    ref, used = chi_and_bytes(eng, good)
    dmma = chi_on_dmma(bad, used)
    for _ in range(2):                         # the second round replays captured graphs
        assert np.array_equal(chi_and_bytes(eng, bad)[0], dmma)
        assert np.array_equal(chi_and_bytes(eng, good)[0], ref)
    eng.close()


def test_negative_factors(engine):
    """A few inverted transitions (D < 0) that leave eps positive definite."""
    inst = molecule(10, 70, 400, 3, seed=6)
    inst.occupation[9], inst.occupation[10] = 0.5, 1.5
    check(engine, inst)


def test_frequency_groups_and_mixed_batch(engine):
    """A batch in which some problems take the digit products and some the DMMA kernel gives
    what each gives alone."""
    insts = [make_instance(4, 30, 70, 8, seed=41), make_instance(9, 80, 400, 16, seed=42),
             make_instance(12, 100, 520, 12, seed=43)]
    alone = [engine.g0w0(i) for i in insts]
    for a, b in zip(alone, engine.g0w0_batch(insts)):
        assert abs(a.erpa - b.erpa) <= 1e-12 * abs(a.erpa)
        assert np.abs(a.sigma_calc - b.sigma_calc).max() <= 1e-12 * np.abs(a.sigma_calc).max()


def sigma_reference(inst, omega, weight, z):
    no, nv = inst.nocc, inst.nvirt
    de = (inst.energy[no:][None, :] - inst.energy[:no][:, None]).ravel()
    docc = (inst.occupation[:no][:, None] - inst.occupation[no:][None, :]).ravel()
    m = inst.m_ia.reshape(no * nv, -1)
    out, erpa = np.zeros((2, z.size), complex), 0.0
    for w, wt in zip(omega, weight):
        eps = np.eye(inst.naux) + m.T @ (m * (2.0 * docc * de / (w * w + de * de))[:, None])
        for s in range(2):
            v = np.einsum("pi,pi->p", inst.m_sigma[s], np.linalg.solve(eps, inst.m_sigma[s].T).T) - \
                np.sum(inst.m_sigma[s] ** 2, axis=1)
            x = z[:, None] - inst.energy[None, :]
            out[s] -= wt / (2 * np.pi) * ((1.0 / (x + 1j * w) + 1.0 / (x - 1j * w)) @ v)
        erpa += wt / (2 * np.pi) * (np.linalg.slogdet(eps)[1] + inst.naux - np.trace(eps))
    return out, erpa


@pytest.mark.parametrize("nocc,nvirt,naux,nomega", [
    # on DMMA: too few frequencies for their panels
    (9, 60, 769, 3),
    (8, 70, 1030, 5),
    (10, 65, 1100, 2),
    (6, 86, 3200, 1),
    # as many frequencies as the digit products take up (frequencies x panels^2 >= 800)
    (9, 60, 769, 17),      # seven panels in groups of two: the last group has one
    (8, 70, 1030, 10),     # nine panels, one column block of the right-hand sides ends early
    (10, 65, 1100, 10),    # M columns that end inside a 128-column block
    (6, 86, 3200, 2),      # 25 panels in groups of four: the last group has one
])
@pytest.mark.parametrize("qp_only", [False, True])
def test_factorization_updates_by_digits(engine, nocc, nvirt, naux, nomega, qp_only):
    """The updates between panel groups on digit products: chi from the identity part and
    Sigma_c from the M columns.  |U^-T M|^2 - |M|^2 is a difference of sums of naux terms, each
    rounded: 1e-13 of the largest Sigma covers naux u sqrt(naux) for these sizes.  The integrand of
    E_RPA is a difference of two sums of naux terms of about 1, on either side; a sum in blocks
    rounds log2(naux) times, by up to u naux: 4 log2(naux) u naux sum |weight| / (2 pi)."""
    from molgw_b200.rigw import imag_grid
    inst = molecule(nocc, nvirt, naux, nomega, seed=naux)
    if not qp_only:
        check(engine, inst)
    om, wt = imag_grid(nomega)
    out = engine.g0w0(inst, qp_only=qp_only)
    ef = 0.5 * (inst.energy[nocc - 1] + inst.energy[nocc])
    ref, erpa = sigma_reference(inst, om, wt, ef + 1j * inst.step_sigma_calc * np.arange(inst.nomega_sigma_calc))
    assert np.abs(out.sigma_calc - ref).max() <= 1e-13 * np.abs(ref).max()
    assert abs(out.erpa - erpa) <= 4 * np.log2(naux) * 2.0 ** -53 * naux * np.abs(wt).sum() / (2 * np.pi)


@pytest.mark.parametrize("sizes,nomega", [
    ((900, 1000, 420), 7),     # two that factorize on DMMA alone and on digit products together
    ((780, 700, 500), 18),     # one that takes digits alone and leaves them beside the others
])
def test_a_batch_takes_up_the_digits_together(engine, sizes, nomega):
    """The factorization of a batch takes digit products, beside problems too small for them, or none,
    and gives what each problem gives alone."""
    insts = [make_instance(8, 90, n, nomega, seed=n) for n in sizes]
    for one, both in zip([engine.g0w0(i) for i in insts], engine.g0w0_batch(insts)):
        assert abs(one.erpa - both.erpa) <= 1e-10 * abs(one.erpa)
        assert np.abs(one.sigma_calc - both.sigma_calc).max() <= 1e-12 * np.abs(one.sigma_calc).max()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_input_is_reported(engine, bad):
    inst = molecule(9, 64, 384, 2, seed=8)
    inst.m_ia[3, 5, 17] = bad
    with pytest.raises(RigwError):
        engine.g0w0(inst)
    check(engine, molecule(9, 64, 384, 2, seed=8))      # the context stays usable


def test_without_room_for_the_digits(engine):
    """A budget that holds one frequency without the digit buffers (about 115 MB) but not with
    them (205 MB): the problem still runs, on DMMA."""
    inst = molecule(30, 547, 390, 2, seed=9)
    ref = engine.g0w0(inst)
    small = Engine(0, hbm_budget_bytes=160 << 20)
    out = small.g0w0(inst)
    small.close()
    assert abs(out.erpa - ref.erpa) <= 1e-10
    assert np.abs(out.sigma_calc - ref.sigma_calc).max() <= 1e-11 * np.abs(ref.sigma_calc).max()


def test_a_small_batch_does_without_digits_before_it_is_cut():
    """A budget that holds the batch in one plan without the digit buffers only: one plan, kept."""
    inst = make_instance(9, 90, 400, 16, seed=12)
    eng = Engine(0)
    ref = eng.g0w0(inst)
    peak = eng.last_stats()["device_bytes_peak"]
    eng.close()
    eng = Engine(0, hbm_budget_bytes=peak - (4 << 20))
    for k in range(3):
        out = eng.g0w0(inst)
        st = eng.last_stats()
        assert (st["waves"], st["graph_replayed"]) == (1, k > 0)
        assert np.abs(out.sigma_calc - ref.sigma_calc).max() <= 1e-11 * np.abs(ref.sigma_calc).max()
    eng.close()


def test_every_budget_finds_chunks_that_fit():
    """Chunks of fewer frequencies keep all their operand planes at once and can need more memory than
    longer ones (digits 57 MB a frequency here, up to 18 of them at once or 8 in turn): no budget
    above that of one frequency is refused."""
    inst = molecule(30, 547, 390, 90, seed=9)
    eng = Engine(0)
    ref = eng.g0w0(inst, qp_only=True)
    peak = eng.last_stats()["device_bytes_peak"]
    eng.close()
    for budget in range(240 << 20, peak, 10 << 20):
        eng = Engine(0, hbm_budget_bytes=budget)
        out = eng.g0w0(inst, qp_only=True)
        eng.close()
        assert np.abs(out.sigma_calc - ref.sigma_calc).max() <= 1e-11 * np.abs(ref.sigma_calc).max()
