"""The persistent FP64 solve (k_f64_solve) at the edges of its tiles, k-blocks and shares:
sizes about one 16-row k-block, one 32- and one 64-edge tile, the tile-edge rule's line
(416), and sizes whose tiles are cut between CTAs, for the plain solve and the response;
and a solve that spans several launches.

FP64 sums of n terms differ by at most n eps relative to the sum of magnitudes between two
orders, and the recursion of a gapped chain does not amplify: with 14 steps of n <= 1100
that is 14 * 1100 * 1.1e-16 = 2e-12."""
import numpy as np
import pytest

import sp2_oracle as O
import sp2b
from sp2b import modelham as M

pytestmark = pytest.mark.gpu
TOL = 2e-12


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 33, 65, 127, 385, 416, 417, 449, 700, 1089])
def test_solve_and_response_against_oracle(cuda, n):
    h = M.two_band_1d(n, seed=n)
    if n == 1:
        h = np.array([[0.0]])      # degenerate bounds: refused
        with pytest.raises(sp2b.SP2Error):
            sp2b.sp2_alg2(h, 1.0)
        return
    bndfil = ((n + 1) // 2) / n
    ref = O.sp2_alg2_genseq(h, bndfil, 0, 100, "None", 1e-10)
    got = sp2b.sp2_alg2_genseq(h, bndfil, 0, 100, "None", 1e-10)
    k = min(len(got.pp), len(ref.pp)) - 2      # the last branches of a converged loop are ties
    assert got.pp[:k] == ref.pp[:k]
    assert np.linalg.norm(got.rho - ref.rho) <= TOL * np.linalg.norm(ref.rho)
    assert np.array_equal(got.rho, got.rho.T)
    assert np.allclose(got.vv[:k], ref.vv[:k], rtol=TOL, atol=TOL)
    h1 = M.random_symmetric(n, seed=n + 1)
    rho_r, rho1_r, _ = O.compute_response_sp2(h, h1, bndfil, 0, 100, "None", 1e-10)
    rho, rho1, _, _ = sp2b.compute_response_sp2(h, h1, bndfil, 0, 100, "None", 1e-10)
    assert np.linalg.norm(rho - rho_r) <= TOL * np.linalg.norm(rho_r)
    # {X, Delta} doubles the terms of each sum
    assert np.linalg.norm(rho1 - rho1_r) <= 2 * TOL * np.linalg.norm(rho1_r)
    assert np.array_equal(rho1, rho1.T)


@pytest.mark.parametrize("n", [300, 600])
def test_submatrix_core_rows_and_bad_input(cuda, n):
    h = M.two_band_1d(n, seed=3)
    emin, emax = O.gershgorin(h)
    pp = [1, 0, 1, 1, 0, 0, 1, 0]
    for core in (1, 33, n - 1, n):
        vv, vv_ref = np.full(8, 0.5), np.full(8, 0.5)
        ref = O.sp2_submatrix(h, pp, 8, vv_ref, emin, emax, core)
        got = sp2b.sp2_submatrix(h, pp, 8, vv, emin, emax, core)
        assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref)
        assert np.allclose(vv, vv_ref, rtol=TOL, atol=0)
    for bad in (np.nan, np.inf):
        hb = h.copy()
        hb[5, 7] = hb[7, 5] = bad
        with pytest.raises(sp2b.SP2Error):
            sp2b.sp2_alg2(hb, 0.5, 0, 100, "None", 1e-10)
    assert np.isfinite(sp2b.sp2_alg2(h, 0.5, 0, 100, "None", 1e-10).rho).all()


def test_solve_of_several_launches(cuda):
    """A 16^3 lattice (n = 4096, about 50 steps, 29 steps a launch): the replay of the
    generated sequence, and plain FP64 products, give the same density."""
    torch = cuda
    n = 4096
    h = M.cubic_3d(16, seed=0)
    got = sp2b.sp2_alg2_genseq(h, 0.5, 0, 100, "None", 1e-10)
    assert got.icount > 32
    emin, emax = O.gershgorin(h)
    x = torch.from_numpy(O.normalize_bounds(h, emin, emax)).cuda()
    for b in got.pp:
        x2 = x @ x
        x = x2 if b == 1 else 2.0 * x - x2
    ref = 2.0 * x.cpu().numpy()
    # rounding near the chemical potential is amplified by up to ~1 / gap, 1e4 here
    assert np.linalg.norm(got.rho - ref) <= 1e-9 * np.linalg.norm(ref)
    seq = sp2b.sp2_alg2_seq(h, got.pp, got.icount)
    assert np.array_equal(seq.rho, got.rho)


@pytest.mark.parametrize("wait", [1, 2])
def test_a_wait_that_runs_out_is_reported(cuda, wait):
    """The waits for another CTA's piece of a tile, or at the grid barrier, run out in the last
    step of a solve: the call says so although other CTAs finished and published that step,
    and the next solve is sound."""
    from sp2b import _lib
    L = _lib.lib()
    for _ in range(3):
        assert L.sp2b_selftest_solve_timeout(wait) == _lib.SP2B_TIMEOUT
        assert "timed out" in _lib.last_error()
    h = M.two_band_1d(448, seed=448)
    ref = O.sp2_alg2(h, 0.5, 0, 100, "None", 1e-10)
    got = sp2b.sp2_alg2(h, 0.5, 0, 100, "None", 1e-10)
    assert np.linalg.norm(got.rho - ref.rho) <= TOL * np.linalg.norm(ref.rho)


@pytest.mark.parametrize("n", [500, 1000, 1300])
def test_recorded_choices_change_no_bit(cuda, n):
    """No recorded decision changes a result: the edge of single FP64 products ("f64-step/...")
    is theirs alone, measured on them, and either one gives the same bits, in a solve and in a
    refinement by FP64 products; the solve's own edge is a rule on n, whatever a decision file
    holds for it."""
    h = M.two_band_1d(n, seed=5)
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    key = f"f64-step/sm{sms}/np{(n + 127) // 128 * 128}"

    def results():
        r = sp2b.sp2_alg2(h, 0.5, 0, 100, "Rel", 1e-10)
        m = sp2b.sp2_alg2(h, 0.5, 0, 100, "None", 1e-10, precision=sp2b.PREC_MIXED_FP16,
                          mcweeny_products=sp2b.MCW_FP64)
        return r.rho, m.rho
    first = results()
    choice, ms = sp2b.tune_get(key)
    assert choice in (64, 128)
    if len(ms) == 2:
        assert ms[(128, 64).index(choice)] == min(ms)
    try:
        for c in (64, 128):
            sp2b.tune_set(key, c)
            sp2b.tune_set(key.replace("step", "solve"), c)
            for a, b in zip(results(), first):
                assert np.array_equal(a, b)
    finally:
        sp2b.tune_set(key, choice)
