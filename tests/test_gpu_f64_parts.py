"""The persistent FP64 sub-graph solve (k_f64_parts) at the edges of its tiles: parts of one
16-row k-block, one 32- and one 64-edge tile and either side of them, a part above 512 and
parts without core rows, against the oracle's prg_sp2_submatrix per part, with both tile edges
giving the same rows.  (Parts about the extraction's limit: tests/test_gpu_extraction.py.)

Sums of n <= 600 terms over 12 steps: 12 * 600 * 1.1e-16 = 8e-13 between two orders."""
import numpy as np
import pytest

import sp2_oracle as O
import sp2b
from sp2b import modelham as M

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _parts(sizes, n, rng):
    hp = np.zeros(len(sizes) + 1, dtype=np.int64)
    hp[1:] = np.cumsum(sizes)
    # scattered node lists, in no order (core nodes first is only a convention of the rows)
    hidx = np.concatenate([rng.permutation(n)[:s] for s in sizes]).astype(np.int32)
    return hp, hidx


@pytest.mark.parametrize("sizes", [[1, 15, 16, 17, 31, 32, 33], [63, 64, 65, 127, 128, 129, 191],
                                   [512, 95, 2], [600, 97, 40]])
def test_parts_against_oracle_with_both_edges(cuda, sizes):
    rng = np.random.default_rng(sum(sizes))
    n = 640
    h = M.two_band_1d(n, seed=5)
    h_csr = sp2b.dense_to_csr(h)
    emin, emax = O.gershgorin(h)
    pp = [1, 0, 1, 1, 0, 0, 1, 0, 1, 1, 0, 1]
    hp, hidx = _parts(sizes, n, rng)
    lls = np.array([max(1, s // 2) for s in sizes], dtype=np.int32)
    lls[-1] = 0
    vv_ref = np.zeros(len(pp))
    want = []
    for q, s in enumerate(sizes):
        if lls[q] == 0:
            continue
        ix = hidx[hp[q]:hp[q + 1]]
        rho = O.sp2_submatrix(h[np.ix_(ix, ix)], pp, len(pp), vv_ref, emin, emax, int(lls[q]))
        want.append(rho[:lls[q]].reshape(-1))
    want = np.concatenate(want)

    def solve():
        return sp2b.subgraph_sp2_loop(n, h_csr, hp, hidx, lls, pp, len(pp), emin, emax,
                                      precision=sp2b.PREC_FP64, dense=False, core=True)
    _, core, vv = solve()
    assert np.linalg.norm(core - want) <= TOL * np.linalg.norm(want)
    assert np.allclose(vv, np.sqrt(vv_ref), rtol=TOL, atol=0)
    hist = {}
    for s in sizes:
        p = (s + 127) // 128 * 128
        hist[p] = hist.get(p, 0) + 1
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    key = f"subgraph/f64/sm{sms}/" + "".join(f"{p}x{k}," for p, k in sorted(hist.items()))
    ch = sp2b.tune_get(key)[0]
    try:
        sp2b.tune_set(key, 96 - ch)
        _, core2, vv2 = solve()
    finally:
        sp2b.tune_set(key, ch)
    assert np.array_equal(core, core2)
    assert np.allclose(vv2, vv, rtol=TOL, atol=0)


def test_a_wait_that_runs_out_is_reported(cuda):
    """A part's second step waits for a tile that nothing finishes: every thread of the launch
    leaves, the error is on record, and the next solve is sound."""
    from sp2b import _lib
    L = _lib.lib()
    for _ in range(3):
        assert L.sp2b_selftest_solve_timeout(3) == _lib.SP2B_TIMEOUT, _lib.last_error()
    test_parts_against_oracle_with_both_edges(cuda, [63, 64, 65])
