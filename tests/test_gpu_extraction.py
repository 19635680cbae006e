"""Core+halo extraction about the limit of its one-pass form (a part's padded size of 2048: eight
rows and the node list in 147 KB of shared memory) in every precision and in the FP64 re-solve,
and entries of H that are not numbers."""
import functools

import numpy as np
import pytest

import sp2_oracle as O
import sp2b
from sp2b import modelham as M

pytestmark = pytest.mark.gpu
N = 2304
PP = [1, 0, 1, 1]


@functools.lru_cache(maxsize=2)
def _job(big):
    """One part of `big` scattered nodes and a small one; core rows and vv of the oracle."""
    rng = np.random.default_rng(big)
    h = M.two_band_1d(N, seed=7)
    emin, emax = O.gershgorin(h)
    sizes, lls = [big, 70], np.array([150, 41], dtype=np.int32)
    hp = np.array([0, big, big + 70], dtype=np.int64)
    hidx = np.concatenate([rng.permutation(N)[:s] for s in sizes]).astype(np.int32)
    vv = np.zeros(len(PP))
    rows = []
    for q in range(2):
        ix = hidx[hp[q]:hp[q + 1]]
        rho = O.sp2_submatrix(h[np.ix_(ix, ix)], PP, len(PP), vv, emin, emax, int(lls[q]))
        rows.append(rho[:lls[q]].reshape(-1))
    return sp2b.dense_to_csr(h), emin, emax, hp, hidx, lls, np.concatenate(rows), np.sqrt(vv)


def _solve(job, prec, tol=0.0, h=None):
    h_csr, emin, emax, hp, hidx, lls, _, _ = job
    _, core, vv = sp2b.subgraph_sp2_loop(N, h or h_csr, hp, hidx, lls, PP, len(PP), emin, emax,
                                         precision=prec, dense=False, core=True, refine_tol=tol)
    return core, vv


@pytest.mark.parametrize("big", [2048, 2049])
def test_parts_about_the_extraction_limit(cuda, big):
    job = _job(big)
    want, vv_want = job[6:]
    norm = np.linalg.norm(want)
    c64, vv = _solve(job, sp2b.PREC_FP64)
    # sums of 2049 terms over four steps: 4 * 2049 * 1.1e-16 = 9e-13 between two orders
    assert np.linalg.norm(c64 - want) <= 1e-12 * norm
    assert np.allclose(vv, vv_want, rtol=1e-12, atol=0)
    # the digit form rounds to 2^-31 once a step
    c8, vv = _solve(job, sp2b.PREC_EXACT_INT8)
    assert np.linalg.norm(c8 - want) <= 1e-7 * norm
    assert np.allclose(vv, vv_want, rtol=1e-5, atol=2e-6)
    # hi + lo: a step errs by 2 (K/16 + 8) 2^-23 (tests/test_gpu_split_small.py), and a
    # step at most doubles what it is given: 15 times that after four
    c16, vv = _solve(job, sp2b.PREC_MIXED_FP16)
    assert np.linalg.norm(c16 - want) <= 15 * 2 * (2176 / 16 + 8) * 2.0 ** -23 * norm
    # the FP64 re-solve of both parts (their sums of (X - X^2)_ii are far above the threshold)
    for prec in (sp2b.PREC_MIXED_FP16, sp2b.PREC_EXACT_INT8):
        again, _ = _solve(job, prec, tol=1e-6)
        assert sp2b.last_subgraph_refined(2)[0] == [0, 1]
        assert np.array_equal(again, c64)


@pytest.mark.parametrize("big", [300, 2049])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_entries_that_are_not_numbers(cuda, big, bad):
    """The FP64 form refuses them; the digit form, whose grid has no such value, keeps them
    inside the parts that hold them.  A sound call afterwards is unaffected."""
    job = _job(big)
    (rp, col, val), hidx, lls = job[0], job[4], job[5]
    good8 = _solve(job, sp2b.PREC_EXACT_INT8)[0]
    node = int(hidx[0])                       # a core row of the large part ...
    small = set(int(i) for i in hidx[big:])
    e = next(e for e in range(rp[node], rp[node + 1]) if col[e] == node)
    v = val.copy()
    v[e] = bad
    with pytest.raises(sp2b.SP2Error):
        _solve(job, sp2b.PREC_FP64, h=(rp, col, v))
    if node not in small:                     # ... that the small one does not hold
        c8 = _solve(job, sp2b.PREC_EXACT_INT8, h=(rp, col, v))[0]
        k = int(lls[0]) * big
        assert np.array_equal(c8[k:], good8[k:])
    assert np.linalg.norm(_solve(job, sp2b.PREC_FP64)[0] - job[6]) <= 1e-12 * np.linalg.norm(job[6])
