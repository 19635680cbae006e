"""The exact INT8 form's integer arithmetic (residues by FP32 rounding, Chinese remaindering
in FP64, row norms carried from step to step) at sizes about one 32-block and one 128-tile,
against a host model: X rounded to 2^-S and squared exactly with Python integers."""
import numpy as np
import pytest

import sp2_oracle as O
import sp2b
from sp2b import modelham as M

pytestmark = pytest.mark.gpu
MODULI = [255, 253, 251, 247, 241, 239, 233, 229, 256]


def _scale(x, n_pad):
    """The largest S with (2^S max row norm + sqrt(n)/2)^2 < prod/2."""
    prod = 1
    for m in MODULI:
        prod *= m
    lim = np.sqrt(prod / 2.0) * (1.0 - 1e-12)
    r, e = np.sqrt(np.max(np.sum(x * x, axis=1))), 0.5 * np.sqrt(n_pad)
    s = int(np.floor(np.log2((lim - e) / r)))
    while np.ldexp(r, s) + e >= lim:
        s -= 1
    return s


@pytest.mark.parametrize("n", [2, 31, 33, 127, 130])
def test_exact_steps_against_integers(cuda, n):
    h = M.two_band_1d(n, seed=n)
    emin, emax = O.gershgorin(h)
    pp = [1, 0, 1, 0, 0, 1]
    got = sp2b.sp2_alg2_seq_inplace(h, pp, len(pp), emin, emax, precision=sp2b.PREC_EXACT_INT8)
    alpha, beta = -1.0 / (emax - emin), emax / (emax - emin)
    x = alpha * h + beta * np.eye(n)
    vv = []
    for b in pp:
        s = _scale(x, (n + 127) // 128 * 128)
        m = np.rint(np.ldexp(x, s)).astype(np.int64).astype(object)
        x2 = np.array([[float(v) for v in row] for row in m.dot(m)]) * 2.0 ** (-2 * s)
        vv.append(np.linalg.norm(x - x2))
        x = x2 if b == 1 else 2.0 * x - x2
    # the squares are exact but for one rounding to FP64 and X0 for its last bit, which the
    # 2^-S grid (S ~ 35) can turn into one grid step of single elements
    assert np.linalg.norm(got.rho - 2.0 * x) <= 2.0 ** -33 * np.sqrt(n) * np.linalg.norm(x)
    assert np.allclose(got.vv, vv, rtol=1e-8, atol=2.0 ** -32 * n)


@pytest.mark.parametrize("n", [33, 130])
def test_row_norms_above_the_integer_range(cuda, n):
    """Bounds narrower than the spectrum: the iterate grows, and 32-element shares of its row
    norms pass 2^8, where the scale's bound takes the largest share for every one of a row."""
    h = M.two_band_1d(n, seed=n)
    emin, emax = O.gershgorin(h)
    mid, half = 0.5 * (emin + emax), 0.05 * (emax - emin)
    pp = [1, 1, 1]
    got = sp2b.sp2_alg2_seq_inplace(h, pp, len(pp), mid - half, mid + half,
                                    precision=sp2b.PREC_EXACT_INT8)
    x = (mid + half) / (2 * half) * np.eye(n) - h / (2 * half)
    for _ in pp[1:]:
        x = x @ x
    assert np.max(np.sum(x * x, axis=1)) > 2.0 ** 13   # so one of its shares is above 2^8
    x = x @ x
    # 2^S r >= 2^35.9 / (2 * 2) for rows of up to 5 shares: elements are rounded by 2^-35 r, the
    # matrix by e = 2^-35 sqrt(n) r, and each squaring doubles the relative error: 14 e
    assert np.linalg.norm(got.rho - 2.0 * x) <= 2.0 ** -31 * np.sqrt(n) * np.linalg.norm(2.0 * x)
