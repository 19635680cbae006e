"""Split-precision products at the sizes where the paired kernel takes 64-column tiles (np up
to 1280, odd multiples of 128 included), just past them, and where it cuts the last wave's
tiles in two (2560, 3072), against an FP64 product: the SP2 step on the split form and the
reverse step {G, X}.

hi + lo keeps 22 bits and the dropped lo lo term is 2^-22 relative.  The FP32 accumulators
take K in chunks of 16, each addition losing at most one unit of the last place of the
partial sum, 2^-23 of it: (K/16 + 8) 2^-23 relative for sums that do not cancel, taken
twice for those that do; K is the padded size, twice that for {G, X}."""
import numpy as np
import pytest

from sp2b import modelham as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 128, 200, 300, 640, 896, 1000, 1152, 1280, 1281, 1408, 2560, 3072])
def test_split_step_and_reverse_step(cuda, n):
    torch = cuda
    from sp2b import _lib
    L = _lib.lib()
    npad = int(L.sp2b_split_dim(n))
    rng = np.random.default_rng(n)
    # a symmetric iterate, spectrum in [0, 1]
    q, _ = torch.linalg.qr(torch.from_numpy(rng.normal(size=(n, n))).cuda())
    x = ((q * torch.from_numpy(rng.uniform(0.0, 1.0, n)).cuda()) @ q.T).cpu().numpy()
    g = M.random_symmetric(n, seed=n)
    st = torch.cuda.current_stream().cuda_stream

    def split(a):
        s = torch.empty(2, npad, npad, dtype=torch.float16, device="cuda")
        f = torch.from_numpy(0.5 * (a + a.T)).float().cuda()
        _lib.check(L.sp2b_dev_f32_to_split(f.data_ptr(), n, s[0].data_ptr(), s[1].data_ptr(), st), "")
        return s, f.double()

    def full(s):
        y = torch.empty(n, n, dtype=torch.float32, device="cuda")
        _lib.check(L.sp2b_dev_split_to_f32(s[0].data_ptr(), s[1].data_ptr(), n, 1.0, y.data_ptr(), st), "")
        return y.double()
    tol = 2.0 * (npad / 16 + 8) * 2.0 ** -23
    xs, xd = split(x)
    gs, gd = split(g)
    for branch in (0, 1):
        y = torch.full((2, npad, npad), float("nan"), dtype=torch.float16, device="cuda")
        _lib.check(L.sp2b_dev_sp2_step_split(xs[0].data_ptr(), xs[1].data_ptr(), y[0].data_ptr(),
                                             y[1].data_ptr(), n, branch, st), "")
        ref = xd @ xd if branch else 2.0 * xd - xd @ xd
        got = full(y)
        assert float((got - ref).norm()) <= tol * float(ref.norm())
        assert torch.equal(got, got.T)
        assert not y.isnan().any()                     # the padding is written (zeros)
        assert float(y[:, n:, :].abs().sum()) == 0.0
        o = torch.full((2, npad, npad), float("nan"), dtype=torch.float16, device="cuda")
        _lib.check(L.sp2b_dev_adjoint_step_split(gs[0].data_ptr(), gs[1].data_ptr(), xs[0].data_ptr(),
                                                 xs[1].data_ptr(), o[0].data_ptr(), o[1].data_ptr(),
                                                 n, branch, st), "")
        anti = gd @ xd + xd @ gd
        ref = anti if branch else 2.0 * gd - anti
        got = full(o)
        assert float((got - ref).norm()) <= 2.0 * tol * float(ref.norm())
        assert torch.equal(got, got.T)


@pytest.mark.parametrize("n", [2300, 2560, 3072, 3328, 3840, 4352])
def test_dense_solve_where_the_last_wave_is_cut(cuda, n):
    """The dense solve at the sizes whose last wave's tiles are cut in two: the sums that a step
    leaves for the next one's branch (its record) against the iterate it wrote, and the
    McWeeny combine product on the same tiles."""
    import ctypes as C

    torch = cuda
    from sp2b import _lib
    L = _lib.lib()
    npad = int(L.sp2b_split_dim(n))
    h = torch.from_numpy(M.two_band_1d(n, seed=n)).cuda()
    rho = torch.empty_like(h)
    st = torch.cuda.current_stream().cuda_stream
    o = _lib.make_opts(precision=_lib.PREC_MIXED_FP16, mcweeny=0, device_ptrs=True, stream=st)
    off = h.abs().sum(0) - h.diagonal().abs()
    emin, emax = float((h.diagonal() - off).min()), float((h.diagonal() + off).max())
    x0 = (emax * torch.eye(n, dtype=h.dtype, device="cuda") - h) / (emax - emin)
    tol = 2.0 * (npad / 16 + 8) * 2.0 ** -23
    for branch in (1, 0):
        pp, vv = np.array([branch], dtype=np.int32), np.zeros(1)
        _lib.check(L.sp2b_sp2_alg2_seq(h.data_ptr(), rho.data_ptr(), n, 0.0, pp.ctypes.data, 1,
                                       vv.ctypes.data, 0, C.byref(o)), "seq")
        recs = np.zeros((2, 9))
        it = C.c_int(0)
        _lib.check(L.sp2b_last_solve_info(C.byref(it), C.byref(it), C.byref(it), C.byref(it),
                                          recs.ctypes.data, 2), "info")
        x = 0.5 * rho
        p = x0 @ x0
        want = p if branch else 2.0 * x0 - p
        assert float((x - want).norm()) <= tol * float(want.norm())
        assert torch.equal(x, x.T)
        # {trx, trx_data, fro2, ..., trp}: sums of what was stored, but for its rounding to hi + lo
        _, trx, fro2, *_, trp = recs[1]
        assert abs(trx - float(x.trace())) <= 2.0 ** -20 * float(x.diagonal().abs().sum())
        assert abs(fro2 - float(x.norm()) ** 2) <= 2.0 ** -20 * float(x.norm()) ** 2
        assert abs(trp - float(p.trace())) <= tol * float(p.trace())
        res = float((x0 - p).norm())
        assert abs(vv[0] - res) <= tol * float(p.norm()) + 2.0 ** -21 * float(x0.norm())
    # a whole solve: the refined density of a gapped system, as tests/test_gpu_dense.py bounds it
    o = _lib.make_opts(precision=_lib.PREC_MIXED_FP16, device_ptrs=True, stream=st)
    o64 = _lib.make_opts(precision=_lib.PREC_FP64, device_ptrs=True, stream=st)
    ref = torch.empty_like(h)
    for out, opts in ((rho, o), (ref, o64)):
        _lib.check(L.sp2b_sp2_alg2(h.data_ptr(), out.data_ptr(), n, 0.0, 0.5, 0, 100, b"Rel", 1e-10, 0,
                                   C.byref(opts), None), "alg2")
    assert float((rho - ref).norm()) / n <= 1e-6
    assert float((rho - ref).abs().max()) <= 1e-6      # in no tile more than elsewhere
    assert torch.equal(rho, rho.T)
