"""GPU: errors of the eigensolver that do not average out.

The eigenvalues' root sum of squares is the matrix's Frobenius norm.  Each
rounding of a backward-stable solve moves it either way, so the mean over
several dense matrices stays well below eps; a step that rounds one way in
every merge shows as a mean of that size.  And for the smallest orders the
mean error of the eigenvalues is compared with LAPACK's (of the same order: no
more than half as much again allowed)."""
import ctypes as C

import numpy as np
import pytest

from tblite_b200 import capi

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _dense(n, rng):
    a = rng.standard_normal((n, n))
    return 0.5 * (a + a.T)


@pytest.mark.parametrize("n", [200, 256])
def test_norm_is_kept_in_the_mean(n):
    import torch
    rng = np.random.default_rng(n)
    S = torch.eye(n, dtype=torch.float64, device="cuda")
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    c = torch.empty((n, n), dtype=torch.float64, device="cuda")
    lost = []
    for _ in range(16):
        H = _dense(n, rng)
        h = torch.from_numpy(H).cuda()
        assert capi.load_library().tb_sygvd_noalloc(C.c_int32(n), *[C.c_void_p(x.data_ptr()) for x in (h, S, w, c)],
                                                    C.c_void_p(0)) == 0
        f = (H.astype(np.longdouble) ** 2).sum()
        lost.append(float(((w.cpu().numpy().astype(np.longdouble) ** 2).sum() / f - 1) / 2))
    assert abs(np.mean(lost)) <= 0.25 * EPS


@pytest.mark.parametrize("n", [2, 3, 4, 6, 9, 12])
def test_smallest_orders_against_lapack(n):
    rng = np.random.default_rng(n)
    Hs = [_dense(n, rng) for _ in range(200)]
    st, out = capi.sygvd_batch(Hs, [np.eye(n)] * len(Hs))
    assert st == capi.TB_OK
    ours, lapack = [], []
    for H, (w, _) in zip(Hs, out):
        w0, v = np.linalg.eigh(H)
        v = v.astype(np.longdouble)
        exact = (v * (H.astype(np.longdouble) @ v)).sum(0) / (v * v).sum(0)
        scale = np.abs(exact).max()
        ours.append(float(np.abs(w - exact).max() / scale))
        lapack.append(float(np.abs(w0 - exact).max() / scale))
    assert np.mean(ours) <= 1.5 * np.mean(lapack), (np.mean(ours), np.mean(lapack))
