"""GPU: the blocked overlap factorisation (k_factor) through the generalized
eigensolver's entry points: overlaps with nearly dependent functions, and
overlaps that are not positive definite where a cluster of CTAs owns the
block columns."""
import ctypes as C

import numpy as np
import pytest

from tblite_b200 import capi

pytestmark = pytest.mark.gpu


def _paired_overlap(n, apart, rng):
    """Overlap of n unit vectors in neighbouring pairs, their differences of length about `apart`."""
    h = (n + 1) // 2
    a = rng.standard_normal((2 * n, h))
    a = np.c_[a, a[:, :n - h] + apart * rng.standard_normal((2 * n, n - h))]
    a = a[:, np.argsort(np.r_[np.arange(h) * 2, np.arange(n - h) * 2 + 1])]
    a /= np.linalg.norm(a, axis=0)
    s = a.T @ a
    return 0.5 * (s + s.T)


@pytest.mark.parametrize("n", [64, 65, 97, 138, 256, 300])
def test_nearly_dependent_functions(n):
    # Cholesky by substitution leaves |S - L L^T| of a few n u whatever the condition of
    # its diagonal blocks, so the equations' residual is that times the vectors (which
    # grow as the square root of the condition) times the eigenvalues.  u = eps / 2;
    # rounding errors of the n terms of S C and of the factor add as their square
    # roots: n u |C| |w|, four times that allowed.
    rng = np.random.default_rng(n)
    S = _paired_overlap(n, 10 ** -5.5, rng)
    a = rng.standard_normal((n, n))
    H = 0.5 * (a + a.T)
    st, out = capi.sygvd_batch([H], [S])
    assert st == capi.TB_OK
    w, V = out[0]
    u = 0.5 * np.finfo(float).eps
    scale = np.abs(V).max() * np.abs(w).max()
    V = V.astype(np.longdouble)
    assert np.abs(H @ V - S @ V * w).max() <= 4 * n * u * scale


@pytest.mark.parametrize("n", [65, 192, 256])
def test_not_positive_definite_in_any_block_column(n):
    # alone, a matrix is factorised by a cluster whose ranks own the block columns in turn
    import torch
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    c = torch.empty((n, n), dtype=torch.float64, device="cuda")
    h = torch.diag(torch.arange(n, dtype=torch.float64, device="cuda"))

    def solve(s):
        return capi.load_library().tb_sygvd_noalloc(C.c_int32(n), *[C.c_void_p(x.data_ptr()) for x in (h, s, w, c)],
                                                    C.c_void_p(0))

    for bad in sorted({0, 63, 64, n // 2, n - 1}):
        s = torch.eye(n, dtype=torch.float64, device="cuda")
        s[bad, bad] = -1.0
        assert solve(s) == capi.TB_NOT_SPD
        assert capi.sygvd_batch([np.eye(n)], [s.cpu().numpy()])[0] == capi.TB_NOT_SPD
        s[bad, bad] = 1.0  # the next call starts afresh
        assert solve(s) == capi.TB_OK
        np.testing.assert_allclose(w.cpu().numpy(), np.arange(n), atol=8 * n * np.finfo(float).eps * n, rtol=0)
