"""GPU: k_syev on one CTA and on clusters, k_syev_small below 64 AOs.

The eigensolver's units of work depend on the matrix order alone, so a
structure gives the same bits alone (a cluster of CTAs) and in a batch of
several waves (one CTA per structure).  Orders at the edges of its tiles
(walk shapes change at 224 and 448 rows, leaves at 24 rows, Q in 16-reflector
blocks; the small kernel's leaves at 13, 26 and 52 rows, its padded row strides
at multiples of 16, rows past one warp's 32 columns) are compared with numpy through the allocation-free entry point.
"""
import ctypes as C

import numpy as np
import pytest

from tblite_b200 import capi
from tblite_b200 import geometry as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 13, 14, 15, 16, 26, 27, 31, 32, 33, 48, 51, 53, 62, 63, 64, 65, 97, 112, 129, 193, 223, 224, 225, 226, 240, 255, 256])
def test_orders_at_tile_edges(n):
    import torch
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    H = 0.5 * (a + a.T)
    if n in (33, 51, 129):  # threefold degenerate
        H = np.diag(np.repeat(np.arange(n / 3.0), 3))
    b = 0.1 * rng.standard_normal((n, n))
    S = np.eye(n) + b @ b.T / n
    h, s = torch.from_numpy(H).cuda(), torch.from_numpy(S).cuda()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    c = torch.empty((n, n), dtype=torch.float64, device="cuda")
    st = capi.load_library().tb_sygvd_noalloc(C.c_int32(n), *[C.c_void_p(x.data_ptr()) for x in (h, s, w, c)],
                                              C.c_void_p(0))
    assert st == 0, capi.last_error()
    W, V = w.cpu().numpy(), c.cpu().numpy()
    li = np.linalg.inv(np.linalg.cholesky(S))
    scale = max(1.0, np.abs(H).sum(axis=1).max())
    tol = 8 * n * np.finfo(float).eps  # backward stable: a few n eps of the norm
    np.testing.assert_allclose(W, np.linalg.eigvalsh(li @ H @ li.T), atol=tol * scale, rtol=0)
    np.testing.assert_allclose(V.T @ S @ V, np.eye(n), atol=tol, rtol=0)
    np.testing.assert_allclose(H @ V, S @ V * W, atol=tol * scale, rtol=0)


@pytest.mark.parametrize("n", [65, 97, 130, 200, 256])
def test_runs_of_close_eigenvalues(n):
    # chains of deflated pairs, shorter and longer than the 32 entries tested at once
    import torch
    rng = np.random.default_rng(7 * n)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    lam = np.concatenate([1.0 + 1e-16 * np.arange(n // 2), np.repeat([2.0, 3.0], (n - n // 2) // 3),
                          4.0 + 1e-13 * np.arange(n - n // 2 - 2 * ((n - n // 2) // 3))])
    H = (q * lam) @ q.T
    H = 0.5 * (H + H.T)
    h, s = torch.from_numpy(H).cuda(), torch.eye(n, dtype=torch.float64, device="cuda")
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    c = torch.empty((n, n), dtype=torch.float64, device="cuda")
    st = capi.load_library().tb_sygvd_noalloc(C.c_int32(n), *[C.c_void_p(x.data_ptr()) for x in (h, s, w, c)],
                                              C.c_void_p(0))
    assert st == 0, capi.last_error()
    W, V = w.cpu().numpy(), c.cpu().numpy()
    tol = 8 * n * np.finfo(float).eps  # backward stable: a few n eps of the norm (4)
    np.testing.assert_allclose(W, np.linalg.eigvalsh(H), atol=4 * tol, rtol=0)
    np.testing.assert_allclose(V.T @ V, np.eye(n), atol=tol, rtol=0)
    np.testing.assert_allclose(H @ V, V * W, atol=4 * tol, rtol=0)


def test_cluster_and_one_cta_give_the_same_bits(gpu_calc):
    rng = np.random.default_rng(17)
    mols = [g.water_cluster(k, rng) for k in (11, 16, 22, 37, 38, 64)]
    # 68, 224, 446, 452, 662 AOs, and 194, 386, 392, 770, 794 with leaves at two depths
    mols += [g.alkane(k, rng) for k in (11, 37, 74, 75, 110, 32, 64, 65, 128, 132)]
    fill = g.water_clusters(700, seed=9, nmin=11, nmax=14)     # several waves: one CTA each
    batch = gpu_calc.singlepoint_batch(mols + fill, solver=1)
    few = gpu_calc.singlepoint_batch(mols, solver=1)
    for i, m in enumerate(mols):
        alone = gpu_calc.singlepoint_batch([m], solver=1)[0]
        for r in (batch[i], few[i]):
            assert alone["status"] == r["status"] == 0
            assert alone["energy"] == r["energy"] and alone["iterations"] == r["iterations"]
            np.testing.assert_array_equal(alone["qat"], r["qat"])


def test_mixed_form_cluster_and_one_cta_give_the_same_bits(gpu_calc):
    # k_syev (68, 224, 446 AOs) and the small solvers (2, 24, 48 AOs)
    rng = np.random.default_rng(23)
    mols = [g.water_cluster(k, rng) for k in (4, 8)] + [g.alkane(k, rng) for k in (11, 37, 74)]
    mols.append(g.Molecule(np.array([0, 0], np.int32), np.array([[0, 0, 0], [0, 0, 1.4]], float)))
    fill = g.water_clusters(400, seed=3, nmin=11, nmax=12)
    batch = gpu_calc.singlepoint_batch(mols + fill, precision=1, solver=1)
    plain = gpu_calc.singlepoint_batch(mols, solver=1, accuracy=0.01)
    for m, rb, rp in zip(mols, batch, plain):
        alone = gpu_calc.singlepoint_batch([m], precision=1, solver=1)[0]
        assert alone["status"] == rb["status"] == rp["status"] == 0
        assert alone["energy"] == rb["energy"] and alone["iterations"] == rb["iterations"]
        np.testing.assert_array_equal(alone["qat"], rb["qat"])
        assert abs(alone["energy"] - rp["energy"]) < 1e-6  # the mixed form's bound


# AOs of batches that k_syev (two CTAs per SM) solves: from one CTA per structure
# throughout, and with clusters of two for the largest (tests/test_plan.py holds the plans)
NARROW_LARGE = [446, 384, 228, 224, 222, 132, 66]


def narrow_sizes(fill):
    return NARROW_LARGE + [6 * (11 + i * 62 // (fill - 1)) for i in range(fill)]


@pytest.mark.parametrize("fill", [900, 700])
def test_narrow_kernel_gives_the_bits_of_the_wide_one(gpu_calc, fill):
    rng = np.random.default_rng(fill)
    sizes = narrow_sizes(fill)
    mols = [g.alkane((n - 2) // 6, rng) if n % 6 == 2 else g.water_cluster(n // 6, rng) for n in sizes]
    batch = gpu_calc.singlepoint_batch(mols, solver=1)
    assert [r["nao"] for r in batch] == sizes
    probe = list(range(len(NARROW_LARGE))) + [len(NARROW_LARGE) + i for i in range(0, fill, 90)]
    for i in probe:  # alone: a cluster of the wide kernel
        alone = gpu_calc.singlepoint_batch([mols[i]], solver=1)[0]
        assert alone["status"] == batch[i]["status"] == 0
        assert alone["energy"] == batch[i]["energy"] and alone["iterations"] == batch[i]["iterations"]
        np.testing.assert_array_equal(alone["qat"], batch[i]["qat"])


def test_narrow_kernel_at_its_largest_orders():
    rng = np.random.default_rng(449)
    pairs = []
    for n in (449, 448, 225, 224):
        a = rng.standard_normal((n, n))
        b = 0.1 * rng.standard_normal((n, n))
        pairs.append((0.5 * (a + a.T), np.eye(n) + b @ b.T / n))
    many = pairs * 74  # 296 matrices: enough for the narrow kernel
    st, out = capi.sygvd_batch([p[0] for p in many], [p[1] for p in many])
    assert st == capi.TB_OK
    for i, (h, s) in enumerate(pairs):
        st, alone = capi.sygvd_batch([h], [s])
        assert st == capi.TB_OK
        for j in (i, 4 * 73 + i):
            np.testing.assert_array_equal(out[j][0], alone[0][0])
            np.testing.assert_array_equal(out[j][1], alone[0][1])
