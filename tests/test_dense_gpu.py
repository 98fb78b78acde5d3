"""Small dense pieces of the Rayleigh-Ritz step on the GPU.

* bdgd_chol_inverse: Z upper triangular with Z^T G Z = I, at the edges of its
  register blocks (32 columns, 16 rows) and of its range (1, 192), for badly
  scaled Gs; the smallest pivot is that of numpy's factor, and not positive for
  an indefinite matrix, a singular one and one with NaN.
  Tolerance: the factor and inverse of a scaled matrix of condition c carry
  errors of a few k c eps; with c <= 50 and k <= 192 that is below 1e-11.
* the solver's result does not depend on whether Cholesky or the
  eigen-decompositions (BDG_SMALL_EIG=1) give the coefficients.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chol(bdg, torch, G, ldg):
    k = G.shape[0]
    f = bdg.lib().bdgd_chol_inverse
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_void_p]
    dc = bdg.DeviceContext(1, [16], [1.0], False)
    g = torch.zeros((k, ldg), dtype=torch.float64)
    g[:, :k] = torch.tensor(G)
    g = g.cuda()
    z = torch.full((k, k), 7.0, dtype=torch.float64, device="cuda")
    p = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = f(dc.ptr, g.data_ptr(), k, ldg, z.data_ptr(), p.data_ptr())
    dc.synchronize()
    dc.close()
    return rc, z.cpu().numpy().T, float(p[0])  # column-major to row index first


@pytest.mark.parametrize("k", [1, 2, 15, 16, 17, 31, 32, 33, 48, 64, 65, 96, 97, 128, 160, 161, 191, 192])
def test_cholesky_coefficients(k, bdg):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(k)
    q, _ = np.linalg.qr(rng.standard_normal((k, k)))
    G = (q * np.linspace(1.0, 50.0, k)) @ q.T if k > 1 else np.array([[3.0]])
    s = 10.0 ** rng.uniform(-6, 6, k)  # column norms of a basis may differ by much
    G = s[:, None] * (0.5 * (G + G.T)) * s[None, :]
    rc, Z, piv = _chol(bdg, torch, G, k + 3)
    assert rc == 0
    assert np.array_equal(Z, np.triu(Z))
    assert np.max(np.abs(Z.T @ G @ Z - np.eye(k))) < 1e-11
    d = 1.0 / np.sqrt(np.diag(G))
    L = np.linalg.cholesky(d[:, None] * G * d[None, :])
    assert abs(piv - np.min(np.diag(L)) ** 2) < 1e-11


def test_cholesky_reports_unusable_matrices(bdg):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(1)
    B = rng.standard_normal((40, 40))
    G = B @ B.T + 40 * np.eye(40)
    bad = G.copy()
    bad[7, 7] = -1.0
    assert _chol(bdg, torch, bad, 40)[2] <= 0.0
    dup = G.copy()
    dup[:, 9] = dup[:, 3]
    dup[9, :] = dup[3, :]
    dup[9, 9] = dup[3, 3]
    assert _chol(bdg, torch, dup, 40)[2] < 1e-12
    nan = G.copy()
    nan[11, 5] = np.nan
    assert _chol(bdg, torch, nan, 40)[2] <= 0.0
    assert _chol(bdg, torch, np.eye(193), 193)[0] == -3


@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_solver_result_same_with_either_coefficients(precision, bdg, monkeypatch):
    from bdg_lobpcg_b200 import problems

    cfg = problems.config(16, box=12.0, nev=4, seed=3)
    psi, mu, _, _, V = problems.ground_state(bdg, cfg)
    out = []
    for eig in ("0", "1"):
        monkeypatch.setenv("BDG_SMALL_EIG", eig)
        p, _ = problems.build(bdg, cfg, psi, mu, V, precision=precision)
        assert p.solve() == 0 and p.converged() >= 4
        out.append((p.eigenvalues()[:4].copy(), p.stats()["iterations"]))
        p.close()
    assert np.max(np.abs(out[0][0] - out[1][0]) / out[1][0]) < 1e-11
    assert abs(out[0][1] - out[1][1]) <= 5
