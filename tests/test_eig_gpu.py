"""The eigensolver of the Rayleigh-Ritz step (bdgd_eig_top) against numpy.

All eigenvalues and the nv largest vectors of symmetric matrices at the edges of
the register blocks (32 columns), of the rule that gives the scalar work a warp of
its own (up to 96 columns) and of the range (3, 192): full spectra, graded,
clustered, degenerate, identity, diagonal, split into two blocks, zero, and scaled
to where squares leave the range of a double.

Tolerances: Householder reduction and bisection are backward stable, so values
carry an error of order k eps ||A|| and vectors a residual of that order; 8 k eps
with eps = 2.2e-16 leaves room for the constant.  The reported check is the
residual of the tridiagonal problem, a few eps: within the 2e-15 up to which the
solver takes the result, and large for matrices with NaN or infinities.  Vectors
are of unit length to 1e-13; those of separated values (a gap of 1e-2 ||A||)
orthogonal to 8 k eps / 1e-2.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.2e-16


def _sym(a):
    return 0.5 * (a + a.T)


def _matrices(k, rng):
    q, _ = np.linalg.qr(rng.standard_normal((k, k)))
    h = k // 2
    spectra = {
        "linear": np.linspace(-1.0, 1.0, k), "graded": np.logspace(-12, 0, k), "theta": 1.0 / np.linspace(0.5, 30.0, k) ** 2,
        "clustered": np.r_[1.0 + 1e-13 * rng.standard_normal(h), np.linspace(0.0, 0.5, k - h)],
        "degenerate": np.r_[np.full(k - k // 3, 0.3), np.full(k // 3, 2.0)], "identity": np.ones(k),
        "one large": np.r_[np.logspace(-4, -3.9, k - 1), 1.0],
    }
    out = [(n, _sym((q * e) @ q.T)) for n, e in spectra.items()]
    split = _sym(rng.standard_normal((k, k)))
    split[:h, h:] = split[h:, :h] = 0.0
    ones = np.ones(k - 1)
    out += [("random", _sym(rng.standard_normal((k, k)))), ("diagonal", np.diag(rng.standard_normal(k))), ("split", split),
            ("wilkinson", np.diag(np.abs(np.arange(k) - 0.5 * (k - 1))) + np.diag(ones, 1) + np.diag(ones, -1))]
    base = _sym((q * np.linspace(0.1, 1.0, k)) @ q.T)
    out += [("scaled %g" % s, base * s) for s in (1e-290, 1e-170, 1e-80, 1e80, 1e170, 1e290)]
    return out


class _Eig:
    def __init__(self, bdg, torch):
        self.torch = torch
        self.f, self.work = bdg.lib().bdgd_eig_top, bdg.lib().bdgd_eig_work
        self.f.restype, self.f.argtypes = C.c_int, [C.c_void_p, C.c_void_p, C.c_int, C.c_int] + [C.c_void_p] * 4
        self.work.restype, self.work.argtypes = C.c_size_t, [C.c_int]
        self.dc = bdg.DeviceContext(1, [16], [1.0], False)

    def __call__(self, A, nv):
        torch, k = self.torch, A.shape[0]
        new = lambda *s: torch.full(s, 7.0, dtype=torch.float64, device="cuda")
        a, w, y, chk = torch.tensor(A).cuda(), new(k), new(max(nv, 1), k), new(1)
        work = new(self.work(k) // 8)
        torch.cuda.synchronize()
        rc = self.f(self.dc.ptr, a.data_ptr(), k, nv, w.data_ptr(), y.data_ptr(), work.data_ptr(), chk.data_ptr())
        self.dc.synchronize()
        assert np.array_equal(a.cpu().numpy(), A, equal_nan=True)
        return rc, w.cpu().numpy(), y.cpu().numpy().T, float(chk[0])


@pytest.fixture(scope="module")
def eig(bdg):
    e = _Eig(bdg, pytest.importorskip("torch"))
    yield e
    e.dc.close()


@pytest.mark.parametrize("k", [3, 4, 16, 31, 32, 33, 64, 65, 96, 97, 128, 129, 160, 161, 191, 192])
def test_largest_pairs(k, eig):
    rng = np.random.default_rng(k)
    for name, A in _matrices(k, rng):
        want = np.linalg.eigvalsh(A)
        nrm = np.max(np.abs(want))
        for nv in sorted({1, max(1, k // 3), k}):
            rc, w, Y, chk = eig(A, nv)
            what = (name, nv)
            assert rc == 0 and 0.0 <= chk <= 2e-15, what
            assert np.max(np.abs(w - want)) < 8 * k * EPS * nrm, what
            assert np.max(np.abs(np.linalg.norm(Y, axis=0) - 1.0)) < 1e-13, what
            top = w[k - nv:]
            assert np.max(np.linalg.norm((A / nrm) @ Y - Y * (top / nrm), axis=0)) < 8 * k * EPS, what
            apart = np.abs(top[:, None] - top[None, :]) > 1e-2 * nrm
            assert np.max(np.abs(Y.T @ Y)[apart], initial=0.0) < 800 * k * EPS, what


def test_zero_and_unusable_matrices(eig):
    rc, w, Y, chk = eig(np.zeros((40, 40)), 10)
    assert rc == 0 and np.max(np.abs(w)) < 1e-13 and chk < 1e-14
    assert np.max(np.abs(np.linalg.norm(Y, axis=0) - 1.0)) < 1e-13
    for k in (20, 100):
        for bad in (np.nan, np.inf):
            A = np.eye(k)
            A[5, 3] = A[3, 5] = bad
            assert eig(A, 7)[3] > 1.0
    for k, nv in ((2, 1), (193, 10), (20, 0), (20, 21)):
        assert eig(np.eye(k), nv)[0] == -3


@pytest.mark.parametrize("nev", [4, 20])
def test_solver_result_same_with_syevd(nev, bdg, monkeypatch):
    """BDG_SMALL_EIG=2 leaves the pencil's eigenproblem to syevd, as a declined
    result does; sizeSub 8 and 40 (up to 120 columns)."""
    from bdg_lobpcg_b200 import problems

    cfg = problems.config(16, box=12.0, nev=nev, seed=3)
    psi, mu, _, _, V = problems.ground_state(bdg, cfg)
    out = []
    for mode in ("0", "2"):
        monkeypatch.setenv("BDG_SMALL_EIG", mode)
        p, _ = problems.build(bdg, cfg, psi, mu, V)
        assert p.solve() == 0 and p.converged() >= nev
        out.append((p.eigenvalues()[:nev].copy(), p.stats()["iterations"]))
        p.close()
    assert np.max(np.abs(out[0][0] - out[1][0]) / out[1][0]) < 1e-11
    assert abs(out[0][1] - out[1][1]) <= 5
