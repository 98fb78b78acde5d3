"""A Cholesky factor that the Rayleigh-Ritz step rejects moves that step alone.

The start block holds a nearly dependent pair: column m is column 1 plus a
direction d of size 7e-4, so the scaled pivot of its Gram matrix is about 5e-7
(rejected below 1e-6), and d is nearly orthogonal between its u and v parts, so its
Ritz value theta is 1e-5 of the others (a spread above 1e4).  All vectors are
orthogonal to psi0 and, but for the pair, to one another, so d couples to nothing
else and the block is B-positive.  The first step takes the eigen-decompositions;
the later ones, whose factors are good, have to take the Cholesky path again.
Each step of either path launches a fixed number of the library's kernels (11
with Cholesky: the preparation, the factor, four of the eigensolver, two more
factors, two of the coefficients, one of H; 8 with the eigen-decompositions),
so the launches per iteration tell them apart: they equal those of a solve from
a good block to within one.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_rejected_factor_is_not_latched(bdg):
    from bdg_lobpcg_b200 import problems

    cfg = problems.config(16, box=12.0, nev=4, seed=3)
    m = cfg["sizeSub"]
    psi, mu, _, _, V = problems.ground_state(bdg, cfg)
    rng = np.random.default_rng(7)
    S = psi.size
    q, _ = np.linalg.qr(np.column_stack([psi, rng.standard_normal((S, m + 1))]))
    good = q[:, 1:m + 1].T.copy()
    n1, n2 = q[:, m], q[:, m + 1]
    good = np.concatenate([good, good], axis=1)
    bad = good.copy()
    bad[m - 1] = bad[0] + 7e-4 * np.concatenate([n1, 1e-5 * n1 + n2])
    out = {}
    for name, X0 in (("good", good), ("bad", bad)):
        p, _ = problems.build(bdg, cfg, psi, mu, V)
        p.set_initial_block(X0)
        l0 = bdg.lib().bdgd_launch_count()
        assert p.solve() == 0 and p.converged() >= cfg["nev"]
        out[name] = (p.eigenvalues()[:4].copy(), (bdg.lib().bdgd_launch_count() - l0) / p.stats()["iterations"])
        p.close()
    assert np.max(np.abs(out["good"][0] - out["bad"][0]) / out["good"][0]) < 1e-10
    assert abs(out["good"][1] - out["bad"][1]) < 1.0, out
