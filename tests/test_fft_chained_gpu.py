"""Operator applies that follow each other without a wait of the host.

The kernels of an apply are launched programmatically, so a kernel is resident
while the one before it still writes what it reads: the spectra, and x where it
is the y of the apply before.  A chain x -> op x -> op op x ... queued at once
therefore has to give the bits that the same chain gives with a wait of the host
after every apply.  The grids: odd planes and odd nx/2 + 1, where neighbouring
blocks share 32-byte sectors of the spectra, and planes of one and of several
blocks an SM.  The entries are scaled down by the operator's norm through small
fields, so that a chain of eight stays finite.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [
    ([9, 4, 25], False, 3), ([45, 50, 36], False, 5), ([50, 45, 36], False, 5), ([33, 20, 14], True, 4),
    ([16, 16, 16], False, 1), ([64, 64, 64], False, 2), ([48, 48, 48], False, 1), ([128, 128, 32], False, 2),
]


@pytest.mark.parametrize("prec", [0, 1], ids=["f64", "f32"])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g[0])) + ("-z" if g[1] else "-d"))
def test_queued_applies_equal_waited_ones(grid, prec, bdg, monkeypatch):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("BDG_FFT_PATH", "reg")
    N, cplx, ncol = grid
    rng = np.random.default_rng(13)
    S = int(np.prod(N))
    H = S if cplx else (N[0] // 2 + 1) * S // N[0]
    dc = bdg.DeviceContext(3, N, [4.0 * n for n in N], cplx)
    wf = rng.standard_normal(S) + (1j * rng.standard_normal(S) if cplx else 0.0)
    dc.set_fields(ltK=0.5 * rng.random(S), ltM=0.5 * rng.random(S), wf=0.3 * wf, pK=0.5 + rng.random(S),
                  pM=0.5 + rng.random(S), mu=0.9, vdd=0.1 * rng.standard_normal(H), g_ddi=0.6, dipolar=True)
    dt = {(0, False): torch.float64, (1, False): torch.float32, (0, True): torch.complex128,
          (1, True): torch.complex64}[prec, cplx]
    for op, halves in ((bdg.OP_LREP, 2), (bdg.OP_TLREP, 2), (bdg.OP_K, 1), (bdg.OP_M, 1)):
        n = halves * S
        bufs = [[torch.zeros((ncol, n), dtype=dt, device="cuda") for _ in range(9)] for _ in range(2)]
        x = torch.tensor(rng.standard_normal((ncol, n)) + (1j * rng.standard_normal((ncol, n)) if cplx else 0.0)).to(dt).cuda()
        for b in bufs:
            b[0].copy_(x)
        torch.cuda.synchronize()
        for b, wait in zip(bufs, (False, True)):
            for i in range(8):
                dc.apply_ptr(op, prec, b[i].data_ptr(), n, b[i + 1].data_ptr(), n, ncol)
                if wait:
                    dc.synchronize()
            dc.synchronize()
        for q, w in zip(*bufs):
            assert torch.isfinite(torch.view_as_real(w) if cplx else w).all() and torch.equal(q, w), op
        assert float(bufs[1][8].abs().max()) > 0.0
    dc.close()
