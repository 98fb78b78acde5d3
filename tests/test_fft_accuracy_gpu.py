"""Accuracy of the plane passes on axes with factors 3 to 13, against 80 bits.

The register DFTs take their constants from compile-time trigonometry; constants a
few units of the last place off are an error that every element shares.  T (weight,
transform, divide, back, weight) of random columns is compared with scipy's
transforms in extended precision.  The generic kernels, whose tables are rounded to
nearest, are the yardstick: both families do the same number of roundings per
point to within a few, so the relative L2 errors may differ by 30%.  In FP32 both
errors are of the single precision's rounding.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [([50, 50, 36], False), ([169, 26, 26], False), ([121, 22, 33], False), ([81, 18, 27], False), ([225, 30, 15], False),
         ([49, 28, 21], False), ([65, 39, 26], True), ([45, 50, 36], True)]


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g[0])) + ("-z" if g[1] else "-d"))
def test_planes_are_as_accurate_as_tables(grid, bdg, monkeypatch):
    torch = pytest.importorskip("torch")
    import scipy.fft as sf

    N, cplx = grid
    rng = np.random.default_rng(6)
    S = int(np.prod(N))
    L = [12.0] * 3
    w, mu = 0.5 + rng.random(S), 0.9
    dc = bdg.DeviceContext(3, N, L, cplx)
    dc.set_fields(ltK=w, ltM=w, wf=w + (0j if cplx else 0.0), pK=w, pM=w, mu=mu)
    x = rng.standard_normal((2, S)) + (1j * rng.standard_normal((2, S)) if cplx else 0.0)
    ld = np.longdouble
    k = [(2 * np.pi / l * sf.fftfreq(n, 1.0 / n)) ** 2 for n, l in zip(N, L)]
    k2 = k[2][:, None, None] + k[1][None, :, None] + k[0][None, None, :]
    pre = 1 / (ld(mu) + k2.astype(ld) / 2)
    wl = w.reshape(N[::-1]).astype(ld)

    def exact(v):
        v = v.reshape(N[::-1]).astype(np.clongdouble)
        y = wl * sf.ifftn(sf.fftn(v * wl) * pre)
        return (y if cplx else y.real).ravel()

    want = np.stack([exact(v) for v in x])
    for prec in (0, 1):
        dt = {(0, False): torch.float64, (1, False): torch.float32, (0, True): torch.complex128,
              (1, True): torch.complex64}[prec, cplx]
        xt = torch.tensor(x).to(dt).cuda()
        err = {}
        for path in ("reg", "generic"):
            monkeypatch.setenv("BDG_FFT_PATH", path)
            y = torch.zeros_like(xt)
            torch.cuda.synchronize()
            l0 = bdg.lib().bdgd_launch_count()
            dc.apply_ptr(bdg.OP_TK, prec, xt.data_ptr(), S, y.data_ptr(), S, 2)
            dc.synchronize()
            assert path == "generic" or bdg.lib().bdgd_launch_count() - l0 == 3  # planes ran
            d = y.cpu().numpy() - want
            err[path] = float(np.sqrt(np.sum(np.abs(d) ** 2) / np.sum(np.abs(want) ** 2)))
        assert err["reg"] < 1.3 * err["generic"], (prec, err)
    dc.close()
