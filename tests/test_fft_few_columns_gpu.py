"""Which passes an apply of one to three columns takes when nothing chooses them.

The autotuner times applies of four columns or more.  Below, plane passes serve
the grids where they pay and line passes the others, by a rule on sizes, precision
and operator.  An apply that nothing chooses equals, bit for bit, the one of the
family that the rule names, and launches as many kernels (planes 3, or 4 with a
half of two fields; lines 3 and two for each half); the two families agree to 1e-12 (FP64) and 2e-5
(FP32) of the largest entry.  Also where a block was tuned before: the tuner's
choice of planes is one for many columns.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# grid, complex, precision, operator, columns, family
CASES = [
    ([32, 32, 32], False, 0, "M", 1, "reg"), ([16, 16, 16], False, 1, "K", 1, "reg"), ([128, 128, 128], False, 1, "M", 1, "reg"),
    ([48, 48, 96], False, 0, "L", 3, "reg"), ([64, 32, 64], True, 0, "T", 1, "reg"), ([32, 32, 128], True, 1, "L", 2, "reg"),
    ([128, 128, 16], True, 1, "M", 1, "lines"), ([128, 128, 32], False, 0, "M", 3, "lines"), ([32, 32, 256], False, 0, "M", 1, "lines"),
    ([256, 32, 32], False, 1, "K", 1, "lines"), ([256, 64, 64], True, 1, "T", 1, "lines"), ([64, 64, 64], True, 0, "M", 1, "lines"),
    ([96, 128, 64], True, 1, "M", 1, "lines"),
    # no line passes for these lengths
    ([50, 45, 36], False, 0, "M", 1, "reg"), ([33, 20, 14], True, 1, "L", 2, "reg"),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(["x".join(map(str, c[0])), "z" if c[1] else "d",
                                                                 "f32" if c[2] else "f64", c[3], str(c[4])]))
def test_family_of_few_columns(case, bdg, monkeypatch):
    torch = pytest.importorskip("torch")
    monkeypatch.delenv("BDG_FFT_PATH", raising=False)
    N, cplx, prec, o, ncol, family = case
    op, halves = {"K": (bdg.OP_K, 1), "M": (bdg.OP_M, 1), "L": (bdg.OP_LREP, 2), "T": (bdg.OP_TLREP, 2)}[o]
    rng = np.random.default_rng(3)
    S = int(np.prod(N))
    H = S if cplx else (N[0] // 2 + 1) * S // N[0]
    dc = bdg.DeviceContext(3, N, [0.5 * n for n in N], cplx)
    wf = rng.standard_normal(S) + (1j * rng.standard_normal(S) if cplx else 0.0)
    dc.set_fields(ltK=1 + rng.random(S), ltM=2 + rng.random(S), wf=wf, pK=0.5 + rng.random(S), pM=0.5 + rng.random(S),
                  mu=0.9, vdd=rng.standard_normal(H), g_ddi=0.6, dipolar=True)
    dt = {(0, False): torch.float64, (1, False): torch.float32, (0, True): torch.complex128,
          (1, True): torch.complex64}[prec, cplx]
    n = halves * S
    x = torch.randn((8, n), dtype=dt, device="cuda")

    def apply(path, cols=ncol):
        if path:
            monkeypatch.setenv("BDG_FFT_PATH", path)
        else:
            monkeypatch.delenv("BDG_FFT_PATH", raising=False)
        y = torch.zeros((cols, n), dtype=dt, device="cuda")
        torch.cuda.synchronize()
        l0 = bdg.lib().bdgd_launch_count()
        dc.apply_ptr(op, prec, x.data_ptr(), n, y.data_ptr(), n, cols)
        dc.synchronize()
        return y, bdg.lib().bdgd_launch_count() - l0

    planes, nplanes = apply("reg")
    other, nother = apply("lines")
    assert nplanes == (4 if o in "ML" else 3)
    got, ngot = apply(None)
    want = (planes, nplanes) if family == "reg" else (other, nother)
    assert ngot == want[1] and torch.equal(got, want[0])
    scale = float(planes.abs().max())
    assert float((planes - other).abs().max()) < (2e-5 if prec else 1e-12) * scale
    apply(None, 8)  # tunes, where there is a choice
    path = dc.fft_tuning(op, prec)[0]
    again, nagain = apply(None)
    if path != 2 and nagain != nother:  # the tuner took neither shared-memory stages nor lines
        assert nagain == want[1] and torch.equal(again, want[0])
    dc.close()
