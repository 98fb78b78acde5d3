"""3D applies as line passes (BDG_FFT_PATH=lines), and which family ran.

`reg` takes plane passes wherever a plane fits, so the line passes, which the
autotuner can choose and which serve planes too large for an SM and most small
applies, are asked for by name here: every length of their register kernels (16,
32, 48, 64, 96, 128, 256) on each axis, real and complex fields, FP64 and FP32, the
two-field M half as well as the one-field ones, against the generic kernels, and a
64^3 dipolar problem against the oracle.  A random dipolar kernel, not symmetric
under k -> -k, checks the DC and Nyquist terms of real rows.  The number of launches
says which family ran: line passes take three for the y and z axes and two for each
half, plane passes three and one more for a half of two fields, the generic
kernels five.

Tolerance: 1e-12 relative (max-norm) between FP64 results; FP32 results
against the FP64 generic path to 2e-5.
"""
import numpy as np
import pytest

from oracle import bdg_oracle as O

pytestmark = pytest.mark.gpu


def _problem(bdg, N, cplx, seed):
    rng = np.random.default_rng(seed)
    S = int(np.prod(N))
    H = S if cplx else (N[0] // 2 + 1) * S // N[0]
    dc = bdg.DeviceContext(3, N, [0.5 * n for n in N], cplx)
    wf = rng.standard_normal(S) + (1j * rng.standard_normal(S) if cplx else 0.0)
    dc.set_fields(ltK=1 + rng.random(S), ltM=2 + rng.random(S), wf=wf, pK=0.5 + rng.random(S), pM=0.5 + rng.random(S),
                  mu=0.9, vdd=rng.standard_normal(H), g_ddi=0.6, dipolar=True)
    return dc, rng, S


def _apply(bdg, torch, monkeypatch, dc, op, prec, x, path):
    """(y, launches) of one apply by a family."""
    monkeypatch.setenv("BDG_FFT_PATH", path)
    if prec:
        x = x.to(torch.complex64 if x.is_complex() else torch.float32)
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    l0 = bdg.lib().bdgd_launch_count()
    dc.apply_ptr(op, prec, x.data_ptr(), x.shape[1], y.data_ptr(), x.shape[1], x.shape[0])
    dc.synchronize()
    return y, bdg.lib().bdgd_launch_count() - l0


GRIDS = [
    ([16, 32, 48], False), ([32, 48, 64], False), ([48, 64, 96], False), ([64, 96, 16], False), ([96, 128, 32], False),
    ([128, 16, 32], False), ([256, 32, 16], False), ([32, 256, 16], False), ([16, 16, 128], False), ([16, 16, 256], False),
    ([16, 64, 32], True), ([32, 16, 128], True), ([48, 32, 16], True), ([64, 48, 16], True), ([96, 16, 48], True),
    ([128, 96, 16], True), ([256, 16, 16], True), ([16, 256, 16], True), ([16, 128, 96], True), ([16, 16, 256], True),
]


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g[0])) + ("-z" if g[1] else "-d"))
def test_lines_match_generic(grid, bdg, monkeypatch):
    torch = pytest.importorskip("torch")
    N, cplx = grid
    dc, rng, S = _problem(bdg, N, cplx, 11)
    for op, halves in ((bdg.OP_LREP, 2), (bdg.OP_TLREP, 2), (bdg.OP_M, 1), (bdg.OP_K, 1)):
        n = halves * S
        x = torch.tensor(rng.standard_normal((3, n)) + (1j * rng.standard_normal((3, n)) if cplx else 0.0)).cuda()
        ref, _ = _apply(bdg, torch, monkeypatch, dc, op, 0, x, "generic")
        scale = float(ref.abs().max())
        got, launches = _apply(bdg, torch, monkeypatch, dc, op, 0, x, "lines")
        assert launches == 3 + 2 * halves
        assert float((got - ref).abs().max()) < 1e-12 * scale, op
        got, launches = _apply(bdg, torch, monkeypatch, dc, op, 1, x, "lines")
        assert launches == 3 + 2 * halves
        assert float((got - ref).abs().max()) < 2e-5 * scale, op
    dc.close()


def test_lines_against_oracle_64cubed(bdg, monkeypatch):
    torch = pytest.importorskip("torch")
    dim, N, L = 3, [64, 64, 64], [10.0, 10.0, 10.0]
    rng = np.random.default_rng(22)
    oc = O.Ctx(dim, N, L, False)
    O.set_system(oc)
    S = oc.size
    oc.localTermK, oc.localTermM = 1.0 + rng.random(S), 2.0 + rng.random(S)
    oc.precond_sqrtK, oc.precond_sqrtM = 0.5 + rng.random(S), 0.5 + rng.random(S)
    oc.mu = 0.8
    oc.wf = rng.standard_normal(S)
    O.dipolar_set_kernel(oc, 0.7, [0.0, 0.0, 1.0], 4.0)
    oc.dipolar = True
    dc = bdg.DeviceContext(dim, N, L, False)
    dc.set_fields(ltK=oc.localTermK, ltM=oc.localTermM, wf=oc.wf, pK=oc.precond_sqrtK, pM=oc.precond_sqrtM,
                  mu=oc.mu, vdd=oc.longRngInt, g_ddi=oc.g_ddi, dipolar=True)
    X = rng.standard_normal((2, 2 * S))
    for op, ref in ((bdg.OP_LREP, O.matmulLrep), (bdg.OP_TLREP, O.precondLrep)):
        got, _ = _apply(bdg, torch, monkeypatch, dc, op, 0, torch.tensor(X).cuda(), "lines")
        for c in range(X.shape[0]):
            want = ref(oc, X[c])
            assert np.max(np.abs(got[c].cpu().numpy() - want)) < 1e-12 * np.max(np.abs(want)), (op, c)
    dc.close()


# grid, complex, whether a plane of FP64 spectra fits an SM
FITS = [
    ([4, 4, 4], False, True), ([45, 50, 36], False, True), ([50, 45, 36], False, True), ([169, 6, 4], False, True),
    ([128, 128, 4], False, True), ([256, 100, 4], False, True), ([256, 104, 4], False, False), ([121, 100, 4], True, True),
    ([256, 60, 4], True, False), ([128, 128, 4], True, False),
]


@pytest.mark.parametrize("case", FITS, ids=lambda c: "x".join(map(str, c[0])) + ("-z" if c[1] else "-d"))
def test_planes_run_where_they_fit(case, bdg, monkeypatch):
    """`reg` is plane passes there and another family elsewhere; in FP32 all of these fit."""
    torch = pytest.importorskip("torch")
    N, cplx, fits = case
    dc, rng, S = _problem(bdg, N, cplx, 12)
    x = torch.tensor(rng.standard_normal((3, S)) + (1j * rng.standard_normal((3, S)) if cplx else 0.0)).cuda()
    for op, planes in ((bdg.OP_K, 3), (bdg.OP_M, 4)):
        ref, generic = _apply(bdg, torch, monkeypatch, dc, op, 0, x, "generic")
        assert generic >= 5
        got, launches = _apply(bdg, torch, monkeypatch, dc, op, 0, x, "reg")
        assert launches == planes if fits else launches >= 5
        assert float((got - ref).abs().max()) < 1e-12 * float(ref.abs().max())
        assert _apply(bdg, torch, monkeypatch, dc, op, 1, x, "reg")[1] == planes
    dc.close()
