"""The plane passes of 3D operator applies against the runtime-sized kernels.

BDG_FFT_PATH=reg runs an apply as plane passes where the grid allows it and
`generic` as runtime-sized shared-memory stages.  The grids here are the edges
of the plane passes: the shortest lengths (4), lengths that split into unequal
or prime factors, an odd y extent (rows then go in unpaired), an odd or even x
extent (no Nyquist column, or one), switch sizes below and above 8, the cubes
with compiled-in sizes, one plane that just fits an SM and one that does not
(the apply then takes another family), leading dimensions that are odd, and
one column.  The dipolar kernel is random, so the DC and Nyquist columns of
real rows are checked too.

Tolerance: FP64 1e-12 relative in the maximum norm, as between the other pass
families; FP32 against FP64 2e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [
    ([4, 4, 4], False), ([9, 4, 25], False), ([10, 16, 9], False), ([22, 26, 13 * 2], False), ([26, 22, 39], False),
    ([45, 50, 36], False), ([50, 45, 36], False), ([13 * 13, 6, 4], False), ([16, 16, 16], False), ([32, 32, 32], False),
    ([48, 48, 48], False), ([96, 96, 96], False), ([256, 100, 4], False), ([256, 104, 4], False),
    ([4, 9, 16], True), ([33, 20, 14], True), ([96, 64, 6], True), ([121, 100, 4], True), ([256, 60, 4], True),
]


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g[0])) + ("-z" if g[1] else "-d"))
def test_planes_match_generic(grid, bdg, monkeypatch):
    torch = pytest.importorskip("torch")
    N, cplx = grid
    rng = np.random.default_rng(5)
    S = int(np.prod(N))
    H = S if cplx else (N[0] // 2 + 1) * S // N[0]
    dc = bdg.DeviceContext(3, N, [0.5 * n for n in N], cplx)
    wf = rng.standard_normal(S) + (1j * rng.standard_normal(S) if cplx else 0.0)
    dc.set_fields(ltK=1 + rng.random(S), ltM=2 + rng.random(S), wf=wf, pK=0.5 + rng.random(S), pM=0.5 + rng.random(S),
                  mu=0.9, vdd=rng.standard_normal(H), g_ddi=0.6, dipolar=True)

    def apply(op, prec, x, path):
        monkeypatch.setenv("BDG_FFT_PATH", path)
        y = torch.zeros_like(x)
        torch.cuda.synchronize()
        dc.apply_ptr(op, prec, x.data_ptr(), x.shape[1], y.data_ptr(), x.shape[1], x.shape[0])
        dc.synchronize()
        return y

    for op, halves in ((bdg.OP_LREP, 2), (bdg.OP_TLREP, 2), (bdg.OP_M, 1), (bdg.OP_K, 1), (bdg.OP_DIPCONV, 1)):
        ncol = 1 if op == bdg.OP_M else 3
        ld = halves * S + (1 if op == bdg.OP_LREP else 0)  # an odd leading dimension for Lrep
        x = torch.tensor(rng.standard_normal((ncol, ld)) + (1j * rng.standard_normal((ncol, ld)) if cplx else 0.0)).cuda()
        ref = apply(op, 0, x, "generic")
        got = apply(op, 0, x, "reg")
        scale = float(ref.abs().max())
        assert float((got - ref).abs().max()) < 1e-12 * scale, op
        assert float(got[:, halves * S:].abs().max() if ld > halves * S else 0.0) == 0.0  # nothing past a column
        got32 = apply(op, 1, x.to(torch.complex64 if cplx else torch.float32), "reg")
        assert float((got32 - ref).abs().max()) < 2e-5 * scale, op
    dc.close()


# large applies prefetch into L2 (both plane kernels where a plane fills an SM):
# the arithmetic is the same, so every column equals that of a one-column apply,
# which is too small to prefetch, bit for bit
PREFETCH = [
    ([128, 128, 128], False, 3, "KM"), ([64, 64, 64], False, 8, "KML"), ([250, 75, 4], False, 70, "KML"),
    ([256, 60, 4], True, 50, "KML"), ([48, 64, 96], True, 5, "KML"),
]


@pytest.mark.parametrize("case", PREFETCH, ids=lambda c: "x".join(map(str, c[0])) + ("-z" if c[1] else "-d"))
def test_large_applies_equal_single_columns(case, bdg, monkeypatch):
    torch = pytest.importorskip("torch")
    N, cplx, ncol, ops = case
    monkeypatch.setenv("BDG_FFT_PATH", "reg")
    rng = np.random.default_rng(8)
    S = int(np.prod(N))
    H = S if cplx else (N[0] // 2 + 1) * S // N[0]
    dc = bdg.DeviceContext(3, N, [0.5 * n for n in N], cplx)
    wf = rng.standard_normal(S) + (1j * rng.standard_normal(S) if cplx else 0.0)
    dc.set_fields(ltK=1 + rng.random(S), ltM=2 + rng.random(S), wf=wf, pK=0.5 + rng.random(S), pM=0.5 + rng.random(S),
                  mu=0.9, vdd=rng.standard_normal(H), g_ddi=0.6, dipolar=True)
    for o in ops:
        op, n = {"K": (bdg.OP_K, S), "M": (bdg.OP_M, S), "L": (bdg.OP_LREP, 2 * S)}[o]
        x = torch.randn((ncol, n), dtype=torch.complex128 if cplx else torch.float64, device="cuda")
        y, y1 = torch.zeros_like(x), torch.zeros_like(x)
        torch.cuda.synchronize()
        dc.apply_ptr(op, 0, x.data_ptr(), n, y.data_ptr(), n, ncol)
        for j in range(ncol):
            dc.apply_ptr(op, 0, x[j].data_ptr(), n, y1[j].data_ptr(), n, 1)
        dc.synchronize()
        assert float(y.abs().max()) > 0.0 and torch.equal(y, y1), o
    dc.close()
