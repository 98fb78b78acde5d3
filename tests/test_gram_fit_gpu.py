"""Gram and update kernels on blocks narrower than a 64-column tile.

The kernels multiply with as many 8-column fragments as a block needs (16, 32,
48 or 64 columns a tile; stages of 64, 32 or 16 rows).  Column counts at the
edges of those, more than one tile with a narrow last one, and row counts that
are no multiple of a stage, against the same product in torch FP64.

Tolerance: a dot product over n rows carries at most n eps relative to
|a|^T |b|; normwise the sums here stay below 1e-13 for n < 10^4 (the other Gram
tests take 1e-12).  FP32 inputs are exact in FP64, so the same bound holds
where they are multiplied as FP64; the integer tensor-core path (above 48
columns) rounds inputs to 31 bits of the column maximum: 1e-8.
"""
import pytest

pytestmark = pytest.mark.gpu


def _torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device for torch")
    return torch


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("k", [1, 8, 15, 16, 17, 32, 33, 48, 49, 64, 65, 80, 112])
def test_gram_narrow_blocks(k, prec, bdg):
    torch = _torch()
    g = torch.Generator(device="cuda").manual_seed(k)
    dt = torch.float32 if prec else torch.float64
    dc = bdg.DeviceContext(1, [16], [1.0], False)
    for half in (20, 1000, 4098):
        ld = 2 * half + 4
        S = torch.randn((k, ld), generator=g, device="cuda", dtype=dt)
        AS = torch.randn((k, ld), generator=g, device="cuda", dtype=dt)
        out = torch.full((4, k, k), 9.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        dc.gram_ptr(prec, False, half, k, S.data_ptr(), ld, AS.data_ptr(), ld, out.data_ptr())
        dc.synchronize()
        u, v = S[:, :half].double(), S[:, half:2 * half].double()
        a = AS[:, :2 * half].double()
        ref = torch.stack([u @ u.T, v @ v.T, v @ u.T, a @ S[:, :2 * half].double().T])
        err = float((out - ref).norm() / ref.norm())
        assert err < (1e-8 if prec and k > 48 else 1e-13), (half, err)
    dc.close()


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("k", [1, 8, 16, 17, 31, 33, 48, 64, 80])
def test_gram_narrow_complex_blocks(k, prec, bdg):
    torch = _torch()
    g = torch.Generator(device="cuda").manual_seed(200 + k)
    dt = torch.float32 if prec else torch.float64
    dc = bdg.DeviceContext(1, [16], [1.0], True)
    for half in (20, 1000, 4098):
        ld = 2 * half + 4
        S, AS = (torch.view_as_complex(torch.randn((k, ld, 2), generator=g, device="cuda", dtype=dt)) for _ in range(2))
        out = torch.full((4, k, k), 9.0, dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
        dc.gram_ptr(prec, True, half, k, S.data_ptr(), ld, AS.data_ptr(), ld, out.data_ptr())
        dc.synchronize()
        wide = torch.complex128
        u, v = S[:, :half].to(wide), S[:, half:2 * half].to(wide)
        ref = torch.stack([u @ u.conj().T, v @ v.conj().T, v @ u.conj().T,
                           AS[:, :2 * half].to(wide) @ S[:, :2 * half].to(wide).conj().T])
        assert float((out - ref).norm() / ref.norm()) < 1e-13, half
    dc.close()


@pytest.mark.parametrize("m,act", [(1, 1), (8, 7), (15, 16), (17, 16), (32, 24), (33, 31), (48, 49), (64, 63), (65, 20), (80, 66)])
def test_update_narrow_outputs(m, act, bdg):
    torch = _torch()
    g = torch.Generator(device="cuda").manual_seed(100 + m)
    dc = bdg.DeviceContext(1, [16], [1.0], False)

    def rnd(*s):
        return torch.randn(s, generator=g, device="cuda", dtype=torch.float64)

    n, ld, k = 1234, 1240, m + act
    X, W, C, D = rnd(m, ld), rnd(act, ld), rnd(m, k), rnd(act, act)
    for beta in (0.0, 1.0):
        Y, Q = rnd(m, ld), rnd(act, ld)
        y0, q0 = Y.clone(), Q.clone()
        torch.cuda.synchronize()
        c = C.data_ptr()
        rc = dc.block_update(0, False, n, ld, [
            (Y.data_ptr(), m, -1.0, beta, [(X.data_ptr(), m, c, k), (W.data_ptr(), act, c + 8 * m, k)]),
            (Q.data_ptr(), act, 1.0, beta, [(W.data_ptr(), act, D.data_ptr(), act)])])
        assert rc == 0
        dc.synchronize()
        ry = -(C[:, :m] @ X + C[:, m:] @ W) + beta * y0
        rq = D @ W + beta * q0
        assert float((Y - ry)[:, :n].norm() / ry[:, :n].norm()) < 1e-13
        assert float((Q - rq)[:, :n].norm() / rq[:, :n].norm()) < 1e-13
        assert torch.equal(Y[:, n:], y0[:, n:]) and torch.equal(Q[:, n:], q0[:, n:])
    dc.close()
