"""Operator applies at the limits of their scratch and staging buffers.

* the autotuner times a large block on a part of its columns: the first apply,
  which tunes, and the second are right on every column;
* plane passes over several chunks of columns (BDG_SPEC_CAP_MB) give the bits of
  one chunk;
* the FP32 plane kernels that prefetch (large applies) give the bits of
  one-column applies, which do not;
* host applies below, at and above the largest pinned staging buffer, growing
  and shrinking, before and after such buffers are made (32 calls of a size), and
  from several threads at once, more than there are buffers, give the bits of
  device applies.

Tolerance against the generic kernels: 1e-12 of the largest entry (FP64).
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(bdg, N, cplx, seed):
    rng = np.random.default_rng(seed)
    S = int(np.prod(N))
    H = S if cplx else (N[0] // 2 + 1) * S // N[0]
    dc = bdg.DeviceContext(3, N, [0.5 * n for n in N], cplx)
    wf = rng.standard_normal(S) + (1j * rng.standard_normal(S) if cplx else 0.0)
    dc.set_fields(ltK=1 + rng.random(S), ltM=2 + rng.random(S), wf=wf, pK=0.5 + rng.random(S), pM=0.5 + rng.random(S),
                  mu=0.9, vdd=rng.standard_normal(H), g_ddi=0.6, dipolar=True)
    return dc, S


def _apply(torch, dc, op, prec, x, n):
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    dc.apply_ptr(op, prec, x.data_ptr(), n, y.data_ptr(), n, x.shape[0])
    dc.synchronize()
    return y


@pytest.mark.parametrize("case", [([64, 64, 64], False, 40), ([32, 64, 64], True, 70), ([256, 64, 32], False, 20)],
                         ids=lambda c: "x".join(map(str, c[0])) + ("-z" if c[1] else "-d"))
def test_tuning_on_part_of_a_block(case, bdg, monkeypatch):
    torch = pytest.importorskip("torch")
    N, cplx, ncol = case
    dc, S = _problem(bdg, N, cplx, 4)
    assert ncol > ((1 << 23) + S - 1) // S  # more columns than the tuner times
    n = 2 * S
    x = torch.randn((ncol, n), dtype=torch.complex128 if cplx else torch.float64, device="cuda")
    monkeypatch.setenv("BDG_FFT_PATH", "generic")
    ref = _apply(torch, dc, bdg.OP_LREP, 0, x, n)
    monkeypatch.delenv("BDG_FFT_PATH")
    assert dc.fft_tuning(bdg.OP_LREP, 0)[0] == 0
    first = _apply(torch, dc, bdg.OP_LREP, 0, x, n)
    assert dc.fft_tuning(bdg.OP_LREP, 0)[0] in (1, 2)
    second = _apply(torch, dc, bdg.OP_LREP, 0, x, n)
    scale = float(ref.abs().max())
    assert float((first - ref).abs().max()) < 1e-12 * scale
    assert torch.equal(first, second)  # the last apply of the first call ran by the family chosen
    dc.close()


@pytest.mark.parametrize("case", [([64, 64, 64], False, 7), ([50, 45, 36], False, 40), ([48, 64, 96], True, 3)],
                         ids=lambda c: "x".join(map(str, c[0])) + ("-z" if c[1] else "-d"))
def test_planes_in_chunks(case, bdg, monkeypatch):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("BDG_FFT_PATH", "reg")
    N, cplx, ncol = case
    whole, S = _problem(bdg, N, cplx, 6)
    monkeypatch.setenv("BDG_SPEC_CAP_MB", "15")  # read when a context is made
    parts, _ = _problem(bdg, N, cplx, 6)
    n = 2 * S
    x = torch.randn((ncol, n), dtype=torch.complex128 if cplx else torch.float64, device="cuda")
    out, launches = [], []
    for dc in (whole, parts):
        l0 = bdg.lib().bdgd_launch_count()
        out.append(_apply(torch, dc, bdg.OP_LREP, 0, x, n))
        launches.append(bdg.lib().bdgd_launch_count() - l0)
    assert launches[0] == 4 and launches[1] >= 8 and torch.equal(*out)
    whole.close()
    parts.close()


@pytest.mark.parametrize("case", [([128, 128, 128], False, 3), ([64, 64, 64], False, 16), ([250, 75, 4], False, 140),
                                  ([48, 64, 96], True, 10), ([128, 128, 16], True, 12)],
                         ids=lambda c: "x".join(map(str, c[0])) + ("-z" if c[1] else "-d"))
def test_large_f32_applies_equal_single_columns(case, bdg, monkeypatch):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("BDG_FFT_PATH", "reg")
    N, cplx, ncol = case
    dc, S = _problem(bdg, N, cplx, 9)
    for op, n in ((bdg.OP_LREP, 2 * S), (bdg.OP_TLREP, 2 * S)):
        x = torch.randn((ncol, n), dtype=torch.complex64 if cplx else torch.float32, device="cuda")
        assert x.nbytes * 3.5 > 80 << 20  # x, y and three or two half spectra: above the size that prefetches
        y = _apply(torch, dc, op, 1, x, n)
        y1 = torch.cat([_apply(torch, dc, op, 1, x[j:j + 1].contiguous(), n) for j in range(ncol)])
        assert float(y.abs().max()) > 0.0 and torch.equal(y, y1), op
    dc.close()


@pytest.mark.parametrize("cplx", [False, True], ids=["d", "z"])
def test_host_applies_around_the_pinned_buffers(cplx, bdg, monkeypatch):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("BDG_FFT_PATH", "reg")
    N = [32, 32, 32]
    dc, S = _problem(bdg, N, cplx, 2)
    n = 2 * S
    col = n * (16 if cplx else 8)
    full = (8 << 20) // col  # columns that fill the largest buffer
    rng = np.random.default_rng(1)
    for repeat in (1, 36):
        for ncol in (1, full, full + 1, 2, 3 * full, full - 1, 1):
            X = rng.standard_normal((ncol, n)) + (1j * rng.standard_normal((ncol, n)) if cplx else 0.0)
            want = _apply(torch, dc, bdg.OP_LREP, 0, torch.tensor(X).cuda(), n).cpu().numpy()
            for _ in range(repeat):
                assert np.array_equal(dc.apply_host(bdg.OP_LREP, X), want), ncol
    # buffers given back in between
    bdg.lib().bdgd_trim(dc.ptr)
    for _ in range(36):
        assert np.array_equal(dc.apply_host(bdg.OP_LREP, X), want)
    dc.close()


def test_host_applies_from_threads(bdg, monkeypatch):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("BDG_FFT_PATH", "reg")
    rng = np.random.default_rng(4)
    jobs = []
    for i in range(7):
        dc, S = _problem(bdg, [16, 16, 16 if i % 2 else 32], False, 20 + i)
        X = rng.standard_normal((1 + i, 2 * S))
        jobs.append((dc, X, _apply(torch, dc, bdg.OP_LREP, 0, torch.tensor(X).cuda(), 2 * S).cpu().numpy()))
    bad = []

    def work(dc, X, want, trim):
        for k in range(80):
            if not np.array_equal(dc.apply_host(bdg.OP_LREP, X), want):
                bad.append(k)
            if trim and k % 20 == 19:
                bdg.lib().bdgd_trim(dc.ptr)

    threads = [threading.Thread(target=work, args=j + (i == 3,)) for i, j in enumerate(jobs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    for dc, _, _ in jobs:
        dc.close()
