"""Device memory of a batch does not grow with the number of its problems.

A set of cuBLAS and cuSOLVER handles holds hundreds of MB of device memory.
bdg_solve_batch keeps one set for each solve in flight, whatever the number of
problems, and gives all of it back.  The free memory is sampled while batches of
4 and of 12 problems run two at a time.  Bound: with a set for each problem the
longer batch would need eight sets more, so half a set a problem tells the two
apart.  What the device holds after a batch differs by less than one set too
(modules and pools that stay loaded are there from the first batch on).  The
eigenvalues equal those of a solve by itself to 1e-10: their error is of second
order in the residual, 1e-8, whichever FFT family the tuner takes.
"""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _peak_use(bdg, torch, build, n, precision):
    probs = [build(precision) for _ in range(n)]
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    least, stop = [before], threading.Event()

    def sample():
        torch.cuda.set_device(0)
        while not stop.is_set():
            least[0] = min(least[0], torch.cuda.mem_get_info()[0])
            time.sleep(0.001)

    t = threading.Thread(target=sample)
    t.start()
    rcs, _ = bdg.solve_batch(probs, concurrency=2, graphs=True)
    stop.set()
    t.join()
    assert rcs == [0] * n
    lam = [p.eigenvalues().copy() for p in probs]
    for p in probs:
        p.close()
    return before - least[0], before - torch.cuda.mem_get_info()[0], lam


@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_batch_memory_is_flat(precision, bdg):
    torch = pytest.importorskip("torch")
    from bdg_lobpcg_b200 import problems

    cfg = problems.config(16, box=12.0, nev=4, seed=3)
    psi, mu, _, _, V = problems.ground_state(bdg, cfg)

    def build(prec):
        return problems.build(bdg, cfg, psi, mu, V, precision=prec)[0]

    _peak_use(bdg, torch, build, 2, precision)  # loads what the process keeps
    p = build(precision)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    assert p.solve() == 0
    one = free - torch.cuda.mem_get_info()[0]  # workspace and handles of one solve
    want = p.eigenvalues().copy()
    p.close()
    few, left, _ = _peak_use(bdg, torch, build, 4, precision)
    many, left2, lam = _peak_use(bdg, torch, build, 12, precision)
    assert many - few < 4 * one, (one, few, many)
    assert left2 < one, (one, left, left2)
    for e in lam:
        assert np.max(np.abs(e - want) / want) < 1e-10


def test_batch_takes_problems_solved_before(bdg):
    """Problems that hold handles and a workspace of their own, and one that fails."""
    from bdg_lobpcg_b200 import problems

    cfg = problems.config(16, box=12.0, nev=4, seed=3)
    psi, mu, _, _, V = problems.ground_state(bdg, cfg)
    probs = [problems.build(bdg, cfg, psi, mu, V, precision="mixed" if i % 2 else "f64")[0] for i in range(5)]
    for p in probs[:2]:
        assert p.solve() == 0
    want = probs[0].eigenvalues().copy()
    probs[3].set_solver_params(4, 3, 100, 1e-8)  # sizeSub below nev
    for _ in range(2):
        rcs, _ = bdg.solve_batch(probs, concurrency=2, graphs=False)
        assert [r == 0 for r in rcs] == [True, True, True, False, True]
        for i in (0, 1, 2, 4):
            assert np.max(np.abs(probs[i].eigenvalues() - want) / want) < 1e-10
    assert probs[0].solve() == 0
    for p in probs:
        p.close()
