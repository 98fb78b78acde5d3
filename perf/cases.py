"""Performance cases of the library: what programs that use it have it do.

A program sets a dipolar trap up, solves for its lowest BdG modes (`Problem.solve`), and, where it brings an
eigensolver or a propagator of its own, calls the block entry points on device memory: operator applies
(`DeviceContext.apply_ptr`), the Gram blocks of a Rayleigh-Ritz step (`gram_ptr`) and the basis update
(`block_update`), or the single-column host operators of the reference API (`OperatorContext.apply`).  Grids run
from 16 to 128 points an axis, the lengths of the benchmark configurations (32, 64, 128) among others of the same
range, smooth ones, uneven ones and odd ones; blocks hold from one column to the 64 of a 128^3 solve.
"""
import math

import numpy as np
import torch

import bdg_lobpcg_b200 as B
from bdg_lobpcg_b200 import problems

REAL = {"f64": torch.float64, "f32": torch.float32, "c128": torch.float64, "c64": torch.float32}
CPLX = {"f64": False, "f32": False, "c128": True, "c64": True}
OPS = {"lrep": B.OP_LREP, "tlrep": B.OP_TLREP, "m": B.OP_M, "k": B.OP_K}
RC, MU, BOX = 8.0, 9.0, 20.0  # dipolar cutoff radius, chemical potential, box length per axis


def listed():
    def apply(name, op, n, dtype, cols):
        return {"name": name, "kind": "apply", "op": op, "nx": n[0], "ny": n[1], "nz": n[2], "dtype": dtype, "cols": cols}

    return [
        # one column of host memory through the reference's own operator call: a port of its callers and tests
        {"name": "host_lrep_32", "kind": "host", "op": "lrep", "nx": 32, "ny": 32, "nz": 32, "dtype": "f64"},
        # one device column: a step of the conjugate gradients and propagators that run on M
        apply("m_48_one_column", "m", (48, 48, 48), "f64", 1),
        # the block of a 64^3 solve (sizeSub 32)
        apply("lrep_64_f64", "lrep", (64, 64, 64), "f64", 32),
        # the preconditioner on the block of a 128^3 solve (sizeSub 64): the largest FP64 apply
        apply("tlrep_128_f64", "tlrep", (128, 128, 128), "f64", 64),
        # the same block in the FP32 phase of a mixed-precision solve
        apply("lrep_128_f32", "lrep", (128, 128, 128), "f32", 64),
        # a complex condensate in an uneven box
        apply("lrep_48x64x96_c128", "lrep", (96, 64, 48), "c128", 24),
        # axes that are no powers of two, one of them odd: a box chosen by its physics
        apply("lrep_50x45x36_f64", "lrep", (50, 45, 36), "f64", 16),
        # Rayleigh-Ritz blocks of [X, P, W] of a 32^3 solve (sizeSub 16) and of a 128^3 solve (sizeSub 64)
        {"name": "gram_32_k48", "kind": "gram", "rows": 32 ** 3, "k": 48, "dtype": "f64"},
        {"name": "gram_128_k192", "kind": "gram", "rows": 128 ** 3, "k": 192, "dtype": "f64"},
        # X, AX, P, AP of the next iteration of a 64^3 solve (sizeSub 32, 24 active columns)
        {"name": "update_64_m32", "kind": "update", "rows": 2 * 64 ** 3, "m": 32, "act": 24},
        # whole solves: the 32^3 configuration in FP64, the 64^3 one in mixed precision
        {"name": "solve_32_f64", "kind": "solve", "grid": 32, "nev": 8, "eps_dd": 0.5, "mixed": False},
        {"name": "solve_64_mixed", "kind": "solve", "grid": 64, "nev": 16, "eps_dd": 0.7, "mixed": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(n):
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def draw(rng):
    kind = rng.choice(["apply"] * 6 + ["gram"] * 2 + ["update"] * 2 + ["solve", "host"])
    if kind in ("apply", "host"):
        style = rng.choice(["cube", "smooth", "smooth", "any"])
        if style == "cube":
            n = [rng.choice([16, 32, 48, 64, 96, 128])] * 3
        elif style == "smooth":
            n = [rng.choice([16, 20, 24, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 80, 90, 96, 100, 108, 120, 128])
                 for _ in range(3)]
        else:  # any length the library takes: no prime factor above 13
            n = [rng.choice([k for k in range(16, 81) if _smooth(k)]) for _ in range(3)]
        size = n[0] * n[1] * n[2]
        op = rng.choice(["lrep", "lrep", "tlrep", "m", "k"])
        if kind == "host":
            return {"kind": "host", "op": op, "nx": n[0], "ny": n[1], "nz": n[2], "dtype": rng.choice(["f64", "c128"])}
        most = max(1, min(64, 64 * 128 ** 3 // (8 * size) if style == "any" else 32 * 128 ** 3 // size))
        return {"kind": "apply", "op": op, "nx": n[0], "ny": n[1], "nz": n[2],
                "dtype": rng.choice(["f64", "f64", "f32", "c128", "c64"]), "cols": _log(rng, 1, most)}
    if kind == "gram":
        dtype = rng.choice(["f64", "f64", "f32", "c128"])
        rows = _log(rng, 16 ** 3, 96 ** 3)
        return {"kind": "gram", "rows": rows, "k": _log(rng, 12, 120 if dtype == "c128" else 192), "dtype": dtype}
    if kind == "update":
        m = _log(rng, 8, 64)
        return {"kind": "update", "rows": 2 * _log(rng, 16 ** 3, 96 ** 3), "m": m, "act": rng.randint(max(1, m // 2), m)}
    grid = rng.choice([16, 24, 32, 40, 48])
    return {"kind": "solve", "grid": grid, "nev": rng.randint(4, 12), "eps_dd": round(rng.uniform(0.1, 0.7), 3),
            "mixed": rng.random() < 0.3}


# ---- fields of a trapped condensate (x fastest, the library's layouts) ----------------------------------------------
def _fields(case):
    n = (case["nx"], case["ny"], case["nz"])
    cplx = CPLX[case["dtype"]]
    ax = [(np.arange(k) - 0.5 * k) * BOX / k for k in n]
    Z, Y, X = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    V = 0.5 * (X * X + Y * Y + 4.0 * Z * Z)
    g, gdd = 1000.0, 500.0
    dens = np.exp(-(X * X + Y * Y + 4.0 * Z * Z) / 8.0) + 0.0
    dens /= dens.sum() * (BOX ** 3 / dens.size)
    psi = np.sqrt(dens)
    if cplx:
        psi = psi * np.exp(1j * (0.7 + 0.3 * X))
    ltK = V + g * dens - MU
    ltM = ltK + 2.0 * g * dens
    kk = [(2.0 * math.pi / BOX * np.where(np.arange(k) <= k // 2, np.arange(k), np.arange(k) - k)) ** 2 for k in n]
    kx2 = kk[0] if cplx else kk[0][: n[0] // 2 + 1]
    k2 = kk[2][:, None, None] + kk[1][None, :, None] + kx2[None, None, :]
    with np.errstate(all="ignore"):
        q = np.sqrt(k2) * RC
        vdd = (3.0 * kk[2][:, None, None] / k2 - 1.0) * (1.0 + 3.0 * np.cos(q) / q ** 2 - 3.0 * np.sin(q) / q ** 3)
    vdd[0, 0, 0] = 0.0
    pre = [1.0 / np.sqrt(np.fmax(1e-8, a)) for a in (ltK, ltM)]
    pre = [np.fmin(p, 10.0) for p in pre]
    return {"psi": psi, "ltK": ltK, "ltM": ltM, "pK": pre[0], "pM": pre[1], "vdd": vdd, "k2": k2, "gdd": gdd}


_context = {}


def _device_context(key, make):
    """The context of one grid.  A program keeps one and runs its blocks through it in turn, whatever it gets as input:
    so the states of one case share theirs (and its stream); the context of another case is not kept beside it."""
    if key not in _context:
        _context.clear()
        _context[key] = make()
    return _context[key]


def _operators(case):
    """Device context of the case's grid with the condensate's fields."""
    f = _fields(case)
    cplx = CPLX[case["dtype"]]
    ctx = B.DeviceContext(3, [case["nx"], case["ny"], case["nz"]], [BOX] * 3, cplx)
    ctx.set_fields(f["ltK"].ravel(), f["ltM"].ravel(), f["psi"].ravel(), f["pK"].ravel(), f["pM"].ravel(), MU,
                   f["vdd"].ravel(), f["gdd"], True)
    return ctx


def _dense(cplx):
    """Context for the dense block calls, which take any: its stream and workspaces."""
    return _device_context(("dense", cplx), lambda: B.DeviceContext(3, [16, 16, 16], [BOX] * 3, cplx))


def _halves(case):
    return 2 if case["op"] in ("lrep", "tlrep") else 1


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(shape, dtype, seed):
    """Columns as the eigensolver starts from: N(0, 1) entries."""
    x = torch.randn(tuple(shape) + ((2,) if CPLX[dtype] else ()), generator=_gen(seed), device="cuda", dtype=REAL[dtype])
    return torch.view_as_complex(x) if CPLX[dtype] else x


def _block(rows, k, dtype, seed):
    """Basis columns of falling size, as [X, P, W] holds them."""
    x = _randn((k, rows), dtype, seed)
    s = torch.logspace(0.0, -3.0, k, dtype=REAL[dtype], device="cuda")
    return x * s[:, None]


def _host_column(case, seed):
    """One column of host memory, made from the seed."""
    n = _halves(case) * case["nx"] * case["ny"] * case["nz"]
    r = np.random.default_rng(seed)
    return r.standard_normal(n) + 1j * r.standard_normal(n) if CPLX[case["dtype"]] else r.standard_normal(n)


def _update_inputs(case, seed):
    """Blocks X, P, W, AX, AP, AW and coefficients C_x ((m + 2 act) x m), C_p ((2 act) x act), column-major."""
    m, a, rows = case["m"], case["act"], case["rows"]
    blocks = [_randn((c, rows), "f64", seed * 16 + i) for i, c in enumerate((m, a, a, m, a, a))]
    k = m + 2 * a
    cx = _randn((m, k), "f64", seed * 16 + 6) / math.sqrt(k)
    cp = _randn((a, 2 * a), "f64", seed * 16 + 7) / math.sqrt(2 * a)
    return blocks, cx, cp


def _solve_config(case, seed):
    """The trap of the benchmark family; the seed moves its coupling a little and makes the start block."""
    cfg = problems.config(case["grid"], eps_dd=case["eps_dd"], nev=case["nev"], seed=seed,
                          g=1000.0 + 5.0 * (seed % 17), box=16.0 if case["grid"] <= 32 else 24.0)
    return cfg


def prepare(case, seed):
    kind = case["kind"]
    if kind == "apply":
        n = [case["nx"], case["ny"], case["nz"]]
        ctx = _device_context(tuple(n) + (CPLX[case["dtype"]],), lambda: _operators(case))
        x = _randn((case["cols"], _halves(case) * n[0] * n[1] * n[2]), case["dtype"], seed)
        prec = B.F32 if case["dtype"] in ("f32", "c64") else B.F64
        return {"kind": kind, "ctx": ctx, "op": OPS[case["op"]], "prec": prec, "x": x, "y": torch.empty_like(x)}
    if kind == "host":
        f = _fields(case)
        ctx = B.OperatorContext(3, [case["nx"], case["ny"], case["nz"]], [BOX] * 3, CPLX[case["dtype"]])
        for name, a in (("localTermK", "ltK"), ("localTermM", "ltM"), ("precond_sqrtK", "pK"), ("precond_sqrtM", "pM"),
                        ("wf", "psi")):
            ctx.set(name, f[a])
        ctx.set_scalar("mu", MU)
        ctx.set_dipolar_kernel(f["gdd"], [0.0, 0.0, 1.0], RC)
        ctx.set_scalar("dipolar", 1)
        call = {"lrep": "matmulLrep", "tlrep": "precondLrep", "m": "matmulM", "k": "matmulK"}[case["op"]]
        return {"kind": kind, "ctx": ctx, "call": call, "x": _host_column(case, seed)}
    if kind == "gram":
        ctx = _dense(CPLX[case["dtype"]])
        S = _block(2 * case["rows"], case["k"], case["dtype"], 2 * seed)
        AS = _block(2 * case["rows"], case["k"], case["dtype"], 2 * seed + 1)
        out = torch.zeros((4, case["k"], case["k"]), device="cuda",
                          dtype=torch.complex128 if CPLX[case["dtype"]] else torch.float64)
        prec = B.F32 if case["dtype"] == "f32" else B.F64
        return {"kind": kind, "ctx": ctx, "S": S, "AS": AS, "out": out, "prec": prec, "rows": case["rows"],
                "cplx": CPLX[case["dtype"]]}
    if kind == "update":
        ctx = _dense(False)
        blocks, cx, cp = _update_inputs(case, seed)
        m, a, rows = case["m"], case["act"], case["rows"]
        outs = [torch.empty((c, rows), dtype=torch.float64, device="cuda") for c in (m, m, a, a)]
        return {"kind": kind, "ctx": ctx, "blocks": blocks, "cx": cx, "cp": cp, "outs": outs, "m": m, "a": a, "rows": rows}
    cfg = _solve_config(case, seed)
    psi, mu, _, _, V = problems.ground_state(B, cfg)
    p, _ = problems.build(B, cfg, psi, mu, V, precision="mixed" if case["mixed"] else "f64")
    return {"kind": kind, "problem": p}


def run(state):
    kind = state["kind"]
    if kind == "apply":
        x, y = state["x"], state["y"]
        state["ctx"].apply_ptr(state["op"], state["prec"], x.data_ptr(), x.shape[1], y.data_ptr(), y.shape[1], x.shape[0])
        return y
    if kind == "host":
        return state["ctx"].apply(state["call"], state["x"])
    if kind == "gram":
        S, AS, out = state["S"], state["AS"], state["out"]
        state["ctx"].gram_ptr(state["prec"], state["cplx"], state["rows"], S.shape[0], S.data_ptr(), S.shape[1],
                              AS.data_ptr(), AS.shape[1], out.data_ptr())
        return out
    if kind == "update":
        m, a, rows = state["m"], state["a"], state["rows"]
        k = m + 2 * a
        cx, cp = state["cx"].data_ptr(), state["cp"].data_ptr()
        X, P, W, AX, AP, AW = (t.data_ptr() for t in state["blocks"])
        oX, oAX, oP, oAP = (t.data_ptr() for t in state["outs"])
        outs = [(oX, m, 1.0, 0.0, [(X, m, cx, k), (P, a, cx + 8 * m, k), (W, a, cx + 8 * (m + a), k)]),
                (oAX, m, 1.0, 0.0, [(AX, m, cx, k), (AP, a, cx + 8 * m, k), (AW, a, cx + 8 * (m + a), k)]),
                (oP, a, 1.0, 0.0, [(P, a, cp, 2 * a), (W, a, cp + 8 * a, 2 * a)]),
                (oAP, a, 1.0, 0.0, [(AP, a, cp, 2 * a), (AW, a, cp + 8 * a, 2 * a)])]
        rc = state["ctx"].block_update(B.F64, False, rows, rows, outs)
        if rc:
            raise RuntimeError("block_update: %d" % rc)
        return state["outs"]
    p = state["problem"]
    rc = p.solve()
    if rc:
        raise RuntimeError("solve: %d" % rc)
    # the modes of degenerate pairs are fixed up to a rotation only; the eigenvalues are the solve's numbers
    return p.eigenvalues()


def work(case):
    kind = case["kind"]
    if kind in ("apply", "host"):
        size = case["nx"] * case["ny"] * case["nz"]
        dtype, op = case["dtype"], case["op"]
        el = {"f64": 8, "f32": 4, "c128": 16, "c64": 8}[dtype]
        re = 8 if dtype in ("f64", "c128") else 4
        spec = size if CPLX[dtype] else size // case["nx"] * (case["nx"] // 2 + 1)
        cols = case.get("cols", 1)
        ffts = {"lrep": 6, "tlrep": 4, "m": 4, "k": 2}[op]
        fields = {"lrep": 2 * re * size + el * size + 8 * spec, "tlrep": 2 * re * size, "m": re * size + el * size + 8 * spec,
                  "k": re * size}[op]
        flops = ffts * (5.0 if CPLX[dtype] else 2.5) * size * math.log2(size) * cols
        return {"bytes": 2.0 * _halves(case) * el * size * cols + fields, "flops": flops}
    if kind == "gram":
        el = {"f64": 8, "f32": 4, "c128": 16}[case["dtype"]]
        rows, k = case["rows"], case["k"]
        flops = (8.0 if CPLX[case["dtype"]] else 2.0) * rows * (k * (k + 1.0) + k * k + 2.0 * k * k)
        return {"bytes": 4.0 * rows * k * el + 4.0 * k * k * (16 if CPLX[case["dtype"]] else 8), "flops": flops}
    if kind == "update":
        m, a, rows = case["m"], case["act"], case["rows"]
        k = m + 2 * a
        return {"bytes": 8.0 * rows * (2 * k + 2 * (m + a)) + 8.0 * (k * m + 2 * a * a),
                "flops": 4.0 * rows * (k * m + 2 * a * a)}
    # a solve: about 60 iterations, each with Lrep and T on about 3/4 of the block, 19 block products of the Gram
    # stage and 12 of the update
    n, m = 2 * case["grid"] ** 3, 2 * case["nev"]
    return {"bytes": 60.0 * 8 * n * m * 12, "flops": 60.0 * 2 * n * m * m * 31}


def _spectral(x, n, mult):
    """F^-1[mult F x] of columns (cols, nz, ny, nx)."""
    if x.is_complex():
        return torch.fft.ifftn(torch.fft.fftn(x, dim=(1, 2, 3)) * mult, dim=(1, 2, 3))
    return torch.fft.irfftn(torch.fft.rfftn(x, dim=(1, 2, 3)) * mult, s=(n[2], n[1], n[0]), dim=(1, 2, 3))


def _exact_apply(case, x):
    f = {k: torch.as_tensor(v, device="cuda") if isinstance(v, np.ndarray) else v for k, v in _fields(case).items()}
    n = (case["nx"], case["ny"], case["nz"])
    kin, inv = 0.5 * f["k2"], MU + 0.5 * f["k2"]

    def K(u):
        return _spectral(u, n, kin) + f["ltK"] * u

    def M(v):
        return _spectral(v, n, kin) + f["ltM"] * v + 2.0 * f["gdd"] * f["psi"] * _spectral(f["psi"].conj() * v, n, f["vdd"])

    def T(p):
        return lambda v: p * _spectral(p * v, n, 1.0 / inv)

    ops = {"lrep": (K, M), "tlrep": (T(f["pK"]), T(f["pM"])), "m": (M,), "k": (K,)}[case["op"]]
    out = torch.empty(x.shape, dtype=torch.complex128 if x.is_complex() else torch.float64, device="cuda")
    size = n[0] * n[1] * n[2]
    for c in range(0, x.shape[0], 4):
        for h, op in enumerate(ops):
            part = x[c:c + 4, h * size:(h + 1) * size].to(out.dtype).reshape(-1, n[2], n[1], n[0])
            out[c:c + 4, h * size:(h + 1) * size] = op(part).reshape(part.shape[0], -1)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "apply":
        cols, rows = case["cols"], _halves(case) * case["nx"] * case["ny"] * case["nz"]
        return _exact_apply(case, _randn((cols, rows), case["dtype"], seed))
    if kind == "host":
        x = torch.as_tensor(_host_column(case, seed), device="cuda")
        return _exact_apply(case, x[None, :])[0].cpu().numpy()
    if kind == "gram":
        rows, k = case["rows"], case["k"]
        wide = torch.complex128 if CPLX[case["dtype"]] else torch.float64
        S = _block(2 * rows, k, case["dtype"], 2 * seed)
        AS = _block(2 * rows, k, case["dtype"], 2 * seed + 1)
        out = torch.zeros((4, k, k), dtype=wide, device="cuda")
        step = 1 << 16
        for r in range(0, rows, step):
            e = min(rows, r + step)
            u, v = S[:, r:e].to(wide), S[:, rows + r:rows + e].to(wide)
            au, av = AS[:, r:e].to(wide), AS[:, rows + r:rows + e].to(wide)
            # column-major blocks: out[j, i] = a_i^H b_j
            out[0] += u @ u.conj().T
            out[1] += v @ v.conj().T
            out[2] += v @ u.conj().T
            out[3] += au @ u.conj().T + av @ v.conj().T
        return out
    if kind == "update":
        blocks, cx, cp = _update_inputs(case, seed)
        m, a = case["m"], case["act"]
        X, P, W, AX, AP, AW = blocks

        def both(x, p, w):
            return (cx[:, :m] @ x + cx[:, m:m + a] @ p + cx[:, m + a:] @ w, cp[:, :a] @ p + cp[:, a:] @ w)

        (x1, p1), (ax1, ap1) = both(X, P, W), both(AX, AP, AW)
        return [x1, ax1, p1, ap1]
    return None  # a solve to tolerance in plain 64-bit torch takes minutes
