"""Performance cases of the engine: what a user's program has it do, from one site's contractions to
whole RK4 steps of trajectories, density matrices and batches, through the public entry points.

A case is a dict of plain values with a ``kind``:

* ``site``   the contractions of one site in both sweep directions (C ABI op level, device buffers):
             prod_AOR, prod_LR, update_re and prod_AOL, prod_LR, update_le;
* ``qr``     one Householder QR of a site (leftorth! / rightorth!), Q and optionally R;
* ``step``   one RK4 step RK4stp_apply_H_half!: trajectories (d = 2, w = 4, the 11-argument form,
             then normalize_lo!) and density matrices (d = 4, the 10-argument in-place form);
             ``batch`` > 0 runs that many copies in batch handles; ``slices`` is the context's
             contraction precision (0 = FP64, 6 = int8 slices);
* ``jump``   a trajectory's jump step: a waveguide jump (compress_var_apply_H!, one sweep pair,
             normalize_lo!) and a local decay (apply_site_operator!, leftorthonormalizationQR!);
* ``observe`` the measurements of a density matrix: its trace and every population.

Inputs are generic: left-canonical matrix product states at full bond dimension with decaying
bond weights, and the waveguide generators with couplings and positions drawn from the seed.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.getcwd(), "matrixproductstates.jl_b200"))
from mpsb200 import _lib, core as K  # noqa: E402

C128 = torch.complex128


def listed():
    return [
        # the smallest work: one ragged site of a small trajectory, op by op (latency and launches)
        {"name": "site_37x29_d2", "kind": "site", "chil": 37, "chir": 29, "d": 2, "w": 4},
        # an interior site of the chi = 128 density matrix
        {"name": "site_128_d4", "kind": "site", "chil": 128, "chir": 128, "d": 4, "w": 8},
        # gauge moves: the site of a small trajectory, of the chi = 128 and of the chi = 512 density matrix
        {"name": "qr_64x32", "kind": "qr", "m": 64, "n": 32, "r": True},
        {"name": "qr_512x128", "kind": "qr", "m": 512, "n": 128, "r": False},
        {"name": "qr_2048x512", "kind": "qr", "m": 2048, "n": 512, "r": False},
        # the CPU-sized trajectory configuration
        {"name": "trajectory_n20_chi32", "kind": "step", "na": 20, "chi": 32, "d": 2, "w": 4, "batch": 0, "slices": 0},
        # the FP64 density-matrix workload
        {"name": "density_n40_chi128", "kind": "step", "na": 40, "chi": 128, "d": 4, "w": 8, "batch": 0, "slices": 0},
        # the interior of the chi = 512 density matrix (a shorter chain), split precision
        {"name": "density_n14_chi512_s6", "kind": "step", "na": 14, "chi": 512, "d": 4, "w": 8, "batch": 0, "slices": 6},
        # buckets of the batched trajectory engine: a middle cap off the tile grid, and the largest cap
        {"name": "batch16_n32_chi81_s6", "kind": "step", "na": 32, "chi": 81, "d": 2, "w": 4, "batch": 16, "slices": 6},
        {"name": "batch8_n24_chi256_s6", "kind": "step", "na": 24, "chi": 256, "d": 2, "w": 4, "batch": 8, "slices": 6},
        # a jump step of a plain trajectory
        {"name": "jump_n64_chi100", "kind": "jump", "na": 64, "chi": 100, "d": 2},
        # the measurements every few steps of the density-matrix loop
        {"name": "observe_n40_chi128", "kind": "observe", "na": 40, "chi": 128, "d": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["site", "qr", "trajectory", "density", "split", "batch", "batch", "jump", "observe"])
    if kind == "site":
        return {"kind": "site", "chil": _log_int(rng, 3, 256), "chir": _log_int(rng, 3, 256), "d": rng.choice([2, 4]),
                "w": rng.choice([2, 4, 6, 8])}
    if kind == "qr":
        n = _log_int(rng, 4, 512)
        return {"kind": "qr", "m": rng.randint(n, min(2048, 4 * n)), "n": n, "r": rng.random() < 0.5}
    if kind == "trajectory":
        return {"kind": "step", "na": rng.randint(8, 64), "chi": _log_int(rng, 8, 160), "d": 2, "w": 4, "batch": 0,
                "slices": rng.choice([0, 0, 6])}
    if kind == "density":
        return {"kind": "step", "na": rng.randint(6, 40), "chi": _log_int(rng, 8, 128), "d": 4, "w": rng.choice([6, 8]),
                "batch": 0, "slices": 0}
    if kind == "split":
        return {"kind": "step", "na": rng.randint(8, 13), "chi": _log_int(rng, 130, 500), "d": 4, "w": rng.choice([6, 8]),
                "batch": 0, "slices": 6}
    if kind == "batch":
        slices = rng.choice([0, 6, 6])
        chi = _log_int(rng, 8, 200 if slices else 128)
        most = max(2, min(16, int(6 * 256 ** 3 / chi ** 3)))
        return {"kind": "step", "na": rng.randint(8, 24), "chi": chi, "d": 2, "w": 4, "batch": rng.randint(2, most),
                "slices": slices}
    if kind == "jump":
        return {"kind": "jump", "na": rng.randint(16, 64), "chi": _log_int(rng, 8, 128), "d": 2}
    return {"kind": "observe", "na": rng.randint(8, 40), "chi": _log_int(rng, 8, 128), "d": 4}


# ------------------------------------------------------------------ inputs (plain torch)

def _dims(na, chi, d):
    return [min(chi, d ** min(k, 12), d ** min(na - k, 12)) for k in range(na + 1)]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + 17)


def _randn(gen, *shape):
    return torch.randn(*shape, dtype=C128, device="cuda", generator=gen)


def _isometry(x):
    """(Q, R) of x (..., m, n), full column rank, by two Cholesky passes."""
    r = None
    for _ in range(2):
        c = torch.linalg.cholesky(x.mH @ x).mH
        x = torch.linalg.solve_triangular(c, x, upper=True, left=False)
        r = c if r is None else c @ r
    return x, r


def _mps(gen, dims, d, batch=1):
    """Sites (batch, chiL, d, chiR) of normalised left-canonical states: a bulk whose bond weights
    decay from 1 to 0.1, as on bonds whose cap is in use, between ends of full bond dimension."""
    na = len(dims) - 1
    sites, r = [], torch.ones(batch, 1, 1, dtype=C128, device="cuda")
    for k in range(na):
        l, n = dims[k], dims[k + 1]
        if n == l * d and k < na - 1:          # the left end: unitary, nothing to carry
            q, _ = torch.linalg.qr(_randn(gen, batch, n, n))
            sites.append(q.reshape(batch, l, d, n))
            r = torch.eye(n, dtype=C128, device="cuda").expand(batch, n, n)
            continue
        if l == d * n:                         # the right end: unitary from the right
            a = torch.linalg.qr(_randn(gen, batch, l, l))[0].reshape(batch, l, d, n)
        else:
            a = _randn(gen, batch, l, d, n) * 0.1 ** (torch.arange(n, dtype=torch.float64, device="cuda") / n)
        a = (r @ a.reshape(batch, l, d * n)).reshape(batch, l, d, n)
        if k == na - 1:
            sites.append(a / torch.linalg.vector_norm(a, dim=(1, 2, 3), keepdim=True))
            break
        q, r = _isometry(a.reshape(batch, l * d, n))
        r = r / torch.linalg.vector_norm(r, dim=(1, 2), keepdim=True)
        sites.append(q.reshape(batch, l, d, n))
    return sites


def _slab(sites):
    """The device layout: every site column-major, back to back, per copy."""
    return torch.cat([a.permute(0, 3, 2, 1).reshape(a.shape[0], -1) for a in sites], dim=1)


I2 = np.eye(2)
EE = np.diag([0.0, 1.0])
SM = np.array([[0.0, 1.0], [0.0, 0.0]])
SP = SM.T


def _chain(case, seed):
    """Couplings and positions of the waveguide chain, from the seed."""
    r = np.random.default_rng(seed)
    na = case["na"]
    return {"g": 1.0 + 0.2 * r.uniform(-1, 1, na), "x": np.arange(na) + 0.1 * r.uniform(-1, 1, na), "omega": 0.5,
            "k": 0.5 * np.pi}


def _ends(sites):
    sites[0] = sites[0][:1]
    sites[-1] = sites[-1][:, :, -1:]
    return [np.ascontiguousarray(o, dtype=np.complex128) for o in sites]


def _h_mpo(p, con, delt):
    """con + delt * (-i H_eff) of the driven chain, w = 4, d = 2: O[wL, out, wR, in]."""
    na, out = len(p["g"]), []
    for j in range(na):
        ph = np.exp(1j * p["k"] * (p["x"][min(j + 1, na - 1)] - p["x"][j]))
        c = np.sqrt(delt * p["g"][j] / 2)
        o = np.zeros((4, 2, 4, 2), dtype=complex)
        o[0, :, 0], o[0, :, 1], o[0, :, 2] = I2, -c * ph * SP, -c * ph * SM
        o[1, :, 1] = o[2, :, 2] = ph * I2
        o[0, :, 3] = con / na * I2 + delt * (-p["g"][j] / 2 * EE + 1j * p["omega"] * (SP + SM))
        o[1, :, 3], o[2, :, 3], o[3, :, 3] = c * SM, c * SP, I2
        out.append(o)
    return _ends(out)


def _l_mpo(p, con, delt, w):
    """con + delt * Lindbladian of the driven chain for a vectorised density matrix, d = 4."""
    na, out, k = len(p["g"]), [], np.kron
    ii, gphi, geg = k(I2, I2), 0.1, 0.1
    for j in range(na):
        q = np.exp(1j * p["k"] * (p["x"][min(j + 1, na - 1)] - p["x"][j]))
        c, g = np.sqrt(delt * p["g"][j] / 2), p["g"][j] + geg
        o = np.zeros((w, 4, w, 4), dtype=complex)
        o[0, :, 0] = ii
        o[0, :, 1], o[0, :, 2] = c * q * (k(I2, SM) - k(SP, I2)), c * q * k(SM, I2)
        o[0, :, 3], o[0, :, 4] = np.conj(c * q) * k(I2, SM), np.conj(c * q) * (k(SM, I2) - k(I2, SP))
        o[1, :, 1] = o[2, :, 2] = q * ii
        o[3, :, 3] = o[4, :, 4] = np.conj(q) * ii
        x = SP + SM
        o[0, :, w - 1] = con / na * ii + delt * (
            g * (k(SM, SM) - 0.5 * k(EE, I2) - 0.5 * k(I2, EE)) + 1j * p["omega"] * (k(x, I2) - k(I2, x))
            + gphi * (k(EE, EE) - 0.5 * k(EE, I2) - 0.5 * k(I2, EE)))
        o[1, :, w - 1], o[2, :, w - 1] = c * k(SM, I2), -c * (k(SP, I2) - k(I2, SM))
        o[3, :, w - 1], o[4, :, w - 1] = -np.conj(c) * (k(I2, SP) - k(SM, I2)), np.conj(c) * k(I2, SM)
        o[w - 1, :, w - 1] = ii
        out.append(o)
    return _ends(out)


def _jump_mpo(p):
    """sum_j i sqrt(g/2) e^{-i k x_j} sigma-_j, w = 2, d = 2."""
    out = []
    for g, x in zip(p["g"], p["x"]):
        o = np.zeros((2, 2, 2, 2), dtype=complex)
        o[0, :, 0] = o[1, :, 1] = I2
        o[0, :, 1] = 1j * np.sqrt(g / 2) * np.exp(-1j * p["k"] * x) * SM
        out.append(o)
    return _ends(out)


def _generators(case, seed):
    p, dt = _chain(case, seed), _dt(case)
    one = (lambda con, delt: _l_mpo(p, con, delt, case["w"])) if case["d"] == 4 else (lambda con, delt: _h_mpo(p, con, delt))
    return [one(1, dt / 2), one(0, 1), one(1, dt / 2)]


def _dt(case):
    return 0.005 if case["d"] == 4 else 0.01


def _site_inputs(case, seed):
    gen, d, w = _gen(seed), case["d"], case["w"]
    l, r = case["chil"], case["chir"]
    a = _randn(gen, l, d, r) / math.sqrt(l * d)
    a0 = _randn(gen, l, d, r) / math.sqrt(l * d)
    o = _randn(gen, w, d, w, d) / math.sqrt(w * d)
    return a, a0, o, _randn(gen, l, w, l) / l, _randn(gen, r, w, r) / r


def _qr_input(case, seed):
    """A site's matrix: columns mixed from directions whose weights span two decades."""
    gen, m, n = _gen(seed), case["m"], case["n"]
    w = 10.0 ** (-2.0 * torch.arange(n, dtype=torch.float64, device="cuda") / n)
    return (_randn(gen, m, n) * w) @ (_randn(gen, n, n) / math.sqrt(n))


# ------------------------------------------------------------------ the passes

class _Device:
    """`n` complex128 at a device address, for torch; keeps the handle that owns them alive."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<c16", "data": (ptr, False), "version": 2}


def _view(mps):
    """The whole slab of an MPS handle (every copy) as one tensor."""
    n = mps.batch * sum(mps.dims[k] * mps.d * mps.dims[k + 1] for k in range(mps.na))
    return torch.as_tensor(_Device(mps, mps.site_ptr(0), n), device="cuda")


def _fmt(t):
    """The column-major buffer of an index-ordered tensor."""
    return t.permute(*reversed(range(t.dim()))).contiguous().reshape(-1)


_contexts = {}


def _ctx(slices=0):
    """The program's context of one contraction precision."""
    if slices not in _contexts:
        _contexts[slices] = K.Context(0)
        _contexts[slices].set_precision(slices)
    return _contexts[slices]


def _new_mps(ctx, dims, d, batch, sites=None):
    m = K.MPS(dims, d, ctx, batch or None)
    if sites is not None:
        _view(m).copy_(_slab(sites).reshape(-1))
    return m


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    kind, s = case["kind"], {"kind": case["kind"]}
    if kind == "site":
        a, a0, o, L, R = _site_inputs(case, seed)
        l, r, d, w = case["chil"], case["chir"], case["d"], case["w"]
        s.update(ctx=_ctx(), sizes=(l, r, d, w), ins=[_fmt(t) for t in (a, a0, o, L, R)])
        s["outs"] = [torch.empty(n, dtype=C128, device="cuda") for n in
                     (l * w * d * r, l * d * r, l * w * l, l * d * r * w, l * d * r, r * w * r)]
    elif kind == "qr":
        x = _qr_input(case, seed)
        s.update(ctx=_ctx(), m=case["m"], n=case["n"], x=_fmt(x), q=torch.empty(x.numel(), dtype=C128, device="cuda"))
        s["r"] = torch.empty(case["n"] ** 2, dtype=C128, device="cuda") if case["r"] else None
    elif kind == "observe":
        ctx, dims = _ctx(), _dims(case["na"], case["chi"], 4)
        s["rho"] = _new_mps(ctx, dims, 4, 0, _mps(_gen(seed), dims, 4))
        tr, see = np.array([1, 0, 0, 1.0]), np.array([0, 0, 0, 1.0])
        product = lambda at: K.MPS.from_sites([(see if j == at else tr).astype(complex).reshape(1, 4, 1)  # noqa: E731
                                               for j in range(case["na"])], ctx)
        s["functionals"] = [product(at) for at in range(-1, case["na"])]
    elif kind == "jump":
        ctx, na, dims = _ctx(), case["na"], _dims(case["na"], case["chi"], 2)
        s["A"] = _new_mps(ctx, dims, 2, 0, _mps(_gen(seed), dims, 2))
        s["A_r"], s["A_d"] = s["A"].clone(), s["A"].clone()
        s["envop"] = K.build_env(dims, dims, [2] * (na + 1), ctx)
        s["jump"] = K.MPO.from_sites(_jump_mpo(_chain(case, seed)), ctx)
        s["site"] = na // 2
    else:
        ctx, na, d, b = _ctx(case["slices"]), case["na"], case["d"], case["batch"]
        dims = _dims(na, case["chi"], d)
        s["psi"] = _new_mps(ctx, dims, d, b, _mps(_gen(seed), dims, d, b or 1))
        s["out"], *s["stages"] = (_new_mps(ctx, dims, d, b) for _ in range(4))
        s["env"] = [K.build_env(dims, dims, None, ctx, b or None) for _ in range(3)]
        s["env"].append(K.build_env(dims, dims, [case["w"]] * (na + 1), ctx, b or None))
        s["H"] = [K.MPO.from_sites(h, ctx) for h in _generators(case, seed)]
        s["dt"], s["d"], s["batch"] = _dt(case), d, b
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "site":
        (l, r, d, w), h = s["sizes"], s["ctx"].h
        a, a0, o, L, R = (_p(t) for t in s["ins"])
        aor, x, re, aol, y, le = (_p(t) for t in s["outs"])
        _lib.call("mpsb_op_prod_AOR", h, a, o, R, aor, l, d, r, w, w, r)
        _lib.call("mpsb_op_prod_LR_3_4", h, L, aor, x, l, w, l, d, r)
        _lib.call("mpsb_op_update_re", h, a0, aor, re, l, w, d, r, l)
        _lib.call("mpsb_op_prod_AOL", h, a, o, L, aol, l, d, r, w, w, l)
        _lib.call("mpsb_op_prod_LR_4_3", h, aol, R, y, l, d, r, w, r)
        _lib.call("mpsb_op_update_le", h, a0, aol, le, l, d, r, w, r)
        return s["outs"]
    if kind == "qr":
        _lib.call("mpsb_op_qr", s["ctx"].h, _p(s["x"]), _p(s["q"]), _p(s["r"]) if s["r"] is not None else None, s["m"], s["n"])
        return [s["q"]] if s["r"] is None else [s["q"], s["r"]]
    if kind == "observe":
        v = [K.scal_prod_no_conj(f, s["rho"]) for f in s["functionals"]]
        return [v[0].real, v[0].imag, np.array(v[1:])]
    if kind == "jump":
        K.compress_var_apply_H_(s["A_r"], s["envop"], s["A"], s["A"], s["jump"], 1)
        p_r = K.normalize_lo_(s["A_r"])
        s["A_d"].copy_from(s["A"])
        K.apply_site_operator_(s["A_d"], s["site"], SM)
        p_d = K.leftorthonormalizationQR_(s["A_d"])
        return [_view(s["A_r"]), p_r, _view(s["A_d"]), p_d]
    if s["d"] == 4:   # the in-place form of the density-matrix loop, from a saved state
        s["out"].copy_from(s["psi"])
        K.RK4stp_apply_H_half_(s["dt"], s["H"], s["out"], *s["stages"], *s["env"])
        return [_view(s["out"])]
    K.RK4stp_apply_H_half_(s["dt"], s["H"], s["out"], s["psi"], *s["stages"], *s["env"])
    p = K.normalize_lo_batch(s["out"]) if s["batch"] else K.normalize_lo_(s["out"])
    return [_view(s["out"]), p]


# ------------------------------------------------------------------ what a pass cannot do without

def _contraction(dl, dr, d, wl, wr):
    """flops of applying one site's effective operator (A, O, one environment, then the other)."""
    return 8.0 * dl * d * wr * dr * dr + 8.0 * dl * dr * (d * wr) * (wl * d), 8.0 * dl * dl * wl * d * dr


def _qr_flops(m, n):
    return 16.0 * (m * n * n - n ** 3 / 3.0)


def _half_sweep_flops(dims, d, w, plain, right):
    na, f = len(dims) - 1, 0.0
    for k in range(na):
        dl, dr = dims[k], dims[k + 1]
        wl, wr = (w if k else 1), (w if k < na - 1 else 1)
        if right:
            dl, dr, wl, wr = dr, dl, wr, wl
        first, second = _contraction(dl, dr, d, wl, wr)
        pl = 8.0 * d * dl * dr * (dl + dr) * plain
        f += first + second + pl                                           # the site
        last = (k == na - 1) if right else (k == 0)
        if not last:
            f += _qr_flops(d * dr, dl) + second + 8.0 * d * dl * dl * dr * plain   # gauge move and environments
        start = (k >= 1) if right else (k < na - 1)
        if start:                                                          # initial environments of the sweep
            f += 8.0 * d * dr * dr * wr * dl + 8.0 * dl * dr * d * d * wl * wr + 8.0 * d * dl * dl * wl * dr
            f += 16.0 * d * dl * dl * dr * plain
    return f


def work(case):
    kind, d = case["kind"], case.get("d")
    if kind == "site":
        l, r, w = case["chil"], case["chir"], case["w"]
        a, b = _contraction(l, r, d, w, w)
        e, f = _contraction(r, l, d, w, w)
        elems = 2 * l * d * r + (w * d) ** 2 + w * (l * l + r * r) + 2 * w * l * d * r + 2 * l * d * r + w * (l * l + r * r)
        return {"bytes": 16.0 * elems, "flops": a + 2 * b + e + 2 * f}
    if kind == "qr":
        return {"bytes": 32.0 * case["m"] * case["n"], "flops": _qr_flops(case["m"], case["n"])}
    dims = _dims(case["na"], case["chi"], d)
    state = 16.0 * sum(dims[k] * d * dims[k + 1] for k in range(case["na"]))
    if kind == "observe":
        f = sum(8.0 * d * dims[k] * dims[k + 1] for k in range(case["na"]))
        return {"bytes": state * (case["na"] + 1), "flops": f * (case["na"] + 1)}
    if kind == "jump":
        f = sum(_half_sweep_flops(dims, d, 2, 0, right) for right in (False, True))
        f += sum(_qr_flops(d * dims[k], dims[k + 1]) + 8.0 * dims[k + 1] ** 2 * d * dims[min(k + 2, case["na"])]
                 for k in range(case["na"] - 1))
        return {"bytes": 3 * state, "flops": f}
    b = max(1, case["batch"])
    f = sum(_half_sweep_flops(dims, d, case["w"], pl, right) for pl, right in ((0, False), (1, True), (1, False), (3, True)))
    return {"bytes": 2 * b * state, "flops": b * f}


# ------------------------------------------------------------------ the same in plain torch

def _orth_right(a):
    """rightorth!: QR of reshape(a, l, d r) transposed, rows in column-major order."""
    l, d, r = a.shape
    q, _ = torch.linalg.qr(a.permute(2, 1, 0).reshape(r * d, l))
    return q.reshape(r, d, l).permute(2, 1, 0)


def _orth_left(a, with_r=False):
    l, d, r = a.shape
    q, c = torch.linalg.qr(a.permute(1, 0, 2).reshape(d * l, r))
    q = q.reshape(d, l, r).permute(1, 0, 2)
    return (q, c) if with_r else q


# environments [bra bond, operator bond, ket bond]; e = torch.einsum over at most two tensors
_e = torch.einsum


def _left(env, bra, o, ket):
    return _e("xpcd,xpy->ycd", _e("xwsd,wpcs->xpcd", _e("xwz,zsd->xwsd", env, ket), o), bra.conj())


def _right(env, bra, o, ket):
    return _e("zwpy,xpy->xwz", _e("zscy,wpcs->zwpy", _e("zsd,ycd->zscy", ket, env), o), bra.conj())


def _apply(left, o, ket, right):
    t = _e("xwsd,wpcs->xpcd", _e("xwz,zsd->xwsd", left, ket), o)
    return _e("xpcd,ycd->xpy", t, right)


def _half_sweep(right, bra, coef, terms, H, lefts=None):
    """One half sweep of the variational compression of sum_l coef[l] terms[l], the last through H;
    returns the new sites.  Plain terms are terms through the identity (operator bond 1)."""
    na, d = len(bra), bra[0].shape[1]
    one = torch.ones(1, 1, 1, dtype=C128, device="cuda")
    ident = torch.eye(d, dtype=C128, device="cuda").reshape(1, d, 1, d)
    ops = [[ident] * na] * (len(terms) - 1) + [H]
    new = [None] * na
    order = range(na) if right else range(na - 1, -1, -1)
    far = [[None] * (na + 1) for _ in terms]      # the environments of the guess, ahead of the sweep
    near = [c * one for c in coef]                 # the environments of the new sites, behind it
    for l, (t, o) in enumerate(zip(terms, ops)):
        far[l][na if right else 0] = one
        for k in (range(na - 1, 0, -1) if right else range(na - 1)):
            if right:
                far[l][k] = _right(far[l][k + 1], bra[k], o[k], t[k])
            else:
                far[l][k + 1] = _left(far[l][k], bra[k], o[k], t[k])
    for k in order:
        x = sum(_apply(near[l], o[k], t[k], far[l][k + 1]) if right else _apply(far[l][k], o[k], t[k], near[l])
                for l, (t, o) in enumerate(zip(terms, ops)))
        if k != (na - 1 if right else 0):
            x = _orth_left(x) if right else _orth_right(x)
            near = [(_left if right else _right)(near[l], x, o[k], t[k]) for l, (t, o) in enumerate(zip(terms, ops))]
        new[k] = x
    return new


def _rk4(psi, H, dt):
    p1 = _half_sweep(False, psi, [1.0], [psi], H[0])
    p2 = _half_sweep(True, p1, [1.0, dt / 2], [psi, p1], H[1])
    p3 = _half_sweep(False, p2, [1.0, dt], [psi, p2], H[1])
    return _half_sweep(True, p3, [-1 / 3, 1 / 3, 2 / 3, 1 / 3], [psi, p1, p2, p3], H[2])


def _jump(psi, H):
    """compress_var_apply_H! with one sweep pair."""
    na = len(psi)
    one = torch.ones(1, 1, 1, dtype=C128, device="cuda")
    left, right, new = [one] + [None] * na, [None] * na + [one], list(psi)
    for k in range(na - 1):
        left[k + 1] = _left(left[k], psi[k], H[k], psi[k])
    for k in range(na - 1, 0, -1):
        new[k] = _orth_right(_apply(left[k], H[k], psi[k], right[k + 1]))
        right[k] = _right(right[k + 1], new[k], H[k], psi[k])
    for k in range(na):
        new[k] = _apply(left[k], H[k], psi[k], right[k + 1])
        if k < na - 1:
            new[k] = _orth_left(new[k])
            left[k + 1] = _left(left[k], new[k], H[k], psi[k])
    return new


def _normalized(sites):
    p = torch.linalg.vector_norm(sites[-1]) ** 2
    return sites[:-1] + [sites[-1] / torch.sqrt(p)], float(p)


def _flat(sites):
    return _slab([a.unsqueeze(0) for a in sites]).reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "site":
        a, a0, o, L, R = _site_inputs(case, seed)   # L is stored [ket, w, bra], conjugated on use
        aor = _e("zsd,dcy->zscy", a, R)
        aor = _e("zscy,wpcs->zwpy", aor, o)
        aol = _e("zwx,zsd->xwsd", L.conj(), a)
        aol = _e("xwsd,wpcs->xpdc", aol, o)
        return [_fmt(t) for t in (aor, _e("zwx,zwpy->xpy", L.conj(), aor), _e("zwpy,xpy->zwx", aor, a0.conj()), aol,
                                  _e("xpdc,dcy->xpy", aol, R), _e("xpdc,xpy->dcy", aol.conj(), a0))]
    if kind == "qr":
        q, r = torch.linalg.qr(_qr_input(case, seed))
        return [_fmt(q), _fmt(r)] if case["r"] else [_fmt(q)]
    dims = _dims(case["na"], case["chi"], case["d"])
    states = _mps(_gen(seed), dims, case["d"], case.get("batch") or 1)
    psi = [a[0] for a in states]
    if kind == "observe":
        tr = torch.tensor([1, 0, 0, 1], dtype=C128, device="cuda")
        see = torch.tensor([0, 0, 0, 1], dtype=C128, device="cuda")
        v = []
        for at in range(-1, case["na"]):
            e = torch.ones(1, dtype=C128, device="cuda")
            for j, a in enumerate(psi):
                e = e @ _e("s,lsr->lr", see if j == at else tr, a)
            v.append(complex(e[0]))
        return [v[0].real, v[0].imag, np.array(v[1:])]
    up = lambda sites: [torch.from_numpy(o).cuda() for o in sites]  # noqa: E731
    if kind == "jump":
        new, p_r = _normalized(_jump(psi, up(_jump_mpo(_chain(case, seed)))))
        at = case["na"] // 2 - 1
        sm = torch.from_numpy(SM.astype(complex)).cuda()
        dec = list(psi)
        dec[at] = _e("ps,lsr->lpr", sm, dec[at])
        for k in range(case["na"] - 1):
            dec[k], c = _orth_left(dec[k], True)
            dec[k + 1] = _e("xl,lsr->xsr", c, dec[k + 1])
        dec, p_d = _normalized(dec)
        return [_flat(new), p_r, _flat(dec), p_d]
    H = [up(h) for h in _generators(case, seed)]
    if case["d"] == 4:
        return [_flat(_rk4(psi, H, _dt(case)))]
    done = [_normalized(_rk4([a[b] for a in states], H, _dt(case))) for b in range(case["batch"] or 1)]
    norms = np.array([p for _, p in done]) if case["batch"] else done[0][1]
    return [torch.cat([_flat(x) for x, _ in done]), norms]
