"""The work that users of mfix_b200 have it do, as cases whose time can be compared.

Every case goes through the package's public entry points (mfix_b200.leq) and
uses the repository's own generators' recipes (mfix_b200/systems.py), restated
here in torch so that the inputs are made on the GPU.  Sizes are interior cells
per axis; the arrays carry MFIX's one-cell wall layer.

`exact` is plain torch in 64 bits: for a solve stopped by ITMAX the same
BiCGSTAB steps, for a solve run to TOL the solution itself.
"""
import math
import types

import numpy as np
import torch

from mfix_b200 import leq

DEV = "cuda"
F64 = torch.float64


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # One 2-D transport equation of a SIMPLE iteration, host arrays through the Fortran
        # signature, with the reference's defaults LEQ_IT = 20, LEQ_TOL = 1e-4: the smallest call.
        {"name": "dropin_2d_64", "kind": "dropin", "i": 64, "j": 64, "k": 0, "itmax": 20, "tol": 1e-4},
        # The momentum equations of a SIMPLE iteration (LEQ_IT(3..5) = 5): three phases' calls queued
        # and solved as one batch, host arrays, odd sizes.
        {"name": "momentum_3x_41", "kind": "momentum", "i": 41, "j": 51, "k": 37, "itmax": 5, "tol": 1e-4},
        # The pressure correction of a SIMPLE iteration on device fields: assembly and a solve with
        # LEQ_IT(1) = 20, one solids phase.
        {"name": "pp_step_96", "kind": "pp", "i": 96, "j": 128, "k": 96, "itmax": 20, "tol": 1e-4},
        # One 64^3 convection-diffusion system, mixed precision, device arrays (the benchmark's small
        # configuration), run to a tight tolerance as the known-answer tests do.
        {"name": "mixed_64", "kind": "solve", "i": 64, "j": 64, "k": 64, "prec": 1, "itmax": 500, "tol": 1e-10},
        # An ordinary size with ragged extents, mixed precision.
        {"name": "mixed_ragged_150", "kind": "solve", "i": 143, "j": 171, "k": 98, "prec": 1, "itmax": 500,
         "tol": 1e-10},
        # The benchmark's headline system, mixed precision.
        {"name": "mixed_256", "kind": "solve", "i": 256, "j": 256, "k": 256, "prec": 1, "itmax": 500, "tol": 1e-8},
        # The FP64 drop-in on device arrays, odd line length (JMAX2 odd).
        {"name": "fp64_ragged_odd", "kind": "solve", "i": 127, "j": 145, "k": 120, "prec": 0, "itmax": 500,
         "tol": 1e-10},
        # The FP64 drop-in at the headline size.
        {"name": "fp64_256", "kind": "solve", "i": 256, "j": 256, "k": 256, "prec": 0, "itmax": 500, "tol": 1e-8},
        # Independent systems of uneven sizes (U{16..96} per axis) solved together, mixed precision.
        {"name": "batch_48", "kind": "batch", "count": 48, "lo": 16, "hi": 96, "prec": 1, "itmax": 500, "tol": 1e-8,
         "mix": 11},
        # A burst of requests to the server: sizes log-uniform 24..160, a fifth of them pressure
        # corrections, TOL 1e-6 or 1e-8.
        {"name": "serve_burst_48", "kind": "serve", "count": 48, "lo": 24, "hi": 160, "prec": 1, "mix": 12},
        # One application of the LINE preconditioner on device arrays, as a host with its own Krylov
        # loop calls it.
        {"name": "msolve_130", "kind": "msolve", "i": 130, "j": 190, "k": 126},
        # The residual check of such a host: a matrix-vector product and a dot product, odd sizes.
        {"name": "residual_201", "kind": "residual", "i": 201, "j": 203, "k": 155},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "momentum", "pp", "solve", "solve", "solve", "batch", "serve", "msolve", "residual"])
    if kind == "dropin":
        two = rng.random() < 0.5
        hi = 160 if two else 48
        return {"kind": kind, "i": _size(rng, 16, hi), "j": _size(rng, 16, hi), "k": 0 if two else _size(rng, 16, hi),
                "itmax": rng.choice([5, 20]), "tol": 1e-4}
    if kind == "momentum":
        return {"kind": kind, "i": _size(rng, 16, 72), "j": _size(rng, 16, 72), "k": _size(rng, 16, 72), "itmax": 5,
                "tol": 1e-4}
    if kind == "pp":
        return {"kind": kind, "i": _size(rng, 24, 160), "j": _size(rng, 24, 200), "k": _size(rng, 24, 160),
                "itmax": 20, "tol": 1e-4}
    if kind == "solve":
        return {"kind": kind, "i": _size(rng, 24, 256), "j": _size(rng, 24, 256), "k": _size(rng, 24, 256),
                "prec": rng.choice([1, 1, 0]), "itmax": 500, "tol": 1e-10}
    if kind == "batch":
        return {"kind": kind, "count": _size(rng, 4, 48), "lo": 16, "hi": rng.choice([64, 96]),
                "prec": rng.choice([1, 1, 0]), "itmax": 500, "tol": 1e-8, "mix": rng.randrange(1000)}
    if kind == "serve":
        return {"kind": kind, "count": _size(rng, 8, 48), "lo": 24, "hi": rng.choice([96, 160]), "prec": 1,
                "mix": rng.randrange(1000)}
    return {"kind": kind, "i": _size(rng, 24, 240), "j": _size(rng, 24, 240), "k": _size(rng, 24, 240)}


# ---------------------------------------------------------------- inputs
def _box(i, j, k):
    return i + 2, j + 2, (k + 2 if k else 1)


def _interior(i2, j2, k2):
    m = torch.zeros((k2, i2, j2), dtype=torch.bool, device=DEV)
    m[(slice(1, -1) if k2 > 1 else slice(None)), 1:-1, 1:-1] = True
    return m


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _rand(g, shape):
    return torch.rand(shape, generator=g, dtype=F64, device=DEV)


# (axis of the [k, i, j] grid, diagonal of the low cell's row, of the high cell's)
_FACES = ((1, 4, 2), (2, 5, 1), (0, 6, 0))


def _system(i, j, k, seed, kind):
    """A_M as (7, n) and B_M as (n,): conv_diff or pressure_like of mfix_b200/systems.py."""
    i2, j2, k2 = _box(i, j, k)
    g = _gen(seed)
    inter = _interior(i2, j2, k2)
    a = torch.zeros((7, k2, i2, j2), dtype=F64, device=DEV)
    eps = _void_fraction(i2, j2, k2, g) if kind == "pressure_like" else None
    for ax, lo, hi in _FACES:
        m = inter.shape[ax]
        if m < 2:
            continue
        both = (inter.narrow(ax, 0, m - 1) & inter.narrow(ax, 1, m - 1)).to(F64)
        D = 0.5 + _rand(g, both.shape)
        if kind == "pressure_like":
            c_lo = c_hi = 0.5 * (eps.narrow(ax, 0, m - 1) + eps.narrow(ax, 1, m - 1)) * D
        else:
            F = 0.5 * torch.randn(both.shape, generator=g, dtype=F64, device=DEV)
            c_lo, c_hi = D + (-F).clamp(min=0), D + F.clamp(min=0)
        a[lo].narrow(ax, 0, m - 1).copy_(c_lo * both)
        a[hi].narrow(ax, 1, m - 1).copy_(c_hi * both)
    off = a[0] + a[1] + a[2] + a[4] + a[5] + a[6]
    excess = 1e-6 if kind == "pressure_like" else 1e-3
    a[3] = torch.where(inter, -off * (1.0 + excess), torch.full_like(off, -1.0))
    b = torch.where(inter, 2.0 * _rand(g, inter.shape) - 1.0, torch.zeros_like(off))
    return a.reshape(7, -1), b.reshape(-1)


def _void_fraction(i2, j2, k2, g):
    """0.4 with bubbles of 0.95, their number and radius scaled with the box (pressure_scaled)."""
    s = ((i2 - 2) * (j2 - 2) * (k2 - 2) / (192.0 * 384.0 * 192.0)) ** (1.0 / 3.0)
    count, rmin = max(1, round(40 * s ** 3)), max(1.5, 6.0 * s)
    rmax = max(rmin + 1.0, 20.0 * s)
    u = _rand(g, (count, 4)).cpu().numpy()
    eps = torch.full((k2, i2, j2), 0.4, dtype=F64, device=DEV)
    kk = torch.arange(k2, device=DEV, dtype=F64)[:, None, None]
    ii = torch.arange(i2, device=DEV, dtype=F64)[None, :, None]
    jj = torch.arange(j2, device=DEV, dtype=F64)[None, None, :]
    for q in range(count):
        r2 = ((kk - (1 + u[q, 0] * (k2 - 2))) ** 2 + (ii - (1 + u[q, 1] * (i2 - 2))) ** 2
              + (jj - (1 + u[q, 2] * (j2 - 2))) ** 2)
        eps[r2 <= (rmin + u[q, 3] * (rmax - rmin)) ** 2] = 0.95
    return eps


def _dims(case):
    """The systems' interior sizes, generators and tolerances of a batch or a burst."""
    rs = np.random.RandomState(case["mix"])
    out = []
    for _ in range(case["count"]):
        if case["kind"] == "batch":
            d = [int(v) for v in rs.randint(case["lo"], case["hi"] + 1, 3)]
            out.append((d, "conv_diff", case["tol"], case["itmax"]))
        else:
            v = np.exp(rs.uniform(math.log(case["lo"]), math.log(case["hi"] + 1), 3))
            d = [int(min(math.floor(x), case["hi"])) for x in v]
            pressure, loose = rs.rand() < 0.2, rs.rand() < 0.5
            out.append((d, "pressure_like" if pressure else "conv_diff", 1e-6 if loose else 1e-8,
                        5000 if pressure else 500))
    return out


class _Many:
    """Device systems in flat buffers (each array on a 256-byte boundary), with their pristine inputs."""

    def __init__(self, specs, seed):
        self.sys, self.at = [], []
        na = nb = 0
        for (i, j, k), _, tol, itmax in specs:
            i2, j2, k2 = _box(i, j, k)
            n = i2 * j2 * k2
            self.sys.append(types.SimpleNamespace(imax2=i2, jmax2=j2, kmax2=k2, do_k=1 if k else 0, n=n, tol=tol,
                                                  itmax=itmax))
            self.at.append((na, nb))
            na += -(-7 * n // 32) * 32
            nb += -(-n // 32) * 32
        self.a0 = torch.zeros(na, dtype=F64, device=DEV)
        self.b0 = torch.zeros(nb, dtype=F64, device=DEV)
        for q, ((i, j, k), kind, _, _) in enumerate(specs):
            a, b = _system(i, j, k, seed * 1009 + q, kind)
            (pa, pb), n = self.at[q], self.sys[q].n
            self.a0[pa:pa + 7 * n] = a.reshape(-1)
            self.b0[pb:pb + n] = b
        self.a, self.b = torch.empty_like(self.a0), torch.empty_like(self.b0)
        self.x = torch.empty_like(self.b0)
        self.ptr = [(self.a.data_ptr() + 8 * pa, self.b.data_ptr() + 8 * pb, self.x.data_ptr() + 8 * pb)
                    for pa, pb in self.at]

    def assemble(self):
        """What the host's assembly leaves in A_M, B_M and VAR before a solve (the solve scales A_M
        and B_M in place); the library's streams do not wait for torch's, so torch's is waited for."""
        self.a.copy_(self.a0)
        self.b.copy_(self.b0)
        self.x.zero_()
        torch.cuda.current_stream().synchronize()

    def outputs(self, ier):
        return {"x": self.x, "a": self.a, "b": self.b, "ier": np.array(ier, dtype=np.int32)}


def _fields(case, seed):
    """Device fields of the pressure-correction assembly (pp_fields of mfix_b200/systems.py): one
    solids phase, a pressure-outflow patch and an obstacle."""
    i2, j2, k2 = _box(case["i"], case["j"], case["k"])
    n, g = i2 * j2 * k2, _gen(seed)
    flag = torch.where(_interior(i2, j2, k2), 1, 100).to(torch.int32)
    flag[k2 // 3:2 * k2 // 3, i2 // 3:2 * i2 // 3, j2 - 1] = 11
    flag[k2 // 2 - 1:k2 // 2 + 1, i2 // 2 - 1:i2 // 2 + 1, j2 // 3:j2 // 3 + 2] = 100
    lim = {"rop_ge": (.5, 1.5), "rop_gn": (.5, 1.5), "rop_gt": (.5, 1.5), "ayz": (.8, 1.2), "axz": (.8, 1.2),
           "axy": (.8, 1.2), "u_g": (-1, 1), "v_g": (-1, 1), "w_g": (-1, 1), "rop_g": (.9, 1.1), "rop_go": (.9, 1.1),
           "vol": (.9, 1.1), "sum_r_g": (-.01, .01), "d_e": (.1, 1), "d_n": (.1, 1), "d_t": (.1, 1),
           "rop_se": (.1, .5), "rop_sn": (.1, .5), "rop_st": (.1, .5), "u_s": (-.5, .5), "v_s": (-.5, .5),
           "w_s": (-.5, .5), "rop_s": (.1, .3), "rop_so": (.1, .3), "sum_r_s": (-.001, .001)}
    f = {"flag": flag.reshape(-1)}
    for name, (lo, hi) in lim.items():
        f[name] = lo + (hi - lo) * _rand(g, (2 * n if name in ("d_e", "d_n", "d_t") else n,))
    return f, (i2, j2, k2), n


def _host_system(case, seed):
    a, b = _system(case["i"], case["j"], case["k"], seed, "conv_diff")
    return a.cpu().pin_memory(), b.cpu().pin_memory()


def prepare(case, seed):
    kind = case["kind"]
    s = types.SimpleNamespace(case=case, kind=kind)
    if kind in ("dropin", "momentum"):
        s.box = _box(case["i"], case["j"], case["k"])
        s.n = s.box[0] * s.box[1] * s.box[2]
        s.do_k = 1 if case["k"] else 0
        phases = 3 if kind == "momentum" else 1
        made = [_host_system(case, seed * 1009 + q) for q in range(phases)]
        s.a0 = torch.stack([m[0] for m in made]).pin_memory()  # A_M(DIMENSION_3, -3:3, 0:DIMENSION_M)
        s.b0 = torch.stack([m[1] for m in made]).pin_memory()
        s.a, s.b = torch.empty_like(s.a0).pin_memory(), torch.empty_like(s.b0).pin_memory()
        s.x = [torch.zeros(s.n, dtype=F64).pin_memory() for _ in range(phases)]
        return s
    if kind in ("solve", "batch", "serve"):
        if kind == "solve":
            specs = [((case["i"], case["j"], case["k"]), "conv_diff", case["tol"], case["itmax"])]
        else:
            specs = _dims(case)
        s.m = _Many(specs, seed)
        if kind == "serve":
            s.server = leq.Server(precision=case["prec"], max_systems=256, check_every=8, hbm_budget=40e9)
        return s
    if kind == "pp":
        s.f, s.box, s.n = _fields(case, seed)
        s.rec = types.SimpleNamespace(mmax=1, close_packed=np.zeros(1, dtype=np.int32), odt=100.0, ijk_p_g=0)
        s.ptrs = {k: v.data_ptr() for k, v in s.f.items()}
        s.a = torch.empty(7 * s.n, dtype=F64, device=DEV)
        s.b, s.bmmax, s.x = (torch.empty(s.n, dtype=F64, device=DEV) for _ in range(3))
        s.sys = types.SimpleNamespace(imax2=s.box[0], jmax2=s.box[1], kmax2=s.box[2], do_k=1, n=s.n, tol=case["tol"],
                                      itmax=case["itmax"])
        return s
    i2, j2, k2 = _box(case["i"], case["j"], case["k"])
    s.n, s.geom = i2 * j2 * k2, leq.geom(i2, j2, k2, 1)
    s.a, s.b = _system(case["i"], case["j"], case["k"], seed, "conv_diff")
    s.a /= s.a.abs().amax(dim=0)  # row-scaled, as the solver's own preconditioner sees it
    s.x = torch.empty(s.n, dtype=F64, device=DEV)
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    case, kind = s.case, s.kind
    if kind in ("dropin", "momentum"):
        s.a.copy_(s.a0)  # the host's assembly
        s.b.copy_(s.b0)
        phases = len(s.x)
        leq.init_geometry(*s.box, s.do_k, s.n, phases - 1)
        A, B, X = s.a.numpy(), s.b.numpy(), [x.numpy() for x in s.x]
        ier = []
        for m in range(phases):
            X[m][:] = 0.0
            call = leq.solve_lin_eq if phases == 1 else leq.defer_lin_eq
            ier.append(call("U_g", 3, X[m], A, B, m, case["itmax"], 2, "RSRS", case["tol"], "LINE"))
        if phases > 1:
            leq.flush_lin_eq()
            ier = [c.value for c in ier]
        return {"x": s.x, "a": s.a, "b": s.b, "ier": np.array(ier, dtype=np.int32)}
    if kind in ("solve", "batch"):
        s.m.assemble()
        _, res = leq.batch_solve(s.m.sys, precision=case["prec"], on_device=True, pointers=s.m.ptr)
        return s.m.outputs([r.ier for r in res])
    if kind == "serve":
        s.m.assemble()
        tickets = [s.server.submit(q, on_device=True, pointers=p) for q, p in zip(s.m.sys, s.m.ptr)]
        return s.m.outputs([s.server.wait(t)["ier"] for t in tickets])
    if kind == "pp":
        i2, j2, k2 = s.box
        leq.init_geometry(i2, j2, k2, 1, s.n, 1)
        s.x.zero_()
        torch.cuda.current_stream().synchronize()
        leq.conv_source_pp_g(s.rec, s.a.data_ptr(), s.b.data_ptr(), s.bmmax.data_ptr(), device_ptrs=s.ptrs)
        _, res = leq.batch_solve([s.sys], precision=0, on_device=True,
                                 pointers=[(s.a.data_ptr(), s.b.data_ptr(), s.x.data_ptr())])
        return {"x": s.x, "a": s.a, "b": s.b, "bmmax": s.bmmax, "ier": res[0].ier}
    if kind == "msolve":
        leq.leq_msolve(s.geom, s.b.data_ptr(), s.a.data_ptr(), s.x.data_ptr(), "RSRS", "LINE")
        return s.x
    leq.leq_matvec(s.geom, s.a.data_ptr(), s.b.data_ptr(), s.x.data_ptr())
    return {"y": s.x, "dot": leq.dot_product_par(s.x.data_ptr(), s.b.data_ptr(), s.n)}


# ---------------------------------------------------------------- what a pass cannot do without
def _iterations(tol, itmax):
    """Iterations a convergence to `tol` takes on these systems (about 6 per decade), or ITMAX."""
    return min(itmax, round(-7.5 * math.log10(tol)))


def _solve_work(n, prec, tol, itmax):
    """A, B and VAR in, A, B and VAR out; and per iteration, whose two reductions depend on each
    other, the matrix once before each of them and the vectors that must live from one to the next."""
    e = 4 if prec else 8
    it = _iterations(tol, itmax)
    per = (2 * 7 + 14) * e
    return {"bytes": n * (17 * 8 + it * per), "flops": n * it * 2 * (13 + 2 * 2 * 14 + 8)}


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        w = [_solve_work((d[0] + 2) * (d[1] + 2) * (d[2] + 2), case["prec"], tol, 500) for d, _, tol, _ in _dims(case)]
        return {m: sum(x[m] for x in w) for m in ("bytes", "flops")}
    i2, j2, k2 = _box(case["i"], case["j"], case["k"])
    n = i2 * j2 * k2
    if kind == "solve":
        return _solve_work(n, case["prec"], case["tol"], case["itmax"])
    if kind in ("dropin", "momentum", "pp"):
        w = _solve_work(n, 0, 1e-30, case["itmax"])
        m = 3 if kind == "momentum" else 1
        fields = n * (4 + 28 * 8 + 9 * 8) if kind == "pp" else 0
        return {"bytes": m * w["bytes"] + fields, "flops": m * w["flops"] + (80 * n if kind == "pp" else 0)}
    if kind == "msolve":  # the matrix and B in, VAR out; two red/black passes of line solves
        return {"bytes": 9 * 8 * n, "flops": n * (3 + 2 * 14)}
    return {"bytes": 9 * 8 * n, "flops": 15 * n}


def tolerance(case):
    kind = case["kind"]
    if kind == "msolve" or kind == "residual":
        return {"rel": 1e-13, "max": 1e-11}  # sums in another order, 64 bits
    if kind in ("dropin", "momentum", "pp"):
        # a fixed number of BiCGSTAB steps, whose scalars amplify the order of the sums: up to 2e-9 off
        # `exact` after 20 steps, 1e-15 after 5
        return {"rel": 1e-8, "max": 1e-6} if case["itmax"] > 5 else {"rel": 1e-11, "max": 1e-9}
    if kind == "serve":
        # each solution is defined up to its request's TOL times the operator's condition: the FP64
        # and the mixed server differ by 3e-4
        return {"rel": 5e-3, "max": 5e-2}
    # solved to TOL: the FP64 and the mixed form differ by up to 185 TOL
    return {"rel": 1000 * case["tol"], "max": 10000 * case["tol"]}


# ---------------------------------------------------------------- 64-bit results in plain torch
def _shift(x, ax, s):
    """x at the neighbour s = -1 / +1 along ax, clamped at the array edge."""
    m = x.shape[ax]
    idx = (torch.arange(m, device=x.device) + s).clamp(0, m - 1)
    return x.index_select(ax, idx)


def _matvec(A, X):
    y = A[1] * _shift(X, 2, -1) + A[2] * _shift(X, 1, -1) + A[3] * X + A[4] * _shift(X, 1, 1) + A[5] * _shift(X, 2, 1)
    if X.shape[0] > 1:
        y = y + A[0] * _shift(X, 0, -1) + A[6] * _shift(X, 0, 1)
    return y


class _Line:
    """LEQ_MSOLVE with RSRS: two passes of red, then black J-line solves (Thomas, all lines at once)."""

    def __init__(self, A):
        self.A, (self.k2, self.i2, self.j2) = A, A.shape[1:]
        kk = torch.arange(self.k2, device=A.device)[:, None] + 1
        ii = torch.arange(self.i2, device=A.device)[None, :] + 1
        odd = (ii + kk) % 2 == 1 if self.k2 > 1 else ((ii % 2 == 1) & (kk > 0))
        self.colour = [odd[..., None], ~odd[..., None]]
        sub, dia, sup = (A[q].permute(2, 0, 1).contiguous() for q in (1, 3, 5))
        self.l, self.u, self.c = torch.zeros_like(sub), dia.clone(), sup
        for r in range(1, self.j2):
            self.l[r] = sub[r] / self.u[r - 1]
            self.u[r] = dia[r] - self.l[r] * sup[r - 1]

    def __call__(self, B):
        X = B.clone()
        for _ in range(2):
            for colour in self.colour:
                f = B - self.A[2] * _shift(X, 1, -1) - self.A[4] * _shift(X, 1, 1)
                if self.k2 > 1:
                    f = f - self.A[0] * _shift(X, 0, -1) - self.A[6] * _shift(X, 0, 1)
                f = f.permute(2, 0, 1).contiguous()
                for r in range(1, self.j2):
                    f[r] -= self.l[r] * f[r - 1]
                f[-1] /= self.u[-1]
                for r in range(self.j2 - 2, -1, -1):
                    f[r] = (f[r] - self.c[r] * f[r + 1]) / self.u[r]
                X = torch.where(colour, f.permute(1, 2, 0), X)
        return X


def _mix64(z):
    with np.errstate(over="ignore"):
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


def _rtilde(n):
    """The stream that stands for RANDOM_NUMBER in Rtilde (option rtilde_seed at its default)."""
    m = (1 << 64) - 1
    key = (0x5EED * 0x9E3779B97F4A7C15 + 0xA1 * 0xD1B54A32D192ED03 + 0x632BE59BD9B4E019) & m
    key = _mix64(np.array([key], dtype=np.uint64))
    with np.errstate(over="ignore"):
        v = _mix64(key + (np.arange(n, dtype=np.uint64) + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15))
    return torch.from_numpy((v >> np.uint64(11)).astype(np.float64) * 2.0 ** -53).to(DEV)


def _scaled(a, b, box):
    shape = (box[2], box[0], box[1])
    oam = 1.0 / a.abs().amax(dim=0)
    return (a * oam).reshape(7, *shape), (b * oam).reshape(shape)


def _capped(A, B, itmax, tol):
    """BiCGSTAB's solution from zero after ITMAX steps or at TOL (model/leq_bicgs.f), LINE preconditioner."""
    M, X, R = _Line(A), torch.zeros_like(B), B.clone()
    rn0 = R.norm()
    Rt = R + ((2.0 * _rtilde(R.numel()) - 1.0) * 1e-6 * rn0).reshape(R.shape)
    rho = (Rt * R).sum()
    P = R
    for _ in range(itmax):
        Ph = M(P)
        V = _matvec(A, Ph)
        alpha = rho / (Rt * V).sum()
        S = R - alpha * V
        Sh = M(S)
        T = _matvec(A, Sh)
        omega = (T * S).sum() / (T * T).sum()
        X = X + alpha * Ph + omega * Sh
        R = S - omega * T
        if float(R.norm()) <= tol * float(rn0):
            break
        rho1 = (Rt * R).sum()
        P = R + (rho1 / rho) * (alpha / omega) * (P - omega * V)
        rho = rho1
    return X


def _solution(A, B):
    """A x = B to 64-bit accuracy: diagonally preconditioned BiCGSTAB with restarts on the true residual."""
    D, X, R = 1.0 / A[3], torch.zeros_like(B), B.clone()
    bn = float(B.norm())
    for _ in range(40):
        Rt, P, V = R.clone(), torch.zeros_like(R), torch.zeros_like(R)
        rho = alpha = omega = torch.ones((), dtype=F64, device=B.device)
        r0 = float(R.norm())
        for it in range(2000):
            rho1 = (Rt * R).sum()
            P = R + (rho1 / rho) * (alpha / omega) * (P - omega * V)
            Ph = D * P
            V = _matvec(A, Ph)
            alpha = rho1 / (Rt * V).sum()
            S = R - alpha * V
            Sh = D * S
            T = _matvec(A, Sh)
            omega = (T * S).sum() / (T * T).sum()
            X = X + alpha * Ph + omega * Sh
            R = S - omega * T
            rho = rho1
            if it % 16 == 15 and float(R.norm()) <= max(1e-4 * r0, 1e-15 * bn):
                break
        R = B - _matvec(A, X)
        if float(R.norm()) <= 1e-13 * bn:
            break
    return X


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return None  # solutions to 1e-6 and 1e-8 of systems whose condition reaches 1e6: no digits to hold to
    if kind in ("dropin", "momentum"):
        s = prepare(case, seed)
        done = [_scaled(s.a0[q].to(DEV), s.b0[q].to(DEV), s.box) for q in range(len(s.x))]
        x = [_capped(A, B, case["itmax"], case["tol"]) for A, B in done]
        return {"x": [v.reshape(-1).cpu() for v in x],
                "a": torch.stack([A.reshape(7, -1) for A, _ in done]).cpu(),
                "b": torch.stack([B.reshape(-1) for _, B in done]).cpu(), "ier": None}
    if kind in ("solve", "batch"):
        if kind == "solve" and (case["i"] + 2) * (case["j"] + 2) * (case["k"] + 2) > 9e6:
            return None  # over 20 seconds
        specs = _dims(case) if kind == "batch" else [((case["i"], case["j"], case["k"]), "conv_diff", case["tol"], 0)]
        m = _Many(specs, seed)
        m.x.zero_()
        m.a.zero_()
        m.b.zero_()
        for q, (pa, pb) in zip(m.sys, m.at):
            A, B = _scaled(m.a0[pa:pa + 7 * q.n].reshape(7, -1), m.b0[pb:pb + q.n], (q.imax2, q.jmax2, q.kmax2))
            m.a[pa:pa + 7 * q.n], m.b[pb:pb + q.n] = A.reshape(-1), B.reshape(-1)
            m.x[pb:pb + q.n] = _solution(A, B).reshape(-1)
        return {"x": m.x, "a": m.a, "b": m.b, "ier": None}
    if kind == "pp":
        return _exact_pp(case, seed)
    s = prepare(case, seed)
    shape = (s.geom.kmax2, s.geom.imax2, s.geom.jmax2)
    A, B = s.a.reshape(7, *shape), s.b.reshape(shape)
    if kind == "msolve":
        return _Line(A)(B).reshape(-1)
    y = _matvec(A, B)
    return {"y": y.reshape(-1), "dot": float((y * B).sum())}


def _exact_pp(case, seed):
    """CONV_PP_G and SOURCE_PP_G for one solids phase (model/conv_pp_g.f:80-178,
    model/source_pp_g.f:87-162), then ITMAX steps of BiCGSTAB."""
    f, box, n = _fields(case, seed)
    shape = (box[2], box[0], box[1])
    v = {k: t.reshape(-1, *shape) for k, t in f.items()}
    one = {k: t[0] for k, t in v.items()}
    odt = 100.0
    A = torch.zeros((7, *shape), dtype=F64, device=DEV)
    mx = torch.zeros(shape, dtype=F64, device=DEV)
    B = torch.zeros(shape, dtype=F64, device=DEV)
    for ph, (re, rn, rt, u, vv, w, rop, ropo, src) in enumerate(
            (("rop_ge", "rop_gn", "rop_gt", "u_g", "v_g", "w_g", "rop_g", "rop_go", "sum_r_g"),
             ("rop_se", "rop_sn", "rop_st", "u_s", "v_s", "w_s", "rop_s", "rop_so", "sum_r_s"))):
        terms = [(one[rop] - one[ropo]) * one["vol"] * odt]
        for ax, r, area, vel, d, hi, lo in ((1, re, "ayz", u, "d_e", 4, 2), (2, rn, "axz", vv, "d_n", 5, 1),
                                            (0, rt, "axy", w, "d_t", 6, 0)):
            face = one[r] * one[area]
            below, flux = _shift(face, ax, -1), face * one[vel]
            A[hi] += face * v[d][ph]
            A[lo] += below * _shift(v[d][ph], ax, -1)
            terms += [flux, -_shift(flux, ax, -1)]
        gain = one[src] * one["vol"]
        B += sum(terms) - gain
        if ph == 0:
            mx = torch.stack([t.abs() for t in terms + [gain]]).amax(dim=0)
    A[3] = -(A[0] + A[1] + A[2] + A[4] + A[5] + A[6])
    flow = one["flag"] == 11  # links to pressure-flow cells are cut
    for ax, hi, lo in ((1, 4, 2), (2, 5, 1), (0, 6, 0)):
        A[hi][_shift(flow, ax, 1)] = 0.0
        A[lo][_shift(flow, ax, -1)] = 0.0
    fluid = one["flag"] == 1
    A = torch.where(fluid, A, torch.zeros_like(A))
    A[3] = torch.where(fluid, A[3], torch.full_like(A[3], -1.0))
    B, mx = torch.where(fluid, B, torch.zeros_like(B)), torch.where(fluid, mx, torch.zeros_like(mx))
    As, Bs = _scaled(A.reshape(7, -1), B.reshape(-1), box)
    x = _capped(As, Bs, case["itmax"], case["tol"])
    return {"x": x.reshape(-1), "a": As.reshape(-1), "b": Bs.reshape(-1),
            "bmmax": mx.reshape(-1), "ier": None}
