"""The work that users of this library run, as timed cases.

A user of the library advances boundary-layer runs: the RK4 step of the plain
FP64 form (the drop-in) and of the mixed form, in every physics form, alone
and as an ensemble; or a host program calls single operators of the stage.
The grids are those of trans_bl_gb300/configs.py (the flat-plate TS cases from
385 x 129 in 2D to 1025 x 193 with 32 and 64 modes, and the uneven grids of
the ensemble), and `draw` gives more of the same ranges.

Every step case starts from the Blasius base flow plus a seeded smooth
disturbance past the forcing ramp, as bench.py does, and each pass advances
the run by one step; the six fields stay on the device and are returned as
views of them.  The operator cases run on seeded smooth fields.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from trans_bl_gb300 import api, configs

NAMES = ("ux", "uy", "uz", "wx", "wy", "wz")


def listed():
    return [
        # 2D TS run, drop-in form: one Fourier mode, the smallest call, where latency counts
        {"name": "step_plain_2d", "kind": "step", "form": "plain", "nx": 385, "ny": 129, "K": 1, "P": 2, "msh": 3},
        # 3D run of the drop-in form, FP64 everywhere
        {"name": "step_plain_3d", "kind": "step", "form": "plain", "nx": 513, "ny": 129, "K": 8, "P": 16, "msh": 4},
        # the smallest member of the ensemble workload run on its own
        {"name": "step_mixed_small", "kind": "step", "form": "mixed", "nx": 257, "ny": 97, "K": 8, "P": 16, "msh": 4},
        # an ordinary 3D run
        {"name": "step_mixed_mid", "kind": "step", "form": "mixed", "nx": 769, "ny": 129, "K": 16, "P": 32, "msh": 4},
        # the benchmark's 3D run
        {"name": "step_mixed_large", "kind": "step", "form": "mixed", "nx": 1025, "ny": 193, "K": 32, "P": 64, "msh": 4},
        # LES with a wall roughness element at 64 modes: the largest run here
        {"name": "step_les_roughness", "kind": "les", "form": "mixed", "nx": 1025, "ny": 193, "K": 64, "P": 128, "msh": 4},
        # Goertler vortices: linear modes about the base flow
        {"name": "step_gortler", "kind": "gortler", "form": "mixed", "nx": 257, "ny": 65, "K": 8, "P": 16, "msh": 4},
        # heated wall: a seventh field, FP64 transforms
        {"name": "step_thermal", "kind": "thermal", "form": "mixed", "nx": 257, "ny": 97, "K": 16, "P": 32, "msh": 4},
        # four uneven runs advanced together, one launch per step
        {"name": "ensemble_4", "kind": "ensemble", "form": "mixed", "members": 4, "pick": 20261203},
        # a Fortran host's calls of derparx and derparxx on its own arrays
        {"name": "xderiv_host", "kind": "xderiv", "form": "plain", "nx": 385, "ny": 129, "K": 8, "P": 16, "msh": 3},
        # filter_trid on a host program's device buffers, no context and no allocation
        {"name": "filter_noalloc", "kind": "filter", "nx": 513, "ny": 97, "K": 32},
    ]


def draw(rng):
    """One more case: the same kinds of call on other grids.  nx - 1 and ny - 1
    are multiples of 2^(msh-1), as the multigrid levels need, and K is any
    number of modes up to P/2."""
    kind = rng.choice(["plain", "mixed", "mixed", "mixed", "les", "gortler", "thermal", "ensemble", "xderiv", "filter"])

    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def modes(lo, hi):
        k = log_int(lo, hi)
        p = 2
        while p < 2 * k:
            p *= 2
        return k, p

    ny = 1 + 8 * rng.randint(8, 24)                       # 65 .. 193
    if kind == "plain":
        k, p = modes(1, 8)
        return {"kind": "step", "form": "plain", "nx": 1 + 8 * log_int(16, 64), "ny": 1 + 8 * rng.randint(8, 16), "K": k,
                "P": p, "msh": rng.choice([3, 4])}
    if kind == "mixed":
        k, p = modes(2, 32)
        return {"kind": "step", "form": "mixed", "nx": 1 + 32 * log_int(6, 32), "ny": ny, "K": k, "P": p, "msh": 4}
    if kind == "les":
        k, p = modes(4, 48)
        return {"kind": "les", "form": "mixed", "nx": 1 + 32 * log_int(8, 32), "ny": ny, "K": k, "P": p, "msh": 4}
    if kind in ("gortler", "thermal"):
        k, p = modes(2, 16)
        return {"kind": kind, "form": rng.choice(["mixed", "mixed", "plain"]), "nx": 1 + 32 * log_int(4, 16),
                "ny": 1 + 8 * rng.randint(8, 16), "K": k, "P": p, "msh": 4}
    if kind == "ensemble":
        return {"kind": "ensemble", "form": "mixed", "members": rng.randint(2, 5), "pick": rng.randint(1, 10 ** 6)}
    if kind == "xderiv":
        k, p = modes(1, 16)
        return {"kind": "xderiv", "form": "plain", "nx": 1 + 4 * log_int(32, 256), "ny": 1 + 4 * rng.randint(8, 32), "K": k,
                "P": p, "msh": 3}
    nx = log_int(65, 1025)
    nyf = rng.randint(33, 193)
    return {"kind": "filter", "nx": nx, "ny": nyf, "K": max(1, min(rng.randint(1, 32), (2 ** 21 - 4096) // (nx * nyf)))}


# ---- configurations -------------------------------------------------------
def config_of(c):
    prec = api.FORM_PLAIN_FP64 if c["form"] == "plain" else api.FORM_MIXED
    kw = dict(precision=prec, amp2d=1e-4, amp3d=1e-5)
    if c["nx"] < 257:      # a short domain keeps the streamwise resolution of the TS wave
        kw.update(n_lambda=4.0, strip=(1.0, 1.6))
    if c["kind"] == "les":
        # the physics of configs.config5 (LES with van Driest damping on |wall
        # vorticity|, a roughness element, TS and oblique forcing at 3e-3)
        kw.update(my_form=4, tol=1e-8, amp2d=3e-3, amp3d=3e-3)
    elif c["kind"] == "gortler":
        kw.update(my_form=1)
    elif c["kind"] == "thermal":
        kw.update(my_form=2)
    cfg = configs.blasius_ts_config(c["nx"], c["ny"], c["K"], c["P"], c["msh"], **kw)
    cfg.stpp = configs.stable_steps_per_period(cfg)
    if c["kind"] == "gortler":
        cfg.go_number = 2.0
    if c["kind"] == "les":
        dstar = configs.BLASIUS_DSTAR / math.sqrt(cfg.Re)
        cfg.ibm = 1
        cfg.ibm_xc = cfg.x0 + 0.25 * (cfg.nx - 1) * cfg.dx
        cfg.ibm_zc = math.pi / cfg.beta
        cfg.ibm_h = 0.5 * dstar
        cfg.ibm_R = 1.0 * dstar
        cfg.irf = -min(0.1 * cfg.Re, 2.0 / (2.0 * math.pi / cfg.omega / cfg.stpp))
        cfg.C_s = 0.1
        cfg.A_plus = 26.0
        cfg.les_damping = 3
    return cfg


def ensemble_configs(c):
    return configs.config3(seed=c["pick"], members=c["members"], precision=api.FORM_MIXED)


# ---- inputs ----------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def blasius_profile(h=1.0 / 256.0, eta_max=12.0):
    """f, f', f'' of f''' + f f'' = 0 on a fine grid of eta (RK4)."""
    n = int(round(eta_max / h))
    out = np.zeros((n + 1, 3))
    out[0] = 0.0, 0.0, 0.4695999883610132

    def rate(y):
        return np.array([y[1], y[2], -y[0] * y[2]])

    for q in range(n):
        y = out[q]
        a = rate(y)
        b = rate(y + 0.5 * h * a)
        c = rate(y + 0.5 * h * b)
        d = rate(y + h * c)
        out[q + 1] = y + h / 6.0 * (a + 2.0 * b + 2.0 * c + d)
    return out


def blasius(cfg):
    """Blasius base flow (ux, uy, wz) on cfg's grid (fac_y = 1).  A user's
    program reads it from its file, so it is made here quickly, by Hermite
    interpolation of one profile, and not by the library's shooting."""
    h = 1.0 / 256.0
    p = blasius_profile(h)
    x = cfg.x0 + cfg.dx * np.arange(cfg.nx)[None, :]
    y = cfg.dy * (cfg.stf ** np.arange(cfg.ny) - 1.0)[:, None] / (cfg.stf - 1.0)
    s = np.sqrt(0.5 * cfg.Re / x)
    eta = y * s
    q = np.minimum((eta / h).astype(int), len(p) - 2)
    t = np.minimum(eta / h - q, 1.0)

    def hermite(v, d):
        return ((1 + 2 * t) * (1 - t) ** 2 * v[q] + t * (1 - t) ** 2 * h * d[q] + t * t * (3 - 2 * t) * v[q + 1] +
                t * t * (t - 1) * h * d[q + 1])

    f = hermite(p[:, 0], p[:, 1]) + np.maximum(eta - (len(p) - 1) * h, 0.0)
    f1 = hermite(p[:, 1], p[:, 2])
    f2 = hermite(p[:, 2], -p[:, 0] * p[:, 2])
    return f1, (eta * f1 - f) * np.sqrt(0.5 / (x * cfg.Re)), s * f2


class _Device:
    """Device memory of a context's field as torch sees it; keeps its owner alive."""

    def __init__(self, ptr, shape, owner):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 2}
        self.owner = owner


class _Run:
    """A context (or an ensemble and its members), closed in the right order."""

    def __init__(self, ctxs, ens=None):
        self.ctxs, self.ens = ctxs, ens

    def __del__(self):
        if self.ens is not None:
            self.ens.close()
        for g in self.ctxs:
            g.close()


def smooth(shape, gen, scale):
    """Smooth complex field (K, ny, nx, 2): three waves per mode, mode 0 real, amplitude scale / (1 + k)."""
    K, ny, nx = shape
    d = dict(device="cuda", dtype=torch.float64)
    a, b = (torch.rand((K, 3), generator=gen, **d) * 3.5 + 0.5 for _ in range(2))
    px, py = (torch.rand((K, 3), generator=gen, **d) * 2 * math.pi for _ in range(2))
    re, im = (torch.randn((K, 3), generator=gen, **d) for _ in range(2))
    im[0] = 0.0
    x, y = torch.linspace(0, 1, nx, **d), torch.linspace(0, 1, ny, **d)
    sx = torch.sin(a[..., None] * math.pi * x + px[..., None])
    cy = torch.cos(b[..., None] * math.pi * y + py[..., None])
    s = scale / (1.0 + torch.arange(K, **d))[:, None]
    f = torch.stack([torch.einsum("kp,kpy,kpx->kyx", w * s, cy, sx) for w in (re, im)], dim=-1)
    return f.contiguous()


def fill(ctx, cfg, base, gen, owner):
    """The disturbed start state into the context's resident fields; their views."""
    shape = (cfg.kfour, cfg.ny, cfg.nx)
    views = [torch.as_tensor(_Device(ctx.device_field(q), shape + (2,), owner), device="cuda") for q in range(6)]
    mean = {"ux": base[0], "uy": base[1], "wz": base[2]} if cfg.my_form in (0, 4) else {}
    for n, v in zip(NAMES, views):
        f = smooth(shape, gen, 1e-3)
        if n in ("ux", "uy", "uz"):
            f[:, 0] = 0.0          # no slip
        if n in mean:
            f[0, :, :, 0] += torch.from_numpy(mean[n]).to("cuda")
        v.copy_(f)
    return views


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    kind = case["kind"]
    if kind == "filter":
        shape = (case["K"], case["ny"], case["nx"])
        f = [smooth(shape, gen, 1.0) + 1e-2 * torch.randn(shape + (2,), generator=gen, device="cuda", dtype=torch.float64)
             for _ in range(3)]
        torch.cuda.synchronize()
        return {"kind": kind, "case": case, "f": f}
    if kind == "xderiv":
        cfg = config_of(case)
        ctx = api.Context(cfg, api.generate_coefs(cfg.stf, cfg.msh), blasius(cfg))
        f = smooth((case["K"], case["ny"], case["nx"]), gen, 1.0).cpu().numpy().view(np.complex128)[..., 0]
        return {"kind": kind, "ctx": ctx, "run": _Run([ctx]), "f": f}
    cfgs = ensemble_configs(case) if kind == "ensemble" else [config_of(case)]
    ctxs, bases = [], []
    for cfg in cfgs:
        bases.append(blasius(cfg))
        ctxs.append(api.Context(cfg, api.generate_coefs(cfg.stf, cfg.msh), bases[-1]))
    ens = api.Ensemble(ctxs) if kind == "ensemble" else None
    run_ = _Run(ctxs, ens)
    views = [fill(g, cfg, base, gen, run_) for g, cfg, base in zip(ctxs, cfgs, bases)]
    if kind == "thermal":
        cfg = cfgs[0]
        ctxs[0].set_baseflow_th(configs.base_temperature(cfg, bases[0]))
        th = smooth((cfg.kfour, cfg.ny, cfg.nx), gen, 1e-3)
        th[:, 0] = 0.0
        th[:, -1] = 0.0
        ctxs[0].put_th(th.cpu().numpy().view(np.complex128)[..., 0])
    torch.cuda.synchronize()
    # past the forcing ramp of one period
    return {"kind": kind, "run": run_, "ctx": ctxs[0], "ens": ens, "views": views, "t": [c.stpp + 1 for c in cfgs]}


def run(state):
    kind = state["kind"]
    if kind == "filter":
        c, f = state["case"], state["f"]
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        p = [ctypes.c_void_p(x.data_ptr()) for x in f]
        api.check(api.load().tb_filter_trid_noalloc(p[0], p[1], p[2], c["nx"], c["ny"], c["K"], 0.48, stream),
                  "tb_filter_trid_noalloc")
        return f
    if kind == "xderiv":
        return [state["ctx"].derparx(state["f"]), state["ctx"].derparxx(state["f"])]
    if kind == "ensemble":
        state["ens"].step(state["t"])
    else:
        state["ctx"].step(state["t"][0])
    state["t"] = [t + 1 for t in state["t"]]
    out = [v for views in state["views"] for v in views]
    if kind == "thermal":
        out.append(state["ctx"].get_th())
    return out


# ---- what one pass cannot do without ------------------------------------
def work(case):
    """Every input read once and every output written once.  The operations
    of a step, per point and stage: 16 compact line operators (10 a real
    part), two pentadiagonal solves (20), and one residual (22) and three
    relaxations (24) of the v-Poisson problem; the transforms add 9 real FFTs
    of length P over the modes."""
    if case["kind"] == "ensemble":
        grids = [(c.nx, c.ny, c.kfour, c.kphys) for c in ensemble_configs(case)]
    else:
        grids = [(case["nx"], case["ny"], case["K"], case.get("P", 2))]
    total = {"bytes": 0.0, "flops": 0.0}
    for nx, ny, K, P in grids:
        n = float(nx) * ny * K
        if case["kind"] == "filter":
            total["bytes"] += 3 * 2 * 16 * n
            total["flops"] += 3 * 2 * 12 * n
        elif case["kind"] == "xderiv":
            total["bytes"] += 3 * 16 * n
            total["flops"] += 2 * 2 * 9 * n
        else:
            fields = 7 if case["kind"] == "thermal" else 6
            total["bytes"] += fields * 2 * 16 * n
            total["flops"] += 4 * 2 * (16 * 10 + 2 * 20 + 22 + 3 * 24) * n + 4 * 9 * 2.5 * P * math.log2(max(P, 2)) * nx * ny
    return total


# ---- the operators in 64 bits ----------------------------------------------
def line_operator(n, lhs, rhs):
    """The dense pair (A, B) of a compact scheme A y = B f along a line of n
    points: `lhs` and `rhs` give the rows at the low end, the rows at the high
    end (counted and indexed from that end) and the interior row as
    (column or offset, value) pairs."""
    pair = []
    for low, high, inner in (lhs, rhs):
        M = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        for r, cols in enumerate(low):
            for c, v in cols:
                M[r, c] = v
        for r, cols in enumerate(high):
            for c, v in cols:
                M[n - 1 - r, n - 1 - c] = v
        i = torch.arange(len(low), n - len(high), device="cuda")
        for off, v in inner:
            M[i, i + off] = v
        pair.append(M)
    return pair


def along_x(pair, x):
    """y of A y = B f for every line of x (K, ny, nx, 2)."""
    A, B = pair
    n = A.shape[0]
    f = x.permute(2, 0, 1, 3).reshape(n, -1)
    return torch.linalg.solve(A, B @ f).reshape(n, *x.shape[:2], 2).permute(1, 2, 0, 3).contiguous()


def en(*v):
    return list(enumerate(v))


def exact(case, seed):
    n = case.get("nx")
    if case["kind"] == "filter":
        # the three rows at each end explicit, the interior with alpha_f =
        # 0.48; the fields' first row and first column stay as they are
        al = 0.48
        w = [(11 + 10 * al) / 16, (15 + 34 * al) / 64, (-3 + 6 * al) / 32, (1 - 2 * al) / 64]
        one = [[(r, 1.0)] for r in range(3)]
        end = [[(q, v / 16.0) for q, v in en(*row)] for row in ((15, 4, -6, 4, -1), (1, 12, 6, -4, 1), (-1, 4, 10, 4, -1))]
        op = line_operator(n, (one, one, [(-1, al), (0, 1.0), (1, al)]),
                           (end, end, [(0, w[0])] + [(s * q, w[q]) for q in (1, 2, 3) for s in (1, -1)]))
        out = []
        for x in prepare(case, seed)["f"]:
            y = along_x(op, x)
            y[:, 0] = x[:, 0]
            y[:, :, 0] = x[:, :, 0]
            out.append(y)
        return out
    if case["kind"] == "xderiv":
        state = prepare(case, seed)
        h = state["ctx"].cfg.dx
        d1 = line_operator(n, ([en(1.0), en(1.0, 6.0, 2.0)], [en(1.0, 4.0), en(1.0, 6.0, 2.0)], [(-1, 1.0), (0, 3.0), (1, 1.0)]),
                           ([[(q, v / (12 * h)) for q, v in en(-25, 48, -36, 16, -3)],
                             [(q, v / (120 * h)) for q, v in en(-406, -300, 760, -80, 30, -4)]],
                            [[(q, v / (-24 * h)) for q, v in en(-74, 16, 72, -16, 2)],
                             [(q, v / (-120 * h)) for q, v in en(-406, -300, 760, -80, 30, -4)]],
                            [(s * q, s * v / (12 * h)) for q, v in ((1, 28.0), (2, 1.0)) for s in (1, -1)]))
        end = [[(q, v / (60 * h * h)) for q, v in en(9775, -20285, 11170, -550, -145, 35)],
               [(q, v / (360 * h * h)) for q, v in en(4834, -8424, 1890, 2320, -810, 216, -26)]]
        lhs = [en(13.0, 137.0), en(1.0, 12.0, 3.0)]
        d2 = line_operator(n, (lhs, lhs, [(-1, 2.0), (0, 11.0), (1, 2.0)]),
                           (end, end, [(0, -102 / (4 * h * h))] +
                            [(s * q, v / (4 * h * h)) for q, v in ((1, 48.0), (2, 3.0)) for s in (1, -1)]))
        f = torch.from_numpy(state["f"].view(np.float64).reshape(state["f"].shape + (2,))).to("cuda")
        return [along_x(op, f).cpu().numpy().view(np.complex128)[..., 0] for op in (d1, d2)]
    return None
