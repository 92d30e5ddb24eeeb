"""Rounding of the y-derivatives against the compact schemes solved in extended
precision: no more than the reference's order of operations leaves, which the
oracle runs with every product rounded."""
import numpy as np
import pytest

from trans_bl_gb300 import api, configs

pytestmark = pytest.mark.gpu

LD = np.longdouble


def exact(cfg, coefs, op, f):
    """dery, deryfv and deryy (derivs_par.f:116-177, 400-611, 1040-1142) of f (ny, nx) in extended precision."""
    n, p = cfg.ny, 0
    part = {}
    for name, m in (("fp1", 6), ("sp1", 9), ("cp1", 8), ("pp1", 9), ("lp1", 7), ("fp2", 8), ("sp2", 10), ("cp2", 8), ("pp2", 10),
                    ("lp2", 8)):
        part[name] = np.asarray(coefs[p:p + m]).astype(LD)
        p += m
    d = "2" if op == "deryy" else "1"
    fp, sp, cp, pp, lp = (part[k + d] for k in ("fp", "sp", "cp", "pp", "lp"))
    q = 1 / (LD(cfg.dy) * LD(cfg.stf) ** np.arange(n))
    if d == "2":
        q = q * q
    a, b, c = np.zeros(n, LD), np.ones(n, LD), np.zeros(n, LD)
    if op != "deryfv":
        b[0] = fp[0]
    if d == "2":
        c[0] = fp[1]
    a[1], b[1], c[1] = sp[:3]
    a[2:n - 2], b[2:n - 2], c[2:n - 2] = cp[0], cp[1], cp[2]
    a[n - 2], b[n - 2], c[n - 2] = pp[2], pp[1], pp[0]
    a[n - 1], b[n - 1] = lp[1], lp[0]
    f = f.astype(np.clongdouble)
    r = np.zeros_like(f)
    wall, top = (fp[1:], (5, 6)) if d == "1" else (fp[2:], (6, 7))
    if op != "deryfv":
        r[0] = sum(wall[m] * f[m] for m in range(top[0])) * q[0]
    r[1] = sum(sp[3 + m] * f[m] for m in range(top[1])) * q[0]
    r[2:n - 2] = sum(cp[3 + m] * f[m:n - 4 + m] for m in range(5)) * q[:n - 4, None]
    r[n - 2] = sum(pp[3 + m] * f[n - 1 - m] for m in range(top[1])) * q[n - 6 if d == "1" else n - 7]
    r[n - 1] = sum(lp[2 + m] * f[n - 1 - m] for m in range(top[0])) * q[n - 5 if d == "1" else n - 6]
    # Gaussian elimination of the tridiagonal system
    for j in range(1, n):
        w = a[j] / b[j - 1]
        b[j] = b[j] - w * c[j - 1]
        r[j] = r[j] - w * r[j - 1]
    r[n - 1] /= b[n - 1]
    for j in range(n - 2, -1, -1):
        r[j] = (r[j] - c[j] * r[j + 1]) / b[j]
    return r


@pytest.mark.parametrize("ny", [97, 129, 161, 193, 257])
def test_y_derivatives_round_no_more_than_the_reference(oracle_built, ny):
    nx, K = 257, 2
    cfg = configs.blasius_ts_config(nx, ny, K, 4, 3)
    coefs = api.generate_coefs(cfg.stf, cfg.msh)
    base = [np.zeros((ny, nx))] * 3
    g, o = api.Context(cfg, coefs, base), oracle_built.Oracle(cfg, coefs, base)
    f = configs.smooth_random((K, ny, nx), np.random.default_rng(ny), 1.0)
    for op in ("dery", "deryfv", "deryy"):
        want = exact(cfg, coefs, op, f[1])
        rms = [float(np.sqrt(np.mean(np.abs(getattr(c, op)(f)[1] - want) ** 2))) for c in (g, o)]
        assert rms[0] <= rms[1], (op, rms)
