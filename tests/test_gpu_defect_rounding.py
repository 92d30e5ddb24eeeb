"""Rounding of the mixed form's FP64 defect, which decides when a solve stops.

A field u whose source is L u to the last digit leaves a defect of rounding
alone, and a solve with a tolerance that any defect meets reports its largest
value per mode without changing u.  The same defect summed term by term in
64 bits on the host, every product rounded, is what the GPU's fused
multiply-adds may not exceed.
"""
import numpy as np
import pytest

from trans_bl_gb300 import api, configs

pytestmark = pytest.mark.gpu

LD = np.longdouble
K = 32


def operator(cfg, coefs, k, u, T):
    """L u of mode k term by term in precision T (defect, poisson_par.f:543-793)."""
    ny, msh, b = cfg.ny, cfg.msh, np.asarray(coefs[83:]).astype(T)
    SP, CP, PP, LP = b, b[7 * msh:], b[15 * msh:], b[19 * msh:]
    dy = LD(cfg.dy) * LD(cfg.stf) ** np.arange(ny)
    q2 = (1 / (dy * dy)).astype(T)
    den, ify = T(1) / (T(12) * T(cfg.dx) ** 2 * T(cfg.fac_y)), T(1) / T(cfg.fac_y)
    k2 = -(T(k) * T(cfg.beta)) ** 2
    u = u.astype(np.clongdouble if T is LD else np.complex128)
    x = np.zeros_like(u)
    x[:, 2:-2] = -u[:, :-4] + T(16) * u[:, 1:-3] - T(30) * u[:, 2:-2] + T(16) * u[:, 3:-1] - u[:, 4:]
    for i, e in ((1, 1), (cfg.nx - 2, -1)):
        x[:, i] = (T(10) * u[:, i - e] - T(15) * u[:, i] - T(4) * u[:, i + e] + T(14) * u[:, i + 2 * e] - T(6) * u[:, i + 3 * e] +
                   u[:, i + 4 * e])
    L = np.zeros_like(u)
    L[1] = ((SP[1] * x[1] + SP[2] * x[2]) * den + sum(SP[3 + q] * u[q] for q in range(4)) * q2[0] +
            k2 * (SP[1] * u[1] + SP[2] * u[2]) * ify)
    n = ny - 3      # rows 2 .. ny-3
    cc = sum(CP[3 + q] * u[q:n - 1 + q] for q in range(5))
    L[2:n + 1] = (sum(CP[q] * x[1 + q:n + q] for q in range(3)) * den + cc * q2[:n - 1, None] +
                  k2 * sum(CP[q] * u[1 + q:n + q] for q in range(3)) * ify)
    m = ny - 2
    L[m] = x[m] * den + (PP[3] * u[m + 1] + PP[2] * u[m] + PP[1] * u[m - 1]) * q2[m - 1] + k2 * u[m] * ify
    m = ny - 1
    L[m] = (x[m] * den + (LP[2] * u[m] + LP[3] * u[m - 1] + LP[4] * u[m - 2]) * q2[m - 2] + k2 * u[m] * ify -
            LP[1] * np.sqrt((T(cfg.alpha) ** 2 - k2) * ify) * np.sqrt(q2[m - 2]) * u[m])
    return L


def source(cfg, coefs, S, T):
    """function_source (poisson_par.f:111-164) of S, zero on the top row."""
    msh, b = cfg.msh, np.asarray(coefs[83:]).astype(T)
    SP, CP = b, b[7 * msh:]
    s = np.zeros_like(S)
    s[1] = SP[1] * S[1] + SP[2] * S[2]
    s[2:-2] = CP[0] * S[1:-3] + CP[1] * S[2:-2] + CP[2] * S[3:-1]
    s[-2] = S[-2]
    return s


def invert_source(cfg, coefs, s):
    """S with source(S) = s, rows 1 .. ny-2, by elimination from the top."""
    msh, b = cfg.msh, np.asarray(coefs[83:]).astype(LD)
    SP, CP, n = b, b[7 * msh:], cfg.ny
    S = np.zeros_like(s)
    # S_j = r_j + c_j S_{j-1}
    r, c = np.zeros_like(s), np.zeros(n, LD)
    r[n - 2] = s[n - 2]
    for j in range(n - 3, 1, -1):
        p = CP[1] + CP[2] * c[j + 1]
        r[j], c[j] = (s[j] - CP[2] * r[j + 1]) / p, -CP[0] / p
    S[1] = (s[1] - SP[2] * r[2]) / (SP[1] + SP[2] * c[2])
    for j in range(2, n - 1):
        S[j] = r[j] + c[j] * S[j - 1]
    return S


@pytest.mark.parametrize("nx,ny", [(129, 97), (257, 129), (129, 193), (97, 257)])
def test_defect_rounds_no_more_than_its_terms(nx, ny):
    """The modes' largest rounding errors, their root mean square (31 of them)."""
    nl = 12.0 * (nx - 1) / 1024
    cfg = configs.blasius_ts_config(nx, ny, K, 2 * K, 4, n_lambda=nl, strip=(0.3 * nl, 0.4 * nl), precision=api.FORM_MIXED)
    coefs = api.generate_coefs(cfg.stf, cfg.msh)
    ctx = api.Context(cfg, coefs, [np.zeros((ny, nx))] * 3)
    y = np.arange(ny) / (ny - 1.0)
    shape = np.where(y < 0.9, (y * (1 - y / 0.9)) ** 2, 0.0)[:, None]   # zero at the wall and near the top
    u = configs.smooth_random((K, ny, nx), np.random.default_rng(nx), 1.0) * (1.0 + np.arange(K))[:, None, None] * shape
    st = {n: np.zeros((K, ny, nx), complex) for n in configs.NAMES}
    st["uy"] = u
    d = np.zeros((K, ny, nx), complex)
    host = np.zeros(K)
    for k in range(1, K):
        d[k] = -invert_source(cfg, coefs, operator(cfg, coefs, k, u[k], LD)).astype(complex)
        r = source(cfg, coefs, -d[k], float) - operator(cfg, coefs, k, u[k], float)
        host[k] = np.max(np.abs(r[1:, 1:-1]))
    ctx.put_state(st)
    ctx.poi_uy(d, 1e300)
    got = np.array(ctx.poisson_stats()["residual"])
    rms = [float(np.sqrt(np.mean(v[1:] ** 2))) for v in (got, host)]
    assert rms[0] <= rms[1], rms


@pytest.mark.parametrize("n_lambda,counts", [(6.0, [7, 6, 6, 6]), (3.0, [7, 7, 7, 6])])
def test_257_rows_converge_at_1e_8(n_lambda, counts):
    """The 257-row grid of the roughness runs (first cell 0.005 delta*) at their
    tolerance, not far above the defect's rounding there, with their x spacing and
    half of it: every mode converges, with the corrections of a defect that forms
    the operator's terms one by one."""
    kw = dict(amp2d=3e-3, amp3d=3e-3, strip=(0.5, 1.0), n_lambda=n_lambda)
    cfg = configs.blasius_ts_config(513, 257, 4, 8, 4, max_vcycles=11, precision=api.FORM_MIXED, **kw)
    # the base flow of 17 stations, repeated
    base = [np.ascontiguousarray(np.resize(b.T, (513, 257)).T)
            for b in api.baseflow_fs(configs.blasius_ts_config(17, 257, 4, 8, 2, **kw), 0.0)]
    ctx = api.Context(cfg, api.generate_coefs(cfg.stf, cfg.msh), base)
    ctx.put_state(configs.disturbed_state(cfg, base, np.random.default_rng(23), 1e-3))
    ctx.poi_uy(ctx.outuy(), 1e-8)
    ps = ctx.poisson_stats()
    assert ps["noconv"] == 0 and ps["vcycles"] == counts
