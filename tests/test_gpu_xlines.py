"""The x-line solves at the edges of their chunks against dense 64-bit algebra.

A warp owns a line in 32 chunks of ceil(n / 32) rows: lengths around multiples
of 32, the shortest lines, empty last chunks, and lines so long that the row
tables stay in global memory; the filter for pivots that settle at once,
after tens of rows, and not within one kernel argument.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def filter_matrices(n, al):
    A, B = np.eye(n), np.zeros((n, n))
    ends = [[15, 4, -6, 4, -1], [1, 12, 6, -4, 1], [-1, 4, 10, 4, -1]]
    for r in range(3):
        B[r, :5] = np.array(ends[r]) / 16.0
        B[n - 1 - r, n - 5:] = np.array(ends[r])[::-1] / 16.0
    w = [(11 + 10 * al) / 16, (15 + 34 * al) / 64, (-3 + 6 * al) / 32, (1 - 2 * al) / 64]
    for i in range(3, n - 3):
        A[i, i - 1] = A[i, i + 1] = al
        for q in range(4):
            B[i, i - q] = B[i, i + q] = w[q]
    return A, B


def derivative_matrices(n, dx):
    """derparx's and derparxx's (A, B), derivs_par.f:259-397, 980-1037."""
    A1, A2, B1, B2 = (np.zeros((n, n)) for _ in range(4))
    for i in range(2, n - 2):
        A1[i, i - 1:i + 2] = 1, 3, 1
        A2[i, i - 1:i + 2] = 2, 11, 2
        B1[i, i - 2:i + 3] = np.array([-1, -28, 0, 28, 1]) / (12 * dx)
        B2[i, i - 2:i + 3] = np.array([1, 16, -34, 16, 1]) * 3 / (4 * dx * dx)
    A1[0, 0] = 1
    A1[1, :3] = 1, 6, 2
    A1[n - 2, n - 3:] = 2, 6, 1
    A1[n - 1, n - 2:] = 4, 1
    B1[0, :5] = np.array([-25, 48, -36, 16, -3]) / (12 * dx)
    B1[1, :6] = np.array([-406, -300, 760, -80, 30, -4]) / (120 * dx)
    B1[n - 2, n - 6:] = np.array([4, -30, 80, -760, 300, 406]) / (120 * dx)
    B1[n - 1, n - 5:] = np.array([-2, 16, -72, -16, 74]) / (24 * dx)
    ends = [([13, 137], [9775, -20285, 11170, -550, -145, 35], 60), ([1, 12, 3], [4834, -8424, 1890, 2320, -810, 216, -26], 360)]
    for r, (a, b, d) in enumerate(ends):
        A2[r, :len(a)] = a
        B2[r, :len(b)] = np.array(b) / (d * dx * dx)
        A2[n - 1 - r, n - len(a):] = a[::-1]
        B2[n - 1 - r, n - len(b):] = B2[r, :len(b)][::-1]
    return (A1, B1), (A2, B2)


@pytest.mark.parametrize("al", [0.48, 0.0, -0.3, 0.4999999])
@pytest.mark.parametrize("nx,ny,kfour", [(8, 3, 2), (9, 2, 1), (31, 3, 2), (32, 3, 2), (33, 3, 2), (64, 3, 1), (65, 3, 1),
                                         (97, 5, 3), (513, 9, 2), (1025, 3, 1), (2049, 2, 1), (4096, 2, 1)])
def test_noalloc_filter_lines(nx, ny, kfour, al):
    """Rows i >= 2 of the lines j >= 2 are filtered, the rest stays.  The bound:
    both LHS and RHS act on values of size 1, so the error is a few roundings
    per row times the condition of the LHS, at most (1 + 2|al|) / (1 - 2|al|)
    and no more than the line's length squared."""
    import torch
    from trans_bl_gb300 import api
    rng = np.random.default_rng(nx)
    f = rng.uniform(-1, 1, (3, kfour, ny, nx, 2))
    t = [torch.from_numpy(x.copy()).cuda() for x in f]
    rc = api.load().tb_filter_trid_noalloc(*[ctypes.c_void_p(x.data_ptr()) for x in t], nx, ny, kfour, al,
                                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    api.check(rc, "tb_filter_trid_noalloc")
    torch.cuda.synchronize()
    A, B = filter_matrices(nx, al)
    want = f.copy()
    lines = np.moveaxis(f[:, :, 1:], 3, 0).reshape(nx, -1)
    got = np.linalg.solve(A, B @ lines).reshape((nx,) + np.moveaxis(f[:, :, 1:], 3, 0).shape[1:])
    want[:, :, 1:, 1:] = np.moveaxis(got, 0, 3)[:, :, :, 1:]
    cond = min((1 + 2 * abs(al)) / (1 - 2 * abs(al)), float(nx) ** 2)
    for a, b in zip(t, want):
        assert np.max(np.abs(a.cpu().numpy() - b)) < 64 * EPS * max(cond, 16.0)
        assert np.array_equal(a.cpu().numpy()[:, 0], b[:, 0]) and np.array_equal(a.cpu().numpy()[:, :, 0], b[:, :, 0])


def test_noalloc_filter_same_field_three_times():
    """One buffer given as all three fields is filtered three times, in order."""
    import torch
    from trans_bl_gb300 import api
    nx, ny = 65, 4
    f = np.random.default_rng(3).uniform(-1, 1, (1, ny, nx, 2))
    t = torch.from_numpy(f.copy()).cuda()
    p = ctypes.c_void_p(t.data_ptr())
    api.check(api.load().tb_filter_trid_noalloc(p, p, p, nx, ny, 1, 0.48,
                                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "filter")
    torch.cuda.synchronize()
    A, B = filter_matrices(nx, 0.48)
    want = f.copy()
    for _ in range(3):
        y = np.moveaxis(np.linalg.solve(A, B @ np.moveaxis(want, 2, 0).reshape(nx, -1)).reshape(nx, 1, ny, 2), 0, 2)
        want[:, 1:, 1:] = y[:, 1:, 1:]
    assert np.max(np.abs(t.cpu().numpy() - want)) < 3 * 64 * EPS * 49.0


@pytest.mark.parametrize("nx", [17, 33, 65, 97, 129, 1025, 2049])
def test_derivatives_of_lines(oracle_built, nx):
    """derparx, derparxx and the context's filter against the oracle.  The
    derivatives' bound: each side rounds a row's up to 7 products, the sums and
    the sweep's up to 8 operations, 16 roundings of terms no larger than the sum
    of |weight| times the largest value, seen through the inverse of the LHS;
    the end rows' weights reach 10^4 / dx^2 and cancel, so for the shortest dx
    here that is far above the last digit of the result.  The filter has
    weights below 1: the parity tests' tolerance."""
    from tests.helpers import perturbed_state, rel, small_case
    from trans_bl_gb300 import api, configs
    kw = dict(ny=17, kfour=2, kphys=4, msh=2)
    cfg = configs.small(nx=nx, **kw)
    _, coefs, base = small_case(nx=17, **kw)
    base = [np.ascontiguousarray(np.resize(b.T, (nx, 17)).T) for b in base]   # its stations, repeated
    g = api.Context(cfg, coefs, base)
    o = oracle_built.Oracle(cfg, coefs, base)
    st = perturbed_state(cfg, base, np.random.default_rng(nx))
    g.put_state(st)
    o.put_state(st)
    f = np.ascontiguousarray(st["wy"])
    for op, (A, B) in zip(("derparx", "derparxx"), derivative_matrices(nx, cfg.dx)):
        want = getattr(o, op)(f)
        amp = np.max(np.abs(np.linalg.inv(A)) @ np.abs(B).sum(1)) * np.max(np.abs(f)) / np.max(np.abs(want))
        assert rel(getattr(g, op)(f), want) < 2 * 16 * EPS * amp
    g.filter_trid()
    o.filter_trid()
    a, b = g.get_state(), o.get_state()
    for n in ("wx", "wy", "wz"):
        assert rel(a[n], b[n]) < 1e-12
