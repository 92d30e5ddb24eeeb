"""x-lines in numbers that make the kernels keep their row tables in shared
memory, which they do only where every SM has several lines in turn.

The pentadiagonal solves: runs of lines that cross Fourier modes (the tables
are replaced on the way), pairs of warps with a second line, and lines so long
that the tables stay in global memory all the same.  The derivatives and the
filter: pairs with several lines, at the edges of the chunks.
"""
import numpy as np
import pytest

from tests.helpers import perturbed_state, rel
from tests.test_gpu_xlines import EPS, derivative_matrices
from trans_bl_gb300 import api, configs

pytestmark = pytest.mark.gpu


def pair(oracle_built, nx, ny, modes, **kw):
    kw = dict(kfour=modes, kphys=2 * modes, **kw)
    cfg = configs.small(nx=nx, ny=ny, msh=2, **kw)
    # the base flow of 17 stations, repeated
    base = [np.ascontiguousarray(np.resize(b.T, (nx, ny)).T) for b in api.baseflow_fs(configs.small(nx=17, ny=ny, msh=2, **kw), 0.0)]
    coefs = api.generate_coefs(cfg.stf, cfg.msh)
    g, o = api.Context(cfg, coefs, base), oracle_built.Oracle(cfg, coefs, base)
    st = perturbed_state(cfg, base, np.random.default_rng(nx * ny))
    g.put_state(st)
    o.put_state(st)
    return cfg, g, o, st


# 8 lines an SM are 1216 on 152 SMs; 50 rows a mode are no multiple of a block's 8 lines
@pytest.mark.parametrize("nx,ny,modes", [(17, 51, 32), (33, 51, 32), (63, 51, 32), (65, 51, 32), (1025, 51, 32), (2177, 41, 32)])
def test_penta_runs_of_lines(oracle_built, nx, ny, modes):
    """poi_ux and poi_uz to the tolerance the parity tests give them."""
    _, g, o, _ = pair(oracle_built, nx, ny, modes)
    g.poi_ux()
    b = o.poi_ux()
    assert rel(g.get_state()["ux"], o.get_state()["ux"]) < 1e-11
    g.poi_uz(b)
    o.poi_uz(b)
    assert rel(g.get_state()["uz"], o.get_state()["uz"]) < 1e-11


# 4864 lines are one a pair for the short lines, 1216 for those of 1025 points
@pytest.mark.parametrize("nx,ny,modes", [(17, 153, 64), (33, 153, 64), (97, 153, 64), (1025, 51, 32)])
def test_line_operators_in_turn(oracle_built, nx, ny, modes):
    """derparx, derparxx and the context's filter, to the bounds the line tests
    derive: 16 roundings on either side of terms as large as the sum of
    |weight| allows, through the inverse of the LHS; the filter's weights are
    below 1."""
    cfg, g, o, st = pair(oracle_built, nx, ny, modes)
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
