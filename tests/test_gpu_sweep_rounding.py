"""Rounding of the plain form's line solves: what three sweeps leave of a
solved problem.

From a field whose source is L u to the last digit the pre-sweeps of the first
V-cycle can only add rounding, and the defect after them, which a solve with a
tolerance that any defect meets reports, is the size of it.  The oracle runs the
same sweeps line by line in the reference's order.
"""
import numpy as np
import pytest

from tests.test_gpu_defect_rounding import LD, invert_source, operator
from trans_bl_gb300 import api, configs

pytestmark = pytest.mark.gpu


# modes: few take four warps a line (one row a lane on 129 rows), many take two
@pytest.mark.parametrize("nx,ny,modes,draws", [(33, 129, 8, 4), (65, 129, 8, 4), (33, 129, 32, 1)])
def test_sweeps_round_as_sequential_ones(oracle_built, nx, ny, modes, draws):
    """Root mean square over modes and draws (28 or 31) of the largest defect.
    Each maximum scatters by about an eighth, so two such means of equal
    errors differ by 3 % and rarely by 10."""
    nl = 12.0 * (nx - 1) / 1024
    cfg = configs.blasius_ts_config(nx, ny, modes, 2 * modes, 3, n_lambda=nl, strip=(0.3 * nl, 0.4 * nl))
    coefs = api.generate_coefs(cfg.stf, cfg.msh)
    base = [np.zeros((ny, nx))] * 3
    g, o = api.Context(cfg, coefs, base), oracle_built.Oracle(cfg, coefs, base)
    y = np.arange(ny) / (ny - 1.0)
    shape = np.where(y < 0.9, (y * (1 - y / 0.9)) ** 2, 0.0)[:, None]   # zero at the wall and near the top
    rng = np.random.default_rng(nx + modes)
    got, want = [], []
    for _ in range(draws):
        u = configs.smooth_random((modes, ny, nx), rng, 1.0) * (1.0 + np.arange(modes))[:, None, None] * shape
        st = {n: np.zeros((modes, ny, nx), complex) for n in configs.NAMES}
        st["uy"] = u
        d = np.zeros((modes, ny, nx), complex)
        for k in range(1, modes):
            d[k] = -invert_source(cfg, coefs, operator(cfg, coefs, k, u[k], LD)).astype(complex)
        g.put_state(st)
        o.put_state(st)
        g.poi_uy(d, 1e300)
        o.poi_uy(d, 1e300)
        got += list(g.poisson_stats()["residual"][1:])
        want += list(o.poisson_stats()[1][1:])
    rms = [float(np.sqrt(np.mean(np.square(v)))) for v in (got, want)]
    assert rms[0] <= 1.15 * rms[1], rms
