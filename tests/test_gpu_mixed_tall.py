"""The mixed form's multigrid on grids of more than 272 rows, whose finest
levels relax a line on a warp (9, 11, 13, 15 or 17 rows a lane) and hand over to
the strips below: 273 and 505 rows, the first beyond 288, 352, 416 and 480, one
and several levels with all rows.  The corrections are those of the same
multigrid with every level relaxed so, from the same states.
"""
import numpy as np
import pytest

from tests.helpers import perturbed_state, rel
from trans_bl_gb300 import api, configs

pytestmark = pytest.mark.gpu

GRIDS = [(97, 273, 1, [5]), (193, 289, 2, [7, 6]), (97, 353, 3, [5, 4, 4]), (129, 417, 2, [4, 4]), (97, 481, 1, [5]),
         (257, 505, 2, [5, 4])]   # nx, ny, modes, corrections to 1e-5


@pytest.mark.parametrize("nx,ny,modes,counts", GRIDS)
def test_poi_uy_of_tall_grids(oracle_built, nx, ny, modes, counts):
    kw = dict(kfour=modes, kphys=max(2, 1 << (2 * modes - 1).bit_length()), max_vcycles=40)
    cfg = configs.small(precision=api.FORM_MIXED, nx=nx, ny=ny, msh=4, **kw)
    # the base flow of 17 stations, repeated
    base = [np.ascontiguousarray(np.resize(b.T, (nx, ny)).T) for b in api.baseflow_fs(configs.small(nx=17, ny=ny, msh=2, **kw), 0.0)]
    coefs = api.generate_coefs(cfg.stf, cfg.msh)
    g, o = api.Context(cfg, coefs, base), oracle_built.Oracle(cfg, coefs, base)
    st = perturbed_state(cfg, base, np.random.default_rng(nx + ny))
    g.put_state(st)
    o.put_state(st)
    d = o.outuy()
    g.outuy()
    erro = 1e-5
    g.poi_uy(d, erro)
    o.poi_uy(d, erro)
    ps = g.poisson_stats()
    assert ps["noconv"] == 0
    assert ps["vcycles"][:modes] == counts
    assert max(ps["residual"][:modes]) < erro
    assert rel(g.get_state()["uy"], o.get_state()["uy"]) < 10 * erro
