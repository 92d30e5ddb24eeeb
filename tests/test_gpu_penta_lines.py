"""Pentadiagonal x-lines at the edges of their chunks and blocks against the
oracle: line lengths around multiples of 32 (a pair of warps in 32 chunks), tables
too long for shared memory, and runs of lines that cross modes."""
import numpy as np
import pytest

from tests.helpers import perturbed_state, rel
from trans_bl_gb300 import api, configs

pytestmark = pytest.mark.gpu


def pair(oracle_built, nx, ny, modes):
    kw = dict(kfour=modes, kphys=2 * modes if modes != 3 else 8)
    cfg = configs.small(nx=nx, ny=ny, msh=2, **kw)
    base = [np.ascontiguousarray(np.resize(b.T, (nx, ny)).T) for b in api.baseflow_fs(configs.small(nx=17, ny=ny, msh=2, **kw), 0.0)]
    coefs = api.generate_coefs(cfg.stf, cfg.msh)
    g, o = api.Context(cfg, coefs, base), oracle_built.Oracle(cfg, coefs, base)
    st = perturbed_state(cfg, base, np.random.default_rng(nx * ny))
    g.put_state(st)
    o.put_state(st)
    return g, o, st


@pytest.mark.parametrize("nx,ny,modes", [(17, 17, 2), (33, 17, 3), (63, 17, 2), (65, 25, 4), (129, 33, 16), (1025, 17, 3), (2049, 17, 2)])
def test_penta_lines(oracle_built, nx, ny, modes):
    """poi_ux and poi_uz to the tolerance the parity tests give them."""
    g, o, _ = pair(oracle_built, nx, ny, modes)
    g.poi_ux()
    b = o.poi_ux()
    assert rel(g.get_state()["ux"], o.get_state()["ux"]) < 1e-11
    g.poi_uz(b)
    o.poi_uz(b)
    assert rel(g.get_state()["uz"], o.get_state()["uz"]) < 1e-11
