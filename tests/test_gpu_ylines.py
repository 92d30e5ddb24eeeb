"""y-lines of the shortest length and around multiples of their eight-row window
against the oracle."""
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


@pytest.mark.parametrize("ny", [17, 19, 25, 27, 33, 35, 129])
def test_y_lines(oracle_built, ny):
    """dery, deryfv and deryy.  The bound: up to 7 products, their sums and the
    sweeps round about 16 times a row on either side, terms as large as the
    operator's absolute row sum (its dense matrix, from the oracle) allows, with a
    factor 2 for what cancels between its factors."""
    g, o, st = pair(oracle_built, 17, ny, 2)
    f = np.ascontiguousarray(st["ux"])
    unit = np.zeros((ny,) + f.shape, dtype=complex)
    for j in range(ny):
        unit[j, :, j] = 1.0
    for op in ("dery", "deryfv", "deryy"):
        want = getattr(o, op)(f)
        dense = np.array([getattr(o, op)(u)[0, :, 0].real for u in unit]).T
        amp = np.max(np.abs(dense).sum(1)) * np.max(np.abs(f)) / np.max(np.abs(want))
        assert rel(getattr(g, op)(f), want) < 64 * np.finfo(np.float64).eps * amp
