"""Plain-form Poisson solves at the edges of the line groups and of the wavefront.

The lexicographic sweeps keep the reference's iterates whatever the shape of
a launch, so uy after the solve and every mode's number of V-cycles are the
oracle's.  The grids reach: a coarsest level of too few lines for the wavefront
and the smallest one for it; 1, 2 and 4 warps a line, with lines that fill their
lanes (33, 65, 129 points) and that leave some empty; 2, 3, 4 and more rows a lane;
coarsest sweeps that wrap round the cluster's line groups and that do not (nx
of 385 and more on two levels); and modes enough for fewer warps a line.
"""
import numpy as np
import pytest

from trans_bl_gb300 import api, configs
from tests.helpers import perturbed_state, rel

pytestmark = pytest.mark.gpu

GRIDS = [   # nx, ny, msh, modes
    (17, 17, 2, 1), (25, 17, 3, 2), (33, 33, 3, 1), (49, 65, 3, 2), (65, 129, 4, 1), (33, 101, 3, 1), (33, 193, 3, 1),
    (33, 257, 3, 1), (33, 321, 3, 1), (33, 449, 3, 1), (385, 33, 2, 1), (25, 129, 3, 40), (25, 257, 3, 64),
]


@pytest.mark.parametrize("nx,ny,msh,modes", GRIDS)
def test_poi_uy_of_grids(oracle_built, nx, ny, msh, modes):
    """The parity tests' tolerance of one solve.  The defect's rounding floor grows
    with the number of rows (the oracle's own stalls at 9e-10 for 257, 2e-9 for 289),
    so the tall grids stop well above it."""
    phys = 2
    while phys < 2 * modes:
        phys *= 2
    kw = dict(kfour=modes, kphys=phys, max_vcycles=12)
    cfg = configs.small(nx=nx, ny=ny, msh=msh, **kw)
    # the base flow of 17 stations, repeated
    base = [np.ascontiguousarray(np.resize(b.T, (nx, ny)).T) for b in api.baseflow_fs(configs.small(nx=17, ny=ny, msh=2, **kw), 0.0)]
    coefs = api.generate_coefs(cfg.stf, cfg.msh)
    g = api.Context(cfg, coefs, base)
    o = oracle_built.Oracle(cfg, coefs, base)
    st = perturbed_state(cfg, base, np.random.default_rng(nx + ny))
    g.put_state(st)
    o.put_state(st)
    d = o.outuy()
    g.outuy()
    for erro in (1e-3, 1e-9 if ny < 200 else 1e-6):
        g.poi_uy(d, erro)
        o.poi_uy(d, erro)
        assert g.poisson_stats()["vcycles"] == o.poisson_stats()[0]
        assert rel(g.get_state()["uy"], o.get_state()["uy"]) < 1e-9
