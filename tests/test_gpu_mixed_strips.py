"""The mixed form's multigrid on grids at the edges of its strips and chunks.

A kernel of the V-cycle holds 32 elements of each colour plane (plane
elements: nx // 3 + 1) in overlapping strips, 16 row chunks of S rows each,
S picked from a fixed list by the number of rows.  The grids below sit on both
sides of the strip counts (one strip up to 32 elements, then 27 or 26 more per
strip), take the three remainders of nx by 3 (the plane of the last border
line), every S, ragged last chunks, and x-only and full coarsening.  A wrong
halo or remainder leaves the FP64 stopping rule intact but spoils the
contraction, so the corrections are checked too: the counts are those of the
same multigrid run line by line, one kernel per relaxation colour, from the
same states.
"""
import numpy as np
import pytest

from tests.helpers import perturbed_state, rel, small_case

pytestmark = pytest.mark.gpu

# nx, ny, kfour, msh, tolerance of the solve, corrections per mode: the FP64
# defect of a grid with more than 200 rows (first cell below 0.02 delta*)
# carries round-off near 1e-9
GRIDS = [(25, 17, 1, 2, 1e-9, [6]),            # one strip, S = 2, the smallest coarsening
         (93, 33, 2, 3, 1e-9, [9, 7]),         # 32 elements: one full strip
         (97, 65, 3, 3, 1e-9, [8, 7, 6]),      # 33 elements: two strips, S = 5
         (177, 49, 2, 3, 1e-9, [6, 6]),        # 60 elements, S = 4
         (181, 77, 2, 3, 1e-9, [10, 10]),      # 61 elements, ragged rows
         (185, 109, 1, 3, 1e-9, [7]),          # S = 7
         (273, 137, 2, 4, 1e-9, [7, 7]),       # 92 elements: four strips, S = 9
         (129, 201, 2, 4, 1e-8, [5, 6]),       # S = 13
         (97, 265, 1, 4, 1e-7, [7]),           # S = 17
         (97, 297, 1, 4, 1e-7, [7])]           # S = 33


@pytest.mark.parametrize("nx,ny,kfour,msh,erro,counts", GRIDS)
def test_poi_uy_at_strip_edges(oracle_built, nx, ny, kfour, msh, erro, counts):
    from trans_bl_gb300 import api
    cfg, coefs, base = small_case(precision=api.FORM_MIXED, max_vcycles=40, nx=nx, ny=ny, kfour=kfour,
                                  kphys=max(2, 1 << (2 * kfour - 1).bit_length()), msh=msh)
    g = api.Context(cfg, coefs, base)
    o = oracle_built.Oracle(cfg, coefs, base)
    st = perturbed_state(cfg, base, np.random.default_rng(nx + ny))
    g.put_state(st)
    o.put_state(st)
    d = o.outuy()
    g.outuy()
    g.poi_uy(d, erro)
    o.poi_uy(d, erro)
    ps = g.poisson_stats()
    assert ps["noconv"] == 0
    assert ps["vcycles"][:kfour] == counts
    assert max(ps["residual"][:kfour]) < erro
    assert rel(g.get_state()["uy"], o.get_state()["uy"]) < 10 * erro
