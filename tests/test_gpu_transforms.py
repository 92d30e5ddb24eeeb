"""The FP64 spanwise transforms and what is built on them, for every number of
physical points, against the oracle: one thread a grid line up to 64 points and
two at 128, all modes and fewer, grid lines that do not fill the last block."""
import math

import numpy as np
import pytest

from tests.helpers import perturbed_state, rel
from trans_bl_gb300 import api, configs

pytestmark = pytest.mark.gpu


def pair(oracle_built, modes, phys, my_form=0, ibm=0):
    cfg = configs.small(nx=17, ny=17, msh=2, kfour=modes, kphys=phys, my_form=my_form)
    cfg.ibm = ibm
    dstar = 1.7208 / math.sqrt(cfg.Re)
    cfg.C_s, cfg.A_plus, cfg.les_damping, cfg.irf = 0.1, 26.0, 3, -500.0
    cfg.ibm_xc = cfg.x0 + 0.25 * (cfg.nx - 1) * cfg.dx
    cfg.ibm_zc, cfg.ibm_h, cfg.ibm_R = math.pi / cfg.beta, 3.0 * dstar, 8.0 * dstar
    base = api.baseflow_fs(cfg, 0.0)
    coefs = api.generate_coefs(cfg.stf, cfg.msh)
    g, o = api.Context(cfg, coefs, base), oracle_built.Oracle(cfg, coefs, base)
    st = perturbed_state(cfg, base, np.random.default_rng(phys + modes))
    g.put_state(st)
    o.put_state(st)
    return g, o, st


@pytest.mark.parametrize("modes,phys", [(1, 2), (2, 4), (3, 8), (8, 16), (11, 32), (16, 32), (32, 64), (33, 128), (64, 128)])
def test_transforms(oracle_built, modes, phys):
    """A value passes 7 stages at most, a few roundings each; products twice that."""
    g, o, _ = pair(oracle_built, modes, phys)
    rng = np.random.default_rng(phys)
    c = rng.normal(size=g.shape) + 1j * rng.normal(size=g.shape)
    p = rng.normal(size=(phys,) + g.shape[1:])
    assert rel(g.f_to_p(c), o.f_to_p(c)) < 1e-12
    assert rel(g.p_to_f(p), o.p_to_f(p)) < 1e-12
    for a, b in zip(g.nlterms(), o.nlterms()):
        assert rel(a, b) < 1e-12


@pytest.mark.parametrize("modes,phys", [(5, 16), (32, 64), (33, 128), (64, 128)])
def test_les_and_roughness_force(oracle_built, modes, phys):
    """To the tolerance of the tests of both terms at 8 points; a line outside the
    roughness has no force, and one with a NaN has it everywhere."""
    g, o, st = pair(oracle_built, modes, phys, my_form=4, ibm=1)
    for a, b in zip(g.les_terms(), o.les_terms()):
        assert rel(a, b) < 1e-11
    for a, b in zip(g.cvirt(), o.cvirt()):
        assert rel(a, b) < 1e-11
        outside = np.all(b == 0, axis=0)
        assert outside.any() and np.max(np.abs(a[:, outside])) < 1e-13   # components below 1e-14 are dropped
    st["ux"][modes - 1, 15, 14] = np.nan   # far from the roughness
    g.put_state(st)
    o.put_state(st)
    for a, b in zip(g.cvirt(), o.cvirt()):
        assert np.array_equal(np.isnan(a.real), np.isnan(b.real))
        ok = np.isfinite(b)
        assert rel(a[ok], b[ok]) < 1e-11
