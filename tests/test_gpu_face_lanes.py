"""Faces with the nonlinear weights, few and many to a warp, against the
oracle: a warp with up to twelve of them reconstructs each with a lane a
field, one with more a face a thread.

Bound: the states are those on which the tests of all-sensed sweeps hold the
fluxes to 1e-12 of a component's largest value (WENO5 on the smooth layer and
vortex; WENO7 on 20 % noise, where its smoothness indicators do not cancel);
flagging fewer points leaves every sensed face one of theirs."""
import numpy as np
import pytest

import workloads as W
from phd_gb300.izem import IzemGPU

pytestmark = pytest.mark.gpu


# part of the points flagged: a face a few warps, a few a warp, around the
# line, most of them
@pytest.mark.parametrize("part", [0.002, 0.02, 0.07, 0.5])
@pytest.mark.parametrize("name,ng", [("tgv", 3), ("mix", 3), ("mix", 4)])
def test_euler_flux_partly_sensed(name, ng, part):
    cfg, thd, adi, dxi, st, info, orc = W.case(name, 12, ng=ng)
    if ng == 4:
        W.perturb(st, 0.2, seed=9)
        orc.update_primitives(st)
    rng = np.random.Generator(np.random.PCG64(int(1000 * part)))
    i = (slice(ng, -ng),) * 3
    st["shock_sensor"][...] = 0
    st["shock_sensor"][i] = rng.random(st["shock_sensor"][i].shape) < part
    assert st["shock_sensor"].any()
    g = IzemGPU(cfg, thd, adi)
    g.set_grid(*dxi)
    g.upload(**st)
    fl = np.zeros((cfg.nx, cfg.ny, cfg.nz, 5 + cfg.nrv), order="F")
    for d in range(3):
        orc.euler_flux(st, d, fl)
        g.euler_LLF(d)
    got = g.flux()
    g.close()
    err = W.normwise(got, fl)
    assert np.all(err <= 1e-12), err


# grids whose sweeps take two lanes (tgv 18) and one lane (tgv 24, mix 30) to a
# face, where those above take four; 20 % noise on all, so that the finer grids'
# indicators do not cancel either
@pytest.mark.parametrize("part", [0.02, 0.5])
@pytest.mark.parametrize("name,n", [("tgv", 18), ("tgv", 24), ("mix", 30)])
def test_euler_flux_lanes_to_a_face(name, n, part):
    cfg, thd, adi, dxi, st, info, orc = W.case(name, n)
    W.perturb(st, 0.2, seed=9)
    orc.update_primitives(st)
    rng = np.random.Generator(np.random.PCG64(n))
    i = (slice(3, -3),) * 3
    st["shock_sensor"][...] = 0
    st["shock_sensor"][i] = rng.random(st["shock_sensor"][i].shape) < part
    g = IzemGPU(cfg, thd, adi)
    g.set_grid(*dxi)
    g.upload(**st)
    fl = np.zeros((cfg.nx, cfg.ny, cfg.nz, 5 + cfg.nrv), order="F")
    for d in range(3):
        orc.euler_flux(st, d, fl)
        g.euler_LLF(d)
    got = g.flux()
    g.close()
    err = W.normwise(got, fl)
    assert np.all(err <= 1e-12), err
