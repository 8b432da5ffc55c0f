"""The EGLIB point kernel inside, at the ends of and outside the tabulated
temperature range (128 K <= T < 4096 K), against the oracle.

Bound: of the quantities a flux takes from EGLIB the thermal diffusion ratios
carry the largest error, the solution of an ill-conditioned 9 x 9 system: up to
2.6e-12 of the largest ratio for the FP64 evaluation on either side (4000
random states against 80-bit arithmetic); the flux differences of two such
evaluations, over stencils whose weights sum to 3 in magnitude, stay below
3 x 2 x 2.6e-12 = 1.6e-11 of a component's largest value."""
import numpy as np
import pytest

import oracle  # noqa: F401
import workloads as W
from phd_gb300.izem import IzemGPU
from phd_gb300.thd import eglib_link, load_species

pytestmark = pytest.mark.gpu


# the layer's 1036 .. 1164 K scaled across the lower end, inside, across the
# middle temperature of the fits, across the upper end, and beyond
@pytest.mark.parametrize("scale", [0.05, 0.117, 0.3, 0.9, 3.74, 5.0])
def test_visc_flux_over_the_table(scale):
    cfg, thd, adi, dxi, st, info, orc = W.case("mix", 16, eglib=True)
    st["T"] *= scale
    fl = np.zeros((cfg.nx, cfg.ny, cfg.nz, 14), order="F")
    orc.visc_flux(st, fl)
    g = IzemGPU(cfg, thd, adi)
    g.set_grid(*dxi)
    g.set_eglib(eglib_link(load_species("h2air9")))
    g.upload(**st)
    g.zero_flux()
    g.viscflux_xyz()
    got = g.flux()
    g.close()
    err = W.normwise(got, fl)
    assert np.all(err <= 1.6e-11), err
