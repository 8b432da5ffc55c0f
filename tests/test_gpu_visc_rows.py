"""Viscous fluxes of grids whose gradients and divergences are shared by all,
by some and by one block row.

A flow that repeats itself in z, its ghost planes the images of its interior
ones, has the fluxes of one period in every period, and a point's flux comes
from the same operations whichever block row takes a component of it: the
same bits, no tolerance."""
import numpy as np
import pytest

import workloads as W
from phd_gb300.izem import IzemGPU

pytestmark = pytest.mark.gpu


def _visc_flux(cfg, thd, adi, dxi, st):
    g = IzemGPU(cfg, thd, adi)
    g.set_grid(*dxi)
    g.upload(**st)
    g.zero_flux()
    g.viscflux_xyz()
    got = g.flux()
    g.close()
    return got


# one and eight periods of 4000 points, one and four of 32 000
@pytest.mark.parametrize("n,periods", [(20, 8), (40, 4)])
def test_visc_flux_rows(n, periods):
    cfg, thd, adi, dxi, st, info, orc = W.case("mix", n)
    W.perturb(st, 0.01, seed=5)
    orc.update_primitives(st)
    ng, nz = 3, cfg.nz

    def repeat(a, m):
        inner = np.concatenate([a[:, :, ng:-ng]] * m, axis=2)
        return np.asfortranarray(np.concatenate([inner[:, :, -ng:], inner, inner[:, :, :ng]], axis=2))

    def spacing(m):   # one value: the metric's own last bits differ from plane to plane
        return dxi[0], dxi[1], np.full(m * nz + 2 * ng, dxi[2][ng])

    one = _visc_flux(cfg, thd, adi, spacing(1), {k: repeat(a, 1) for k, a in st.items()})
    cfg.nz = periods * nz
    many = _visc_flux(cfg, thd, adi, spacing(periods), {k: repeat(a, periods) for k, a in st.items()})
    assert np.abs(one[..., 5:]).max() > 0
    for m in range(periods):
        np.testing.assert_array_equal(many[:, :, m * nz:(m + 1) * nz], one)
