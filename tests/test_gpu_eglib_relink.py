"""One context given one set of EGLIB linking data, then another, then the first
again: each flux is the oracle's for the data set last, from the first call
after the change on.  Bound: that of test_gpu_eglib_table.py."""
import numpy as np
import pytest

import workloads as W
from phd_gb300.izem import IzemGPU
from phd_gb300.thd import eglib_link, load_species

pytestmark = pytest.mark.gpu


def _link(shift):
    """The H2/air set, its viscosities and diffusion coefficients scaled by e^shift."""
    link = eglib_link(load_species("h2air9"))
    for k in range(link.ns):
        link.cofe[k][0] += shift
        for l in range(link.ns):
            link.cofd[k][l][0] += shift
    return link


def test_linking_data_set_again():
    cfg, thd, adi, dxi, st, info, orc = W.case("mix", 16, eglib=True)
    shifts = (0.25, 0.0, 0.25)
    want = []
    for s in shifts:
        orc.set_eglib(_link(s))
        fl = np.zeros((cfg.nx, cfg.ny, cfg.nz, 14), order="F")
        orc.visc_flux(st, fl)
        want.append(fl)
    assert np.max(W.normwise(want[0], want[1])) > 0.1   # the data matter
    g = IzemGPU(cfg, thd, adi)
    g.set_grid(*dxi)
    g.upload(**st)
    for s, ref in zip(shifts, want):
        g.set_eglib(_link(s))
        g.zero_flux()
        g.viscflux_xyz()
        err = W.normwise(g.flux(), ref)
        assert np.all(err <= 1.6e-11), (s, err)
    g.close()
