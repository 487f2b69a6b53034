"""1D grids that take one launch per pass: a polar ring with a planet, and a tube through the
drop-in entry points.  Needs a B200."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from penguin_b200 import initial as I
from penguin_b200 import params as P
from penguin_b200.disk import Disk

pytestmark = pytest.mark.gpu

T0 = 5.0 * 2.0 * np.pi


def l1(a, b):
    return np.abs(a - b).sum() / np.abs(b).sum()


@pytest.mark.parametrize("lft,rgh", [(1, 1), (1, 2), (2, 1)])
@pytest.mark.parametrize("n", [28, 30, 64])
def test_polar_ring_with_a_planet_matches_the_oracle(n, lft, rgh):
    """One row, so the planet's table has one row: no pass has another to read.  The row lies at
    azimuth 0, where the oracle takes it to be.  The two sides solve the slope weights of the
    logarithmic radii with roundings of their own, 1e-9 of a slope; a slope is a tenth of the
    field on 28 radii, a face carries it on by the Courant number 0.3: 3e-10 after 10 steps (the
    planet itself moves the density by 1e-2)."""
    p = P.planet_disk(n, 96).replace(ndim=1, yres=1, ymin=-np.pi, ymax=np.pi, visc_flag=0, OrbAdv_flag=0, kill_flag=0,
                                     bound_lft=lft, bound_rgh=rgh)
    st = I.disk_state(p, seed=n)
    o = Oracle(p, st, T0)
    o.run(10)
    ref = o.interior()
    o.close()
    d = Disk(p)
    d.set_state(T0, st)
    d.run(10)
    d.check()
    g = d.get_state()
    d.close()
    errs = {k: l1(g[k], ref[k]) for k in ("r", "p", "v")}
    # the radial velocity starts at zero: its rounding is that of the speeds it is made of
    errs["u"] = np.abs(g["u"] - ref["u"]).max() / np.abs(ref["v"]).max()
    assert all(e < 3e-10 for e in errs.values()), errs
