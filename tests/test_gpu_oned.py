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


def test_drop_in_tube_carries_both_transverse_velocities():
    """Cartesian v and w are transported by the same expressions and enter the energy through
    v^2 + w^2 alone, so a tube with v = 3 s, w = 4 s that takes one launch per pass moves like
    one with v = 5 s, w = 0 in the tube's own kernel.  40 steps at an ulp each, without growth
    at CFL 0.5 (1e-13 of a field's size)."""
    from penguin_b200.grid import ReferenceLoop

    p = P.sod_tube(94)
    rng = np.random.default_rng(7)
    s = 0.1 * rng.uniform(-1, 1, (1, 94))
    st = I.sod_state(p)
    d = Disk(p)
    d.set_state(0.0, dict(st, v=5.0 * s))
    d.step_host(40)
    ref = d.get_state()
    d.close()
    loop = ReferenceLoop(p, 0.0, dict(st, v=3.0 * s))
    cells = loop._keep["C"].view(p.yarr, p.xarr, 5)
    cells[0, 3:-3, 4] = loop.torch.from_numpy(4.0 * s[0]).cuda()
    loop.torch.cuda.synchronize()
    loop.step(40)
    g = loop.interior()
    loop.close()
    want = dict(ref, v=0.6 * ref["v"], w=0.8 * ref["v"])
    for k in "rpuvw":
        assert np.abs(g[k] - want[k]).max() < 1e-13 * np.abs(want[k]).max(), k
