"""Passes whose warps march along a line of cells: 30 or 32 radii across a warp, a run
of rows along it.  Grids on either side of those widths and run lengths against the
oracle, and run lengths against one another bit for bit.  Needs a B200."""
import numpy as np
import pytest

from oracle.oracle import Oracle, Oracle3
from penguin_b200 import initial as I
from penguin_b200 import params as P
from penguin_b200.disk import Disk
from penguin_b200.disk3 import Disk3
from penguin_b200.ensemble import Ensemble

pytestmark = pytest.mark.gpu

T0 = 5.0 * 2.0 * np.pi

# radii (always even): one warp not full, exactly full at 30 (radial sweep, kicks) and at 32
# (azimuthal passes), two radii into the next warp, two and three warps; azimuths: a last
# run of one row
SIZES = [(28, 90), (30, 91), (32, 96), (34, 97), (60, 127), (62, 128), (64, 129), (66, 190), (96, 191)]


def l1(a, b):
    return np.abs(a - b).sum() / np.abs(b).sum()


def momentum(a, b, keys):
    return (sum(np.abs(a["r"] * a[k] - b["r"] * b[k]).sum() for k in keys)
            / sum(np.abs(b["r"] * b[k]).sum() for k in keys))


@pytest.mark.parametrize("size", SIZES, ids=lambda s: f"{s[0]}x{s[1]}")
def test_disk_matches_oracle(size):
    """Viscosity and orbital advection, no planet and no damping: both sides agree to
    rounding, 10 steps of some 1e3 operations a cell at 1.1e-16, whose errors add as a
    random walk (100 * 1.1e-16) with the local slopes' factor of at most ten."""
    p = P.reference_disk(*size).replace(planet_mass=0.0, kill_flag=0)
    st = I.disk_state(p, seed=size[0])
    o = Oracle(p, st, T0)
    o.run(10)
    ref = o.interior()
    d = Disk(p)
    d.set_state(T0, st)
    d.run(10)
    d.check()
    g = d.get_state()
    d.close()
    errs = {k: l1(g[k], ref[k]) for k in ("r", "p")}
    errs["momentum"] = momentum(g, ref, "uv")
    assert all(e < 1e-13 for e in errs.values()), errs


@pytest.mark.parametrize("size", [(30, 91), (62, 128)], ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("other", ["averages", "dust"])
def test_kick2_instances_agree_bitwise(size, other):
    """A disk that averages or carries dust takes the other instance of the second half-kick, with
    planet, stress and damping: the gas keeps its bits (the dust, slower than the gas's signals
    here, does not bind the time step)."""
    p = P.reference_disk(*size)
    st = I.disk_state(p, seed=7)
    out = []
    for plain in (True, False):
        d = Disk(p if plain or other != "dust" else p.replace(dust_flag=1, Stokes=0.05))
        d.set_state(T0, st)
        if not plain and other == "averages":
            d.set_average(1.0)
        d.run(20)
        d.check()
        out.append((d.get_state(), d.clock()))
        d.close()
    assert out[0][1] == out[1][1]
    for k in ("r", "p", "u", "v"):
        assert np.array_equal(out[0][0][k], out[1][0][k]), k


@pytest.mark.parametrize("size", [(34, 97), (62, 300)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_run_lengths_agree_bitwise(size):
    """The ten run lengths and one CTA per SM (several runs a warp) of the FP64 passes, and
    the two lists of runs of the FP32 passes."""
    p = P.reference_disk(*size)
    st = I.disk_state(p, seed=5)
    out = []
    for v in range(-1, 10):
        d = Disk(p)
        d.set_state(T0, st)
        if v >= 0:
            d.set_tuning(dict(zip(Disk.TUNING, (v, v, v, 1, 1, 1, 1, 1))))
        d.run(6)
        d.check()
        out.append(d.get_state())
        d.close()
    for v, g in enumerate(out[1:]):
        for k in ("r", "p", "u", "v"):
            assert np.array_equal(g[k], out[0][k]), (v, k)


# the FP32 form takes 64 cells per axis at least
@pytest.mark.parametrize("size", [(64, 96), (66, 129), (90, 127), (92, 131), (96, 200)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("dust", [0, 1], ids=["gas", "dust"])
def test_fp32_tracks_fp64(size, dust):
    """Gas against the FP64 oracle, dust against the FP64 path: FP32 residuals against the
    initial disk carry the density to 2e-6 and the velocities to 1e-4 of their deviation,
    the bounds of the 64x192 disk."""
    p = (P.dust_disk(*size, stokes=0.05) if dust else P.reference_disk(*size))
    st = I.disk_state(p, seed=size[1])
    d = Disk(p)
    d.set_state(T0, st)
    base = d.get_dust() if dust else None
    d.step_host(20)
    e = Ensemble([p])
    e.set_state(0, T0, st)
    e.run(20)
    e.sync()
    e.check()
    pairs = [(e.get_state(0), d.get_state(), st)]
    if dust:
        pairs.append((e.get_dust(0), d.get_dust(), base))
    else:
        o = Oracle(p, st, T0)
        o.run(20)
        pairs.append((pairs[0][0], o.interior(), st))
    e.close()
    d.close()
    for got, ref, start in pairs:
        assert l1(got["r"], ref["r"]) < 2e-6
        for k in ("u", "v"):
            assert np.abs(got[k] - ref[k]).sum() < 1e-4 * np.abs(ref[k] - start[k]).sum(), k


# the last: the radial sweep's other instance (create3, pg_3d.cu)
@pytest.mark.parametrize("size", [(28, 9, 7), (30, 8, 12), (32, 13, 9), (34, 7, 8), (62, 6, 10), (96, 96, 96)],
                         ids=lambda s: "x".join(map(str, s)))
def test_box_matches_oracle(size):
    """Uniform cartesian cells leave only rounding: the 40 passes of 8 steps round a cell to
    a few ulp each, a random walk of some 20 ulp, which the flow carries on as it does the
    one-ulp noise that a second oracle run starts with.  Within 64 of its response."""
    p = P.cartesian_box(*size)
    st = I.box_state(p, seed=size[0])
    d = Disk3(p)
    d.set_state(0.0, st)
    d.run(8)
    d.check()
    g = d.get_state()
    d.close()
    rng = np.random.default_rng(size[0])
    runs = []
    for noise in (0.0, 2.0 ** -52):
        o = Oracle3(p, {k: v * (1.0 + noise * rng.integers(-1, 2, v.shape)) for k, v in st.items()}, 0.0)
        o.run(8)
        runs.append(o.interior())
        o.close()
    ref, ulp = runs
    for k in ("r", "p"):
        assert l1(g[k], ref[k]) < 64 * l1(ulp[k], ref[k]), k
    assert momentum(g, ref, "uvw") < 64 * momentum(ulp, ref, "uvw")
    print([l1(g[k], ref[k]) / l1(ulp[k], ref[k]) for k in "rp"], momentum(g, ref, "uvw") / momentum(ulp, ref, "uvw"))
