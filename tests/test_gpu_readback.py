"""Reading a state back: small reads, reads cut into chunks for several threads (from 8 MB on,
with a last chunk of any size) and reads into page-locked arrays.  Needs a B200."""
import ctypes

import numpy as np
import pytest
import torch

from penguin_b200 import initial as I
from penguin_b200 import params as P
from penguin_b200._lib import check, lib
from penguin_b200.disk import Disk
from penguin_b200.disk3 import Disk3
from penguin_b200.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def _ptr(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


# 2^18 cells are the 8 MB of four planes; 2^15 doubles a chunk
@pytest.mark.parametrize("size", [(510, 514), (512, 512), (514, 513), (1030, 777)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_get_state_returns_what_was_set(size):
    p = P.reference_disk(*size)
    st = I.disk_state(p, seed=3)
    d = Disk(p)
    d.set_state(0.0, st)
    for _ in range(2):  # the second read finds the slots made by the first
        g = d.get_state()
        for k in ("r", "u", "v"):
            assert np.array_equal(g[k], st[k]), k
    locked = [torch.empty(p.yres, p.xres, dtype=torch.float64).pin_memory().numpy() for _ in range(4)]
    check(lib().pg_disk_get_state(d._h, *(_ptr(a) for a in locked), None))
    for a, k in zip(locked, ("r", "p", "u", "v")):
        assert np.array_equal(a, g[k]), k
    d.close()


def test_get_state_of_a_disk_on_the_per_thread_stream():
    """Every host thread has a per-thread stream of its own: a large read on that stream is not
    split over threads, and follows the steps queued before it."""
    p = P.reference_disk(512, 1024)
    st = I.disk_state(p, seed=4)
    out = []
    for stream in (None, 2):  # 2: cudaStreamPerThread
        d = Disk(p, stream=stream)
        d.set_state(0.0, st)
        d.get_state()
        d.run(60)
        out.append(d.get_state())
        d.close()
    for k in ("r", "p", "u", "v"):
        assert np.array_equal(out[0][k], out[1][k]), k


def test_get_state_into_one_array_leaves_the_last_plane():
    """A caller who wants one field may hand one array for the others: the planes are written in
    their order."""
    p = P.reference_disk(512, 1024)
    st = I.disk_state(p, seed=4)
    d = Disk(p)
    d.set_state(0.0, st)
    d.run(3)
    g = d.get_state()
    v, rest = np.zeros_like(g["v"]), np.zeros_like(g["r"])
    check(lib().pg_disk_get_state(d._h, _ptr(rest), _ptr(rest), _ptr(rest), _ptr(v), None))
    d.close()
    assert np.array_equal(rest, g["u"]) and np.array_equal(v, g["v"])


# three planes of 8 MB and more
@pytest.mark.parametrize("size", [(592, 591), (1030, 777)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_dust_and_ensemble_reads_return_what_was_set(size):
    """FP64 dust as set; FP32 members to the residuals' rounding, 2^-24 of the deviation from the
    initial disk (below 2 in all fields here)."""
    p = P.dust_disk(*size)
    st = I.disk_state(p, seed=3)
    d = Disk(p)
    d.set_state(0.0, st)
    dust = d.get_dust()
    rng = np.random.default_rng(1)
    dust = {k: v * (1.0 + 1e-3 * rng.uniform(-1, 1, v.shape)) for k, v in dust.items()}
    d.set_dust(dust)
    g = d.get_dust()
    d.close()
    for k in ("r", "u", "v"):
        assert np.array_equal(g[k], dust[k]), k
    e = Ensemble([p, P.planet_disk(64, 96)])
    e.set_state(0, 0.0, st)
    e.set_dust(0, dust)
    for _ in range(2):
        g, q = e.get_state(0), e.get_dust(0)
        for k in ("r", "u", "v"):
            assert np.abs(g[k] - st[k]).max() < 2.0 * 2.0 ** -24, k
            assert np.abs(q[k] - dust[k]).max() < 2.0 * 2.0 ** -24, k
    e.close()


def test_get_state_3d_returns_what_was_set():
    p = P.cartesian_box(66, 61, 63)
    st = I.box_state(p, seed=3)
    d = Disk3(p)
    d.set_state(0.0, st)
    g = d.get_state()
    for k in "rpuvw":
        assert np.array_equal(g[k], st[k]), k
    d.close()
