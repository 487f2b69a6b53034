"""The 1D tube's device-resident loop (one launch for many steps, a cluster of
CTAs) against the same steps as one launch per pass."""
import numpy as np
import pytest

from penguin_b200 import params as P

pytestmark = pytest.mark.gpu

# sizes: the smallest, one warp's 30 outputs, one CTA's four warps, where the cluster
# grows and where its CTAs get more warps, ragged last CTAs, the largest and the first beyond
SIZES = (6, 30, 32, 90, 118, 122, 238, 482, 1024, 1922, 4098, 7680, 7682)


def state(n, seed, transverse):
    rng = np.random.default_rng(seed)
    x = np.arange(n) / n
    left = x < 0.4
    s = {"r": np.where(left, 1.0, 0.125) * (1 + 0.05 * rng.uniform(-1, 1, n)),
         "p": np.where(left, 1.0, 0.1) * (1 + 0.05 * rng.uniform(-1, 1, n)), "u": 0.2 * rng.uniform(-1, 1, n),
         "v": 0.3 * rng.uniform(-1, 1, n) if transverse else np.zeros(n)}
    return {k: v[None].copy() for k, v in s.items()}


def both(p, st, steps):
    """The state, clock and planet after `steps` of the one-launch loop, and of the same
    steps as one launch per pass (Disk.profile); then the states three steps on."""
    from penguin_b200.disk import Disk

    out = []
    for passes in (False, True):
        d = Disk(p)
        d.set_state(0.0, st)
        if passes:
            d.profile(steps)
        else:
            d.run(steps)
        d.check()
        out.append((d.get_state(), d.clock(), d.planet()))
        d.run(3)
        out[-1] += (d.get_state(),)
        d.close()
    return out


@pytest.mark.parametrize("n", SIZES)
def test_tube_loop_matches_the_passes(n):
    """Same cells, same arithmetic: the only freedom is how the compiler contracts
    sums of products in the two kernels, an ulp a step; a tube at CFL 0.5 carries it
    on without growth, so 40 steps stay within 1e-13 of the field's size."""
    p = P.sod_tube(n)
    a, b = both(p, state(n, n, False), 40)
    for k in ("r", "p", "u"):
        assert np.abs(a[0][k] - b[0][k]).max() <= 1e-13 * np.abs(b[0][k]).max(), k
        assert np.abs(a[3][k] - b[3][k]).max() <= 2e-13 * np.abs(b[3][k]).max(), k
    assert a[1][2] == b[1][2] == 40
    assert abs(a[1][0] - b[1][0]) <= 1e-13 * b[1][0]
    assert abs(a[2]["y"] - b[2]["y"]) < 1e-13 and a[2]["m"] == b[2]["m"]


@pytest.mark.parametrize("lft,rgh", [(1, 2), (2, 1), (2, 2), (0, 0)])
@pytest.mark.parametrize("eos,ie", [(2, 0), (2, 1), (0, 1)])
def test_tube_loop_boundaries_and_equations_of_state(lft, rgh, eos, ie):
    p = P.sod_tube(94).replace(bound_lft=lft, bound_rgh=rgh, EOS_flag=eos, internal_e_flag=ie,
                               gam=1.4 if eos else 1.0, sc_h=0.8)
    a, b = both(p, state(94, 3, True), 50)
    for k in ("r", "p", "u", "v"):
        assert np.abs(a[0][k] - b[0][k]).max() <= 1e-13 * np.abs(b[0][k]).max(), k


def test_tube_loop_stops_at_its_end_time():
    """The step that crosses end_time is clipped, later launches do nothing, and the
    next run starts from the step the clip replaced."""
    from penguin_b200.disk import Disk

    p = P.sod_tube(1024)
    st = state(1024, 1, False)
    d = Disk(p)
    d.set_state(0.0, st)
    d.run(100000, end_time=0.2)
    t, dt, n = d.clock()
    h = Disk(p)
    h.set_state(0.0, st)
    nh = h.step_host(100000, 0.2)
    assert t == pytest.approx(0.2, abs=1e-15) and n == nh
    a, b = d.get_state(), h.get_state()
    for k in ("r", "p", "u"):
        assert np.array_equal(a[k], b[k]), k
    d.run(100000, end_time=0.3)
    t, dt, m = d.clock()
    assert t == pytest.approx(0.3, abs=1e-15) and m > n
    d.check()
    d.close()
    h.close()


@pytest.mark.parametrize("finite", [False, True])
def test_tube_loop_longer_than_a_launch(finite):
    """A launch takes up to 2048 steps and hands state, clock and signal rate to the next: 4100
    steps (without an end time), or as many as an end time after some 2500 takes, against the same
    steps launched one by one with the host's clock, bit for bit."""
    from penguin_b200.disk import Disk

    p = P.sod_tube(90)
    st = state(90, 4, False)
    end = 1.0e30
    if finite:
        h = Disk(p)
        h.set_state(0.0, st)
        h.step_host(2500)
        end = h.t + 0.5 * h.dt
        h.close()
    d, h = Disk(p), Disk(p)
    for x in (d, h):
        x.set_state(0.0, st)
    steps = 100000 if finite else 4100
    d.run(steps, end_time=end)
    nh = h.step_host(steps, end)
    t, dt, n = d.clock()
    assert n == nh and n > 2048 and (not finite or n < 4096)
    assert t == h.t and dt == h.dt
    a, b = d.get_state(), h.get_state()
    for k in ("r", "p", "u"):
        assert np.array_equal(a[k], b[k]), k
    d.check()
    d.close()
    h.close()


def test_tubes_made_and_run_by_several_threads():
    """Every tube asks its own device for the largest cluster when it is made: threads that make
    and run tubes at the same time (16 CTAs each) get the states that one thread gets."""
    import threading

    from penguin_b200.disk import Disk

    p = P.sod_tube(1024)
    st = state(1024, 2, False)
    out = [None] * 5

    def work(k):
        d = Disk(p)
        d.set_state(0.0, st)
        d.run(30)
        d.check()
        out[k] = d.get_state()
        d.close()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    work(4)
    for g in out[:4]:
        for k in ("r", "p", "u"):
            assert np.array_equal(g[k], out[4][k]), k


@pytest.mark.parametrize("n,transverse", [(94, True), (1024, False)])
def test_averages_leave_the_tube_as_it_is(n, transverse):
    """A tube that averages takes one launch per pass: the same bits and the same clock."""
    from penguin_b200.disk import Disk

    p = P.sod_tube(n)
    st = state(n, n, transverse)
    out = []
    for average in (False, True):
        d = Disk(p)
        d.set_state(0.0, st)
        if average:
            d.set_average(0.1)
        d.run(200)
        d.check()
        out.append((d.get_state(), d.clock()))
        d.close()
    assert out[0][1] == out[1][1]
    for k in ("r", "p", "u", "v"):
        assert np.array_equal(out[0][0][k], out[1][0][k]), k


@pytest.mark.parametrize("n,average,launches", [(1024, 0.0, 1), (7680, 0.0, 1), (7682, 0.0, 4), (1024, 0.1, 4)])
def test_launches_of_a_step(n, average, launches):
    from penguin_b200.disk import Disk

    d = Disk(P.sod_tube(n))
    d.set_average(average)
    assert d.kernels_per_step == launches
    d.close()
