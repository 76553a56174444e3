"""The plain form's tile kernels against its ring-array path, bit for bit, at the sizes and states where
they can differ: grids smaller than a tile, multiples of the 8 x 16 tile and one cell either way, bulk
tiles at every border, odd step counts between uploads, moving-frame shifts and smoothing pre-steps
(which take the other path and reset the tile words), dense random states, values outside [0, 1] and
non-finite ones.

The tile kernels take models with symmetric pair constants only.  An isotropic model does not read dab,
so making dab asymmetric sends the same physics through the ring-array path.  Anisotropic models are
compared with the oracle.
"""
import numpy as np
import pytest

import microsim_b200 as mb
from microsim_b200 import configs
from oracle import gp_oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(4, 4), (7, 15), (8, 16), (9, 17), (16, 33), (40, 70), (64, 128), (5, 200)]


def _alloy(kind, mx, my, bc):
    if kind in ("obstacle", "well", "gradient"):
        c = configs.binary_case(mx, my, gap=1.0, supersat=0.5, eps=3.0, dt=0.05, tau=1.3332,
                                function_w=2 if kind == "well" else 1, seed=(0, 0, 0.3 * min(mx, my) + 1), bc=bc)
        if kind == "gradient":
            c.tempgrady = (0.97, 0.08, float(my), 2.0, 0.5)
        return c
    if kind == "three":
        c = configs.Case(mesh_x=mx, mesh_y=my, dx=1.0, dt=0.04, N=3, K=3, epsilon=4.0, tau=1.0, gamma=[1.0, 1.2, 0.8],
                         tau_ab=[1.0, 1.1, 1.3], aniso=0, dab=[0.0] * 3, function_w=1, gamma_abc=[3.0],
                         diffusivity=[(1, 0, 0.0, 0.0), (1, 1, 0.0, 0.0), (1, 2, 1.0, 0.7)],
                         A=[(0, 1.0, 1.0, 0.0), (1, 1.0, 1.0, 0.0), (2, 1.0, 1.0, 0.0)],
                         ceq=[(0, 0, 0.4, 0.1), (0, 2, -0.2, -0.2), (2, 0, -0.2, -0.2), (1, 1, 0.1, 0.4),
                              (1, 2, -0.2, -0.2), (2, 1, -0.2, -0.2), (2, 2, -0.2, -0.2)],
                         cfill=[(0, 0, 0.4, 0.1), (0, 2, -0.2, -0.2), (2, 0, -0.2, -0.2), (1, 1, 0.1, 0.4),
                                (1, 2, -0.2, -0.2), (2, 1, -0.2, -0.2), (2, 2, -0.1, -0.1)],
                         slopes=[(0, 0, 0.45, 0.45), (0, 2, 0.45, 0.45), (2, 0, 0.45, 0.45), (1, 1, 0.45, 0.45),
                                 (1, 2, 0.45, 0.45), (2, 1, 0.45, 0.45)], bc_phi=bc, bc_mu=bc,
                         solver="DILUTE", phases=["a", "b", "l"], components=["X", "Y", "Z"])
    else:
        c = configs.c3(steps=10, mesh=max(mx, 16), nseeds=4, rng_seed=5)
        c.mesh_x, c.mesh_y, c.bc_phi, c.bc_mu, c.aniso, c.fills = mx, my, bc, bc, 0, []
    r = max(1.5, 0.2 * min(mx, my))
    c.fills = [("FILLCYLINDER", [0, mx // 4, my // 4, 0, 0, r]),
               ("FILLCYLINDER", [1, (3 * mx) // 4, (2 * my) // 3, 0, 0, r])]
    return c


def _pair(m):
    other = m.copy()
    d = other.arr("dab")
    d[0, 1], d[1, 0] = 0.25, 0.5  # not read by an isotropic model
    return mb.Context(m, mb.GP_FP64), mb.Context(other, mb.GP_FP64)


def _same(a, b, what):
    pa, ua = a.download()
    pb, ub = b.download()
    assert np.array_equal(pa, pb, equal_nan=True), what
    assert np.array_equal(ua, ub, equal_nan=True), what
    assert np.array_equal(a.download_dphi(), b.download_dphi(), equal_nan=True), what
    return pa, ua


@pytest.mark.parametrize("kind", ["obstacle", "well", "gradient", "three", "four"])
@pytest.mark.parametrize("bc", [(1, 1, 1, 1), (3, 3, 1, 1), (3, 3, 3, 3)])
@pytest.mark.parametrize("size", SIZES)
def test_tiles_equal_the_ring_array_path(size, bc, kind):
    m, phi, mu = mb.load_case(_alloy(kind, *size, bc))
    a, b = _pair(m)
    with a, b:
        for c in (a, b):
            c.upload(phi, mu)
            c.step(1)
        _same(a, b, "first step")
        for n in (8, 3, 17):
            for c in (a, b):
                c.step(n)
            _same(a, b, f"{n} more steps")
        for c in (a, b):  # an upload of the same state between steps
            c.upload(*c.download())
            c.step(5)
        _same(a, b, "after an upload")
        if kind != "gradient":
            for c in (a, b):
                c.shift_y(2)
                c.step(3)
                c.shift_y(1)
                c.step(8)
            _same(a, b, "after shifts")
        for c in (a, b):
            c.smooth(3)
            c.step(9)
        _same(a, b, "after smoothing")


@pytest.mark.parametrize("kind", ["obstacle", "well", "three", "four"])
def test_tiles_equal_the_ring_array_path_on_wild_states(kind):
    m, phi, mu = mb.load_case(_alloy(kind, 37, 51, (3, 3, 1, 1)))
    rng = np.random.default_rng(4)
    dense = rng.random(phi.shape)
    outside = np.where(rng.random(phi.shape) < 0.1, rng.uniform(-0.2, 1.2, phi.shape), phi)
    tiny = np.where(rng.random(phi.shape) < 0.2, 10.0 ** rng.uniform(-300, -1, phi.shape), phi)
    bad = phi.copy()
    bad[0, 20, 30], bad[-1, 5, 5] = np.nan, np.inf
    for name, p in (("dense", dense), ("outside", outside), ("tiny", tiny), ("bad", bad), ("minus zero", phi * -0.0 + phi)):
        a, b = _pair(m)
        with a, b:
            for c in (a, b):
                c.upload(p, mu)
                c.step(2)
            _same(a, b, name)


@pytest.mark.parametrize("spacing", [(1.0, 1.0), (0.5, 2.0), (4.0, 0.25), (0.7, 1.3)])  # the last: no tiles
@pytest.mark.parametrize("size", [(33, 47), (64, 64)])
def test_anisotropic_tiles_equal_the_oracle(size, spacing):
    mx, my = size
    c = configs.binary_case(mx, my, gap=1.0, supersat=0.5, eps=3.0, delta=0.04, theta=17.0, dt=0.05, tau=1.3332,
                            seed=(0, 0, 9.0))
    m, phi, mu = mb.load_case(c)
    m.dx, m.dy = spacing
    m.dt *= min(1.0, min(spacing) ** 2)
    om = O.OracleModel(
        N=m.N, K1=m.K1, mesh_x=mx, mesh_y=my, dx=m.dx, dy=m.dy, dt=m.dt, epsilon=m.epsilon, tau=m.tau, T=m.T, Teq=m.Teq,
        obstacle=m.obstacle, anisotropy=m.anisotropy, binary=1, ternary=0, dilute=0, bc_phi=tuple(m.bc_phi),
        bc_mu=tuple(m.bc_mu), Gamma=m.arr("Gamma")[:2, :2], tau_ab=m.arr("tau_ab")[:2, :2], cmu=m.arr("cmu")[:2, :1, :1],
        A=m.arr("A")[:2, :1, :1], Beq=m.arr("Beff")[:2, :1], dBbdT=np.zeros((2, 1)), B=m.arr("B")[:2, :1],
        C=m.arr("C")[:2], Diff=m.arr("Diff")[:2, :1, :1], dab=m.arr("dab")[:2, :2],
        R=np.pad(m.arr("R")[:2, :2], ((0, 0), (0, 0), (0, 1), (0, 1))),
        Rinv=np.pad(m.arr("Rinv")[:2, :2], ((0, 0), (0, 0), (0, 1), (0, 1))))
    gp, gm = np.zeros((2, mx + 6, my + 6)), np.zeros((1, mx + 6, my + 6))
    gp[:, 3:-3, 3:-3], gm[:, 3:-3, 3:-3] = phi, mu
    O.apply_bc(om, gp, gm)
    O.step(om, gp, gm, 203)
    with mb.Context(m, mb.GP_FP64) as ctx:
        ctx.upload(phi, mu)
        ctx.step(203)
        p, u = ctx.download()
    assert np.array_equal(p, gp[:, 3:-3, 3:-3]) and np.array_equal(u, gm[:, 3:-3, 3:-3])


def _write(c, k):
    """Fields as a caller writes them into the device buffers: another phase's patch across tile borders, a
    gradient beside it, a negative zero in a pure region, mu changed in the bulk."""
    phi, mu = c.device_state()
    N, mx, my = phi.shape[0], int(c.model.mesh_x), int(c.model.mesh_y)
    x0, y0 = (5 * k) % max(1, mx - 6), (11 * k) % max(1, my - 9)
    phi[:, x0:x0 + 6, y0:y0 + 8] = 0.0
    phi[k % N, x0:x0 + 6, y0:y0 + 8] = 1.0
    phi[0, x0 + 2, y0 + 8:y0 + 9], phi[-1, x0 + 2, y0 + 8:y0 + 9] = 0.25, 0.75
    phi[:, mx - 1, my - 1] = 0.0
    phi[-1, mx - 1, my - 1] = 1.0
    phi[0, mx - 1, my - 1] = -0.0
    mu[:, mx // 2, :my] += 0.01
    c.state_changed()


@pytest.mark.parametrize("kind", ["obstacle", "well", "gradient", "three", "four"])
@pytest.mark.parametrize("size", SIZES + [(129, 130)])
def test_tiles_equal_the_ring_array_path_after_a_callers_writes(size, kind):
    import torch
    m, phi, mu = mb.load_case(_alloy(kind, *size, (1, 1, 1, 1)))
    a, b = _pair(m)
    with a, b:
        for c in (a, b):
            c.upload(phi, mu)
            c.step(3)
        for k, n in enumerate((1, 1, 1, 8, 3, 9)):
            for c in (a, b):
                c.sync()
                _write(c, k)
                torch.cuda.synchronize()
                c.step(n)
            _same(a, b, f"write {k}, {n} steps")


def test_a_changed_state_costs_a_survey_not_the_bulk():
    """A caller that writes rows every step (slabs exchanging halos): one more pass over phi, not every bulk tile
    through the interface kernel.  On this grid (8,192 tiles, a few dozen with an interface) the latter took 3.8
    times a plain step, the survey takes 1.4 times."""
    import time
    m, phi, mu = mb.load_case(configs.c2(mesh=1024))
    with mb.Context(m, mb.GP_FP64) as c:
        c.upload(phi, mu)
        c.step(48)
        c.sync()

        def best(changed):
            t = []
            for _ in range(5):
                t0 = time.perf_counter()
                for _ in range(64):
                    c.step(1)
                    if changed:
                        c.state_changed()
                c.sync()
                t.append(time.perf_counter() - t0)
            return min(t)

        best(True)
        plain, changed = best(False), best(True)
    assert changed < 2.5 * plain, (changed / 64, plain / 64)


def _dense(mx, my, seed=6):
    """A well alloy (isotropic: _pair) whose grains leave hardly a tile without an interface."""
    c = configs.binary_case(mx, my, gap=1.0, supersat=0.5, eps=4.0, dt=0.05, tau=1.7776, function_w=2, seed=(0, 0, 5.0))
    m, phi, mu = mb.load_case(c)
    x, y = np.mgrid[0:mx, 0:my]
    rng = np.random.default_rng(seed)
    d = np.min([np.hypot(x - a, y - b) for a, b in rng.uniform(0, 1, (mx * my // 1500, 2)) * (mx, my)], 0) - 12.0
    phi[0] = 0.5 - 0.5 * np.sin(np.pi * np.clip(d / 9.6, -0.5, 0.5))
    phi[1] = 1.0 - phi[0]
    return m, phi, mu


def test_the_path_follows_the_share_of_listed_tiles_and_the_bits_do_not():
    """A dense state (through the ring array once the host has seen the count), a sparse one written over it
    (back to the tiles when the count is taken anew), shifts and smoothing in between, against the ring array
    throughout."""
    m, phi, mu = _dense(300, 280)
    sparse = np.zeros_like(phi)
    sparse[0, :20, :20] = 1.0
    sparse[1] = 1.0 - sparse[0]
    a, b = _pair(m)
    with a, b:
        for state in (phi, sparse, phi):
            for c in (a, b):
                c.upload(state, mu)
            for n in (1, 3, 8, 17, 64, 5):
                for c in (a, b):
                    c.step(n)
                _same(a, b, n)
            for c in (a, b):
                c.shift_y(3)
                c.step(9)
                c.smooth(2)
                c.step(600)  # past the next count
                c.step(1)
            _same(a, b, "long")


def test_dense_two_phase_states_are_not_slower_than_the_ring_array():
    """684 tiles, all listed: 40 us per step through the tile kernels, 29 through the ring array."""
    import time
    m, phi, mu = _dense(300, 280)
    best = []
    for c in _pair(m):
        with c:
            c.upload(phi, mu)
            c.step(32)
            c.sync()
            t = []
            for _ in range(6):
                t0 = time.perf_counter()
                c.step(64)
                c.sync()
                t.append(time.perf_counter() - t0)
            best.append(min(t))
    assert best[0] < 1.2 * best[1], best


def test_creating_a_context_stays_cheap_and_many_of_them_keep_apart():
    """A context takes about as long with the host's word for its tile count as without one (a grid that one round
    of blocks covers has none); page-locked memory of its own took 1 to 3 ms more.  Contexts created and closed
    in turn, more than the page has words, and dense and sparse ones alive together keep their own counts."""
    import time
    dense, phi, mu = _dense(300, 280)
    sparse, sp, su = mb.load_case(_alloy("obstacle", 300, 280, (1, 1, 1, 1)))
    small = mb.load_case(_alloy("obstacle", 128, 128, (1, 1, 1, 1)))[0]
    t = ([], [])
    for _ in range(25):  # in turn: the host's allocations take longer at some times than at others
        for m, v in zip((small, mb.load_case(_alloy("obstacle", 128, 300, (1, 1, 1, 1)))[0]), t):
            t0 = time.perf_counter()
            c = mb.Context(m, mb.GP_FP64)
            v.append(time.perf_counter() - t0)
            c.close()
    assert min(t[1]) < min(t[0]) + 0.5e-3, (min(t[0]), min(t[1]))
    for _ in range(1100):
        mb.Context(dense, mb.GP_FP64).close()
    a, b = _pair(dense)
    c, d = _pair(sparse)
    with a, b, c, d:
        for x in (a, b):
            x.upload(phi, mu)
        for x in (c, d):
            x.upload(sp, su)
        for n in (9, 40, 17):
            for x in (a, c, b, d):
                x.step(n)
            _same(a, b, n)
            _same(c, d, n)
