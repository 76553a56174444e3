"""What an FP32 context and a batch choose by themselves against a batch told to use 16x32 tiles, 256
threads and (by odd step counts) direct launches: bit for bit, on grids either side of the lines where
the small tiles give way (1,184 tiles of 8x32, 832 with a well) and the wide blocks do (a well, 296), isothermal and in a frozen gradient, across a switch of
the accumulation mode (which drops the captured steps) and runs split so that both replayed and direct
steps occur."""
import numpy as np
import pytest

import microsim_b200 as mb
from microsim_b200 import configs

pytestmark = pytest.mark.gpu

SIZES = [(4, 4), (8, 32), (9, 33), (70, 90), (592, 512), (600, 512),  # the last two: 1,184 and 1,200 tiles
         (296, 256), (304, 256), (416, 512), (424, 512)]              # 296, 304, 832 and 848


def _case(kind, mx, my):
    if kind == "four":
        c = configs.c3(steps=10, mesh=max(mx, 16), nseeds=6, rng_seed=8)
        c.mesh_x, c.mesh_y = mx, my
        c.fills = [("FILLCYLINDER", [i, (i + 1) * mx // 4, my // 3, 0, 0, max(1.5, min(mx, my) / 9.0)]) for i in range(3)]
        return c
    c = configs.binary_case(mx, my, gap=1.0, supersat=0.5, eps=4.0, delta=0.03, theta=10.0, dt=0.05, tau=1.7776,
                            function_w=2 if kind == "well" else 1, seed=(0, 0, 0.3 * min(mx, my)))
    if kind == "gradient":
        c.tempgrady = (0.97, 0.08, float(my), 2.0, 0.5)
    return c


@pytest.mark.parametrize("kind", ["obstacle", "well", "gradient", "four"])
@pytest.mark.parametrize("size", SIZES)
def test_defaults_equal_large_tiles_and_direct_steps(size, kind):
    m, phi, mu = mb.load_case(_case(kind, *size))
    with mb.Context(m, mb.GP_FP32) as c, mb.Batch([m]) as d, mb.Batch([m]) as b:
        b.set_tile(16, 32)
        if kind != "four":
            b.set_block(256)
        c.upload(phi, mu)
        d.upload(0, phi, mu)
        b.upload(0, phi, mu)
        for n, comp in ((3, False), (64, False), (21, True), (75, True), (9, False), (135, True), (40, False), (17, False)):
            c.set_compensated(comp)
            d.set_compensated(comp)
            b.set_compensated(comp)
            c.step(n)
            d.step(n)
            for _ in range(n):
                b.step(1)
            pc, uc = c.download()
            pd, ud = d.download(0)
            pb, ub = b.download(0)
            assert np.array_equal(pc, pb) and np.array_equal(uc, ub), (n, comp)
            assert np.array_equal(pd, pb) and np.array_equal(ud, ub), (n, comp)


@pytest.mark.parametrize("size", [(300, 280), (400, 416), (512, 416), (592, 512)])
def test_the_default_shape_does_not_lose_on_well_grains(size):
    """A well potential's tails leave few pure tiles: the shape a context and a batch choose against 16x32 tiles
    with 256 threads, which they had everywhere before small tiles existed (8x32/512 on the last grid: 1.2 times
    their time)."""
    import time
    mx, my = size
    m, phi, mu = mb.load_case(_case("well", mx, my))
    x, y = np.mgrid[0:mx, 0:my]
    c = np.random.default_rng(6).uniform(0, 1, (30, 2)) * (mx, my)
    d = np.min([np.hypot(x - a, y - b) for a, b in c], 0) - 0.15 * min(mx, my)
    phi[0] = 0.5 - 0.5 * np.sin(np.pi * np.clip(d / 9.6, -0.5, 0.5))
    phi[1] = 1.0 - phi[0]
    best = []
    for given in (False, True):
        with mb.Batch([m]) as b:
            if given:
                b.set_tile(16, 32)
                b.set_block(256)
            b.upload(0, phi, mu)
            b.step(64)
            b.sync()
            t = []
            for _ in range(6):
                t0 = time.perf_counter()
                b.step(64)
                b.sync()
                t.append(time.perf_counter() - t0)
            best.append(min(t))
    assert best[0] < 1.12 * best[1], best


@pytest.mark.parametrize("n", [64, 100])
def test_a_short_run_does_not_pay_for_a_capture(n):
    """A new context's only call takes no more than the same steps in calls of twenty, which are direct: less than
    a third of the 200 us of a capture apart."""
    import time
    m, phi, mu = mb.load_case(_case("obstacle", 600, 512))
    best = []
    for split in (1, n // 20):
        t = []
        for _ in range(9):
            with mb.Context(m, mb.GP_FP32) as c:
                c.upload(phi, mu)
                c.sync()
                t0 = time.perf_counter()
                for _ in range(split):
                    c.step(n // split)
                c.sync()
                t.append(time.perf_counter() - t0)
        best.append(min(t))
    assert best[0] < best[1] + 60e-6, best
