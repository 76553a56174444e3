"""The adjoint's tiled kernels at the sizes where they can go wrong: grids smaller than a tile, exact
multiples of the 8 x 32 tile and one cell either way, interfaces crossing every border, each boundary
type per axis, and segments whose Delta-phi is recomputed state by state.

The yardstick is a directional central difference of the FP64 forward (the initial-state adjoint and the
mobility/diffusivity gradients in one number each): with h = 1e-6 its own error is about 1e-9 relative from
rounding plus h^2 from the third derivative, far below the 1e-4 asked for."""
import numpy as np
import pytest

import microsim_b200 as mb
from microsim_b200 import adjoint, configs

pytestmark = pytest.mark.gpu

SIZES = [(4, 4), (7, 31), (8, 32), (9, 33), (16, 64), (17, 65), (23, 5), (5, 70)]


def _case(mx, my, bc, well):
    c = configs.binary_case(mx, my, gap=1.0, supersat=0.5, eps=3.0, delta=0.03, theta=12.0, dt=0.05, tau=1.3332,
                            function_w=2 if well else 1, seed=(0, 0, 0.4 * max(mx, my)), bc=bc)
    return mb.load_case(c)


@pytest.mark.parametrize("well", [0, 1])
@pytest.mark.parametrize("bc", [(1, 1, 1, 1), (3, 3, 1, 1), (1, 1, 3, 3), (3, 3, 3, 3)])
@pytest.mark.parametrize("size", SIZES)
def test_adjoint_matches_directional_differences(size, bc, well):
    m, phi, mu = _case(*size, bc, well)
    rng = np.random.default_rng(1)
    with mb.Context(m, mb.GP_FP64) as c:  # a state with a developed interface, off the projection's corners
        c.upload(phi, mu)
        c.step(60)
        phi, mu = c.download()
    steps = 5
    wp, wu = rng.standard_normal(phi.shape), rng.standard_normal(mu.shape)
    inside = (phi > 1e-3) & (phi < 1 - 1e-3)
    dphi, dmu = rng.standard_normal(phi.shape) * inside, rng.standard_normal(mu.shape)
    dp = np.array([0.3, 0.0, 0.2, 0.3])
    p = adjoint.params_of(m)

    def forward(h, every=0, back=False):
        with adjoint.Adjoint(adjoint.with_params(m, p + h * dp), mb.GP_FP64) as a:
            q, u = a.forward(phi + h * dphi, mu + h * dmu, steps, every)
            if back:
                return a.backward(wp, wu, initial=True)
            return float((wp * q).sum() + (wu * u).sum())

    g, lphi, lmu = forward(0.0, back=True)
    an = float((lphi * dphi).sum() + (lmu * dmu).sum() + g @ dp)
    h = 1e-6
    fd = (forward(h) - forward(-h)) / (2 * h)
    scale = np.abs(lphi * dphi).sum() + np.abs(lmu * dmu).sum() + np.abs(g * dp).sum()
    assert abs(an - fd) <= 1e-4 * scale, (an, fd, scale)
    for every in (1, 2, steps):
        g2, lphi2, lmu2 = forward(0.0, every, True)
        np.testing.assert_allclose(g2, g, rtol=1e-9, atol=1e-12 * np.abs(g).max())
        np.testing.assert_allclose(lphi2, lphi, rtol=1e-9, atol=1e-11 * np.abs(lphi).max())


def test_forward_is_the_plain_step_at_every_size():
    for size in SIZES:
        m, phi, mu = _case(*size, (3, 3, 1, 1), 0)
        with adjoint.Adjoint(m, mb.GP_FP64) as a:
            pa, ua = a.forward(phi, mu, 40)
        with mb.Context(m, mb.GP_FP64) as c:
            c.upload(phi, mu)
            c.step(40)
            pp, up = c.download()
        assert np.abs(pa - pp).max() <= 1e-10 and np.abs(ua - up).max() <= 1e-10, size


def test_runs_of_different_lengths_on_one_object():
    """The kept workspaces serve shorter, longer and shorter runs again, each as a fresh object's."""
    m, phi, mu = _case(33, 40, (1, 1, 1, 1), 0)
    w = np.random.default_rng(2).standard_normal(phi.shape)
    with adjoint.Adjoint(m, mb.GP_FP64) as a:
        for steps, every in ((9, 0), (50, 0), (4, 1), (50, 25), (1, 0)):
            q, u = a.forward(phi, mu, steps, every)
            g = a.backward(w)
            with adjoint.Adjoint(m, mb.GP_FP64) as b:
                q2, u2 = b.forward(phi, mu, steps, every)
                g2 = b.backward(w)
            assert np.array_equal(q, q2) and np.array_equal(u, u2)
            np.testing.assert_allclose(g, g2, rtol=1e-10)


@pytest.mark.parametrize("precision", [mb.GP_FP64, mb.GP_FP32])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_loss_that_does_not_see_a_nonfinite_cell_has_finite_gradients(bad, precision):
    """mu is not finite in one cell of the bulk liquid, the loss takes phi around the crystal alone: where no
    adjoint arrives, none leaves, whatever the fields hold there."""
    m, phi, mu = _case(48, 90, (1, 1, 1, 1), 0)
    with mb.Context(m, mb.GP_FP64) as c:
        c.upload(phi, mu)
        c.step(60)
        phi, mu = c.download()
    assert phi[1, 36:, 70:].min() == 1.0  # bulk there
    w = np.random.default_rng(3).standard_normal(phi.shape) * ((phi > 0) & (phi < 1))
    spoilt = mu.copy()
    spoilt[0, 42, 80] = bad
    got = []
    for u in (mu, spoilt):
        with adjoint.Adjoint(m, precision) as a:
            a.forward(phi, u, 3)
            got.append(a.backward(w, None, initial=True))
    rtol = 1e-9 if precision == mb.GP_FP64 else 1e-4  # the order of the atomic additions
    for clean, x in zip(*got):
        assert np.isfinite(x).all()
        np.testing.assert_allclose(x, clean, rtol=rtol, atol=rtol * np.abs(clean).max())


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


def test_a_long_runs_memory_is_given_back_by_a_short_one():
    m, phi, mu = _case(512, 512, (1, 1, 1, 1), 0)
    with adjoint.Adjoint(m, mb.GP_FP32) as a:
        a.forward(phi, mu, 4)
        short = _free()
        a.forward(phi, mu, 900)  # 60 states of 3 MB and 30 slots of 3 MB
        long = _free()
        a.forward(phi, mu, 4)
        assert long < short - (200 << 20)
        assert _free() > short - (80 << 20)


def test_slots_leave_memory_to_others_and_one_slot_gives_the_same():
    """With about 2.4 GB free: 65 states of 12.6 MB fit, a slot for each of a segment's 64 states would take
    as much again and more than half of what is free."""
    import torch
    m, phi, mu = _case(1024, 1024, (1, 1, 1, 1), 0)
    w = np.random.default_rng(2).standard_normal(phi.shape)
    got = []
    for tight in (False, True):
        hog = None
        with adjoint.Adjoint(m, mb.GP_FP32) as a:
            if tight:
                torch.cuda.empty_cache()
                hog = torch.empty(_free() - 2400 * (1 << 20), dtype=torch.uint8, device="cuda")
            a.forward(phi, mu, 64, 64)
            if tight:
                assert _free() > 1300 * (1 << 20)
            got.append(a.backward(w, None, initial=True))
        del hog
        torch.cuda.empty_cache()
    for x, y in zip(*got):
        np.testing.assert_allclose(x, y, rtol=1e-4, atol=1e-4 * np.abs(x).max())


SPACINGS = [(0.5, 2.0), (0.7, 1.3)]  # products with reciprocals, quotients


@pytest.mark.parametrize("well", [0, 1])
@pytest.mark.parametrize("size", [(9, 33), (33, 47)])
@pytest.mark.parametrize("spacing", SPACINGS)
def test_adjoint_at_other_spacings(spacing, size, well):
    """FP64 against directional differences (as above), FP32 against FP64 for the obstacle potential: its fields and
    adjoints are rounded at every one of five steps and reverses, a few times 6e-8 each, which the antitrapping
    term's quotients grow tenfold (2e-6 seen); a wrong or swapped spacing is an error of its own size.  (In a well's
    tails 1 - phi is below FP32's resolution of phi: which phases are active there is a matter of rounding at
    any spacing, and random weights see it.)"""
    m, phi, mu = _case(*size, (1, 1, 1, 1), well)
    m.dx, m.dy = spacing
    m.dt *= 0.4
    with mb.Context(m, mb.GP_FP64) as c:
        c.upload(phi, mu)
        c.step(60)
        phi, mu = c.download()
        c.step(5)
        want = c.download()
    rng = np.random.default_rng(7)
    wp, wu = rng.standard_normal(phi.shape), rng.standard_normal(mu.shape)
    dphi = rng.standard_normal(phi.shape) * ((phi > 1e-3) & (phi < 1 - 1e-3))
    dmu, dp, p = rng.standard_normal(mu.shape), np.array([0.3, 0.0, 0.2, 0.3]), adjoint.params_of(m)

    def forward(h, precision=mb.GP_FP64, back=False):
        with adjoint.Adjoint(adjoint.with_params(m, p + h * dp), precision) as a:
            q, u = a.forward(phi + h * dphi, mu + h * dmu, 5)
            return (a.backward(wp, wu, initial=True), q, u) if back else float((wp * q).sum() + (wu * u).sum())

    (g, lphi, lmu), q, u = forward(0.0, back=True)
    assert np.abs(q - want[0]).max() <= 1e-10 and np.abs(u - want[1]).max() <= 1e-10
    an = float((lphi * dphi).sum() + (lmu * dmu).sum() + g @ dp)
    fd = (forward(1e-6) - forward(-1e-6)) / 2e-6
    scale = np.abs(lphi * dphi).sum() + np.abs(lmu * dmu).sum() + np.abs(g * dp).sum()
    assert abs(an - fd) <= 1e-4 * scale, (an, fd, scale)
    if well:
        return
    (g32, lphi32, lmu32), _, _ = forward(0.0, mb.GP_FP32, True)
    for a, b in ((lphi32, lphi), (lmu32, lmu)):
        assert np.linalg.norm(a - b) <= 2e-5 * np.linalg.norm(b)
    assert np.abs(g32 - g).max() <= 2e-5 * np.abs(g).max()


@pytest.mark.parametrize("spacing", [(1.0, 1.0)] + SPACINGS)
def test_fp32_adjoint_sums_are_rounded_at_their_own_scale(spacing):
    """The adjoint of mu after five reverse steps, FP32 against FP64.  A cell's four faces are summed apart and
    added once, a rounding of at most 2^-24 = 6e-8 of its value per step (3.4e-8 root mean square, so 7.7e-8 over
    five steps if all were as large as the result; 5.4e-8 to 6.4e-8 measured); four additions in turn gave 9.1e-8
    to 1.06e-7."""
    m, phi, mu = _case(33, 47, (1, 1, 1, 1), 0)
    m.dx, m.dy = spacing
    m.dt *= 1.0 if spacing == (1.0, 1.0) else 0.4
    with mb.Context(m, mb.GP_FP64) as c:
        c.upload(phi, mu)
        c.step(60)
        phi, mu = c.download()
    rng = np.random.default_rng(7)
    wp, wu = rng.standard_normal(phi.shape), rng.standard_normal(mu.shape)
    lmu = []
    for precision in (mb.GP_FP64, mb.GP_FP32):
        with adjoint.Adjoint(m, precision) as a:
            a.forward(phi, mu, 5)
            lmu.append(a.backward(wp, wu, initial=True)[2])
    assert np.linalg.norm(lmu[1] - lmu[0]) <= 7.7e-8 * np.linalg.norm(lmu[0])


@pytest.mark.parametrize("precision", [mb.GP_FP64, mb.GP_FP32])
def test_a_face_without_adjoint_leaves_the_diffusivity_gradient_finite(precision):
    """phi of the liquid is infinite in one bulk cell that the loss does not see.  That cell's own update makes the
    other gradients NaN (0 times its mobility's terms, whichever kernels run); its faces have a zero adjoint."""
    m, phi, mu = _case(48, 90, (1, 1, 1, 1), 0)
    with mb.Context(m, mb.GP_FP64) as c:
        c.upload(phi, mu)
        c.step(60)
        phi, mu = c.download()
    w = np.random.default_rng(3).standard_normal(phi.shape) * ((phi > 0) & (phi < 1))
    spoilt = phi.copy()
    spoilt[1, 42, 80] = np.inf
    got = []
    for p in (phi, spoilt):
        with adjoint.Adjoint(m, precision) as a:
            a.forward(p, mu, 1)
            got.append(a.backward(w)[3])
    np.testing.assert_allclose(got[1], got[0], rtol=1e-9 if precision == mb.GP_FP64 else 1e-4)
