"""The interior test of the Mandelbrot kernels (interior_c in
csrc/chaos_device.cuh): where it says yes, the rounded orbit never escapes.

With w = z - p about the attracting fixed point (mu = 2p, c = mu/2 - mu^2/4)
the step is w' = mu w + w^2, and the critical orbit w_k(mu) from w_1 = -mu^2/4
is a polynomial in mu; so are the products D_kn = prod (mu + 2 w_j), k <= j < n,
that carry an error of step k to step n.  Both are bounded on the whole disc
|mu| <= rho by their largest modulus on its rim (for the sum of |D_kn| over k
too: it is subharmonic), which ball arithmetic bounds here over the full rim:

  * |w_n| <= delta / 8 at n = 800 (delta = 1 - rho = 2^-7), and T >= sum_k |D_kn|
    for every n up to there.  An orbit whose every step is off by at most eta
    then stays within E = 2 eta T of w_n when 4 eta T^2 <= 1 (induction:
    e_n <= T (eta + E^2) = eta T (1 + 4 eta T^2)).
  * |w| <= delta / 4 maps into itself with steps off by eta when
    eta <= (3 delta / 4)(delta / 4), and |z| stays below 1.

eta = 2^-21 covers a binary32 step for |z| <= 1.25, the widest either orbit
gets: (2|z|^2 + |z'|, |z|^2 + |z'|) 2^-24 bounds the two coordinates' errors,
5.2 x 2^-24 in all; the other arithmetics round less.  The period-2 disc
(c = -1 + m/4, delta = 2^-6) goes the same way about its 2-cycle."""
import numpy as np

ETA = 2.0 ** -21


def rim(rho, boxes):
    """Centres of `boxes` arcs of the upper half of |mu| = rho (the lower is its conjugate) and their radius."""
    th = (np.arange(boxes) + 0.5) * (np.pi / boxes)
    return rho * np.exp(1j * th), rho * np.pi / (2 * boxes)


def test_cardioid_orbits_fall_into_the_invariant_disc():
    delta = 2.0 ** -7
    mu, eps = rim(1 - delta, 120_000)
    w, r = -mu * mu / 4, np.full(mu.size, eps * 0.5 + eps * eps)
    t = np.zeros(mu.size)
    t_max, w_max = 0.0, 0.0
    for _ in range(800):
        d = np.abs(mu + 2 * w)
        t = t * (d + 2 * r + eps) + 1
        r = r * (d + r + eps) + eps * np.abs(w) + 1e-15
        w = w * (w + mu)
        t_max, w_max = max(t_max, t.max()), max(w_max, (np.abs(w) + r).max())
    err = 2 * ETA * t_max
    assert 4 * ETA * t_max ** 2 <= 1
    assert (np.abs(w) + r).max() <= delta / 8 and delta / 8 + err <= delta / 4
    assert ETA <= (3 * delta / 4) * (delta / 4)
    assert 0.5 + w_max + err < 1.25


def test_period_two_orbits_fall_into_the_invariant_disc():
    delta = 2.0 ** -6
    m, eps = rim(1 - delta, 60_000)
    c = -1 + m / 4
    s = np.sqrt(1 - m)
    p = [(-1 - s) / 2, (-1 + s) / 2]  # the cycle; the orbit starts at c, next to the first
    eps_p = eps / (4 * (np.abs(s) - eps / np.abs(s)))
    u, r = c - p[0], eps / 4 + eps_p
    t = np.zeros(m.size)
    t_max, z_max = 0.0, 0.0
    for k in range(1000):
        d = 2 * np.abs(u + p[k & 1])
        t = t * (d + 2 * r + 2 * eps_p) + 1
        r = r * (d + r + 2 * eps_p) + 2 * eps_p * np.abs(u) + 1e-15
        u = u * (u + 2 * p[k & 1])
        t_max, z_max = max(t_max, t.max()), max(z_max, (np.abs(u + p[(k + 1) & 1]) + r).max())
    err = 2 * ETA * t_max
    assert 4 * ETA * t_max ** 2 <= 1
    ball = delta / 32
    assert (np.abs(u) + r).max() + err <= ball
    # two steps from |v| <= ball about either point: |v''| <= |v| (|m| + 7 |v|) + 3.5 eta
    assert ball * (1 - delta + 7 * ball) + 3.5 * ETA <= ball
    assert z_max + err < 1.25


def test_the_binary32_test_accepts_no_other_point():
    """interior_c restated in binary32 with each square root off by 2^-23 upwards, against the multipliers in
    extended precision, at points on both sides of its bounds."""
    f = np.float32
    rng = np.random.default_rng(3)
    n = 2_000_000
    rho = 1 - 2.0 ** -7 + rng.uniform(-3e-4, 3e-4, n)
    mu = rho * np.exp(2j * np.pi * np.concatenate([rng.uniform(0, 1, n // 2), rng.uniform(-1e-3, 1e-3, n - n // 2)]))
    disc = -1 + (1 - 2.0 ** -6 + rng.uniform(-3e-4, 3e-4, n)) / 4 * np.exp(2j * np.pi * rng.uniform(0, 1, n))
    c = np.concatenate([mu / 2 - mu * mu / 4, disc])
    cx, cy = c.real.astype(f), c.imag.astype(f)
    up = f(1 + 2.0 ** -22)
    with np.errstate(invalid="ignore"):
        y2 = cy * cy
        a = f(1) - f(4) * cx
        big = np.sqrt(a * a + f(16) * y2) * up
        re = np.sqrt(f(0.5) * big + f(0.5) * a) * up
        yes = (f(2) * re - big >= f(0.0158)) | ((cx + f(1)) * (cx + f(1)) + y2 <= f(0.0605))
    z = cx.astype(np.longdouble) + 1j * cy.astype(np.longdouble)
    inside = (np.abs(1 - np.sqrt(1 - 4 * z)) <= 1 - 2.0 ** -7) | (4 * np.abs(z + 1) <= 1 - 2.0 ** -6)
    assert yes.any() and not (yes & ~inside).any()
