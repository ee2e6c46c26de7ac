"""The arithmetic of the kernels' Lanczos runs, restated here in FP64, against the
reference's scheme (src/hydrodynamics.cpp:146-264), and the refined reciprocal square
root of device_physics.cuh against its error bound.

Both kernels run cold (30 steps, projections on the whole basis where BasisLoss of
integrator_team.cuh asks for them, below 3N = 64 in every step) and warm (8 steps of the
three-term recurrence alone); the reference projects every vector on the whole basis.
Bounds:
- orthogonality of a cold basis: the square root of the products' rounding, the level up
  to which the tridiagonal is the projection of D to rounding (Simon): 2^-26 in FP64;
  on FP32 products (error 1e-7 of the largest entries) 1e-3;
- extreme eigenvalues: 1e-10 relative. A relative change x of a bound moves a
  Chebyshev result by about x times its order (some 20) times its truncation error
  (2.5e-3 at most), the noise enters with sqrt(dt) (0.03): 1e-10 moves a step by
  1.5e-13, within the 1e-12 that the steps are held to. On FP32 products: the largest
  within 1e-4, the smallest within the smaller of 0.1 of itself and 1e-5 of the largest
  (the bounds are padded by 2% and a factor of two), against the
  reference's scheme on the same products;
- where the reference's own value moves by more under a rounding error in D (the
  smallest one of a long-symmetric chain, not converged in 30 steps), 100 times that.
"""
from fractions import Fraction

import numpy as np
import pytest

from bdsim_b200 import gaussian_chain

COLD, WARM = 30, 8
ORTHOGONAL = 2.0 ** -26
BOUNDS_TOL = 1e-10


def rpy(R, h):
    N = len(R)
    d = R[None, :, :] - R[:, None, :]
    r = np.sqrt(np.maximum((d * d).sum(-1), 1e-12))
    a = np.sqrt(np.pi) * h
    far = 0.75 * a / r * (1 + 2 * np.pi / 3 * (h / r) ** 2), 0.75 * a / r ** 3 * (1 - 2 * np.pi * (h / r) ** 2)
    near = 1 - 0.75 / np.sqrt(np.pi) * 0.375 * r / h, 0.09375 / np.sqrt(np.pi) / (h * r)
    o1, o2 = (np.where(r >= 2 * a, f, n) for f, n in zip(far, near))
    np.fill_diagonal(o1, 1.0)
    np.fill_diagonal(o2, 0.0)
    D = o1[:, :, None, None] * np.eye(3) + o2[:, :, None, None] * d[..., :, None] * d[..., None, :]
    return D.transpose(0, 2, 1, 3).reshape(3 * N, 3 * N)


def product(D, u, mixed):
    return (D.astype(np.float32) @ u.astype(np.float32)).astype(np.float64) if mixed else D @ u


def reference_run(D, v, m, mixed=False):
    V, al, be, b, vp = [], [], [], 0.0, 0.0 * v
    for _ in range(min(m, len(v))):
        V.append(v)
        w = product(D, v, mixed)
        al.append(v @ w)
        w = w - al[-1] * v - b * vp
        for x in V:
            w = w - (w @ x) * x
        b = np.sqrt(w @ w)
        if b < 1e-10 or len(V) == min(m, len(v)):
            break
        be.append(b)
        vp, v = v, w / b
    return np.array(V), np.array(al), np.array(be[:len(al) - 1])


F = np.float32


class BasisLoss:
    def __init__(self, eps, tol, tiny):
        self.eps, self.tol, self.tiny = F(eps), F(tol), F(tiny)
        self.w = self.wp = self.bmax = F(0)
        self.again = False

    def project(self, j, al, bt, ww):
        if j == 0:
            self.lo = self.hi = F(al)
            bt = 0.0
        a, b, sq = F(al), F(bt), F(ww - al * al - bt * bt)
        self.lo, self.hi, self.bmax = min(self.lo, a), max(self.hi, a), max(self.bmax, b)
        lost = not sq > self.tiny * F(ww)
        bn = F(1) if lost else np.sqrt(sq)
        f = max(self.hi - a, a - self.lo) + F(2) * max(self.bmax, bn)
        wn = (f * self.w + b * self.wp + self.eps * (abs(a) + b + bn)) / bn
        hit = lost or not wn <= self.tol
        now = hit or self.again
        self.again = lost or (hit and not self.again)
        self.wp, self.w = self.w, self.eps if now else wn
        return now


def kernel_run(D, v, m, cold, mixed=False):
    n, V, al, be, u, vp = len(v), [], [], [], v, 0.0 * v
    loss = BasisLoss(1e-7, 3e-4, 1e-5) if mixed else BasisLoss(4e-16, 1e-8, 1e-10)
    m = min(n, m)
    for j in range(m):
        w = product(D, u, mixed)
        bsq = u @ u
        if j > 0 and bsq < 1e-20:
            break
        ib = 1.0 / np.sqrt(bsq)
        a, bt, ww = (u @ w) * ib * ib, bsq * ib, (w @ w) * ib * ib
        al.append(a)
        if j > 0:
            be.append(bt)
        v = u * ib
        V.append(v)
        u = w * ib - a * v
        if j > 0:
            u = u - bt * vp
        vp = v
        if cold and (n < 64 or loss.project(j, a, bt, ww)):
            B = np.array(V)
            u = u - B.T @ (B @ u)
    return np.array(V), np.array(al), np.array(be)


def ritz(V, al, be):
    e, y = np.linalg.eigh(np.diag(al) + np.diag(be, 1) + np.diag(be, -1))
    return e[0], e[-1], V.T @ y[:, 0], V.T @ y[:, -1]


def positions(kind, N):
    t = np.arange(N)
    if kind == "coil":
        return gaussian_chain(N, bond_std=1.0, seed=N)
    if kind == "rod":
        return np.stack([1.3 * t, 0 * t, 0 * t], 1)
    if kind == "ring":
        x = 2 * np.pi * t / N
        return N / 5.0 * np.stack([np.cos(x), np.sin(x), 0 * t], 1)
    if kind == "planar":
        return gaussian_chain(N, bond_std=1.0, seed=N) * [1.0, 1.0, 0.0]
    if kind == "compact":
        return gaussian_chain(N, bond_std=1.0, seed=N) * 0.2
    if kind == "stretched":
        return gaussian_chain(N, bond_std=1.0, seed=N) * [8.0, 0.3, 0.3]
    return gaussian_chain(N, bond_std=1.0, seed=N) * float(kind)  # (collapsed by a factor)


def moved(D, v, m, rng, mixed=False):
    """The reference run's extreme eigenvalues, and how far rounding errors in D move them."""
    e = ritz(*reference_run(D, v, m, mixed))[:2]
    move = [0.0, 0.0]
    for _ in range(3):
        P = 1.0 + 2.0 ** (-23 if mixed else -52) * rng.uniform(-1, 1, D.shape)
        g = ritz(*reference_run(D * (P + P.T) / 2, v, m, mixed))[:2]
        move = [max(x, abs(g[k] - e[k])) for k, x in enumerate(move)]
    return e, move


KINDS = ["coil", "rod", "ring", "planar", "compact", "stretched", "0.1", "0.02", "0.005"]
SIZES = [2, 3, 5, 10, 21, 22, 24, 35, 50, 120, 200]


def start(kind, N, h):
    n = 3 * N
    seed = np.sin(0.7654321 * (np.arange(n) + 1)) + 0.5
    return rpy(positions(kind, N), h), seed / np.linalg.norm(seed)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("N", SIZES)
def test_extreme_eigenvalues(kind, N):
    rng = np.random.default_rng(N)
    for h in (0.05, 0.25, 0.5):
        D, seed = start(kind, N, h)
        got = kernel_run(D, seed, COLD, True)
        V = got[0]
        assert np.max(np.abs(V @ V.T - np.eye(len(V)))) <= ORTHOGONAL
        want, move = moved(D, seed, COLD, rng)
        g = ritz(*got)
        for k in (0, 1):
            assert abs(g[k] - want[k]) <= max(BOUNDS_TOL * abs(want[k]), 100 * move[k]), (h, k)
        # the next step's warm run, from the sum of the Ritz vectors
        w = ritz(*reference_run(D, seed, COLD))
        v = w[2] + w[3] + 0.01 * seed
        v /= np.linalg.norm(v)
        D = rpy(positions(kind, N) * (1.0 + 1e-3 * rng.standard_normal((N, 3))), h)
        got = kernel_run(D, v, WARM, False)
        if len(reference_run(D, v, WARM)[1]) < 4 or len(got[1]) < 4:
            continue  # too short: both start again cold
        want, move = moved(D, v, WARM, rng)
        g = ritz(*got)
        for k in (0, 1):
            assert abs(g[k] - want[k]) <= max(BOUNDS_TOL * abs(want[k]), 100 * move[k]), (h, k)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("N", [n for n in SIZES if n >= 22])
def test_extreme_eigenvalues_of_fp32_products(kind, N):
    rng = np.random.default_rng(N)
    for h in (0.05, 0.25, 0.5):
        D, seed = start(kind, N, h)
        got = kernel_run(D, seed, COLD, True, mixed=True)
        V = got[0]
        assert np.max(np.abs(V @ V.T - np.eye(len(V)))) <= 1e-3
        want, move = moved(D, seed, COLD, rng, mixed=True)
        g = ritz(*got)
        assert abs(g[1] - want[1]) <= 1e-4 * want[1]
        assert abs(g[0] - want[0]) <= max(min(0.1 * want[0], 1e-5 * want[1]), 100 * move[0])


def test_refined_reciprocal_square_root():
    """y (1 + e/2 + 3 e^2/8), e = 1 - s y^2, from any estimate within 2^-21: e is
    off by the rounding of s y (2^-53), half of which reaches the result, which is
    rounded once more (2^-53); the smaller terms fit in the 2^-52 asserted (one unit in
    the last place, as CUDA's own rsqrt())."""
    rng = np.random.default_rng(1)

    def rnd(x):  # one rounding to double
        return Fraction(float(x))

    half, c = Fraction(1, 2), Fraction(3, 8)
    for _ in range(20000):
        s = float(2.0 ** rng.uniform(-99, 126))
        y = float(np.float32(s ** -0.5 * (1.0 + rng.uniform(-1, 1) * 2.0 ** -21.2)))
        fs, fy = Fraction(s), Fraction(y)
        e = rnd(1 - rnd(fs * fy) * fy)
        r = rnd(rnd(fy * e) * rnd(e * c + half) + fy)
        assert abs(r * r * fs - 1) / 2 <= Fraction(1, 2 ** 52)
