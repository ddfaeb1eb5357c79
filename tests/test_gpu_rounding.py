"""Rounding of the operators that take gradients at the Gauss points (reinitialisation, normal and curvature
right-hand sides, banded projection): they may be no further from 80-bit values than plain quadrature sums in the
operator's own precision, on nearly constant fields, where a gradient is a small difference of large values."""
import numpy as np
import pytest

from tests.gpu_util import to_gpu

pytestmark = pytest.mark.gpu

LD = np.longdouble


def lagrange(nodes, x):
    """Values and derivatives of the Lagrange polynomials of `nodes` at `x` (rows: points)."""
    n = len(nodes)
    V, G = np.ones((len(x), n), LD), np.zeros((len(x), n), LD)
    for a in range(n):
        rest = [b for b in range(n) if b != a]
        for b in rest:
            V[:, a] *= (x - nodes[b]) / (nodes[a] - nodes[b])
        for c in rest:
            t = np.full(len(x), 1 / (nodes[a] - nodes[c]))
            for b in rest:
                if b != c:
                    t = t * (x - nodes[b]) / (nodes[a] - nodes[b])
            G[:, a] += t
    return V, G


def rule(k):
    """Gauss-Lobatto nodes, Gauss points and weights on [0, 1] by Newton's method in 80 bits."""
    def newton(c, x):
        x = x.astype(LD)
        for _ in range(4):
            x = x - polyval(c, x) / polyval(polyder(c), x)
        return x

    def polyval(c, x):
        s = np.zeros_like(x)
        for a in c[::-1]:
            s = s * x + a
        return s

    polyder = lambda c: np.array([j * c[j] for j in range(1, len(c))] or [LD(0)], LD)  # noqa: E731
    legendre = [np.array([1], LD), np.array([0, 1], LD)]
    for j in range(2, k + 2):
        p = np.zeros(j + 1, LD)
        p[1:] = (2 * j - 1) * legendre[-1] / LD(j)
        p[:j - 1] -= (j - 1) * legendre[-2] / LD(j)
        legendre.append(p)
    q = newton(legendre[k + 1], np.polynomial.legendre.leggauss(k + 1)[0])
    w = 2 / ((1 - q * q) * polyval(polyder(legendre[k + 1]), q) ** 2)
    d = polyder(legendre[k])
    inner = newton(d, np.sort(np.roots(d[::-1].astype(float)).real)) if k > 1 else np.zeros(0, LD)
    nodes = (1 + np.concatenate([[LD(-1)], inner, [LD(1)]])) / 2
    return nodes, (1 + q) / 2, w / 2


class Sums:
    """Plain quadrature sums over all nodes of a cell, in precision T."""

    def __init__(self, mesh, T):
        k = mesh.degree
        nodes, q, w = rule(k)
        V, G = lagrange(nodes, q)
        h = [LD(length / m) for length, m in zip(mesh.length, mesh.cells)]
        self.T, self.mesh, self.n = T, mesh, k + 1
        c = lambda a: a.astype(T)  # noqa: E731
        three = lambda z, y, x: np.einsum("al,bj,ci->abclji", c(z), c(y), c(x)).reshape(self.n ** 3, -1)  # noqa: E731
        self.phi = three(V, V, V)
        self.grad = [three(V, V, G / h[0]), three(V, G / h[1], V), three(G / h[2], V, V)]
        self.jxw = c(h[0] * h[1] * h[2] * np.einsum("a,b,c->abc", w, w, w).reshape(-1))
        at = [k * np.arange(m)[:, None] + np.arange(self.n)[None, :] for m in mesh.cells]
        n0, n1 = mesh.n[0], mesh.n[1]
        self.idx = (at[0][None, None, :, None, None, :] + n0 * (at[1][None, :, None, None, :, None] +
                    n1 * at[2][:, None, None, :, None, None])).reshape(-1, self.n ** 3)

    def cells(self, u):
        return np.asarray(u).astype(self.T)[self.idx]

    def value(self, u):
        return self.cells(u) @ self.phi.T

    def gradient(self, u):
        return [self.cells(u) @ g.T for g in self.grad]

    def test(self, value, flux):
        cell = 0
        if value is not None:
            cell = (value * self.jxw) @ self.phi
        if flux is not None:
            cell = cell + sum((f * self.jxw) @ g for f, g in zip(flux, self.grad))
        out = np.zeros(self.mesh.ndofs, self.T)
        np.add.at(out, self.idx, cell)
        return out


def unit(v):
    norm = np.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
    return [c / norm for c in v]


def check(got, form, mesh, T):
    ref = form(Sums(mesh, LD))
    norm = lambda a: np.sqrt((a.astype(LD) ** 2).sum())  # noqa: E731
    err, plain = norm(got.cpu().numpy() - ref), norm(form(Sums(mesh, T)) - ref)
    assert err <= plain, (float(err / norm(ref)), float(plain / norm(ref)))


@pytest.mark.parametrize("degree,m", [(1, (12, 10, 9)), (2, (7, 6, 5)), (3, (5, 4, 4)), (2, (34, 5, 2))])
@pytest.mark.parametrize("fp32", [False, True])
def test_gradients_of_nearly_constant_fields(degree, m, fp32):
    import torch

    from meltpooldg_b200.operators import HeatDiffuseOperator, Mesh, OlssonOperator

    mesh = Mesh(degree, m, length=(1.0, 0.9, 1.1))
    T, dt = (np.float32, torch.float32) if fp32 else (np.float64, torch.float64)
    rng = np.random.default_rng(3)
    level = 1.0 + 0.01 * rng.random(mesh.ndofs)
    normal = [c + 0.01 * rng.random(mesh.ndofs) for c in (1.0, -0.5, 0.7)]
    x = to_gpu(level, dt)
    level_t = x.double().cpu().numpy()  # as the kernel gets it

    # reinitialisation without its mass term (dt = 1e30)
    eps_n, eps_t = 0.1, 0.025
    op = OlssonOperator(mesh, dt=1e30, eps_normal=eps_n, eps_tangential=eps_t)
    op.set_normal(*[to_gpu(c) for c in normal])
    y = torch.empty_like(x)

    def tangent(s, u=level_t):
        n, g = unit([s.value(c) for c in normal]), s.gradient(u)
        gn = sum(a * b for a, b in zip(g, n))
        return s.test(None, [s.T(eps_t) * a + s.T(eps_n - eps_t) * gn * b for a, b in zip(g, n)])

    op.vmult(y, x)
    check(y, tangent, mesh, T)
    # the banded projection's stiffness, every point in the band
    band = HeatDiffuseOperator(mesh, rho_cp=1.0, dt=1e30, conductivity=0.3)
    band.set_narrow_band(to_gpu(np.zeros(mesh.ndofs)), 1.0)
    band.vmult(y, x)
    check(y, lambda s: s.test(None, [s.T(0.3) * g for g in s.gradient(level_t)]), mesh, T)
    assert op.device_errors() == 0 and band.device_errors() == 0
    if fp32:
        return
    # at |psi| = 1 + O(0.01) the compressive flux is as small as the diffusive one
    r = torch.empty_like(x)
    op.create_rhs(r, x)

    def rhs(s):
        n, c = unit([s.value(c) for c in normal]), s.value(level)
        return s.test(None, [s.T(0.5) * (1 - c * c) * b for b in n]) - tangent(s)

    check(r, rhs, mesh, T)
    for banded in (False, True):
        p = HeatDiffuseOperator(mesh, rho_cp=1.0, dt=1.0, conductivity=1.0)
        if banded:
            p.set_narrow_band(x, 2.0)
        out = [torch.zeros_like(x) for _ in range(3)]
        p.level_set_normal_rhs(x, *out)
        for d in range(3):
            check(out[d], lambda s, d=d: s.test(s.gradient(level)[d], None), mesh, T)
            out[d].zero_()
        p.level_set_normal_rhs(x, *out, normalized=True)
        for d in range(3):
            check(out[d], lambda s, d=d: s.test(unit(s.gradient(level))[d], None), mesh, T)
        p.level_set_curvature_rhs(r, *[to_gpu(c) for c in normal], 1e-10)
        check(r, lambda s: -s.test(sum(s.gradient(c)[d] for d, c in enumerate(unit([c.astype(s.T) for c in normal]))), None), mesh, T)
        assert p.device_errors() == 0
