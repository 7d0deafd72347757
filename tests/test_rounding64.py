"""Rounding error of the FP64 hydro step against 80-bit arithmetic.

The same step is evaluated in three ways: exactly (numpy's 80-bit long double), in FP64 with
every operation of the scheme rounded once and the multiply-adds fused, and by the kernel.  The
kernel's rms error may not pass the second's by more than 2 %.  That is the scatter allowed: over
2 x 10^4 cells whose errors are sums of some eight roundings, an rms is known to 1 / (2 sqrt(n)) =
0.4 %, the ratio of two to 0.5 %.  One rounding more per sweep in a momentum adds some 6 %."""
import numpy as np
import pytest

import diskgpu as D
from fake_lib import fake_child, fake_lib  # noqa: F401 (a fixture)

LD = np.longdouble


def step(T, fma, S, u, w, dt, K, gamma, GM, R, Rf, dphi):
    """DiskHydro::step without self-gravity, in type T; fma(a, b, c) = a b + c."""
    R, Rf, dt, dphi, K, gm, half = R.astype(T)[:, None], Rf.astype(T)[:, None], T(dt), T(dphi), T(K), T(gamma), T(0.5)
    up, dn = (lambda a: np.concatenate([a[1:], a[-1:]])), (lambda a: np.concatenate([a[:1], a[:-1]]))
    E, W = (lambda a: np.roll(a, -1, 1)), (lambda a: np.roll(a, 1, 1))  # values of cells j + 1, j - 1
    dR = Rf[1:] - Rf[:-1]
    vol = R * dR * dphi

    def limit(a, b):
        p = a * b
        return np.where(p > 0, 2 * p / np.where(p > 0, a + b, T(1)), T(0))

    P = K * (S * S) if gamma == 2.0 else K * S ** gm
    aR = fma(w, w * (1 / R), fma(-((up(P) - dn(P)) * (1 / (up(R) - dn(R)))), 1 / S, -T(GM) / (R * R)))
    ap = fma(-1 / (2 * dphi * R), (E(P) - W(P)) * (1 / S), -(u * (w * (1 / R))))
    u, w = fma(dt, aR, u), fma(dt, ap, w)

    def sweep(qc, left, kl, right, kr, vf, h, A, diff):  # cells; either side of the faces, with slopes
        f = [fma(h, np.where(vf > 0, k, m), np.where(vf > 0, a, b)) for a, k, b, m in zip(left, kl, right, kr)]
        F = vf * f[0] * A
        cv = dt * (1 / vol)
        n = fma(cv, diff(F), qc[0])
        d = np.maximum(n, T(1e-10))
        return [n] + [fma(qc[0], a, cv * diff(F * x)) / d for a, x in zip(qc[1:], f[1:])]

    qc = [S, u, w]
    kq = []
    for a in qc:
        k = np.zeros_like(a)
        k[1:-1] = limit(a[2:] - a[1:-1], a[1:-1] - a[:-2])
        kq.append(k)
    vf = half * (u[:-1] + u[1:])
    h = np.where(vf > 0, fma(-vf, half * dt / dR[:-1], half), fma(-vf, half * dt / dR[1:], -half))
    z = lambda F: np.concatenate([np.zeros_like(F[:1]), F, np.zeros_like(F[:1])])  # noqa: E731
    qc = sweep(qc, [a[:-1] for a in qc], [k[:-1] for k in kq], [a[1:] for a in qc], [k[1:] for k in kq], vf, h,
                Rf[1:-1] * dphi, lambda F: z(F)[:-1] - z(F)[1:])
    kq = [limit(E(a) - a, a - W(a)) for a in qc]
    vf = half * (W(qc[2]) + qc[2])
    h = fma(-vf, half * dt / (R * dphi), np.where(vf > 0, half, -half))
    return sweep(qc, [W(a) for a in qc], [W(k) for k in kq], qc, kq, vf, h, dR, lambda F: F - E(F))


@pytest.mark.gpu
@pytest.mark.parametrize("Nu,Nphi,gamma", [(128, 160, 2.0), (160, 128, 1.6)])
def test_step_rounds_no_more_than_the_scheme_needs(Nu, Nphi, gamma):
    r = np.random.RandomState(Nu)
    dk = D.DiskHydro(Nu, Nphi, gamma=gamma)
    j = np.arange(Nphi) * 2 * np.pi / Nphi
    S = 0.4 + 0.2 * np.cos(2 * j)[None] * r.uniform(0.5, 1, (Nu, 1)) + r.uniform(0, 0.05, (Nu, Nphi))
    u = 0.1 * np.sin(j)[None] + r.uniform(-0.05, 0.05, (Nu, Nphi))
    w = 0.8 + 0.2 * np.cos(j + 1)[None] + r.uniform(0, 0.1, (Nu, Nphi))
    dk.Sig, dk.vR, dk.vp = S.copy(), u.copy(), w.copy()
    dt = 1e-3
    dk.step(dt)
    got = [dk.Sig, dk.vR, dk.vp]
    args = (dt, 0.25, gamma, 0.6, dk.R, dk.Rf, dk.dphi)
    want = step(LD, lambda a, b, c: a * b + c, *(a.astype(LD) for a in (S, u, w)), *args)
    once = step(np.float64, lambda a, b, c: (np.asarray(a, LD) * b + c).astype(np.float64), S, u, w, *args)
    for g, o, e in zip(got, once, want):
        rms = [float(np.sqrt(np.mean((x.astype(LD) - e) ** 2))) for x in (g, o)]
        assert rms[0] <= 1.02 * rms[1], rms


CHILD = r"""
import ctypes as C, json
import numpy as np
L = D.lib()
L.fake_copy.restype = C.POINTER(C.c_double)
Nu, Nphi, G = json.loads(arg)
p = D.default_params(Nu=Nu, Nphi=Nphi, G=G)
h = C.c_void_p()
assert L.dg_create(C.byref(p), C.byref(h)) == 0
R, Rf, Vol = np.empty(Nu), np.empty(Nu + 1), np.empty(Nu)
L.dg_grid(h, D._dp(R), D._dp(Rf), D._dp(Vol))
n, copies = C.c_longlong(), []
for k in range(L.fake_copies()):
    q = L.fake_copy(k, C.byref(n))
    if n.value == Nu:
        copies.append(np.ctypeslib.as_array(q, (Nu,)).astype(np.longdouble))
LD, du, dphi = np.longdouble, (np.log(1.0) - np.log(0.25)) / Nu, 2.0 * np.pi / Nphi
r = R.astype(LD)
worst = []
for want in (r * np.sqrt(r), -LD(G) * LD(du) * LD(dphi) / (LD(2 * Nu) * LD(Nphi)) / np.sqrt(r)):
    ulp = np.spacing(abs(want).astype(np.float64)).astype(LD)
    worst.append(min(float(np.max(abs(c - want) / ulp)) for c in copies))
print(json.dumps(worst))
"""


@pytest.mark.parametrize("Nu,Nphi,G", [(512, 512, 1.0), (240, 180, 1.0), (300, 64, 0.7)])
def test_row_factors_of_the_gravity_are_rounded_once(fake_lib, Nu, Nphi, G):
    """What a row is multiplied by before and after the transforms, R^{3/2} and
    -G du dphi / (M Nphi sqrt(R)), errs alike in every step.  Each is the nearest double to the
    80-bit value (half a unit in the last place, and what 80 bits leave of it)."""
    for w in fake_child(fake_lib, CHILD, [Nu, Nphi, G]):
        assert w <= 0.5 + 2.0 ** -9
