"""The FP32 column solve's arithmetic (column_finish, shoc_tr_tile.cuh) as FP32_COMP
takes it, restated in numpy: its first solve is no further from the 64-bit one than the Thomas solve with
FP64 factors rounded once (the lower diagonal, 1 / div and the elimination factor
cm1 / div), where a factor made of two rounded ones is; after the FP64 residual and
the correction, eliminated from the top, the error is that of the FP32 diffusivity.
"""
import numpy as np
import pytest

f4 = np.float32


def fma(a, b, c):  # one rounding (48-bit products are exact in FP64)
    return (a.astype(float) * b + c).astype(f4)


def column(nk, ncol, thin, kz, rng, dt=60.0):
    dz = np.full((nk, ncol), 5.0)
    if thin:
        dz[:] = np.geomspace(20.0, 0.5, nk)[:, None]
    dz *= rng.uniform(0.9, 1.1, (1, ncol))
    K = np.exp(rng.uniform(*np.log(kz), (nk, ncol)))
    cm = np.zeros((nk, ncol))
    cm[1:] = -K[1:] / (0.5 * (dz[1:] + dz[:-1]))
    cp = np.vstack([cm[1:], np.zeros((1, ncol))])
    return dz / dt, cm, dz / dt - cm - cp, np.exp(rng.normal(size=(nk, ncol))).astype(f4)


def solve64(dzdt, cm, C, a):
    div, e, x = C.copy(), C.copy(), dzdt * a
    for k in range(1, len(C)):
        div[k] -= cm[k] * (cm[k] / div[k - 1])
        x[k] -= cm[k] * x[k - 1] / div[k - 1]
    x[-1] /= div[-1]
    for k in range(len(C) - 2, -1, -1):
        x[k] = (x[k] - cm[k + 1] * x[k + 1]) / div[k]
        e[k] -= cm[k + 1] * (cm[k + 1] / e[k + 1])
    return x, div, e


def rms(x, ref):
    return np.sqrt((((x.astype(float) - ref) / ref) ** 2).mean())


@pytest.mark.parametrize("nk", [2, 6, 20, 50, 128])
@pytest.mark.parametrize("thin", [False, True])
@pytest.mark.parametrize("kz", [(1e-6, 1e-1), (1e-2, 1.0)])
def test_first_solve(nk, thin, kz):
    rng = np.random.default_rng(nk)
    dzdt, cm, C, a = column(nk, 4000, thin, kz, rng)
    X, div, e = solve64(dzdt, cm, C, a)
    ud64 = np.zeros_like(cm)
    ud64[1:] = cm[1:] / div[:-1]
    b, m, rd, ud = (dzdt.astype(f4) * a), cm.astype(f4), (1 / div).astype(f4), ud64.astype(f4)
    # Thomas, every factor rounded once: s = (b - cm1 s) / div, x = s - ud x
    s = np.zeros_like(b)
    s[0] = b[0] * rd[0]
    # the kernel: z = b - ud z, s = z / div, x = s - ud x
    z = b.copy()
    for k in range(1, nk):
        s[k] = fma(-m[k], s[k - 1], b[k]) * rd[k]
        z[k] = fma(-ud[k], z[k - 1], b[k])
    x, t = z * rd, s.copy()
    for k in range(nk - 2, -1, -1):
        t[k] = fma(-ud[k + 1], t[k + 1], s[k])
        x[k] = fma(-ud[k + 1], x[k + 1], x[k])
    assert rms(x, X) <= 1.002 * rms(t, X)
    # the correction: h = r - cm1 (h / e) downwards, d = (h - cm1 d) / e upwards
    re = (1 / e).astype(f4)
    m64, xd = m.astype(float), x.astype(float)
    r = dzdt * (a - xd)
    r[1:] -= m64[1:] * (xd[:-1] - xd[1:])
    r[:-1] -= m64[1:] * (xd[1:] - xd[:-1])
    h = r.astype(f4)
    for k in range(nk - 2, -1, -1):
        h[k] = fma(-m[k + 1], h[k + 1] * re[k + 1], h[k])
    d = h * re
    for k in range(1, nk):
        d[k] = fma(-m[k], d[k - 1], h[k]) * re[k]
    # what is left is the rounding of cm1 (2^-24) acting on the solution's gradients,
    # of which a row has two, and of the correction itself
    fin = xd + d
    assert rms(fin, X) <= 2.0 ** -24 and rms(fin, X) < 0.3 * rms(x, X)
