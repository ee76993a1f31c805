"""The mixed-precision streamfunction solve equals, bit for bit, its plain
restatement here: FP64 defect correction around FP32 zebra line relaxation with
every line eliminated row after row, each operation rounded to FP32 (numpy).
The lanes that share a line on the device (warpline.cuh) must not show in the
result, whichever number of lanes and rows a lane a line's length selects.

Grids n = 4 k + 2 have one level, so a cycle is nrel relaxations.  Both sides
do the same IEEE operations, so the comparison has no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def _tdma(a, b, c, n):
    """Pivots and multipliers in FP64, as the tables keep them in FP32: F, 1/b', c."""
    fact, bp = np.zeros(n), np.zeros(n)
    bp[0] = b[0]
    for k in range(1, n):
        fact[k] = a[k] / bp[k - 1]
        bp[k] = b[k] - fact[k] * c[k - 1]
    return fact.astype(F), (1.0 / bp).astype(F), np.asarray(c).astype(F)


def _lines(tab, x):
    """x[line, row] in place; tab's arrays [row] or [row, line]."""
    fact, ib, c = tab
    n = x.shape[1]
    for k in range(1, n):
        x[:, k] = x[:, k] - fact[k] * x[:, k - 1]
    x[:, n - 1] = x[:, n - 1] * ib[n - 1]
    for k in range(n - 2, -1, -1):
        x[:, k] = (x[:, k] - c[k] * x[:, k + 1]) * ib[k]
    return x


def _solve(nr, nz, r0, rmax, zmax, rhs, tol, nrel):
    dr, dz = (rmax - r0) / nr, zmax / nz
    hr, hhr, hhz = dr, dr * dr, dz * dz
    rv = np.arange(nr + 1) * hr + r0
    q = rv[1:nr]
    rt = _tdma(1 / hhr - 0.5 / hr / q, -2 / hhr - 2 / hhz - 1 / (q * q), 1 / hhr + 0.5 / hr / q, nr - 1)
    zt = [_tdma(np.full(nz - 1, 1 / hhz), np.full(nz - 1, -2 / hhr - 2 / hhz - 1 / (v * v)), np.full(nz - 1, 1 / hhz), nz - 1) for v in q]
    zt = [np.stack([t[k] for t in zt], axis=1) for k in range(3)]
    drdz = 2 * (1 / hhr + 1 / hhz)
    r32, hr32, hhr32, hhz32 = rv.astype(F), F(hr), F(hhr), F(hhz)
    psi = np.zeros((nr + 1, nz + 1))
    res0 = None
    for cycles in range(50):
        p = psi
        t = (p[2:, 1:-1] + p[:-2, 1:-1]) / hhr + (p[2:, 1:-1] - p[:-2, 1:-1]) * 0.5 / hr / q[:, None] - p[1:-1, 1:-1] / (q * q)[:, None] \
            + (p[1:-1, 2:] + p[1:-1, :-2]) / hhz - p[1:-1, 1:-1] * drdz
        r = rhs[1:-1, 1:-1] - t
        res = np.abs(r).max()
        res0 = res if res0 is None else res0
        if res < tol * res0:
            return psi, cycles, tol * res0
        f = np.zeros((nr + 1, nz + 1), F)
        f[1:-1, 1:-1] = r.astype(F)
        v = np.zeros((nr + 1, nz + 1), F)
        for _ in range(nrel):
            for c in (1, 2):
                j = np.arange(c, nz, 2)
                x = -(v[1:nr][:, j + 1] + v[1:nr][:, j - 1]) / hhz32 + f[1:nr][:, j]
                v[1:nr, j] = _lines(rt, x.T.copy()).T
            for c in (1, 2):
                i = np.arange(c, nr, 2)
                vp, vm = v[i + 1, 1:nz], v[i - 1, 1:nz]
                x = -(vp + vm) / hhr32 + f[i, 1:nz] - (vp - vm) * F(0.5) / r32[i][:, None] / hr32
                v[i, 1:nz] = _lines([t[:, i - 1] for t in zt], x)
        psi = psi + v.astype(np.float64)
    raise AssertionError("no convergence")


# (nr, nz): rows a line n - 1 of 5 .. 33 (4 or 8 lanes), 65 (16), 129 .. 253
# (32 lanes of 8 rows), 257 and more (16 rows a lane); zmax sets how strongly
# a line's rows are coupled: passes run from two to one per lane
@pytest.mark.parametrize("nr,nz,zmax", [(6, 10, 0.5), (34, 66, 0.5), (130, 30, 0.5), (254, 66, 2.0), (66, 258, 0.1), (258, 34, 4.0),
                                        (34, 510, 0.05)])
def test_equals_serial_elimination(gblib, nr, nz, zmax):
    from codesthesis_dir_gb300 import axi
    rng = np.random.default_rng(nr * 1000 + nz)
    rhs = np.zeros((nr + 1, nz + 1))
    rhs[1:-1, 1:-1] = rng.standard_normal((nr - 1, nz - 1))
    want, cycles, tolcon = _solve(nr, nz, 0.5, 1.0, zmax, rhs, 0.7, 2)
    g = axi.AXI(nr, nz, r0=0.5, rmax=1.0, zmax=zmax, tolcon=tolcon, smoother=1, precision=1, nrel=2)
    g.set("omegn", rhs)
    assert g.poisson() == cycles > 0
    np.testing.assert_array_equal(g.get("phi"), want)
    g.close()
