"""The adaptive eigenvalue estimate on ill-conditioned systems.

ITPACK's stopping test divides by 1 - cme, and cme is the last point of
zbrent's search, which its tolerance 10^-max(4, -log10(zeta)) leaves beside
the eigenvalue.  Where cme is close to 1 that place decides when a solve
stops, so the iteration counts must be the oracle's (sequential sums, its own
zbrent), and the estimate returned in RPARM(2) agrees to 1e-12.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ZETAS = (1e-2, 1e-3, 1e-4, 5e-6, 1e-7, 1e-10)


def _laplacian(nx, ny, eps, seed):
    """A 5-point operator with random couplings; eps is the excess of its
    diagonal: the smaller, the closer cme is to 1."""
    rng = np.random.default_rng(seed)
    n = nx * ny
    idx = np.arange(n).reshape(nx, ny)
    p = np.concatenate([np.stack([idx[:-1].ravel(), idx[1:].ravel()]),
                        np.stack([idx[:, :-1].ravel(), idx[:, 1:].ravel()])], axis=1)
    v = -rng.uniform(0.3, 1.0, p.shape[1])
    row, col, val = np.concatenate([p[0], p[1]]), np.concatenate([p[1], p[0]]), np.concatenate([v, v])
    o = np.lexsort((col, row))
    row, col, val = row[o], col[o], val[o]
    slot = np.arange(row.size) - np.searchsorted(row, np.arange(n))[row]
    maxnz = int(slot.max()) + 2
    jcoef = np.zeros((n, maxnz), np.int32, order="F")
    coef = np.zeros((n, maxnz), order="F")
    jcoef[:, 0] = np.arange(1, n + 1)
    coef[:, 0] = np.bincount(row, np.abs(val), n) * (1.0 + eps * rng.uniform(0.2, 1.0, n))
    jcoef[row, slot + 1] = col + 1
    coef[row, slot + 1] = val
    return n, maxnz, jcoef, coef, rng.standard_normal(n)


def _solve(fns, n, maxnz, jcoef, coef, rhs, zeta, itmax=400):
    from adcirc_b200._lib import dp_, ip_, ptr
    jcg, dfault, reset = fns
    reset()
    j, c, r, u = jcoef.copy(order="F"), coef.copy(order="F"), rhs.copy(), np.zeros(n)
    iparm, rparm = np.zeros(12, np.int32), np.zeros(12)
    dfault(ptr(iparm, ip_), ptr(rparm, dp_))
    iparm[0], rparm[0] = itmax, zeta
    nw = 4 * n + 4 * itmax
    wksp, iwksp, ier = np.zeros(nw), np.zeros(3 * n, np.int32), C.c_int(-1)
    jcg(C.byref(C.c_int(n)), C.byref(C.c_int(n)), C.byref(C.c_int(maxnz)), ptr(j, ip_), ptr(c, dp_),
        ptr(r, dp_), ptr(u, dp_), ptr(iwksp, ip_), C.byref(C.c_int(nw)), ptr(wksp, dp_),
        ptr(iparm, ip_), ptr(rparm, dp_), C.byref(ier))
    return ier.value, int(iparm[0]), float(rparm[1])


@pytest.mark.parametrize("nx,ny,zetas", [(10, 10, ZETAS), (26, 27, ZETAS), (54, 55, ZETAS), (170, 173, ZETAS),
                                         (806, 803, (1e-3, 5e-6))])   # cluster, grid, two blocks an SM
@pytest.mark.parametrize("eps", [1.0, 1e-1, 1e-2, 1e-3])
def test_iterations_and_estimate(lib, nx, ny, zetas, eps):
    import oracle
    orc = oracle.load()
    bad = []
    for seed in range(3 if nx < 100 else 1):
        sysargs = _laplacian(nx, ny, eps, 1000 * seed + nx)
        for zeta in zetas:
            g = _solve((lib.adc_jcg, lib.adc_dfault, lib.adc_jcg_reset), *sysargs, zeta)
            o = _solve((orc.orc_jcg, orc.orc_dfault, orc.orc_itpack_reset), *sysargs, zeta)
            if g[:2] != o[:2] or not abs(g[2] - o[2]) <= 1e-12:
                bad.append((seed, zeta, g, o))
    assert not bad, bad


@pytest.mark.parametrize("nx,eps,zeta", [(3000, 1e-3, 1e-6), (3000, 1e-4, 1e-4), (3000, 1e-6, 1e-6), (8000, 1e-4, 1e-6)])
def test_many_iterations(lib, nx, eps, zeta):
    """475 to 1,400 iterations: the determinants of the CG tridiagonal leave
    the range in which quotients are formed by reciprocals, and ITMAX is met."""
    import oracle
    orc = oracle.load()
    sysargs = _laplacian(nx, 1, eps, 5)
    g = _solve((lib.adc_jcg, lib.adc_dfault, lib.adc_jcg_reset), *sysargs, zeta, itmax=1400)
    o = _solve((orc.orc_jcg, orc.orc_dfault, orc.orc_itpack_reset), *sysargs, zeta, itmax=1400)
    assert g[:2] == o[:2] and o[1] >= 400
    assert abs(g[2] - o[2]) <= 1e-12


def test_estimate_of_steps(lib, orc, tmp_path):
    """The estimate that adc_timestep, adc_gwce_new, adc_run, adc_get_scalars
    and a dump report is the oracle's of the same solve, though the solve has
    stopped by bounds of it; after a dump is read back too."""
    import ctypes as C

    from adcirc_b200 import _lib, model
    case0, case = model.channel_case(prep=orc.mesh_prep()), model.channel_case()
    om, gm = orc.OracleModel(case0), model.GpuModel(case)
    want = [om.step(it).cme for it in range(1, 13)]

    def same(x, y):
        return abs(x - y) <= 1e-12 * max(abs(y), 1.0)

    for it in range(1, 5):
        assert same(gm.step(it).cme, want[it - 1]), it
        assert same(gm.scalars()["rparm2"], want[it - 1]), it
    out = _lib.AdcStepOut()
    for it in (5, 6):
        s = C.byref(case.schedule.step(it))
        assert lib.adc_shift_friction(gm.h, s) == 0
        assert lib.adc_gwce_new(gm.h, s, C.byref(out)) == 0
        assert same(out.cme, want[it - 1]), it
        assert lib.adc_wetdry(gm.h, s, C.byref(out)) == 0
        assert same(out.cme, want[it - 1]), it
        assert lib.adc_momentum(gm.h, s) == 0
    _, last = gm.run(7, 3)
    assert same(last.cme, want[8])
    gm.hotstart_write(tmp_path / "a")
    gm.run(10, 3)
    assert same(gm.scalars()["rparm2"], want[11])
    gm.hotstart_read(tmp_path / "a")
    assert same(gm.scalars()["rparm2"], want[8])
    gm.hotstart_write(tmp_path / "b")
    assert (tmp_path / "a").read_bytes() == (tmp_path / "b").read_bytes()
    gm.close()
    om.close()
