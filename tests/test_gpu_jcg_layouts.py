"""The JCG kernels' launch shapes against the oracle's jcg.

adc_jcg chooses a layout by the number of rows: one cluster of 1 to 16
blocks with one or two 32-row slices per warp, the whole grid with one to
nine, parts of the matrix in registers, in shared memory or streamed, and
jcg_kernel beyond.  Each size below sits at an edge of that choice or of a
tile; `wide` gives some rows more neighbours than one group of eight slots
holds, `huge` some more than a staging buffer.  Solutions agree with the
oracle to 1e-9 (the tolerance of the other JCG parity tests), iteration
counts exactly, and a second call (drifted COEF, saved q1) does too.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL_TOL = 1e-9


def _system(n, seed, wide=0, huge=0):
    """A symmetric matrix with a dominant diagonal: a ring of +-1, +-2, +-41
    neighbours (fewer at the ends), and `wide`/`huge` rows with 4 to 30 more."""
    rng = np.random.default_rng(seed)
    pairs = []
    for d in (1, 2, 41):
        i = np.arange(max(n - d, 0))
        pairs.append(np.stack([i, i + d]))
    for k, cnt in ((4, wide), (30, huge)):
        for r in rng.choice(n, min(cnt, n), replace=False) if cnt else ():
            j = np.unique(rng.integers(0, n, k))
            j = j[(np.abs(j - r) > 2) & (np.abs(j - r) != 41)]
            pairs.append(np.stack([np.minimum(j, r), np.maximum(j, r)]))
    p = np.unique(np.concatenate(pairs, axis=1), axis=1)
    v = rng.uniform(-0.2, 0.4, p.shape[1])
    row = np.concatenate([p[0], p[1]])
    col = np.concatenate([p[1], p[0]])
    val = np.concatenate([v, v])
    o = np.lexsort((col, row))
    row, col, val = row[o], col[o], val[o]
    start = np.searchsorted(row, np.arange(n))
    slot = np.arange(row.size) - start[row]
    maxnz = int(slot.max(initial=0)) + 2
    jcoef = np.zeros((n, maxnz), np.int32, order="F")
    coef = np.zeros((n, maxnz), order="F")
    jcoef[:, 0] = np.arange(1, n + 1)
    coef[:, 0] = 0.5 + np.bincount(row, np.abs(val), n) * rng.uniform(1.05, 1.3, n)
    jcoef[row, slot + 1] = col + 1
    coef[row, slot + 1] = val
    return maxnz, jcoef, coef, rng.standard_normal(n), 1e-2 * rng.standard_normal(n)


def _solve(jcg, dfault, n, maxnz, jcoef, coef, rhs, u):
    from adcirc_b200._lib import dp_, ip_, ptr
    iparm, rparm = np.zeros(12, np.int32), np.zeros(12)
    dfault(ptr(iparm, ip_), ptr(rparm, dp_))
    iparm[0], rparm[0] = 200, 1e-10
    nw = 4 * n + 4 * 200
    wksp, iwksp, ier = np.zeros(nw + 16), np.zeros(3 * n, np.int32), C.c_int(-1)
    jcg(C.byref(C.c_int(n)), C.byref(C.c_int(n)), C.byref(C.c_int(maxnz)), ptr(jcoef, ip_),
        ptr(coef, dp_), ptr(rhs, dp_), ptr(u, dp_), ptr(iwksp, ip_), C.byref(C.c_int(nw)),
        ptr(wksp, dp_), ptr(iparm, ip_), ptr(rparm, dp_), C.byref(ier))
    return ier.value, int(iparm[0])


@pytest.mark.parametrize("n,wide,huge", [
    (1, 0, 0), (31, 0, 0), (33, 0, 0), (480, 5, 0), (481, 0, 0), (7_680, 40, 6), (7_681, 0, 0),
    (15_360, 30, 0), (15_361, 30, 0), (71_040, 0, 0), (71_041, 100, 10), (150_001, 200, 0),
    (300_007, 0, 20), (430_003, 300, 40), (639_360, 2000, 60), (645_001, 0, 0)])
def test_layouts(n, wide, huge):
    import oracle
    from adcirc_b200 import _lib
    lib, orc = _lib.load(), oracle.load()
    maxnz, jc, cf, rhs, u0 = _system(n, n, wide, huge)
    state = {}
    for name, jcg, dfault, reset in (("gpu", lib.adc_jcg, lib.adc_dfault, lib.adc_jcg_reset),
                                     ("oracle", orc.orc_jcg, orc.orc_dfault, orc.orc_itpack_reset)):
        reset()
        j, c, got = jc.copy(order="F"), cf.copy(order="F"), []
        for _ in range(2):
            r, u = rhs.copy(), u0.copy()
            ier, its = _solve(jcg, dfault, n, maxnz, j, c, r, u)
            got.append((ier, its, u, r))
        state[name] = (got, c, j)
    (g, cg, jg), (o, co, jo) = state["gpu"], state["oracle"]
    for (ie, it, u, r), (ie2, it2, u2, r2) in zip(g, o):
        assert (ie, it) == (ie2, it2)
        assert np.abs(u - u2).max() <= REL_TOL * np.abs(u2).max()
        assert np.abs(r - r2).max() <= REL_TOL * np.abs(r2).max()
    assert np.array_equal(jg, jo)
    assert np.abs(cg - co).max() <= 1e-14 * np.abs(co).max()


@pytest.mark.parametrize("n,pad", [(1, 3), (33, 1), (500, 7), (20_001, 31)])
def test_padded_columns(n, pad):
    """COEF with NDIM > N and a column of empty slots: the solution, the
    drifted COEF and its untouched parts as the oracle leaves them (COEF to
    1e-13, as in the other drop-in tests)."""
    import oracle
    from adcirc_b200 import _lib
    lib, orc = _lib.load(), oracle.load()
    from adcirc_b200._lib import dp_, ip_, ptr
    maxnz, jc, cf, rhs, u0 = _system(n, n + 1)
    ndim, maxnz = n + pad, maxnz + 1
    jcoef = np.full((ndim, maxnz), 9, np.int32, order="F")
    coef = np.full((ndim, maxnz), 7.5, order="F")
    jcoef[:n], coef[:n] = 0, 0.0
    jcoef[:n, :-1], coef[:n, :-1] = jc, cf
    got = []
    for jcg, dfault, reset in ((lib.adc_jcg, lib.adc_dfault, lib.adc_jcg_reset),
                               (orc.orc_jcg, orc.orc_dfault, orc.orc_itpack_reset)):
        reset()
        j, c, r, u = jcoef.copy(order="F"), coef.copy(order="F"), rhs.copy(), u0.copy()
        iparm, rparm = np.zeros(12, np.int32), np.zeros(12)
        dfault(ptr(iparm, ip_), ptr(rparm, dp_))
        iparm[0], rparm[0] = 200, 1e-10
        nw = 4 * n + 4 * 200
        wksp, iwksp, ier = np.zeros(nw + 16), np.zeros(3 * n, np.int32), C.c_int(-1)
        jcg(C.byref(C.c_int(n)), C.byref(C.c_int(ndim)), C.byref(C.c_int(maxnz)), ptr(j, ip_), ptr(c, dp_),
            ptr(r, dp_), ptr(u, dp_), ptr(iwksp, ip_), C.byref(C.c_int(nw)), ptr(wksp, dp_),
            ptr(iparm, ip_), ptr(rparm, dp_), C.byref(ier))
        got.append((ier.value, iparm[0], j, c, r, u))
    g, o = got
    assert g[:2] == o[:2]
    assert np.array_equal(g[2], o[2]) and np.array_equal(g[3][n:], coef[n:])
    assert np.abs(g[3] - o[3]).max() <= 1e-13 * np.abs(o[3]).max()
    assert np.abs(g[4] - o[4]).max() <= 1e-13 * max(np.abs(o[4]).max(), 1e-30)
    assert np.abs(g[5] - o[5]).max() <= REL_TOL * max(np.abs(o[5]).max(), 1e-30)
