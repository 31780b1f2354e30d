"""The resident JCG kernel's launch shapes where shared memory runs out.

Its instances of one and two slices per warp keep a row's first eight slots
in registers and read further ones from shared memory, so every slice wider
than eight slots must be resident there.  ITMAX takes 32 bytes of shared
memory an iteration, and a block of wide rows takes more than its share.  The
planner is checked on the host (148 SMs of 227 KB, a B200); the same systems
solved on the device agree with the oracle to 1e-9, the tolerance of the
other JCG parity tests, with the same iteration counts.
"""
import ctypes as C

import numpy as np
import pytest

SMS, SMEM = 148, 227 * 1024 - 1024   # less the kernel's static part


def _band(n, near, lo=0, hi=0, far=0):
    """Columns and lengths of a symmetric band |i - j| <= near, widened to
    <= far between the rows lo..hi-1; slots in column order."""
    m = max(near, far)
    d = np.concatenate([np.arange(-m, 0), np.arange(1, m + 1)])
    j = np.arange(n)[:, None] + d[None, :]
    i = np.arange(n)[:, None]
    ok = (j >= 0) & (j < n) & ((np.abs(d) <= near)[None, :] |
                               ((i >= lo) & (i < hi) & (j >= lo) & (j < hi)))
    o = np.argsort(~ok, axis=1, kind="stable")
    rlen = ok.sum(1).astype(np.int32)
    w = int(rlen.max())
    return np.take_along_axis(j, o, 1)[:, :w].astype(np.int32), rlen


def _shape(lib, cols, rlen, itmax, blocks=0):
    from adcirc_b200._lib import ip_, ptr
    n, w = cols.shape
    nsl = (n + 31) // 32
    full = np.zeros((nsl * 32, w), np.int32)
    full[:n] = cols
    ln = np.zeros(nsl * 32, np.int32)
    ln[:n] = rlen
    sl_w = ln.reshape(nsl, 32).max(1).astype(np.int32)
    sl_ptr = np.concatenate([[0], np.cumsum(32 * sl_w)]).astype(np.int32)
    col = np.concatenate([full[32 * s:32 * s + 32, :sl_w[s]].T.ravel() for s in range(nsl)]).astype(np.int32)
    out = np.zeros(4, np.int32)
    assert lib.adc_selftest_jcg_shape(n, ptr(sl_ptr, ip_), ptr(sl_w, ip_), ptr(col, ip_), ptr(ln, ip_),
                                      itmax, blocks, SMS, SMEM, ptr(out, ip_)) == 0
    return dict(zip(("form", "k", "loose", "misread"), out.tolist()))


# (rows, band, wide rows lo..hi, their band, ITMAX)
TIGHT = [
    (140_000, 6, 0, 0, 0, 1900), (140_000, 6, 0, 0, 0, 2000), (140_000, 6, 0, 0, 0, 2130),
    (140_001, 3, 30 * 32 * 5, 30 * 32 * 5 + 18 * 32, 14, 200),
    (140_000, 3, 0, 18 * 32, 14, 200),
]


@pytest.mark.parametrize("n,near,lo,hi,far,itmax", TIGHT)
def test_wide_slices_are_resident_or_staged(lib, n, near, lo, hi, far, itmax):
    s = _shape(lib, *_band(n, near, lo, hi, far), itmax)
    assert s["misread"] == 0, s
    assert s["form"] == 1 and s["loose"] > 0, s   # shared memory did run out


@pytest.mark.parametrize("n,near,itmax,k,loose", [
    (140_000, 3, 200, 2, 0), (140_000, 3, 2900, 2, None), (71_040, 3, 200, 1, 0), (71_040, 6, 1000, 1, 0)])
def test_narrow_or_resident_slices_keep_their_instance(lib, n, near, itmax, k, loose):
    s = _shape(lib, *_band(n, near), itmax)
    assert (s["form"], s["k"], s["misread"]) == (1, k, 0), s
    assert loose is None or s["loose"] == loose, s


@pytest.mark.gpu
@pytest.mark.parametrize("n,near,lo,hi,far,itmax", TIGHT)
def test_tight_shapes_solve(lib, n, near, lo, hi, far, itmax):
    import oracle
    from adcirc_b200._lib import dp_, ip_, ptr
    orc = oracle.load()
    cols, rlen = _band(n, near, lo, hi, far)
    rng = np.random.default_rng(n + itmax)
    i = np.arange(n)[:, None]
    # symmetric values from the pair, a dominant diagonal
    a, b = np.minimum(cols, i).astype(np.int64), np.maximum(cols, i).astype(np.int64)
    v = ((a * 7919 + b * 104729) % 1009) / 1009.0 * 0.6 - 0.2
    v[np.arange(cols.shape[1])[None, :] >= rlen[:, None]] = 0.0
    maxnz = cols.shape[1] + 1
    jcoef = np.zeros((n, maxnz), np.int32, order="F")
    coef = np.zeros((n, maxnz), order="F")
    jcoef[:, 0] = np.arange(1, n + 1)
    coef[:, 0] = 0.5 + np.abs(v).sum(1) * rng.uniform(1.05, 1.3, n)
    jcoef[:, 1:] = np.where(v != 0.0, cols + 1, 0)
    coef[:, 1:] = v
    rhs, u0 = rng.standard_normal(n), 1e-2 * rng.standard_normal(n)
    got = []
    for jcg, dfault, reset in ((lib.adc_jcg, lib.adc_dfault, lib.adc_jcg_reset),
                               (orc.orc_jcg, orc.orc_dfault, orc.orc_itpack_reset)):
        reset()
        j, c, r, u = jcoef.copy(order="F"), coef.copy(order="F"), rhs.copy(), u0.copy()
        iparm, rparm = np.zeros(12, np.int32), np.zeros(12)
        dfault(ptr(iparm, ip_), ptr(rparm, dp_))
        iparm[0], rparm[0] = itmax, 1e-10
        nw = 4 * n + 4 * itmax
        wksp, iwksp, ier = np.zeros(nw), np.zeros(3 * n, np.int32), C.c_int(-1)
        jcg(C.byref(C.c_int(n)), C.byref(C.c_int(n)), C.byref(C.c_int(maxnz)), ptr(j, ip_), ptr(c, dp_),
            ptr(r, dp_), ptr(u, dp_), ptr(iwksp, ip_), C.byref(C.c_int(nw)), ptr(wksp, dp_),
            ptr(iparm, ip_), ptr(rparm, dp_), C.byref(ier))
        got.append((ier.value, int(iparm[0]), u, c))
    (ie, it, u, c), (ie2, it2, u2, c2) = got
    assert (ie, it) == (ie2, it2)
    assert np.abs(u - u2).max() <= 1e-9 * np.abs(u2).max()
    assert np.abs(c - c2).max() <= 1e-14 * np.abs(c2).max()


@pytest.mark.gpu
def test_staged_slices_of_uneven_width(lib):
    """Blocks of 4,320 rows (nine slices a warp, most of them streamed).  In
    each, a warp's first slice has rows of 12 neighbours, the last of them the
    block's row 4,094 or 4,095, whose column word 0x7ff0 or 0x7ff8 is the top
    of a double that is no number; the third has rows of one neighbour, so
    that its buffer still holds words of the first past its own end."""
    import oracle
    from adcirc_b200._lib import dp_, ip_, ptr
    orc = oracle.load()
    per = 15 * 9 * 32
    n = SMS * per
    i = np.arange(n)
    local = i % per
    k = local // 32 // 15
    cols = np.zeros((n, 12), np.int64)
    use = np.zeros((n, 12), bool)
    for q in range(11):
        cols[:, q] = i ^ (q + 1)
        use[:, q] = (k == 0) | (q == 0) | ((q == 1) & (k != 2))
    cols[:, 11] = i - local + 4094 + i % 2
    use[:, 11] = k == 0
    v = np.where(use, 0.05 + 0.3 * ((np.minimum(cols, i[:, None]) * 7919) % 1009) / 1009.0, 0.0)
    v[:, 11] *= 1e-6
    rng = np.random.default_rng(12)
    jcoef = np.zeros((n, 13), np.int32, order="F")
    coef = np.zeros((n, 13), order="F")
    jcoef[:, 0] = i + 1
    coef[:, 0] = 0.5 + np.abs(v).sum(1) * rng.uniform(1.05, 1.3, n)
    jcoef[:, 1:] = np.where(use, cols + 1, 0)
    coef[:, 1:] = v
    rhs, u0 = rng.standard_normal(n), 1e-2 * rng.standard_normal(n)
    got = []
    for jcg, dfault, reset in ((lib.adc_jcg, lib.adc_dfault, lib.adc_jcg_reset),
                               (orc.orc_jcg, orc.orc_dfault, orc.orc_itpack_reset)):
        reset()
        j, c, r, u = jcoef.copy(order="F"), coef.copy(order="F"), rhs.copy(), u0.copy()
        iparm, rparm = np.zeros(12, np.int32), np.zeros(12)
        dfault(ptr(iparm, ip_), ptr(rparm, dp_))
        iparm[0], rparm[0] = 200, 1e-8
        nw = 4 * n + 800
        wksp, iwksp, ier = np.zeros(nw), np.zeros(3 * n, np.int32), C.c_int(-1)
        jcg(C.byref(C.c_int(n)), C.byref(C.c_int(n)), C.byref(C.c_int(13)), ptr(j, ip_), ptr(c, dp_),
            ptr(r, dp_), ptr(u, dp_), ptr(iwksp, ip_), C.byref(C.c_int(nw)), ptr(wksp, dp_),
            ptr(iparm, ip_), ptr(rparm, dp_), C.byref(ier))
        got.append((ier.value, int(iparm[0]), u))
    (ie, it, u), (ie2, it2, u2) = got
    assert (ie, it) == (ie2, it2)
    assert np.abs(u - u2).max() <= 1e-9 * np.abs(u2).max()
