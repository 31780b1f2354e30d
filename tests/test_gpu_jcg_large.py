"""FP64 meshes beyond the resident kernel's 639,360 rows.

They are solved by the kernel with two row blocks an SM and block-local
tables (jcg_ordered.cu) up to about a million rows, not by jcg_kernel, which
takes up to twice its time there.  adc_jcg_layout tells the two apart; the
step is compared with the oracle as in test_gpu_parity, and adc_jcg, which
starts from the caller's ITPACK scalars and forms peror's norms, with the
oracle's jcg.
"""
import ctypes as C

import numpy as np
import pytest

from test_gpu_jcg_layouts import REL_TOL, _system
from test_gpu_parity import _check, _pair

pytestmark = pytest.mark.gpu


def _case(nx, ny, **k):
    from adcirc_b200 import meshgen, model
    raw = meshgen.channel_mesh(nx=nx, ny=ny, lx=100.0 * nx, ly=100.0 * ny, depth0=6.0, depth1=-0.5)
    eta0 = np.where(raw.dp > 0.05, np.random.default_rng(7).uniform(-0.2, 0.4, raw.dp.size), 0.0)
    tides = [(1e-3, 0.0, 1.0, np.full(raw.open_nodes.size, 0.5), np.zeros(raw.open_nodes.size))]
    return model.build_case(raw, model.default_params(1.0), model.Schedule(dt=1.0, nramp=0), tides,
                            eta0=eta0, **k)


@pytest.mark.parametrize("nx,ny,tables", [(2131, 300, 1), (2200, 301, 1), (2300, 310, 1)])
def test_layout(lib, nx, ny, tables):
    from adcirc_b200 import model
    gpu = model.GpuModel(_case(nx, ny))
    rb, res = C.c_int(-1), C.c_int(-1)
    assert lib.adc_jcg_layout(gpu.h, C.byref(rb), C.byref(res)) == 0
    gpu.close()
    assert res.value == tables, (nx * ny, rb.value)


def test_steps_against_oracle(lib, orc):
    c0, cg, io, ig = _pair(lambda **k: _case(2200, 301, **k), 6, use_run=True)
    _check(c0, cg, io, ig)
    assert 0 < (cg.arrays["nodecode"] == 0).sum() < cg.sizes["np"]


@pytest.mark.parametrize("n,tol", [(645_001, 1e-10), (700_003, 1e-5)])
def test_dropin_digits(lib, orc, n, tol):
    """digit1 and digit2 are logarithms of the stopping test and of the
    residual; solutions agreeing to 1e-13 change a residual of 1e-10 by
    1e-3 of itself, a digit by 1e-2 at most."""
    import oracle
    from adcirc_b200._lib import dp_, ip_, ptr
    o = oracle.load()
    maxnz, jc, cf, rhs, u0 = _system(n, n)
    got = []
    for jcg, dfault, reset in ((lib.adc_jcg, lib.adc_dfault, lib.adc_jcg_reset),
                               (o.orc_jcg, o.orc_dfault, o.orc_itpack_reset)):
        reset()
        j, c, r, u = jc.copy(order="F"), cf.copy(order="F"), rhs.copy(), u0.copy()
        iparm, rparm = np.zeros(12, np.int32), np.zeros(12)
        dfault(ptr(iparm, ip_), ptr(rparm, dp_))
        iparm[0], rparm[0] = 200, tol
        nw = 4 * n + 800
        wksp, iwksp, ier = np.zeros(nw), np.zeros(3 * n, np.int32), C.c_int(-1)
        jcg(C.byref(C.c_int(n)), C.byref(C.c_int(n)), C.byref(C.c_int(maxnz)), ptr(j, ip_), ptr(c, dp_),
            ptr(r, dp_), ptr(u, dp_), ptr(iwksp, ip_), C.byref(C.c_int(nw)), ptr(wksp, dp_),
            ptr(iparm, ip_), ptr(rparm, dp_), C.byref(ier))
        got.append((ier.value, iparm, rparm, u, r, c))
    g, w = got
    assert g[0] == w[0] == 0 and np.array_equal(g[1], w[1])
    assert np.abs(g[2][10:] - w[2][10:]).max() <= 1e-2, (g[2], w[2])
    assert np.abs(g[3] - w[3]).max() <= REL_TOL * np.abs(w[3]).max()
    assert np.abs(g[4] - w[4]).max() <= REL_TOL * np.abs(w[4]).max()
    assert np.abs(g[5] - w[5]).max() <= 1e-14 * np.abs(w[5]).max()
