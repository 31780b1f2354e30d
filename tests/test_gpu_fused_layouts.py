"""The fused step against the four phase calls, for every form of the solver
that solves in FP64 and for the split element pass.

As test_gpu_fused_step, on meshes past the cluster form: 20,163 nodes with the
row blocks set so that each grid instance runs (one, two, four, six and nine
slices a warp, the last two with u in memory), and so few that jcg_kernel does
(D1 a launch of its own); 45,933 nodes, whose 91,000 elements are beyond one
wave, so that the element pass is two kernels.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(nx, ny):
    from adcirc_b200 import meshgen, model
    raw = meshgen.channel_mesh(nx=nx, ny=ny, lx=100.0 * nx, ly=100.0 * ny, depth0=3.0, depth1=-1.5)
    eta0 = np.where(raw.dp > 0.05, np.random.default_rng(3).uniform(-0.4, 0.9, raw.dp.size), 0.0)
    tides = [(1e-3, 0.0, 1.0, np.full(raw.open_nodes.size, 0.5), np.zeros(raw.open_nodes.size))]
    return model.build_case(raw, model.default_params(0.5), model.Schedule(dt=0.5, nramp=0), tides, eta0=eta0)


# (nx, ny, row blocks, block-local tables): 631 slices in 43, 22, 11, 7, 5 and 3 blocks of 15 row warps
@pytest.mark.parametrize("nx,ny,blocks,tables", [
    (141, 143, 0, 1), (141, 143, 43, 1), (141, 143, 22, 1), (141, 143, 11, 1), (141, 143, 7, 1),
    (141, 143, 5, 1), (141, 143, 3, 0), (251, 183, 0, 1)])
def test_run_equals_phases(lib, nx, ny, blocks, tables):
    from adcirc_b200 import _lib, model
    n, out = 25, []
    for phases in (False, True):
        case = _case(nx, ny)
        gpu = model.GpuModel(case)
        assert lib.adc_set_jcg_blocks(gpu.h, blocks) == 0
        rb, res = C.c_int(-1), C.c_int(-1)
        assert lib.adc_jcg_layout(gpu.h, C.byref(rb), C.byref(res)) == 0
        assert res.value == tables and (blocks == 0 or rb.value == blocks), (rb.value, res.value)
        if phases:
            o, numitr = _lib.AdcStepOut(), []
            for it in range(1, n + 1):
                s = C.byref(case.schedule.step(it))
                assert lib.adc_shift_friction(gpu.h, s) == 0
                assert lib.adc_gwce_new(gpu.h, s, C.byref(o)) == 0
                numitr.append(o.numitr)
                assert lib.adc_wetdry(gpu.h, s, C.byref(o)) == 0
                assert lib.adc_momentum(gpu.h, s) == 0
        else:
            numitr, _ = gpu.run(1, n)
        gpu.sync_to_host()
        sc = gpu.scalars()
        gpu.close()
        out.append((dict(case.arrays, numitr=np.asarray(numitr)), sc))
    (a, sa), (b, sb) = out
    bad = [k for k in a if not np.array_equal(a[k], b[k])]
    assert not bad, f"arrays differ: {bad}"
    assert sa == sb
    assert 0 < (a["nodecode"] == 0).sum() < a["nodecode"].size
