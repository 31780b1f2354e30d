"""The fused step against the four phase calls.

adc_run and adc_timestep fold passes that the phase calls keep apart: D1 of
the wet/dry pass into the solve, ALPHAL into the momentum terms, the step's
bookkeeping into the last kernel.  The same operations in the same order on
the same values must leave every array the same, bit for bit.  The meshes
have a node count below one block, one that no block size divides, and
drying fronts; the modes reach each solver kernel.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(name):
    from adcirc_b200 import meshgen, model
    if name == "channel+vortex":
        return model.channel_case(vortex=True)
    if name == "beach":
        return model.beach_case()
    nx, ny = {"small": (13, 7), "ragged": (83, 61)}[name]
    raw = meshgen.channel_mesh(nx=nx, ny=ny, lx=100.0 * nx, ly=100.0 * ny, depth0=3.0, depth1=-1.5)
    eta0 = np.where(raw.dp > 0.05, np.random.default_rng(3).uniform(-0.4, 0.9, raw.dp.size), 0.0)
    tides = [(1e-3, 0.0, 1.0, np.full(raw.open_nodes.size, 0.5), np.zeros(raw.open_nodes.size))]
    return model.build_case(raw, model.default_params(0.5), model.Schedule(dt=0.5, nramp=0), tides, eta0=eta0)


@pytest.mark.parametrize("prec", [0, 1, 18])
@pytest.mark.parametrize("name", ["small", "ragged", "beach", "channel+vortex"])
def test_run_equals_phases(lib, name, prec):
    from adcirc_b200 import _lib, model
    n, out = 60, []
    for phases in (False, True):
        case = _case(name)
        gpu = model.GpuModel(case, prec)
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
    assert sa["ncchange"] == sb["ncchange"] and sa["ep"] == sb["ep"]
    if name in ("ragged", "beach"):
        assert 0 < (a["nodecode"] == 0).sum() < a["nodecode"].size
