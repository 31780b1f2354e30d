"""Expired waits inside the solver.

Every wait of the persistent solver kernels is bounded.  With a limit of one
cycle (adc_set_wait_cycles) the first wait that is not over at once expires,
in some blocks before others: the call returns ADC_ERR_TIMEOUT and the device
and the context stay usable.  One case per kernel form: one block, a cluster
with one and two slices a warp, the grid with the matrix resident and
streamed, two blocks an SM in a mode with FP32 parts and in FP64.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = {
    "block": (21, 20, 0), "cluster": (121, 41, 0), "cluster2": (181, 71, 0), "grid": (250, 160, 0),
    "streamed": (1000, 300, 0), "ordered32": (121, 41, 18), "ordered64": (2200, 301, 0),
}


def _case(nx, ny):
    from adcirc_b200 import meshgen, model
    raw = meshgen.channel_mesh(nx=nx, ny=ny, lx=100.0 * nx, ly=100.0 * ny, depth0=6.0, depth1=2.0)
    tides = [(1e-3, 0.0, 1.0, np.full(raw.open_nodes.size, 0.5), np.zeros(raw.open_nodes.size))]
    return model.build_case(raw, model.default_params(1.0), model.Schedule(dt=1.0, nramp=0), tides)


def _run(case, prec, n):
    from adcirc_b200 import model
    gpu = model.GpuModel(case, prec)
    its, _ = gpu.run(1, n)
    gpu.sync_to_host()
    gpu.close()
    return np.asarray(its), {k: v.copy() for k, v in case.arrays.items()}


@pytest.mark.parametrize("form", FORMS)
def test_expired_wait_is_an_error(lib, form):
    from adcirc_b200 import model
    nx, ny, prec = FORMS[form]
    its, want = _run(_case(nx, ny), prec, 6)
    gpu = model.GpuModel(_case(nx, ny), prec)
    gpu.run(1, 3)
    assert lib.adc_set_wait_cycles(gpu.h, 1) == 0
    for call in (lambda: gpu.run(4, 2), lambda: gpu.step(6)):
        with pytest.raises(model.AdcError, match="status -5"):
            call()
    gpu.sync_to_host()
    gpu.close()
    # the device as before, and another context
    its2, got = _run(_case(nx, ny), prec, 6)
    assert np.array_equal(its, its2)
    assert all(np.array_equal(want[k], got[k]) for k in want)


@pytest.mark.parametrize("form", FORMS)
def test_hotstart_resumes_after_an_expired_wait(lib, tmp_path, form):
    """A dump taken before, read back into the same context: the run goes on
    bit for bit, whatever the failed solve had exchanged."""
    from adcirc_b200 import model
    nx, ny, prec = FORMS[form]
    its, want = _run(_case(nx, ny), prec, 8)
    case = _case(nx, ny)
    gpu = model.GpuModel(case, prec)
    got = list(gpu.run(1, 4)[0])
    gpu.hotstart_write(tmp_path / "hs")
    assert lib.adc_set_wait_cycles(gpu.h, 1) == 0
    for _ in range(3):
        with pytest.raises(model.AdcError, match="status -5"):
            gpu.step(5)
    assert lib.adc_set_wait_cycles(gpu.h, 0) == 0
    gpu.hotstart_read(tmp_path / "hs")
    got += list(gpu.run(5, 4)[0])
    gpu.sync_to_host()
    gpu.close()
    assert np.array_equal(its, got)
    bad = [k for k in want if not np.array_equal(want[k], case.arrays[k])]
    assert not bad, bad
