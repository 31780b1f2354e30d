"""adc_sync_to_host returns every bound array as it was uploaded, through
the pinned block (small states, one piece and several; odd counts leave half a word at the
end of an integer array) and array by array (large ones)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 2), (13, 7), (12, 8), (61, 55), (151, 131), (401, 301)])
def test_round_trip(lib, nx, ny):
    from adcirc_b200 import meshgen, model
    raw = meshgen.channel_mesh(nx=nx, ny=ny, lx=100.0 * nx, ly=100.0 * ny, depth0=5.0, depth1=3.0)
    tides = [(1e-3, 0.0, 1.0, np.full(raw.open_nodes.size, 0.5), np.zeros(raw.open_nodes.size))]
    case = model.build_case(raw, model.default_params(1.0), model.Schedule(dt=1.0, nramp=0), tides)
    rng = np.random.default_rng(nx)
    a = case.arrays
    for k in model.STATE_F64 + model.STATE_I32:
        v = rng.integers(0, 2, a[k].shape) if k in model.STATE_I32 else rng.standard_normal(a[k].shape)
        a[k][...] = v
    slot = np.arange(case.sizes["mnei"])[None, :]
    a["coef"][...] = np.where(slot < a["nneigh"][:, None], rng.standard_normal(a["coef"].shape), 0.0)
    want = {k: v.copy() for k, v in a.items()}
    gpu = model.GpuModel(case)
    for k in model.STATE_F64 + model.STATE_I32:
        if a[k].size:
            a[k][...] = 7
    gpu.sync_to_host()
    gpu.close()
    bad = [k for k in want if not np.array_equal(want[k], a[k])]
    assert not bad, f"arrays differ: {bad}"
