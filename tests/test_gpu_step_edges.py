"""Whole steps at the sizes where the column kernels' level blocks end: the
EOS pass with the column depths and live spans (blocks of four levels, two
ahead), and the 1-2-1 smoothing (eight interfaces a thread; ks taking kt's
values or smoothed on its own), against the oracle, bit for bit; the mixed
solve's tracer pairs with an odd tracer left over, within the 1e-6 of the mixed
form."""
import numpy as np
import pytest

from tests._cases import assert_bitwise, columns, hot_cfg, oracle_state

pytestmark = pytest.mark.gpu
DT = 3600.0


@pytest.fixture(scope="module")
def VP():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from roundabout_b200.column import VerticalPhysics

    return VerticalPhysics


def pair(VP, oracle, cfg, **shape):
    cols = columns(**shape)
    st = oracle_state(oracle, cols, cfg)
    vp = VP(cols.nx, cols.ny, cols.nz, len(cols.tracers), cfg)
    vp.load_columns(cols)
    return st, vp


@pytest.mark.parametrize("nz", [1, 2, 3, 4, 5, 7, 8, 9, 16, 17, 127])
def test_step(VP, oracle, nz):
    cfg = hot_cfg(ntr=3)
    st, vp = pair(VP, oracle, cfg, nx=67, ny=5, nz=nz, ntr=3, seed=300 + nz, thin_frac=0.2)
    assert st.call("vpo_step", cfg, DT, 2) == 0
    vp.step(DT, 2)
    for n in ("rho", "kv", "kt", "ks", "u", "v", "bl_depth", "b0"):
        assert_bitwise(n, vp.get(n), getattr(st, n))
    for t in range(3):
        assert_bitwise(f"tracer{t}", vp.get_tracer(t), st.tracers[t])


@pytest.mark.parametrize("nz", [1, 2, 9, 10, 18])
@pytest.mark.parametrize("over", [dict(), dict(bkgnd_profile=0, kt_bg=2e-5, ks_bg=7e-6)])
def test_smoothing(VP, oracle, nz, over):
    cfg = hot_cfg(kd_smooth_iterations=2, **over)
    st, vp = pair(VP, oracle, cfg, nx=33, ny=9, nz=nz, seed=400 + nz)
    st.call("vpo_eos_wright", cfg)
    st.call("vpo_build_coefficients", cfg)
    vp.eos()
    vp.assemble()
    for n in ("kv", "kt", "ks"):
        assert_bitwise(n, vp.get(n), getattr(st, n))


@pytest.mark.parametrize("ntr", [1, 2, 3, 5])
@pytest.mark.parametrize("nz", [3, 8, 9, 85, 86, 127])
def test_mixed_pairs(VP, oracle, ntr, nz):
    """nz = 85 / 86: three and two warps per lane quarter of the tensor memory."""
    cfg = hot_cfg(ntr=ntr, eos_in_step=0)
    cols = columns(nx=45, ny=4, nz=nz, ntr=max(ntr, 2), seed=500 + nz + ntr, passive_init="uniform")
    cols.tracers = cols.tracers[:ntr]
    cols.q_heat[...] = -np.abs(cols.q_heat)
    if ntr == 1:
        cfg.idx_temperature = -1
    st = oracle_state(oracle, cols, cfg)
    st.rho[...] = 1027.0 - 0.5 * np.arange(nz)[None, None, :] / nz
    vp = VP(cols.nx, cols.ny, nz, ntr, cfg)
    vp.load_columns(cols)
    vp.set("rho", st.rho)
    st.call("vpo_build_coefficients", cfg)
    vp.assemble()
    st.call("vpo_vdiff_tracers", cfg, DT)
    st.call("vpo_nonlocal", cfg, DT)
    cfg.mixed_precision = 1
    vp.set_config(cfg)
    vp.set_variants("registers", "tmem_rows")
    vp.vdiff_tracers_nonlocal(DT)
    for t in range(ntr):
        assert np.abs(vp.get_tracer(t) - st.tracers[t]).max() <= 1e-6
