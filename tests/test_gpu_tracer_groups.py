"""The exact tracer solve's groups (at most five tracers per thread, as even as
they come: 5 / 6 / 11 / 16 tracers are one, two, three and four groups) and block
remainders, against the oracle, bit for bit, with one factorisation and with
two, with and without the budgets that read the column to the bed."""
import numpy as np
import pytest

from tests._cases import assert_bitwise, columns, hot_cfg, oracle_state

pytestmark = pytest.mark.gpu
DT = 3600.0


@pytest.mark.parametrize("ntr", [1, 2, 3, 5, 6, 7, 11, 16])
@pytest.mark.parametrize("over", [dict(), dict(bkgnd_profile=0, kt_bg=2e-5, ks_bg=7e-6), dict(budgets=1)])
def test_groups(oracle, ntr, over):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from roundabout_b200.column import VerticalPhysics

    cols = columns(nx=70, ny=6, nz=21, ntr=max(ntr, 2), seed=200 + ntr, thin_frac=0.1, passive_init="uniform")
    cols.tracers = cols.tracers[:ntr]
    cols.q_heat[...] = -np.abs(cols.q_heat)
    cfg = hot_cfg(ntr=ntr, eos_in_step=0, **over)
    if ntr == 1:   # one tracer: salinity alone
        cfg.idx_temperature = -1
        cfg.buoyancy_coeffs = 0
    st = oracle_state(oracle, cols, cfg)
    st.rho[...] = 1027.0 - 0.5 * np.arange(cols.nz)[None, None, :] / cols.nz
    vp = VerticalPhysics(cols.nx, cols.ny, cols.nz, ntr, cfg)
    vp.load_columns(cols)
    vp.set("rho", st.rho)
    st.call("vpo_build_coefficients", cfg)
    vp.assemble()
    st.call("vpo_vdiff_tracers", cfg, DT)
    st.call("vpo_nonlocal", cfg, DT)
    vp.vdiff_tracers_nonlocal(DT)
    for t in range(ntr):
        assert_bitwise(f"tracer{t}", vp.get_tracer(t), st.tracers[t])
    if cfg.budgets:
        for n in ("heat_budget", "salt_budget"):
            if ntr > 1 or n == "salt_budget":
                assert_bitwise(n, vp.get(n), getattr(st, n))


@pytest.mark.parametrize("ntr", [6, 8, 9, 10, 11, 16])
@pytest.mark.parametrize("nz", [1, 2, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("over", [dict(), dict(bkgnd_profile=0, kt_bg=2e-5, ks_bg=7e-6), dict(budgets=1),
                                  dict(column_integrals=1)])
def test_shallow_columns(oracle, nz, ntr, over):
    """Columns of up to eight levels (four with nine or ten tracers; with budgets and more than eight tracers three, or
    none up to ten) on a grid that fills the chip: every tracer in one thread; one level more, and it is the groups."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from roundabout_b200.column import VerticalPhysics

    cols = columns(nx=70, ny=80, nz=nz, ntr=ntr, seed=240 + ntr + nz, thin_frac=0.1, passive_init="uniform")
    cols.q_heat[...] = -np.abs(cols.q_heat)
    cfg = hot_cfg(ntr=ntr, eos_in_step=0, **over)
    st = oracle_state(oracle, cols, cfg)
    st.rho[...] = 1027.0 - 0.5 * np.arange(nz)[None, None, :] / nz
    vp = VerticalPhysics(70, 80, nz, ntr, cfg)
    vp.load_columns(cols)
    vp.set("rho", st.rho)
    st.call("vpo_build_coefficients", cfg)
    vp.assemble()
    old = st.column_content(False)
    st.call("vpo_vdiff_tracers", cfg, DT)
    if cfg.column_integrals:   # the two calls apart: the content is the diffusion's
        new = st.column_content(True)
        vp.vdiff_tracers(DT)
        assert_bitwise("content_old", vp.get("content_old"), old)
        assert_bitwise("content_new", vp.get("content_new"), new)
        vp.nonlocal_tendencies(DT)
    else:
        vp.vdiff_tracers_nonlocal(DT)
    st.call("vpo_nonlocal", cfg, DT)
    for t in range(ntr):
        assert_bitwise(f"tracer{t}", vp.get_tracer(t), st.tracers[t])
    if cfg.budgets:
        for n in ("heat_budget", "salt_budget"):
            assert_bitwise(n, vp.get(n), getattr(st, n))
