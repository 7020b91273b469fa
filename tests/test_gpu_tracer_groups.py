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
