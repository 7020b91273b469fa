"""Whole steps at the sizes where the column kernels' level blocks end,
against the oracle, bit for bit.  67 x 5 columns run the forms of grids that do not
fill the chip: the EOS pass with the column depths and live spans in blocks of
eight levels, the assembly with three layers loaded a block ahead.  The same
columns 120 times over run the forms of large grids: the EOS pass in blocks of
four, the assembly in blocks of one (FP64) or three (FP32) layers.  Then operands
outside the range of the exact solves' branch-free quotients, the 1-2-1 smoothing
(eight interfaces a thread; ks taking kt's values or smoothed on its own), and the
mixed solve's tracer pairs with an odd tracer left over, within the 1e-6 of the
mixed form."""
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


@pytest.mark.parametrize("level", [0, 2])
@pytest.mark.parametrize("nz", [1, 2, 3, 4, 5, 7, 8, 9, 74, 75, 76])
def test_step_of_a_large_grid(VP, oracle, nz, level):
    """1200 EOS and 600 assembly blocks.  The rows repeat, with no flow between the copies, so every copy is the
    small grid: FP64 is the oracle's bits, mixed level 2 the small grid's."""
    copies, over = 120, dict(mixed_precision=level)
    cols = columns(nx=67, ny=5, nz=nz, ntr=2, seed=330 + nz, thin_frac=0.2)
    cfg = hot_cfg(ntr=2, **over)
    big = VP(67, 5 * copies, nz, 2, cfg)
    for n in ("h", "u", "q_heat", "q_salt", "wet", "tau_x"):
        big.set(n, np.concatenate([getattr(cols, n)] * copies, axis=1))
    for n in ("v", "tau_y"):
        a = getattr(cols, n)
        assert (a[:, 0] == 0).all() and (a[:, -1] == 0).all()
        big.set(n, np.concatenate([a[:, :-1]] * copies + [a[:, -1:]], axis=1))
    for t in range(2):
        big.set_tracer(t, np.concatenate([cols.tracers[t]] * copies, axis=1))
    big.stress_mag()
    fields = ("rho", "kv", "kt", "ks", "u", "bl_depth", "b0")
    if level == 0:
        st = oracle_state(oracle, cols, cfg)
        assert st.call("vpo_step", cfg, DT, 1) == 0
        want = {n: getattr(st, n) for n in fields}
        want.update({f"tracer{t}": st.tracers[t] for t in range(2)})
    else:
        small = VP(67, 5, nz, 2, cfg)
        small.load_columns(cols)
        for vp in (small, big):
            vp.set_variants("registers", "tmem_rows")
        small.step(DT, 1)
        want = {n: small.get(n) for n in fields + ("tracer0", "tracer1")}
    big.step(DT, 1)
    for n, w in want.items():
        got = big.get(n)
        for c in (0, 1, 59, copies - 1):
            assert_bitwise(n, got[:, 5 * c:5 * c + 5], w)


@pytest.mark.parametrize("over", [dict(), dict(bkgnd_profile=0, kt_bg=2e-5, ks_bg=7e-6), dict(remnant=1)])
def test_operands_out_of_range(VP, oracle, over):
    """A dye released in one layer (near the bed, midway, at the surface) and a spin-up from rest: away from the
    release and the wind the values fall by orders of magnitude a level, through 2^-511, where the exact
    solves leave the branch-free quotients, to zero."""
    cfg = hot_cfg(ntr=7, implicit_stress=1, bkgnd_kd_sfc=1e-6, bkgnd_kd_deep=1e-6, pp81_nu_bg=1e-6,
                  pp81_kappa_bg=1e-6, **over)
    cols = columns(nx=67, ny=5, nz=75, ntr=7, seed=350, passive_init="uniform")
    cols.u[...] = cols.v[...] = 0.0
    cols.tracers[0][...] = 35.0   # stably stratified: no shear mixing below the wind's layer
    cols.tracers[1][...] = 2.0 + 18.0 * np.arange(75) / 75.0
    for t, k in ((2, 74), (3, 37), (5, 20), (6, 30)):
        cols.tracers[t][...] = 0.0
        cols.tracers[t][:, :, k] = cols.wet
    st = oracle_state(oracle, cols, cfg)
    vp = VP(67, 5, 75, 7, cfg)
    vp.load_columns(cols)
    for steps in (1, 3):
        assert st.call("vpo_step", cfg, DT, steps) == 0
        vp.step(DT, steps)
        for n in ("kv", "kt", "ks", "u", "v") + (("visc_rem_u", "visc_rem_v") if cfg.remnant else ()):
            assert_bitwise(n, vp.get(n), getattr(st, n))
        for t in range(7):
            assert_bitwise(f"tracer{t}", vp.get_tracer(t), st.tracers[t])
        for a in (st.u, st.tracers[2], st.tracers[3]):
            a = np.abs(a)
            assert ((a > 0) & (a < 2.0 ** -511)).sum() > 100


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
@pytest.mark.parametrize("nz", [3, 8, 9, 80, 81, 85, 86, 127])
def test_mixed_pairs(VP, oracle, ntr, nz):
    """nz = 80 / 81: three and two warps per lane quarter of the tensor memory."""
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
