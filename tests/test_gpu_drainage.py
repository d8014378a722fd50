"""GPU parity of the drainage kernels through the C ABI (libsbs.so) against the oracle.

Bars:
  * bit-exact against the kernel-order oracle (same f32 arithmetic), both semantics, all sizes;
  * CPU semantics vs the f64 restatement of drainage.rs: relative L-inf <= 1e-5 per step and,
    after 1000 steps of config 0, <= 1e-4 (plain f32) / <= 1e-8 (compensated f32x2);
  * WGSL semantics vs the drainage.wgsl operation order: <= 1e-5 per pass, <= 1e-4 after 1000;
  * FP64 film volume within 1e-12 relative of the oracle's sum.
"""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel_linf(a, b):
    return float(np.max(np.abs(np.asarray(a, np.float64) - b)) / np.max(np.abs(b)))


def make_sim(sbs, res, precision="f32x2"):
    cfg = sbs.SimulationConfig()
    cfg.resolution = res
    c = cfg.to_c()
    h = ctypes.c_void_p()
    prec = sbs._native.DRAIN_F32X2 if precision == "f32x2" else sbs._native.DRAIN_F32
    sbs._native.call("sbs_drainage_create_ex", ctypes.byref(c), prec, ctypes.byref(h))
    sim = sbs.DrainageSimulator.__new__(sbs.DrainageSimulator)
    sbs.drainage._Handle.__init__(sim)
    sim._h = h
    sim._config = cfg
    return sim


def field64(sbs, sim):
    nt, np_ = sim.grid()
    out = np.empty(nt * np_, dtype=np.float64)
    sbs._native.call("sbs_drainage_get_thickness_field_f64", sim.handle, sbs._native.dptr(out), out.size)
    return out.reshape(nt, np_)


def set64(sbs, sim, h):
    a = np.ascontiguousarray(h, dtype=np.float64)
    sbs._native.call("sbs_drainage_set_thickness_f64", sim.handle, sbs._native.dptr(a), a.size)


ORC_PREC = {"f32": "f32k", "f32x2": "f32x2"}


# --------------------------------------------------------------------------------------------
# CPU semantics (DrainageSimulator)
# --------------------------------------------------------------------------------------------
@pytest.mark.parametrize("precision", ["f32x2", "f32"])
@pytest.mark.parametrize("res", [3, 8, 33, 64, 130])
def test_cpu_semantics_bit_exact(sbs, orc, precision, res):
    """Single steps and graph-replayed chunks, TFE fronts active (dt 0.01 s: first spawn at step
    50), odd and non-multiple-of-4 widths; every cell equal to the kernel-order oracle."""
    from soap_bubble_simulation_gb300 import synthetic

    h0 = synthetic.bubble_c0(res, seed=res)
    if precision == "f32":
        h0 = h0.astype(np.float32).astype(np.float64)
    sim = make_sim(sbs, res, precision)
    set64(sbs, sim, h0)
    ref = orc.CpuSim(resolution=res, precision=ORC_PREC[precision])
    ref.set_field(h0)
    for _ in range(10):
        sim.step(0.01)
        ref.step(0.01)
    np.testing.assert_array_equal(field64(sbs, sim), ref.field())
    sim.step_n(0.01, 190)
    ref.step_n(0.01, 190)
    got, want = field64(sbs, sim), ref.field()
    assert sim.active_tfe_count() == ref.active_tfe_count()
    assert sim.current_time() == ref.current_time()
    if not np.array_equal(got, want):
        bad = np.argwhere(got != want)
        pytest.fail(f"{len(bad)} cells differ, first {bad[:5].tolist()}, "
                    f"max rel {rel_linf(got, want):.3e}")
    if res >= 33:
        assert sim.active_tfe_count() >= 1
        assert (got < h0 * 0.99999).any()  # fronts thinned something


def set_cpu_blocking(sbs, sim, k):
    sbs._native.call("sbs_drainage_set_time_blocking", sim.handle, k)


def cpu_blocking(sbs, sim):
    out = ctypes.c_int()
    sbs._native.call("sbs_drainage_time_blocking", sim.handle, ctypes.byref(out))
    return out.value


@pytest.mark.parametrize("precision", ["f32x2", "f32"])
@pytest.mark.parametrize("res", [10, 12, 64, 130, 256])
def test_cpu_time_blocking_bit_identical(sbs, orc, precision, res):
    """K = 1..4 steps per launch (the blocked kernel's polar strips form each step's ring means
    as exact integer sums across their blocks): the same bits as single steps and as the
    kernel-order oracle, with fronts active (first spawn at step 50), a frozen critical patch,
    volume checks and chunk ends at every K."""
    from soap_bubble_simulation_gb300 import synthetic

    h0 = synthetic.bubble_c0(res, seed=res + 1)
    h0[res // 3, : res // 2] = 5e-9  # below the 10 nm critical thickness: frozen
    if precision == "f32":
        h0 = h0.astype(np.float32).astype(np.float64)
    results = []
    for k in (1, 2, 3, 4):
        sim = make_sim(sbs, res, precision)
        assert cpu_blocking(sbs, sim) == (3 if precision == "f32x2" else 4)  # the defaults
        set_cpu_blocking(sbs, sim, k)
        assert cpu_blocking(sbs, sim) == k
        set64(sbs, sim, h0)
        sim.step_n(0.01, 23)
        vols = sim.run_checked(0.01, 60, 20)
        for _ in range(3):
            sim.step(0.01)
        results.append((field64(sbs, sim), vols, sim.active_tfe_count()))
        sim.close()
    for f, v, n in results[1:]:
        np.testing.assert_array_equal(f, results[0][0])
        np.testing.assert_allclose(v, results[0][1], rtol=1e-12)
        assert n == results[0][2]
    ref = orc.CpuSim(resolution=res, precision=ORC_PREC[precision])
    ref.set_field(h0)
    ref.step_n(0.01, 86)
    np.testing.assert_array_equal(results[0][0], ref.field())
    assert results[0][2] == ref.active_tfe_count() >= 1


@pytest.mark.parametrize("precision", ["f32x2", "f32"])
@pytest.mark.parametrize("res", [1024, 1500])
def test_cpu_single_steps_many_column_blocks(sbs, orc, precision, res):
    """Single steps (K = 1) on grids of 2048 and 3000 columns (many column blocks, the last one
    partly filled: 3000 = 5 x 512 + 440), the phi wrap at both ends, fronts active from step 50
    (dt 0.01 s), volume checks: every cell equal to the kernel-order oracle."""
    from soap_bubble_simulation_gb300 import synthetic

    h0 = synthetic.smooth_modes(res, 2 * res, seed=res)
    if precision == "f32":
        h0 = h0.astype(np.float32).astype(np.float64)
    sim = make_sim(sbs, res, precision)
    set_cpu_blocking(sbs, sim, 1)
    set64(sbs, sim, h0)
    sim.step_n(0.01, 47)
    vols = sim.run_checked(0.01, 16, 8)
    ref = orc.CpuSim(resolution=res, precision=ORC_PREC[precision], threads=0)
    ref.set_field(h0)
    ref.step_n(0.01, 55)
    v0 = orc.film_volume(ref.field(), 0.025)
    ref.step_n(0.01, 8)
    got, want = field64(sbs, sim), ref.field()
    assert sim.active_tfe_count() == ref.active_tfe_count() >= 1
    np.testing.assert_array_equal(got, want)
    assert vols[0] == pytest.approx(v0, rel=1e-12)
    assert vols[1] == pytest.approx(orc.film_volume(want, 0.025), rel=1e-12)


def test_cpu_time_blocking_needs_even_resolution(sbs):
    sim = make_sim(sbs, 33)  # 66 columns: not a multiple of 4
    assert cpu_blocking(sbs, sim) == 1
    with pytest.raises(sbs.SbsError, match="even resolution"):
        set_cpu_blocking(sbs, sim, 4)
    set_cpu_blocking(sbs, sim, 1)
    sim.step_n(0.001, 5)
    small = make_sim(sbs, 4)  # fewer than 2 (K + 1) rows for any K
    assert cpu_blocking(sbs, small) == 1
    with pytest.raises(sbs.SbsError):
        set_cpu_blocking(sbs, small, 4)


def test_step_n_equals_repeated_steps(sbs):
    from soap_bubble_simulation_gb300 import synthetic

    h0 = synthetic.bubble_c0(64, seed=3)
    a, b = make_sim(sbs, 64), make_sim(sbs, 64)
    set64(sbs, a, h0)
    set64(sbs, b, h0)
    a.step_n(0.002, 333)
    for _ in range(333):
        b.step(0.002)
    np.testing.assert_array_equal(field64(sbs, a), field64(sbs, b))
    assert a.current_time() == b.current_time()


@pytest.mark.parametrize("precision,tol", [("f32", 1e-4), ("f32x2", 1e-8)])
def test_c0_1000_steps_vs_f64_reference(sbs, orc, precision, tol):
    """Config 0: resolution 128, h = 500 nm (1 + 0.05 U[-1,1]) seed 0, defaults, dt 1e-3,
    1000 steps, TFE on. Relative L-inf against the f64 restatement of drainage.rs."""
    from soap_bubble_simulation_gb300 import synthetic

    h0 = synthetic.bubble_c0(128, seed=0).astype(np.float32).astype(np.float64)
    sim = make_sim(sbs, 128, precision)
    set64(sbs, sim, h0)
    ref = orc.CpuSim(resolution=128, precision="f64", threads=0)
    ref.set_field(h0)
    # per-step bar over the first steps, from the same input each time
    for k in range(5):
        ref_step = orc.CpuSim(resolution=128, precision="f64")
        ref_step.set_field(field64(sbs, sim))
        sim.step(0.001)
        ref_step.step(0.001)
        assert rel_linf(field64(sbs, sim), ref_step.field()) <= 1e-5
    ref.step_n(0.001, 5)
    sim.step_n(0.001, 995)
    ref.step_n(0.001, 995)
    err = rel_linf(field64(sbs, sim), ref.field())
    assert err <= tol, err
    assert sim.active_tfe_count() == ref.active_tfe_count() >= 1


# --- the reference's drainage.rs unit tests on the GPU path (drainage.rs:636-719) ------------
def test_reference_unit_tests_on_gpu(sbs):
    cfg = sbs.SimulationConfig.default()
    sim = sbs.DrainageSimulator(cfg)
    assert abs(sim.current_time()) < 1e-300 and not sim.has_critical_region()
    assert abs(sim.get_thickness(0.5, 1.0) - sim.get_thickness(1.5, 3.0)) < 1e-15
    assert abs(sim.get_thickness(1.0, 0.0) - sim.get_thickness(1.0, 2 * math.pi)) < 1e-12
    before = sim.get_thickness(0.1, 0.0)
    sim.step(cfg.dt)
    assert abs(sim.current_time() - 0.001) < np.finfo(float).eps
    for _ in range(99):
        sim.step(cfg.dt)
    assert sim.get_thickness(0.1, 0.0) < before
    sim.reset(600e-9)
    assert sim.current_time() == 0.0
    assert abs(sim.get_thickness(0.5, 0.5) - 600e-9) < 1e-15
    assert sim.critical_thickness() == pytest.approx(10e-9)
    f = sim.thickness_field()
    assert f.num_theta() == 128 and f.num_phi() == 256


def test_query_batch_matches_oracle(sbs, orc):
    from soap_bubble_simulation_gb300 import synthetic

    h0 = synthetic.bubble_c0(48, seed=9)
    sim = make_sim(sbs, 48)
    set64(sbs, sim, h0)
    ref = orc.CpuSim(resolution=48, precision="f32x2")
    ref.set_field(h0)
    sim.step_n(0.001, 20)
    ref.step_n(0.001, 20)
    g = np.random.default_rng(1)
    th = np.concatenate([g.uniform(-0.5, math.pi + 0.5, 500), [0.0, math.pi, 1.0, 1.0]])
    ph = np.concatenate([g.uniform(-10, 10, 500), [0.0, 2 * math.pi, -2 * math.pi, 4 * math.pi - 1e-12]])
    got = sim.get_thickness_batch(th, ph)
    want = np.array([ref.get_thickness(a, b) for a, b in zip(th, ph)])
    np.testing.assert_array_equal(got, want)


def test_volume_checks_match_oracle(sbs, orc):
    from soap_bubble_simulation_gb300 import synthetic

    h0 = synthetic.bubble_c0(96, seed=4)
    sim = make_sim(sbs, 96)
    set64(sbs, sim, h0)
    ref = orc.CpuSim(resolution=96, precision="f32x2")
    ref.set_field(h0)
    vols = sim.run_checked(0.01, 300, 100)
    assert vols.shape == (3,)
    for k in range(3):
        ref.step_n(0.01, 100)
        want = orc.film_volume(ref.field(), 0.025)
        assert vols[k] == pytest.approx(want, rel=1e-12)
    np.testing.assert_array_equal(field64(sbs, sim), ref.field())
    assert sim.film_volume() == pytest.approx(orc.film_volume(ref.field(), 0.025), rel=1e-12)
    mn, mx = sim.min_max()
    assert mn == ref.min_thickness() and mx == ref.max_thickness()


def test_marginal_regeneration_controls(sbs, orc):
    sim = make_sim(sbs, 64)
    ref = orc.CpuSim(resolution=64, precision="f32x2")
    sim.set_tfe_thickness_ratio(0.2)
    assert sim.tfe_thickness_ratio() == 0.5
    sim.set_tfe_thickness_ratio(0.9)
    ref.set_tfe_thickness_ratio(0.9)
    assert sim.marginal_regeneration_enabled()
    sim.step_n(0.01, 120)
    ref.step_n(0.01, 120)
    assert sim.active_tfe_count() == ref.active_tfe_count() >= 1
    np.testing.assert_array_equal(field64(sbs, sim), ref.field())
    sim.set_marginal_regeneration(False)
    ref.set_marginal_regeneration(False)
    assert sim.active_tfe_count() == 0 and not sim.marginal_regeneration_enabled()
    sim.step_n(0.01, 50)
    ref.step_n(0.01, 50)
    np.testing.assert_array_equal(field64(sbs, sim), ref.field())


def test_critical_cells_frozen_and_detected(sbs):
    h0 = np.full((32, 64), 500e-9)
    h0[10, 5] = 5e-9
    sim = make_sim(sbs, 32)
    set64(sbs, sim, h0)
    assert sim.has_critical_region()
    sim.step_n(0.001, 10)
    # frozen at its stored value: 5 nm as a hi + lo f32 pair
    hi = np.float32(5e-9)
    assert field64(sbs, sim)[10, 5] == float(hi) + float(np.float32(5e-9 - float(hi)))


def test_errors_are_reported(sbs):
    with pytest.raises(sbs.SbsError):
        make_sim(sbs, 2)
    sim = make_sim(sbs, 16)
    with pytest.raises(ValueError):
        sim.set_thickness_array(np.zeros((15, 32), np.float32))
    short = np.zeros(15 * 32, np.float32)
    with pytest.raises(sbs.SbsError, match="expected 16 x 32"):
        sbs._native.call("sbs_drainage_set_thickness", sim.handle, sbs._native.ptr(short), short.size,
                         sbs._native.MEM_HOST)
    with pytest.raises(sbs.SbsError):
        sim.step(float("nan"))
    with pytest.raises(sbs.SbsError, match="WGSL"):
        sbs._native.call("sbs_gpu_drainage_run", sim.handle, 1)
    g = sbs.GPUDrainageSimulator(None, 500e-9, 16, 8)
    with pytest.raises(sbs.SbsError, match="CPU"):
        sbs._native.call("sbs_drainage_step", g.handle, 0.001)
    with pytest.raises(sbs.SbsError):
        sbs.GPUDrainageSimulator(None, 500e-9, 2, 8)


def test_film_volume_device_stateless(sbs, orc):
    from soap_bubble_simulation_gb300 import synthetic

    sim = sbs.GPUDrainageSimulator(None, 500e-9, 128, 64)
    h = synthetic.smooth_modes(64, 128).astype(np.float32)
    sim.set_thickness_array(h)
    d = sim.current_thickness_buffer()
    v = sbs.film_volume_device(d.ptr, 64, 128, d.pitch, 0.025)
    assert v == pytest.approx(orc.film_volume(h, 0.025), rel=1e-12)


# --------------------------------------------------------------------------------------------
# WGSL semantics (GPUDrainageSimulator)
# --------------------------------------------------------------------------------------------
@pytest.mark.parametrize("W,H", [(128, 64), (130, 33), (3, 3), (5, 7), (512, 200)])
@pytest.mark.parametrize("marangoni", [0, 1])
def test_wgsl_semantics_bit_exact(sbs, orc, W, H, marangoni):
    from soap_bubble_simulation_gb300 import synthetic

    h = synthetic.smooth_modes(H, W, seed=W + H).astype(np.float32)
    h[H // 2, W // 2] = 20e-9  # below the 30 nm critical thickness: copied
    c = synthetic.surfactant_noise(H, W, seed=7)
    sim = sbs.GPUDrainageSimulator(None, 500e-9, W, H)
    sim.set_thickness_array(h)
    sim.set_concentration_array(c)
    if marangoni:
        sim.set_marangoni_enabled(True)
    sim.run(37)
    p = orc.wgsl_params(grid_width=W, grid_height=H, marangoni_enabled=marangoni)
    hk, ck = orc.wgsl_run(p, h, c, 37, "kernel")
    np.testing.assert_array_equal(sim.thickness_array(), hk)
    np.testing.assert_array_equal(sim.concentration_array(), ck)


@pytest.mark.parametrize("marangoni", [0, 1])
def test_wgsl_semantics_vs_wgsl_operation_order(sbs, orc, marangoni):
    from soap_bubble_simulation_gb300 import synthetic

    W, H = 128, 64
    h = synthetic.smooth_modes(H, W).astype(np.float32)
    c = synthetic.surfactant_noise(H, W)
    sim = sbs.GPUDrainageSimulator(None, 500e-9, W, H)
    sim.set_thickness_array(h)
    sim.set_concentration_array(c)
    sim.set_marangoni_enabled(bool(marangoni))
    p = orc.wgsl_params(marangoni_enabled=marangoni)
    sim.run(1)
    h1, c1 = orc.wgsl_run(p, h, c, 1, "wgsl")
    assert rel_linf(sim.thickness_array(), h1) <= 1e-5
    assert np.max(np.abs(sim.concentration_array() - c1)) <= 1e-5
    sim.run(999)
    hN, cN = orc.wgsl_run(p, h, c, 1000, "wgsl")
    assert rel_linf(sim.thickness_array(), hN) <= 1e-4
    assert np.max(np.abs(sim.concentration_array() - cN)) <= 1e-4


def test_wgsl_step_clock_and_enable(sbs):
    sim = sbs.GPUDrainageSimulator(None, 500e-9, 128, 64)
    before = sim.thickness_array()
    sim.step(1.0 / 60.0)  # disabled by default (gpu_drainage.rs:339-341)
    np.testing.assert_array_equal(sim.thickness_array(), before)
    assert sim.current_time() == 0.0
    sim.enabled = True
    sim.step(1.0 / 60.0)
    step_dt = np.float32(np.float32(1.0 / 60.0) * np.float32(100.0)) / np.float32(10)
    assert sim.current_time() == pytest.approx(10 * float(step_dt), rel=1e-12)
    assert sim.grid_size() == (128, 64)
    p = sim.params()
    assert p.grid_width == 128 and p.dt == pytest.approx(0.001)


def test_wgsl_buffers_and_reset(sbs, orc):
    """current_buffer() is the last pass's input (gpu_drainage.rs:473-479): its film volume equals
    the field before the pass; current_thickness_buffer() holds the output."""
    from soap_bubble_simulation_gb300 import synthetic

    h = synthetic.smooth_modes(64, 128).astype(np.float32)
    sim = sbs.GPUDrainageSimulator(None, 500e-9, 128, 64)
    sim.set_thickness_array(h)
    sim.run(3)
    prev = orc.wgsl_run(orc.wgsl_params(), h, np.full_like(h, 0.5), 2, "kernel")[0]
    cur = sim.thickness_array()
    stale, new = sim.current_buffer(), sim.current_thickness_buffer()
    assert stale.ptr != new.ptr
    v_stale = sbs.film_volume_device(stale.ptr, 64, 128, stale.pitch, 0.025)
    v_new = sbs.film_volume_device(new.ptr, 64, 128, new.pitch, 0.025)
    assert v_stale == pytest.approx(orc.film_volume(prev, 0.025), rel=1e-12)
    assert v_new == pytest.approx(orc.film_volume(cur, 0.025), rel=1e-12)
    sim.reset(400e-9)
    np.testing.assert_array_equal(sim.thickness_array(), np.float32(400e-9))
    np.testing.assert_array_equal(sim.concentration_array(), np.float32(0.5))
    assert sim.current_time() == 0.0


def test_wgsl_params_setters(sbs, orc):
    from soap_bubble_simulation_gb300 import synthetic

    W, H = 128, 64
    h = synthetic.smooth_modes(H, W).astype(np.float32)
    c = synthetic.surfactant_noise(H, W)
    sim = sbs.GPUDrainageSimulator(None, 500e-9, W, H)
    sim.set_thickness_array(h)
    sim.set_concentration_array(c)
    sim.set_dt(0.002)
    sim.set_physics(0.002, 1100.0, 9.0, 2e-9)
    sim.set_bubble_radius(0.01)
    sim.set_marangoni_params(0.07, 0.05, 3e-9, 0.02)
    sim.set_marangoni_enabled(True)
    sim.run(25)
    p = orc.wgsl_params(dt=0.002, viscosity=0.002, density=1100.0, gravity=9.0, diffusion_coeff=2e-9,
                        bubble_radius=0.01, gamma_air=0.07, gamma_reduction=0.05, surfactant_diffusion=3e-9,
                        marangoni_coeff=0.02, marangoni_enabled=1)
    hk, ck = orc.wgsl_run(p, h, c, 25, "kernel")
    np.testing.assert_array_equal(sim.thickness_array(), hk)
    np.testing.assert_array_equal(sim.concentration_array(), ck)


def test_wgsl_volume_checks(sbs, orc):
    from soap_bubble_simulation_gb300 import synthetic

    W, H = 256, 128
    h = synthetic.smooth_modes(H, W).astype(np.float32)
    c = synthetic.surfactant_noise(H, W)
    sim = sbs.GPUDrainageSimulator(None, 500e-9, W, H)
    sim.set_thickness_array(h)
    sim.set_concentration_array(c)
    vols = sim.run_checked(0.0, 200, 50)
    p = orc.wgsl_params(grid_width=W, grid_height=H)
    cur_h, cur_c = h, c
    for k in range(4):
        cur_h, cur_c = orc.wgsl_run(p, cur_h, cur_c, 50, "kernel")
        assert vols[k] == pytest.approx(orc.film_volume(cur_h, 0.025), rel=1e-12)


# --------------------------------------------------------------------------------------------
# Temporal blocking (several WGSL steps per launch) must not change a single bit
# --------------------------------------------------------------------------------------------
def set_blocking(sbs, sim, k):
    sbs._native.call("sbs_gpu_drainage_set_time_blocking", sim.handle, k)


@pytest.mark.parametrize("W,H", [(4096, 300), (512, 200), (8, 5), (132, 40), (248, 9)])
@pytest.mark.parametrize("marangoni", [0, 1])
def test_time_blocking_bit_identical(sbs, orc, W, H, marangoni):
    from soap_bubble_simulation_gb300 import synthetic

    h = synthetic.smooth_modes(H, W, seed=W * 7 + H).astype(np.float32)
    h[H // 3, : W // 5] = 25e-9  # a patch below the critical thickness
    c = synthetic.surfactant_noise(H, W, seed=H)
    results = []
    for k in (1, 2, 3, 4):
        sim = sbs.GPUDrainageSimulator(None, 500e-9, W, H)
        set_blocking(sbs, sim, k)
        sim.set_thickness_array(h)
        sim.set_concentration_array(c)
        sim.set_marangoni_enabled(bool(marangoni))
        sim.run(23)
        sim.run(18)
        results.append((sim.thickness_array(), sim.concentration_array()))
    for hk, ck in results[1:]:
        np.testing.assert_array_equal(hk, results[0][0])
        np.testing.assert_array_equal(ck, results[0][1])
    if W * H <= 512 * 200:
        p = orc.wgsl_params(grid_width=W, grid_height=H, marangoni_enabled=marangoni)
        ho, co = orc.wgsl_run(p, h, c, 41, "kernel")
        np.testing.assert_array_equal(results[0][0], ho)
        np.testing.assert_array_equal(results[0][1], co)


def test_time_blocking_keeps_previous_buffer_one_pass_behind(sbs, orc):
    from soap_bubble_simulation_gb300 import synthetic

    h = synthetic.smooth_modes(64, 128).astype(np.float32)
    sim = sbs.GPUDrainageSimulator(None, 500e-9, 128, 64)
    out = ctypes.c_int()
    sbs._native.call("sbs_gpu_drainage_time_blocking", sim.handle, ctypes.byref(out))
    assert out.value == 4
    sim.set_thickness_array(h)
    sim.run(9)  # two 4-step launches and one single step
    prev = orc.wgsl_run(orc.wgsl_params(), h, np.full_like(h, 0.5), 8, "kernel")[0]
    stale = sim.current_buffer()
    v = sbs.film_volume_device(stale.ptr, 64, 128, stale.pitch, 0.025)
    assert v == pytest.approx(orc.film_volume(prev, 0.025), rel=1e-12)


def test_time_blocking_needs_width_multiple_of_4(sbs):
    sim = sbs.GPUDrainageSimulator(None, 500e-9, 130, 20)
    with pytest.raises(sbs.SbsError, match="multiple of 4"):
        set_blocking(sbs, sim, 4)
    set_blocking(sbs, sim, 1)
    sim.run(5)


@pytest.mark.parametrize("marangoni", [0, 1])
@pytest.mark.parametrize("W,H", [(9, 5), (11, 40), (119, 37), (121, 64), (122, 33), (243, 70), (1037, 131)])
def test_ragged_widths_blocked_by_default_match_single_steps(sbs, orc, W, H, marangoni):
    """Widths that are no multiple of four cells (the seam inside a lane's window, one and several
    120-column segments, a window that wraps more than once) run blocked by default: the bits of
    single steps and of the kernel-order oracle, volumes, and the fused caustic map."""
    from soap_bubble_simulation_gb300 import synthetic

    h = synthetic.smooth_modes(H, W, seed=W + H).astype(np.float32)
    h[H // 3, : W // 4] = 25e-9  # a patch below the critical thickness
    h[2 * H // 3, W // 2] = 1e-4  # a spike that is clamped at zero around it
    c = synthetic.surfactant_noise(H, W, seed=H)
    c[1, :3] = (0.0, 1.0, 0.5)
    out = []
    for single in (False, True):
        sim = sbs.GPUDrainageSimulator(None, 500e-9, W, H)
        if single:
            set_blocking(sbs, sim, 1)
        sim.set_thickness_array(h)
        sim.set_concentration_array(c)
        sim.set_marangoni_enabled(bool(marangoni))
        vols = sim.run_checked(0.001, 22, 11)
        cau = sim.run_caustic_map(9)
        out.append((sim.thickness_array(), sim.concentration_array(), cau, vols))
    for a, b in zip(out[0][:3], out[1][:3]):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_allclose(out[0][3], out[1][3], rtol=1e-12)
    p = orc.wgsl_params(grid_width=W, grid_height=H, marangoni_enabled=marangoni)
    ho, co = orc.wgsl_run(p, h, c, 31, "kernel")
    np.testing.assert_array_equal(out[0][0], ho)
    np.testing.assert_array_equal(out[0][1], co)


@pytest.mark.parametrize("precision", ["f32x2", "f32"])
@pytest.mark.parametrize("res", [9, 11, 33, 61, 121, 305])
def test_odd_resolutions_blocked_by_default_match_single_steps(sbs, orc, precision, res):
    """Odd resolutions (rows of 2 r cells, no multiple of four; pole rings of one and several blocks)
    run blocked by default: the bits of single steps and of the kernel-order oracle, fronts active
    (first spawn at step 50), volumes."""
    from soap_bubble_simulation_gb300 import synthetic

    h0 = synthetic.bubble_c0(res, seed=res)
    h0[res // 3, : res // 2] = 5e-9  # below the 10 nm critical thickness: frozen
    h0[1, : res // 3] *= 40.0
    if precision == "f32":
        h0 = h0.astype(np.float32).astype(np.float64)
    out = []
    for single in (False, True):
        sim = make_sim(sbs, res, precision)
        if single:
            set_cpu_blocking(sbs, sim, 1)
        set64(sbs, sim, h0)
        sim.step_n(0.01, 47)
        vols = sim.run_checked(0.01, 34, 17)
        out.append((field64(sbs, sim), vols))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=1e-12)
    ref = orc.CpuSim(resolution=res, precision=ORC_PREC[precision])
    ref.set_field(h0)
    ref.step_n(0.01, 81)
    np.testing.assert_array_equal(out[0][0], ref.field())


@pytest.mark.parametrize("res", [64, 121, 256])
def test_pole_rings_of_very_large_words_use_the_wide_sums(sbs, orc, res):
    """Ring words around the 128-bit sums' range (4096 m) on some or all of the ring's blocks, negative
    low words, and words below 2^-96 m: the kernel-order oracle's bits."""
    from soap_bubble_simulation_gb300 import synthetic

    base = synthetic.bubble_c0(res, seed=5)
    for hi in (4000.0, 5000.0, 1e9):
        h0 = base.copy()
        h0[1, 3] = hi
        h0[res - 2, res : res + 40] = hi / 3.0
        h0[1, 9] = 1e-30
        sim = make_sim(sbs, res, "f32x2")
        set64(sbs, sim, h0)
        sim.step_n(1e-9, 3)
        ref = orc.CpuSim(resolution=res, precision=ORC_PREC["f32x2"])
        ref.set_field(h0)
        ref.step_n(1e-9, 3)
        np.testing.assert_array_equal(field64(sbs, sim), ref.field())


@pytest.mark.parametrize("marangoni", [0, 1])
@pytest.mark.parametrize("W,H", [(3, 3), (7, 4), (128, 3), (130, 90), (255, 160), (640, 310), (1027, 500), (2048, 160)])
def test_resident_chunks_match_single_steps(sbs, orc, W, H, marangoni):
    """Grids that stay on the chip for a chunk of passes (default): one and several rows per block,
    one to sixteen warps per row, the seam inside a lane's window, chunks of 256 and a remainder, the
    field one pass behind the newest, volumes: the bits of single steps."""
    from soap_bubble_simulation_gb300 import synthetic

    h = synthetic.smooth_modes(H, W, seed=W + H).astype(np.float32)
    h[H // 2, : W // 3] = 25e-9  # below the critical thickness
    c = synthetic.surfactant_noise(H, W, seed=H)
    c[H // 2, -1] = 1.0
    out = []
    for single in (False, True):
        sim = sbs.GPUDrainageSimulator(None, 500e-9, W, H)
        if single:
            set_blocking(sbs, sim, 1)
        sim.set_thickness_array(h)
        sim.set_concentration_array(c)
        sim.set_marangoni_enabled(bool(marangoni))
        sim.run(1)
        sim.run(2)
        vols = sim.run_checked(0.001, 300, 130)
        stale = sim.current_buffer()
        v = sbs.film_volume_device(stale.ptr, H, W, stale.pitch, 0.025)
        out.append((sim.thickness_array(), sim.concentration_array(), vols, v, sim.current_time()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_allclose(out[0][2], out[1][2], rtol=1e-12)
    assert out[0][3] == pytest.approx(out[1][3], rel=1e-12) and out[0][4] == out[1][4]


@pytest.mark.parametrize("precision", ["f32x2", "f32"])
@pytest.mark.parametrize("res", [3, 4, 64, 153, 200, 320, 330])
def test_resident_cpu_chunks_match_single_steps(sbs, precision, res):
    """The same in DrainageSimulator semantics, with fronts (the first at step 50) over several rows of
    a block, and both poles in one block at the smallest sizes."""
    from soap_bubble_simulation_gb300 import synthetic

    h0 = synthetic.bubble_c0(res, seed=res)
    h0[res // 3, : res // 2] = 5e-9
    out = []
    for single in (False, True):
        sim = make_sim(sbs, res, precision)
        if single:
            set_cpu_blocking(sbs, sim, 1)
        set64(sbs, sim, h0)
        sim.step(0.01)
        sim.step_n(0.01, 300)
        vols = sim.run_checked(0.01, 40, 20)
        out.append((field64(sbs, sim), vols, sim.active_tfe_count()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=1e-12)
    assert out[0][2] == out[1][2] >= 1


@pytest.mark.parametrize("semantics,nt,np_,routes", [
    ("wgsl", 64, 128, ("resident", "blocked", "single")), ("wgsl", 33, 131, ("resident", "blocked", "single")),
    ("wgsl", 3, 7, ("resident", "single")), ("wgsl", 40, 2052, ("blocked", "single")),
    ("wgsl", 40, 2051, ("blocked", "single")), ("cpu", 64, 128, ("resident", "blocked", "single")),
    ("cpu", 61, 122, ("resident", "blocked", "single")), ("cpu", 4, 8, ("resident", "single")),
    ("cpu", 1026, 2052, ("blocked", "single"))])
def test_routes_are_chosen_and_reported(sbs, semantics, nt, np_, routes):
    """Every route that a grid allows, from any other, in the middle of a run: the same bits; a route that
    it does not allow is refused and leaves the one in use."""
    from soap_bubble_simulation_gb300 import synthetic

    def make():
        if semantics == "cpu":
            return make_sim(sbs, nt)
        sim = sbs.GPUDrainageSimulator(None, 500e-9, np_, nt)
        sim.set_thickness_array(synthetic.smooth_modes(nt, np_, seed=nt).astype(np.float32))
        return sim

    def run(sim, n):
        sim.step_n(1e-4, n) if semantics == "cpu" else sim.run(n)

    sim, ref = make(), make()
    ref.route = "single"
    assert sim.route == routes[0] and ref.route == "single"
    for route in ("blocked", "auto", "single", "resident", "blocked", "single", "auto"):
        before = sim.route
        if route == "auto" or route in routes:
            sim.route = route
            assert sim.route == (routes[0] if route == "auto" else route)
        else:
            with pytest.raises(sbs.SbsError, match="fit|small"):
                sim.route = route
            assert sim.route == before
        run(sim, 13)
        run(ref, 13)
        np.testing.assert_array_equal(sim.thickness_array(), ref.thickness_array())
    with pytest.raises(ValueError):
        sim.route = "fast"
    out = ctypes.c_int()
    sbs._native.call("sbs_drainage_time_blocking", sim.handle, ctypes.byref(out))
    if np_ % 4 == 0 and "blocked" in routes:  # a chosen K leaves the resident route, and stays until "auto"
        set_cpu_blocking(sbs, sim, 2)
        assert sim.route == "blocked"
        sim.route = "blocked"
        assert cpu_blocking(sbs, sim) == 2
        sim.route = "auto"
        assert sim.route == routes[0] and cpu_blocking(sbs, sim) == out.value
    run(sim, 13)
    run(ref, 13)
    np.testing.assert_array_equal(sim.thickness_array(), ref.thickness_array())


@pytest.mark.parametrize("W,H", [(2051, 200), (2500, 121), (2501, 500), (8, 30)])
def test_marangoni_strips_match_single_steps(sbs, W, H):
    """Blocked steps with Marangoni, whose strips have their own height, and the plain ones of the same
    handle: single steps' bits, volumes, the shorter launches of a remainder."""
    from soap_bubble_simulation_gb300 import synthetic

    h = synthetic.smooth_modes(H, W, seed=W + H).astype(np.float32)
    c = synthetic.surfactant_noise(H, W, seed=H)
    out = []
    for route in ("blocked", "single"):
        sim = sbs.GPUDrainageSimulator(None, 500e-9, W, H)
        sim.route = route
        sim.set_thickness_array(h)
        sim.set_concentration_array(c)
        vols = []
        for marangoni in (1, 0, 1):
            sim.set_marangoni_enabled(bool(marangoni))
            vols.append(sim.run_checked(0.0, 22, 11))
            sim.run(4)
        out.append((sim.thickness_array(), sim.concentration_array(), np.concatenate(vols)))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_allclose(out[0][2], out[1][2], rtol=1e-12)


@pytest.mark.parametrize("marangoni", [0, 1])
@pytest.mark.parametrize("W,H", [(7, 3), (128, 64), (1037, 517), (1501, 900), (1999, 1300), (1600, 2000)])
def test_runs_of_few_passes_match_single_steps(sbs, W, H, marangoni):
    """Runs on both sides of the numbers of passes from which the resident kernel takes them, on grids of
    every class of that rule: bits, the field one pass behind the newest, volumes, the caustic map."""
    from soap_bubble_simulation_gb300 import synthetic

    h = synthetic.smooth_modes(H, W, seed=W + H).astype(np.float32)
    c = synthetic.surfactant_noise(H, W, seed=H)
    out = []
    for route in ("auto", "resident", "single"):
        sim = sbs.GPUDrainageSimulator(None, 500e-9, W, H)
        sim.route = route
        assert sim.route == ("single" if route == "single" else "resident")
        sim.set_thickness_array(h)
        sim.set_concentration_array(c)
        sim.set_marangoni_enabled(bool(marangoni))
        behind = []
        for k in (1, 2, 3, 5, 6, 15, 16):
            sim.run(k)
            stale = sim.current_buffer()
            behind.append(sbs.film_volume_device(stale.ptr, H, W, stale.pitch, 0.025))
        vols = sim.run_checked(0.0, 24, 6)
        cau = sim.run_caustic_map(5)
        out.append((sim.thickness_array(), sim.concentration_array(), cau, vols, behind))
    for got in out[:2]:
        for a, b in zip(got[:3], out[2][:3]):
            np.testing.assert_array_equal(a, b)
        np.testing.assert_allclose(got[3], out[2][3], rtol=1e-12)
        np.testing.assert_allclose(got[4], out[2][4], rtol=1e-12)


@pytest.mark.parametrize("marangoni", [0, 1])
@pytest.mark.parametrize("W,H", [(9, 5), (11, 40), (119, 37), (121, 64), (122, 33), (243, 70), (1037, 131), (2051, 40),
                                 (2177, 33), (4099, 20)])
def test_ragged_widths_on_the_blocked_route_match_single_steps(sbs, orc, W, H, marangoni):
    """Widths that are no multiple of four cells in the blocked kernel (the seam inside a lane's window, one
    and several 120-column segments, a window that wraps more than once; rows of more than 2048 columns are
    blocked by default): the bits of single steps and of the kernel-order oracle, volumes, and the fused
    caustic map after every remainder."""
    from soap_bubble_simulation_gb300 import synthetic

    h = synthetic.smooth_modes(H, W, seed=W + H).astype(np.float32)
    h[H // 3, : W // 4] = 25e-9  # a patch below the critical thickness
    h[2 * H // 3, W // 2] = 1e-4  # a spike that is clamped at zero around it
    c = synthetic.surfactant_noise(H, W, seed=H)
    c[1, :3] = (0.0, 1.0, 0.5)
    out = []
    for route in ("blocked", "single"):
        sim = sbs.GPUDrainageSimulator(None, 500e-9, W, H)
        if W <= 2048 or route == "single":
            sim.route = route
        assert sim.route == route
        sim.set_thickness_array(h)
        sim.set_concentration_array(c)
        sim.set_marangoni_enabled(bool(marangoni))
        vols = sim.run_checked(0.001, 22, 11)
        maps = [sim.run_caustic_map(n) for n in (3, 4, 6, 9, 11)]
        out.append((sim.thickness_array(), sim.concentration_array(), vols, maps))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_allclose(out[0][2], out[1][2], rtol=1e-12)
    for a, b in zip(out[0][3], out[1][3]):
        np.testing.assert_array_equal(a, b)
    p = orc.wgsl_params(grid_width=W, grid_height=H, marangoni_enabled=marangoni)
    ho, co = orc.wgsl_run(p, h, c, 55, "kernel")
    np.testing.assert_array_equal(out[0][0], ho)
    np.testing.assert_array_equal(out[0][1], co)


@pytest.mark.parametrize("precision", ["f32x2", "f32"])
@pytest.mark.parametrize("res", [11, 33, 61, 121, 305, 1025])
def test_odd_resolutions_on_the_blocked_route_match_single_steps(sbs, orc, precision, res):
    """Odd resolutions (rows of 2 r cells, no multiple of four; pole rings of one and several blocks) in
    the blocked kernel (1025 by default): the bits of single steps and, the smaller ones, of the
    kernel-order oracle, fronts active (first spawn at step 50), volumes."""
    from soap_bubble_simulation_gb300 import synthetic

    h0 = synthetic.bubble_c0(res, seed=res)
    h0[res // 3, : res // 2] = 5e-9  # below the 10 nm critical thickness: frozen
    h0[1, : res // 3] *= 40.0
    if precision == "f32":
        h0 = h0.astype(np.float32).astype(np.float64)
    dt = 0.01 if res < 1000 else 2e-5
    out = []
    for route in ("blocked", "single"):
        sim = make_sim(sbs, res, precision)
        if res < 1000 or route == "single":
            sim.route = route
        assert sim.route == route
        if res >= 1000:
            sim.step_n(0.01, 70)  # a uniform film stays stable; its clock brings the first front
        set64(sbs, sim, h0)
        sim.step_n(dt, 47)
        vols = sim.run_checked(dt, 34, 17)
        out.append((field64(sbs, sim), vols, sim.active_tfe_count()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=1e-12)
    assert out[0][2] == out[1][2] >= 1
    if res < 1000:
        ref = orc.CpuSim(resolution=res, precision=ORC_PREC[precision])
        ref.set_field(h0)
        ref.step_n(dt, 81)
        np.testing.assert_array_equal(out[0][0], ref.field())


RING_EDGES = {  # words of a ring around the range of its 128-bit sums: [2^-47, 2^-16) m and 0, low words to 2^-41 m
    "below 2^-16": np.nextafter(np.float32(2.0**-16), np.float32(0)), "2^-16": 2.0**-16,
    "below 2^-16, low word 2^-41": float(np.nextafter(np.float32(2.0**-16), np.float32(0))) - 2.0**-41,
    "below 2^-16, low word over it": float(np.nextafter(np.float32(2.0**-16), np.float32(0))) + 2.0**-41 - 2.0**-66,
    "2^-47": 2.0**-47, "below 2^-47": np.nextafter(np.float32(2.0**-47), np.float32(0)), "zero": 0.0,
    "tiny": 1e-30, "large": 5.0, "huge": 1e9}


@pytest.mark.parametrize("route", ["resident", 2, 3, 4])
@pytest.mark.parametrize("res", [33, 256, 512])
def test_pole_ring_words_at_the_edges_of_the_narrow_sums(sbs, orc, res, route):
    """Such words in the first, the last or all of the ring's column blocks (1, 2 and 3 of them in the
    blocked kernel, one in the resident one), at either pole: the kernel-order oracle's bits."""
    from soap_bubble_simulation_gb300 import synthetic

    base = synthetic.bubble_c0(res, seed=5)
    np_ = 2 * res
    sim = make_sim(sbs, res, "f32x2")
    if route == "resident" or res % 2:  # odd: blocked with the default K
        sim.route = "resident" if route == "resident" else "blocked"
    else:
        set_cpu_blocking(sbs, sim, route)
    assert sim.route == ("resident" if route == "resident" else "blocked")
    for k, value in enumerate(RING_EDGES.values()):
        h0 = base.copy()
        h0[1, (3, np_ - 2, np_ // 2)[k % 3]] = value
        h0[res - 2, (np_ - 1, slice(0, np_, 7), 0)[k % 3]] = value
        set64(sbs, sim, h0)
        sim.step_n(1e-9, 13)
        ref = orc.CpuSim(resolution=res, precision=ORC_PREC["f32x2"])
        ref.set_field(h0)
        ref.step_n(1e-9, 13)
        np.testing.assert_array_equal(field64(sbs, sim), ref.field())


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, -1.0, 3e38, 1e-42])
@pytest.mark.parametrize("marangoni", [0, 1])
@pytest.mark.parametrize("W,H", [(132, 40), (131, 40)])
def test_unusual_values_are_the_same_on_every_route(sbs, W, H, marangoni, bad):
    """NaN, infinities, negative, enormous and denormal cells in either field (WGSL semantics)."""
    from soap_bubble_simulation_gb300 import synthetic

    h = synthetic.smooth_modes(H, W, seed=W).astype(np.float32)
    c = synthetic.surfactant_noise(H, W, seed=H)
    for k, (i, j) in enumerate([(1, 0), (H - 2, W - 1), (H // 2, W // 2), (7, 120)]):
        (h if k % 2 else c)[i, j] = np.float32(bad)
    h[20, 3] = np.float32(bad)
    out = []
    for route in ("single", "blocked", "resident"):
        sim = sbs.GPUDrainageSimulator(None, 500e-9, W, H)
        sim.route = route
        sim.set_thickness_array(h)
        sim.set_concentration_array(c)
        sim.set_marangoni_enabled(bool(marangoni))
        sim.run(14)
        out.append((sim.thickness_array(), sim.concentration_array()))
    for got in out[1:]:
        for a, b in zip(got, out[0]):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, -1.0, 3e38, 1e-42])
@pytest.mark.parametrize("precision", ["f32x2", "f32"])
@pytest.mark.parametrize("res", [66, 61])
def test_unusual_cpu_values_are_the_same_on_every_route(sbs, res, precision, bad):
    """The same in DrainageSimulator semantics, in a pole ring and inside, a front active."""
    from soap_bubble_simulation_gb300 import synthetic

    h0 = synthetic.bubble_c0(res, seed=res)
    for i, j in [(1, 0), (res - 2, 2 * res - 1), (res // 2, res), (9, 119)]:
        h0[i, j] = np.float32(bad)
    out = []
    for route in ("single", "blocked", "resident"):
        sim = make_sim(sbs, res, precision)
        sim.route = route
        sim.step_n(0.01, 60)  # the first front
        set64(sbs, sim, h0)
        sim.step_n(1e-4, 13)
        out.append(field64(sbs, sim))
    np.testing.assert_array_equal(out[1], out[0])
    np.testing.assert_array_equal(out[2], out[0])


def test_handles_of_several_threads(sbs):
    """Handles of every route stepped at once by several threads: the fields of one thread alone."""
    from concurrent.futures import ThreadPoolExecutor

    from soap_bubble_simulation_gb300 import synthetic

    jobs = [("wgsl", 64, 128, "resident"), ("wgsl", 700, 1400, "resident"), ("cpu", 128, 0, "resident"),
            ("cpu", 256, 0, "blocked"), ("wgsl", 300, 2052, "blocked"), ("cpu", 512, 0, "resident")]

    def run(job):
        kind, nt, np_, route = job
        if kind == "cpu":
            sim = make_sim(sbs, nt)
            set64(sbs, sim, synthetic.bubble_c0(nt, seed=nt))
        else:
            sim = sbs.GPUDrainageSimulator(None, 500e-9, np_, nt)
            sim.set_thickness_array(synthetic.smooth_modes(nt, np_, seed=nt).astype(np.float32))
            sim.set_dt(1e-5)
        sim.route = route
        for _ in range(12):
            sim.step_n(1e-6, 70) if kind == "cpu" else sim.run(70)
        return sim.thickness_array()

    want = [run(j) for j in jobs]
    with ThreadPoolExecutor(len(jobs)) as pool:
        for got, w in zip(pool.map(run, jobs), want):
            np.testing.assert_array_equal(got, w)


@pytest.mark.parametrize("marangoni", [0, 1])
def test_handles_that_share_the_chip(sbs, orc, marangoni):
    """Eight threads with handles that alone fill the chip leave the resident route while they run at once:
    the fields of one thread alone, volumes, the caustic map."""
    from concurrent.futures import ThreadPoolExecutor

    from soap_bubble_simulation_gb300 import synthetic

    sizes = [(512, 1024), (517, 1037), (300, 600), (64, 128), (900, 1801), ("cpu", 512), ("cpu", 305), (40, 2051)]

    def run(size):
        if size[0] == "cpu":
            sim = make_sim(sbs, size[1])
            set64(sbs, sim, synthetic.bubble_c0(size[1], seed=size[1]))
        else:
            nt, np_ = size
            sim = sbs.GPUDrainageSimulator(None, 500e-9, np_, nt)
            sim.set_thickness_array(synthetic.smooth_modes(nt, np_, seed=nt).astype(np.float32))
            sim.set_dt(1e-5)
            sim.set_marangoni_enabled(bool(marangoni))
        vols, maps = [], []
        for n in (300, 7, 64, 100, 33):
            vols.append(sim.run_checked(1e-6, n, 25))
            if size[0] != "cpu":
                maps.append(sim.run_caustic_map(9))
        return sim.thickness_array(), maps, np.concatenate(vols)

    want = [run(s) for s in sizes]
    with ThreadPoolExecutor(len(sizes)) as pool:
        for _ in range(3):
            for got, w in zip(pool.map(run, sizes), want):
                np.testing.assert_array_equal(got[0], w[0])
                for a, b in zip(got[1], w[1]):
                    np.testing.assert_array_equal(a, b)
                np.testing.assert_allclose(got[2], w[2], rtol=1e-12)
