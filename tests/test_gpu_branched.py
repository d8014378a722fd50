"""Branched flow on the GPU (sbs_branched_flow) against the oracle's literal restatement of
branched_flow_compute.wgsl: the texture bit for bit. Every operation is the same FP32 sequence on
both sides (acos / atan2 / exp included: the library's own published approximations) and the
deposits are integer atomic adds, whose order does not matter."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def br(sbs):
    from soap_bubble_simulation_gb300 import branched

    return branched


def field(nt=64, np_=128, seed=3, scale=1.0):
    from soap_bubble_simulation_gb300 import synthetic as S

    return (S.smooth_modes(nt, np_, seed=seed) * scale).astype(np.float32)


@pytest.mark.parametrize("kw", [{}, {"patch_enabled": 0}, {"particle_weight": 0.6, "bend_strength": 9.0},
                                {"entry_point": (0.0, 1.0, 0.0), "patch_enabled": 0},
                                {"intensity_falloff": 0.02, "spread_angle": 1.2}])
def test_texture_matches_oracle(sbs, orc, br, kw):
    p = br.BranchedFlowParams.default()
    p.num_rays = 2048
    for k, v in kw.items():
        if k == "entry_point":
            for i, x in enumerate(v):
                p.entry_point[i] = x
        else:
            setattr(p, k, v)
    th = field(scale=2e4)  # thickness in um-ish units so that the GRIN kick matters
    sc = br.generate_scatterers(p, time=1.5)
    tex0 = np.random.default_rng(0).integers(0, 5000, (p.tex_height, p.tex_width)).astype(np.uint32)
    got = br.branched_flow_step(p, th, sc, tex0, fade=True)
    want = orc.branched_flow(p, th, sc, tex0, fade=True)
    assert np.array_equal(got, want), (int(np.abs(got.astype(np.int64) - want).max()), int((got != want).sum()))
    assert got.sum() > tex0.sum() * 0.85 * 0.9  # the rays deposited


def test_simulator_steps(sbs, br):
    sim = br.BranchedFlowSimulator()
    sim.params.num_rays = 4096
    sim.params.patch_enabled = 0  # the default entry point (u = 0.75) lies outside the default patch
    th = field(scale=2e4)
    t1 = sim.step(th, 0.0).copy()
    t2 = sim.step(th, 0.016)
    assert t1.sum() > 0 and t2.sum() > t1.sum()  # fade x 0.85 plus a new frame of deposits
    assert sim.texture_size() == (512, 256)


def test_bad_arguments(sbs, br):
    p = br.BranchedFlowParams.default()
    with pytest.raises(ValueError):
        br.branched_flow_step(p, field(), np.zeros((10, 4), np.float32), np.zeros((256, 512), np.uint32))
    p.tex_width = 1
    with pytest.raises(sbs.SbsError):
        br.branched_flow_step(p, field(), br.generate_scatterers(br.BranchedFlowParams.default()),
                              np.zeros((256, 1), np.uint32))


@pytest.mark.parametrize("rays", [1, 33, 10000, 10001, 24000, 24001])
def test_every_number_of_lanes_per_ray_matches_oracle(sbs, orc, br, rays):
    """Ray counts at the edges of the rule that gives a ray 4, 2 or 1 lanes; scatterers of very
    different cutoffs (one covers the whole film, one nothing), more than 128 of them in a cell's list."""
    p = br.BranchedFlowParams.default()
    p.num_rays, p.patch_enabled, p.ray_steps, p.num_scatterers = rays, 0, 60, 700
    g = np.random.default_rng(rays)
    sc = br.generate_scatterers(p, time=0.5)
    sc[:200, :2] = 0.45 + 0.1 * g.random((200, 2))
    sc[5, 3], sc[6, 3], sc[7, 3] = 0.5, 1e9, 40.0
    th = field(scale=2e4)
    tex0 = np.zeros((p.tex_height, p.tex_width), np.uint32)
    got = br.branched_flow_step(p, th, sc, tex0, fade=False)
    assert np.array_equal(got, orc.branched_flow(p, th, sc, tex0, False))
    assert got.sum() > 0


@pytest.mark.parametrize("kw,scale", [({"bend_strength": 1e17}, 2e4), ({"bend_strength": 1e24}, 2e4),
                                      ({"bend_strength": -1e33, "particle_weight": 0.5}, 2e4),
                                      ({"spread_angle": 1e16}, 2e4), ({"spread_angle": 1e23}, 2e4),
                                      ({}, 1e43), ({"step_size": 1e30}, 2e4)])
@pytest.mark.parametrize("rays", [2000, 30000])
def test_values_whose_squares_overflow_match_oracle(sbs, orc, br, kw, scale, rays):
    """Velocities and positions on both sides of where a length's square is infinite: the division by
    an infinite length gives zero, and the ray goes on."""
    p = br.BranchedFlowParams.default()
    p.num_rays, p.patch_enabled, p.ray_steps = rays, 0, 40
    for k, v in kw.items():
        setattr(p, k, v)
    with np.errstate(over="ignore"):
        th = field(scale=scale)
    sc = br.generate_scatterers(p, time=1.5)
    tex0 = np.zeros((p.tex_height, p.tex_width), np.uint32)
    got = br.branched_flow_step(p, th, sc, tex0, fade=False)
    assert np.array_equal(got, orc.branched_flow(p, th, sc, tex0, False))


@pytest.mark.parametrize("scatterers,clustered", [(0, 0), (1, 0), (12, 0), (40, 8), (40, 9), (60, 33)])
@pytest.mark.parametrize("rays", [500, 25000])
def test_short_lists_match_oracle(sbs, orc, br, rays, scatterers, clustered):
    """Lists of no scatterers up to both sides of the length that is walked without masks."""
    p = br.BranchedFlowParams.default()
    p.num_rays, p.patch_enabled, p.ray_steps, p.num_scatterers = rays, 0, 60, scatterers
    sc = br.generate_scatterers(p, time=0.5)
    if clustered:  # `clustered` of them share a cell, the others one far away
        g = np.random.default_rng(clustered)
        sc[:clustered, :2] = 0.72 + 0.06 * g.random((clustered, 2))
        sc[clustered:, :2] = 0.03 + 0.005 * np.arange(scatterers - clustered)[:, None] * np.array([[0.0, 1.0]])
    th = field(scale=2e4)
    tex0 = np.zeros((p.tex_height, p.tex_width), np.uint32)
    got = br.branched_flow_step(p, th, sc, tex0, fade=False)
    assert np.array_equal(got, orc.branched_flow(p, th, sc, tex0, False))


def test_threads_with_different_numbers_of_scatterers(sbs, br):
    """Calls of several threads whose blocks want different amounts of shared memory."""
    from concurrent.futures import ThreadPoolExecutor

    th = field(scale=2e4)

    def run(n, times=1):
        p = br.BranchedFlowParams.default()
        p.num_rays, p.patch_enabled, p.ray_steps, p.num_scatterers = 300, 0, 5, n
        sc = br.generate_scatterers(p, time=0.5)
        return [br.branched_flow_step(p, th, sc, np.zeros((p.tex_height, p.tex_width), np.uint32), fade=False)
                for _ in range(times)]

    sizes = (0, 400, 1200, 2000)
    want = [run(n)[0] for n in sizes]
    with ThreadPoolExecutor(4) as pool:
        for got, w in zip(pool.map(lambda n: run(n, 40), sizes), want):
            for t in got:
                np.testing.assert_array_equal(t, w)
