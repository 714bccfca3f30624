"""Edges of the engine's dispatch: launch shapes by block count, domain sizes of the
compaction, the stresses' fallback, adaptive graphs, and the differentiable rollout's
particle order and tiles.  Where two routes compute the same thing, they are
compared bit for bit; the stresses against the FP64 oracle."""
import math

import numpy as np
import pytest

from ckmpm_b200 import Scene, scenes
from ckmpm_b200 import _capi as capi
from ckmpm_b200.engine import MPMConfig, MPMMaterial, MPMModel, compute_lame_parameters

pytestmark = pytest.mark.gpu


def rotations(rng, n):
    q, _ = np.linalg.qr(rng.normal(size=(n, 3, 3)))
    q[np.linalg.det(q) < 0, :, 0] *= -1
    return q


def box_scene(n, blocks, dx=1 / 64, ppc=8, kind="fixed_corotated", seed=0, v0=(0.4, -1.0, 0.3)):
    """A jittered cube of about n particles in the middle of a domain of `blocks`, at cell size dx."""
    rng = np.random.default_rng(seed)
    half = 0.5 * (n / ppc) ** (1 / 3) * dx
    c = 2.0 * np.asarray(blocks) * dx + 0.1 * dx
    x = scenes.box_particles(c - half, c + half, dx, ppc, rng)
    lam, mu = compute_lame_parameters(5e4, 0.3)
    mat = MPMMaterial.fluid(1e4, 7.15, 0.1) if kind == "fluid" else getattr(MPMMaterial, kind)(lam, mu)
    vol = dx ** 3 / ppc
    v = (np.asarray(v0) + 4.0 * (x - c)[:, [1, 2, 0]]).astype(np.float32)
    return MPMConfig(dx=dx, domain_blocks=tuple(blocks)), [MPMModel(1000 * vol, vol, x, v, mat)]


def run(cfg, models, steps, tuning=None, dt=1e-4):
    s = Scene(cfg)
    for m in models:
        s.add_model(m)
    if tuning:
        s.set_tuning(*tuning)
    s.setup()
    s.step(steps, dt)
    return s


def assert_same(a, b, what):
    for name in ("x", "v", "F", "aux"):
        p, q = getattr(a, name), getattr(b, name)
        assert np.array_equal(p.view(np.uint32), q.view(np.uint32)), (what, name)
    assert np.array_equal(a.id, b.id), what


@pytest.mark.parametrize("kind", ["fixed_corotated", "drucker_prager", "fluid"])
@pytest.mark.parametrize("n,blocks", [(40, 12), (17000, 12), (45000, 14), (100000, 16)])
def test_split_blocks_give_the_same_bits(engine_lib, kind, n, blocks):
    """The default shape (blocks split over clusters of 4 or 2 CTAs, or not, by their number)
    against one CTA per block, with the particles crossing block faces."""
    cfg, models = box_scene(n, (blocks,) * 3, kind=kind)
    a = run(cfg, models, 33)
    b = run(cfg, models, 33, (256, 4, 8))
    c = run(cfg, models, 33, (1024, 1, 8))
    assert_same(a.state(0), b.state(0), "default")
    assert_same(c.state(0), b.state(0), "clusters")
    for which in (0, 1, 2):
        for p, q in zip(a.blocks(0, which), b.blocks(0, which)):
            assert np.array_equal(p, q)


def test_a_spreading_scene_outgrows_its_clusters(engine_lib):
    """A cloud set up with so few blocks that each is split over 4 CTAs, flying apart to more blocks than
    clusters within its graphs: the same bits as with one CTA per block throughout, and no slower than that
    (2.7 times as slow while the split stayed as it was set up; the bound is 1.4)."""
    cfg, models = box_scene(17000, (20, 20, 20), kind="drucker_prager", v0=(0.0, 0.0, 0.0))
    cfg.gravity = 0.0
    x = models[0].particle_position
    models[0].particle_velocity = (30.0 * (x - x.mean(0))).astype(np.float32)
    scene = [run(cfg, models, 0), run(cfg, models, 0, (256, 4, 8))]
    sms = 148
    assert scene[0].tuning()["threads"] == 1024 and len(scene[0].blocks(0, 0)[1]) <= sms
    for _ in range(5):
        for s in scene:
            s.step(56, 1e-4)
        assert_same(scene[0].state(0), scene[1].state(0), "spreading")
    assert len(scene[0].blocks(0, 0)[1]) > 2 * sms
    ms = [min(s.step_profiled(16, 1e-7)[0] for _ in range(5)) for s in scene]
    assert ms[0] < 1.4 * ms[1], ms


@pytest.mark.parametrize("n,small,large", [(130000, 16, 26), (460000, 24, 26)])
def test_small_domain_is_no_slower_than_a_large_one(engine_lib, n, small, large):
    """A body of many blocks in a domain whose compaction also zeroes the next windows, against the same body
    in the smallest domain that gives the zeroing a launch of its own: no slower (1.2
    times as slow at 343 blocks while one CTA per tile did the zeroing; the bound is 1.1)."""
    import time
    scene = [run(*box_scene(n, (b,) * 3, kind="drucker_prager", v0=(0.0, 0.0, 0.0)), 0) for b in (small, large)]
    seconds = [math.inf, math.inf]
    for _ in range(9):
        for k, s in enumerate(scene):
            t = time.perf_counter()
            s.step(64, 1e-7)
            seconds[k] = min(seconds[k], time.perf_counter() - t)
    assert len(scene[0].blocks(0, 0)[1]) >= 300
    assert seconds[0] < 1.1 * seconds[1], seconds


@pytest.mark.parametrize("blocks,bodies", [(12, 1), (12, 2), (26, 2)])
def test_profiled_substeps_are_the_ones_that_run(engine_lib, blocks, bodies):
    """step_profiled launches the kernels of step, in small and large domains, for one model and two, and moves
    the scene alike."""
    torch = pytest.importorskip("torch")
    cfg, models = box_scene(5000, (blocks,) * 3)
    if bodies == 2:
        models += box_scene(3000, (blocks,) * 3, kind="fluid", seed=1)[1]
    plain, profiled = run(cfg, models, 0), run(cfg, models, 0)

    def kernels(step):
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            step()
            torch.cuda.synchronize()
        return sorted((e.key, e.count) for e in prof.key_averages() if "compact" in e.key or "zero_windows" in e.key)

    a, b = kernels(lambda: plain.step(7, 1e-4)), kernels(lambda: profiled.step_profiled(7, 1e-4))
    if not a and not b:
        pytest.skip("no kernel records here (another profiler holds them)")
    assert a == b
    for m in range(bodies):
        assert_same(profiled.state(m), plain.state(m), m)


@pytest.mark.parametrize("n", [40, 17000, 60000])
def test_cam_clay_gives_the_same_bits_everywhere(engine_lib, n):
    """Cam-clay's F jumps with its last bit (F = U diag(S) V, V not transposed), so its own
    transfers must agree bit for bit between launch shapes."""
    cfg, models = box_scene(n, (14, 14, 14))
    lam, mu = compute_lame_parameters(2e4, 0.4)
    models[0].material = MPMMaterial.nacc(mu, lam, -0.01, 0.5, 0.8, 2.36, True)
    a = run(cfg, models, 33, (256, 4, 8)).state(0)
    for shape in (None, (128, 5, 8), (192, 4, 8), (1024, 1, 8)):
        assert_same(run(cfg, models, 33, shape).state(0), a, shape)


@pytest.mark.parametrize("n,dx", [(40, 1 / 64), (17000, 1 / 64), (17000, 1 / 37)])
def test_cam_clay_gives_the_same_bits_in_every_kernel(engine_lib, n, dx):
    """The rigid form and the mixed kernel of a batch (a von Mises scene beside two of clay) against the single
    scene's kernel, with particles on the faces of cells and blocks and an ulp beside them: every stencil lies in
    its block's window (a base cell other than the binning's raises a status)."""
    from ckmpm_b200.batch import SceneBatch
    cfg, models = box_scene(n, (14, 14, 14), dx=dx, v0=(0.4, -3.0, 0.3))
    lam, mu = compute_lame_parameters(2e4, 0.4)
    body = models[0]
    body.material = MPMMaterial.nacc(mu, lam, -0.01, 0.5, 0.8, 2.36, True)
    x = body.particle_position
    cells = np.rint(x[::3] / dx - 0.25) + 0.75  # faces of grid -dx/4's cells
    x[::3] = (cells * dx).astype(np.float32)
    x[::6] = np.nextafter(x[::6], np.float32(0))
    x[1::6] = np.nextafter(x[1::6], np.float32(1e3))
    ref = run(cfg, models, 33, (256, 4, 8))
    rigid = Scene(cfg)
    rigid.add_model(body)
    rigid.set_rigid(1, (0.1, 0.0, 0.0))
    rigid.setup()
    rigid.step(33, 1e-4)
    assert_same(rigid.state(0), ref.state(0), "rigid")
    metal = MPMModel(body.particle_mass, body.particle_volume, x, body.particle_velocity,
                     MPMMaterial.von_mises(mu, lam, 500.0))
    batch = SceneBatch(cfg, [body, metal, body])
    batch.setup()
    batch.step(33, 1e-4)
    for i in (0, 2):
        assert_same(batch.scene_state(i), ref.state(0), i)


@pytest.mark.parametrize("dims", [(9, 11, 13), (25, 25, 26), (26, 26, 26), (64, 17, 16)])
def test_domain_size_does_not_matter(engine_lib, dims):
    """The compaction's small and large tiles, odd extents among them: the same body far from
    any wall moves alike in every domain (positions are taken relative to its block)."""
    cfg, models = box_scene(5000, (10, 10, 10))
    ref = run(cfg, models, 40, (256, 4, 8))
    big = MPMConfig(dx=cfg.dx, domain_blocks=dims)
    s = run(big, models, 40)
    assert_same(s.state(0), ref.state(0), dims)
    for p, q in zip(s.blocks(0, 0), ref.blocks(0, 0)):
        assert np.array_equal(p, q)


@pytest.mark.parametrize("kind", [capi.FIXED_COROTATED, capi.DRUCKER_PRAGER, capi.VON_MISES])
def test_stress_of_ill_conditioned_deformation(engine_lib, oracle_mod, kind):
    """Stretches from well within to far beyond the ratio of 4 at which the return maps go back to
    the full SVD, and inverted ones for the fixed-corotated model.  The stretches are known to
    rounding of the largest, so log s to 2^-23 s_max / s_min: the tolerance on tau is
    8 of those times the stiffness."""
    rng = np.random.default_rng(11)
    n = 384
    ratio = np.exp(rng.uniform(0, math.log(40.0), n))
    s = np.stack([np.ones(n), ratio ** -rng.uniform(0, 1, n), 1 / ratio], 1) * np.exp(rng.uniform(-0.3, 0.3, (n, 1)))
    if kind == capi.FIXED_COROTATED:
        s[::7, 2] *= -1
    F = (rotations(rng, n) * s[:, None, :]) @ rotations(rng, n).transpose(0, 2, 1)
    F = F.astype(np.float32)
    lam, mu = 2.0e4, 3.0e4
    params = {capi.VON_MISES: [mu, lam, 500.0, 0.0]}.get(kind, [lam, mu, 0.0, 0.0])
    mat = capi.Material()
    mat.kind = kind
    for i, p in enumerate(params):
        mat.p[i] = p
    aux = np.full(n, 1.0 if kind == capi.VON_MISES else 0.0, np.float32)
    Fg, ag, tau = F.copy(), aux.copy(), np.zeros_like(F)
    C = np.zeros((n, 3, 3), np.float32)
    capi.check(engine_lib.ckmpm_debug_constitutive(mat, n, capi.fptr(C), 0.0, capi.fptr(Fg), capi.fptr(ag),
                                                   capi.fptr(tau), None, None, None), "debug")
    for i in range(n):
        Fo, ao, to = oracle_mod.constitutive(kind, params, np.zeros((3, 3)), 0.0, F[i].astype(np.float64), float(aux[i]))
        eps = 2.0 ** -23 * float(ratio[i])
        assert np.abs(tau[i] - to).max() <= 8 * eps * 5 * max(lam, mu) + 2e-5 * np.abs(to).max(), i
        assert np.abs(Fg[i] - Fo).max() <= 16 * eps + 2e-6, i


@pytest.mark.parametrize("branch", ["tension", "elastic", "plastic"])
def test_inverted_sand_leaves_unreflected(engine_lib, oracle_mod, branch):
    """Drucker-Prager writes F = U diag(exp h) V^T with rotations U and V, so an inverted F leaves with a positive
    determinant in every branch, at stretch ratios under and over the 4 at which the return map goes back to the
    full SVD.  F and the FP64 oracle's differ by the singular vectors' error, 2^-23 over the smallest gap of the
    squared stretches to the largest (the stretches are kept apart), times exp h: the tolerance is 32 of those."""
    rng = np.random.default_rng(5)
    n = 240
    ratio = np.exp(rng.uniform(math.log(1.3), math.log(40.0), n))
    s = np.stack([np.ones(n), ratio ** -rng.uniform(0.35, 0.65, n), 1 / ratio], 1)
    gap = np.minimum(1 - s[:, 1] ** 2, s[:, 1] ** 2 - s[:, 2] ** 2)
    s *= np.exp(rng.uniform(-0.3, 0.3, (n, 1)))
    volume = np.log(s).sum(1)
    aux = {"tension": 1.0 - volume, "elastic": np.full(n, -30.0), "plastic": -0.05 - volume}[branch].astype(np.float32)
    s[:, 2] *= -1
    F = ((rotations(rng, n) * s[:, None, :]) @ rotations(rng, n).transpose(0, 2, 1)).astype(np.float32)
    lam, mu = 2.0e4, 3.0e4
    mat = capi.Material()
    mat.kind = capi.DRUCKER_PRAGER
    mat.p[0], mat.p[1] = lam, mu
    Fg, ag, tau = F.copy(), aux.copy(), np.zeros_like(F)
    capi.check(engine_lib.ckmpm_debug_constitutive(mat, n, capi.fptr(np.zeros_like(F)), 0.0, capi.fptr(Fg),
                                                   capi.fptr(ag), capi.fptr(tau), None, None, None), "debug")
    assert (np.linalg.det(Fg.astype(np.float64)) > 0).all()
    for i in range(n):
        Fo, ao, to = oracle_mod.constitutive(capi.DRUCKER_PRAGER, [lam, mu, 0.0, 0.0], np.zeros((3, 3)), 0.0,
                                             F[i].astype(np.float64), float(aux[i]))
        eps = 2.0 ** -23
        assert np.abs(Fg[i] - Fo).max() <= 32 * eps / gap[i] * max(1.0, np.abs(Fo).max()), i
        assert np.abs(tau[i] - to).max() <= 8 * eps * float(ratio[i]) * 5 * max(lam, mu) + 2e-5 * np.abs(to).max(), i
        assert abs(ag[i] - ao) <= 16 * eps * float(ratio[i]), i


@pytest.mark.parametrize("boundary", ["sticky_blocks", "slip_floor"])
def test_adaptive_frame_equals_its_substeps(engine_lib, boundary):
    """A frame in one call (substeps replayed from graphs, the dt taken on the device) against the
    same frame one substep per call, and two frames of different bounds on one scene."""
    cfg, models = box_scene(6000, (12,) * 3, v0=(3.0, -4.0, 2.0))
    cfg.boundary = boundary
    whole, single = Scene(cfg), Scene(cfg)
    for s in (whole, single):
        s.add_model(models[0])
        s.setup()
    for dt, cfl, frame in ((1e-4, 0.02, 2.3e-3), (7e-5, 0.5, 1.7e-3)):
        whole.step_adaptive(1 << 20, dt, cfl, frame)
        left = frame
        while True:
            single.step_adaptive(1, dt, cfl, left)
            left = 0.0
            t, end = single.time()
            if not end - t > 0.0:
                break
        assert whole.counters()["steps"] == single.counters()["steps"]
        assert whole.time() == single.time()
    assert_same(whole.state(0), single.state(0), boundary)


@pytest.mark.parametrize("n,spread,every", [(1, 0.0, 1), (129, 0.02, 1), (700, 0.3, 4), (3000, 0.1, 1), (3000, 0.1, 7)])
def test_rollout_does_not_depend_on_the_particle_order(engine_lib, n, spread, every):
    """The rollout sorts its particles and deposits through per-CTA tiles, or directly where a CTA's
    particles lie too far apart (a sparse cloud): permuted inputs give permuted outputs and gradients,
    bit for bit, for every checkpoint interval."""
    torch = pytest.importorskip("torch")
    from ckmpm_b200.diff import DiffRollout
    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(n)
    cfg = MPMConfig(dx=1 / 64, domain_blocks=(16,) * 3)
    x = (0.5 + spread * (rng.random((n, 3)) * 2 - 1)).astype(np.float32)
    v = rng.normal(scale=0.5, size=(n, 3)).astype(np.float32)
    logE = (math.log(5e4) + 0.2 * rng.standard_normal(n)).astype(np.float32)
    gx, gF = rng.normal(size=(n, 3)).astype(np.float32), rng.normal(size=(n, 3, 3)).astype(np.float32)
    vol = (1 / 64) ** 3 / 8

    def outputs(order, k):
        t = [torch.from_numpy(np.ascontiguousarray(a[order])).to(dev) for a in (x, v, logE, gx, gF)]
        sim = DiffRollout(cfg, n, 1000 * vol, vol, nu=0.3, nsteps=9, dt=1e-4, checkpoint_every=k)
        res = []
        for _ in range(2):  # the second pass finds every sum as the first left it
            out = sim.forward(*t[:3])
            res.append([a.cpu().numpy() for a in (*out, *sim.backward(t[3], t[4], dev))])
        for a, b in zip(*res):
            assert np.array_equal(a, b)
        sim.close()
        return res[1]

    ref = outputs(np.arange(n), every)
    order = rng.permutation(n)
    for a, b in zip(ref, outputs(order, every)):
        assert np.array_equal(a[order], b)
    for a, b in zip(ref, outputs(np.arange(n), 2)):
        assert np.array_equal(a, b)
