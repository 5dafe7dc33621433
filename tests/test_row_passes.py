"""The row passes at the row counts where another kernel or lane count takes them: eight lanes a
row up to 16,384 fluid rows, four up to 49,152, a thread above.  Forward passes add a row's terms
in list order on every path, so a scene gives the same bits on each; adjoint sums are split over
lanes and agree to rounding."""
import numpy as np
import pytest

from vtp import scenes

pytestmark = pytest.mark.gpu


def _filler(kind, n):
    """n fluid particles at rest spacing in a box of their own; a batch of them and another scene
    has that many rows more."""
    sp = 0.02 if kind == "PBF" else 0.01
    side = int(np.ceil(n ** (1 / 3)))
    g = (np.arange(side, dtype=np.float32) + np.float32(5)) * np.float32(sp)
    z, y, x = np.meshgrid(g, g, g, indexing="ij")
    p = scenes.jitter(np.stack([x.ravel(), y.ravel(), z.ravel()], 1)[:n], 0.05, sp, n)
    make = scenes.pbf_config if kind == "PBF" else scenes.dfsph_config
    cfg = make(dt=1.0 / 240.0 if kind == "PBF" else 1e-3, r=sp / 2, lb=(0.0,) * 3, size=((side + 10) * sp,) * 3)
    return scenes.Scene(kind, cfg, [scenes.SceneObject("fluid", p, 0)])


def _state(s, lo, hi):
    names = ("pos", "vel", "density")
    return [s.get_field(k)[lo:hi].copy() for k in names]


@pytest.mark.parametrize("kind", ["PBF", "DFSPH"])
@pytest.mark.parametrize("n_probe", [33, 3000])
def test_rows_give_the_same_bits_on_every_path(vtp_gpu, kind, n_probe):
    """A scene alone (eight lanes a row) and behind a filler of such a size that the solver's rows
    are the last of one path or the first of the next; its rows then begin anywhere in a block."""
    probe = scenes.dam_break(kind, n_probe, seed=n_probe)
    nf = probe.n_fluid
    s = vtp_gpu.solver_from_scene(probe)
    assert s.tickNsteps(3), s.last_error
    want = _state(s, 0, probe.n_total)
    iters = s.stats()["total_div_iters"]
    s.destroy()
    assert np.isfinite(want[0]).all()
    for rows in (16384, 16385, 49152, 49153):
        b, ranges = vtp_gpu.solver_from_scenes([_filler(kind, rows - nf), probe])
        assert b.initialize(), b.last_error
        assert b.tickNsteps(3), b.last_error
        lo, hi = ranges[1]
        for name, x, y in zip(("pos", "vel", "density"), _state(b, lo, hi), want):
            assert np.array_equal(x, y), (rows, name)
        if kind == "DFSPH":
            assert b.scene_stats(1)["total_div_iters"] == iters
        b.destroy()


@pytest.mark.parametrize("kind", ["PBF", "DFSPH"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33])
def test_smallest_scenes_match_the_oracle(vtp_gpu, oracle_lib, kind, n):
    """A block of lanes with rows to spare, one row short and one over.  FP32 against FP64 over one
    substep: positions and velocities within the 1e-5 of their largest value that the one-substep
    parity tests allow (a step moves a particle by well under its spacing)."""
    sc = _filler(kind, n)
    s = vtp_gpu.solver_from_scene(sc)
    assert s.tickNsteps(1), s.last_error
    o = oracle_lib.OracleSolver(sc)
    o.step(1)
    for got, want in ((s.get_field("pos"), o.pos), (s.get_field("vel"), o.vel)):
        # the velocity is (x1 - x0) / dt in FP32: an ulp of x, 240 times over, for PBF
        floor = np.abs(want).max() + (np.abs(o.pos).max() * 240 if kind == "PBF" else 0.0)
        assert np.abs(got.astype(np.float64) - want).max() <= 1e-5 * floor
    s.destroy()


@pytest.mark.parametrize("n", [400, 26000, 52000])
def test_adjoint_lanes_chosen_by_rows_match_one_thread(vtp_gpu, n):
    """8 lanes a row up to 24,576 fluid rows, 4 up to 49,152, 2 above, against one thread.  A sum of
    60 terms in another order is off by at most 60 * 2^-24 = 3.6e-6 of its terms' size; two substeps
    of four iterations of three passes carry 24 of them: 1e-4."""
    from vtp import diff
    sc = scenes.dam_break("PBF", n, seed=n)
    mask = diff.fluid_mask(sc)
    rng = np.random.default_rng(n)
    bar = np.where(mask[:, None], rng.normal(size=(mask.size, 3)), 0.0).astype(np.float32)
    got = []
    for extra in ({}, {"adjointLanes": 1}):
        s = diff.pbf_solver(sc, extra=extra)
        diff.diff_forward(s, 2, 1)
        got.append(diff.diff_backward(s, bar, None))
        s.destroy()
    for a, b in zip(got[0][:2], got[1][:2]):
        assert np.linalg.norm(a[mask].astype(np.float64) - b[mask]) <= 1e-4 * np.linalg.norm(b[mask])
    assert abs(got[0][2] - got[1][2]) <= 1e-4 * abs(got[1][2]) + 1e-12


def test_fractions_are_read_in_attach_order(vtp_gpu):
    """The boundary's fractions are the attached ones, and the fluid's follow their particles: before
    any exchange every particle holds its own layer's, whatever order the rows are in."""
    sc = scenes.layered_mixture("IMM", 12, seed=2)
    fluid = np.concatenate([np.full(o.n, o.material == 0) for o in sc.objects])
    s = vtp_gpu.solver_from_scene(sc)
    assert s.initialize(), s.last_error
    first = s.get_field("vol_frac")
    attached = np.concatenate([np.tile(np.asarray(o.phase_fraction, np.float32), (o.n, 1)) for o in sc.objects
                               if o.material == 0])
    assert np.array_equal(first[fluid], attached)
    assert s.tickNsteps(3), s.last_error
    after = s.get_field("vol_frac")
    assert np.array_equal(after[~fluid], first[~fluid])
    assert np.array_equal(s.get_field("vol_frac"), after)
    assert np.abs(after[fluid].astype(np.float64).sum(1) - 1.0).max() < 1e-5
    s.destroy()


def _bits(s, lo, hi):
    return _state(s, lo, hi) + [np.array([s.stats()[k] for k in ("total_div_iters", "total_incomp_iters")])]


@pytest.mark.parametrize("n_side, tension", [(7, 0.001), (13, 0.001), (13, 0.0)])
def test_tension_and_objects_give_the_same_bits_on_every_path(vtp_gpu, n_side, tension):
    """Two fluid objects (a residual mean each) with and without surface tension: alone (eight lanes a
    row), in a batch whose rows are the last of one path or the first of the next, and with a thread
    per row asked for by "persistentTiles"."""
    probe = scenes.colliding_blocks(3, tension, n_side=n_side)
    nf = probe.n_fluid
    s = vtp_gpu.solver_from_scene(probe)
    assert s.tickNsteps(6), s.last_error
    want = _bits(s, 0, probe.n_total)
    s.destroy()
    assert np.isfinite(want[0]).all() and want[3].min() > 0
    t = vtp_gpu.solver_from_scene(probe, extra={"persistentTiles": True})
    assert t.tickNsteps(6), t.last_error
    for x, y in zip(_bits(t, 0, probe.n_total), want):
        assert np.array_equal(x, y)
    t.destroy()
    for rows in (16384, 16385, 49152, 49153):
        filler = _filler("DFSPH", rows - nf)
        filler.config["DFSPH"]["Required"]["surfaceTensionCoefficient"] = tension
        b, ranges = vtp_gpu.solver_from_scenes([filler, probe])
        assert b.initialize(), b.last_error
        assert b.tickNsteps(6), b.last_error
        for name, x, y in zip(("pos", "vel", "density"), _state(b, *ranges[1]), want):
            assert np.array_equal(x, y), (rows, name)
        stats = b.scene_stats(1)
        assert [stats["total_div_iters"], stats["total_incomp_iters"]] == list(want[3]), rows
        b.destroy()


@pytest.mark.parametrize("kind, extra", [("PBF", {"pbfFormulation": "standard"}), ("DFSPH", {"cfl": 0.4}),
                                         ("DFSPH", {"blockSize": 96}), ("DFSPH", {"blockSize": 256, "unroll": 1})])
@pytest.mark.parametrize("n", [3000, 30000])
def test_options_give_the_same_bits_with_and_without_teams(vtp_gpu, kind, extra, n):
    """Eight and four lanes a row against a thread: the standard PBF kernels, the adaptive step, and
    residual tiles of three and eight warps."""
    sc = scenes.dam_break(kind, n, seed=n)
    got = []
    for more in ({}, {"persistentTiles": True}):
        s = vtp_gpu.solver_from_scene(sc, extra={**extra, **more})
        assert s.tickNsteps(4), s.last_error
        got.append(_bits(s, 0, sc.n_total))
        s.destroy()
    for x, y in zip(*got):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("kind", ["IMM", "IMMCT"])
def test_unroll_of_one_gives_a_small_mixture_the_same_bits(vtp_gpu, kind):
    """The entries of a row are used in list order whatever "unroll" is.  (Larger mixtures agree to
    rounding: which product the drift and diffusion sums fuse is the compiler's choice for each.)"""
    sc = scenes.layered_mixture(kind, 14, seed=3)
    got = []
    for unroll in (4, 2, 1):
        s = vtp_gpu.solver_from_scene(sc, extra={"unroll": unroll})
        assert s.tickNsteps(3), s.last_error
        got.append([s.get_field(k) for k in ("pos", "vel", "vol_frac", "phase_vel")])
        s.destroy()
    for other in got[1:]:
        for x, y in zip(got[0], other):
            assert np.array_equal(x, y)


def test_a_staged_solver_takes_a_thread_per_row(vtp_gpu):
    """The staged solve's kernels read a list's entries a thread per row, in lists laid out for that;
    the other passes then read the same lists, whatever the row count."""
    import torch
    s = vtp_gpu.solver_from_scene(scenes.dam_break("DFSPH", 3000, seed=2), extra={"stagedSolve": True})
    assert s.initialize(), s.last_error
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        s.profile_kernels(1)
        torch.cuda.synchronize()
    names = " ".join(e.key for e in prof.key_averages())
    s.destroy()
    assert "k_solve_a_staged" in names and "k_viscosity" in names and "k_team" not in names
