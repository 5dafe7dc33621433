"""Neighbour lists of particles that do not lie as a fluid at rest: crowded cells, sparse clouds, and
occupancies that leave groups of every size.  The lists are the oracle's, and their time follows the
number of candidates: a crowded cell is spread over the GPU, and fewer candidates take no longer."""
import ctypes as C

import numpy as np
import pytest

from vtp import scenes

pytestmark = pytest.mark.gpu

R = 0.005
H = 4 * R
LB = -0.05


def _cloud(n, spacing, crowd=0, seed=0):
    """n points, a jittered lattice `spacing` cells apart with `crowd` of them moved into one cell, and
    the size of a box around them."""
    side = int(np.ceil(n ** (1 / 3)))
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(side, dtype=np.float32)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    p = spacing * H * (g + 0.2 * rng.uniform(-1, 1, g.shape))
    p[rng.permutation(n)[:crowd]] = np.floor(0.5 * side * spacing) * H + rng.uniform(0.01, 0.99, (crowd, 3)) * H
    return p.astype(np.float32), side * spacing * H + 0.1


def _scene(p, size, walls=None, max_nbr=60):
    cfg = scenes.pbf_config(dt=1e-7, r=R, lb=(LB,) * 3, size=(size,) * 3, max_nbr=max_nbr)
    half = len(p) // 2
    objs = [scenes.SceneObject("a", p[:half], 0), scenes.SceneObject("b", p[half:], 0)]
    if walls is not None:   # attached between the fluid objects: a cell's two runs interleave
        objs.insert(1, scenes.SceneObject("wall", walls, 1))
    return scenes.Scene("PBF", cfg, objs)


def _noalloc(vtp, p, size, max_nbr, repeats=1):
    """Counts, entries and the shortest time (ms) of the allocation-free lists."""
    import torch
    n = len(p)
    pos = torch.from_numpy(p).cuda()
    cnt = torch.empty(n, dtype=torch.int32, device="cuda")
    nbr = torch.empty((n, max_nbr), dtype=torch.int32, device="cuda")
    best = np.inf
    for _ in range(repeats):
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        rc = vtp.lib().vtp_ugns_neighbors_noalloc(pos.data_ptr(), n, (C.c_float * 3)(LB, LB, LB),
                                                  (C.c_float * 3)(size, size, size), H, max_nbr, cnt.data_ptr(),
                                                  nbr.data_ptr(), torch.cuda.current_stream().cuda_stream)
        t1.record()
        assert rc == 0, vtp.lib().vtp_last_error().decode()
        torch.cuda.synchronize()
        best = min(best, t0.elapsed_time(t1))
    return cnt.cpu().numpy().view(np.uint32), nbr.cpu().numpy().view(np.uint32), best


def _build_ms(vtp, sc):
    """The shortest list build (ms) of a few substeps from the scene's own positions."""
    s = vtp.solver_from_scene(sc)
    assert s.initialize(), s.last_error
    pos, best = s.get_field("pos"), np.inf
    for _ in range(5):
        s.set_field("pos", pos)
        best = min(best, s.profile_kernels(1)["ugns_lists"][0])
    s.destroy()
    return best


# Row counts on both sides of each builder's range, spacings from three rows a cell to none beside
# it, and crowds of one group more or less than the size from which small groups are not walked.
@pytest.mark.parametrize("n, spacing, crowd, max_nbr", [
    (5, 1.0, 5, 60), (1500, 0.35, 0, 60), (1500, 0.5, 63, 96), (1500, 0.7, 65, 96), (1500, 1.0, 70, 3),
    (16384, 0.7, 700, 60), (16385, 0.7, 700, 60), (16385, 1.6, 0, 60), (16385, 0.35, 64, 60),
    (40000, 0.5, 1500, 60), (131072, 0.8, 65, 60), (131073, 0.8, 65, 60), (131073, 0.5, 17, 60), (131073, 0.35, 0, 96),
])
@pytest.mark.parametrize("walls", [False, True])
def test_lists_match_the_oracle(vtp_gpu, oracle_lib, n, spacing, crowd, max_nbr, walls):
    p, size = _cloud(n, spacing, crowd, seed=n)
    sc = _scene(p, size, _cloud(max(n // 8, 2), spacing, min(crowd, n // 16), n + 1)[0] if walls else None, max_nbr)
    grid = oracle_lib.make_grid(sc.config["PBF"]["Required"])
    s = vtp_gpu.solver_from_scene(sc)
    assert s.initialize(), s.last_error
    want_cnt, want_nbr, _, _ = oracle_lib.neighbors(s.get_field("pos"), grid)
    cnt, nbr = s.get_neighbors(max_nbr)
    s.destroy()
    assert np.array_equal(cnt, want_cnt) and np.array_equal(nbr, want_nbr)
    if not walls:
        cnt, nbr, _ = _noalloc(vtp_gpu, p, size, max_nbr)
        assert np.array_equal(cnt, want_cnt) and np.array_equal(nbr, want_nbr)


def test_a_crowded_cell_costs_what_its_candidates_do(vtp_gpu):
    """10,000 particles in one cell test 1e8 candidates, as 463,000 particles of a fluid at rest do
    (216 each).  Ten times their time leaves room for the lanes and warps a single cell cannot fill;
    one warp for the whole cell took over a hundred times."""
    crowd, crowd_size = _cloud(20000, 0.5, 10000)
    even, even_size = _cloud(463000, 0.5)
    t_even = _noalloc(vtp_gpu, even, even_size, 60, repeats=4)[2]
    assert _noalloc(vtp_gpu, crowd, crowd_size, 60, repeats=4)[2] <= 10 * t_even
    t_even = _build_ms(vtp_gpu, _scene(even, even_size))
    assert _build_ms(vtp_gpu, _scene(crowd, crowd_size)) <= 10 * t_even


@pytest.mark.parametrize("n", [30000, 100000, 250000])
def test_a_sparse_cloud_costs_no_more_than_a_fluid(vtp_gpu, n):
    """A particle a cell has an eighth of the candidates of a fluid at rest."""
    fluid, fluid_size = _cloud(n, 0.5)
    spray, spray_size = _cloud(n, 1.0)
    assert _noalloc(vtp_gpu, spray, spray_size, 60, 6)[2] <= _noalloc(vtp_gpu, fluid, fluid_size, 60, 6)[2]
    assert _build_ms(vtp_gpu, _scene(spray, spray_size)) <= _build_ms(vtp_gpu, _scene(fluid, fluid_size))


def test_a_crowded_cell_of_interleaved_objects_merges_its_runs_once(vtp_gpu):
    """Fluid and wall particles of one cell whose attach ids interleave are merged by id.  A binary
    search per candidate looks 13 times at 4,000 + 4,000 particles, against 8 instructions for each
    row that tests the candidate; a merge that starts again for each 320 candidates looks 4,000 times."""
    p, size = _cloud(30000, 0.5, 4000)
    walls = _cloud(30000, 0.5, 4000, seed=1)[0]
    after = _scene(p, size)
    after.objects.append(scenes.SceneObject("wall", walls, 1))
    assert _build_ms(vtp_gpu, _scene(p, size, walls)) <= 2 * _build_ms(vtp_gpu, after)


@pytest.mark.parametrize("kind", ["PBF", "IMM"])   # lists of both shapes at this size
def test_list_lanes_choose_the_builder(vtp_gpu, kind):
    """"listLanes": a thread per row (1), rows of a cell together (8), by row count (0)."""
    import torch
    sc = _scene(*_cloud(3000, 0.5)) if kind == "PBF" else scenes.layered_mixture("IMM", 14, seed=3)
    used = []
    for lanes in (0, 1, 8):
        s = vtp_gpu.solver_from_scene(sc, extra={"listLanes": lanes})
        assert s.initialize(), s.last_error
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            s.get_neighbors(60)
            torch.cuda.synchronize()
        names = [e.key for e in prof.key_averages()]
        used.append({b for b in ("k_walk_lists", "k_build_lists") if any(b in n for n in names)})
        s.destroy()
    assert used == [{"k_build_lists"}, {"k_walk_lists"}, {"k_build_lists"}]


@pytest.mark.parametrize("cull", [False, True])
@pytest.mark.parametrize("attach", ["after", "before", "between"])
@pytest.mark.parametrize("n", [3000, 131073])
def test_a_thread_per_row_matches_the_oracle(vtp_gpu, oracle_lib, n, attach, cull):
    """Every order of a cell's two runs, with and without cell culling, in lists of both shapes."""
    p, size = _cloud(n, 0.5, 100, seed=2)
    wall = scenes.SceneObject("wall", _cloud(n // 8, 0.6, 50, seed=3)[0], 1)
    sc = _scene(p, size)
    sc.objects.insert({"after": 2, "before": 0, "between": 1}[attach], wall)
    s = vtp_gpu.solver_from_scene(sc, extra={"listLanes": 1, "cellCull": cull})
    assert s.initialize(), s.last_error
    want = oracle_lib.neighbors(s.get_field("pos"), oracle_lib.make_grid(sc.config["PBF"]["Required"]))
    cnt, nbr = s.get_neighbors(60)
    s.destroy()
    assert np.array_equal(cnt, want[0]) and np.array_equal(nbr, want[1])


def test_scan_of_a_large_grid_runs_at_memory_rate(vtp_gpu):
    """27 million buckets are read twice, zeroed and written: 16 bytes each, 66 us at 6.5 TB/s, three
    launches.  Three times that leaves room for the launches and for reads that miss the L2."""
    sc = _scene(*_cloud(8000, 0.5))
    sc.config["PBF"]["Required"]["simSpaceSize"] = [300 * H] * 3
    s = vtp_gpu.solver_from_scene(sc)
    assert s.initialize(), s.last_error
    best = min(s.profile_kernels(1)["ugns_cell_scan"][0] for _ in range(5))
    s.destroy()
    assert best <= 3 * 300 ** 3 * 16 / 6.5e9
