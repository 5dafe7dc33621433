"""What a solver takes of the device's memory, and when."""
import numpy as np
import pytest

from vtp import scenes

pytestmark = pytest.mark.gpu

PAGE = 2 << 20   # cudaMalloc takes pages of this size from the device


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_reading_the_fractions_allocates_nothing(vtp_gpu):
    """What the read needs beside its staging buffer is there from initialize on: the first frame of a
    fresh solver costs what the next one does."""
    sc = scenes.layered_mixture("IMM", 90, seed=1)
    s = vtp_gpu.solver_from_scene(sc)
    assert s.initialize(), s.last_error
    s.get_field("pos")   # a staging buffer of three floats a particle, the fractions' size
    before = _free()
    fractions = s.get_field("vol_frac")
    assert fractions.nbytes == 12 * sc.n_total > 2 * PAGE
    assert before - _free() < PAGE
    s.destroy()


def _fluid(kind, n, max_nbr=60):
    sp = 0.02 if kind == "PBF" else 0.01
    side = int(np.ceil(n ** (1 / 3)))
    g = (np.arange(side, dtype=np.float32) + np.float32(5)) * np.float32(sp)
    z, y, x = np.meshgrid(g, g, g, indexing="ij")
    p = scenes.jitter(np.stack([x.ravel(), y.ravel(), z.ravel()], 1)[:n], 0.05, sp, n)
    make = scenes.pbf_config if kind == "PBF" else scenes.dfsph_config
    cfg = make(dt=1e-3, r=sp / 2, lb=(0.0,) * 3, size=((side + 10) * sp,) * 3, max_nbr=max_nbr)
    return scenes.Scene(kind, cfg, [scenes.SceneObject("fluid", p, 0)])


def _taken(vtp, sc):
    """Device memory of an initialized solver."""
    s = vtp.solver_from_scene(sc)
    before = _free()
    assert s.initialize(), s.last_error
    taken = before - _free()
    s.destroy()
    return taken


def test_lists_of_large_solvers_hold_no_more_than_they_may(vtp_gpu):
    """A thread per row reads lists of any length: three neighbours more are three words a row more
    (the list and the page ends of the arrays around it leave four pages open)."""
    n = 1_000_000
    _taken(vtp_gpu, _fluid("PBF", n, 57))   # modules and streams are loaded
    more = _taken(vtp_gpu, _fluid("PBF", n, 60)) - _taken(vtp_gpu, _fluid("PBF", n, 57))
    assert more <= 3 * 4 * n + 4 * PAGE


def test_dfsph_scene_that_just_fits(vtp_gpu):
    """The second array of packed rows is taken only where it leaves room: a scene that fits without
    it initializes, and gives the same bits."""
    import torch
    n = 1_000_000
    sc = _fluid("DFSPH", n)
    want = []
    for _ in range(2):   # the second time everything around the solver is loaded
        s = vtp_gpu.solver_from_scene(sc)
        before = _free()
        assert s.initialize(), s.last_error
        taken = before - _free()
        assert s.tickNsteps(2), s.last_error
        want = [s.get_field("pos"), s.get_field("vel"), s.stats()["total_div_iters"], s.stats()["total_incomp_iters"]]
        s.destroy()
    s = vtp_gpu.solver_from_scene(sc)
    torch.cuda.empty_cache()
    filler = torch.empty(_free() - (taken - 32 * n // 2), dtype=torch.uint8, device="cuda")
    assert s.initialize(), s.last_error   # half of the second array short
    del filler
    torch.cuda.empty_cache()
    assert s.tickNsteps(2), s.last_error
    got = [s.get_field("pos"), s.get_field("vel"), s.stats()["total_div_iters"], s.stats()["total_incomp_iters"]]
    s.destroy()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]) and got[2:] == want[2:]


def test_a_slab_worker_holds_one_array_of_packed_rows(vtp_gpu):
    """Its rows' own state: two load slots and objects, the slot map, ghost flags, four targets."""
    from vtp.domain import LibraryStages
    n = 1_000_000
    sc = _fluid("DFSPH", n)
    p = sc.objects[0].pos
    _taken(vtp_gpu, sc)
    solver = _taken(vtp_gpu, sc)
    before = _free()
    d = LibraryStages(sc.config, p[:1000], p[1000:1100] + np.float32(0.004), np.arange(n, n + 100, dtype=np.uint32),
                      False, n, 1)
    taken = before - _free()
    d.close()
    own = (4 * 4 + 4 + 1 + 4 + 8 * 4) * n
    assert taken <= solver - 32 * n + own + 8 * PAGE


def test_a_solver_that_does_not_fit_leaves_the_next_one_alone(vtp_gpu):
    import torch
    sc = _fluid("PBF", 1_000_000)
    taken = _taken(vtp_gpu, sc)
    torch.cuda.empty_cache()
    filler = torch.empty(_free() - taken // 2, dtype=torch.uint8, device="cuda")
    s = vtp_gpu.solver_from_scene(sc)
    with pytest.raises(vtp_gpu.VtpError, match="out of device memory"):
        s.initialize()
    s.destroy()
    del filler
    torch.cuda.empty_cache()
    small = vtp_gpu.solver_from_scene(_fluid("PBF", 1000))
    assert small.initialize() and small.tickNsteps(1), small.last_error
    small.destroy()
