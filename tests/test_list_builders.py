"""Neighbour-list builders and the cell scan at the row counts where another one is chosen,
with cells denser than a builder's window and lists cut at maxNeighborNum: counts, entries and
order are whole numbers and equal the oracle's."""
import ctypes as C

import numpy as np
import pytest

from vtp import scenes

pytestmark = pytest.mark.gpu

R = 0.125        # h = 0.5, cells of 0.5
SPACING = 0.25


def _points(n, seed, clump=400):
    """n points: a jittered lattice with `clump` of them (at most half) moved into one cell."""
    side = int(np.ceil(n ** (1 / 3)))
    g = np.arange(side, dtype=np.float32) * np.float32(SPACING)
    z, y, x = np.meshgrid(g, g, g, indexing="ij")
    rng = np.random.default_rng(seed)
    p = np.stack([x.ravel(), y.ravel(), z.ravel()], 1)[:n] + rng.uniform(-0.05, 0.05, (n, 3))
    k = min(clump, n // 2)
    p[rng.permutation(n)[:k]] = 0.5 * (side // 8) + rng.uniform(0.01, 0.49, (k, 3))
    return p.astype(np.float32)


def _scene(n, n_b, max_nbr, cells, attach, seed):
    cfg = scenes.pbf_config(dt=1e-3, r=R, lb=(-1.0,) * 3, size=(0.5 * cells,) * 3, max_nbr=max_nbr)
    f = _points(n, seed)
    objs = [scenes.SceneObject("fluid", f, 0)]
    if n_b:
        wall = scenes.SceneObject("wall", _points(n_b, seed + 1, 40) + np.float32(0.07), 1)
        objs = {"after": [*objs, wall], "before": [wall, *objs],
                "between": [scenes.SceneObject("a", f[: n // 2], 0), wall,
                            scenes.SceneObject("b", f[n // 2:], 0)]}[attach]
    return scenes.Scene("PBF", cfg, objs)


# Rows: one, one warp and its neighbours, the last row count of the builder with four rows a warp
# (16,384), of the builder with a warp per cell (300,000) and of the lists of 8 x 4 segments
# (49,152), and the first of what follows.  Cells per axis: 126 gives 127^3 buckets or 128^3 in
# bricks (1,024 tiles of 2,048, one launch of the scan) and 150 more tiles than one launch takes.
@pytest.mark.parametrize("n, n_b, max_nbr, cells, order, attach", [
    (1, 0, 60, 12, "brick", "after"),
    (2, 1, 60, 12, "linear", "before"),
    (31, 33, 3, 12, "brick", "between"),
    (33, 31, 60, 12, "brick", "before"),
    (1000, 500, 400, 24, "linear", "between"),
    (1001, 501, 7, 24, "brick", "after"),
    (3000, 900, 60, 126, "brick", "after"),
    (3000, 900, 60, 150, "brick", "before"),
    (3000, 900, 60, 150, "linear", "between"),
    (16384, 2000, 60, 40, "brick", "between"),
    (16385, 16385, 60, 40, "brick", "after"),
    (16385, 900, 250, 40, "linear", "between"),
    (49153, 900, 60, 50, "brick", "before"),
    (300000, 20000, 60, 80, "brick", "between"),
    (300001, 20000, 60, 80, "brick", "between"),
])
def test_lists_and_order_match_the_oracle(vtp_gpu, oracle_lib, n, n_b, max_nbr, cells, order, attach):
    sc = _scene(n, n_b, max_nbr, cells, attach, seed=n)
    s = vtp_gpu.solver_from_scene(sc, extra={"cellOrder": order})
    assert s.initialize(), s.last_error
    grid = oracle_lib.make_grid(sc.config["PBF"]["Required"])
    cnt, nbr, ids, keys = oracle_lib.neighbors(s.get_field("pos"), grid)
    got_cnt, got_nbr = s.get_neighbors(max_nbr)
    got_ids, got_keys = s.get_sorted_order()
    s.destroy()
    assert np.array_equal(got_cnt, cnt)
    assert np.array_equal(got_nbr, nbr)
    alive = ids.size
    assert np.array_equal(got_ids[:alive], ids) and np.array_equal(got_keys[:alive], keys)


@pytest.mark.parametrize("n, max_nbr", [(1, 60), (7, 1), (33, 8), (1000, 61), (1000, 400), (20001, 60)])
def test_allocation_free_lists_of_dense_cells_match_the_oracle(vtp_gpu, oracle_lib, n, max_nbr):
    import torch
    req = {"particleRadius": R, "simSpaceLB": [-1.0] * 3, "simSpaceSize": [20.0] * 3, "maxNeighborNum": max_nbr}
    pos = _points(n, seed=n)
    cnt, nbr, _, _ = oracle_lib.neighbors(pos, oracle_lib.make_grid(req))
    d_pos = torch.from_numpy(pos).cuda()
    d_cnt = torch.empty(n, dtype=torch.int32, device="cuda")
    d_nbr = torch.empty(n * max_nbr, dtype=torch.int32, device="cuda")
    rc = vtp_gpu.lib().vtp_ugns_neighbors_noalloc(
        d_pos.data_ptr(), n, (C.c_float * 3)(-1.0, -1.0, -1.0), (C.c_float * 3)(20.0, 20.0, 20.0), 4 * R, max_nbr,
        d_cnt.data_ptr(), d_nbr.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0, vtp_gpu.lib().vtp_last_error().decode()
    got_cnt = d_cnt.cpu().numpy().view(np.uint32)
    got_nbr = d_nbr.cpu().numpy().view(np.uint32).reshape(n, max_nbr)
    assert np.array_equal(got_cnt, cnt)
    for i in range(n):
        assert np.array_equal(got_nbr[i, : cnt[i]], nbr[i, : cnt[i]])
