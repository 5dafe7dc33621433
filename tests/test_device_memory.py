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
