"""Device memory a loaded patch takes: what its arrays need. Only blocks small
enough to be kept between calls are rounded up."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_large_arrays_take_what_they_need(cuda_lib):
    import torch

    from pystamps_b200 import stage2 as S
    from pystamps_b200 import synth

    n, m, cells = 2000, 244, 200
    p = S.prepare_patch(synth.make_patch(n, m, cells, 41, seed=21, n_rand=1000), nr=np.ones(100))
    p = dataclasses.replace(p, clap_window=24)
    w = -(-p.n_i // 6) - 3, -(-p.n_j // 6) - 3
    blocks = (-(-w[0] // 4)) * (-(-w[1] // 4))
    win, part, grid = 8 * w[0] * w[1] * 576 * m, 16 * blocks * 42 * 42 * m, 8 * p.n_i * p.n_j * m
    assert win > 1 << 30 and part > 400 << 20 and grid < 100 << 20
    torch.zeros(1, device="cuda")
    with S.Stage2Context() as c:
        before = torch.cuda.mem_get_info()[0]
        c.load(p, "fp32")
        taken = before - torch.cuda.mem_get_info()[0]
    # grid and patch phase rounded by up to a sixteenth, the rows' arrays and the
    # driver's own pages below 30 MB
    assert taken <= win + part + 2 * grid * 17 / 16 + (30 << 20)
