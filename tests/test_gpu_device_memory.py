"""Device memory a loaded patch takes: what its arrays need. Only blocks small
enough to be kept between calls are rounded up, and what is kept can be given back."""
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


def test_kept_memory_is_given_back(cuda_lib):
    import torch

    from pystamps_b200 import _lib
    from pystamps_b200 import stage2 as S
    from pystamps_b200 import synth

    p = S.prepare_patch(synth.make_patch(40_000, 60, 40, 41, seed=22, n_rand=1000), nr=np.ones(100))
    torch.zeros(1, device="cuda")
    _lib.release_kept()
    with S.Stage2Context() as c:
        c.load(p, "fp32")
        c.iterate(1)
        first = c.download(("K_ps",))["K_ps"].copy()
    held = torch.cuda.mem_get_info()[0]
    freed = _lib.release_kept()
    assert 0 < freed <= 512 << 20
    # the driver returns whole 2 MB pages
    assert torch.cuda.mem_get_info()[0] - held >= freed // 2
    assert _lib.release_kept() == 0
    with S.Stage2Context() as c:  # blocks, streams and a loaded context after it work as before
        c.load(p, "fp32")
        _lib.release_kept()
        c.iterate(1)
        np.testing.assert_array_equal(c.download(("K_ps",))["K_ps"], first)
