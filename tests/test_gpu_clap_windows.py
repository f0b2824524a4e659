"""Window sizes that 4 does not divide: n_inc = n_win // 4 then leaves up to 8
windows (10 with the clamped ones at an edge) over a cell along an axis, where a
multiple of 4 has 4 or 5. Filter against the oracle's FP64 CLAP, coherence and
gradient against the FP64 torch restatement, the loop's two forms against each
other."""
import dataclasses

import numpy as np
import pytest

from torch_coherence_ref import geometry, torch_coherence

pytestmark = pytest.mark.gpu


# as in test_clap_window_sizes: 64 eps of the grid's largest (an FP32 transform of
# the same sums by the oracle is within 0.5 eps of it at every size here)
@pytest.mark.parametrize("n_win", [5, 6, 7, 9, 10, 11, 14, 15, 18, 19, 22, 23, 26, 27, 31])
@pytest.mark.parametrize("n_i,n_j", [(41, 35), (33, 48)])
def test_filter(cuda_lib, oracle, n_win, n_i, n_j):
    from pystamps_b200 import kernels as K
    from pystamps_b200 import stage2 as S

    rng = np.random.default_rng(n_win * 10 + n_j)
    g = (rng.standard_normal((n_i, n_j, 5)) + 1j * rng.standard_normal((n_i, n_j, 5))).astype(np.complex64)
    lp = S.build_low_pass(32.0, 800.0, 50.0)
    out = K.run_stage2_clap_filter_kernel(g, 1.0, 0.3, lp, n_win)
    ref = oracle.clap_filter_grid_stack(g.astype(np.complex128), 1.0, 0.3, lp, n_win, fp64=True)
    assert np.abs(out - ref).max() <= 64 * np.finfo(np.float32).eps * np.abs(ref).max()


def _patch(n_win, m=5):
    from pystamps_b200 import stage2, synth

    patch = synth.make_patch(4000, m, 33, 41, seed=380 + n_win, n_rand=1000, stable_fraction=1.0)
    return patch, dataclasses.replace(stage2.prepare_patch(patch, nr=np.ones(100)), clap_window=n_win)


# the adjoint's own tolerances: 1e-9 of the coherence, here with the rounding of its FP32
# result (2^-24) on top, and 1e-6 of the gradients
@pytest.mark.parametrize("n_win", [6, 7, 11, 23])
def test_coherence_and_gradient(cuda_lib, n_win):
    import torch

    from pystamps_b200 import autograd as AG

    patch, prep = _patch(n_win)
    dev = torch.device("cuda", 0)
    ph = torch.from_numpy(np.ascontiguousarray(prep.ph_nm, np.complex64)).to(dev)
    K = torch.from_numpy(patch["truth"]["K_ps"].astype(np.float32)).to(dev)
    w = torch.ones(4000, device=dev)
    gcoh = torch.full((4000,), 1.0 / 4000, device=dev)
    with AG.CoherenceMap(prep, 0, "fp64") as c:
        coh = c.forward(ph, K, w, 1.0, 0.3)
        gph, gK, _ = c.backward(ph, K, w, 1.0, 0.3, gcoh)
    ph64 = ph.cpu().to(torch.complex128).requires_grad_(True)
    K64 = K.cpu().double().requires_grad_(True)
    want = torch_coherence(geometry(prep, torch.device("cpu")), ph64, K64, w.cpu().double(),
                           torch.tensor(1.0, dtype=torch.float64), torch.tensor(0.3, dtype=torch.float64))
    assert float((coh.cpu().double() - want.detach()).abs().max()) <= 2.0 ** -24 + 1e-9
    (want * gcoh.cpu().double()).sum().backward()
    for got, ref in ((gph, ph64.grad), (gK, K64.grad)):
        assert float((got.cpu().to(ref.dtype) - ref).abs().norm() / ref.abs().norm()) <= 1e-6


@pytest.mark.parametrize("n_win", [6, 7, 11, 23])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_loop_forms(cuda_lib, n_win, precision):
    from pystamps_b200 import stage2 as S

    _, prep = _patch(n_win)
    out = []
    with S.Stage2Context() as c:
        c.load(prep, precision)
        for form in (0, 1):
            c.launch_shapes([0, 0, 0, 0, form])
            c.reset()
            c.iterate(2)
            out.append(c.download(["ph_patch", "K_ps", "coh_ps"]))
    if precision == "fp32":
        for k in out[0]:
            np.testing.assert_array_equal(out[0][k], out[1][k])
    else:  # the two forms add a cell's windows in FP64 in different orders
        assert np.abs(out[0]["ph_patch"] - out[1]["ph_patch"]).max() <= 1e-9


# grids either side of the lines between 4 and 8 warps a block: one round of blocks of
# 4, one of 8, two of 4, and the padding's share; alone and in window blocks
@pytest.mark.parametrize("cells,m", [(30, 4), (40, 100), (40, 116), (40, 148), (64, 28), (64, 68), (64, 76)])
def test_warps_a_block(cuda_lib, cells, m):
    from pystamps_b200 import stage2 as S
    from pystamps_b200 import synth

    prep = S.prepare_patch(synth.make_patch(2500, m, cells, 41, seed=390 + m, n_rand=1000), nr=np.ones(100))
    out = []
    with S.Stage2Context() as c:
        c.load(prep)
        for warps, form in ((0, 0), (4, 0), (8, 0), (0, 1)):
            c.launch_shapes([0, warps, 0, 0, form])
            c.reset()
            c.iterate(1)
            out.append(c.download(["ph_patch"])["ph_patch"])
    for o in out[1:]:
        np.testing.assert_array_equal(o, out[0])
