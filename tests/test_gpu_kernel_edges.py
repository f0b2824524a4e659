"""Kernel variants at the edges of their ranges: window sizes and padded columns
of the FP32 CLAP filter and its adjoint, even and odd grid strides of the stage-3
patch filter, trial and column counts of the random-phase histogram, and the shared trial phasors of the
near-maximum topofit."""
import dataclasses
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(cuda_lib):
    from pystamps_b200 import stage2

    return stage2


# the transforms' rounding is ~10 eps of a window's largest element; gain and
# overlap sums of up to 16 windows bring it below 64 eps of the grid's largest
@pytest.mark.parametrize("n_win", [4, 8, 12, 24, 32])
@pytest.mark.parametrize("m,alpha", [(1, 1.0), (5, 1.7), (8, 1.0)])
def test_clap_window_sizes(cuda_lib, S, oracle, n_win, m, alpha):
    from pystamps_b200 import kernels as K

    rng = np.random.default_rng(n_win * 10 + m)
    g = (rng.standard_normal((41, 35, m)) + 1j * rng.standard_normal((41, 35, m))).astype(np.complex64)
    lp = S.build_low_pass(32.0, 800.0, 50.0)
    out = K.run_stage2_clap_filter_kernel(g, alpha, 0.3, lp, n_win)
    ref = oracle.clap_filter_grid_stack(g.astype(np.complex128), alpha, 0.3, lp, n_win, fp64=True)
    assert np.abs(out - ref).max() <= 64 * np.finfo(np.float32).eps * np.abs(ref).max()


# warps a block (0: the rule), window stack or window blocks: every form the same bits
@pytest.mark.parametrize("n_win", [8, 16, 24, 32])
@pytest.mark.parametrize("m", [3, 8, 41])
def test_clap_forms_give_the_same_bits(S, n_win, m):
    from pystamps_b200 import synth

    prep = S.prepare_patch(synth.make_patch(3000, m, 40, 41, seed=360 + m, n_rand=1000), nr=np.ones(100))
    with S.Stage2Context() as c:
        c.load(dataclasses.replace(prep, clap_window=n_win))
        out = []
        for warps in (0, 4, 8):
            for form in (0, 1):
                c.launch_shapes([0, warps, 0, 0, form])
                c.reset()
                c.iterate(2)
                out.append(c.download(["ph_grid", "ph_patch", "K_ps", "coh_ps"]))
    for o in out[1:]:
        for k in o:
            np.testing.assert_array_equal(o[k], out[0][k])


@pytest.mark.parametrize("m", [3, 4, 7, 10])
@pytest.mark.parametrize("slc_osf", [1, 2])
def test_stage3_patches_at_even_and_odd_strides(cuda_lib, oracle, m, slc_osf):
    from pystamps_b200 import stage2, stage3, synth

    patch = synth.make_patch(600, m, 34, 41, seed=320 + m, n_rand=1000)
    prep = stage2.prepare_patch(patch, nr=np.ones(100))
    rng = np.random.default_rng(m)
    grid = (rng.standard_normal((prep.n_i, prep.n_j, m)) + 1j * rng.standard_normal((prep.n_i, prep.n_j, m))).astype(
        np.complex64)
    sel = np.arange(0, 600, 3)
    gij = np.rint(prep.grid_ij).astype(np.int64)
    args = (grid, gij, sel, prep.ph_nm, np.asarray(prep.bperp, np.float64), np.arange(m))
    g = stage3.reestimate(*args, clap_alpha=1.0, clap_beta=0.3, low_pass=prep.low_pass, n_trial_wraps=2.4,
                          slc_osf=slc_osf)
    o = oracle.s3_reestimate(*args, alpha=1.0, beta=0.3, low_pass=prep.low_pass, n_trial_wraps=2.4, slc_osf=slc_osf)
    # the bound of the larger selection: 2e-6 of the largest value
    assert np.abs(g["ph_patch2"] - o["ph_patch2"]).max() <= 2e-6 * np.abs(o["ph_patch2"]).max()


# 0.3 rad noise on every PS keeps the patch phases away from |f| = 0, where FP32's
# rounding (~1e-6 through the two transforms) would be amplified by thousands
@pytest.mark.parametrize("n_win", [6, 12, 24, 32])
@pytest.mark.parametrize("m", [5, 40])
def test_adjoint_window_sizes(cuda_lib, n_win, m):
    import torch

    from pystamps_b200 import autograd as AG
    from pystamps_b200 import stage2, synth

    patch = synth.make_patch(4000, m, 33, 41, seed=340 + m, n_rand=1000, stable_fraction=1.0)
    prep = dataclasses.replace(stage2.prepare_patch(patch, nr=np.ones(100)), clap_window=n_win)
    dev = torch.device("cuda", 0)
    ph = torch.from_numpy(np.ascontiguousarray(prep.ph_nm, np.complex64)).to(dev)
    K = torch.from_numpy(patch["truth"]["K_ps"].astype(np.float32)).to(dev)
    w = torch.ones(4000, device=dev)
    gcoh = torch.full((4000,), 1.0 / 4000, device=dev)
    with AG.CoherenceMap(prep, 0) as c32, AG.CoherenceMap(prep, 0, "fp64") as c64:
        a = c32.backward(ph, K, w, 1.0, 0.3, gcoh)
        b = c64.backward(ph, K, w, 1.0, 0.3, gcoh)
    for x, y in zip(a, b):
        assert float((x - y).abs().norm() / y.abs().norm()) <= 1e-3


# trials around the 32-lane rounds; rows around the 8 (up to 64 columns) or 4 a warp
@pytest.mark.parametrize("m,n_trial_wraps,n_rand", [(2, 0.0, 1), (3, 2.0, 1001), (9, 1.9, 37), (64, 4.0, 999),
                                                    (65, 4.0, 999), (64, 3.9, 8), (65, 6.0, 5), (256, 0.6, 130)])
def test_random_histogram_edges(S, oracle, m, n_trial_wraps, n_rand):
    bp = np.random.default_rng(m).uniform(-300, 300, m)
    a, am = S.random_coherence_histogram(bp, n_trial_wraps, n_rand)
    b, bm = oracle.random_hist(bp, n_trial_wraps, n_rand=n_rand)
    np.testing.assert_array_equal(a, b)
    assert am == bm and a.sum() == n_rand


# rows and table sizes either side of the rule for shared phasors: the general
# path (a baseline matrix with equal rows) evaluates the same expressions
@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n,m,n_trial_wraps", [(1, 7, 1.0), (63, 30, 5.0), (64, 30, 5.0), (300, 1, 0.0), (300, 33, 4.0),
                                               (70, 131, 500.0), (70, 132, 500.0)])
def test_shared_baselines_give_the_general_path(cuda_lib, dtype, n, m, n_trial_wraps):
    from pystamps_b200 import kernels as K

    rng = np.random.default_rng(n + m)
    z = np.exp(1j * rng.uniform(-math.pi, math.pi, (n, m))).astype(dtype)
    z[::5, m // 2] = 0  # rows with a dropped column, whose own range may differ
    z[n // 2] = 0
    bp = rng.uniform(-300, 300, m).astype(z.real.dtype)
    for b in (bp, np.full_like(bp, 25.0)):
        one = K.run_stage2_topofit_row_invariant_kernel(z, b, n_trial_wraps)
        gen = K._near_max(z, np.tile(b, (n, 1)), False, n_trial_wraps, K.NEAR_MAX_COH_TOL, dtype == np.complex64)
        for x, y in zip(one, gen):
            np.testing.assert_array_equal(x, y)
