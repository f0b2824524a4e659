"""Rows of the plain FP64 topofit that the trial chains do not decide: the trial
is the direct sum's where the direct sums differ beyond their own rounding, and
one of the tied trials where they do not."""
import dataclasses
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

QPI = math.pi / 4


def _run(p):
    from pystamps_b200 import stage2 as S

    with S.Stage2Context() as c:
        c.load(p, "fp64")
        c.iterate(1)
        return c.download(("K_ps", "coh_ps", "N_opt", "ph_patch"))


def _direct(z, theta, half):
    return np.stack([np.abs((z * np.exp(-1j * (theta * t))).sum(1)) ** 2 for t in range(-half, half + 1)], 1)


def _refined(z, b, k0):
    r = z * np.exp(-1j * k0[:, None] * b)
    wgt = np.abs(z)
    ang = np.angle(r * np.conj(r.sum(1))[:, None])
    K = k0 + (wgt * b * wgt * ang).sum(1) / np.maximum(((wgt * b) ** 2).sum(1), 1e-300)
    s = (z * np.exp(-1j * K[:, None] * b)).sum(1)
    return K, np.abs(s) / np.maximum(wgt.sum(1), 1e-300), (np.abs(np.abs(ang) - math.pi) < 1e-9).any(1)


def test_close_baselines_far_from_zero(cuda_lib):
    """Baselines of 2e8 within 2e3: an argument theta m of the direct sum is rounded
    by up to 5e-10, which decides between two trials that lie closer than that."""
    from pystamps_b200 import stage2 as S
    from pystamps_b200 import synth

    n, m, half = 20_000, 40, 60
    patch = synth.make_patch(2 * n, m, 40, 41, seed=11, n_rand=1000)
    p = S.prepare_patch(patch, nr=np.ones(100))
    rng = np.random.default_rng(12)
    b = (2e8 + rng.uniform(-1e3, 1e3, (2 * n, m))).astype(np.float32)
    b64 = b.astype(np.float64)
    span = b64.max(1) - b64.min(1)
    theta = (b64 / span[:, None]) * QPI
    # the first n rows fill the grid; the others have no weight in it, and with the
    # same patch phase again two equal maxima either side of a trial
    w = np.asarray(p.weight0).copy()
    w[n:] = 0.0
    p = dataclasses.replace(p, bperp=b, weight0=w, n_trial_wraps=(half - 0.5) / 8.0, gamma_max_iterations=1)
    f = _run(p)["ph_patch"][n:]
    d = theta[n:] - theta[n:].mean(1, keepdims=True)
    k, t0 = rng.integers(8, 40, (n, 1)), rng.integers(-15, 16, (n, 1))
    ph = np.asarray(p.ph_nm).copy()
    ph[n:] = f * np.cos(d * k) * np.exp(1j * d * t0)
    g = _run(dataclasses.replace(p, ph_nm=ph))
    np.testing.assert_array_equal(g["ph_patch"][n:], f)
    z = np.conj(f) * ph[n:]
    direct, ranked = _direct(z, theta[n:], half), _direct(z, d, half)
    order = np.sort(direct, 1)
    # 40 terms of 2^-52 each in a sum of at most 40, and its square
    decided = (z != 0).all(1) & (order[:, -1] - order[:, -2] > 1e-10)
    K, coh, wrap = _refined(z, b64[n:], QPI / span[n:] * (direct.argmax(1) - half))
    ok = decided & ~wrap
    assert (ok & (direct.argmax(1) != ranked.argmax(1))).sum() >= 5 and ok.sum() > 0.9 * n
    # neighbouring trials are pi / 4 / span apart, a refinement K off by far less
    assert np.abs(g["K_ps"][n:] - K)[ok].max() * 2e3 <= 0.05
    assert np.abs(g["coh_ps"][n:] - coh)[ok].max() <= 1e-6


# every trial ties: one baseline for all columns, one column, one trial
@pytest.mark.parametrize("m,trials,n", [(1, 41, 297), (7, 3, 301), (9, 19, 303), (33, 81, 201), (150, 35, 101), (7, 1, 55)])
def test_tied_trials(cuda_lib, m, trials, n):
    from pystamps_b200 import stage2 as S
    from pystamps_b200 import synth

    half = (trials - 1) // 2
    p = S.prepare_patch(synth.make_patch(n, max(m, 3), 28, 41, seed=200 + m, n_rand=1000), nr=np.ones(100))
    b = np.full((n, m), 25.0, np.float32)
    ph = np.ascontiguousarray(p.ph_nm[:, :m])
    ph[n // 2, m // 2] = 0
    p = dataclasses.replace(p, n_ifg=m, ph_nm=ph, amp=np.ascontiguousarray(p.amp[:, :m]), bperp=b,
                            bperp_nm=p.bperp_nm[:m], n_trial_wraps=max(0.0, (half - 0.5) / 8.0))
    g = _run(p)
    z = np.conj(g["ph_patch"]) * ph
    good = (z != 0).all(1)
    assert good.sum() == n - 1 and np.array_equal(g["N_opt"] == 1, good) and np.isnan(g["K_ps"][~good]).all()
    b64 = b.astype(np.float64)
    sq = _direct(z, b64 * QPI, half)
    near = np.full(n, np.inf)
    cohs = np.full(n, np.inf)
    for t in range(trials):
        K, coh, wrap = _refined(z, b64, np.full(n, QPI * (t - half)))
        tied = sq[:, t] >= sq.max(1) - 1e-11 * m * m
        # the step from K0 is a weighted mean angle over b; an angle at +-pi may go either way
        err = np.where(tied & ~wrap, np.abs(g["K_ps"] - K), np.inf)
        cohs = np.where(err < near, np.abs(g["coh_ps"] - coh), cohs)
        near = np.minimum(near, err)
    ok = good & np.isfinite(near)
    assert ok.sum() > 0.9 * n
    np.testing.assert_allclose(near[ok], 0.0, atol=1e-10 * max(1.0, QPI * half))
    np.testing.assert_allclose(cohs[ok], 0.0, atol=1e-11)


# 16 lanes take a row above 64 columns or in launches of few rows, 8 the others: 8-lane
# launches at the edges of the lanes and trial blocks, and either side of the column rule
@pytest.mark.parametrize("m,trials", [(7, 1), (8, 17), (9, 19), (31, 41), (33, 35), (64, 33), (65, 33)])
def test_launches_of_many_rows(cuda_lib, m, trials):
    from test_gpu_topofit_f64 import test_trial_and_refinement as check

    check(cuda_lib, m, trials, 5003, False)
