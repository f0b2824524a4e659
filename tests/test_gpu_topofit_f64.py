"""The plain FP64 topofit at the edges of its row groups, lanes and trial blocks,
against the direct evaluation of every trial in numpy on the same patch phases:
the same trial, and K and coherence to rounding."""
import dataclasses
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# columns around the 8 lanes and the 32-lane rounds, up to the largest; trials
# around the blocks of 8 magnitudes; rows around the 4 of a warp and the 8 of a block
CASES = [(1, 41, 297, False), (7, 1, 300, False), (7, 3, 301, True), (8, 17, 302, False), (9, 19, 303, True), (31, 41, 200, False),
         (33, 81, 201, True), (64, 33, 202, False), (150, 175, 100, False), (256, 35, 121, False)]


@pytest.mark.parametrize("m,trials,n,same_baseline", CASES)
def test_trial_and_refinement(cuda_lib, m, trials, n, same_baseline):
    from pystamps_b200 import stage2 as S
    from pystamps_b200 import synth

    patch = synth.make_patch(n, max(m, 3), 28, 41, seed=100 + m, n_rand=1000)
    p = S.prepare_patch(patch, nr=np.ones(100))
    half = (trials - 1) // 2
    bp = np.ascontiguousarray(p.bperp[:, :m])
    if same_baseline:
        bp[:] = np.float32(25.0)
    ph = np.ascontiguousarray(p.ph_nm[:, :m])
    ph[n // 2, m // 2] = 0  # one invalid row
    p = dataclasses.replace(p, n_ifg=m, ph_nm=ph, amp=np.ascontiguousarray(p.amp[:, :m]), bperp=bp,
                            bperp_nm=p.bperp_nm[:m], n_trial_wraps=max(0.0, (half - 0.5) / 8.0))
    with S.Stage2Context() as c:
        c.load(p, "fp64")
        c.iterate(1)
        g = c.download(("K_ps", "C_ps", "coh_ps", "N_opt", "ph_patch", "ph_res"))
    z = np.conj(g["ph_patch"]) * ph
    bad = (z == 0).any(1)
    assert bad[n // 2] and np.array_equal(np.isnan(g["K_ps"]), bad) and np.array_equal(g["N_opt"] == 0, bad)
    b = bp.astype(np.float64)
    span = b.max(1) - b.min(1)
    span[span == 0] = 1.0
    theta = b / span[:, None] * (math.pi / 4)
    sq = np.stack([np.abs((z * np.exp(-1j * theta * t)).sum(1)) ** 2 for t in range(-half, half + 1)], 1)
    order = np.sort(sq, 1)
    # rows whose best trial leads by more than the rounding of either evaluation
    clear = ~bad & (order[:, -1] - (order[:, -2] if trials > 1 else -1.0) > 1e-11 * m * m)
    if not same_baseline and m > 1:
        assert clear.sum() > 0.9 * n
    k0 = (math.pi / 4) / span * (sq.argmax(1) - half)
    r = z * np.exp(-1j * k0[:, None] * b)
    wgt = np.abs(z)
    num = (wgt * b * wgt * np.angle(r * np.conj(r.sum(1))[:, None])).sum(1)
    K = k0 + num / np.maximum(((wgt * b) ** 2).sum(1), 1e-300)
    s = (z * np.exp(-1j * K[:, None] * b)).sum(1)
    # a residual angle within 1e-9 of +-pi may round to either side
    wrap = (np.abs(np.abs(np.angle(r * np.conj(r.sum(1))[:, None])) - math.pi) < 1e-9).any(1)
    ok = clear & ~wrap
    np.testing.assert_allclose(g["K_ps"][ok], K[ok], rtol=1e-10, atol=1e-12)
    np.testing.assert_allclose(g["coh_ps"][ok], np.abs(s)[ok] / wgt[ok].sum(1), rtol=0, atol=1e-11)
    assert np.all(g["coh_ps"][~bad] <= 1 + 1e-12)
