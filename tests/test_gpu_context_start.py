"""A context loaded into device blocks that an earlier one filled: what can be read
before the first iteration is zero, not the other patch's data."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("weighting", ["P-square", "SNR"])
def test_readable_state_before_the_first_iteration(cuda_lib, precision, weighting):
    from pystamps_b200 import stage2 as S
    from pystamps_b200 import synth

    n, m = 3000, 14
    keys = ("K_ps", "C_ps", "coh_ps", "N_opt", "ph_grid")
    patch = synth.make_patch(n, m, 26, 41, seed=15, gamma_max_iterations=3, n_rand=1000)
    patch["parms"]["filter_weighting"] = weighting
    p = S.prepare_patch(patch, nr=np.ones(100))
    assert p.psquare == (weighting == "P-square")
    with S.Stage2Context() as c:
        c.load(p, precision)
        c.run()
        assert c.download(("ph_grid",))["ph_grid"].any()
        used = c.export_state()
    with S.Stage2Context() as c:
        c.load(p, precision)
        first = c.download(keys)
        state = c.export_state()
    for k in keys:
        assert not first[k].any(), k
    assert len(state) == len(used)
    if weighting == "SNR":  # the residual phases end the blob
        tail = n * m * (8 if precision == "fp64" else 4)
        assert any(used[-tail:]) and not any(state[-tail:])
