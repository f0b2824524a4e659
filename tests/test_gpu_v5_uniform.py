"""The random-phase histogram's uniform stream, drawn on the GPU in segments of
1,024 draws whose start states come from jump tables of 256 segments a row:
histograms equal to the oracle's serial generator at the edges of a segment and
of a table row, for one column, odd columns and small baselines."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rand,m", [(1, 3), (341, 3), (1023, 5), (1024, 4), (1025, 7), (3500, 75), (3496, 75), (9001, 61)])
def test_histogram_equals_serial_stream(cuda_lib, oracle, n_rand, m):
    from pystamps_b200 import stage2 as S

    bp = np.random.default_rng(n_rand + m).uniform(-300.0, 300.0, m)
    got, top = S.random_coherence_histogram(bp, 2.4, n_rand)
    want, want_top = oracle.random_hist(bp, 2.4, n_rand=n_rand)
    np.testing.assert_array_equal(got, want)
    assert top == want_top and got.sum() == n_rand


def test_draws_past_the_kept_tables(cuda_lib, oracle):
    """84.6 million draws: the last rows of segment starts are not among the 320 the
    process keeps."""
    from pystamps_b200 import stage2 as S

    n_rand, bp = 28_200_000, np.array([-120.0, 35.0, 260.0])
    assert 3 * n_rand > 320 * 256 * 1024
    got, top = S.random_coherence_histogram(bp, 0.1, n_rand)
    want, want_top = oracle.random_hist(bp, 0.1, n_rand=n_rand)
    np.testing.assert_array_equal(got, want)
    assert top == want_top and got.sum() == n_rand
