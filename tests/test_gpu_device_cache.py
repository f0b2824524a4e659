"""Device blocks and streams kept between calls: calls of changing sizes, from
several threads at once, give what each gives alone; a context loaded into
blocks that another one filled starts from the same state."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(n, m, seed):
    r = np.random.default_rng(seed)
    return np.exp(1j * r.uniform(-3.0, 3.0, (n, m))).astype(np.complex64), r.uniform(-200.0, 200.0, (n, m)).astype(np.float32)


@pytest.mark.parametrize("threads", [1, 4])
def test_calls_in_any_order_and_thread(cuda_lib, threads):
    from pystamps_b200 import kernels as K
    from pystamps_b200 import stage2 as S

    sizes = [(1, 5), (700, 9), (33, 60), (5000, 20), (2, 3), (4000, 31)]
    rows = [_rows(n, m, k) for k, (n, m) in enumerate(sizes)]

    def call(k):
        z, b = rows[k % len(rows)]
        return (*K.run_stage2_topofit_kernel(z, b, 3.0), S.random_coherence_histogram(b[0].astype(np.float64), 1.5, 500 + k % 6)[0])

    want = [call(k) for k in range(len(rows))]
    with ThreadPoolExecutor(threads) as ex:
        for k, got in enumerate(ex.map(call, range(5 * len(rows)))):
            for a, b in zip(got, want[k % len(rows)]):
                np.testing.assert_array_equal(a, b)


def test_context_in_used_blocks(cuda_lib):
    from pystamps_b200 import stage2 as S
    from pystamps_b200 import synth

    p = S.prepare_patch(synth.make_patch(3000, 14, 26, 41, seed=5, gamma_max_iterations=3))
    keys = ("K_ps", "C_ps", "coh_ps", "N_opt", "ph_grid")
    with S.Stage2Context() as c:
        c.load(p, "fp32")
        before = c.download(("C_ps", "N_opt"))
        c.run()
        first = c.download(keys)
    with S.Stage2Context() as c:
        c.load(p, "fp32")
        again = c.download(("C_ps", "N_opt"))
        c.run()
        second = c.download(keys)
    assert not again["C_ps"].any() and not again["N_opt"].any()
    np.testing.assert_array_equal(before["C_ps"], again["C_ps"])
    for k in keys:
        np.testing.assert_array_equal(first[k], second[k])


def test_download_vectors_are_not_overwritten(cuda_lib):
    """The context hands out its result memory again only when no vector of an
    earlier download is left."""
    from pystamps_b200 import stage2 as S
    from pystamps_b200 import synth

    p = S.prepare_patch(synth.make_patch(2000, 12, 26, 41, seed=6, gamma_max_iterations=2))
    with S.Stage2Context() as c:
        c.load(p, "fp32")
        c.iterate(1)
        first = c.download(("K_ps", "coh_ps"))
        kept, tail = first["K_ps"].copy(), first["coh_ps"][7:]
        tail_kept = tail.copy()
        c.iterate(1)
        second = c.download(("K_ps", "coh_ps"))
        assert not np.array_equal(first["K_ps"], second["K_ps"])
        np.testing.assert_array_equal(first["K_ps"], kept)
        del first, second  # `tail` still refers to the first download's memory
        third = c.download(("K_ps", "coh_ps", "C_ps"))
        np.testing.assert_array_equal(tail, tail_kept)
        assert all(v.flags.c_contiguous and v.flags.writeable and v.shape == (2000,) for v in
                   (third["K_ps"], third["coh_ps"], third["C_ps"]))
