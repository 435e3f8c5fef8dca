"""GPU: the double-precision path at the edges of its kernels: rows padded to 2, 4, 8, 16 and 32
dimensions (longer rows take the warp-per-point kernel), mean sets around one shared-memory tile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,d", [(257, 5, 1), (700, 2049, 2), (256, 1023, 3), (300, 1025, 4), (513, 511, 5), (300, 513, 8),
                                   (255, 257, 9), (1000, 256, 16), (300, 129, 17), (400, 128, 32), (200, 60, 33), (1, 1, 7)])
def test_f64_matches_the_oracle_at_tile_edges(pkg, torch_cuda, oracle_mod, n, k, d):
    rng = np.random.default_rng(n + 31 * k + d)
    rows = rng.standard_normal((n, d))
    centres = np.resize(rows, (k, d)) + (rng.integers(0, 2, (k, 1)) * 0.1)      # repeated rows: exact ties, the lower index wins
    for lay, laym in ((0, 0), (1, 0), (0, 1), (1, 1)):
        data = rows.reshape(-1) if lay == 0 else np.ascontiguousarray(rows.T).reshape(-1)
        m0 = centres.reshape(-1) if laym == 0 else np.ascontiguousarray(centres.T).reshape(-1)
        means, asg = pkg.kmeans_host_f64(data, m0, n, k, d, 1, lay, laym)
        assert np.array_equal(asg, oracle_mod.assign_f64(data, m0, n, k, d, lay, laym, threads=8)), (lay, laym)
        want, _ = oracle_mod.update_d(data, asg, n, k, d, lay, laym)
        # sums of at most n terms in another order: n * 2^-53 of the sum of absolute values (below 6 per term)
        assert np.allclose(means, want, rtol=0, atol=6 * n * 2.0 ** -53), (lay, laym)
