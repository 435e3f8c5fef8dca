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


@pytest.mark.parametrize("k", [1, 3, 4, 7, 8, 130])
@pytest.mark.parametrize("blocks_x256,extra", [(2, 0), (2, 1), (1, 0), (1, 1), (4, 1)])
def test_f64_lanes_per_point(pkg, torch_cuda, oracle_mod, k, blocks_x256, extra):
    """Around 512, 256 and 1024 points per SM, where the lanes per point change (as far as k allows)."""
    sms = torch_cuda.cuda.get_device_properties(0).multi_processor_count
    n, d = sms * 256 * blocks_x256 + extra, 3
    rng = np.random.default_rng(n + k)
    data = rng.integers(0, 4, (n, d)).astype(np.float64).reshape(-1)            # coarse: exact ties, the lower index wins
    m0 = rng.integers(0, 4, (k, d)).astype(np.float64).reshape(-1)
    means, asg = pkg.kmeans_host_f64(data, m0, n, k, d, 1, 0, 0)
    assert np.array_equal(asg, oracle_mod.assign_f64(data, m0, n, k, d, 0, 0, threads=8))
    want, _ = oracle_mod.update_d(data, asg, n, k, d, 0, 0)
    assert np.allclose(means, want, rtol=0, atol=4 * n * 2.0 ** -53)            # (integers: the sums are exact)
