"""GPU: the two smallest values of a point's row come from two partitions of the means (by index mod 16, and into
groups of 16 neighbours).  A second mean as close as the first has to be seen wherever it lies: in the same
group, in the same position of another group, chunk, mean tile or column part."""
import numpy as np
import pytest

from helpers import DeviceArrays, rows_to_layout

pytestmark = pytest.mark.gpu

# CUDA cores (one and two tiles of means), a resident mean tile, mean tiles in a ring, CTA pairs, the K loop
SHAPES = [(3, 48), (8, 1100), (16, 33), (16, 256), (12, 600), (24, 600), (32, 1024), (64, 700), (70, 300), (128, 1024), (300, 2100)]


@pytest.mark.parametrize("apart", [1, 15, 16, 17, 31, 32, 64, 128, 256, 512, 1024])
@pytest.mark.parametrize("d,k", SHAPES)
def test_second_mean_at_every_distance(pkg, torch_cuda, oracle_mod, d, k, apart):
    if apart >= k:
        pytest.skip("no two means lie so far apart")
    rng = np.random.default_rng(1000 * d + k + apart)
    n = 515
    means = rng.random((k, d), dtype=np.float32)
    first = rng.choice(k - apart, size=min(24, k - apart), replace=False)
    used = set()
    for t, i in enumerate(first):
        if i in used or i + apart in used:
            continue
        used |= {i, i + apart}
        means[i + apart] = means[i]
        if t % 2:                                    # not equal, but closer than the pass can tell apart
            means[i + apart, t % d] = np.nextafter(means[i, t % d], np.float32(t % 4), dtype=np.float32)
    near = means[rng.choice(np.array(sorted(used)), n)]
    rows = (near + 0.01 * rng.standard_normal((n, d))).astype(np.float32)
    for lay, laym in ((0, 0), (1, 1)):
        data, m = rows_to_layout(rows, lay), rows_to_layout(means, laym)
        want = oracle_mod.assign(data, m, n, k, d, lay, laym, threads=8)
        for variant in [pkg.ASSIGN_TC] + ([pkg.ASSIGN_SIMT] if d <= 8 else []):
            dev = DeviceArrays(torch_cuda, pkg, data, m, n, k, d)
            pkg.assign(dev.points.data_ptr(), dev.means.data_ptr(), dev.assignment.data_ptr(), n, k, d, lay, laym,
                       dev.ws_ptr, dev.ws_bytes_avail, variant=variant)
            pkg.workspace_check(dev.ws_ptr)
            got = dev.asg_host()
            assert np.array_equal(got, want), (lay, pkg.ASSIGN_NAMES[variant], int((got != want).sum()))
