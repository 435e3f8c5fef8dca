"""GPU: points near the bisector of two means, at every distance from it that the band of the CUDA-core pass could get
wrong: from a fraction of a spacing of its values to several times the band.  The labels are the serial arithmetic's."""
import numpy as np
import pytest

from helpers import DeviceArrays, rows_to_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", [1.0, 0.03, 1e-3])      # distance of the means from each other against the distance from the centre
@pytest.mark.parametrize("d", range(1, 9))
def test_gaps_of_a_few_spacings(pkg, torch_cuda, oracle_mod, d, spread):
    rng = np.random.default_rng(100 * d + int(1000 * spread))
    n, k = 120000, 48
    clusters = rng.random((6, d)) * 4.0
    means = (clusters[rng.integers(0, 6, k)] + spread * (rng.random((k, d)) - 0.5)).astype(np.float32)
    wide = means.astype(np.float64)
    dist = ((wide[:, None] - wide[None]) ** 2).sum(2)
    np.fill_diagonal(dist, np.inf)
    a = rng.integers(0, k, n)
    b = dist.argmin(1)[a]                            # the nearest other mean: no third one is nearer to the middle
    along = wide[b] - wide[a]
    length = np.sqrt((along ** 2).sum(1, keepdims=True)) + 1e-30
    centred = wide - wide.mean(0)
    binade = 2.0 ** np.ceil(np.log2(2.5 * 2.0 * (centred ** 2).sum(1).max()))
    gap = rng.uniform(-1, 1, (n, 1)) * 2.0 ** rng.uniform(-2, 6, (n, 1)) * binade * 2.0 ** -23
    across = rng.standard_normal((n, d)) * 0.1 * length
    across -= along * ((across * along).sum(1, keepdims=True) / length ** 2)
    rows = ((wide[a] + wide[b]) / 2 + across + along / length * (gap / (2 * length))).astype(np.float32)
    for lay, laym in ((0, 0), (1, 1)):
        data, m = rows_to_layout(rows, lay), rows_to_layout(means, laym)
        want = oracle_mod.assign(data, m, n, k, d, lay, laym, threads=8)
        dev = DeviceArrays(torch_cuda, pkg, data, m, n, k, d)
        pkg.assign(dev.points.data_ptr(), dev.means.data_ptr(), dev.assignment.data_ptr(), n, k, d, lay, laym,
                   dev.ws_ptr, dev.ws_bytes_avail, variant=pkg.ASSIGN_SIMT)
        pkg.workspace_check(dev.ws_ptr)
        got = dev.asg_host()
        assert np.array_equal(got, want), (lay, int((got != want).sum()))
    # the form that settles its near-ties itself
    km = pkg.KMeans(layout=0, variant_assign=pkg.ASSIGN_SIMT)
    km.initialize(d, k, n, 1, rows.reshape(-1), means.reshape(-1))
    km.set_option("fuse_update", 2)
    km.run(1)
    want = oracle_mod.assign(rows.reshape(-1), means.reshape(-1), n, k, d, 0, 0, threads=8)
    got = km.getAssignment()
    km.cleanup()
    assert np.array_equal(got, want), int((got != want).sum())
