"""GPU: the exact re-check in its forms for short lists, lists of pairs and points settled in the fast
pass, and the sorted update at the edges of its chunk sizes, against the oracle."""
import numpy as np
import pytest

from helpers import DeviceArrays, means_close, rows_to_layout

pytestmark = pytest.mark.gpu


def _assign(pkg, torch, data, means, n, k, d, lay, laym, variant):
    dev = DeviceArrays(torch, pkg, data, means, n, k, d)
    pkg.assign(dev.points.data_ptr(), dev.means.data_ptr(), dev.assignment.data_ptr(), n, k, d, lay, laym,
               dev.ws_ptr, dev.ws_bytes_avail, variant=variant)
    pkg.workspace_check(dev.ws_ptr)
    return dev.asg_host()


@pytest.mark.parametrize("n", [1, 33, 5000, 300000])
@pytest.mark.parametrize("k,d", [(2, 1), (5, 2), (127, 3), (64, 4), (600, 6), (512, 8), (37, 12), (256, 16)])
def test_lists_of_small_mean_sets(pkg, torch_cuda, oracle_mod, n, k, d):
    """Every mean exists twice, so every point is queued: one point to one list longer than the grid, with
    as many lanes per point as that leaves, and mean counts that are no multiple of the lanes.  The
    lower index of two equal distances wins."""
    rng = np.random.default_rng(n + k + d)
    centres = rng.random((k, d), dtype=np.float32)
    centres[(k + 1) // 2:] = centres[:k // 2]
    rows = rng.random((n, d), dtype=np.float32)
    lay, laym = (n + k) % 2, d % 2
    data, means = rows_to_layout(rows, lay), rows_to_layout(centres, laym)
    got = _assign(pkg, torch_cuda, data, means, n, k, d, lay, laym, pkg.ASSIGN_TC if d > 8 else pkg.ASSIGN_SIMT)
    assert np.array_equal(got, oracle_mod.assign(data, means, n, k, d, lay, laym, threads=8))


@pytest.mark.parametrize("lay,laym", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("n,k,d", [(1500, 1024, 256), (700, 1100, 300), (400, 2050, 513)])
def test_near_ties_of_two_and_of_more_means_in_the_k_loop(pkg, torch_cuda, oracle_mod, n, k, d, lay, laym):
    """A third of the means exists twice (exactly, or apart by a few roundings), another third three times:
    the points of the former are settled between two candidates, those of the latter go through the list."""
    rng = np.random.default_rng(k + d)
    centres = rng.standard_normal((k, d)).astype(np.float32)
    t = k // 6
    centres[t:2 * t] = centres[:t]
    centres[t:t + t // 2, 0] = np.nextafter(centres[t:t + t // 2, 0], np.float32(9))
    centres[3 * t:4 * t] = centres[2 * t:3 * t]
    centres[4 * t:5 * t] = centres[2 * t:3 * t]
    rows = (centres[rng.integers(0, k, n)] + 0.3 * rng.standard_normal((n, d))).astype(np.float32)
    data, means = rows_to_layout(rows, lay), rows_to_layout(centres, laym)
    want = oracle_mod.assign(data, means, n, k, d, lay, laym, threads=8)
    km = pkg.KMeans(layout=lay, layout_means=laym, variant_assign=pkg.ASSIGN_TC)
    km.initialize(d, k, n, 1, data, means)
    assert km.assign_plan()["block_split"] == 2
    km.run(1)
    got, info = km.getAssignment(), km.counters()
    km.cleanup()
    assert info["rechecked"] >= n // 2
    assert np.array_equal(got, want), int((got != want).sum())
    assert np.array_equal(_assign(pkg, torch_cuda, data, means, n, k, d, lay, laym, pkg.ASSIGN_TC), want)


@pytest.mark.parametrize("blocks_x2,chunk,d", [(2, 512, 2), (1, 2048, 2), (2, 2048, 2), (2, 512, 16), (5, 512, 16), (5, 1024, 16), (5, 2048, 16)])
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_sorted_update_at_chunk_edges(pkg, torch_cuda, oracle_mod, blocks_x2, chunk, d, extra):
    """Half a block of 2048 points per SM (up to 8 dimensions) and two and a half blocks per SM (longer rows), where
    the chunk of the sorted update changes, and full last chunks of each size."""
    sms = torch_cuda.cuda.get_device_properties(0).multi_processor_count
    n, k = sms * blocks_x2 // 2 * chunk + extra, 9
    rng = np.random.default_rng(chunk + extra)
    rows = rng.random((n, d), dtype=np.float32)
    asg = rng.integers(0, k, n).astype(np.uint32)
    dev = DeviceArrays(torch_cuda, pkg, rows.reshape(-1), rows[:k].reshape(-1).copy(), n, k, d)
    dev.assignment.copy_(torch_cuda.from_numpy(asg.view(np.int32)))
    pkg.update(dev.points.data_ptr(), dev.assignment.data_ptr(), dev.means_out.data_ptr(), dev.sizes.data_ptr(), n, k, d, 0, 0,
               dev.ws_ptr, dev.ws_bytes_avail, variant=pkg.UPDATE_SORTED)
    pkg.workspace_check(dev.ws_ptr)
    want, want_sizes = oracle_mod.update_f64(rows.reshape(-1), asg, n, k, d, 0, 0)
    assert np.array_equal(dev.sizes.cpu().numpy().view(np.uint32), want_sizes)
    ok, err = means_close(dev.means_out.cpu().numpy(), want)
    assert ok, err


@pytest.mark.parametrize("share", [0.02, 0.3, 1.0])
@pytest.mark.parametrize("n", [1, 130, 1100, 9000])
@pytest.mark.parametrize("k,d", [(1, 3), (2, 1), (7, 2), (9, 8), (64, 4), (600, 2), (1000, 8), (1024, 5)])
def test_near_ties_settled_in_the_fused_pass(pkg, torch_cuda, oracle_mod, n, k, d, share):
    """From one near-tie per warp to all of its points, each with as many lanes as that leaves: a share of the
    points lies at means that exist twice (the lower index wins), the others far from them."""
    rng = np.random.default_rng(n + 3 * k + d)
    centres = rng.random((k, d), dtype=np.float32)
    half = k // 2
    centres[half:2 * half:2] = centres[:half:2]            # every second mean of the first half exists twice
    twice, once = np.arange(0, max(half, 1), 2), np.arange(1 if half > 1 else 0, max(half, 1), 2 if half > 1 else 1)
    pick = np.where(rng.random(n) < share, rng.choice(twice, n), rng.choice(once, n))
    rows = (centres[pick] + np.float32(1e-3) * rng.standard_normal((n, d)).astype(np.float32)).astype(np.float32)
    lay, laym = (n + k) % 2, d % 2
    data, means = rows_to_layout(rows, lay), rows_to_layout(centres, laym)
    km = pkg.KMeans(layout=lay, layout_means=laym, variant_assign=pkg.ASSIGN_SIMT)
    km.initialize(d, k, n, 1, data, means)
    km.set_option("fuse_update", 2)
    km.run(1)
    got, cur, sizes, info = km.getAssignment(), km.getMeans(), km.getSizes(), km.counters()
    km.cleanup()
    assert info["update_variant"] == "fused"
    want = oracle_mod.assign(data, means, n, k, d, lay, laym, threads=8)
    assert np.array_equal(got, want), int((got != want).sum())
    assert info["rechecked"] >= (np.isin(pick, twice).sum() if half > 1 else 0)
    want_means, want_sizes = oracle_mod.update(data, want, n, k, d, lay, laym)
    assert np.array_equal(sizes, want_sizes)
    ok, err = means_close(cur, want_means)
    assert ok, err
