"""GPU: the stateless runner entry points called the way the reference's drivers call their runners -
every iteration, on one workspace, with the same (immutable) points.  The workspace keeps the
operands derived from the points between calls; these tests check that a repeated call gives the
same (oracle) result, that NEW data at the same address and shape is noticed, and that
bkm_iterate_f32's single pass (assignment kernel accumulating the update sums) equals the oracle's
iteration (serial.hpp:21-73 restated in oracle/)."""
import numpy as np
import pytest

from helpers import DeviceArrays, means_close, rows_to_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,d,layout,variant", [(20000, 512, 32, 1, 3), (9000, 300, 20, 0, 3), (30000, 64, 2, 0, 2), (5000, 17, 7, 1, 2)])
def test_repeated_calls_reuse_the_workspace_and_notice_new_points(pkg, torch_cuda, oracle_mod, n, k, d, layout, variant):
    torch = torch_cuda
    rng = np.random.default_rng(n + k + d)
    rows_a = rng.random((n, d), dtype=np.float32)
    rows_b = (rng.random((n, d), dtype=np.float32) * 3.0 - 1.0).astype(np.float32)       # other values, larger norms
    means_1 = rng.random((k, d), dtype=np.float32)
    means_2 = rng.random((k, d), dtype=np.float32)
    dev = DeviceArrays(torch, pkg, rows_to_layout(rows_a, layout), rows_to_layout(means_1, layout), n, k, d)

    def call(rows, means):
        dev.means.copy_(torch.from_numpy(rows_to_layout(means, layout)).to("cuda:0"))
        pkg.assign(dev.points.data_ptr(), dev.means.data_ptr(), dev.assignment.data_ptr(), n, k, d, layout, layout,
                   dev.ws_ptr, dev.ws_bytes_avail, variant=variant)
        pkg.workspace_check(dev.ws_ptr)
        want = oracle_mod.assign(rows_to_layout(rows, layout), rows_to_layout(means, layout), n, k, d, layout, layout, threads=8)
        got = dev.asg_host()
        assert np.array_equal(got, want), int((got != want).sum())

    call(rows_a, means_1)            # first call: operands are derived
    call(rows_a, means_2)            # same points: operands reused, new means
    call(rows_a, means_1)
    # new data at the same address and shape: the fingerprint differs, the operands are derived again
    dev.points.copy_(torch.from_numpy(rows_to_layout(rows_b, layout)).to("cuda:0"))
    call(rows_b, means_2)
    call(rows_b, means_1)
    # an update on the same workspace in between must not disturb what the assignment keeps there
    pkg.update(dev.points.data_ptr(), dev.assignment.data_ptr(), dev.means_out.data_ptr(), dev.sizes.data_ptr(),
               n, k, d, layout, layout, dev.ws_ptr, dev.ws_bytes_avail)
    pkg.workspace_check(dev.ws_ptr)
    call(rows_b, means_2)


@pytest.mark.parametrize("n,k,d,layout,layout_means,want_asg", [
    (20000, 1024, 32, 1, 1, True),     # CTA-pair kernel: single pass
    (7001, 512, 24, 1, 0, False),      # same, no assignment output, other means layout
    (9000, 300, 20, 0, 0, True),       # row-major points: two passes
    (30000, 64, 2, 0, 0, True),        # CUDA cores: single pass (every warp sorts its points by cluster)
    (12345, 100, 7, 1, 0, False),      # same, dimension-major points, no assignment output
    (12345, 300, 2, 1, 0, False),      # more means: two passes
    (12345, 512, 7, 0, 1, True),       # longer rows, as many as the single pass takes by itself
    (65537, 257, 4, 0, 0, True),       # one more point and mean than that: two passes
    (70000, 10, 3, 0, 0, True),        # more points in few clusters: two passes
    (5000, 2000, 3, 0, 0, True),       # CUDA cores, more means than the single pass takes: two passes
])
def test_iterate_matches_oracle_iteration(pkg, torch_cuda, oracle_mod, n, k, d, layout, layout_means, want_asg):
    torch = torch_cuda
    rng = np.random.default_rng(n * 3 + k)
    rows = rng.random((n, d), dtype=np.float32)
    data = rows_to_layout(rows, layout)
    means = rows_to_layout(np.ascontiguousarray(rows[:k]), layout_means)
    dev = DeviceArrays(torch, pkg, data, means, n, k, d)
    cur = means.copy()
    for it in range(3):
        dev.means.copy_(torch.from_numpy(cur).to("cuda:0"))
        pkg.iterate(dev.points.data_ptr(), dev.means.data_ptr(), dev.means_out.data_ptr(), dev.sizes.data_ptr(),
                    dev.assignment.data_ptr() if want_asg else 0, n, k, d, layout, layout_means, dev.ws_ptr, dev.ws_bytes_avail)
        pkg.workspace_check(dev.ws_ptr)
        asg = oracle_mod.assign(data, cur, n, k, d, layout, layout_means, threads=8)
        if want_asg:
            assert np.array_equal(dev.asg_host(), asg), it
        want_means, want_sizes = oracle_mod.update(data, asg, n, k, d, layout, layout_means)
        assert np.array_equal(dev.sizes.cpu().numpy().view(np.uint32), want_sizes), it
        got = dev.means_out.cpu().numpy()
        ok, err = means_close(got, want_means)
        assert ok, (it, err)
        cur = got.copy()


@pytest.mark.parametrize("n,d,variant,small,large", [(5000, 24, 3, 40, 300), (3000, 70, 3, 40, 700), (9000, 4, 2, 20, 700)])
@pytest.mark.parametrize("layout", [0, 1])
def test_one_workspace_serves_calls_with_different_numbers_of_means(pkg, torch_cuda, oracle_mod, n, d, variant, small, large, layout):
    """The operands kept in a workspace lie behind ranges whose sizes depend on k: the same points with another
    k (a sweep over k on a workspace sized for the largest), and an update, a bucketing or an exact assignment
    with another k in between, must have them derived again."""
    torch = torch_cuda
    rng = np.random.default_rng(n + d)
    rows = rng.standard_normal((n, d)).astype(np.float32)
    data = rows_to_layout(rows, layout)
    dev = DeviceArrays(torch, pkg, data, rows_to_layout(rows[:large], layout), n, large, d)
    means = {k: rows_to_layout(rng.standard_normal((k, d)).astype(np.float32), layout) for k in (small, large)}
    want = {k: oracle_mod.assign(data, m, n, k, d, layout, layout, threads=8) for k, m in means.items()}

    def assign(k, v=variant):
        m = torch.from_numpy(means[k]).to("cuda:0")
        pkg.assign(dev.points.data_ptr(), m.data_ptr(), dev.assignment.data_ptr(), n, k, d, layout, layout, dev.ws_ptr, dev.ws_bytes_avail, variant=v)
        pkg.workspace_check(dev.ws_ptr)
        got = dev.asg_host()
        assert np.array_equal(got, want[k]), (k, v, int((got != want[k]).sum()))

    for k in (large, small, large, large, small):
        assign(k)
    # the workspace now remembers the points for `small`
    pkg.update(dev.points.data_ptr(), dev.assignment.data_ptr(), dev.means_out.data_ptr(), dev.sizes.data_ptr(), n, large, d, layout, layout,
               dev.ws_ptr, dev.ws_bytes_avail)
    assign(small)
    pkg.bucket_sums(dev.points.data_ptr(), dev.assignment.data_ptr(), dev.means_out.data_ptr(), n, large, d, layout, dev.ws_ptr, dev.ws_bytes_avail)
    assign(small)
    assign(large, 1)
    assign(small)
    # fewer points: the same ranges mean something else again
    pkg.update(dev.points.data_ptr(), dev.assignment.data_ptr(), dev.means_out.data_ptr(), dev.sizes.data_ptr(), n // 2, small, d, 0, layout,
               dev.ws_ptr, dev.ws_bytes_avail)
    assign(small)


def test_threads_that_replace_each_others_plans(pkg, torch_cuda, oracle_mod):
    """The library keeps eight tensor-core plans; three threads with six shapes each keep replacing the others'
    while their calls are being enqueued, each on a stream and workspaces of its own."""
    import threading
    torch = torch_cuda
    n = 700

    def job(t, errors):
        try:
            torch.cuda.set_device(0)
            stream = torch.cuda.Stream()
            rng = np.random.default_rng(t)
            work = []
            for k, d in ((20 + t, 16), (40 + t, 32), (300 + t, 32), (300 + t, 64), (40 + t, 90), (1030 + t, 260)):
                data, means = (rng.standard_normal(m * d).astype(np.float32) for m in (n, k))
                work.append((k, d, DeviceArrays(torch, pkg, data, means, n, k, d), oracle_mod.assign(data, means, n, k, d, 0, 0, threads=2)))
            torch.cuda.synchronize()
            for _ in range(20):
                for k, d, dev, _want in work:
                    pkg.assign(dev.points.data_ptr(), dev.means.data_ptr(), dev.assignment.data_ptr(), n, k, d, 0, 0, dev.ws_ptr, dev.ws_bytes_avail,
                               variant=pkg.ASSIGN_TC, stream=stream.cuda_stream)
            stream.synchronize()
            for k, d, dev, want in work:
                if not np.array_equal(dev.asg_host(), want):
                    errors.append((t, k, d))
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append((t, repr(e)))

    errors = []
    threads = [threading.Thread(target=job, args=(t, errors)) for t in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
