"""GPU: the fp16 operand pairs of the tensor-core assignment where their range and resolution matter,
every point against the oracle (the exact re-check makes the assignment bit-identical), at the edges of
the operand rows (16 words, 32 words, slices of 16 words) and of the kernels that read them."""
import numpy as np
import pytest

from helpers import DeviceArrays, means_close, rows_to_layout

pytestmark = pytest.mark.gpu


def _rows(kind, n, k, d, rng):
    rows = rng.standard_normal((n, d)).astype(np.float32)
    means = None
    if kind == "outliers":           # a few points far beyond what the sampled scale leaves room for
        rows[rng.integers(0, n, max(1, n // 100))] *= np.float32(1e6)
    elif kind == "mixed-scales":     # dimensions whose ranges differ by five orders of magnitude
        rows *= np.logspace(-5, 0, d, dtype=np.float32)
    elif kind == "tiny":
        rows *= np.float32(1e-12)
    elif kind == "huge":
        rows *= np.float32(1e12)
    elif kind == "far-means":        # means that the scale of the points cannot hold: every point is re-checked
        means = rows[:k].copy()
        means[::3] *= np.float32(1e5)
    elif kind == "constant":         # the sample shows no deviation at all
        rows[:] = np.float32(0.3)
        rows[n // 2] = np.float32(7.0)
    return rows, (rows[:k].copy() if means is None else means)


@pytest.mark.parametrize("n,k,d", [(1000, 40, 16), (1500, 300, 17), (1301, 300, 32), (1300, 513, 33), (900, 300, 48), (900, 257, 64),
                                   (700, 40, 65), (700, 600, 97), (300, 257, 47)])
@pytest.mark.parametrize("kind", ["outliers", "mixed-scales", "tiny", "huge", "far-means", "constant"])
def test_operand_ranges_match_oracle(pkg, torch_cuda, oracle_mod, n, k, d, kind):
    rows, mrows = _rows(kind, n, k, d, np.random.default_rng(n + d))
    for layout in (0, 1):
        data, means = rows_to_layout(rows, layout), rows_to_layout(mrows, layout)
        want = oracle_mod.assign(data, means, n, k, d, layout, layout, threads=8)
        dev = DeviceArrays(torch_cuda, pkg, data, means, n, k, d)
        pkg.assign(dev.points.data_ptr(), dev.means.data_ptr(), dev.assignment.data_ptr(), n, k, d, layout, layout,
                   dev.ws_ptr, dev.ws_bytes_avail, variant=pkg.ASSIGN_TC)
        pkg.workspace_check(dev.ws_ptr)
        got = dev.asg_host()
        assert np.array_equal(got, want), (layout, int((got != want).sum()))


@pytest.mark.parametrize("n,kind", [(2560, "mixed-scales"), (2047, "mixed-scales"), (129, "mixed-scales"), (16384, "beyond"), (16383, "beyond")])
@pytest.mark.parametrize("d,layout", [(32, 1), (20, 1), (32, 0)])
def test_fused_sums_come_from_the_raw_rows(pkg, torch_cuda, oracle_mod, n, d, layout, kind):
    """The CTA-pair kernel adds the points themselves, not what its operands hold of them: dimensions
    of very different ranges keep their precision, and a point beyond the operands' range (far outside of
    what the sample showed) reaches only the sum of its own cluster - an addition and subtraction of 1e6
    elsewhere would leave 0.1 behind.  Rows that start on 16-byte boundaries (n a multiple of 4) and rows
    that do not."""
    k = 300 if n > 300 else 260
    rng = np.random.default_rng(7 * n + d)
    rows, _ = _rows(kind, n, k, d, rng)
    if kind == "beyond":
        unseen = np.setdiff1d(np.arange(k, n), (np.arange(8192, dtype=np.int64) * n) // 8192)     # points that the sample leaves out
        rows[rng.choice(unseen, 40, replace=False)] *= np.float32(1e6)
    mrows = np.ascontiguousarray(np.resize(rows, (k, d)))
    data, means = rows_to_layout(rows, layout), rows_to_layout(mrows, layout)
    km = pkg.KMeans(layout=layout, variant_assign=pkg.ASSIGN_TC, variant_update=pkg.UPDATE_ROWS)
    km.initialize(d, k, n, 1, data, means)
    km.run(1)
    asg, cur, sizes = km.getAssignment(), km.getMeans(), km.getSizes()
    info = km.counters()
    km.cleanup()
    assert info["update_variant"] == "fused"
    assert np.array_equal(asg, oracle_mod.assign(data, means, n, k, d, layout, layout, threads=8))
    want, want_sizes = oracle_mod.update(data, asg, n, k, d, layout, layout)
    assert np.array_equal(sizes, want_sizes)
    # per dimension: 32-bit sums of some dozen points (at most a hundred), each step within 2^-24 of the sum of absolute values
    got2, want2 = (np.asarray(a, np.float64).reshape((k, d) if layout == 0 else (d, k)) for a in (cur, want))
    if layout == 1:
        got2, want2 = got2.T, want2.T
    scale = np.zeros((k, d))
    np.add.at(scale, asg, np.abs(rows.astype(np.float64)))
    scale /= np.maximum(sizes, 1)[:, None]
    assert np.all(np.abs(got2 - want2) <= 100 * 2.0 ** -24 * scale + 1e-300)


def test_scale_is_taken_again_when_the_first_chunk_misleads(pkg, torch_cuda, oracle_mod):
    """Host points of 32 MB and more travel in chunks and the first one sets the scale: points that grow
    by orders of magnitude behind it must not all end up in the exact kernel."""
    n, k, d = 350003, 64, 24
    rng = np.random.default_rng(3)
    rows = rng.standard_normal((n, d)).astype(np.float32)
    rows[:60000] *= np.float32(1e-6)
    mrows = np.ascontiguousarray(rows[-k:])
    data, means = rows_to_layout(rows, 0), rows_to_layout(mrows, 0)
    km = pkg.KMeans(layout=0)
    km.initialize(d, k, n, 1, data, means)
    km.run(1)
    asg, cur, info = km.getAssignment(), km.getMeans(), km.counters()
    km.cleanup()
    assert info["assign_variant"] == "tc" and info["rechecked"] < n // 4, info
    assert np.array_equal(asg, oracle_mod.assign(data, means, n, k, d, 0, 0, threads=8))
    ok, err = means_close(cur, oracle_mod.update(data, asg, n, k, d, 0, 0)[0])
    assert ok, err
