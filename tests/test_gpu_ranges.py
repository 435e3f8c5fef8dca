"""GPU: the label of every point is the serial arithmetic's also where that arithmetic leaves the range of
32-bit numbers - squares that vanish or lose bits (the lowest index of several equal distances wins), squares
or sums that become infinite, coordinates that are infinite or not a number - in every assignment variant."""
import numpy as np
import pytest

from helpers import DeviceArrays, rows_to_layout

pytestmark = pytest.mark.gpu

TC_SHAPES = [(1500, 40, 16), (1500, 40, 32), (900, 300, 32), (900, 300, 64), (700, 40, 97), (300, 300, 513), (300, 1100, 260)]
SIMT_SHAPES = [(3001, 40, 1), (3000, 40, 3), (2000, 300, 8), (900, 1100, 4)]
FACTORS = [1e-38, 1e-30, 1e-24, 1e-22, 1e-21, 1e-20, 1e-18, 1e17, 1e18, 1e19, 1e21, 1e30, 1e37]


def _inputs(n, k, d, factor):
    rng = np.random.default_rng(n + 7 * k + d)
    rows = (rng.standard_normal((n, d)) * factor).astype(np.float32)
    means = (rng.standard_normal((k, d)) * factor).astype(np.float32)
    return rows, means


def _spoil(rows, means, kind):
    """Puts what is not finite into single coordinates of points ("p-...") or of means ("m-...")."""
    rng = np.random.default_rng(len(rows) + len(means))
    n, d = rows.shape
    k = len(means)
    value = {"nan": np.nan, "+inf": np.inf, "-inf": -np.inf}[kind[2:]]
    if kind[0] == "p":
        for i in rng.choice(n, n // 50, replace=False):
            rows[i, rng.integers(0, d)] = value
    else:
        for m in set(rng.choice(np.arange(1, k), max(1, k // 10), replace=False)) | {1}:
            means[m, rng.integers(0, d)] = value
        if len(rows) % 2:
            means[0, 0] = value
    return rows, means


def _check_assign(pkg, torch, oracle_mod, rows, mrows, variant, layouts=((0, 0), (1, 1), (0, 1), (1, 0))):
    (n, d), k = rows.shape, len(mrows)
    for lay, laym in layouts:
        data, means = rows_to_layout(rows, lay), rows_to_layout(mrows, laym)
        want = oracle_mod.assign(data, means, n, k, d, lay, laym, threads=8)
        dev = DeviceArrays(torch, pkg, data, means, n, k, d)
        pkg.assign(dev.points.data_ptr(), dev.means.data_ptr(), dev.assignment.data_ptr(), n, k, d, lay, laym,
                   dev.ws_ptr, dev.ws_bytes_avail, variant=variant)
        pkg.workspace_check(dev.ws_ptr)
        got = dev.asg_host()
        assert np.array_equal(got, want), (lay, laym, int((got != want).sum()))


@pytest.mark.parametrize("factor", FACTORS)
@pytest.mark.parametrize("n,k,d", TC_SHAPES)
def test_tensor_core_labels_where_squares_underflow_or_overflow(pkg, torch_cuda, oracle_mod, n, k, d, factor):
    _check_assign(pkg, torch_cuda, oracle_mod, *_inputs(n, k, d, factor), pkg.ASSIGN_TC, ((0, 0), (1, 1)))


@pytest.mark.parametrize("kind", ["p-nan", "p-+inf", "p--inf", "m-nan", "m-+inf", "m--inf"])
@pytest.mark.parametrize("n,k,d", TC_SHAPES + [(901, 300, 32)])
def test_tensor_core_labels_of_values_that_are_not_finite(pkg, torch_cuda, oracle_mod, n, k, d, kind):
    _check_assign(pkg, torch_cuda, oracle_mod, *_spoil(*_inputs(n, k, d, 1.0), kind), pkg.ASSIGN_TC, ((0, 0), (1, 1)))


def _check_handle(pkg, oracle_mod, rows, mrows, layout, variant_assign, variant_update, fused_name, options=()):
    """One iteration through a handle whose assignment pass adds the points up itself."""
    (n, d), k = rows.shape, len(mrows)
    data, means = rows_to_layout(rows, layout), rows_to_layout(mrows, layout)
    km = pkg.KMeans(layout=layout, variant_assign=variant_assign, variant_update=variant_update)
    km.initialize(d, k, n, 1, data, means)
    for name, value in options:
        km.set_option(name, value)
    km.run(1)
    asg, cur, sizes, info = km.getAssignment(), km.getMeans(), km.getSizes(), km.counters()
    km.cleanup()
    assert info["update_variant"] == fused_name
    want_asg = oracle_mod.assign(data, means, n, k, d, layout, layout, threads=8)
    assert np.array_equal(asg, want_asg), int((asg != want_asg).sum())
    want, want_sizes = oracle_mod.update(data, want_asg, n, k, d, layout, layout)
    assert np.array_equal(sizes, want_sizes)
    got, want = (np.asarray(a, np.float64).reshape((k, d) if layout == 0 else (d, k)) for a in (cur, want))
    if layout == 1:
        got, want = got.T, want.T
    # What is not finite is the same value.  The rest: a sum takes its points and, added and subtracted again,
    # those that the pass had put there first (their nearest mean in real numbers); each of these steps is
    # within 2^-24 of the sum of the absolute values.
    finite = np.isfinite(want)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(got[~finite & ~np.isnan(want)], want[~finite & ~np.isnan(want)])
    rows64, means64 = rows.astype(np.float64), mrows.astype(np.float64)
    scale, steps = np.zeros((k, d)), want_sizes.astype(np.float64)
    with np.errstate(invalid="ignore"):
        first = np.argmin((means64 ** 2).sum(1) - 2.0 * rows64 @ means64.T, axis=1)
        for labels in (asg, first, first):
            np.add.at(scale, labels, np.abs(rows64))
    steps += 2.0 * np.bincount(first, minlength=k)
    bound = 2.0 ** -24 * (scale * (steps / np.maximum(want_sizes, 1))[:, None] + np.abs(want)) + 1e-44
    assert np.all(np.abs(got - want)[finite] <= bound[finite])


@pytest.mark.parametrize("kind", ["1e-30", "1e-22", "1e18", "1e19", "1e30", "p-nan", "p-+inf", "m-nan", "m--inf"])
@pytest.mark.parametrize("n,k,d,layout", [(2501, 300, 32, 1), (2500, 600, 20, 0), (3000, 1024, 32, 1)])
def test_sums_of_the_cta_pair_pass_where_squares_leave_the_range(pkg, torch_cuda, oracle_mod, n, k, d, layout, kind):
    """Points that the pass cannot place are added once, by the exact kernel: an addition to a wrong sum and
    the subtraction after it would leave rounding errors or, with infinities, nothing but NaN."""
    if kind[0] in "pm":
        rows, means = _spoil(*_inputs(n, k, d, 1.0), kind)
    else:
        rows, means = _inputs(n, k, d, float(kind))
    _check_handle(pkg, oracle_mod, rows, means, layout, pkg.ASSIGN_TC, pkg.UPDATE_ROWS, "fused")


@pytest.mark.parametrize("factor", FACTORS)
@pytest.mark.parametrize("n,k,d", SIMT_SHAPES)
def test_cuda_core_labels_where_squares_underflow_or_overflow(pkg, torch_cuda, oracle_mod, n, k, d, factor):
    _check_assign(pkg, torch_cuda, oracle_mod, *_inputs(n, k, d, factor), pkg.ASSIGN_SIMT, ((0, 0), (1, 1)))


@pytest.mark.parametrize("kind", ["p-nan", "p-+inf", "p--inf", "m-nan", "m-+inf", "m--inf"])
@pytest.mark.parametrize("n,k,d", SIMT_SHAPES)
def test_cuda_core_labels_of_values_that_are_not_finite(pkg, torch_cuda, oracle_mod, n, k, d, kind):
    _check_assign(pkg, torch_cuda, oracle_mod, *_spoil(*_inputs(n, k, d, 1.0), kind), pkg.ASSIGN_SIMT, ((0, 0), (1, 1)))


@pytest.mark.parametrize("kind", ["1e-30", "1e-22", "5e18", "1e19", "1e30", "p-nan", "p-+inf", "m-nan", "m--inf"])
@pytest.mark.parametrize("n,k,d,layout", [(3001, 40, 1, 0), (3000, 60, 3, 1), (2000, 300, 8, 0)])
def test_sums_of_the_cuda_core_pass_where_squares_leave_the_range(pkg, torch_cuda, oracle_mod, n, k, d, layout, kind):
    if kind[0] in "pm":
        rows, means = _spoil(*_inputs(n, k, d, 1.0), kind)
    else:
        rows, means = _inputs(n, k, d, float(kind))
    _check_handle(pkg, oracle_mod, rows, means, layout, pkg.ASSIGN_SIMT, pkg.UPDATE_AUTO, "fused", (("fuse_update", 2),))


@pytest.mark.parametrize("kind", ["p-nan", "p-+inf", "m-nan", "m--inf", "1e-24", "1e19"])
@pytest.mark.parametrize("n,k,d", [(301, 70, 3), (300, 70, 40), (201, 33, 513), (200, 1, 2)])
def test_exact_variant_and_double_precision_outside_the_range(pkg, torch_cuda, oracle_mod, n, k, d, kind):
    """A mean whose distance is not a number never wins, but must not hide the means behind it either."""
    if kind[0] in "pm":
        rows, means = _inputs(n, k, d, 1.0)
        if k > 1:
            rows, means = _spoil(rows, means, kind)
    else:
        rows, means = _inputs(n, k, d, float(kind))
    _check_assign(pkg, torch_cuda, oracle_mod, rows, means, pkg.ASSIGN_EXACT)
    if kind == "1e-24" or kind == "1e19":
        rows, means = rows.astype(np.float64) * float(kind) ** 7.2, means.astype(np.float64) * float(kind) ** 7.2
    for lay, laym in ((0, 0), (1, 1), (0, 1), (1, 0)):
        data, m0 = (np.ascontiguousarray(a if lx == 0 else a.T, dtype=np.float64).reshape(-1) for a, lx in ((rows, lay), (means, laym)))
        got = pkg.kmeans_host_f64(data, m0, n, k, d, 1, lay, laym)[1]
        assert np.array_equal(got, oracle_mod.assign_f64(data, m0, n, k, d, lay, laym, threads=8)), (lay, laym)
