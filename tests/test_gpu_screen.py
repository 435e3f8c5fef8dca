"""GPU: rows longer than 64 dimensions go through a pass with the fp16 high parts alone first; the points it leaves open
through the pass with all three products (gathered from a list), and the rest of them to the exact kernel.  The labels are
the serial arithmetic's whatever the share of open points."""
import numpy as np
import pytest

from helpers import rows_to_layout

pytestmark = pytest.mark.gpu


def _handle(pkg, rows, mrows, lay, laym):
    (n, d), k = rows.shape, len(mrows)
    km = pkg.KMeans(layout=lay, layout_means=laym, variant_assign=pkg.ASSIGN_TC)
    km.initialize(d, k, n, 2, rows_to_layout(rows, lay), rows_to_layout(mrows, laym))
    km.set_option("tc_screen", 2)                    # (these shapes are smaller than where it pays)
    return km


def _check(pkg, oracle_mod, rows, mrows, layouts=((0, 0), (1, 1))):
    (n, d), k = rows.shape, len(mrows)
    for lay, laym in layouts:
        want = oracle_mod.assign(rows_to_layout(rows, lay), rows_to_layout(mrows, laym), n, k, d, lay, laym, threads=8)
        km = _handle(pkg, rows, mrows, lay, laym)
        km.run(1)
        got = km.getAssignment()
        km.cleanup()
        assert np.array_equal(got, want), (lay, int((got != want).sum()))


# one slice of 64 dimensions and a bit, whole slices, half slices, rows that stay and rows that stream; mean tiles
# that are full and that hold one mean; an odd last tile of points
@pytest.mark.parametrize("n,k,d", [(1, 257, 65), (300, 300, 96), (20480, 512, 128), (20481, 513, 130), (9000, 260, 322), (4095, 300, 512), (5000, 280, 520)])
@pytest.mark.parametrize("kind", ["uniform", "clusters", "twins"])
def test_labels_match_the_oracle(pkg, torch_cuda, oracle_mod, n, k, d, kind):
    rng = np.random.default_rng(n + k + d)
    means = rng.random((k, d), dtype=np.float32)
    if kind == "uniform":
        rows = rng.random((n, d), dtype=np.float32)
    else:
        if kind == "twins":                          # every point is as close to a second mean: nothing is settled by the high parts
            means[k // 2:2 * (k // 2)] = means[:k // 2]
        rows = means[rng.integers(0, k, n)] + np.float32(0.02) * rng.standard_normal((n, d), dtype=np.float32)
    _check(pkg, oracle_mod, rows, means, ((0, 0), (1, 1)) if d < 300 else ((0, 1),))


def test_points_behind_the_first_wave_are_left_open_where_screening_does_not_help(pkg, torch_cuda, oracle_mod):
    """More than six waves of points, means in pairs: the first launch leaves all of its points open, the second
    does not multiply."""
    rng = np.random.default_rng(3)
    n, k, d = 120011, 300, 66
    means = rng.random((k, d), dtype=np.float32)
    means[150:] = means[:150]
    rows = means[rng.integers(0, k, n)] + np.float32(0.02) * rng.standard_normal((n, d), dtype=np.float32)
    _check(pkg, oracle_mod, rows, means, ((0, 0),))


def test_values_out_of_range_and_iterations(pkg, torch_cuda, oracle_mod):
    """Points beyond what the operands hold, and what is not finite, among ordinary ones; then two iterations of the handle
    (the counts of one iteration must not reach the next)."""
    rng = np.random.default_rng(8)
    n, k, d = 15666, 270, 70
    rows = rng.standard_normal((n, d)).astype(np.float32)
    means = rows[:k].copy()
    wild = rows.copy()
    wild[1000:1040] *= np.float32(1e4)
    wild[5000:5010, 3] = np.inf
    wild[7000:7010, 69] = np.nan
    _check(pkg, oracle_mod, wild, means, ((0, 0),))
    km = _handle(pkg, rows, means, 0, 0)
    km.run(1)
    want = oracle_mod.assign(rows.reshape(-1), means.reshape(-1), n, k, d, 0, 0, threads=8)
    assert np.array_equal(km.getAssignment(), want)
    second = km.getMeans().copy()
    km.run(1)
    want = oracle_mod.assign(rows.reshape(-1), second, n, k, d, 0, 0, threads=8)
    assert np.array_equal(km.getAssignment(), want)
    km.cleanup()


def test_the_rule_and_the_general_pass_agree(pkg, torch_cuda, oracle_mod):
    """The stateless call at a size where the rule takes the pass, against the pass with all products, and a sample against
    the oracle."""
    torch = torch_cuda
    n, k, d = 100003, 1024, 128
    gen = torch.Generator(device="cuda").manual_seed(5)
    pts = torch.randn((n, d), generator=gen, device="cuda")
    means = pts[:k].clone()
    ws_bytes = pkg.workspace_bytes(n, k, d)
    ws = torch.full((ws_bytes,), 0x7F, dtype=torch.uint8, device="cuda")
    got = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    for _ in range(2):                               # the second call finds the operands of the points in the workspace
        pkg.assign(pts.data_ptr(), means.data_ptr(), got.data_ptr(), n, k, d, 0, 0, ws.data_ptr(), ws_bytes)
        pkg.workspace_check(ws.data_ptr())
        km = pkg.KMeans(layout=0, variant_assign=pkg.ASSIGN_TC)
        km.initialize(d, k, n, 1, pts.cpu().numpy().reshape(-1), means.cpu().numpy().reshape(-1))
        km.set_option("tc_screen", 0)
        km.run(1)
        labels = got.cpu().numpy().view(np.uint32)
        assert np.array_equal(labels, km.getAssignment())
        km.cleanup()
    pick = np.random.default_rng(1).choice(n, 3000, replace=False)
    want = oracle_mod.assign(pts.cpu().numpy()[pick].reshape(-1), means.cpu().numpy().reshape(-1), len(pick), k, d, 0, 0, threads=8)
    assert np.array_equal(labels[pick], want)
