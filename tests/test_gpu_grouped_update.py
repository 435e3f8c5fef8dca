"""GPU: the update of long row-major rows for many clusters, which sorts all points by cluster first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# columns of one warp, of one and a bit, of several; the fewest and the most clusters; clusters of every size, empty ones among them
@pytest.mark.parametrize("n,k,d", [(17000, 1025, 256), (20011, 1100, 260), (70001, 4096, 384), (131072, 8192, 256), (24000, 1200, 516)])
@pytest.mark.parametrize("skew", [False, True])
def test_sums_and_sizes(pkg, torch_cuda, n, k, d, skew):
    torch = torch_cuda
    gen = torch.Generator(device="cuda").manual_seed(n + k + d)
    pts = torch.randn((n, d), generator=gen, device="cuda")
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    asg = ((u ** 6 if skew else u) * (k - 1)).to(torch.int32)          # (the last cluster stays empty)
    size = pkg.workspace_bytes(n, k, d)
    ws = torch.full((size,), 0x5A, dtype=torch.uint8, device="cuda")
    means = torch.full((k, d), float("nan"), device="cuda")
    sizes = torch.full((k,), -1, dtype=torch.int32, device="cuda")
    wide = torch.zeros((k, d), dtype=torch.float64, device="cuda").index_add_(0, asg.long(), pts.double())
    mass = torch.zeros((k, d), dtype=torch.float64, device="cuda").index_add_(0, asg.long(), pts.double().abs())
    want = torch.bincount(asg.long(), minlength=k)
    for _ in range(2):
        pkg.update(pts.data_ptr(), asg.data_ptr(), means.data_ptr(), sizes.data_ptr(), n, k, d, 0, 0, ws.data_ptr(), size)
        pkg.workspace_check(ws.data_ptr())
        assert torch.equal(sizes.long(), want)
        # a sum of m terms in any order is within m * 2^-24 of the sum of their magnitudes; the division adds half an ulp
        count = want.clamp(min=1).double()[:, None]
        bound = (count + 1) * 2.0 ** -24 * mass / count + 1e-30
        assert bool(((means.double() - wide / count).abs() <= bound).all())


def test_bad_indices_are_reported_and_left_out(pkg, torch_cuda):
    torch = torch_cuda
    n, k, d = 20000, 1100, 256
    pts = torch.ones((n, d), device="cuda")
    asg = (torch.arange(n, device="cuda") % k).to(torch.int32)
    asg[17] = k
    asg[n - 1] = 0x7fffffff
    size = pkg.workspace_bytes(n, k, d)
    ws = torch.zeros(size, dtype=torch.uint8, device="cuda")
    means = torch.empty((k, d), device="cuda")
    sizes = torch.empty(k, dtype=torch.int32, device="cuda")
    pkg.update(pts.data_ptr(), asg.data_ptr(), means.data_ptr(), sizes.data_ptr(), n, k, d, 0, 0, ws.data_ptr(), size)
    with pytest.raises(pkg.BkmError):
        pkg.workspace_check(ws.data_ptr())
    assert int(sizes.sum()) == n - 2 and bool((means == 1.0).all())
