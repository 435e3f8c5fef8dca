"""What is timed: the calls a program makes of this library, over the range of sizes it makes them with.

Kinds of work (every case is one of them):
  restart   the fixed-iteration loop on points that already lie on the GPU behind a KMeans handle: set the
            initial means, run, fetch means and sizes (k-means is restarted from several initialisations on
            one data set; the labels stay on the GPU for whatever follows)
  encode    assignment only, the stateless call: batches of vectors that have not been seen before are
            labelled against a fixed codebook (vector quantisation, prediction for new points)
  iterate   the stateless one-iteration call in a loop of the caller's own, means double-buffered (how a host
            program with its own driver uses the kernel runners)
  update    the bucketed sum / count / divide alone, for labels that the caller already has
  host      the whole job on host buffers in one call: upload, iterations, results back
  host64    the same in double precision
Layouts: "aos" = rows of points, "soa" = one array per dimension; the means may have the other layout.
"""
import math

import numpy as np
import torch

from __graft_entry__ import load

LAYOUT = {"aos": 0, "soa": 1}

MAX_PAIR_COST = 3.0e-2      # seconds a drawn case may cost at the rough rates of pass_cost()
MAX_INPUT_BYTES = 5.0e9


def listed():
    return [
        # 64 Ki four-dimensional points in 16 clusters: a job of ten launch-bound iterations
        dict(name="restart-small", kind="restart", n=1 << 16, d=4, k=16, iters=10, layout="aos", layout_means="aos", data="mixture"),
        # the headline shape of the benchmark: 2 Mi uniform points of 32 dimensions, 1024 clusters, dimension-major
        dict(name="restart-headline", kind="restart", n=1 << 21, d=32, k=1024, iters=4, layout="soa", layout_means="soa", data="uniform"),
        # two-dimensional positions in few clusters of very different sizes
        dict(name="restart-plane", kind="restart", n=1 << 24, d=2, k=64, iters=5, layout="aos", layout_means="aos", data="zipf"),
        # normalised embeddings against many clusters: the dense contraction
        dict(name="restart-embeddings", kind="restart", n=1 << 20, d=512, k=4096, iters=2, layout="aos", layout_means="aos", data="sphere"),
        # one GPU's part of a very large set of 16-dimensional points
        dict(name="restart-shard", kind="restart", n=1 << 26, d=16, k=256, iters=3, layout="aos", layout_means="aos", data="mixture"),
        # sizes that divide nothing: features of 50 dimensions, 1000 clusters, means in the other layout
        dict(name="restart-ragged", kind="restart", n=300007, d=50, k=1000, iters=5, layout="aos", layout_means="soa", data="mixture"),
        # product quantisation: 8-dimensional sub-vectors against a 256-entry codebook, batch after batch
        dict(name="encode-subvectors", kind="encode", n=250000, d=8, k=256, iters=4, layout="aos", layout_means="aos", data="normal"),
        # coarse quantisation of 128-dimensional descriptors, batches of an odd size
        dict(name="encode-descriptors", kind="encode", n=100003, d=128, k=1024, iters=3, layout="aos", layout_means="aos", data="normal"),
        # colours of a thumbnail clustered by a program with its own loop: the smallest calls
        dict(name="iterate-colours", kind="iterate", n=20011, d=3, k=10, iters=6, layout="soa", layout_means="aos", data="uniform"),
        # the update step alone at the size of the reference's bucketing study
        dict(name="update-rows", kind="update", n=1 << 23, d=32, k=1024, iters=1, layout="aos", layout_means="aos", data="mixture"),
        # host program, one call, pinned buffers
        dict(name="host-job", kind="host", n=1 << 20, d=32, k=1024, iters=4, layout="soa", layout_means="soa", data="uniform"),
        # the same in double precision
        dict(name="host-job-double", kind="host64", n=1 << 18, d=8, k=64, iters=5, layout="aos", layout_means="aos", data="mixture"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def pass_cost(kind, n, d, k, iters):
    """A rough upper estimate of the seconds of one pass, to keep drawn cases within the listed ones' cost."""
    pairs = float(n) * k * iters
    if kind == "host64":
        return pairs * (10e-12 + 6e-12 * d) + n * d * 8 / 1e10
    compute = 0.0 if kind == "update" else pairs * (0.6e-12 + 0.012e-12 * d)
    return compute + iters * float(n) * d * 4 / 1e12 + (n * d * 4 / 1e10 if kind == "host" else 0.0)


def draw(rng):
    kind = rng.choice(["restart"] * 8 + ["encode"] * 4 + ["iterate"] * 3 + ["update"] * 2 + ["host"] * 2 + ["host64"])
    d = _log_int(rng, 1, 512) if kind != "host64" else _log_int(rng, 1, 32)
    k = _log_int(rng, 2, 4096) if kind != "host64" else _log_int(rng, 2, 256)
    iters = 1 if kind == "update" else rng.randint(2, 5)
    n_max = 1 << (24 if kind in ("restart", "update") else 21 if kind == "iterate" else 20 if kind != "host64" else 18)
    n = _log_int(rng, max(4 * k, 2000), max(n_max, 8 * k))
    while n > 4 * k and (pass_cost(kind, n, d, k, iters) > MAX_PAIR_COST or n * d * 4.0 * (iters if kind == "encode" else 1) > MAX_INPUT_BYTES):
        n = n // 2 + 1
    if rng.random() < 0.3:
        n = (n + 127) // 128 * 128
    layout = rng.choice(["aos", "soa"])
    means = layout if rng.random() < 0.7 else ("soa" if layout == "aos" else "aos")
    data = rng.choice(["mixture", "uniform", "normal", "zipf"] if d < 128 else ["sphere", "normal", "mixture"])
    return dict(kind=kind, n=n, d=d, k=k, iters=iters, layout=layout, layout_means=means, data=data)


# ---- inputs -------------------------------------------------------------------------------------------------

def _rows(case, gen, count):
    """(points [count, d] on the GPU, generating component of every point)."""
    n, d, k, kind = count, case["d"], case["k"], case["data"]
    out = torch.empty((n, d), dtype=torch.float32, device="cuda")
    which = torch.empty(n, dtype=torch.int32, device="cuda")
    centres = torch.rand((k, d), generator=gen, device="cuda")
    weights = 1.0 / torch.arange(1, k + 1, device="cuda", dtype=torch.float64) ** (1.1 if kind == "zipf" else 0.0)
    edges = torch.cumsum(weights / weights.sum(), 0)
    step = max(1, (1 << 26) // d)
    for a in range(0, n, step):
        b = min(n, a + step)
        pick = torch.searchsorted(edges, torch.rand(b - a, generator=gen, device="cuda", dtype=torch.float64)).clamp_(max=k - 1)
        which[a:b] = pick
        if kind == "uniform":
            out[a:b] = torch.rand((b - a, d), generator=gen, device="cuda")
            continue
        noise = torch.randn((b - a, d), generator=gen, device="cuda")
        if kind == "sphere":
            out[a:b] = noise / noise.norm(dim=1, keepdim=True)
        elif kind == "normal":
            out[a:b] = noise
        else:
            out[a:b] = centres[pick] + noise * (0.01 if kind == "zipf" else 0.05 / math.sqrt(d / 4.0))
    return out, which


def _flat(rows, layout):
    return (rows if layout == "aos" else rows.t().contiguous()).reshape(-1)


class _DeviceView:
    """Lets torch read a device buffer of the library; keeps its owner alive."""

    def __init__(self, owner, ptr, count):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<i4", "data": (ptr, False), "version": 3}


def prepare(case, seed):
    bkm = load()
    n, d, k, kind = case["n"], case["d"], case["k"], case["kind"]
    lay, laym = LAYOUT[case["layout"]], LAYOUT[case["layout_means"]]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = dict(case, bkm=bkm, lay=lay, laym=laym)
    batches = case["iters"] if kind == "encode" else 1
    rows, which = _rows(case, gen, n)
    means = rows[:k].clone()                      # the first k points
    s["points"] = [_flat(rows, case["layout"])]
    for _ in range(batches - 1):
        s["points"].append(_flat(_rows(case, gen, n)[0], case["layout"]))
    s["means"] = _flat(means, case["layout_means"])

    if kind == "restart":
        km = bkm.KMeans(layout=lay, layout_means=laym, device=torch.cuda.current_device())
        torch.cuda.synchronize()                  # the handle works on a stream of its own
        km.initialize_device(d, k, n, case["iters"], s["points"][0].data_ptr(), s["means"].data_ptr())
        s["km"] = km
        s["init"] = s["means"].cpu().numpy()
        s["assignment"] = torch.as_tensor(_DeviceView(km, km.device_assignment(), n), device="cuda")
        return s
    if kind in ("host", "host64"):
        f = torch.float64 if kind == "host64" else torch.float32
        s["points"] = s["points"][0].to(f).cpu().pin_memory().numpy()
        s["means"] = s["means"].to(f).cpu().numpy()
        return s
    size = bkm.workspace_bytes(n, k, d)
    s["workspace"] = torch.empty(size, dtype=torch.uint8, device="cuda")
    s["workspace_size"] = size
    if kind == "encode":
        s["labels"] = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(batches)]
        return s
    s["labels"] = which if kind == "update" else torch.empty(n, dtype=torch.int32, device="cuda")
    s["out"] = [torch.empty(k * d, dtype=torch.float32, device="cuda") for _ in range(2)]
    s["sizes"] = torch.empty(k, dtype=torch.int32, device="cuda")
    return s


# ---- one pass -----------------------------------------------------------------------------------------------

def run(s):
    bkm, n, d, k, kind, lay, laym = s["bkm"], s["n"], s["d"], s["k"], s["kind"], s["lay"], s["laym"]
    if kind == "restart":
        km = s["km"]
        km.set_means(s["init"])
        km.run()
        return {"means": km.getMeans(), "sizes": km.getSizes().astype(np.float64), "assignment": s["assignment"]}
    if kind in ("host", "host64"):
        job = bkm.kmeans_host if kind == "host" else bkm.kmeans_host_f64
        means, assignment = job(s["points"], s["means"], n, k, d, s["iters"], lay, laym, torch.cuda.current_device())
        return {"means": means, "assignment": assignment}
    ws, size = s["workspace"].data_ptr(), s["workspace_size"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "encode":
        means = s["means"].data_ptr()
        for points, labels in zip(s["points"], s["labels"]):
            bkm.assign(points.data_ptr(), means, labels.data_ptr(), n, k, d, lay, laym, ws, size, stream=stream)
        return s["labels"]
    points, labels, sizes, out = s["points"][0].data_ptr(), s["labels"].data_ptr(), s["sizes"].data_ptr(), s["out"]
    if kind == "update":
        bkm.update(points, labels, out[0].data_ptr(), sizes, n, k, d, lay, laym, ws, size, stream=stream)
        return {"means": out[0], "sizes": s["sizes"]}
    current = s["means"]
    for t in range(s["iters"]):
        bkm.iterate(points, current.data_ptr(), out[t & 1].data_ptr(), sizes, labels, n, k, d, lay, laym, ws, size, stream=stream)
        current = out[t & 1]
    return {"means": current, "sizes": s["sizes"].double(), "assignment": s["labels"]}


# ---- what a pass cannot do without --------------------------------------------------------------------------

def work(case):
    n, d, k, kind, iters = case["n"], case["d"], case["k"], case["kind"], case["iters"]
    word = 8 if kind == "host64" else 4
    reads = iters * (n * d + k * d) * word                # every iteration (or batch) reads points and means
    if kind == "update":
        return {"bytes": reads + 4 * n + 4 * k, "flops": n * d}
    if kind == "encode":
        return {"bytes": reads + iters * 4 * n, "flops": iters * 2.0 * n * k * d}
    # labels written every iteration, new means and sizes
    return {"bytes": reads + iters * (4 * n + k * d * word + 4 * k), "flops": iters * (2.0 * n * k * d + n * d)}


def tolerance(case):
    """Labels for given means are exact.  Over several iterations the order of the sums moves the means in the
    last bits, a point half-way between two means then falls to the other one, and each such point moves two
    means: four runs of the same job on the same inputs (60 drawn cases) differed by up to 6.5e-3 (2-norm), 0.2
    (one coordinate) and 1.2e-3 of the labels, with sums and counts that are each correct to 32 bits."""
    kind = case["kind"]
    if kind == "encode":
        return "exact"
    if kind == "update":
        return {"rel": 2e-6, "max": 2e-5}
    if kind == "host64":
        return {"rel": 1e-9, "max": 1e-6, "differ": 1e-6}
    return {"rel": 1e-2, "max": 0.4, "differ": 3e-3}
