"""The work that users of this engine have it do, as timed cases.

A case names an entry point (its "kind"), sizes, element type and options.
`prepare` makes what a program holds before the call (rows on the device or in
host memory, centroids, a handle, a fitted proposer), `run` is one call through
the public API, `work` what the call cannot do without, and `exact` the same
results in 64-bit arithmetic by plain torch.

Rows are generated on the GPU from the seed, with the distributions of the
engine's own workloads (datasets.py): Gaussian blobs, low-rank unit-norm
embeddings, int8 codes of such embeddings, byte features, Student-t mixtures.
"""
import importlib
import math

import numpy as np
import torch

emb = importlib.import_module("e-means_b200")

DEV = "cuda"


def listed():
    return [
        # A handful of new rows labelled by the default assigner from a numpy array: an
        # online service's request, all latency and launches.
        {"name": "assign_request", "kind": "assign", "data": "blobs", "dtype": "f32", "precision": "fp32", "bits": 0,
         "where": "numpy", "bias": False, "m": 100, "d": 96, "k": 1024},
        # A ragged mini-batch under a balance bias, d and k multiples of nothing: what a
        # training loop of one's own around the Assigner calls.
        {"name": "assign_ragged_bias", "kind": "assign", "data": "blobs", "dtype": "f32", "precision": "bf16",
         "bits": 0, "where": "device", "bias": True, "m": 20011, "d": 100, "k": 1031},
        # The exact closing pass over a trained corpus with the default (FP32) search.
        {"name": "assign_fp32", "kind": "assign", "data": "blobs", "dtype": "f32", "precision": "fp32", "bits": 0,
         "where": "device", "bias": False, "m": 200000, "d": 96, "k": 1024},
        # The headline: a corpus of embeddings against a large codebook.
        {"name": "assign_embeddings", "kind": "assign", "data": "embeddings", "dtype": "f32", "precision": "bf16x1",
         "bits": 0, "where": "device", "bias": False, "m": 1000000, "d": 128, "k": 16384},
        # A chunk of a corpus that lives in (pinned) host memory, labels and distances back to the host.
        {"name": "assign_host", "kind": "assign", "data": "embeddings", "dtype": "f32", "precision": "bf16x1",
         "bits": 0, "where": "pinned", "bias": False, "m": 262144, "d": 128, "k": 4096},
        # Quantised rows against int8 centroids (the integer assigner).
        {"name": "assign_int8", "kind": "assign", "data": "embeddings", "dtype": "i8", "precision": "fp32", "bits": 8,
         "where": "device", "bias": False, "m": 500000, "d": 512, "k": 4096},
        # Training, the README's own size: many small batches.
        {"name": "train_blobs", "kind": "train", "data": "blobs", "precision": "bf16", "n": 200000, "d": 96, "k": 1024,
         "epochs": 5.0},
        # Training a larger codebook on embeddings: fewer, larger batches.
        {"name": "train_embeddings", "kind": "train", "data": "embeddings", "precision": "bf16x1", "n": 500000,
         "d": 128, "k": 4096, "epochs": 2.0},
        # Refining the lists of an inverted file: many uneven instances at once.
        {"name": "train_lists", "kind": "lists", "lists": 48, "median": 20000, "d": 64, "epochs": 5.0},
        # Calibrating the int8 quantizer on resident rows.
        {"name": "quantizer_fit", "kind": "fit", "data": "embeddings", "n": 500000, "d": 512, "quantile": 1.0},
        # The cluster report of a large clustering, from the resident results of its assign.
        {"name": "report", "kind": "report", "data": "embeddings", "n": 1000000, "d": 128, "k": 16384},
        # A very large codebook searched through the learned proposer.
        {"name": "assign_proposed", "kind": "proposed", "n": 1000000, "d": 96, "k": 65536, "steps": 500},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges: odd sizes, every element type and option."""
    kind = rng.choice(["assign"] * 6 + ["train"] * 2 + ["lists", "fit", "report", "proposed"])
    if kind == "assign":
        dtype, bits = rng.choice([("f32", 0), ("f32", 0), ("f32", 0), ("u8", 0), ("i8", 0), ("i8", 8)])
        precision = rng.choice(["fp32", "bf16", "bf16x1"])
        where = rng.choice(["numpy", "device", "device", "pinned"])
        d = _log(rng, 16, 512 if bits == 8 else 256)
        if rng.random() < 0.5:
            d = (d + 15) // 16 * 16
        k = _log(rng, 200, 16384 if precision != "fp32" and bits == 0 else 4096)
        most = {"fp32": 4e10, "bf16": 1.4e12, "bf16x1": 4e12}[precision] if bits == 0 else 2e12
        m = min(_log(rng, 100, 1000000), max(100, int(most / (2.0 * d * k))))
        if where != "device":
            m = min(m, 32_000_000 // d)
        return {"kind": kind, "data": rng.choice(["blobs", "embeddings"]), "dtype": dtype, "precision": precision,
                "bits": bits, "where": where, "bias": rng.random() < 0.25, "m": m, "d": d, "k": k}
    if kind == "train":
        k = _log(rng, 64, 4096)
        return {"kind": kind, "data": rng.choice(["blobs", "embeddings"]),
                "precision": rng.choice(["fp32", "bf16", "bf16x1"]), "n": max(10 * k, _log(rng, 20000, 500000)),
                "d": 4 * _log(rng, 5, 32), "k": k, "epochs": float(rng.choice([1, 2, 2.5, 3]))}
    if kind == "lists":
        return {"kind": kind, "lists": rng.randint(4, 48), "median": _log(rng, 3000, 20000),
                "d": 4 * _log(rng, 2, 24), "epochs": float(rng.choice([2, 3, 5]))}
    if kind == "fit":
        d = _log(rng, 32, 512)
        return {"kind": kind, "data": rng.choice(["blobs", "embeddings"]), "n": _log(rng, 10000, 250_000_000 // 512),
                "d": d, "quantile": rng.choice([1.0, 0.9999])}
    if kind == "report":
        k = _log(rng, 256, 16384)
        return {"kind": kind, "data": rng.choice(["blobs", "embeddings"]), "n": max(20 * k, _log(rng, 20000, 1000000)),
                "d": _log(rng, 16, 128), "k": k}
    return {"kind": kind, "n": _log(rng, 100000, 1000000), "d": rng.choice([64, 96]), "k": 1 << rng.randint(14, 16),
            "steps": 300}


# ---- inputs ------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32)


def _rows(data, n, d, g):
    if data == "blobs":  # 4096 centres N(0, 4^2), unit spread
        centres = _randn(g, 4096, d) * 4.0
        x = centres[torch.randint(0, 4096, (n,), generator=g, device=DEV)]
        return x.add_(_randn(g, n, d))
    if data == "heavy":  # Student-t (nu = 3) latents around 8192 offsets through a random map
        w = _randn(g, 32, d)
        offsets = _randn(g, 8192, 32) * 3.0
        z = _randn(g, n, 32)
        chi = _randn(g, n, 32, 3).square_().sum(2).div_(3.0)
        z = z / chi.sqrt_() + offsets[torch.randint(0, 8192, (n,), generator=g, device=DEV)]
        return _matmul(z, w)
    latent = 64 if d > 256 else 32  # embeddings: low-rank latent plus noise, unit norm
    w = _randn(g, latent, d)
    x = _matmul(_randn(g, n, latent), w)
    x.add_(_randn(g, n, d), alpha=0.1)
    return x.div_(x.square().sum(1, keepdim=True).sqrt_())


def _matmul(a, b):
    """f32 matrix product, one rank at a time: the same bits whatever library mode is set."""
    out = a[:, :1] * b[:1]
    for i in range(1, a.shape[1]):
        out.addcmul_(a[:, i:i + 1], b[i:i + 1])
    return out


def _centroids(x, k):
    """Centroids as an earlier training left them: two Lloyd steps of plain torch over
    at most 64 rows a centroid (sums in 64-bit integers: the same bits every time)."""
    n = min(x.shape[0], 64 * k)
    xs = x[:n]
    c = xs[torch.arange(k, device=DEV) * (n // k)].clone() if n >= k else xs[torch.arange(k, device=DEV) % n] * 1.01
    scale = 2.0 ** 24
    for _ in range(2):
        nrm = c.square().sum(1)
        ch = c.to(torch.bfloat16).t().contiguous()
        lab = torch.cat([(nrm - 2.0 * (xs[r:r + 65536].to(torch.bfloat16) @ ch).float()).argmin(1)
                         for r in range(0, n, 65536)])
        sums = torch.zeros(k, x.shape[1], dtype=torch.int64, device=DEV)
        sums.index_add_(0, lab, (xs * scale).round_().to(torch.int64))
        cnt = torch.zeros(k, dtype=torch.int64, device=DEV).index_add_(0, lab, torch.ones_like(lab))
        mean = (sums.double() / (scale * cnt.clamp(min=1).double()[:, None])).float()
        c = torch.where(cnt[:, None] > 0, mean, c)
    return c


def _typed(x, dtype):
    """f32 rows, or their int8 / byte codes (faiss calibration: one power-of-two scale)."""
    if dtype == "f32":
        return x
    if dtype == "u8":
        lo, hi = x.min(), x.max()
        return ((x - lo) * (255.0 / (hi - lo))).round_().to(torch.uint8)
    peak = x.abs().max()
    scale = torch.exp2(torch.floor(torch.log2(112.0 / peak)))
    return (x * scale).round_().clamp_(-128, 127).to(torch.int8)


def _list_sizes(case):
    rng = np.random.default_rng(case["median"])
    n = np.clip(np.round(rng.lognormal(np.log(case["median"]), 1.0, case["lists"])), 2000, 200000).astype(np.int64)
    return n, np.maximum(16, n // 256)


def _assign_inputs(case, seed):
    g = _gen(seed)
    x = _typed(_rows(case["data"], case["m"] if case["m"] >= 4 * case["k"] else 4 * case["k"], case["d"], g),
               case["dtype"])
    c = _centroids(x.float(), case["k"])
    bias = None
    if case["bias"]:  # a balance penalty: a few percent of the typical distance, more for some clusters
        typical = (x[:4096].float() - c[torch.arange(min(4096, x.shape[0]), device=DEV) % case["k"]]).square().sum(1).mean()
        bias = torch.rand(case["k"], generator=g, device=DEV) * (0.05 * typical)
    return x[:case["m"]].contiguous(), c, bias


def _heavy_inputs(case, seed):
    x = _rows("heavy", case["n"], case["d"], _gen(seed))
    return x, _centroids(x, case["k"])


# ---- state and run -----------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "assign":
        x, c, bias = _assign_inputs(case, seed)
        a = emb.B200Assigner(0, precision=case["precision"], centroid_bits=case["bits"])
        a.set_centroids(c.cpu().numpy())
        if bias is not None:
            a.set_bias(bias.cpu().numpy())
        state = {"kind": kind, "where": case["where"], "a": a, "m": case["m"],
                 "dtype": {"f32": emb.EMB200_F32, "i8": emb.EMB200_I8, "u8": emb.EMB200_U8}[case["dtype"]]}
        if case["where"] == "numpy":
            state["x"] = x.cpu().numpy()
        else:
            dev = DEV if case["where"] == "device" else "cpu"
            pin = case["where"] == "pinned"
            state["x"] = x if dev == DEV else x.cpu().pin_memory()
            state["labels"] = torch.empty(case["m"], dtype=torch.int32, device=dev, pin_memory=pin)
            state["dist"] = torch.empty(case["m"], dtype=torch.float32, device=dev, pin_memory=pin)
        return state
    if kind == "train":
        x = _rows(case["data"], case["n"], case["d"], _gen(seed))
        a = emb.B200Assigner(0, precision=case["precision"])
        a.load_rows(x.cpu().numpy())
        return {"kind": kind, "a": a, "k": case["k"], "cfg": emb.Config(nepochs=case["epochs"])}
    if kind == "lists":
        sizes, ks = _list_sizes(case)
        g = _gen(seed)
        parts = []
        for n in sizes:  # a list: its own centre, 64 sub-clusters around it, spread 0.5
            subs = _randn(g, 1, case["d"]) * 4.0 + _randn(g, 64, case["d"])
            parts.append(subs[torch.randint(0, 64, (int(n),), generator=g, device=DEV)]
                         + _randn(g, int(n), case["d"]) * 0.5)
        a = emb.B200Assigner(0)
        a.load_rows(torch.cat(parts).cpu().numpy())
        starts = np.concatenate([[0], np.cumsum(sizes)])
        inst = [(int(starts[i]), int(sizes[i]), int(ks[i])) for i in range(case["lists"])]
        return {"kind": kind, "a": a, "inst": inst, "cfg": emb.Config(nepochs=case["epochs"])}
    if kind == "fit":
        a = emb.B200Assigner(0)
        a.load_rows(_rows(case["data"], case["n"], case["d"], _gen(seed)).cpu().numpy())
        cal = emb.Calibration.faiss() if case["quantile"] == 1.0 else emb.Calibration.clipped(case["quantile"])
        return {"kind": kind, "a": a, "cal": cal}
    if kind == "report":
        x = _rows(case["data"], case["n"], case["d"], _gen(seed))
        a = emb.B200Assigner(0, precision="bf16x1")
        a.set_centroids(_centroids(x, case["k"]).cpu().numpy())
        a.load_rows(x.cpu().numpy())
        a.assign_resident(want_host=False)
        return {"kind": kind, "a": a}
    x, c = _heavy_inputs(case, seed)
    a = emb.B200Assigner(0, precision="bf16x1")
    a.load_rows(x.cpu().numpy())
    a.set_centroids(c.cpu().numpy())
    labels, _ = a.assign_resident()
    a.proposer_init(groups=256, hidden=512, top=32, seed=7)
    a.proposer_train(labels, case["steps"])
    a.proposer_set("mlp", 32, 0.99, 0.9995)
    return {"kind": kind, "a": a, "x": x, "labels": torch.empty(case["n"], dtype=torch.int32, device=DEV),
            "dist": torch.empty(case["n"], dtype=torch.float32, device=DEV)}


def _padded(values, n):
    """As many entries as there are clusters, -1 past the last."""
    return np.concatenate([np.asarray(values, np.int64), np.full(n - len(values), -1, np.int64)])


def run(state):
    kind, a = state["kind"], state["a"]
    if kind == "assign":
        if state["where"] == "numpy":
            labels, dist = a.assign(state["x"])
            return {"labels": labels, "dist": dist}
        call = a.assign_device if state["where"] == "device" else a.assign_host_ptr
        call(state["x"].data_ptr(), state["dtype"], state["m"], state["labels"].data_ptr(), state["dist"].data_ptr())
        return {"labels": state["labels"], "dist": state["dist"]}
    if kind == "train":
        out = a.train_resident(state["k"], state["cfg"])
        return {"centroids": out.centroids, "labels": out.labels, "objective": out.objective, "splits": out.n_splits}
    if kind == "lists":
        outs = a.train_batched(state["inst"], state["cfg"])
        return {"centroids": np.concatenate([o.centroids.reshape(-1) for o in outs]),
                "labels": np.concatenate([o.labels for o in outs]),
                "objective": np.concatenate([o.objective for o in outs]),
                "splits": np.array([o.n_splits for o in outs])}
    if kind == "fit":
        q = emb.Int8Quantizer.fit_resident(a, state["cal"])
        return {"shift": q.shift, "scale": float(q.scale)}
    if kind == "report":
        r = emb.report_resident(a)
        out = {f: r.clusters[f].copy() for f in emb.CLUSTER_STATS.names}
        out.update(local_z=r.local_z, global_z=r.global_z,
                   medians=np.array([r.median_dist, r.median_rms, r.median_nearest_dist], np.float32),
                   leaders=_padded([f.leader for f in r.families], a.k),
                   sizes=_padded([f.size for f in r.families], a.k),
                   members=_padded(np.concatenate([f.members for f in r.families]), a.k))
        return out
    a.assign_proposed_device(state["x"].data_ptr(), state["x"].shape[0], state["labels"].data_ptr(),
                             state["dist"].data_ptr())
    return {"labels": state["labels"], "dist": state["dist"]}


def work(case):
    kind = case["kind"]
    if kind == "assign":
        m, d, k = case["m"], case["d"], case["k"]
        return {"bytes": m * d * (4 if case["dtype"] == "f32" else 1) + 4 * k * d + 8 * m, "flops": 2.0 * m * d * k}
    if kind == "train":
        rows = case["n"] * case["epochs"]
        return {"bytes": 4.0 * rows * case["d"] + 8.0 * rows + 8.0 * case["k"] * case["d"],
                "flops": 2.0 * rows * case["d"] * case["k"]}
    if kind == "lists":
        n, k = _list_sizes(case)
        rows = float(n.sum()) * case["epochs"]
        return {"bytes": 4.0 * rows * case["d"] + 8.0 * rows,
                "flops": 2.0 * case["epochs"] * case["d"] * float((n * k).sum())}
    if kind == "fit":  # the rows are read for the mean, then for the peak around it
        return {"bytes": 8.0 * case["n"] * case["d"], "flops": 3.0 * case["n"] * case["d"]}
    if kind == "report":  # every pair of centroids once; rows' labels and distances in, two scores out
        return {"bytes": 16.0 * case["n"] + 4.0 * case["k"] * case["d"], "flops": 1.5 * case["k"] ** 2 * case["d"]}
    d, hidden, groups = case["d"], 512, 256  # the network, then an eighth of the groups a row
    return {"bytes": 4.0 * case["n"] * d + 8.0 * case["n"] + 4.0 * case["k"] * d,
            "flops": 2.0 * case["n"] * (d * hidden + hidden * hidden + hidden * groups + d * case["k"] / 8)}


# ---- 64-bit results ------------------------------------------------------------

def _search64(x, c, bias=None):
    """(nearest centroid, its squared distance without the bias) in float64."""
    c = c.double()
    nrm = c.square().sum(1)
    off = nrm if bias is None else nrm + bias.double()
    step = max(1, (1 << 28) // c.shape[0])
    labels, dist = [], []
    for r in range(0, x.shape[0], step):
        xs = x[r:r + step].double()
        best, j = (off - 2.0 * (xs @ c.t())).min(1)
        labels.append(j)
        dist.append((best + xs.square().sum(1)).clamp_(min=0))
    return torch.cat(labels), torch.cat(dist)


def exact(case, seed):
    kind = case["kind"]
    if kind == "assign":
        x, c, bias = _assign_inputs(case, seed)
        if case["bits"] == 8:  # the integer assigner's centroids: rounded half away from zero
            c = (torch.sign(c) * torch.floor(c.abs().double() + 0.5)).clamp(-128, 127)
            bias = None if bias is None else torch.floor(bias.double() + 0.5)
        return {"labels": None, "dist": _search64(x, c, bias)[1]}
    if kind == "fit":
        x = _rows(case["data"], case["n"], case["d"], _gen(seed))
        total, peaks = torch.zeros(case["d"], dtype=torch.float64, device=DEV), []
        for r in range(0, case["n"], 65536):
            total += x[r:r + 65536].double().sum(0)
        shift = total / case["n"]
        for r in range(0, case["n"], 65536):
            mag = (x[r:r + 65536].double() - shift).abs_().reshape(-1)
            peaks.append(mag.max()[None] if case["quantile"] == 1.0 else mag.float())
        if case["quantile"] == 1.0:
            return {"shift": shift, "scale": float(2.0 ** math.floor(math.log2(112.0 / float(torch.cat(peaks).max()))))}
        mags = torch.cat(peaks).sort()[0]
        return {"shift": shift, "scale": 127.0 / float(mags[round((mags.numel() - 1) * case["quantile"])])}
    if kind == "report":
        return _report64(case, seed)
    return None


def _report64(case, seed):
    x = _rows(case["data"], case["n"], case["d"], _gen(seed))
    c = _centroids(x, case["k"])
    labels, sq = _search64(x, c)
    labels, dist, k = labels.cpu().numpy(), sq.sqrt().cpu().numpy(), case["k"]

    def by_cluster(v):
        order = np.lexsort((v, labels))
        return v[order], np.searchsorted(labels[order], np.arange(k + 1))

    def at(v, s, q):
        n = np.diff(s)
        return np.where(n > 0, v[np.minimum(s[:-1] + np.floor(np.maximum(n - 1, 0) * q + 0.5).astype(np.int64),
                                            v.size - 1)], 0.0)

    def median(v):
        return np.sort(v)[int(math.floor((v.size - 1) * 0.5 + 0.5))]

    v, s = by_cluster(dist)
    size = np.diff(s)
    live = size > 0
    total = np.concatenate([[0.0], np.cumsum(v * v)])
    med = at(v, s, 0.5)
    mad = at(*by_cluster(np.abs(dist - med[labels])), 0.5)
    near = np.full(k, np.inf)
    c64, alive = c.double(), torch.from_numpy(live).to(DEV)
    nrm = c64.square().sum(1)
    for r in range(0, k, 2048):
        e = (nrm[r:r + 2048, None] + nrm[None] - 2.0 * (c64[r:r + 2048] @ c64.t())).clamp_(min=0)
        e[:, ~alive] = math.inf
        e[torch.arange(e.shape[0], device=DEV), torch.arange(r, r + e.shape[0], device=DEV)] = math.inf
        near[r:r + 2048] = e.min(1)[0].sqrt().cpu().numpy()
    g_med = median(dist)
    g_scale = 1.4826 * median(np.abs(dist - g_med))
    gz = (dist - g_med) / g_scale
    own = mad[labels] > 0
    small = (size[labels] < 30) | ~own
    lz = np.where(small, gz, (dist - med[labels]) / np.where(own, 1.4826 * mad[labels], 1.0))
    rms = np.sqrt(np.diff(total[s]) / np.maximum(size, 1))
    return {"rms": rms, "median": med, "mad": mad, "p90": at(v, s, 0.9), "p99": at(v, s, 0.99), "max": at(v, s, 1.0),
            "nearest_dist": near, "local_z": lz, "global_z": gz,
            "medians": np.array([g_med, median(rms[live]), median(near[live])])}
