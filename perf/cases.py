"""Performance cases: what a user of this framework runs, through its public
entry points, over the sizes, data kinds and options that are used in earnest.

A case's ``path`` is one of

* ``host``    -- ``gpu_search``: host queries in, host ids out (synchronous);
* ``search``  -- ``search_device``: the plain search on device buffers;
* ``prec``    -- ``search_device_ex`` with BF16 / FP8 rows and the FP32 re-rank;
* ``learned`` -- ``search_device_ex`` from the tensor-core entry stage's hubs;
* ``hamming`` -- ``search_device`` on sign codes;
* ``knn``     -- ``exact_knn_device``: the exact ground truth;
* ``bithash`` -- ``BitHash.project_device``: sign-random-projection codes;
* ``build``   -- ``build_graph``: the NSW graph of host rows.

Searches run on graphs that the framework's own builder makes, as a user's
program would have them.  The data kinds are the shapes of the reference's
benchmarks: ``int`` (SIFT-shaped integers in [0, 255]), ``angular``
(GloVe-shaped, L2-normalised), ``l1`` (non-negative, L1-normalised) and
``gist`` (GIST-shaped: ``l1`` with a low-rank spread per component).
"""
import importlib
import math

import numpy as np
import torch

song = importlib.import_module("2020_song_ex_b200")


def listed():
    return [
        # one query with the reference's default parameters: an interactive lookup
        dict(name="host_one_query", path="host", data="int", n=100_000, dim=128, nq=1, k=10, ef=50, bf=256, trace=False),
        # a small host batch with the per-query trace, as the reference's GPU bench runs it
        dict(name="host_l1_100d", path="host", data="l1", n=60_000, dim=100, nq=512, k=10, ef=128, bf=256, trace=True),
        # the bench workload: 1M x 128 integers, 10,000 queries, queue and filter for recall@10 >= 0.95
        dict(name="search_int_1m", path="search", data="int", n=1_000_000, dim=128, nq=10_000, k=10, ef=576, bf=512),
        # GloVe-shaped floats at the queue size that reaches recall 0.95
        dict(name="search_angular_200d", path="search", data="angular", n=200_000, dim=200, nq=10_000, k=10, ef=512, bf=512),
        # GIST-shaped floats, a medium batch with k = 100
        dict(name="search_gist_960d", path="search", data="gist", n=40_000, dim=960, nq=1_000, k=100, ef=256, bf=256),
        # the precision form on the same shape: FP8 rows, exact re-rank
        dict(name="prec_fp8_960d", path="prec", data="gist", n=40_000, dim=960, nq=4_000, k=10, ef=384, bf=512, prec="fp8"),
        # the learned form without a model's choice: entry stage, beam 4, two Bloom hashes
        dict(name="learned_int_128d", path="learned", data="int", n=200_000, dim=128, nq=10_000, k=10, ef=64, bf=512),
        # sign codes of 512 bits, reference queue sizes and up
        dict(name="hamming_512b", path="hamming", data="angular", n=200_000, dim=256, bits=512, nq=10_000, k=10, ef=256, bf=256),
        # ground truth of the bench workload
        dict(name="knn_int_1m", path="knn", data="int", n=1_000_000, dim=128, nq=10_000, k=10),
        # ground truth of a small ragged float set, k = 100
        dict(name="knn_l1_ragged", path="knn", data="l1", n=99_991, dim=100, nq=777, k=100),
        # codes of the Hamming workload's base
        dict(name="bithash_290k", path="bithash", data="angular", n=290_000, dim=256, bits=512),
        # the graph of a mid-sized base
        dict(name="build_int_100k", path="build", data="int", n=100_000, dim=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(("host", "search", "search", "prec", "learned", "hamming", "knn", "bithash", "build"))
    if path == "bithash":
        return dict(path=path, data=rng.choice(("angular", "int")), n=_log(rng, 1_000, 400_000),
                    dim=_log(rng, 24, 960), bits=32 * rng.choice((4, 8, 16, 32)))
    if path == "knn":
        data = rng.choice(("int", "l1", "angular"))
        return dict(path=path, data=data, n=_log(rng, 5_000, 500_000), dim=_log(rng, 24, 256),
                    nq=_log(rng, 50, 10_000), k=rng.choice((1, 10, 50, 100)))
    if path == "build":
        data = rng.choice(("int", "angular"))
        return dict(path=path, data=data, n=_log(rng, 5_000, 120_000), dim=_log(rng, 32, 256))
    k = rng.choice((1, 10, 10, 100))
    ef = max(k, _log(rng, 32, 768))
    c = dict(path=path, n=_log(rng, 10_000, 150_000), nq=_log(rng, 1, 10_000), k=k, ef=ef,
             bf=rng.choice((256, 300, 512, 1024)))
    if path == "host":
        c.update(data=rng.choice(("int", "l1", "angular")), dim=_log(rng, 24, 256), nq=_log(rng, 1, 4_000),
                 trace=rng.choice((True, False)))
    elif path == "search":
        c.update(data=rng.choice(("int", "l1", "angular", "gist")), dim=_log(rng, 24, 320))
        if c["data"] == "gist":
            c.update(dim=rng.randrange(400, 1000), n=_log(rng, 10_000, 40_000), nq=_log(rng, 1, 2_000))
    elif path == "prec":
        c.update(data=rng.choice(("gist", "angular")), dim=_log(rng, 100, 960), prec=rng.choice(("bf16", "fp8")),
                 n=_log(rng, 10_000, 60_000), nq=_log(rng, 1, 4_000))
    elif path == "learned":
        c.update(data=rng.choice(("int", "angular")), dim=_log(rng, 32, 200), ef=max(k, _log(rng, 32, 256)))
    else:
        c.update(data="angular", dim=rng.choice((128, 200, 256)), bits=32 * rng.choice((4, 8, 16, 32)))
    # no more gathered values than the GloVe-shaped listed case
    c["nq"] = max(1, min(c["nq"], 10_000 * 512 * 200 // (c["ef"] * c["dim"])))
    return c


# ------------------------------------------------------------------- inputs

def _draw_rows(data, n, dim, pars, g, dev):
    """n rows of one mixture (its parameters in `pars`) as FP32 on the GPU."""
    out = torch.empty((n, dim), device=dev)
    step = 1 << 13 if data == "gist" else 1 << 18
    for s in range(0, n, step):
        m = min(step, n - s)
        c = torch.randint(pars["centres"].shape[0], (m,), generator=g, device=dev)
        x = pars["centres"][c]
        z = torch.randn((m, dim), generator=g, device=dev)
        if data == "int":
            x = (x + 20.0 * z).round_().clamp_(0.0, 255.0)
        elif data == "angular":
            x = x + pars["scales"][c] * z
            x = x / x.norm(dim=1, keepdim=True).clamp_min(1e-12)
        elif data == "l1":
            x = (x + 0.5 * z).clamp_min_(0.0)
            x = x / x.sum(dim=1, keepdim=True).clamp_min(1e-12)
        else:
            w = torch.randn((m, 1, 16), generator=g, device=dev)
            x = x + 0.1 * z + torch.bmm(w, pars["basis"][c]).squeeze(1)
            x = x.clamp_min_(0.0)
            x = x / x.sum(dim=1, keepdim=True).clamp_min(1e-12)
        out[s:s + m] = x
    return out


def _rows(data, n, nq, dim, seed):
    """Base and query rows (device FP32) of one seeded mixture."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(int(seed))
    comp = max(16, min(1024, n // 1000)) if data != "gist" else 64
    pars = {}
    if data == "int":
        pars["centres"] = 255.0 * torch.rand((comp, dim), generator=g, device=dev)
    elif data == "angular":
        pars["centres"] = torch.randn((comp, dim), generator=g, device=dev)
        pars["scales"] = torch.exp(0.5 * torch.randn((comp, dim), generator=g, device=dev) - 0.5)
    else:
        u = torch.rand((2, comp, dim), generator=g, device=dev).clamp_min_(1e-7)
        pars["centres"] = -u.log().sum(dim=0)  # Gamma(2, 1)
        if data == "gist":
            pars["basis"] = (0.7 / 4.0) * torch.randn((comp, 16, dim), generator=g, device=dev)
    base = _draw_rows(data, n, dim, pars, g, dev)
    queries = _draw_rows(data, nq, dim, pars, g, dev) if nq else None
    return base, queries


def _params(case):
    return song.Params(pq_size=max(case.get("ef", 50), case.get("k", 10)), bf_words=case.get("bf", 256),
                       hash_bits=case.get("bits", 256))


def _codes(case, x, seed):
    bh = song.BitHash(case["dim"], seed=int(seed) % 1000, hash_bits=case["bits"])
    R = torch.from_numpy(bh.R).cuda()
    codes = torch.empty((x.shape[0], bh.hash_words), dtype=torch.int32, device="cuda")
    bh.project_device(R, x, x.shape[0], codes)
    return codes


def prepare(case, seed):
    path, n, dim = case["path"], case["n"], case["dim"]
    nq, k = case.get("nq", 0), case.get("k", 0)
    base, q = _rows(case["data"], n, nq, dim, seed)
    st = dict(case=dict(case), path=path)
    if path == "build":
        st["rows"] = base.cpu().numpy()
        return st
    if path == "bithash":
        st["bh"] = song.BitHash(dim, seed=int(seed) % 1000, hash_bits=case["bits"])
        st["R"] = torch.from_numpy(st["bh"].R).cuda()
        st["x"] = base
        st["codes"] = torch.empty((n, case["bits"] // 32), dtype=torch.int32, device="cuda")
        return st
    if path != "host":
        st["ids"] = torch.empty((nq, k), dtype=torch.int32, device="cuda")
    if path in ("knn", "prec", "learned"):
        st["dists"] = torch.empty((nq, k), dtype=torch.float32, device="cuda")
    if path == "knn":
        st["base"], st["q"] = base, q
        return st
    p = _params(case)
    if path == "hamming":
        both = _codes(case, torch.cat((base, q)), seed)
        codes = both[:n].cpu().numpy().view(np.uint32)
        adj = song.build_graph(codes, p, song.KIND_HAMMING)
        st["g"] = song.HashKernelGraph(n, codes, p, adj=adj)
        st["q"] = both[n:].clone()
    else:
        rows = base.cpu().numpy()
        st["g"] = song.KernelGraph(n, dim, rows, p, adj=song.build_graph(rows, p))
        st["q"] = q.cpu().numpy() if path == "host" else q
    g = st["g"]
    g.upload_to_gpu()
    if path == "prec":
        prec = song.PREC_FP8 if case["prec"] == "fp8" else song.PREC_BF16
        song.set_precision(g, prec)
        st["opts"] = song.SearchOpts(precision=prec, rerank=True)
    if path == "learned":
        # the models are trained for a moment only, on a sample of the base: this
        # form takes the entry stage's nearest hubs and never stops early, so it
        # reads no weight
        own = torch.arange(0, n, n // 1024, device="cuda", dtype=torch.int32)
        song.learn(g, base[own.long()].contiguous(), own.numel(), own,
                   song.LearnParams(ef=64, entry_steps=4, stop_steps=4, batch=256,
                                    entry_hubs=min(8192, n // 8)))
        st["opts"] = song.SearchOpts(learned=True, stop_threshold=1.0, beam=4, bloom_hashes=2,
                                     entry=song.ENTRY_NEAREST)
    return st


def run(st):
    c, path = st["case"], st["path"]
    if path == "build":
        return song.build_graph(st["rows"])
    if path == "bithash":
        st["bh"].project_device(st["R"], st["x"], c["n"], st["codes"])
        return st["codes"]
    if path == "knn":
        song.exact_knn_device(st["base"], c["n"], c["dim"], st["q"], c["nq"], c["k"], st["ids"], st["dists"])
        return st["ids"], st["dists"]
    if path == "host":
        tr = song.GpuSearchTrace() if c["trace"] else None
        ids = song.gpu_search(st["g"], st["q"], c["nq"], c["k"], ef_search=c["ef"], trace=tr)
        return (ids, tr.queries) if c["trace"] else ids
    if path in ("search", "hamming"):
        song.search_device(st["g"], st["q"], c["nq"], c["k"], c["ef"], st["ids"])
        return st["ids"]
    song.search_device_ex(st["g"], st["opts"], st["q"], c["nq"], c["k"], c["ef"], st["ids"], st["dists"])
    return st["ids"], st["dists"]


def work(case):
    """Bytes and operations of one pass.  A graph search expands about 1.2
    nodes and evaluates about 4 distances per queue slot (measured on the
    integer mixtures); it cannot do without the rows and adjacency rows of
    those.  Integer rows are counted as bytes, compressed rows at their width."""
    path, n, dim = case["path"], case["n"], case["dim"]
    nq, k = case.get("nq", 0), case.get("k", 0)
    if path == "knn":
        return {"bytes": 4.0 * (n * dim + nq * dim + 2 * nq * k), "flops": 2.0 * n * nq * dim}
    if path == "bithash":
        return {"bytes": 4.0 * n * dim + n * case["bits"] / 8 + 4.0 * dim * case["bits"],
                "flops": 2.0 * n * dim * case["bits"]}
    width = dim if case["data"] == "int" else 4 * dim
    if path == "prec":
        width = dim * (1 if case["prec"] == "fp8" else 2)
    if path == "hamming":
        width = case["bits"] / 8
    if path == "build":  # one search with EF_CONSTRUCTION = 150 per node, rows in, graph out
        return {"bytes": n * (600.0 * width + 180.0 * 128 + 128.0 + 4.0 * dim), "flops": 3.0 * n * 600 * dim}
    ef = case["ef"]
    per = 4.0 * ef * width + 1.2 * ef * 128 + 4.0 * dim + 4.0 * k
    flops = 12.0 * ef * dim
    if path == "prec":
        per += 4.0 * dim * ef
        flops += 3.0 * ef * dim
    if path == "learned":
        flops += 2.0 * min(8192, n // 8) * dim
    return {"bytes": nq * per, "flops": nq * flops}


def exact(case, seed):
    """Exact kNN distances in 64 bits.  Ids of all paths, codes and graphs are
    whole numbers; a graph search's distances belong to the ids that it found
    on its own graph and have no value apart from it."""
    if case["path"] != "knn":
        return None
    base, q = _rows(case["data"], case["n"], case["nq"], case["dim"], seed)
    best = torch.full((case["nq"], case["k"]), math.inf, dtype=torch.float64, device=q.device)
    q = q.double()
    for s in range(0, case["n"], 1 << 15):
        b = base[s:s + (1 << 15)].double()
        for r in range(0, case["nq"], 4096):
            d = (q[r:r + 4096].square().sum(1, keepdim=True) - 2.0 * (q[r:r + 4096] @ b.T)) + b.square().sum(1)
            both = torch.cat((best[r:r + 4096], d), dim=1)
            best[r:r + 4096] = both.topk(case["k"], dim=1, largest=False, sorted=True).values
    return None, best
