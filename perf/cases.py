"""The work that users of this framework have it do, as timed cases: batched graph search (with and without
the exact rerank), multiprobe search, search on sign-bit codes, bulk index build, incremental insertion,
encoding and exact ground truth, all through the public calls of ``cphnsw_b200.CPHNSWIndex``.

Data are the mixtures of ``cphnsw_b200.synthetic`` drawn on the GPU: unit vectors of a Gaussian mixture with
about 1,000 points per cluster (sigma 0.3), non-negative where the dimension is that of image descriptors
(960), one entry node to score for every 122 base vectors (8,192 at 1M) of which the best 32 seed the walk.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sparse-text-kmeans_b200"))
import cphnsw_b200 as cp  # noqa: E402

EF_CONSTRUCTION = 200
K_ENTRY = 32


def listed():
    return [
        # one user's query at a time, as a service answers it (host arrays in and out): latency
        dict(name="search_one", kind="search", n=100_000, dim=128, K=32, M=32, nq=1, k=10, ef=100, rerank_k=500, io="host"),
        # a small ragged batch of plain searches (no rerank) at the wide end of the ef sweep, d=96 base vectors
        dict(name="search_61", kind="search", n=300_007, dim=96, K=32, M=32, nq=61, k=10, ef=400, rerank_k=0, io="host"),
        # the headline: 10,000 queries against 1M x 128, queries and results in device memory
        dict(name="search_10k", kind="search", n=1_000_000, dim=128, K=32, M=32, nq=10_000, k=10, ef=100, rerank_k=500, io="dev"),
        # image descriptors, d=960 padded to 1024, two-byte components, wide beam and rerank
        dict(name="search_960", kind="search", n=100_003, dim=960, K=32, M=32, nq=2_000, k=10, ef=200, rerank_k=1000, io="host"),
        # the unified index's sign-bit codes: walk under the Hamming distance, rerank of the beam
        dict(name="search_binary", kind="binary", n=200_000, dim=128, K=64, M=32, nq=5_000, k=10, ef=200, rerank_k=200, io="host"),
        # a batch of 1,024 queries, four probe codes each
        dict(name="multiprobe_1k", kind="multiprobe", n=200_000, dim=128, K=32, M=32, nq=1_024, k=10, ef=100, probes=4),
        # an index that grows: 1,000 new vectors join 100,000
        dict(name="insert_1k", kind="insert", n=100_000, dim=128, K=32, M=32, add=1_000),
        # a small index built from host vectors from nothing, handle creation included, links read back
        dict(name="build_20k", kind="build", n=20_011, dim=96, K=32, M=32, io="host"),
        # the bulk build's stages on device memory: encode, kNN graph, pruning
        dict(name="build_500k", kind="build", n=500_000, dim=128, K=32, M=32, io="dev"),
        # the same on d=960 descriptors with two-byte components
        dict(name="build_960", kind="build", n=100_003, dim=960, K=32, M=32, io="dev"),
        # encoding alone, the size of a whole base set
        dict(name="encode_1m", kind="encode", n=1_000_000, dim=128, K=32),
        # exact ground truth that recall is measured against
        dict(name="exact_2k", kind="exact", n=500_000, dim=128, nq=2_000, k=10),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["search", "search", "search", "binary", "multiprobe", "insert", "build", "build", "encode", "exact"])
    wide = kind in ("search", "build", "encode", "binary") and rng.random() < 0.3  # padded dimensions above 128
    dim = rng.choice([200, 256, 300, 384, 512, 768, 960, 1000, 1024]) if wide else rng.choice([32, 50, 64, 96, 100, 120, 128, 128, 128])
    K = 32 if wide else rng.choice([16, 32, 32, 32, 64])
    M = rng.choice([16, 24, 32, 32])
    n = spread(20_000, 100_000 if wide else 300_000)
    io = rng.choice(["host", "dev"])
    if kind == "search":
        ef = spread(50, 400)
        rerank_k = rng.choice([0, ef, spread(ef, 1000)])
        return dict(kind=kind, n=n, dim=dim, K=K, M=M, nq=spread(1, 2_000 if wide else 10_000), k=rng.choice([1, 10, 10, 32]), ef=ef,
                    rerank_k=rerank_k, io=io)
    if kind == "binary":
        ef = spread(50, 400)
        return dict(kind=kind, n=n, dim=dim, K=rng.choice([32, 64, 64]), M=M, nq=spread(1, 10_000), k=10, ef=ef,
                    rerank_k=rng.choice([0, ef]), io=io)
    if kind == "multiprobe":
        return dict(kind=kind, n=n, dim=dim, K=K, M=M, nq=spread(1, 2_000), k=10, ef=spread(50, 400), probes=rng.choice([1, 4, 16]))
    if kind == "insert":
        return dict(kind=kind, n=n, dim=dim, K=K, M=M, add=spread(1, 10_000))
    if kind == "build":
        return dict(kind=kind, n=spread(5_000, 100_000 if wide else 300_000), dim=dim, K=K, M=M, io=io)
    if kind == "encode":
        return dict(kind=kind, n=spread(100, 200_000 if wide else 1_000_000), dim=dim, K=K)
    return dict(kind=kind, n=n, dim=dim, nq=spread(10, 2_000), k=rng.choice([1, 10, 100]))


def padded(dim):
    return 1 << (dim - 1).bit_length()


def component_bytes(case):
    return 2 if padded(case["dim"]) > 128 and case["kind"] != "binary" else 1


class Mixture:
    """Unit vectors of a mixture with about 1,000 points per cluster, on the GPU; non-negative above 512 dimensions."""

    def __init__(self, n, dim, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.positive = dim > 512
        self.centres = torch.randn((max(1, n // 1000), dim), generator=self.gen, device="cuda")
        if self.positive:
            self.centres.abs_()

    def draw(self, m):
        dim = self.centres.shape[1]
        out = torch.empty((m, dim), device="cuda")
        for i in range(0, m, 1 << 18):
            j = min(m, i + (1 << 18))
            a = torch.randint(0, self.centres.shape[0], (j - i,), generator=self.gen, device="cuda")
            x = torch.randn((j - i, dim), generator=self.gen, device="cuda").mul_(0.3).add_(self.centres[a])
            if self.positive:
                x.abs_()
            out[i:j] = x / x.norm(dim=1, keepdim=True).clamp_min_(1e-10)
        return out


def new_index(case):
    if case["kind"] == "binary":
        idx = cp.CPHNSWIndex.binary(case["dim"], M=case["M"], ef_construction=EF_CONSTRUCTION, K=case["K"])
    else:
        idx = cp.CPHNSWIndex(case["dim"], M=case.get("M", 32), ef_construction=EF_CONSTRUCTION, K=case.get("K", 32),
                             component_bytes=component_bytes(case))
    idx.set_param("k_entry", K_ENTRY)
    idx.set_param("entry_scan", entry_scan(case))
    return idx


def entry_scan(case):
    return max(K_ENTRY, case["n"] // 122)


def stage_buffers(case):
    """Device outputs of the build stages: codes, kNN candidates, adjacency."""
    n, M = case["n"], case["M"]
    codes = torch.empty((n, case["K"]), dtype=torch.uint8 if component_bytes(case) == 1 else torch.int16, device="cuda")
    cand = torch.empty((n, min(2 * M, 64)), dtype=torch.int32, device="cuda")
    adj = torch.empty((n, M), dtype=torch.int32, device="cuda")
    return codes, cand, adj


def build_stages(idx, x, codes, cand, adj):
    n, k, M = cand.shape[0], cand.shape[1], adj.shape[1]
    st = torch.cuda.current_stream().cuda_stream
    idx.encode_dev(x.data_ptr(), n, codes.data_ptr(), stream=st)
    idx.knn_graph_dev(codes.data_ptr(), n, k, 0, n, cand.data_ptr(), stream=st)
    idx.select_neighbors_dev(codes.data_ptr(), n, cand.data_ptr(), k, 0, n, M, True, adj.data_ptr(), stream=st)


def prepare(case, seed):
    kind, n, dim = case["kind"], case["n"], case["dim"]
    mix = Mixture(n, dim, seed)
    x = mix.draw(n)
    s = dict(case=case)
    if kind == "exact":
        s["idx"] = new_index(case)
        s["base"], s["q"] = x, mix.draw(case["nq"])
    elif kind == "encode":
        s["idx"] = new_index(case)
        s["base"] = x
        s["codes"] = torch.empty((n, case["K"]), dtype=torch.uint8 if component_bytes(case) == 1 else torch.int16, device="cuda")
    elif kind == "build":
        if case["io"] == "host":
            s["base"] = x.cpu().numpy()
        else:
            s["idx"] = new_index(case)
            s["base"], s["stages"] = x, stage_buffers(case)
    else:
        idx = s["idx"] = new_index(case)
        codes, cand, adj = stage_buffers(case)
        build_stages(idx, x, codes, cand, adj)
        if kind == "insert":
            s["graph"] = (x, codes, adj)
            s["new"] = mix.draw(case["add"]).cpu().numpy()
            return s
        idx.install_dev(x.data_ptr(), codes.data_ptr(), adj.data_ptr(), n, stream=torch.cuda.current_stream().cuda_stream)
        s["q"] = mix.draw(case["nq"])
        if case.get("io", "host") == "host":
            s["q"] = s["q"].cpu().numpy()
    if "nq" in case and (kind == "exact" or case.get("io") == "dev"):
        s["ids"] = torch.empty((case["nq"], case["k"]), dtype=torch.int32, device="cuda")
        s["dist"] = torch.empty((case["nq"], case["k"]), dtype=torch.float32, device="cuda")
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    st = torch.cuda.current_stream().cuda_stream
    if kind in ("search", "binary"):
        if case["io"] == "dev":
            s["idx"].search_dev(s["q"].data_ptr(), case["nq"], case["k"], case["ef"], case["rerank_k"], s["ids"].data_ptr(),
                                s["dist"].data_ptr(), stream=st)
            return s["ids"], s["dist"]
        if case["rerank_k"]:
            return s["idx"].search_and_rerank_batch(s["q"], case["k"], case["ef"], case["rerank_k"])
        return s["idx"].search_batch(s["q"], case["k"], case["ef"])
    if kind == "multiprobe":
        return s["idx"].search_multiprobe_batch(s["q"], case["k"], case["ef"], case["probes"])
    if kind == "insert":
        # every pass starts from the same graph: it is installed again, then the new vectors join it
        x, codes, adj = s["graph"]
        s["idx"].install_dev(x.data_ptr(), codes.data_ptr(), adj.data_ptr(), case["n"], stream=st)
        s["idx"].add_batch(s["new"])
        return s["idx"].codes(), s["idx"].adjacency()
    if kind == "build":
        if case["io"] == "host":
            idx = new_index(case)
            idx.add_batch_parallel(s["base"])
            out = idx.codes(), idx.adjacency()
            idx.close()
            return out
        build_stages(s["idx"], s["base"], *s["stages"])
        return s["stages"]
    if kind == "encode":
        s["idx"].encode_dev(s["base"].data_ptr(), case["n"], s["codes"].data_ptr(), stream=st)
        return s["codes"]
    s["idx"].exact_search_dev(s["base"].data_ptr(), case["n"], s["q"].data_ptr(), case["nq"], case["k"], s["ids"].data_ptr(),
                              s["dist"].data_ptr(), stream=st)
    return s["ids"], s["dist"]


def work(case):
    """Bytes: inputs read once and outputs written once.  Operations: the additions of the transforms, one compare and
    one add per component of a code distance (each unordered pair once in a graph build), one add per component of a
    score, a multiply and an add per coordinate of a dot product."""
    kind, n, dim = case["kind"], case["n"], case["dim"]
    K, M = case.get("K", 32), case.get("M", 32)
    P, row = padded(dim), K * component_bytes(case)
    stored = K / 8 if kind == "binary" else row  # bytes of a node's code that the walk reads
    transform = K * 3 * P * math.log2(max(2, P))
    if kind == "encode":
        return {"bytes": n * (dim * 4 + row), "flops": n * transform}
    if kind == "exact":
        return {"bytes": (n + case["nq"]) * dim * 4 + case["nq"] * case["k"] * 8, "flops": 2.0 * n * case["nq"] * dim}
    if kind == "build":
        k = min(2 * M, 64)
        return {"bytes": n * (dim * 4 + row + (k if case["io"] == "dev" else 0) * 4 + M * 4),
                "flops": n * transform + n * (n - 1.0) * K + n * k * M * K}
    if kind == "insert":
        a = case["add"]
        beam = max(EF_CONSTRUCTION, 64)
        return {"bytes": 2 * n * (dim * 4 + row + M * 4) + a * (dim * 4 + row + M * 4) + (n + a) * (row + M * 4),
                "flops": a * (transform + 2.0 * K * (entry_scan(case) + beam) + 64 * M * K)}
    # searches: every walk expands the members of its final beam, reads their links and codes, and scores the entry nodes
    walks = case["nq"] * case.get("probes", 1)
    rerank_k = case.get("rerank_k", 0)
    beam = max(case["ef"], case["k"], rerank_k)
    nodes = min(n, walks * beam)
    vectors = min(n, case["nq"] * rerank_k)
    return {"bytes": case["nq"] * (dim * 4 + case["k"] * 8) + nodes * (M * 4 + stored) + entry_scan(case) * stored + vectors * dim * 4,
            "flops": case["nq"] * transform + walks * K * float(entry_scan(case) + beam) + case["nq"] * rerank_k * 2.0 * dim}


def tolerance(case):
    if case["kind"] in ("build", "insert", "encode", "multiprobe"):
        return "exact"  # integer codes, links and code distances, ties by id
    if case["kind"] == "binary" and not case["rerank_k"]:
        return "exact"
    # fp32 sums of up to 1,024 terms; two candidates whose sums tie within that may trade places
    return {"rel": 1e-5, "max": 1e-4, "differ": 1e-3}
