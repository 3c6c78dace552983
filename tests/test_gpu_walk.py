"""The beam walk where its dispatch turns (csrc/search_walk.cu): a block or a warp per query, with and without the entry
scan, the narrow and the wide rerank, beams at the edges of their steps.  Without statistics asked for the walk keeps a
lossy filter of the nodes it has seen; ids and distances are those of the one-warp kernel and of the oracle all the same,
bit for bit."""
import numpy as np
import pytest

from cphnsw_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,K,cb,M,k,ef,rerank,entries,seeds", [
    (128, 32, 1, 32, 10, 100, 500, 500, 32),   # K = 32, P = 128: the specialised scores
    (96, 16, 1, 16, 1, 1, 0, 64, 1),           # a beam of one
    (40, 33, 1, 24, 32, 33, 40, 100, 31),      # a second, ragged block of rotations
    (300, 16, 2, 32, 10, 64, 64, 32, 32),      # two-byte components; every entry is a seed: no scan
    (128, 32, 1, 32, 10, 65, 0, 100, 33),      # more seeds than the scan keeps
    (960, 8, 2, 32, 10, 1000, 1024, 7, 32),    # a table of 32 KB; fewer entries than seeds; a full list to rerank
])
@pytest.mark.parametrize("nq", [1, 149, 297, 593])
def test_walk_matches_one_warp_kernel_and_oracle(cp, oracle, dim, K, cb, M, k, ef, rerank, entries, seeds, nq):
    n = 3001
    base, q = synthetic.gaussian_mixture(n, nq, dim, 12, 0.3, dim + nq)
    idx = cp.CPHNSWIndex(dim, M=M, ef_construction=max(200, M), K=K, component_bytes=cb, fht_convention=2)
    idx.set_param("entry_scan", entries)
    idx.set_param("k_entry", seeds)
    idx.add_batch_parallel(base)
    run = (lambda: idx.search_and_rerank_batch(q, k, ef, rerank)) if rerank else (lambda: idx.search_batch(q, k, ef))
    ids, dist = run()
    idx.set_param("search_kernel", 1)
    wi, wd = run()
    assert np.array_equal(ids, wi) and np.array_equal(dist, wd)
    if not rerank:
        _, rot, _ = oracle.encode(q[:20], K, cb, oracle.sign_tables(dim, K, 42), 2, want_rotated=True)
        oi, od = oracle.search(rot, idx.codes(), idx.adjacency(), idx.entry_ids(), max(ef, k), k, n_seed=seeds)
        assert np.array_equal(ids[:20], oi) and np.array_equal(dist[:20], od)


# a block or a warp per query under the symmetric metrics: one-byte and two-byte components, sign bits with and without residual
# bits; a fifth of the vectors are copies of one (their distances tie, by id) and the beam is wider than the cluster
@pytest.mark.parametrize("kind,dim,K,ef", [("bytes", 100, 33, 40), ("bytes", 300, 16, 300), ("binary", 128, 64, 200), ("residual", 64, 32, 65)])
@pytest.mark.parametrize("nq", [1, 592, 593])
def test_few_queries_under_the_symmetric_metrics(cp, kind, dim, K, ef, nq):
    n = 3001
    base, q = synthetic.gaussian_mixture(n, nq, dim, 12, 0.3, dim + nq)
    base[::5] = base[0]
    if kind == "bytes":
        idx = cp.CPHNSWIndex(dim, M=24, ef_construction=200, K=K, component_bytes=2 if dim > 128 else 1)
    else:
        idx = cp.CPHNSWIndex.binary(dim, M=32, ef_construction=200, K=K)
    if kind == "residual":
        idx.set_param("residual_bits", 16)
    idx.set_param("entry_scan", 200)
    idx.set_param("k_entry", 32)
    idx.add_batch_parallel(base)
    run = (lambda: idx.search_multiprobe_batch(q, 10, ef, 1)) if kind == "bytes" else (lambda: idx.search_batch(q, 10, ef))
    ids, dist = run()
    idx.set_param("search_kernel", 1)
    wi, wd = run()
    assert np.array_equal(ids, wi) and np.array_equal(dist, wd)


# as many queries as go a block each, and one more: in eighths of a query an SM by links, beam, the size of the query table and the
# blocks that fit an SM (a beam of 4,096: three)
@pytest.mark.parametrize("kind,dim,K,M,ef,eighths", [
    ("bytes", 64, 16, 16, 199, 16), ("bytes", 64, 16, 16, 200, 24), ("bytes", 128, 32, 17, 63, 24), ("bytes", 128, 32, 32, 64, 30),
    ("bytes", 64, 16, 32, 4096, 24),
    ("wide", 300, 16, 32, 40, 32), ("wide", 300, 16, 32, 4096, 32), ("binary", 128, 64, 32, 40, 32), ("binary", 128, 64, 32, 4096, 27)])
def test_as_many_queries_as_go_a_block_each(cp, kind, dim, K, M, ef, eighths):
    import torch
    most = torch.cuda.get_device_properties(0).multi_processor_count * eighths // 8
    n = 4500
    base, q = synthetic.gaussian_mixture(n, most + 1, dim, 12, 0.3, dim + ef)
    if kind == "binary":
        idx = cp.CPHNSWIndex.binary(dim, M=M, ef_construction=200, K=K)
    else:
        idx = cp.CPHNSWIndex(dim, M=M, ef_construction=200, K=K, component_bytes=2 if dim > 128 else 1)
    idx.set_param("entry_scan", 200)
    idx.set_param("k_entry", 32)
    idx.add_batch_parallel(base)
    ids, dist = idx.search_batch(q, 10, ef)
    fewer = idx.search_batch(q[:most], 10, ef)
    idx.set_param("search_kernel", 1)
    wi, wd = idx.search_batch(q, 10, ef)
    assert np.array_equal(ids, wi) and np.array_equal(dist, wd)
    assert np.array_equal(fewer[0], wi[:most]) and np.array_equal(fewer[1], wd[:most])


# a base beyond L2 that is read many times over: the queries are taken by their nearest entry nodes (more queries than one pass of
# the block that orders them, fewer seeds than it looks at)
@pytest.mark.parametrize("n,dim,nq,rerank,seeds", [(40_003, 960, 601, 1000, 32), (70_001, 512, 2_500, 500, 3)])
def test_queries_in_order_of_their_entry_nodes(cp, n, dim, nq, rerank, seeds):
    base, q = synthetic.gaussian_mixture(n, nq, dim, 40, 0.3, nq)
    idx = cp.CPHNSWIndex(dim, M=32, ef_construction=200, K=16, component_bytes=2)
    idx.set_param("entry_scan", 300)
    idx.set_param("k_entry", seeds)
    idx.add_batch_parallel(base)
    ids, dist = idx.search_and_rerank_batch(q, 10, 100, rerank)
    idx.set_param("search_kernel", 1)
    wi, wd = idx.search_and_rerank_batch(q, 10, 100, rerank)
    assert np.array_equal(ids, wi) and np.array_equal(dist, wd)


# the order is taken, a launch more, from a node beyond L2 and a query beyond 2 GB of reads on; a node is 32 links, a code row of 32 bytes
# and its vector, and 1,000 are read for a query
def test_where_the_order_of_queries_begins(cp):
    import torch
    dim, node = 960, 32 * 4 + 32 + 960 * 4
    most_nodes = torch.cuda.get_device_properties(0).L2_cache_size // node
    most = int(2e9 // (1000 * node))
    base, q = synthetic.gaussian_mixture(most_nodes + 1, most + 1, dim, 40, 0.3, 17)
    launches = {}
    for n in (most_nodes, most_nodes + 1):
        idx = cp.CPHNSWIndex(dim, M=32, ef_construction=200, K=16, component_bytes=2)
        idx.set_param("entry_scan", 300)
        idx.set_param("k_entry", 32)
        idx.add_batch_parallel(base[:n])
        found = {}
        for nq in (most, most + 1):
            before = idx.launch_count()
            found[nq] = idx.search_and_rerank_batch(q[:nq], 10, 100, 1000)
            launches[n, nq] = idx.launch_count() - before
        for a, b in zip(found[most], found[most + 1]):
            assert np.array_equal(a, b[:most])
    few = launches[most_nodes, most]
    assert launches[most_nodes, most + 1] == few and launches[most_nodes + 1, most] == few
    assert launches[most_nodes + 1, most + 1] == few + 1


@pytest.mark.parametrize("M", [24, 32])
@pytest.mark.parametrize("row,a,b", [(0, 0, 1), (0, 0, 16), (0, 7, 23), (256, 3, 20)])
def test_repeated_ids_in_a_row_count_once(cp, oracle, M, row, a, b):
    # one row of the graph names a node twice, at places 1 to 17 apart; the last row is the last of a ragged group of rows
    n, dim = 257, 128
    base, q = synthetic.gaussian_mixture(n, 30, dim, 2, 0.5, M + b)
    ref = cp.CPHNSWIndex(dim, M=M, ef_construction=64, K=32, component_bytes=1, fht_convention=2)
    ref.add_batch_parallel(base)
    codes, adj = ref.codes(), ref.adjacency()
    rng = np.random.default_rng(b)
    for r in {0, row}:
        adj[r] = rng.choice(np.setdiff1d(np.arange(n), [r]), M, replace=False)
    adj[row, b] = adj[row, a]
    idx = cp.CPHNSWIndex(dim, M=M, ef_construction=64, K=32, component_bytes=1, fht_convention=2)
    idx.set_param("k_entry", 4)
    idx.set_param("entry_scan", 4)
    idx.install(base, codes, adj)
    _, rot, _ = oracle.encode(q, 32, 1, oracle.sign_tables(dim, 32, 42), 2, want_rotated=True)
    for kernel in (0, 1):
        idx.set_param("search_kernel", kernel)
        ids, dist = idx.search_batch(q, 20, 200)
        wi, wd = oracle.search(rot, codes, adj, idx.entry_ids(), 200, 20, n_seed=4)
        assert np.array_equal(ids, wi) and np.array_equal(dist, wd)


# nodes by eights with the same links in another order each: what one warp of a block finds in a step, the others find as well, and
# of the keys listed up to seven are struck out while other warps still compare theirs
@pytest.mark.parametrize("M,nq", [(16, 1), (32, 40), (32, 149)])
def test_ids_found_by_many_rows_of_a_step_count_once(cp, oracle, M, nq):
    n, dim = 2000, 128
    base, q = synthetic.gaussian_mixture(n, nq, dim, 4, 0.5, M + nq)
    rng = np.random.default_rng(M)
    ref = cp.CPHNSWIndex(dim, M=M, ef_construction=64, K=32, component_bytes=1, fht_convention=2)
    codes = ref.encode(base)
    adj = np.empty((n, M), np.uint32)
    for i in range(0, n, 8):
        links = rng.choice(n, M, replace=False)
        for r in range(i, i + 8):
            adj[r] = rng.permutation(np.where(links == r, (r + 8) % n, links))
    idx = cp.CPHNSWIndex(dim, M=M, ef_construction=64, K=32, component_bytes=1, fht_convention=2)
    idx.set_param("k_entry", 32)
    idx.set_param("entry_scan", 32)
    idx.install(base, codes, adj)
    _, rot, _ = oracle.encode(q, 32, 1, oracle.sign_tables(dim, 32, 42), 2, want_rotated=True)
    for ef in (40, 300):
        ids, dist = idx.search_batch(q, 20, ef)
        wi, wd = oracle.search(rot, codes, adj, idx.entry_ids(), ef, 20, n_seed=32)
        assert np.array_equal(ids, wi) and np.array_equal(dist, wd)


def test_wide_rows_with_the_walk_asked_for(cp):
    # M = 48: a search under the asymmetric score is refused, walks under the code distance take the one-warp kernel
    base, q = synthetic.gaussian_mixture(1200, 20, 64, 4, 0.3, 3)
    out = []
    for kernel in (2, 1):
        idx = cp.CPHNSWIndex(64, M=48, ef_construction=64, K=32)
        idx.set_param("search_kernel", kernel)
        idx.add_batch_parallel(base[:1000])
        idx.add_batch(base[1000:])
        ids, dist = idx.search_multiprobe_batch(q, 10, 100, 3)
        out.append((idx.adjacency(), ids, dist))
        if kernel == 2:
            with pytest.raises(cp.CPHNSWError):
                idx.search_batch(q, 10, 100)
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("dim,K,cb,M,k,ef,rerank,entries,seeds", [
    (128, 32, 1, 32, 10, 100, 500, 700, 100),  # a list of 128 seeds per query
    (128, 64, 1, 32, 10, 50, 0, 900, 64),      # a beam narrower than the seeds
    (960, 16, 2, 24, 10, 300, 300, 333, 34),
    (96, 16, 1, 16, 10, 20, 0, 100, 100),      # no scan: all entries are offered, more of them than the beam takes
    (300, 40, 2, 32, 10, 64, 64, 33, 33),
])
@pytest.mark.parametrize("nq", [1, 150, 600])
def test_many_seeds_match_one_warp_kernel(cp, dim, K, cb, M, k, ef, rerank, entries, seeds, nq):
    base, q = synthetic.gaussian_mixture(3001, nq, dim, 12, 0.3, dim + nq)
    idx = cp.CPHNSWIndex(dim, M=M, ef_construction=max(200, M), K=K, component_bytes=cb)
    idx.set_param("entry_scan", entries)
    idx.set_param("k_entry", seeds)
    idx.add_batch_parallel(base)
    runs = [lambda: idx.search_and_rerank_batch(q, k, ef, rerank) if rerank else idx.search_batch(q, k, ef),
            lambda: idx.search_batch(q, k, ef, want_stats=True)]
    if nq < 600:
        runs.append(lambda: idx.search_multiprobe_batch(q, k, ef, 3))
    for run in runs:
        idx.set_param("search_kernel", 0)
        got = run()
        idx.set_param("search_kernel", 1)
        for a, b in zip(got, run()):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("dim,K,cb", [(128, 32, 1), (128, 64, 1), (100, 17, 1), (960, 32, 2), (300, 40, 2)])
@pytest.mark.parametrize("nq", [2, 700])
def test_rows_of_new_neighbours_match_one_warp_kernel(cp, dim, K, cb, nq):
    # no clusters: nearly every link of a row is a candidate, and a lane scores one (up to eight share their lookups by four)
    rng = np.random.default_rng(dim + K)
    base, q = rng.standard_normal((4000, dim)).astype(np.float32), rng.standard_normal((nq, dim)).astype(np.float32)
    idx = cp.CPHNSWIndex(dim, M=32, K=K, component_bytes=cb)
    idx.add_batch_parallel(base)
    got = idx.search_batch(q, 20, 150)
    idx.set_param("search_kernel", 1)
    for a, b in zip(got, idx.search_batch(q, 20, 150)):
        assert np.array_equal(a, b)
