"""Exact search through the tensor-core filter (csrc/exact_mma.cu) against the CPU loop and the plain kernel: ids and
distances are those of fp32 sums in d order, so every comparison is exact."""
import numpy as np
import pytest

from cphnsw_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cp():
    import cphnsw_b200
    return cphnsw_b200


def exact(cp, base, q, k):
    idx = cp.CPHNSWIndex(base.shape[1], K=8, M=4, ef_construction=8)
    idx.set_exact_base(base)
    return idx, idx.exact_search_batch(q, k)


def cpu(base, q, k):
    """The k smallest (0 - dot, id) of fp32 sums in d order."""
    with np.errstate(all="ignore"):
        dots = np.zeros((q.shape[0], base.shape[0]), np.float32)
        for d in range(base.shape[1]):
            dots += q[:, d:d + 1] * base[:, d][None, :]
        dist = np.float32(0) - dots
    part = np.argpartition(dist, k, axis=1)[:, :k]
    worst = np.take_along_axis(dist, part, 1).max(axis=1)
    ids = np.empty((q.shape[0], k), np.uint32)
    for i in range(q.shape[0]):
        c = np.flatnonzero(dist[i] <= worst[i])
        ids[i] = c[np.argsort(dist[i][c], kind="stable")[:k]]
    return ids, np.take_along_axis(dist, ids.astype(np.int64), 1)


def plain(base, q, k):
    """The plain kernel on pieces too small for the filter, joined."""
    ids, dist = [], []
    for r in range(0, base.shape[0], 16000):
        _, (i, d) = exact(cp_module(), base[r:r + 16000], q, k)
        ids.append(i.astype(np.int64) + r)
        dist.append(d)
    ids, dist = np.concatenate(ids, 1), np.concatenate(dist, 1)
    order = np.lexsort((ids, dist), axis=1)[:, :k]
    return np.take_along_axis(ids, order, 1).astype(np.uint32), np.take_along_axis(dist, order, 1)


def cp_module():
    import cphnsw_b200
    return cphnsw_b200


# groups of 32 vectors, tiles of 256 vectors and 256 queries, dims padded to 16; the least sizes the filter takes
@pytest.mark.parametrize("n,nq,dim,k", [(16384, 1, 128, 1), (16385, 257, 128, 10), (20011, 100, 96, 100), (33000, 300, 50, 32),
                                        (16639, 64, 17, 64), (40000, 513, 3, 10), (70001, 200, 128, 128)])
def test_filter_equals_cpu_loop(cp, n, nq, dim, k):
    base, q = synthetic.gaussian_mixture(n, nq, dim, max(1, n // 1000), 0.3, n + k)
    _, (ids, dist) = exact(cp, base, q, k)
    wi, wd = cpu(base, q, k)
    assert np.array_equal(ids, wi) and np.array_equal(dist, wd)


@pytest.mark.parametrize("kind", ["scales", "equal", "near", "zeros", "inf", "nan", "tiny", "negative"])
def test_awkward_values(cp, kind):
    rng = np.random.default_rng(5)
    n, nq, dim, k = 17000, 70, 64, 10
    base = rng.standard_normal((n, dim)).astype(np.float32)
    q = rng.standard_normal((nq, dim)).astype(np.float32)
    if kind == "scales":  # rows and queries of very different lengths
        base *= np.exp2(rng.integers(-12, 12, (n, 1))).astype(np.float32)
        q *= np.exp2(rng.integers(-30, 30, (nq, 1))).astype(np.float32)
    if kind == "equal":  # one vector n times: every product ties, far more candidates than the buffers hold
        base[:] = base[0]
    if kind == "near":  # products that differ by less than the bound on the error
        base[:] = base[0] + np.float32(1e-5) * base
    if kind == "zeros":
        base[:] = 0
        q[::2] = 0
    if kind == "inf":
        base[77, 3] = np.inf
    if kind == "nan":  # a query that cannot be scaled goes the plain way, the others do not mind
        q[5, 1] = np.inf
    if kind == "tiny":
        base *= np.float32(1e-30)
        q *= np.float32(1e-25)
    if kind == "negative":  # all products negative
        base, q = -np.abs(base), np.abs(q)
    with np.errstate(all="ignore"):
        _, (ids, dist) = exact(cp, base, q, k)
        wi, wd = plain(base, q, k)
    assert np.array_equal(ids, wi) and np.array_equal(dist, wd, equal_nan=True)


# tiles of 256 vectors below the smallest coordinate that is searched (2^-63) in a base that is: the larger vectors, one in every
# second tile, are far from the queries, so all neighbours are in coordinates that count as much as theirs
@pytest.mark.parametrize("k", [1, 10])
@pytest.mark.parametrize("tops", [(-62.0,), (-62.0, -64.0, -70.0), (-60.0, -63.5)])
def test_tiles_on_both_sides_of_the_smallest_coordinate(cp, k, tops):
    rng = np.random.default_rng(11)
    n, nq, dim = 20000, 70, 32
    base = (rng.uniform(-1, 1, (n, dim)) * 2.0 ** -63.2).astype(np.float32)
    q = np.abs(rng.standard_normal((nq, dim))).astype(np.float32)
    for i, row in enumerate(range(100, n, 512)):
        base[row, i % dim] = -2.0 ** tops[i % len(tops)]
    _, (ids, dist) = exact(cp, base, q, k)
    wi, wd = cpu(base, q, k)
    assert np.array_equal(ids, wi) and np.array_equal(dist, wd)


def test_lost_wait_costs_no_result(cp):
    # the sweep's first wait gets no polls: every query is answered the plain way, and nothing is left behind that a later
    # call on the handle would report as its own
    base, q = synthetic.gaussian_mixture(17000, 300, 64, 17, 0.3, 9)
    idx = cp.CPHNSWIndex(64, K=32, M=16)
    idx.set_exact_base(base)
    idx.set_param("first_wait_polls", 0)
    ids, dist = idx.exact_search_batch(q, 10)
    wi, wd = cpu(base, q, 10)
    assert np.array_equal(ids, wi) and np.array_equal(dist, wd)
    idx.check_device_status()
    idx.set_param("first_wait_polls", 1 << 22)
    idx.add_batch_parallel(base[:5000])
    assert idx.size() == 5000


def test_beside_a_graph_on_another_stream(cp):
    # a kNN graph and an exact search of one handle in flight on two streams: no workspace in common
    import torch
    n, nq, dim = 40000, 400, 128
    base, q = synthetic.gaussian_mixture(n, nq, dim, 40, 0.3, 21)
    idx = cp.CPHNSWIndex(dim, K=32)
    d_base, d_q = torch.from_numpy(base).cuda(), torch.from_numpy(q).cuda()
    codes = torch.from_numpy(idx.encode(base)).cuda()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()

    def graph():
        nbrs = torch.empty((n, 64), dtype=torch.int32, device="cuda")
        idx.knn_graph_dev(codes.data_ptr(), n, 64, 0, n, nbrs.data_ptr(), stream=a.cuda_stream)
        return nbrs

    def search():
        ids, dist = torch.empty((nq, 10), dtype=torch.int32, device="cuda"), torch.empty((nq, 10), device="cuda")
        idx.exact_search_dev(d_base.data_ptr(), n, d_q.data_ptr(), nq, 10, ids.data_ptr(), dist.data_ptr(), stream=b.cuda_stream)
        return ids

    torch.cuda.synchronize()
    g0 = graph()
    torch.cuda.synchronize()
    s0 = search()
    torch.cuda.synchronize()
    got = [(graph(), search()) for _ in range(4)]
    torch.cuda.synchronize()
    for g, s in got:
        assert bool((g == g0).all()) and bool((s == s0).all())


def test_no_room_for_the_filters(cp, oracle):
    # the workspaces of both filters above the limit: the kernels without one answer
    base, q = synthetic.gaussian_mixture(17000, 40, 64, 17, 0.3, 33)
    idx = cp.CPHNSWIndex(64, K=32)
    idx.set_param("workspace_limit_mb", 2)
    idx.set_exact_base(base)
    before = idx.launch_count()
    ids, dist = idx.exact_search_batch(q, 10)
    assert idx.launch_count() - before <= 2
    wi, wd = cpu(base, q, 10)
    assert np.array_equal(ids, wi) and np.array_equal(dist, wd)
    codes = idx.encode(base[:5000])
    before = idx.launch_count()
    nbrs, d = idx.knn_graph(codes, 32)
    assert idx.launch_count() - before <= 2
    wn, wd = oracle.knn_graph(codes, 32, 0, 5000)
    assert np.array_equal(nbrs, wn) and np.array_equal(d, wd)
    idx.set_param("knn_kernel", 3)
    with pytest.raises(cp.CPHNSWError):
        idx.knn_graph(codes, 32)
    idx.set_param("workspace_limit_mb", 0)
    assert np.array_equal(idx.knn_graph(codes, 32)[0], wn)
