"""The kNN graph with the tensor cores as a filter (csrc/knn_mma.cu, knn_kernel = 3) against the CPU oracle: neighbour
ids and distances are integers with ties broken by id, so every comparison is exact."""
import numpy as np
import pytest

from cphnsw_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cp():
    import cphnsw_b200
    return cphnsw_b200


@pytest.fixture(scope="module")
def oracle():
    import oracle
    return oracle


def index(cp, dim, K, cb):
    idx = cp.CPHNSWIndex(dim, K=K, component_bytes=cb)
    idx.set_param("knn_kernel", 3)
    return idx


def check(idx, oracle, codes, k, rows=None):
    n = codes.shape[0]
    rb, re = rows or (0, n)
    nbrs, dist = idx.knn_graph(codes, k, rb, re)
    wn, wd = oracle.knn_graph(codes, k, rb, re)
    assert np.array_equal(nbrs, wn) and np.array_equal(dist, wd)


# tiles are 256 rows by 256 candidates; 8 symbols up to K = 32, 4 up to K = 64
@pytest.mark.parametrize("n,k,K,cb,dim", [(1, 4, 32, 1, 128), (255, 64, 32, 1, 128), (256, 127, 32, 1, 128), (257, 1, 16, 1, 100),
                                          (513, 40, 2, 1, 64), (3000, 64, 32, 1, 128), (2999, 32, 24, 1, 96), (2049, 64, 33, 1, 128),
                                          (4100, 64, 64, 1, 128), (1500, 127, 61, 1, 128), (2300, 64, 32, 2, 960), (1200, 20, 64, 2, 300)])
def test_shapes(cp, oracle, n, k, K, cb, dim):
    base, _ = synthetic.gaussian_mixture(n, 1, dim, max(1, n // 400), 0.3, n + K)
    codes = oracle.encode(base, K, cb, oracle.sign_tables(dim, K, 42))
    idx = index(cp, dim, K, cb)
    check(idx, oracle, codes, k)
    if n > 600:
        check(idx, oracle, codes, k, (n // 3, n // 3 + 300))  # a row block across a tile edge


# the row buffers overflow many times: unclustered rows, identical rows, rows that differ in one component only
@pytest.mark.parametrize("kind", ["random", "equal", "near"])
def test_full_buffers_and_ties(cp, oracle, kind):
    rng = np.random.default_rng(7)
    n, K = 6000, 32
    codes = rng.integers(0, 256, (n, K)).astype(np.uint8)
    if kind == "equal":
        codes[:] = codes[0]
    if kind == "near":
        codes[:] = codes[0]
        codes[np.arange(n), rng.integers(0, K, n)] = rng.integers(0, 256, n)
    idx = index(cp, 128, K, 1)
    check(idx, oracle, codes, 64, (0, 700))
    check(idx, oracle, codes, 127, (n - 300, n))


def test_many_clusters_against_the_bit_sliced_kernel(cp):
    # row tiles in a full wave of blocks and in a split one; both kernels are exact, so they agree
    base, _ = synthetic.gaussian_mixture(70_001, 1, 128, 70, 0.3, 11)
    idx = index(cp, 128, 32, 1)
    codes = idx.encode(base)
    a = idx.knn_graph(codes, 64)
    idx.set_param("knn_kernel", 2)
    b = idx.knn_graph(codes, 64)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


# the operand's length turns (64 values a step; 28 components are the first whose rows share tensor memory with the scales), in
# 149 row tiles: a full wave of blocks, and one row tile that all of them share
@pytest.mark.parametrize("K", [9, 10, 18, 19, 27, 28, 31, 42, 43, 64])
def test_operand_lengths(cp, K):
    base, _ = synthetic.gaussian_mixture(38_100, 1, 96, 38, 0.3, K)
    idx = index(cp, 96, K, 1)
    codes = idx.encode(base)
    a = idx.knn_graph(codes, 40)
    idx.set_param("knn_kernel", 1)
    b = idx.knn_graph(codes, 40)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("K,cb", [(32, 1), (32, 2)])
def test_codes_off_a_sector_boundary(cp, oracle, K, cb):
    # 16-byte aligned device codes are read by 16 bytes, 32-byte aligned ones by 32
    import torch
    n, k = 1500, 64
    codes = np.random.default_rng(K + cb).integers(0, 16, (n, K)).astype(np.uint8 if cb == 1 else np.uint16)
    wn, wd = oracle.knn_graph(codes, k, 0, n)
    buf = torch.zeros(n * K * cb + 64, dtype=torch.uint8, device="cuda")
    idx = index(cp, 128 if cb == 1 else 300, K, cb)
    for offset in (0, 16):
        buf[offset:offset + n * K * cb] = torch.from_numpy(codes.reshape(-1).view(np.uint8)).cuda()
        nbrs = torch.zeros((n, k), dtype=torch.int32, device="cuda")
        idx.knn_graph_dev(buf.data_ptr() + offset, n, k, 0, n, nbrs.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        assert np.array_equal(nbrs.cpu().numpy().view(np.uint32), wn)


def test_two_byte_codes_at_an_odd_address(cp, oracle):
    # rows of 20 bytes are copied byte by byte into padded ones: any address will do
    import torch
    n, K, k = 4200, 10, 20
    codes = np.random.default_rng(8).integers(0, 8, (n, K)).astype(np.uint16)
    wn, _ = oracle.knn_graph(codes, k, 0, n)
    idx = cp.CPHNSWIndex(300, K=K, component_bytes=2)
    buf = torch.zeros(n * K * 2 + 16, dtype=torch.uint8, device="cuda")
    nbrs = torch.zeros((n, k), dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    for offset in (0, 1, 2):
        buf[offset:offset + n * K * 2] = torch.from_numpy(codes.reshape(-1).view(np.uint8)).cuda()
        nbrs.zero_()
        idx.knn_graph_dev(buf.data_ptr() + offset, n, k, 0, n, nbrs.data_ptr(), stream=st)
        assert np.array_equal(nbrs.cpu().numpy().view(np.uint32), wn)
    idx.set_param("knn_kernel", 3)
    with pytest.raises(ValueError):
        idx.knn_graph_dev(buf.data_ptr() + 1, n, k, 0, n, nbrs.data_ptr(), stream=st)


def test_lost_wait_is_reported(cp, oracle):
    # the first wait gets no polls: every role of the block ends and the call reports it; the handle stays usable
    codes = np.random.default_rng(3).integers(0, 256, (3000, 32)).astype(np.uint8)
    idx = index(cp, 128, 32, 1)
    idx.set_param("first_wait_polls", 0)
    with pytest.raises(cp.CPHNSWError) as err:
        idx.knn_graph(codes, 16)
    assert "[%d]" % cp.E_DEVICE_WAIT in str(err.value)
    idx.set_param("first_wait_polls", 1 << 22)
    check(idx, oracle, codes, 16)


def test_lost_wait_leaves_empty_rows(cp, oracle):
    # the buffers' lengths of an earlier graph are still in the workspace: none of them may be read as this one's
    import torch
    codes = np.random.default_rng(4).integers(0, 256, (6000, 32)).astype(np.uint8)
    idx = index(cp, 128, 32, 1)
    d_codes = torch.from_numpy(codes).cuda()
    nbrs = torch.zeros((6000, 64), dtype=torch.int32, device="cuda")
    dist = torch.zeros((6000, 64), dtype=torch.int16, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    idx.knn_graph_dev(d_codes.data_ptr(), 6000, 64, 0, 6000, nbrs.data_ptr(), dist.data_ptr(), stream=st)
    idx.set_param("first_wait_polls", 0)
    idx.knn_graph_dev(d_codes.data_ptr(), 6000, 64, 0, 6000, nbrs.data_ptr(), dist.data_ptr(), stream=st)
    torch.cuda.synchronize()
    assert bool((nbrs == -1).all()) and bool((dist == -1).all())
    with pytest.raises(cp.CPHNSWError):
        idx.check_device_status()
    idx.set_param("first_wait_polls", 1 << 22)
    check(idx, oracle, codes, 64, (0, 300))


def test_lost_handover_is_reported(cp, oracle):
    # no polls for the stages that the products hand back: the wait for the first of them is lost, and the call reports it
    codes = np.random.default_rng(5).integers(0, 256, (4300, 32)).astype(np.uint8)
    idx = index(cp, 128, 32, 1)
    idx.set_param("handover_polls", 0)
    with pytest.raises(cp.CPHNSWError) as err:
        idx.knn_graph(codes, 16)
    assert "[%d]" % cp.E_DEVICE_WAIT in str(err.value)
    idx.set_param("handover_polls", idx.get_param("first_wait_polls"))
    check(idx, oracle, codes, 16)


# the data decide between the filter and a kernel without one: byte-wise (few components in all; widths the bit planes do
# not serve) or bit-sliced; clustered and unclustered rows, all of them and a block
@pytest.mark.parametrize("n,K,cb,dim", [(8192, 32, 1, 128), (9000, 64, 1, 128), (17000, 64, 1, 128), (8200, 24, 1, 96), (8500, 32, 2, 960),
                                        (8300, 16, 2, 300)])
@pytest.mark.parametrize("clustered", [True, False])
def test_picked_kernel(cp, oracle, n, K, cb, dim, clustered):
    rng = np.random.default_rng(n + K)
    if clustered:
        base, _ = synthetic.gaussian_mixture(n, 1, dim, n // 500, 0.2, n + K)
        codes = oracle.encode(base, K, cb, oracle.sign_tables(dim, K, 42))
    else:
        codes = rng.integers(0, 2 * (1 << (dim - 1).bit_length()), (n, K)).astype(np.uint8 if cb == 1 else np.uint16)
    idx = cp.CPHNSWIndex(dim, K=K, component_bytes=cb)
    check(idx, oracle, codes, 40, (n // 3, n // 3 + 200))
    nbrs, dist = idx.knn_graph(codes, 64)
    idx.set_param("knn_kernel", 1)
    wn, wd = idx.knn_graph(codes, 64)
    assert np.array_equal(nbrs, wn) and np.array_equal(dist, wd)


def test_unclustered_data_do_not_go_through_the_filter(cp):
    # 20,000 points of the unit sphere: the filter takes 3.1 ms, the byte-wise kernel 1.55, the sample and what it skips 0.2
    import torch
    n = 20000
    x = torch.randn((n, 128), device="cuda")
    idx = cp.CPHNSWIndex(128, K=32)
    codes = torch.empty((n, 32), dtype=torch.uint8, device="cuda")
    nbrs = torch.empty((n, 64), dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    idx.encode_dev(x.data_ptr(), n, codes.data_ptr(), stream=st)
    time = {}
    for kernel in (0, 3):
        idx.set_param("knn_kernel", kernel)
        ms = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            idx.knn_graph_dev(codes.data_ptr(), n, 64, 0, n, nbrs.data_ptr(), stream=st)
            b.record()
            torch.cuda.synchronize()
            ms.append(a.elapsed_time(b))
        time[kernel] = min(ms[1:])
    assert time[0] < 0.85 * time[3]


def test_unsupported_codes_are_refused(cp):
    idx = index(cp, 128, 100, 1)
    with pytest.raises(cp.CPHNSWError):
        idx.knn_graph(np.zeros((10, 100), np.uint8), 4)
