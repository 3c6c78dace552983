"""The kNN graph's tensor-core sweep that takes every pair once, in an order of groups, by phases (csrc/knn_mma.cu): sizes where
its routes turn, against the byte-wise kernel, which knows none of them.  Both are exact, ties by id, so they agree in every entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cp():
    import cphnsw_b200
    return cphnsw_b200


def mixture_codes(idx, n, dim, per, sigma, K, cb, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    c = torch.randn((max(1, n // per), dim), generator=g, device="cuda")
    x = c[torch.randint(0, len(c), (n,), generator=g, device="cuda")] + sigma * torch.randn((n, dim), generator=g, device="cuda")
    x /= x.norm(dim=1, keepdim=True)
    codes = torch.empty((n, K), dtype=torch.uint8 if cb == 1 else torch.int16, device="cuda")
    idx.encode_dev(x.data_ptr(), n, codes.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
    return codes


def graph(idx, codes, k, rb, re):
    import torch
    nbrs = torch.empty((re - rb, k), dtype=torch.int32, device="cuda")
    dist = torch.empty((re - rb, k), dtype=torch.int16, device="cuda")
    idx.knn_graph_dev(codes.data_ptr(), codes.shape[0], k, rb, re, nbrs.data_ptr(), dist.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    idx.check_device_status()
    return nbrs, dist


def agree(cp, idx, dim, K, cb, codes, k, rb, re):
    import torch
    plain = cp.CPHNSWIndex(dim, K=K, component_bytes=cb)
    plain.set_param("knn_kernel", 1)
    a, b = graph(idx, codes, k, rb, re), graph(plain, codes, k, rb, re)
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


# 4,096 nodes: by default through the filter and in an order from here on; 8,192: the sample is taken, and data that are not calm
# (sigma 0.5 and above) take the near columns first, 24,321 nodes and more with second bounds; 32,001: near columns first on any
# data; 32,513: phases; 32,769: a third joining of groups, second bounds on any data; 1 and 256 nodes: a tile or less; 296 row
# tiles: two whole waves and none left over, an even number; 297: odd, one left over; blocks of rows against all nodes, one of
# them on either side of the near columns; clusters far larger than what lies beside a row (several phases); two-byte and
# four-symbol codes; no clusters at all
@pytest.mark.parametrize("n,k,dim,K,cb,per,sigma,rows", [
    (10239, 64, 128, 32, 1, 1000, 0.3, None), (10240, 64, 128, 32, 1, 1000, 0.3, None), (10241, 1, 128, 32, 1, 1000, 0.3, None),
    (32256, 64, 96, 32, 1, 1000, 0.3, None), (32512, 127, 128, 32, 1, 1000, 0.3, None), (75776, 64, 128, 16, 1, 1000, 0.3, None),
    (75777, 32, 64, 32, 1, 1000, 0.3, None), (40001, 64, 128, 32, 1, 1000, 0.3, (5003, 29007)), (36000, 64, 128, 32, 1, 18000, 0.3, None),
    (20001, 64, 300, 32, 2, 1000, 0.4, None), (7001, 64, 300, 32, 2, 1, 0.3, None), (33001, 64, 128, 64, 1, 500, 0.4, (0, 33000)), (12000, 64, 128, 32, 1, 1, 0.3, None),
    (34000, 20, 64, 10, 1, 1000, 0.3, None),
    (1, 5, 64, 32, 1, 1, 0.3, None), (256, 127, 64, 32, 1, 100, 0.3, None), (257, 64, 64, 32, 1, 100, 0.3, None),
    (4095, 64, 128, 32, 1, 1000, 0.3, None), (4096, 64, 128, 32, 1, 1000, 0.3, None), (4097, 64, 300, 32, 2, 500, 0.4, None),
    (8191, 64, 128, 32, 1, 1000, 0.7, None), (8192, 64, 128, 64, 1, 1000, 0.7, None), (14001, 32, 300, 32, 2, 1000, 0.6, None),
    (24320, 64, 128, 32, 1, 1000, 0.7, None), (24321, 64, 128, 32, 1, 1000, 0.7, None), (24577, 127, 300, 32, 2, 1000, 0.6, None),
    (32000, 64, 128, 32, 1, 1000, 0.3, None), (32001, 64, 128, 32, 1, 1000, 0.6, None), (32513, 64, 128, 32, 1, 1000, 0.5, None),
    (32768, 64, 128, 16, 1, 1000, 0.6, None), (32769, 64, 128, 16, 1, 1000, 0.6, None),
    (40001, 64, 128, 32, 1, 1000, 0.5, (1000, 33000)), (40001, 64, 128, 32, 1, 1000, 0.5, (1000, 33001))])
@pytest.mark.parametrize("kernel", [0, 3])
def test_routes(cp, n, k, dim, K, cb, per, sigma, rows, kernel):
    idx = cp.CPHNSWIndex(dim, K=K, component_bytes=cb)
    codes = mixture_codes(idx, n, dim, per, sigma, K, cb, n + k)
    idx.set_param("knn_kernel", kernel)
    agree(cp, idx, dim, K, cb, codes, k, *(rows or (0, n)))


# hundreds to thousands of equal codes: more ties than a row's neighbours are taken from by id (in one phase a buffer holds n k / 256
# entries), or their rows' buffers run over twice and the row is compared with every node
@pytest.mark.parametrize("n,equal", [(5000, 390), (11000, 700), (11000, 2740), (11000, 5000), (34000, 3000)])
def test_equal_codes(cp, n, equal):
    import torch
    idx = cp.CPHNSWIndex(128, K=32)
    codes = mixture_codes(idx, n, 128, 1000, 0.3, 32, 1, n)
    codes[torch.randperm(n, device="cuda")[:equal]] = codes[0].clone()
    idx.set_param("knn_kernel", 3)
    agree(cp, idx, 128, 32, 1, codes, 64, 0, n)


def test_rows_in_blocks_where_the_workspace_is_small(cp):
    # 60,000 rows: 169 MB with all rows' buffers at once, 122 in two blocks
    idx = cp.CPHNSWIndex(128, K=32)
    codes = mixture_codes(idx, 60000, 128, 1000, 0.3, 32, 1, 5)
    idx.set_param("knn_kernel", 3)
    idx.set_param("workspace_limit_mb", 130)
    agree(cp, idx, 128, 32, 1, codes, 64, 0, 60000)
    idx.set_param("workspace_limit_mb", 20)
    with pytest.raises(cp.CPHNSWError):
        graph(idx, codes, 64, 0, 60000)


# entries of a row's buffer are one word up to 2^25 - 1 nodes and two above; nodes behind 2^27 are served like the others.  The wanted
# rows are the last 600, in six clusters whose other members lie anywhere, and 30 of them in none
@pytest.mark.parametrize("n", [(1 << 25) - 1, 1 << 25, (1 << 27) + 301])
def test_many_nodes(cp, n):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    K, rows, k = 16, 600, 20
    codes = torch.empty((n, K), dtype=torch.uint8, device="cuda")
    for i in range(0, n, 1 << 24):
        codes[i:i + (1 << 24)] = torch.randint(0, 256, (min(n - i, 1 << 24), K), generator=g, device="cuda", dtype=torch.uint8)
    centres = torch.randint(0, 256, (6, K), generator=g, device="cuda", dtype=torch.uint8)

    def member(c, m):
        own = torch.rand((m, K), generator=g, device="cuda") < 0.25
        return torch.where(own, torch.randint(0, 256, (m, K), generator=g, device="cuda", dtype=torch.uint8), centres[c])

    for c in range(6):
        codes[n - rows + 100 * c:n - rows + 100 * c + 95] = member(c, 95)
        codes[torch.randint(0, n - rows, (40,), generator=g, device="cuda")] = member(c, 40)
    idx = cp.CPHNSWIndex(64, K=K)
    idx.set_param("knn_kernel", 3)
    agree(cp, idx, 64, K, 1, codes, k, n - rows, n)
    idx.close()


# the byte-wise kernel's rows a warp, six or eight of 32 bytes: 10,656 rows are a wave of sixes, 14,208 one of eights (three blocks
# on each of 148 SMs)
@pytest.mark.parametrize("rows", [10656, 10657, 14208, 14209])
@pytest.mark.parametrize("k", [20, 64, 127])
def test_rows_a_warp(cp, rows, k):
    idx = cp.CPHNSWIndex(128, K=32)
    codes = mixture_codes(idx, 15000, 128, 1000, 0.3, 32, 1, rows)
    idx.set_param("knn_kernel", 2)
    agree(cp, idx, 128, 32, 1, codes, k, 500, 500 + rows)


# points without clusters, whose sweep finds nearly all groups of 32 rows and 32 columns: up to 65,024 nodes they have room in one list,
# above in sections of one, of which there are enough at 80,000 (the last phase has 3.2M groups, the sections room for 5.5M).  At
# 200,000 (9.8M) blocks compare what has no room
@pytest.mark.parametrize("n,dim,K,cb,rows", [
    (65024, 128, 32, 1, None), (65025, 128, 32, 1, None), (80000, 64, 16, 1, None), (200000, 128, 32, 1, None), (200000, 300, 64, 2, None),
    (200000, 300, 32, 2, (20001, 180000))])
def test_more_hits_than_the_list_has_room_for(cp, n, dim, K, cb, rows):
    idx = cp.CPHNSWIndex(dim, K=K, component_bytes=cb)
    codes = mixture_codes(idx, n, dim, 1, 1.0, K, cb, 9)
    idx.set_param("knn_kernel", 3)
    agree(cp, idx, dim, K, cb, codes, 64, *(rows or (0, n)))
