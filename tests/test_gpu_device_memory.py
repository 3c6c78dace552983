"""Device memory kept between handles (csrc/device_memory.cu): reused, bounded, given back on request."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def free_mb():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0] / MB


def use(cp, n, dim=64):
    rng = np.random.default_rng(n)
    idx = cp.CPHNSWIndex(dim, M=8, K=16)
    base = rng.standard_normal((n, dim)).astype(np.float32)
    idx.set_exact_base(base)
    ids, _ = idx.exact_search_batch(base[:8], 1)
    assert np.array_equal(ids[:, 0], np.argmax(base[:8] @ base.T, 1))
    return idx


def test_kept_memory_is_bounded_and_given_back(cp):
    use(cp, 1000).close()  # modules and contexts are loaded
    cp.release_memory()
    before = free_mb()
    idx = use(cp, 600_000)  # 150 MB of vectors, as much again of workspace
    idx.close()
    kept = before - free_mb()
    assert kept <= 384 + 64
    use(cp, 600_000).close()  # the same sizes again: no more is kept
    assert before - free_mb() <= 384 + 64
    cp.release_memory()
    assert abs(before - free_mb()) <= 32
    use(cp, 3_000_000).close()  # more than is kept without handles
    assert before - free_mb() <= 384 + 64
    cp.release_memory()
    with pytest.raises(ValueError):
        cp.release_memory(999)


def test_handles_of_several_threads(cp):
    errors = []

    def work(seed):
        try:
            for i in range(4):
                use(cp, 20_000 + 1000 * seed + i).close()
                if i == 2:
                    cp.release_memory()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors


def test_a_large_graph_workspace_does_not_stay_with_the_index(cp):
    # 1.3M nodes: 2.2 GB of buffers for the kNN graph, which the index has no use for once it is searched
    import torch
    use(cp, 1000).close()
    cp.release_memory()
    rng = np.random.default_rng(3)
    n, dim = 1_300_000, 32
    base = (rng.standard_normal((1300, dim)).repeat(1000, 0) + 0.1 * rng.standard_normal((n, dim))).astype(np.float32)
    before = free_mb()
    idx = cp.CPHNSWIndex(dim, M=8, K=16)
    idx.add_batch_parallel(base)
    held = before - free_mb()  # vectors 160, links 40, candidates 80, codes 20; 1,024 at most are kept for other buffers
    assert held <= 1024 + 512
    # by the stages on device arrays: they enqueue only, so the workspace goes when the index is installed
    x = torch.from_numpy(base).cuda()
    codes = torch.empty((n, 16), dtype=torch.uint8, device="cuda")
    cand = torch.empty((n, 16), dtype=torch.int32, device="cuda")
    idx.close()
    cp.release_memory()
    before = free_mb()
    idx = cp.CPHNSWIndex(dim, M=8, K=16)
    st = torch.cuda.current_stream().cuda_stream
    idx.encode_dev(x.data_ptr(), n, codes.data_ptr(), stream=st)
    idx.knn_graph_dev(codes.data_ptr(), n, 16, 0, n, cand.data_ptr(), stream=st)
    assert before - free_mb() > 2000
    adj = cand[:, :8].contiguous()
    idx.install_dev(x.data_ptr(), codes.data_ptr(), adj.data_ptr(), n, stream=st)
    assert before - free_mb() <= 1024 + 512
    idx.close()
    cp.release_memory()
