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
