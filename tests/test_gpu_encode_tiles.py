"""Encoding at the edges of the kernels' tiles and padded dimensions (csrc/encode.cu) against the oracle: codes, rotated
values and magnitudes are those of fp32 sums in the reference's stage order, so every comparison is exact.  The inputs
include one-hot and small-integer vectors, whose transforms are full of equal magnitudes (the lowest index wins)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,cb", [(17, 1), (32, 1), (33, 1), (64, 2), (65, 1), (129, 2), (256, 2), (257, 2), (510, 2), (512, 2), (513, 2),
                                    (1023, 2), (1024, 2)])
@pytest.mark.parametrize("n,K,conv", [(1, 5, 1), (129, 8, 2), (2050, 19, 0)])
def test_encode_tiles_match_oracle(oracle, dim, cb, n, K, conv):
    import cphnsw_b200 as cp
    rng = np.random.default_rng(dim + n)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    x[0::3] = np.eye(dim, dtype=np.float32)[rng.integers(0, dim, len(x[0::3]))]
    x[1::3] = rng.integers(-1, 2, x[1::3].shape)
    idx = cp.CPHNSWIndex(dim, M=8, ef_construction=8, K=K, component_bytes=cb, fht_convention=conv)
    signs = oracle.sign_tables(dim, K, 42)
    want, wrot, wmag = oracle.encode(x, K, cb, signs, conv, want_rotated=True)
    assert np.array_equal(idx.encode(x), want)
    codes, rot, mag = idx.encode_queries(x)
    assert np.array_equal(codes, want)
    assert np.array_equal(mag, wmag)
    assert np.array_equal(rot, wrot)  # a zero's sign apart


@pytest.mark.parametrize("dim,cb", [(20, 1), (64, 1), (100, 1), (256, 2), (500, 2), (700, 2)])
@pytest.mark.parametrize("n", [1, 300])
def test_rotated_vectors_to_any_float_address(dim, cb, n):
    # the buffer for the rotated vectors starts one to three floats past a 16-byte boundary
    import torch
    import cphnsw_b200 as cp
    K = 12
    x = torch.randn((n, dim), device="cuda")
    idx = cp.CPHNSWIndex(dim, M=8, ef_construction=8, K=K, component_bytes=cb)
    P = 1 << (dim - 1).bit_length()
    st = torch.cuda.current_stream().cuda_stream
    codes = torch.empty(n * K * cb, dtype=torch.uint8, device="cuda")
    want = None
    for off in range(4):
        buf = torch.full((n * K * P + 8,), 7.0, device="cuda")
        idx.encode_dev(x.data_ptr(), n, codes.data_ptr(), buf.data_ptr() + 4 * off, stream=st)
        assert bool((buf[:off] == 7).all()) and bool((buf[off + n * K * P:] == 7).all())
        rot = buf[off:off + n * K * P].cpu().numpy()
        want = rot if want is None else want
        assert np.array_equal(rot, want)
