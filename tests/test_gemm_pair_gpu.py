"""The split-precision GEMM with B shared by two CTAs (an even number of 64-row tiles of C) and
without (an odd number), at the edges of its tiles: one tile, one pair, more tiles than SMs, one
K-slice and several, ragged last tiles and slices. Against numpy in complex128: the pieces hold
24 bits and a slice of 32 K-steps loses up to an ulp of FP32 a step in one direction, at most
512 * 2^-24 = 3.1e-5 of the magnitudes; measured 4.7e-7 relative L2, and the bar is 2e-6."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 8), (64, 256, 256), (65, 255, 257), (128, 257, 300), (129, 64, 512),
                                   (192, 700, 520), (256, 40, 1030), (1280, 2049, 264), (1344, 1800, 264),
                                   (4096, 300, 40)])
def test_pairs_of_row_tiles(M, N, K):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    a = (rng.standard_normal((M, K)) + 1j * rng.standard_normal((M, K))) / np.sqrt(K)
    b = rng.standard_normal((K, N)) + 1j * rng.standard_normal((K, N))
    old = q.get_gemm_precision()
    q.take_device_errors()
    q.set_gemm_precision(q.GEMM_BF16X3)
    try:
        res = q.contract(q.Tensor(q.DENSE, [], [M, K], torch.from_numpy(a.reshape(-1)).cuda()),
                         q.Tensor(q.DENSE, [], [K, N], torch.from_numpy(b.reshape(-1)).cuda()), [(1, 0)])[0]
        torch.cuda.synchronize()
    finally:
        q.set_gemm_precision(old)
    assert q.take_device_errors() == 0
    out, ref = res.data.cpu().numpy().reshape(M, N), a @ b
    assert np.linalg.norm(out - ref) < 2e-6 * np.linalg.norm(ref)
