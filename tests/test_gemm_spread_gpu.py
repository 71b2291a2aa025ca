"""The FP64 GEMM of small results (threads spread over the outputs and over K) through
Tensor::contract, against a plain complex128 matrix product.

Tolerance: K products summed in FP64 with one rounding each, K <= 5000: relative L2 well
below K^(1/2) 2^-52 times a condition of order 10 for Gaussian operands, 1e-13."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu


# one output; fewer outputs than SMs; K below and above the threads of an output; 64 outputs a
# block with a remainder; just below and above the share of the SMs' time that 64 x 64 tiles
# fill (9/10 of 152 tiles); M 1 and N 1
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (1, 1, 5000), (3, 5, 2), (151, 1, 37), (1, 153, 300), (77, 39, 45),
                                   (130, 75, 16), (64, 64, 64), (767, 700, 3), (768, 768, 3), (832, 768, 3)])
def test_small_fp64_gemm_matches_matmul(m, n, k):
    rng = np.random.default_rng(m * 7 + n * 3 + k)
    a = rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))
    b = rng.standard_normal((k, n)) + 1j * rng.standard_normal((k, n))
    old = q.get_gemm_precision()
    q.set_gemm_precision(q.GEMM_FP64)
    try:
        t = [q.Tensor(q.DENSE, [], list(x.shape), torch.from_numpy(x.reshape(-1)).cuda()) for x in (a, b)]
        out, _, _, _ = q.contract(t[0], t[1], [(1, 0)])
    finally:
        q.set_gemm_precision(old)
    ref = a @ b
    assert np.linalg.norm(out.data.cpu().numpy().reshape(m, n) - ref) <= 1e-13 * np.linalg.norm(ref)
