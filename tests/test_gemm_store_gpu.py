"""Split-precision contractions of one K-slice write C in whole 32-byte sectors wherever 16 columns of
a row are there: rows of odd length (every other one starts inside a sector), an output that starts
inside one itself, last columns and rows that fill no tile. An element depends on its row of A and
its column of B alone, so every element has the bits that it has in a product with more rows and columns; and
nothing beside the output is written."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(64, 256, 16), (1, 1, 3), (65, 15, 40), (63, 17, 16), (130, 31, 64), (64, 255, 8),
                                   (77, 257, 512), (200, 289, 33), (3, 1000, 64), (320, 511, 100)])
@pytest.mark.parametrize("offset", [0, 1])
def test_rows_of_any_length(M, N, K, offset):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    rng = np.random.default_rng(M + 1000 * N)
    M2, N2 = (M + 64) // 64 * 64, (N + 256) // 256 * 256
    a = torch.from_numpy(rng.standard_normal((M2, K)) + 1j * rng.standard_normal((M2, K))).cuda()
    b = torch.from_numpy(rng.standard_normal((K, N2)) + 1j * rng.standard_normal((K, N2))).cuda()
    buf = torch.full((M * N + 4,), -7.0, dtype=torch.complex128, device="cuda")
    out = buf[offset:offset + M * N]
    old = q.get_gemm_precision()
    q.set_gemm_precision(q.GEMM_BF16X3)
    try:
        q.take_device_errors()
        q.contract(q.Tensor(q.DENSE, [], [M, K], a[:M].contiguous().reshape(-1)),
                   q.Tensor(q.DENSE, [], [K, N], b[:, :N].contiguous().reshape(-1)), [(1, 0)], out=out)
        ref = q.contract(q.Tensor(q.DENSE, [], [M2, K], a.reshape(-1)), q.Tensor(q.DENSE, [], [K, N2], b.reshape(-1)),
                         [(1, 0)])[0].data
        assert q.take_device_errors() == 0
    finally:
        q.set_gemm_precision(old)
    assert torch.equal(torch.view_as_real(out.reshape(M, N)), torch.view_as_real(ref.reshape(M2, N2)[:M, :N]))
    exact = a[:M] @ b[:, :N]
    assert torch.linalg.vector_norm(out.reshape(M, N) - exact) < 2e-6 * torch.linalg.vector_norm(exact)
    assert (buf[:offset] == -7).all() and (buf[offset + M * N:] == -7).all()
