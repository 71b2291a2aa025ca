"""4-qubit reduced density matrices against a plain complex128 matrix product of the same
state. Tolerance: FP64 sums of at most 2^14 products, relative L2 well below 2^7 2^-52 for
positive diagonal sums, 1e-13; the result is exactly Hermitian with a real diagonal."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu


# 4: one column; 6: fewer columns than a chunk; 17 and 18: on either side of the chunks' change
# at 64 columns an SM; 20: several chunks a block
@pytest.mark.parametrize("n,qubits", [(4, (3, 0, 2, 1)), (6, (0, 1, 4, 5)), (9, (8, 3, 0, 5)), (17, (16, 2, 9, 0)),
                                      (18, (4, 17, 5, 6)), (20, (19, 18, 1, 7))])
@pytest.mark.parametrize("precision", [q.STATE_C64, q.STATE_C128], ids=["c64", "c128"])
def test_rdm4_matches_matrix_product(n, qubits, precision):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    psi = torch.randn(2 ** n, dtype=torch.complex128, device="cuda", generator=g)
    psi /= torch.linalg.vector_norm(psi)
    st = psi if precision == q.STATE_C128 else psi.to(torch.complex64)
    rho = q.rdm4(precision, st, n, list(qubits))
    x = torch.movedim(st.to(torch.complex128).reshape([2] * n), qubits, (0, 1, 2, 3)).reshape(16, -1)
    ref = x @ x.conj().T
    assert torch.linalg.vector_norm(rho - ref) <= 1e-13 * torch.linalg.vector_norm(ref)
    assert torch.equal(rho.imag.diagonal(), torch.zeros(16, dtype=torch.float64, device="cuda"))
