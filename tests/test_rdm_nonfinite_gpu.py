"""4-qubit reduced density matrices of states that hold an infinity or a NaN: every entry of that
row and column is not finite in either part, the diagonal's imaginary part included
(x x* = inf * 0 - 0 * inf), every other entry is the finite state's. And of finite states: Hermitian to
the bit. Sizes on either side of the change of chunks. Tolerance of the finite entries: FP64 sums of at
most 2^15 products, 1e-13 relative to the matrix (test_rdm_gpu.py)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,qubits", [(4, (0, 1, 2, 3)), (6, (5, 2, 0, 3)), (12, (0, 11, 6, 2)), (19, (18, 1, 9, 4))])
@pytest.mark.parametrize("bad", [None, complex(np.inf, 0.5), complex(0.5, -np.inf), complex(np.nan, 0.5)],
                         ids=["finite", "inf", "ninf", "nan"])
@pytest.mark.parametrize("precision", [q.STATE_C64, q.STATE_C128], ids=["c64", "c128"])
def test_rdm4_of_states_with_infinities(n, qubits, bad, precision):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    psi = torch.randn(2 ** n, dtype=torch.complex128, device="cuda", generator=g)
    psi /= torch.linalg.vector_norm(psi)
    if precision == q.STATE_C64:
        psi = psi.to(torch.complex64)
    x = torch.movedim(psi.to(torch.complex128).reshape([2] * n), qubits, (0, 1, 2, 3)).reshape(16, -1)
    ref = x @ x.conj().T
    st, row = psi.clone(), 11
    if bad is not None:
        flat = torch.arange(2 ** n, device="cuda").reshape([2] * n)
        at = torch.movedim(flat, qubits, (0, 1, 2, 3)).reshape(16, -1)[row, -1]
        st[at] = bad
    rho = q.rdm4(precision, st, n, list(qubits))
    keep = torch.ones(16, 16, dtype=torch.bool, device="cuda")
    if bad is not None:
        keep[row, :] = keep[:, row] = False
        assert not torch.isfinite(torch.view_as_real(rho)[~keep]).any()
        assert torch.isnan(rho.imag[row, row])
    else:
        assert torch.equal(rho, rho.conj().T.resolve_conj())
    assert torch.isfinite(torch.view_as_real(rho)[keep]).all()
    assert torch.linalg.vector_norm((rho - ref)[keep]) <= 1e-13 * torch.linalg.vector_norm(ref)
    assert (rho.imag.diagonal()[keep.diagonal()] == 0).all()
