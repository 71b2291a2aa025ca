"""Gates on two qutrits (nine amplitudes per group) on either side of the line between the form that
shares a group among threads and the one that keeps it in one: about 400 groups per SM. Against
complex128 products: float-float keeps 46 bits, 9 products a sum; the bar is 1e-12 of the largest."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", [q.ARITH_F32X2, q.ARITH_BF16X6])
@pytest.mark.parametrize("per_sm,more", [(400, -1), (400, 0), (400, 1), (0, 1), (1, 5)])
@pytest.mark.parametrize("first", [True, False])
def test_nine_amplitudes(per_sm, more, first, arith):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    groups = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    rng = np.random.default_rng(groups)
    u = np.linalg.qr(rng.standard_normal((9, 9)) + 1j * rng.standard_normal((9, 9)))[0]
    gate = torch.from_numpy(u).cuda()
    x = torch.from_numpy(rng.standard_normal((9, groups)) + 1j * rng.standard_normal((9, groups))).cuda()
    x[4, groups // 2] *= 1e40  # beyond the split range
    ref = gate.T @ x
    dims, targets, state = ([3, 3, groups], [0, 1], x) if first else ([groups, 3, 3], [1, 2], x.T)
    state = state.contiguous().reshape(-1)
    old = q.get_arithmetic()
    q.set_arithmetic(arith)
    try:
        q.apply_gate(state, dims, targets, gate.reshape(-1))
    finally:
        q.set_arithmetic(old)
    out = state.reshape(9, groups) if first else state.reshape(groups, 9).T
    err = (out - ref).abs().amax(dim=0) / ref.abs().amax(dim=0)
    assert err.max().item() < 1e-12
