"""The last pass of a run of fused gate pairs, whose outputs are doubles, with an operator whose rows
lie more than 2^62 apart: every row of it is cut at its own scale, so its outputs are as accurate
relative to themselves as the largest row's. States on either side of the size up to which the
passes share one launch, with and without a permutation behind the last pass. Against the same gates in
FP64, every output row of the operator relative to its own magnitude: a pass costs about 1e-14
relative L2 (test_gate_chain_gpu.py), five passes stay below 1e-12."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu


def gate(rng, rows):
    """Haar-random, output row o scaled by 2^rows[o]; elements [in, out]."""
    z = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
    u, r = np.linalg.qr(z)
    u = (u * (np.diag(r) / np.abs(np.diag(r)))).T * np.exp2(np.array(rows, dtype=np.float64))
    return torch.from_numpy(np.ascontiguousarray(u.reshape(-1))).cuda()


@pytest.mark.parametrize("n", [11, 13, 19, 23])
@pytest.mark.parametrize("rows", [(0, -40, 0, -33), (-50, 0, -31, 31), (0, -25, -5, 0)], ids=["80", "162", "50"])
@pytest.mark.parametrize("permuted", [False, True], ids=["in_place", "permuted"])
def test_rows_keep_their_own_scale(n, rows, permuted):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    rng = np.random.default_rng(n)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    psi = torch.randn(2 ** n, dtype=torch.complex128, device="cuda", generator=gen)
    psi /= torch.linalg.vector_norm(psi)
    gates = []
    for k in range(5):
        t = [int(x) for x in rng.choice(n, size=4, replace=False)]
        r = rows if k == 4 else (0, 0, 0, 0)
        gates += [(t[:2], gate(rng, r)), (t[2:], gate(rng, r))]
    dims, old = [2] * n, q.get_arithmetic()
    ptup = [int(x) for x in rng.permutation(n)]
    try:
        q.set_arithmetic(q.ARITH_FP64)
        ref = psi.clone()
        for targets, g in gates:
            q.apply_gate(ref, dims, targets, g)
        q.set_arithmetic(q.ARITH_BF16X6)
        q.take_device_errors()
        runs = [(gates, ptup), ([], None)] if permuted else [(gates, None)]
        out = q.apply_gate_runs(psi, torch.empty_like(psi), dims, runs)
        assert q.take_device_errors() == 0
    finally:
        q.set_arithmetic(old)
    if permuted:
        out = q.permute(out, dims, [int(x) for x in np.argsort(ptup)])  # back to the gates' axes

    def by_row(x):  # output rows of the last operator
        return torch.movedim(x.reshape(dims), t, (0, 1, 2, 3)).reshape(16, -1)

    err = torch.linalg.vector_norm(by_row(out) - by_row(ref), dim=1) / torch.linalg.vector_norm(by_row(ref), dim=1)
    assert torch.all(err < 1e-12), err
