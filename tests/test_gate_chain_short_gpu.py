"""Short runs of fused gate pairs on states that L2 holds: one and two passes after the first are launches
of their own (three share one; its tables are not worth preparing for fewer), also where a
launch is full and one pass is left. Counted in the allocations that the calls make (the
shared launch takes a workspace for its tables beside the records'), and against the gates in FP64 (the
chain's bar of 1e-12 relative L2, test_gate_chain_gpu.py)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu


def haar(rng):
    z = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
    u, r = np.linalg.qr(z)
    return torch.from_numpy(np.ascontiguousarray((u * (np.diag(r) / np.abs(np.diag(r)))).T.reshape(-1))).cuda()


def workspaces():
    allocs, used = ctypes.c_uint64(), ctypes.c_uint64()
    q.check(q.lib().qtnh_workspace_stats(ctypes.byref(allocs), ctypes.byref(used)))
    return allocs.value


@pytest.mark.parametrize("n", [11, 16, 20])
@pytest.mark.parametrize("pairs,perm,shared", [(2, None, 0), (3, None, 0), (3, 1, 0), (4, None, 1), (4, 2, 1), (66, 64, 1), (67, 65, 1)])
def test_few_passes(n, pairs, perm, shared):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    rng = np.random.default_rng(n + 100 * pairs)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    psi = torch.randn(2 ** n, dtype=torch.complex128, device="cuda", generator=g)
    psi /= torch.linalg.vector_norm(psi)
    dims, runs, gates = [2] * n, [], []
    for k in range(pairs):
        t = [int(x) for x in rng.choice(n, size=4, replace=False)]
        gates += [(t[:2], haar(rng)), (t[2:], haar(rng))]
        if k == perm:
            runs.append((gates, [int(x) for x in rng.permutation(n)]))
            gates = []
    runs.append((gates, None))
    old = q.get_arithmetic()
    try:
        q.set_arithmetic(q.ARITH_FP64)
        ref = psi.clone()
        for gl, pt in runs:
            for targets, gate in gl:
                q.apply_gate(ref, dims, targets, gate)
            if pt is not None:
                ref = q.permute(ref, dims, pt)
        q.set_arithmetic(q.ARITH_BF16X6)
        q.take_device_errors()
        before = workspaces()
        out = q.apply_gate_runs(psi, torch.empty_like(psi), dims, runs)
        taken = workspaces() - before
        assert q.take_device_errors() == 0
    finally:
        q.set_arithmetic(old)
    assert torch.linalg.vector_norm(out - ref) < 1e-12 * torch.linalg.vector_norm(ref)
    assert taken == 1 + shared
