"""Runs of fused gate pairs that stay resident in L2 (all passes after the first in one
launch) and the size where every pass becomes a launch of its own, against the oracle.

Tolerance: the chain's bar of 1e-12 relative L2. A pass cuts the state at 48 bits of its
largest magnitude and drops products below 2^-48, about 1e-14 relative L2 a pass; the
errors of the passes are independent, so 130 passes stay below 2e-13."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.complex128).reshape(-1)).cuda()


def haar(rng):
    z = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
    u, r = np.linalg.qr(z)
    return (u * (np.diag(r) / np.abs(np.diag(r)))).T.reshape(-1)


def oracle_runs(psi, n, runs):
    t = orc.Tensor(orc.DENSE, [], [2] * n, psi)
    for gates, pt in runs:
        for targets, els in gates:
            t, _, _ = orc.contract(t, orc.Tensor(orc.SYMM, [], [2] * 4, els), [(targets[0], 0), (targets[1], 1)])
        if pt is not None:
            t = orc.Tensor(orc.DENSE, [], [2] * n, orc.permute(t.els.reshape([2] * n), pt).reshape(-1))
    return t.els


# 11: one tile; 13: eight tiles; 19: 256 tiles, more than one for some SMs; 130 passes: three
# launches, a permutation at the end of one; scale: a gate out of the digit range in the
# middle (that pass in FP64, the next from doubles), rows of very different scale
@pytest.mark.parametrize("n,passes,perms,scale", [(11, 130, (63, 64, 100), None), (12, 3, (), None), (13, 9, (1, 5), 1e230),
                                                  (13, 6, (), "rows"), (19, 4, (2,), None), (22, 3, (1,), None),
                                                  (23, 3, (1,), None)])
def test_chain_passes_match_oracle(n, passes, perms, scale):
    rng = np.random.default_rng(1000 * n + passes)
    psi = rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)
    psi /= np.linalg.norm(psi)
    runs, gates = [], []
    for k in range(passes):
        q4 = [int(x) for x in rng.choice(n, size=4, replace=False)]
        if k % 3 == 0:
            q4[k % 4] = n - 1 if n - 1 not in q4 else q4[k % 4]  # the innermost axis among the targets
        a, b = haar(rng), haar(rng)
        if scale == "rows":
            a = a * np.repeat([1.0, 1e3, 1.0, 1e-3], 4).reshape(4, 4).T.reshape(-1)
        elif scale is not None and k == passes // 2:
            a = a * scale
        elif scale is not None and k == passes // 2 + 1:
            a = a / scale
        gates += [(q4[:2], a), (q4[2:], b)]
        if k in perms:
            runs.append((gates, [int(x) for x in rng.permutation(n)]))
            gates = []
    runs.append((gates, None))
    old = q.get_arithmetic()
    q.set_arithmetic(q.ARITH_BF16X6)
    try:
        q.take_device_errors()
        st, sc = dev(psi), dev(np.zeros_like(psi))
        out = q.apply_gate_runs(st, sc, [2] * n, [([(t, dev(g)) for t, g in gl], pt) for gl, pt in runs])
        assert q.take_device_errors() == 0
    finally:
        q.set_arithmetic(old)
    ref = oracle_runs(psi, n, runs)
    assert np.linalg.norm(out.cpu().numpy() - ref) / np.linalg.norm(ref) < 1e-12
