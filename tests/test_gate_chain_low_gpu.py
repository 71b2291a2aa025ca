"""Chain passes on a state too large for the resident kernel, with targets among the lowest bits:
each of the three lowest bits alone, in every role of the two gates, together, and none; a
permutation that puts neighbouring outputs apart or together; and a state whose buffer is only
16-byte aligned. Against the gates applied one at a time in FP64 (the bar of the chain: 1e-12
relative L2; a pass costs about 1e-14, see test_gate_chain_gpu.py)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu
N = 23  # 2^23 amplitudes: a launch per pass


def haar(rng):
    z = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
    u, r = np.linalg.qr(z)
    return torch.from_numpy(np.ascontiguousarray((u * (np.diag(r) / np.abs(np.diag(r)))).T.reshape(-1))).cuda()


def axes(bits):  # bit 0 is the innermost axis
    return [N - 1 - b for b in bits]


# target bits (a0 a1 b0 b1) of each pass
@pytest.mark.parametrize("passes,perm,offset", [
    ([(9, 5, 20, 3), (0, 9, 17, 4), (12, 0, 7, 9), (5, 8, 0, 22), (9, 5, 10, 0)], None, 0),
    ([(9, 5, 20, 3), (1, 9, 17, 4), (12, 8, 7, 1), (5, 2, 11, 22), (2, 5, 10, 19)], None, 0),
    ([(0, 5, 20, 3), (1, 0, 17, 4), (12, 2, 7, 0), (2, 1, 0, 22), (3, 2, 1, 0), (8, 1, 2, 9)], None, 0),
    ([(9, 5, 20, 3), (0, 9, 17, 4), (3, 0, 1, 2), (5, 8, 0, 22)], None, 1),
    ([(9, 5, 20, 3), (0, 9, 17, 4), (5, 8, 0, 22)], "swap0", 0),
    ([(9, 5, 20, 3), (4, 9, 17, 6), (5, 8, 0, 22)], "swap0", 0),
    ([(9, 5, 20, 3), (0, 9, 17, 4), (5, 8, 2, 22)], "high", 1),
])
def test_low_targets(passes, perm, offset):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    rng = np.random.default_rng(len(passes) + offset)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    buf = torch.randn(2 ** N + 2, dtype=torch.complex128, device="cuda", generator=gen)
    psi = buf[offset:offset + 2 ** N]
    psi /= torch.linalg.vector_norm(psi)
    ref, scratch = psi.clone(), torch.empty(2 ** N + 2, dtype=torch.complex128, device="cuda")[offset:offset + 2 ** N]
    gates = [(axes(b[:2]), axes(b[2:]), haar(rng), haar(rng)) for b in passes]
    flat = [g for a, b, ga, gb in gates for g in ((a, ga), (b, gb))]
    pt = None
    if perm is not None:  # after the second pass
        pt = list(range(N))
        i, j = (N - 1, N - 5) if perm == "swap0" else (0, 7)
        pt[i], pt[j] = j, i
    dims, old = [2] * N, q.get_arithmetic()
    try:
        q.set_arithmetic(q.ARITH_FP64)
        for k, (t, g) in enumerate(flat):
            q.apply_gate(ref, dims, t, g)
            if pt is not None and k == 3:
                ref = q.permute(ref, dims, pt)
        q.set_arithmetic(q.ARITH_BF16X6)
        q.take_device_errors()
        runs = [(flat, None)] if pt is None else [(flat[:4], pt), (flat[4:], None)]
        out = q.apply_gate_runs(psi, scratch, dims, runs)
        torch.cuda.synchronize()
        assert q.take_device_errors() == 0
    finally:
        q.set_arithmetic(old)
    assert torch.linalg.vector_norm(out - ref) < 1e-12 * torch.linalg.vector_norm(ref)
