"""States of 2^31 elements and more: the index forms that smaller ones never take (gates with 64-bit
offsets; diagonals by the 32-bit division that keeps its carry, 2^31 to 2^32 elements, and with
64-bit indices, by shifts and by divisions). A state whose elements follow from their index, checked
at the first and last elements, around 2^31 and 2^32 and at random ones. Tolerance: float-float
keeps 46 bits, a gate sums at most 9 products; the bar is the plain complex128 one, 1e-12 of the
largest magnitude (below 1)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu


def value(e):
    return torch.complex(((e * 2654435761) % 1000003).double() / 1000003 - 0.5,
                         ((e * 40503 + 77) % 999983).double() / 999983 - 0.5)


def fill(x):
    for s in range(0, x.numel(), 1 << 27):
        x[s:s + (1 << 27)] = value(torch.arange(s, min(x.numel(), s + (1 << 27)), device="cuda"))


@pytest.mark.parametrize("dims", [[3] * 20, [2] * 32, [5] * 14], ids=["3^20", "2^32", "5^14"])
def test_states_beyond_31_bits(dims):
    n = int(np.prod(dims, dtype=np.int64))
    if torch.cuda.mem_get_info()[0] < 16 * n + (8 << 30):
        pytest.skip("not enough device memory")
    strides = [int(np.prod(dims[i + 1:], dtype=np.int64)) for i in range(len(dims))]
    g = torch.Generator(device="cuda")
    g.manual_seed(n % 1000)
    e = torch.cat([torch.randint(0, n, (1 << 17,), device="cuda", generator=g)] +
                  [torch.arange(max(0, c - 1024), min(n, c + 1024), device="cuda") for c in (0, n, 1 << 31, 1 << 32) if c <= n])
    x = torch.empty(n, dtype=torch.complex128, device="cuda")
    last = len(dims) - 1
    digit = lambda e, i: (e // strides[i]) % dims[i]
    close = lambda ref: (x[e] - ref).abs().max().item() < 1e-12
    rng = np.random.default_rng(7)
    for targets in ([0, 1], [last, 2], [0, 3, 5, last]):
        d = torch.from_numpy(np.exp(1j * rng.uniform(0, 6.28, [dims[t] for t in targets]))).cuda()
        for arith in (q.ARITH_FP64, q.ARITH_F32X2, q.ARITH_BF16X6):
            old = q.get_arithmetic()
            q.set_arithmetic(arith)
            try:
                fill(x)
                q.apply_diag(x, dims, targets, d.reshape(-1))
            finally:
                q.set_arithmetic(old)
            assert close(value(e) * d[tuple(digit(e, t) for t in targets)])
    phases = torch.from_numpy(np.exp(1j * rng.uniform(0, 6.28, sum(dims)))).cuda()
    fill(x)
    q.apply_diag_layer(x, dims, list(range(len(dims))), phases)
    ref = value(e)
    for i in range(len(dims)):
        ref = ref * phases[sum(dims[:i]) + digit(e, i)]
    assert close(ref)
    for targets in ([3], [last, 0] if dims[0] < 4 else [last]):
        td = [dims[t] for t in targets]
        D = int(np.prod(td))
        u = torch.from_numpy(np.linalg.qr(rng.standard_normal((D, D)) + 1j * rng.standard_normal((D, D)))[0].copy()).cuda()
        fill(x)
        if D in (2, 3, 4, 9):  # (others go out of a copy of the state)
            q.apply_gate(x, dims, targets, u.reshape(-1))
            base, out = e.clone(), torch.zeros_like(e)
            for t in targets:
                base = base - digit(e, t) * strides[t]
                out = out * dims[t] + digit(e, t)
            ref = torch.zeros(len(e), dtype=torch.complex128, device="cuda")
            for c, multi in enumerate(np.ndindex(*td)):
                ref += u[c][out] * value(base + sum(int(m) * strides[t] for m, t in zip(multi, targets)))
            assert close(ref)
    del x
    torch.cuda.empty_cache()
