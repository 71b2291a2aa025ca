"""Lone gates and diagonals on states of any extents: the float-float kernels in packed FP32
(gate_kernel_f32x2, diag_kernel_f32x2, layer_apply_kernel_f32x2) where their index forms,
remainders and fall-backs change: extents that are powers of two, odd and mixed; targets first,
last and out of order; states smaller than a block, not a multiple of a thread's step and of
several steps of the ring; diagonals split by each block (up to 256 entries) and ahead (above);
elements outside the split range. Against numpy in complex128. Float-float keeps 46 bits, and an
element is a sum of at most 9 products: 9 * 2^-46 = 1.3e-13 of the largest product; the bar is
1e-12 of the largest magnitude, the plain complex128 one."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.fixture(scope="module", autouse=True)
def _setup():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    q.lib()


@pytest.fixture(params=[q.ARITH_F32X2, q.ARITH_BF16X6], ids=["f32x2", "bf16x6"])
def arith(request):
    old = q.get_arithmetic()
    q.set_arithmetic(request.param)
    yield request.param
    q.set_arithmetic(old)


def state(rng, dims, scale):
    x = rng.standard_normal(dims) + 1j * rng.standard_normal(dims)
    if scale == "range":  # one element beyond the split range, one zero
        f = x.reshape(-1)
        f[len(f) // 3] *= 1e40
        f[0] = 0
    return x


def run(x, f):
    t = torch.from_numpy(np.ascontiguousarray(x).reshape(-1)).cuda()
    f(t)
    torch.cuda.synchronize()
    return t.cpu().numpy().reshape(x.shape)


def close(out, ref):
    assert np.max(np.abs(out - ref)) <= TOL * np.max(np.abs(ref))


@pytest.mark.parametrize("scale", ["unit", "range"])
@pytest.mark.parametrize("dims,targets", [([2], [0]), ([2, 257], [0]), ([257, 2], [1]), ([2] * 15, [7]),
                                          ([3, 5, 7, 11], [0]), ([5, 7, 3], [2]), ([3] * 9, [8, 0]), ([3] * 11, [3, 4]),
                                          ([3, 3], [1, 0]), ([9, 129], [0]), ([1, 5, 4, 6], [2]), ([2, 3, 2, 65], [2, 0]),
                                          ([1, 77], [0])])
def test_lone_gate_any_extents(dims, targets, scale, arith):
    rng = np.random.default_rng(sum(dims) * 31 + len(dims) + targets[0])
    td = [dims[t] for t in targets]
    D = int(np.prod(td))
    u = np.linalg.qr(rng.standard_normal((D, D)) + 1j * rng.standard_normal((D, D)))[0]
    x = state(rng, dims, scale)
    gate = torch.from_numpy(np.ascontiguousarray(u)).reshape(-1).cuda()  # elements [in, out]
    out = run(x, lambda t: q.apply_gate(t, dims, targets, gate))
    m = np.moveaxis(x, targets, range(len(targets)))
    ref = np.moveaxis((u.T @ m.reshape(D, -1)).reshape(m.shape), range(len(targets)), targets)
    close(out, ref)


@pytest.mark.parametrize("scale", ["unit", "range"])
@pytest.mark.parametrize("dims,targets", [([2], [0]), ([2] * 14, [13, 2]), ([2] * 17, list(range(8))), ([3] * 9, [8, 0]),
                                          ([3, 5, 7, 11], [2, 0]), ([7, 1, 300], [2]), ([16, 17, 61], [1, 0]),
                                          ([767], [0]), ([4, 769], []), ([3, 256, 1031], [1])])
def test_diagonal_any_extents(dims, targets, scale, arith):
    rng = np.random.default_rng(sum(dims) * 17 + len(targets))
    td = [dims[t] for t in targets]
    d = np.exp(1j * rng.uniform(0, 6.28, td))
    x = state(rng, dims, scale)
    dd = torch.from_numpy(np.ascontiguousarray(d).reshape(-1)).cuda()
    out = run(x, lambda t: q.apply_diag(t, dims, targets, dd))
    shape = [1] * len(dims)
    for t in targets:
        shape[t] = dims[t]
    ref = x * np.transpose(d, np.argsort(targets)).reshape(shape) if targets else x * d
    close(out, ref)


@pytest.mark.parametrize("scale", ["unit", "range"])
@pytest.mark.parametrize("dims,axes", [([2] * 16, list(range(16))), ([2] * 13, [12, 0, 5]), ([3] * 11, list(range(11))),
                                       ([5000, 3], [0, 1]), ([3, 5, 7, 11, 13], [4, 2, 0]), ([2], [0]), ([6, 1, 5], [2, 1])])
def test_diagonal_layer_any_extents(dims, axes, scale, arith):
    rng = np.random.default_rng(sum(dims) * 13 + len(axes))
    fac = [np.exp(1j * rng.uniform(0, 6.28, dims[a])) for a in axes]
    x = state(rng, dims, scale)
    ff = torch.from_numpy(np.concatenate(fac)).cuda()
    out = run(x, lambda t: q.apply_diag_layer(t, dims, axes, ff))
    ref = x
    for a, f in zip(axes, fac):
        shape = [1] * len(dims)
        shape[a] = dims[a]
        ref = ref * f.reshape(shape)
    close(out, ref)


# Entries that are exactly 1 (kept as they are where whole warps share them): targets above and
# among the lowest five bits, more and fewer ones than a quarter, and an entry next to 1.
@pytest.mark.parametrize("n,targets", [(5, [0]), (6, [0]), (12, [1, 4]), (12, [6, 7]), (13, [0, 12]), (16, [3, 0, 9]), (14, [])])
@pytest.mark.parametrize("ones", ["phase", "most", "few", "next", "all"])
def test_diagonal_with_ones(n, targets, ones, arith):
    rng = np.random.default_rng(n + len(targets))
    m = 2 ** len(targets)
    d = np.exp(1j * rng.uniform(0.1, 6.2, m))
    if ones == "phase":
        d[:-1] = 1
    elif ones == "most":
        d[1:] = 1
    elif ones == "few":
        d[0] = 1
    elif ones == "next":
        d[:] = 1 + 2.0 ** -52
    else:
        d[:] = 1
    x = state(rng, [2] * n, "unit")
    bad = x.copy()
    bad.reshape(-1)[2 ** n // 2] = complex(np.inf, 1)
    bad.reshape(-1)[2 ** n // 2 + 1] = complex(1, np.nan)
    td = torch.from_numpy(d).cuda()
    f = np.ones([2] * n, dtype=np.complex128)
    shape = [1] * n
    for t in targets:
        shape[t] = 2
    f = f * (np.transpose(d.reshape([2] * len(targets)), np.argsort(targets)).reshape(shape) if targets else d)
    close(run(x, lambda t: q.apply_diag(t, [2] * n, targets, td)), x * f)
    out = run(bad, lambda t: q.apply_diag(t, [2] * n, targets, td))
    with np.errstate(invalid="ignore"):
        ref = bad * f
    fin = np.isfinite(ref)
    assert np.array_equal(np.isfinite(out), fin)
    close(out[fin], ref[fin])
