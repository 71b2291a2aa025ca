"""Reduced density matrices where there is no memory for the blocks' sums: they are added in place, as
the call did before it had a workspace, in another order (FP64 sums of 2^(n-4) terms: the bar is
1e-13 of the largest entry). Entries that are not finite stay so. The allocation is refused on the
host: the library's own objects linked with a cudaMallocAsync that returns the error."""
import glob
import importlib.util
import os
import subprocess

import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q
from qtnh_gb300 import build as b

pytestmark = pytest.mark.gpu

FAKE = """
#include <cuda_runtime.h>
static int calls = 0;
extern "C" int fake_calls() { return calls; }
extern "C" cudaError_t __wrap_cudaMallocAsync(void**, size_t, cudaStream_t) {
  ++calls;
  return cudaErrorMemoryAllocation;
}
"""


@pytest.fixture(scope="module")
def refusing(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    d = tmp_path_factory.mktemp("refusing")
    src, so = d / "fake.cpp", d / "libqtnh_cuda_no_memory.so"
    src.write_text(FAKE)
    objs = sorted(glob.glob(os.path.join(b.BUILD, "*.cu.o")) + glob.glob(os.path.join(b.BUILD, "plan.cpp.o")))
    subprocess.run([b._nvcc(), "-shared", "-gencode", "arch=compute_103a,code=sm_103a", "-Xcompiler", "-fPIC", "-Xlinker",
                    "--wrap=cudaMallocAsync", "-o", str(so), str(src)] + objs, check=True)
    spec = importlib.util.spec_from_file_location("qtnh_no_memory", q.__file__)
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    m.LIB_PATH = str(so)
    return m


@pytest.mark.parametrize("precision", [q.STATE_C128, q.STATE_C64])
@pytest.mark.parametrize("n,qubits", [(4, [3, 0, 2, 1]), (11, [0, 10, 4, 7]), (19, [18, 2, 3, 5])])
@pytest.mark.parametrize("finite", [True, False])
def test_sums_in_place(refusing, n, qubits, precision, finite):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    psi = torch.randn(2**n, dtype=torch.complex128, device="cuda", generator=g) * 2 ** (-n / 2)
    psi = psi.to(torch.complex64 if precision == q.STATE_C64 else torch.complex128)
    if not finite:
        psi[2**n // 3] = float("inf")
    calls = refusing.lib().fake_calls()
    rho, ref = refusing.rdm4(precision, psi, n, qubits), q.rdm4(precision, psi, n, qubits)
    assert refusing.lib().fake_calls() == calls + 1
    a, c = torch.view_as_real(rho), torch.view_as_real(ref)
    assert torch.equal(a.isfinite(), c.isfinite()) and torch.equal(a.isnan(), c.isnan())
    ok = c.isfinite()
    assert (a[ok] - c[ok]).abs().max() < 1e-13 * c[ok].abs().max()
