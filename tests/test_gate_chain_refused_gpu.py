"""Runs of fused gate pairs where the launch that all passes share is refused (a context with a share of the
SMs cannot hold it as a whole, and its CTAs wait for one another) or there is no memory for its tables:
the passes go one by one and give the same bits. The refusals are made on the host: the
library's own objects linked with a cudaLaunchCooperativeKernel and a cudaMallocAsync that return
the errors."""
import glob
import importlib.util
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q
from qtnh_gb300 import build as b

pytestmark = pytest.mark.gpu

FAKE = """
#include <cuda_runtime.h>
static int calls = 0, memory = 0;
extern "C" int fake_calls() { return calls; }
extern "C" void fake_memory(int on) { memory = on; }
extern "C" cudaError_t __wrap_cudaLaunchCooperativeKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) {
  ++calls;
  return cudaErrorCooperativeLaunchTooLarge;
}
extern "C" cudaError_t __real_cudaMallocAsync(void**, size_t, cudaStream_t);
extern "C" cudaError_t __wrap_cudaMallocAsync(void** p, size_t bytes, cudaStream_t s) {
  if (memory && bytes > 32768) {
    ++calls;
    return cudaErrorMemoryAllocation;
  }
  return __real_cudaMallocAsync(p, bytes, s);
}
"""


@pytest.fixture(scope="module")
def refusing(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    d = tmp_path_factory.mktemp("refusing")
    src, so = d / "fake.cpp", d / "libqtnh_cuda_refusing.so"
    src.write_text(FAKE)
    objs = sorted(glob.glob(os.path.join(b.BUILD, "*.cu.o")) + glob.glob(os.path.join(b.BUILD, "plan.cpp.o")))
    subprocess.run([b._nvcc(), "-shared", "-gencode", "arch=compute_103a,code=sm_103a", "-Xcompiler", "-fPIC", "-Xlinker",
                    "--wrap=cudaLaunchCooperativeKernel", "-Xlinker", "--wrap=cudaMallocAsync", "-o", str(so), str(src)] + objs, check=True)
    spec = importlib.util.spec_from_file_location("qtnh_refusing", q.__file__)
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    m.LIB_PATH = str(so)
    return m


def haar(rng):
    z = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
    u, r = np.linalg.qr(z)
    return torch.from_numpy(np.ascontiguousarray((u * (np.diag(r) / np.abs(np.diag(r)))).T.reshape(-1))).cuda()


@pytest.mark.parametrize("what", ["launch", "memory"])
@pytest.mark.parametrize("n,pairs,perms", [(12, 5, ()), (12, 9, (2, 6)), (20, 5, (1, 2)), (11, 70, (66,))])
def test_refused(refusing, n, pairs, perms, what):
    rng = np.random.default_rng(n + pairs)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    psi = torch.randn(2 ** n, dtype=torch.complex128, device="cuda", generator=g)
    psi /= torch.linalg.vector_norm(psi)
    runs, gates = [], []
    for k in range(pairs):
        t = [int(x) for x in rng.choice(n, size=4, replace=False)]
        gates += [(t[:2], haar(rng)), (t[2:], haar(rng))]
        if k in perms:
            runs.append((gates, [int(x) for x in rng.permutation(n)]))
            gates = []
    runs.append((gates, None))
    refusing.lib().fake_memory(1 if what == "memory" else 0)
    outs, calls = [], refusing.lib().fake_calls()
    for m in (q, refusing):
        old = m.get_arithmetic()
        m.set_arithmetic(m.ARITH_BF16X6)
        m.take_device_errors()
        st = psi.clone()
        m.gate_timing(True)
        outs.append(m.apply_gate_runs(st, torch.empty_like(st), [2] * n, runs))
        assert m.gate_timing(False)[1] == pairs  # every pass counted once
        assert m.take_device_errors() == 0
        m.set_arithmetic(old)
    assert refusing.lib().fake_calls() == calls + (2 if pairs > 65 else 1)
    assert torch.equal(torch.view_as_real(outs[0]), torch.view_as_real(outs[1]))
