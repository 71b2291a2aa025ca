"""Runs of fused gate pairs recorded into a CUDA graph and replayed: the replay reads nothing but device
memory and the launches' own arguments, so it gives the bits of the call, whatever the host has done
since. Sizes with all passes in one launch (12, 20 qubits) and with a launch per pass (23), without
permutations and with two that are folded into passes. And on two streams from two host threads at
once, beside a contraction on a third: the bits of the calls one after the other."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _setup():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    old = q.get_arithmetic()
    q.set_arithmetic(q.ARITH_BF16X6)
    q.take_device_errors()
    yield
    q.set_arithmetic(old)


def haar(rng):
    z = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
    u, r = np.linalg.qr(z)
    return torch.from_numpy(np.ascontiguousarray((u * (np.diag(r) / np.abs(np.diag(r)))).T.reshape(-1))).cuda()


def make(n, pairs, perms, seed):
    """A state and runs of `pairs` pairs, permutations after the passes `perms` (an even number)."""
    rng = np.random.default_rng(seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    psi = torch.randn(2 ** n, dtype=torch.complex128, device="cuda", generator=g)
    psi /= torch.linalg.vector_norm(psi)
    runs, gates = [], []
    for k in range(pairs):
        t = [int(x) for x in rng.choice(n, size=4, replace=False)]
        gates += [(t[:2], haar(rng)), (t[2:], haar(rng))]
        if k in perms:
            runs.append((gates, [int(x) for x in rng.permutation(n)]))
            gates = []
    return psi, runs + [(gates, None)]


@pytest.mark.parametrize("n,pairs", [(12, 2), (12, 7), (20, 3), (20, 7), (23, 4)])
@pytest.mark.parametrize("perms", [(), (1, 2)], ids=["plain", "permuted"])
def test_replayed_graph(n, pairs, perms):
    perms = perms if pairs > 2 else ((0, 1) if perms else ())
    psi, runs = make(n, pairs, perms, n + pairs)
    dims = [2] * n
    ref = psi.clone()
    scratch = torch.empty_like(psi)
    for _ in range(2):
        ref = q.apply_gate_runs(ref, scratch, dims, runs)
    state = psi.clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        assert q.apply_gate_runs(state, scratch, dims, runs) is state
    make(10, 12, (3, 5), 1)  # the host goes on
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert q.take_device_errors() == 0
    assert torch.equal(torch.view_as_real(state), torch.view_as_real(ref))


def test_two_streams_from_two_threads():
    rng = np.random.default_rng(3)
    jobs = []
    for n, pairs, perms in ((12, 9, (2, 5)), (20, 6, ()), (16, 3, (0, 1)), (22, 5, ())):
        psi, runs = make(n, pairs, perms, 7 * n)
        ref, scratch = psi.clone(), torch.empty_like(psi)
        for _ in range(6):
            ref = q.apply_gate_runs(ref, scratch, [2] * n, runs)
        jobs.append((n, runs, psi, ref))
    a = torch.from_numpy(rng.standard_normal((512, 512)) + 1j * rng.standard_normal((512, 512))).cuda()
    A = q.Tensor(q.DENSE, [], [512, 512], a.reshape(-1))
    prod = q.contract(A, A, [(1, 0)])[0].data
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(3)]
    out, errors = {}, []

    def gates(s, mine):
        try:
            with torch.cuda.stream(streams[s]):
                for j in mine:
                    n, runs, psi, _ = jobs[j]
                    st, scratch = psi.clone(), torch.empty_like(psi)
                    for _ in range(6):
                        q.apply_gate_runs(st, scratch, [2] * n, runs)
                    out[j] = (st, scratch)
                streams[s].synchronize()
        except Exception as e:  # reported by the test, not by the thread
            errors.append(e)

    threads = [threading.Thread(target=gates, args=(0, (0, 1))), threading.Thread(target=gates, args=(1, (3, 2)))]
    for t in threads:
        t.start()
    res = []
    with torch.cuda.stream(streams[2]):
        for _ in range(20):
            res.append(q.contract(A, A, [(1, 0)])[0].data)
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    assert q.take_device_errors() == 0
    for j, (_, _, _, ref) in enumerate(jobs):
        assert torch.equal(torch.view_as_real(out[j][0]), torch.view_as_real(ref)), j
    for r in res:
        assert torch.equal(torch.view_as_real(r), torch.view_as_real(prod))
