"""Runs of fused gate pairs on states whose groups lie further apart than the chain's one digit
scale carries: the passes of the one launch go in FP64, 32 groups a warp, spread over all CTAs. One
CTA, two, as many as a warp's share leaves idle, all SMs with several shares; permutations in between.
Against the oracle, relative to the largest amplitude: FP64 products of 16 terms round below 2e-15 a
pass, the first pass's digits below 1e-14; the bar is the chain's 1e-12."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q
from tests.test_gate_chain_gpu import dev, haar, oracle_runs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,pairs,perms", [(11, 4, ()), (12, 5, (1, 2)), (13, 4, ()), (17, 4, (2,)), (22, 4, (1,))])
def test_wide_states_in_one_launch(n, pairs, perms):
    rng = np.random.default_rng(31 * n + pairs)
    psi = (rng.standard_normal(2**n) + 1j * rng.standard_normal(2**n)) * 2.0 ** (-n / 2)
    psi[5] = 1e9
    runs, gates = [], []
    for k in range(pairs):
        q4 = [int(x) for x in rng.choice(n, size=4, replace=False)]
        gates += [(q4[:2], haar(rng)), (q4[2:], haar(rng))]
        if k in perms:
            runs.append((gates, [int(x) for x in rng.permutation(n)]))
            gates = []
    runs.append((gates, None))
    st, sc = dev(psi), dev(np.zeros_like(psi))
    out = q.apply_gate_runs(st, sc, [2] * n, [([(t, dev(g)) for t, g in gl], pt) for gl, pt in runs])
    assert q.take_device_errors() == 0
    ref, got = oracle_runs(psi, n, runs), out.cpu().numpy()
    assert np.max(np.abs(got - ref)) < 1e-12 * np.max(np.abs(ref))
