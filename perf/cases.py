"""Performance cases: the work a user of this framework has it do, through its public
entry points (the Python binding of the C ABI), over the range of sizes it is used at.

Every case is a dict of plain values. `prepare` makes what a program holds before the call
(device states, gates, plans), `run` is one pass, `work` the bytes and operations that
pass cannot do without, `exact` the outputs of the first pass in 64-bit arithmetic by plain
torch. States are updated in place, as the engine's in-place contractions are, so a second
pass continues from the first one's result; every operation on a state is unitary.
"""
import cmath
import math

import numpy as np
import torch

import qtnh_gb300 as q
from qtnh_gb300 import workload as wl
from qtnh_gb300.circuit import DeviceCircuit


def listed():
    return [
        # A small simulation: the random layered circuit on 12 qubits (64 KiB state), all of
        # its 40 layers in one runner call. Launches and their latency are the cost.
        {"name": "circuit_n12", "kind": "circuit", "n": 12, "depth": 40},
        # The same circuit family at an everyday size (16 MiB state, resident in L2).
        {"name": "circuit_n20", "kind": "circuit", "n": 20, "depth": 40},
        # The headline size, 2^28 complex128 amplitudes (4 GiB): one period of the headline
        # circuit, eight layers with two phase layers and one redistribution.
        {"name": "circuit_n28", "kind": "circuit", "n": 28, "depth": 8},
        # The 16-qubit quantum Fourier transform, one Tensor::contract call per gate: Hadamards,
        # controlled phases and the final swaps. The smallest calls a program makes.
        {"name": "qft_n16", "kind": "qft", "n": 16},
        # Gates that come alone (no neighbour to fuse with) on a large state, one on each of
        # one, two, three and four qubits.
        {"name": "lone_gates_n26", "kind": "gates", "n": 26},
        # Qutrits: a state whose axes are not powers of two; one- and two-qutrit gates, a
        # two-qutrit diagonal and a permutation.
        {"name": "qutrits_n14", "kind": "qudits", "d": 3, "n": 14},
        # Data movement and streaming on a large state: a controlled phase, a layer of phases
        # on every qubit, a swap of the outermost axes, a redistribution of the top three.
        {"name": "streaming_n27", "kind": "streaming", "n": 27},
        # A small dense contraction as tensor networks have by the hundred, odd dimensions.
        {"name": "dense_small", "kind": "dense", "dims1": "5x7x9x11", "dims2": "9x13x5x3",
         "wires": "0-2 2-0", "precision": "oz6"},
        # A dense pair of the precision study's shape (wired indices at scattered positions) in
        # the default, FP64-accurate arithmetic: M 4096, N 2048, K 1024.
        {"name": "dense_oz6", "kind": "dense", "dims1": "32x16x64x64x2", "dims2": "64x2x16x64x16",
         "wires": "1-2 3-0", "precision": "oz6"},
        # A pair of the same study in split precision (BF16x3): M 4096, N 8192, K 2048.
        {"name": "dense_bf16x3", "kind": "dense", "dims1": "64x32x16x64x4", "dims2": "64x32x16x64x4",
         "wires": "1-1 3-0", "precision": "bf16x3"},
        # Many independent circuits of uneven size in one compiled batch, mixed precision, with
        # 64 amplitudes queried of each.
        {"name": "batch_mixed", "kind": "batch", "count": 64, "n_lo": 10, "n_hi": 22, "d_lo": 8, "d_hi": 16,
         "precision": "c64"},
        # One round of the request loop over resident states of uneven size: four layers for
        # every state (the last with phases and a qubit exchange), a renormalisation, and the
        # answers (256 amplitudes or a 4-qubit reduced density matrix).
        {"name": "serve_mixed", "kind": "serve", "count": 16, "n_lo": 12, "n_hi": 24, "layers": 4, "precision": "c64"},
    ]


def _dense_shape(case):
    """(dims1, dims2, wires) of a dense case: dims as "5x7", wires as "0-2 2-0"."""
    return ([int(d) for d in case["dims1"].split("x")], [int(d) for d in case["dims2"].split("x")],
            [tuple(int(i) for i in w.split("-")) for w in case["wires"].split()])


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["circuit", "circuit", "qft", "gates", "qudits", "streaming", "dense", "dense", "dense", "batch",
                       "serve"])
    if kind == "circuit":
        n = rng.randint(8, 28)
        return {"kind": kind, "n": n, "depth": rng.randint(1, 8 if n > 26 else 40)}
    if kind in ("qft", "gates", "streaming"):
        return {"kind": kind, "n": rng.randint(6, 22) if kind == "qft" else rng.randint(12, 27)}
    if kind == "qudits":
        d = rng.choice([3, 5, 6, 7])
        return {"kind": kind, "d": d, "n": rng.randint(4, int(math.log(2 ** 24) / math.log(d)))}
    if kind == "dense":
        # sizes log-uniform, each split into one to three axes; odd ones among them
        while True:
            sizes = []
            for _ in range(3):
                axes = [_logint(rng, 2, 64) for _ in range(rng.randint(1, 3))]
                if rng.random() < 0.5:
                    axes = [2 ** int(round(math.log2(a))) for a in axes]
                sizes.append(axes)
            m, n, k = (math.prod(a) for a in sizes)
            if max(m * k, k * n, m * n) <= 2 ** 24 and 2 ** 12 <= m * n * k <= 2 ** 35:
                break
        d1, p1 = _shuffled(rng, sizes[0] + sizes[2])
        d2, p2 = _shuffled(rng, sizes[1] + sizes[2])
        wires = [[p1[len(sizes[0]) + j], p2[len(sizes[1]) + j]] for j in range(len(sizes[2]))]
        return {"kind": kind, "dims1": "x".join(map(str, d1)), "dims2": "x".join(map(str, d2)),
                "wires": " ".join("%d-%d" % tuple(w) for w in wires),
                "precision": rng.choice(["oz6", "oz6", "bf16x3", "fp64"] if m * n * k <= 2 ** 30 else ["oz6", "bf16x3"])}
    lo = rng.randint(8, 14)
    hi = rng.randint(lo, 21)
    if kind == "batch":
        return {"kind": kind, "count": _logint(rng, 2, 64), "n_lo": lo, "n_hi": hi, "d_lo": 2, "d_hi": rng.randint(2, 16),
                "precision": rng.choice(["c64", "c64", "c128"])}
    return {"kind": kind, "count": _logint(rng, 1, 24), "n_lo": lo, "n_hi": hi, "layers": rng.randint(1, 8),
            "precision": rng.choice(["c64", "c64", "c128"])}


def _shuffled(rng, dims):
    """The dims in a random order and the new position of each."""
    order = list(range(len(dims)))
    rng.shuffle(order)
    pos = [0] * len(dims)
    for new, old in enumerate(order):
        pos[old] = new
    return [dims[i] for i in order], pos


# ---- inputs ---------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _random_state(size, gen):
    """I.i.d. complex Gaussian amplitudes of unit norm."""
    psi = torch.randn(size, dtype=torch.complex128, device="cuda", generator=gen)
    psi /= torch.linalg.vector_norm(psi)
    return psi


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.complex128).reshape(-1)).cuda()


def _circuit(case, seed):
    return wl.random_circuit(case["n"], case["depth"], seed=seed)


def _lone_gates(case, seed):
    """[(targets, SymmTensor elements)]: one gate on each of 1, 2, 3 and 4 random qubits."""
    rng = np.random.default_rng(seed)
    out = []
    for k in (1, 2, 3, 4):
        targets = [int(x) for x in rng.choice(case["n"], size=k, replace=False)]
        out.append((targets, wl.gate_elements(wl.haar_unitary(rng, 2 ** k))))
    return out


def _qudit_ops(case, seed):
    """Gates on one and two qudits, a two-qudit diagonal and a permutation."""
    rng = np.random.default_rng(seed)
    d, n = case["d"], case["n"]
    t1 = [int(rng.integers(n))]
    t2 = [int(x) for x in rng.choice(n, size=2, replace=False)]
    t3 = [int(x) for x in rng.choice(n, size=2, replace=False)]
    return {"one": (t1, wl.gate_elements(wl.haar_unitary(rng, d))),
            "two": (t2, wl.gate_elements(wl.haar_unitary(rng, d * d))),
            "diag": (t3, np.exp(1j * rng.uniform(0, 2 * math.pi, d * d))),
            "ptup": [int(x) for x in rng.permutation(n)]}


def _streaming_ops(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    pair = [int(x) for x in rng.choice(n, size=2, replace=False)]
    ptup = list(range(n))
    local = rng.choice(np.arange(3, n), size=3, replace=False)
    for k in range(3):
        ptup[k], ptup[int(local[k])] = int(local[k]), k
    return {"pair": pair, "cphase": np.array([1, 1, 1, cmath.exp(1j * math.pi / 8)]),
            "phases": rng.uniform(0.0, 2.0 * math.pi, n), "ptup": ptup}


def _spread(lo, hi, i, count):
    """The i-th of `count` sizes spread evenly over lo .. hi."""
    return lo + (hi - lo + 1) * i // count if count > 1 else hi


def _batch_circuits(case, seed):
    """[(circuit, 64 query indices)]: qubits spread over n_lo .. n_hi, depths over d_lo .. d_hi in
    another order; phases after every 4th layer, now and then an exchange of two qubits."""
    rng = np.random.default_rng(seed)
    count, out = case["count"], []
    for i in range(count):
        n = _spread(case["n_lo"], case["n_hi"], i, count)
        depth = _spread(case["d_lo"], case["d_hi"], (i * 7 + 3) % count, count)
        us = wl.haar_unitaries(rng, depth * (n // 2), 4)
        c = wl.Circuit(n)
        for li in range(depth):
            order = [int(x) for x in rng.permutation(n)]
            layer = wl.Layer([(order[2 * j], order[2 * j + 1]) for j in range(n // 2)],
                             [wl.gate_elements(u) for u in us[li * (n // 2):(li + 1) * (n // 2)]])
            if (li + 1) % 4 == 0:
                layer.phases = rng.uniform(0.0, 2.0 * math.pi, n)
            if li % 4 == 1:
                layer.ptup = list(range(n))
                layer.ptup[order[0]], layer.ptup[order[-1]] = order[-1], order[0]
            c.layers.append(layer)
        out.append((c, rng.integers(0, 2 ** n, size=64, dtype=np.uint64)))
    return out


def _serve_qubits(case):
    """Qubit counts of the resident states, log-uniform over n_lo .. n_hi."""
    lo, hi, count = math.log(case["n_lo"]), math.log(case["n_hi"]), case["count"]
    return [int(round(math.exp(lo + (hi - lo) * (i + 0.5) / count))) for i in range(count)]


def _serve_requests(case, seed):
    """[(n, layers, query)]: a layer is (pairs, gates, phases or None, exchange or None); the
    query is 256 amplitude indices or 4 qubits, in turn."""
    rng = np.random.default_rng(seed)
    out = []
    for i, n in enumerate(_serve_qubits(case)):
        layers = []
        for li in range(case["layers"]):
            order = [int(x) for x in rng.permutation(n)]
            pairs = [(order[2 * j], order[2 * j + 1]) for j in range(n // 2)]
            gates = [wl.gate_elements(u) for u in wl.haar_unitaries(rng, n // 2, 4)]
            last = (li + 1) % 4 == 0
            layers.append((pairs, gates, rng.uniform(0.0, 2.0 * math.pi, n) if last else None,
                           (order[0], order[-1]) if last else None))
        if i % 2 == 0:
            query = ("amps", rng.integers(0, 2 ** n, size=256, dtype=np.uint64))
        else:
            query = ("rdm", np.sort(rng.choice(n, size=4, replace=False)).astype(np.uint16))
        out.append((n, layers, query))
    return out


_STATE = {"c64": q.STATE_C64, "c128": q.STATE_C128}
_GEMM = {"oz6": q.GEMM_OZ6, "bf16x3": q.GEMM_BF16X3, "fp64": q.GEMM_FP64}


def prepare(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    s = {"case": case}
    if kind == "circuit":
        s["circuit"] = DeviceCircuit(_circuit(case, seed))
        s["psi"] = _random_state(2 ** case["n"], gen)
        s["scratch"] = torch.empty_like(s["psi"])
    elif kind == "qft":
        n = case["n"]
        s["state"] = q.Tensor(q.DENSE, [], [2] * n, _random_state(2 ** n, gen))
        s["spare"] = torch.empty_like(s["state"].data)
        r = 2 ** -0.5
        s["h"] = q.Tensor(q.SYMM, [], [2, 2], _dev([r, r, r, -r]))
        s["cp"] = [None] + [q.Tensor(q.DIAG, [], [2] * 4, _dev([1, 1, 1, cmath.exp(1j * math.pi / 2 ** k)]))
                            for k in range(1, n)]
        s["swap"] = q.Tensor(q.SWAP, [], [2] * 4)
    elif kind == "gates":
        s["psi"] = _random_state(2 ** case["n"], gen)
        s["gates"] = [(t, _dev(g)) for t, g in _lone_gates(case, seed)]
    elif kind == "qudits":
        ops = _qudit_ops(case, seed)
        s["psi"] = _random_state(case["d"] ** case["n"], gen)
        s["spare"] = torch.empty_like(s["psi"])
        s["ops"] = {k: (v if k == "ptup" else (v[0], _dev(v[1]))) for k, v in ops.items()}
    elif kind == "streaming":
        ops = _streaming_ops(case, seed)
        s["psi"] = _random_state(2 ** case["n"], gen)
        s["spare"] = torch.empty_like(s["psi"])
        s["pair"], s["ptup"] = ops["pair"], ops["ptup"]
        s["cphase"], s["factors"] = _dev(ops["cphase"]), _dev(wl.phase_factors(ops["phases"]))
    elif kind == "dense":
        dims1, dims2, wires = _dense_shape(case)
        a, b = _dense_operands(case, gen)
        s["a"], s["b"], s["wires"] = q.Tensor(q.DENSE, [], dims1, a), q.Tensor(q.DENSE, [], dims2, b), wires
    elif kind == "batch":
        circuits = _batch_circuits(case, seed)
        b = q.Batch([c.n for c, _ in circuits], precision=_STATE[case["precision"]])
        for i, (c, idx) in enumerate(circuits):
            b.set_state(i, _random_state(2 ** c.n, gen))
            b.add_circuit(i, c, idx)
        b.compile()
        s["batch"] = b
    else:
        s["requests"] = _serve_requests(case, seed)
        s["states"] = [_serve_state(n, case, gen) for n, _, _ in s["requests"]]
    return s


def _dense_operands(case, gen):
    """Gaussian entries scaled by 1 / sqrt(contracted size)."""
    dims1, dims2, wires = _dense_shape(case)
    k = math.prod(dims1[w[0]] for w in wires)
    a = torch.randn(math.prod(dims1), dtype=torch.complex128, device="cuda", generator=gen)
    b = torch.randn(math.prod(dims2), dtype=torch.complex128, device="cuda", generator=gen)
    return a / math.sqrt(k), b / math.sqrt(k)


def _serve_state(n, case, gen):
    psi = _random_state(2 ** n, gen)
    if case["precision"] == "c128":
        return psi
    return q.state_convert(q.STATE_C64, psi, torch.empty(2 ** n, dtype=torch.complex64, device="cuda"))


# ---- one pass -------------------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "circuit":
        out = s["circuit"].run(s["psi"], s["scratch"])
        if out is s["scratch"]:
            s["psi"], s["scratch"] = s["scratch"], s["psi"]
        return out
    if kind == "qft":
        n, st = case["n"], s["state"]
        for i in range(n):
            st = q.contract(st, s["h"], [(i, 0)], out=st.data)[0]
            for j in range(i + 1, n):
                st = q.contract(st, s["cp"][j - i], [(i, 0), (j, 1)], out=st.data)[0]
        for k in range(n // 2):
            before = st.data
            st = q.contract(st, s["swap"], [(k, 0), (n - 1 - k, 1)], out=s["spare"])[0]
            s["spare"] = before
        s["state"] = st
        return st.data
    if kind == "gates":
        dims = [2] * case["n"]
        for targets, gate in s["gates"]:
            q.apply_gate(s["psi"], dims, targets, gate)
        return s["psi"]
    if kind == "qudits":
        dims, ops = [case["d"]] * case["n"], s["ops"]
        q.apply_gate(s["psi"], dims, *ops["one"])
        q.apply_gate(s["psi"], dims, *ops["two"])
        q.apply_diag(s["psi"], dims, *ops["diag"])
        q.permute(s["psi"], dims, ops["ptup"], out=s["spare"])
        s["psi"], s["spare"] = s["spare"], s["psi"]
        return s["psi"]
    if kind == "streaming":
        n = case["n"]
        dims = [2] * n
        q.apply_diag(s["psi"], dims, s["pair"], s["cphase"])
        q.apply_diag_layer(s["psi"], dims, list(range(n)), s["factors"])
        q.swap(s["psi"], dims, 0, n - 1, out=s["spare"])
        q.permute(s["spare"], dims, s["ptup"], out=s["psi"])
        return s["psi"]
    if kind == "dense":
        before = q.get_gemm_precision()
        q.set_gemm_precision(_GEMM[case["precision"]])
        try:
            return q.contract(s["a"], s["b"], s["wires"])[0].data
        finally:
            q.set_gemm_precision(before)
    if kind == "batch":
        s["batch"].run()
        return s["batch"].results()
    return _run_serve(s)


def _run_serve(s):
    case = s["case"]
    precision = _STATE[case["precision"]]
    for li in range(case["layers"]):
        q.group_layer(precision, [(st, n) + layers[li] for st, (n, layers, _) in zip(s["states"], s["requests"])])
    q.group_renorm(precision, [(st, n) for st, (n, _, _) in zip(s["states"], s["requests"])])
    answers = []
    for st, (n, _, (what, arg)) in zip(s["states"], s["requests"]):
        answers.append(q.gather(precision, st, n, arg) if what == "amps" else q.rdm4(precision, st, n, arg))
    return {"answers": answers, "states": s["states"]}


# ---- what a pass cannot do without ------------------------------------------------------

def _gate_flops(size, d):
    """A d x d complex gate on a state of `size` amplitudes: d multiply-adds of 8 flop each."""
    return 8 * d * size


def work(case):
    kind = case["kind"]
    if kind == "circuit":
        n, depth = case["n"], case["depth"]
        flops = depth * (n // 2) * _gate_flops(2 ** n, 4) + (depth // 4) * 6 * 2 ** n
        return {"bytes": 32 * 2 ** n, "flops": flops}
    if kind == "qft":
        n = case["n"]
        # a controlled phase multiplies a quarter of the amplitudes
        return {"bytes": 32 * 2 ** n, "flops": n * _gate_flops(2 ** n, 2) + n * (n - 1) // 2 * 6 * 2 ** (n - 2)}
    if kind == "gates":
        size = 2 ** case["n"]
        return {"bytes": 4 * 32 * size, "flops": sum(_gate_flops(size, 2 ** k) for k in (1, 2, 3, 4))}
    if kind == "qudits":
        d, size = case["d"], case["d"] ** case["n"]
        return {"bytes": 4 * 32 * size, "flops": _gate_flops(size, d) + _gate_flops(size, d * d) + 6 * size}
    if kind == "streaming":
        size = 2 ** case["n"]
        # the controlled phase multiplies a quarter of the amplitudes
        return {"bytes": 4 * 32 * size, "flops": 6 * size + 6 * size // 4}
    if kind == "dense":
        d1, d2, wires = _dense_shape(case)
        k = math.prod(d1[w[0]] for w in wires)
        m, n = math.prod(d1) // k, math.prod(d2) // k
        return {"bytes": 16 * (m * k + k * n + m * n), "flops": 8 * m * n * k}
    amp = 8 if case["precision"] == "c64" else 16
    count = case["count"]
    if kind == "batch":
        sizes = [(_spread(case["n_lo"], case["n_hi"], i, count), _spread(case["d_lo"], case["d_hi"], (i * 7 + 3) % count, count))
                 for i in range(count)]
    else:
        sizes = [(n, case["layers"]) for n in _serve_qubits(case)]
    return {"bytes": sum(2 * amp * 2 ** n for n, _ in sizes),
            "flops": sum(depth * (n // 2) * _gate_flops(2 ** n, 4) for n, depth in sizes)}


# ---- the first pass's outputs in 64 bits -----------------------------------------------

def _apply(psi, dims, targets, els):
    """psi'[.., o, ..] = sum_in els[in, o] psi[.., in, ..] over the target axes."""
    d = math.prod(dims[t] for t in targets)
    els = np.asarray(els, dtype=np.complex128).reshape(d, d)
    x = torch.movedim(psi.reshape(dims), targets, list(range(len(targets))))
    shape = x.shape
    x = x.reshape(d, -1)
    y = torch.empty_like(x)
    for o in range(d):
        torch.mul(x[0], complex(els[0, o]), out=y[o])
        for i in range(1, d):
            y[o].add_(x[i], alpha=complex(els[i, o]))
    del x
    return torch.movedim(y.reshape(shape), list(range(len(targets))), targets).reshape(-1)


def _apply_phases(psi, n, axes, factors):
    """psi *= the product of per-axis diagonals (1, f)."""
    x = psi.clone()
    for a, f in zip(axes, factors):
        x.reshape(2 ** a, 2, -1)[:, 1, :].mul_(complex(f))
    return x


def _permute(psi, dims, ptup):
    order = [0] * len(dims)
    for old, new in enumerate(ptup):
        order[new] = old
    return psi.reshape(dims).permute(order).reshape(-1)


def _merged(n, targets):
    """The state's axes with runs of untouched qubits merged: dims and the targets' positions."""
    dims, pos, last = [], {}, -1
    for t in sorted(targets):
        if t - last > 1:
            dims.append(2 ** (t - last - 1))
        pos[t] = len(dims)
        dims.append(2)
        last = t
    if last < n - 1:
        dims.append(2 ** (n - 1 - last))
    return dims, [pos[t] for t in targets]


def _apply_qubits(psi, n, targets, els):
    dims, pos = _merged(n, targets)
    return _apply(psi, dims, pos, els)


def _swap_qubits(psi, n, a, b):
    dims, (pa, pb) = _merged(n, (a, b))
    return psi.reshape(dims).transpose(pa, pb).reshape(-1)


def _apply_circuit(psi, circuit):
    n = circuit.n
    for layer in circuit.layers:
        for pair, els in zip(layer.pairs, layer.gates):
            psi = _apply_qubits(psi, n, list(pair), els)
        if layer.phases is not None:
            psi = _apply_phases(psi, n, range(n), np.exp(1j * np.asarray(layer.phases)))
        if layer.ptup is not None:
            for a, b in enumerate(layer.ptup):
                if b > a:  # the permutations are disjoint exchanges
                    psi = _swap_qubits(psi, n, a, b)
    return psi


def exact(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    if kind == "circuit":
        return _apply_circuit(_random_state(2 ** case["n"], gen), _circuit(case, seed))
    if kind == "qft":
        n = case["n"]
        return torch.fft.ifft(_random_state(2 ** n, gen), norm="ortho")
    if kind == "gates":
        psi = _random_state(2 ** case["n"], gen)
        for targets, els in _lone_gates(case, seed):
            psi = _apply_qubits(psi, case["n"], targets, els)
        return psi
    if kind == "qudits":
        dims, ops = [case["d"]] * case["n"], _qudit_ops(case, seed)
        psi = _random_state(case["d"] ** case["n"], gen)
        psi = _apply(psi, dims, *ops["one"])
        psi = _apply(psi, dims, *ops["two"])
        t, diag = ops["diag"]
        x = torch.movedim(psi.reshape(dims), t, [0, 1])
        x = x * _dev(diag).reshape([case["d"]] * 2 + [1] * (case["n"] - 2))
        return _permute(torch.movedim(x, [0, 1], t).reshape(-1), dims, ops["ptup"])
    if kind == "streaming":
        n, ops = case["n"], _streaming_ops(case, seed)
        psi = _random_state(2 ** n, gen)
        dims, pos = _merged(n, ops["pair"])
        x = torch.movedim(psi.reshape(dims), pos, [0, 1])
        x[1, 1].mul_(complex(ops["cphase"][3]))
        psi = _apply_phases(psi, n, range(n), np.exp(1j * ops["phases"]))
        psi = _swap_qubits(psi, n, 0, n - 1)
        for a, b in enumerate(ops["ptup"]):
            if b > a:
                psi = _swap_qubits(psi, n, a, b)
        return psi
    if kind == "dense":
        d1, d2, wires = _dense_shape(case)
        a, b = _dense_operands(case, gen)
        return torch.tensordot(a.reshape(d1), b.reshape(d2), dims=([w[0] for w in wires], [w[1] for w in wires])).reshape(-1)
    if kind == "batch":
        out = []
        for c, idx in _batch_circuits(case, seed):
            psi = _apply_circuit(_random_state(2 ** c.n, gen), c)
            out.append(psi[torch.from_numpy(idx.astype(np.int64)).cuda()])
        return torch.cat(out)
    return _exact_serve(case, seed, gen)


def _exact_serve(case, seed, gen):
    answers, states = [], []
    requests = _serve_requests(case, seed)
    initial = []
    for n, _, _ in requests:
        psi = _random_state(2 ** n, gen)
        initial.append(psi if case["precision"] == "c128" else psi.to(torch.complex64).to(torch.complex128))
    for (n, layers, (what, arg)), psi in zip(requests, initial):
        for pairs, gates, phases, swap in layers:
            for pair, els in zip(pairs, gates):
                psi = _apply_qubits(psi, n, list(pair), els)
            if phases is not None:
                psi = _apply_phases(psi, n, range(n), np.exp(1j * phases))
            if swap is not None:
                psi = _swap_qubits(psi, n, *swap)
        psi = psi / torch.linalg.vector_norm(psi)
        states.append(psi)
        if what == "amps":
            answers.append(psi[torch.from_numpy(arg.astype(np.int64)).cuda()])
        else:
            dims, pos = _merged(n, [int(x) for x in arg])
            x = torch.movedim(psi.reshape(dims), pos, [0, 1, 2, 3]).reshape(16, -1)
            answers.append(x @ x.conj().T)
    return {"answers": answers, "states": states}
