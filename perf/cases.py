"""Performance cases: the work a user of the simulator has it do, through its
public entry points, from the smallest circuits to the largest states.

A case is a dict of plain values; its "kind" says which path it takes:

circuit  a Circuit of the default mode (complex128, one gate at a time) run
         from |0...0> with a measure_all: what a q1tsim program does
calls    gates applied one by one through VectorState.apply_gate, as a host
         program bound to the backend's trait does
brick    the random U3/CX brick circuit, the state's amplitudes as the result
qft      the quantum Fourier transform of a random state, in place
shots    sampling of a prepared state (peek_all_into)
midway   measurements and resets in the middle of a circuit, with gates
         conditioned on their results
batch    many small independent circuits in one call
product  a state prepared from single-qubit coefficients
"""
import math

import numpy as np
import torch

from q1tsim_gb300 import Circuit, Rng, VectorState, workloads
from q1tsim_gb300 import gates as G
from q1tsim_gb300.batch import Batch
from q1tsim_gb300.sharded import EngineShard


def listed():
    return [
        # the reference's own benchmark sizes: a small circuit, where each call's latency counts
        {"name": "circuit_10q", "kind": "circuit", "n": 10, "depth": 8, "shots": 1024},
        # the benchmark's 16-qubit circuit of 20 layers and 8192 runs
        {"name": "circuit_16q", "kind": "circuit", "n": 16, "depth": 20, "shots": 8192},
        # a bound host program that applies one gate of any kind per call
        {"name": "calls_13q_c128", "kind": "calls", "n": 13, "gates": 48, "precision": "c128"},
        # the default mode on a state far larger than the caches
        {"name": "brick_26q_c128", "kind": "brick", "n": 26, "depth": 6, "precision": "c128", "width": 0},
        # complex128 with gates fused (as Circuit allows it)
        {"name": "brick_25q_c128_fused", "kind": "brick", "n": 25, "depth": 10, "precision": "c128", "width": 5},
        # complex64 fused, a request of middle size
        {"name": "brick_21q_c64_fused", "kind": "brick", "n": 21, "depth": 30, "precision": "c64", "width": 5},
        # the benchmark's headline circuit
        {"name": "brick_30q_c64_fused", "kind": "brick", "n": 30, "depth": 24, "precision": "c64", "width": 5},
        # the benchmark's QFT on a random state
        {"name": "qft_28q_c64", "kind": "qft", "n": 28, "precision": "c64", "width": 5},
        # a million shots of a large state
        {"name": "shots_29q_c64", "kind": "shots", "n": 29, "shots": 1000000, "precision": "c64"},
        # error-correction style circuits: measure, act on the result, reset
        {"name": "midway_23q_c128", "kind": "midway", "n": 23, "measures": 3, "shots": 4096},
        # independent circuits of uneven sizes with a mid-circuit measurement each
        {"name": "batch_160", "kind": "batch", "circuits": 160, "qmin": 8, "qmax": 17, "dmin": 10, "dmax": 30,
         "shots": 1024},
        # a large state prepared from its qubits' coefficients
        {"name": "product_27q_c128", "kind": "product", "n": 27, "precision": "c128"},
    ]


def draw(rng):
    kind = rng.choice(["circuit", "calls", "brick", "brick", "brick", "qft", "shots", "midway", "batch", "product"])
    if kind == "circuit":
        return {"kind": kind, "n": rng.randint(6, 17), "depth": rng.randint(2, 20), "shots": _log(rng, 100, 10000)}
    if kind == "calls":
        return {"kind": kind, "n": rng.randint(6, 21), "gates": rng.randint(20, 60),
                "precision": rng.choice(["c128", "c64"])}
    if kind == "brick":
        precision, width = rng.choice([("c128", 0), ("c128", 5), ("c64", 5), ("c64", 5)])
        top, deep = {("c128", 0): (26, 6), ("c128", 5): (25, 10), ("c64", 5): (29, 24)}[precision, width]
        n = rng.randint(11, top)
        return {"kind": kind, "n": n, "depth": rng.randint(3, deep), "precision": precision, "width": width}
    if kind == "qft":
        precision = rng.choice(["c64", "c64", "c128"])
        return {"kind": kind, "n": rng.randint(11, 28 if precision == "c64" else 24), "precision": precision, "width": 5}
    if kind == "shots":
        return {"kind": kind, "n": rng.randint(11, 29), "shots": _log(rng, 1000, 1000000),
                "precision": rng.choice(["c64", "c128"])}
    if kind == "midway":
        return {"kind": kind, "n": rng.randint(8, 23), "measures": rng.randint(1, 3), "shots": _log(rng, 1000, 8192)}
    if kind == "batch":
        qmax = rng.randint(12, 17)
        return {"kind": kind, "circuits": _log(rng, 16, 160), "qmin": 8, "qmax": qmax, "dmin": 5, "dmax": 30,
                "shots": _log(rng, 100, 2048)}
    return {"kind": kind, "n": rng.randint(10, 27), "precision": rng.choice(["c128", "c64"])}


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


# ---------------------------------------------------------------- inputs

def _random_calls(n, count, seed):
    """(gate, qubits): what the gate set offers, one kind after the other."""
    rng = np.random.default_rng(seed)
    ang = lambda: float(rng.uniform(0.0, 2 * math.pi))  # noqa: E731
    kinds = [lambda: G.U3(ang(), ang(), ang()), lambda: G.CX(), lambda: G.H(), lambda: G.CU1(ang()), lambda: G.T(),
             lambda: G.RX(ang()), lambda: G.Swap(), lambda: G.CCX(), lambda: G.Kron(G.U3(ang(), ang(), ang()), G.H()),
             lambda: G.CRY(ang()), lambda: G.RZ(ang()), lambda: _block3(ang(), ang())]
    out = []
    for i in range(count):
        g = kinds[i % len(kinds)]()
        out.append((g, [int(q) for q in rng.choice(n, g.nr_affected_bits(), replace=False)]))
    return out


def _block3(a, b):
    c = G.Composite("block", 3)
    c.add_gate(G.H(), [0])
    c.add_gate(G.CRX(a), [0, 1])
    c.add_gate(G.U2(a, b), [2])
    c.add_gate(G.CX(), [1, 2])
    return c


def _midway_circuit(n, measures, seed):
    """Layers of U3 and CX; after each a Z or X measurement into classical bit
    j and an X conditioned on it; at the end one more qubit reset."""
    rng = np.random.default_rng(seed)
    c = Circuit(n, max(measures, 1))

    def layer(start):
        for q in range(n):
            c.add_gate(G.U3(*rng.uniform(0.0, 2 * math.pi, 3)), [q])
        for q in range(start, n - 1, 2):
            c.add_gate(G.CX(), [q, q + 1])

    layer(0)
    for j in range(measures):
        q = int(rng.integers(n))
        c.measure(q, j, "z" if j % 2 == 0 else "x")
        c.add_conditional_gate([j], 1, G.X(), [int(rng.integers(n))])
        layer((j + 1) % 2)
    c.reset(int(rng.integers(n)))
    return c


def _coefficients(n, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(size=2 * n) + 1j * rng.normal(size=2 * n)


def _random_state(n, seed, precision):
    """A random unit vector on the GPU, in the state's precision."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    real = torch.float64 if precision == "c128" else torch.float32
    v = torch.randn(1 << n, 2, generator=g, dtype=real, device="cuda")
    v /= torch.linalg.vector_norm(v, dtype=torch.float64).to(real)
    return torch.view_as_complex(v)


def _state_of(n, shots, precision, amplitudes):
    shard = EngineShard(n, shots, precision)
    shard.amplitudes().copy_(amplitudes)
    shard.amplitudes_written()
    return shard.state


def _amplitudes(state):
    """A state's amplitudes where they are on the GPU, column after column;
    the tensor keeps the state that owns them."""
    shard = EngineShard.__new__(EngineShard)
    shard.state, shard.precision = state, state.precision
    a = shard.amplitudes()
    a.owner = shard
    return a


def _all_columns(case, a):
    """Zeros for the columns that a rare certain outcome left out, so that the
    result's length does not depend on the draw."""
    full = 1 << (case["n"] + case["measures"] + 1)
    return a if a.numel() == full else torch.nn.functional.pad(a, (0, full - a.numel()))


def prepare(case, seed):
    k = case["kind"]
    s = {"case": case, "seed": seed}
    if k == "circuit":
        s["circuit"] = workloads.brick(case["n"], case["depth"], seed, precision="c128", fusion_width=0)
    elif k == "calls":
        s["calls"] = _random_calls(case["n"], case["gates"], seed)
        s["state"] = VectorState(case["n"], 1, case["precision"])
    elif k == "brick":
        s["circuit"] = workloads.brick(case["n"], case["depth"], seed, precision=case["precision"],
                                       fusion_width=case["width"], measure=False)
    elif k == "qft":
        s["circuit"] = workloads.qft(case["n"], precision=case["precision"], fusion_width=case["width"], measure=False)
        s["state"] = _state_of(case["n"], 1, case["precision"], _random_state(case["n"], seed, case["precision"]))
    elif k == "shots":
        s["state"] = _state_of(case["n"], case["shots"], case["precision"],
                               _random_state(case["n"], seed, case["precision"]))
        s["words"] = np.zeros(case["shots"], dtype=np.uint64)
    elif k == "midway":
        s["circuit"] = _midway_circuit(case["n"], case["measures"], seed)
    elif k == "batch":
        s["batch"] = Batch(4)
        circuits = workloads.batch_workload(case["circuits"], seed, case["qmin"], case["qmax"], case["dmin"], case["dmax"])
        for i, c in enumerate(circuits):
            s["batch"].add(c, case["shots"], seed + i)
    elif k == "product":
        s["coefs"] = _coefficients(case["n"], seed)
    return s


def run(s):
    case, k = s["case"], s["case"]["kind"]
    if k == "circuit":
        s["circuit"].execute(case["shots"], Rng(s["seed"]))
        return s["circuit"].cstate().view(np.int64)
    if k == "calls":
        st = s["state"]
        st.reset_all()
        for g, bits in s["calls"]:
            st.apply_gate(g, bits)
        return _amplitudes(st)
    if k == "brick":
        s["circuit"].execute(1, Rng(s["seed"]))
        return _amplitudes(s["circuit"].q_state)
    if k == "qft":
        s["circuit"].execute_with(1, Rng(s["seed"]), s["state"])
        return _amplitudes(s["state"])
    if k == "shots":
        s["state"].peek_all_into(list(range(case["n"])), s["words"], rng=Rng(s["seed"]))
        return s["words"].view(np.int64)
    if k == "midway":
        s["circuit"].execute(case["shots"], Rng(s["seed"]))
        return {"words": s["circuit"].cstate().view(np.int64),
                "amplitudes": _all_columns(case, _amplitudes(s["circuit"].q_state))}
    if k == "batch":
        return np.concatenate(s["batch"].run()).view(np.int64)
    s["state"] = VectorState.from_qubit_coefs(s["coefs"], 1, case["precision"])
    return _amplitudes(s["state"])


# ---------------------------------------------------------------- work

def _bytes_per(precision):
    return 16 if precision == "c128" else 8


def _brick_flops(n, depth):
    """A 2x2 complex update of a pair takes 28 operations, a CX none."""
    return 14.0 * (1 << n) * n * depth


def work(case):
    k = case["kind"]
    if k == "circuit":
        # matrices in, words out
        return {"bytes": 64 * case["n"] * case["depth"] + 8 * case["shots"], "flops": _brick_flops(case["n"], case["depth"])}
    if k == "calls":
        return {"bytes": _bytes_per(case["precision"]) << case["n"], "flops": 10.0 * (1 << case["n"]) * case["gates"]}
    if k == "brick":
        return {"bytes": _bytes_per(case["precision"]) << case["n"], "flops": _brick_flops(case["n"], case["depth"])}
    if k == "qft":
        return {"bytes": 2 * _bytes_per(case["precision"]) << case["n"], "flops": 5.0 * (1 << case["n"]) * case["n"]}
    if k == "shots":
        return {"bytes": (_bytes_per(case["precision"]) << case["n"]) + 8 * case["shots"], "flops": 3.0 * (1 << case["n"])}
    if k == "midway":
        # each measurement and the reset write the columns that they split
        m = case["measures"]
        return {"bytes": (16 << case["n"]) * ((1 << (m + 1)) - 1), "flops": _brick_flops(case["n"], 1) * ((1 << (m + 1)) - 1)}
    if k == "batch":
        q = 0.5 * (case["qmin"] + case["qmax"])
        return {"bytes": 8 * case["circuits"] * case["shots"],
                "flops": case["circuits"] * 2 * 14.0 * 2.0 ** q * q * 0.5 * (case["dmin"] + case["dmax"])}
    return {"bytes": _bytes_per(case["precision"]) << case["n"], "flops": 6.0 * (1 << case["n"])}


# ---------------------------------------------------------------- 64-bit results

def _apply(x, mat, bits, n):
    """The gate on qubits `bits` (the first is the matrix's highest bit) of
    the columns x (ncols, 2^n), qubit 0 the highest index bit."""
    m = torch.as_tensor(np.ascontiguousarray(mat), dtype=torch.complex128, device=x.device)
    k = len(bits)
    order = sorted(range(k), key=lambda j: bits[j])
    shape, at = [x.shape[0]], 0
    for j in order:
        shape += [1 << (bits[j] - at), 2]
        at = bits[j] + 1
    shape.append(1 << (n - at))
    v = x.reshape(shape)
    dim_of = {j: 2 * i + 2 for i, j in enumerate(order)}
    front = [dim_of[j] for j in range(k)]
    rest = [d for d in range(len(shape)) if d not in front]
    perm = front + rest
    w = v.permute(perm)
    y = (m @ w.reshape(1 << k, -1)).reshape(w.shape)
    back = [perm.index(d) for d in range(len(shape))]
    return y.permute(back).reshape(x.shape)


def _splitmix(seed, counter):
    z = (seed + (counter + 1) * 0x9E3779B97F4A7C15) & (2 ** 64 - 1)
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & (2 ** 64 - 1)
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & (2 ** 64 - 1)
    return ((z ^ (z >> 31)) >> 11) * (1.0 / 9007199254740992.0)


def _binomial(n, p, u):
    """The smallest k whose cumulative probability exceeds u."""
    if n == 0 or p <= 0.0:
        return 0
    if p >= 1.0:
        return n
    cdf, lp, lq = 0.0, math.log(p), math.log1p(-p)
    for j in range(n + 1):
        cdf += math.exp(math.lgamma(n + 1) - math.lgamma(j + 1) - math.lgamma(n - j + 1) + j * lp + (n - j) * lq)
        if u < cdf:
            return j
    return n


def _measure(x, counts, q, n, seed, counter):
    """(columns, counts, each new column's outcome) of a Z measurement."""
    cols, new, bits = [], [], []
    for c in range(x.shape[0]):
        v = x[c].reshape(1 << q, 2, -1)
        w0 = float((v[:, 0].abs() ** 2).sum())
        n0 = _binomial(counts[c], min(w0, 1.0), _splitmix(seed, counter + c))
        for bit, runs, w in ((0, n0, w0), (1, counts[c] - n0, 1.0 - w0)):
            if runs:
                y = torch.zeros_like(v)
                y[:, bit] = v[:, bit] / math.sqrt(w)
                cols.append(y.reshape(-1))
                new.append(runs)
                bits.append(bit)
    return torch.stack(cols), new, bits


def _exact_midway(case, seed):
    n = case["n"]
    x = torch.zeros(1, 1 << n, dtype=torch.complex128, device="cuda")
    x[0, 0] = 1.0
    counts, words, ctr = [case["shots"]], [0], 0
    h = G.H().matrix()
    flip = G.X().matrix()

    def measured(q):
        nonlocal x, counts, words, ctr
        old = x.shape[0]
        src = []
        y, new, bits = _measure(x, counts, q, n, seed, ctr)
        left, c = counts[0], 0
        for runs in new:     # which old column each new one comes from
            src.append(c)
            left -= runs
            if left == 0 and c + 1 < old:
                c += 1
                left = counts[c]
        ctr += old
        words = [words[s] for s in src]
        x, counts = y, new
        return bits

    def conditional(apply, mat, bits):
        for c in range(x.shape[0]):
            if apply[c]:
                x[c] = _apply(x[c:c + 1], mat, bits, n)[0]

    for op in _midway_circuit(n, case["measures"], seed).ops:
        if op[0] == "gate":
            x = _apply(x, op[1].matrix(), op[2], n)
        elif op[0] == "measure":
            _, q, cbit, basis = op
            if basis == "x":
                x = _apply(x, h, [q], n)
            bits = measured(q)
            words = [w & ~(1 << cbit) | b << cbit for w, b in zip(words, bits)]
            if basis == "x":
                x = _apply(x, h, [q], n)
        elif op[0] == "cgate":
            conditional([w >> op[1][0] & 1 for w in words], op[3].matrix(), op[4])
        elif op[0] == "reset":
            conditional(measured(op[1]), flip, [op[1]])
    return {"words": None, "amplitudes": _all_columns(case, x.reshape(-1))}


def exact(case, seed):
    """run()'s result in 64 bits, without the engine's kernels: the gates'
    matrices applied by torch, the QFT as an inverse FFT."""
    k = case["kind"]
    if k in ("calls", "brick"):
        n = case["n"]
        if n > 28:
            return None      # takes too long
        if k == "calls":
            ops = [(g.matrix(), bits) for g, bits in _random_calls(n, case["gates"], seed)]
        else:
            c = workloads.brick(n, case["depth"], seed, measure=False)
            ops = [(op[1].matrix(), op[2]) for op in c.ops]
        x = torch.zeros(1, 1 << n, dtype=torch.complex128, device="cuda")
        x[0, 0] = 1.0
        for m, bits in ops:
            x = _apply(x, m, bits, n)
        return x.reshape(-1)
    if k == "qft":
        v = _random_state(case["n"], seed, case["precision"]).to(torch.complex128)
        return torch.fft.ifft(v, norm="ortho")
    if k == "midway":
        return _exact_midway(case, seed)
    if k == "product":
        c = torch.as_tensor(_coefficients(case["n"], seed).reshape(-1, 2), device="cuda")
        c = c / torch.linalg.vector_norm(c, dim=1, keepdim=True)
        x = c[0]
        for q in range(1, case["n"]):
            x = (x[:, None] * c[q][None, :]).reshape(-1)
        return x
    return None              # words only
