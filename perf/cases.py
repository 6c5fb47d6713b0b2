"""The work that programs have this engine do, as cases that can be timed and compared.

Every case goes through the package's public entry points (`GpuStateVector`, `TrajectoryBatch`,
`GpuSparseVector`, `FrameSampler`).  The kinds:

- ``gates``     gates applied one by one from the host, then a readout (a program that builds its circuit as it goes);
- ``layers``    `run` of a random-layer circuit on a dense register (H/S/T/SQRT_X/RZ on every qubit, a CZ matching);
- ``noisy``     one noisy trajectory with measurements, resets and Pauli channels between the gates;
- ``unitaries`` dense matrices on k qubits (`apply_matrix`), small and wide ones;
- ``readout``   the observables of a state: a spin-chain Hamiltonian's expectation, norm, overlap, Born samples;
- ``fused``     `run_fused` of a random-layer circuit on a complex64 register;
- ``batch``     many noisy trajectories of mixed sizes in one batch;
- ``sparse``    permutation/diagonal circuits on registers whose states stay sparse (up to 64 qubits);
- ``wide``      the same on registers wider than 64 qubits;
- ``frames``    bulk sampling of a noisy Clifford circuit by Pauli frames.
"""
import ctypes
import math
import random

import numpy as np
import torch

import ncsim_b200 as nb

ONE = ("H", "S", "T", "SQRT_X", "RZ")


def listed():
    return [
        # a small interactive register driven gate by gate: latency of the single calls
        {"name": "gates_n12", "kind": "gates", "n": 12, "gates": 96, "precision": "c128"},
        # the benchmark's 20-qubit circuit: a register that fits the L2
        {"name": "layers_n20", "kind": "layers", "n": 20, "depth": 40},
        # a register far larger than the L2, as the 30-qubit configuration (4 GiB of complex128)
        {"name": "layers_n28", "kind": "layers", "n": 28, "depth": 20},
        # one trajectory of an error-correction style circuit on an odd register
        {"name": "noisy_n17", "kind": "noisy", "n": 17, "rounds": 8, "p": 0.01},
        # unitaries a program computed itself, from 3 qubits to wide blocks
        {"name": "unitaries_n24", "kind": "unitaries", "n": 24, "ks": "3,4,5,6,7,9", "precision": "c128"},
        # the inner step of a variational program: energy, overlap, samples
        {"name": "readout_n24", "kind": "readout", "n": 24, "shots": 100000},
        # the tensor-core form where launches and planning count, and where the register streams from HBM
        {"name": "fused_n21", "kind": "fused", "n": 21, "depth": 20},
        {"name": "fused_n30", "kind": "fused", "n": 30, "depth": 8},
        # an eighth of the benchmark's batch of noisy trajectories
        {"name": "batch_512", "kind": "batch", "count": 512, "n_lo": 16, "n_span": 7, "depth": 30, "p": 1e-3},
        # the 31-qubit reversible configuration: 2^16 entries, 2000 gates
        {"name": "sparse_n31", "kind": "sparse", "n": 31, "inputs": 16, "gates": 2000},
        # the reference's published sparse workload: a Toffoli/CNOT ripple at n = 1000
        {"name": "wide_n1000", "kind": "wide", "n": 1000, "inputs": 10, "gates": 1996, "ripple": True},
        # the reference's published frame-sampler workload
        {"name": "frames_n1000", "kind": "frames", "n": 1000, "rounds": 20, "meas": 100, "p": 1e-3, "shots": 100000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gates", "layers", "noisy", "unitaries", "readout", "fused", "batch", "sparse", "wide", "frames"])
    if kind == "gates":
        return {"kind": kind, "n": rng.randint(5, 24), "gates": _log(rng, 16, 200), "precision": rng.choice(["c128", "c64"])}
    if kind == "layers":
        return {"kind": kind, "n": rng.randint(10, 27), "depth": _log(rng, 4, 40)}
    if kind == "noisy":
        return {"kind": kind, "n": rng.randint(6, 23), "rounds": rng.randint(2, 12), "p": rng.choice([0.001, 0.01, 0.05])}
    if kind == "unitaries":
        n = rng.randint(12, 25)
        ks = sorted(rng.randint(2, 10) for _ in range(rng.randint(2, 6)))
        return {"kind": kind, "n": n, "ks": ",".join(map(str, ks)), "precision": rng.choice(["c128", "c64"])}
    if kind == "readout":
        return {"kind": kind, "n": rng.randint(8, 26), "shots": _log(rng, 100, 200000)}
    if kind == "fused":
        return {"kind": kind, "n": rng.randint(13, 29), "depth": _log(rng, 4, 20)}
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 24, 512), "n_lo": rng.randint(13, 18), "n_span": rng.randint(1, 5),
                "depth": _log(rng, 6, 30), "p": rng.choice([1e-3, 1e-2])}
    if kind == "sparse":
        return {"kind": kind, "n": rng.randint(17, 60), "inputs": rng.randint(3, 16), "gates": _log(rng, 50, 2000)}
    if kind == "wide":
        return {"kind": kind, "n": rng.randint(65, 1000), "inputs": rng.randint(3, 13), "gates": _log(rng, 50, 2000),
                "ripple": rng.random() < 0.3}
    return {"kind": kind, "n": _log(rng, 12, 1000), "rounds": rng.randint(3, 20), "meas": _log(rng, 8, 100),
            "p": rng.choice([1e-4, 1e-3, 1e-2]), "shots": _log(rng, 1000, 100000)}


# ---------------------------------------------------------------------------
# circuits as lists of (name, argument, qubits), made from the seed alone
# ---------------------------------------------------------------------------
def _token(name, arg):
    return name if arg is None else "%s(%r)" % (name, arg)


def _text(n, gates):
    return "QUBITS %d\n" % n + "".join("%s %s\n" % (_token(g, a), " ".join(map(str, qs))) for g, a, qs in gates)


def _layers(n, depth, seed):
    r = random.Random(seed)
    gates = []
    for _ in range(depth):
        for q in range(n):
            g = r.choice(ONE)
            gates.append((g, r.uniform(0, 2 * math.pi) if g == "RZ" else None, (q,)))
        perm = list(range(n))
        r.shuffle(perm)
        gates += [("CZ", None, (perm[i], perm[i + 1])) for i in range(0, n - 1, 2)]
    return gates


def _mixed(n, count, seed):
    r = random.Random(seed)
    gates = []
    for _ in range(count):
        g = r.choice(["H", "T", "S", "X", "RX", "RY", "RZ", "CX", "CZ", "SWAP", "CCX"])
        k = {"CX": 2, "CZ": 2, "SWAP": 2, "CCX": 3}.get(g, 1)
        gates.append((g, r.uniform(0, 2 * math.pi) if g[0] == "R" else None, tuple(r.sample(range(n), k))))
    return gates


def _noisy_text(n, rounds, p, seed):
    r = random.Random(seed)
    lines = ["QUBITS %d" % n]
    for _ in range(rounds):
        for q in range(n):
            lines.append("%s %d" % (r.choice(["H", "S", "T", "SQRT_X", "RY(0.7)"]), q))
        for q in range(r.randrange(2), n - 1, 2):
            lines.append("%s %d %d" % (r.choice(["CX", "CZ"]), q, q + 1))
            lines.append("DEPOLARIZE2(%r) %d %d" % (p, q, q + 1))
        a, b = r.sample(range(n), 2)
        lines.append("MPP %s%d*%s%d" % (r.choice("XYZ"), a, r.choice("XYZ"), b))
        for q in r.sample(range(n), max(1, n // 4)):
            lines.append("M %d" % q)
        lines.append("R %d" % r.randrange(n))
        lines.append("DEPOLARIZE1(%r) %d" % (p, r.randrange(n)))
    return "\n".join(lines) + "\n"


def _rank(rows):
    rows, rank = list(rows), 0
    for b in reversed(range(8)):
        piv = next((i for i in range(rank, len(rows)) if rows[i] >> b & 1), None)
        if piv is None:
            continue
        rows[rank], rows[piv] = rows[piv], rows[rank]
        rows = [v ^ rows[rank] if i != rank and v >> b & 1 else v for i, v in enumerate(rows)]
        rank += 1
    return rank


def _terms(r, nv, count):
    return [(1 + r.randrange(7), tuple(r.sample(range(nv), min(nv, 1 + r.randrange(3))))) for _ in range(count)]


def _reversible(n, inputs, gates, seed):
    """H on the first `inputs` qubits, then CX, CCX, CCZ, 40-term diagonals and 8-qubit affine monomials alike often."""
    r = random.Random(seed)
    ops = [("H", None, (q,)) for q in range(inputs)]
    for _ in range(gates):
        g = r.choice(["CX", "CCX", "CCZ", "DIAG", "MONOMIAL"])
        if g == "DIAG":
            ops.append((g, _terms(r, n, 40), tuple(range(n))))
        elif g == "MONOMIAL":
            while True:
                rows = [r.randrange(256) for _ in range(8)]
                if _rank(rows) == 8:
                    break
            ops.append((g, (rows, r.randrange(256), _terms(r, 8, 8)), tuple(r.sample(range(n), 8))))
        else:
            ops.append((g, None, tuple(r.sample(range(n), 2 if g == "CX" else 3))))
    return ops


def _reversible_text(n, ops):
    def terms(ts):
        return "".join(";%d:%s" % (c, ",".join(str(1 << v) for v in vs)) for c, vs in ts)

    lines = ["QUBITS %d" % n]
    for g, a, qs in ops:
        if g == "DIAG":
            g = "DIAG(3;0%s)" % terms(a)
        elif g == "MONOMIAL":
            g = "MONOMIAL(%s;%d;3;0%s;0,0,0)" % (",".join(map(str, a[0])), a[1], terms(a[2]))
        lines.append("%s %s" % (g, " ".join(map(str, qs))))
    return "\n".join(lines) + "\n"


def _wide_ops(case, seed):
    r = random.Random(seed)
    n, ops = case["n"], [("H", None, (q,)) for q in range(case["inputs"])]
    if case["ripple"]:
        # the published ripple; the seed says which qubits start flipped
        ops += [("X", None, (r.randrange(n),)) for _ in range(4)]
        tail = []
        for q in range(n - 2):
            tail += [("CCX", None, (q, q + 1, q + 2)), ("CX", None, (q, q + 2))]
        return ops + tail[: case["gates"]]
    hot = r.sample(range(n), min(n, 40)) + list(range(case["inputs"]))
    for _ in range(case["gates"]):
        g = r.choice(["CX", "CX", "CCX", "SWAP", "CCZ", "CZ", "T", "S", "X"])
        k = {"CX": 2, "SWAP": 2, "CZ": 2, "CCX": 3, "CCZ": 3}.get(g, 1)
        while True:
            qs = r.sample(hot if r.random() < 0.7 else range(n), k)
            if len(set(qs)) == k:
                break
        ops.append((g, None, tuple(qs)))
    return ops


def _chain(n, seed):
    """Terms (coefficient, x mask, z mask, phase) of a spin chain with random couplings and fields."""
    r = random.Random(seed)
    terms = []
    for q in range(n - 1):
        m = 3 << q
        terms += [(r.uniform(-1, 1), m, 0, 0), (r.uniform(-1, 1), m, m, 2), (r.uniform(-1, 1), 0, m, 0)]
    for q in range(n):
        terms.append((r.uniform(-1, 1), 0, 1 << q, 0))
        if q % 3 == 0:
            terms.append((r.uniform(-1, 1), 1 << q, 0, 0))
    return terms


# ---------------------------------------------------------------------------
# states
# ---------------------------------------------------------------------------
def _amplitudes(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    v = torch.randn(1 << n, 2, generator=g, device="cuda", dtype=torch.float32)
    v /= v.norm()
    return torch.view_as_complex(v)


def _register(n, seed, precision=nb.C128):
    """A state holding the seed's amplitudes, and a tensor over them that keeps the state alive."""
    sv = nb.GpuStateVector(n, precision)
    view = sv.torch_view()
    view.copy_(_amplitudes(n, seed))
    torch.cuda.synchronize()
    view.owner = sv
    return sv, view


def _unitaries(case, seed):
    r = random.Random(seed)
    out = []
    for j, k in enumerate(int(t) for t in case["ks"].split(",")):
        g = torch.Generator()
        g.manual_seed(seed + j)
        m = torch.linalg.qr(torch.randn(1 << k, 1 << k, dtype=torch.complex128, generator=g))[0]
        out.append((m.numpy(), r.sample(range(case["n"]), k)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "rng": nb.StdRng(seed)}
    if kind == "gates":
        s["sv"], _ = _register(case["n"], seed, nb.C128 if case["precision"] == "c128" else nb.C64)
        s["gates"] = [(nb.Gate.parse(_token(g, a)), list(qs)) for g, a, qs in _mixed(case["n"], case["gates"], seed)]
        s["pauli"] = nb.Pauli.from_string(case["n"], "X0*Y3*Z4")
    elif kind in ("layers", "fused"):
        s["sv"], s["view"] = _register(case["n"], seed, nb.C64 if kind == "fused" else nb.C128)
        s["circuit"] = nb.Circuit.parse(_text(case["n"], _layers(case["n"], case["depth"], seed)))
    elif kind == "noisy":
        s["sv"], s["view"] = _register(case["n"], seed)
        s["circuit"] = nb.Circuit.parse(_noisy_text(case["n"], case["rounds"], case["p"], seed))
    elif kind == "unitaries":
        s["sv"], s["view"] = _register(case["n"], seed, nb.C128 if case["precision"] == "c128" else nb.C64)
        s["matrices"] = _unitaries(case, seed)
    elif kind == "readout":
        n = case["n"]
        s["sv"], s["view"] = _register(n, seed)
        s["other"], s["other_view"] = _register(n, seed + 1)
        s["terms"] = [(c, nb.Pauli(n, x, z, ph)) for c, x, z, ph in _chain(n, seed)]
        s["shots"], s["index"] = case["shots"], random.Random(seed).randrange(1 << n)
    elif kind == "batch":
        s["batch"] = nb.TrajectoryBatch.random_layers(case["count"], seed0=1 + (seed << 12), n_lo=case["n_lo"],
                                                      n_span=case["n_span"], depth=case["depth"], p=case["p"])
    elif kind == "sparse":
        s["n"] = case["n"]
        s["circuit"] = nb.Circuit.parse(_reversible_text(case["n"], _reversible(case["n"], case["inputs"], case["gates"], seed)))
    elif kind == "wide":
        s["n"] = case["n"]
        s["circuit"] = nb.Circuit.parse(_text(case["n"], _wide_ops(case, seed)))
    else:
        s["shots"] = case["shots"]
        circuit = nb.Circuit.frames_workload(case["n"], case["rounds"], case["meas"], case["p"], seed)
        s["sampler"] = nb.FrameSampler(circuit, seed)
        s["out"] = np.zeros((s["sampler"].m, nb.FrameSampler.words(case["shots"])), dtype=np.uint64)
    return s


def _packed_entries(sv):
    """Keys as (entries, words) and amplitudes, through the C interface: `entries` makes Python integers of wide keys."""
    m = sv.num_entries()
    keys, amps = np.empty((m, sv.words), dtype=np.uint64), np.empty(m, dtype=np.complex128)
    u64, f64 = ctypes.POINTER(ctypes.c_uint64), ctypes.POINTER(ctypes.c_double)
    status = nb.lib().ncsim_sparse_get_entries(sv._h, keys.ctypes.data_as(u64), amps.ctypes.data_as(f64), m)
    if status:
        raise RuntimeError("ncsim_sparse_get_entries: %d" % status)
    return keys, amps


def run(state):
    kind = state["kind"]
    if kind == "gates":
        sv = state["sv"]
        for gate, qubits in state["gates"]:
            sv.apply_gate(gate, qubits)
        return {"expectation": np.array([sv.expectation(state["pauli"])]), "amplitudes": _small(sv)}
    if kind == "layers":
        state["sv"].run(state["circuit"], state["rng"])
        return state["view"]
    if kind == "fused":
        state["sv"].run_fused(state["circuit"], state["rng"])
        return state["view"]
    if kind == "noisy":
        record = state["sv"].run(state["circuit"], state["rng"])
        return {"record": np.array(record, dtype=np.int64), "amplitudes": state["view"]}
    if kind == "unitaries":
        for matrix, qubits in state["matrices"]:
            state["sv"].apply_matrix(matrix, qubits)
        return state["view"]
    if kind == "readout":
        sv = state["sv"]
        return {"energy": np.array([sv.expectation_sum(state["terms"])]), "norm": np.array([sv.norm_sq()]),
                "overlap": np.array([sv.inner(state["other"])]), "probability": sv.probability(state["index"]),
                "samples": sv.sample(state["rng"], state["shots"])}
    if kind == "batch":
        state["batch"].run()
        n, record, z0, norm = state["batch"].results()
        # sums over complex64 amplitudes: 32-bit numbers
        return {"qubits": n.astype(np.int64), "records": record, "readouts": np.stack([z0, norm]).astype(np.float32)}
    if kind in ("sparse", "wide"):
        sv = nb.GpuSparseVector.zero_state(state["n"])
        sv.run(state["circuit"], state["rng"])
        keys, amps = _packed_entries(sv)
        return {"keys": keys, "amplitudes": amps}
    seeds = [state["rng"].next_u64() for _ in range(-(-state["shots"] // nb.FrameSampler.BATCH))]
    return state["sampler"].sample_packed_seeds(state["shots"], seeds, state["out"])


def _small(sv):
    """What an interactive program looks at: every amplitude of a small register, the first ones of a larger one."""
    return sv.to_vector_range(0, 1 << min(sv.n, 12)).astype(np.complex128 if sv.precision == nb.C128 else np.complex64)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _gate_flops(gates, n):
    """Per gate: a dense 2x2 takes 14 flops an amplitude, a phase 6 on the amplitudes that it changes, a swap none."""
    dense = sum(g in ("H", "SQRT_X", "RX", "RY") for g, _, _ in gates)
    half = sum(g in ("S", "T") for g, _, _ in gates)
    full = sum(g == "RZ" for g, _, _ in gates)
    return float(1 << n) * (14.0 * dense + 3.0 * half + 6.0 * full)


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "gates":
        item = 16 if case["precision"] == "c128" else 8
        return {"bytes": 2.0 * item * (1 << n), "flops": _gate_flops(_mixed(n, case["gates"], 1), n)}
    if kind in ("layers", "fused"):
        item = 16 if kind == "layers" else 8
        return {"bytes": 2.0 * item * (1 << n), "flops": _gate_flops(_layers(n, case["depth"], 1), n)}
    if kind == "noisy":
        return {"bytes": 2.0 * 16 * (1 << n), "flops": 8.0 * case["rounds"] * n * (1 << n)}
    if kind == "unitaries":
        item = 16 if case["precision"] == "c128" else 8
        ks = [int(t) for t in case["ks"].split(",")]
        return {"bytes": 2.0 * item * (1 << n) + 16.0 * sum(4 ** k for k in ks),
                "flops": sum(8.0 * (1 << k) for k in ks) * (1 << n)}
    if kind == "readout":
        return {"bytes": 2.0 * 16 * (1 << n) + 16.0 * case["shots"], "flops": 4.0 * len(_chain(n, 1)) * (1 << n)}
    if kind == "batch":
        sizes = range(case["n_lo"], case["n_lo"] + case["n_span"])
        each = case["count"] / case["n_span"]
        return {"bytes": each * sum(2.0 * 8 * (1 << m) for m in sizes),
                "flops": each * sum((0.4 * 14 + 0.4 * 3 + 0.2 * 6) * case["depth"] * m * (1 << m) for m in sizes)}
    if kind == "sparse":
        return {"bytes": 24.0 * (1 << case["inputs"]), "flops": 28.0 * case["gates"] * (1 << case["inputs"])}
    if kind == "wide":
        return {"bytes": (8.0 * (4 if n <= 256 else 16) + 16) * (1 << case["inputs"]),
                "flops": 2.0 * case["gates"] * (1 << case["inputs"])}
    return {"bytes": case["rounds"] * case["meas"] * math.ceil(case["shots"] / 64) * 8.0,
            "flops": case["rounds"] * (n / 2) * case["shots"] / 64 * 4.0}


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain torch
# ---------------------------------------------------------------------------
def _matrix(g, arg):
    w = complex(0.5, 0.5)
    h = math.sqrt(0.5)
    if g in ("RX", "RY"):
        c, s = math.cos(arg / 2), math.sin(arg / 2)
        return [[c, -1j * s], [-1j * s, c]] if g == "RX" else [[c, -s], [s, c]]
    return {"H": [[h, h], [h, -h]], "SQRT_X": [[w, w.conjugate()], [w.conjugate(), w]], "X": [[0, 1], [1, 0]]}[g]


def _phases(g, arg):
    if g == "RZ":
        return complex(math.cos(arg / 2), -math.sin(arg / 2)), complex(math.cos(arg / 2), math.sin(arg / 2))
    return 1.0, {"S": 1j, "T": complex(math.sqrt(0.5), math.sqrt(0.5))}[g]


def _split(n, qubits):
    """The register's shape with an axis of 2 for each qubit, and the axis of each."""
    shape, axis, at = [], {}, n
    for q in sorted(qubits, reverse=True):
        shape += [1 << (at - q - 1), 2]
        axis[q] = len(shape) - 1
        at = q
    return shape + [1 << at], axis


def _apply(v, n, g, arg, qubits):
    shape, axis = _split(n, qubits)
    t = v.view(shape)
    at = {axis[q]: 1 for q in qubits}

    def part(ones):
        return t[tuple(ones.get(a, slice(None)) for a in range(len(shape)))]

    if g in ("S", "T", "RZ"):
        for b, ph in enumerate(_phases(g, arg)):
            if ph != 1.0:
                part({axis[qubits[0]]: b}).mul_(ph)
    elif g == "CZ":
        part(at).neg_()
    elif g in ("CX", "CCX", "SWAP"):
        if g == "SWAP":
            a, b = part({axis[qubits[0]]: 1, axis[qubits[1]]: 0}), part({axis[qubits[0]]: 0, axis[qubits[1]]: 1})
        else:
            a, b = part({**at, axis[qubits[-1]]: 0}), part(at)
        old = a.clone()
        a.copy_(b)
        b.copy_(old)
    else:
        m = _matrix(g, arg)
        a, b = t[:, 0], t[:, 1]
        new = m[0][0] * a
        new.add_(b, alpha=m[0][1])
        b.mul_(m[1][1]).add_(a, alpha=m[1][0])
        a.copy_(new)


def _apply_dense(v, n, matrix, qubits):
    shape, axis = _split(n, qubits)
    front = [axis[q] for q in reversed(qubits)]
    order = front + [a for a in range(len(shape)) if a not in front]
    t = v.view(shape).permute(order)
    got = torch.from_numpy(matrix).to(v.device) @ t.reshape(1 << len(qubits), -1)
    back = [order.index(a) for a in range(len(shape))]
    return got.view(t.shape).permute(back).reshape(-1)


def _parity(v):
    for s in (32, 16, 8, 4, 2, 1):
        v = v ^ (v >> s)
    return v & 1


def _expect(v, x, z, phase, index):
    """<v| i^phase X^x Z^z |v>."""
    sign = (1 - 2 * _parity(index & z)).to(torch.float64)
    w = v * sign
    total = torch.vdot(v.index_select(0, index ^ x), w) if x else torch.vdot(v, w)
    return complex(total) * 1j ** phase


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind in ("noisy", "batch", "frames"):
        return None  # their random draws are the engine's own generator's
    if kind in ("sparse", "wide"):
        return {"keys": None, "amplitudes": _exact_sparse(case, seed)}
    if kind == "unitaries" and sum(4 ** int(k) for k in case["ks"].split(",")) * (1 << n) > 1 << 46:
        return None
    v = _amplitudes(n, seed).to(torch.complex128)
    if kind == "gates":
        for g in _mixed(n, case["gates"], seed):
            _apply(v, n, *g)
        e = _expect(v, 0b1001, 0b11000, 1, torch.arange(1 << n, device="cuda"))
        return {"expectation": np.array([e]), "amplitudes": v[: 1 << min(n, 12)]}
    if kind in ("layers", "fused"):
        for g in _layers(n, case["depth"], seed):
            _apply(v, n, *g)
        return v
    if kind == "unitaries":
        for matrix, qubits in _unitaries(case, seed):
            v = _apply_dense(v, n, matrix, qubits)
        return v
    index = torch.arange(1 << n, device="cuda")
    energy = sum(c * _expect(v, x, z, ph, index) for c, x, z, ph in _chain(n, seed))
    norm = float(torch.vdot(v, v).real)
    other = _amplitudes(n, seed + 1).to(torch.complex128)
    p = complex(v[random.Random(seed).randrange(1 << n)])
    return {"energy": np.array([energy]), "norm": np.array([complex(norm)]), "overlap": np.array([complex(torch.vdot(v, other))]),
            "probability": abs(p) ** 2 / norm, "samples": None}


def _exact_sparse(case, seed):
    """Bits of every entry as rows of 0/1, entries in the order of their start; phases as eighths of a turn."""
    n, m = case["n"], 1 << case["inputs"]
    ops = _reversible(n, case["inputs"], case["gates"], seed) if case["kind"] == "sparse" else _wide_ops(case, seed)
    bits = torch.zeros(n, m, dtype=torch.int32, device="cuda")
    start = torch.arange(m, device="cuda", dtype=torch.int32)
    for q in range(case["inputs"]):
        bits[q] = (start >> q) & 1
    f = torch.zeros(m, dtype=torch.int32, device="cuda")
    for g, a, qs in ops:
        if g == "H":
            continue
        if g in ("DIAG", "MONOMIAL"):
            for c, vs in a if g == "DIAG" else a[2]:
                p = bits[qs[vs[0]]]
                for v in vs[1:]:
                    p = p & bits[qs[v]]
                f += c * p
        if g == "MONOMIAL":
            old = bits[list(qs)]
            for i, row in enumerate(a[0]):
                new = torch.full((m,), (a[1] >> i) & 1, dtype=torch.int32, device="cuda")
                for j in range(8):
                    if row >> j & 1:
                        new ^= old[j]
                bits[qs[i]] = new
        elif g == "X":
            bits[qs[0]] ^= 1
        elif g == "CX":
            bits[qs[1]] ^= bits[qs[0]]
        elif g == "CCX":
            bits[qs[2]] ^= bits[qs[0]] & bits[qs[1]]
        elif g == "SWAP":
            bits[list(qs)] = bits[[qs[1], qs[0]]]
        elif g in ("CZ", "CCZ", "T", "S"):
            p = bits[qs[0]]
            for q in qs[1:]:
                p = p & bits[q]
            f += {"T": 1, "S": 2}.get(g, 4) * p
    turn = (f.to(torch.float64) % 8) * (math.pi / 4)
    return torch.polar(torch.full_like(turn, m ** -0.5), turn)
