"""Measured cases of the engine: what a VQE program calls, at the sizes it calls them.

``listed()`` names them; ``draw(rng)`` gives more of the same ranges; ``prepare`` builds
what a program holds before the call (engine, circuit, Pauli sum, angles on the GPU),
``run`` makes one pass through the public entry points, ``exact`` the same numbers in
64 bits with plain torch (an exact matrix product state: every CX doubles a bond).
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT / "graph-vqe_b200") not in sys.path:
    sys.path.insert(0, str(ROOT / "graph-vqe_b200"))

import vqemps  # noqa: E402
from vqemps import mpnn  # noqa: E402
from vqemps.reverse import ReverseMPS  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # one objective evaluation of a small problem, with the value of every word: the smallest call
        dict(name="plain_12q", kind="energy", n=12, terms=300, wmax=4, reps=4, gates="ry", pattern="linear", batch=1,
             per_term=True),
        # one SPSA update: the candidate and the next two probes
        dict(name="update_40q", kind="energy", n=40, terms=5000, wmax=6, reps=4, gates="ry", pattern="reverse_linear",
             batch=3, per_term=False),
        # many SPSA probes at once: the benchmark's step
        dict(name="probes_40q", kind="energy", n=40, terms=5000, wmax=6, reps=4, gates="ry", pattern="reverse_linear",
             batch=256, per_term=False),
        # the reference's default ansatz gates (complex amplitudes), an odd width, a middling batch
        dict(name="ryrz_27q", kind="energy", n=27, terms=1300, wmax=4, reps=3, gates="ryrz", pattern="linear", batch=45,
             per_term=True),
        # the warm start's judgement: proposal and zero angles on the widest Hamiltonians
        dict(name="judge_96q", kind="energy", n=96, terms=40000, wmax=4, reps=4, gates="ry", pattern="linear", batch=2,
             per_term=False),
        # one L-BFGS point: host angles in, host value and gradient out
        dict(name="lbfgs_40q", kind="value_grad", n=40, terms=5000, wmax=6, reps=4, gates="ry", pattern="reverse_linear",
             batch=1),
        # a batch of gradients of a large problem: the largest case
        dict(name="grad_64q", kind="grad", n=64, terms=20000, wmax=6, reps=4, gates="ry", pattern="linear", batch=32),
        # gradients with complex amplitudes, odd sizes
        dict(name="grad_ryrz_21q", kind="grad", n=21, terms=790, wmax=4, reps=3, gates="ryrz", pattern="linear", batch=7),
        # the partition warm start's round: 64 local problems of uneven width in one call
        dict(name="partitions_64", kind="partitions", parts=64, nmin=8, nmax=48, tmin=200, tmax=3000, gates="ry", reps=4,
             copies=1, shots=0),
        # the same with 1,000 shots each, bitstrings and shot energies
        dict(name="partition_shots", kind="partitions", parts=64, nmin=8, nmax=48, tmin=200, tmax=3000, gates="ry", reps=4,
             copies=1, shots=1000),
        # the 1000-shot objective with the plugin's streams (X/Y words analytic), an SPSA pair
        dict(name="objective_shots", kind="shots", n=22, terms=400, wmax=4, reps=4, gates="ryrz", pattern="linear", batch=2,
             shots=1000, rng="splitmix", mode="plugin"),
        # one training step of the warm-start network: forward, loss, backward, Adam
        dict(name="train_32", kind="train", graphs=32, nmin=16, nmax=48),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["energy", "energy", "energy", "grad", "grad", "value_grad", "partitions", "partitions", "shots", "train"])
    gates = rng.choice(["ry", "ry", "ryrz"])
    pattern = rng.choice(["linear", "reverse_linear"])
    reps = rng.choice([2, 3, 4, 4, 4])
    if kind == "energy":
        n = _log(rng, 6, 96)
        terms = _log(rng, 60, 420 * n)
        most = min(256, int((12e6 if gates == "ryrz" else 51e6) // (n * terms)))
        return dict(kind=kind, n=n, terms=terms, wmax=rng.randint(2, 6), reps=reps, gates=gates, pattern=pattern,
                    batch=_log(rng, 1, max(most, 1)), per_term=rng.random() < 0.5)
    if kind == "grad":
        n = _log(rng, 6, 64)
        terms = _log(rng, 60, 310 * n)
        most = min(32, int((4e6 if gates == "ryrz" else 40e6) // (n * terms)))
        return dict(kind=kind, n=n, terms=terms, wmax=rng.randint(2, 6), reps=reps, gates=gates, pattern=pattern,
                    batch=_log(rng, 1, max(most, 1)))
    if kind == "value_grad":
        n = _log(rng, 6, 48)
        return dict(kind=kind, n=n, terms=_log(rng, 60, 125 * n), wmax=rng.randint(2, 6), reps=reps, gates=gates,
                    pattern=pattern, batch=1)
    if kind == "partitions":
        nmax = rng.randint(8, 48)
        tmax = _log(rng, 100, 3000)
        return dict(kind=kind, parts=_log(rng, 2, 64), nmin=rng.randint(3, 8), nmax=nmax, tmin=rng.randint(20, 100), tmax=tmax,
                    gates=gates, reps=reps, copies=rng.randint(1, 2), shots=rng.choice([0, 0, rng.randint(100, 1000)]))
    if kind == "shots":
        return dict(kind=kind, n=rng.randint(6, 24), terms=_log(rng, 40, 400), wmax=4, reps=reps, gates=gates, pattern=pattern,
                    batch=rng.randint(1, 2), shots=_log(rng, 100, 1000), rng=rng.choice(["splitmix", "philox"]),
                    mode=rng.choice(["plugin", "shared"]))
    nmin = rng.randint(8, 40)
    return dict(kind="train", graphs=rng.randint(1, 32), nmin=nmin, nmax=rng.randint(nmin, 48))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def circuit(n, reps, gates, pattern):
    """Hardware-efficient ansatz: one rotation per gate letter pair and qubit, then a CX chain,
    ``reps`` times, and a last rotation layer; angles in (layer, qubit, gate) order."""
    kinds = {"ry": ("ry",), "ryrz": ("ry", "rz")}[gates]
    pairs = [(q, q + 1) for q in range(n - 1)]
    if pattern == "reverse_linear":
        pairs = pairs[::-1]
    ops, k = [], 0
    for layer in range(reps + 1):
        for q in range(n):
            for g in kinds:
                ops.append((g, q, k))
                k += 1
        if layer < reps:
            ops.extend(("cx", a, b) for a, b in pairs)
    return ops, k


def pauli_sum(rng, n, terms, wmax):
    """Codes [terms, n] (0 I, 1 X, 2 Y, 3 Z) and coefficients: weight U{1..wmax} on distinct qubits,
    90 % Z words, coefficients N(0, 1) with 20 % penalties of +-U(100, 1000)."""
    w = rng.integers(1, min(wmax, n) + 1, terms)
    where = np.argsort(rng.random((terms, n)), axis=1)[:, :min(wmax, n)]
    codes = np.zeros((terms, n), dtype=np.uint8)
    letters = np.where((rng.random(terms) < 0.9)[:, None], 3, rng.integers(1, 4, where.shape))
    for j in range(where.shape[1]):
        on = np.nonzero(j < w)[0]
        codes[on, where[on, j]] = letters[on, j]
    sign = np.where(rng.random(terms) < 0.5, 1.0, -1.0)
    coeffs = np.where(rng.random(terms) < 0.8, rng.normal(size=terms), sign * rng.uniform(100.0, 1000.0, terms))
    return codes, coeffs


def strings(codes):
    text = np.frombuffer(b"IXYZ", dtype=np.uint8)[codes]
    return [row.tobytes().decode("ascii") for row in text]


def inputs(case, seed):
    """Numbers of one problem: circuit, words, coefficients, angles [batch, P]."""
    rng = np.random.default_rng([seed, 17])
    ops, count = circuit(case["n"], case["reps"], case["gates"], case["pattern"])
    codes, coeffs = pauli_sum(rng, case["n"], case["terms"], case["wmax"])
    B = case["batch"]
    if B > 1 and case["kind"] == "energy":      # SPSA probes around a point
        x = rng.uniform(-np.pi, np.pi, count) + 0.1 * rng.choice([-1.0, 1.0], size=(B, count))
    else:
        x = rng.uniform(-np.pi, np.pi, (B, count))
    return ops, codes, coeffs, x


def parts_of(case, seed):
    rng = np.random.default_rng([seed, 23])
    out = []
    for _ in range(case["parts"]):
        n = int(rng.integers(case["nmin"], case["nmax"] + 1))
        ops, count = circuit(n, case["reps"], case["gates"], "linear")
        codes, coeffs = pauli_sum(rng, n, int(rng.integers(case["tmin"], case["tmax"] + 1)), 4)
        out.append((n, ops, codes, coeffs, rng.uniform(-np.pi, np.pi, (case["copies"], count))))
    return out


def graphs_of(case, seed):
    """Coupling graphs with their features, target angles, and the network's weights."""
    rng = np.random.default_rng([seed, 31])
    slog = lambda v: np.sign(v) * np.log1p(np.abs(v))  # noqa: E731
    graphs, targets = [], []
    for _ in range(case["graphs"]):
        n = int(rng.integers(case["nmin"], case["nmax"] + 1))
        a, b = np.triu_indices(n, 1)
        keep = (b - a == 1) | (rng.random(a.size) < 1.0 - math.exp(-125.0 / max(n - 1, 1)))
        a, b = a[keep], b[keep]
        big = lambda m: np.where(rng.random(m) < 0.8, rng.normal(size=m), rng.uniform(-1000.0, 1000.0, m))  # noqa: E731
        node = np.stack([slog(big(n)) / 5, slog(np.abs(big(n)) * 60) / 10, np.arange(n) / (n - 1),
                         ((np.arange(n) == 0) | (np.arange(n) == n - 1)).astype(float)], axis=1)
        f = np.stack([slog(big(a.size) * (rng.random(a.size) < 0.5)) / 5, slog(np.abs(big(a.size)) * 8) / 10,
                      (b - a == 1).astype(float)], axis=1)
        index = np.array([np.stack([a, b], 1).reshape(-1), np.stack([b, a], 1).reshape(-1)])
        graphs.append((node.astype(np.float32), index.astype(np.int64), np.repeat(f, 2, axis=0).astype(np.float32)))
        t = np.zeros((n, 5))
        t[:, 4] = np.arccos(rng.uniform(-1, 1, n))
        targets.append(t.astype(np.float32))
    weights = []
    for shape in weight_shapes():
        lim = math.sqrt(6.0 / shape[0]) * (0.1 if shape[-1] == 5 and len(shape) == 2 else 1.0)
        weights.append(rng.uniform(-lim, lim, shape) if len(shape) == 2 else 0.02 * rng.normal(size=shape))
    return graphs, np.concatenate(targets), [w.astype(np.float32) for w in weights]


def weight_shapes(width=128, layers=3, out=5):
    shapes = [(4, width), (width,)]
    for _ in range(layers):
        shapes += [(width + 3, width), (width,), (2 * width, width), (width,)]
    return shapes + [(width, out), (out,)]


# ---------------------------------------------------------------------------
# state and pass
# ---------------------------------------------------------------------------
class Loaded:
    """A Pauli sum or partition set of an engine, given back with its state."""

    def __init__(self, eng, thing, free):
        self.eng, self.thing, self.free = eng, thing, free

    def __del__(self):
        if self.eng.ctx:
            self.free(self.thing)


_HELD = {}


def engine(key, spec=None):
    """One engine per circuit, as a solver holds it while it loads one Pauli sum after another."""
    if key not in _HELD:
        _HELD.clear()
        eng = vqemps.Engine(0, 16)
        if spec is not None:
            eng.set_spec(spec)
        _HELD[key] = eng
    return _HELD[key]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        graphs, target, weights = graphs_of(case, seed)
        net = mpnn.MPNN(0, params=np.concatenate([w.reshape(-1) for w in weights]))
        return dict(case=case, net=net, batch=mpnn.make_batch(graphs, net.device), target=torch.tensor(target, device=DEV))
    if kind == "value_grad":
        ops, codes, coeffs, x = inputs(case, seed)
        spec = dict(n=case["n"], ops=ops, initial=None, count=x.shape[1])
        return dict(case=case, problem=ReverseMPS(spec, strings(codes), coeffs), x=x[0])
    if kind == "partitions":
        parts = parts_of(case, seed)
        eng = engine("partitions")
        pset = eng.set_partitions([(n, ops, strings(codes), coeffs) for n, ops, codes, coeffs, _ in parts])
        theta = pset.pack_theta([p[4] for p in parts], copies=case["copies"], device=eng.device)
        return dict(case=case, eng=eng, pset=pset, held=Loaded(eng, pset, eng.free_partitions), theta=theta,
                    seed=seed & 0xFFFF)
    ops, codes, coeffs, x = inputs(case, seed)
    eng = engine((case["n"], case["reps"], case["gates"], case["pattern"]),
                 dict(n=case["n"], ops=ops, initial=None, count=x.shape[1]))
    ham = eng.set_hamiltonian(strings(codes), coeffs)
    return dict(case=case, eng=eng, ham=ham, held=Loaded(eng, ham, eng.free_hamiltonian), theta=torch.tensor(x, device=eng.device), seed=seed & 0xFFFF)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "energy":
        return state["eng"].energy(state["ham"], state["theta"], per_term=case["per_term"], check_status=False)
    if kind == "value_grad":
        return state["problem"].value_gradient(state["x"])
    if kind == "grad":
        return state["eng"].energy_grad(state["ham"], state["theta"])
    if kind == "partitions":
        if case["shots"]:
            return state["eng"].partition_sampled_energy(state["pset"], state["theta"], case["shots"], state["seed"], "philox",
                                                         copies=case["copies"], return_bits=True)
        return state["eng"].partition_energy(state["pset"], state["theta"], copies=case["copies"], check_status=False)
    if kind == "shots":
        return state["eng"].sampled_energy(state["ham"], state["theta"], case["shots"], state["seed"], case["rng"],
                                           case["mode"], per_term=True, check_status=False)
    loss = state["net"].train_step(state["batch"], state["target"], lr=1e-3)
    return dict(loss=loss, grad=state["net"].grad)


def work(case):
    """One multiply-add for each of the 256 numbers of a bond-16 environment at every site a word passes,
    three times that for a gradient; angles, words and coefficients read and the results written once."""
    kind = case["kind"]
    if kind == "train":
        nodes = case["graphs"] * (case["nmin"] + case["nmax"]) / 2
        edges = nodes * (case["nmin"] + case["nmax"]) / 2
        weights = sum(int(np.prod(s)) for s in weight_shapes())
        flops = 3 * 2 * (nodes * (4 * 128 + 3 * 256 * 128 + 128 * 5) + edges * 3 * 131 * 128)
        return dict(bytes=nodes * (4 + 5) * 4 + edges * (3 * 4 + 3 * 4) + weights * 4 * 7, flops=flops)
    if kind == "partitions":
        n, t = (case["nmin"] + case["nmax"]) / 2, (case["tmin"] + case["tmax"]) / 2
        states = case["parts"] * case["copies"]
        shot = states * case["shots"] * n
        return dict(bytes=states * (n * (case["reps"] + 1) * 8 + 8) + case["parts"] * t * (n / 4 + 8) + shot / 8,
                    flops=states * t * n * 512 + shot * 512)
    n, t, B = case["n"], case["terms"], case["batch"]
    P = n * (case["reps"] + 1) * (2 if case["gates"] == "ryrz" else 1)
    flops = B * t * n * 512.0 * (3 if kind in ("grad", "value_grad") else 1)
    out = B * 8 * (1 + (P if kind in ("grad", "value_grad") else 0) + (t if case.get("per_term") or kind == "shots" else 0))
    if kind == "shots":
        flops += B * case["shots"] * n * 512.0 * (t if case["mode"] == "plugin" else 1)
    return dict(bytes=B * P * 8 + t * (n / 4 + 8) + out, flops=flops)


# ---------------------------------------------------------------------------
# 64 bits, plain torch
# ---------------------------------------------------------------------------
def _sites(n, ops, x, dtype):
    """Site tensors [B, left, 2, right] of the circuit at angles x [B, P]; a CX copies its control
    into a new bond index and flips its target by it."""
    B = x.shape[0]
    A = [torch.zeros((B, 1, 2, 1), dtype=dtype, device=x.device) for _ in range(n)]
    for t in A:
        t[:, 0, 0, 0] = 1
    for op in ops:
        if op[0] == "cx":
            c, t = op[1], op[2]
            L = A[c]
            A[c] = torch.stack([L * torch.tensor([1, 0], dtype=dtype, device=x.device)[None, None, :, None],
                                L * torch.tensor([0, 1], dtype=dtype, device=x.device)[None, None, :, None]], dim=-1).flatten(-2)
            A[t] = torch.stack([A[t], A[t].flip(2)], dim=2).flatten(1, 2)
            continue
        h = x[:, op[2]] / 2
        if op[0] == "ry":
            U = torch.stack([torch.stack([h.cos(), -h.sin()], -1), torch.stack([h.sin(), h.cos()], -1)], -2).to(dtype)
        else:
            z = torch.zeros_like(h)
            U = torch.stack([torch.stack([torch.complex(h.cos(), -h.sin()), torch.complex(z, z)], -1),
                             torch.stack([torch.complex(z, z), torch.complex(h.cos(), h.sin())], -1)], -2)
        A[op[1]] = torch.einsum("bij,bljr->blir", U, A[op[1]])
    return A


PAULI = [np.eye(2), np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]]), np.array([[1, 0], [0, -1]])]


def _values(A, codes):
    """Re <P_t> [B, T] of every word: one environment per distinct prefix, closed against the rest's norm."""
    n = len(A)
    B, dev = A[0].shape[0], A[0].device
    dtype = A[0].dtype
    real = not dtype.is_complex
    right = [None] * (n + 1)
    right[n] = torch.ones((B, 1, 1), dtype=dtype, device=dev)
    for s in range(n - 1, -1, -1):
        right[s] = torch.einsum("baic,bcd,beid->bae", A[s].conj(), right[s + 1], A[s])
    last = np.where(codes.any(1), n - 1 - np.argmax(codes[:, ::-1] != 0, axis=1), -1)
    pieces, order = [], []
    none = np.nonzero(last < 0)[0]
    if none.size:
        pieces.append(right[0][:, 0, 0].real.unsqueeze(1).expand(B, none.size))
        order.append(none)
    active = np.nonzero(last >= 0)[0]
    node = np.zeros(active.size, dtype=np.int64)
    # real amplitudes: the environment is i^k times a real matrix, k the number of Y so far
    phase = np.zeros(1, dtype=np.int64)
    env = torch.ones((B, 1, 1, 1), dtype=dtype, device=dev)
    for s in range(n):
        key = node * 4 + codes[active, s]
        keys, node = np.unique(key, return_inverse=True)
        parent, code = keys // 4, keys % 4
        l, r = A[s].shape[1], A[s].shape[3]
        parts = []
        for c in range(4):
            k = np.nonzero(code == c)[0]
            if not k.size:
                continue
            if real:
                P = torch.tensor((PAULI[c] if c != 2 else np.array([[0, -1], [1, 0]])).real.copy(), dtype=dtype, device=dev)
            else:
                P = torch.tensor(PAULI[c].astype(complex), dtype=dtype, device=dev)
            PA = torch.einsum("ij,bajr->bair", P, A[s])
            E = env[:, torch.as_tensor(parent[k], device=dev)]
            S = torch.matmul(E.reshape(B, -1, l), PA.reshape(B, l, 2 * r)).reshape(B, k.size, l, 2, r)
            Y = torch.matmul(A[s].conj().reshape(B, 1, l * 2, r).transpose(2, 3), S.reshape(B, k.size, l * 2, r))
            parts.append((k, Y))
        where = np.argsort(np.concatenate([k for k, _ in parts]), kind="stable")
        new = torch.cat([y for _, y in parts], dim=1)[:, torch.as_tensor(where, device=dev)]
        phase = (phase[parent] + (code == 2)) % 4
        done = last[active] == s
        if done.any():
            nd = node[done]
            v = (new * right[s + 1].unsqueeze(1)).sum((2, 3))[:, torch.as_tensor(nd, device=dev)]
            if real:
                v = v * torch.tensor(np.array([1.0, 0.0, -1.0, 0.0])[phase[nd]], dtype=v.dtype, device=dev)
            pieces.append(v.real)
            order.append(active[done])
        active, node = active[~done], node[~done]
        if not active.size:
            break
        keep, node = np.unique(node, return_inverse=True)
        env, phase = new[:, torch.as_tensor(keep, device=dev)], phase[keep]
    inverse = np.argsort(np.concatenate(order), kind="stable")
    return torch.cat(pieces, dim=1)[:, torch.as_tensor(inverse, device=dev)]


def _energies(n, ops, gates, codes, coeffs, x):
    dtype = torch.float64 if gates == "ry" else torch.complex128
    step = max(1, int(4e5 // codes.shape[0]))
    vals = []
    with torch.no_grad():
        for b in range(0, x.shape[0], step):
            xb = torch.tensor(x[b:b + step], device=DEV)
            vals.append(_values(_sites(n, ops, xb, dtype), codes))
    v = torch.cat(vals)
    return v @ torch.tensor(coeffs, device=DEV), v


def _gradients(n, ops, gates, codes, coeffs, x):
    dtype = torch.float64 if gates == "ry" else torch.complex128
    order = np.lexsort(codes.T[::-1])
    es, gs = [], []
    step = 8
    for b in range(0, x.shape[0], step):
        xb = torch.tensor(x[b:b + step], device=DEV, requires_grad=True)
        A = _sites(n, ops, xb, dtype)
        leaf = [t.detach().requires_grad_(True) for t in A]
        e = torch.zeros(xb.shape[0], dtype=torch.float64, device=DEV)
        for t in range(0, order.size, 1000):
            w = order[t:t + 1000]
            part = _values(leaf, codes[w]) @ torch.tensor(coeffs[w], device=DEV)
            part.sum().backward()
            e += part.detach()
        torch.autograd.backward(A, [t.grad for t in leaf])
        es.append(e)
        gs.append(xb.grad)
    return torch.cat(es), torch.cat(gs)


def _training_step(graphs, target, weights):
    w = [torch.tensor(v, device=DEV, dtype=torch.float64, requires_grad=True) for v in weights]
    off, nodes, src, dst, feats = 0, [], [], [], []
    for node, index, ef in graphs:
        nodes.append(node)
        src.append(index[0] + off)
        dst.append(index[1] + off)
        feats.append(ef)
        off += node.shape[0]
    t = lambda v: torch.tensor(np.concatenate(v), device=DEV)  # noqa: E731
    src, dst, ef = t(src), t(dst), t(feats).double()
    x = torch.relu(t(nodes).double() @ w[0] + w[1])
    degree = torch.zeros(off, dtype=torch.float64, device=DEV).index_add_(0, dst, torch.ones(dst.numel(), dtype=torch.float64, device=DEV))
    for k in range(3):
        wm, bm, wu, bu = w[2 + 4 * k:6 + 4 * k]
        m = torch.relu(torch.cat([x[src], ef], 1) @ wm + bm)
        a = torch.zeros_like(x).index_add_(0, dst, m) / degree.clamp(min=1)[:, None]
        x = x + torch.relu(torch.cat([x, a], 1) @ wu + bu)
    theta = math.pi * torch.tanh(x @ w[14] + w[15])
    loss = (1 - torch.cos(theta - torch.tensor(target, device=DEV).double())).mean()
    loss.backward()
    return dict(loss=loss.detach().reshape(1), grad=torch.cat([v.grad.reshape(-1) for v in w]))


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _training_step(*graphs_of(case, seed))
    if kind == "partitions":
        if case["shots"]:
            return None          # a shot energy has no value apart from its draws
        es = []
        for n, ops, codes, coeffs, x in parts_of(case, seed):
            es.append(_energies(n, ops, case["gates"], codes, coeffs, x)[0])
        return torch.cat(es)
    if kind == "shots":
        return None
    ops, codes, coeffs, x = inputs(case, seed)
    if kind == "energy":
        e, v = _energies(case["n"], ops, case["gates"], codes, coeffs, x)
        return (e, v) if case["per_term"] else e
    e, g = _gradients(case["n"], ops, case["gates"], codes, coeffs, x)
    return (float(e[0]), g[0].cpu().numpy()) if kind == "value_grad" else (e, g)
