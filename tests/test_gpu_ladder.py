"""GPU: ladder kernels (environments as Pauli components, no site tensors) against the
oracle's bond-doubling state, the gate chain's kernels and themselves.

Tolerance: a value is a sum of at most 256 products of components bounded by 1, each
the result of at most 5 n fused operations, so its error stays below 256 * 5 n * eps / 2,
2e-12 at the widest state here; 1e-12 is what all variants promise per term."""
import numpy as np
import pytest
import torch

from oracle import mps_oracle as O
from oracle import workloads as W

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.fixture(scope="module")
def vq(cuda_device):
    import vqemps
    return vqemps


def _words(rng, n, count):
    words = ["I" * n, "Z" * n, "X" + "I" * (n - 1), "I" * (n - 1) + "Y", "Y" * n]
    for _ in range(count):
        words.append("".join(rng.choice(list("IIIXYZ"), n)))
    return words + words[:2]


def _energy(vq, spec, words, coeffs, x, order="msb"):
    eng = vq.Engine(0, 16)
    eng.set_spec(spec, site_order=order)
    ham = eng.set_hamiltonian(words, coeffs)
    x = np.atleast_2d(x)
    assert eng.level_variant(ham, x.shape[0]) == "ladder"
    e, pt = eng.energy(ham, x, per_term=True)
    out = e.cpu().numpy(), pt.cpu().numpy()
    eng.close()
    return out


@pytest.mark.parametrize("gates", [("ry",), ("ry", "rz"), ("rx", "rz")])
@pytest.mark.parametrize("pattern", ["linear", "reverse_linear"])
@pytest.mark.parametrize("order", ["msb", "qubit"])
def test_ladder_values_match_bond_doubling_state(vq, gates, pattern, order):
    rng = np.random.default_rng(7)
    for n, reps, initial in ((2, 4, None), (3, 1, "+"), (5, 2, "1"), (6, 3, "-"), (11, 4, None)):
        spec = O.hardware_efficient_spec(n, reps, gates, pattern)
        spec["initial"] = initial
        words = _words(rng, n, 40)
        coeffs = rng.normal(size=len(words))
        x = rng.uniform(-np.pi, np.pi, (3, spec["count"]))
        e, pt = _energy(vq, spec, words, coeffs, x, order)
        for b in range(3):
            ref = O.expect_words(O.bond_doubling_sites(spec, x[b]), words).real
            np.testing.assert_allclose(pt[b], ref, rtol=0, atol=TOL)
            assert abs(e[b] - coeffs @ ref) <= TOL * np.abs(coeffs).sum()


@pytest.mark.parametrize("gates", [("ry",), ("ry", "rz")])
def test_ladder_values_do_not_depend_on_task_list_or_batch(vq, monkeypatch, gates):
    rng = np.random.default_rng(11)
    n = 13
    spec = O.hardware_efficient_spec(n, 4, gates, "linear")
    words, coeffs = W.random_hamiltonian(rng, n, 400, 5)
    x = rng.uniform(-np.pi, np.pi, (19, spec["count"]))
    out = []
    for name in ("0", "1", "2"):
        monkeypatch.setenv("VQEMPS_LADDER_LIST", name)
        for B in (1, 2, 7, 8, 19):
            out.append((B, _energy(vq, spec, words, coeffs, x[:B])))
    ref = out[-1][1]
    for B, (e, pt) in out:
        assert np.array_equal(e, ref[0][:B]) and np.array_equal(pt, ref[1][:B])
    monkeypatch.delenv("VQEMPS_LADDER_LIST")
    eng = vq.Engine(0, 16)
    eng.set_evolve_mode("chain")
    eng.set_level_variant("dmma3_pf")
    eng.set_spec(spec)
    _, pt = eng.energy(eng.set_hamiltonian(words, coeffs), x, per_term=True)
    np.testing.assert_allclose(ref[1], pt.cpu().numpy(), rtol=0, atol=1e-11)


def test_ladder_passes_split_large_batches(vq):
    """More states than one pass holds (the environments of a pass stay within 8 GB)."""
    spec, words, coeffs, x = W.batched_40q(2, batch=8)
    eng = vq.Engine(0, 16)
    eng.set_spec(spec)
    ham = eng.set_hamiltonian(words, coeffs)
    slots = eng.ladder_info(ham, 8)["slots"]
    B = 2 * int((8 << 30) // (slots * 4 * 36 * 8)) + 5
    th = torch.tensor(np.tile(x, (B // 8 + 1, 1))[:B], device=eng.device)
    e = eng.energy(ham, th).cpu().numpy()
    ref = eng.energy(ham, x).cpu().numpy()
    assert np.array_equal(e, np.tile(ref, B // 8 + 1)[:B])
    eng.close()


def test_circuits_that_are_not_ladders_keep_their_kernels(vq):
    rng = np.random.default_rng(3)
    u = np.linalg.qr(rng.normal(size=(2, 2)))[0]
    lay = lambda k: [("ry", q, 4 * k + q) for q in range(4)]  # noqa: E731
    chain = [("cx", 0, 1), ("cx", 1, 2), ("cx", 2, 3)]
    other = {
        "direction changes": lay(0) + chain + lay(1) + [("cx", 1, 0), ("cx", 2, 1), ("cx", 3, 2)],
        "a gate between the two CX of a site": lay(0) + [chain[0], ("ry", 1, 4), chain[1], chain[2]],
        "a bond without CX": lay(0) + [chain[0], chain[2]] + lay(1),
        "order changes": lay(0) + chain + lay(1) + chain[::-1],
        "a user's matrix": lay(0) + chain + [("u1", 2, u)],
        "no CX": lay(0),
    }
    words = _words(rng, 4, 30)
    coeffs = rng.normal(size=len(words))
    for name, ops in other.items():
        eng = vq.Engine(0, 16)
        eng.set_circuit(4, ops)
        ham = eng.set_hamiltonian(words, coeffs)
        assert eng.level_variant(ham, 2) != "ladder", name
        x = rng.uniform(-np.pi, np.pi, (2, eng.P))
        _, pt = eng.energy(ham, x, per_term=True)
        named = [op for op in ops if op[0] != "u1"]
        if len(named) == len(ops):
            spec = dict(n=4, ops=ops, initial=None, count=eng.P)
            ref = O.dense_expectations(O.dense_statevector(spec, x[1]), words).real
            np.testing.assert_allclose(pt[1].cpu().numpy(), ref, rtol=0, atol=1e-11)
        eng.close()
    spec = O.hardware_efficient_spec(4, 2, ("ry",), "linear")
    for make in (lambda e: e.set_evolve_mode("pair"), lambda e: e.set_split_mode("off"),
                 lambda e: e.set_level_variant("dmma3_pf")):
        eng = vq.Engine(0, 16)
        make(eng)
        eng.set_spec(spec)
        assert eng.level_variant(eng.set_hamiltonian(words, coeffs), 1) != "ladder"
        eng.close()
    for args in ((2, 0.0, 0.0), (16, 1e-9, 0.0), (16, 0.0, 1e-9)):        # bond 4 needed; cutoffs
        eng = vq.Engine(0, *args)
        eng.set_spec(spec)
        assert eng.level_variant(eng.set_hamiltonian(words, coeffs), 1) != "ladder"
        eng.close()


def test_sites_after_ladder_energies_are_the_gate_chains(vq):
    rng = np.random.default_rng(5)
    spec = O.hardware_efficient_spec(9, 3, ("ry",), "reverse_linear")
    x = rng.uniform(-np.pi, np.pi, (4, spec["count"]))
    got = []
    for mode in ("auto", "chain"):
        eng = vq.Engine(0, 16)
        eng.set_evolve_mode(mode)
        eng.set_spec(spec)
        eng.energy(eng.set_hamiltonian(["ZIIIIIIIZ"], [1.0]), x)
        got.append([eng.sites(b) for b in range(4)])
        eng.close()
    assert all(np.array_equal(a, b) for a, b in zip(*got))


def test_angles_that_are_not_finite(vq):
    """Before a site's last CX they fail the state (as the gate chain's SVD does), after it
    every value is NaN; the other states of the batch are untouched."""
    spec = O.hardware_efficient_spec(5, 2, ("ry",), "linear")
    words, coeffs = ["ZIIII", "IIIII", "IIXXI"], np.array([1.0, 0.5, 0.25])
    x = np.random.default_rng(1).uniform(-1, 1, (3, spec["count"]))
    eng = vq.Engine(0, 16)
    eng.set_spec(spec)
    ham = eng.set_hamiltonian(words, coeffs)
    good = eng.energy(ham, x).cpu().numpy()
    bad = x.copy()
    bad[1, 3] = np.nan
    with pytest.raises(vq.EngineError, match="nonfinite"):
        eng.energy(ham, bad)
    e = eng.energy(ham, bad, check_status=False).cpu().numpy()
    assert np.isnan(e[1]) and e[0] == good[0] and e[2] == good[2]
    late = x.copy()
    late[1, -1] = np.inf
    e, pt = eng.energy(ham, late, per_term=True)
    e, pt = e.cpu().numpy(), pt.cpu().numpy()
    assert np.isnan(e[1]) and np.isnan(pt[1]).all() and e[0] == good[0] and e[2] == good[2]
    eng.close()


def test_split_evaluation_asked_for_runs_as_asked(vq):
    """vqemps_set_split_mode: 'on' is the split plan and 'off' the prefix plan, for energies, gradients and the analytic
    words of a shot estimate alike; the ladder kernels answer where the choice is left to the engine."""
    rng = np.random.default_rng(6)
    spec = O.hardware_efficient_spec(9, 3, ("ry", "rz"), "linear")
    words, coeffs = W.random_hamiltonian(rng, 9, 60, 3, z_fraction=0.4)
    x = rng.uniform(-np.pi, np.pi, (2, spec["count"]))
    out = {}
    for mode in ("on", "off", "auto"):
        eng = vq.Engine(0, 16)
        eng.set_spec(spec)
        eng.set_split_mode(mode)
        ham = eng.set_hamiltonian(words, coeffs)
        assert (eng.level_variant(ham, 2) == "ladder") == (mode == "auto")
        assert (eng.plan_stats(ham)["cut"] >= 0) or mode != "on"
        _, g = eng.energy_grad(ham, x)
        eng.set_grad_variant("dmma3")
        _, g3 = eng.energy_grad(ham, x)
        assert torch.equal(g, g3) == (mode != "auto")
        _, pt = eng.sampled_energy(ham, x, 300, 5, "philox", "shared", per_term=True)
        out[mode] = pt.cpu().numpy()
        eng.close()
    for mode in ("on", "off"):
        np.testing.assert_allclose(out[mode], out["auto"], rtol=0, atol=1e-11)


def test_autotuner_at_40_qubits(vq):
    """A circuit that is no ladder (CX in both directions): the level kernels are tuned, among them the real ones."""
    n, count = 40, 0
    _, words, coeffs, _ = W.batched_40q(0, batch=1)
    ops = []
    for layer in range(4):
        ops += [("ry", q, count + q) for q in range(n)]
        ops += [("cx", q, q + 1) if layer % 2 else ("cx", q + 1, q) for q in range(n - 1)]
        count += n
    spec = dict(n=n, ops=ops, initial=None, count=count)
    x = np.random.default_rng(9).uniform(-np.pi, np.pi, (16, count))
    eng = vq.Engine(0, 16)
    eng.set_spec(spec)
    ham = eng.set_hamiltonian(words, coeffs)
    e = eng.energy(ham, x).cpu().numpy()
    assert eng.level_variant(ham, 16) in set(vq.Engine.LEVEL_VARIANTS) - {"ladder"}
    for b in (0, 9):
        ref = float(np.dot(O.expect_words(O.svd_evolve(spec, x[b], 16), words).real, coeffs))
        assert abs(e[b] - ref) <= 1e-9 * max(1.0, abs(ref))
    eng.close()


def test_workspace_budget(vq, monkeypatch):
    """VQEMPS_LADDER_BYTES: passes of fewer states (one at least) give the same bits; where a gradient's state does not
    fit, the level kernels answer. A state takes some 220 KB for an energy and 730 KB for a gradient here."""
    spec, words, coeffs, x = W.plain_12q(3)
    x = x * np.linspace(0.2, 1.0, 19)[:, None]
    out = []
    for budget, variant in ((None, None), (str(1500 << 10), None), (str(7 << 20), None), ("1", None), (None, "dmma3")):
        monkeypatch.delenv("VQEMPS_LADDER_BYTES", raising=False)
        if budget:
            monkeypatch.setenv("VQEMPS_LADDER_BYTES", budget)
        eng = vq.Engine(0, 16)
        if variant:
            eng.set_grad_variant(variant)
        eng.set_spec(spec)
        ham = eng.set_hamiltonian(words, coeffs)
        e, pt = eng.energy(ham, x, per_term=True)
        eg, g = eng.energy_grad(ham, x)
        out.append([v.cpu().numpy() for v in (e, pt, eg, g)])
        eng.close()
    for got in out[1:]:
        assert np.array_equal(got[0], out[0][0]) and np.array_equal(got[1], out[0][1])
    for got in out[1:3]:
        assert np.array_equal(got[2], out[0][2]) and np.array_equal(got[3], out[0][3])
    assert np.array_equal(out[3][2], out[4][2]) and np.array_equal(out[3][3], out[4][3])
    assert not np.array_equal(out[0][3], out[4][3])


@pytest.mark.parametrize("gates", [("ry",), ("ry", "rz"), ("rx", "h", "s")])
@pytest.mark.parametrize("pattern", ["linear", "reverse_linear"])
@pytest.mark.parametrize("order", ["msb", "qubit"])
def test_clifford_circuits_give_whole_numbers(vq, gates, pattern, order):
    """At angles of zero every gate's Bloch matrix has entries of 0 and +-1, so every value is -1, 0 or 1 without
    rounding, whichever axis the bonds take (rotations from half angles or a rounded H leave a bias per layer)."""
    n, L, ops, k = 40, 4, [], 0
    pairs = [(q, q + 1) for q in range(n - 1)][::1 if pattern == "linear" else -1]
    for layer in range(L + 1):
        for q in range(n):
            for g in gates:
                if g in ("h", "s"):
                    ops.append((g, q))
                else:
                    ops.append((g, q, k))
                    k += 1
        if layer < L:
            ops += [("cx", a, b) for a, b in pairs]
    eng = vq.Engine(0, 16)
    eng.set_circuit(n, ops, site_order=order)
    words = _words(np.random.default_rng(3), n, 200)
    ham = eng.set_hamiltonian(words, np.ones(len(words)))
    assert eng.level_variant(ham, 1) == "ladder"
    _, pt = eng.energy(ham, np.zeros((2, eng.P)), per_term=True)
    v = pt.cpu().numpy()
    assert np.array_equal(v, np.rint(v)) and np.abs(v).max() == 1.0
    if gates[0] == "ry":                               # the state stays |0 .. 0>
        assert np.array_equal(v[0], [float(set(w) <= set("IZ")) for w in words])
    eng.close()
