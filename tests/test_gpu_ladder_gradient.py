"""GPU: ladder gradient kernels against the oracle's adjoint gradient, the level kernels and
themselves. Tolerance: a derivative is a sum over words of c times a value bounded by 1
(rotations by half angles), computed to 1e-12 like the values themselves."""
import numpy as np
import pytest
import torch

from oracle import mps_oracle as O
from oracle import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vq(cuda_device):
    import vqemps
    return vqemps


def _grad(vq, spec, words, coeffs, x, order="msb", variant=None):
    eng = vq.Engine(0, 16)
    if variant:
        eng.set_grad_variant(variant)
    eng.set_spec(spec, site_order=order)
    e, g = eng.energy_grad(eng.set_hamiltonian(words, coeffs), np.atleast_2d(x))
    out = e.cpu().numpy(), g.cpu().numpy()
    eng.close()
    return out


@pytest.mark.parametrize("gates", [("ry",), ("ry", "rz"), ("rx", "rz")])
@pytest.mark.parametrize("pattern", ["linear", "reverse_linear"])
@pytest.mark.parametrize("order", ["msb", "qubit"])
def test_ladder_gradient_matches_oracle(vq, gates, pattern, order):
    rng = np.random.default_rng(17)
    for n, reps, initial in ((2, 4, None), (3, 1, "+"), (5, 2, "1"), (6, 3, "-"), (9, 4, None)):
        spec = O.hardware_efficient_spec(n, reps, gates, pattern)
        spec["initial"] = initial
        words, coeffs = W.random_hamiltonian(rng, n, 50, min(n, 4), z_fraction=0.4)
        words += ["I" * n, words[0], "X" + "I" * (n - 1), "I" * (n - 1) + "Z"]
        coeffs = np.append(coeffs, rng.normal(size=4))
        x = rng.uniform(-np.pi, np.pi, (2, spec["count"]))
        e, g = _grad(vq, spec, words, coeffs, x, order)
        tol = 1e-12 * np.abs(coeffs).sum()
        for b in range(2):
            ref, gref = O.reverse_value_gradient(spec, words, coeffs, x[b])
            assert abs(e[b] - ref) <= tol
            np.testing.assert_allclose(g[b], gref, rtol=0, atol=tol)


def test_constant_gates_scales_and_shared_parameters(vq):
    """Fixed gates in a layer, rotations with a scale or a constant angle, a parameter used twice."""
    rng = np.random.default_rng(23)
    n, ops = 4, []
    chain = [("cx", q, q + 1) for q in range(n - 1)]
    for layer in range(2):
        for q in range(n):
            ops += [("h", q), ("ry", q, (layer * n + q) % 6, 0.7), ("z", q), ("rx", q, 6 + q), ("ry", q, None, 0.3), ("s", q)]
        ops += chain
    ops += [("rz", q, 2, -1.3) for q in range(n)]
    words, coeffs = W.random_hamiltonian(rng, n, 30, 4, z_fraction=0.3)
    eng = vq.Engine(0, 16)
    eng.set_circuit(n, ops)
    ham = eng.set_hamiltonian(words, coeffs)
    assert eng.level_variant(ham, 1) == "ladder"
    x = rng.uniform(-np.pi, np.pi, (3, eng.P))
    e, g = (v.cpu().numpy() for v in eng.energy_grad(ham, x))
    eng.set_grad_variant("dmma")
    e0, g0 = (v.cpu().numpy() for v in eng.energy_grad(ham, x))
    tol = 1e-11 * np.abs(coeffs).sum()
    np.testing.assert_allclose(e, e0, rtol=0, atol=tol)
    np.testing.assert_allclose(g, g0, rtol=0, atol=tol)
    eng.close()


@pytest.mark.parametrize("gates", [("ry",), ("ry", "rz")])
def test_ladder_gradient_does_not_depend_on_batch_and_agrees_over_lists(vq, monkeypatch, gates):
    """Within a task list the bits do not depend on the batch; lists sum a site's steps in other orders."""
    rng = np.random.default_rng(29)
    n = 12
    spec = O.hardware_efficient_spec(n, 4, gates, "linear")
    words, coeffs = W.random_hamiltonian(rng, n, 300, 5)
    x = rng.uniform(-np.pi, np.pi, (35, spec["count"]))
    e0, g0 = _grad(vq, spec, words, coeffs, x[:8], variant="dmma")
    tol = 1e-11 * np.abs(coeffs).sum()
    for name in ("0", "1", "2"):
        monkeypatch.setenv("VQEMPS_LADDER_LIST", name)
        e, g = _grad(vq, spec, words, coeffs, x)
        np.testing.assert_allclose(e[:8], e0, rtol=0, atol=tol)
        np.testing.assert_allclose(g[:8], g0, rtol=0, atol=tol)
        for B in (1, 5, 9):
            eb, gb = _grad(vq, spec, words, coeffs, x[:B])
            assert np.array_equal(eb, e[:B]) and np.array_equal(gb, g[:B])


def test_ladder_gradient_passes_split_large_batches(vq):
    """More states than one pass holds (16 GB): 64 qubits, 20,000 words."""
    from vqemps import workloads as VW
    spec, words, coeffs, x = VW.gradient_64q(seed=3, batch=4)
    eng = vq.Engine(0, 16)
    eng.set_spec(spec)
    ham = eng.set_hamiltonian(words, coeffs)
    B = 150
    e, g = eng.energy_grad(ham, torch.tensor(np.tile(x, (B // 4 + 1, 1))[:B], device=eng.device))
    e, g = e.cpu().numpy(), g.cpu().numpy()
    assert np.array_equal(e[:4], e[144:148]) and np.array_equal(g[:4], g[144:148])
    eng.set_grad_variant("dmma3")
    e0, g0 = (v.cpu().numpy() for v in eng.energy_grad(ham, x[:2]))
    np.testing.assert_allclose(e[:2], e0, rtol=1e-10)
    np.testing.assert_allclose(g[:2], g0, rtol=0, atol=1e-10 * np.abs(g0).max())
    eng.close()


def test_gradient_at_angles_that_are_not_finite(vq):
    spec = O.hardware_efficient_spec(5, 2, ("ry",), "linear")
    words, coeffs = ["ZZIII", "IIXXI"], np.array([1.0, 0.25])
    x = np.random.default_rng(1).uniform(-1, 1, (3, spec["count"]))
    good = _grad(vq, spec, words, coeffs, x)
    x[1, 2] = np.nan
    e, g = _grad(vq, spec, words, coeffs, x)
    assert np.isnan(e[1]) and np.isnan(g[1]).all()
    for b in (0, 2):
        assert e[b] == good[0][b] and np.array_equal(g[b], good[1][b])


@pytest.mark.parametrize("gates", [("ry",), ("ry", "rz")])
@pytest.mark.parametrize("count, B", [(2, 1), (3, 1), (16, 3), (17, 1), (300, 8)])
def test_many_words_that_close_at_one_step(vq, gates, count, B):
    """Words in one half close at the identity chain's steps: few directly, more in sums of chunks of
    16 and sums of those. Against the level kernels."""
    n = 14
    rng = np.random.default_rng(count)
    spec = O.hardware_efficient_spec(n, 3, gates, "linear")
    tails = sorted({"".join(rng.choice(list("XYZ"), 4)) + "".join(rng.choice(list("IXYZ"), 5))
                    for _ in range(4 * count)})[:count]
    words = ["I" * 5 + t for t in tails] + [("I" * 5 + t)[::-1] for t in tails] + ["ZZ" + "I" * 12]
    coeffs = rng.normal(size=len(words))
    x = rng.uniform(-np.pi, np.pi, (B, spec["count"]))
    e, g = _grad(vq, spec, words, coeffs, x)
    e1, g1 = _grad(vq, spec, words, coeffs, x, variant="dmma")
    tol = 1e-12 * np.abs(coeffs).sum()
    np.testing.assert_allclose(e, e1, rtol=0, atol=tol)
    np.testing.assert_allclose(g, g1, rtol=0, atol=tol)


@pytest.mark.parametrize("gates, n, terms", [(("ry",), 40, 5000), (("ry", "rz"), 30, 3000)])
def test_default_gradients_do_not_depend_on_the_batch(vq, gates, n, terms):
    """Problems large enough for each task list to be the fastest at some batch size: the same bits for all."""
    rng = np.random.default_rng(41)
    spec = O.hardware_efficient_spec(n, 4, gates, "linear")
    words, coeffs = W.random_hamiltonian(rng, n, terms, 5)
    x = rng.uniform(-np.pi, np.pi, (32, spec["count"]))
    e, g = _grad(vq, spec, words, coeffs, x)
    for B in (1, 3, 8):
        eb, gb = _grad(vq, spec, words, coeffs, x[:B])
        assert np.array_equal(eb, e[:B]) and np.array_equal(gb, g[:B]), B


def test_captured_gradient_after_a_larger_batch(vq):
    """What a call of a larger batch has allocated and made serves a smaller one: it can be captured at once."""
    spec, words, coeffs, x = W.batched_40q(seed=2, batch=32)
    eng = vq.Engine(0, 16)
    eng.set_spec(spec)
    ham = eng.set_hamiltonian(words, coeffs)
    th = torch.tensor(x, device=eng.device)
    e, g = eng.energy_grad(ham, th)
    small, out = th[:2].clone(), []
    graph = eng.capture(lambda: out.append(eng.energy_grad(ham, small)), warmup=0)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out[0][0], e[:2]) and torch.equal(out[0][1], g[:2])
    del graph
    eng.close()


def test_checkpointing_asked_for_runs_the_kernels_that_checkpoint(vq):
    """An interval set by the caller is kept to: the level kernels', bit for bit (vqemps_set_grad_checkpoint)."""
    spec, words, coeffs, x = W.plain_12q(6)
    x = np.stack([x, -x])
    out = []
    for asked in ((), ("checkpoint",), ("variant",), ("variant", "checkpoint")):
        eng = vq.Engine(0, 16)
        eng.set_spec(spec)
        if "variant" in asked:
            eng.set_grad_variant("dmma3")
        if "checkpoint" in asked:
            eng.set_grad_checkpoint(3)
        e, g = eng.energy_grad(eng.set_hamiltonian(words, coeffs), x)
        out.append((e.cpu().numpy(), g.cpu().numpy()))
        eng.close()
    for e, g in out[2:]:
        assert np.array_equal(e, out[1][0]) and np.array_equal(g, out[1][1])
    assert not np.array_equal(out[0][1], out[1][1])
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=0, atol=1e-11 * np.abs(coeffs).sum())


@pytest.mark.parametrize("gates", [("ry",), ("ry", "rz")])
def test_gradient_of_sums_without_closures(vq, gates):
    """Identity words and, with real gates, words with an odd number of Y: nothing to walk, derivatives of zero."""
    spec = O.hardware_efficient_spec(4, 2, gates, "linear")
    x = np.random.default_rng(2).uniform(-np.pi, np.pi, (3, spec["count"]))
    words = ["IIII", "IIII"] + (["YIII", "IYZX"] if gates == ("ry",) else [])
    e, g = _grad(vq, spec, words, np.arange(1.0, 1.0 + len(words)), x)
    np.testing.assert_allclose(e, np.full(3, 3.0), rtol=0, atol=1e-14)
    assert np.array_equal(g, np.zeros_like(g))


def test_first_gradient_on_the_next_pauli_sum_allocates_nothing(vq):
    """Its task list is made with the sum, and buffers that have grown once hold a little more: the first call can be
    captured."""
    rng = np.random.default_rng(8)
    spec = O.hardware_efficient_spec(30, 4, ("ry",), "linear")
    eng = vq.Engine(0, 16)
    eng.set_spec(spec)
    th = torch.tensor(rng.uniform(-np.pi, np.pi, (8, spec["count"])), device=eng.device)
    for terms in (1500, 2600):
        eng.energy_grad(eng.set_hamiltonian(*W.random_hamiltonian(rng, 30, terms, 5)), th)
    ham = eng.set_hamiltonian(*W.random_hamiltonian(rng, 30, 2680, 5))
    out = []
    graph = eng.capture(lambda: out.append(eng.energy_grad(ham, th)), warmup=0)
    graph.replay()
    torch.cuda.synchronize()
    e, g = eng.energy_grad(ham, th)
    assert torch.equal(out[0][0], e) and torch.equal(out[0][1], g)
    del graph
    eng.close()
