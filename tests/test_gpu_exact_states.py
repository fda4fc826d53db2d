"""GPU: the exact bond-doubling state that replaces the gate chain where its SVDs discard
nothing, against the dense state and the chain. Values are sums of products of components bounded by
1 over at most 16 x 16 bonds: 1e-11, the tolerance of the other dense comparisons."""
import numpy as np
import pytest

from oracle import mps_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vq(cuda_device):
    import vqemps
    return vqemps


def _circuits():
    rng = np.random.default_rng(31)
    chain = [("cx", q, q + 1) for q in range(4)]
    lay = lambda k: [(g, q, 10 * k + 2 * q + i) for q in range(5) for i, g in enumerate(("ry", "rz"))]  # noqa: E731
    yield "orders and directions mixed", lay(0) + chain + lay(1) + [("cx", 3, 2), ("cx", 1, 0)] + lay(2) + chain[::-1]
    yield "four CX on one bond", [("h", 0)] + [op for k in range(4) for op in (("rx", 1, k), ("cx", 0, 1))] + [("ry", 4, 4)]
    yield "more events than are staged at once", lay(0) + chain + [("ry", 2, int(k), 0.1) for k in rng.integers(0, 10, 90)] + \
        [("cx", 2, 1)] + [("rx", 2, 3)]
    yield "no CX", lay(0)


@pytest.mark.parametrize("order", ["msb", "qubit"])
def test_states_match_dense_and_sites_are_the_chains(vq, order):
    rng = np.random.default_rng(2)
    words = ["".join(rng.choice(list("IXYZ"), 5)) for _ in range(40)]
    coeffs = rng.normal(size=40)
    for name, ops in _circuits():
        got = []
        for mode in ("auto", "chain"):
            eng = vq.Engine(0, 16)
            eng.set_evolve_mode(mode)
            eng.set_level_variant("simt")
            eng.set_circuit(5, ops, site_order=order)
            x = np.random.default_rng(3).uniform(-np.pi, np.pi, (2, eng.P))
            _, pt = eng.energy(eng.set_hamiltonian(words, coeffs), x, per_term=True)
            got.append((pt.cpu().numpy(), [eng.sites(b) for b in range(2)]))
            eng.close()
        if all(len(op) == 3 for op in ops if op[0] != "h"):
            spec = dict(n=5, ops=ops, initial=None, count=x.shape[1])
            for b in range(2):
                ref = O.dense_expectations(O.dense_statevector(spec, x[b]), words).real
                np.testing.assert_allclose(got[0][0][b], ref, rtol=0, atol=1e-11, err_msg=name)
        np.testing.assert_allclose(got[0][0], got[1][0], rtol=0, atol=1e-11, err_msg=name)
        assert all(np.array_equal(a, b) for a, b in zip(got[0][1], got[1][1])), name


def test_states_that_fail(vq):
    """An angle that is not finite fails its state when a CX follows it on its site, as in the chain."""
    spec = O.hardware_efficient_spec(5, 2, ("ry",), "linear")
    x = np.random.default_rng(1).uniform(-1, 1, (3, spec["count"]))
    eng = vq.Engine(0, 16)
    eng.set_spec(spec)
    eng.set_level_variant("dmma3_pf")
    ham = eng.set_hamiltonian(["ZIIII", "IIXXI"], [1.0, 0.5])
    good = eng.energy(ham, x).cpu().numpy()
    x[1, 4] = np.inf
    with pytest.raises(vq.EngineError, match="nonfinite"):
        eng.energy(ham, x)
    with pytest.raises(vq.EngineError, match="nonfinite"):
        eng.sample(x, 10, 1)
    e = eng.energy(ham, x, check_status=False).cpu().numpy()
    assert np.isnan(e[1]) and e[0] == good[0] and e[2] == good[2]
    x[1, 4], x[1, -1] = 0.3, np.nan
    assert np.isnan(eng.energy(ham, x).cpu().numpy()[1])
    ps = eng.set_partitions([(5, spec["ops"], ["ZIIII"], [1.0])] * 3)
    x[1, -1], x[2, 0] = 0.1, np.nan
    with pytest.raises(vq.EngineError, match="nonfinite"):
        eng.partition_energy(ps, ps.pack_theta(x, device=eng.device))
    eng.close()


def test_bond_limits_keep_the_chain(vq):
    """A doubled bond above max_bond, where the compressed state still fits: 4 layers on 3 qubits."""
    spec = O.hardware_efficient_spec(3, 4, ("ry",), "linear")
    x = np.random.default_rng(5).uniform(-np.pi, np.pi, spec["count"])
    words = ["ZZI", "XIX", "YIY"]
    ref = O.dense_expectations(O.dense_statevector(spec, x), words).real
    for max_bond in (2, 4, 16):
        eng = vq.Engine(0, max_bond)
        eng.set_spec(spec)
        _, pt = eng.energy(eng.set_hamiltonian(words, [1.0, 1.0, 1.0]), x, per_term=True)
        np.testing.assert_allclose(pt[0].cpu().numpy(), ref, rtol=0, atol=1e-11)
        eng.close()
