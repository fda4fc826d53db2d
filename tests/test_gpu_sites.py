"""GPU: vqemps_copy_sites answers for the last call's angles, whatever call that was, and leaves that
call's statuses alone. The chain gives the same states bit for bit in every mode and batch size, so the
sites equal those of an energy call with a chain asked for by name."""
import numpy as np
import pytest

from oracle import mps_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vq(cuda_device):
    import vqemps
    return vqemps


LADDER = O.hardware_efficient_spec(6, 3, ("ry", "rz"), "linear")
OTHER = dict(n=5, initial=None, count=10, ops=[("ry", q, q) for q in range(5)] + [("cx", q, q + 1) for q in range(4)] +
             [("rx", q, 5 + q) for q in range(5)] + [("cx", 3, 2), ("cx", 1, 0)])


@pytest.mark.parametrize("variant", [None, "dmma"])
@pytest.mark.parametrize("spec", [LADDER, OTHER], ids=["ladder", "other"])
def test_sites_after_a_gradient_are_its_own(vq, spec, variant):
    rng = np.random.default_rng(4)
    n = spec["n"]
    words, coeffs = ["Z" * n, "X" + "I" * (n - 1)], [1.0, 0.5]
    first, x = rng.uniform(-np.pi, np.pi, (2, spec["count"])), rng.uniform(-np.pi, np.pi, (3, spec["count"]))
    ref = vq.Engine(0, 16)
    ref.set_evolve_mode("chain")
    ref.set_spec(spec)
    ref.energy(ref.set_hamiltonian(words, coeffs), x)
    want = [ref.sites(b) for b in range(3)]
    eng = vq.Engine(0, 16)
    eng.set_spec(spec)
    if variant:
        eng.set_grad_variant(variant)
    ham = eng.set_hamiltonian(words, coeffs)
    eng.energy(ham, first)
    eng.energy_grad(ham, x)
    for b in (2, 0, 1, 2):
        assert np.array_equal(eng.sites(b), want[b])
    e = eng.energy(ham, first[:1])
    assert not np.array_equal(eng.sites(0), want[0])
    assert e.item() == eng.energy(ham, first[:1]).item()
    with pytest.raises(vq.EngineError):
        eng.sites(1)
    ref.close()
    eng.close()


@pytest.mark.parametrize("call", ["energy", "energy_grad"])
def test_sites_leave_the_statuses_of_the_call(vq, call):
    """A gradient does not fail at an angle that is not finite (its values are NaN); the chain behind sites() does."""
    x = np.random.default_rng(1).uniform(-1, 1, (3, LADDER["count"]))
    x[1, 2] = np.nan
    eng = vq.Engine(0, 16)
    eng.set_spec(LADDER)
    ham = eng.set_hamiltonian(["ZZIIII"], [1.0])
    out = eng.energy(ham, x, check_status=False) if call == "energy" else eng.energy_grad(ham, x)[0]
    assert np.isnan(out[1].item())
    for _ in range(2):
        if call == "energy":
            with pytest.raises(vq.EngineError, match="nonfinite"):
                eng.check_status(3)
        else:
            assert eng.check_status(3) == [0, 0, 0]
        eng.sites(0)
        eng.sites(1)
    eng.close()
