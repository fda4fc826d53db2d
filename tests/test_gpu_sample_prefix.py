"""Shot prefixes shared through a table, and parities of 32 shots at a time.

A shot's bits depend on the state, the seed and its index only, so the first shots of a large call
(prefix table, one or two launches) equal those of a call too small for a table, bit for bit."""
import numpy as np
import pytest

from oracle import mps_oracle as O

pytestmark = pytest.mark.gpu


def _bits(packed):
    return packed.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("gates", [("ry",), ("ry", "rz")])
@pytest.mark.parametrize("n, shots", [(2, 64), (3, 5000), (11, 63), (11, 64), (13, 1000), (20, 5000), (70, 2100)])
def test_first_shots_do_not_depend_on_the_prefix_table(cuda_device, gates, n, shots):
    import vqemps
    rng = np.random.default_rng(n + shots)
    spec = O.hardware_efficient_spec(n, 3, gates, "linear")
    x = rng.uniform(-np.pi, np.pi, (2, spec["count"]))
    eng = vqemps.Engine(0, 16)
    eng.set_spec(spec)
    for kind in ("splitmix", "philox"):
        many = _bits(eng.sample(x, shots, 11, kind))
        few = _bits(eng.sample(x, 40, 11, kind))
        assert many.shape[1] == shots
        assert np.array_equal(many[:, :40], few)


@pytest.mark.parametrize("n, shots", [(5, 31), (9, 512), (12, 513), (66, 1000)])
def test_parity_sums_equal_host_popcounts(cuda_device, n, shots):
    """Z words of weight 1 to n over shared shots; counts are whole numbers, so per-term values are equal."""
    import vqemps
    rng = np.random.default_rng(shots)
    spec = O.hardware_efficient_spec(n, 2, ("ry",), "linear")
    masks = rng.random((300, n)) < rng.random((300, 1))
    masks[0], masks[1] = True, False
    masks[1, n - 1] = True
    words = ["".join("Z" if z else "I" for z in m) for m in masks]
    eng = vqemps.Engine(0, 16)
    eng.set_spec(spec)
    ham = eng.set_hamiltonian(words, np.ones(len(words)))
    x = rng.uniform(-np.pi, np.pi, (1, spec["count"]))
    out = eng.sampled_energy(ham, x, shots, 5, "philox", mode="shared", per_term=True)
    pt = out[1].cpu().numpy()[0]
    packed = _bits(eng.sample(x, shots, 5, "philox"))[0]
    bits = np.array([(packed[:, q >> 6] >> np.uint64(q & 63)) & np.uint64(1) for q in range(n)]).T.astype(int)
    for t, m in enumerate(masks):
        assert pt[t] == np.sum(1 - 2 * (bits[:, m].sum(axis=1) % 2)) / shots
