"""GPU: the network's products at the sizes where their tiles and splits change -- more
edge rows than 148 tiles of 64, rows that fill no tile, graphs without edges -- against the numpy
oracle with the same BF16 operand rounding and the tolerances of the other network tests."""
import numpy as np
import pytest
import torch

from oracle import mpnn_oracle as MO

pytestmark = pytest.mark.gpu


def _graph(rng, n, pairs):
    a, b = np.triu_indices(n, 1)
    keep = rng.permutation(a.size)[:pairs]
    a, b = a[keep], b[keep]
    index = np.array([np.stack([a, b], 1).reshape(-1), np.stack([b, a], 1).reshape(-1)]).reshape(2, -1)
    return (rng.normal(size=(n, 4)).astype(np.float32), index.astype(np.int64),
            np.repeat(0.5 * rng.normal(size=(a.size, 3)), 2, axis=0).astype(np.float32))


@pytest.mark.parametrize("sizes", [((40, 780),) * 7, ((17, 1), (3, 0)), ((9, 0),), ((2, 1),), ((48, 1128),) * 3])
def test_products_match_oracle_at_tile_edges(cuda_device, sizes):
    from vqemps import mpnn
    rng = np.random.default_rng(len(sizes) + sizes[0][0])
    net = mpnn.MPNN(0, seed=4)
    flat = net.params().astype(np.float64)
    flat[np.abs(flat) < 1e-12] = 0.01
    net.set_params(flat.astype(np.float32))
    flat = net.params().astype(np.float64)
    batch = mpnn.make_batch([_graph(rng, n, m) for n, m in sizes], net.device)
    h = batch.host
    g = dict(node=h["node"].astype(np.float64), src=h["src"], dst=h["dst"], ef=h["ef"].astype(np.float64))
    p, names = MO.unflatten(flat)
    theta = net.forward(batch).cpu().numpy()
    ref, cache = MO.forward(p, 3, g, bf16=True)
    assert np.linalg.norm(theta - ref) <= 2e-3 * np.linalg.norm(ref)
    dtheta = rng.normal(size=theta.shape).astype(np.float32)
    grad = net.backward(batch, torch.tensor(dtheta, device=net.device)).cpu().numpy()
    ref_g = MO.backward(p, 3, g, cache, dtheta.astype(np.float64), bf16=True)
    o = 0
    for name in names:
        want = ref_g[name].reshape(-1)
        assert np.linalg.norm(grad[o:o + want.size] - want) <= 1e-2 * np.linalg.norm(want) + 1e-30, name
        o += want.size
