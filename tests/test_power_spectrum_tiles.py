"""Power spectrum values alone with a warp per centre, at the edges of its
tiles: one to five species (four are the most it takes), one to nine radial
functions (eight are), odd counts, centres that miss some species, one centre
and more than a CTA holds.

Against the FP64 dense form, whose contraction is a kernel of its own: 1e-12
of the largest value (sums of at most 17 products at 1e-16 each, and
coefficients that agree to 1e-14).
"""
import numpy as np
import pytest

import rascaline_b200 as rb
from rascaline_b200 import workloads

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from rascaline_b200 import torch_api  # noqa: E402

TYPES = (1, 6, 7, 8, 9)


@pytest.mark.parametrize("atoms,species,max_radial,max_angular", [
    (1, 1, 0, 0), (8, 1, 7, 8), (9, 2, 2, 3), (33, 3, 7, 6), (40, 4, 7, 6), (40, 4, 4, 5), (25, 3, 8, 4), (30, 5, 7, 2),
])
def test_values(atoms, species, max_radial, max_angular):
    rng = np.random.default_rng(atoms)
    types = rng.permutation([TYPES[k % species] for k in range(atoms)])
    positions = rng.uniform(0.0, 2.2 * atoms ** (1 / 3), (atoms, 3))
    calculator = rb.SoapPowerSpectrum(**workloads.hypers(2.6, max_radial, max_angular))
    system = workloads.system_dict(types, positions, np.zeros((3, 3)))
    result = calculator.compute([system])
    dense, _ = torch_api.dense_power_spectrum(calculator, torch.tensor(positions, device="cuda"), types,
                                              np.zeros((1, 9)), [atoms], 64)
    dense = dense.cpu().numpy()
    present = sorted(set(types.tolist()))
    pairs = [(a, b) for i, a in enumerate(present) for b in present[i:]]
    seen = np.zeros(dense.shape[:2], dtype=bool)
    for key, block in zip(result.keys.values.tolist(), result.blocks()):
        pair = pairs.index((key[1], key[2]))
        rows = np.asarray(block.samples.values)[:, 1]
        expected = dense[rows, pair].reshape(np.asarray(block.values).shape)
        np.testing.assert_allclose(block.values, expected, rtol=0.0, atol=1e-12 * np.abs(dense).max())
        seen[rows, pair] = True
    np.testing.assert_array_equal(dense[~seen], 0.0)


def test_every_slot_of_many_centres():
    """Rows of one to ten slots a centre, thousands of warps in flight: no part
    of a tile is dropped, and repeated calls agree to the last bit."""
    systems = workloads.molecules(256, seed=3)
    sizes = [len(m["types"]) for m in systems]
    types = np.concatenate([m["types"] for m in systems])
    positions = np.concatenate([m["positions"] for m in systems])
    calculator = rb.SoapPowerSpectrum(**workloads.hypers(3.0, 7, 3))
    dense, _ = torch_api.dense_power_spectrum(calculator, torch.tensor(positions, device="cuda"), types,
                                              np.zeros((len(sizes), 9)), sizes, 64)
    dense = dense.cpu().numpy()
    start = np.concatenate([[0], np.cumsum(sizes)])
    present = sorted(set(types.tolist()))
    pairs = [(a, b) for i, a in enumerate(present) for b in present[i:]]
    first = None
    for _ in range(3):
        result = calculator.compute(systems)
        found = np.zeros_like(dense)
        for key, block in zip(result.keys.values.tolist(), result.blocks()):
            samples = np.asarray(block.samples.values)
            found[start[samples[:, 0]] + samples[:, 1], pairs.index((key[1], key[2]))] = np.asarray(block.values)
        np.testing.assert_allclose(found, dense, rtol=0.0, atol=1e-12 * np.abs(dense).max())
        first = found if first is None else first
        np.testing.assert_array_equal(found, first)
