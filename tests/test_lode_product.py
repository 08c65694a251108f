"""LODE values and positions gradients at the edges of the product's tiles
(64 rows, 56 or 64 columns of one parity of l, 16 k-vectors, splits of the
k-vectors), against the oracle.

Bound: |x - ref| <= 1e-10 |ref| + 1e-12 max|ref|.  Both sides sum the same K
<= 2000 FP64 terms in different orders; rounding is a random walk of sqrt(K)
half-ulps over sums of absolute terms at most about 100 times the largest
value, 45 x 1.1e-16 x 100 = 5e-13 of it.
"""
import numpy as np
import pytest

import rascaline_b200 as rb
from oracle import lode as oracle_lode

pytestmark = pytest.mark.gpu


def _box(n, seed):
    rng = np.random.default_rng(seed)
    length = (n / 0.1) ** (1.0 / 3.0)
    cell = length * (np.eye(3) + rng.uniform(-0.1, 0.1, (3, 3)))
    types = np.array([1, 8], dtype=np.int32)[(np.arange(n) % 3 == 0).astype(int)]
    return {"types": types, "positions": rng.uniform(0.0, 1.0, (n, 3)) @ cell, "cell": cell}


@pytest.mark.parametrize("atoms,max_radial,max_angular,smearing,gradients", [
    (1, 0, 0, 0.6, ()),  # one row, one column
    (5, 2, 1, 0.9, ("positions",)),  # odd columns of both parities, 3 rows per task across tiles
    (21, 3, 4, 1.0, ("positions",)),  # 64 rows and one more
    (64, 6, 3, 1.0, ()),  # one full row tile, 56 odd columns
    (65, 7, 6, 0.8, ()),  # a row past the tile, 224 and 168 columns, several splits
])
def test_tile_edges(atoms, max_radial, max_angular, smearing, gradients):
    hypers = {"density": {"type": "SmearedPowerLaw", "smearing": smearing, "exponent": 1, "center_atom_weight": 0.5},
              "basis": {"type": "TensorProduct", "max_angular": max_angular, "spline_accuracy": None,
                        "radial": {"type": "Gto", "max_radial": max_radial, "radius": 3.0}}}
    system = _box(atoms, 10 + atoms)
    calculator = rb.LodeSphericalExpansion(**hypers)
    ours = calculator.compute(rb.System.from_dict(system), gradients=list(gradients)).to_dict(gradients)
    reference = oracle_lode.compute(hypers, [system], gradients)
    np.testing.assert_array_equal(ours["keys"], reference["keys"])
    for pick in (lambda b: b["values"],) + tuple(lambda b, g=g: b["gradients"][g]["values"] for g in gradients):
        x = np.concatenate([pick(b).reshape(-1) for b in ours["blocks"]])
        y = np.concatenate([pick(b).reshape(-1) for b in reference["blocks"]])
        assert np.all(np.abs(x - y) <= 1e-10 * np.abs(y) + 1e-12 * np.max(np.abs(y)))


def test_splits_memory():
    """Splits of the k-vectors keep a partial sum each, 512 MB together at most:
    49 344 atoms and 9605 k-vectors, whose waves seven splits of 155 MB would
    fill best.  Beside them a call keeps its phases, table and output, and the
    small arrays and the pool's granularity below 200 MB."""
    torch = pytest.importorskip("torch")
    hypers = {"density": {"type": "SmearedPowerLaw", "smearing": 1.0, "exponent": 1},
              "basis": {"type": "TensorProduct", "max_angular": 6, "radial": {"type": "Gto", "max_radial": 7, "radius": 3.0}}}
    cell = 27.7 * np.eye(3)
    atoms, k, columns = 49344, 9616, 392

    def run(n):
        positions = np.random.default_rng(n).uniform(0.0, 27.7, (n, 3))
        calculator = rb.LodeSphericalExpansion(**hypers)
        system = rb.System.from_dict({"types": np.ones(n, dtype=np.int32), "positions": positions, "cell": cell})
        return calculator, calculator.compute(system)

    run(100)
    before = torch.cuda.mem_get_info()[0]
    calculator, result = run(atoms)
    used = before - torch.cuda.mem_get_info()[0]
    del result
    assert calculator is not None
    expected = 8 * (2 * atoms * k + k * columns + atoms * columns)
    assert expected - (64 << 20) <= used <= expected + (512 << 20) + (200 << 20)
