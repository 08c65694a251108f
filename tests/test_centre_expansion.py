"""Values of the spherical expansion by the kernel with one CTA per centre
against the two kernels over pair records: the same operations in the same
order, so the drop-in's values are bit-identical, and the dense FP64 form
(with FMA contraction) agrees to 1e-13 of its largest value (sums of at most
100 products of O(1) terms, 1e-14 each).  Edges: one and sixteen radial
functions, lmax 0 and 8, more and fewer than 32 directions per centre, one
and several species, an atom without neighbours, periodic self-images, and
channels with different knots.
"""
import numpy as np
import pytest

import rascaline_b200 as rb
from rascaline_b200 import _c_api as C
from rascaline_b200 import workloads

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(autouse=True)
def restore_engine():
    yield
    C.check(C.lib().featomic_b200_set_expansion_engine(1))


def _small_cell():
    rng = np.random.default_rng(7)
    cell = np.array([[4.2, 0.0, 0.0], [0.6, 4.4, 0.0], [0.3, -0.4, 4.6]])
    return workloads.system_dict(rng.choice([1, 6, 8], size=9), rng.uniform(0.0, 1.0, (9, 3)) @ cell, cell)


def _isolated():
    return workloads.system_dict([1, 8, 8], [[0.0, 0.0, 0.0], [1.0, 0.0, 0.1], [50.0, 0.0, 0.0]], np.zeros((3, 3)))


@pytest.mark.parametrize("system,cutoff,max_radial,max_angular", [
    (_small_cell, 4.5, 7, 6),
    (_small_cell, 4.0, 3, 8),  # two groups of knots
    (_isolated, 3.0, 0, 0),
    (lambda: workloads.random_box(60, seed=3, species=(1,)), 4.5, 15, 8),  # 38 directions, 16 radial functions
    (lambda: workloads.random_box(70, seed=4, species=(1, 6, 7, 8, 9, 16)), 3.5, 4, 5),  # odd rows
])
def test_values_are_those_of_the_pair_records(system, cutoff, max_radial, max_angular):
    system = system()
    hypers = workloads.hypers(cutoff, max_radial, max_angular)
    calculator = rb.SphericalExpansion(**hypers)
    results = []
    for engine in (1, 0):
        C.check(C.lib().featomic_b200_set_expansion_engine(engine))
        results.append(calculator.compute(rb.System.from_dict(system)).to_dict())
    a, b = results
    np.testing.assert_array_equal(a["keys"], b["keys"])
    for x, y in zip(a["blocks"], b["blocks"]):
        np.testing.assert_array_equal(x["values"], y["values"])

    from rascaline_b200.torch_api import dense_spherical_expansion
    types = np.asarray(system["types"])
    positions = torch.tensor(system["positions"], device="cuda")
    dense, _ = dense_spherical_expansion(calculator, positions, types, np.asarray(system["cell"]).reshape(1, 9),
                                         [len(types)], 64)
    dense = dense.cpu().numpy()
    species = np.unique(types)
    scale = np.max(np.abs(dense))
    for key, block in zip(b["keys"], b["blocks"]):
        l, t = int(key[0]), int(np.searchsorted(species, key[3]))
        rows = dense[block["samples"][:, 1], t].reshape(-1, (max_angular + 1) ** 2, max_radial + 1)
        assert np.max(np.abs(rows[:, l * l:(l + 1) ** 2] - block["values"])) <= 1e-13 * scale
