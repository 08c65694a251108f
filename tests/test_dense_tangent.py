"""Forward-mode derivative of the dense forms by centre, at the edges of its
chunks and tiles: a batch whose systems hold no pair, one pair and more than
32 directions per centre, in and out of a cell, one to five species, odd, few
and more than eight radial functions, l from 0 to 9.

* FP64: the tangent is the transpose of the adjoint, <G, J u> = <J^T G, u>,
  to 1e-12 of the sum of sizes (sums of 1e3 terms at 1e-16 each, with a
  factor 10);
* FP32 against FP64: 2e-5 of the largest value, the bound of the FP32 forms
  (6e-8 per operation, some 30 operations deep, with a factor 10);
* FP32 values on tensor cores against the CUDA cores: 2e-6 of the largest
  (TF32 hi + lo drops 2^-22 of a product).
"""
import numpy as np
import pytest

import rascaline_b200 as rb
from rascaline_b200 import _c_api as C
from rascaline_b200 import workloads

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from rascaline_b200 import torch_api  # noqa: E402

TYPES = (1, 6, 7, 8, 9)


@pytest.fixture(autouse=True)
def restore_engine():
    yield
    C.check(C.lib().featomic_b200_set_contraction_engine(1, 1))


def _systems(species):
    rng = np.random.default_rng(species)
    types = lambda n: rng.permutation([TYPES[k % species] for k in range(n)])  # noqa: E731
    cluster = rng.uniform(0.0, 4.0, (40, 3))
    return [
        (types(1), np.array([[0.3, 0.1, 0.2]]), np.zeros((3, 3))),
        (types(2), np.array([[0.0, 0.0, 0.0], [0.4, 1.1, 0.7]]), np.zeros((3, 3))),
        (types(12), rng.uniform(0.0, 4.5, (12, 3)), np.diag([4.4, 4.7, 5.0]) + rng.uniform(-0.2, 0.2, (3, 3))),
        (types(40), cluster, np.zeros((3, 3))),
    ]


@pytest.mark.parametrize("species,max_radial,max_angular", [
    (1, 0, 0), (1, 7, 9), (2, 2, 3), (3, 7, 6), (4, 4, 5), (4, 7, 2), (5, 5, 4), (3, 11, 5),
])
def test_tangent(species, max_radial, max_angular):
    systems = _systems(species)
    hypers = workloads.hypers(3.6, max_radial, max_angular)
    calculator = rb.SoapPowerSpectrum(**hypers)
    types = np.concatenate([s[0] for s in systems])
    positions = torch.tensor(np.concatenate([s[1] for s in systems]), device="cuda")
    cells = np.stack([s[2].reshape(9) for s in systems])
    sizes = [len(s[0]) for s in systems]
    generator = torch.Generator().manual_seed(4)
    move = torch.randn((len(types), 3), dtype=torch.float64, generator=generator).cuda()
    strain = torch.randn((len(systems), 3, 3), dtype=torch.float64, generator=generator).cuda()
    results = {}
    for precision, engine in ((64, 1), (32, 1), (32, 0)):
        C.check(C.lib().featomic_b200_set_contraction_engine(engine, 1))
        values, state = torch_api.dense_power_spectrum(calculator, positions, types, cells, sizes, precision)
        tangents = torch_api.dense_jvp(state, move.to(values.dtype), strain.to(values.dtype))
        results[precision, engine] = tangents[0].double()
        if precision == 64:
            gradient = torch.randn(values.shape, dtype=torch.float64, generator=generator).cuda()
            at_positions, _, at_cell = torch_api.dense_backward(state, gradient, len(systems), strain=False, cell=True)
            left = float((gradient * tangents[0]).sum())
            right = float((at_positions * move).sum() + (at_cell * strain).sum())
            size = float((gradient.abs() * tangents[0].abs()).sum())
            assert abs(left - right) <= 1e-12 * size
    fast, exact, cores = results[32, 1], results[64, 1], results[32, 0]
    assert float((fast - exact).abs().max()) <= 2e-5 * float(exact.abs().max())
    assert float((fast - cores).abs().max()) <= 2e-6 * float(exact.abs().max())


@pytest.mark.parametrize("species,max_radial,max_angular", [(1, 0, 0), (2, 2, 3), (3, 7, 6), (4, 4, 5), (4, 7, 8)])
def test_contraction_in_64_bits(species, max_radial, max_angular):
    """The FP32 tangent of the power spectrum from its own FP32 coefficients and
    their tangents: products and sums in 64 bits, one rounding at the end, so
    |x - ref| <= 2^-24 |ref| + 2^-48 of the sum of sizes."""
    systems = _systems(species)
    hypers = workloads.hypers(3.6, max_radial, max_angular)
    types = np.concatenate([s[0] for s in systems])
    positions = torch.tensor(np.concatenate([s[1] for s in systems]), device="cuda")
    cells = np.stack([s[2].reshape(9) for s in systems])
    sizes = [len(s[0]) for s in systems]
    move = torch.randn((len(types), 3), generator=torch.Generator().manual_seed(4)).cuda()
    c, state = torch_api.dense_spherical_expansion(rb.SphericalExpansion(**hypers), positions, types, cells, sizes, 32)
    state.expansion_width = c.shape[2]
    _, d = torch_api.dense_jvp(state, move, values=False, coefficients=True)
    _, state = torch_api.dense_power_spectrum(rb.SoapPowerSpectrum(**hypers), positions, types, cells, sizes, 32)
    tangent, _ = torch_api.dense_jvp(state, move)
    N, S = max_radial + 1, c.shape[1]
    c, d = (x.double().reshape(len(types), S, (max_angular + 1) ** 2, N) for x in (c, d))
    key = 0
    for a in range(S):
        for b in range(a, S):
            for l in range(max_angular + 1):
                x, y = (c[:, s, l * l:(l + 1) ** 2] for s in (a, b))
                dx, dy = (d[:, s, l * l:(l + 1) ** 2] for s in (a, b))
                scale = (-1) ** l / np.sqrt(2 * l + 1) * (np.sqrt(2) if a != b else 1)
                product = lambda u, v: torch.einsum("cmp,cmq->cpq", u, v).reshape(len(types), -1)  # noqa: E731
                reference = scale * (product(dx, y) + product(x, dy))
                size = abs(scale) * (product(dx.abs(), y.abs()) + product(x.abs(), dy.abs()))
                found = tangent[:, key, l * N * N:(l + 1) * N * N].double()
                assert bool(((found - reference).abs() <= 2.0 ** -24 * reference.abs() + 2.0 ** -48 * size).all())
            key += 1


@pytest.mark.parametrize("atoms,max_radial,max_angular", [
    (600, 1, 1), (700, 1, 1), (700, 7, 3), (700, 3, 3), (1000, 3, 1), (1100, 3, 1), (1100, 7, 2),
])
def test_both_sides_of_the_rule(atoms, max_radial, max_angular):
    """Around 24 000 (FP64) and 40 000 (FP32) directions, bases below and above
    the line: the same bounds as above, whichever way the tangent goes."""
    box = workloads.random_box(atoms, seed=atoms, species=TYPES[:2])
    calculator = rb.SoapPowerSpectrum(**workloads.hypers(4.5, max_radial, max_angular))
    positions, cell = torch.tensor(box["positions"], device="cuda"), np.asarray(box["cell"]).reshape(1, 9)
    generator = torch.Generator().manual_seed(4)
    move = torch.randn((atoms, 3), dtype=torch.float64, generator=generator).cuda()
    strain = torch.randn((1, 3, 3), dtype=torch.float64, generator=generator).cuda()
    values, state = torch_api.dense_power_spectrum(calculator, positions, box["types"], cell, [atoms], 64)
    exact, _ = torch_api.dense_jvp(state, move, strain)
    gradient = torch.randn(values.shape, dtype=torch.float64, generator=generator).cuda()
    at_positions, _, at_cell = torch_api.dense_backward(state, gradient, 1, strain=False, cell=True)
    left, right = float((gradient * exact).sum()), float((at_positions * move).sum() + (at_cell * strain).sum())
    assert abs(left - right) <= 1e-12 * float((gradient.abs() * exact.abs()).sum())
    _, state = torch_api.dense_power_spectrum(calculator, positions, box["types"], cell, [atoms], 32)
    fast, _ = torch_api.dense_jvp(state, move.float(), strain.float())
    assert float((fast.double() - exact).abs().max()) <= 2e-5 * float(exact.abs().max())
