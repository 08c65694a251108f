"""Warp-per-centre contractions of the dense forms at the edges of their
tiles: one to six species (four are the most that are known at compile time),
one to forty radial functions (odd, fewer and more than eight, across blocks
of 32), l up to 8, one centre and more than a CTA holds.

* values and dL/dpositions, FP32 against the CUDA-core kernels: 2e-6 of the
  largest value, the bound of the tensor-core kernels (TF32 hi + lo drops
  2^-22 of a product; sums of at most 17 x 40 products);
* FP64 values against the contraction in torch, and the FP64 gradient against
  the transposed forward-mode derivative <G, J u> = <J^T G, u>: 1e-12 of the
  sum of sizes (rounding of 1e3-term sums, 1e-16 each, with a factor 10);
* a batch with weights by species against the same batch with every atom's
  row given: 2e-6 on gradients, 1e-5 on energies (FP32 sums of 4480 terms).
"""
import numpy as np
import pytest

import rascaline_b200 as rb
from rascaline_b200 import _c_api as C
from rascaline_b200 import workloads

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from rascaline_b200 import torch_api  # noqa: E402

TYPES = (1, 6, 7, 8, 9, 16)


@pytest.fixture(autouse=True)
def restore_engine():
    yield
    C.check(C.lib().featomic_b200_set_contraction_engine(1, 1))


def _forward(calculator, system, precision):
    positions = torch.tensor(system["positions"], device="cuda")
    cell = np.asarray(system["cell"]).reshape(1, 9)
    return torch_api.dense_power_spectrum(calculator, positions, system["types"], cell, [len(system["types"])], precision)


@pytest.mark.parametrize("atoms,species,max_radial,max_angular", [
    (1, 1, 0, 0), (9, 1, 7, 8), (20, 2, 2, 3), (33, 3, 5, 6), (40, 4, 7, 6), (40, 4, 4, 5), (30, 6, 7, 2),
    (20, 3, 11, 4), (12, 1, 15, 3),
])
def test_values_and_gradients(atoms, species, max_radial, max_angular):
    if atoms > 1:
        system = workloads.random_box(atoms, seed=atoms, species=TYPES[:species])
    else:
        system = workloads.system_dict([1], [[0.1, 0.2, 0.3]], np.zeros((3, 3)))
    hypers = workloads.hypers(4.0, max_radial, max_angular)
    calculator = rb.SoapPowerSpectrum(**hypers)
    results = []
    for engine in (1, 0):
        C.check(C.lib().featomic_b200_set_contraction_engine(engine, 1))
        values, state = _forward(calculator, system, 32)
        gradient = torch.randn(values.shape, generator=torch.Generator().manual_seed(3)).cuda()
        results.append([values] + [x for x in torch_api.dense_backward(state, gradient, 1) if x is not None])
    for a, b in zip(*results):
        assert float((a - b).abs().max()) <= 2e-6 * max(float(b.abs().max()), 1e-30)

    values, state = _forward(calculator, system, 64)
    positions = torch.tensor(system["positions"], device="cuda")
    c, _ = torch_api.dense_spherical_expansion(rb.SphericalExpansion(**hypers), positions, system["types"],
                                               np.asarray(system["cell"]).reshape(1, 9), [atoms], 64)
    N, S = max_radial + 1, c.shape[1]
    c = c.reshape(atoms, S, (max_angular + 1) ** 2, N)
    key = 0
    for a in range(S):
        for b in range(a, S):
            for l in range(max_angular + 1):
                x, y = (c[:, s, l * l:(l + 1) ** 2] for s in (a, b))
                scale = (-1) ** l / np.sqrt(2 * l + 1) * (np.sqrt(2) if a != b else 1)
                reference = torch.einsum("cmp,cmq->cpq", x, y).reshape(atoms, -1) * scale
                size = torch.einsum("cmp,cmq->cpq", x.abs(), y.abs()).reshape(atoms, -1) * abs(scale)
                found = values[:, key, l * N * N:(l + 1) * N * N]
                assert bool(((found - reference).abs() <= 1e-12 * size + 1e-300).all())
            key += 1
    gradient = torch.randn(values.shape, generator=torch.Generator().manual_seed(4), dtype=torch.float64).cuda()
    move = torch.randn((atoms, 3), generator=torch.Generator().manual_seed(5), dtype=torch.float64).cuda()
    forces, _, _ = torch_api.dense_backward(state, gradient, 1, cell=False)
    tangent, _ = torch_api.dense_jvp(state, move)
    size = float((gradient.abs() * tangent.abs()).sum())
    assert abs(float((gradient * tangent).sum() - (forces * move).sum())) <= 1e-12 * size + 1e-300


@pytest.mark.parametrize("molecules,species,max_radial,max_angular", [(1, 1, 1, 2), (12, 2, 7, 4), (40, 4, 7, 6), (9, 4, 4, 3)])
def test_batch_weights_by_species(molecules, species, max_radial, max_angular):
    systems = workloads.molecules(molecules, seed=5)
    sizes = [len(m["types"]) for m in systems]
    rng = np.random.default_rng(6)
    types = rng.choice(TYPES[:species], size=sum(sizes)).astype(np.int32)
    positions = torch.tensor(np.concatenate([m["positions"] for m in systems]), device="cuda")
    batch = torch_api.Batch(rb.SoapPowerSpectrum(**workloads.hypers(4.5, max_radial, max_angular)), sizes, types,
                            TYPES[:species])
    batch.config = dict(batch.config, pipeline=1)
    weights = torch.tensor(rng.normal(size=(species, batch.n_keys, batch.n_properties)), dtype=torch.float32, device="cuda")
    out = batch.run(positions, batch.outputs(strain=True), weights=weights)
    rows = weights[torch.tensor(np.searchsorted(TYPES[:species], types), device="cuda")].contiguous()
    given = batch.run(positions, batch.outputs(energies=False, strain=True), grad_values=rows)
    assert torch.equal(out["values"], given["values"])
    for name in ("gradients", "strain"):
        assert float((out[name] - given[name]).abs().max()) <= 2e-6 * float(given[name].abs().max())
    per_atom = (given["values"].double() * rows.double()).flatten(1)
    energies = torch.stack([x.sum() for x in torch.split(per_atom, sizes)])
    size = torch.stack([x.abs().sum() for x in torch.split(per_atom, sizes)])
    assert bool(((out["energies"] - energies).abs() <= 1e-5 * size).all())


@pytest.mark.parametrize("atoms,species,max_radial,max_angular", [(40, 17, 7, 1), (30, 2, 3, 16), (24, 3, 2, 18)])
def test_large_bases_keep_fp32_products(atoms, species, max_radial, max_angular):
    """More than 128 (s, n) or l from 16 on: FP32 multiply-adds, as with the
    tensor cores off, so that every value is within (M + 2) 2^-24 of the sum of
    sizes of the products of its FP32 coefficients (M <= 2 l + 1 of them, and
    the scale)."""
    types = np.random.default_rng(atoms).permutation([1 + k % species for k in range(atoms)])
    system = workloads.random_box(atoms, seed=atoms, species=(1,))
    positions, cell = torch.tensor(system["positions"], device="cuda"), np.asarray(system["cell"]).reshape(1, 9)
    hypers = workloads.hypers(3.5, max_radial, max_angular)
    calculator = rb.SoapPowerSpectrum(**hypers)
    results = []
    for engine in (1, 0):
        C.check(C.lib().featomic_b200_set_contraction_engine(engine, 1))
        results.append(torch_api.dense_power_spectrum(calculator, positions, types, cell, [atoms], 32)[0])
    assert torch.equal(*results)
    c, _ = torch_api.dense_spherical_expansion(rb.SphericalExpansion(**hypers), positions, types, cell, [atoms], 32)
    N = max_radial + 1
    c = c.double().reshape(atoms, species, (max_angular + 1) ** 2, N)
    key = 0
    for a in range(species):
        for b in range(a, species):
            for l in range(max_angular + 1):
                x, y = (c[:, s, l * l:(l + 1) ** 2] for s in (a, b))
                scale = (-1) ** l / np.sqrt(2 * l + 1) * (np.sqrt(2) if a != b else 1)
                reference = torch.einsum("cmp,cmq->cpq", x, y).reshape(atoms, -1) * scale
                size = torch.einsum("cmp,cmq->cpq", x.abs(), y.abs()).reshape(atoms, -1) * abs(scale)
                found = results[0][:, key, l * N * N:(l + 1) * N * N].double()
                assert bool(((found - reference).abs() <= (2 * l + 3) * 2.0 ** -24 * size + 1e-40).all())
            key += 1


def test_batch_energies_keep_small_terms():
    """An atom's energy of 64 terms 1 (l = 0) and 2304 of 0.9 x 2^-25 (l > 0),
    which an FP32 sum that runs on over l drops one by one (16 units of 2^-24 of
    the sum).  With the sums over l in FP64 a term 1 is rounded once, the small
    ones lose 2^-24 of themselves, and the energy is rounded once: 3 units."""
    types = np.array(TYPES[:4], dtype=np.int32)
    positions = torch.tensor([[0.0, 0.0, 0.0], [1.1, 0.2, 0.1], [0.1, 1.3, 0.4], [0.3, 0.5, 1.2]], dtype=torch.float64,
                             device="cuda")
    batch = torch_api.Batch(rb.SoapPowerSpectrum(**workloads.hypers(4.5, 7, 6)), [4], types, TYPES[:4])
    batch.config = dict(batch.config, pipeline=1)
    weights = torch.zeros((4, batch.n_keys, batch.n_properties), device="cuda")
    values = batch.run(positions, batch.outputs(), weights=weights)["values"].reshape(weights.shape)
    terms = torch.zeros_like(weights)
    terms[0, 0, :64] = 1.0
    terms[0, :, 64:] = 0.9 * 2.0 ** -25
    used = (terms != 0) & (values.abs() > 1e-20)
    weights[used] = terms[used] / values[used]
    assert int(used.sum()) > 2300
    energy = batch.run(positions, batch.outputs(), weights=weights)["energies"].double().cpu()
    terms = values.double() * weights.double()
    assert float((energy - terms.sum().cpu()).abs().max()) <= 3 * 2.0 ** -24 * float(terms.abs().sum())


@pytest.mark.parametrize("atoms,species,max_radial,max_angular", [
    (30, 9, 7, 3), (20, 16, 7, 2), (17, 5, 12, 2), (12, 6, 15, 2), (25, 20, 7, 1),
])
def test_blocks_of_many_functions(atoms, species, max_radial, max_angular):
    """65 to 160 (s, n): three to five blocks of 32, species that begin in one and
    end in the next.  FP64 within 1e-12 of the sum of sizes, FP32
    within 2e-6 of the largest value (as above), from the coefficients."""
    types = np.random.default_rng(atoms).permutation([1 + k % species for k in range(atoms)])
    system = workloads.random_box(atoms, seed=atoms, species=(1,))
    positions, cell = torch.tensor(system["positions"], device="cuda"), np.asarray(system["cell"]).reshape(1, 9)
    hypers = workloads.hypers(4.0, max_radial, max_angular)
    N = max_radial + 1
    for precision in (64, 32):
        values, _ = torch_api.dense_power_spectrum(rb.SoapPowerSpectrum(**hypers), positions, types, cell, [atoms], precision)
        c, _ = torch_api.dense_spherical_expansion(rb.SphericalExpansion(**hypers), positions, types, cell, [atoms], precision)
        c = c.double().reshape(atoms, species, (max_angular + 1) ** 2, N)
        largest = float(values.abs().max())
        key = 0
        for a in range(species):
            for b in range(a, species):
                for l in range(max_angular + 1):
                    x, y = (c[:, s, l * l:(l + 1) ** 2] for s in (a, b))
                    scale = (-1) ** l / np.sqrt(2 * l + 1) * (np.sqrt(2) if a != b else 1)
                    reference = torch.einsum("cmp,cmq->cpq", x, y).reshape(atoms, -1) * scale
                    size = torch.einsum("cmp,cmq->cpq", x.abs(), y.abs()).reshape(atoms, -1) * abs(scale)
                    error = (values[:, key, l * N * N:(l + 1) * N * N].double() - reference).abs()
                    assert bool((error <= (1e-12 * size + 1e-300 if precision == 64 else 2e-6 * largest)).all())
                key += 1


@pytest.mark.parametrize("atoms,species,max_radial,max_angular", [
    (1199, 4, 7, 1), (1200, 4, 15, 1), (1199, 4, 15, 1), (1200, 5, 7, 1), (2000, 1, 2, 9), (1999, 1, 2, 9),
])
def test_fp64_on_both_sides_of_its_rule(atoms, species, max_radial, max_angular):
    """The number of atoms, the fill of the blocks of 32 and lmax decide which
    kernel makes the FP64 values: within 1e-12 of the sum of sizes on both
    sides, from the coefficients."""
    system = workloads.random_box(atoms, seed=atoms, species=TYPES[:species])
    positions, cell = torch.tensor(system["positions"], device="cuda"), np.asarray(system["cell"]).reshape(1, 9)
    hypers = workloads.hypers(2.5, max_radial, max_angular)
    values, _ = torch_api.dense_power_spectrum(rb.SoapPowerSpectrum(**hypers), positions, system["types"], cell, [atoms], 64)
    c, _ = torch_api.dense_spherical_expansion(rb.SphericalExpansion(**hypers), positions, system["types"], cell, [atoms], 64)
    N = max_radial + 1
    c = c.reshape(atoms, species, (max_angular + 1) ** 2, N)
    key = 0
    for a in range(species):
        for b in range(a, species):
            for l in range(max_angular + 1):
                x, y = (c[:, s, l * l:(l + 1) ** 2] for s in (a, b))
                scale = (-1) ** l / np.sqrt(2 * l + 1) * (np.sqrt(2) if a != b else 1)
                reference = torch.einsum("cmp,cmq->cpq", x, y).reshape(atoms, -1) * scale
                size = torch.einsum("cmp,cmq->cpq", x.abs(), y.abs()).reshape(atoms, -1) * abs(scale)
                found = values[:, key, l * N * N:(l + 1) * N * N]
                assert bool(((found - reference).abs() <= 1e-12 * size + 1e-300).all())
            key += 1
