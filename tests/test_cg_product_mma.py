"""FP64 Clebsch-Gordan products of more than 16 properties a side (the
tensor-core kernel) at the edges of its 8-wide tiles and 32-wide blocks, with
odd rows, wider outputs and infinities, against the oracle's coefficients.

Bound: every output is a sum of at most 2 (2 l1 + 1) <= 18 products of three
factors; each adds at most three roundings to its own size, and summing adds
18 more to the sum of sizes, so |x - ref| <= 64 u sum |C a b| holds for both
summation orders (u = 1.1e-16).
"""
import numpy as np
import pytest

from oracle import clebsch_gordan as ocg
from rascaline_b200 import clebsch_gordan as cg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _product(samples, n1, n2, l1, l2, column, width, seed, poison=False):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((samples, 2 * l1 + 1, n1))
    b = rng.standard_normal((samples, 2 * l2 + 1, n2))
    if poison:
        a[1, 0, 3] = np.inf
        b[2, 2 * l2, 5] = np.nan
    ta, tb = torch.tensor(a, device="cuda"), torch.tensor(b, device="cuda")
    tasks, outs = [], []
    for lam in range(abs(l1 - l2), l1 + l2 + 1):
        out = torch.full((samples, 2 * lam + 1, width or n1 * n2), 7.0, dtype=torch.float64, device="cuda")
        tasks.append((ta, tb, out, lam, column) if width else (ta, tb, out, lam))
        outs.append((lam, out))
    cg.cg_tensor_products(tasks)
    return a, b, outs


@pytest.mark.parametrize("samples,n1,n2,l1,l2,column,width", [
    (1, 17, 17, 0, 0, 0, 0),  # the smallest, odd rows: 8-byte stores
    (5, 24, 32, 1, 2, 0, 0),  # full tiles
    (3, 32, 32, 4, 4, 0, 0),  # the largest tile, several rows groups
    (2, 33, 40, 2, 1, 0, 0),  # blocks of 24 + 9 and 24 + 16
    (4, 18, 70, 1, 3, 2, 18 * 70 + 6),  # three blocks, columns of a wider output
    (2, 20, 20, 3, 0, 1, 20 * 20 + 3),  # an odd column and pitch
])
def test_against_the_oracle(samples, n1, n2, l1, l2, column, width):
    a, b, outs = _product(samples, n1, n2, l1, l2, column, width, 3)
    for lam, out in outs:
        c = ocg.real_cg(l1, l2, lam)
        reference = np.einsum("xyz,sxp,syq->szpq", c, a, b).reshape(samples, 2 * lam + 1, -1)
        size = np.einsum("xyz,sxp,syq->szpq", np.abs(c), np.abs(a), np.abs(b)).reshape(reference.shape)
        found = out.cpu().numpy()
        inside = found[:, :, column:column + n1 * n2]
        assert np.all(np.abs(inside - reference) <= 64 * 1.1e-16 * size)
        assert np.all(np.delete(found, np.s_[column:column + n1 * n2], axis=2) == 7.0)


def test_infinities_stay_in_the_rows_they_couple_to():
    l1, l2 = 1, 2
    a, b, outs = _product(4, 20, 24, l1, l2, 0, 0, 5, poison=True)
    for lam, out in outs:
        c = ocg.real_cg(l1, l2, lam)
        reference = np.zeros((4, 2 * lam + 1, 20, 24))
        for x, y, z in zip(*np.nonzero(np.abs(c) > 1e-12)):
            reference[:, z] += c[x, y, z] * a[:, x, :, None] * b[:, y, None, :]
        found = out.cpu().numpy().reshape(reference.shape)
        np.testing.assert_array_equal(np.isnan(found), np.isnan(reference))
        np.testing.assert_array_equal(np.isinf(found), np.isinf(reference))
        fine = np.isfinite(reference)
        assert np.all(np.abs(found[fine] - reference[fine]) <= 1e-13)
