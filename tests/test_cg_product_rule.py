"""FP64 Clebsch-Gordan products on both sides of the rule that takes them to the
tensor-core kernel (enough output for its tables), at the edges of its 8-wide
tiles and 32-wide blocks, with odd rows, wider outputs and infinities, against
the oracle's coefficients; the kernel that ran is read from the profiler.

Bound: as for the kernel itself, |x - ref| <= 64 u sum |C a b| (u = 1.1e-16).
"""
import numpy as np
import pytest

from oracle import clebsch_gordan as ocg
from rascaline_b200 import clebsch_gordan as cg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _run(samples, n1, n2, l1, l2, column, width, poison=False):
    generator = torch.Generator().manual_seed(n1)
    a = torch.randn((samples, 2 * l1 + 1, n1), dtype=torch.float64, generator=generator).cuda()
    b = torch.randn((samples, 2 * l2 + 1, n2), dtype=torch.float64, generator=generator).cuda()
    if poison:
        a[1, 0, 3] = np.inf
        b[2, 2 * l2, 5] = np.nan
    tasks, outs = [], []
    for lam in range(abs(l1 - l2), l1 + l2 + 1):
        out = torch.full((samples, 2 * lam + 1, width or n1 * n2), 7.0, dtype=torch.float64, device="cuda")
        tasks.append((a, b, out, lam, column) if width else (a, b, out, lam))
        outs.append((lam, out))
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as profiler:
        cg.cg_tensor_products(tasks)
        torch.cuda.synchronize()
    names = [e.name for e in profiler.events()]
    return a, b, outs, any("cg_product_mma_kernel" in name for name in names)


# rows of the tables times 32 bytes and 6000 more, times 2500 (even rows) or 60
SHAPES = [
    (17, 17, 0, 0, 0, 0, 620),  # odd rows
    (24, 32, 1, 2, 0, 0, 240),  # full tiles
    (32, 32, 4, 4, 0, 0, 145),  # the largest tile, several groups of rows
    (33, 40, 2, 1, 0, 0, 160),  # blocks of 24 + 9 and 24 + 16
    (18, 70, 1, 3, 2, 18 * 70 + 6, 105),  # three blocks, columns of a wider output
    (20, 20, 3, 0, 1, 20 * 20 + 3, 120),  # an odd column and pitch
]


@pytest.mark.parametrize("mma", [False, True])
@pytest.mark.parametrize("n1,n2,l1,l2,column,width,samples", SHAPES)
def test_both_sides(n1, n2, l1, l2, column, width, samples, mma):
    a, b, outs, ran = _run(samples if mma else 1, n1, n2, l1, l2, column, width)
    assert ran == mma
    for lam, out in outs:
        c = torch.tensor(ocg.real_cg(l1, l2, lam), device="cuda")
        reference = torch.einsum("xyz,sxp,syq->szpq", c, a, b).flatten(2)
        size = torch.einsum("xyz,sxp,syq->szpq", c.abs(), a.abs(), b.abs()).flatten(2)
        inside = out[:, :, column:column + n1 * n2]
        assert bool(((inside - reference).abs() <= 64 * 1.1e-16 * size).all())
        assert bool((out[:, :, :column] == 7.0).all()) and bool((out[:, :, column + n1 * n2:] == 7.0).all())


def test_infinities_stay_in_the_rows_they_couple_to():
    l1, l2 = 1, 2
    a, b, outs, ran = _run(400, 20, 24, l1, l2, 0, 0, poison=True)
    assert ran
    for lam, out in outs:
        c = ocg.real_cg(l1, l2, lam)
        reference = torch.zeros((400, 2 * lam + 1, 20, 24), dtype=torch.float64, device="cuda")
        for x, y, z in zip(*np.nonzero(np.abs(c) > 1e-12)):
            reference[:, z] += c[x, y, z] * a[:, x, :, None] * b[:, y, None, :]
        found = out.reshape(reference.shape)
        assert bool((found.isnan() == reference.isnan()).all()) and bool((found.isinf() == reference.isinf()).all())
        fine = reference.isfinite()
        assert bool(((found - reference)[fine].abs() <= 1e-13).all())
