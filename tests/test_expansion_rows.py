"""Rows of the spherical expansion from the neighbourhood tables built on the
device against those from the host's tables (a caller's own pairs): the same
labels and the same bits, for values and every gradient.  Periodic images of
a neighbour and of the atom itself, an atom without neighbours, one and six
species, one and many coefficients per row.
"""
import numpy as np
import pytest

import rascaline_b200 as rb
from rascaline_b200 import workloads

pytestmark = pytest.mark.gpu


def _small_cell():
    rng = np.random.default_rng(7)
    cell = np.array([[4.2, 0.0, 0.0], [0.6, 4.4, 0.0], [0.3, -0.4, 4.6]])
    return workloads.system_dict(rng.choice([1, 6, 8], size=9), rng.uniform(0.0, 1.0, (9, 3)) @ cell, cell)


def _isolated():
    return workloads.system_dict([1, 8, 8], [[0.0, 0.0, 0.0], [1.0, 0.0, 0.1], [50.0, 0.0, 0.0]], np.zeros((3, 3)))


@pytest.mark.parametrize("system,cutoff,max_radial,max_angular,gradients", [
    (_small_cell, 4.5, 3, 4, ["positions", "strain", "cell"]),
    (_small_cell, 4.5, 3, 4, ["strain"]),
    (_isolated, 3.0, 0, 0, ["positions", "cell"]),
    (lambda: workloads.random_box(70, seed=4, species=(1, 6, 7, 8, 9, 16)), 3.5, 7, 8, ["positions"]),
    (lambda: workloads.random_box(40, seed=5, species=(1,)), 4.0, 4, 9, ["positions", "strain"]),  # pair records
    (lambda: workloads.random_box(30, seed=6), 3.5, 2, 3, []),
])
def test_device_tables_give_the_rows_of_the_host_tables(system, cutoff, max_radial, max_angular, gradients):
    d = system()
    calculator = rb.SphericalExpansion(**workloads.hypers(cutoff, max_radial, max_angular))
    ours = calculator.compute(rb.System.from_dict(d), gradients=gradients).to_dict(gradients)
    pairs = rb.neighbor_list(d["positions"], d["cell"], cutoff)
    given = calculator.compute(rb.System.from_dict(dict(d, pairs=pairs)), gradients=gradients,
                               use_native_system=False).to_dict(gradients)
    np.testing.assert_array_equal(ours["keys"], given["keys"])
    for a, b in zip(ours["blocks"], given["blocks"]):
        np.testing.assert_array_equal(a["samples"], b["samples"])
        np.testing.assert_array_equal(a["values"], b["values"])
        for g in gradients:
            np.testing.assert_array_equal(a["gradients"][g]["samples"], b["gradients"][g]["samples"])
            np.testing.assert_array_equal(a["gradients"][g]["values"], b["gradients"][g]["values"])


def test_growing_neighbourhoods_keep_their_staging():
    """Twenty steps of a box that shrinks, each with more pairs than the last:
    the pinned buffer of the neighbourhood tables grows by a quarter at a time,
    here once at most, where an exact size would be freed at every step."""
    torch = pytest.importorskip("torch")
    from torch.profiler import ProfilerActivity, profile

    box = workloads.random_box(200, seed=1, species=(1, 8))
    calculator = rb.SphericalExpansion(**workloads.hypers(4.0, 2, 1))

    def step(k):
        f = 1.0 - 0.002 * k
        calculator.compute([workloads.system_dict(box["types"], np.asarray(box["positions"]) * f, np.asarray(box["cell"]) * f)],
                           gradients=["positions"])

    step(0)
    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as profiler:
        for k in range(1, 21):
            step(k)
    calls = [e.name for e in profiler.events()]
    assert any("LaunchKernel" in name for name in calls)
    assert sum("FreeHost" in name for name in calls) <= 1
