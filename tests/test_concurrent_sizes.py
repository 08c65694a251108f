"""Calls of different sizes from two threads: each needs its own amount of
dynamic shared memory of the same kernels (above and below the 48 KB that a
kernel has without asking), and none may take it from the other.  Results equal
those of the same calls one after the other, to the last bit."""
import threading

import numpy as np
import pytest

import rascaline_b200 as rb
from rascaline_b200 import clebsch_gordan as cg
from rascaline_b200 import workloads

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from rascaline_b200 import torch_api  # noqa: E402


def _product(l1, l2, lam):
    # enough samples for the tensor-core kernel
    generator = torch.Generator().manual_seed(l1)
    a = torch.randn((2000, 2 * l1 + 1, 20), generator=generator, dtype=torch.float64).cuda()
    b = torch.randn((2000, 2 * l2 + 1, 20), generator=generator, dtype=torch.float64).cuda()
    out = torch.empty((2000, 2 * lam + 1, 400), dtype=torch.float64, device="cuda")

    def call():
        cg.cg_tensor_products([(a, b, out, lam)])
        return out
    return call


def _expansion(max_radial, max_angular, precision):
    system = workloads.random_box(20, seed=3, species=(1, 6))
    calculator = rb.SphericalExpansion(**workloads.hypers(3.0, max_radial, max_angular))
    positions = torch.tensor(system["positions"], device="cuda")
    cell = np.asarray(system["cell"]).reshape(1, 9)
    return lambda: torch_api.dense_spherical_expansion(calculator, positions, system["types"], cell, [20], precision)[0]


@pytest.mark.parametrize("large,small", [
    (lambda: _product(12, 12, 3), lambda: _product(1, 1, 1)),  # 58 and 9 KB
    (lambda: _expansion(15, 8, 64), lambda: _expansion(3, 2, 64)),  # 59 and 7 KB
])
def test_two_threads(large, small):
    calls = [large(), small()]
    references = [call().clone() for call in calls]
    torch.cuda.synchronize()
    wrong, errors = [], []
    begin = threading.Barrier(2)

    def work(call, reference):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                begin.wait()
                for _ in range(8000):
                    found = call()
                torch.cuda.current_stream().synchronize()
                if not torch.equal(found, reference):
                    wrong.append(reference.shape)
        except Exception as error:  # noqa: BLE001
            errors.append(error)

    threads = [threading.Thread(target=work, args=x) for x in zip(calls, references)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert not errors
    assert not wrong
