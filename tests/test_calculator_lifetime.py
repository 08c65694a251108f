"""A calculator dropped right after a dense form has returned, with its kernels
still queued, while another thread makes calculators of its own: the tables of
the first must stay as they are until its kernels are done.  Both threads' results
equal those of the same calls one after the other, to the last bit (every
reduction has a fixed order)."""
import threading

import numpy as np
import pytest

import rascaline_b200 as rb
from rascaline_b200 import workloads

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from rascaline_b200 import torch_api  # noqa: E402


def _values(system, hypers, precision):
    positions = torch.tensor(system["positions"], device="cuda")
    cell = np.asarray(system["cell"]).reshape(1, 9)
    values, state = torch_api.dense_power_spectrum(rb.SoapPowerSpectrum(**hypers), positions, system["types"], cell,
                                                   [len(system["types"])], precision)
    del state  # and with it the calculator
    return values


@pytest.mark.parametrize("precision", [32, 64])
def test_dropped_with_work_in_flight(precision):
    system = workloads.random_box(1500, seed=1, species=(1, 6, 8))
    small = workloads.random_box(60, seed=2, species=(1, 6, 8))
    hypers, others = workloads.hypers(4.5, 7, 6), [workloads.hypers(3.0 + 0.1 * k, 5, 4) for k in range(4)]
    reference = _values(system, hypers, precision)
    references = [_values(small, h, 64) for h in others]
    torch.cuda.synchronize()
    wrong, errors = [], []

    def work(rounds, calls):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(rounds):
                    for h, box, bits, expected in calls:
                        found = _values(box, h, bits)
                        torch.cuda.current_stream().synchronize()
                        if not torch.equal(found, expected):
                            wrong.append(h)
        except Exception as error:  # noqa: BLE001
            errors.append(error)

    threads = [threading.Thread(target=work, args=(12, [(hypers, system, precision, reference)])),
               threading.Thread(target=work, args=(12, [(h, small, 64, r) for h, r in zip(others, references)]))]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert not errors
    assert not wrong
