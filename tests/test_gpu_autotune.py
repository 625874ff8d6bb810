"""Builds of a tuned engine against builds of an untuned one: results, and time."""
import importlib

import numpy as np
import pytest

lai = importlib.import_module("libaccint-public_b200")

pytestmark = pytest.mark.gpu


def _ms(eng, d, stream):
    """Time of one build: the shortest of five groups of ten."""
    import torch
    J, K = torch.empty_like(d), torch.empty_like(d)
    best = 1e30
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for _ in range(10):
            eng.jk_device(d.data_ptr(), J.data_ptr(), K.data_ptr(), stream=stream.cuda_stream)
        b.record(stream)
        b.synchronize()
        best = min(best, a.elapsed_time(b) / 10)
    return best, J.cpu().numpy(), K.cpu().numpy()


# many small launches (666 blocks), few functions with them, and launches that fill the device
@pytest.mark.parametrize("name", ["h2o1_ccpvqz", "h2o2_ccpvdz", "h2o16_ccpvdz"])
def test_tuned_engine_is_not_slower(name):
    import torch
    w = lai.workloads.make(name)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        d = torch.from_numpy(w.D).cuda()
        plain, tuned = lai.Engine(w.basis), lai.Engine(w.basis)
        tuned.autotune(d.data_ptr(), stream=stream.cuda_stream)
        t0, J0, K0 = _ms(plain, d, stream)
        t1, J1, K1 = _ms(tuned, d, stream)
        t0 = min(t0, _ms(plain, d, stream)[0])
    # launches that add in another order
    assert np.max(np.abs(J1 - J0)) < 1e-12 * np.max(np.abs(J0))
    assert np.max(np.abs(K1 - K0)) < 1e-12 * np.max(np.abs(K0))
    assert t1 < 1.05 * t0, (t1, t0)
