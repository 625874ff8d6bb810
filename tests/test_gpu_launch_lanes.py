"""Builds spread over several streams against the same launches on one stream, and
the pool of stream sets that outlives an engine."""
import importlib
import threading

import numpy as np
import pytest

lai = importlib.import_module("libaccint-public_b200")

pytestmark = pytest.mark.gpu

# the launches' atomics add in another order: a few hundred roundings of terms below
# the result's largest element
REL = 1e-13


def _device_build(eng, D, stream, **opts):
    import torch
    with torch.cuda.stream(stream):
        d = torch.from_numpy(D).cuda()
        J, K = torch.empty_like(d), torch.empty_like(d)
        eng.jk_device(d.data_ptr(), J.data_ptr(), K.data_ptr(), stream=stream.cuda_stream, **opts)
        return J.cpu().numpy(), K.cpu().numpy()


@pytest.mark.parametrize("name", ["h2o1_sto3g", "h2o2_631g", "h2o2_ccpvdz", "h2o1_ccpvtz"])
@pytest.mark.parametrize("fp32_cut", [0.0, 1e-7])
def test_spread_build_equals_one_stream(name, fp32_cut):
    import torch
    w = lai.workloads.make(name)
    eng = lai.Engine(w.basis)
    one = _device_build(eng, w.D, torch.cuda.Stream(), profile=True, fp32_cut=fp32_cut)
    for _ in range(3):
        got = _device_build(eng, w.D, torch.cuda.Stream(), fp32_cut=fp32_cut)
        for a, b in zip(one, got):
            assert np.max(np.abs(a - b)) < REL * np.max(np.abs(a))
    graph = _device_build(eng, w.D, torch.cuda.Stream(), graph=True, fp32_cut=fp32_cut)
    for a, b in zip(one, graph):
        assert np.max(np.abs(a - b)) < REL * np.max(np.abs(a))


def test_engines_of_several_threads_share_the_pool():
    w = lai.workloads.make("h2o2_631g")
    eng = lai.Engine(w.basis)
    J0, K0, _ = eng.jk(w.D)
    bad = []

    def work():
        for _ in range(4):
            e = lai.Engine(w.basis)
            J, K, _ = e.jk(w.D)
            if max(np.max(np.abs(J - J0)), np.max(np.abs(K - K0))) > REL * np.max(np.abs(J0)):
                bad.append(1)
            e.close()

    threads = [threading.Thread(target=work) for _ in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
