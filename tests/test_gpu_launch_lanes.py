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


@pytest.mark.parametrize("call", ["jk", "gradient"])
def test_calls_beside_a_capture_that_is_still_open(call):
    """Between a captured call and the end of its capture, the engine's side streams are the
    capture's: a call on another stream runs beside it, and the capture stays good."""
    import torch
    w = lai.workloads.make("h2o2_631g")
    eng = lai.Engine(w.basis)
    J0, K0, _ = eng.jk(w.D)
    g0 = eng.gradient(w.D)
    d = torch.from_numpy(w.D).cuda()
    out = [[torch.empty_like(d) for _ in range(2)] for _ in range(2)]
    grad = [torch.empty(eng.natom(), 3, dtype=torch.float64, device="cuda") for _ in range(2)]

    def run(k, stream):
        if call == "jk":
            eng.jk_device(d.data_ptr(), out[k][0].data_ptr(), out[k][1].data_ptr(), stream=stream.cuda_stream)
        else:
            lai._lib.check(lai._lib.lib().lai_jk_gradient_device(eng._h, d.data_ptr(), grad[k].data_ptr(),
                                                                 stream.cuda_stream))

    graph, inside, beside = torch.cuda.CUDAGraph(), torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=inside, capture_error_mode="thread_local"):
        run(0, inside)
        run(1, beside)
    beside.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    for k in range(2):
        if call == "jk":
            for a, b in zip(out[k], (J0, K0)):
                assert np.max(np.abs(a.cpu().numpy() - b)) < REL * np.max(np.abs(b))
        else:
            assert np.max(np.abs(grad[k].cpu().numpy() - g0)) < 1e-12 * np.max(np.abs(g0))


@pytest.mark.parametrize("system", ["alkane6_ccpvtz", "h2o1_ccpvqz"])
def test_shared_launches_do_not_cost_time(system):
    """The plain build shares launches among a class's blocks; with a mixed-precision cut
    below every bound the same quartets run one launch per block."""
    import time

    import torch
    if system == "alkane6_ccpvtz":
        basis = lai.BasisSet.from_atoms(*lai.molecules.alkane(6), "cc-pvtz")
    else:
        basis = lai.workloads.make(system).basis
    eng = lai.Engine(basis)
    d = torch.from_numpy(lai.molecules.random_density(basis.nbf, 10, np.random.default_rng(0))).cuda()
    J, K = torch.empty_like(d), torch.empty_like(d)
    stream = torch.cuda.Stream()

    def ms(cut):
        best = 1e9
        for _ in range(6):
            torch.cuda.synchronize()
            t = time.perf_counter()
            eng.jk_device(d.data_ptr(), J.data_ptr(), K.data_ptr(), stream=stream.cuda_stream, fp32_cut=cut)
            torch.cuda.synchronize()
            best = min(best, 1e3 * (time.perf_counter() - t))
        return best

    ms(0.0)
    shared, single = ms(0.0), ms(1e-25)
    # launches that fill the device gain nothing by sharing one, and lost 6.6 % by it
    assert shared < 1.035 * single, (shared, single)
