"""Rounding of the sums of J and K: a build against its shards added up."""
import importlib

import numpy as np
import pytest

lai = importlib.import_module("libaccint-public_b200")

pytestmark = pytest.mark.gpu


# 25 functions per molecule; norm of what one accumulator per matrix and four of them leave
# (measured): 1.9e-15 and 6.5e-16 at 175 functions, 3.2e-15 and 1.1e-15 at 400, 4.5e-15 and
# 1.5e-15 at 725
@pytest.mark.parametrize("n,bound", [(7, 1.2e-15), (16, 2e-15), (29, 2.8e-15)])
def test_build_equals_its_shards(n, bound):
    import torch
    rng = np.random.default_rng(0)
    Z, xyz = lai.molecules.water_cluster_n(n, rng)
    basis = lai.BasisSet.from_atoms(Z, xyz, "cc-pvdz")
    eng = lai.Engine(basis)
    C = rng.normal(0, 1 / np.sqrt(basis.nbf), size=(basis.nbf, 5 * n))
    D = torch.from_numpy(C @ C.T).cuda()

    def build(shard):
        J, K = torch.empty_like(D), torch.empty_like(D)
        eng.jk_device(D.data_ptr(), J.data_ptr(), K.data_ptr(), stream=torch.cuda.current_stream().cuda_stream,
                      shard=shard)
        return J, K

    J, K = build((0, 1))
    parts = [build((s, 24)) for s in range(24)]
    for full, part in ((J, sum(p[0] for p in parts)), (K, sum(p[1] for p in parts))):
        assert float((full - part).norm()) < bound * float(full.norm())
