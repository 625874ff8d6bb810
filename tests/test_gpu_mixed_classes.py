"""Which classes a mixed-precision build runs in FP32: quartets counted class by class."""
import importlib
import itertools

import numpy as np
import pytest

lai = importlib.import_module("libaccint-public_b200")

pytestmark = pytest.mark.gpu


def _components(l0, l1):
    return sum((l + 1) * (l + 2) // 2 for l in range(l0, l1 + 1))


def _runs_fp32(la, lb, lc, ld):
    """Classes up to f with at most (dd|dd)'s 961 integrals (e0|f0), and (gs|ss)."""
    if la == 4:
        return (lb, lc, ld) == (0, 0, 0)
    return _components(la, la + lb) * _components(lc, lc + ld) <= 961


@pytest.mark.parametrize("ls", [(4, 1, 0), (3, 2, 1, 0), (3, 3, 2, 2, 1), (4, 3, 2, 1, 0)])
def test_fp32_classes_of_a_mixed_build(ls):
    rng = np.random.default_rng(2)
    shells = [lai.Shell(l, rng.normal(size=3), [rng.uniform(0.3, 2.0)], [1.0], i) for i, l in enumerate(ls)]
    basis = lai.BasisSet(shells)
    pairs = [tuple(sorted((ls[i], ls[j]), reverse=True)) for i in range(len(ls)) for j in range(i + 1)]
    want = sum(_runs_fp32(*max(a, b), *min(a, b)) for a, b in itertools.combinations_with_replacement(pairs, 2))
    total = len(pairs) * (len(pairs) + 1) // 2
    eng = lai.Engine(basis, threshold=0.0)
    for _ in range(2):
        rep = eng.jk(np.eye(basis.nbf), fp32_cut=1e30)[2]
        assert (rep.quartets_fp32, rep.quartets_fp64) == (want, total - want)
