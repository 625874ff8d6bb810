"""Raw integrals of the low classes (Boys rows, vertical recurrence, Rys fits) against the
oracle where the argument T = rho R^2 of the Boys function meets the ends of its tables."""
import importlib

import numpy as np
import pytest

lai = importlib.import_module("libaccint-public_b200")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [0.0, 1e-12, 0.049999, 0.05, 7.3, 39.94, 39.95, 39.96, 44.9, 45.0, 45.94, 45.95, 45.96,
                               60.0, 400.0])
def test_integrals_at_table_ends(T, oracle):
    # one-centre pairs of exponent 1 + 1 at distance R: rho = 1 and T = R^2 exactly in the
    # s classes; a shifted third centre gives pairs with P - A and Q - C non-zero
    R = np.sqrt(T)
    u = np.array([0.6, -0.48, 0.64])
    shells = [lai.Shell(l, np.zeros(3), [1.0], [1.0], 0) for l in (0, 1, 2, 3)]
    shells += [lai.Shell(l, R * u, [1.0], [1.0], 1) for l in (0, 1)]
    shells += [lai.Shell(l, R * u + np.array([0.3, -0.2, 0.1]), [1.0], [1.0], 2) for l in (0, 1)]
    b = lai.BasisSet(shells)
    eng = lai.Engine(b, threshold=0.0)
    bra = [(0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (3, 0), (1, 4), (2, 4)]
    ket = [(4, 4), (5, 4), (6, 4), (7, 4), (5, 6), (5, 5)]
    q = np.array([(*x, *y) for x in bra for y in ket], dtype=np.int32)
    values, meta = eng.eri_quartets(q)
    for row, m in zip(q, meta):
        n = int(m[5] * m[6] * m[7] * m[8])
        ref = np.asarray(oracle.orc_quartet(b, *[int(s) for s in row])).reshape(-1)
        got = values[m[0]:m[0] + n]
        # rounding of some ten terms, none more than ten times the s integral at the same T
        scale = max(np.max(np.abs(ref)), 1e-3 / max(1.0, R))
        assert np.max(np.abs(got - ref)) < 2e-14 * max(1.0, scale), (row, np.max(np.abs(got - ref)))
