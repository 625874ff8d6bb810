"""The block-per-quartet J/K kernel against J and K contracted on the host from the raw
integrals (another kernel family), in every class up to (gg|gg)."""
import importlib

import numpy as np
import pytest

lai = importlib.import_module("libaccint-public_b200")

pytestmark = pytest.mark.gpu


def _basis(shells):
    """[(l, primitives)] on three centres."""
    rng = np.random.default_rng(5)
    centres = np.array([[0.0, 0.0, 0.0], [0.3, 1.1, -0.7], [-0.9, 0.4, 0.8]])
    out = []
    for i, (l, k) in enumerate(shells):
        e = np.sort(rng.uniform(0.3, 2.5, k))[::-1] * (3.0 ** np.arange(k)[::-1])
        out.append(lai.Shell(l, centres[i % 3], e, rng.uniform(0.3, 1.0, k), i % 3))
    return lai.BasisSet(out)


def _host_jk(eng, n, D):
    values, meta = eng.compute_batch_screened()
    T = np.zeros((n, n, n, n))
    for off, fa, fb, fc, fd, na, nb, nc, nd in meta:
        g = values[off:off + na * nb * nc * nd].reshape(na, nb, nc, nd)
        a, b, c, d = slice(fa, fa + na), slice(fb, fb + nb), slice(fc, fc + nc), slice(fd, fd + nd)
        for g1, x, y in ((g, a, b), (g.transpose(1, 0, 2, 3), b, a)):
            for g2, z, w in ((g1, c, d), (g1.transpose(0, 1, 3, 2), d, c)):
                T[x, y, z, w] = g2
                T[z, w, x, y] = g2.transpose(2, 3, 0, 1)
    return np.einsum("abcd,cd->ab", T, D), np.einsum("acbd,cd->ab", T, D)


# one primitive per shell (no list), several (list, table batches, quartets shared by
# blocks), a mixture with g shells, and enough pairs for several quartets per block
@pytest.mark.parametrize("shells", [
    [(4, 1), (4, 1), (3, 1), (2, 1), (1, 1), (0, 1)],
    [(3, 3), (3, 1), (2, 2), (1, 4), (0, 6)],
    [(4, 2), (2, 1), (0, 9), (1, 3)],
    [(2, 1)] * 6 + [(1, 2)] * 4 + [(3, 1)] * 2,
])
def test_block_kernel_equals_host_digestion(shells):
    basis = _basis(shells)
    n = basis.nbf
    rng = np.random.default_rng(1)
    D = rng.normal(size=(n, n))
    D = D + D.T
    eng = lai.Engine(basis, threshold=0.0)
    J, K, _ = eng.jk(D)
    Jh, Kh = _host_jk(eng, n, D)
    # sums of at most n^2 products of 1e-15 relative error each
    bound = 1e-15 * n * n
    assert np.max(np.abs(J - Jh)) < bound * np.max(np.abs(Jh))
    assert np.max(np.abs(K - Kh)) < bound * np.max(np.abs(Kh))
    Jm, Km, rep = eng.jk(D, fp32_cut=1e30)
    assert rep.quartets_fp32 > 0
    # FP32 roots, tables and primitive sums: 24-bit rounding of terms up to some ten times
    # the sum (recurrences with both signs)
    assert np.max(np.abs(Jm - Jh)) < 1e-5 * np.max(np.abs(Jh))
    assert np.max(np.abs(Km - Kh)) < 1e-5 * np.max(np.abs(Kh))


@pytest.mark.parametrize("ls", [(2,), (3,), (2, 3), (3, 4)])
def test_transfer_on_both_sides_keeps_precision(ls):
    """d, f and g shells on three centres: the transfer of (ff|ff) and its neighbours, done
    once per quartet, must not lose what doing it per root keeps (the raw integrals' kernel)."""
    rng = np.random.default_rng(3)
    Z, xyz = lai.molecules.water_cluster_n(1, rng)
    basis = lai.BasisSet([s for s in lai.BasisSet.from_atoms(Z, xyz, "cc-pvqz").shells if s.l in ls])
    n = basis.nbf
    C = rng.normal(size=(n, 5)) / np.sqrt(n)
    D = C @ C.T
    eng = lai.Engine(basis, threshold=0.0)
    J, K, _ = eng.jk(D)
    Jh, Kh = _host_jk(eng, n, D)
    # both routes round some hundred terms per element to 1e-16, their errors independent:
    # 2e-15 of the norm, 7e-15 in the d shells' K, small by cancellation in D.  Transferred
    # about the first shell's centre on both sides, K' of (3,) is off by 4e-14
    assert np.linalg.norm(J - Jh) < 5e-15 * np.linalg.norm(Jh)
    assert np.linalg.norm(K - Kh) < 1e-14 * np.linalg.norm(Kh)


# contracted g, f and d shells on different centres: primitives away from the expansion centre
@pytest.mark.parametrize("shells", [[(4, 2), (4, 1), (3, 2), (0, 1)], [(4, 1), (3, 3), (2, 3), (2, 2), (1, 2)]])
def test_contracted_pairs_of_two_centres(shells):
    test_block_kernel_equals_host_digestion(shells)
