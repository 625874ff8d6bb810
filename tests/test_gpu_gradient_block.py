"""The block-per-quartet gradient kernel, in classes up to (gg|gg) and with contracted
shells, against central differences of the energy of the J/K build, and its split over
lanes and blocks in the low classes."""
import importlib

import numpy as np
import pytest

lai = importlib.import_module("libaccint-public_b200")

pytestmark = pytest.mark.gpu


def _basis(shells, centres):
    rng = np.random.default_rng(5)
    out = []
    for i, (l, k) in enumerate(shells):
        e = np.sort(rng.uniform(0.3, 1.5, k))[::-1] * (2.5 ** np.arange(k)[::-1])
        out.append(lai.Shell(l, centres[i % len(centres)], e, rng.uniform(0.3, 1.0, k), i % len(centres)))
    return lai.BasisSet(out)


@pytest.mark.parametrize("shells", [
    [(4, 1), (3, 1), (2, 1), (1, 1)],
    [(3, 2), (3, 1), (1, 3), (0, 4)],
    [(4, 2), (0, 5), (2, 2)],
    [(2, 1), (2, 1), (1, 1), (1, 2), (1, 1), (0, 9), (0, 1)],
])
def test_gradient_matches_differences(shells):
    c0 = np.array([[0.0, 0.0, 0.0], [0.4, 1.3, -0.8], [-1.1, 0.5, 0.9]])[:min(3, len(shells))]
    basis = _basis(shells, c0)
    n = basis.nbf
    rng = np.random.default_rng(1)
    C = rng.normal(size=(n, 4)) / np.sqrt(n)
    D = C @ C.T
    g = lai.Engine(basis, threshold=0.0).gradient(D)

    def energy(c):
        J, K, _ = lai.Engine(_basis(shells, c), threshold=0.0).jk(D)
        return 0.5 * np.sum(D * J) - 0.25 * np.sum(D * K)

    h = 2e-3
    fd = np.zeros_like(c0)
    for a in range(c0.shape[0]):
        for x in range(3):
            e = []
            for k in (-2, -1, 1, 2):
                c = c0.copy()
                c[a, x] += k * h
                e.append(energy(c))
            fd[a, x] = (e[0] - 8 * e[1] + 8 * e[2] - e[3]) / (12 * h)
    # differences: h^4/30 E^(5) and 1e-15 |E| / h
    assert np.max(np.abs(g - fd)) < 1e-8 * max(1.0, np.max(np.abs(fd)))
    assert np.max(np.abs(g.sum(axis=0))) < 1e-11 * max(1.0, np.max(np.abs(g)))


def test_gradient_from_two_threads_on_one_engine():
    import threading
    w = lai.workloads.make("h2o2_631g")
    eng = lai.Engine(w.basis)
    g0 = eng.gradient(w.D)
    bad = []

    def work():
        for _ in range(5):
            if np.max(np.abs(eng.gradient(w.D) - g0)) > 1e-12 * np.max(np.abs(g0)):
                bad.append(1)

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("ls", [(3,), (2, 3), (3, 4)])
def test_gradient_does_not_depend_on_the_order_of_shells(ls):
    """The order decides which shell of a pair the transfer starts from; with d, f and g
    shells on three atoms the terms of a badly placed one cancel."""
    for seed in (3, 4, 5, 6):
        rng = np.random.default_rng(seed)
        Z, xyz = lai.molecules.water_cluster_n(1, rng)
        shells = [s for s in lai.BasisSet.from_atoms(Z, xyz, "cc-pvqz").shells if s.l in ls]
        at = np.cumsum([0] + [s.n_functions for s in shells])
        n = int(at[-1])
        C = rng.normal(size=(n, 5)) / np.sqrt(n)
        D = C @ C.T
        orders = [range(len(shells)), range(len(shells) - 1, -1, -1),
                  sorted(range(len(shells)), key=lambda i: -min(shells[i].exps))]
        got = []
        for order in orders:
            idx = np.concatenate([np.arange(at[i], at[i + 1]) for i in order])
            got.append(lai.Engine(lai.BasisSet([shells[i] for i in order]), threshold=0.0).gradient(D[np.ix_(idx, idx)]))
        # each is off by 1e-15 to 5e-15 of its norm; with the transfer started from a
        # shell's centre on both sides by 2e-14 to 2e-13
        for g in got[1:]:
            assert np.linalg.norm(g - got[0]) < 1.2e-14 * np.linalg.norm(got[0]), (seed, np.linalg.norm(g - got[0]))


# pairs of g and f shells on different centres: 165 rows about the charge, contracted shells
# whose other primitives lie away from it, kets that stay about their first shell
@pytest.mark.parametrize("shells", [[(4, 1), (4, 1), (3, 1)], [(4, 1), (3, 2), (4, 1), (2, 2), (2, 1)]])
def test_gradient_of_two_centre_pairs(shells):
    test_gradient_matches_differences(shells)
