"""Device memory while an engine is made, and the bounds of a basis whose primitive pairs
are formed in many pieces."""
import importlib
import threading

import numpy as np
import pytest

lai = importlib.import_module("libaccint-public_b200")

pytestmark = pytest.mark.gpu


def _far_apart(n, spacing=14.0):
    """n water molecules on a line: 37 primitives each in cc-pVDZ, pairs of two molecules
    below any cut."""
    one = np.array([[0.0, 0.0, 0.0], [0.0, 1.43, 1.11], [0.0, -1.43, 1.11]])
    xyz = np.concatenate([one + [spacing * i, 0.0, 0.0] for i in range(n)])
    return lai.BasisSet.from_atoms(np.array([8, 1, 1] * n), xyz, "cc-pvdz")


def test_engine_set_up_holds_no_table_of_every_primitive_pair():
    import torch
    lai.Engine(_far_apart(1)).close()  # context, lookup tables, pools
    basis = _far_apart(110)  # 8.3e6 primitive pairs, 2.8 GB of unsorted tables
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    least, done = [before], threading.Event()

    def watch():
        while not done.is_set():
            least[0] = min(least[0], torch.cuda.mem_get_info()[0])

    t = threading.Thread(target=watch)
    t.start()
    eng = lai.Engine(basis)
    done.set()
    t.join()
    kept = before - torch.cuda.mem_get_info()[0]
    # the pieces, 16 bytes for each pair or primitive pair (bounds, order, pair lists), and
    # allocation granularity
    nprim, nsh = sum(len(s.exps) for s in basis.shells), basis.n_shells
    pairs = (nprim * nprim + nsh * nsh) // 2
    assert before - least[0] < kept + (256 << 20) + 16 * pairs + (64 << 20), (before - least[0], kept)
    # bounds of the last molecule's shells, of the last pieces, as those of the molecule alone
    one = lai.Engine(_far_apart(1)).schwarz()
    m = len(one)
    assert np.max(np.abs(eng.schwarz()[-m:, -m:] - one)) < 1e-13 * np.max(one)


def test_builds_with_bounds_made_in_pieces():
    """J and K of a molecule far from 109 others, against the molecule alone."""
    one, many = _far_apart(1), _far_apart(110)
    n = one.nbf
    rng = np.random.default_rng(0)
    C = rng.normal(size=(n, 5)) / np.sqrt(n)
    D = np.zeros((many.nbf, many.nbf))
    D[-n:, -n:] = C @ C.T
    J, K, _ = lai.Engine(many).jk(D)
    J1, K1, _ = lai.Engine(one).jk(C @ C.T)
    # the cut of 1e-12 is relative to other partners in the larger system
    assert np.max(np.abs(J[-n:, -n:] - J1)) < 1e-10
    assert np.max(np.abs(K[-n:, -n:] - K1)) < 1e-10
