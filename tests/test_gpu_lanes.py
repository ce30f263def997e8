"""Quartets shared by several lanes: contractions whose primitive counts are odd, prime,
one, or below and above the lane counts, on shells of every angular momentum."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _functions(counts, ls, seed):
    from mmd.integrals.twoe import Basis
    rng = np.random.default_rng(seed)
    ours, ref = [], []
    for k, (n, l) in enumerate(zip(counts, ls)):
        centre = rng.uniform(-1.2, 1.2, 3) + [0.0, 0.0, 0.7 * (k % 3)]
        exps = 10.0 ** rng.uniform(-0.7, 2.0, n)
        coefs = rng.uniform(0.2, 1.0, n)
        for x in range(l, -1, -1):
            for y in range(l - x, -1, -1):
                shell = (x, y, l - x - y)
                ours.append(Basis(centre, shell, n, exps, coefs))
                ref.append(O.Basis(centre, shell, n, exps, coefs))
    return ours, ref


@pytest.mark.parametrize("counts,ls", [
    ((1,), (0,)),                                # one primitive quartet: nothing to share
    ((33,), (0,)),                               # one heavy quartet on a full warp
    ((7, 1, 5), (0, 0, 0)),
    ((9, 3, 1), (1, 0, 1)),
    ((2, 5, 1), (0, 1, 2)),
    ((1, 2), (2, 2)),
    ((3, 5), (2, 0)),
])
def test_shared_quartets_equal_the_oracle(counts, ls):
    from mmd.integrals.fock import formPT
    from mmd.integrals.twoe import doERIs
    ours, ref = _functions(counts, ls, seed=len(counts) + sum(counts))
    N = len(ours)
    T = doERIs(N, np.zeros((N,) * 4), ours)
    To = O.doERIs(N, np.zeros((N,) * 4), ref)
    assert np.abs(T - To).max() < 1e-12
    scr = O.screen_table(ref)
    A = np.random.default_rng(N).standard_normal((N, N))
    P = 0.5 * (A + A.T)
    G = formPT(P, np.zeros_like(P), ours, N, scr, 1e-12)
    Go = O.formPT(P, np.zeros_like(P), ref, N, scr, 1e-12)
    assert np.abs(G - Go).max() < 1e-11  # a sum of up to N^2 ERIs, each to 1e-12, over |P| ~ 1
