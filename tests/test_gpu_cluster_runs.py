"""Cluster engine, tiles with few run heads: their roots and flips go by runs instead of by sites.

A run is a maximal row segment of occupied y-bonds; the rule is two run heads for each word of 32 sites.  Lattices
without an open bond, with long runs that begin and end anywhere in a word, on both sides of the rule, and half
ordered, half disordered (the two passes in one lattice) are compared with the oracle, with and without records.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cuts(L, rng, cut_y, cut_x):
    """Couplings with antiferromagnetic (at all spins up: open) y- and x-bonds at the given rates."""
    J = np.ones((L, L, 2), dtype=np.int8)
    J[..., 0][rng.random((L, L)) < cut_x] = -1
    J[..., 1][rng.random((L, L)) < cut_y] = -1
    return J


def _half(L, rng):
    J = _cuts(L, rng, 0.0, 0.0)
    J[L // 2:] = _cuts(L, rng, 0.4, 0.4)[L // 2:]
    return J


@pytest.mark.parametrize("L", [257, 313, 314, 362, 363, 404, 405, 512, 627, 700, 1001, 1024])
def test_tiles_of_few_runs(rb, orc, L):
    rng = np.random.default_rng(L)
    # Heads a word: about 32 cut_y (the rule lies at 1 / 16), and one for each row start.
    couplings = [_cuts(L, rng, 0.0, 0.0), _cuts(L, rng, 0.01, 0.3), _cuts(L, rng, 0.055, 0.02),
                 _cuts(L, rng, 0.07, 0.5), _cuts(L, rng, 0.0, 1.0), _half(L, rng)]
    starts = [np.ones(L * L, dtype=np.int8)] * len(couplings)
    wall = np.ones((L, L), dtype=np.int8)
    wall[:, L // 3:] = -1
    wall[L // 5:] *= -1
    couplings.append(couplings[0])
    starts.append(wall.reshape(-1))
    specs, packed = [], []
    for i, J in enumerate(couplings):
        packed.append(rb.packing.pack_couplings(J.reshape(-1), L))
        specs += [rb.ChainSpec(L=L, realization=i, key=0x52 + 17 * i + L, beta=50.0, n_therm=1, n_bins=1,
                               sweeps_per_bin=2, records=records) for records in (False, True)]
    cs = rb.ChainSet(specs, packed)
    for k, s in enumerate(specs):
        cs.set_spins(k, rb.packing.pack_spins(starts[s.realization], L))
    cs.run_batched(3)
    cs.check_status()
    for i, J in enumerate(couplings):
        k, s = 2 * i, specs[2 * i]
        thr = rb.packing.threshold(s.beta)
        spins = starts[i].copy()
        rows = [orc.sw_sweep(L, spins, J.reshape(-1), s.key, thr, t, measure=True) for t in range(3)][1:]
        ib, _, end = orc.run_chain(L, J.reshape(-1), s.key, thr, n_therm=1, n_bins=1, sweeps_per_bin=2,
                                   spins=starts[i])
        for at in (k, k + 1):
            assert np.array_equal(cs.bins(at)[0], ib), (L, i)
            assert np.array_equal(cs.spins(at), end.astype(np.int64)), (L, i)
        assert np.array_equal(cs.chain_records(k + 1), np.array(rows, dtype=np.int64)), (L, i)
