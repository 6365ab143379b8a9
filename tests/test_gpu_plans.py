"""Default launch plans: cluster plans at the edges of their ranges, with and without per-sweep records, and the CTA
sizes of launches of few lattices.

The magnetization of the largest cluster is summed with the merged sizes, or by popcounts when it is a tile's likely
largest cluster, or by a pass over the sites: with records, and when it lies inside one tile without being that
tile's likely largest.  The temperatures below have a spanning cluster, clusters of all sizes, and only small
clusters.  The integer sums and the spins are compared exactly.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [257, 313, 314, 362, 363, 404, 405, 512, 513, 572, 573, 627, 628, 768, 769, 809, 810, 1001])
def test_cluster_plan_edges_match_oracle(rb, orc, L):
    rng = np.random.default_rng(L)
    # (p, T, hot start): spanning, critical, frustrated, small clusters only, one cluster of every site.
    cases = [(0.0, 1.5, False), (0.0, 2.27, True), (0.5, 1.0, True), (0.1, 12.0, True), (0.0, 0.05, False)]
    for hot in (True, False):
        specs, packed, bonds = [], [], []
        for i, (p, T, _) in enumerate(c for c in cases if c[2] == hot):
            J = np.where(rng.random(2 * L * L) < p, -1, 1).astype(np.int8)
            bonds.append(J)
            packed.append(rb.packing.pack_couplings(J, L))
            specs += [rb.ChainSpec(L=L, realization=i, key=0xC1A5 + 97 * i + L, beta=1.0 / T, n_therm=1, n_bins=2,
                                   sweeps_per_bin=2, records=records) for records in (False, True)]
        cs = rb.ChainSet(specs, packed)
        cs.init_spins(hot=hot)
        cs.run_batched(5)
        cs.check_status()
        for k, s in enumerate(specs):
            ib, _, spins = orc.run_chain(L, bonds[s.realization], s.key, rb.packing.threshold(s.beta), hot=hot,
                                         n_therm=1, n_bins=2, sweeps_per_bin=2)
            gi, _ = cs.bins(k)
            assert np.array_equal(gi, ib), (L, hot, s)
            assert np.array_equal(cs.spins(k), spins.astype(np.int64)), (L, hot, s)


@pytest.mark.parametrize("n", [2, 149, 300, 600, 1300])
def test_few_lattice_cta_sizes_match_oracle(rb, orc, n):
    """The CTA size of a launch of few lattices: never above the occupancy bound, a supported size from the
    library's default on, and the same chains whatever it is."""
    occ = rb.engine.occupancy_threads
    for L in range(3, 200):
        d = rb._native.lib().rbim_resident_threads(L)
        t = occ(d, n, 148, L * L)
        assert d <= t <= occ(d, n, 148) and t in (32, 64, 128, 256, 512, 1024), (L, n)
    for L in (7, 16, 32, 45, 96):
        J = np.where(np.random.default_rng(L).random(2 * L * L) < 0.1, -1, 1).astype(np.int8)
        specs = [rb.ChainSpec(L=L, realization=0, key=31 * L + i, beta=1.0 / (0.8 + 0.3 * (i % 8)), n_therm=1, n_bins=2,
                              sweeps_per_bin=2) for i in range(n)]
        cs = rb.ChainSet(specs, [rb.packing.pack_couplings(J, L)])
        cs.init_spins(hot=True)
        cs.run_batched(5)
        cs.check_status()
        for i in sorted({0, 1, n // 2, n - 2, n - 1}):
            s = specs[i]
            ib, _, spins = orc.run_chain(L, J, s.key, rb.packing.threshold(s.beta), hot=True, n_therm=1, n_bins=2,
                                         sweeps_per_bin=2)
            gi, _ = cs.bins(i)
            assert np.array_equal(gi, ib), (L, n, i)
            assert np.array_equal(cs.spins(i), spins.astype(np.int64)), (L, n, i)
