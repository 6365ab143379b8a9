"""Default cluster plans at the edges of their ranges, with and without per-sweep records.

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
