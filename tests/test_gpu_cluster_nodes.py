"""Node tables of the cluster engine: a lattice whose last site's node has its root in the table's last slot.

At L = 1024 a tile has 65536 sites and a table of 4096 slots.  Key 65535 is the last site of the lattice; joined only
to its row's start, across the y seam, it merges with the cluster of that site, whose smallest site ``key`` of the
last tile is one that the multiplicative hash sends to slot 4095.  Every other site is alone.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L, TILE = 1024, 65536
KEYS = [k for k in range(TILE) if ((k * 0x9E3779B1) & 0xFFFFFFFF) >> 20 == 4095]


@pytest.mark.parametrize("records", [False, True])
def test_last_site_with_a_root_in_the_last_slot(rb, orc, records):
    base = L * L - TILE
    keys = [k for k in KEYS if k % L < L - 2][:6]
    assert keys
    specs, packed, host = [], [], []
    for i, k in enumerate(keys):
        J = -np.ones((L, L, 2), dtype=np.int8)  # spins up, beta = 50: only bonds with J = +1 are occupied
        x, y = divmod(base + k, L)
        J[x: L - 1, y, 0] = 1  # down to the last row
        J[L - 1, :y, 1] = 1    # along it to its start
        J[L - 1, L - 1, 1] = 1  # across the y seam from the last site
        host.append(J.reshape(-1))
        packed.append(rb.packing.pack_couplings(host[-1], L))
        specs += [rb.ChainSpec(L=L, realization=i, key=0x5107 + 7 * i + 1000 * j, beta=50.0, n_therm=0, n_bins=1,
                               sweeps_per_bin=1, records=records) for j in range(3)]
    cs = rb.ChainSet(specs, packed)
    cs.init_spins(hot=False)
    cs.run_batched(1)
    cs.check_status()
    for i, s in enumerate(specs):
        thr = rb.packing.threshold(s.beta)
        ib, _, spins = orc.run_chain(L, host[s.realization], s.key, thr, hot=False, n_therm=0, n_bins=1, sweeps_per_bin=1)
        assert np.array_equal(cs.bins(i)[0], ib), keys[s.realization]
        assert np.array_equal(cs.spins(i), spins.astype(np.int64)), keys[s.realization]
        if records:
            ref = np.ones(L * L, dtype=np.int8)
            r = orc.sw_sweep(L, ref, host[s.realization], s.key, thr, 0, measure=True)
            assert tuple(int(v) for v in cs.chain_records(i)[0]) == tuple(int(v) for v in r)
