"""Run links, union lists and their edges: every CTA size on sizes where the bands of words are ragged.

The open labelling splits a lattice's words in one band per warp, links run heads row by row inside a band and lists
the remaining bonds per warp; a warp may have no word, one word, or words whose bonds overflow its list (a CTA of many
threads on a small lattice has the shortest lists).  The integer sums and the spins are compared exactly; the double
sums follow from the same integers (the device fuses the product of an M^4 sum, which can differ from the oracle's in
the last bit on large ordered lattices).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,threads", [(3, 32), (3, 1024), (6, 256), (11, 64), (16, 32), (16, 1024), (31, 64), (32, 512),
                                       (33, 32), (33, 1024), (47, 128), (63, 1024), (65, 256), (96, 256), (97, 512),
                                       (120, 256), (127, 256), (128, 256), (128, 512), (129, 1024), (181, 512),
                                       (184, 512), (185, 1024), (255, 1024), (256, 1024)])
def test_resident_bands_match_oracle(rb, orc, L, threads):
    rng = np.random.default_rng(100 * L + threads)
    # Hot and critical, nearly full (long runs, one cluster), nearly empty, and frustrated.
    cases = [(0.0, 2.2), (0.0, 0.4), (0.1, 1.3), (0.5, 0.9), (0.3, 8.0)]
    specs, packed, bonds = [], [], []
    for i, (p, T) in enumerate(cases):
        J = np.where(rng.random(2 * L * L) < p, -1, 1).astype(np.int8)
        bonds.append(J)
        packed.append(rb.packing.pack_couplings(J, L))
        specs.append(rb.ChainSpec(L=L, realization=i, key=0xA11CE + 31 * i + L, beta=1.0 / T, n_therm=2, n_bins=2,
                                  sweeps_per_bin=2, records=True))
    cs = rb.ChainSet(specs, packed)
    cs.init_spins(hot=True)
    cs.run_batched(6, threads=threads)
    cs.check_status()
    for i, s in enumerate(specs):
        ib, _, spins = orc.run_chain(L, bonds[i], s.key, rb.packing.threshold(s.beta), hot=True, n_therm=2, n_bins=2,
                                      sweeps_per_bin=2)
        gi, _ = cs.bins(i)
        assert np.array_equal(gi, ib), (L, threads, cases[i])
        assert np.array_equal(cs.spins(i), spins.astype(np.int64)), (L, threads, cases[i])
