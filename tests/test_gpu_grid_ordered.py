"""Ordered lattices on the grid engine: one cluster of every tile must not leave a chain of nodes as long as the grid.

The descriptor's walk_cap bounds every union-find walk, so a tree that is too deep shows as an error of the call.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [256, 512, 768, 1024])
def test_walks_of_an_ordered_lattice_stay_short(rb, L):
    """256 and 1024: tiles of whole rows, whose only bonds out of a tile lead to the next one.  In a tile a row's
    32 words and its rows' links make walks of up to 41 steps."""
    J = np.ones(2 * L * L, dtype=np.int8)
    spec = rb.ChainSpec(L=L, realization=0, key=11 + L, beta=50.0, n_therm=2, n_bins=1, sweeps_per_bin=6)
    cs = rb.ChainSet([spec], [rb.packing.pack_couplings(J, L)])
    cs.init_spins(hot=False)
    cs.set_descriptor_field(0, "walk_cap", 48)
    cs.run_grid(8)
    cs.check_status()
    ints = cs.bins(0)[0][0]
    assert ints[8] == 6 and ints[5] == 6 * L * L and ints[11] == 6  # one cluster a sweep, of every site, wrapping
