"""sw_sweep after a device error: the call that met it raises, the next one starts with a clear status word."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [64, 200])
def test_error_of_one_call_is_not_the_next_ones(rb, orc, L):
    """The descriptor's walk_cap = 1 makes the walk bounds fire (one CTA at L = 64, the grid engine at L = 200)."""
    lattice, J = rb.build_lattice(L), np.ones(2 * L * L, dtype=np.int8)
    beta, key = 1.0 / 2.2, 17
    spins = orc.initial_spins(L * L, key, hot=False).astype(np.int64)
    ref = spins.astype(np.int8).copy()
    rb.sw_sweep(spins, lattice, J, beta, key=key, sweep=0)
    orc.sw_sweep(L, ref, J, key, rb.packing.threshold(beta), 0, measure=False)
    state = rb.swendsen_wang._sweep_state(L, None)
    state.desc["walk_cap"] = 1
    try:
        with pytest.raises(rb.RbimError, match="status word"):
            rb.sw_sweep(spins, lattice, J, beta, key=key, sweep=1)
    finally:
        state.desc["walk_cap"] = 0
    assert np.array_equal(spins, ref.astype(np.int64))  # left as they were
    for t in range(1, 4):
        res = rb.sw_sweep(spins, lattice, J, beta, key=key, sweep=t)
        r = orc.sw_sweep(L, ref, J, key, rb.packing.threshold(beta), t, measure=True)
        assert np.array_equal(spins, ref.astype(np.int64))
        assert (res.energy, res.n_clusters, res.largest_abs_magnetization) == (r[0], r[2], r[4])
