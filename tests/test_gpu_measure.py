"""Measured sweeps of ordered lattices whose clusters are known in advance: domains, stripes, ties and tiny seconds.

At beta = 50 every satisfied bond is occupied, so the clusters of the first sweep are the chosen domains: two of equal
size, a largest one that few of the sampled sites share (the one "likely" to be the largest is then another), one that
holds every site from an even index on, or a second largest one at the very end of the lattice.  Bin sums, per-sweep
records (the magnetizations of the two largest clusters among them) and spins are compared with the oracle exactly,
with and without records: the largest cluster's magnetization takes another route in each.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BETA = 50.0


def _stripes(L, k, columns):
    """Spins of two domains: +1 in the first k rows (or columns), -1 in the others."""
    s = np.ones((L, L), dtype=np.int8)
    if columns:
        s[:, k:] = -1
    else:
        s[k:] = -1
    return s.reshape(-1)


def _fence(L, sites):
    """Couplings that cut the given sites (all spins up, beta = 50) from the rest: -1 across the boundary."""
    inside = np.zeros(L * L, dtype=bool)
    inside[list(sites)] = True
    g = inside.reshape(L, L)
    J = np.ones((L, L, 2), dtype=np.int8)
    J[..., 0][g != np.roll(g, -1, 0)] = -1
    J[..., 1][g != np.roll(g, -1, 1)] = -1
    return J.reshape(-1)


def _check(rb, orc, L, starts, run, beta=BETA, sweeps=1):
    """Chains of the given (couplings, spins), each with and without records, advanced by `run` and compared."""
    specs, packed = [], []
    for i, (J, _) in enumerate(starts):
        packed.append(rb.packing.pack_couplings(J, L))
        specs += [rb.ChainSpec(L=L, realization=i, key=0xD0A + 101 * i + L, beta=beta, n_therm=0, n_bins=1,
                               sweeps_per_bin=sweeps, records=records) for records in (False, True)]
    cs = rb.ChainSet(specs, packed)
    for k, s in enumerate(specs):
        cs.set_spins(k, rb.packing.pack_spins(starts[s.realization][1], L))
    run(cs)
    cs.check_status()
    for k, s in enumerate(specs):
        J, start = starts[s.realization]
        thr = rb.packing.threshold(beta)
        ib, _, spins = orc.run_chain(L, J, s.key, thr, n_therm=0, n_bins=1, sweeps_per_bin=sweeps, spins=start)
        assert np.array_equal(cs.bins(k)[0], ib), (L, s)
        assert np.array_equal(cs.spins(k), spins.astype(np.int64)), (L, s)
        if s.records:
            ref = start.copy()
            rows = [orc.sw_sweep(L, ref, J, s.key, thr, t, measure=True) for t in range(sweeps)]
            assert np.array_equal(cs.chain_records(k), np.array(rows, dtype=np.int64)), (L, s)


@pytest.mark.parametrize("columns", [False, True])
@pytest.mark.parametrize("L,threads", [(255, 0), (256, 0), (256, 128), (256, 512)])
def test_striped_starts(rb, orc, L, threads, columns):
    J = np.ones(2 * L * L, dtype=np.int8)
    starts = [(J, _stripes(L, k, columns)) for k in (100, 125, 126, 128, 140)]
    _check(rb, orc, L, starts, lambda cs: cs.run_batched(1, threads=threads))


@pytest.mark.parametrize("L,sites", [(256, (65534, 65535)), (256, (65533, 65534, 65535)), (256, range(65280, 65536)),
                                     (256, range(32768, 65536)), (255, (65023, 65024)), (64, (4094, 4095)),
                                     (32, (1022, 1023))])
def test_second_cluster_at_the_end(rb, orc, L, sites):
    starts = [(_fence(L, sites), np.ones(L * L, dtype=np.int8))]
    _check(rb, orc, L, starts, lambda cs: cs.run_batched(1))


def _blocks(L, seed, n=6):
    """Couplings of a lattice cut into blocks of three colours (all spins up, beta = 50): many clusters of like size,
    so that the largest one is often not the one most of the sampled sites share."""
    rng = np.random.default_rng(seed)
    edges = [np.searchsorted(np.sort(rng.integers(1, L, n - 1)), np.arange(L), side="right") for _ in (0, 1)]
    g = rng.integers(0, 3, (n, n))[edges[0]][:, edges[1]]
    J = np.ones((L, L, 2), dtype=np.int8)
    J[..., 0][g != np.roll(g, -1, 0)] = -1
    J[..., 1][g != np.roll(g, -1, 1)] = -1
    return J.reshape(-1)


@pytest.mark.parametrize("L,threads", [(9, 32), (31, 64), (32, 512), (40, 64), (63, 128), (64, 1024), (96, 256),
                                       (97, 512), (128, 256), (129, 1024), (181, 512), (255, 1024), (256, 1024)])
def test_blocks_on_one_cta(rb, orc, L, threads):
    starts = [(_blocks(L, 31 * L + i, 3 + 2 * i), np.ones(L * L, dtype=np.int8)) for i in range(6)]
    _check(rb, orc, L, starts, lambda cs: cs.run_batched(1, threads=threads))


@pytest.mark.parametrize("L", [257, 313, 314, 404, 512, 627, 628, 810, 1001, 1024])
def test_blocks_and_stripes_on_clusters(rb, orc, L):
    ones, J1 = np.ones(L * L, dtype=np.int8), np.ones(2 * L * L, dtype=np.int8)
    starts = [(_blocks(L, 17 * L + i, 4 + 3 * i), ones) for i in range(4)]
    starts += [(J1, _stripes(L, L // 2 + d, columns)) for columns in (False, True) for d in (0, 3)]
    _check(rb, orc, L, starts, lambda cs: cs.run_batched(1))


@pytest.mark.parametrize("L", [64, 249, 256, 700])
def test_blocks_and_stripes_on_the_grid(rb, orc, L):
    ones, J1 = np.ones(L * L, dtype=np.int8), np.ones(2 * L * L, dtype=np.int8)
    starts = [(_blocks(L, 13 * L + i, 4 + 3 * i), ones) for i in range(3)]
    starts += [(J1, _stripes(L, L // 2 + d, True)) for d in (0, 3)]
    _check(rb, orc, L, starts, lambda cs: cs.run_grid(1))


@pytest.mark.parametrize("L,threads", [(3, 32), (11, 64), (16, 1024), (33, 32), (47, 128), (65, 256), (97, 512),
                                       (127, 256), (181, 512), (185, 1024), (256, 1024), (313, 0), (363, 0), (512, 0),
                                       (769, 0), (1001, 0)])
def test_records_of_disordered_chains(rb, orc, L, threads):
    """Records sweep by sweep at the sizes where the bands of words, the CTA sizes and the cluster plans change."""
    rng = np.random.default_rng(L + threads)
    for p, T in ((0.0, 2.27), (0.1, 1.3), (0.5, 0.9)):
        J = np.where(rng.random(2 * L * L) < p, -1, 1).astype(np.int8)
        start = np.where(rng.random(L * L) < 0.5, -1, 1).astype(np.int8)
        _check(rb, orc, L, [(J, start)], lambda cs: cs.run_batched(3, threads=threads), beta=1.0 / T, sweeps=3)
