"""CTA-size rules of the resident engine at the edges of their ranges, as measured (no GPU)."""

import pytest


def test_single_lattice_cta_sizes(rb):
    """512 threads up to L = 32 and from 97 to 128, 1024 elsewhere up to the engine's largest lattice."""
    size = rb.engine.single_cta_threads
    assert {L: size(L) for L in (3, 24, 32, 33, 64, 96, 97, 112, 128, 129, 144, 181, 192, 224, 255, 256)} == {
        3: 512, 24: 512, 32: 512, 33: 1024, 64: 1024, 96: 1024, 97: 512, 112: 512, 128: 512, 129: 1024, 144: 1024,
        181: 1024, 192: 1024, 224: 1024, 255: 1024, 256: 1024}


@pytest.mark.parametrize("default,lattices,L,threads", [
    # The measured points of the rule's description.
    (32, 296, 32, 256), (32, 148, 16, 128), (32, 1280, 32, 64), (32, 888, 32, 128), (128, 592, 48, 256),
    (128, 296, 64, 256), (256, 148, 128, 512), (256, 296, 128, 512),
    # Both sides of each least number of sites: up to 512 threads an SM ...
    (32, 148, 5, 32), (32, 148, 6, 64), (32, 148, 11, 64), (32, 148, 12, 128), (32, 148, 22, 128), (32, 148, 23, 256),
    (32, 148, 32, 256), (32, 148, 33, 512),
    # ... up to 768 ...
    (64, 6 * 148, 19, 64), (64, 6 * 148, 20, 128), (128, 3 * 148, 31, 128), (128, 3 * 148, 32, 256),
    # ... and up to 1024.
    (64, 8 * 148, 22, 64), (64, 8 * 148, 23, 128), (128, 4 * 148, 35, 128), (128, 4 * 148, 36, 256),
    (256, 2 * 148, 95, 256), (256, 2 * 148, 96, 512), (512, 148, 135, 512), (512, 148, 136, 1024),
    # More than 1024 threads an SM are never taken.
    (32, 32 * 148 + 1, 256, 32), (512, 149, 256, 512)])
def test_cta_sizes_of_launches_of_few_lattices(rb, default, lattices, L, threads):
    assert rb.engine.occupancy_threads(default, lattices, 148, L * L) == threads


@pytest.mark.parametrize("L,engine", [(64, "batched"), (96, "batched"), (108, "batched"), (109, "grid"), (112, "grid"),
                                      (128, "grid")])
def test_one_lattice_takes_the_faster_engine(rb, L, engine):
    """Up to L = 108 one CTA, from L = 112 the grid engine was measured faster."""
    spec = rb.ChainSpec(L=L, realization=0, key=1, beta=0.5, n_therm=0, n_bins=1, sweeps_per_bin=1)
    assert rb.engine.auto_engine([spec], lambda L: (148, 512)) == engine
