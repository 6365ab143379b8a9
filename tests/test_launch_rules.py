"""CTA-size rules of the resident engine at the edges of their ranges, as measured (no GPU)."""

import pytest


def test_single_lattice_cta_sizes(rb):
    """512 threads up to L = 32 and from 97 to 128, 1024 elsewhere up to the engine's largest lattice."""
    size = rb.engine.single_cta_threads
    assert {L: size(L) for L in (3, 24, 32, 33, 64, 96, 97, 112, 128, 129, 144, 181, 192, 224, 255, 256)} == {
        3: 512, 24: 512, 32: 512, 33: 1024, 64: 1024, 96: 1024, 97: 512, 112: 512, 128: 512, 129: 1024, 144: 1024,
        181: 1024, 192: 1024, 224: 1024, 255: 1024, 256: 1024}
