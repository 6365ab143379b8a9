"""Host copies: labels widened through pinned chunks, sw_sweep's one copy each way."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks,extra", [(0, 0), (0, 1), (1, -1), (1, 0), (1, 1), (2, 0), (3, 7)])
def test_labels_widened_in_chunks(rb, chunks, extra):
    import torch

    stage = rb.clusters._STAGE
    n = chunks * stage + extra
    t = (torch.arange(n, dtype=torch.int32, device="cuda") * 3 - 5).view(1, n)
    out = rb.clusters._to_host_int64(t)
    assert out.dtype == np.int64 and out.shape == (1, n) and out.flags.writeable
    assert np.array_equal(out[0], np.arange(n, dtype=np.int64) * 3 - 5)


@pytest.mark.parametrize("form", ["bool", "uint8", "int64", "strided"])
def test_mask_forms_label_alike(rb, orc, form):
    L = 20
    mask = np.random.default_rng(3).random((3, 2 * L * L)) < 0.5
    given = {"bool": mask, "uint8": mask.astype(np.uint8), "int64": mask.astype(np.int64),
             "strided": np.repeat(mask, 2, axis=1)[:, ::2]}[form]
    ncl, labels, wraps = rb.label_and_wrap_many(given, L)
    for k in range(3):
        n, lab, wx, wy = orc.label_and_wrap(mask[k], L)
        assert ncl[k] == n and np.array_equal(labels[k], lab) and tuple(wraps[k]) == (wx, wy)


def test_sw_sweep_after_an_error_and_in_threads(rb, orc):
    L = 24
    lattice = rb.build_lattice(L)
    J = np.where(np.random.default_rng(1).random(2 * L * L) < 0.1, -1, 1).astype(np.int8)
    with pytest.raises(ValueError):
        rb.sw_sweep(np.zeros(L * L, dtype=np.int64), lattice, J, 0.5, key=3)

    def run(key, bad):
        spins = orc.initial_spins(L * L, key, hot=True).astype(np.int64)
        ref = spins.astype(np.int8).copy()
        for t in range(20):
            res = rb.sw_sweep(spins, lattice, J, 0.5, key=key, sweep=t)
            r = orc.sw_sweep(L, ref, J, key, rb.packing.threshold(0.5), t, measure=True)
            if not np.array_equal(spins, ref) or res.energy != r[0] or res.n_clusters != r[2]:
                bad.append((key, t))

    bad = []
    threads = [threading.Thread(target=run, args=(k, bad)) for k in (11, 12, 13)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
