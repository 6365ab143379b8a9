"""Host arrays as callers hold them: read-only and memory-mapped masks are labelled without a warning."""

import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [bool, np.uint8, np.int64])
@pytest.mark.parametrize("form", ["frozen", "memmap", "frozen strided"])
def test_read_only_masks_label_quietly(rb, orc, tmp_path, form, dtype):
    import torch

    L = 20
    mask = np.random.default_rng(5).random((3, 2 * L * L)) < 0.5
    given = mask.astype(dtype)
    if form == "memmap":
        np.save(tmp_path / "mask.npy", given)
        given = np.load(tmp_path / "mask.npy", mmap_mode="r")
    elif form == "frozen strided":
        given = np.repeat(given, 2, axis=1)[:, ::2]
    if form != "memmap":
        given.setflags(write=False)
    torch.set_warn_always(True)  # torch gives this warning once per process otherwise
    try:
        with warnings.catch_warnings():
            warnings.simplefilter("error")
            ncl, labels, wraps = rb.label_and_wrap_many(given, L)
    finally:
        torch.set_warn_always(False)
    for k in range(3):
        n, lab, wx, wy = orc.label_and_wrap(mask[k], L)
        assert ncl[k] == n and np.array_equal(labels[k], lab) and tuple(wraps[k]) == (wx, wy)
    assert not given.flags.writeable and np.array_equal(given, mask.astype(dtype))
