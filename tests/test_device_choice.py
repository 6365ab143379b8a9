"""Which device a call means: resolved to an index when it is given, not when it is used (no GPU)."""

import pytest


@pytest.mark.parametrize("given,current,index", [(None, 1, 1), ("cuda", 0, 0), ("cuda", 1, 1), ("cuda:0", 1, 0),
                                                 ("cuda:3", 1, 3)])
def test_device_index_is_resolved(rb, monkeypatch, given, current, index):
    import torch

    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: current)
    for form in (given, given and torch.device(given)):
        assert rb.engine.require_cuda(form) == torch.device("cuda", index)


def test_other_devices_stay_refused(rb, monkeypatch):
    import torch

    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    with pytest.raises(rb.RbimError, match="CUDA devices only"):
        rb.engine.require_cuda("cpu")
