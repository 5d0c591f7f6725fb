"""stream_handle hands out streams of CUDA devices only."""
import pytest
import torch

from flowmc_gb300 import _lib


@pytest.mark.parametrize("device", ["cpu:0", "cpu", "meta"])
def test_other_devices_are_refused(device, monkeypatch):
    monkeypatch.setattr(_lib, "_raw_stream", lambda index: 0)   # no GPU needed to ask
    with pytest.raises(Exception):
        _lib.stream_handle(torch.device(device))


def test_indexed_cuda_device_takes_the_raw_handle(monkeypatch):
    monkeypatch.setattr(_lib, "_raw_stream", lambda index: 40 + index)
    assert _lib.stream_handle(torch.device("cuda", 2)) == 42
