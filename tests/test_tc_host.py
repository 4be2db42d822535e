"""Host side of the tensor-core GEMM wrapper, without a GPU."""
import pytest
import torch

from pot3d_b200 import tc


@pytest.fixture
def one_device(monkeypatch):
    """Device 1 of a machine with several, its flags in host memory."""
    zeros = torch.zeros
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 1)
    monkeypatch.setattr(torch, "zeros", lambda *a, device=None, **k: zeros(*a, **k))
    monkeypatch.setattr(tc, "_err", {})


@pytest.mark.parametrize("asked", ["cuda", "cuda:1", torch.device("cuda"), torch.device("cuda", 1)])
def test_check_errors_reads_the_flag_that_products_write(one_device, asked):
    flag = tc._err_flag(torch.device("cuda", 1))  # a tensor's device always has its index
    tc.check_errors(asked)
    flag.fill_(1)
    with pytest.raises(RuntimeError):
        tc.check_errors(asked)
    with pytest.raises(RuntimeError):
        tc.check_errors()
    tc.check_errors("cuda:0")


def test_raw_stream_without_the_private_name(monkeypatch):
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda i: type("Stream", (), {"cuda_stream": 1000 + i})())
    assert tc.raw_stream(3) == 1003


def test_unknown_activation_is_refused():
    a = torch.zeros((16, 64), dtype=torch.bfloat16)
    with pytest.raises(ValueError):
        tc.tc_gemm(a, a, act="relu")
