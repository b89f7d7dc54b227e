"""The stream that captured steps branch onto."""
import gc

import pytest
import torch

import cbis_b200      # noqa: F401
from cbis_b200.engine.runner import ModelRunner

pytestmark = pytest.mark.gpu


def test_no_other_stream_is_the_branch_stream(monkeypatch):
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    runner = object.__new__(ModelRunner)
    runner._branch, runner.device = None, torch.device("cuda", 0)
    side = runner.branch_stream()
    assert side is runner.branch_stream()
    assert side.cuda_stream not in {torch.cuda.Stream().cuda_stream for _ in range(100)} | {torch.cuda.current_stream().cuda_stream}
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        x = torch.ones(1000, device="cuda") * 3
    torch.cuda.current_stream().wait_stream(side)
    assert x.sum().item() == 3000
    del runner, side
    gc.collect()
