"""A torch allocation that runs out is made once more after the library gave back what its contexts
keep; a second failure is the caller's."""
import contextlib

import pytest
import torch

from quanty_gb300 import api


class Eng:
    device, torch = 0, torch

    def __init__(self):
        self.trimmed = 0
        self.L = self

    def qg_trim(self, device):
        self.trimmed += 1
        return 0

    def check(self, st):
        assert st == 0

    def on_stream(self):
        return contextlib.nullcontext()


@pytest.mark.parametrize("failures", [0, 1, 2])
def test_tried_again_once(failures):
    eng, calls = Eng(), []

    def make(dev):
        calls.append(dev)
        if len(calls) <= failures:
            raise torch.cuda.OutOfMemoryError("short")
        return len(calls)

    if failures == 2:
        with pytest.raises(torch.cuda.OutOfMemoryError):
            api._allocate(eng, make)
    else:
        assert api._allocate(eng, make) == failures + 1
    assert eng.trimmed == min(failures, 1) and calls == ["cuda:0"] * min(failures + 1, 2)
