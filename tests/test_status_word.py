"""What `check_status` makes of each code that kernels write into the status word."""
import glob
import os
import re

import pytest
import torch

from picolm_b200 import ops
from picolm_b200.ops import _lib

CSRC = os.path.join(os.path.dirname(_lib.__file__), "..", "csrc")


def _waits_in_the_sources():
    """The codes that bounded waits are given in the kernels' sources."""
    text = "".join(open(f).read() for pattern in ("*.cu", "*.cuh") for f in glob.glob(os.path.join(CSRC, pattern)))
    return sorted({int(n) for n in re.findall(r"mbar_wait(?:_warp)?\([^;]*?status, (\d+)\)", text)} - {0})


def _message(code, monkeypatch):
    monkeypatch.setitem(_lib._status, torch.device("cpu"), torch.tensor([code], dtype=torch.int32))
    with pytest.raises(ops.KernelError) as e:
        ops.check_status("cpu")
    ops.check_status("cpu")                                  # reading it cleared it
    return str(e.value)


def test_every_wait_that_runs_out_is_called_a_wait(monkeypatch):
    codes = _waits_in_the_sources()
    assert {1, 2, 3, 40, 41, 42, 43, 51, 52, 53, 54} <= set(codes)
    for code in codes:
        assert "gave up waiting" in _message(code, monkeypatch) and code in _lib._WAITS, code


@pytest.mark.parametrize("code,what", [(16, "page number"), (17, "sequence index"), (18, "position"), (19, "row index")])
def test_what_the_checked_build_meets(code, what, monkeypatch):
    assert what in _message(code, monkeypatch)
