"""Arguments that the kernels' C entry points refuse before any launch, so that it shows without a device."""
import ctypes

import pytest


def _entry(library, name):
    from picolm_b200.csrc.build import load_library
    from picolm_b200.ops import _lib
    f = getattr(load_library(library), name)
    f.argtypes, f.restype = _lib._SIGNATURES[name], ctypes.c_int
    return f


@pytest.mark.parametrize("max_new", [95, 96, 400])
def test_a_decay_from_logits_wants_its_bias(max_new):
    """Every kernel that linear attention may run for a decay per key channel, whatever the prompt's length."""
    some = ctypes.create_string_buffer(64)                   # an address; nothing is read behind it
    T, H, N, P, bf16 = max_new, 2, 64, 64, 1
    row = H * N
    assert _entry("scan_chunk", "plm_sigmoid_chunk_scan")(
        some, some, some, some, bf16, row, row, H * P, row, None, 1.0, 0.5, some, H * N * P, some, some, 1 << 20, some, some, T, 1, max_new, H, N, P, 1,
        None, None) == -2
    assert _entry("recurrent", "plm_sigmoid_decay")(some, bf16, row, None, 0.5, some, T, row, None) == -2
    mode = 2                                                 # the decay from logits
    assert _entry("recurrent", "plm_linear_scan")(
        some, some, some, some, bf16, row, row, H * P, row, mode, None, None, None, 1.0, 0.5, some, H * N * P, some, H * P, some, some, 1, H, N,
        P, 1, max_new, 1, None, None, 0, None) == -2


@pytest.mark.gpu
@pytest.mark.parametrize("n", [95, 96, 400])
@pytest.mark.parametrize("N", [64, 160])
def test_linear_attention_without_a_bias_is_refused(n, N):
    """At every length, and for key sizes that only the general scan takes."""
    import torch
    import types
    from picolm_b200 import ops
    H, P = 2, 32
    rows = lambda c: torch.zeros(n, c, dtype=torch.bfloat16, device="cuda:0")
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda:0")
    step = types.SimpleNamespace(n_seqs=1, n_tokens=n, max_new=n, is_decode=False, seq_start=i32([0, n]), seq_slot=i32([0]))
    with pytest.raises(ops.KernelError, match="refused"):
        ops.linear_scan(rows(H * N), rows(H * N), rows(H * P), rows(H * N), ops.DECAY_SIGMOID, None, None, None, 1.0, 0.5,
                        torch.zeros(1, H * N * P, device="cuda:0"), step, H, N, P)
