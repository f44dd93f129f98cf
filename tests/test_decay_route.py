"""When a constant decay's recurrence over rotated rows runs 128 tokens at a time: by what a step's sequences bring, in a captured
step as in one that is launched kernel by kernel."""
import types

import pytest
import torch

from picolm_b200.config.spec import PartSpec
from picolm_b200.ops import StepShape, recurrent
from picolm_b200.parts import build_part


@pytest.mark.parametrize("lens,expected", [([64], False), ([129], True), ([200], True), ([2048], True), ([129] * 4, False), ([170] * 3, False),
                                           ([256] * 4, False), ([100] * 16, False), ([2048, 1, 1, 1], True), ([700] + [60] * 20, False),
                                           ([1024] * 2, True)])
def test_by_the_sequences(lens, expected):
    assert recurrent.decay_in_128(StepShape.of(lens), 16, 128, 256) == expected


@pytest.mark.parametrize("lens,tokens,seqs,expected", [([200], 256, 2, True), ([129], 192, 2, True), ([170] * 3, 512, 5, False), ([600] * 3, 2048, 5, True)])
def test_a_captured_step_goes_by_its_shape_and_not_by_its_bounds(lens, tokens, seqs, expected):
    step = types.SimpleNamespace(n_tokens=tokens, n_seqs=seqs, max_new=tokens, shape=StepShape.of(lens))
    floats = recurrent._decay_tc_floats(step, 16, 128, 256, types.SimpleNamespace(half=64))
    assert floats == (2 * (tokens // 128 + seqs) * 16 * 128 * 256 if expected else 0)


@pytest.mark.parametrize("tokens,expected", [(127 * 128 + 127, True), (128 * 128, False), (40000, False)])
def test_no_more_workspace_than_half_a_gigabyte(tokens, expected):
    """Beyond that a step runs 64 tokens at a time, whose workspace is a state a segment."""
    step = types.SimpleNamespace(n_tokens=tokens, n_seqs=1, max_new=tokens)
    floats = recurrent._decay_tc_floats(step, 16, 128, 256, types.SimpleNamespace(half=64))
    assert (floats > 0) == expected and floats * 4 <= 512 << 20


def test_a_part_says_how_it_runs_a_shape():
    def part(dtype, dim, vdim):
        params = dict(hidden_size=64, heads=16, dim=dim, vdim=vdim, decay=[0.9] * 16, eps=1e-5, position=None)
        return build_part("mixer", PartSpec("retention", params), types.SimpleNamespace(dtype=dtype))
    p = part(torch.bfloat16, 128, 256)
    assert p.chooses_by_shape and p.step_route(StepShape.of([200])) != p.step_route(StepShape.of([100] * 16))
    assert not part(torch.float32, 128, 256).chooses_by_shape and not part(torch.bfloat16, 96, 256).chooses_by_shape
