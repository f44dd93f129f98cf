"""Which steps the recurrences with a decay per key channel run 64 tokens at a time: by what the step's sequences bring, in
captured steps too, whose bounds are those of all batches of their size."""
import json

import pytest

from picolm_b200 import ops
from picolm_b200.ops import StepShape


# lengths and whether 64 tokens at a time was the faster way (8 heads of 128 x 128, microseconds that way and token by token)
@pytest.mark.parametrize("lens,chunks", [
    ([48], True),                    # 41, 45
    ([40], False),                   # 43, 38
    ([64], True),                    # 44, 59
    ([129], True),                   # 51, 115
    ([16] * 32, False),              # 190, 57
    ([63] * 32, False),              # 207, 194
    ([128] * 32, True),              # 305, 564
    ([64] + [1] * 63, False),        # 355, 69
    ([100] + [16] * 31, False),      # 196, 100
    ([200] + [1] * 31, False),       # 200, 179
    ([1000] + [20] * 8, True),       # 137, 892
])
def test_delta_rule(lens, chunks):
    assert ops.delta_scan_in_chunks(StepShape.of(lens), 8, 128, 128) == chunks


# 8 heads of 128 x 256
@pytest.mark.parametrize("lens,chunks", [
    ([95], False), ([96], True),     # (at 96) 44, 49
    ([96] * 2, False),               # 56, 49
    ([128] * 2, True),               # 57, 63
    ([128] * 16, True),              # 131, 183
    ([100] + [16] * 31, False),      # 142, 84
    ([64] + [1] * 63, False),        # 354, 82
    ([200] + [1] * 31, True),        # 146, 267 (in segments)
    ([1000] + [20] * 8, True),       # 112, 299 (in segments)
])
def test_linear_attention(lens, chunks):
    route = ops.linear_scan_route(StepShape.of(lens), 8, 128, 256)
    assert route == (ops.IN_CHUNKS if chunks else ops.ONE_PASS)


def test_the_shape_of_a_step():
    import types
    assert StepShape.of([130, 1, 64]) == (130, 195, 3, 5)
    made = types.SimpleNamespace(shape=StepShape.of([16] * 32), max_new=512, n_tokens=512, n_seqs=33)
    assert ops.step_shape(made).longest == 16
    bounds = types.SimpleNamespace(max_new=512, n_tokens=512, n_seqs=33)
    assert ops.step_shape(bounds) == (512, 512, 33, 41)


@pytest.mark.gpu
@pytest.mark.parametrize("design", ["tebasun", "potuzen"])
def test_captured_steps_go_by_the_batch_at_hand(design, tmp_path, monkeypatch):
    """32 prompts of 16 tokens and one of 481 beside 31 single tokens have one size; their graphs run the recurrence in
    different ways, and both give the logits of the step launched kernel by kernel."""
    import importlib
    from picolm_b200.engine import Engine
    from picolm_b200.ops import recurrent
    tests = importlib.import_module(f"test_gpu_{design}")
    if design == "tebasun":
        config, names = tests._config([tests._parallel()]), ("plm_delta_channel_scan", "plm_delta_scan")
    else:
        config = tests._config([{"type": "gla", "mixer": {"heads": 2, "dim": 16, "vdim": 24, "tau": 16.0, "decay_rank": 4}, "mlp": None}])
        names = "plm_sigmoid_chunk_scan", "plm_linear_scan"
    folder = tests._make(tmp_path, "shape", json.loads(json.dumps(config)), seed=4)[0]
    ran, find = [], recurrent._fn
    monkeypatch.setattr(recurrent, "_fn", lambda library, name, *more: (ran.append(name), find(library, name, *more))[1])
    engines = [Engine.from_folder(folder, dtype="bfloat16", max_tokens=64 * 80, max_seqs=32, use_graphs=graphs) for graphs in (None, False)]
    assert engines[0].prompt_graphs
    from util import random_tokens
    for turn in range(2):
        for lens, in_chunks in (([16] * 32, False), ([481] + [1] * 31, True)):
            logits = []
            for eng in engines:
                ran.clear()
                slots = [eng.new_sequence() for _ in lens]
                logits.append(eng.step([(s, random_tokens(n, 97, 7 * i + n)) for i, (s, n) in enumerate(zip(slots, lens))]).float().clone())
                for s in slots:
                    eng.end_sequence(s)
                if turn == 0 or eng is engines[1]:
                    assert names[not in_chunks] in ran and names[in_chunks] not in ran
            assert (logits[0] - logits[1]).abs().max() <= 0.02 * logits[1].std()
    assert len(engines[0]._prompt_graphs) == 2
