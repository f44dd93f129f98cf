"""Recurrences with a decay per key channel, 64 tokens at a time (csrc/scan_chunk.cu): against the recurrence in float64,
at the edges of chunks, blocks and tiles."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _step(lens):
    start = [0]
    for n in lens:
        start.append(start[-1] + n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    return types.SimpleNamespace(n_seqs=len(lens), n_tokens=start[-1], max_new=max(lens), is_decode=max(lens) == 1, seq_start=i32(start),
                                 seq_slot=i32(list(range(len(lens)))[::-1]))


def _recurrence(q, k, v, decay, beta, state, lens):
    """float64; `state` [sequences, H, N, P] in the order of the slots."""
    outs, states, at = [], [None] * len(lens), 0
    for b, n in enumerate(lens):
        S = state[len(lens) - 1 - b].double()
        for t in range(at, at + n):
            S = S * decay[t][:, :, None]
            u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
            S = S + k[t][:, :, None] * u[:, None]
            outs.append(torch.bmm(q[t][:, None], S)[:, 0])
        states[len(lens) - 1 - b] = S
        at += n
    return torch.stack(outs), torch.stack(states)


def _off(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


LENS = [[64], [65, 1, 63], [16, 130, 3], [200]]
SIZES = [(2, 1, 128, 128), (3, 3, 64, 72), (2, 2, 48, 6), (1, 1, 20, 33), (2, 1, 100, 260)]
# The state and the outputs are sums of at most a few hundred terms in float32 whose factors (exponentials of sums of at most
# 64 logarithms, products of three of them) are each off by a few units of 2^-24: 1e-6 over vectors whose errors do not align.
BOUND = 1e-6


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("H,G,N,P", SIZES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("head_decay", [False, True])
def test_delta_rule_in_chunks(lens, H, G, N, P, dtype, head_decay):
    from picolm_b200 import ops
    if head_decay and dtype == torch.bfloat16:
        pytest.skip("one decay a head in bfloat16 has kernels of its own")
    torch.manual_seed(sum(lens) + N + P)
    T, step = sum(lens), _step(lens)
    unit = lambda: torch.nn.functional.normalize(torch.randn(T, G, N, device=DEV) + 0.3, dim=-1).reshape(T, G * N).contiguous()
    q, k, v = unit(), unit(), torch.randn(T, H * P, device=DEV).to(dtype)
    # decays from almost one to almost nothing, neighbours of very different strength
    decay = -torch.exp(3 * torch.randn(T, H if head_decay else H * N, device=DEV) - 3)
    beta = torch.rand(T, H, device=DEV)
    state0 = torch.randn(len(lens) + 1, H, N, P, device=DEV)
    state = state0.clone().view(len(lens) + 1, -1)
    y = ops.delta_scan(q, k, (q.view(T, G, N) * k.view(T, G, N)).sum(-1).contiguous(), decay, beta, v, state, step, H, N, P,
                       heads_per_group=H // G, head_decay=head_decay)
    wide = lambda x: x.double().view(T, G, N).repeat_interleave(H // G, 1)
    d = torch.exp(decay.double()).view(T, H, -1).expand(T, H, N)
    o, S = _recurrence(wide(q), wide(k), v.double().view(T, H, P), d, beta.double(), state0, lens)
    assert _off(y.view(T, H, P), o) < BOUND and _off(state.view(-1, H, N, P)[:len(lens)], S) < BOUND
    assert torch.equal(state[len(lens)], state0[len(lens)].view(-1))


@pytest.mark.parametrize("lens", [[128], [129], [191], [400]] + [[65, 130, 3], [192, 64, 1]])
@pytest.mark.parametrize("H,G,N,P", SIZES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_linear_attention_in_chunks(lens, H, G, N, P, dtype):
    """Column slices of a wider projection, and a group of heads that shares keys and queries."""
    from picolm_b200 import ops
    torch.manual_seed(sum(lens) + N + P)
    T, step = sum(lens), _step(lens)
    rows = torch.randn(T, 2 * G * N + H * P + H * N + 3, device=DEV).to(dtype)
    q, k, v, raw = (t[:, :w] for t, w in ((rows, G * N), (rows[:, G * N:], G * N), (rows[:, 2 * G * N:], H * P),
                                          (rows[:, 2 * G * N + H * P:], H * N)))
    bias, power = torch.rand(H * N, device=DEV) * 8 - 4, 1.0 / 16.0
    state0 = torch.randn(len(lens) + 1, H, N, P, device=DEV)
    state = state0.clone().view(len(lens) + 1, -1)
    y = ops.linear_scan(q, k, v, raw, ops.DECAY_SIGMOID, bias, None, None, N ** -0.5, power, state, step, H, N, P, heads_per_group=H // G)
    wide = lambda x: x.double().reshape(T, G, N).repeat_interleave(H // G, 1)
    d = (torch.sigmoid(raw.double() + bias.double()) ** power).view(T, H, N)
    o, S = _recurrence(wide(q) * N ** -0.5, wide(k), v.double().reshape(T, H, P), d, None, state0, lens)
    assert _off(y.view(T, H, P), o) < BOUND and _off(state.view(-1, H, N, P)[:len(lens)], S) < BOUND
    assert torch.equal(state[len(lens)], state0[len(lens)].view(-1))


def _rows_before(lens, poisoned):
    """Per token: whether what it sees (its own sequence up to itself) is clean of the poisoned tokens."""
    out, at = [], 0
    for n in lens:
        bad = False
        for t in range(at, at + n):
            bad = bad or t in poisoned
            out.append(not bad)
        at += n
    return torch.tensor(out, device=DEV)


@pytest.mark.parametrize("H,G,N,P", [(2, 1, 128, 128), (3, 3, 48, 72), (2, 2, 100, 33)])
@pytest.mark.parametrize("where", ["v", "k", "q", "decay"])
@pytest.mark.parametrize("what", [float("inf"), float("nan")])
@pytest.mark.parametrize("rule", ["channel", "head", "linear"])
def test_what_is_not_finite_reaches_no_earlier_token(H, G, N, P, where, what, rule):
    """Poisoned tokens at the places of a block of four, of sixteen and of a chunk: the tokens before them and the other
    sequences have the bits that they have without, and one value column of v touches that column alone."""
    from picolm_b200 import ops
    lens = [200, 96, 130]
    T, step, poisoned = sum(lens), _step(lens), {2, 61, 200 + 79, 200 + 96 + 128}
    torch.manual_seed(N + P)
    x = {n: torch.randn(T, c, device=DEV) for n, c in (("q", G * N), ("k", G * N), ("v", H * P), ("decay", H if rule == "head" else H * N))}
    x["k"] = torch.nn.functional.normalize(x["k"].view(T, G, N), dim=-1).reshape(T, G * N).contiguous()
    if rule != "linear":
        x["decay"] = -x["decay"].abs()
    beta, bias = torch.rand(T, H, device=DEV), torch.rand(H * N, device=DEV)
    state0 = torch.randn(len(lens), H * N * P, device=DEV)

    def run(x):
        state = state0.clone()
        if rule == "linear":
            y = ops.linear_scan(x["q"], x["k"], x["v"], x["decay"], ops.DECAY_SIGMOID, bias, None, None, 1.0, 1 / 16, state, step, H, N, P,
                                heads_per_group=H // G)
        else:
            y = ops.delta_scan(x["q"], x["k"], torch.ones(T, G, device=DEV), x["decay"], beta, x["v"], state, step, H, N, P,
                               heads_per_group=H // G, head_decay=rule == "head")
        return y
    clean = run(x)
    assert torch.isfinite(clean).all()
    column = 5                                                           # of the first head
    for t in poisoned:
        if where == "v":
            x["v"][t, column] = what
        else:
            x[where][t] = what if where != "decay" or rule == "linear" else -abs(what)
    y = run(x)
    before = _rows_before(lens, poisoned)
    assert before.sum() > 100 and torch.equal(y[before], clean[before])
    if where == "v":
        others = torch.arange(H * P, device=DEV) != column
        assert torch.equal(y[:, others], clean[:, others])
        assert not torch.isfinite(y[sorted(poisoned), column]).any()


@pytest.mark.parametrize("H,G,N,P", [(2, 1, 128, 128), (3, 3, 48, 72)])
@pytest.mark.parametrize("rule", ["channel", "linear"])
@pytest.mark.parametrize("slots", [1, 3, 8])
def test_a_workspace_that_does_not_hold_the_step(H, G, N, P, rule, slots, monkeypatch):
    """Room for one chunk, three and eight: the step goes some chunks of some sequences at a time, to the same bits."""
    from picolm_b200 import ops
    from picolm_b200.ops import recurrent
    lens = [200, 1, 96, 330, 64]
    T, step = sum(lens), _step(lens)
    torch.manual_seed(N + P)
    q, k, v = torch.randn(T, G * N, device=DEV), torch.randn(T, G * N, device=DEV) * N ** -0.5, torch.randn(T, H * P, device=DEV)
    decay, beta, bias = torch.randn(T, H * N, device=DEV), torch.rand(T, H, device=DEV), torch.rand(H * N, device=DEV)
    state0 = torch.randn(len(lens), H * N * P, device=DEV)

    def run():
        state = state0.clone()
        if rule == "linear":
            return ops.linear_scan(q, k, v, decay, ops.DECAY_SIGMOID, bias, None, None, 1.0, 1 / 16, state, step, H, N, P, heads_per_group=H // G), state
        return ops.delta_scan(q, k, torch.ones(T, G, device=DEV), -decay.abs(), beta, v, state, step, H, N, P, heads_per_group=H // G), state
    whole = run()
    ops.check_status(DEV)
    each = recurrent._chunk_floats[N, P] * H
    monkeypatch.setattr(recurrent, "SCAN_CHUNK_FLOATS", slots * each)
    floats, stretches = recurrent.scan_chunk_plan(T, len(lens), max(lens), H, N, P)
    assert floats == slots * each and stretches == {1: 30, 3: 12, 8: 6}[slots]
    before = ops.launch_count()
    parts = run()
    ops.check_status(DEV)
    assert ops.launch_count() - before == (4 if rule == "linear" else 3) * stretches
    assert torch.equal(parts[0], whole[0]) and torch.equal(parts[1], whole[1])


@pytest.mark.parametrize("rule", ["channel", "linear"])
def test_long_prompts_take_a_bounded_workspace(rule):
    """One prompt of 40,000 tokens, 8 heads of 128 x 128: 1.1 GB for all its chunks."""
    from picolm_b200 import ops
    T, H, N, P = 40000, 8, 128, 128
    step = _step([T])
    q, k, v = [torch.randn(T, H * N, device=DEV) * N ** -0.5 for _ in range(3)]
    decay, beta, state = -torch.rand(T, H * N, device=DEV), torch.rand(T, H, device=DEV), torch.zeros(1, H * N * P, device=DEV)
    bias, qk = torch.rand(H * N, device=DEV), torch.ones(T, H, device=DEV)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    held = torch.cuda.memory_allocated()
    if rule == "linear":
        y = ops.linear_scan(q, k, v, decay, ops.DECAY_SIGMOID, bias, None, None, 1.0, 1 / 16, state, step, H, N, P)
    else:
        y = ops.delta_scan(q, k, qk, decay, beta, v, state, step, H, N, P)
    ops.check_status(DEV)
    assert torch.isfinite(y).all()
    assert torch.cuda.max_memory_allocated() - held <= y.numel() * 4 + (520 << 20)
