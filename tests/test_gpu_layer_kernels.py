"""Kernels of the recurrent layers that are chosen by size or alignment, against the forms that take anything and against
plain computations."""
import math
import types
from unittest import mock

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def _step(lens):
    start = [sum(lens[:b]) for b in range(len(lens) + 1)]
    return types.SimpleNamespace(n_seqs=len(lens), n_tokens=start[-1], max_new=max(lens), is_decode=False, seq_start=_i32(start), seq_slot=_i32(list(range(len(lens)))),
                                 tok_seq=_i32([b for b, n in enumerate(lens) for _ in range(n)]))


@pytest.mark.parametrize("K", [8, 16, 32])
@pytest.mark.parametrize("M,N", [(1, 4), (3, 1028), (17, 512), (50, 516), (33, 1028), (130, 516), (1025, 1028), (2050, 516)])
def test_products_with_few_terms_give_the_bits_of_the_general_one(M, N, K):
    from picolm_b200 import ops
    torch.manual_seed(M + N + K)
    wide = torch.randn(M, K + 6).to(torch.bfloat16).to(DEV)
    w = torch.randn(N, K).to(torch.bfloat16).to(DEV)
    a = wide[:, 3:3 + K]
    out = ops.gemm_simt(a, w, torch.bfloat16)
    general = torch.cat([ops.gemm_simt(a, w[:N - N % 4 - 1], torch.bfloat16), ops.gemm_simt(a, w[1 - 4:], torch.bfloat16)], 1)   # odd widths
    assert torch.equal(out[:, :N - N % 4 - 1], general[:, :N - N % 4 - 1]) and torch.equal(out[:, 1 - 4:], general[:, 1 - 4:])


@pytest.mark.parametrize("lens", [[1], [2, 1, 3], [5, 4, 70, 1, 1, 9], [64, 3]])
@pytest.mark.parametrize("C", [8, 1032])
def test_convolution_of_four_taps(lens, C):
    """Sequences that begin and end inside a thread's four tokens, old inputs from the state."""
    from picolm_b200 import ops
    torch.manual_seed(sum(lens) + C)
    step = _step(lens)
    wide = torch.randn(sum(lens), C + 8).to(torch.bfloat16).to(DEV)
    u, w = wide[:, :C], torch.randn(4, C, device=DEV)
    state = torch.randn(len(lens), 3 * C, device=DEV)
    back = [torch.cat([state[b].view(3, C).double(), u[s:s + n].double()]) for b, (s, n) in enumerate(zip([sum(lens[:b]) for b in range(len(lens))], lens))]
    raw = torch.cat([sum(x[j:j + n] * w[j].double() for j in range(4)) for x, n in zip(back, lens)])
    before = state.clone()
    got = ops.causal_conv(u, w, None, state, step)
    want = torch.nn.functional.silu(raw)
    # sums of four terms in fp32 (the activation's slope is at most 1.1), the activation within 2^-20, one rounding to bfloat16
    mag = torch.cat([sum((x[j:j + n] * w[j].double()).abs() for j in range(4)) for x, n in zip(back, lens)])
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1.1 * 2.0 ** -22 * mag + 2.0 ** -130).all()
    assert torch.equal(state.double().view(len(lens), 3, C), torch.stack([x[-3:] for x in back]))
    # a fifth tap of zero takes the kernel for any number of taps
    w5, state5 = torch.cat([torch.zeros(1, C, device=DEV), w]), torch.cat([torch.zeros(len(lens), C, device=DEV), before], 1)
    assert torch.equal(got, ops.causal_conv(u, w5, None, state5, step))


def test_activations_of_the_convolution_far_from_zero():
    """Inputs down to -88: a result is as exact as one rounding to bfloat16 lets it be, also where it is tiny."""
    from picolm_b200 import ops
    C, T = 64, 177
    x = torch.linspace(-88, 88, T, dtype=torch.float64).to(torch.bfloat16)
    w = torch.zeros(4, C, device=DEV)
    w[3] = 1.0
    got = ops.causal_conv(x[:, None].expand(T, C).contiguous().to(DEV), w, None, torch.zeros(1, 3 * C, device=DEV), _step([T]))
    want = torch.nn.functional.silu(x.double()).to(DEV)[:, None]
    assert ((got.double() - want).abs() <= (2.0 ** -8 + 2.0 ** -20) * want.abs()).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,G,H,N,per_head", [(1, 1, 1, 64, False), (5, 3, 6, 64, False), (33, 2, 4, 128, False), (9, 3, 3, 64, True), (7, 2, 6, 128, True)])
def test_delta_prep_by_fours(dtype, T, G, H, N, per_head):
    """Rows that can be read by fours against rows off that boundary, which the general kernel takes."""
    from picolm_b200 import ops
    torch.manual_seed(T + G + H + N)
    ND = 1 if per_head else N
    make = lambda c: torch.randn(T, c).to(dtype).to(DEV)
    q, k, z, b = make(G * N), make(G * N), make(H * ND), make(H)
    a_log, bias = torch.randn(H, device=DEV), torch.randn(H * ND, device=DEV)

    def off(x):                                              # the same values, rows one element off
        wide = torch.zeros(T, x.shape[1] + 9, dtype=dtype, device=DEV)
        wide[:, 1:1 + x.shape[1]] = x
        return wide[:, 1:1 + x.shape[1]]

    run = lambda f: ops.delta_prep(f(q), f(k), f(z), f(b), a_log, bias, 1e-6, N ** -0.5, H, N, heads_per_group=H // G, head_decay=per_head)
    for got, want in zip(run(lambda x: x), run(off)):
        # (sums of N squares in another order: at most N roundings of 2^-24 of a sum of positive terms; q . k of terms of both signs)
        assert (got - want).abs().max() <= N * 2.0 ** -24 * max(1.0, want.abs().max().item())


def _scan(q, k, v, log_decay, beta=None):
    """float64, token by token: [T, H, N], [T, H, N], [T, H, P], [T, H, N], beta [T, H] or None."""
    T, H, N = k.shape
    S, out = torch.zeros((H, N, v.shape[2]), dtype=torch.float64, device=v.device), []
    for t in range(T):
        S = S * log_decay[t].exp()[:, :, None]
        u = v[t] if beta is None else beta[t, :, None] * (v[t] - torch.bmm(k[t, :, None], S)[:, 0])
        S = S + k[t, :, :, None] * u[:, None]
        out.append(torch.bmm(q[t, :, None], S)[:, 0])
    return torch.stack(out), S


@pytest.mark.parametrize("N,P", [(128, 128), (128, 256), (64, 68), (40, 200), (100, 132)])
@pytest.mark.parametrize("lens", [[64], [65, 130], [300, 1, 128, 7]])
def test_chunk_products(N, P, lens):
    """Linear attention and the delta rule for states of more than 64 columns (whose chunks' products run on the tensor cores):
    ragged columns and channels, chunks that end early, more units than CTAs."""
    from picolm_b200 import ops
    torch.manual_seed(N + P + sum(lens))
    H, T = 6, sum(lens)
    step = _step(lens)
    q, k, v, raw = (torch.randn(T, H * c, device=DEV) for c in (N, N, P, N))
    bias = torch.randn(H * N, device=DEV)
    q, k = q * N ** -0.5, k * N ** -0.5
    start = [sum(lens[:b]) for b in range(len(lens))]
    state = torch.zeros(len(lens), H * N * P, device=DEV)
    assert ops.delta_scan_in_chunks(ops.step_shape(step), H, N, P)
    logs = torch.nn.functional.logsigmoid(raw.double() + bias.double()) / 16.0
    view = lambda x, s, n, c: x[s:s + n].double().view(n, H, c)
    got = ops.linear_scan(q, k, v, raw, ops.DECAY_SIGMOID, bias, None, None, 1.0, 1.0 / 16.0, state, step, H, N, P)
    for b, (s, n) in enumerate(zip(start, lens)):
        want, S = _scan(view(q, s, n, N), view(k, s, n, N), view(v, s, n, P), view(logs, s, n, N))
        # sums in fp32 of float32 operands: some hundred roundings of 2^-24 at most, most of them far smaller than the sum
        assert (got[s:s + n].double() - want.reshape(n, -1)).norm() <= 2e-6 * want.norm(), (b, n)
        assert (state[b].double() - S.reshape(-1)).norm() <= 2e-6 * S.norm()
    state.zero_()
    qn, kn = (torch.nn.functional.normalize(x.view(T, H, N), dim=2).view(T, H * N) for x in (q, k))
    beta, dec = torch.rand(T, H, device=DEV), -torch.rand(T, H * N, device=DEV) * 0.2
    got = ops.delta_scan(qn, kn, (qn * kn).view(T, H, N).sum(2).contiguous(), dec, beta, v, state, step, H, N, P)
    for b, (s, n) in enumerate(zip(start, lens)):
        want, S = _scan(view(qn, s, n, N), view(kn, s, n, N), view(v, s, n, P), view(dec, s, n, N), beta[s:s + n].double())
        assert (got[s:s + n].double() - want.reshape(n, -1)).norm() <= 4e-6 * want.norm(), (b, n)
        assert (state[b].double() - S.reshape(-1)).norm() <= 4e-6 * S.norm()
    ops.check_status(DEV)


def test_chunk_products_keep_what_is_not_finite_where_it_belongs():
    """An infinity and a NaN in a token's values reach its column's later results and no earlier one."""
    from picolm_b200 import ops
    torch.manual_seed(3)
    H, N, P, T = 2, 128, 128, 200
    step = _step([T])
    q, k, v, raw = (torch.randn(T, H * c, device=DEV) * 0.1 for c in (N, N, P, N))
    bias = torch.zeros(H * N, device=DEV)
    run = lambda x: ops.linear_scan(q, k, x, raw, ops.DECAY_SIGMOID, bias, None, None, 1.0, 1.0 / 16.0, torch.zeros(1, H * N * P, device=DEV), step, H, N, P)
    clean = run(v)
    bad = v.clone()
    bad[100, 5], bad[150, 200] = math.inf, math.nan
    got = run(bad)
    assert torch.equal(got[:100], clean[:100]) and torch.isfinite(got[:150, 128:]).all()
    assert not torch.isfinite(got[100:, 5]).any() and torch.isnan(got[150:, 200]).all()
    keep = [c for c in range(H * P) if c not in (5, 200)]
    assert torch.equal(got[:, keep], clean[:, keep])


@pytest.mark.parametrize("N", [40, 64, 128])
def test_units_of_one_cta_keep_their_own_marks(N):
    """More than three units a CTA, and values that are not finite in units that one CTA takes one after the other, in a state and
    in the values: each reaches its own column's later results, whichever unit comes before or behind it."""
    from picolm_b200 import ops
    torch.manual_seed(N)
    H, P, lens = 8, 128, [64 * 37, 64 * 37 - 5]                  # 592 units: 148 CTAs take four each
    T, step = sum(lens), _step(lens)
    q, k, v, raw = (torch.randn(T, H * c, device=DEV) * 0.1 for c in (N, N, P, N))
    bias, state = torch.zeros(H * N, device=DEV), torch.randn(2, H * N * P, device=DEV)
    run = lambda x, s: ops.linear_scan(q, k, x, raw, ops.DECAY_SIGMOID, bias, None, None, 1.0, 1.0 / 16.0, s, step, H, N, P)
    clean = run(v, state.clone())
    bad, old = v.clone(), state.clone()
    # a column of every head: from the state on, from a token of every third chunk on (the column is of no number from the first
    # on, so each chunk has one of its own)
    marks = [(t, (c % H) * P + 3 * c + 1) for c, t in enumerate(range(7, T, 64 * 3)) if t < T]
    for i, (t, c) in enumerate(marks):
        bad[t, c] = (math.inf, -math.inf, math.nan)[i % 3]
    old.view(2, H, N, P)[1, 2, 5, 127] = math.nan
    ends = lambda t: lens[0] if t < lens[0] else T
    for _ in range(3):
        got = run(bad, old.clone())
        rest = torch.ones(T, H * P, dtype=torch.bool, device=DEV)
        for t, c in marks + [(lens[0], 2 * P + 127)]:
            assert not torch.isfinite(got[t:ends(t), c]).any(), (t, c)
            rest[t:ends(t), c] = False
        assert torch.equal(got[rest], clean[rest])
    ops.check_status(DEV)


@pytest.mark.parametrize("small,large", [(1e-36, 1e30), (1e-41, 1e34), (1e-12, 1e33)])
def test_chunk_products_of_the_smallest_and_largest_values(small, large):
    """Values whose last bits bfloat16 has no place for against large queries."""
    from picolm_b200 import ops
    torch.manual_seed(4)
    H, N, P, T = 3, 64, 128, 190
    step = _step([T])
    q, k, v, raw = (torch.randn(T, H * c, device=DEV) for c in (N, N, P, N))
    q, k, v, bias = q * large, k * N ** -0.5, v * small, torch.zeros(H * N, device=DEV)
    state = torch.zeros(1, H * N * P, device=DEV)
    got = ops.linear_scan(q, k, v, raw, ops.DECAY_SIGMOID, bias, None, None, 1.0, 1.0 / 16.0, state, step, H, N, P)
    view = lambda x, c: x.double().view(T, H, c)
    want, S = _scan(view(q, N), view(k, N), view(v, P), view(torch.nn.functional.logsigmoid(raw.double()) / 16.0, N))
    # (as for ordinary numbers; a value of the state may be subnormal)
    assert (state.double() - S.reshape(-1)).abs().max() <= 2e-6 * S.abs().max() + 4 * 2.0 ** -149
    if small > 1e-38:
        assert (got.double() - want.reshape(T, -1)).norm() <= 2e-6 * want.norm()


def _retention(N, P, lens, H=3, positions=0, odd=None, rotary_dim=None):
    """ops.decay_scan over rotated rows, its inputs, and the same in float64 with everything that the kernels are handed."""
    from picolm_b200 import ops
    from picolm_b200.ops import recurrent
    torch.manual_seed(N + P + sum(lens))
    T = sum(lens)
    start = [sum(lens[:b]) for b in range(len(lens))]
    step = _step(lens)
    step.tok_pos = _i32([positions + p for n in lens for p in range(n)])
    step.max_position = positions + max(lens) - 1
    rows = torch.randn(T, 2 * H * N + H * P).to(torch.bfloat16).to(DEV)
    q, k, v = rows[:, :H * N], rows[:, H * N:2 * H * N], rows[:, 2 * H * N:]
    if odd:
        for t, c, x in odd:
            v[t, c] = x
    decay = torch.tensor([1.0 - 2.0 ** (-3.0 - 2 * h) for h in range(H)], dtype=torch.float64)
    half = (N if rotary_dim is None else rotary_dim) // 2
    angle = torch.arange(positions + max(lens), dtype=torch.float64)[:, None] * 10000.0 ** (-torch.arange(half, dtype=torch.float64) / half)
    rotation = types.SimpleNamespace(cos=angle.cos().float().to(DEV), sin=angle.sin().float().to(DEV), rotary_dim=2 * half, pairing="half") if half else None
    state = torch.randn(len(lens), H * N * P, device=DEV)
    before = state.clone()
    with mock.patch.object(recurrent, "decay_in_128", lambda *a: True):                # (whatever the rule would choose)
        y = ops.decay_scan(q, k, v, decay.float().to(DEV), ops.decay_powers(decay).to(DEV), state, step, H, N, P, rotation=rotation, k_scale=N ** -0.5)
    want, states = [], []
    for b, n in enumerate(lens):
        c, s = (f[positions:positions + n].to(DEV).float().double()[:, None] for f in (angle.cos(), angle.sin()))
        turn = lambda x: (lambda u, w, r: torch.cat([u * c - w * s, w * c + u * s, r], -1))(*x[start[b]:start[b] + n].double().view(n, H, N).split([half, half, N - 2 * half], -1))
        qq, kk, vv = turn(q), turn(k) * N ** -0.5, v[start[b]:start[b] + n].double().view(n, H, P)
        S, out = before[b].double().view(H, N, P), []
        for i in range(n):
            S = S * decay.to(DEV)[:, None, None] + kk[i][:, :, None] * vv[i][:, None]
            out.append(torch.bmm(qq[i][:, None], S)[:, 0].reshape(-1))
        want += [torch.stack(out)] if out else []
        states.append(S.reshape(-1))
    ops.check_status(DEV)
    return y, torch.cat(want), state, torch.stack(states)


@pytest.mark.parametrize("N,P", [(64, 128), (128, 128), (128, 256), (64, 384)])
@pytest.mark.parametrize("lens", [[129], [128, 150, 200], [513, 70, 3], [400, 257]])
def test_retention_128_tokens_at_a_time(N, P, lens):
    """Chunks that end early, sequences in the midst of others, several value tiles, a state that is carried on, positions that do
    not begin at 0."""
    y, want, state, states = _retention(N, P, lens, positions=17)
    # operands in two bf16 terms: 2^-17 of each at most, two or three a product
    assert (y.double() - want).norm() <= 3 * 2.0 ** -17 * want.norm() and (state.double() - states).norm() <= 3 * 2.0 ** -17 * states.norm()
    for t in range(0, want.shape[0], 37):
        assert (y[t].double() - want[t]).norm() <= 6 * 2.0 ** -17 * want[t].norm()


@pytest.mark.parametrize("N,rotary_dim", [(64, 0), (64, 16), (128, 32), (128, 112)])
def test_retention_with_part_of_a_head_rotated(N, rotary_dim):
    y, want, state, states = _retention(N, 128, [200, 131], positions=5, rotary_dim=rotary_dim)
    assert (y.double() - want).norm() <= 3 * 2.0 ** -17 * want.norm() and (state.double() - states).norm() <= 3 * 2.0 ** -17 * states.norm()


@pytest.mark.parametrize("lens", [[0, 140, 0, 0, 1, 300, 0], [(7 * i) % 40 for i in range(70)], [300] + [i % 3 for i in range(1100)] + [129]])
def test_retention_chunks_find_their_sequences(lens):
    """Sequences of no tokens, more sequences than a warp has lanes, more than a warp's square."""
    y, want, state, states = _retention(64, 128, lens, H=1)
    assert (y.double() - want).norm() <= 3 * 2.0 ** -17 * want.norm() and (state.double() - states).norm() <= 3 * 2.0 ** -17 * states.norm()


def test_many_retention_chunks_share_their_weights_between_value_tiles():
    y, want, state, states = _retention(128, 256, [1200, 1100], H=9)
    assert (y.double() - want).norm() <= 3 * 2.0 ** -17 * want.norm() and (state.double() - states).norm() <= 3 * 2.0 ** -17 * states.norm()


@pytest.mark.parametrize("H", [2, 40])
def test_retention_keeps_what_is_not_finite_where_it_belongs(H):
    """(2 heads: a CTA a value tile; 40: a CTA all of them)"""
    N, P, lens = 64, 256, [300, 200]
    clean, _, _, _ = _retention(N, P, lens, H=H)
    odd = [(40, 5, math.inf), (170, 140, math.nan), (299, 3, -math.inf), (300, 200, math.inf)]
    y, _, state, _ = _retention(N, P, lens, H=H, odd=odd)
    for t, c, _ in odd:
        end = 300 if t < 300 else 500
        assert not torch.isfinite(y[t:end, c]).any()
        assert torch.equal(y[:t, c], clean[:t, c]) and torch.equal(y[end:, c], clean[end:, c])
        assert not torch.isfinite(state.view(2, H, N, P)[t // 300, c // P, :, c % P]).all()
    rest = [c for c in range(H * P) if c not in (5, 140, 3, 200)]
    assert torch.equal(y[:, rest], clean[:, rest])


@pytest.mark.parametrize("types_", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float32, torch.float32)])
@pytest.mark.parametrize("T,E,K", [(64, 32, 132), (2049, 1, 2052), (683, 3, 2052), (1024, 24, 260), (1025, 24, 260), (2731, 48, 388), (10923, 12, 128), (10923, 24, 132), (10925, 25, 4)])
def test_router_logits_have_the_same_bits_in_every_tile(T, E, K, types_):
    """Pairs on both sides of each line between tiles, tokens and rows that fill no tile, K with and without whole groups of steps."""
    from picolm_b200 import ops
    torch.manual_seed(T + E + K)
    h, w = torch.randn(T, K).to(types_[0]).to(DEV), torch.randn(E, K).to(types_[1]).to(DEV)
    odd = torch.empty(T * K + 1, dtype=types_[0], device=DEV)[1:].view(T, K).copy_(h)      # rows on no boundary: the general form
    got = ops.router_logits(h, w)
    assert torch.equal(got, ops.router_logits(odd, w))
    ref = h.double() @ w.double().t()
    # a lane's K / 32 terms one after the other, then five additions: each rounds a sum of at most `size`
    size = h.double().abs() @ w.double().abs().t()
    assert ((got.double() - ref).abs() <= (K / 32 + 9) * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("scores", ["sigmoid", "softmax", "logits"])
@pytest.mark.parametrize("E,top", [(5, 5), (33, 1), (64, 32), (70, 33), (130, 70)])
def test_choices_among_equal_scores(E, top, scores):
    """Many ties and scores of both zeros' signs and of minus infinity: the lowest expert first, weights in the choices' order."""
    from picolm_b200 import ops
    T = 9
    torch.manual_seed(E + top)
    z = torch.randint(-6, 7, (T, E)).float() / 4
    if scores == "logits":
        z[z == 0] = -0.0
        z[1, ::2] = 0.0
        z[2, 1:E - top + 1 if top < E else 1] = -math.inf
    ids, weights, _ = ops.route_topk(z.to(DEV), E, top, scores=scores)
    order = torch.sort(z.double(), dim=1, descending=True, stable=True).indices[:, :top]
    assert torch.equal(ids.cpu().long(), order)
    chosen = z.double().gather(1, order)
    s = torch.sigmoid(chosen) if scores == "sigmoid" else torch.softmax(z.double(), 1).gather(1, order) if scores == "softmax" else torch.softmax(chosen, 1)
    want = s / s.sum(1, keepdim=True)
    # an exponential within 2 units, a sum of E or `top` terms, three more roundings
    assert ((weights.cpu().double() - want).abs() <= (E + top + 16) * 2.0 ** -24 * want).all()
