"""Kernels of the recurrent layers that are chosen by size or alignment, against the forms that take anything and against
plain computations."""
import math
import types

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
@pytest.mark.parametrize("M,N", [(1, 4), (17, 512), (50, 516), (33, 1028)])
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
    got = ops.causal_conv(u, w, None, state, step)
    want = torch.nn.functional.silu(raw)
    # sums of four terms in fp32, the activation within 2^-20, one rounding to bfloat16
    mag = torch.cat([sum((x[j:j + n] * w[j].double()).abs() for j in range(4)) for x, n in zip(back, lens)])
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -19 * (mag + 1)).all()
    assert torch.equal(state.double().view(len(lens), 3, C), torch.stack([x[-3:] for x in back]))


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
    assert ops.delta_scan_in_chunks(ops.step_shape(step), H, N, P) and sum(lens) // 64 * 6 + 6 >= 1
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
