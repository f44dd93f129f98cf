"""The experts' products of prompts on tcgen05 with the weights on the MMA's rows (csrc/routed_tc.cu) and the router's
logits by tiles: at the edges of their tiles and chunks."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("bm", [16, 128])
@pytest.mark.parametrize("mode", ["gate_up", "up", "down"])
# few rows an expert, experts without rows, one with more than 256 rows (two chunks), K that ends inside a stage, weight rows
# that end inside a tile of 256 and of 128
@pytest.mark.parametrize("T,E,top,N,K", [(5, 9, 2, 128, 64), (300, 4, 2, 384, 96), (700, 3, 1, 640, 328), (130, 40, 4, 256, 200)])
def test_experts_products_against_float64(bm, mode, T, E, top, N, K):
    from picolm_b200 import ops
    torch.manual_seed(T + N + bm)
    ids = torch.multinomial(torch.rand(T, E, device=DEV) ** 4 + 1e-6, top).to(torch.int32)
    ids[: T // 2, 0] = torch.where((ids[: T // 2, 1:] == E - 1).any(1), ids[: T // 2, 0], E - 1)        # one busy expert
    pairs = ops.moe_align(ids, E, bm)
    used = pairs.sorted >= 0
    h = torch.randn(T, K, device=DEV).to(torch.bfloat16)
    x = ops.moe_gather(h, pairs)
    e = pairs.tile_expert.long().repeat_interleave(bm)[used]
    if mode == "gate_up":
        gate, up = [(torch.randn(E, N, K, device=DEV) * K ** -0.5).to(torch.bfloat16) for _ in range(2)]
        got = ops.moe_gate_up_tc(x, torch.stack([ops.interleave_gate_up(a, b) for a, b in zip(gate, up)]), pairs)
        g, u = [torch.einsum("rk,rnk->rn", x[used].double(), w[e].double()) for w in (gate, up)]
        want = torch.nn.functional.silu(g) * u
    else:
        w = (torch.randn(E, N, K, device=DEV) * K ** -0.5).to(torch.bfloat16)
        got = ops.moe_up_tc(x, w, pairs) if mode == "up" else ops.moe_down_tc(x, w, pairs)
        z = torch.einsum("rk,rnk->rn", x[used].double(), w[e].double())
        want = torch.relu(z) ** 2 if mode == "up" else z
    ops.check_status(DEV)
    if mode == "down":                       # fp32 sums of K products of size K^(-1/2)
        assert torch.allclose(got[used].double(), want, atol=1e-5, rtol=1e-5)
    else:                                    # branches and results rounded to bf16: three roundings of 2^-9 at most
        assert torch.allclose(got[used].double(), want, atol=1e-2, rtol=1.2e-2)


@pytest.mark.parametrize("epilogue", [0, 1, 2])
# K in whole and in ragged pairs of 64 (3.5 and 8 of them: the ring of three or four stages comes round), and one that only the
# form with single stages takes
@pytest.mark.parametrize("K", [448, 1024, 456])
def test_every_cta_takes_several_units(epilogue, K):
    """Both forms on the same rows, from the C entry, which is told by the number of pairs which to take: over 450 units, so that every
    CTA uses both accumulators again, and an expert with 300 rows among some with 30: two or three chunks of its tokens."""
    import ctypes
    from picolm_b200 import ops
    from picolm_b200.csrc.build import load_library
    from picolm_b200.ops import _lib
    product = load_library("routed_tc").plm_moe_tc
    product.argtypes = _lib._SIGNATURES["plm_moe_tc"]
    E, F = 12, 5120 + (0 if epilogue == 1 else 40)           # (weight rows that end inside a tile of 128)
    torch.manual_seed(K + epilogue)
    rows_of = [300, 0, 1, 16, 17, 64, 65, 129, 33, 30, 30, 30]
    ids = torch.tensor([e for e, n in enumerate(rows_of) for _ in range(n)], dtype=torch.int32)[torch.randperm(sum(rows_of))]
    pairs = ops.moe_align(ids[:, None].contiguous().to(DEV), E, 16)
    x = ops.moe_gather(torch.randn(len(ids), K, device=DEV).to(torch.bfloat16), pairs)
    w = (torch.randn(E, F, K, device=DEV) * K ** -0.5).to(torch.bfloat16)
    used = (pairs.sorted >= 0).nonzero()[:, 0]
    of = pairs.tile_expert.long().repeat_interleave(16)[used]
    want = torch.empty(len(used), F // 2 if epilogue == 1 else F, dtype=torch.float64, device=DEV)
    for e in range(E):
        z = x[used[of == e]].double() @ w[e].double().T
        if epilogue == 1:
            z = z.view(len(z), F // 128, 2, 64)
            z = (torch.nn.functional.silu(z[:, :, 0]) * z[:, :, 1]).reshape(len(z), F // 2)
        want[of == e] = torch.relu(z) ** 2 if epilogue == 2 else z
    outs = []
    for n_pairs in (1, 1 << 20):                             # 128 tokens and pairs of stages (K a multiple of 64), 256 and single ones
        out = torch.full((pairs.rows, want.shape[1]), float("nan"), dtype=torch.bfloat16 if epilogue else torch.float32, device=DEV)
        assert product(x.data_ptr(), w.data_ptr(), out.data_ptr(), 1 if epilogue else 0, epilogue, n_pairs, pairs.tile_expert.data_ptr(),
                       pairs.max_tiles, 16, E, F, K, out.shape[1], ops.status_word(DEV).data_ptr(),
                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        ops.check_status(DEV)
        outs.append(out[used])
        if epilogue == 0:                    # sums of up to K / 16 steps, each rounded at 2^-23 of a partial sum of some 4 at most
            assert (out[used].double() - want).abs().max() <= K / 16 * 4 * 2.0 ** -23
        else:                                # branches and results rounded to bf16: three roundings of 2^-9 at most
            assert torch.allclose(out[used].double(), want, atol=1e-2, rtol=1.2e-2)
    assert torch.allclose(outs[0].float(), outs[1].float(), atol=1e-4, rtol=2.0 ** -7)


@pytest.mark.parametrize("E", [31, 33, 64, 1000, 1024])
def test_many_experts(E):
    """The table of units by expert: a part of 32 experts, a whole one, many; experts without rows among them."""
    from picolm_b200 import ops
    torch.manual_seed(E)
    T, N, K = 3 * E, 200, 64
    ids = torch.randint(0, E, (T, 2), device=DEV, dtype=torch.int32)
    ids[: T // 8] = E - 1
    pairs = ops.moe_align(ids, E, 16)
    x = ops.moe_gather(torch.randn(T, K, device=DEV).to(torch.bfloat16), pairs)
    w = (torch.randn(E, N, K, device=DEV) * K ** -0.5).to(torch.bfloat16)
    got = ops.moe_down_tc(x, w, pairs)
    ops.check_status(DEV)
    used = pairs.sorted >= 0
    e = pairs.tile_expert.long().repeat_interleave(16)[used]
    want = torch.cat([torch.einsum("rk,rnk->rn", a.double(), w[b].double()) for a, b in zip(x[used].split(512), e.split(512))])
    assert torch.allclose(got[used].double(), want, atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("types", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("T,E,K", [(1, 5, 64), (8, 16, 4096), (3, 1, 132), (2050, 33, 260), (1185, 32, 2048)])
def test_router_tiles_give_the_bits_of_the_general_kernel(types, T, E, K):
    """Both tile sizes, ragged edges of tokens, experts and K; the general kernel takes rows off the four-value boundary."""
    from picolm_b200 import ops
    torch.manual_seed(T + E + K)
    flat = torch.randn(T * K + 1, device=DEV).to(types[0])
    odd = flat[1:].view(T, K)
    w = torch.randn(E, K, device=DEV).to(types[1])
    tiles, general = ops.router_logits(odd.clone(), w), ops.router_logits(odd, w)
    assert torch.equal(tiles, general)
    # 32 chains of K / 32 terms and five sums: at most K / 32 + 5 roundings of partial sums
    bound = (K / 32 + 6) * 2.0 ** -24 * (odd.double().abs() @ w.double().abs().T)
    assert ((tiles.double() - odd.double() @ w.double().T).abs() <= bound).all()
