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
