"""The experts' products that stream their weights through one CTA an SM (csrc/routed_stream.cu): the bits of the kernel
for other sizes, over unused tiles, several tiles an expert, odd numbers of column pieces and K that ends inside a stage."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("mode", ["gate_up", "gate_up_interleaved", "up", "down"])
@pytest.mark.parametrize("T,E,top,N,K", [(1, 4, 2, 64, 64), (3, 32, 2, 96, 192), (8, 16, 4, 1344, 320), (48, 6, 3, 160, 128), (70, 3, 2, 2048, 1088)])
def test_streamed_products_give_the_same_bits(mode, T, E, top, N, K, monkeypatch):
    from picolm_b200 import ops
    from picolm_b200.ops import routed
    if mode == "gate_up_interleaved" and N % 64:
        pytest.skip("gate and up rows come in turns of 64")
    torch.manual_seed(T * E + N)
    # choices that leave experts out and give others several tiles
    ids = torch.multinomial(torch.rand(T, E, device=DEV) ** 3 + 1e-6, top).to(torch.int32)
    pairs = ops.moe_align(ids, E, 16)
    rows = pairs.rows if mode == "down" else T
    a = torch.randn(rows, K, device=DEV).to(torch.bfloat16)
    w = (torch.randn(E, (2 if "gate" in mode else 1) * N, K, device=DEV) * K ** -0.5).to(torch.bfloat16)

    def run():
        if mode == "down":
            return ops.moe_down(a, w, pairs)
        return ops.moe_up(a, w, pairs) if mode == "up" else ops.moe_gate_up(a, w, pairs, interleaved="inter" in mode)
    streamed = run()
    ops.check_status(streamed.device)
    monkeypatch.setattr(routed, "STREAM_TILES", 0)
    plain = run()
    used = pairs.sorted >= 0
    assert used.sum().item() == T * top
    assert torch.equal(streamed[used], plain[used]) and torch.isfinite(plain[used].float()).all()
    # row by row against float64: fp32 sums of K products, at most K roundings, then the result's own
    entry = pairs.sorted[used].long()
    x = (a[used] if mode == "down" else a[entry // top]).double()
    e = pairs.tile_expert.long().repeat_interleave(16)[used]
    z = torch.einsum("rk,rnk->rn", x, w[e].double())
    if mode == "down":
        assert torch.allclose(streamed[used].double(), z, atol=1e-4, rtol=1e-5)
    elif mode == "up":
        assert torch.allclose(streamed[used].double(), torch.relu(z) ** 2, atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("mode", ["gate_up", "up", "down"])
@pytest.mark.parametrize("T,E,busy", [(1300, 40, 1), (700, 24, 3), (16 * 380, 100, 1)])
def test_experts_with_many_tiles(mode, T, E, busy, monkeypatch):
    """All tokens but a few at one expert or three: runs of hundreds of tiles between experts of one tile and of none."""
    from picolm_b200 import ops
    from picolm_b200.ops import routed
    torch.manual_seed(T)
    N, K = 96, 128
    ids = torch.randint(0, busy, (T, 1), device=DEV, dtype=torch.int32) * 7 + 2
    ids[::97, 0] = torch.randint(0, E, (len(ids[::97]),), device=DEV, dtype=torch.int32)
    pairs = ops.moe_align(ids, E, 16)
    assert pairs.max_tiles <= routed.STREAM_TILES and T <= routed.STREAM_PAIRS * E
    a = torch.randn(pairs.rows if mode == "down" else T, K, device=DEV).to(torch.bfloat16)
    w = (torch.randn(E, (2 if mode == "gate_up" else 1) * N, K, device=DEV) * K ** -0.5).to(torch.bfloat16)
    product = {"gate_up": ops.moe_gate_up, "up": ops.moe_up, "down": ops.moe_down}[mode]
    streamed = product(a, w, pairs)
    ops.check_status(DEV)
    monkeypatch.setattr(routed, "STREAM_TILES", 0)
    used = pairs.sorted >= 0
    assert torch.equal(streamed[used], product(a, w, pairs)[used])


@pytest.mark.parametrize("T", [1, 8])
def test_more_sms_than_pieces(T):
    """Fewer pieces of columns than SMs: every CTA has one or none."""
    from picolm_b200 import ops
    torch.manual_seed(T)
    ids = torch.zeros((T, 1), dtype=torch.int32, device=DEV)
    pairs = ops.moe_align(ids, 2, 16)
    h, w = torch.randn(T, 128, device=DEV).to(torch.bfloat16), torch.randn(2, 64, 128, device=DEV).to(torch.bfloat16) * 0.1
    got = ops.moe_up(h, w, pairs)[pairs.where.long()]
    want = torch.relu(h.double() @ w[0].double().T) ** 2
    assert torch.allclose(got.double(), want, atol=2e-2, rtol=1e-2)
