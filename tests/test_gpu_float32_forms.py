"""The forms of the float32 product and of the CUDA-core attention that are chosen by size: every form gives the bits of
the general one, so a row does not depend on how many rows stand beside it."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, DT, _paged

SIZES = [(M, N, K) for M in (1, 8, 9, 32, 33, 65, 200, 530) for N, K in ((16, 4), (130, 20), (129, 100), (300, 64), (2064, 132))]
# ragged edges of each of the five tiles, by rows and by columns
SIZES += [(5, 2070, 132), (24, 4100, 132), (24, 8190, 132), (61, 4100, 36), (150, 8190, 36), (462, 2050, 132), (462, 16390, 132), (530, 32001, 36)]


def _form(M, N):
    from picolm_b200.csrc.build import load_library
    return load_library("gemm_simt").plm_gemm_simt_form(M, N)


def test_every_form_of_the_float32_product_is_tested():
    """(8 x 16, 32 x 16, 32 x 32, 64 x 64, 64 x 128: at least two sizes each, with rows and columns that end inside a tile)"""
    tiles = [(8, 16), (32, 16), (32, 32), (64, 64), (64, 128)]
    for form, (bm, bn) in enumerate(tiles):
        of_it = [(M, N) for M, N, _ in SIZES if _form(M, N) == form]
        assert len(of_it) >= 2 and any(M % bm and N % bn for M, N in of_it), (form, of_it)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", SIZES)
def test_float32_product_forms_agree_to_the_bit(M, N, K):
    """Few rows, many rows, ragged edges of every tile: against the general kernel (which takes rows that do not start on
    16-byte boundaries), against float64, and row by row."""
    from picolm_b200 import ops
    torch.manual_seed(M * 7 + N + K)
    wide = torch.randn(M, K + 4, device=DEV)
    w = torch.randn(N, K, device=DEV)
    odd = wide[:, 1:1 + K]                                   # the general kernel's: K a multiple of 4, rows off by 4 bytes
    out, general = ops.gemm_simt(odd.contiguous(), w, torch.float32), ops.gemm_simt(odd, w, torch.float32)
    assert torch.equal(out, general)
    assert torch.equal(out[M // 2:M // 2 + 1], ops.gemm_simt(odd[M // 2:M // 2 + 1].contiguous(), w, torch.float32))
    ref = odd.double() @ w.double().T
    # a piece of 16 terms: at most 16 roundings of partial sums, then one to the result
    bound = 17 * 2.0 ** -24 * (odd.double().abs() @ w.double().abs().T)
    assert ((out.double() - ref).abs() <= bound).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,G,hd", [(5, 5, 16), (6, 2, 48), (16, 4, 64), (8, 1, 128), (4, 2, 80), (3, 1, 256), (80, 2, 32)])
@pytest.mark.parametrize("extra", [False, True])
def test_attention_tile_form_agrees_to_the_bit(dtype, H, G, hd, extra):
    """Prompts of unequal lengths in one step, some behind earlier positions, tiles that hold several sequences: the tile
    form against the row form.  The last value of each sequence is infinite: rows before it must not see it."""
    from picolm_b200 import ops
    torch.manual_seed(H * 100 + hd)
    lens, new = [100, 1, 65, 33, 7, 64], [90, 1, 65, 2, 7, 31]
    ks = [torch.randn(n, G, hd) for n in lens]
    vs = [torch.randn(n, G, hd) for n in lens]
    for v in vs:
        v[-1] = math.inf
    kc, vc, table = _paged(ks, vs, lens, 16, DT[dtype], 5)
    q = torch.randn(sum(new), H, hd).to(DT[dtype]).to(DEV)
    pos = torch.tensor([p for n, m in zip(lens, new) for p in range(n - m, n)], dtype=torch.int32, device=DEV)
    seq = torch.tensor([b for b, m in enumerate(new) for _ in range(m)], dtype=torch.int32, device=DEV)
    start = torch.tensor([sum(new[:b]) for b in range(len(new) + 1)], dtype=torch.int32, device=DEV)
    more = dict(sink=torch.randn(H, device=DEV), slopes=torch.rand(H, device=DEV) * 0.1) if extra else {}
    rows, tiles = (ops.attention_rows(q, kc.to(DEV), vc.to(DEV), pos, seq, table.to(DEV), G, hd ** -0.5, longest=max(new), seq_start=st, **more)
                   for st in (None, start))
    assert torch.isfinite(rows).any()
    assert torch.equal(torch.nan_to_num(rows.float(), nan=7.0), torch.nan_to_num(tiles.float(), nan=7.0))


@pytest.mark.parametrize("longest,max_position,rows,tiles", [(7, 5000, 1 << 20, False), (8, 30, 8191, False), (8, 31, 256, True), (8, 8, 8192, True)])
def test_when_rows_share_keys(longest, max_position, rows, tiles):
    from picolm_b200.ops.attention import shares_keys
    assert shares_keys(longest, max_position, rows) == tiles


@pytest.mark.gpu
def test_single_tokens_beside_a_prompt_have_tiles_of_their_own():
    """More sequences than a block has threads, heads in pairs: every sequence's rows against the row form."""
    from picolm_b200 import ops
    torch.manual_seed(11)
    H, G, hd = 4, 2, 16
    new = [1] * 70 + [33] + [1] * 80 + [9, 0, 2]
    lens = [n + 40 + 3 * b for b, n in enumerate(new)]
    ks, vs = [torch.randn(n, G, hd) for n in lens], [torch.randn(n, G, hd) for n in lens]
    kc, vc, table = _paged(ks, vs, lens, sum((n + 63) // 64 for n in lens) + 8, torch.float32, 6)
    q = torch.randn(sum(new), H, hd, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    pos = i32([p for n, m in zip(lens, new) for p in range(n - m, n)])
    seq = i32([b for b, m in enumerate(new) for _ in range(m)])
    start = i32([sum(new[:b]) for b in range(len(new) + 1)])
    rows, tiles = (ops.attention_rows(q, kc.to(DEV), vc.to(DEV), pos, seq, table.to(DEV), G, hd ** -0.5, longest=33, seq_start=st) for st in (None, start))
    assert torch.equal(rows, tiles) and torch.isfinite(rows).all()
