"""The float32 product on the tensor cores: every form against float64 and against one another, bit for bit, and what is not
finite."""
import math

import pytest
import torch

DEV = "cuda:0"
ROWS, CLUSTERS = (16, 32, 64, 96), (1, 2, 4, 8)


def _forms():
    return [r + 1000 * c for r in ROWS for c in CLUSTERS if r < 96 or c == 1]


def test_every_form_is_chosen_somewhere():
    from picolm_b200.csrc.build import load_library
    form = load_library("gemm_f32_tc").plm_gemm_f32_tc_form
    met = {form(M, N, K) for M in (1, 8, 24, 40, 64, 100, 200, 462, 1300) for N in (64, 130, 512, 1000, 2048, 3072, 16384, 32000)
           for K in (64, 1024, 2048, 4096, 8192, 14336)}
    assert met <= set(_forms()) and {f % 1000 for f in met} == set(ROWS) and {f // 1000 for f in met} == set(CLUSTERS), sorted(met)


# edges of the tiles by rows and columns; K of less than a stage, of a stage, of parts of stages, of one segment, just over one,
# of several segments and more segments than a cluster has CTAs
@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (5, 64, 20), (16, 128, 32), (17, 129, 100), (33, 130, 1024), (97, 300, 1028), (200, 520, 3000),
                                   (63, 257, 8192), (9, 140, 9300)])
def test_float32_tc_forms(M, N, K):
    from picolm_b200 import ops
    torch.manual_seed(M + 3 * N + 7 * K)
    a, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    out = ops.gemm_f32_tc(a, w)
    for form in _forms():
        for _ in range(3):                                   # (a wait that passes too early shows only now and then)
            assert torch.equal(ops.gemm_f32_tc(a, w, form), out), form
    assert torch.equal(ops.gemm_f32_tc(a[M // 2:M // 2 + 1], w), out[M // 2:M // 2 + 1])
    wide = torch.randn(M, K + 8, device=DEV)                 # rows of a wider matrix
    wide[:, 4:4 + K] = a
    assert torch.equal(ops.gemm_f32_tc(wide[:, 4:4 + K], w), out)
    ref, mag = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    # a piece of 32 terms: 12 truncations (a bit of 2^-23 each) of sums of at most the terms' magnitudes, two of them of whole
    # ones, the others 2^-8 and less; left-out products below 2^-25; the roundings of three pieces' sum; one to the result
    assert ((out.double() - ref).abs() <= (2 * 2.0 ** -23 + 2.0 ** -25 + 4 * 2.0 ** -24 + 2.0 ** -26) * mag).all()
    old = ops.gemm_simt(a, w, torch.float32)
    if M * N >= 10000:                                       # the error is no larger than the CUDA cores' (1.31e-7 / 2 against 1.26)
        assert (out.double() - ref).norm() <= 1.02 * (old.double() - ref).norm()
    assert int(ops.status_word(DEV).item()) == 0


# what rows hold: the products of a gated feed-forward, whose sums must be as exact as on the CUDA cores (the norms of 61,440 errors
# lie within 2 %), and terms of one sign, which come out low
@pytest.mark.gpu
@pytest.mark.parametrize("what", ["gated", "one sign", "one sign, several decades"])
@pytest.mark.parametrize("K", [128, 2048, 8192])
def test_float32_tc_error_by_what_rows_hold(what, K):
    from picolm_b200 import ops
    torch.manual_seed(K)
    x, y, w = torch.randn(96, K, device=DEV), torch.randn(96, K, device=DEV), torch.randn(640, K, device=DEV)
    a = torch.nn.functional.silu(x) * y if what == "gated" else x.abs()
    if what != "gated":
        w = w.abs()
    if what == "one sign, several decades":
        a, w = (2 * a).exp(), (2 * w).exp()
    got, ref = ops.gemm_f32_tc(a, w), a.double() @ w.double().T
    if what == "gated":
        old = ops.gemm_simt(a, w, torch.float32)
        assert (got.double() - ref).norm() <= 1.02 * (old.double() - ref).norm()
        return
    # a whole-sized MMA (two a piece, one of them of half the sum) truncates its result (2^-23) and cuts its 17 addends off two
    # bits below that, all of the largest one's size at most; then the bounds of sums of both signs
    cut = 17 * 2.0 ** -25 if what == "one sign, several decades" else 17 / 4 * 2.0 ** -25     # (the largest of 16: a quarter of them at most)
    assert (got.double() - ref).norm() <= (1.5 * (2.0 ** -23 + cut) + 4 * 2.0 ** -24) * ref.norm()


@pytest.mark.gpu
@pytest.mark.parametrize("form", [0, 1016, 4016, 8032, 2064, 1096])
def test_float32_tc_values_that_are_not_finite(form):
    """Infinities, values next to the largest one, NaN and overflowing sums: what fused multiply-adds make of them, and rows
    and columns without them as they are."""
    from picolm_b200 import ops
    torch.manual_seed(5)
    M, N, K = 70, 140, 2100
    a, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    clean = ops.gemm_f32_tc(a, w, form)
    a[3, 5], a[4, 2000], a[5, 7], a[6, :2] = math.inf, -math.inf, math.nan, torch.tensor([math.inf, -math.inf], device=DEV)
    w[:, 5] = w[:, 5].abs() + 0.1
    clean5 = ops.gemm_f32_tc(torch.where(torch.isfinite(a), a, torch.zeros_like(a)), w, form)
    a[8, 0], w[9, 0] = 3.4e38, 0.5                           # rounds up to infinity in bfloat16
    a[10, :2], w[11, :2] = 3e38, 1.0
    got, want = ops.gemm_f32_tc(a, w, form), ops.gemm_simt(a, w, torch.float32)
    assert (torch.isinf(got[3]) & (got[3] > 0)).all() and torch.isnan(got[5]).all()
    # (of row 10 only the column that must overflow: with terms of both signs it depends on the order whether a sum does)
    assert got[10, 11] == math.inf == want[10, 11]
    got[10], want[10] = 0.0, 0.0
    finite = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    assert torch.equal(got[~finite & ~torch.isnan(want)], want[~finite & ~torch.isnan(want)])
    mag = torch.where(torch.isfinite(a), a, torch.zeros_like(a)).double().abs() @ w.double().abs().T
    assert ((got.double() - want.double()).abs()[finite] <= 1e-6 * mag[finite]).all()
    keep = [m for m in range(M) if m not in (3, 4, 5, 6, 8, 10)]
    cols = [n for n in range(N) if n not in (9, 11)]
    assert torch.equal(got[keep][:, cols], clean5[keep][:, cols]) and clean.shape == got.shape


@pytest.mark.gpu
@pytest.mark.parametrize("small,large", [(1e-36, 1e30), (1e-39, 1e30), (2e-44, 1e36), (1e-33, 1e-6), (1e-20, 1e-21), (1e-3, 1e26), (1e-5, 1e33)])
def test_float32_tc_of_the_smallest_and_largest_operands(small, large):
    """Operands next to and below the smallest normal number, whose last bits bfloat16 has no place for, and large ones: as exact
    as any others.  Rows of ordinary numbers beside them stay as they are."""
    from picolm_b200 import ops
    torch.manual_seed(8)
    M, N, K = 40, 140, 300
    a, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    plain = ops.gemm_f32_tc(a, w)
    a[::2] *= small
    w[::2] *= large
    got, ref, mag = ops.gemm_f32_tc(a, w), a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    # (16 fused multiply-adds one after the other where the sums are taken again; a result may be subnormal)
    assert ((got.double() - ref).abs() <= 16 * 2.0 ** -24 * mag + 2.0 ** -149).all()
    assert (got.double() - ref)[::2, ::2].norm() <= 2 * 2.0 ** -24 * ref[::2, ::2].norm() + 2.0 ** -149 * (M * N) ** 0.5
    assert torch.equal(got[1::2, 1::2], plain[1::2, 1::2])
    assert int(ops.status_word(DEV).item()) == 0


@pytest.mark.gpu
def test_linear_of_float32_rows_off_their_boundaries_takes_the_cuda_cores():
    from picolm_b200 import ops
    torch.manual_seed(6)
    wide, w = torch.randn(20, 68, device=DEV), torch.randn(2100, 64, device=DEV)
    odd = wide[:, 1:65]
    assert torch.equal(ops.linear(odd, w, torch.float32), ops.gemm_simt(odd, w, torch.float32))
    assert torch.equal(ops.linear(odd.contiguous(), w, torch.float32), ops.gemm_f32_tc(odd.contiguous(), w))
    with pytest.raises(ops.KernelError):
        ops.gemm_f32_tc(odd, w)


@pytest.mark.gpu
@pytest.mark.parametrize("N,K,tensor_cores", [(64, 64, False), (2048, 64, False), (2052, 64, True), (128, 1024, False), (64, 1028, True)])
def test_linear_of_small_float32_weights_takes_the_cuda_cores(N, K, tensor_cores):
    """By the weights' sizes alone, so that a row's bits are the same beside any number of others."""
    from picolm_b200 import ops
    torch.manual_seed(7)
    a, w = torch.randn(600, K, device=DEV), torch.randn(N, K, device=DEV)
    out = ops.linear(a, w, torch.float32)
    assert torch.equal(out, ops.gemm_f32_tc(a, w) if tensor_cores else ops.gemm_simt(a, w, torch.float32))
    for rows in (1, 7, 33, 300):
        assert torch.equal(ops.linear(a[:rows], w, torch.float32), out[:rows])
