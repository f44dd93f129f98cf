"""The kernels' safety nets, made to act: a bounded wait that runs out (the kernel returns, the status word
says where, the next kernel runs as if nothing had happened), and the checked build of the kernels that walk
page tables (a page number, position or row outside its bounds is recorded and replaced, not followed)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_a_wait_that_runs_out_is_reported_not_hung():
    """A test build of the decode-shaped product (short wait limit, a switch that makes the producer announce
    more bytes than it loads): with the switch on no stage of the ring ever fills, every wait of the kernel
    runs out, the kernel returns, and `check_status` raises; with the switch off again the same library gives
    the right product."""
    from picolm_b200 import ops
    from picolm_b200.csrc.build import load_library
    lib = load_library("gemm_tc_skinny@stall", ["-DPLM_WAIT_LIMIT=20000", "-DPLM_TEST_STALL"])
    vp, i, l = ctypes.c_void_p, ctypes.c_int, ctypes.c_long
    lib.plm_gemm_tc_skinny.argtypes = [vp, vp, vp, i, i, i, i, i, l, l, l, vp, vp]
    lib.plm_test_stall.argtypes = [i, vp]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    T, F, K = 8, 512, 1024
    torch.manual_seed(3)
    x = (torch.randn(T, K) / K ** 0.25).to(torch.bfloat16).to(DEV)
    w = (torch.randn(F, K) / K ** 0.25).to(torch.bfloat16).to(DEV)
    out = torch.zeros((T, F), dtype=torch.float32, device=DEV)
    status = ops.status_word(DEV)
    ops.check_status(DEV)                                        # clean before the test

    def product():
        return lib.plm_gemm_tc_skinny(x.data_ptr(), w.data_ptr(), out.data_ptr(), 0, 0, T, F, K, K, K, F,
                                      status.data_ptr(), stream)

    assert lib.plm_test_stall(1, stream) == 0
    assert product() == 0                                        # launched; it gives up on the device
    torch.cuda.synchronize()                                     # ... and returns
    assert int(status.item()) in (1, 2, 3)
    with pytest.raises(ops.KernelError, match="gave up waiting"):
        ops.check_status(DEV)
    ops.check_status(DEV)                                        # reading the status cleared it
    assert lib.plm_test_stall(0, stream) == 0
    assert product() == 0
    torch.cuda.synchronize()
    ops.check_status(DEV)
    ref = x.double().cpu() @ w.double().cpu().t()
    assert torch.allclose(out.double().cpu(), ref, atol=2e-3, rtol=1e-4)


@pytest.mark.parametrize("epilogue", [0, 1, 2])
@pytest.mark.parametrize("how", [1, 2])
def test_the_experts_product_gives_up_as_one(epilogue, how):
    """The same for the experts' product with the weights on the MMA's rows, whose gated epilogue has barriers inside sets of
    four warps: with no stage ever filling (1), and with a single warp that gives up on its CTA's second unit while the others
    go on (2), the kernel says so and returns; switched off again the same library gives the right product."""
    from picolm_b200 import ops
    from picolm_b200.csrc.build import load_library
    from picolm_b200.ops import _lib
    lib = load_library("routed_tc@give_up", ["-DPLM_WAIT_LIMIT=20000", "-DPLM_TEST_GIVE_UP"])
    lib.plm_moe_tc.argtypes = _lib._SIGNATURES["plm_moe_tc"]
    lib.plm_test_give_up.argtypes = [ctypes.c_int, ctypes.c_void_p]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    E, F, K, T = 8, 8192, 128, 100                              # 512 units or more: every CTA has at least three
    torch.manual_seed(5)
    ids = torch.randint(0, E, (T, 1), device=DEV, dtype=torch.int32)
    pairs = ops.moe_align(ids, E, 16)
    x = ops.moe_gather((torch.randn(T, K, device=DEV) / K ** 0.25).to(torch.bfloat16), pairs)
    w = (torch.randn(E, F, K, device=DEV) / K ** 0.25).to(torch.bfloat16)
    out = torch.zeros((pairs.rows, F // 2 if epilogue == 1 else F), dtype=torch.bfloat16 if epilogue else torch.float32, device=DEV)
    status = ops.status_word(DEV)
    ops.check_status(DEV)

    def product():
        return lib.plm_moe_tc(x.data_ptr(), w.data_ptr(), out.data_ptr(), 1 if epilogue else 0, epilogue, T, pairs.tile_expert.data_ptr(),
                              pairs.max_tiles, pairs.bm, E, F, K, out.shape[1], status.data_ptr(), stream)

    assert lib.plm_test_give_up(how, stream) == 0
    assert product() == 0
    torch.cuda.synchronize()
    assert int(status.item()) in ((51, 52, 53, 54) if how == 1 else (54,))
    with pytest.raises(ops.KernelError, match="gave up waiting"):
        ops.check_status(DEV)
    assert lib.plm_test_give_up(0, stream) == 0
    assert product() == 0
    torch.cuda.synchronize()
    ops.check_status(DEV)
    used = pairs.sorted >= 0
    z = torch.einsum("rk,rnk->rn", x[used].double(), w.double()[pairs.tile_expert.long().repeat_interleave(16)[used]])
    if epilogue == 1:
        z = z.view(len(z), F // 128, 2, 64)
        z = (torch.nn.functional.silu(z[:, :, 0]) * z[:, :, 1]).reshape(len(z), F // 2)
    elif epilogue == 2:
        z = torch.relu(z) ** 2
    assert torch.allclose(out[used].double(), z, atol=2e-3 if epilogue == 0 else 2e-2, rtol=1e-4 if epilogue == 0 else 1.2e-2)


@pytest.mark.parametrize("form", [16 + 8000, 32 + 2000, 64 + 1000, 96 + 1000])
@pytest.mark.parametrize("how", [1, 2])
def test_the_float32_product_gives_up(form, how):
    """The same for the float32 product on the tensor cores, alone and in clusters, whose ring has been round more than once
    when one of the warps that add sums up gives up (2)."""
    from picolm_b200 import ops
    from picolm_b200.csrc.build import load_library
    from picolm_b200.ops import _lib
    lib = load_library("gemm_f32_tc@give_up", ["-DPLM_WAIT_LIMIT=20000", "-DPLM_TEST_GIVE_UP"])
    lib.plm_gemm_f32_tc.argtypes = _lib._SIGNATURES["plm_gemm_f32_tc"]
    lib.plm_test_give_up.argtypes = [ctypes.c_int, ctypes.c_void_p]
    stream = torch.cuda.current_stream().cuda_stream
    M, N, K = 90, 300, 9000
    torch.manual_seed(6)
    a, w, out = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV), torch.zeros(M, N, device=DEV)
    status = ops.status_word(DEV)
    ops.check_status(DEV)

    def product():
        return lib.plm_gemm_f32_tc(a.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, K, K, N, form, status.data_ptr(), stream)

    assert lib.plm_test_give_up(how, stream) == 0
    assert product() == 0
    torch.cuda.synchronize()
    assert int(status.item()) in ((60, 61, 62, 63) if how == 1 else (63,))
    with pytest.raises(ops.KernelError, match="gave up waiting"):
        ops.check_status(DEV)
    assert lib.plm_test_give_up(0, stream) == 0
    assert product() == 0
    torch.cuda.synchronize()
    ops.check_status(DEV)
    assert torch.equal(out, ops.gemm_f32_tc(a, w))


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("how", [1, 2])
def test_the_chunk_products_give_up(N, how, monkeypatch):
    """The same for the chunk products of a recurrence, with several units a CTA."""
    import types
    from picolm_b200 import ops
    from picolm_b200.csrc.build import load_library
    from picolm_b200.ops import _lib
    H, P, T = 8, 128, 64 * 40
    torch.manual_seed(7)
    q, k, v, raw = (torch.randn(T, H * c, device=DEV) * 0.1 for c in (N, N, P, N))
    bias = torch.zeros(H * N, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    step = types.SimpleNamespace(n_seqs=1, n_tokens=T, max_new=T, is_decode=False, seq_start=i32([0, T]), seq_slot=i32([0]), tok_seq=i32([0] * T))
    run = lambda: ops.linear_scan(q, k, v, raw, ops.DECAY_SIGMOID, bias, None, None, 1.0, 1.0 / 16.0, torch.zeros(1, H * N * P, device=DEV), step, H, N, P)
    ops.check_status(DEV)
    want = run()
    flags = ["-DPLM_WAIT_LIMIT=20000", "-DPLM_TEST_GIVE_UP"]
    lib = load_library("scan_chunk@give_up", flags)
    lib.plm_test_give_up.argtypes = [ctypes.c_int, ctypes.c_void_p]
    stream = torch.cuda.current_stream().cuda_stream
    monkeypatch.setitem(_lib.VARIANT_OF, "scan_chunk", ("scan_chunk@give_up", flags))
    assert lib.plm_test_give_up(how, stream) == 0
    run()
    torch.cuda.synchronize()
    assert int(ops.status_word(DEV).item()) in ((44, 45, 46, 47) if how == 1 else (47,))
    with pytest.raises(ops.KernelError, match="gave up waiting"):
        ops.check_status(DEV)
    assert lib.plm_test_give_up(0, stream) == 0
    assert torch.equal(run(), want)
    ops.check_status(DEV)


CHECKED_SCRIPT = r'''
import os, sys, json
sys.path.insert(0, sys.argv[1]); sys.path.insert(0, os.path.join(sys.argv[1], "tests"))
import torch
from picolm_b200 import ops
from picolm_b200.ops import _lib
assert _lib.CHECKED
from picolm_b200.engine import Engine
from harness import run_batch, run_tail, run_whole
from plain import llama_plain as P
from util import assert_close, random_tokens
out = {}
# 1. the tiny models through the checked kernels, in both precisions and every cut: nothing is out of bounds
for d, vocab in ((sys.argv[2], 256), (sys.argv[3], 384)):
    cfg, w = P.load_model(d)
    for dtype in ("float32", "bfloat16"):
        eng = Engine.from_folder(d, dtype=dtype, max_tokens=64 * 12, max_seqs=4)
        a, b = random_tokens(100, vocab, 1), random_tokens(41, vocab, 2)
        act = torch.bfloat16 if dtype == "bfloat16" else None
        ra, rb = P.forward(cfg, w, a, act_dtype=act), P.forward(cfg, w, b, act_dtype=act)
        assert_close(run_whole(eng, a), ra, dtype, "whole")
        assert_close(run_tail(eng, b, tail=32), rb, dtype, "tail")
        for got, ref in zip(run_batch(eng, [a, b], [70, 5]), (ra, rb)):
            assert_close(got, ref, dtype, "batch")
        ops.check_status()
out["models"] = "clean"
# 2. a page table with a page number beyond the cache's pages (the tensors below have room to spare, so
#    that nothing could leave allocated memory even if the check did not act): recorded, not followed
G, hd, H = 2, 16, 4
cache_k = torch.randn(8, G, 64, hd, device="cuda")
cache_v = torch.randn(8, G, 64, hd, device="cuda")
q = torch.randn(1, H, hd, device="cuda")
pos = torch.tensor([70], dtype=torch.int32, device="cuda")
seq = torch.zeros(1, dtype=torch.int32, device="cuda")
good = torch.tensor([[1, 2, 0, 0]], dtype=torch.int32, device="cuda")
ops.attention_rows(q, cache_k[:5], cache_v[:5], pos, seq, good, G, 0.25)
torch.cuda.synchronize(); ops.check_status()
bad = torch.tensor([[1, 6, 0, 0]], dtype=torch.int32, device="cuda")          # page 6 of a cache of 5 pages
ops.attention_rows(q, cache_k[:5], cache_v[:5], pos, seq, bad, G, 0.25)
torch.cuda.synchronize()
try:
    ops.check_status()
    out["bad_page"] = "missed"
except ops.KernelError as e:
    out["bad_page"] = str(e)
far = torch.tensor([300], dtype=torch.int32, device="cuda")                   # position 300 of a table of 4 pages
ops.attention_rows(q, cache_k[:5], cache_v[:5], far, seq, good, G, 0.25)
torch.cuda.synchronize()
try:
    ops.check_status()
    out["bad_position"] = "missed"
except ops.KernelError as e:
    out["bad_position"] = str(e)
print(json.dumps(out))
'''


def test_the_checked_build_runs_clean_and_catches_a_bad_page(model_dirs):
    """A process of its own with PICOLM_B200_CHECK=1: the page-walking kernels are compiled with their
    bounds checks, the tiny models run through them in every cut with a clean status word, and a page number
    and a position outside their bounds are reported instead of followed."""
    import json
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PICOLM_B200_CHECK="1")
    r = subprocess.run([sys.executable, "-c", CHECKED_SCRIPT, root, model_dirs["A_sharp"], model_dirs["B_sharp"]],
                       capture_output=True, text=True, env=env, timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out["models"] == "clean"
    assert "page number outside its bounds" in out["bad_page"]
    assert "position outside its bounds" in out["bad_position"]
