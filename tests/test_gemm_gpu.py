"""The batched / prefill W4 dequant-GEMM on tcgen05 (q4_matmul_q4_batched) against the oracle: every row of Y is the
reference's matmul(QWeight) of that row of X (gpu_kernels.h:179-248), within the fp16 tolerance."""
import numpy as np
import pytest
import torch

from conftest import assert_close
from llama_cu_awq_b200 import ops, synth
from oracle import q4_oracle as O

pytestmark = pytest.mark.gpu


def interleave(dst, src, K, N):
    ops.check(ops._lib.lib().q4_gemm_interleave_weights(ops._stream(), ops._p(dst), ops._p(src), K, N), "interleave_weights")


def _case(M, K, N, seed, interleave):
    rng = np.random.default_rng(seed)
    q = synth.synth_qweight(rng, K, N)
    x = rng.standard_normal((M, K)).astype(np.float16)
    W = ops.QWeight.from_numpy(q)
    mm = ops.BatchedMatmul(W, K, N, M, interleave=interleave)
    xd = torch.from_numpy(x).cuda()
    y = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    mm(y, xd, M)
    assert mm.status() == 0
    return q, x, y.cpu().numpy(), mm, xd


@pytest.mark.parametrize("interleave", [True, False])
@pytest.mark.parametrize("M,K,N", [(16, 256, 128), (16, 128, 128), (1, 384, 136), (5, 1024, 8), (17, 640, 264), (64, 2048, 384), (100, 896, 520),
                                    (300, 512, 128)])
def test_small_shapes_against_the_oracle_rows(M, K, N, interleave):
    """Tails everywhere: rows that do not fill a batch tile, features that do not fill a 128-row tile, a last chunk of
    128 inputs, one to several K splits. Each row against the oracle's GEMV in the reference's summation order."""
    q, x, y, _, _ = _case(M, K, N, seed=M * 7 + K + N, interleave=interleave)
    for m in sorted({0, M // 2, M - 1}):
        assert_close(y[m], O.matvec(x[m], q, K, N, order=1), f"row {m} of {M}x{K}x{N}", max_rel=4e-3)
    w = O.dequant(q, K, N).astype(np.float64)     # [N][K], bit-exact dequantised weights
    assert_close(y, x.astype(np.float64) @ w.T, f"{M}x{K}x{N} vs f64", max_rel=4e-3)


@pytest.mark.parametrize("M,K,N", [(31, 256, 256), (32, 384, 248), (33, 512, 264), (65, 4096, 72), (97, 640, 4096), (160, 2048, 520), (223, 1024, 1000), (256, 1152, 16),
                                    (257, 896, 776), (385, 5120, 256), (700, 256, 2056)])
def test_batch_tiles_and_shares(M, K, N):
    """Batch tiles of every size (32 .. 256 rows, one to several), feature tiles that are not full on either CTA of a pair,
    shares that cut tiles into two and more parts; against an fp64 product of the bit-exact weights."""
    q, x, y, mm, xd = _case(M, K, N, seed=M + K + N, interleave=True)
    w = O.dequant(q, K, N).astype(np.float64)
    assert_close(y, x.astype(np.float64) @ w.T, f"{M}x{K}x{N} vs f64", max_rel=4e-3)
    y2 = torch.empty_like(torch.from_numpy(y)).cuda()
    mm(y2, xd, M)
    assert mm.status() == 0 and (y2.cpu().numpy().view(np.uint16) == y.view(np.uint16)).all()


def test_more_rows_than_a_million():
    """A narrow matrix and so many rows that the tile counters are nearly used up (8192 tiles of 256 rows are accepted)."""
    M, K, N = 1_060_000, 128, 8
    q = synth.synth_qweight(np.random.default_rng(0), K, N)
    mm = ops.BatchedMatmul(ops.QWeight.from_numpy(q), K, N, M)
    x = torch.randn((M, K), device="cuda", generator=torch.Generator("cuda").manual_seed(1)).half()
    y = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    mm(y, x, M)
    assert mm.status() == 0
    w = torch.from_numpy(O.dequant(q, K, N)).cuda()
    assert_close(y.cpu().numpy(), (x.double() @ w.double().T).cpu().numpy(), "a million rows vs f64", max_rel=4e-3)


@pytest.mark.parametrize("M", [16, 64, 512])
@pytest.mark.parametrize("K,N", [(4096, 12288), (4096, 22016), (11008, 4096), (4096, 4096)])
def test_7b_projection_shapes(M, K, N):
    """The four Llama-2-7B projection shapes (fused QKV, fused gate/up, down, O) at the three batch sizes: a few rows
    against the oracle's GEMV, the whole result against an fp32 product of the bit-exact dequantised weights."""
    q, x, y, mm, xd = _case(M, K, N, seed=K + N + M, interleave=True)
    for m in (0, M - 1):
        assert_close(y[m], O.matvec(x[m], q, K, N, order=0), f"row {m} of {M}x{K}x{N}", max_rel=4e-3)
    torch.backends.cuda.matmul.allow_tf32 = False
    w = torch.from_numpy(O.dequant(q, K, N)).cuda()
    ref = (xd.float() @ w.t()).cpu().numpy()
    assert_close(y, ref, f"{M}x{K}x{N} vs fp32 product", max_rel=4e-3)
    # a second call on the same workspace (tile counters back at zero) and bit-equal results (fixed summation order)
    y2 = torch.empty_like(torch.from_numpy(y)).cuda()
    mm(y2, xd, M)
    assert mm.status() == 0
    assert (y2.cpu().numpy().view(np.uint16) == y.view(np.uint16)).all()


def test_back_to_back_launches_are_bit_reproducible():
    """Forty launches queued back to back on one workspace (their prologues overlap the previous launch's tail through
    programmatic dependent launch): every result equals the first, bit for bit."""
    M, K, N = 512, 4096, 11008
    q, x, y, mm, xd = _case(M, K, N, seed=3, interleave=True)
    first = torch.from_numpy(y).cuda()
    outs = [torch.zeros_like(first) for _ in range(8)]
    for _ in range(5):
        for o in outs:
            mm(o, xd, M)
        torch.cuda.synchronize()
        for o in outs:
            assert torch.equal(o, first)
    assert mm.status() == 0


@pytest.mark.parametrize("M,K,N", [(64, 4096, 22016), (33, 512, 264)])
def test_weights_written_by_the_kernel_before(M, K, N):
    """A call behind the kernel that wrote its packed words, without a wait between them: two matrices in turn in one buffer, the bits of
    the calls on settled words each time."""
    rng = np.random.default_rng(K)
    xd = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float16)).cuda()
    W = [ops.QWeight.from_numpy(synth.synth_qweight(rng, K, N)) for _ in range(2)]
    mm = ops.BatchedMatmul(W[0], K, N, M)
    other = ops.BatchedMatmul(W[1], K, N, M)
    want = torch.empty((2, M, N), dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    mm(want[0], xd, M)
    mm.wi, other.wi = other.wi, mm.wi
    mm(want[1], xd, M)
    y = torch.empty((20, M, N), dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    for i in range(20):
        interleave(mm.wi, W[i % 2].weight, K, N)
        mm(y[i], xd, M)
    assert mm.status() == 0
    for i in range(20):
        assert (y[i].view(torch.int16) == want[i % 2].view(torch.int16)).all(), i


@pytest.mark.parametrize("M,K,N", [(64, 4096, 22016), (17, 512, 264)])
@pytest.mark.parametrize("behind", ["gemm", "gemv", "gemv stream", "rows"])
def test_weights_of_a_writer_that_lets_the_next_kernel_in_early(M, K, N, behind):
    """The kernel in front signals its dependents first and writes the packed words late. A GEMM on those words reads them when it has ended; a product
    behind a GEMM on another matrix, whose words may be read ahead of its own wait, starts only when the GEMM has waited."""
    from llama_cu_awq_b200 import _lib
    L = _lib.test_lib()
    rng = np.random.default_rng(K)
    xd = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float16)).cuda()
    front = ops.BatchedMatmul(ops.QWeight.from_numpy(synth.synth_qweight(rng, K, N)), K, N, M)
    K2, N2 = {"gemm": (K, N), "gemv": (1024, 1024), "gemv stream": (11008, 4096), "rows": (1024, 1024)}[behind]
    q = synth.synth_qweight(rng, K2, N2)
    W, src = ops.QWeight.from_numpy(q), [torch.from_numpy(synth.synth_qweight(rng, K2, N2)["weight"].view(np.int32)).cuda() for _ in range(2)]
    x2 = torch.from_numpy(rng.standard_normal((M if behind == "gemm" else 8, K2)).astype(np.float16)).cuda()
    mm = ops.BatchedMatmul(W, K2, N2, M, interleave=False)
    out = torch.empty((10, M if behind == "gemm" else 8, N2), dtype=torch.float16, device="cuda")
    yf = torch.empty((M, N), dtype=torch.float16, device="cuda")

    def product(y):
        if behind == "gemm":
            mm(y, x2, M)
        elif behind == "rows":
            ops.matmul_rows(y, x2, W, 8, K2, N2)
        else:
            ops.matmul(y[0], x2[0], W, K2, N2)

    want = torch.zeros_like(out[:2])
    out.zero_()
    for i in range(2):
        W.weight.copy_(src[i])
        torch.cuda.synchronize()
        product(want[i])
        torch.cuda.synchronize()
    for i in range(10):
        assert L.q4_test_write_late(ops._stream(), ops._p(W.weight), ops._p(src[i % 2]), W.weight.numel(), 40000) == 0
        if behind != "gemm":
            front(yf, xd, M)
        product(out[i])
    torch.cuda.synchronize()
    assert mm.status() == 0 and front.status() == 0
    for i in range(10):
        assert torch.equal(out[i], want[i % 2]), i


@pytest.mark.parametrize("M,K,N", [(40, 1024, 520), (300, 4096, 256), (512, 11008, 512)])
def test_residual_epilogue(M, K, N):
    """y = product + y * scale in place (q4_matmul_q4_batched_residual), whole tiles and tiles in several parts."""
    from llama_cu_awq_b200 import _lib
    q, x, y, mm, xd = _case(M, K, N, seed=M, interleave=True)
    r = np.random.default_rng(1).standard_normal((M, N)).astype(np.float16)
    yd = torch.from_numpy(r).cuda()
    e = _lib.lib().q4_matmul_q4_batched_residual(ops._stream(), ops._p(yd), ops._p(xd), mm.w.ref, ops._p(mm.wi), M, K, N, ops._p(yd), 0.5, ops._p(mm.ws), mm.ws_bytes)
    assert e == 0 and mm.status() == 0
    w = O.dequant(q, K, N).astype(np.float64)
    assert_close(yd.cpu().numpy(), x.astype(np.float64) @ w.T + 0.5 * r, f"{M}x{K}x{N} + residual", max_rel=4e-3)


@pytest.mark.parametrize("offset", [1, 4])
@pytest.mark.parametrize("M,K,N", [(1, 128, 8), (33, 512, 264), (300, 4096, 520)])
def test_y_of_any_alignment(M, K, N, offset):
    """A result (and a residual in it) that does not start on 16 bytes: the bits of the aligned call, and nothing written around it."""
    from llama_cu_awq_b200 import _lib
    q, x, y, mm, xd = _case(M, K, N, seed=M + K, interleave=True)
    buf = torch.full((M * N + 16,), 7.0, dtype=torch.float16, device="cuda")
    view = buf[offset : offset + M * N].view(M, N)
    mm(view, xd, M)
    assert mm.status() == 0 and (view.cpu().numpy().view(np.uint16) == y.view(np.uint16)).all()
    assert (buf[:offset] == 7).all() and (buf[offset + M * N :] == 7).all()
    outs = []
    for out in (torch.ones((M, N), dtype=torch.float16, device="cuda"), view.fill_(1)):
        assert _lib.lib().q4_matmul_q4_batched_residual(ops._stream(), ops._p(out), ops._p(xd), mm.w.ref, ops._p(mm.wi), M, K, N, ops._p(out), 0.5, ops._p(mm.ws),
                                                        mm.ws_bytes) == 0
        outs.append(out.cpu().numpy().view(np.uint16))
    assert mm.status() == 0 and (outs[0] == outs[1]).all()


@pytest.mark.parametrize("M,K,N", [(16, 128, 128), (64, 4096, 4096), (300, 11008, 520), (512, 1024, 22016)])
def test_calls_behind_a_recorded_time_out_end(M, K, N):
    """A status word that already holds a time-out (what calls queued behind one that ran out of time meet): every role gives up at
    its first unfinished wait, the calls end and report the status; with the workspace zeroed the next call is right again."""
    from llama_cu_awq_b200 import _lib
    q, x, y, mm, xd = _case(M, K, N, seed=M + N, interleave=True)
    y2 = torch.empty((M, N), dtype=torch.float16, device="cuda")
    mm.ws.view(torch.int32)[0] = _lib.Q4_ERR_TIMEOUT
    for _ in range(4):
        mm(y2, xd, M)
    assert mm.status() == _lib.Q4_ERR_TIMEOUT
    mm.ws.zero_()
    mm(y2, xd, M)
    assert mm.status() == 0 and (y2.cpu().numpy().view(np.uint16) == y.view(np.uint16)).all()


@pytest.mark.parametrize("M", [40, 512])
def test_gate_up_epilogue_values(M):
    """silu(gate) * up as the GEMM's epilogue forms it, for gates and ups that the test chooses (one weight of a row is not zero): the
    result is the rounding of a value within the fp32 evaluation's error of the 64-bit one. That error: expf 2 ulp (2^-22), then
    one rounding each (2^-24) of 1 + e, of the division and of the two products."""
    from llama_cu_awq_b200 import _lib
    L = _lib.test_lib()
    K, hid = 128, 2048
    rng = np.random.default_rng(M)
    w = np.zeros((2 * hid, 16), np.uint32)
    w[0::2, 0], w[1::2, 0] = 1, 1 << 4   # gate = scale * x[0], up = x[1] (zero points 0)
    scales = np.ones((2 * hid, 1), np.float16)
    scales[0::2, 0] = rng.uniform(0.5, 1.0, hid).astype(np.float16)
    q = ops.QWeight.from_numpy({"weight": w, "zeros": np.zeros((2 * hid, 1), np.uint32), "scales": scales})
    x = np.zeros((M, K), np.float16)
    x[:, 0] = rng.uniform(-20.0, -8.0, M)              # where the exponential decides the bits
    x[: M // 4, 0] = rng.uniform(-8.0, 100.0, M // 4)
    x[:4, 0] = [0.0, -0.0, -100.0, 100.0]
    x[:, 1] = np.where(x[:, 0] < -8, 6e4, 90.0) * rng.uniform(0.5, 1.0, M) * rng.choice([-1, 1], M)
    mm = ops.BatchedMatmul(q, K, 2 * hid, M)
    y = torch.full((M, hid), float("nan"), dtype=torch.float16, device="cuda")
    xd = torch.from_numpy(x).cuda()
    assert L.q4_test_gemm_silu(ops._stream(), ops._p(y), ops._p(xd), q.ref, ops._p(mm.wi), M, K, 2 * hid, ops._p(mm.ws), mm.ws_bytes) == 0 and mm.status() == 0
    gate = (x[:, :1].astype(np.float32) * scales[0::2, 0].astype(np.float32)).astype(np.float16).astype(np.float64)
    ref = gate / (1.0 + np.exp(-gate)) * x[:, 1:2].astype(np.float64)
    d = 2.0**-22 + 4 * 2.0**-24
    a, b = (ref * (1 - d)).astype(np.float16), (ref * (1 + d)).astype(np.float16)
    got = y.cpu().numpy()
    wrong = (got < np.minimum(a, b)) | (got > np.maximum(a, b)) | ~np.isfinite(got)
    assert not wrong.any(), f"{wrong.sum()} of {wrong.size}"


def test_rejects_unsupported_arguments():
    from llama_cu_awq_b200 import _lib
    rng = np.random.default_rng(0)
    q = synth.synth_qweight(rng, 96, 8)
    W = ops.QWeight.from_numpy(q)
    x = torch.zeros((4, 96), dtype=torch.float16, device="cuda")
    y = torch.zeros((4, 8), dtype=torch.float16, device="cuda")
    ws = torch.zeros(4096, dtype=torch.uint8, device="cuda")
    L = _lib.lib()
    s = ops._stream()
    assert L.q4_matmul_q4_batched(s, ops._p(y), ops._p(x), W.ref, None, 4, 96, 8, ops._p(ws), 4096) == _lib.Q4_ERR_UNSUPPORTED_SIZE   # K % 128
    q = synth.synth_qweight(rng, 128, 8)
    W = ops.QWeight.from_numpy(q)
    x = torch.zeros((4, 128), dtype=torch.float16, device="cuda")
    assert L.q4_matmul_q4_batched(s, ops._p(y), ops._p(x), W.ref, None, 4, 128, 8, ops._p(ws), 16) == _lib.Q4_ERR_LIMIT   # workspace too small
    assert L.q4_matmul_q4_batched(s, ops._p(y), ops._p(x), W.ref, None, 0, 128, 8, ops._p(ws), 4096) == _lib.Q4_ERR_INVALID
    nb = L.q4_matmul_q4_batched_workspace_bytes(4, 128, 8)
    big = torch.zeros(nb, dtype=torch.uint8, device="cuda")
    c = W.c
    for part in ((None, c.zeros, c.scales), (c.weight, None, c.scales), (c.weight, c.zeros, None)):   # a matrix without one of its parts
        assert L.q4_matmul_q4_batched(s, ops._p(y), ops._p(x), _lib.q4_qweight(*part), None, 4, 128, 8, ops._p(big), nb) == _lib.Q4_ERR_INVALID
