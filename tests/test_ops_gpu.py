"""GPU parity of RMSNorm, RoPE, attention, the fp16 classifier GEMV, embedding gather and the greedy hand-off."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import assert_close
from llama_cu_awq_b200 import _lib, ops
from oracle import q4_oracle as O

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("n", [8, 128, 1000, 4096, 5120, 8192])
def test_rmsnorm(n):
    rng = np.random.default_rng(n)
    x = (rng.standard_normal(n) * 3).astype(np.float16)
    w = rng.uniform(0.5, 1.5, n).astype(np.float16)
    o = torch.empty(n, dtype=torch.float16, device="cuda")
    ops.rmsnorm(o, dev(x), dev(w), n)
    ref = O.rmsnorm(x, w)
    got = o.cpu().numpy()
    assert_close(got, ref, "rmsnorm", max_rel=2e-3)
    def key(a):
        u = a.view(np.uint16).astype(np.int32)
        return np.where(u & 0x8000, -(u & 0x7FFF), u)
    assert np.abs(key(got) - key(ref)).max() <= 1  # at most 1 fp16 step
    xd = dev(x)
    ops.rmsnorm(xd, xd, dev(w), n)  # in place, as the final norm does (llama2_q4.cu:528)
    assert (xd.cpu().numpy().view(np.uint16) == got.view(np.uint16)).all()


# one and two pieces per thread, the largest row that stays in registers (8192 at 512 threads, 16384 at 1024), one past it
@pytest.mark.parametrize("n", [8, 4088, 4104, 8184, 8192, 16384, 16392])
def test_rmsnorm_in_registers_and_not(n):
    rng = np.random.default_rng(n)
    x = (rng.standard_normal(n) * 3).astype(np.float16)
    w = rng.uniform(0.5, 1.5, n).astype(np.float16)
    o = torch.empty(n + 8, dtype=torch.float16, device="cuda")
    wd = dev(np.r_[w[:1], w])          # w again, two bytes further
    xd = dev(x)
    got = []
    for ov, wv in ((o[:n], dev(w)), (o[1:n + 1], dev(w)), (o[:n], wd[1:])):     # the last two do not start on 16 bytes
        ops.rmsnorm(ov, xd, wv, n)
        got.append(ov.cpu().numpy().copy())
    assert_close(got[0], O.rmsnorm(x, w), "rmsnorm", max_rel=2e-3)
    for g in got[1:]:
        assert (g.view(np.uint16) == got[0].view(np.uint16)).all()      # same sums in the same order, one rounding


# several pairs per thread (head size 512), heads and key heads that end inside a block, a head size that is no power of two
@pytest.mark.parametrize("heads,kv_heads,hs,pos", [(6, 6, 512, 11), (5, 2, 256, 70), (7, 3, 96, 9), (1, 1, 2, 3)])
def test_rope_pairs_per_thread(heads, kv_heads, hs, pos):
    test_rope(heads, kv_heads, hs, pos)


@pytest.mark.parametrize("heads,kv_heads,hs,pos", [(2, 2, 64, 0), (32, 32, 128, 17), (8, 1, 128, 4095), (4, 2, 128, 300)])
def test_rope(heads, kv_heads, hs, pos):
    rng = np.random.default_rng(pos + heads)
    q = rng.standard_normal(heads * hs).astype(np.float16)
    seq, layers = pos + 2, 2
    kv_dim = kv_heads * hs
    kc = rng.standard_normal(layers * seq * kv_dim).astype(np.float16)
    loff = 1 * seq * kv_dim
    qd, kd = dev(q), dev(kc)
    ops.RoPERotation(qd, kd, heads, kv_heads, hs, torch.tensor([pos], dtype=torch.int32, device="cuda"), loff, 10000.0)
    row = slice(loff + pos * kv_dim, loff + (pos + 1) * kv_dim)
    qr, kr = O.rope(q, kc[row], heads, kv_heads, hs, pos, 10000.0)
    # sin/cos of large arguments differ by a few ulp of fp32 between libm and CUDA; outputs are fp16
    assert_close(qd.cpu().numpy(), qr, "rope q", max_rel=2e-3)
    k_out = kd.cpu().numpy()
    assert_close(k_out[row], kr, "rope k", max_rel=2e-3)
    k_out[row] = kc[row]
    assert (k_out.view(np.uint16) == kc.view(np.uint16)).all(), "touched other cache rows"


@pytest.mark.parametrize("heads,kv_mul,hs,pos", [(2, 1, 64, 0), (4, 1, 128, 5), (32, 1, 128, 15), (32, 1, 128, 271), (8, 8, 128, 1000),
                                               (64, 8, 128, 33), (40, 1, 128, 2047), (2, 2, 256, 77)])
def test_attention(heads, kv_mul, hs, pos):
    rng = np.random.default_rng(pos * 3 + heads)
    kv_stride = heads * hs // kv_mul
    seq = pos + 3
    q = rng.standard_normal(heads * hs).astype(np.float16)
    kc = (rng.standard_normal((seq, kv_stride)) * 0.5).astype(np.float16)
    vc = rng.standard_normal((seq, kv_stride)).astype(np.float16)
    kc[pos + 1:] = np.float16(100.0)  # rows beyond pos must not be read
    vc[pos + 1:] = np.float16(-1000.0)
    out = torch.full((heads * hs,), float("nan"), dtype=torch.float16, device="cuda")
    scratch = ops.attention_scratch(heads, hs)
    ops.MultiHeadAttention(out, dev(q), dev(kc), dev(vc), scratch, heads, hs, kv_mul, seq, torch.tensor([pos], dtype=torch.int32, device="cuda"))
    ref = O.attention(q, kc, vc, heads, hs, kv_mul, pos)
    # the reference rounds probabilities to fp16 before the V product; the split softmax here stays in fp32
    assert_close(out.cpu().numpy(), ref, f"attention pos={pos}", max_rel=5e-3)


def _attention(heads, kv_mul, hs, pos, q, kc, vc):
    out = torch.full((heads * hs,), float("nan"), dtype=torch.float16, device="cuda")
    ops.MultiHeadAttention(out, dev(q), dev(kc), dev(vc), ops.attention_scratch(heads, hs), heads, hs, kv_mul, pos + 1,
                           torch.tensor([pos], dtype=torch.int32, device="cuda"))
    return out.cpu().numpy()


# both sides of every line between clusters of eight, four, two and one (37, 74 and 148 heads), shares that are empty, end on a step of
# 64 positions or one past it
@pytest.mark.parametrize("heads,kv_mul,hs", [(1, 1, 128), (15, 1, 128), (16, 1, 256), (37, 1, 64), (38, 2, 64), (64, 8, 128), (74, 2, 64), (75, 5, 64), (148, 4, 64), (149, 1, 64), (150, 3, 256)])
@pytest.mark.parametrize("pos", [0, 31, 32, 255, 256, 511, 512, 600])
def test_attention_clusters_and_share_edges(heads, kv_mul, hs, pos):
    rng = np.random.default_rng(pos * 7 + heads)
    stride = heads * hs // kv_mul
    q = rng.standard_normal(heads * hs).astype(np.float16)
    kc, vc = ((rng.standard_normal((pos + 1, stride)) * s).astype(np.float16) for s in (0.5, 1.0))
    assert_close(_attention(heads, kv_mul, hs, pos, q, kc, vc), O.attention(q, kc, vc, heads, hs, kv_mul, pos), f"{heads} heads, pos {pos}", max_rel=5e-3)


@pytest.mark.parametrize("heads", [4, 149])     # eight blocks per head, one
def test_attention_with_scores_that_are_not_finite(heads):
    """A score of -infinity (rounded to fp16) has weight 0, also where it is the first or the only one a lane group sees; a NaN reaches
    its own head's outputs and no other's."""
    hs, pos = 128, 40
    rng = np.random.default_rng(heads)
    q = np.abs(rng.standard_normal(heads * hs)).astype(np.float16) + np.float16(0.5)
    kc = (rng.standard_normal((pos + 1, heads * hs)) * 0.5).astype(np.float16)
    vc = rng.standard_normal((pos + 1, heads * hs)).astype(np.float16)
    low = [0, 1, 2, 33]
    kc[low] = np.float16(-60000.0)             # scores far below -65504
    want = O.attention(q, np.delete(kc, low, 0), np.delete(vc, low, 0), heads, hs, 1, pos - len(low))
    assert_close(_attention(heads, 1, hs, pos, q, kc, vc), want, "scores of -infinity", max_rel=5e-3)
    kc[35, hs] = np.nan                        # head 1
    got = _attention(heads, 1, hs, pos, q, kc, vc)
    assert np.isnan(got[hs:2 * hs]).all()
    rest = np.r_[0:hs, 2 * hs:heads * hs]
    assert_close(got[rest], want[rest], "other heads", max_rel=5e-3)


@pytest.mark.parametrize("n,d", [(8, 8), (256, 40), (4096, 1000), (5120, 4000), (4096, 32000)])
def test_classifier_matvec_f16(n, d):
    rng = np.random.default_rng(n + d)
    W = (rng.standard_normal((d, n)) * 0.02).astype(np.float16)
    x = rng.standard_normal(n).astype(np.float16)
    y = torch.empty(d, dtype=torch.float16, device="cuda")
    ops.matmul(y, dev(x), dev(W), n, d)
    assert_close(y.cpu().numpy(), O.matvec_f16(x, W, n, d, order=1), "classifier", max_rel=2e-3)


@pytest.mark.parametrize("d", [8, 592, 600, 1184, 1192, 2368, 2376])
@pytest.mark.parametrize("n", [8, 1032, 4096])
def test_classifier_matvec_f16_split_edges(n, d):
    """The sizes on both sides of every split of a row over warps, rows shorter than the split and rows with a remainder. Against
    64 bits: one rounding to fp16 (2^-11 of the value, 2^-25 where it is a denormal) and fp32 roundings of a chain of n / 32 fused
    multiply-adds in a lane (rounded up to a 16-byte piece), five additions of lanes and at most eight of warps."""
    rng = np.random.default_rng(n * d)
    W = (rng.standard_normal((d, n)) * 0.02).astype(np.float16)
    x = rng.standard_normal(n).astype(np.float16)
    y = torch.full((d,), float("nan"), dtype=torch.float16, device="cuda")
    ops.matmul(y, dev(x), dev(W), n, d)
    ref = W.astype(np.float64) @ x.astype(np.float64)
    terms = np.abs(W).astype(np.float64) @ np.abs(x).astype(np.float64)
    bound = np.abs(ref) * 2.0**-11 + 2.0**-25 + 1.01 * (n / 32 + 8 + 5 + 8) * 2.0**-24 * terms
    assert (np.abs(y.cpu().numpy().astype(np.float64) - ref) <= bound).all()


def _pinned_mailbox():
    t = torch.zeros(4 + 64, dtype=torch.int32).pin_memory()
    return t  # [0] = pos, [4:] = tokens (layout is private to this test)


def test_embed_and_argmax_handoff():
    rng = np.random.default_rng(0)
    V, dim = 1000, 256
    table = rng.standard_normal((V, dim)).astype(np.float16)
    mb = _pinned_mailbox()
    mb[4 + 3] = 777
    pos_dev = torch.tensor([3], dtype=torch.int32, device="cuda")
    mb[0] = 3
    x = torch.empty(dim, dtype=torch.float16, device="cuda")
    tokens_ptr = mb.data_ptr() + 16
    ops.copy_embedding(x, dev(table), dim, tokens_ptr, pos_dev)
    torch.cuda.synchronize()
    assert (x.cpu().numpy().view(np.uint16) == table[777].view(np.uint16)).all()

    logits = rng.standard_normal(V).astype(np.float16)
    logits[[123, 600]] = np.float16(9.0)  # tie: lowest index wins
    ops.sample_greedy(dev(logits), V, tokens_ptr, mb.data_ptr(), pos_dev, True)
    torch.cuda.synchronize()
    assert int(mb[0]) == 4 and int(pos_dev.item()) == 4 and int(mb[4 + 4]) == 123 == O.argmax(logits)
    ops.sample_greedy(dev(logits), V, tokens_ptr, mb.data_ptr(), pos_dev, False)  # prompt phase: position only
    torch.cuda.synchronize()
    assert int(mb[0]) == 5 and int(mb[4 + 5]) == 0


@pytest.mark.parametrize("size", [8, 1000, 32000])
def test_argmax_matches_oracle(size):
    rng = np.random.default_rng(size)
    for trial in range(3):
        logits = (rng.standard_normal(size) * 2).astype(np.float16)  # fp16 values collide often at 32000
        mb = _pinned_mailbox()
        pos_dev = torch.zeros(1, dtype=torch.int32, device="cuda")
        ops.sample_greedy(dev(logits), size, mb.data_ptr() + 16, mb.data_ptr(), pos_dev, True)
        torch.cuda.synchronize()
        assert int(mb[4 + 1]) == O.argmax(logits)


# one load per thread and several, remainders behind the last eight, logits that do not start on 16 bytes
@pytest.mark.parametrize("size", [1, 7, 8, 9, 8191, 8200, 32771, 70003])
@pytest.mark.parametrize("shift", [0, 1])
def test_argmax_ties_and_remainders(size, shift):
    rng = np.random.default_rng(size)
    base = rng.standard_normal(size).astype(np.float16)
    cases = [(base, None), (np.full(size, -np.inf, np.float16), 0), (np.full(size, np.nan, np.float16), 0)]
    for a, b in ((0, size - 1), (size // 2, size - 1), (size // 3, size // 3)):     # the lowest of two equal maxima
        v = base.copy()
        v[[a, b]] = 9.0
        v[max(a - 1, 0):a] = np.nan                                                 # a NaN in front does not win
        cases.append((v, a))
    for v, want in cases:
        buf = torch.empty(size + 8, dtype=torch.float16, device="cuda")
        x = buf[shift:shift + size]
        x.copy_(torch.from_numpy(v))
        mb = _pinned_mailbox()
        pos_dev = torch.zeros(1, dtype=torch.int32, device="cuda")
        ops.sample_greedy(x, size, mb.data_ptr() + 16, mb.data_ptr(), pos_dev, True)
        torch.cuda.synchronize()
        assert int(mb[4 + 1]) == (int(np.argmax(v)) if want is None else want)
