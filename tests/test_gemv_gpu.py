"""GPU parity of the W4 g128 dequant + GEMV kernels against the CPU oracle, through the C ABI."""
import numpy as np
import pytest
import torch

from conftest import assert_close
from llama_cu_awq_b200 import _lib, ops, synth
from oracle import q4_oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(128, 8), (256, 16), (384, 8), (96, 8), (40, 16), (1024, 24), (2048, 40), (4096, 64), (640, 5120 // 8 * 0 + 64), (3584, 32),
          (11008, 32), (13824, 16), (4096, 4096)]


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def mk(K, N, seed=0):
    rng = np.random.default_rng(seed)
    q = synth.synth_qweight(rng, K, N)
    x = rng.standard_normal(K).astype(np.float16)
    return q, x, rng


@pytest.mark.parametrize("K,N", [(128, 8), (384, 16), (4096, 64), (11008, 8), (96, 8)])
def test_unpack_and_dequant_bit_exact(K, N):
    q, _, _ = mk(K, N, seed=K)
    W = ops.QWeight.from_numpy(q)
    qd, zd = ops.unpack_nibbles(W, K, N)
    qo, zo = O.unpack(q, K, N)
    assert (qd.cpu().numpy() == qo).all() and (zd.cpu().numpy() == zo).all()
    w = ops.dequant(W, K, N).cpu().numpy()
    assert (w.view(np.uint32) == O.dequant(q, K, N).view(np.uint32)).all()


@pytest.mark.parametrize("K,N", SHAPES)
def test_matvec_parity(K, N):
    q, x, _ = mk(K, N, seed=K * 7 + N)
    W = ops.QWeight.from_numpy(q)
    y = torch.full((N,), float("nan"), dtype=torch.float16, device="cuda")
    ops.matmul(y, dev(x), W, K, N)
    torch.cuda.synchronize()
    ref = O.matvec(x, q, K, N, order=1)
    r, _ = assert_close(y.cpu().numpy(), ref, f"matvec {K}x{N}")
    assert r < 4e-3  # well inside the tolerance; also compared with the unrounded sum:
    assert_close(y.cpu().numpy(), O.matvec_f32(x, q, K, N), f"matvec {K}x{N} vs f64", max_rel=4e-3)


def test_config0_single_layer():
    """The single-layer configuration of the metric: fp16 [1,4096] ~ N(0,1), 4096x4096 W4 g128, scales U[0.002,0.02], seed 0."""
    q, x, _ = mk(4096, 4096, seed=0)
    W = ops.QWeight.from_numpy(q)
    y = torch.empty(4096, dtype=torch.float16, device="cuda")
    ops.matmul(y, dev(x), W, 4096, 4096)
    r, c = assert_close(y.cpu().numpy(), O.matvec(x, q, 4096, 4096, order=1), "cfg0")
    assert r < 3e-3 and c > 0.99999


@pytest.mark.parametrize("g,K,N", [(1, 1024, 256), (2, 1024, 256), (8, 1024, 256), (2, 11008, 4096)])
def test_matvec_accum_residual(g, K, N):
    q, x, rng = mk(K, N, seed=g)
    W = ops.QWeight.from_numpy(q)
    y0 = (rng.standard_normal(N) * 5).astype(np.float16)
    y = dev(y0.copy())
    ops.matmul(y, dev(x), W, K, N, accum=True, gpu_count=g)
    assert_close(y.cpu().numpy(), O.matvec(x, q, K, N, y_old=y0, gpu_count=g, order=1), "accum", max_rel=4e-3)


def test_matvec_kv_cache_offset():
    K, N, seq, layers = 512, 64, 8, 3
    q, x, _ = mk(K, N, seed=5)
    W = ops.QWeight.from_numpy(q)
    cache = torch.zeros(layers * seq * N, dtype=torch.float16, device="cuda")
    pos = torch.tensor([5], dtype=torch.int32, device="cuda")
    loff = 2 * seq * N
    ops.matmul(cache, dev(x), W, K, N, loff=loff, pPos=pos)
    c = cache.cpu().numpy()
    ref = O.matvec(x, q, K, N, order=1)
    assert_close(c[loff + 5 * N: loff + 6 * N], ref, "kv row", max_rel=4e-3)
    c[loff + 5 * N: loff + 6 * N] = 0
    assert not c.any(), "wrote outside the cache row"


@pytest.mark.parametrize("K,Nq,Nkv", [(256, 256, 256), (512, 512, 128), (4096, 4096, 4096), (8192, 1024, 128), (256, 16000, 12000), (1024, 24000, 24000)])
def test_qkv_matvec(K, Nq, Nkv):
    rng = np.random.default_rng(K + Nkv)
    qs = [synth.synth_qweight(rng, K, n) for n in (Nq, Nkv, Nkv)]
    x = rng.standard_normal(K).astype(np.float16)
    Ws = [ops.QWeight.from_numpy(q) for q in qs]
    seq, l = 6, 1
    qo = torch.empty(Nq, dtype=torch.float16, device="cuda")
    kc = torch.zeros(2 * seq * Nkv, dtype=torch.float16, device="cuda")
    vc = torch.zeros(2 * seq * Nkv, dtype=torch.float16, device="cuda")
    pos = torch.tensor([3], dtype=torch.int32, device="cuda")
    loff = l * seq * Nkv
    ops.qkv_matvec(qo, kc, vc, dev(x), *Ws, K, Nq, loff, pos, kvSize=Nkv)
    row = slice(loff + 3 * Nkv, loff + 4 * Nkv)
    assert_close(qo.cpu().numpy(), O.matvec(x, qs[0], K, Nq, order=1), "q", max_rel=4e-3)
    assert_close(kc.cpu().numpy()[row], O.matvec(x, qs[1], K, Nkv, order=1), "k", max_rel=4e-3)
    assert_close(vc.cpu().numpy()[row], O.matvec(x, qs[2], K, Nkv, order=1), "v", max_rel=4e-3)
    assert int((kc != 0).sum()) <= Nkv and int((vc != 0).sum()) <= Nkv


@pytest.mark.parametrize("K,N", [(256, 8), (512, 1376), (4096, 11008), (5120, 1728), (256, 20000), (1024, 24000)])
def test_ffn_matvec_silu(K, N):
    rng = np.random.default_rng(K + N)
    gate, up = synth.synth_qweight(rng, K, N), synth.synth_qweight(rng, K, N)
    x = (rng.standard_normal(K) * 0.25).astype(np.float16)
    h = torch.empty(N, dtype=torch.float16, device="cuda")
    ops.ffn_matvec_silu(h, dev(x), ops.QWeight.from_numpy(gate), ops.QWeight.from_numpy(up), K, N)
    assert_close(h.cpu().numpy(), O.ffn_silu(x, gate, up, K, N, order=1), "ffn")


def test_linearity_full_size():
    """Size-independent property at the 7B down-projection size: W(a*x1 + x2) == a*W(x1) + W(x2)."""
    K, N = 11008, 4096
    q, x1, rng = mk(K, N, seed=11)
    x2 = rng.standard_normal(K).astype(np.float16)
    W = ops.QWeight.from_numpy(q)
    xs = 2.0 * x1.astype(np.float32) + x2.astype(np.float32)
    outs = []
    for x in (x1, x2, xs.astype(np.float16)):
        y = torch.empty(N, dtype=torch.float16, device="cuda")
        ops.matmul(y, dev(x), W, K, N)
        outs.append(y.float().cpu().numpy())
    assert_close(outs[2], 2.0 * outs[0] + outs[1], "linearity", max_rel=5e-3)


def test_zero_padding_nibbles_are_never_read():
    """Unused nibbles of the last zeros word may hold garbage (the reference packer leaves it there)."""
    K, N = 384, 16  # 3 groups -> 5 unused nibbles per zeros word
    q, x, _ = mk(K, N, seed=2)
    a = dict(q)
    b = dict(q)
    b["zeros"] = (q["zeros"] & np.uint32(0x00000FFF)) | np.uint32(0xABCDE000)
    ys = []
    for w in (a, b):
        y = torch.empty(N, dtype=torch.float16, device="cuda")
        ops.matmul(y, dev(x), ops.QWeight.from_numpy(w), K, N)
        ys.append(y.cpu().numpy())
    assert (ys[0].view(np.uint16) == ys[1].view(np.uint16)).all()


def test_unsupported_sizes_return_status():
    q, x, _ = mk(128, 8)
    W = ops.QWeight.from_numpy(q)
    y = torch.empty(16, dtype=torch.float16, device="cuda")
    for K, N in [(124, 8), (128, 12), (0, 8)]:
        with pytest.raises(ops.Q4Error) as e:
            ops.matmul(y, dev(x), W, K, N)
        assert e.value.status == _lib.Q4_ERR_UNSUPPORTED_SIZE
    with pytest.raises(ops.Q4Error) as e:
        ops.matmul(y, dev(x), dev(x), 12, 8)
    assert e.value.status == _lib.Q4_ERR_UNSUPPORTED_SIZE


@pytest.mark.parametrize("K,N", [(256, 8 * 297), (520, 1184 * 8 + 8), (1024, 40008), (8192, 4744 * 8), (28672, 24), (4352, 2376),
                                 (4352, 10400), (520, 90000), (4096, 11008), (4096, 3 * 148 * 8)])
def test_matvec_splits(K, N):
    """Both forms of the kernel as the launch chooses them. Direct: fewer items than warps, pairs beyond a multiple of 16, more tiles than
    one pass holds. Stream: short rows of many tiles, more tiles than one pass holds, several pairs per warp, pairs beyond a multiple of 16.
    Bound: the rounding of the result to fp16 (2^-11 of
    each value, relative to the largest at most 4.9e-4) and the fixed-point step of x (2^-16 of a group's largest, averaged over K)."""
    q, x, _ = mk(K, N, seed=K + N)
    W = ops.QWeight.from_numpy(q)
    y = torch.full((N,), float("nan"), dtype=torch.float16, device="cuda")
    ops.matmul(y, dev(x), W, K, N)
    assert_close(y.cpu().numpy(), O.matvec_f32(x, q, K, N), f"matvec {K}x{N}", max_rel=1e-3)


def no_weight_on(q, K, ks):
    """Gives every column the weight zero (nibble = zero point) on the inputs ks."""
    for k in ks:
        g, shift = k // 128, np.uint32(4 * (k % 8))
        z = (q["zeros"][:, g // 8] >> np.uint32(4 * (g % 8))) & np.uint32(15)
        w = q["weight"][:, k // 8]
        q["weight"][:, k // 8] = (w & ~(np.uint32(15) << shift)) | (z << shift)
    return q


def check_against_64_bits(got, q, x, K, N, what):
    """fp16 result of fp32 sums: half a unit of the result's last place (2^-11 of it, 2^-25 at least), 2^-23 per addition of a sum of K / 128
    group sums, whose sizes are bounded by the sums of the magnitudes, and half a step of the group's fixed point, 2^(e - 26) with e the
    exponent of its largest input, for each input below 2^(e - 15) where 32 or more are not."""
    x = x.astype(np.float64)
    step = np.zeros(K)
    for g in range(0, K, 128):
        a = np.abs(x[g:g + 128])
        e = np.floor(np.log2(a.max()))
        if (a >= 2.0 ** (e - 15)).sum() >= 32:
            step[g:g + 128] = np.where((a > 0) & (a < 2.0 ** (e - 15)) & (e >= 2), 2.0 ** (e - 26), 0)
    w = O.dequant(q, K, N).astype(np.float64)
    ref = w @ x
    bound = 2.0**-11 * np.abs(ref) + 2.0**-25 + 2.0**-23 * (2 * K / 128 + 8) * np.abs(w * x).sum(axis=1) + np.abs(w) @ step
    worst = np.max(np.abs(got.astype(np.float64) - ref) / bound)
    assert worst <= 1.0, f"{what}: {worst:.2f} of the bound"


@pytest.mark.parametrize("large", [(3,), (64,), (1, 2, 3, 4, 5, 6, 7, 8, 9)])     # in each group: odd, even, many
@pytest.mark.parametrize("ratio", [100.0, 5000.0, 3e4, 1e6])
@pytest.mark.parametrize("K,N", [(520, 64), (4096, 64), (11008, 32), (4360, 10400)])
def test_matvec_small_inputs_beside_large_ones(K, N, ratio, large):
    """Columns that give no weight to a group's large inputs: the small ones' products must come out as if they were alone."""
    q, x, rng = mk(K, N, seed=K + int(ratio))
    ks = [k for k in range(K) if k % 128 in large]
    x = (x.astype(np.float32) * (16000.0 / ratio)).astype(np.float16)
    x[ks] = (16000.0 * rng.choice([-1, 1], len(ks))).astype(np.float16)
    q["scales"] = (q["scales"].astype(np.float32) * min(1.0, ratio / 16000.0)).astype(np.float16)
    no_weight_on(q, K, ks)
    y = torch.empty(N, dtype=torch.float16, device="cuda")
    ops.matmul(y, dev(x), ops.QWeight.from_numpy(q), K, N)
    check_against_64_bits(y.cpu().numpy(), q, x, K, N, f"{K}x{N}, 1 : {ratio:g}")


@pytest.mark.parametrize("large", [(64,), (1, 2, 3, 4, 5, 6, 7, 8, 9)])
@pytest.mark.parametrize("K,N", [(2040, 19608), (8192, 2072), (13824, 640), (16640, 1192)])
def test_streamed_small_inputs_beside_large_ones(K, N, large):
    """The same in the stream form: no pairs of a warp's own, two, three, four and some left over."""
    test_matvec_small_inputs_beside_large_ones(K, N, 5000.0, large)


def test_products_of_several_matrices_with_small_inputs_beside_large_ones():
    """q|k|v, gate/up and the accumulating form: fewer pairs than warps, some left over, and the stream form with matrices that end inside a CTA's tiles."""
    for K, N, Nkv in [(384, 2368, 2368), (5000, 1024, 256), (4104, 4952, 4952)]:
        rng = np.random.default_rng(K)
        x = (rng.standard_normal(K) * 0.01).astype(np.float16)
        ks = list(range(5, K, 128))
        x[ks] = 2000.0
        qs = [no_weight_on(synth.synth_qweight(rng, K, n), K, ks) for n in (N, Nkv, Nkv)]
        qo, kc, vc = (torch.zeros(n, dtype=torch.float16, device="cuda") for n in (N, Nkv, Nkv))
        pos = torch.zeros(1, dtype=torch.int32, device="cuda")
        Ws = [ops.QWeight.from_numpy(q) for q in qs]
        ops.qkv_matvec(qo, kc, vc, dev(x), *Ws, K, N, 0, pos, kvSize=Nkv)
        for got, q, n in zip((qo, kc, vc), qs, (N, Nkv, Nkv)):
            check_against_64_bits(got.cpu().numpy(), q, x, K, n, f"q|k|v {K}x{n}")
        ops.matmul(qo, dev(x), Ws[0], K, N, accum=True)     # twice the product: half of one rounding and one of the sum
        got = qo.cpu().numpy().astype(np.float64) / 2
        ref = O.dequant(qs[0], K, N).astype(np.float64) @ x.astype(np.float64)
        assert np.abs(got - ref).max() <= 1.5 * 2.0**-11 * 1.01 * np.abs(ref).max()
        h = torch.empty(Nkv, dtype=torch.float16, device="cuda")
        ops.ffn_matvec_silu(h, dev(x), Ws[1], Ws[2], K, Nkv)
        gate, up = (O.dequant(q, K, Nkv).astype(np.float64) @ x.astype(np.float64) for q in qs[1:])
        want = gate / (1 + np.exp(-gate)) * up
        # fp16 rounding of the result; expf and the reciprocal are good to a few units of 2^-23
        assert np.abs(h.cpu().numpy() - want).max() <= 2.0**-11 * 1.02 * np.abs(want).max() + 1e-6


@pytest.mark.parametrize("K,N", [(1032, 33160), (2040, 9432), (4096, 4400), (4352, 4232), (4360, 4240), (8192, 2072), (11008, 1640),
                                 (13824, 640), (16384, 1104), (16640, 1192), (28672, 168), (41088, 120),
                                 (1032, 38800), (2040, 19608), (4096, 9800), (4352, 9200), (4360, 9176), (8064, 5560)])
def test_matvec_stream_edges(K, N):
    """The form that long and large products take, and sizes close to the line on its other side: five pairs for 16 warps, one to four pairs per warp and none to 15 left over, a last pair with one
    group and a last group that is not full, fewer tiles than SMs, tiles that do not divide by them, more than one pass of tiles."""
    q, x, _ = mk(K, N, seed=K + N)
    y = torch.full((N,), float("nan"), dtype=torch.float16, device="cuda")
    ops.matmul(y, dev(x), ops.QWeight.from_numpy(q), K, N)
    check_against_64_bits(y.cpu().numpy(), q, x, K, N, f"{K}x{N}")


@pytest.mark.parametrize("NQ,NKV,NGU,ND", [(2376, 1192, 16800, 1640), (4952, 2456, 19408, 3640)])
def test_streamed_products_of_several_matrices(NQ, NKV, NGU, ND):
    """q|k|v whose matrices end inside a CTA's tiles, gate/up in more than one pass of tiles, and the accumulating form; on both sides of 20 MB."""
    K = 4104
    rng = np.random.default_rng(5)
    x = rng.standard_normal(K).astype(np.float16)
    qs = [synth.synth_qweight(rng, K, n) for n in (NQ, NKV, NKV)]
    Ws = [ops.QWeight.from_numpy(q) for q in qs]
    qo = torch.zeros(NQ, dtype=torch.float16, device="cuda")
    kc, vc = (torch.zeros((3, NKV), dtype=torch.float16, device="cuda") for _ in range(2))
    ops.qkv_matvec(qo, kc, vc, dev(x), *Ws, K, NQ, 0, torch.full((1,), 2, dtype=torch.int32, device="cuda"), kvSize=NKV)
    assert not kc[:2].any() and not vc[:2].any()
    for got, q, n in zip((qo, kc[2], vc[2]), qs, (NQ, NKV, NKV)):
        check_against_64_bits(got.cpu().numpy(), q, x, K, n, f"q|k|v {K}x{n}")
    K, N = 1032, NGU     # 8400 and 9704 tiles: 57 and 66 for some CTAs
    x = (rng.standard_normal(K) * 0.1).astype(np.float16)
    gate, up = (synth.synth_qweight(rng, K, N) for _ in range(2))
    h = torch.empty(N, dtype=torch.float16, device="cuda")
    ops.ffn_matvec_silu(h, dev(x), ops.QWeight.from_numpy(gate), ops.QWeight.from_numpy(up), K, N)
    g, u = (O.dequant(q, K, N).astype(np.float64) @ x.astype(np.float64) for q in (gate, up))
    want = g / (1 + np.exp(-g)) * u
    # fp16 rounding of the result; expf and the reciprocal are good to a few units of 2^-23
    assert np.abs(h.cpu().numpy() - want).max() <= 2.0**-11 * 1.02 * np.abs(want).max() + 1e-6
    K, N = 11008, ND
    q, x, _ = mk(K, N, seed=9)
    W, y = ops.QWeight.from_numpy(q), torch.zeros(N, dtype=torch.float16, device="cuda")
    for _ in range(2):
        ops.matmul(y, dev(x), W, K, N, accum=True)     # twice the product: half of one rounding and one of the sum
    ref = O.dequant(q, K, N).astype(np.float64) @ x.astype(np.float64)
    assert np.abs(y.cpu().numpy().astype(np.float64) / 2 - ref).max() <= 1.5 * 2.0**-11 * 1.01 * np.abs(ref).max()


@pytest.mark.parametrize("held", [16, 31, 32, 80])
def test_matvec_small_inputs_beside_many_held_ones(held):
    """`held` inputs of a group within 2^-15 of its largest, the others far below: rounded from 32 held ones on, exact below that."""
    K, N = 1024, 64
    q, _, rng = mk(K, N, seed=held)
    x = (rng.standard_normal(K) * 1e-4).astype(np.float16)
    big = np.concatenate([g * 128 + rng.permutation(128)[:held] for g in range(K // 128)])
    x[big] = (rng.choice([-1, 1], big.size) * rng.uniform(4, 32, big.size)).astype(np.float16)
    if held < 32:
        no_weight_on(q, K, big)
    y = torch.empty(N, dtype=torch.float16, device="cuda")
    ops.matmul(y, dev(x), ops.QWeight.from_numpy(q), K, N)
    check_against_64_bits(y.cpu().numpy(), q, x, K, N, f"{held} held")


@pytest.mark.parametrize("K,N", [(512, 64), (4104, 9800), (16640, 1192)])      # direct; stream with a last group of eight inputs; four pairs and some left
@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
def test_matvec_non_finite_inputs(value, K, N):
    """A NaN in x makes every output NaN, an infinity makes it infinite with the weight's sign, or NaN where the weight is zero."""
    q, x, _ = mk(K, N, seed=3)
    x[300] = value
    x[37] = value                       # an odd position of another group
    W = ops.QWeight.from_numpy(q)
    y = torch.empty(N, dtype=torch.float16, device="cuda")
    ops.matmul(y, dev(x), W, K, N)
    w = O.dequant(q, K, N)[:, 300]
    with np.errstate(invalid="ignore"):
        want = w * np.float32(value) + O.dequant(q, K, N)[:, 37] * np.float32(value)
    assert np.array_equal(y.float().cpu().numpy(), want, equal_nan=True)


@pytest.mark.parametrize("K,N", [(512, 128), (4104, 9800)])
def test_matvec_opposite_infinities(K, N):
    """Infinities of both signs in one group, and of one sign in two groups: what IEEE sums of the products give."""
    q, x, _ = mk(K, N, seed=8)
    x[[130, 201]] = np.inf, -np.inf
    x[[3, 400]] = np.inf
    y = torch.empty(N, dtype=torch.float16, device="cuda")
    ops.matmul(y, dev(x), ops.QWeight.from_numpy(q), K, N)
    with np.errstate(invalid="ignore"):
        want = (O.dequant(q, K, N)[:, [130, 201, 3, 400]] * x[[130, 201, 3, 400]].astype(np.float32)).sum(axis=1)
    assert np.array_equal(y.float().cpu().numpy(), want, equal_nan=True) and np.isnan(want).any() and np.isinf(want).any()


@pytest.mark.parametrize("K,N", [(1024, 1024), (4352, 10400)])
def test_scales_changed_by_the_kernel_in_front(K, N):
    """Both forms of the kernel: scales rewritten in place on the stream directly before the call, with no wait in between."""
    q, x, _ = mk(K, N, seed=4)
    W, xd = ops.QWeight.from_numpy(q), dev(x)
    base = W.scales.clone()
    want = []
    for f in (0.5, 1.0):
        W.scales.copy_(base * f)
        torch.cuda.synchronize()
        y = torch.empty(N, dtype=torch.float16, device="cuda")
        ops.matmul(y, xd, W, K, N)
        torch.cuda.synchronize()
        want.append(y)
    out = torch.empty((200, N), dtype=torch.float16, device="cuda")
    for i in range(200):
        torch.mul(base, (0.5, 1.0)[i & 1], out=W.scales)
        ops.matmul(out[i], xd, W, K, N)
    assert all(torch.equal(out[i], want[i & 1]) for i in range(200))
