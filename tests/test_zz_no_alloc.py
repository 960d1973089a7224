"""q4_attention_static: the attention entry point for callers that cannot allocate device memory (hosts with all
device memory handed out at start-up, plugins that only receive the owning runtime's pointers). Checked against the oracle and, bit for bit, against q4_attention, on two
calls in a row and on calls that overlap on different streams (nothing is kept between calls)."""
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


def run_both(heads, kv_mul, hs, pos, seed):
    rng = np.random.default_rng(seed)
    stride = heads * hs // kv_mul
    host = [rng.standard_normal(heads * hs).astype(np.float16), (rng.standard_normal((pos + 1, stride)) * 0.5).astype(np.float16),
            rng.standard_normal((pos + 1, stride)).astype(np.float16)]
    q, kc, vc = map(dev, host)
    pd = torch.tensor([pos], dtype=torch.int32, device="cuda")
    ref = torch.empty(heads * hs, dtype=torch.float16, device="cuda")
    ops.MultiHeadAttention(ref, q, kc, vc, ops.attention_scratch(heads, hs), heads, hs, kv_mul, pos + 1, pd)
    out = torch.full((heads * hs,), float("nan"), dtype=torch.float16, device="cuda")
    L = _lib.lib()
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    st = L.q4_attention_static(s, C.c_void_p(out.data_ptr()), C.c_void_p(q.data_ptr()), C.c_void_p(kc.data_ptr()), C.c_void_p(vc.data_ptr()),
                               heads, hs, kv_mul, pos + 1, C.c_void_p(pd.data_ptr()))
    assert st == _lib.Q4_OK
    torch.cuda.synchronize()
    assert_close(out.cpu().numpy(), O.attention(*host, heads, hs, kv_mul, pos), f"{heads} heads, pos {pos} against the oracle", max_rel=5e-3)
    return out.cpu().numpy(), ref.cpu().numpy()


def test_static_scratch_matches_caller_scratch_twice_in_a_row():
    # two different problems back to back
    for heads, kv_mul, hs, pos, seed in [(32, 1, 128, 300, 1), (8, 4, 128, 37, 2)]:
        out, ref = run_both(heads, kv_mul, hs, pos, seed)
        assert_close(out, ref, f"static vs caller scratch ({heads} heads, pos {pos})")
        assert (out.view(np.uint16) == ref.view(np.uint16)).all()  # same kernels, same arithmetic


def test_static_call_allocates_and_frees_nothing():
    """The advertised property: a call leaves the device's free memory exactly where it was - nothing is allocated, nothing is
    freed (the first call may load the kernel). head_size 64 rides along."""
    out, ref = run_both(16, 2, 64, 90, 3)     # first use of this shape; also the head_size 64 case
    assert (out.view(np.uint16) == ref.view(np.uint16)).all()
    rng = np.random.default_rng(5)
    heads, kv_mul, hs, pos = 32, 1, 128, 200
    q = dev(rng.standard_normal(heads * hs).astype(np.float16))
    kc = dev((rng.standard_normal((pos + 1, heads * hs)) * 0.5).astype(np.float16))
    vc = dev(rng.standard_normal((pos + 1, heads * hs)).astype(np.float16))
    pd = torch.tensor([pos], dtype=torch.int32, device="cuda")
    out = torch.empty(heads * hs, dtype=torch.float16, device="cuda")
    L = _lib.lib()
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    args = (s, C.c_void_p(out.data_ptr()), C.c_void_p(q.data_ptr()), C.c_void_p(kc.data_ptr()), C.c_void_p(vc.data_ptr()), heads, hs, kv_mul, pos + 1,
            C.c_void_p(pd.data_ptr()))
    assert L.q4_attention_static(*args) == _lib.Q4_OK
    torch.cuda.synchronize()
    free_before, _ = torch.cuda.mem_get_info()
    for _ in range(3):
        assert L.q4_attention_static(*args) == _lib.Q4_OK
    torch.cuda.synchronize()
    free_after, _ = torch.cuda.mem_get_info()
    assert free_after == free_before


def test_static_calls_that_overlap_on_different_streams():
    heads, hs, pos, n = 32, 128, 1500, 4
    L = _lib.lib()
    rng = np.random.default_rng(11)
    pd = torch.tensor([pos], dtype=torch.int32, device="cuda")
    work, want = [], []
    for _ in range(n):
        q, kc, vc = dev(rng.standard_normal(heads * hs).astype(np.float16)), *(dev(rng.standard_normal((pos + 1, heads * hs)).astype(np.float16) * np.float16(0.5)) for _ in range(2))
        ref = torch.empty(heads * hs, dtype=torch.float16, device="cuda")
        ops.MultiHeadAttention(ref, q, kc, vc, ops.attention_scratch(heads, hs), heads, hs, 1, pos + 1, pd)
        work.append((q, kc, vc, torch.empty_like(ref), torch.cuda.Stream()))
        want.append(ref)
    torch.cuda.synchronize()
    for _ in range(20):
        for q, kc, vc, out, s in work:
            assert L.q4_attention_static(C.c_void_p(s.cuda_stream), C.c_void_p(out.data_ptr()), C.c_void_p(q.data_ptr()), C.c_void_p(kc.data_ptr()), C.c_void_p(vc.data_ptr()), heads, hs,
                                         1, pos + 1, C.c_void_p(pd.data_ptr())) == _lib.Q4_OK
    torch.cuda.synchronize()
    for (_, _, _, out, _), ref in zip(work, want):
        assert (out.view(torch.int16) == ref.view(torch.int16)).all()


def test_static_scratch_rejects_oversized_shapes():
    L = _lib.lib()
    heads, hs = 1024, 256
    assert L.q4_attention_scratch_bytes(heads, hs) > 256 * 1024
    x = torch.zeros(8, dtype=torch.float16, device="cuda")
    pd = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = C.c_void_p(x.data_ptr())
    st = L.q4_attention_static(C.c_void_p(torch.cuda.current_stream().cuda_stream), p, p, p, p, heads, hs, 1, 8, C.c_void_p(pd.data_ptr()))
    assert st == _lib.Q4_ERR_LIMIT
