"""Arguments of the op wrappers' native module (csrc/q4_pyops.c): wrong ones raise before anything is launched (no GPU needed)."""
import pytest

from llama_cu_awq_b200 import _lib, ops


class Stream:
    cuda_stream = 0


class Tensor:
    def data_ptr(self):
        return 4096


class Weight:
    def __init__(self):
        self.c = _lib.q4_qweight(4096, 4096, 4096)


S, T = Stream(), Tensor()


@pytest.mark.parametrize("call,error", [
    (lambda: ops.RoPERotation(T, T, "8", 8, 128, T, 0, 1e4, stream=S), TypeError),             # a size that is no number, tensors behind it
    (lambda: ops.RoPERotation(T, T, 8, 8, 128, T, 0, "theta", stream=S), TypeError),
    (lambda: ops.MultiHeadAttention(T, T, T, T, T, 8, 128.5, 1, 64, T, stream=S), TypeError),
    (lambda: ops.rmsnorm(T, T, T, 2**40, stream=S), OverflowError),
    (lambda: ops.rmsnorm(T, 4096, T, 512, stream=S), AttributeError),                          # an address where a tensor belongs
    (lambda: ops.qkv_matvec(T, T, T, T, Weight(), Weight(), T, 128, 128, 0, T, stream=S), AttributeError),   # a tensor where a matrix belongs
    (lambda: ops.copy_embedding(T, T, 128, T, T, stream=S), TypeError),                        # a tensor where a host address belongs
    (lambda: ops.sample_greedy(T, 512, 4096, T, T, True, stream=S), TypeError),
    (lambda: ops.sample_topp(T, 512, 1.0, 0.9, 0.5, T, 4096, T, stream=S), TypeError),
    (lambda: ops.rmsnorm(T, T, T, 512, stream=7), AttributeError),
])
def test_wrong_arguments_raise_what_they_are(call, error):
    with pytest.raises(error):
        call()


def test_matrix_is_read_from_the_weight_at_each_call():
    """The matrix's pointers are those of QWeight.c when the call is made (a call that is refused before its launch tells them apart)."""
    w = Weight()
    call = lambda: ops._n().matmul_q4_batched(S, T, T, w, None, 4, 128, 8, T, 1)   # noqa: E731
    assert call() == _lib.Q4_ERR_LIMIT   # a workspace of one byte
    w.c = _lib.q4_qweight(4096, None, 4096)
    assert call() == _lib.Q4_ERR_INVALID   # no zero points
    w.c = b"x"
    with pytest.raises(TypeError):
        call()


def test_library_is_built_without_the_python_headers(tmp_path, monkeypatch, capsys):
    """Without Python.h (or a C compiler) the C library and the programs are still built, and the module's absence is announced."""
    from llama_cu_awq_b200 import build as b
    assert b.PYOPS.endswith(b.sysconfig.get_config_var("EXT_SUFFIX")) and ops._n().__file__ == b.PYOPS
    monkeypatch.setattr(b, "PYOPS", str(tmp_path / "_q4ops.so"))
    monkeypatch.setattr(b.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    assert b.build() == b.LIB
    assert "not built" in capsys.readouterr().err
