"""How many of a prompt's positions the token kernel takes in one launch (positions_at_once), on the CPU."""
import pytest

from llama_cu_awq_b200 import _lib, synth


def _bytes(cfg, pos):
    """What a position reads: the packed layers, the classifier, the cache."""
    dim, hid, L, H, KV, V = cfg[:6]
    kvd = dim * KV // H
    shapes = [(dim, dim), (dim, kvd), (dim, kvd), (dim, dim), (dim, hid), (dim, hid), (hid, dim)]
    return L * (sum(synth.qweight_bytes(k, n) for k, n in shapes) + 4 * kvd * pos) + 2 * V * dim


@pytest.mark.parametrize("model,most", [("llama2-7b", 4), ("llama2-13b", 2), ("llama2-70b", 1), ("tiny", 32)])
def test_a_launch_of_several_positions_leaves_room_for_other_streams(model, most):
    """A launch keeps every SM: as many positions as take about 4 ms, never none."""
    L, cfg = _lib.test_lib(), synth.CONFIGS[model]
    n = [L.q4_test_positions_at_once(_bytes(cfg, pos), cfg[2]) for pos in (0, 100, cfg[6])]
    assert 1 <= n[-1] <= n[1] <= n[0] <= most
    assert n[0] == most or n[0] >= most - 1 > 0


def test_positions_at_once_has_bounds():
    L = _lib.test_lib()
    assert L.q4_test_positions_at_once(1e3, 1) == 32
    assert L.q4_test_positions_at_once(1e15, 80) == 1
    for layers in (1, 10, 1000, 6000, 20000):      # tags of a launch's positions stay within half of their 16 bits
        n = L.q4_test_positions_at_once(1e3, layers)
        assert n == 1 or n * (5 * layers + 3) <= 32768
