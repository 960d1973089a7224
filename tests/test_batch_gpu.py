"""Prompt prefill in one pass (q4_model_prefill) and batched decode of several sequences (q4_batch_*): both run the
projections as W4 dequant-GEMMs on the tensor cores and must agree with the token-by-token decode paths and the oracle."""
import numpy as np
import pytest

from conftest import MAX_REL, assert_close
from llama_cu_awq_b200 import _lib, synth
from llama_cu_awq_b200.model import Batch, Transformer
from oracle import q4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mid_path(tmp_path_factory):
    p = tmp_path_factory.mktemp("models") / "mid_gqa.bin"
    synth.write_model_file(str(p), "mid-gqa", seed=4)
    return str(p)


def token_by_token(path, tokens, fwd_path, keep):
    t = Transformer(path)
    t.reset(tokens, 0)
    out = {}
    for pos in range(len(tokens)):
        t.forward(gen_token=False, path=fwd_path)
        if pos in keep:
            t.synchronize()
            out[pos] = t.logits()
    t.synchronize()
    assert t.status() == 0
    t.close()
    return out


@pytest.mark.parametrize("n_prompt", [1, 5, 37, 100])
def test_prefill_matches_token_by_token_and_the_oracle(mid_path, n_prompt):
    """The prompt in one pass, then decoding goes on through the fused path on the cache the prefill filled: logits of the
    last prompt position and of later positions against the oracle and against the token-by-token run."""
    vocab = synth.CONFIGS["mid-gqa"][5]
    extra = 6
    tokens = np.random.default_rng(n_prompt).integers(3, vocab, size=n_prompt + extra, dtype=np.int32)
    keep = {n_prompt - 1, n_prompt + 2, n_prompt + extra - 1}
    ref = token_by_token(mid_path, tokens, 1, keep)
    t = Transformer(mid_path)
    assert t.best_path() == 2
    t.reset(tokens, 0)
    t.prefill(n_prompt, gen_token=False)
    t.synchronize()
    got = {n_prompt - 1: t.logits()}
    assert t.shared().pos == n_prompt
    for pos in range(n_prompt, n_prompt + extra):
        t.forward(gen_token=False, path=2)
        if pos in keep:
            t.synchronize()
            got[pos] = t.logits()
    t.synchronize()
    assert t.status() == 0
    t.close()
    m = O.Model(open(mid_path, "rb").read())
    for pos, tok in enumerate(tokens):
        m.forward(int(tok), pos, order=0)
        if pos in keep:
            assert_close(got[pos], m.logits(), f"prefill {n_prompt}, logits at pos {pos} vs oracle")
            assert_close(got[pos], ref[pos], f"prefill {n_prompt}, logits at pos {pos} vs token by token", max_rel=2 * MAX_REL)
    m.close()


@pytest.mark.parametrize("cfg,history,n", [("mid-gqa", 0, 17), ("mid-gqa", 3, 18), ("mid", 0, 17), ("mid", 40, 65)])
def test_a_prompts_last_layer_keeps_keys_and_values_of_all_rows(tmp_path, cfg, history, n):
    """In a prompt's last layer k and v alone are computed for all rows and q for the last one: its logits, and those of the next token, which
    reads the last layer's rows of all positions, against the oracle."""
    path = str(tmp_path / "m.bin")
    synth.write_model_file(path, cfg, seed=6)
    tokens = np.random.default_rng(n).integers(3, synth.CONFIGS[cfg][5], size=history + n + 1, dtype=np.int32)
    t = Transformer(path)
    t.reset(tokens, 0)
    if history:
        t.prefill(history, gen_token=False)
    t.prefill(n, gen_token=False)
    t.synchronize()
    got = [t.logits()]
    t.forward(gen_token=False, path=1)
    t.synchronize()
    got.append(t.logits())
    assert t.status() == 0
    t.close()
    m = O.Model(open(path, "rb").read())
    for pos, tok in enumerate(tokens):
        m.forward(int(tok), pos, order=0)
        if pos >= history + n - 1:
            # (the next token's own path is up to 1.1e-2 off the oracle on these models; another token at one position of the prompt moves
            # its logits by 6e-2 at least)
            assert_close(got[pos - (history + n - 1)], m.logits(), f"{cfg}, {n} rows behind {history}, logits at {pos} vs oracle", max_rel=2 * MAX_REL)
    m.close()


def test_prefill_hand_off_and_pieces(mid_path):
    """gen_token writes the greedy id after the prompt; a prompt fed in two pieces gives the same cache (to tolerance)."""
    vocab = synth.CONFIGS["mid-gqa"][5]
    tokens = np.random.default_rng(7).integers(3, vocab, size=48, dtype=np.int32)
    t = Transformer(mid_path)
    t.reset(tokens[:40], 0)
    t.prefill(40, gen_token=True)
    t.synchronize()
    one = t.logits()
    assert int(t.shared().tokens[40]) == O.argmax(one) and t.shared().pos == 40
    t.reset(tokens[:40], 0)
    t.prefill(23, gen_token=False)
    t.prefill(17, gen_token=True)
    t.synchronize()
    two = t.logits()
    assert t.shared().pos == 40
    assert_close(two, one, "prompt in two pieces vs one piece", max_rel=2 * MAX_REL)
    # a prompt that does not fit what is left of the sequence is refused
    L = _lib.lib()
    import ctypes as C
    assert L.q4_model_prefill(t.h, C.c_void_p(t.stream.cuda_stream), synth.CONFIGS["mid-gqa"][6], 0) == _lib.Q4_ERR_LIMIT
    t.close()


@pytest.fixture(scope="module")
def long_path(tmp_path_factory):
    p = tmp_path_factory.mktemp("models") / "mid_long.bin"
    synth.write_model_file(str(p), "mid-long", seed=6)
    return str(p)


@pytest.mark.parametrize("history,n", [(0, 64), (0, 65), (1, 63), (63, 17), (64, 64), (30, 129)])
def test_prefill_attention_at_chunk_edges(long_path, history, n):
    """The prompt attention works on 64 query rows and 64 keys at a time: prompts that end on, before and behind such an edge,
    and whose diagonal crosses a chunk elsewhere because of a history, against the token-by-token run."""
    vocab = synth.CONFIGS["mid-long"][5]
    tokens = np.random.default_rng(history + n).integers(3, vocab, size=history + n, dtype=np.int32)
    ref = token_by_token(long_path, tokens, 1, {history + n - 1})
    t = Transformer(long_path)
    t.reset(tokens, 0)
    for pos in range(history):
        t.forward(gen_token=False, path=1)
    t.prefill(n, gen_token=False)
    t.synchronize()
    got = t.logits()
    assert t.status() == 0 and t.shared().pos == history + n
    t.close()
    assert_close(got, ref[history + n - 1], f"{n} tokens behind {history}", max_rel=2 * MAX_REL)   # both sides are within MAX_REL of the oracle


def test_generate_with_the_prompt_in_one_pass(mid_path):
    """q4_generate with Q4_PATH_PROMPT_ONE_PASS: same ids as prefill of the prompt but its last position followed by the
    token loop done by hand, the same count of timed tokens as the plain loop, and a sampled run draws the coins the token
    loop would have drawn (so the same seed gives the same ids as prefill-by-hand plus sampling)."""
    vocab = synth.CONFIGS["mid-gqa"][5]
    prompt = np.random.default_rng(11).integers(3, vocab, size=12, dtype=np.int32)
    steps = 30
    t = Transformer(mid_path)
    plain, timed_plain, _ = t.generate(prompt, steps, path=2)
    one, timed_one, _ = t.generate(prompt, steps, path=2, prompt_one_pass=True)
    assert (one[:12] == prompt).all()
    t.reset(prompt, 0)
    t.prefill(11, gen_token=False)
    for pos in range(11, steps):
        t.forward(gen_token=True, path=2)
        t.synchronize()
        if pos > 0 and int(t.shared().tokens[pos]) == 2:
            break
    by_hand = np.array(t.shared().tokens[:steps + 1])
    n = min(timed_one + 1, steps)
    assert (one[:n + 1] == by_hand[:n + 1]).all()
    if (plain[:13] == one[:13]).all():       # same first generated id: then the counts agree as well
        assert abs(timed_plain - timed_one) <= steps
    # sampling: two runs with one seed agree, and the one-pass run consumes one coin per prompt position like the loop
    for run in range(2):
        t.set_sampler(0.8, 0.9, 1234)
        a, _, _ = t.generate(prompt, steps, path=2, prompt_one_pass=True)
        if run == 0:
            keep = a
    assert (a == keep).all()
    t.set_sampler(0.0, 0.9, 0)
    assert t.status() == 0
    t.close()


@pytest.fixture(scope="module")
def path_7b4l(tmp_path_factory):
    p = tmp_path_factory.mktemp("models") / "7b4l.bin"
    synth.write_model_file(str(p), "llama2-7b-4l", seed=0)
    return str(p)


def test_prefill_512_tokens_on_7b_layer_shapes(path_7b4l):
    """512 prompt positions through four layers of the 7B shapes: last-position logits against the per-op kernels fed token
    by token (the path that follows the reference's arithmetic op by op). At position 511 of this random-weight model any
    two of the three paths lie about 2e-2 apart (fused vs per-op 2.0e-2, prefill vs per-op 2.3e-2, prefill vs fused 1.8e-2;
    the long-context case against the oracle itself is the next test), so the bound here is 3e-2 and the cosine limit holds."""
    tokens = np.random.default_rng(1).integers(3, 32000, size=512, dtype=np.int32)
    ref = token_by_token(path_7b4l, tokens, 1, {511})
    t = Transformer(path_7b4l)
    t.reset(tokens, 0)
    t.prefill(512, gen_token=False)
    t.synchronize()
    assert t.status() == 0
    assert_close(t.logits(), ref[511], "512-token prefill vs token-by-token per-op path", max_rel=3 * MAX_REL)
    t.close()


def test_prefill_long_prompt_against_the_oracle(tmp_path):
    """600 positions in one pass on the long-context model (ten 64-row attention tiles, ragged last one): the last position's
    logits against the CPU oracle that walked the same 600 tokens one by one."""
    path = str(tmp_path / "midlong.bin")
    synth.write_model_file(path, "mid-long", seed=2)
    vocab = synth.CONFIGS["mid-long"][5]
    tokens = np.random.default_rng(5).integers(3, vocab, size=600, dtype=np.int32)
    t = Transformer(path)
    t.reset(tokens, 0)
    t.prefill(600, gen_token=False)
    t.synchronize()
    got = t.logits()
    assert t.status() == 0
    t.close()
    m = O.Model(open(path, "rb").read())
    for pos, tok in enumerate(tokens):
        m.forward(int(tok), pos, order=0)
    assert_close(got, m.logits(), "600-token prefill, last logits vs oracle")
    m.close()


def test_prefill_and_batched_decode_are_bit_reproducible(path_7b4l):
    """Two different prompts alternate through the same model object (so that stale rows of the other prompt would show);
    every run of a prompt must give the same bits, for the 512-token prefill and for eight sequences decoded together."""
    prompts = [np.random.default_rng(s).integers(3, 32000, size=512, dtype=np.int32) for s in (1, 2)]
    t = Transformer(path_7b4l)
    first = {}
    for rep in range(10):
        k = rep & 1
        t.reset(prompts[k], 0)
        t.prefill(512, gen_token=False)
        t.synchronize()
        bits = t.logits().view(np.uint16)
        assert (first.setdefault(k, bits) == bits).all(), f"prefill run {rep} differs from the first run of prompt {k}"
    b = Batch(t, 8)
    sets = [np.stack([synth.synth_prompt(16, 32000, seed=s * 100 + i) for i in range(8)]) for s in (1, 2)]
    first = {}
    for rep in range(6):
        k = rep & 1
        b.reset(sets[k])
        for _ in range(40):
            b.forward()
        t.synchronize()
        bits, toks = b.logits().view(np.uint16), b.tokens(41)
        ref = first.setdefault(k, (bits, toks))
        assert (ref[0] == bits).all() and (ref[1] == toks).all(), f"batched decode run {rep} differs from the first run of prompt set {k}"
    assert t.status() == 0
    b.close()
    t.close()


def test_the_first_prompt_in_new_buffers():
    """The GEMM's tile counters must read zero when the first prompt of a length that grows the buffers starts, on a stream that does not
    wait for the default one: the same bits as that prompt again."""
    dim, hid, _, H, KV, _, S, theta = synth.CONFIGS["llama2-7b"]
    for seed in range(3):
        t = Transformer(None, synthetic=((dim, hid, 1, H, KV, 512, S, theta), seed))
        ids = np.random.default_rng(seed).integers(3, 512, size=333, dtype=np.int32)
        for n in (17, 64, 77, 200, 333):
            got = []
            for _ in range(2):
                t.reset(ids, 0)
                t.prefill(n, gen_token=False)
                t.synchronize()
                got.append(t.logits().view(np.uint16))
            assert (got[0] == got[1]).all(), n
        assert t.status() == 0
        t.close()


@pytest.mark.parametrize("n_seq", [1, 8])
def test_batched_decode_matches_single_sequence_decode(mid_path, n_seq):
    """n_seq sequences with different prompts advance together; each one's logits equal (to tolerance) what the single-
    sequence path computes when it is fed that sequence's tokens, and the ids it generated are the argmax of its logits."""
    vocab = synth.CONFIGS["mid-gqa"][5]
    n_prompt, steps = 5, 14
    prompts = np.random.default_rng(3).integers(3, vocab, size=(n_seq, n_prompt), dtype=np.int32)
    t = Transformer(mid_path)
    b = Batch(t, n_seq)
    b.reset(prompts)
    per_step = []
    for _ in range(steps):
        b.forward()
        per_step.append(b.logits())
    toks = b.tokens(steps + 1)
    assert (toks[:, :n_prompt] == prompts).all()
    for s in range(n_seq):
        for pos in range(n_prompt - 1, steps):
            assert toks[s, pos + 1] == O.argmax(per_step[pos][s]), (s, pos)
    b.close()
    for s in range(n_seq):
        t.reset(toks[s], 0)
        for pos in range(steps):
            t.forward(gen_token=False, path=1)
            if pos in (0, n_prompt - 1, steps - 1):
                t.synchronize()
                assert_close(per_step[pos][s], t.logits(), f"sequence {s} of {n_seq}, pos {pos}", max_rel=2 * MAX_REL)
    t.close()


def test_a_smaller_batch_does_not_lower_the_plain_classifiers_limit():
    """A vocabulary of no whole 16s goes through the classifier that keeps the rows in shared memory (64 KB for 16 rows of 2048):
    a batch of one sequence, created after it, must leave the limit of the wide one's launch alone."""
    cfg = (2048, 512, 1, 16, 16, 40, 32, 10000.0)
    t = Transformer(None, synthetic=(cfg, 3))
    wide, narrow = Batch(t, 16), Batch(t, 1)
    prompts = np.random.default_rng(0).integers(3, cfg[5], size=(16, 3), dtype=np.int32)
    wide.reset(prompts)
    for _ in range(3):
        wide.forward()
    got = wide.logits()
    for s in (0, 7, 15):
        t.reset(prompts[s], 0)
        for _ in range(3):
            t.forward(gen_token=False, path=1)
        t.synchronize()
        assert_close(got[s], t.logits(), f"sequence {s}", max_rel=2 * MAX_REL)
    wide.close()
    narrow.close()
    t.close()


def test_failed_set_up_of_the_rows_publishes_nothing(mid_path):
    """An allocation that fails anywhere in the set-up of a prompt's rows (weight copies, rotation table, row buffers) fails that call
    only: the next one starts over and gives the bits of a model whose set-up went through; so with buffers that have to grow."""
    L = _lib.test_lib()
    vocab, layers = synth.CONFIGS["mid-gqa"][5], synth.CONFIGS["mid-gqa"][2]
    tokens = np.random.default_rng(8).integers(3, vocab, size=110, dtype=np.int32)

    def prefilled(t, n):
        t.reset(tokens[:n], 0)
        t.prefill(n, gen_token=False)
        t.synchronize()
        assert t.status() == 0
        return t.logits().view(np.uint16)

    t = Transformer(mid_path, lib=L)
    want = {n: prefilled(t, n) for n in (40, 110)}
    t.close()
    try:
        for fail_at in (0, 1, 2, 3, layers * 8 - 1, layers * 8, layers * 8 + 1, layers * 8 + 12):   # a layer: four words, two zeros and scales
            t = Transformer(mid_path, lib=L)
            t.reset(tokens[:40], 0)
            L.q4_test_fail_rows_alloc(fail_at)
            with pytest.raises(_lib.Q4Error):
                t.prefill(40, gen_token=False)
            assert (prefilled(t, 40) == want[40]).all()
            t.reset(tokens, 0)
            L.q4_test_fail_rows_alloc(3)   # the larger row buffers
            with pytest.raises(_lib.Q4Error):
                t.prefill(110, gen_token=False)
            assert (prefilled(t, 40) == want[40]).all() and (prefilled(t, 110) == want[110]).all()
            t.close()
    finally:
        L.q4_test_fail_rows_alloc(-1)


def test_failed_launch_behind_a_prompts_layers_is_reported(mid_path):
    """The launch that moves the position words fails (injected): the call says so with and without logits, the model's own position
    has not moved, and the same prompt goes through afterwards."""
    L = _lib.test_lib()
    vocab = synth.CONFIGS["mid-gqa"][5]
    tokens = np.random.default_rng(9).integers(3, vocab, size=20, dtype=np.int32)
    t = Transformer(mid_path, lib=L)
    t.reset(tokens, 0)
    L.q4_test_fail_set_pos()
    with pytest.raises(_lib.Q4Error):
        t.prefill(20, gen_token=False)
    t.prefill(20, gen_token=False)
    t.synchronize()
    assert t.shared().pos == 20
    got = t.logits().view(np.uint16)
    L.q4_test_fail_set_pos()
    with pytest.raises(_lib.Q4Error):
        t.generate(tokens, 24, path=2, prompt_one_pass=True)
    t.reset(tokens, 0)
    t.prefill(20, gen_token=False)
    t.synchronize()
    assert (t.logits().view(np.uint16) == got).all()
    t.close()
