"""Decode steps of few sequences as one persistent kernel (tuning key "few"): against the oracle and against the same
steps launched one kernel per operation."""
import numpy as np
import pytest

import b200nn
import np_ref
from b200nn import DecodeSession, Gpt2Config, Gpt2Model, Int4Gpt2Model, synth
from oracle import oracle
from test_gpu_model import MAX_ABS, REL_RMS, _check_tokens, _int4_oracle_weights

pytestmark = pytest.mark.gpu


def _steps(reg, m, prompts, n_new, few, flags=0):
    reg.set_tuning("few", few)
    try:
        B, P = prompts.shape
        s = DecodeSession(m, batch=B, capacity=P + n_new, flags=flags)
        s.prefill(prompts)
        s.step(1)
        launches = reg.launch_count()
        s.step(n_new - 2)
        return s.tokens(), s.logits(), reg.launch_count() - launches
    finally:
        reg.set_tuning("few", 1)


# The narrowest model (12 blocks, one K unit per part, fewer tiles of the output matrix than blocks); contexts that cross one
# and three context splits of 120 rows; three of four row slots; more steps than a launch takes; an odd group of 192;
# one, three and two K parts of the projections (GPT-2 XL's, Small's and Medium's widths); an output matrix of 22 tiles a block.
@pytest.mark.parametrize("family,d,layers,vocab,B,P,N,group", [
    ("f32", 64, 1, 131, 4, 9, 5, 0), ("f32", 128, 2, 257, 3, 117, 8, 0), ("int4", 128, 3, 257, 2, 9, 40, 64),
    ("int4", 192, 2, 1031, 1, 357, 7, 192), ("f32", 768, 2, 50257, 1, 33, 5, 0), ("f32", 1024, 1, 3001, 4, 20, 5, 0),
    ("int4", 768, 2, 5003, 2, 250, 5, 128), ("int4", 1600, 2, 50257, 1, 77, 5, 128)])
def test_steps_in_one_kernel_match_oracle_and_per_operation_path(reg, family, d, layers, vocab, B, P, N, group):
    cfg = Gpt2Config(n_layer=layers, n_embd=d, n_head=d // 64, vocab_size=vocab, n_positions=400)
    w = synth.gpt2_weights(cfg, base_seed=70 + d, std=0.08 if d < 512 else 0.02, random_ln=True)
    m = Gpt2Model(w, cfg, reg) if family == "f32" else Int4Gpt2Model(w, cfg, reg, flags=b200nn.QUANT_LM_HEAD, group_size=group)
    prompts = synth.token_ids(d + B, (B, P), vocab)
    tok, lg, launches = _steps(reg, m, prompts, N, 1)
    tok_o, lg_o, launches_o = _steps(reg, m, prompts, N, 0)
    assert reg.device_error() == 0
    assert launches == (N - 2 + 31) // 32 and launches_o > launches * layers
    # The paths differ by the order of f32 sums, and where that turns the fp16 rounding of a cached value, by 2^-11 of it:
    # under 1e-3 in logits of spread one.  A near-tie may turn a pick, and all that follows it.
    same = (tok == tok_o).all(axis=1)
    assert same.sum() >= B - 1
    assert not same.any() or np.abs(lg - lg_o)[same].max() < 1e-3
    if d <= 768 and vocab < 10000:
        om = oracle.Model(cfg.as_dict(), w if family == "f32" else _int4_oracle_weights(m, cfg, w, True))
        for b in sorted({0, B - 1}):
            ref, lr = om.generate_cached(prompts[b], N, flags=oracle.KV_FP16, want_logits=True)
            _check_tokens(np.concatenate([prompts[b], tok[b]]), ref, lr, P)
            if np.array_equal(tok[b], ref[P:]):
                assert np.abs(lg[b] - lr[-1]).max() < MAX_ABS and np_ref.rel_rms(lg[b], lr[-1]) < REL_RMS


def test_steps_in_one_kernel_rewind_and_last_index_picks(reg):
    """Steps taken again after a rewind (from the last token picked) are those of the per-operation path.  Equal logits
    everywhere: the last index wins when asked for."""
    cfg = Gpt2Config(n_layer=2, n_embd=128, n_head=2, vocab_size=259, n_positions=64)
    w = dict(synth.gpt2_weights(cfg, base_seed=3, std=0.08))
    m = Gpt2Model(w, cfg, reg)
    prompts = synth.token_ids(4, (2, 9), cfg.vocab_size)

    def again(few):
        reg.set_tuning("few", few)
        try:
            s = DecodeSession(m, batch=2, capacity=40)
            s.prefill(prompts)
            s.step(12)
            out = [s.logits()]
            for back, n in ((20, 1), (13, 6), (10, 30)):
                s.rewind(back)
                s.step(n)
                out += [s.logits(), s.tokens()]
            return out
        finally:
            reg.set_tuning("few", 1)
    for a, b in zip(again(1), again(0)):
        assert a.shape == b.shape and np.isfinite(a).all()
        # the order of f32 sums and what it turns in the fp16 cache, as above
        assert np.array_equal(a, b) if a.dtype == np.uint32 else np.abs(a - b).max() < 1e-3
    w["wte"] = np.zeros_like(w["wte"])
    flat = Gpt2Model(w, cfg, reg)
    for flags, pick in ((0, 0), (b200nn.ARGMAX_LAST, cfg.vocab_size - 1)):
        assert (_steps(reg, flat, prompts, 5, 1, flags)[0] == pick).all()


def test_steps_in_one_kernel_wait_runs_out_and_session_recovers(reg):
    cfg = Gpt2Config(n_layer=3, n_embd=128, n_head=2, vocab_size=257, n_positions=64)
    m = Gpt2Model(synth.gpt2_weights(cfg, base_seed=77, std=0.08, random_ln=True), cfg, reg)
    prompts = synth.token_ids(5, (2, 9), cfg.vocab_size)
    s = DecodeSession(m, batch=2, capacity=40)

    def run():
        s.prefill(prompts)
        s.step(6)
        return s.tokens(), s.logits()
    good = run()
    reg.set_tuning("persist_wait_kcycles", 2000)  # about a millisecond of SM clocks
    reg.set_tuning("few_fault_layer", 1)
    try:
        with pytest.raises(b200nn.NnError) as e:
            run()
        assert e.value.code == b200nn.ERR_DEVICE and reg.device_error() == 0
    finally:
        reg.set_tuning("few_fault_layer", -1)
        reg.set_tuning("persist_wait_kcycles", 0)
    again = run()  # a new prompt starts the exchanged words over
    assert np.array_equal(again[0], good[0]) and np.array_equal(again[1], good[1]) and reg.device_error() == 0


def test_steps_given_up_are_reported_until_the_session_starts_over(reg):
    """Words that were published and not taken back must not pass for later values, whoever else has met the error."""
    cfg = Gpt2Config(n_layer=3, n_embd=128, n_head=2, vocab_size=257, n_positions=64)
    m = Gpt2Model(synth.gpt2_weights(cfg, base_seed=77, std=0.08, random_ln=True), cfg, reg)
    prompts = synth.token_ids(5, (2, 9), cfg.vocab_size)
    reg.set_tuning("few", 1)
    s, other = (DecodeSession(m, batch=2, capacity=40) for _ in range(2))

    def read(x):
        return x.tokens(), x.logits()

    def given_up(x):
        with pytest.raises(b200nn.NnError) as e:
            x.tokens()
        return e.value.code == b200nn.ERR_DEVICE

    s.prefill(prompts)
    s.step(6)
    good = read(s)
    other.prefill(prompts)
    for layer in (0, 1, 2):
        s.prefill(prompts)
        reg.set_tuning("persist_wait_kcycles", 2000)  # about a millisecond of SM clocks
        reg.set_tuning("few_fault_layer", layer)
        try:
            s.step(6)
        finally:
            reg.set_tuning("few_fault_layer", -1)
            reg.set_tuning("persist_wait_kcycles", 0)
        other.step(6)  # behind the error, which is not its own
        assert given_up(other)  # the context's error word goes to whoever asks first
        assert all(np.array_equal(a, b) for a, b in zip(read(other), good))
        assert given_up(s) and given_up(s)  # kept although the context's word has been cleared
        s.step(1)  # refused by the kernel
        assert given_up(s)
        s.rewind(9)
        s.step(6)  # the prompt's pick is still in place: what was given up has stored nothing
        assert all(np.array_equal(a, b) for a, b in zip(read(s), good)) and reg.device_error() == 0
        other.prefill(prompts)


# one layer less than the rule asks for, and as many; narrower than any; a vocabulary that asks for twice the layers
@pytest.mark.parametrize("family,d,layers,vocab,one", [
    ("f32", 512, 6, 300, True), ("f32", 512, 5, 300, False), ("f32", 448, 12, 300, False), ("int4", 512, 11, 300, False), ("int4", 512, 12, 300, True),
    ("int4", 640, 6, 300, True), ("f32", 512, 11, 131072, False), ("f32", 512, 12, 131072, True)])
def test_steps_in_one_kernel_only_where_they_are_faster(reg, family, d, layers, vocab, one):
    cfg = Gpt2Config(n_layer=layers, n_embd=d, n_head=d // 64, vocab_size=vocab, n_positions=64)
    w = synth.gpt2_weights(cfg, base_seed=1, std=0.05)
    m = Gpt2Model(w, cfg, reg) if family == "f32" else Int4Gpt2Model(w, cfg, reg, flags=b200nn.QUANT_LM_HEAD, group_size=64)
    prompts = synth.token_ids(2, (1, 5), vocab)
    default = _steps(reg, m, prompts, 10, -1)
    assert (default[2] == 1) is one
    forced = _steps(reg, m, prompts, 10, 1)
    assert forced[2] == 1 and np.array_equal(forced[0], default[0]) and np.abs(forced[1] - default[1]).max() < 1e-3


@pytest.mark.parametrize("layers,steps", [(3, 32), (48, 6), (400, 1)])
def test_a_launch_takes_no_more_steps_than_about_five_milliseconds(reg, layers, steps):
    cfg = Gpt2Config(n_layer=layers, n_embd=64, n_head=1, vocab_size=99, n_positions=128)
    m = Gpt2Model(synth.gpt2_weights(cfg, base_seed=1, std=0.05), cfg, reg)
    prompts = synth.token_ids(2, (1, 5), 99)
    tok, lg, launches = _steps(reg, m, prompts, 2 * steps + 3, 1)  # two steps are not counted
    assert launches == 3 and reg.device_error() == 0
    tok_o, lg_o, _ = _steps(reg, m, prompts, 2 * steps + 3, 0)
    assert np.array_equal(tok, tok_o) and np.abs(lg - lg_o).max() < 1e-3


# contexts around 1000 with as few splits as the widths leave (f32, four sequences: three, 340 rows a block; int4, two: two, 512),
# several turns of 120 rows each; the cache's last position
@pytest.mark.parametrize("family,d,layers,B,P,N,group", [("f32", 768, 2, 4, 1010, 14, 0), ("int4", 1600, 2, 2, 955, 12, 128), ("f32", 1024, 1, 1, 1000, 8, 0),
                                                         ("int4", 768, 2, 1, 480, 6, 128)])
def test_steps_in_one_kernel_with_long_contexts(reg, family, d, layers, B, P, N, group):
    cfg = Gpt2Config(n_layer=layers, n_embd=d, n_head=d // 64, vocab_size=1031, n_positions=1024)
    w = synth.gpt2_weights(cfg, base_seed=90 + d, std=0.02, random_ln=True)
    m = Gpt2Model(w, cfg, reg) if family == "f32" else Int4Gpt2Model(w, cfg, reg, flags=b200nn.QUANT_LM_HEAD, group_size=group)
    prompts = synth.token_ids(d + B, (B, P), 1031)
    tok, lg, launches = _steps(reg, m, prompts, N, 1)
    tok_o, lg_o, launches_o = _steps(reg, m, prompts, N, 0)
    assert reg.device_error() == 0 and launches == 1 and launches_o > layers
    same = (tok == tok_o).all(axis=1)
    assert same.sum() >= B - 1  # a near-tie may turn a pick
    assert np.abs(lg - lg_o)[same].max() < 1e-3


def test_a_session_turns_to_steps_in_one_kernel_and_back(reg):
    """A narrow model's session prepares nothing until it is asked to; each way goes on where the other has stopped."""
    cfg = Gpt2Config(n_layer=2, n_embd=128, n_head=2, vocab_size=257, n_positions=64)
    m = Gpt2Model(synth.gpt2_weights(cfg, base_seed=8, std=0.08, random_ln=True), cfg, reg)
    prompts = synth.token_ids(6, (2, 9), cfg.vocab_size)

    def run(ways):
        try:
            reg.set_tuning("few", ways[0])
            s = DecodeSession(m, batch=2, capacity=60)
            s.prefill(prompts)
            for few in ways:
                reg.set_tuning("few", few)
                launches = reg.launch_count()
                s.step(3)
                assert (reg.launch_count() - launches == 1) is (few == 1)
            return s.tokens(), s.logits()
        finally:
            reg.set_tuning("few", 1)
    a, b = run((-1, 1, 0, 1, -1, 1, 1)), run((0,) * 7)
    assert np.array_equal(a[0], b[0]) and np.abs(a[1] - b[1]).max() < 1e-3 and reg.device_error() == 0
