"""Parts that make much of a last bit (recurrences, routed experts) inside the engine's steps: which forms of the
kernels a step takes."""

import pytest
import torch

import besorax_cases
import gegorax_cases
import karupel_cases
import plain_karupel
import vavupel_cases

pytestmark = pytest.mark.gpu

MODELS = {"karupel": (karupel_cases.MIXED, plain_karupel.random_weights),
          "vavupel": (vavupel_cases.MIXED, vavupel_cases.random_weights),
          "gegorax": (gegorax_cases.MIXED, gegorax_cases.random_weights)}


@pytest.mark.parametrize("name", sorted(MODELS))
def test_long_prompts_walk_token_by_token_unless_asked_otherwise(name, monkeypatch):
    """The recurrences in chunks are further from 64 bits than those token by token (1.3e-7 to 1.7e-7 against
    0.9e-7), so an engine takes them only where its owner says so: by default every bit is as without them."""
    from strata_inference_b200 import Engine, spec_from_config
    from strata_inference_b200.kernels import native
    cfg, weights_of = MODELS[name]
    weights, tokens = weights_of(cfg, seed=7), [(17 * i + 5) % cfg["vocab"] for i in range(300)]
    native.library()

    def logits(chunked):
        eng = Engine(spec_from_config(cfg)[1], weights, dtype="float32", max_tokens=1024, max_seq_len=512)
        if chunked is not None:
            eng.rt.chunked_scans = chunked
        return eng.step([(eng.new_sequence(), tokens)], [list(range(len(tokens)))])

    got, asked = logits(None), logits(True)
    monkeypatch.setattr(native, "CHUNKED_SCAN_MIN_ROWS", 1 << 30)
    want = logits(True)
    assert torch.equal(got, want)
    assert not torch.equal(asked, want)
    assert (asked - want).abs().max() <= 1e-4 * want.abs().max()


ATTENTION = karupel_cases.attention(4, 2, 64, 64, scale=0.125, ff=128)
DECODED = {
    # (layers, weights, whether its attention shares blocks out by the rows' lengths)
    "attention alone": (karupel_cases.model(64, 200, [ATTENTION]), plain_karupel.random_weights, True),
    "beside a recurrence": (karupel_cases.model(64, 200, [ATTENTION, karupel_cases.delta(2, 1, 32, 32, 4)]),
                            plain_karupel.random_weights, False),
    "in chunks": (besorax_cases.model(64, 200, [besorax_cases.attention(4, 2, 64, 64, 5000, mlp=besorax_cases.dense(64))]),
                  besorax_cases.random_weights, True),
    "ahead of routed experts": (besorax_cases.model(64, 200, [
        besorax_cases.attention(4, 2, 64, 64, 0, mlp=besorax_cases.moe(4, 2, 32))]), besorax_cases.random_weights, False),
}


@pytest.mark.parametrize("name", sorted(DECODED))
def test_parts_that_make_much_of_a_last_bit_keep_the_order_of_sums(name, monkeypatch):
    """40 sequences of 100 to 1 100 tokens: a model with such parts gives a sequence the same bits whatever the
    others' lengths are; other models' blocks are shared out by the lengths."""
    from strata_inference_b200 import Engine, spec_from_config
    from strata_inference_b200.kernels import native
    cfg, weights_of, shares = DECODED[name]
    native.library()
    slots, plain = [], native.attention_decode
    monkeypatch.setattr(native, "attention_decode", lambda *a, **kw: (slots.append(kw.get("slots", 0)), plain(*a, **kw))[1])
    weights = weights_of(cfg, seed=5)
    logits = []
    for short in (100, 700):
        eng = Engine(spec_from_config(cfg)[1], weights, dtype="bfloat16", max_tokens=65536, max_seq_len=1536)
        seqs = [eng.new_sequence() for _ in range(40)]
        lens = [1100] + [short] * 19 + [900] * 20
        for s, n in zip(seqs, lens):
            eng.step([(s, [(7 * s + 3 * i) % 200 for i in range(n)])])
        eng.decode_step(seqs, [11] * 40)
        logits.append(eng.last_logits[20:].float().clone())
    assert slots and all((n > 0) == shares for n in slots), slots
    if not shares:
        assert torch.equal(*logits)
