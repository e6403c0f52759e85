"""Recurrent layers inside the engine's steps: which form of a recurrence a step takes."""

import pytest
import torch

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
