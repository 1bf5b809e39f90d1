"""Rows that are handed on whole (up to 1024 logits, no threshold): the survivor stage's lists cut them by ranges of a fixed width.
Logits whose spread is a fraction of a range, a few ranges or far beyond the last, ties, masked entries --
token ids, survivor counts and statuses as the checker's, log-probs within 1e-5."""
import numpy as np
import pytest

import gpu_harness as gh
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab", [1, 2, 33, 300, 511, 513, 700, 1017, 1024])
@pytest.mark.parametrize("settings", [
    dict(top_k=1), dict(top_k=20, top_p=0.9, temperature=0.7), dict(top_k=200, min_p=0.001), dict(top_k=513), dict(top_p=0.95), dict(top_p=0.4, temperature=3.0),
    dict(top_p=0.9, min_p=0.02, repetition_penalty=0.8), dict(min_p=0.1, temperature=0.2),
], ids=str)
def test_rows_handed_on_whole(vocab, settings):
    rng = np.random.RandomState(vocab)
    logits = rng.randn(10, vocab) * 3.0
    logits[1] *= 0.01                       # all in one range
    logits[2] *= 100.0                      # most beyond the last
    logits[3] = np.round(logits[3])
    logits[4] = 0.25
    logits[5, rng.rand(vocab) < 0.9] = -1e9
    logits[6, rng.randint(vocab)] = 60.0
    logits[7] -= 1000.0
    logits[8] = -np.abs(logits[8]) * 1e4
    logits[9, -1] = logits[9].max()
    hist = rng.randint(0, vocab, size=(10, 12)).astype(np.int64)
    eos = [int(logits[0].argmax()), vocab // 2]
    for extra in (dict(), dict(min_new_tokens=1, eos_token_ids=eos)):
        if vocab <= 2 and extra:
            continue
        cfg = ol.make_config(max_new_tokens=2, do_sample=True, **settings, **extra)
        gh.check_rows_against_oracle(logits.astype(np.float32), hist, np.arange(11, dtype=np.int64) * 12, cfg, np.arange(10, dtype=np.uint64) + vocab)


@pytest.mark.parametrize("vocab", [1, 2, 33, 700, 1024, 1025, 20000])
@pytest.mark.parametrize("settings", [dict(top_k=30), dict(top_p=0.9), dict(min_p=0.1)], ids=str)
def test_quotients_that_overflow_on_lists(vocab, settings):
    # T = 1e-36: below -340 a quotient is -inf and the token removed, alone or with all the others
    if settings.get("top_k", 0) >= vocab:
        settings = dict(top_p=0.5)
    rng = np.random.RandomState(vocab)
    logits = rng.randn(5, vocab) * 3.0
    logits[1] -= 1000.0
    logits[2, ::3] = -1000.0
    logits[3] = -400.0
    logits[4] *= 20.0  # (up to 300: 3e38 after the divide, still a float)
    hist = np.zeros((5, 1), dtype=np.int64)
    cfg = ol.make_config(max_new_tokens=1, do_sample=True, temperature=1e-36, **settings)
    (_, _, status, _), _ = gh.check_rows_against_oracle(logits.astype(np.float32), hist, np.arange(6, dtype=np.int64), cfg,
                                                        np.arange(5, dtype=np.uint64), expect_ok=False)
    assert status[1] == status[3] == 5 and status[0] == 0
