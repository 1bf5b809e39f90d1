"""Rows that the survivor stage's lists held only after a look at what they are made of.

Rows that are handed on whole (up to 1024 logits, no threshold): the survivor stage's lists cut them by ranges of a fixed width.
Logits whose spread is a fraction of a range, a few ranges or far beyond the last, ties, masked entries --
token ids, survivor counts and statuses as the checker's, log-probs within 1e-5.  Rows masked by a number: whole parts of them are equal."""
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


@pytest.mark.parametrize("rows,vocab", [(1, 50000), (3, 128256), (40, 151936)])
@pytest.mark.parametrize("settings", [
    dict(do_sample=False), dict(top_k=1), dict(top_k=5, temperature=0.8, top_p=0.9), dict(top_p=0.95), dict(min_p=0.05, temperature=1.5),
    dict(top_p=0.9, temperature=1000.0),  # (at 1e7 a token of probability exp(-65504) is drawn, whose log-probability is -inf on both sides)
], ids=str)
def test_rows_masked_by_a_number(rows, vocab, settings):
    rng = np.random.RandomState(vocab)
    logits = rng.randn(rows, vocab) * 2.5
    for r in range(rows):
        mask = np.ones(vocab, dtype=bool)
        mask[rng.randint(vocab, size=rng.choice([1, 7, 60]))] = False
        logits[r, mask] = [-1e9, -65504.0, -200.0][r % 3]
    hist = rng.randint(0, vocab, size=(rows, 8)).astype(np.int64)
    for penalty in (1.0, 1.3, 0.7):
        cfg = ol.make_config(max_new_tokens=1, **{"do_sample": True, "repetition_penalty": penalty, **settings})
        gh.check_rows_against_oracle(logits.astype(np.float32), hist, np.arange(rows + 1, dtype=np.int64) * 8, cfg, np.arange(rows, dtype=np.uint64))


@pytest.mark.parametrize("settings", [dict(do_sample=False), dict(do_sample=True, top_k=1)], ids=str)
def test_a_masked_row_takes_no_longer_than_others(settings):
    # (7 and 33 times as long when the parts without a live logit left their lists)
    import torch
    plain = torch.randn((1, 50000), device="cuda")
    masked = torch.full_like(plain, -1e9)
    masked[0, :50] = plain[0, :50]
    uniforms, config = torch.rand(1, dtype=torch.float64, device="cuda"), gh.psx_config(ol.make_config(max_new_tokens=1, **settings))

    def best(x):
        out, times = gh.ctx().alloc_outputs(1), []
        for _ in range(30):
            begin, end = torch.cuda.Event(True), torch.cuda.Event(True)
            begin.record()
            gh.ctx().sample_rows(x, None, None, config, uniforms, out=out)
            end.record()
            end.synchronize()
            times.append(begin.elapsed_time(end))
        return min(times)

    assert best(masked) < 3 * best(plain)


@pytest.mark.parametrize("rows,vocab", [(1, 50000), (20, 151936)])
@pytest.mark.parametrize("k", [100, 180, 200, 256])
def test_more_candidates_than_2048_at_the_threshold(rows, vocab, k):
    # (a k of some 200 from every part)
    logits, hist = ol.synth_rows(np.arange(rows) + k, vocab, 2.5, 0.0, 20)
    logits[0] = np.round(logits[0] * 8) / 8
    for settings in (dict(), dict(top_p=0.9, temperature=0.7, repetition_penalty=1.2)):
        cfg = ol.make_config(max_new_tokens=1, do_sample=True, top_k=k, **settings)
        gh.check_rows_against_oracle(logits, hist, np.arange(rows + 1, dtype=np.int64) * 20, cfg, np.arange(rows, dtype=np.uint64))
