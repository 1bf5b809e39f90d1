"""Sampling with no filter (whole_rows.cu): segments of 512 columns, a run of several segments per thread of the
drawing kernel beyond 131,072 columns, rows off the 16-byte grid, everything banned in a segment.  Token ids, statuses
and survivor counts as the reference's; the distance of the draw from its bucket's edges, which both sides form from
sums over the whole row, agrees to what the reference's sequential double sums may be off by: 3 sums of `vocab` terms
of at most 1 in all, each addition rounded at 2^-53."""
import numpy as np
import pytest

import gpu_harness as gh
import oracle_lib as ol
import pulsatrix_b200 as psx

pytestmark = pytest.mark.gpu


def _run(vocab, rows, settings, **kw):
    logits, hist = ol.synth_rows(np.arange(rows) + 7 * vocab, vocab, 2.0, 0.7, 40)
    hist[:, 3] = hist[:, 5]  # an id twice
    cfg = ol.make_config(max_new_tokens=4, do_sample=True, **settings)
    (_, _, _, diag), want = gh.check_rows_against_oracle(logits, hist, np.arange(rows + 1, dtype=np.int64) * 40, cfg,
                                                         np.arange(rows, dtype=np.uint64) + vocab, **kw)
    assert np.abs(diag["draw_margin"] - want["draw_margin"]).max() <= 3 * vocab * 2.0**-53


@pytest.mark.parametrize("vocab", [1025, 1537, 4095, 4097, 20011, 131072, 131073, 262144, 300007])
@pytest.mark.parametrize("settings", [dict(), dict(temperature=0.9, repetition_penalty=1.2)], ids=["plain", "processed"])
def test_edges_of_segments(vocab, settings):
    _run(vocab, 5, settings)


def test_rows_off_the_vector_grid():
    for shift in (1, 2, 3):
        _run(5003, 6, dict(temperature=1.4, repetition_penalty=0.8), pad_columns=shift, shift=shift)


def test_many_rows_share_a_warp():
    _run(12289, 300, dict(temperature=0.7, repetition_penalty=1.1))


def test_banned_segments_and_failed_rows():
    vocab, rows = 2048, 4
    logits = np.full((rows, vocab), -3.0, dtype=np.float32)
    logits[:, 700] = 1000.0  # everything else has no mass in double precision
    logits[1, 2047] = np.inf
    cfg = ol.make_config(max_new_tokens=2, do_sample=True, min_new_tokens=1, eos_token_ids=list(range(512)))
    hist, offsets = np.zeros((rows, 1), dtype=np.int64), np.arange(rows + 1, dtype=np.int64)
    (tokens, _, status, _), _ = gh.check_rows_against_oracle(logits, hist, offsets, cfg, np.arange(rows, dtype=np.uint64), expect_ok=False)
    assert status[1] == psx.ROW_NON_FINITE and (tokens[[0, 2, 3]] == 700).all()


# The first and the last segment of a row have slots that lie outside it; none of them may weigh anything.
@pytest.mark.parametrize("vocab", [1025, 50021])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("settings", [dict(temperature=50.0), dict(temperature=100.0), dict(temperature=1000.0),
                                      dict(temperature=100.0, repetition_penalty=1.2), dict(temperature=0.05)], ids=str)
def test_slots_outside_the_row_weigh_nothing(vocab, shift, settings):
    _run(vocab, 5, settings, pad_columns=shift, shift=shift)


def test_slots_outside_the_row_beside_a_banned_maximum():
    # the last segment's largest logit is banned and lies 200 above the others: at T = 0.2 anything derived from it outweighs the row
    vocab, rows = 1500, 4
    logits, hist = ol.synth_rows(np.arange(rows) + 31, vocab, 2.0, 0.7, 4)
    logits[:, 1490] = 200.0
    cfg = ol.make_config(max_new_tokens=2, do_sample=True, temperature=0.2, min_new_tokens=1, eos_token_ids=[1490])
    (_, _, _, diag), want = gh.check_rows_against_oracle(logits, hist, np.arange(rows + 1, dtype=np.int64) * 4, cfg, np.arange(rows, dtype=np.uint64))
    assert np.abs(diag["draw_margin"] - want["draw_margin"]).max() <= 3 * vocab * 2.0**-53


def test_slots_outside_the_row_beside_a_maximum_that_690_does_not_move():
    vocab, rows = 1025, 3  # the last segment: this one column
    logits, hist = ol.synth_rows(np.arange(rows) + 5, vocab, 2.0, 0.7, 4)
    logits[:, -1] = 1e11
    for settings in (dict(), dict(temperature=0.9, repetition_penalty=1.2)):
        cfg = ol.make_config(max_new_tokens=1, do_sample=True, **settings)
        gh.check_rows_against_oracle(logits, hist, np.arange(rows + 1, dtype=np.int64) * 4, cfg, np.arange(rows, dtype=np.uint64))


@pytest.mark.parametrize("penalty", [1.0, 1.5])
def test_quotients_that_fall_to_minus_infinity_are_not_alive(penalty):
    # -1000 / 1e-36 is -inf (removed, as by the reference), the positive logits' quotients are finite
    vocab, rows = 3001, 4
    logits, hist = ol.synth_rows(np.arange(rows) + 77, vocab, 2.0, 0.7, 30)
    logits[:, ::7] = -1000.0
    logits[:, 1500] = 50.0
    hist[:, 0], hist[:, 1] = 7, 1500
    cfg = ol.make_config(max_new_tokens=1, do_sample=True, temperature=1e-36, repetition_penalty=penalty)
    _, want = gh.check_rows_against_oracle(logits, hist, np.arange(rows + 1, dtype=np.int64) * 30, cfg, np.arange(rows, dtype=np.uint64))
    assert (want["survivors"] < vocab).all()


@pytest.mark.parametrize("settings", [dict(temperature=1e-38), dict(repetition_penalty=1e-38), dict(temperature=1e-38, repetition_penalty=1.5)], ids=str)
def test_quotients_that_overflow(settings):
    # every probability of the reference is NaN: its walk ends at the last column
    vocab, rows = 3001, 4
    logits, hist = ol.synth_rows(np.arange(rows) + 78, vocab, 2.0, 0.7, 30)
    logits[:, 1500] = 6.0  # 6 / 1.5 / 1e-38 = 4e38, above the largest float (5 would give 3.33e38, below it)
    hist[:, 0] = 1500
    cfg = ol.make_config(max_new_tokens=1, do_sample=True, **settings)
    (tokens, _, _, _), _ = gh.check_rows_against_oracle(logits, hist, np.arange(rows + 1, dtype=np.int64) * 30, cfg, np.arange(rows, dtype=np.uint64))
    assert (tokens == vocab - 1).all()


def test_uniforms_outside_the_unit_interval():
    vocab = 5003
    logits, _ = ol.synth_rows(np.arange(5) + 79, vocab, 2.0, 0.7, 4)
    uniforms = np.array([-0.25, -1e300, 1.0, 7.5, np.nan])
    for settings in (dict(), dict(temperature=0.8)):
        cfg = ol.make_config(max_new_tokens=1, do_sample=True, **settings)
        tokens, _, status, _ = gh.sample_on_gpu(logits, None, None, cfg, uniforms)
        assert (status == 0).all() and tokens.tolist() == [0, 0, vocab - 1, vocab - 1, vocab - 1]
