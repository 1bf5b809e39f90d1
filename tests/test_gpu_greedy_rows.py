"""Greedy decoding of more rows than the survivor stage has blocks for: a warp decides a row, and what it cannot is left to its block.

Row counts around the line and off a multiple of the blocks; lists longer than a warp's look; ties at the maximum, rows masked by a number
(their parts' lists overflow), constant rows, failed rows between good ones, EOS bans, penalties on either side of one."""
import numpy as np
import pytest

import gpu_harness as gh
import oracle_lib as ol
import pulsatrix_b200 as psx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,vocab", [(444, 1025), (445, 1025), (451, 1024), (453, 5003), (460, 20011), (450, 49152), (450, 65536),
                                        (450, 65537), (447, 131072), (449, 131073)])
@pytest.mark.parametrize("settings", [dict(), dict(repetition_penalty=1.3), dict(repetition_penalty=0.7, min_new_tokens=1)], ids=str)
def test_a_warp_per_row(rows, vocab, settings):
    if vocab > 100000:
        base = np.random.RandomState(7).randn(16, vocab).astype(np.float32) * 3
        logits = base[np.arange(rows) % 16]
    else:
        logits = np.random.RandomState(rows).randn(rows, vocab).astype(np.float32) * 3
    rng = np.random.RandomState(rows + 1)
    logits[3] = 0.25                                                  # constant
    logits[9, rng.rand(vocab) < 0.99] = -1e9                          # masked by a number
    logits[17, rng.randint(0, vocab, 200)] = logits[17].max()         # ties at the maximum
    logits[18] = np.round(logits[18])
    logits[rows - 1, rng.randint(0, vocab, 40)] = logits[rows - 1].max() + 1.0
    hist = rng.randint(0, vocab, size=(rows, 12)).astype(np.int64)
    hist[17, :4] = np.argsort(-logits[17])[:4]
    extra = dict(eos_token_ids=[int(logits[0].argmax()), vocab // 2]) if "min_new_tokens" in settings else {}
    cfg = ol.make_config(max_new_tokens=2, do_sample=False, **settings, **extra)
    gh.check_rows_against_oracle(logits, hist, np.arange(rows + 1, dtype=np.int64) * 12, cfg, np.arange(rows, dtype=np.uint64))


def test_failed_rows_among_many():
    rows, vocab = 470, 3001
    logits = np.random.RandomState(1).randn(rows, vocab).astype(np.float32)
    logits[5, 77] = np.nan
    logits[6, 0] = -np.inf
    logits[300, vocab - 1] = np.inf
    hist = np.zeros((rows, 1), dtype=np.int64)
    cfg = ol.make_config(max_new_tokens=1, do_sample=False)
    (_, _, status, _), _ = gh.check_rows_against_oracle(logits, hist, np.arange(rows + 1, dtype=np.int64), cfg, np.arange(rows, dtype=np.uint64),
                                                        expect_ok=False)
    assert np.nonzero(status)[0].tolist() == [5, 6, 300] and (status[[5, 6, 300]] == psx.ROW_NON_FINITE).all()


@pytest.mark.parametrize("vocab", [1500, 2048, 20003])
@pytest.mark.parametrize("settings", [dict(), dict(repetition_penalty=1.3), dict(repetition_penalty=0.7, min_new_tokens=1)], ids=str)
def test_rows_that_no_list_holds(vocab, settings):
    """Constant rows next to one another, every third row and the last ones: the first column of the maximum, whatever the history and the ban name."""
    rows = 900
    rng = np.random.RandomState(vocab)
    logits = rng.randn(rows, vocab).astype(np.float32)
    constant = np.zeros(rows, dtype=bool)
    constant[100:240] = constant[rows - 70:] = True
    constant[400:700:3] = True
    logits[constant] = np.float32(2.0)
    logits[110] = -1.0                                                       # a penalty below one lifts what the history names
    logits[111] = np.where(np.arange(vocab) % 2 == 0, np.float32(-0.0), np.float32(0.0))
    logits[112, 1:] = -3.0                                                   # the maximum is in the history: not the maximum any more
    logits[113, vocab - 1] = np.nan
    logits[rows - 1, 7] = np.inf
    hist = rng.randint(0, vocab, size=(rows, 9)).astype(np.int64)
    hist[100:240:2, :3] = [0, 1, 2]
    hist[112, 0] = 0
    extra = dict(eos_token_ids=[0, 3]) if "min_new_tokens" in settings else {}
    cfg = ol.make_config(max_new_tokens=2, do_sample=False, **settings, **extra)
    (_, _, status, _), _ = gh.check_rows_against_oracle(logits, hist, np.arange(rows + 1, dtype=np.int64) * 9, cfg,
                                                        np.arange(rows, dtype=np.uint64), expect_ok=False)
    assert np.nonzero(status)[0].tolist() == [113, rows - 1]
