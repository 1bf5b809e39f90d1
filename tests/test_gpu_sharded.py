"""The vocabulary-sharded entry points on one GPU: the eight column shards of workload C5 are
scanned one after another into the buffer an all-gather would fill, then merged; the result must
equal the reference fixture (and therefore the unsharded path) bit for bit.  The collective itself
is covered by tests/test_sharding_cpu.py (gloo) and by the multi-GPU benchmark."""
from pathlib import Path

import numpy as np
import pytest

import gpu_harness as gh
import oracle_lib as ol
import pulsatrix_b200 as psx
import workload_rows
from pulsatrix_b200.sharded import gathered_layout, row_bounds, shard_bounds
from pulsatrix_b200.workloads import WORKLOADS

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"


def run_sharded(logits, hist_flat, offsets, cfg, uniforms, world, merge_blocks=1):
    """merge_blocks > 1: the rows are decided block by block, as that many ranks would share them out."""
    import torch
    rows, vocab = logits.shape
    ctx = gh.ctx()
    config = gh.psx_config(cfg)
    record = ctx.shard_record_bytes(config)
    layout, per = gathered_layout(rows, record, world)
    gathered = torch.zeros(world * per, dtype=torch.uint8, device="cuda")
    d_logits = torch.from_numpy(logits).cuda()
    d_hist = torch.from_numpy(hist_flat).cuda()
    d_off = torch.from_numpy(offsets).cuda()
    for s in range(world):
        begin, cols = shard_bounds(vocab, world, s)
        shard = d_logits[:, begin: begin + cols]  # a strided view: row stride stays the full vocabulary
        ctx.shard_scan(shard, begin, vocab, d_hist, d_off, config, gathered[layout[s]: layout[s] + per])
    d_u = torch.from_numpy(uniforms).cuda() if uniforms is not None else None
    if merge_blocks == 1:
        out = ctx.shard_merge(gathered, world, rows, vocab, config, d_u)
        torch.cuda.synchronize()
        return out["tokens"].cpu().numpy(), out["log_probs"].cpu().numpy(), out["status"].cpu().numpy()
    pieces = []
    for b in range(merge_blocks):
        begin, count, _ = row_bounds(rows, merge_blocks, b)
        if count == 0:
            continue
        out = ctx.shard_merge(gathered, world, rows, vocab, config, d_u, row_begin=begin, row_count=count)
        torch.cuda.synchronize()
        pieces.append([out[k].cpu().numpy() for k in ("tokens", "log_probs", "status")])
    return tuple(np.concatenate([p[i] for p in pieces]) for i in range(3))


def test_c5_in_eight_shards_matches_the_reference_fixture():
    w = WORKLOADS["c5"]
    gold = np.load(GOLDEN / "workload_c5.npz")
    cfg = workload_rows.config_of(w)
    ids = np.arange(0, 96)
    logits, hist, offsets, seeds = workload_rows.build("c5", ids)
    tokens, logp, status = run_sharded(logits, hist.ravel(), offsets, cfg, psx.uniforms_mt19937_64(seeds), w.shards)
    assert (status == 0).all(), status
    assert tokens.tolist() == gold["token"][ids].tolist()
    assert (np.abs(logp - gold["log_prob"][ids]) <= 1e-5 * np.abs(gold["log_prob"][ids]) + 1e-9).all()


def test_rows_shared_out_among_the_ranks_give_the_same_answers():
    w = WORKLOADS["c5"]
    gold = np.load(GOLDEN / "workload_c5.npz")
    ids = np.arange(96, 133)  # 37 rows in 8 blocks: the last blocks are short or empty
    logits, hist, offsets, seeds = workload_rows.build("c5", ids)
    tokens, logp, status = run_sharded(logits, hist.ravel(), offsets, workload_rows.config_of(w),
                                       psx.uniforms_mt19937_64(seeds), w.shards, merge_blocks=8)
    assert (status == 0).all() and tokens.tolist() == gold["token"][ids].tolist()
    assert (np.abs(logp - gold["log_prob"][ids]) <= 1e-5 * np.abs(gold["log_prob"][ids]) + 1e-9).all()


@pytest.mark.parametrize("world", [2, 3, 8])
def test_sharded_equals_unsharded_for_greedy_and_top_k(world):
    rng = np.random.RandomState(world)
    rows, vocab, hlen = 24, 50000, 100
    logits = (rng.randn(rows, vocab) * 3).astype(np.float32)
    logits[5, [11, 20000, 49999]] = logits[5].max() + 2.0  # ties across shards: lowest column wins
    hist = rng.randint(0, vocab, size=(rows, hlen)).astype(np.int64)
    offsets = np.arange(rows + 1, dtype=np.int64) * hlen
    seeds = np.arange(rows, dtype=np.uint64) + 100
    u = psx.uniforms_mt19937_64(seeds)
    for cfg in (ol.make_config(max_new_tokens=1, repetition_penalty=1.3),
                ol.make_config(max_new_tokens=1, do_sample=True, top_k=40, top_p=0.9, temperature=0.8,
                               repetition_penalty=1.1)):
        want = ol.rows("oracle", logits, hist.ravel(), offsets, cfg, seeds)
        tokens, logp, status = run_sharded(logits, hist.ravel(), offsets, cfg, u, world)
        assert (status == 0).all()
        assert tokens.tolist() == want["token"].tolist()
        assert (np.abs(logp - want["log_prob"]) <= 1e-5 * np.abs(want["log_prob"]) + 1e-9).all()


def test_a_shard_scan_may_be_the_first_call_of_a_process():
    """The kernels' shared-memory limits are lifted by whichever entry point runs first: a fresh
    process whose first call is psx_b200_shard_scan must work like any other."""
    import subprocess
    import sys
    done = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-p", "no:cacheprovider",
                           f"{Path(__file__).resolve()}::test_c5_in_eight_shards_matches_the_reference_fixture"],
                          capture_output=True, text=True, timeout=600)
    assert done.returncode == 0, done.stdout[-2000:] + done.stderr[-2000:]


@pytest.mark.parametrize("world", [2, 4, 5, 8, 9])
@pytest.mark.parametrize("rows", [444, 445, 450])
def test_many_greedy_rows_over_few_shards(world, rows):
    """More rows than the survivor stage has blocks for, records of 64 slots; a record that overflows is reported, as it is with fewer rows."""
    rng = np.random.RandomState(rows + world)
    vocab = 6000
    logits = (rng.randn(rows, vocab) * 3).astype(np.float32)
    logits[5, [11, 3000, 5999]] = logits[5].max() + 2.0  # ties across shards: lowest column wins
    logits[rows - 1, [4500, 100]] = logits[rows - 1].max() + 1.0
    logits[200:212] = 1.0                                # constant: no record holds their ties
    logits[300, 5000] = np.nan
    hist = rng.randint(0, vocab, size=(rows, 10)).astype(np.int64)
    offsets = np.arange(rows + 1, dtype=np.int64) * 10
    seeds = np.arange(rows, dtype=np.uint64)
    cfg = ol.make_config(max_new_tokens=1, repetition_penalty=1.3)
    want = ol.rows("oracle", logits, hist.ravel(), offsets, cfg, seeds)
    tokens, logp, status = run_sharded(logits, hist.ravel(), offsets, cfg, None, world)
    few_tokens, few_logp, few_status = run_sharded(logits, hist.ravel(), offsets, cfg, None, world, merge_blocks=3)
    assert (tokens == few_tokens).all() and (status == few_status).all() and np.abs(logp - few_logp).max() <= 1e-6
    ok = np.ones(rows, dtype=bool)
    ok[200:212] = ok[300] = False
    assert (status[ok] == 0).all() and status[300] == psx.ROW_NON_FINITE and (status[200:212] == psx.ROW_TOO_WIDE).all()
    assert tokens[ok].tolist() == want["token"][ok].tolist()
    assert (np.abs(logp[ok] - want["log_prob"][ok]) <= 1e-5 * np.abs(want["log_prob"][ok]) + 1e-9).all()
