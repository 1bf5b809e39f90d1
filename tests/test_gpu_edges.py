"""The sizes at which the kernels change their way: the widest row of each softmax kernel, rows off the 16-byte boundary, the
slices and the k of each top_k kernel with ties at the cut, sliding windows that leave most of a cache unread, and the
survivor stage's lists when they are full, empty of decisions or one entry long."""
import numpy as np
import pytest

import gpu_harness as gh
import oracle_lib as ol
import test_gpu_decode_attention as attention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [1, 127, 129, 253, 257, 509, 1021, 1024, 1025, 2045, 4096, 4099, 8189, 8192, 16381, 16387, 32765, 32769, 131072, 131073])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_softmax_and_logsumexp_at_the_edges_of_their_kernels(cols, shift):
    import torch
    rows = 5
    gen = torch.Generator(device="cuda")
    gen.manual_seed(cols * 4 + shift)
    flat = torch.full((rows * cols + 8,), float("nan"), device="cuda")
    x = flat[shift: shift + rows * cols].view(rows, cols)
    x.copy_(torch.randn((rows, cols), generator=gen, device="cuda") * 3.0)
    want = torch.softmax(x.double(), dim=1)
    # exp of a difference d by one float ex2 of d * log2(e): |d| <= 30 here, the rounded exponent is off by 43 * 2^-24 at most, ex2 by
    # 2^-22, the sum and the quotient by a few 2^-24: 4e-6 in all
    for out in (torch.empty_like(x), None):  # (out of its own allocation: another offset from the boundary when shift is odd)
        got = gh.ctx().softmax_rows(x, out=out) if out is not None else gh.ctx().softmax_rows(x)
        assert ((got.double() - want).abs() / want).max().item() < 4e-6
    before = flat[:shift].clone(), flat[shift + rows * cols:].clone()
    inside = x.clone()
    gh.ctx().softmax_rows(x, out=x)
    assert ((x.double() - want).abs() / want).max().item() < 4e-6
    assert flat[:shift].isnan().all() and flat[shift + rows * cols:].isnan().all() and before[0].isnan().all() and before[1].isnan().all()
    lse = gh.ctx().logsumexp_rows(inside).double()
    assert (lse - torch.logsumexp(inside.double(), dim=1)).abs().max().item() < 4e-6 * 20  # (values up to 20)


@pytest.mark.parametrize("cols", [33, 2047, 4096, 4097, 16383, 16384, 16385, 32769, 65536, 131072, 131077])
@pytest.mark.parametrize("k", [1, 2, 31, 33, 64, 65, 128, 129, 256, 257])
def test_top_k_at_the_edges_of_its_kernels(cols, k):
    import torch
    if k > cols:
        pytest.skip("k exceeds the row")
    rng = np.random.RandomState(cols + k)
    for shift, largest in ((0, True), (1, False)):
        x = rng.randn(6, cols).astype(np.float32)
        x[1] = np.round(x[1] * 4) / 4          # a few dozen values only: ties at every cut
        x[2, : cols // 2] = x[2, cols // 2: 2 * (cols // 2)]  # every value twice
        x[3, rng.randint(cols, size=3)] = np.nan
        x[4] = 0.5
        flat = torch.zeros(x.size + 4, device="cuda")
        view = flat[shift: shift + x.size].view(*x.shape)
        view.copy_(torch.from_numpy(x))
        values, indices = (t.cpu().numpy() for t in gh.ctx().top_k_rows(view, k, largest=largest))
        want_values, want_indices = ol.top_k_rows("oracle", x, k, largest)
        assert (indices == want_indices).all()
        assert ((values == want_values) | (np.isnan(values) & np.isnan(want_values))).all()


@pytest.mark.parametrize("d,window,cached,q_len", [(64, 1, 500, 1), (128, 31, 700, 1), (100, 257, 3000, 2), (256, 33, 900, 1), (132, 600, 1500, 2), (64, 2000, 900, 1)])
@pytest.mark.parametrize("padding", [False, True])
def test_sliding_windows_over_long_caches(d, window, cached, q_len, padding):
    attention._case(batch=3, heads=4, kv_heads=2, q_len=q_len, d=d, cached=cached, max_len=cached + q_len + 3, seed=d + window,
                    window=window, padding=padding)


def _check(logits, seed, **settings):
    rows = logits.shape[0]
    hist = np.random.RandomState(seed).randint(0, logits.shape[1], size=(rows, 20)).astype(np.int64)
    gh.check_rows_against_oracle(logits.astype(np.float32), hist, np.arange(rows + 1, dtype=np.int64) * 20, ol.make_config(max_new_tokens=1, **settings),
                                 np.arange(rows, dtype=np.uint64) + seed)


@pytest.mark.parametrize("vocab", [1025, 20000, 50021, 128256])
@pytest.mark.parametrize("settings", [
    dict(top_k=1), dict(top_k=2, top_p=0.01), dict(top_k=64, temperature=0.3), dict(top_k=65, top_p=0.99, min_p=0.001), dict(top_k=256, top_p=0.5),
    dict(top_p=0.3), dict(top_p=0.95, temperature=1.7), dict(top_p=0.9, min_p=0.01, repetition_penalty=0.9), dict(min_p=0.05), dict(min_p=0.9),
], ids=str)
def test_lists_of_every_length(vocab, settings):
    rng = np.random.RandomState(vocab)
    logits = rng.randn(9, vocab) * 3.0
    logits[1] *= 0.2                                   # thousands of near-equal logits: more than the lists hold
    logits[2] = 0.0
    logits[2, 7:vocab:vocab // 50] = 4.0               # fifty ties at the top, nothing between them and the rest
    logits[3] = np.round(logits[3])                    # ties everywhere
    logits[4, rng.randint(vocab)] = 60.0               # one logit has it all
    logits[5, vocab // 3: vocab // 3 + 700] += 12.0    # the survivors side by side
    logits[6, -1] = logits[6].max() + 1.0              # the last column
    _check(logits, vocab, do_sample=True, **settings)
    _check(logits, vocab, do_sample=False)


@pytest.mark.parametrize("cols", [1, 3, 126, 128, 254, 512, 1021, 1023, 1025, 2046, 4093, 4096, 8187, 8189, 8192])
@pytest.mark.parametrize("shift,out_shift", [(0, 1), (0, 2), (1, 0), (2, 1), (3, 2), (1, 3)])
def test_softmax_into_a_buffer_that_lies_differently(cols, shift, out_shift):
    import torch
    rows = 19
    gen = torch.Generator(device="cuda")
    gen.manual_seed(cols * 16 + shift * 4 + out_shift)
    x = torch.randn((rows * cols + 8,), generator=gen, device="cuda")[shift: shift + rows * cols].view(rows, cols)
    flat = torch.full((rows * cols + 8,), float("nan"), device="cuda")
    out = flat[out_shift: out_shift + rows * cols].view(rows, cols)
    gh.ctx().softmax_rows(x, out=out)
    want = torch.softmax(x.double(), dim=1)
    assert ((out.double() - want).abs() / want).max().item() < 4e-6  # (as above)
    assert flat[:out_shift].isnan().all() and flat[out_shift + rows * cols:].isnan().all()


def test_a_narrow_softmax_into_a_buffer_that_lies_differently_takes_a_warp_per_row():
    # 512 threads for a row of 128 columns took 34 times as long as a warp does; a scalar write in place of a vector 1.5 times
    import torch
    x = torch.randn((65536 * 128 + 4,), device="cuda")
    like, other = x[:-4].view(65536, 128), x[1:-3].view(65536, 128)
    out = torch.empty_like(like)

    def best(source):
        times = []
        for _ in range(20):
            begin, end = torch.cuda.Event(True), torch.cuda.Event(True)
            begin.record()
            gh.ctx().softmax_rows(source, out=out)
            end.record()
            end.synchronize()
            times.append(begin.elapsed_time(end))
        return min(times)

    assert best(other) < 6 * best(like)


@pytest.mark.parametrize("batch", [1, 200])
@pytest.mark.parametrize("q_len,padding", [(1, False), (2, False), (2, True)])
def test_scores_of_minus_infinity_in_a_window(batch, q_len, padding):
    # Every product overflows to -inf: what the mask hides weighs more than what it shows, in the window and before it.
    import torch
    heads, kv_heads, d, cached, window = 2, 1, 64, 1500, 800
    rng = np.random.RandomState(q_len)
    total = cached + q_len
    q = np.full((batch, heads, q_len, d), 1e30, dtype=np.float32)
    keys = np.full((batch, kv_heads, total + 2, d), -1e30, dtype=np.float32)
    values = rng.randn(batch, kv_heads, total + 2, d).astype(np.float32)
    q[0, 1] = 1.0  # (a row of ordinary scores beside it)
    keep = None
    if padding:
        keep = (rng.rand(batch, total) > 0.3).astype(np.float32)
        keep[batch - 1] = 0.0
    few = slice(0, 3) if batch > 3 else slice(None)
    want = ol.decode_attention("oracle", q[few], keys[few], values[few], cached, 1.0, True, window, None if keep is None else keep[few])
    got, status = gh.ctx().decode_attention(*(torch.from_numpy(x).cuda() for x in (q, keys, values)), cached, scale=1.0, window=window,
                                            key_keep=None if keep is None else torch.from_numpy(keep).cuda())
    assert int(status[0]) == 0
    # 1500 terms, each weight and each sum rounded: 1e-4 as the other cases
    assert np.abs(got[few].cpu().numpy() - want).max() < 1e-4
