"""Attention of the new positions over the KV cache (psx_b200_decode_attention) against the CPU restatement
of MultiHeadAttentionModule::forward_cached's core (src/multihead_attention_module.cpp:562-586), which
tests/test_oracle_pins.py pins to the compiled reference: within the reference's own CPU/GPU equivalence
tolerance, 1e-4 (tests/backend_primitive_equivalence_cases.hpp:22).  Grouped-query heads, several new
positions, causal masks with a cache offset, sliding windows, key padding, fully masked rows, caches of one
position and of thousands (several slices per head)."""
import numpy as np
import pytest

import gpu_harness as gh
import oracle_lib as ol
import pulsatrix_b200 as psx

pytestmark = pytest.mark.gpu
TOLERANCE = 1e-4


def _case(batch, heads, kv_heads, q_len, d, cached, max_len, seed, causal=True, window=0, padding=False, scale=None):
    import torch
    rng = np.random.RandomState(seed)
    q = rng.randn(batch, heads, q_len, d).astype(np.float32)
    keys = rng.randn(batch, kv_heads, max_len, d).astype(np.float32)
    values = rng.randn(batch, kv_heads, max_len, d).astype(np.float32)
    total = cached + q_len
    keys[:, :, total:] = np.nan   # what lies beyond the cached positions must never be read into a result
    values[:, :, total:] = np.nan
    keep = None
    if padding:
        keep = (rng.rand(batch, total) > 0.3).astype(np.float32)
        keep[0, :] = 0.0          # a fully masked batch entry: uniform attention, as the reference gives
    scale = float(1.0 / np.sqrt(np.float32(d))) if scale is None else scale
    want = ol.decode_attention("oracle", q, np.nan_to_num(keys), np.nan_to_num(values), cached, scale, causal, window, keep)
    got, status = gh.ctx().decode_attention(torch.from_numpy(q).cuda(), torch.from_numpy(keys).cuda(), torch.from_numpy(values).cuda(),
                                            cached, scale=scale, causal=causal, window=window,
                                            key_keep=None if keep is None else torch.from_numpy(keep).cuda())
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    got = got.cpu().numpy()
    assert np.isfinite(got).all()
    err = np.abs(got - want) / np.maximum(1.0, np.abs(want))
    assert err.max() <= TOLERANCE, (err.max(), np.unravel_index(err.argmax(), err.shape))


@pytest.mark.parametrize("cached", [0, 1, 31, 32, 33, 127, 1000, 4097])
def test_one_new_position_over_caches_of_every_length(cached):
    _case(batch=3, heads=8, kv_heads=2, q_len=1, d=64, cached=cached, max_len=cached + 5, seed=cached)


@pytest.mark.parametrize("heads,kv_heads,q_len,d", [(4, 4, 1, 128), (8, 1, 1, 64), (16, 2, 1, 128), (6, 3, 2, 32), (4, 2, 4, 96),
                                                    (2, 2, 8, 4), (12, 12, 3, 80), (4, 2, 1, 256), (8, 8, 1, 160), (2, 1, 2, 192), (8, 1, 1, 256)])
def test_head_layouts_and_several_new_positions(heads, kv_heads, q_len, d):
    _case(batch=2, heads=heads, kv_heads=kv_heads, q_len=q_len, d=d, cached=300, max_len=512, seed=heads * 100 + d)


def test_masks():
    _case(batch=2, heads=4, kv_heads=2, q_len=2, d=64, cached=500, max_len=600, seed=1, causal=True, window=64)
    _case(batch=3, heads=4, kv_heads=4, q_len=1, d=64, cached=200, max_len=256, seed=2, causal=True, padding=True)
    _case(batch=2, heads=4, kv_heads=1, q_len=2, d=32, cached=90, max_len=128, seed=3, causal=False)
    _case(batch=2, heads=2, kv_heads=2, q_len=3, d=64, cached=40, max_len=64, seed=4, causal=False, padding=True, scale=0.3)


def test_many_slices_and_many_heads():
    _case(batch=1, heads=8, kv_heads=8, q_len=1, d=128, cached=20000, max_len=20001, seed=5)    # few heads, long cache: slices
    _case(batch=40, heads=16, kv_heads=8, q_len=1, d=128, cached=700, max_len=768, seed=6)      # many heads: one slice each


def test_bad_arguments_are_refused():
    import torch
    ctx = gh.ctx()
    q = torch.zeros((1, 6, 1, 64), device="cuda")
    kv = torch.zeros((1, 4, 16, 64), device="cuda")
    with pytest.raises(psx.PsxError):   # heads not a multiple of kv_heads
        ctx.decode_attention(q, kv, kv, 3)
    q = torch.zeros((1, 4, 1, 64), device="cuda")
    with pytest.raises(psx.PsxError):   # the cache is full
        ctx.decode_attention(q, kv, kv, 16)
    q = torch.zeros((1, 16, 4, 64), device="cuda")
    kv = torch.zeros((1, 1, 64, 64), device="cuda")
    with pytest.raises(psx.PsxError) as e:   # 64 query rows per kv head
        ctx.decode_attention(q, kv, kv, 8)
    assert e.value.status == psx.ERR_UNSUPPORTED


def _small_call(ctx, **kw):
    import torch
    q = torch.zeros((1, 2, 1, 64), device="cuda")
    kv = torch.zeros((1, 2, 16, 64), device="cuda")
    return lambda: ctx.decode_attention(q, kv, kv, 7, **kw)[1]


@pytest.mark.parametrize("explicit", [False, True])
def test_status_words_belong_to_their_calls_stream(explicit):
    # a call on one stream waits behind long work; a call on another stream must not depend on anything that waits there
    import torch
    ctx, a, b = psx.Context(0), torch.cuda.Stream(), torch.cuda.Stream()
    _small_call(psx.Context(0))()  # (the kernel is loaded)
    first, second = _small_call(ctx, stream=a.cuda_stream if explicit else None), _small_call(ctx, stream=b.cuda_stream if explicit else None)
    with torch.cuda.stream(a):
        stale = [torch.full((256,), -1, dtype=torch.int32, device="cuda") for _ in range(64)]
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        del stale  # (what this stream allocates next holds -1)
        torch.cuda._sleep(400_000_000)  # some 0.2 s
        mine = first()
    with torch.cuda.stream(b):
        other = second()
    b.synchronize()
    assert int(other.cpu()) == 0
    other.fill_(1)
    torch.cuda.synchronize()
    assert int(mine.cpu()) == 0 and int(other.cpu()) == 1
    assert mine.untyped_storage().data_ptr() != other.untyped_storage().data_ptr()


def test_a_captured_call_zeroes_its_status_in_every_replay():
    import torch
    ctx = psx.Context(0)
    call = _small_call(ctx)
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        status = call()
    eager = call()  # (a word handed out after the capture)
    for _ in range(2):
        status.fill_(1)
        graph.replay()
        torch.cuda.synchronize()
        assert int(status.cpu()) == 0
    assert int(eager.cpu()) == 0


def test_status_on_the_default_stream_given_by_its_handle():
    ctx = psx.Context(0)
    assert int(_small_call(ctx, stream=0)().cpu()) == 0


def test_a_second_device_of_the_process():
    # (more shared memory per block than the default limit, which is raised device by device)
    import torch
    if torch.cuda.device_count() < 2:
        pytest.skip("one GPU")
    rng = np.random.RandomState(0)
    q, kv = rng.randn(2, 4, 1, 128).astype(np.float32), rng.randn(2, 2, 2, 40, 128).astype(np.float32)
    got = []
    for d in (0, 1):
        on = [torch.from_numpy(x).to(f"cuda:{d}") for x in (q, kv[0], kv[1])]
        got.append(psx.Context(d).decode_attention(*on, 33)[0].cpu())
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("window", [2001, 2002, 2**31, 2**62, 2**63 - 1])
def test_a_window_wider_than_the_cache_is_none(window):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    q = torch.randn((2, 4, 1, 64), generator=gen, device="cuda")
    keys, values = (torch.randn((2, 2, 2010, 64), generator=gen, device="cuda") for _ in range(2))
    got, want = (gh.ctx().decode_attention(q, keys, values, 2000, window=w)[0] for w in (window, 0))
    assert torch.equal(got, want)
