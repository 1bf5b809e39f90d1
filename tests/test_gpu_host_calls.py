"""The entry points that take rows in host memory (psx_b200_sample_rows_host, psx_b200_process_logits_host) when a call ends early."""
import numpy as np
import pytest

import gpu_harness as gh
import oracle_lib as ol
import pulsatrix_b200 as psx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["sample", "process"])
def test_nothing_is_in_flight_after_an_error(which):
    # The settings are refused once the inputs are on their way (more EOS ids than the library takes); the copies wait behind
    # other work on the context's stream, and the next call reuses the memory that they read.
    import torch
    ctx = psx.Context(0)
    rows, vocab = 3, 20011
    logits, hist = ol.synth_rows(np.arange(rows) + 40, vocab, 2.0, 1.0, 16)
    offsets, uniforms = np.arange(rows + 1, dtype=np.int64) * 16, psx.uniforms_mt19937_64(np.arange(rows, dtype=np.uint64))
    settings = dict(do_sample=True, temperature=0.9, top_k=40, top_p=0.9, repetition_penalty=1.1)
    refused = psx.SamplingConfig.make(min_new_tokens=1, eos_token_ids=[0] * ((1 << 20) + 1), **settings)
    taken = psx.SamplingConfig.make(**settings)

    def call(config, rows_of):
        if which == "sample":
            return ctx.sample_rows_host(rows_of, hist.ravel(), offsets, config, uniforms)[0]
        return ctx.process_logits_host(rows_of, hist.ravel(), offsets, config)

    call(taken, logits.copy())
    stream = torch.cuda.ExternalStream(ctx.stream)
    with torch.cuda.stream(stream):
        torch.cuda._sleep(400_000_000)  # some 0.2 s
    with pytest.raises(psx.PsxError) as error:
        call(refused, logits.copy())
    assert error.value.status == psx.ERR_UNSUPPORTED and "eos" in str(error.value)
    assert stream.query()
    if which == "sample":
        want = ol.rows("oracle", logits, hist.ravel(), offsets, ol.make_config(max_new_tokens=1, **settings), np.arange(rows, dtype=np.uint64))
        assert call(taken, logits).tolist() == want["token"].tolist()
