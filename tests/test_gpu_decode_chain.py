"""The chain of step kernels (default decode path) where it can go wrong: contexts of several key rounds per split,
projections longer than their ring, two to four sessions against one at a time."""
import dataclasses
import time

import numpy as np
import pytest

from conftest import logits_close, seeded_ids

pytestmark = pytest.mark.gpu


def image(mio, cfg):
    return mio.export_model_litertlm(cfg, mio.build_weights_record(cfg))


@pytest.mark.parametrize("kv_dtype", [0, 1])
@pytest.mark.parametrize("prompt", [33, 2048, 2049, 5003])       # one key, one round per split, one key more, several rounds
def test_long_contexts_agree_with_the_streaming_kernel(pkg, mio, prompt, kv_dtype):
    cfg = dataclasses.replace(mio.config_small(), max_ctx=6144, window=2500, kv_dtype=kv_dtype)
    img = image(mio, cfg)
    ids = seeded_ids(prompt, cfg.vocab, prompt)
    chain, stream = (pkg.B200LlmExecutor(img, decode_mode=m) for m in (pkg.DECODE_CHAINED, pkg.DECODE_PERSISTENT))
    assert stream.GetDecodeMode() == pkg.DECODE_PERSISTENT
    for ex in (chain, stream):
        ex.Prefill(ids)
    for step in range(3):
        a, b = (ex.DecodeLogits(None if step == 0 else 5 + step).ravel().astype(np.float64) for ex in (chain, stream))
        assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b), step


@pytest.mark.parametrize("d_model,ffn,vocab", [(64, 64, 16), (448, 4096, 40000), (1152, 12800, 2048)])   # fewer tiles than CTAs .. streamed
def test_odd_projections_agree_with_the_streaming_kernel(pkg, mio, d_model, ffn, vocab):
    cfg = dataclasses.replace(mio.config_small(), n_layers=2, d_model=d_model, ffn=ffn, vocab=vocab, max_ctx=256)
    img = image(mio, cfg)
    ids = seeded_ids(3, cfg.vocab, 70)
    out = []
    for mode in (pkg.DECODE_CHAINED, pkg.DECODE_PERSISTENT_BASIC):
        ex = pkg.B200LlmExecutor(img, decode_mode=mode)
        ex.Prefill(ids)
        out.append(ex.DecodeLogits().ravel().astype(np.float64))
    assert np.linalg.norm(out[0] - out[1]) <= 1e-4 * np.linalg.norm(out[1])


@pytest.mark.parametrize("sessions", [2, 3, 4])
def test_sessions_in_lockstep_agree_with_one_at_a_time(pkg, models, sessions):
    cfg, _, img = models("small")
    prompts = [seeded_ids(40 + i, cfg.vocab, 30 + 41 * i) for i in range(sessions)]
    ex = pkg.B200LlmExecutor(img, n_sessions=sessions)
    for i, p in enumerate(prompts):
        ex.PrefillSession(i, p)
    got = ex.DecodeTokensBatch(6)
    for i, p in enumerate(prompts):
        solo = pkg.B200LlmExecutor(img)
        solo.Prefill(p)
        assert list(solo.DecodeTokens(6)) == list(got[:, i]), i
        ex.SelectSession(i)
        a, b = (e.DecodeLogits().ravel().astype(np.float64) for e in (ex, solo))
        assert np.linalg.norm(a - b) <= 2e-3 * np.linalg.norm(b), i     # two int8 terms with three or four sessions


@pytest.mark.parametrize("kv_dtype", [0, 1])
@pytest.mark.parametrize("heads,kv_heads", [(1, 1), (2, 1), (2, 2), (4, 1), (4, 2)])
@pytest.mark.parametrize("prompt", [1, 33, 1100])              # one key in one split, two splits, all 32 and a window's 20
def test_heads_of_128_one_to_a_slice(pkg, mio, heads, kv_heads, prompt, kv_dtype):
    """A slice of the O projection's K is one head of 128 where there are one, two or four of them: the narrowest form of the
    short combine, alone and with two and four sessions, against the streaming kernel."""
    cfg = dataclasses.replace(mio.config_small(), n_layers=2, n_q_heads=heads, n_kv_heads=kv_heads, head_dim=128, d_model=192, ffn=256, vocab=512,
                              max_ctx=1280, window=600, global_period=2, kv_dtype=kv_dtype)
    img = image(mio, cfg)
    ids = [seeded_ids(prompt + i, cfg.vocab, max(1, prompt - 31 * i)) for i in range(4)]

    def logits(sessions, mode):
        ex = pkg.B200LlmExecutor(img, n_sessions=sessions, decode_mode=mode)
        for i in range(sessions):
            ex.PrefillSession(i, ids[i])
        tokens = ex.DecodeTokensBatch(3)
        out = []
        for i in range(sessions):
            ex.SelectSession(i)
            out.append(ex.DecodeLogits().ravel().astype(np.float64))
        return tokens, out

    # fp32 sums in another order, and two int8 terms with four sessions.  Either may round a value of a bf16 cache the
    # other way: 2^-8 of it, and at most that of a result over few rows.
    for sessions, tol in ((1, 1e-4), (2, 1e-4), (4, 2e-3)):
        tol += kv_dtype * 2.0 ** -8
        (ta, la), (tb, lb) = (logits(sessions, m) for m in (pkg.DECODE_CHAINED, pkg.DECODE_PERSISTENT))
        assert np.array_equal(ta, tb)
        for a, b in zip(la, lb):
            assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)


@pytest.mark.parametrize("d_model,ffn", [(4096, 512), (4160, 512), (6144, 256), (256, 24576)])   # 4, 5 and 6 float4 a thread; down's 6
def test_two_sessions_over_wide_vectors(pkg, mio, d_model, ffn):
    cfg = dataclasses.replace(mio.config_small(), n_layers=2, d_model=d_model, ffn=ffn, n_q_heads=2, head_dim=128, vocab=256, max_ctx=256)
    img = image(mio, cfg)
    ids = [seeded_ids(80 + i, cfg.vocab, 40 - 17 * i) for i in range(2)]
    ex = pkg.B200LlmExecutor(img, n_sessions=2, decode_mode=pkg.DECODE_CHAINED)
    assert ex.GetDecodeMode() == pkg.DECODE_CHAINED
    for i, p in enumerate(ids):
        ex.PrefillSession(i, p)
    got = ex.DecodeTokensBatch(4)
    for i, p in enumerate(ids):
        solo = pkg.B200LlmExecutor(img)
        solo.Prefill(p)
        assert list(solo.DecodeTokens(4)) == list(got[:, i])
        ex.SelectSession(i)
        a, b = (e.DecodeLogits().ravel().astype(np.float64) for e in (ex, solo))
        assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b)


def test_timeline_covers_every_kernel_of_the_step(pkg, models):
    cfg, _, img = models("small")
    ex = pkg.B200LlmExecutor(img)
    ex.Prefill(seeded_ids(1, cfg.vocab, 20))
    tok, stamps, khz = ex.TraceDecodeStep()
    pts = ex.last_trace_points
    assert stamps.shape[0] == 5 * cfg.n_layers + 2 and khz == 1000000 and 0 <= tok < cfg.vocab
    for k in range(5 * cfg.n_layers + 1):
        p = pts[k][pts[k][:, 4] > 0]
        assert len(p) and (np.diff(p[:, :5], axis=1) >= 0).all(), k


@pytest.mark.parametrize("d_model,ffn,heads,sessions,mode", [
    (64, 6208, (4, 1, 256), 2, 2),      # ffn = 64 * 97 has no K split: too long for two sessions, the persistent kernel
    (64, 6208, (4, 1, 256), 4, 4),      # too much staging for that with four: the chain, one session after another
    (6208, 64, (4, 1, 256), 2, 4),      # a residual that the persistent kernel does not take either
    (64, 24896, (2, 2, 32), 1, 1),      # 64 * 389, too long for one session: one kernel per phase
])
def test_geometries_beyond_the_chain_have_a_fallback(pkg, orc, mio, d_model, ffn, heads, sessions, mode):
    cfg = dataclasses.replace(mio.config_small(), n_layers=2, d_model=d_model, ffn=ffn, n_q_heads=heads[0], n_kv_heads=heads[1],
                              head_dim=heads[2], vocab=512, max_ctx=256)
    record = mio.build_weights_record(cfg)
    ex = pkg.B200LlmExecutor(mio.export_model_litertlm(cfg, record), n_sessions=sessions)
    assert ex.GetDecodeMode() == mode
    prompts = [seeded_ids(60 + i, cfg.vocab, 20 + 9 * i) for i in range(sessions)]
    for i, p in enumerate(prompts):
        ex.PrefillSession(i, p)
    got = ex.DecodeTokensBatch(3)
    model = orc.OracleModel(record)
    for i, p in enumerate(prompts):
        ref = orc.OracleExecutor(model)
        assert ref.prefill(p) == 0
        for step in range(3):                # teacher-forced: the device's id is one the oracle puts at its best, within the prefill's tolerance
            rc, want = ref.decode_logits()
            assert rc == 0 and want[got[step, i]] >= want.max() - 2e-2 * (want.max() - want.min()), (i, step)
            assert ref.prefill(got[step:step + 1, i].copy()) == 0
        ex.SelectSession(i)
        rc, want = ref.decode_logits()
        cos, err = logits_close(ex.DecodeLogits(), want)
        assert rc == 0 and cos >= 0.999 and err <= 2e-2, (i, cos, err)


def test_every_requested_mode_finds_kernels(pkg, mio):
    cfg = dataclasses.replace(mio.config_small(), n_layers=1, d_model=64, ffn=6208, vocab=512, max_ctx=256)
    img = image(mio, cfg)
    want = {(pkg.DECODE_PHASE_KERNELS, 4): 1, (pkg.DECODE_PERSISTENT, 1): 2, (pkg.DECODE_PERSISTENT, 4): 4, (pkg.DECODE_PERSISTENT_BASIC, 2): 3,
            (pkg.DECODE_CHAINED, 1): 4, (pkg.DECODE_CHAINED, 2): 2}
    for (mode, n), runs in want.items():
        assert pkg.B200LlmExecutor(img, n_sessions=n, decode_mode=mode).GetDecodeMode() == runs, (mode, n)
    with pytest.raises(Exception, match="shared memory"):
        pkg.B200LlmExecutor(img, n_sessions=4, decode_mode=pkg.DECODE_PERSISTENT_BASIC)


def test_the_first_decode_call_does_not_wait_for_a_graph(pkg, mio):
    """A step is 121 launches here; capturing and instantiating its graph takes the host longer than the GPU needs for
    the step (2.3 times the time of a later call, where plain launches take 1.2 times).  Least of eight executors; and
    every call gives the same logits, launched or replayed."""
    cfg = dataclasses.replace(mio.config_small(), n_layers=24, d_model=64, ffn=128, vocab=512, max_ctx=256)
    owner = pkg.B200LlmExecutor(image(mio, cfg))
    ids = seeded_ids(8, cfg.vocab, 20)
    times, logits = [], []
    for _ in range(8):
        ex = owner.CreateShared()
        row = []
        for _ in range(7):
            ex.Reset()
            ex.Prefill(ids)
            t0 = time.perf_counter()
            logits.append(ex.DecodeLogits().ravel().copy())
            row.append(time.perf_counter() - t0)
        times.append(row)
    least = np.min(times, axis=0)
    assert least[0] <= 1.8 * least[4:].min(), (least * 1e6).round().tolist()
    assert all(np.array_equal(x, logits[0]) for x in logits)


@pytest.mark.parametrize("sessions", [1, 3, 6])               # the chain, and the wide step
def test_the_callers_stream_may_be_the_default_stream(pkg, models, sessions):
    cfg, _, img = models("small")
    out = []
    for stream in (0, 1):                                     # an own stream; cudaStreamLegacy, which cannot be captured
        ex = pkg.B200LlmExecutor(img, n_sessions=sessions, stream=stream)
        for i in range(sessions):
            ex.PrefillSession(i, seeded_ids(70 + i, cfg.vocab, 25 + 7 * i))
        out.append((ex.DecodeTokensBatch(8), ex.DecodeLogits().copy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
