"""The prefill's KV append in groups of eight positions: chunks that begin and end inside a group, and inside a page."""
import numpy as np
import pytest

from conftest import logits_close, seeded_ids

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cuts", [(2,), (9, 12, 18), (8, 17), (254, 262)])
def test_append_in_chunks_agrees_with_one_prefill(pkg, models, cuts):
    cfg, _, img = models("gemma3-4b-slice")
    ids = seeded_ids(77, cfg.vocab, 280)
    one, parts = pkg.B200LlmExecutor(img), pkg.B200LlmExecutor(img)
    one.Prefill(ids)
    for a, b in zip((0,) + cuts, cuts + (len(ids),)):
        parts.Prefill(ids[a:b])
    cos, err = logits_close(parts.DecodeLogits().ravel(), one.DecodeLogits().ravel())
    assert cos >= 0.9995 and err <= 1e-2, (cos, err)
    for pos in {c - 1 for c in cuts} | set(cuts) | {0, 278}:
        for is_v in (False, True):
            got, want = (e.ReadKvRow(0, is_v, cfg.n_kv_heads - 1, pos)[0][:cfg.head_dim] for e in (parts, one))
            assert np.abs(got - want).max() <= 1e-3 * np.abs(want).max(), (pos, is_v)
