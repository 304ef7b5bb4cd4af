"""Edges of the top-k kernels (csrc/sampling.cuh) through oxg4_topk_noalloc: part of a chunk, a chunk and one more, fewer candidates
than places, ties, signed zeros, infinities and NaN."""
import ctypes as C

import numpy as np
import pytest

from util import build_pair, pkg, small_cfg

pytestmark = pytest.mark.gpu


def _topk(logits, seen, penalty, k):
    import torch
    N = pkg._native
    rows, V = logits.shape
    d_logits, d_seen = torch.from_numpy(logits).cuda(), None if seen is None else torch.from_numpy(seen).cuda()
    ids = torch.zeros((rows, k), dtype=torch.int32, device="cuda")
    scores = torch.zeros((rows, k), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    N.check(N.lib().oxg4_topk_noalloc(C.c_void_p(d_logits.data_ptr()), rows, V, None if seen is None else C.c_void_p(d_seen.data_ptr()),
                                      penalty, k, C.c_void_p(ids.data_ptr()), C.c_void_p(scores.data_ptr()), None))
    torch.cuda.synchronize()
    return ids.cpu().numpy().view(np.uint32), scores.cpu().numpy()


def _want(row, seen, penalty, k):
    s = row.astype(np.float32).copy()
    if seen is not None and penalty > 1.0:
        hit = seen != 0
        s[hit] = np.where(s[hit] >= 0, s[hit] / np.float32(penalty), s[hit] * np.float32(penalty))
    s[np.isnan(s)] = -np.inf
    order = np.lexsort((np.arange(s.size), -s))[:k]
    order = order[s[order] > -np.inf]
    ids, scores = np.zeros(k, dtype=np.uint32), np.full(k, -np.inf, dtype=np.float32)
    ids[:order.size], scores[:order.size] = order, s[order]
    return ids, scores


@pytest.mark.parametrize("k", [1, 2, 33, 64])
@pytest.mark.parametrize("vocab", [64, 255, 257, 2047, 2048, 2049, 70000])
def test_random_rows_with_ties(vocab, k):
    rng = np.random.default_rng(vocab + k)
    logits = np.round(rng.standard_normal((3, vocab)) * 8).astype(np.float32) / 8          # many equal scores
    seen = (rng.random((3, vocab)) < 0.3).astype(np.uint8)
    for mask, penalty in ((None, 1.0), (seen, 1.3)):
        ids, scores = _topk(logits, mask, penalty, k)
        for r in range(3):
            want_ids, want_scores = _want(logits[r], None if mask is None else mask[r], penalty, k)
            assert ids[r].tolist() == want_ids.tolist()
            np.testing.assert_array_equal(scores[r], want_scores)


def test_rows_with_few_candidates():
    """Infinities, signed zeros and denormals in order; NaN and minus infinity are never selected, places that stay empty are 0, -inf."""
    logits = np.full((4, 4100), -np.inf, dtype=np.float32)
    logits[0, [4099, 7, 2048, 9, 300]] = [np.inf, -0.0, 0.0, 1e-42, np.float32(-3.4028235e38)]
    logits[1, :] = np.nan
    logits[2, 5::2] = -0.0
    logits[2, 4::2] = 0.0
    logits[3, 4000:] = np.arange(100, dtype=np.float32) - 50.0
    ids, scores = _topk(logits, None, 1.0, 40)
    for r in range(4):
        want_ids, want_scores = _want(logits[r], None, 1.0, 40)
        assert ids[r].tolist() == want_ids.tolist(), r
        np.testing.assert_array_equal(scores[r], want_scores)
        np.testing.assert_array_equal(np.signbit(scores[r]), np.signbit(want_scores))


def test_lists_fill_shared_memory():
    """966 chunks of 2048 scores with 30 candidates each take 231840 of the 232448 bytes that a block can have: the merge may need next to
    nothing beside the lists."""
    k, vocab = 30, 966 * 2048 - 5
    gpu, _ = build_pair(small_cfg(hidden=16, layers=1, heads=1, kv_heads=1, head_dim=64, inter=32, vocab=vocab, window=8), "bf16",
                        kv_bf16=False, want_oracle=False)
    a, b = gpu.new_cache_table(4, kv_dtype=pkg.F32), gpu.new_cache_table(4, kv_dtype=pkg.F32)
    want_ids, want_scores = _want(gpu.decode_token(7, a), None, 1.0, k)
    got = gpu.decode_topk(7, b, k, 1.0, False)
    assert [i for i, _ in got] == want_ids.tolist()
    np.testing.assert_array_equal(np.array([s for _, s in got], dtype=np.float32), want_scores)
