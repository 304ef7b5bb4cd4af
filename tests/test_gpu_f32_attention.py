"""Attention in f32 (csrc/attention.cuh) for the rows of a prompt: more query heads per key/value head than the CTAs of a launch with many
rows have warps."""
import numpy as np
import pytest

from util import build_pair, pkg, small_cfg, syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,kv,page,tol", [("f32", "f32", 32, 1e-3), ("bf16", "f32", 32, 2e-2), ("bf16", "bf16", 7, 2e-2)])
@pytest.mark.parametrize("head_dim,heads,kv_heads", [(64, 8, 1), (128, 8, 1), (256, 8, 1), (128, 16, 2)])
def test_eight_query_heads_of_a_key_head(dtype, kv, page, tol, head_dim, heads, kv_heads):
    cfg = small_cfg(hidden=128, layers=2, heads=heads, kv_heads=kv_heads, head_dim=head_dim, inter=128, vocab=600, window=40,
                    layer_types=["sliding_attention", "full_attention"])
    gpu, oracle = build_pair(cfg, dtype, kv_bf16=(kv == "bf16"), norm_jitter=0.1)
    tokens = syn.prompt_ids(600, 281, seed=head_dim)
    table = gpu.new_cache_table(281, page_tokens=page, kv_dtype=pkg.BF16 if kv == "bf16" else pkg.F32)
    places = [0, 3, 41, 199]
    got = dict(zip(places, gpu.extend(tokens[:200], table, want=places)))
    got[279] = gpu.extend(tokens[200:280], table, want=[79])[0]
    got[280] = gpu.decode_token(int(tokens[280]), table)
    cache = oracle.new_cache(281)
    for i, t in enumerate(tokens):
        if i in got:
            assert np.abs(got[i] - cache.decode_logits(int(t))).max() <= tol, i
        else:
            cache.prefill_token(int(t))
