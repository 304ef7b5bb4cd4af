"""Row kernels of decode steps on the tensor-core path: as many rows as SMs and one more (the norm and query kernels change their form
there), rows that end inside a thread's first, second and third group of values, KV types and head sizes."""
import numpy as np
import pytest

from util import build_pair, pkg, small_cfg

pytestmark = pytest.mark.gpu

# relative 2-norm of a row's logits: the two layers and the head round eight operands to BF16 (2^-9 each), and two orders of the same
# sums may round any of them the other way
TOL = 8 * 2.0 ** -9


@pytest.mark.parametrize("hidden,head_dim,heads,kv_heads,batch,kv", [
    (200, 64, 2, 1, 9, "bf16"), (200, 64, 4, 4, 149, "bf16"), (2056, 128, 2, 1, 16, "bf16"), (2056, 128, 2, 2, 148, "f32"),
    (4104, 256, 2, 1, 8, "bf16"), (4104, 256, 1, 1, 150, "f32")])
def test_every_row_of_a_step_matches_the_oracle(hidden, head_dim, heads, kv_heads, batch, kv):
    cfg = small_cfg(hidden=hidden, layers=2, heads=heads, kv_heads=kv_heads, head_dim=head_dim, inter=128, vocab=300, window=3,
                    layer_types=["sliding_attention", "full_attention"])
    gpu, oracle = build_pair(cfg, "bf16", kv_bf16=(kv == "bf16"), norm_jitter=0.1)
    table = gpu.new_cache_table([8] * batch, batch=batch, page_tokens=16, kv_dtype=pkg.BF16 if kv == "bf16" else pkg.F32)
    cache = oracle.new_cache(8)
    for token in (5, 77, 299, 6):
        want = cache.decode_logits(token)
        got = gpu.decode_token(np.full(batch, token, dtype=np.uint32), table)
        assert (np.linalg.norm(got - want[None], axis=1) / np.linalg.norm(want)).max() <= TOL
