"""Row kernels of decode steps on the tensor-core path: as many rows as SMs and one more (the norm and query kernels change their form
there), rows that end inside a thread's first, second and third group of values, KV types and head sizes."""
import numpy as np
import pytest

from util import build_pair, pkg, small_cfg, syn

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


@pytest.mark.parametrize("hidden,head_dim,heads,kv_heads,batch,kv", [
    (256, 64, 4, 2, 9, "bf16"), (256, 64, 2, 1, 149, "bf16"), (256, 128, 2, 2, 148, "f32"), (512, 256, 2, 1, 16, "bf16")])
def test_rows_with_tokens_and_positions_of_their_own(hidden, head_dim, heads, kv_heads, batch, kv):
    """Five sequences of unequal lengths in turn, at places inside different pages, each row with its own sequence's next token: a row that
    took another one's token, position, page or partial outputs gets another sequence's logits."""
    cfg = small_cfg(hidden=hidden, layers=2, heads=heads, kv_heads=kv_heads, head_dim=head_dim, inter=128, vocab=300, window=20,
                    layer_types=["sliding_attention", "full_attention"])
    gpu, oracle = build_pair(cfg, "bf16", kv_bf16=(kv == "bf16"), norm_jitter=0.1)
    starts, steps = [1, 15, 16, 33, 50], 3
    seqs = [syn.prompt_ids(300, n + steps, seed=60 + i) for i, n in enumerate(starts)]
    want = []
    for s, n in zip(seqs, starts):
        cache = oracle.new_cache(len(s))
        for t in s[:n]:
            cache.prefill_token(int(t))
        want.append([cache.decode_logits(int(t)) for t in s[n:]])
    of = [b % 5 for b in range(batch)]
    table = gpu.new_cache_table([starts[i] + steps for i in of], batch=batch, page_tokens=16, kv_dtype=pkg.BF16 if kv == "bf16" else pkg.F32)
    gpu.prefill_prompt(np.concatenate([seqs[i][:starts[i]] for i in of]), table, lens=[starts[i] for i in of], want_logits=False)
    for t in range(steps):
        got = gpu.decode_token(np.array([seqs[i][starts[i] + t] for i in of], dtype=np.uint32), table)
        ref = np.stack([want[i][t] for i in of])
        assert (np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)).max() <= TOL
