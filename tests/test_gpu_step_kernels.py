"""Kernels of decode steps with few sequences at the sizes where they can go wrong: projections through shared memory
(csrc/gemv_mma.cuh, csrc/gemv_rows.cuh) with columns and rows that fill no box, and the attention of one token (csrc/attention.cuh) with units of fewer
heads than a key/value head has, positions around split and window edges."""
import numpy as np
import pytest

import layered_util
from util import build_pair, pkg, small_cfg, syn

pytestmark = pytest.mark.gpu

# relative 2-norm of a row's logits: a layer and the head round four operands to BF16 (2^-9 each), and two orders of the same sums
# may round any of them the other way
TOL = 4 * 2.0 ** -9


@pytest.fixture(params=["short", "long"])
def launches(request):
    """Makes a BF16 model take the one-row projections of short or of long launches."""
    def choose(state):
        pkg._native.check(pkg._native.lib().oxg4_debug_long_launches(state._h, int(request.param == "long")))
        return request.param
    return choose


@pytest.mark.parametrize("hidden,inter,heads,head_dim,vocab,batch,tcgen05", [
    (72, 40, 1, 64, 37, 1, True),           # columns of a box past the end, fewer column blocks than warps
    (2560, 4768, 8, 64, 4111, 1, True),     # 17 and 18 rows per CTA, 16 and 17 pairs: two boxes, the second nearly empty
    (3072, 160, 4, 256, 5003, 1, True),     # norm weights in registers: the widest row
    (3080, 160, 4, 256, 300, 1, True),      # one past it
    (5632, 96, 2, 64, 300, 1, True),        # the widest hidden row
    (264, 136, 2, 64, 301, 2, True), (1160, 2080, 2, 128, 301, 3, True), (264, 96, 2, 64, 20011, 7, True), (2056, 10272, 2, 64, 300, 7, True),
    # several rows without tcgen05, as models with per-layer embeddings and tensor-parallel ranks have them
    (264, 136, 2, 64, 301, 2, False),       # intermediate size no multiple of 32: activations in f32 between gate/up and down
    (1160, 2080, 2, 128, 301, 3, False),    # three rows share four teams of warps
    (3080, 96, 2, 64, 300, 4, False), (264, 96, 2, 64, 20011, 7, False), (72, 40, 1, 64, 37, 8, False),
    (264, 20000, 2, 64, 300, 7, False), (264, 20008, 2, 64, 300, 8, False),     # as many rows of the down projection as fit, twice
    (264, 136, 2, 64, 301, 9, False), (1160, 2080, 2, 128, 20011, 15, False),   # csrc/gemv_rows.cuh
    (264, 96, 2, 64, 301, 17, False),       # sixteen rows and one
    (264, 20000, 2, 64, 300, 9, False)])    # nine rows, of the down projection five at a time
def test_projections_of_few_rows(hidden, inter, heads, head_dim, vocab, batch, tcgen05, launches, monkeypatch):
    cfg = small_cfg(hidden=hidden, layers=1, heads=heads, kv_heads=1 if heads != 8 else 4, head_dim=head_dim, inter=inter, vocab=vocab,
                    window=64, layer_types=["full_attention"])
    gpu, oracle = build_pair(cfg, "bf16", kv_bf16=True, norm_jitter=0.1)
    if launches(gpu) == "long" and batch > 1:
        pytest.skip("one row only")
    if not tcgen05:
        monkeypatch.setenv("OXG4_DISABLE_TCGEN05", "1")        # looked at when a table is made
    table = gpu.new_cache_table([8] * batch, batch=batch, page_tokens=16, kv_dtype=pkg.BF16)
    caches = [oracle.new_cache(8) for _ in range(batch)]
    for t in range(3):
        tokens = np.array([(5 + 11 * b + 7 * t) % vocab for b in range(batch)], dtype=np.uint32)
        want = np.stack([c.decode_logits(int(x)) for c, x in zip(caches, tokens)])
        got = np.atleast_2d(gpu.decode_token(tokens, table))
        assert (np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)).max() <= TOL
        if t == 0:                                             # the fused arg-max, one position on
            best = gpu.decode_topk(tokens, table, 1, 1.0, False)
            best = np.array([[best[0][0]]]) if batch == 1 else best[0].astype(np.int64)
            want = np.stack([c.decode_logits(int(x)) for c, x in zip(caches, tokens)])
            top = np.take_along_axis(want, best, 1)[:, 0]
            assert (want.max(1) - top <= 2 * TOL * np.linalg.norm(want, axis=1)).all()


# f32 cache: rounding of f32 sums. BF16 cache: a key's element (up to 4 after its norm) that lies between two BF16 values may round to
# the other one, 2^-6 away at most; with |q| up to 4 that moves a score by 2^-4, its softmax weight p by the factor exp(2^-4) and the
# head's output by p (1 - p) 2^-4 <= 2^-6 of the values' size
@pytest.mark.parametrize("kv", ["f32", "bf16"])
@pytest.mark.parametrize("head_dim,heads,kv_heads,batch,room", [
    (64, 1, 1, 1, 0), (64, 8, 1, 1, 0), (128, 4, 1, 1, 0), (256, 2, 2, 1, 0), (256, 8, 1, 1, 0), (128, 16, 8, 1, 0), (64, 8, 2, 3, 0), (256, 4, 1, 5, 0),
    # tables with room for so many positions that the other kernel attends in the global layer: with four and sixteen warps per CTA
    (64, 1, 1, 1, 20000), (128, 4, 2, 1, 20000), (256, 8, 1, 5, 20000), (64, 8, 2, 3, 20000), (256, 2, 2, 1, 20000), (256, 8, 2, 24, 600)])
def test_attention_of_one_token(head_dim, heads, kv_heads, batch, room, kv):
    cfg = small_cfg(hidden=128, layers=2, heads=heads, kv_heads=kv_heads, head_dim=head_dim, inter=128, vocab=600, window=40,
                    layer_types=["sliding_attention", "full_attention"])
    gpu, oracle = build_pair(cfg, "f32", kv_bf16=(kv == "bf16"), norm_jitter=0.1)
    n = 300
    seqs = [syn.prompt_ids(600, n, seed=10 * head_dim + b) for b in range(batch)]
    # a table for more positions than are used (sixteen splits) and, for one sequence, one for a handful (a split or two)
    table = gpu.new_cache_table([n + room + 30 * b for b in range(batch)], batch=batch, page_tokens=16, kv_dtype=pkg.F32 if kv == "f32" else pkg.BF16)
    small = gpu.new_cache_table(20, page_tokens=16, kv_dtype=pkg.F32 if kv == "f32" else pkg.BF16) if batch == 1 else None
    caches = [oracle.new_cache(n) for _ in range(batch)]
    look = {0, 1, 7, 15, 16, 17, 31, 32, 33, 39, 40, 41, 127, 128, 129, 255, 256, 257, 299}
    for t in range(n):
        tokens = np.array([s[t] for s in seqs], dtype=np.uint32)
        if t not in look:
            for c, s in zip(caches, seqs):
                c.prefill_token(int(s[t]))
            gpu.prefill_token(tokens, table)
            if small is not None and t < 20:
                gpu.prefill_token(tokens, small)
            continue
        want = np.stack([c.decode_logits(int(s[t])) for c, s in zip(caches, seqs)])
        off = np.atleast_2d(gpu.decode_token(tokens, table)) - want
        assert np.abs(off).max() <= 1e-3 if kv == "f32" else np.linalg.norm(off) <= 2.0 ** -6 * np.linalg.norm(want), t
        if small is not None and t < 20:
            off = gpu.decode_token(tokens, small) - want[0]
            assert np.abs(off).max() <= 1e-3 if kv == "f32" else np.linalg.norm(off) <= 2.0 ** -6 * np.linalg.norm(want), t


@pytest.mark.parametrize("head_dim,heads,kv_heads,batch,room", [
    (64, 2, 2, 2, 0), (64, 2, 2, 2, 5000), (128, 8, 1, 5, 2000), (256, 2, 1, 3, 9000), (256, 8, 2, 8, 0), (64, 8, 1, 5, 9000)])
def test_one_launch_or_three_beside_tcgen05(head_dim, heads, kv_heads, batch, room):
    """Batches whose global layer attends by attn_step_kernel, attn_decode_kernel (with BF16 output) or the tensor-core attention, by
    what the table has room for: the same logits to the rounding of BF16 operands."""
    cfg = small_cfg(hidden=256, layers=1, heads=heads, kv_heads=kv_heads, head_dim=head_dim, inter=128, vocab=600, window=40, layer_types=["full_attention"])
    gpu, oracle = build_pair(cfg, "bf16", kv_bf16=True, norm_jitter=0.1)
    n = 40
    seqs = [syn.prompt_ids(600, n, seed=40 * head_dim + b) for b in range(batch)]
    table = gpu.new_cache_table([n + room] * batch, batch=batch, page_tokens=16, kv_dtype=pkg.BF16)
    caches = [oracle.new_cache(n) for _ in range(batch)]
    for t in range(n):
        tokens = np.array([s[t] for s in seqs], dtype=np.uint32)
        want = np.stack([c.decode_logits(int(x)) for c, x in zip(caches, tokens)])
        got = gpu.decode_token(tokens, table)
        # with the bound on the attention's output above
        assert (np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)).max() <= TOL + 2.0 ** -6, t


# a mechanism alone: BF16 operands of its projections and of the head, recurrent state or cache beside them
@pytest.mark.parametrize("layer", [
    layered_util.wkv(2, 64, ff=96), layered_util.lightning(2, 32, 64, (0.9, 0.99), ff=72), layered_util.latent(3, 32, 48, 64, 80, 16, ff=136),
    layered_util.retention(3, 32, 64, (0.8, 0.95, 0.99), ff=200), layered_util.attention(4, 2, 32, 64, ff=104)], ids=lambda x: x["type"])
def test_one_row_of_listed_layers(layer, launches):
    pair = layered_util.Pair(layered_util.config([layer], width=100), "bf16", seed=5)
    launches(pair.state)
    tokens = pair.prompt(30, 6)
    assert layered_util.error(layered_util.feed(pair, pair.table(40), tokens, [1]), pair.want(tokens)) <= 3e-2
