"""Prompt passes of more than 256 rows that attend slice by slice (BF16 weights with an f32 cache, or with pages of no multiple of 16
tokens), against the CPU oracle; the row counts at which a pass changes its projections (96) and its attention (64); the same passes
made twice."""
import numpy as np
import pytest

from util import build_pair, pkg, small_cfg, syn

pytestmark = pytest.mark.gpu

TOL_BF16 = 2e-2                    # of logits, as in the other comparisons of BF16 weights with the oracle


def _cfg(head_dim, heads, kv_heads, window):
    return small_cfg(hidden=128, layers=2, heads=heads, kv_heads=kv_heads, head_dim=head_dim, inter=256, vocab=700, window=window,
                     layer_types=["sliding_attention", "full_attention"])


def _oracle(oracle, tokens, want, max_seq):
    cache, out = oracle.new_cache(max_seq), {}
    for i, t in enumerate(tokens):
        if i in want:
            out[i] = cache.decode_logits(int(t))
        else:
            cache.prefill_token(int(t))
    return out


# a ring of window + 255 rows, rounded up to 16: 304 rows, which the second slice wraps; pages of 7 leave slices' ends inside pages
@pytest.mark.parametrize("head_dim,heads,kv_heads,kv,page", [(64, 4, 2, "f32", 256), (128, 4, 1, "f32", 16), (256, 2, 2, "f32", 32), (64, 2, 1, "bf16", 7)])
def test_one_prompt_of_three_slices_and_a_later_portion(head_dim, heads, kv_heads, kv, page):
    gpu, oracle = build_pair(_cfg(head_dim, heads, kv_heads, 40), "bf16", kv_bf16=(kv == "bf16"), norm_jitter=0.1)
    tokens = syn.prompt_ids(700, 902, seed=head_dim)
    table = gpu.new_cache_table(902, page_tokens=page, kv_dtype=pkg.BF16 if kv == "bf16" else pkg.F32)
    first, second = [0, 39, 40, 255, 256, 257, 295, 511, 512, 599], [600, 855, 856, 899]
    got = dict(zip(first, gpu.extend(tokens[:600], table, want=first)))
    got.update(zip(second, gpu.extend(tokens[600:900], table, want=[p - 600 for p in second])))
    for p in (900, 901):
        got[p] = gpu.decode_token(int(tokens[p]), table)
    for p, ref in _oracle(oracle, tokens, set(got), 902).items():
        assert np.abs(got[p] - ref).max() <= TOL_BF16, p


@pytest.mark.parametrize("heads,kv_heads", [(4, 2), (8, 1)])
def test_unequal_prompts_across_slices(heads, kv_heads):
    """Runs that end at, before and behind a slice's end, several in one slice and one over three; then portions, some of them empty."""
    gpu, oracle = build_pair(_cfg(64, heads, kv_heads, 33), "bf16", kv_bf16=False, norm_jitter=0.1)
    lens, more = [3, 250, 5, 254, 1, 600, 130], [300, 0, 1, 40, 2, 257, 0]
    seqs = [syn.prompt_ids(700, a + b, seed=40 + i) for i, (a, b) in enumerate(zip(lens, more))]
    table = gpu.new_cache_table([len(s) + 1 for s in seqs], batch=7, page_tokens=48, kv_dtype=pkg.F32)
    got = gpu.prefill_prompt(np.concatenate([s[:n] for s, n in zip(seqs, lens)]), table, lens=lens)
    ends, fed = np.cumsum(more), [i for i in range(7) if more[i]]
    got2 = gpu.extend(np.concatenate([s[n:] for s, n in zip(seqs, lens)]), table, lens=more, want=[int(ends[i]) - 1 for i in fed])
    for i in range(7):
        ref = _oracle(oracle, seqs[i], {lens[i] - 1, len(seqs[i]) - 1}, len(seqs[i]) + 1)
        assert np.abs(got[i] - ref[lens[i] - 1]).max() <= TOL_BF16, i
        if more[i]:
            assert np.abs(got2[fed.index(i)] - ref[len(seqs[i]) - 1]).max() <= TOL_BF16, i


@pytest.mark.parametrize("kv", ["f32", "bf16"])
def test_passes_at_the_row_counts_where_the_kernels_change(kv):
    gpu, oracle = build_pair(_cfg(64, 4, 2, 50), "bf16", kv_bf16=(kv == "bf16"), norm_jitter=0.1)
    sizes = [63, 64, 96, 97]
    tokens = syn.prompt_ids(700, sum(sizes), seed=9)
    kv_dtype = pkg.BF16 if kv == "bf16" else pkg.F32
    table, probe = (gpu.new_cache_table(len(tokens), page_tokens=16, kv_dtype=kv_dtype) for _ in range(2))
    got, at = {}, 0
    for n in sizes:
        want = [0, n // 2, n - 1]
        got.update(zip([at + w for w in want], gpu.extend(tokens[at:at + n], table, want=want)))
        kinds = gpu.profile_extend(tokens[at:at + n], probe)
        assert ("geglu" in kinds) == (n <= 96)                       # SM pairs have the activation in the projection
        assert ("kv_append" in kinds) == (kv == "bf16" and n >= 64)  # prompt_attn_kernel
        at += n
    for p, ref in _oracle(oracle, tokens, set(got), len(tokens)).items():
        assert np.abs(got[p] - ref).max() <= TOL_BF16, p


@pytest.mark.parametrize("kv", ["f32", "bf16"])
def test_the_same_passes_give_the_same_bits(kv):
    """Cut tiles, split positions and their merges add in a fixed order: a call that is repeated on a new table gives the same bits. (It
    need not give those of a call with other neighbours: which tiles are cut, and where, depends on all rows of the pass.)"""
    gpu, _ = build_pair(_cfg(64, 4, 2, 50), "bf16", kv_bf16=(kv == "bf16"), norm_jitter=0.1, want_oracle=False)
    lens = [310, 97, 1, 140]
    tokens, more = syn.prompt_ids(700, sum(lens), seed=3), syn.prompt_ids(700, 400, seed=4)
    out = []
    for _ in range(3):
        table = gpu.new_cache_table([n + 110 for n in lens], batch=4, page_tokens=16, kv_dtype=pkg.BF16 if kv == "bf16" else pkg.F32)
        out.append(np.concatenate([gpu.prefill_prompt(tokens, table, lens=lens), gpu.extend(more, table, lens=[100] * 4, want=[0, 99, 250, 399]),
                                   gpu.decode_token(more[:4], table)]))
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
