"""GPU parity of the prompt attention kernel (csrc/prompt_attn.cuh) against the CPU oracle, which ingests prompts token by
token: rows of one tile and of several, unequal prompts in one pass, portions into a filled cache (keys from the pages and
from the pass), a prompt longer than a pass whose sliding ring wraps many times, split positions with their merge."""
import numpy as np
import pytest

from util import build_pair, pkg, small_cfg, syn

pytestmark = pytest.mark.gpu

TOL_BF16 = 2e-2


def _cfg(head_dim, heads, kv_heads, window):
    return small_cfg(hidden=128, layers=2, heads=heads, kv_heads=kv_heads, head_dim=head_dim, inter=256, vocab=700, window=window,
                     layer_types=["sliding_attention", "full_attention"])


def _oracle(oracle, tokens, want, max_seq):
    """Logits behind the tokens at the places `want`."""
    cache, out = oracle.new_cache(max_seq), []
    for i, t in enumerate(tokens):
        if i in want:
            out.append(cache.decode_logits(int(t)))
        else:
            cache.prefill_token(int(t))
    return np.stack(out)


# head sizes and group sizes: 128, 64, 32 and 16 tokens per tile; page sizes that are and are not multiples of a tile
@pytest.mark.parametrize("head_dim,heads,kv_heads,page", [(64, 2, 2, 16), (64, 8, 1, 48), (128, 4, 2, 256), (256, 4, 1, 32), (256, 2, 1, 7)])
def test_portions_into_a_filled_cache(head_dim, heads, kv_heads, page):
    """Portions of 65 (one tile, mostly empty), 200, 97 and 129 tokens: from the second on the keys come from pages and pass;
    the window of 50 is shorter than a portion, so the first rows see pages and the last ones do not."""
    gpu, oracle = build_pair(_cfg(head_dim, heads, kv_heads, 50), "bf16", kv_bf16=True, norm_jitter=0.1)
    sizes = [65, 200, 97, 129]
    tokens = syn.prompt_ids(700, sum(sizes) + 3, seed=head_dim + heads)
    table = gpu.new_cache_table(len(tokens), page_tokens=page, kv_dtype=pkg.BF16)
    got, at, places = [], 0, []
    for n in sizes:
        want = sorted({0, n // 2, n - 1})
        got.append(gpu.extend(tokens[at:at + n], table, want=want))
        places += [at + w for w in want]
        at += n
    for t in tokens[at:]:
        got.append(gpu.decode_token(int(t), table)[None])
        places.append(at)
        at += 1
    ref = _oracle(oracle, tokens, set(places), len(tokens))
    assert np.abs(np.concatenate(got) - ref).max() <= TOL_BF16


def test_prompt_longer_than_a_pass():
    """2300 tokens: two passes, the ring of the sliding layer (window 40) is overwritten by each of them."""
    gpu, oracle = build_pair(_cfg(64, 4, 2, 40), "bf16", kv_bf16=True, norm_jitter=0.1)
    tokens = syn.prompt_ids(700, 2303, seed=5)
    table = gpu.new_cache_table(len(tokens), page_tokens=64, kv_dtype=pkg.BF16)
    got = [gpu.prefill_prompt(tokens[:2300], table)] + [gpu.decode_token(int(t), table) for t in tokens[2300:]]
    ref = _oracle(oracle, tokens, {2299, 2300, 2301, 2302}, len(tokens))
    assert np.abs(np.stack(got) - ref).max() <= TOL_BF16


def test_unequal_prompts_of_one_pass():
    """Nine prompts of 1 to 400 tokens in one pass, then a further portion of each, some of them empty."""
    gpu, oracle = build_pair(_cfg(128, 4, 2, 100), "bf16", kv_bf16=True, norm_jitter=0.1)
    lens, more = [1, 400, 63, 64, 65, 127, 128, 129, 2], [5, 0, 130, 1, 64, 0, 33, 200, 3]
    seqs = [syn.prompt_ids(700, a + b, seed=20 + i) for i, (a, b) in enumerate(zip(lens, more))]
    table = gpu.new_cache_table([len(s) + 1 for s in seqs], batch=9, page_tokens=32, kv_dtype=pkg.BF16)
    got = gpu.prefill_prompt(np.concatenate([s[:n] for s, n in zip(seqs, lens)]), table, lens=lens)
    ends = np.cumsum(more)
    fed = [i for i in range(9) if more[i]]
    got2 = gpu.extend(np.concatenate([s[n:] for s, n in zip(seqs, lens)]), table, lens=more, want=[int(ends[i]) - 1 for i in fed])
    for i in range(9):
        places = {lens[i] - 1} | ({len(seqs[i]) - 1} if more[i] else set())
        ref = _oracle(oracle, seqs[i], places, len(seqs[i]) + 1)
        assert np.abs(got[i] - ref[0]).max() <= TOL_BF16
        if more[i]:
            assert np.abs(got2[fed.index(i)] - ref[-1]).max() <= TOL_BF16


@pytest.mark.parametrize("page,mma", [(16, True), (48, True), (7, False), (24, False), (1, False)])
def test_pages_of_odd_sizes_keep_queries_in_f32(page, mma):
    """Pages of a multiple of 16 tokens attend on the tensor cores, with queries and softmax weights as pairs of BF16 values (2^-17),
    steps and prompts alike. With any other page size both are held in f32, and a prompt has to go through the same kernel as a step."""
    gpu, _ = build_pair(_cfg(64, 4, 2, 50), "bf16", kv_bf16=True, want_oracle=False)
    table = gpu.new_cache_table(310, page_tokens=page, kv_dtype=pkg.BF16)
    for n in (63, 64, 97, 80):
        kinds = gpu.profile_extend(syn.prompt_ids(700, n, seed=n), table)
        assert ("kv_append" in kinds) == (mma and n >= 64)       # prompt_attn_kernel ran
        assert mma or "attn_merge" not in kinds                  # no tensor-core attention at all


@pytest.mark.parametrize("head_dim,heads,kv_heads", [(64, 4, 2), (64, 4, 1), (128, 2, 1), (256, 2, 2)])
@pytest.mark.parametrize("kind,window", [("full_attention", 9), ("sliding_attention", 70)])
def test_attention_keeps_the_low_parts_of_queries_and_weights(head_dim, heads, kv_heads, kind, window):
    """The same prompt with pages of 16 tokens (this kernel) and of 24 (queries and softmax weights in f32), from equal projections of a
    one-layer model: in one pass, then a portion into the filled cache.

    The kernels' sums differ by about 2^-17 of a value, one value in 2^9 rounds to the other BF16 number: of the 256 of a row none or one,
    so that six rows in ten have no such value (of 512 with heads of 256, whose weights are sharper). Weights without their low parts are off by 2^-10, one value
    in four rounds the other way, 2^-9 in the 2-norm; queries without theirs move scores, whose spread is sqrt(head_dim), by a
    percent and the weights as much. Measured on such kernels, 2-norm of the median row's difference: 2.2e-3 and more, 4.4e-3
    and more."""
    cfg = small_cfg(hidden=256, layers=1, heads=heads, kv_heads=kv_heads, head_dim=head_dim, inter=128, vocab=700, window=window,
                    layer_types=[kind])
    gpu, _ = build_pair(cfg, "bf16", kv_bf16=True, norm_jitter=0.1, want_oracle=False)
    tokens = syn.prompt_ids(700, 400, seed=head_dim)
    out = []
    for page in (16, 24):
        table = gpu.new_cache_table(400, page_tokens=page, kv_dtype=pkg.BF16)
        out.append(np.concatenate([gpu.extend(tokens[:270], table, want=list(range(270))), gpu.extend(tokens[270:], table, want=list(range(130)))]))
    rows = np.linalg.norm(out[0] - out[1], axis=1) / np.linalg.norm(out[1], axis=1)
    assert np.median(rows) <= 2.0 ** -10 and rows.max() <= 2.0 ** -7
