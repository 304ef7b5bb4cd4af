"""Prompt passes of more than 96 rows of BF16 listed-layer models (csrc/pair_gemm.cuh around the mixers): against the plain
implementation, and against portions of at most 64 rows, which take the weight-streaming projections."""
import numpy as np
import pytest

from layered_util import Pair, attention, config, error, feed, latent, lightning, retention, wkv

pytestmark = pytest.mark.gpu

TOL = 3e-2                   # one layer in BF16, as in the tests of the single mechanisms
MODELS = {
    "wkv": [wkv(3, 20, ff=30)],
    "lightning": [lightning(3, 12, 28, (0.5, 0.93, 1.0), ff=50)],
    "latent": [latent(5, 24, 20, 36, 44, 10, ff=72)],
    "latent_512": [latent(9, 32, 128, 64, 512, 64, ff=16)],
    "retention": [retention(3, 12, 28, (0.5, 0.93, 1.0), ff=50)],
    "attention": [attention(6, 2, 24, 20, ff=40)],
}


@pytest.mark.parametrize("portions", [[97], [128, 257], [256, 1, 300]], ids=str)
@pytest.mark.parametrize("name", sorted(MODELS))
def test_portions(name, portions):
    """Row counts around the limit, a row tile and a slice; the second portion starts inside a filled cache."""
    pair = Pair(config(MODELS[name], width=100 if name != "wkv" else 64), "bf16", seed=13)
    tokens = pair.prompt(sum(portions))
    assert error(feed(pair, pair.table(len(tokens) + 2, page_tokens=48), tokens, portions), pair.want(tokens)) <= TOL


@pytest.mark.parametrize("name", sorted(MODELS))
def test_prompt_longer_than_a_pass(name):
    """2300 tokens: a pass of eight slices and one that goes on from its states, then a step."""
    pair = Pair(config(MODELS[name]), "bf16", seed=14)
    tokens = pair.prompt(2301)
    wide, narrow = pair.table(2304), pair.table(2304)
    got = [pair.state.prefill_prompt(tokens[:2300], wide), pair.state.decode_token(int(tokens[2300]), wide)]
    for at in range(0, 2300, 64):
        part = tokens[at:min(2300, at + 64)]
        want = pair.state.extend(part, narrow, want=[len(part) - 1])[0]
    want = [want, pair.state.decode_token(int(tokens[2300]), narrow)]
    for g, w in zip(got, want):
        assert error(g, w) <= TOL


@pytest.mark.parametrize("name", sorted(MODELS))
def test_unequal_prompts_of_one_pass(name):
    """Runs that begin and end anywhere in the slices, one of them across two borders, then a further portion of each."""
    lens, more = [1, 60, 530, 2, 64, 65, 127, 3], [5, 100, 130, 1, 64, 0, 33, 20]
    pair = Pair(config(MODELS[name]), "bf16", seed=15)
    seqs = [pair.prompt(a + b, seed=30 + i) for i, (a, b) in enumerate(zip(lens, more))]
    table = pair.table([len(s) + 1 for s in seqs], batch=len(seqs), page_tokens=32)
    got = pair.state.prefill_prompt(np.concatenate([s[:n] for s, n in zip(seqs, lens)]), table, lens=lens)
    ends = np.cumsum(more)
    fed = [i for i in range(len(seqs)) if more[i]]
    got2 = pair.state.extend(np.concatenate([s[n:] for s, n in zip(seqs, lens)]), table, lens=more, want=[int(ends[i]) - 1 for i in fed])
    for i, s in enumerate(seqs):
        want = pair.want(s)
        assert error(got[i], want[lens[i] - 1]) <= TOL, i
        if more[i]:
            assert error(got2[fed.index(i)], want[-1]) <= TOL, i
