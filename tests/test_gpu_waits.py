"""Bounded waits of the tensor-core pipelines (csrc/tc_gemm.cuh). No GPU fault, trap or hang: every wait here has a limit, and what is
waited for is a flag that comes late or never."""
import ctypes as C
import time

import numpy as np
import pytest

from util import build_pair, pkg, small_cfg, syn

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def model():
    return build_pair(small_cfg(hidden=128, layers=2, heads=2, kv_heads=1, head_dim=64, inter=256, vocab=500, window=16), "bf16",
                      kv_bf16=True, want_oracle=False)[0]


def test_lanes_of_a_warp_hear_one_answer(model):
    """A phase completes after the budget of half the lanes ran out, and another one never: both times all lanes go on together with
    "ran out" (a lane on its own way would leave the rest of its warp at an .aligned instruction)."""
    table = model.new_cache_table(16, kv_dtype=pkg.BF16)
    N = pkg._native
    status = N.lib().oxg4_debug_wait_timeout(model._h, table._h, 1, 1000)
    assert N.STATUS_NAMES[status] == "TIMEOUT", N.lib().oxg4_last_error()
    assert b"mbarrier wait" in N.lib().oxg4_last_error()


@pytest.mark.parametrize("gate_up", [False, True])
@pytest.mark.parametrize("N,K,M", [(8, 8, 2), (520, 136, 257), (2560, 10240, 300), (4104, 320, 2000)])
def test_pair_projection_behind_a_failure_returns_without_output(N, K, M, gate_up):
    """One tile and many, whole and cut ones; a bounded wait that ran out in it would take a second."""
    w, x, out = np.zeros((N, K), dtype=np.uint16), np.zeros((M, K), dtype=np.uint16), np.zeros((M, N), dtype=np.float32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    fn, n = pkg._native.lib().oxg4_debug_pair_gemm, pkg._native.STATUS_NAMES
    assert n[fn(p(w), p(w) if gate_up else None, p(x), N, K, M, 0, p(out), None)] == "OK" and (out == 0).all()
    start = time.monotonic()
    assert n[fn(p(w), p(w) if gate_up else None, p(x), N, K, M, 4, p(out), None)] == "TIMEOUT"
    assert np.isnan(out).all() and time.monotonic() - start < 1.0
    assert n[fn(p(w), p(w) if gate_up else None, p(x), N, K, M, 0, p(out), None)] == "OK" and (out == 0).all()


def test_calls_behind_a_failure_report_it_and_the_next_ones_work(model):
    """A prompt on SM pairs with prompt attention, a short portion on the weight-streaming projections with the paged attention, and
    steps of eight sequences: each behind a set status word. No launch may use up a wait's limit (a second each)."""
    N = pkg._native
    tokens = syn.prompt_ids(500, 8 * 40, seed=3)
    lens = [40] * 8

    calls = [lambda table: model.prefill_prompt(tokens, table, lens=lens),
             lambda table: model.extend(tokens[:16], table, lens=[2] * 8, want=[15]),
             lambda table: model.decode_token(tokens[:8], table),
             lambda table: model.decode_greedy(tokens[:8], table, 4)[0]]
    new = lambda: model.new_cache_table([64] * 8, batch=8, page_tokens=16, kv_dtype=pkg.BF16)  # noqa: E731
    table = new()
    clean = [call(table) for call in calls]
    for i, call in enumerate(calls):
        table = new()
        for earlier in calls[:i]:
            earlier(table)
        N.check(N.lib().oxg4_debug_set_status(model._h, table._h, 12))
        start = time.monotonic()
        with pytest.raises(N.Oxg4Error, match="TIMEOUT"):
            call(table)
        assert time.monotonic() - start < 1.0
        table.reset()
        for again, want in zip(calls[:i + 1], clean):
            assert np.array_equal(again(table), want)


@pytest.mark.parametrize("kv", [pkg.F32, pkg.BF16])
@pytest.mark.parametrize("batch,ple", [(1, False), (1, True), (3, True), (9, True)])
def test_small_batch_projections_behind_a_failure_report_it(model, batch, ple, kv):
    """The same for calls whose BF16 projections are all of the small-batch kind, with and without tensor-core attention beside them: one
    sequence, and a model with per-layer embeddings with one, a few and more than eight rows."""
    N = pkg._native
    if ple:
        model = build_pair(syn.e_tiny_cfg(), "bf16", kv_bf16=True, want_oracle=False)[0]
    tokens = syn.prompt_ids(500, batch * 12, seed=4)
    calls = [lambda table: model.prefill_prompt(tokens, table, lens=[12] * batch),
             lambda table: model.decode_token(tokens[:batch], table),
             lambda table: model.decode_greedy(tokens[:batch], table, 3)[0],
             lambda table: model.decode_trace(tokens[:batch], table)[0]]
    if batch == 1:
        calls.append(lambda table: model.cached_attention_smoke(int(tokens[0]), 0, table))
    new = lambda: model.new_cache_table([32] * batch, batch=batch, page_tokens=16, kv_dtype=kv)  # noqa: E731
    table = new()
    clean = [call(table) for call in calls]
    for i, call in enumerate(calls):
        table = new()
        for earlier in calls[:i]:
            earlier(table)
        N.check(N.lib().oxg4_debug_set_status(model._h, table._h, 7))
        start = time.monotonic()
        with pytest.raises(N.Oxg4Error, match="TIMEOUT"):
            call(table)
        assert time.monotonic() - start < 1.0
        table.reset()
        for again, want in zip(calls[:i + 1], clean):
            assert np.array_equal(again(table), want)
