"""Bounded waits of the tensor-core pipelines (csrc/tc_gemm.cuh). No GPU fault, trap or hang: every wait here has a limit, and what is
waited for is a flag that comes late or never."""
import pytest

from util import build_pair, pkg, small_cfg

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
