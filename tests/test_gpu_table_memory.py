"""Device memory of a cache table's workspace."""
import pytest

from util import build_pair, pkg, small_cfg

pytestmark = pytest.mark.gpu


def test_prompt_passes_hold_no_buffers_of_the_small_batch_kernels():
    """A pass of 2048 rows with 32768 gated columns needs them in BF16 (134 MB), a pass of up to 96 rows both projections' partial outputs
    (at most two splits, 50 MB). The small-batch kernels' f32 outputs (268 MB for 2048 rows) belong to the step's one row."""
    import torch
    gpu, _ = build_pair(small_cfg(hidden=128, layers=1, heads=2, kv_heads=1, head_dim=64, inter=32768, vocab=300, window=16), "bf16",
                        kv_bf16=True, want_oracle=False)
    gpu.new_cache_table(16, kv_dtype=pkg.BF16).close()      # kernels loaded
    for kv in (pkg.BF16, pkg.F32):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        table = gpu.new_cache_table(2048, kv_dtype=kv)
        torch.cuda.synchronize()
        assert before - torch.cuda.mem_get_info()[0] < 250e6
        table.close()
