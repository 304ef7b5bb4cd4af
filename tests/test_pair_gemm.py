"""GPU parity test of the SM-pair projection (tcgen05, cta_group::2) against a float64 matmul of the same BF16 values: whole
tiles and tiles cut over several pairs, ragged rows, columns and depths, gate and up in one launch."""
import ctypes as C

import numpy as np
import pytest

from util import pkg, syn

pytestmark = pytest.mark.gpu


def bf16(rng, shape, std):
    bits = syn.f32_to_bf16_bits((rng.standard_normal(shape) * std).astype(np.float32)).reshape(shape)
    return bits, syn.bf16_bits_to_f32(bits).reshape(shape).astype(np.float64)


def launch(w, w1, x, M):
    N, K = w.shape
    out, slots = np.zeros((M, N), dtype=np.float32), C.c_int32(0)
    p = lambda a: None if a is None else a.ctypes.data_as(C.c_void_p)  # noqa: E731
    pkg._native.check(pkg._native.lib().oxg4_debug_pair_gemm(p(w), p(w1), p(x), N, K, M, 0, p(out), C.byref(slots)))
    return out, slots.value


# (1, 8, 1): one value; 128 / 129 / 256 / 257 rows: edges of the CTA's and the pair's tile; K 64 / 72 / 2664: one k-block, a
# ragged last one; N 1003: scalar stores; the rest: tiles cut into ranges (slots > 1) and whole tiles in several rounds
@pytest.mark.parametrize("N,K,M", [(1, 8, 1), (256, 64, 128), (256, 72, 129), (512, 512, 256), (520, 136, 257), (1003, 2664, 999),
                                   (2560, 10240, 300), (1152, 6912, 97), (2560, 2048, 2048), (4104, 320, 2000)])
def test_store(N, K, M):
    rng = np.random.default_rng(N + K + M)
    (w, wd), (x, xd) = bf16(rng, (N, K), 0.05), bf16(rng, (M, K), 1.0)
    out, slots = launch(w, None, x, M)
    ref = xd @ wd.T
    # products are exact in f32; what differs is the order of K + slots additions
    assert slots >= 1 and np.isfinite(out).all()
    assert np.abs(out - ref).max() <= 2e-5 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("N,K,M", [(8, 8, 2), (1000, 72, 129), (1024, 520, 513), (6912, 1152, 300), (130, 256, 257)])
def test_gate_and_up(N, K, M):
    rng = np.random.default_rng(N + K + M)
    (w, wd), (w1, wd1), (x, xd) = bf16(rng, (N, K), 0.05), bf16(rng, (N, K), 0.05), bf16(rng, (M, K), 1.0)
    out, _ = launch(w, w1, x, M)
    g = xd @ wd.T
    ref = 0.5 * g * (1.0 + np.tanh(0.7978845608 * (g + 0.044715 * g ** 3))) * (xd @ wd1.T)
    # one rounding to BF16 (2^-9) on top of f32 arithmetic; near zero the f32 sums' absolute error
    assert (np.abs(out - ref) <= 2.0 ** -8 * np.abs(ref) + 1e-4 * np.abs(ref).max()).all()
