"""The streaming decode kernel against the oracle: widths that straddle bytes (bf16) and f16, at the edges of its
16-row tiles, of its K slices (a last slice that ends inside 256 k, K longer than one trip) and of its token tiles."""
import numpy as np
import pytest

import mlx_b200 as mb
import oracle as O
from util import col_scale, from_torch, make_w, make_x, qmm_close, to_torch, u32_to_torch

pytestmark = pytest.mark.gpu


def check(dtype, M, N, K, g, bits, rel):
    wq, s, b = O.quantize(make_w(M + N, (N, K), dtype), g, bits, dtype)
    x = make_x(M + K, (M, K), dtype)
    ref = O.qmm_f32_from(x, wq, s, b, dtype, transpose=True, group_size=g, bits=bits)
    y = mb.quantized_matmul(to_torch(x, dtype), u32_to_torch(wq), to_torch(s, dtype), to_torch(b, dtype), group_size=g, bits=bits)
    ok, err = qmm_close(O.to_f32(from_torch(y), dtype), ref, rel)
    assert ok, err


@pytest.mark.parametrize("bits", (3, 5, 6))
@pytest.mark.parametrize("M,N,K,g", [(1, 16, 256, 128), (2, 17, 384, 32), (3, 1000, 640, 32), (8, 47, 4224, 64), (9, 520, 1280, 128),
                                     (16, 2311, 2048, 64), (1, 333, 14336, 64)])
def test_bf16(bits, M, N, K, g):
    check("bf16", M, N, K, g, bits, 1e-2)


@pytest.mark.parametrize("bits", (2, 4, 8))
@pytest.mark.parametrize("M,N,K,g", [(1, 16, 256, 128), (2, 17, 512, 64), (3, 1000, 640, 64), (8, 47, 4224, 64), (9, 520, 1280, 128),
                                     (16, 2311, 2048, 64), (20, 333, 2816, 128), (1, 333, 14336, 64)])
def test_f16(bits, M, N, K, g):
    check("f16", M, N, K, g, bits, 2e-3)   # the weights keep their fp32 value: only the result is rounded


def test_scales_of_very_different_magnitude():
    """Scales with no room for the factor 2^133 take the general unpack, one branch per warp."""
    N, K, g, bits, M = 96, 1024, 64, 6, 4
    wf = np.random.default_rng(3).standard_normal((N, K)).astype(np.float32)
    wf *= (2.0 ** np.random.default_rng(4).integers(-24, 9, size=(N, 1))).astype(np.float32)
    wf[5] = 0.0
    wq, s, b = O.quantize(O.to_dtype(wf, "bf16"), g, bits, "bf16")
    x = make_x(41, (M, K), "bf16")
    ref = O.qmm_f32_from(x, wq, s, b, "bf16", transpose=True, group_size=g, bits=bits)
    y = mb.quantized_matmul(to_torch(x, "bf16"), u32_to_torch(wq), to_torch(s, "bf16"), to_torch(b, "bf16"), group_size=g, bits=bits)
    ok, err = qmm_close(O.to_f32(from_torch(y), "bf16"), ref, 1e-2, col_scale(wq, s, b, x, "bf16", g, bits)[None, :])
    assert ok, err
