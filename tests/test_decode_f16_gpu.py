"""Half-precision decode through the row-owning kernel: every instantiation, K in several phases, ragged rows, two
passes, and activations and biases at the ends of the half-precision range (x is scaled by a power of two per
warp and token, the bias sums travel as two half numbers)."""
import numpy as np
import pytest
import torch

import mlx_b200 as mb
import oracle as O
from util import from_torch, make_w, make_x, qmm_close, to_torch, u32_to_torch

pytestmark = pytest.mark.gpu


def product(x, q, g, bits):
    ref = O.qmm_f32_from(x, *q, "f16", transpose=True, group_size=g, bits=bits)
    y = mb.quantized_matmul(to_torch(x, "f16"), u32_to_torch(q[0]), to_torch(q[1], "f16"), to_torch(q[2], "f16"), group_size=g, bits=bits)
    return O.to_f32(from_torch(y), "f16"), ref


@pytest.mark.parametrize("bits,g", [(2, 64), (2, 128), (4, 32), (4, 64), (4, 128), (8, 32), (8, 64), (8, 128)])
@pytest.mark.parametrize("M,N,K", [(1, 2504, 4096), (8, 24, 2048), (9, 1000, 6144), (16, 67, 14336), (20, 520, 4096)])
def test_every_instantiation(bits, g, M, N, K):
    assert mb.qmm_kernel_name(torch.float16, M, N, K, g, bits) == "qmv_rows"
    got, ref = product(make_x(M + K, (M, K), "f16"), O.quantize(make_w(M + N, (N, K), "f16"), g, bits, "f16"), g, bits)
    ok, err = qmm_close(got, ref, 2e-3)   # the weights keep their fp32 value: only the result is rounded
    assert ok, err


@pytest.mark.parametrize("bits", (4, 8))
def test_range_of_half(bits):
    M, N, K, g = 4, 256, 2048, 64
    xf = np.random.default_rng(8).standard_normal((M, K)).astype(np.float32)
    xf[0] *= 300.0
    xf[1] *= 2.0 ** -14          # subnormal numbers among them
    xf[2, ::7] *= 2.0 ** 10
    x = O.to_dtype(xf, "f16")
    w = np.random.default_rng(9).standard_normal((N, K)).astype(np.float32) * 0.02 + 0.5   # large biases: they must not drown the rest
    got, ref = product(x, O.quantize(O.to_dtype(w, "f16"), g, bits, "f16"), g, bits)
    for m in range(M):           # rows differ by many binades: row by row
        if not np.isfinite(O.to_f32(O.to_dtype(ref[m], "f16"), "f16")).all():
            continue
        ok, err = qmm_close(got[m:m + 1], ref[m:m + 1], 2e-3)
        assert ok, (m, err)
