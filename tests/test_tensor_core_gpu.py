"""The tensor-core kernel at the edges of its tiles: every way it forms the weight operand (bf16 rounded, f16
split in two, packed along the output columns), against the oracle's fp32 accumulation.

Sizes: one stage of 128 k and odd numbers of stages, token counts around 32, 128 and 256, output columns that
end inside a block's or a pair's half of a tile, one scale per stage at an odd position of its 4-byte
word, and few tiles with a long K (K shared by several pairs of thread blocks)."""
import numpy as np
import pytest
import torch

import mlx_b200 as mb
import oracle as O
from util import from_torch, make_w, make_x, qmm_close, to_torch, u32_to_torch

pytestmark = pytest.mark.gpu
DT = {"bf16": torch.bfloat16, "f16": torch.float16}


def check(dtype, M, N, K, g, bits, transpose, rel):
    w = make_w(M + N, (N, K) if transpose else (K, N), dtype)
    wq, s, b = O.quantize(w, g, bits, dtype)
    x = make_x(M + K, (M, K), dtype)
    if bits != 8 or (dtype == "bf16" and transpose):
        assert mb.qmm_kernel_name(DT[dtype], M, N, K, g, bits, transpose) == "qmm_tcgen05"
    ref = O.qmm_f32_from(x, wq, s, b, dtype, transpose=transpose, group_size=g, bits=bits)
    args = (to_torch(x, dtype), u32_to_torch(wq), to_torch(s, dtype), to_torch(b, dtype))
    for _ in range(2):   # the second call finds the counters and partial sums the first has left
        y = mb.quantized_matmul(*args, transpose=transpose, group_size=g, bits=bits)
    ok, err = qmm_close(O.to_f32(from_torch(y), dtype), ref, rel)
    assert ok, err


@pytest.mark.parametrize("bits", (2, 3, 4, 5, 6, 8))
@pytest.mark.parametrize("M,N,K,g", [(33, 130, 128, 128), (96, 257, 384, 128), (257, 385, 640, 64), (129, 128, 1152, 32)])
def test_transposed(bits, M, N, K, g):
    check("bf16", M, N, K, g, bits, True, 1e-2)
    check("f16", M, N, K, g, bits, True, 2e-3)   # the weights keep their fp32 value: only the result is rounded


@pytest.mark.parametrize("dtype,rel", [("bf16", 6e-3), ("f16", 2e-3)])
@pytest.mark.parametrize("bits", (2, 3, 4, 5, 6, 8))
@pytest.mark.parametrize("M,N,K,g", [(17, 128, 8, 128), (33, 384, 200, 64), (257, 256, 136, 32), (128, 640, 1000, 128)])
def test_not_transposed(dtype, rel, bits, M, N, K, g):
    check(dtype, M, N, K, g, bits, False, rel)


@pytest.mark.parametrize("dtype", ("bf16", "f16"))
@pytest.mark.parametrize("M,N,K,g,bits", [(57, 512, 8192, 64, 4), (40, 300, 5504, 128, 3), (200, 256, 4224, 32, 8)])
def test_k_shared_by_pairs_of_blocks(dtype, M, N, K, g, bits):
    check(dtype, M, N, K, g, bits, True, 1e-2)


@pytest.mark.parametrize("dtype", ("bf16", "f16"))
@pytest.mark.parametrize("M,N,K,g,bits,transpose", [(57, 19500, 1024, 64, 4, True), (40, 28601, 1152, 128, 3, True),
                                                    (600, 6300, 1152, 32, 8, True), (300, 9728, 1032, 64, 4, False)])
def test_tiles_left_over_from_whole_waves(dtype, M, N, K, g, bits, transpose):
    """One to 38 tiles more than there are pairs of blocks: their stages are cut into ranges that end inside tiles."""
    check(dtype, M, N, K, g, bits, transpose, 1e-2)


@pytest.mark.parametrize("bits", (5, 6, 8))
def test_experts_with_an_odd_number_of_stages(bits):
    """Nine stages per tile and several tiles per pair of blocks: the unpack warps' turns cross tile borders."""
    E, tokens, N, K, g = 16, 96, 640, 1152, 64
    wq, s, b = O.quantize(make_w(5, (E, N, K), "bf16"), g, bits, "bf16")
    x = to_torch(make_x(6, (tokens, 1, K), "bf16"), "bf16")
    wt, st, bt = u32_to_torch(wq), to_torch(s, "bf16"), to_torch(b, "bf16")
    rhs = torch.arange(tokens, device="cuda") * 7 % E
    y = mb.gather_qmm(x, wt, st, bt, rhs_indices=rhs, group_size=g, bits=bits)
    for e in range(E):
        rows = torch.nonzero(rhs == e).flatten()
        ref = O.qmm_f32_from(from_torch(x[rows, 0]), wq[e], s[e], b[e], "bf16", transpose=True, group_size=g, bits=bits)
        ok, err = qmm_close(O.to_f32(from_torch(y[rows, 0]), "bf16"), ref)
        assert ok, (e, err)


def at_odd_address(t):
    """The same values, contiguous, 2 bytes past a 16-byte boundary: a slice of a flat buffer."""
    flat = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    assert flat.data_ptr() % 16 == 0
    return flat[1:1 + t.numel()].view(t.shape).copy_(t)


@pytest.mark.parametrize("bits", (2, 3, 4, 5, 6, 8))
@pytest.mark.parametrize("E,tokens,N,K,g", [(2, 90, 65, 128, 128), (3, 70, 300, 640, 64), (4, 200, 200, 1152, 32), (3, 40, 65, 384, 128)])
def test_experts_with_scales_at_odd_addresses(bits, E, tokens, N, K, g):
    wq, s, b = O.quantize(make_w(7, (E, N, K), "bf16"), g, bits, "bf16")
    x = to_torch(make_x(8, (tokens, 1, K), "bf16"), "bf16")
    st, bt = at_odd_address(to_torch(s, "bf16")), at_odd_address(to_torch(b, "bf16"))
    rhs = torch.arange(tokens, device="cuda") * 5 % E
    for _ in range(2):   # through plain arrays of pairs, then through views of them
        y = mb.gather_qmm(x, u32_to_torch(wq), st, bt, rhs_indices=rhs, group_size=g, bits=bits)
        for e in range(E):
            rows = torch.nonzero(rhs == e).flatten()
            ref = O.qmm_f32_from(from_torch(x[rows, 0]), wq[e], s[e], b[e], "bf16", transpose=True, group_size=g, bits=bits)
            ok, err = qmm_close(O.to_f32(from_torch(y[rows, 0]), "bf16"), ref)
            assert ok, (e, err)


@pytest.mark.parametrize("bits", (3, 4, 8))
@pytest.mark.parametrize("dtype,transpose,rel", [("bf16", True, 1e-2), ("f16", True, 2e-3), ("bf16", False, 6e-3), ("f16", False, 2e-3)])
@pytest.mark.parametrize("M,N,K,g", [(40, 384, 640, 32), (64, 128, 1152, 128), (300, 256, 512, 64)])
def test_scales_at_odd_addresses(bits, dtype, transpose, rel, M, N, K, g):
    wq, s, b = O.quantize(make_w(M, (N, K) if transpose else (K, N), dtype), g, bits, dtype)
    x = make_x(K, (M, K), dtype)
    ref = O.qmm_f32_from(x, wq, s, b, dtype, transpose=transpose, group_size=g, bits=bits)
    y = mb.quantized_matmul(to_torch(x, dtype), u32_to_torch(wq), at_odd_address(to_torch(s, dtype)), at_odd_address(to_torch(b, dtype)),
                            transpose=transpose, group_size=g, bits=bits)
    ok, err = qmm_close(O.to_f32(from_torch(y), dtype), ref, rel)
    assert ok, err


@pytest.mark.parametrize("dtype", ("bf16", "f16"))
@pytest.mark.parametrize("M,N", [(33, 129), (40, 132), (100, 250), (257, 517), (300, 34), (600, 9477)])
def test_rows_of_y_off_16_byte_boundaries(dtype, M, N):
    """Widths that are no multiple of 8 (an output head): columns stored one by one; nothing past the last one."""
    import ctypes

    from mlx_b200 import _lib

    lib, P, K, g, bits = _lib.load(), lambda t: ctypes.c_void_p(t.data_ptr()), 384, 64, 4
    wq, s, b = O.quantize(make_w(M, (N, K), dtype), g, bits, dtype)
    x = make_x(N, (M, K), dtype)
    ref = O.qmm_f32_from(x, wq, s, b, dtype, transpose=True, group_size=g, bits=bits)
    xt, wt, st, bt = to_torch(x, dtype), u32_to_torch(wq), to_torch(s, dtype), to_torch(b, dtype)
    dt = {"bf16": _lib.BF16, "f16": _lib.F16}[dtype]
    ws = torch.zeros(lib.b200q_qmm_workspace_bytes(dt, 1, M, N, K, g, bits, 1), dtype=torch.uint8, device="cuda")
    for before in (0, 1, 8):   # y itself at 16, 2 and 16 bytes past a boundary
        flat = torch.full((before + M * N + 64,), 7.0, dtype=DT[dtype], device="cuda")
        y = flat[before:before + M * N].view(M, N)
        _lib.check(lib.b200q_qmm(P(xt), P(wt), P(st), P(bt), P(y), dt, 1, M, N, K, g, bits, 1, 0, P(ws), ws.numel(),
                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        ok, err = qmm_close(O.to_f32(from_torch(y), dtype), ref, 1e-2 if dtype == "bf16" else 2e-3)
        assert ok, err
        assert bool((flat[:before] == 7).all()) and bool((flat[before + M * N:] == 7).all())


def test_workspace_off_a_16_byte_boundary():
    """A caller's workspace may lie anywhere a 4-byte word may; its tiles are then not shared between pairs of blocks."""
    import ctypes

    from mlx_b200 import _lib

    lib, P = _lib.load(), lambda t: ctypes.c_void_p(t.data_ptr())
    M, N, K, g, bits = 57, 512, 8192, 64, 4   # few tiles, a long K
    wq, s, b = O.quantize(make_w(1, (N, K), "bf16"), g, bits, "bf16")
    x = make_x(2, (M, K), "bf16")
    need = lib.b200q_qmm_workspace_bytes(_lib.BF16, 1, M, N, K, g, bits, 1)
    ws = torch.zeros(need + 256, dtype=torch.uint8, device="cuda")[8:8 + need]
    xt, wt, st, bt = to_torch(x, "bf16"), u32_to_torch(wq), to_torch(s, "bf16"), to_torch(b, "bf16")
    y = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(lib.b200q_qmm(P(xt), P(wt), P(st), P(bt), P(y), _lib.BF16, 1, M, N, K, g, bits, 1, 0, P(ws), need, stream))
    ok, err = qmm_close(O.to_f32(from_torch(y), "bf16"), O.qmm_f32_from(x, wq, s, b, "bf16", transpose=True, group_size=g, bits=bits))
    assert ok, err
    assert int(ws.max()) == 0


def dense(wq, s, b, g, bits, dtype):
    """The weights in 64 bits."""
    K = wq.shape[-1] * 32 // bits
    stream = np.unpackbits(np.ascontiguousarray(wq).view(np.uint8), axis=-1, bitorder="little").reshape(wq.shape[0], K, bits)
    q = (stream.astype(np.float64) * 2.0 ** np.arange(bits)).sum(-1)
    wide = lambda t: np.repeat(O.to_f32(t, dtype).astype(np.float64), g, -1)
    return q * wide(s) + wide(b)


SPLIT = [("f16", True, 40, 257, 640, 64, 4), ("f16", True, 57, 512, 8192, 64, 4), ("f16", True, 300, 132, 512, 32, 3),
         ("f16", False, 64, 256, 392, 64, 6), ("f16", False, 300, 384, 1032, 128, 4), ("bf16", False, 64, 256, 392, 64, 4)]


@pytest.mark.parametrize("dtype,transpose,M,N,K,g,bits", SPLIT[:5])
def test_weights_beyond_the_range_of_half(dtype, transpose, M, N, K, g, bits):
    """Scales and biases are half precision, s*q+b need not be: some weights of a few rows lie between 65504 and 700000, x
    is small enough for every result to be a half.  Whole tiles, tiles shared between pairs of blocks, columns stored one by one."""
    rng = np.random.default_rng(M + K)
    rows, cols = (N, K) if transpose else (K, N)
    wq, s, b = O.quantize(make_w(M, (rows, cols), dtype), g, bits, dtype)
    sf = O.to_f32(s, dtype).copy()
    for r in rng.choice(rows, size=4, replace=False):
        sf[r, rng.integers(sf.shape[1])] = rng.uniform(2e4, 4e4)
    s = O.to_dtype(sf, dtype)
    w = dense(wq, s, b, g, bits, dtype)
    assert (np.abs(w) > 131008).any() and np.isfinite(w).all()
    x = O.to_dtype((rng.standard_normal((M, K)) * 1e-4).astype(np.float32), dtype)
    xf = O.to_f32(x, dtype).astype(np.float64)
    ref = xf @ (w.T if transpose else w)
    size = np.abs(xf) @ np.abs(w.T if transpose else w)
    got = mb.quantized_matmul(to_torch(x, dtype), u32_to_torch(wq), to_torch(s, dtype), to_torch(b, dtype), transpose=transpose,
                              group_size=g, bits=bits)
    got = O.to_f32(from_torch(got), dtype).astype(np.float64)
    # the result's rounding (2^-11 of it, 2^-25 where it is subnormal), and fp32 sums of K terms of that size in any order
    assert (np.abs(got - ref) <= 2.0 ** -11 * np.abs(ref) + 2.0 ** -25 + K * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("dtype,transpose,M,N,K,g,bits", SPLIT)
def test_activations_and_weights_that_are_not_finite(dtype, transpose, M, N, K, g, bits):
    """One infinity in a row of x times a weight is an infinity of the sign of both; so is one infinite bias; NaN stays NaN.
    The next call finds the workspace clear."""
    rng = np.random.default_rng(M + N)
    rows, cols = (N, K) if transpose else (K, N)
    wq, s, b = O.quantize(make_w(N, (rows, cols), dtype), g, bits, dtype)
    xf = rng.standard_normal((M, K)).astype(np.float32)
    xf[1, 3], xf[2, K - 1], xf[5, 7] = np.inf, -np.inf, np.nan
    bf = O.to_f32(b, dtype).copy()
    bf[rows - 2, 0] = np.inf
    x, b = O.to_dtype(xf, dtype), O.to_dtype(bf, dtype)
    w = dense(wq, s, b, g, bits, dtype)
    with np.errstate(invalid="ignore"):
        ref = O.to_f32(x, dtype).astype(np.float64) @ (w.T if transpose else w)
    odd = ~np.isfinite(ref)
    assert odd.any() and not odd.all()
    for _ in range(2):
        got = mb.quantized_matmul(to_torch(x, dtype), u32_to_torch(wq), to_torch(s, dtype), to_torch(b, dtype), transpose=transpose,
                                  group_size=g, bits=bits)
        got = O.to_f32(from_torch(got), dtype)
        assert np.array_equal(got[odd], ref[odd].astype(np.float32), equal_nan=True)
        ok, err = qmm_close(got[~odd], ref[~odd], 6e-3 if dtype == "bf16" else 2e-3)
        assert ok, err
    from mlx_b200 import ops
    assert int(ops._workspaces.get(torch.device("cuda", torch.cuda.current_device()), 0, "qmm").max()) == 0


def test_autograd_worker_thread():
    """The backward pass runs in a thread of its own, which has made no CUDA call yet."""
    from mlx_b200 import grad

    M, N, K = 64, 256, 384
    wq, s, b = O.quantize(make_w(8, (N, K), "bf16"), 64, 4, "bf16")
    x = to_torch(make_x(9, (M, K), "bf16"), "bf16").requires_grad_(True)
    dy = make_x(10, (M, N), "bf16")
    y = grad.quantized_matmul(x, u32_to_torch(wq), to_torch(s, "bf16"), to_torch(b, "bf16"))
    dx, = torch.autograd.grad(y, x, to_torch(dy, "bf16"))
    ref = O.qmm_f32_from(dy, wq, s, b, "bf16", transpose=False, group_size=64, bits=4)
    ok, err = qmm_close(O.to_f32(from_torch(dx), "bf16"), ref)
    assert ok, err


@pytest.mark.parametrize("M,bits,dtype,transpose", [(8, 4, "bf16", False), (8, 8, "f16", False), (64, 8, "bf16", False), (64, 4, "f16", True)])
def test_every_kernel_as_the_first_call_of_an_autograd_worker(M, bits, dtype, transpose):
    """A process of its own, so that nothing has used its worker thread before; the backward product is the row-owning
    kernel, the one for 8-bit weights, or the one for pairs of blocks."""
    import os
    import subprocess
    import sys

    code = f"""
import torch, mlx_b200 as mb
from mlx_b200 import grad
G = torch.Generator(device="cuda").manual_seed(1)
dt = {DT[dtype]}
w = mb.quantize(torch.randn(1024, 2048, generator=G, device="cuda", dtype=dt) * 0.02, 64, {bits})
x = torch.randn({M}, {2048 if transpose else 1024}, generator=G, device="cuda", dtype=dt, requires_grad=True)
dy = torch.randn({M}, {1024 if transpose else 2048}, generator=G, device="cuda", dtype=dt)
dx, = torch.autograd.grad(grad.quantized_matmul(x, *w, {transpose}, 64, {bits}), x, dy)
assert torch.equal(dx, mb.quantized_matmul(dy, *w, {not transpose}, 64, {bits}))
print("worker-ok")
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "worker-ok" in res.stdout, res.stdout + res.stderr
