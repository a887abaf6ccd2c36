"""Index pairs read in place: strided, broadcast, 32- and 64-bit and defaulted indices give what plain arrays of pairs
give, and the tile table of many experts (some without a row, one with several tiles) is right."""
import numpy as np
import pytest
import torch

import mlx_b200 as mb
import oracle as O
from util import from_torch, make_w, make_x, qmm_close, to_torch, u32_to_torch

pytestmark = pytest.mark.gpu


def setup(E, tokens, N, K, g=64, bits=4, seed=0):
    wq, s, b = O.quantize(make_w(50 + seed, (E, N, K), "bf16"), g, bits, "bf16")
    x = make_x(60 + seed, (tokens, 1, 1, K), "bf16")
    return x, (wq, s, b), to_torch(x, "bf16"), (u32_to_torch(wq), to_torch(s, "bf16"), to_torch(b, "bf16"))


def expected(x, q, lhs, rhs, g=64, bits=4):
    flat = x.reshape(-1, 1, x.shape[-1])
    return O.gather_qmm(O.to_f32(flat, "bf16"), q[0], O.to_f32(q[1], "bf16"), O.to_f32(q[2], "bf16"), lhs.ravel().astype(np.uint32),
                        rhs.ravel().astype(np.uint32), True, g, bits, "f32")


@pytest.mark.parametrize("kind", ("int64", "int32", "strided", "lhs_given", "column"))
def test_views(kind):
    E, tokens, top, N, K = 6, 40, 3, 200, 256
    x, q, xt, qt = setup(E, tokens, N, K)
    rhs = np.random.default_rng(1).integers(0, E, (tokens, top))
    lhs = np.broadcast_to(np.arange(tokens)[:, None], rhs.shape)
    rt = torch.from_numpy(rhs).cuda()
    kw = {}
    if kind == "int32":
        rt = rt.to(torch.int32)
    elif kind == "strided":
        rt = rt.t().contiguous().t()
    elif kind == "lhs_given":
        lhs = np.random.default_rng(2).integers(0, tokens, (tokens, 1))
        kw["lhs_indices"] = torch.from_numpy(lhs).cuda()
        lhs = np.broadcast_to(lhs, rhs.shape)
    elif kind == "column":
        rhs, rt = np.broadcast_to(rhs[:, :1], (tokens, 1)), rt[:, :1]
        lhs = lhs[:, :1]
    ref = expected(x, q, lhs, rhs)
    for _ in range(2):   # the second call finds the scratch buffer of the first and takes the native path
        y = mb.gather_qmm(xt, *qt, rhs_indices=rt, **kw)
        assert tuple(y.shape) == rhs.shape + (1, N)
        ok, err = qmm_close(O.to_f32(from_torch(y), "bf16").reshape(ref.shape), ref)
        assert ok, err


def test_many_experts_uneven():
    E, tokens, N, K = 300, 700, 64, 128
    x, q, xt, qt = setup(E, tokens, N, K, seed=1)
    rhs = np.random.default_rng(3).integers(0, E, tokens)
    rhs[:400] = 17        # several tiles of one expert
    rhs[rhs > 250] = 3    # and many experts without a row
    ref = expected(x, q, np.arange(tokens), rhs)
    xt3 = xt.reshape(tokens, 1, K)
    for _ in range(2):
        y = mb.gather_qmm(xt3, *qt, rhs_indices=torch.from_numpy(rhs).cuda())
        ok, err = qmm_close(O.to_f32(from_torch(y), "bf16").reshape(ref.shape), ref)
        assert ok, err


def test_gated_experts_native_equals_three_calls():
    E, tokens, top, H, K = 8, 5, 2, 256, 384
    _, _, xt, gate = setup(E, tokens, H, K, seed=2)
    up = setup(E, tokens, H, K, seed=3)[3]
    down = setup(E, tokens, K, H, seed=4)[3]
    idx = torch.from_numpy(np.random.default_rng(5).permuted(np.tile(np.arange(E), (tokens, 1)), axis=1)[:, :top].copy()).cuda()
    a, u = mb.gather_qmm(xt, *gate, rhs_indices=idx), mb.gather_qmm(xt, *up, rhs_indices=idx)
    h = (torch.nn.functional.silu(a.float()) * u.float()).to(torch.bfloat16)
    ref = mb.gather_qmm(h, *down, lhs_indices=torch.arange(tokens * top, device="cuda").reshape(tokens, top), rhs_indices=idx)
    for _ in range(2):
        y = mb.gather_qmm_swiglu(xt, gate, up, down, idx)
        assert tuple(y.shape) == (tokens, top, 1, K)
        assert torch.allclose(y.float(), ref.float(), rtol=2e-2, atol=2e-2 * float(ref.float().abs().max()))
