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


# Few rows per expert: tiles of up to 8 rows of the row-owning kernel.  Columns off the 16-row groups, one and two phases
# over K, every field width it has, an expert with more rows than a tile, one row in all, two rows per pair.
@pytest.mark.parametrize("E,tokens,top,rows,N,K,bits,group", [
    (8, 4, 2, 1, 200, 1024, 4, 64), (64, 1, 1, 1, 16, 1024, 4, 64), (16, 16, 4, 1, 1000, 512, 4, 32), (4, 5, 1, 2, 72, 12288, 4, 64),
    (8, 10, 2, 1, 136, 6144, 8, 128), (5, 7, 2, 1, 344, 3072, 2, 64), (32, 9, 1, 3, 64, 2048, 2, 128), (300, 500, 2, 1, 24, 512, 8, 32)])
def test_few_rows_per_expert(E, tokens, top, rows, N, K, bits, group):
    wq, s, b = O.quantize(make_w(70, (E, N, K), "bf16"), group, bits, "bf16")
    x = make_x(71, (tokens, rows, K), "bf16")
    rng = np.random.default_rng(72)
    rhs = rng.integers(0, E, (tokens, top))
    rhs[: min(tokens, 10)] = E - 1   # more than a tile of one expert, where there are enough
    lhs = np.broadcast_to(np.arange(tokens)[:, None], rhs.shape)
    ref = O.gather_qmm(O.to_f32(x, "bf16"), wq, O.to_f32(s, "bf16"), O.to_f32(b, "bf16"), lhs.ravel().astype(np.uint32),
                       rhs.ravel().astype(np.uint32), True, group, bits, "f32")
    args = to_torch(x, "bf16"), u32_to_torch(wq), to_torch(s, "bf16"), to_torch(b, "bf16")
    idx = {"lhs_indices": torch.from_numpy(lhs.copy()).cuda(), "rhs_indices": torch.from_numpy(rhs).cuda()}
    for _ in range(2):
        y = mb.gather_qmm(*args, **idx, group_size=group, bits=bits)
        ok, err = qmm_close(O.to_f32(from_torch(y), "bf16").reshape(ref.shape), ref)
        assert ok, err


@pytest.mark.parametrize("E,tokens,top,H,K,N2,bits", [(8, 4, 2, 1024, 1024, 200, 4), (16, 30, 2, 2048, 1024, 72, 4), (4, 1, 1, 3072, 6144, 16, 8),
                                                      (6, 11, 2, 2048, 12288, 40, 4)])
def test_few_rows_gated(E, tokens, top, H, K, N2, bits):
    make = lambda seed, shape: O.quantize(make_w(seed, shape, "bf16"), 64, bits, "bf16")
    dev = lambda q: (u32_to_torch(q[0]), to_torch(q[1], "bf16"), to_torch(q[2], "bf16"))
    gate, up, down = make(80, (E, H, K)), make(81, (E, H, K)), make(82, (E, N2, H))
    x = make_x(83, (tokens, 1, K), "bf16")
    rhs = np.random.default_rng(84).integers(0, E, (tokens, top))
    xt, rt = to_torch(x, "bf16")[:, None], torch.from_numpy(rhs).cuda()
    a, u = (mb.gather_qmm(xt, *dev(q), rhs_indices=rt, bits=bits).float() for q in (gate, up))
    h = (torch.nn.functional.silu(a) * u).to(torch.bfloat16).reshape(tokens * top, 1, H)
    ref = O.gather_qmm(O.to_f32(from_torch(h), "bf16"), down[0], O.to_f32(down[1], "bf16"), O.to_f32(down[2], "bf16"),
                       np.arange(tokens * top, dtype=np.uint32), rhs.ravel().astype(np.uint32), True, 64, bits, "f32")
    for _ in range(2):
        y = mb.gather_qmm_swiglu(xt, dev(gate), dev(up), dev(down), rt, bits=bits)
        assert tuple(y.shape) == (tokens, top, 1, N2)
        ok, err = qmm_close(O.to_f32(from_torch(y), "bf16").reshape(ref.shape), ref)
        assert ok, err


@pytest.mark.parametrize("bits,rows", [(2, 32), (4, 32), (4, 33), (8, 32), (8, 33)])
@pytest.mark.parametrize("skew", (False, True))
def test_both_sides_of_the_rule_for_few_rows(bits, rows, skew):
    """8 experts: the last number of rows that takes the row-owning kernel and the first that does not; routing spread
    evenly, and all rows on one expert."""
    E, N, K, g = 8, 264, 1024, 64
    wq, s, b = O.quantize(make_w(90, (E, N, K), "bf16"), g, bits, "bf16")
    x = make_x(91, (rows, 1, K), "bf16")
    rhs = np.full(rows, 5) if skew else np.arange(rows) * 3 % E
    ref = O.gather_qmm(O.to_f32(x, "bf16"), wq, O.to_f32(s, "bf16"), O.to_f32(b, "bf16"), np.arange(rows, dtype=np.uint32),
                       rhs.astype(np.uint32), True, g, bits, "f32")
    for _ in range(2):
        y = mb.gather_qmm(to_torch(x, "bf16"), u32_to_torch(wq), to_torch(s, "bf16"), to_torch(b, "bf16"),
                          rhs_indices=torch.from_numpy(rhs).cuda(), group_size=g, bits=bits)
        ok, err = qmm_close(O.to_f32(from_torch(y), "bf16").reshape(ref.shape), ref)
        assert ok, err
