"""The row-owning decode kernel where its forms and layouts can go wrong: widths whose fields straddle bytes and words, groups
kept apart in MMA columns, K in phases that end inside a warp's share, rows of scales off 16-byte boundaries, row counts that leave
a pair of rows half empty, and sums that are not finite."""
import numpy as np
import pytest
import torch

import mlx_b200 as mb
import oracle as O
from util import from_torch, make_w, make_x, qmm_close, to_torch, u32_to_torch

pytestmark = pytest.mark.gpu
DT = {"bf16": torch.bfloat16, "f16": torch.float16}


def product(dtype, M, N, K, g, bits, seed=0, x=None):
    wq, s, b = O.quantize(make_w(M + N + seed, (N, K), dtype), g, bits, dtype)
    x = make_x(M + K, (M, K), dtype) if x is None else x
    assert mb.qmm_kernel_name(DT[dtype], M, N, K, g, bits) == "qmv_rows"
    ref = O.qmm_f32_from(x, wq, s, b, dtype, transpose=True, group_size=g, bits=bits)
    for _ in range(2):
        y = mb.quantized_matmul(to_torch(x, dtype), u32_to_torch(wq), to_torch(s, dtype), to_torch(b, dtype), group_size=g, bits=bits)
    return O.to_f32(from_torch(y), dtype), ref


def norm_error(got, ref):
    return np.linalg.norm(got.astype(np.float64) - ref) / np.linalg.norm(ref)


def limit(dtype, n):
    """Of norm_error over n results where the weights keep their value and only the result is rounded, to 8 bits or to 11.  An error is
    spread evenly over the unit in the last place: 2^-8 / sqrt(3) (2^-11 / sqrt(3)) binades over the mantissas' root mean square,
    which is 1.36 at least: 1.66e-3 (2.07e-4).  The squares of evenly spread errors deviate by 0.9 of their mean and the largest third
    of normally spread results carries the norm, so n results deviate by 0.45 sqrt(3 / n) of it: four times that.  (Weights rounded to
    8 bits as well: 2.1e-3 and more.)"""
    return (1.66e-3 if dtype == "bf16" else 2.07e-4) * (1 + 3.1 / np.sqrt(n)) + 1e-5   # fp32 sums


def check(dtype, *args, **kw):
    got, ref = product(dtype, *args, **kw)
    assert norm_error(got, ref) < limit(dtype, ref.size), norm_error(got, ref)
    assert qmm_close(got, ref, 1e-2)[0]


@pytest.mark.parametrize("dtype", ("bf16", "f16"))
@pytest.mark.parametrize("bits,g", [(b, g) for b in (3, 5, 6) for g in (32, 64, 128)] + [(2, 32)])
@pytest.mark.parametrize("M,N,K", [(1, 1031, 128), (2, 17, 2176), (4, 250, 4224), (3, 8, 8448)])
def test_runs(dtype, bits, g, M, N, K):
    """One chunk of 128, 17 and 33 (a warp's second chunk, or a second phase, that most warps do not have), 66 in phases."""
    check(dtype, M, N, K, g, bits)


@pytest.mark.parametrize("dtype", ("bf16", "f16"))
@pytest.mark.parametrize("M,K", [(1, 4608), (8, 8192), (3, 8192)])
def test_two_bits_with_all_of_a_long_row_in_one_phase(dtype, M, K):
    """Groups of 64 from 16384 output columns on; shares that end early, a last row group of one row."""
    check(dtype, M, 16385, K, 64, 2)


@pytest.mark.parametrize("dtype", ("bf16", "f16"))
@pytest.mark.parametrize("M,g,bits", [(8, 64, 5), (5, 64, 3), (16, 128, 6), (9, 128, 3)])
def test_runs_in_two_column_tiles(dtype, M, g, bits):
    check(dtype, M, 300, 2304, g, bits)


@pytest.mark.parametrize("dtype", ("bf16", "f16"))
@pytest.mark.parametrize("bits,g,K", [(4, 32, 128), (4, 64, 384), (4, 128, 1792), (4, 64, 6912), (8, 32, 256), (8, 128, 4480), (8, 64, 5248),
                                      (2, 64, 3328), (2, 128, 384), (2, 64, 17408), (2, 128, 4224), (2, 128, 8192), (4, 128, 16768), (8, 64, 11136)])
@pytest.mark.parametrize("M,N", [(1, 9), (8, 1201), (11, 100)])
def test_units_with_k_of_any_length(dtype, bits, g, K, M, N):
    """Fewer groups than warps, shares that end early, odd numbers of groups (scales at 2-byte addresses), several phases."""
    check(dtype, M, N, K, g, bits)


@pytest.mark.parametrize("dtype,top", [("bf16", 3e38), ("f16", 6e4)])
@pytest.mark.parametrize("bits,g", [(4, 64), (6, 32), (8, 128), (2, 32)])
def test_infinite_and_largest_activations(dtype, top, bits, g):
    """An infinite x times a weight has the weight's sign; a token with the type's largest number among small ones stays finite where
    the sum is, and a NaN stays in its token.  The factored sums alone give NaN for the first."""
    M, N, K = 4, 130, 1280
    xf = O.to_f32(make_x(3, (M, K), dtype), dtype).astype(np.float32)
    xf[0, 77] = np.inf
    xf[1, 5] = top
    xf[2, 300] = np.nan
    x = O.to_dtype(xf, dtype)
    wq, s, b = O.quantize(make_w(5, (N, K), dtype), g, bits, dtype)
    y = mb.quantized_matmul(to_torch(x, dtype), u32_to_torch(wq), to_torch(s, dtype), to_torch(b, dtype), group_size=g, bits=bits)
    got = O.to_f32(from_torch(y), dtype)
    product_of = lambda rows: O.qmm_f32_from(O.to_dtype(rows, dtype), wq, s, b, dtype, transpose=True, group_size=g, bits=bits)
    one = np.zeros((1, K), np.float32)
    one[0, 77] = 1.0
    w = product_of(one)[0]   # the weights' own values
    assert np.array_equal(got[0][w != 0], np.where(w > 0, np.inf, -np.inf)[w != 0].astype(np.float32))
    ref = product_of(xf[1:2])[0]
    finite = np.abs(ref) < (3e38 if dtype == "bf16" else 6.5e4)
    # the result's rounding; and where the two parts of the sum cancel (s * sum of x q, b * sum of x), what fp32 loses of each: a group's
    # sums, the largest x among them, pass up to 8 MMAs, which bring 17 addends to the largest one's exponent and may cut each off there
    part = float(np.abs(xf[1]).max()) * float((np.abs(O.to_f32(s, dtype)) * (2 ** bits - 1) + np.abs(O.to_f32(b, dtype))).max())
    assert finite.any() and np.allclose(got[1][finite], ref[finite], rtol=2.0 ** (-8 if dtype == "bf16" else -11), atol=8 * 17 * 2.0 ** -24 * part)
    assert np.isnan(got[2]).all()
    ref = O.qmm_f32_from(x[3:], wq, s, b, dtype, transpose=True, group_size=g, bits=bits)
    assert qmm_close(got[3:], ref, 1e-2)[0]


@pytest.mark.parametrize("bits,g", [(3, 64), (6, 32), (2, 32), (4, 64), (8, 128)])
@pytest.mark.parametrize("x_exp,s_exp", [(0, -100), (0, -115), (60, -120), (-60, -50), (-40, 60), (100, -20), (-100, 110)])
def test_results_of_any_magnitude(bits, g, x_exp, s_exp):
    """Activations and weights at the ends of what bf16 holds: results that are normal numbers have the bits of the same product nearer
    to 1, scaled by the power of two.  (The sums are kept times a power of two, which must not take them below fp32's range.)"""
    M, N, K = 3, 70, 2304
    G = torch.Generator(device="cuda").manual_seed(bits)
    x = torch.randn(M, K, generator=G, device="cuda").bfloat16()
    wq, s, b = mb.quantize(torch.randn(N, K, generator=G, device="cuda").bfloat16(), g, bits)
    ref = mb.quantized_matmul(x, wq, s, b, group_size=g, bits=bits)
    f = lambda t, e: torch.ldexp(t.double(), torch.tensor(e, device="cuda")).bfloat16()
    got = mb.quantized_matmul(f(x, x_exp), wq, f(s, s_exp), f(b, s_exp), group_size=g, bits=bits)
    want = f(ref, x_exp + s_exp)
    # (half a unit in the last place of either, where a tie or the order of sums computed again decides)
    assert float((got.double() - want.double()).norm() / want.double().norm()) < 2.0 ** -8


@pytest.mark.parametrize("bits,g", [(4, 64), (6, 128), (2, 32)])
@pytest.mark.parametrize("dtype", ("bf16", "f16"))
def test_nan_costs_no_time(dtype, bits, g):
    """A NaN in a row of x, the last element of it, leaves the launch as long as it is: nothing is computed again for what stays NaN.
    (Every output once more from the weights is a hundred times the product; the bound is far from both.)  Other rows are as without."""
    M, N, K = 4, 14336, 4096
    x = torch.randn(M, K, device="cuda").to(DT[dtype])
    w = mb.quantize((torch.randn(N, K, device="cuda") * 0.02).to(DT[dtype]), g, bits)
    bad = x.clone()
    bad[:3, -1] = float("nan")
    ref, got = (mb.quantized_matmul(v, *w, group_size=g, bits=bits) for v in (x, bad))
    assert got[:3].isnan().all() and torch.equal(got[3], ref[3])

    def us(v):
        t = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                mb.quantized_matmul(v, *w, group_size=g, bits=bits)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b) * 100)
        return min(t)

    assert us(bad) < 8 * us(x), (us(bad), us(x))


@pytest.mark.parametrize("bits,g", [(4, 64), (3, 64), (8, 128)])
def test_sums_that_are_not_finite_in_several_tiles(bits, g):
    """Infinities in some of 16 rows, which two warps sum, and in rows of a gated expert layer: each result is the weights' sign times
    infinity, and rows without one keep their bits."""
    M, N, K = 16, 270, 4352
    if bits == 3:
        M = 8
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = mb.quantize(torch.randn(N, K, device="cuda", dtype=torch.bfloat16) * 0.02, g, bits)
    ref = mb.quantized_matmul(x, *w, group_size=g, bits=bits)
    W = mb.dequantize(*w, g, bits).float()
    rows = [1, M - 2]
    bad = x.clone()
    for i in rows:
        bad[i, 300 * i] = float("-inf")
    got = mb.quantized_matmul(bad, *w, group_size=g, bits=bits)
    for i in range(M):
        if i in rows:
            sign = W[:, 300 * i]
            assert torch.equal(got[i][sign != 0], torch.where(sign > 0, float("-inf"), float("inf")).bfloat16()[sign != 0])
        else:
            assert torch.equal(got[i], ref[i])
    E = 3
    G = torch.Generator(device="cuda").manual_seed(bits)
    mk = lambda a, c: mb.quantize(torch.randn(E, a, c, generator=G, device="cuda", dtype=torch.bfloat16) * 0.02, g, bits)
    gate, up = mk(256, K), mk(256, K)
    down = mk(K, 256)
    xe = x[:6].view(6, 1, 1, K).clone()
    idx = torch.tensor([0, 1, 2, 0, 1, 2], device="cuda").view(6, 1)
    ref = mb.gather_qmm_swiglu(xe, gate, up, down, idx, group_size=g, bits=bits)
    xe[4, 0, 0, 7] = float("inf")
    xe[2, 0, 0, 9] = float("nan")
    got = mb.gather_qmm_swiglu(xe, gate, up, down, idx, group_size=g, bits=bits)
    assert got[2].isnan().all() and not got[4].isfinite().any()
    for i in (0, 1, 3, 5):
        assert torch.equal(got[i], ref[i])


@pytest.mark.parametrize("bits,g,K", [(3, 32, 640), (6, 64, 1152), (5, 128, 1280), (2, 32, 384), (4, 128, 1792), (8, 64, 4224)])
@pytest.mark.parametrize("gated", (False, True))
def test_experts(bits, g, K, gated):
    """Few rows per expert (none for some, more than a tile's for one), K that is no whole turn of the warps; gated: both products of a
    row group meet in one warp."""
    E, H, tokens = 9, 384, 18
    G = torch.Generator(device="cuda").manual_seed(bits + g)
    draw = lambda a, c: torch.randn(E, a, c, generator=G, device="cuda", dtype=torch.bfloat16) * 0.02
    idx = (torch.arange(tokens, device="cuda") * 5 % (E - 1)).view(tokens, 1)
    idx[:10] = 3
    x = torch.randn(tokens, 1, 1, K, generator=G, device="cuda", dtype=torch.bfloat16)
    q = {"group_size": g, "bits": bits}
    gate, up = mb.quantize(draw(H, K), **q), mb.quantize(draw(H, K), **q)
    if gated:
        down = mb.quantize(draw(K, H), **q)
        y = mb.gather_qmm_swiglu(x, gate, up, down, idx, **q)
        # the same from separate products, whose roundings are the same
        a = mb.gather_qmm(x, *gate, rhs_indices=idx, **q).float()
        c = mb.gather_qmm(x, *up, rhs_indices=idx, **q).float()
        h = (a * torch.sigmoid(a) * c).to(torch.bfloat16)
        ref = mb.gather_qmm(h, *down, lhs_indices=torch.arange(tokens, device="cuda").view(tokens, 1), rhs_indices=idx, **q)
        err = float((y.float() - ref.float()).norm() / ref.float().norm())
        assert err < 1e-2, err
    else:
        y = mb.gather_qmm(x, *gate, rhs_indices=idx, **q)
        wq, s, b = (from_torch(t) for t in gate)
        for e in range(E - 1):
            rows = torch.nonzero(idx[:, 0] == e).flatten()
            if len(rows):
                ref = O.qmm_f32_from(from_torch(x[rows, 0, 0]), wq[e].view(np.uint32), s[e], b[e], "bf16", transpose=True, group_size=g, bits=bits)
                assert norm_error(O.to_f32(from_torch(y[rows, 0, 0]), "bf16"), ref) < limit("bf16", ref.size)


@pytest.mark.parametrize("bits,g,line", [(2, 64, 8), (4, 64, 6), (8, 64, 6), (3, 128, 6), (6, 64, 4), (6, 32, 2), (2, 32, 2)])
@pytest.mark.parametrize("beyond", (0, 1))
def test_experts_on_both_sides_of_the_rule_for_few_rows(bits, g, line, beyond):
    """The last row count of the row-owning kernel (tiles full, an expert with more rows than a tile's) and the first of the
    tensor-core kernel, which rounds the weights."""
    E, N, K = 3, 100, 384
    rows = line * E + beyond
    wq, s, b = O.quantize(make_w(bits, (E, N, K), "bf16"), g, bits, "bf16")
    x = make_x(line, (rows, 1, K), "bf16")
    idx = np.sort(np.arange(rows) % (E + 1)) % E   # expert 0 has about twice the others' rows
    y = mb.gather_qmm(to_torch(x, "bf16"), u32_to_torch(wq), to_torch(s, "bf16"), to_torch(b, "bf16"),
                      rhs_indices=torch.from_numpy(idx.astype(np.int64)).cuda(), group_size=g, bits=bits)
    for e in range(E):
        mine = np.flatnonzero(idx == e)
        ref = O.qmm_f32_from(x[mine, 0], wq[e], s[e], b[e], "bf16", transpose=True, group_size=g, bits=bits)
        got = O.to_f32(from_torch(y[torch.from_numpy(mine).cuda(), 0]), "bf16")
        assert qmm_close(got, ref, 1e-2)[0]
        if not beyond:
            assert norm_error(got, ref) < limit("bf16", ref.size)
