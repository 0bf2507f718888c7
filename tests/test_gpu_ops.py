"""Numerics of the sm_100a compute kernels against plain PyTorch fp32 references
computed from the same bf16 inputs.  Tolerances are those of one bf16 rounding of
the output (2^-8 relative) plus fp32 accumulation-order noise."""

import contextlib
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def close(got, want, rtol=1.6e-2, atol=1e-2, frobenius=1.5e-2):
    """Element-wise bound (absolute part scaled by the largest entry) AND a bound on the relative Frobenius error: the
    first alone would let small entries be entirely wrong."""
    got, want = got.float(), want.float()
    err = (got - want).abs()
    tol = atol * want.abs().max().clamp_min(1e-6) + rtol * want.abs()
    assert bool((err <= tol).all()), f"max err {err.max().item():.4g} (|want| max {want.abs().max().item():.4g})"
    if want.norm().item() > 0:
        rel = (err.norm() / want.norm()).item()
        assert rel <= frobenius, f"relative Frobenius error {rel:.4g} > {frobenius}"


def gelu_slope(x):
    """d/dx of the exact GELU: Phi(x) + x * phi(x)."""
    x = x.float()
    return 0.5 * (1 + torch.erf(x * 0.7071067811865476)) + x * torch.exp(-0.5 * x * x) * 0.3989422804014327


def rnd(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).bfloat16()


@pytest.fixture(autouse=True)
def no_gemm_timeouts():
    yield
    from tandem_b200.ops.gemm import gemm_error

    torch.cuda.synchronize()
    assert not gemm_error(), "a GEMM wait ran out"


@pytest.fixture(autouse=True)
def planner_left_alone():
    """Whatever a test pins (tile shape, number of k-parts) is unpinned again when it ends, also when it fails."""
    yield
    from tandem_b200.ops._lib import lib

    lib().tb_gemm_force_tile(-1)
    lib().tb_gemm_force_splits(0)


@pytest.fixture
def force_tile():
    """Pins the GEMM's tile shape (0: 256x256, 1: 128x256, 2: 128x128, 3/4: CTA-pair 256x256 / 256x128, 5: 128x192) for one test."""
    from tandem_b200.ops._lib import lib

    yield lib().tb_gemm_force_tile
    lib().tb_gemm_force_tile(-1)


@pytest.mark.parametrize("tile", [-1, 0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (128, 256, 128), (256, 384, 768), (1024, 2304, 768), (512, 65, 768),
                                   (384, 768, 3072), (130, 72, 200)])
def test_gemm_three_layouts(M, N, K, tile, force_tile):
    from tandem_b200.ops._lib import empty_padded
    from tandem_b200.ops.gemm import gemm

    force_tile(tile)

    def padded(rows, cols):
        t = empty_padded(rows, cols, torch.bfloat16, "cuda")
        t.copy_(rnd(rows, cols, scale=0.5))
        return t

    a, b = padded(M, K), padded(N, K)  # forward: A K-major, B K-major
    out = gemm(a, b, M, N, K, a.stride(0), b.stride(0), False, False)
    close(out, a.float() @ b.float().t())
    bt = padded(K, N)  # dX-style: B is [K, N] with N contiguous
    out = gemm(a, bt, M, N, K, a.stride(0), bt.stride(0), False, True)
    close(out, a.float() @ bt.float())
    at = padded(K, M)  # dW-style: both MN-major
    out = gemm(at, bt, M, N, K, at.stride(0), bt.stride(0), True, True)
    close(out, at.float().t() @ bt.float())
    out32 = gemm(at, bt, M, N, K, at.stride(0), bt.stride(0), True, True, out_dtype=torch.float32)
    close(out32, at.float().t() @ bt.float(), rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("splits", [2, 3, 8])
@pytest.mark.parametrize("tile", [-1, 0, 1, 2, 5])
@pytest.mark.parametrize("M,N,K", [(768, 768, 8192), (384, 200, 2048), (130, 72, 4096), (1024, 2304, 768)])
def test_gemm_split_k(M, N, K, splits, tile, force_tile):
    """The reduction cut into parts inside one kernel: producers park fp32 partial tiles, the consumer folds them in and runs
    the epilogue.  Weight-gradient shapes (both operands MN-major) and a forward shape with bias, GELU and residual."""
    from tandem_b200.ops import gemm as G
    from tandem_b200.ops._lib import empty_padded, lib

    force_tile(tile)
    lib().tb_gemm_force_splits(splits)
    try:
        a2, b2 = empty_padded(K, M, torch.bfloat16, "cuda"), empty_padded(K, N, torch.bfloat16, "cuda")
        a2.copy_(rnd(K, M, scale=0.5)), b2.copy_(rnd(K, N, scale=0.5))
        want = a2.float().t() @ b2.float()
        out = G.gemm(a2, b2, M, N, K, a2.stride(0), b2.stride(0), True, True)
        close(out, want)
        again = G.gemm(a2, b2, M, N, K, a2.stride(0), b2.stride(0), True, True)
        assert torch.equal(out, again)  # the parts are folded in a fixed order
        acc = torch.ones_like(out)
        G.gemm(a2, b2, M, N, K, a2.stride(0), b2.stride(0), True, True, G.ACCUMULATE, out=acc)
        close(acc, want + 1)
        if N % 8 == 0:
            x, w, bias, res = rnd(M, K, scale=0.5), rnd(N, K, scale=0.5), rnd(N), rnd(M, N)
            ref = x.float() @ w.float().t() + bias.float()
            close(G.gemm(x, w, M, N, K, K, K, False, False, G.BIAS | G.RESIDUAL, bias, res), ref + res.float())
            slope = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
            act = G.gemm(x, w, M, N, K, K, K, False, False, G.BIAS | G.GELU, bias, None, slope)
            close(slope, gelu_slope(ref))
            close(act, torch.nn.functional.gelu(ref))
    finally:
        lib().tb_gemm_force_splits(0)


@pytest.mark.parametrize("tile", [0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("M,N,K", [(2300, 1100, 136), (1281, 3000, 64), (4224, 4200, 72)])
def test_gemm_raster_and_edges(M, N, K, tile, force_tile):
    """Several raster groups, the last one short, and an unfinished last column of tiles; rows and columns that fit no tile, chunks
    that start beyond the last column, bias and aux at the edges.  Sums of at most 136 products: fp32 order is far below the
    bf16 rounding that `close` allows for."""
    from tandem_b200.ops import gemm as G
    from tandem_b200.ops._lib import empty_padded

    force_tile(tile)
    x, w, bias = rnd(M, K, scale=0.5), rnd(N, K, scale=0.5), rnd(N)
    res = empty_padded(M, N, torch.bfloat16, "cuda")
    res.copy_(rnd(M, N))
    ref = x.float() @ w.float().t() + bias.float()
    close(G.gemm(x, w, M, N, K, K, K, False, False, G.BIAS, bias), ref)
    out = empty_padded(M, N, torch.bfloat16, "cuda")
    close(G.gemm(x, w, M, N, K, K, K, False, False, G.BIAS | G.RESIDUAL, bias, res, out=out), ref + res.float())
    close(G.gemm(x, w, M, N, K, K, K, False, False, G.DGELU, None, res, out=out), (ref - bias.float()) * res.float())
    slope = empty_padded(M, N, torch.bfloat16, "cuda")
    close(G.gemm(x, w, M, N, K, K, K, False, False, G.BIAS | G.GELU, bias, None, slope, out=out), torch.nn.functional.gelu(ref))
    close(slope, gelu_slope(ref))


@pytest.mark.parametrize("tile", [0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("M,N", [(33, 72), (700, 1090), (3900, 4168)])
def test_gemm_accumulates_in_place(M, N, tile, force_tile):
    """The output's old values come in through the blocks that the sums leave from: fewer blocks than chunks, clipped chunks and
    rows, several tiles per CTA.  Sums of 64 products of -1, 0 and 1 and a small integer are exact in bf16."""
    from tandem_b200.ops import gemm as G
    from tandem_b200.ops._lib import empty_padded

    force_tile(tile)
    x, w = (torch.randint(-1, 2, (rows, 64), device="cuda").bfloat16() for rows in (M, N))
    out = empty_padded(M, N, torch.bfloat16, "cuda")
    old = torch.randint(-8, 9, (M, N), device="cuda").bfloat16()
    out.copy_(old)
    want = old.float()
    for _ in range(3):
        G.gemm(x, w, M, N, 64, 64, 64, False, False, G.ACCUMULATE, out=out)
        want = want + x.float() @ w.float().t()
        assert torch.equal(out.float(), want)


@pytest.mark.parametrize("exponent", [0, 1, 8, 64, 99])
def test_gelu_reciprocal_against_a_division(exponent):
    """Every significand at a few powers of two (a power of two scales the whole computation exactly): one Newton step from an
    approximation within one unit in the last place rounds correctly, but for the significand of all ones."""
    from tandem_b200.ops._lib import lib

    d = (torch.arange(1 << 23, device="cuda", dtype=torch.int32) + ((127 + exponent) << 23)).view(torch.float32)
    d = d.clamp(max=1e30)
    out = torch.empty_like(d)
    assert lib().tb_gemm_reciprocals(d.data_ptr(), out.data_ptr(), d.numel(), torch.cuda.current_stream().cuda_stream) == 0
    want = (1 / d.double()).float()  # never near a rounding tie: 1 / d is at least 2^-48 away from one
    off = (out.view(torch.int32) - want.view(torch.int32)).abs()
    assert off[:-1].max() == 0 and off[-1] <= 1


@pytest.mark.parametrize("tile,N", [(5, 384), (2, 96), (1, 160), (4, 352), (3, 416), (0, 288)])
def test_gemm_store_blocks_with_odd_chunk_counts(tile, N, force_tile):
    """Six tiles and more per CTA whose epilogue warps write an odd number of 32-column blocks each: a tile's first block is the
    one that the tile before stored last.  One k-block, so that the epilogue follows on the tile before at once.  Sums of 64
    products of -1, 0 and 1 are exact in bf16."""
    from tandem_b200.ops import gemm as G

    force_tile(tile)
    M, K = 148 * 128 * 6, 64
    x, w = (torch.randint(-1, 2, (rows, K), device="cuda").bfloat16() for rows in (M, N))
    res = torch.randint(-1, 2, (M, N), device="cuda").bfloat16()
    ref = x.float() @ w.float().t()
    for _ in range(4):
        assert torch.equal(G.gemm(x, w, M, N, K, K, K, False, False).float(), ref)
        assert torch.equal(G.gemm(x, w, M, N, K, K, K, False, False, G.RESIDUAL, None, res).float(), ref + res.float())


def test_gelu_epilogue_at_the_extremes(force_tile):
    """GELU and its derivative where the reciprocal and the exponential saturate, and for infinities and NaN."""
    from tandem_b200.ops import gemm as G

    M, N, K = 128, 128, 64
    values = torch.tensor([0.0, 1e-20, 0.5, 3.0, 9.0, 60.0, 1e4, 1e20, 3e38, float("inf"), float("nan")], device="cuda").bfloat16()
    values = torch.cat([values, -values])
    x = torch.zeros(M, K, device="cuda", dtype=torch.bfloat16)
    w = torch.zeros(N, K, device="cuda", dtype=torch.bfloat16)
    bias = torch.zeros(N, device="cuda", dtype=torch.bfloat16)
    bias[:values.numel()] = values
    slope = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    out = G.gemm(x, w, M, N, K, K, K, False, False, G.BIAS | G.GELU, bias, None, slope)
    v = values.double()
    cdf = 0.5 * torch.special.erfc(-v / 2**0.5)
    want, want_slope = v * cdf, cdf + v * torch.exp(-v * v / 2) / (2 * torch.pi) ** 0.5
    got, got_slope = out[5, :v.numel()].double(), slope[5, :v.numel()].double()
    finite = v.isfinite()
    # the formula's 1.5e-7 absolute error, times |x| for gelu, and one bf16 rounding
    assert ((got - want).abs()[finite] <= 2.0**-8 * want.abs()[finite] + 2e-7 * v.abs()[finite].clamp(min=1)).all()
    assert ((got_slope - want_slope).abs()[finite] <= 2.0**-8 * want_slope.abs()[finite] + 1e-6).all()
    assert got[v == float("inf")].item() == float("inf") and got[v.isnan()].isnan().all()


SPLIT = [(3, 2), (3, 8), (4, 3), (4, 2)]  # CTA-pair tile shape, parts


@pytest.mark.parametrize("M,N,K,tile,splits", [(*shape, *how) for shape in [(768, 768, 8192), (384, 200, 2048), (130, 72, 4096), (21100, 250, 2048)] for how in SPLIT]
                         + [(2304, 1030, 1160, 4, 3), (2304, 1030, 1160, 4, 2), (5000, 2100, 520, 3, 2), (4864, 1030, 520, 4, 3)])
def test_gemm_pair_split_k(M, N, K, tile, splits, force_tile):
    """The CTA-pair kernel with the reduction of its last round cut into parts: both CTAs' eight warps park and fold their
    own rows.  From 2304 rows on there are whole rounds before the split one."""
    import ctypes

    from tandem_b200.ops import gemm as G
    from tandem_b200.ops._lib import empty_padded, lib

    force_tile(tile)
    lib().tb_gemm_force_splits(splits)
    plan = (ctypes.c_int * 4)()
    lib().tb_gemm_plan(M, N, K, plan)
    assert list(plan[:3]) == [512, 256 if tile == 3 else 128, splits] and (plan[3] > 0) == (M >= 2304)
    a2, b2 = empty_padded(K, M, torch.bfloat16, "cuda"), empty_padded(K, N, torch.bfloat16, "cuda")
    a2.copy_(rnd(K, M, scale=0.5)), b2.copy_(rnd(K, N, scale=0.5))
    want = a2.float().t() @ b2.float()
    out = G.gemm(a2, b2, M, N, K, a2.stride(0), b2.stride(0), True, True)
    close(out, want)
    for _ in range(3):
        assert torch.equal(out, G.gemm(a2, b2, M, N, K, a2.stride(0), b2.stride(0), True, True))
    bias, res = rnd(N), empty_padded(M, N, torch.bfloat16, "cuda")
    res.copy_(rnd(M, N))
    out = empty_padded(M, N, torch.bfloat16, "cuda")
    close(G.gemm(a2, b2, M, N, K, a2.stride(0), b2.stride(0), True, True, G.BIAS | G.RESIDUAL, bias, res, out=out), want + bias.float() + res.float())


def test_gemm_planner_splits_where_tiles_are_few():
    import ctypes

    from tandem_b200.ops._lib import lib

    def plan(m, n, k):
        three = (ctypes.c_int * 4)()
        lib().tb_gemm_plan(m, n, k, three)
        return tuple(three)

    assert plan(768, 768, 8192)[2] > 1      # a few dozen output tiles, 128 k-blocks: the square weight gradient
    assert plan(1024, 768, 768)[2] == 1     # twelve k-blocks: folding would cost more than it saves
    bm, bn, splits, whole = plan(8192, 768, 3072)
    rows, units = (256, 74) if bm == 512 else (bm, 148)  # 512 marks the 256-row tiles of a CTA pair
    tiles = -(-8192 // rows) * -(-768 // bn)
    assert splits == 1 or (0 < tiles - whole and (tiles - whole) * splits <= units)  # only the last, partial round is ever split


@pytest.mark.parametrize("tile", [-1, 1, 3, 5])
def test_gemm_epilogues(tile, force_tile):
    from tandem_b200.ops import gemm as G

    force_tile(tile)

    M, N, K = 256, 512, 384
    a, w, bias, res = rnd(M, K, scale=0.5), rnd(N, K, scale=0.5), rnd(N), rnd(M, N)
    ref = a.float() @ w.float().t() + bias.float()
    close(G.gemm(a, w, M, N, K, K, K, False, False, G.BIAS, bias), ref)
    close(G.gemm(a, w, M, N, K, K, K, False, False, G.BIAS | G.RESIDUAL, bias, res), ref + res.float())
    slope = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    act = G.gemm(a, w, M, N, K, K, K, False, False, G.BIAS | G.GELU, bias, None, slope)
    close(slope, gelu_slope(ref))  # the forward epilogue saves gelu'(pre-activation) ...
    close(act, torch.nn.functional.gelu(ref))
    x = ref.clone().requires_grad_()
    torch.nn.functional.gelu(x).sum().backward()
    close(slope, x.grad)           # ... which is autograd's derivative of the exact (erf) GELU
    close(G.gemm(a, w, M, N, K, K, K, False, False, G.DGELU, None, slope), (a.float() @ w.float().t()) * slope.float())
    acc = torch.ones(M, N, dtype=torch.float32, device="cuda")
    G.gemm(a, w, M, N, K, K, K, False, False, G.ACCUMULATE, out=acc)
    close(acc, a.float() @ w.float().t() + 1, rtol=2e-3, atol=2e-3)
    acc16 = torch.ones(M, N, dtype=torch.bfloat16, device="cuda")
    G.gemm(a, w, M, N, K, K, K, False, False, G.ACCUMULATE, out=acc16)
    close(acc16, a.float() @ w.float().t() + 1)


@pytest.mark.parametrize("N", [768, 65])
def test_linear_autograd_matches_fp32(N):
    from tandem_b200 import ops

    B, T, K = 4, 96, 256
    x, w, b = rnd(B, T, K).requires_grad_(), rnd(N, K, scale=0.1).requires_grad_(), rnd(N).requires_grad_()
    res = rnd(B, T, N).requires_grad_() if N % 8 == 0 else None
    y = ops.linear(x, w, b, residual=res)
    dy = rnd(B, T, N)
    y.backward(dy)
    xf, wf, bf = (t.detach().float().requires_grad_() for t in (x, w, b))
    yf = torch.nn.functional.linear(xf, wf, bf)
    if res is not None:
        rf = res.detach().float().requires_grad_()
        yf = yf + rf
    yf.backward(dy.float())
    close(y, yf)
    close(x.grad, xf.grad)
    close(w.grad, wf.grad)
    close(b.grad, bf.grad)
    if res is not None:
        close(res.grad, rf.grad)


def test_mlp_autograd_matches_fp32():
    from tandem_b200 import ops

    B, T, D = 2, 128, 256
    x = rnd(B, T, D).requires_grad_()
    w1, b1 = rnd(4 * D, D, scale=0.05).requires_grad_(), rnd(4 * D, scale=0.1).requires_grad_()
    w2, b2 = rnd(D, 4 * D, scale=0.05).requires_grad_(), rnd(D, scale=0.1).requires_grad_()
    res = rnd(B, T, D).requires_grad_()
    y = ops.mlp(x, w1, b1, w2, b2, res)
    dy = rnd(B, T, D)
    y.backward(dy)
    f = [t.detach().float().requires_grad_() for t in (x, w1, b1, w2, b2, res)]
    F = torch.nn.functional
    yf = f[5] + F.linear(F.gelu(F.linear(f[0], f[1], f[2])), f[3], f[4])
    yf.backward(dy.float())
    close(y, yf)
    for got, want in zip((x, w1, b1, w2, b2, res), f):
        close(got.grad, want.grad, rtol=3e-2, atol=2e-2)


@pytest.mark.parametrize("D", [256, 768, 2048])
def test_layer_norm_matches_fp32(D):
    from tandem_b200 import ops

    x, w, b = rnd(3, 100, D, scale=2).requires_grad_(), rnd(D).requires_grad_(), rnd(D).requires_grad_()
    y = ops.layer_norm(x, w, b, 1e-5)
    dy = rnd(3, 100, D)
    y.backward(dy)
    xf, wf, bf = (t.detach().float().requires_grad_() for t in (x, w, b))
    yf = torch.nn.functional.layer_norm(xf, (D,), wf, bf, 1e-5)
    yf.backward(dy.float())
    close(y, yf)
    close(x.grad, xf.grad)
    close(w.grad, wf.grad)
    close(b.grad, bf.grad)


# widths on both sides of every vector count; rows: fewer than a block's, ragged, one and several slices per block (148 or 296
# blocks are resident), one to more rows per warp than the ring holds, forward with and without early gains
@pytest.mark.parametrize("D", [8, 256, 264, 768, 776, 1024, 1032, 1536, 2040])
@pytest.mark.parametrize("M", [1, 13, 1187, 2375, 4801, 21001])
def test_layer_norm_rings_and_slices(M, D):
    from tandem_b200.ops._lib import lib, stream

    x, dy, add, w, b = rnd(M, D), rnd(M, D), rnd(M, D), rnd(D), rnd(D)
    xf, dyf, addf, wf, bf = (t.double() for t in (x, dy, add, w, b))
    mean, std = xf.mean(1, keepdim=True), (xf.var(1, unbiased=False, keepdim=True) + 1e-5).sqrt()
    xh, g = (xf - mean) / std, dyf * wf
    dxf = (g - g.mean(1, keepdim=True) - xh * (g * xh).mean(1, keepdim=True)) / std
    y, dx, dw, db = torch.empty_like(x), torch.empty_like(x), torch.empty_like(w), torch.empty_like(w)
    stats = torch.empty(2, M, device="cuda")
    L, s, scratch = lib(), stream(x), torch.empty(lib().tb_layernorm_bwd_blocks(M) * 2 * D, device="cuda")
    assert L.tb_layernorm_fwd(x.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), stats[0].data_ptr(), stats[1].data_ptr(), M, D, 1e-5, s) == 0
    # one bf16 rounding (2^-9 of the value) and fp32 sums: 1e-5 of the largest term covers 2048 or 21001 of them
    def near(got, want, terms):
        assert ((got.double() - want).abs() <= want.abs() * 2**-8 + 1e-5 * terms).all()

    near(y, xh * wf + bf, (xh * wf).abs().max() + bf.abs().max())
    for second in (None, add, dx):  # without a second gradient, with one, with one that dx is written over
        if second is dx:
            dx.copy_(add)
        assert L.tb_layernorm_bwd_add(dy.data_ptr(), x.data_ptr(), w.data_ptr(), stats[0].data_ptr(), stats[1].data_ptr(),
                                      None if second is None else second.data_ptr(), dx.data_ptr(), dw.data_ptr(), db.data_ptr(),
                                      scratch.data_ptr(), M, D, s) == 0
        near(dx, dxf if second is None else dxf + addf, dxf.abs().max() + addf.abs().max())
        near(dw, (dyf * xh).sum(0), (dyf * xh).abs().sum(0))
        near(db, dyf.sum(0), dyf.abs().sum(0))


def test_residual_layer_norm_sums_both_gradients():
    from tandem_b200 import ops

    M, D = 300, 768
    x = rnd(M, D).requires_grad_()
    w, b = (1 + rnd(D, scale=0.1)).requires_grad_(), rnd(D, scale=0.1).requires_grad_()
    xr, n = ops.residual_layer_norm(x, w, b)
    up, un = rnd(M, D), rnd(M, D)
    (xr.float() * up.float()).sum().backward(retain_graph=True)  # only the residual branch: the gradient passes through
    close(x.grad, up)
    x.grad = None
    ((xr.float() * up.float()).sum() + (n.float() * un.float()).sum()).backward()
    xf, wf, bf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_(), b.detach().float().requires_grad_()
    nf = torch.nn.functional.layer_norm(xf, (D,), wf, bf)
    ((xf * up.float()).sum() + (nf * un.float()).sum()).backward()
    close(n, nf)
    close(x.grad, xf.grad)
    close(w.grad, wf.grad, rtol=3e-2, atol=3e-2)
    close(b.grad, bf.grad, rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("V", [65, 50304])
def test_cross_entropy_matches_fp32(V):
    from tandem_b200 import ops
    from tandem_b200.ops._lib import empty_padded

    rows = 300
    logits = empty_padded(rows, V, torch.bfloat16, "cuda")
    logits.copy_(rnd(rows, V, scale=3))
    ref_in = logits.detach().float().clone().requires_grad_()
    targets = torch.randint(0, V, (rows,), device="cuda")
    leaf = logits.detach().requires_grad_()
    loss = ops.cross_entropy(leaf, targets)
    want = torch.nn.functional.cross_entropy(ref_in, targets)
    (loss * 0.5).backward()
    (want * 0.5).backward()
    assert abs(loss.item() - want.item()) < 1e-4 * max(1.0, abs(want.item()))
    close(leaf.grad, ref_in.grad, rtol=2e-2, atol=1e-3)


def test_embedding_matches_fp32():
    from tandem_b200 import ops

    V, S, D, B, T = 65, 128, 256, 4, 128
    tok, pos = rnd(V, D).requires_grad_(), rnd(S, D).requires_grad_()
    idx = torch.randint(0, V, (B, T), device="cuda")
    y = ops.embedding(idx, tok, pos)
    dy = rnd(B, T, D)
    y.backward(dy)
    tf, pf = tok.detach().float().requires_grad_(), pos.detach().float().requires_grad_()
    yf = tf[idx] + pf[torch.arange(T, device="cuda")]
    yf.backward(dy.float())
    close(y, yf)
    close(tok.grad, tf.grad)
    close(pos.grad, pf.grad)


@pytest.mark.parametrize("B,T,V,D", [(1, 1, 3, 8), (3, 7, 65, 24), (5, 130, 1003, 136)])
def test_embedding_backward_vectors_and_a_misaligned_gradient(B, T, V, D):
    """Vector tails, every batch count of the position sums' unrolled loop, and a gradient that is a contiguous slice starting in
    mid-vector: the kernels read a copy of it.  Sums of integers up to 8 are exact in fp32, in any order."""
    from tandem_b200 import ops

    tok, pos = rnd(V, D).requires_grad_(), rnd(T + 2, D).requires_grad_()
    idx = torch.randint(0, V, (B, T), device="cuda")
    store = torch.randint(-8, 9, (B * T * D + 8,), device="cuda").bfloat16()
    for first in (0, 1, 4):
        dy = store[first:first + B * T * D].view(B, T, D)
        assert (dy.data_ptr() % 16 == 0) == (first == 0)
        got_tok, got_pos = torch.autograd.grad(ops.embedding(idx, tok, pos), [tok, pos], dy)
        want = torch.zeros(V, D, device="cuda").index_add_(0, idx.view(-1), dy.float().view(-1, D))
        assert torch.equal(got_tok, want.bfloat16())
        assert torch.equal(got_pos[:T], dy.float().sum(0).bfloat16()) and (got_pos[T:] == 0).all()


@pytest.mark.parametrize("sizes,offset", [([1, 15, 16, 17, 4096], 0), ([4 * 16 * 256 + 5] * 3, 0), ([70_000_003], 0), ([33_000_000, 40], 1),
                                          ([7] * 100 + [1 << 20] * 5, 0)])
def test_multi_copy_tails_and_large_tensors(sizes, offset):
    """Byte tails, misaligned tensors, more tensors than one launch takes, and tensors that take the whole GPU several turns."""
    from tandem_b200.ops.elementwise import multi_copy

    pairs = []
    for n in sizes:
        src = torch.randint(0, 256, (n + 32,), dtype=torch.uint8, device="cuda")
        dst = torch.zeros(n + 32, dtype=torch.uint8, device="cuda")
        pairs.append((dst, src, n))
    multi_copy(pairs[0][0], [(d[offset:offset + n], s[offset:offset + n]) for d, s, n in pairs])
    for d, s, n in pairs:
        assert torch.equal(d[offset:offset + n], s[offset:offset + n])
        assert (d[:offset] == 0).all() and (d[offset + n:] == 0).all()


def test_gpt_on_b200_kernels_tracks_torch_path():
    """Same weights, same batch: loss and gradients of the kernel path stay within bf16 noise of the torch path."""
    from tandem_b200.model import GPT, Config

    torch.manual_seed(0)
    cfg_t = Config(vocab=65, seq=128, layers=2, heads=4, dim=256, kernels="torch")
    cfg_k = Config(vocab=65, seq=128, layers=2, heads=4, dim=256, kernels="b200")
    ref = GPT(cfg_t).cuda()
    ker = GPT(cfg_k).cuda().bfloat16()
    ker.load_state_dict({k: v.bfloat16() for k, v in ref.state_dict().items()})
    ref.load_state_dict({k: v.float() for k, v in ker.state_dict().items()})  # identical (bf16-representable) weights
    x = torch.randint(0, 65, (4, 128), device="cuda")
    y = torch.randint(0, 65, (4, 128), device="cuda")
    lk = ker(x, y)
    lk.backward()
    lr = ref(x, y)
    lr.backward()
    assert abs(lk.item() - lr.item()) < 2e-2, (lk.item(), lr.item())
    for (name, pk), (_, pr) in zip(ker.named_parameters(), ref.named_parameters()):
        g, w = pk.grad.float(), pr.grad
        denom = w.norm().clamp_min(1e-6)
        assert ((g - w).norm() / denom).item() < 6e-2, (name, ((g - w).norm() / denom).item())


def test_twenty_training_steps_track_torch_autocast():
    """Mixed precision end to end: the bf16 kernel path (bf16 parameters, fp32 master weights and moments in BucketAdamW)
    against the same model trained by torch with fp32 parameters under bf16 autocast and torch's AdamW.  Twenty steps on
    the same batches from the same initial weights: the loss curves must stay together and both must fall."""
    import tandem_b200
    from tandem_b200.data import synthetic
    from tandem_b200.ddp import DDP, BucketAdamW
    from tandem_b200.model import GPT, Config

    text = synthetic(60_000)
    shape = dict(vocab=256, seq=128, layers=3, heads=4, dim=256)
    torch.manual_seed(0)
    ref = GPT(Config(kernels="torch", **shape)).cuda()
    torch.manual_seed(0)
    ker = GPT(Config(kernels="b200", **shape)).cuda().bfloat16()
    group = tandem_b200.Group(0, 1, "cuda:0", job=f"curve{torch.randint(0, 1 << 30, (1,)).item()}")
    wrapped = DDP(ker, group, rebuild=False)
    opt_k = BucketAdamW(wrapped, lr=1e-3, weight_decay=0.1)
    opt_r = torch.optim.AdamW(ref.parameters(), lr=1e-3, weight_decay=0.1)
    ours, theirs = [], []
    for step in range(20):
        x, y = text.batch(step, 16, shape["seq"], device="cuda")
        loss = wrapped(x, y)
        loss.backward()
        opt_k.step()
        opt_k.zero_grad()
        ours.append(loss.item())
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = ref(x, y)
        loss.backward()
        opt_r.step()
        opt_r.zero_grad()
        theirs.append(loss.item())
    group.close()
    assert all(a == a for a in ours)
    assert max(abs(a - b) for a, b in zip(ours, theirs)) < 0.05, (ours, theirs)
    assert ours[-1] < ours[0] - 0.5 and theirs[-1] < theirs[0] - 0.5, (ours, theirs)


@pytest.mark.parametrize("B,T,H,hd", [(2, 128, 2, 64), (2, 512, 3, 64), (1, 256, 2, 128), (3, 1024, 2, 64), (1, 384, 2, 128), (2, 640, 1, 64),
                                      (1, 2048, 2, 128)])
@pytest.mark.parametrize("spread", [1.0, 3.0])
def test_causal_attention_matches_fp32(B, T, H, hd, spread):
    """Odd and even numbers of 128-row tiles (the forward pairs them up), both head sizes, and scores spread widely
    enough that the running maximum keeps moving (the lazy accumulator rescale in the forward kernel)."""
    from tandem_b200 import ops
    from tandem_b200.ops.attention import attention_error

    d = H * hd
    qkv = rnd(B, T, 3 * d, scale=spread).requires_grad_()
    y = ops.causal_attention(qkv, H)
    dy = rnd(B, T, d)
    y.backward(dy)
    ref = qkv.detach().float().requires_grad_()
    q, k, v = (z.view(B, T, H, hd).transpose(1, 2) for z in ref.split(d, dim=2))
    yf = torch.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True).transpose(1, 2).reshape(B, T, d)
    yf.backward(dy.float())
    torch.cuda.synchronize()
    assert not attention_error(), "an attention wait ran out"
    close(y, yf, rtol=2e-2, atol=1e-2)
    close(qkv.grad, ref.grad, rtol=4e-2, atol=2e-2)
    for part in range(3):  # dq, dk and dv each on their own scale
        close(qkv.grad[..., part * d:(part + 1) * d], ref.grad[..., part * d:(part + 1) * d], rtol=4e-2, atol=2e-2, frobenius=1e-2)


# more tiles than SMs (backward) and than two per SM (forward), by one and by several rounds; one to eight tiles per head; heads that
# fill no whole group of the work list
@pytest.mark.parametrize("B,T,H", [(149, 128, 1), (297, 128, 1), (25, 256, 13), (10, 640, 8), (13, 1024, 12), (40, 1024, 5)])
def test_causal_attention_work_lists(B, T, H):
    """CTAs that take item after item against a CTA for every item: a sequence by itself has fewer tiles than the GPU has SMs."""
    from tandem_b200 import ops
    from tandem_b200.ops.attention import attention_error

    qkv, dy = rnd(B, T, 3 * H * 64), rnd(B, T, H * 64)
    x = qkv.clone().requires_grad_()
    y = ops.causal_attention(x, H)
    (g,) = torch.autograd.grad(y, x, dy)
    for b in range(B):
        one = qkv[b:b + 1].clone().requires_grad_()
        alone = ops.causal_attention(one, H)
        assert torch.equal(y[b:b + 1], alone)
        assert torch.equal(g[b:b + 1], torch.autograd.grad(alone, one, dy[b:b + 1])[0])
    torch.cuda.synchronize()
    assert not attention_error(), "an attention wait ran out"


@pytest.mark.parametrize("hd", [64, 128])
def test_causal_attention_keeps_nan_queries_from_later_keys(hd):
    """The value gradient of a key is a sum over the queries from that key on: a query that is NaN reaches no key after it."""
    from tandem_b200 import ops

    T, H, row = 256, 2, 133
    qkv, dy = rnd(1, T, 3 * H * hd), rnd(1, T, H * hd)
    want = torch.autograd.grad(ops.causal_attention(x := qkv.clone().requires_grad_(), H), x, dy)[0][..., 2 * H * hd:]
    qkv[0, row, :hd] = float("nan")
    got = torch.autograd.grad(ops.causal_attention(x := qkv.clone().requires_grad_(), H), x, dy)[0][..., 2 * H * hd:]
    assert got[0, row, :hd].isnan().all()
    assert torch.equal(got[0, row + 1:], want[0, row + 1:]) and torch.equal(got[..., hd:], want[..., hd:])


def test_causal_attention_is_deterministic():
    """No atomics anywhere: two runs give the same bits."""
    from tandem_b200 import ops

    qkv = rnd(2, 512, 3 * 256).requires_grad_()
    dy = rnd(2, 512, 256)
    outs = []
    for _ in range(2):
        qkv.grad = None
        y = ops.causal_attention(qkv, 4)
        y.backward(dy)
        outs.append((y.detach().clone(), qkv.grad.clone()))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("n,rank", [(1, 0), (4, 2), (8, 7)])
def test_gemm_with_fused_weight_gather(n, rank):
    """The weight lives in `n` shards of a flat buffer (here all on this GPU, standing in for the peers'
    symmetric memory); the kernel assembles it in `full` while it multiplies."""
    from tandem_b200.ops.gemm import GatheredLinear
    from tandem_b200.parallel.symm import split_offsets

    M, N, K = 1024, 2304, 768
    before, after = 1536, 2304 + 1003
    flat = rnd(before + N * K + after, scale=0.3)
    offs = split_offsets(flat.numel(), n)
    shards = [flat[offs[q]:offs[q + 1]].clone() for q in range(n)]
    full = torch.zeros_like(flat)
    x, bias = rnd(M, K, scale=0.5), rnd(N)
    op = GatheredLinear([s.data_ptr() for s in shards], offs, rank, full, before, N, K)
    w = flat[before:before + N * K].view(N, K)
    for _ in range(2):  # the second call reuses the flags with a new epoch
        full.zero_()
        y = op(x, bias)
        close(y, x.float() @ w.float().t() + bias.float())
        assert torch.equal(full[before:before + N * K], flat[before:before + N * K])
    # the bias sits right behind the weight in the flat buffer and is fetched with it
    op2 = GatheredLinear([s.data_ptr() for s in shards], offs, rank, full, before, N, K, bias_follows=True)
    b2 = flat[before + N * K:before + N * K + N]
    for _ in range(2):
        full.zero_()
        y = op2(x, None)
        close(y, x.float() @ w.float().t() + b2.float())
        assert torch.equal(full[before:before + N * K + N], flat[before:before + N * K + N])


def optimizer_timing_rank(g, during_backward, graphed):
    """DDP on the hand-written kernels in bf16 with the replicated optimizer applied after backward or span by span
    during it; eager or replayed from a CUDA graph."""
    from tandem_b200.data import synthetic
    from tandem_b200.ddp import DDP, BucketAdamW
    from tandem_b200.model import Config, GPT
    from tandem_b200.parallel.graph import GraphedStep

    torch.manual_seed(0)
    cfg = Config(seq=128, layers=2, heads=2, dim=128, kernels="b200")
    text = synthetic(50_000)
    model = GPT(cfg).to(g.device).bfloat16()
    wrapped = DDP(model, g, bucket_bytes=128 << 10, rebuild=False)
    opt = BucketAdamW(wrapped, lr=1e-3, weight_decay=0.1, during_backward=during_backward)
    batches = [text.batch(step, 8, cfg.seq, rank=g.rank, world=g.size, device=g.device) for step in range(8)]
    losses = []
    if graphed:
        step_fn = GraphedStep(wrapped, opt, *batches[0], warmup=3)
        for x, y in batches[3:]:
            losses.append(step_fn(x, y).item())
    else:
        for k, (x, y) in enumerate([batches[0]] * 3 + batches[3:]):
            loss = wrapped(x, y)
            loss.backward()
            opt.step()
            opt.zero_grad()
            if k >= 3:
                losses.append(loss.item())
    g.check()
    return losses, torch.cat([p.detach().float().reshape(-1) for p in model.parameters()]).cpu()


def test_optimizer_during_backward_equals_optimizer_after_backward():
    from tandem_b200 import launch

    after = launch(optimizer_timing_rank, 1, False, False, device="cuda")[0]
    during = launch(optimizer_timing_rank, 1, True, False, device="cuda")[0]
    replayed = launch(optimizer_timing_rank, 1, True, True, device="cuda")[0]
    assert after[0] == during[0], (after[0], during[0])
    assert torch.equal(after[1], during[1])  # the same arithmetic on the same gradients: bit for bit
    assert after[0] == replayed[0] and torch.equal(after[1], replayed[1])


@pytest.mark.parametrize("V,ld,first", [(65, 72, 0), (1003, 1003, 0), (1003, 1008, 0), (8200, 8200, 3), (50304, 50304, 0), (2049, 2056, 8),
                                         (256, 256, 0), (512, 512, 0), (505, 512, 0), (517, 520, 0), (300, 301, 1)])
def test_cross_entropy_row_layouts(V, ld, first):
    """Rows that can and cannot be read in 16-byte vectors (odd strides, a first element in mid-vector), vector tails and
    batches of loads that end early; gradients land in place and nothing outside the columns changes."""
    from tandem_b200 import ops

    rows = 37
    store = torch.full((rows * ld + first + 8,), 7.0, dtype=torch.bfloat16, device="cuda")
    logits = store[first:first + rows * ld].view(rows, ld)[:, :V]
    logits.copy_(rnd(rows, V) * 3)
    targets = torch.randint(0, V, (rows,), device="cuda")
    targets[0], targets[1] = 0, V - 1
    z = logits.detach().double().requires_grad_()
    want = torch.nn.functional.cross_entropy(z, targets)
    (want * 2).backward()
    x = logits.detach().requires_grad_()
    loss = ops.cross_entropy(x, targets)
    (grad,) = torch.autograd.grad(loss * 2, x)
    assert abs(loss.item() - want.item()) < 1e-5 * want.item()
    # one bf16 rounding, and exp(z - lse) with lse ~ 10 rounded to fp32
    assert ((grad.double() - z.grad).abs() <= 2.0**-8 * z.grad.abs() + 2e-6 / rows).all()
    if first:
        assert (store[:first] == 7).all()
    assert (store[first + rows * ld:] == 7).all()


@pytest.mark.parametrize("n,offset", [(1, 0), (3, 0), (511, 0), (513, 0), (4097, 0), (4096, 1), (1000003, 0), (1000002, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_fused_adamw_alignment_and_tails(n, offset, dtype):
    """Arrays that start off a 16-byte boundary take the element-wise loop, aligned ones four elements at a time plus a tail:
    the arithmetic is the same, so both must agree bit for bit."""
    from tandem_b200.ops import fused_adamw

    scalars = (1 - 3e-5, 0.1, 0.999, 0.001, 0.0316, 1e-8, -3e-3)

    def run(at):
        gen = torch.Generator(device="cuda").manual_seed(3)
        arrays = [torch.zeros(n + 8, device="cuda") for _ in range(3)] + [torch.zeros(n + 8, device="cuda", dtype=dtype), torch.zeros(n + 8, device="cuda", dtype=torch.bfloat16)]
        p, m, v, g, shadow = (a[at:at + n] for a in arrays)
        p.copy_(torch.randn(n, device="cuda", generator=gen)), m.copy_(torch.randn(n, device="cuda", generator=gen) * 0.1)
        v.copy_(torch.rand(n, device="cuda", generator=gen)), g.copy_(torch.randn(n, device="cuda", generator=gen))
        fused_adamw(p, g, m, v, scalars, True, shadow)
        for a in arrays:
            assert (a[:at] == 0).all() and (a[at + n:] == 0).all()
        return p, m, v, shadow

    for a, b in zip(run(offset), run(5)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("M,N,ld", [(1, 64, 64), (300, 72, 72), (2048, 768, 768), (5000, 200, 208), (8191, 4104, 4104)])
def test_column_sums_in_vectors(M, N, ld):
    from tandem_b200.ops._lib import lib

    x = rnd(M, ld)
    scratch = torch.empty(32 * N, dtype=torch.float32, device="cuda")
    out, again = (torch.empty(N, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    s = torch.cuda.current_stream().cuda_stream
    assert lib().tb_col_sum(x.data_ptr(), M, N, ld, out.data_ptr(), scratch.data_ptr(), s) == 0
    assert lib().tb_col_sum(x.data_ptr(), M, N, ld, again.data_ptr(), scratch.data_ptr(), s) == 0
    want = x[:, :N].double().sum(0)
    # fp32 partial sums of M unit normals (error ~ sqrt(M) * 6e-8 * a few), then one bf16 rounding
    assert ((out.double() - want).abs() <= 2.0**-8 * want.abs() + 1e-5 * M**0.5).all()
    assert torch.equal(out, again)


@pytest.mark.parametrize("M,N", [(2048, 3072), (4096, 4096), (6145, 4104), (300, 5128), (1536, 8192), (9000, 16392)])
def test_wide_column_sums_equal_narrow_ones(M, N):
    """Wide matrices take a kernel with more columns per block: every sum is the one that a few columns by themselves get."""
    from tandem_b200.ops._lib import lib

    x = rnd(M, N)
    scratch = torch.empty(32 * N, dtype=torch.float32, device="cuda")
    wide, narrow = (torch.empty(N, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    s = torch.cuda.current_stream().cuda_stream
    assert lib().tb_col_sum(x.data_ptr(), M, N, N, wide.data_ptr(), scratch.data_ptr(), s) == 0
    for a in range(0, N, 1024):
        n = min(1024, N - a)
        assert lib().tb_col_sum(x[:, a:].data_ptr(), M, n, N, narrow[a:].data_ptr(), scratch.data_ptr(), s) == 0
    assert torch.equal(wide, narrow)
    want = x.double().sum(0)
    assert ((wide.double() - want).abs() <= 2.0**-8 * want.abs() + 1e-5 * M**0.5).all()


def test_operators_without_gradients_equal_those_with():
    """Where gradients are off the operators skip the autograd node: same results, and transforms that the node refuses still
    meet it.  A saved-tensor hook sees what a node saves where gradients are on, and nothing where they are off."""
    from tandem_b200 import ops

    x, w, b = rnd(256, 128), rnd(384, 128, scale=0.05), rnd(384)
    ln_w, ln_b, w2, b2 = rnd(128), rnd(128), rnd(128, 384, scale=0.05), rnd(128)
    qkv = rnd(2, 128, 3 * 128)
    idx, tok, pos = torch.randint(0, 50, (2, 128), device="cuda"), rnd(50, 128), rnd(128, 128)
    calls = [lambda: ops.linear(x, w, b), lambda: ops.layer_norm(x, ln_w, ln_b), lambda: ops.residual_layer_norm(x, ln_w, ln_b)[1],
             lambda: ops.mlp(x, w, b, w2, b2, x), lambda: ops.causal_attention(qkv, 2), lambda: ops.embedding(idx, tok, pos),
             lambda: ops.cross_entropy(x, torch.zeros(256, dtype=torch.long, device="cuda"))]
    for call in calls:
        want = call()
        with torch.no_grad():
            got = call()
        assert torch.equal(got, want) and not got.requires_grad
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t.shape) or t, lambda t: t):
        with torch.no_grad():
            ops.linear(x, w, b)
        assert not seen
        y = ops.linear(x, w.clone().requires_grad_(), b)
        assert seen == [x.shape, w.shape]
    assert torch.equal(y, ops.linear(x, w, b))
    with torch.no_grad(), pytest.raises(RuntimeError):
        torch.func.vmap(lambda v: ops.linear(v, w, b))(x.unsqueeze(0))
    with torch.no_grad(), torch.autograd.forward_ad.dual_level(), pytest.raises((RuntimeError, NotImplementedError)):
        ops.linear(torch.autograd.forward_ad.make_dual(x, torch.ones_like(x)), w, b)


def _operator_forms():
    """Every operator with the forms of input that it accepts: leading dimensions, strides, offsets, odd widths, missing and
    frozen operands, few and many rows (below and above the second stream's limit).  Name -> (function, inputs, which need gradients)."""
    from tandem_b200 import ops

    def leaf(*shape):
        return rnd(*shape, scale=0.5)

    forms = {}
    for rows, inner, outer in [((1,), 64, 64), ((33,), 72, 65), ((3, 40), 100, 96), ((2, 3, 7), 8, 1003), ((4200,), 136, 128), ((), 64, 24), ((2, 130), 65, 40)]:
        x, w, b = leaf(*rows, inner), leaf(outer, pad8(inner))[:, :inner], leaf(outer)
        forms[f"linear {rows} {inner} {outer}"] = (ops.linear, [x, w, b], [1, 1, 1])
        forms[f"linear {rows} {inner} {outer} no bias"] = (ops.linear, [x, w, None], [1, 1, 0])
        forms[f"linear {rows} {inner} {outer} frozen"] = (ops.linear, [x, w, b], [1, 0, 0])
        forms[f"linear {rows} {inner} {outer} first layer"] = (ops.linear, [x, w, b], [0, 1, 1])
        if outer % 8 == 0:
            forms[f"linear {rows} {inner} {outer} residual"] = (lambda x, w, b, r: ops.linear(x, w, b, residual=r), [x, w, b, leaf(*rows, outer)], [1, 1, 1, 1])
    wide = leaf(40, 3 * 64)
    for name, x in {"columns": wide[:, 64:128], "odd columns": wide[:, 3:67], "transposed": leaf(64, 40).t(), "every other row": leaf(80, 64)[::2],
                    "swapped": leaf(5, 6, 64).transpose(0, 1), "expanded": leaf(1, 64).expand(40, 64), "offset": leaf(40 * 64 + 1)[1:].view(40, 64)}.items():
        forms[f"linear of {name}"] = (ops.linear, [x, leaf(96, 64), leaf(96)], [1, 1, 1])
        forms[f"layer_norm of {name}"] = (ops.layer_norm, [x, leaf(64), leaf(64)], [1, 1, 1])
    def offset(*shape):  # contiguous, and not on a 16-byte boundary
        return leaf(math.prod(shape) + 1)[1:].view(*shape)

    x, w, r, every_other, expanded = leaf(40, 64), leaf(96, 64), offset(40, 96), leaf(192)[::2], leaf(1).expand(96)
    for name, b in {"every other": every_other, "expanded": expanded, "offset": offset(96)}.items():
        forms[f"linear with {name} bias"] = (ops.linear, [x, w, b], [1, 1, 1])
        forms[f"layer_norm with {name} weight"] = (ops.layer_norm, [leaf(40, 96), b, leaf(96)], [1, 1, 1])
        forms[f"layer_norm with {name} bias"] = (ops.layer_norm, [leaf(40, 96), leaf(96), b], [1, 1, 1])
    forms["linear with offset residual"] = (lambda x, w, b, r: ops.linear(x, w, b, residual=r), [x, w, leaf(96), r], [1, 1, 1, 1])
    forms["mlp with offset residual"] = (ops.mlp, [x, leaf(128, 64), leaf(128), leaf(96, 128), leaf(96), r], [1] * 6)
    forms["residual_layer_norm of offset"] = (ops.residual_layer_norm, [r, leaf(96), leaf(96)], [1, 1, 1])
    for rows in [(1,), (2, 77), (4100,)]:
        x, r = leaf(*rows, 72), leaf(*rows, 40)
        forms[f"mlp {rows}"] = (ops.mlp, [x, leaf(96, 72), leaf(96), leaf(40, 96), leaf(40), r], [1] * 6)
        forms[f"mlp {rows} frozen"] = (ops.mlp, [x, leaf(96, 72), None, leaf(40, 96), None, r], [1, 0, 0, 1, 0, 0])
        forms[f"residual_layer_norm {rows}"] = (ops.residual_layer_norm, [x, leaf(72), leaf(72)], [1, 1, 1])
        forms[f"normalized alone {rows}"] = (lambda *a: ops.residual_layer_norm(*a)[1], [x, leaf(72), leaf(72)], [1, 1, 1])
    for heads, hd in [(1, 64), (3, 64), (2, 128)]:
        forms[f"attention {heads} {hd}"] = (lambda q, h=heads: ops.causal_attention(q, h), [leaf(2, 256, 3 * heads * hd)], [1])
    forms["attention of a slice"] = (lambda q: ops.causal_attention(q, 2), [leaf(2, 128, 2 * 384)[:, :, :384]], [1])
    idx = torch.randperm(60, device="cuda")[:2 * 20].view(2, 20)
    forms["embedding"] = (lambda t, p: ops.embedding(idx, t, p), [leaf(60, 40), leaf(32, 40)], [1, 1])
    forms["embedding in views"] = (lambda t, p: ops.embedding(idx, t, p), [leaf(60, 48)[:, 8:48], offset(32, 40)], [1, 1])
    forms["embedding of transposed ids"] = (lambda t, p: ops.embedding(idx.t(), t, p), [leaf(60, 40), leaf(32, 40)], [1, 1])
    for V, ld in [(65, 72), (65, 65), (1003, 1008), (64, 200)]:
        forms[f"cross_entropy {V} {ld}"] = (lambda z: ops.cross_entropy(z * 1.0 if z.stride(0) == z.shape[1] else z, torch.arange(30, device="cuda") % V),
                                            [leaf(30, ld)[:, :V]], [1])
    forms["cross_entropy of one row for all"] = (lambda z: ops.cross_entropy(z, torch.arange(30, device="cuda")), [leaf(1, 64).expand(30, 64)], [1])
    return forms


def pad8(n):
    return (n + 7) // 8 * 8


def test_native_operators_equal_the_python_ones(monkeypatch):
    """Outputs, gradients, saved tensors and second uses, bit for bit, over all forms; and what is refused is refused alike."""
    from tandem_b200 import ops
    from tandem_b200.ops import _lib

    assert _lib.native() is not None
    torch.manual_seed(0)
    forms = _operator_forms()

    def outcome(function, inputs, needs):
        inputs = [t if t is None or not n else t.detach().requires_grad_() for t, n in zip(inputs, needs)]
        saved = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: saved.append((t.dtype, t.shape)) or t, lambda t: t):
            out = function(*inputs)
        outs = out if isinstance(out, tuple) else (out,)
        torch.manual_seed(1)
        grads = [torch.randn_like(o) for o in outs]
        kept = [o.detach().clone() for o in outs]
        wanted = [t for t, n in zip(inputs, needs) if n]
        got = torch.autograd.grad(outs, wanted, grads)
        with pytest.raises(RuntimeError, match="second time"):
            torch.autograd.grad(outs, wanted, grads)
        return saved, [(o.shape, o.stride(), o.is_contiguous()) for o in outs], kept + [g.clone() for g in got]

    for name, (function, inputs, needs) in forms.items():
        fresh = [None if t is None else t.detach().clone(memory_format=torch.preserve_format) if "cross" in name else t for t in inputs]
        native = outcome(function, fresh, needs)
        with monkeypatch.context() as m:
            m.setattr(_lib, "native", lambda: None)
            python = outcome(function, inputs, needs)
        assert native[:2] == python[:2], name
        for a, b in zip(native[2], python[2]):
            assert a.shape == b.shape and a.stride() == b.stride() and torch.equal(a, b), name

    x, w, b = rnd(40, 64), rnd(96, 64), rnd(96)
    refused = [lambda: ops.linear(x.float(), w, b), lambda: ops.linear(x, w.cpu(), b), lambda: ops.linear(x, rnd(65, 64), None, residual=rnd(40, 65)),
               lambda: ops.linear(x, w, b, residual=rnd(96, 40).t()), lambda: ops.mlp(x, w, b, rnd(40, 96), b, None),
               lambda: ops.mlp(x, rnd(65, 64), None, rnd(40, 65), None, rnd(40, 40)), lambda: ops.layer_norm(rnd(4, 12), rnd(12), rnd(12)),
               lambda: ops.causal_attention(rnd(1, 100, 192), 1), lambda: ops.causal_attention(rnd(1, 128, 96), 1), lambda: ops.causal_attention(rnd(128, 192), 1),
               lambda: ops.causal_attention(rnd(1, 128, 192), 0), lambda: ops.embedding(torch.zeros(3, dtype=torch.long, device="cuda"), w, w),
               lambda: ops.cross_entropy(rnd(2, 3, 8), torch.zeros(2, dtype=torch.long, device="cuda"))]

    def refusal(call):
        try:
            call()
        except Exception as e:
            return type(e)
        return None

    native = [refusal(call) for call in refused]
    monkeypatch.setattr(_lib, "native", lambda: None)
    assert native == [refusal(call) for call in refused] and None not in native


@pytest.mark.parametrize("python", [False, True])
def test_operators_of_views_equal_those_of_copies(python, monkeypatch):
    """What the kernels cannot read where it lies is copied: strides, offsets and expanded operands change no bit."""
    from tandem_b200.ops import _lib

    if python:
        monkeypatch.setattr(_lib, "native", lambda: None)
    torch.manual_seed(0)

    def outcome(function, inputs, needs):
        inputs = [t if t is None or not n else t.detach().requires_grad_() for t, n in zip(inputs, needs)]
        out = function(*inputs)
        outs = out if isinstance(out, tuple) else (out,)
        torch.manual_seed(1)
        return [o.detach().clone() for o in outs] + list(torch.autograd.grad(outs, [t for t, n in zip(inputs, needs) if n], [torch.randn_like(o) for o in outs]))

    for name, (function, inputs, needs) in _operator_forms().items():
        copies = [None if t is None else t.clone(memory_format=torch.contiguous_format) for t in inputs]
        if name.startswith("linear"):
            copies[1] = inputs[1]  # a weight has to have 16-byte rows, which an odd width takes padding for
        for a, b in zip(outcome(function, inputs, needs), outcome(function, copies, needs)):
            assert torch.equal(a, b), name


@pytest.mark.parametrize("python", [False, True])
@pytest.mark.parametrize("hook", ["save_on_cpu", "offset copies", "transposed copies"])
def test_saved_tensors_may_come_back_elsewhere(hook, python, monkeypatch):
    """A saved-tensor hook may hand backward a tensor with other strides, or one that starts off a 16-byte boundary."""
    from tandem_b200.ops import _lib

    if python:
        monkeypatch.setattr(_lib, "native", lambda: None)
    torch.manual_seed(0)

    def offset(t):
        room = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
        return room[1:].view(t.shape).copy_(t)

    def transposed(t):
        return t.t().contiguous().t() if t.dim() == 2 else t.clone()

    hooks = {"save_on_cpu": torch.autograd.graph.save_on_cpu(), "offset copies": torch.autograd.graph.saved_tensors_hooks(lambda t: t.clone(), offset),
             "transposed copies": torch.autograd.graph.saved_tensors_hooks(lambda t: t.clone(), transposed)}

    def gradients(function, inputs, needs, around):
        inputs = [t if t is None or not n else t.detach().requires_grad_() for t, n in zip(inputs, needs)]
        with around:
            out = function(*inputs)
        outs = out if isinstance(out, tuple) else (out,)
        torch.manual_seed(1)
        return torch.autograd.grad(outs, [t for t, n in zip(inputs, needs) if n], [torch.randn_like(o) for o in outs])

    for name, (function, inputs, needs) in _operator_forms().items():
        hooked = gradients(function, inputs, needs, hooks[hook])  # first: cross_entropy writes its gradient over what it saved
        for a, b in zip(hooked, gradients(function, inputs, needs, contextlib.nullcontext())):
            assert torch.equal(a, b), name


@pytest.mark.parametrize("python", [False, True])
def test_linear_of_an_empty_batch(python, monkeypatch):
    """Its weight gradient is a sum over no rows: zeros, not what the memory held before."""
    from tandem_b200 import ops
    from tandem_b200.ops import _lib

    if python:
        monkeypatch.setattr(_lib, "native", lambda: None)
    for inner, outer in [(64, 96), (68, 96), (64, 0)]:
        x, w, b = rnd(0, inner).requires_grad_(), rnd(outer, pad8(inner))[:, :inner].detach().requires_grad_(), rnd(outer).requires_grad_()
        del_me = [torch.full((96, pad8(inner)), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(8)]
        del del_me
        y = ops.linear(x, w, b if outer else None)
        y.sum().backward()
        assert y.shape == (0, outer) and x.grad.shape == x.shape and torch.equal(w.grad, torch.zeros_like(w))
        assert not outer or torch.equal(b.grad, torch.zeros_like(b))
    x = rnd(40, 64).requires_grad_()
    (g,) = torch.autograd.grad(ops.linear(x, rnd(0, 64)), x, rnd(40, 0))
    assert torch.equal(g, torch.zeros_like(x))
    assert torch.equal(ops.linear(rnd(40, 0), rnd(96, 0)), torch.zeros(40, 96, device="cuda"))
    with pytest.raises(ValueError, match="no columns"):
        ops.linear(rnd(40, 0), rnd(96, 0), rnd(96))


@pytest.mark.parametrize("python", [False, True])
def test_operators_notice_a_changed_input(python, monkeypatch):
    """What backward reads again must not have changed in between; a gradient has no gradient of its own."""
    from tandem_b200 import ops
    from tandem_b200.ops import _lib

    if python:
        monkeypatch.setattr(_lib, "native", lambda: None)
    x, w = rnd(40, 64), rnd(96, 64).requires_grad_()
    y = ops.linear(x, w)
    x.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()
    x.requires_grad_()
    (g,) = torch.autograd.grad(ops.linear(x, w).float().square().sum(), x, create_graph=True)
    assert not g.requires_grad  # as of a constant


def test_stream_wait_from_two_threads():
    """Each thread orders its own pair of streams through one native call, many times over."""
    import threading

    from tandem_b200.ops._lib import stream_wait

    bad = []

    def work():
        torch.cuda.set_device(0)
        first, second = torch.cuda.Stream(), torch.cuda.Stream()
        x = torch.zeros(1 << 20, device="cuda")
        torch.cuda.synchronize()
        for i in range(50):
            with torch.cuda.stream(first):
                x.fill_(float(i))
            stream_wait(second.cuda_stream, first.cuda_stream)
            with torch.cuda.stream(second):
                y = x + 1
            stream_wait(first.cuda_stream, second.cuda_stream)
            second.synchronize()
            if not (y == i + 1).all():
                bad.append(i)

    threads = [threading.Thread(target=work) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_stream_waits_of_many_threads_share_their_events():
    """A program that starts a thread per step makes no event per thread."""
    import threading

    from tandem_b200.ops._lib import lib, stream_wait

    first, second = torch.cuda.Stream(), torch.cuda.Stream()

    def work():
        torch.cuda.set_device(0)
        stream_wait(second.cuda_stream, first.cuda_stream)

    work()
    before = lib().tb_stream_wait_events()
    for _ in range(20):
        t = threading.Thread(target=work)
        t.start()
        t.join()
    assert lib().tb_stream_wait_events() == before


def test_products_and_sums_of_two_threads():
    """Split products and column sums that two host threads launch on streams of their own equal those of one thread."""
    import threading

    from tandem_b200.ops import gemm as G

    dy, x = rnd(2048, 768), rnd(2048, 384)
    results = [[], []]

    def work(mine, rounds):
        torch.cuda.set_device(0)
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.default_stream())
        with torch.cuda.stream(s):
            for _ in range(rounds):
                mine.append((G._grad_weight(dy, 768, x, 384, torch.bfloat16), G._grad_bias(dy, 768)))
        s.synchronize()

    work(results[0], 1)
    (want,) = results[0]
    threads = [threading.Thread(target=work, args=(mine, 200)) for mine in results]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(torch.equal(a, b) for mine in results for got in mine for a, b in zip(got, want))
