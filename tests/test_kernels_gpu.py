"""Numerics of every hand-written CUDA kernel against a plain PyTorch fp32 statement of the op."""
import math

import pytest
import torch

from oneflow_b200.ops import gemm as G
from oneflow_b200.ops import kernels as K
from oneflow_b200.ops import _native

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16


def close(a, b, rtol=1e-2, atol=None):
    """Element-wise bound ``|a - b| <= atol + rtol * |b|`` against the fp32 statement. ``rtol`` covers the rounding of a
    bf16 result (2^-8) with margin; ``atol`` defaults to 1 % of the reference's RMS, which is what cancellation in an
    fp32-accumulated sum of bf16 products can leave on elements that are themselves close to zero."""
    a, b = a.float().cpu(), b.float().cpu()
    assert a.shape == b.shape, (a.shape, b.shape)
    if atol is None:
        atol = 1e-2 * float(b.pow(2).mean().sqrt()) + 1e-6
    bad = (a - b).abs() > atol + rtol * b.abs()
    if bad.any():
        idx = torch.nonzero(bad)[0].tolist()
        raise AssertionError(f"{int(bad.sum())} of {bad.numel()} elements outside atol={atol:.3g} rtol={rtol}: first at {idx}, "
                             f"got {a[tuple(idx)].item()}, expected {b[tuple(idx)].item()}, max err {(a - b).abs().max().item()}")


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    torch.cuda.synchronize()
    assert _native.read_status() == (0, 0)


@pytest.mark.parametrize("al,bl", [("mk", "nk"), ("mk", "kn"), ("km", "nk"), ("km", "kn")])
@pytest.mark.parametrize("shape", [(128, 128, 64), (520, 392, 264), (2048, 1024, 512)])
def test_gemm_layouts(al, bl, shape):
    M, N, K_ = shape
    torch.manual_seed(1)
    a = torch.randn((M, K_) if al == "mk" else (K_, M), device=DEV, dtype=BF)
    b = torch.randn((N, K_) if bl == "nk" else (K_, N), device=DEV, dtype=BF)
    out = G.gemm(a, b, a_layout=al, b_layout=bl)
    ref = G.gemm_reference(a.cpu(), b.cpu(), al, bl)
    close(out, ref)


@pytest.mark.parametrize("al,bl", [("mk", "nk"), ("mk", "kn"), ("km", "nk"), ("km", "kn")])
@pytest.mark.parametrize("shape", [(512, 768, 320), (1031, 520, 264), (256, 256, 64)])
def test_gemm_two_sm_kernel_layouts(al, bl, shape):
    """The cta_group::2 kernel (256 x 256 tiles over a CTA pair), forced with bn=512 on small and ragged problems."""
    M, N, K_ = shape
    torch.manual_seed(5)
    a = torch.randn((M, K_) if al == "mk" else (K_, M + (-M) % 8), device=DEV, dtype=BF)
    if al == "km":
        a = a[:, :M] if a.shape[1] != M else a
    b = torch.randn((N, K_) if bl == "nk" else (K_, N), device=DEV, dtype=BF)
    out = G.gemm(a, b, a_layout=al, b_layout=bl, bn=512)
    close(out, G.gemm_reference(a.cpu(), b.cpu(), al, bl))


@pytest.mark.parametrize("shape", [(512, 768, 320), (1031, 520, 264)])
def test_gemm_two_sm_kernel_epilogues(shape):
    M, N, K_ = shape
    torch.manual_seed(6)
    a = torch.randn(M, K_, device=DEV, dtype=BF)
    b = torch.randn(N, K_, device=DEV, dtype=BF)
    bias = torch.randn(N, device=DEV, dtype=BF)
    res = torch.randn(M, N, device=DEV, dtype=BF)
    for act in (0, 1, 2, 3):
        out, aux = G.gemm(a, b, bias=bias, act=act, residual=res, want_aux=True, bn=512)
        ref, raux = G.gemm_reference(a.cpu(), b.cpu(), bias=bias.cpu(), act=act, residual=res.cpu(), want_aux=True)
        close(out, ref)
        close(aux, raux)
        if act:
            out = G.gemm(a, b, aux_in=res, act=act, bn=512)
            close(out, G.gemm_reference(a.cpu(), b.cpu(), aux_in=res.cpu(), act=act))
    acc = torch.randn(M, N, device=DEV, dtype=torch.float32)
    ref = G.gemm_reference(a.cpu(), b.cpu(), out=acc.cpu().clone(), accumulate=True, out_dtype=torch.float32, alpha=0.5)
    close(G.gemm(a, b, out=acc, accumulate=True, alpha=0.5, bn=512), ref)
    out32 = G.gemm(a, b, out_dtype=torch.float32, bn=512)
    close(out32, G.gemm_reference(a.cpu(), b.cpu(), out_dtype=torch.float32), rtol=1e-3)


def test_gelu_of_the_epilogue_against_64_bits():
    """Every bf16 value of magnitude 2^-20 .. 12 (and the extremes) through the epilogue's GELU and its gradient, fp32 results."""
    pos = torch.arange(0x3580, 0x4141, dtype=torch.int32).to(torch.int16).view(BF)          # 2^-20 .. 12
    x = torch.cat([pos, -pos, torch.tensor([0.0, 1e4, -1e4, 3e38], dtype=BF)])
    x = torch.nn.functional.pad(x, (0, -x.numel() % 128)).view(-1, 128).to(DEV)
    eye = torch.eye(128, device=DEV, dtype=BF)
    y = G.gemm(x.clone(), eye, act="gelu", out_dtype=torch.float32)
    xd = x.double().requires_grad_(True)
    ref = xd * 0.5 * torch.erfc(-xd * 0.5 ** 0.5)     # erfc keeps the relative accuracy of the negative tail
    ref.sum().backward()
    # relative: 1.5e-7 of the fit, 2 units in the last place each of the exponential and the reciprocal, a dozen roundings; the
    # exponent 0.72 x^2 and its constant are rounded to 2^-24 each, which the exponential turns into 6e-8 x^2
    assert bool(((y.double() - ref).abs() <= (1.5e-6 + 6e-8 * xd.detach() ** 2) * ref.abs() + 1e-36).all())
    ones = torch.ones(x.shape[0], 8, device=DEV, dtype=BF)
    one = torch.zeros(128, 8, device=DEV, dtype=BF)
    one[:, 0] = 1
    g = G.gemm(ones, one, aux_in=x, act="gelu", out_dtype=torch.float32)
    assert bool(((g.double() - xd.grad).abs() <= 1e-6 * xd.grad.abs() + 5e-7).all())


@pytest.mark.parametrize("M,N,K,a_layout,b_layout", [(16006, 304, 3528, "mk", "nk"), (2638, 2040, 6936, "mk", "kn"),
                                                     (9904, 520, 3728, "km", "kn"), (9472, 3328, 136, "km", "kn"), (2331, 768, 3072, "mk", "nk")])
def test_gemm_chooses_a_tiling_close_to_the_best(M, N, K, a_layout, b_layout):
    """Sizes whose tilings differ by a fifth and more: the one that is chosen against each of the three by force."""
    a = torch.randn((M, K) if a_layout == "mk" else (K, M), device=DEV, dtype=BF)
    b = torch.randn((N, K) if b_layout == "nk" else (K, N), device=DEV, dtype=BF)
    call = lambda bn: lambda: G.gemm(a, b, a_layout=a_layout, b_layout=b_layout, bn=bn)  # noqa: E731
    chosen, *forced = timed_in_turn(*(call(bn) for bn in (0, 128, 256, 512)), n=5)
    assert chosen < 1.12 * min(forced), (chosen, forced)


@pytest.mark.parametrize("K", [256, 320, 328, 384, 392])
def test_gemm_short_k_on_both_sides_of_the_line(K):
    """Many tiles and few K blocks, ragged rows and columns: the epilogue-bound kernel up to K = 384 (320 without operands in the
    epilogue), pairs above."""
    torch.manual_seed(25)
    a, b = torch.randn(5003, K, device=DEV, dtype=BF), torch.randn(1160, K, device=DEV, dtype=BF)
    bias = torch.randn(1160, device=DEV, dtype=BF)
    out, aux = G.gemm(a, b, bias=bias, act="gelu", want_aux=True)
    ref, raux = G.gemm_reference(a.cpu(), b.cpu(), bias=bias.cpu(), act="gelu", want_aux=True)
    close(out, ref)
    close(aux, raux)
    close(G.gemm(a, b), G.gemm_reference(a.cpu(), b.cpu()))


def test_gemm_keeps_to_the_limit_of_ctas():
    """48 tiles of 256 x 256 (or 192 of 128 x 128) on two CTAs or one take many times as long as on all, and one longer than two."""
    a, b = torch.randn(3072, 512, device=DEV, dtype=BF), torch.randn(1024, 512, device=DEV, dtype=BF)
    free, two, one = timed_in_turn(*(lambda c=c: G.gemm(a, b, max_ctas=c) for c in (0, 2, 1)), n=3)
    assert two > 10 * free and one > 1.3 * two, (free, two, one)
    close(G.gemm(a, b, max_ctas=1), G.gemm_reference(a.cpu(), b.cpu()))


def test_gemm_default_dispatch_reaches_two_sm_kernel():
    """A problem large enough for the dispatcher's own choice of the two-SM kernel (>= 74 tiles of 256 x 256)."""
    torch.manual_seed(7)
    M, N, K_ = 2560, 2048, 256
    a = torch.randn(M, K_, device=DEV, dtype=BF)
    b = torch.randn(N, K_, device=DEV, dtype=BF)
    bias = torch.randn(N, device=DEV, dtype=BF)
    out = G.gemm(a, b, bias=bias, act=2)
    close(out, G.gemm_reference(a.cpu(), b.cpu(), bias=bias.cpu(), act=2))


@pytest.mark.parametrize("kind,code", [(0, 1), (1, 2), (2, 2)])
def test_bounded_wait_runs_out_and_context_stays_usable(kind, code):
    """Every device-side wait of the library has a limit. Here a one-block kernel waits 5 ms for something that never
    happens (kind 0: an mbarrier nobody arrives on; 1: a peer flag nobody writes; 2: a counter nobody advances): it must
    return by itself, leave the matching status code (1 = mbarrier time-out, 2 = peer time-out), and the next kernel
    must run normally."""
    import ctypes
    from ctypes import c_int, c_longlong, c_void_p
    lib = _native.kernels()
    torch.cuda.synchronize()
    assert _native.read_status() == (0, 0)
    elapsed = torch.zeros(1, dtype=torch.int32, device=DEV)
    rc = lib.ofb_wait_probe(c_int(kind), c_longlong(5_000_000), c_void_p(elapsed.data_ptr()), _native.stream_ptr())
    assert rc == 0
    torch.cuda.synchronize()
    st = _native.read_status()          # reads and clears
    assert st[0] == code and st[1] == 7001 + kind, st
    us = int(elapsed.item())
    assert 4_000 <= us <= 500_000, us   # gave up after the limit, not before, and nowhere near the default of seconds
    # the context is intact: a GEMM right after it computes the right thing and the status stays clean
    a = torch.randn(256, 128, device=DEV, dtype=BF)
    b = torch.randn(128, 128, device=DEV, dtype=BF)
    close(G.gemm(a, b), G.gemm_reference(a.cpu(), b.cpu()))
    torch.cuda.synchronize()
    assert _native.read_status() == (0, 0)


@pytest.mark.parametrize("bn", [128, 256])
def test_gemm_epilogues(bn):
    torch.manual_seed(2)
    M, N, K_ = 384, 512, 256
    a = torch.randn(M, K_, device=DEV, dtype=BF)
    b = torch.randn(N, K_, device=DEV, dtype=BF)
    bias = torch.randn(N, device=DEV, dtype=BF)
    res = torch.randn(M, N, device=DEV, dtype=BF)
    for act in (1, 2, 3):
        out, aux = G.gemm(a, b, bias=bias, act=act, residual=res, want_aux=True, bn=bn)
        ref, raux = G.gemm_reference(a.cpu(), b.cpu(), bias=bias.cpu(), act=act, residual=res.cpu(), want_aux=True)
        close(out, ref)
        close(aux, raux)
        out = G.gemm(a, b, aux_in=res, act=act, bn=bn)
        close(out, G.gemm_reference(a.cpu(), b.cpu(), aux_in=res.cpu(), act=act))
    acc = torch.randn(M, N, device=DEV, dtype=torch.float32)
    ref = G.gemm_reference(a.cpu(), b.cpu(), out=acc.cpu().clone(), accumulate=True, out_dtype=torch.float32, alpha=0.5)
    out = G.gemm(a, b, out=acc, accumulate=True, alpha=0.5, bn=bn)
    close(out, ref)


@pytest.mark.parametrize("cols", [64, 1024, 4096, 8192])
def test_layer_norm(cols):
    torch.manual_seed(3)
    rows = 515
    x = torch.randn(rows, cols, device=DEV, dtype=BF) * 2 + 0.5
    g = torch.randn(cols, device=DEV, dtype=BF)
    b = torch.randn(cols, device=DEV, dtype=BF)
    y, mean, rstd = K.layer_norm_fwd(x, g, b, 1e-5)
    ry, rmean, rrstd = K.layer_norm_fwd(x.cpu(), g.cpu(), b.cpu(), 1e-5)
    close(y, ry)
    close(mean, rmean, 1e-3, 1e-3)
    close(rstd, rrstd, 1e-3, 1e-3)
    ref = torch.nn.functional.layer_norm(x.float().cpu(), (cols,), g.float().cpu(), b.float().cpu(), 1e-5)
    close(y, ref)
    dy = torch.randn(rows, cols, device=DEV, dtype=BF)
    add = torch.randn(rows, cols, device=DEV, dtype=BF)
    dx, dg, db = K.layer_norm_bwd(dy, x, g, mean, rstd, add_to_dx=add)
    rdx, rdg, rdb = K.layer_norm_bwd(dy.cpu(), x.cpu(), g.cpu(), rmean, rrstd, add_to_dx=add.cpu())
    close(dx, rdx)
    close(dg, rdg, 2e-2, 5e-2)
    close(db, rdb, 2e-2, 5e-2)


@pytest.mark.parametrize("rows,cols", [(1, 8), (17, 256), (9, 264), (2500, 512), (130, 520), (1300, 1024), (7, 1032), (1, 2048), (300, 2056),
                                       (1184, 512), (1185, 512), (1184, 1024), (1185, 1024), (4, 1536), (5, 1536), (148, 1032), (149, 1032), (740, 2048), (741, 2048), (1185, 2048), (1777, 2048),
                                       (64, 512), (65, 512), (148, 1024), (149, 1024), (1000, 256), (1100, 248)])
def test_layer_norm_narrow_rows(rows, cols):
    """Widths on both sides of what a warp's lanes hold (256, 512, 1024, 2048), one row to more rows than warps, and the numbers of
    rows at which another kernel takes over."""
    torch.manual_seed(17)
    x = torch.randn(rows, cols, device=DEV, dtype=BF) * 0.5 + 3.0
    g, b = torch.randn(cols, device=DEV, dtype=BF), torch.randn(cols, device=DEV, dtype=BF)
    dy, add = torch.randn(rows, cols, device=DEV, dtype=BF), torch.randn(rows, cols, device=DEV, dtype=BF)
    y, mean, rstd = K.layer_norm_fwd(x, g, b, 1e-5)
    xd, gd, bd = (t.double().requires_grad_(True) for t in (x, g, b))
    ref = torch.nn.functional.layer_norm(xd, (cols,), gd, bd, 1e-5)
    ref.backward(dy.double())
    # one rounding of the result to bf16 (2^-8); fp32 sums: 2^-24 of |x| <= 6 against a spread of 0.5, a few times over
    close(y, ref, 2.0 ** -8 * 1.02, 2e-5)
    close(mean, xd.mean(1), 1e-6, 1e-6)
    dx, dg, db = K.layer_norm_bwd(dy, x, g, mean, rstd, add_to_dx=add)
    close(dx, xd.grad + add.double(), 2.0 ** -8 * 1.02, 1e-4)
    close(dg, gd.grad, 1e-4, 1e-4 * rows ** 0.5)
    close(db, bd.grad, 1e-5, 1e-5 * rows ** 0.5)
    _, hg, hb = K.layer_norm_bwd(dy, x, g, mean, rstd, add_to_dx=add, param_dtype=BF)
    assert torch.equal(hg, dg.to(BF)) and torch.equal(hb, db.to(BF))      # the same fp32 sums, rounded once
    acc_g, acc_b = torch.ones(cols, device=DEV), torch.ones(cols, device=DEV)
    dx2, _, _ = K.layer_norm_bwd(dy, x, g, mean, rstd, dgamma=acc_g, dbeta=acc_b)
    close(dx2, xd.grad, 2.0 ** -8 * 1.02, 1e-4)
    close(acc_g, gd.grad + 1, 1e-4, 1e-4 * rows ** 0.5)
    close(acc_b, bd.grad + 1, 1e-5, 1e-5 * rows ** 0.5)
    plain, _, _ = K.layer_norm_fwd(x, None, None, 1e-5)
    close(plain, torch.nn.functional.layer_norm(xd, (cols,)), 2.0 ** -8 * 1.02, 2e-5)


def test_rows_without_columns_are_refused():
    """They have neither a mean nor a column to sum; without rows there is nothing to do."""
    x = torch.empty(4, 0, device=DEV, dtype=BF)
    with pytest.raises(_native.NativeLibraryError):
        K.layer_norm_fwd(x, None, None, 1e-5)
    for dt in (torch.float32, BF):
        with pytest.raises(_native.NativeLibraryError):
            K.column_sum(x, out_dtype=dt)
    none = torch.empty(0, 64, device=DEV, dtype=BF)
    assert K.layer_norm_fwd(none, None, None, 1e-5)[0].shape == (0, 64)
    assert not K.column_sum(none).any() and K.column_sum(none).shape == (64,)


@pytest.mark.parametrize("rows,cols", [(2331, 264), (2331, 768), (2331, 1000), (2331, 1280), (2331, 2040)])
def test_layer_norm_mean_is_rounded_once(rows, cols):
    """Row means of values around 1, no power of two in a row, against 64 bits."""
    g = torch.Generator(device=DEV).manual_seed(3)
    x = (torch.randn(rows, cols, device=DEV, generator=g) + 1).to(BF)
    _, mean, rstd = K.layer_norm_fwd(x, None, None, 1e-5)
    ref = x.double().mean(1)
    # half a unit in the last place (2^-24 above 1, 2^-25 below). A lane's sum of at most 64 bf16 values rounds away a last bit now
    # and then: up to 8 % more over such rows in an emulation on the CPU, where 32-bit sums across the lanes are up to 4 times off
    bound = torch.where(ref >= 1, 2.0 ** -24, 2.0 ** -25) * 1.25
    assert bool(((mean.double() - ref).abs() <= bound).all())
    # the square sum of short chains, a division, rsqrtf to two units: 1.5e-7 each at most, 1e-7 root mean square in all
    r64 = 1 / torch.sqrt(x.double().var(1, unbiased=False) + 1e-5)
    assert float((rstd.double() / r64 - 1).pow(2).mean().sqrt()) < 1e-7


@pytest.mark.parametrize("rows,C,residual", [(1, 8, False), (37, 96, True), (5003, 64, True), (4099, 64, False), (130, 2048, True)])
def test_batch_norm_sign_mask(rows, C, residual):
    """The backward from the forward's one-bit mask: the same masked gradient as from y (bit for bit), and right against 64 bits.
    Channel counts that do and do not divide a block, rows around the ones a thread keeps in flight."""
    from oneflow_b200.ops import cnn as N
    torch.manual_seed(18)
    x, dy = torch.randn(rows, C, device=DEV, dtype=BF), torch.randn(rows, C, device=DEV, dtype=BF)
    res = torch.randn(rows, C, device=DEV, dtype=BF) if residual else None
    g, b = torch.rand(C, device=DEV) + 0.5, torch.randn(C, device=DEV)
    mask = torch.empty(rows * C // 8, device=DEV, dtype=torch.uint8)
    y, mean, rstd = N.bn_train_fwd(x, g, b, res, True, mask=mask)
    bits = (mask.view(-1, 1) >> torch.arange(8, device=DEV, dtype=torch.uint8)) & 1
    assert torch.equal(bits.view(rows, C).bool(), y > 0)
    dx, dres, dg, db = N.bn_train_bwd(dy, x, None, mean, rstd, g, True, residual, mask=mask)
    dx2, dres2, dg2, db2 = N.bn_train_bwd(dy, x, y, mean, rstd, g, True, residual)
    masked = torch.where(y > 0, dy, torch.zeros_like(dy))
    if residual:
        assert torch.equal(dres, masked) and torch.equal(dres2, masked)
    gd = masked.double()
    xh = (x.double() - mean.double()) * rstd.double()
    s1, s2 = gd.sum(0), (gd * xh).sum(0)
    ref = g.double() * rstd.double() * (gd - s1 / rows - xh * s2 / rows)
    # the sums in a given workspace, the parameter gradients written and added in place
    work, grads = torch.zeros(4 * C, device=DEV), [torch.full((C,), 7.0, device=DEV), torch.full((C,), -3.0, device=DEV)]
    y3, mean3, rstd3 = N.bn_train_fwd(x, g, b, res, True, mask=mask, sums=work[:2 * C])
    close(mean3, x.double().mean(0), 1e-5, 1e-6)
    dx3, _, dg3, db3 = N.bn_train_bwd(dy, x, None, mean3, rstd3, g, True, residual, mask, work[2 * C:], grads, (False, True))
    assert dg3 is grads[0] and db3 is grads[1]
    for d, sg, sb in ((dx, dg, db), (dx2, dg2, db2), (dx3, dg3, db3 + 3.0)):
        # fp32 sums of up to 5003 terms in any order, 2^-24 each against their magnitude; dx rounded to bf16 once
        close(sg, s2, 1e-5, 1e-5 * rows ** 0.5)
        close(sb, s1, 1e-5, 1e-5 * rows ** 0.5)
        close(d, ref, 2.0 ** -8 * 1.02, 1e-5 * float(rstd.max()))


@pytest.mark.parametrize("N,H,W,C,R,stride,pad,ldc", [(2, 224, 224, 3, 7, 2, 3, 152), (1, 9, 11, 3, 7, 2, 3, 152), (3, 5, 7, 4, 3, 1, 1, 40),
                                                      (1, 1, 1, 1, 3, 1, 1, 16), (1, 4, 5000, 8, 3, 2, 1, 72),
                                                      (1, 97, 95, 3, 7, 2, 3, 152), (700, 33, 45, 3, 7, 2, 3, 160), (600, 3, 1300, 3, 7, 2, 3, 152),
                                                      (2, 120, 5000, 3, 7, 2, 3, 152), (3, 150, 701, 4, 3, 1, 1, 40), (40, 64, 65, 4, 3, 1, 1, 40),
                                                      (1, 40, 41, 130, 15, 1, 7, 29256)])
def test_im2col_small(N, H, W, C, R, stride, pad, ldc):
    """Odd sizes, padding columns, one pixel; more and less than 2^20 vectors of results (read directly, or staged); output rows in
    one piece and in several (few of them; too wide for shared memory); windows too large for it; copies, so bit for bit."""
    from oneflow_b200.ops import cnn
    x = torch.randn(N, H, W, C, device=DEV, dtype=BF)
    got, hw = cnn.im2col_small(x, R, R, stride, pad, ldc)
    ref, hw2 = cnn.im2col_small(x.cpu(), R, R, stride, pad, ldc)
    assert hw == hw2 and torch.equal(got.cpu(), ref)


@pytest.mark.parametrize("N,H,W,C", [(2, 7, 9, 8), (1, 1, 1, 16), (3, 56, 56, 24), (2, 113, 57, 40), (1, 2, 301, 8), (5, 64, 1, 16)])
def test_pool_and_stride_index_kernels(N, H, W, C):
    from oneflow_b200.ops import cnn
    x = torch.randn(N, H, W, C, device=DEV, dtype=BF)
    y, idx = cnn.maxpool3x3s2_fwd(x)
    ry, ridx = cnn.maxpool3x3s2_fwd(x.cpu())
    assert torch.equal(y.cpu(), ry)
    dy = torch.randn_like(y)
    # the taps point at the maxima; ties between equal pixels may choose either of them, so the gradient is checked for these taps
    OH, OW = y.shape[1:3]
    tap = idx.long()
    h = 2 * torch.arange(OH, device=DEV).view(1, -1, 1, 1) - 1 + tap // 3
    w = 2 * torch.arange(OW, device=DEV).view(1, 1, -1, 1) - 1 + tap % 3
    assert bool(((h >= 0) & (h < H) & (w >= 0) & (w < W)).all())
    flat = ((torch.arange(N, device=DEV).view(-1, 1, 1, 1) * H + h) * W + w) * C + torch.arange(C, device=DEV)
    assert torch.equal(x.flatten()[flat], y)
    want = torch.zeros(x.numel(), device=DEV, dtype=torch.float64).scatter_add_(0, flat.flatten(), dy.double().flatten())
    size = torch.zeros_like(want).scatter_add_(0, flat.flatten(), dy.double().abs().flatten())
    got = cnn.maxpool3x3s2_bwd(dy, idx, (N, H, W, C)).double().flatten()
    # up to four bf16 gradients meet in fp32 (three roundings of 2^-24 of their size) and are rounded once to bf16
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 3 * 2.0 ** -24 * size).all())
    s = cnn.subsample2(x)
    assert torch.equal(s, x[:, ::2, ::2])
    up = cnn.upsample2_zero(s, (N, H, W, C))
    ref = torch.zeros_like(x)
    ref[:, ::2, ::2] = s
    assert torch.equal(up, ref)


def test_index_kernels_beyond_32_bits():
    """2^31 vectors and a few: the instances of the index kernels that divide in 64 bits (34 GB of results; the pooling and
    subsampling kernels read four times as much and share the same arithmetic)."""
    from oneflow_b200.ops import cnn
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 60 GB")
    N, H, W, C = 1032, 65, 64, 4096          # 2,197,946,368 vectors of 8
    assert N * H * W * (C // 8) > 1 << 31
    dy = torch.randn(N, C, device=DEV, dtype=BF)
    dx = cnn.avgpool_bwd(dy, (N, H, W, C))
    want = (dy.float() * (1.0 / (H * W))).to(BF)
    for n in range(N):
        assert bool((dx[n] == want[n]).all()), n
    del dx
    dy = torch.randn(N, (H + 1) // 2, W // 2, C, device=DEV, dtype=BF)
    dx = cnn.upsample2_zero(dy, (N, H, W, C))
    for n in range(N):
        assert torch.equal(dx[n, ::2, ::2], dy[n]) and not dx[n, 1::2].any() and not dx[n, :, 1::2].any(), n


@pytest.mark.parametrize("act", [1, 2, 3])
def test_bias_act(act):
    torch.manual_seed(4)
    x = torch.randn(300, 1024, device=DEV, dtype=BF)
    b = torch.randn(1024, device=DEV, dtype=BF)
    dy = torch.randn(300, 1024, device=DEV, dtype=BF)
    close(K.bias_act_fwd(x, b, act), K.bias_act_fwd(x.cpu(), b.cpu(), act))
    close(K.bias_act_bwd(x, b, dy, act), K.bias_act_bwd(x.cpu(), b.cpu(), dy.cpu(), act))


def test_bias_mask_scale_and_dropout_mask():
    torch.manual_seed(5)
    x = torch.randn(257, 512, device=DEV, dtype=BF)
    b = torch.randn(512, device=DEV, dtype=BF)
    add = torch.randn(257, 512, device=DEV, dtype=BF)
    mask = K.dropout_mask(x.shape, 0.1, seed=1234, device=DEV)
    keep = mask.float().mean().item()
    assert abs(keep - 0.9) < 0.01
    mask2 = K.dropout_mask(x.shape, 0.1, seed=1234, device=DEV)
    assert torch.equal(mask, mask2)
    y = K.bias_mask_scale(x, b, mask, 1 / 0.9, add)
    close(y, K.bias_mask_scale(x.cpu(), b.cpu(), mask.cpu(), 1 / 0.9, add.cpu()))


@pytest.mark.parametrize("rows,cols", [(1, 8), (31, 64), (256, 72), (1025, 776), (5000, 128), (3, 4096), (8200, 1024)])
def test_column_sum_outputs(rows, cols):
    """Rows around what a cluster takes per step (256, unrolled 1024), columns around the 64 it owns, and a matrix on the other side
    of the size limit; all three outputs."""
    torch.manual_seed(19)
    x = torch.randn(rows, cols, device=DEV, dtype=BF)
    ref = x.double().sum(0)
    out = K.column_sum(x)
    close(out, ref, 1e-6, 1e-6 * rows ** 0.5 * 4)       # fp32 sums in a tree of short chains
    # one rounding to bf16 (2^-8); beside it only the order of the atomics of a large matrix
    close(K.column_sum(x, out_dtype=BF), ref, 2.0 ** -8 * 1.01, 1e-6 * rows ** 0.5 * 4)
    acc = torch.full((cols,), 2.0, device=DEV)
    assert K.column_sum(x, out=acc) is acc
    close(acc, ref + 2.0, 1e-6, 1e-6 * rows ** 0.5 * 4)


def timed_in_turn(*calls, n=20, rounds=5):
    """Device time of each call (best of several rounds, the calls in turn, captured so that the host does not count), in ms."""
    graphs = []
    for fn in calls:
        fn()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(n):
                fn()
        graphs.append(g)
    best = [1e9] * len(calls)
    for _ in range(rounds):
        for i, g in enumerate(graphs):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            g.replay()
            b.record()
            torch.cuda.synchronize()
            best[i] = min(best[i], a.elapsed_time(b) / n)
    return best


@pytest.mark.parametrize("rows,cols", [(100000, 64), (25488, 40), (512, 16384), (8192, 256)])
def test_column_sum_takes_the_kernel_that_suits_the_shape(rows, cols):
    """Tall or wide matrices: returning the sums costs no more than clearing a buffer and adding them to it (five times as much
    by the kernel for small matrices)."""
    x = torch.randn(rows, cols, device=DEV, dtype=BF)
    got, want = timed_in_turn(lambda: K.column_sum(x), lambda: K.column_sum(x, out=torch.zeros(cols, device=DEV)))
    assert got < 1.25 * want + 0.0003, (got, want)


def test_cast_scale_column_sum():
    torch.manual_seed(6)
    x = torch.randn(1000, 776, device=DEV, dtype=BF)
    st = torch.tensor([0.25], device=DEV)
    y = K.cast_scale(x, 2.0, torch.float32, st)
    close(y, x.float().cpu() * 0.5, 1e-3, 1e-3)
    close(K.column_sum(x), x.float().cpu().sum(0), 1e-2, 1e-2)


@pytest.mark.parametrize("cols", [128, 512, 2048])
def test_softmax_tril(cols):
    torch.manual_seed(7)
    x = torch.randn(2, 3, cols, cols, device=DEV, dtype=BF)
    mask = K.dropout_mask(x.shape, 0.1, seed=7, device=DEV)
    y, sm = K.softmax_fwd(x, scale=0.125, tril=True, dropout_mask=mask, dropout_scale=1 / 0.9, want_softmax=True)
    ry, rsm = K.softmax_fwd(x.cpu(), scale=0.125, tril=True, dropout_mask=mask.cpu(), dropout_scale=1 / 0.9,
                            want_softmax=True)
    close(y, ry)
    close(sm, rsm)
    dy = torch.randn_like(x)
    dx = K.softmax_bwd(sm, dy, scale=0.125, tril=True, dropout_mask=mask, dropout_scale=1 / 0.9)
    rdx = K.softmax_bwd(rsm, dy.cpu(), scale=0.125, tril=True, dropout_mask=mask.cpu(), dropout_scale=1 / 0.9)
    close(dx, rdx, 2e-2, 1e-3)


def test_softmax_attn_mask():
    torch.manual_seed(8)
    B, H, S = 2, 4, 256
    x = torch.randn(B, H, S, S, device=DEV, dtype=BF)
    am = (torch.rand(S, S, device=DEV) > 0.2)
    y = K.softmax_fwd(x, scale=0.5, attn_mask=am)
    ry = K.softmax_fwd(x.cpu(), scale=0.5, attn_mask=am.cpu())
    close(y, ry)


@pytest.mark.parametrize("vocab", [1024, 50304])
def test_xent(vocab):
    torch.manual_seed(9)
    rows = 300
    logits = torch.randn(rows, vocab, device=DEV, dtype=BF) * 3
    labels = torch.randint(0, vocab, (rows,), device=DEV)
    labels[5] = -100
    st = K.xent_stats(logits, labels)
    loss, d = K.xent_grad(logits, labels, st, grad_scale=0.5)
    ref = torch.nn.functional.cross_entropy(logits.float().cpu(), labels.cpu(), reduction="none", ignore_index=-100)
    close(loss, ref, 1e-3, 1e-3)
    lf = logits.float().cpu().requires_grad_(True)
    torch.nn.functional.cross_entropy(lf, labels.cpu(), reduction="sum", ignore_index=-100).mul(0.5).backward()
    close(d, lf.grad, 2e-2, 1e-3)
    # vocabulary-sharded path: two shards merged
    half = vocab // 2
    p0 = K.xent_stats(logits[:, :half].contiguous(), labels, 0)
    p1 = K.xent_stats(logits[:, half:].contiguous(), labels, half)
    merged = K.xent_merge(torch.stack([p0, p1]))
    close(merged[:, 2], st[:, 2], 1e-3, 1e-3)
    l2, _ = K.xent_grad(logits[:, half:].contiguous(), labels, merged, vocab_start=half)
    close(l2, ref, 1e-3, 1e-3)


@pytest.mark.parametrize("rows,cols", [(4096, 1000), (4096, 8192), (296, 8200), (4096, 16392), (4096, 50304)])
def test_xent_sum_accuracy(rows, cols):
    """The sum of exponentials of unit-normal logits against 64 bits, for every number of threads a row is given."""
    err = []
    for rep in range(max(1, 8192 // rows)):
        g = torch.Generator(device=DEV).manual_seed(40 + rep)
        x = torch.randn(rows, cols, device=DEV, generator=g).to(BF)
        st = K.xent_stats(x, torch.zeros(rows, dtype=torch.long, device=DEV))
        xd = x.double()
        err.append(st[:, 1].double() / torch.exp(xd - xd.max(1, keepdim=True).values).sum(1) - 1)
    err = torch.cat(err)
    # One rounding to fp32 is 2^-24 / sqrt(3) = 3.4e-8 of the power of two below, 2.5e-8 of the value on average; the threads'
    # own sums and exponentials average out over 128 threads or more. A sum added in fp32 throughout adds a second rounding of
    # that size (the last levels of the tree): 3.5e-8 before anything else.
    assert float(err.pow(2).mean().sqrt()) < 3.5e-8
    assert abs(float(err.mean())) < 1e-8      # __expf errs by a few units in the last place, not to one side


@pytest.mark.parametrize("rows,cols,expanded", [(1, 8, False), (3, 4096, True), (5, 16384 + 8, False), (1200, 2 * 16384 - 8, True),
                                                 (300, 4104, False), (297, 8184, True), (297, 8200, False), (300, 16384, True),
                                                 (4, 16392, False), (9600, 264, False)])
def test_xent_row_scale_and_extremes(rows, cols, expanded):
    """Widths around the 4096, 8192 and 16384 elements a block of 128, 256 and 512 threads takes per step and around those at which
    the number of threads changes, more rows than blocks in the gradient (1184) and in the statistics (9472), incoming gradients per
    row or one value; entries of -inf, the type's lowest value and a row maximum that comes last."""
    torch.manual_seed(16)
    logits = torch.randn(rows, cols, device=DEV, dtype=BF) * 3
    labels = torch.randint(0, cols, (rows,), device=DEV)
    logits[0, : cols // 2] = float("-inf")
    labels[0] = cols - 1
    logits[-1, -1] = 40.0
    if rows > 2:
        logits[1] = torch.finfo(BF).min
        logits[1, 3] = 1.0
        labels[1] = 3
        labels[2] = -100
    g = torch.rand(1 if expanded else rows, device=DEV).add(0.5).expand(rows)
    st = K.xent_stats(logits, labels)
    loss, d = K.xent_grad(logits, labels, st, row_scale=g)
    lf = logits.double().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(lf, labels, reduction="none", ignore_index=-100)
    (ref * g.double()).sum().backward()
    # fp32 sums of exponentials that are good to 2 units in the last place; the gradient is rounded to bf16 once
    close(loss, ref, 1e-5, 1e-5)
    close(d, lf.grad, 2.0 ** -8 * 1.05, 1e-6)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_fmha_fwd(D, causal):
    torch.manual_seed(10)
    B, S, H = 2, 384, 3
    qkv = torch.randn(B, S, 3, H, D, device=DEV, dtype=BF)
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    out, lse = K.fmha_fwd(q, k, v, causal=causal)
    ro, rl = K.fmha_reference(q.cpu(), k.cpu(), v.cpu(), causal, 1 / math.sqrt(D))
    close(out, ro)
    close(lse, rl, 1e-2, 1e-2)


def test_fmha_fwd_padding_and_ragged():
    torch.manual_seed(11)
    B, S, H, D = 3, 200, 2, 64
    q = torch.randn(B, S, H, D, device=DEV, dtype=BF)
    k = torch.randn(B, S, H, D, device=DEV, dtype=BF)
    v = torch.randn(B, S, H, D, device=DEV, dtype=BF)
    kv_len = torch.tensor([200, 77, 130], dtype=torch.int32)
    out, lse = K.fmha_fwd(q, k, v, causal=False, kv_len=kv_len)
    ro, rl = K.fmha_reference(q.cpu(), k.cpu(), v.cpu(), False, 1 / math.sqrt(D), kv_len)
    close(out, ro)
    close(lse, rl, 1e-2, 1e-2)


# Forward: pairs of query tiles (at least 148 of them: many heads) and key tiles split between the two streams of a CTA (few);
# edges of the 128-row tiles, a pair whose second tile has no rows, odd numbers of key tiles, rows that see no key, short kv_len.
# Backward: one and several key tiles, a single row, both head sizes.
@pytest.mark.parametrize("B,H,Hk,Sq,Sk,D,causal,lens", [
    (10, 15, 15, 100, 129, 64, False, None),     # 150 pairs, second tile empty
    (5, 16, 4, 257, 257, 128, True, None),       # 160 pairs, one row in the last tile
    (5, 16, 16, 300, 140, 64, True, None),       # rows above the shifted diagonal see nothing; first tile of a pair may be idle
    (37, 4, 2, 129, 385, 64, False, (0, 1, 128, 129, 385)),
    (2, 3, 1, 257, 300, 128, True, None),        # split: one, two and three key tiles for a row tile
    (1, 2, 2, 1, 1, 64, False, None),
    (1, 2, 2, 130, 640, 64, False, (513,)),
    (2, 2, 2, 200, 100, 128, True, None),
])
def test_fmha_streams_and_tile_edges(B, H, Hk, Sq, Sk, D, causal, lens):
    torch.manual_seed(15)
    q = torch.randn(B, Sq, H, D, device=DEV, dtype=BF)
    k, v = (torch.randn(B, Sk, Hk, D, device=DEV, dtype=BF) for _ in range(2))
    kv_len = None if lens is None else torch.tensor([lens[i % len(lens)] for i in range(B)], dtype=torch.int32, device=DEV)
    sc = 1 / math.sqrt(D)
    out, lse = K.fmha_fwd(q, k, v, causal=causal, kv_len=kv_len)
    ro, rl = K.fmha_reference(q, k, v, causal, sc, kv_len)
    # P is rounded to bf16 (half a unit in the last place is at most 2^-8 of the value) before it multiplies v, and both results
    # are rounded to bf16: the difference is at most 2^-8 sum p |v| + 2 * 2^-8 |o|, with 2 % for the fp32 parts
    ab, _ = K.fmha_reference(q, k, v.abs(), causal, sc, kv_len)
    assert bool(((out.float() - ro.float()).abs() <= 1.02 * (ab.float() / 256 + ro.float().abs() / 128) + 1e-6).all())
    seen = torch.isfinite(rl)
    assert torch.equal(seen, torch.isfinite(lse))
    close(lse[seen], rl[seen], 1e-2, 1e-2)
    d_o = torch.randn_like(out)
    got = K.fmha_bwd(q, k, v, out, d_o, lse, causal=causal, kv_len=kv_len, separate=True)
    assert all(t.is_contiguous() for t in got)
    for g, r in zip(got, K.fmha_bwd_reference(q, k, v, out, d_o, lse, causal, sc, kv_len)):
        close(g, r, 3e-2, 2e-2)


def _attention_backward_with_bounds(q, k, v, o, d_o, causal, kv_len, p, keep):
    """(reference, bound) of dq, dk, dv in fp32 for the forward's own (rounded) output: the kernel rounds P and dS to bf16, half a
    unit in the last place each (at most 2^-8 of the value, and dS is formed from the rounded P), and every result once; 5 % for
    the fp32 parts."""
    B, Sq, H, D = q.shape
    Sk, Hk = k.shape[1:3]
    qf, kf, vf, of, df = (t.float().permute(0, 2, 1, 3) for t in (q, k, v, o, d_o))
    kx, vx = kf.repeat_interleave(H // Hk, 1), vf.repeat_interleave(H // Hk, 1)
    s = qf @ kx.transpose(-1, -2) / math.sqrt(D)
    if causal:
        s = s.masked_fill(~torch.ones(Sq, Sk, dtype=torch.bool, device=q.device).tril(Sk - Sq), float("-inf"))
    if kv_len is not None:
        s = s.masked_fill(torch.arange(Sk, device=q.device) >= kv_len[:, None, None, None], float("-inf"))
    pr = torch.nan_to_num(torch.softmax(s, -1))          # rows that see no key
    z = 1.0 if keep is None else keep.float() / (1 - p)
    ds = pr * (df @ vx.transpose(-1, -2) * z - (df * of).sum(-1, keepdim=True)) / math.sqrt(D)
    pd = pr * z

    def fold(t):        # sum over the query heads of a group
        return t.view(B, Hk, H // Hk, Sk, D).sum(2)
    dst, adst, pdt = ds.transpose(-1, -2), ds.abs().transpose(-1, -2), pd.transpose(-1, -2)
    ref = (ds @ kx, fold(dst @ qf), fold(pdt @ df))
    terms = (2.0 ** -7 * (ds.abs() @ kx.abs()), 2.0 ** -7 * fold(adst @ qf.abs()), 2.0 ** -8 * fold(pdt @ df.abs()))
    return [(r.permute(0, 2, 1, 3), (1.05 * (t + r.abs() * 2.0 ** -8) + 1e-5).permute(0, 2, 1, 3)) for r, t in zip(ref, terms)]


# Which form of the forward kernel the sizes choose is said beside them; "items" are what a CTA of the 148 works through in turn, so that
# every slot and phase of its barriers comes round more than once.
@pytest.mark.parametrize("B,H,Hk,Sq,Sk,D,causal,lens,p", [
    (50, 16, 16, 200, 200, 64, False, None, 0.2),                       # 800 pairs (5 items), 1600 key tiles (11 items)
    (50, 16, 4, 256, 320, 128, True, None, 0.2),                        # 800 pairs, 600 key tiles of four heads each
    (50, 16, 16, 300, 140, 64, True, (0, 140, 65, 0, 129, 64, 140), 0.2),   # 1600 pairs: empty, of one stream only, one or two tiles
    (50, 16, 16, 300, 140, 128, True, (0, 140, 65, 0, 129, 64, 140), 0.0),
    (60, 16, 8, 129, 513, 64, False, (513, 0, 128, 385, 1, 257, 512), 0.0),  # 960 pairs of one to five tiles, 2400 key tiles
    (3, 4, 2, 130, 100, 128, True, None, 0.2),                          # one key tile in halves
    (2, 8, 8, 200, 64, 64, False, None, 0.2),                           # only its first half
    (1, 4, 4, 1, 128, 128, False, None, 0.0),
    (2, 3, 3, 7, 65, 64, False, None, 0.0),                             # one key in the second half
    (40, 16, 16, 64, 128, 64, False, None, 0.0),                        # one key tile, 640 pairs
    (3, 4, 4, 100, 300, 64, False, (300, 129, 320), 0.2),               # split, three tiles: the last halved; two tiles
    (3, 4, 4, 100, 641, 128, True, (641, 577, 576), 0.2),               # split, five tiles and a key, then halves of one key and none
    (20, 16, 4, 3, 641, 128, False, None, 0.0),                         # split for its length, in three waves
    (90, 8, 8, 20, 385, 64, False, None, 0.2),                          # split with dropout, five waves
])
def test_fmha_items_halves_and_dropout(B, H, Hk, Sq, Sk, D, causal, lens, p):
    torch.manual_seed(24)
    q, d_o = torch.randn(B, Sq, H, D, device=DEV, dtype=BF), torch.randn(B, Sq, H, D, device=DEV, dtype=BF)
    k, v = (torch.randn(B, Sk, Hk, D, device=DEV, dtype=BF) for _ in range(2))
    kv_len = None if lens is None else torch.tensor([lens[i % len(lens)] for i in range(B)], dtype=torch.int32, device=DEV).clamp(max=Sk)
    sc, drop = 1 / math.sqrt(D), dict(dropout_p=p, seed=0x1234567890ABCDEF, offset=9)
    keep = K.fmha_dropout_mask(B, H, Sq, Sk, p, drop["seed"], 9, DEV) if p else None
    out, lse = K.fmha_fwd(q, k, v, causal=causal, kv_len=kv_len, **drop)
    ro, rl = K.fmha_reference(q, k, v, causal, sc, kv_len, p, keep)
    ab, _ = K.fmha_reference(q, k, v.abs(), causal, sc, kv_len, p, keep)
    # as in the test above: P and both results are rounded to bf16
    assert bool(((out.float() - ro.float()).abs() <= 1.02 * (ab.float() / 256 + ro.float().abs() / 128) + 1e-6).all())
    seen = torch.isfinite(rl)
    assert torch.equal(seen, torch.isfinite(lse))
    close(lse[seen], rl[seen], 1e-5, 1e-5)       # fp32 on both sides
    got = K.fmha_bwd(q, k, v, out, d_o, lse, causal=causal, kv_len=kv_len, separate=True, **drop)
    for g, (r, bound) in zip(got, _attention_backward_with_bounds(q, k, v, out, d_o, causal, kv_len, p, keep)):
        assert bool(((g.float() - r).abs() <= bound).all())


def test_multi_tensor_adamw_sgd_and_norm():
    torch.manual_seed(12)
    sizes = [1000, 65536 + 8, 300000, 16]
    def mk(dt=torch.float32):
        return [torch.randn(n, device=DEV, dtype=dt) for n in sizes]
    w, g, m, v = mk(), mk(BF), [t.abs() * 0 for t in mk()], [t.abs() * 0 for t in mk()]
    c = [torch.empty(n, device=DEV, dtype=BF) for n in sizes]
    wc, gc, mc, vc = [[t.cpu().clone() for t in L] for L in (w, g, m, v)]
    cc = [t.cpu().clone() for t in c]
    kw = dict(lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, scale=0.5, step=3)
    K.multi_tensor_adamw(g, w, c, m, v, **kw)
    K.multi_tensor_adamw(gc, wc, cc, mc, vc, **kw)
    for a, b in zip(w + m + v, wc + mc + vc):
        close(a, b, 1e-3, 1e-4)
    for a, b in zip(c, cc):  # bf16 copies: one rounding step apart at most
        close(a, b, 1e-2, 1e-2)
    # SGD momentum
    w, g, m = mk(), mk(), [t * 0 for t in mk()]
    wc, gc, mc = [[t.cpu().clone() for t in L] for L in (w, g, m)]
    kw = dict(lr=0.1, momentum=0.9, nesterov=True, weight_decay=1e-4, l2=1e-3, scale=2.0)
    K.multi_tensor_sgd(g, w, None, m, **kw)
    K.multi_tensor_sgd(gc, wc, None, mc, **kw)
    for a, b in zip(w + m, wc + mc):
        close(a, b, 1e-3, 1e-4)
    g[1][7] = float("inf")
    out = K.multi_tensor_sqsum(g)
    ref = K.multi_tensor_sqsum([t.cpu() for t in g])
    close(out[:1], ref[:1], 1e-3, 1e-3)
    assert int(out[1].item()) == 1
    f, found, norm = K.clip_factor(out, 1.0)
    assert int(found.item()) == 1 and f.item() <= 1.0


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_fmha_bwd(D, causal):
    torch.manual_seed(13)
    B, S, H = 2, 384, 2
    qkv = torch.randn(B, S, 3, H, D, device=DEV, dtype=BF)
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    out, lse = K.fmha_fwd(q, k, v, causal=causal)
    d_o = torch.randn_like(out)
    dq, dk, dv = K.fmha_bwd(q, k, v, out, d_o, lse, causal=causal)
    rq, rk, rv = K.fmha_bwd_reference(q.cpu(), k.cpu(), v.cpu(), out.cpu(), d_o.cpu(), lse.cpu(), causal,
                                      1 / math.sqrt(D))
    close(dq, rq, 3e-2, 2e-2)
    close(dk, rk, 3e-2, 2e-2)
    close(dv, rv, 3e-2, 2e-2)


def test_fmha_bwd_padding_ragged():
    torch.manual_seed(14)
    B, S, H, D = 2, 200, 2, 64
    qkv = torch.randn(B, S, 3, H, D, device=DEV, dtype=BF)
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    kv_len = torch.tensor([200, 90], dtype=torch.int32)
    out, lse = K.fmha_fwd(q, k, v, causal=False, kv_len=kv_len)
    d_o = torch.randn_like(out)
    dq, dk, dv = K.fmha_bwd(q, k, v, out, d_o, lse, causal=False, kv_len=kv_len)
    rq, rk, rv = K.fmha_bwd_reference(q.cpu(), k.cpu(), v.cpu(), out.cpu(), d_o.cpu(), lse.cpu(), False,
                                      1 / math.sqrt(D), kv_len)
    close(dq, rq, 3e-2, 2e-2)
    close(dk, rk, 3e-2, 2e-2)
    close(dv, rv, 3e-2, 2e-2)


@pytest.mark.parametrize("D,causal,Sq,Sk,H,Hk", [(64, True, 200, 456, 4, 2), (128, True, 384, 256, 4, 1), (64, False, 130, 300, 6, 3),
                                                 (128, True, 256, 256, 8, 2), (64, True, 300, 100, 2, 2)])
def test_fmha_grouped_heads_and_unequal_lengths(D, causal, Sq, Sk, H, Hk):
    """Grouped-query heads (H query heads on Hk key/value heads) and Sq != Sk with the causal diagonal at the bottom-right
    corner (Sq > Sk leaves the first rows without any visible key: zero output, zero gradient), forward and backward."""
    torch.manual_seed(21)
    B = 2
    q = torch.randn(B, Sq, H, D, device=DEV, dtype=BF)
    kv = torch.randn(B, Sk, 2, Hk, D, device=DEV, dtype=BF)
    k, v = kv[:, :, 0], kv[:, :, 1]
    sc = 1 / math.sqrt(D)
    out, lse = K.fmha_fwd(q, k, v, causal=causal)
    ro, rl = K.fmha_reference(q.cpu(), k.cpu(), v.cpu(), causal, sc)
    # probabilities are rounded to bf16 (2^-9 relative) before they multiply V ~ N(0, 1): rows that see a handful of keys sum a
    # few terms of magnitude ~0.3 that partly cancel, so the absolute bound is set from that, not from the output's RMS (which
    # the all-zero rows above the shifted diagonal pull down)
    close(out, ro, 1e-2, 5e-3)
    live = torch.isfinite(rl)
    assert torch.equal(torch.isfinite(lse.cpu()), live)
    close(lse.cpu()[live], rl[live], 1e-2, 1e-2)
    d_o = torch.randn_like(out)
    dq, dk, dv = K.fmha_bwd(q, k, v, out, d_o, lse, causal=causal)
    assert dk.shape == (B, Sk, Hk, D) and dq.shape == (B, Sq, H, D)
    rq, rk, rv = K.fmha_bwd_reference(q.cpu(), k.cpu(), v.cpu(), out.cpu(), d_o.cpu(), lse.cpu(), causal, sc)
    close(dq, rq, 3e-2, 2e-2)
    close(dk, rk, 3e-2, 2e-2 * math.sqrt(H // Hk))
    close(dv, rv, 3e-2, 2e-2 * math.sqrt(H // Hk))


@pytest.mark.parametrize("D,causal,p", [(64, True, 0.1), (128, False, 0.3)])
def test_fmha_dropout_follows_its_philox_mask(D, causal, p):
    """The kernels drop probabilities by a Philox stream indexed by position; forward and backward agree with the fp32
    statement that applies the same mask (written out by the mask kernel), the mask keeps about 1 - p of the entries,
    and another offset gives another mask."""
    torch.manual_seed(22)
    B, S, H = 2, 320, 3
    qkv = torch.randn(B, S, 3, H, D, device=DEV, dtype=BF)
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    sc = 1 / math.sqrt(D)
    seed, off = 0x1234567890ABCDEF, 7
    mask = K.fmha_dropout_mask(B, H, S, S, p, seed, off, DEV)
    frac = mask.float().mean().item()
    assert abs(frac - (1 - p)) < 5e-3, frac
    assert not torch.equal(mask, K.fmha_dropout_mask(B, H, S, S, p, seed, off + 1, DEV))
    assert torch.equal(mask, K.fmha_dropout_mask(B, H, S, S, p, seed, off, DEV))
    out, lse = K.fmha_fwd(q, k, v, causal=causal, dropout_p=p, seed=seed, offset=off)
    ro, rl = K.fmha_reference(q.cpu(), k.cpu(), v.cpu(), causal, sc, None, p, mask.cpu())
    close(out, ro)
    close(lse, rl, 1e-2, 1e-2)
    d_o = torch.randn_like(out)
    dq, dk, dv = K.fmha_bwd(q, k, v, out, d_o, lse, causal=causal, dropout_p=p, seed=seed, offset=off)
    rq, rk, rv = K.fmha_bwd_reference(q.cpu(), k.cpu(), v.cpu(), out.cpu(), d_o.cpu(), lse.cpu(), causal, sc, None, p, mask.cpu())
    close(dq, rq, 3e-2, 2e-2)
    close(dk, rk, 3e-2, 2e-2)
    close(dv, rv, 3e-2, 2e-2)


def test_sdpa_entry_point_runs_the_fused_kernels():
    """flow.nn.functional.scaled_dot_product_attention with grouped heads, Sq != Sk and dropout: fused kernels (the launch
    counter moves), gradients flow, eval-mode result equals torch's op on the same inputs."""
    import oneflow_b200 as flow
    torch.manual_seed(23)
    B, H, Hk, Sq, Sk, D = 2, 4, 2, 128, 256, 64
    q = torch.randn(B, H, Sq, D, device=DEV, dtype=BF, requires_grad=True)
    k = torch.randn(B, Hk, Sk, D, device=DEV, dtype=BF, requires_grad=True)
    v = torch.randn(B, Hk, Sk, D, device=DEV, dtype=BF, requires_grad=True)
    n0 = K.launch_count
    y = flow.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True)
    assert K.launch_count > n0
    kk, vv = (t.repeat_interleave(H // Hk, dim=1) for t in (k, v))
    m = torch.ones(Sq, Sk, dtype=torch.bool, device=DEV).tril(Sk - Sq)
    ref = torch.nn.functional.scaled_dot_product_attention(q.float(), kk.float(), vv.float(), attn_mask=m)
    close(y, ref)
    y2 = flow.nn.functional.scaled_dot_product_attention(q, k, v, dropout_p=0.2)
    y2.float().sum().backward()
    assert q.grad is not None and k.grad.shape == k.shape and torch.isfinite(v.grad.float()).all()


@pytest.mark.parametrize("self_inter,T,D", [(False, 26, 128), (True, 26, 128), (False, 7, 64), (False, 31, 32)])
def test_dot_feature_interaction(self_inter, T, D):
    from oneflow_b200.ops.interaction import dot_feature_interaction, dot_feature_interaction_reference
    torch.manual_seed(3)
    B = 517
    dense = (torch.randn(B, D, device="cuda") * 0.5).bfloat16().requires_grad_()
    sparse = (torch.randn(B, T, D, device="cuda") * 0.5).bfloat16().requires_grad_()
    F = T + 1
    npairs = F * (F + 1) // 2 if self_inter else F * (F - 1) // 2
    pad = (-(D + npairs)) % 8 or 8
    n0 = K.launch_count
    out = dot_feature_interaction([dense, sparse], output_concat=dense, self_interaction=self_inter, output_padding=pad)
    assert K.launch_count == n0 + 1, "native interaction kernel did not run"
    d32, s32 = dense.detach().float().requires_grad_(), sparse.detach().float().requires_grad_()
    ref = dot_feature_interaction_reference([d32, s32], output_concat=d32, self_interaction=self_inter, output_padding=pad)
    assert out.shape == ref.shape
    torch.testing.assert_close(out.float(), ref, atol=0.06, rtol=0.02)
    g = (torch.randn_like(ref) * 0.5).bfloat16()
    out.backward(g)
    ref.backward(g.float())
    torch.testing.assert_close(dense.grad.float(), d32.grad, atol=0.15, rtol=0.03)
    torch.testing.assert_close(sparse.grad.float(), s32.grad, atol=0.15, rtol=0.03)


@pytest.mark.parametrize("B", [1, 3, 445, 1333, 6000])
@pytest.mark.parametrize("T", [1, 26, 31])
def test_dot_feature_interaction_backward_tiles(B, T):
    """Three samples a tile, tiles in turn over the SMs and two sets of builder warps: one tile, a tile of one sample, a second tile for
    one SM, a third, several rounds."""
    from oneflow_b200.ops.interaction import dot_feature_interaction, dot_feature_interaction_reference
    torch.manual_seed(5)
    dense = (torch.randn(B, 128, device=DEV) * 0.5).to(BF).requires_grad_()
    sparse = (torch.randn(B, T, 128, device=DEV) * 0.5).to(BF).requires_grad_()
    pad = -(T * (T + 1) // 2) % 8
    out = dot_feature_interaction([dense, sparse], output_concat=dense, output_padding=pad)
    d64, s64 = dense.detach().double().requires_grad_(), sparse.detach().double().requires_grad_()
    ref = dot_feature_interaction_reference([d64, s64], output_concat=d64, output_padding=pad)
    g = torch.randn(out.shape, device=DEV).to(BF)
    out.backward(g)
    ref.backward(g.double())
    # fp32 sums of up to 33 products below 16, at most 33 roundings of 2^-24 on partial sums below 64, then one rounding to bf16
    torch.testing.assert_close(dense.grad.double(), d64.grad.double(), rtol=2.0 ** -8, atol=33 * 2.0 ** -18)
    torch.testing.assert_close(sparse.grad.double(), s64.grad.double(), rtol=2.0 ** -8, atol=33 * 2.0 ** -18)


@pytest.mark.parametrize("N,H,W,Cin,Cout,R", [(4, 56, 56, 64, 64, 3), (3, 28, 28, 128, 128, 3), (5, 14, 14, 256, 256, 3),
                                              (6, 7, 7, 512, 512, 3), (2, 19, 13, 64, 128, 3), (2, 16, 16, 64, 64, 5)])
def test_conv_implicit_gemm(N, H, W, Cin, Cout, R):
    from oneflow_b200.ops import conv as C
    torch.manual_seed(0)
    x = torch.randn(N, H, W, Cin, device="cuda").bfloat16()
    w = (torch.randn(Cout, R, R, Cin, device="cuda") / math.sqrt(R * R * Cin)).bfloat16()
    dy = torch.randn(N, H, W, Cout, device="cuda").bfloat16()
    x32 = x.float().requires_grad_()
    w32 = w.float().requires_grad_()
    ref = C._ref_conv(x32, w32)
    ref.backward(dy.float())
    y = C.conv_fprop(x, w)
    torch.testing.assert_close(y.float(), ref.detach(), atol=3e-2, rtol=2e-2)
    dx = C.conv_dgrad(dy, w)
    torch.testing.assert_close(dx.float(), x32.grad, atol=3e-2, rtol=2e-2)
    dw = C.conv_wgrad(x, dy, (R, R))
    scale = w32.grad.abs().max().item()
    assert (dw - w32.grad).abs().max().item() <= 1e-2 * scale + 1e-3
    dw2 = C.conv_wgrad(x, dy, (R, R), out=dw.clone(), accumulate=True)
    assert (dw2 - 2 * w32.grad).abs().max().item() <= 2e-2 * scale + 2e-3
    torch.cuda.synchronize()
    assert _native.read_status() == (0, 0)


@pytest.mark.parametrize("N,H,W,Cin,Cout,R", [(4, 56, 56, 128, 128, 3), (19, 14, 14, 512, 512, 3), (3, 10, 10, 256, 256, 3),
                                              (2, 19, 13, 64, 128, 3), (2, 9, 16, 128, 64, 5), (1, 1, 1, 64, 64, 3), (70, 56, 56, 128, 64, 3)])
def test_conv_implicit_gemm_stride2(N, H, W, Cin, Cout, R):
    """Every other pixel by the tensor map, the input gradient by the parity of its pixel: even and odd maps, all tilings."""
    from oneflow_b200.ops import conv as C
    torch.manual_seed(0)
    x = torch.randn(N, H, W, Cin, device="cuda").bfloat16()
    w = (torch.randn(Cout, R, R, Cin, device="cuda") / math.sqrt(R * R * Cin)).bfloat16()
    dy = torch.randn(N, (H + 1) // 2, (W + 1) // 2, Cout, device="cuda").bfloat16()
    x64, w64 = x.double().requires_grad_(), w.double().requires_grad_()
    ref = torch.nn.functional.conv2d(x64.permute(0, 3, 1, 2), w64.permute(0, 3, 1, 2), stride=2, padding=(R - 1) // 2).permute(0, 2, 3, 1)
    ref.backward(dy.double())
    # results are rounded to bf16 once (2^-9 of their size); the fp32 chain of at most R R C / 16 = 288 sums of size below 43 loses
    # no more than 288 * 43 * 2^-23
    y = C.conv_fprop(x, w, 2)
    torch.testing.assert_close(y.double(), ref.detach(), atol=1.5e-3, rtol=2.0 ** -8)
    dx = C.conv_dgrad(dy, w, stride=2, in_hw=(H, W))
    torch.testing.assert_close(dx.double(), x64.grad, atol=1.5e-3, rtol=2.0 ** -8)
    # fp32 results: a chain of N OH OW / 16 sums at most
    dw = C.conv_wgrad(x, dy, (R, R), stride=2)
    size = w64.grad.abs().max().item()
    tol = max(1e-5, dy[..., 0].numel() / 16 * 2.0 ** -23) * max(size, 1.0)
    assert (dw - w64.grad).abs().max().item() <= tol
    dw2 = C.conv_wgrad(x, dy, (R, R), out=dw.clone(), accumulate=True, stride=2)
    assert (dw2 - 2 * w64.grad).abs().max().item() <= 2 * tol
    torch.cuda.synchronize()
    assert _native.read_status() == (0, 0)


@pytest.mark.parametrize("N,H,W,Cin,Cout,R,stride", [(3, 30, 28, 64, 192, 3, 1), (3, 31, 29, 192, 64, 3, 2), (8, 96, 100, 64, 64, 3, 1),
                                                     (10, 90, 100, 64, 64, 3, 2), (2, 9, 7, 64, 64, 3, 2), (1, 8, 8, 320, 320, 3, 1),
                                                     (2, 12, 20, 192, 64, 5, 1), (1, 3, 5, 64, 128, 7, 1)])
def test_conv_channel_boxes(N, H, W, Cin, Cout, R, stride):
    """Tiles of 64 channels, alone and as the last part of wider ones; a few tiles and more than four per SM; taps in every order."""
    from oneflow_b200.ops import conv as C
    torch.manual_seed(42)
    x = torch.randn(N, H, W, Cin, device=DEV).to(BF)
    w = (torch.randn(Cout, R, R, Cin, device=DEV) / math.sqrt(R * R * Cin)).to(BF)
    x64, w64 = x.double().requires_grad_(), w.double().requires_grad_()
    ref = torch.nn.functional.conv2d(x64.permute(0, 3, 1, 2), w64.permute(0, 3, 1, 2), stride=stride, padding=R // 2).permute(0, 2, 3, 1)
    dy = torch.randn(ref.shape, device=DEV).to(BF)
    ref.backward(dy.double())
    # fp32 sums of n terms: at most n / 16 (16 terms an instruction) roundings of 2^-23 on partial sums below 8 (32 for the gradient of x,
    # whose terms are not normalised, 8 sqrt(n) for that of w); results in bf16 another 2^-9 of their size
    n = R * R * max(Cin, Cout)
    torch.testing.assert_close(C.conv_fprop(x, w, stride).double(), ref.detach(), rtol=2.0 ** -8, atol=n / 16 * 2.0 ** -20 + 1e-6)
    torch.testing.assert_close(C.conv_dgrad(dy, w, None, stride, (H, W)).double(), x64.grad, rtol=2.0 ** -8, atol=n / 16 * 2.0 ** -18 + 1e-6)
    px = N * ref.shape[1] * ref.shape[2]
    torch.testing.assert_close(C.conv_wgrad(x, dy, (R, R), stride=stride).double(), w64.grad, rtol=1e-5, atol=px / 16 * 2.0 ** -20 * px ** 0.5)
    torch.cuda.synchronize()
    assert _native.read_status() == (0, 0)


def test_conv_stride_arguments():
    from oneflow_b200.ops import conv as C
    x, w = torch.zeros(1, 6, 6, 64, device="cuda", dtype=BF), torch.zeros(64, 3, 3, 64, device="cuda", dtype=BF)
    dy = torch.zeros(1, 3, 3, 64, device="cuda", dtype=BF)
    for call in (lambda: C.conv_fprop(x, w, 3), lambda: C.conv_fprop(x, w[:, :1, :1].contiguous(), 2), lambda: C.conv_dgrad(dy, w, stride=2),
                 lambda: C.conv_dgrad(dy, w, stride=2, in_hw=(7, 7)), lambda: C.conv_wgrad(x, dy, (3, 3))):
        with pytest.raises(ValueError):
            call()


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (1, 1032, 72), (15, 128, 64), (16, 136, 1000), (17, 4096, 4096), (33, 264, 136), (64, 50304, 256),
                                   (64, 120, 16384), (40, 33024, 64), (65, 256, 512)])
@pytest.mark.parametrize("layout", ["nk", "kn"])
def test_gemm_few_rows(M, N, K, layout):
    """Edges of the row classes (16, 32, 64), ragged columns, one K block and K ranges shared by up to eight CTAs; every epilogue."""
    from oneflow_b200.ops import gemm as G
    torch.manual_seed(40)
    x = torch.randn(M, K, device=DEV, dtype=BF)
    w = torch.randn(N, K, device=DEV, dtype=BF) * K ** -0.5
    wl = w if layout == "nk" else w.t().contiguous()
    b, r, h = torch.randn(N, device=DEV, dtype=BF), torch.randn(M, N, device=DEV, dtype=BF), torch.randn(M, N, device=DEV, dtype=BF)
    p = x.double() @ w.double().t()
    # fp32 sums of K products of size K^-1/2: at most K / 16 roundings of 2^-23 on partial sums below 8; bf16 results 2^-9 of their size
    atol = K / 16 * 2.0 ** -20 + 1e-6
    torch.testing.assert_close(G.gemm(x, wl, b_layout=layout, out_dtype=torch.float32).double(), p, rtol=1e-6, atol=atol)
    y, aux = G.gemm(x, wl, b_layout=layout, bias=b, act="gelu", want_aux=True, residual=r)
    pre = p + b.double()
    torch.testing.assert_close(aux.double(), pre, rtol=2.0 ** -8, atol=atol)
    # the activation's own approximation is good to 2e-6 (tests of the element-wise kernels)
    torch.testing.assert_close(y.double(), torch.nn.functional.gelu(pre) + r.double(), rtol=2.0 ** -8, atol=atol + 1e-5)
    d = G.gemm(x, wl, b_layout=layout, aux_in=h, act="relu")
    torch.testing.assert_close(d.double(), p * (h > 0), rtol=2.0 ** -8, atol=atol)
    acc = torch.randn(M, N, device=DEV)
    out = G.gemm(x, wl, b_layout=layout, out=acc.clone(), accumulate=True)
    torch.testing.assert_close(out.double(), acc.double() + p, rtol=1e-6, atol=atol)
    acc = r.clone()
    G.gemm(x, wl, b_layout=layout, out=acc, accumulate=True)
    torch.testing.assert_close(acc.double(), p + r.double(), rtol=2.0 ** -7, atol=atol + 2.0 ** -8 * float(p.abs().max()))
    # a slice of a wider matrix: leading dimensions that are not the row length
    wide = torch.zeros(M, N + 24, device=DEV, dtype=BF)
    G.gemm(x, wl, b_layout=layout, out=wide[:, 8:N + 8])
    torch.testing.assert_close(wide[:, 8:N + 8].double(), p, rtol=2.0 ** -8, atol=atol)
    assert not wide[:, :8].any() and not wide[:, N + 8:].any()
    torch.cuda.synchronize()
    assert _native.read_status() == (0, 0)


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (64, 136, 72), (129, 72, 64), (300, 264, 256), (257, 1032, 512), (4096, 512, 640), (2000, 64, 1024)])
@pytest.mark.parametrize("layout", ["nk", "kn"])
@pytest.mark.parametrize("bias", [False, True])
def test_gemm_masked_residual(M, N, K, layout, bias):
    """One and two SMs a tile, up to 64 rows, rows of the mask that are and are not whole words; what the mask hides may be NaN."""
    from oneflow_b200.ops import gemm as G
    torch.manual_seed(41)
    x = torch.randn(M, K, device=DEV, dtype=BF)
    w = torch.randn(N, K, device=DEV, dtype=BF) * K ** -0.5
    r = torch.randn(M, N, device=DEV, dtype=BF)
    b = torch.randn(N, device=DEV, dtype=BF) if bias else None
    mask = torch.randint(0, 256, (M, N // 8), device=DEV, dtype=torch.uint8)
    keep = ((mask.view(M, N // 8, 1) >> torch.arange(8, device=DEV, dtype=torch.uint8)) & 1).view(M, N) != 0
    r = torch.where(keep, r, float("nan"))
    y = G.gemm(x, w if layout == "nk" else w.t().contiguous(), b_layout=layout, bias=b, residual=r, residual_mask=mask)
    ref = x.double() @ w.double().t() + torch.where(keep, r, 0.).double()
    # fp32 sums of K products of size K^-1/2: at most K / 16 roundings of 2^-23 on partial sums below 8; bf16 results 2^-9 of their size
    torch.testing.assert_close(y.double(), ref if b is None else ref + b.double(), rtol=2.0 ** -8, atol=K / 16 * 2.0 ** -20 + 1e-6)
    with pytest.raises(ValueError):
        G.gemm(x, w, residual=r, residual_mask=mask.view(-1)[1:])
    with pytest.raises(ValueError):
        G.gemm(x, w, residual_mask=mask)


@pytest.mark.parametrize("N", [8, 56, 64, 72, 128, 184, 192, 200])
@pytest.mark.parametrize("bn", [0, 128, 256])
def test_gemm_narrow_tile(N, bn):
    """All of N in one tile, from a part of one 64-row box of weights to the whole tile; all layouts, a last K block that is not full."""
    from oneflow_b200.ops import gemm as G
    torch.manual_seed(43)
    M, K = 328, 200
    x, w = torch.randn(M, K, device=DEV, dtype=BF), torch.randn(N, K, device=DEV, dtype=BF) * K ** -0.5
    ref = x.double() @ w.double().t()
    for al in ("mk", "km"):
        for bl in ("nk", "kn"):
            y = G.gemm(x if al == "mk" else x.t().contiguous(), w if bl == "nk" else w.t().contiguous(), a_layout=al, b_layout=bl, bn=bn,
                       out_dtype=torch.float32)
            # fp32 sums of K products of size K^-1/2: at most K / 16 roundings of 2^-23 on partial sums below 8
            torch.testing.assert_close(y.double(), ref, rtol=1e-6, atol=K / 16 * 2.0 ** -20)
    torch.cuda.synchronize()
    assert _native.read_status() == (0, 0)


def test_flow_conv2d_channels_last_uses_igemm():
    import oneflow_b200 as flow
    torch.manual_seed(0)
    conv = flow.nn.Conv2d(64, 128, 3, padding=1, bias=True).cuda().bfloat16().to(memory_format=torch.channels_last)
    x = torch.randn(4, 64, 20, 20, device="cuda").bfloat16().to(memory_format=torch.channels_last).requires_grad_()
    n0 = K.launch_count
    y = conv(x)
    assert K.launch_count == n0 + 1, "the eligible convolution must run on the implicit-GEMM kernel"
    assert y.shape == (4, 128, 20, 20) and y.is_contiguous(memory_format=torch.channels_last)
    ref = torch.nn.functional.conv2d(x.detach().float(), conv.weight.detach().float(), conv.bias.detach().float(), padding=1)
    torch.testing.assert_close(y.float(), ref, atol=5e-2, rtol=3e-2)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    wr = conv.weight.detach().float().requires_grad_()
    torch.nn.functional.conv2d(xr, wr, None, padding=1).backward(g.float())
    torch.testing.assert_close(x.grad.float(), xr.grad, atol=8e-2, rtol=3e-2)
    assert (conv.weight.grad.float() - wr.grad).abs().max() <= 2e-2 * wr.grad.abs().max() + 1e-2
    # a strided convolution takes the library path and still works
    conv2 = flow.nn.Conv2d(64, 64, 3, stride=2, padding=1).cuda().bfloat16()
    assert conv2(x.detach()).shape == (4, 64, 10, 10)


def test_profiler_reports_native_kernels_with_bandwidth():
    """Inside flow.profiler.profile the native kernel calls appear by name with device time, input shapes and a bandwidth
    (bytes of the operands / device time); ATen ops appear beside them."""
    import oneflow_b200 as flow
    x = torch.randn(4096, 4096, device=DEV, dtype=BF)
    w = torch.randn(4096, 4096, device=DEV, dtype=BF)
    g, b = torch.ones(4096, device=DEV, dtype=BF), torch.zeros(4096, device=DEV, dtype=BF)
    G.gemm(x, w)
    with flow.profiler.profile(record_shapes=True, record_attrs=True, record_bandwidth_for_cuda=True) as prof:
        with flow.profiler.record_function("step"):
            for _ in range(3):
                y = G.gemm(x, w)
            K.layer_norm_fwd(y, g, b)
            torch.relu(y)
    avg = prof.key_averages(group_by_input_shape=True, group_by_attributes=True)
    by = {e.name: e for e in avg}
    assert by["gemm_bf16"].count == 3 and by["layer_norm_fwd"].count == 1 and by["aten::relu"].count == 1 and by["step"].count == 1
    ge = by["gemm_bf16"]
    assert ge.cuda_time > 20 and ge.flops == 3 * 2.0 * 4096 ** 3         # a 4096^3 GEMM takes > 20 us on any B200
    assert ge.input_shapes == "[(4096,4096), (4096,4096), (4096,4096)]" and "act=0" in ge.attributes
    ln = by["layer_norm_fwd"]
    assert ln.bandwidth is not None and 50 < ln.bandwidth < 20000       # GB/s: two 32 MB passes in some tens of microseconds
    assert by["step"].cuda_time_total >= ge.cuda_time_total
    t = avg.table()
    assert "Bandwidth" in t.splitlines()[0] and "GB/s" in t and "gemm_bf16" in t
    # the library is handed out unwrapped again
    assert type(_native.kernels()).__name__ == "CDLL"


def test_remat_on_cuda_matches_unbounded_run():
    """flow.remat.scope on CUDA tensors: eviction really lowers torch's allocated bytes, backward (on autograd's device thread)
    recomputes what it needs, gradients equal the unbounded run."""
    import oneflow_b200 as flow
    torch.manual_seed(3)
    layers = torch.nn.ModuleList([torch.nn.Linear(1024, 1024) for _ in range(8)]).to(DEV)
    x = torch.randn(2048, 1024, device=DEV)

    def run():
        h = x
        for l in layers:
            h = torch.tanh(l(h)) + h
        return h.pow(2).mean()
    ref = run()
    ref.backward()
    g_ref = [p.grad.clone() for p in layers.parameters()]
    for p in layers.parameters():
        p.grad = None
    act = 2048 * 1024 * 4
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    with flow.remat.scope(budget=10 * act) as r:
        loss = run()
        assert r.stats["forced_eviction_num"] > 0
        assert torch.cuda.memory_allocated() - base <= 11 * act      # 24 activations were produced, at most the budget is held
        loss.backward()
        assert r.stats["recomputation_num"] > 0
    torch.cuda.synchronize()
    assert torch.allclose(loss, ref)
    for a, p in zip(g_ref, layers.parameters()):
        assert torch.allclose(a, p.grad, atol=1e-6, rtol=1e-5)


def test_mlp_unit_folds_the_activation_gradient_into_the_gemm():
    """fused_ops.mlp == linear(gelu(linear(x))) + residual with the same gradients as the fp32 statement; its backward issues one
    kernel less than the two separate linears (the GELU gradient rides in the second layer's data-gradient GEMM)."""
    from oneflow_b200.framework import fused_ops as FO
    torch.manual_seed(31)
    T, H, F_ = 512, 256, 1024
    x = (torch.randn(T, H, device=DEV) * 0.5).to(BF).requires_grad_()
    w1 = (torch.randn(F_, H, device=DEV) * 0.05).to(BF).requires_grad_()
    b1 = (torch.randn(F_, device=DEV) * 0.1).to(BF).requires_grad_()
    w2 = (torch.randn(H, F_, device=DEV) * 0.05).to(BF).requires_grad_()
    b2 = (torch.randn(H, device=DEV) * 0.1).to(BF).requires_grad_()
    res = (torch.randn(T, H, device=DEV) * 0.5).to(BF).requires_grad_()
    gy = torch.randn(T, H, device=DEV).to(BF)

    def run(fused):
        for t in (x, w1, b1, w2, b2, res):
            t.grad = None
        n0 = K.launch_count
        if fused:
            y = FO.mlp(x, w1, b1, w2, b2, act="gelu", residual=res)
        else:
            y = FO.linear(FO.linear(x, w1, b1, act="gelu"), w2, b2, residual=res)
        y.backward(gy)
        return y.detach(), [t.grad.clone() for t in (x, w1, b1, w2, b2, res)], K.launch_count - n0
    y_f, g_f, n_f = run(True)
    y_s, g_s, n_s = run(False)
    assert n_f == n_s - 1, (n_f, n_s)
    xf, w1f, b1f, w2f, b2f, rf = (t.detach().float().requires_grad_() for t in (x, w1, b1, w2, b2, res))
    ref = torch.nn.functional.linear(torch.nn.functional.gelu(torch.nn.functional.linear(xf, w1f, b1f)), w2f, b2f) + rf
    ref.backward(gy.float())
    close(y_f, ref.detach())

    def rms(t):
        return float(t.float().pow(2).mean().sqrt())
    # gradients pass through two bf16 roundings of [T, ffn]-sized intermediates (one in the folded form): elements that nearly
    # cancel carry an absolute error of a few percent of the tensor's RMS
    for got, want in zip(g_f, (xf, w1f, b1f, w2f, b2f, rf)):
        close(got, want.grad, 2e-2, 3e-2 * rms(want.grad))
    for a, b in zip(g_f, g_s):
        close(a, b.float(), 2e-2, 3e-2 * rms(b))


def test_fused_mlp_chain_on_cuda():
    """flow._C.fused_mlp on bf16 CUDA tensors: three linear + ReLU layers, each ReLU gradient folded into the next layer's
    data-gradient GEMM (no separate activation-gradient kernel runs), values and gradients against the fp32 statement."""
    import oneflow_b200 as flow
    torch.manual_seed(32)
    T = 384
    dims = [256, 512, 384, 128]
    x = (torch.randn(T, dims[0], device=DEV) * 0.5).to(BF).requires_grad_()
    ws = [(torch.randn(dims[i + 1], dims[i], device=DEV) * 0.06).to(BF).requires_grad_() for i in range(3)]
    bs = [(torch.randn(dims[i + 1], device=DEV) * 0.1).to(BF).requires_grad_() for i in range(3)]
    gy = torch.randn(T, dims[-1], device=DEV).to(BF)
    n0 = K.launch_count
    y = flow._C.fused_mlp(x, ws, bs, skip_final_activation=True)
    y.backward(gy)
    # 3 forward GEMMs; backward: 3 data-gradient + 3 weight-gradient GEMMs + 3 bias column sums, no activation-gradient kernel
    assert K.launch_count - n0 == 12, K.launch_count - n0
    # fp32 statement that rounds the hidden activations to bf16 where the kernels store them (straight-through for the
    # gradient): ReLU is discontinuous, so a statement with unrounded hidden values switches a few units per token the other
    # way (|pre-activation| below the rounding noise of its inputs) and its gradients then differ by several percent of
    # their RMS on whole rows: measured 10 - 30 % of the elements beyond 3 % of RMS, against none for GELU
    ref_in = [t.detach().float().requires_grad_() for t in [x] + ws + bs]
    h = ref_in[0]
    for i in range(3):
        h = torch.nn.functional.linear(h, ref_in[1 + i], ref_in[4 + i])
        if i < 2:
            h = torch.relu(h)
            h = h + (h.bfloat16().float() - h).detach()
    h.backward(gy.float())
    close(y, h.detach())

    def rms(t):
        return float(t.float().pow(2).mean().sqrt())
    # even so a hidden value can round to the neighbouring bf16 number in the kernel (other summation order), which now and
    # then switches a unit of the next layer: up to 1 % of the elements may sit outside the bound, none far outside
    for got, want in zip([x] + ws + bs, ref_in):
        g, w_ = got.grad.float(), want.grad
        r = rms(w_)
        bad = (g - w_).abs() > 3e-2 * r + 2e-2 * w_.abs()
        assert bad.float().mean().item() < 0.01, bad.float().mean().item()
        assert (g - w_).abs().max().item() < 0.5 * r
    # and the folded form equals the layer-by-layer form bit for bit
    got = [t.grad.clone() for t in [x] + ws + bs]
    for t in [x] + ws + bs:
        t.grad = None
    from oneflow_b200.framework import fused_ops as FO
    h2 = x
    for i in range(3):
        h2 = FO.linear(h2, ws[i], bs[i], act=("relu" if i < 2 else 0))
    h2.backward(gy)
    for a, t in zip(got, [x] + ws + bs):
        assert torch.equal(a, t.grad)
