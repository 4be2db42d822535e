"""Kernels of the learned operator at the sizes where they can go wrong:
permutations through shared-memory tiles (remainders in both tiled axes,
padding, cropping, accumulation), products with a split K, a strided or
unaligned output and the GELU epilogue, the fused layer sum, column sums and
the loss over many blocks.  References are torch on the same inputs in FP64;
permutations are exact, FP32 sums of n terms are held to 4 sqrt(n) roundings
of the sum of magnitudes, BF16 outputs to their rounding."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS32, EPS16 = 2.0 ** -24, 2.0 ** -8


def _t(shape, cuda, seed=0, dtype=None):
    import torch
    g = torch.Generator(device=cuda).manual_seed(seed)
    x = torch.randn(shape, device=cuda, generator=g)
    return x.to(dtype) if dtype else x


@pytest.mark.parametrize("perm", [(0, 1, 3, 2), (0, 3, 1, 2), (0, 2, 3, 1), (2, 3, 0, 1), (0, 1, 2, 3), (3, 0, 1, 2)])
@pytest.mark.parametrize("dims", [(2, 3, 130, 65), (1, 2, 1, 33), (3, 1, 257, 16), (5, 4, 7, 3), (2, 129, 16, 32), (33, 5, 15, 32)])
def test_permute_pads_crops_and_adds(cuda, perm, dims):
    import torch
    from pot3d_b200.fno import permute
    for src, dst, add in (("bf16", "bf16", False), ("f32", "bf16", False), ("bf16", "f32", True), ("f32", "f32", False)):
        dt = {"bf16": torch.bfloat16, "f32": torch.float32}
        x = _t(dims, cuda, 1, dt[src])
        out_dims = [dims[p] for p in perm]
        out_dims[3] += 5      # padded
        out_dims[2] = max(1, out_dims[2] - 1)  # cropped
        out = _t(out_dims, cuda, 2, dt[dst]) if add else torch.full(out_dims, 7.0, device=cuda, dtype=dt[dst])
        ref = x.permute(*perm)[:, :, :out_dims[2]].float()
        ref = torch.nn.functional.pad(ref, (0, 5))
        ref = (out.float() + ref if add else ref).to(dt[dst])
        permute(x, dims, out, out_dims, perm, add=add)
        assert torch.equal(out, ref), (src, dst, add)


def test_permute_of_short_axes_costs_no_more_than_its_elements(cuda):
    """The same elements with axes of 1 x 1 and of 64 x 64 to turn; a tile an
    element took 300 times as long as an element at a time."""
    import torch
    from pot3d_b200.fno import permute
    n, ms = 1 << 23, []
    x, out = _t((n,), cuda, 19), torch.empty(n, device=cuda)
    for k in (1, 64):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        for timed in (False, True):
            e[0].record()
            permute(x, (1, n // (k * k), k, k), out, (1, n // (k * k), k, k), (0, 1, 3, 2))
            e[1].record()
            torch.cuda.synchronize()
        assert torch.equal(out.view(-1, k, k), x.view(-1, k, k).transpose(1, 2))
        ms.append(e[0].elapsed_time(e[1]))
    assert ms[0] < 30 * ms[1], ms


@pytest.mark.parametrize("b,m,n,k", [(1, 32, 64, 64 * 67), (1, 128, 128, 64 * 300), (1, 130, 16, 64 * 64),
                                     (2, 32, 32, 64 * 65), (1, 1000, 48, 64), (33, 16, 16, 64 * 67), (30, 100, 16, 64 * 80)])
def test_gemm_split_k_strides_and_act(cuda, b, m, n, k):
    import torch
    from pot3d_b200.tc import check_errors, k_splits, tc_gemm
    A, B, bias = _t((b, m, k), cuda, 3, torch.bfloat16), _t((b, n, k), cuda, 4, torch.bfloat16), _t((n,), cuda, 5)
    ref = A.double() @ B.double().transpose(1, 2) + bias.double()
    mag = A.double().abs() @ B.double().abs().transpose(1, 2) + bias.double().abs()
    tol = 4 * EPS32 * np.sqrt(k) * mag
    splits = k_splits(b, m, n, k)
    assert (splits > 1) == (k >= 64 * 64 and b * -(-m // 128) * 2 <= k // 64)
    assert bool(((tc_gemm(A, B, bias=bias).double() - ref).abs() <= tol).all())
    acc = _t((b, m, n), cuda, 6)
    got = tc_gemm(A, B, bias=bias, out=acc.clone(), accumulate=True)
    assert bool(((got.double() - ref - acc.double()).abs() <= tol + EPS32 * (ref + acc.double()).abs()).all())
    g = torch.nn.functional.gelu(ref, approximate="tanh")
    assert bool(((tc_gemm(A, B, bias=bias, act="gelu").double() - g).abs() <= 2 * tol + 16 * EPS32 * g.abs()).all())
    wide = torch.full((b, m, n + 3), 7.0, device=cuda)  # a row stride that rules out vector stores
    tc_gemm(A, B, bias=bias, out=wide, ldd=n + 3)
    assert bool(((wide[..., :n].double() - ref).abs() <= tol).all()) and bool((wide[..., n:] == 7.0).all())
    if splits == 1:  # the BF16 output is the FP32 one rounded
        assert torch.equal(tc_gemm(A, B, bias=bias, out_dtype=torch.bfloat16), tc_gemm(A, B, bias=bias).bfloat16())
    check_errors()


def test_a_product_whose_wait_ran_out_is_reported(cuda):
    import torch
    from pot3d_b200.tc import _err_flag, check_errors, tc_gemm
    out = tc_gemm(_t((16, 64), cuda, 17, torch.bfloat16), _t((16, 64), cuda, 18, torch.bfloat16))
    check_errors()
    flag = _err_flag(out.device)
    flag.fill_(1)  # as the kernel does
    try:
        with pytest.raises(RuntimeError):
            check_errors()
    finally:
        flag.zero_()
    check_errors()


@pytest.mark.parametrize("b,w,nph,nth", [(1, 32, 3, 33), (2, 17, 5, 31), (1, 64, 2, 96)])
def test_spec_act(cuda, b, w, nph, nth):
    import torch
    from pot3d_b200.fno import spec_act
    pth = (nth + 63) // 64 * 64
    pre = _t((b * nph * nth, w), cuda, 7)
    spec = _t((b, w, nph, pth), cuda, 8, torch.bfloat16)
    s = pre + spec[..., :nth].permute(0, 2, 3, 1).reshape(-1, w).float()
    for gelu in (False, True):
        p = pre.clone()
        v = spec_act(p, spec, b, w, nph, nth, pth, gelu, keep=gelu)
        assert torch.equal(p, s if gelu else pre)
        ref = torch.nn.functional.gelu(s.double(), approximate="tanh") if gelu else s.double()
        assert bool(((v[:, :w].double() - ref).abs() <= (EPS16 + 32 * EPS32) * ref.abs() + 1e-7).all())
        assert not v[:, w:].any()


@pytest.mark.parametrize("b,npos,R,ldp", [(1, 1, 1, 64), (3, 2049, 125, 128), (2, 70000, 61, 64),
                                           (70000, 1, 3, 4), (65537, 9, 1, 1), (3, 4096, 1, 1),
                                           (2, 2000, 5, 9), (64, 1030, 17, 20), (1, 1 << 17, 1, 2)])
def test_relmse_and_colsum(cuda, b, npos, R, ldp):
    import torch
    from pot3d_b200 import _lib
    from pot3d_b200.fno import _L, colsum, new
    pred, tgt = _t((b, npos, ldp), cuda, 9), _t((b, npos, R), cuda, 10, torch.bfloat16)
    d = pred[..., :R].double() - tgt.double()
    den = tgt.double().square().sum((1, 2))
    loss = d.square().sum((1, 2)) / den
    gref = torch.nn.functional.pad(2.0 * 0.25 * d / den.view(-1, 1, 1), (0, ldp - R))
    tol = 8 * EPS32 * np.sqrt(npos * R)
    L = _L()
    for scratch in (True, False):
        grad, got = torch.full_like(pred, 7.0), torch.zeros(b, device=cuda)
        args = [C.c_void_p(pred.data_ptr()), ldp, C.c_void_p(tgt.data_ptr()), 1, b, C.c_longlong(npos), R,
                C.c_float(0.25), C.c_void_p(grad.data_ptr()), C.c_void_p(got.data_ptr())]
        if scratch:
            ws = new((L.pot3d_fno_relmse_scratch(b),), "f32")
            _lib.check(L.pot3d_fno_relmse_ws(*args, C.c_void_p(ws.data_ptr()), None))
        else:
            _lib.check(L.pot3d_fno_relmse(*args, None))
        torch.cuda.synchronize()
        assert bool(((got.double() - loss).abs() <= tol * loss).all())
        assert bool(((grad.double() - gref).abs() <= (tol + 8 * EPS32) * gref.abs() + 4 * EPS32 * 0.5 / den.view(-1, 1, 1) *
                     (pred.abs().double().amax() + tgt.abs().double().amax())).all())
    flat = pred.reshape(-1, ldp)
    s = colsum(flat, R, ldp, new((R,), "f32"))
    ref = flat[:, :R].double().sum(0)
    assert bool(((s.double() - ref).abs() <= 4 * EPS32 * np.sqrt(b * npos) * flat[:, :R].double().abs().sum(0) + 1e-30).all())


@pytest.mark.parametrize("m,c,ld", [(1, 1, 1), (255, 33, 40), (257, 32, 32), (16384 + 31, 125, 128), (5 * 16384 + 300, 7, 64),
                                    (40 * 16384 + 255, 1, 3), (2 * 16384, 8, 8), (300, 2, 2), (20 * 16384 + 1, 9, 9)])
def test_colsum_order(cuda, m, c, ld):
    """Bit for bit the stated order: 64 blocks of 256 chains of rows, a binary
    tree over a block's chains, then the blocks one after the other."""
    import torch
    from pot3d_b200.fno import colsum, new
    x = _t((m, ld), cuda, 16)
    steps = -(-m // (64 * 256))
    rows = torch.zeros((steps * 64 * 256, c), device=cuda)
    rows[:m] = x[:, :c]
    rows = rows.view(steps, 64, 256, c)
    s = torch.zeros((64, 256, c), device=cuda)
    for k in range(steps):
        s = s + rows[k]
    while s.shape[1] > 1:
        h = s.shape[1] // 2
        s = s[:, :h] + s[:, h:]
    ref = torch.zeros(c, device=cuda)
    for b in range(64):
        ref = ref + s[b, 0]
    assert torch.equal(colsum(x, c, ld, new((c,), "f32")), ref)


@pytest.mark.parametrize("rows,cols,out_cols", [(1, 4, 8), (1001, 32, 64), (37, 128, 128), (5, 64, 32), (9, 12, 40)])
def test_permute_rows_eight_columns_a_thread(cuda, rows, cols, out_cols):
    import torch
    from pot3d_b200.fno import permute
    x = _t((2, 3, rows, cols), cuda, 11)
    ref = torch.nn.functional.pad(x[..., :out_cols], (0, max(0, out_cols - cols))).bfloat16()
    shifted = torch.empty(2 * 3 * rows * cols + 1, device=cuda)[1:].view(x.shape).copy_(x)  # not 16-byte aligned
    for src in (x, shifted):
        out = torch.full((2, 3, rows, out_cols), 7.0, device=cuda, dtype=torch.bfloat16)
        assert torch.equal(permute(src, x.shape, out, out.shape, (0, 1, 2, 3)), ref)
    out = torch.full((3, 2, rows, out_cols), 7.0, device=cuda, dtype=torch.bfloat16)
    assert torch.equal(permute(x, x.shape, out, out.shape, (1, 0, 2, 3)), ref.transpose(0, 1))


@pytest.mark.parametrize("rows,c,ldo", [(1, 1, 1), (3001, 1, 3), (2047, 40, 64), (2048, 31, 31), (2049, 40, 64), (5, 1000, 1001)])
def test_gelu_and_guess_of_any_width(cuda, rows, c, ldo):
    import torch
    from pot3d_b200 import _lib
    from pot3d_b200.fno import _L, act
    pre, grad = _t((rows, c), cuda, 20), _t((rows, c), cuda, 21, torch.bfloat16)
    x = pre.double().requires_grad_(True)
    ref = torch.nn.functional.gelu(x, approximate="tanh")
    (dref,) = torch.autograd.grad(ref, x, grad.double())
    for mode, want in (("gelu", ref.detach()), ("dgelu", dref)):
        out = torch.full((rows, ldo), 7.0, device=cuda)
        act(pre, c, c, out, ldo, mode, grad=grad, ldg=c)
        # tanh of u to 2 ulp of 1, u's own rounding times u, and a few products
        assert bool(((out[:, :c].double() - want).abs() <= 32 * EPS32 * (1 + pre.abs().double() ** 3) *
                     (1 + grad.abs().double())).all()), mode
        assert not out[:, c:].any()
    for b in (1, 2):
        sigma, x0 = _t((b,), cuda, 22, torch.float64), torch.empty((b, rows, c), device=cuda, dtype=torch.float64)
        y = _t((b, rows, ldo), cuda, 23)
        _lib.check(_L().pot3d_fno_guess(C.c_void_p(y.data_ptr()), b, rows, ldo, c, C.c_void_p(sigma.data_ptr()),
                                        C.c_void_p(x0.data_ptr()), None))
        torch.cuda.synchronize()
        assert torch.equal(x0, y[..., :c].double() * sigma.view(-1, 1, 1))


@pytest.mark.parametrize("b,npos,rs,r", [(1, 1, 2, 1), (2, 1201, 125, 253), (1, 2500, 768, 800), (1, 9, 769, 31),
                                         (2, 1500, 125, 31), (1, 2100, 125, 62), (3, 800, 70, 33), (1, 2500, 70, 70)])
def test_guess_resampled(cuda, b, npos, rs, r):
    import torch
    from pot3d_b200 import _lib
    from pot3d_b200.fno import _L
    rp = (rs + 63) // 64 * 64
    out = _t((b, npos, rp), cuda, 12)
    hi = rp - 1 if (rs, r) == (70, 70) else rs - 1  # once every index inside a row, padding included
    idx = torch.randint(0, hi, (r,), device=cuda, dtype=torch.int32, generator=torch.Generator(cuda).manual_seed(13))
    w, sigma = 1.2 * _t((r,), cuda, 14, torch.float64), _t((b,), cuda, 15, torch.float64)
    x = torch.empty((b, npos, r), device=cuda, dtype=torch.float64)
    _lib.check(_L().pot3d_fno_guess_resampled(*[C.c_void_p(out.data_ptr()), b, npos, rp, rs], C.c_void_p(idx.data_ptr()),
                                              C.c_void_p(w.data_ptr()), r, C.c_void_p(sigma.data_ptr()),
                                              C.c_void_p(x.data_ptr()), None))
    torch.cuda.synchronize()
    lo, hi = out.double()[..., idx.long()], out.double()[..., idx.long() + 1]
    # the same operations but for the fma's missing rounding: two roundings of the terms' magnitudes and the product's
    tol = 4 * 2.0 ** -53 * (lo.abs() + (w * (hi - lo)).abs()) * sigma.abs().view(-1, 1, 1)
    assert bool(((x - (lo + w * (hi - lo)) * sigma.view(-1, 1, 1)).abs() <= tol).all())
