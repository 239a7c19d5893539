"""Kernels whose work split depends on sizes or alignment, at the edges of those splits, against the CPU oracle."""
import ctypes as C

import numpy as np
import pytest

import om_binding as omb
from backends import scaled_diff
from om_binding import f32, i32, i64

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K(oracle_built):
    return oracle_built


def normal(seed, *shape, scale=1.0):
    return (np.random.default_rng(seed).standard_normal(shape) * scale).astype(np.float32)


def table(pointers):
    return (C.c_void_p * len(pointers))(*pointers)


class SgdHyper(C.Structure):
    _fields_ = [(n, C.c_float) for n in ("lr", "weight_decay", "momentum", "dampening", "grad_scale")] + [("nesterov", C.c_int32), ("has_momentum", C.c_int32)]


@pytest.mark.parametrize("sizes", [[1, 3, 1023, 1024, 1025, 4099], [8 * 148 * 4096 - 5, 4, 9], [8 * 148 * 4096 + 3, 4097, 2]])
@pytest.mark.parametrize("momentum,nesterov,wd", [(0.0, 0, 0.0), (0.9, 1, 0.1)])
def test_sgd_visits_are_bit_exact(ctx, K, sizes, momentum, nesterov, wd):
    """Edges of the visits (1024 or 4096 elements by the launch's total), their ragged ends, and tensors that start off a
    16-byte boundary (every second one): the bits of the reference's update."""
    shift = [i % 2 for i in range(len(sizes))]
    ps, bufs = ([normal(7 * i + j, n) for i, n in enumerate(sizes)] for j in (0, 1))
    P, B = ([ctx.to_device(np.concatenate([np.zeros(s, np.float32), a])) for a, s in zip(arrs, shift)] for arrs in (ps, bufs))
    at = lambda arrs: table([a.ptr.value + 4 * s for a, s in zip(arrs, shift)])  # noqa: E731
    hyper = SgdHyper(0.05, wd, momentum, 0.1, 1.0, nesterov, int(momentum != 0.0))
    for step in range(2):
        gs = [normal(100 + 7 * i + step, n) for i, n in enumerate(sizes)]
        G = [ctx.to_device(np.concatenate([np.zeros(s, np.float32), a])) for a, s in zip(gs, shift)]
        ctx.call("om_optim_sgd_step", ctx.handle, i32(len(sizes)), at(P), at(G), at(B), omb.int_array([int(step == 0)] * len(sizes)),
                 omb.int_array(sizes, C.c_int64), C.byref(hyper), None)
        for p, g, b in zip(ps, gs, bufs):
            K.sgd_step(p, g, b, step == 0, 0.05, wd, momentum, 0.1, bool(nesterov))
    for i, s in enumerate(shift):
        assert np.array_equal(P[i].numpy()[s:], ps[i]), sizes[i]
        if momentum:
            assert np.array_equal(B[i].numpy()[s:], bufs[i]), sizes[i]


@pytest.mark.parametrize("tf32", [0, 1])
@pytest.mark.parametrize("b,h,lq,lk,d,batched", [(2, 3, 128, 128, 32, 1), (3, 2, 97, 61, 32, 1), (2, 2, 100, 128, 64, 0), (2, 2, 129, 130, 32, 1),
                                                 (2, 2, 320, 320, 32, 1), (1, 3, 200, 259, 64, 0), (2, 1, 256, 384, 64, 1)])
def test_attention_masks_of_every_alignment(ctx, K, tf32, b, h, lq, lk, d, batched):
    """The mask is brought in by rows and turned: one tile and several, ragged rows and columns, rows off the 16-byte grid, a
    mask base off it, a mask for all batches and one for each, padded keys with a large negative score and with -inf. Three
    chained TF32 products: 2e-3 scaled, the gate of the attention tests without a mask."""
    ctx.set_flags(omb.OM_TF32 if tf32 else 0)
    try:
        q, k, v, g = (normal(i, b, h, l, d) for i, l in ((1, lq), (2, lk), (3, lk), (4, lq)))
        r = np.random.default_rng(5)
        mask = normal(6, *((b, lq, lk) if batched else (lq, lk)))
        mask[..., lk - lk // 4:] = np.where(r.random(mask[..., lk - lk // 4:].shape) < 0.5, np.float32(-1e9), np.float32(-np.inf))
        scale = 1.0 / np.sqrt(d)
        for shift in (0, 1):
            Q, Kk, V, G = (ctx.to_device(a) for a in (q, k, v, g))
            M = ctx.to_device(np.concatenate([np.zeros(shift, np.float32), mask.reshape(-1)]))
            O, LSE = ctx.empty(q.shape), ctx.empty((b, h, lq))
            DQ, DK, DV = ctx.empty(q.shape), ctx.empty(k.shape), ctx.empty(v.shape)
            at = C.c_void_p(M.ptr.value + 4 * shift)
            mbs = lq * lk if batched else 0
            ctx.call("om_attention_fwd", ctx.handle, Q.ptr, Kk.ptr, V.ptr, at, i64(mbs), i32(b), i32(h), i32(lq), i32(lk), i32(d), f32(scale), O.ptr, LSE.ptr)
            ctx.call("om_attention_bwd", ctx.handle, G.ptr, Q.ptr, Kk.ptr, V.ptr, at, i64(mbs), LSE.ptr, i32(b), i32(h), i32(lq), i32(lk), i32(d), f32(scale),
                     DQ.ptr, DK.ptr, DV.ptr)
            dq, dk, dv = K.attention_bwd(g, q, k, v, mask)
            for got, want in ((O, K.attention_fwd(q, k, v, mask)), (DQ, dq), (DK, dk), (DV, dv)):
                assert scaled_diff(got.numpy(), want) <= (2e-3 if tf32 else 1e-4)
    finally:
        ctx.set_flags(0)


class ConvShape(C.Structure):
    _fields_ = [(n, C.c_int32) for n in ("n", "cin", "h", "w", "cout", "kh", "kw", "stride_h", "stride_w", "pad_top", "pad_left",
                                         "pad_bottom", "pad_right", "dil_h", "dil_w", "groups")]


def to_tf32(a):
    """Round to nearest even at 10 mantissa bits."""
    u = a.view(np.uint32).astype(np.uint64)
    return ((u + 0xFFF + ((u >> 13) & 1)) & ~np.uint64(0x1FFF)).astype(np.uint32).view(np.float32)


def conv_case(n, cin, h, w, cout, kh, kw, sh, sw, pads, dh, dw, seed=0):
    """Geometry, TF32-valued operands and the exact results (float64 PyTorch on the CPU)."""
    import torch
    pt, pl, pb, pr = pads
    s = ConvShape(n, cin, h, w, cout, kh, kw, sh, sw, pt, pl, pb, pr, dh, dw, 1)
    x, wt, b = to_tf32(normal(seed, n, cin, h, w)), to_tf32(normal(seed + 1, cout, cin, kh, kw, scale=0.2)), normal(seed + 2, cout)
    xt, wtt = (torch.from_numpy(a).double().requires_grad_(True) for a in (x, wt))
    y = torch.nn.functional.conv2d(torch.nn.functional.pad(xt, (pl, pr, pt, pb)), wtt, torch.from_numpy(b).double(), (sh, sw), 0, (dh, dw))
    g = to_tf32(normal(seed + 3, *y.shape))
    y.backward(torch.from_numpy(g).double())
    return s, x, wt, b, g, y.detach().numpy(), xt.grad.numpy(), wtt.grad.numpy()


def run_conv(ctx, s, x, wt, b, g):
    X, W, B, G = (ctx.to_device(a) for a in (x, wt, b, g))
    Y, DX, DW = ctx.empty(g.shape), ctx.empty(x.shape), ctx.empty(wt.shape)
    ctx.call("om_conv2d_fwd", ctx.handle, C.byref(s), X.ptr, W.ptr, B.ptr, Y.ptr)
    ctx.call("om_conv2d_dgrad", ctx.handle, C.byref(s), G.ptr, W.ptr, DX.ptr)
    ctx.call("om_conv2d_wgrad", ctx.handle, C.byref(s), G.ptr, X.ptr, DW.ptr, i32(0))
    first = DW.numpy().copy()
    ctx.call("om_conv2d_wgrad", ctx.handle, C.byref(s), G.ptr, X.ptr, DW.ptr, i32(1))
    ctx.sync()
    return Y.numpy(), DX.numpy(), first, DW.numpy()


CONV_EDGES = [
    # n, cin, h, w, cout, kh, kw, sh, sw, (top, left, bottom, right), dh, dw
    (2, 4, 8, 8, 5, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1),            # one ragged tile of everything
    (4, 8, 5, 7, 130, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1),          # planes off the 16-byte grid, a second block of channels
    (20, 8, 32, 32, 200, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1),       # two accumulators, the second ragged
    (20, 8, 32, 32, 384, 1, 1, 1, 1, (0, 0, 0, 0), 1, 1),       # two accumulators, then one
    (4, 12, 9, 11, 20, 3, 3, 2, 2, (1, 1, 1, 1), 1, 1),         # classes of a strided gradient of different sizes
    (4, 16, 8, 6, 12, 1, 1, 2, 2, (0, 0, 0, 0), 1, 1),          # classes that no tap reaches
    (4, 8, 13, 10, 12, 3, 2, 1, 2, (2, 0, 1, 1), 1, 1),         # strides and pads of their own
    (4, 4, 20, 18, 9, 5, 5, 1, 1, (4, 4, 4, 4), 2, 2),          # dilation, 25 taps
    (4, 4, 12, 12, 9, 4, 8, 2, 1, (1, 3, 2, 4), 1, 1),          # 32 taps
    (4, 4, 12, 12, 9, 6, 6, 1, 1, (2, 2, 2, 2), 1, 1),          # 36 taps: the unfolded matrix
    (4, 4, 14, 14, 9, 3, 3, 3, 3, (1, 1, 1, 1), 1, 1),          # nine classes: the unfolded matrix for the input gradient
    (3, 4, 64, 4, 136, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1),         # planes of whole stages: the gradient by TMA
    (64, 160, 4, 4, 144, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1),       # several column tiles, planes of half a stage
]


@pytest.mark.parametrize("case", CONV_EDGES)
def test_conv2d_without_an_unfolded_matrix(ctx, case):
    """TF32-valued operands, so that only the order of the fp32 sums is left: 2e-5 scaled, the gate of the plain products."""
    s, x, wt, b, g, y, dx, dw = conv_case(*case)
    ctx.set_flags(omb.OM_TF32)
    try:
        Y, DX, DW, DW2 = run_conv(ctx, s, x, wt, b, g)
    finally:
        ctx.set_flags(0)
    assert scaled_diff(Y, y) <= 2e-5
    assert scaled_diff(DX, dx) <= 2e-5
    assert scaled_diff(DW, dw) <= 2e-5
    assert scaled_diff(DW2, 2 * dw) <= 2e-5


@pytest.mark.parametrize("tf32", [0, 1])
@pytest.mark.parametrize("case", [
    (3, 3, 45, 51, 24, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1), (3, 24, 11, 13, 48, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1),
    (1, 1, 9, 7, 33, 3, 3, 2, 2, (1, 1, 1, 1), 1, 1), (2, 33, 7, 9, 64, 1, 1, 1, 1, (0, 0, 0, 0), 1, 1),
    (3, 32, 5, 5, 65, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1),      # the weight and input gradients on the unfolded matrix
    (3, 33, 5, 5, 7, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1),       # 297 terms: forward and weight gradient on the unfolded matrix
    (1, 2, 11, 10, 5, 4, 8, 2, 1, (1, 3, 2, 4), 2, 1)] + [c for c in CONV_EDGES if c[0] == 4])
def test_conv2d_on_the_fma_pipe(ctx, case, tf32):
    """fp32 products without an unfolded matrix where they are small, in both tiers (with TF32 asked for: planes off the 16-byte
    grid). The operands are TF32 values, so every path is held to the fp32 gates: 1e-6 a short sum, 1e-5 a sum over pixels."""
    s, x, wt, b, g, y, dx, dw = conv_case(*case)
    ctx.set_flags(omb.OM_TF32 if tf32 else 0)
    try:
        Y, DX, DW, DW2 = run_conv(ctx, s, x, wt, b, g)
    finally:
        ctx.set_flags(0)
    tc = tf32 and (s.n * y.shape[2] * y.shape[3]) % 4 == 0
    assert scaled_diff(Y, y) <= (2e-5 if tc else 1e-6)
    assert scaled_diff(DX, dx) <= (2e-5 if tc else 1e-6)
    assert scaled_diff(DW, dw) <= (2e-5 if tc else 1e-5)
    assert scaled_diff(DW2, 2 * dw) <= (2e-5 if tc else 1e-5)


@pytest.mark.parametrize("n,cin,h,w,cout,k,stride", [
    (3, 8, 20, 24, 40, 3, 1), (3, 9, 20, 24, 40, 3, 1), (36, 8, 20, 24, 40, 3, 1), (36, 9, 20, 24, 40, 3, 1),       # 72 and 81 terms, few and many CTAs
    (36, 32, 20, 24, 48, 3, 1), (36, 33, 20, 24, 48, 3, 1), (31, 32, 20, 24, 48, 3, 1), (32, 32, 20, 24, 32, 3, 2),  # 288 and 297 terms, either side of 120 CTAs
    (36, 28, 20, 24, 64, 3, 1), (36, 27, 20, 24, 64, 3, 1), (36, 64, 10, 24, 65, 1, 1), (2, 1, 33, 31, 3, 5, 2)])
def test_conv2d_fp32_bits_do_not_depend_on_the_kernel(ctx, K, n, cin, h, w, cout, k, stride):
    """Either side of the lines between the kernels without an unfolded matrix and the product on one, the forward and the input gradient have the
    bits of the reference's order: one chain over (channel, ky, kx), and tap by tap one chain over the output channels."""
    ctx.set_flags(0)
    pad = k // 2
    x, wt, b = normal(1, n, cin, h, w), normal(2, cout, cin, k, k, scale=0.2), normal(3, cout)
    y = K.conv2d_fwd(x, wt, b, stride, pad)
    g = normal(4, *y.shape)
    dx = K.conv2d_bwd(g, x, wt, stride, pad)[0]
    s = ConvShape(n, cin, h, w, cout, k, k, stride, stride, pad, pad, pad, pad, 1, 1, 1)
    Y, DX, _, _ = run_conv(ctx, s, x, wt, b, g)
    assert np.array_equal(Y, y)
    assert np.array_equal(DX, dx)


def test_ctc_chains_and_classes_are_bit_exact(ctx, K):
    """Extended targets of more positions than a CTA has threads, repeated labels, an empty target, more labels than steps, no steps, and a
    number of steps whose rows no longer fit on the chip: the reference's doubles bit for bit."""
    r = np.random.default_rng(4)
    for t, c, tl, il in ((150, 7, [70, 0, 3, 149, 2], [150, 150, 2, 150, 0]), (1300, 5, [90, 1], [1300, 640])):
        tl, il = np.array(tl, np.int32), np.array(il, np.int32)
        b = len(tl)
        z = r.standard_normal((t, b, c))
        lp = (z - np.log(np.exp(z).sum(-1, keepdims=True))).astype(np.float32)
        tg = r.integers(1, c, int(tl.sum())).astype(np.int32)
        for red in (0, 1, 2):
            g = normal(red, b if red == 0 else 1)
            LP, TG, TL, IL, G = (ctx.to_device(a) for a in (lp, tg, tl, il, g))
            NLL, L, GR = ctx.empty((b,)), ctx.empty(()), ctx.empty(lp.shape)
            ctx.call("om_ctc_loss", ctx.handle, LP.ptr, i32(t), i32(b), i32(c), TG.ptr, TL.ptr, IL.ptr, i32(0), i32(red), i32(1), NLL.ptr, L.ptr)
            ctx.call("om_ctc_grad", ctx.handle, G.ptr, LP.ptr, i32(t), i32(b), i32(c), TG.ptr, TL.ptr, IL.ptr, None, i32(0), i32(red), i32(1), GR.ptr)
            ctx.sync()
            assert np.array_equal(NLL.numpy(), K.ctc_loss(lp, tg, tl, il, 0, red, True)[1])
            assert np.array_equal(GR.numpy(), K.ctc_grad(g, lp, tg, tl, il, 0, red))


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(16, 16, 64), (17, 15, 65), (1, 1, 1), (16, 128, 63), (10, 512, 128), (389, 389, 129), (4 * 148 * 16, 16, 3), (4 * 148 * 16 + 1, 16, 3)])
def test_small_fp32_products_are_bit_exact(ctx, K, ta, tb, m, n, k):
    """Either side of the line between one output a thread and tiles of 64 x 64, ragged tiles and k's: the scalar chain's bits,
    with and without a bias, accumulating or not."""
    ctx.set_flags(0)
    a, b = normal(m + k, *((k, m) if ta else (m, k))), normal(n + 3 * k, *((n, k) if tb else (k, n)))
    A, B, Cm = ctx.to_device(a), ctx.to_device(b), ctx.empty((m, n))
    ref = K.gemm(a, b, bool(ta), bool(tb))
    for acc in (0, 1):
        ctx.call("om_matmul", ctx.handle, i32(ta), i32(tb), i32(m), i32(n), i32(k), A.ptr, i32(a.shape[1]), B.ptr, i32(b.shape[1]), Cm.ptr, i32(n), i32(acc))
        assert np.array_equal(Cm.numpy(), ref + ref if acc else ref)
    if not ta and tb:
        bias = normal(9, n)
        Bv = ctx.to_device(bias)
        ctx.call("om_linear_fwd", ctx.handle, A.ptr, B.ptr, Bv.ptr, i32(m), i32(k), i32(n), Cm.ptr)
        assert np.array_equal(Cm.numpy(), ref + bias)


@pytest.mark.parametrize("t,b,h", [(3, 5, 64), (4, 33, 144), (3, 17, 272), (3, 40, 400), (5, 16, 16)])
def test_whole_sequence_lstm_shapes(ctx, K, t, b, h):
    """Widths off the eight k lanes and off the 256 columns of a round, row groups with idle rows, both directions: fp32 products, 1e-4, the gate of the exact tier (only the order of the recurrent sums differs)."""
    r = np.random.default_rng(h)
    bound = 1.0 / np.sqrt(h)
    gx = r.standard_normal((t, b, 12)).astype(np.float32)
    w_ih, w_hh = (r.uniform(-bound, bound, (4 * h, n)).astype(np.float32) for n in (12, h))
    b_ih, b_hh = (r.uniform(-bound, bound, 4 * h).astype(np.float32) for _ in range(2))
    proj = r.standard_normal((t, b, h)).astype(np.float32)
    results = []
    for flags in (0, omb.OM_SEQ_KERNELS):
        ctx.set_flags(flags)
        try:
            out = []
            for reverse in (False, True):
                x, ws = omb.Tensor.from_numpy(gx, requires_grad=True), [omb.Tensor.from_numpy(a, requires_grad=True) for a in (w_ih, w_hh, b_ih, b_hh)]
                y = omb.call("lstm_layer", [x] + ws, ints=[int(reverse)])
                omb.call("sum", [omb.call("mul", [y, omb.Tensor.from_numpy(proj)])]).backward()
                out += [y.numpy(), x.grad.numpy()] + [w.grad.numpy() for w in ws]
            results.append(out)
        finally:
            ctx.set_flags(0)
    for k, (p, q) in enumerate(zip(*results)):
        assert scaled_diff(q, p) <= 1e-4, k


@pytest.mark.parametrize("tf32", [0, 1])
@pytest.mark.parametrize("off", [(1, 0), (0, 1), (1, 1)])
def test_linear_bias_off_the_16_byte_grid(ctx, tf32, off):
    """Bias and outputs one float past a 16-byte boundary, where the fp32 product adds the bias in a pass of its own: the bits of the aligned call (TF32: 2e-5)."""
    m, n, k = 640, 256, 36
    x, w, b = to_tf32(normal(1, m, k)), to_tf32(normal(2, n, k)), normal(3, n)
    ctx.set_flags(omb.OM_TF32 if tf32 else 0)
    try:
        X, W = ctx.to_device(x), ctx.to_device(w)
        out = []
        for shift in ((0, 0), off):
            B, Y = ctx.to_device(np.concatenate([np.zeros(shift[0], np.float32), b])), ctx.empty((m * n + shift[1],))
            ctx.call("om_linear_fwd", ctx.handle, X.ptr, W.ptr, C.c_void_p(B.ptr.value + 4 * shift[0]), i32(m), i32(k), i32(n), C.c_void_p(Y.ptr.value + 4 * shift[1]))
            out.append(Y.numpy()[shift[1]:])
    finally:
        ctx.set_flags(0)
    assert scaled_diff(out[1], out[0]) <= 2e-5 if tf32 else np.array_equal(out[0], out[1])


@pytest.mark.parametrize("off", [(1, 0, 0), (0, 1, 0), (0, 0, 1)])
def test_lstm_of_arrays_off_the_16_byte_grid(ctx, off):
    """Recurrent weights, initial state and outputs one float past a 16-byte boundary under OM_SEQ_KERNELS: the values of the step-by-step form, both directions
    of the pass."""
    t, b, n, h = 3, 5, 12, 32
    x, w_ih, w_hh, h0, gy = normal(1, t, b, n), normal(2, 4 * h, n, scale=0.2), normal(3, 4 * h, h, scale=0.2), normal(4, b, h), normal(5, t, b, h)
    runs = []
    for flags, shift in ((0, (0, 0, 0)), (omb.OM_SEQ_KERNELS, off)):
        ctx.set_flags(flags)
        try:
            X, WI, GY = (ctx.to_device(a) for a in (x, w_ih, gy))
            WH, H0 = (ctx.to_device(np.concatenate([np.zeros(k, np.float32), a.ravel()])) for a, k in ((w_hh, shift[0]), (h0, shift[1])))
            Y = ctx.empty((t * b * h + shift[2],))
            G, CC, TC, DX, DWI, DWH = (ctx.empty(s) for s in ((t, b, 4 * h), (t, b, h), (t, b, h), (t, b, n), w_ih.shape, w_hh.shape))
            pw, p0, py = (C.c_void_p(a.ptr.value + 4 * k) for a, k in zip((WH, H0, Y), shift))
            sizes = [i32(t), i32(b), i32(n), i32(h)]
            ctx.call("om_lstm_layer_fwd", ctx.handle, i32(0), *sizes, X.ptr, WI.ptr, pw, None, None, p0, None, py, G.ptr, CC.ptr, TC.ptr)
            ctx.call("om_lstm_layer_bwd", ctx.handle, i32(0), *sizes, GY.ptr, None, None, X.ptr, py, WI.ptr, pw, p0, None, G.ptr, CC.ptr, TC.ptr, DX.ptr, DWI.ptr, DWH.ptr,
                     None, None, None, None)
            ctx.sync()
            runs.append([Y.numpy()[shift[2]:], DX.numpy(), DWI.numpy(), DWH.numpy()])
        finally:
            ctx.set_flags(0)
    for p, q in zip(*runs):
        assert scaled_diff(q, p) <= 1e-4


@pytest.mark.parametrize("case", [
    (80, 32, 16, 16, 96, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1), (20, 48, 32, 32, 64, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1),     # half a block of channels empty
    (33, 64, 16, 16, 129, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1),     # a second block of one channel, images that no box divides
    (64, 64, 16, 16, 256, 3, 3, 2, 2, (1, 1, 1, 1), 1, 1), (130, 96, 17, 15, 64, 3, 3, 2, 2, (1, 1, 1, 1), 1, 1),   # strided, odd planes
    (256, 64, 32, 32, 128, 1, 1, 2, 2, (0, 0, 0, 0), 1, 1),    # classes that no tap reaches
    (24, 32, 20, 44, 32, 5, 5, 1, 1, (4, 4, 4, 4), 2, 2), (160, 64, 32, 4, 128, 3, 2, 1, 2, (2, 0, 1, 1), 1, 1),
    (128, 128, 4, 4, 256, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1)])
def test_conv2d_from_channels_last_copies(ctx, case):
    """Boxes of 128 and of 32 pixels over several images and rows, ragged boxes and channel blocks: TF32-valued operands, 2e-5 scaled."""
    s, x, wt, b, g, y, dx, dw = conv_case(*case)
    assert 2.0 * g.size * s.cin * s.kh * s.kw >= 1e9
    ctx.set_flags(omb.OM_TF32)
    try:
        Y, DX, DW, DW2 = run_conv(ctx, s, x, wt, b, g)
    finally:
        ctx.set_flags(0)
    for got, want in ((Y, y), (DX, dx), (DW, dw), (DW2, 2 * dw)):
        assert scaled_diff(got, want) <= 2e-5


@pytest.mark.parametrize("case", [
    (33, 64, 16, 16, 96, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1), (72, 64, 16, 16, 96, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1), (64, 64, 16, 16, 256, 3, 3, 2, 2, (1, 1, 1, 1), 1, 1),
    (40, 72, 17, 15, 160, 3, 3, 2, 2, (1, 1, 1, 1), 1, 1), (256, 64, 32, 32, 128, 1, 1, 2, 2, (0, 0, 0, 0), 1, 1),
    (24, 32, 20, 44, 32, 5, 5, 1, 1, (4, 4, 4, 4), 2, 2), (160, 64, 32, 4, 128, 3, 2, 1, 2, (2, 0, 1, 1), 1, 1), (37, 48, 11, 12, 96, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1)])
def test_conv2d_input_gradient_has_the_bits_of_product_and_fold(ctx, case):
    """The TF32 product W^T g on its own (k = output channels) and its fold, one tap after the other in float32: the same bits, so the sums are no
    less exact than those, whatever the kernel. An infinite and a NaN weight reach exactly the values whose taps lie inside the gradient's plane."""
    s, x, wt, b, g, y, dx, dw = conv_case(*case)
    n, cin, h, w, cout, kh, kw, sh, sw, (pt, pl, pb, pr), dh, dw_ = case
    oh, ow = g.shape[2:]
    kk, pixels = cin * kh * kw, n * oh * ow
    assert cout < 512 and pixels % 4 == 0 and kk % 4 == 0      # (the product does not split k)
    wt[3, 5, 0, 0], wt[1, cin - 1, kh - 1, kw - 1] = np.inf, np.nan
    G, W, DX, D = ctx.to_device(g), ctx.to_device(wt), ctx.empty(x.shape), ctx.empty((kk, pixels))
    GT = ctx.to_device(np.ascontiguousarray(g.transpose(1, 0, 2, 3).reshape(cout, pixels)))
    ctx.set_flags(omb.OM_TF32)
    try:
        ctx.call("om_conv2d_dgrad", ctx.handle, C.byref(s), G.ptr, W.ptr, DX.ptr)
        ctx.call("om_matmul", ctx.handle, i32(1), i32(0), i32(kk), i32(pixels), i32(cout), W.ptr, i32(kk), GT.ptr, i32(pixels), D.ptr, i32(pixels), i32(0))
        cols, got = D.numpy().reshape(cin, kh, kw, n, oh, ow).transpose(3, 0, 1, 2, 4, 5), DX.numpy()
    finally:
        ctx.set_flags(0)
    want = np.zeros((n, cin, h + pt + pb + dh * kh, w + pl + pr + dw_ * kw), np.float32)
    for ky in range(kh):
        for kx in range(kw):
            want[:, :, ky * dh:ky * dh + oh * sh:sh, kx * dw_:kx * dw_ + ow * sw:sw] += cols[:, :, ky, kx]
    want = want[:, :, pt:pt + h, pl:pl + w]
    assert np.array_equal(got, want, equal_nan=True)
    assert np.isfinite(want[:, 5]).any() and not np.isfinite(want[:, 5]).all() and np.isnan(want[:, cin - 1]).any()


@pytest.mark.parametrize("n,cin,h,w,cout", [(128, 128, 8, 8, 128), (64, 256, 8, 8, 512), (16, 64, 20, 32, 64), (61, 40, 20, 32, 40), (37, 48, 11, 12, 96), (7, 24, 30, 28, 200), (60, 128, 8, 54, 256)])
def test_conv2d_sums_are_no_less_exact_than_the_plain_products(ctx, n, cin, h, w, cout):
    """Forward and weight gradient against float64, beside om_matmul on the unfolded input, which splits k (the tensor core's accumulator loses bits
    with the length of a sum): values of one sign on one side, as behind a rectifier, and 5 % for the order of the sums."""
    s, x, wt, b, g, y, dx, dw = conv_case(n, cin, h, w, cout, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1)
    x = np.maximum(x, 0)
    pad, kk, pixels = np.pad(x, ((0, 0), (0, 0), (1, 1), (1, 1))), cin * 9, n * h * w
    cols = np.stack([pad[:, :, i:i + h, j:j + w] for i in range(3) for j in range(3)], 2).transpose(1, 2, 0, 3, 4).reshape(kk, pixels)
    gt, wm = np.ascontiguousarray(g.transpose(1, 0, 2, 3).reshape(cout, pixels)), wt.reshape(cout, kk)
    CO, GT, W, PY, PW = ctx.to_device(cols), ctx.to_device(gt), ctx.to_device(wm), ctx.empty((cout, pixels)), ctx.empty((cout, kk))
    ctx.set_flags(omb.OM_TF32)
    try:
        Y, DX, DW, DW2 = run_conv(ctx, s, x, wt, np.zeros_like(b), g)
        ctx.call("om_matmul", ctx.handle, i32(0), i32(0), i32(cout), i32(pixels), i32(kk), W.ptr, i32(kk), CO.ptr, i32(pixels), PY.ptr, i32(pixels), i32(0))
        ctx.call("om_matmul", ctx.handle, i32(0), i32(1), i32(cout), i32(kk), i32(pixels), GT.ptr, i32(pixels), CO.ptr, i32(pixels), PW.ptr, i32(kk), i32(0))
        py, pw = PY.numpy(), PW.numpy()
    finally:
        ctx.set_flags(0)
    far = lambda got, want: np.linalg.norm(got.astype(np.float64) - want)  # noqa: E731
    want = wm.astype(np.float64) @ cols.astype(np.float64)
    assert far(Y.transpose(1, 0, 2, 3).reshape(cout, pixels), want) <= 1.05 * far(py, want)
    want = gt.astype(np.float64) @ cols.T.astype(np.float64)
    assert far(DW.reshape(cout, kk), want) <= 1.05 * far(pw, want)


@pytest.mark.parametrize("tf32", [0, 1])
@pytest.mark.parametrize("case", [(4, 8, 8, 8, 12, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1), (4, 4, 14, 14, 9, 3, 3, 3, 3, (1, 1, 1, 1), 1, 1), (4, 4, 12, 12, 9, 6, 6, 1, 1, (2, 2, 2, 2), 1, 1),
                                  (33, 64, 16, 16, 96, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1), (8, 64, 8, 8, 64, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1)])
def test_conv2d_of_arrays_off_the_16_byte_grid(ctx, case, tf32):
    """Every array one float past a 16-byte boundary, as a slice of a larger tensor may be: the values of the aligned call (2e-5, another order of sums)."""
    s, x, wt, b, g, y, dx, dw = conv_case(*case)
    ctx.set_flags(omb.OM_TF32 if tf32 else 0)
    off = lambda a: C.c_void_p(a.ptr.value + 4)  # noqa: E731
    try:
        X, W, B, G = (ctx.to_device(np.concatenate([np.zeros(1, np.float32), a.ravel()])) for a in (x, wt, b, g))
        Y, DX, DW = (ctx.empty((a.size + 1,)) for a in (g, x, wt))
        ctx.call("om_conv2d_fwd", ctx.handle, C.byref(s), off(X), off(W), off(B), off(Y))
        ctx.call("om_conv2d_dgrad", ctx.handle, C.byref(s), off(G), off(W), off(DX))
        ctx.call("om_conv2d_wgrad", ctx.handle, C.byref(s), off(G), off(X), off(DW), i32(0))
        ctx.sync()
        for got, want in ((Y, y), (DX, dx), (DW, dw)):
            assert scaled_diff(got.numpy()[1:].reshape(want.shape), want) <= 2e-5
    finally:
        ctx.set_flags(0)


@pytest.mark.parametrize("n,cout,h,w", [(1, 3, 2, 2), (5, 7, 4, 16), (17, 2, 33, 31), (3, 4, 1, 3), (40, 5, 40, 64)])
def test_conv2d_bias_gradient_planes(ctx, n, cout, h, w):
    """Planes smaller and larger than a CTA's stride, of a multiple of four floats or not: sums in double, 1e-6."""
    s, g = ConvShape(n, 1, h, w, cout, 1, 1, 1, 1, 0, 0, 0, 0, 1, 1, 1), normal(n, n, cout, h, w)
    G, DB = ctx.to_device(g), ctx.empty((cout,))
    ctx.call("om_conv2d_dbias", ctx.handle, C.byref(s), G.ptr, DB.ptr, i32(0))
    want = g.astype(np.float64).sum((0, 2, 3))
    assert np.max(np.abs(DB.numpy() - want) / np.abs(g).astype(np.float64).sum((0, 2, 3))) <= 1e-6


@pytest.mark.parametrize("planes,h,w,kh,kw", [(3, 4, 8, 2, 2), (2, 6, 12, 3, 1), (5, 4, 4, 4, 4), (1, 2, 4, 1, 2), (2, 5, 8, 2, 2), (300, 8, 20, 4, 1)])
def test_max_pool_windows_are_bit_exact(ctx, K, planes, h, w, kh, kw):
    """Windows that tile the plane: ties go to the first, NaN wins, all -inf; the bits and the indices of the oracle (a height that the window
    does not divide keeps the general kernels)."""
    x = np.round(normal(kh * 10 + kw, 1, planes, h, w) * 2) / 2
    x.reshape(-1)[::17], x[0, 0, :kh, :kw] = np.nan, -np.inf
    y, idx = K.maxpool_fwd(x, kh, kw, kh, kw, 0, 0)
    X, Y, I = ctx.to_device(x), ctx.empty(y.shape), ctx.empty(y.shape, np.int32)
    geometry = [i32(v) for v in (planes, h, w, kh, kw, kh, kw, 0, 0)]
    ctx.call("om_maxpool_fwd", ctx.handle, X.ptr, *geometry, Y.ptr, I.ptr)
    assert np.array_equal(Y.numpy(), y, equal_nan=True) and np.array_equal(I.numpy(), idx)
    g = normal(3, *y.shape)
    G, DX = ctx.to_device(g), ctx.empty(x.shape)
    ctx.call("om_maxpool_bwd", ctx.handle, G.ptr, I.ptr, i32(planes), i32(h), i32(w), i32(y.shape[2]), i32(y.shape[3]), i32(kh), i32(kw), i32(kh), i32(kw), i32(0),
             i32(0), DX.ptr)
    want = np.zeros(x.size, np.float32)
    want[idx.reshape(-1)] = g.reshape(-1)
    assert np.array_equal(DX.numpy().reshape(-1), want)


@pytest.mark.parametrize("rows,cols", [(1, 320), (7, 64), (2367, 128), (2369, 256), (296 * 56 + 1, 32), (5000, 384)])
def test_layer_norm_backward_rows_per_cta(ctx, K, rows, cols):
    """Eight rows a CTA, the next step of eight, and the most: 1e-4, the gate of the layer norm tests; parameter sums in double."""
    x, g, gamma = normal(1, rows, cols), normal(2, rows, cols), normal(3, cols)
    beta = normal(4, cols)
    X, G, GA, BE = (ctx.to_device(a) for a in (x, g, gamma, beta))
    Y, M, I, DX, DG, DB = ctx.empty(x.shape), ctx.empty((rows,)), ctx.empty((rows,)), ctx.empty(x.shape), ctx.empty((cols,)), ctx.empty((cols,))
    ctx.call("om_layernorm_fwd", ctx.handle, X.ptr, GA.ptr, BE.ptr, i32(rows), i32(cols), f32(1e-5), Y.ptr, M.ptr, I.ptr)
    ctx.call("om_layernorm_bwd", ctx.handle, G.ptr, X.ptr, GA.ptr, M.ptr, I.ptr, i32(rows), i32(cols), DX.ptr, DG.ptr, DB.ptr, i32(0))
    x64, g64 = x.astype(np.float64), g.astype(np.float64)
    inv = 1.0 / np.sqrt(x64.var(1, keepdims=True) + 1e-5)
    xh, dh = (x64 - x64.mean(1, keepdims=True)) * inv, g64 * gamma
    assert scaled_diff(DX.numpy(), inv * (dh - dh.mean(1, keepdims=True) - xh * (dh * xh).mean(1, keepdims=True))) <= 1e-4
    assert scaled_diff(DG.numpy(), (g64 * xh).sum(0)) <= 1e-4 and scaled_diff(DB.numpy(), g64.sum(0)) <= 1e-4


@pytest.mark.parametrize("rows,cols,ld", [(3, 4096, 4096), (2, 4099, 4100), (5, 8193, 8196), (300, 16385, 16392), (2, 30522, 30528), (2, 32768, 32768), (2, 32769, 32772),
                                          (2, 4099, 4099)])
def test_cross_entropy_of_wide_rows(ctx, rows, cols, ld):
    """Rows held in registers and the widths on either side of them, ragged ends, pitched rows: against float64, 1e-6 of the largest value forward, 1e-5
    backward (the log-softmax is rounded to fp32 before its exponential)."""
    x = normal(cols, rows, ld, scale=3.0)
    t = np.random.default_rng(1).integers(0, cols, rows)
    t[-1] = -100
    x64 = x[:, :cols].astype(np.float64)
    lse = np.log(np.exp(x64 - x64.max(1, keepdims=True)).sum(1, keepdims=True)) + x64.max(1, keepdims=True)
    X, T = ctx.to_device(x), ctx.to_device(t)
    LP, L, N, D, G = ctx.to_device(np.zeros_like(x)), ctx.empty(()), ctx.empty((1,), np.int32), ctx.to_device(np.zeros_like(x)), ctx.to_device(np.ones(1, np.float32))
    ctx.call("om_cross_entropy_fwd_ld", ctx.handle, X.ptr, T.ptr, i32(omb.OM_I64), i32(rows), i32(cols), i32(ld), i32(1), i64(-100), f32(0.0), LP.ptr, L.ptr, N.ptr)
    ctx.call("om_cross_entropy_bwd_ld", ctx.handle, G.ptr, LP.ptr, T.ptr, i32(omb.OM_I64), i32(rows), i32(cols), i32(ld), i32(1), i64(-100), f32(0.0), D.ptr)
    want = np.exp(x64 - lse)
    want[np.arange(rows - 1), t[:-1]] -= 1.0
    want[-1] = 0.0
    assert scaled_diff(LP.numpy()[:, :cols], x64 - lse) <= 1e-6
    assert scaled_diff(D.numpy()[:, :cols], want / (rows - 1)) <= 1e-5
    assert abs(float(L.numpy()) - (lse[:-1, 0] - x64[np.arange(rows - 1), t[:-1]]).mean()) <= 1e-5 * 10
    assert int(N.numpy()[0]) == rows - 1 and not LP.numpy()[:, cols:].any() and not D.numpy()[:, cols:].any()


@pytest.mark.parametrize("tf32", [0, 1])
@pytest.mark.parametrize("case", [(33, 64, 16, 16, 96, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1), (64, 64, 16, 16, 256, 3, 3, 2, 2, (1, 1, 1, 1), 1, 1),
                                  (80, 32, 16, 16, 97, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1), (3, 5, 9, 7, 6, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1)])
def test_conv2d_backward_in_one_call(ctx, case, tf32):
    """Together and one by one: the same bits (the bias gradient, another order of sums in double, within 1e-6), each result left out too."""
    s, x, wt, b, g, y, dx, dw = conv_case(*case)
    ctx.set_flags(omb.OM_TF32 if tf32 else 0)
    try:
        X, W, G = (ctx.to_device(a) for a in (x, wt, g))
        DX, DW, DB = (ctx.empty(a) for a in (x.shape, wt.shape, b.shape))
        apart = run_conv(ctx, s, x, wt, b, g)
        want = g.astype(np.float64).sum((0, 2, 3))
        for skip in (None, 0, 1, 2):
            out = [None if skip == i else a.ptr for i, a in enumerate((DX, DW, DB))]
            ctx.call("om_conv2d_bwd", ctx.handle, C.byref(s), G.ptr, X.ptr, W.ptr, out[0], out[1], i32(0), out[2], i32(0))
            assert skip == 0 or np.array_equal(DX.numpy(), apart[1])
            assert skip == 1 or np.array_equal(DW.numpy(), apart[2])
            assert skip == 2 or np.max(np.abs(DB.numpy() - want) / np.abs(g).astype(np.float64).sum((0, 2, 3))) <= 1e-6
        ctx.call("om_conv2d_bwd", ctx.handle, C.byref(s), G.ptr, X.ptr, W.ptr, DX.ptr, DW.ptr, i32(1), DB.ptr, i32(1))
        assert np.array_equal(DW.numpy(), apart[3]) and scaled_diff(DB.numpy(), 2 * want) <= 2e-6
    finally:
        ctx.set_flags(0)


@pytest.mark.parametrize("tf32", [0, 1])
@pytest.mark.parametrize("case", [(48, 64, 16, 16, 96, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1), (64, 64, 16, 16, 256, 3, 3, 2, 2, (1, 1, 1, 1), 1, 1), (3, 5, 9, 7, 6, 3, 3, 1, 1, (1, 1, 1, 1), 1, 1)])
def test_conv2d_parameter_gradients_before_the_input_gradient(ctx, case, tf32):
    """The two calls give the bits of the one; after the first the parameters' gradients are there and nothing of the input gradient is."""
    s, x, wt, b, g, y, dx, dw = conv_case(*case)
    ctx.set_flags(omb.OM_TF32 if tf32 else 0)
    try:
        X, W, G = (ctx.to_device(a) for a in (x, wt, g))
        DX, DW, DB, DX2, DW2, DB2 = (ctx.empty(a) for a in (x.shape, wt.shape, b.shape) * 2)
        floats = C.c_int64()
        ctx.call("om_conv2d_bwd_workspace", ctx.handle, C.byref(s), C.byref(floats))
        assert (floats.value > 0) == bool(tf32 and g.size > 1e5)
        ws = ctx.empty((max(4, floats.value),))        # (not looked at where nothing is shared)
        ctx.call("om_conv2d_bwd", ctx.handle, C.byref(s), G.ptr, X.ptr, W.ptr, DX.ptr, DW.ptr, i32(0), DB.ptr, i32(0))
        ctx.call("om_memset", ctx.handle, DX2.ptr, i32(0x2b), C.c_size_t(x.nbytes))
        ctx.call("om_conv2d_bwd_params", ctx.handle, C.byref(s), G.ptr, X.ptr, DW2.ptr, i32(0), DB2.ptr, i32(0), ws.ptr)
        assert np.array_equal(DW2.numpy(), DW.numpy()) and np.array_equal(DB2.numpy(), DB.numpy())
        assert (DX2.numpy().view(np.uint32) == 0x2b2b2b2b).all()
        ctx.call("om_conv2d_bwd_input", ctx.handle, C.byref(s), G.ptr, W.ptr, DX2.ptr, ws.ptr)
        assert np.array_equal(DX2.numpy(), DX.numpy())
    finally:
        ctx.set_flags(0)


@pytest.mark.parametrize("n,c,h,w,offset", [(2, 3, 1, 1, 0.0), (5, 2, 3, 1, 0.0), (17, 4, 7, 9, 1e4), (33, 3, 16, 16, -1e4), (3, 2, 128, 130, 100.0), (1, 5, 1, 4, 0.0)])
def test_batch_norm_statistics_and_sums(ctx, n, c, h, w, offset):
    """Empty and ragged slices, planes on and off four values, pieces smaller and larger than a CTA's registers, and channels whose mean is ten
    thousand deviations away (nothing may cancel): the saved statistics within 1e-6 of float64, gradients within 1e-4."""
    x, g = (normal(n + c, n, c, h, w) + np.float32(offset)).astype(np.float32), normal(7, n, c, h, w)
    gamma, beta = normal(8, c), normal(9, c)
    X, G, GA, BE, RM, RV = (ctx.to_device(a) for a in (x, g, gamma, beta, np.zeros(c, np.float32), np.ones(c, np.float32)))
    Y, M, I, DX, DG, DB = ctx.empty(x.shape), ctx.empty((c,)), ctx.empty((c,)), ctx.empty(x.shape), ctx.empty((c,)), ctx.empty((c,))
    ctx.call("om_batchnorm_fwd", ctx.handle, X.ptr, GA.ptr, BE.ptr, RM.ptr, RV.ptr, i32(n), i32(c), i32(h * w), i32(1), f32(0.1), f32(1e-5), Y.ptr, M.ptr, I.ptr)
    ctx.call("om_batchnorm_bwd", ctx.handle, G.ptr, X.ptr, GA.ptr, M.ptr, I.ptr, i32(n), i32(c), i32(h * w), i32(1), DX.ptr, DG.ptr, DB.ptr, i32(0))
    x64, g64 = x.astype(np.float64), g.astype(np.float64)
    mu, var, m = x64.mean((0, 2, 3)), x64.var((0, 2, 3)), n * h * w
    assert np.max(np.abs(M.numpy() - mu) / np.maximum(np.abs(mu), 1e-3)) <= 1e-6
    assert np.max(np.abs(I.numpy() * np.sqrt(var + 1e-5) - 1)) <= 1e-6
    assert np.max(np.abs(RV.numpy() - (0.9 + 0.1 * var * m / max(m - 1, 1)))) <= 1e-6 * (1 + np.max(var))
    mean, inv = (a.numpy().astype(np.float64)[None, :, None, None] for a in (M, I))     # (the gradient is that of the saved statistics)
    xh = (x64 - mean) * inv
    sb, sg = g64.sum((0, 2, 3)), (g64 * xh).sum((0, 2, 3))
    assert np.max(np.abs(DB.numpy() - sb)) <= 1e-5 * max(1.0, np.max(np.abs(sb)))
    assert np.max(np.abs(DG.numpy() - sg)) <= 1e-4 * max(1.0, np.max(np.abs(sg)))
    want = gamma[None, :, None, None] * inv * (g64 - sb[None, :, None, None] / m - xh * sg[None, :, None, None] / m)
    assert np.max(np.abs(DX.numpy() - want)) <= 1e-4 * max(1.0, np.max(np.abs(want)))


@pytest.mark.parametrize("n,c,h,w,training", [(5, 3, 4, 4, 1), (3, 2, 3, 5, 1), (17, 4, 16, 20, 1), (4, 3, 7, 4, 0)])
def test_batch_norm_with_its_rectifier(ctx, n, c, h, w, training):
    """One call against the norm followed by the rectifier: the same bits forward and backward, negative and zero inputs and a NaN among them."""
    x, g = normal(1, n, c, h, w), normal(2, n, c, h, w)
    gamma, beta = normal(3, c), normal(4, c)
    gamma[0] = 0.0                       # a channel whose rectifier sees beta alone
    if not training:
        x[0, 1, 0, 0] = np.nan
    X, G, GA, BE = (ctx.to_device(a) for a in (x, g, gamma, beta))
    geometry = [i32(n), i32(c), i32(h * w)]
    out = {}
    for fused in (0, 1):
        RM, RV = ctx.to_device(np.full(c, 0.1, np.float32)), ctx.to_device(np.full(c, 2.0, np.float32))
        Y, M, I, DX, DG, DB, U = ctx.empty(x.shape), ctx.empty((c,)), ctx.empty((c,)), ctx.empty(x.shape), ctx.empty((c,)), ctx.empty((c,)), ctx.empty((c,))
        args = [X.ptr, GA.ptr, BE.ptr, RM.ptr, RV.ptr, *geometry, i32(training), f32(0.1), f32(1e-5)]
        if fused:
            ctx.call("om_batchnorm_relu_fwd", ctx.handle, *args, Y.ptr, M.ptr, I.ptr, U.ptr)
            ctx.call("om_batchnorm_relu_bwd", ctx.handle, G.ptr, X.ptr, GA.ptr, U.ptr, M.ptr, I.ptr, *geometry, i32(training), DX.ptr, DG.ptr, DB.ptr, i32(0))
            assert np.array_equal(U.numpy(), beta)
        else:
            Z, GZ = ctx.empty(x.shape), ctx.empty(x.shape)
            ctx.call("om_batchnorm_fwd", ctx.handle, *args, Z.ptr, M.ptr, I.ptr)
            ctx.call("om_unary", ctx.handle, i32(1), Z.ptr, Y.ptr, i64(x.size))
            ctx.call("om_unary_bwd", ctx.handle, i32(1), G.ptr, Y.ptr, GZ.ptr, i64(x.size))
            ctx.call("om_batchnorm_bwd", ctx.handle, GZ.ptr, X.ptr, GA.ptr, M.ptr, I.ptr, *geometry, i32(training), DX.ptr, DG.ptr, DB.ptr, i32(0))
        out[fused] = [a.numpy().copy() for a in (Y, M, I, RM, RV, DX, DG, DB)]
    for a, b in zip(out[0], out[1]):
        assert np.array_equal(a, b, equal_nan=True)


def test_batch_norm_relu_backward_needs_the_beta_of_the_forward(ctx):
    """The forward may leave it out (no gradient wanted); the backward without it is refused on the host."""
    X, V = ctx.to_device(normal(1, 2, 3, 2, 2)), ctx.to_device(np.ones(3, np.float32))
    with pytest.raises(omb.OmError) as e:
        ctx.call("om_batchnorm_relu_bwd", ctx.handle, X.ptr, X.ptr, V.ptr, None, V.ptr, V.ptr, i32(2), i32(3), i32(4), i32(1), None, None, None, i32(0))
    assert e.value.status == 8      # OM_ERR_ARG
    ctx.sync()


@pytest.mark.parametrize("relu", [0, 1])
@pytest.mark.parametrize("off", [(1, 1, 1, 1), (1, 0, 0, 0), (0, 1, 0, 0), (0, 0, 1, 0), (0, 0, 0, 1)])
def test_batch_norm_of_planes_off_the_16_byte_grid(ctx, relu, off):
    """x, y, g and dx one float past a 16-byte boundary, together and alone, planes of whole float4s: the bits of the aligned calls where the statistics'
    own accesses are the same, and 1e-6 where their double sums run in another order."""
    n, c, h, w = 5, 3, 4, 8
    x, g, gamma, beta = normal(1, n, c, h, w), normal(2, n, c, h, w), normal(3, c), normal(4, c)
    out = []
    for shift in ((0, 0, 0, 0), off):
        X, G = (ctx.to_device(np.concatenate([np.zeros(k, np.float32), a.ravel()])) for a, k in ((x, shift[0]), (g, shift[2])))
        Y, DX = (ctx.empty((x.size + k,)) for k in (shift[1], shift[3]))
        GA, BE, RM, RV = (ctx.to_device(a) for a in (gamma, beta, np.zeros(c, np.float32), np.ones(c, np.float32)))
        M, I, DG, DB, U = (ctx.empty((c,)) for _ in range(5))
        px, py, pg, pd = (C.c_void_p(a.ptr.value + 4 * k) for a, k in zip((X, Y, G, DX), shift))
        geometry, last = [i32(n), i32(c), i32(h * w)], [i32(1), pd, DG.ptr, DB.ptr, i32(0)]
        ctx.call("om_batchnorm_relu_fwd" if relu else "om_batchnorm_fwd", ctx.handle, px, GA.ptr, BE.ptr, RM.ptr, RV.ptr, *geometry, i32(1), f32(0.1), f32(1e-5), py, M.ptr, I.ptr,
                 *([U.ptr] if relu else []))
        ctx.call("om_batchnorm_relu_bwd" if relu else "om_batchnorm_bwd", ctx.handle, pg, px, GA.ptr, *([U.ptr] if relu else []), M.ptr, I.ptr, *geometry, *last)
        ctx.sync()
        out.append([Y.numpy()[shift[1]:], DX.numpy()[shift[3]:], M.numpy(), I.numpy(), DG.numpy(), DB.numpy()])
    for a, b in zip(*out):
        assert np.array_equal(a, b) if not (off[0] or off[2]) else np.max(np.abs(a - b)) <= 1e-6 * np.max(np.abs(a))


@pytest.mark.parametrize("v,dim,n", [(50, 16, 20), (7, 3, 5), (300, 8, 64)])
def test_kernels_of_a_chain_read_what_the_chain_wrote(ctx, v, dim, n):
    """A count that one kernel of a chain leaves and others read, while a slow kernel in front lets the whole chain queue up: every round has
    another number of rows, and the dense form is that of float32 additions in position order."""
    r = np.random.default_rng(v)
    slow, S = ctx.to_device(normal(1, 4096)), ctx.empty((1,))
    cap = min(n, v)
    rows, values, count = ctx.empty((cap,), np.int32), ctx.empty((cap, dim)), ctx.to_device(np.zeros(1, np.int32))
    for distinct in (cap, 1, cap // 2, 2, cap):
        ids = r.permutation(v)[:distinct][r.integers(0, distinct, n)].astype(np.int32)
        g = normal(distinct, n, dim)
        I, G, D = ctx.to_device(ids), ctx.to_device(g), ctx.to_device(np.zeros((v, dim), np.float32))
        for _ in range(4):
            ctx.call("om_reduce_fwd", ctx.handle, slow.ptr, i64(1), i64(4096), i64(1), i32(0), S.ptr)
        ctx.call("om_embedding_bwd_sparse", ctx.handle, G.ptr, I.ptr, i32(1), i64(n), i32(v), i32(dim), i64(-1), rows.ptr, values.ptr, i32(cap), count.ptr)
        ctx.call("om_rowsparse_add_to", ctx.handle, rows.ptr, values.ptr, count.ptr, i32(cap), i32(dim), D.ptr, i32(v))
        want = np.zeros((v, dim), np.float32)
        np.add.at(want, ids, g)
        assert count.numpy()[0] == np.unique(ids).size
        assert np.array_equal(D.numpy(), want)


@pytest.mark.parametrize("n,c,h,w", [(6, 3, 4, 4), (5, 3, 3, 5), (70, 3, 16, 8)])
def test_batch_norm_statistics_with_infinities(ctx, n, c, h, w):
    """An infinite value makes its channel's mean infinite (and the running mean), both signs make it NaN; the other channel is unharmed."""
    x = normal(1, n, c, h, w)
    x[1, 0, 1, 2] = np.inf
    x[0, 1, 0, 0], x[n - 1, 1, 2, 1] = np.inf, -np.inf
    X, GA, BE, RM, RV = (ctx.to_device(a) for a in (x, np.ones(c, np.float32), np.zeros(c, np.float32), np.zeros(c, np.float32), np.ones(c, np.float32)))
    Y, M, I = ctx.empty(x.shape), ctx.empty((c,)), ctx.empty((c,))
    ctx.call("om_batchnorm_fwd", ctx.handle, X.ptr, GA.ptr, BE.ptr, RM.ptr, RV.ptr, i32(n), i32(c), i32(h * w), i32(1), f32(0.1), f32(1e-5), Y.ptr, M.ptr, I.ptr)
    mean, running = M.numpy(), RM.numpy()
    assert mean[0] == np.inf and running[0] == np.inf and np.isnan(mean[1]) and np.isnan(running[1])
    assert np.isnan(I.numpy()[:2]).all() and np.isfinite(Y.numpy()[:, 2]).all()
    assert abs(mean[2] - x[:, 2].astype(np.float64).mean()) <= 1e-6
