"""sparse_conv2d (1x1) on the GPU over the reference's encoding, checked against the dense
convolution on the densified weights (int8: exact oracle; fp32: the ARM accumulation order)."""
import numpy as np
import pytest
import torch

from helpers import O, assert_f32_close

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def sparse_weights(seed, cout, cin, semi, keep=0.2):
    rng = np.random.default_rng(seed)
    w = (rng.standard_normal((cout, cin)) * 0.05).astype(np.float32)
    if semi:
        mask = np.repeat(rng.random(((cout + 1) // 2, cin)) < keep, 2, axis=0)[:cout]
    else:
        mask = rng.random((cout, cin)) < keep
    return (w * mask).astype(np.float32)


# cin, cout, hw side, batch
SHAPES = [(32, 64, 12, 2), (128, 128, 14, 2), (256, 256, 7, 3), (109, 33, 5, 1), (512, 512, 7, 1),
          # images of more than 1024 pixels (several blocks of the shared-memory slab kernels, ragged last block),
          # channel counts on each side of the slab kernels' pixels-per-thread thresholds, odd pixel counts
          (24, 40, 36, 1), (48, 16, 34, 2), (100, 20, 33, 1), (150, 8, 36, 1),
          # fp32 pixel-tile kernel: 16 and 8 lanes per output channel (cin > 128, > 256), ragged last tile, cin > 512 (fallback)
          (200, 96, 16, 2), (512, 48, 12, 1), (130, 37, 30, 1), (520, 24, 8, 1)]


@pytest.mark.parametrize("impl", [1, 2, 0], ids=["walk", "densified", "auto"])
@pytest.mark.parametrize("semi", [False, True], ids=["unstructured", "semi"])
@pytest.mark.parametrize("cin,cout,side,batch", SHAPES)
def test_sparse_int8(plb, ctx, cin, cout, side, batch, semi, impl):
    wf = sparse_weights(cin + cout, cout, cin, semi)
    wq, ws = O.quantize_per_channel(wf)
    rng = np.random.default_rng(5)
    xq, in_s = O.quantize_per_tensor(rng.standard_normal((batch, cin, side, side)).astype(np.float32))
    bias = (rng.standard_normal(cout) * 0.1).astype(np.float32)
    enc = O.sparse_encode(wq, side * side, semi=semi)
    assert np.array_equal(O.sparse_decode(enc, cout, cin, side * side), wq)
    acc = O.conv_acc_i32(xq, wq[:, :, None, None])
    y_ref = O.epilogue(acc, ws, in_s, bias, O.ACT_RELU, 0.0)
    out_s = float(np.abs(y_ref).max() / 127)
    q_ref = O.epilogue(acc, ws, in_s, bias, O.ACT_RELU, 0.0, out_scale=out_s)
    args = (enc["nonzero_weights"], enc["oc_nonzeros"], enc["diffs"], enc["first_ic"], enc["flag_semi"])
    kw = dict(cin=cin, cout=cout, in_hw=(side, side), wscale=ws, in_scale=in_s, bias=bias, act=O.ACT_RELU,
              impl=impl)
    x = dev(xq)
    y = plb.SparseConv(ctx, *args, **kw).run(x).cpu().numpy()
    q = plb.SparseConv(ctx, *args, out_scale=out_s, **kw).run(x).cpu().numpy()
    ctx.sync()
    assert np.array_equal(y, y_ref)
    assert np.array_equal(q, q_ref)


@pytest.mark.parametrize("semi", [False, True], ids=["unstructured", "semi"])
@pytest.mark.parametrize("cin,cout,side,batch", SHAPES[:4] + SHAPES[5:])  # (512 x 512 takes the oracle too long)
def test_sparse_fp32(plb, ctx, cin, cout, side, batch, semi):
    wf = sparse_weights(cin * 3 + cout, cout, cin, semi)
    rng = np.random.default_rng(6)
    x = rng.standard_normal((batch, cin, side, side)).astype(np.float32)
    bias = (rng.standard_normal(cout) * 0.1).astype(np.float32)
    enc = O.sparse_encode(wf, side * side, semi=semi)
    y_ref = O.sparse_conv_f32(x, wf, bias, O.ACT_RELU)
    y64 = O.sparse_conv_f32(x, wf, bias, O.ACT_RELU, f64=True)
    sp = plb.SparseConv(ctx, enc["nonzero_weights"], enc["oc_nonzeros"], enc["diffs"], enc["first_ic"],
                        enc["flag_semi"], cin=cin, cout=cout, in_hw=(side, side), bias=bias, act=O.ACT_RELU)
    y = sp.run(dev(x)).cpu().numpy()
    ctx.sync()
    assert np.array_equal(y, y_ref), "fp32 sparse differs from the ordered fma oracle"
    # against fp64: 1e-5 of the output range (single fp32 sums of ~0.2*cin products carry ~1e-7)
    assert_f32_close(y, y64, rel=1e-5, floor=float(np.abs(y64).max()))


# fp32 walk over tensor memory: row lengths 0 and up to 20 of every remainder of a batch, chunks of channels with empty rows
# in front, between and behind, pixel groups across images, teams that share a group, planes of whole 16-byte groups or not
@pytest.mark.parametrize("cin,cout,h,w,batch", [(8, 23, 4, 4, 1), (128, 25, 5, 5, 7), (129, 30, 8, 4, 70), (300, 41, 3, 11, 5),
                                                (64, 4, 1, 1, 3), (640, 9, 7, 7, 12), (32, 3, 40, 40, 60), (40, 70, 9, 7, 40)])
@pytest.mark.parametrize("act,alpha", [(0, 0.0), (2, 1.5), (3, 0.1)])
def test_sparse_fp32_row_lengths(plb, ctx, cin, cout, h, w, batch, act, alpha):
    rng = np.random.default_rng(cin + cout)
    wf = np.zeros((cout, cin), np.float32)
    for oc in range(cout):
        cols = rng.permutation(cin)[:min(cin, oc if oc < 21 else 3)]
        if oc % 5 == 4:
            cols = cols[cols >= min(cin - 1, 128)]
        wf[oc, cols] = rng.standard_normal(len(cols))
    x = rng.standard_normal((batch, cin, h, w)).astype(np.float32)
    bias = rng.standard_normal(cout).astype(np.float32) if act else None
    enc = O.sparse_encode(wf, h * w)
    sp = plb.SparseConv(ctx, enc["nonzero_weights"], enc["oc_nonzeros"], enc["diffs"], enc["first_ic"], enc["flag_semi"],
                        cin=cin, cout=cout, in_hw=(h, w), bias=bias, act=act, alpha=alpha)
    y_ref = O.sparse_conv_f32(x, wf, bias if bias is not None else np.zeros(cout, np.float32), act, alpha)
    for offset in (0, 1):  # the second one: tensors off the 16-byte grid
        xd = torch.empty(x.size + offset, device="cuda")[offset:].view(x.shape)
        xd.copy_(dev(x))
        yd = torch.full((y_ref.size + offset,), 7.0, device="cuda")[offset:].view(y_ref.shape)
        sp.run(xd, out=yd)
        ctx.sync()
        assert np.array_equal(yd.cpu().numpy(), y_ref)


def special_values(plb, ctx, cin, hw):
    """Only the non-zeros take part: infinities and NaN in a channel reach exactly the outputs that read it, and a sum of
    negative zeros stays one."""
    cout = 12
    rng = np.random.default_rng(3)
    wf = np.where(rng.random((cout, cin)) < 0.1, rng.standard_normal((cout, cin)), 0).astype(np.float32)
    wf[3, :] = 0
    x = rng.standard_normal((2, cin, hw, hw)).astype(np.float32)
    x[0, 5], x[1, 140], x[0, 70, 2, 3] = np.inf, np.nan, -np.inf
    bias = rng.standard_normal(cout).astype(np.float32)
    bias[3] = -0.0
    enc = O.sparse_encode(wf, hw * hw)
    y = plb.SparseConv(ctx, enc["nonzero_weights"], enc["oc_nonzeros"], enc["diffs"], enc["first_ic"], enc["flag_semi"],
                       cin=cin, cout=cout, in_hw=(hw, hw), bias=bias).run(dev(x)).cpu().numpy()
    ctx.sync()
    y_ref = O.sparse_conv_f32(x, wf, bias, O.ACT_NONE)
    assert np.array_equal(np.isnan(y), np.isnan(y_ref)) and np.isnan(y_ref).any()
    ok = ~np.isnan(y_ref)
    assert np.array_equal(y[ok].view(np.int32), y_ref[ok].view(np.int32))
    assert np.all(np.signbit(y[:, 3]))


def test_sparse_fp32_special_values(plb, ctx):
    special_values(plb, ctx, 150, 6)


# The two tests above on the tensor-memory kernel whatever the choice between kernels says: 1, 2, 3 and 5 chunks of channels,
# on and off the 16-byte grid.
@pytest.mark.parametrize("cin,cout,h,w,batch", [(60, 23, 4, 4, 40), (129, 30, 8, 4, 9), (300, 41, 3, 11, 5), (300, 41, 4, 12, 5),
                                                (640, 9, 7, 7, 12), (640, 26, 8, 8, 3)])
@pytest.mark.parametrize("act,alpha", [(0, 0.0), (2, 1.5), (3, 0.1)])
def test_sparse_fp32_row_lengths_in_tensor_memory(plb, ctx, monkeypatch, cin, cout, h, w, batch, act, alpha):
    monkeypatch.setenv("PLB_SPARSE_TMEM", "1")
    before = ctx.sparse_tmem_launch_count()
    test_sparse_fp32_row_lengths(plb, ctx, cin, cout, h, w, batch, act, alpha)
    assert ctx.sparse_tmem_launch_count() == before + 2


@pytest.mark.parametrize("cin,hw", [(150, 6), (150, 5), (300, 6), (600, 6), (600, 5)])
def test_sparse_fp32_special_values_in_tensor_memory(plb, ctx, monkeypatch, cin, hw):
    monkeypatch.setenv("PLB_SPARSE_TMEM", "1")
    before = ctx.sparse_tmem_launch_count()
    special_values(plb, ctx, cin, hw)
    assert ctx.sparse_tmem_launch_count() == before + 1


# (cin, cout, h, w, batch, density, kernel): both sides of the lines between tensor memory, shared-memory tiles and one thread
# per output
@pytest.mark.parametrize("cin,cout,h,w,batch,density,tmem", [
    (489, 33, 18, 18, 2, 0.08, False), (128, 46, 30, 30, 17, 0.1, True), (329, 43, 16, 16, 7, 0.06, False),
    (192, 82, 5, 5, 12, 0.15, False), (224, 101, 5, 5, 2, 0.31, False), (448, 150, 33, 33, 4, 0.3, True), (100, 40, 5, 5, 3, 0.2, True),
])
def test_sparse_fp32_kernel_choice(plb, ctx, cin, cout, h, w, batch, density, tmem):
    rng = np.random.default_rng(cin)
    wf = np.where(rng.random((cout, cin)) < density, rng.standard_normal((cout, cin)), 0).astype(np.float32)
    x = rng.standard_normal((batch, cin, h, w)).astype(np.float32)
    bias = rng.standard_normal(cout).astype(np.float32)
    enc = O.sparse_encode(wf, h * w)
    before = ctx.sparse_tmem_launch_count()
    y = plb.SparseConv(ctx, enc["nonzero_weights"], enc["oc_nonzeros"], enc["diffs"], enc["first_ic"], enc["flag_semi"],
                       cin=cin, cout=cout, in_hw=(h, w), bias=bias, act=O.ACT_RELU).run(dev(x))
    ctx.sync()
    assert ctx.sparse_tmem_launch_count() - before == (1 if tmem else 0)
    assert np.array_equal(y.cpu().numpy(), O.sparse_conv_f32(x, wf, bias, O.ACT_RELU))


# the sparse_conv benchmark shapes: MobileNetV1 pointwise layers at batch 256, 80 % of the weights masked
CONFIG5 = [(32, 64, 112), (128, 128, 56), (256, 256, 28), (512, 512, 14), (1024, 1024, 7)]


@pytest.mark.parametrize("semi", [False, True], ids=["unstructured", "semi"])
@pytest.mark.parametrize("cin,cout,side", CONFIG5)
def test_sparse_int8_benchmark_size(plb, ctx, cin, cout, side, semi):
    """Full benchmark size (batch 256).  The oracle cannot run 2 GOP per case in seconds, so the whole output is
    checked through an exact integer identity and three images are checked element by element:
    * with unit scales, no bias and no activation the fp32 output IS the int32 accumulator (|acc| < 2^24), and
      sum over pixels of acc[n, oc, :] = sum_ic W[oc, ic] * (sum over pixels of x[n, ic, :])  -- exact in int64;
    * images 0, 100 and 255 of the int8-out layer (per-channel scales, bias, ReLU) equal the oracle bit for bit."""
    batch = 256
    hw = side * side
    wf = sparse_weights(7 * cin + cout, cout, cin, semi)
    wq, ws = O.quantize_per_channel(wf)
    enc = O.sparse_encode(wq, hw, semi=semi)
    args = (enc["nonzero_weights"], enc["oc_nonzeros"], enc["diffs"], enc["first_ic"], enc["flag_semi"])
    g = torch.Generator(device="cuda").manual_seed(cin + side)
    x = torch.randint(-127, 128, (batch, cin, side, side), dtype=torch.int8, device="cuda", generator=g)
    # 1. accumulators of the whole batch through the fp32-out kernel
    ident = plb.SparseConv(ctx, *args, cin=cin, cout=cout, in_hw=(side, side), wscale=np.ones(cout, np.float32),
                           in_scale=1.0)
    acc = ident.run(x)
    ctx.sync()
    got = acc.view(batch, cout, hw).to(torch.int64).sum(dim=2).cpu().numpy()
    xsum = x.view(batch, cin, hw).to(torch.int64).sum(dim=2).cpu().numpy()       # [batch, cin]
    want = xsum @ wq.astype(np.int64).T                                          # [batch, cout]
    assert np.array_equal(got, want), "pixel sums of the accumulators break the linear identity"
    del acc
    # 2. int8-out layer, three images against the oracle
    rng = np.random.default_rng(cin)
    bias = (rng.standard_normal(cout) * 0.1).astype(np.float32)
    in_s, out_s = 0.02, 0.06
    q = plb.SparseConv(ctx, *args, cin=cin, cout=cout, in_hw=(side, side), wscale=ws, in_scale=in_s, bias=bias,
                       act=O.ACT_RELU, out_scale=out_s).run(x)
    ctx.sync()
    for n in (0, 100, 255):
        xs = x[n:n + 1].cpu().numpy()
        a = O.conv_acc_i32(xs, wq[:, :, None, None])
        q_ref = O.epilogue(a, ws, in_s, bias, O.ACT_RELU, 0.0, out_scale=out_s)
        assert np.array_equal(q[n:n + 1].cpu().numpy(), q_ref), "image %d differs from the oracle" % n


def test_sparse_errors(plb, ctx):
    wq = np.zeros((4, 8), dtype=np.int8)
    wq[1, 3] = 5
    enc = O.sparse_encode(wq, 4)
    with pytest.raises(plb.PlbError):
        plb.SparseConv(ctx, enc["nonzero_weights"], enc["oc_nonzeros"], enc["diffs"], enc["first_ic"], 0,
                       cin=8, cout=4, in_hw=(2, 2), wscale=np.ones(3, np.float32), in_scale=1.0)
    bad = enc["diffs"].copy()
    bad[:] = 3  # not a multiple of the channel pitch
    with pytest.raises(plb.PlbError):
        plb.SparseConv(ctx, np.array([5, 6], np.int8), np.array([0, 2, 2, 2], np.uint32),
                       np.array([3, 3], np.int32), 3, 0, cin=8, cout=4, in_hw=(2, 2),
                       wscale=np.ones(4, np.float32), in_scale=1.0)
