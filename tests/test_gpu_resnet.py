"""Channels-last ResNet stage kernels and layers against fp32 PyTorch (bf16 tolerance 2e-2):
patch gather and its adjoint, batch norm with batch statistics, pooling, one bottleneck block at
ResNet-152's own dimensions, and a small bottleneck ResNet through the public API (loss and every
gradient tensor against the oracle)."""
import ctypes
import os
import sys

import pytest
import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from oracle import resnet_ref  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = 2e-2


@pytest.fixture(scope="module")
def L():
    from bamboo_b200 import lib
    lib.load()
    return lib


def _rel(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-12)).item()


@pytest.mark.parametrize("k,stride,C,H", [(3, 1, 16, 14), (3, 2, 64, 15), (7, 2, 8, 32), (1, 2, 32, 8)])
def test_patch_gather_and_its_adjoint(L, k, stride, C, H):
    g = torch.Generator(device="cuda").manual_seed(1)
    N, W, pad = 2, H + 3, (k - 1) // 2
    x = torch.randn(N, H, W, C, device="cuda", generator=g).bfloat16()
    Ho, Wo = (H + 2 * pad - k) // stride + 1, (W + 2 * pad - k) // stride + 1
    col = torch.empty(N * Ho * Wo, k * k * C, dtype=torch.bfloat16, device="cuda")
    L.im2col(x, col, k, stride, pad, Ho, Wo)
    # torch.unfold orders columns (c, r, s); ours (r, s, c)
    ref = F.unfold(x.float().permute(0, 3, 1, 2), k, padding=pad, stride=stride)          # [N, C*k*k, Ho*Wo]
    ref = ref.view(N, C, k * k, Ho * Wo).permute(0, 3, 2, 1).reshape(N * Ho * Wo, k * k * C)
    assert torch.equal(col.float(), ref)                                                   # a gather: exact
    # adjoint: <im2col(x), d> == <x, col2im(d)> ; compare with fold
    d = torch.randn(N * Ho * Wo, k * k * C, device="cuda", generator=g).bfloat16()
    dx = torch.empty_like(x)
    L.col2im(d, dx, k, stride, pad, Ho, Wo)
    dref = d.float().view(N, Ho * Wo, k * k, C).permute(0, 3, 2, 1).reshape(N, C * k * k, Ho * Wo)
    want = F.fold(dref, (H, W), k, padding=pad, stride=stride).permute(0, 2, 3, 1)
    assert _rel(dx, want) <= 5e-3
    torch.cuda.synchronize()
    assert L.read_status() == 0


@pytest.mark.parametrize("rows,C,relu,res", [(1000, 64, True, True), (4096, 256, True, False), (333, 2048, False, False),
                                             (50000, 16, True, True)])
def test_batch_norm_forward_backward(L, rows, C, relu, res):
    g = torch.Generator(device="cuda").manual_seed(2)
    y = (torch.randn(rows, C, device="cuda", generator=g) * 2 + 0.5).bfloat16()
    gamma = (1 + 0.2 * torch.randn(C, device="cuda", generator=g)).bfloat16()
    beta = (0.1 * torch.randn(C, device="cuda", generator=g)).bfloat16()
    r = torch.randn(rows, C, device="cuda", generator=g).bfloat16() if res else None
    dz = torch.randn(rows, C, device="cuda", generator=g).bfloat16()
    mean, rstd = torch.empty(C, device="cuda"), torch.empty(C, device="cuda")
    L.bn_stats(y, mean, rstd, 1e-5)
    z = torch.empty_like(y)
    L.bn_apply(y, mean, rstd, gamma, beta, r, z, relu)
    yf = y.float().requires_grad_(True)
    gf, bf_ = gamma.float().requires_grad_(True), beta.float().requires_grad_(True)
    rf = r.float().requires_grad_(True) if res else None
    zr = F.batch_norm(yf, None, None, gf, bf_, training=True, eps=1e-5)
    if res:
        zr = zr + rf
    if relu:
        zr = F.relu(zr)
    assert (mean - yf.detach().mean(0)).abs().max().item() <= 1e-3
    assert _rel(z, zr.detach()) <= TOL
    # backward uses the kernel's own z for the ReLU mask; elements within bf16 rounding of 0 may differ
    zr.backward(dz.float())
    dy = torch.empty_like(y)
    dres = torch.empty_like(y) if res else None
    dg, db = torch.zeros(C, device="cuda"), torch.zeros(C, device="cuda")
    L.bn_bwd(dz, z, y, mean, rstd, gamma, dy, dres, dg, db, relu)
    assert _rel(dy, yf.grad) <= TOL
    assert _rel(dg, gf.grad) <= TOL and _rel(db, bf_.grad) <= TOL
    if res:
        assert _rel(dres, rf.grad) <= TOL
    torch.cuda.synchronize()
    assert L.read_status() == 0


def test_pooling(L):
    g = torch.Generator(device="cuda").manual_seed(3)
    x = F.relu(torch.randn(3, 17, 22, 32, device="cuda", generator=g)).bfloat16()          # many exact ties at 0
    from bamboo_b200 import resnet
    xr = x.float().permute(0, 3, 1, 2).requires_grad_(True)
    want = F.max_pool2d(xr, 3, 2, 1)
    xs = x.clone().requires_grad_(True)
    got = resnet._MaxPoolFn.apply(xs)
    assert torch.equal(got.float(), want.detach().permute(0, 2, 3, 1))
    d = torch.randn_like(got)
    got.backward(d)
    want.backward(d.float().permute(0, 3, 1, 2))
    assert _rel(xs.grad, xr.grad.permute(0, 2, 3, 1)) <= 5e-3
    x2 = torch.randn(4, 7, 7, 2048, device="cuda", generator=g).bfloat16().requires_grad_(True)
    a = resnet._AvgPoolFn.apply(x2)
    assert _rel(a, x2.detach().float().mean((1, 2))) <= 5e-3
    a.backward(torch.ones_like(a))
    assert _rel(x2.grad, torch.full_like(x2, 1 / 49.0)) <= 5e-3


@pytest.mark.parametrize("cin,cout,k,stride,hw", [(8, 64, 7, 2, 64), (64, 64, 3, 1, 28), (64, 128, 3, 2, 28), (256, 512, 1, 2, 14),
                                                  (64, 256, 1, 1, 28)])
def test_conv_bn_layer_without_relu(L, cin, cout, k, stride, hw):
    """Convolution + batch norm with no ReLU behind it (no activation mask that bf16 rounding could
    flip): output, input gradient, weight gradient and batch-norm gradients at 2e-2."""
    from bamboo_b200 import resnet
    from bamboo_b200.arena import ParamArena
    m = resnet.ConvBN(cin, cout, k, stride=stride, relu=False, generator=torch.Generator().manual_seed(9))
    w_ref = m.weight.detach().float().view(cout, k, k, cin).permute(0, 3, 1, 2).contiguous().cuda().requires_grad_(True)
    g_ref = torch.ones(cout, device="cuda", requires_grad=True)
    b_ref = torch.zeros(cout, device="cuda", requires_grad=True)
    ParamArena(list(m.parameters()), torch.device("cuda"), torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(4, hw, hw, cin, device="cuda", generator=g).bfloat16().requires_grad_(True)
    out = m(x)
    xr = x.detach().float().permute(0, 3, 1, 2).requires_grad_(True)
    y = F.conv2d(xr, w_ref, None, stride=stride, padding=(k - 1) // 2)
    want = F.batch_norm(y, None, None, g_ref, b_ref, training=True, eps=1e-5)
    assert _rel(out, want.detach().permute(0, 2, 3, 1)) <= TOL
    d = torch.randn_like(out)
    out.backward(d)
    want.backward(d.float().permute(0, 3, 1, 2))
    errs = {"dx": _rel(x.grad, xr.grad.permute(0, 2, 3, 1)),
            "dW": _rel(m.weight.main_grad.view(cout, k, k, cin).permute(0, 3, 1, 2), w_ref.grad),
            "dgamma": _rel(m.bn_weight.main_grad, g_ref.grad), "dbeta": _rel(m.bn_bias.main_grad, b_ref.grad)}
    print(f"conv {cin}->{cout} k{k} s{stride}: {errs}")
    assert max(errs.values()) <= TOL, errs
    torch.cuda.synchronize()
    assert L.read_status() == 0


# rows: fewer than one per thread group, around a thread's four rows in flight, many; channels: the narrowest (one
# 16-byte chunk), ordinary, the widest (a row per block)
@pytest.mark.parametrize("rows,C", [(1, 8), (255, 8), (3, 64), (129, 64), (1025, 256), (7, 2048), (50, 2048), (40000, 64)])
def test_batch_norm_backward_mask_from_y_equals_mask_from_z(L, rows, C):
    """bb_conv_bn_bwd_affine takes the ReLU mask from y: the same values as the general entry point, which reads the
    stored output, in every bit (same kernels, same order of sums), a channel that
    is zero throughout included."""
    from bamboo_b200 import resnet
    from bamboo_b200.arena import ParamArena
    m = resnet.ConvBN(8, C, 1, relu=True, generator=torch.Generator().manual_seed(5))
    with torch.no_grad():
        m.bn_weight.copy_(torch.linspace(-1.0, 1.5, C)); m.bn_bias.copy_(torch.linspace(0.5, -0.5, C))
        m.bn_weight[0] = 0.0; m.bn_bias[0] = 0.0                  # z = 0 everywhere: nothing passes
    ParamArena(list(m.parameters()), torch.device("cuda"), torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(1, 1, rows, 8, device="cuda", generator=g).bfloat16()
    x[..., 0] = 0.0
    d = resnet._conv_desc(m, 1, 1, rows, 8, True)
    y, z = torch.empty(rows, C, dtype=torch.bfloat16, device="cuda"), torch.empty(1, 1, rows, C, dtype=torch.bfloat16, device="cuda")
    stats = torch.empty(4, C, device="cuda")
    L.conv_bn_fwd(d, x, None, y, z, stats[0], stats[1], torch.empty(max(d._fwd_scratch, 16), dtype=torch.uint8, device="cuda"), stats[2:])
    dz = torch.randn(1, 1, rows, C, device="cuda", generator=g).bfloat16()
    out = []
    for residual in (True, False):
        for p in (m.weight, m.bn_weight, m.bn_bias):
            p.main_grad.zero_()
        dx = torch.empty_like(x)
        scratch = torch.zeros(d._bwd_scratch[1], dtype=torch.uint8, device="cuda")
        L.conv_bn_bwd(d, x, y, z, stats[0], stats[1], dz, dx, None, scratch, residual=residual, affine=None if residual else stats[2:])
        out.append((scratch[:rows * C * 2].view(torch.bfloat16).clone(), m.bn_weight.main_grad.clone(), m.bn_bias.main_grad.clone()))
    for a, b in zip(*out):
        assert torch.equal(a.nan_to_num(), b.nan_to_num()) and torch.equal(a.isnan(), b.isnan())
    # (the values themselves, against fp32: masked gradient through batch norm)
    yf = y.float().requires_grad_(True)
    if rows > 3:
        ga, be = m.bn_weight.detach().float().requires_grad_(True), m.bn_bias.detach().float().requires_grad_(True)
        zf = F.batch_norm(yf, None, None, ga, be, training=True, eps=m.eps)
        zf.backward(torch.where(z.view(rows, C) > 0, dz.view(rows, C).float(), torch.zeros((), device="cuda")))
        assert _rel(out[1][0].view(rows, C), yf.grad) <= TOL and _rel(out[1][1], ga.grad) <= TOL


@pytest.mark.parametrize("residual", [False, True])
def test_relu_mask_is_that_of_the_forward_pass(L, residual):
    """Gain and bias that change between a layer's forward and backward pass (an update while a micro-batch is in flight)
    do not move the ReLU mask: the bias gradient stays the sum of dz over the positive outputs."""
    from bamboo_b200 import resnet
    from bamboo_b200.arena import ParamArena
    C, rows = 64, 300
    m = resnet.ConvBN(16, C, 1, relu=True, generator=torch.Generator().manual_seed(5))
    ParamArena(list(m.parameters()), torch.device("cuda"), torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn(1, 1, rows, 16, device="cuda", generator=g).bfloat16().requires_grad_(True)
    res = torch.randn(1, 1, rows, C, device="cuda", generator=g).bfloat16() if residual else None
    z = m(x, res)
    with torch.no_grad():
        m.bn_bias.add_(1.0)
        m.bn_weight.mul_(-1.0)
    dz = torch.randint(-8, 9, z.shape, device="cuda", generator=g).bfloat16()
    z.backward(dz)
    # whole numbers below 2^24: the sums are exact
    want = torch.where(z > 0, dz.float(), torch.zeros((), device="cuda")).sum((0, 1, 2))
    assert torch.equal(m.bn_bias.main_grad.view(-1), want)


# (channels in / out, window, stride, image side): reductions of one to several 64-channel blocks, output rows that no
# 128-row tile divides, images smaller than the window, an even window (asymmetric turned padding), both tile widths (and
# CTA pairs for the weight gradient of 128 -> 512; the other two products: next test), channel counts that only one direction
# can gather
@pytest.mark.parametrize("cin,cout,k,stride,hw", [(64, 64, 3, 1, 1), (64, 64, 3, 1, 2), (64, 16, 3, 1, 5), (192, 64, 3, 1, 11),
                                                  (64, 64, 2, 1, 6), (64, 64, 7, 1, 9), (64, 128, 7, 2, 13), (128, 64, 3, 2, 15),
                                                  (64, 128, 1, 2, 7), (256, 256, 3, 1, 14), (256, 256, 3, 2, 29), (512, 128, 3, 1, 7),
                                                  (8, 64, 3, 1, 10), (64, 8, 3, 1, 9), (128, 512, 3, 1, 35)])
def test_convolution_with_gathered_patches(L, cin, cout, k, stride, hw):
    check_convolution(L, cin, cout, k, stride, hw, 9)


# enough images that the input gradient is gathered as well: images smaller than the window, an even window, rows that no tile
# divides, fewer input channels than a tile has columns, one of two tile widths
@pytest.mark.parametrize("cin,cout,k,hw,N", [(64, 64, 3, 1, 30001), (64, 64, 3, 2, 7003), (32, 64, 5, 5, 2001), (192, 64, 3, 11, 201),
                                             (64, 64, 2, 6, 701), (64, 64, 7, 9, 301), (512, 128, 3, 7, 211)])
def test_convolution_with_gathered_input_gradient(L, cin, cout, k, hw, N):
    d = check_convolution(L, cin, cout, k, 1, hw, N)
    assert L.load().bb_conv_bn_launches(ctypes.byref(d), 1, 1) == (5 if cin % 64 == 0 else 6)


def check_convolution(L, cin, cout, k, stride, hw, N):
    """The convolution alone (what the layer feeds into batch norm, and the gradients that come out of it) against
    conv2d in fp32 on the same bf16 operands.  One bf16 rounding of each result: 2^-9 of the value, so 4e-3 in the
    2-norm; the weight gradient is summed and kept in fp32 (1e-4: order of the sums)."""
    from bamboo_b200 import resnet
    from bamboo_b200.arena import ParamArena
    m = resnet.ConvBN(cin, cout, k, stride=stride, relu=False, generator=torch.Generator().manual_seed(11))
    ParamArena(list(m.parameters()), torch.device("cuda"), torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(12)
    x = torch.randn(N, hw, hw, cin, device="cuda", generator=g).bfloat16()
    ho = (hw + 2 * m.pad - k) // stride + 1
    P = N * ho * ho
    y = torch.empty(P, cout, dtype=torch.bfloat16, device="cuda")
    z = torch.empty(N, ho, ho, cout, dtype=torch.bfloat16, device="cuda")
    stats = torch.empty(2, cout, device="cuda")
    d = resnet._conv_desc(m, N, hw, hw, cin, True)
    scratch = torch.empty(max(d._fwd_scratch, 16), dtype=torch.uint8, device="cuda")
    L.conv_bn_fwd(d, x, None, y, z, stats[0], stats[1], scratch)
    w = m.weight.detach().float().view(cout, k, k, cin).permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    xr = x.float().permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    with torch.backends.cudnn.flags(allow_tf32=False):
        want = F.conv2d(xr, w, None, stride=stride, padding=m.pad)
        assert _rel(y.view(N, ho, ho, cout), want.detach().permute(0, 2, 3, 1)) <= 4e-3
        dz = torch.randn(N, ho, ho, cout, device="cuda", generator=g).bfloat16()
        dx = torch.empty_like(x)
        bwd = torch.empty(d._bwd_scratch[1], dtype=torch.uint8, device="cuda")
        L.conv_bn_bwd(d, x, y, z, stats[0], stats[1], dz, dx, None, bwd)
        dy = bwd[:P * cout * 2].view(torch.bfloat16).view(N, ho, ho, cout)      # the scratch starts with dy
        want.backward(dy.float().permute(0, 3, 1, 2).contiguous())
    # a strided layer rounds every tap's contribution to bf16 before they are summed: k * k roundings instead of one
    assert _rel(dx, xr.grad.permute(0, 2, 3, 1)) <= 8e-3
    assert _rel(m.weight.main_grad.view(cout, k, k, cin).permute(0, 3, 1, 2), w.grad) <= 1e-4
    torch.cuda.synchronize()
    assert L.read_status() == 0
    return d


def test_convolution_with_gathered_patches_on_cta_pairs(L):
    """256 -> 256, 3 x 3, nine images of 53 x 53: forward product and input gradient are planned to CTA pairs (two waves of
    99 tiles of 256 x 256 are expected to take 39.6 us, 128 x 256 tiles 40.4, 128 x 128 44), seen in the captured call's cluster sizes."""
    from bamboo_b200 import resnet
    from bamboo_b200.arena import ParamArena
    from test_gpu_overlap import captured, kernel_nodes
    m = resnet.ConvBN(256, 256, 3, relu=False, generator=torch.Generator().manual_seed(11))
    ParamArena(list(m.parameters()), torch.device("cuda"), torch.bfloat16)
    x = torch.randn(9, 53, 53, 256, device="cuda").bfloat16().requires_grad_(True)
    dz = torch.ones_like(m(x))
    graph, handle, rt = captured(lambda: torch.autograd.grad(m(x), x, dz))
    clusters = [rt.cudaGraphKernelNodeGetAttribute(n, rt.cudaLaunchAttributeID.cudaLaunchAttributeClusterDimension)[1].clusterDim.x
                for n in kernel_nodes(handle, rt)]
    assert sum(c == 2 for c in clusters) >= 2, clusters
    check_convolution(L, 256, 256, 3, 1, 53, 9)


def _block_params(blk, prefix):
    out = {}
    for name in ("conv1", "conv2", "conv3", "down"):
        m = getattr(blk, name)
        if m is None:
            continue
        cout = m.weight.shape[0]
        cin = m.weight.shape[1] // (m.k * m.k)
        out[f"{prefix}.{name}.weight"] = m.weight.detach().float().view(cout, m.k, m.k, cin).permute(0, 3, 1, 2).contiguous()
        out[f"{prefix}.{name}.bn_weight"] = m.bn_weight.detach().float().clone()
        out[f"{prefix}.{name}.bn_bias"] = m.bn_bias.detach().float().clone()
    return out


@pytest.mark.parametrize("cin,mid,stride,down,hw", [(256, 64, 1, False, 56), (256, 128, 2, True, 56), (1024, 256, 1, False, 14)])
def test_bottleneck_at_resnet152_dimensions(L, cin, mid, stride, down, hw):
    """One block with ResNet-152's channel counts and feature-map sizes against the same block in
    fp32 PyTorch: output and input gradient."""
    from bamboo_b200 import resnet
    from bamboo_b200.arena import ParamArena
    blk = resnet.Bottleneck(cin, mid, stride=stride, downsample=down, seed=5)
    P = {k: v.cuda().requires_grad_(True) for k, v in _block_params(blk, "1").items()}
    ParamArena(list(blk.parameters()), torch.device("cuda"), torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(4, hw, hw, cin, device="cuda", generator=g).bfloat16().requires_grad_(True)
    out = blk(x)
    xr = x.detach().float().permute(0, 3, 1, 2).requires_grad_(True)
    identity = resnet_ref._conv_bn(P, "1.down", xr, stride, 1, False) if down else xr
    y = resnet_ref._conv_bn(P, "1.conv1", xr, 1, 1, True)
    y = resnet_ref._conv_bn(P, "1.conv2", y, stride, 3, True)
    want = resnet_ref._conv_bn(P, "1.conv3", y, 1, 1, True, residual=identity)
    assert _rel(out, want.detach().permute(0, 2, 3, 1)) <= TOL
    d = torch.randn_like(out)
    out.backward(d)
    want.backward(d.float().permute(0, 3, 1, 2))
    # Gradients behind three ReLUs: wherever a pre-activation lies within bf16 rounding of zero the
    # mask differs from the fp32 reference's, and a fraction f of flipped elements costs about
    # sqrt(f) in relative L2 error (f ~ 0.3 % per ReLU here; with a random upstream gradient the
    # weight-gradient sums do not average it out).  Yardstick: the same block in bf16 on torch's
    # own kernels; the CUDA layers must be as close to fp32 as that pipeline (factor 1.5).
    P16 = {k: v.detach().bfloat16().requires_grad_(True) for k, v in P.items()}
    x16 = x.detach().permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    id16 = resnet_ref._conv_bn(P16, "1.down", x16, stride, 1, False) if down else x16
    y16 = resnet_ref._conv_bn(P16, "1.conv1", x16, 1, 1, True)
    y16 = resnet_ref._conv_bn(P16, "1.conv2", y16, stride, 3, True)
    resnet_ref._conv_bn(P16, "1.conv3", y16, 1, 1, True, residual=id16).backward(d.permute(0, 3, 1, 2))
    m = blk.conv2
    ours = {"dx": x.grad, "dW": m.weight.main_grad.view(mid, 3, 3, mid).permute(0, 3, 1, 2), "dgamma": blk.conv3.bn_weight.main_grad}
    bf16 = {"dx": x16.grad.permute(0, 2, 3, 1), "dW": P16["1.conv2.weight"].grad, "dgamma": P16["1.conv3.bn_weight"].grad}
    fp32 = {"dx": xr.grad.permute(0, 2, 3, 1), "dW": P["1.conv2.weight"].grad, "dgamma": P["1.conv3.bn_weight"].grad}
    for key in ours:
        e_o, e_b = _rel(ours[key], fp32[key]), _rel(bf16[key], fp32[key])
        print(f"bottleneck {cin}/{mid}/s{stride} {key}: ours {e_o:.4f}  torch-bf16 {e_b:.4f}")
        assert e_o <= max(1.5 * e_b, TOL), (key, e_o, e_b)
    torch.cuda.synchronize()
    assert L.read_status() == 0


def test_small_resnet_training_steps_match_oracle():
    """Bottleneck ResNet (one block per stage, width 64, 128 x 128 images, 40 classes) through
    PipelineModule / initialize / train_batch.  The loss must match the fp32 oracle at 2e-2.  For the
    gradients an fp32 reference alone is the wrong yardstick in a ReLU / max-pool network: wherever
    a pre-activation lies within bf16 rounding of zero (or two window entries within rounding of
    each other) the mask differs, and every such flip is a full-size element-wise error that the
    batch-norm backward passes spread further.  So the same oracle is also run in bf16 on the GPU
    (torch / cuDNN kernels, rounding at the same points): the CUDA layers must be as close to the
    fp32 oracle as that bf16 pipeline is (factor 1.5), tensor by tensor and for the whole model."""
    from bamboo_b200 import api, resnet
    from bamboo_b200.module import PipelineModule
    os.environ["BAMBOO_QUIET"] = "1"
    blocks, width, classes, size = (1, 1, 1, 1), 64, 40, 128
    mb, gas, lr = 8, 2, 1e-3
    model = PipelineModule(resnet.resnet_layer_specs(blocks, classes, width, seed=0), num_stages=1,
                           loss_fn=resnet.resnet_loss(classes), partition_method="uniform")
    engine, *_ = api.initialize(model=model, config={
        "train_micro_batch_size_per_gpu": mb, "gradient_accumulation_steps": gas, "bf16": {"enabled": True},
        "optimizer": {"type": "Adam", "params": {"lr": lr}}})
    engine.capture_grads = True
    ref = resnet_ref.RefTrainer(blocks, classes, width, seed=0, lr=lr, micro_batches=gas)
    arena = engine.arenas[0]
    names = [n for n, _ in engine.module.get_named_param(0)]

    def ours_layout(name, g):
        if name.endswith(".weight") and g.dim() == 4:
            co, ci, k, _ = g.shape
            return g.permute(0, 2, 3, 1).reshape(co, k * k * ci)
        return g

    for step, batches in enumerate(resnet_ref.synthetic_batches(mb, gas, 2, size=size, classes=classes, seed=1)):
        if step > 0:
            # after an Adam update from gradients that differ at the bf16 level the two weight sets are
            # no longer the same point (Adam normalises the step size): only the loss is compared
            want = ref.train_batch(batches)
            got = float(engine.train_batch(data_iter=iter([(resnet_ref.to_channels_last_8(x), y) for x, y in batches])))
            assert got == pytest.approx(want, rel=TOL)
            continue
        # the bf16 torch pipeline from the oracle's current weights
        P16 = {k: v.detach().cuda().bfloat16().requires_grad_(True) for k, v in ref.P.items()}
        for images, labels in batches:
            (resnet_ref.forward_loss(P16, images.cuda().bfloat16(), labels.cuda(), blocks) / gas).backward()
        want = ref.train_batch(batches)
        got = float(engine.train_batch(data_iter=iter([(resnet_ref.to_channels_last_8(x), y) for x, y in batches])))
        assert got == pytest.approx(want, rel=TOL)
        flat = engine.last_grads[0].cpu()
        n_o = n_b = den = 0.0
        for name, (i, off, n) in zip(names, arena.named_slices()):
            g_ref = ours_layout(name, ref.last_grads[name])
            g_b16 = ours_layout(name, P16[name].grad.float().cpu()) if P16[name].grad is not None else torch.zeros_like(g_ref)
            g_got = flat[off:off + n].view(arena.params[i].shape)
            assert g_got.shape == g_ref.shape, name
            e_o, e_b = _rel(g_got, g_ref), _rel(g_b16, g_ref)
            n_o += float((g_got - g_ref).double().pow(2).sum()); n_b += float((g_b16 - g_ref).double().pow(2).sum())
            den += float(g_ref.double().pow(2).sum())
            print(f"   {name}: ours {e_o:.4f}  torch-bf16 {e_b:.4f}")
            assert e_o <= max(1.5 * e_b, 2 * TOL), (name, e_o, e_b)
        e_o, e_b = (n_o / den) ** 0.5, (n_b / den) ** 0.5
        print(f"small resnet step: loss {got:.5f} vs {want:.5f}; gradients vs fp32: ours {e_o:.4f}, torch bf16 {e_b:.4f}")
        assert e_o <= max(1.5 * e_b, TOL)
    from bamboo_b200 import lib
    torch.cuda.synchronize()
    assert lib.read_status() == 0


# (k, stride, pad): one to four taps along a dimension at strides 1 and 2, and what stays with the general kernel
@pytest.mark.parametrize("k,stride,pad", [(1, 2, 0), (2, 2, 0), (3, 2, 1), (4, 2, 1), (5, 2, 2), (7, 2, 3), (1, 1, 0), (2, 1, 1), (3, 1, 1),
                                          (4, 1, 0), (5, 1, 2), (3, 3, 1), (9, 2, 4), (1, 2, 1)])
@pytest.mark.parametrize("n,size,c", [(1, 9, 8), (3, 14, 24), (2, 33, 64)])
def test_patch_adjoint_sums_every_tap_once(L, k, stride, pad, n, size, c):
    """Whole numbers whose sums (at most 81 of magnitude 3) are exact in bf16's eight bits: equal to the fold bit for bit."""
    torch.manual_seed(9)
    out = (size + 2 * pad - k) // stride + 1
    cols = torch.randint(-3, 4, (n, out, out, k * k, c), device="cuda")
    col = torch.full((n * out * out, k * k * c + 8), 5.0, device="cuda", dtype=torch.bfloat16)
    col[:, :k * k * c] = cols.reshape(n * out * out, -1).bfloat16()
    dx = torch.empty(n, size, size, c, device="cuda", dtype=torch.bfloat16)
    L.col2im(col[:, :k * k * c], dx, k, stride, pad, out, out)
    folded = F.fold(cols.permute(0, 4, 3, 1, 2).reshape(n, c * k * k, out * out).float(), size, k, padding=pad, stride=stride)
    assert torch.equal(dx.float(), folded.permute(0, 2, 3, 1))


# few pixels and a reduction of k * k * Cout: the gathered input gradient is split over clusters; the last on a budget, which keeps it whole
@pytest.mark.parametrize("n,hw,cin,cout,k,max_ctas,kernels", [(32, 7, 64, 64, 7, 0, 5), (1, 28, 512, 256, 7, 0, 5), (8, 14, 128, 256, 5, 0, 5),
                                                              (6, 14, 256, 2048, 3, 0, 6), (32, 7, 64, 64, 7, -1, 6)])
def test_input_gradient_is_priced_as_it_is_planned(L, monkeypatch, n, hw, cin, cout, k, max_ctas, kernels):
    monkeypatch.setattr(L, "GEMM_MAX_CTAS", max_ctas)
    d = check_convolution(L, cin, cout, k, 1, hw, n)
    assert L._conv_launches(d, 1, 1) == kernels


@pytest.mark.parametrize("n,hw,cin,cout,k", [(32, 7, 512, 512, 3), (5, 9, 64, 64, 7)])
def test_gathered_products_split_inside_a_cluster(L, n, hw, cin, cout, k):
    """Few pixels and a long reduction: forward product and, where it is gathered, input gradient as clusters (kernels of 608 threads)."""
    from bamboo_b200 import resnet
    from bamboo_b200.arena import ParamArena
    from cuda.bindings import driver
    from test_gpu_overlap import captured, kernel_nodes
    d = check_convolution(L, cin, cout, k, 1, hw, n)
    m = resnet.ConvBN(cin, cout, k, relu=False, generator=torch.Generator().manual_seed(11))
    ParamArena(list(m.parameters()), torch.device("cuda"), torch.bfloat16)
    x = torch.randn(n, hw, hw, cin, device="cuda").bfloat16().requires_grad_(True)
    dz = torch.ones_like(m(x))
    graph, handle, rt = captured(lambda: torch.autograd.grad(m(x), x, dz))
    threads = [driver.cuGraphKernelNodeGetParams(driver.CUgraphNode(int(v)))[1].blockDimX for v in kernel_nodes(handle, rt)]
    assert threads.count(608) >= (2 if L._conv_launches(d, 1, 1) == 5 else 1), threads
