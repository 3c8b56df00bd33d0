"""Which route a convolution's geometry takes, and its limits, as far as the library decides them on the host."""
import ctypes
import subprocess
import sys

import pytest


# (H, k, stride): the output side is (H - k) / stride + 1 = 0 or below
@pytest.mark.parametrize("H,k,stride", [(2, 3, 1), (1, 4, 1), (2, 4, 2), (1, 3, 2)])
def test_patch_gather_without_windows_is_an_empty_call(H, k, stride):
    """A window that does not fit makes an empty patch matrix: a call that does nothing, and no host fault (in a child
    process: a division by zero ends the process that makes it)."""
    side = int((H - k) / stride) + 1
    code = f"""
import ctypes
from bamboo_b200 import lib as L
i = ctypes.c_int
rc = L.load().bb_im2col_nhwc(ctypes.c_void_p(1 << 20), ctypes.c_void_p(1 << 21), i(3), i({H}), i({H}), i(8), i({k}), i({stride}), i(0),
                             i({side}), i({side}), ctypes.c_longlong({k * k * 8}), None)
assert rc == 0, (rc, L.load().bb_last_error())
"""
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, (done.returncode, done.stderr[-500:])


# (H, W, k, stride, pad): Ho or Wo = 1 by rounding towards zero, although the window is larger than the padded image
@pytest.mark.parametrize("H,W,k,stride,pad", [(2, 2, 4, 3, 0), (1, 9, 2, 2, 0), (9, 1, 2, 2, 0), (1, 1, 7, 8, 2)])
def test_overhanging_windows_are_gathered_into_a_patch_matrix(H, W, k, stride, pad):
    """The im2col loads have no box for them, so the layer's scratch has to hold the patch matrix."""
    from bamboo_b200 import lib as L
    N, cin, cout = 5, 64, 64
    fake = 1 << 20
    d = L.ConvDesc(N=N, H=H, W=W, Cin=cin, Cout=cout, k=k, stride=stride, pad=pad, relu=0, eps=1e-5, max_ctas=0, w=fake, gamma=fake, beta=fake)
    windows = N * (int((H + 2 * pad - k) / stride) + 1) * (int((W + 2 * pad - k) / stride) + 1)
    assert L.load().bb_conv_bn_scratch_bytes(ctypes.byref(d), 0, 0) >= windows * k * k * cin * 2


@pytest.mark.parametrize("pad", [1, 3])
def test_padded_pointwise_convolution_is_not_read_from_the_activations(pad):
    """A 1 x 1 convolution with padding has more output positions than input pixels: read as the patch matrix, the
    activation tensor would end too early."""
    from bamboo_b200 import lib as L
    N, side, cin, cout = 2, 5, 64, 64
    fake = 1 << 20
    d = L.ConvDesc(N=N, H=side, W=side, Cin=cin, Cout=cout, k=1, stride=1, pad=pad, relu=0, eps=1e-5, max_ctas=0, w=fake, gamma=fake, beta=fake)
    assert L.load().bb_conv_bn_scratch_bytes(ctypes.byref(d), 0, 0) >= N * (side + 2 * pad) ** 2 * cin * 2


# (images, side, channels in / out, window, kernels of a backward call with input gradient).  Batch norm takes three, each
# product one, a stored patch matrix one more in each direction
@pytest.mark.parametrize("N,hw,cin,cout,k,launches", [(28, 77, 8, 2048, 7, 7), (4, 79, 8, 1024, 7, 7), (32, 14, 16, 256, 3, 7), (5, 8, 256, 1024, 7, 6),
                                                      (6, 14, 256, 2048, 3, 6), (32, 56, 64, 64, 3, 5), (32, 28, 128, 128, 3, 5),
                                                      (9, 53, 256, 256, 3, 5), (16, 56, 32, 64, 5, 6)])
def test_input_gradient_is_gathered_where_that_is_quicker(N, hw, cin, cout, k, launches):
    """Few input channels leave most of a gathered product's columns empty (8 -> 2048, 7 x 7: 6.0 ms instead of 2.7), few
    pixels most of the machine: those keep the patch-gradient matrix."""
    from bamboo_b200 import lib as L
    fake = 1 << 20
    d = L.ConvDesc(N=N, H=hw, W=hw, Cin=cin, Cout=cout, k=k, stride=1, pad=(k - 1) // 2, relu=0, eps=1e-5, max_ctas=0, w=fake, gamma=fake, beta=fake)
    assert L.load().bb_conv_bn_launches(ctypes.byref(d), 1, 1) == launches


# (N, H, W, C, k): a row of windows, a row of pixels, and the rows of all images beyond 31 bits
@pytest.mark.parametrize("N,H,W,C,k", [(1, 64, (1 << 19) + 63, 8, 64), (1, 1, 1 << 22, 4096, 1), (1 << 16, 1 << 15, 1, 8, 1)])
@pytest.mark.parametrize("adjoint", [False, True])
def test_patch_kernels_accept_rows_beyond_31_bits(N, H, W, C, k, adjoint):
    """34 GB of patches fit a GPU.  Without one the launch fails, but the geometry is not refused."""
    import torch
    from bamboo_b200 import lib as L
    if torch.cuda.is_available():
        pytest.skip("the pointers are no device memory")
    i, fn = ctypes.c_int, L.load().bb_col2im_nhwc if adjoint else L.load().bb_im2col_nhwc
    rc = fn(ctypes.c_void_p(1 << 20), ctypes.c_void_p(1 << 21), i(N), i(H), i(W), i(C), i(k), i(1), i(0), i(H - k + 1), i(W - k + 1),
            ctypes.c_longlong(k * k * C), None)
    assert rc == -2, (rc, L.load().bb_last_error())
