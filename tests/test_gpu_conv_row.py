"""The 3x3 convolution with the column taps side by side (image widths 8 to 128,
channels in blocks of 32) at the edges of its tiles: one tile and many, rows that
do not fill a pair of pixel tiles, row neighbours inside a warp (W = 8 to 32) and
across warps (64, 128), weights resident and streamed, 32 and 64 channel tiles,
two inputs, more tiles than CTAs, both output types; against a float64
convolution of the same bf16 operands.  Tolerance: bf16 outputs round to 2^-9
relative, fp32 sums of up to 9 x 512 products of bf16 values to 1e-5 in the norm."""
import ctypes

import pytest
import torch
import torch.nn.functional as F

from test_gpu_conv import _conv, _input, _lib, _p, _rel, _weights

pytestmark = pytest.mark.gpu

CASES = [  # (n, H, W, [channels], cout)
    (1, 16, 8, [32], 32), (1, 16, 8, [64], 64), (3, 48, 8, [32, 32], 64), (1, 8, 16, [64], 32), (2, 24, 16, [256], 256),
    (1, 4, 32, [32], 64), (5, 20, 32, [128], 128), (3, 12, 32, [128, 256], 128), (1, 2, 64, [64], 64),
    (7, 6, 64, [64, 128], 64), (40, 64, 64, [64], 64), (2, 10, 64, [32], 96), (1, 1, 128, [32], 32),
    (2, 5, 128, [64], 64), (1, 7, 128, [160], 32), (3, 130, 128, [96, 32], 192), (1, 8, 16, [512], 64),
]


@pytest.mark.parametrize("case", CASES)
def test_conv_row(case):
    L = _lib()
    lib = L.lib()
    n, H, W, chans, cout = case
    gen = torch.Generator().manual_seed(H * 1000 + W + sum(chans) + cout)
    srcs = [(torch.randn((n, H, W, ch), generator=gen).to(torch.bfloat16).cuda(), ch, 0) for ch in chans]
    wb, w4 = _weights(cout, sum(chans), gen)
    bias = (0.1 * torch.randn(cout, generator=gen)).cuda()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    c = _conv(n, H, W, srcs, cout)
    s = L.stream_ptr()
    ref = F.conv2d(_input(srcs), w4, bias.double(), padding=1).permute(0, 2, 3, 1)
    # a guard after the outputs: the stores stay inside
    out = torch.full((n * H * W + 64, cout), 7.0, dtype=torch.bfloat16, device="cuda")
    outf = torch.full((n * H * W + 64, cout), 7.0, dtype=torch.float32, device="cuda")
    L.check(lib.agd_conv3x3_forward(ctypes.byref(c), _p(wb), _p(bias), 1, _p(out), None, _p(err), s))
    L.check(lib.agd_conv3x3_forward(ctypes.byref(c), _p(wb), None, 0, None, _p(outf), _p(err), s))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert float((out[n * H * W:].float() - 7.0).abs().max()) == 0.0
    assert float((outf[n * H * W:] - 7.0).abs().max()) == 0.0
    assert _rel(out[: n * H * W].double().view_as(ref), F.relu(ref)) < 4e-3
    assert _rel(outf[: n * H * W].double().view_as(ref), ref - bias.double()) < 1e-5
