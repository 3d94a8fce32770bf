"""The activation quantizers at the edges of their kernels' tiles, bit for bit against the CPU oracle: rows held in registers
(up to 4096 values, or 32768 in batches of up to 256 rows; 32 values to a thread), 32 x 512 tiles of NVFP4 blocks."""
import ctypes

import numpy as np
import pytest
import torch

from crit_kernels_b200 import cabi
from oracle import decode_gemv_oracle as oc
from oracle import quantize_oracle as qo

pytestmark = pytest.mark.gpu


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def inputs(m, k):
    g = torch.Generator().manual_seed(m * 7 + k)
    x = torch.randn(m, k, generator=g) * torch.exp2(torch.randint(-9, 6, (m, 1), generator=g).float())
    x[m // 2, : k // 3] = 0
    return x.to(torch.bfloat16)


@pytest.mark.parametrize("m,k", [(1, 8), (3, 248), (9, 264), (33, 1016), (257, 1032), (5, 4096), (300, 4096), (300, 4104),
                                 (256, 4104), (257, 5120), (2, 32768), (2, 32776), (1200, 1024)])
def test_fp8_rows_at_the_edges_of_their_kernels(m, k):
    x = inputs(m, k)
    x[0, k - 1] = -448.0
    xd = x.cuda()
    q = torch.full((m, k), 0x55, dtype=torch.uint8, device="cuda")
    scale = torch.empty(m, device="cuda")
    assert cabi.load().dg_enqueue_quantize_fp8_rows(_ptr(xd), k, m, k, _ptr(q), k, _ptr(scale), None) == 0
    torch.cuda.synchronize()
    want_q, want_scale = qo.fp8_rows(x)
    assert np.array_equal(scale.cpu().numpy().view(np.uint32), want_scale.view(np.uint32))
    assert np.array_equal(q.cpu().numpy(), want_q)


@pytest.mark.parametrize("m,k", [(1, 16), (8, 496), (31, 512), (33, 528), (127, 1040), (129, 560), (97, 64)])
@pytest.mark.parametrize("offset", [0, 4])                         # of the tiled scales from 16 bytes
def test_nvfp4_at_the_edges_of_its_tiles(m, k, offset):
    x = inputs(m, k)
    xd = x.cuda()
    codes = torch.full((m, k // 2), 0x55, dtype=torch.uint8, device="cuda")
    buffer = torch.full((oc.blocked_numel(m, k) + offset,), 0x55, dtype=torch.uint8, device="cuda")
    scales = buffer[offset:]
    g, r = ctypes.c_float(300.0), ctypes.c_float(np.float32(1.0) / np.float32(300.0))
    assert cabi.load().dg_enqueue_quantize_nvfp4(_ptr(xd), k, m, k, g, r, _ptr(codes), _ptr(scales), None) == 0
    torch.cuda.synchronize()
    want_codes, want_blocked = qo.nvfp4_blocked(x, 300.0)
    assert np.array_equal(codes.cpu().numpy(), want_codes)
    assert np.array_equal(scales.cpu().numpy(), want_blocked)
    assert bool((buffer[:offset] == 0x55).all())


@pytest.mark.parametrize("large", [7.6e5, 8.1e5, 9.9e7, 1.01e8, 3e38])        # about scales of 2^17 and values of 1e8 the division changes its way
@pytest.mark.parametrize("input_scale", [2688.0 / 8.0, 2e-5, 1e25])
def test_nvfp4_blocks_of_tiny_values_beside_large_ones(large, input_scale):
    """Quotients that FP32 rounds to zero, negative ones and negative zeros among them, beside a block's largest value."""
    g = torch.Generator().manual_seed(5)
    x = torch.randn(40, 1024, generator=g) * torch.exp2(torch.randint(-149, -80, (40, 1024), generator=g).float())
    x[:, 3::16] = -0.0
    x[::2, 7::16] = large
    x[1::4, 9::16] = -large * torch.rand(10, 64, generator=g)
    x = x.to(torch.bfloat16)
    codes = torch.full((40, 512), 0x55, dtype=torch.uint8, device="cuda")
    scales = torch.full((oc.blocked_numel(40, 1024),), 0x55, dtype=torch.uint8, device="cuda")
    s, r = np.float32(input_scale), np.float32(1.0) / np.float32(input_scale)
    xd = x.cuda()
    assert cabi.load().dg_enqueue_quantize_nvfp4(_ptr(xd), 1024, 40, 1024, ctypes.c_float(s), ctypes.c_float(r), _ptr(codes),
                                                 _ptr(scales), None) == 0
    torch.cuda.synchronize()
    want_codes, want_blocked = qo.nvfp4_blocked(x, input_scale)
    assert np.array_equal(codes.cpu().numpy(), want_codes)
    assert np.array_equal(scales.cpu().numpy(), want_blocked)
