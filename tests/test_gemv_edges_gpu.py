"""The GEMV kernels at the edges of their tiles and dispatch rules, against the CPU oracle's exact products: shares of a CTA of
one tile and of several, windows that end with the row and short of it, activations that no tensor copy can bring (K no
multiple of 64), gathered scales, and chunks with activations outside the range that FP16 holds after the usual
scaling (above 2^8, below 2^-24). Every row's bits are those it has alone."""
import pytest
import torch

from oracle import decode_gemv_oracle as oc
from oracle import workloads as wl
from tests import helpers as h

pytestmark = pytest.mark.gpu
MAKE = {"nvfp4": wl.cfg_nvfp4, "fp8": wl.cfg_fp8, "mxfp8": wl.cfg_mxfp8, "bf16": wl.cfg_bf16}


def gemv_abi(fmt, x, t):
    out = torch.full((x.shape[0], t[0].shape[0]), float("nan"), device="cuda")
    call = {"nvfp4": h.abi_nvfp4, "fp8": h.abi_fp8, "mxfp8": h.abi_fp8, "bf16": h.abi_bf16}[fmt]
    assert call(x, *t, out) == 0
    return out


@pytest.mark.parametrize("fmt,n,k", [
    ("nvfp4", 3, 32), ("nvfp4", 593, 1056), ("nvfp4", 4736, 512), ("nvfp4", 9473, 2080), ("nvfp4", 1200, 8192),
    ("fp8", 4736, 1024), ("fp8", 4737, 1040), ("fp8", 149, 4160), ("fp8", 600, 28672),
    ("mxfp8", 4737, 544), ("mxfp8", 1185, 2048), ("mxfp8", 700, 5024),
    ("bf16", 4736, 512), ("bf16", 4745, 520), ("bf16", 600, 8192)])
@pytest.mark.parametrize("wild", [False, True])
def test_tile_edges_and_wild_activations(fmt, n, k, wild):
    host = MAKE[fmt](n, k, seed=n + k)
    host = host if isinstance(host, tuple) else (host,)
    t = tuple(part.cuda() for part in host)
    g = torch.Generator().manual_seed(n)
    x = torch.randn(16, k, generator=g)
    if wild:
        x[1, k // 2] = 300.0
        x[2, 0] = 1e-9
        x[5, k - 1] = -2.0 ** 20
        x[11] *= 1e-12
        x[12, :: max(1, k // 7)] = 0.0
    x = x.to(torch.bfloat16)
    xd = x.cuda()
    batch = gemv_abi(fmt, xd, t)
    values = oc.values_of(fmt, host)
    assert oc.within_fp32_bound(batch.cpu(), x, values)
    for rows in (1, 2, 3, 4, 5, 8, 9):
        assert torch.equal(gemv_abi(fmt, xd[:rows].contiguous(), t), batch[:rows]), rows
    for row in (5, 11):
        assert torch.equal(gemv_abi(fmt, xd[row:row + 1].contiguous(), t)[0], batch[row]), row
