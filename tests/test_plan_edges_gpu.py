"""Launches at the edges of the planner's rules: a CTA's range that is one tile only in stages of one step, that has two stages of two
steps instead of three, and windows of activations that up to four rows share with the kernel for five to eight, copied ones in
one tile and in several. The bits of a row are those it has among sixteen, the values the CPU oracle's."""
import pytest
import torch

from oracle import decode_gemv_oracle as oc
from oracle import workloads as wl
from tests import helpers as h

pytestmark = pytest.mark.gpu
MAKE = {"nvfp4": wl.cfg_nvfp4, "fp8": wl.cfg_fp8, "mxfp8": wl.cfg_mxfp8}


@pytest.mark.parametrize("fmt,n,k", [
    ("nvfp4", 148 * 56, 2048), ("nvfp4", 148 * 64 - 5, 8192), ("nvfp4", 148 * 41, 15360), ("nvfp4", 148 * 56 - 1, 16384),
    ("nvfp4", 1300, 28672), ("nvfp4", 148 * 20, 1056), ("nvfp4", 148 * 70, 1056), ("fp8", 148 * 56, 4096), ("fp8", 148 * 50, 8192),
    ("fp8", 148 * 20, 528), ("fp8", 148 * 70, 528), ("mxfp8", 148 * 56, 8192),
    # small NVFP4 launches (up to 72 matrix rows times steps) and what is just none; ranges in which up to four rows have windows or not
    ("nvfp4", 1, 64), ("nvfp4", 149, 1024), ("nvfp4", 148 * 8, 4096), ("nvfp4", 148 * 8 + 1, 4096), ("nvfp4", 148 * 24, 3072),
    ("nvfp4", 148 * 24 + 1, 3072), ("nvfp4", 148 * 8, 9216), ("nvfp4", 148 * 32, 2048), ("nvfp4", 148 * 48, 1024), ("nvfp4", 148 * 48 + 1, 1024),
    ("fp8", 148 * 32, 4096), ("fp8", 148 * 32 + 1, 4096), ("fp8", 148 * 32, 4160)])
def test_launches_at_the_edges_of_the_plans(fmt, n, k):
    host = MAKE[fmt](n, k, seed=n + k)
    t = tuple(part.cuda() for part in host)
    x = torch.randn(16, k, generator=torch.Generator().manual_seed(k))
    x[2, k // 3] = 300.0
    x = x.to(torch.bfloat16)
    xd = x.cuda()
    batch = h.run(fmt, xd, t, torch.full((16, n), float("nan"), device="cuda"))
    picked = torch.randperm(n, generator=torch.Generator().manual_seed(n))[:256].sort().values
    part = tuple(a[picked] for a in host)
    assert oc.within_fp32_bound(batch[:, picked.cuda()].cpu(), x, oc.values_of(fmt, part))
    for rows in (1, 2, 3, 4, 5, 8):
        out = h.run(fmt, xd[:rows].contiguous(), t, torch.full((rows, n), float("nan"), device="cuda"))
        assert torch.equal(out, batch[:rows]), rows
    assert h.cabi.load().dg_take_status() == 0
