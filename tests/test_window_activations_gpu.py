"""Activations of a K that is no multiple of 64: the windows that lie within the rows come by tensor copies, the last one by the copying
warps. K at the edges of windows of one and two steps, rows with gaps, one and several tiles per CTA, batches; the values are the
CPU oracle's, and a row has the bits that it has among sixteen and behind a gap."""
import pytest
import torch

from oracle import decode_gemv_oracle as oc
from oracle import workloads as wl
from tests import helpers as h

pytestmark = pytest.mark.gpu
MAKE = {"nvfp4": wl.cfg_nvfp4, "fp8": wl.cfg_fp8, "mxfp8": wl.cfg_mxfp8, "bf16": wl.cfg_bf16}


# (a window holds 1024 or 2048 values of NVFP4, 512 or 1024 of FP8 and MXFP8, 512 of BF16)
@pytest.mark.parametrize("fmt,n,k", [
    ("nvfp4", 300, 992), ("nvfp4", 300, 1056), ("nvfp4", 148 * 70, 2016), ("nvfp4", 148 * 70, 2080), ("nvfp4", 148 * 56, 4128),
    ("nvfp4", 148 * 20, 16416), ("fp8", 300, 496), ("fp8", 148 * 70, 528), ("fp8", 148 * 70, 1040), ("fp8", 148 * 56, 4112),
    ("mxfp8", 300, 480), ("mxfp8", 148 * 70, 544), ("mxfp8", 148 * 56, 4128), ("bf16", 300, 504), ("bf16", 148 * 70, 520),
    ("bf16", 148 * 20, 4104)])
def test_windows_within_the_rows_and_the_last_one(fmt, n, k):
    host = MAKE[fmt](n, k, seed=n + k)
    host = host if isinstance(host, tuple) else (host,)
    t = tuple(part.cuda() for part in host)
    x = torch.randn(16, k, generator=torch.Generator().manual_seed(k)).to(torch.bfloat16)
    xd = x.cuda()
    batch = h.run(fmt, xd, t, torch.full((16, n), float("nan"), device="cuda"))
    picked = torch.randperm(n, generator=torch.Generator().manual_seed(n))[:256].sort().values
    part = tuple(a[picked] for a in host)
    assert oc.within_fp32_bound(batch[:, picked.cuda()].cpu(), x, oc.values_of(fmt, part))
    for rows in (1, 4, 8, 16):
        wide = torch.full((rows, k + 8), float("nan"), dtype=torch.bfloat16, device="cuda")   # what a copy past a row's end would bring
        wide[:, :k] = xd[:rows]
        out = h.run(fmt, wide[:, :k], t, torch.full((rows, n), float("nan"), device="cuda"))
        assert torch.equal(out, batch[:rows]), rows
    assert h.cabi.load().dg_take_status() == 0
