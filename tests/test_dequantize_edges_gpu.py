"""The dequantizers at the edges of a CTA's run of 1024 output vectors (8 or 16 values each), which may start and end anywhere
in a row: bit for bit against the CPU oracle."""
import ctypes

import pytest
import torch

from crit_kernels_b200 import cabi
from oracle import decode_gemv_oracle as oc
from oracle import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(1, 8192), (1, 16384), (2, 8208), (3, 5472), (16, 512), (17, 1008), (1025, 16)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float8_e4m3fn])
def test_runs_that_cross_rows(n, k, dtype):
    c, s, i = wl.cfg_nvfp4(n, k, seed=n + k)
    i = i * (48.0 if dtype == torch.float8_e4m3fn else 1.0)
    cd, sd, f = c.cuda(), s.cuda(), i.cuda()
    out = torch.full((n * k * dtype.itemsize + 64,), 0x55, dtype=torch.uint8, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    kind = 3 if dtype == torch.float8_e4m3fn else 1
    assert cabi.load().dg_enqueue_dequantize(ptr(cd), ptr(sd), ptr(f), ptr(out), kind, n, k, None) == 0
    torch.cuda.synchronize()
    want = oc.dequantize(c, s, i, dtype)
    assert torch.equal(out[:-64].cpu(), want.view(torch.uint8).flatten())
    assert bool((out[-64:] == 0x55).all())


@pytest.mark.parametrize("n,k,dtype", [(n, k, d) for d, k in ((torch.bfloat16, 8192), (torch.float8_e4m3fn, 16384))
                                       for n in (147, 148, 149)] + [(1, 16, torch.bfloat16), (255, 16, torch.float8_e4m3fn)])
def test_matrices_around_one_run_per_sm(n, k, dtype):
    """Below 1024 output vectors per SM a CTA takes 256 of them."""
    test_runs_that_cross_rows(n, k, dtype)


@pytest.mark.parametrize("n,k", [(40, 1024), (1500, 2048)])             # in one launch the other way of the two
def test_a_chain_of_calls_reads_what_the_one_before_wrote(n, k):
    """The kernels start before the previous one of the stream has finished."""
    import crit_kernels_b200
    kernel = crit_kernels_b200.get_kernel("crit-labs/decode-gemv", version=1)
    mats = [tuple(t.cuda() for t in wl.cfg_nvfp4(n, k, seed=s)) for s in range(2)]
    want = []
    for m in mats:
        w = kernel.decode(*m, torch.empty(n, k, dtype=torch.bfloat16, device="cuda"))
        torch.cuda.synchronize()
        q, scale = kernel.quantize_fp8_rows(w, torch.empty(n, k, dtype=torch.uint8, device="cuda"), torch.empty(n, device="cuda"))
        torch.cuda.synchronize()
        want.append((w, q, scale))
    now = tuple(torch.empty_like(t) for t in mats[0])
    got = [tuple(torch.zeros_like(t) for t in want[0]) for _ in range(12)]
    for i, (w, q, scale) in enumerate(got):
        for t, source in zip(now, mats[i % 2]):
            t.copy_(source)
        kernel.decode(*now, w)
        kernel.quantize_fp8_rows(w, q, scale)
        kernel.decode(*mats[(i + 1) % 2], w)                            # may not overtake the call that reads w
    torch.cuda.synchronize()
    for i, (w, q, scale) in enumerate(got):
        assert torch.equal(w, want[(i + 1) % 2][0]) and torch.equal(q, want[i % 2][1]) and torch.equal(scale, want[i % 2][2])
