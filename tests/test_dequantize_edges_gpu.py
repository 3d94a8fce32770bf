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


@pytest.mark.parametrize("n,k", [(300, 1024), (4096, 4096)])            # in one launch the other way of the two
def test_a_matrix_just_dequantized_is_static_for_the_next_gemv(n, k):
    """With static weights a GEMV reads its matrix before it waits for the kernel in front of it."""
    import crit_kernels_b200
    kernel = crit_kernels_b200.get_kernel("crit-labs/decode-gemv", version=1)
    mats = [tuple(t.cuda() for t in wl.cfg_nvfp4(n, k, seed=s)) for s in range(2)]
    x = wl.activations(3, k, seed=2).cuda()
    want = []
    for m in mats:
        w = kernel.decode(*m, torch.empty(n, k, dtype=torch.bfloat16, device="cuda"))
        torch.cuda.synchronize()
        want.append(kernel.gemv_bf16(x, w, torch.empty(3, n, device="cuda")))
        torch.cuda.synchronize()
    w = torch.zeros(n, k, dtype=torch.bfloat16, device="cuda")
    got = [torch.zeros(3, n, device="cuda") for _ in range(12)]
    previous = cabi.load().dg_set_static_weights(1)
    try:
        for i, out in enumerate(got):
            kernel.decode(*mats[i % 2], w)
            kernel.gemv_bf16(x, w, out)
        torch.cuda.synchronize()
    finally:
        cabi.load().dg_set_static_weights(previous)
    for i, out in enumerate(got):
        assert torch.equal(out, want[i % 2]), i
    assert cabi.load().dg_take_status() == 0


@pytest.mark.parametrize("n,k", [(40, 1024), (1500, 2048)])
def test_factors_and_codes_that_the_kernel_before_writes(n, k):
    """Kernels of the package that let the dequantizer start early write what it reads: the FP8 quantizer its factors, the NVFP4
    quantizer its codes, others with every call."""
    import crit_kernels_b200
    kernel = crit_kernels_b200.get_kernel("crit-labs/decode-gemv", version=1)
    codes, scales, _ = (t.cuda() for t in wl.cfg_nvfp4(n, k, seed=5))
    g = torch.Generator().manual_seed(n)
    rows = [(torch.randn(n, k, generator=g) * 2.0 ** i).to(torch.bfloat16).cuda() for i in range(3)]
    tiles = torch.empty(oc.blocked_numel(n, k), dtype=torch.uint8, device="cuda")
    q, factor, now = torch.empty(n, k, dtype=torch.uint8, device="cuda"), torch.empty(n, device="cuda"), torch.empty_like(codes)
    new = lambda: (torch.zeros(n, k, dtype=torch.bfloat16, device="cuda"), torch.zeros(n, k, dtype=torch.bfloat16, device="cuda"))

    def chain(i, out, between):
        kernel.quantize_fp8_rows(rows[i % 3], q, factor)
        between()
        kernel.decode(codes, scales, factor, out[0])
        between()
        kernel.quantize_nvfp4(rows[(i + 1) % 3], 2688.0 / (8.0 + i % 3), now, tiles)
        between()
        kernel.decode(now, scales, factor, out[1])
        between()
    want = [new() for _ in range(9)]
    for i, out in enumerate(want):
        chain(i, out, torch.cuda.synchronize)
    got = [new() for _ in range(9)]
    for i, out in enumerate(got):
        chain(i, out, lambda: None)
    torch.cuda.synchronize()
    for i in range(9):
        assert torch.equal(got[i][0], want[i][0]) and torch.equal(got[i][1], want[i][1]), i
