"""BF16 activations of the FP8, MXFP8 and NVFP4 GEMVs over BF16's whole range. The kernels multiply a chunk of an activation row
(64 bytes of codes) as FP16 times a power of two when its values lie within 32 binades, as BF16 otherwise: checked at the edges
of these rules against the CPU oracle's exact products, and no kind of activations may cost a GEMV many times what others do."""
import pytest
import torch

from oracle import decode_gemv_oracle as oc
from oracle import workloads as wl
from tests import helpers as h

pytestmark = pytest.mark.gpu
MAKE = {"nvfp4": wl.cfg_nvfp4, "fp8": wl.cfg_fp8, "mxfp8": wl.cfg_mxfp8}
CHUNK = {"nvfp4": 128, "fp8": 64, "mxfp8": 64}          # values


def two_sided(shape, g):
    return torch.randn(shape, generator=g).sign()


def activations(fmt, k, g):
    """16 rows, one rule each; column 0 of every row that has a large value holds it (see the test)."""
    chunk = CHUNK[fmt]
    x = torch.randn(16, k, generator=g)
    x[1] = torch.exp2(torch.randint(-24, 8, (k,), generator=g).float())       # the usual window from end to end
    x[2] = torch.exp2(torch.randint(-23, 9, (k,), generator=g).float())       # one binade up: 32 binades, another power
    x[3] = torch.exp2(torch.randint(-24, 9, (k,), generator=g).float())       # 33 binades
    x[4] *= 2.0 ** 100
    x[5] *= 2.0 ** -120
    x[6] = 2.0 ** -133 * torch.randint(0, 128, (k,), generator=g).float()     # subnormals
    x[7] = torch.exp2(torch.rand(k, generator=g) * 160 - 100) * two_sided(k, g)
    x[8] = 0.0
    x[8, k // 2] = 2.0 ** -30
    x[9, :chunk] = torch.exp2(torch.rand(min(chunk, k), generator=g) * 60 - 40)
    x[10] *= 2.0 ** -30
    x[11] = torch.nn.functional.silu(x[11] * 300) * 300 * torch.randn(k, generator=g)
    x[12] = 0.0
    x[13, ::2] = -0.0
    x[14] = x[14].relu()
    for row, top in ((2, 256.0), (9, 2.0 ** 20), (10, 2.0 ** 2), (13, 2.0 ** 20), (15, 300.0)):
        x[row, 0] = top
    return x.to(torch.bfloat16)


@pytest.mark.parametrize("fmt,n,k", [
    ("nvfp4", 149, 1024), ("nvfp4", 1200, 8192), ("nvfp4", 700, 2080), ("nvfp4", 4800, 512), ("nvfp4", 300, 28672),
    ("fp8", 149, 1024), ("fp8", 2400, 4096), ("fp8", 700, 1040), ("fp8", 300, 28672),
    ("mxfp8", 149, 1024), ("mxfp8", 2400, 2048), ("mxfp8", 700, 1056)])
def test_activations_of_every_range(fmt, n, k):
    host = MAKE[fmt](n, k, seed=n + k)
    # Column 0 of every odd matrix row is zero: such a row's output is made of the small values alone, and dropping them beside
    # a large one would show.
    host[0][1::2, 0] &= 0xF0 if fmt == "nvfp4" else 0
    t = tuple(part.cuda() for part in host)
    x = activations(fmt, k, torch.Generator().manual_seed(n))
    xd = x.cuda()
    out = h.run(fmt, xd, t, torch.full((16, n), float("nan"), device="cuda"))
    values = oc.values_of(fmt, host)
    # FP32 sums, and FP32's smallest steps (a product, a sum and the row scale may each lose half of one)
    bound = oc.gemv_magnitude(x, values) * 2e-5 + 4 * k * 2.0 ** -149
    error = (out.cpu().double() - oc.gemv_exact(x, values)).abs()
    assert bool((error <= bound).all()), [(row, float((error[row] / bound[row]).max())) for row in range(16)]
    for rows in (1, 2, 3, 4, 5, 8, 9):
        assert torch.equal(h.run(fmt, xd[:rows].contiguous(), t, torch.empty(rows, n, device="cuda")), out[:rows]), rows
    for row in range(16):
        assert torch.equal(h.run(fmt, xd[row:row + 1].contiguous(), t, torch.empty(1, n, device="cuda"))[0], out[row]), row


@pytest.mark.parametrize("fmt", list(MAKE))
@pytest.mark.parametrize("rows", [1, 3, 6, 16])
def test_infinities_and_nans_stay_in_their_rows(fmt, rows):
    n, k = 333, 2048
    host = MAKE[fmt](n, k, seed=3)
    t = tuple(part.cuda() for part in host)
    x = torch.randn(rows, k, generator=torch.Generator().manual_seed(4))
    clean = h.run(fmt, x.to(torch.bfloat16).cuda(), t, torch.empty(rows, n, device="cuda"))
    x[0, 5], x[rows // 2, 700], x[rows - 1, 1999] = float("inf"), float("nan"), float("-inf")
    x = x.to(torch.bfloat16)
    out = h.run(fmt, x.cuda(), t, torch.empty(rows, n, device="cuda")).cpu().double()
    want = oc.gemv_exact(x, oc.values_of(fmt, host))
    touched = {0, rows // 2, rows - 1}
    for row in range(rows):
        if row in touched:
            assert torch.equal(out[row].isnan(), want[row].isnan())
            assert torch.equal(out[row][~out[row].isnan()], want[row][~want[row].isnan()])
        else:
            assert torch.equal(out[row], clean[row].cpu().double())


def replay_us(call):
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(20):
            call()
    times = []
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        graph.replay()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) / 20 * 1e3)
    return sorted(times)[3]


@pytest.mark.parametrize("fmt,n,k", [("nvfp4", 8192, 8192), ("nvfp4", 2048, 28672), ("fp8", 8192, 4096), ("mxfp8", 8192, 4096)])
@pytest.mark.parametrize("rows", [1, 4, 8, 16])
def test_no_kind_of_activations_is_many_times_slower(fmt, n, k, rows):
    """A power of two of their own costs chunks little; chunks that stay BF16 take about twice as long. (Multiplied apart after
    the tile, they took 5 to 30 times as long.)"""
    g = torch.Generator().manual_seed(1)
    t = tuple(part.cuda() for part in MAKE[fmt](n, k, seed=2))
    out = torch.empty(rows, n, dtype=torch.bfloat16, device="cuda")
    normal = torch.randn(rows, k, generator=g)
    outlier = normal.clone()
    outlier[:, k // 3] = 300.0
    kinds = {"normal": normal, "outlier": outlier, "large": normal * 4096, "small": normal * 2.0 ** -40, "zeros": normal.relu(),
             "wide": torch.nn.functional.silu(normal * 367) * 367 * torch.randn(rows, k, generator=g)}
    us = {}
    for name, x in kinds.items():
        xd = x.to(torch.bfloat16).cuda()
        us[name] = replay_us(lambda: h.run(fmt, xd, t, out))
    for name, limit in (("outlier", 1.3), ("large", 1.7), ("small", 1.7), ("zeros", 1.7), ("wide", 3.0)):
        assert us[name] <= limit * us["normal"], (name, us)
