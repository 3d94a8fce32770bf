"""Batched launches in which bulk copies bring everything (all of a CTA's other warps then finish tiles): the bits of single
launches, resident activations of several K and of every range among them, and no longer than these take."""
import ctypes

import pytest
import torch

from crit_kernels_b200 import cabi
from crit_kernels_b200 import stack as stacks
from oracle import workloads as wl
from tests import helpers as h
from tests.test_batch_gpu import encode

pytestmark = pytest.mark.gpu
SHAPES = ((96, 256), (1280, 4096), (7168, 1024), (9500, 512), (1024, 8192), (600, 28672), (5, 768))
ROLES = (("qkv", 8192, 10240), ("o", 8192, 8192), ("gate_up", 8192, 57344), ("down", 28672, 8192))


@pytest.mark.parametrize("world", [0, 1])
@pytest.mark.parametrize("m", [1, 3, 4, 5, 8, 9, 16])
def test_a_batch_without_anything_to_copy_gives_the_bits_of_single_calls(m, world):
    lib, dev = cabi.load(), torch.device("cuda")
    flags = torch.zeros(4, dtype=torch.int32, device=dev)
    keep, items, got, want = [], [], [], []
    for i, (n, k) in enumerate(SHAPES):
        t = tuple(part.to(dev) for part in wl.cfg_nvfp4(n, k, seed=20 + i))
        x = wl.activations(m, k, seed=50 + i)
        if i % 2:
            x[i % m, k // 2] = 300.0
            x[(i + 1) % m, 3] = 2.0 ** 40
        x = x.to(dev)
        want.append(h.run("nvfp4", x, t, torch.empty(m, n, dtype=torch.bfloat16, device=dev)))
        out = torch.full((m, n), -1.0, dtype=torch.bfloat16, device=dev)
        peers = (ctypes.c_void_p * 1)(out.data_ptr())
        got.append(out)
        keep.append((t, x, peers))
        items.append(cabi.Nvfp4BatchItem(x=x.data_ptr(), codes=t[0].data_ptr(), scales=t[1].data_ptr(), inverse=t[2].data_ptr(),
                                         out=out.data_ptr(), peer_out=ctypes.cast(peers, ctypes.POINTER(ctypes.c_void_p)),
                                         ldx=k, ldo=n, blocked=0, N=n, K=k))
    host, device = encode(lib, items, m, world, flags, 0, dev)
    for _ in range(2):
        for out in got:
            out.fill_(-1.0)
        torch.cuda.synchronize()
        assert lib.dg_enqueue_batch(ctypes.c_void_p(host.data_ptr()), None) == 0
        torch.cuda.synchronize()
        for out, w in zip(got, want):
            assert torch.equal(out.view(torch.int16), w.view(torch.int16)), (m, tuple(w.shape))
        assert int(flags.abs().sum()) == 0


def us(run):
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    for _ in range(5):
        run.replay()
    b.record()
    torch.cuda.synchronize()
    return a.elapsed_time(b) / 5 * 1e3


@pytest.mark.parametrize("rows", [1, 8, 16])
def test_batched_launches_take_no_longer_than_single_ones(rows):
    """Four GEMVs a launch. (With a single finishing warp, and copying warps that had nothing to copy, they took 1.04 and 1.10 times
    as long as single launches at 8 and 16 rows.)"""
    stack = stacks.ShardedStack.random(4, ROLES, 0, 1, torch.device("cuda"), seed=3)
    single, batched = stack.capture(rows), stack.with_batch(4).capture(rows)
    times = [(us(batched), us(single)) for _ in range(12)][2:]
    ratio = sorted(b / s for b, s in times)[len(times) // 2]
    assert ratio <= 1.035, (ratio, times)
