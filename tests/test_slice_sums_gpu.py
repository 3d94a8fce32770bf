"""The order in which a row's sum is formed is the stated one: eight slices of K (64 bytes of codes of every 512-byte step; BF16
128 of 1 KB), each summed step after step, then added as a balanced tree and multiplied by the row scale. Row invariance alone
would not notice an order that is consistently another one. One value per slice and step is not zero, so that every product
is exact and the rest is FP32 additions, repeated here with numpy bit for bit."""
import numpy as np
import pytest
import torch

from tests import helpers as h

pytestmark = pytest.mark.gpu
CHUNK = {"nvfp4": 128, "fp8": 64, "mxfp8": 64, "bf16": 64}          # values of a slice in a step


def weights(fmt, n, k):
    """Every weight 1.5, row scales 0.75."""
    scale = torch.full((n,), 0.75)
    if fmt == "nvfp4":
        return torch.full((n, k // 2), 0x33, dtype=torch.uint8), torch.full((n, k // 16), 0x38, dtype=torch.uint8), scale
    if fmt == "fp8":
        return torch.full((n, k), 0x3C, dtype=torch.uint8), scale
    if fmt == "mxfp8":
        return torch.full((n, k), 0x3C, dtype=torch.uint8), torch.full((n, k // 32), 127, dtype=torch.uint8)
    return (torch.full((n, k), 1.5, dtype=torch.bfloat16),)


@pytest.mark.parametrize("fmt", list(CHUNK))
@pytest.mark.parametrize("steps", [1, 3])
@pytest.mark.parametrize("rows", [2, 16])
def test_the_eight_slices_are_added_as_a_tree(fmt, steps, rows):
    n, chunk = 37, CHUNK[fmt]
    g = torch.Generator().manual_seed(steps * rows)
    terms = torch.randn(rows, steps, 8, generator=g) * torch.exp2(torch.randint(-14, 6, (rows, steps, 8), generator=g).float())
    terms = terms.to(torch.bfloat16)
    x = torch.zeros(rows, steps, 8, chunk, dtype=torch.bfloat16)
    x[..., 5] = terms
    x = x.view(rows, -1)
    out = h.run(fmt, x.cuda(), tuple(t.cuda() for t in weights(fmt, n, x.shape[1])), torch.empty(rows, n, device="cuda")).cpu().numpy()
    products = terms.float().numpy() * np.float32(1.5)
    slices = np.zeros((rows, 8), np.float32)
    for step in range(steps):
        slices = slices + products[:, step]
    a = [slices[:, i] for i in range(8)]
    tree = ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]))
    if fmt in ("nvfp4", "fp8"):
        tree = tree * np.float32(0.75)
    assert tree.dtype == np.float32
    assert np.array_equal(out.view(np.uint32), np.repeat(tree[:, None], n, 1).view(np.uint32))
    chain = a[0]
    for part in a[1:]:
        chain = chain + part
    assert rows == 2 or bool((chain != (tree / np.float32(0.75) if fmt in ("nvfp4", "fp8") else tree)).any())
