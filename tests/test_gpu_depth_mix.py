"""The weighted average over depth and the norm that reads it, in one kernel."""
import pytest
import torch

from esp_b200.csrc import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows, width, index", [(1, 4, 0), (8, 2048, 7), (3, 1028, 1), (300, 4100, 2), (2, 16384, 12)])
@pytest.mark.parametrize("parts", ["none", "delta", "scaled"])
def test_equals_the_two_kernels(dtype, rows, width, index, parts):
    x, gamma, weights = rnd(rows, width), rnd(width, seed=1), rnd(index + 2, seed=2)
    delta = rnd(rows, width, seed=3) if parts != "none" else None
    scale = rnd(width, seed=4) if parts == "scaled" else None
    history = torch.full((index + 3, rows, width), 7.0, device=DEV)
    history[:index + 1] = rnd(index + 1, rows, width, seed=5)
    x1, hist1, h1 = x.clone(), history.clone(), torch.empty(rows, width, dtype=dtype, device=DEV)
    ops.depth_mix(x1, delta, scale, hist1, weights, index)
    ops.add_rmsnorm(x1, None, gamma, h1, 1e-5)
    x2, hist2, h2 = x.clone(), history.clone(), torch.empty(rows, width, dtype=dtype, device=DEV)
    ops.depth_mix_rmsnorm(x2, delta, scale, hist2, weights, index, gamma, h2, 1e-5)
    assert torch.equal(x1, x2) and torch.equal(hist1, hist2) and torch.equal(h1, h2)
    # and what they mean, in 64 bits
    layer = x.double() + (0 if delta is None else delta.double() * (1 if scale is None else scale.double()))
    want = (weights[:index + 1].double()[:, None, None] * history[:index + 1].double()).sum(0) + weights[index + 1].double() * layer
    normed = want / torch.sqrt((want * want).mean(-1, keepdim=True) + 1e-5) * gamma.double()
    bound = (index + 8) * 2.0 ** -24 if dtype == torch.float32 else 2.0 ** -8
    assert (h2.double() - normed).norm() <= 2 * bound * normed.norm()


@pytest.mark.parametrize("rows, width", [(8, 2048), (400, 2048), (5, 16384)])
def test_reads_what_the_kernel_before_has_written(rows, width):
    """The kernel before (tanh) lets the next one in at once and writes what that one reads: nothing may be asked for ahead of the
    wait.  Over and over in one stream, each time with other numbers in the place of the last ones."""
    gamma, weights, scale = rnd(width, seed=1), rnd(2, seed=2), rnd(width, seed=4)
    z, y = rnd(12, rows, width, seed=5), torch.zeros(rows, width, device=DEV)
    x = rnd(rows, width)
    history = torch.zeros(2, rows, width, device=DEV)
    wanted = []
    for i in range(12):
        ops.tanh(z[i], y)
        torch.cuda.synchronize()
        x1, h = x.clone(), torch.empty(rows, width, device=DEV)
        torch.cuda.synchronize()
        if i % 2:
            ops.depth_mix_rmsnorm(x1, y, scale, history, weights, 0, gamma, h, 1e-5)
        else:
            ops.add_rmsnorm(x1, y, gamma, h, 1e-5)
        wanted.append((x1, h))
    copies = [(x.clone(), torch.empty(rows, width, device=DEV)) for _ in range(12)]
    torch.cuda.synchronize()
    for i, (x1, h) in enumerate(copies):
        ops.tanh(z[i], y)
        if i % 2:
            ops.depth_mix_rmsnorm(x1, y, scale, history, weights, 0, gamma, h, 1e-5)
        else:
            ops.add_rmsnorm(x1, y, gamma, h, 1e-5)
    for (a, b), (c, d) in zip(wanted, copies):
        assert torch.equal(a, c) and torch.equal(b, d)


def test_refusals():
    x, h = rnd(2, 8), torch.empty(2, 8, device=DEV)
    with pytest.raises(Exception, match="too short"):
        ops.depth_mix_rmsnorm(x, None, None, torch.zeros(2, 2, 8, device=DEV), rnd(3), 1, rnd(8), h, 1e-6)
    with pytest.raises(Exception, match="refused"):
        ops.depth_mix_rmsnorm(rnd(2, 6), None, None, torch.zeros(2, 2, 6, device=DEV), rnd(2), 0, rnd(6), torch.empty(2, 6, device=DEV), 1e-6)
    assert not ops.depth_mix_rmsnorm_fits(6) and not ops.depth_mix_rmsnorm_fits(16388) and ops.depth_mix_rmsnorm_fits(16384)
