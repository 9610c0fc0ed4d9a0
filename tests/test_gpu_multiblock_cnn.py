"""Multi-block convolution on CUDA tensors over domains built through the PISOtorch API, against the
reference's own ``MultiblockConv`` outputs and gradients (tests/golden/ref_mbcnn_*.npz)."""
import pytest
import torch

import setups
from test_multiblock_cnn import run_against_fixture, FIXTURES
from pict_b200.multiblock_cnn import MultiblockConv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,k", FIXTURES)
def test_domain_matches_reference_fixture(name, k):
    domain = setups.build_product(setups.mbcnn_case(name), dtype=torch.float64, prepare=False)
    run_against_fixture(domain, name, k, "cuda")


def test_velocity_fields_through_layers():
    """A small multi-block network over a domain's block velocities: shapes per block, gradients reach every block."""
    spec = setups.mbcnn_case("grid2x2_2d")
    domain = setups.build_product(spec, dtype=torch.float32, prepare=False)
    net = torch.nn.ModuleList([MultiblockConv(domain, "ZERO", 2, 8, 3, device="cuda"),
                               MultiblockConv(domain, "ZERO", 8, 2, 5, device="cuda")])
    xs = [torch.randn_like(b.velocity).requires_grad_(True) for b in domain.getBlocks()]
    h = net[0](xs, domain)
    h = [torch.relu(t) for t in h]
    out = net[1](h, domain)
    assert [o.shape for o in out] == [x.shape for x in xs]
    sum(o.square().sum() for o in out).backward()
    assert all(x.grad is not None and torch.isfinite(x.grad).all() and x.grad.abs().sum() > 0 for x in xs)


@pytest.mark.parametrize("name", setups.MBCNN_CASES + setups.MBCNN_CYCLE_CASES)
@pytest.mark.parametrize("k", [3, 5])
def test_padding_kernels_equal_the_index_map(name, k):
    """The library's padding launch (pict_mb_pad_gather) equals the index map applied with index_select on
    CPU tensors, bitwise; its gradient (pict_mb_pad_scatter_sum, a fixed-order gather-sum) equals the
    index_add gradient of the CPU path to round-off."""
    from pict_b200 import _lib
    domain = setups.build_product(setups.mbcnn_case(name), dtype=torch.float64, prepare=False)
    layer = MultiblockConv(domain, "ZERO", 3, 2, k)
    g = torch.Generator().manual_seed(7)
    xs = [torch.randn([2, 3] + list(b.velocity.shape[2:]), generator=g, dtype=torch.float64) for b in domain.getBlocks()]
    ws = None
    grads = []
    outs = []
    for dev in ("cpu", "cuda"):
        layer = layer.to(dev)
        x = [t.detach().clone().to(dev).requires_grad_(True) for t in xs]
        pads = layer.pad(x)
        if ws is None:
            ws = [torch.randn(p.shape, generator=g, dtype=torch.float64) for p in pads]
        sum((p * w.to(dev)).sum() for p, w in zip(pads, ws)).backward()
        outs.append([p.detach().cpu() for p in pads])
        grads.append([t.grad.cpu() for t in x])
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    for a, b in zip(*grads):
        assert torch.allclose(a, b, rtol=1e-13, atol=1e-13)
    assert _lib.load() is not None


@pytest.mark.parametrize("channels", [64, 67])
def test_padding_kernels_with_many_channels_a_thread(channels):
    """Blocks so large that a thread walks 32 channels of its cell and more, eight at a time with a remainder (small
    blocks give every channel its own thread): the padded values bitwise, the gradient to round-off, at the connections
    of a 2 x 2 grid of uneven blocks too; a gradient of -0 gives +0, as adding it to zeros does."""
    from pict_b200 import PISOtorch as P
    dom = P.Domain(2, torch.tensor([1e-3]), name="grid", dtype=torch.float32, device=torch.device("cuda"),
                   passiveScalarChannels=0)
    sizes = [(320, 330), (320, 325), (323, 330), (323, 325)]   # (y, x) per block
    b = [dom.CreateBlockWithSize(P.Int4(x, y, 1, 2), name="b%d" % i) for i, (y, x) in enumerate(sizes)]
    for blk in b:
        blk.CloseAllBoundaries()
    b[0].ConnectBlock("+x", b[1], "-x", "-y")
    b[0].ConnectBlock("+y", b[2], "-y", "-x")
    b[1].ConnectBlock("+y", b[3], "-y", "-x")
    b[2].ConnectBlock("+x", b[3], "-x", "-y")
    layer = MultiblockConv(dom, "ZERO", channels, 1, 3, dtype=torch.float32)
    g = torch.Generator().manual_seed(5)
    xs = [torch.randn((1, channels) + s, generator=g) for s in sizes]
    ws = [torch.randn((1, channels, s[0] + 2, s[1] + 2), generator=g) for s in sizes]
    res = []
    for dev in ("cpu", "cuda"):
        layer = layer.to(dev)
        x = [t.detach().clone().to(dev).requires_grad_(True) for t in xs]
        pads = layer.pad(x)
        torch.autograd.backward(pads, [w.to(dev) for w in ws])
        res.append(([p.detach().cpu() for p in pads], [t.grad.cpu() for t in x]))
    for a, c in zip(res[0][0], res[1][0]):
        assert torch.equal(a, c)
    for a, c in zip(res[0][1], res[1][1]):
        # at most 4 readers a cell, summed in another order: 3 roundings of a sum of 4 values
        assert float((a - c).abs().max()) <= 3 * 4 * 2 ** -24 * float(max(w.abs().max() for w in ws))
    x = [t.detach().clone().cuda().requires_grad_(True) for t in xs]
    torch.autograd.backward(layer.pad(x), [torch.full_like(w, -0.0).cuda() for w in ws])
    assert not any(bool(torch.signbit(t.grad).any()) for t in x)
