"""A forward pass holds the activations that its layers read and no copies of them: decoder
inputs that are read in place are not written out, nor is memory for them kept; on the
other convolution path they are, and switching the path of one network back and forth
gives each path's own output again, bit for bit.

Bound: the buffers' sizes, 2 MB each for the allocator's granularity and 32 MB for kernels
loaded on first use.
"""
import pytest

from phasecon_b200 import warmstart as WS

pytestmark = pytest.mark.gpu


def test_forward_holds_what_its_layers_read():
    import torch
    c, shape = 16, (32, 256, 256)
    x = torch.rand(*shape, device="cuda") * 0.02
    net = WS.UNet(c, seed=1)
    net.forward(x[:8, :8, :8].contiguous())  # kernels loaded, weights laid out
    out = net.forward(x)  # torch's block for the output
    del out
    net.close()
    net = WS.UNet(c, seed=1)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    net.forward(x)
    used = before - torch.cuda.mem_get_info()[0]
    V = [shape[0] * shape[1] * shape[2] >> 3 * l for l in range(4)]
    C = [c << l for l in range(4)]
    bufs = [2 * V[0], 4 * V[0]]                                     # the scaled input, the output
    bufs += [2 * V[l] * C[l] for l in range(4) for _ in range(2)]   # encoder
    bufs += [2 * V[l + 1] * C[l] for l in range(3)]                 # pooled
    bufs += [2 * V[l] * C[l] for l in range(3) for _ in range(3)]   # decoder
    assert used <= sum(bufs) + 2 * 2**20 * len(bufs) + 32 * 2**20


@pytest.mark.parametrize("c,shape", [(16, (16, 24, 40)), (8, (8, 16, 8)), (12, (8, 8, 16))])
def test_switching_the_convolution_path(c, shape):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(3)
    x = torch.rand(*shape, device="cuda", generator=gen) * 0.02
    t = x + 0.003 * torch.randn(*shape, device="cuda", generator=gen)
    net = WS.UNet(c, seed=2)
    net.input_scale = 50.0
    outs, losses = {0: [], 1: []}, {0: [], 1: []}
    for path in (1, 0, 1, 0, 0, 1):
        net.tensor_path = path
        outs[path].append(net.forward(x))
        losses[path].append(net.gradients(x, t)[0])
    for path in (0, 1):
        assert all(torch.equal(outs[path][0], o) for o in outs[path])
        # the loss: FP64 sums of the same terms, added up by atomics
        assert losses[path] == pytest.approx([losses[path][0]] * 3, rel=1e-12)
    net.close()
