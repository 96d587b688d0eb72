"""The network's long sums over voxels (head and last bias gradients) against independent FP64 sums, with more chunks than one
pass of the reduction takes (1280, and 4096 of more than 256 voxels).  A head of one weight at a time makes the output
the last activations themselves, from which the sums follow: dw = sum dout a, db = sum dout, and the last convolution's bias
sum of BF16(dout w) where a > 0.  Tolerance, before the first run: FP32 sums of 4096 partial sums in turn err by about
eps sqrt(4096) = 4e-6 of the size sqrt(n) rms that n terms of random sign reach; 1e-4 of it (a lost chunk is 1e-2 and more)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["mma", "tcgen05"])
@pytest.mark.parametrize("shape", [(64, 32, 160), (128, 128, 72)])
def test_long_sums(sfpkg, gpu_ctx, shape, mode):
    import torch
    from oracle import unet_ref as ref
    g = sfpkg.StaggeredGrid.from_origin(1.0 / shape[0], shape)
    n = g.num_cells
    rng = np.random.default_rng(5)
    P = ref.init_params(16, seed=23)
    P["d0b.b"] = rng.normal(0.2, 0.05, P["d0b.b"].shape).astype(np.float32)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(6)
    feat = torch.randn((n, 16), generator=gen, device="cuda").to(torch.bfloat16)
    dout = torch.randn(n, generator=gen, device="cuda")
    net = sfpkg.Network(gpu_ctx)
    net.set_mode(mode)
    net.set_params(ref.flatten(P))
    G = ref.unflatten(net.gradients(g, feat, dout))

    def close(got, terms):
        want, size = terms.sum().item(), terms.square().sum().sqrt().item()
        assert abs(float(got) - want) <= 1e-4 * size, (got, want, size)

    close(G["head.b"].ravel()[0], dout.double())
    w = np.array(P["head.w"], dtype=np.float32).ravel()
    out = torch.zeros(n, dtype=torch.float32, device="cuda")
    for c in range(16):
        Q = dict(P)
        one = np.zeros_like(P["head.w"])
        one.ravel()[c] = 1.0
        Q["head.w"] = one
        net.set_params(ref.flatten(Q))
        net.forward(g, feat, out)
        a = out.double()
        assert a.max().item() > 0
        close(G["head.w"].ravel()[c], dout.double() * a)
        dy = (dout * float(w[c])).to(torch.bfloat16).double() * (a > 0)
        close(G["d0b.b"].ravel()[c], dy)
    net.close()
