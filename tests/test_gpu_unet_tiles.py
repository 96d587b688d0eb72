"""U-Net kernels at the edges of their tiles and of the rules that choose them, the tensor-core path against the
warp-MMA one.  Forward: FP32 sums in different orders and BF16 activations, relative L2 1e-2.  Weight gradients from the
same BF16 dY and X: FP32 sums of up to 2^19 products in different orders, eps sqrt(n / 2) = 3e-5, relative L2 1e-4."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

LAYERS = [(16, 16, 27), (16, 16, 27), (16, 32, 27), (32, 32, 27), (32, 64, 27), (64, 64, 27), (64, 64, 27), (64, 64, 27),
          (64, 64, 27), (64, 32, 27), (32, 32, 27), (32, 16, 27), (16, 16, 27), (16, 16, 27), (16, 1, 1)]


# (4, 6, 40): the smallest grid of the halo'd weight gradient, (4, 5, 40), (3, 6, 40): below it;
# (34, 33, 32): chunks of the warp-MMA weight gradient longer than one index tile;
# (4, 6, 128), (7, 10, 131): z lines four high; (64, 32, 128), (63, 31, 130): eight high (whole and ragged bricks);
# (64, 32, 160): warp-MMA layers with every output channel in one block (the smaller grids split them)
@pytest.mark.parametrize("shape", [(4, 6, 40), (4, 5, 40), (3, 6, 40), (34, 33, 32), (4, 6, 128), (7, 10, 131),
                                   (64, 32, 128), (63, 31, 130), (64, 32, 160)])
def test_tile_edges(sfpkg, gpu_ctx, shape):
    import torch
    from oracle import unet_ref as ref
    g = sfpkg.StaggeredGrid.from_origin(1.0 / shape[0], shape)
    rng = np.random.default_rng(7)
    P = ref.init_params(16, seed=17)
    for k in P:
        if k.endswith(".b"):
            P[k] = rng.normal(0, 0.05, P[k].shape).astype(np.float32)
    net = sfpkg.Network(gpu_ctx)
    net.set_params(ref.flatten(P))
    feat = torch.from_numpy(ref.bf16(rng.standard_normal(shape + (16,)))).to(torch.bfloat16).cuda().contiguous()
    dout = torch.from_numpy(rng.standard_normal(int(np.prod(shape))).astype(np.float32)).cuda()
    out0 = torch.zeros(g.num_cells, dtype=torch.float32, device="cuda")
    out1 = torch.zeros_like(out0)
    net.set_mode("mma")
    net.forward(g, feat, out0)
    g0 = net.gradients(g, feat, dout)
    net.set_mode("tcgen05_wgrad")
    g1 = net.gradients(g, feat, dout)
    net.set_mode("tcgen05")
    before = net.tc_launches()
    net.forward(g, feat, out1)
    torch.cuda.synchronize()
    assert net.tc_launches() > before
    a, b = out0.cpu().numpy(), out1.cpu().numpy()
    assert np.isfinite(b).all() and rel_l2(b, a) <= 1e-2
    # the head's weight and bias gradients against their definition, from the network's own last activations: db = sum
    # of dout, in FP64
    assert abs(g0[-1] - dout.double().sum().item()) <= 1e-4 * dout.double().abs().sum().item() / np.sqrt(dout.numel())
    off = 0
    for ci, co, taps in LAYERS:
        w, off = slice(off, off + taps * co * ci), off + taps * co * ci + co
        if np.abs(g0[w]).max() > 0:
            assert rel_l2(g1[w], g0[w]) <= 1e-4, (ci, co)
        np.testing.assert_array_equal(g1[w.stop:off], g0[w.stop:off])
    net.close()
