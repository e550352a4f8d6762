"""Edges of the two-CTA tensor-core kernel behind row blocks (k_pair_gemm) and of the row-block predictor kernels:
token tiles of 32 to 256, neurons that do not fill a tile, contraction lengths around a k block, split contractions."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,H,K,act", [
    (9, 64, 64, "relu"),        # one k block, one partial tile, the smallest block of rows
    (33, 192, 65, "silu"),      # 64 tokens of which 33 exist, one neuron beyond a k block, H not a multiple of the tile
    (64, 1024, 1777, "silu"),   # evenly shared neurons, split contraction, odd K (activations through the scratch)
    (256, 320, 132, "relu"),    # the widest token tile
    (257, 256, 200, "gelu_pytorch_tanh"),   # two token tiles, the second with one token less than the first
    (530, 128, 19000, "relu"),  # several waves of tiles: both accumulators and the stage ring wrap around
])
def test_against_torch_fp32(dtype, B, H, K, act):
    from stxgpu import DEV, mlp_forward

    g = torch.Generator().manual_seed(B * 7 + K)
    x = torch.randn(B, H, generator=g).to(dtype).to(DEV)
    cw = (torch.randn(2 * K, H, generator=g) / np.sqrt(H)).to(dtype).to(DEV)
    dp = (torch.randn(K, H, generator=g) / np.sqrt(K)).to(dtype).to(DEV)
    out, comb = mlp_forward(x, cw, dp, act)
    gate, up = (x.double() @ cw.double().t()).chunk(2, dim=-1)
    f = {"relu": torch.relu, "silu": torch.nn.functional.silu,
         "gelu_pytorch_tanh": lambda t: torch.nn.functional.gelu(t, approximate="tanh")}[act]
    a = f(gate) * up
    # one rounding of a result is at most eps/2 of it; fp32 sums of up to 19000 terms stay far below that
    eps = torch.finfo(dtype).eps
    # |a| near zero: the fp32 error of g and u, not the rounding of a, is what is left
    assert bool(((comb[:, :K].double() - a).abs() <= eps * a.abs() + 1e-5 * a.abs().max()).all())
    assert bool(((comb[:, K:].double() - up).abs() <= eps * up.abs() + 1e-5 * up.abs().max()).all())
    ref = comb[:, :K].double() @ dp.double()  # the second contraction on the activations as they were rounded
    assert bool(((out.double() - ref).abs() <= eps * ref.abs() + 1e-4 * ref.abs().max()).all())


@pytest.mark.parametrize("K", [1000, 1016, 8704 + 64])
def test_a_last_tile_for_one_cta_of_the_pair(K):
    """The last tile has eight neurons, all of the even CTA's: no wait of the odd one may run out (each costs about a second)."""
    from stxgpu import DEV, mlp_forward

    H, B = 4096, 64
    g = torch.Generator(device=DEV).manual_seed(K)
    rn = lambda *s: (torch.randn(*s, generator=g, device=DEV) / 64).to(torch.bfloat16)
    x, cw, dp = rn(B, H), rn(2 * K, H), rn(K, H)
    first, slow = None, 0
    for _ in range(150):
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        out, _ = mlp_forward(x, cw, dp, "silu")
        t1.record()
        t1.synchronize()
        slow += t0.elapsed_time(t1) > 300.0
        first = out if first is None else first
        assert torch.equal(out, first)
    assert slow <= 3  # a busy host may stall a call or two


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,H,r,I,density", [
    (9, 4096, 32, 100, 0.1),      # smallest row block
    (65, 512, 64, 1030, 0.002),   # one row beyond a block of the scores kernel, hardly any bit set
    (300, 256, 30, 333, 0.01),    # r that the tensor-core scores do not take
    (1300, 256, 32, 2050, 0.0005),  # three chunks of rows, the union is not full after the first two
    (600, 256, 32, 2050, 0.2),    # the union is full after the first chunk
    (12, 16384, 32, 64, 0.1),     # more chunks than threads
])
def test_row_block_masks_bit_exact(dtype, B, H, r, I, density):
    from statistics import NormalDist
    from stxgpu import DEV, ODT, predict_mask

    g = torch.Generator().manual_seed(B + H + I)
    x = torch.randn(B, H, generator=g).to(dtype)
    A = (torch.randn(r, H, generator=g) * 0.02).to(dtype)
    Bm = (torch.randn(I, r, generator=g) * 0.02).to(dtype)
    tau = 0.02 ** 2 * np.sqrt(H * r) * NormalDist().inv_cdf(1 - density)
    mask, _, bits = predict_mask(x.to(DEV), A.to(DEV), Bm.to(DEV), param=tau, want_scores=False)
    _, s_ref = orc.predictor(x.float().numpy(), A.float().numpy(), Bm.float().numpy(), ODT[dtype])
    _, uni = orc.mask_threshold(s_ref, ODT[dtype], tau)
    assert np.array_equal(mask.cpu().numpy(), uni)
    if I % 32:
        assert int(bits.cpu().numpy().view(np.uint32)[-1]) >> (I % 32) == 0
