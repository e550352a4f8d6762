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


def _rows_of_the_last_tile(K, pairs):
    """Neurons of the last of the evenly shared tiles (one token tile): the layout rule of k_pair_gemm restated."""
    cover = -(-K // 64) * 64
    want = -(-(-(-cover // 128)) // pairs) * pairs
    tw = max(16, -(-(-(-cover // want)) // 8) * 8)
    return (cover - 1) % tw + 1


@pytest.mark.parametrize("B", [16, 64])
def test_a_last_tile_for_one_cta_of_the_pair(B):
    """The last tile has eight neurons, all of the even CTA's.  No bounded wait may run out over many steps with kernels
    of the layers ahead beside the launch: a stack reports that on its next step (the device status word)."""
    from sparse_transformers_b200 import SparseLayer, SparseStack
    from stxgpu import DEV

    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    H, r, L, dt = 4096, 32, 3, torch.bfloat16
    ks = [k for k in range(1024, 9216, 64) if _rows_of_the_last_tile(k, pairs) == 8]
    if not ks:
        pytest.skip("no such K with this number of SMs")
    k = ks[-1]
    I = k + 512
    g = torch.Generator(device=DEV).manual_seed(k)
    rn = lambda *s: (torch.randn(*s, generator=g, device=DEV) / 64).to(dt)
    ws = [(rn(I, H), rn(I, H), rn(H, I), rn(r, H), rn(I, r)) for _ in range(L)]
    layers = [SparseLayer(*w, act="silu", method="topk", param=k, max_batch=B) for w in ws]
    stack = SparseStack(layers, B)
    xs = [(64 * rn(1, H)).expand(B, H).contiguous() for _ in range(4)]  # equal rows: exactly k active neurons
    out = torch.empty(L, B, H, dtype=dt, device=DEV)
    for _ in range(500):
        for x in xs:
            stack.step(x, out)
    torch.cuda.synchronize()
    stack.step(xs[0], out)  # raises where a step before it recorded an expired wait
    torch.cuda.synchronize()
    x, eps = xs[0].double(), torch.finfo(dt).eps
    for l, (gate, up, down, _, _) in zip(range(L), ws):
        on = layers[l].mask()
        assert int(on.sum()) == layers[l].num_active() == k
        a = torch.nn.functional.silu(x @ gate[on].double().t()) * (x @ up[on].double().t())
        d = down[:, on].double().t()
        ref = a @ d
        # one rounding of each activation and of the result, at most eps / 2 of it; the rest is for the fp32 sums
        assert bool(((out[l].double() - ref).abs() <= eps * ref.abs() + eps * (a.abs() @ d.abs())).all())


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
