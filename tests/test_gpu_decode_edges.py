"""Edges of the decode-time kernels: splits of the attention keys, the end of a greedy step, finished masks through the
one-kernel layer path, stacks whose predictors run ahead of their layers."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("hd,heads,kv", [(64, 8, 2), (128, 6, 2), (256, 4, 4), (64, 12, 6), (128, 7, 1), (256, 4, 1), (64, 32, 8), (128, 32, 4), (256, 32, 8)])
def test_attention_splits(dtype, hd, heads, kv):
    from sparse_transformers_b200.llama_skip import LlamaSkipConfig, apply_rope, attn_decode, attn_workspace, rope_tables

    max_len = 8192
    g = torch.Generator(device=DEV).manual_seed(hd + heads)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV).to(dtype)
    cos, sin = rope_tables(LlamaSkipConfig(head_dim=hd, max_len=max_len), DEV)
    kc, vc, ws = rn(kv, max_len, hd), rn(kv, max_len, hd), attn_workspace(heads, hd, DEV)
    eps = torch.finfo(dtype).eps
    for pos in (0, 1, 47, 48, 97, 128, 129, 256, 257, 300, 512, 513, 1023, 1024, 1025, 4097, 8191):  # one block up to two tiles
        qkv = rn((heads + 2 * kv) * hd)
        k0, v0 = kc.clone(), vc.clone()
        out = attn_decode(qkv, cos, sin, torch.tensor([pos], device=DEV), kc, vc, torch.zeros(1, heads * hd, dtype=dtype, device=DEV),
                          heads, kv, hd, ws).view(heads, hd).double()
        q, k, v = qkv.split([heads * hd, kv * hd, kv * hd])
        q = apply_rope(q.view(heads, 1, hd), cos[pos:pos + 1], sin[pos:pos + 1])[:, 0].double()
        k0[:, pos] = apply_rope(k.view(kv, 1, hd), cos[pos:pos + 1], sin[pos:pos + 1])[:, 0]
        v0[:, pos] = v.view(kv, hd)
        assert torch.equal(kc, k0) and torch.equal(vc, v0)
        s = torch.einsum("grd,gnd->grn", q.view(kv, heads // kv, hd), k0[:, :pos + 1].double()) / math.sqrt(hd)
        ref = torch.einsum("grn,gnd->grd", torch.softmax(s, -1), v0[:, :pos + 1].double()).reshape(heads, hd)
        # the result is rounded once (eps / 2); scores of fp32 sums of hd terms move a weight by about 1e-5 of it
        assert bool(((out - ref).abs() <= eps * ref.abs() + 3e-5 * v0.double().abs().max()).all()), pos
    assert int(ws[:4096].view(torch.int32).abs().sum()) == 0, "the arrival counters are left zeroed"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("V", [1, 255, 257, 128256])
def test_decode_finish(dtype, V):
    from sparse_transformers_b200.llama_skip import decode_finish

    g = torch.Generator(device=DEV).manual_seed(V)
    ws = torch.zeros(16, dtype=torch.uint8, device=DEV)
    i64 = lambda *v: torch.tensor(v, dtype=torch.long, device=DEV)
    base = torch.randn(V, generator=g, device=DEV).to(dtype)
    zeros = torch.zeros(V, dtype=dtype, device=DEV)
    zeros[V // 2:] = -0.0
    ties, nan = base.clone(), base.clone()
    ties[[V // 3, V - 1]] = 40.0
    nan[V - 1] = float("nan")
    low = torch.full((V,), torch.finfo(dtype).min, dtype=dtype, device=DEV)
    inf = torch.full((V,), float("-inf"), dtype=dtype, device=DEV)
    for logits in (base, ties, nan, zeros, -zeros, low, inf):
        out, token, pos, gen = torch.zeros(V, device=DEV), i64(-1), i64(6), torch.zeros(4, dtype=torch.long, device=DEV)
        decode_finish(logits, out, token, pos, i64(5), gen, ws)
        want = int(torch.isnan(logits.float()).nonzero()[0]) if torch.isnan(logits.float()).any() else int(
            (logits == logits.max()).nonzero()[0])
        assert int(token) == want and int(pos) == 7 and gen.tolist() == [0, 0, want, 0]
        assert torch.equal(out.nan_to_num(7.5), logits.float().nan_to_num(7.5))
    decode_finish(base, out, token, i64(8), i64(5), gen, ws)  # index 4 lies outside
    assert gen.tolist() == [0, 0, want, 0] and int(ws.sum()) == 0


@pytest.mark.parametrize("rule,param", [("topk", 90), ("topk", 333), ("statistical_topk", 1.0)])
@pytest.mark.parametrize("B,dtype,scale", [(1, torch.float32, 1.0), (1, torch.bfloat16, 1.0), (2, torch.float16, 1.0), (5, torch.bfloat16, 1.0),
                                           (8, torch.float16, 1.0), (3, torch.float16, 90.0)])
def test_finished_masks_through_the_layer(rule, param, B, dtype, scale):
    """scale 90: activations of up to about 1e6, beyond fp16, whose products are in range again."""
    from sparse_transformers_b200 import SparseLayer

    H, I, r = 512, 333, 32
    g = torch.Generator(device=DEV).manual_seed(B + int(param))
    rn = lambda *s, std=1.0: (torch.randn(*s, generator=g, device=DEV) * std).to(dtype)
    gate, up = rn(I, H, std=0.05 * scale), rn(I, H, std=0.05 * scale)
    down, A, Bm = rn(H, I, std=0.05 / scale ** 2), rn(r, H, std=0.02), rn(I, r, std=0.02)
    layer = SparseLayer(gate, up, down, A, Bm, act="silu", method=rule, param=param, max_batch=B)
    for _ in range(3):
        x = rn(B, H, std=2.0 if scale > 1 else 1.0)
        out = layer.step(x).double()
        on = layer.mask()
        assert sorted(layer.active_indices().tolist()) == on.nonzero().flatten().tolist()
        if rule == "topk":
            assert int(on.sum()) >= param
        u = x.double() @ up[on].double().t()
        a = torch.nn.functional.silu(x.double() @ gate[on].double().t()) * u
        ref = a @ down[:, on].double().t()
        size = a.abs() @ down[:, on].double().abs().t()  # of the terms: what the sums' own rounding scales with
        fi = torch.finfo(dtype)
        # fp32 sums of 512 and 333 terms (2e-5), one rounding of the result: half a step of the smallest numbers at least
        assert bool(((out - ref).abs() <= fi.eps * ref.abs() + 2e-5 * size + fi.eps * fi.smallest_normal).all())
        if scale > 1:
            assert float(a.abs().max()) > 65504


def _mlp_terms(x, gate, up, down, on):
    """act(g) * u of the active neurons in 64 bits, the result, and the size of its terms (what the sums' rounding scales with)."""
    a = torch.nn.functional.silu(x.double() @ gate[on].double().t()) * (x.double() @ up[on].double().t())
    d = down[:, on].double().t()
    return a, a @ d, a.abs() @ d.abs()


@pytest.mark.parametrize("dtype,H,I,k,scales,wd", [
    (torch.float16, 4096, 6000, 900, (12000.0, 1.0, 0.1, 0.03), 0.05),   # 20 and more neurons a CTA: several tiles of six
    (torch.float16, 512, 3000, 2500, (3e-3, 3e-3), 1.0),                 # activations around 1e-6, tiles of eight
    (torch.float16, 1024, 4736, 1500, (1.0,) * 8, 0.05),
    (torch.bfloat16, 2048, 6000, 1200, (1e4, 1.0, 1e-4), 0.05),
    (torch.bfloat16, 512, 200, 3, (1.0, 1.0, 1.0, 1.0, 1.0), 0.05),      # fewer neurons than CTAs
])
def test_finished_masks_keep_rows_apart_and_fp32_activations(dtype, H, I, k, scales, wd):
    from sparse_transformers_b200 import SparseLayer

    B, r = len(scales), 32
    g = torch.Generator(device=DEV).manual_seed(H + k)
    rn = lambda *s, std=1.0: (torch.randn(*s, generator=g, device=DEV) * std).to(dtype)
    gate, up, down = rn(I, H, std=0.02), rn(I, H, std=0.02), rn(H, I, std=wd)
    layer = SparseLayer(gate, up, down, rn(r, H, std=0.02), rn(I, r, std=0.02), act="silu", method="topk", param=k, max_batch=B)
    fi = torch.finfo(dtype)
    for _ in range(2):
        x_pred = rn(B, H)
        x = (x_pred.float() * torch.tensor(scales, device=DEV)[:, None]).to(dtype)
        out = layer.step(x_pred, x)
        on = layer.mask()
        _, ref, size = _mlp_terms(x, gate, up, down, on)
        # one rounding of the result (half a step of the smallest numbers at least); fp32 sums of H and of K terms
        bound = fi.eps * ref.abs() + fi.smallest_normal * fi.eps + 2e-5 * size
        fits = ref.abs() < 0.99 * fi.max
        assert bool(((out.double() - ref).abs() <= bound)[fits].all())
        for other in (0.0, float("inf"), float("nan")):  # what stands in row 0 is nothing to the other rows
            x2 = x.clone()
            x2[0] = other
            assert torch.equal(layer.step(x_pred, x2)[1:], out[1:]), other


@pytest.mark.parametrize("B", [2, 8, 12, 70])
def test_stack_with_predictors_ahead_equals_eager_layers(B):
    from sparse_transformers_b200 import SparseLayer, SparseStack

    H, I, r, L, dt = 512, 1030, 32, 3, torch.float16
    g = torch.Generator(device=DEV).manual_seed(B)
    rn = lambda *s, std=1.0: (torch.randn(*s, generator=g, device=DEV) * std).to(dt)
    ws = [(rn(I, H, std=0.05), rn(I, H, std=0.05), rn(H, I, std=0.05), rn(r, H, std=0.02), rn(I, r, std=0.02)) for _ in range(L)]
    tau = 0.02 ** 2 * math.sqrt(H * r) * 1.3
    mk = lambda: [SparseLayer(*w, act="silu", param=tau, max_batch=B) for w in ws]
    eager, stacked = mk(), mk()
    stack = SparseStack(stacked, B)
    out = torch.empty(L, B, H, dtype=dt, device=DEV)
    for _ in range(4):
        x = rn(B, H)
        stack.step(x, out)
        for i, l in enumerate(eager):
            assert torch.equal(l.step(x), out[i])
            assert torch.equal(l.mask(), stacked[i].mask())
            assert torch.equal(l.active_indices(), stacked[i].active_indices())
            assert torch.equal(l.concat_weight(), stacked[i].concat_weight())
    # the same layer twice in one stack: served one after the other
    both = SparseStack([stacked[0], stacked[0]], B)
    two = torch.empty(2, B, H, dtype=dt, device=DEV)
    both.step(x, two)
    assert torch.equal(two[0], out[0]) and torch.equal(two[1], out[0])


@pytest.mark.parametrize("H,I", [(512, 2048), (4096, 8192), (8192, 9000)])
def test_norm_gemv_waits_for_the_kernel_that_writes_its_weights(H, I):
    """The row copies of a cache update let the next kernel of the stream start before they are through."""
    import ctypes

    from stxgpu import Cache, stream

    from sparse_transformers_b200 import _capi as C
    from sparse_transformers_b200.llama_skip import norm_gemv

    dt = torch.float16
    g = torch.Generator(device=DEV).manual_seed(H)
    up = (torch.randn(I, H, generator=g, device=DEV) * 0.02).to(dt)
    cache = Cache(up, up, up.t().contiguous())
    pk = ctypes.c_void_p()
    C.check(C.lib.stx_cache_packed_ptrs(cache.h, None, ctypes.byref(pk), None, None))
    h, a, wn = (torch.randn(1, H, generator=g, device=DEV).to(dt) for _ in range(3))
    masks = [torch.arange(I, device=DEV) % 2 == i for i in (0, 1)]
    K = int(masks[0].sum())
    masks[1][: K - int(masks[1].sum())] = True  # as many in both

    class Packed:
        __cuda_array_interface__ = {"shape": (K * H * 2,), "typestr": "|u1", "data": (pk.value, False), "version": 2}

    W = torch.as_tensor(Packed(), device=DEV).view(dt).view(K, H)
    own = torch.empty(K, H, dtype=dt, device=DEV)
    for it in range(12):
        C.check(C.lib.stx_cache_update(cache.h, masks[it % 2].data_ptr(), stream()))
        first = norm_gemv(h, None, None, 0.0, W) if it % 3 else norm_gemv(h, a, wn, 1e-5, W)
        torch.cuda.synchronize()
        assert torch.equal(first, norm_gemv(h, None, None, 0.0, W) if it % 3 else norm_gemv(h, a, wn, 1e-5, W))
        torch.mul(W, float(it + 1), out=own)  # a torch kernel in front
        first = norm_gemv(h, None, None, 0.0, own)
        torch.cuda.synchronize()
        assert torch.equal(first, norm_gemv(h, None, None, 0.0, own))
