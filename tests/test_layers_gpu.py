"""GPU parity: the decoder-layer drivers (GEMM + attention kernels + torch glue) on one GPU against
the un-sharded numpy layer oracle, at reduced sizes the oracle finishes in seconds.
Tolerance: activations are O(1) and stored in bf16 between kernels, so 6e-2 absolute (a few bf16
ulps accumulated over the block), plus the bf16 relative bound 2e-2."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def f32(t):
    return t.float().cpu().numpy()


def test_gptj_block_prefill(pkg, orc, cuda):
    from oracle import layers_oracle
    layers = importlib.import_module("ixk_b200.layers")
    hidden, heads, hd, rot, ffn, B, S = 512, 2, 256, 64, 1024, 2, 320
    g = torch.Generator().manual_seed(1)
    r = lambda *s: (torch.randn(*s, generator=g) * 0.02).bfloat16()
    full = {"wqkv": r(hidden, 3 * heads * hd), "wo": r(heads * hd, hidden), "w1": r(hidden, ffn), "b1": r(ffn),
            "w2": r(ffn, hidden), "b2": r(hidden)}
    x = torch.randn(B, S, hidden, generator=g).bfloat16()
    w = layers.GptJLayerWeights.shard({k: v.to(cuda) for k, v in full.items()}, heads, hd, rot, 0, 1)
    y = layers.gptj_layer_prefill(x.to(cuda), w, layers.KernelOps(pkg))
    want = layers_oracle.gptj_layer_prefill(f32(x), {k: f32(v) for k, v in full.items()}, heads, hd, rot)
    orc.check_close(f32(y), want, rtol=2e-2, atol=6e-2, what="gptj block")


def test_gemma_decode_step(pkg, orc, cuda):
    from oracle import layers_oracle
    layers = importlib.import_module("ixk_b200.layers")
    hidden, heads, hd, ffn, B, T = 384, 2, 256, 768, 5, 700
    g = torch.Generator().manual_seed(2)
    r = lambda *s: (torch.randn(*s, generator=g) * 0.02).bfloat16()
    full = {"wqkv": r(hidden, 3 * heads * hd), "wo": r(heads * hd, hidden), "wgate": r(hidden, ffn),
            "wup": r(hidden, ffn), "wdown": r(ffn, hidden),
            "norm_attn": r(hidden), "norm_mlp": r(hidden)}
    x = torch.randn(B, 1, hidden, generator=g).bfloat16()
    kc = torch.randn(B, T, heads, hd, generator=g).bfloat16()
    vc = torch.randn(B, T, heads, hd, generator=g).bfloat16()
    w = layers.GemmaLayerWeights.shard({k: v.to(cuda) for k, v in full.items()}, heads, hd, 0, 1)
    kd, vd = kc.to(cuda), vc.to(cuda)
    y = layers.gemma_decode_step(x.to(cuda), w, kd, vd, T - 1, layers.KernelOps(pkg))
    want = layers_oracle.gemma_decode_step(f32(x), {k: f32(v) for k, v in full.items()}, f32(kc), f32(vc), T - 1, heads, hd)
    orc.check_close(f32(y), want, rtol=2e-2, atol=6e-2, what="gemma decode")
    assert not torch.equal(kd[:, T - 1].cpu(), kc[:, T - 1])      # the new key was written into the cache


def test_gptj_block_at_full_width(pkg, orc, cuda):
    """Configuration 4's layer at its real widths (hidden 4096, 16 heads x 256, rotary 64, MLP 16384,
    weights ~ N(0, 0.02)), with batch and sequence cut to what the numpy oracle finishes in seconds
    (2 x 320 tokens instead of 4 x 2048; 320 is not a multiple of the 128-row tiles)."""
    from oracle import layers_oracle
    layers = importlib.import_module("ixk_b200.layers")
    hidden, heads, hd, rot, ffn, B, S = 4096, 16, 256, 64, 16384, 2, 320
    g = torch.Generator().manual_seed(3)
    r = lambda *s: (torch.randn(*s, generator=g) * 0.02).bfloat16()
    full = {"wqkv": r(hidden, 3 * heads * hd), "wo": r(heads * hd, hidden), "w1": r(hidden, ffn), "b1": r(ffn),
            "w2": r(ffn, hidden), "b2": r(hidden)}
    x = torch.randn(B, S, hidden, generator=g).bfloat16()
    w = layers.GptJLayerWeights.shard({k: v.to(cuda) for k, v in full.items()}, heads, hd, rot, 0, 1)
    y = layers.gptj_layer_prefill(x.to(cuda), w, layers.KernelOps(pkg))
    want = layers_oracle.gptj_layer_prefill(f32(x), {k: f32(v) for k, v in full.items()}, heads, hd, rot)
    orc.check_close(f32(y), want, rtol=2e-2, atol=6e-2, what="gptj block, full width")


def test_gemma_decode_step_at_full_width(pkg, orc, cuda):
    """Configuration 5's step at its real widths (hidden 3072, 16 heads x 256, GeGLU 24576: the
    K = 24576 down projection runs split along K), 8 sequences against a cache of 1100 keys
    instead of 64 against 4096."""
    from oracle import layers_oracle
    layers = importlib.import_module("ixk_b200.layers")
    hidden, heads, hd, ffn, B, T = 3072, 16, 256, 24576, 8, 1100
    g = torch.Generator().manual_seed(4)
    r = lambda *s: (torch.randn(*s, generator=g) * 0.02).bfloat16()
    full = {"wqkv": r(hidden, 3 * heads * hd), "wo": r(heads * hd, hidden), "wgate": r(hidden, ffn),
            "wup": r(hidden, ffn), "wdown": r(ffn, hidden),
            "norm_attn": r(hidden), "norm_mlp": r(hidden)}
    x = torch.randn(B, 1, hidden, generator=g).bfloat16()
    kc = torch.randn(B, T, heads, hd, generator=g).bfloat16()
    vc = torch.randn(B, T, heads, hd, generator=g).bfloat16()
    w = layers.GemmaLayerWeights.shard({k: v.to(cuda) for k, v in full.items()}, heads, hd, 0, 1)
    ops = layers.KernelOps(pkg, gemm_workspace=torch.empty(32 << 20, dtype=torch.uint8, device=cuda))
    n0 = pkg.launch_count()
    y = layers.gemma_decode_step(x.to(cuda), w, kc.to(cuda), vc.to(cuda), T - 1, ops)
    assert pkg.launch_count() - n0 >= 5 * 2 + 2       # every projection split along K (+ reduce), attention + combine
    want = layers_oracle.gemma_decode_step(f32(x), {k: f32(v) for k, v in full.items()}, f32(kc), f32(vc), T - 1, heads, hd)
    orc.check_close(f32(y), want, rtol=2e-2, atol=6e-2, what="gemma decode, full width")


@pytest.mark.parametrize("B", [1, 5])
def test_decode_steps_overlap_without_changing_a_bit(pkg, cuda, monkeypatch, B):
    """The kernels of a decode step start while their predecessors run and wait for them in front of their first
    access.  Twelve steps over two layers' weights, each fed by the last, on the same buffers and scratch: the bits
    of the same chain with the device idle before every launch, eagerly and as a graph replay."""
    layers = importlib.import_module("ixk_b200.layers")
    hidden, heads, hd, ffn, T, steps = 1024, 4, 256, 4096, 600, 6
    g = torch.Generator(device=cuda).manual_seed(B)
    r = lambda *s: (torch.randn(*s, generator=g, device=cuda) * 0.02).bfloat16()
    weights = [layers.GemmaLayerWeights(wqkv=r(hidden, 3 * heads * hd), wo=r(heads * hd, hidden), wgateup=r(hidden, 2 * ffn),
                                        wdown=r(ffn, hidden), heads_local=heads, head_dim=hd, norm_attn=r(hidden), norm_mlp=r(hidden))
               for _ in range(2)]
    x0 = torch.randn(B, 1, hidden, generator=g, device=cuda).bfloat16()
    caches = [torch.randn(B, T, heads, hd, generator=g, device=cuda).bfloat16() for _ in range(4)]
    ops = layers.KernelOps(pkg, gemm_workspace=torch.empty(32 << 20, dtype=torch.uint8, device=cuda))
    workspace = torch.empty(8 << 20, dtype=torch.uint8, device=cuda)
    ropes = [layers.rotary_tables(torch.tensor([T - steps + i], device=cuda), hd) for i in range(steps)]

    def chain(c):
        x = x0
        for i in range(steps):
            for n, w in enumerate(weights):
                x = layers.gemma_decode_step(x, w, c[2 * n], c[2 * n + 1], T - steps + i, ops, workspace=workspace, rope=ropes[i])
            x = pkg.residual_add(x, x)      # (no layer between: the next step's first norm reads what this one writes)
        return x
    stream_of = pkg._stream_ptr

    def idle_first(stream):
        torch.cuda.synchronize()
        return stream_of(stream)
    with monkeypatch.context() as m:
        m.setattr(pkg, "_stream_ptr", idle_first)
        apart = [c.clone() for c in caches]
        want = chain(apart)
    torch.cuda.synchronize()
    for _ in range(5):
        together = [c.clone() for c in caches]
        got = chain(together)
        assert torch.equal(got, want) and all(torch.equal(a, b) for a, b in zip(together, apart))
    together = [c.clone() for c in caches]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        got = chain(together)
    for _ in range(3):
        for t, c in zip(together, caches):
            t.copy_(c)
        graph.replay()
        assert torch.equal(got, want) and all(torch.equal(a, b) for a, b in zip(together, apart))
    del graph
