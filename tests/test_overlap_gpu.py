"""GPU: kernels that start while their predecessor runs and wait for it in front of their first access.

Chains of calls, each fed by the last, on the same buffers and scratch: eagerly and as a graph replay they give the bits of
the same chain in a process in which every launch waits for the one before (CUDA_LAUNCH_BLOCKING), kernels of one call
among them."""
import importlib
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def gemma_chain(pkg, dev, B):
    layers = importlib.import_module("ixk_b200.layers")
    hidden, heads, hd, ffn, T, steps = 1024, 4, 256, 4096, 600, 4
    g = torch.Generator(device=dev).manual_seed(B)
    r = lambda *s: (torch.randn(*s, generator=g, device=dev) * 0.02).bfloat16()
    w = [layers.GemmaLayerWeights(wqkv=r(hidden, 3 * heads * hd), wo=r(heads * hd, hidden), wgateup=r(hidden, 2 * ffn), wdown=r(ffn, hidden),
                                  heads_local=heads, head_dim=hd, norm_attn=r(hidden), norm_mlp=r(hidden)) for _ in range(2)]
    x0 = torch.randn(B, 1, hidden, generator=g, device=dev).bfloat16()
    caches = [torch.randn(B, T, heads, hd, generator=g, device=dev).bfloat16() for _ in range(4)]
    ops = layers.KernelOps(pkg, gemm_workspace=torch.empty(32 << 20, dtype=torch.uint8, device=dev))
    workspace = torch.empty(8 << 20, dtype=torch.uint8, device=dev)
    ropes = [layers.rotary_tables(torch.tensor([T - steps + i], device=dev), hd) for i in range(steps)]

    def run():
        c, x = [t.clone() for t in caches], x0
        for i in range(steps):
            for n in range(2):
                x = layers.gemma_decode_step(x, w[n], c[2 * n], c[2 * n + 1], T - steps + i, ops, workspace=workspace, rope=ropes[i])
            x = pkg.residual_add(x, x)      # (no layer between: the next step's first norm reads what this one writes)
        return [x, *c]
    return run


def gptj_chain(pkg, dev):
    layers = importlib.import_module("ixk_b200.layers")
    hidden, heads, hd, rot, ffn, B, S = 512, 2, 256, 64, 1024, 2, 320
    g = torch.Generator(device=dev).manual_seed(1)
    r = lambda *s: (torch.randn(*s, generator=g, device=dev) * 0.05).bfloat16()
    full = {"wqkv": r(hidden, 3 * heads * hd), "wo": r(heads * hd, hidden), "w1": r(hidden, ffn), "b1": r(ffn), "w2": r(ffn, hidden), "b2": r(hidden)}
    w = layers.GptJLayerWeights.shard(full, heads, hd, rot, 0, 1)
    x0, ops = torch.randn(B, S, hidden, generator=g, device=dev).bfloat16(), layers.KernelOps(pkg)
    rope = layers.rotary_tables(torch.arange(S, device=dev), rot)

    def run():
        x = x0
        for _ in range(4):
            x = layers.gptj_layer_prefill(x, w, ops, rope=rope)
        return [x]
    return run


def training_chain(pkg, dev, H, S, causal):
    """Forward and backward, each step's inputs the normalised gradients of the last.  (At most two key blocks up to head
    size 128: two fp32 addends make one sum in either order.)"""
    B, N = 2, 3
    g = torch.Generator(device=dev).manual_seed(H)
    q0, k0, v0, go = (torch.randn(B, N, S, H, generator=g, device=dev).bfloat16() for _ in range(4))
    lse, out = torch.empty(B, N, S, device=dev), torch.empty_like(q0)
    dq, dk, dv = (torch.empty_like(q0) for _ in range(3))
    need = max(pkg.fmha_workspace_bytes(q0, k0, v0, None, out, H ** -0.5, causal),
               pkg.fmha_backward_workspace_bytes(q0, k0, v0, out, None, go, dq, dk, dv, H ** -0.5, causal))
    ws = torch.empty(need, dtype=torch.uint8, device=dev)

    def run():
        q, k, v = q0, k0, v0
        for _ in range(4):
            pkg.fmha_forward_kernel(None, q, k, v, None, None, 0.0, out, lse, H ** -0.5, True, causal=causal, workspace=ws)
            pkg.fmha_backward_kernel(None, q, k, v, out, None, go, lse, dq, dk, dv, H ** -0.5, causal=causal, workspace=ws)
            q, k, v = pkg.row_norm(dq), pkg.row_norm(dk), pkg.row_norm(dv)
        return [q, k, v, out.clone(), lse.clone()]
    return run


def attention_chain(pkg, dev):
    """Short, split and whole prefill, biases by TMA and by words, and decode of one row and several, over one buffer."""
    g = torch.Generator(device=dev).manual_seed(5)
    B, N, H = 1, 4, 128
    r = lambda *s: torch.randn(*s, generator=g, device=dev).bfloat16()
    x0, kv = r(B, N, 1500, H), r(B, N, 1500, H)
    sizes = [(300, 100, None), (1500, 1500, None), (260, 700, 704), (260, 701, 701), (1, 1500, None), (8, 1100, None), (1, 60, None)]
    biases = [None if p is None else r(1, 1, F, p)[..., :T] for F, T, p in sizes]
    ws = torch.empty(64 << 20, dtype=torch.uint8, device=dev)

    def run():
        x, got = x0.clone(), []
        for _ in range(2):
            for (F, T, _), bias in zip(sizes, biases):
                q, o = x[:, :, -F:], x.new_empty(B, N, F, H)
                pkg.fmha_forward_kernel(None, q, x[:, :, :T], kv[:, :, :T], bias, None, 0.0, o, None, H ** -0.5, False, workspace=ws)
                pkg.row_norm(o, out=o)
                pkg.kv_append_(x.permute(0, 2, 1, 3), kv.permute(0, 2, 1, 3).clone(), o[:, :, -1], o[:, :, -1], T - 1)
                got.append(o)
        return got + [x]
    return run


def gemm_chain(pkg, dev):
    """Products of a few rows, of CTA pairs with a bias and C, cut along K, and fp8, each from the last one's result."""
    g = torch.Generator(device=dev).manual_seed(6)
    r = lambda *s: (torch.randn(*s, generator=g, device=dev) * 0.05).bfloat16()
    x0, w1, b1, w2, w3, c3 = r(2600, 512), r(512, 4096), r(4096), r(4096, 512), r(512, 512), r(300, 512)
    f8 = r(4096, 512).to(torch.float8_e4m3fn)
    ws = torch.empty(64 << 20, dtype=torch.uint8, device=dev)

    def run():
        x, got = x0, []
        for rows in (2600, 300, 100, 1, 2600):
            x = x0 if rows == 2600 else x
            h = pkg.row_norm(x[:rows])
            up = pkg.gemm(h, w1, bias=b1, epilogue="BIAS_GELU", workspace=ws)
            x = pkg.gemm(up, w2, c=h, beta=1.0, workspace=ws)
            if rows == 300:
                x = pkg.gemm(x, w3, c=c3, beta=0.5, workspace=ws)
            got += [up, x, pkg.gemm_fp8(up.to(torch.float8_e4m3fn), f8, 0.5, 0.5)]
        return got
    return run


CHAINS = {
    "gemma-1": lambda pkg, dev: gemma_chain(pkg, dev, 1),
    "gemma-5": lambda pkg, dev: gemma_chain(pkg, dev, 5),
    "gptj": gptj_chain,
    "training-64": lambda pkg, dev: training_chain(pkg, dev, 64, 250, False),
    "training-128": lambda pkg, dev: training_chain(pkg, dev, 128, 200, True),
    "training-256": lambda pkg, dev: training_chain(pkg, dev, 256, 300, True),
    "attention": attention_chain,
    "gemm": gemm_chain,
}


def main(path):
    """Every chain, each launch after the end of the one before."""
    sys.path.insert(0, ROOT)
    import __graft_entry__ as entry
    pkg, dev = entry.load_package(), torch.device("cuda:0")
    results = {}
    for name, make in CHAINS.items():
        run = make(pkg, dev)
        run()
        assert torch.cuda.current_stream().query()      # nothing is in flight when a call returns
        results[name] = [t.cpu() for t in run()]
    assert pkg.device_status() == 0
    torch.save(results, path)


@pytest.fixture(scope="module")
def one_at_a_time(cuda, tmp_path_factory):
    path = str(tmp_path_factory.mktemp("chains") / "results.pt")
    r = subprocess.run([sys.executable, os.path.abspath(__file__), path], env={**os.environ, "CUDA_LAUNCH_BLOCKING": "1"},
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    return torch.load(path)


@pytest.mark.parametrize("name", list(CHAINS))
def test_chains_overlap_without_changing_a_bit(pkg, cuda, one_at_a_time, name):
    want = [t.to(cuda) for t in one_at_a_time[name]]
    assert all(torch.isfinite(t.float()).all() for t in want)
    run = CHAINS[name](pkg, cuda)

    def check(got):
        assert len(got) == len(want) and all(torch.equal(a, b) for a, b in zip(got, want))
    for _ in range(5):
        check(run())
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        got = run()
    for _ in range(3):
        for t in got:
            t.zero_()
        graph.replay()
        check(got)
    del graph


if __name__ == "__main__":
    main(sys.argv[1])
