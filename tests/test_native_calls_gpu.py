"""GPU: the native calls (csrc/py_calls.cc) and the Python code behind them are one thing said twice: the same bits and the
same number of launches for what they take, the same errors for what they refuse."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16, F16, F32, F8, I8 = torch.bfloat16, torch.float16, torch.float32, torch.float8_e4m3fn, torch.int8


def both(pkg, monkeypatch, call):
    """call() by the native code and by Python: (bits or error, launches) of each."""
    assert pkg._NATIVE is not None
    answers = []
    for native in (True, False):
        with monkeypatch.context() as m:
            if not native:
                m.setattr(pkg, "_NATIVE", None)
            n0 = pkg.launch_count()
            try:
                got = [t.contiguous().view(torch.uint8).cpu() for t in call()]
            except Exception as e:      # noqa: BLE001 (whatever it is, both have to raise it)
                got = (type(e), str(e), getattr(e, "status", None))
            answers.append((got, pkg.launch_count() - n0))
    return answers


def rnd(*shape, dtype=BF16, seed=0, scale=0.3):
    g = torch.Generator(device="cuda").manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def gemm_calls(pkg):
    x, w, col = rnd(100, 256), rnd(256, 72), rnd(72, 256).t()
    bias, c = rnd(72), rnd(100, 72, seed=1)
    ws = torch.empty(16 << 20, dtype=torch.uint8, device="cuda")
    bx, bw = rnd(3, 40, 64, dtype=F16), rnd(3, 64, 48, dtype=F16)
    long, wide = rnd(300, 8192), rnd(8192, 128)
    i8 = lambda *s: rnd(*s, scale=20).to(I8)
    yield "plain", lambda: [pkg.gemm(x, w)]
    yield "column-major", lambda: [pkg.gemm(x, col, alpha=2.0)]
    yield "column-major operands", lambda: [pkg.gemm(rnd(256, 104).t(), col)]
    yield "column-major result", lambda: [pkg.gemm(x, w, bias=bias, epilogue="BIAS_GELU", out=torch.empty(72, 100, dtype=BF16, device="cuda").t())]
    yield "pitched result and C", lambda: [pkg.gemm(x, w, c=c.repeat(1, 2)[:, 72:], beta=-1, out=torch.empty(100, 144, dtype=BF16, device="cuda")[:, :72])]
    yield "epilogue", lambda: [pkg.gemm(x, w, bias=bias, c=c, beta=0.5, epilogue="BIAS_RELU")]
    yield "fp32 result", lambda: [pkg.gemm(x, w, out_dtype=F32, alpha=0.5)]
    yield "batched", lambda: [pkg.gemm(bx, bw)]
    yield "batched C", lambda: [pkg.gemm(bx, bw, c=rnd(3, 40, 48, dtype=F16), beta=2.0)]
    yield "fp32", lambda: [pkg.gemm(rnd(40, 64, dtype=F32), rnd(64, 32, dtype=F32))]
    yield "int8", lambda: [pkg.gemm(i8(64, 64), i8(64, 32), out_dtype=torch.int32)]
    yield "scratch", lambda: [pkg.gemm(long, wide, workspace=ws), pkg.gemm(long[:5], wide, workspace=ws)]
    yield "stream", lambda: [pkg.gemm(x, w, stream=torch.cuda.current_stream())]
    yield "empty", lambda: [pkg.gemm(x[:0], w)]
    yield "fp8", lambda: [pkg.gemm_fp8(long.to(F8), wide.to(F8), 0.5, 2), pkg.gemm_fp8(x.to(F8), col.to(F8), 0.5, 2.0, bias=bias, epilogue="BIAS")]
    yield "fp8, own result", lambda: [pkg.gemm_fp8(long.to(F8), wide.to(F8), 0.5, 2.0, out=torch.empty(300, 128, dtype=F16, device="cuda"), workspace=ws)]
    yield "fp8, stream", lambda: [pkg.gemm_fp8(long.to(F8), wide.to(F8), 0.5, 2.0, stream=torch.cuda.current_stream())]
    yield "fp8, torch's default type", lambda: [pkg.gemm_fp8(x.to(F8), col.to(F8), 0.5, 2.0, out_dtype=None)]
    yield "geglu", lambda: [pkg.gemm_geglu(x, w[:, :64], workspace=ws), pkg.gemm_geglu(x, w[:, :64]),
                            pkg.gemm_geglu(x, w[:, :64], out=torch.empty(100, 72, dtype=BF16, device="cuda")[:, :32], workspace=ws)]
    for name, bad in (("shape", lambda: pkg.gemm(x, w[:64])), ("layout", lambda: pkg.gemm(x[:, ::2], w)), ("rank", lambda: pkg.gemm(x[0], w)),
                      ("pitch", lambda: pkg.gemm(rnd(100, 250), rnd(250, 72))), ("bias", lambda: pkg.gemm(x, w, bias=bias)),
                      ("epilogue", lambda: pkg.gemm(x, w, epilogue="SILU")), ("host", lambda: pkg.gemm(x, w.cpu())),
                      ("host bias", lambda: pkg.gemm(x, w, bias=bias.cpu(), epilogue="BIAS")), ("type", lambda: pkg.gemm(x, w.double())),
                      ("types", lambda: pkg.gemm(x, w.half())), ("no C", lambda: pkg.gemm(x, w, beta=1.0)),
                      ("C", lambda: pkg.gemm(x, w, c=c.repeat(1, 2)[:, 72:], beta=1.0)), ("C type", lambda: pkg.gemm(x, w, c=c.float(), beta=1.0)),
                      ("alpha", lambda: pkg.gemm(x, w, alpha=float("inf"))), ("fp8 operands", lambda: pkg.gemm_fp8(x, w, 1.0, 1.0)),
                      ("geglu scratch", lambda: pkg.gemm_geglu(x, w[:, :64], workspace=ws[:64])), ("geglu columns", lambda: pkg.gemm_geglu(x, w[:, :72]))):
        yield f"refused: {name}", lambda bad=bad: [bad()]


def layer_calls(pkg):
    x, gain, tall = rnd(5, 7, 512), rnd(512), rnd(30, 6, 128)
    cos, sin = rnd(10, 32, dtype=F32), rnd(10, 32, dtype=F32, seed=2)
    cache, new = rnd(3, 20, 4, 64), rnd(3, 3, 4, 64)
    half = lambda t, **kw: pkg.rotary_interleaved_(t.clone(), cos, sin, 10, 64, **kw)

    def append(position, k=cache, n=new):
        kc, vc = k.clone(), k.clone()
        pkg.kv_append_(kc, vc, n[:, 1], n[:, 2], position)
        return [kc, vc]
    yield "norms", lambda: [pkg.row_norm(x), pkg.row_norm(x.half(), kind=pkg.NORM_RMS, eps=1e-6, gain=gain.half(), gain_offset=1),
                            pkg.row_norm(x, out=torch.empty_like(x), stream=torch.cuda.current_stream())]
    yield "rotary", lambda: [half(tall), half(tall, half_split=True), half(tall.half(), stream=torch.cuda.current_stream()),
                             half(rnd(30, 9, 128))[:, :6], pkg.rotary_half_(tall.clone(), cos, sin, 10, 64)]
    yield "append", lambda: append(0) + append(19) + append(7, cache.permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3))
    yield "residual", lambda: [pkg.residual_add(x, x), pkg.residual_add(x, x.view(35, 512), gain), pkg.residual_add(x, x, out=torch.empty_like(x))]
    for name, bad in (("norm", lambda: pkg.row_norm(x.transpose(0, 1))), ("norm out", lambda: pkg.row_norm(x, out=x[0])), ("norm type", lambda: pkg.row_norm(x.double())),
                      ("gain", lambda: pkg.row_norm(x, gain=gain[:8])), ("kind", lambda: pkg.row_norm(x, kind=7)),
                      ("tables", lambda: pkg.rotary_interleaved_(tall, cos[:5], sin, 10, 64)), ("dim", lambda: pkg.rotary_interleaved_(tall, rnd(10, 128, dtype=F32), rnd(10, 128, dtype=F32), 10, 256)),
                      ("position", lambda: append(20)), ("rows", lambda: append(0, cache, new[:2])), ("residual", lambda: pkg.residual_add(x, x[0])),
                      ("residual type", lambda: pkg.residual_add(x, x.half())), ("residual bias", lambda: pkg.residual_add(x, x, gain[:4]))):
        yield f"refused: {name}", lambda bad=bad: [bad()]


def attention_calls(pkg):
    B, N, F, T, H = 2, 3, 40, 200, 64
    q, k, v = rnd(B, F, N, H).permute(0, 2, 1, 3), rnd(B, T, N, H).permute(0, 2, 1, 3), rnd(B, N, T, H, seed=3)
    bias, shared = rnd(B, 1, F, T), rnd(B, 1, T, H).expand(B, N, T, H)
    go = rnd(B, N, F, H, seed=4)
    ws = torch.empty(16 << 20, dtype=torch.uint8, device="cuda")

    def forward(q=q, k=k, v=v, bias=None, train=False, **kw):
        out = torch.zeros(q.shape, dtype=q.dtype, device="cuda")
        lse = torch.zeros(q.shape[:3], device="cuda") if train else None
        pkg.fmha_forward_kernel(kw.pop("stream", None), q, k, v, bias, kw.pop("dropout", None), kw.pop("prob", 0.0), out, lse,
                                kw.pop("scale", H ** -0.5), train, **kw)
        return [out] + ([lse] if train else [])

    def backward(causal=False, bias=None, scale=0.125, lse_type=F32, **kw):
        out, lse = forward(bias=bias, train=True, causal=causal)
        dq, dk, dv = torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
        pkg.fmha_backward_kernel(None, q, k, v, out, bias, go, lse.to(lse_type), dq, dk, dv, scale, causal=causal, **kw)
        return [dq, dk, dv]
    yield "forward", lambda: forward() + forward(causal=True, train=True) + forward(bias=bias, train=True, workspace=ws)
    yield "shared keys", lambda: forward(k=shared, v=shared, scale=1) + forward(k=shared, v=shared, bias=bias.expand(B, N, F, T))
    yield "row bias", lambda: forward(bias=rnd(1, N, 1, T).expand(1, N, F, T))
    yield "decode", lambda: forward(q=q[:, :, :1], workspace=ws) + forward(q=q[:, :, :3]) + forward(q=q[:, :, :3], bias=bias[:, :, :3], causal=True)
    yield "fp16", lambda: forward(q=q.half(), k=k.half(), v=v.half(), stream=torch.cuda.current_stream(), prob=None)
    yield "backward", lambda: backward(workspace=ws) + backward(causal=True) + backward(bias=bias, workspace=ws)
    for name, bad in (("keys", lambda: forward(k=k[:, :2])), ("type", lambda: forward(k=k.half())), ("host", lambda: forward(v=v.cpu())),
                      ("bias", lambda: forward(bias=bias[:, :, :, :8])), ("bias type", lambda: forward(bias=bias.half())), ("scale", lambda: forward(scale=float("nan"))),
                      ("dropout", lambda: forward(prob=0.5)), ("mask", lambda: forward(dropout=q)), ("q", lambda: forward(q=q[:, :, :1].expand(B, N, 9, H))),
                      ("gradient's lse", lambda: backward(lse_type=F16)), ("gradient's scale", lambda: backward(scale=float("inf"), workspace=ws))):
        yield f"refused: {name}", bad


@pytest.mark.parametrize("family", [gemm_calls, layer_calls, attention_calls])
def test_native_calls_and_their_python_twins(pkg, cuda, monkeypatch, family):
    for name, call in family(pkg):
        (a, la), (b, lb) = both(pkg, monkeypatch, call)
        assert la == lb, name
        if isinstance(a, tuple) or isinstance(b, tuple):
            assert a == b and name.startswith("refused"), (name, a, b)
        else:
            assert not name.startswith("refused"), name
            assert all(torch.equal(s, t) for s, t in zip(a, b)) and len(a) == len(b) and a, name
