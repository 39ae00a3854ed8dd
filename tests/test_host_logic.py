"""CPU: the host-side mirror — layout attributes derived from tensor views, and the checks the
reference's runners make before launching."""
import contextlib
import types

import pytest
import torch


def test_gemm_attrs_row_and_col_major(pkg):
    a = torch.zeros(6, 10, dtype=torch.bfloat16)
    b = torch.zeros(4, 10, dtype=torch.bfloat16).t()       # [10, 4] with K contiguous → column-major
    o = torch.zeros(6, 4, dtype=torch.bfloat16)
    at = pkg.gemm_attrs_for(a, b, o, beta=0.5)
    assert (at["lhs_order"], at["lhs_num_rows"], at["lhs_num_cols"], at["lhs_leading_dim_stride"]) == (0, 6, 10, 10)
    assert (at["rhs_order"], at["rhs_num_rows"], at["rhs_num_cols"], at["rhs_leading_dim_stride"]) == (1, 10, 4, 10)
    assert at["output_order"] == 0 and at["batch_size"] == 1 and at["beta"] == 0.5
    assert at["lhs_layout_dtype"] == pkg.IXK_BF16


def test_gemm_attrs_padded_and_batched(pkg):
    a = torch.zeros(3, 6, 16, dtype=torch.float16)[:, :, :10]   # pitch 16
    b = torch.zeros(3, 10, 8, dtype=torch.float16)
    o = torch.zeros(3, 6, 8, dtype=torch.float32)
    at = pkg.gemm_attrs_for(a, b, o)
    assert at["lhs_leading_dim_stride"] == 16 and at["lhs_batch_stride"] == 96
    assert at["batch_size"] == 3 and at["output_layout_dtype"] == pkg.IXK_F32


def test_gemm_attrs_rejects_doubly_strided(pkg):
    a = torch.zeros(6, 20, dtype=torch.bfloat16)[:, ::2]
    with pytest.raises(pkg.IxkError):
        pkg.gemm_attrs_for(a, torch.zeros(10, 4, dtype=torch.bfloat16), torch.zeros(6, 4, dtype=torch.bfloat16))


def test_unknown_epilogue_name(pkg):
    x = torch.zeros(8, 8, dtype=torch.bfloat16)
    with pytest.raises(pkg.IxkError, match="Unknown Epilogue"):
        pkg.run_gemm_custom_call(x, x, None, x, None, None, pkg.gemm_attrs_for(x, x, x), "SILU")


def test_fmha_desc_from_bsnh_views(pkg):
    B, S, N, H = 2, 12, 3, 64
    q = torch.zeros(B, S, N, H, dtype=torch.bfloat16).permute(0, 2, 1, 3)   # [B,N,S,H] view of [B,S,N,H]
    o = torch.zeros(B, N, S, H, dtype=torch.bfloat16)
    bias = torch.zeros(B, 1, S, S, dtype=torch.bfloat16)
    d = pkg._fmha_desc(q, q, q, bias, o, 0.125, True, 0.0)
    assert list(d.q_strides) == [S * N * H, H, N * H]
    assert list(d.o_strides) == [N * S * H, S * H, H]
    assert list(d.bias_strides) == [S * S, 0, S]          # head-broadcast → stride 0
    assert (d.num_batches, d.num_heads, d.num_queries, d.num_keys, d.head_size, d.causal) == (B, N, S, S, H, 1)


def test_fmha_rejects_dropout_and_strided_head(pkg):
    q = torch.zeros(1, 1, 4, 64, dtype=torch.bfloat16)
    with pytest.raises(pkg.IxkError):
        pkg._fmha_desc(q[..., ::2], q, q, None, q, 1.0, False, 0.0)
    with pytest.raises(pkg.IxkError, match="no CPU path"):
        pkg.fmha_forward_kernel(None, q, q, q, None, torch.zeros(1), 0.5, q, None, 1.0)


def test_quantize_fp8_matches_oracle(pkg, orc):
    import numpy as np
    torch.manual_seed(0)
    x = torch.randn(64, 48)
    for tdt, odt in ((torch.float8_e4m3fn, orc.F8E4M3), (torch.float8_e5m2, orc.F8E5M2)):
        q, s = pkg.quantize_fp8(x, tdt)
        codes, s2 = orc.quantize_fp8(x.numpy(), odt)
        assert s == pytest.approx(s2)
        assert np.array_equal(q.view(torch.uint8).numpy(), codes)


@pytest.mark.parametrize("shape", [(5, 7, 3), (1, 64, 8), (16, 1, 1), (2, 6, 24, 40)], ids=str)
@pytest.mark.parametrize("layout", ["rr", "rc", "cr"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float8_e4m3fn])
def test_packed_gemm_descriptor(pkg, shape, layout, dtype):
    """gemm() packs its descriptor in one go: field for field what the attribute dictionary gives."""
    *batch, m, k, n = shape
    lhs = torch.empty(*batch, m, k).to(dtype) if layout[0] == "r" else torch.empty(*batch, k, m).to(dtype).transpose(-1, -2)
    rhs = torch.empty(*batch, k, n).to(dtype) if layout[1] == "r" else torch.empty(*batch, n, k).to(dtype).transpose(-1, -2)
    out = torch.empty(*batch, m, n + 8, dtype=torch.float32)[..., :n]
    want = pkg.gemm_desc_from_attrs(pkg.gemm_attrs_for(lhs, rhs, out, beta=0.5, alpha=2.0), "BIAS_GELU")
    got = pkg._gemm_desc(*(pkg._matrix_layout(name, t) for name, t in (("lhs", lhs), ("rhs", rhs), ("output", out))),
                         out.shape[0] if out.dim() == 3 else 1, 2.0, 0.5, "BIAS_GELU")
    assert bytes(got) == bytes(want)


class _FakeLibrary:
    """Answers 4096 to every workspace query and records the arguments of the launches."""

    def __init__(self, status=0):
        self.calls, self.status = [], status

    def __getattr__(self, name):
        if name.endswith("_workspace_bytes"):
            return lambda *args: 4096
        return lambda *args: self.calls.append((name, args)) or self.status


@pytest.fixture
def fake_calls(pkg, monkeypatch):
    """The package on a library that launches nothing.  allocated: for each torch.empty the stream whose pool it
    was taken from (None: the current stream's)."""
    lib, scope, allocated, empty = _FakeLibrary(), [None], [], torch.empty

    @contextlib.contextmanager
    def on(stream):
        scope.append(stream)
        yield
        scope.pop()

    def recorded(*args, **kwargs):
        allocated.append(scope[-1])
        return empty(*args, **kwargs)
    monkeypatch.setattr(pkg, "load_library", lambda: lib)
    monkeypatch.setattr(pkg, "_require_cuda", lambda *tensors: None)
    monkeypatch.setattr(torch.cuda, "stream", on)
    monkeypatch.setattr(torch.cuda, "ExternalStream", lambda ptr, device=None: ptr)
    monkeypatch.setattr(torch, "empty", recorded)
    return types.SimpleNamespace(lib=lib, allocated=allocated)


@pytest.mark.parametrize("call", ["forward", "backward", "geglu"])
def test_scratch_comes_from_the_pool_of_the_calls_stream(pkg, fake_calls, call):
    """Scratch that a call takes for itself is free again when the call returns: only in the pool of the stream that
    the call was given does its next tenant wait for the call's kernels."""
    q = torch.zeros(1, 2, 64, 32, dtype=torch.bfloat16)
    lse = torch.zeros(1, 2, 64)
    stream = types.SimpleNamespace(cuda_stream=77)
    own = torch.zeros(8192, dtype=torch.uint8)

    def run(stream, workspace):
        fake_calls.allocated.clear()
        fake_calls.lib.calls.clear()
        if call == "forward":
            pkg.fmha_forward_kernel(stream, q, q, q, None, None, 0.0, q, None, 1.0, False, workspace=workspace)
        elif call == "backward":
            pkg.fmha_backward_kernel(stream, q, q, q, q, None, q, lse, q, q, q, 1.0, workspace=workspace)
        else:
            pkg.gemm_geglu(q[0, 0], torch.zeros(32, 16, dtype=torch.bfloat16), out=q[0, 0, :, :8], workspace=workspace, stream=stream)
        (_, args), = fake_calls.lib.calls
        assert args[-1] == 77 and args[-2] >= 4096 and (workspace is None or args[-3] == workspace.data_ptr())
    run(stream, None)
    assert fake_calls.allocated == [77]
    run(stream, own)
    assert fake_calls.allocated == []


@pytest.mark.parametrize("status", ["IXK_OK", "IXK_WORKSPACE_TOO_SMALL"])
def test_forward_without_memory_for_scratch(pkg, fake_calls, monkeypatch, status):
    """With no device memory left the forward goes in without scratch of its own: a prefill runs unsplit, as it
    always could; only where the library cannot do without is the allocator's error the answer."""
    q = torch.zeros(1, 2, 64, 32, dtype=torch.bfloat16)

    def full(*args, **kwargs):
        raise torch.OutOfMemoryError("no memory")
    monkeypatch.setattr(torch, "empty", full)
    fake_calls.lib.status = getattr(pkg, status)
    for small in (None, torch.zeros(16, dtype=torch.uint8)):
        fake_calls.lib.calls.clear()
        run = lambda: pkg.fmha_forward_kernel(None, q, q, q, None, None, 0.0, q, None, 1.0, False, workspace=small)
        monkeypatch.setattr(pkg, "_stream_ptr", lambda stream: 0)
        if status == "IXK_OK":
            run()
        else:
            with pytest.raises(torch.OutOfMemoryError):
                run()
        (_, args), = fake_calls.lib.calls
        assert args[-3:-1] == ((None, 0) if small is None else (small.data_ptr(), 16))


def test_gemm_refuses_a_residual_that_does_not_lie_like_the_result(pkg, fake_calls):
    """C is read with the result's pitch, order and type: a pitched, transposed, smaller or wider-typed one is an error,
    not a read of other memory; what lies as the result does is taken, whatever it is called."""
    bf16 = torch.bfloat16
    x, w = torch.zeros(6, 16, dtype=bf16), torch.zeros(16, 8, dtype=bf16)
    out = torch.zeros(6, 8, dtype=bf16)
    pitched = torch.zeros(6, 24, dtype=bf16)[:, :8]
    refused = [(out, pitched), (out, torch.zeros(8, 6, dtype=bf16).t()), (out, torch.zeros(8, 6, dtype=bf16)), (out, out.float()),
               (out, torch.zeros(5, 8, dtype=bf16)), (out, torch.zeros(8, dtype=bf16)), (out, torch.zeros(1, 8, dtype=bf16).expand(6, 8)),
               (pitched, out), (torch.zeros(8, 6, dtype=bf16).t(), out), (None, pitched)]
    for o, c in refused:
        with pytest.raises(pkg.IxkError, match="c must have") as e:
            pkg.gemm(x, w, c=c, beta=1.0, out=o, stream=types.SimpleNamespace(cuda_stream=1))
        assert e.value.status == pkg.IXK_INVALID_ARGUMENT
    assert fake_calls.lib.calls == []
    taken = [(out, out), (out, torch.zeros(1, 6, 8, dtype=bf16)), (out, torch.zeros(48, dtype=bf16)), (out, torch.zeros(2, 3, 8, dtype=bf16)),
             (pitched, torch.zeros(6, 24, dtype=bf16)[:, 8:16]), (None, out)]
    for o, c in taken:
        pkg.gemm(x, w, c=c, beta=1.0, out=o, stream=types.SimpleNamespace(cuda_stream=1))
    pkg.gemm(x, w, c=pitched, out=out, stream=types.SimpleNamespace(cuda_stream=1))      # (beta 0: not read)
    one = torch.zeros(1, 24, dtype=bf16)[:, :8]
    pkg.gemm(x[:1], w, c=one, beta=1.0, out=out[:1], stream=types.SimpleNamespace(cuda_stream=1))   # (one row: no pitch)
    b = torch.zeros(2, 6, 8, dtype=bf16)
    pkg.gemm(x.expand(2, 6, 16), w.expand(2, 16, 8), c=b, beta=1.0, out=torch.zeros_like(b), stream=types.SimpleNamespace(cuda_stream=1))
    with pytest.raises(pkg.IxkError, match="c must have"):
        pkg.gemm(x.expand(2, 6, 16), w.expand(2, 16, 8), c=out, beta=1.0, out=b, stream=types.SimpleNamespace(cuda_stream=1))
    assert len(fake_calls.lib.calls) == len(taken) + 3


def test_scratch_of_an_fp8_call(pkg, fake_calls, monkeypatch):
    """A call that makes its own result takes scratch for cutting K too, from the pool of its stream; one into the
    caller's result allocates nothing and hands on the scratch that it was given; with no memory left it runs without."""
    x, w = torch.zeros(16, 32).to(torch.float8_e4m3fn), torch.zeros(32, 48).to(torch.float8_e4m3fn)
    stream = types.SimpleNamespace(cuda_stream=77)
    out, own = torch.zeros(16, 48, dtype=torch.bfloat16), torch.zeros(64, dtype=torch.uint8)

    def run(**kw):
        fake_calls.allocated.clear()
        fake_calls.lib.calls.clear()
        pkg.gemm_fp8(x, w, 0.5, 2.0, stream=stream, **kw)
        (name, args), = fake_calls.lib.calls
        assert name == "ixk_gemm_fp8" and args[-1] == 77
        return args[-3:-1]
    assert run()[1] == 4096 and fake_calls.allocated == [None, 77]      # the result, the scratch
    assert run(out=out) == (None, 0) and fake_calls.allocated == []
    assert run(out=out, workspace=own) == (own.data_ptr(), 64) and fake_calls.allocated == []
    assert run(workspace=own) == (own.data_ptr(), 64) and fake_calls.allocated == [None]

    def full(need, device, stream):
        raise torch.OutOfMemoryError("no memory")
    monkeypatch.setattr(pkg, "_own_scratch", full)
    assert run() == (None, 0)


def _workspace(pkg, B, N, F, T, H, causal):
    import ctypes
    d = pkg._FmhaDesc()
    d.dtype, d.causal = pkg.IXK_BF16, int(causal)
    d.num_batches, d.num_heads, d.head_size, d.num_queries, d.num_keys, d.head_scale = B, N, H, F, T, 1.0
    return pkg.load_library().ixk_fmha_fwd_workspace_bytes(ctypes.byref(d))


def test_scratch_of_a_split_prefill(pkg):
    """The query (made without a GPU for 148 SMs): partials of at most one part per SM, 128 rows of the padded head
    and two statistics each; none with a row of items per SM under the mask, or where the merge costs more."""
    import random
    rng = random.Random(4)
    split = 0
    for _ in range(2000):
        B, N, H = rng.randint(1, 16), rng.randint(1, 16), rng.choice([40, 64, 96, 128, 160, 256])
        F, T, causal = rng.randint(17, 5000), rng.randint(1, 6000), rng.random() < 0.5
        need = _workspace(pkg, B, N, F, T, H, causal)
        padded = 64 if H <= 64 else 128 if H <= 128 else 256
        tiles, rest = divmod(need, 128 * (padded + 2) * 4)
        per_item = 2 if F > 128 and H <= 128 else 1
        assert rest == 0 and tiles % per_item == 0 and tiles // per_item <= 148
        items = -(-F // (128 * per_item)) * B * N
        assert need == 0 or (items < 148 if causal else items % 148 != 0)
        split += need > 0
    assert split > 300
    assert _workspace(pkg, 2, 10, 4096, 4096, 64, False) == 144 * 2 * 128 * 66 * 4          # 24 items in parts of six blocks
    assert _workspace(pkg, 3, 8, 700, 700, 128, True) == 0                                  # slower split than whole
    assert _workspace(pkg, 1, 1, 100000, 100000, 128, True) == 0                            # an item per SM and more


@pytest.mark.parametrize("F", range(1, 17))
def test_scratch_of_a_decode_call(pkg, F):
    """What the key splits need, which a call cannot do without, or the one-pass kernel's partials (at most 4 MiB) where
    those are more; under the mask the key splits alone."""
    import random
    rng = random.Random(F)
    for _ in range(300):
        B, N, T, H = rng.randint(1, 64), rng.randint(1, 32), rng.randint(1, 9000), 8 * rng.randint(1, 32)
        groups = B * N * -(-F // (2 if F > 1 else 1))
        splits = max(min(-(-16 * 148 // groups), -(-T // 256)), 1)
        key_splits = splits * B * N * F * (H + 2) * 4 if splits > 1 else 0
        need = _workspace(pkg, B, N, F, T, H, False)
        assert need == key_splits or key_splits < need <= pkg.STATIC_SCRATCH_BYTES
        assert _workspace(pkg, B, N, F, T, H, True) == key_splits


def test_residual_projection_goes_through_the_gemm_of_the_ops(pkg):
    """A decode step's projections that add the residual are GEMMs like the others: an ops class with a gemm of its own
    (another scratch, a record of the calls) sees them."""
    import importlib
    layers = importlib.import_module("ixk_b200.layers")

    class Ops(layers.KernelOps):
        def gemm(self, x, w, **kw):
            return kw
    r = torch.zeros(2, 8)
    assert Ops(pkg).gemm_residual(torch.zeros(2, 4), torch.zeros(4, 8), r) == {"c": r, "beta": 1.0}
