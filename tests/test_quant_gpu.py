"""The CUDA quantizer kernels against the torch form of the same functions on the same device."""
import pytest
import torch

from llm_decode_kernels_b200 import quant as PQ

pytestmark = pytest.mark.gpu


def weights(N, K, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randn(N, K, generator=g, device="cuda") * 0.02
    w[0, :K // 2] = 0                       # a group without a range
    w[N // 2] = w[N // 2].abs() + 0.5       # no zero crossing: levels far beyond 15 before clamping
    w[N - 1] *= 1e-6                        # scales at their lower bound
    w[torch.rand(N, K, generator=g, device="cuda") < 2e-3] *= 8
    return w.to(dtype)


@pytest.mark.parametrize("N,K,G", [(1, 8, 8), (3, 96, 32), (257, 384, 64), (1000, 1280, 128), (64, 512, 256), (17, 640, 640)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("clip", [False, True])
def test_quantize_kernel_equals_torch_form(N, K, G, dtype, clip):
    w = weights(N, K, dtype, N + K)
    q0, s0, z0 = PQ._quantize_torch(w, G, clip)
    q, s, z = PQ.quantize(w, G, clip)
    same = ((s == s0) & (z == z0)).repeat_interleave(G, 1)
    # clipping: two factors of equal error up to the order of the sum may change places
    assert same.float().mean() >= (1 - 2e-3 if clip else 1)
    assert torch.equal(q[same], q0[same])
    ql = PQ.QuantLinear(w, G, clip=clip)
    assert torch.equal(ql.packed, PQ.pack(q)) and torch.equal(ql.sz, PQ.pack_scale_zero(s, z))
    assert torch.equal(ql.w_ref, PQ.dequantize(q, s, z, G))


@pytest.mark.parametrize("N,K,G,block", [(5, 64, 64, 64), (300, 384, 128, 128), (64, 320, 32, 96), (129, 512, 64, 128)])
@pytest.mark.parametrize("clip", [False, True])
def test_gptq_kernel_equals_torch_loop(monkeypatch, N, K, G, block, clip):
    g = torch.Generator(device="cuda").manual_seed(N)
    w = weights(N, K, torch.float16, 3)
    x = torch.randn(4 * K, K, generator=g, device="cuda")
    H = 2 * x.t() @ (x + 0.5 * x.roll(1, 1)) / x.shape[0]
    H = (H + H.t()) / 2
    H[7] = 0
    H[:, 7] = 0                             # an input that is never active
    got = PQ.quantize_gptq(w, H, G, clip=clip, block=block)
    monkeypatch.setattr(PQ, "_gptq_columns", PQ._gptq_columns_torch)
    ref = PQ.quantize_gptq(w, H, G, clip=clip, block=block)
    assert (got[0] != ref[0]).float().mean() < 2e-3
    assert all((a != b).float().mean() < 2e-3 for a, b in zip(got[1:], ref[1:]))


@pytest.mark.parametrize("form", ["transposed", "columns of a wider matrix", "every second row"])
def test_gptq_kernel_takes_any_strides(form):
    g = torch.Generator(device="cuda").manual_seed(5)
    N, K = 64, 256
    if form == "transposed":
        w = (torch.randn(K, N, generator=g, device="cuda") * 0.02).half().t()
    elif form == "columns of a wider matrix":
        w = (torch.randn(N, K + 64, generator=g, device="cuda") * 0.02).half()[:, 32:K + 32]
    else:
        w = (torch.randn(2 * N, K, generator=g, device="cuda") * 0.02).half()[::2]
    assert w.shape == (N, K) and not w.is_contiguous()
    x = torch.randn(4 * K, K, generator=g, device="cuda")
    H = 2 * x.t() @ x / x.shape[0]
    for a, b in zip(PQ.quantize_gptq(w, H, 64), PQ.quantize_gptq(w.contiguous(), H, 64)):
        assert torch.equal(a, b)


def test_gptq_without_rows_and_with_a_hessian_elsewhere():
    H = torch.eye(128)
    q, s, z = PQ.quantize_gptq(torch.empty(0, 128, device="cuda"), H.cuda(), 64)
    assert q.shape == (0, 128) and s.shape == z.shape == (0, 2)
    with pytest.raises(RuntimeError, match="device"):       # torch's own refusal; no host pointer reaches the kernel
        PQ.quantize_gptq(torch.ones(4, 128, device="cuda"), H, 64)


def damaged(N, K, G, dtype):
    """Groups of every kind a damaged matrix holds, one per row: NaN alone or everywhere, infinities of one or both signs."""
    g = torch.Generator(device="cuda").manual_seed(9)
    w = torch.randn(N, K, generator=g, device="cuda") * 0.02
    nan, inf = float("nan"), float("inf")
    w[0, G + 3] = nan
    w[1, :G] = nan
    w[2, 2 * G - 1], w[2, G] = inf, -inf
    w[3, G + 1] = inf
    w[4, G + 2] = -inf
    w[5, :G] = inf
    w[6, :3] = torch.tensor([nan, inf, -inf])
    return w.to(dtype)


@pytest.mark.parametrize("G", [8, 32, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("clip", [False, True])
def test_quantize_kernel_shows_damaged_weights(G, dtype, clip):
    w = damaged(9, 4 * G, G, dtype)
    q0, s0, z0 = PQ._quantize_torch(w, G, clip)
    q, s, z = PQ.quantize(w, G, clip)
    assert torch.isnan(s0[:2]).any() and torch.isinf(s0[2, 1])
    assert torch.equal(torch.isfinite(s), torch.isfinite(s0)) and torch.equal(torch.isfinite(z), torch.isfinite(z0))
    bad = ~(torch.isfinite(s0) & torch.isfinite(z0))
    assert torch.allclose(s[bad], s0[bad], rtol=0, equal_nan=True) and torch.allclose(z[bad], z0[bad], rtol=0, equal_nan=True)
    rows = bad.repeat_interleave(G, 1)
    assert torch.equal(q[rows], q0[rows])
    ref = PQ.QuantLinear(w, G, clip=clip).w_ref
    assert torch.allclose(ref[rows], PQ.dequantize(q0, s0, z0, G)[rows], rtol=0, equal_nan=True)


@pytest.mark.parametrize("clip", [False, True])
def test_gptq_kernel_shows_damaged_weights(monkeypatch, clip):
    G = 64
    w = damaged(9, 4 * G, G, torch.float32)
    x = torch.randn(2048, 4 * G, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    H = 2 * x.t() @ x / x.shape[0]
    got = PQ.quantize_gptq(w, H, G, clip=clip)
    monkeypatch.setattr(PQ, "_gptq_columns", PQ._gptq_columns_torch)
    ref = PQ.quantize_gptq(w, H, G, clip=clip)
    for a, b in zip(got[1:], ref[1:]):
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.isnan(b[:2]).any()


@pytest.mark.parametrize("dtype,offset", [(torch.float16, 1), (torch.float16, 4), (torch.bfloat16, 3), (torch.float32, 2)])
def test_quantize_takes_views_off_a_16_byte_boundary(dtype, offset):
    flat = torch.randn(offset + 32 * 256, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda").to(dtype)
    w = flat[offset:].view(32, 256)
    assert w.is_contiguous() and w.data_ptr() % 16
    for a, b in zip(PQ.quantize(w, 64), PQ.quantize(w.clone(), 64)):
        assert torch.equal(a, b)
    assert torch.equal(PQ.QuantLinear(w, 64).packed, PQ.QuantLinear(w.clone(), 64).packed)


def test_quantize_under_autograd_and_vmap_is_the_torch_form():
    w = torch.randn(4, 32, 256, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda")
    p = torch.nn.Parameter(w[0].clone())
    _, s, _ = PQ.quantize(p, 64)
    s.float().sum().backward()
    want = w[0].clone().requires_grad_()
    PQ._quantize_torch(want, 64)[1].float().sum().backward()
    assert torch.equal(p.grad, want.grad)
    with torch.no_grad():      # an ordinary parameter, as a loader passes it
        assert not PQ.quantize(p, 64)[1].requires_grad
    for a, b in zip(torch.vmap(lambda m: PQ.quantize(m, 64))(w), map(torch.stack, zip(*(PQ.quantize(m, 64) for m in w)))):
        assert torch.equal(a, b)
