"""The prompt path on the tile-layout weights: GEMM by CTA pairs, prompt attention, batched RoPE + append."""
import numpy as np
import pytest
import torch

from llm_decode_kernels_b200 import ext, quant as PQ
from oracle import quant_oracle as Q

pytestmark = pytest.mark.gpu
dev = "cuda"


@pytest.fixture(scope="module")
def K():
    return ext.load()


def matrix(K, N, Kd, gate_up=False, G=128):
    torch.manual_seed(N + Kd)
    ql = PQ.QuantLinear((torch.randn(N, Kd, device=dev) * 0.02).half(), G, keep_ref=True)
    return ql, K.gemv_tile_repack(ql.packed, ql.sz, G, gate_up=gate_up)


def test_one_hot_rows_are_the_dequantized_weights(K):
    N, Kd, G = 200, 256, 128
    torch.manual_seed(3)
    w = (torch.randn(N, Kd) * 0.05).half()
    w[3] *= 1e-4                                 # a subnormal scale
    q, s, z = PQ.quantize(w, G, False)
    packed, sz = PQ.pack(q).to(dev), PQ.pack_scale_zero(s, z).to(dev)
    tiled = K.gemv_tile_repack(packed, sz, G)
    want = Q.dequantize(q.numpy(), s.numpy(), z.numpy(), G)
    y = torch.full((Kd, N), float("nan"), dtype=torch.half, device=dev)
    K.gemm_w4a16_tiled(tiled, torch.eye(Kd, dtype=torch.half, device=dev), y, N, Kd)
    assert np.array_equal(y.cpu().numpy().view(np.uint16), want.T.copy().view(np.uint16))


# ragged rows and tokens, one unit of K, a tile more than whole ones, more tiles than CTA pairs; every split
@pytest.mark.parametrize("N,Kd,T", [(256, 128, 1), (1003, 1024, 17), (320, 384, 77), (2560, 2048, 256), (2048, 5632, 300),
                                    (512, 256, 129), (5000, 512, 1025)])
@pytest.mark.parametrize("split", [0, 1, 2, 4])
def test_gemm_tiled(K, N, Kd, T, split):
    if split > Kd // 128:
        pytest.skip("more splits than units of K")
    ql, tiled = matrix(K, N, Kd)
    x = torch.randn(T, Kd, device=dev).half()
    y = torch.full((T, N), float("nan"), dtype=torch.half, device=dev)
    K.gemm_w4a16_tiled(tiled, x, y, N, Kd, split=split)
    ref = x.float() @ ql.w_ref.float().t()
    assert ((y.float() - ref).abs().max() / ref.abs().max()).item() <= 2e-3
    assert K.gemm_status() == 0


@pytest.mark.parametrize("I,Kd,T", [(5632, 2048, 256), (1003, 1024, 77), (128, 256, 500)])
@pytest.mark.parametrize("split", [1, 2])
def test_gemm_tiled_swiglu(K, I, Kd, T, split):
    ql, tiled = matrix(K, 2 * I, Kd, gate_up=True)
    x = torch.randn(T, Kd, device=dev).half()
    y = torch.full((T, I), float("nan"), dtype=torch.half, device=dev)
    K.gemm_w4a16_tiled(tiled, x, y, I, Kd, swiglu=True, split=split)
    gu = (x.float() @ ql.w_ref.float().t()).half()
    ref = (torch.nn.functional.silu(gu[:, :I].float()).half() * gu[:, I:]).float()
    assert ((y.float() - ref).abs().max() / ref.abs().max()).item() <= 4e-3
    assert K.gemm_status() == 0


# heads per group 1 .. 8, both head sizes, pages of 8 .. 64 tokens; prompts of one row block and several, with and without
# a context before them, and a few tokens behind a long one (the context is then split between blocks); more than one chunk
# of 4096 tokens
@pytest.mark.parametrize("D,n_q,n_kv,page,start,T", [(64, 8, 8, 16, 0, 130), (64, 8, 4, 8, 37, 65), (64, 8, 2, 64, 0, 33),
                                                     (64, 8, 1, 16, 1500, 5), (64, 16, 2, 16, 700, 200), (128, 8, 1, 16, 0, 70),
                                                     (64, 8, 2, 16, 0, 4500), (128, 8, 1, 16, 300, 4100),
                                                     (128, 4, 4, 16, 1100, 3), (64, 8, 1, 16, 0, 1), (64, 16, 2, 16, 4090, 7),
                                                     (128, 8, 1, 32, 191, 130), (64, 8, 2, 16, 500, 300)])
def test_prefill_equals_stepping(D, n_q, n_kv, page, start, T):
    from llm_decode_kernels_b200.model import DecodeConfig, Model
    from test_model import KERNEL_TOL, hf_cfg, random_state
    c = hf_cfg(512, 2, n_q, n_kv, 1024, 1000, D=D)
    m = Model(random_state(c, 3, D), c, DecodeConfig(group=128, max_ctx=start + T + 16, page=page, seed=1))
    m.prepare(start + T + 8, use_graph=False)
    m.kv.normal_(generator=torch.Generator(device=dev).manual_seed(2))
    before = m.kv.clone()
    ids = torch.randint(0, 1000, (T,), generator=torch.Generator().manual_seed(4))
    m.reset(start)
    want = m.teacher_force(ids, use_graph=False, collect_logits=True).float()
    kv, tok = m.kv.clone().float(), int(m.tok)
    m.kv.copy_(before)
    m.reset(start)
    got = m.prefill(ids, collect_logits=True).float()
    assert (got - want).abs().max() <= KERNEL_TOL * want.abs().max()
    assert torch.equal((m.kv != before).any(-1), (kv != before).any(-1))      # the same cache rows
    assert (m.kv.float() - kv).abs().max() <= KERNEL_TOL * kv.abs().max()
    assert m.host_pos == start + T and int(m.pos) == start + T and m.K.gemm_status() == 0
    top = want[-1].sort(descending=True)[0]
    assert int(m.tok) == tok or top[0] - top[1] <= 2 * KERNEL_TOL * want.abs().max()


# Norms, residual sums and RoPE inside the GEMMs: hidden sizes whose last 256-row tile is half empty, one and several token tiles;
# embeddings and norm weights small and large enough that rows stored as x * w would leave fp16.
# Same tolerance as above, which allows for the stepping path's own roundings. (The norm in front of attention keeps its weights where
# they are large: scores of hundreds would multiply every rounding of either path.)
@pytest.mark.parametrize("H,D,n_q,n_kv,T,emb,ln", [(128, 64, 2, 1, 3, 1.0, 1.0), (384, 64, 6, 3, 33, 1e-3, 0.02), (640, 64, 8, 8, 257, 1.0, 8.0),
                                                   (640, 128, 4, 1, 129, 2000.0, 1.0), (384, 64, 4, 4, 768, 100.0, 0.1),
                                                   (384, 128, 2, 2, 769, 1e-3, 8.0), (2048, 64, 32, 4, 96, 1e-3, 3.0)])
def test_norms_and_rope_inside_the_gemms(H, D, n_q, n_kv, T, emb, ln):
    from llm_decode_kernels_b200.model import DecodeConfig, Model
    from test_model import KERNEL_TOL, hf_cfg, random_state
    c = hf_cfg(H, 3, n_q, n_kv, 512, 1000, D=D)
    sd = random_state(c, 5, D)
    for k in sd:
        if "embed_tokens" in k:
            sd[k] = (sd[k].float() * emb).half()
        elif "norm" in k:
            sd[k] = (sd[k].float() * (min(ln, 1.0) if "input" in k else ln)).half()
    m = Model(sd, c, DecodeConfig(group=128, max_ctx=T + 16, seed=1))
    m.prepare(T + 8, use_graph=False)
    ids = torch.randint(0, 1000, (T,), generator=torch.Generator().manual_seed(6))
    m.reset(0)
    want = m.teacher_force(ids, use_graph=False, collect_logits=True).float()
    kv = m.kv.clone().float()
    m.kv.zero_()
    m.reset(0)
    got = m.prefill(ids, collect_logits=True).float()
    assert torch.isfinite(want).all() and (got - want).abs().max() <= KERNEL_TOL * want.abs().max()
    assert (m.kv.float() - kv).abs().max() <= KERNEL_TOL * kv.abs().max() and m.K.gemm_status() == 0


def prompt_in_64_bits(m, sd, ids):
    """Logits [T, V], K and V rows [T, L, n_kv D] of a prompt at position 0, from the fp16 weights as dequantized."""
    def weight(lin):
        w = torch.empty(lin.packed.shape[0], lin.K, dtype=torch.half, device=dev)
        m.K.dequant_w4a16(lin.packed, lin.sz, w, 128)
        return w.double()
    T, D, n_q, n_kv, d2 = ids.numel(), m.D, m.n_q, m.n_kv, m.D // 2
    cos, sin = m.cos[:T, None].double(), m.sin[:T, None].double()
    norm = lambda x, w: x * torch.rsqrt((x * x).mean(-1, keepdim=True) + m.eps) * w.double()
    rope = lambda v: torch.cat([v[..., :d2] * cos - v[..., d2:] * sin, v[..., d2:] * cos + v[..., :d2] * sin], -1)
    later = torch.ones(T, T, dtype=torch.bool, device=dev).triu(1)
    x, ks, vs = sd["model.embed_tokens.weight"].to(dev)[ids.to(dev)].double(), [], []
    for lw in m.layers:
        q, k, v = (norm(x, lw["ln1"]) @ weight(lw["qkv"]).t()).view(T, -1, D).split([n_q, n_kv, n_kv], 1)
        q, k = rope(q), rope(k)
        ks.append(k.reshape(T, -1)), vs.append(v.reshape(T, -1))
        k, v = (t.repeat_interleave(n_q // n_kv, 1) for t in (k, v))
        s = torch.einsum("thd,shd->hts", q, k) / D ** 0.5
        a = torch.einsum("hts,shd->thd", s.masked_fill(later, float("-inf")).softmax(-1), v).reshape(T, -1)
        x = x + a @ weight(lw["o"]).t()
        gate, up = (norm(x, lw["ln2"]) @ weight(lw["gu"]).t()).split(m.I, 1)
        x = x + (torch.nn.functional.silu(gate) * up) @ weight(lw["down"]).t()
    return norm(x, m.norm_f) @ weight(m.lm_head).t(), torch.stack(ks, 1), torch.stack(vs, 1)


def errors(m, sd, ids):
    """How far a prompt is from 64 bits (2-norms), on the tile layout and operator by operator: {path: {output: error}}."""
    want, T, err = prompt_in_64_bits(m, sd, ids), ids.numel(), {}
    for path in ("tiled", "operators"):
        if path == "operators":
            m._prefill_desc = None          # what a model whose shape rules the tile layout out has there
        m.kv.zero_()
        m.reset(0)
        logits = m.prefill(ids, collect_logits=True)
        rows = m.kv[:, :, m.bt[:-(-T // 16)].long()].permute(1, 2, 4, 0, 3, 5).reshape(2, -1, 2, m.n_kv * m.D)[:, :T]
        assert torch.isfinite(logits).all() and m.K.gemm_status() == 0
        got = {"logits": (logits, want[0]), "k0": (rows[0, :, 0], want[1][:, 0]), "k1": (rows[0, :, 1], want[1][:, 1]),
               "v0": (rows[1, :, 0], want[2][:, 0]), "v1": (rows[1, :, 1], want[2][:, 1])}
        err[path] = {n: ((a.double() - b).norm() / b.norm()).item() for n, (a, b) in got.items()}
    print(err)
    return err


# The rows between the GEMMs of a prompt lose neither range nor precision against RMSNorm as an operator of its own, which the
# row-major path still has: small embeddings under small and large weights, large rows, rows of which one addition makes one channel a
# million times as large as the rest, under weights above 1 (`jump`: by what its weights in o are multiplied; channel 7 and positive
# weights for it give all tokens the same sign there), rows that one channel of weight zero dominates (`massive`: that channel's embedding). K and V
# rows and logits against 64 bits: no further off than the operators, but for 5 % between two sets of roundings.
@pytest.mark.parametrize("H,D,n_q,n_kv,I,T,emb,ln,jump,massive", [
    (512, 64, 8, 2, 512, 40, 0.02, 0.005, 0, 0), (512, 64, 8, 2, 512, 40, 2e-3, 0.02, 0, 0), (512, 128, 4, 2, 512, 40, 2e-3, 0.005, 0, 0),
    (512, 64, 8, 2, 512, 300, 1e-3, 0.02, 0, 0), (512, 64, 8, 2, 512, 40, 1e-4, 1.0, 0, 0), (512, 64, 8, 2, 512, 40, 0.04, 8.0, 800.0, 0),
    (1024, 128, 8, 8, 512, 300, 0.04, 8.0, 400.0, 0), (2048, 64, 32, 4, 512, 40, 0.6, 0.1, 0, 15000.0), (512, 64, 8, 2, 512, 40, 600.0, 1.0, 0, 0)])
def test_norms_inside_the_gemms_lose_nothing(H, D, n_q, n_kv, I, T, emb, ln, jump, massive):
    from llm_decode_kernels_b200.model import DecodeConfig, Model
    from test_model import hf_cfg, random_state
    c = hf_cfg(H, 2, n_q, n_kv, I, 1000, D=D)
    sd = random_state(c, 5, D)
    for k in sd:
        if "norm" in k:
            sd[k] = (sd[k].float() * (min(ln, 1.0) if "input" in k else ln)).half()
            if massive:
                sd[k][5] = 0
    E = sd["model.embed_tokens.weight"] = (sd["model.embed_tokens.weight"].float() * emb).half()
    if jump:
        E[:, 7] = 2
        sd["model.layers.0.self_attn.v_proj.weight"][:, 7].abs_()
        sd["model.layers.0.self_attn.o_proj.weight"][5].abs_().mul_(jump)
    if massive:
        E[:, 5] = massive
    m = Model(sd, c, DecodeConfig(group=128, max_ctx=T + 16, seed=1, keep_packed=True))
    m.prepare(T + 8, use_graph=False)
    ids = torch.randint(0, 1000, (T,), generator=torch.Generator().manual_seed(6))
    err = errors(m, sd, ids)
    for n, e in err["tiled"].items():
        assert e <= 1.05 * err["operators"][n], (n, err)


# The same where a CTA pair walks over several tiles of the qkv, o and down matrices (3400 tokens: 144 to 324 and 108 tiles for 74
# pairs), where four pairs split K in front of RoPE and of a residual row, and where the partials of a split lie over the stages (rows
# of more than 14336 weights and 256-token tiles). By the dispatch's own choice.
@pytest.mark.parametrize("H,D,n_q,n_kv,I,T", [(1536, 128, 12, 12, 256, 3400), (1536, 64, 24, 3, 256, 3391), (8192, 64, 2, 1, 256, 40),
                                              (256, 64, 4, 2, 8192, 37), (4352, 64, 2, 1, 14464, 256)])
def test_epilogues_over_many_tiles_and_splits(H, D, n_q, n_kv, I, T):
    from llm_decode_kernels_b200.model import DecodeConfig, Model
    from llm_decode_kernels_b200.shapes import random_llama_state
    from test_model import hf_cfg
    c = hf_cfg(H, 2, n_q, n_kv, I, 1000, D=D)
    sd, g = random_llama_state(c, dev, 7), torch.Generator(device=dev).manual_seed(8)
    for k in sd:
        if "norm" in k:
            sd[k] = (0.5 + torch.rand(H, generator=g, device=dev)).half()
    m = Model(sd, c, DecodeConfig(group=128, max_ctx=T + 16, seed=1, keep_packed=True))
    m.prepare(T + 8, use_graph=False)
    err = errors(m, sd, torch.randint(0, 1000, (T,), generator=torch.Generator().manual_seed(6)))
    for n, e in err["tiled"].items():
        assert e <= 1.05 * err["operators"][n], (n, err)


# Error of the prompt attention against 64 bits, on the rotated queries and the cache it read. Its output is one fp16 rounding of sums
# that keep the probabilities to 22 bits: the error must be that rounding's (2^-11 / sqrt(12), a little less on average) and 10 % at
# most beside it. fp16 probabilities alone add 17 to 40 %. Flat and peaked rows; whole context and splits.
@pytest.mark.parametrize("D,n_q,n_kv,start,T", [(64, 16, 2, 0, 300), (64, 16, 2, 1800, 100), (128, 8, 1, 0, 200), (128, 8, 1, 1500, 30)])
@pytest.mark.parametrize("peak", [1, 4])
def test_prompt_attention_loses_no_precision(D, n_q, n_kv, start, T, peak):
    from llm_decode_kernels_b200.model import DecodeConfig, Model
    from test_model import hf_cfg, random_state
    c = hf_cfg(n_q * D, 1, n_q, n_kv, 1024, 1000, D=D)
    sd = random_state(c, 5, D, scale=0.02)
    sd["model.layers.0.self_attn.q_proj.weight"] *= peak
    m = Model(sd, c, DecodeConfig(group=128, max_ctx=start + T + 16, page=16, seed=1))
    m.prepare(start + T + 8, use_graph=False)
    m.kv.normal_(generator=torch.Generator(device=dev).manual_seed(2))
    m.reset(start)
    m.prefill(torch.randint(0, 1000, (T,), generator=torch.Generator().manual_seed(3)))
    d, work = m._prefill_desc, m._prefill_work

    def buffer(ptr, width):
        at = ptr - work.data_ptr()
        return work[at:at + 2 * T * width].view(torch.half).view(T, width)
    n = start + T
    k, v = (m.kv[0, i][m.bt[:-(-n // 16)].long()].permute(0, 2, 1, 3).reshape(-1, n_kv, D)[:n].double() for i in (0, 1))
    q = buffer(d.qkv, (n_q + 2 * n_kv) * D)[:, :n_q * D].reshape(T, n_q, D).double()
    hidden = torch.arange(n, device=dev)[None] > start + torch.arange(T, device=dev)[:, None]
    ref = torch.empty_like(q)
    for h in range(n_q):
        s = (q[:, h] @ k[:, h * n_kv // n_q].t() / D ** 0.5).masked_fill(hidden, float("-inf"))
        ref[:, h] = torch.softmax(s, -1) @ v[:, h * n_kv // n_q]
    rounding = (ref.half().double() - ref).norm()
    assert (buffer(d.attn, n_q * D).reshape(T, n_q, D).double() - ref).norm() <= 1.1 * rounding


def test_long_rows_are_split_for_precision(K):
    """The library's own choice at K = 28672 and many tokens, where one accumulation chain per tile is fastest: the error against 64
    bits is no larger than with K split in two (a chain loses the low bits of its addends at every step)."""
    N, Kd, T = 8192, 28672, 256
    ql, tiled = matrix(K, N, Kd)
    x = torch.randn(T, Kd, generator=torch.Generator(device=dev).manual_seed(1), device=dev).half()
    ref = torch.cat([x.double() @ w.double().t() for w in ql.w_ref.split(1024)], 1)
    err = {}
    for split in (0, 1, 2):
        y = torch.empty(T, N, dtype=torch.half, device=dev)
        K.gemm_w4a16_tiled(tiled, x, y, N, Kd, split=split)
        err[split] = ((y.double() - ref).norm() / ref.norm()).item()
    assert err[0] <= err[2] * (1 + 1e-4) < err[1]


# A token whose keys and values are NaN (as after an overflow): the tokens before it are what they are without it - in the same tile
# of 64, in the row block before, and where the context is split between CTAs.
@pytest.mark.parametrize("D,n_q,n_kv,start,T,bad", [(64, 8, 1, 0, 40, 37), (64, 8, 8, 0, 150, 100), (64, 16, 2, 0, 70, 0), (128, 8, 2, 30, 90, 64),
                                                    (64, 8, 1, 1500, 12, 9), (128, 8, 1, 1100, 20, 3)])
def test_tokens_do_not_see_a_later_nan(D, n_q, n_kv, start, T, bad):
    from llm_decode_kernels_b200.model import DecodeConfig, Model
    from test_model import KERNEL_TOL, hf_cfg, random_state
    c = hf_cfg(512, 2, n_q, n_kv, 1024, 1000, D=D)
    m = Model(random_state(c, 3, D), c, DecodeConfig(group=128, max_ctx=start + T + 16, page=16, seed=1))
    m.prepare(start + T + 8, use_graph=False)
    m.kv.normal_(generator=torch.Generator(device=dev).manual_seed(2))
    m.emb[999] = float("inf")
    ids = torch.randint(0, 999, (T,), generator=torch.Generator().manual_seed(4))
    m.reset(start)
    want = m.prefill(ids, collect_logits=True).float()
    ids[bad] = 999
    m.reset(start)
    got = m.prefill(ids, collect_logits=True).float()
    assert torch.isnan(got[bad:]).all()
    assert bad == 0 or (got[:bad] - want[:bad]).abs().max() <= KERNEL_TOL * want.abs().max()


def test_prompts_on_two_streams_keep_their_work_buffer():
    """A prompt on a side stream, then a longer one, which replaces the work buffer: its memory is not handed to the stream it was
    allocated on while the side stream still uses it."""
    from llm_decode_kernels_b200.model import DecodeConfig, Model
    from test_model import hf_cfg, random_state
    c = hf_cfg(512, 2, 8, 2, 1024, 1000)
    m = Model(random_state(c, 3), c, DecodeConfig(group=128, max_ctx=2100, page=16, seed=1))
    m.prepare(2048, use_graph=False)
    # on the host and pinned: neither checking nor copying them waits for the side stream
    ids = torch.randint(0, 1000, (1500,), generator=torch.Generator().manual_seed(4)).pin_memory()
    m.reset(0)
    m.prefill(ids[:700])                    # allocates the buffer, on the current stream
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(1_000_000_000)    # the side stream is busy for about half a second
        m.reset(0)
        m.prefill(ids[:700])
        used = m._prefill_work.data_ptr(), m._prefill_work.numel()
        m.prefill(ids[700:])                # more than the buffer holds: it is replaced
        done = side.record_event()
    assert m._prefill_work.data_ptr() != used[0]
    assert not done.query(), "the host was too slow for this test"
    again = torch.empty(used[1], dtype=torch.uint8, device=dev)     # on the current stream
    assert again.data_ptr() != used[0]
    torch.cuda.synchronize()
