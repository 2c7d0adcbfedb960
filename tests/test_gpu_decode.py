"""
GPU decode path: the CUDA-graph decode step (GEMV / cache-append / split-key attention kernels) against the
op-level KV-cache forward of the same model, and the decode kernels against plain PyTorch fp32 references.
"""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16 = torch.bfloat16


class _Tok:
    SPECIAL = {"<|python_start|>": 2040, "<|python_end|>": 2041, "<|output_start|>": 2042,
               "<|output_end|>": 2043, "<|assistant_end|>": 2044, "<|bos|>": 2045}

    def encode_special(self, s):
        return self.SPECIAL[s]

    def get_bos_token_id(self):
        return 2045

    def encode(self, s, prepend=None):
        return [ord(c) % 256 for c in s]

    def decode(self, ids):
        return "".join(chr(t % 128) for t in ids)


def _model():
    from nanochat_b200.models.gpt import GPT, GPTConfig
    cfg = GPTConfig(sequence_len=256, vocab_size=2048, n_layer=4, n_head=2, n_kv_head=1, n_embd=256, window_pattern="SL")
    torch.manual_seed(3)
    with torch.device("meta"):
        m = GPT(cfg)
    m.to_empty(device="cuda")
    m.init_weights()
    with torch.no_grad():
        for blk in m.transformer.h:
            blk.attn.c_proj.weight.normal_(0, 0.05)
            blk.mlp.c_proj.weight.normal_(0, 0.05)
        m.lm_head.weight.normal_(0, 0.2)
        m.smear_lambda.fill_(0.5)
    return m.eval()


def test_gemv_rows_matches_fp32():
    from nanochat_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(0)
    for B, N, K in ((1, 1664, 1664), (3, 520, 6656), (8, 2048, 256)):
        x = torch.randn(B, K, device="cuda", generator=g).to(BF16)
        W = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(BF16)
        aux = torch.randn(B, N, device="cuda", generator=g).to(BF16)
        out = torch.empty(B, N, dtype=BF16, device="cuda")
        nat._C.gemv_rows(x, W, out, None, 0, False)
        ref = x.float() @ W.float().t()
        assert ((out.float() - ref).norm() / ref.norm()).item() < 1e-2
        nat._C.gemv_rows(x, W, out, aux, 1, False)
        ref2 = torch.relu(ref) ** 2 + aux.float()
        assert ((out.float() - ref2).norm() / ref2.norm()).item() < 1e-2
        nat._C.gemv_rows(x, W, out, None, 0, True)       # rmsnorm of the input rows folded in
        xf = x.float()
        ref3 = (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1.1920929e-07)) @ W.float().t()
        assert ((out.float() - ref3).norm() / ref3.norm()).item() < 1e-2


def test_gemv_with_folded_mix_and_norm_matches_the_separate_kernels():
    from nanochat_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(5)
    lam_r = torch.tensor([1.0, 0.9, 1.1], device="cuda")
    lam_0 = torch.tensor([0.0, 0.2, -0.1], device="cuda")
    for B, N, K, layer in ((1, 4992, 1664, 1), (5, 1000, 256, 2), (8, 768, 2048, 0)):
        x = torch.randn(B, K, device="cuda", generator=g).to(BF16)
        x0 = torch.randn(B, K, device="cuda", generator=g).to(BF16)
        W = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(BF16)
        out = torch.empty(B, N, dtype=BF16, device="cuda")
        xm = torch.zeros(B, K, dtype=BF16, device="cuda")
        xn = torch.zeros(B, K, dtype=BF16, device="cuda")
        nat._C.gemv_rows_mix(x, x0, lam_r, lam_0, layer, W, out, xm, xn)
        # oracle: the stand-alone mix + norm kernel, then fp32 matmul
        xm_ref = torch.empty_like(xm)
        xn_ref = torch.empty_like(xn)
        nat._C.mixnorm_fwd(x, x0, lam_r, lam_0, layer, xm_ref, xn_ref, None)
        assert torch.equal(xm, xm_ref)                                        # same rounding, bit for bit
        assert (xn[:, :16].float() - xn_ref[:, :16].float()).abs().max().item() <= 0.02 * xn_ref.float().abs().max().item()
        assert xn[:, 16:].abs().sum().item() == 0                             # only the gate's slice is written
        xmf = xm_ref.float()
        ref = (xmf * torch.rsqrt(xmf.pow(2).mean(-1, keepdim=True) + 1.1920929e-07)) @ W.float().t()
        assert ((out.float() - ref).norm() / ref.norm()).item() < 1e-2
    nat.check_status()


@pytest.mark.parametrize("B,N,K", [(1, 128, 8), (1, 4992, 1664), (3, 520, 6656), (16, 1000, 72), (17, 1664, 6656), (32, 129, 256),
                                   (33, 2304, 768), (64, 6656, 1664), (64, 32768, 512)])
def test_rows_gemm_matches_fp32(B, N, K):
    from nanochat_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(B + N)
    x = torch.randn(B, K, device="cuda", generator=g).to(BF16)
    W = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).to(BF16)
    aux, x0 = (torch.randn(B, N, device="cuda", generator=g).to(BF16) for _ in range(2))
    lam_r, lam_0 = torch.tensor([1.0, 0.9], device="cuda"), torch.tensor([0.0, 0.2], device="cuda")
    out, xm, xn = torch.empty(B, N, dtype=BF16, device="cuda"), torch.empty(B, N, dtype=BF16, device="cuda"), torch.zeros_like(x)
    logits = torch.empty(B, N, device="cuda")
    ref, xf = x.float() @ W.float().t(), x.float()
    close = lambda a, b: ((a.float() - b).norm() / b.norm()).item() < 4e-3          # a bf16 result is off by at most 2^-9 = 2e-3
    nat._C.rows_gemm(x, W, out, aux, relu2=True, x0=x0, lam_r=lam_r, lam_0=lam_0, layer=1, xm=xm)
    assert close(out, torch.relu(ref) ** 2 + aux.float())
    assert close(xm, 0.9 * out.float() + 0.2 * x0.float())
    nat._C.rows_gemm(x, W, logits=logits, softcap=15.0)
    assert ((logits - 15 * torch.tanh(ref / 15)).norm() / ref.norm()).item() < 1e-5
    rstd = torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1.1920929e-07)
    nat._C.rows_gemm(x, W, out, norm_input=True, xn=xn if K >= 16 else None)
    assert close(out, rstd * ref)
    if K >= 16:
        assert close(xn[:, :16], (rstd * xf)[:, :16]) and xn[:, 16:].abs().sum().item() == 0
    nat.check_status()


def test_decode_embed_matches_fp32():
    from nanochat_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(11)
    V, C, B = 300, 1664, 5
    wte = torch.randn(V, C, device="cuda", generator=g).to(BF16)
    gate_w = torch.randn(24, device="cuda", generator=g) * 0.3
    lam = torch.tensor([0.7], device="cuda")
    prev = torch.randn(B, C, device="cuda", generator=g).to(BF16)
    ids = torch.tensor([[3], [299], [0], [17], [3]], device="cuda")
    out = torch.empty(B, C, dtype=BF16, device="cuda")
    prev_in = prev.clone()
    nat._C.decode_embed(ids, wte, gate_w, lam, prev, out)
    e = wte[ids[:, 0]].float()
    e = (e * torch.rsqrt(e.pow(2).mean(-1, keepdim=True) + 1.1920929e-07)).to(BF16).float()
    gate = lam * torch.sigmoid(e[:, :24] @ gate_w)
    want = e + gate[:, None] * prev_in.float()
    assert torch.equal(prev.float(), e)                                  # the state becomes the normed embedding
    assert (out.float() - want).abs().max().item() < 0.02 * want.abs().max().item()
    zero = torch.zeros_like(prev)                                        # no previous token: the smear term vanishes
    nat._C.decode_embed(ids, wte, gate_w, lam, zero, out)
    assert torch.equal(out.float(), e) and torch.equal(zero.float(), e)


def test_decode_attention_matches_fp32():
    from nanochat_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(1)
    B, H, Hkv, T = 3, 4, 2, 300
    kc = torch.randn(B, T, Hkv, 128, device="cuda", generator=g).to(BF16)
    vc = torch.randn(B, T, Hkv, 128, device="cuda", generator=g).to(BF16)
    q = torch.randn(B, H * 128, device="cuda", generator=g).to(BF16)
    seqlens = torch.tensor([5, 150, 299], dtype=torch.int32, device="cuda")
    scratch = torch.zeros(nat._C.decode_attn_scratch(B, H), dtype=torch.float32, device="cuda")
    for window in (-1, 64):
        y = torch.empty(B, H * 128, dtype=BF16, device="cuda")
        nat._C.decode_attn(q, kc, vc, seqlens, H, Hkv, window, 1.0 / math.sqrt(128), scratch, y)
        for b in range(B):
            pos = int(seqlens[b])
            lo = 0 if window < 0 else max(0, pos - window)
            for h in range(H):
                k = kc[b, lo:pos + 1, h // 2].float()
                v = vc[b, lo:pos + 1, h // 2].float()
                p = torch.softmax(k @ q[b, h * 128:(h + 1) * 128].float() / math.sqrt(128), dim=0)
                ref = p @ v
                got = y[b, h * 128:(h + 1) * 128].float()
                assert ((got - ref).norm() / ref.norm()).item() < 2e-2, (window, b, h)


def test_decode_graph_matches_cached_forward_and_engine_is_greedy_consistent():
    from nanochat_b200 import ops
    from nanochat_b200.engine import Engine
    model = _model()
    prompt = [2045, 5, 9, 200, 41, 7, 1000, 33]
    eng = Engine(model, _Tok())
    fast = [c for c, _ in eng.generate(prompt, num_samples=2, max_tokens=40, temperature=0.0)]
    assert eng._decode_graphs, "the graph decode path was not taken"
    graph = next(iter(eng._decode_graphs.values()))
    assert graph.graph is not None, "the decode step was never captured"
    ops.native_module().check_status()
    # the same generation through the op-level cached forward (no graph, no pooled cache)
    eng2 = Engine(model, _Tok())
    eng2._pooled_cache = lambda *a, **k: None
    slow = [c for c, _ in eng2.generate(prompt, num_samples=2, max_tokens=40, temperature=0.0)]
    # bf16 rounding differs between the two paths; near-ties in the argmax may flip late in the sequence
    agree = 0
    for a, b in zip(fast, slow):
        if a != b:
            break
        agree += 1
    assert agree >= 8, (agree, fast[:12], slow[:12])
    # a second generation reuses the captured graph and gives the same tokens
    again = [c for c, _ in eng.generate(prompt, num_samples=2, max_tokens=40, temperature=0.0)]
    assert again == fast
    # more than 8 rows: the same graph with tensor-core GEMMs instead of the GEMV; every row is the same greedy sequence
    wide = [c for c, _ in eng.generate(prompt, num_samples=12, max_tokens=24, temperature=0.0)]
    assert any(g.graph is not None and g.B == 12 for g in eng._decode_graphs.values())
    assert all(len(set(col)) == 1 for col in wide[:8])
    agree = 0
    for a, b in zip(wide, fast):
        if a[0] != b[0]:
            break
        agree += 1
    assert agree >= 8, (agree, [c[0] for c in wide[:12]], [c[0] for c in fast[:12]])
    ops.native_module().check_status()


@pytest.mark.parametrize("T", [8, 77, 200])
def test_fused_prefill_matches_op_level_cached_forward(T):
    """Prompt into an empty cache: the fused per-layer path against the plain-PyTorch cached forward (logits, the
    cache contents, the smear state), then one decode step on top of each cache."""
    from nanochat_b200 import ops
    from nanochat_b200.engine import KVCache
    model = _model()
    cfg = model.config
    g = torch.Generator(device="cuda").manual_seed(T)
    ids = torch.randint(0, 2040, (1, T), device="cuda", generator=g)
    nxt = torch.randint(0, 2040, (1, 1), device="cuda", generator=g)

    def run():
        cache = KVCache(1, cfg.n_kv_head, 256, 128, cfg.n_layer, "cuda", BF16)
        with torch.inference_mode():
            logits = model(ids, kv_cache=cache)
            step = model(nxt, kv_cache=cache)
        return logits.float(), step.float(), cache

    calls = []
    orig = model._prefill_native
    model._prefill_native = lambda *a, **k: (calls.append(1), orig(*a, **k))[1]
    logits, step, cache = run()
    assert calls, "the fused prefill path was not taken"
    ops.native_module().check_status()
    ops.set_kernel_mode("torch")
    try:
        ref_logits, ref_step, ref_cache = run()
    finally:
        ops.set_kernel_mode("native")
    assert len(calls) == 1
    assert cache.get_pos() == ref_cache.get_pos() == T + 1
    assert cache.cache_seqlens.tolist() == ref_cache.cache_seqlens.tolist() == [T + 1]
    assert (logits - ref_logits).abs().max().item() < 0.25, (logits - ref_logits).abs().max().item()
    assert (logits[0, -1].argmax() == ref_logits[0, -1].argmax()) or (logits[0, -1] - ref_logits[0, -1]).abs().max() < 0.1
    k, rk = cache.k_cache[:, :, :T + 1].float(), ref_cache.k_cache[:, :, :T + 1].float()
    v, rv = cache.v_cache[:, :, :T + 1].float(), ref_cache.v_cache[:, :, :T + 1].float()
    for got, want in ((k, rk), (v, rv)):
        assert (got - want).abs().max().item() < 0.05 + 0.03 * want.abs().max().item()
        assert (got - want).abs().mean().item() < 0.01 * want.abs().mean().item() + 1e-3
    assert cache.k_cache[:, :, T + 1:].abs().sum().item() == 0           # nothing written past the prompt
    assert (step - ref_step).abs().max().item() < 0.25


def test_sampling_kernel_semantics():
    from nanochat_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(7)
    B, V = 4, 32768
    logits = (torch.randn(B, V, device="cuda", generator=g) * 3).float()
    logits[1, 77] = 50.0
    # temperature 0: argmax, first index on ties
    logits[2, 100] = logits[2, 200] = 60.0
    out = nat.sample_next_token(logits, None, 0.0, None)
    assert out[:, 0].tolist() == logits.argmax(dim=-1).tolist() and out[2, 0].item() == 100
    # top-k: every draw lies inside the top-k set; same seed -> same tokens; different seeds differ somewhere
    k = 50
    topk = torch.topk(logits, k, dim=-1).indices
    draws = []
    for seed in (1, 1, 2):
        rng = torch.Generator(device="cuda").manual_seed(seed)
        cols = [nat.sample_next_token(logits, rng, 1.0, k)[:, 0] for _ in range(16)]
        draws.append(torch.stack(cols, 1))
    assert torch.equal(draws[0], draws[1]) and not torch.equal(draws[0], draws[2])
    for b in range(B):
        assert set(draws[0][b].tolist()) <= set(topk[b].tolist())
    assert (draws[0][1] == 77).all()                    # a dominating logit is always drawn
    # distribution: empirical frequencies of the top entries follow softmax over the top-k set
    row = logits[0:1].expand(4096, V).contiguous()
    rng = torch.Generator(device="cuda").manual_seed(3)
    samples = nat.sample_next_token(row, rng, 1.0, k)[:, 0]
    vals, idx = torch.topk(logits[0], k)
    probs = torch.softmax(vals, 0)
    for j in range(3):
        freq = (samples == idx[j]).float().mean().item()
        assert abs(freq - probs[j].item()) < 0.03 + 0.2 * probs[j].item(), (j, freq, probs[j].item())
    # no top-k: full-vocabulary sampling at a low temperature concentrates on the maximum
    rng = torch.Generator(device="cuda").manual_seed(4)
    cold = nat.sample_next_token(logits, rng, 0.05, None)[:, 0]
    assert (cold == logits.argmax(-1)).float().mean().item() >= 0.5


def test_paged_decode_kernels_match_contiguous_cache():
    """The same keys and values behind a shuffled page table: the attention output is bitwise the contiguous one (same
    arithmetic, other addresses), and the append writes the new token's K/V into the page its position maps to."""
    from nanochat_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(11)
    B, H, Hkv, T, P = 3, 4, 2, 320, 64
    kc = torch.randn(B, T, Hkv, 128, device="cuda", generator=g).to(BF16)
    vc = torch.randn(B, T, Hkv, 128, device="cuda", generator=g).to(BF16)
    q = torch.randn(B, H * 128, device="cuda", generator=g).to(BF16)
    seqlens = torch.tensor([5, 150, 299], dtype=torch.int32, device="cuda")
    n_pages = T // P
    perm = torch.randperm(B * n_pages, device="cuda", generator=g)
    table = perm.view(B, n_pages).to(torch.int32).contiguous()
    k_pool = torch.zeros(B * n_pages + 1, P, Hkv, 128, dtype=BF16, device="cuda")
    v_pool = torch.zeros_like(k_pool)
    k_pool[table.long().view(-1)] = kc.view(B * n_pages, P, Hkv, 128)
    v_pool[table.long().view(-1)] = vc.view(B * n_pages, P, Hkv, 128)
    scratch = torch.zeros(nat._C.decode_attn_scratch(B, H), dtype=torch.float32, device="cuda")
    for window in (-1, 64):
        want = torch.empty(B, H * 128, dtype=BF16, device="cuda")
        got = torch.empty_like(want)
        nat._C.decode_attn(q, kc, vc, seqlens, H, Hkv, window, 1.0 / math.sqrt(128), scratch, want)
        nat._C.decode_attn(q, k_pool, v_pool, seqlens, H, Hkv, window, 1.0 / math.sqrt(128), scratch, got, table)
        assert torch.equal(got, want), window
    # append: rotary + norm of k, plain v, written at (row, seqlens[row]) through the table
    qkv = torch.randn(B, (H + 2 * Hkv) * 128, device="cuda", generator=g).to(BF16)
    cos = torch.randn(T, 64, device="cuda", generator=g).to(BF16)
    sin = torch.randn(T, 64, device="cuda", generator=g).to(BF16)
    a, b = qkv.clone(), qkv.clone()
    kc2, vc2 = kc.clone(), vc.clone()
    nat._C.decode_qkv_post(a, H, Hkv, cos, sin, seqlens, None, None, None, None, kc2, vc2)
    nat._C.decode_qkv_post(b, H, Hkv, cos, sin, seqlens, None, None, None, None, k_pool, v_pool, table, T)
    assert torch.equal(a, b)
    for row in range(B):
        pos = int(seqlens[row])
        page = int(table[row, pos // P])
        assert torch.equal(k_pool[page, pos % P], kc2[row, pos])
        assert torch.equal(v_pool[page, pos % P], vc2[row, pos])
    nat.check_status()


def test_paged_engine_cache_holds_the_prompt_once():
    """Many samples of one prompt: the page tables of all rows name the same pages for the prompt's full pages, each
    row owns its partial page and what it decodes, the pool is far smaller than one contiguous cache per row, and the
    tokens are those of the contiguous op-level path."""
    from nanochat_b200 import ops
    from nanochat_b200.engine import Engine, PagedKVCache, PAGE_TOKENS
    model = _model()
    cfg = model.config
    g = torch.Generator().manual_seed(5)
    prompt = torch.randint(0, 2040, (150,), generator=g).tolist()          # 2 full pages + 22 tokens
    rows, new = 8, 20
    eng = Engine(model, _Tok())
    fast = [c for c, _ in eng.generate(prompt, num_samples=rows, max_tokens=new, temperature=0.0)]
    cache = eng._cache_pool[rows]
    assert isinstance(cache, PagedKVCache)
    table = cache.table.cpu()
    full = len(prompt) // PAGE_TOKENS
    assert full == 2
    assert all(table[r, :full].tolist() == [0, 1] for r in range(rows))        # shared prompt pages
    own = table[:, full].tolist()
    assert len(set(own)) == rows and min(own) >= cache.shared_pages            # private continuation pages
    per_token = 2 * cfg.n_layer * cfg.n_kv_head * 128 * 2
    contiguous = rows * (len(prompt) + new) * per_token
    assert cache.pool_bytes() < 0.6 * contiguous, (cache.pool_bytes(), contiguous)
    # every row's keys of the prompt are the shared ones
    k0, _ = cache.gather_row(0, 0)
    k5, _ = cache.gather_row(0, 5)
    assert torch.equal(k0[:len(prompt)], k5[:len(prompt)])
    ops.native_module().check_status()
    eng2 = Engine(model, _Tok())
    eng2._pooled_cache = lambda *a, **k: None
    slow = [c for c, _ in eng2.generate(prompt, num_samples=rows, max_tokens=new, temperature=0.0)]
    agree = 0
    for a, b in zip(fast, slow):
        if a != b:
            break
        agree += 1
    assert agree >= 8, (agree, fast[:10], slow[:10])
    assert all(len(set(col)) == 1 for col in fast[:8])                        # greedy: every row decodes the same tokens
    # a longer request grows the pool; the graph is rebuilt on the new pool and still agrees with itself
    longer = [c for c, _ in eng.generate(prompt, num_samples=rows, max_tokens=new + 70, temperature=0.0)]
    assert longer[:agree] == fast[:agree]
    ops.native_module().check_status()


@pytest.mark.parametrize("B,H,Hkv,T,window,common", [(1, 13, 13, 700, -1, 0), (3, 4, 2, 320, 64, 0), (64, 4, 4, 130, -1, 0),
                                                     (2, 2, 1, 9000, 4000, 0), (2, 13, 13, 700, 130, 9), (5, 4, 2, 320, -1, 1), (8, 13, 13, 700, 300, 10),
                                                     (17, 4, 4, 200, -1, 2), (64, 13, 13, 400, 100, 5), (3, 2, 1, 9000, 4000, 130)])
def test_fused_append_and_attention_matches_the_two_kernels(B, H, Hkv, T, window, common):
    """Same roundings, other summation order: y is bf16 of float sums over up to 9000 keys, so 2^-8 of a value and what the order of
    the sums moves (1e-3). Positions at the ends of splits, batches, pages and the window;
    more pages than the shared-memory table takes (T = 9000)."""
    from nanochat_b200.ops import native as nat
    P, g = 64, torch.Generator(device="cuda").manual_seed(5)
    pages = -(-T // P)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(BF16)
    table = torch.randperm(B * pages, device="cuda", generator=g).view(B, pages).to(torch.int32).contiguous()
    table[:, :common] = table[:1, :common].clone()                       # the first pages are the same for all rows
    k_pool, v_pool = rnd(B * pages + 1, P, Hkv, 128), rnd(B * pages + 1, P, Hkv, 128)
    cos, sin, qkv, xn = rnd(T, 64), rnd(T, 64), rnd(B, (H + 2 * Hkv) * 128), rnd(B, 256)
    wg, ve = torch.randn(Hkv, 12, device="cuda", generator=g), rnd(50, Hkv * 128)
    idx = torch.randint(0, 50, (B,), device="cuda", generator=g)
    scratch = torch.zeros(nat._C.decode_attn_scratch(B, H), dtype=torch.float32, device="cuda")
    for base in (0, 1, 15, 16, 63, 64, 127, T - 1):
        base = max(base, common * P + B) if common else base             # a row appends to pages of its own
        seqlens = torch.tensor([max(0, min(T - 1, base - b)) for b in range(B)], dtype=torch.int32, device="cuda")
        for gated in (False, True):
            extra = (xn, wg, ve, idx) if gated else (None,) * 4
            k1, v1, k2, v2, q1 = k_pool.clone(), v_pool.clone(), k_pool.clone(), v_pool.clone(), qkv.clone()
            want, got = torch.empty(B, H * 128, dtype=BF16, device="cuda"), torch.empty(B, H * 128, dtype=BF16, device="cuda")
            nat._C.decode_qkv_post(q1, H, Hkv, cos, sin, seqlens, *extra, k1, v1, table, T)
            nat._C.decode_attn(q1[:, :H * 128], k1, v1, seqlens, H, Hkv, window, 0.088, scratch, want, table)
            torch.cuda.synchronize()
            nat._C.decode_qkv_attn(qkv, H, Hkv, cos, sin, seqlens, *extra, k2, v2, window, 0.088, got, table, T)
            for a, b in ((k1, k2), (v1, v2)):
                # the norm's sum has another order: a value may round to the neighbouring bf16, 2^-7 of it at most, seldom
                off = (a.float() - b.float()).abs()
                assert (off <= 2.0 ** -7 * a.float().abs() + 1e-6).all() and (off > 0).sum().item() <= 1e-3 * B * Hkv * 256 + 1
            assert ((got.float() - want.float()).norm() / want.float().norm()).item() < 4e-3, (base, gated)
    full = torch.full((B,), T, dtype=torch.int32, device="cuda")        # a full row: recorded, nothing appended
    k2 = k_pool.clone()
    torch.cuda.synchronize()
    nat._C.decode_qkv_attn(qkv, H, Hkv, cos, sin, full, None, None, None, None, k2, v_pool, window, 0.088, got, table, T)
    assert torch.equal(k2, k_pool)
    with pytest.raises(RuntimeError):
        nat.check_status()


@pytest.mark.parametrize("tokens", [2, 63, 64, 65, 200])
def test_prompt_in_one_call_matches_the_op_by_op_forward(tokens):
    """Logits of wanted and of all positions, keys and values: against the same weights without a cache, where every layer runs as
    the training forward does. Two bf16 forwards of four layers; the switch to the few-row products lies at 64 tokens."""
    from nanochat_b200.engine import KVCache
    model = _model()
    cfg = model.config
    ids = torch.randint(0, cfg.vocab_size, (1, tokens), device="cuda", generator=torch.Generator(device="cuda").manual_seed(tokens))
    mk = lambda: KVCache(batch_size=1, num_heads=cfg.n_kv_head, seq_len=256, head_dim=128, num_layers=cfg.n_layer, device="cuda", dtype=BF16)
    with torch.inference_mode():
        want = model.forward(ids)
        a, b, c = mk(), mk(), mk()
        every, some = model.forward(ids, kv_cache=a), model.forward(ids, kv_cache=b, want=[tokens - 1, 0])
        assert model.forward(ids, kv_cache=c, want=[]) is None and c.get_pos() == tokens
        close = lambda x, y: ((x.float() - y.float()).norm() / y.float().norm()).item() < 2e-2
        assert close(every, want) and close(some, want[:, [tokens - 1, 0]])
        for layer in range(cfg.n_layer):
            for x, y in zip(a.get_layer_cache(layer), b.get_layer_cache(layer)):
                assert torch.equal(x, y) and x[:, tokens:].abs().sum().item() == 0 and (x[:, :tokens].abs().sum(-1) > 0).all()
