"""Each kernel alone against its plain reference, at sizes other than the engine's."""
import math

import pytest
import torch

import plain_llama as P

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
TOL = {"float32": 2e-6, "bfloat16": 1e-2}


def close(got, ref, dtype, scale=None):
    ref = ref.to(torch.float64)
    err = float((got.detach().to(torch.float64).cpu() - ref.cpu()).abs().max())
    bound = TOL[dtype] * (scale if scale is not None else float(ref.abs().max()) + 1e-30)
    assert err <= bound, f"max abs err {err:.3e} > {bound:.3e}"


def rnd(shape, dtype, seed, std=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * std).to(DT[dtype]).to(DEV)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_embedding(dtype):
    from libllm_b200.csrc import ops
    table = rnd((1000, 200), dtype, 1)
    ids = torch.tensor([0, 999, 5, 5, 321], dtype=torch.int32, device=DEV)
    out = torch.empty((5, 200), dtype=torch.float32, device=DEV)
    ops.embedding(table, ids, out)
    assert torch.equal(out.cpu(), P.embedding(table.cpu(), ids.tolist()).float())


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("hidden,parts", [(200, 0), (200, 1), (72, 3), (13000, 2)])
def test_add_rmsnorm(dtype, hidden, parts):
    from libllm_b200.csrc import ops
    T = 7
    resid = rnd((T, hidden), "float32", 2)
    delta = rnd((parts, T, hidden), dtype, 3) if parts else None
    w = rnd((hidden,), "float32", 4) * 0.1 + 1
    out = torch.empty((T, hidden), dtype=DT[dtype], device=DEV)
    want = resid.double().cpu() + (delta.double().cpu().sum(0) if parts else 0)
    r2 = resid.clone()
    ops.add_rmsnorm(r2, delta, w, 1e-5, out)
    close(r2, want, "float32")
    close(out, P.rms_norm(want, w.cpu(), 1e-5), dtype)
    # a subset of rows, residual left alone
    rows = torch.tensor([6, 0, 3], dtype=torch.int32, device=DEV)
    r3 = resid.clone()
    out3 = torch.empty((3, hidden), dtype=DT[dtype], device=DEV)
    ops.add_rmsnorm(r3, delta, w, 1e-5, out3, rows)
    assert torch.equal(r3, resid)
    close(out3, P.rms_norm(want[[6, 0, 3]], w.cpu(), 1e-5), dtype)
    # add only
    r4 = resid.clone()
    ops.add_rmsnorm(r4, delta, None, 0.0, None)
    close(r4, want, "float32")


@pytest.mark.parametrize("dtype,in_dtype", [("float32", "float32"), ("bfloat16", "bfloat16"), ("bfloat16", "float32")])
@pytest.mark.parametrize("inter", [173, 176])        # the general kernel, and four values per thread
def test_swiglu(dtype, in_dtype, inter):
    from libllm_b200.csrc import ops
    gu = rnd((9, 2 * inter), in_dtype, 5, 2.0)
    gu[0, 0] = -30.0
    gu[0, 1] = 30.0
    out = torch.empty((9, inter), dtype=DT[dtype], device=DEV)
    ops.swiglu(gu, out)
    close(out, P.swiglu(gu[:, :inter].cpu(), gu[:, inter:].cpu()), dtype)


@pytest.mark.parametrize("dtype,out_dtype", [("float32", "float32"), ("bfloat16", "bfloat16"), ("bfloat16", "float32")])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (5, 7, 3), (513, 2, 513), (70, 130, 1000), (64, 64, 16)])
def test_gemm_plain(dtype, out_dtype, M, N, K):
    from libllm_b200.csrc import ops
    a, w = rnd((M, K), dtype, 6), rnd((N, K), dtype, 7)
    bias = rnd((N,), "float32", 8)
    out = torch.empty((M, N), dtype=DT[out_dtype], device=DEV)
    ops.gemm_plain(a, w, out, bias)
    ref = P.linear(a.cpu(), w.cpu(), bias.cpu())
    close(out, ref, out_dtype, scale=float(ref.abs().max()) + math.sqrt(K) * 1e-1)


def test_gemm_plain_rows_do_not_depend_on_the_batch():
    from libllm_b200.csrc import ops
    a, w = rnd((130, 300), "float32", 9), rnd((77, 300), "float32", 10)
    full = torch.empty((130, 77), device=DEV)
    one = torch.empty((1, 77), device=DEV)
    ops.gemm_plain(a, w, full)
    ops.gemm_plain(a[97:98], w, one)
    assert torch.equal(full[97:98], one)


def paged_cache(n_seqs, lens, n_kv, d, page, dtype, seed):
    """Random keys/values per sequence scattered over shuffled pages."""
    per = [(l + page - 1) // page for l in lens]
    n_pages = sum(per) + 3
    g = torch.Generator().manual_seed(seed)
    perm = torch.randperm(n_pages, generator=g).tolist()
    width = max(per) + 1
    table = torch.zeros((n_seqs, width), dtype=torch.int32)
    K = torch.full((n_pages, n_kv, page, d), 1e4).to(DT[dtype])     # unread places are poisoned
    V = torch.full((n_pages, n_kv, page, d), -1e4).to(DT[dtype])
    ks, vs = [], []
    o = 0
    for s, l in enumerate(lens):
        k = (torch.randn((l, n_kv, d), generator=g)).to(DT[dtype])
        v = (torch.randn((l, n_kv, d), generator=g)).to(DT[dtype])
        ks.append(k)
        vs.append(v)
        for lp in range(per[s]):
            pg = perm[o]
            o += 1
            table[s, lp] = pg
            n = min(page, l - lp * page)
            K[pg, :, :n] = k[lp * page:lp * page + n].transpose(0, 1)
            V[pg, :, :n] = v[lp * page:lp * page + n].transpose(0, 1)
    return K.to(DEV), V.to(DEV), table.to(DEV), ks, vs


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("n_heads,n_kv,d,window", [(4, 2, 16, None), (3, 1, 48, None), (8, 8, 128, None),
                                                     (6, 2, 256, None), (4, 1, 32, 37), (2, 2, 64, 64)])
def test_attention_generic(dtype, n_heads, n_kv, d, window):
    from libllm_b200.csrc import ops
    page = 16
    lens = [1, 70, 33, 130]
    q_lens = [1, 70, 5, 1]          # a whole prompt, the end of one, and single tokens
    K, V, table, ks, vs = paged_cache(4, lens, n_kv, d, page, dtype, 11)
    T = sum(q_lens)
    q = rnd((T, n_heads * d), dtype, 12)
    tok_seq = torch.tensor([s for s, n in enumerate(q_lens) for _ in range(n)], dtype=torch.int32, device=DEV)
    tok_pos = torch.tensor([lens[s] - n + i for s, n in enumerate(q_lens) for i in range(n)], dtype=torch.int32, device=DEV)
    out = torch.empty((T, n_heads * d), dtype=DT[dtype], device=DEV)
    scale = 1 / math.sqrt(d)
    ops.attention_generic(q, out, K, V, tok_seq, tok_pos, table, n_heads, n_kv, d, page, window, scale)
    o = 0
    for s, n in enumerate(q_lens):
        ref = P.attention_scores_softmax_values(q[o:o + n].cpu().view(n, n_heads, d), ks[s], vs[s], window)
        close(out[o:o + n].view(n, n_heads, d), ref, dtype, scale=1.0)
        o += n


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_attention_finds_one_far_key_among_hundreds(dtype):
    """Key 3 of 900 matches the query strongly; its value must dominate the output."""
    from libllm_b200.csrc import ops
    n_heads = n_kv = 1
    d, page, L = 64, 64, 900
    K, V, table, ks, vs = paged_cache(1, [L], n_kv, d, page, dtype, 13)
    q = rnd((1, d), dtype, 14)
    k3 = (q[0].float().cpu() * 3.0).to(DT[dtype])
    pg = int(table[0, 0])
    K[pg, 0, 3] = k3.to(DEV)
    ks[0][3, 0] = k3
    out = torch.empty((1, d), dtype=DT[dtype], device=DEV)
    pos = torch.tensor([L - 1], dtype=torch.int32, device=DEV)
    ops.attention_generic(q, out, K, V, torch.zeros(1, dtype=torch.int32, device=DEV), pos, table, 1, 1, d, page,
                          None, 1 / math.sqrt(d))
    ref = P.attention_scores_softmax_values(q.cpu().view(1, 1, d), ks[0], vs[0])
    close(out.view(1, 1, d), ref, dtype, scale=1.0)
    assert float((out.float().cpu()[0] - vs[0][3, 0].float()).abs().max()) < 0.2


def test_attention_of_more_heads_and_tokens_than_one_grid_takes():
    """One key each, so that every result is its value; 2^31 + 1,024 (token, head) pairs."""
    from libllm_b200.csrc import ops
    T, H = 2 ** 21 + 1, 1024
    i32 = dict(dtype=torch.int32, device=DEV)
    K, V = (torch.full((1, 1, 16, 1), x, dtype=torch.bfloat16, device=DEV) for x in (1.0, 0.75))
    q = torch.zeros((T, H), dtype=torch.bfloat16, device=DEV)
    out = torch.zeros_like(q)
    ops.attention_generic(q, out, K, V, torch.zeros(T, **i32), torch.zeros(T, **i32), torch.zeros((1, 1), **i32), H, 1, 1, 16, None, 1.0)
    assert float(out.min()) == float(out.max()) == 0.75
    del q, out
    torch.cuda.empty_cache()


# blocks of 32 keys of the first, a later and several warps; all but the last key
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("lo,hi", [(0, 32), (32, 64), (32, 160), (0, 199)])
def test_keys_of_score_minus_infinity_weigh_nothing(dtype, lo, hi):
    from libllm_b200.csrc import ops
    d, page, L = 64, 64, 200
    K, V, table, ks, vs = paged_cache(1, [L], 1, d, page, dtype, 18)
    q = rnd((1, d), dtype, 19)
    q[0, 0] = 1.0
    for j in range(lo, hi):
        K[int(table[0, j // page]), 0, j % page, 0] = float("-inf")
    out = torch.empty((1, d), dtype=DT[dtype], device=DEV)
    i32 = dict(dtype=torch.int32, device=DEV)
    ops.attention_generic(q, out, K, V, torch.zeros(1, **i32), torch.tensor([L - 1], **i32), table, 1, 1, d, page, None, 1 / math.sqrt(d))
    seen = [j for j in range(L) if not lo <= j < hi]
    ref = P.attention_scores_softmax_values(q.cpu().view(1, 1, d), ks[0][seen], vs[0][seen])
    close(out.view(1, 1, d), ref, dtype, scale=max(1.0, float(ref.abs().max())))


@pytest.mark.parametrize("dtype,in_dtype", [("float32", "float32"), ("bfloat16", "bfloat16"), ("bfloat16", "float32")])
@pytest.mark.parametrize("n_heads,n_kv,d", [(4, 2, 16), (3, 1, 96)])
def test_rope_and_cache_write(dtype, in_dtype, n_heads, n_kv, d):
    from libllm_b200.csrc import ops
    from helpers import rotary_frequencies
    page, n_pages = 8, 12
    lens_past, q_lens = [0, 13, 40], [9, 1, 3]
    T = sum(q_lens)
    width = (n_heads + 2 * n_kv) * d
    qkv = rnd((T, width), in_dtype, 15)
    qkv0 = qkv.clone()
    q_out = torch.zeros((T, n_heads * d), dtype=DT[dtype], device=DEV)
    freqs = torch.tensor(rotary_frequencies(d, 10000.0, None), dtype=torch.float64)
    pos = torch.arange(64, dtype=torch.float64)
    ang = pos[:, None] * freqs[None]
    table = torch.cat([ang.cos(), ang.sin()], 1).float().to(DEV)
    tok_seq = torch.tensor([s for s, n in enumerate(q_lens) for _ in range(n)], dtype=torch.int32, device=DEV)
    tok_pos = torch.tensor([lens_past[s] + i for s, n in enumerate(q_lens) for i in range(n)], dtype=torch.int32, device=DEV)
    pt = torch.tensor([[3, 7, 0, 0, 0, 0], [1, 2, 0, 0, 0, 0], [4, 5, 6, 8, 9, 10]], dtype=torch.int32, device=DEV)
    K = torch.zeros((n_pages, n_kv, page, d), dtype=DT[dtype], device=DEV)
    V = torch.zeros_like(K)
    ops.rope_cache_write(qkv, q_out, n_heads, n_kv, d, table, tok_seq, tok_pos, pt, K, V, page)
    assert torch.equal(qkv, qkv0)
    x = qkv0.cpu().view(T, n_heads + 2 * n_kv, d)
    positions = tok_pos.cpu().to(torch.float64)
    qr = P.rope_rotate(x[:, :n_heads], positions, freqs)
    kr = P.rope_rotate(x[:, n_heads:n_heads + n_kv], positions, freqs)
    close(q_out.cpu().view(T, n_heads, d), qr, dtype)
    for t in range(T):
        s, p = int(tok_seq[t]), int(tok_pos[t])
        pg = int(pt[s, p // page])
        close(K[pg, :, p % page], kr[t], dtype)
        assert torch.equal(V[pg, :, p % page].cpu(), x[t, n_heads + n_kv:].to(DT[dtype]))
    # places no token was written to stay untouched
    written = {(int(pt[int(tok_seq[t]), int(tok_pos[t]) // page]), int(tok_pos[t]) % page) for t in range(T)}
    for pg in range(n_pages):
        for r in range(page):
            if (pg, r) not in written:
                assert float(K[pg, :, r].abs().max()) == 0.0


def test_argmax_and_ties():
    from libllm_b200.csrc import ops
    logits = rnd((5, 3001), "float32", 16)
    logits[1, 17] = logits[1, 2900] = 50.0          # tie: the lower index wins
    logits[2, 3000] = 60.0
    out = torch.empty(5, dtype=torch.int32, device=DEV)
    ops.argmax(logits, out)
    want = [P.sample_token(logits[i].cpu(), 0.0, 0, 1.0, 0.0) for i in range(5)]
    assert out.tolist() == want and want[1] == 17 and want[2] == 3000


def _interval_ok(logits_row, temperature, top_k, top_p, u, token):
    """``token`` is what the plain sampler returns for a number within 1e-5 of u."""
    return any(P.sample_token(logits_row, temperature, top_k, top_p, min(max(u + du, 0.0), 0.9999999)) == token
               for du in (0.0, -1e-5, 1e-5))


@pytest.mark.parametrize("vocab", [331, 128256])
@pytest.mark.parametrize("temperature,top_k,top_p", [(1.0, 50, 0.8), (0.7, 5, 1.0), (1.3, 1, 0.5), (0.8, 0, 1.0),
                                                      (1.0, 1024, 0.95)])
def test_sampling_matches_plain_sampler(vocab, temperature, top_k, top_p):
    from libllm_b200.csrc import ops
    B = 6
    logits = rnd((B, vocab), "float32", 17, 3.0)
    logits[0, 5] = logits[0, 9] = logits[0].max() + 1.0        # tied leaders
    us = [0.0, 0.1234, 0.5, 0.77, 0.999, 0.31]
    uni = torch.tensor(us, dtype=torch.float32, device=DEV)
    out = torch.empty(B, dtype=torch.int32, device=DEV)
    ops.sample(logits, temperature, top_k, top_p, uni, out)
    for i in range(B):
        assert _interval_ok(logits[i].cpu(), temperature, min(top_k, vocab), top_p, us[i], int(out[i])), (i, int(out[i]))
    # a row's draw does not depend on its neighbours
    out1 = torch.empty(1, dtype=torch.int32, device=DEV)
    ops.sample(logits[3:4], temperature, top_k, top_p, uni[3:4], out1)
    assert int(out1[0]) == int(out[3])
    # temperature 0 is argmax
    ops.sample(logits, 0.0, top_k, top_p, uni, out)
    want = logits.argmax(-1).tolist()
    want[0] = 5                                  # tied leaders: the lower index wins
    assert out.tolist() == want


@pytest.mark.parametrize("case", ["flat", "many_tied_leaders", "ties_at_the_kth", "none_near_the_maximum"])
def test_sampling_rows_that_the_quick_selection_must_get_right_or_hand_on(case):
    """Rows at the edges of the two ways the kernel finds the top_k: all logits equal and thousands
    of tied leaders (more candidates than the quick selection sorts), ties exactly at the k-th place
    inside it (the lower indices are taken), and fewer than top_k logits near the maximum."""
    from libllm_b200.csrc import ops
    V, top_k = 20000, 50
    g = torch.Generator().manual_seed(23)
    if case == "flat":
        row = torch.full((V,), 1.5)
    elif case == "many_tied_leaders":
        row = torch.randn(V, generator=g) - 30.0
        row[torch.randperm(V, generator=g)[:3000]] = 4.0
    elif case == "ties_at_the_kth":
        row = torch.randn(V, generator=g) - 40.0
        idx = torch.randperm(V, generator=g)
        row[idx[:10]] = torch.linspace(5.0, 6.0, 10)
        row[idx[10:1510]] = 4.0
    else:
        row = torch.randn(V, generator=g) * 0.1 - 50.0
        row[torch.randperm(V, generator=g)[:7]] = torch.linspace(1.0, 3.0, 7)
    us = [0.0, 0.21, 0.5, 0.83, 0.97, 0.9999]
    logits = row.to(DEV).repeat(len(us), 1).contiguous()
    uni = torch.tensor(us, dtype=torch.float32, device=DEV)
    out = torch.empty(len(us), dtype=torch.int32, device=DEV)
    for temperature, top_p in ((1.0, 1.0), (0.7, 0.9)):
        ops.sample(logits, temperature, top_k, top_p, uni, out)
        for i, u in enumerate(us):
            assert _interval_ok(row, temperature, top_k, top_p, u, int(out[i])), (case, temperature, top_p, u, int(out[i]))


def test_kernels_refuse_what_they_cannot_do():
    from libllm_b200.csrc import ops
    from libllm_b200.errors import ExtensionError, UnsupportedError
    with pytest.raises(ExtensionError):
        ops.swiglu(torch.zeros(2, 4), torch.zeros(2, 2))          # host tensors: no CPU fallback
    logits = rnd((1, 100), "float32", 18)
    with pytest.raises(UnsupportedError):
        ops.sample(logits, 1.0, 5000, 1.0, torch.zeros(1, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV))


@pytest.mark.parametrize("out_dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("M,N,K", [(1, 96, 64), (8, 200, 80), (3, 331, 176), (16, 2048, 2048), (33, 130, 520),
                                   (64, 1000, 4096), (7, 17, 8)])
def test_small_batch_product(out_dtype, M, N, K):
    from libllm_b200.csrc import ops
    x, w = rnd((M, K), "bfloat16", 20), rnd((N, K), "bfloat16", 21, 0.05)
    out = torch.empty((M, N), dtype=DT[out_dtype], device=DEV)
    ops.gemv_bf16(x, w, out)
    ref = P.linear(x.cpu(), w.cpu())
    close(out, ref, out_dtype, scale=float(ref.abs().max()))
    # one token's result does not depend on the others in the batch: bit for bit when the
    # batch has the same size, to rounding when the size (and with it the K split) differs
    x2 = rnd((M, K), "bfloat16", 99)
    x2[M - 1] = x[M - 1]
    out2 = torch.empty((M, N), dtype=DT[out_dtype], device=DEV)
    ops.gemv_bf16(x2, w, out2)
    assert torch.equal(out2[M - 1], out[M - 1])
    one = torch.empty((1, N), dtype=DT[out_dtype], device=DEV)
    ops.gemv_bf16(x[M - 1:M], w, one)
    close(one, ref[M - 1:M], out_dtype, scale=float(ref.abs().max()))


@pytest.mark.parametrize("M,I,K", [(1, 96, 64), (5, 173, 80), (8, 8192, 2048), (40, 300, 256)])
def test_small_batch_product_with_swiglu(M, I, K):
    from libllm_b200.csrc import ops
    x, w = rnd((M, K), "bfloat16", 22), rnd((2 * I, K), "bfloat16", 23, 0.2)
    out = torch.empty((M, I), dtype=torch.bfloat16, device=DEV)
    ops.gemv_bf16(x, w, out, swiglu=True)
    gu = P.linear(x.cpu(), w.cpu())
    close(out, P.swiglu(gu[:, :I], gu[:, I:]), "bfloat16")


@pytest.mark.parametrize("n_heads,n_kv,d,window", [(4, 2, 16, None), (3, 1, 32, None), (32, 8, 64, None),
                                                     (8, 1, 128, None), (8, 8, 64, None), (6, 2, 128, 100)])
@pytest.mark.parametrize("chunk,n_splits", [(64, 16), (192, 6), (1024, 1)])
def test_attention_decode(n_heads, n_kv, d, window, chunk, n_splits):
    from libllm_b200.csrc import ops
    page = 64
    lens = [1, 70, 333, 1000, 64]
    B = len(lens)
    K, V, table, ks, vs = paged_cache(B, lens, n_kv, d, page, "bfloat16", 24)
    q = rnd((B, n_heads * d), "bfloat16", 25)
    pos = torch.tensor([l - 1 for l in lens], dtype=torch.int32, device=DEV)
    out = torch.empty((B, n_heads * d), dtype=torch.bfloat16, device=DEV)
    ws_o = torch.full((B * n_heads * n_splits * d,), float("nan"), device=DEV)
    ws_ml = torch.full((B * n_heads * n_splits * 2,), float("nan"), device=DEV)
    assert ops.attention_decode_supported(d, n_heads // n_kv)
    ops.attention_decode(q, out, K, V, pos, table, n_heads, n_kv, d, page, chunk, n_splits, window, 1 / math.sqrt(d),
                         ws_o, ws_ml)
    for b in range(B):
        ref = P.attention_scores_softmax_values(q[b:b + 1].cpu().view(1, n_heads, d), ks[b], vs[b], window)
        close(out[b].view(1, n_heads, d), ref, "bfloat16", scale=1.0)


# runs of keys beside the eight asked for together and the 64 whose weights lie in shared memory; one to two channels a thread
@pytest.mark.parametrize("n_heads,n_kv,d", [(2, 1, 16), (4, 1, 64), (1, 1, 128)])
def test_many_runs_of_keys_are_joined(n_heads, n_kv, d):
    from libllm_b200.csrc import ops
    lens, page, n_splits = [511, 512, 513, 4095, 4096, 4097, 4500], 64, 72
    B = len(lens)
    K, V, table, ks, vs = paged_cache(B, lens, n_kv, d, page, "bfloat16", 27)
    q = rnd((B, n_heads * d), "bfloat16", 28)
    pos = torch.tensor([l - 1 for l in lens], dtype=torch.int32, device=DEV)
    out = torch.empty((B, n_heads * d), dtype=torch.bfloat16, device=DEV)
    ws_o, ws_ml = (torch.full((B * n_heads * n_splits * w,), float("nan"), device=DEV) for w in (d, 2))
    ops.attention_decode(q, out, K, V, pos, table, n_heads, n_kv, d, page, 64, n_splits, None, 1 / math.sqrt(d), ws_o, ws_ml)
    for b in range(B):
        ref = P.attention_scores_softmax_values(q[b:b + 1].cpu().view(1, n_heads, d), ks[b], vs[b], None)
        close(out[b].view(1, n_heads, d), ref, "bfloat16", scale=1.0)


def prefill_inputs(lens, q_lens):
    start = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=DEV)
    past = torch.tensor([l - n for l, n in zip(lens, q_lens)], dtype=torch.int32, device=DEV)
    return start, past


@pytest.mark.parametrize("n_heads,n_kv,d,window", [(4, 2, 16, None), (3, 1, 48, None), (32, 8, 64, None),
                                                     (5, 5, 80, None), (8, 2, 128, None), (4, 1, 32, 37),
                                                     (2, 2, 64, 64), (6, 3, 112, 130)])
def test_attention_prefill(n_heads, n_kv, d, window):
    """Whole prompts, the end of a prompt behind cached tokens, tile edges (63, 64, 65 rows) and
    single tokens in one launch, against the plain attention of each sequence."""
    from libllm_b200.csrc import ops
    page = 64
    lens = [1, 70, 333, 200, 64, 65, 63]
    q_lens = [1, 70, 5, 150, 64, 65, 1]
    B = len(lens)
    K, V, table, ks, vs = paged_cache(B, lens, n_kv, d, page, "bfloat16", 31)
    T = sum(q_lens)
    q = rnd((T, n_heads * d), "bfloat16", 32)
    out = torch.full((T, n_heads * d), float("nan"), dtype=torch.bfloat16, device=DEV)
    start, past = prefill_inputs(lens, q_lens)
    assert ops.attention_prefill_supported(d, page)
    ops.attention_prefill(q, out, K, V, start, past, table, B, max(q_lens), n_heads, n_kv, d, page, window,
                          1 / math.sqrt(d))
    o = 0
    for s, n in enumerate(q_lens):
        ref = P.attention_scores_softmax_values(q[o:o + n].cpu().view(n, n_heads, d), ks[s], vs[s], window)
        close(out[o:o + n].view(n, n_heads, d), ref, "bfloat16", scale=1.0)
        o += n


def test_attention_prefill_finds_a_far_key_and_respects_the_window_edge():
    """Row 700 of a 900-token prompt matches key 3 strongly: without a window key 3's value
    dominates that row; with a window of 697 key 3 is the last one outside (700 - 697 = 3) and
    must not be seen, with 698 it is the first one inside."""
    from libllm_b200.csrc import ops
    d, page, L = 64, 64, 900
    K, V, table, ks, vs = paged_cache(1, [L], 1, d, page, "bfloat16", 33)
    q = rnd((L, d), "bfloat16", 34)
    k3 = (q[700].float().cpu() * 3.0).to(torch.bfloat16)
    K[int(table[0, 0]), 0, 3] = k3.to(DEV)
    ks[0][3, 0] = k3
    start, past = prefill_inputs([L], [L])
    for window, sees in ((None, True), (697, False), (698, True)):
        out = torch.empty((L, d), dtype=torch.bfloat16, device=DEV)
        ops.attention_prefill(q, out, K, V, start, past, table, 1, L, 1, 1, d, page, window, 1 / math.sqrt(d))
        ref = P.attention_scores_softmax_values(q.cpu().view(L, 1, d), ks[0], vs[0], window)
        close(out.view(L, 1, d), ref, "bfloat16", scale=1.0)
        near = float((out[700].float().cpu() - vs[0][3, 0].float()).abs().max()) < 0.2
        assert near == sees, (window, near)


def test_attention_prefill_refuses_what_it_cannot_do():
    from libllm_b200.csrc import ops
    from libllm_b200.errors import UnsupportedError
    assert not ops.attention_prefill_supported(256, 64) and not ops.attention_prefill_supported(64, 16)
    assert not ops.attention_prefill_supported(40, 64)
    K, V, table, _, _ = paged_cache(1, [10], 1, 144, 64, "bfloat16", 35)
    q = rnd((10, 144), "bfloat16", 36)
    start, past = prefill_inputs([10], [10])
    with pytest.raises(UnsupportedError):
        ops.attention_prefill(q, torch.empty_like(q), K, V, start, past, table, 1, 10, 1, 1, 144, 64, None, 0.1)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_rope_on_a_part_of_the_channels(dtype):
    """Only the first 16 of 32 channels rotate (pairs (i, i + 8)); the rest pass through.  This is
    the general kernel; heads that rotate whole take the vectorised one."""
    from libllm_b200.csrc import ops
    n_heads, n_kv, d, rot, page = 2, 1, 32, 16, 8
    T = 5
    qkv = rnd((T, (n_heads + 2 * n_kv) * d), dtype, 40)
    q_out = torch.zeros((T, n_heads * d), dtype=DT[dtype], device=DEV)
    freqs = torch.tensor([0.5 ** i for i in range(rot // 2)], dtype=torch.float64)
    ang = torch.arange(16, dtype=torch.float64)[:, None] * freqs[None]
    table = torch.cat([ang.cos(), ang.sin()], 1).float().to(DEV)
    tok_seq = torch.zeros(T, dtype=torch.int32, device=DEV)
    tok_pos = torch.arange(3, 3 + T, dtype=torch.int32, device=DEV)
    pt = torch.tensor([[2, 0, 1, 3]], dtype=torch.int32, device=DEV)
    K = torch.zeros((4, n_kv, page, d), dtype=DT[dtype], device=DEV)
    V = torch.zeros_like(K)
    ops.rope_cache_write(qkv, q_out, n_heads, n_kv, d, table, tok_seq, tok_pos, pt, K, V, page)
    x = qkv.cpu().view(T, n_heads + 2 * n_kv, d)
    want = x[:, :n_heads].clone().double()
    want[..., :rot] = P.rope_rotate(x[:, :n_heads, :rot], tok_pos.cpu().double(), freqs)
    close(q_out.cpu().view(T, n_heads, d), want, dtype)
    kwant = x[:, n_heads:n_heads + n_kv].clone().double()
    kwant[..., :rot] = P.rope_rotate(x[:, n_heads:n_heads + n_kv, :rot], tok_pos.cpu().double(), freqs)
    for t in range(T):
        p = 3 + t
        close(K[int(pt[0, p // page]), :, p % page], kwant[t], dtype)


TC_SHAPES = [(1, 128, 64), (8, 200, 80), (3, 331, 176), (16, 2048, 2048), (17, 130, 520), (64, 300, 128),
             (100, 256, 192), (300, 500, 72), (8, 3072, 2048), (2, 64, 8)]


@pytest.mark.parametrize("out_dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("M,N,K", TC_SHAPES)
def test_tensor_core_product(out_dtype, M, N, K):
    """Sizes that are no multiple of any tile (rows of W, tokens, K), one token, many tokens."""
    from libllm_b200.csrc import ops
    x = rnd((M, K), "bfloat16", 50)
    w = rnd((N, K), "bfloat16", 51, std=0.1)
    out = torch.full((M, N), float("nan"), dtype=DT[out_dtype], device=DEV)
    assert ops.gemm_tc_supported(x, w)
    ops.gemm_tc(x, w, out)
    ops.check_tc_status()
    close(out, P.linear(x.cpu(), w.cpu()), "bfloat16" if out_dtype == "bfloat16" else "float32",
          scale=None if out_dtype == "bfloat16" else 50 * float(P.linear(x.cpu(), w.cpu()).abs().max()))


@pytest.mark.parametrize("M,N,K,parts", [(8, 2048, 2048, 4), (5, 200, 8192, 8), (40, 130, 520, 2), (16, 2048, 8192, 8)])
def test_tensor_core_product_in_parts_of_k(M, N, K, parts):
    from libllm_b200.csrc import ops
    x = rnd((M, K), "bfloat16", 52)
    w = rnd((N, K), "bfloat16", 53, std=0.1)
    out = torch.full((parts, M, N), float("nan"), dtype=torch.float32, device=DEV)
    ops.gemm_tc(x, w, out)
    ops.check_tc_status()
    ref = P.linear(x.cpu(), w.cpu())
    close(out.sum(0), ref, "float32", scale=50 * float(ref.abs().max()))
    assert 1 <= ops.gemm_tc_suggest_parts(M, N, K) <= 8


# one part, several and more than the registers for eight; a width for a block of each size, one for four pieces to a thread and one
# without 16-byte rows; few rows and prompt rows
@pytest.mark.parametrize("hidden", [1000, 1030, 2048, 4096, 4100])
@pytest.mark.parametrize("parts", [1, 2, 6, 12])
def test_what_a_scaled_addition_rounds(hidden, parts):
    """resid + (sum + bias) * scale to the bit: the product rounded, then the sum; both at once for several parts of rows of up to 4,096."""
    from ctypes import c_float, c_int, c_longlong, c_void_p
    from libllm_b200.csrc import ops
    P_, I_ = c_void_p, c_int
    for rows in (5, 1030):
        g = torch.Generator().manual_seed(hidden + parts)
        x, d = torch.randn(rows, hidden, generator=g), torch.randn(parts, rows, hidden, generator=g)
        s, b, w = (torch.randn(hidden, generator=g) for _ in range(3))
        t = d[0].clone()
        for p in range(1, parts):
            t = t + d[p]
        t = t + b
        joined = parts > 1 and hidden % 4 == 0 and hidden <= 4096
        want = (x.double() + t.double() * s.double()).float() if joined else x + t * s      # 48 bits of a product are exact in 64
        X, D, S, B, W = (v.to(DEV) for v in (x, d, s, b, w))
        out = torch.empty_like(X)
        ops._call("elementwise", "llm_add_rmsnorm_scaled", [P_, P_, I_, I_, c_longlong, P_, c_float, P_, I_, P_, I_, I_, P_, P_, P_],
                  X.data_ptr(), D.data_ptr(), 0, parts, rows * hidden, W.data_ptr(), 1e-5, out.data_ptr(), 0, None, rows, hidden,
                  S.data_ptr(), B.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert torch.equal(X.cpu(), want)


# widths at and beside a lane's pieces, the row count at which the prompt kernel takes over and one that leaves a CTA's last warps idle
@pytest.mark.parametrize("hidden", [516, 1024, 1028, 2048, 2052, 3072, 4092, 4096])
@pytest.mark.parametrize("parts,scaled", [(0, False), (1, False), (1, True)])
def test_norm_of_prompt_rows_has_the_bits_of_a_row_alone(hidden, parts, scaled):
    from ctypes import c_float, c_int, c_longlong, c_void_p
    from libllm_b200.csrc import ops
    rows = 1027
    x, w = rnd((rows, hidden), "float32", 94), rnd((hidden,), "float32", 95)
    delta = rnd((rows, hidden), "float32", 96) if parts else None
    cs, cb = (rnd((hidden,), "float32", 97), rnd((hidden,), "float32", 98)) if scaled else (None, None)
    got, one = torch.empty((rows, hidden), dtype=torch.bfloat16, device=DEV), torch.empty((3, hidden), dtype=torch.bfloat16, device=DEV)
    a, b = x.clone(), x[[0, 517, 1026]].contiguous()
    P_, I_ = c_void_p, c_int
    call = lambda r, d, o: ops._call(  # noqa: E731
        "elementwise", "llm_add_rmsnorm_scaled", [P_, P_, I_, I_, c_longlong, P_, c_float, P_, I_, P_, I_, I_, P_, P_, P_],
        r.data_ptr(), d.data_ptr() if d is not None else None, 0, parts, r.numel(), w.data_ptr(), 1e-5, o.data_ptr(), 1, None, r.shape[0], hidden,
        cs.data_ptr() if scaled else None, cb.data_ptr() if scaled else None, torch.cuda.current_stream().cuda_stream)
    call(a, delta, got)
    call(b, delta[[0, 517, 1026]].contiguous() if parts else None, one)
    assert torch.equal(a[[0, 517, 1026]], b) and torch.equal(got[[0, 517, 1026]], one)
    v = x.double() + (0 if not parts else (delta.double() + cb.double()) * cs.double() if scaled else delta.double())
    ref = v / (v * v).mean(-1, keepdim=True).add(1e-5).sqrt() * w.double()
    assert bool(((got.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-6).all())


def test_32_bit_product_of_more_rows_than_one_launch_takes():
    from libllm_b200.csrc import ops
    M = 65535 * 32 + 40
    x, w = rnd((M, 4), "float32", 64), rnd((3, 4), "float32", 65)
    out = torch.full((M, 3), float("nan"), device=DEV)
    ops.gemm_plain(x, w, out)
    ref = x.double() @ w.double().T
    assert float((out.double() - ref).abs().max()) < 8 * 2 ** -24 * float((x.double().abs() @ w.double().abs().T).max())     # 4 products, 8 roundings at most


# one part with work and eight, parts that end inside a block, widths beside the tiles; 4-byte rows take the general kernel
@pytest.mark.parametrize("K,N", [(4, 1), (36, 15), (252, 16), (260, 17), (1028, 130), (2048, 64), (97, 33)])
def test_32_bit_product_rows_do_not_depend_on_the_batch(K, N):
    """Every number of rows at which another kernel takes over gives a row the same bits, and rounding alone lies between
    them and 64 bits: each part adds at most K / 8 + 32 products one behind the other."""
    from libllm_b200.csrc import ops
    a = rnd((130, K), "float32", 91)
    w = rnd((N, K), "float32", 92)
    bias = rnd((N,), "float32", 93)
    rows = {}
    for M in (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 130):
        out = torch.full((M, N), float("nan"), dtype=torch.float32, device=DEV)
        ops.gemm_plain(a[:M], w, out, bias)
        rows[M] = out
    ref = a.double() @ w.double().T + bias.double()
    bound = (K / 8 + 40) * 2 ** -24 * (a.abs().double() @ w.abs().double().T + bias.abs().double()) if K % 4 == 0 else K * 2 ** -24 * (a.abs().double() @ w.abs().double().T + 1)
    assert bool(((rows[130].double() - ref).abs() <= bound).all())
    for M, out in rows.items():
        assert torch.equal(out, rows[130][:M]), M


# widths and numbers of rows that whole models have, ragged ones beside them
@pytest.mark.parametrize("K,N", [(1024, 256), (1028, 257), (1060, 300), (2048, 2048), (2052, 9600), (8192, 384)])
def test_32_bit_product_of_large_matrices(K, N):
    """A row has the same bits in every call, from rows with gaps between them too, and the error against 64 bits is that of 32-bit additions."""
    from libllm_b200.csrc import ops
    a = rnd((300, K + 8), "float32", 97)[:, :K]
    w = rnd((N, K + 4), "float32", 98)[:, :K]
    bias = rnd((N,), "float32", 99)
    full = torch.full((300, N + 3), float("nan"), device=DEV)
    ops.gemm_plain(a, w, full[:, :N], bias)
    assert bool(torch.isnan(full[:, N:]).all())
    full = full[:, :N]
    ref = a.double() @ w.double().T + bias.double()
    bound = (K / 8 + 40) * 2 ** -24 * (a.abs().double() @ w.abs().double().T + bias.abs().double())     # a part's chain of K / 8 and the parts'
    assert bool(((full.double() - ref).abs() <= bound).all())
    whole, wide = a.contiguous(), w.contiguous()
    for M in (1, 2, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129):
        out = torch.full((M, N), float("nan"), device=DEV)
        ops.gemm_plain(whole[:M], wide, out, bias)
        assert torch.equal(out, full[:M]), M
    # operands of one sign: sums in 16 chains of K / 16 and 11 additions to join them, each addition off by 2^-23 / sqrt(12) of what it has so far at most (2-norm),
    # a quarter above that for the share of small magnitudes
    out = torch.empty((300, N), device=DEV)
    ops.gemm_plain(whole.abs(), wide.abs(), out)
    ref = whole.abs().double() @ wide.abs().double().T
    assert float((out.double() - ref).norm() / ref.norm()) <= 1.25 * math.sqrt(K / 16 / 3 / 16 + 11 / 3) * 2 ** -23 / math.sqrt(12)
    # a single product each is rounded once: nothing of the operands is left out
    one = torch.zeros((64, K), device=DEV)
    at = torch.arange(64, device=DEV) * (K // 64)
    for value in (torch.ones(64, device=DEV), whole[:64, 0]):
        one[torch.arange(64), at] = value
        ops.gemm_plain(one, wide, out[:64])
        assert torch.equal(out[:64], value[:, None] * wide[:, at].T)
    # nor of values near the end of the type's range, down to where a product has fewer bits itself
    for power in (-100, -126):
        small = (whole[:64].double() * 2.0 ** power).float()
        ops.gemm_plain(small, wide, out[:64])
        ref = small.double() @ wide.double().T
        bound = (K / 8 + 40) * 2 ** -24 * (small.abs().double() @ wide.abs().double().T) + K * 2.0 ** -149
        assert bool(((out[:64].double() - ref).abs() <= bound).all()), power


def test_32_bit_product_of_large_matrices_with_values_that_are_not_finite():
    from libllm_b200.csrc import ops
    K, N = 2048, 512
    for M in (3, 40, 130):
        a, w = rnd((M, K), "float32", 101), rnd((N, K), "float32", 102)
        a[0, 5] = math.inf
        a[1, 700] = -math.inf
        a[2, 2047] = math.nan
        w[7, 5] = 0.0                                  # infinity times nought
        w[300, 9] = 3e38
        a[M - 1, 9] = 2.0 if M > 3 else a[M - 1, 9]    # a product beyond the type's range
        out = torch.empty((M, N), device=DEV)
        ops.gemm_plain(a, w, out)
        ref = a.double() @ w.double().T
        want = torch.where(ref.abs() > 3.4028235e38, torch.copysign(torch.full_like(ref, math.inf), ref), ref)
        assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(torch.isinf(out), torch.isinf(want))
        assert torch.equal(out[torch.isinf(out)].double(), want[torch.isinf(want)])
        ok = torch.isfinite(want)
        bound = (K / 8 + 40) * 2 ** -24 * (a.abs().double() @ w.abs().double().T)
        assert bool(((out.double() - want).abs()[ok] <= bound[ok]).all())


# widths of whole groups of 16 (gate and up rows in turns) and others; rows at the tiles' edges
@pytest.mark.parametrize("M,I,K", [(1, 64, 64), (5, 173, 80), (8, 8192, 2048), (40, 300, 256), (200, 128, 136), (257, 391, 200),
                                   (1000, 1024, 512), (1, 16, 8), (16, 48, 136), (17, 80, 72), (33, 208, 200), (64, 1040, 64), (65, 48, 64),
                                   (512, 4752, 8), (640, 3216, 72), (1025, 1904, 200),        # two SMs to a tile, ragged on both sides
                                   (2000, 5136, 456), (1280, 8208, 1096)])      # ... every pair's ring and both accumulators used again
def test_tensor_core_product_with_swiglu(M, I, K):
    from libllm_b200.csrc import ops
    x = rnd((M, K), "bfloat16", 54)
    w = rnd((2 * I, K), "bfloat16", 55, std=0.1)
    out = torch.full((M, I), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.gemm_tc(x, w, out, swiglu=True)
    ops.check_tc_status()
    gu = P.linear(x.cpu(), w.cpu())
    close(out, P.swiglu(gu[:, :I], gu[:, I:]), "bfloat16")


# tiles of 32 rows (up to 37 tiles of 128, parts counted; 32 tokens) and of 64 (up to 74, 48 tokens), the edges of a tile and of a stage of several blocks of K
@pytest.mark.parametrize("M,N,K,parts", [(1, 4736, 8, 1), (16, 4737, 328, 1), (17, 31, 264, 1), (32, 9472, 128, 1), (33, 97, 1096, 1), (48, 4700, 520, 1), (49, 300, 136, 1),
                                         (5, 2050, 1992, 2), (20, 1100, 2048, 5), (40, 1000, 1000, 4), (2, 9473, 192, 1)])
def test_tensor_core_product_in_tiles_of_fewer_rows(M, N, K, parts):
    """A row's sum is the same whatever the tile: the bits of the same rows in a matrix whose tiles have 128."""
    from libllm_b200.csrc import ops
    x = rnd((M, K), "bfloat16", 190)
    w = rnd((N, K), "bfloat16", 191, std=0.1)
    out = torch.full((parts, M, N), float("nan"), device=DEV) if parts > 1 else torch.full((M, N), float("nan"), device=DEV)
    ops.gemm_tc(x, w, out)
    wide = torch.cat([w, torch.zeros((19200 - N, K), dtype=torch.bfloat16, device=DEV)])       # 150 tiles of 128
    ref = torch.full((parts, M, 19200), float("nan"), device=DEV) if parts > 1 else torch.full((M, 19200), float("nan"), device=DEV)
    ops.gemm_tc(x, wide, ref)
    ops.check_tc_status()
    assert torch.equal(out, ref[..., :N])


def test_tensor_core_product_rows_do_not_depend_on_the_batch():
    """A token's row is the same alone and among 200 others: each token is its own column of the tile."""
    from libllm_b200.csrc import ops
    x = rnd((200, 256), "bfloat16", 56)
    w = rnd((384, 256), "bfloat16", 57, std=0.1)
    full = torch.empty((200, 384), dtype=torch.float32, device=DEV)
    ops.gemm_tc(x, w, full)
    for r in (0, 17, 199):
        one = torch.empty((1, 384), dtype=torch.float32, device=DEV)
        ops.gemm_tc(x[r:r + 1].contiguous(), w, one)
        assert torch.equal(one[0], full[r])
    ops.check_tc_status()


@pytest.mark.parametrize("n_heads,n_kv,d,window", [(4, 2, 16, None), (3, 1, 32, None), (32, 8, 64, None), (8, 1, 128, None),
                                                     (8, 8, 64, None), (6, 2, 128, 100), (10, 2, 48, None)])
# up to 16 splits are joined through a cluster's shared memory, more through scratch in global memory;
# chunk 0: each length cut into 5 runs
@pytest.mark.parametrize("chunk,n_splits", [(64, 16), (64, 18), (192, 6), (1024, 1), (0, 5)])
def test_attention_decode_fused(n_heads, n_kv, d, window, chunk, n_splits):
    """Rotation, cache append, attention and the joining of splits in one launch: the outputs
    against the plain rotation + attention, the cache rows it must have written, and a second
    launch one position later (the counters must have come back to zero)."""
    from libllm_b200.csrc import ops
    from helpers import rotary_frequencies
    page = 64
    lens = [1, 70, 333, 1000, 64, 65]        # cached tokens, the new one included
    B = len(lens)
    K, V, table_pt, ks, vs = paged_cache(B, [l + 1 for l in lens], n_kv, d, page, "bfloat16", 60)
    freqs = torch.tensor(rotary_frequencies(d, 10000.0, None), dtype=torch.float64)
    ang = torch.arange(1100, dtype=torch.float64)[:, None] * freqs[None]
    table = torch.cat([ang.cos(), ang.sin()], 1).float().to(DEV)
    counters = torch.zeros(B * n_kv, dtype=torch.int32, device=DEV)
    for step in range(2):
        pos = [l - 1 + step for l in lens]
        gen = torch.Generator().manual_seed(61 + step)
        if step == 0:
            qkv = torch.randn((B, (n_heads + 2 * n_kv) * d), generator=gen).to(DEV)
            qkv_in = qkv
        else:       # the stacked product in three parts over K, which the kernel adds in order
            qkv_in = torch.randn((3, B, (n_heads + 2 * n_kv) * d), generator=gen).to(DEV)
            qkv = (qkv_in[0] + qkv_in[1]) + qkv_in[2]
        out = torch.full((B, n_heads * d), float("nan"), dtype=torch.bfloat16, device=DEV)
        ws_o = torch.full((B * n_heads * n_splits * d,), float("nan"), device=DEV)
        ws_ml = torch.full((B * n_heads * n_splits * 2,), float("nan"), device=DEV)
        tok_pos = torch.tensor(pos, dtype=torch.int32, device=DEV)
        assert ops.attention_decode_tc_supported(d, page, n_heads // n_kv)
        ops.attention_decode_tc(qkv_in, out, table, K, V, tok_pos, table_pt, n_heads, n_kv, d, page, chunk, n_splits, window,
                                1 / math.sqrt(d), True, ws_o, ws_ml, counters, max_len=1100)
        assert int(counters.abs().sum()) == 0
        x = qkv.cpu().view(B, n_heads + 2 * n_kv, d)
        for b in range(B):
            p = torch.tensor([pos[b]], dtype=torch.float64)
            q = P.rope_rotate(x[b:b + 1, :n_heads], p, freqs).to(torch.bfloat16)
            k_new = P.rope_rotate(x[b:b + 1, n_heads:n_heads + n_kv], p, freqs).to(torch.bfloat16)
            v_new = x[b:b + 1, n_heads + n_kv:].to(torch.bfloat16)
            # the plain side's cache: the rows before the new token as they were, then the new one
            ks[b][pos[b]] = k_new[0]
            vs[b][pos[b]] = v_new[0]
            pg = int(table_pt[b, pos[b] // page])
            assert torch.equal(K[pg, :, pos[b] % page].cpu(), k_new[0]) or \
                float((K[pg, :, pos[b] % page].cpu().float() - k_new[0].float()).abs().max()) <= 2 ** -7 * float(k_new.abs().max())
            assert torch.equal(V[pg, :, pos[b] % page].cpu(), v_new[0])
            ref = P.attention_scores_softmax_values(q, ks[b][:pos[b] + 1], vs[b][:pos[b] + 1], window)
            # bfloat16 rounds relative to the value: a sequence of one or two keys returns values of up to 4
            close(out[b].view(1, n_heads, d), ref, "bfloat16", scale=max(1.0, float(ref.abs().max())))


# last rows that share a warp with rows beyond the sequence (length no multiple of 32), in the first tile and in later ones
@pytest.mark.parametrize("form", [1, 2])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("window,sink", [(None, 0), (100, 3)])
def test_prompt_attention_does_not_hang_on_old_pages(d, form, window, sink):
    """A sequence's bits are the same whatever its last page held before, also where the rows that share a warp with its last ones
    have far larger queries."""
    from libllm_b200.csrc import ops
    if form == 2 and sink:
        pytest.skip("kept first positions are the first form's")
    page, H, G, lens = 64, 4, 2, [16, 80, 200, 335]
    for n in lens:
        K, V, table, _, _ = paged_cache(2, [n, 90], G, d, page, "bfloat16", 171)
        q = rnd((n + 90, H * d), "bfloat16", 172)
        q[n:] *= 30
        start, past = prefill_inputs([n, 90], [n, 90])
        results = []
        for factor in (0.0, 30.0):
            last = int(table[0, (n - 1) // page])
            K[last, :, (n - 1) % page + 1:] = rnd((G, page - 1 - (n - 1) % page, d), "bfloat16", 174) * factor
            V[last, :, (n - 1) % page + 1:] = rnd((G, page - 1 - (n - 1) % page, d), "bfloat16", 175) * factor
            out = torch.empty((n + 90, H * d), dtype=torch.bfloat16, device=DEV)
            ops.attention_prefill_tc(q, out, K, V, start, past, table, 2, max(n, 90), H, G, d, page, window, 1 / math.sqrt(d), form, sink=sink)
            ops.check_tc_status()
            results.append(out[:n].cpu())
        assert torch.equal(results[0], results[1]), n


@pytest.mark.parametrize("n_heads,n_kv,d,window", [(32, 8, 64, None), (3, 1, 64, None), (8, 2, 128, None), (2, 2, 64, 64),
                                                     (6, 3, 128, 130), (4, 1, 64, 37)])
@pytest.mark.parametrize("form", [1, 2])
def test_attention_prefill_on_tcgen05(n_heads, n_kv, d, window, form):
    """The tcgen05 kernel on the cases of the mma.sync one: whole prompts, the end of a prompt behind
    cached tokens, tile edges (127, 128, 129 rows), single tokens, windows."""
    from libllm_b200.csrc import ops
    page = 64
    lens = [1, 70, 333, 200, 128, 129, 127, 300]
    q_lens = [1, 70, 5, 150, 128, 129, 1, 300]
    B = len(lens)
    K, V, table, ks, vs = paged_cache(B, lens, n_kv, d, page, "bfloat16", 71)
    T = sum(q_lens)
    q = rnd((T, n_heads * d), "bfloat16", 72)
    out = torch.full((T, n_heads * d), float("nan"), dtype=torch.bfloat16, device=DEV)
    start, past = prefill_inputs(lens, q_lens)
    assert ops.attention_prefill_tc_supported(d, page)
    ops.attention_prefill_tc(q, out, K, V, start, past, table, B, max(q_lens), n_heads, n_kv, d, page, window,
                             1 / math.sqrt(d), form)
    ops.check_tc_status()
    o = 0
    for s, n in enumerate(q_lens):
        ref = P.attention_scores_softmax_values(q[o:o + n].cpu().view(n, n_heads, d), ks[s], vs[s], window)
        close(out[o:o + n].view(n, n_heads, d), ref, "bfloat16", scale=max(1.0, float(ref.abs().max())))
        o += n


@pytest.mark.parametrize("form", [1, 2])
def test_attention_prefill_on_tcgen05_finds_a_far_key_and_respects_the_window_edge(form):
    from libllm_b200.csrc import ops
    d, page, L = 64, 64, 900
    K, V, table, ks, vs = paged_cache(1, [L], 1, d, page, "bfloat16", 73)
    q = rnd((L, d), "bfloat16", 74)
    k3 = (q[700].float().cpu() * 3.0).to(torch.bfloat16)
    K[int(table[0, 0]), 0, 3] = k3.to(DEV)
    ks[0][3, 0] = k3
    start, past = prefill_inputs([L], [L])
    for window, sees in ((None, True), (697, False), (698, True)):
        out = torch.empty((L, d), dtype=torch.bfloat16, device=DEV)
        ops.attention_prefill_tc(q, out, K, V, start, past, table, 1, L, 1, 1, d, page, window, 1 / math.sqrt(d), form)
        ops.check_tc_status()
        ref = P.attention_scores_softmax_values(q.cpu().view(L, 1, d), ks[0], vs[0], window)
        close(out.view(L, 1, d), ref, "bfloat16", scale=max(1.0, float(ref.abs().max())))
        near = float((out[700].float().cpu() - vs[0][3, 0].float()).abs().max()) < 0.2
        assert near == sees, (window, near)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("step_nats", [6.5, 2.0, -6.5])
@pytest.mark.parametrize("form", [1, 2])
def test_attention_prefill_on_tcgen05_when_the_maximum_moves_from_tile_to_tile(d, step_nats, form):
    """The kernel moves a row's exponent reference only when a tile's maximum exceeds it by 2^8, and
    then rescales the output row in tensor memory.  Random scores settle the reference in the first
    tile; here every 64 keys the scores step up by 6.5 nats (the reference moves in every tile and
    earlier tiles all but vanish), by 2 nats (it lags behind the maximum, moving every third tile or
    so, and the probabilities in between exceed 1), or down (it never moves after the first tile)."""
    from libllm_b200.csrc import ops
    page, L, n_heads, n_kv = 64, 700, 2, 1
    K, V, table, ks, vs = paged_cache(1, [L], n_kv, d, page, "bfloat16", 75)
    q = rnd((L, n_heads * d), "bfloat16", 76, 0.3)
    q.view(L, n_heads, d)[:, :, 0] = math.sqrt(d)              # channel 0 alone gives key j's score k[j, 0]
    k = ks[0][:, 0].float() * 0.3
    k[:, 0] = step_nats * (torch.arange(L) // 64).float()
    ks[0][:, 0] = k.to(torch.bfloat16)
    for lp in range((L + page - 1) // page):
        n = min(page, L - lp * page)
        K[int(table[0, lp]), 0, :n] = ks[0][lp * page:lp * page + n, 0].to(DEV)
    start, past = prefill_inputs([L], [L])
    out = torch.full((L, n_heads * d), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.attention_prefill_tc(q, out, K, V, start, past, table, 1, L, n_heads, n_kv, d, page, None, 1 / math.sqrt(d), form)
    ops.check_tc_status()
    ref = P.attention_scores_softmax_values(q.cpu().view(L, n_heads, d), ks[0], vs[0], None)
    close(out.view(L, n_heads, d), ref, "bfloat16", scale=max(1.0, float(ref.abs().max())))


@pytest.mark.parametrize("d,n_heads,n_kv", [(64, 32, 8), (128, 8, 2)])
@pytest.mark.parametrize("form", [1, 2])
def test_attention_prefill_on_tcgen05_with_a_prompt_of_2048_tokens(d, n_heads, n_kv, form):
    """A prompt as long as the benchmark's: 16 query tiles a head and up to 32 key tiles a CTA, so the
    rings of key/value stages and the two score buffers go round many times, with queries that lie
    strided in the stacked q|k|v rows as the engine has them.  Every 97th row is checked against
    the plain attention."""
    from libllm_b200.csrc import ops
    page, L = 64, 2048
    K, V, table, ks, vs = paged_cache(1, [L], n_kv, d, page, "bfloat16", 81)
    qkv = rnd((L, (n_heads + 2 * n_kv) * d), "bfloat16", 82)
    q = qkv[:, :n_heads * d]
    start, past = prefill_inputs([L], [L])
    out = torch.full((L, n_heads * d), float("nan"), dtype=torch.bfloat16, device=DEV)
    for _ in range(3):          # the same launch again: a race shows in some runs only
        ops.attention_prefill_tc(q, out, K, V, start, past, table, 1, L, n_heads, n_kv, d, page, None, 1 / math.sqrt(d), form)
        ops.check_tc_status()
        assert bool(torch.isfinite(out.float()).all())
        rows = list(range(0, L, 97)) + [L - 1]
        qs = q[rows].cpu().view(len(rows), n_heads, d)
        for i, r in enumerate(rows):
            ref = P.attention_scores_softmax_values(qs[i:i + 1], ks[0][:r + 1], vs[0][:r + 1], None)
            close(out[r].view(1, n_heads, d), ref, "bfloat16", scale=max(1.0, float(ref.abs().max())))


def test_copy_words_between_pinned_host_memory_and_the_device():
    """The small copies inside a single-token step's graph are kernels that read and write pinned
    host memory directly: both directions, an odd count, and a refusal of pageable memory."""
    from libllm_b200.csrc import ops
    from libllm_b200.errors import ExtensionError
    n = 2353
    host = torch.arange(n, dtype=torch.int32).pin_memory()
    dev = torch.full((n + 7,), -1, dtype=torch.int32, device=DEV)
    ops.copy_words(host, dev, n)
    torch.cuda.synchronize()
    assert torch.equal(dev[:n].cpu(), host) and bool((dev[n:] == -1).all())
    back = torch.zeros(n, dtype=torch.int32).pin_memory()
    ops.copy_words(dev * 3, back, n)
    torch.cuda.synchronize()
    assert torch.equal(back, host * 3)
    with pytest.raises(ExtensionError):
        ops.copy_words(torch.zeros(4, dtype=torch.int32), dev, 4)


# ---------------------------------------------------------------- a chain of products and norms in one launch
def _chain_case(T, Kq, H, inter, V, parts_o, parts_d, seed, repeats=3):
    from libllm_b200.csrc import ops
    eps = 3e-5
    x0 = rnd((T, Kq), "bfloat16", seed)
    wo = rnd((H, Kq), "bfloat16", seed + 1, Kq ** -0.5)
    wgu = rnd((2 * inter, H), "bfloat16", seed + 2, H ** -0.5)
    wd = rnd((H, inter), "bfloat16", seed + 3, inter ** -0.5)
    wh = rnd((V, H), "bfloat16", seed + 4, H ** -0.5)
    n1 = (1 + 0.1 * rnd((H,), "float32", seed + 5))
    n2 = (1 + 0.1 * rnd((H,), "float32", seed + 6))
    resid0 = rnd((T, H), "float32", seed + 7)
    rows = torch.tensor([T - 1, 0, T // 2][:min(3, T)], dtype=torch.int32, device=DEV)
    W = rows.numel()

    # the plain computation, rounding to bfloat16 where the chain does
    def norm(v, w):
        return (v * w * torch.rsqrt((v * v).mean(-1, keepdim=True) + eps)).to(torch.bfloat16)
    o = x0.float() @ wo.float().T
    v1 = resid0 + o
    h1 = norm(v1, n1)
    gu = h1.float() @ wgu.float().T
    m = (torch.nn.functional.silu(gu[:, :inter]) * gu[:, inter:]).to(torch.bfloat16)
    d = m.float() @ wd.float().T
    v2 = v1 + d
    h2 = norm(v2[rows.long()], n2)
    logits_ref = h2.float() @ wh.float().T

    counters = torch.zeros(16, dtype=torch.int32, device=DEV)
    for _ in range(repeats):
        resid = resid0.clone()
        o_parts = torch.full((parts_o, T, H), float("nan"), dtype=torch.float32, device=DEV)
        h1_out = torch.empty((T, H), dtype=torch.bfloat16, device=DEV)
        m_out = torch.empty((T, inter), dtype=torch.bfloat16, device=DEV)
        d_parts = torch.full((parts_d, T, H), float("nan"), dtype=torch.float32, device=DEV)
        h2_out = torch.empty((W, H), dtype=torch.bfloat16, device=DEV)
        logits = torch.full((W, V), float("nan"), dtype=torch.float32, device=DEV)
        jobs = [
            ops.chain_product(x0, wo, o_parts),
            ops.chain_norm(resid, o_parts, n1, eps, h1_out, deps=(0, -1)),
            ops.chain_product(h1_out, wgu, m_out, swiglu=True, deps=(1, -1)),
            ops.chain_product(m_out, wd, d_parts, deps=(2, -1)),
            ops.chain_norm(resid, d_parts, n2, eps, h2_out, rows=rows, deps=(3, 1)),
            ops.chain_product(h2_out, wh, logits, deps=(4, -1)),
        ]
        ops.gemm_chain(jobs, counters)
        torch.cuda.synchronize()
        ops.check_tc_status()
        assert int(counters.abs().sum()) == 0, "the chain left its counters non-zero"
        close(resid, v1, "bfloat16")
        close(h1_out.float(), h1.float(), "bfloat16")
        close(m_out.float(), m.float(), "bfloat16")
        close(h2_out.float(), h2.float(), "bfloat16")
        close(logits, logits_ref, "bfloat16")


@pytest.mark.parametrize("T,Kq,H,inter,V,parts_o,parts_d", [
    (5, 136, 200, 328, 1000, 2, 3),          # sizes that are no power of two, few tiles
    (16, 512, 1024, 2816, 20000, 4, 8),      # several tiles per CTA and job
    (23, 264, 520, 1096, 3001, 1, 2),        # 32-token shape, one part
    (40, 512, 1024, 1536, 9000, 2, 4),       # 64-token shape
    (1, 2048, 2048, 8192, 32000, 8, 8),      # the engine's widths at batch 1
])
def test_gemm_chain_layer(T, Kq, H, inter, V, parts_o, parts_d):
    _chain_case(T, Kq, H, inter, V, parts_o, parts_d, seed=11)


def test_gemm_chain_refuses():
    from libllm_b200.csrc import ops
    from libllm_b200.errors import UnsupportedError
    counters = torch.zeros(16, dtype=torch.int32, device=DEV)
    x = rnd((65, 64), "bfloat16", 1)
    w = rnd((128, 64), "bfloat16", 2)
    out = torch.empty((65, 128), dtype=torch.float32, device=DEV)
    with pytest.raises(UnsupportedError):
        ops.gemm_chain([ops.chain_product(x, w, out)], counters)          # more tokens than a chain takes
    x = rnd((4, 64), "bfloat16", 1)
    out = torch.empty((4, 128), dtype=torch.float32, device=DEV)
    with pytest.raises(UnsupportedError):
        ops.gemm_chain([ops.chain_product(x, w, out, deps=(0, -1))], counters)   # depends on itself
    with pytest.raises(UnsupportedError):
        ops.gemm_chain([ops.chain_product(x, w, out)] * 9, counters)      # more jobs than one launch holds
