"""The mechanisms Sobezen adds, each alone (a part built from its description, run through the host library's part
handle) against the plain implementation's function for it: the rotation table of neighbouring pairs with the
ramp between kept and slowed frequencies, attention whose values are its keys, latent attention with rows of its
own and with borrowed rows, the delta rule with a decay per key channel and its carried state, the clamped gated
unit, and a sublayer's scale per channel.  Attention is run with a score scale that makes one key stand out for
almost every query, wherever it lies (far back, next to a page border, the query's own position), so that a mask or
a page one position off shows; prompts, portions and single tokens share the calls."""
import math

import pytest
import torch

import plain_sobezen as P
import sobezen_helpers as S
from test_parts_gpu import PAGE, Step, act, part, summed

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DTYPES = ["float32", "bfloat16"]
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
# on |got - ref| / (|ref| + mean |ref|), element by element
TOL = {"float32": 3e-5, "bfloat16": 3e-2}


def bf(t):
    return t.to(torch.bfloat16).float()


def close(got, ref, dtype, what, roundings=1.0):
    assert got.shape == ref.shape, f"{what}: {tuple(got.shape)} vs {tuple(ref.shape)}"
    assert torch.isfinite(got.float()).all(), f"{what}: not finite"
    ref = ref.to(torch.float64)
    d = (got.to(torch.float64).cpu() - ref).abs()
    e = float((d / (ref.abs() + ref.abs().mean())).max())
    assert e < TOL[dtype] * roundings, f"{what}: error {e:.3e} ({dtype})"


def mixer_of(layers, i, dtype, seed, ranks=(6, 9), max_positions=1024):
    """Layer i's mixer of a model of `layers`, as the configuration's reader describes it, with weights of its own."""
    from libllm_b200 import _lib
    c = S.config(64, WIDTH, EPS, layers)
    spec = _lib.describe_model(c, dtype)["spec"]["layers"][i]["mixer"]
    w = {k: v for k, v in S.random_weights(c, seed, ranks).items() if k.startswith(f"l{i}.mix.")}
    m = part("mixer", spec, dtype, max_positions)
    m.load(w)
    return m, {k: v.double() for k, v in w.items()}, spec


WIDTH, EPS = 56, 1e-5


def run_in_portions(mixers, caches, x, portions, dtype, lens, state=None, slots=None):
    """Sequences of `lens` tokens of x (a list of [n, WIDTH]) brought in `portions` (a list of lists: new tokens per
    sequence and call, 0 = the sequence sits the call out) through every mixer of `mixers` in turn (they share the
    step; mixer j reads and writes caches[j]).  Returns per mixer and sequence the rows of the result."""
    done = [0] * len(lens)
    got = [[[] for _ in lens] for _ in mixers]
    pages = sum((n + PAGE - 1) // PAGE for n in lens) + 4
    for por in portions:
        seqs = [b for b in range(len(lens)) if por[b] > 0]
        step = Step([por[b] for b in seqs], [done[b] for b in seqs])
        # pages of a sequence stay its own from call to call: logical page j of sequence b is page (j * 5 + b * 2 + 1) % pages
        width = max((done[b] + por[b] + PAGE - 1) // PAGE for b in seqs)
        table = torch.tensor([[PAGE_OF[(b, j)] for j in range(width)] for b in seqs], dtype=torch.int32, device=DEV)
        if slots is not None:
            step.keep["seq_slot"].copy_(torch.tensor([slots[b] for b in seqs], dtype=torch.int32))
            step.json["slots"] = [slots[b] for b in seqs]
        xs = torch.cat([x[b][done[b]:done[b] + por[b]] for b in seqs]).to(DT[dtype]).to(DEV)
        for j, m in enumerate(mixers):
            call = dict(step=step.json, x=act(xs))
            if caches[j] is not None:
                k, v, writes = caches[j]
                call["cache"] = dict(k=k.data_ptr(), v=v.data_ptr() if v is not None else 0, n_pages=k.shape[0],
                                     page_table=table.data_ptr(), table_width=width, writes=writes)
            if state is not None:
                call["state"] = state
            out = summed(m.forward(call)["out"]).cpu()
            at = 0
            for b in seqs:
                got[j][b].append(out[at:at + por[b]])
                at += por[b]
        for b in seqs:
            done[b] += por[b]
    assert done == list(lens)
    return [[torch.cat(rows) for rows in per] for per in got]


# logical page j of sequence b -> a page of the store, scattered and never shared
PAGE_OF = {(b, j): 3 + b + 4 * j if j % 2 == 0 else 40 - b - 4 * j for b in range(4) for j in range(5)}
assert len(set(PAGE_OF.values())) == len(PAGE_OF) and min(PAGE_OF.values()) >= 0
N_PAGES = max(PAGE_OF.values()) + 1
LENS = [300, 66, 130]
# a prompt each; single tokens over the page border at 64 / 128 / 192 (the second sequence ends first); portions of
# two and three tokens; most of the rest of the first sequence in one portion; single tokens past 256 positions (where
# a token's keys are shared out over two runs); the last of it
PORTIONS = [[60, 63, 120]] + [[1, 1, 1]] * 3 + [[2, 0, 3], [1, 0, 1], [3, 0, 2], [1, 0, 1]] + [[200, 0, 0]] + [[1, 0, 0]] * 2 + [[28, 0, 0]]
assert [sum(p[b] for p in PORTIONS) for b in range(3)] == LENS


def sharp_inputs(seed, lens=LENS):
    g = torch.Generator().manual_seed(seed)
    return [bf(torch.randn(n, WIDTH, generator=g)) for n in lens]


def check_sharpness(shares, what):
    """The test means something only if most queries give most of their weight to one key, and those keys lie
    anywhere: many far back, some on either side of a page border, some the query's own position."""
    a = shares[0]                                       # [H, T, T]
    top, where = a.max(-1)
    T = a.shape[1]
    i = torch.arange(T)[None, :].expand_as(where)
    sharp = top > 0.6
    assert float(sharp.float().mean()) > 0.5, f"{what}: the scores are not sharp enough to show a misplaced key"
    far = (sharp & (i - where > 64)).sum()
    own = (sharp & (where == i) & (i > 0)).sum()
    edge = (sharp & ((where % PAGE == 0) | (where % PAGE == PAGE - 1)) & (i - where > 1)).sum()
    assert far > 20 and own > 3 and edge > 3, f"{what}: far {int(far)}, own {int(own)}, at a page's edge {int(edge)}"


# ---------------------------------------------------------------- the rotation's table
@pytest.mark.parametrize("rot", [S.rot(8, 5e4, S.Y1), S.rot(32, 1e6, S.Y2), S.rot(6, 2e3, S.Y3), S.rot(12, 500.0), S.rot(2, 1e4)])
def test_pair_table_holds_the_ramped_frequencies_and_the_magnitude(rot):
    """The position part of a latent layer: row p holds cos and sin of p * f_i, both times 0.1 ln(factor) + 1."""
    layers = [S.layer(S.latent(2, 8, rot["dims"], 8, 16, 8, base=rot["base"], scale=0.3,
                               scaling=tuple(rot["scaling"][k] for k in ("factor", "original", "fast", "slow")) if "scaling" in rot else None), None)]
    from libllm_b200 import _lib
    spec = _lib.describe_model(S.config(64, WIDTH, EPS, layers), "float32")["spec"]["layers"][0]["mixer"]["position"]
    assert spec["pairing"] == "interleaved"
    pos = part("position", spec, "float32", 300)
    pos.load({})
    table = pos.forward(dict(step=Step([1], [0]).json))["table"].torch().cpu().double()      # [positions, cosines | sines]
    n = rot["dims"]
    angle = torch.arange(300, dtype=torch.float64)[:, None] * P.pair_frequencies(rot)[None, :]
    m = P.table_magnitude(rot)
    assert table.shape == (300, n)
    assert float((table[:, :n // 2] - torch.cos(angle) * m).abs().max()) < 2e-5 * max(1.0, 300 * float(P.pair_frequencies(rot).max()))
    assert float((table[:, n // 2:] - torch.sin(angle) * m).abs().max()) < 2e-5 * max(1.0, 300 * float(P.pair_frequencies(rot).max()))
    if "scaling" in rot:
        assert abs(m - 1.0) > 0.05
        f_plain = P.pair_frequencies(dict(dims=n, base=rot["base"]))
        ratio = P.pair_frequencies(rot) / f_plain
        assert float(ratio.min()) < 0.99 and float(ratio.max()) <= 1.0        # some pair is slowed, none is sped up


# ---------------------------------------------------------------- latent attention
# heads, dim, rot_dim, vdim, kv_rank, q_rank, scale: sizes the tiled kernels take (five heads in a tile of 32 and
# values narrower than their tile; 34 heads over two tiles with a rotated part as wide as the rest) and sizes they
# do not (no 16-byte rows), which go the plain kernels' way
LATENT_SIZES = [(5, 24, 8, 40, 48, 20, 1.3), (34, 16, 16, 16, 32, 24, 2.0), (3, 6, 6, 10, 22, 14, 1.8)]


def latent_pair(sizes, dtype, seed):
    H, d, r, dv, R, Q, scale = sizes
    own = S.latent(H, d, r, dv, R, Q, base=3e3, scale=scale, scaling=S.Y1)
    lent = S.latent(H, d, r, dv, R, Q, base=3e3, scale=scale, scaling=S.Y1, kv_from=0)
    layers = [S.layer(own, None), S.layer(lent, None)]
    return layers, [mixer_of(layers, i, dtype, seed) for i in range(2)]


def plain_latent_pair(layers, weights, x, rounded):
    """Both layers over whole sequences: per layer and sequence the result, and the first layer's shares."""
    ref, shares = [[], []], []
    for xb in x:
        pos = torch.arange(xb.shape[0])
        h = xb.double()
        rows = P.latent_rows(weights[0], "l0.mix.", layers[0]["mixer"], h, pos, EPS)
        if rounded:
            rows = (bf(rows[0]).double(), bf(rows[1]).double())        # what a bfloat16 cache holds
        for i in range(2):
            sh = []
            ref[i].append(P.latent_attention(weights[i], f"l{i}.mix.", layers[i]["mixer"], h, pos, EPS, rows, sh))
            if i == 0:
                shares.append(sh)
    return ref, shares


@pytest.mark.parametrize("sizes", LATENT_SIZES)
@pytest.mark.parametrize("dtype", DTYPES)
def test_latent_attention_with_sharp_scores(sizes, dtype):
    """Prompts from the first token, single tokens across page borders and past 256 positions, portions of two and
    three tokens and a long one behind cached rows, for three sequences at once; the second mixer has no rows of
    its own and reads the first's."""
    layers, built = latent_pair(sizes, dtype, 11)
    x = sharp_inputs(5)
    ref, shares = plain_latent_pair(layers, [b[1] for b in built], x, dtype == "bfloat16")
    check_sharpness(shares[0], "latent attention")
    row = sizes[4] + sizes[2]
    k = torch.zeros(N_PAGES, PAGE, row, dtype=DT[dtype], device=DEV)
    got = run_in_portions([b[0] for b in built], [(k, None, True), (k, None, False)], x, PORTIONS, dtype, LENS)
    for i in range(2):
        for b in range(len(LENS)):
            close(got[i][b], ref[i][b], dtype, f"latent layer {i}, sequence {b}", roundings=6.0 if dtype == "bfloat16" else 4.0)


@pytest.mark.parametrize("sizes", LATENT_SIZES[:2])
def test_latent_prompt_and_token_by_token_are_one_function(sizes):
    """The two forms of the kernel (heads materialised for a prompt; all heads over the cached rows otherwise) agree:
    a prompt at once against the same tokens one at a time."""
    layers, built = latent_pair(sizes, "bfloat16", 12)
    x = sharp_inputs(6, [150])
    row = sizes[4] + sizes[2]
    results = []
    for portions in ([[150]], [[1]] * 150, [[2]] * 75):
        k = torch.zeros(N_PAGES, PAGE, row, dtype=torch.bfloat16, device=DEV)
        results.append(run_in_portions([b[0] for b in built], [(k, None, True), (k, None, False)], x, portions, "bfloat16", [150]))
    for other in results[1:]:
        for i in range(2):
            close(other[i][0], results[0][i][0].double(), "bfloat16", f"latent layer {i} in single tokens", roundings=4.0)


def test_latent_tokens_behind_cached_rows_are_the_same_alone_and_together():
    """Eighty tokens behind 220 cached ones, at once and one at a time: below 512 positions a token's keys are one run whatever else
    the step holds, so the results are the same bits."""
    layers, built = latent_pair(LATENT_SIZES[1], "bfloat16", 13)
    x = sharp_inputs(7, [300])
    row = LATENT_SIZES[1][4] + LATENT_SIZES[1][2]
    results = []
    for portions in ([[220], [80]], [[220]] + [[1]] * 80):
        k = torch.zeros(N_PAGES, PAGE, row, dtype=torch.bfloat16, device=DEV)
        results.append(run_in_portions([b[0] for b in built], [(k, None, True), (k, None, False)], x, portions, "bfloat16", [300]))
    for i in range(2):
        assert torch.equal(results[0][i][0], results[1][i][0]), f"latent layer {i}"


# runs at and beyond the eight whose values a thread of the join asks for together, some without keys; widths that leave threads idle and that
# take them all, output rows on 8 bytes and not
@pytest.mark.parametrize("R,rot,heads,row_gap", [(64, 16, 5, 0), (512, 32, 3, 2), (512, 64, 2, 0), (96, 8, 33, 4)])
@pytest.mark.parametrize("n_splits", [1, 7, 8, 9, 17, 40])
def test_latent_runs_are_joined(n_splits, R, rot, heads, row_gap):
    """All heads of two tokens over the cached rows, against the softmax in 64 bits; probabilities are rounded to bfloat16 in the kernel."""
    from ctypes import c_float, c_int, c_longlong, c_void_p
    from libllm_b200.csrc import ops
    g = torch.Generator().manual_seed(R + n_splits)
    lens, row = [1290, 700], R + rot
    pages = [(n + PAGE - 1) // PAGE for n in lens]
    order = torch.randperm(sum(pages), generator=g)
    table = torch.zeros(2, max(pages), dtype=torch.int32)
    cache = torch.zeros(sum(pages), PAGE, row)
    data, at = [], 0
    for b, n in enumerate(lens):
        rows = bf(torch.randn(n, row, generator=g))
        data.append(rows.double())
        for j in range(pages[b]):
            table[b, j] = order[at]
            part = rows[j * PAGE:(j + 1) * PAGE]
            cache[order[at], :len(part)] = part
            at += 1
    q = bf(torch.randn(2, heads * row, generator=g))
    out = torch.zeros(2, heads * R + row_gap, dtype=torch.bfloat16, device=DEV)
    ws = torch.full((2 * heads * n_splits * (R + 2),), float("nan"), device=DEV)
    i32 = dict(dtype=torch.int32, device=DEV)
    qd, cd, td, seq, pos = q.to(torch.bfloat16).to(DEV), cache.to(torch.bfloat16).to(DEV), table.to(DEV), torch.arange(2, **i32), torch.tensor(lens, **i32) - 1
    scale = 2.0 / row ** 0.5
    ops._call("latent_tc", "llm_latent_decode", [c_void_p, c_longlong, c_void_p, c_int] + [c_void_p] * 3 + [c_int] * 6 + [c_float, c_void_p, c_longlong,
              c_void_p, c_int, c_void_p], qd.data_ptr(), qd.stride(0), cd.data_ptr(), PAGE, seq.data_ptr(), pos.data_ptr(), td.data_ptr(), td.stride(0),
              2, heads, R, rot, n_splits, scale, out.data_ptr(), out.stride(0), ws.data_ptr(), 0, torch.cuda.current_stream().cuda_stream)
    for b in range(2):
        p = torch.softmax(q[b].double().view(heads, row) @ data[b].T * scale, -1)
        want, size = p @ data[b][:, :R], p @ data[b][:, :R].abs()
        got = out[b, :heads * R].double().cpu().view(heads, R)
        # a probability's rounding (2^-9) and the result's, of the terms' sizes; 32-bit sums and exponentials beside them are nothing
        assert bool(((got - want).abs() <= 2.2 * 2 ** -9 * (size + want.abs()) + 1e-6).all())
    assert float(out[:, heads * R:].abs().max() if row_gap else 0.0) == 0.0


# tokens at which another instantiation takes over, heads of one and of several fetches of w_uk, latents with an odd width
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,H,d,rot,R,dv", [(1, 2, 6, 2, 22, 10), (2, 3, 64, 32, 512, 64), (3, 1, 65, 0, 33, 7), (4, 2, 80, 4, 520, 9),
                                            (5, 2, 64, 8, 130, 64), (9, 1, 130, 6, 48, 24), (17, 2, 33, 2, 600, 5)])
def test_queries_take_in_the_keys_matrix_and_results_are_expanded(T, H, d, rot, R, dv, dtype):
    """latent_absorb and latent_expand against 64 bits: a sum of n products is off by at most n + 2 roundings of its terms'
    absolute sum, and a 16-bit result by one of its own."""
    from ctypes import c_int, c_longlong, c_void_p
    from libllm_b200.csrc import ops
    g = torch.Generator().manual_seed(T * R + d)
    row, dt = R + rot, DT[dtype]
    q = torch.randn(T, H * (d + rot), generator=g)
    w_uk, w_uv = (torch.randn(H * n, R, generator=g).to(dt) for n in (d, dv))
    table = torch.randn(9, max(rot, 1), generator=g)
    pos = torch.randint(0, 9, (T,), generator=g).int()
    out = torch.full((T, H * row), float("nan"), dtype=dt, device=DEV)
    dev = [t.to(DEV) for t in (q, w_uk, table, pos, w_uv)]
    stream = torch.cuda.current_stream().cuda_stream
    code = 0 if dtype == "float32" else 1
    ops._call("latent", "llm_latent_absorb",
              [c_int, c_void_p, c_longlong, c_void_p, c_void_p, c_longlong] + [c_int] * 5 + [c_void_p, c_int, c_int, c_void_p, c_void_p],
              code, dev[0].data_ptr(), q.shape[1], dev[1].data_ptr(), out.data_ptr(), H * row, T, H, d, rot, R, dev[2].data_ptr(), 9, 1,
              dev[3].data_ptr(), stream)
    got, q3 = out.cpu().double().view(T, H, row), q.double().view(T, H, d + rot)
    w3 = w_uk.double().view(H, d, R)
    result = 2 ** -8 if dtype == "bfloat16" else 0.0
    ref = torch.einsum("thi,hic->thc", q3[..., :d], w3)
    room = (d + 2) * 2 ** -24 * torch.einsum("thi,hic->thc", q3[..., :d].abs(), w3.abs()) + result * ref.abs()
    assert bool(((got[..., :R] - ref).abs() <= room).all())
    if rot:
        a, b = q3[..., d::2], q3[..., d + 1::2]
        c, s = (table[pos.long()].double()[:, None, i * rot // 2:(i + 1) * rot // 2] for i in range(2))
        for part_, want in ((got[..., R::2], a * c - b * s), (got[..., R + 1::2], b * c + a * s)):
            assert bool(((part_ - want).abs() <= 4 * 2 ** -24 * (a.abs() * c.abs().maximum(s.abs()) + b.abs() * c.abs().maximum(s.abs())) + result * want.abs()).all())
    x = torch.randn(T, H * R, generator=g).to(dt)
    y = torch.full((T, H * dv), float("nan"), dtype=dt, device=DEV)
    xd = x.to(DEV)
    ops._call("latent", "llm_latent_expand", [c_int, c_void_p, c_longlong, c_void_p, c_void_p, c_longlong] + [c_int] * 4 + [c_void_p],
              code, xd.data_ptr(), H * R, dev[4].data_ptr(), y.data_ptr(), H * dv, T, H, R, dv, stream)
    x3, v3 = x.double().view(T, H, R), w_uv.double().view(H, dv, R)
    ref = torch.einsum("thc,hjc->thj", x3, v3)
    room = (R / 32 + 8) * 2 ** -24 * torch.einsum("thc,hjc->thj", x3.abs(), v3.abs()) + result * ref.abs()
    assert bool(((y.cpu().double().view(T, H, dv) - ref).abs() <= room).all())


# ranks on either side of the sixteen values a thread holds, CTAs whose channels begin inside a head and end in another key head's
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,G,d,dv,ranks", [(6, 2, 50, 44, (16, 17)), (5, 5, 96, 64, (40, 3)), (8, 1, 64, 80, (15, 33))])
def test_channel_delta_with_ranks_and_heads_beside_a_threads_share(H, G, d, dv, ranks, dtype):
    """Prompts, portions and single tokens of the gated delta rule, state carried in slots out of order."""
    m, w, _ = mixer_of([S.layer(S.delta(H, G, d, dv, 3), None)], 0, dtype, 21, ranks)
    sizes = dict(heads=H, kv_heads=G, dim=d, vdim=dv)
    lens = [70, 9]
    x = sharp_inputs(22, lens)
    kept = {n["name"]: (torch.zeros([4, *n["shape"]], dtype=DT[n["dtype"]], device=DEV), n) for n in m.description["state"]}
    state = [dict(name=k, ptr=t.data_ptr(), shape=n["shape"], dtype=n["dtype"], n_slots=4) for k, (t, n) in kept.items()]
    got = run_in_portions([m], [None], x, [[33, 1], [1, 1], [35, 6], [1, 1]], dtype, lens, state=state, slots=[2, 0])
    for b in range(2):
        survives = []
        ref = P.channel_delta(w, "l0.mix.", sizes, x[b].double(), EPS, survives)
        # a head's norm divides by the head: rows where one all but cancels hang on the roundings of its 16-bit inputs
        clear = survives[0] > (0.0 if dtype == "float32" else 0.1 * float(survives[0].mean()))
        e = (got[0][b].double() - ref).norm(dim=-1) / ref.norm(dim=-1).mean()
        assert int(clear.sum()) > len(ref) // 2
        assert float(e[clear].max()) < (1e-4 if dtype == "float32" else 16 * 2 ** -8), (b, float(e[clear].max()))
