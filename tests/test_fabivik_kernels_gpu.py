"""Each mechanism of the Fabivik design alone on the GPU, against the plain oracle's function for it."""
import math

import fabivik_helpers as H
import pytest
import torch

from oracle import fabivik_oracle as F

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16]
LIMIT = {torch.float32: 2e-5, torch.bfloat16: 0.04}
SCHEDULES = {
    "whole": [[(0, 150)], [(1, 70)], [(2, 1)]],
    "portions": [[(0, n)] for n in (2, 62, 2, 3, 1, 31, 33, 2, 1, 13)] + [[(1, 64)], [(1, 6)], [(2, 1)]],
    "tokens": [[(0, 1)]] * 150 + [[(1, 1)]] * 70 + [[(2, 1)]],
    "batch": [[(0, 64), (1, 2)], [(1, 3), (2, 1), (0, 1)], [(0, 1), (1, 1)], [(1, 20), (0, 2)], [(0, 60)], [(1, 1), (0, 2)], [(0, 20), (1, 43)]],
}


def close(got, want, dtype, factor=1.0):
    """Every row within the limit; in 16 bits a row in which large terms cancel may be off by a few times its share."""
    want = want.float()
    e = (got.float().cpu() - want).square().mean(-1).sqrt() / want.square().mean().sqrt()
    limit = LIMIT[dtype] * factor
    if dtype == torch.float32:
        return float(e.max()) < limit
    return float(e.max()) < 4 * limit and float((e > limit).float().sum()) <= 0.02 * e.numel()


def bf(t):
    return t.to(torch.bfloat16).float()


def rows(n, width, seed):
    return bf(torch.randn(n, width, generator=torch.Generator().manual_seed(seed)))


def one_layer(layer, dtype, width=96, eps=1e-5, seed=0, **kw):
    cfg = H.config([layer] if isinstance(layer, dict) else layer, width=width, eps=eps)
    w = H.weights(cfg, seed=seed)
    model, ctx, _ = H.build(cfg, w, dtype, **kw)
    return cfg, w, {k: v.double() for k, v in w.items()}, model, ctx


MIXERS = {
    "wkv": (H.wkv(mlp=None), H.wkv(heads=2, dim=64, rank=16, mlp=None), H.wkv(heads=1, dim=12, rank=5, mlp=None),
            H.wkv(heads=2, dim=128, rank=40, mlp=None), H.wkv(heads=1, dim=256, rank=8, mlp=None)),
    "delta": (H.delta(mlp=None), H.delta(heads=2, kv_heads=2, dim=64, vdim=64, conv=2, mlp=None),
              H.delta(heads=4, kv_heads=1, dim=128, vdim=72, conv=6, mlp=None), H.delta(heads=3, kv_heads=1, dim=20, vdim=11, conv=1, mlp=None),
              H.delta(heads=1, kv_heads=1, dim=256, vdim=300, conv=8, mlp=None)),
}


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("kind,which", [(k, i) for k in MIXERS for i in range(5)])
def test_recurrent_mixers(kind, which, dtype):
    """Whole prompts, portions, single tokens and unequal batches give the same rows; slots are used again all the time."""
    layer = MIXERS[kind][which]
    cfg, _, w, model, ctx = one_layer(layer, dtype)
    hs = [rows(n, 96, 5 + i) for i, n in enumerate((150, 70, 1))]
    fn = F.wkv if kind == "wkv" else F.gated_delta
    want = [fn(h.double(), w, "l0.mix", layer["mixer"], 1e-5) for h in hs]
    for name, schedule in SCHEDULES.items():
        got = H.run_mixer(model, ctx, 0, hs, schedule)
        assert all(close(g, x, dtype) for g, x in zip(got, want)), name
    assert len(ctx._free_state_slots) == ctx.num_state_slots


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,dim", [(2, 64), (3, 36), (1, 128)])
def test_wkv_rows_that_end_inside_a_block(heads, dim, dtype):
    """Blocks of four tokens, prepared 32 tokens at a time for long rows and 16 for short ones: rows that end before, at and behind both, in one step and
    continued in another one."""
    layer = H.wkv(heads=heads, dim=dim, rank=8, mlp=None)
    _, _, w, model, ctx = one_layer(layer, dtype)
    hs = [rows(n, 96, 15 + i) for i, n in enumerate((193, 66, 131, 4))]
    want = [F.wkv(h.double(), w, "l0.mix", layer["mixer"], 1e-5) for h in hs]
    for schedule in ([[(0, 193), (1, 66), (2, 131)], [(3, 4)]], [[(0, 17), (1, 1), (2, 3), (3, 4)], [(0, 176), (1, 65), (2, 128)]]):
        got = H.run_mixer(model, ctx, 0, hs, schedule)
        assert all(close(g, x, dtype) for g, x in zip(got, want)), schedule


class WkvCase:
    """Inputs of the wkv scan alone, with a state in front of every row (slots 0 to ``most`` - 1; row i writes slot ``most`` + i)."""

    def __init__(self, heads, dim, tokens, most, dtype, seed):
        g = torch.Generator(device="cuda").manual_seed(seed)

        def r(*shape):
            return torch.randn(*shape, generator=g, device="cuda")

        n = heads * dim
        self.heads, self.dim, self.n, self.most, self.dtype = heads, dim, n, most, dtype
        self.proj, self.z, self.state0 = r(tokens, 3 * n).to(dtype), r(1, tokens, n), r(2 * most, heads, dim, dim)
        self.bias, self.bonus, self.norm = (r(n).to(dtype) for _ in range(3))

    def scan(self, lens):
        """Rows of ``lens`` tokens from the first token on: (o [tokens][n] in 32 bits, the rows' states)."""
        from megatron_mixtera_b200 import _lib, ops

        T, rows_, state = sum(lens), len(lens), self.state0.clone()
        cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
        rd = torch.arange(rows_, dtype=torch.int32, device="cuda")
        wr, o, z = rd + self.most, torch.zeros(T, self.n, device="cuda"), self.z[:, :T].contiguous()
        a = _lib.RecurrenceArgs()
        a.kind, a.heads, a.kv_heads, a.dim, a.vdim, a.num_tokens, a.num_rows, a.norm_per_head = 0, self.heads, self.heads, self.dim, self.dim, T, rows_, 1
        a.proj, a.proj_ld, a.off_r, a.off_k, a.off_v = self.proj.data_ptr(), 3 * self.n, 0, self.n, 2 * self.n
        a.decay_bias, a.bonus, a.norm_weight, a.z, a.z_splits = self.bias.data_ptr(), self.bonus.data_ptr(), self.norm.data_ptr(), z.data_ptr(), 1
        a.state, a.state_in, a.state_out, a.state_slots, a.cu_tokens = state.data_ptr(), rd.data_ptr(), wr.data_ptr(), 2 * self.most, cu.data_ptr()
        a.o_f32, a.dtype, a.eps = o.data_ptr(), ops.dtype_code(self.dtype), 1e-5
        ops.struct_kernel("recurrence_scan", a, state)
        return o, state[self.most: self.most + rows_]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,dim", [(2, 64), (1, 128), (2, 20)])
@pytest.mark.parametrize("at", [3, 38, 129, 0])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_wkv_scan_looks_at_no_later_token(dtype, heads, dim, at, value):
    """A token that is no number (the fourth, third and second of a block, and the first) changes no bit of the tokens before it, nor of other rows: long rows
    and short ones."""
    for lens in ([131, 150, 3], [5] * 26 + [1] + [150] + [3] * 20):
        c = WkvCase(heads, dim, sum(lens), len(lens), dtype, 20)
        o, new = c.scan(lens)
        row = lens.index(150)
        t, end = sum(lens[:row]) + at, sum(lens[: row + 1])
        c.proj[t] = value
        o2, new2 = c.scan(lens)
        assert torch.equal(o2[:t], o[:t]) and torch.equal(o2[end:], o[end:]) and bool(o2[t].isnan().any())
        assert torch.equal(new2[:row], new[:row]) and torch.equal(new2[row + 1:], new[row + 1:])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("dim", [64, 40, 128])
def test_wkv_scan_of_a_row_in_any_company(dim, dtype):
    """A row alone, among enough rows of its length for two CTAs an SM, and beside many short rows.  Four lanes a column sum in one order, so the first two agree in
    every bit; short rows' eight lanes split a head's channels further, so the third agrees within a few roundings of 32-bit sums.  States have one order."""
    heads, n = 16, 67
    many = 8 * torch.cuda.get_device_properties(0).multi_processor_count // heads + 3
    c = WkvCase(heads, dim, many * n, many, dtype, 21)
    found = [c.scan(lens) for lens in ([n], [n] * many, [n] + [2] * 40)]
    (o, s), (o2, s2), (o3, s3) = ((o[:n], s[0]) for o, s in found)
    assert torch.equal(o, o2) and torch.equal(s, s2) and torch.equal(s, s3)
    assert float((o - o3).abs().max()) < 2.0 ** -24 * 16 * float(o.abs().max())
    assert bool(found[1][0].isfinite().all()) and bool(found[1][0][-n:].abs().max() > 0)


@pytest.mark.parametrize("heads,dim,lens", [(8, 64, [401]), (4, 128, [401]), (8, 64, [30, 31, 33, 29]), (4, 128, [30, 31, 33, 29])])
def test_wkv_states_are_rounded_no_more_than_a_token_at_a_time(heads, dim, lens):
    """Against 64 bits, the states' error is no larger than that of S <- fma(w, S, k v) for every token in 32 bits with the same decays (which 64 bits restate: a
    product of 24-bit numbers is exact there)."""
    off = plain = 0.0
    for seed in (1, 2, 3):
        c = WkvCase(heads, dim, sum(lens), len(lens), torch.float32, seed)
        c.z = c.z * 0.5 - 2
        new, at = c.scan(lens)[1].double(), 0
        k, v = (c.proj[:, i * c.n: (i + 1) * c.n].double().view(-1, heads, dim) for i in (1, 2))
        w = torch.exp(-torch.exp(c.z[0].double() + c.bias.double())).view(-1, heads, dim)
        w32 = torch.exp(-torch.exp(c.z[0] + c.bias)).double().view(-1, heads, dim)
        for row, n in enumerate(lens):
            S = c.state0[row].double().transpose(1, 2)
            P = S
            for t in range(at, at + n):
                kv = k[t][:, :, None] * v[t][:, None, :]
                S, P = w[t][:, :, None] * S + kv, (w32[t][:, :, None] * P + kv.float().double()).float().double()
            off += float((new[row].transpose(1, 2) - S).square().sum())
            plain += float((P - S).square().sum())
            at += n
    assert off <= plain, math.sqrt(off / plain)


@pytest.mark.parametrize("kind", ["wkv", "delta", "memory"])
@pytest.mark.parametrize("dim", [64, 48, 128])
def test_recurrent_decode_shares_a_row_between_warps(kind, dim):
    """One, two or four warps for a (row, head), by how many there are: the states are the same bits whichever takes a row, outputs up to the order of a head
    norm's sum (bf16: one rounding apart)."""
    from megatron_mixtera_b200 import _lib, ops

    heads, most, rank, splits = 16, 90, 24, 3
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(11)

    def r(*shape, scale=1.0):
        return torch.randn(*shape, generator=g, device="cuda") * scale

    def b(*shape, scale=1.0):
        return r(*shape, scale=scale).bfloat16()

    n, kv = heads * dim, heads // 2
    channels = 2 * kv * dim + n
    width = {"wkv": 4 * n, "memory": 4 * n, "delta": channels + n + 2 * heads}[kind]
    x = dict(proj=b(most, width), norm=b(n), state0=r(2 * most, heads, dim + (kind == "memory"), dim, scale=0.3), top0=r(2 * most, heads), bias=b(max(n, 2 * heads)),
             z=r(splits, most, 2 * heads), lora=b(most, rank), w2=b(n, rank, scale=rank ** -0.5), bonus=b(n), rate=b(heads), filter=b(4, channels, scale=0.4),
             conv0=b(2 * most, 3, channels))
    found = {}
    for rows_ in (most, max(2, 5 * sms // heads), 3):
        state, top, conv = x["state0"].clone(), x["top0"].clone(), x["conv0"].clone()
        at = torch.arange(rows_, dtype=torch.int32, device="cuda")
        rd, wr = at, at + most
        out = torch.zeros(rows_, n, dtype=torch.bfloat16, device="cuda")
        z = x["z"][:, :rows_].contiguous()
        a = _lib.RecurrenceArgs()
        a.kind = {"wkv": 0, "delta": 1, "memory": 2}[kind]
        a.heads, a.kv_heads, a.dim, a.vdim, a.num_tokens, a.num_rows, a.norm_per_head = heads, kv if kind == "delta" else heads, dim, dim, rows_, rows_, int(kind != "delta")
        a.proj, a.proj_ld, a.decay_bias, a.norm_weight, a.out = x["proj"].data_ptr(), width, x["bias"].data_ptr(), x["norm"].data_ptr(), out.data_ptr()
        a.off_r, a.off_k, a.off_v, a.off_g = 0, n, 2 * n, 3 * n
        if kind == "wkv":
            a.lora, a.rank, a.w2, a.bonus = x["lora"].data_ptr(), rank, x["w2"].data_ptr(), x["bonus"].data_ptr()
        elif kind == "memory":
            a.z, a.z_splits, a.z_ld, a.top, a.gate_cap, a.out_scale = z.data_ptr(), splits, 2 * heads, top.data_ptr(), 15.0, 1.0
        else:
            a.off_g, a.off_b, a.off_a = channels, channels + n, channels + n + heads
            a.decay_rate, a.conv_filter, a.conv_state, a.taps = x["rate"].data_ptr(), x["filter"].data_ptr(), conv.data_ptr(), 4
        a.state, a.state_in, a.state_out, a.state_slots = state.data_ptr(), rd.data_ptr(), wr.data_ptr(), 2 * most
        a.dtype, a.unit_eps, a.eps = ops.dtype_code(torch.bfloat16), 1e-6, 1e-5
        ops.struct_kernel("recurrence_decode", a, state)
        found[rows_] = (out, state[most: most + rows_], top[most: most + rows_], conv[most: most + rows_])
        assert torch.equal(state[:most], x["state0"][:most]) and torch.equal(state[most + rows_:], x["state0"][most + rows_:])
        assert bool(out.float().isfinite().all()) and float(out.float().abs().max()) > 0
    sizes = sorted(found)
    for few, many in zip(sizes, sizes[1:]):
        a, b_ = found[few], found[many]
        assert all(torch.equal(u, v[:few]) for u, v in zip(a[1:], b_[1:]))
        d = (a[0].float() - b_[0][:few].float()).abs()
        assert bool((d <= 2.0 ** -7 * a[0].float().abs() + 1e-6).all())


@pytest.mark.parametrize("kind", list(MIXERS))
def test_recurrent_state_after_a_portion(kind):
    """The state itself, and that a padding row or another request's slot is left alone."""
    layer = MIXERS[kind][0]
    cfg, _, w, model, ctx = one_layer(layer, torch.float32)
    h = rows(37, 96, 1)
    H.run_mixer(model, ctx, 0, [torch.cat([h, h])], [[(0, 37)]])
    side = int(ctx.request_state_side[0]) * ctx.num_state_slots + int(ctx.request_state_slots[0])
    buffers = ctx.recurrent_state(1)
    scan = F.wkv_scan(*F.wkv_inputs(h.double(), w, "l0.mix", layer["mixer"])[:4], w["l0.mix.u"]) if kind == "wkv" else \
        F.delta_scan(*F.delta_inputs(h.double(), w, "l0.mix", layer["mixer"]))
    S = scan[1].transpose(1, 2).float()
    assert float((buffers["state"][side].cpu() - S).abs().max() / S.abs().max()) < 1e-5
    if kind == "wkv":
        assert torch.equal(buffers["shift"][side].cpu(), h[-1])
    else:
        u = torch.cat([h.double() @ w["l0.mix." + k].T for k in "qkv"], dim=1)[-3:].float()
        assert float((buffers["conv"][side].cpu() - u).abs().max()) < 1e-4
    others = [i for i in range(2 * ctx.num_state_slots) if i != side]
    assert all(float(b[others].abs().max()) == 0.0 for b in buffers.values())


ATTENTIONS = [H.attention(mlp=None), H.attention(heads=3, kv_heads=3, dim=64, vdim=64, size=64, conv=2, v_mix=False, mlp=None),
              H.attention(heads=4, kv_heads=1, dim=128, vdim=128, size=100, v_mix=False, mlp=None),
              H.attention(heads=16, kv_heads=1, dim=72, vdim=16, size=5, conv=7, v_mix=False, mlp=None),
              H.attention(heads=5, kv_heads=1, dim=16, vdim=128, size=None, v_mix=False, mlp=None),
              H.attention(heads=2, kv_heads=2, dim=11, vdim=7, size=40, conv=1, v_mix=False, mlp=None),
              H.attention(heads=2, kv_heads=1, dim=200, vdim=256, size=90, conv=3, v_mix=False, mlp=None)]


def attention_oracle(h, w, layer, index=0, first=None):
    p, m = f"l{index}.mix", layer["mixer"]
    v = F.attention_values(h, w, p, m)
    if first is not None:
        v = (1 - w[p + ".vmix"]) * v + w[p + ".vmix"] * first
    return F.attention(h, w, p, m, 1e-5, v)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("which", range(len(ATTENTIONS)))
def test_attention(which, dtype):
    layer = ATTENTIONS[which]
    cfg, _, w, model, ctx = one_layer(layer, dtype)
    hs = [rows(n, 96, 5 + i) for i, n in enumerate((150, 70, 1))]
    want = [attention_oracle(h.double(), w, layer) for h in hs]
    for name, schedule in SCHEDULES.items():
        got = H.run_mixer(model, ctx, 0, hs, schedule)
        assert all(close(g, x, dtype) for g, x in zip(got, want)), name


@pytest.mark.parametrize("dtype", DTYPES)
def test_value_mixing(dtype):
    """The second mixing layer blends in the first one's values, with a layer that does not mix in between."""
    layers = [H.attention(mlp=None), H.attention(heads=4, kv_heads=4, dim=16, vdim=8, v_mix=False, mlp=None), H.attention(heads=2, mlp=None)]
    cfg, _, w, model, ctx = one_layer(layers, dtype)
    hs = [rows(n, 96, 5 + i) for i, n in enumerate((150, 70, 1))]
    want = [attention_oracle(h.double(), w, layers[2], 2, F.attention_values(h.double(), w, "l0.mix", layers[0]["mixer"])) for h in hs]
    plain = [attention_oracle(h.double(), w, layers[2], 2) for h in hs]
    for schedule in SCHEDULES.values():
        got = H.run_mixer(model, ctx, 2, hs, schedule)
        assert all(close(g, x, dtype) for g, x in zip(got, want))
    assert min(H.rel(a, b) for a, b in zip(plain, want)) > 0.1  # (mixing matters)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("size,key", [(96, 63), (96, 64), (64, 100), (65, 0), (1, 40), (2, 127), (None, 3), (130, 30)])
def test_one_key_stands_out(size, key, dtype):
    """One key that outweighs hundreds of others: queries just inside the window answer with its value, those just outside do not, in a
    prompt, in portions cut beside it, and decoded; every other pool slot a page holds is poisoned."""
    heads, dim, W, T = 2, 64, 96, 260
    layer = H.attention(heads=heads, kv_heads=1, dim=dim, vdim=32, size=size, v_mix=False, scale=2.0 / math.sqrt(dim), mlp=None)
    cfg = H.config([layer], width=W)
    w = H.weights(cfg, seed=1)
    g = torch.Generator().manual_seed(2)
    axis = torch.eye(W)
    asks, shown, s = axis[0] * 8, axis[1] * 8, torch.randn(dim, generator=g)
    small = 0.2 / math.sqrt(W)
    w["l0.mix.q"] = (torch.randn(heads * dim, W, generator=g) * small + torch.outer(s.repeat(heads), axis[0])).to(torch.bfloat16)
    w["l0.mix.k"] = (torch.randn(dim, W, generator=g) * small + torch.outer(s, axis[1])).to(torch.bfloat16)
    for k in ("q", "k"):  # positions stay sharp: the newest input outweighs the older ones
        w[f"l0.mix.{k}.conv"] *= 0.05
        w[f"l0.mix.{k}.conv"][:, -1] = 1.0
        w[f"l0.mix.{k}.norm"] = torch.full((dim,), 1.5).to(torch.bfloat16)
    h = rows(T, W, 9)
    h[:, :2] *= 0.02
    h[key] = bf(h[key] * 0.1 + shown)
    reach = size if size is not None else T
    places = sorted({p for p in (key, key + 1, key + 2, key + reach - 2, key + reach - 1, key + reach, key + reach + 1, key + 63, key + 64, T - 1)
                     if key < p < T})
    for p in places:
        h[p] = bf(h[p] * 0.1 + asks)
    wd = {k: v.double() for k, v in w.items()}
    want = attention_oracle(h.double(), wd, layer)
    value = F.attention_values(h.double(), wd, "l0.mix", layer["mixer"])[key, 0].repeat(heads) @ wd["l0.mix.o"].T
    for p in places:  # (what the case claims)
        near = float((want[p] - value).norm() / value.norm())
        assert (near < 0.2) == (p - key < reach), (p, near)
    model, ctx, _ = H.build(cfg, w, dtype)
    ctx.token_rows(1).fill_(30.0)  # nothing may be read from slots that hold no token of the request
    for schedule in ([T], [key + 1, 1, T - key - 2] if key + 2 < T else [T], [64] * 4 + [4], [key + 1] + [1] * (T - key - 1), [2] * (T // 2)):
        got = H.run_mixer(model, ctx, 0, [h], [[(0, n)] for n in schedule if n])[0]
        assert H.rel(got[places], want[places]) < 2 * LIMIT[dtype], schedule[:4]
        assert H.rel(got, want) < 2 * LIMIT[dtype], schedule[:4]
        ctx.token_rows(1).fill_(30.0)


def test_decode_attention_split_over_the_context():
    """Long rows: several splits of one window, rows shorter than a split beside them."""
    layer = H.attention(heads=4, kv_heads=2, dim=128, vdim=128, size=3000, v_mix=False, mlp=None)
    cfg, _, w, model, ctx = one_layer(layer, torch.bfloat16, max_cached_tokens=9000, max_sequence_length=4096, max_step_tokens=4096)
    from megatron_mixtera_b200.transformer.attention import choose_attention_splits

    assert choose_attention_splits(2, 2, 3064, 64) > 1
    hs = [rows(n, 96, 3 + i) for i, n in enumerate((3500, 40))]
    want = [attention_oracle(h.double(), w, layer) for h in hs]
    got = H.run_mixer(model, ctx, 0, hs, [[(0, 3490)], [(1, 30)]] + [[(0, 1), (1, 1)]] * 10)
    assert max(H.rel(g, x) for g, x in zip(got, want)) < LIMIT[torch.bfloat16]


def add_up(model, index, x, out):
    """out + the mixture of layer ``index`` for the rows ``x``."""
    from megatron_mixtera_b200 import ops

    with torch.inference_mode():
        hidden = out.cuda()
        ops.residual_norm(hidden, ops.PendingRows(experts=model.layers[index].moe(x.cuda().to(model.config.params_dtype))), [], [], eps=1.0)
    return hidden.cpu()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("tokens", [1, 7, 64, 300, 2000])
@pytest.mark.parametrize("case", range(6))
def test_experts(case, tokens, dtype):
    """Routing, the sort, the grouped products and the sum, over one to many tokens per expert and tile."""
    mlp = (H.experts(), H.experts(40, 5, 100, 2.0, 130), H.experts(3, 3, 64, 0.5, 64), H.experts(1, 1, 8, 1.0, None), H.experts(130, 1, 24, 3.0, 16),
           H.experts(9, 9, 70, 1.0, None))[case]
    width = 100 if case == 2 else 96
    cfg, _, w, model, _ = one_layer(H.wkv(mlp=mlp), dtype, width=width)
    x, base = rows(tokens, width, 4), torch.randn(tokens, width, generator=torch.Generator().manual_seed(8))
    got = add_up(model, 0, x, base)
    check = list(range(tokens)) if tokens <= 64 else list(range(0, tokens, tokens // 50))
    score = torch.sigmoid(x.double() @ w["l0.mlp.router"].T).sort(-1, descending=True).values
    top = mlp["router"]["top"]
    sure = [t for t in check if top == score.shape[1] or score[t, top - 1] - score[t, top] > 1e-6]
    want = base[sure].double() + F.mixture(x[sure].double(), w, "l0.mlp", mlp)
    assert H.rel(got[sure], want) < LIMIT[dtype] / 4
    from megatron_mixtera_b200 import ops

    assert int(ops.moe_counters(torch.device("cuda", 0), mlp["router"]["experts"])[: 4 * (mlp["router"]["experts"] + 1)].max()) == 0


@pytest.mark.parametrize("dtype", DTYPES)
def test_experts_all_tokens_at_one(dtype):
    """Every token chooses the same experts (the others get none), scores of zero and one included; limits bite on both sides."""
    mlp = H.experts(6, 2, 64, 0.3, 64, 0.2)
    cfg, w0, w, model, _ = one_layer(H.wkv(mlp=mlp), dtype)
    x = rows(500, 96, 4)
    x[:, 0] = 6.0
    for r in range(6):
        w0["l0.mlp.router"][r] *= 0.02
        w0["l0.mlp.router"][r, 0] = (-20.0, 3.0, -3.0, 20.0, -1.0, 0.0)[r]
    model.load_checkpoint(w0)
    w = {k: v.double() for k, v in w0.items()}
    got = add_up(model, 0, x, torch.zeros(500, 96))
    assert H.rel(got[::9], F.mixture(x[::9].double(), w, "l0.mlp", mlp)) < LIMIT[dtype] / 4


@pytest.mark.parametrize("tile", [32, 64, 128, 256])
def test_expert_tiles(tile, monkeypatch):
    from megatron_mixtera_b200.transformer.moe import MixtureOfExperts

    mlp = H.experts(5, 2, 72, 1.0, 200)
    cfg, _, w, model, _ = one_layer(H.wkv(mlp=mlp), torch.bfloat16, width=200)
    monkeypatch.setattr(MixtureOfExperts, "tile_tokens", staticmethod(lambda *a: tile))
    for tokens in (1, 31, 700):
        x = rows(tokens, 200, 4)
        got = add_up(model, 0, x, torch.zeros(tokens, 200))
        pick = list(range(0, tokens, max(1, tokens // 40)))
        assert H.rel(got[pick], F.mixture(x[pick].double(), w, "l0.mlp", mlp)) < LIMIT[torch.bfloat16] / 4


def test_expert_pairs_over_several_units_each():
    """More than two 256 x 256 tiles for each of the 74 pairs of SMs: tiles of the shared expert (four blocks of features, K 328 up and 456 down), then the
    experts' (two blocks, the last one partly filled, K 328 and 200), so that ring stages and accumulators are carried from one problem's tiles into the
    other's; one expert takes part in most choices, one in none, and the last tile of each holds a remainder."""
    experts, top, ff, shared_ff, width, tokens = 12, 3, 200, 456, 328, 7000
    mlp = H.experts(experts, top, ff, 1.0, shared_ff)
    cfg, w0, _, model, _ = one_layer(H.wkv(mlp=mlp), torch.bfloat16, width=width)
    w0["l0.mlp.router"][0, 0], w0["l0.mlp.router"][3, 0] = 0.5, -30.0
    model.load_checkpoint(w0)
    w = {k: v.double() for k, v in w0.items()}
    x = rows(tokens, width, 4)
    x[:, 0] = 6.0
    moe = model.layers[0].moe
    assert moe.tile_tokens(tokens * top, experts, False) == 256
    shared_tiles, least = -(-tokens // 256), tokens * top // 256  # (tiles of 256 rows; experts' remainders come on top)
    assert min(-(-2 * shared_ff // 256) * shared_tiles + 2 * least, -(-width // 256) * shared_tiles + 2 * least) > 2 * 74
    got = add_up(model, 0, x, torch.zeros(tokens, width))
    score = torch.sigmoid(x.double() @ w["l0.mlp.router"].T)
    chosen, order = torch.topk(score, top).indices, score.sort(-1, descending=True).values
    counts = chosen.flatten().bincount(minlength=experts)
    assert counts[3] == 0 and counts[0] > 2 * counts.double().mean()
    pick = torch.cat([(chosen == e).any(-1).nonzero()[-9:, 0] for e in range(experts)] + [torch.arange(0, tokens, 97)]).unique()  # (each expert's last tile)
    pick = [t for t in pick.tolist() if order[t, top - 1] - order[t, top] > 1e-6]
    assert H.rel(got[pick], F.mixture(x[pick].double(), w, "l0.mlp", mlp)) < LIMIT[torch.bfloat16] / 4
    assert not torch.isnan(got).any()


@pytest.mark.parametrize("width,top,splits", [(520, 3, 2), (1024, 4, 1), (1032, 1, 3), (2048, 5, 0), (4096, 8, 1), (4104, 2, 1), (8192, 4, 1)])
def test_residual_norm_of_many_rows(width, top, splits):
    """More rows than two for every SM: sums of the branch, expert rows (some missing), a gated shared expert's and the stream; two norms.  32-bit sums of bf16
    values in the stream (1e-5 of its scale), one rounding to bf16 in the norms (2^-8 of a value)."""
    from megatron_mixtera_b200 import _lib, ops

    g = torch.Generator(device="cuda").manual_seed(3)
    T, E = 2 * torch.cuda.get_device_properties(0).multi_processor_count + 5, 7

    def r(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    hidden, part, rows_, shared, gate = r(T, width), r(max(splits, 1), T, width), r(T * top, width).bfloat16(), r(T, width).bfloat16(), torch.rand(T, generator=g, device="cuda")
    expert = torch.randint(0, E, (T * top,), generator=g, device="cuda")
    counts = torch.bincount(expert, minlength=E)
    offsets = torch.cat([counts.new_zeros(1), counts.cumsum(0)])
    rank = torch.empty_like(expert)
    order = torch.argsort(expert, stable=True)
    rank[order] = torch.arange(T * top, device="cuda") - offsets[expert[order]]
    at = (offsets[expert] + rank).view(T, top)
    weight = torch.rand(T, top, generator=g, device="cuda")
    lost = torch.zeros(T * top, dtype=torch.bool, device="cuda")
    lost[::11] = True  # an expert that does not exist
    pairs = torch.stack([torch.where(lost, E + 3, expert), rank], dim=1).int().contiguous()
    gammas = [(0.3 * r(width)).bfloat16() for _ in range(2)]
    out = [torch.empty(T, width, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    want = hidden.double() + (part.double().sum(0) if splits else 0.0) + gate.double()[:, None] * shared.double()
    for j in range(top):
        want += (weight[:, j].double() * ~lost.view(T, top)[:, j])[:, None] * rows_[at[:, j]].double()
    a = _lib.ResidualNormArgs()
    a.hidden, a.rows, a.source_rows, a.width, a.eps, a.gain, a.out_scale, a.dtype = hidden.data_ptr(), T, T, width, 1e-3, 1.0, 0.5, ops.dtype_code(torch.bfloat16)
    if splits:
        a.partials, a.num_splits = part.data_ptr(), splits
    a.expert_rows, a.expert_row_count, a.pairs, a.offsets, offsets32 = rows_.data_ptr(), T * top, pairs.data_ptr(), 0, offsets.int()
    a.offsets, a.top, a.experts, a.pair_weight = offsets32.data_ptr(), top, E, weight.data_ptr()
    a.shared_rows, a.shared_gate = shared.data_ptr(), gate.data_ptr()
    for i in range(2):
        a.gamma[i], a.y[i] = gammas[i].data_ptr(), out[i].data_ptr()
    ops.struct_kernel("residual_norm", a, hidden)
    assert float((hidden.double() - want).abs().max()) < 1e-5 * float(want.abs().max())
    for o, gamma in zip(out, gammas):
        y = 0.5 * want / torch.sqrt((want * want).mean(-1, keepdim=True) + 1e-3) * (1.0 + gamma.double())
        assert bool(((o.double() - y).abs() <= 2.0 ** -8 * y.abs() + 1e-5).all())


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [32, 100, 101, 160, 1028, 2056, 4100, 8200])
def test_residual_stream_and_norms(width, dtype):
    """Embedding start, partial sums, two norms of one row, picked rows, the scale of the output."""
    from megatron_mixtera_b200 import ops

    g = torch.Generator().manual_seed(0)
    T, V = 9, 20
    table = bf(torch.randn(V, width, generator=g))
    gam = [bf(0.3 * torch.randn(width, generator=g)) for _ in range(2)]
    ids = torch.randint(0, V, (T,), generator=g)
    hidden = torch.empty((T, width), dtype=torch.float32, device="cuda")
    dev = [t.cuda().to(dtype) for t in (table, *gam)]
    out = [torch.empty((T, width), dtype=dtype, device="cuda") for _ in range(2)]
    ops.residual_norm(hidden, ops.PendingRows(table=dev[0], ids=ids.cuda(), table_scale=3.7), dev[1:], out, eps=1e-3)
    x = table[ids] * 3.7
    assert float((hidden.cpu() - x).abs().max()) < 1e-5
    tol = 1e-5 if dtype == torch.float32 else 2e-2
    for o, w in zip(out, gam):
        assert float((o.float().cpu() - F.layer_norm(x.double(), w.double(), 1e-3)).abs().max()) < tol
    K = 64
    a, b = bf(torch.randn(T, K, generator=g)), bf(torch.randn(width, K, generator=g))
    pick = torch.tensor([8, 0, 3])
    picked = torch.empty((3, width), dtype=dtype, device="cuda")
    pend = lambda: ops.PendingRows(partials=ops.linear_partials(a.cuda().to(dtype), b.cuda().to(dtype)))  # noqa: E731
    ops.residual_norm(hidden, pend(), dev[1:2], [picked], eps=1e-3, out_scale=0.5, row_index=pick.cuda())
    assert float((hidden.cpu() - x).abs().max()) < 1e-5  # (picked rows leave the stream as it is)
    y = x.double() + a.double() @ b.double().T
    assert float((picked.float().cpu() - 0.5 * F.layer_norm(y[pick], gam[0].double(), 1e-3)).abs().max()) < tol
    ops.residual_norm(hidden, pend(), [], [], eps=1.0)
    assert float((hidden.cpu() - y).abs().max()) < 1e-4


def test_wrong_arguments_are_refused():
    """The host checks turn impossible sizes into errors before anything is launched."""
    from megatron_mixtera_b200 import _lib, ops

    x = torch.zeros(8, device="cuda")
    for name, args in (("residual_norm", _lib.ResidualNormArgs()), ("conv_qkv", _lib.ConvArgs()), ("token_shift", _lib.ShiftArgs()),
                       ("recurrence_scan", _lib.RecurrenceArgs()), ("moe_up", _lib.MoeArgs())):
        with pytest.raises(ops.B200Error):
            ops.struct_kernel(name, args, x)
