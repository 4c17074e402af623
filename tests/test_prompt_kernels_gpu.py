"""Kernels for many tokens (prompts) at the edges of their tiles: GEMMs of CTA pairs, attention over blocks of 256 query rows."""
import ctypes
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16 = torch.bfloat16


@pytest.fixture(scope="module")
def ops():
    from megatron_mixtera_b200 import build, ops as _ops

    build.build_torch_ops()
    yield _ops
    torch.cuda.synchronize()
    assert _ops.device_status() == 0, "a kernel abandoned a bounded wait"


def randn(*shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * scale).to(BF16)


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


# ---------------------------------------------------------------------------------------------------------------------
# GEMM: 256 x 256 tiles.  One bf16 rounding of an fp32 sum is 2^-9 / sqrt(3) = 1.1e-3 of a value, 1.7e-3 over a binade; 3e-3 is the limit of the
# other GEMM tests.
# ---------------------------------------------------------------------------------------------------------------------
SHAPES = [
    (257, 14336, 128),   # one token in the second token block
    (1000, 4868, 72),    # K of one block and a bit, N 4 past a tile
    (4097, 1128, 512),   # N inside the last tile's first half
    (2048, 2560, 1000),  # K no multiple of a block
    (5000, 1160, 64),    # a single K block
    (300, 16384, 192),
    (129, 18828, 136),   # one token block, half of it used
    # (the pairs take these; of the ones above, which the streaming kernel takes, its SwiGLU only)
    (257, 19204, 1352),  # one token in the second token block, N 4 past a tile, K of 21 blocks and a bit
    (4097, 2312, 1280),  # N inside the last tile's first half
    (129, 38532, 1288),  # one token block, half of it used
    (700, 6400, 5000),   # two waves: long K only
]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_pair_gemm_matches_the_fp32_product(ops, M, N, K):
    x, w, b = randn(M, K, seed=1), randn(N, K, seed=2, scale=K ** -0.5), randn(N, seed=3)
    ref = x.float() @ w.float().T
    assert rel(ops.gemm(x, w), ref) < 3e-3
    assert rel(ops.gemm(x, w, b), ref.to(BF16).float() + b.float()) < 3e-3
    assert rel(ops.linear(x, w, act="relu2"), torch.relu(ref).square()) < 3e-3
    parts = ops.gemm_splitk(x, w)
    got = parts.buf.view(torch.float32)[: parts.num_splits * M * N].view(parts.num_splits, M, N).sum(0)
    assert rel(got, x.double() @ w.double().T) < 1e-5  # fp32 sums of up to 1000 products
    assert ops.gemm_num_splits(None, M, N, K) == parts.num_splits
    wide = torch.zeros(M, N + 3, dtype=BF16, device="cuda")  # rows that no vector store can take
    ops.linear(x, w, out=wide[:, :N])
    assert torch.equal(wide[:, :N], ops.gemm(x, w)) and not wide[:, N:].any()


# Tiles are walked in groups of 16 token blocks, or of 8 where a token is more than 8 KB, every other group from the last features to the first: three groups of
# each kind, the last one partial, features that end inside a tile.
@pytest.mark.parametrize("M,N,K", [(4400, 1160, 4104), (8500, 1160, 1280)])
def test_pair_gemm_walks_groups_of_tiles_to_and_fro(ops, M, N, K):
    x, w = randn(M, K, seed=11), randn(N, K, seed=12, scale=K ** -0.5)
    y = torch.full((M, N), float("nan"), dtype=BF16, device="cuda")
    assert rel(ops.gemm(x, w, out=y), x.float() @ w.float().T) < 3e-3 and not bool(y.isnan().any())


@pytest.mark.parametrize("M,N,K", [(4400, 1160, 8320), (8500, 1160, 1152)])
def test_pair_gemm_mxfp8_walks_groups_of_tiles_to_and_fro(ops, M, N, K):
    from oracle import decode_oracle as O

    x, w = randn(M, K, seed=13), randn(N, K, seed=14)
    xd, wd = (O.dequantize_mxfp8(*O.quantize_mxfp8(t.cpu())).cuda() for t in (x, w))
    y = torch.full((M, N), float("nan"), dtype=BF16, device="cuda")
    assert rel(ops.gemm_mxfp8(ops.quantize_mxfp8(x), ops.quantize_mxfp8_weight(w), out=y), xd.float() @ wd.float().T) < 3e-3 and not bool(y.isnan().any())


@pytest.mark.parametrize("M,F,K", [(257, 7168, 256), (2048, 1280, 512), (1500, 3200, 72), (300, 9664, 1352)])
def test_pair_gemm_swiglu_equals_gemm_then_activation(ops, M, F, K):
    x, w = randn(M, K, seed=4), randn(2 * F, K, seed=5, scale=K ** -0.5)
    assert ops.gemm_swiglu_supported(M, 2 * F, K)
    got = ops.gemm_swiglu(x, ops.interleave_gate_up(w))
    assert torch.equal(got, ops.activation(ops.gemm(x, w), "swiglu"))


@pytest.mark.parametrize("M,N,K", [(257, 14336, 128), (1000, 4864, 384), (4097, 1152, 512), (2048, 2560 + 40, 1024), (257, 14592, 1152), (4097, 1128, 1024),
                                   (3000, 3328, 640)])  # (the pairs take the last four)
def test_pair_gemm_mxfp8_matches_the_dequantised_product(ops, M, N, K):
    from oracle import decode_oracle as O

    # scales that differ from row to row and block to block: a scale taken from another place shows
    def spread(rows, seed):
        s = torch.randint(-3, 4, (rows, K // 32), generator=torch.Generator().manual_seed(seed)).float().exp2().cuda()
        return (randn(rows, K, seed=seed).float() * s.repeat_interleave(32, 1)).to(BF16)

    x, w = spread(M, 6), spread(N, 7)
    xd, wd = (O.dequantize_mxfp8(*O.quantize_mxfp8(t.cpu())).cuda() for t in (x, w))
    ref = xd.double() @ wd.double().T
    xq, wq = ops.quantize_mxfp8(x), ops.quantize_mxfp8_weight(w)
    assert rel(ops.gemm_mxfp8(xq, wq), ref) < 3e-3
    parts = ops.gemm_splitk(xq, wq)
    got = parts.buf.view(torch.float32)[: parts.num_splits * M * N].view(parts.num_splits, M, N).sum(0)
    assert rel(got, ref) < 1e-5
    b = randn(N, seed=8)
    assert rel(ops.gemm_mxfp8(xq, wq, b), ref.to(BF16).double() + b.double()) < 3e-3


@pytest.mark.parametrize("M,F,K", [(257, 7168, 256), (1500, 2176, 384), (2048, 1280, 1024), (257, 7168, 1024), (1500, 2176, 1152), (1100, 2048, 1024)])
def test_pair_gemm_mxfp8_swiglu_equals_gemm_then_activation(ops, M, F, K):
    x, w = ops.quantize_mxfp8(randn(M, K, seed=9)), ops.quantize_mxfp8_weight(randn(2 * F, K, seed=10, scale=K ** -0.5))
    y = ops.gemm_mxfp8(x, w)
    assert torch.equal(ops.gemm_mxfp8_swiglu(x, w, quantize=False), ops.activation(y, "swiglu"))
    got, want = ops.gemm_mxfp8_swiglu(x, w), ops.activation_mxfp8(y, "swiglu")
    r, b = torch.arange(M)[:, None], torch.arange(F // 32)[None, :]
    at = ((r // 128) * (F // 128) * 512 + (b // 4) * 512 + (r % 32) * 16 + ((r % 128) // 32) * 4 + b % 4).reshape(-1).cuda()
    assert torch.equal(got.q, want.q) and torch.equal(got.sf[at], want.sf[at])


# ---------------------------------------------------------------------------------------------------------------------
# Attention over prompts: units of several requests in one CTA, portions behind a past, short last units, every option of the separate layouts,
# NaN in every pool row that no token wrote.  The output's bf16 rounding is 1.7e-3; the weights' hi + lo terms and fp32 sums add less than 1e-4.
# ---------------------------------------------------------------------------------------------------------------------
LENS, PAST = [700, 333, 1, 300, 900, 64], [0, 0, 300, 513, 64, 1]


@pytest.mark.parametrize("form,heads,groups,dim,vdim,chunk,options", [
    ("fused", 32, 8, 128, 128, 64, {}),
    ("fused", 16, 16, 64, 64, 256, {}),
    ("separate", 16, 8, 128, 128, 128, {"window": 200}),
    ("separate", 24, 8, 64, 128, 64, {}),
    ("separate", 16, 8, 128, 128, 64, {"window": 1}),
    ("extra", 16, 8, 96, 72, 64, {"window": 150, "keep": 5, "sinks": True}),
    ("extra", 16, 8, 128, 128, 256, {"window": 300, "cap": 5.0, "gates": "head"}),
    ("extra", 16, 8, 128, 128, 64, {"window": 300, "keep": 70, "bias": 100, "cap": 7.0, "sinks": True}),
    ("extra", 48, 8, 64, 64, 64, {"bias": 40}),
    ("extra", 16, 16, 128, 128, 64, {"sinks": True, "gates": "value"}),
    ("maps", 16, 8, 64, 128, 64, {}),
])
def test_prompt_attention_matches_the_plain_one(ops, form, heads, groups, dim, vdim, chunk, options):
    prompt_attention(ops, form, heads, groups, dim, vdim, chunk, options, LENS, PAST, 1)


# Lists of short and long requests: two kernels share them by groups of four units.  Groups of one, two and more requests, of two that see few or many
# tiles, padding behind the list; every value of the hint, whatever the list holds.
MIXED = [1] * 9 + [300, 5, 64, 64, 200, 700, 1, 33] + [16] * 5 + [2, 400, 1]
MIXED_PAST = [40, 700, 0, 1, 63, 64, 65, 130, 7] + [0, 900, 0, 0, 513, 1, 64, 3] + [0] * 5 + [600, 0, 250]


@pytest.mark.parametrize("mix", [0, 1, 2])
@pytest.mark.parametrize("form,heads,groups,dim,vdim,chunk,options", [
    ("fused", 32, 8, 128, 128, 64, {}),
    ("fused", 64, 16, 64, 64, 64, {}),
    ("separate", 16, 8, 128, 128, 128, {"window": 200}),
    ("extra", 16, 16, 128, 128, 64, {"window": 300, "keep": 70, "bias": 100, "cap": 7.0, "sinks": True}),
    ("maps", 16, 8, 64, 128, 64, {}),
])
def test_prompt_attention_of_mixed_lists(ops, form, heads, groups, dim, vdim, chunk, options, mix):
    prompt_attention(ops, form, heads, groups, dim, vdim, chunk, options, MIXED, MIXED_PAST, mix)


def prompt_attention(ops, form, heads, groups, dim, vdim, chunk, options, lens, past, mix):
    from megatron_mixtera_b200 import _lib

    o = {"window": 0, "keep": 0, "sinks": False, "cap": 0.0, "bias": 0, "gates": None, **options}
    maps, dev = 2 if form == "maps" else 1, "cuda"
    group, T, kv = heads // groups, sum(lens), [n + p for n, p in zip(lens, past)]
    blocks = [-(-n // chunk) for n in kv]
    order = torch.randperm(sum(blocks), generator=torch.Generator().manual_seed(1)).tolist()
    table = torch.zeros(len(kv), max(blocks), dtype=torch.int32)
    key_width = groups * maps * dim
    width = key_width + groups * vdim
    pool = torch.full((sum(blocks) + 1, chunk, width), float("nan"), dtype=BF16, device=dev)
    keys, values = [], []
    for r, n in enumerate(kv):
        k, v = randn(n, key_width, seed=100 + r), randn(n, groups * vdim, seed=200 + r)
        keys.append(k.view(n, groups, maps, dim)), values.append(v.view(n, groups, vdim))
        rows = torch.cat([k, v], dim=1)
        for b in range(blocks[r]):
            table[r, b] = order.pop()
            part = rows[b * chunk: (b + 1) * chunk]
            pool[int(table[r, b]), : len(part)] = part
    q = randn(T, groups, group, maps, dim, seed=3)
    lengths = torch.cat([torch.arange(p + 1, p + n + 1) for n, p in zip(lens, past)]).int().to(dev)
    unit, units, t = 64 // group, [], 0
    for r, n in enumerate(lens):
        units += [(r, t + a, min(unit, n - a), 0) for a in range(0, n, unit)]
        t += n
    units += [(0, 0, 0, 0)] * 3  # padding entries
    units, table = torch.tensor(units, dtype=torch.int32, device=dev), table.to(dev)
    assert -(-(-(-T // unit)) // 4) * groups * maps * 2 >= 148  # (fewer take the kernel for few units)
    out = torch.full((T, heads * vdim), float("nan"), dtype=BF16, device=dev)

    a = _lib.AttentionArgs()
    if form == "fused":
        qkv = torch.zeros(T, groups, group + 2, dim, dtype=BF16, device=dev)
        qkv[:, :, :group] = q[:, :, :, 0]
        pools = [pool[..., :key_width].contiguous(), pool[..., key_width:].contiguous()]
        a.qkv, a.k_cache, a.v_cache = qkv.data_ptr(), pools[0].data_ptr(), pools[1].data_ptr()
    else:
        a.qkv, a.k_cache, a.v_cache = q.data_ptr(), pool.data_ptr(), pool.data_ptr() + 2 * key_width
        a.separate, a.value_dim, a.pool_row_elems, a.window = (1 if form == "separate" else 2), vdim, width, o["window"]
    sinks = torch.randn(heads, generator=torch.Generator().manual_seed(4)).to(dev)
    bias = torch.randn(heads, max(o["bias"], 1), generator=torch.Generator().manual_seed(5)).to(dev)
    gates = randn(T, heads * (vdim if o["gates"] != "head" else 1), seed=6)
    work = torch.empty(T * 2 * heads * 129, device=dev)
    if a.separate == 2:
        a.out_scale, a.keep_first, a.softcap = 0.75, o["keep"], o["cap"]
        if o["sinks"]:
            a.sinks = sinks.data_ptr()
        if o["bias"]:
            a.distance_bias, a.bias_len = bias.data_ptr(), o["bias"]
        if o["gates"] or maps == 2:
            a.gate, a.gate_ld, a.value_gates = gates.data_ptr(), gates.shape[1], int(o["gates"] == "value")
    if maps == 2:
        a.maps, a.diff_scale, a.eps, a.workspace, a.workspace_bytes = 2, 0.7, 1e-5, work.data_ptr(), work.numel() * 4
        a.lambda_ = 0.4
    a.unit_mix = mix
    a.block_table, a.kv_seq_lengths, a.out = table.data_ptr(), lengths.data_ptr(), out.data_ptr()
    a.num_tokens, a.num_q_heads, a.num_kv_heads, a.head_dim, a.chunk_size = T, heads, groups, dim, chunk
    a.num_chunks, a.max_chunks_per_row, a.num_splits = pool.shape[0], table.shape[1], 1
    rc = _lib.load().b200_paged_prefill_attention(ctypes.byref(a), units.data_ptr(), len(units), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0 and ops.device_status() == 0

    def plain(qs, ks, vs, past, n):  # [n, heads, dim], [keys, groups, dim], [keys, groups, vdim]
        ks, vs = (x.double().repeat_interleave(group, 1) for x in (ks, vs))
        s = torch.einsum("qhd,khd->hqk", qs.double(), ks) * dim ** -0.5
        age = torch.arange(past, past + n, device=dev)[:, None] - torch.arange(past + n, device=dev)[None]
        seen = age >= 0
        if o["window"]:
            seen &= (age < o["window"]) | (torch.arange(past + n, device=dev) < o["keep"])
        if o["cap"]:
            s = o["cap"] * torch.tanh(s / o["cap"])
        if o["bias"]:
            s = s + bias.double()[:, age.clamp(0, o["bias"] - 1)]
        s = s.masked_fill(~seen, -math.inf)
        if o["sinks"]:
            s = torch.cat([s, sinks.double()[:, None, None].expand(-1, n, 1)], dim=-1)
        return torch.einsum("hqk,khv->qhv", torch.softmax(s, dim=-1)[..., : past + n], vs)

    want, t = [], 0
    for r, (n, p) in enumerate(zip(lens, past)):
        qs = q[t: t + n].reshape(n, heads, maps, dim)
        y = [plain(qs[:, :, m], keys[r][:, :, m], values[r], p, n) for m in range(maps)]
        y = y[0] if maps == 1 else y[0] - 0.4 * y[1]
        if maps == 2:
            y = y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5) * 0.7
        g = torch.sigmoid(gates[t: t + n].double())
        if maps == 2 or o["gates"] == "value":
            y = y * g.view(n, heads, vdim)
        elif o["gates"] == "head":
            y = y * g[:, :, None]
        want.append(y * (0.75 if a.separate == 2 else 1.0))
        t += n
    want = torch.cat(want).reshape(T, -1)
    assert not torch.isnan(out.float()).any()
    assert rel(out, want) < (4e-3 if maps == 2 else 2.5e-3)
    # one bf16 rounding is at most 2^-9 of a value; what the weights and sums add is small beside the outputs' scale
    off = (out.double() - want).abs() - 2 ** -8 * want.abs()
    assert float(off.max() / want.square().mean().sqrt()) < 1e-2


# ---------------------------------------------------------------------------------------------------------------------
# Latent attention of prompts on expanded keys: rows that start and that continue, windows, value and head gates, key sizes of one to three tiles of 64.
# ---------------------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dim,rot,vdim,window,gates,sinks", [
    (128, 64, 128, None, "head", False), (24, 16, 40, 33, "head", False), (64, 32, 64, 1, "head", True), (112, 8, 72, 150, "value", True),
    (72, 0, 128, None, "value", True), (128, 64, 128, 257, "head", False)])
def test_latent_prompts_match_the_plain_attention(ops, dim, rot, vdim, window, gates, sinks):
    latent_prompts(ops, dim, rot, vdim, window, gates, sinks, (dim + rot) ** -0.5)


@pytest.mark.parametrize("scale", [-0.1, 0.0])
@pytest.mark.parametrize("window", [None, 150])
def test_latent_prompts_with_a_scale_that_is_not_positive(ops, window, scale):
    latent_prompts(ops, 128, 64, 128, window, "head", False, scale)  # (scores would be masked with -inf in front of the scale)


def latent_prompts(ops, dim, rot, vdim, window, gates, sinks, scale):
    from megatron_mixtera_b200 import _lib

    heads, lens, past, dev = 40, [300, 1, 700, 257], [0, 40, 65, 0], "cuda"
    T, rows = sum(lens), len(lens)
    first = [0 if window is None else max(0, p - window + 1) for p in past]
    count = [n + p - f for n, p, f in zip(lens, past, first)]
    E, kv_pad = sum(count), 48
    width = -(-(kv_pad + rot) // 32) * 32
    kv = randn(E, heads * (dim + vdim), seed=1)
    key_rows = randn(E, width, seed=2)
    key_rows[:, kv_pad + rot:] = 0
    q, gate = randn(T, heads, dim + rot, seed=3), randn(T, heads * (vdim if gates == "value" else 1), seed=4)
    gate_at = heads * (dim + rot)
    proj = torch.zeros(T, gate_at + -(-gate.shape[1] // 8) * 8, dtype=BF16, device=dev)
    proj[:, :gate_at], proj[:, gate_at: gate_at + gate.shape[1]] = q.reshape(T, -1), gate
    q_rot = torch.zeros(T, heads, max(width - kv_pad, 8), dtype=BF16, device=dev)
    q_rot[..., :rot] = q[..., dim:]
    sink = torch.randn(heads, generator=torch.Generator().manual_seed(5)).to(dev)
    out = torch.full((T, heads * vdim), float("nan"), dtype=BF16, device=dev)

    def running(xs):
        return torch.tensor([0] + xs).cumsum(0).int().to(dev)

    cu_tokens, cu_keys, key_start = running(lens), running(count), torch.tensor(first, dtype=torch.int32, device=dev)
    a = _lib.LatentArgs()
    a.proj, a.proj_ld, a.gate_offset, a.value_gates = proj.data_ptr(), proj.shape[1], gate_at, int(gates == "value")
    a.q_full, a.q_stride, a.q_rot_at, a.out = q_rot.data_ptr(), q_rot.shape[2], 0, out.data_ptr()
    a.num_tokens, a.heads, a.dim, a.rot_dim, a.rot_dims, a.vdim = T, heads, dim, rot, rot, vdim
    a.kv_rank, a.kv_pad, a.row_width, a.window, a.scale = kv_pad, kv_pad, width, window or 0, scale
    a.dtype, a.max_positions, a.num_splits, a.chunk_size, a.num_chunks, a.pool = ops.dtype_code(BF16), 1, 1, 64, 1, key_rows.data_ptr()
    if sinks:
        a.sinks = sink.data_ptr()
    a.cu_tokens, a.cu_keys, a.key_start, a.key_rows, a.key_values = (t.data_ptr() for t in (cu_tokens, cu_keys, key_start, key_rows, kv))
    a.num_rows, a.num_keys, a.max_row_tokens = rows, E, max(lens)
    assert -(-max(lens) // 256) * rows * heads * 2 >= 148  # (fewer take the kernel of 64 queries)
    ops.latent_prompt_attention(a, kv)
    torch.cuda.synchronize()
    t = e = 0
    want = torch.empty(T, heads, vdim, dtype=torch.float64, device=dev)
    for n, p, f, c in zip(lens, past, first, count):
        k = torch.cat([kv[e: e + c, : heads * dim].view(c, heads, dim), key_rows[e: e + c, None, kv_pad: kv_pad + rot].expand(-1, heads, -1)], dim=-1).double()
        v = kv[e: e + c, heads * dim:].view(c, heads, vdim).double()
        s = torch.einsum("qhd,khd->hqk", q[t: t + n].double(), k) * a.scale
        age = torch.arange(p, p + n, device=dev)[:, None] - torch.arange(f, f + c, device=dev)[None]
        s = s.masked_fill((age < 0) | (age >= (window or 1 << 30)), -math.inf)
        if sinks:
            s = torch.cat([s, sink.double()[:, None, None].expand(-1, n, 1)], dim=-1)
        want[t: t + n] = torch.einsum("hqk,khv->qhv", torch.softmax(s, dim=-1)[..., :c], v)
        t, e = t + n, e + c
    want *= torch.sigmoid(gate.double()).view(T, heads, -1)
    want = want.reshape(T, -1)
    assert not torch.isnan(out.float()).any() and rel(out, want) < 2.5e-3
    off = (out.double() - want).abs() - 2 ** -8 * want.abs()
    assert float(off.max() / want.square().mean().sqrt()) < 1e-2


# ---------------------------------------------------------------------------------------------------------------------
# Blockwise FP8 over pairs of weight tiles (more than 128 tokens): an odd tile at the end, tokens inside the last block, K split or not.
# ---------------------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("M,N,K", [(129, 384, 512), (200, 2560, 4096), (257, 640, 128), (1000, 4224, 384), (4097, 1024, 512)])
def test_blockwise_gemm_over_pairs_of_weight_tiles(ops, M, N, K):
    from oracle import decode_oracle as O

    x, w, b = randn(M, K, seed=1), randn(N, K, seed=2, scale=K ** -0.5), randn(N, seed=3)
    xd, wd = O.dequantize_fp8_rowblock(*O.quantize_fp8_rowblock(x.cpu())), O.dequantize_fp8_block_weight(*O.quantize_fp8_block_weight(w.cpu()))
    ref = (xd.double() @ wd.double().T).cuda()
    xq, wq = ops.quantize_fp8_rowblock(x), ops.quantize_fp8_weight_block128(w)
    assert rel(ops.gemm_fp8_block(xq, wq), ref) < 3e-3
    assert rel(ops.gemm_fp8_block(xq, wq, b), ref.to(BF16).double() + b.double()) < 3e-3
    parts = ops.gemm_splitk(xq, wq)
    got = parts.buf.view(torch.float32)[: parts.num_splits * M * N].view(parts.num_splits, M, N).sum(0)
    assert rel(got, ref) < 1e-5


# ---------------------------------------------------------------------------------------------------------------------
# Scans start their longest rows first (up to 32 rows): the bits of every row are those of the row alone, whatever its place.
# ---------------------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("heads,dim,rows", [(2, 64, 32), (2, 64, 33), (1, 128, 5), (1, 48, 1)])
def test_scanned_rows_do_not_depend_on_the_others(ops, heads, dim, rows):
    from test_zinurax_kernels_gpu import DeltaCase

    rank, lens = 16, [(7 * i + 3) % 41 for i in range(rows)]  # ties, and a row of no token from 6 rows on
    T = sum(lens)
    c = DeltaCase(heads, dim, rank, T, torch.bfloat16, seed=50)
    at = torch.tensor([0] + lens).cumsum(0).int()
    slots = torch.arange(rows, dtype=torch.int32)
    z = None
    results = []
    for alone in (False, True):
        state = torch.randn(rows, heads, dim, dim, generator=torch.Generator().manual_seed(51)).cuda()
        o, out = torch.zeros(T, c.n, device="cuda"), torch.empty(T, c.n, dtype=BF16, device="cuda")
        lora = torch.empty(T, rank, dtype=BF16, device="cuda")
        for group in ([[r] for r in range(rows)] if alone else [list(range(rows))]):
            rd = slots[group[0]: group[-1] + 1].cuda()
            cu = at[group[0]: group[-1] + 2].cuda()
            a = c.args(state, rd, rd, out)
            a.num_rows, a.cu_tokens, a.o_f32, a.lora = len(group), cu.data_ptr(), o.data_ptr(), lora.data_ptr()
            if z is None:
                ops.delta_lora(a, state)
                z = ops.linear(lora, c.dev[1])
            a.z = z.data_ptr()
            ops.delta_scan(a, state)
            torch.cuda.synchronize()
        results.append((o, state))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


def test_a_row_that_ends_before_it_starts_is_left_out(ops):
    from test_zinurax_kernels_gpu import DeltaCase

    T = 40
    c = DeltaCase(2, 64, 16, T, torch.bfloat16, seed=50)
    before = torch.randn(3, 2, 64, 64, generator=torch.Generator().manual_seed(51)).cuda()
    slots = torch.arange(3, dtype=torch.int32, device="cuda")
    o, out, lora = torch.zeros(T, c.n, device="cuda"), torch.empty(T, c.n, dtype=BF16, device="cuda"), torch.empty(T, 16, dtype=BF16, device="cuda")
    state = before.clone()
    a = c.args(state, slots, slots, out)
    whole, torn = (torch.tensor(at, dtype=torch.int32, device="cuda") for at in ([0, 20, 20, 40], [0, 20, 10, 40]))  # (rows 0 and 2 share tokens 10 to 19)
    a.num_rows, a.cu_tokens, a.o_f32, a.lora = 3, whole.data_ptr(), o.data_ptr(), lora.data_ptr()
    ops.delta_lora(a, state)
    z = ops.linear(lora, c.dev[1])
    a.z, a.cu_tokens = z.data_ptr(), torn.data_ptr()
    ops.delta_scan(a, state)
    torch.cuda.synchronize()
    assert torch.equal(state[1], before[1]) and not torch.equal(state[0], before[0]) and not torch.equal(state[2], before[2])


# ---------------------------------------------------------------------------------------------------------------------
# K splits as clusters: bf16 out of the sums of partial tiles, against the same sums through `gemm_splitk` (same splits, same order: same bits).
# ---------------------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("M,N,K", [(1, 10304, 2048), (4, 2560, 512), (33, 384, 1024), (64, 6144, 4096), (100, 6144, 4096), (128, 132, 4096), (17, 1000, 640)])
def test_splits_in_clusters_give_the_bits_of_the_summed_partials(ops, M, N, K):
    x, w, b = randn(M, K, seed=1), randn(N, K, seed=2, scale=K ** -0.5), randn(N, seed=3)
    parts = ops.gemm_splitk(x, w)
    assert parts.num_splits > 1
    p = parts.buf.view(torch.float32)[: parts.num_splits * M * N].view(parts.num_splits, M, N).clone()
    total = p[0].clone()
    for s in range(1, parts.num_splits):
        total += p[s]
    y = ops.gemm(x, w)
    assert torch.equal(y, total.to(BF16))
    assert torch.equal(ops.gemm(x, w, b), (total.to(BF16).float() + b.float()).to(BF16))
    assert torch.equal(ops.linear(x, w, act="relu2"), torch.relu(total).square().to(BF16))
    wide = torch.zeros(M, N + 3, dtype=BF16, device="cuda")
    ops.linear(x, w, out=wide[:, :N])
    assert torch.equal(wide[:, :N], y) and not wide[:, N:].any()
    if K % 128 == 0:
        xq, wq = ops.quantize_mxfp8(x), ops.quantize_mxfp8_weight(w)
        parts = ops.gemm_splitk(xq, wq)
        p = parts.buf.view(torch.float32)[: parts.num_splits * M * N].view(parts.num_splits, M, N).clone()
        total = p[0].clone()
        for s in range(1, parts.num_splits):
            total += p[s]
        assert torch.equal(ops.gemm_mxfp8(xq, wq), total.to(BF16))


# Both sides of the limits of clusters: four splits, 24 rows, N a multiple of 4 (of the shapes above, those of 33 rows and more do not form any).  K splits of
# bf16 and MXFP8, and whether they form clusters, which need no scratch.
@pytest.mark.parametrize("M,N,K,bf16,mxfp8", [
    (24, 4700, 1024, (4, True), (2, True)),    # the most rows and splits; N 92 past a tile
    (25, 4700, 1024, (4, False), (2, False)),  # one row more
    (31, 388, 768, (3, False), None),
    (32, 4700, 2048, (8, False), (4, False)),  # a full tile
    (8, 384, 1280, (5, False), (2, True)),     # one split more
    (12, 388, 768, (3, True), None),
    (3, 390, 1024, (4, False), (2, False)),    # N even only
    (24, 4700, 2048, (8, False), (4, True)),
    (7, 132, 1536, (6, False), (3, True)),
    (1, 4, 1024, (4, True), (2, True)),        # the smallest N
    (2, 128, 2560, (10, False), (5, False)),
])
def test_splits_on_both_sides_of_the_cluster_limits(ops, M, N, K, bf16, mxfp8):
    from megatron_mixtera_b200 import _lib

    lib = _lib.load()
    for recipe, scratch, expected in ((None, lib.b200_gemm_bf16_workspace_bytes, bf16), ("mxfp8", lib.b200_gemm_mxfp8_workspace_bytes, mxfp8)):
        if expected is not None:
            assert (ops.gemm_num_splits(recipe, M, N, K), scratch(M, N, K) == 0) == expected
    test_splits_in_clusters_give_the_bits_of_the_summed_partials(ops, M, N, K)


# ---------------------------------------------------------------------------------------------------------------------
# Output norm: few rows and many, one to eight vectors per thread, widths that end inside a thread's vectors.  fp32 sums of up to 8192 terms: 1e-5.
# ---------------------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("accumulate", [0, 1])
@pytest.mark.parametrize("rows,width,splits", [(1, 2048, 8), (5, 1000, 3), (3, 1028, 1), (296, 4096, 2), (7, 8192, 5), (2, 4100, 1), (297, 2048, 1), (300, 96, 2),
                                               (400, 2052, 1), (310, 4096, 2), (298, 8188, 1), (3, 8200, 2)])
def test_output_norm_by_rows_and_width(ops, rows, width, splits, accumulate):
    p = torch.randn(splits, rows, width, generator=torch.Generator().manual_seed(1)).cuda()
    gamma, before = randn(width, seed=2), torch.randn(rows, width, generator=torch.Generator().manual_seed(3)).cuda()
    hidden = before.clone()
    y = ops.out_norm(ops.GemmPartials(p, splits, (rows, width)), gamma, eps=1e-5, hidden=hidden, accumulate=bool(accumulate))
    x = p.double().sum(0)
    x = x - x.mean(-1, keepdim=True)
    want = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * gamma.double() + accumulate * before.double()
    assert float((hidden.double() - want).abs().max()) < 1e-5 * float(want.abs().max())
    assert torch.equal(y, hidden.to(BF16))


# One row more than SMs, and than twice as many, with two, three and four vectors a thread; three on 256 threads.
@pytest.mark.parametrize("accumulate", [0, 1])
@pytest.mark.parametrize("rows,width,splits", [(148, 2052, 1), (148, 6144, 3), (148, 8192, 2), (149, 2052, 2), (149, 3076, 1), (149, 4100, 1), (149, 8188, 3),
                                               (296, 6144, 2), (297, 3072, 1), (297, 3076, 2), (297, 6144, 1), (297, 6148, 3)])
def test_output_norm_by_rows_on_an_sm(ops, rows, width, splits, accumulate):
    test_output_norm_by_rows_and_width(ops, rows, width, splits, accumulate)
