"""Kernels for many tokens (prompts) at the edges of their tiles: GEMMs of CTA pairs."""
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
    (1000, 4100, 72),    # K of one block and a bit, N 4 past a tile
    (4097, 1000, 512),   # N inside the last tile's first half
    (2048, 2048, 1000),  # K no multiple of a block
    (5000, 1160, 64),    # a single K block
    (300, 16384, 192),
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


@pytest.mark.parametrize("M,F,K", [(257, 7168, 256), (2048, 1024, 512), (1500, 3200, 72)])
def test_pair_gemm_swiglu_equals_gemm_then_activation(ops, M, F, K):
    x, w = randn(M, K, seed=4), randn(2 * F, K, seed=5, scale=K ** -0.5)
    assert ops.gemm_swiglu_supported(M, 2 * F, K)
    got = ops.gemm_swiglu(x, ops.interleave_gate_up(w))
    assert torch.equal(got, ops.activation(ops.gemm(x, w), "swiglu"))


@pytest.mark.parametrize("M,N,K", [(257, 14336, 128), (1000, 4224, 384), (4097, 1024, 512), (2048, 2048 + 40, 1024)])
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


@pytest.mark.parametrize("M,F,K", [(257, 7168, 256), (1500, 2176, 384), (2048, 1024, 1024)])
def test_pair_gemm_mxfp8_swiglu_equals_gemm_then_activation(ops, M, F, K):
    x, w = ops.quantize_mxfp8(randn(M, K, seed=9)), ops.quantize_mxfp8_weight(randn(2 * F, K, seed=10, scale=K ** -0.5))
    y = ops.gemm_mxfp8(x, w)
    assert torch.equal(ops.gemm_mxfp8_swiglu(x, w, quantize=False), ops.activation(y, "swiglu"))
    got, want = ops.gemm_mxfp8_swiglu(x, w), ops.activation_mxfp8(y, "swiglu")
    r, b = torch.arange(M)[:, None], torch.arange(F // 32)[None, :]
    at = ((r // 128) * (F // 128) * 512 + (b // 4) * 512 + (r % 32) * 16 + ((r % 128) // 32) * 4 + b % 4).reshape(-1).cuda()
    assert torch.equal(got.q, want.q) and torch.equal(got.sf[at], want.sf[at])
