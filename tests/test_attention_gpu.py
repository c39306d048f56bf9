"""Fused causal attention (tb_attention_fwd / tb_attention_bwd) against the CPU oracle's
scores -> mask -> softmax -> P V chain and its backward (model/attention.c:32-60;
model/gpu_train.c:435-455), through the C ABI.  Metric: max|got-want| / max|want|."""
import numpy as np
import pytest
import torch

from conftest import rel_to_maxabs
from oracle.pyoracle import BF16, FP32

pytestmark = pytest.mark.gpu

TOL_FWD = 1e-2        # bf16 P and V operands; P is rounded against the running maximum
TOL_BWD = 2e-2        # the BF16-mode bound


def make_qkv(oracle, B, H, T, hd, seed):
    rng = np.random.default_rng(seed)
    q, k, v = (oracle.round(rng.standard_normal((B * H, T, hd)).astype(np.float32), BF16) for _ in range(3))
    return q, k, v


def dev16(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda().to(torch.bfloat16)


@pytest.mark.parametrize("dims", [(1, 2, 12, 16), (2, 2, 200, 32), (1, 3, 320, 64), (1, 2, 1024, 64), (2, 1, 130, 8)])
def test_attention_fwd_bwd_matches_oracle(tb, oracle, dims):
    B, H, T, hd = dims
    D = H * hd
    scale = float(1.0 / np.sqrt(np.float32(hd)))
    q, k, v = make_qkv(oracle, B, H, T, hd, 3)
    Q, K, V = dev16(q), dev16(k), dev16(v)
    att = torch.full((B * T, D), float("nan"), device="cuda", dtype=torch.bfloat16)
    lse = torch.zeros(B * H, T, device="cuda")
    tb.attention_fwd(Q, K, V, att, lse, B, H, T, hd, scale)
    tb.sync_check()
    O, P = oracle.attention_fwd(q, k, v, scale, mode=BF16, want_P=True)
    want = oracle.heads_merge(O, B, T, H, hd)
    got = att.float().cpu().numpy()
    assert np.isfinite(got).all()
    assert rel_to_maxabs(got, want) <= TOL_FWD
    assert rel_to_maxabs(got, oracle.heads_merge(oracle.attention_fwd(q, k, v, scale, mode=FP32), B, T, H, hd)) <= 2e-2
    # log-sum-exp of the masked, scaled scores
    S = np.einsum("zid,zjd->zij", q.astype(np.float64), k.astype(np.float64)) * scale
    S = np.where(np.tril(np.ones((T, T), bool))[None], S, -np.inf)
    want_lse = np.log(np.exp(S - S.max(-1, keepdims=True)).sum(-1)) + S.max(-1)
    assert np.abs(lse.cpu().numpy() - want_lse).max() <= 1e-3

    rng = np.random.default_rng(4)
    datt = oracle.round(rng.standard_normal((B * T, D)).astype(np.float32), BF16)
    dQ, dK, dV = (torch.full((B * H, T, hd), float("nan"), device="cuda") for _ in range(3))
    delta = torch.zeros(B * H, T, device="cuda")
    tb.attention_bwd(Q, K, V, att, dev16(datt), lse, delta, dQ, dK, dV, B, H, T, hd, scale)
    tb.sync_check()
    dO = oracle.heads_split(datt, B, T, H, hd)
    wq, wk, wv = oracle.attention_bwd(q, k, v, dO, scale, mode=BF16)
    for got_t, want_a, name in ((dQ, wq, "dQ"), (dK, wk, "dK"), (dV, wv, "dV")):
        g = got_t.cpu().numpy()
        assert np.isfinite(g).all(), name
        assert rel_to_maxabs(g, want_a) <= TOL_BWD, name


@pytest.mark.parametrize("dims", [(2, 1, 2, 8), (1, 3, 16, 40), (2, 2, 17, 32), (1, 2, 64, 64), (3, 1, 127, 64), (50, 6, 128, 64)])
def test_attention_of_one_block(tb, oracle, dims):
    """Sequences of up to 128 positions have a backward kernel of their own: edges of its products' 16-row steps and of
    the block, narrow heads, more heads than fit on the device at a time."""
    test_attention_fwd_bwd_matches_oracle(tb, oracle, dims)


@pytest.mark.parametrize("dims", [(2, 6, 1024, 64), (3, 6, 777, 64), (4, 3, 200, 32), (8, 6, 1000, 16)])
def test_probabilities_are_rounded_against_the_rows_maximum(tb, dims):
    """Rows in which a few keys have most of the weight (q four times as large): the largest probability is 1 and exact in
    bf16, so what is left of the forward pass's error is mostly the rounding of its bf16 output.  That is uniform within half a
    unit in the last place, 2^-8 of a power of two: 2^-8 / sqrt(3) times the root of the mean of 1 / m^2 over mantissas m
    whose logarithm is uniform, 0.736, so 1.66e-3 in the 2-norm.  The roundings of P may add half as much in quadrature; with P
    taken against an older maximum they add 0.65 times as much at 777 keys and up."""
    B, H, T, hd = dims
    gen = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(B * H, T, hd, device="cuda", generator=gen) for _ in range(3))
    q, k, v = (4 * q).bfloat16(), k.bfloat16(), v.bfloat16()
    att = torch.empty(B * T, H * hd, device="cuda", dtype=torch.bfloat16)
    lse = torch.empty(B * H, T, device="cuda")
    tb.attention_fwd(q, k, v, att, lse, B, H, T, hd, float(hd) ** -0.5)
    tb.sync_check()
    s = (q.double() @ k.double().transpose(1, 2)) * float(hd) ** -0.5
    s = s.masked_fill(torch.ones(T, T, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    want = (s.softmax(-1) @ v.double()).view(B, H, T, hd).transpose(1, 2).reshape(B * T, H * hd)
    output_rounding = 2.0 ** -8 / np.sqrt(3.0) * 0.736
    assert float((att.double() - want).norm() / want.norm()) <= output_rounding * np.sqrt(1 + 0.5 ** 2)


def test_attention_properties_at_benchmark_size(tb):
    """B=16, H=6, T=1024, hd=64 (the attention configuration of the benchmark): rows of P sum to 1
    (V = 1 gives O = 1), and a change in later keys/values leaves earlier outputs bit-identical."""
    B, H, T, hd = 16, 6, 1024, 64
    D = H * hd
    scale = 0.125
    g = torch.Generator(device="cuda").manual_seed(2)
    Q = torch.randn(B * H, T, hd, device="cuda", generator=g).to(torch.bfloat16)
    K = torch.randn(B * H, T, hd, device="cuda", generator=g).to(torch.bfloat16)
    V = torch.ones(B * H, T, hd, device="cuda", dtype=torch.bfloat16)
    att = torch.zeros(B * T, D, device="cuda", dtype=torch.bfloat16)
    lse = torch.zeros(B * H, T, device="cuda")
    tb.attention_fwd(Q, K, V, att, lse, B, H, T, hd, scale)
    tb.sync_check()
    assert (att.float() - 1.0).abs().max().item() <= 1e-2
    V = torch.randn(B * H, T, hd, device="cuda", generator=g).to(torch.bfloat16)
    a1 = torch.zeros_like(att)
    tb.attention_fwd(Q, K, V, a1, lse, B, H, T, hd, scale)
    K2, V2 = K.clone(), V.clone()
    K2[:, 700:] = 3.0
    V2[:, 700:] = -2.0
    a2 = torch.zeros_like(att)
    tb.attention_fwd(Q, K2, V2, a2, lse, B, H, T, hd, scale)
    tb.sync_check()
    a1 = a1.view(B, T, D)
    a2 = a2.view(B, T, D)
    assert torch.equal(a1[:, :700], a2[:, :700])
    assert not torch.equal(a1[:, 700:], a2[:, 700:])
    a3 = torch.zeros_like(att)
    tb.attention_fwd(Q, K, V, a3, lse, B, H, T, hd, scale)
    tb.sync_check()
    assert torch.equal(a3.view(B, T, D), a1)          # bitwise reproducible


def test_strided_qkv_projection_rope_then_attention_at_benchmark_size(tb, oracle):
    """The attention configuration of the benchmark (B=16, H=6, T=1024, hd=64) from the reference's strided
    layout: q, k, v are column slices of one [B*T, 3D] projection (model/attention.c:26-29,50-53).  The QKV GEMM
    with the fused position embedding and head split is compared with the oracle's projection + k_qkv_rope_split
    restatement (cuda/train_kernels.cu:573-597) on every element; fused attention forward and backward then run
    on that output for all 96 heads and are compared with the oracle on a handful of them."""
    import os
    B, H, T, hd = 16, 6, 1024, 64
    D, N = H * hd, B * T
    scale = float(1.0 / np.sqrt(np.float32(hd)))
    oracle.set_threads(min(os.cpu_count() or 8, 64))
    rng = np.random.default_rng(2)
    X = oracle.round(rng.standard_normal((N, D)).astype(np.float32), BF16)
    W = oracle.round((rng.standard_normal((D, 3 * D)) / np.sqrt(D)).astype(np.float32), BF16)   # q, k, v ~ N(0, 1)
    bias = (0.1 * rng.standard_normal(3 * D)).astype(np.float32)
    cos_t, sin_t = oracle.rope_tables(T, hd)
    qkv16 = torch.full((3, B, H, T, hd), float("nan"), device="cuda", dtype=torch.bfloat16)
    tb.gemm_qkv_rope_bf16(dev16(X), dev16(W), torch.from_numpy(bias).cuda(), torch.from_numpy(cos_t).cuda(),
                          torch.from_numpy(sin_t).cuda(), B, T, H, hd, qkv16)
    tb.sync_check()
    want_qkv = oracle.gemm_bias(X, W, bias, None, mode=BF16)
    wq, wk, wv = oracle.qkv_rope_split(want_qkv, B, T, H, hd)
    got = qkv16.float().cpu().numpy().reshape(3, B * H, T, hd)
    assert np.isfinite(got).all()
    for g, w, name in zip(got, (wq, wk, wv), "QKV"):
        assert rel_to_maxabs(g, w) <= 4e-3, name            # one bf16 rounding of the stored value (2^-9 of it)

    # attention on the stored bf16 q, k, v: all heads on the device, a handful against the oracle
    Q, K, V = qkv16[0].reshape(B * H, T, hd), qkv16[1].reshape(B * H, T, hd), qkv16[2].reshape(B * H, T, hd)
    att = torch.full((N, D), float("nan"), device="cuda", dtype=torch.bfloat16)
    lse = torch.zeros(B * H, T, device="cuda")
    tb.attention_fwd(Q, K, V, att, lse, B, H, T, hd, scale)
    datt = oracle.round(np.random.default_rng(5).standard_normal((N, D)).astype(np.float32), BF16)
    dQ, dK, dV = (torch.full((B * H, T, hd), float("nan"), device="cuda") for _ in range(3))
    delta = torch.zeros(B * H, T, device="cuda")
    tb.attention_bwd(Q, K, V, att, dev16(datt), lse, delta, dQ, dK, dV, B, H, T, hd, scale)
    tb.sync_check()
    heads = [0, 17, 40, 63, 95]                                # (batch, head) = divmod(index, H)
    q, k, v = (got[i][heads] for i in range(3))
    O = oracle.attention_fwd(q, k, v, scale, mode=BF16)
    att_h = att.float().cpu().numpy().reshape(B, T, H, hd)
    dO = np.stack([datt.reshape(B, T, H, hd)[z // H, :, z % H, :] for z in heads])
    wdq, wdk, wdv = oracle.attention_bwd(q, k, v, dO, scale, mode=BF16)
    for i, z in enumerate(heads):
        assert rel_to_maxabs(att_h[z // H, :, z % H, :], O[i]) <= TOL_FWD, z
        for got_t, want_a, name in ((dQ, wdq, "dQ"), (dK, wdk, "dK"), (dV, wdv, "dV")):
            assert rel_to_maxabs(got_t[z].cpu().numpy(), want_a[i]) <= TOL_BWD, (z, name)
    assert torch.isfinite(att.float()).all() and all(torch.isfinite(t).all() for t in (dQ, dK, dV))
