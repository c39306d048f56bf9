"""Parity of the sm_100a GEMM path with the CPU oracle, through the C ABI.

Two comparisons per case, both with the reference's metric max|got-want| / max|want|
(tests/test_gpu_train.c:53-66):
  * against the oracle with operands rounded to bf16 first -- only the float32 summation order
    differs, so the bound is 2e-5;
  * against the float32 oracle -- the BF16-mode bound 2e-2 the task states.
"""
import json
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from conftest import golden_path, rel_to_maxabs
from oracle.pyoracle import BF16, FP32

pytestmark = pytest.mark.gpu

TOL_SAME_OPERANDS = 2e-5
TOL_BF16_MODE = 2e-2

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

KINDS = {"NN": 0, "NT": 1, "TN": 2}


def stored_shapes(kind, M, N, K):
    a = (K, M) if kind == 2 else (M, K)
    b = (N, K) if kind == 1 else (K, N)
    return a, b


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("kind", ["NN", "NT", "TN"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (4, 5, 3), (64, 48, 32), (127, 129, 65), (128, 128, 64),
                                   (200, 100, 72), (300, 260, 520), (1024, 384, 384)])
def test_gemm_f32_matches_oracle(tb, oracle, kind, shape):
    M, N, K = shape
    k = KINDS[kind]
    rng = np.random.default_rng(hash((kind, shape)) % (1 << 31))
    (ar, ac), (br, bc) = stored_shapes(k, M, N, K)
    A = rng.standard_normal((ar, ac)).astype(np.float32)
    B = (rng.standard_normal((br, bc)) * 0.02).astype(np.float32)
    C = torch.full((M, N), float("nan"), device="cuda")
    tb.gemm_f32(k, dev(A), dev(B), C, M, N, K, ac, bc, N)
    tb.sync_check()
    got = C.cpu().numpy()
    want16 = oracle.gemm(k // 2, k % 2, A, B, M, N, K, mode=BF16).reshape(M, N)
    want32 = oracle.gemm(k // 2, k % 2, A, B, M, N, K, mode=FP32).reshape(M, N)
    assert np.isfinite(got).all()
    assert rel_to_maxabs(got, want16) <= TOL_SAME_OPERANDS
    assert rel_to_maxabs(got, want32) <= TOL_BF16_MODE


TOL_TF32_MODE = 5e-3
TOL_FP32_MODE = 1e-5


@pytest.mark.parametrize("kind", ["NN", "NT", "TN"])
@pytest.mark.parametrize("shape", [(4, 5, 3), (127, 129, 65), (200, 100, 72), (300, 260, 520), (1024, 384, 384),
                                   (512, 1152, 384)])
def test_tf32_and_fp32_modes(tb, oracle, kind, shape):
    """TF32 mode: <= 5e-3 against the float32 oracle and <= 2e-5 against the oracle on tf32-truncated
    operands.  FP32 mode (three tf32 products): <= 1e-5 against the float64 product."""
    from oracle.pyoracle import TF32
    M, N, K = shape
    k = KINDS[kind]
    rng = np.random.default_rng(hash((kind, shape, 1)) % (1 << 31))
    (ar, ac), (br, bc) = stored_shapes(k, M, N, K)
    A = rng.standard_normal((ar, ac)).astype(np.float32)
    B = (rng.standard_normal((br, bc)) * 0.02).astype(np.float32)
    want32 = oracle.gemm(k // 2, k % 2, A, B, M, N, K, mode=FP32).reshape(M, N)
    want_tf = oracle.gemm(k // 2, k % 2, A, B, M, N, K, mode=TF32).reshape(M, N)
    truth = oracle.gemm_f64(k // 2, k % 2, A, B, M, N, K)
    C = torch.full((M, N), float("nan"), device="cuda")
    tb.gemm_f32(k, dev(A), dev(B), C, M, N, K, ac, bc, N, precision=tb.PREC_TF32)
    tb.sync_check()
    got = C.cpu().numpy()
    assert rel_to_maxabs(got, want_tf) <= TOL_SAME_OPERANDS
    assert rel_to_maxabs(got, want32) <= TOL_TF32_MODE
    C = torch.full((M, N), float("nan"), device="cuda")
    tb.gemm_f32(k, dev(A), dev(B), C, M, N, K, ac, bc, N, precision=tb.PREC_FP32)
    tb.sync_check()
    got = C.cpu().numpy()
    assert rel_to_maxabs(got, truth) <= TOL_FP32_MODE
    assert rel_to_maxabs(got, want32) <= TOL_FP32_MODE


@pytest.mark.parametrize("kind", ["NN", "NT", "TN"])
@pytest.mark.parametrize("shape", [(513, 1030, 44), (777, 384, 2112), (1024, 300, 2080), (2049, 700, 260), (512, 384, 2048)])
def test_tf32_and_fp32_modes_on_pair_tiles(tb, oracle, kind, shape):
    """Sizes at which float32 operands take 256 x 256 and 256 x 384 tiles of a CTA pair, ragged in every dimension."""
    test_tf32_and_fp32_modes(tb, oracle, kind, shape)


def test_modes_with_bias_residual_batch(tb, oracle):
    """Strided, batched, alpha/beta and bias+residual forms in the TF32 and FP32 modes."""
    rng = np.random.default_rng(33)
    M, N, K, batch = 70, 52, 40, 3
    lda, ldb, ldc = 44, 56, 60
    sA, sB, sC = M * lda + 4, K * ldb + 8, M * ldc + 4
    A = rng.standard_normal(batch * sA).astype(np.float32)
    B = rng.standard_normal(batch * sB).astype(np.float32)
    C0 = rng.standard_normal(batch * sC).astype(np.float32)
    want = oracle.gemm(0, 0, A, B, M, N, K, lda, ldb, ldc, batch, sA, sB, sC, alpha=0.5, beta=2.0, C_in=C0)
    for prec, tol in ((tb.PREC_TF32, TOL_TF32_MODE), (tb.PREC_FP32, TOL_FP32_MODE)):
        C = dev(C0.copy())
        tb.gemm_f32(0, dev(A), dev(B), C, M, N, K, lda, ldb, ldc, batch, sA, sB, sC, alpha=0.5, beta=2.0, precision=prec)
        tb.sync_check()
        assert rel_to_maxabs(C.cpu().numpy(), want) <= tol
    M, N, K = 260, 96, 384
    A = rng.standard_normal((M, K)).astype(np.float32)
    B = (rng.standard_normal((K, N)) * 0.02).astype(np.float32)
    bias = rng.standard_normal(N).astype(np.float32)
    res = rng.standard_normal((M, N)).astype(np.float32)
    want = oracle.gemm_bias(A, B, bias, res)
    for prec, tol in ((tb.PREC_TF32, TOL_TF32_MODE), (tb.PREC_FP32, TOL_FP32_MODE)):
        C = torch.zeros(M, N, device="cuda")
        tb.gemm_bias_f32(dev(A), dev(B), dev(bias), dev(res), C, M, N, K, precision=prec)
        tb.sync_check()
        assert rel_to_maxabs(C.cpu().numpy(), want) <= tol


def test_known_answer_vectors(tb):
    ka = json.load(open(golden_path("matmul_known_answers.json")))
    for name in ("test_tensor_2x2", "test_cuda_4x3x5"):
        c = ka[name]
        A, B = np.array(c["A"], np.float32), np.array(c["B"], np.float32)
        M, K = A.shape
        N = B.shape[1]
        out = np.zeros((M, N), np.float32)
        tb.matmul_host(A, B, out, M, K, N)          # small integers and halves: exact in bf16
        assert out.tolist() == c["C"], name
    c = ka["test_tensor_2x2_transposed_view"]
    At, B = np.array(c["A_stored"], np.float32), np.array(c["B"], np.float32)
    C = torch.zeros(2, 2, device="cuda")
    tb.gemm_f32(2, dev(At), dev(B), C, 2, 2, 2, 2, 2, 2)
    assert C.cpu().numpy().tolist() == c["C"]


def test_strided_batched_alpha_beta(tb, oracle):
    """The gemm()/bf16_gemm() interface in full: leading dimensions larger than the rows,
    batch strides, alpha and beta (model/gpu_train.c:45-78)."""
    rng = np.random.default_rng(3)
    M, N, K, batch = 70, 50, 40, 3
    lda, ldb, ldc = 44, 53, 57
    sA, sB, sC = M * lda + 5, K * ldb + 3, M * ldc + 7
    A = rng.standard_normal(batch * sA).astype(np.float32)
    B = rng.standard_normal(batch * sB).astype(np.float32)
    C0 = rng.standard_normal(batch * sC).astype(np.float32)
    C = dev(C0.copy())
    tb.gemm_f32(0, dev(A), dev(B), C, M, N, K, lda, ldb, ldc, batch, sA, sB, sC, alpha=0.5, beta=2.0)
    tb.sync_check()
    want = oracle.gemm(0, 0, A, B, M, N, K, lda, ldb, ldc, batch, sA, sB, sC, alpha=0.5, beta=2.0, C_in=C0, mode=BF16)
    got = C.cpu().numpy()
    assert rel_to_maxabs(got, want) <= TOL_SAME_OPERANDS
    # elements outside the [M,N] windows are untouched
    mask = np.ones(batch * sC, bool)
    for z in range(batch):
        for i in range(M):
            mask[z * sC + i * ldc: z * sC + i * ldc + N] = False
    assert np.array_equal(got[mask], C0[mask])


def test_gemm_bias_residual(tb, oracle):
    """k_bf16_gemm_nn_bias semantics: NULL bias / residual are skipped (train_kernels.cu:226-329)."""
    rng = np.random.default_rng(4)
    M, N, K = 260, 96, 384
    A = rng.standard_normal((M, K)).astype(np.float32)
    B = (rng.standard_normal((K, N)) * 0.02).astype(np.float32)
    bias = rng.standard_normal(N).astype(np.float32)
    res = rng.standard_normal((M, N)).astype(np.float32)
    for b, r in ((bias, res), (bias, None), (None, res), (None, None)):
        C = torch.zeros(M, N, device="cuda")
        tb.gemm_bias_f32(dev(A), dev(B), None if b is None else dev(b), None if r is None else dev(r), C, M, N, K)
        tb.sync_check()
        want = oracle.gemm_bias(A, B, b, r, mode=BF16)
        assert rel_to_maxabs(C.cpu().numpy(), want) <= TOL_SAME_OPERANDS


@pytest.mark.parametrize("precision", ["bf16", "tf32", "fp32"])
@pytest.mark.parametrize("name", ["qkv", "out", "gate_up", "down"])
def test_layer_gemms_fwd_dx_dw(tb, oracle, name, precision):
    """One layer's linear GEMMs at M = 4*256 tokens: forward, dX = dY W^T, dW = X^T dY, in each of the three
    operand precisions with its stated bound against the float32 oracle: 2e-2 (BF16), 5e-3 (TF32), 1e-5 (FP32)
    (the float32 oracle results are pinned to the reference by tests/golden/gemm_layer_digests.json)."""
    import os, sys
    from oracle.pyoracle import TF32
    sys.path.insert(0, os.path.dirname(golden_path("x")))
    from make_golden import gemm_inputs
    prec, mode_tol, same_mode = {"bf16": (tb.PREC_BF16, TOL_BF16_MODE, BF16), "tf32": (tb.PREC_TF32, TOL_TF32_MODE, TF32),
                                 "fp32": (tb.PREC_FP32, TOL_FP32_MODE, None)}[precision]
    d = json.load(open(golden_path("gemm_layer_digests.json")))[name]
    M, K, N = d["M"], d["K"], d["N"]
    X, W, dY = gemm_inputs(d["seed"], M, K, N)
    dX_, dW_, dY_ = dev(X), dev(W), dev(dY)
    C = torch.zeros(M, N, device="cuda")
    dX = torch.zeros(M, K, device="cuda")
    dW = torch.zeros(K, N, device="cuda")
    tb.gemm_f32(0, dX_, dW_, C, M, N, K, K, N, N, precision=prec)
    tb.gemm_f32(1, dY_, dW_, dX, M, K, N, N, N, K, precision=prec)
    tb.gemm_f32(2, dX_, dY_, dW, K, N, M, K, N, N, precision=prec)
    tb.sync_check()
    for got, (ta, tb_, A, B, m, n, k), key in (
            (C, (0, 0, X, W, M, N, K), "C"), (dX, (0, 1, dY, W, M, K, N), "dX"), (dW, (1, 0, X, dY, K, N, M), "dW")):
        got = got.cpu().numpy().reshape(-1)
        want32 = oracle.gemm(ta, tb_, A, B, m, n, k)
        step = max(1, want32.size // 16)
        assert np.allclose(want32[::step][:16], d[key + "_sample"], rtol=0, atol=0)   # same oracle as the fixture
        if same_mode is not None:
            want_same = oracle.gemm(ta, tb_, A, B, m, n, k, mode=same_mode)
            assert rel_to_maxabs(got, want_same) <= TOL_SAME_OPERANDS, key
        else:
            # the float32 oracle itself carries the rounding of a sequential float32 sum over k (up to 1024
            # terms); the float64 product is the truth the 1e-5 bound is stated against
            truth = oracle.gemm_f64(ta, tb_, A, B, m, n, k).reshape(-1)
            assert rel_to_maxabs(got, truth) <= TOL_FP32_MODE, key
        assert rel_to_maxabs(got, want32) <= mode_tol, key


@pytest.mark.parametrize("kind", ["NN", "NT", "TN"])
def test_bf16_entry_tiles_splits_outputs(tb, oracle, kind):
    """The native entry point: both tile widths, split-K with fixed-order partials, float32 and
    bf16 outputs, bias and beta; split results are bitwise reproducible."""
    k = KINDS[kind]
    rng = np.random.default_rng(10 + k)
    M, N, K = 384, 200, 4096
    (ar, ac), (br, bc) = stored_shapes(k, M, N, K)
    lda, ldb = (ac + 7) // 8 * 8, (bc + 7) // 8 * 8
    A = np.zeros((ar, lda), np.float32)
    B = np.zeros((br, ldb), np.float32)
    A[:, :ac] = oracle.round(rng.standard_normal((ar, ac)).astype(np.float32), BF16)
    B[:, :bc] = oracle.round(rng.standard_normal((br, bc)).astype(np.float32), BF16)
    A16, B16 = dev(A).to(torch.bfloat16), dev(B).to(torch.bfloat16)
    bias = rng.standard_normal(N).astype(np.float32)
    C0 = rng.standard_normal((M, N)).astype(np.float32)
    want = oracle.gemm(k // 2, k % 2, A, B, M, N, K, lda, ldb, N, beta=1.0, C_in=C0).reshape(M, N) + bias
    results = []
    for tile_n, splits in ((128, 1), (64, 1), (192, 1), (256, 1), (128, 8), (64, 5), (192, 3), (256, 4), (0, 0)):
        C = dev(C0.copy())
        C16 = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
        tb.gemm_bf16(k, A16, B16, M, N, K, lda, ldb, C32=C, ldc32=N, C16=C16, ldc16=N, bias=dev(bias), beta=1.0,
                     splits=splits, tile_n=tile_n)
        tb.sync_check()
        got = C.cpu().numpy()
        assert rel_to_maxabs(got, want) <= TOL_SAME_OPERANDS, (tile_n, splits)
        assert rel_to_maxabs(C16.float().cpu().numpy(), want) <= 1e-2
        C2 = dev(C0.copy())
        tb.gemm_bf16(k, A16, B16, M, N, K, lda, ldb, C32=C2, ldc32=N, bias=dev(bias), beta=1.0, splits=splits,
                     tile_n=tile_n)
        assert torch.equal(C, C2), "same launch twice must be bitwise identical"
        results.append(got)


@pytest.mark.parametrize("kind", ["NN", "TN"])
@pytest.mark.parametrize("shape", [(777, 384, 2112), (512, 300, 4160), (1024, 384, 4096), (130, 264, 200)])
def test_bf16_entry_384_column_pair_tiles(tb, oracle, kind, shape):
    """256 x 384 tiles on a CTA pair (three 128-column tensor-core instructions per K step, one accumulator): the form
    the LM-head gradients take (N = d_model <= 384, K = vocabulary or tokens).  B must be stored [K, N]."""
    k = KINDS[kind]
    M, N, K = shape
    rng = np.random.default_rng(40 + k + M)
    (ar, ac), (br, bc) = stored_shapes(k, M, N, K)
    lda, ldb = (ac + 7) // 8 * 8, (bc + 7) // 8 * 8
    A = np.zeros((ar, lda), np.float32)
    B = np.zeros((br, ldb), np.float32)
    A[:, :ac] = oracle.round(rng.standard_normal((ar, ac)).astype(np.float32), BF16)
    B[:, :bc] = oracle.round(rng.standard_normal((br, bc)).astype(np.float32), BF16)
    A16, B16 = dev(A).to(torch.bfloat16), dev(B).to(torch.bfloat16)
    bias = rng.standard_normal(N).astype(np.float32)
    C0 = rng.standard_normal((M, N)).astype(np.float32)
    want = oracle.gemm(k // 2, k % 2, A, B, M, N, K, lda, ldb, N, beta=1.0, C_in=C0).reshape(M, N) + bias
    for tile_n, splits in ((384, 1), (384, 2), (384, 3), (0, 0)):
        C = dev(C0.copy())
        tb.gemm_bf16(k, A16, B16, M, N, K, lda, ldb, C32=C, ldc32=N, bias=dev(bias), beta=1.0, splits=splits, tile_n=tile_n)
        tb.sync_check()
        assert rel_to_maxabs(C.cpu().numpy(), want) <= TOL_SAME_OPERANDS, (tile_n, splits)
        C2 = dev(C0.copy())
        tb.gemm_bf16(k, A16, B16, M, N, K, lda, ldb, C32=C2, ldc32=N, bias=dev(bias), beta=1.0, splits=splits, tile_n=tile_n)
        assert torch.equal(C, C2), "same launch twice must be bitwise identical"
    if kind == "NN":        # the same product with B stored [N, K] cannot take this tile
        Bt = dev(np.ascontiguousarray(np.zeros((N, (K + 7) // 8 * 8), np.float32))).to(torch.bfloat16)
        with pytest.raises(Exception):
            tb.gemm_bf16(KINDS["NT"], A16, Bt, M, N, K, lda, Bt.shape[1], C32=dev(C0.copy()), ldc32=N, tile_n=384)
            tb.sync_check()


def test_causal_modes(tb, oracle):
    """Batched square attention products restricted to the lower triangle."""
    rng = np.random.default_rng(20)
    T, hd, BH = 320, 64, 3
    Q = oracle.round(rng.standard_normal((BH, T, hd)).astype(np.float32), BF16)
    Kk = oracle.round(rng.standard_normal((BH, T, hd)).astype(np.float32), BF16)
    Q16, K16 = dev(Q).to(torch.bfloat16), dev(Kk).to(torch.bfloat16)
    S = torch.full((BH, T, T), float("nan"), device="cuda")
    tb.gemm_bf16(1, Q16, K16, T, T, hd, hd, hd, BH, T * hd, T * hd, C32=S, ldc32=T, sC32=T * T, causal=tb.CAUSAL_SKIP_UPPER)
    tb.sync_check()
    want = oracle.gemm(0, 1, Q, Kk, T, T, hd, batch=BH, sA=T * hd, sB=T * hd, sC=T * T).reshape(BH, T, T)
    got = S.cpu().numpy()
    low = np.tril(np.ones((T, T), bool))
    assert rel_to_maxabs(got[:, low], want[:, low]) <= TOL_SAME_OPERANDS
    # lower-triangular P times V with the k range cut at the tile's last row
    P = np.tril(rng.standard_normal((BH, T, T))).astype(np.float32)
    P = oracle.round(P, BF16)
    V = oracle.round(rng.standard_normal((BH, T, hd)).astype(np.float32), BF16)
    O = torch.zeros(BH, T, hd, device="cuda")
    tb.gemm_bf16(0, dev(P).to(torch.bfloat16), dev(V).to(torch.bfloat16), T, hd, T, T, hd, BH, T * T, T * hd,
                 C32=O, ldc32=hd, sC32=T * hd, causal=tb.CAUSAL_K_PREFIX)
    dV = torch.zeros(BH, T, hd, device="cuda")
    tb.gemm_bf16(2, dev(P).to(torch.bfloat16), dev(V).to(torch.bfloat16), T, hd, T, T, hd, BH, T * T, T * hd,
                 C32=dV, ldc32=hd, sC32=T * hd, causal=tb.CAUSAL_K_SUFFIX)
    tb.sync_check()
    wantO = oracle.gemm(0, 0, P, V, T, hd, T, batch=BH, sA=T * T, sB=T * hd, sC=T * hd)
    wantdV = oracle.gemm(1, 0, P, V, T, hd, T, batch=BH, sA=T * T, sB=T * hd, sC=T * hd)
    assert rel_to_maxabs(O.cpu().numpy().reshape(-1), wantO) <= TOL_SAME_OPERANDS
    assert rel_to_maxabs(dV.cpu().numpy().reshape(-1), wantdV) <= TOL_SAME_OPERANDS


def test_linearity_at_benchmark_size(tb):
    """Size-independent property at the benchmark's M = 8192: (A1 + A2) W = A1 W + A2 W up to
    float32 summation error, and the ragged 31,769-column head writes nothing past its edge."""
    torch.manual_seed(0)
    M, K, N = 8192, 384, 1152
    A1 = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    A2 = (torch.randn(M, K, device="cuda") * 4).to(torch.bfloat16)
    W = (torch.randn(K, N, device="cuda") * 0.02).to(torch.bfloat16)
    # pick A1, A2 with an exactly representable sum
    A1 = (A1.float() * 0 + torch.round(A1.float() * 8) / 8).to(torch.bfloat16)
    A2 = (torch.round(A2.float() * 8) / 8).to(torch.bfloat16)
    As = (A1.float() + A2.float()).to(torch.bfloat16)
    assert torch.equal(As.float(), A1.float() + A2.float())
    outs = []
    for A in (A1, A2, As):
        C = torch.zeros(M, N, device="cuda")
        tb.gemm_bf16(0, A, W, M, N, K, K, N, C32=C, ldc32=N)
        outs.append(C)
    tb.sync_check()
    err = (outs[2] - (outs[0] + outs[1])).abs().max().item() / outs[2].abs().max().item()
    assert err <= 1e-5
    V, ld = 31769, 31776
    nf = torch.randn(256, K, device="cuda").to(torch.bfloat16)
    E = (torch.randn(V, K, device="cuda") * 0.02).to(torch.bfloat16)
    logits = torch.full((256, ld), -7.0, device="cuda")
    tb.gemm_bf16(1, nf, E, 256, V, K, K, K, C32=logits, ldc32=ld)
    tb.sync_check()
    assert (logits[:, V:] == -7.0).all()
    want = nf.float() @ E.float().T
    assert ((logits[:, :V] - want).abs().max() / want.abs().max()).item() <= TOL_SAME_OPERANDS


def test_rejects_bad_arguments(tb):
    A = torch.zeros(8, 8, device="cuda", dtype=torch.bfloat16)
    C = torch.zeros(8, 8, device="cuda")
    with pytest.raises(tb.TbError):
        tb.gemm_bf16(0, A, A, 8, 8, 8, 7, 8, C32=C, ldc32=8)       # leading dimension not a multiple of 8
    with pytest.raises(tb.TbError):
        tb.gemm_bf16(0, A, A, 0, 8, 8, 8, 8, C32=C, ldc32=8)       # empty problem
    with pytest.raises(tb.TbError):
        tb.gemm_f32(0, C, C, C, 8, 8, 8, 8, 8, 8, precision=7)             # unknown precision mode


@pytest.mark.parametrize("shape", [(8192, 1024, 384), (200, 64, 72), (64, 128, 384), (333, 192, 96)])
def test_gemm_swiglu_epilogue(tb, oracle, shape):
    """tb_gemm_swiglu_bf16 against the oracle's two steps: the BF16-mode gate|up projection with bias
    (bf16_gemm_bias) and swiglu_fwd on it.  h and the kept gate|up are bf16, so the bound is the BF16
    mode's plus one bf16 rounding of the result."""
    import torch
    from oracle import pyoracle
    from turkce_llm_b200 import lib
    M, F, K = shape
    rng = np.random.default_rng(21)
    X = rng.standard_normal((M, K)).astype(np.float32)
    W = (rng.standard_normal((K, 2 * F)) * 0.05).astype(np.float32)
    bias = (rng.standard_normal(2 * F) * 0.1).astype(np.float32)
    gu_want = oracle.gemm_bias(X, W, bias, None, mode=pyoracle.BF16)
    h_want = oracle.swiglu_fwd(gu_want)
    x16 = torch.from_numpy(X).cuda().to(torch.bfloat16)
    w16 = torch.from_numpy(W).cuda().to(torch.bfloat16)
    b = torch.from_numpy(bias).cuda()
    h16 = torch.full((M, F), 7.0, device="cuda", dtype=torch.bfloat16)
    gu16 = torch.full((M, 2 * F), 7.0, device="cuda", dtype=torch.bfloat16)
    lib.gemm_swiglu_bf16(x16, w16, b, h16, gu16)
    h_only = torch.full((M, F), 7.0, device="cuda", dtype=torch.bfloat16)
    lib.gemm_swiglu_bf16(x16, w16, b, h_only, None)
    lib.sync_check()
    assert rel_to_maxabs(gu16.float().cpu().numpy(), gu_want) <= 2e-2
    assert rel_to_maxabs(h16.float().cpu().numpy(), h_want) <= 2e-2
    assert torch.equal(h16, h_only)
    # bit-for-bit the same as the unfused route on the device: float32 projection, then bf16 SwiGLU of it
    gu32 = torch.empty(M, 2 * F, device="cuda")
    lib.gemm_bf16(0, x16, w16, M, 2 * F, K, K, 2 * F, C32=gu32, ldc32=2 * F, bias=b, splits=1)
    lib.sync_check()
    g, u = gu32[:, :F], gu32[:, F:]
    assert torch.equal(gu16, gu32.to(torch.bfloat16))
    h_ref = (g * (1.0 / (1.0 + torch.exp(-g))) * u)
    assert rel_to_maxabs(h16.float().cpu().numpy(), h_ref.cpu().numpy()) <= 1e-2


def test_matmul_host_from_several_threads(tb, oracle):
    """gpu_matmul is called from many worker threads at once in the reference's data-parallel step
    (model/gpu_ops.c:78-134): every thread has its own buffers, results are unaffected by the others, and a
    thread's repeated calls reuse its buffers (shapes shrink and grow)."""
    import threading
    rng = np.random.default_rng(77)
    shapes = [(64, 48, 32), (200, 384, 130), (17, 5, 300), (128, 1024, 384)]
    cases = []
    for M, K, N in shapes:
        A = rng.standard_normal((M, K)).astype(np.float32)
        B = (rng.standard_normal((K, N)) * 0.05).astype(np.float32)
        cases.append((A, B, oracle.gemm(0, 0, A, B, M, N, K, mode=BF16).reshape(M, N)))
    errors = []

    def worker(order):
        try:
            for _ in range(3):
                for i in order:
                    A, B, want = cases[i]
                    M, K = A.shape
                    N = B.shape[1]
                    out = np.zeros((M, N), np.float32)
                    tb.matmul_host(A, B, out, M, K, N)
                    if rel_to_maxabs(out, want) > TOL_SAME_OPERANDS:
                        errors.append((i, rel_to_maxabs(out, want)))
        except Exception as e:          # noqa: BLE001 -- reported by the assertion below
            errors.append(repr(e))
    threads = [threading.Thread(target=worker, args=(o,)) for o in ([0, 1, 2, 3], [3, 2, 1, 0], [1, 3, 0, 2], [2, 0, 3, 1])]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("pinned", [(1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1)])
@pytest.mark.parametrize("shape", [(300, 200, 100), (1030, 701, 777)])
def test_matmul_host_with_pinned_arrays(tb, shape, pinned):
    """Pinned host memory is copied as it is, each operand for itself; the arrays may change as soon as the call is back."""
    import torch
    M, K, N = shape
    a, b, c = (torch.empty(s, pin_memory=bool(p)) for s, p in zip(((M, K), (K, N), (M, N)), pinned))
    gen = torch.Generator().manual_seed(3)
    for _ in range(3):
        a.normal_(generator=gen), b.normal_(generator=gen)
        want = a.double() @ b.double()
        tb.matmul_host(a, b, c, M, K, N, tb.PREC_FP32)
        a.fill_(float("nan")), b.fill_(float("nan"))
        assert rel_to_maxabs(c, want) <= 1e-5


def test_pinned_arrays_are_not_staged(tb):
    """The copies of 48 MB from and to pinned memory take the bus's time: well under what the staging threads' copies add."""
    import time
    import torch
    M = N = 3000
    K = 40
    best = {}
    for pin in (False, True):
        a, b, c = (torch.zeros(s, pin_memory=pin) for s in ((M, K), (K, N), (M, N)))
        for _ in range(8):
            t0 = time.perf_counter()
            tb.matmul_host(a, b, c, M, K, N, tb.PREC_BF16)
            best[pin] = min(best.get(pin, 1e9), time.perf_counter() - t0)
    assert best[True] < 0.8 * best[False], best


@pytest.mark.parametrize("missing", [0, 1, 2])
def test_matmul_host_refuses_a_null_array(tb, missing):
    """(it is read and written by the host's own copies, not by the driver, which would refuse it)"""
    arrays = [np.ones((64, 64), np.float32) for _ in range(3)]
    arrays[missing] = None
    with pytest.raises(tb.TbError, match="NULL"):
        tb.matmul_host(*arrays, 64, 64, 64)


def test_matmul_host_from_more_threads_than_there_are_copy_buffers(tb):
    """Sixteen threads with products of one row block and of several: more transfers at a time than there are helper threads or
    pinned buffers, so that all three ways to copy are taken."""
    import threading
    rng = np.random.default_rng(79)
    cases = []
    for M, K, N in ((600, 900, 1000), (300, 400, 500), (64, 64, 64)):
        A, B = rng.standard_normal((M, K)).astype(np.float32), (rng.standard_normal((K, N)) * 0.05).astype(np.float32)
        cases.append((A, B, A.astype(np.float64) @ B.astype(np.float64)))
    errors, start = [], threading.Barrier(16)

    def worker(first):
        try:
            start.wait()
            for i in range(30):
                A, B, want = cases[(first + i) % len(cases)]
                out = np.zeros(want.shape, np.float32)
                tb.matmul_host(A, B, out, A.shape[0], A.shape[1], B.shape[1], tb.PREC_FP32)
                if rel_to_maxabs(out, want) > 1e-5:
                    errors.append(rel_to_maxabs(out, want))
        except Exception as e:          # noqa: BLE001 -- reported by the assertion below
            errors.append(repr(e))
    threads = [threading.Thread(target=worker, args=(t,)) for t in range(16)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("precision", ["bf16", "fp32"])
def test_matmul_host_in_row_blocks_beside_other_calls(tb, oracle, precision):
    """Products large enough for row blocks from several threads, with shapes that shrink and grow, while another thread has
    the device's scratch memory packed with operands of its own."""
    import threading
    import torch
    prec = {"bf16": tb.PREC_BF16, "fp32": tb.PREC_FP32}[precision]
    tol = {"bf16": 2e-2, "fp32": 1e-5}[precision]
    rng = np.random.default_rng(78)
    cases = []
    for M, K, N in ((1024, 512, 700), (700, 1024, 1024), (129, 64, 40), (2000, 300, 512)):
        A, B = rng.standard_normal((M, K)).astype(np.float32), (rng.standard_normal((K, N)) * 0.05).astype(np.float32)
        cases.append((A, B, A.astype(np.float64) @ B.astype(np.float64)))
    errors, done = [], threading.Event()

    def worker(order):
        try:
            for _ in range(6):
                for i in order:
                    A, B, want = cases[i]
                    out = np.zeros(want.shape, np.float32)
                    tb.matmul_host(A, B, out, A.shape[0], A.shape[1], B.shape[1], prec)
                    if rel_to_maxabs(out, want) > tol:
                        errors.append((i, rel_to_maxabs(out, want)))
        except Exception as e:          # noqa: BLE001 -- reported by the assertion below
            errors.append(repr(e))

    x, w = torch.randn(640, 500, device="cuda"), torch.randn(500, 330, device="cuda") * 0.05
    y, want_y = torch.empty(640, 330, device="cuda"), x.double() @ w.double()

    def device_calls():
        try:
            while not done.is_set():
                tb.gemm_f32(tb.NN, x, w, y, 640, 330, 500, 500, 330, 330, precision=prec)
                err = float((y.double() - want_y).abs().max() / want_y.abs().max())
                if err > tol:
                    errors.append(("device", err))
        except Exception as e:          # noqa: BLE001
            errors.append(repr(e))
    tb.gemm_f32(tb.NN, x, w, y, 640, 330, 500, 500, 330, 330, precision=prec)      # (sizes the device's scratch memory)
    threads = [threading.Thread(target=worker, args=(o,)) for o in ([0, 1, 2, 3], [3, 2, 1, 0], [1, 3, 0, 2])]
    beside = threading.Thread(target=device_calls)
    for t in threads + [beside]:
        t.start()
    for t in threads:
        t.join()
    done.set()
    beside.join()
    assert not errors, errors


@pytest.mark.parametrize("precision", ["bf16", "tf32", "fp32"])
@pytest.mark.parametrize("shape", [(255, 1031, 900), (257, 2000, 1025), (1030, 701, 777), (128, 300, 20000), (2049, 513, 1)])
def test_matmul_host_in_row_blocks(tb, oracle, shape, precision):
    """Host products around the sizes where they are cut into row blocks and the copies go through several threads: short
    last blocks, one block only, a result of one column."""
    M, K, N = shape
    rng = np.random.default_rng(5)
    A = rng.standard_normal((M, K)).astype(np.float32)
    B = (rng.standard_normal((K, N)) * 0.05).astype(np.float32)
    want = A.astype(np.float64) @ B.astype(np.float64)
    out = np.full((M, N), np.nan, np.float32)
    prec = {"bf16": tb.PREC_BF16, "tf32": tb.PREC_TF32, "fp32": tb.PREC_FP32}[precision]
    for _ in range(2):                       # (the second call finds the first one's buffers and packed operands)
        tb.matmul_host(A, B, out, M, K, N, prec)
        assert rel_to_maxabs(out, want) <= {"bf16": 2e-2, "tf32": 5e-3, "fp32": 1e-5}[precision]
        A *= -1.0
        want *= -1.0


@pytest.mark.parametrize("precision", ["bf16", "tf32"])
@pytest.mark.parametrize("kind", ["NN", "NT", "TN"])
@pytest.mark.parametrize("shape", [(200, 72, 1100, 2), (130, 260, 2048, 3), (384, 136, 1024, 5), (64, 64, 4096, 7), (257, 44, 2080, 8), (129, 131, 1500, 0)])
def test_splits_added_inside_a_cluster(tb, monkeypatch, kind, shape, precision):
    """Products split along K whose parts a cluster adds: ragged tiles, rows that do not divide by the splits, bias, alpha and beta, a
    leading dimension that keeps the output from 16-byte accesses, against float64 and the reduction kernel."""
    M, N, K, splits = shape
    rng = np.random.default_rng(M + N)
    A = rng.standard_normal((K, M) if kind == "TN" else (M, K)).astype(np.float32)
    B = (rng.standard_normal((N, K) if kind == "NT" else (K, N)) * 0.1).astype(np.float32)
    kn = {"NN": tb.NN, "NT": tb.NT, "TN": tb.TN}[kind]
    C0 = rng.standard_normal((M, N + 3)).astype(np.float32)
    got = []
    for off in (False, True):
        if off:
            monkeypatch.setenv("TB_GEMM_NO_CLUSTER_SPLIT", "1")
        before = tb.launch_count()
        if precision == "bf16":
            # (rows of 16 bytes for the operands)
            pad = lambda X: np.pad(X, ((0, 0), (0, -X.shape[1] % 8)))
            a, b = torch.from_numpy(pad(A)).cuda().bfloat16(), torch.from_numpy(pad(B)).cuda().bfloat16()
            C = torch.from_numpy(C0).cuda()
            bias = torch.from_numpy(C0[0, :N].copy()).cuda()
            tb.gemm_bf16(kn, a, b, M, N, K, a.shape[1], b.shape[1], C32=C, ldc32=N + 3, bias=bias, alpha=0.5, beta=2.0, splits=splits)
            want_a, want_b = a.double().cpu().numpy()[:, :A.shape[1]], b.double().cpu().numpy()[:, :B.shape[1]]
            want = 0.5 * ((want_a.T if kind == "TN" else want_a) @ (want_b.T if kind == "NT" else want_b)) + C0[0, :N].astype(np.float64) + 2.0 * C0[:, :N]
            launches = 1
            bound = 2e-5
        else:
            C = torch.from_numpy(C0).cuda()
            tb.gemm_f32(kn, torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), C, M, N, K, A.shape[1], B.shape[1], N + 3, alpha=0.5, beta=2.0,
                        precision=tb.PREC_TF32)
            want = 0.5 * ((A.T if kind == "TN" else A).astype(np.float64) @ (B.T if kind == "NT" else B).astype(np.float64)) + 2.0 * C0[:, :N]
            launches = None
            bound = 5e-3
        out = C.cpu().numpy()
        tb.sync_check()
        if launches is not None and splits:
            assert tb.launch_count() - before == (2 if off else launches)
        assert np.abs(out[:, :N] - want).max() <= bound * np.abs(want).max()
        assert np.array_equal(out[:, N:], C0[:, N:])
        got.append(out)
    if precision == "bf16" and splits:
        # the same parts in the same order
        assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("shape", [(64, 72, 1100, 4, 64), (200, 72, 1100, 2, 64), (130, 264, 2048, 8, 64), (384, 520, 2048, 4, 128),
                                   (640, 384, 4096, 8, 128), (640, 376, 2600, 7, 128), (1024, 512, 1024, 3, 128), (300, 568, 2608, 5, 192),
                                   (384, 1152, 2048, 6, 192)])
def test_cluster_sums_round_like_the_reduction_kernel(tb, monkeypatch, shape):
    """Whoever adds them, the parts of a product are as many and come in the same order: the same bits, in one launch and in two."""
    M, N, K, splits, bn = shape
    A, B = (torch.randn(r, c, device="cuda").bfloat16() for r, c in ((M, (K + 7) // 8 * 8), (K, N)))
    got = []
    for off in (False, True):
        if off:
            monkeypatch.setenv("TB_GEMM_NO_CLUSTER_SPLIT", "1")
        C = torch.empty(M, N, device="cuda")
        before = tb.launch_count()
        tb.gemm_bf16(tb.NN, A, B, M, N, K, A.shape[1], N, C32=C, ldc32=N, splits=splits, tile_n=bn)
        tb.sync_check()
        assert tb.launch_count() - before == (2 if off else 1)
        got.append(C)
    assert torch.equal(*got)


@pytest.mark.parametrize("kind", ["NN", "NT", "TN"])
@pytest.mark.parametrize("shape", [(4, 4, 192), (100, 68, 228), (132, 132, 420), (200, 72, 1100), (384, 1152, 1024), (1000, 260, 2048), (64, 2048, 384)])
def test_float32_product_splits_its_slices_on_chip(tb, monkeypatch, kind, shape):
    """Float32 accuracy in one launch: ragged tiles and slices, clusters of one to eight, an output that is not 16-byte
    addressable, bias, alpha, beta.  Bound per element: a rest is below 2^-10 of x and loses 2^-10 of itself, the product of two rests
    2^-20, three times 2^-20 of the sum of magnitudes in all; every addition of eight products may lose 2^-23 of it."""
    M, N, K = shape
    rng = np.random.default_rng(M + K)
    A = rng.standard_normal((K, M) if kind == "TN" else (M, K)).astype(np.float32)
    B = rng.standard_normal((N, K) if kind == "NT" else (K, N)).astype(np.float32)
    a64, b64 = (A.T if kind == "TN" else A).astype(np.float64), (B.T if kind == "NT" else B).astype(np.float64)
    C0 = rng.standard_normal((M, N + 3)).astype(np.float32)
    want = 0.5 * (a64 @ b64) + 2.0 * C0[:, :N]
    bound = (3 * 2.0 ** -20 + (K / 8 + 4) * 2.0 ** -23) * (0.5 * (np.abs(a64) @ np.abs(b64)) + 2.0 * np.abs(C0[:, :N]))
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()

    def run(C):
        out = torch.from_numpy(C).cuda()
        before = tb.launch_count()
        tb.gemm_f32({"NN": tb.NN, "NT": tb.NT, "TN": tb.TN}[kind], dA, dB, out, M, N, K, A.shape[1], B.shape[1], C.shape[1], alpha=0.5, beta=2.0,
                    precision=tb.PREC_FP32)
        tb.sync_check()
        return out.cpu().numpy(), tb.launch_count() - before

    one, launches = run(C0)
    assert launches == 1
    assert (np.abs(one[:, :N] - want) <= bound).all()
    assert np.array_equal(one[:, N:], C0[:, N:])
    assert np.array_equal(run(np.ascontiguousarray(C0[:, :N]))[0], one[:, :N]) and np.array_equal(run(C0)[0], one)
    if kind == "NN":
        bias, y = torch.from_numpy(C0[0, :N].copy()).cuda(), torch.zeros(M, N, device="cuda")
        tb.gemm_bias_f32(dA, dB, bias, None, y, M, N, K, precision=tb.PREC_FP32)
        assert (np.abs(y.cpu().numpy() - (a64 @ b64 + C0[0, :N])) <= 2 * bound + 2.0 ** -22 * np.abs(C0[0, :N])).all()
    # an infinity and a NaN: where the pieces written out in memory give none, none here
    dA[0, 0], dB[0, 1] = float("inf"), float("nan")
    special = run(C0)[0]
    monkeypatch.setenv("TB_GEMM_NO_X3", "1")
    pieces, launches = run(C0)
    assert launches >= 2 and np.array_equal(np.isfinite(special), np.isfinite(pieces))


def test_float32_product_over_its_operand_and_with_rows_that_repeat(tb):
    """Where C lies over A, or a leading dimension of zero repeats one row, the operands' pieces are written out first, as they were
    before there was a way without: the same result as with arrays apart."""
    n = 256
    A, B = torch.randn(n, n, device="cuda"), torch.randn(n, n, device="cuda")
    want = A.double() @ B.double()
    bound = (3 * 2.0 ** -20 + (n / 8 + 4) * 2.0 ** -23) * (A.double().abs() @ B.double().abs())
    C = A.clone()
    tb.gemm_f32(tb.NN, C, B, C, n, n, n, n, n, n, precision=tb.PREC_FP32)
    tb.sync_check()
    assert bool(((C.double() - want).abs() <= bound).all())
    tb.gemm_f32(tb.NN, A, B, C, n, n, n, 0, n, n, precision=tb.PREC_FP32)
    tb.sync_check()
    assert bool(((C.double() - want[:1]).abs() <= bound[:1]).all())


@pytest.mark.parametrize("over", ["A", "B"])
def test_split_product_over_its_operand(tb, over):
    """A product split along K writes C when its operands have been read, if C lies over one of them: the same bits as apart."""
    n = 512
    A, B = torch.randn(n, n, device="cuda"), torch.randn(n, n, device="cuda")
    got = []
    for apart in (True, False):
        a, b = A.clone(), B.clone()
        C = torch.empty_like(A) if apart else (a if over == "A" else b)
        tb.gemm_f32(tb.NN, a, b, C, n, n, n, n, n, n, precision=tb.PREC_TF32)
        tb.sync_check()
        got.append(C)
    assert torch.equal(*got)


@pytest.mark.parametrize("shape", [(4739, 390, 2100), (9601, 190, 2104), (9601, 150, 1190), (8300, 570, 1030), (5000, 1000, 700)])
@pytest.mark.parametrize("tf32", [False, True], ids=["bf16", "tf32"])
def test_192_column_tiles_on_cta_pairs(tb, monkeypatch, shape, tf32):
    """B stored [N, K], tiles of 256 x 192: ragged rows, columns and K, previous contents and bias, against float64 and single CTAs.
    Operands are exact in either type, so what differs is the sum: every addition of a K step may lose 2^-23 of the magnitudes."""
    M, N, K = shape
    rng = np.random.default_rng(M)
    ld = (K + 7) // 8 * 8
    A, B = torch.zeros(M, ld, device="cuda", dtype=torch.bfloat16), torch.zeros(N, ld, device="cuda", dtype=torch.bfloat16)
    A[:, :K] = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).cuda().bfloat16()
    B[:, :K] = torch.from_numpy(rng.standard_normal((N, K)).astype(np.float32)).cuda().bfloat16()
    C0 = torch.from_numpy(rng.standard_normal((M, N)).astype(np.float32)).cuda()
    bias = C0[0].clone()
    want = A[:, :K].double() @ B[:, :K].double().T + 2.0 * C0.double()
    bound = (K / 8 + 4) * 2.0 ** -23 * (A[:, :K].double().abs() @ B[:, :K].double().abs().T + 2.0 * C0.abs())
    if not tf32:
        want, bound = want + bias, bound + 2.0 ** -22 * bias.abs()
    a32, b32, got = A.float(), B.float(), []
    for single in (False, True):
        if single:
            monkeypatch.setenv("TB_GEMM_NO_PAIR", "1")
        C = C0.clone()
        tb.profile_begin()
        if tf32:
            tb.gemm_f32(tb.NT, a32, b32, C, M, N, K, ld, ld, N, beta=2.0, precision=tb.PREC_TF32)
        else:
            tb.gemm_bf16(tb.NT, A, B, M, N, K, ld, ld, C32=C, ldc32=N, bias=bias, beta=2.0, tile_n=192)
        tags = [t for t in tb.profile_end(torch.cuda.current_stream().cuda_stream) if t.startswith("gemm_")]
        assert len(tags) == 1 and (tags[0].endswith("bn192:pair") != single), tags
        tb.sync_check()
        assert bool(((C.double() - want).abs() <= bound).all())
        got.append(C)
    assert bool(((got[0] - got[1]).abs() <= 2 * bound).all())


@pytest.mark.parametrize("precision", ["native", "tf32", "fp32"])
def test_parts_of_a_split_product_are_scaled_before_they_are_added(tb, precision):
    """Each part is 2^126 or below and eight of them leave float32's range, but not alpha times them: every value here is a power of
    two or a sum of equal ones, so the result is exact."""
    n, K = 128, 1024
    A, B = torch.full((n, K), 2.0 ** 60, device="cuda"), torch.full((K, n), 2.0 ** 59, device="cuda")
    C = torch.zeros(n, n, device="cuda")
    before = tb.launch_count()
    if precision == "native":
        tb.gemm_bf16(tb.NN, A.bfloat16(), B.bfloat16(), n, n, K, K, n, C32=C, ldc32=n, alpha=2.0 ** -4, splits=8)
    else:
        tb.gemm_f32(tb.NN, A, B, C, n, n, K, K, n, n, alpha=2.0 ** -4, precision={"tf32": tb.PREC_TF32, "fp32": tb.PREC_FP32}[precision])
    tb.sync_check()
    assert tb.launch_count() - before == 1
    assert bool((C == 2.0 ** 125).all())


def test_clusters_keep_to_the_sms_that_are_not_reserved():
    """TB_SM_RESERVE leaves SMs to another library's kernels.  With 40 of them reserved, 15 tiles in clusters of eight do not fit into
    the rest (two launches instead of one), and a float32 product takes no more CTAs than there are SMs left."""
    code = """
import torch
from turkce_llm_b200 import lib as tb
tb.init(0)
left = torch.cuda.get_device_properties(0).multi_processor_count - 40
A, B, C = torch.randn(1920, 2048, device="cuda").bfloat16(), torch.randn(2048, 128, device="cuda").bfloat16(), torch.zeros(1920, 128, device="cuda")
before = tb.launch_count()
tb.gemm_bf16(tb.NN, A, B, 1920, 128, 2048, 2048, 128, C32=C, ldc32=128, splits=8, tile_n=128)
print("launches", tb.launch_count() - before)
tb.profile_begin()
for M, N, K in ((1024, 1152, 384), (1024, 384, 1152), (384, 1152, 1024), (1024, 1024, 1024), (640, 640, 640)):
    x, w, y = torch.randn(M, K, device="cuda"), torch.randn(K, N, device="cuda"), torch.zeros(M, N, device="cuda")
    tb.gemm_f32(tb.NN, x, w, y, M, N, K, K, N, N, precision=tb.PREC_FP32)
for tag in tb.profile_end(torch.cuda.current_stream().cuda_stream):
    if tag.startswith("gemm_x3"):
        _, _, shape, _, s, _, bn = tag.split(":")[:7]
        M, N, K = (int(v) for v in shape.split("x"))
        ctas = -(-M // 128) * -(-N // int(bn[2:])) * int(s[1:])
        print("ctas", tag, ctas)
        assert ctas <= left, tag
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=ROOT, env={**os.environ, "TB_SM_RESERVE": "40"})
    assert r.returncode == 0, r.stderr
    assert "launches 2" in r.stdout and "ctas" in r.stdout, r.stdout


@pytest.mark.parametrize("outputs", ["C16", "both"])
@pytest.mark.parametrize("pad", [0, 3], ids=["by_four", "by_one"])
@pytest.mark.parametrize("shape", [(3, 72, 1024, 8, 64), (16, 136, 1024, 5, 128), (130, 70, 2048, 3, 64), (257, 90, 1024, 2, 128), (129, 388, 1024, 3, 192)])
def test_cluster_sums_of_few_rows_and_bf16_outputs(tb, monkeypatch, shape, pad, outputs):
    """Fewer rows than CTAs, a last tile of one or two rows, bf16 outputs that can and cannot be written four at a time, with bias and
    previous contents: the bits of the reduction kernel, and nothing written past a row's end."""
    M, N, K, splits, bn = shape
    A, B = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(K, (N + 7) // 8 * 8, device="cuda").bfloat16()
    bias, C0 = torch.randn(N, device="cuda"), torch.randn(M, N + pad, device="cuda")
    got = []
    for off in (False, True):
        if off:
            monkeypatch.setenv("TB_GEMM_NO_CLUSTER_SPLIT", "1")
        C, C16 = C0.clone(), C0.bfloat16()
        before = tb.launch_count()
        tb.gemm_bf16(tb.NN, A, B, M, N, K, K, B.shape[1], C32=C if outputs == "both" else None, ldc32=N + pad, C16=C16, ldc16=N + pad, bias=bias,
                     alpha=0.75, beta=0.5, splits=splits, tile_n=bn)
        tb.sync_check()
        assert tb.launch_count() - before == (2 if off else 1)
        assert torch.equal(C[:, N:], C0[:, N:]) and torch.equal(C16[:, N:], C0.bfloat16()[:, N:])
        got.append((C, C16))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    want = 0.75 * (A.double() @ B[:, :N].double()) + bias.double() + (0.5 * C0[:, :N].double() if outputs == "both" else 0.0)
    assert ((got[0][1][:, :N].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * want.abs().max()).all()


def tile_of(tb, call):
    """Tile width, splits and shape that a call's product was launched with, from the profile's tags."""
    tb.profile_begin()
    call()
    tags = [t for t in tb.profile_end(torch.cuda.current_stream().cuda_stream) if t.startswith("gemm_")]
    assert len(tags) == 1, tags
    _, _, shape, _, s, _, bn = tags[0].split(":")[:7]
    return int(bn[2:]), int(s[1:]), tuple(int(v) for v in shape.split("x"))


@pytest.mark.parametrize("M,N,K,wide", [(384, 1152, 8192, False), (384, 696, 12000, False), (384, 1496, 10000, False), (384, 2048, 5000, False),
                                        (384, 2048, 14336, True)])
def test_wide_tiles_of_a_weight_gradient_alone_only_where_they_gain(tb, M, N, K, wide):
    """Float32 operands read as tf32: 384 columns formed the other way round took 1.1 to 1.5 times as long as the usual tile with few
    tiles or a short K, and 0.86 at the last of these shapes."""
    A, B, C = torch.randn(K, M, device="cuda"), torch.randn(K, N, device="cuda"), torch.zeros(M, N, device="cuda")
    bn, _, shape = tile_of(tb, lambda: tb.gemm_f32(tb.TN, A, B, C, M, N, K, M, N, N, beta=1.0, precision=tb.PREC_TF32))
    assert (bn == 384) == wide and shape == ((N, M, K) if wide else (M, N, K))


@pytest.mark.parametrize("beta", [0.0, 1.0])
@pytest.mark.parametrize("M,N", [(300, 1994), (260, 2049), (384, 1802)])
def test_weight_gradient_formed_the_other_way_round(tb, M, N, beta):
    """C^T = B^T A in 384-column tiles, turned back by the reduction: rows and columns that end inside its 32 x 32 blocks, a leading
    dimension beyond the columns, against float64.  Operands are exact in tf32, so what differs is the sum: every addition of eight
    products may lose 2^-23 of the magnitudes."""
    K = 14000
    A, B = torch.randn(K, M, device="cuda").bfloat16().float(), torch.randn(K, N, device="cuda").bfloat16().float()
    C0 = torch.randn(M, N + 5, device="cuda")
    C = C0.clone()
    bn, splits, shape = tile_of(tb, lambda: tb.gemm_f32(tb.TN, A, B, C, M, N, K, M, N, N + 5, beta=beta, precision=tb.PREC_TF32))
    assert bn == 384 and splits > 1 and shape == (N, M, K)
    want = A.double().T @ B.double() + beta * C0[:, :N].double()
    bound = (K / 8 + 4) * 2.0 ** -23 * (A.double().abs().T @ B.double().abs() + beta * C0[:, :N].abs())
    assert bool(((C[:, :N].double() - want).abs() <= bound).all())
    assert torch.equal(C[:, N:], C0[:, N:])


def test_products_that_a_cluster_adds_reserve_no_memory_for_their_parts():
    """The device's scratch memory grows by a device-wide wait and an allocation: not for partial sums that nobody writes."""
    code = """
import torch
from turkce_llm_b200 import lib as tb
tb.init(0)
def product(M, N, K, tf32):
    A, B, C = torch.randn(M, K, device="cuda"), torch.randn(K, N, device="cuda"), torch.zeros(M, N, device="cuda")
    before = tb.launch_count()
    if tf32: tb.gemm_f32(tb.NN, A, B, C, M, N, K, K, N, N, precision=tb.PREC_TF32)
    else: tb.gemm_bf16(tb.NN, A.bfloat16(), B.bfloat16(), M, N, K, K, N, C32=C, ldc32=N, splits=8, tile_n=128)
    tb.sync_check()
    assert tb.launch_count() - before == 1
for tf32 in (False, True):
    M, N, K = (1408, 256, 1024) if tf32 else (640, 384, 4096)
    product(128, 128, 512, tf32)          # the kernel's code and a first scratch allocation
    product(M, N, 64, True)               # torch's own memory (unsplit)
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    product(M, N, K, tf32)
    torch.cuda.empty_cache()
    left = torch.cuda.mem_get_info()[0]
    print("taken", free - left)
    assert free - left < 4 << 20          # slabs of 7.9 and 8.7 MB, and a quarter
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stdout + r.stderr


def test_short_float32_products_of_many_tiles_keep_their_pieces_in_memory(tb):
    """K = 168 on most SMs took 9.7 us split on chip and 9.1 over pieces written out, which run unsplit there; with a longer K or fewer tiles
    the chip is faster."""
    for M, N, K, launches in ((1503, 448, 168, 2), (1774, 568, 168, 2), (1503, 448, 172, 1), (355, 800, 168, 1)):
        A, B, C = torch.randn(M, K, device="cuda"), torch.randn(N, K, device="cuda"), torch.zeros(M, N, device="cuda")
        before = tb.launch_count()
        tb.gemm_f32(tb.NT, A, B, C, M, N, K, K, K, N, precision=tb.PREC_FP32)
        tb.sync_check()
        assert tb.launch_count() - before == launches
        want = A.double() @ B.double().T
        assert bool(((C.double() - want).abs() <= (3 * 2.0 ** -20 + (3 * K / 8 + 4) * 2.0 ** -23) * (A.double().abs() @ B.double().abs().T)).all())
