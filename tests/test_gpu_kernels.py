"""Parity of every CUDA entry point (called through the C ABI) with the oracle and
with the fixtures written by the reference's own code.

Tolerances (from the stated parity bar): packed words and dequantized values
bit-exact; scales exact (<= 1e-3 relative allowed); >= 99.5 % of the int4 codes equal;
Hessian-weighted reconstruction error within 1 % relative.
"""
import os

import numpy as np
import pytest
import torch

from moe_quant_b200 import _lib, ops, synthetic
from moe_quant_b200._lib import MATH_FP32, MATH_TENSOR, MoeQuantError, lib
from oracle import gptq_oracle as O

pytestmark = pytest.mark.gpu

CODE_AGREEMENT = 0.995
SCALE_RTOL = 1e-3
RECON_RTOL = 0.01


@pytest.fixture(params=["fp32", "tensor"])
def precision(request):
    math = MATH_FP32 if request.param == "fp32" else MATH_TENSOR
    return ops.Precision(math=math, split_hessian=3, split_hinv=3, split_sweep=3)


# ------------------------------------------------------------------ packing
def test_pack_golden_vectors(cuda):
    z = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "pack_int4.npz"))
    for key in z.files:
        if key.startswith("v_"):
            v = torch.from_numpy(z[key])
            got = ops.pack_int4((v + 8).to(torch.uint8).to(cuda)).cpu()
            assert torch.equal(got, torch.from_numpy(z["p_" + key[2:]])), key


@pytest.mark.parametrize("shape", [(1, 16), (7, 2048), (33, 264), (5, 13), (128, 7168), (3, 1), (0, 64), (4, 0)])
def test_pack_random_shapes(cuda, shape):
    g = torch.Generator().manual_seed(shape[0] * 131 + shape[1])
    codes = torch.randint(0, 16, shape, generator=g, dtype=torch.uint8)
    got = ops.pack_int4(codes.to(cuda)).cpu()
    want = O.pack_to_int32(codes.to(torch.int8) - 8, 4) if codes.numel() else torch.empty(shape[0], (shape[1] + 7) // 8, dtype=torch.int32)
    assert got.shape == want.shape and torch.equal(got, want)


def test_pack_with_zero_points(cuda):
    g = torch.Generator().manual_seed(5)
    codes = torch.randint(0, 16, (9, 64), generator=g, dtype=torch.uint8)
    zero = torch.randint(6, 10, (9, 2), generator=g, dtype=torch.int8)
    shifted = codes.to(torch.int8) - zero.repeat_interleave(32, dim=-1)
    shifted = shifted.clamp(-8, 7)
    codes = (shifted + zero.repeat_interleave(32, dim=-1)).to(torch.uint8)
    got = ops.pack_int4(codes.to(cuda), zero.to(cuda), 32).cpu()
    assert torch.equal(got, O.pack_to_int32(shifted, 4))


def test_pack_unpack_round_trip_full_size(cuda):
    """Property at the full down_proj size: unpacking the words gives the codes back."""
    g = torch.Generator(device="cuda").manual_seed(1)
    codes = torch.randint(0, 16, (7168, 2048), generator=g, dtype=torch.uint8, device=cuda)
    words = ops.pack_int4(codes)
    shifts = torch.arange(8, device=cuda, dtype=torch.int32) * 4
    back = ((words.unsqueeze(-1) >> shifts) & 0xF).reshape(7168, 2048).to(torch.uint8)
    assert torch.equal(back, codes)


def test_pack_golden_layers(cuda, golden):
    got = ops.pack_int4(golden.t("qweight").to(cuda)).cpu()
    assert torch.equal(got, golden.t("weight_packed"))


# ------------------------------------------------------------------ dequantize
def test_dequantize_golden(cuda, golden):
    q = golden.t("qweight").to(cuda)
    s = golden.t("scale", typed=True).to(cuda)
    zr = golden.t("zero", typed=True).to(cuda)
    got = ops.dequantize(q, s, zr, golden.group, 4, golden.dtype).cpu()
    assert torch.equal(got.float(), golden.t("dequantized", typed=True).float())
    got2 = ops.dequantize(q, s, None, golden.group, 4, golden.dtype).cpu()
    assert torch.equal(got2.float(), got.float())


def test_relative_error_golden(cuda, golden, precision):
    """get_relative_mse_error on the engine against the number the reference's own function
    returned for the fixture (src/quant_utils.py:259-264)."""
    from moe_quant_b200 import quant_utils
    ops.set_default_precision(precision)
    try:
        deq = golden.t("dequantized", typed=True).float().to(cuda)
        rel = quant_utils.get_relative_mse_error(deq, golden.W.float().to(cuda), golden.t("H_damped").to(cuda))
    finally:
        ops.set_default_precision(ops.Precision())
    want = float(golden.t("rel_error"))
    assert rel.dtype == torch.float32 and rel.dim() == 0
    assert abs(float(rel) - want) <= 2e-4 * want
    plain = quant_utils.get_relative_mse_error(deq, golden.W.float().to(cuda))
    d = deq.cpu() - golden.W.float()
    assert abs(float(plain) - float(d.pow(2).mean() / golden.W.float().pow(2).mean())) <= 1e-5 * float(plain)


# ------------------------------------------------------------------ Hessian
def test_hessian_accum_golden(cuda, golden, precision):
    C = golden.W.shape[1]
    H = torch.zeros(C, C, dtype=torch.float32, device=cuda)
    n = 0
    for k, x in enumerate(golden.batches):
        m = x.shape[0]
        ops.hessian_accum(H, x.to(cuda), n / (n + m), 2.0 / (n + m), precision)
        n += m
        if k == 0 and len(golden.batches) > 1:
            torch.testing.assert_close(H.cpu(), golden.t("H_after0"), rtol=2e-5, atol=1e-5)
    Hc = H.cpu()
    torch.testing.assert_close(Hc, golden.t("H_final"), rtol=2e-5, atol=1e-5)
    assert torch.equal(Hc, Hc.t()), "both triangles must hold the same numbers"


@pytest.mark.parametrize("m,C,dtype", [(1, 128, torch.float32), (37, 256, torch.bfloat16), (513, 384, torch.float16),
                                       (1000, 1024, torch.bfloat16), (300, 2048, torch.float32), (0, 128, torch.bfloat16)])
def test_hessian_accum_ragged(cuda, precision, m, C, dtype):
    x = synthetic.activations(max(m, 1), C, 3, dtype)[:m]
    H0 = synthetic.layer_weight(C, C, 9)
    H0 = (H0 + H0.t()).contiguous()
    H = H0.clone().to(cuda)
    ops.hessian_accum(H, x.to(cuda), 0.25, 0.5, precision)
    want = 0.25 * H0.double() + 0.5 * (x.double().t() @ x.double())
    err = (H.cpu().double() - want).abs().max() / want.abs().max()
    assert float(err) < 5e-6   # tensor-core fp32 accumulation truncates; fp32 FMA path reaches ~3e-7


@pytest.mark.parametrize("pad,offset", [(8, 0), (3, 0), (8, 1), (10, 2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_hessian_accum_activation_views(cuda, dtype, pad, offset):
    """16-bit activations are read in place through a tensor map when their rows are 16-byte
    aligned (pad 8, offset 0); a row stride that is not a multiple of 8 elements or a start that is
    not 16-byte aligned goes through the transposed copy.  Both must give the same Hessian, with
    ragged token and channel counts."""
    m, C = 333, 1000
    g = torch.Generator().manual_seed(17)
    big = torch.randn(m, C + pad + offset, generator=g).to(dtype)
    xd = big.to(cuda)[:, offset:offset + C]
    assert xd.stride(0) == C + pad + offset and xd.stride(1) == 1
    H0 = synthetic.layer_weight(C, C, 5)
    H0 = (H0 + H0.t()).contiguous()
    H = H0.clone().to(cuda)
    ops.hessian_accum(H, xd, 0.75, 2.0 / m, ops.Precision(math=MATH_TENSOR))
    x = big[:, offset:offset + C].double()
    want = 0.75 * H0.double() + (2.0 / m) * (x.t() @ x)
    Hc = H.cpu()
    assert float((Hc.double() - want).abs().max() / want.abs().max()) < 5e-6
    assert torch.equal(Hc, Hc.t())


@pytest.mark.parametrize("C", [8, 129, 250, 256, 1000, 1031])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_hessian_accum_first_batch_reads_nothing(cuda, precision, C, dtype):
    """With beta = 0 every element of both triangles is written and none is read: a handle's first batch goes into memory as the
    allocator gives it.  Every route: rows read in place, the transposed copy, planes of fp32, the CUDA cores."""
    for m in (1, 37, 333):
        for offset in (0, 1):
            gen = torch.Generator().manual_seed(100 * m + offset)
            big = torch.randn(m, C + 8, generator=gen).to(dtype)
            H = torch.full((C, C), float("nan"), device=cuda)
            ops.hessian_accum(H, big.to(cuda)[:, offset : offset + C], 0.0, 2.0 / m, precision)
            x = big[:, offset : offset + C].double()
            want = (2.0 / m) * (x.t() @ x)
            got = H.cpu()
            assert float((got.double() - want).abs().max() / want.abs().max()) < 5e-6
            assert torch.equal(got, got.t())


@pytest.mark.parametrize("C,pad", [(256, 0), (264, 8), (3335, 9), (3336, 0)])
@pytest.mark.parametrize("m", [1, 320, 1100])
@pytest.mark.parametrize("beta", [0.0, 0.25])
def test_hessian_accum_in_tile_pairs(cuda, C, pad, m, beta):
    """One tile, a ragged last tile, rows of the Hessian that are not 16-byte aligned, and 105 tiles for 74 pairs of CTAs with one,
    five and eighteen slabs of tokens for a ring of six.  fp32 sums of m products: 2^-24 m of the sum of their sizes at most."""
    gen = torch.Generator().manual_seed(C + m)
    big = torch.randn(m, C + pad, generator=gen).to(torch.bfloat16)
    H0 = torch.randn(C, C, generator=gen)
    H0 = H0 + H0.t()
    H = H0.to(cuda) if beta else torch.full((C, C), float("nan"), device=cuda)
    ops.hessian_accum(H, big.to(cuda)[:, :C], beta, 0.5)
    x = big[:, :C].to(cuda).double()
    want, size = 0.5 * (x.t() @ x), 0.5 * (x.abs().t() @ x.abs())
    if beta:
        want, size = want + beta * H0.to(cuda).double(), size + beta * H0.to(cuda).double().abs()
    assert bool(((H.double() - want).abs() <= 2.0 ** -24 * (m + 3) * size).all())
    assert torch.equal(H, H.t())


# ------------------------------------------------------------------ prepare
def test_prepare_golden(cuda, golden):
    H = golden.t("H_final").clone().to(cuda)
    W = golden.W.float().to(cuda)
    flags = ops.hessian_prepare(H, W, 1e-2).cpu().tolist()
    torch.testing.assert_close(H.cpu(), golden.t("H_damped"), rtol=1e-6, atol=1e-7)
    dead = len(golden.meta.get("dead", ()))
    zero_w = len(golden.meta.get("zero_w", ()))
    assert flags == [0, dead, dead + zero_w, 0]
    for j in golden.meta.get("dead", ()):
        assert float(W[:, j].abs().max()) == 0.0


def test_prepare_nan_hessian_becomes_identity(cuda):
    H = torch.eye(64, device=cuda) * 3
    H[5, 7] = float("nan")
    flags = ops.hessian_prepare(H, None, 0.5).cpu().tolist()
    assert flags[0] == 1
    torch.testing.assert_close(H.cpu(), torch.eye(64) * 1.5)


# ------------------------------------------------------------------ scales
def test_scales_golden(cuda, golden):
    _, Wf, _, _ = O.pre_step(golden.t("H_final").clone(), golden.W)
    got = ops.absmax_scales(Wf.to(cuda), golden.group, 4, golden.dtype).cpu()
    assert torch.equal(got, golden.t("scale", typed=True).float())


@pytest.mark.parametrize("g", [4, 8, 32, 64, 128, 256, 1024])
def test_scales_group_sizes(cuda, g):
    W = synthetic.layer_weight(19, 1024, 4)
    for dt in (torch.float32, torch.bfloat16, torch.float16):
        want, _, _ = O.symmetric_grid(W, g, 4, dt)
        got = ops.absmax_scales(W.to(cuda), g, 4, dt).cpu()
        assert torch.equal(got, want)


# ------------------------------------------------------------------ Hessian inverse factor
def test_hinv_golden(cuda, golden, precision):
    U, flags, _ = ops.hinv_upper(golden.t("H_damped").clone().to(cuda), precision)
    assert flags.cpu().tolist()[3] == 0
    Uc = U.cpu()
    assert float(Uc.tril(-1).abs().max()) == 0.0
    assert torch.equal(Uc.diag(), torch.ones(Uc.shape[0]))
    torch.testing.assert_close(Uc, golden.t("Uhat"), rtol=2e-3, atol=2e-5)


@pytest.mark.parametrize("C", [128, 136, 640, 1000, 1536])
def test_hinv_sizes(cuda, precision, C):
    x = synthetic.activations(C // 2 + 11, C, 21)
    H, _ = O.hessian_update(None, 0, x)
    W = synthetic.layer_weight(8, C, 2)
    want, failed = O.hessian_inverse(H, W, 1e-2)  # damps H in place
    assert not failed
    U, flags, _ = ops.hinv_upper(H.clone().to(cuda), precision)
    assert flags.cpu().tolist()[3] == 0
    rel = (U.cpu() - want).norm() / want.norm()
    assert float(rel) < 2e-4


def test_hinv_not_positive_definite_gives_identity(cuda, precision):
    H = torch.eye(256)
    H[200, 200] = -1.0
    U, flags, _ = ops.hinv_upper(H.to(cuda), precision)
    assert flags.cpu().tolist()[3] == 201
    assert torch.equal(U.cpu(), torch.eye(256))


def test_inv_sym_seam(cuda, precision):
    from moe_quant_b200 import linalg_utils
    x = synthetic.activations(400, 256, 8)
    H, _ = O.hessian_update(None, 0, x)
    H += 0.1 * torch.eye(256)
    got = linalg_utils.inv_sym(H.to(cuda), precision).cpu().double()
    eye = got @ H.double()
    assert float((eye - torch.eye(256, dtype=torch.float64)).abs().max()) < 5e-3


# ------------------------------------------------------------------ sweep
def _grid(golden):
    _, Wf, _, _ = O.pre_step(golden.t("H_final").clone(), golden.W)
    scale, _, _ = O.symmetric_grid(Wf, golden.group, 4, golden.dtype)
    return Wf, scale


def test_sweep_with_reference_factor(cuda, golden, precision):
    Wf, scale = _grid(golden)
    R, C = Wf.shape
    codes, deq = ops.gptq_sweep(Wf.to(cuda), golden.t("Uhat").to(cuda), scale.to(cuda), None, golden.group,
                                C // golden.group, 1, 4, golden.dtype, True, precision)
    assert O.code_agreement(codes.cpu(), golden.t("qweight")) >= 0.999
    want = O.dequantize_linear_weight(codes.cpu(), golden.t("scale", typed=True), golden.t("zero", typed=True))
    assert torch.equal(deq.cpu().float(), want.float())


def test_gptq_loop_seam(cuda, golden, precision):
    """The reference's inner seam: transposed weight, per-element scale and zero."""
    from moe_quant_b200 import gptq_loop
    ops.set_default_precision(precision)
    try:
        Wf, scale = _grid(golden)
        g = golden.group
        sf = scale.repeat_interleave(g, -1)
        zf = torch.full_like(sf, 8.0)
        wt = Wf.t().contiguous().to(cuda)
        q = gptq_loop.gptq_loop(wt, golden.t("Uhat").to(cuda), sf.t().contiguous().to(cuda), zf.t().contiguous().to(cuda),
                                torch.tensor(15.0, device=cuda), golden.dtype, 128)
    finally:
        ops.set_default_precision(ops.Precision())
    assert q.shape == wt.shape and q.dtype == torch.float32
    codes = q.t().contiguous().to(torch.uint8).cpu()
    assert O.code_agreement(codes, golden.t("qweight")) >= 0.999
    deq = O.dequantize_linear_weight(codes, golden.t("scale", typed=True), golden.t("zero", typed=True))
    assert torch.equal(wt.t().cpu().to(golden.dtype).float(), deq.float())


# ------------------------------------------------------------------ argument errors (no fallback, loud failures)
def test_cpu_tensor_is_rejected():
    with pytest.raises(MoeQuantError):
        ops.pack_int4(torch.zeros(4, 8, dtype=torch.uint8))


def test_bad_group_is_rejected(cuda):
    with pytest.raises(MoeQuantError):
        ops.absmax_scales(torch.zeros(4, 96, device=cuda), 64, 4, torch.float32)


# ------------------------------------------------------------------ the GEMM engine alone, against torch fp32
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (128, 128, 64), (130, 257, 128), (300, 1000, 100), (2048, 640, 128),
                                   (257, 129, 1000), (512, 512, 4096)])
@pytest.mark.parametrize("layout", ["nn", "tn", "nt"])
def test_gemm_engine_against_torch(cuda, precision, M, N, K, layout):
    g = torch.Generator().manual_seed(M * 7 + N * 3 + K)
    A = torch.randn(M, K, generator=g)
    B = torch.randn(K, N, generator=g)
    C0 = torch.randn(M, N, generator=g)
    Ad = A.to(cuda) if layout != "tn" else A.t().contiguous().to(cuda).t()     # column-major A
    Bd = B.to(cuda) if layout != "nt" else B.t().contiguous().to(cuda).t()     # column-major B
    Cd = C0.clone().to(cuda)
    ops.gemm(Ad, Bd, Cd, alpha=-0.5, beta=1.0, precision=precision)
    want = C0.double() - 0.5 * (A.double() @ B.double())
    err = float((Cd.cpu().double() - want).abs().max() / want.abs().max())
    # the tensor pipe truncates when it aligns addends, so its error grows ~linearly with K;
    # fp32 FMAs round to nearest and stay near sqrt(K) * 6e-8
    tol = 5e-6 * max(1.0, K / 256.0) if precision.math == MATH_TENSOR else 5e-6
    assert err < tol, f"relative error {err:.3e} (tolerance {tol:.1e})"


def test_gemm_engine_two_plane_split_is_coarser_but_close(cuda):
    g = torch.Generator().manual_seed(9)
    A, B = torch.randn(256, 128, generator=g), torch.randn(128, 384, generator=g)
    want = A.double() @ B.double()
    errs = {}
    for split in (1, 2, 3):
        C = torch.zeros(256, 384, device=cuda)
        ops.gemm(A.to(cuda), B.to(cuda), C, precision=ops.Precision(math=MATH_TENSOR), split=split)
        errs[split] = float((C.cpu().double() - want).abs().max() / want.abs().max())
    assert errs[1] < 2e-2 and errs[2] < 1e-4 and errs[3] < 5e-6
    assert errs[3] < errs[2] < errs[1]


def test_gemm_engine_upper_tiles_only(cuda, precision):
    g = torch.Generator().manual_seed(4)
    P = torch.randn(640, 128, generator=g)
    C0 = torch.randn(640, 640, generator=g)
    Cd = C0.clone().to(cuda)
    Pd = P.to(cuda)
    ops.gemm(Pd, Pd.t(), Cd, alpha=-1.0, beta=1.0, upper_tiles_only=True, precision=precision)
    want = C0.double() - P.double() @ P.double().t()
    got = Cd.cpu().double()
    blocks = torch.arange(640) // 128
    upper = blocks[:, None] <= blocks[None, :]
    assert float((got - want)[upper].abs().max() / want.abs().max()) < 5e-6
    assert torch.equal(got[~upper], C0.double()[~upper]), "tiles below the diagonal must not be touched"


@pytest.mark.parametrize("beta", [0.0, 1.0, 0.5])
@pytest.mark.parametrize("upper,N", [(False, 2780), (False, 2777), (True, 3304)])
@pytest.mark.parametrize("deep", [False, True])
def test_gemm_engine_rank128_update_many_tiles(cuda, beta, upper, N, deep):
    """Rank-128 updates with at least two tiles per SM leave through the TMA unit (store for
    beta 0, add at the L2 for beta 1); any other beta, or fewer tiles, goes through the warps'
    own loads and stores, and so does an N that is not a multiple of 4.  Ragged edges (M, N not
    multiples of the 32-wide boxes) and a C that is a window of a wider matrix must not touch
    anything outside the window.  `deep`: the same with 512 (and a ragged 300) contraction
    columns, the persistent streaming kernel that the two-level updates of the factorisation
    and of the sweep use."""
    M, K = (N, 128) if upper else (2500, 100)
    if deep:
        K = 512 if upper else 300
    g = torch.Generator().manual_seed(11)
    A, B = torch.randn(M, K, generator=g), torch.randn(K, N, generator=g)
    if upper:
        B = A.t().clone()
    big = torch.randn(M + 3, (N + 43) // 4 * 4, generator=g)   # row stride is a multiple of 4 floats
    big_d = big.clone().to(cuda)
    Cd = big_d[2:2 + M, 8:8 + N]                      # 16-byte aligned window of a wider matrix
    ops.gemm(A.to(cuda), B.to(cuda), Cd, alpha=-1.0, beta=beta, upper_tiles_only=upper,
             precision=ops.Precision(math=MATH_TENSOR))
    want = beta * big[2:2 + M, 8:8 + N].double() - A.double() @ B.double()
    got = big_d.cpu()
    win = got[2:2 + M, 8:8 + N].double()
    mask = torch.ones(M, N, dtype=torch.bool)
    if upper:
        blocks_m, blocks_n = torch.arange(M) // 128, torch.arange(N) // 128
        mask = blocks_m[:, None] <= blocks_n[None, :]
        assert torch.equal(win[~mask], big[2:2 + M, 8:8 + N].double()[~mask])
    assert float((win - want)[mask].abs().max() / want.abs().max()) < 5e-6
    outside = torch.ones_like(big, dtype=torch.bool)
    outside[2:2 + M, 8:8 + N] = False
    assert torch.equal(got[outside], big[outside]), "elements outside the C window were modified"


@pytest.mark.parametrize("M,N,K,upper", [(300, 1000, 200, False), (2048, 256, 96, True), (2048, 256, 300, True), (1000, 1000, 64, True),
                                         (129, 257, 1000, False), (4000, 4000, 130, True), (1500, 1500, 4096, True)])
def test_gemm_engine_one_plane_persistent(cuda, M, N, K, upper):
    """One bf16 plane and N >= 256: the persistent kernel (one CTA per SM walking 128 x 256 tiles).
    Inputs are bf16-representable, so one plane is exact and the result must agree with float64 to
    accumulation error; tiles below the diagonal stay untouched with upper_tiles_only, also when the
    matrix has more rows than columns."""
    g = torch.Generator().manual_seed(M + N + K)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16).float()
    B = torch.randn(K, N, generator=g).to(torch.bfloat16).float()
    C0 = torch.randn(M, N, generator=g)
    Cd = C0.clone().to(cuda)
    ops.gemm(A.to(cuda), B.to(cuda), Cd, alpha=0.5, beta=-1.0, upper_tiles_only=upper,
             precision=ops.Precision(math=MATH_TENSOR), split=1)
    want = 0.5 * (A.double() @ B.double()) - C0.double()
    got = Cd.cpu().double()
    must = torch.ones(M, N, dtype=torch.bool)
    if upper:
        # guaranteed: every 128-block on or above the diagonal is computed; nothing below the
        # diagonal's 256-wide tile is touched (K <= 128 runs in the 128 x 128 panel kernel, larger
        # K in 128 x 256 tiles, and what lies between the two tilings may be either)
        must = (torch.arange(N)[None, :] // 128) >= (torch.arange(M)[:, None] // 128)
        never = ((torch.arange(N)[None, :] // 256) * 256 + 256) <= ((torch.arange(M)[:, None] // 128) * 128)
        assert torch.equal(got[never], C0.double()[never])
    assert float((got - want)[must].abs().max() / want.abs().max()) < 5e-6 * max(1.0, K / 256.0)


# ------------------------------------------------------------------ inverse-free form of the sweep
def test_unit_factor_is_inverse_of_reference_factor(cuda, golden, precision):
    H = golden.t("H_damped").clone().to(cuda)
    flags, diag = ops.chol_unit_factor(H, precision)
    assert flags.cpu().tolist()[3] == 0
    Ut = H.cpu().double()
    assert float(Ut.tril(-1).abs().max()) == 0.0 and torch.equal(Ut.diag(), torch.ones(Ut.shape[0], dtype=torch.float64))
    eye = Ut @ golden.t("Uhat").double()
    assert float((eye - torch.eye(Ut.shape[0], dtype=torch.float64)).abs().max()) < 2e-3
    # diag(T)^2 reproduces the pivots: H = Utilde diag(T)^2 Utilde^T
    back = (Ut * diag.cpu().double()[None, :] ** 2) @ Ut.t()
    Hd = golden.t("H_damped").double()
    assert float((back - Hd).abs().max() / Hd.abs().max()) < 1e-5


def test_sweep_inverse_free_form_matches_reference_codes(cuda, golden, precision):
    Wf, scale = _grid(golden)
    R, C = Wf.shape
    Ut = torch.linalg.inv(golden.t("Uhat").double()).float().contiguous()
    codes, deq = ops.gptq_sweep(Wf.clone().to(cuda), Ut.to(cuda), scale.to(cuda), None, golden.group, C // golden.group, 1,
                                4, golden.dtype, True, precision, W_original=Wf.to(cuda))
    assert O.code_agreement(codes.cpu(), golden.t("qweight")) >= 0.999
    want = O.dequantize_linear_weight(codes.cpu(), golden.t("scale", typed=True), golden.t("zero", typed=True))
    assert torch.equal(deq.cpu().float(), want.float())


@pytest.mark.parametrize("R,C,g", [(1, 8, 8), (3, 40, 8), (5, 24, 12), (7, 1056, 1056), (33, 2048, 64), (2, 28, 4), (130, 4096, 128)])
@pytest.mark.parametrize("out", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("held", [torch.bfloat16, torch.float16, torch.float32, torch.float64])
def test_dequantize_every_type_and_group(cuda, R, C, g, out, held):
    """Vector and element paths, scales held in the layer's type or another one: bit-exact."""
    gen = torch.Generator().manual_seed(R * 7 + C + g)
    codes = torch.randint(0, 256, (R, C), generator=gen, dtype=torch.uint8)
    scale = (torch.rand(R, C // g, generator=gen) * 0.01 + 1e-3).to(held)
    zero = torch.randint(0, 16, (R, C // g), generator=gen).to(held)
    wide_s, wide_z = (t.float().repeat_interleave(g, -1) for t in (scale, zero))
    for z, zf in ((zero, wide_z), (None, 8.0), (zero.to(torch.int32), wide_z)):
        got = ops.dequantize(codes.to(cuda), scale.to(cuda), None if z is None else z.to(cuda), g, 4, out).cpu()
        assert torch.equal(got, ((codes.float() - zf) * wide_s).to(out))


# ------------------------------------------------------------------ operand pairs of the factorisation and the sweep
@pytest.mark.parametrize("C,tokens,spread", [(8, 40, 1.0), (128, 200, 1.0), (136, 300, 1.0), (520, 700, 1.0), (640, 640, 2.0), (1032, 1500, 1.0),
                                             (1544, 2000, 3.0)])
@pytest.mark.parametrize("units", [1.0, 1e-12, 1e10])
def test_factor_of_operand_pairs_against_fp64(cuda, C, tokens, spread, units):
    """Super-panel edges (512), ragged last panels, channels whose scales spread over decades and
    Hessians far from 1: the factor is as close to fp64 as the one of the fp32 CUDA cores, whose error is the
    rounding of the same sums (2x: another order of additions)."""
    gen = torch.Generator().manual_seed(C)
    X = torch.randn(tokens, C, generator=gen, dtype=torch.float64) * torch.exp(spread * torch.randn(C, generator=gen, dtype=torch.float64))
    H = X.T @ X * (units / tokens)
    H.diagonal().add_(0.01 * H.diagonal().mean())
    H32 = H.float()
    T = torch.linalg.cholesky(H32.double().flip(0, 1)).flip(0, 1)
    U64 = T / T.diagonal()[None, :]

    def error(math):
        U = H32.to(cuda)
        flags, diag = ops.chol_unit_factor(U, ops.Precision(math=math))
        assert int(flags[3]) == 0
        e = ((U.cpu().double() - U64).norm(dim=0) / U64.norm(dim=0)).norm()
        return float(e), float(((diag.cpu().double() - T.diagonal()) / T.diagonal()).abs().max())

    got, ref = error(MATH_TENSOR), error(MATH_FP32)
    assert got[0] <= 2 * ref[0] + 1e-6 and got[1] <= 2 * ref[1] + 1e-6


@pytest.mark.parametrize("R,C,g,dtype", [(1, 648, 8, torch.bfloat16), (129, 1032, 24, torch.float16), (257, 1664, 128, torch.bfloat16),
                                         (300, 776, 97 * 8, torch.float32), (40, 1280, 64, torch.bfloat16)])
@pytest.mark.parametrize("size", [1.0, 1e-6, 1e3])
def test_sweep_of_operand_pairs_against_fp32_math(cuda, R, C, g, dtype, size):
    """Deep updates whose last 256 x 256 tile is ragged in rows and columns, rows of very different size,
    a row of zeros: the codes of the fp32 CUDA cores."""
    if dtype == torch.float16 and size < 1:
        size = 1e-2     # the scales must be representable
    W = synthetic.layer_weight(R, C, 5, torch.float32) * size
    W[::3] *= 0.125
    if R > 2:
        W[2] = 0.0
    W = W.to(dtype)
    X = synthetic.activations(2 * C, C, 6, torch.bfloat16).float()
    H = X.T @ X / C

    def run(math):
        p = ops.Precision(math=math)
        codes, scales, _, flags = ops.quantize_layer([W.to(cuda)], H.to(cuda), g, 4, 1e-2, precision=p)
        assert int(flags[3]) == 0
        return codes[0].cpu(), scales[0].cpu()

    (q, s), (q0, s0) = run(MATH_TENSOR), run(MATH_FP32)
    assert torch.equal(s, s0)
    assert O.code_agreement(q, q0) >= CODE_AGREEMENT


@pytest.mark.parametrize("C,g", [(136, 8), (648, 8), (1280, 32), (1664, 128)])
@pytest.mark.parametrize("kind", ["plain", "small_first", "big_first", "by_group"])
@pytest.mark.parametrize("split", [3, 4])
def test_sweep_running_values_against_fp64(cuda, C, g, kind, split):
    """What every column has received from the tiles in front of it, against fp64 sums over the same errors, for rows whose
    groups differ by up to 2^28.  Bound per element: products of pairs 2^-22 (lo lo left out) + 2 * 2^-23, the tensor
    core's truncations four times 2^-23 of a part of the sum: 2^-20 of the sum of absolute products; and one fp32
    rounding of the running value per update."""
    R = 40
    W = synthetic.layer_weight(R, C, 5, torch.float32)
    gen = torch.Generator().manual_seed(C + g)
    if kind == "small_first":
        W[:, : C // 2] *= 2.0 ** -28
    elif kind == "big_first":
        W[:, C // 2 :] *= 2.0 ** -28
    elif kind == "by_group":
        W *= torch.exp2(-torch.randint(0, 21, (R, C // g), generator=gen).float()).repeat_interleave(g, -1)
    X = synthetic.activations(2 * C, C, 6, torch.bfloat16).double()
    H = X.T @ X / C
    H.diagonal().add_(0.01 * H.diagonal().mean())
    T = torch.linalg.cholesky(H.flip(0, 1)).flip(0, 1)
    U = (T / T.diagonal()[None, :]).float().contiguous()
    w, run = W.to(cuda), W.to(cuda)
    scale = ops.absmax_scales(w, g, 4, torch.float32)
    _, deq = ops.gptq_sweep(run, U.to(cuda), scale, None, g, C // g, 1, 4, torch.float32, True, ops.Precision(split_sweep=split), W_original=w)
    E, U64 = (W - deq.cpu()).double(), U.double()
    for j in range(128, C, 128):
        e, u = E[:, :j], U64[:j, j : j + 128]
        size = e.abs() @ u.abs()
        want = W[:, j : j + 128].double() + e @ u
        got = run[:, j : j + 128].cpu().double()
        bound = 2.0 ** -20 * size + (C // 128 + 3) * 2.0 ** -24 * (W[:, j : j + 128].abs().double() + size)
        assert bool(((got - want).abs() <= bound).all()), float(((got - want).abs() / bound).max())


@pytest.mark.parametrize("R,C", [(2600, 2600), (7000, 1800), (1024, 5640), (576, 7176)])
def test_sweep_running_values_where_super_blocks_go_together(cuda, R, C):
    """As above, with enough tiles that two super-blocks of 512 columns share an update (and a last one that does not): tile by tile,
    and by launches of 512 columns (up to 1024 rows)."""
    g = 8
    W = synthetic.layer_weight(R, C, 5, torch.float32).to(cuda)
    X = synthetic.activations(2 * C, C, 6, torch.bfloat16).to(cuda).double()
    H = X.T @ X / C
    H.diagonal().add_(0.01 * H.diagonal().mean())
    T = torch.linalg.cholesky(H.flip(0, 1)).flip(0, 1)
    U = (T / T.diagonal()[None, :]).float().contiguous()
    run = W.clone()
    scale = ops.absmax_scales(W, g, 4, torch.float32)
    _, deq = ops.gptq_sweep(run, U, scale, None, g, C // g, 1, 4, torch.float32, True, ops.Precision(), W_original=W)
    E, U64 = (W - deq).double(), U.double()
    for j in range(128, C, 128):
        e, u = E[:, :j], U64[:j, j : j + 128]
        size = e.abs() @ u.abs()
        want = W[:, j : j + 128].double() + e @ u
        bound = 2.0 ** -20 * size + (C // 128 + 3) * 2.0 ** -24 * (W[:, j : j + 128].abs().double() + size)
        assert bool(((run[:, j : j + 128].double() - want).abs() <= bound).all()), j


@pytest.mark.parametrize("C", [3592, 4104, 5640])
def test_factor_where_super_panels_go_together(cuda, C):
    """Updates 1024 columns deep, of as many tokens as columns, against those of 512 and fp64: the sums of 64 of k are the same, and one rounding
    of the trailing matrix less counts for more than the longer sums do (0.989 to 0.999 of the error, seed by seed, from 4104 columns on)."""
    gen = torch.Generator(device=cuda).manual_seed(C)
    X = torch.randn(C, C, generator=gen, device=cuda, dtype=torch.float64) * torch.exp(torch.randn(C, generator=gen, device=cuda, dtype=torch.float64))
    H = X.T @ X * (2.0 / C)
    H.diagonal().add_(0.01 * H.diagonal().mean())
    H = H.float()
    T = torch.linalg.cholesky(H.double().flip(0, 1)).flip(0, 1)
    U64 = T / T.diagonal()[None, :]

    def error(many_tokens):
        U = H.clone()
        flags, _ = ops.chol_unit_factor(U, ops.Precision(many_tokens=many_tokens))
        assert int(flags[3]) == 0 and not bool(torch.tril(U, -1).any())
        return float((U.double() - U64).norm() / torch.triu(U64, 1).norm())

    assert error(True) < error(False) < 1e-6


def test_updates_go_deeper_only_for_many_tokens(cuda):
    """Of 4104 columns, 700 tokens: the last 3080 columns of the factor are those of the trailing block by itself, which has too few tiles for
    deeper updates, bit for bit.  A caller that gives H of as many tokens as columns may say so, and gets other sums."""
    C, k = 4104, 1024
    X = torch.randn(700, C, generator=torch.Generator(device=cuda).manual_seed(1), device=cuda)
    H = X.T @ X / 700
    H.diagonal().add_(0.01 * H.diagonal().mean())

    def factor(A, **kw):
        A = A.clone().contiguous()
        ops.chol_unit_factor(A, ops.Precision(split_hinv=3, **kw))
        return A

    trailing = factor(H[k:, k:])
    assert torch.equal(factor(H)[k:, k:], trailing)
    assert not torch.equal(factor(H, many_tokens=True)[k:, k:], trailing)
    assert torch.equal(factor(H[k:, k:], many_tokens=True), trailing)


@pytest.mark.parametrize("C,tokens", [(648, 110), (1024, 174), (1544, 260)])
def test_all_products_where_the_sums_cancel(cuda, C, tokens):
    """A Hessian of few tokens: the product of the low pieces takes error off the factor (its 2^-22 per product is most of
    what a pair loses; the mean of eight seeds differs by several per cent), and the explicit inverse has it by itself.
    Up to 512 columns there are no pairs and the two are the same bits."""
    def errors(split, seed):
        gen = torch.Generator().manual_seed(seed)
        X = torch.randn(tokens, C, generator=gen, dtype=torch.float64) * torch.exp(torch.randn(C, generator=gen, dtype=torch.float64))
        H = X.T @ X * (2.0 / tokens)
        H.diagonal().add_(0.01 * H.diagonal().mean())
        H = H.float()
        T = torch.linalg.cholesky(H.double().flip(0, 1)).flip(0, 1)
        U64 = T / T.diagonal()[None, :]
        U = H.to(cuda)
        flags, _ = ops.chol_unit_factor(U, ops.Precision(split_hinv=split))
        assert int(flags[3]) == 0
        return float((U.cpu().double() - U64).norm() / torch.triu(U64, 1).norm())

    three, four = (sum(errors(split, seed) for seed in range(8)) for split in (3, 4))
    assert four < 0.99 * three

    X = torch.randn(2 * C, C, generator=torch.Generator().manual_seed(C))
    H = (X.T @ X / C).to(cuda)
    assert torch.equal(ops.hinv_upper(H.clone(), ops.Precision(split_hinv=3))[0], ops.hinv_upper(H.clone(), ops.Precision(split_hinv=4))[0])
    narrow = [H[:512, :512].clone() for _ in range(2)]
    for U, split in zip(narrow, (3, 4)):
        ops.chol_unit_factor(U, ops.Precision(split_hinv=split))
    assert torch.equal(*narrow)


@pytest.mark.parametrize("C,tokens", [(520, 88), (1032, 1032)])
def test_factor_takes_all_products_unless_told(cuda, C, tokens):
    X = torch.randn(tokens, C, generator=torch.Generator().manual_seed(C))
    H = X.T @ X / tokens
    H.diagonal().add_(0.01 * H.diagonal().mean())
    own, four, three = (H.to(cuda) for _ in range(3))
    ops.chol_unit_factor(own)
    ops.chol_unit_factor(four, ops.Precision(split_hinv=4))
    ops.chol_unit_factor(three, ops.Precision(split_hinv=3))
    assert torch.equal(own, four) and not torch.equal(own, three)


@pytest.mark.parametrize("C", [136, 384, 512])
def test_narrow_sweep_keeps_whole_operands(cuda, C):
    """One product per column: up to 512 columns an error and an entry of the factor enter an update with all of their 24
    bits, so a single product is off by its own rounding and what three planes leave out, below 2^-23 together."""
    gen = torch.Generator().manual_seed(C)
    R = 64
    W = 0.02 * torch.randn(R, C, generator=gen)
    W[:, 128:] = 0.0
    U = torch.eye(C)
    rows = torch.randint(0, 128, (C - 128,), generator=gen)
    U[rows, torch.arange(128, C)] = 0.5 * torch.randn(C - 128, generator=gen)
    w, run = W.to(cuda), W.to(cuda)
    scale = ops.absmax_scales(w[:, :128].contiguous(), 8, 4, torch.bfloat16)
    scale = torch.cat([scale, torch.ones(R, (C - 128) // 8, device=cuda)], 1).contiguous()
    # inside the first tile the factor is the identity, so its errors are those of plain rounding (to bf16: exact in fp32)
    _, deq = ops.gptq_sweep(run, U.to(cuda), scale, None, 8, C // 8, 1, 4, torch.bfloat16, True, ops.Precision(), W_original=w)
    e = (W - deq.cpu().float())[:, rows].double()
    want = e * U[rows, torch.arange(128, C)].double()
    assert bool(((run.cpu()[:, 128:].double() - want).abs() <= 2.0 ** -23 * want.abs()).all())


@pytest.mark.parametrize("rel_damp", [0.0, 1e-6, 1e-2])
@pytest.mark.parametrize("spread", [1.0, 2.5])
@pytest.mark.parametrize("C", [520, 1544])
def test_layer_with_little_damping_against_fp32_math(cuda, rel_damp, spread, C):
    """Channels over e^+-7 and a damping that does not lift the small ones: the factor's columns are scaled from one bound
    over the whole matrix, and the codes are still those of the fp32 CUDA cores."""
    gen = torch.Generator().manual_seed(C)
    X = torch.randn(2 * C, C, generator=gen, dtype=torch.float64) * torch.exp(spread * torch.randn(C, generator=gen, dtype=torch.float64))
    H = (X.T @ X / C).float()
    W = synthetic.layer_weight(200, C, 5, torch.bfloat16)

    def run(math):
        codes, _, _, flags = ops.quantize_layer([W.to(cuda)], H.to(cuda), 8, 4, rel_damp, precision=ops.Precision(math=math))
        assert int(flags[3]) == 0
        return codes[0].cpu()

    assert O.code_agreement(run(MATH_TENSOR), run(MATH_FP32)) >= CODE_AGREEMENT


@pytest.mark.parametrize("C", [520, 1544])
@pytest.mark.parametrize("large", ["first", "last"])
@pytest.mark.parametrize("tied", [1, 2])
def test_undamped_layer_with_a_few_large_channels(cuda, C, large, tied):
    """Small channels that depend on each other, column j on column j - 128, beside independent ones 2^32 as large: a bound
    over the whole matrix says nothing about the columns of the small ones, which are scaled by their own maxima."""
    gen = torch.Generator().manual_seed(C)
    n = 256 if C == 520 else 1024
    T = torch.eye(n, dtype=torch.float64)
    j = torch.arange(128, n)
    T[j - 128, j] = 0.5 + 0.5 * torch.rand(n - 128, generator=gen, dtype=torch.float64)
    big = 2.0 ** 64 * torch.eye(C - n, dtype=torch.float64)
    H = torch.block_diag(*((big, T @ T.T) if large == "first" else (T @ T.T, big))).float()
    W = [synthetic.layer_weight(200, C, 5 + i, torch.bfloat16).to(cuda) for i in range(tied)]

    def run(math):
        codes, _, _, flags = ops.quantize_layer(W, H.to(cuda), 8, 4, 0.0, precision=ops.Precision(math=math))
        assert int(flags[3]) == 0
        return torch.cat(codes).cpu()

    assert O.code_agreement(run(MATH_TENSOR), run(MATH_FP32)) >= CODE_AGREEMENT


# ------------------------------------------------------------------ MSE scale search
@pytest.mark.parametrize("R,C,g,dtype", [(64, 512, 128, torch.bfloat16), (40, 256, 32, torch.float16),
                                         (24, 384, 64, torch.float32), (8, 2048, 2048, torch.bfloat16)])
def test_mse_scales_match_oracle(cuda, R, C, g, dtype):
    """The shrink-factor search of src/quant_utils.py:104-139.  The loss sums |.|^2.4 over the
    group in an order the reference leaves open, so a candidate next to the minimum may win on
    one side and not the other: nearly all scales must be identical, every scale must be one of
    the candidates, and its loss must equal the oracle's minimum to rounding."""
    W = synthetic.layer_weight(R, C, 91, dtype).float()
    s0, zero, maxq = O.symmetric_grid(W, g, 4, dtype)
    want = O.mse_scale(W.unflatten(-1, (-1, g)), s0, zero, maxq, dtype)
    got = ops.mse_scales(W.to(cuda), ops.absmax_scales(W.to(cuda), g, 4, dtype), g, 4, dtype).cpu()
    assert float((got == want).float().mean()) >= 0.97
    p = torch.linspace(1, 0.2, 100)
    cands = O.round_fp(s0[..., None] * p, dtype)
    assert bool((cands == got[..., None]).any(-1).all())

    def loss(s):
        Wg = W.unflatten(-1, (-1, g))
        q = torch.clamp(torch.floor((Wg / s[..., None] + 8.0) + 0.5), 0.0, 15.0)
        y = O.round_fp((q - 8.0) * s[..., None], dtype)
        return ((y - Wg).abs().log() * 2.4).exp().sum(-1)

    torch.testing.assert_close(loss(got), loss(want), rtol=1e-3, atol=0)


@pytest.mark.parametrize("R,C,g,factor,dtype", [
    (16, 384, 384, 1.0, torch.bfloat16),      # wide groups: partial sums are compared on the way
    (5, 1536, 256, 1.0, torch.float32), (1300, 264, 264, 1.0, torch.bfloat16), (7, 248, 248, 1.0, torch.float16),
    (1299, 264, 264, 1.0, torch.float16), (1340, 688, 688, 1.0, torch.bfloat16), (1313, 688, 688, 1.0, torch.float32),   # either side of the line
    (9, 1056, 1056, 1e-6, torch.float32),     # a last trip of the lanes that is not full
    (16, 96, 24, 1.0, torch.float16),         # fewer elements than lanes
    (12, 256, 32, 1e-10, torch.bfloat16),
    (12, 512, 128, 1e4, torch.float32),
    (12, 512, 64, 1e-20, torch.float32),      # scales below the range of the reciprocal: the division
])
@pytest.mark.parametrize("outliers", [False, True])
def test_mse_scales_skip_no_winner(cuda, R, C, g, factor, dtype, outliers):
    """The search drops candidates by a lower bound of their loss.  No candidate may have a smaller
    loss in fp64 than the chosen one by more than fp32 sums allow: terms of one sign, g additions,
    about ten roundings in a term, |d|^norm of a d that cancels against x with |x| / |d| up to 2^8
    on the elements that matter: 1e-4 covers them."""
    norm = 1.0 if factor < 1e-12 else 2.4        # |d|^2.4 would leave fp32's range
    W = synthetic.layer_weight(R, C, 17 + g, torch.float32)
    if outliers:
        W[:, ::max(g // 2, 1)] *= 6.0
        W[0] = 0.0
    W = W * factor
    base = ops.absmax_scales(W.to(cuda), g, 4, dtype)
    s0 = base.cpu()
    got = ops.mse_scales(W.to(cuda), base, g, 4, dtype, norm=norm).cpu()
    cands = O.round_fp(s0[..., None] * torch.linspace(1, 0.2, 100), dtype)
    Wg = W.unflatten(-1, (-1, g))

    def loss(s):
        s = s[..., None]
        # an all-zero group has scale 0 in fp16 (1e-12 underflows): any code gives loss 0
        q = torch.clamp(torch.floor(((Wg / s).nan_to_num(0.0) + 8.0) + 0.5), 0.0, 15.0)
        return (O.round_fp((q - 8.0) * s, dtype) - Wg).double().abs().pow(norm).sum(-1)

    assert bool((cands == got[..., None]).any(-1).all())
    best = torch.stack([loss(cands[..., i]) for i in range(cands.shape[-1])]).amin(0)
    assert bool((loss(got) <= best * (1 + 1e-4)).all())


# ------------------------------------------------------------------ compact launches
@pytest.mark.parametrize("R,C,g,dtype,math", [(200, 512, 128, torch.bfloat16, MATH_TENSOR), (64, 384, 64, torch.float16, MATH_TENSOR),
                                              (333, 640, 32, torch.float32, MATH_TENSOR), (130, 512, 512, torch.bfloat16, MATH_FP32),
                                              (96, 392, 56, torch.float16, MATH_TENSOR), (2500, 256, 64, torch.bfloat16, MATH_TENSOR)])
def test_compact_sweep_is_bit_identical(cuda, R, C, g, dtype, math):
    """MQ_MATH_COMPACT changes how a launch is laid out (rows per CTA, a panel of the factorisation in one launch or two): codes,
    dequantized values, packed words and scales must be the same bits, through the whole-layer call and through the sweep
    alone with zero points and the factor of the inverse (the reference's form of the recurrence).  Group 56 crosses
    sub-blocks, 392 columns end on a tile of eight; 2500 rows are swept tile by tile, and that case is also held to the
    CPU oracle."""
    W = synthetic.layer_weight(R, C, 3, dtype).to(cuda)
    X = synthetic.activations(2 * C, C, 4, dtype).to(cuda)
    H = torch.zeros(C, C, device=cuda)
    ops.hessian_accum(H, X, 0.0, 2.0 / X.shape[0])
    outs = []
    for compact in (False, True):
        p = ops.Precision(math=math, compact=compact)
        outs.append(ops.quantize_layer([W], H.clone(), g, 4, 1e-2, want_dequantized=True, precision=p, want_packed=True))
    (c0, s0, d0, f0, p0), (c1, s1, d1, f1, p1) = outs
    assert torch.equal(c0[0], c1[0]) and torch.equal(s0[0], s1[0]) and torch.equal(p0[0], p1[0])
    assert torch.equal(d0[0].float(), d1[0].float()) and torch.equal(f0, f1)
    if R > 2368:
        want = O.quantize_layer(W.cpu(), H.cpu().clone(), bits=4, group_size=g, rel_damp=1e-2, block_size=128)
        assert torch.equal(s0[0].cpu(), want["scale"].float())
        assert O.code_agreement(c0[0].cpu(), want["qweight"]) >= CODE_AGREEMENT

    # the sweep alone: factor of the inverse, per-group zero points
    Hd = H.clone()
    ops.hessian_prepare(Hd, W.float(), 1e-2)
    U, _, _ = ops.hinv_upper(Hd, ops.Precision(math=math))
    scale = ops.absmax_scales(W.float(), g, 4, dtype)
    gen = torch.Generator().manual_seed(1)
    zero = torch.randint(6, 11, scale.shape, generator=gen).float().to(cuda)
    res = []
    for compact in (False, True):
        p = ops.Precision(math=math, compact=compact)
        res.append(ops.gptq_sweep(W.float().clone(), U, scale, zero, g, C // g, 1, 4, dtype, True, p))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1].float(), res[1][1].float())


# ------------------------------------------------------------------ one launch per panel
@pytest.mark.parametrize("C,tokens", [(136, 200), (392, 100), (1160, 1500), (4840, 1000), (9544, 700)])
def test_panel_in_one_launch_is_bit_identical(cuda, C, tokens):
    """The block and the solve in one launch against one launch each (compact): the same operations in the same order.
    One, two and four groups of rows per warp (from 4705 and 9409 rows on), first panels of 8 and 72 columns."""
    R = 24
    W = synthetic.layer_weight(R, C, 3, torch.bfloat16).to(cuda)
    X = synthetic.activations(tokens, C, 4, torch.bfloat16).to(cuda)
    H = torch.zeros(C, C, device=cuda)
    ops.hessian_accum(H, X, 0.0, 2.0 / tokens)

    def layer(compact):
        # the call leaves the factor, and behind it its diagonal, at the front of its workspace
        damped, nbytes = H.clone(), lib().mq_quantize_layer_workspace_bytes(1, R, C, MATH_TENSOR, 3, 3)
        _lib.workspace(damped.device, nbytes).zero_()
        out = ops.quantize_layer([W], damped, C, 4, 1e-2, want_dequantized=True, precision=ops.Precision(compact=compact))
        words = _lib.workspace(damped.device, nbytes)[: 4 * C * (C + 1)].clone().view(torch.float32)
        factor, diag = words[: C * C].view(C, C).triu(), words[C * C :]
        # (the matrix is scaled by powers of two, and the last pivot is the root of its element)
        scale = torch.log2(diag[-1] / damped[-1, -1].sqrt())
        assert bool((diag > 0).all()) and abs(float(scale - scale.round())) < 1e-5 and int((factor != 0).sum()) > C * C // 3
        return out, factor, diag

    ((c0, s0, d0, f0), u0, t0), ((c1, s1, d1, f1), u1, t1) = layer(False), layer(True)
    assert f0.tolist() == f1.tolist() and int(f0[3]) == 0
    assert torch.equal(u0, u1) and torch.equal(t0, t1)
    assert torch.equal(c0[0], c1[0]) and torch.equal(s0[0], s1[0]) and torch.equal(d0[0], d1[0])


# ------------------------------------------------------------------ row groups of the sweep tile
@pytest.mark.parametrize("R", [1, 7, 8, 9, 33, 1184, 1185, 4737, 9473])
@pytest.mark.parametrize("C,g", [(24, 24), (136, 8), (256, 32)])
def test_sweep_tile_row_groups(cuda, R, C, g):
    """One chain warp or two, groups that are not full, more groups than CTAs, a last tile of 8 columns,
    scales per sub-block and per column.  Rows are independent: every row's codes equal those of the
    same row swept in another grouping (the compact one, and alone)."""
    gen = torch.Generator().manual_seed(R + C)
    base = 0.02 * torch.randn(64, C, generator=gen)
    W = base[torch.arange(R) % 64].contiguous()
    U = torch.triu(0.2 * torch.randn(C, C, generator=gen), 1) + torch.eye(C)

    def sweep(w, precision):
        s = ops.absmax_scales(w, g, 4, torch.bfloat16)
        codes, deq = ops.gptq_sweep(w.clone(), U.to(cuda), s, None, g, C // g, 1, 4, torch.bfloat16, True, precision, W_original=w)
        assert torch.equal(deq, ops.dequantize(codes, s, None, g, 4, torch.bfloat16))
        return codes.cpu()

    got = sweep(W.to(cuda), ops.Precision())
    want = sweep(base[: min(R, 64)].to(cuda), ops.Precision())
    assert torch.equal(got, want[torch.arange(R) % 64])
    assert torch.equal(got, sweep(W.to(cuda), ops.Precision(compact=True)))


# ------------------------------------------------------------------ super-blocks of the sweep
@pytest.mark.parametrize("R", [1, 9, 1024, 1025])
@pytest.mark.parametrize("C,g", [(24, 8), (136, 136), (520, 8), (1160, 40), (1536, 128)])
@pytest.mark.parametrize("inverse_free", [True, False])
def test_sweep_by_super_blocks(cuda, R, C, g, inverse_free):
    """Up to 1024 rows a launch takes 512 columns: last blocks of eight columns and of one tile, CTAs that are not full, scales per
    sub-block and per column with zero points of their own, both recurrences, and the row behind the last that goes this way.
    Codes as on the fp32 CUDA cores, the compact launch's bits."""
    W = synthetic.layer_weight(R, C, 5, torch.bfloat16).float().to(cuda)
    X = synthetic.activations(2 * C, C, 6, torch.bfloat16).double()
    H = X.T @ X / C
    H.diagonal().add_(0.01 * H.diagonal().mean())
    U = H.float().to(cuda)
    if inverse_free:
        ops.chol_unit_factor(U)
    else:
        U = ops.hinv_upper(U)[0]
    scale = ops.absmax_scales(W, g, 4, torch.bfloat16)
    zero = (8 - torch.arange(scale.numel(), device=cuda).reshape(scale.shape) % 3).float().contiguous()

    def sweep(precision):
        return ops.gptq_sweep(W.clone(), U, scale, zero, g, C // g, 1, 4, torch.bfloat16, True, precision, W_original=W if inverse_free else None)

    (q, deq), (q0, _), (q1, deq1) = sweep(ops.Precision()), sweep(ops.Precision(math=MATH_FP32)), sweep(ops.Precision(compact=True))
    # a code on a rounding boundary takes others of its row along: of few codes those of one row in a hundred may differ
    assert int((q != q0).sum()) <= max(0.005 * q.numel(), 0.01 * C)
    assert R == 1 or int((q != q0).sum(0).max()) <= max(1, 0.1 * R)     # and no column is wrong as a whole
    assert torch.equal(q, q1) and torch.equal(deq, deq1)
    assert torch.equal(deq, ops.dequantize(q, scale, zero, g, 4, torch.bfloat16))


# ------------------------------------------------------------------ the weights' way in, the diagonal pass
@pytest.mark.parametrize("R,C,g", [(1, 8, 8), (65, 136, 8), (7, 160, 32), (64, 192, 64), (130, 1152, 128), (3, 9216, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("offset", [0, 2])
def test_layer_preparation_against_oracle(cuda, R, C, g, dtype, offset):
    """Dead channels, all-zero columns, ragged column blocks, more channels than one pass over the diagonal
    keeps, weights that start off a vector boundary: scales, damped Hessian and flags."""
    gen = torch.Generator().manual_seed(R + C)
    W = (0.02 * torch.randn(R, C, generator=gen)).to(dtype)
    W[:, 3] = 0.0
    H = torch.diag(torch.rand(C, generator=gen) + 0.5)
    H[0, 5] = H[5, 0] = 0.1
    H[3, 4] = H[4, 3] = 0.2
    H[6] = 0.0
    H[:, 6] = 0.0
    store = torch.empty(offset + R * C, dtype=dtype, device=cuda)
    w = store[offset:].view(R, C)
    w.copy_(W)
    Hd = H.to(cuda)
    _, scales, _, flags = ops.quantize_layer([w], Hd, g, 4, 1e-2)
    Wm = W.float().clone()
    Wm[:, 6] = 0.0
    s0, _, _ = O.symmetric_grid(Wm, g, 4, dtype)
    assert torch.equal(scales[0].cpu(), s0.float().reshape(R, C // g))
    zero_cols = int((Wm == 0).all(0).sum())
    assert flags.tolist()[:3] == [0, 1, zero_cols] and int(flags[3]) == 0
    want = H.clone()
    for c in torch.nonzero((Wm == 0).all(0)).flatten().tolist():
        want[c] = 0.0
        want[:, c] = 0.0
        want[c, c] = 1.0
    want.diagonal().add_(1e-2 * want.diagonal().double().mean().float())
    torch.testing.assert_close(Hd.cpu(), want, rtol=2e-6, atol=0)   # the mean's sum in another order


# ------------------------------------------------------------------ quadratic forms
@pytest.mark.parametrize("R,C", [(1, 1), (3, 13), (255, 64), (257, 200), (40, 257), (300, 1031), (512, 768)])
@pytest.mark.parametrize("kind", ["hessian", "unsymmetric", "spread", "tiny", "huge"])
def test_quadratic_forms_against_fp64(cuda, R, C, kind):
    """Ragged tiles in rows, columns and k; any square H, not only symmetric ones; scales over many decades; row
    strides.  Error: three of four half products of 22-bit pairs, 2^-22 each, sums of 64 of k in the
    tensor core (four truncations at 2^-23): below 2^-20 of the sum of absolute products."""
    gen = torch.Generator().manual_seed(R * 1000 + C)
    X = torch.randn(2 * C + 3, C, generator=gen, dtype=torch.float64)
    if kind == "spread":
        X *= torch.exp(3.0 * torch.randn(C, generator=gen, dtype=torch.float64))
    H = (X.T @ X / X.shape[0]).float()
    if kind == "unsymmetric":
        H = torch.randn(C, C, generator=gen)
    q, w = torch.randn(R, C, generator=gen), torch.randn(R, C, generator=gen)
    if kind == "tiny":
        q, w, H = q * 1e-9, w * 1e-12, H * 1e-20
    if kind == "huge":
        q, w, H = q * 1e-2, w * 1e-2, H * 2.0 ** 117
    wide = torch.empty(R, C + 5, device=cuda)
    wide[:, :C] = q.to(cuda)
    got = ops.error_forms(wide[:, :C], w.to(cuda), H.to(cuda)).cpu()
    one = ops.quadratic_form(w.to(cuda), H.to(cuda)).cpu()
    for a, g in (((q - w), got[0]), (w, got[1]), (w, one)):
        a, h = a.double(), H.double()
        want, size = float(((a @ h) * a).sum()), float(((a.abs() @ h.abs()) * a.abs()).sum())
        assert abs(float(g) - want) <= 2.0 ** -20 * size


@pytest.mark.parametrize("R,widths", [(1, (1, 64, 65, 150, 200, 257, 330, 400, 450)), (300, (40, 128, 250, 320, 513)), (300, (5000,))])
def test_quadratic_forms_back_to_back(cuda, R, widths):
    """One to eight slabs of k, one tile per CTA pair and several: whatever use of the ring is the last one, the pair leaves
    with its commits and copies received, and the launch that follows on the same SMs finds its barriers its own (no wait
    expires, which is checked after every test, and every result of the series is right)."""
    gen = torch.Generator().manual_seed(R + len(widths))
    cases = []
    for C in widths:
        X = torch.randn(C + 3, C, generator=gen)
        cases.append((torch.randn(R, C, generator=gen), torch.randn(R, C, generator=gen), X.T @ X / C))
    dev = [tuple(t.to(cuda) for t in c) for c in cases]
    got = [[ops.error_forms(*c) for c in dev] for _ in range(6)]
    for i, (q, w, H) in enumerate(cases):
        for a, k in ((q - w, 0), (w, 1)):
            a, h = a.double(), H.double()
            want, size = float(((a @ h) * a).sum()), float(((a.abs() @ h.abs()) * a.abs()).sum())
            for series in got:      # bound: as in test_quadratic_forms_against_fp64
                assert abs(float(series[i][k]) - want) <= 2.0 ** -20 * size


# ------------------------------------------------------------------ column permutation
@pytest.mark.parametrize("R,C", [(1, 1), (3, 7), (130, 1032), (1300, 64), (2, 24577)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.uint8])
def test_permute_columns(cuda, R, C, dtype):
    """Rows that fit the staging and rows that do not, ragged widths, row strides, a row index, groups."""
    gen = torch.Generator().manual_seed(R + C)
    src = torch.randint(0, 255, (R, C + 3), generator=gen).to(dtype)[:, :C]
    cols, rows = torch.randperm(C, generator=gen), torch.randint(0, R, (R + 2,), generator=gen)
    dev = torch.empty(R, C + 3, dtype=dtype, device=cuda)[:, :C]
    dev.copy_(src)
    c32, r32 = cols.int().to(cuda), rows.int().to(cuda)
    assert torch.equal(ops.permute_columns(dev, c32).cpu(), src[:, cols])
    assert torch.equal(ops.permute_columns(dev, c32, rows=r32).cpu(), src[rows][:, cols])
    few = src[:, : (C + 7) // 8].contiguous()
    assert torch.equal(ops.permute_columns(few.to(cuda), c32, group=8).cpu(), few.repeat_interleave(8, -1)[:, cols])
