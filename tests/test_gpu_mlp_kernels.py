"""The surrogate's launch-saving kernels at the edges of their ranges: every
block width of the default contraction, the multi-layer training kernels
against their single-matrix forms, and the ensemble statistics."""
import ctypes

import numpy as np
import pytest

from oracle import mlp_oracle as MO

pytestmark = pytest.mark.gpu


def _bf(a):
    import torch
    return torch.from_numpy(np.asarray(a, np.float32)).cuda().to(torch.bfloat16)


# (M, N): blocks of 64, 128 and 256 columns; K: fewer tiles than stages, a ring that wraps
@pytest.mark.parametrize("M,N", [(128, 256), (2432, 1024), (2432, 4096)])
@pytest.mark.parametrize("K", [64, 640])
@pytest.mark.parametrize("pad", [0, 2])
def test_gemm_block_widths_vs_numpy(cuda_device, M, N, K, pad):
    """pad: output and mask rows that do not start on 16-byte boundaries (the older epilogue)."""
    import torch
    from cupyram_b200 import surrogate as S
    rng = np.random.default_rng(7)
    A, B = rng.normal(size=(M, K)), rng.normal(size=(N, K))
    bias = rng.normal(size=N).astype(np.float32)
    ref = MO.to_bf16(A) @ MO.to_bf16(B).T
    scale = np.abs(ref).max()
    Ab, Bb, bt = _bf(A), _bf(B), torch.from_numpy(bias).cuda()
    mask = _bf(rng.normal(size=(M, N + pad)))[:, :N]
    S.tc_error_flag().zero_()
    out = torch.full((M, N + pad), float("nan"), device="cuda")[:, :N]
    ob = torch.full((M, N + pad), float("nan"), dtype=torch.bfloat16, device="cuda")[:, :N]
    S.gemm(S.EPI_F32, Ab, Bb, out, tc=True)
    assert np.abs(out.cpu().numpy() - ref).max() < 1e-5 * scale * K
    S.gemm(S.EPI_BIAS_F32, Ab, Bb, out, bias=bt, tc=True)
    assert np.abs(out.cpu().numpy() - (ref + bias)).max() < 1e-5 * scale * K
    S.gemm(S.EPI_BIAS_RELU_BF16, Ab, Bb, ob, bias=bt, tc=True)
    want = np.maximum(ref + bias, 0)
    assert np.abs(ob.float().cpu().numpy() - want).max() <= 2 ** -7 * np.abs(want).max() + 1e-3
    S.gemm(S.EPI_RELU_MASK_BF16, Ab, Bb, ob, mask=mask, tc=True)
    want = np.where(mask.float().cpu().numpy() > 0, ref, 0.0)
    assert np.abs(ob.float().cpu().numpy() - want).max() <= 2 ** -7 * scale + 1e-3
    assert int(S.tc_error_flag().item()) == 0


@pytest.mark.parametrize("dims,batch", [([128, 256], 128), ([128, 384, 256], 256), ([128] * 19 + [256], 128)])
def test_training_step_matches_single_matrix_kernels(cuda_device, dims, batch):
    """One backward and step of the whole network against the transpose, column
    sum and Adam calls layer by layer (19 layers take two launches)."""
    import torch
    from cupyram_b200 import surrogate as S
    m = S.MLP(dims, seed=2)
    g = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randn(batch, dims[0], generator=g, device="cuda").to(torch.bfloat16)
    m.forward(X)
    dout = m.grad_buffer(batch)
    dout.copy_(torch.randn(batch, dims[-1], generator=g, device="cuda"))
    m.backward(dout)
    H, _, dH, _, _ = m._buffers(batch)
    L = len(m.W)
    for l in range(L):
        want = torch.empty_like(m.gW[l])
        S.gemm(S.EPI_F32, dH[l].t().contiguous(), (X if l == 0 else H[l]).t().contiguous(), want)
        assert torch.equal(m.gW[l], want), l
        # the same column sum, and within FP32 rounding of the FP64 one (512 terms)
        ref = dH[l].double().sum(0)
        assert (m.gb[l].double() - ref).abs().max() <= 1e-5 * dH[l].double().abs().sum(0).max(), l
    before = [[t.clone() for t in lst] for lst in (m.W, m.mW, m.vW, m.b, m.mb, m.vb)]
    m.step(1e-3, weight_decay=0.01)
    k = S.kernels()
    for l in range(L):
        w, mw, vw, b, mb, vb = (lst[l] for lst in before)
        w16 = torch.empty_like(m.Wb[l])
        for p, gr, mo, ve, h, wd in ((w, m.gW[l], mw, vw, w16, 0.01), (b, m.gb[l], mb, vb, None, 0.0)):
            assert k.cr_mlp_adam(S._p(p), S._p(gr), S._p(mo), S._p(ve), S._p(h), p.numel(), 1e-3, 0.9, 0.999, 1e-8, 1,
                                 wd, S._stream()) == 0
        for a, c in ((m.W[l], w), (m.mW[l], mw), (m.vW[l], vw), (m.b[l], b), (m.mb[l], mb), (m.vb[l], vb),
                     (m.Wb[l], w16), (m.WTb[l], w16.t())):
            assert torch.equal(a, c), l


@pytest.mark.parametrize("members", [1, 2, 3, 4, 5, 64])
@pytest.mark.parametrize("n", [4, 1020, 300004])
def test_ensemble_statistics(cuda_device, members, n):
    import torch
    from cupyram_b200 import surrogate as S
    g = torch.Generator(device="cuda").manual_seed(3)
    preds = [2.0 * torch.randn(n, generator=g, device="cuda") for _ in range(members)]
    preds[-1][1] = float("nan")
    preds[0][2] = float("inf")
    mean, spread = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
    ptrs = (ctypes.c_void_p * members)(*[p.data_ptr() for p in preds])
    assert S.kernels().cr_mlp_ensemble_stats(ptrs, members, n, 25.0, 90.0, 20.0, 150.0, S._p(mean), S._p(spread),
                                             S._stream()) == 0
    tl = (torch.stack(preds) * 25.0 + 90.0).clamp(20.0, 150.0).double()
    assert torch.isnan(mean[1]) and torch.isnan(spread[1])
    ok = torch.arange(n, device="cuda") != 1
    # FP32 sums of up to 64 values of at most 150
    assert (mean[ok].double() - tl.mean(0)[ok]).abs().max() < 64 * 150 * 6e-8
    assert (spread[ok].double() - tl.std(0, unbiased=False)[ok]).abs().max() < 1e-3
    assert S.kernels().cr_mlp_ensemble_stats(ptrs, members, n - 1, 25.0, 90.0, 20.0, 150.0, S._p(mean), S._p(spread),
                                             S._stream()) != 0


# one block per CTA, several, rings that wrap within a block, no hidden layer; 384: not the fused path
@pytest.mark.parametrize("dims", [[128, 256], [128, 256, 512, 4096], [192 * 2, 256, 768], [128, 384, 256]])
@pytest.mark.parametrize("members", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("batch", [128, 2432])
def test_ensemble_predict_matches_forward_and_statistics(cuda_device, dims, members, batch):
    import torch
    from cupyram_b200 import surrogate as S
    models = [S.MLP(dims, seed=k) for k in range(members)]
    g = torch.Generator(device="cuda").manual_seed(2)
    for m in models:
        for b in m.b:
            b.copy_(torch.randn(b.shape, generator=g, device="cuda"))
    X = torch.randn(batch, dims[0], generator=g, device="cuda").to(torch.bfloat16)
    n = batch * dims[-1]
    S.tc_error_flag().zero_()
    mean, spread, m0, s0 = (torch.full((batch, dims[-1]), float("nan"), device="cuda") for _ in range(4))
    e = S.Ensemble.__new__(S.Ensemble)
    e.models = models
    e._predict_chunk(X, mean, spread)
    preds = [m.forward(X) for m in models]
    ptrs = (ctypes.c_void_p * members)(*[p.data_ptr() for p in preds])
    assert S.kernels().cr_mlp_ensemble_stats(ptrs, members, n, S.TL_SCALE, S.TL_MID, S.TL_LO, S.TL_HI, S._p(m0),
                                             S._p(s0), S._stream()) == 0
    # the same sums over K in the same order; at most the statistics' own FP32 rounding of values up to 150
    assert (mean - m0).abs().max() <= 150 * 2 ** -22
    assert (spread - s0).abs().max() <= 1e-3
    assert int(S.tc_error_flag().item()) == 0
