"""GPU parity of the KNN consumers (through the C-ABI): inverse-distance interpolation and the
neighbourhood max-pool, against the numpy oracle, against vectors from the reference's own Python,
and against the unfused torch formulation of the reference on the same device."""
import os

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

G = np.load(os.path.join(os.path.dirname(__file__), "golden", "knn_consumers_reference.npz"))


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _scene():
    return _dev(G["src"]), _dev(G["qry"]), _dev(G["so"]), _dev(G["qo"])


@pytest.mark.parametrize("tag,K", [("k3", 3), ("k5", 5)])
def test_interpolation_fp32_bit_exact_vs_oracle_and_reference(tag, K):
    from swin3d_b200.sparse_dl.knn import knn_linear_interpolation
    src, qry, so, qo = _scene()
    feat = _dev(G[f"interp.{tag}.feat"]).requires_grad_(True)
    out = knn_linear_interpolation(src, qry, feat, so, qo, K=K)
    out.backward(_dev(G[f"interp.{tag}.dout"]))
    idx, d2 = O.knn(K, G["src"], G["qry"], G["so"], G["qo"])
    ref = O.knn_interpolate(idx, np.sqrt(d2), G[f"interp.{tag}.feat"])
    assert np.array_equal(out.detach().cpu().numpy(), ref)                # same operation order
    np.testing.assert_allclose(out.detach().cpu().numpy(), G[f"interp.{tag}.f32.out"], rtol=2e-6, atol=1e-7)
    # tolerance of the gradient: fp32 sums in a different order (atomics), 1e-5 relative
    np.testing.assert_allclose(feat.grad.cpu().numpy(), G[f"interp.{tag}.f32.dsrc"], rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("tag,K", [("k3", 3), ("k5", 5)])
def test_interpolation_fp16(tag, K):
    from swin3d_b200.sparse_dl.knn import knn_linear_interpolation
    src, qry, so, qo = _scene()
    feat = _dev(G[f"interp.{tag}.feat"]).half().requires_grad_(True)
    out = knn_linear_interpolation(src, qry, feat, so, qo, K=K)
    out.backward(_dev(G[f"interp.{tag}.dout"]).half())
    idx, d2 = O.knn(K, G["src"], G["qry"], G["so"], G["qo"])
    ref = O.knn_interpolate(idx, np.sqrt(d2), G[f"interp.{tag}.feat"].astype(np.float16))
    assert np.array_equal(out.detach().cpu().numpy(), ref)                # rounding after every neighbour
    ref_d = G[f"interp.{tag}.f16.dsrc"]
    err = np.max(np.abs(feat.grad.float().cpu().numpy() - ref_d))
    assert err <= 2e-2 * max(1.0, np.max(np.abs(ref_d)))                  # fp16 tolerance of the suite


def test_interpolation_matches_unfused_torch_on_large_input():
    """The reference's formulation (swin3d_layers.py:64-72) evaluated with torch ops on the GPU."""
    from swin3d_b200.sparse_dl.knn import KNN, KNNInterpolate
    g = torch.Generator(device="cuda").manual_seed(5)
    Ns, Nq, C, K = 20_000, 60_000, 96, 3
    src = torch.rand(Ns, 3, device="cuda", generator=g) * 10
    qry = torch.rand(Nq, 3, device="cuda", generator=g) * 10
    so = torch.tensor([Ns], dtype=torch.int32, device="cuda")
    qo = torch.tensor([Nq], dtype=torch.int32, device="cuda")
    feat = torch.randn(Ns, C, device="cuda", generator=g, requires_grad=True)
    idx, dist = KNN.apply(K, src, qry, so, qo)
    out = KNNInterpolate.apply(feat, idx, dist)
    dout = torch.randn(Nq, C, device="cuda", generator=g)
    out.backward(dout)
    mine, feat.grad = feat.grad.clone(), None
    weight = 1.0 / (dist + 1e-8)
    weight = weight / torch.sum(weight, dim=1, keepdim=True)
    ref = torch.zeros((Nq, C), dtype=feat.dtype, device="cuda")
    for i in range(K):
        ref = ref + feat[idx[:, i].long(), :] * weight[:, i].unsqueeze(-1)
    ref.backward(dout)
    # torch's own kernels may associate the sum over K and round the division differently: last-bit tolerance
    assert torch.allclose(out, ref, rtol=2e-6, atol=1e-6)
    assert torch.allclose(mine, feat.grad, rtol=1e-4, atol=1e-5)
    # linearity in the features: interpolating a constant field returns the constant
    ones = KNNInterpolate.apply(torch.ones(Ns, 8, device="cuda"), idx, dist)
    assert torch.allclose(ones, torch.ones_like(ones), atol=1e-6)


def test_interpolation_argument_errors():
    from swin3d_b200.sparse_dl.knn import KNNInterpolate
    idx = torch.zeros((4, 3), dtype=torch.int32, device="cuda")
    dist = torch.ones((4, 3), device="cuda")
    with pytest.raises(ValueError):
        KNNInterpolate.apply(torch.ones(5, 6, device="cuda"), idx, dist)        # C not a multiple of 4
    with pytest.raises(ValueError):
        KNNInterpolate.apply(torch.ones(5, 8, device="cuda").double(), idx, dist)
    empty = KNNInterpolate.apply(torch.ones(5, 8, device="cuda"), idx[:0], dist[:0])
    assert empty.shape == (0, 8)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_maxpool_vs_oracle(dtype):
    from swin3d_b200.sparse_dl.knn import KNN, KNNMaxPool
    src, qry, so, qo = _scene()
    K = 16
    rng = np.random.default_rng(11)
    g_np = rng.normal(size=(G["src"].shape[0], 40)).astype(np.float32)
    g_np[:, :4] = np.round(g_np[:, :4])                    # ties: the first maximum must win
    g = _dev(g_np).to(dtype).requires_grad_(True)
    idx, _ = KNN.apply(K, src, qry, so, qo)
    out, arg = KNNMaxPool.apply(g, idx)
    dout_np = rng.normal(size=tuple(out.shape)).astype(np.float32)
    out.backward(_dev(dout_np).to(dtype))
    oidx, _ = O.knn(K, G["src"], G["qry"], G["so"], G["qo"])
    ref_out, ref_arg = O.knn_maxpool(oidx, g.detach().cpu().numpy())
    assert np.array_equal(out.detach().cpu().numpy(), ref_out)
    assert np.array_equal(arg.cpu().numpy(), ref_arg)
    ref_dg = O.knn_maxpool_bwd(ref_arg, _dev(dout_np).to(dtype).float().cpu().numpy(), g.shape[0])
    tol = 1e-5 if dtype == torch.float32 else 2e-2
    assert np.max(np.abs(g.grad.float().cpu().numpy() - ref_dg)) <= tol * max(1.0, np.max(np.abs(ref_dg)))


def test_downsample_tail_matches_reference_vectors():
    """gather + LayerNorm + Linear + MaxPool1d(16) of GridKNNDownsample.forward, evaluated as
    LayerNorm + Linear per source row followed by the fused neighbourhood max-pool."""
    from swin3d_b200.sparse_dl.knn import knn_max_pool
    src, qry, so, qo = _scene()
    feat = _dev(G["down.feat"]).requires_grad_(True)
    norm = torch.nn.LayerNorm(feat.shape[1]).cuda()
    linear = torch.nn.Linear(feat.shape[1], G["down.lin_w"].shape[0], bias=False).cuda()
    with torch.no_grad():
        norm.weight.copy_(_dev(G["down.norm_w"]))
        norm.bias.copy_(_dev(G["down.norm_b"]))
        linear.weight.copy_(_dev(G["down.lin_w"]))
    out = knn_max_pool(16, src, qry, linear(norm(feat)), so, qo)      # fp32 GEMM (TF32 is off by default)
    out.backward(_dev(G["down.dout"]))
    np.testing.assert_allclose(out.detach().cpu().numpy(), G["down.out"], rtol=1e-4, atol=1e-5)
    np.testing.assert_allclose(feat.grad.cpu().numpy(), G["down.dfeat"], rtol=1e-3, atol=1e-4)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("K,C,n_src,Nq", [(3, 8, 1, 1), (3, 80, 4095, 1000), (3, 48, 4097, 12_293), (16, 40, 300, 65),
                                          (5, 320, 70, 129), (64, 16, 257, 64)])
def test_gather_backwards_match_the_scatter(dtype, K, C, n_src, Nq):
    """Gradient gathered per source row against the scatter form and fp64: sources without an entry,
    ends of the scan's tiles, one query, lists longer than a warp, every K of the templates."""
    from swin3d_b200.sparse_dl.knn import KNNInterpolate, KNNMaxPool, consumers
    g = torch.Generator(device="cuda").manual_seed(K * Nq)
    idx = torch.randint(0, n_src, (Nq, K), generator=g, device="cuda", dtype=torch.int32)
    dist = torch.rand((Nq, K), generator=g, device="cuda")
    feat = torch.randn((n_src, C), generator=g, device="cuda").to(dtype).requires_grad_()
    dout = torch.randn((Nq, C), generator=g, device="cuda").to(dtype)
    w = 1.0 / (dist + 1e-8)
    w = (w / w.sum(1, keepdim=True)).double()
    want = torch.zeros((n_src, C), dtype=torch.float64, device="cuda")
    size = torch.zeros((n_src, C), dtype=torch.float64, device="cuda")
    for i in range(K):
        want.index_add_(0, idx[:, i].long(), w[:, i, None] * dout.double())
        size.index_add_(0, idx[:, i].long(), w[:, i, None] * dout.double().abs())
    # fp32 sums of n terms: n eps of the sum of magnitudes at most (n <= a few hundred), then one rounding to dtype
    eps = 2.0 ** -24 if dtype == torch.float32 else 2.0 ** -11
    n_max = int(torch.bincount(idx.flatten().long(), minlength=n_src).max()) + 8
    bound = size * n_max * 2.0 ** -24 + want.abs() * eps + 2.0 ** -24
    was = consumers.GATHER_MOST_PER_SOURCE
    try:
        for most in (0, 1 << 30):
            consumers.GATHER_MOST_PER_SOURCE = most
            (got,) = torch.autograd.grad(KNNInterpolate.apply(feat, idx, dist), [feat], dout)
            assert ((got.double() - want).abs() <= bound).all()
    finally:
        consumers.GATHER_MOST_PER_SOURCE = was
    out, arg = KNNMaxPool.apply(feat, idx)
    (ref,) = torch.autograd.grad(out, [feat], dout)
    out2 = consumers._KNNMaxPoolSlots.apply(feat, idx)
    (got,) = torch.autograd.grad(out2, [feat], dout)
    assert torch.equal(out, out2)
    size = torch.zeros((n_src, C), dtype=torch.float64, device="cuda").scatter_add_(0, arg.long(), dout.double().abs())
    if K <= n_src:                                    # a row listed twice by a query: the first position counts, as here
        assert ((got.double() - ref.double()).abs() <= size * n_max * 2.0 ** -23 + 2 * ref.double().abs() * eps + 2.0 ** -24).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("K,C,n_src,Nq,counts", [(3, 80, 500, 3_000, (64, 65, 66)), (3, 640, 40, 3_000, (1279, 1280, 1281, 2561)),
                                                 (16, 8, 300, 5_000, (255, 256, 257, 511, 512, 513)), (3, 16, 20_000, 40_000, (20_000, 70, 65)),
                                                 (1, 4, 3, 3_000, (700, 2_000)), (3, 2064, 9, 700, (100, 300))])
def test_gather_backwards_of_long_rows(dtype, K, C, n_src, Nq, counts):
    """Source rows with more entries than a thread sums (64) and than a block takes at a time (the larger of 256 and 2 C),
    each side of both, among rows without any; more pieces in a row than threads in a block."""
    if dtype == torch.float16 and C % 8:
        pytest.skip("rows of fp16 are whole 16-byte pieces")
    from swin3d_b200.sparse_dl.knn import KNNInterpolate, consumers
    g = torch.Generator(device="cuda").manual_seed(C + Nq)
    rest = torch.randint(len(counts) + 1, max(n_src, len(counts) + 2), (Nq * K - sum(counts),), generator=g, device="cuda") % n_src
    idx = torch.cat([torch.full((c,), i, device="cuda") for i, c in enumerate(counts)] + [rest])
    idx = idx[torch.randperm(Nq * K, generator=g, device="cuda")].view(Nq, K).int()
    dist = torch.rand((Nq, K), generator=g, device="cuda")
    feat = torch.randn((n_src, C), generator=g, device="cuda").to(dtype).requires_grad_()
    dout = torch.randn((Nq, C), generator=g, device="cuda").to(dtype)
    w = 1.0 / (dist + 1e-8)
    w = (w / w.sum(1, keepdim=True)).double()
    size, want = (torch.zeros((n_src, C), dtype=torch.float64, device="cuda") for _ in range(2))
    for i in range(K):
        want.index_add_(0, idx[:, i].long(), w[:, i, None] * dout.double())
        size.index_add_(0, idx[:, i].long(), w[:, i, None] * dout.double().abs())
    eps = 2.0 ** -24 if dtype == torch.float32 else 2.0 ** -11
    n_max = int(torch.bincount(idx.flatten().long(), minlength=n_src).max()) + 8
    was, consumers.GATHER_MOST_PER_SOURCE = consumers.GATHER_MOST_PER_SOURCE, 1 << 30
    try:
        (got,) = torch.autograd.grad(KNNInterpolate.apply(feat, idx, dist), [feat], dout)
        out = consumers._KNNMaxPoolSlots.apply(feat, idx)
        (pooled,) = torch.autograd.grad(out, [feat], dout)
    finally:
        consumers.GATHER_MOST_PER_SOURCE = was
    assert ((got.double() - want).abs() <= size * n_max * 2.0 ** -24 + want.abs() * eps + 2.0 ** -24).all()
    arg = torch.gather(idx.long()[:, :, None].expand(-1, -1, C), 1, feat.detach()[idx.long()].argmax(1, keepdim=True))[:, 0]
    ref, size = (torch.zeros((n_src, C), dtype=torch.float64, device="cuda").scatter_add_(0, arg, d) for d in (dout.double(), dout.double().abs()))
    assert ((pooled.double() - ref).abs() <= size * n_max * 2.0 ** -24 + ref.abs() * eps + 2.0 ** -24).all()


@pytest.mark.parametrize("dtype,per_source,gathered", [(torch.float16, 190, True), (torch.float16, 200, False), (torch.float32, 22, True),
                                                       (torch.float32, 26, False)])
def test_pooling_either_side_of_the_gather(dtype, per_source, gathered):
    """knn_max_pool takes the gathered backward up to its limit of entries per source, and both give the same gradient."""
    from swin3d_b200.sparse_dl.knn import KNN, KNNMaxPool, knn_max_pool
    K, n_src = 16, 800
    rng = np.random.default_rng(per_source)
    src, qry = (rng.random((n, 3), dtype=np.float32) for n in (n_src, per_source * n_src // K))
    a = [_dev(src), _dev(qry)]
    so, qo = _dev(np.array([len(src)], np.int32)), _dev(np.array([len(qry)], np.int32))
    g = torch.randn((n_src, 16), device="cuda").to(dtype).requires_grad_()
    dout = torch.randn((len(qry), 16), device="cuda").to(dtype)
    out = knn_max_pool(K, *a, g, so, qo)
    assert type(out.grad_fn).__name__ == ("_KNNMaxPoolSlotsBackward" if gathered else "KNNMaxPoolBackward")
    ref = KNNMaxPool.apply(g, KNN.apply(K, *a, so, qo)[0])[0]
    assert torch.equal(out, ref)
    (x,), (y,) = torch.autograd.grad(out, [g], dout), torch.autograd.grad(ref, [g], dout)
    # both sum in fp32, in another order, and round once
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -16
    assert ((x.double() - y.double()).abs() <= 2 * eps * y.double().abs() + 2.0 ** -14).all()
