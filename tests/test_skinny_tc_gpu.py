"""The projection kernel that splits K over a cluster, forced for every shape and split (a shape outside its domain is then an
error): edges of its tiles (128 rows of W, 64 pairs), of its 64-column blocks, of the split (fewer blocks than CTAs, slices of
unequal length), of the rows, and more tiles than clusters with 8 and with 16 rows."""
import numpy as np
import pytest

from test_skinny_gemm_gpu import rmsnorm16, w16

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 1, 2, 3, 5, 7, 8], ids=lambda c: f"cluster-{c or 'chosen'}", autouse=True)
def cluster(b200p, request):
    b200p.set_tuning("runtime_skinny", 3)
    b200p.set_tuning("skinny_cluster", request.param)
    yield request.param
    b200p.set_tuning("runtime_skinny", -1)
    b200p.set_tuning("skinny_cluster", -1)


# the last one has more tiles than clusters and more columns than the two other kernels hold
@pytest.mark.parametrize("M,N,K", [(1, 128, 512), (4, 70, 16), (12, 140, 144), (2, 130, 528), (3, 65, 1040), (5, 257, 1600), (8, 127, 576), (9, 200, 2048), (16, 96, 544), (13, 2048, 5632), (16, 19400, 8192), (7, 40100, 1024)])
def test_all_prologues_and_plain_epilogues(b200p, torch_cuda, cluster, M, N, K):
    torch, kind = torch_cuda, "f16" if M == 5 else "bf16"
    rng = np.random.default_rng(M * 1000 + K)
    if cluster and -(-K // 64 // cluster) * (8 if M <= 8 else 16) > 1088:
        pytest.skip("the slice of X does not fit")
    Wf, W = w16(torch, rng, (N, K), kind, 0.05)
    Xf, X = w16(torch, rng, (M, K), kind)
    res = rng.standard_normal((M, N)).astype(np.float32)
    out = torch.from_numpy(res.copy()).cuda()
    b200p.skinny_gemm(W, out, x16=X, epilogue="acc32")
    ref = res.astype(np.float64) + Xf @ Wf.T
    # fp32 sums of K products in any order: sqrt(K) roundings of the partial sums, far below 1e-4 of the largest output
    assert np.abs(out.cpu().numpy() - ref).max() < 1e-4 * max(1.0, np.abs(ref).max())
    wide = torch.full((M, K + 24), float("nan"), dtype=X.dtype, device="cuda")     # a strided matrix; what lies past its columns is not read
    wide[:, :K] = X
    out2 = torch.from_numpy(res.copy()).cuda()
    b200p.skinny_gemm(W, out2, x16=wide[:, :K], epilogue="acc32")
    assert torch.equal(out, out2)
    nwf, nw = w16(torch, rng, (K,), kind)
    x = rng.standard_normal((M, K)).astype(np.float32)
    ref = rmsnorm16(x.astype(np.float64), nwf, kind) @ Wf.T
    out = torch.full((M + 1, N), 7.0, dtype=torch.float32, device="cuda")
    b200p.skinny_gemm(W, out[:M], x32=torch.from_numpy(x).cuda(), norm_w=nw, epilogue="store32")
    assert np.abs(out[:M].cpu().numpy() - ref).max() < 2e-3 * np.abs(ref).max()     # 1-ulp flips of normalised activations
    assert (out[M] == 7.0).all()


@pytest.mark.parametrize("M,F,K", [(1, 40, 512), (4, 63, 528), (8, 300, 512), (11, 65, 1040), (16, 5632, 2048)])
def test_gated_epilogues(b200p, torch_cuda, M, F, K):
    torch = torch_cuda
    rng = np.random.default_rng(F + M)
    Wf, W = w16(torch, rng, (2 * F, K), "bf16", 3.0 / np.sqrt(K))
    Xf, X = w16(torch, rng, (M, K), "bf16")
    g, u = Xf @ Wf[:F].T, Xf @ Wf[F:].T
    ref = 0.5 * g * (1.0 + np.tanh(np.sqrt(2 / np.pi) * (g + 0.044715 * g ** 3))) * u
    out = torch.zeros((M, F), dtype=torch.bfloat16, device="cuda")
    b200p.skinny_gemm(W, out, x16=X, epilogue="gelu16")
    assert (np.abs(out.float().cpu().numpy() - ref) < 2.0 ** -8 * np.abs(ref) + 2e-4).all()
    nwf, nw = w16(torch, rng, (K,), "bf16")
    x = rng.standard_normal((M, K)).astype(np.float32)
    X = rmsnorm16(x.astype(np.float64), nwf, "bf16")
    g, u = X @ Wf[:F].T, X @ Wf[F:].T
    ref = g / (1.0 + np.exp(-g)) * u
    b200p.skinny_gemm(W, out, x32=torch.from_numpy(x).cuda(), norm_w=nw, epilogue="silu16")
    assert np.abs(out.float().cpu().numpy() - ref).max() < (2.0 ** -8 + 3e-3) * max(1e-3, np.abs(ref).max())


@pytest.mark.parametrize("M,N,K", [(8, 300, 8192), (16, 300, 4096), (16, 520, 2048), (11, 200, 1040)])
def test_products_of_one_sign_are_not_truncated_in_long_chains(b200p, torch_cuda, cluster, M, N, K):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(K)
    W, X = (torch.randn(s, device="cuda", generator=g).abs().bfloat16() for s in ((N, K), (M, K)))
    out = torch.zeros((M, N), device="cuda")
    b200p.skinny_gemm(W, out, x16=X, epilogue="acc32")
    ref = X.double() @ W.double().T
    # two truncated additions lose at most 2^-23 of the sum each; the fp32 sums after them round to nearest, which averages
    # out, below 2^-24.  One accumulator for all of K = 4096: 256 truncations, 5e-6.
    assert ((out.double() - ref).norm() / ref.norm()).item() < 2 * 2.0 ** -23 + 2.0 ** -24


def test_a_shape_outside_the_kernel_is_refused_when_it_is_forced(b200p, torch_cuda, cluster):
    torch = torch_cuda
    K = 64 * 1100                                            # 8 CTAs: 138 blocks of 8 rows, more than lie beside the ring
    W, X = torch.zeros((16, K), device="cuda").bfloat16(), torch.zeros((8, K), device="cuda").bfloat16()
    with pytest.raises(b200p.B200PError) as e:
        b200p.skinny_gemm(W, torch.zeros((8, 16), device="cuda"), x16=X, epilogue="acc32")
    assert e.value.status == -10
