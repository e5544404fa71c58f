"""Which kernel a projection takes by default: the one that splits K over a cluster gives other bits than the streaming and
register kernels (another order of summation), so its own result, forced, tells."""
import pytest

pytestmark = pytest.mark.gpu


# on both sides of 96 KB of X (16 rows of 3072 columns, 8 of 6144, 4 of 12288) and of the least W of a call without a
# session; wide projections over few columns (a head, gate/up of a small model) stay with the streaming kernel
@pytest.mark.parametrize("M,N,K,split", [
    (16, 4096, 3072, False), (16, 4096, 3088, True), (9, 32000, 2048, False), (9, 32000, 1024, False), (16, 5632, 2048, False),
    (16, 1024, 5632, False), (16, 2048, 5632, True), (8, 6000, 6144, False), (8, 6000, 6160, True), (5, 4096, 6400, False), (4, 6000, 12288, False)])
def test_default_kernel(b200p, torch_cuda, M, N, K, split):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(N + K)
    W, X = (torch.randn(s, device="cuda", generator=g).bfloat16() for s in ((N, K), (M, K)))
    outs = []
    try:
        for kind in (-1, 3):
            b200p.set_tuning("runtime_skinny", kind)
            outs.append(b200p.skinny_gemm(W, torch.zeros((M, N), device="cuda"), x16=X, epilogue="acc32"))
    finally:
        b200p.set_tuning("runtime_skinny", -1)
    assert torch.equal(*outs) == split
