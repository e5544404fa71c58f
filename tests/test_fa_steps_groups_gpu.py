"""Step kernels whose warps are two groups that take every other tile of keys: one tile (one group), an odd number of tiles, a last tile of
one key in either group's turn, scores that differ by much between the groups, and more CTAs than SMs (step 2 has one buffer of V, in 16 bits and 128 columns one of K too)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("S,heads", [(1, 1), (63, 3), (64, 2), (65, 1), (128, 1), (129, 5), (192, 1), (193, 40), (321, 2), (640, 8),
                                     (128, 24), (192, 16), (256, 12), (320, 8), (384, 8)])                    # (128 ... 384: more CTAs than SMs)
def test_groups(b200p, torch_cuda, S, heads, D):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(S + D)
    for dtype, eps in ((torch.float32, 2.0 ** -23), (torch.float16, 2.0 ** -10), (torch.bfloat16, 2.0 ** -7)):
        if dtype != torch.float32 and S % 64:
            continue
        q, k, v = (torch.randn((1, heads, S, D), device="cuda", generator=g) for _ in range(3))
        k[:, :, S // 2:] *= 4                                    # the running maxima of the groups end far apart
        q, k, v = (x.to(dtype) for x in (q, k, v))
        p = torch.softmax(q.double() @ k.double().transpose(2, 3) * D ** -0.5, -1)
        want = p @ v.double()
        # fp32 sums of D products and S weights, exponentials of arguments up to about 50 off by eps each, and the output's own rounding
        bound = (100 * 2.0 ** -23 + eps) * (p @ v.double().abs()) + 1e-7
        if dtype != torch.float32:
            bound = bound + 2.0 ** -16 * (p @ v.double().abs())  # __expf
        outs = [b200p.fa_step(s, q, k, v) for s in ("naive", "dpp", "dme")]
        for o in outs:
            assert ((o - want).abs() <= bound).all(), (dtype, ((o - want).abs() / bound).max())
        assert torch.equal(outs[1], outs[2])
