"""Decode attention whose splits are one thread-block cluster (513 .. 2048 keys): edges of the range and of the tiles, clusters of two to
eight, strided caches, key counts that leave splits empty, scratch sized for one split only, and sessions of such lengths."""
import numpy as np
import pytest

from oracle import runtime_ref as rr
from test_runtime_gpu import check_logits, to_device
from test_skinny_sessions_gpu import llama

pytestmark = pytest.mark.gpu


def expect(torch, q, K, V, N):
    """In 64 bits, and a bound: softmax weights and outputs of 11 (8) bits, scores of fp32 sums."""
    g = q.shape[1] // K.shape[1]
    k, v = (x[:, :, :N].double().repeat_interleave(g, 1) for x in (K, V))
    p = torch.softmax((k @ q.double()[..., None])[..., 0] * q.shape[-1] ** -0.5, -1)[:, :, None]
    return (p @ v)[:, :, 0], (2.0 ** (-10 if q.dtype == torch.float16 else -7) + 1e-4) * (p @ v.abs())[:, :, 0]


def case(torch, B, H, G, cap, D, dtype):
    g = torch.Generator(device="cuda").manual_seed(B * cap + D)
    return [torch.randn(s, device="cuda", generator=g).to(dtype) for s in ((B, H, D), (B, G, cap, D), (B, G, cap, D))]


@pytest.mark.parametrize("B,H,G,D", [(1, 4, 4, 64), (1, 32, 8, 128), (3, 16, 1, 64), (5, 28, 7, 128), (8, 32, 8, 64)])
@pytest.mark.parametrize("N", [512, 513, 640, 1000, 1024, 1025, 1999, 2048, 2049])
def test_lengths(b200p, torch_cuda, B, H, G, D, N):
    torch = torch_cuda
    for dtype in (torch.float16, torch.bfloat16):
        q, K, V = case(torch, B, H, G, 2100, D, dtype)
        got = b200p.decode(q, K, V, N=N)
        want, bound = expect(torch, q, K, V, N)
        assert ((got - want).abs() <= bound).all()
        small = torch.empty(b200p.decode_workspace(q, K[:, :, :512].contiguous(), 512).numel(), dtype=torch.uint8, device="cuda")
        if N <= 1024:                                            # scratch of one split
            assert ((b200p.decode(q, K, V, N=N, workspace=small) - want).abs() <= bound).all()
        assert ((b200p.decode_noalloc(q, K, V, N=N) - want).abs() <= bound).all()


def test_counts_on_the_device(b200p, torch_cuda):
    torch = torch_cuda
    q, K, V = case(torch, 2, 16, 4, 1500, 128, torch.bfloat16)
    ws = b200p.decode_workspace(q, K, 1500)
    for n in (1, 127, 128, 129, 700, 1281, 1500):
        got = b200p.decode_dyn(q, K, V, torch.tensor([n], dtype=torch.int32, device="cuda"), N=1500, workspace=ws)
        want, bound = expect(torch, q, K, V, n)
        assert ((got - want).abs() <= bound).all(), n
        assert b200p.workspace_status(ws) == 0


# one split up to 1024 keys, one per 256 above (few units): what a caller may have sized, whichever form the splits take
@pytest.mark.parametrize("N,splits", [(700, 1), (1024, 1), (1025, 5), (2000, 8)])
def test_scratch_of_the_stated_size_is_enough_and_less_is_refused(b200p, torch_cuda, N, splits):
    torch = torch_cuda
    q, K, V = case(torch, 1, 32, 32, 2100, 64, torch.float16)
    ws = b200p.decode_workspace(q, K, N)
    up = lambda n: -(-n // 256) * 256
    assert ws.numel() == 256 + up(32 * 4) + up(32 * splits * 8) + 32 * splits * 64 * 4
    want, bound = expect(torch, q, K, V, N)
    assert ((b200p.decode(q, K, V, N=N, workspace=ws) - want).abs() <= bound).all()
    with pytest.raises(b200p.B200PError) as e:
        b200p.decode(q, K, V, N=N, workspace=ws[:-256])
    assert e.value.status == -7


# bounds on both sides of the one below which a count on the device takes no cluster
@pytest.mark.parametrize("bound", [513, 1000, 1024, 1025, 2048, 2049])
@pytest.mark.parametrize("B,H,G,D", [(1, 32, 8, 128), (5, 8, 8, 64)])
def test_counts_below_the_bound(b200p, torch_cuda, bound, B, H, G, D):
    torch = torch_cuda
    q, K, V = case(torch, B, H, G, 2100, D, torch.float16)
    for n in (1, 60, 128, 300, 512, 513, bound):
        got = b200p.decode_dyn(q, K, V, torch.tensor([n], dtype=torch.int32, device="cuda"), N=bound)
        want, limit = expect(torch, q, K, V, n)
        assert ((got - want).abs() <= limit).all(), n


@pytest.mark.parametrize("max_seq,batch", [(1025, 16), (1100, 2), (2047, 8)])
def test_sessions(b200p, torch_cuda, max_seq, batch):
    """(Their scratch was sized at 1024 keys and every step refused.)"""
    cfg = llama(16, 4, 64, ffn=256, hidden=256)
    w = rr.make_weights(cfg, seed=9, kind="bf16", std=0.05, bias=False)
    ref, sess = rr.RefSession(cfg, w, max_seq, batch, "bf16"), b200p.Session(cfg, to_device(torch_cuda, w, "bf16"), max_seq, batch)
    rng = np.random.default_rng(max_seq)
    ids = rng.integers(0, 300, (batch, 140)).astype(np.int32)
    check_logits(sess.prefill_logits(ids), ref.prefill_logits(ids))
    for _ in range(2):
        nxt = rng.integers(0, 300, batch).astype(np.int32)
        check_logits(sess.step_logits(nxt), ref.step_logits(nxt))
    sess.close()
