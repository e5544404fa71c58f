"""Decode steps whose norms are folded into the projections around them (bf16): x * w rounded by whoever adds to x, 1 / rms from
partial sums.  Sizes where the partial sums end inside a vector, pass the vectors a lane loads at once or are made by the kernel that
splits K; one and two fragments of rows; sums that only the GEMM takes; and rows of X by bulk copies, with half stages where X leaves room
for one whole stage only."""
import numpy as np
import pytest

from oracle import runtime_ref as rr
import test_hybrid_gpu as hybrid
from test_hybrid_gpu import knob, opened  # noqa: F401 (fixtures)
from test_runtime_gpu import check_logits, to_device
from test_skinny_sessions_gpu import llama

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,batch", [(16, 1), (48, 9), (144, 2), (144, 16), (528, 7), (1040, 8), (2064, 3), (4112, 2), (4112, 16)])
def test_sums_of_every_width(b200p, torch_cuda, hidden, batch):
    cfg = llama(4, 2, 64, ffn=144, hidden=hidden)
    # rows of the projections near unit length, so that the softmax does not magnify where x * w was rounded
    w = rr.make_weights(cfg, seed=3, kind="bf16", std=min(0.05, hidden ** -0.5), bias=batch % 2 == 0)
    ref, sess = rr.RefSession(cfg, w, 16, batch, "bf16"), b200p.Session(cfg, to_device(torch_cuda, w, "bf16"), 16, batch)
    rng = np.random.default_rng(batch)
    ids = rng.integers(0, cfg["vocab_size"], (batch, 5)).astype(np.int32)
    check_logits(sess.prefill_logits(ids), ref.prefill_logits(ids))
    for _ in range(3):
        nxt = rng.integers(0, cfg["vocab_size"], batch).astype(np.int32)
        check_logits(sess.step_logits(nxt), ref.step_logits(nxt))
    sess.close()
    assert b200p.device_status() == 0


# x * w is outside fp16's range (its sessions normalise first), and far above 1 in bf16
@pytest.mark.parametrize("kind", ["f16", "bf16"])
def test_large_residual(b200p, torch_cuda, kind):
    cfg = llama(4, 2, 64, ffn=256, hidden=256)
    w = rr.make_weights(cfg, seed=5, kind=kind, std=0.05, bias=False)
    w["embed_tokens"] = w["embed_tokens"] * np.float32(32768)
    w["final_norm"] = w["final_norm"] * np.float32(64)
    ref, sess = rr.RefSession(cfg, w, 8, 3, kind), b200p.Session(cfg, to_device(torch_cuda, w, kind), 8, 3)
    ids = np.arange(9, dtype=np.int32).reshape(3, 3)
    check_logits(sess.prefill_logits(ids), ref.prefill_logits(ids))
    nxt = np.array([4, 8, 15], np.int32)
    check_logits(sess.step_logits(nxt), ref.step_logits(nxt))
    sess.close()


@pytest.mark.parametrize("M,N,K", [(1, 48, 16), (2, 40, 5632), (7, 33, 2064), (8, 64, 6144), (9, 100, 3008), (16, 2400, 3072), (16, 64, 2048)])
def test_rows_by_copies(b200p, torch_cuda, M, N, K):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(K + M)
    W, wide = (torch.randn(s, device="cuda", generator=g).bfloat16() for s in ((N, K), (M, K + 24)))
    X, out = wide[:, :K], torch.zeros((M, N), device="cuda")
    b200p.skinny_gemm(W, out, x16=X, epilogue="store32")
    want = X.double() @ W.double().T
    # products of 16-bit values are exact in fp32; K sums of them, each rounded: error below K eps of the sum of magnitudes, sqrt(K) of it in the mean
    bound = 2.0 ** -24 * 8 * K ** 0.5 * (X.double().abs() @ W.double().abs().T)
    assert ((out - want).abs() <= bound).all()


# an MLP's rows that no kernel with the form takes: the sum comes from the GEMM, its folded form from a kernel of its own.  The first
# layer's MLP is followed by a norm and the last one's by the head; 5 and 8 rows, 16 rows
@pytest.mark.parametrize("batch", [5, 8, 16])
def test_sums_of_the_gemm(b200p, torch_cuda, opened, knob, batch):  # noqa: F811
    knob("skinny_cluster", 1)
    s, cfg = opened("wide_mlp", "bf16", 64, batch), hybrid.CONFIGS["wide_mlp"]
    ids = [hybrid.tokens(cfg, 9, b) for b in range(batch)]
    got = [s.extend([i[:3] for i in ids], [2])]
    for t in range(3, 9):
        got.append(s.extend([i[t:t + 1] for i in ids], [0]))
    for b in range(batch):
        hybrid.check(np.concatenate([g[b] for g in got]), hybrid.reference("wide_mlp", ids[b])[2:], "bf16", b)
