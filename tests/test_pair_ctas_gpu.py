"""Projections of 149 to 296 groups of rows, a stage long: one CTA per group, two on an SM.  The ends of that range on both sides, K up to
a whole stage and with a remainder, every prologue and epilogue that launches it, and that what is launched so is the bounded form."""
import os
import re

import numpy as np
import pytest

from oracle import runtime_ref as rr
from test_latent_gpu import check, config, mixer, opened, reference, run, tokens  # noqa: F401 (opened is a fixture)
from test_runtime_gpu import check_logits, to_device
from test_skinny_sessions_gpu import llama

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "amd-incstinct-labs_b200", "csrc")


def test_one_group_launches_take_the_bounded_kernel():
    src = open(os.path.join(CSRC, "skinny_gemm.cuh")).read()
    params, bound = re.search(r"template <([^<>]*)>\n__global__ void __launch_bounds__\(kSkinnyStreamThreads, (.*?)\)\nskinny_stream_kernel", src).groups()
    assert params.endswith("bool PAIR") and bound == "PAIR ? 2 : 1"
    assert re.search(r"if \(one_group_ctas\) sk = skinny_stream_kernel<T, PRO, EPI, MH, true>;", src)


@pytest.mark.gpu
@pytest.mark.parametrize("groups", [148, 149, 296, 297])
@pytest.mark.parametrize("M,K", [(1, 2048), (3, 64), (8, 1040), (5, 2048), (2, 2064)])
def test_plain_projections(b200p, torch_cuda, groups, M, K):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(groups + K)
    W, X = (torch.randn(s, device="cuda", generator=g).bfloat16() for s in ((16 * groups - 5, K), (M, K)))
    out, start = torch.empty((M, W.shape[0]), device="cuda"), torch.randn((M, W.shape[0]), device="cuda", generator=g)
    want, size = X.double() @ W.double().T, X.double().abs() @ W.double().abs().T
    bound = 2.0 ** -24 * 8 * K ** 0.5 * size                       # sums of K exact products, sqrt(K) roundings in the mean
    b200p.skinny_gemm(W, out, x16=X, epilogue="store32")
    assert ((out - want).abs() <= bound).all()
    acc = start.clone()
    b200p.skinny_gemm(W, acc, x16=X, epilogue="acc32")
    assert ((acc - start.double() - want).abs() <= bound + 2.0 ** -23 * (start.abs() + size)).all()
    # gated: 8 rows of each half per group
    W2 = torch.randn((2 * (8 * groups - 3), K), device="cuda", generator=g).mul(K ** -0.5).bfloat16()
    a, b = (X.double() @ W2.double().T).chunk(2, 1)
    act = torch.empty((M, 8 * groups - 3), device="cuda", dtype=torch.bfloat16)
    b200p.skinny_gemm(W2, act, x16=X, epilogue="gelu16")
    want = torch.nn.functional.gelu(a, approximate="tanh") * b
    assert ((act - want).abs() <= 2.0 ** -8 * want.abs() + 2e-4).all()


# adds of 150 and 296 groups with the folded norm, gated projections of 150 and 296 that read it; fp16 normalises in the projection
@pytest.mark.gpu
@pytest.mark.parametrize("hidden,ffn,batch,kind", [(2400, 1200, 1, "bf16"), (2400, 1200, 7, "f16"), (256, 2368, 8, "bf16"), (4736, 160, 3, "bf16")])
def test_sessions(b200p, torch_cuda, hidden, ffn, batch, kind):
    cfg = llama(4, 2, 64, ffn=ffn, hidden=hidden)
    w = rr.make_weights(cfg, seed=7, kind=kind, std=min(0.05, hidden ** -0.5), bias=False)
    ref, sess = rr.RefSession(cfg, w, 16, batch, kind), b200p.Session(cfg, to_device(torch_cuda, w, kind), 16, batch)
    rng = np.random.default_rng(batch)
    ids = rng.integers(0, cfg["vocab_size"], (batch, 3)).astype(np.int32)
    check_logits(sess.prefill_logits(ids), ref.prefill_logits(ids))
    for _ in range(3):
        nxt = rng.integers(0, cfg["vocab_size"], batch).astype(np.int32)
        check_logits(sess.step_logits(nxt), ref.step_logits(nxt))
    sess.close()
    assert b200p.device_status() == 0


# rotated queries of 13 heads (156 groups) and 24 (288) from latents of 768 and 2000 columns; an MLP of 150 groups behind the post-norm prologue
@pytest.mark.gpu
@pytest.mark.parametrize("heads,q", [(13, 768), (24, 2000)])
def test_latent(b200p, opened, heads, q):  # noqa: F811
    name = f"queries of {heads} heads"
    cfg = config(96, 90, [("", mixer(heads, 128, 64, 32, 64, q), 1200), ("_2", mixer(heads, 128, 64, 32, 64, q), 1200)])
    ids = tokens(cfg, 12, heads)
    s = opened(name, "bf16", cfg=cfg)
    for n in (1, 2, 4, 8):
        check(run(s, ids, [n]), reference(name, ids, cfg), "bf16", n)
