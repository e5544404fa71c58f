"""Decode steps of sessions on the projection kernel that splits K over a cluster, and what a session does where that kernel
cannot run."""
import numpy as np
import pytest

from oracle import runtime_ref as rr
from test_runtime_gpu import check_logits, to_device

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def knobs(b200p):
    yield
    for k in ("runtime_skinny", "skinny_cluster"):
        b200p.set_tuning(k, -1)


def llama(heads, kv, D, ffn=1024, hidden=512):
    return dict(n_layers=2, hidden=hidden, n_heads=heads, n_kv_heads=kv, head_dim=D, ffn_dim=ffn, vocab_size=300, rope_theta=10000.0)


def steps(b200p, torch, cfg, kind, bias, batch, T=5, n=3):
    """Prompt and teacher-forced steps: the later ones read what the earlier ones scattered into the cache."""
    w = rr.make_weights(cfg, seed=3, kind=kind, std=0.05, bias=bias)
    ref, sess = rr.RefSession(cfg, w, 16, batch, kind), b200p.Session(cfg, to_device(torch, w, kind), 16, batch)
    rng = np.random.default_rng(batch)
    ids = rng.integers(0, cfg["vocab_size"], (batch, T)).astype(np.int32)
    check_logits(sess.prefill_logits(ids), ref.prefill_logits(ids))
    for _ in range(n):
        nxt = rng.integers(0, cfg["vocab_size"], batch).astype(np.int32)
        check_logits(sess.step_logits(nxt), ref.step_logits(nxt))
    sess.close()
    assert b200p.device_status() == 0


def test_rows_too_long_for_every_allowed_split_take_the_gemm(b200p, torch_cuda):
    """8 rows of 12304 columns fit no streaming kernel, and one CTA of the cluster kernel neither."""
    b200p.set_tuning("skinny_cluster", 1)
    steps(b200p, torch_cuda, llama(4, 2, 64, ffn=12304, hidden=256), "bf16", False, 8)
