"""Decode steps of sessions on the projection kernel that splits K over a cluster: the forms that only sessions launch (rotated
Q/K/V with the scatter into the cache, rotated query pairs, the prologue that adds the last sublayer's output), and what a
session does where that kernel cannot run."""
import numpy as np
import pytest

from oracle import runtime_ref as rr
from test_latent_gpu import check, opened, reference, tokens  # noqa: F401 (opened is a fixture)
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


# rows that fit the register kernel, but neither two stages of the streaming one beside them nor one CTA of the cluster kernel: the
# down projection's, with 16 and with 8 sequences, and the O projection's
@pytest.mark.parametrize("heads,kv,ffn,batch", [(4, 2, 5632, 16), (4, 2, 9856, 8), (88, 8, 512, 16)])
def test_rows_that_no_kernel_with_a_folded_norm_takes(b200p, torch_cuda, heads, kv, ffn, batch):
    b200p.set_tuning("skinny_cluster", 1)
    steps(b200p, torch_cuda, llama(heads, kv, 64, ffn=ffn, hidden=256), "bf16", False, batch)


# heads whose rows fill the 128-row tiles and not, one head a tile and two, biases, one and two fragments of rows
@pytest.mark.parametrize("cluster", [0, 1, 3, 8])
@pytest.mark.parametrize("heads,kv,D,kind,bias,batch", [(8, 2, 64, "bf16", False, 1), (3, 3, 64, "f16", True, 3), (4, 1, 128, "bf16", True, 9), (5, 5, 64, "bf16", True, 16),
                                                        (3, 1, 128, "f16", False, 16)])
def test_rotated_projections(b200p, torch_cuda, cluster, heads, kv, D, kind, bias, batch):
    b200p.set_tuning("runtime_skinny", 3)
    b200p.set_tuning("skinny_cluster", cluster)
    steps(b200p, torch_cuda, llama(heads, kv, D), kind, bias, batch)


# 1 .. 4 rows form the residual sum in the next projection's prologue, more in a kernel of its own; then single tokens, which
# read the cache that those rows wrote
@pytest.mark.parametrize("cluster", [0, 1, 2, 8])
@pytest.mark.parametrize("name", ["odd", "many_heads", "real_heads", "wide_mlp"])
def test_latent_decoder(b200p, opened, name, cluster):  # noqa: F811
    from test_latent_gpu import CONFIGS, run
    b200p.set_tuning("runtime_skinny", 3)
    b200p.set_tuning("skinny_cluster", cluster)
    s, ids = opened(name, "bf16"), tokens(CONFIGS[name], 20, 2)
    want = reference(name, ids)
    for n in (1, 2, 3, 4, 5, 9, 16):
        check(run(s, ids, [n, 1]), want, "bf16", n)
