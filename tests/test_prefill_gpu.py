"""Prefill attention on tcgen05 (through the C ABI) against the oracle's cpu_prefill on
the reference's own test matrix and seeds, plus ragged and full-size cases.
Tolerance: max|delta| < 2e-2 for fp16/bf16 I/O (the reference gates at
0.15 and records 4e-5 .. 6.6e-4 for fp16)."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu
TOL = 2e-2


def dev16(torch, f32, kind):
    t = torch.from_numpy(np.ascontiguousarray(f32)).cuda()
    return t.half() if kind == "f16" else t.bfloat16()


@pytest.mark.parametrize("kind", ["bf16", "f16"])
@pytest.mark.parametrize("D", [128, 64])
def test_raw_score_tile_probe(b200p, torch_cuda, D, kind):
    """Known-answer probe of the tensor-core operand layouts: the raw S = Q.K^T tile the
    kernel holds in tensor memory equals a plain fp32 matmul of the same 16-bit inputs."""
    torch = torch_cuda
    g = torch.Generator(device="cuda"); g.manual_seed(5)
    dt = torch.bfloat16 if kind == "bf16" else torch.float16
    Q = (torch.randn(1, 1, 512, D, device="cuda", generator=g) * 0.5).to(dt)
    K = (torch.randn(1, 1, 512, D, device="cuda", generator=g) * 0.5).to(dt)
    V = (torch.randn(1, 1, 512, D, device="cuda", generator=g) * 0.5).to(dt)
    raw = torch.full((128, 128), float("nan"), device="cuda")
    O = b200p.prefill(Q, K, V, causal=False, raw_scores=raw)
    assert b200p.device_status() == 0
    ref = Q[0, 0, 256:384].float() @ K[0, 0, :128].float().T       # last 256-row block, its first tile
    assert torch.isfinite(raw).all()
    assert (raw - ref).abs().max().item() < 1e-3
    refO = torch.softmax((Q[0, 0].float() @ K[0, 0].float().T) / D ** 0.5, dim=-1) @ V[0, 0].float()
    assert (O[0, 0].float() - refO).abs().max().item() < TOL


# cdna3-prims/tests/validate_attention_api.hip:154-162: seed 42, N(0,0.5), Q then K then V
API_CASES = [(128, 256, 256, 2, 2, 1, 0), (128, 256, 256, 4, 2, 1, 0), (128, 256, 256, 2, 2, 1, 1), (128, 256, 256, 4, 2, 1, 1),
             (64, 256, 256, 2, 2, 1, 0), (128, 1024, 1024, 8, 8, 1, 0), (128, 512, 512, 32, 8, 1, 1)]


@pytest.mark.parametrize("kind", ["f16", "bf16"])
@pytest.mark.parametrize("D,sq,sk,nqh,nkvh,batch,causal", API_CASES)
def test_reference_api_matrix(b200p, torch_cuda, D, sq, sk, nqh, nkvh, batch, causal, kind):
    torch = torch_cuda
    q, k, v = orc.gen_qkv_mt19937(42, 0.5, batch * nqh * sq * D, batch * nkvh * sk * D)
    ref = orc.cpu_prefill(q, k, v, D, sq, sk, nqh, nkvh, batch, causal, threads=8)
    got = b200p.prefill(dev16(torch, q.reshape(batch, nqh, sq, D), kind), dev16(torch, k.reshape(batch, nkvh, sk, D), kind),
                        dev16(torch, v.reshape(batch, nkvh, sk, D), kind), causal=bool(causal))
    assert b200p.device_status() == 0
    err = np.abs(got.float().cpu().numpy() - ref).max()
    assert err < TOL, err
    if kind == "f16":
        assert err < 3e-3, err


# research/flash-attention-mi300x/fa_naive.hip:258-268 (and fa_dpp/fa_dme/fa_mfma2): B1 H8 S512 D64, seed 42, N(0,0.5),
# non-causal.  The reference checks head 0 only; all 8 heads here.
def test_step_config_all_heads(b200p, torch_cuda):
    torch = torch_cuda
    D, S, H = 64, 512, 8
    q, k, v = orc.gen_qkv_mt19937(42, 0.5, H * S * D, H * S * D)
    ref = orc.cpu_prefill(q, k, v, D, S, S, H, H, 1, 0, threads=8)
    got = b200p.prefill(dev16(torch, q.reshape(1, H, S, D), "f16"), dev16(torch, k.reshape(1, H, S, D), "f16"),
                        dev16(torch, v.reshape(1, H, S, D), "f16"))
    assert np.abs(got.float().cpu().numpy() - ref).max() < 1e-3


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("sq,sk,causal", [(128, 128, 1), (200, 333, 0), (130, 130, 1), (16, 64, 0), (384, 1000, 0), (640, 640, 1), (100, 700, 1)])
def test_ragged_shapes(b200p, torch_cuda, D, sq, sk, causal):
    torch = torch_cuda
    rng = np.random.default_rng(sq * 7 + sk)
    batch, nqh, nkvh = 2, 4, 2
    q = orc.round_to(rng.standard_normal((batch, nqh, sq, D)).astype(np.float32), "bf16")
    k = orc.round_to(rng.standard_normal((batch, nkvh, sk, D)).astype(np.float32), "bf16")
    v = orc.round_to(rng.standard_normal((batch, nkvh, sk, D)).astype(np.float32), "bf16")
    ref = orc.cpu_prefill(q, k, v, D, sq, sk, nqh, nkvh, batch, causal, threads=8)
    got = b200p.prefill(dev16(torch, q, "bf16"), dev16(torch, k, "bf16"), dev16(torch, v, "bf16"), causal=bool(causal))
    assert b200p.device_status() == 0
    assert np.abs(got.float().cpu().numpy() - ref).max() < TOL


def test_argument_errors(b200p, torch_cuda):
    torch = torch_cuda
    Q = torch.zeros(1, 2, 128, 96, device="cuda", dtype=torch.float16)
    with pytest.raises(b200p.B200PError) as e:
        b200p.prefill(Q, Q, Q)                             # D = 96 -> hipErrorInvalidValue in the reference
    assert e.value.status == -6
    Q = torch.zeros(1, 3, 128, 64, device="cuda", dtype=torch.float16)
    K = torch.zeros(1, 2, 128, 64, device="cuda", dtype=torch.float16)
    with pytest.raises(b200p.B200PError):
        b200p.prefill(Q, K, K)


def test_full_size_config_sampled(b200p, torch_cuda):
    """BASELINE config 3 at full size: batch 8, 32 heads, seq 4096, D 128, causal, bf16,
    N(0,1)*0.5.  Three (batch, head) units against the oracle, every unit through
    run-to-run identity and the row-sum property of softmax (V = 1 gives O = 1)."""
    torch = torch_cuda
    B, H, S, D = 8, 32, 4096, 128
    g = torch.Generator(device="cuda"); g.manual_seed(0xB203)
    Q = (torch.randn(B, H, S, D, device="cuda", generator=g) * 0.5).bfloat16()
    K = (torch.randn(B, H, S, D, device="cuda", generator=g) * 0.5).bfloat16()
    V = (torch.randn(B, H, S, D, device="cuda", generator=g) * 0.5).bfloat16()
    O = b200p.prefill(Q, K, V, causal=True)
    assert b200p.device_status() == 0
    for (b, h) in ((0, 0), (3, 17), (7, 31)):
        ref = orc.cpu_prefill(Q[b, h].float().cpu().numpy(), K[b, h].float().cpu().numpy(), V[b, h].float().cpu().numpy(),
                              D, S, S, 1, 1, 1, 1, threads=1)[0, 0]
        assert np.abs(O[b, h].float().cpu().numpy() - ref).max() < TOL
    assert torch.equal(b200p.prefill(Q, K, V, causal=True), O)
    ones = torch.ones_like(V)
    O1 = b200p.prefill(Q, K, ones, causal=True)
    assert (O1.float() - 1.0).abs().max().item() < 1e-2


@pytest.mark.parametrize("causal", [1, 0])
@pytest.mark.parametrize("D", [128, 64])
def test_more_work_items_than_sms(b200p, torch_cuda, D, causal):
    """The kernel's CTAs are persistent (one per SM) and draw 256-row work items from a device
    counter.  Here there are more items than SMs (2 x 20 heads x 5 query blocks = 200), of
    unequal length under the causal mask, a ragged last block and GQA; every output row against
    the oracle; the one-CTA-per-item launch (knob bit 1) gives the same bits."""
    torch = torch_cuda
    rng = np.random.default_rng(41 + D + causal)
    batch, nqh, nkvh, sq = 2, 20, 4, 1200
    q = orc.round_to((rng.standard_normal((batch, nqh, sq, D)) * 0.5).astype(np.float32), "bf16")
    k = orc.round_to((rng.standard_normal((batch, nkvh, sq, D)) * 0.5).astype(np.float32), "bf16")
    v = orc.round_to((rng.standard_normal((batch, nkvh, sq, D)) * 0.5).astype(np.float32), "bf16")
    ref = orc.cpu_prefill(q, k, v, D, sq, sq, nqh, nkvh, batch, causal, threads=8)
    Q, K, V = dev16(torch, q, "bf16"), dev16(torch, k, "bf16"), dev16(torch, v, "bf16")
    got = b200p.prefill(Q, K, V, causal=bool(causal))
    assert b200p.device_status() == 0
    assert np.abs(got.float().cpu().numpy() - ref).max() < TOL
    b200p.set_tuning("prefill_variant", 2)
    try:
        assert torch.equal(b200p.prefill(Q, K, V, causal=bool(causal)), got)
    finally:
        b200p.set_tuning("prefill_variant", -1)


def test_launches_on_two_streams_do_not_share_a_work_counter(b200p, torch_cuda):
    """Two prefill launches in flight at once on different streams each draw their items from
    their own counter slot: both results equal the single-stream ones."""
    torch = torch_cuda
    g = torch.Generator(device="cuda"); g.manual_seed(77)
    mk = lambda b, h, s: (torch.randn(b, h, s, 128, device="cuda", generator=g) * 0.5).bfloat16()
    A = [mk(4, 16, 2048) for _ in range(3)]
    Bq = [mk(2, 24, 1536) for _ in range(3)]
    ref_a = b200p.prefill(*A, causal=True)
    ref_b = b200p.prefill(*Bq, causal=True)
    torch.cuda.synchronize()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    outs = []
    for _ in range(3):
        with torch.cuda.stream(s1):
            oa = b200p.prefill(*A, causal=True)
        with torch.cuda.stream(s2):
            ob = b200p.prefill(*Bq, causal=True)
        outs.append((oa, ob))
    torch.cuda.synchronize()
    for oa, ob in outs:
        assert torch.equal(oa, ref_a) and torch.equal(ob, ref_b)
    assert b200p.device_status() == 0


# rows that end inside, at and just past a tile and a pair of tiles; runs of rows that wrap to the next head inside a tile; one
# row per head; fewer and more items than SMs; keys of one tile and of many
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("batch,heads,kv,S", [(1, 4, 1, 1), (2, 8, 2, 20), (1, 8, 1, 127), (1, 4, 4, 128), (3, 8, 2, 129), (1, 6, 2, 255), (2, 4, 1, 257), (1, 8, 4, 385), (2, 32, 4, 555), (1, 8, 8, 700)])
def test_work_items_of_every_form_give_the_same_bits(b200p, torch_cuda, D, causal, batch, heads, kv, S):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(S * 7 + heads)
    q, k, v = (torch.randn((batch, h, S, D), device="cuda", generator=g).bfloat16() for h in (heads, kv, kv))
    outs = []
    try:
        for variant in (16, 20, 24, 28, -1):                     # pairs, single tiles, both packed, the rule's choice
            b200p.set_tuning("prefill_variant", variant)
            outs.append(b200p.prefill(q, k, v, causal=causal))
    finally:
        b200p.set_tuning("prefill_variant", -1)
    for o in outs[1:]:
        assert torch.equal(o, outs[0])
    qd, kd, vd = q.double(), k.double().repeat_interleave(heads // kv, 1), v.double().repeat_interleave(heads // kv, 1)
    s = qd @ kd.transpose(-1, -2) * D ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    assert (outs[0].double() - s.softmax(-1) @ vd).abs().max() < 2e-2


# lengths whose last tile is not full, groups, sizes at which the heads of a group would fit fewer rounds of items as one run of rows
@pytest.mark.parametrize("batch,heads,kv,S,D", [(2, 32, 4, 555, 64), (2, 32, 8, 1111, 128), (8, 8, 1, 1111, 64), (8, 64, 8, 128, 64), (8, 64, 8, 384, 64), (1, 8, 8, 300, 64)])
def test_values_behind_a_rows_position_do_not_reach_it(b200p, torch_cuda, batch, heads, kv, S, D):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn((batch, h, S, D), device="cuda", generator=g).bfloat16() for h in (heads, kv, kv))
    clean = b200p.prefill(q, k, v, causal=True)
    for bad in (float("nan"), float("inf")):
        v2 = v.clone(); v2[:, :, S - 3:] = bad
        first = (S - 3) // 128 * 128                                 # rows that share a tile of keys with the bad ones may see 0 x bad
        assert torch.equal(b200p.prefill(q, k, v2, causal=True)[:, :, :first], clean[:, :, :first])


# rows wider than the head, other pitches for O than for Q, other lengths of Q and K: the heads of a group still follow one
# another, so that they can be one run of rows; and token-major rows, where they cannot
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D,batch,heads,kv,seqQ,seqK,q_pitch,o_pitch", [
    (64, 2, 8, 2, 77, 200, 80, 64), (64, 1, 32, 4, 555, 130, 64, 72), (128, 2, 6, 2, 130, 700, 136, 160), (64, 2, 4, 1, 1, 300, 72, 64), (128, 1, 8, 1, 300, 1, 128, 128), (64, 2, 8, 4, 96, 96, 0, 0)])
def test_packed_rows_of_strided_views(b200p, torch_cuda, causal, D, batch, heads, kv, seqQ, seqK, q_pitch, o_pitch):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(seqQ)
    if q_pitch:
        view = lambda t: t[..., :D]
        qb, shape = torch.randn((batch, heads, seqQ, q_pitch), device="cuda", generator=g).bfloat16(), (batch, heads, seqQ, o_pitch)
    else:                                                                  # [batch, seq, heads, D]
        view = lambda t: t.transpose(1, 2)
        qb, shape = torch.randn((batch, seqQ, heads, D), device="cuda", generator=g).bfloat16(), (batch, seqQ, heads, D)
    k, v = (torch.randn((batch, kv, seqK, D), device="cuda", generator=g).bfloat16() for _ in range(2))
    outs = []
    try:
        for variant in (16, 20, 24, 28, -1):                     # as in test_work_items_of_every_form_give_the_same_bits
            b200p.set_tuning("prefill_variant", variant)
            ob = torch.full(shape, 7.0, device="cuda").bfloat16()
            b200p.prefill_strided(view(qb), k, v, view(ob), causal=causal)
            outs.append(ob)
    finally:
        b200p.set_tuning("prefill_variant", -1)
    for o in outs[1:]:
        assert torch.equal(o, outs[0])
    if q_pitch:
        assert (outs[0][..., D:] == 7.0).all()
    qd, kd, vd = view(qb).double(), k.double().repeat_interleave(heads // kv, 1), v.double().repeat_interleave(heads // kv, 1)
    s = qd @ kd.transpose(-1, -2) * D ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(seqQ, seqK, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    assert (view(outs[0]).double() - s.softmax(-1) @ vd).abs().max() < 2e-2      # 16-bit weights and outputs of size up to 4
