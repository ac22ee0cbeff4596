"""The rows next to the hot path, on the GPU (``-m gpu``), through the C ABI: causal masks over
unequal lengths in both alignments, the split-KV decode forward, dropout with a Philox mask
regenerated by the oracle and the bounded wait's give-up path.  Tolerances as everywhere: 2e-2 on 16-bit tensors, 1e-3 on fp32 and lse."""

import os

import numpy as np
import pytest
import torch

from oracle import restatement as R
from oracle import sdpa_oracle as O
from oracle.philox import keep_mask
from tests.helpers import TOL_16BIT, TOL_FP32, TOL_LSE, assert_within
from torch_mojo_backend_b200 import _lib, raw

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def tol_for(dtype):
    return TOL_FP32 if dtype == torch.float32 else TOL_16BIT


def draw(dtype, B, Hq, Hkv, Sq, Sk, D, seed):
    g = torch.Generator().manual_seed(seed)
    q = (torch.randn(B, Hq, Sq, D, generator=g) * 0.5).to(dtype)
    k = (torch.randn(B, Hkv, Sk, D, generator=g) * 0.5).to(dtype)
    v = (torch.randn(B, Hkv, Sk, D, generator=g) * 0.5).to(dtype)
    dout = torch.randn(B, Hq, Sq, D, generator=g).to(dtype)
    return q, k, v, dout


def run(q, k, v, dout, causal, scale, simt=False, dropout=None):
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    qc, kc, vc = q.cuda(), k.cuda(), v.cuda()
    out, lse = raw.flash_fwd(qc, kc, vc, causal=causal, scale=scale, status=status, simt=simt, dropout=dropout)
    dq, dk, dv = raw.flash_bwd(dout.cuda(), qc, kc, vc, out, lse, causal=causal, scale=scale, status=status, simt=simt,
                               dropout=dropout)
    torch.cuda.synchronize()
    assert int(status.item()) == 0, f"kernel status word 0x{int(status.item()) & 0xffffffff:x}"
    return out, lse, dq, dk, dv


def t64(x):
    return x.float().numpy().astype(np.float64)


# Forward calls with few (batch, head, query tile) units.  The K/V blocks of the first three, the fifth and
# the sixth are dealt to the CTAs of clusters (unequal shares, shares without a block, ragged edges); the
# others are too short for that.
SPLIT = [
    # dtype, B, Hq, Hkv, Sq, Sk, D, mode
    (torch.bfloat16, 1, 2, 1, 256, 4224, 128, 2),
    (torch.float16, 1, 3, 3, 300, 2000, 128, 2),
    (torch.bfloat16, 1, 8, 8, 1024, 1024, 128, 1),
    (torch.float16, 1, 2, 1, 600, 300, 128, 2),
    (torch.bfloat16, 1, 4, 4, 129, 1153, 64, 2),
    (torch.float16, 2, 2, 2, 1000, 1000, 64, 1),
    (torch.bfloat16, 1, 2, 2, 33, 700, 64, 0),
    (torch.bfloat16, 1, 2, 2, 20, 1025, 128, 1),
    (torch.float16, 1, 4, 2, 257, 1, 128, 0),
]


@pytest.mark.parametrize("dtype,B,Hq,Hkv,Sq,Sk,D,mode", SPLIT)
def test_forward_split_over_clusters(dtype, B, Hq, Hkv, Sq, Sk, D, mode):
    q, k, v, _ = draw(dtype, B, Hq, Hkv, Sq, Sk, D, Sq + Sk)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.full((B, Sq, Hq, D), float("nan"), dtype=dtype, device="cuda").transpose(1, 2)
    _, lse = raw.flash_fwd(q.cuda(), k.cuda(), v.cuda(), causal=mode, scale=D ** -0.5, out=out, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    ref_out, ref_lse = O.sdpa_forward(q, k, v, mode, D ** -0.5)
    assert_within("out", out, ref_out, TOL_16BIT, dtype)
    sees = torch.arange(Sq) + (Sk - Sq if mode == 2 else 0) >= 0    # a row without a key has lse -inf
    seen = sees.expand(B, Hq, Sq)
    assert torch.equal(seen, torch.isfinite(lse.cpu()))
    assert (lse.cpu() - ref_lse)[seen].abs().max().item() < TOL_LSE


# every cluster size at both head dimensions, rows without a key among them
SPLIT_COUNTS = [
    # dtype, B, Hq, Hkv, Sq, Sk, D, mode, CTAs per query unit
    (torch.bfloat16, 1, 8, 8, 1584, 1982, 128, 0, 2),
    (torch.float16, 1, 6, 3, 1300, 1200, 128, 2, 2),
    (torch.float16, 1, 10, 5, 1111, 1500, 64, 0, 2),
    (torch.bfloat16, 1, 8, 8, 1472, 1662, 64, 2, 2),
    (torch.bfloat16, 1, 4, 4, 1537, 1000, 128, 2, 4),
    (torch.float16, 1, 2, 1, 2600, 2300, 64, 2, 4),
    (torch.float16, 1, 2, 2, 1500, 1300, 128, 2, 8),
    (torch.bfloat16, 1, 1, 1, 2600, 2300, 64, 2, 8),
]


@pytest.mark.parametrize("dtype,B,Hq,Hkv,Sq,Sk,D,mode,splits", SPLIT_COUNTS)
def test_forward_split_over_each_cluster_size(dtype, B, Hq, Hkv, Sq, Sk, D, mode, splits):
    assert _lib.fwd_splits(B, Hq, Sq, Sk, D, _lib.BF16, mode) == splits
    q, k, v, _ = draw(dtype, B, Hq, Hkv, Sq, Sk, D, Sq + Sk)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, lse = raw.flash_fwd(q.cuda(), k.cuda(), v.cuda(), causal=mode, scale=D ** -0.5, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    ref_out, ref_lse = O.sdpa_forward(q, k, v, mode, D ** -0.5)
    keyless = max(0, Sq - Sk) if mode == 2 else 0     # these rows are 0 with lse -inf
    assert not bool(out[:, :, :keyless].any()) and bool((lse[:, :, :keyless] == -float("inf")).all())
    assert_within("out", out[:, :, keyless:], ref_out[:, :, keyless:], TOL_16BIT, dtype)
    assert (lse.cpu() - ref_lse)[:, :, keyless:].abs().max().item() < TOL_LSE


@pytest.mark.parametrize("Hq,Sq,Sk,D,mode", [(1, 256, 4096, 128, 2), (2, 300, 3000, 64, 0), (64, 1024, 1024, 128, 1)])
def test_a_launch_whose_status_word_is_set_writes_nothing(Hq, Sq, Sk, D, mode):
    """Whether the K/V blocks are dealt to clusters (the first two shapes) or not."""
    q, k, v, _ = draw(torch.bfloat16, 1, Hq, Hq, Sq, Sk, D, 3)
    qc, kc, vc = q.cuda(), k.cuda(), v.cuda()
    status = torch.full((1,), 0x57410100, dtype=torch.int32, device="cuda")
    out, lse = torch.full_like(qc, 7.0), torch.full((1, Hq, Sq), 7.0, device="cuda")
    raw.flash_fwd(qc, kc, vc, causal=mode, out=out, lse=lse, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0x57410100
    assert bool((out == 7.0).all()) and bool((lse == 7.0).all())
    status.zero_()
    raw.flash_fwd(qc, kc, vc, causal=mode, out=out, lse=lse, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert_within("out", out, O.sdpa_forward(q, k, v, mode, D ** -0.5)[0], TOL_16BIT, torch.bfloat16)


@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk,D,mode", [(8, 4, 4, 1024, 1024, 64, 1), (4, 8, 2, 500, 3000, 128, 2),
                                                  (6, 16, 4, 2, 9000, 128, 2), (9, 2, 2, 1, 5000, 64, 0)])
def test_a_shard_that_is_told_the_whole_has_its_bits(B, Hq, Hkv, Sq, Sk, D, mode):
    q, k, v, _ = (t.cuda() for t in draw(torch.float16, B, Hq, Hkv, Sq, Sk, D, 9))
    forward = raw.flash_fwd_splitkv if Hq // Hkv * Sq <= 16 else raw.flash_fwd
    out, lse = forward(q, k, v, causal=mode)
    for hs, ks in ((slice(None), slice(None)), (slice(Hq // 2, Hq), slice(Hkv // 2, Hkv))):   # an entry, half its heads
        part_out, part_lse = forward(q[1:2, hs], k[1:2, ks], v[1:2, ks], causal=mode, whole_heads=B * Hq)
        assert torch.equal(part_out, out[1:2, hs]) and torch.equal(part_lse, lse[1:2, hs])


@pytest.mark.parametrize("D", [64, 128])
def test_an_infinity_behind_a_vanished_probability_spreads_split_or_not(D):
    """Zero times infinity is NaN (as in the softmax written out), also where the keys whose probabilities
    vanish are a thread block's whole share."""
    q = torch.ones(1, 2, 256, D, dtype=torch.float16, device="cuda")
    k, v = torch.full((1, 2, 4096, D), 4.0, dtype=torch.float16, device="cuda"), torch.ones_like(q[:, :, :1]).repeat(1, 1, 4096, 1)
    k[:, :, 2000:] = -12.0      # 16 sqrt(D) lower: 2^-184 at D = 64
    v[0, 1, 4000, 5] = float("inf")
    assert _lib.fwd_splits(1, 2, 256, 4096, D, _lib.F16, 0) > 1
    out, lse = raw.flash_fwd(q, k, v, causal=0)
    _lib.set_fwd_tiles(1 if D == 64 else 2)     # a forced shape is never split
    try:
        whole, whole_lse = raw.flash_fwd(q, k, v, causal=0)
    finally:
        _lib.set_fwd_tiles(0)
    assert bool(whole[0, 1, :, 5].isnan().all()) and int(whole.isnan().sum()) == 256
    assert torch.equal(out.isnan(), whole.isnan()) and torch.equal(out.nan_to_num(), whole.nan_to_num())
    assert torch.allclose(lse, whole_lse, atol=1e-5)


ALIGNED = [
    # dtype, B, Hq, Hkv, Sq, Sk, D, mode (1 top-left = torch's is_causal, 2 bottom-right = the reference kernels' rule)
    (torch.bfloat16, 2, 4, 2, 128, 320, 128, 1),
    (torch.bfloat16, 2, 4, 2, 128, 320, 128, 2),
    (torch.float16, 1, 4, 4, 300, 1000, 64, 2),
    (torch.bfloat16, 1, 2, 2, 1000, 300, 64, 1),     # key rows past the last query are seen by nobody
    (torch.bfloat16, 1, 2, 1, 1, 777, 128, 2),       # one new token against a cache: sees every key
    (torch.bfloat16, 1, 2, 1, 1, 777, 128, 1),       # ... and under torch's rule only key 0
    (torch.bfloat16, 1, 3, 3, 513, 640, 64, 2),
    (torch.float32, 1, 2, 2, 100, 260, 64, 2),
    (torch.float32, 1, 2, 1, 260, 100, 128, 1),
]


@pytest.mark.parametrize("dtype,B,Hq,Hkv,Sq,Sk,D,mode", ALIGNED)
def test_causal_mask_over_unequal_lengths_both_alignments(dtype, B, Hq, Hkv, Sq, Sk, D, mode):
    """Oracle: torch CPU SDPA (is_causal for the top-left rule, an explicit mask for the
    bottom-right rule of fa4_fwd_kernel.mojo:266-273) and the float64 restatement."""
    q, k, v, dout = draw(dtype, B, Hq, Hkv, Sq, Sk, D, 20260910 + Sq + Sk + mode)
    scale = D ** -0.5
    ref_out, ref_lse = O.sdpa_forward(q, k, v, mode, scale)
    _, rdq, rdk, rdv = O.sdpa_backward(q, k, v, dout, mode, scale)
    r_out, r_lse = R.forward(t64(q), t64(k), t64(v), mode, scale)
    assert np.abs(r_out - ref_out.numpy()).max() < 1e-4 and np.abs(r_lse - ref_lse.numpy()).max() < 1e-4
    tol = tol_for(dtype)
    for simt in ([False, True] if dtype != torch.float32 else [False]):
        out, lse, dq, dk, dv = run(q, k, v, dout, mode, scale, simt=simt)
        tag = "simt " if simt else ""
        assert_within(tag + "out", out, ref_out, tol, dtype)
        assert_within(tag + "lse", lse, ref_lse, TOL_LSE)
        assert_within(tag + "dq", dq, rdq, tol, dtype)
        assert_within(tag + "dk", dk, rdk, tol, dtype)
        assert_within(tag + "dv", dv, rdv, tol, dtype)


@pytest.mark.parametrize("dtype,Sq,Sk,D", [(torch.bfloat16, 700, 260, 128), (torch.float16, 300, 100, 64),
                                           (torch.float32, 200, 72, 64)])
def test_bottom_right_mask_with_more_queries_than_keys_has_rows_that_see_nothing(dtype, Sq, Sk, D):
    """Sq > Sk under the bottom-right rule: the first Sq - Sk query rows see no key; they get
    out = 0, lse = -inf and zero gradients (torch would give NaN for such rows, so the oracle
    here is the float64 restatement)."""
    B, Hq, Hkv = 1, 4, 2
    q, k, v, dout = draw(dtype, B, Hq, Hkv, Sq, Sk, D, 20260911 + Sq)
    scale = D ** -0.5
    r_out, r_lse = R.forward(t64(q), t64(k), t64(v), 2, scale)
    r_dq, r_dk, r_dv = R.backward(t64(q), t64(k), t64(v), t64(dout), 2, scale)
    tol = tol_for(dtype)
    for simt in ([False, True] if dtype != torch.float32 else [False]):
        out, lse, dq, dk, dv = run(q, k, v, dout, 2, scale, simt=simt)
        blind = Sq - Sk
        assert torch.all(out[:, :, :blind] == 0) and torch.all(lse[:, :, :blind] == float("-inf"))
        assert torch.all(dq[:, :, :blind] == 0)
        assert_within("out", out, torch.from_numpy(r_out), tol, dtype)
        assert_within("lse", lse[:, :, blind:], torch.from_numpy(r_lse[:, :, blind:]), TOL_LSE)
        assert_within("dq", dq, torch.from_numpy(r_dq), tol, dtype)
        assert_within("dk", dk, torch.from_numpy(r_dk), tol, dtype)
        assert_within("dv", dv, torch.from_numpy(r_dv), tol, dtype)


DECODE = [
    # dtype, B, Hq, Hkv, Sq, Sk, D, mode
    (torch.bfloat16, 2, 8, 2, 1, 4096, 128, 0),
    (torch.bfloat16, 3, 8, 8, 1, 1000, 64, 2),
    (torch.float16, 1, 16, 2, 2, 5000, 128, 2),     # 8 heads x 2 rows = 16 rows per kv head
    (torch.bfloat16, 1, 4, 1, 4, 777, 64, 2),
    (torch.bfloat16, 2, 4, 4, 16, 600, 128, 2),
    (torch.float32, 1, 4, 2, 1, 2000, 64, 0),
    (torch.bfloat16, 1, 8, 2, 1, 40000, 128, 2),    # long cache: many splits per kv head
    (torch.bfloat16, 1, 2, 2, 3, 513, 128, 1),      # torch's rule: the three rows see 1, 2 and 3 keys
    (torch.float16, 2, 12, 4, 4, 1531, 64, 2),      # 12 rows: two row tiles, four padding rows
    (torch.bfloat16, 1, 10, 2, 1, 3001, 128, 0),    # 5 rows: three padding rows in the tile
    (torch.bfloat16, 2, 6, 2, 5, 2050, 64, 2),      # 15 rows, a causal diagonal inside the last keys
    (torch.float16, 1, 8, 1, 1, 9000, 128, 2),      # 8 rows: a full tile
    (torch.float32, 1, 8, 2, 3, 700, 128, 2),       # fp32 keeps the scalar kernel: 12 rows, two groups of warps
]


@pytest.mark.parametrize("dtype,B,Hq,Hkv,Sq,Sk,D,mode", DECODE)
def test_split_kv_decode_forward_matches_oracle_and_prefill_kernel(dtype, B, Hq, Hkv, Sq, Sk, D, mode):
    q, k, v, _ = draw(dtype, B, Hq, Hkv, Sq, Sk, D, 20260912 + Sk)
    scale = D ** -0.5
    ref_out, ref_lse = O.sdpa_forward(q, k, v, mode, scale)
    qc, kc, vc = q.cuda(), k.cuda(), v.cuda()
    before = _lib.launch_count()
    out, lse = raw.flash_fwd_splitkv(qc, kc, vc, causal=mode, scale=scale)
    assert _lib.launch_count() - before == 1   # the last thread block of a KV head merges its splits
    p_out, p_lse = raw.flash_fwd(qc, kc, vc, causal=mode, scale=scale)
    torch.cuda.synchronize()
    tol = tol_for(dtype)
    assert_within("out", out, ref_out, tol, dtype)
    assert_within("lse", lse, ref_lse, TOL_LSE)
    assert_within("out vs prefill kernel", out, p_out.float(), tol, dtype)
    assert_within("lse vs prefill kernel", lse, p_lse, TOL_LSE)
    # K and V stored (B, S, H, D) and handed over as transposed views: same bits
    kt = kc.transpose(1, 2).contiguous().transpose(1, 2)
    vt = vc.transpose(1, 2).contiguous().transpose(1, 2)
    out_t, lse_t = raw.flash_fwd_splitkv(qc, kt, vt, causal=mode, scale=scale)
    assert torch.equal(out_t, out) and torch.equal(lse_t, lse)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,D", [(1, 1, 1, 1, 64), (1, 4, 1, 3, 128), (3, 10, 2, 3, 64), (19, 16, 8, 5, 128), (57, 1, 1, 2, 128)])
def test_split_kv_merges_as_a_cluster_or_through_the_workspace(dtype, B, Hq, Hkv, Sq, D):
    """One split, clusters of 2 to 16 of them, and more splits or more clusters than that: the same numbers as the exact-fp32
    forward within the contract's tolerance, and the same bits whichever piece of a batch they are computed for."""
    for Sk in (500, 512, 700, 1100, 1900, 2304, 4000, 4400, 9000):
        if B * Hkv * Sk > 400000:
            continue
        q, k, v, _ = (t.cuda() for t in draw(dtype, B, Hq, Hkv, Sq, Sk, D, 31 + Sk))
        out, lse = raw.flash_fwd_splitkv(q, k, v, causal=2)
        ref_out, ref_lse = raw.flash_fwd(q, k, v, causal=2, simt=True)
        assert_within("out", out, ref_out.float(), tol_for(dtype), dtype)
        assert_within("lse", lse, ref_lse, TOL_LSE)
        part_out, part_lse = raw.flash_fwd_splitkv(q[:1], k[:1], v[:1], causal=2, whole_heads=B * Hq)
        assert torch.equal(part_out, out[:1]) and torch.equal(part_lse, lse[:1])


DROPOUT = [
    # dtype, B, Hq, Hkv, Sq, Sk, D, mode, p
    (torch.bfloat16, 2, 4, 2, 256, 256, 128, 1, 0.1),
    (torch.float16, 1, 4, 4, 384, 384, 64, 0, 0.25),
    (torch.bfloat16, 1, 2, 1, 193, 193, 64, 1, 0.5),
    (torch.bfloat16, 1, 2, 2, 130, 400, 128, 2, 0.2),
    (torch.float32, 1, 2, 2, 100, 100, 64, 1, 0.3),
]


@pytest.mark.parametrize("dtype,B,Hq,Hkv,Sq,Sk,D,mode,p", DROPOUT)
def test_dropout_uses_the_documented_philox_stream_forward_and_backward(dtype, B, Hq, Hkv, Sq, Sk, D, mode, p):
    """The oracle regenerates the mask from (seed, offset) with its own Philox4x32-10 and applies
    it in torch CPU ops (and in the float64 restatement): parity is exact-mask, not statistical."""
    seed, offset = 0x9E3779B97F4A7C15, 1000 + Sq
    q, k, v, dout = draw(dtype, B, Hq, Hkv, Sq, Sk, D, 20260913 + Sq)
    scale = D ** -0.5
    keep, keep_scale = keep_mask(B, Hq, Sq, Sk, p, seed, offset)
    assert abs(keep.mean() - (1 - _lib.dropout_threshold(p) / 256)) < 0.02
    ref_out, ref_lse, rdq, rdk, rdv = O.sdpa_dropout(q, k, v, dout, mode, scale, torch.from_numpy(keep), keep_scale)
    r_out, _ = R.forward(t64(q), t64(k), t64(v), mode, scale, keep, keep_scale)
    assert np.abs(r_out - ref_out.numpy()).max() < 1e-4
    tol = tol_for(dtype)
    for simt in ([False, True] if dtype != torch.float32 else [False]):
        out, lse, dq, dk, dv = run(q, k, v, dout, mode, scale, simt=simt, dropout=(p, seed, offset))
        tag = "simt " if simt else ""
        assert_within(tag + "out", out, ref_out, tol, dtype)
        assert_within(tag + "lse", lse, ref_lse, TOL_LSE)
        assert_within(tag + "dq", dq, rdq, tol, dtype)
        assert_within(tag + "dk", dk, rdk, tol, dtype)
        assert_within(tag + "dv", dv, rdv, tol, dtype)
    # another offset draws another mask
    other = run(q, k, v, dout, mode, scale, dropout=(p, seed, offset + B * Hq))[0]
    assert not torch.equal(other, out)


def test_dropout_through_the_mojo_device_regenerates_the_mask_in_backward(mojo_registered):
    """F.scaled_dot_product_attention(dropout_p=...) on mojo tensors: the rng_state slot of the
    aten tuple holds the (seed, offset) the mask came from, and the gradients match the oracle
    given that mask."""
    torch.mojo.manual_seed_all(4242)
    B, H, S, D, p = 2, 4, 256, 64, 0.2
    q, k, v, dout = draw(torch.bfloat16, B, H, H, S, S, D, 77)
    scale = D ** -0.5
    seed, offset = torch.mojo._reserve_philox_state(0, 0)
    keep, keep_scale = keep_mask(B, H, S, S, p, seed, offset)
    ref_out, _, rdq, rdk, rdv = O.sdpa_dropout(q, k, v, dout, 1, scale, torch.from_numpy(keep), keep_scale)
    mq, mk, mv = (t.to("mojo").requires_grad_() for t in (q, k, v))
    out = torch.nn.functional.scaled_dot_product_attention(mq, mk, mv, dropout_p=p, is_causal=True)
    out.backward(dout.to("mojo"))
    torch.mojo.synchronize()
    assert_within("out", out.cpu(), ref_out, TOL_16BIT, torch.bfloat16)
    assert_within("dq", mq.grad.cpu(), rdq, TOL_16BIT, torch.bfloat16)
    assert_within("dk", mk.grad.cpu(), rdk, TOL_16BIT, torch.bfloat16)
    assert_within("dv", mv.grad.cpu(), rdv, TOL_16BIT, torch.bfloat16)
    res = torch.ops.aten._scaled_dot_product_flash_attention.default(mq.detach(), mk.detach(), mv.detach(), p, True, False)
    assert res[6].cpu().tolist() == [4242, B * H]


def test_a_wait_that_runs_out_reports_a_status_and_leaves_the_gpu_usable():
    """The give-up path of the kernels' bounded waits, exercised by a one-warp kernel that waits
    a millisecond's worth of cycles on a barrier nobody arrives at: the kernel returns, the
    status word says where it gave up, and the next attention call on the same stream is fine."""
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    before = _lib.launch_count()
    assert _lib.selftest_wait_timeout(status.data_ptr(), 2_000_000, stream, 0) == _lib.OK
    torch.cuda.synchronize()
    assert _lib.launch_count() - before == 1
    value = int(status.item()) & 0xFFFFFFFF
    assert value == 0x5741FFFE
    assert _lib.status_to_error(value) == _lib.ERR_TIMEOUT
    # an attention kernel handed a status word that is already set leaves at once (its output is
    # not to be trusted and the word is preserved); with a clean word it runs as usual
    q, k, v, _ = draw(torch.bfloat16, 1, 2, 2, 256, 256, 64, 5)
    qc, kc, vc = q.cuda(), k.cuda(), v.cuda()
    raw.flash_fwd(qc, kc, vc, causal=True, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) & 0xFFFFFFFF == 0x5741FFFE
    status.zero_()
    out, lse = raw.flash_fwd(qc, kc, vc, causal=True, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    ref_out, _ = O.sdpa_forward(q, k, v, True, 64 ** -0.5)
    assert_within("out after a timed-out wait", out, ref_out, TOL_16BIT, torch.bfloat16)


def test_the_mojo_device_surfaces_a_timed_out_wait_at_synchronize(mojo_registered):
    from torch_mojo_backend_b200 import flash_ops

    q = torch.randn(1, 2, 128, 64).bfloat16().to("mojo")
    torch.nn.functional.scaled_dot_product_attention(q, q, q, is_causal=True)
    torch.mojo.synchronize()   # clean
    stream = torch.cuda.current_stream(0).cuda_stream
    assert _lib.selftest_wait_timeout(flash_ops._status_ptr(0), 1_000_000, stream, 0) == _lib.OK
    with pytest.raises(_lib.B200FAError) as err:
        torch.mojo.synchronize()
    assert err.value.code == _lib.ERR_TIMEOUT
    torch.mojo.synchronize()   # the word was cleared; the device carries on
    out = torch.nn.functional.scaled_dot_product_attention(q, q, q, is_causal=True)
    torch.mojo.synchronize()
    assert not torch.isnan(out.cpu().float()).any()


def test_extended_golden_fixtures_on_the_gpu():
    """The committed ext_* fixtures (mask alignments over unequal lengths, rows that see no key,
    dropout with a stored mask) against the tensor-core and the exact-fp32 kernels."""
    from tests.helpers import ext_golden_names, load_ext_golden

    for name in ext_golden_names():
        meta, q, k, v, dout, exp = load_ext_golden(name)
        tol = tol_for(meta["dtype"])
        for simt in (False, True):
            out, lse, dq, dk, dv = run(q, k, v, dout, meta["mode"], meta["scale"], simt=simt, dropout=meta["dropout"])
            fin = torch.isfinite(exp["lse"])
            assert torch.equal(torch.isfinite(lse.cpu()), fin), name
            assert_within(name + " out", out, exp["out"], tol, meta["dtype"])
            assert_within(name + " lse", lse.cpu()[fin], exp["lse"][fin], TOL_LSE)
            assert_within(name + " dq", dq, exp["dq"], tol, meta["dtype"])
            assert_within(name + " dk", dk, exp["dk"], tol, meta["dtype"])
            assert_within(name + " dv", dv, exp["dv"], tol, meta["dtype"])


TILE_SHAPES = [
    # dtype, B, Hq, Hkv, Sq, Sk, D, mode, dropout p
    (torch.bfloat16, 2, 4, 2, 700, 700, 64, 1, 0.0),
    (torch.float16, 1, 3, 3, 1, 1, 64, 1, 0.0),
    (torch.bfloat16, 1, 4, 4, 1333, 1333, 128, 1, 0.0),
    (torch.bfloat16, 2, 2, 1, 300, 1000, 128, 2, 0.0),
    (torch.float16, 3, 4, 2, 640, 640, 128, 0, 0.0),
    (torch.bfloat16, 1, 2, 2, 515, 515, 64, 1, 0.2),
]


@pytest.mark.parametrize("dtype,B,Hq,Hkv,Sq,Sk,D,mode,p", TILE_SHAPES)
def test_both_shapes_of_the_forward_kernel_give_the_same_result(dtype, B, Hq, Hkv, Sq, Sk, D, mode, p):
    """One query tile per thread block (two blocks per SM) and two tiles per block are two schedules
    of the same arithmetic: bit-identical out and lse, and both within tolerance of the exact-fp32 kernel."""
    q, k, v, _ = draw(dtype, B, Hq, Hkv, Sq, Sk, D, seed=99 + Sq)
    scale = D ** -0.5
    dropout = (p, 0x5EED, 8) if p else None
    qc, kc, vc = q.cuda(), k.cuda(), v.cuda()
    results = {}
    try:
        for tiles in (1, 2):
            _lib.set_fwd_tiles(tiles)
            assert _lib.fwd_tiles() == tiles
            status = torch.zeros(1, dtype=torch.int32, device="cuda")
            out, lse = raw.flash_fwd(qc, kc, vc, causal=mode, scale=scale, status=status, dropout=dropout)
            torch.cuda.synchronize()
            assert int(status.item()) == 0
            results[tiles] = (out.cpu(), lse.cpu())
    finally:
        _lib.set_fwd_tiles(0)
    assert torch.equal(results[1][0], results[2][0])
    assert torch.equal(results[1][1], results[2][1])
    s_out, s_lse = raw.flash_fwd(qc, kc, vc, causal=mode, scale=scale, simt=True, dropout=dropout)
    assert_within("out vs exact fp32 kernel", results[1][0], s_out, TOL_16BIT, dtype)
    assert_within("lse vs exact fp32 kernel", results[1][1], s_lse, TOL_LSE)


@pytest.mark.parametrize("dtype,Sq,Sk,D,mode", [(torch.float16, 300, 1, 64, 0), (torch.float16, 640, 1, 128, 1),
                                                (torch.float16, 257, 130, 128, 0), (torch.bfloat16, 300, 1, 64, 0)])
def test_key_columns_past_the_last_key_stay_out_of_dq_when_logits_are_large(dtype, Sq, Sk, D, mode):
    """With large logits a row's logsumexp can be very negative; the zero-filled key rows past Sk then
    have an enormous would-be probability, which must be blanked before it reaches the 16-bit dS
    (inf times the zero K row would be NaN in dQ)."""
    g = torch.Generator().manual_seed(4242 + Sq)
    q = (torch.randn(2, 4, Sq, D, generator=g) * 3.0).to(dtype)
    k = (torch.randn(2, 2, Sk, D, generator=g) * 3.0).to(dtype)
    v = (torch.randn(2, 2, Sk, D, generator=g) * 0.5).to(dtype)
    dout = torch.randn(2, 4, Sq, D, generator=g).to(dtype)
    scale = D ** -0.5
    out, lse, dq, dk, dv = run(q, k, v, dout, mode, scale)
    s_out, s_lse, s_dq, s_dk, s_dv = run(q, k, v, dout, mode, scale, simt=True)
    for name, got, ref in (("out", out, s_out), ("dq", dq, s_dq), ("dk", dk, s_dk), ("dv", dv, s_dv)):
        assert torch.isfinite(got.float()).all(), name
        assert_within(name, got, ref, TOL_16BIT, dtype)


def test_split_kv_of_one_split_has_nothing_to_merge():
    """Many short caches of 16 query rows: each KV head is one block, which writes its rows without the walk through a
    cluster's peers (measured 1.67 of the time a copy takes to read K and V, with it 2.16)."""
    B, Hq, Hkv, Sq, Sk, D = 64, 96, 12, 2, 600, 128
    assert _lib.fwd_splitkv_workspace_bytes(B, Hq, Hkv, Sq, Sk, D) // (B * Hq * Sq * (D + 2) * 4) == 1
    g = torch.Generator(device="cuda").manual_seed(6)
    rand = lambda *shape: torch.randn(shape, generator=g, device="cuda", dtype=torch.bfloat16)
    q, caches = rand(B, Hq, Sq, D), [(rand(B, Hkv, Sk, D), rand(B, Hkv, Sk, D)) for _ in range(4)]   # larger than L2
    big = torch.empty(1 << 30, dtype=torch.uint8, device="cuda")
    other = torch.empty_like(big)

    def ms(call, times):
        call()
        start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        start.record()
        for _ in range(times):
            call()
        end.record()
        end.synchronize()
        return start.elapsed_time(end) / times

    out, lse = raw.flash_fwd_splitkv(q, *caches[0], causal=2)
    ref_out, ref_lse = raw.flash_fwd(q, *caches[0], causal=2, simt=True)
    assert_within("out", out, ref_out.float(), TOL_16BIT, torch.bfloat16)
    assert_within("lse", lse, ref_lse, TOL_LSE)
    workspace = torch.empty(_lib.fwd_splitkv_workspace_bytes(B, Hq, Hkv, Sq, Sk, D), dtype=torch.uint8, device="cuda")

    def calls():
        for k, v in caches:
            raw.flash_fwd_splitkv(q, k, v, causal=2, out=out, lse=lse, workspace=workspace)

    per_call = min(ms(calls, 5) for _ in range(5)) / len(caches)
    read = min(ms(lambda: other.copy_(big), 3) for _ in range(3)) / (2 * big.numel()) * caches[0][0].numel() * 2 * 2
    assert per_call < 1.9 * read, (per_call, read)
