"""Grouped decode attention (csrc/attn_decode_gqa.cu): the number of key ranges that the rule picks (attn_decode_gqa_splits) -- one range, because nothing else runs in
one round of CTAs; clusters of several sizes; ranges merged through the workspace -- against one range, against the scalar kernel, and as a captured step."""
import pytest
import torch

from oracle import model_ref as M
from lit_gpt_b200 import kernels as K

pytestmark = pytest.mark.gpu

HS = 128


def _case(B, G, qpk, max_seq, pos):
    g = torch.Generator(device="cuda").manual_seed(B * 1000 + G * 100 + max_seq)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()   # noqa: E731
    kc, vc = r(B, G, max_seq, HS), r(B, G, max_seq, HS)
    kc[:, :, pos:], vc[:, :, pos:] = 1e4, 1e4   # stale rows past the filled region must never be read
    cos, sin = M.build_rope_cache(max_seq, HS, pos_dtype=torch.float32)
    return r(B, (qpk + 2) * G * HS), cos.cuda(), sin.cuda(), torch.tensor([pos], device="cuda"), kc, vc


def _run(case, G, qpk, splits):
    qkv, cos, sin, pos, kc, vc = case
    k, v = kc.clone(), vc.clone()
    return K.attn_decode(qkv, cos, sin, pos, k, v, G * qpk, G, HS, HS, num_splits=splits), k, v


# (sequences, groups, heads of a group, cache rows, position)
@pytest.mark.parametrize("B,G,qpk,max_seq,pos", [
    (16, 8, 4, 1024, 1000),    # 128 pairs: one range
    (10, 8, 2, 900, 899),      # 80 pairs: not as many clusters of two at once
    (20, 8, 4, 520, 300),      # 160 pairs: more than SMs
    (8, 8, 4, 3008, 3000),     # 64 pairs: clusters of two
    (9, 8, 4, 2048, 1500),     # 72 pairs: about as many clusters of two as run at once
    (2, 8, 4, 3900, 3899),     # 16 pairs: clusters of several
    (1, 8, 8, 4096, 100),      # far fewer keys than rows: most ranges are empty
    (1, 1, 16, 16384, 16000),  # one pair over a long cache: ranges merged through the workspace
    (1, 2, 4, 8192, 8191),
    (3, 1, 2, 257, 256),
    (1, 4, 16, 64, 0),
])
def test_ranges_by_the_rule(B, G, qpk, max_seq, pos):
    case = _case(B, G, qpk, max_seq, pos)
    got, k, v = _run(case, G, qpk, 0)
    one, k1, v1 = _run(case, G, qpk, 1)
    assert torch.equal(k, k1) and torch.equal(v, v1)
    prev = K.attn_decode_tune(force_scalar=True)
    try:
        scalar = _run(case, G, qpk, 1)[0]
    finally:
        K.attn_decode_tune(force_scalar=prev)
    # bf16 outputs of fp32 sums: probabilities are rounded to bf16 on either side (2^-9 of each), the result once more
    for other in (one, scalar):
        assert (got.float() - other.float()).norm() <= 2**-7 * other.float().norm()
    for _ in range(3):   # the counters of the merge clean up after themselves
        assert torch.equal(_run(case, G, qpk, 0)[0], got)


def test_ranges_under_capture():
    case = _case(8, 8, 4, 3008, 3000)
    want = _run(case, 8, 4, 0)[0]
    qkv, cos, sin, pos, kc, vc = case
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = K.attn_decode(qkv, cos, sin, pos, kc, vc, 32, 8, HS, HS)
    graph.replay()
    assert torch.equal(got, want)


@pytest.mark.parametrize("B,G,qpk,max_seq,pos", [(4, 8, 4, 3008, 3000), (2, 2, 8, 1024, 1000), (1, 4, 16, 2048, 2000), (1, 2, 9, 700, 600)])
@pytest.mark.parametrize("splits", [0, 1, 3, 12])
def test_close_to_64_bits_whatever_the_ranges(B, G, qpk, max_seq, pos, splits):
    """P enters as two 16-bit numbers: what is left is the rounding of the result, and 2^-17 of P and fp32 sums beside it.  (With more than eight heads a group and ranges
    that fill the SMs it is one number, good to 2^-9: as much again.)"""
    case = _case(B, G, qpk, max_seq, pos)
    qkv, _, _, p, kc, vc = case
    one, zero = torch.ones(max_seq, HS, device="cuda"), torch.zeros(max_seq, HS, device="cuda")   # (no rotation: the queries as they are)
    y, k, v = _run((qkv, one, zero, p, kc, vc), G, qpk, splits)
    q = qkv.view(B, G, qpk + 2, HS)[:, :, :qpk].double()
    att = torch.softmax(torch.einsum("bgqd,bgkd->bgqk", q, k[:, :, : pos + 1].double()) * HS**-0.5, -1)
    want = torch.einsum("bgqk,bgkd->bgqd", att, v[:, :, : pos + 1].double()).reshape(B, -1)
    rounding = (want.bfloat16().double() - want).norm()
    one_number = qpk > 8 and (splits == 0 or splits >= min(-(-148 // (B * G)), -(-max_seq // 256)))
    assert (y.double() - want).norm() <= 1.02 * rounding + (2**-9 if one_number else 2**-15) * want.norm()


@pytest.mark.parametrize("qpk", [4, 12])
def test_infinite_values(qpk):
    """An infinite value in one column: that column's outputs, and no other's."""
    B, G, max_seq, pos = 2, 2, 512, 500
    case = _case(B, G, qpk, max_seq, pos)
    want = _run(case, G, qpk, 0)[0].view(B, G, qpk, HS)
    case[5][1, 0, 77, 9] = float("inf")
    got = _run(case, G, qpk, 0)[0].view(B, G, qpk, HS)
    assert (got[1, 0, :, 9] == float("inf")).all()
    keep = torch.ones(B, G, qpk, HS, dtype=torch.bool, device="cuda")
    keep[1, 0, :, 9] = False
    assert torch.equal(got[keep], want[keep])
