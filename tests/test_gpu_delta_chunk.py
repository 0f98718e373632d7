"""The gated delta rule in chunks of 32 tokens against the same recurrence in 64 bits, beside the token-by-token kernel: chunk edges, sequences
shorter than a chunk or a token, key and value sizes off every tile, grouped heads, states carried in, several segments of scratch."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from lit_gpt_b200 import kernels

    return kernels


def _inputs(lens, starts, H, G, dk, dv, channel, dtype, seed, pad):
    g = torch.Generator().manual_seed(seed)
    n = sum(lens)
    unit = lambda t: t / t.norm(dim=-1, keepdim=True)   # noqa: E731
    pitch = lambda t: torch.cat((t, torch.zeros(n, pad)), 1)[:, : t.shape[1]]   # noqa: E731  (pad: rows that do not start on 16-byte boundaries)
    q = pitch(unit(torch.randn(n, G, dk, generator=g)).reshape(n, G * dk) * dk ** -0.5)
    k = pitch(unit(torch.randn(n, G, dk, generator=g)).reshape(n, G * dk))
    v = pitch(torch.randn(n, H * dv, generator=g))
    beta, dec = torch.randn(n, H, generator=g).to(dtype), torch.randn(n, H * (dk if channel else 1), generator=g).to(dtype)
    a_log = (torch.rand(H, generator=g) * 2.5 - 1).to(dtype)
    bias = (torch.rand(H * (dk if channel else 1), generator=g) * 6 - 5).to(dtype)
    slots = len(lens) + 1
    S0 = torch.randn(slots, H, dk, dv, generator=g)
    seqs, first = [], 0
    for i, (m, s) in enumerate(zip(lens, starts)):
        seqs.append((first, m, s, slots - 1 - i))
        first += m
    return q, k, v, beta, dec, a_log, bias, S0, torch.tensor(seqs, dtype=torch.int32)


def _exact(q, k, v, beta, dec, a_log, bias, S0, seqs, H, G, dk, dv, channel):
    d = lambda t: t.double()   # noqa: E731
    g = torch.exp(-torch.exp(d(a_log))[None, :, None] * torch.nn.functional.softplus((d(dec) + d(bias)).view(len(q), H, -1)))
    out, S1 = torch.zeros(len(q), H, dv, dtype=torch.float64), d(S0).clone()
    kk, qq = (d(t).reshape(len(q), G, dk).repeat_interleave(H // G, 1) for t in (k, q))
    vv, bb = d(v).reshape(len(q), H, dv), torch.sigmoid(d(beta))
    for first, m, start, slot in seqs.tolist():
        S = d(S0[slot]).clone() if start else torch.zeros(H, dk, dv, dtype=torch.float64)
        for t in range(first, first + m):
            S = S * g[t][:, :, None]
            u = bb[t][:, None] * (vv[t] - torch.einsum("hij,hi->hj", S, kk[t]))
            S = S + kk[t][:, :, None] * u[:, None]
            out[t] = torch.einsum("hij,hi->hj", S, qq[t])
        S1[slot] = S
    return out.reshape(len(q), -1), S1


def _stored(S, dk, L):
    """(slots, H, dk, dv) -> the order the kernels keep a state in: runs of L keys, zeros up to a whole run"""
    slots, H, _, dv = S.shape
    pad = torch.zeros(slots, H, -dk % L, dv, dtype=S.dtype)
    return torch.cat((S, pad), 2).view(slots, H, -1, L, dv).transpose(3, 4).reshape(slots, -1)


@pytest.mark.parametrize("lens,starts,H,G,dk,dv,dtype,pad", [
    ((64,), (0,), 2, 2, 128, 128, torch.bfloat16, 0),
    ((65, 1, 31, 32, 33), (0, 7, 0, 3, 0), 4, 2, 64, 64, torch.bfloat16, 0),
    ((200, 96), (11, 0), 3, 1, 72, 136, torch.float32, 0),
    ((95,), (0,), 2, 1, 7, 5, torch.float32, 3),
    ((130,), (4,), 1, 1, 63, 1, torch.bfloat16, 1),
    ((300,), (0,), 16, 16, 128, 128, torch.float32, 0),
    ((128, 64), (0, 0), 2, 2, 1, 20, torch.bfloat16, 0),
])
@pytest.mark.parametrize("channel", [False, True])
def test_delta_chunks_against_exact(K, lens, starts, H, G, dk, dv, dtype, pad, channel):
    data = _inputs(lens, starts, H, G, dk, dv, channel, dtype, dk + dv, pad)
    ref, S_ref = _exact(*data, H, G, dk, dv, channel)
    q, k, v, beta, dec, a_log, bias, S0, seqs = data
    L = 4 if dk <= 64 else 8

    def cuda(t):   # keeps the row pitch
        return torch.zeros(t.shape[0], t.stride(0), dtype=t.dtype, device="cuda")[:, : t.shape[1]].copy_(t)

    def run(chunked):
        state = _stored(S0, dk, L).float().cuda()
        K.DELTA_CHUNKED = chunked
        try:
            o = K.delta_rule(cuda(q), cuda(k), cuda(v), beta.cuda(), dec.cuda(), a_log.cuda(), bias.cuda(), state, seqs.cuda(), H, G, dk, dv, channel,
                             max_rows=max(lens))
        finally:
            K.DELTA_CHUNKED = True
        return o.cpu().double(), state.cpu().double()

    (o1, s1), (o0, s0) = run(True), run(False)
    s_ref = _stored(S_ref, dk, L)
    # both sum the same fp32 terms in another order: neither may be far worse than the other, nor than a few roundings of the largest number
    for new, old, exact in ((o1, o0, ref), (s1, s0, s_ref)):
        scale = exact.abs().max()
        assert (new - exact).abs().max() <= 2 * (old - exact).abs().max() + 4 * 2.0 ** -23 * scale
    assert torch.equal(s1[0], _stored(S0, dk, L)[0].double())   # the slot no sequence uses


@pytest.mark.parametrize("chunks", [1, 3])
def test_delta_chunks_in_segments(K, chunks):
    """Less scratch than the prompt's chunks: the same launches over runs of chunks, the state handed on through the slot."""
    from lit_gpt_b200 import _cabi as C

    H, G, dk, dv, lens = 2, 2, 128, 40, (170, 70)
    q, k, v, beta, dec, a_log, bias, S0, seqs = _inputs(lens, (0, 5), H, G, dk, dv, True, torch.float32, 5, 0)
    dev = [t.cuda() for t in (q, k, v.contiguous(), beta, dec, a_log, bias, seqs)]
    state = _stored(S0, dk, 8).float().cuda()
    whole = state.clone()
    want = K.delta_rule(*dev[:7], whole, dev[7], H, G, dk, dv, True, max_rows=max(lens))
    lib = C.load()
    full = lib.b200_delta_rule_workspace_bytes(max(lens), 2, H, dk, dv)
    nbytes = full // 6 * chunks            # the longer sequence has six chunks
    ws, out = torch.empty(nbytes, dtype=torch.uint8, device="cuda"), torch.empty(sum(lens), H * dv, device="cuda")
    a = C.DeltaRuleArgs(q=dev[0].data_ptr(), k=dev[1].data_ptr(), v=dev[2].data_ptr(), ldq=G * dk, ldk=G * dk, ldv=H * dv, beta_in=dev[3].data_ptr(),
                        ld_beta=H, decay_in=dev[4].data_ptr(), ld_decay=H * dk, a_log=dev[5].data_ptr(), dt_bias=dev[6].data_ptr(),
                        state=state.data_ptr(), state_slot_stride=state.stride(0), out=out.data_ptr(), ldo=H * dv, seqs=dev[7].data_ptr(), n_seqs=2,
                        heads=H, kv_heads=G, dk=dk, dv=dv, channel_decay=1, dtype=C.F32, max_rows=max(lens))
    C.check(lib.b200_delta_rule_chunked(ctypes.byref(a), ws.data_ptr(), nbytes, C.stream_ptr()), "delta_rule")
    assert torch.equal(out, want) and torch.equal(state, whole)


@pytest.mark.parametrize("lens,hint", [((200, 10), 110), ((100, 1, 1), 64), ((70, 300, 5), 64), ((33, 0, 100, 64), 65)])
def test_delta_chunks_compute_every_row_whatever_the_hint(K, monkeypatch, lens, hint):
    """max_rows picks the kernel; rows past it are computed all the same, and a sequence without rows starts its slot from zero as before."""
    monkeypatch.setattr(K, "DELTA_CHUNKED", True)
    H, G, dk, dv = 4, 2, 64, 40
    starts = [7 * (i % 2) for i in range(len(lens))]
    data = _inputs(lens, starts, H, G, dk, dv, True, torch.float32, 11, 0)
    dev = [t.contiguous().cuda() for t in data[:7]]
    out = {}
    for rows in (hint, max(lens), 0):   # 0: token by token
        state = _stored(data[7], dk, 4).float().cuda()
        out[rows] = K.delta_rule(*dev, state, data[8].cuda(), H, G, dk, dv, True, max_rows=rows), state
    (a, sa), (b, sb), (c, sc) = out[hint], out[max(lens)], out[0]
    assert torch.equal(a, b) and torch.equal(sa, sb)
    assert (a - c).abs().max() <= 1e-4 * c.abs().max() and (sa - sc).abs().max() <= 1e-4 * sc.abs().max()


@pytest.mark.parametrize("rows", [40, 1, 0])
@pytest.mark.parametrize("start", [0, 9])
def test_delta_chunks_of_a_short_sequence_in_a_long_buffer(K, monkeypatch, rows, start):
    """One sequence whose rows are fewer than the buffer's and than the hint says: its rows and its state, as token by token."""
    H, G, dk, dv = 2, 1, 64, 24
    data = _inputs((100,), (start,), H, G, dk, dv, True, torch.float32, 2, 0)
    dev, seqs = [t.contiguous().cuda() for t in data[:7]], torch.tensor([[0, rows, start, 1]], dtype=torch.int32).cuda()
    out = []
    for chunked in (True, False):
        monkeypatch.setattr(K, "DELTA_CHUNKED", chunked)
        state = _stored(data[7], dk, 4).float().cuda()
        out.append((K.delta_rule(*dev, state, seqs, H, G, dk, dv, True, max_rows=100)[:rows], state))
    (a, sa), (b, sb) = out
    assert rows == 0 or (a - b).abs().max() <= 1e-4 * b.abs().max()
    assert (sa - sb).abs().max() <= 1e-4 * sb.abs().max()


def test_delta_chunk_scratch_follows_the_rows(K, monkeypatch):
    """One prompt among many single rows takes scratch for the rows there are; without memory for it the call runs token by token."""
    H, G, dk, dv, lens = 2, 2, 128, 32, (96,) + (1,) * 40
    data = _inputs(lens, [3] * len(lens), H, G, dk, dv, False, torch.bfloat16, 3, 0)
    dev, seqs = [t.contiguous().cuda() for t in data[:7]], data[8].cuda()
    empty, asked = torch.empty, []

    def run(limit):
        def alloc(*a, **kw):
            if kw.get("dtype") == torch.uint8:
                asked.append(a[0])
                if a[0] > limit:
                    raise torch.OutOfMemoryError("scratch")
            return empty(*a, **kw)

        state = _stored(data[7], dk, 8).float().cuda()
        monkeypatch.setattr(torch, "empty", alloc)
        y = K.delta_rule(*dev, state, seqs, H, G, dk, dv, False, max_rows=96)
        monkeypatch.undo()
        return y, state

    monkeypatch.setattr(K, "DELTA_CHUNKED", True)
    a, sa = run(1 << 40)
    monkeypatch.setattr(K, "DELTA_CHUNKED", True)
    b, sb = run(0)
    from lit_gpt_b200 import _cabi as C
    chunk = C.load().b200_delta_rule_workspace_bytes(64, 1, H, dk, dv) // 2
    assert asked[0] == (sum(lens) + 31 * 2) // 32 * chunk   # two sequences of 64 rows at most, whatever their number
    assert (a - b).abs().max() <= 1e-4 * b.abs().max() and (sa - sb).abs().max() <= 1e-4 * sb.abs().max()


def test_delta_chunks_or_tokens(K):
    """What a step's rows decide: a prompt alone or beside single rows, many long sequences that fill the GPU token by token, short prompts, wide keys."""
    from lit_gpt_b200 import _cabi as C

    pays = C.load().b200_delta_rule_in_chunks
    for channel in (0, 1):
        for heads in (4, 16, 32):
            assert pays(512, 512, 1, heads, 128, 128, channel) and pays(1024 + 32, 1024, 33, heads, 128, 128, channel)
            assert not pays(63, 63, 1, heads, 128, 128, channel) and not pays(4096, 4096, 1, heads, 129, 128, channel)
        assert not pays(64 + 32, 64, 33, 16, 128, 128, channel) and not pays(64 * 64, 64, 64, 16, 128, 128, channel)
    assert pays(64, 64, 1, 16, 128, 128, 1) and not pays(64, 64, 1, 16, 128, 128, 0) and not pays(10, 100, 1, 16, 128, 128, 1)


def test_delta_chunk_rule(K):
    """What stays with the token-by-token kernel: single rows, short portions, wide keys, unknown lengths."""
    from lit_gpt_b200 import _cabi as C

    need = C.load().b200_delta_rule_workspace_bytes
    assert need(1, 8, 16, 128, 128) == need(63, 1, 16, 128, 128) == need(4096, 1, 4, 129, 128) == need(0, 1, 4, 64, 64) == 0
    assert 0 < need(64, 1, 16, 128, 128) < need(2048, 1, 16, 128, 128) <= 256 << 20
    assert need(1 << 20, 8, 32, 128, 128) <= 256 << 20
