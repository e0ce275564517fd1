"""The recurrences eight tokens at a time (csrc/chunk_scan.cu) against float64 loops, at the edges of chunks, tiles and column
blocks, beside the token-by-token kernels on the same inputs."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

P_, I_, F_, L_ = ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_longlong
LENS = [1, 7, 8, 9, 16, 17, 131, 30]


def entry(name, restype, *argtypes):
    from inferllm_b200.kernels import ops
    f = getattr(ops.load(), name)
    f.restype, f.argtypes = restype, list(argtypes)
    return f


def p(t):
    return None if t is None else t.data_ptr()


def layout():
    cu = np.concatenate([[0], np.cumsum(LENS)])
    ints = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device="cuda")  # noqa: E731
    pos, seq = np.concatenate([np.arange(n) for n in LENS]), np.repeat(np.arange(len(LENS)), LENS)
    return cu, ints(cu), ints(pos), ints(seq), ints(np.arange(len(LENS))[::-1].copy()), ints(LENS)


@pytest.mark.parametrize("d,dv,nh,off", [(128, 128, 3, 0), (128, 64, 2, 4), (20, 130, 2, 0), (9, 7, 1, 1), (100, 65, 2, 0), (64, 200, 1, 0)])
@pytest.mark.parametrize("segments", [1, 2, 5])
def test_linear_attention(d, dv, nh, off, segments):
    g = torch.Generator().manual_seed(d + dv)
    cu, cu_d, pos, _, slots, _ = layout()
    T, B, C = int(cu[-1]), len(LENS), nh * (2 * d + dv) + off
    x = torch.randn(T, C, generator=g)
    S0 = torch.randn(B, nh, dv, d, generator=g)
    decay = torch.tensor([0.3, 0.97, 0.9999][:nh])
    q_off, k_off, v_off = off, off + nh * d, off + 2 * nh * d
    xd, Sd, out, dd = x.cuda(), S0.cuda(), torch.full((T, nh * dv), float("nan"), device="cuda"), decay.cuda()
    n = entry("illm_decay_chunk_scratch", L_, I_, I_, I_, I_, I_, I_)(T, B, nh, d, dv, segments)
    rec, err = torch.full((n,), float("nan"), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = entry("illm_decay_chunk_scan", I_, P_, I_, I_, I_, I_, I_, I_, I_, I_, I_, I_, P_, I_, I_, F_, P_, P_, P_, P_, P_, P_, I_, I_, I_, P_, P_, P_)(
        p(xd), T, C, q_off, k_off, v_off, nh, d, dv, 0, 0, None, 0, 0, 1.0, p(dd), p(Sd), p(slots), p(cu_d), p(pos), p(out), B, max(LENS), segments, p(err), p(rec),
        torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    got, state = out.cpu().double().numpy().reshape(T, nh, dv), Sd.cpu().double().numpy()
    q, k, v = (x[:, o:o + nh * w].double().numpy().reshape(T, nh, w) for o, w in ((q_off, d), (k_off, d), (v_off, dv)))
    a = decay.double().numpy()
    # a term goes through at most d + 2 roundings in sums over rows, 2 per chunk or segment in the state, one per token of a segment in
    # the powers of the decay (twice: a fold and a read-out), and 20 more
    bound = 2.0 ** -24 * (d + 2 * (max(LENS) / 8) + 22 + (2 * max(LENS) if segments > 1 else 0))
    for b in range(B):
        s = B - 1 - b
        S, M = S0[s].double().numpy().copy(), S0[s].abs().double().numpy()
        for t in range(cu[b], cu[b + 1]):
            S = a[:, None, None] * S + v[t][:, :, None] * k[t][:, None, :]
            M = a[:, None, None] * M + np.abs(v[t])[:, :, None] * np.abs(k[t])[:, None, :]
            ref, mag = np.einsum("hvd,hd->hv", S, q[t]), np.einsum("hvd,hd->hv", M, np.abs(q[t]))
            assert (np.abs(got[t] - ref) <= bound * mag).all(), (b, t - cu[b])
        assert (np.abs(state[s] - S) <= bound * M).all()


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("segments,at", [(1, 19), (1, 23), (1, 8), (2, 90)])
def test_linear_attention_keeps_a_value_from_earlier_tokens(segments, at, bad):
    """A value that is no finite number at token `at` leaves the bits of all tokens before it as they are."""
    d, dv, nh, n = 64, 64, 2, 131
    g = torch.Generator().manual_seed(at)
    x, C = torch.randn(n, nh * (2 * d + dv), generator=g), nh * (2 * d + dv)
    ints = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")  # noqa: E731
    outs = []
    for planted in (False, True):
        xd, out, Sd = x.cuda(), torch.full((n, nh * dv), 7.0, device="cuda"), torch.zeros(1, nh, dv, d, device="cuda")
        if planted:
            xd[at, 2 * nh * d:] = bad
        size = entry("illm_decay_chunk_scratch", L_, I_, I_, I_, I_, I_, I_)(n, 1, nh, d, dv, segments)
        rec, err, decay = torch.empty(size, device="cuda"), ints([0]), torch.tensor([0.9, 0.99], device="cuda")
        zero, cu, pos = ints([0]), ints([0, n]), ints(list(range(n)))
        rc = entry("illm_decay_chunk_scan", I_, P_, I_, I_, I_, I_, I_, I_, I_, I_, I_, I_, P_, I_, I_, F_, P_, P_, P_, P_, P_, P_, I_, I_, I_, P_, P_, P_)(
            p(xd), n, C, 0, nh * d, 2 * nh * d, nh, d, dv, 0, 0, None, 0, 0, 1.0, p(decay), p(Sd), p(zero), p(cu), p(pos), p(out), 1, n, segments, p(err), p(rec),
            torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        outs.append(out.cpu())
    assert torch.equal(outs[0][:at], outs[1][:at]) and not torch.isfinite(outs[1][at]).any()


@pytest.mark.parametrize("head_decay", [0, 1])
@pytest.mark.parametrize("d,dv,nh,nkv", [(128, 128, 4, 2), (128, 64, 1, 1), (20, 130, 2, 2), (9, 7, 3, 1), (100, 65, 2, 1)])
@pytest.mark.parametrize("strong", [False, True])
def test_delta_rule(head_decay, d, dv, nh, nkv, strong):
    """The recurrence feeds its own output back, so the reference for its rounding is the token-by-token kernel: no more than twice as
    far from float64 (both measured as 2-norms over a sequence).  strong: decays down to e^-60."""
    taps = 2
    g = torch.Generator().manual_seed(d * dv + head_decay)
    cu, cu_d, pos, seq, slots, lens = layout()
    T, B = int(cu[-1]), len(LENS)
    C = 2 * nkv * d + nh * dv
    ld = C + nh
    x = torch.randn(T, ld, generator=g)
    na = nh if head_decay else nh * d
    a = torch.randn(T, na, generator=g) * (20.0 if strong else 1.0)
    conv = [torch.randn(w, taps, generator=g) for w in (nkv * d, nkv * d, nh * dv)]
    a_log, dt = torch.randn(nh, generator=g) * 0.5, torch.randn(na, generator=g)
    elems = nh * d * dv + (taps - 1) * C
    S0 = torch.randn(B, elems, generator=g)
    f = entry("illm_delta_rule", I_, P_, I_, I_, I_, I_, I_, I_, P_, I_, I_, I_, I_, I_, I_, I_, P_, P_, P_, P_, P_, F_, P_, L_, P_, P_, P_, P_, P_, P_, P_, P_, P_, I_,
              I_, P_, P_)
    n = entry("illm_delta_chunk_scratch", L_, I_, I_, I_)(T, B, nh)
    dev = [t.cuda() for t in (x, a, *conv, a_log, dt)]

    def run(chunks):
        S = S0.cuda()
        qkv, gg, beta = torch.empty(T, C, device="cuda"), torch.empty(T, na, device="cuda"), torch.empty(T, nh, device="cuda")
        out = torch.full((T, nh * dv), float("nan"), device="cuda")
        rec = torch.full((n,), float("nan"), device="cuda") if chunks else None
        rc = f(p(dev[0]), T, ld, 0, nkv * d, 2 * nkv * d, C, p(dev[1]), na, head_decay, nh, nkv, d, dv, taps, p(dev[2]), p(dev[3]), p(dev[4]), p(dev[5]),
               p(dev[6]), d ** -0.5, p(S), elems, p(slots), p(cu_d), p(pos), p(seq), p(lens), p(qkv), p(gg), p(beta), p(out), B, max(LENS), p(rec),
               torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        return [t.cpu().double().numpy() for t in (out, S, qkv, gg, beta)]

    chunked, (out, S, qkv, gg, beta) = run(True), run(False)
    share = nh // nkv
    # what the preparation makes of the projection (fast exponentials in silu: 1e-5)
    sig = lambda z: 1.0 / (1.0 + np.exp(-z))  # noqa: E731
    raw = x[:, :C].double().numpy()
    taps_all = np.concatenate([c.double().numpy() for c in conv])
    y = raw * taps_all[:, 1]
    y[1:] += raw[:-1] * taps_all[:, 0] * (pos.cpu().numpy()[1:, None] > 0)
    y = y * sig(y)
    for lo in range(0, 2 * nkv * d, d):
        head = y[:, lo:lo + d]
        y[:, lo:lo + d] = head / np.sqrt((head * head).sum(-1, keepdims=True) + 1e-6) * (d ** -0.5 if lo < nkv * d else 1.0)
    assert np.abs(qkv - y).max() <= 3e-5 * max(1.0, np.abs(y).max())
    z = a.double().numpy() + dt.double().numpy()
    rate = np.exp(a_log.double().numpy())
    want = np.exp(-(rate if head_decay else np.repeat(rate, d)) * np.logaddexp(0.0, z))
    assert np.abs(gg - want).max() <= 2e-5 and np.abs(beta - sig(x[:, C:].double().numpy())).max() <= 1e-6
    for b in range(B):
        s = B - 1 - b
        refs = []
        St = S0[s, :nh * d * dv].double().numpy().reshape(nh, dv, d).copy()
        for t in range(cu[b], cu[b + 1]):
            q, k, v = qkv[t, :nkv * d].reshape(nkv, d).repeat(share, 0), qkv[t, nkv * d:2 * nkv * d].reshape(nkv, d).repeat(share, 0), qkv[t, 2 * nkv * d:].reshape(nh, dv)
            St = St * (gg[t].reshape(nh, 1, 1) if head_decay else gg[t].reshape(nh, 1, d))
            u = beta[t][:, None] * (v - np.einsum("hvd,hd->hv", St, k))
            St = St + u[:, :, None] * k[:, None, :]
            refs.append(np.einsum("hvd,hd->hv", St, q).reshape(-1))
        refs, rows = np.array(refs), slice(cu[b], cu[b + 1])
        for mine, token, ref in ((chunked[0][rows], out[rows], refs), (chunked[1][s, :nh * d * dv], S[s, :nh * d * dv], St.reshape(-1))):
            assert np.isfinite(mine).all()
            floor = 2.0 ** -24 * np.linalg.norm(ref)
            assert np.linalg.norm(mine - ref) <= 2 * np.linalg.norm(token - ref) + 4 * floor
        assert np.array_equal(chunked[1][s, nh * d * dv:], S[s, nh * d * dv:])       # the convolution's rows


@pytest.mark.parametrize("taps,d,dv,nh,nkv", [(4, 128, 64, 2, 1), (3, 16, 20, 3, 3), (2, 4, 4, 2, 2)])
@pytest.mark.parametrize("head_decay", [0, 1])
def test_delta_preparation_of_many_tokens(taps, d, dv, nh, nkv, head_decay):
    """A step of 512 tokens and more, which the preparation takes by eights of rows: sequences that meet inside an eight, some of them behind
    a past whose convolution rows lie in the state.  The bits are those of each sequence in a step of its own (one row at a time),
    and q, k, v, decays and write strengths those of float64."""
    lens, past = [1, 2, 3, 5, 130, 7, 201, 9, 166, 1], [0, 2, 1, 0, 5, 0, 1, 9, 0, 3]
    g = torch.Generator().manual_seed(taps * d + head_decay)
    T, B, C = sum(lens), len(lens), 2 * nkv * d + nh * dv
    assert T >= 512 and T % 8
    ld, na, elems = (C + nh + 3) // 4 * 4, nh if head_decay else nh * d, nh * d * dv + (taps - 1) * C
    x, a = torch.randn(T, ld, generator=g), torch.randn(T, na, generator=g)
    conv = [torch.randn(w, taps, generator=g) for w in (nkv * d, nkv * d, nh * dv)]
    a_log, dt, S0 = torch.randn(nh, generator=g) * 0.5, torch.randn(na, generator=g), torch.randn(B, elems, generator=g)
    f = entry("illm_delta_rule", I_, P_, I_, I_, I_, I_, I_, I_, P_, I_, I_, I_, I_, I_, I_, I_, P_, P_, P_, P_, P_, F_, P_, L_, P_, P_, P_, P_, P_, P_, P_, P_, P_, I_,
              I_, P_, P_)
    weights = [t.cuda() for t in (*conv, a_log, dt)]
    ints = lambda v: torch.tensor(list(v), dtype=torch.int32, device="cuda")  # noqa: E731

    def run(seqs, rows):
        n = [lens[b] for b in seqs]
        xd, ad, S = x[rows].cuda(), a[rows].cuda(), S0.cuda()
        cu, pos = ints([0, *np.cumsum(n)]), ints(past[b] + i for b in seqs for i in range(lens[b]))
        seq, slots, total = ints(i for i, b in enumerate(seqs) for _ in range(lens[b])), ints(seqs), ints(past[b] + lens[b] for b in seqs)
        outs = [torch.full((sum(n), w), float("nan"), device="cuda") for w in (C, na, nh, nh * dv)]
        rc = f(p(xd), sum(n), ld, 0, nkv * d, 2 * nkv * d, C, p(ad), na, head_decay, nh, nkv, d, dv, taps, *(p(t) for t in weights), d ** -0.5, p(S), elems, p(slots),
               p(cu), p(pos), p(seq), p(total), *(p(t) for t in outs), len(n), max(n), None, torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        return [t.cpu() for t in (*outs, S)]

    whole, cu = run(range(B), slice(0, T)), [0, *np.cumsum(lens)]
    sig = lambda z: 1.0 / (1.0 + np.exp(-z))  # noqa: E731
    taps_all = np.concatenate([c.double().numpy() for c in conv])
    for b in range(B):
        rows = slice(int(cu[b]), int(cu[b + 1]))
        one = run([b], rows)
        for mine, alone in zip(whole[:4], one[:4]):
            assert torch.equal(mine[rows], alone)
        assert torch.equal(whole[4][b], one[4][b])
        raw = np.concatenate([S0[b, nh * d * dv:].double().numpy().reshape(taps - 1, C), x[rows, :C].double().numpy()])
        raw[:max(0, taps - 1 - past[b])] = 0.0                 # positions before the sequence's start
        y = sum(raw[j:j + lens[b]] * taps_all[:, j] for j in range(taps))
        y = y * sig(y)
        for lo in range(0, 2 * nkv * d, d):
            head = y[:, lo:lo + d]
            y[:, lo:lo + d] = head / np.sqrt((head * head).sum(-1, keepdims=True) + 1e-6) * (d ** -0.5 if lo < nkv * d else 1.0)
        # fast exponentials in silu, whose error the norm of a head of small values enlarges
        assert np.abs(whole[0][rows].double().numpy() - y).max() <= 3e-5 * max(1.0, np.abs(y).max())
        z, rate = a[rows].double().numpy() + dt.double().numpy(), np.exp(a_log.double().numpy())
        want = np.exp(-(rate if head_decay else np.repeat(rate, d)) * np.logaddexp(0.0, z))
        assert np.abs(whole[1][rows].double().numpy() - want).max() <= 2e-5
        assert np.abs(whole[2][rows].double().numpy() - sig(x[rows, C:C + nh].double().numpy())).max() <= 1e-6


@pytest.mark.parametrize("d,dv,nh,nkv", [(128, 64, 2, 1), (64, 64, 4, 2), (20, 30, 2, 2), (9, 7, 3, 1)])
def test_delta_rule_own_chunks(d, dv, nh, nkv):
    """The delta rule's own chunks for the head sizes that chunk_scan.cu takes too: no more than twice as far from float64 as token by token."""
    taps, g = 2, torch.Generator().manual_seed(d * dv)
    cu, cu_d, pos, seq, slots, lens = layout()
    T, B, C = int(cu[-1]), len(LENS), 2 * nkv * d + nh * dv
    ld, elems = C + nh, nh * d * dv + (taps - 1) * C
    x, a = torch.randn(T, ld, generator=g), torch.randn(T, nh, generator=g)
    weights = [torch.randn(*s, generator=g).cuda() for s in ((nkv * d, taps), (nkv * d, taps), (nh * dv, taps), (nh,), (nh,))]
    S0, xd, ad = torch.randn(B, elems, generator=g), x.cuda(), a.cuda()
    f = entry("illm_delta_rule_form", I_, P_, I_, I_, I_, I_, I_, I_, P_, I_, I_, I_, I_, I_, I_, I_, P_, P_, P_, P_, P_, F_, P_, L_, P_, P_, P_, P_, P_, P_, P_, P_, P_, I_,
              I_, P_, I_, P_)
    n = entry("illm_delta_chunk_scratch", L_, I_, I_, I_)(T, B, nh)

    def run(own):
        S, out = S0.cuda(), torch.full((T, nh * dv), float("nan"), device="cuda")
        mid = [torch.empty(T, w, device="cuda") for w in (C, nh, nh)]
        rec = torch.full((n,), float("nan"), device="cuda") if own else None
        rc = f(p(xd), T, ld, 0, nkv * d, 2 * nkv * d, C, p(ad), nh, 1, nh, nkv, d, dv, taps, *(p(t) for t in weights), d ** -0.5, p(S), elems, p(slots), p(cu_d), p(pos), p(seq),
               p(lens), *(p(t) for t in mid), p(out), B, max(LENS), p(rec), own, torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        return [t.cpu().double().numpy() for t in (out, S, *mid)]

    chunked, (out, S, qkv, gg, beta) = run(1), run(0)
    share = nh // nkv
    for b in range(B):
        s, refs = B - 1 - b, []
        St = S0[s, :nh * d * dv].double().numpy().reshape(nh, dv, d).copy()
        for t in range(cu[b], cu[b + 1]):
            q, k, v = (qkv[t, lo:lo + w * e].reshape(w, e) for lo, w, e in ((0, nkv, d), (nkv * d, nkv, d), (2 * nkv * d, nh, dv)))
            q, k = q.repeat(share, 0), k.repeat(share, 0)
            St = St * gg[t].reshape(nh, 1, 1)
            St = St + (beta[t][:, None] * (v - np.einsum("hvd,hd->hv", St, k)))[:, :, None] * k[:, None, :]
            refs.append(np.einsum("hvd,hd->hv", St, q).reshape(-1))
        refs, rows = np.array(refs), slice(cu[b], cu[b + 1])
        for mine, token, ref in ((chunked[0][rows], out[rows], refs), (chunked[1][s, :nh * d * dv], S[s, :nh * d * dv], St.reshape(-1))):
            assert np.linalg.norm(mine - ref) <= 2 * np.linalg.norm(token - ref) + 4 * 2.0 ** -24 * np.linalg.norm(ref)
