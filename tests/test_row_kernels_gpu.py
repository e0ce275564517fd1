"""The kernels that keep a token's row in registers (norms, the preparation of q, k and v) and differential attention on tensor
memory, at the edges of their pieces, against float64 and against the kernels they stand in for."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_chunk_scan_gpu import F_, I_, L_, P_, entry, p   # noqa: E402

WIDTHS = [4, 36, 128, 516, 2048, 4096, 4100, 8192, 8196, 16384, 16388, 30, 4097]     # the last three: not whole pieces, or too wide


def stream():
    return torch.cuda.current_stream().cuda_stream


def close(got, ref, roundings, mag=None):
    """At most so many float32 roundings of the magnitude, plus the output's own rounding."""
    tol = roundings * 2.0 ** -24 + (2.0 ** -8 if got.dtype == torch.bfloat16 else 0.0)
    mag = np.abs(ref) if mag is None else mag
    assert (np.abs(got.cpu().double().numpy() - ref) <= tol * mag + 1e-30).all()


@pytest.mark.parametrize("H", [4, 8, 30, 1028, 4096])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("off_table,off_out", [(0, 0), (1, 0), (0, 1), (3, 2)])
def test_scaled_embedding_at_any_address(H, dtype, off_table, off_out):
    """Tables and outputs on 16-byte boundaries and off them, widths that are whole pieces or not: exact (one product per value)."""
    g = torch.Generator().manual_seed(H)
    V, T = 9, 5
    table, ids = torch.randn(V, H, generator=g).to(dtype), torch.tensor([8, 0, 3, 3, 7], dtype=torch.int32)
    held, out = torch.zeros(V * H + 8, dtype=dtype, device="cuda"), torch.full((T * H + 8,), float("nan"), device="cuda")
    held[off_table:off_table + V * H] = table.reshape(-1).cuda()
    err, idd = torch.zeros(1, dtype=torch.int32, device="cuda"), ids.cuda()
    rc = entry("illm_embedding_scaled", I_, P_, P_, P_, I_, P_, I_, I_, I_, F_, P_, P_, P_)(
        p(idd), p(idd), held[off_table:].data_ptr(), 1 if dtype == torch.bfloat16 else 0, out[off_out:].data_ptr(), T, H, V, 1.5, None, p(err), stream())
    assert rc == 0 and int(err) == 0
    assert torch.equal(out[off_out:off_out + T * H].cpu().view(T, H), table.float()[ids.long()] * 1.5)
    assert torch.isnan(out[:off_out]).all() and torch.isnan(out[off_out + T * H:]).all()


@pytest.mark.parametrize("H", WIDTHS)
@pytest.mark.parametrize("splits", [0, 3, 9])
def test_scale_add_rmsnorm(H, splits):
    g = torch.Generator().manual_seed(H + splits)
    n, alpha, eps = 3, 1.5, 1e-5
    x, w = torch.randn(n, H, generator=g), torch.randn(H, generator=g)
    add = torch.randn(max(1, splits), n, H, generator=g)
    xd, wd, ad = x.cuda(), w.cuda(), add.cuda()
    y = torch.empty(n, H, dtype=torch.bfloat16, device="cuda")
    rc = entry("illm_scale_add_rmsnorm", I_, P_, P_, I_, P_, P_, I_, I_, I_, F_, F_, P_, I_, L_, P_)(
        p(xd), None if splits else p(ad), 0, p(wd), p(y), 1, n, H, alpha, eps, p(ad) if splits else None, splits, n * H, stream())
    assert rc == 0
    v = alpha * x.double().numpy() + add.double().numpy().sum(0)
    mag = alpha * x.abs().double().numpy() + add.abs().double().numpy().sum(0)
    inv = 1.0 / np.sqrt((v * v).mean(-1, keepdims=True) + eps)
    ref, m = v * inv * w.double().numpy(), mag * inv * w.abs().double().numpy()
    for got in (xd, y):
        close(got, ref, 2 * math.sqrt(H) + 16, m)


@pytest.mark.parametrize("H", WIDTHS)
@pytest.mark.parametrize("center", [0, 1])
@pytest.mark.parametrize("with_y,with_rows", [(True, False), (False, True), (True, True)])
def test_norm_sandwich(H, center, with_y, with_rows):
    g = torch.Generator().manual_seed(H + center)
    n, eps, post = 4, 1e-5, 1.0 if center else 0.5
    x, y, wb, w = torch.randn(n, H, generator=g), torch.randn(n, H, generator=g), torch.randn(H, generator=g), torch.randn(H, generator=g)
    rows = torch.tensor([3, 1], dtype=torch.int32) if with_rows else None
    xd, yd, wbd, wd, rd = x.cuda(), y.cuda(), wb.cuda(), w.cuda(), rows.cuda() if with_rows else None
    n_out = 2 if with_rows else n
    out = torch.empty(n_out, H, dtype=torch.bfloat16, device="cuda")
    rc = entry("illm_norm_sandwich", I_, P_, P_, P_, P_, P_, I_, P_, I_, I_, F_, I_, I_, F_, P_)(
        p(xd), p(yd) if with_y else None, p(wbd) if with_y else None, p(wd), p(out), 1, p(rd), n_out, H, eps, 0 if with_rows else 1, center, post, stream())
    assert rc == 0

    def norm(v, weight):
        v = v - v.mean(-1, keepdims=True) if center else v
        return v / np.sqrt((v * v).mean(-1, keepdims=True) + eps) * weight.double().numpy()

    v = x.double().numpy() + (post * norm(y.double().numpy(), wb) if with_y else 0.0)
    if not with_rows:
        close(xd, v, 2 * math.sqrt(H) + 16, np.abs(v) + np.abs(x.double().numpy()) + 4)
    ref = norm(v, w)[[3, 1]] if with_rows else norm(v, w)
    close(out, ref, 4 * math.sqrt(H) + 32, np.abs(ref) + 4 * w.abs().double().numpy())


@pytest.mark.parametrize("H", [64, 4096, 5120, 8192, 12288, 20480, 4097])
@pytest.mark.parametrize("center", [0, 1])
def test_norm_sandwich_rows_do_not_depend_on_the_step(H, center):
    """A row of many (more than the SMs, which take another form of the kernel) has the bits that it has alone."""
    g = torch.Generator().manual_seed(H + center)
    n, post = 400, 1.0 if center else 0.5
    x, y, wb, w = (torch.randn(*s, generator=g).cuda() for s in ((n, H), (n, H), (H,), (H,)))
    f = entry("illm_norm_sandwich", I_, P_, P_, P_, P_, P_, I_, P_, I_, I_, F_, I_, I_, F_, P_)

    def run(at, rows):
        xd, yd, out = x[at:at + rows].clone(), y[at:at + rows].clone(), torch.empty(rows, H, device="cuda")
        assert f(p(xd), p(yd), p(wb), p(w), p(out), 0, None, rows, H, 1e-5, 1, center, post, stream()) == 0
        return xd, out

    many = run(0, n)
    for at in (0, 7, n - 1):
        for a, b in zip(run(at, 1), many):
            assert torch.equal(a[0], b[at])


@pytest.mark.parametrize("name", ["illm_norm_sandwich", "illm_add2_rmsnorm", "illm_scaled_add_rmsnorm"])
def test_norms_of_wide_rows_take_their_bytes_time(name):
    """2,048 rows of 20,480 channels beside as many of 8,192, both at the rate of memory: 2.5 times the bytes, at most twice that in time."""
    f = entry(name, I_, P_, P_, P_, P_, P_, I_, P_, I_, I_, F_, I_, I_, F_, P_) if "sandwich" in name else entry(name, I_, P_, P_, P_, P_, P_, I_, I_, I_, F_, P_)
    n, times = 2048, []
    for H in (8192, 20480):
        x, a, b, w = (torch.randn(*s, device="cuda") for s in ((n, H), (n, H), (n, H), (H,)))
        y = torch.empty(n, H, dtype=torch.bfloat16, device="cuda")
        args = {"illm_norm_sandwich": (p(x), p(a), p(w), p(w), p(y), 1, None, n, H, 1e-5, 1, 0, 0.5), "illm_add2_rmsnorm": (p(x), p(a), p(b), p(w), p(y), 1, n, H, 1e-5),
                "illm_scaled_add_rmsnorm": (p(x), p(a), p(w), p(w), p(y), 1, n, H, 1e-5)}[name]
        best = float("inf")
        for _ in range(5):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            assert f(*args, stream()) == 0
            torch.cuda._sleep(1 << 21)
            begin.record()
            for _ in range(5):
                f(*args, stream())
            end.record()
            end.synchronize()
            best = min(best, begin.elapsed_time(end))
        times.append(best)
    assert times[1] <= 5 * times[0], times


@pytest.mark.parametrize("width,group", [(2048, 2048), (1032, 516), (8192, 8192), (1024, 128), (12, 4), (8196, 8196), (30, 15)])
@pytest.mark.parametrize("act", [1, 2])
def test_group_norm_gate(width, group, act):
    g = torch.Generator().manual_seed(width + act)
    T, eps = 3, 1e-5
    o, gate, w = torch.randn(T, width, generator=g), torch.randn(T, width + 4, generator=g), torch.randn(group, generator=g)
    y, od, gd, wd = torch.empty(T, width, device="cuda"), o.cuda(), gate.cuda(), w.cuda()
    rc = entry("illm_group_norm_gate_ex", I_, P_, I_, I_, I_, P_, I_, F_, P_, I_, I_, I_, P_, I_, P_, P_, I_, P_, I_, P_)(
        p(od), T, width, group, p(wd), group, eps, p(gd), width + 4, act, 0, None, 0, None, None, 0, p(y), 0, stream())
    assert rc == 0
    v, z = o.double().numpy().reshape(T, -1, group), gate.double().numpy()[:, :width]
    sig = 1.0 / (1.0 + np.exp(-z))
    ref = (v / np.sqrt((v * v).mean(-1, keepdims=True) + eps) * w.double().numpy()).reshape(T, width) * (z * sig if act == 1 else sig)
    close(y, ref, 2 * math.sqrt(group) + 24)


@pytest.mark.parametrize("nh,nkv,d,dv,rot,pairs,norm,qt,mix,own", [
    (8, 2, 128, 128, 64, 1, "whole", 0, False, True), (8, 2, 128, 128, 64, 1, "head", 0, False, True), (4, 4, 64, 96, 30, 0, "none", 4, False, True),
    (5, 1, 36, 20, 36, 1, "none", 0, True, True), (6, 2, 16, 16, 6, 0, "head", 0, False, True), (16, 4, 128, 128, 128, 0, "whole", 0, False, False),
    (32, 8, 128, 128, 0, 1, "none", 16, False, True), (3, 3, 4, 4, 4, 1, "whole", 0, True, True), (40, 40, 128, 128, 64, 1, "none", 0, False, True)])
def test_qk_prep_by_pieces(nh, nkv, d, dv, rot, pairs, norm, qt, mix, own):
    """Rows that begin on 16-byte boundaries (four channels per thread) and the same rows one float further on (the channel by channel
    kernel) give the same values up to the order of a norm's sum."""
    g = torch.Generator().manual_seed(nh * d + rot)
    T, page, n_pos = 5, 8, 64
    nq, nk, nv = nh * d, nkv * d, nkv * dv
    cols = nq + (nk + nv if own else 0)
    rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    x, bq, bk, bv = rnd(T, cols), rnd(nq), rnd(nk), rnd(nv)
    wq, wk = (rnd(nq), rnd(nk)) if norm == "whole" else (rnd(d), rnd(d))
    cs, first, lam = rnd(n_pos, max(1, rot // 2), 2), rnd(T, nv), torch.tensor([0.3])
    pos, seq = torch.tensor([0, 7, 8, 30, 63], dtype=torch.int32), torch.tensor([0, 0, 0, 1, 1], dtype=torch.int32)
    table = torch.arange(16, dtype=torch.int32).view(2, 8).flip(0).contiguous()
    f = entry("illm_qk_prep_heads", I_, P_, I_, I_, I_, I_, I_, I_, I_, I_, I_, P_, P_, P_, P_, P_, F_, P_, I_, I_, I_, P_, P_, P_, I_, I_, P_, P_, P_, I_, I_, P_, F_,
              I_, P_, I_, P_, P_, I_, P_)
    keep = [t.cuda() for t in (bq, bk, bv, wq, wk, cs, first, lam, pos, seq, table)]

    def run(shift):
        xd = torch.zeros(T, cols + 4, device="cuda")
        xd[:, shift:shift + cols] = x.cuda()
        q = torch.full((T, nq), float("nan"), device="cuda")
        kc, vc = torch.zeros(16, nkv, page, d, device="cuda"), torch.zeros(16, nkv, page, dv, device="cuda")
        kept, err = torch.zeros(T, nv, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        bqd, bkd, bvd, wqd, wkd, csd, fd, ld, pd, sd, td = keep
        rc = f(p(xd), 0, cols + 4, shift, shift + nq if own else -1, shift + nq + nk if own else -1, nh, nkv, d, dv, p(bqd), p(bkd) if own else None,
               p(bvd) if own else None, None if norm == "none" else p(wqd), None if norm == "none" or not own else p(wkd), 1e-5, p(csd), rot, pairs, n_pos, p(pd),
               p(sd), p(td), 8, page, p(q), p(kc) if own else None, p(vc) if own else None, 0, T, p(err), 0.25, qt, p(fd) if mix else None, nv,
               p(ld) if mix else None, p(kept) if mix else None, 1 if norm == "head" else 0, stream())
        assert rc == 0 and int(err) == 0
        return [t.cpu() for t in (q, kc, vc, kept)]

    for a, b in zip(run(0), run(1)):
        assert torch.isfinite(a).all()
        assert (a - b).abs().max() <= (2 * math.sqrt(nq) + 8) * 2.0 ** -24 * max(1.0, float(b.abs().max()))
    assert not own or float(run(0)[1].abs().sum()) > 0


@pytest.mark.parametrize("nh,nkv,d,rot,pairs,norm,mix", [(32, 8, 128, 128, 0, "whole", False), (32, 8, 128, 64, 1, "head", True), (8, 2, 64, 30, 0, "none", True),
                                                        (40, 40, 128, 128, 0, "head", False), (6, 2, 20, 20, 1, "whole", True), (5, 5, 30, 30, 0, "whole", True)])
def test_qk_prep_rows_do_not_depend_on_the_step(nh, nkv, d, rot, pairs, norm, mix):
    """A token of many (more than the SMs, which take another form of the kernel) has the bits that it has alone."""
    g = torch.Generator().manual_seed(nh * d + rot)
    T, page = 320, 64
    nq, nk = nh * d, nkv * d
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    x, bq, bk, bv, first, lam, cs = rnd(T, nq + 2 * nk), rnd(nq), rnd(nk), rnd(nk), rnd(T, nk), torch.tensor([0.3]).cuda(), rnd(T, max(1, rot // 2), 2)
    wq, wk = (rnd(nq), rnd(nk)) if norm == "whole" else (rnd(d), rnd(d))
    pos, seq = torch.arange(T, dtype=torch.int32).cuda(), torch.zeros(T, dtype=torch.int32).cuda()
    table = torch.arange(T // page, dtype=torch.int32).view(1, -1).cuda()
    f = entry("illm_qk_prep_heads", I_, P_, I_, I_, I_, I_, I_, I_, I_, I_, I_, P_, P_, P_, P_, P_, F_, P_, I_, I_, I_, P_, P_, P_, I_, I_, P_, P_, P_, I_, I_, P_, F_,
              I_, P_, I_, P_, P_, I_, P_)

    def run(at, n):
        q, kept, err = torch.empty(n, nq, device="cuda"), torch.empty(n, nk, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        kc, vc = (torch.zeros(T // page, nkv, page, d, device="cuda") for _ in range(2))
        own = [t[at:at + n].contiguous() for t in (x, pos, seq, first)]
        assert f(p(own[0]), 0, nq + 2 * nk, 0, nq, nq + nk, nh, nkv, d, d, p(bq), p(bk), p(bv), None if norm == "none" else p(wq), None if norm == "none" else p(wk),
                 1e-5, p(cs), rot, pairs, T, p(own[1]), p(own[2]), p(table), T // page, page, p(q), p(kc), p(vc), 0, n, p(err), 0.25, 16, p(own[3]) if mix else None,
                 nk, p(lam) if mix else None, p(kept) if mix else None, 1 if norm == "head" else 0, stream()) == 0
        rows = [c[:, :, :].transpose(1, 2).reshape(T, nk)[at:at + n] for c in (kc, vc)]
        assert int(err) == 0
        return [q, *rows] + ([kept] if mix else [])

    many = run(0, T)
    for at in (0, 77, T - 1):
        for a, b in zip(run(at, 1), many):
            assert torch.equal(a[0], b[at])


def test_qk_prep_of_many_tokens_takes_its_bytes_time():
    """2,000 tokens of 32 + 2 x 8 heads of 128, rotate-half and norms over all heads: 47 us with two blocks an SM, 68 with one."""
    nh, nkv, d, T, page = 32, 8, 128, 2000, 64
    nq, nk, w = nh * d, nkv * d, -(-T // 64)
    x, wq, wk, cs = torch.randn(T, nq + 2 * nk, device="cuda"), torch.randn(nq, device="cuda"), torch.randn(nk, device="cuda"), torch.randn(T, d // 2, 2, device="cuda")
    pos, seq, table = (torch.as_tensor(a, dtype=torch.int32).cuda() for a in (np.arange(T), np.zeros(T), np.arange(w)[None]))
    q, err = torch.empty(T, nq, dtype=torch.bfloat16, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    kc, vc = (torch.zeros(w, nkv, page, d, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    f = entry("illm_qk_prep_heads", I_, P_, I_, I_, I_, I_, I_, I_, I_, I_, I_, P_, P_, P_, P_, P_, F_, P_, I_, I_, I_, P_, P_, P_, I_, I_, P_, P_, P_, I_, I_, P_, F_,
              I_, P_, I_, P_, P_, I_, P_)
    best = float("inf")
    for _ in range(5):
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda._sleep(1 << 21)
        begin.record()
        for _ in range(10):
            assert f(p(x), 0, nq + 2 * nk, 0, nq, nq + nk, nh, nkv, d, d, None, None, None, p(wq), p(wk), 1e-5, p(cs), d, 0, T, p(pos), p(seq), p(table), w, page, p(q),
                     p(kc), p(vc), 1, T, p(err), 0.0, 0, None, 0, None, None, 0, stream()) == 0
        end.record()
        end.synchronize()
        best = min(best, begin.elapsed_time(end) * 100)
    assert best <= 58, best          # microseconds


@pytest.mark.parametrize("nh,nkv,window,lens", [(4, 2, 0, [1, 63, 64, 65, 300]), (8, 1, 0, [129]), (3, 3, 70, [200, 5]), (2, 1, 1, [70])])
def test_differential_attention_on_tensor_memory(nh, nkv, window, lens):
    """Beside the warp-level MMA kernel, both against float64: no farther from it than that one by more than a half, and within two
    bfloat16 roundings of the output."""
    d, dv, page = 64, 128, 64
    g = torch.Generator().manual_seed(nh + window)
    T, B = sum(lens), len(lens)
    width = max(-(-n // page) for n in lens) + 1
    n_pages = B * width
    table = torch.randperm(n_pages, generator=g).to(torch.int32).view(B, width)
    q = (torch.randn(T, nh * 2 * d, generator=g)).bfloat16()
    ks, vs = [torch.randn(n, nkv, 2 * d, generator=g).bfloat16() for n in lens], [torch.randn(n, nkv, dv, generator=g).bfloat16() for n in lens]
    kc, vc = (torch.full((n_pages, nkv, page, w), float("nan"), dtype=torch.bfloat16) for w in (2 * d, dv))
    for b, n in enumerate(lens):
        for t in range(n):
            kc[table[b, t // page], :, t % page], vc[table[b, t // page], :, t % page] = ks[b][t], vs[b][t]
    cu = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32)
    dev = [t.cuda() for t in (q, kc, vc, table.contiguous(), cu, torch.tensor(lens, dtype=torch.int32))]
    scale, lam, eps, factor = d ** -0.5, 0.45, 1e-6, 0.6
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    maps = torch.empty(T, nh, 2, dv, device="cuda")
    outs = [torch.full((T, nh * dv), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    rc = entry("illm_attention_diff_tc", I_, P_, I_, I_, P_, P_, L_, P_, I_, P_, P_, P_, P_, I_, I_, I_, I_, I_, I_, I_, I_, F_, F_, F_, F_, P_, P_)(
        p(dev[0]), nh * 2 * d, T, p(dev[1]), p(dev[2]), n_pages, p(dev[3]), width, p(dev[4]), p(dev[5]), p(maps), p(outs[0]), B, max(lens), nh, nkv, d, dv, page,
        window, scale, lam, eps, factor, p(err), stream())
    assert rc == 0
    rc = entry("illm_attention_diff_mma", I_, P_, I_, P_, P_, P_, I_, P_, P_, P_, I_, I_, I_, I_, I_, I_, I_, I_, F_, F_, F_, F_, P_)(
        p(dev[0]), nh * 2 * d, p(dev[1]), p(dev[2]), p(dev[3]), width, p(dev[4]), p(dev[5]), p(outs[1]), B, max(lens), nh, nkv, d, dv, page, window, scale, lam, eps,
        factor, stream())
    assert rc == 0 and int(err) == 0
    got, other = (o.cpu().double().numpy().reshape(T, nh, dv) for o in outs)
    for b, n in enumerate(lens):
        qq = q[cu[b]:cu[b + 1]].double().numpy().reshape(n, nh, 2, d)
        i, j = np.arange(n)[:, None], np.arange(n)[None]
        hide = (j > i) | ((i - j >= window) if window else False)
        ref = np.zeros((n, nh, dv))
        for h in range(nh):
            k, v = ks[b][:, h // (nh // nkv)].double().numpy().reshape(n, 2, d), vs[b][:, h // (nh // nkv)].double().numpy()
            a = []
            for m in range(2):
                s = np.where(hide, -np.inf, qq[:, h, m] @ k[:, m].T * scale)
                e = np.exp(s - s.max(-1, keepdims=True))
                a.append(e / e.sum(-1, keepdims=True) @ v)
            o = a[0] - lam * a[1]
            ref[:, h] = o / np.sqrt((o * o).mean(-1, keepdims=True) + eps) * factor
        mine, theirs = (np.abs(x[cu[b]:cu[b + 1]] - ref) for x in (got, other))
        assert (mine <= 2.0 ** -7 * np.abs(ref) + 2.0 ** -9).all()
        assert np.linalg.norm(mine) <= 1.5 * np.linalg.norm(theirs) + 1e-6


@pytest.mark.parametrize("heads", [1, 2, 5])
def test_differential_attention_in_passes_over_heads(heads):
    """Any number of heads per pass gives the bits of one pass over all, and a pass's scratch is bounded."""
    nh, nkv, d, dv, page, lens = 6, 2, 64, 128, 64, [5, 200, 64]
    g = torch.Generator().manual_seed(heads)
    _, pools, table = paged(lens, nkv, (2 * d, dv), g)
    T, B, width, n_pages = sum(lens), len(lens), table.shape[1], pools[0].shape[0]
    q = torch.randn(T, nh * 2 * d, generator=g).bfloat16()
    cu = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32)
    dev = [t.cuda() for t in (q, *pools, table, cu, torch.tensor(lens, dtype=torch.int32))]
    err, outs = torch.zeros(1, dtype=torch.int32, device="cuda"), []
    for n in (nh, heads):
        guard = 64
        maps = torch.full((T * n * 2 * dv + guard,), -7.0, device="cuda")
        out = torch.full((T, nh * dv), float("nan"), dtype=torch.bfloat16, device="cuda")
        rc = entry("illm_attention_diff_tc_sliced", I_, P_, I_, I_, P_, P_, L_, P_, I_, P_, P_, P_, P_, I_, I_, I_, I_, I_, I_, I_, I_, F_, F_, F_, F_, I_, P_, P_)(
            p(dev[0]), nh * 2 * d, T, p(dev[1]), p(dev[2]), n_pages, p(dev[3]), width, p(dev[4]), p(dev[5]), p(maps), p(out), B, max(lens), nh, nkv, d, dv, page, 0,
            d ** -0.5, 0.45, 1e-6, 0.6, n, p(err), stream())
        assert rc == 0 and (maps[-guard:] == -7.0).all()
        outs.append(out.cpu())
    assert int(err) == 0 and torch.isfinite(outs[0].float()).all() and torch.equal(outs[0], outs[1])
    per_pass = entry("illm_attention_diff_tc_heads", I_, L_, I_, I_)
    for T in (1, 1777, 4096, 16384, 65536, 1 << 20):
        n = per_pass(T, 32, dv)
        assert 1 <= n <= 32 and (n == 1 or n * T * 2 * dv * 4 <= 128 << 20)
    assert per_pass(4096, 32, dv) == 32


@pytest.mark.parametrize("H", [4, 516, 4096, 4100, 16384])
@pytest.mark.parametrize("n1,n2", [(1, 1), (3, 1), (9, 2), (17, 0)])
def test_addends_as_slices(H, n1, n2):
    """What the norms make of one or two addends that come as K slices, against float64: add2_rmsnorm, scaled_add_rmsnorm and
    norm_sandwich (whose first norm reads the sum)."""
    g = torch.Generator().manual_seed(H + n1)
    T, eps = 3, 1e-5
    x, w, ls = torch.randn(T, H, generator=g), torch.randn(H, generator=g), torch.randn(H, generator=g)
    a, b = torch.randn(n1, T, H, generator=g), torch.randn(max(1, n2), T, H, generator=g)
    xs, s1, s2 = x.double().numpy(), a.double().numpy().sum(0), b.double().numpy().sum(0) if n2 else 0.0
    dev = [t.cuda() for t in (a, b, w, ls)]
    y = torch.empty(T, H, device="cuda")
    tol = 4 * math.sqrt(H) + 40 + n1

    def norm(v, weight):
        return v / np.sqrt((v * v).mean(-1, keepdims=True) + eps) * weight.double().numpy()

    big = 4.0 * (n1 + n2 + 2) * w.abs().double().numpy() + 1e-3
    xd = x.cuda()
    rc = entry("illm_add2_rmsnorm_slices", I_, P_, P_, I_, L_, P_, I_, L_, P_, P_, I_, I_, I_, F_, P_)(
        p(xd), p(dev[0]), n1, T * H, p(dev[1]) if n2 else None, max(1, n2), T * H, p(dev[2]), p(y), 0, T, H, eps, stream())
    assert rc == 0
    close(xd, xs + s1 + s2, n1 + n2 + 4, np.abs(xs) + 4.0 * (n1 + n2))
    close(y, norm(xs + s1 + s2, w), tol, big)
    xd = x.cuda()
    rc = entry("illm_scaled_add_rmsnorm_slices", I_, P_, P_, I_, L_, P_, P_, P_, I_, I_, I_, F_, P_)(
        p(xd), p(dev[0]), n1, T * H, p(dev[3]), p(dev[2]), p(y), 0, T, H, eps, stream())
    assert rc == 0
    v = xs + s1 * ls.double().numpy()
    close(y, norm(v, w), tol, big * (1 + ls.abs().double().numpy()) + np.abs(norm(v, w)))
    xd = x.cuda()
    rc = entry("illm_norm_sandwich_slices", I_, P_, P_, I_, L_, P_, P_, P_, I_, P_, I_, I_, F_, I_, I_, F_, P_)(
        p(xd), p(dev[0]), n1, T * H, p(dev[3]), p(dev[2]), p(y), 0, None, T, H, eps, 1, 0, 0.5, stream())
    assert rc == 0
    v = xs + 0.5 * norm(s1, ls)
    close(y, norm(v, w), tol, big * (1 + ls.abs().double().numpy()) + np.abs(norm(v, w)))


def paged(lens, nkv, widths, g, page=64):
    """Keys and values of sequences in pages dealt out at random, rows that nothing wrote full of NaN: the rows, the pools and the table."""
    width = max(-(-n // page) for n in lens) + 1
    table = torch.randperm(len(lens) * width, generator=g).to(torch.int32).view(len(lens), width)
    rows = [[torch.randn(n, nkv, w, generator=g).bfloat16() for n in lens] for w in widths]
    pools = [torch.full((len(lens) * width, nkv, page, w), float("nan"), dtype=torch.bfloat16) for w in widths]
    for pool, of in zip(pools, rows):
        for b, n in enumerate(lens):
            for t in range(n):
                pool[table[b, t // page], :, t % page] = of[b][t]
    return rows, pools, table


def weights_of(q, k, scale, window, cap=0.0, sink=None):
    """Float64 softmax weights of the last token's heads [heads, d] over keys [n, d]."""
    s = q @ k.T * scale
    s = np.tanh(s / cap) * cap if cap else s
    if window:
        s[:, :max(0, k.shape[0] - window)] = -np.inf
    top = s.max(-1, keepdims=True) if sink is None else np.maximum(s.max(-1, keepdims=True), sink[:, None])
    e = np.exp(s - top)
    return e / (e.sum(-1, keepdims=True) + (0.0 if sink is None else np.exp(sink[:, None] - top)))


@pytest.mark.parametrize("nh,nkv,window,lens", [(8, 1, 0, [1, 64, 65, 700]), (32, 4, 0, [1821]), (3, 3, 70, [200, 5]), (2, 1, 1, [70])])
@pytest.mark.parametrize("splits", [1, 3, 16])
def test_differential_attention_of_single_tokens(nh, nkv, window, lens, splits):
    """Beside the kernel on CUDA cores, both against float64: as near to it as that one (both round their output to bfloat16)."""
    d, dv, page, T = 64, 128, 64, len(lens)
    g = torch.Generator().manual_seed(nh + window + splits)
    (ks, vs), pools, table = paged(lens, nkv, (2 * d, dv), g)
    q = torch.randn(T, nh * 2 * d, generator=g).bfloat16()
    width, n_pages = table.shape[1], pools[0].shape[0]
    dev = [t.cuda() for t in (q, *pools, table, torch.tensor(lens, dtype=torch.int32) - 1, torch.arange(T, dtype=torch.int32))]
    scale, lam, eps, factor = d ** -0.5, 0.45, 1e-6, 0.6
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    outs = [torch.full((T, nh * dv), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    acc, ml = torch.empty(T * nh * 2 * splits * dv, device="cuda"), torch.empty(T * nh * 2 * splits * 2, device="cuda")
    rc = entry("illm_attention_diff_ring", I_, P_, I_, P_, P_, L_, P_, I_, P_, P_, P_, P_, P_, I_, I_, I_, I_, I_, I_, I_, F_, I_, F_, F_, F_, P_, P_)(
        p(dev[0]), nh * 2 * d, p(dev[1]), p(dev[2]), n_pages, p(dev[3]), width, p(dev[4]), p(dev[5]), p(acc), p(ml), p(outs[0]), T, nh, nkv, d, dv, page, window,
        scale, splits, lam, eps, factor, p(err), stream())
    assert rc == 0
    scratch = torch.empty(T * nh * 2 * 64 * (dv + 2), device="cuda")
    rc = entry("illm_attention_diff_decode", I_, P_, I_, P_, P_, P_, I_, P_, P_, P_, I_, I_, I_, I_, I_, I_, I_, F_, F_, F_, F_, L_, I_, P_, P_)(
        p(dev[0]), nh * 2 * d, p(dev[1]), p(dev[2]), p(dev[3]), width, p(dev[4]), p(dev[5]), p(outs[1]), T, nh, nkv, d, dv, page, window, scale, lam, eps, factor,
        max(lens), 4, p(scratch), stream())
    assert rc == 0 and int(err) == 0
    ref = np.zeros((T, nh, dv))
    for b in range(T):
        kv = np.arange(nh) // (nh // nkv)
        qq, k, v = q[b].double().numpy().reshape(nh, 2, d), ks[b].double().numpy().reshape(-1, nkv, 2, d), vs[b].double().numpy()
        for h in range(nh):
            a = [weights_of(qq[h:h + 1, m], k[:, kv[h], m], scale, window) @ v[:, kv[h]] for m in range(2)]
            o = (a[0] - lam * a[1])[0]
            ref[b, h] = o / np.sqrt((o * o).mean() + eps) * factor
    mine, theirs = (np.abs(o.cpu().double().numpy().reshape(T, nh, dv) - ref) for o in outs)
    # the output's rounding, and 2^-16 of the values' size for the weights' two terms, the products and the powers of two
    assert (mine <= 2.0 ** -8 * np.abs(ref) + 2.0 ** -12).all()
    print("errors", np.linalg.norm(mine) / np.linalg.norm(ref), np.linalg.norm(theirs) / np.linalg.norm(ref))
    assert np.linalg.norm(mine) <= 1.01 * np.linalg.norm(theirs) + 1e-6


def test_merge_of_shares_at_any_address():
    """The shares' words need no more than a float's alignment: the same bits from scratch that starts one float further on."""
    nh, d, dv, splits, lens = 4, 64, 128, 3, [300, 65]
    g = torch.Generator().manual_seed(3)
    _, pools, table = paged(lens, 1, (2 * d, dv), g)
    T, outs = len(lens), []
    dev = [t.cuda() for t in (torch.randn(T, nh * 2 * d, generator=g).bfloat16(), *pools, table, torch.tensor(lens, dtype=torch.int32) - 1, torch.arange(T, dtype=torch.int32))]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for off in (0, 1):
        acc, ml = (torch.empty(T * nh * 2 * splits * w + off, device="cuda")[off:] for w in (dv, 2))
        out = torch.full((T, nh * dv), float("nan"), dtype=torch.bfloat16, device="cuda")
        rc = entry("illm_attention_diff_ring", I_, P_, I_, P_, P_, L_, P_, I_, P_, P_, P_, P_, P_, I_, I_, I_, I_, I_, I_, I_, F_, I_, F_, F_, F_, P_, P_)(
            p(dev[0]), nh * 2 * d, p(dev[1]), p(dev[2]), pools[0].shape[0], p(dev[3]), table.shape[1], p(dev[4]), p(dev[5]), p(acc), p(ml), p(out), T, nh, 1, d, dv, 64,
            0, d ** -0.5, splits, 0.45, 1e-6, 0.6, p(err), stream())
        assert rc == 0 and int(err) == 0
        outs.append(out.cpu())
    assert torch.isfinite(outs[0].float()).all() and torch.equal(*outs)


def shares(acc, ml, base2):
    """(acc, maximum, sum) of a head's shares put together in float64; base2: the maxima are in units of log2."""
    m, l = ml[..., 0].double(), ml[..., 1].double()
    w = torch.exp2(m - m.amax(-1, keepdim=True)) if base2 else torch.exp(m - m.amax(-1, keepdim=True))
    live = (w > 0)[..., None]
    return ((torch.where(live, acc.double(), 0.0) * w[..., None]).sum(-2) / (l * w).sum(-1)[..., None]).cpu().numpy()


@pytest.mark.parametrize("maps", [1, 2])
@pytest.mark.parametrize("sharp", [0.3, 1.0, 4.0])
def test_ring_attention_keeps_float32_weights(maps, sharp):
    """Single tokens of differential heads (two maps) and of a group of 32 heads: what the shares hold before the output is rounded is no
    farther from float64 than the float32 kernel's on CUDA cores.  sharp: the scores' spread."""
    nh, nkv, d, dv, page, splits = 32, 4 if maps == 2 else 1, 64 if maps == 2 else 128, 128, 64, 4
    lens = [17, 400, 2100]
    T, scale = len(lens), sharp * d ** -0.5
    g = torch.Generator().manual_seed(maps)
    (ks, vs), pools, table = paged(lens, nkv, (maps * d, dv), g)
    q = torch.randn(T, nh * maps * d, generator=g).bfloat16()
    width, n_pages = table.shape[1], pools[0].shape[0]
    dev = [t.cuda() for t in (q, *pools, table, torch.tensor(lens, dtype=torch.int32) - 1, torch.arange(T, dtype=torch.int32))]
    err, out = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.empty(T, nh * dv, dtype=torch.bfloat16, device="cuda")
    acc, ml = torch.empty(T, nh, maps, splits, dv, device="cuda"), torch.empty(T, nh, maps, splits, 2, device="cuda")
    old = torch.empty(T, nh, splits, maps, dv + 2, device="cuda")
    if maps == 2:
        rc = entry("illm_attention_diff_ring", I_, P_, I_, P_, P_, L_, P_, I_, P_, P_, P_, P_, P_, I_, I_, I_, I_, I_, I_, I_, F_, I_, F_, F_, F_, P_, P_)(
            p(dev[0]), nh * 2 * d, p(dev[1]), p(dev[2]), n_pages, p(dev[3]), width, p(dev[4]), p(dev[5]), p(acc), p(ml), p(out), T, nh, nkv, d, dv, page, 0, scale,
            splits, 0.4, 1e-6, 1.0, p(err), stream())
        rc |= entry("illm_attention_diff_decode", I_, P_, I_, P_, P_, P_, I_, P_, P_, P_, I_, I_, I_, I_, I_, I_, I_, F_, F_, F_, F_, L_, I_, P_, P_)(
            p(dev[0]), nh * 2 * d, p(dev[1]), p(dev[2]), p(dev[3]), width, p(dev[4]), p(dev[5]), p(out), T, nh, nkv, d, dv, page, 0, scale, 0.4, 1e-6, 1.0, max(lens),
            splits, p(old), stream())
    else:
        rc = entry("illm_attention_decode_ring_shared", I_, P_, I_, P_, P_, L_, P_, I_, P_, P_, P_, P_, P_, I_, I_, I_, I_, I_, I_, F_, I_, P_, I_, P_, P_, I_, I_, F_, I_,
                   P_)(p(dev[0]), nh * d, p(dev[1]), p(dev[2]), n_pages, p(dev[3]), width, p(dev[4]), p(dev[5]), p(acc), p(ml), p(out), T, nh, nkv, d, page, 0, scale,
                       splits, p(err), 1, None, None, 0, 0, 0.0, 2, stream())
        rc |= entry("illm_attention_one_decode", I_, P_, I_, P_, P_, P_, I_, P_, P_, P_, I_, I_, I_, I_, I_, I_, I_, F_, F_, P_, P_, I_, I_, L_, I_, P_, P_)(
            p(dev[0]), nh * d, p(dev[1]), p(dev[2]), p(dev[3]), width, p(dev[4]), p(dev[5]), p(out), T, nh, nkv, d, d, page, 0, scale, 0.0, None, None, 0, 0, max(lens),
            splits, p(old), stream())
    assert rc == 0 and int(err) == 0
    ring, cores = shares(acc, ml, True), shares(old[..., 2:].transpose(2, 3), old[..., :2].transpose(2, 3), False)
    num = [0.0, 0.0]
    for b in range(T):
        qq, k, v = q[b].double().numpy().reshape(nh, maps, d), ks[b].double().numpy().reshape(-1, nkv, maps, d), vs[b].double().numpy()
        for h in range(nh):
            hk = h // (nh // nkv)
            for m in range(maps):
                ref = (weights_of(qq[h:h + 1, m], k[:, hk, m], scale, 0) @ v[:, hk])[0]
                for i, got in enumerate((ring, cores)):
                    num[i] += (np.linalg.norm(got[b, h, m] - ref) / np.linalg.norm(ref)) ** 2
    ours, theirs = (math.sqrt(x / (T * nh * maps)) for x in num)
    print("errors before the output's rounding:", maps, sharp, ours, theirs)
    assert ours <= theirs


@pytest.mark.parametrize("maps", [1, 2])
@pytest.mark.parametrize("splits", [1, 3])
def test_ring_attention_of_infinite_keys(maps, splits):
    """A key with an infinite channel whose scores are minus infinity has weight 0 in its own map and the other map does not see it, among
    other keys and as the only one of the last 16 (differential heads; a group of 32 heads)."""
    nh, nkv, d, dv, page = 32, 4 if maps == 2 else 1, 64 if maps == 2 else 128, 128, 64
    lens, far = [40, 65, 300, 300], [3, 64, 17, 299]
    T, scale = len(lens), d ** -0.5
    g = torch.Generator().manual_seed(maps)
    q = torch.randn(T, nh, maps, d, generator=g).bfloat16()
    q[:, :, maps - 1, 5] = -q[:, :, maps - 1, 5].abs() - 0.1
    width = max(-(-n // page) for n in lens)
    table = torch.arange(T * width, dtype=torch.int32).view(T, width)
    ks, vs = [[torch.randn(n, nkv, w, generator=g).bfloat16() for n in lens] for w in (maps * d, dv)]
    kc, vc = (torch.full((T * width, nkv, page, w), float("nan"), dtype=torch.bfloat16) for w in (maps * d, dv))
    for b, n in enumerate(lens):
        ks[b][far[b], :, (maps - 1) * d + 5] = float("inf")
        for t in range(n):
            kc[table[b, t // page], :, t % page], vc[table[b, t // page], :, t % page] = ks[b][t], vs[b][t]
    dev = [t.cuda() for t in (q.reshape(T, -1), kc, vc, table, torch.tensor(lens, dtype=torch.int32) - 1, torch.arange(T, dtype=torch.int32))]
    err, out = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.empty(T, nh * dv, dtype=torch.bfloat16, device="cuda")
    acc, ml = torch.empty(T * nh * maps * splits * dv, device="cuda"), torch.empty(T * nh * maps * splits * 2, device="cuda")
    lam, eps = 0.4, 1e-6
    if maps == 2:
        rc = entry("illm_attention_diff_ring", I_, P_, I_, P_, P_, L_, P_, I_, P_, P_, P_, P_, P_, I_, I_, I_, I_, I_, I_, I_, F_, I_, F_, F_, F_, P_, P_)(
            p(dev[0]), nh * 2 * d, p(dev[1]), p(dev[2]), T * width, p(dev[3]), width, p(dev[4]), p(dev[5]), p(acc), p(ml), p(out), T, nh, nkv, d, dv, page, 0, scale,
            splits, lam, eps, 1.0, p(err), stream())
    else:
        rc = entry("illm_attention_decode_ring_shared", I_, P_, I_, P_, P_, L_, P_, I_, P_, P_, P_, P_, P_, I_, I_, I_, I_, I_, I_, F_, I_, P_, I_, P_, P_, I_, I_, F_, I_,
                   P_)(p(dev[0]), nh * d, p(dev[1]), p(dev[2]), T * width, p(dev[3]), width, p(dev[4]), p(dev[5]), p(acc), p(ml), p(out), T, nh, nkv, d, page, 0, scale,
                       splits, p(err), 1, None, None, 0, 0, 0.0, 2, stream())
    assert rc == 0 and int(err) == 0
    got = out.cpu().double().numpy().reshape(T, nh, dv)
    for b in range(T):
        for h in range(nh):
            k, v = ks[b][:, h // (nh // nkv)].double().numpy().reshape(-1, maps, d), vs[b][:, h // (nh // nkv)].double().numpy()
            a = [(weights_of(q[b, h, m:m + 1].double().numpy(), k[:, m], scale, 0) @ v)[0] for m in range(maps)]
            ref = a[0]
            if maps == 2:
                o = a[0] - lam * a[1]
                ref = o / np.sqrt((o * o).mean() + eps)
            assert (np.abs(got[b, h] - ref) <= 2.0 ** -8 * np.abs(ref) + 2.0 ** -12).all(), (b, h)


@pytest.mark.parametrize("nh,nkv,alias,d", [(32, 1, 2, 128), (20, 1, 2, 64), (96, 2, 3, 64), (128, 1, 8, 128), (6, 2, 3, 128), (4, 4, 1, 64)])
@pytest.mark.parametrize("window,cap,sinks", [(0, 0.0, False), (70, 20.0, True)])
@pytest.mark.parametrize("splits", [1, 5])
def test_single_tokens_with_a_group_over_several_blocks(nh, nkv, alias, d, window, cap, sinks, splits):
    """Against float64, and beside the kernel on CUDA cores."""
    lens, page = [1, 64, 300], 64
    T, scale = len(lens), d ** -0.5
    g = torch.Generator().manual_seed(nh + window)
    (ks, vs), pools, table = paged(lens, nkv, (d, d), g)
    q, sink = torch.randn(T, nh * d, generator=g).bfloat16(), torch.randn(nh, generator=g)
    dev = [t.cuda() for t in (q, *pools, table, torch.tensor(lens, dtype=torch.int32) - 1, torch.arange(T, dtype=torch.int32), sink)]
    width, n_pages = table.shape[1], pools[0].shape[0]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    outs = [torch.full((T, nh * d), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    acc, ml = torch.empty(T * nh * splits * d, device="cuda"), torch.empty(T * nh * splits * 2, device="cuda")
    sp = p(dev[6]) if sinks else None
    rc = entry("illm_attention_decode_ring_shared", I_, P_, I_, P_, P_, L_, P_, I_, P_, P_, P_, P_, P_, I_, I_, I_, I_, I_, I_, F_, I_, P_, I_, P_, P_, I_, I_, F_, I_, P_)(
        p(dev[0]), nh * d, p(dev[1]), p(dev[2]), n_pages, p(dev[3]), width, p(dev[4]), p(dev[5]), p(acc), p(ml), p(outs[0]), T, nh, nkv, d, page, window, scale, splits,
        p(err), 1, sp, None, 0, 0, cap, alias, stream())
    assert rc == 0
    scratch = torch.empty(T * nh * 64 * (d + 2), device="cuda")
    rc = entry("illm_attention_one_decode", I_, P_, I_, P_, P_, P_, I_, P_, P_, P_, I_, I_, I_, I_, I_, I_, I_, F_, F_, P_, P_, I_, I_, L_, I_, P_, P_)(
        p(dev[0]), nh * d, p(dev[1]), p(dev[2]), p(dev[3]), width, p(dev[4]), p(dev[5]), p(outs[1]), T, nh, nkv, d, d, page, window, scale, cap, sp, None, 0, 0,
        max(lens), 2, p(scratch), stream())
    assert rc == 0 and int(err) == 0
    ref = np.zeros((T, nh, d))
    for b in range(T):
        qq, k, v = q[b].double().numpy().reshape(nh, d), ks[b].double().numpy(), vs[b].double().numpy()
        for hk in range(nkv):
            of = slice(hk * nh // nkv, (hk + 1) * nh // nkv)
            ref[b, of] = weights_of(qq[of], k[:, hk], scale, window, cap, sink.double().numpy()[of] if sinks else None) @ v[:, hk]
    mine, theirs = (np.abs(o.cpu().double().numpy().reshape(T, nh, d) - ref) for o in outs)
    assert (mine <= 2.0 ** -8 * np.abs(ref) + 2.0 ** -13).all()
    print("errors", np.linalg.norm(mine) / np.linalg.norm(ref), np.linalg.norm(theirs) / np.linalg.norm(ref))
    assert np.linalg.norm(mine) <= 1.01 * np.linalg.norm(theirs) + 1e-6


@pytest.mark.parametrize("nh,nkv,d", [(4, 4, 128), (6, 2, 64), (32, 2, 128)])
@pytest.mark.parametrize("splits", [1, 2, 32])
@pytest.mark.parametrize("window", [0, 40])
def test_ring_attention_loads_no_more_than_the_last_tiles_keys(nh, nkv, d, splits, window):
    """Contexts that end in each of a tile's four groups of 16 keys, against float64; every row that nothing wrote is NaN."""
    g = torch.Generator().manual_seed(d + splits)
    lens, page = [1, 15, 16, 17, 31, 33, 47, 48, 49, 63, 64, 65, 80, 97, 128, 129, 200, 2047], 64
    T, scale = len(lens), d ** -0.5
    (ks, vs), pools, table = paged(lens, nkv, (d, d), g)
    q = torch.randn(T, nh * d, generator=g).bfloat16()
    dev = [t.cuda() for t in (q, *pools, table, torch.tensor(lens, dtype=torch.int32) - 1, torch.arange(T, dtype=torch.int32))]
    err, out = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.empty(T, nh * d, dtype=torch.bfloat16, device="cuda")
    acc, ml = torch.full((T * nh * splits * d,), float("nan"), device="cuda"), torch.empty(T * nh * splits * 2, device="cuda")
    ring = entry("illm_attention_decode_ring", I_, P_, I_, P_, P_, L_, P_, I_, P_, P_, P_, P_, P_, I_, I_, I_, I_, I_, I_, F_, I_, P_, P_)
    assert ring(p(dev[0]), nh * d, p(dev[1]), p(dev[2]), pools[0].shape[0], p(dev[3]), table.shape[1], p(dev[4]), p(dev[5]), p(acc), p(ml), p(out), T, nh, nkv, d, page,
                window, scale, splits, p(err), stream()) == 0
    got = out.cpu().double().numpy().reshape(T, nh, d)
    assert int(err) == 0
    for b in range(T):
        qq = q[b].double().numpy().reshape(nh, d)
        for h in range(nh):
            k, v = ks[b][:, h // (nh // nkv)].double().numpy(), vs[b][:, h // (nh // nkv)].double().numpy()
            w = weights_of(qq[h:h + 1], k, scale, window)
            # every weight and the output rounded to bfloat16
            assert (np.abs(got[b, h] - (w @ v)[0]) <= 2.0 ** -8 * ((w @ np.abs(v))[0] + np.abs((w @ v)[0])) + 2.0 ** -20).all()
