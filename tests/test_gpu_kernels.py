"""Each kernel alone against the plain implementation's function for the same op, at sizes other
than the engine's tiny models: odd widths, head sizes in steps of 16, odd head and group counts."""
import math

import pytest
import torch

from tests.plain import llama_plain as plain

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DT = [torch.float32, torch.bfloat16]
IDS = ["f32", "bf16"]
# elementwise results: float32 to rounding; bfloat16 outputs are rounded once to 8 bits (2^-9 relative)
ETOL = {torch.float32: 2e-6, torch.bfloat16: 2 ** -8}


def rel(a, b):
    return float((a.double().cpu() - b.double().cpu()).abs().max() / b.double().abs().max().clamp_min(1e-30))


def K():
    from vllm_oxide_b200 import kernels
    return kernels


def test_embed():
    g = torch.Generator().manual_seed(0)
    for dt in DT:
        table = torch.randn(301, 72, generator=g).to(dt).to(DEV)
        toks = torch.tensor([0, 300, 17, 17, 5], dtype=torch.int32, device=DEV)
        out = torch.empty(5, 72, dtype=torch.float32, device=DEV)
        flag = torch.zeros(1, dtype=torch.int32, device=DEV)
        K().embed(table, toks, out, flag)
        want = plain.embedding(table.double().cpu(), toks.tolist())
        assert torch.equal(out.double().cpu(), want) and int(flag) == 0
        bad = torch.tensor([1, 301, 2, 3, 4], dtype=torch.int32, device=DEV)
        K().embed(table, bad, out, flag)
        assert int(flag) == 1 and float(out[1].abs().max()) == 0.0      # out of range: zeros and a raised flag


@pytest.mark.parametrize("dt", DT, ids=IDS)
@pytest.mark.parametrize("h", [19, 100, 2048, 4100])
def test_add_rmsnorm(dt, h):
    g = torch.Generator().manual_seed(h)
    T = 7
    resid = torch.randn(T, h, generator=g).to(DEV)
    delta = (torch.randn(T, h, generator=g) * 0.5).to(dt).to(DEV)
    w = (1 + 0.3 * torch.randn(h, generator=g)).to(DEV)
    eps = 3e-5
    r0 = resid.clone()
    out = torch.empty(T, h, dtype=dt, device=DEV)
    K().add_rmsnorm(resid, delta, w, eps, out)
    x = r0.double().cpu() + delta.double().cpu()
    assert rel(resid, x) <= 2e-7                                       # the residual sum stays float32
    assert rel(out, plain.rms_norm(x, w.double().cpu(), eps)) <= ETOL[dt]
    # without delta, and with a row list: the residual is left alone
    r1 = resid.clone()
    rows = torch.tensor([6, 0, 3], dtype=torch.int32, device=DEV)
    out2 = torch.empty(3, h, dtype=dt, device=DEV)
    K().add_rmsnorm(resid, delta, w, eps, out2, rows)
    assert torch.equal(resid, r1)
    x2 = (r1.double().cpu() + delta.double().cpu())[[6, 0, 3]]
    assert rel(out2, plain.rms_norm(x2, w.double().cpu(), eps)) <= ETOL[dt]
    out3 = torch.empty(T, h, dtype=dt, device=DEV)
    K().add_rmsnorm(resid, None, w, eps, out3)
    assert rel(out3, plain.rms_norm(r1.double().cpu(), w.double().cpu(), eps)) <= ETOL[dt]


def test_rmsnorm_refuses_too_wide_rows():
    from vllm_oxide_b200.errors import ShapeError
    with pytest.raises(ShapeError, match="limit"):
        K().add_rmsnorm(torch.zeros(1, 20000, device=DEV), None, torch.ones(20000, device=DEV), 1e-5,
                        torch.zeros(1, 20000, device=DEV))


@pytest.mark.parametrize("dt", DT, ids=IDS)
@pytest.mark.parametrize("I", [5, 224, 1000])
def test_swiglu(dt, I):
    g = torch.Generator().manual_seed(I)
    gu = (torch.randn(6, 2 * I, generator=g) * 3).to(dt).to(DEV)
    out = torch.empty(6, I, dtype=dt, device=DEV)
    K().swiglu(gu, out)
    want = plain.swiglu(gu[:, :I].double().cpu(), gu[:, I:].double().cpu())
    assert rel(out, want) <= ETOL[dt]


@pytest.mark.parametrize("M,N,K_", [(1, 1, 1), (7, 37, 21), (64, 64, 16), (65, 130, 257), (3, 1000, 96), (200, 50, 2048)])
def test_gemm_f32(M, N, K_):
    # odd sizes against the 64x64x16 tiling (the reference tests 7x21 -> 37: crates/engine/src/backend/cpu/tests.rs:37-59)
    g = torch.Generator().manual_seed(M * 1000 + N)
    a = torch.randn(M, K_, generator=g).to(DEV)
    w = torch.randn(N, K_, generator=g).to(DEV)
    out = torch.empty(M, N, device=DEV)
    K().gemm_f32(a, w, out)
    # one chain of K float32 FMAs per element: rounding errors of 2^-24 each add up like a random
    # walk, sqrt(K) * 2^-24 of the running sum; twice that as the bound (1e-6 at the reference's K = 21)
    tol = max(1e-6, 2.0 ** -23 * math.sqrt(K_))
    assert rel(out, plain.linear(a.double().cpu(), w.double().cpu())) <= tol
    # a row's value does not depend on the rows around it: bitwise
    out1 = torch.empty(1, N, device=DEV)
    K().gemm_f32(a[M - 1:M], w, out1)
    assert torch.equal(out1[0], out[M - 1])
    # strided views (a column slice of a wider buffer)
    wide = torch.randn(M, K_ + 8, generator=g).to(DEV)
    outw = torch.zeros(M, N + 4, device=DEV)
    K().gemm_f32(wide[:, 4:4 + K_], w, outw[:, 2:2 + N])
    assert rel(outw[:, 2:2 + N], plain.linear(wide[:, 4:4 + K_].double().cpu(), w.double().cpu())) <= tol
    assert float(outw[:, :2].abs().max()) == 0.0 and float(outw[:, 2 + N:].abs().max()) == 0.0


@pytest.mark.parametrize("N,K_", [(1, 4), (63, 128), (65, 132), (200, 1020), (64, 1024), (130, 2052), (2048, 2048), (72, 8192), (66, 14336), (70, 131)])
def test_gemm_f32_kernels_agree_to_the_bit(N, K_):
    """One order of summation everywhere: rows of a batch on the kernel of few rows (every size it is built for, and a K cut
    over one to eight blocks) and on tiles of 32, 64 and 128 rows (a block or eight to a tile) give the same bits."""
    g = torch.Generator().manual_seed(N + K_)
    a, w, bias = torch.randn(300, K_, generator=g).to(DEV), torch.randn(N, K_, generator=g).to(DEV), torch.randn(N, generator=g).to(DEV)
    full = torch.full((301, N), 7.0, device=DEV)
    K().gemm_f32(a, w, full[:300], bias)
    want = a.double() @ w.double().T + bias.double()
    # chains of 64, their sum, a segment's chunks, eight segments, the bias: one rounding of 2^-24 each, of at most the sum of magnitudes
    roundings = 64 + 1 + -(-(-(-K_ // 128)) // 8) + 8 + 1
    bound = roundings * 2.0 ** -24 * 1.01 * (a.double().abs() @ w.double().abs().T + bias.double().abs())
    assert bool(((full[:300].double() - want).abs() <= bound).all()) and bool((full[300] == 7.0).all())
    for M in (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 100, 129, 257):
        for lo in (0, 300 - M):
            out = torch.full((M + 1, N), 7.0, device=DEV)
            K().gemm_f32(a[lo:lo + M], w, out[:M], bias)
            assert torch.equal(out[:M], full[lo:lo + M]) and bool((out[M] == 7.0).all()), (M, lo)


@pytest.mark.parametrize("dt", DT, ids=IDS)
def test_a_matrix_written_by_the_kernel_in_front(dt):
    """`w` of a product may be what the kernel in front writes, with a bias and without: nothing of it is read before that kernel is
    done unless the caller says that no kernel writes it. (bfloat16 without a bias always takes `w` for weights.)"""
    g = torch.Generator().manual_seed(5)
    N, Kd, inner = 512 if dt == torch.float32 else 32, 1024, 2048         # (few rows of `w`: written by this package's kernel)
    x = torch.randn(16, Kd, generator=g).to(dt).to(DEV)
    w_t = torch.randn(Kd, inner, generator=g).to(dt).to(DEV)
    bias = torch.randn(N, generator=g).to(dt).to(DEV)
    k = K()
    makers = [torch.randn(N, inner, generator=g).to(dt).to(DEV) for _ in range(12)]
    w = torch.zeros(N, Kd, dtype=dt, device=DEV)
    for M in (1, 3, 16):
        outs = [torch.empty(M, N, dtype=dt, device=DEV) for _ in makers]
        torch.cuda.synchronize()
        for a, out in zip(makers, outs):
            k.linear(a, w_t, w)                    # w = a @ w_t^T
            k.linear(x[:M], w, out, bias)
        for a, out in zip(makers, outs):
            k.linear(a, w_t, w)
            torch.cuda.synchronize()
            again = torch.empty_like(out)
            k.linear(x[:M], w, again, bias)
            assert torch.equal(out, again), M
            if dt == torch.float32:                # read early or not: the same bits
                k.linear(x[:M], w, again, bias, fixed_w=True)
                assert torch.equal(out, again), M


def test_gemm_f32_shape_errors():
    from vllm_oxide_b200.errors import ShapeError
    with pytest.raises(ShapeError):
        K().gemm_f32(torch.zeros(2, 3, device=DEV), torch.zeros(4, 5, device=DEV), torch.zeros(2, 4, device=DEV))
    with pytest.raises(ShapeError):
        K().gemm_f32(torch.zeros(2, 3, device=DEV), torch.zeros(4, 3, device=DEV), torch.zeros(2, 5, device=DEV))


def test_linear_bf16_library_product():
    g = torch.Generator().manual_seed(3)
    a = torch.randn(9, 200, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(77, 200, generator=g).to(torch.bfloat16).to(DEV)
    want = plain.linear(a.double().cpu(), w.double().cpu())
    o32 = torch.empty(9, 77, dtype=torch.float32, device=DEV)
    K().linear(a, w, o32)
    assert rel(o32, want) <= 1e-5                                      # bf16 inputs are exact; float32 accumulation
    o16 = torch.empty(9, 77, dtype=torch.bfloat16, device=DEV)
    K().linear(a, w, o16)
    assert rel(o16, want) <= 2 ** -8


def _paged_case(dt, H, KV, hd, page, seqs, seed, scale_key=None, poison=False):
    """seqs: list of (context_len, num_new). Returns tensors for the kernel and per-sequence q/k/v."""
    g = torch.Generator().manual_seed(seed)
    total_pages = sum(-(-(c + n) // page) for c, n in seqs) + 3
    perm = torch.randperm(total_pages, generator=g).tolist()          # shuffled, non-identity tables
    kc = torch.randn(total_pages, KV, page, hd, generator=g).to(dt)   # stale values everywhere
    vc = torch.randn(total_pages, KV, page, hd, generator=g).to(dt)
    if poison:                                                        # what no request wrote is NaN: it must reach no result
        kc.fill_(float("nan"))
        vc.fill_(float("nan"))
    max_pages = max(-(-(c + n) // page) for c, n in seqs) + 1
    bt = torch.full((len(seqs), max_pages), -1, dtype=torch.int32)
    qs, ks, vs, row_seq, positions = [], [], [], [], []
    for s, (c, n) in enumerate(seqs):
        L = c + n
        k = torch.randn(L, KV * hd, generator=g).to(dt)
        v = torch.randn(L, KV * hd, generator=g).to(dt)
        q = torch.randn(L, H * hd, generator=g).to(dt)
        if scale_key is not None:
            j = scale_key(L)
            k[j] *= 6.0                       # one key stands out: a wrong or missing key shows
        np_ = -(-L // page)
        for i in range(np_):
            bt[s, i] = perm.pop()
        for p in range(L):
            pg, off = int(bt[s, p // page]), p % page
            kc[pg, :, off, :] = k[p].view(KV, hd)
            vc[pg, :, off, :] = v[p].view(KV, hd)
        qs.append(q), ks.append(k), vs.append(v)
        row_seq += [s] * n
        positions += list(range(c, L))
    qrows = torch.cat([q[c:] for q, (c, n) in zip(qs, seqs)])
    return (qrows, kc, vc, bt, torch.tensor(row_seq, dtype=torch.int32), torch.tensor(positions, dtype=torch.int32),
            qs, ks, vs)


def _last_row(q, k, v, H, KV, hd, window=0):
    """Attention of a request's last row in float64: q [H * hd], k and v [L, KV * hd]."""
    L = len(k)
    k, v = (x.double().view(L, KV, 1, hd)[-(window or L):].expand(-1, -1, H // KV, -1).reshape(-1, H, hd) for x in (k, v))
    p = torch.softmax(torch.einsum("hd,lhd->hl", q.double().view(H, hd), k) / math.sqrt(hd), -1)
    return torch.einsum("hl,lhd->hd", p, v).reshape(1, H * hd)


ATOL = {torch.float32: 1e-5, torch.bfloat16: 2 ** -7}      # reference: 1e-5 relative for paged attention (cpu/tests.rs:161-334)


@pytest.mark.parametrize("dt", DT, ids=IDS)
@pytest.mark.parametrize("H,KV,hd,page", [(6, 2, 16, 4), (3, 1, 32, 8), (5, 5, 48, 16), (8, 2, 64, 16), (4, 2, 128, 16),
                                          (2, 1, 256, 32), (7, 7, 80, 8)])
def test_paged_attention_prefill_and_decode_shapes(dt, H, KV, hd, page):
    # (context, new): mid-page, zero context, page edge, a decode row, a long one
    seqs = [(5, 6), (0, 3), (2 * page, page), (37, 1), (0, 1), (3 * page - 1, 2)]
    qrows, kc, vc, bt, row_seq, pos, qs, ks, vs = _paged_case(dt, H, KV, hd, page, seqs, seed=hd + H)
    out = torch.empty_like(qrows).to(DEV)
    K().paged_attention(qrows.to(DEV), out, kc.to(DEV), vc.to(DEV), bt.to(DEV), row_seq.to(DEV), pos.to(DEV),
                        H, KV, hd, 1.0 / math.sqrt(hd))
    r = 0
    for s, (c, n) in enumerate(seqs):
        want = plain.causal_attention(qs[s].double(), ks[s].double(), vs[s].double(), H, KV, hd)[c:]
        got = out[r:r + n]
        assert rel(got, want) <= ATOL[dt], (s, c, n)
        r += n


@pytest.mark.parametrize("dt", DT, ids=IDS)
def test_paged_attention_far_key_among_hundreds(dt):
    """One key far back dominates the softmax; it must be found at any distance, across pages."""
    H, KV, hd, page = 4, 2, 64, 16
    seqs = [(700, 1), (0, 333), (511, 2)]
    qrows, kc, vc, bt, row_seq, pos, qs, ks, vs = _paged_case(dt, H, KV, hd, page, seqs, seed=1, scale_key=lambda L: 3)
    out = torch.empty_like(qrows).to(DEV)
    K().paged_attention(qrows.to(DEV), out, kc.to(DEV), vc.to(DEV), bt.to(DEV), row_seq.to(DEV), pos.to(DEV),
                        H, KV, hd, 1.0 / math.sqrt(hd))
    r = 0
    for s, (c, n) in enumerate(seqs):
        want = plain.causal_attention(qs[s].double(), ks[s].double(), vs[s].double(), H, KV, hd)[c:]
        assert rel(out[r:r + n], want) <= ATOL[dt]
        r += n


@pytest.mark.parametrize("dt", DT, ids=IDS)
@pytest.mark.parametrize("window", [1, 5, 16, 17, 40])
def test_paged_attention_window_edge(dt, window):
    H, KV, hd, page = 4, 2, 32, 8
    seqs = [(0, 50), (44, 3), (window, 1), (max(window - 1, 0), 1)]
    # the key just outside the window stands out: reading it would change everything
    qrows, kc, vc, bt, row_seq, pos, qs, ks, vs = _paged_case(dt, H, KV, hd, page, seqs, seed=window,
                                                             scale_key=lambda L: max(L - 1 - window, 0))
    out = torch.empty_like(qrows).to(DEV)
    K().paged_attention(qrows.to(DEV), out, kc.to(DEV), vc.to(DEV), bt.to(DEV), row_seq.to(DEV), pos.to(DEV),
                        H, KV, hd, 0.3, window)
    r = 0
    for s, (c, n) in enumerate(seqs):
        want = plain.causal_attention(qs[s].double(), ks[s].double(), vs[s].double(), H, KV, hd, window=window, scale=0.3)[c:]
        assert rel(out[r:r + n], want) <= ATOL[dt]
        r += n


@pytest.mark.parametrize("H,KV,hd,page,window", [(4, 4, 64, 16, 0), (8, 2, 64, 8, 33), (6, 2, 128, 16, 0), (16, 2, 128, 24, 40), (32, 8, 64, 16, 0),
                                                 (5, 1, 64, 16, 100), (2, 1, 128, 8, 0), (8, 1, 64, 16, 1)])
def test_f32_attention_of_portions_and_of_single_tokens_agree_to_the_bit(H, KV, hd, page, window):
    """The 32-bit engine's two kernels (single tokens over one to eight blocks, rows of portions) give a row the same bits, whatever
    shares its block; a padding row gives zeros; an infinity among a later token's values reaches no earlier row."""
    seqs = [(0, 70), (131, 1), (30, 5), (0, 1), (31, 2), (63, 66), (700, 1), (255, 200)]
    qrows, kc, vc, bt, row_seq, pos, qs, ks, vs = _paged_case(torch.float32, H, KV, hd, page, seqs, seed=H + hd + window, poison=True,
                                                             scale_key=lambda L: L // 2)
    # the last token of the first request: values that are infinite
    vc[int(bt[0, 69 // page]), :, 69 % page, :] = float("inf")
    pad = 3
    T = len(pos) + pad
    qrows, row_seq, pos = torch.cat([qrows, qrows[:pad]]).to(DEV), torch.cat([row_seq, row_seq[:pad]]).to(DEV), torch.cat([pos, pos[:pad] * 0 - 1]).to(DEV)
    kc, vc, bt = kc.to(DEV), vc.to(DEV), bt.to(DEV)

    def go(singles, rows=slice(0, T), portions=0):
        out = torch.full_like(qrows[rows], 7.0)
        K().paged_attention(qrows[rows], out, kc, vc, bt, row_seq[rows].contiguous(), pos[rows].contiguous(), H, KV, hd, 1.0 / math.sqrt(hd), window, singles,
                            portions)
        return out
    full = go(0, portions=-1)
    assert bool((full[-pad:] == 0).all())
    same = lambda a, b: torch.equal(torch.nan_to_num(a, 9e9), torch.nan_to_num(b, 9e9))  # noqa: E731
    for singles in (1, 2, 50, T - 1, T):
        assert same(go(singles), full) and same(go(singles, portions=-1), full), singles
    for portions in (0, 1, 8, 100):
        assert same(go(0, portions=portions), full), portions
    # several rows a block: row counts around its choices, with padding rows among them
    for n in (75, 149, 296, 297, 340, T):
        assert same(go(n, slice(T - n, T)), full[T - n:]), n
    for lo, n in ((0, 1), (3, 40), (69, 3), (13, 300), (T - 9, 9)):
        assert same(go(0, slice(lo, lo + n)), full[lo:lo + n]) and same(go(n, slice(lo, lo + n)), full[lo:lo + n]), (lo, n)
    r = 0
    for s, (c, n) in enumerate(seqs):
        want = plain.causal_attention(qs[s].double(), ks[s].double(), vs[s].double(), H, KV, hd, window=window or None)[c:]
        m = n - 1 if s == 0 else n
        assert rel(full[r:r + m], want[:m]) <= ATOL[torch.float32], s
        r += n


@pytest.mark.parametrize("hd,H,KV,window", [(64, 8, 2, 0), (128, 4, 4, 0), (64, 5, 1, 150)])
def test_f32_attention_keys_of_minus_infinite_score_weigh_nothing(hd, H, KV, window):
    """Keys whose score is minus infinity, for whole tiles of 32 and 64 at the front, in the middle and at the end of a row's keys:
    the row is what its other keys give, in both of the 32-bit engine's kernels."""
    # (context, rows): the infinite tiles lie at keys 0-31, 64-127 and 160-191 of each request
    seqs = [(150, 1), (32, 260), (191, 1), (0, 400), (223, 1)]
    qrows, kc, vc, bt, row_seq, pos, qs, ks, vs = _paged_case(torch.float32, H, KV, hd, 16, seqs, seed=hd + window)
    qrows[:, ::hd] = 1.0
    for s, (c, n) in enumerate(seqs):
        qs[s][:, ::hd] = 1.0
        for j in (*range(32), *range(64, 128), *range(160, 192)):
            if j < c + n:
                kc[int(bt[s, j // 16]), :, j % 16, 0] = float("-inf")
                ks[s][j].view(KV, hd)[:, 0] = float("-inf")
    T = len(pos)
    for singles in (0, T):
        out = torch.full((T, H * hd), 7.0, device=DEV)
        K().paged_attention(qrows.to(DEV), out, kc.to(DEV), vc.to(DEV), bt.to(DEV), row_seq.to(DEV), pos.to(DEV), H, KV, hd, 1.0 / math.sqrt(hd), window, singles,
                            -1)
        r = 0
        for s, (c, n) in enumerate(seqs):
            # (rows 0-31 have no other key: not asked)
            want = plain.causal_attention(qs[s].double(), ks[s].double(), vs[s].double(), H, KV, hd, window=window or None)[max(c, 32):]
            assert rel(out[r + max(c, 32) - c:r + n], want) <= ATOL[torch.float32], (s, singles)
            r += n


def test_paged_attention_refuses_bad_sizes():
    from vllm_oxide_b200.errors import ShapeError
    q = torch.zeros(1, 4 * 20, device=DEV)
    kc = torch.zeros(2, 2, 8, 20, device=DEV)
    z = torch.zeros(1, dtype=torch.int32, device=DEV)
    with pytest.raises(ShapeError, match="head_dim 20"):
        K().paged_attention(q, q.clone(), kc, kc, torch.zeros(1, 2, dtype=torch.int32, device=DEV), z, z, 4, 2, 20, 1.0)
    q = torch.zeros(1, 3 * 16, device=DEV)
    kc = torch.zeros(2, 2, 8, 16, device=DEV)
    with pytest.raises(ShapeError, match="multiple"):
        K().paged_attention(q, q.clone(), kc, kc, torch.zeros(1, 2, dtype=torch.int32, device=DEV), z, z, 3, 2, 16, 1.0)


@pytest.mark.parametrize("dt", DT, ids=IDS)
@pytest.mark.parametrize("T,pad", [(11, 0), (70, 0), (70, 1)])      # few tokens; many (16-byte accesses); many, rows not 16-byte aligned
@pytest.mark.parametrize("H,KV,hd,page", [(6, 2, 16, 4), (3, 1, 32, 8), (5, 5, 48, 16), (32, 8, 64, 16), (2, 1, 256, 16)])
def test_rope_kv_write(dt, H, KV, hd, page, T, pad):
    g = torch.Generator().manual_seed(hd)
    cfg = {"head_dim": hd, "hidden_size": H * hd, "num_attention_heads": H, "rope_theta": 500000.0,
           "rope_scaling": {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                            "original_max_position_embeddings": 64}}
    inv = plain.rope_inv_freq(cfg)
    qkv = torch.randn(T, (H + 2 * KV) * hd, generator=g).to(dt)
    positions = ([0, 1, 2, 63, 64, 65, 1000, 4095, 7, 7, 300] + list(range(100, 100 + T)))[:T]
    pages = -(-T // page) + 9
    slots = torch.randperm(pages * page, generator=g)[:T].to(torch.int32)
    slots[4] = -1                                                       # this token writes nothing
    kc = torch.full((pages, KV, page, hd), 7.0).to(dt)
    vc = torch.full((pages, KV, page, hd), 7.0).to(dt)
    d_kc, d_vc = kc.to(DEV), vc.to(DEV)
    d_qkv = torch.zeros(T, qkv.shape[1] + pad, dtype=dt, device=DEV)[:, :qkv.shape[1]]
    d_qkv.copy_(qkv)
    q, k, v = d_qkv[:, :H * hd], d_qkv[:, H * hd:(H + KV) * hd], d_qkv[:, (H + KV) * hd:]
    K().rope_kv_write(q, k, v, torch.tensor(positions, dtype=torch.int32, device=DEV), slots.to(DEV), inv.to(DEV),
                      d_kc, d_vc, H, KV, hd)
    wq = plain.rope(qkv[:, :H * hd].double(), positions, inv, hd)
    wk = plain.rope(qkv[:, H * hd:(H + KV) * hd].double(), positions, inv, hd)
    tol = 3e-6 if dt == torch.float32 else 2 ** -8
    assert rel(q, wq) <= tol and rel(k, wk) <= tol
    for t in range(T):
        s = int(slots[t])
        if s < 0:
            continue
        pg, off = s // page, s % page
        assert rel(d_kc[pg, :, off, :].reshape(-1), wk[t]) <= tol
        assert torch.equal(d_vc[pg, :, off, :].reshape(-1).cpu(), qkv[t, (H + KV) * hd:])
    written = {int(s) for s in slots if s >= 0}
    for s in range(pages * page):
        if s not in written:
            assert float((d_kc[s // page, :, s % page, :].float() - 7.0).abs().max()) == 0.0     # nothing else is touched


def test_pick_tokens_greedy_cases():
    # crates/engine/src/backend/cpu/tests.rs:129-144: ties -> first, all equal -> 0, NaN -> error
    V = 10007
    logits = torch.full((5, V), -1.0, device=DEV)
    logits[0, 5000] = 5.0
    logits[0, 9000] = 5.0
    logits[1] = 0.0
    logits[2, V - 1] = 3.0
    logits[3, 0] = 2.0
    logits[4, 77] = float("nan")
    k = K()
    sp = k.pick_splits(V)
    out = torch.zeros(5, dtype=torch.int32, device=DEV)
    flags = torch.zeros(5, dtype=torch.int32, device=DEV)
    k.pick_tokens(logits, out, flags, torch.empty(5 * sp, device=DEV), torch.empty(5 * sp, dtype=torch.int32, device=DEV))
    assert out.tolist() == [5000, 0, V - 1, 0, -1]
    assert flags.tolist() == [0, 0, 0, 0, 0]          # the flag is cleared once it has been turned into -1
    want = [plain.argmax_first(r) for r in logits[:4].double().cpu()]
    assert out.tolist()[:4] == want


def test_pick_writes_its_tokens_to_further_places():
    """`also`: the pick kernel writes the same tokens to up to two more places, a device tensor and a
    page-locked host buffer that the device addresses directly (no copy behind the kernel); both the
    two-pass pick and the final pass alone; what lies around the rows stays as it was."""
    from vllm_oxide_b200.errors import ShapeError
    V = 10007
    logits = torch.full((5, V), -1.0, device=DEV)
    for r, i in enumerate([5000, 3, V - 1, 0, 77]):
        logits[r, i] = 2.0 + r
    logits[4, 78] = float("nan")
    k = K()
    sp = k.pick_splits(V)
    host = k.HostInts((2, 8))
    host.tensor.fill_(-7)
    dev2 = torch.full((9,), -7, dtype=torch.int32, device=DEV)
    out = torch.zeros(5, dtype=torch.int32, device=DEV)
    flags = torch.zeros(5, dtype=torch.int32, device=DEV)
    val, idx = torch.empty(5 * sp, device=DEV), torch.empty(5 * sp, dtype=torch.int32, device=DEV)
    k.pick_tokens(logits, out, flags, val, idx, also=[dev2[2:7], host.at(8 + 1)])
    torch.cuda.synchronize()
    want = [5000, 3, V - 1, 0, -1]
    assert out.tolist() == want and dev2.tolist() == [-7, -7] + want + [-7, -7]
    assert host.tensor.tolist() == [[-7] * 8, [-7] + want + [-7, -7]]
    # the final pass alone, pairs given: one destination only
    part_val = torch.tensor([[1.0, 5.0, 5.0], [0.0, -1.0, 7.0]], device=DEV)
    part_idx = torch.tensor([[9, 4, 6], [1, 2, 3]], dtype=torch.int32, device=DEV)
    out2 = torch.zeros(2, dtype=torch.int32, device=DEV)
    k.pick_final(part_val, part_idx, 2, 100, torch.zeros(2, dtype=torch.int32, device=DEV), out2, also=[host.at(0)])
    torch.cuda.synchronize()
    assert out2.tolist() == [4, 3] and host.tensor[0].tolist() == [4, 3] + [-7] * 6
    with pytest.raises(ShapeError, match="room for"):
        k.pick_final(part_val, part_idx, 2, 100, flags, out2, also=[host.at(15)])
    with pytest.raises(ShapeError, match="at most two"):
        k.pick_final(part_val, part_idx, 2, 100, flags, out2, also=[out2, out2, out2])
    with pytest.raises(ShapeError):
        k.pick_tokens(logits, out, flags, val, idx, also=[dev2[:3]])


def test_pick_tokens_temperature_matches_plain_and_law():
    V = 997
    g = torch.Generator().manual_seed(5)
    logits = (torch.randn(6, V, generator=g) * 2).to(DEV)
    temps = torch.tensor([0.7, 0.0, 1.3, 0.7, 0.7, 0.2], device=DEV)
    seeds = torch.tensor([[1, 0], [2, 0], [3, 7], [1, 0], [9, 1], [4, 4]], dtype=torch.int32, device=DEV)
    steps = torch.tensor([0, 5, 2, 1, 0, 3], dtype=torch.int32, device=DEV)
    k = K()
    sp = k.pick_splits(V)
    out = torch.zeros(6, dtype=torch.int32, device=DEV)
    k.pick_tokens(logits, out, torch.zeros(6, dtype=torch.int32, device=DEV), torch.empty(6 * sp, device=DEV),
                  torch.empty(6 * sp, dtype=torch.int32, device=DEV), temps, seeds, steps)
    for r in range(6):
        seed = (int(seeds[r, 1]) << 32) | int(seeds[r, 0])
        assert int(out[r]) == plain.temperature_pick(logits[r].double().cpu(), float(temps[r]), seed, int(steps[r]))
    # the law: many steps of one request over small logits follow softmax(logits / t)
    small = torch.tensor([[2.0, 1.0, 0.0, -1.0, -30.0]], device=DEV).repeat(64, 1)
    n, counts = 0, torch.zeros(5)
    for it in range(40):
        st = torch.arange(it * 64, it * 64 + 64, dtype=torch.int32, device=DEV)
        o = torch.zeros(64, dtype=torch.int32, device=DEV)
        k.pick_tokens(small, o, torch.zeros(64, dtype=torch.int32, device=DEV), torch.empty(64, device=DEV),
                      torch.empty(64, dtype=torch.int32, device=DEV), torch.full((64,), 0.7, device=DEV),
                      torch.tensor([[11, 3]] * 64, dtype=torch.int32, device=DEV), st)
        counts += torch.bincount(o.cpu(), minlength=5).float()
        n += 64
    p = torch.softmax(small[0].cpu().double() / 0.7, 0)
    for i in range(5):
        assert abs(float(counts[i]) / n - float(p[i])) < 4 * math.sqrt(float(p[i]) * (1 - float(p[i])) / n) + 2e-3


def test_cpu_tensors_are_refused():
    from vllm_oxide_b200.errors import KernelError
    with pytest.raises(KernelError, match="no CPU path"):
        K().gemm_f32(torch.zeros(2, 2), torch.zeros(2, 2), torch.zeros(2, 2))


# ----------------------------------------------------------------------------- tensor-core attention (bfloat16)
def _starts_ctx(seqs):
    starts, ctxs, r = [0], [], 0
    for c, n in seqs:
        r += n
        starts.append(r)
        ctxs.append(c)
    return torch.tensor(starts, dtype=torch.int32, device=DEV), torch.tensor(ctxs, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("H,KV,hd,page", [(8, 2, 64, 16), (3, 1, 64, 8), (4, 4, 128, 32), (6, 2, 128, 16), (32, 8, 64, 64)])
def test_attn_prefill_mma(H, KV, hd, page, window):
    dt = torch.bfloat16
    # portions that start mid-page, at a page edge, at zero; single tokens beside them; > one row tile
    seqs = [(5, 6), (0, 3), (2 * page, page), (137, 1), (0, 1), (3 * page - 1, 2), (0, 150), (201, 77)]
    sk = (lambda L: max(L - 1 - window, 0)) if window else (lambda L: min(3, L - 1))
    qrows, kc, vc, bt, row_seq, pos, qs, ks, vs = _paged_case(dt, H, KV, hd, page, seqs, seed=hd + H + page, scale_key=sk)
    starts, ctxs = _starts_ctx(seqs)
    out = torch.empty_like(qrows).to(DEV)
    K().attn_prefill_mma(qrows.to(DEV), out, kc.to(DEV), vc.to(DEV), bt.to(DEV), starts, ctxs, len(seqs),
                         max(n for _, n in seqs), H, KV, hd, 1.0 / math.sqrt(hd), window)
    r = 0
    for s, (c, n) in enumerate(seqs):
        want = plain.causal_attention(qs[s].double(), ks[s].double(), vs[s].double(), H, KV, hd, window=window or None)[c:]
        assert rel(out[r:r + n], want) <= 2 ** -6, (s, c, n)     # P is rounded to bfloat16 before P V: one more 2^-9 rounding per key
        r += n


@pytest.mark.parametrize("H,KV,hd,page", [(8, 2, 64, 16), (3, 3, 64, 8), (16, 2, 64, 32), (32, 8, 64, 64), (2, 1, 64, 128),
                                          (6, 2, 64, 16), (5, 1, 64, 8), (4, 2, 128, 16), (24, 8, 128, 32), (8, 8, 128, 128), (7, 1, 128, 8)])
def test_attn_prefill_sm100(H, KV, hd, page):
    """The tcgen05 kernel for prompt portions: portions that start mid-page, at a page edge, at
    zero; single tokens beside them; more than one row tile and more than one key tile; one key far
    back scaled so that a wrong or missing key shows. Cache slots no request wrote hold NaN."""
    dt = torch.bfloat16
    seqs = [(5, 6), (0, 3), (2 * page, page), (137, 1), (0, 1), (3 * page - 1, 2), (0, 150), (201, 77), (0, 300), (250, 130)]
    qrows, kc, vc, bt, row_seq, pos, qs, ks, vs = _paged_case(dt, H, KV, hd, page, seqs, seed=hd + H + page,
                                                              scale_key=lambda L: min(3, L - 1), poison=True)
    starts, ctxs = _starts_ctx(seqs)
    out = torch.full_like(qrows, 7.0).to(DEV)
    k = K()
    assert k.attn_prefill_sm100_supported(H, KV, hd, page, bt.shape[1])
    args = (qrows.to(DEV), out, kc.to(DEV), vc.to(DEV), bt.to(DEV), starts, ctxs, len(seqs), max(n for _, n in seqs),
            H, KV, hd, 1.0 / math.sqrt(hd))
    k.attn_prefill_sm100(*args)
    torch.cuda.synchronize()
    k.gemm_sm100_check()
    r = 0
    for s, (c, n) in enumerate(seqs):
        want = plain.causal_attention(qs[s].double(), ks[s].double(), vs[s].double(), H, KV, hd)[c:]
        assert rel(out[r:r + n], want) <= 2 ** -6, (s, c, n)     # P is rounded to bfloat16 before P V
        r += n
    first = out.clone()
    out.fill_(3.0)
    k.attn_prefill_sm100(*args)                                   # nothing needs resetting between launches
    assert torch.equal(out, first)


def test_attn_prefill_sm100_far_key_and_refusals():
    from vllm_oxide_b200.errors import ShapeError
    k = K()
    H, KV, hd, page = 4, 1, 64, 16
    seqs = [(0, 1000), (900, 100)]
    qrows, kc, vc, bt, row_seq, pos, qs, ks, vs = _paged_case(torch.bfloat16, H, KV, hd, page, seqs, seed=5,
                                                              scale_key=lambda L: 3, poison=True)
    starts, ctxs = _starts_ctx(seqs)
    out = torch.empty_like(qrows).to(DEV)
    k.attn_prefill_sm100(qrows.to(DEV), out, kc.to(DEV), vc.to(DEV), bt.to(DEV), starts, ctxs, 2, 1000, H, KV, hd, 0.125)
    r = 0
    for s, (c, n) in enumerate(seqs):
        want = plain.causal_attention(qs[s].double(), ks[s].double(), vs[s].double(), H, KV, hd)[c:]
        assert rel(out[r:r + n], want) <= 2 ** -6, (s, c, n)
        r += n
    k.gemm_sm100_check()
    assert k.attn_prefill_sm100_supported(6, 2, 64, 16, 64) and k.attn_prefill_sm100_supported(4, 2, 128, 16, 64)
    assert not k.attn_prefill_sm100_supported(4, 2, 48, 16, 64) and not k.attn_prefill_sm100_supported(4, 2, 64, 24, 64)
    assert not k.attn_prefill_sm100_supported(4, 2, 64, 4, 64) and not k.attn_prefill_sm100_supported(258, 2, 64, 16, 64)
    assert not k.attn_prefill_sm100_supported(4, 2, 64, 16, 1 << 20)  # the page list would not fit shared memory
    q = torch.zeros(1, 4 * 48, dtype=torch.bfloat16, device=DEV)
    kc6 = torch.zeros(2, 2, 16, 48, dtype=torch.bfloat16, device=DEV)
    z = torch.zeros(2, dtype=torch.int32, device=DEV)
    with pytest.raises(ShapeError, match="not supported"):
        k.attn_prefill_sm100(q, q.clone(), kc6, kc6, torch.zeros(1, 2, dtype=torch.int32, device=DEV), z, z, 1, 1, 4, 2, 48, 1.0)


@pytest.mark.parametrize("splits", [1, 3, 8])
@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("H,KV,hd,page", [(8, 2, 64, 16), (3, 1, 64, 8), (4, 4, 128, 32), (32, 2, 128, 16)])
def test_attn_decode_mma(H, KV, hd, page, window, splits):
    dt = torch.bfloat16
    seqs = [(700, 1), (0, 1), (63, 1), (64, 1), (65, 1), (333, 1), (5, 1)]
    sk = (lambda L: max(L - 1 - window, 0)) if window else (lambda L: min(3, L - 1))
    qrows, kc, vc, bt, row_seq, pos, qs, ks, vs = _paged_case(dt, H, KV, hd, page, seqs, seed=hd + H + page + splits, scale_key=sk)
    # a padding row: position -1, attends to nothing, must come out as zeros
    qrows = torch.cat([qrows, torch.randn(1, H * hd).to(dt)])
    pos = torch.cat([pos, torch.tensor([-1], dtype=torch.int32)])
    bt = torch.cat([bt, bt[:1]])
    out = torch.full_like(qrows, 7.0).to(DEV)
    k = K()
    k.attn_decode_mma(qrows.to(DEV), out, kc.to(DEV), vc.to(DEV), bt.to(DEV), pos.to(DEV), H, KV, hd,
                      1.0 / math.sqrt(hd), window, splits)
    for s, (c, n) in enumerate(seqs):
        want = plain.causal_attention(qs[s].double(), ks[s].double(), vs[s].double(), H, KV, hd, window=window or None)[c:]
        assert rel(out[s:s + 1], want) <= 2 ** -6, (s, c)
    assert float(out[len(seqs)].float().abs().max()) == 0.0


@pytest.mark.parametrize("H,KV,hd,page,window,splits", [(8, 2, 64, 16, 0, 37), (6, 2, 128, 32, 0, 64), (4, 4, 64, 8, 300, 19),
                                                        (8, 2, 64, 64, 0, 9)])
def test_attn_decode_mma_merge_through_global_memory(H, KV, hd, page, window, splits):
    """Up to 64 blocks per request without a cluster: long and short requests in one launch (a
    short one uses one block and the others leave), a far key that decides the result, a padding
    row; and a second launch on the same counters, which the first must have left at zero."""
    dt = torch.bfloat16
    seqs = [(5000, 1), (0, 1), (130, 1), (700, 1), (64 * splits * 2 - 1, 1)]
    sk = (lambda L: max(L - 1 - window, 0)) if window else (lambda L: min(3, L - 1))
    qrows, kc, vc, bt, row_seq, pos, qs, ks, vs = _paged_case(dt, H, KV, hd, page, seqs, seed=hd + H + page + splits, scale_key=sk)
    qrows = torch.cat([qrows, torch.randn(1, H * hd).to(dt)])
    pos = torch.cat([pos, torch.tensor([-1], dtype=torch.int32)])
    bt = torch.cat([bt, bt[:1]])
    k = K()
    S = qrows.shape[0]
    partials = torch.full((k.attn_decode_partial_floats(S, KV, hd, splits),), float("nan"), device=DEV)
    arrived = torch.zeros(S * KV, dtype=torch.int32, device=DEV)
    args = (kc.to(DEV), vc.to(DEV), bt.to(DEV), pos.to(DEV), H, KV, hd, 1.0 / math.sqrt(hd), window, splits, partials, arrived)
    for _ in range(2):
        out = torch.full_like(qrows, 7.0).to(DEV)
        k.attn_decode_mma(qrows.to(DEV), out, *args)
        for s, (c, n) in enumerate(seqs):
            want = plain.causal_attention(qs[s].double(), ks[s].double(), vs[s].double(), H, KV, hd, window=window or None)[c:]
            assert rel(out[s:s + 1], want) <= 2 ** -6, (s, c)
        assert float(out[len(seqs)].float().abs().max()) == 0.0
        assert int(arrived.abs().max()) == 0
    from vllm_oxide_b200.errors import ShapeError
    with pytest.raises(ShapeError, match="splits must be"):
        k.attn_decode_mma(qrows.to(DEV), out, *args[:9], 65, partials, arrived)
    with pytest.raises(ShapeError, match="splits must be"):
        k.attn_decode_mma(qrows.to(DEV), out, *args[:9], 9)
    with pytest.raises(ShapeError, match="partials must be"):
        k.attn_decode_mma(qrows.to(DEV), out, *args[:10], partials[:100], arrived)


@pytest.mark.parametrize("H,KV,hd,page,S,balance,most", [(8, 2, 64, 16, 1, 2, 400), (8, 2, 64, 16, 1, 64, 9000), (6, 2, 128, 32, 12, 37, 3000),
                                                         (32, 8, 64, 16, 33, 55, 1500), (4, 4, 64, 8, 70, 3, 300), (3, 1, 128, 64, 128, 64, 700),
                                                         (16, 1, 64, 16, 128, 5, 64), (8, 2, 64, 64, 20, 2, 5000)])
def test_attn_decode_mma_balanced(H, KV, hd, page, S, balance, most):
    """Blocks dealt out by length: one long request among short ones, all alike, single keys, padding rows in between, tile edges,
    as many requests as a launch takes and few blocks for them; what one block per request computes, up to rounding, and
    counters left at zero."""
    g = torch.Generator().manual_seed(S + most)
    k = K()
    pages = -(-most // page)
    spread = torch.exp(torch.rand(S, generator=g) * math.log(most)).long().clamp(1, most)
    one = torch.ones(S, dtype=torch.long)
    one[S // 2] = most
    edges = torch.tensor([[1, 63, 64, 65, 128, 0][i % 6] for i in range(S)]).clamp(max=most)
    bt = torch.arange(S * pages, dtype=torch.int32).view(S, pages)[:, torch.randperm(pages, generator=g)].contiguous().to(DEV)
    kc = torch.randn(S * pages, KV, page, hd, generator=g).to(torch.bfloat16).to(DEV)
    vc = torch.randn(S * pages, KV, page, hd, generator=g).to(torch.bfloat16).to(DEV)
    q = (2 * torch.randn(S, H * hd, generator=g)).to(torch.bfloat16).to(DEV)
    partials = torch.full((k.attn_decode_partial_floats(1, KV, hd, 2 * balance),), float("nan"), device=DEV)
    arrived = torch.zeros(S * KV, dtype=torch.int32, device=DEV)
    for lens in (spread, one, torch.full((S,), most), edges, one * 0):
        pos = (lens - 1).to(torch.int32).to(DEV)
        want, got = torch.full_like(q, 7.0), torch.full_like(q, 7.0)
        args = (kc, vc, bt, pos, H, KV, hd, 1.0 / math.sqrt(hd))
        k.attn_decode_mma(q, want, *args)
        k.attn_decode_mma(q, got, *args, 0, 1, partials, arrived, balance=balance)
        # P is rounded to bfloat16 relative to another maximum, and so is the result: two roundings of 2^-8 at most
        assert rel(got, want.double().cpu()) <= 2 ** -7 if int(lens.max()) else bool((got == 0).all())
        assert bool((got[pos < 0] == 0).all()) and int(arrived.abs().max()) == 0
    from vllm_oxide_b200.errors import ShapeError
    with pytest.raises(ShapeError, match="balance must be"):
        k.attn_decode_mma(q, got, *args, 0, 1, partials, arrived, balance=65)
    with pytest.raises(ShapeError, match="balance must be"):
        k.attn_decode_mma(q, got, *args, 0, 1, balance=balance)
    with pytest.raises(ShapeError, match="partials must be"):
        k.attn_decode_mma(q, got, *args, 0, 1, partials[:100], arrived, balance=balance)


@pytest.mark.parametrize("H,KV,hd,page,window,splits", [(8, 2, 64, 1, 0, 1), (8, 2, 64, 4, 0, 1), (6, 2, 128, 2, 0, 2), (4, 4, 64, 1, 1500, 1), (8, 2, 64, 16, 0, 1),
                                                        (4, 1, 128, 8, 0, 1)])
def test_attn_decode_mma_page_list_is_refilled(H, KV, hd, page, window, splits):
    """Beside a table whose pages no block could hold, its list of 1,024 is filled again, half by half, as the block walks on: requests
    of lengths around its halves, in clusters, with the merge through global memory and balanced. The bits are those of a table just
    wide enough."""
    half = 512 * page
    seqs = [(n - 1, 1) for n in (2 * half - 1, 2 * half + 1, 3 * half, 5 * half + 70, 64, 3 * half + 65)]
    dt = torch.bfloat16
    qrows, kc, vc, bt, row_seq, pos, qs, ks, vs = _paged_case(dt, H, KV, hd, page, seqs, seed=hd + page, scale_key=lambda L: max(L - 3 - page, 0))
    want = torch.cat([_last_row(qs[s][-1], ks[s], vs[s], H, KV, hd, window) for s in range(len(seqs))])
    k = K()
    wide = torch.full((len(seqs), 131072), -1, dtype=torch.int32)
    wide[:, :bt.shape[1]] = bt
    caches, tables = (kc.to(DEV), vc.to(DEV)), (bt.to(DEV), wide.to(DEV))
    arrived = torch.zeros(len(seqs) * KV, dtype=torch.int32, device=DEV)

    def go(*more, **kw):
        outs = []
        for table in tables:
            outs.append(torch.full_like(qrows, 7.0).to(DEV))
            k.attn_decode_mma(qrows.to(DEV), outs[-1], *caches, table, pos.to(DEV), H, KV, hd, 1.0 / math.sqrt(hd), *more, **kw)
            assert rel(outs[-1], want) <= 2 ** -6
        assert torch.equal(*outs)
    go(window, splits)
    go(window, 2, torch.empty(k.attn_decode_partial_floats(len(seqs), KV, hd, 2), device=DEV), arrived)
    if not window:
        go(0, 1, torch.empty(k.attn_decode_partial_floats(1, KV, hd, 4), device=DEV), arrived, balance=2)


@pytest.mark.parametrize("page,balance", [(16, 37), (1, 37), (16, 0)])
def test_attn_decode_mma_takes_block_tables_of_any_width(page, balance):
    """What a block needs in shared memory does not grow with the longest request that the block table could hold: 32 short requests
    beside a table of 524,288 tokens, head size 128, with the bits of the same launch on a table just wide enough."""
    H, KV, hd, S = 16, 8, 128, 32
    g = torch.Generator().manual_seed(page)
    lens = torch.randint(1, 200, (S,), generator=g)
    pages = 200 // page + 1
    narrow = torch.randperm(S * pages, generator=g).to(torch.int32).view(S, pages).to(DEV)
    wide = torch.full((S, 524288 // page), -1, dtype=torch.int32, device=DEV)
    wide[:, :pages] = narrow
    kc, vc = (torch.randn(S * pages, KV, page, hd, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
    q = torch.randn(S, H * hd, generator=g).to(torch.bfloat16).to(DEV)
    k = K()
    partials = torch.empty(k.attn_decode_partial_floats(1, KV, hd, max(2 * balance, 2)), device=DEV) if balance else None
    arrived = torch.zeros(S * KV, dtype=torch.int32, device=DEV) if balance else None
    got = []
    for bt in (narrow, wide):
        out = torch.full_like(q, 7.0)
        k.attn_decode_mma(q, out, kc, vc, bt, (lens - 1).to(torch.int32).to(DEV), H, KV, hd, 1.0 / math.sqrt(hd), 0, 1, partials, arrived, balance=balance)
        got.append(out)
    assert torch.equal(*got) and bool(torch.isfinite(got[0]).all())


def test_attn_mma_refusals():
    from vllm_oxide_b200.errors import ShapeError
    k = K()
    assert k.attn_mma_supported(32, 8, 64, 16, True) and k.attn_mma_supported(24, 8, 128, 16, False)
    assert not k.attn_mma_supported(4, 2, 48, 16, False) and not k.attn_mma_supported(4, 2, 64, 24, False)
    assert not k.attn_mma_supported(34, 2, 64, 16, True) and k.attn_mma_supported(34, 2, 64, 16, False)
    q = torch.zeros(1, 4 * 48, dtype=torch.bfloat16, device=DEV)
    kc = torch.zeros(2, 2, 16, 48, dtype=torch.bfloat16, device=DEV)
    z = torch.zeros(2, dtype=torch.int32, device=DEV)
    with pytest.raises(ShapeError, match="not supported"):
        k.attn_prefill_mma(q, q.clone(), kc, kc, torch.zeros(1, 2, dtype=torch.int32, device=DEV), z, z, 1, 1, 4, 2, 48, 1.0)
    with pytest.raises(ShapeError, match="bfloat16 only"):
        k.attn_prefill_mma(q.float(), q.float(), kc.float(), kc.float(), torch.zeros(1, 2, dtype=torch.int32, device=DEV), z, z, 1, 1, 4, 2, 48, 1.0)


# ----------------------------------------------------------------------------- tcgen05 matrix product (bfloat16)
@pytest.mark.parametrize("T,N,Kd", [(1, 128, 64), (3, 200, 136), (8, 3072, 2048), (16, 130, 2048), (17, 2048, 2048), (32, 77, 200), (33, 256, 512)])
def test_linear_bf16_with_a_bias(T, N, Kd):
    """A bias is added to the float32 sum before the result is rounded, once under a split of K too: one rounding to bfloat16 away
    from float64, on this package's product (up to `TUNING.few_rows` rows) and on the library's behind it."""
    g = torch.Generator().manual_seed(T + N)
    a, w = (torch.randn(n, Kd, generator=g).to(torch.bfloat16).to(DEV) for n in (T, N))
    bias = (30 * torch.randn(N, generator=g)).to(torch.bfloat16).to(DEV)
    want = a.double() @ w.double().T + bias.double()
    # half a unit in the last of bfloat16's 8 bits (2^-8 of the value at most), and float32 sums of Kd products
    bound = 2.0 ** -8 * 1.01 * want.abs() + Kd * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    for fixed_w in (False, True):                  # read before the kernels in front are done, or not
        out = torch.full((T + 1, N), 7.0, dtype=torch.bfloat16, device=DEV)
        K().linear(a, w, out[:T], bias, fixed_w)
        assert bool(((out[:T].double() - want).abs() <= bound).all()) and bool((out[T] == 7.0).all())


@pytest.mark.parametrize("odt", [torch.bfloat16, torch.float32], ids=["bf16out", "f32out"])
@pytest.mark.parametrize("T,N,Kd,splits", [
    (1, 128, 64, 1), (8, 128, 256, None), (5, 640, 8192, 8), (8, 2048, 2048, 3), (16, 256, 512, 2), (17, 200, 136, None),
    (33, 200, 136, None), (64, 2048, 2048, None), (100, 300, 520, None), (129, 1000, 1032, None), (300, 520, 264, None),
    (700, 384, 96, None)])
def test_gemm_sm100(T, N, Kd, splits, odt):
    """TMA + tcgen05 product against float64: rows and features that are no multiple of a tile,
    K that is no multiple of 64, every token-tile width (16 ... 256), K split over a cluster."""
    g = torch.Generator().manual_seed(T * 7 + N)
    a = torch.randn(T, Kd, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(N, Kd, generator=g).to(torch.bfloat16).to(DEV)
    out = torch.full((T, N), 7.0, dtype=odt, device=DEV)
    k = K()
    k.gemm_sm100(a, w, out, splits)
    torch.cuda.synchronize()
    k.gemm_sm100_check()
    want = plain.linear(a.double().cpu(), w.double().cpu())
    # bfloat16 inputs are exact and products accumulate in float32: sqrt(K) * 2^-24 like the float32
    # kernel; a bfloat16 result adds one rounding of 2^-9
    tol = (2.0 ** -8) if odt == torch.bfloat16 else max(2e-6, 2.0 ** -22 * math.sqrt(Kd))
    assert rel(out, want) <= tol
    # a row's value does not depend on the rows beside it (same tile width): bitwise
    if T > 1:
        bt = 16 if T <= 16 else 32 if T <= 32 else 64 if T <= 64 else 128 if T <= 128 else 256
        lo = max(0, T - 2) if (T - 1) // bt == 0 or bt == 16 else T - 1
        sub = torch.empty((T - lo, N), dtype=odt, device=DEV)
        if (T - lo <= 16) == (T <= 16) and splits == 1:
            k.gemm_sm100(a[lo:].contiguous(), w, sub, splits)
            assert torch.equal(sub, out[lo:])
    # replay: nothing needs resetting between launches
    out2 = torch.zeros_like(out)
    k.gemm_sm100(a, w, out2, splits)
    assert torch.equal(out2, out)


def test_gemm_sm100_strided_and_refusals():
    from vllm_oxide_b200.errors import ShapeError
    k = K()
    g = torch.Generator().manual_seed(1)
    wide = torch.randn(9, 96, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(50, 64, generator=g).to(torch.bfloat16).to(DEV)
    outw = torch.zeros(9, 80, dtype=torch.bfloat16, device=DEV)
    k.gemm_sm100(wide[:, 16:80], w, outw[:, 8:58])             # column slices of wider buffers
    want = plain.linear(wide[:, 16:80].double().cpu(), w.double().cpu())
    assert rel(outw[:, 8:58], want) <= 2 ** -8
    assert float(outw[:, :8].float().abs().max()) == 0.0 and float(outw[:, 58:].float().abs().max()) == 0.0
    assert not k.gemm_sm100_supported(wide[:, 1:65], w)         # rows not 16-byte aligned
    assert not k.gemm_sm100_supported(wide[:, :60], w[:, :60])  # K no multiple of 8
    with pytest.raises(ShapeError):
        k.gemm_sm100(wide[:, :60], w[:, :60], outw[:, :50])
    # linear() falls back to the library product for such operands instead of failing
    o = torch.empty(9, 50, dtype=torch.bfloat16, device=DEV)
    k.linear(wide[:, :60].contiguous(), w[:, :60].contiguous(), o)
    assert rel(o, plain.linear(wide[:, :60].double().cpu(), w[:, :60].double().cpu())) <= 2 ** -8


# ----------------------------------------------------------------------------- fused epilogues of the tcgen05 product
@pytest.mark.parametrize("T,I,Kd,splits", [(1, 128, 64, 1), (8, 8192, 2048, None), (5, 224, 96, 1), (16, 300, 520, 3), (32, 1000, 256, 2), (17, 128, 1024, 8),
                                            (33, 224, 96, 1), (64, 8192, 2048, None), (50, 300, 520, 3)])
def test_gemm_swiglu(T, I, Kd, splits):
    g = torch.Generator().manual_seed(T + I)
    a = torch.randn(T, Kd, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(2 * I, Kd, generator=g) / math.sqrt(Kd) * 2).to(torch.bfloat16).to(DEV)
    out = torch.full((T, I), 7.0, dtype=torch.bfloat16, device=DEV)
    k = K()
    k.gemm_swiglu(a, w, out, splits)
    torch.cuda.synchronize()
    k.gemm_sm100_check()
    gate = plain.linear(a.double().cpu(), w[:I].double().cpu())
    up = plain.linear(a.double().cpu(), w[I:].double().cpu())
    assert rel(out, plain.swiglu(gate, up)) <= 2 ** -8
    out2 = torch.zeros_like(out)
    k.gemm_swiglu(a, w, out2, splits)
    assert torch.equal(out, out2)


@pytest.mark.parametrize("rope", [True, False])
@pytest.mark.parametrize("T,H,KV,hd,Kd,page,splits", [(8, 32, 8, 64, 2048, 16, None), (1, 4, 2, 64, 128, 16, 1), (13, 3, 1, 32, 96, 8, 1),
                                                      (32, 6, 2, 16, 200, 8, 2), (5, 2, 2, 128, 512, 32, 4), (20, 5, 5, 64, 320, 16, 5),
                                                      (64, 32, 8, 64, 2048, 16, None), (41, 3, 1, 32, 96, 8, 2)])
def test_gemm_qkv_rope(T, H, KV, hd, Kd, page, splits, rope):
    g = torch.Generator().manual_seed(T + H + hd)
    a = torch.randn(T, Kd, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn((H + 2 * KV) * hd, Kd, generator=g) / math.sqrt(Kd)).to(torch.bfloat16).to(DEV)
    cfg = {"head_dim": hd, "hidden_size": H * hd, "num_attention_heads": H, "rope_theta": 500000.0,
           "rope_scaling": {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                            "original_max_position_embeddings": 64}}
    inv = plain.rope_inv_freq(cfg)
    positions = [(37 * i + 5) % 3000 for i in range(T)]
    pages = -(-T // page) + 4
    slots = torch.randperm(pages * page, generator=g)[:T].to(torch.int32)
    if T > 2:
        slots[2] = -1                                                   # this token writes nothing
    kc = torch.full((pages, KV, page, hd), 7.0, dtype=torch.bfloat16, device=DEV)
    vc = torch.full((pages, KV, page, hd), 7.0, dtype=torch.bfloat16, device=DEV)
    q = torch.full((T, H * hd), 7.0, dtype=torch.bfloat16, device=DEV)
    k = K()
    k.gemm_qkv_rope(a, w, q, torch.tensor(positions, dtype=torch.int32, device=DEV), slots.to(DEV),
                    inv.to(DEV) if rope else None, kc, vc, H, KV, hd, splits)
    torch.cuda.synchronize()
    k.gemm_sm100_check()
    qkv = plain.linear(a.double().cpu(), w.double().cpu())
    wq, wk, wv = qkv[:, :H * hd], qkv[:, H * hd:(H + KV) * hd], qkv[:, (H + KV) * hd:]
    if rope:
        wq, wk = plain.rope(wq, positions, inv, hd), plain.rope(wk, positions, inv, hd)
    assert rel(q, wq) <= 2 ** -8
    written = set()
    for t in range(T):
        s_ = int(slots[t])
        if s_ < 0:
            continue
        written.add(s_)
        pg, off = s_ // page, s_ % page
        assert rel(kc[pg, :, off, :].reshape(-1), wk[t]) <= 2 ** -8
        assert rel(vc[pg, :, off, :].reshape(-1), wv[t]) <= 2 ** -8
    for s_ in range(pages * page):
        if s_ not in written:
            assert float((kc[s_ // page, :, s_ % page, :].float() - 7.0).abs().max()) == 0.0
            assert float((vc[s_ // page, :, s_ % page, :].float() - 7.0).abs().max()) == 0.0


def test_fused_gemm_refusals():
    from vllm_oxide_b200.errors import ShapeError
    k = K()
    a = torch.zeros(70, 64, dtype=torch.bfloat16, device=DEV)
    w = torch.zeros(256, 64, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(ShapeError, match="at most 64"):
        k.gemm_swiglu(a, w, torch.zeros(70, 128, dtype=torch.bfloat16, device=DEV))
    assert not k.gemm_qkv_rope_supported(48) and k.gemm_qkv_rope_supported(64)


def _folded_input(T, Kd, g):
    """A residual x [T, Kd], the next norm's weight, and what the folded form hands to a product:
    bf16(x * weight) and the sums of squares of x per 128-feature tile."""
    x = torch.randn(T, Kd, generator=g) * 1.5
    wn = 1.0 + 0.3 * torch.randn(Kd, generator=g)
    xn = (x * wn).to(torch.bfloat16)
    tiles = -(-Kd // 128)
    ssq = torch.zeros(tiles, 64)
    for i in range(tiles):
        ssq[i, :T] = (x[:, i * 128:(i + 1) * 128] ** 2).sum(1)
    return x, wn, xn, ssq


@pytest.mark.parametrize("T,N,Kd,splits", [(1, 128, 128, 1), (8, 2048, 2048, None), (20, 200, 320, 2), (32, 640, 8192, 8),
                                           (33, 200, 320, 1), (64, 2048, 8192, None), (47, 384, 256, 3)])
def test_gemm_fused_residual_and_folded_norm(T, N, Kd, splits):
    """EPI_RESID with the RMSNorm of the input folded in: resid += rmsnorm(x) W^T (the norm as a
    per-token scale of the accumulator), the next norm's input bf16(resid * next_w) and the
    per-tile sums of squares of the new residual come out of the same kernel."""
    from vllm_oxide_b200.kernels import EPI_RESID, EPI_STORE
    g = torch.Generator().manual_seed(T * 3 + N)
    eps = 1e-5
    x, wn, xn, ssq = _folded_input(T, Kd, g)
    w = (torch.randn(N, Kd, generator=g) / math.sqrt(Kd)).to(torch.bfloat16)
    resid0 = torch.randn(T, N, generator=g)
    next_w = 1.0 + 0.3 * torch.randn(N, generator=g)
    k = K()
    resid = resid0.clone().to(DEV)
    xn_out = torch.full((T, N), 7.0, dtype=torch.bfloat16, device=DEV)
    ssq_out = torch.full((-(-N // 128), 64), 7.0, device=DEV)
    k.gemm_fused(xn.to(DEV), w.to(DEV), None, EPI_RESID, N, ssq_in=ssq.to(DEV), eps=eps,
                 resid=(resid, next_w.to(DEV), xn_out, ssq_out), splits=splits)
    torch.cuda.synchronize()
    k.gemm_sm100_check()
    # the plain norm of x with weight wn (x * wn rounded to bfloat16 as the kernel's operand), then the product
    inv = 1.0 / torch.sqrt((x.double() ** 2).mean(1) + eps)
    want_delta = plain.linear(xn.double(), w.double()) * inv[:, None]
    want_resid = resid0.double() + want_delta
    assert rel(resid, want_resid) <= max(2e-6, 2.0 ** -22 * math.sqrt(Kd)) * 4
    assert rel(xn_out, want_resid * next_w.double()) <= 2 ** -8
    got = resid.double().cpu()
    for i in range(-(-N // 128)):
        want_ssq = (got[:, i * 128:(i + 1) * 128] ** 2).sum(1)
        assert rel(ssq_out[i, :T], want_ssq) <= 1e-5
    # the same scale on a plain store
    out = torch.empty(T, N, device=DEV)
    k.gemm_fused(xn.to(DEV), w.to(DEV), out, EPI_STORE, N, ssq_in=ssq.to(DEV), eps=eps, splits=splits)
    assert rel(out, want_delta) <= max(2e-6, 2.0 ** -22 * math.sqrt(Kd)) * 4


@pytest.mark.parametrize("N,Kd,splits", [(640, 320, 5), (392, 1344, 6), (4096, 4096, 7), (512, 832, 7), (4096, 14336, 7)])
@pytest.mark.parametrize("T", [1, 8, 16, 24, 32])
def test_few_row_product_on_clusters_of_five_to_seven(T, N, Kd, splits):
    """K shared by five, six and seven blocks, the last with less of it than the others: the residual epilogue and the plain one. Seven is what
    4,096 features get."""
    from vllm_oxide_b200.kernels import EPI_RESID
    k = K()
    if N == 4096:
        assert k._pick_splits(T, N, Kd, torch.device("cuda", 0)) == splits
    g = torch.Generator().manual_seed(T * 3 + N + Kd)
    a = torch.randn(T, Kd, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(N, Kd, generator=g) / math.sqrt(Kd)).to(torch.bfloat16).to(DEV)
    want = a.double() @ w.double().t()
    tol = max(2e-6, 2.0 ** -22 * math.sqrt(Kd))
    out = torch.full((T, N), 7.0, device=DEV)
    k.gemm_sm100(a, w, out, splits)
    assert rel(out, want.cpu()) <= tol
    resid0, next_w = torch.randn(T, N, generator=g).to(DEV), (1.0 + 0.3 * torch.randn(N, generator=g)).to(DEV)
    resid = resid0.clone()
    xn_out = torch.full((T, N), 7.0, dtype=torch.bfloat16, device=DEV)
    ssq_out = torch.full((-(-N // 128), 64), 7.0, device=DEV)
    k.gemm_fused(a, w, None, EPI_RESID, N, resid=(resid, next_w, xn_out, ssq_out), splits=splits)
    torch.cuda.synchronize()
    k.gemm_sm100_check()
    want_resid = resid0.double() + want
    assert rel(resid, want_resid.cpu()) <= tol
    assert rel(xn_out, (want_resid * next_w.double()).cpu()) <= 2 ** -8
    for i in range(-(-N // 128)):
        assert rel(ssq_out[i, :T], (resid.double()[:, i * 128:(i + 1) * 128] ** 2).sum(1).cpu()) <= 1e-5


@pytest.mark.parametrize("N,Kd", [(16390, 2000), (16384, 1024), (8200, 4096), (4100, 8192), (500, 8200), (32777, 1536)])
def test_gemm_f32_few_rows_chunks_of_a_block(N, Kd):
    """A block of the few-row kernel that has all, half or a quarter of K's chunks, and rows taken eight at a time: every count of rows
    gives the bits that the same rows have in a product of 40, which the tiles compute."""
    g = torch.Generator().manual_seed(N + Kd)
    a = torch.randn(40, Kd, generator=g).to(DEV)
    w = torch.randn(N, Kd, generator=g).to(DEV)
    k = K()
    want = torch.empty(40, N, device=DEV)
    k.gemm_f32(a, w, want)
    assert rel(want[:2], (a[:2].double() @ w.double().t()).cpu()) <= 2.0 ** -22 * math.sqrt(Kd)
    for M in (1, 2, 3, 4, 5, 8, 9, 16, 17, 24, 25):
        out = torch.full((M, N), 7.0, device=DEV)
        k.gemm_f32(a[:M], w, out)
        assert torch.equal(out, want[:M]), M


def test_gemm_f32_few_rows_stages():
    """Three and four rows have a ring of three stages where the grid fills at most two waves (two cost up to a quarter of the time) and
    two blocks still find room on an SM, or all blocks an SM each; two elsewhere and where a block adds up more than an eighth of K. All give
    the bits of the tiles."""
    from vllm_oxide_b200 import kernels
    plan = kernels._fn("gemm_f32", "vob_gemm_f32_few_plan", [kernels._I] * 4)
    for M in (3, 4):
        for N, Kd, stages in ((3072, 1024, 3), (1024, 8960, 3), (896, 14336, 3), (500, 516, 3), (49152, 1280, 2), (16384, 2048, 2), (1024, 11008, 2),
                              (4100, 14336, 2), (2048, 14336, 2)):
            assert plan(M, N, Kd, 64) % 8 == stages, (M, N, Kd)
    assert {plan(M, 3072, 1024, 64) % 8 for M in (1, 2, 5, 8, 9, 16)} == {2}
    g = torch.Generator().manual_seed(3)
    for N, Kd in ((3072, 1024), (897, 14336), (500, 516), (9000, 1280), (1025, 11008)):
        a, w = torch.randn(40, Kd, generator=g).to(DEV), torch.randn(N, Kd, generator=g).to(DEV)
        want = torch.empty(40, N, device=DEV)
        kernels.gemm_f32(a, w, want)
        for M in (3, 4):
            out = torch.full((M, N), 7.0, device=DEV)
            kernels.gemm_f32(a[:M], w, out)
            assert torch.equal(out, want[:M]), (M, N, Kd)


def test_gemm_f32_few_rows_waves():
    """With one and two rows a block of the few-row kernel takes more than an eighth of K only where its waves of blocks are at least 0.7 full (sizes
    above one wave lost up to a fifth); wherever it is cut, a row has the bits it has in the tiles."""
    from vllm_oxide_b200 import kernels
    plan = kernels._fn("gemm_f32", "vob_gemm_f32_few_plan", [kernels._I] * 4)
    longer = 0
    for N in list(range(64, 34000, 1088)) + [6144, 11008, 16384, 22016, 28672, 128256]:
        for Kd in (516, 2048, 2560, 4096, 8192, 14336):
            for M in (1, 2):
                nc = -(-Kd // 128)
                q = plan(M, N, Kd, 64) // 8
                if q == ((nc + 7) // 8 + 3) // 4 * 4:
                    continue
                smem = 4 * (8 * 2 * 32 * 32 + 4 * 128 * M + q * M * 64)
                waves = -(-N // 64) * -(-nc // q) / (148 * min(3, 227 * 1024 // (smem + 1024)))
                assert waves <= 1.05 or waves >= 0.7 * math.ceil(waves), (N, Kd, M, q)
                longer += 1
    assert longer > 40 and plan(2, 6144, 8192, 64) // 8 == 8 and plan(1, 16384, 2048, 64) // 8 == 16 and plan(4, 11008, 4096, 64) // 8 == 16
    g = torch.Generator().manual_seed(4)
    for N, Kd in ((6144, 4096), (11008, 2048), (22016, 1280)):
        a, w = torch.randn(40, Kd, generator=g).to(DEV), torch.randn(N, Kd, generator=g).to(DEV)
        want = torch.empty(40, N, device=DEV)
        kernels.gemm_f32(a, w, want)
        for M in (1, 2, 4, 8):
            out = torch.full((M, N), 7.0, device=DEV)
            kernels.gemm_f32(a[:M], w, out)
            assert torch.equal(out, want[:M]), (M, N, Kd)


@pytest.mark.parametrize("N,Kd", [(500, 4612), (764, 4992), (768, 4612), (500, 5120), (1024, 4100), (2048, 5000), (3200, 4100), (3204, 4100), (3072, 16512), (3076, 16388)])
def test_gemm_f32_rows_by_eights(N, Kd):
    """On both sides of the lines between rows taken eight at a time and the tiles: the bits of a product of 40 rows, and as many launches
    counted as there are."""
    from vllm_oxide_b200 import kernels
    pieces = kernels._fn("gemm_f32", "vob_gemm_f32_launches", [kernels._I] * 3)
    narrow = N < 768 and Kd < 4993 or N > 3072 and Kd > 16384
    g = torch.Generator().manual_seed(N + Kd)
    a, w = torch.randn(40, Kd, generator=g).to(DEV), torch.randn(N, Kd, generator=g).to(DEV)
    want = torch.empty(40, N, device=DEV)
    kernels.gemm_f32(a, w, want)
    for M in (8, 9, 16, 17, 24, 25):
        by_eights = 8 < M <= 16 and not narrow or 16 < M <= 24 and 1536 <= N <= 3200 and 33e6 < 4 * N * Kd <= 70e6
        assert pieces(M, N, Kd) == (-(-M // 8) if by_eights else 1), M
        out = torch.full((M, N), 7.0, device=DEV)
        before = kernels.launch_count()
        kernels.gemm_f32(a[:M], w, out)
        assert kernels.launch_count() - before == pieces(M, N, Kd), M
        assert torch.equal(out, want[:M]), M


@pytest.mark.parametrize("N,Kd,M,tr,c", [
    (65, 516, 17, 2, 1), (65, 1028, 17, 2, 8), (1541, 516, 65, 4, 1), (65, 1028, 177, 4, 8), (8201, 516, 65, 5, 1), (65, 1028, 300, 5, 8),
    (4101, 516, 350, 6, 1), (501, 1028, 81, 6, 8), (3101, 516, 640, 7, 1), (501, 1028, 97, 7, 8), (8201, 516, 225, 8, 1), (501, 1028, 113, 8, 8),
    (65, 130, 17, 2, 1), (65, 1030, 17, 2, 8), (1541, 130, 65, 4, 1), (65, 1030, 130, 4, 8), (4101, 130, 65, 5, 1), (65, 1030, 300, 5, 8),
    (8201, 130, 81, 6, 1), (201, 1030, 177, 6, 8), (3101, 130, 640, 7, 1), (501, 1030, 97, 7, 8), (12301, 130, 350, 8, 1), (501, 1030, 113, 8, 8)])
def test_gemm_f32_tile_choice(N, Kd, M, tr, c):
    """Every tile height with and without a shared K, operands that come by 16 and by 4 bytes: the choice that the rule makes at these sizes, and the
    bits that the few-row kernel or, where operands come by 4 bytes, tiles of 32 rows give."""
    from vllm_oxide_b200 import kernels
    choice = kernels._fn("gemm_f32", "vob_gemm_f32_tile", [kernels._I] * 4)
    assert divmod(choice(M, N, Kd, int(Kd % 4 == 0)), 16) == (tr, c)
    g = torch.Generator().manual_seed(N + Kd + M)
    a, w = torch.randn(M, Kd, generator=g).to(DEV), torch.randn(N, Kd, generator=g).to(DEV)
    want = torch.empty(M, N, device=DEV)
    for r in range(0, M, 8):
        kernels.gemm_f32(a[r:r + 8], w, want[r:r + 8])
    assert rel(want, (a.double() @ w.double().t()).cpu()) <= 2.0 ** -22 * math.sqrt(Kd)
    out = torch.full((M + 1, N), 7.0, device=DEV)
    kernels.gemm_f32(a, w, out[:M])
    assert torch.equal(out[:M], want)
    assert float((out[M:] - 7.0).abs().max()) == 0.0


def test_gemm_f32_tiles_of_an_idle_chip():
    """Where every tile has an SM to itself the smallest tiles are the fastest, whatever rows of them are not there (higher ones, chosen by their
    waves alone, took half as long again)."""
    from vllm_oxide_b200 import kernels
    choice = kernels._fn("gemm_f32", "vob_gemm_f32_tile", [kernels._I] * 4)
    for M in (17, 33, 65, 72, 81, 97, 130, 160, 260, 400, 700, 1000, 2048):
        for N in (1, 64, 200, 500, 1000, 2048):
            tiles = -(-M // 32) * -(-N // 64)
            if tiles <= 48:
                assert all(choice(M, N, Kd, v) // 16 == 2 for Kd in (128, 516, 892) for v in (0, 1)), (M, N)
            if tiles <= 8:
                assert all(choice(M, N, Kd, 1) == 2 * 16 + 8 for Kd in (1024, 2048, 8192)), (M, N)


@pytest.mark.parametrize("N,Kd", [(70, 53252), (70, 61440), (70, 61444), (33, 65536), (1024, 65536)])
def test_gemm_f32_few_rows_of_a_k_without_room(N, Kd):
    """A K whose chunks' sums find no room in a block of the few-row kernel goes to the tiles, rows taken eight at a time too: the
    bits of a product of 40 rows, up to the longest K that fits and beyond it."""
    g = torch.Generator().manual_seed(N + Kd)
    a = torch.randn(40, Kd, generator=g).to(DEV)
    w = torch.randn(N, Kd, generator=g).to(DEV)
    k = K()
    want = torch.empty(40, N, device=DEV)
    k.gemm_f32(a, w, want)
    assert rel(want[:2], (a[:2].double() @ w.double().t()).cpu()) <= 2.0 ** -22 * math.sqrt(Kd)
    for M in (1, 4, 8, 9, 12, 16, 17, 24):
        out = torch.full((M, N), 7.0, device=DEV)
        k.gemm_f32(a[:M], w, out)
        assert torch.equal(out, want[:M]), M


@pytest.mark.parametrize("N,Kd", [(2100, 1152), (9000, 200), (2050, 1155), (9000, 203), (16384, 1028), (70, 2052), (740, 200), (740, 203)])
def test_gemm_f32_tiles_of_every_height(N, Kd):
    """Tiles of 80, 96 and 112 rows beside those of 32, 64 and 128, K shared over a cluster and not, operands that come by 16 and by 4
    bytes: whatever the launcher takes, a row has the bits it has in the few-row kernel or in another tile."""
    g = torch.Generator().manual_seed(N + Kd)
    a = torch.randn(640, Kd, generator=g).to(DEV)
    w = torch.randn(N, Kd, generator=g).to(DEV)
    k = K()
    want = torch.empty(640, N, device=DEV)
    for r in range(0, 640, 8):
        k.gemm_f32(a[r:r + 8], w, want[r:r + 8])
    assert rel(want[:64], (a[:64].double() @ w.double().t()).cpu()) <= 2.0 ** -22 * math.sqrt(Kd)
    for M in (65, 70, 80, 81, 90, 96, 97, 100, 112, 113, 150, 160, 200, 224, 260, 288, 300, 400, 517, 640):
        out = torch.full((M + 1, N), 7.0, device=DEV)
        k.gemm_f32(a[:M], w, out[:M])
        assert torch.equal(out[:M], want[:M]), M
        assert float((out[M:] - 7.0).abs().max()) == 0.0


@pytest.mark.parametrize("I,Kd", [(1, 4), (33, 64), (40, 516), (96, 1152), (160, 4100), (64, 8192), (8200, 2000)])
@pytest.mark.parametrize("M", [1, 2, 3, 8, 9, 16])
def test_gemm_f32_swiglu(M, I, Kd):
    """Gate/up and activation in the few-row product's epilogue: the bits of the product and the activation kernel one behind the
    other, for features that are no multiple of a block's 32, K of one chunk to many; other sizes are refused."""
    from vllm_oxide_b200.errors import ShapeError
    g = torch.Generator().manual_seed(M * 1000 + I + Kd)
    a = torch.randn(M, Kd + 4, generator=g).to(DEV)[:, :Kd]
    w = (torch.randn(2 * I, Kd, generator=g) / math.sqrt(Kd) * 2).to(DEV)
    k = K()
    out = torch.full((M, I + 3), 7.0, device=DEV)
    assert not k.gemm_f32_swiglu_supported(a[:, :Kd - 1], w[:, :Kd - 1]) and not k.gemm_f32_swiglu_supported(a.repeat(17, 1), w)
    if not k.gemm_f32_swiglu_supported(a, w):
        assert M > (4 if Kd <= 64 else 8)
        with pytest.raises(ShapeError):
            k.gemm_f32_swiglu(a, w, out[:, :I])
        return
    torch.cuda.synchronize()
    k.gemm_f32_swiglu(a, w, out[:, :I], fixed_w=True)
    gu, want = torch.empty(M, 2 * I, device=DEV), torch.empty(M, I, device=DEV)
    k.gemm_f32(a, w, gu)
    k.glu(gu, want)
    assert torch.equal(out[:, :I], want)
    assert float((out[:, I:] - 7.0).abs().max()) == 0.0


# ----------------------------------------------------------------------------- tcgen05 product on pairs of SMs
@pytest.mark.parametrize("odt", [torch.bfloat16, torch.float32], ids=["bf16out", "f32out"])
@pytest.mark.parametrize("T,N,Kd", [(1, 8, 64), (256, 256, 64), (300, 520, 264), (129, 1000, 1032), (700, 384, 96), (1030, 2048, 512)])
def test_gemm_sm100_pair(T, N, Kd, odt):
    """The two-SM product (tcgen05.mma.cta_group::2) against float64: rows and features that are no
    multiple of a tile, K that is no multiple of 64, one tile and many, both output types."""
    g = torch.Generator().manual_seed(T * 5 + N)
    a = torch.randn(T, Kd, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(N, Kd, generator=g).to(torch.bfloat16).to(DEV)
    out = torch.full((T, N), 7.0, dtype=odt, device=DEV)
    k = K()
    k.gemm_sm100_pair(a, w, out)
    torch.cuda.synchronize()
    k.gemm_sm100_check()
    want = plain.linear(a.double().cpu(), w.double().cpu())
    tol = (2.0 ** -8) if odt == torch.bfloat16 else max(2e-6, 2.0 ** -22 * math.sqrt(Kd))
    assert rel(out, want) <= tol
    out2 = torch.zeros_like(out)
    k.gemm_sm100_pair(a, w, out2)                                # nothing needs resetting between launches
    assert torch.equal(out2, out)
    # a row's value does not depend on the rows beside it
    if T > 2:
        sub = torch.empty((2, N), dtype=odt, device=DEV)
        k.gemm_sm100_pair(a[T - 2:].contiguous(), w, sub)
        assert torch.equal(sub, out[T - 2:])


@pytest.mark.parametrize("odt", [torch.bfloat16, torch.float32], ids=["bf16out", "f32out"])
@pytest.mark.parametrize("T,N,Kd,bn", [(513, 16392, 520, 192), (1000, 16384, 456, 256)])
def test_gemm_sm100_pair_wide_token_tiles(T, N, Kd, bn, odt):
    """The plain store with tiles of 192 and 256 tokens, several to a pair of SMs, and a ring that wraps."""
    from vllm_oxide_b200 import kernels
    assert kernels._fn("gemm_sm100_pair", "vob_gemm_sm100_pair_tokens", [kernels._I] * 4)(T, N, 0, 74) == bn
    g = torch.Generator().manual_seed(T + N)
    a = torch.randn(T, Kd, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(N, Kd, generator=g).to(torch.bfloat16).to(DEV)
    out = torch.full((T + 1, N), 7.0, dtype=odt, device=DEV)
    kernels.gemm_sm100_pair(a, w, out[:T])
    torch.cuda.synchronize()
    kernels.gemm_sm100_check()
    assert rel(out[:T], (a.double() @ w.double().t()).cpu()) <= (2.0 ** -8 if odt == torch.bfloat16 else max(2e-6, 2.0 ** -22 * math.sqrt(Kd)))
    assert float((out[T:].float() - 7.0).abs().max()) == 0.0


def test_gemm_sm100_pair_narrow_output_rows():
    """An output whose rows are not 16-byte aligned takes the element-wise store path."""
    g = torch.Generator().manual_seed(3)
    a = torch.randn(200, 128, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(100, 128, generator=g).to(torch.bfloat16).to(DEV)
    wide = torch.full((200, 101), 7.0, dtype=torch.bfloat16, device=DEV)
    k = K()
    k.gemm_sm100_pair(a, w, wide[:, :100])
    assert rel(wide[:, :100], plain.linear(a.double().cpu(), w.double().cpu())) <= 2 ** -8
    assert float((wide[:, 100].float() - 7.0).abs().max()) == 0.0


@pytest.mark.parametrize("T,I,Kd", [(1, 64, 64), (256, 128, 64), (300, 300, 264), (700, 224, 96), (1100, 1000, 256)])
def test_gemm_pair_swiglu(T, I, Kd):
    g = torch.Generator().manual_seed(T + I)
    a = torch.randn(T, Kd, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(2 * I, Kd, generator=g) / math.sqrt(Kd) * 2).to(torch.bfloat16).to(DEV)
    out = torch.full((T, I), 7.0, dtype=torch.bfloat16, device=DEV)
    k = K()
    k.gemm_pair_swiglu(a, w, out)
    torch.cuda.synchronize()
    k.gemm_sm100_check()
    gate = plain.linear(a.double().cpu(), w[:I].double().cpu())
    up = plain.linear(a.double().cpu(), w[I:].double().cpu())
    assert rel(out, plain.swiglu(gate, up)) <= 2 ** -8
    out2 = torch.zeros_like(out)
    k.gemm_pair_swiglu(a, w, out2)
    assert torch.equal(out, out2)


# tokens, features, K, weights asked for early, tokens of a tile on 74 pairs of SMs
PAIR_TOKEN_TILES = [(33, 8192, 64, True, 64), (64, 128, 832, True, 32), (100, 64, 704, False, 32), (300, 8192, 72, True, 160), (517, 4224, 128, False, 160),
                    (600, 8192, 64, True, 224), (1201, 640, 200, True, 96), (120, 9472, 712, True, 128), (350, 5632, 584, True, 128), (517, 8192, 520, True, 192),
                    (600, 8192, 520, False, 224), (1000, 8192, 456, True, 256), (700, 14336, 456, False, 256)]


def test_gemm_pair_token_tiles_are_all_tested():
    from vllm_oxide_b200 import kernels
    pick = kernels._fn("gemm_sm100_pair", "vob_gemm_sm100_pair_tokens", [kernels._I] * 4)
    assert [pick(T, I, 1, 74) for T, I, *_ in PAIR_TOKEN_TILES] == [bn for *_, bn in PAIR_TOKEN_TILES]
    assert {bn for *_, bn in PAIR_TOKEN_TILES} == {pick(T, I, 1, 74) for T in range(1, 2049, 3) for I in (64, 640, 1024, 2816, 4224, 5632, 8192, 9472, 14336)}
    # several tiles a pair and more K blocks than the ring has stages (ten, or what 192 KB hold)
    for bn in (128, 192, 224, 256):
        assert any(b == bn and -(-T // b) * -(-I // 128) > 74 and -(-Kd // 64) > min(10, 196608 // (16384 + 64 * b))
                   for T, I, Kd, _, b in PAIR_TOKEN_TILES), bn


@pytest.mark.parametrize("T,I,Kd,early,bn", PAIR_TOKEN_TILES)
def test_gemm_pair_swiglu_token_tiles(T, I, Kd, early, bn):
    """Token tiles of every width the launcher picks (32 to 256), more K blocks than a ring of ten stages holds, several tiles a
    pair of SMs; weights asked for before the kernels in front are done or behind them: the same bits."""
    g = torch.Generator().manual_seed(T * 3 + I)
    a = torch.randn(T, Kd, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(2 * I, Kd, generator=g) / math.sqrt(Kd) * 2).to(torch.bfloat16).to(DEV)
    out, other = (torch.full((T, I), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    k = K()
    torch.cuda.synchronize()
    k.gemm_pair_swiglu(a, w, out, fixed_w=early)
    k.gemm_pair_swiglu(a, w, other, fixed_w=not early)
    torch.cuda.synchronize()
    k.gemm_sm100_check()
    want = plain.swiglu(plain.linear(a.double(), w[:I].double()), plain.linear(a.double(), w[I:].double()))
    assert rel(out, want.cpu()) <= 2 ** -8                       # one rounding to bfloat16, as above
    assert torch.equal(out, other)


def test_a_wait_that_runs_out_raises_the_error_word_and_harms_nothing():
    """The give-up path of the tensor-core kernels: a one-block launch of the few-token product is
    told to expect 16 bytes more than its loads bring, with the wait limit lowered to 10 ms. The
    kernel returns (no hang, no fault), the error word turns into a KernelError, and the next
    ordinary launch on the same context is correct."""
    from vllm_oxide_b200 import kernels
    from vllm_oxide_b200.errors import KernelError
    g = torch.Generator().manual_seed(90)
    a = torch.randn(8, 256, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(128, 256, generator=g).to(torch.bfloat16).to(DEV)
    out = torch.zeros(8, 128, dtype=torch.float32, device=DEV)
    kernels.gemm_sm100(a, w, out, splits=1)
    torch.cuda.synchronize()
    kernels.gemm_sm100_check()                                   # nothing wrong so far
    want = a.double().cpu() @ w.double().cpu().t()
    assert rel(out.cpu(), want) <= 1e-5
    kernels.gemm_sm100_test_hooks(extra_tx_bytes=16, wait_limit_ms=10.0)
    try:
        kernels.gemm_sm100(a, w, torch.zeros_like(out), splits=1)
        torch.cuda.synchronize()                           # returns after some 10 ms
    finally:
        kernels.gemm_sm100_test_hooks(0, 0.0)
    with pytest.raises(KernelError, match="bounded wait"):
        kernels.gemm_sm100_check()
    kernels.gemm_sm100_check()                                   # the word was cleared by the check
    out2 = torch.zeros_like(out)
    kernels.gemm_sm100(a, w, out2, splits=1)
    big = torch.zeros(8, 2048, dtype=torch.float32, device=DEV)
    w2 = torch.randn(2048, 256, generator=g).to(torch.bfloat16).to(DEV)
    kernels.gemm_sm100(a, w2, big)                               # and a launch with a cluster split
    torch.cuda.synchronize()
    kernels.gemm_sm100_check()
    assert rel(out2.cpu(), want) <= 1e-5
    assert rel(big.cpu(), a.double().cpu() @ w2.double().cpu().t()) <= 1e-5


@pytest.mark.parametrize("T,V,Kd", [(1, 128, 64), (8, 128256, 256), (5, 1000, 96), (16, 301, 128), (33, 5000, 64), (64, 2048, 320)])
def test_output_head_that_picks_in_its_epilogue(T, V, Kd):
    """EPI_PICK + pick_final against the logits (EPI_STORE) + pick_tokens: the same tokens for greedy
    and sampled rows, ties kept at the first index, a NaN row flagged, with the folded norm's scale."""
    from vllm_oxide_b200 import kernels
    g = torch.Generator().manual_seed(V + T)
    x, wn, xn, ssq = _folded_input(T, Kd, g)
    w = (torch.randn(V, Kd, generator=g) * 0.2).to(torch.bfloat16)
    if V > 40:
        w[37] = w[11]                                      # a tie between two logits of every row: the first index wins
        w[V - 1] = w[11]
    w, xn, ssq = w.to(DEV), xn.to(DEV), ssq.to(DEV)
    if T > 2:
        xn[2] = float("nan")                               # row 2 holds NaN logits
    temps = torch.tensor([0.0 if i % 3 else 0.8 for i in range(T)], device=DEV)
    temps[0] = 0.0
    seeds = torch.tensor([[i + 1, 7 * i] for i in range(T)], dtype=torch.int32, device=DEV)
    steps = torch.arange(T, dtype=torch.int32, device=DEV) + 3
    logits = torch.empty(T, V, dtype=torch.float32, device=DEV)
    kernels.gemm_fused(xn, w, logits, kernels.EPI_STORE, V, ssq_in=ssq, eps=1e-5)
    sp = kernels.pick_splits(V)
    want = torch.zeros(T, dtype=torch.int32, device=DEV)
    kernels.pick_tokens(logits, want, torch.zeros(T, dtype=torch.int32, device=DEV), torch.empty(T * sp, device=DEV),
                        torch.empty(T * sp, dtype=torch.int32, device=DEV), temps, seeds, steps)
    tiles = kernels.pick_tiles(V)
    pv = torch.full((T, tiles + 3), float("nan"), device=DEV)
    pi = torch.full((T, tiles + 3), -5, dtype=torch.int32, device=DEV)
    flags = torch.zeros(T, dtype=torch.int32, device=DEV)
    got = torch.full((T,), -9, dtype=torch.int32, device=DEV)
    kernels.gemm_fused(xn, w, None, kernels.EPI_PICK, V, ssq_in=ssq, eps=1e-5, pick=(temps, seeds, steps, pv, pi, flags))
    kernels.pick_final(pv[:, :tiles].contiguous(), pi[:, :tiles].contiguous(), T, V, flags, got)
    assert got.tolist() == want.tolist()
    if T > 2:
        assert got[2].item() == -1 and int(flags.sum()) == 0          # flagged, and the flag was put back
    if V > 40:
        assert got[0].item() != 37 and got[0].item() != V - 1         # never the later twin of a tie
    # greedy without sampling parameters at all
    got2 = torch.full((T,), -9, dtype=torch.int32, device=DEV)
    kernels.gemm_fused(xn, w, None, kernels.EPI_PICK, V, ssq_in=ssq, eps=1e-5, pick=(None, None, None, pv, pi, flags))
    kernels.pick_final(pv[:, :tiles].contiguous(), pi[:, :tiles].contiguous(), T, V, flags, got2)
    ref = torch.where(torch.isnan(logits).any(1), torch.full_like(want, -1), logits.argmax(1).to(torch.int32))
    assert got2.tolist() == ref.tolist()
