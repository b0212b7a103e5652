"""Each CUDA kernel alone against a plain float32 torch formula, at sizes the engine's tiny
models do not use (odd widths, head sizes in steps of 16, group sizes, long rows)."""
import math

import pytest
import torch

import plain_gemma2 as plain

pytestmark = pytest.mark.gpu

DT = [torch.float32, torch.bfloat16]
PAGE = 64


@pytest.fixture(scope="module")
def ops():
    from trapetum_b200.csrc import ops as o
    assert torch.cuda.is_available(), "these tests need a GPU"
    return o


def tol(dt):
    return 2e-6 if dt == torch.float32 else 1e-2


def close(got, want, dt, scale=1.0):
    got, want = got.float().cpu(), want.float().cpu()
    err = float((got - want).abs().max())
    ref = float(want.abs().max()) + 1e-6
    assert err <= tol(dt) * scale * max(ref, 1.0), f"max abs err {err} (ref max {ref})"


def rnd(*shape, dt=torch.float32, s=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + sum(shape))
    return (torch.randn(*shape, device="cuda", generator=g) * s).to(dt)


# ---------------------------------------------------------------------------
@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("V,H", [(50, 24), (301, 1000), (1024, 2304)])
def test_embed(ops, dt, V, H):
    table = rnd(V, H, dt=dt)
    ids = torch.tensor([0, V - 1, 3, 3, V // 2], dtype=torch.int32, device="cuda")
    out = ops.embed(ids, table, 7.5)
    assert out.dtype == torch.float32
    assert torch.equal(out, table.float()[ids.long()] * 7.5)
    bad = ops.embed(torch.tensor([V, -1], dtype=torch.int32, device="cuda"), table, 1.0)
    assert torch.isnan(bad).all()                     # an id outside the table cannot pass for a result


def test_gather_rows(ops):
    x = rnd(37, 131)
    rows = torch.tensor([36, 0, 5, 5], dtype=torch.int32, device="cuda")
    assert torch.equal(ops.gather_rows(x, rows), x[rows.long()])


@pytest.mark.parametrize("xdt", DT)
@pytest.mark.parametrize("wdt", DT)
@pytest.mark.parametrize("odt", DT)
@pytest.mark.parametrize("rows,width,eps,off", [(3, 17, 1e-6, 1.0), (5, 2304, 1e-5, 1.0), (2, 5000, 1e-3, 0.0)])
def test_rmsnorm(ops, xdt, wdt, odt, rows, width, eps, off):
    x, w = rnd(rows, width, dt=xdt, s=3.0), rnd(width, dt=wdt, s=0.3)
    got = ops.rmsnorm(x, w, eps, off, odt)
    xf, wf = x.float(), w.float()
    want = xf * torch.rsqrt((xf * xf).mean(-1, keepdim=True) + eps) * (off + wf)
    close(got, want, odt)


@pytest.mark.parametrize("adt", DT)
@pytest.mark.parametrize("odt", DT)
@pytest.mark.parametrize("rows,width", [(4, 72), (3, 2304), (1, 4099)])
def test_add_rmsnorm(ops, adt, odt, rows, width):
    h0, a = rnd(rows, width, s=2.0), rnd(rows, width, dt=adt, s=5.0, seed=1)
    wa, wb = rnd(width, dt=odt, s=0.2, seed=2), rnd(width, dt=odt, s=0.2, seed=3)
    af = a.float()
    add = af * torch.rsqrt((af * af).mean(-1, keepdim=True) + 1e-6) * (1.0 + wa.float())
    h = h0.clone()
    assert ops.add_rmsnorm(h, a, wa, 1e-6, 1.0) is None
    close(h, h0 + add, torch.float32, 2.0)
    h = h0.clone()
    x = ops.add_rmsnorm(h, a, wa, 1e-6, 1.0, wb, 1e-5, 0.0, odt)
    hn = h0 + add
    close(h, hn, torch.float32, 2.0)
    close(x, hn * torch.rsqrt((hn * hn).mean(-1, keepdim=True) + 1e-5) * wb.float(), odt, 2.0)
    h = h0.clone()
    ops.residual_add(h, a)
    close(h, h0 + af, torch.float32)


@pytest.mark.parametrize("odt", DT)
@pytest.mark.parametrize("rows,width", [(64, 2304), (100, 3584), (65, 4608), (300, 520), (70, 72), (64, 5120)])
def test_add_rmsnorm_many_rows(ops, odt, rows, width):
    """Many rows take the warp-per-row kernel (32-bit branch, bfloat16 weights); same numbers as the formula."""
    h0, a = rnd(rows, width, s=2.0), rnd(rows, width, s=5.0, seed=1)
    wa, wb = rnd(width, dt=torch.bfloat16, s=0.2, seed=2), rnd(width, dt=torch.bfloat16, s=0.2, seed=3)
    add = a * torch.rsqrt((a * a).mean(-1, keepdim=True) + 1e-6) * (1.0 + wa.float())
    hn = h0 + add
    h = h0.clone()
    x = ops.add_rmsnorm(h, a, wa, 1e-6, 1.0, wb, 1e-5, 1.0, odt)
    close(h, hn, torch.float32, 2.0)
    close(x, hn * torch.rsqrt((hn * hn).mean(-1, keepdim=True) + 1e-5) * (1.0 + wb.float()), odt, 2.0)
    h = h0.clone()
    assert ops.add_rmsnorm(h, a, wa, 1e-6, 1.0) is None
    close(h, hn, torch.float32, 2.0)


@pytest.mark.parametrize("rows,width,splits", [(8, 2304, 8), (3, 72, 2), (1, 12000, 5)])
def test_add_rmsnorm_from_partial_sums(ops, rows, width, splits):
    part = rnd(splits, rows, width, s=2.0)
    h0 = rnd(rows, width, seed=5)
    wa, wb = rnd(width, dt=torch.bfloat16, s=0.2, seed=2), rnd(width, dt=torch.bfloat16, s=0.2, seed=3)
    a = part[0].clone()
    for s_ in range(1, splits):
        a += part[s_]                                                # the kernel adds in split order too
    h1, h2 = h0.clone(), h0.clone()
    x1 = ops.add_rmsnorm(h1, a, wa, 1e-6, 1.0, wb, 1e-6, 1.0, torch.bfloat16)
    x2 = ops.add_rmsnorm(h2, part, wa, 1e-6, 1.0, wb, 1e-6, 1.0, torch.bfloat16)
    assert torch.equal(h1, h2) and torch.equal(x1, x2)
    assert torch.equal(ops.sum_partials(part), a)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("act", ["gelu_tanh", "silu"])
def test_gated_act(ops, dt, act):
    gu = rnd(5, 2 * 333, dt=dt, s=2.0)
    g, u = gu.float()[:, :333], gu.float()[:, 333:]
    want = (plain.gelu_tanh(g) if act == "gelu_tanh" else g * torch.sigmoid(g)) * u
    close(ops.gated_act(gu, act, dt), want, dt)


@pytest.mark.parametrize("adt,wdt,odt", [(torch.float32, torch.float32, torch.float32),
                                         (torch.bfloat16, torch.bfloat16, torch.bfloat16),
                                         (torch.bfloat16, torch.float32, torch.float32),
                                         (torch.bfloat16, torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (7, 301, 100), (65, 130, 77), (200, 64, 1030)])
def test_gemm_simt(ops, adt, wdt, odt, M, N, K):
    a, w = rnd(M, K, dt=adt, s=0.5), rnd(N, K, dt=wdt, s=0.5, seed=1)
    want = a.double() @ w.double().T
    close(ops.gemm_simt(a, w, odt), want, odt, scale=math.sqrt(K))
    close(ops.gemm_simt(a, w, torch.float32, softcap=3.0), 3.0 * torch.tanh(want / 3.0), torch.float32, scale=4.0)


def test_gemm_simt_row_does_not_depend_on_the_batch(ops):
    a, w = rnd(50, 333), rnd(97, 333, seed=1)
    full = ops.gemm_simt(a, w, torch.float32)
    one = ops.gemm_simt(a[17:18].contiguous(), w, torch.float32)
    assert torch.equal(full[17:18], one)


def recorded(ops, monkeypatch):
    """The names of the kernel entries that calls go through from here on."""
    names, check = [], ops._check

    def record(lib, status, what, kernels=1):
        names.append(what)
        return check(lib, status, what, kernels)
    monkeypatch.setattr(ops, "_check", record)
    return names


@pytest.mark.parametrize("heads,P,N,groups,lens,span", [(2, 64, 128, 1, [128], 1.0), (3, 8, 8, 1, [65, 1, 7], 0.1), (4, 72, 40, 2, [129, 300], 1.0),
                                                        (2, 64, 64, 2, [3, 127, 513], 30.0), (1, 16, 120, 1, [64], 1e4)])
def test_mamba2_prompts_as_products(ops, monkeypatch, heads, P, N, groups, lens, span):
    """The product form against the recurrence (which a step that does not say its longest prompt takes): the same
    convolution, so the states differ by the order of 32-bit sums (up to N + 128 terms and as many products, in rms
    about 1e-6) and the outputs by that and one bfloat16 rounding.  ``span``: how far the decays reach."""
    T, B, inner, ch = sum(lens), len(lens), heads * P, heads * P + 2 * groups * N
    proj, dt = rnd(T, inner + ch, dt=torch.bfloat16), rnd(T, heads, seed=1)
    small = [rnd(ch, 4, s=0.3, seed=2), rnd(ch, s=0.1, seed=3), rnd(heads, seed=4) - 2, rnd(heads, s=0.5, seed=5) + math.log(span), rnd(heads, seed=6)]
    norm = rnd(inner, s=0.1, seed=7) + 1
    first = rnd(B + 1, ops.mamba2_state_size(heads, P, N, groups, 4), seed=8)
    starts = torch.tensor([sum(lens[:i]) for i in range(B + 1)], dtype=torch.int32, device="cuda")
    seq = torch.repeat_interleave(torch.arange(B), torch.tensor(lens)).to("cuda", torch.int32)
    slots = torch.arange(B, 0, -1, dtype=torch.int32, device="cuda")
    got, ran = [], recorded(ops, monkeypatch)
    for longest in (0, max(lens)):
        state = first.clone()
        out = ops.mamba2(proj, dt, heads, P, N, groups, 4, 1, *small, norm, 1e-6, state, starts, seq, slots, B, False, longest)
        got.append((out.double(), state.double()))
    assert ran.count("mamba2_scan") == 1 and ran.count("mamba2_prompts") == 1                       # each form once
    assert torch.equal(got[0][1][0], got[1][1][0])                       # a slot that is not in the step
    assert (got[1][1] - got[0][1]).norm() <= 3e-6 * got[0][1].norm()
    assert (got[1][0] - got[0][0]).norm() <= 3e-3 * got[0][0].norm()
    assert torch.isfinite(got[1][0]).all()


@pytest.mark.parametrize("bad", [math.nan, math.inf, -math.inf])
@pytest.mark.parametrize("at", [0, 17, 127, 128, 200])
def test_mamba2_prompts_stay_causal(ops, bad, at):
    """A number that is not finite in one token's x of one channel: the tokens before it give what they give without it,
    and a NaN shows wherever the recurrence shows it."""
    heads, P, N, groups, lens = 2, 64, 64, 1, [230, 40]
    T, B, inner, ch = sum(lens), len(lens), heads * P, heads * P + 2 * groups * N
    proj, dt = rnd(T, inner + ch, dt=torch.bfloat16), rnd(T, heads, seed=1)
    small = [rnd(ch, 4, s=0.3, seed=2), rnd(ch, s=0.1, seed=3), rnd(heads, seed=4) - 2, rnd(heads, s=0.5, seed=5), rnd(heads, seed=6)]
    norm = rnd(inner, s=0.1, seed=7) + 1
    first = rnd(B, ops.mamba2_state_size(heads, P, N, groups, 4), seed=8)
    starts, slots = torch.tensor([0, lens[0], T], dtype=torch.int32, device="cuda"), torch.arange(B, dtype=torch.int32, device="cuda")
    seq = torch.repeat_interleave(torch.arange(B), torch.tensor(lens)).to("cuda", torch.int32)

    def run(rows, longest):
        state = first.clone()
        return ops.mamba2(rows, dt, heads, P, N, groups, 4, 1, *small, norm, 1e-6, state, starts, seq, slots, B, False, longest)
    clean, spoilt = run(proj, max(lens)), proj.clone()
    spoilt[at, inner + 5] = bad
    got, scan = run(spoilt, max(lens)), run(spoilt, 0)
    assert torch.equal(got[:at], clean[:at]) and torch.equal(got[lens[0]:], clean[lens[0]:])
    if math.isnan(bad):
        assert torch.equal(got.isnan(), scan.isnan())


@pytest.mark.parametrize("bad", [math.nan, math.inf, -math.inf])
@pytest.mark.parametrize("at", [0, 13, 16, 150])
def test_gla_prompts_stay_causal(ops, bad, at):
    """The same of gated linear attention, a value that is not finite."""
    heads, D, V, rank, lens = 2, 64, 128, 16, [170, 30]
    T, B = sum(lens), len(lens)
    proj, low = rnd(T, 2 * heads * (D + V), dt=torch.bfloat16), rnd(1, T, rank, seed=1)
    a2, bias, norm = rnd(heads * D, rank, s=0.3, seed=2), rnd(heads * D, seed=3) + 2, rnd(V, s=0.1, seed=4) + 1
    first = rnd(B, heads * D * V, seed=5)
    starts, slots = torch.tensor([0, lens[0], T], dtype=torch.int32, device="cuda"), torch.arange(B, dtype=torch.int32, device="cuda")
    seq = torch.repeat_interleave(torch.arange(B), torch.tensor(lens)).to("cuda", torch.int32)

    def run(rows, longest):
        state = first.clone()
        return ops.gla(rows, low, a2, bias, 8.0, D ** -0.5, norm, 1e-6, heads, D, V, state, starts, seq, slots, B, longest)
    clean, spoilt = run(proj, max(lens)), proj.clone()
    spoilt[at, 2 * heads * D + V + 9] = bad
    got, scan = run(spoilt, max(lens)), run(spoilt, 0)
    assert torch.equal(got[:at], clean[:at]) and torch.equal(got[lens[0]:], clean[lens[0]:])
    if math.isnan(bad):
        assert torch.equal(got.isnan(), scan.isnan())


@pytest.mark.parametrize("heads,D,V,lens,span", [(8, 128, 256, [700, 15], 1.0), (2, 72, 128, [16, 33, 1], 0.01), (3, 64, 128, [32], 30.0),
                                                 (1, 8, 144, [300, 257], 1.0), (2, 128, 256, [65], 1e3)])
def test_gla_prompts_in_blocks(ops, monkeypatch, heads, D, V, lens, span):
    """The block form against the recurrence (which a step that does not say its longest prompt takes): states by the
    order of 32-bit sums, outputs by that and one bfloat16 rounding.  ``span``: how far the decays reach."""
    monkeypatch.setattr(ops, "GLA_BLOCKS_FROM", 1)                       # also where the recurrence is the faster one
    T, B, rank = sum(lens), len(lens), 16
    proj, low = rnd(T, 2 * heads * (D + V), dt=torch.bfloat16), rnd(1, T, rank, seed=1)
    a2, bias, norm = rnd(heads * D, rank, s=0.3, seed=2), rnd(heads * D, seed=3) + 2, rnd(V, s=0.1, seed=4) + 1
    first = rnd(B + 1, heads * D * V, seed=5)
    starts = torch.tensor([sum(lens[:i]) for i in range(B + 1)], dtype=torch.int32, device="cuda")
    seq = torch.repeat_interleave(torch.arange(B), torch.tensor(lens)).to("cuda", torch.int32)
    slots = torch.arange(B, 0, -1, dtype=torch.int32, device="cuda")
    got, ran = [], recorded(ops, monkeypatch)
    for longest in (0, max(lens)):
        state = first.clone()
        out = ops.gla(proj, low, a2, bias, 8.0 / span, D ** -0.5, norm, 1e-6, heads, D, V, state, starts, seq, slots, B, longest)
        got.append((out.double(), state.double()))
    assert ran.count("gla_scan") == 1 and ran.count("gla_blocks") == 1                       # each form once
    assert torch.equal(got[0][1][0], got[1][1][0])                       # a slot that is not in the step
    assert (got[1][1] - got[0][1]).norm() <= 3e-6 * got[0][1].norm()
    assert (got[1][0] - got[0][0]).norm() <= 3e-3 * got[0][0].norm()
    assert torch.isfinite(got[1][0]).all()


# sequences, heads, latent, rotary, rows, window
LATENT_CLUSTERS = [(1, 5, 64, 16, 33, 0), (1, 16, 448, 64, 700, 0), (3, 20, 96, 0, 500, 0), (8, 16, 512, 64, 900, 0),
                   (40, 16, 128, 64, 300, 0), (40, 3, 448, 64, 640, 200), (2, 33, 512, 512, 130, 0)]


@pytest.mark.parametrize("B,heads,C,R,longest,window", LATENT_CLUSTERS)
def test_latent_decode_pieces(ops, B, heads, C, R, longest, window):
    """Keys cut for clusters (alone, two, four, eight), heads and rows that fill no tile, one to two tiles a ring.  The pool
    holds NaN wherever no key of the step lies.  Weights and result are rounded to bfloat16 once each."""
    KD, lens = C + R, [max(1, longest - 37 * b % longest) for b in range(B)]
    pages = (longest + PAGE - 1) // PAGE
    pool = torch.full((B * pages, 1, PAGE, KD), float("nan"), dtype=torch.bfloat16, device="cuda")
    table = torch.arange(B * pages, dtype=torch.int32, device="cuda").flip(0).view(B, pages).contiguous()
    q, sink, rows = rnd(B, heads * KD, dt=torch.bfloat16), rnd(heads, seed=1), rnd(B, longest, KD, dt=torch.bfloat16, seed=2)
    want = torch.empty(B, heads * C, dtype=torch.float64, device="cuda")
    for b, n in enumerate(lens):
        first = max(0, n - window) if window else 0
        view = pool[table[b].long()].reshape(-1, KD)
        view[first:n] = rows[b, first:n]
        pool[table[b].long()] = view.view(pages, 1, PAGE, KD)
        k = rows[b, first:n].double()
        s = torch.cat([q[b].double().view(heads, KD) @ k.T * 0.1, sink.double()[:, None]], -1)
        want[b] = (torch.softmax(s, -1)[:, :-1] @ k[:, :C]).reshape(-1)
    got = ops.latent_decode(q, pool, table, torch.tensor(lens, dtype=torch.int32, device="cuda"), sink, heads, C, R, 0.1, longest, window)
    assert (got.double() - want).norm() <= 4e-3 * want.norm()
    assert ops.kernel_errors() == {}


def state_error(state, want):
    return float((state.double() - want).norm() / want.norm())


@pytest.mark.parametrize("n,B,heads,N,log_a", [(100, 1, 4, 128, 0.0), (300, 2, 3, 64, 0.0), (2048, 1, 2, 128, -2.0), (1000, 2, 2, 128, -8.0)])
def test_mamba2_products_lose_nothing_in_the_state(ops, n, B, heads, N, log_a):
    """The 32-bit state against 64 bits: as near as the recurrence leaves it (a fifth more: both are sums of the same
    roundings in another order), also where decays are close to 1 and all terms have one sign, so that sums which are cut
    off would show.  The convolution copies numbers of 32 to 64, which silu leaves as they are."""
    P, T, inner, ch = 64, n * B, heads * 64, heads * 64 + 2 * N
    g = torch.Generator(device="cuda").manual_seed(n + N)
    proj, dt = (torch.rand(T, inner + ch, device="cuda", generator=g) * 31 + 32).bfloat16(), rnd(T, heads, seed=1)
    taps = torch.tensor([0.0, 0.0, 0.0, 1.0], device="cuda").repeat(ch, 1)
    small = [taps, torch.zeros(ch, device="cuda"), rnd(heads, seed=4) - 2, rnd(heads, s=0.5, seed=5) + log_a, rnd(heads, seed=6)]
    starts, slots = torch.arange(0, T + 1, n, dtype=torch.int32, device="cuda"), torch.arange(B, dtype=torch.int32, device="cuda")
    seq = torch.arange(B, device="cuda").repeat_interleave(n).to(torch.int32)
    x, Bm = (t.double().view(B, n, -1) for t in (proj[:, inner:2 * inner], proj[:, 2 * inner:2 * inner + N]))
    step = torch.nn.functional.softplus(dt.double() + small[2].double()).view(B, n, heads)
    decay = torch.exp(-torch.exp(small[3].double()) * step)
    S = torch.zeros(B, heads, P, N, dtype=torch.float64, device="cuda")
    for t in range(n):
        S = decay[:, t, :, None, None] * S + (step[:, t, :, None] * x[:, t].view(B, heads, P))[..., None] * Bm[:, t, None, None]
    err = []
    for longest in (0, n):
        state = torch.zeros(B, ops.mamba2_state_size(heads, P, N, 1, 4), device="cuda")
        ops.mamba2(proj, dt, heads, P, N, 1, 4, 1, *small, torch.ones(inner, device="cuda"), 1e-6, state, starts, seq, slots, B, False, longest)
        err.append(state_error(state[:, :heads * P * N].view(B, heads, P, N), S))
    assert err[1] <= 1.2 * err[0], err


def test_mamba2_prompts_do_not_depend_on_the_step(ops):
    """A sequence alone and beside others, where a thread of the convolution takes two tokens and eight: the same bits."""
    heads, P, N, lens = 64, 64, 128, [400, 30, 41]
    T, inner, ch = sum(lens), heads * P, heads * P + 2 * N
    proj, dt = rnd(T, inner + ch, dt=torch.bfloat16), rnd(T, heads, seed=1)
    small = [rnd(ch, 4, s=0.3, seed=2), rnd(ch, s=0.1, seed=3), rnd(heads, seed=4) - 2, rnd(heads, s=0.5, seed=5), rnd(heads, seed=6)]
    norm, first = rnd(inner, s=0.1, seed=7) + 1, rnd(3, ops.mamba2_state_size(heads, P, N, 1, 4), seed=8)

    def run(which):
        n = [lens[i] for i in which]
        rows = torch.cat([torch.arange(sum(lens[:i]), sum(lens[:i + 1])) for i in which]).cuda()
        starts = torch.tensor([sum(n[:i]) for i in range(len(n) + 1)], dtype=torch.int32, device="cuda")
        seq = torch.repeat_interleave(torch.arange(len(n)), torch.tensor(n)).to("cuda", torch.int32)
        state, slots = first.clone(), torch.tensor(which, dtype=torch.int32, device="cuda")
        out = ops.mamba2(proj[rows], dt[rows], heads, P, N, 1, 4, 1, *small, norm, 1e-6, state, starts, seq, slots, len(n), False, 400)
        return out, state[which]
    out, state = run([0, 1, 2])
    for i in range(3):
        alone = run([i])
        assert torch.equal(alone[0], out[sum(lens[:i]):sum(lens[:i + 1])]) and torch.equal(alone[1][0], state[i])


@pytest.mark.parametrize("layer", ["mamba2", "gla"])
def test_prompts_take_the_form_with_less_scratch_where_memory_is_short(ops, monkeypatch, layer):
    """No memory for the states between the chunks: the recurrence, which needed little before and still does, to the
    last bit."""
    heads, lens = 8, [700, 40]
    T, B = sum(lens), len(lens)
    starts = torch.tensor([0, lens[0], T], dtype=torch.int32, device="cuda")
    seq = torch.repeat_interleave(torch.arange(B), torch.tensor(lens)).to("cuda", torch.int32)
    slots, real = torch.arange(B, dtype=torch.int32, device="cuda"), torch.empty
    if layer == "mamba2":
        P = N = 64
        inner, ch = heads * P, heads * P + 2 * N
        proj, dt = rnd(T, inner + ch, dt=torch.bfloat16), rnd(T, heads, seed=1)
        small = [rnd(ch, 4, s=0.3, seed=2), rnd(ch, s=0.1, seed=3), rnd(heads, seed=4) - 2, rnd(heads, s=0.5, seed=5), rnd(heads, seed=6)]
        state, limit, at = torch.zeros(B, ops.mamba2_state_size(heads, P, N, 1, 4), device="cuda"), 7 * heads * P * N, "MAMBA2_PRODUCTS_FROM"
        run = lambda: ops.mamba2(proj, dt, heads, P, N, 1, 4, 1, *small, torch.ones(inner, device="cuda"), 1e-6, state.zero_(), starts, seq, slots, B, False, 700)
    else:
        D, V = 128, 256
        proj, low = rnd(T, 2 * heads * (D + V), dt=torch.bfloat16), rnd(1, T, 16, seed=1)
        a2, bias = rnd(heads * D, 16, s=0.3, seed=2), rnd(heads * D, seed=3) + 2
        state, limit, at = torch.zeros(B, heads * D * V, device="cuda"), 3 * heads * D * V, "GLA_BLOCKS_FROM"
        run = lambda: ops.gla(proj, low, a2, bias, 8.0, D ** -0.5, torch.ones(V, device="cuda"), 1e-6, heads, D, V, state.zero_(), starts, seq, slots, B, 700)

    def short(*size, **kw):                                              # (the chunks' states are asked for as one row of numbers)
        if isinstance(size[0], int) and size[0] >= limit:
            raise torch.OutOfMemoryError("none left")
        return real(*size, **kw)
    with monkeypatch.context() as m:
        m.setattr(ops, at, 1 << 30)
        scans = [run(), state.clone()]
    with monkeypatch.context() as m:
        m.setattr(torch, "empty", short)
        got = [run(), state.clone()]
    assert torch.equal(got[0], scans[0]) and torch.equal(got[1], scans[1])
    run()
    assert not torch.equal(state, scans[1])                              # with memory: the other form, whose sums are in another order


def device_time(call, reps=20):
    """Least time of ``reps`` calls in a row, of five tries, in ms."""
    best = math.inf
    for _ in range(5):
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        call()
        begin.record()
        for _ in range(reps):
            call()
        end.record()
        torch.cuda.synchronize()
        best = min(best, begin.elapsed_time(end))
    return best


@pytest.mark.parametrize("lens", [[64] + 63 * [5], [64] + 15 * [5], [8 + 7 * i % 57 for i in range(64)], [300] + 31 * [9]])
def test_mamba2_short_prompts_are_not_slower_than_the_recurrence(ops, monkeypatch, lens):
    """Many short prompts in a step whose longest one asks for the product form: no state goes through scratch for them,
    and the step takes at most a quarter more than the recurrence (five times as much before)."""
    heads, P, N = 64, 64, 128
    T, B, inner, ch = sum(lens), len(lens), heads * P, heads * P + 2 * N
    proj, dt = rnd(T, inner + ch, dt=torch.bfloat16), rnd(T, heads, seed=1)
    small = [rnd(ch, 4, s=0.3, seed=2), rnd(ch, s=0.1, seed=3), rnd(heads, seed=4) - 2, rnd(heads, s=0.5, seed=5), rnd(heads, seed=6)]
    starts = torch.tensor([sum(lens[:i]) for i in range(B + 1)], dtype=torch.int32, device="cuda")
    seq = torch.repeat_interleave(torch.arange(B), torch.tensor(lens)).to("cuda", torch.int32)
    slots = torch.arange(B, dtype=torch.int32, device="cuda")
    state, norm = torch.zeros(B, ops.mamba2_state_size(heads, P, N, 1, 4), device="cuda"), torch.ones(inner, device="cuda")
    times = []
    for least in (ops.MAMBA2_PRODUCTS_FROM, 1 << 30):
        monkeypatch.setattr(ops, "MAMBA2_PRODUCTS_FROM", least)
        times.append(device_time(lambda: ops.mamba2(proj, dt, heads, P, N, 1, 4, 1, *small, norm, 1e-6, state, starts, seq, slots, B, False, max(lens))))
    assert times[0] <= 1.25 * times[1], times


@pytest.mark.parametrize("n,B,heads,bias", [(100, 1, 4, 0.0), (100, 2, 4, 2.0), (2048, 1, 4, 0.0), (2048, 1, 4, 6.0), (2048, 16, 10, 10.0)])
def test_gla_blocks_lose_nothing_in_the_state(ops, n, B, heads, bias):
    """The same of gated linear attention, prompts in several chunks and (16 of them) in one.  ``bias`` 10: decays of 0.99999."""
    D, V, rank, T = 64, 128, 16, n * B
    proj, low = rnd(T, 2 * heads * (D + V), dt=torch.bfloat16).abs(), rnd(1, T, rank, seed=1)
    a2, b2 = rnd(heads * D, rank, s=0.3, seed=2), rnd(heads * D, seed=3) + bias
    starts, slots = torch.arange(0, T + 1, n, dtype=torch.int32, device="cuda"), torch.arange(B, dtype=torch.int32, device="cuda")
    seq = torch.arange(B, device="cuda").repeat_interleave(n).to(torch.int32)
    k, v = (t.double().reshape(B, n, heads, -1) for t in (proj[:, heads * D:2 * heads * D], proj[:, 2 * heads * D:2 * heads * D + heads * V]))
    decay = torch.exp(torch.nn.functional.logsigmoid(low[0].double() @ a2.double().T + b2.double()) / 8.0).view(B, n, heads, D)
    S = torch.zeros(B, heads, D, V, dtype=torch.float64, device="cuda")
    for t in range(n):
        S = decay[:, t, :, :, None] * S + k[:, t, :, :, None] * v[:, t, :, None, :]
    err = []
    for longest in (0, n):
        state = torch.zeros(B, heads * D * V, device="cuda")
        ops.gla(proj, low, a2, b2, 8.0, D ** -0.5, torch.ones(V, device="cuda"), 1e-6, heads, D, V, state, starts, seq, slots, B, longest)
        err.append(state_error(state.view(B, heads, D, V), S))
    assert err[1] <= 1.2 * err[0], err


# sequences, heads, latent, rotary, bucket of rows, window, sink
LATENT_FOLDED = [(1, 16, 448, 64, 4096, 0, True), (3, 16, 448, 64, 4096, 0, False), (8, 5, 64, 16, 8192, 0, True), (1, 33, 96, 32, 8192, 0, True),
                 (40, 16, 448, 64, 2048, 0, True), (10, 16, 512, 64, 4096, 3000, False), (12, 20, 128, 0, 4096, 0, True)]


@pytest.mark.parametrize("B,heads,C,R,bucket,window,has_sink", LATENT_FOLDED)
def test_latent_decode_pieces_that_a_launch_folds(ops, monkeypatch, B, heads, C, R, bucket, window, has_sink):
    """More pieces than a cluster takes, and contexts from one row up to the bucket's last: pieces without a key."""
    KD, lens, ran = C + R, [[bucket, 1, bucket // 2, 33, 64, bucket - 31, 700][b % 7] for b in range(B)], []
    pages = (bucket + PAGE - 1) // PAGE
    pool = torch.full((B * pages, 1, PAGE, KD), float("nan"), dtype=torch.bfloat16, device="cuda")
    table = torch.arange(B * pages, dtype=torch.int32, device="cuda").flip(0).view(B, pages).contiguous()
    q, rows = rnd(B, heads * KD, dt=torch.bfloat16), rnd(B, bucket, KD, dt=torch.bfloat16, seed=2)
    sink = rnd(heads, seed=1) if has_sink else None
    want = torch.empty(B, heads * C, dtype=torch.float64, device="cuda")
    for b, n in enumerate(lens):
        first = max(0, n - window) if window else 0
        view = pool[table[b].long()].reshape(-1, KD)
        view[first:n] = rows[b, first:n]
        pool[table[b].long()] = view.view(pages, 1, PAGE, KD)
        k = rows[b, first:n].double()
        s = q[b].double().view(heads, KD) @ k.T * 0.1
        if has_sink:
            s = torch.cat([s, sink.double()[:, None]], -1)
        want[b] = (torch.softmax(s, -1)[:, :n - first] @ k[:, :C]).reshape(-1)
    check = ops._check
    monkeypatch.setattr(ops, "_check", lambda lib, status, what, kernels=1: (ran.append((what, kernels)), check(lib, status, what, kernels))[1])
    got = ops.latent_decode(q, pool, table, torch.tensor(lens, dtype=torch.int32, device="cuda"), sink, heads, C, R, 0.1, bucket, window)
    assert ran == [("latent_decode_mma", 2)]                             # (with the launch that folds)
    assert (got.double() - want).norm() <= 4e-3 * want.norm()
    assert ops.kernel_errors() == {}


@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (8, 17, 60), (9, 16, 2048), (16, 1100, 4100), (17, 63, 256), (65, 65, 2052), (70, 130, 8196)])
def test_gemm_simt_rows_and_tiles(ops, M, N, K):
    """32-bit operands in whole 16-byte pieces: rows that are not full, tails of a k-tile, stage and segment; a row is
    the same alone (the rows kernel) as among the others (the tiles kernel from 17 rows on)."""
    a, w = rnd(M, K, s=0.5), rnd(N, K, s=0.5, seed=1)
    want = a.double() @ w.double().T
    got = ops.gemm_simt(a, w, torch.float32)
    close(got, want, torch.float32, scale=math.sqrt(K))
    close(ops.gemm_simt(a, w, torch.bfloat16, softcap=3.0, out_scale=0.5), 1.5 * torch.tanh(want / 3.0), torch.bfloat16, scale=4.0)
    i = M - 1
    assert torch.equal(got[i:i + 1], ops.gemm_simt(a[i:i + 1].contiguous(), w, torch.float32))


@pytest.mark.parametrize("odt", DT)
@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (3, 40, 72), (16, 384, 96), (17, 130, 64), (64, 2304, 2048),
                                   (100, 512, 520), (128, 256, 64), (129, 256, 64), (300, 520, 200),
                                   (1000, 301 * 8, 1032), (2048, 1024, 2304), (2048, 10240, 128)])
@pytest.mark.parametrize("pair", [0, 1])
def test_gemm_tc(ops, odt, M, N, K, pair):
    """Few tokens (swapped tiles), many tokens on single SMs and on pairs of SMs (one tile a pair, and several)."""
    if pair and (M <= 128 or N < 256):
        pytest.skip("the pair kernel takes more than 128 tokens and at least 256 weight rows")
    a, w = rnd(M, K, dt=torch.bfloat16, s=0.5), rnd(N, K, dt=torch.bfloat16, s=0.5, seed=1)
    assert ops.gemm_tc_takes(a, w)
    want = a.double() @ w.double().T
    was = ops.gemm_tc_set_pair(pair)
    try:
        got = ops.gemm_tc(a, w, odt)
    finally:
        ops.gemm_tc_set_pair(was)
    torch.cuda.synchronize()
    assert ops.gemm_tc_error() == 0
    if odt == torch.float32:
        assert float((got.double() - want).norm() / want.norm()) < 2e-5
    else:
        assert float((got.double() - want).norm() / want.norm()) < 4e-3


# tokens, weight rows, K and the form that the cost picks on 148 SMs (1000 x CTAs a tile + columns, + 100000 for pairs)
GEMM_FORMS = [(300, 300, 64, 1128), (1500, 2400, 1032, 1256), (129, 520, 1040, 4128), (200, 2300, 2040, 3128), (300, 2304, 2048, 2128),
              (300, 3584, 14336, 3256), (257, 2304, 9216, 4256), (700, 2300, 2040, 101128), (1500, 2304, 2048, 101192),
              (1000, 3580, 4088, 101224), (2047, 2304, 2048, 101256), (513, 18432, 136, 1256)]


@pytest.mark.parametrize("M,N,K,form", GEMM_FORMS)
def test_gemm_tc_forms(ops, M, N, K, form):
    """Every form of a product of many tokens at sizes with remainders: 32-bit and bfloat16 results, the gate where the
    rows allow it, a cap, and a result whose rows are not whole 16-byte pieces.  32-bit: sums of K products of which each
    is exact; bfloat16: one rounding."""
    from trapetum_b200.csrc import build
    if ops.sm_count() == 148:
        assert build.load("gemm_tc").tb_gemm_tc_form(M, N, K, 148) == form
    a, w = rnd(M, K, dt=torch.bfloat16, s=0.5), rnd(N, K, dt=torch.bfloat16, s=0.5, seed=1)
    want = a.double() @ w.double().T
    off = torch.full((M, N + 3), 7.0, device="cuda")
    for got, truth, tol in ((ops.gemm_tc(a, w, torch.float32), want, 2e-5), (ops.gemm_tc(a, w, torch.bfloat16), want, 4e-3),
                            (ops.gemm_tc(a, w, torch.float32, 20.0), 20 * torch.tanh(want / 20), 2e-5),
                            (ops.gemm_tc(a, w, torch.float32, out=off[:, 1:N + 1]), want, 2e-5)):
        assert float((got.double() - truth).norm() / truth.norm()) < tol
    assert bool((off[:, 0] == 7).all() and (off[:, N + 1:] == 7).all())
    if N % 32 == 0:
        blocks = want.view(M, N // 32, 2, 16)
        gated = (torch.nn.functional.silu(blocks[:, :, 0]) * blocks[:, :, 1]).reshape(M, N // 2)
        got = ops.gemm_tc(a, w, torch.bfloat16, gated_act="silu")
        assert float((got.double() - gated).norm() / gated.norm()) < 4e-3
    assert ops.gemm_tc_error() == 0


@pytest.mark.parametrize("M,N,K,splits", [(8, 2304, 2048, 8), (64, 640, 9216, 5), (1, 136, 1024, 16), (33, 100 * 8, 520, 3)])
def test_gemm_tc_split_k(ops, M, N, K, splits):
    a, w = rnd(M, K, dt=torch.bfloat16, s=0.5), rnd(N, K, dt=torch.bfloat16, s=0.5, seed=1)
    want = a.double() @ w.double().T
    got = ops.gemm_tc(a, w, torch.float32, 0.0, splits)
    again = ops.gemm_tc(a, w, torch.float32, 0.0, splits)
    assert torch.equal(got, again)                                  # fixed summation order
    assert float((got.double() - want).norm() / want.norm()) < 2e-5
    capped = ops.gemm_tc(a, w, torch.float32, 5.0, splits)
    assert float((capped.double() - 5 * torch.tanh(want / 5)).abs().max()) < 1e-4
    assert ops.gemm_tc_error() == 0


@pytest.mark.parametrize("act", ["gelu_tanh", "silu"])
@pytest.mark.parametrize("M,I,K", [(1, 160, 96), (8, 9216, 2304), (40, 128, 64), (64, 1024, 512), (128, 176, 72),
                                   (129, 160, 96), (700, 1296, 520), (2048, 2048, 256)])
@pytest.mark.parametrize("pair", [0, 1])
def test_gemm_tc_gated_epilogue(ops, act, M, I, K, pair):
    """act(x Wg^T) * (x Wu^T) in the product's epilogue, swapped tiles (few tokens) and token-major ones, these on
    single SMs and on pairs."""
    if pair and M <= 128:
        pytest.skip("the pair kernel takes more than 128 tokens")
    x = rnd(M, K, dt=torch.bfloat16, s=1.0)
    wg, wu = rnd(I, K, dt=torch.bfloat16, s=0.1, seed=1), rnd(I, K, dt=torch.bfloat16, s=0.1, seed=2)
    g, u = x.double() @ wg.double().T, x.double() @ wu.double().T
    want = (plain.gelu_tanh(g) if act == "gelu_tanh" else g * torch.sigmoid(g)) * u
    was = ops.gemm_tc_set_pair(pair)
    try:
        got = ops.gemm_tc(x, ops.interleave_gate_up(wg, wu), torch.bfloat16, gated_act=act)
    finally:
        ops.gemm_tc_set_pair(was)
    assert got.shape == (M, I) and got.dtype == torch.bfloat16
    assert float((got.double() - want).norm() / want.norm()) < 4e-3
    assert ops.gemm_tc_error() == 0


def test_gemm_tc_pair_policy_and_cap(ops):
    """The default policy sends a long product to pairs of SMs and a short one to single SMs; either way the result
    is the same up to the order of additions inside an instruction, with a soft cap and through a row-strided view."""
    big = rnd(2048, 2 * 4096, dt=torch.bfloat16, s=0.5)
    a = big[:, 4096:]                                                # row stride 8192
    w = rnd(16384 + 8, 4096, dt=torch.bfloat16, s=0.05, seed=1)      # 8 x 65 tiles of 64 k-blocks: long enough for the pair
    want = 5 * torch.tanh(a.double() @ w.double().T / 5)
    outs = []
    for mode in (0, 1, 2):
        was = ops.gemm_tc_set_pair(mode)
        try:
            outs.append(ops.gemm_tc(a, w, torch.float32, 5.0))
        finally:
            ops.gemm_tc_set_pair(was)
    assert was == 2                                                  # the default
    for got in outs:
        assert float((got.double() - want).abs().max()) < 1e-4
    assert torch.equal(outs[2], outs[1])                             # where the pair pays
    short = rnd(520, 64, dt=torch.bfloat16, s=0.5, seed=2)
    x = rnd(300, 64, dt=torch.bfloat16, s=0.5, seed=3)
    ops.gemm_tc_set_pair(0)
    try:
        single = ops.gemm_tc(x, short, torch.float32)
    finally:
        ops.gemm_tc_set_pair(2)
    assert torch.equal(ops.gemm_tc(x, short, torch.float32), single)  # a short product stays on single SMs
    assert ops.gemm_tc_error() == 0


def test_gemm_tc_views_and_refusals(ops):
    big = rnd(40, 3 * 256, dt=torch.bfloat16, s=0.5)
    w = rnd(96, 256, dt=torch.bfloat16, s=0.5, seed=1)
    a = big[:, 256:512]                                              # a column slice: row stride 768
    got = ops.gemm_tc(a, w, torch.float32)
    assert float((got.double() - a.double() @ w.double().T).abs().max()) < 1e-3
    assert not ops.gemm_tc_takes(rnd(4, 100, dt=torch.bfloat16), rnd(8, 100, dt=torch.bfloat16))   # K % 8
    assert not ops.gemm_tc_takes(rnd(4, 64), rnd(8, 64))                                         # float32
    with pytest.raises(ops.KernelError, match="does not take"):
        ops.gemm_tc(rnd(4, 100, dt=torch.bfloat16), rnd(8, 100, dt=torch.bfloat16), torch.float32)


def test_gemm_tc_token_rows_do_not_depend_on_the_batch(ops):
    """The same token row gives the same bits alone (swapped tiles) and among 40 rows."""
    a, w = rnd(40, 512, dt=torch.bfloat16, s=0.5), rnd(384, 512, dt=torch.bfloat16, s=0.5, seed=1)
    full = ops.gemm_tc(a, w, torch.float32, splits=1)
    one = ops.gemm_tc(a[7:8].contiguous(), w, torch.float32, splits=1)
    assert torch.equal(full[7:8], one)


# ---------------------------------------------------------------------------
def paged(k, v, lens, ring_rows, n_pages, seed=0):
    """Scatter dense per-sequence k, v ([len, nkv, hd] each) into scrambled pages; untouched rows are NaN."""
    nkv, hd = k[0].shape[1:]
    dt = k[0].dtype
    kp = torch.full((n_pages, nkv, PAGE, hd), float("nan"), dtype=dt, device="cuda")
    vp = torch.full((n_pages, nkv, PAGE, hd), float("nan"), dtype=dt, device="cuda")
    perm = torch.randperm(n_pages, generator=torch.Generator().manual_seed(seed)).tolist()
    width = max((min(n, ring_rows) if ring_rows else n) + PAGE - 1 for n in lens) // PAGE
    table = torch.zeros(len(lens), width, dtype=torch.int32)
    for b, n in enumerate(lens):
        rows = min(n, ring_rows) if ring_rows else n
        for pg in range((rows + PAGE - 1) // PAGE):
            table[b, pg] = perm.pop()
        for p in range(max(0, n - ring_rows) if ring_rows else 0, n):
            r = p % ring_rows if ring_rows else p
            page = int(table[b, r // PAGE])
            kp[page, :, r % PAGE, :] = k[b][p]
            vp[page, :, r % PAGE, :] = v[b][p]
    return kp, vp, table.cuda()


def ref_attention_one(q, k, v, scale, cap, window):
    """q [nh, hd] at position len-1 against k, v [len, nkv, hd] -> [nh, hd] (float64)."""
    n, nkv, hd = k.shape
    nh = q.shape[0]
    out = torch.zeros(nh, hd, dtype=torch.float64)
    lo = max(0, n - window) if window else 0
    for h in range(nh):
        kh = h // (nh // nkv)
        s = (k[lo:, kh].double() @ q[h].double()) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        p = torch.softmax(s, 0)
        out[h] = p @ v[lo:, kh].double()
    return out


def decode_impls(ops, dt, nh, nkv, hd):
    """The generic kernel always; the bulk-copy kernel too where it takes the shape."""
    import functools
    impls = [ops.attn_decode_simt]
    if ops.attn_decode_takes(dt, nh, nkv, hd):
        impls.append(ops.attn_decode_tma)
        if ops.attn_decode_stream_takes(dt, nh, nkv, hd, 64):
            # the stream partition, with CTA counts that leave parts of a sequence to several CTAs, one page to
            # each CTA (more CTAs than pages), and everything to one CTA; `splits` is not used by it
            for n_ctas in (None, 7, 1, 1000):
                def stream(q, kp, vp, table, la, nh, nkv, hd, scale, cap, window, ring, splits, n_ctas=n_ctas):
                    return ops.attn_decode_stream(q, kp, vp, table, la, nh, nkv, hd, scale, cap, window, ring, n_ctas)
                stream.__name__ = f"attn_decode_stream[{n_ctas}]"
                impls.append(stream)
        if nh // nkv in (1, 2, 4, 8):
            lanes = functools.partial(ops.attn_decode_tma, variant="lanes")
            lanes.__name__ = "attn_decode_lanes"
            impls.append(lanes)
    return impls


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("nh,nkv,hd,cap,window,splits", [
    (4, 2, 16, 50.0, 0, 1), (6, 1, 32, 0.0, 40, 3), (3, 3, 48, 20.0, 70, 2), (8, 4, 256, 50.0, 0, 4),
    (5, 5, 80, 0.0, 128, 7), (8, 2, 128, 30.0, 100, 1), (8, 1, 64, 10.0, 0, 2), (4, 4, 32, 0.0, 64, 5),
    (16, 2, 256, 50.0, 200, 3), (2, 1, 128, 0.0, 0, 9), (8, 8, 64, 0.0, 300, 1), (6, 2, 64, 25.0, 90, 2),
    (5, 1, 128, 0.0, 0, 3), (14, 2, 256, 50.0, 0, 2)])
def test_attn_decode(ops, dt, nh, nkv, hd, cap, window, splits):
    lens = [1, 37, 64, 65, 200, 333]
    ring = ((window + PAGE - 1) // PAGE) * PAGE if window else 0
    ks = [rnd(n, nkv, hd, dt=dt, seed=i).cpu() for i, n in enumerate(lens)]
    vs = [rnd(n, nkv, hd, dt=dt, seed=10 + i).cpu() for i, n in enumerate(lens)]
    q = rnd(len(lens), nh * hd, dt=dt, seed=99)
    kp, vp, table = paged([k.cuda() for k in ks], [v.cuda() for v in vs], lens, ring, 64, seed=hd)
    la = torch.tensor(lens, dtype=torch.int32, device="cuda")
    scale = 0.37 / math.sqrt(hd)
    for impl in decode_impls(ops, dt, nh, nkv, hd):
        got = impl(q, kp, vp, table, la, nh, nkv, hd, scale, cap, window, ring, splits)
        assert torch.isfinite(got.float()).all(), f"{impl.__name__}: a row outside the sequence's own keys was read"
        for b, n in enumerate(lens):
            want = ref_attention_one(q[b].view(nh, hd).cpu(), ks[b], vs[b], scale, cap, window)
            close(got[b].view(nh, hd), want, dt, 2.0)
    torch.cuda.synchronize()
    assert ops.attn_decode_error() == 0


@pytest.mark.parametrize("splits", [17, 33, 64, 70])
def test_attn_decode_in_many_pieces(ops, splits):
    """A long sequence cut into many pieces: the fold inside the kernel takes up to 32 pieces at a time and holds
    the weights of 64; more than 64 pieces go to the fold launch."""
    dt, nh, nkv, hd = torch.bfloat16, 4, 2, 64
    lens = [PAGE * 70 + 5, 300]
    ks = [rnd(n, nkv, hd, dt=dt, seed=i).cpu() for i, n in enumerate(lens)]
    vs = [rnd(n, nkv, hd, dt=dt, seed=10 + i).cpu() for i, n in enumerate(lens)]
    q = rnd(len(lens), nh * hd, dt=dt, seed=99)
    kp, vp, table = paged([k.cuda() for k in ks], [v.cuda() for v in vs], lens, 0, 80, seed=3)
    la = torch.tensor(lens, dtype=torch.int32, device="cuda")
    scale = 0.37 / math.sqrt(hd)
    for rep in range(2):                                                # twice: the tickets are used again
        got = ops.attn_decode_tma(q, kp, vp, table, la, nh, nkv, hd, scale, 30.0, 0, 0, splits)
        assert torch.isfinite(got.float()).all()
        for b, n in enumerate(lens):
            want = ref_attention_one(q[b].view(nh, hd).cpu(), ks[b], vs[b], scale, 30.0, 0)
            close(got[b].view(nh, hd), want, dt, 2.0)
    torch.cuda.synchronize()
    assert ops.attn_decode_error() == 0


@pytest.mark.parametrize("nh,nkv,hd,rot,cap,window", [(8, 4, 256, 256, 50.0, 0), (8, 4, 256, 256, 50.0, 128), (6, 2, 64, 32, 0.0, 70),
                                                     (5, 5, 128, 0, 0.0, 0), (14, 2, 256, 64, 30.0, 200), (4, 1, 128, 128, 0.0, 64)])
def test_attn_decode_that_rotates_and_appends_by_itself(ops, nh, nkv, hd, rot, cap, window):
    """Given the partial sums of the q/k/v product, the tensor-core decode kernel must do what the rotation kernel
    followed by the attention kernel does: the same output, and the same new rows in the cache, bit for bit (same
    sums in the same order).  The new token lies on a page's first row, last row and in the middle, among the 16 rows
    of each of the four warps that put it into the page's copy in shared memory; in a ring it overwrites the oldest row."""
    dt = torch.bfloat16
    lens = [1, 64, 65, 200, 333, 128, 21, 175]
    assert {(n - 1) % PAGE // 16 for n in lens} == {0, 1, 2, 3}
    ring = ((window + PAGE - 1) // PAGE) * PAGE if window else 0
    ks = [rnd(n, nkv, hd, dt=dt, seed=i).cpu() for i, n in enumerate(lens)]
    vs = [rnd(n, nkv, hd, dt=dt, seed=10 + i).cpu() for i, n in enumerate(lens)]
    kp, vp, table = paged([k.cuda() for k in ks], [v.cuda() for v in vs], lens, ring, 64, seed=hd)
    la = torch.tensor(lens, dtype=torch.int32, device="cuda")
    B, width = len(lens), (nh + 2 * nkv) * hd
    part = rnd(3, B, width, dt=torch.float32, s=0.6, seed=5)         # three splits of the product
    inv_freq = (1.0 / (10000.0 ** (torch.arange(0, rot, 2, dtype=torch.float32) / rot))).cuda() if rot else None
    pos = (la - 1).contiguous()
    seq = torch.arange(B, dtype=torch.int32, device="cuda")
    scale = 0.37 / math.sqrt(hd)
    # the two-kernel path, on its own copy of the cache
    kp1, vp1 = kp.clone(), vp.clone()
    qkv = torch.empty(B, width, dtype=dt, device="cuda")
    ops.rope_kv(qkv, nh, nkv, hd, rot, inv_freq, pos, seq, la, kp1, vp1, table, ring, part)
    want = ops.attn_decode_tma(qkv[:, :nh * hd], kp1, vp1, table, la, nh, nkv, hd, scale, cap, window, ring, 2)
    runs = [("split 1", lambda k, v: ops.attn_decode_tma(part, k, v, table, la, nh, nkv, hd, scale, cap, window, ring, 1, "mma", (inv_freq, rot))),
            ("split 3", lambda k, v: ops.attn_decode_tma(part, k, v, table, la, nh, nkv, hd, scale, cap, window, ring, 3, "mma", (inv_freq, rot)))]
    for n_ctas in (None, 5, 1, 1000):
        runs.append((f"stream {n_ctas}", lambda k, v, n_ctas=n_ctas: ops.attn_decode_stream(
            part, k, v, table, la, nh, nkv, hd, scale, cap, window, ring, n_ctas, (inv_freq, rot))))
    for name, run in runs:
        kp2, vp2 = kp.clone(), vp.clone()
        got = run(kp2, vp2)
        torch.cuda.synchronize()
        assert torch.isfinite(got.float()).all(), name
        # NaN marks rows that no token has written: equal_nan compares them too
        assert torch.equal(torch.nan_to_num(kp2.float(), nan=-7.0), torch.nan_to_num(kp1.float(), nan=-7.0)), f"{name}: k rows"
        assert torch.equal(torch.nan_to_num(vp2.float(), nan=-7.0), torch.nan_to_num(vp1.float(), nan=-7.0)), f"{name}: v rows"
        close(got, want, dt, 2.0)
    assert ops.attn_decode_error() == 0


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("n", [14, 30, 56])
def test_attn_decode_divides_with_one_rounding(ops, hd, n):
    """n keys of equal score, half of them with the value a and half with the next bfloat16 number b: weights, sums and
    their number are exact and the mean is the midpoint of a and b, so the result is the even one of the two.  The sum
    times a rounded 1 / n passes the midpoint for a third of the a's."""
    nh, nkv, dt = 4, 2, torch.bfloat16
    a = 1.0 + (torch.arange(hd) % 128) / 128.0
    v = torch.stack([a + (i % 2) / 128.0 for i in range(n)])[:, None, :].expand(n, nkv, hd).to(dt)
    assert torch.equal(v.float()[0, 0], a) and torch.equal(v.float()[1, 0], a + 1 / 128)
    kp, vp, table = paged([torch.zeros(n, nkv, hd, dtype=dt).cuda()], [v.cuda()], [n], 0, 4, seed=1)
    la = torch.tensor([n], dtype=torch.int32, device="cuda")
    q = rnd(1, nh * hd, dt=dt)
    want = (a + 1 / 256).to(dt).expand(nh, hd)                          # ties go to the even one
    part = torch.zeros(2, 1, (nh + 2 * nkv) * hd, device="cuda")
    part[0, 0, :nh * hd] = q.float()[0]
    part[1, 0, (nh + nkv) * hd:] = v[n - 1].reshape(-1).float().cuda()
    for name, got in (("split", ops.attn_decode_tma(q, kp, vp, table, la, nh, nkv, hd, 1.0, 0.0, 0, 0, 1)),
                      ("stream", ops.attn_decode_stream(q, kp, vp, table, la, nh, nkv, hd, 1.0, 0.0, 0, 0)),
                      ("fused split", ops.attn_decode_tma(part, kp, vp, table, la, nh, nkv, hd, 1.0, 0.0, 0, 0, 1, "mma", (None, 0))),
                      ("fused stream", ops.attn_decode_stream(part, kp, vp, table, la, nh, nkv, hd, 1.0, 0.0, 0, 0, None, (None, 0)))):
        assert torch.equal(got.view(nh, hd).cpu(), want), name
    assert ops.attn_decode_error() == 0


@pytest.mark.parametrize("dt", DT)
def test_attn_decode_far_key_and_window_edge(ops, dt):
    """One key is made to stand out.  Among hundreds it must win the softmax; one step outside the
    window it must be invisible; on the window's first row it must be seen."""
    nh, nkv, hd, n, W = 2, 1, 32, 500, 128
    ring = 128
    for marked, sees in ((3, "full only"), (n - W - 1, "full only"), (n - W, "both"), (n - 1, "both")):
        k = rnd(n, nkv, hd, dt=dt, s=0.1, seed=marked)
        v = rnd(n, nkv, hd, dt=dt, s=1.0, seed=marked + 1)
        q = rnd(1, nh * hd, dt=dt, s=0.1, seed=7)
        k[marked, 0] = (q.view(nh, hd)[0].float() * 400).to(dt)        # q0 . k_marked is huge
        la = torch.tensor([n], dtype=torch.int32, device="cuda")
        for window, rr in ((0, 0), (W, ring)):
            kp, vp, table = paged([k], [v], [n], rr, 16, seed=1)
            for impl in decode_impls(ops, dt, nh, nkv, hd):
                got = impl(q, kp, vp, table, la, nh, nkv, hd, 1.0, 0.0, window, rr, 3).view(nh, hd)
                visible = window == 0 or sees == "both"
                hit = float((got[0].float() - v[marked, 0].float()).abs().max()) < 2e-2
                assert hit == visible, f"{impl.__name__}: key {marked}, window {window}: expected visible={visible}"


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("nh,nkv,hd,cap,window", [(4, 2, 16, 50.0, 8), (6, 1, 32, 0.0, 16), (3, 3, 48, 20.0, 0),
                                                  (2, 1, 256, 50.0, 50), (4, 4, 112, 0.0, 0), (4, 2, 64, 0.0, 64),
                                                  (2, 2, 128, 30.0, 65), (8, 4, 256, 50.0, 0)])
def test_attn_prefill(ops, dt, nh, nkv, hd, cap, window):
    lens = [1, 70, 9, 33, 200, 64, 129]
    T = sum(lens)
    qkv = rnd(T, (nh + 2 * nkv) * hd, dt=dt, s=0.7)
    q, k, v = qkv[:, :nh * hd], qkv[:, nh * hd:(nh + nkv) * hd], qkv[:, (nh + nkv) * hd:]
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    seq_start = torch.tensor(starts, dtype=torch.int32, device="cuda")
    token_seq = torch.repeat_interleave(torch.arange(len(lens), dtype=torch.int32), torch.tensor(lens)).cuda()
    scale = 1.0 / math.sqrt(hd)
    impls = [lambda: ops.attn_prefill_simt(q, k, v, seq_start, token_seq, nh, nkv, hd, scale, cap, window)]
    if ops.attn_prefill_takes(dt, hd) and hd in (16, 32, 48, 64, 128, 256):
        impls.append(lambda: ops.attn_prefill_mma(q, k, v, seq_start, nh, nkv, hd, scale, cap, window, max(lens)))
    if ops.attn_prefill_tc_takes(dt, hd):
        impls.append(lambda: ops.attn_prefill_tc(q, k, v, seq_start, lens, nh, nkv, hd, scale, cap, window))
    wants = []
    for b, n in enumerate(lens):
        s = slice(starts[b], starts[b + 1])
        wants.append(plain.attention(q[s].float().cpu().view(n, nh, hd), k[s].float().cpu().view(n, nkv, hd),
                                     v[s].float().cpu().view(n, nkv, hd), scale, cap or None, window or None))
    for impl in impls:
        got = impl()
        for b, n in enumerate(lens):
            close(got[starts[b]:starts[b + 1]].view(n, nh, hd), wants[b], dt, 2.0)
    if ops.attn_prefill_tc_takes(dt, hd):
        torch.cuda.synchronize()
        assert ops.attn_prefill_tc_error(hd) == 0


@pytest.mark.parametrize("nh,nkv,hd,cap,window,lens", [(8, 4, 256, 50.0, 0, [1000]), (8, 4, 256, 50.0, 300, [700, 64, 129]),
                                                       (4, 1, 128, 0.0, 0, [513, 1]), (2, 2, 64, 20.0, 100, [400, 333]),
                                                       (4, 2, 256, 50.0, 1024, [2500]), (4, 2, 128, 30.0, 0, [2100, 700])])
def test_attn_prefill_tc_long(ops, nh, nkv, hd, cap, window, lens):
    """Long sequences: many key blocks, the lazy rescaling of O, the window's trailing edge, and query
    tiles whose rows belong to the next sequence of the packed batch."""
    T = sum(lens)
    qkv = rnd(T, (nh + 2 * nkv) * hd, dt=torch.bfloat16, s=1.0)
    # make the scores grow along each sequence, so that the running maximum keeps moving
    ramp = torch.cat([torch.linspace(0.2, 2.0, n) for n in lens]).cuda().bfloat16()
    qkv[:, nh * hd:(nh + nkv) * hd] *= ramp[:, None]
    q, k, v = qkv[:, :nh * hd], qkv[:, nh * hd:(nh + nkv) * hd], qkv[:, (nh + nkv) * hd:]
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    seq_start = torch.tensor(starts, dtype=torch.int32, device="cuda")
    scale = 1.0 / math.sqrt(hd)
    got = ops.attn_prefill_tc(q, k, v, seq_start, lens, nh, nkv, hd, scale, cap, window)
    ref = ops.attn_prefill_mma(q, k, v, seq_start, nh, nkv, hd, scale, cap, window, max(lens))
    torch.cuda.synchronize()
    assert ops.attn_prefill_tc_error(hd) == 0
    assert torch.isfinite(got.float()).all()
    for b, n in enumerate(lens):
        s = slice(starts[b], starts[b + 1])
        sub = slice(0, n) if n <= 400 else slice(n - 200, n)
        want = plain.attention(q[s].float().cpu().view(n, nh, hd), k[s].float().cpu().view(n, nkv, hd),
                               v[s].float().cpu().view(n, nkv, hd), scale, cap or None, window or None)
        close(got[s].view(n, nh, hd)[sub], want[sub], torch.bfloat16, 2.0)
        close(ref[s].view(n, nh, hd)[sub], want[sub], torch.bfloat16, 2.0)


def moe_rule(ops, T, top, E, W, ff, gated):
    return ops.moe_tile(T * top, E, (3 if gated else 2) * W * ff * 2)


def test_moe_few_pairs_are_grouped_where_they_share_enough(ops):
    """Pairs, experts, an expert's bytes: on either side of the lines that the rule draws for fewer than 128 pairs."""
    mb = 1 << 20
    for pairs, experts, size, tile in ((48, 32, 12 * mb, 16), (47, 32, 12 * mb, 0), (79, 32, 3 * mb, 0), (80, 32, 3 * mb, 16), (64, 64, 4 * mb, 16),
                                       (64, 64, 3 * mb, 0), (96, 64, 3 * mb, 16),
                                       (64, 128, 4 * mb, 0), (96, 128, 4 * mb, 16), (127, 2048, 12 * mb, 0), (127, 4096, 12 * mb, 0), (128, 4096, mb, 16)):
        assert ops.moe_tile(pairs, experts, size) == tile, (pairs, experts, size)


# tokens, experts a token, experts, width, ff, the tile that the rule picks
MOE_TILES = [(12, 4, 32, 2048, 1024, 16), (33, 4, 8, 136, 48, 32), (200, 2, 16, 96, 208, 64), (700, 2, 6, 72, 16, 128), (128, 1, 40, 264, 144, 16)]


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("on", ["input", "output"])
@pytest.mark.parametrize("T,top,E,W,ff,tile", MOE_TILES)
def test_moe_experts_by_tiles(ops, gated, on, T, top, E, W, ff, tile):
    """Experts' products grouped in tiles of every size: some experts without a pair, one with more than a tile's, sizes
    that fill no tile of weight rows.  act and the operands are rounded to bfloat16 once each, sums are 32-bit."""
    assert moe_rule(ops, T, top, E, W, ff, gated) == tile or not gated
    g = torch.Generator().manual_seed(T)
    idx = torch.stack([torch.randperm(E - 1, generator=g)[:top] for _ in range(T)])          # the last expert has none
    idx[: T // 2, 0] = torch.where((idx[: T // 2] == 1).any(1), idx[: T // 2, 0], torch.ones(T // 2, dtype=torch.long))
    idx, weight = idx.to("cuda", torch.int32), rnd(T, top, seed=3).abs() + 0.1
    x = rnd(T, W, dt=torch.bfloat16)
    gw, uw, dw = (rnd(E, *s, dt=torch.bfloat16, s=0.1, seed=i) for i, s in enumerate(((ff, W), (ff, W), (W, ff))))
    both = torch.stack([ops.interleave_gate_up(gw[e], uw[e]) for e in range(E)]) if gated else None
    got = ops.moe_experts(x, gw if gated else None, uw, dw, idx, weight, gate_up_w=both, weight_on=on)
    want = torch.zeros(T, W, dtype=torch.float64, device="cuda")
    for k in range(top):
        e, w = idx[:, k].long(), weight[:, k, None].double()
        xs = x.double() * (w if on == "input" else 1.0)
        u = torch.stack([uw[e[t]].double() @ xs[t] for t in range(T)])
        a = torch.relu(u) ** 2
        if gated:
            a = torch.nn.functional.silu(torch.stack([gw[e[t]].double() @ xs[t] for t in range(T)])) * u
        want += torch.stack([dw[e[t]].double() @ a[t] for t in range(T)]) * (1.0 if on == "input" else w)
    assert float((got.double() - want).norm() / want.norm()) < 4e-3
    assert ops.kernel_errors() == {}


def off_16_bytes(t):
    """The same numbers, contiguous, in memory that begins 2 bytes past a 16-byte boundary."""
    room = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    room[1:] = t.reshape(-1)
    return room[1:].view(t.shape)


def moe_case(ops, T, top, E, W, ff, gated):
    g = torch.Generator().manual_seed(T)
    idx = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).to("cuda", torch.int32)
    weight, x = rnd(T, top, seed=3).abs() + 0.1, rnd(T, W, dt=torch.bfloat16)
    gw, uw, dw = (rnd(E, *s, dt=torch.bfloat16, s=0.1, seed=i) for i, s in enumerate(((ff, W), (ff, W), (W, ff))))
    both = torch.stack([ops.interleave_gate_up(gw[e], uw[e]) for e in range(E)]) if gated else None
    want = torch.zeros(T, W, dtype=torch.float64, device="cuda")
    for e in range(E):
        t, k = torch.nonzero(idx == e, as_tuple=True)
        u = x[t].double() @ uw[e].double().T
        a = torch.nn.functional.silu(x[t].double() @ gw[e].double().T) * u if gated else torch.relu(u) ** 2
        want.index_add_(0, t, a @ dw[e].double().T * weight[t, k, None].double())
    return idx, weight, x, gw if gated else None, uw, dw, both, want


@pytest.mark.parametrize("which", ["gate and up", "gate and up alone", "down", "joint", "up without a gate", "down without a gate"])
@pytest.mark.parametrize("T,top,E,W,ff", [(16, 4, 16, 2048, 1024), (60, 4, 12, 136, 48), (300, 4, 12, 136, 48)])
def test_moe_experts_whose_matrices_begin_off_16_bytes(ops, which, T, top, E, W, ff):
    """Contiguous matrices may begin anywhere: what the tensor cores' copies cannot fetch is read another way, at counts of
    pairs that run pair by pair (where such matrices were always taken) and at those that run grouped."""
    gated = "without" not in which
    idx, weight, x, gw, uw, dw, both, want = moe_case(ops, T, top, E, W, ff, gated)
    assert moe_rule(ops, T, top, E, W, ff, gated) > 0
    if which.startswith("gate and up") or which.startswith("up"):
        gw, uw = off_16_bytes(gw) if gated else None, off_16_bytes(uw)
    elif which.startswith("down"):
        dw = off_16_bytes(dw)
    else:
        both = off_16_bytes(both)
    got = ops.moe_experts(x, gw, uw, dw, idx, weight, gate_up_w=None if which.endswith("alone") else both)
    assert float((got.double() - want).norm() / want.norm()) < 4e-3
    assert ops.kernel_errors() == {}


def test_moe_tiles_refuse_scratch_that_is_too_small(ops, monkeypatch):
    idx, weight, x, gw, uw, dw, both, want = moe_case(ops, 60, 4, 12, 136, 48, True)
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *s, **k: empty(s[0] - 256, **k) if k.get("dtype") == torch.uint8 else empty(*s, **k))
    with pytest.raises(ops.KernelError, match="scratch"):
        ops.moe_experts(x, gw, uw, dw, idx, weight, gate_up_w=both)


@pytest.mark.parametrize("T", [24, 60, 300])
def test_moe_experts_leave_a_joint_matrix_that_is_not_packed_unread(ops, T):
    """The interleaved gate and up rows only speed the products up: if they are not [E, 2 ff, W], packed, of x's dtype the
    single matrices are read."""
    idx, weight, x, gw, uw, dw, both, want = moe_case(ops, T, 4, 12, 1024, 512, True)
    wide = torch.zeros(12, 1024, 1024 + 64, dtype=torch.bfloat16, device="cuda")
    wide[:, :, :1024] = both
    for joint in (wide[:, :, :1024], both.float(), both[:, :512].contiguous(), None):
        got = ops.moe_experts(x, gw, uw, dw, idx, weight, gate_up_w=joint)
        assert float((got.double() - want).norm() / want.norm()) < 4e-3
    assert ops.kernel_errors() == {}


@pytest.mark.parametrize("T, E, tile", [(4, 12, 0), (24, 12, 16), (60, 12, 32), (120, 12, 64), (255, 12, 128)])
def test_moe_gate_far_below_zero(ops, T, E, tile):
    """silu(-88) = -88 e^-88 is a bfloat16 number (-5e-37), pair by pair and in tiles of every size below 1,024 pairs."""
    W, ff, top = 1024, 512, 4
    assert moe_rule(ops, T, top, E, W, ff, True) == tile and T * top < ops.MOE_EXACT_BELOW
    x = torch.zeros(T, W, dtype=torch.bfloat16, device="cuda")
    x[:, 0] = 1.0
    gw, uw = (torch.zeros(E, ff, W, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    gw[:, :, 0], uw[:, :, 0] = -88.0, 1.0
    dw = torch.ones(E, W, ff, dtype=torch.bfloat16, device="cuda")
    both = torch.stack([ops.interleave_gate_up(gw[e], uw[e]) for e in range(E)])
    idx = torch.stack([torch.randperm(E, generator=torch.Generator().manual_seed(t))[:top] for t in range(T)]).to("cuda", torch.int32)
    got = ops.moe_experts(x, gw, uw, dw, idx, torch.ones(T, top, device="cuda"), gate_up_w=both)
    want = -88.0 * math.exp(-88.0) * ff * top
    assert float((got.double() / want - 1.0).abs().max()) < 4e-3          # the activations are rounded to bfloat16


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("reach", [0.3, 1.0, 30.0, 3000.0])
def test_attn_prefill_cap_near_and_far(ops, hd, reach):
    """The soft cap where all scores lie within half of it, around half of it and far past it (``reach``: scores over the
    cap at most), every warp with some rows of each; probabilities and the result are rounded to bfloat16 once each."""
    n, cap = 333, 8.0
    q, k, v = (rnd(n, hd, dt=torch.bfloat16, seed=i) for i in range(3))
    most = float((q.double() @ k.double().T).abs().max())
    scale = reach * cap / most
    q[::3] *= 0.25
    starts = torch.tensor([0, n], dtype=torch.int32, device="cuda")
    for sign in (1.0, -1.0):                                            # the negative of a query mirrors its scores about 0
        got = ops.attn_prefill_tc(sign * q, k, v, starts, [n], 1, 1, hd, scale, cap, 0).double()
        s = cap * torch.tanh(sign * q.double() @ k.double().T * scale / cap)
        s = s.masked_fill(torch.ones(n, n, device="cuda", dtype=torch.bool).triu(1), -math.inf)
        want = torch.softmax(s, -1) @ v.double()
        assert float((got - want).norm() / want.norm()) < 5e-3
    assert ops.attn_prefill_tc_error(hd) == 0


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("spread", [0.5, 1.3, 20.0])
def test_attn_prefill_cap_of_a_row_goes_by_its_own_keys(ops, hd, window, spread):
    """What the soft cap makes of a score must not depend on scores that the query does not see: a prompt's rows are the
    same bits alone, before a prompt of huge scores and behind one, and with huge queries, keys and values from some later
    token on (also one that shares a tile, a warp and a block of keys with them).  ``spread``: the scores' standard
    deviation, with which all rows, some of them or none stay within half the cap."""
    n, cap, scale = 333, 8.0, spread / math.sqrt(hd)
    q, k, v = (rnd(n, hd, dt=torch.bfloat16, seed=i) for i in range(3))

    def run(prompts):
        qs, ks, vs = (torch.cat(x) for x in zip(*prompts))
        lens = [p[0].shape[0] for p in prompts]
        starts = torch.tensor([0] + lens, dtype=torch.int32, device="cuda").cumsum(0).int()
        return ops.attn_prefill_tc(qs, ks, vs, starts, lens, 1, 1, hd, scale, cap, window)

    alone = run([(q, k, v)])
    huge = tuple(rnd(77, hd, dt=torch.bfloat16, s=100.0, seed=9 + i) for i in range(3))
    assert torch.equal(run([(q, k, v), huge])[:n], alone)
    assert torch.equal(run([huge, (q, k, v)])[77:], alone)
    for at in (300, 273, 129, 70):
        later = tuple(torch.cat([x[:at], x[at:] * 100]) for x in (q, k, v))
        assert torch.equal(run([later])[:at], alone[:at]), at
    assert ops.attn_prefill_tc_error(hd) == 0


def test_attn_prefill_far_key_and_window_edge(ops):
    """A key made to stand out is seen from far away without a window, and exactly up to the window's
    edge with one; on tensor cores and on the generic kernel alike."""
    nh, nkv, hd, n, W = 2, 1, 64, 300, 100
    qkv = rnd(n, (nh + 2 * nkv) * hd, dt=torch.bfloat16, s=0.1)
    q, k, v = qkv[:, :nh * hd], qkv[:, nh * hd:(nh + nkv) * hd], qkv[:, (nh + nkv) * hd:]
    marked = 37
    k[marked] = (q[250, :hd].float() * 300).to(torch.bfloat16)          # query 250, head 0 loves key 37
    for i in (marked + W - 1, marked + W, 250):
        q[i, :hd] = q[250, :hd]
    seq_start = torch.tensor([0, n], dtype=torch.int32, device="cuda")
    token_seq = torch.zeros(n, dtype=torch.int32, device="cuda")
    for window in (0, W):
        for got in (ops.attn_prefill_simt(q, k, v, seq_start, token_seq, nh, nkv, hd, 1.0, 0.0, window),
                    ops.attn_prefill_mma(q, k, v, seq_start, nh, nkv, hd, 1.0, 0.0, window, n),
                    ops.attn_prefill_tc(q, k, v, seq_start, [n], nh, nkv, hd, 1.0, 0.0, window)):
            got = got.view(n, nh, hd).float()
            hit = lambda i: float((got[i, 0] - v[marked].float()).abs().max()) < 3e-2
            assert hit(marked + W - 1)                                  # the window's last row that still sees it
            assert hit(marked + W) == (window == 0)                     # one further: only without a window
            assert hit(250) == (window == 0)


@pytest.mark.parametrize("nh,nkv,hd,rot,n", [(24, 16, 128, 128, 129), (20, 20, 256, 256, 128), (5, 1, 80, 32, 131), (32, 17, 512, 512, 128)])
def test_rope_kv_of_many_heads(ops, nh, nkv, hd, rot, n):
    """Prompts whose tokens have more work items and copied pieces than their threads hold at a time, against the same rows in
    pieces of fewer than 128 tokens, which another kernel takes: both round 32-bit results once (two units of bfloat16's last
    place, 2^-7, where a product is contracted in one and not in the other)."""
    qkv = rnd(n, (nh + 2 * nkv) * hd, dt=torch.bfloat16)
    pos, seq, after = torch.arange(n).int().cuda() + 40, torch.zeros(n).int().cuda(), torch.tensor([n + 40]).int().cuda()
    table = torch.tensor([[3, 0, 2]]).int().cuda()
    inv = (1e4 ** -(torch.arange(0, rot, 2).float() / rot)).cuda()
    pools = [torch.zeros(4, nkv, PAGE, hd, dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    want = qkv.clone()
    ops.rope_kv(qkv, nh, nkv, hd, rot, inv, pos, seq, after, *pools[:2], table, 0)
    for lo in range(0, n, 100):
        part = slice(lo, min(n, lo + 100))
        ops.rope_kv(want[part], nh, nkv, hd, rot, inv, pos[part], seq[part], after, *pools[2:], table, 0)
    for got, ref in ((qkv, want), (pools[0], pools[2]), (pools[1], pools[3])):
        torch.testing.assert_close(got.float(), ref.float(), rtol=2 ** -7, atol=1e-6)
    assert torch.equal(pools[1], pools[3])


@pytest.mark.parametrize("nh,nkv,hd,rot", [(12, 2, 64, 64), (14, 2, 64, 64), (3, 1, 128, 32), (2, 4, 64, 0)])
def test_rope_kv_of_few_heads(ops, nh, nkv, hd, rot):
    """More than 1,536 tokens of up to 64 work items take 64 threads a token: the same bits as in pieces that take 128."""
    n = 1600
    qkv = rnd(n, (nh + 2 * nkv) * hd, dt=torch.bfloat16)
    pos, seq, after = torch.arange(n).int().cuda(), torch.zeros(n).int().cuda(), torch.tensor([n]).int().cuda()
    table = torch.arange(n // PAGE - 1, -1, -1).int().cuda()[None].contiguous()
    inv = (1e4 ** -(torch.arange(0, rot, 2).float() / rot)).cuda() if rot else None
    pools = [torch.zeros(n // PAGE, nkv, PAGE, hd, dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    want = qkv.clone()
    ops.rope_kv(qkv, nh, nkv, hd, rot, inv, pos, seq, after, *pools[:2], table, 0)
    for part in (slice(0, 1400), slice(1400, n)):
        ops.rope_kv(want[part], nh, nkv, hd, rot, inv, pos[part], seq[part], after, *pools[2:], table, 0)
    assert torch.equal(qkv, want) and torch.equal(pools[0], pools[2]) and torch.equal(pools[1], pools[3])
    assert torch.equal(pools[1].transpose(1, 2).flip(0).reshape(n, nkv * hd), qkv[:, (nh + nkv) * hd:])


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd,rot,ring,theta", [(16, 16, 0, 1e4), (48, 48, 128, 5e4), (256, 256, 64, 1e4), (32, 16, 0, 1e3), (64, 0, 0, 1.0),
                                               (640, 640, 0, 1e4), (576, 530, 64, 1e4)])     # more pairs than a CTA has threads for
def test_rope_kv(ops, dt, hd, rot, ring, theta):
    nh, nkv = 3, 2
    lens_before, new = [0, 0, 0], [5, 150, 70]                      # a first step
    for lens_before, new in (([0, 0, 0], [5, 150, 70]), ([5, 150, 70], [1, 1, 1])):
        B, T = len(new), sum(new)
        qkv = rnd(T, (nh + 2 * nkv) * hd, dt=dt, seed=T)
        orig = qkv.clone()
        pos = torch.cat([torch.arange(b, b + n) for b, n in zip(lens_before, new)]).int().cuda()
        tseq = torch.repeat_interleave(torch.arange(B), torch.tensor(new)).int().cuda()
        after = [b + n for b, n in zip(lens_before, new)]
        la = torch.tensor(after, dtype=torch.int32, device="cuda")
        n_pages = 16
        kp = torch.full((n_pages, nkv, PAGE, hd), float("nan"), dtype=dt, device="cuda")
        vp = torch.full_like(kp, float("nan"))
        width = max(((min(a, ring) if ring else a) + PAGE - 1) // PAGE for a in after)
        table = torch.zeros(B, width, dtype=torch.int32)
        perm = torch.randperm(n_pages, generator=torch.Generator().manual_seed(3)).tolist()
        for b, a in enumerate(after):
            for pg in range(((min(a, ring) if ring else a) + PAGE - 1) // PAGE):
                table[b, pg] = perm.pop()
        table = table.cuda()
        inv = (1.0 / (torch.tensor(theta) ** (torch.arange(0, rot, 2).float() / rot))).cuda() if rot else None
        if dt == torch.bfloat16 and T <= 16:
            # the same values as three partial sums: the kernel adds them, rotates in 32-bit, rounds once
            part = torch.stack([orig.float() * 0.5, orig.float() * 0.25, orig.float() * 0.25])
            dst = torch.full_like(qkv, float("nan"))
            kp2, vp2 = kp.clone(), vp.clone()
            ops.rope_kv(dst, nh, nkv, hd, rot, inv, pos, tseq, la, kp2, vp2, table, ring, partial=part)
        ops.rope_kv(qkv, nh, nkv, hd, rot, inv, pos, tseq, la, kp, vp, table, ring)
        if dt == torch.bfloat16 and T <= 16:
            assert torch.equal(dst, qkv) and torch.equal(torch.nan_to_num(kp2.float()), torch.nan_to_num(kp.float())) \
                and torch.equal(torch.nan_to_num(vp2.float()), torch.nan_to_num(vp.float()))
        o = orig.float().cpu().view(T, nh + 2 * nkv, hd)
        want = o.clone()
        if rot:
            want[:, :nh + nkv, :rot] = plain.rope(o[:, :nh + nkv, :rot], pos.cpu(), theta)
        got = qkv.float().cpu().view(T, nh + 2 * nkv, hd)
        close(got, want, dt, 2.0)
        assert torch.equal(got[:, nh + nkv:], o[:, nh + nkv:])       # v is not rotated
        # every token that must be in the cache is there, at its row, and nothing else was written
        written = 0
        for t in range(T):
            b, p = int(tseq[t]), int(pos[t])
            if ring and p < after[b] - ring:
                continue
            r = p % ring if ring else p
            page = int(table[b, r // PAGE])
            assert torch.equal(kp[page, :, r % PAGE].float().cpu(), got[t, nh:nh + nkv])
            assert torch.equal(vp[page, :, r % PAGE].float().cpu(), got[t, nh + nkv:])
            written += 1
        assert int((~torch.isnan(kp.float()[:, 0, :, 0])).sum()) == written


# ---------------------------------------------------------------------------
def test_argmax_ties_and_rows(ops):
    V = 256000
    x = rnd(5, V)
    x[0, 1234] = x[0, 200000] = 50.0            # a tie: the smaller index wins
    x[1, V - 1] = 60.0
    x[2, 0] = 60.0
    x[3, :] = -1.0                              # all equal
    x[4, 8191] = x[4, 8192] = 70.0              # a tie across the border of two stage-one chunks
    got = ops.argmax(x).cpu().tolist()
    assert got == [1234, V - 1, 0, 0, 8191]
    assert ops.argmax(rnd(3, 301)).cpu().tolist() == rnd(3, 301).argmax(-1).cpu().tolist()


def _args(rows, temperature, top_p, penalty, draws):
    f = lambda v: torch.full((rows,), float(v), device="cuda") if not isinstance(v, torch.Tensor) else v.cuda().float()
    return f(temperature), f(top_p), f(penalty), f(draws)


def test_wide_sampling_reads_no_scratch_it_did_not_write(ops):
    """Rows without a nucleus (top_p 1) beside rows with one, on scratch memory that held other bytes before: the
    draws are those of clean memory."""
    V, rows = 256000, 8
    x = rnd(rows, V, s=2.0, seed=3)
    u = torch.linspace(0.001, 0.999, rows)
    top_p = torch.tensor([1.0, 0.9, 1.0, 1.0, 0.5, 1.0, 0.95, 1.0])
    t, p, pen, ud = _args(rows, 1.0, top_p, 1.0, u)
    torch.cuda.empty_cache()
    want = ops.sample(x.clone(), t, p, pen, ud, None).cpu()
    for fill in (0xFF, 0x01, 0x7F):
        junk = [torch.full((n,), fill, dtype=torch.uint8, device="cuda") for n in (1 << 16, 1 << 18, 1 << 20, 1 << 22, 1 << 24)]
        del junk                                  # the allocator hands these blocks out again, bytes and all
        assert torch.equal(ops.sample(x.clone(), t, p, pen, ud, None).cpu(), want)
    for i in range(rows):
        probs = plain.nucleus(x[i].cpu(), 1.0, float(top_p[i]))
        cdf = torch.cumsum(probs, 0)
        tok = int(want[i])
        assert probs[tok] > 0 and float(cdf[tok] - probs[tok]) - 1e-4 <= float(u[i]) <= float(cdf[tok]) + 1e-4


@pytest.mark.parametrize("V", [1000, 40001])      # one CTA a row; several CTAs a row (the ids lie in different chunks)
def test_sample_greedy_and_penalty(ops, V):
    a, b, c, d = 10, V - 7, V // 2 + 3, 5
    x = rnd(4, V)
    x[:, a] = 9.0; x[:, b] = 8.0
    recent = torch.full((4, 128), -1, dtype=torch.int32, device="cuda")
    recent[1, :3] = torch.tensor([a, a, d], dtype=torch.int32)          # a twice: penalised once
    recent[1, 100] = a
    recent[2, 0] = b
    x[3, a] = -0.5; x[3, b] = -0.6; x[3, c] = -0.55
    x[3, :] = torch.minimum(x[3, :], torch.tensor(-0.5, device="cuda"))
    recent[3, 0] = a
    before = x.clone()
    t, p, pen, u = _args(4, 0.0, 0.95, 1.2, 0.5)
    got = ops.sample(x, t, p, pen, u, recent).cpu().tolist()
    want = [plain.greedy(plain.repetition_penalty(before[i].cpu(), recent[i].cpu().tolist(), 1.2)) for i in range(4)]
    assert got == want and got[0] == a and got[1] == b and got[2] == a
    assert float(x[1, a]) == pytest.approx(9.0 / 1.2) and float(x[1, d]) == pytest.approx(
        float(before[1, d]) / 1.2 if before[1, d] > 0 else float(before[1, d]) * 1.2)


@pytest.mark.parametrize("V", [301, 256000])
@pytest.mark.parametrize("temperature,top_p", [(1.0, 1.0), (0.7, 0.95), (1.5, 0.5), (0.3, 0.9)])
def test_sample_draws_follow_the_inverse_cdf(ops, V, temperature, top_p):
    rows = 32
    x = rnd(rows, V, s=2.0, seed=V)
    u = torch.linspace(0.001, 0.999, rows)
    t, p, pen, ud = _args(rows, temperature, top_p, 1.0, u)
    got = ops.sample(x.clone(), t, p, pen, ud, None).cpu().tolist()
    for i in range(rows):
        probs = plain.nucleus(x[i].cpu(), temperature, top_p)          # float64, renormalised over the nucleus
        cdf = torch.cumsum(probs, 0)
        tok = got[i]
        assert probs[tok] > 0, "a token outside the nucleus was drawn"
        lo = float(cdf[tok] - probs[tok])
        assert lo - 1e-4 <= float(u[i]) <= float(cdf[tok]) + 1e-4


@pytest.mark.parametrize("V", [16384, 40001, 256000])
@pytest.mark.parametrize("kind", ["equal", "three values", "masked", "flat", "spike", "narrow", "two zeros", "neighbours"])
def test_sample_where_logits_crowd(ops, V, kind):
    """Rows whose threshold falls among more elements than a row lists (equal logits), that hold -inf, whose logits lie
    close together, or one far above the rest; tokens as the float64 nucleus in index order gives them."""
    rows = 24
    x = rnd(rows, V, s=2.0, seed=V)
    if kind == "equal":
        x[:] = 1.5
    elif kind == "three values":
        x = torch.round(x / 4.0).clamp(-1, 1) + 0.0                     # (no -0: its key is below that of 0)
    elif kind == "masked":
        x[:, V // 50:] = -math.inf
    elif kind == "flat":
        x *= 1e-3
    elif kind == "spike":
        x = (x * 1e-2)
        x[:, V // 3] = 10.0
    elif kind == "narrow":                                              # the bulk in one or two of the steps of the row's range
        x = (x * 1e-4)
        x[:, V // 3] = 8.0
    elif kind == "two zeros":                                           # many of 0, half of them -0, the next lower key
        x = torch.round(x / 4.0)
    else:                                                               # thousands each of four numbers that the row's range cannot tell apart
        x = 1.0 + torch.remainder(torch.arange(V, device="cuda") * 7919, 4).float().expand(rows, V) * 2.0 ** -23
        x[:, V // 3] = 8.0
    u = torch.linspace(0.001, 0.999, rows)
    t, p, pen, ud = _args(rows, 0.9, 0.6, 1.0, u)
    got = ops.sample(x.clone(), t, p, pen, ud, None).cpu().tolist()
    for i in range(rows):
        row = x[i].double().cpu()
        if kind == "two zeros":
            row = torch.where((row == 0) & torch.signbit(row), torch.full_like(row, -1e-30), row)
        m = torch.exp((row - row.max()) / 0.9)
        order = torch.sort(row, descending=True).values                  # equal logits are kept or left together, by their value
        cum = torch.cumsum(torch.exp((order - row.max()) / 0.9), 0)
        thr = order[min(V - 1, int((cum < 0.6 * m.sum() * (1 - 1e-6)).sum()))]
        m[row < thr] = 0.0
        cdf = torch.cumsum(m, 0) / m.sum()
        tok = got[i]
        assert m[tok] > 0, "a token outside the nucleus was drawn"
        assert float(cdf[tok] - m[tok] / m.sum()) - 1e-4 <= float(u[i]) <= float(cdf[tok]) + 1e-4


@pytest.mark.parametrize("rows, V", [(4, 32768), (4, 256000), (32, 256000)])
def test_sample_takes_about_as_long_where_logits_crowd(ops, rows, V):
    """Rows with too many elements in the threshold's step to list: within three times the time of ordinary rows (up to
    24 times before; 1.2 to 2.0 measured)."""
    ordinary = rnd(rows, V, s=2.0, seed=V)
    narrow = ordinary * 1e-3
    narrow[:, V // 3] = 8.0
    t, p, pen, u = _args(rows, 0.8, 0.95, 1.0, torch.linspace(0.1, 0.9, rows))
    times = [device_time(lambda: ops.sample(x, t, p, pen, u, None)) for x in (ordinary, narrow, torch.round(ordinary) / 2)]
    assert max(times[1:]) <= 3.0 * times[0], times


@pytest.mark.parametrize("V", [500, 20011])
def test_sample_mixed_rows(ops, V):
    x = rnd(3, V, s=3.0)
    t = torch.tensor([0.0, 1.0, 0.0]); p = torch.tensor([1.0, 1.0, 1.0])
    got = ops.sample(x.clone(), t.cuda(), p.cuda(), torch.ones(3).cuda(), torch.tensor([0.3, 0.3, 0.3]).cuda(), None)
    assert got[0] == x[0].argmax() and got[2] == x[2].argmax()


def test_refusals(ops):
    with pytest.raises(ops.KernelError, match="GPU only"):
        ops.rmsnorm(torch.zeros(2, 4), torch.zeros(4), 1e-6, 1.0, torch.float32)
    with pytest.raises(ops.KernelError, match="heads"):
        ops.attn_prefill_simt(rnd(2, 48), rnd(2, 32), rnd(2, 32), torch.zeros(2, dtype=torch.int32, device="cuda"),
                              torch.zeros(2, dtype=torch.int32, device="cuda"), 3, 2, 16, 1.0, 0.0, 0)
    with pytest.raises(ops.KernelError, match="512"):
        ops.attn_prefill_simt(rnd(2, 1024), rnd(2, 1024), rnd(2, 1024), torch.zeros(2, dtype=torch.int32, device="cuda"),
                              torch.zeros(2, dtype=torch.int32, device="cuda"), 1, 1, 1024, 1.0, 0.0, 0)
    with pytest.raises(ops.KernelError, match="float32 and bfloat16"):
        ops.rmsnorm(torch.zeros(2, 4, device="cuda", dtype=torch.float16), torch.zeros(4, device="cuda"), 1e-6, 1.0,
                    torch.float32)


def test_attn_decode_ctas_per_sm(ops):
    """The tensor-core decode kernel's stream partition is budgeted (shared memory to the byte, registers by its
    launch bounds) for two CTAs an SM at heads narrower than 256: if a change breaks the budget the kernel still
    computes the same, only slower, so the fit is checked here.  (2: the split partition that adds up, rotates and appends.)"""
    from trapetum_b200.csrc import build
    lib = build.load("attention_decode")
    for hd in (64, 128, 256):
        assert lib.tb_attn_decode_occupancy(hd, 0) == 1, hd
        assert lib.tb_attn_decode_occupancy(hd, 1) == (2 if hd <= 128 else 1), hd
        assert lib.tb_attn_decode_occupancy(hd, 2) == 1, hd
