"""Kernels that a rule on sizes, types or alignment chooses, at the sizes where each can go wrong: edges of tiles,
remainders, the smallest and the largest of the rule's range."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _k():
    from ccinfer_b200 import kernels
    return kernels


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rel(got, ref):
    got, ref = got.double(), ref.double()
    assert torch.isfinite(got).all()
    return float((got - ref).abs().max() / ref.abs().max().clamp_min(1e-30))


# rows kernel: 1, 2, 3, 5, 9, 16 rows; tiles from 17 rows on; K of less than a segment, of whole segments and with a remainder; rows
# that start on no 16 bytes; more tiles than two rounds
@pytest.mark.parametrize("M,N,K,pad,batch", [
    (1, 1, 1, 0, 1), (2, 15, 31, 0, 1), (3, 17, 256, 0, 2), (4, 33, 260, 1, 1), (5, 64, 2048, 0, 1), (8, 300, 1001, 3, 1),
    (9, 16, 8192, 0, 1), (16, 2049, 512, 4, 3), (17, 129, 511, 0, 1), (32, 128, 512, 0, 2), (33, 257, 516, 0, 1),
    (64, 100, 4100, 2, 1), (65, 128, 1024, 0, 1), (120, 300, 100, 0, 1), (128, 1000, 2048, 0, 1), (300, 16384, 544, 0, 1),
    (1030, 5000, 72, 0, 1)])
def test_float_product_of_every_shape_is_one_order_of_sums(M, N, K, pad, batch):
    """Against float64: eight chains of K / 8 float multiply-adds and seven sums stay within (K / 8 + 8) roundings of
    the sum of magnitudes; and a row alone gives the bits that it has among others."""
    g = _gen(M + 7 * N + 13 * K)
    a = torch.randn((batch, M, K + pad), generator=g, device="cuda")[:, :, :K]
    w = torch.randn((batch, N, K + pad), generator=g, device="cuda")[:, :, :K]
    c = torch.full((batch, M, N), float("nan"), device="cuda")
    k = _k()
    if batch > 1:
        k.gemm_f32_batched(c, a, w)
    else:
        k.gemm_f32(c[0], a[0], w[0])
    ref = a.double() @ w.double().transpose(1, 2)
    size = a.double().abs() @ w.double().abs().transpose(1, 2)
    assert ((c.double() - ref).abs() <= (K / 8 + 8) * 2.0 ** -24 * size).all()
    for rows in (1, 7, 20):   # a few rows by themselves: other kernels, the same sums
        n = min(rows, M)
        c1 = torch.full((n, N), float("nan"), device="cuda")
        k.gemm_f32(c1, a[0, M - n:], w[0])
        assert torch.equal(c1, c[0, M - n:])


# numbers of rows between those of the tiles' heights, at a few, some and many columns (every tile: the test below)
@pytest.mark.parametrize("M", [20, 21, 23, 29, 31, 41, 47, 50, 57, 63, 77, 79, 90, 96, 101, 107, 112, 125, 140, 175, 223])
@pytest.mark.parametrize("N,K", [(200, 1030), (3001, 96), (640, 2048)])
def test_float_product_of_every_tile_height(M, N, K):
    """As above, beside the rows by themselves: sixteen at a time have a kernel without tiles."""
    g = _gen(M + 7 * N + 13 * K)
    a, w = torch.randn((M, K), generator=g, device="cuda"), torch.randn((N, K), generator=g, device="cuda")
    k = _k()
    c = torch.full((M, N), float("nan"), device="cuda")
    k.gemm_f32(c, a, w)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert ((c.double() - ref).abs() <= (K / 8 + 8) * 2.0 ** -24 * size).all()
    for r in range(0, M, 16):
        c1 = torch.empty((min(16, M - r), N), device="cuda")
        k.gemm_f32(c1, a[r:r + 16], w)
        assert torch.equal(c1, c[r:r + 16])


# a shape for each height of a tile, columns a thread, warps and, in lines of their own, whole or shared by a cluster that the rule takes
@pytest.mark.parametrize("M,N,K,batch", [
    (2132, 421, 33, 1), (3337, 285, 33, 1), (3628, 803, 33, 1), (1732, 2005, 33, 1), (338, 9840, 35, 1),
    (442, 144, 108, 1), (525, 150, 123, 1), (1514, 132, 197, 1), (1576, 153, 219, 1), (1793, 151, 207, 1),
    (31, 138, 33, 1), (1878, 132, 33, 1), (2447, 134, 35, 1), (3083, 137, 35, 1), (3627, 134, 34, 1), (3311, 525, 34, 1),
    (26, 131, 72, 1), (176, 132, 79, 1), (230, 136, 84, 1), (281, 138, 105, 1), (361, 132, 102, 1), (977, 133, 157, 1),
    (57, 19213, 35, 1), (67, 29287, 33, 1), (82, 31452, 35, 1), (30, 61839, 34, 1),
    (17, 145, 104, 8), (59, 996, 98, 1), (67, 978, 118, 1), (81, 2106, 187, 1), (193, 1225, 192, 1), (126, 2091, 216, 1)])
def test_float_product_of_every_tile(M, N, K, batch):
    """As above: a segment is 32 k or more, a chain of as many roundings, and eight sums are added."""
    g = _gen(M + 7 * N + 13 * K)
    a, w = torch.randn((batch, M, K), generator=g, device="cuda"), torch.randn((batch, N, K), generator=g, device="cuda")
    c = torch.full((batch, M, N), float("nan"), device="cuda")
    k = _k()
    if batch > 1:
        k.gemm_f32_batched(c, a, w)
    else:
        k.gemm_f32(c[0], a[0], w[0])
    ref, size = a.double() @ w.double().mT, a.double().abs() @ w.double().abs().mT
    assert ((c.double() - ref).abs() <= (-(-K // 256) * 32 + 8) * 2.0 ** -24 * size).all()
    for r in range(0, M, 16):
        c1 = torch.empty((min(16, M - r), N), device="cuda")
        k.gemm_f32(c1, a[0, r:r + 16], w[0])
        assert torch.equal(c1, c[0, r:r + 16])


def _recurrence64(q, k, v, g, beta, S):
    """Token by token in float64: q, k [n, H, dk], v [n, H, dv], g [n, H, dk or 1], beta [n, H] or None, S [H, dv, dk]."""
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * g[t][:, None, :]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - (S * k[t][:, None, :]).sum(-1))
        S = S + u[:, :, None] * k[t][:, None, :]
        out[t] = (S * q[t][:, None, :]).sum(-1)
    return out, S


# decays: of every size down to zero; near one; strong ones beside weak ones (runs of tokens far below float's range)
@pytest.mark.parametrize("decay", ["any", "slow", "strong"])
@pytest.mark.parametrize("rule", ["delta", "head delta", "linear", "head linear"])
@pytest.mark.parametrize("H,G,dk,dv", [(2, 2, 128, 128), (4, 2, 128, 32), (2, 1, 64, 96), (3, 3, 64, 64)])
def test_recurrence_in_chunks(H, G, dk, dv, rule, decay):
    """Portions of one token up to several chunks against the recurrence in float64.  An operand as two bfloat16 is right
    to 2^-17, a product of two to 2^-16 of its factors' norms; an output has passed four of them in a row: 2^-14 of the
    largest."""
    delta, head = "delta" in rule, "head" in rule
    g = _gen(dk + dv + len(rule) + len(decay))
    lens = [1, 2, 15, 16, 17, 63, 64, 65, 130, 200]
    n_slots, first = len(lens) + 2, 2   # the first two entries of the step are somebody else's
    T = sum(lens)

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    q, k = (torch.nn.functional.normalize(rnd(T, G, dk), dim=-1) for _ in range(2))
    v = rnd(T, H, dv)
    shape = (T, H) if head else (T, H, dk)
    u = torch.rand(shape, generator=g, device="cuda")
    a = {"any": u, "slow": 1 - 0.02 * u, "strong": torch.where(u < 0.1, torch.zeros_like(u), torch.where(u < 0.3, 1e-30 * u, 0.9 + 0.1 * u))}[decay]
    beta = torch.rand((T, H), generator=g, device="cuda") if delta else None
    state = rnd(n_slots, H, dv, dk)
    slots = torch.randperm(n_slots, generator=torch.Generator().manual_seed(3)).tolist()
    cu = [0] + torch.tensor(lens).cumsum(0).tolist()
    want, after = torch.zeros(T, H, dv, dtype=torch.float64, device="cuda"), state.double()
    for e, slot in enumerate(slots[:len(lens)]):
        if e < first:
            continue
        s = slice(cu[e], cu[e + 1])
        rep = H // G
        want[s], after[slot] = _recurrence64(
            q[s].double().repeat_interleave(rep, 1), k[s].double().repeat_interleave(rep, 1), v[s].double(),
            (a[s, :, None] if head else a[s]).double(), beta[s].double() if delta else None, state[slot].double())
    out = torch.zeros(T, H, dv, device="cuda")
    bufs = {}

    def scratch(key, per, shape, dtype):
        n = T if per == "tokens" else T // 64 + len(lens)
        bufs[key] = torch.full((n,) + tuple(shape), float("nan"), dtype=dtype, device="cuda")
        return bufs[key]

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")

    _k().chunk_recurrence(scratch, q.clone(), k.clone(), v.clone(), a.clone(), beta, state, out, dev(cu), dev(slots[:len(lens)]),
                          first, len(lens) - first, max(lens), G, H, dk, dv)
    assert torch.isfinite(out).all() and torch.isfinite(state).all()
    assert (out.double() - want).abs().max() <= 2.0 ** -14 * want.abs().max()
    assert (state.double() - after).abs().max() <= 2.0 ** -14 * after.abs().max()


# one team of 16 columns, two teams of 16, two of 32 (75 blocks and more)
@pytest.mark.parametrize("H,G,N,P", [(4, 2, 128, 64), (2, 1, 128, 16), (3, 3, 64, 48), (4, 1, 64, 32), (15, 3, 128, 64), (8, 2, 64, 128)])
def test_state_space_recurrence_in_chunks(H, G, N, P):
    """Portions of a prompt beside single tokens, from the projection's rows: the chunks' rows and the recurrence in float64.
    An operand as two bfloat16 is right to 2^-17; sums of logarithms over 64 tokens that cancel to 2^-18 of 64 steps."""
    k, g = _k(), _gen(H + G + N + P)
    lens = [1, 1, 2, 63, 64, 65, 150]
    T, taps, C = sum(lens), 4, H * P + 2 * G * N

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")

    width = -(-(C + H) // 8) * 8
    proj = rnd(T, width).to(torch.bfloat16)
    conv_w, conv_b, dt_bias = 0.5 * rnd(taps, C), rnd(C), rnd(H) - 2
    A_log = torch.log(1 + 15 * torch.rand(H, generator=g, device="cuda"))
    conv = torch.zeros(len(lens), taps - 1, C, dtype=torch.bfloat16, device="cuda")
    state = rnd(len(lens), H, P, N)
    first, slots = state.double(), dev(list(range(len(lens)))[::-1])
    cu = dev([0] + torch.tensor(lens).cumsum(0).tolist())
    entry = dev([e for e, n in enumerate(lens) for _ in range(n)])
    xs, bs, cs = (torch.full(s, float("nan"), device="cuda") for s in ((T, H, P), (T, G, N), (T, G, N)))
    dts, decay, log_a, log_dt = (torch.full((T, H), float("nan"), device="cuda") for _ in range(4))
    halves = [torch.full((T, G, N), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    out = torch.full((T, H, P), float("nan"), device="cuda")
    chunk = (2, *halves, log_a, log_dt)
    k.ssm_prepare(proj, 0, C, conv_w, conv_b, taps, conv, A_log, dt_bias, entry, cu, slots, xs, bs, cs, dts, decay, H, P, G, N,
                  chunk=chunk)
    k.ssm_recurrence(cs, bs, xs, decay, dts, state, out, cu, slots, 2, G, H, N, P)
    k.ssm_chunks(chunk, xs, state, out, cu, slots, 2, len(lens) - 2, G, H, N, P)
    for e, n in enumerate(lens):
        r0 = int(cu[e])
        x = proj[r0:r0 + n, :C].double()
        pad = torch.cat([x.new_zeros(taps - 1, C), x])
        y = torch.nn.functional.silu(sum(pad[j:j + n] * conv_w[j].double() for j in range(taps)) + conv_b.double())
        v, b, c = y[:, :H * P].view(n, H, P), y[:, H * P:H * P + G * N].view(n, G, N), y[:, H * P + G * N:].view(n, G, N)
        dt = torch.nn.functional.softplus(proj[r0:r0 + n, C:C + H].double() + dt_bias.double())
        a = torch.exp(-torch.exp(A_log.double()) * dt)
        rep, slot = H // G, len(lens) - 1 - e
        want, after = _recurrence64(c.repeat_interleave(rep, 1), b.repeat_interleave(rep, 1), v * dt[..., None], a[..., None],
                                    None, first[slot])
        assert (out[r0:r0 + n].double() - want).abs().max() <= 2.0 ** -14 * want.abs().max()
        assert (state[slot].double() - after).abs().max() <= 2.0 ** -14 * after.abs().max()


# what the rows of chunks are made from, on no 16 bytes: the bias of the convolution, its one tap's weights, its state
@pytest.mark.parametrize("moved,taps", [("conv_bias", 4), ("conv", 1), ("state", 4)])
def test_state_space_portions_whose_weights_or_state_start_anywhere(moved, taps):
    """The layer takes them token by token.  Against the layer that has them on 16 bytes: rows between differ by their last
    bfloat16 place at most, 2^-8, and so do the results; the memory by what chunks leave, as above."""
    from ccinfer_b200.engine.runtime import Runtime
    from ccinfer_b200.parts import SelectiveStateSpace
    D, H, P, N, G = 64, 4, 32, 64, 2
    lens, g = [1, 170, 200], _gen(taps)
    part = SelectiveStateSpace(D, H, P, N, G, taps, 2, 1e-5, {k: k for k in ("in", "conv", "conv_bias", "dt_bias", "A_log", "D", "norm", "o")})
    w = {s.name: torch.randn(s.shape, generator=g, device="cuda") * (0.125 if len(s.shape) == 2 else 0.5) for s in part.tensor_specs()}
    w = {n: t.to(torch.bfloat16) if n in ("in", "o") else t for n, t in w.items()}
    x = torch.randn((sum(lens), D), generator=g, device="cuda").to(torch.bfloat16)
    memory = torch.randn((len(lens), H, P, N), generator=g, device="cuda")
    ring = torch.randn((len(lens), max(taps - 1, 1), part.conv_width), generator=g, device="cuda").to(torch.bfloat16)

    def elsewhere(t, name):
        if name != moved:
            return t.clone()
        out = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape)
        out.copy_(t)
        assert out.data_ptr() & 15
        return out

    def run(place):
        rt = Runtime("cuda:0", torch.bfloat16, sum(lens), len(lens))
        part.bind(rt, lambda n: place(w[n], n))
        state = {"S": memory.clone(), "conv": place(ring, "state")}
        step = _Step([(3, n) for n in lens], 16, 1).step
        out = part.forward(x, step, None, state).double()
        rt.check_status()
        return out, state["S"].double(), state["conv"].clone()

    (want, after, rows), (got, got_after, got_rows) = run(lambda t, n: t.clone()), run(elsewhere)
    assert (got - want).norm() <= 2.0 ** -8 * want.norm()
    assert (got_after - after).abs().max() <= 2.0 ** -14 * after.abs().max()
    assert torch.equal(got_rows, rows)


# steps and rates up to where a token keeps nothing; three such tokens before slow ones; steps of nothing; whole chunks of both
@pytest.mark.parametrize("decay", ["strong", "then slow", "extreme"])
@pytest.mark.parametrize("H,G,N,P", [(4, 2, 128, 64), (2, 1, 64, 48), (40, 1, 64, 128)])
def test_state_space_chunks_under_strong_decays(H, G, N, P, decay):
    """Every output against float64, within what rounds on its way: queries, keys, weighted scores or memory, and values, each
    right to 2^-17, and one more 2^-17 for the weights, of the sum of magnitudes."""
    k, g = _k(), _gen(H + N + len(decay))
    lens = [1, 64, 65, 150, 200]
    T = sum(lens)

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")

    b, c, v, state = rnd(T, G, N), rnd(T, G, N), rnd(T, H, P), rnd(len(lens), H, P, N)
    u = torch.rand((T, H), generator=g, device="cuda")
    dt = {"strong": 20 * u, "then slow": torch.where(torch.arange(T, device="cuda")[:, None] % 29 < 3, 15 + 5 * u, 1e-3 * u),
          "extreme": torch.where(u < 0.1, 0 * u, torch.where(u < 0.2, 1e6 * u, u))}[decay]
    log_a, log_dt = -16 * dt, dt.log()
    halves = []
    for x in (b, c):
        halves += [x.to(torch.bfloat16), (x - x.to(torch.bfloat16).float()).to(torch.bfloat16)]
    first = state.double()
    out = torch.full((T, H, P), float("nan"), device="cuda")
    cu = [0] + torch.tensor(lens).cumsum(0).tolist()
    k.ssm_chunks((0, *halves, log_a, log_dt), v, state, out, dev(cu), dev(list(range(len(lens)))), 0, len(lens), G, H, N, P)
    for e, n in enumerate(lens):
        s, rep = slice(cu[e], cu[e + 1]), H // G
        args = [c[s].double().repeat_interleave(rep, 1), b[s].double().repeat_interleave(rep, 1),
                v[s].double() * log_dt[s].double().exp()[..., None], log_a[s].double().exp()[..., None], None, first[e]]
        want, after = _recurrence64(*args)
        size, size_after = _recurrence64(*(x if x is None else x.abs() for x in args))
        assert ((out[s].double() - want).abs() <= 5 * 2.0 ** -17 * size + 1e-35).all()
        assert ((state[e].double() - after).abs() <= 5 * 2.0 ** -17 * size_after + 1e-35).all()


def _same_where_finite(got, want, bound):
    """Numbers where the reference has numbers, within ``bound`` of the largest; none where it has none."""
    ok = torch.isfinite(want)
    assert not torch.isfinite(got[~ok]).any()
    assert torch.isfinite(got[ok]).all()
    assert (got.double() - want)[ok].abs().max() <= bound * want[ok].abs().max()


# one number that is none, within a run, at its first and at its last token, in the first and in a later chunk
@pytest.mark.parametrize("at", [0, 37, 47, 64, 90])
@pytest.mark.parametrize("what", ["q", "k", "v", "decay", "beta"])
@pytest.mark.parametrize("rule", ["delta", "head delta", "linear", "head linear"])
def test_recurrence_in_chunks_keeps_what_is_no_number_to_later_tokens(rule, what, at):
    """Tokens before it, requests, heads and value columns beside it stay what they are, as token by token in float64."""
    delta, head = "delta" in rule, "head" in rule
    if what == "beta" and not delta:
        pytest.skip("no such factor")
    H, dk, dv, lens, g = 2, 64, 64, [70, 130], _gen(at + len(what))
    T, row = sum(lens), 70 + at

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")

    q, k = (torch.nn.functional.normalize(rnd(T, H, dk), dim=-1) for _ in range(2))
    v, state, beta = rnd(T, H, dv), rnd(2, H, dv, dk), torch.rand((T, H), generator=g, device="cuda") if delta else None
    a = 1 - 0.1 * torch.rand((T, H) if head else (T, H, dk), generator=g, device="cuda")
    if what == "beta":
        beta[row, 1] = float("nan")
    elif what == "decay" and head:
        a[row, 1] = float("nan")
    else:
        {"q": q, "k": k, "v": v, "decay": a}[what][row, 1, 21] = float("nan") if what == "decay" or at % 2 else float("-inf" if at == 90 else "inf")
    want, after, cu = torch.empty(T, H, dv, dtype=torch.float64, device="cuda"), state.double(), [0, 70, 200]
    for e in range(2):
        s = slice(cu[e], cu[e + 1])
        want[s], after[e] = _recurrence64(q[s].double(), k[s].double(), v[s].double(), (a[s, :, None] if head else a[s]).double(),
                                          beta[s].double() if delta else None, after[e])
    assert torch.isfinite(want[:row]).all() and torch.isfinite(want[:, 0]).all() and not torch.isfinite(want[row, 1]).all()

    def scratch(key, per, shape, dtype):
        return torch.full((T,) + tuple(shape), float("nan"), dtype=dtype, device="cuda")

    out = torch.zeros(T, H, dv, device="cuda")
    _k().chunk_recurrence(scratch, q, k, v, a, beta, state, out, dev(cu), dev([0, 1]), 0, 2, 130, H, H, dk, dv)
    _same_where_finite(out, want, 2.0 ** -14)
    _same_where_finite(state, after, 2.0 ** -14)


@pytest.mark.parametrize("at", [0, 37, 47, 64, 90])
@pytest.mark.parametrize("what", ["b", "c", "x", "log_a", "log_dt"])
@pytest.mark.parametrize("P", [16, 32, 64])
def test_state_space_chunks_keep_what_is_no_number_to_later_tokens(P, what, at):
    """As above; one team, two teams of 16 and (with enough heads) of 32 columns."""
    H, N, lens, g = 40, 64, [70, 130], _gen(at + P + len(what))
    T, row = sum(lens), 70 + at

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")

    b, c, x, state = rnd(T, 2, N).to(torch.bfloat16), rnd(T, 2, N).to(torch.bfloat16), rnd(T, H, P), rnd(2, H, P, N)
    log_dt = torch.log(0.1 + torch.rand((T, H), generator=g, device="cuda"))
    log_a = -0.1 * log_dt.exp()
    {"b": b, "c": c, "x": x, "log_a": log_a, "log_dt": log_dt}[what].view(T, -1)[row, 11] = float("nan") if what[0] == "l" or at % 2 else float("-inf" if at == 90 else "inf")
    want, after, cu = torch.empty(T, H, P, dtype=torch.float64, device="cuda"), state.double(), [0, 70, 200]
    for e in range(2):
        s = slice(cu[e], cu[e + 1])
        want[s], after[e] = _recurrence64(c[s].double().repeat_interleave(H // 2, 1), b[s].double().repeat_interleave(H // 2, 1),
                                          x[s].double() * log_dt[s].double().exp()[..., None], log_a[s].double().exp()[..., None],
                                          None, after[e])
    assert torch.isfinite(want[:row]).all() and not torch.isfinite(want[row]).all() and torch.isfinite(want[row]).any()
    out, zero = torch.full((T, H, P), 7.0, device="cuda"), torch.zeros_like(b)
    _k().ssm_chunks((0, b, zero, c, zero, log_a, log_dt), x, state, out, dev(cu), dev([0, 1]), 0, 2, 2, H, N, P)
    _same_where_finite(out, want, 2.0 ** -14)
    _same_where_finite(state, after, 2.0 ** -14)


class _Step:
    """The arrays of a step whose requests have (cached, new) tokens each, single tokens first, on shuffled pages."""

    def __init__(self, entries, page, seed):
        from ccinfer_b200.engine.step import GroupStep, StepContext
        counts = [n for _, n in entries]
        s = self.step = StepContext()

        def dev(x):
            return torch.tensor(x, dtype=torch.int32, device="cuda")

        s.n_tokens, s.n_entries, s.n_single = sum(counts), len(entries), sum(n == 1 for n in counts)
        s.max_q_len, s.max_ctx = max(counts), max(p + n for p, n in entries)
        s.positions = dev([p + i for p, n in entries for i in range(n)])
        s.entry_of_token = dev([e for e, n in enumerate(counts) for _ in range(n)])
        cu = [0]
        for n in counts:
            cu.append(cu[-1] + n)
        s.cu_q, s.pos0, s.state_slot = dev(cu), dev([p for p, _ in entries]), dev(list(range(len(entries))))
        pages = [-(-(p + n) // page) for p, n in entries]
        order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(seed)).tolist()
        table = torch.full((len(entries), max(pages)), -1, dtype=torch.int32)
        self.slots, at = [], 0
        for e, k in enumerate(pages):
            table[e, :k] = torch.tensor(order[at:at + k])
            at += k
            j = torch.arange(sum(entries[e]))
            self.slots.append((table[e, j // page].long() * page + j % page))
        new = torch.cat([x[p:] for x, (p, _) in zip(self.slots, entries)]).int()
        s.groups = [GroupStep(0, page, sum(pages), None, new.cuda(), table.cuda(), new.numpy(), table.numpy())]


# d, r, rotated, value and latent sizes: one and two blocks of 64 key and value columns, sizes that fill none; windows
# that end in a tile, at a tile's edge, none; heads in groups
@pytest.mark.parametrize("d,r,dims,dv,R,H,window,groups", [
    (64, 64, 64, 128, 512, 4, 130, False), (128, 64, 64, 128, 64, 3, None, False), (64, 32, 16, 64, 128, 2, 128, False),
    (40, 16, 0, 24, 48, 5, 256, True), (72, 8, 0, 72, 512, 2, 1, False), (64, 64, 64, 128, 128, 6, 300, True)])
def test_latent_attention_over_made_keys_and_values(monkeypatch, d, r, dims, dv, R, H, window, groups):
    """Portions beside single tokens: against float64, no further off than the form that stays in the latent space (both round
    queries, keys or latent queries, weights and results to bfloat16 once), with a third in hand for their different sums."""
    from ccinfer_b200 import kernels
    from ccinfer_b200.engine.runtime import Runtime
    from ccinfer_b200.engine.step import LayerCache
    from ccinfer_b200.parts import LatentAttention
    D, page, scale, base, eps = 96, 16, (d + r) ** -0.5, 10000.0, 1e-5
    entries = [(0, 1), (300, 1), (0, 2), (0, 33), (127, 128), (250, 129), (129, 200)]
    g = _gen(d + r + dv + R + H)
    shapes = {"q": (H * (d + r), D), "dkv": (R + r, D), "uk": (H * d, R), "uv": (H * dv, R), "o": (D, H * dv), "g": (H, D)}
    w = {k: (torch.randn(s, generator=g, device="cuda") * s[1] ** -0.5).to(torch.bfloat16) for k, s in shapes.items()}
    w["dkv_norm"], w["sink"] = 1 + 0.1 * torch.randn(R, generator=g, device="cuda"), torch.randn(H, generator=g, device="cuda")
    made = _Step(entries, page, 5)
    step, T = made.step, made.step.n_tokens
    x = torch.randn((T, D), generator=g, device="cuda").to(torch.bfloat16)
    old = [torch.randn((p, R + r), generator=g, device="cuda").to(torch.bfloat16) for p, _ in entries]

    def run():
        part = LatentAttention(D, H, d, r, dv, R, window, scale, base, dims, eps, {k: k for k in w})
        rt = Runtime("cuda:0", torch.bfloat16, T, len(entries))
        part.bind(rt, w.__getitem__)
        cache = torch.zeros((step.groups[0].num_pages, page, R + r), dtype=torch.bfloat16, device="cuda")
        for rows, at in zip(old, made.slots):
            cache.view(-1, R + r)[at[:rows.shape[0]].cuda()] = rows
        out = part.forward(x, step, LayerCache({"latent": cache}, step.groups[0], True), None).double()
        rt.check_status()
        return out

    launched = []
    real = kernels.attention_prefill_dense
    monkeypatch.setattr(kernels, "attention_prefill_dense", lambda *a, **k: (launched.append(a[9]), real(*a, **k)))
    if groups:   # two heads at a time
        monkeypatch.setattr(kernels, "LATENT_DENSE_ELEMENTS", 2 * 64 * (-(-d // 64) - (-dv // 64)) * 4096)
    got = run()
    assert launched and (not groups or len(launched) > 1)
    monkeypatch.setattr(kernels, "LATENT_DENSE_MIN_TOKENS", 1 << 30)
    n = len(launched)
    before = run()
    assert len(launched) == n
    W = {k: v.double() for k, v in w.items()}
    freq = base ** (-torch.arange(0, dims, 2, device="cuda").double() / max(dims, 1))
    want, at = torch.empty(T, D, dtype=torch.float64, device="cuda"), 0

    def turn(y, pos):
        a, h = torch.outer(pos.double(), freq), dims // 2
        u, v = y[..., :h], y[..., h:dims]
        a = a.view(a.shape[0], *([1] * (y.dim() - 2)), h)
        return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin(), y[..., dims:]], -1)

    for (p, m), rows in zip(entries, old):
        h = x[at:at + m].double()
        pos = torch.arange(p, p + m, device="cuda")
        q = (h @ W["q"].T).view(m, H, d + r)
        q = torch.cat([q[..., :d], turn(q[..., d:], pos)], -1)
        c = h @ W["dkv"].T
        new = torch.cat([c[:, :R] / (c[:, :R].square().mean(-1, keepdim=True) + eps).sqrt() * W["dkv_norm"], turn(c[:, R:], pos)], -1)
        seen = torch.cat([rows.double(), new])
        k = torch.cat([(seen[:, :R] @ W["uk"].T).view(-1, H, d), seen[:, None, R:].expand(-1, H, r)], -1)
        v = (seen[:, :R] @ W["uv"].T).view(-1, H, dv)
        s = torch.einsum("ihd,jhd->hij", q, k) * scale
        i, j = pos[:, None], torch.arange(p + m, device="cuda")[None]
        s.masked_fill_((j > i) | ((i - j >= window) if window else (j < 0)), float("-inf"))
        s = torch.softmax(torch.cat([s, W["sink"][:, None, None].expand(H, m, 1)], -1), -1)[..., :-1]
        o = torch.einsum("hij,jhd->ihd", s, v) * torch.sigmoid(h @ W["g"].T)[..., None]
        want[at:at + m] = o.reshape(m, -1) @ W["o"].T
        at += m
    e_new, e_old = ((y - want).norm() / want.norm() for y in (got, before))
    assert e_new <= 1.33 * e_old and e_old < 0.02
    assert (got - want).abs().max() <= 2 * max((before - want).abs().max(), 2.0 ** -8 * want.abs().max())


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("BM", [64, 320])
@pytest.mark.parametrize("N,K", [(256, 64), (40, 72), (264, 200), (1024, 512)])
def test_grouped_products_of_experts(mode, N, K, BM):
    """Experts with no row, one, and numbers around the steps of 32 columns, the accumulators of 256 and the tiles of 64 and 320 rows, against float64: float
    results to K roundings of the sum of magnitudes, 16-bit ones to theirs (2^-8) beside that."""
    k, g = _k(), _gen(N + K + mode)
    counts = [0, 1, 31, 32, 33, 0, 64, 65, 255, 256, 257, 300, 320, 321, 700, 2]
    E, pairs = len(counts), sum(counts)

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(pairs, generator=torch.Generator().manual_seed(1))]
    idx = idx.to(torch.int32).cuda().view(pairs, 1)
    wts = torch.rand((pairs, 1), generator=g, device="cuda") + 0.5
    i32 = dict(dtype=torch.int32, device="cuda")
    src, pos, row_w = torch.empty(pairs, **i32), torch.empty(pairs, **i32), torch.empty(pairs, device="cuda")
    tiles = [torch.empty(k.moe_max_tiles(pairs, E, BM), **i32) for _ in range(3)]
    k.moe_sort(idx, wts, E, BM, src, row_w, pos, *tiles)
    x = rnd(pairs, K).to(torch.bfloat16)
    xs = torch.empty_like(x)
    k.moe_gather_rows(xs, x, src)
    status = torch.zeros(1, **i32)
    w = (rnd(N, E * K) if mode == 1 else rnd(E * N, K)).mul(K ** -0.5).to(torch.bfloat16)
    c = torch.full((pairs, N // 2 if mode == 2 else N), float("nan"), dtype=torch.float32 if mode == 1 else torch.bfloat16, device="cuda")
    k.moe_grouped_tc(c, xs, w, row_w, *tiles, N, K, K if mode == 1 else N, mode, status=status, BM=BM)
    assert int(status.item()) == 0
    order = idx.view(-1)[src.long()].long()   # the expert of every sorted row
    assert (order[1:] >= order[:-1]).all()
    for e in range(E):
        rows = (order == e).nonzero().view(-1)
        if not rows.numel():
            continue
        we = (w[:, e * K:(e + 1) * K] if mode == 1 else w[e * N:(e + 1) * N]).double()
        a = xs[rows].double()
        ref, size = a @ we.T, a.abs() @ we.abs().T
        slack = K * 2.0 ** -24 * size
        got = c[rows].double()
        if mode == 1:
            assert ((got - ref).abs() <= slack).all()
            continue
        rw = row_w[rows].double()[:, None]
        if mode == 0:
            ref, slack = ref.clamp_min(0) ** 2 * rw, 2 * ref.abs() * slack * rw + slack ** 2 * rw
        else:
            gate, up = ref[:, ::2], ref[:, 1::2]
            sg, su = slack[:, ::2], slack[:, 1::2]
            ref = torch.nn.functional.silu(gate) * up * rw
            slack = (1.1 * sg * up.abs() + gate.abs() * su + sg * su) * rw + 2.0 ** -20 * ref.abs()   # (silu's slope is below 1.1)
        assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + slack + 1e-30).all()


# rows around the runs of four, requests of one row beside longer ones (their first rows read the convolution's state),
# heads that fill a warp's 128 channels and that do not; steps of few rows take a warp a row, those with a long request runs
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("more", [0, 1, 3])
@pytest.mark.parametrize("lens,taps,G,H,dk,dv", [
    ([5], 4, 1, 2, 128, 128), ([1, 1, 2, 4, 9], 4, 2, 2, 64, 32), ([3, 1, 1, 7], 2, 1, 1, 4, 128), ([6, 2], 1, 2, 4, 36, 12),
    ([1, 8, 3], 3, 1, 3, 128, 4), ([2, 1], 4, 1, 2, 128, 128)])
def test_delta_rows_in_runs(lens, taps, G, H, dk, dv, more, dtype):
    """Against float64: a row's sums of ``taps`` products, one activation and one norm over dk squares."""
    lens = lens + [16384 // (2 * G + 2 * H) + more] if more else lens
    k, g = _k(), _gen(sum(lens) + taps + dk)
    T, C = sum(lens), 2 * G * dk + H * dv
    ob = -(-C // 8) * 8
    width = ob + -(-H // 8) * 8

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    proj, a = rnd(T, width).to(dtype), rnd(T, H * dk).to(dtype)
    state, w = rnd(len(lens), max(taps - 1, 1), C).to(dtype), 0.5 * rnd(taps, C)
    A_log, dt_bias = rnd(H), rnd(H * dk)
    i32 = dict(dtype=torch.int32, device="cuda")
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), **i32)
    entry = torch.tensor([e for e, n in enumerate(lens) for _ in range(n)], **i32)
    slots = torch.tensor(list(range(len(lens)))[::-1], **i32)
    qn, kn, vv, gg, bb = (torch.full(s, float("nan"), device="cuda") for s in ((T, G, dk), (T, G, dk), (T, H, dv), (T, H, dk), (T, H)))
    k.delta_prepare(proj, (0, G * dk, 2 * G * dk, ob), a, w, taps, state, A_log, dt_bias, entry, cu, slots, qn, kn, vv, gg, bb,
                    G, H, dk, dv, dk ** -0.5, 1e-6)
    x, rows = proj.double(), []
    for e, n in enumerate(lens):
        r0 = int(cu[e])
        pad = torch.cat([state[len(lens) - 1 - e, :taps - 1].double(), x[r0:r0 + n, :C]])
        rows.append(torch.nn.functional.silu(sum(pad[j:j + n] * w[j].double() for j in range(taps))))
    y = torch.cat(rows)
    q, kk, v = y[:, :G * dk].view(T, G, dk), y[:, G * dk:2 * G * dk].view(T, G, dk), y[:, 2 * G * dk:].view(T, H, dv)
    q, kk = (t / (t.square().sum(-1, keepdim=True) + 1e-6).sqrt() for t in (q, kk))
    decay = torch.exp(-torch.exp(A_log.double())[:, None] * torch.nn.functional.softplus(a.double() + dt_bias.double()).view(T, H, dk))
    for got, want in ((qn, q * dk ** -0.5), (kn, kk), (vv, v), (gg, decay), (bb, torch.sigmoid(x[:, ob:ob + H]))):
        assert (got.double() - want).abs().max() <= 64 * 2.0 ** -24 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,P,parts", [(1, 4, 1), (4, 8, 8), (2, 64, 1), (3, 44, 1), (8, 64, 2), (16, 64, 1), (64, 64, 4), (257, 4, 1)])
@pytest.mark.parametrize("few", [True, False])
def test_state_space_gate_and_norm(H, P, parts, few, dtype):
    """Slices of 4 to 1,024 channels in a warp's registers, a longer one and one that starts nowhere in particular; few
    slices: a block each."""
    k, g = _k(), _gen(H * P + parts)
    T, inner = 5 if few else 1024 // parts + 1, H * P

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    o, xs, proj, skip, w = rnd(T, H, P), rnd(T, H, P), rnd(T, 2 * inner + 8).to(dtype), rnd(H), rnd(inner)
    z = proj[:, 8:8 + inner].double()
    v = (o.double() + skip.double()[:, None] * xs.double()).view(T, inner) * torch.nn.functional.silu(z)
    s = v.view(T, parts, -1)
    want = (s / (s.square().mean(-1, keepdim=True) + 1e-5).sqrt()).reshape(T, inner) * w.double()
    for off in (8, 9):
        moved = proj if off == 8 else torch.cat([proj[:, -1:], proj[:, :-1]], 1).contiguous()
        y = torch.full((T, inner), float("nan"), dtype=dtype, device="cuda")
        k.ssm_gate_norm(y, o, xs, moved, off, skip, w, H, P, parts, 1e-5)
        tol = 2.0 ** -8 if dtype == torch.bfloat16 else 64 * 2.0 ** -24
        assert ((y.double() - want).abs() <= tol * want.abs() + 64 * 2.0 ** -24 * want.abs().max()).all()


# one block a row and group, pieces of at least 4, 16 and 32 tiles of 64 keys: contexts at the pieces' edges beside short ones
@pytest.mark.parametrize("rows,min_tiles", [(1, None), (4, None), (8, None), (12, None), (16, None), (24, None), (48, None), (49, None), (5, 1)])
def test_decode_of_ragged_contexts(rows, min_tiles):
    """Every row against float64, split as the plan for so many rows says; counters are left zero."""
    k, g = _k(), _gen(rows)
    nq, nkv, hd, page = 8, 2 if rows == 5 else 8, 128, 16
    edges = [1, 63, 64, 65, 256, 257, 1024, 1025, 2047, 2048, 2049, 4096, 4097, 4160]
    ctx = [edges[i % len(edges)] for i in range(rows)]
    pages = [-(-c // page) for c in ctx]
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(2)).to(torch.int32)
    table, at = torch.full((rows, max(pages)), -1, dtype=torch.int32), 0
    for r, n in enumerate(pages):
        table[r, :n] = order[at:at + n]
        at += n
    kc, vc = (torch.randn((sum(pages), nkv, page, hd), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    q = torch.randn((rows, nq, hd), generator=g, device="cuda").to(torch.bfloat16)
    splits, tiles, in_kernel, n_acc, n_ml = k.attention_decode_plan(rows, nq, nkv, hd)
    assert rows != 48 or (splits, tiles, in_kernel) == (4, 32, True)
    acc, ml = torch.full((n_acc,), float("nan"), device="cuda"), torch.full((n_ml,), float("nan"), device="cuda")
    count = torch.zeros(8192, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.full_like(q, float("nan"))
    i32 = dict(dtype=torch.int32, device="cuda")
    k.attention_decode_tma(q, kc, vc, out, acc, ml, torch.tensor([c - 1 for c in ctx], **i32), torch.arange(rows, **i32),
                           table.cuda(), rows, 0, rows, 0, hd ** -0.5, splits, status=status,
                           merge_counters=count if in_kernel else None, min_tiles=min_tiles or tiles)
    assert int(status.item()) == 0 and int(count.abs().sum()) == 0
    for r, c in enumerate(ctx):
        at = table[r, :pages[r]].long().cuda()
        keys, values = (t[at].transpose(1, 2).reshape(-1, nkv, hd)[:c].double() for t in (kc, vc))
        s = torch.einsum("hd,jhd->hj", q[r].double(), keys.repeat_interleave(nq // nkv, 1)) * hd ** -0.5
        want = torch.einsum("hj,jhd->hd", torch.softmax(s, -1), values.repeat_interleave(nq // nkv, 1))
        # (weights are rounded to bfloat16 for their product, results once more)
        assert (out[r].double() - want).abs().max() <= 2.0 ** -7 * values.abs().max()


# ten pieces of a row, whose results a thread of the merging block holds at once, eleven and more, which go through shared
# memory; heads of one group and of two blocks of a group
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("extras", [False, True])
@pytest.mark.parametrize("nq,nkv", [(8, 2), (40, 2)])
@pytest.mark.parametrize("ctx,pieces", [(2304, 9), (2560, 10), (2561, 11), (4160, 17), (8192, 32)])
def test_decode_merges_pieces_of_a_long_context(ctx, pieces, nq, nkv, extras, fused):
    """One request against float64, with a sink and a gate of the output's heads or without."""
    k, g = _k(), _gen(ctx + nq + extras)
    hd, page = 128, 16
    n = ctx // page + 1

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)

    table = torch.randperm(n, generator=torch.Generator().manual_seed(2)).to(torch.int32).view(1, n)
    kc, vc, qkv = rnd(n, nkv, page, hd), rnd(n, nkv, page, hd), rnd(1, (nq + 2 * nkv) * hd)
    q = qkv[:, :nq * hd].view(1, nq, hd).contiguous()
    at = table[0].long().cuda()
    keys, values = (t[at].transpose(1, 2).reshape(-1, nkv, hd)[:ctx].double() for t in (kc, vc))
    if fused:   # (the row's own key and value come with it)
        keys[-1], values[-1] = (qkv[0, (nq + i * nkv) * hd:(nq + (i + 1) * nkv) * hd].view(nkv, hd).double() for i in (0, 1))
    sink, gate = (4 * torch.randn(nq, generator=g, device="cuda"), rnd(1, nq + 8)) if extras else (None, None)
    splits, tiles, in_kernel, n_acc, n_ml = k.attention_decode_plan(1, nq, nkv, hd)
    assert in_kernel and min(splits, -(-(-(-ctx // 64)) // tiles)) == pieces
    i32 = dict(dtype=torch.int32, device="cuda")
    acc, ml = torch.full((n_acc,), float("nan"), device="cuda"), torch.full((n_ml,), float("nan"), device="cuda")
    count, status, out = torch.zeros(8192, **i32), torch.zeros(1, **i32), torch.full_like(q, float("nan"))
    args = (kc, vc, out, acc, ml, torch.tensor([ctx - 1], **i32), torch.zeros(1, **i32), table.cuda(), 1, 0, 1)
    more = dict(status=status, merge_counters=count, sink=sink, gate=gate, min_tiles=tiles)
    if fused:
        k.attention_decode_tma_fused(qkv, *args, nq, 0, hd ** -0.5, splits, None, None, 1e-6, torch.zeros(hd // 2, device="cuda"), **more)
    else:
        k.attention_decode_tma(q, *args, 0, hd ** -0.5, splits, **more)
    assert int(status.item()) == 0 and int(count.abs().sum()) == 0
    assert (torch.isfinite(ml[:2 * nq * splits].view(nq, splits, 2)).all(-1).sum(-1) == pieces).all()
    s = torch.einsum("hd,jhd->hj", q[0].double(), keys.repeat_interleave(nq // nkv, 1)) * hd ** -0.5
    if extras:
        s = torch.cat([s, sink.double()[:, None]], 1)
    want = torch.einsum("hj,jhd->hd", torch.softmax(s, -1)[:, :ctx], values.repeat_interleave(nq // nkv, 1))
    if extras:
        want *= torch.sigmoid(gate[0, :nq].double())[:, None]
    # (weights are rounded to bfloat16 for their product, results once more)
    assert (out[0].double() - want).abs().max() <= 2.0 ** -7 * values.abs().max()


# rows whose lengths are alike stay in one piece (or two: 16 rows), a long one among short ones is cut; 40 rows: always
@pytest.mark.parametrize("rows,even_pieces,ragged_pieces", [(16, 2, 4), (24, 1, 3), (36, 1, 3), (40, 3, 3)])
@pytest.mark.parametrize("window", [0, 3000])
def test_decode_cuts_long_rows_of_ragged_batches_only(rows, even_pieces, ragged_pieces, window):
    """Every row against float64, and how many pieces left results (a row of one piece leaves none)."""
    k, g = _k(), _gen(rows)
    nq, nkv, hd, page, most = 16, 8, 128, 64, 4160
    n = -(-most // page)
    kc, vc = (torch.randn((n, nkv, page, hd), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    table = torch.stack([torch.randperm(n, generator=torch.Generator().manual_seed(r)) for r in range(rows)]).to(torch.int32)
    q = torch.randn((rows, nq, hd), generator=g, device="cuda").to(torch.bfloat16)
    splits, tiles, in_kernel, n_acc, n_ml = k.attention_decode_plan(rows, nq, nkv, hd)
    even = k.attention_decode_even(rows, nq, nkv, hd)
    i32 = dict(dtype=torch.int32, device="cuda")
    count, status = torch.zeros(8192, **i32), torch.zeros(1, **i32)
    for ragged in (False, True):
        ctx = [most - 5 * r for r in range(rows)] if not ragged else [most if r == 7 else 100 + 3 * r for r in range(rows)]
        acc, ml, out = torch.full((n_acc,), float("nan"), device="cuda"), torch.full((n_ml,), float("nan"), device="cuda"), torch.full_like(q, float("nan"))
        entry = torch.arange(rows, **i32)
        entry[3] = -1   # a row that pads the step
        k.attention_decode_tma(q, kc, vc, out, acc, ml, torch.tensor([c - 1 for c in ctx], **i32), entry, table.cuda(), rows, 0, rows,
                               window, hd ** -0.5, splits, status=status, merge_counters=count, min_tiles=tiles, even=even)
        assert int(status.item()) == 0 and int(count.abs().sum()) == 0
        left = torch.isfinite(ml[:2 * rows * nq * splits].view(rows, nq, splits, 2)).all(-1).sum(-1)
        if not window:
            assert (left[7] == (ragged_pieces if ragged else even_pieces if even_pieces > 1 else 0)).all()
        for r in (0, 3, 7, rows - 1):
            if r == 3:
                assert not out[r].any()
                continue
            at = table[r].long().cuda()
            keys, values = (t[at].transpose(1, 2).reshape(-1, nkv, hd)[max(0, ctx[r] - window) if window else 0:ctx[r]].double() for t in (kc, vc))
            s = torch.einsum("hd,jhd->hj", q[r].double(), keys.repeat_interleave(nq // nkv, 1)) * hd ** -0.5
            want = torch.einsum("hj,jhd->hd", torch.softmax(s, -1), values.repeat_interleave(nq // nkv, 1))
            assert (out[r].double() - want).abs().max() <= 2.0 ** -7 * values.abs().max()


# one block a head from 16 requests of 32 heads on where key and value sizes are over 64; else a cluster a head
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("E,G,H,dk,dv", [(16, 32, 32, 128, 128), (16, 16, 32, 100, 68), (17, 16, 32, 68, 128), (15, 32, 32, 128, 128),
                                         (16, 32, 32, 128, 64), (16, 32, 32, 64, 128), (32, 8, 16, 128, 128)])
def test_delta_step_of_many_heads(E, G, H, dk, dv, dtype):
    """One token of each request against float64; a request without a slot leaves its row and every state alone."""
    k, g = _k(), _gen(E + dk + dv)
    C = 2 * G * dk + H * dv
    pad = -(-(C + 2 * H) // 8) * 8
    off, width = (0, G * dk, 2 * G * dk, C, C + H, pad), pad + H * dv

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    conv_w, A_log, dt_bias, w, S = rnd(1, C), rnd(H), rnd(H), rnd(dv), rnd(E, H, dv, dk)
    rule = k.HeadDelta(off, conv_w, A_log, dt_bias, G, H, dk, dv, dk ** -0.5, 1e-6)
    proj, ring, before = rnd(E, width).to(dtype), torch.zeros(E, 1, C, dtype=dtype, device="cuda"), S.double()
    i32 = dict(dtype=torch.int32, device="cuda")
    slots = torch.arange(E - 1, -1, -1, **i32)
    slots[1] = -1
    y = torch.full((E, H * dv), 7.0, dtype=dtype, device="cuda")
    k.delta_head_step(rule, proj, ring, S, w, 1e-5, torch.full((E,), 9, **i32), torch.arange(E + 1, **i32), slots, y, E)
    x = proj.double()
    c = torch.nn.functional.silu(x[:, :C] * conv_w[0].double())
    q, key = (t.reshape(E, G, dk).repeat_interleave(H // G, 1) for t in (c[:, :G * dk], c[:, G * dk:2 * G * dk]))
    q, key = (t / (t.square().sum(-1, keepdim=True) + 1e-6).sqrt() for t in (q, key))
    v, beta = c[:, 2 * G * dk:].view(E, H, dv), torch.sigmoid(x[:, C:C + H])
    decay = torch.exp(-torch.exp(A_log.double()) * torch.nn.functional.softplus(x[:, C + H:C + 2 * H] + dt_bias.double()))
    old = before[slots.long()] * decay[..., None, None]
    put = beta[..., None] * (v - torch.einsum("ehvk,ehk->ehv", old, key))
    after = old + put[..., None] * key[:, :, None]
    o = torch.einsum("ehvk,ehk->ehv", after, q) * dk ** -0.5
    o = o / (o.square().mean(-1, keepdim=True) + 1e-5).sqrt() * w.double()
    want = o.reshape(E, H * dv) * torch.nn.functional.silu(x[:, pad:])
    want[1], after[1] = 7.0, before[E - 2]
    # (sums of up to 128 products in any order; y is rounded once)
    assert (S[torch.arange(E - 1, -1, -1)].double() - after).abs().max() <= 128 * 2.0 ** -24 * after.abs().max()
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0
    assert ((y.double() - want).abs() <= tol * want.abs() + 256 * 2.0 ** -24 * want.abs().max()).all()


# enough rows that a thread takes four of them: requests of one row (their state moves on) before long ones that end within a
# run and beside its edges; rows of no request, and a request without a slot
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("taps,H,P,G,N,last", [(4, 4, 64, 1, 64, 0), (3, 8, 16, 2, 4, 1), (2, 2, 128, 2, 128, 2), (1, 4, 64, 1, 64, 3)])
def test_state_space_rows_in_runs(taps, H, P, G, N, last, dtype):
    """Against float64: a row's sum of ``taps`` products and its activation, a head's step and decay."""
    k, g = _k(), _gen(taps + H + N)
    C = H * P + 2 * G * N
    lens = [1, 1, 1, 2, 3, 9, 1 << 10, 1000000 // (C // 4 + H) + last]
    T = sum(lens) + 2   # (two rows that pad the step)
    first = 5           # rows from the fourth request on go to the chunks

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    proj, width = rnd(T, C + 8 + -(-H // 8) * 8).to(dtype), C + 8
    conv_w, conv_b, dt_bias, A_log = 0.5 * rnd(taps, C), rnd(C), rnd(H) - 2, torch.log(1 + rnd(H).abs())
    conv = rnd(len(lens), max(taps - 1, 1), C).to(dtype)
    old = conv.double()
    i32 = dict(dtype=torch.int32, device="cuda")
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), **i32)
    entry = torch.tensor([e for e, n in enumerate(lens) for _ in range(n)] + [-1, -1], **i32)
    slots = torch.arange(len(lens) - 1, -1, -1, **i32)
    slots[4] = -1
    nan = float("nan")
    xs, bs, cs = (torch.full(s, nan, device="cuda") for s in ((T, H, P), (T, G, N), (T, G, N)))
    dts, decay, log_a, log_dt = (torch.full((T, H), nan, device="cuda") for _ in range(4))
    halves = [torch.full((T, G, N), nan, dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    chunk = (first, *halves, log_a, log_dt) if dtype == torch.bfloat16 else None
    k.ssm_prepare(proj, 8, width, conv_w, conv_b, taps, conv if taps > 1 else None, A_log, dt_bias, entry, cu, slots, xs, bs, cs,
                  dts, decay, H, P, G, N, shift_single=True, chunk=chunk)
    x, rows, after = proj.double(), [], old.clone()
    for e, n in enumerate(lens):
        r0, at = int(cu[e]), len(lens) - 1 - e
        part = x[r0:r0 + n, 8:8 + C]
        before = old[at, :taps - 1] if e != 4 else torch.zeros_like(old[0, :taps - 1])
        pad = torch.cat([before, part])
        rows.append(torch.nn.functional.silu(conv_b.double() + sum(pad[j:j + n] * conv_w[j].double() for j in range(taps))))
        if n == 1 and taps > 1:
            after[at, :taps - 1] = pad[1:]
    want = torch.cat(rows + [torch.zeros_like(x[:2, :C])])
    tol = 64 * 2.0 ** -24 * float(want.abs().max())
    b, c = want[:, H * P:H * P + G * N].view(T, G, N), want[:, H * P + G * N:].view(T, G, N)
    dt = torch.nn.functional.softplus(x[:, width:width + H] + dt_bias.double())
    n1 = first if chunk is not None else T
    assert (xs.double() - want[:, :H * P].view(T, H, P)).abs().max() <= tol
    assert (bs[:n1].double() - b[:n1]).abs().max() <= tol and (cs[:n1].double() - c[:n1]).abs().max() <= tol
    live = entry[:n1] >= 0
    assert (dts[:n1][live].double() - dt[:n1][live]).abs().max() <= 64 * 2.0 ** -24 * dt.max()
    assert (decay[:n1][live].double() - torch.exp(-A_log.double().exp() * dt[:n1][live])).abs().max() <= 64 * 2.0 ** -24 * 8
    if chunk is not None:
        for hi, lo, w in ((halves[0], halves[1], b), (halves[2], halves[3], c)):   # (two bfloat16: 2^-17)
            assert (hi[n1:].double() + lo[n1:].double() - w[n1:]).abs().max() <= 2.0 ** -17 * w.abs().max() + tol
        s = slice(n1, T - 2)
        assert (log_a[s].double() + A_log.double().exp() * dt[s]).abs().max() <= 64 * 2.0 ** -24 * 16 * dt.max()
        assert (log_dt[s].double() - dt[s].log()).abs().max() <= 64 * 2.0 ** -24 * 16
    assert torch.equal(conv.double(), after)


# sizes of a state that fill no lane's four, no warp's eight or sixteen channels; more requests than SMs; slots that are none
@pytest.mark.parametrize("kind", ["delta", "linear", "state space"])
@pytest.mark.parametrize("E,H,G,dk,dv", [(9, 17, 17, 128, 128), (160, 2, 1, 68, 64), (75, 8, 4, 100, 36), (40, 10, 5, 124, 68),
                                        (150, 1, 1, 128, 128), (3, 50, 25, 72, 128)])
def test_single_tokens_of_many_requests_stream_their_states(kind, E, H, G, dk, dv):
    """One token each against float64: sums of dk products, sizes of some 1; a state that no request of the step has stays."""
    from ccinfer_b200 import kernels as k
    if kind == "linear":
        G = H
    assert E * H * dv >= 148 * 128   # (from here on)
    g = _gen(E + H + dk + dv)

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")

    q, kk = (torch.nn.functional.normalize(rnd(E, G, dk), dim=-1) for _ in range(2))
    v, beta = rnd(E, H, dv), torch.rand((E, H), generator=g, device="cuda")
    decay = torch.rand((E, H) if kind == "state space" else (E, H, dk), generator=g, device="cuda")
    state = rnd(E + 3, H, dv, dk)
    slots = torch.randperm(E + 3, generator=torch.Generator().manual_seed(E)).tolist()[:E]
    dead = {1, E - 1}
    before, out = state.double(), torch.full((E, H, dv), float("nan"), device="cuda")
    args = (dev(list(range(E + 1))), dev([-1 if e in dead else s for e, s in enumerate(slots)]), E)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    if kind == "delta":
        k.delta_recurrence(q, kk, v, decay, beta, state, out, *args, G, H, dk, dv, single=True, status=status)
    elif kind == "linear":
        k.gated_linear_recurrence(q, kk, v, decay, state, out, *args, H, dk, dv, single=True, status=status)
    else:
        k.ssm_recurrence(q, kk, v, decay, beta, state, out, *args, G, H, dk, dv, single=True, status=status)
    rep = H // G
    want, after = out.double(), before.clone()
    for e, s in enumerate(slots):
        if e in dead:
            continue
        put = v[e:e + 1].double() * (beta[e:e + 1, :, None].double() if kind == "state space" else 1)
        want[e:e + 1], after[s] = _recurrence64(
            q[e:e + 1].double().repeat_interleave(rep, 1), kk[e:e + 1].double().repeat_interleave(rep, 1), put,
            (decay[e:e + 1, :, None] if kind == "state space" else decay[e:e + 1]).double(),
            beta[e:e + 1].double() if kind == "delta" else None, before[s])
    live = [e for e in range(E) if e not in dead]
    assert int(status) == 0 and torch.isnan(out[list(dead)]).all()   # (nobody writes the others)
    # a sum of dk terms in float, in some ten additions one after another, and few operations around it
    assert (out[live].double() - want[live]).abs().max() <= 2.0 ** -20 * want[live].abs().max()
    assert (state.double() - after).abs().max() <= 2.0 ** -20 * after.abs().max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("E,H,G,dk,dv,taps", [(5, 37, 37, 128, 128, 4), (150, 2, 1, 68, 36, 1), (30, 10, 5, 100, 64, 6), (40, 8, 2, 72, 100, 2)])
def test_one_token_of_the_head_delta_rule_beside_its_blocks(E, H, G, dk, dv, taps, dtype):
    """The stream of states beside the blocks of few requests (the same step in parts small enough for them)."""
    from ccinfer_b200 import kernels as k
    g = _gen(E + H + dk + dv)

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    C = 2 * G * dk + H * dv
    offsets = [0, G * dk, 2 * G * dk, C, C + H, C + 2 * H]
    width = -(-(C + 2 * H + H * dv) // 8) * 8
    proj, w = rnd(E, width).to(dtype), rnd(dv)
    rule = k.HeadDelta(tuple(offsets), 0.5 * rnd(taps, C), torch.log(1 + 15 * torch.rand(H, generator=g, device="cuda")), rnd(H) - 2,
                       G, H, dk, dv, dk ** -0.5, 1e-6)
    ring, state = rnd(E, taps, C).to(dtype), rnd(E, H, dv, dk)
    i32 = {"dtype": torch.int32, "device": "cuda"}
    pos, slots = torch.arange(E, **i32) % 7, torch.randperm(E, generator=torch.Generator().manual_seed(1)).to(**i32)
    slots[2] = -1
    status = torch.zeros(1, **i32)
    got = [t.clone() for t in (ring, state)] + [torch.zeros(E, H * dv, dtype=dtype, device="cuda")]
    want = [t.clone() for t in (ring, state)] + [torch.zeros(E, H * dv, dtype=dtype, device="cuda")]
    assert E * H >= 148
    k.delta_head_step(rule, proj, got[0], got[1], w, 1e-5, pos, torch.arange(E + 1, **i32), slots, got[2], E, status=status)
    n = 147 // H   # (requests of a part)
    for e in range(0, E, n):
        m = min(n, E - e)
        k.delta_head_step(rule, proj[e:e + m], want[0], want[1], w, 1e-5, pos[e:e + m].contiguous(), torch.arange(m + 1, **i32),
                          slots[e:e + m].contiguous(), want[2][e:e + m], m)
    assert int(status) == 0 and torch.equal(got[0], want[0])
    # the same float operations but for the order of sums of dk and dv terms; rows rounded to the compute type
    assert (got[1] - want[1]).abs().max() <= 2.0 ** -19 * want[1].abs().max()
    near = 2.0 ** -19 if dtype == torch.float32 else 2.0 ** -7
    assert (got[2].float() - want[2].float()).abs().max() <= near * want[2].float().abs().max()


# one and two tiles of heads, whole and in part; pages smaller than, as and larger than a tile of 32 keys; rows in one piece and many
@pytest.mark.parametrize("H,R,r,page,window,splits", [
    (16, 512, 64, 16, 1 << 30, 1), (5, 512, 64, 8, 1 << 30, 7), (32, 512, 64, 32, 100, 3), (17, 256, 64, 64, 1 << 30, 64), (1, 128, 64, 16, 33, 2),
    (48, 128, 64, 8, 1 << 30, 1), (16, 112, 80, 16, 64, 5)])
def test_latent_attention_of_single_tokens(H, R, r, page, window, splits):
    """Against float64, in pages anywhere.  What a token does not see (rows after it, pages before its window) is no number.
    Weights and results are rounded to bfloat16: 2^-9 of the largest coordinate each."""
    k, g = _k(), _gen(H + R + page + splits)
    ctx = [1, 31, 32, 33, 64, 200, 999]   # (keys that a token sees without a window, its own among them)
    E, W, scale = len(ctx) + 1, R + r, 0.06
    pages = [-(-n // page) for n in ctx] + [1]
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(splits)).tolist()
    cache = torch.full((sum(pages), page, W), float("nan"), dtype=torch.bfloat16, device="cuda")
    table = torch.full((E, max(pages)), -1, dtype=torch.int32)
    qa = torch.randn((E, H, W), generator=g, device="cuda").to(torch.bfloat16).float()
    sink = torch.randn(H, generator=g, device="cuda")
    gate = torch.randn((E, H + 3), generator=g, device="cuda").to(torch.bfloat16)[:, :H]
    want, largest = torch.zeros(E, H, R, dtype=torch.float64, device="cuda"), 0.0
    at = 0
    for e, n in enumerate(ctx):
        lo = max(0, n - window)
        rows = torch.randn((n, W), generator=g, device="cuda").to(torch.bfloat16)
        for i in range(pages[e]):
            if (i + 1) * page <= lo:
                continue   # (a page before the window is gone)
            table[e, i] = order[at + i]
            a, b = max(lo, i * page), min(n, (i + 1) * page)
            cache[order[at + i], a - i * page:b - i * page] = rows[a:b]
        at += pages[e]
        c = rows[lo:].double()
        s = torch.cat([qa[e].double() @ c.T * scale, sink.double()[:, None]], 1)
        want[e] = torch.softmax(s, -1)[:, :-1] @ c[:, :R] * torch.sigmoid(gate[e].double())[:, None]
        largest = max(largest, float(c[:, :R].abs().max()))

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")

    out = torch.full((E, H, R), 7.0, dtype=torch.bfloat16, device="cuda")
    want[E - 1] = 7.0   # (a row that pads the step)
    acc, ml = (torch.full((E * H * splits * m,), float("nan"), device="cuda") for m in (R, 2))
    status = dev([0])
    k.latent_attention_mma(qa, cache, sink, gate, out, dev(list(range(E + 1))), dev([n - 1 for n in ctx] + [0]),
                           dev(list(range(E - 1)) + [-1]), table.cuda(), 0, E, 1, page, window, scale, splits, acc, ml, status)
    assert int(status) == 0
    assert (out.double() - want).abs().max() <= 2.0 ** -8 * largest
    table[5, (ctx[5] - 1) // page] = sum(pages)   # a page that does not exist
    k.latent_attention_mma(qa, cache, sink, gate, out, dev(list(range(E + 1))), dev([n - 1 for n in ctx] + [0]),
                           dev(list(range(E - 1)) + [-1]), table.cuda(), 0, E, 1, page, window, scale, splits, acc, ml, status)
    assert int(status) == 4


# rows x heads from which on a warp takes four heads: left-over heads, lanes without channels, a gate inside wider rows
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("silu", [False, True])
@pytest.mark.parametrize("T,H,dv", [(2763, 3, 128), (8289, 1, 4), (830, 10, 100), (8287, 1, 64), (3947, 3, 128), (11841, 1, 4)])
def test_gated_head_norm_of_many_rows(T, H, dv, silu, dtype):
    """Against float64: the norm, a weight and the gate, rounded once."""
    k, g = _k(), _gen(T + dv)
    o, w = torch.randn((T, H, dv), generator=g, device="cuda"), torch.randn(dv, generator=g, device="cuda")
    wide = 4 * torch.randn((T, H * dv + 8), generator=g, device="cuda").to(dtype)
    gate, y = wide[:, 8:], torch.full((T, H * dv), float("nan"), dtype=dtype, device="cuda")
    k.gated_head_rmsnorm(y, o, gate, w, H, dv, 1e-5, silu_gate=silu)
    z = gate.double().view(T, H, dv)
    x = o.double()
    want = x / torch.sqrt(x.square().mean(-1, keepdim=True) + 1e-5) * w.double() * torch.sigmoid(z) * (z if silu else 1)
    rel = (2.0 ** -8 if dtype == torch.bfloat16 else 0) + 2.0 ** -19   # (a sum of dv squares and some twenty operations; the rounding)
    assert ((y.double().view(T, H, dv) - want).abs() <= rel * want.abs() + 1e-30).all()


# portions around the runs of 16 and chunks of 64, behind single tokens; rows and decays inside wider rows; with and without a bias
@pytest.mark.parametrize("H,dk,dv,tau,bias", [(3, 128, 128, 16.0, True), (2, 64, 32, 1.0, False), (1, 128, 64, 0.5, True)])
def test_gated_linear_chunks_from_the_projections_rows(H, dk, dv, tau, bias):
    """Against float64 from the same bfloat16 rows: operands as two bfloat16 (2^-17 each), as the chunks from float rows."""
    k, g = _k(), _gen(H + dk + dv)
    lens, first = [1, 1, 2, 15, 17, 64, 65, 130], 2
    T, oq, ok, ov = sum(lens), 4, 4 + H * dk, 8 + 2 * H * dk
    proj = torch.randn((T, 12 + 2 * H * dk + H * dv), generator=g, device="cuda").to(torch.bfloat16)
    a = (3 * torch.randn((T, H * dk + 1), generator=g, device="cuda")).to(torch.bfloat16)[:, 1:]
    b = 2 + torch.randn(H * dk, generator=g, device="cuda") if bias else None
    state = torch.randn((len(lens) + 1, H, dv, dk), generator=g, device="cuda")
    slots = torch.randperm(len(lens) + 1, generator=torch.Generator().manual_seed(2)).tolist()[:len(lens)]
    slots[4] = -1
    cu = [0] + torch.tensor(lens).cumsum(0).tolist()

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")

    def scratch(key, per, shape, dtype):
        return torch.full((T if per == "tokens" else T // 64 + len(lens),) + tuple(shape), float("nan"), dtype=dtype, device="cuda")

    q, key = (proj[:, o:o + H * dk].double().view(T, H, dk) for o in (oq, ok))
    v = proj[:, ov:ov + H * dv].double().view(T, H, dv)
    decay = torch.sigmoid(a.double() + (b.double() if bias else 0)).view(T, H, dk) ** (1 / tau)
    out, after = torch.full((T, H, dv), 7.0, device="cuda"), state.double()
    want = out.double()
    for e, slot in enumerate(slots):
        if e >= first and slot >= 0:
            s = slice(cu[e], cu[e + 1])
            want[s], after[slot] = _recurrence64(0.3 * q[s], key[s], v[s], decay[s], None, state[slot].double())
    work = [torch.full((T, H, dk), float("nan"), device="cuda") for _ in range(2)]
    k.chunk_recurrence_raw(scratch, proj, (oq, ok, ov), a, b, *work, state, out, dev(cu), dev(slots), first, len(lens) - first,
                           max(lens), H, dk, dv, 0.3, tau)
    assert (out.double() - want).abs().max() <= 2.0 ** -14 * want.abs().max()
    assert (state.double() - after).abs().max() <= 2.0 ** -14 * after.abs().max()


# slow decays, ordinary ones and such that keep nothing of a run; the rows' decays inside wider rows
@pytest.mark.parametrize("shift", [-8.0, 0.0, 6.0])
@pytest.mark.parametrize("H,G,dk,dv", [(2, 2, 128, 128), (4, 2, 64, 32)])
def test_delta_chunks_that_make_their_decays(H, G, dk, dv, shift):
    """Against float64 from the same bfloat16 rows, and that only the single tokens' decays are made beforehand."""
    k, g = _k(), _gen(H + dk + dv + int(shift))
    lens, first = [1, 1, 2, 15, 17, 64, 65, 130], 2
    T = sum(lens)

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")

    def scratch(key, per, shape, dtype):
        return torch.full((T if per == "tokens" else T // 64 + len(lens),) + tuple(shape), float("nan"), dtype=dtype, device="cuda")

    cu, slots = [0] + torch.tensor(lens).cumsum(0).tolist(), list(range(len(lens)))[::-1]
    slots[4] = -1
    a, A_log, dt_bias = rnd(T, H * dk + 5).bfloat16()[:, 5:], rnd(H), rnd(H * dk) + shift
    ob = 2 * G * dk + H * dv
    proj, state = rnd(T, ob + H).bfloat16(), rnd(len(lens), H, dv, dk)
    entry = dev([e for e, n in enumerate(lens) for _ in range(n)])
    rows = [torch.full(s, float("nan"), device="cuda") for s in ((T, G, dk), (T, G, dk), (T, H, dv), (T, H, dk), (T, H))]
    k.delta_prepare(proj, (0, G * dk, 2 * G * dk, ob), a, rnd(1, ob), 1, rnd(len(lens), 0, ob).bfloat16(), A_log, dt_bias, entry, dev(cu),
                    dev(slots), *rows, G, H, dk, dv, dk ** -0.5, 1e-6, decays=first)
    assert torch.isfinite(rows[3][:first]).all() and torch.isnan(rows[3][first:]).all()
    q, kk, v, _, beta = (r.double() for r in rows)
    decay = torch.exp(-torch.exp(A_log.double())[:, None] * torch.nn.functional.softplus(a.double() + dt_bias.double()).view(T, H, dk))
    out, after = torch.full((T, H, dv), 7.0, device="cuda"), state.double()
    want = out.double()
    for e, slot in enumerate(slots):
        if e >= first and slot >= 0:
            s = slice(cu[e], cu[e + 1])
            want[s], after[slot] = _recurrence64(q[s].repeat_interleave(H // G, 1), kk[s].repeat_interleave(H // G, 1), v[s], decay[s],
                                                 beta[s], state[slot].double())
    k.chunk_recurrence(scratch, *rows, state, out, dev(cu), dev(slots), first, len(lens) - first, max(lens), G, H, dk, dv,
                       decay_rows=(a, dt_bias, A_log))
    assert (out.double() - want).abs().max() <= 2.0 ** -14 * want.abs().max()
    assert (state.double() - after).abs().max() <= 2.0 ** -14 * after.abs().max()


# walks in which a tile is cut by the ring's end or passes over slots (rows / 32 rounded up: 8 6 6 10, 9 8 3, 7 8 8 8, 5 5 5 5 5 6 ...),
# by one pair of SMs in this order, and by all of them over many columns
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("K", [64, 256, 2048])
@pytest.mark.parametrize("N,sms", [(256, 2), (4096, None)])
def test_grouped_products_of_long_walks(N, sms, K, mode, monkeypatch):
    """Tensor memory taken in turn by tiles of mixed sizes, against float64 with the bounds of
    test_grouped_products_of_experts: every walk goes round it many times (as tests/test_slot_ring.py follows)."""
    k, g = _k(), _gen(N + K + mode)
    slots = [8, 6, 6, 10, 9, 8, 3, 7, 8, 8, 8, 8, 6, 8, 8, 5, 5, 5, 5, 5, 6, 1, 10, 10, 10, 1, 1, 9, 9, 2, 4]
    slots += torch.randint(1, 11, (29,), generator=torch.Generator().manual_seed(K)).tolist()
    rows = [32 * s - (7 * i) % 32 for i, s in enumerate(slots)]
    E, pairs = 16, sum(rows)
    if sms is not None:
        monkeypatch.setattr(k, "sm_count", lambda: sms)
    else:
        assert len(rows) * (N // 256) >= 12 * (k.sm_count() // 2)

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")

    r0 = [0] + torch.tensor(rows).cumsum(0).tolist()[:-1]
    xs, row_w = rnd(pairs, K).to(torch.bfloat16), torch.rand(pairs, generator=g, device="cuda") + 0.5
    w = (rnd(N, E * K) if mode == 1 else rnd(E * N, K)).mul(K ** -0.5).to(torch.bfloat16)
    c = torch.full((pairs, N // 2 if mode == 2 else N), float("nan"), dtype=torch.float32 if mode == 1 else torch.bfloat16, device="cuda")
    status = dev([0])
    k.moe_grouped_tc(c, xs, w, row_w, dev([i % E for i in range(len(rows))] + [0]), dev(r0 + [0]), dev(rows + [0]), N, K,
                     K if mode == 1 else N, mode, status=status, BM=320)
    assert int(status.item()) == 0
    for i, n in enumerate(rows):
        e, at = i % E, slice(r0[i], r0[i] + n)
        we = (w[:, e * K:(e + 1) * K] if mode == 1 else w[e * N:(e + 1) * N]).double()
        a, got = xs[at].double(), c[at].double()
        ref, size = a @ we.T, a.abs() @ we.abs().T
        slack = K * 2.0 ** -24 * size
        if mode == 1:
            assert ((got - ref).abs() <= slack).all(), i
            continue
        rw = row_w[at].double()[:, None]
        if mode == 0:
            ref, slack = ref.clamp_min(0) ** 2 * rw, 2 * ref.abs() * slack * rw + slack ** 2 * rw
        else:
            gate, up = ref[:, ::2], ref[:, 1::2]
            sg, su = slack[:, ::2], slack[:, 1::2]
            ref = torch.nn.functional.silu(gate) * up * rw
            slack = (1.1 * sg * up.abs() + gate.abs() * su + sg * su) * rw + 2.0 ** -20 * ref.abs()   # (silu's slope is below 1.1)
        assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + slack + 1e-30).all(), i


@pytest.mark.parametrize("pdl", [1, 2])
@pytest.mark.parametrize("kind", ["delta", "linear", "state space"])
@pytest.mark.parametrize("E,H,dk,dv", [(48, 16, 128, 128), (160, 2, 68, 64), (150, 1, 128, 128)])
def test_tokens_in_a_row_on_the_same_states(kind, pdl, E, H, dk, dv):
    """Calls directly behind one another, each with the states that the last one left, with early launches: against float64 as in
    test_single_tokens_of_many_requests_stream_their_states, whose bound a token of each of four calls adds once."""
    k, g = _k(), _gen(E + H + dk + dv + pdl)
    n = 4

    def rnd(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    q, kk = (torch.nn.functional.normalize(rnd(n, E, H, dk), dim=-1) for _ in range(2))
    v, beta = rnd(n, E, H, dv), torch.rand((n, E, H), generator=g, device="cuda")
    decay = 0.5 + 0.5 * torch.rand((n, E, H) if kind == "state space" else (n, E, H, dk), generator=g, device="cuda")
    state, out = rnd(E, H, dv, dk), torch.full((n, E, H, dv), float("nan"), device="cuda")
    before = state.double()
    args = (torch.arange(E + 1, dtype=torch.int32, device="cuda"), torch.arange(E, dtype=torch.int32, device="cuda").flip(0), E)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    was = k._pdl
    k.set_pdl(pdl)
    try:
        for i in range(n):
            if kind == "delta":
                k.delta_recurrence(q[i], kk[i], v[i], decay[i], beta[i], state, out[i], *args, H, H, dk, dv, single=True, status=status)
            elif kind == "linear":
                k.gated_linear_recurrence(q[i], kk[i], v[i], decay[i], state, out[i], *args, H, dk, dv, single=True, status=status)
            else:
                k.ssm_recurrence(q[i], kk[i], v[i], decay[i], beta[i], state, out[i], *args, H, H, dk, dv, single=True, status=status)
        torch.cuda.synchronize()
    finally:
        k.set_pdl(was or 0)
    want, after = out.double(), before.clone()
    for e in range(E):
        put = v[:, e].double() * (beta[:, e, :, None].double() if kind == "state space" else 1)
        want[:, e], after[E - 1 - e] = _recurrence64(
            q[:, e].double(), kk[:, e].double(), put, (decay[:, e, :, None] if kind == "state space" else decay[:, e]).double(),
            beta[:, e].double() if kind == "delta" else None, before[E - 1 - e])
    assert int(status) == 0
    assert (out.double() - want).abs().max() <= n * 2.0 ** -20 * want.abs().max()
    assert (state.double() - after).abs().max() <= n * 2.0 ** -20 * after.abs().max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("layer", ["delta", "state space"])
def test_float_rows_of_many_tokens_have_float_activations(layer, dtype):
    """x sigmoid(x) of an input that is exact (one tap of weight one), as rows that go into a float memory: an exponential right to
    one unit of the last place, a sum, a division and a product right to half of one, so to 2.5 together; over inputs of both signs."""
    k, g = _k(), _gen(5)
    T, H, d = 16384, 4, 64

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")

    x = (60 * torch.rand((T, 3 * H * d + H), generator=g, device="cuda") - 30).to(dtype)
    entry, cu, slots = torch.zeros(T, dtype=torch.int32, device="cuda"), dev([0, T]), dev([0])
    heads = torch.zeros(H, device="cuda")
    q, kk, v = (torch.full((T, H, d), float("nan"), device="cuda") for _ in range(3))
    if layer == "delta":
        gg, bb = torch.empty((T, H, d), device="cuda"), torch.empty((T, H), device="cuda")
        k.delta_prepare(x, (0, H * d, 2 * H * d, 3 * H * d), x[:, :H * d], torch.ones((1, 3 * H * d), device="cuda"), 1,
                        torch.zeros((1, 0, 3 * H * d), dtype=dtype, device="cuda"), heads, torch.zeros(H * d, device="cuda"), entry, cu, slots,
                        q, kk, v, gg, bb, H, H, d, d, 1.0, 1e-6)
        want = x[:, 2 * H * d:3 * H * d]
    else:
        dts, decay = (torch.empty((T, H), device="cuda") for _ in range(2))
        k.ssm_prepare(x, 0, 3 * H * d, torch.ones((1, 3 * H * d), device="cuda"), torch.zeros(3 * H * d, device="cuda"), 1, None, heads, heads,
                      entry, cu, slots, v, kk, q, dts, decay, H, d, H, d, shift_single=True, chunk=None)
        want = x[:, :H * d]
    want = torch.nn.functional.silu(want.double()).view(T, H, d)
    assert ((v.double() - want).abs() <= 2.5 * 2.0 ** -23 * want.abs()).all()


@pytest.mark.parametrize("n", [41, 100, 500, 1700])
def test_latent_pieces_of_single_tokens_round_beside_their_own_largest_weight(n):
    """Where a launch has a piece for each tile of 32 keys, or for every second one, weights are rounded beside their piece's
    largest, and the error against float64 is that of these roundings (and of the result's) made in float64: but for the few weights so near
    the middle of two that a float sum's order decides."""
    k, g = _k(), _gen(n)
    E, H, R, W, page, splits = 8, 16, 512, 576, 16, 64
    pages, scale = -(-n // page), 576 ** -0.5
    cache = torch.randn((E * pages, page, W), generator=g, device="cuda").to(torch.bfloat16)
    qa, sink = torch.randn((E, H, W), generator=g, device="cuda").to(torch.bfloat16).float(), torch.randn(H, generator=g, device="cuda")
    out = torch.empty((E, H, R), dtype=torch.bfloat16, device="cuda")
    acc, ml = (torch.empty(E * H * splits * m, device="cuda") for m in (R, 2))

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")

    status = dev([0])
    k.latent_attention_mma(qa, cache, sink, None, out, dev(list(range(E + 1))), dev([n - 1] * E), dev(list(range(E))),
                           torch.arange(E * pages, dtype=torch.int32, device="cuda").view(E, pages), 0, E, 1, page, 1 << 30, scale, splits, acc, ml,
                           status)
    rows = cache.view(E, pages * page, W)[:, :n].double()
    s = torch.einsum("ehw,enw->ehn", qa.double(), rows) * scale
    want = torch.einsum("ehn,enr->ehr", torch.softmax(torch.cat([s, sink.double()[None, :, None].expand(E, H, 1)], -1), -1)[..., :-1], rows[..., :R])
    per = 32 * -(-(-(-n // 32)) // splits)
    total, weight = torch.zeros_like(want), torch.exp(sink.double())[None, :, None].expand(E, H, 1)
    for a in range(0, n, per):
        top = s[..., a:a + per].amax(-1, keepdim=True)
        if a == 0:
            top = torch.maximum(top, sink.double()[None, :, None])   # (the first piece has the sink)
        p = torch.exp(s[..., a:a + per] - top)
        weight = weight + torch.exp(top) * p.sum(-1, keepdim=True)
        total = total + torch.exp(top) * torch.einsum("ehn,enr->ehr", p.bfloat16().double(), rows[:, a:a + per, :R])
    rounded = (total / weight).bfloat16().double()
    assert int(status) == 0
    assert (out.double() - want).norm() <= 1.004 * (rounded - want).norm()


def test_latent_position_beyond_the_table_of_pages():
    """The last request's position lies past its table's columns, and its window begins inside of them: the status says so, no
    page is looked up beyond the table, and the other requests have their results."""
    k, g = _k(), _gen(3)
    E, H, R, W, page, cols, window = 3, 16, 512, 576, 16, 8, 40
    cache = torch.randn((E * cols, page, W), generator=g, device="cuda").to(torch.bfloat16)
    qa, sink = torch.randn((E, H, W), generator=g, device="cuda").to(torch.bfloat16).float(), torch.randn(H, generator=g, device="cuda")

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")

    table = torch.arange(E * cols, dtype=torch.int32).view(E, cols)
    table[:, :5] = -1   # (pages before the windows are gone)
    status, outs = dev([0]), []
    for last in (127, 160):   # (the last one's window: rows 88 to 127; 121 to 160, of which the table has 121 to 127)
        if last == 160:
            table[2, :7] = -1   # (so rows 96 to 111 of the walk's first tile lie before the window, and their page is gone)
        out = torch.zeros((E, H, R), dtype=torch.bfloat16, device="cuda")
        k.latent_attention_mma(qa, cache, sink, None, out, dev(list(range(E + 1))), dev([127, 120, last]), dev(list(range(E))), table.cuda(), 0, E,
                               1, page, window, 0.05, status=status)
        outs.append(out)
        assert int(status) == (0 if last == 127 else 4)
    assert torch.equal(outs[0][:2], outs[1][:2]) and torch.isfinite(outs[1].float()).all()
