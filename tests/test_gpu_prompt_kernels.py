"""Kernels that prompts take, alone against float64 at the sizes where they can go wrong: remainders of tiles, every split of a state over
lanes, rows on no 16-byte boundary, windows and kept keys, portions that start inside a page."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
F64 = torch.float64
U = 2.0 ** -24                                              # half a unit in the last place of 1.0 in float32


def _step(starts, news):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    cu = [0]
    for n in news:
        cu.append(cu[-1] + n)
    return SimpleNamespace(n_tokens=cu[-1], n_seqs=len(news), cu_tokens=i32(cu), seq_slots=i32(list(range(len(news)))), seq_starts=i32(starts),
                           seq_new=i32(news), max_new=max(news), token_slot=i32([s for s, n in enumerate(news) for _ in range(n)]),
                           positions=i32([a + t for a, n in zip(starts, news) for t in range(n)]), host_new=news, cu=cu)


def _recurrence(q, k, v, a, c, skip, state, cu, scale):
    """y and S in float64; with every operand replaced by its magnitude it is the sum that bounds the rounding."""
    y, out = torch.zeros(v.shape, dtype=F64, device=DEV), []
    for s in range(len(cu) - 1):
        S = state[s].clone()
        for t in range(cu[s], cu[s + 1]):
            S = S * a[t][:, :, None] + (c[t][:, None] * k[t])[:, :, None] * v[t][:, None, :]
            y[t] = (q[t][:, None] @ S)[:, 0] * scale + skip[:, None] * v[t]
        out.append(S)
    return y, torch.stack(out)


# heads, groups, N, P: N fills 4, 8, 16 and 32 lanes or leaves some empty; P of one column pair, of a remainder of a CTA's columns; odd
# sizes that no 16-byte copy takes; many heads, so that the larger pieces of S are chosen
@pytest.mark.parametrize("heads,groups,n,p", [(1, 1, 4, 4), (4, 2, 16, 8), (3, 3, 9, 6), (5, 1, 33, 14), (2, 1, 128, 64), (2, 2, 500, 4), (1, 1, 512, 2),
                                              (64, 1, 128, 64), (16, 16, 64, 128), (96, 32, 20, 50)])
@pytest.mark.parametrize("form", ["head", "row", "normaliser"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_recurrence_of_prompts(heads, groups, n, p, form, dtype):
    _check_recurrence(heads, groups, n, p, form, dtype, [39, 1, 16, 5])


# 32 lanes a column and three pairs of columns: 96 threads would be whole warps but no multiple of four columns
@pytest.mark.parametrize("heads,groups,n,p", [(2, 1, 65, 6), (2, 2, 128, 6), (1, 1, 256, 6), (1, 1, 500, 6), (3, 3, 100, 2), (2, 1, 72, 10)])
@pytest.mark.parametrize("form", ["head", "row", "normaliser"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("news", [[39, 1, 16, 5], [1, 1, 1, 1]])
def test_recurrence_of_few_columns_over_all_lanes(heads, groups, n, p, form, dtype, news):
    _check_recurrence(heads, groups, n, p, form, dtype, news)


# at most one, two, four and eight tokens a sequence: columns of S in fours and in twos (S read and written once) and what goes by slabs; a
# remainder of a CTA's columns, one and several CTAs of columns, more rows than a round of a CTA's threads
@pytest.mark.parametrize("heads,groups,n,p", [(2, 1, 4, 4), (3, 3, 64, 68), (2, 2, 128, 132), (40, 8, 20, 200), (1, 1, 1000, 12), (2, 1, 130, 8), (2, 1, 24, 10),
                                               (8, 1, 32, 30), (4, 2, 21, 50), (6, 3, 64, 130), (16, 16, 7, 18), (40, 8, 90, 66)])
@pytest.mark.parametrize("form", ["head", "row", "normaliser"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_recurrence_of_a_few_tokens(heads, groups, n, p, form, dtype):
    for news in ([1, 1, 1, 1], [2, 1, 2, 2], [4, 3, 1, 4], [8, 5, 7, 8]):
        _check_recurrence(heads, groups, n, p, form, dtype, news)


def _check_recurrence(heads, groups, n, p, form, dtype, news):
    from kuiperllama_b200.csrc import ops
    step = _step([0] * len(news), news)
    rows = step.n_tokens
    g = torch.Generator(device=DEV).manual_seed(heads * n + p)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    q, k, v = rand(rows, groups * n).to(dtype), (0.3 * rand(rows, groups * n)).to(dtype), rand(rows, heads * p).to(dtype)
    a = 0.75 + 0.25 * torch.rand(rows, heads * n if form == "row" else heads, device=DEV, generator=g)
    a[3] = 0.0                                             # a decay that underflowed: what was before is gone
    c, skip = torch.rand(rows, heads, device=DEV, generator=g), rand(heads)
    size = heads * n * p
    state0 = torch.cat([0.1 * rand(4, size), 0.1 * rand(4, heads * n)], dim=1)
    state = state0.clone()
    y = torch.full((rows, heads * p), 7.0, device=DEV)
    norm, floor, den = None, torch.full((rows, heads), 0.05, device=DEV), torch.empty(rows, heads, device=DEV)
    if form == "normaliser":
        norm = (state[:, size:], floor, den, 1e-3)
    ops.outer_recurrence(q, k, v, a, state, y, step, heads, groups, n, p, c=c, skip=skip, q_scale=0.7, normaliser=norm)
    wide = lambda x: x.double().view(rows, groups, n).repeat_interleave(heads // groups, dim=1)
    args = [wide(q), wide(k), v.double().view(rows, heads, p), a.double().view(rows, heads, -1), c.double(), skip.double(),
            state0[:, :size].double().view(4, heads, n, p)]
    want, S = _recurrence(*args, step.cu, 0.7)
    most, S_most = _recurrence(*[x.abs() for x in args], step.cu, 0.7)
    # an element of S takes three roundings a token, y one more for each of n terms and a few for scale and skip
    tokens = max(step.host_new)
    assert bool(((y.double().view(want.shape) - want).abs() <= (3 * tokens + n + 8) * U * most).all())
    assert bool(((state[:, :size].double().view(S.shape) - S).abs() <= (3 * tokens + 2) * U * S_most).all())
    if form == "normaliser":
        args[2], args[5], args[6] = torch.ones(rows, heads, 1, dtype=F64, device=DEV), torch.zeros(heads, dtype=F64, device=DEV), state0[:, size:].double().view(4, heads, n, 1)
        dot, z = _recurrence(*args, step.cu, 0.7)
        dot_most, z_most = _recurrence(*[x.abs() for x in args], step.cu, 0.7)
        near = (3 * tokens + n + 8) * U * dot_most[:, :, 0] + 4 * U
        assert bool(((den.double() - (torch.clamp(dot[:, :, 0].abs(), min=0.05) + 1e-3)).abs() <= near).all())
        assert bool(((state[:, size:].double().view(z.shape) - z).abs() <= (3 * tokens + 2) * U * z_most).all())
    else:
        assert torch.equal(state[:, size:], state0[:, size:])


# rows of S on both sides of 64 and 128, columns of one 16, of a remainder of a CTA's 32 and of several CTAs; chunks of one token, of the first
# block alone, whole ones and remainders; operands as they come and as columns of wider rows
@pytest.mark.parametrize("heads,groups,n,p", [(2, 1, 8, 16), (4, 2, 64, 48), (3, 3, 72, 32), (6, 2, 128, 64), (5, 5, 128, 16)])
@pytest.mark.parametrize("form", ["head", "row"])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("near", [False, True])
def test_recurrence_in_chunks(heads, groups, n, p, form, wide, near):
    from kuiperllama_b200.csrc import ops
    news = [64, 1, 97, 16, 33, 300]
    step = _step([0] * len(news), news)
    rows, dtype = step.n_tokens, torch.float32 if form == "head" else torch.bfloat16
    g = torch.Generator(device=DEV).manual_seed(heads * n + p)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)

    def placed(x):
        if not wide:
            return x
        room = torch.full((rows, x.shape[1] + 24), float("nan"), dtype=dtype, device=DEV)
        room[:, 8:8 + x.shape[1]] = x
        return room[:, 8:8 + x.shape[1]]

    q, k, v = (placed(x.to(dtype)) for x in (rand(rows, groups * n), 0.3 * rand(rows, groups * n), rand(rows, heads * p)))
    a = torch.rand(rows, heads * n if form == "row" else heads, device=DEV, generator=g)
    a = a ** 0.0625 if near else a ** 4                    # decays near one, and ones whose products underflow within a chunk
    a[3] = 0.0
    c, skip = torch.rand(rows, heads, device=DEV, generator=g), rand(heads)
    size = heads * n * p
    state0 = 0.1 * rand(len(news), size + 4)
    state, y = state0.clone(), torch.full((rows, heads * p), 7.0, device=DEV)
    ops.outer_recurrence(q, k, v, a, state, y, step, heads, groups, n, p, c=c, skip=skip, q_scale=0.7, chunked=True)
    spread = lambda x: x.double().reshape(rows, groups, n).repeat_interleave(heads // groups, dim=1)
    args = [spread(q), spread(k), v.double().reshape(rows, heads, p), a.double().view(rows, heads, -1), c.double(), skip.double(),
            state0[:, :size].double().view(len(news), heads, n, p)]
    want, S = _recurrence(*args, step.cu, 0.7)
    most, S_most = _recurrence(*[x.abs() for x in args], step.cu, 0.7)
    # within a chunk a term takes at most 36 roundings of decays and factors and a few for its pieces; a sum of n terms one for every 16 and
    # a few; S four a chunk
    chunks = 300 / 32
    assert bool(((y.double().view(want.shape) - want).abs() <= (36 + n / 16 + 4 * chunks + 16) * U * most).all())
    assert bool(((state[:, :size].double().view(S.shape) - S).abs() <= (36 + 4 * chunks + 16) * U * S_most).all())
    assert torch.equal(state[:, size:], state0[:, size:])
    walked = torch.empty_like(y)
    ops.outer_recurrence(q, k, v, a, state0.clone(), walked, step, heads, groups, n, p, c=c, skip=skip, q_scale=0.7, chunked=False)
    off = lambda x: float((x.double().view(want.shape) - want).norm() / want.norm())
    assert off(y) <= 1.5 * off(walked) + U                 # no less exact than token by token


# decays as the layers have them (sigmoid(z) ** (1 / tau)) and stronger ones; a few tokens behind a chunk and whole prompts
@pytest.mark.parametrize("heads,n,p,tau", [(16, 64, 128, 16.0), (8, 64, 128, 4.0), (8, 64, 128, 2.0), (4, 128, 128, 4.0), (4, 128, 64, 8.0), (4, 128, 64, 16.0)])
@pytest.mark.parametrize("news", [[33], [500]])
def test_recurrence_in_chunks_is_as_exact_as_token_by_token(heads, n, p, tau, news):
    from kuiperllama_b200.csrc import ops
    step, g = _step([0], news), torch.Generator(device=DEV).manual_seed(5)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    q, k, v = (rand(news[0], heads * w).bfloat16() for w in (n, n, p))
    a, state0 = torch.sigmoid(rand(news[0], heads * n)) ** (1 / tau), torch.zeros(1, heads * n * p, device=DEV)
    one = torch.ones(news[0], heads, dtype=F64, device=DEV)
    want, S = _recurrence(q.double().view(-1, heads, n), k.double().view(-1, heads, n), v.double().view(-1, heads, p), a.double().view(-1, heads, n), one,
                          0 * one[0], state0.double().view(1, heads, n, p), step.cu, 0.125)
    off = {}
    for chunked in (False, True):
        state, y = state0.clone(), torch.empty(news[0], heads * p, device=DEV)
        ops.outer_recurrence(q, k, v, a, state, y, step, heads, heads, n, p, q_scale=0.125, chunked=chunked)
        off[chunked] = float((y.double().view(want.shape) - want).norm() / want.norm()), float((state.double().view(S.shape) - S).norm() / S.norm())
    assert off[True][0] <= off[False][0], off
    assert off[True][1] <= max(off[False][1], U), off      # (of S one rounding of a sum's last bits: 2^-24 at most)


@pytest.mark.parametrize("form", ["head", "row"])
@pytest.mark.parametrize("what", ["v", "q", "k", "a", "c", "state", "grows", "huge"])
def test_recurrence_in_chunks_keeps_what_is_not_finite_where_it_arises(form, what):
    """NaN, infinities, numbers too large for the products and decays above one: the same places are not finite as token by token, and the
    others are as close as sums in another order are."""
    from kuiperllama_b200.csrc import ops
    heads, n, p = 4, 64, 48
    groups, dtype = (1, torch.float32) if form == "head" else (heads, torch.bfloat16)
    step = _step([0, 0], [100, 70])
    g = torch.Generator(device=DEV).manual_seed(1)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    q, k, v = rand(170, groups * n).to(dtype), (0.3 * rand(170, groups * n)).to(dtype), rand(170, heads * p).to(dtype)
    a, c = torch.rand(170, heads * n if form == "row" else heads, device=DEV, generator=g) ** 0.1, torch.rand(170, heads, device=DEV, generator=g)
    state0 = 0.1 * rand(2, heads * n * p)
    if what in ("v", "q", "k", "a", "c"):
        {"v": v, "q": q, "k": k, "a": a, "c": c}[what][40, 2], {"v": v, "q": q, "k": k, "a": a, "c": c}[what][120, 1] = float("nan"), float("inf")
    elif what == "state":
        state0[1, 100], state0[0, 7] = float("inf"), 1e30
    elif what == "grows":
        a[20:30] = 1.5
    else:
        v[50], k[90] = 1e12, 1e9
    got = []
    for chunked in (False, True):
        state, y = state0.clone(), torch.empty(170, heads * p, device=DEV)
        ops.outer_recurrence(q, k, v, a, state, y, step, heads, groups, n, p, c=c, q_scale=0.7, chunked=chunked)
        got += [y, state]
    for x, z in ((got[0], got[2]), (got[1], got[3])):
        fine = torch.isfinite(x)
        assert torch.equal(fine, torch.isfinite(z))
        assert bool(((x - z)[fine].abs() <= 1e-4 * x[fine].abs() + 1e-5 * x[fine].abs().median()).all()) or what in ("huge", "state"), what
        assert float((x - z)[fine].double().norm()) <= 2e-6 * float(x[fine].double().norm()), what


def test_recurrence_of_steps_that_the_chunks_do_not_take():
    """Rows between 16-byte boundaries, odd sizes, a normaliser and many short sequences go token by token."""
    from kuiperllama_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(2)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    for n, p, shift, news in ((64, 32, 1, [80]), (20, 32, 0, [80]), (64, 20, 0, [80]), (136, 32, 0, [80]), (64, 32, 0, [64] + [1] * 40)):
        step = _step([0] * len(news), news)
        rows = step.n_tokens
        wide = rand(rows, 4 * n + 4)
        q, k, v, a = wide[:, shift:shift + 2 * n], wide[:, 2 * n:4 * n], rand(rows, 2 * p), torch.rand(rows, 2, device=DEV, generator=g)
        out = []
        for chunked in (None, False):
            state, y = torch.zeros(len(news), 2 * n * p, device=DEV), torch.empty(rows, 2 * p, device=DEV)
            ops.outer_recurrence(q, k, v, a, state, y, step, 2, 2, n, p, chunked=chunked)
            out.append((y, state))
        assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("channels", [4, 36, 512, 1028])
@pytest.mark.parametrize("dtype,out_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_four_taps_in_tiles(channels, dtype, out_dtype):
    """The vector form against the plain one (the same rows at a stride that it does not take): the same bits, outputs and state."""
    from kuiperllama_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(channels)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    w, b = rand(channels, 4), rand(channels)
    for news in ([1, 1, 1], [2, 4, 3], [3, 17, 1], [70, 5, 33], [500]):
        step = _step([0] * len(news), news)
        x = rand(step.n_tokens, channels).to(dtype)
        loose = torch.zeros(step.n_tokens, channels + 1, dtype=dtype, device=DEV)
        loose[:, :channels] = x
        state0 = rand(len(news), 3 * channels)
        for add, silu in ((True, False), (False, True)):
            got = []
            for rows in (x, loose[:, :channels]):
                state, out = state0.clone(), torch.empty(step.n_tokens, channels, dtype=out_dtype, device=DEV)
                ops.short_conv(rows, w, b, state, step, out, add_input=add, silu=silu)
                got.append((out, state))
            assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]), (news, add)


@pytest.mark.parametrize("rows,channels", [(1, 5), (3, 256), (65, 300), (700, 1024)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_low_rank_decays_of_rank_16(rows, channels, dtype):
    from kuiperllama_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(rows)
    r1 = torch.randn(rows, 40, device=DEV, generator=g).to(dtype)[:, 3:19]
    W2, b = torch.randn(channels, 16, device=DEV, generator=g), 8.0 * torch.randn(channels, device=DEV, generator=g)
    a = torch.empty(rows, channels, device=DEV)
    ops.decay_lowrank(r1, W2, b, 16.0, rows, a)
    z = r1.double() @ W2.double().T + b.double()
    want = torch.exp(-torch.nn.functional.softplus(-z, threshold=200.0) / 16.0)
    most = r1.double().abs() @ W2.double().abs().T + b.double().abs()
    # 17 roundings of z, whose error enters the exponent by at most a sixteenth, and a few units for exp and log1p
    assert bool(((a.double() - want).abs() <= want * (17 * U * most / 16 + 32 * U)).all())


@pytest.mark.parametrize("heads,dim", [(1, 1028), (2, 2048), (1, 4096), (1, 4100), (1, 8192)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gated_norm_of_long_heads(heads, dim, dtype):
    """One pass in registers: the gate before and after the norm, a divisor; off by a sum of dim squares and the output's rounding."""
    from kuiperllama_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(dim)
    x, gate = 3 * torch.randn(37, heads * dim, device=DEV, generator=g), torch.randn(37, heads * dim, device=DEV, generator=g).to(dtype)
    w, div = 1 + 0.2 * torch.randn(heads * dim, device=DEV, generator=g), 0.5 + torch.rand(37, heads, device=DEV, generator=g)
    for first in (True, False):
        out = torch.empty(37, heads * dim, dtype=dtype, device=DEV)
        ops.head_rmsnorm_gate(x, gate, w, out, heads, dim, 1e-5, gate_first=first, out_scale=0.7, divisor=div)
        xs, gs = x.double().view(37, heads, dim) / div.double()[..., None], torch.nn.functional.silu(gate.double()).view(37, heads, dim)
        y = xs * gs if first else xs
        y = y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5) * w.double().view(heads, dim)
        want = (y if first else y * gs) * 0.7
        tol = (dim ** 0.5 + 32) * U + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
        assert bool(((out.double().view(want.shape) - want).abs() <= tol * want.abs() + 1e-9).all())


# heads on key/value heads with keys and values of one size, window, kept first keys
@pytest.mark.parametrize("H,G,d,window,keep", [(32, 8, 64, 96, 16), (16, 4, 64, 0, 0), (32, 16, 32, 130, 64), (16, 2, 32, 40, 5), (32, 2, 64, 1, 3),
                                               (32, 16, 64, 70, 0)])
def test_mixed_heads_on_the_tensor_cores(H, G, d, window, keep):
    """Outputs are off by their own rounding (2^-9) and by what 32-bit scores, exponentials and sums leave: scores up to 30 in magnitude
    after the soft cap have errors of a few 2^-24 * 30, which the exponential passes on as a relative error of about 1e-5."""
    from kuiperllama_b200.csrc import ops
    T, dev, dt = 256, DEV, torch.bfloat16
    g = torch.Generator().manual_seed(H + G + d)
    table = torch.tensor([[5, 2, 9, 0], [1, 7, 3, 11], [4, 6, 8, 10]], dtype=torch.int32, device=dev)
    ks, vs = (torch.randn(3, T, G, d, generator=g).to(dt).to(dev) for _ in range(2))
    qs, gates = (1.5 * torch.randn(3, T, H, d, generator=g)).to(dt).to(dev), torch.randn(3, T, H, generator=g).to(dt).to(dev)
    kc, vc = torch.zeros(12, G, 64, d, dtype=dt, device=dev), torch.zeros(12, G, 64, d, dtype=dt, device=dev)
    for s in range(3):
        for p in range(T):
            kc[int(table[s, p // 64]), :, p % 64], vc[int(table[s, p // 64]), :, p % 64] = ks[s, p], vs[s, p]
    r1, r2 = (torch.rand(H, generator=g) * 0.5 + 0.1).to(dev), (torch.rand(H, generator=g) + 0.05).to(dev)
    talk = (torch.eye(H) + 0.4 * torch.randn(H, H, generator=g)).to(dev)
    i, j = torch.arange(T, device=dev)[:, None], torch.arange(T, device=dev)[None]
    hidden = (j > i) | ((i - j >= window) & (j >= keep) if window else torch.zeros(T, T, dtype=torch.bool, device=dev))
    for full in (True, False):
        want, most = [], []
        for s in range(3):
            sc = torch.einsum("ihd,jhd->hij", qs[s].double(), ks[s].double().repeat_interleave(H // G, 1)) * 0.3
            if full:
                sc = 30.0 * torch.tanh(sc / 30.0) - r1.double()[:, None, None] * torch.log1p(r2.double()[:, None, None] * (i - j).clamp(min=0).double())
            w = torch.softmax(sc.masked_fill(hidden, float("-inf")), -1)
            u = torch.einsum("hg,gij->hij", talk.double().abs(), w) if full else w
            w = torch.einsum("hg,gij->hij", talk.double(), w) if full else w
            gate = 1.25 * (torch.sigmoid(gates[s].double()) if full else torch.ones(T, H, dtype=F64, device=dev))[..., None]
            v = vs[s].double().repeat_interleave(H // G, 1)
            want.append(torch.einsum("hij,jhd->ihd", w, v) * gate)
            most.append(torch.einsum("hij,jhd->ihd", u, v.abs()) * gate)
        for starts, news in (([0, 0, 0], [256, 1, 67]), ([100, 63, 200], [30, 2, 56]), ([0, 39, 129], [5, 110, 127])):
            step = _step(starts, news)
            cut = lambda x: torch.cat([x[s][a:a + n].reshape(n, -1) for s, (a, n) in enumerate(zip(starts, news))]).contiguous()
            ref, bound = cut(want), cut(most)
            for tiled in (None, True):                      # the kernel that the sizes choose and the tiled one, within the same bound
                out = torch.full((step.n_tokens, H * d), 9.0, dtype=dt, device=dev)
                ops.attention_mixed(cut(qs), cut(gates) if full else None, out, kc, vc, table, step, H, G, d, d, 0.3, 30.0 if full else 0.0,
                                    r1 if full else None, r2 if full else None, talk if full else None, window, keep, 1.25, tiled=tiled)
                off = (out.double() - ref).abs()
                assert bool((off <= 2.0 ** -8 * ref.abs() + 2e-5 * bound + 1e-30).all()), (full, starts, tiled, float((off / (bound + 1e-30)).max()))


@pytest.mark.parametrize("H,G,d", [(32, 8, 64), (16, 2, 32)])
def test_mixed_heads_with_scores_that_overflow(H, G, d):
    """Keys and queries whose products pass the largest float32: the soft cap takes infinite scores to +-cap, as in the tiled kernel."""
    from kuiperllama_b200.csrc import ops
    g = torch.Generator().manual_seed(d)
    dt, T = torch.bfloat16, 100
    table = torch.tensor([[1, 0]], dtype=torch.int32, device=DEV)
    kc, vc = torch.randn(2, G, 64, d, generator=g).to(dt).to(DEV), torch.randn(2, G, 64, d, generator=g).to(dt).to(DEV)
    q, talk = torch.randn(T, H * d, generator=g).to(dt).to(DEV), (torch.eye(H) + 0.2 * torch.randn(H, H, generator=g)).to(DEV)
    kc[1, :, 3] = kc[1, :, 40] = 3e19                       # one sign a row: a score is +-inf, never inf - inf
    q[10:60] = 2e19
    q[60:] = q[60:].abs()
    q[20] = -2e19
    step, got = _step([0], [T]), []
    for tiled in (None, True):
        out = torch.full((T, H * d), 9.0, dtype=dt, device=DEV)
        ops.attention_mixed(q, None, out, kc, vc, table, step, H, G, d, d, 1.0, 20.0, None, None, talk, 0, 0, 1.0, tiled=tiled)
        got.append(out.float())
    assert bool(torch.isfinite(got[1]).all())
    # both round to bfloat16 sums of 32-bit weights of at most sum |talk| of order one
    assert bool(((got[0] - got[1]).abs() <= 2.0 ** -7 * got[1].abs() + 1e-3).all())


@pytest.mark.parametrize("H,G,d", [(32, 8, 64), (16, 2, 32)])
@pytest.mark.parametrize("splits", [(1, 1), (3, 1), (2, 3), (16, 16)])
def test_mixed_heads_in_pieces(monkeypatch, H, G, d, splits):
    """However many pieces a tile's chunks are dealt to, also pieces without a chunk, and scores on both sides of where tanh is a polynomial
    (0.6 of the cap): float64 within what the test above allows."""
    from kuiperllama_b200.csrc import ops
    monkeypatch.setattr(ops, "MIXED_SPLITS", splits)
    g = torch.Generator().manual_seed(H + splits[0])
    bf, T = torch.bfloat16, 200
    table = torch.tensor([[3, 0, 2, 1]], dtype=torch.int32, device=DEV)
    k, v = (torch.randn(T, G, d, generator=g).to(bf).to(DEV) for _ in range(2))
    kc, vc = torch.zeros(4, G, 64, d, dtype=bf, device=DEV), torch.zeros(4, G, 64, d, dtype=bf, device=DEV)
    for p in range(T):
        kc[int(table[0, p // 64]), :, p % 64], vc[int(table[0, p // 64]), :, p % 64] = k[p], v[p]
    q, gate = torch.randn(T, H, d, generator=g).to(bf).to(DEV), torch.randn(T, H, generator=g).to(bf).to(DEV)
    q[:100:3] *= 6                                         # (the tiles of the other tokens see small scores alone)
    r1, r2 = (torch.rand(H, generator=g) * 0.5 + 0.1).to(DEV), (torch.rand(H, generator=g) + 0.05).to(DEV)
    talk = (torch.eye(H) + 0.3 * torch.randn(H, H, generator=g)).to(DEV)
    i, j = torch.arange(T, device=DEV)[:, None], torch.arange(T, device=DEV)[None]
    for starts, news, window, keep in (([0], [T], 0, 0), ([0], [T], 70, 20), ([130], [70], 70, 0), ([195], [5], 0, 0)):
        step = _step(starts, news)
        rows = slice(starts[0], T)
        hidden = (j > i) | ((i - j >= window) & (j >= keep) if window else torch.zeros(T, T, dtype=torch.bool, device=DEV))
        sc = torch.einsum("ihd,jhd->hij", q.double(), k.double().repeat_interleave(H // G, 1)) * 0.2
        assert float(sc[:, 104:].abs().max()) < 0.6 * 20 < float(sc[:, :100:3].abs().max())
        sc = 20.0 * torch.tanh(sc / 20.0) - r1.double()[:, None, None] * torch.log1p(r2.double()[:, None, None] * (i - j).clamp(min=0).double())
        w = torch.softmax(sc.masked_fill(hidden, float("-inf")), -1)
        f = torch.sigmoid(gate.double())[..., None]
        values = v.double().repeat_interleave(H // G, 1)
        want = (torch.einsum("hg,gij,jhd->ihd", talk.double(), w, values) * f)[rows]
        most = (torch.einsum("hg,gij,jhd->ihd", talk.double().abs(), w, values.abs()) * f)[rows]
        out = torch.full((news[0], H * d), 9.0, dtype=bf, device=DEV)
        ops.attention_mixed(q[rows].reshape(news[0], -1).contiguous(), gate[rows].contiguous(), out, kc, vc, table, step, H, G, d, d, 0.2, 20.0, r1, r2, talk, window, keep, 1.0)
        off = (out.double().view(want.shape) - want).abs()
        assert bool((off <= 2.0 ** -8 * want.abs() + 2e-5 * most + 1e-30).all()), (splits, starts, float((off / most).max()))


@pytest.mark.parametrize("H,G,d,n,longest,window,keep", [
    (32, 8, 64, 3, 2500, 0, 0), (32, 8, 64, 40, 97, 0, 0), (5, 5, 32, 2, 65, 40, 3), (24, 3, 128, 20, 300, 100, 40), (64, 8, 64, 2, 700, 0, 0),
    (16, 16, 64, 150, 64, 0, 0), (40, 8, 32, 1, 1, 1, 0)])
def test_mixed_heads_of_single_tokens(H, G, d, n, longest, window, keep):
    """Clusters of eight, four, two and one CTAs, CTAs without a chunk, chunks with one key and with all, scores in rounds (more chunks than a CTA
    is planned for), heads that are no whole tiles, NaN in the cache past the last key and in pages of others: float64 within a result's
    rounding and 2e-5 of the sum's largest terms (32-bit sums of 32-bit numbers)."""
    from kuiperllama_b200.csrc import ops
    g = torch.Generator().manual_seed(H + n)
    bf = torch.bfloat16
    contexts = [max(1, longest - 31 * (i % 5) - i % 2) for i in range(n)]
    pages = -(-longest // 64)
    table = torch.randperm(n * pages, generator=g).to(torch.int32).view(n, pages).to(DEV)
    kc, vc = (torch.full((n * pages, G, 64, d), float("nan"), dtype=bf, device=DEV) for _ in range(2))
    ks, vs = [], []
    for b, c in enumerate(contexts):
        for cache, kept in ((kc, ks), (vc, vs)):
            x = torch.full((pages * 64, G, d), float("nan"))
            x[:c] = torch.randn(c, G, d, generator=g)
            x = x.to(bf).to(DEV)
            cache[table[b].long()] = x.view(pages, 64, G, d).transpose(1, 2)
            kept.append(x[:c].double().repeat_interleave(H // G, 1))
    q, gate = torch.randn(n, H, d, generator=g).to(bf).to(DEV), torch.randn(n, H, generator=g).to(bf).to(DEV)
    q[::2] *= 6                                            # (scores on both sides of where tanh is a polynomial)
    r1, r2 = (torch.rand(H, generator=g) * 0.5 + 0.1).to(DEV), (torch.rand(H, generator=g) + 0.05).to(DEV)
    talk = (torch.eye(H) + 0.3 * torch.randn(H, H, generator=g)).to(DEV)
    step = _step([c - 1 for c in contexts], [1] * n)
    for full in (True, False):
        out = torch.full((n, H * d), 9.0, dtype=bf, device=DEV)
        ops.attention_mixed(q.view(n, -1), gate if full else None, out, kc, vc, table, step, H, G, d, d, 0.2, 20.0 if full else 0.0, r1 if full else None,
                            r2 if full else None, talk if full else None, window, keep, 1.5)
        for b, c in enumerate(contexts):
            away = torch.arange(c - 1, -1, -1, device=DEV).double()
            sc = torch.einsum("hd,jhd->hj", q[b].double(), ks[b]) * 0.2
            if full:
                sc = 20.0 * torch.tanh(sc / 20.0) - r1.double()[:, None] * torch.log1p(r2.double()[:, None] * away)
            if window:
                sc = sc.masked_fill((away >= window) & (torch.arange(c, device=DEV) >= keep), float("-inf"))
            w, f = torch.softmax(sc, -1), torch.full((H, 1), 1.5, dtype=torch.float64, device=DEV)
            mixed, mass = (talk.double() @ w, talk.double().abs() @ w) if full else (w, w)
            if full:
                f = f * torch.sigmoid(gate[b].double())[:, None]
            want, most = torch.einsum("hj,jhd->hd", mixed, vs[b]) * f, torch.einsum("hj,jhd->hd", mass, vs[b].abs()) * f
            off = (out[b].double().view(H, d) - want).abs()
            assert bool((off <= 2.0 ** -8 * want.abs() + 2e-5 * most + 1e-30).all()), (b, c, full, float((off / most).max()))


@pytest.mark.parametrize("what", ["value inf", "value nan", "key nan", "key inf", "all keys -inf", "talk inf"])
def test_mixed_heads_of_single_tokens_not_finite(what):
    """Infinities and NaN come out where the kernel of 32-bit multiply-adds has them, as the same."""
    from kuiperllama_b200.csrc import ops
    H, G, d, n, T, bf = 8, 2, 32, 2, 150, torch.bfloat16
    g = torch.Generator().manual_seed(3)
    table = torch.tensor([[4, 1, 3], [0, 5, 2]], dtype=torch.int32, device=DEV)
    kc, vc = (torch.randn(6, G, 64, d, generator=g).to(bf).to(DEV) for _ in range(2))
    q = torch.rand(n, H * d, generator=g).add(0.1).to(bf).to(DEV)
    talk = (torch.eye(H) + 0.3 * torch.rand(H, H, generator=g)).to(DEV)
    if what == "value inf": vc[1, 0, 9, 5] = float("inf")
    elif what == "value nan": vc[1, 0, 9, 5] = float("nan")
    elif what == "key nan": kc[4, 1, 7, 3] = float("nan")
    elif what == "key inf": kc[4, 1, 7, 3] = float("inf")
    elif what == "all keys -inf": kc[..., 2] = float("-inf")
    else: talk[3, 2] = float("inf")
    step, outs = _step([T - 1, T - 2], [1, 1]), []
    for tiled in (None, True):
        for mix in (talk, None):
            out = torch.full((n, H * d), 9.0, dtype=bf, device=DEV)
            ops.attention_mixed(q, None, out, kc, vc, table, step, H, G, d, d, 0.1, 0.0, None, None, mix, 60 if what == "key inf" else 0, 8, 1.0, tiled=tiled)
            outs.append(out.float())
    for new, old in zip(outs[:2], outs[2:]):
        assert bool((new.isnan() == old.isnan()).all()) and bool((new.isinf() == old.isinf()).all())
        assert bool(((new - old).abs()[new.isfinite()] <= 2.0 ** -7 * old.abs()[new.isfinite()] + 1e-3).all())
        assert bool((new[new.isinf()] == old[new.isinf()]).all())


@pytest.mark.parametrize("H,G,d", [(32, 8, 64), (16, 2, 32)])
@pytest.mark.parametrize("single", [True, False])
def test_mixed_heads_do_not_notice_keys_that_they_do_not_see(H, G, d, single):
    """Rows past the last key hold what an earlier sequence left there, and a token's tile holds keys of the tokens after it: whatever those are, the
    bits stay.  Every score is 1e5 and a little, so that its last bit is seen in the weights."""
    from kuiperllama_b200.csrc import ops
    g = torch.Generator().manual_seed(H)
    bf, T = torch.bfloat16, 44
    table = torch.zeros(1, 1, dtype=torch.int32, device=DEV)
    kc, vc = (0.5 * torch.randn(1, G, 64, d, generator=g) for _ in range(2))
    q = 0.5 * torch.randn(T, H, d, generator=g)
    kc[..., 0], q[..., 0] = 316.0, 316.0
    kc[:, :, T:], vc[:, :, T:] = 0.0, 0.0
    outs = []
    for far in (False, True):
        k = kc.clone()
        if far:
            k[:, :, T - 1 if not single else T:] = 3000.0  # (scores past the cap)
        step = _step([T - 1], [1]) if single else _step([0], [T])
        rows = step.n_tokens
        out = torch.empty(rows, H * d, dtype=bf, device=DEV)
        ops.attention_mixed(q[-rows:].reshape(rows, -1).to(bf).to(DEV), None, out, k.to(bf).to(DEV), vc.to(bf).to(DEV), table, step, H, G, d, d, 1.0, 3e5,
                            None, None, None, 0, 0, 1.0)
        outs.append(out if single else out[:-1])
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16)) and bool(torch.isfinite(outs[0]).all())


def _score_errors(H, G, d, q, k, cap, single, tiled):
    """What a kernel's scores of q [H, d] and k [G, d] (bfloat16 numbers, products about 2^20) are off by.  Two keys: the first one's score less a
    distance bias of the score itself, rounded to float32, is as good as zero, and so is the second one's; the first one's weight is its result."""
    from kuiperllama_b200.csrc import ops
    bf, T = torch.bfloat16, 2 if single else 8
    kc, vc = torch.zeros(1, G, 64, d, dtype=bf, device=DEV), torch.zeros(1, G, 64, d, dtype=bf, device=DEV)
    kc[0, :, 0], vc[0, :, 0] = k.to(bf).to(DEV), 1.0
    step = _step([1], [1]) if single else _step([0], [T])
    qs = torch.zeros(step.n_tokens, H, d, dtype=bf, device=DEV)
    qs[0 if single else 1] = q.to(bf).to(DEV)
    exact = (q.double() * k.double().repeat_interleave(H // G, 0)).sum(-1)
    if cap:
        exact = cap * torch.tanh(exact / cap)
    bias = exact.float()
    out = torch.empty(step.n_tokens, H * d, dtype=bf, device=DEV)
    ops.attention_mixed(qs.view(step.n_tokens, -1), None, out, kc, vc, torch.zeros(1, 1, dtype=torch.int32, device=DEV), step, H, G, d, d, 1.0, cap,
                        (bias * 2.0 ** 30).to(DEV), torch.full((H,), 2.0 ** -30, device=DEV), None, 0, 0, 1.0, tiled=tiled)
    w = out.view(-1, H, d)[0 if single else 1, :, 0].double().cpu()
    return torch.log(w / (1 - w)) + bias.double() - exact, exact


def test_mixed_heads_of_single_tokens_add_scores_with_rounding():
    """Sums of 128 products on the tensor cores are no less exact than the chain of 32-bit multiply-adds."""
    g, H, G, d, off = torch.Generator().manual_seed(5), 24, 3, 128, {None: [], True: []}
    for _ in range(40):
        q, k = ((300.0 * torch.randn(n, d, generator=g)).bfloat16() for n in (H, G))
        mass = (q.double() * k.double().repeat_interleave(H // G, 0)).abs().sum(-1)
        for tiled, errors in off.items():
            errors.append(_score_errors(H, G, d, q, k, 0.0, True, tiled)[0] / (U * mass))
    rms = {tiled: float(torch.cat(errors).square().mean().sqrt()) for tiled, errors in off.items()}
    assert rms[None] <= rms[True], rms


@pytest.mark.parametrize("single", [True, False])
@pytest.mark.parametrize("lo,hi", [(0.3, 0.59), (0.61, 1.2)])
def test_mixed_heads_divide_by_the_cap_as_exactly_as_before(single, lo, hi):
    """A cap whose reciprocal float32 rounds by half a unit; one product a score, so that nothing else is rounded before the quotient.  On both sides of
    where tanh is a polynomial, no further from float64 than the kernel that divides."""
    g, H, G, d, cap, off = torch.Generator().manual_seed(6), 32, 8, 64, 2096640.0, {None: [], True: []}
    for _ in range(30):
        q, k = torch.zeros(H, d), torch.zeros(G, d)
        k[:, 3] = (1000.0 * (1.0 + 0.01 * torch.rand(G, generator=g))).bfloat16().float()
        q[:, 3] = ((lo + (hi - lo) * torch.rand(H, generator=g)) * cap / 1015.0).bfloat16().float()
        for tiled, errors in off.items():
            e, s = _score_errors(H, G, d, q, k, cap, single, tiled)
            errors.append(e / (U * s))
    rms = {tiled: float(torch.cat(errors).square().mean().sqrt()) for tiled, errors in off.items()}
    assert rms[None] <= 1.02 * rms[True], rms              # (960 samples each)


@pytest.mark.parametrize("which", ["keys", "values"])
def test_mixed_heads_of_caches_on_eight_bytes(which):
    """A cache that starts between two 16-byte boundaries is served as before, by the kernel that copies smaller pieces."""
    from kuiperllama_b200.csrc import ops
    H, G, d, T, dt = 16, 4, 64, 70, torch.bfloat16
    g = torch.Generator().manual_seed(1)
    rand = lambda *s: torch.randn(*s, generator=g).to(dt).to(DEV)
    table, step = torch.tensor([[1, 0]], dtype=torch.int32, device=DEV), _step([0], [T])
    q, caches = rand(T, H * d), {"keys": rand(2, G, 64, d), "values": rand(2, G, 64, d)}
    outs = []
    for shift in (0, 4):
        c = dict(caches)
        room = torch.empty(c[which].numel() + 8, dtype=dt, device=DEV)
        c[which] = room[shift:shift + c[which].numel()].view(2, G, 64, d).copy_(caches[which])
        out = torch.empty(T, H * d, dtype=dt, device=DEV)
        ops.attention_mixed(q, None, out, c["keys"], c["values"], table, step, H, G, d, d, 0.125, 0.0, None, None, None, 0, 0, 1.0)
        outs.append(out.float())
    assert bool(((outs[0] - outs[1]).abs() <= 2.0 ** -7 * outs[0].abs() + 1e-4).all())


@pytest.mark.parametrize("H,KV,hd,vd", [(4, 2, 64, 64), (2, 1, 128, 128), (3, 3, 20, 20), (4, 1, 48, 32)])
def test_float32_attention_of_runs_has_the_same_bits(H, KV, hd, vd):
    """Tiles of eight rows, a CTA per row, and the plain kernel (which a distance bias of zeros asks for): prompts, portions, single tokens
    and padding rows in one step, with and without a sink, and a cache that holds infinities past every row's keys."""
    from kuiperllama_b200.csrc import ops
    g = torch.Generator().manual_seed(hd)
    table = torch.tensor([[5, 2, 9, 0], [1, 7, 3, 11], [4, 6, 8, 10]], dtype=torch.int32, device=DEV)
    kc, vc = torch.randn(12, KV, 64, hd, generator=g).to(DEV), torch.randn(12, KV, 64, hd, generator=g).to(DEV)
    for starts, news in (([0, 0, 0], [200, 1, 67]), ([100, 63, 200], [30, 2, 56]), ([150, 64, 255], [1, 1, 1]), ([0, 39, 129], [8, 16, 9])):
        pos = [a + t for a, n in zip(starts, news) for t in range(n)] + [0, 0, 0]
        slot = [s for s, n in enumerate(news) for _ in range(n)] + [-1, -1, -1]
        pos, slot = (torch.tensor(x, dtype=torch.int32, device=DEV) for x in (pos, slot))
        ks, vs = kc.clone(), vc.clone()
        for s, (a, n) in enumerate(zip(starts, news)):
            for p in range(a + n, 256):
                ks[int(table[s, p // 64]), :, p % 64], vs[int(table[s, p // 64]), :, p % 64] = float("inf"), float("nan")
        q = torch.randn(len(pos), H * hd, generator=g).to(DEV)
        for sink in (None, torch.randn(H, generator=g).to(DEV)):
            got = []
            for runs, zeros in ((False, None), (True, None), (False, torch.zeros(H, 1, device=DEV))):
                out = torch.full((len(pos), H * vd), 3.0, device=DEV)
                ops.attention_simt(q, H * hd, out, ks, vs, table, pos, slot, len(pos), H, KV, hd, 0.2, value_dim=vd, sink=sink, distance_bias=zeros, runs=runs)
                got.append(out)
            assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2]) and bool(torch.isfinite(got[0]).all()) and bool((got[0][-3:] == 3.0).all())


# four and two rows a lane of the kernel of prompts, four, two and one heads together, runs that end within a CTA's rows, single rows between them
@pytest.mark.parametrize("H,KV,hd,vd,starts,news", [(32, 8, 64, 64, [3, 70, 0], [600, 1, 9]), (16, 8, 32, 28, [0], [619]), (12, 4, 96, 96, [0, 40], [500, 333]),
                                                    (32, 8, 128, 128, [100, 0], [130, 20]), (20, 10, 36, 64, [0, 5], [90, 100]), (5, 5, 64, 32, [0, 33], [250, 250])])
def test_float32_attention_of_long_prompts_has_the_same_bits(H, KV, hd, vd, starts, news):
    from kuiperllama_b200.csrc import ops
    g = torch.Generator().manual_seed(H * hd)
    pages = 11
    table = torch.randperm(len(news) * pages, generator=g).to(torch.int32).view(len(news), pages).to(DEV)
    kc, vc = torch.randn(len(news) * pages, KV, 64, hd, generator=g).to(DEV), torch.randn(len(news) * pages, KV, 64, vd, generator=g).to(DEV)
    for s, (a, n) in enumerate(zip(starts, news)):
        for p in range(a + n, pages * 64):
            kc[int(table[s, p // 64]), :, p % 64], vc[int(table[s, p // 64]), :, p % 64] = float("inf"), float("nan")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pos = i32([a + t for a, n in zip(starts, news) for t in range(n)] + [0, 0])
    slot = i32([s for s, n in enumerate(news) for _ in range(n)] + [-1, -1])
    q, sink = torch.randn(len(pos), H * hd, generator=g).to(DEV), torch.randn(H, generator=g).to(DEV)
    for sink in (None, sink):
        got = []
        for runs, zeros in ((True, None), (0, torch.zeros(H, 1, device=DEV))):
            out = torch.full((len(pos), H * vd), 3.0, device=DEV)
            ops.attention_simt(q, H * hd, out, kc, vc, table, pos, slot, len(pos), H, KV, hd, 0.2, value_dim=vd, sink=sink, distance_bias=zeros, runs=runs)
            got.append(out)
        assert torch.equal(got[0], got[1]) and bool(torch.isfinite(got[0]).all()) and bool((got[0][-2:] == 3.0).all())


# rows x heads on both sides of what tiles of eight rows, tiles of one row and a CTA per row each take; rows of 32 columns read at a time
# and a remainder; values in one to sixteen columns a lane
@pytest.mark.parametrize("H,KV,hd,vd,starts,news", [(8, 2, 64, 64, [0, 200], [390, 56]), (4, 4, 128, 128, [0], [256]), (4, 1, 36, 32, [5, 0], [240, 250]),
                                                    (32, 8, 64, 64, [250, 30, 63], [1, 1, 1]), (32, 8, 64, 64, [100] * 3, [4, 5, 6]), (40, 8, 100, 96, [90], [6]),
                                                    (64, 1, 128, 64, [300, 20], [1, 2]), (16, 2, 32, 20, [0], [30])])
def test_float32_attention_by_tiles_and_by_rows_has_the_same_bits(H, KV, hd, vd, starts, news):
    from kuiperllama_b200.csrc import ops
    g = torch.Generator().manual_seed(H + hd)
    pages = 8
    table = torch.randperm(len(news) * pages, generator=g).to(torch.int32).view(len(news), pages).to(DEV)
    kc, vc = torch.randn(len(news) * pages, KV, 64, hd, generator=g).to(DEV), torch.randn(len(news) * pages, KV, 64, vd, generator=g).to(DEV)
    pos = torch.tensor([a + t for a, n in zip(starts, news) for t in range(n)], dtype=torch.int32, device=DEV)
    slot = torch.tensor([s for s, n in enumerate(news) for _ in range(n)], dtype=torch.int32, device=DEV)
    q, got = torch.randn(len(pos), H * hd, generator=g).to(DEV), []
    for runs, zeros in ((False, None), (True, None), (False, torch.zeros(H, 1, device=DEV))):
        out = torch.full((len(pos), H * vd), 3.0, device=DEV)
        ops.attention_simt(q, H * hd, out, kc, vc, table, pos, slot, len(pos), H, KV, hd, 0.2, value_dim=vd, distance_bias=zeros, runs=runs)
        got.append(out)
    assert torch.equal(got[0], got[2]) and torch.equal(got[1], got[2])
    flat = lambda c, s: c[table[s].long()].permute(1, 0, 2, 3).reshape(KV, pages * 64, -1).double().repeat_interleave(H // KV, 0)
    for s in range(len(news)):
        mine = slot == s
        sc = torch.einsum("thd,hjd->thj", q[mine].double().view(-1, H, hd), flat(kc, s)) * 0.2
        sc = sc.masked_fill(torch.arange(pages * 64, device=DEV)[None, None] > pos[mine][:, None, None], float("-inf"))
        w, v = torch.softmax(sc, -1), flat(vc, s)
        want, most = torch.einsum("thj,hjd->thd", w, v), torch.einsum("thj,hjd->thd", w, v.abs())
        # a score is off by hd roundings of its largest partial sum, which the exponential passes on; the sums by one rounding a key
        score = 0.2 * torch.einsum("thd,hjd->thj", q[mine].double().abs().view(-1, H, hd), flat(kc, s).abs()).amax()
        assert bool(((got[0][mine].double().view(want.shape) - want).abs() <= (2 * (hd + 4) * score + 512 + 32) * U * most).all())


@pytest.mark.parametrize("H,G,d,dv", [(4, 2, 16, 24), (2, 1, 32, 8), (4, 4, 64, 48), (2, 1, 100, 36), (3, 1, 256, 20)])
def test_delta_rule_has_the_same_bits_however_a_prompt_is_cut(H, G, d, dv):
    """Whole tiles of eight tokens and tokens one by one, over every number of lanes a column is cut into."""
    from kuiperllama_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(d)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    C, T = 2 * G * d + H * dv, 37
    proj, taps = rand(T, C + 2 * H), rand(C, 4)
    A_log, dt_bias = 0.1 * rand(H), rand(H) - 3.0
    got = []
    for cuts in ([T], [8, 8, 21], [1] * T, [5, 16, 3, 13]):
        state, outs, at = torch.zeros(1, H * d * dv + 3 * C, device=DEV), [], 0
        for n in cuts:
            out = torch.empty(n, H * dv, device=DEV)
            ops.gated_delta_rule(proj[at:at + n], 0, C, C + H, taps, A_log, dt_bias, state, H * d * dv, out, _step([at], [n]), H, G, d, dv, d ** -0.5, 1e-6)
            outs.append(out)
            at += n
        got.append((torch.cat(outs), state))
    for out, state in got[1:]:
        assert torch.equal(out, got[0][0]) and torch.equal(state, got[0][1])


# ------------------------------------------------------------------------------------------------ products with few tiles

def _rand(rows, cols, seed):
    return (torch.randn(rows, cols, generator=torch.Generator().manual_seed(seed)) / cols ** 0.25).to(torch.bfloat16).to(DEV)


@pytest.mark.parametrize("M,N,K", [(1, 8, 64), (64, 1024, 72), (127, 136, 8), (129, 128, 512), (200, 2056, 640), (1025, 2048, 1032), (640, 3712, 128)])
@pytest.mark.parametrize("f32_out", [False, True])
def test_tiles_of_128_features_give_the_sums_of_the_larger_tiles(M, N, K, f32_out):
    from kuiperllama_b200.csrc import ops
    # the first rows of a product with too many tokens for the small tiles have the same sums, added in the same order
    many = 128 * (148 // -(-N // 128) + 2)
    if M >= many:
        many = M + 128
    a, w = _rand(many, K, seed=M), _rand(N, K, seed=N)
    dt = torch.float32 if f32_out else torch.bfloat16
    few, all_rows = torch.full((M + 1, N), 7.0, dtype=dt, device=DEV), torch.empty(many, N, dtype=dt, device=DEV)
    assert ops.one_wave(M, N) and not ops.one_wave(many, N)
    ops.gemm_tcgen05(a[:M], w, few[:M])
    ops.gemm_tcgen05(a, w, all_rows)
    assert torch.equal(few[:M], all_rows[:M])
    assert bool((few[M] == 7.0).all())
    exact = a[:M].double() @ w.double().T
    # K exact products added in 32 bits (and one rounding to 8 bits of the bfloat16 result)
    bound = (a[:M].double().abs() @ w.double().abs().T) * K * 2.0 ** -24 + (0 if f32_out else exact.abs() * 2.0 ** -8) + 1e-30
    assert bool(((few[:M].double() - exact).abs() <= bound).all())


@pytest.mark.parametrize("M", [16, 17, 32, 33, 128, 129, 512, 513])
@pytest.mark.parametrize("N,K", [(256, 2048), (256, 2056), (2048, 4096), (1280, 4104), (19072, 256), (8192, 2048)])
def test_products_on_both_sides_of_the_lines_between_the_ways_round(M, N, K):
    from kuiperllama_b200.csrc import ops
    a, w = _rand(M, K, seed=M), _rand(N, K, seed=K)
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    ops.matmul(a, w, out)
    exact = a.double() @ w.double().T
    bound = (a.double().abs() @ w.double().abs().T) * K * 2.0 ** -24 + exact.abs() * 2.0 ** -8 + 1e-30
    assert bool(((out.double() - exact).abs() <= bound).all())
    # the gated form of the same product: rows alternate 64 gate rows and 64 up rows
    gated = torch.empty(M, N // 2, dtype=torch.bfloat16, device=DEV)
    ops.matmul_swiglu(a, w, gated)
    blocks = exact.view(M, N // 128, 2, 64)
    g, u = blocks[:, :, 0].reshape(M, -1), blocks[:, :, 1].reshape(M, -1)
    want = g * torch.sigmoid(g) * u
    slack = (a.double().abs() @ w.double().abs().T).view(M, N // 128, 2, 64) * K * 2.0 ** -24
    dg, du = slack[:, :, 0].reshape(M, -1), slack[:, :, 1].reshape(M, -1)
    # |d silu / dg| <= 1.1; the two units' exponential and quotient are good to about 2^-20; one rounding to 8 bits
    bound = 1.1 * dg * u.abs() + (g * torch.sigmoid(g)).abs() * du + want.abs() * (2.0 ** -8 + 2.0 ** -18) + 1e-30
    assert bool(((gated.double() - want).abs() <= bound + 1e-6).all())


def _softmax_over_keys(sc, hidden, sink):
    """[T, heads, keys] scores in float64 -> weights; a sink joins the denominator."""
    sc = sc.masked_fill(hidden, float("-inf"))
    top = sc.amax(-1, keepdim=True)
    if sink is not None:
        top = torch.maximum(top, sink.double()[None, :, None])
    e = torch.exp(sc - top)
    return e / (e.sum(-1, keepdim=True) + (0.0 if sink is None else torch.exp(sink.double()[None, :, None] - top)))


# heads on key/value heads in groups of 1 to 16; windows of one key, inside a page, over pages and longer than the prompts; portions that
# start in the middle of a page, whose earlier pages have gone back to the pool
@pytest.mark.parametrize("H,KV,hd", [(8, 8, 64), (8, 2, 64), (4, 1, 128), (16, 1, 64), (6, 2, 128)])
@pytest.mark.parametrize("window", [1, 40, 64, 130, 1000, 0])
@pytest.mark.parametrize("with_sink", [False, True])
def test_attention_tcgen05_with_windows_and_sinks(H, KV, hd, window, with_sink):
    """Outputs are off by their own rounding (2^-9) and by the weights' (2^-9 of each): 2^-8 of sum w |v|, and 2^-8 of the result."""
    from kuiperllama_b200.csrc import ops
    g = torch.Generator().manual_seed(H + hd + window)
    bf, pages = torch.bfloat16, 8
    table = torch.randperm(3 * pages, generator=g).to(torch.int32).view(3, pages)
    kc, vc = (torch.randn(3 * pages, KV, 64, hd, generator=g).to(bf) for _ in range(2))
    sink = torch.randn(H, generator=g) * 3 if with_sink else None
    for starts, news in (([0, 0, 0], [300, 8, 129]), ([100, 63, 200], [30, 12, 256]), ([0, 250, 64], [512, 9, 64])):
        step = _step(starts, news)
        q = (2 * torch.randn(step.n_tokens, H * hd + 16, generator=g)).to(bf)
        k, v, used = kc.clone(), vc.clone(), table.clone()
        for s, (a, n) in enumerate(zip(starts, news)):
            before = max(0, a - window + 1) // 64 if window else 0
            for b in range(before):                        # what a window leaves behind belongs to others now
                k[int(table[s, b])] = v[int(table[s, b])] = float("nan")
                used[s, b] = -1
        out = torch.full((step.n_tokens, H * hd), 9.0, dtype=bf, device=DEV)
        ops.attention_tcgen05(q.to(DEV)[:, :H * hd], H * hd + 16, out, k.to(DEV), v.to(DEV), used.to(DEV), step.cu_tokens, step.seq_slots, step.seq_starts,
                              step.seq_new, 3, step.max_new, step.n_tokens, H, KV, hd, hd ** -0.5, window, None if sink is None else sink.to(DEV))
        ops.check_status(out.device)
        for s, (a, n) in enumerate(zip(starts, news)):
            flat = lambda c: c[table[s].long()].permute(1, 0, 2, 3).reshape(KV, pages * 64, hd).double().repeat_interleave(H // KV, 0).to(DEV)
            i, j = torch.arange(a, a + n, device=DEV)[:, None], torch.arange(pages * 64, device=DEV)[None]
            hidden = (j > i) | ((i - j >= window) if window else torch.zeros(n, pages * 64, dtype=torch.bool, device=DEV))
            rows = slice(step.cu[s], step.cu[s + 1])
            sc = torch.einsum("thd,hjd->thj", q[rows, :H * hd].double().view(n, H, hd).to(DEV), flat(kc)) * hd ** -0.5
            w = _softmax_over_keys(sc, hidden[:, None], None if sink is None else sink.to(DEV))
            want, most = torch.einsum("thj,hjd->thd", w, flat(vc)), torch.einsum("thj,hjd->thd", w, flat(vc).abs())
            off = (out[rows].double().view(n, H, hd) - want).abs()
            assert bool((off <= 2.0 ** -8 * (want.abs() + most)).all()), (s, float((off / most).max()))


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("window", [1024, 0])
def test_attention_into_rows_between_16_byte_boundaries(hd, window):
    """Results that start on a 4-byte boundary are written by the kernel whose stores are that small; asked for by name, tcgen05 refuses them."""
    from kuiperllama_b200.csrc import ops
    g, bf, H, KV, T = torch.Generator().manual_seed(hd), torch.bfloat16, 8, 2, 700
    kc, vc = (torch.randn(11, KV, 64, hd, generator=g).to(bf).to(DEV) for _ in range(2))
    q, table = torch.randn(T, H * hd, generator=g).to(bf).to(DEV), torch.arange(11, dtype=torch.int32, device=DEV).view(1, 11)
    step = _step([0], [T])
    step.is_decode, step.max_context = False, T
    room = torch.full((T * H * hd + 8,), 7.0, dtype=bf, device=DEV)
    out, aligned = room[2:2 + T * H * hd].view(T, H * hd), torch.empty(T, H * hd, dtype=bf, device=DEV)
    for o in (out, aligned):
        ops.attention(q, H * hd, o, kc, vc, table, step, H, KV, hd, hd ** -0.5, window)
    assert float((out.double() - aligned.double()).norm() / aligned.double().norm()) <= 2.0 ** -7      # (two kernels: weights and results rounded to 2^-9)
    assert bool((room[:2] == 7.0).all()) and bool((room[2 + T * H * hd:] == 7.0).all())
    with pytest.raises(ops.KernelError):
        ops.attention_tcgen05(q, H * hd, out, kc, vc, table, step.cu_tokens, step.seq_slots, step.seq_starts, step.seq_new, 1, T, T, H, KV, hd, hd ** -0.5, window)


# a head's own 64 or 128 columns beside 16 to 64 rotated ones, ranks on both sides of a slab of 64, one to several tiles of 128 rows
@pytest.mark.parametrize("H,d,rd,r", [(3, 64, 32, 256), (2, 64, 16, 72), (2, 64, 64, 64), (2, 128, 64, 256), (1, 128, 48, 512), (5, 64, 48, 128)])
@pytest.mark.parametrize("window,with_sink,with_gate", [(0, True, True), (0, False, False), (70, True, False), (300, False, True)])
def test_latent_attention_with_keys_of_every_heads_own(H, d, rd, r, window, with_sink, with_gate):
    """Rotation, norm, the rows of the latent, and scores and sums over every head's own keys and values; one prompt's latent is not
    finite and no other prompt notices.  Keys, values, weights and results are rounded to bfloat16 (2^-9 each); scores are at most a few units, whose
    errors of 2^-9 from keys and queries the weights pass on."""
    from kuiperllama_b200.csrc import ops
    g = torch.Generator().manual_seed(H + d + r + window)
    bf, news, bad = torch.bfloat16, [300, 128, 7, 200], 2
    step = _step([0, 0, 0, 0], news)
    step.host_starts, step.captured, step.padded = [0, 0, 0, 0], False, False
    n, width = step.n_tokens, H * (d + rd)
    proj = torch.randn(n, width + r + rd + 8, generator=g).to(bf)
    proj[step.cu[bad]:step.cu[bad + 1], width:] = float("inf")
    w_norm, freq = 1 + 0.1 * torch.randn(r, generator=g), torch.rand(rd // 2, generator=g)
    w = (torch.randn(2 * H * d, r, generator=g) * r ** -0.5).to(bf)
    sink, gate = torch.randn(H, generator=g), torch.randn(n, H + 8, generator=g).to(bf)
    table = torch.randperm(24, generator=g).to(torch.int32).view(4, 6).to(DEV)
    cache = torch.zeros(24, 1, 64, r + rd, dtype=bf, device=DEV)
    p = proj.to(DEV)
    q = p[:, :width]
    assert ops.latent_expands(step, q) and ops.latent_expandable(bf, d, rd, d, r, 0.1)
    rows = torch.zeros(ops.latent_rows(step), r, dtype=bf, device=DEV)
    ops.latent_prepare(p, 0, width, w_norm.to(DEV), 1e-6, freq.to(DEV), rd, 1.25, True, step.positions, step.token_slot, table, cache, None, n, H, d, rd, r,
                       rows=rows, step=step)
    # against the kernel that leaves the queries where they lie: the same cache, the same rotated parts
    qfull, other = torch.zeros(n, H * (r + rd), dtype=bf, device=DEV), torch.zeros_like(cache)
    ops.latent_prepare(proj.to(DEV), 0, width, w_norm.to(DEV), 1e-6, freq.to(DEV), rd, 1.25, True, step.positions, step.token_slot, table, other, qfull, n, H, d, rd, r)
    same = lambda x, y: torch.equal(x.view(torch.int16), y.view(torch.int16))
    assert same(cache, other) and same(q.reshape(n, H, d + rd)[..., d:].contiguous(), qfull.view(n, H, r + rd)[..., r:].contiguous())
    assert same(q.reshape(n, H, d + rd)[..., :d].contiguous(), proj[:, :width].to(DEV).reshape(n, H, d + rd)[..., :d].contiguous())
    kv = torch.empty(rows.shape[0], 2 * H * d, dtype=bf, device=DEV)
    ops.matmul(rows, w.to(DEV), kv)
    scale, out = 0.3 * (d + rd) ** -0.5, torch.full((n, H * d), 9.0, dtype=bf, device=DEV)
    ops.latent_expanded(q, kv, out, cache, table, step, H, d, rd, d, r, scale, sink.to(DEV) if with_sink else None, window,
                        gate.to(DEV)[:, 4:4 + H] if with_gate else None)
    ops.check_status(out.device)
    for s, m in enumerate(news):
        if s == bad:
            continue
        mine = slice(step.cu[s], step.cu[s + 1])
        flat = cache[table[s].long()].reshape(-1, r + rd)[:m].double()
        k, v = (flat[:, :r] @ x.to(DEV).double().T for x in (w[:H * d], w[H * d:]))
        k = torch.cat([k.view(m, H, d), flat[:, None, r:].expand(m, H, rd)], -1)
        i, j = torch.arange(m, device=DEV)[:, None], torch.arange(m, device=DEV)[None]
        hidden = (j > i) | ((i - j >= window) if window else torch.zeros(m, m, dtype=torch.bool, device=DEV))
        sc = torch.einsum("thd,jhd->thj", q[mine].double().view(m, H, d + rd), k) * scale
        weight = _softmax_over_keys(sc, hidden[:, None], sink.to(DEV) if with_sink else None)
        f = torch.sigmoid(gate[mine, 4:4 + H].to(DEV).double())[..., None] if with_gate else 1.0
        want = torch.einsum("thj,jhd->thd", weight, v.view(m, H, d)) * f
        most = torch.einsum("thj,jhd->thd", weight, v.view(m, H, d).abs()) * f
        # a score's error: 2^-9 of |q| |k| over the own columns of k, in root mean square over d terms a few times less
        err = scale * 2.0 ** -9 * torch.einsum("thd,jhd->thj", q[mine].double().view(m, H, d + rd).abs()[..., :d], k.abs()[..., :d]).amax()
        off = (out[mine].double().view(m, H, d) - want).abs()
        assert bool((off <= 2.0 ** -8 * want.abs() + (2.0 ** -7 + 2 * float(err)) * most).all()), (s, float((off / most).max()))
        assert float((out[mine].double().view(m, H, d) - want).norm() / want.norm()) <= 6e-3


def _delta_inputs(H, G, d, dv, rows, n_seqs, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    C = 2 * G * d + H * dv
    room = torch.full((rows, -(-(C + 2 * H + 12) // 4) * 4), float("nan"), dtype=torch.bfloat16, device=DEV)
    room[:, 4:4 + C + 2 * H] = rand(rows, C + 2 * H)
    A_log, dt_bias = torch.log(1 + 15 * torch.rand(H, device=DEV, generator=g)), rand(H) - 4.0
    return dict(proj=room, taps=0.5 * rand(C, 4), A_log=A_log, dt_bias=dt_bias, state=0.1 * rand(n_seqs, H * d * dv + 3 * C + 4), C=C)


def _delta(x, step, H, G, d, dv, chunked, scale=0.1):
    from kuiperllama_b200.csrc import ops
    state, out = x["state"].clone(), torch.full((step.n_tokens, H * dv), 7.0, device=DEV)
    ops.gated_delta_rule(x["proj"], 4, 4 + x["C"], 4 + x["C"] + H, x["taps"], x["A_log"], x["dt_bias"], state, H * d * dv, out, step, H, G, d, dv, scale, 1e-6,
                         chunked=chunked)
    return out, state


# keys of one slab of 64 and of two, with a remainder; values of one 16 and of more than 128; heads that share keys; chunks of one token, of the
# first block alone, whole ones and remainders
@pytest.mark.parametrize("H,G,d,dv", [(4, 1, 128, 128), (3, 3, 64, 32), (2, 1, 40, 144), (6, 2, 128, 16), (2, 2, 72, 48)])
@pytest.mark.parametrize("news", [[200, 1, 33, 64], [96]])
def test_delta_rule_in_chunks(H, G, d, dv, news):
    """As exact as token by token, with the convolution from and into its state; both are off by sums of float32 numbers of order one: a few
    units of 2^-24 a token at most, whose effect the rule itself damps."""
    step = _step([0] * len(news), news)
    x = _delta_inputs(H, G, d, dv, step.n_tokens, len(news), d + dv)
    C, wide, S, want = x["C"], x["proj"].double(), [], []
    for s in range(len(news)):
        rows = slice(step.cu[s], step.cu[s + 1])
        past = x["state"][s, H * d * dv:H * d * dv + 3 * C].double().view(3, C)
        pad = torch.cat([past, wide[rows, 4:4 + C]])
        y = sum(pad[j:j + news[s]] * x["taps"].double()[:, j] for j in range(4))
        y = y * torch.sigmoid(y)
        q, k, v = y[:, :G * d].view(-1, G, d), y[:, G * d:2 * G * d].view(-1, G, d), y[:, 2 * G * d:].view(-1, H, dv)
        q, k = ((z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1) for z in (q, k))
        beta = torch.sigmoid(wide[rows, 4 + C:4 + C + H])
        decay = torch.exp(-torch.exp(x["A_log"].double()) * torch.nn.functional.softplus(wide[rows, 4 + C + H:4 + C + 2 * H] + x["dt_bias"].double()))
        M = x["state"][s, :H * d * dv].double().view(H, d, dv).clone()
        for t in range(news[s]):
            M = M * decay[t][:, None, None]
            M = M + k[t][:, :, None] * (beta[t][:, None] * (v[t] - torch.einsum("hd,hdv->hv", k[t], M)))[:, None]
            want.append(0.1 * torch.einsum("hd,hdv->hv", q[t], M))
        S.append(M)
    want, S = torch.stack(want), torch.stack(S)
    off = lambda r: (float((r[0].double().view(want.shape) - want).norm() / want.norm()), float((r[1][:, :H * d * dv].double().view(S.shape) - S).norm() / S.norm()))
    walked, chunked = _delta(x, step, H, G, d, dv, False), _delta(x, step, H, G, d, dv, True)
    for a, b in zip(off(chunked), off(walked)):
        assert a <= 1.5 * b + 2 * U and a <= 64 * U
    assert torch.equal(walked[1][:, H * d * dv:], chunked[1][:, H * d * dv:])              # the convolution's state, and what lies behind it
    again = _delta(x, step, H, G, d, dv, True)
    assert torch.equal(again[0], chunked[0]) and torch.equal(again[1], chunked[1])


@pytest.mark.parametrize("what", ["q", "k", "v", "beta", "decay", "state", "large"])
def test_delta_rule_in_chunks_keeps_what_is_not_finite_where_it_arises(what):
    H, G, d, dv, news = 4, 2, 64, 32, [100, 70]
    step = _step([0, 0], news)
    x = _delta_inputs(H, G, d, dv, 170, 2, 3)
    C, p = x["C"], x["proj"]
    bad = float("nan")
    if what == "state":
        x["state"][1, 77] = float("inf")
    elif what == "large":
        p[50, 4 + 2 * G * d + 3] = 1e9
    else:
        col = {"q": 4 + 5, "k": 4 + G * d + 70, "v": 4 + 2 * G * d + 40, "beta": 4 + C + 1, "decay": 4 + C + H + 2}[what]
        p[40, col], p[130, col] = bad, float("inf") if what != "v" else bad
    (a, sa), (b, sb) = _delta(x, step, H, G, d, dv, False), _delta(x, step, H, G, d, dv, True)
    for y, z in ((a, b), (sa, sb)):
        fine = torch.isfinite(y)
        assert torch.equal(fine, torch.isfinite(z))
        assert float((y - z)[fine].double().norm()) <= 4e-6 * float(y[fine].double().norm())


def test_delta_rule_of_steps_that_the_chunks_do_not_take():
    """float32 rows (whose bits do not depend on how a prompt is cut), odd sizes, rows between 8-byte boundaries and short sequences go token by token."""
    from kuiperllama_b200.csrc import ops
    for d, dv, dtype, shift, news in ((64, 32, torch.float32, 4, [130]), (20, 32, torch.bfloat16, 4, [130]), (64, 20, torch.bfloat16, 4, [130]),
                                      (64, 32, torch.bfloat16, 3, [130]), (64, 32, torch.bfloat16, 4, [90]), (64, 32, torch.bfloat16, 4, [100, 1, 1, 1])):
        step = _step([0] * len(news), news)
        x = _delta_inputs(2, 1, d, dv, step.n_tokens, len(news), d)
        proj = x["proj"].nan_to_num(0.0).to(dtype)
        got = []
        for chunked in (None, False):
            state, out = x["state"].clone(), torch.empty(step.n_tokens, 2 * dv, device=DEV)
            ops.gated_delta_rule(proj, shift, shift + x["C"], shift + x["C"] + 2, x["taps"], x["A_log"], x["dt_bias"], state, 2 * d * dv, out, step, 2, 1, d, dv, 0.1,
                                 1e-6, chunked=chunked)
            got.append((out, state))
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("news", [[700], [200, 1, 333, 64, 40], [97, 96]])
@pytest.mark.parametrize("chunks", [0, 1, 7, 12])
def test_chunks_in_portions_have_the_same_bits(monkeypatch, news, chunks):
    """What a step's chunks take is bounded: beyond it a step is worked in portions, one chunk a sequence at the least, with the same results."""
    from kuiperllama_b200.csrc import ops
    step, H, G, d, dv = _step([0] * len(news), news), 4, 2, 64, 32
    x = _delta_inputs(H, G, d, dv, step.n_tokens, len(news), 9)
    g = torch.Generator(device=DEV).manual_seed(7)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    n, p, rows = 64, 48, step.n_tokens
    q, k, v = (rand(rows, 2 * n), 0.3 * rand(rows, 2 * n), rand(rows, 4 * p))
    decay = {False: torch.rand(rows, 4, device=DEV, generator=g) ** 0.1, True: torch.rand(rows, 4 * n, device=DEV, generator=g) ** 0.1}
    qb, kb, state0 = rand(rows, 4 * n).bfloat16(), rand(rows, 4 * n).bfloat16(), 0.1 * rand(len(news), 4 * n * p)

    def outer(per_row):
        state, y = state0.clone(), torch.full((rows, 4 * p), 7.0, device=DEV)
        ops.outer_recurrence(qb if per_row else q, kb if per_row else k, v.bfloat16() if per_row else v, decay[per_row], state, y, step, 4, 4 if per_row else 2, n, p,
                             q_scale=0.7, chunked=True)
        return y, state

    whole = [_delta(x, step, H, G, d, dv, True), outer(False), outer(True)]
    # bytes of a chunk of every sequence: the pieces of q and k for every unit, and what the products and factors take
    sizes = [2 * 24576 + 4 * (12288 + 6144 + 512 + 4096), 2 * 24576 + 2 * (32 * 36 + 4) * 4 + 4 * (32 * 20 + 4) * 4, 4 * (24576 + 6144 + 512)]
    for want, one, run in zip(whole, sizes, (lambda: _delta(x, step, H, G, d, dv, True), lambda: outer(False), lambda: outer(True))):
        monkeypatch.setattr(ops, "CHUNK_SCRATCH", one * chunks * len(news))
        before = ops.launch_count
        got = run()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        portions = -(-(-(-max(news) // 32)) // max(1, chunks))
        if chunks <= 1 or len(news) == 1:
            assert ops.launch_count - before in (2 * portions, 2 * portions + 1)
        monkeypatch.undo()


def test_scratch_of_a_long_step_is_bounded():
    from kuiperllama_b200.csrc import ops
    import ctypes
    limit = ctypes.c_longlong(ops.CHUNK_SCRATCH)
    for n, seqs in ((32768, 1), (131072, 1), (131072, 8)):
        outer = ops.lib("outer_chunked").kl_outer_chunked_scratch(n, seqs, n, 64, 1, 128, 0, limit)
        rows = n * (2 * 4 * 128 + 16 * 128 + 32) * 4                           # what is prepared of every row, as token by token
        delta = ops.lib("delta_chunked").kl_delta_chunked_scratch(n, seqs, n, 16, 4, 128, 128, limit) - rows
        assert outer <= ops.CHUNK_SCRATCH + 4096 and delta <= ops.CHUNK_SCRATCH + 4096, (outer, delta)


def test_delta_rule_with_taps_between_16_byte_boundaries():
    """A contiguous view of the taps at another offset is served as before, token by token."""
    from kuiperllama_b200.csrc import ops
    H, G, d, dv = 2, 1, 64, 32
    step = _step([0], [130])
    x = _delta_inputs(H, G, d, dv, 130, 1, 4)
    room = torch.empty(x["C"] * 4 + 4, device=DEV)
    taps = room[1:1 + x["C"] * 4].view(x["C"], 4)
    taps.copy_(x["taps"])
    walked = _delta(x, step, H, G, d, dv, False)
    got = _delta(dict(x, taps=taps), step, H, G, d, dv, None)
    assert torch.equal(got[0], walked[0]) and torch.equal(got[1], walked[1])
    with pytest.raises(ops.KernelError):
        _delta(dict(x, taps=taps), step, H, G, d, dv, True)


# both sides of where products of few tokens cut K, take the weights as tile rows, and need a second wave of tiles; chunks of 16 tokens with a remainder
@pytest.mark.parametrize("M,N,K", [(33, 3072, 1024), (48, 6144, 512), (64, 200, 1024), (24, 520, 4096), (17, 1024, 264), (64, 2048, 2048)])
def test_products_of_few_tokens(M, N, K):
    """float64 within the rounding of the result and 2^-18 of the sum of the terms' magnitudes (32-bit sums of K terms in any order)."""
    from kuiperllama_b200.csrc import ops
    g = torch.Generator().manual_seed(M * N)
    a, w = torch.randn(M, K, generator=g).bfloat16().to(DEV), torch.randn(N, K, generator=g).bfloat16().to(DEV)
    want, most = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    ops.matmul(a, w, out)
    pieces = ops.gemm_skinny_partials(a, w)
    assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * most).all())
    assert pieces is None or bool(((pieces.double().sum(0) - want).abs() <= 2.0 ** -18 * most).all())


@pytest.mark.parametrize("M,I,K", [(24, 256, 520), (32, 64, 128), (48, 9536, 64), (64, 9536, 72), (33, 512, 192)])
@pytest.mark.parametrize("activation", ["silu", "relu"])
def test_gate_up_products_of_few_tokens(M, I, K, activation):
    """The same; the gate's factor has a slope of at most 1.1, so act(g) u is off by no more than 1.1 |u| dg + |act(g)| du beside the rounding of the
    result, whose bound of 2^-8 is twice what rounding takes and holds the factor's own error (2^-17 where exp is large)."""
    from kuiperllama_b200.csrc import ops
    g = torch.Generator().manual_seed(M + I)
    a = torch.randn(M, K, generator=g).bfloat16().to(DEV)
    gate, up = (torch.randn(I, K, generator=g).bfloat16().to(DEV) for _ in range(2))
    w = ops.interleave_gate_up(gate, up)
    G, U = a.double() @ gate.double().T, a.double() @ up.double().T
    dG, dU = (2.0 ** -18 * (a.double().abs() @ x.double().abs().T) for x in (gate, up))
    act = torch.nn.functional.silu(G) if activation == "silu" else torch.relu(G)
    out = torch.empty(M, I, dtype=torch.bfloat16, device=DEV)
    ops.matmul_swiglu(a, w, out, activation)
    assert bool(((out.double() - act * U).abs() <= 2.0 ** -8 * (act * U).abs() + 1.1 * U.abs() * dG + act.abs() * dU + dG * dU + 1e-30).all())
