"""Recurrences with one decay per head walked sixteen tokens at a time (``kernels.block_walk``) against the recurrences
themselves, token by token in 64 bits."""
import numpy as np
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


def _recurrence(q, k, v, g, w, S, delta, skip):
    """q, k [T, heads, N], v [T, heads, V], g and w [T, heads], S [heads, N, V], all float64."""
    out = []
    for t in range(q.shape[0]):
        S = g[t][:, None, None] * S
        u = w[t][:, None] * (v[t] - (np.einsum("hnv,hn->hv", S, k[t]) if delta else 0.0))
        S = S + k[t][:, :, None] * u[:, None, :]
        out.append(np.einsum("hnv,hn->hv", S, q[t]) + skip[:, None] * v[t])
    return np.stack(out), S


@pytest.mark.parametrize("heads,G,N,V,lens,slow", [
    (2, 1, 128, 128, [100, 1, 16, 33, 2], True), (24, 8, 72, 64, [50, 3, 16], False),
    (60, 20, 64, 36, [17, 31, 1], False), (150, 50, 12, 12, [33], False), (4, 4, 64, 64, [17, 48], False), (3, 1, 20, 12, [64, 5], True), (6, 2, 68, 36, [40, 15, 1, 1], False),
    (1, 1, 4, 4, [33], False), (32, 1, 128, 64, [50], True)])
@pytest.mark.parametrize("form", ["delta", "weights", "decay"])
def test_block_walk_follows_the_recurrence(form, heads, G, N, V, lens, slow):
    """Blocks that end inside a portion, single tokens beside portions, sizes that fill no fragment, a q/k head shared by
    several heads, decays that hardly decay, new requests and old ones, both layouts of the state.  A product of two
    float32 numbers loses 3 * 2^-22 at most and a block rounds its state once: 1e-5 of the largest value covers 100
    tokens of it."""
    from aien_sovereign_core_mv_b200 import kernels as K
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    f64 = lambda a: a.double().cpu().numpy()
    g_ = torch.Generator().manual_seed(heads * 1000 + N + V)
    T, S, delta, act, state_vn = sum(lens), len(lens), form == "delta", form == "decay", form == "weights"
    GN, s_off, extra = G * N, 5, 3
    rows = torch.randn(T, 4 + 2 * GN + heads * V + 4, generator=g_)
    k = rows[:, 4 + GN:4 + 2 * GN]
    if delta:                                              # unit keys, as the delta rule has them
        k /= k.reshape(T, G, N).norm(dim=-1).repeat_interleave(N, dim=1)
    gates = torch.rand(T, 2 * heads + 1, generator=g_)
    gates[:, :heads] = 1.0 - gates[:, :heads] * (1e-4 if slow else 0.9)
    decay = 1.0 - torch.rand(heads, generator=g_) * (1e-4 if slow else 0.5)
    skip = torch.randn(heads, generator=g_)
    state = torch.randn(S + 2, s_off + heads * N * V + extra, generator=g_)
    slots = [S - s for s in range(S)]
    fresh = [s % 2 == 1 for s in range(S)]
    q0 = [sum(lens[:s]) for s in range(S + 1)]
    dev = state.clone().cuda()
    out = torch.full((T, heads * V), 9.0).cuda()
    blocks = torch.full((K.block_walk_scratch(T, S, heads, G, N, V, act),), float("nan")).cuda()
    took = K.block_walk(rows.cuda(), 4, 4 + GN, 4 + 2 * GN, None if act else gates.cuda(), 0, -1 if act else heads, decay.cuda() if act else None,
                        dev, s_off, i32(slots), i32(q0), i32([(0 if fresh[s] else 7) + p for s, n in enumerate(lens) for p in range(n)]), out, S, heads,
                        G, N, V, blocks, delta=delta, act=act, skip=skip.cuda() if state_vn else None, state_vn=state_vn)
    assert took
    a = f64(rows)
    if act:
        a = a / (1.0 + np.exp(-a))
    for s in range(S):
        r = slice(q0[s], q0[s + 1])
        qk = lambda off: np.repeat(a[r, off:off + GN].reshape(-1, G, N), heads // G, axis=1)
        v = a[r, 4 + 2 * GN:4 + 2 * GN + heads * V].reshape(-1, heads, V)
        S0 = f64(state[slots[s], s_off:s_off + heads * N * V]).reshape((heads, V, N) if state_vn else (heads, N, V))
        S0 = S0.transpose(0, 2, 1) if state_vn else S0
        n = lens[s]
        g, w = (np.tile(f64(decay), (n, 1)), np.ones((n, heads))) if act else (f64(gates[r, :heads]), f64(gates[r, heads:2 * heads]))
        want, last = _recurrence(qk(4), qk(4 + GN), v, g, w, S0 * 0.0 if fresh[s] else S0, delta, f64(skip) if state_vn else np.zeros(heads))
        H.assert_close(out[r].cpu().numpy().reshape(n, heads, V), want, 1e-5, f"request {s}")
        got = dev[slots[s], s_off:s_off + heads * N * V].cpu().numpy().reshape((heads, V, N) if state_vn else (heads, N, V))
        H.assert_close(got.transpose(0, 2, 1) if state_vn else got, last, 1e-5, f"state of request {s}")
    keep = [i for i in range(S + 2) if i not in slots]
    assert torch.equal(dev[keep].cpu(), state[keep]) and torch.equal(dev[:, :s_off].cpu(), state[:, :s_off]) and torch.equal(dev[:, -extra:].cpu(), state[:, -extra:])


@pytest.mark.parametrize("form", ["linear", "duality", "delta"])
@pytest.mark.parametrize("slow", [False, True])
def test_long_portions_lose_no_more_than_token_by_token(form, slow):
    """2,048 tokens whose keys, queries and values are mostly of one sign, so that a rounding that always cuts off would add
    up, under decays that hardly decay (one for all tokens, whose products are the same in every block) and ordinary ones:
    the state is rounded once a block, 128 times, at 2^-25 on the average and either way (3.4e-7 together), and no more
    than as much again comes from what is added to it; relative 2-norms."""
    from aien_sovereign_core_mv_b200 import kernels as K
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    g_ = torch.Generator(device="cuda").manual_seed(7)
    T, heads, G, N, V = 2048, 4, {"linear": 4, "duality": 1, "delta": 2}[form], 128, 64
    silu = lambda x: x * torch.sigmoid(x)
    GN = G * N
    rows = torch.randn(T, 2 * GN + heads * V, generator=g_, device="cuda")
    if form != "linear":
        rows = silu(rows)
    if form == "delta":
        for at in (0, GN):
            part = rows[:, at:at + GN].view(T, G, N)
            rows[:, at:at + GN] = (part / part.norm(dim=-1, keepdim=True)).reshape(T, GN)
    span = 1e-4 if slow else 0.1
    gates = torch.cat([1.0 - span * torch.rand(T, heads, generator=g_, device="cuda"), torch.rand(T, heads, generator=g_, device="cuda")], 1)
    decay = 1.0 - span * (0.1 + 0.9 * torch.rand(heads, generator=g_, device="cuda"))
    act = form == "linear"
    state, out = torch.zeros(1, heads * N * V).cuda(), torch.zeros(T, heads * V).cuda()
    blocks = torch.empty(K.block_walk_scratch(T, 1, heads, G, N, V, act)).cuda()
    assert K.block_walk(rows, 0, GN, 2 * GN, None if act else gates, 0, -1 if act else heads, decay if act else None, state, 0, i32([0]), i32([0, T]),
                        i32(list(range(T))), out, 1, heads, G, N, V, blocks, delta=form == "delta", act=act)
    a = silu(rows.double()) if act else rows.double()
    q, k = (a[:, at:at + GN].view(T, G, N).repeat_interleave(heads // G, dim=1) for at in (0, GN))
    v = a[:, 2 * GN:].view(T, heads, V)
    S, want = torch.zeros(heads, N, V, dtype=torch.float64, device="cuda"), []
    for t in range(T):
        S = (decay if act else gates[t, :heads]).double()[:, None, None] * S
        u = v[t] - torch.einsum("hnv,hn->hv", S, k[t]) if form == "delta" else v[t]
        S = S + k[t][:, :, None] * (u if act else gates[t, heads:].double()[:, None] * u)[:, None]
        want.append(torch.einsum("hnv,hn->hv", S, q[t]))
    rel = lambda x, y: float((x.double().flatten() - y.flatten()).norm() / y.norm())
    assert rel(out, torch.stack(want)) <= 7e-7 and rel(state, S) <= 7e-7


def test_tokens_that_know_nothing_of_one_another_return_their_values_to_the_bit():
    """Every token's key and query is a unit vector of its own, so its result is its own value times one: what lies inside a block is
    multiplied and added in float32, and the state that a query reads is zero there."""
    from aien_sovereign_core_mv_b200 import kernels as K
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    heads, N, V, lens = 3, 64, 48, [37, 16, 1]
    T, S = sum(lens), len(lens)
    g_ = torch.Generator().manual_seed(3)
    rows = torch.zeros(T, 2 * N + heads * V)
    at = torch.cat([torch.randperm(N, generator=g_)[:n] for n in lens])
    rows[torch.arange(T), at] = 1.0
    rows[torch.arange(T), N + at] = 1.0
    rows[:, 2 * N:] = torch.randn(T, heads * V, generator=g_)
    gates = torch.cat([1.0 - 0.5 * torch.rand(T, heads, generator=g_), torch.ones(T, heads)], 1)
    state, out = torch.randn(S, heads * N * V).cuda(), torch.full((T, heads * V), 9.0).cuda()
    q0 = [sum(lens[:s]) for s in range(S + 1)]
    blocks = torch.empty(K.block_walk_scratch(T, S, heads, 1, N, V)).cuda()
    assert K.block_walk(rows.cuda(), 0, N, 2 * N, gates.cuda(), 0, heads, None, state, 0, i32(list(range(S))), i32(q0),
                        i32([p for n in lens for p in range(n)]), out, S, heads, 1, N, V, blocks, delta=False)
    assert torch.equal(out.cpu(), rows[:, 2 * N:])


def test_many_heads_over_one_group_walk_by_blocks():
    """The duality form needs no 16 x 16 system a head, so heads that are too many for the delta rule are not for it."""
    from aien_sovereign_core_mv_b200 import kernels as K
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    T, heads, G, N, V = 40, 128, 1, 128, 4
    assert K.block_walk_takes(torch.bfloat16, 2048, 1, heads, G, N, 64) and not K.block_walk_takes(torch.bfloat16, 2048, 1, heads, G, N, 64, delta=True)
    g_ = torch.Generator().manual_seed(1)
    rows, gates = torch.randn(T, 2 * N + heads * V, generator=g_), 1.0 - 0.9 * torch.rand(T, 2 * heads, generator=g_)
    state, out = torch.zeros(1, heads * N * V).cuda(), torch.zeros(T, heads * V).cuda()
    run = lambda delta: K.block_walk(rows.cuda(), 0, N, 2 * N, gates.cuda(), 0, heads, None, state, 0, i32([0]), i32([0, T]), i32(list(range(T))), out, 1,
                                     heads, G, N, V, torch.empty(K.block_walk_scratch(T, 1, heads, G, N, V)).cuda(), delta=delta, state_vn=True)
    with pytest.raises(K.KernelError):
        run(True)
    assert run(False)
    a, ga = rows.double().numpy(), gates.double().numpy()
    qk = lambda off: np.repeat(a[:, off:off + N].reshape(T, 1, N), heads, axis=1)
    want, last = _recurrence(qk(0), qk(N), a[:, 2 * N:].reshape(T, heads, V), ga[:, :heads], ga[:, heads:], np.zeros((heads, N, V)), False, np.zeros(heads))
    H.assert_close(out.cpu().numpy().reshape(T, heads, V), want, 1e-5, "results")
    H.assert_close(state.cpu().numpy().reshape(heads, V, N).transpose(0, 2, 1), last, 1e-5, "state")


@pytest.mark.parametrize("form", ["delta", "duality"])
@pytest.mark.parametrize("lens", [[1, 40, 1, 33, 1, 1], [2, 1, 17], [50, 1]])
def test_single_tokens_beside_portions(form, lens):
    """Requests of one token go token by token beside the walk of the others: every request against 64 bits, with the walk for
    all of them and for the portions alone, where the single tokens have the bits of the token kernel."""
    from aien_sovereign_core_mv_b200 import kernels as K
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    g_ = torch.Generator().manual_seed(len(lens))
    T, S, heads, G, N, V = sum(lens), len(lens), 6, 2, 68, 36
    GN, s_off, delta = G * N, 3, form == "delta"
    rows = torch.randn(T, 2 * GN + heads * V, generator=g_)
    rows[:, GN:2 * GN] /= rows[:, GN:2 * GN].reshape(T, G, N).norm(dim=-1).repeat_interleave(N, dim=1)
    gb = torch.rand(T, 2 * heads, generator=g_) * 0.9 + 0.1
    dtr, A, bias, D = torch.randn(T, heads, generator=g_), torch.rand(heads, generator=g_), torch.randn(heads, generator=g_) - 2.0, torch.randn(heads, generator=g_)
    state = torch.randn(S, s_off + heads * N * V, generator=g_)
    q0, pos = [sum(lens[:s]) for s in range(S + 1)], [p + (0 if s % 2 else 7) for s, n in enumerate(lens) for p in range(n)]
    singles = [t for s, t in enumerate(q0[:-1]) if lens[s] == 1]
    got = []
    for blocks, alone in ((True, 0), (True, len(singles)), (False, 0)):
        st, out = state.clone().cuda(), torch.zeros(T, heads * V).cuda()
        scratch = torch.full((K.block_walk_scratch(T, S, heads, G, N, V),), float("nan")).cuda() if blocks else None
        common = (st, s_off, i32(list(range(S))), i32(q0), i32(pos), out, S, heads)
        if delta:
            K.delta_rule(rows.cuda(), 0, GN, 2 * GN, gb.cuda(), *common, G, N, V, scratch, alone)
        else:
            K.ssd_scan(rows.cuda(), 2 * GN, GN, 0, dtr.cuda(), A.cuda(), bias.cuda(), D.cuda(), *common, V, G, N, blocks=scratch, alone=alone)
        got.append((out.cpu(), st.cpu()))
    assert torch.equal(got[1][0][singles], got[2][0][singles])
    a = rows.double().numpy()
    dt = np.logaddexp(0.0, (dtr + bias).double().numpy())
    g, w = (gb[:, :heads].double().numpy(), gb[:, heads:].double().numpy()) if delta else (np.exp(-A.double().numpy() * dt), dt)
    for s in range(S):
        r = slice(q0[s], q0[s + 1])
        qk = lambda off: np.repeat(a[r, off:off + GN].reshape(-1, G, N), heads // G, axis=1)
        S0 = state[s, s_off:].double().numpy().reshape((heads, N, V) if delta else (heads, V, N))
        S0 = (S0 if delta else S0.transpose(0, 2, 1)) * (0.0 if s % 2 else 1.0)
        want, last = _recurrence(qk(0), qk(GN), a[r, 2 * GN:].reshape(-1, heads, V), g[r], w[r], S0, delta, np.zeros(heads) if delta else D.double().numpy())
        for out, st in got:
            H.assert_close(out[r].numpy().reshape(want.shape), want, 1e-5, f"request {s}")
            end = st[s, s_off:].numpy().reshape((heads, N, V) if delta else (heads, V, N))
            H.assert_close(end if delta else end.transpose(0, 2, 1), last, 1e-5, f"state of request {s}")


def test_which_steps_walk_by_blocks():
    """By counts alone: enough tokens behind each request's first, and portions that are not short on the average."""
    from aien_sovereign_core_mv_b200 import kernels as K
    takes = lambda T, S, singles: K.block_walk_takes(torch.bfloat16, T, S, 16, 8, 64, 64, singles=singles, least=K.BLOCK_WALK_LEAST)
    assert takes(97, 65, 64) and takes(33, 1, 0) and takes(320, 64, 0) and takes(88, 56, 48)
    assert not takes(128, 64, 0) and not takes(192, 64, 0) and not takes(112, 80, 64) and not takes(32, 1, 0) and not takes(64, 64, 64)
    assert K.block_walk_takes(torch.bfloat16, 128, 64, 16, 16, 64, 64)                 # without a least: linear attention


def test_block_walk_declines_rows_off_the_boundary():
    from aien_sovereign_core_mv_b200 import kernels as K
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    rows, out, state = torch.zeros(40, 26).cuda(), torch.full((40, 8), 3.0).cuda(), torch.ones(2, 64).cuda()
    blocks = torch.empty(K.block_walk_scratch(40, 1, 1, 1, 8, 8)).cuda()
    assert not K.block_walk(rows, 0, 8, 16, None, 0, -1, torch.ones(1).cuda(), state, 0, i32([0]), i32([0, 40]), i32(list(range(40))), out, 1, 1, 1, 8, 8,
                            blocks)
    assert float((out - 3.0).abs().max()) == 0.0 and float((state - 1.0).abs().max()) == 0.0
    assert not K.block_walk_takes(torch.float32, 4096, 1, 4, 2, 64, 64) and not K.block_walk_takes(torch.bfloat16, 64, 64, 4, 2, 64, 64)
    assert not K.block_walk_takes(torch.bfloat16, 4096, 1, 4, 2, 130, 64) and K.block_walk_takes(torch.bfloat16, 4096, 1, 4, 2, 128, 64)


@pytest.mark.parametrize("heads,G,N,V", [(2, 1, 128, 32), (4, 2, 64, 20), (150, 50, 12, 36), (1, 1, 36, 16)])
@pytest.mark.parametrize("form", ["delta", "weights", "decay"])
@pytest.mark.parametrize("where", ["value", "key", "gate", "state"])
@pytest.mark.parametrize("odd", [float("inf"), float("nan")])
def test_a_number_that_is_not_finite_reaches_what_follows_it(odd, where, form, heads, G, N, V):
    """An infinity or NaN in one token's value, key or gate, or in a request's state: every number that the recurrence, token
    by token, leaves finite is the one it would be without blocks (the tokens before it in its block, the other columns,
    heads and requests), and where the recurrence is not, neither is this.  Without the delta rule nothing but sums of one
    infinity is made of an infinite state: it stays one."""
    from aien_sovereign_core_mv_b200 import kernels as K
    if where == "gate" and form == "decay":
        pytest.skip("one decay for all tokens")
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    g_ = torch.Generator().manual_seed(heads + N)
    lens, at = [41, 20], 21                                   # the sixth token of the second block
    T, S, GN, delta, act, vn = sum(lens), 2, G * N, form == "delta", form == "decay", form == "weights"
    rows = torch.randn(T, 2 * GN + heads * V, generator=g_)
    if delta:
        rows[:, GN:2 * GN] /= rows[:, GN:2 * GN].reshape(T, G, N).norm(dim=-1).repeat_interleave(N, dim=1)
    gates = 1.0 - 0.9 * torch.rand(T, 2 * heads, generator=g_)
    decay, skip = 1.0 - 0.5 * torch.rand(heads, generator=g_), torch.randn(heads, generator=g_)
    state = torch.randn(S, heads * N * V, generator=g_)
    h = heads - 1
    if where == "value":
        rows[at, 2 * GN + h * V + V - 1] = odd
    elif where == "key":
        rows[at, 2 * GN - 1] = odd
    elif where == "gate":
        gates[at, h] = odd
    else:
        state[0, h * N * V + 3] = odd
    dev, out = state.clone().cuda(), torch.zeros(T, heads * V).cuda()
    blocks = torch.empty(K.block_walk_scratch(T, S, heads, G, N, V, act)).cuda()
    assert K.block_walk(rows.cuda(), 0, GN, 2 * GN, None if act else gates.cuda(), 0, -1 if act else heads, decay.cuda() if act else None, dev, 0,
                        i32([0, 1]), i32([0, lens[0], T]), i32(list(range(5, 5 + lens[0])) + list(range(9, 9 + lens[1]))), out, S, heads, G, N, V,
                        blocks, delta=delta, act=act, skip=skip.cuda() if vn else None, state_vn=vn)
    a = rows.double().numpy()
    with np.errstate(all="ignore"):
        if act:
            a = a / (1.0 + np.exp(-a))
        for s, r in ((0, slice(0, lens[0])), (1, slice(lens[0], T))):
            qk = lambda off: np.repeat(a[r, off:off + GN].reshape(-1, G, N), heads // G, axis=1)
            S0 = state[s].double().numpy().reshape((heads, V, N) if vn else (heads, N, V))
            S0 = S0.transpose(0, 2, 1) if vn else S0
            g, w = (np.tile(decay.double().numpy(), (lens[s], 1)), np.ones((lens[s], heads))) if act else (gates[r, :heads].double().numpy(), gates[r, heads:].double().numpy())
            want, last = _recurrence(qk(0), qk(GN), a[r, 2 * GN:].reshape(-1, heads, V), g, w, S0, delta, skip.double().numpy() if vn else np.zeros(heads))
            got = out[r].cpu().double().numpy().reshape(want.shape)
            end = dev[s].cpu().double().numpy().reshape((heads, V, N) if vn else (heads, N, V))
            end = end.transpose(0, 2, 1) if vn else end
            for x, y, what in ((got, want, "results"), (end, last, "state")):
                assert np.array_equal(np.isfinite(x), np.isfinite(y)), f"{what} of request {s}"
                ok = np.isfinite(y)
                assert np.abs((x - y)[ok]).max(initial=0.0) <= 1e-5 * np.abs(y[ok]).max(initial=0.0), f"{what} of request {s}"
            assert s == 1 or not np.isfinite(last).all()
            if s == 0 and where == "state" and not delta and np.isinf(odd):
                assert np.isinf(end).sum() == 1 and np.isinf(got).sum() == lens[0]
    assert np.isfinite(out.cpu().numpy()[:at if where != "state" else 0]).all()
