"""Steps of single tokens through the recurrences with a float32 state, whose kernels read whole vectors of it where it lies on
16-byte boundaries, against the recurrences in 64 bits; off the boundaries the general kernels serve the same call."""
import numpy as np
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu

I32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")


def _step(lens, seed):
    """(generator, q_start, positions, slots): every second request is new, slots in no order."""
    q0 = [sum(lens[:s]) for s in range(len(lens) + 1)]
    pos = [p + (0 if s % 2 else 7) for s, n in enumerate(lens) for p in range(n)]
    return torch.Generator().manual_seed(seed), q0, pos, [(s * 2 + 1) % len(lens) for s in range(len(lens))]


def _walk(q, k, v, g, w, S, delta, skip):
    out = []
    for t in range(q.shape[0]):
        S = g[t][:, None, None] * S
        u = w[t][:, None] * (v[t] - (np.einsum("hnv,hn->hv", S, k[t]) if delta else 0.0))
        S = S + k[t][:, :, None] * u[:, None, :]
        out.append(np.einsum("hnv,hn->hv", S, q[t]) + skip[:, None] * v[t])
    return np.stack(out) if out else np.zeros((0,) + v.shape[1:]), S


# heads, q/k groups, N, V, the state's first number; lens: single tokens, a portion beside an empty request, one request
SIZES = [(4, 2, 128, 128, 8), (6, 3, 128, 64, 4), (3, 1, 100, 128, 4), (2, 2, 4, 64, 0), (4, 2, 128, 128, 5), (5, 1, 128, 24, 4), (2, 1, 132, 128, 4), (33, 1, 128, 8, 0)]


@pytest.mark.parametrize("heads,G,N,V,s_off", SIZES)
@pytest.mark.parametrize("lens", [[1, 1, 1, 1, 1], [3, 0, 1, 0, 1], [1]])
@pytest.mark.parametrize("form", ["delta", "duality"])
def test_single_tokens_follow_the_recurrence(form, heads, G, N, V, s_off, lens):
    from aien_sovereign_core_mv_b200 import kernels as K
    g_, q0, pos, slots = _step(lens, heads + N + V)
    T, S, GN, delta = sum(lens), len(lens), G * N, form == "delta"
    rows = torch.randn(T, 2 * GN + heads * V + (-(2 * GN + heads * V)) % 4, generator=g_)
    rows[:, GN:2 * GN] /= rows[:, GN:2 * GN].reshape(T, G, N).norm(dim=-1).repeat_interleave(N, dim=1)
    gb = torch.rand(T, 2 * heads, generator=g_) * 0.9 + 0.1
    dtr, A, bias, D = torch.randn(T, heads, generator=g_), torch.rand(heads, generator=g_), torch.randn(heads, generator=g_) - 2.0, torch.randn(heads, generator=g_)
    width = s_off + heads * N * V
    state = torch.randn(S, width + (-width) % 4, generator=g_)
    dev, out = state.clone().cuda(), torch.full((T, heads * V), 9.0).cuda()
    common = (dev, s_off, I32(slots), I32(q0), I32(pos), out, S, heads)
    if delta:
        K.delta_rule(rows.cuda(), 0, GN, 2 * GN, gb.cuda(), *common, G, N, V)
    else:
        K.ssd_scan(rows.cuda(), 2 * GN, GN, 0, dtr.cuda(), A.cuda(), bias.cuda(), D.cuda(), *common, V, G, N)
    a = rows.double().numpy()
    dt = np.logaddexp(0.0, (dtr + bias).double().numpy())
    g, w = (gb[:, :heads].double().numpy(), gb[:, heads:].double().numpy()) if delta else (np.exp(-A.double().numpy() * dt), dt)
    left = state.clone()
    for s in range(S):
        r = slice(q0[s], q0[s + 1])
        qk = lambda off: np.repeat(a[r, off:off + GN].reshape(-1, G, N), heads // G, axis=1)
        S0 = state[slots[s], s_off:width].double().numpy().reshape((heads, N, V) if delta else (heads, V, N))
        S0 = (S0 if delta else S0.transpose(0, 2, 1)) * (0.0 if s % 2 else 1.0)
        if lens[s] == 0:
            continue                                            # its slot stays as it was
        want, last = _walk(qk(0), qk(GN), a[r, 2 * GN:2 * GN + heads * V].reshape(-1, heads, V), g[r], w[r], S0, delta, np.zeros(heads) if delta else D.double().numpy())
        # float32 sums of up to 132 products: 132 * 2^-24 of the largest
        H.assert_close(out[r].cpu().numpy().reshape(want.shape), want, 1e-5, f"request {s}")
        left[slots[s], s_off:width] = torch.tensor((last if delta else last.transpose(0, 2, 1)).reshape(-1), dtype=torch.float32)
    H.assert_close(dev.cpu().numpy(), left.numpy(), 1e-5, "states")


@pytest.mark.parametrize("form", ["delta", "duality"])
def test_single_tokens_beside_portions_keep_off_them(form):
    """The token kernels serve the requests of one token and leave the portions to the walk (128 x 128 and 128 x 64 states)."""
    from aien_sovereign_core_mv_b200 import kernels as K
    lens, heads, G, N = [1, 40, 1, 33, 1], 4, 1, 128
    V, delta = (128, True) if form == "delta" else (64, False)
    g_, q0, pos, slots = _step(lens, 5)
    T, S, GN = sum(lens), len(lens), G * N
    rows = torch.randn(T, 2 * GN + heads * V, generator=g_)
    rows[:, GN:2 * GN] /= rows[:, GN:2 * GN].norm(dim=-1, keepdim=True)
    gb = torch.rand(T, 2 * heads, generator=g_) * 0.9 + 0.1
    dtr, A, bias, D = torch.randn(T, heads, generator=g_), torch.rand(heads, generator=g_), torch.randn(heads, generator=g_) - 2.0, torch.randn(heads, generator=g_)
    state = torch.randn(S, heads * N * V, generator=g_)
    got = []
    for alone in (0, 3):
        dev, out = state.clone().cuda(), torch.full((T, heads * V), 9.0).cuda()
        scratch = torch.full((K.block_walk_scratch(T, S, heads, G, N, V),), float("nan")).cuda()
        common = (dev, 0, I32(slots), I32(q0), I32(pos), out, S, heads)
        if delta:
            K.delta_rule(rows.cuda(), 0, GN, 2 * GN, gb.cuda(), *common, G, N, V, scratch, alone)
        else:
            K.ssd_scan(rows.cuda(), 2 * GN, GN, 0, dtr.cuda(), A.cuda(), bias.cuda(), D.cuda(), *common, V, G, N, blocks=scratch, alone=alone)
        got.append((out.cpu().numpy(), dev.cpu().numpy()))
    for name, a, b in (("results", got[0][0], got[1][0]), ("states", got[0][1], got[1][1])):
        H.assert_close(b, a, 1e-5, name)


@pytest.mark.parametrize("H_,dim,vd", [(4, 128, 128), (3, 64, 64), (2, 100, 128), (5, 4, 64), (2, 128, 36), (2, 132, 64)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_decay_linear_attention_of_single_tokens(H_, dim, vd, dtype):
    from aien_sovereign_core_mv_b200 import kernels as K
    lens = [1] * 5
    g_, q0, pos, slots = _step(lens, dim + vd)
    proj = torch.randn(5, 2 * H_ * dim + H_ * vd, generator=g_).to(dtype)
    decay, state = torch.rand(H_, generator=g_), torch.randn(5, H_, dim, vd, generator=g_)
    dev, out = state.clone().cuda(), torch.full((5, H_ * vd), 9.0).cuda()
    K.decay_linear_attention(proj.cuda(), 0, H_ * dim, 2 * H_ * dim, decay.cuda(), dev, I32(slots), I32(q0), I32(pos), out, 5, H_, dim, vd, single_tokens=True)
    a = proj.double().numpy()
    a = a / (1.0 + np.exp(-a))
    for s in range(5):
        cut = lambda lo, n: a[s:s + 1, lo:lo + H_ * n].reshape(1, H_, n)
        S0 = state[slots[s]].double().numpy() * (0.0 if s % 2 else 1.0)
        want, last = _walk(cut(0, dim), cut(H_ * dim, dim), cut(2 * H_ * dim, vd), decay.double().numpy()[None], np.ones((1, H_)), S0, False, np.zeros(H_))
        H.assert_close(out[s].cpu().numpy().reshape(want.shape), want, 1e-5, f"request {s}")
        H.assert_close(dev[slots[s]].cpu().numpy(), last, 1e-5, f"state {s}")


@pytest.mark.parametrize("inner,N,s_off,b_off", [(130, 16, 4, 0), (64, 32, 0, 4), (7, 64, 8, 0), (130, 16, 5, 0), (130, 16, 4, 1), (40, 12, 4, 0), (33, 128, 0, 0)])
@pytest.mark.parametrize("lens", [[1, 1, 1], [2, 0, 1]])
def test_selective_scan_of_single_tokens(inner, N, s_off, b_off, lens):
    from aien_sovereign_core_mv_b200 import kernels as K
    g_, q0, pos, slots = _step(lens, inner + N)
    r = lambda *n: torch.randn(*n, generator=g_)
    x, dtz, z, bc = r(3, inner), r(3, inner) - 1.0, r(3, inner), r(3, 2 * N + 8)
    A, bias, D = -torch.rand(inner, N, generator=g_) * 3.0, r(inner) - 2.0, r(inner)
    state = r(3, s_off + inner * N + (-(s_off + inner * N)) % 4)
    dev, out = state.clone().cuda(), torch.full((3, inner), 9.0).cuda()
    K.selective_scan(x.cuda(), dtz.cuda(), bc.cuda(), b_off, b_off + N, z.cuda(), A.cuda(), bias.cuda(), D.cuda(), dev, s_off, I32(slots), I32(q0), I32(pos), out, 3, N)
    f = lambda t: t.double().numpy()
    dt = np.logaddexp(0.0, f(dtz + bias))
    for s, n in enumerate(lens):
        S = f(state[slots[s], s_off:s_off + inner * N]).reshape(inner, N) * (0.0 if s % 2 else 1.0)
        for t in range(q0[s], q0[s] + n):
            S = np.exp(dt[t][:, None] * f(A)) * S + (dt[t] * f(x[t]))[:, None] * f(bc[t, b_off:b_off + N])
            y = (S @ f(bc[t, b_off + N:b_off + 2 * N]) + f(D) * f(x[t])) * f(z[t]) / (1.0 + np.exp(-f(z[t])))
            H.assert_close(out[t].cpu().numpy(), y, 1e-5, f"token {t}")
        if n:
            H.assert_close(dev[slots[s], s_off:s_off + inner * N].cpu().numpy().reshape(inner, N), S, 1e-5, f"state {s}")


@pytest.mark.parametrize("form", ["delta", "linear"])
@pytest.mark.parametrize("S,heads,dim", [(9, 8, 128), (33, 32, 64), (64, 16, 128)])
def test_single_tokens_are_as_near_to_64_bits_in_whole_vectors_as_number_by_number(form, S, heads, dim):
    """The same tokens over states on 16-byte boundaries and four bytes beside them, which the general kernels take: a relative 2-norm of
    results and states no larger but for the luck of the draw: the norm of n independent errors scatters by 1 / sqrt(2 n), the ratio of two by
    1 / sqrt(n), and three times that is allowed (3 % of 9,216 results, 0.8 % of 131,072)."""
    from aien_sovereign_core_mv_b200 import kernels as K
    g = torch.Generator(device="cuda").manual_seed(S + dim)
    R = lambda *s: torch.randn(*s, generator=g, device="cuda")
    n = heads * dim * dim
    init, order = R(S, heads, dim, dim), [I32(list(range(S))), I32(list(range(S + 1))), I32([5] * S)]
    rows, gates = R(S, 3 * heads * dim), torch.rand(S, 2 * heads, generator=g, device="cuda")
    decay = 1.0 - 2.0 ** (-5 - 3 * torch.arange(heads, device="cuda") / (heads - 1))
    if form == "delta":
        rows[:, :2 * heads * dim] = torch.nn.functional.normalize(rows[:, :2 * heads * dim].reshape(S, 2 * heads, dim), dim=-1).view(S, -1)
        gates[:, :heads] = 1.0 - 0.3 * gates[:, :heads]
        q, k, v = (rows.double().view(S, 3, heads, dim)[:, i] for i in range(3))
        ga, beta = gates.double()[:, :heads, None], gates.double()[:, heads:, None]
        u = beta * (v - ga * torch.einsum("shnv,shn->shv", init.double(), k))
        last = ga[..., None] * init.double() + k[..., None] * u[:, :, None]
    else:
        q, k, v = (torch.nn.functional.silu(rows.double()).view(S, 3, heads, dim)[:, i] for i in range(3))
        last = decay.double()[:, None, None] * init.double() + k[..., None] * v[:, :, None]
    want = torch.einsum("shnv,shn->shv", last, q).reshape(S, -1)
    off = []
    for beside in (0, 1):
        out = torch.full((S, heads * dim), 9.0, device="cuda")
        if form == "delta":
            state = torch.zeros(S, n + 4, device="cuda")
            state[:, beside:beside + n] = init.view(S, n)
            K.delta_rule(rows, 0, heads * dim, 2 * heads * dim, gates, state, beside, *order, out, S, heads, heads, dim, dim)
            got = state[:, beside:beside + n]
        else:
            state = torch.zeros(S * n + 4, device="cuda")[beside:beside + S * n].view(S, heads, dim, dim)
            state.copy_(init)
            K.decay_linear_attention(rows, 0, heads * dim, 2 * heads * dim, decay, state, *order, out, S, heads, dim, dim, single_tokens=True)
            got = state.reshape(S, n)
        off.append([float((a.double() - b).norm() / b.norm()) for a, b in ((out, want), (got, last.reshape(S, n)))])
    for now, before, n_ in ((off[0][0], off[1][0], want.numel()), (off[0][1], off[1][1], last.numel())):
        assert now <= (1.0 + 3.0 * n_ ** -0.5) * before, off
