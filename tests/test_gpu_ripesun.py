"""The Ripesun design in the engine against its plain implementation (``plain_ripesun``): each mechanism alone, then
whole models under every way of cutting the work, in float32 and bfloat16.

The configurations are small and differ from one another in every size and constant: head counts that fill no warp or
block of heads evenly, latent sizes that are no multiple of 32, windows of less than a page, of several pages and none,
two layers that share one cache under different windows, decays of 0 and 1, a layer without a feed-forward, models
with and without the token side input, the soft cap, the embedding scale and the residual multiplier.  Where random
weights would hide a fault the inputs are made so that it shows: keys just inside and just outside a window are scaled
until their scores stand out, a sink is made large, a far key is made the only one that matters.
"""
import copy
import json
import math
import os

import numpy as np
import pytest
import torch

import helpers as H
import plain_ripesun as pr

pytestmark = pytest.mark.gpu


def _latent(heads, dim, rot_dim, vdim, kv_rank, q_rank, window, scale, base=10000.0, kv_from=None):
    m = {"heads": heads, "dim": dim, "rot_dim": rot_dim, "vdim": vdim, "kv_rank": kv_rank, "q_rank": q_rank, "scale": scale,
         "rot": {"base": base, "dims": rot_dim}, "mask": {"size": window} if window else None}
    if kv_from is not None:
        m["kv_from"] = kv_from
    return m


def _light(heads, dim, vdim, decay):
    return {"heads": heads, "dim": dim, "vdim": vdim, "decay": decay}


def _dense(ff):
    return {"kind": "dense", "ff": ff}


CONFIGS = {
    # five heads, latent of 40, windows of 21 and 9 on one shared cache, decays 0.5 / 0.9 / 1, a layer without feed-forward
    "A": {"architecture": "Ripesun", "vocab": 333, "width": 96, "norm": {"eps": 1e-5}, "embedding": {"scale": 3.0},
          "residual_mult": 0.7, "logit_softcap": 20.0, "token_side": {"dim": 8}, "layers": [
              {"type": "lightning", "mixer": _light(3, 20, 12, [0.5, 0.9, 1.0]), "mlp": _dense(80)},
              {"type": "latent_attention", "mixer": _latent(5, 24, 8, 16, 40, 48, 21, 0.2), "mlp": _dense(64)},
              {"type": "mingru", "mixer": {"width": 72}, "mlp": None},
              {"type": "latent_attention", "mixer": _latent(5, 12, 8, 20, 40, 24, 9, 0.3, kv_from=1), "mlp": _dense(48)},
              {"type": "lightning", "mixer": _light(2, 16, 40, [0.0, 0.97]), "mlp": _dense(40)}]},
    # no side input, no cap, no scale, multiplier 1; one head, a latent of 96, no mask at all (every key stays), a reader of it
    "B": {"architecture": "Ripesun", "vocab": 257, "width": 64, "norm": {"eps": 3e-6}, "layers": [
        {"type": "mingru", "mixer": {"width": 100}, "mlp": _dense(96)},
        {"type": "latent_attention", "mixer": _latent(1, 16, 16, 16, 96, 16, 0, 0.25, 1e6), "mlp": None},
        {"type": "latent_attention", "mixer": _latent(3, 8, 16, 8, 96, 40, 0, 0.35, 1e6, kv_from=1), "mlp": _dense(72)}]},
    # sizes the tensor-core products take; 17 heads (two blocks of heads), a window of four pages, a window of one page
    "C": {"architecture": "Ripesun", "vocab": 512, "width": 128, "norm": {"eps": 1e-6}, "embedding": {"scale": 8.0},
          "residual_mult": 0.5, "logit_softcap": 30.0, "token_side": {"dim": 16}, "layers": [
              {"type": "latent_attention", "mixer": _latent(17, 64, 32, 64, 128, 64, 64, 0.1, 50000.0), "mlp": _dense(256)},
              {"type": "lightning", "mixer": _light(4, 64, 64, [0.8, 0.95, 0.99, 0.999]), "mlp": _dense(256)},
              {"type": "mingru", "mixer": {"width": 256}, "mlp": _dense(128)},
              {"type": "latent_attention", "mixer": _latent(4, 32, 64, 32, 64, 128, 16, 0.12, 777.0), "mlp": _dense(128)}]},
    # no attention at all (no paged cache group), sizes no vector or tensor-core kernel takes: width 90, heads of 10 / 6, 50 channels
    "D": {"architecture": "Ripesun", "vocab": 101, "width": 90, "norm": {"eps": 1e-5}, "residual_mult": 0.9, "token_side": {"dim": 9}, "layers": [
        {"type": "mingru", "mixer": {"width": 50}, "mlp": _dense(30)},
        {"type": "lightning", "mixer": _light(3, 10, 6, [0.25, 0.75, 0.995]), "mlp": None},
        {"type": "mingru", "mixer": {"width": 34}, "mlp": _dense(22)}]},
    # attention only (no state group), odd sizes: 3 heads of 10 + 6 rotated, latent of 18, windows of 5 and 33 on caches of their own
    "E": {"architecture": "Ripesun", "vocab": 130, "width": 70, "norm": {"eps": 1e-6}, "embedding": {"scale": 0.5}, "logit_softcap": 5.0, "layers": [
        {"type": "latent_attention", "mixer": _latent(3, 10, 6, 14, 18, 14, 5, 0.4, 77.0), "mlp": _dense(50)},
        {"type": "latent_attention", "mixer": _latent(2, 6, 2, 6, 18, 22, 33, 0.5, 1e5), "mlp": None}]},
}
PAGE = {"A": 16, "B": 8, "C": 16, "D": 16, "E": 8}
LENGTHS = {"A": [1, 9, 50, 131], "B": [2, 20, 77], "C": [5, 70, 150], "D": [3, 40, 90], "E": [2, 41, 95]}
FP32_TOL, BF16_TOL = 1e-4, 4e-2
DTYPES = [("float32", FP32_TOL), ("bfloat16", BF16_TOL)]


def load_plain(folder):
    from aien_sovereign_core_mv_b200.weights.safetensors_io import CheckpointFiles
    with open(os.path.join(folder, "config.json")) as f:
        cfg = json.load(f)
    files = CheckpointFiles(folder)
    tensors = {n: files.tensor(n).float().numpy().astype(np.float64) for n in files.names()}
    files.close()
    return cfg, tensors


def tokens(which, n, seed):
    return [int(t) for t in np.random.default_rng(seed).integers(0, CONFIGS[which]["vocab"], n)]


@pytest.fixture(scope="module")
def models(tmp_path_factory):
    from aien_sovereign_core_mv_b200 import write_random_model
    root = tmp_path_factory.mktemp("ripesun")
    out = {}
    for i, which in enumerate(CONFIGS):
        d = write_random_model(os.path.join(str(root), which), CONFIGS[which], 70 + i)
        cfg, tensors = load_plain(d)
        reqs = {j + 1: tokens(which, n, 100 * i + n) for j, n in enumerate(LENGTHS[which])}
        want = {rid: pr.forward(cfg, tensors, toks) for rid, toks in reqs.items()}
        out[which] = (d, reqs, want)
    return out


def check(collected, want, tol, what):
    assert collected, f"{what}: nothing was collected"
    for rid, rows in collected.items():
        pos = sorted(rows)
        got, ref = np.stack([rows[p] for p in pos]), want[rid][pos]
        H.assert_close(got, ref, tol, f"{what} request {rid} (positions {pos[0]}..{pos[-1]})")


def make_ctx(dtype, positions, seq_of_token, q_start, ctx_len, groups=()):
    from test_gpu_parts import make_ctx as mk
    return mk(dtype, positions, seq_of_token, q_start, ctx_len, groups)


def i32(a):
    return torch.tensor(a, dtype=torch.int32, device="cuda")


# ------------------------------------------------------------------ mechanisms alone
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width,parts", [(72, 1), (2304, 3), (90, 2)])
def test_scaled_sum_of_a_normed_branch_and_the_next_norm(dtype, width, parts):
    from aien_sovereign_core_mv_b200 import kernels as K
    g = torch.Generator().manual_seed(width)
    T, eps, eps2, mult = 5, 1e-5, 3e-6, 0.37
    w = (torch.rand(width, generator=g) * 0.4 + 0.8).to(torch.bfloat16).cuda()
    w2 = (torch.rand(width, generator=g) * 0.4 + 0.8).to(torch.bfloat16).cuda()
    x0 = torch.randn(T, width, generator=g).cuda()
    a = torch.randn(parts, T, width, generator=g).cuda() if parts > 1 else torch.randn(T, width, generator=g).to(dtype).cuda()
    y = a.double().sum(0).cpu().numpy() if parts > 1 else a.double().cpu().numpy()
    want_x = x0.double().cpu().numpy() + mult * pr.rms_norm(y, w.double().cpu().numpy(), eps)
    tol_h = 2e-6 if dtype == torch.float32 else 8e-3
    # the sum and the next norm
    x, h = x0.clone(), torch.empty(T, width, dtype=dtype).cuda()
    K.post_norm_add(x, a, w, eps, mult, w2, eps2, h)
    H.assert_close(x.cpu().numpy(), want_x, 2e-6, "stream")
    H.assert_close(h.float().cpu().numpy(), pr.rms_norm(want_x, w2.double().cpu().numpy(), eps2), tol_h, "next norm")
    # the sum and the plain copy; the sum alone
    x, h = x0.clone(), torch.empty(T, width, dtype=dtype).cuda()
    K.post_norm_add(x, a, w, eps, mult, None, 0.0, h)
    H.assert_close(h.float().cpu().numpy(), want_x, tol_h, "copy")
    x = x0.clone()
    K.post_norm_add(x, a, w, eps, mult)
    H.assert_close(x.cpu().numpy(), want_x, 2e-6, "stream alone")


def test_scaled_embedding_side_gate_and_soft_cap():
    from aien_sovereign_core_mv_b200 import kernels as K
    g = torch.Generator().manual_seed(1)
    table = torch.randn(50, 36, generator=g).to(torch.bfloat16).cuda()
    ids = i32([3, 49, 0, 17])
    x = torch.empty(4, 36, dtype=torch.float32).cuda()
    K.embed_gather_scaled(table, ids, x, 2.5)
    H.assert_close(x.cpu().numpy(), table.float().cpu().numpy()[[3, 49, 0, 17]] * 2.5, 1e-7, "scaled rows")
    z = torch.randn(4, 5, generator=g).cuda() * 2
    out = torch.empty(4, 5, dtype=torch.float32).cuda()
    K.gelu_times_table(z, table, 30, ids, out)
    want = pr.gelu_tanh(z.double().cpu().numpy()) * table.double().cpu().numpy()[[3, 49, 0, 17]][:, 30:35]
    H.assert_close(out.cpu().numpy(), want, 2e-6, "gelu(z) * columns of the token's row")
    v = (torch.randn(3, 11, generator=g) * 40).cuda()
    want = 15.0 * np.tanh(v.double().cpu().numpy() / 15.0)
    K.softcap(v, 15.0)
    H.assert_close(v.cpu().numpy(), want, 2e-6, "soft cap")


def _state_group(shape, slots):
    from aien_sovereign_core_mv_b200.parts import GroupView
    st = torch.full((2, slots + 1) + tuple(shape), 7.5, dtype=torch.float32).cuda()      # what a slot held before must not matter
    return st, lambda slot_list: GroupView("state", 16, 0, 0, None, i32(slot_list), {"state": st})


@pytest.mark.parametrize("chunked", [False, True])
@pytest.mark.parametrize("heads,dim,vdim,decay", [(3, 20, 12, [0.5, 0.9, 1.0]), (2, 64, 70, [0.0, 0.999]), (1, 130, 8, [0.97])])
def test_decayed_linear_attention_in_one_step_and_in_pieces(heads, dim, vdim, decay, chunked):
    """Two requests of unequal length in one step against the token-by-token recurrence; then the same tokens in pieces
    (65, 1, 1, 2, the rest: across the kernels' chunks of 32 and 64) through a slot that another request used before.
    ``chunked``: the form whose chunks run side by side (portions of prompts), else the one that walks them in order."""
    from aien_sovereign_core_mv_b200 import kernels as K
    g = torch.Generator().manual_seed(dim)
    D, eps = 48, 1e-5
    lens = [150, 5]
    T = sum(lens)
    scratch = lambda n, S: torch.full((K.decay_linear_attention_scratch(n, S, heads, dim, vdim),), float("nan")).cuda() if chunked else None
    p = {n: (torch.randn(r, D, generator=g) / math.sqrt(D)).double().numpy() for n, r in
         (("q", heads * dim), ("k", heads * dim), ("v", heads * vdim), ("g", heads * vdim))}
    h = torch.randn(T, D, generator=g).double().numpy()
    proj = torch.tensor(np.concatenate([h @ p["q"].T, h @ p["k"].T, h @ p["v"].T, h @ p["g"].T], axis=1), dtype=torch.float32).cuda()
    dec = torch.tensor(decay, dtype=torch.float32).cuda()
    st, _ = _state_group((heads, dim, vdim), 3)

    def plain(rows, state=None):
        T_ = rows.shape[0]
        q, k, v = (pr.silu(rows @ p[n].T) for n in ("q", "k", "v"))
        q, k, v = q.reshape(T_, heads, dim), k.reshape(T_, heads, dim), v.reshape(T_, heads, vdim)
        S = np.zeros((heads, dim, vdim)) if state is None else state.copy()
        o = np.zeros((T_, heads, vdim))
        for t in range(T_):
            for hd in range(heads):
                S[hd] = decay[hd] * S[hd] + np.outer(k[t, hd], v[t, hd])
                o[t, hd] = S[hd].T @ q[t, hd]
        return o.reshape(T_, heads * vdim), S

    want0, S0 = plain(h[:lens[0]])
    want1, S1 = plain(h[lens[0]:])
    out = torch.zeros(T, heads * vdim, dtype=torch.float32).cuda()
    K.decay_linear_attention(proj, 0, heads * dim, 2 * heads * dim, dec, st[1], i32([2, 0]), i32([0, lens[0], T]),
                             i32(list(range(lens[0])) + list(range(lens[1]))), out, 2, heads, dim, vdim, scratch(T, 2))
    H.assert_close(out.cpu().numpy(), np.concatenate([want0, want1]), 2e-5, "two requests in one step")
    H.assert_close(st[1, 2].cpu().numpy(), S0, 2e-5, "state of the first")
    H.assert_close(st[1, 0].cpu().numpy(), S1, 2e-5, "state of the second")
    assert float((st[0] - 7.5).abs().max()) == 0.0 and float((st[1, 1] - 7.5).abs().max()) == 0.0     # other runs and slots untouched
    # the first request again, in pieces, through slot 0 (which holds the second request's state): position 0 starts from zero
    at, got = 0, []
    for n in [65, 1, 1, 2, lens[0] - 69]:
        o = torch.zeros(n, heads * vdim, dtype=torch.float32).cuda()
        K.decay_linear_attention(proj[at:at + n], 0, heads * dim, 2 * heads * dim, dec, st[1], i32([0]), i32([0, n]),
                                 i32(list(range(at, at + n))), o, 1, heads, dim, vdim, scratch(n, 1))
        got.append(o.cpu().numpy())
        at += n
    H.assert_close(np.concatenate(got), want0, 2e-5, "the same tokens in pieces")
    H.assert_close(st[1, 0].cpu().numpy(), S0, 2e-5, "state after the pieces")
    # both requests once more, token by token in steps of two single tokens (the kernel made for such steps), slots swapped
    got0, got1 = [], []
    for i in range(lens[1]):
        rows = torch.cat([proj[i:i + 1], proj[lens[0] + i:lens[0] + i + 1]]).contiguous()
        o = torch.zeros(2, heads * vdim, dtype=torch.float32).cuda()
        K.decay_linear_attention(rows, 0, heads * dim, 2 * heads * dim, dec, st[1], i32([1, 2]), i32([0, 1, 2]), i32([i, i]), o, 2,
                                 heads, dim, vdim, single_tokens=True)
        got0.append(o[0].cpu().numpy()); got1.append(o[1].cpu().numpy())
    H.assert_close(np.stack(got0), want0[:lens[1]], 2e-5, "single tokens, first request")
    H.assert_close(np.stack(got1), want1, 2e-5, "single tokens, second request")
    H.assert_close(st[1, 2].cpu().numpy(), S1, 2e-5, "state after single tokens")


@pytest.mark.parametrize("segments", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [72, 300])
def test_gated_recurrence_in_one_step_and_in_pieces(dtype, width, segments):
    from aien_sovereign_core_mv_b200 import kernels as K
    g = torch.Generator().manual_seed(width)
    lens = [141, 6]
    T = sum(lens)
    proj = (torch.randn(T, 3 * width, generator=g) * 2).cuda()
    bz, bx = torch.randn(width, generator=g).cuda(), torch.randn(width, generator=g).cuda()
    st, _ = _state_group((width,), 2)
    pz, px, pg = (proj[:, i * width:(i + 1) * width].double().cpu().numpy() for i in range(3))

    def plain(lo, hi, S=None):
        z = pr.sigmoid(pz[lo:hi] + bz.double().cpu().numpy())
        u = px[lo:hi] + bx.double().cpu().numpy()
        cand = np.where(u >= 0, u + 0.5, pr.sigmoid(u))
        S = np.zeros(width) if S is None else S.copy()
        o = np.zeros((hi - lo, width))
        for t in range(hi - lo):
            S = (1 - z[t]) * S + z[t] * cand[t]
            o[t] = S
        return o * pr.silu(pg[lo:hi]), S

    want0, S0 = plain(0, lens[0])
    want1, S1 = plain(lens[0], T)
    tol = 2e-5 if dtype == torch.float32 else 8e-3
    out = torch.zeros(T, width, dtype=dtype).cuda()
    K.gated_recurrence(proj, 0, width, 2 * width, bz, bx, st[0], i32([1, 0]), i32([0, lens[0], T]),
                       i32(list(range(lens[0])) + list(range(lens[1]))), out, 2, width, segments)
    H.assert_close(out.float().cpu().numpy(), np.concatenate([want0, want1]), tol, "two requests in one step")
    H.assert_close(st[0, 1].cpu().numpy(), S0, 2e-5, "state of the first")
    at, got = 0, []
    for n in [3, 1, 2, 5, 33, lens[0] - 44]:
        o = torch.zeros(n, width, dtype=dtype).cuda()
        K.gated_recurrence(proj[at:at + n], 0, width, 2 * width, bz, bx, st[0], i32([0]), i32([0, n]), i32(list(range(at, at + n))), o, 1, width, segments)
        got.append(o.float().cpu().numpy())
        at += n
    H.assert_close(np.concatenate(got), want0, tol, "the same tokens in pieces, through a slot used before")
    H.assert_close(st[0, 0].cpu().numpy(), S0, 2e-5, "state after the pieces")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("q_rank,kv_rank,rot_dim", [(48, 40, 8), (16, 96, 16), (130, 64, 0)])
def test_latents_norms_rotation_and_cache_rows(dtype, q_rank, kv_rank, rot_dim):
    from aien_sovereign_core_mv_b200 import kernels as K
    g = torch.Generator().manual_seed(q_rank)
    T, eps, base = 6, 1e-5, 777.0
    pos = [0, 1, 17, 64, 1000, 70001]
    d = torch.randn(T, q_rank + kv_rank + rot_dim, generator=g).cuda()
    wq = (torch.rand(q_rank, generator=g) * 0.4 + 0.8).to(torch.bfloat16).cuda()
    wkv = (torch.rand(kv_rank, generator=g) * 0.4 + 0.8).to(torch.bfloat16).cuda()
    cos = sin = None
    if rot_dim:
        ang = np.asarray(pos, dtype=np.float64)[:, None] * np.array([base ** (-2.0 * i / rot_dim) for i in range(rot_dim // 2)])[None]
        cos, sin = torch.tensor(np.cos(ang), dtype=torch.float32).cuda(), torch.tensor(np.sin(ang), dtype=torch.float32).cuda()
    slots = i32([3, 9, 0, -1, 5, 8])
    cache = torch.zeros(12, kv_rank + rot_dim, dtype=dtype).cuda()
    cq = torch.empty(T, q_rank, dtype=dtype).cuda()
    K.latent_prepare(d, q_rank, wq, eps, cq, q_rank, kv_rank, rot_dim, rot_dim, wkv, cos, sin, slots, cache)
    dn = d.double().cpu().numpy()
    tol = 3e-6 if dtype == torch.float32 else 8e-3
    H.assert_close(cq.float().cpu().numpy(), pr.rms_norm(dn[:, :q_rank], wq.double().cpu().numpy(), eps), tol, "query latent")
    c = pr.rms_norm(dn[:, q_rank:q_rank + kv_rank], wkv.double().cpu().numpy(), eps)
    kr = pr.rotate_pairs(dn[:, q_rank + kv_rank:], pos, base, rot_dim) if rot_dim else dn[:, q_rank + kv_rank:]
    for t, s in enumerate(slots.tolist()):
        if s >= 0:
            H.assert_close(cache[s].float().cpu().numpy(), np.concatenate([c[t], kr[t]]), tol, f"cache row of token {t}")
    used = [s for s in slots.tolist() if s >= 0]
    assert all(float(cache[s].abs().max()) == 0.0 for s in range(12) if s not in used)     # a token without a slot writes nothing
    if rot_dim:                                                       # the query's rotated part, moved behind its latent
        heads, dim = 3, 10
        q = torch.randn(T, heads * (dim + rot_dim), generator=g).cuda()
        qf = torch.zeros(T, heads * (kv_rank + rot_dim), dtype=torch.float32).cuda()
        K.rotate_pairs_rows(q, dim + rot_dim, dim, qf, kv_rank + rot_dim, kv_rank, heads, rot_dim, rot_dim, cos, sin)
        qh = q.double().cpu().numpy().reshape(T, heads, dim + rot_dim)
        H.assert_close(qf.cpu().numpy().reshape(T, heads, -1)[:, :, kv_rank:], pr.rotate_pairs(qh[:, :, dim:], pos, base, rot_dim), 3e-6, "rotated query part")
        assert float(qf.reshape(T, heads, -1)[:, :, :kv_rank].abs().max()) == 0.0


@pytest.mark.parametrize("dtype,wdt", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("q_rank,kv_rank,rot_dim,rot_dims,lead", [(2048, 1024, 64, 64, 0), (2052, 64, 4, 4, 0), (1028, 1028, 0, 0, 0), (0, 512, 300, 8, 4), (4, 4, 4, 2, 0), (1536, 512, 6, 6, 0),
                                                                  (64, 64, 8, 8, 2), (1024, 0, 0, 0, 0)])
def test_latents_in_whole_vectors(dtype, wdt, q_rank, kv_rank, rot_dim, rot_dims, lead):
    """Ranks at and beyond what the vector form's threads hold, rotated parts longer than its idle threads and no multiples of
    four, rows that start off the 16-byte boundary (``lead``), no query latent, no cache; the forms agree with 64 bits."""
    from aien_sovereign_core_mv_b200 import kernels as K
    g = torch.Generator().manual_seed(q_rank + kv_rank)
    T, eps, pos = 5, 1e-5, [0, 3, 64, 1000, 70001]
    width = q_rank + kv_rank + rot_dim
    d = torch.randn(T, lead + width + (-(lead + width)) % 4, generator=g).cuda()[:, lead:lead + width]
    weight = lambda n: (torch.rand(n, generator=g) * 0.4 + 0.8).to(wdt).cuda() if n else None
    wq, wkv = weight(q_rank), weight(kv_rank)
    ang = np.asarray(pos, dtype=np.float64)[:, None] * np.array([777.0 ** (-2.0 * i / max(rot_dims, 1)) for i in range(rot_dims // 2)])[None]
    cos, sin = (torch.tensor(f(ang), dtype=torch.float32).cuda() if rot_dims else None for f in (np.cos, np.sin))
    slots = i32([3, -1, 0, 6, 5])
    cache = torch.full((7, kv_rank + rot_dim), 9.0, dtype=dtype).cuda() if kv_rank else None
    cq = torch.empty(T, q_rank, dtype=dtype).cuda() if q_rank else None
    K.latent_prepare(d, q_rank, wq, eps, cq, q_rank, kv_rank, rot_dim, rot_dims, wkv, cos, sin, slots if kv_rank else None, cache)
    dn, tol = d.double().cpu().numpy(), 3e-6 if dtype == torch.float32 else 8e-3
    if q_rank:
        H.assert_close(cq.float().cpu().numpy(), pr.rms_norm(dn[:, :q_rank], wq.double().cpu().numpy(), eps), tol, "query latent")
    if kv_rank:
        c, kr = pr.rms_norm(dn[:, q_rank:q_rank + kv_rank], wkv.double().cpu().numpy(), eps), dn[:, q_rank + kv_rank:].copy()
        if rot_dims:
            kr[:, :rot_dims] = pr.rotate_pairs(kr[:, :rot_dims], pos, 777.0, rot_dims)
        for t, s in enumerate(slots.tolist()):
            if s >= 0:
                H.assert_close(cache[s].float().cpu().numpy(), np.concatenate([c[t], kr[t]]), tol, f"cache row of token {t}")
        assert all((cache[s] == 9.0).all() for s in range(7) if s not in slots.tolist())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,n,k", [(5, 40, 24), (17, 128, 64), (1, 7, 3)])
def test_one_product_per_head(dtype, heads, n, k):
    from aien_sovereign_core_mv_b200 import kernels as K
    g = torch.Generator().manual_seed(n)
    T = 9
    a = torch.randn(T, heads * (k + 4), generator=g).to(dtype).cuda()                # four numbers of something else behind every head
    w = (torch.randn(heads, n, k, generator=g) / math.sqrt(k)).to(dtype).cuda()
    out = torch.zeros(T, heads * (n + 2) + 1, dtype=torch.float32).cuda()
    K.head_project(a, k + 4, 0, w, out, n + 2, 1)
    ah = a.double().cpu().numpy().reshape(T, heads, k + 4)[:, :, :k]
    want = np.einsum("thk,hnk->thn", ah, w.double().cpu().numpy())
    got = out.cpu().numpy()[:, 1:].reshape(T, heads, n + 2)
    H.assert_close(got[:, :, :n], want, 2e-6, "products")
    assert float(np.abs(got[:, :, n:]).max()) == 0.0 and float(out[:, 0].abs().max()) == 0.0


@pytest.mark.parametrize("dtype,impl", [(torch.float32, "plain"), (torch.bfloat16, "plain"), (torch.bfloat16, "tc"), (torch.bfloat16, "tc_split"),
                                        (torch.bfloat16, "tc_small")])
@pytest.mark.parametrize("window,page,heads,r,rd", [(21, 16, 5, 40, 8), (64, 16, 17, 128, 32), (0, 8, 1, 96, 16), (16, 16, 4, 64, 64),
                                                     (7, 32, 3, 520, 0), (100, 16, 6, 256, 16), (0, 16, 16, 512, 64)])
def test_latent_attention_sees_its_window_and_the_sink(dtype, impl, window, page, heads, r, rd):
    """Portions at several places of a request of 150 tokens whose pages lie scattered (each portion as a request of its
    own over the same pages): the first tokens, both sides of a page border, the end.  The keys just inside the window
    (distance window - 1), just outside (distance window) and at position 0 are scaled so that each would take nearly all
    the weight if it were seen; one head's sink is made large.  ``impl``: the plain kernel, or the tensor-core one."""
    from aien_sovereign_core_mv_b200 import kernels as K
    if impl.startswith("tc") and not K.latent_attention_tc_supports(dtype, r, rd):
        pytest.skip("the tensor-core kernel does not take this size")
    g = torch.Generator().manual_seed(window + r)
    n, D, scale = 150, r + rd, 0.2
    rows = torch.randn(n, D, generator=g) * 0.5
    portions = [(0, 3), (page - 2, 4), (2 * page, 1), (60, 70), (149, 1)]
    if impl == "tc_small":                                            # the tiles of 16 rows are for requests that bring one token each
        portions = [(p, 1) for p in (0, 1, page - 1, page, 2 * page, 99, 100, 149)]
    qpos = [p0 + i for p0, m in portions for i in range(m)]
    loud = {p - far for p in qpos for far in ([window - 1, window] if window else [p]) if p - far >= 0}
    for j in sorted(loud):
        rows[j] *= 3.0
    rows = rows.to(dtype)
    order = list(np.random.default_rng(3).permutation((n + page - 1) // page + 3))
    cache = torch.zeros((max(order) + 1) * page, D, dtype=dtype)
    for j in range(n):
        cache[order[j // page] * page + j % page] = rows[j]
    bt = torch.full((len(portions), 64), -1, dtype=torch.int32)
    bt[:, :(n + page - 1) // page] = torch.tensor(order[:(n + page - 1) // page], dtype=torch.int32)
    qdt = torch.bfloat16 if impl.startswith("tc") else torch.float32
    q = (torch.randn(len(qpos), heads * D, generator=g) * 0.7).to(qdt)
    sinks = torch.randn(heads, generator=g)
    sinks[0] = 6.0
    out = torch.zeros(len(qpos), heads * r, dtype=dtype).cuda()
    seq_of = [s for s, (_, m) in enumerate(portions) for _ in range(m)]
    starts = [0]
    for _, m in portions:
        starts.append(starts[-1] + m)
    if impl.startswith("tc"):
        ksplit = {"tc": 1, "tc_split": 3, "tc_small": 2}[impl]
        scratch = torch.full((K.latent_attention_tc_scratch(len(qpos), heads, r, ksplit),), float("nan")).cuda() if ksplit > 1 else None
        K.latent_attention_tc(q.cuda(), cache.cuda(), bt.cuda(), 64, i32(starts), i32(qpos), out, len(portions), heads, r, rd, page, window,
                              scale, sinks.cuda(), ksplit, scratch, small_tiles=(impl == "tc_small"))
    else:
        K.latent_attention(q.cuda(), cache.cuda(), bt.cuda(), 64, i32(seq_of), i32(qpos), out, heads, r, rd, page, window, scale, sinks.cuda())
    rn, qn = rows.double().numpy(), q.double().numpy().reshape(len(qpos), heads, D)
    want = np.zeros((len(qpos), heads, r))
    for t, p in enumerate(qpos):
        seen = [j for j in range(n) if j <= p and (window == 0 or p - j < window)]
        for hd in range(heads):
            sc = np.array([qn[t, hd] @ rn[j] * scale for j in seen])
            m = max(sc.max(), float(sinks[hd]))
            e = np.exp(sc - m)
            want[t, hd] = (e[:, None] * rn[seen][:, :r]).sum(0) / (e.sum() + math.exp(float(sinks[hd]) - m))
    H.assert_close(out.float().cpu().numpy().reshape(len(qpos), heads, r), want, 1e-5 if dtype == torch.float32 else 1.5e-2, "weighted latents")


@pytest.mark.parametrize("heads,r,rd,page,window,ksplit", [(16, 512, 0, 16, 0, 1), (16, 512, 64, 16, 0, 3), (33, 512, 8, 24, 100, 2), (5, 256, 0, 8, 0, 4), (16, 200, 24, 24, 0, 1),
                                                            (16, 128, 72, 32, 40, 1), (17, 104, 0, 16, 0, 9)])
def test_latent_attention_of_single_tokens(heads, r, rd, page, window, ksplit):
    """Contexts from one key to more blocks of 32 than the stages hold, borders of blocks and pages (of 24 tokens too), rows
    wider and narrower than whole vectors, more CTAs a token than it has blocks, the step's tokens and a list of them."""
    from aien_sovereign_core_mv_b200 import kernels as K
    g = torch.Generator().manual_seed(heads + r + page)
    ctx, D, scale = [1, 31, 32, 33, 97, 300, 64, 161], r + rd, 0.1
    pages = [(n + page - 1) // page for n in ctx]
    order = torch.randperm(sum(pages), generator=g)
    cache = torch.zeros(sum(pages) * page, D, dtype=torch.bfloat16)
    bt, rows, at = torch.full((len(ctx), max(pages)), -1, dtype=torch.int32), [], 0
    for s_, n in enumerate(ctx):
        bt[s_, :pages[s_]] = order[at:at + pages[s_]].to(torch.int32)
        at += pages[s_]
        rows.append((torch.randn(n, D, generator=g) * 0.7).to(torch.bfloat16))
        for j in range(n):
            cache[int(bt[s_, j // page]) * page + j % page] = rows[-1][j]
    T = len(ctx)
    q = torch.randn(T, heads * D, generator=g).to(torch.bfloat16)
    sinks = torch.randn(heads, generator=g)
    want = np.zeros((T, heads, r))
    for t, n in enumerate(ctx):
        k = rows[t].double().numpy()[max(0, n - window) if window else 0:]
        z = q[t].double().numpy().reshape(heads, D) @ k.T * scale
        m = np.maximum(z.max(1), sinks.double().numpy())
        e = np.exp(z - m[:, None])
        want[t] = (e @ k[:, :r]) / (e.sum(1) + np.exp(sinks.double().numpy() - m))[:, None]
    scratch = torch.full((K.latent_attention_tc_scratch(T, heads, r, ksplit) + 1,), float("nan")).cuda()
    for tokens in (None, "listed"):
        out = torch.full((T, heads * r), 9.0, dtype=torch.bfloat16).cuda()
        starts = list(range(T + 1))
        K.latent_attention_tc(q.cuda(), cache.cuda(), bt.cuda(), bt.shape[1], i32(starts), i32([n - 1 for n in ctx]), out, T, heads, r, rd, page, window, scale,
                              sinks.cuda(), ksplit, scratch, True, None if tokens is None else i32(list(range(T))), 0 if tokens is None else T)
        H.assert_close(out.float().cpu().numpy().reshape(T, heads, r), want, 1.5e-2, "weighted latents")


# ------------------------------------------------------------------ whole models
@pytest.mark.parametrize("which", list(CONFIGS))
def test_layers_of_a_short_request_float32(models, which):
    """The stream after every layer, so that a fault names its layer."""
    d, reqs, _ = models[which]
    cfg, tensors = load_plain(d)
    toks = reqs[2]
    want = []
    pr.forward(cfg, tensors, toks, want)
    eng = H.engine_for(d, "float32", PAGE[which], 256, replay_steps=False)
    seen = []
    for b in eng.model.blocks:
        def wrapped(ctx, x, delta, run, next_norm=None, _inner=b.forward):
            out = _inner(ctx, x, delta, run, next_norm=next_norm)
            seen.append(x.clone())
            return out
        b.forward = wrapped
    eng.step([(1, toks, [0])])
    assert len(seen) == len(want)
    for i, (a, w) in enumerate(zip(seen, want)):
        H.assert_close(a.cpu().numpy(), w, 2e-5, f"{which}: stream after layer {i} ({cfg['layers'][i]['type']})")


@pytest.mark.parametrize("dtype,tol", DTYPES)
@pytest.mark.parametrize("which", list(CONFIGS))
def test_whole_requests(models, which, dtype, tol):
    d, reqs, want = models[which]
    eng = H.engine_for(d, dtype, PAGE[which], 512)
    steps = [([(rid, toks, list(range(len(toks))))], [rid]) for rid, toks in reqs.items()]
    check(H.run_steps(eng, steps), want, tol, f"{which} {dtype} whole")
    assert eng.cache_state()["check"] == "" and eng.cache_state()["requests"] == 0


@pytest.mark.parametrize("dtype,tol", DTYPES)
@pytest.mark.parametrize("which", list(CONFIGS))
def test_prefill_then_token_by_token(models, which, dtype, tol):
    """Most of the longest request in one step, then 40 tokens one by one: the decoded tokens' windows pass over the
    prompt's end, and pages behind a window are given back while the request runs."""
    d, reqs, want = models[which]
    eng = H.engine_for(d, dtype, PAGE[which], 512)
    rid = max(reqs, key=lambda r: len(reqs[r]))
    toks = reqs[rid]
    cut = len(toks) - 40
    steps = [([(rid, toks[:cut], [0, cut - 1])], [])] + [([(rid, [toks[i]], [0])], []) for i in range(cut, len(toks))]
    check(H.run_steps(eng, steps), want, tol, f"{which} {dtype} decode")
    state = eng.cache_state()
    assert state["check"] == "" and (which in ("B", "D") or state["metrics"]["window_releases"] > 0)     # B keeps every key, D has none


@pytest.mark.parametrize("dtype,tol", DTYPES)
@pytest.mark.parametrize("which", list(CONFIGS))
def test_first_tokens_one_by_one(models, which, dtype, tol):
    d, reqs, want = models[which]
    eng = H.engine_for(d, dtype, PAGE[which], 512)
    rid = max(reqs, key=lambda r: len(reqs[r]))
    steps = [([(rid, [t], [0])], []) for t in reqs[rid][:45]]
    check(H.run_steps(eng, steps), want, tol, f"{which} {dtype} from the first token")


@pytest.mark.parametrize("dtype,tol", DTYPES)
@pytest.mark.parametrize("which", list(CONFIGS))
def test_changing_portions(models, which, dtype, tol):
    d, reqs, want = models[which]
    eng = H.engine_for(d, dtype, PAGE[which], 512)
    sizes = [7, 2, 13, 3, 2, 29, 5, 2, 16, 17, 1, 8, 64, 2, 31]
    for rid, toks in reqs.items():
        steps, at, k = [], 0, rid
        while at < len(toks):
            n = min(sizes[k % len(sizes)], len(toks) - at)
            steps.append(([(rid, toks[at:at + n], list(range(n)))], []))
            at += n
            k += 1
        steps[-1] = (steps[-1][0], [rid])
        check(H.run_steps(eng, steps), want, tol, f"{which} {dtype} portions of request {rid}")
    assert eng.cache_state()["check"] == "" and eng.cache_state()["requests"] == 0


@pytest.mark.parametrize("dtype,tol", DTYPES)
@pytest.mark.parametrize("which", list(CONFIGS))
def test_mixed_batches_on_few_pages_and_slots(models, which, dtype, tol):
    """Unequal requests side by side, portions beside single tokens, with three state slots and a pool so small that
    pages and slots are used again; every logit equals the request's alone."""
    d, reqs, want = models[which]
    page = PAGE[which]
    reqs = dict(reqs)
    reqs.update({rid + 10: toks[: max(1, len(toks) - 3)] for rid, toks in list(reqs.items())})          # more requests than slots
    want = dict(want)
    want.update({rid: want[rid - 10] for rid in reqs if rid > 10})
    longest = max(len(t) for t in reqs.values())
    pool = ((longest + page - 1) // page + 6) * page
    if which == "B":                                               # no mask: every key stays, so the three live requests must fit whole
        pool = (3 * ((longest + page - 1) // page + 1) + 2) * page
    eng = H.engine_for(d, dtype, page, pool, max_requests=3)
    rng = np.random.default_rng(5)
    at = {rid: 0 for rid in reqs}
    waiting, live, steps = sorted(reqs, key=lambda r: (len(reqs[r]), r)), [], []
    held = lambda: sum((at[r] + page - 1) // page + 1 for r in live)
    while waiting or live:
        while waiting and len(live) < 3 and (held() + (len(reqs[waiting[0]]) + page - 1) // page + 2) * page <= pool:
            live.append(waiting.pop(0))
        if not live:
            live.append(waiting.pop(0))
        entries, end = [], []
        for rid in list(live):
            left = len(reqs[rid]) - at[rid]
            n = 1 if rng.random() < 0.4 else int(min(left, rng.integers(2, 40)))
            n = min(n, left)
            if rng.random() < 0.15 and len(live) > 1:
                continue                                            # a request may sit a step out
            entries.append((rid, reqs[rid][at[rid]:at[rid] + n], list(range(n))))
            at[rid] += n
            if at[rid] == len(reqs[rid]):
                end.append(rid)
                live.remove(rid)
        if entries:
            steps.append((entries, end))
    check(H.run_steps(eng, steps), want, tol, f"{which} {dtype} mixed")
    state = eng.cache_state()
    assert state["check"] == "" and state["requests"] == 0


def test_a_window_gives_pages_back_and_takes_them_again(models):
    """A request longer than the pool runs, because only its window is held; a second request then reuses the pages."""
    d, reqs, want = models["A"]                                     # windows of 21 and 9 positions on one cache, pages of 16
    eng = H.engine_for(d, "float32", 16, 6 * 16, max_requests=2, max_batch_tokens=64)
    toks = reqs[4]                                                  # 131 tokens through a pool of 96
    steps, at = [], 0
    for n in [30, 2, 17, 1, 1, 40, 9, 31]:
        steps.append(([(4, toks[at:at + n], list(range(n)))], []))
        at += n
    assert at == len(toks)
    steps[-1] = (steps[-1][0], [4])
    steps.append(([(3, reqs[3], list(range(len(reqs[3]))))], [3]))
    check(H.run_steps(eng, steps), want, FP32_TOL, "A float32 through a pool smaller than the request")
    assert eng.cache_state()["check"] == "" and eng.cache_state()["metrics"]["window_releases"] >= 3


def test_long_decoding_bfloat16_graphs(models):
    """130 decode-only steps of two requests (captured graphs, state slots and windows moving on): along the given tokens
    the logits stay with the plain implementation."""
    d, reqs, want = models["C"]
    eng = H.engine_for(d, "bfloat16", 16, 1024)
    a, b = reqs[3], reqs[2]
    steps = [([(3, a[:15], [14]), (2, b[:4], [3])], [])]
    for i in range(min(len(a) - 15, len(b) - 4)):
        steps.append(([(3, [a[15 + i]], [0]), (2, [b[4 + i]], [0])], []))
    check(H.run_steps(eng, steps), want, BF16_TOL, "C bfloat16 long decoding")
    assert len(eng._graphs) > 0                                     # the decode-only steps ran as captured graphs


def test_greedy_generation_through_the_entry_point(models):
    from aien_sovereign_core_mv_b200.engine.generate import generate
    from aien_sovereign_core_mv_b200.sampling import SamplingParams
    d, reqs, _ = models["A"]
    cfg, tensors = load_plain(d)
    prompts = [reqs[2], reqs[3][:30], reqs[1]]
    n_new = 10
    want = []
    for p in prompts:
        seq, out = list(p), []
        for _ in range(n_new):
            t = int(np.argmax(pr.forward(cfg, tensors, seq)[-1]))
            seq.append(t); out.append(t)
        want.append(out)
    eng = H.engine_for(d, "float32", 16, 512, prefill_chunk_size=16, max_prefill_tokens=32)
    got = generate(eng, prompts, SamplingParams(temperature=0.0, max_tokens=n_new, stop_token_ids=[]))
    assert got == want
    assert eng.cache_state()["requests"] == 0 and eng.cache_state()["check"] == ""


def test_sampling_and_the_command_line(models):
    """Sampling through the scheduler (temperature, top-p, top-k) runs and repeats under the same seed; the command line
    generates the plain implementation's greedy tokens and describes the model."""
    import subprocess
    from aien_sovereign_core_mv_b200.engine.generate import Generator
    from aien_sovereign_core_mv_b200.sampling import SamplingParams
    d, reqs, _ = models["B"]
    eng = H.engine_for(d, "bfloat16", 8, 512)
    params = SamplingParams(temperature=0.8, top_p=0.9, top_k=40, max_tokens=12, stop_token_ids=[], seed=7)
    a = Generator(eng).generate([reqs[2], reqs[1]], params, request_ids=[5, 6])
    b = Generator(eng).generate([reqs[2], reqs[1]], params, request_ids=[5, 6])
    assert [r.tokens for r in a] == [r.tokens for r in b] and all(len(r.tokens) == 12 for r in a)
    cfg, tensors = load_plain(d)
    seq, want = list(reqs[1]), []
    for _ in range(5):
        t = int(np.argmax(pr.forward(cfg, tensors, seq)[-1]))
        seq.append(t); want.append(t)
    exe = os.path.join(H.ROOT, "bin", "aien-b200")
    out = subprocess.run([exe, "generate", "--model-dir", d, "--dtype", "float32", "--prompt-ids", ",".join(map(str, reqs[1])),
                          "--max-tokens", "5", "--temperature", "0", "--stop-token-ids", "", "--json"], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
    assert json.loads(out.stdout.strip().splitlines()[-1])["tokens"] == [want]
    info = subprocess.run([exe, "info", "--model-dir", d], capture_output=True, text=True, timeout=600)
    assert info.returncode == 0, info.stderr[-2000:]
    rec = json.loads(info.stdout.strip().splitlines()[-1])
    assert rec["architecture"] == "Ripesun" and rec["layers"] == 3 and sorted(rec["cache_groups"]) == ["full", "state"]


def test_trace_replay_from_the_command(models, tmp_path):
    d, reqs, want = models["A"]
    toks = reqs[3]
    steps = [{"step": 0, "entries": [{"id": "x", "tokens": toks[:40], "want": [0, 39]}, {"id": 7, "tokens": reqs[1], "want": [0]}], "end": [7]},
             {"step": 1, "entries": [{"id": "x", "tokens": toks[40:42], "want": []}], "end": []},
             {"step": 2, "entries": [{"id": "x", "tokens": toks[42:], "want": [len(toks) - 43]}], "end": ["x"]}]
    out = H.run_trace(d, "float32", str(tmp_path / "out"), 192, steps)
    assert sorted(out) == [0, 2]
    H.assert_close(out[0], np.stack([want[3][0], want[3][39], want[1][0]]), FP32_TOL, "trace step 0")
    H.assert_close(out[2], want[3][-1:], FP32_TOL, "trace step 2")


# ------------------------------------------------------------------ configurations drawn at random
def _random_config(rng):
    """Sizes, order of layers, windows, sharing of caches, decays and constants drawn at random."""
    width = rng.choice([64, 72, 96, 128, 160])
    layers, own = [], []
    for i in range(rng.randint(3, 7)):
        kind = rng.choice(["latent_attention", "lightning", "mingru"])
        mlp = None if rng.random() < 0.2 else _dense(rng.choice([24, 40, 64, 96]))
        if kind == "latent_attention":
            j = rng.choice(own) if own and rng.random() < 0.4 else None
            if j is not None:
                kv_rank, rot_dim, base = layers[j]["mixer"]["kv_rank"], layers[j]["mixer"]["rot_dim"], layers[j]["mixer"]["rot"]["base"]
            else:
                kv_rank, rot_dim, base = rng.choice([16, 24, 40, 64, 128]), rng.choice([8, 16, 32, 6]), rng.choice([1e4, 1e6, 500.0])
            window = rng.choice([0, 5, 16, 33, 40, 100])
            if j is not None and (((layers[j]["mixer"].get("mask") or {}).get("size") or 0) == 0) != (window == 0):
                window = (layers[j]["mixer"].get("mask") or {}).get("size") or 0          # a cache that keeps all has readers that see all
            dim = rng.choice([8, 16, 24, 32, 64])
            layers.append({"type": kind, "mlp": mlp, "mixer": _latent(rng.choice([1, 2, 3, 4, 6, 17]), dim, rot_dim, rng.choice([8, 16, dim, 40]),
                                                                     kv_rank, rng.choice([16, 24, 48, 96]), window, (dim + rot_dim) ** -0.5, base, j)})
            if j is None:
                own.append(i)
        elif kind == "lightning":
            heads = rng.choice([1, 2, 4, 5])
            layers.append({"type": kind, "mlp": mlp, "mixer": _light(heads, rng.choice([8, 16, 64, 20]), rng.choice([8, 32, 12, 72]),
                                                                    [rng.choice([0.5, 0.9, 0.97, 0.999, 1.0]) for _ in range(heads)])})
        else:
            layers.append({"type": kind, "mlp": mlp, "mixer": {"width": rng.choice([32, 50, 128])}})
    cfg = {"architecture": "Ripesun", "vocab": rng.choice([101, 256, 333]), "width": width, "norm": {"eps": rng.choice([1e-5, 1e-6])},
           "embedding": {"scale": rng.choice([1.0, 4.0, 12.0])}, "residual_mult": rng.choice([0.5, 0.7, 1.0]),
           "logit_softcap": rng.choice([15.0, 30.0]), "layers": layers}
    side = rng.choice([0, 4, 8, 24])
    if side:
        cfg["token_side"] = {"dim": side}
    return cfg


@pytest.mark.parametrize("seed", range(8))
def test_configurations_drawn_at_random(seed, tmp_path):
    """Whole prompts, portions of changing size and three requests side by side, against the plain implementation.  float32
    must agree to rounding.  bfloat16 is held to a loose bound only: in a model this small one token whose branch output lies
    near zero before a norm can move a logit by a tenth through rounding alone, while a wrong key, mask or state moves it by
    its whole size."""
    import random
    from aien_sovereign_core_mv_b200 import write_random_model
    rng = random.Random(seed)
    cfg = _random_config(rng)
    d = write_random_model(os.path.join(str(tmp_path), "m"), cfg, 1000 + seed)
    c, tensors = load_plain(d)
    draw = np.random.default_rng(seed)
    reqs = {i + 1: [int(x) for x in draw.integers(0, cfg["vocab"], n)] for i, n in enumerate([rng.randint(1, 30), rng.randint(60, 120), rng.randint(100, 150)])}
    want = {r: pr.forward(c, tensors, t) for r, t in reqs.items()}

    def steps(mode):
        if mode == "whole":
            return [([(rid, t, list(range(len(t))))], [rid]) for rid, t in reqs.items()]
        out = []
        if mode == "portions":
            for rid, t in reqs.items():
                at = 0
                while at < len(t):
                    n = min(rng.choice([1, 2, 3, 7, 16, 33, 64]), len(t) - at)
                    out.append(([(rid, t[at:at + n], list(range(n)))], [rid] if at + n == len(t) else []))
                    at += n
            return out
        at, live = {r: 0 for r in reqs}, list(reqs)
        while live:
            entries, end = [], []
            for rid in list(live):
                n = min(len(reqs[rid]) - at[rid], 1 if rng.random() < 0.5 else rng.randint(2, 50))
                entries.append((rid, reqs[rid][at[rid]:at[rid] + n], list(range(n))))
                at[rid] += n
                if at[rid] == len(reqs[rid]):
                    end.append(rid); live.remove(rid)
            out.append((entries, end))
        return out

    for dtype, tol in (("float32", FP32_TOL), ("bfloat16", 0.25)):
        for mode in ("whole", "portions", "side by side"):
            eng = H.engine_for(d, dtype, rng.choice([8, 16, 32]), 512, max_requests=4)
            check(H.run_steps(eng, steps(mode)), want, tol, f"seed {seed} {dtype} {mode}")
            assert eng.cache_state()["check"] == "" and eng.cache_state()["requests"] == 0



@pytest.mark.parametrize("dim,rot,vdim,heads,q_rank,window,sink", [(128, 64, 128, 3, 48, 200, True), (64, 32, 64, 4, 0, 0, False), (72, 64, 40, 2, 64, 130, True),
                                                                  (16, 8, 64, 5, 0, 50, True), (128, 8, 24, 1, 32, 0, False)])
def test_latent_portions_with_a_rotated_part_expanded_and_absorbed(dim, rot, vdim, heads, q_rank, window, sink):
    """A mixed step (portions that fill no tile, single tokens, a window that has moved on, pages in any order) in both forms
    against 64 bits.  Four roundings to bfloat16 lie on the way of a result (2^-9 each of numbers its own size, a key's under
    the softmax): 3e-2 of the largest."""
    from aien_sovereign_core_mv_b200 import kernels as K
    from aien_sovereign_core_mv_b200.parts import GroupView, RunBinding, StepContext, StepLimits, Workspace
    from aien_sovereign_core_mv_b200.registry import make_part
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(dim + rot)
    width, r, page = 96, 64, 16
    part = make_part("mixer", "latent_attention", hidden_size=width, num_heads=heads, head_dim=dim, rot_dim=rot, value_dim=vdim, kv_rank=r, q_rank=q_rank,
                     window=window, sink=sink, norm_eps=1e-5,
                     position=make_part("position", "rotary", head_dim=rot, theta=10000.0, pairing="interleaved"))
    W = {n: (torch.randn(shape, generator=g, device="cuda") * (shape[-1] ** -0.5 if kind == "matrix" else 1.0)).to(torch.bfloat16)
         for n, (shape, kind) in part.param_shapes().items()}
    part.bind(W)
    bring, held = [150, 1, 40, 1, 2], [37, 260, 300, 0, 11]
    S, T = len(bring), sum(bring)
    h = torch.randn(T, width, generator=g, device="cuda").to(torch.bfloat16)
    q0 = [sum(bring[:s]) for s in range(S + 1)]
    pages = [(a + b + page - 1) // page for a, b in zip(bring, held)]
    order = torch.randperm(sum(pages) + 2, generator=g, device="cuda").to(torch.int32)
    table = torch.full((S, max(pages) + 1), -1, dtype=torch.int32, device="cuda")
    slot = lambda s, p: table[s, p // page].long() * page + p % page
    first = torch.zeros(1, (sum(pages) + 2) * page, r + rot, dtype=torch.bfloat16, device="cuda")
    slots = []
    for s in range(S):
        table[s, :pages[s]] = order[sum(pages[:s]):sum(pages[:s + 1])]
        p = torch.arange(held[s] + bring[s], device="cuda")
        first[0, slot(s, p[:held[s]])] = torch.randn(held[s], r + rot, generator=g, device="cuda").to(torch.bfloat16)
        slots.append(slot(s, p[held[s]:]))
    norm = lambda x, w: x / torch.sqrt(x.square().mean(-1, keepdim=True) + 1e-5) * w

    def turned(x, pos):
        a = pos.double().view(-1, *([1] * (x.dim() - 1))) * 10000.0 ** (-torch.arange(0, rot, 2, device="cuda").double() / rot)
        return torch.stack([x[..., 0::2] * a.cos() - x[..., 1::2] * a.sin(), x[..., 1::2] * a.cos() + x[..., 0::2] * a.sin()], -1).flatten(-2)

    D = {n: t.double() for n, t in W.items()}
    want = []
    for s in range(S):
        x, pos = h[q0[s]:q0[s + 1]].double(), torch.arange(held[s], held[s] + bring[s], device="cuda")
        q = (norm(x @ D["dq_proj"].T, D["dq_norm"]) @ D["uq_proj"].T if q_rank else x @ D["q_proj"].T).view(-1, heads, dim + rot)
        q = torch.cat([q[..., :dim], turned(q[..., dim:], pos)], -1)
        d = x @ D["dkv_proj"].T
        rows = torch.cat([first[0, slot(s, torch.arange(held[s], device="cuda"))].double(), torch.cat([norm(d[:, :r], D["dkv_norm"]), turned(d[:, r:], pos)], -1)])
        k = torch.cat([(rows[:, :r] @ D["uk_proj"].T).view(-1, heads, dim), rows[:, None, r:].expand(-1, heads, -1)], -1)
        z = torch.einsum("tnd,mnd->ntm", q, k) * (dim + rot) ** -0.5
        j = torch.arange(rows.shape[0], device="cuda")
        z = z.masked_fill((j > pos[:, None]) | (j <= pos[:, None] - (window or 1 << 30)), -float("inf"))
        if sink:
            z = torch.cat([z, D["sink"][:, None, None].expand(-1, z.shape[1], 1)], -1)
        o = torch.einsum("ntm,mnv->tnv", z.softmax(-1)[..., :rows.shape[0]], (rows[:, :r] @ D["uv_proj"].T).view(-1, heads, vdim))
        want.append(o.flatten(1) @ D["o_proj"].T)
    want = torch.cat(want).cpu().numpy()
    need = part.cache_need()
    tiles = [(s, q) for s in range(S) for q in range(0, bring[s], 128) if bring[s] > 1]
    lim = StepLimits(max_tokens=T, max_seqs=S, max_context=max(a + b for a, b in zip(bring, held)), itemsize=2)
    saved = K.LATENT_PORTIONS
    try:
        for form in ("absorb", "expand"):
            K.LATENT_PORTIONS = form
            store = first.clone()
            ws = Workspace(1 << 20, part.workspace_bytes(lim) + (1 << 16), torch.device("cuda"))
            ws.begin_layer()
            ctx = StepContext(dtype=torch.bfloat16, num_tokens=T, num_seqs=S, token_ids=i32([0] * T),
                              positions=i32([held[s] + i for s in range(S) for i in range(bring[s])]), seq_of_token=i32([s for s in range(S) for _ in range(bring[s])]),
                              q_start=i32(q0), ctx_len=i32([a + b for a, b in zip(bring, held)]),
                              groups=[GroupView(need.kind, page, need.window, table.shape[1], table, torch.cat(slots).to(torch.int32), {"latent": store})],
                              workspace=ws, max_q_len=max(bring), max_ctx_len=lim.max_context, decode_only=False,
                              prefill_tiles=(i32([s for s, _ in tiles]), i32([q for _, q in tiles]), len(tiles)), single_tokens=(i32([q0[1], q0[3]]), 2))
            y = part.forward(ctx, h, RunBinding(0, 0, True))
            y = (y.float().sum(0) if y.dim() == 3 else y.float()).cpu().numpy()
            H.assert_close(y, want, 3e-2, form)
    finally:
        K.LATENT_PORTIONS = saved


@pytest.mark.parametrize("bring,held", [([300], [0]), ([130, 171], [40, 0]), ([700], [64]), ([1, 260, 40], [90, 0, 200])])
def test_latent_portions_read_no_page_number_that_an_earlier_step_left(bring, held):
    """The expanded form's page table is made by a kernel of the step two launches ahead of the attention.  With the table's room
    holding zeros or other valid page numbers, and the step's launches queued behind work so that they follow one another
    closely, the results are those of a step whose table was there before, to the bit."""
    from aien_sovereign_core_mv_b200 import kernels as K
    from aien_sovereign_core_mv_b200.parts import GroupView, RunBinding, StepContext, StepLimits, Workspace
    from aien_sovereign_core_mv_b200.registry import make_part
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(sum(bring))
    width, heads, r, rot, page, S, T = 256, 4, 64, 64, 16, len(bring), sum(bring)
    part = make_part("mixer", "latent_attention", hidden_size=width, num_heads=heads, head_dim=128, rot_dim=rot, value_dim=128, kv_rank=r, q_rank=128, window=0,
                     norm_eps=1e-5, position=make_part("position", "rotary", head_dim=rot, theta=10000.0, pairing="interleaved"))
    part.bind({n: (torch.randn(shape, generator=g, device="cuda") * (shape[-1] ** -0.5 if kind == "matrix" else 1.0)).to(torch.bfloat16)
               for n, (shape, kind) in part.param_shapes().items()})
    h = torch.randn(T, width, generator=g, device="cuda").to(torch.bfloat16)
    q0 = [sum(bring[:s]) for s in range(S + 1)]
    pages = [(a + b + page - 1) // page for a, b in zip(bring, held)]
    table = torch.full((S, max(pages)), -1, dtype=torch.int32, device="cuda")
    for s in range(S):
        table[s, :pages[s]] = torch.arange(sum(pages[:s]), sum(pages[:s + 1]), dtype=torch.int32, device="cuda").flip(0)
    slots = torch.cat([table[s, p // page].long() * page + p % page for s in range(S) for p in [torch.arange(held[s], held[s] + bring[s], device="cuda")]])
    first = torch.randn(1, sum(pages) * page, r + rot, generator=g, device="cuda").to(torch.bfloat16)
    lim = StepLimits(max_tokens=T, max_seqs=S, max_context=max(a + b for a, b in zip(bring, held)), itemsize=2)
    position = make_part("position", "rotary", head_dim=rot, theta=10000.0, pairing="interleaved")
    ws = Workspace(position.step_workspace_bytes(T) + 4096, part.workspace_bytes(lim) + (1 << 16), torch.device("cuda"))
    tiles = [(s, q) for s in range(S) for q in range(0, bring[s], K.PREFILL_TILE) if bring[s] > 1]
    singles = [q0[s] for s in range(S) if bring[s] == 1]
    need = part.cache_need()
    store = first.clone()
    fixed = dict(dtype=torch.bfloat16, num_tokens=T, num_seqs=S, token_ids=i32([0] * T), positions=i32([held[s] + i for s in range(S) for i in range(bring[s])]),
                 seq_of_token=i32([s for s in range(S) for _ in range(bring[s])]), q_start=i32(q0), ctx_len=i32([a + b for a, b in zip(bring, held)]),
                 groups=[GroupView(need.kind, page, need.window, table.shape[1], table, slots.to(torch.int32), {"latent": store})],
                 workspace=ws, max_q_len=max(bring), max_ctx_len=lim.max_context, decode_only=False,
                 prefill_tiles=(i32([s for s, _ in tiles]), i32([q for _, q in tiles]), len(tiles)), single_tokens=(i32(singles or [0]), len(singles)))
    busy = torch.randn(4096, 4096, device="cuda").to(torch.bfloat16)
    words = ws.buf.view(torch.int32)
    other = torch.arange(words.numel(), dtype=torch.int32, device="cuda").flip(0) % (sum(pages) * page // 128)

    def step(left):
        store.copy_(first)
        if left is not None:
            words.copy_(left)
        ws.reset()
        ws.begin_layer()
        torch.cuda.synchronize()
        for _ in range(8):                                   # the step's launches wait behind this, and then start as close together as they can
            busy @ busy
        y = part.forward(StepContext(**fixed), h, RunBinding(0, 0, True))
        y = (y.float().sum(0) if y.dim() == 3 else y.float()).clone()
        torch.cuda.synchronize()
        return y, store.clone()

    saved = K.LATENT_PORTIONS
    try:
        K.LATENT_PORTIONS = "expand"
        step(torch.zeros_like(words))
        want = step(None)                                    # the table of the step before, which is this step's too
        assert bool(torch.isfinite(want[0]).all())
        for left in (torch.zeros_like(words), other, torch.full_like(words, 0x7fff7fff)):
            got = step(left)
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    finally:
        K.LATENT_PORTIONS = saved
