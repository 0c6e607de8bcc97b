"""Tomodra on the GPU against the plain implementation (tests/plain/tomodra_plain.py, 64-bit): every mechanism alone
through its kernel, then whole models through Engine.step, the scheduler and the trace runner, in float32 and
bfloat16, for configurations that differ in every size and option (tomodra_util.CONFIGS)."""
import tempfile

import numpy as np
import pytest
import torch

import tomodra_util as tu
import util
from plain import tomodra_plain as plain

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def dev(a, dtype=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a)).to(device=DEV, dtype=dtype)


def i32(a):
    return torch.tensor(list(a), dtype=torch.int32, device=DEV)


# ----------------------------------------------------------------------------- mechanisms alone
def test_norm_behind_the_sum():
    from air_b200.csrc import ops
    rng = np.random.default_rng(1)
    T, E = 11, 72
    h, w = rng.normal(size=(T, E)), rng.normal(1, 0.1, size=E)
    a, b, g = rng.normal(size=(3, T, E)), rng.normal(size=(2, T, E)), rng.uniform(size=T)
    want = plain.rms_norm(2.5 * h + a.sum(0) + g[:, None] * b.sum(0), w, 1e-5)
    for out_dtype in (torch.bfloat16, None):
        hd = dev(h)
        out = None if out_dtype is None else torch.empty((T, E), dtype=out_dtype, device=DEV)
        ops.post_norm(hd, 2.5, dev(a), dev(b), dev(g), dev(w), 1e-5, out)
        assert np.abs(hd.cpu().numpy() - want).max() < 1e-5
        if out is not None:
            assert np.abs(out.float().cpu().numpy() - want).max() < 2e-2
    hd = dev(h)
    ops.post_norm(hd, 1.0, dev(a[0]), None, None, dev(w, torch.bfloat16), 1e-5, None)      # one term, a 16-bit weight
    assert np.abs(hd.cpu().numpy() - plain.rms_norm(h + a[0], tu.bf16(w), 1e-5)).max() < 1e-5
    hd = dev(h)
    ops.post_norm(hd, 1.0, None, dev(b[0]), dev(g), None, 0.0, None)                        # the sum alone
    assert np.abs(hd.cpu().numpy() - (h + g[:, None] * b[0])).max() < 1e-5


@pytest.mark.parametrize("H,G,dk,dv,rot,pairing,scaling", [
    (4, 2, 32, 16, 16, "neighbours", (4.0, 64, 16.0, 2.0)), (1, 1, 48, 20, 48, "neighbours", None),
    (3, 3, 24, 40, 12, "half", (2.0, 16, 4.0, 1.0)), (2, 1, 256, 8, 64, "neighbours", (8.0, 1024, 32.0, 1.0)),
    (2, 2, 6, 6, 0, "neighbours", None)])
def test_queries_and_keys_are_normalised_then_rotated(H, G, dk, dv, rot, pairing, scaling):
    """Positions far apart (angles of thousands of turns), pages scattered, two requests: q and the pages against the
    plain functions."""
    from air_b200.csrc import ops
    from air_b200.parts.rope import bent_frequencies
    rng = np.random.default_rng(dk)
    P, base, eps = 16, 5000.0, 1e-5
    sc = dict(zip(("factor", "original", "fast", "slow"), scaling)) if scaling else None
    positions = np.array([0, 1, 15, 16, 17, 100000, 31, 32])
    slots = np.array([1, 1, 1, 1, 1, 0, 0, 0])
    T = len(positions)
    proj = rng.normal(size=(T, (H + G) * dk + G * dv)) * 3
    qw, kw = rng.normal(1, 0.2, size=dk), rng.normal(1, 0.2, size=dk)
    f, mag = plain.yarn_frequencies(rot, base, sc) if rot else (np.zeros(0), 1.0)
    rotate = plain.rotate_neighbours if pairing == "neighbours" else \
        (lambda x, p, f, d, m: plain.rotate_half_split(x, p, f, d) * 1.0)
    q = plain.rms_norm(proj[:, :H * dk].reshape(T, H, dk), qw, eps)
    k = plain.rms_norm(proj[:, H * dk:(H + G) * dk].reshape(T, G, dk), kw, eps)
    if rot:
        q, k = rotate(q, positions, f, rot, mag), rotate(k, positions, f, rot, mag)
    v = proj[:, (H + G) * dk:].reshape(T, G, dv)
    table = torch.full((2, 8192), -1, dtype=torch.int32, device=DEV)
    table[1, :2] = i32([5, 2])
    table[0, [100000 // P, 1, 2]] = i32([7, 0, 3])
    freq = bent_frequencies(rot, base, sc)[0].to(DEV) if rot else None
    if pairing == "half" and sc:
        mag = 1.0           # (the plain half-split rotation has no magnitude)
    cache = torch.zeros((8, G * P * (dk + dv)), device=DEV)
    qo = torch.empty((T, H, dk), device=DEV)
    ops.qk_normed_prepare(dev(proj), dev(qw), dev(kw), eps, freq, pairing, mag, i32(positions), i32(slots), table, qo,
                          cache, G, dv, P)
    assert np.abs(qo.cpu().numpy() - q).max() < 2e-5
    pages = cache.cpu().numpy()
    for t in range(T):
        page = int(table[slots[t], positions[t] // P])
        keys = pages[page, :G * P * dk].reshape(G, P, dk)[:, positions[t] % P]
        values = pages[page, G * P * dk:].reshape(G, P, dv)[:, positions[t] % P]
        assert np.abs(keys - k[t]).max() < 2e-5 and np.abs(values - v[t]).max() < 1e-6
    if rot == 0:      # and without weights nothing is normalised
        ops.qk_normed_prepare(dev(proj), None, None, eps, None, pairing, 1.0, i32(positions), i32(slots), table, qo,
                              cache, G, dv, P)
        assert np.abs(qo.cpu().numpy() - proj[:, :H * dk].reshape(T, H, dk)).max() < 1e-6


def attend(q, k, v, scale, mask, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H, dv], with the plain softmax."""
    H, G = q.shape[1], k.shape[1]
    k, v = np.repeat(k, H // G, axis=1), np.repeat(v, H // G, axis=1)
    a = plain.masked_softmax(np.einsum("thd,shd->hts", q, k) * scale, mask, sink)
    return np.einsum("hts,shd->thd", a, v)


def pointed(rng, T, H, G, d, dv, pairs, scale):
    """Random queries, keys and values in which query i of each pair (i, j) points at key j so strongly that key j,
    if it is seen, takes nearly all the weight; its value is large."""
    q, k, v = rng.normal(size=(T, H, d)), rng.normal(size=(T, G, d)), rng.normal(size=(T, G, dv))
    for i, j in pairs:
        q[i] = np.repeat(k[j], H // G, axis=0) * (14.0 / scale / d)
        v[j] = 20.0 + j / 20.0
    return q, k, v


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind,size", [("window", 50), ("chunk", 40), ("window", 1), ("chunk", 16), ("all", None)])
def test_attention_sees_the_keys_inside_its_mask_and_no_other(kind, size, dtype):
    """One request of 300 tokens over scattered pages of 16.  Queries are made to point at keys far away, at the first
    key that their window or chunk still holds and at the one just outside it; a sink in the softmax.  As rows of
    prompt portions, and token by token."""
    from air_b200.csrc import ops
    rng = np.random.default_rng(size or 0)
    T, P, H, G, d, dv, scale = 300, 16, 4, 2, 32, 24, 0.2
    n = size or T
    if kind == "chunk":
        mask = plain.chunk_mask(T, n)
        pairs = [(299, 299 - 299 % n), (298, 299 - 299 % n - 1), (2 * n - 1, n), (2 * n, 2 * n - 1), (250, 3)]
    else:
        mask = plain.window_mask(T, n)
        pairs = [(299, 299 - n + 1), (298, max(298 - n, 0)), (min(n + 5, 280), 6), (min(n + 4, 279), 3), (250, 3)]
    q, k, v = pointed(rng, T, H, G, d, dv, pairs, scale)
    sink = rng.normal(1.0, 2.0, size=H)
    if dtype == torch.bfloat16:
        q, k, v = (tu.bf16(x).astype(np.float64) for x in (q, k, v))
    want = attend(q, k, v, scale, mask, sink)
    if size and size > 1:
        other = plain.window_mask(T, n + 1) if kind == "window" else plain.chunk_mask(T, n + 1)
        assert np.abs(attend(q, k, v, scale, other, sink) - want).max() > 5.0        # one key more or less shows
    pages = rng.permutation(40)[:-(-T // P)]
    table = torch.full((2, 64), -1, dtype=torch.int32, device=DEV)
    table[1, :len(pages)] = i32(pages)
    cache = torch.zeros((40, G * P * (d + dv)), dtype=dtype, device=DEV)
    for t in range(T):
        page = cache[pages[t // P]]
        page[:G * P * d].view(G, P, d)[:, t % P] = dev(k[t], dtype)
        page[G * P * d:].view(G, P, dv)[:, t % P] = dev(v[t], dtype)
    for cuts in ([2, 61, T - 63], [T - 3, 1, 1, 1]):
        at = 0
        for m in cuts:
            for kernel, more in ((ops.paged_attention_ref, {}), (ops.grouped_attention, {}),
                                 (ops.grouped_attention, {"splits": 3})):
                out = torch.empty((m, H, dv), dtype=dtype, device=DEV)
                kernel(dev(q[at:at + m], dtype), cache, table, i32([1] * m), i32(range(at, at + m)), out,
                       size if kind == "window" else None, scale, kv_heads=G, page_tokens=P,
                       chunk=size if kind == "chunk" else None, sink=dev(sink), **more)
                tol = 3e-4 if dtype == torch.float32 else 0.3          # (values up to 35: bfloat16 holds them to 0.125)
                assert np.abs(out.float().cpu().numpy() - want[at:at + m]).max() < tol, (at, m, kernel.__name__)
            at += m
    if dtype != torch.bfloat16:
        return
    # the same rows as portions of a batch: long portions through the matrix products over gathered keys (in blocks of
    # 100 queries here, so that blocks begin inside windows and chunks), a short one and single tokens of another
    # request through the pages, in one step
    from types import SimpleNamespace
    from air_b200.parts.base import HostBatch, Runtime
    from air_b200.parts.gathered_attention import PortionAttention

    class Road(PortionAttention):
        BLOCK = 100
        rt = Runtime(device=torch.device(DEV), dtype=torch.bfloat16, page_tokens=P)
        heads, kv_heads, window, chunk, sinks = H, G, size if kind == "window" else None, size if kind == "chunk" else None, dev(sink)

    road = Road()
    road.scale = scale
    table[0, :len(pages)] = i32(pages)                  # a second request that holds the same pages
    for counts, lengths, slots in (([1, 33, 1], [40, 0, 299], [0, 1, 0]), ([2, 261], [37, 39], [0, 1]), ([300], [0], [1])):
        q_start = [0] + np.cumsum(counts).tolist()
        batch = HostBatch(counts=counts, lengths=lengths, slots=slots, q_start=q_start)
        plan = road.plan(batch)
        positions = [p for n, l in zip(counts, lengths) for p in range(l, l + n)]
        seq = [s_ for n, s_ in zip(counts, slots) for _ in range(n)]
        ctx = SimpleNamespace(plans={road.plan_key(): SimpleNamespace(small_seq=i32(plan.arrays["small_seq"]), **plan.values)},
                              token_seq=i32(seq), positions=i32(positions))
        out = torch.empty((len(positions), H, dv), dtype=dtype, device=DEV)
        road.attend(dev(q[positions], dtype), cache, table, ctx, out, kv_heads=G, page_tokens=P)
        assert np.abs(out.float().cpu().numpy() - want[positions]).max() < 0.3, counts


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,d,rot,R,dv,window", [(4, 24, 8, 40, 20, 48), (1, 32, 16, 56, 40, None), (3, 8, 4, 300, 8, 17), (16, 32, 16, 112, 24, 40), (7, 16, 8, 600, 8, None)])
def test_latent_attention_through_its_kernels(H, d, rot, R, dv, window, dtype):
    """From the projection's output to the heads' outputs: the rows in the pages, the queries carried through the key
    expansion, attention over the rows, the value expansion.  Against keys and values expanded per head, as the
    equations have them.  Queries point at the first row inside the window and at the one before it."""
    from air_b200.csrc import ops
    rng = np.random.default_rng(R)
    T, P, scale, base, eps = 150, 16, 0.2, 1000.0, 1e-5
    n = window or T
    proj = rng.normal(size=(T, H * (d + rot) + R + rot))
    cw = rng.normal(1, 0.2, size=R)
    uk, uv = rng.normal(size=(H * d, R)) / R ** 0.5, rng.normal(size=(H * dv, R)) / R ** 0.5
    m = dict(kv_rank=R, rot_dim=rot, rot=dict(base=base))
    f = plain.plain_frequencies(rot, base)
    positions = np.arange(T)
    c = plain.rms_norm(proj[:, H * (d + rot):H * (d + rot) + R], cw, eps)
    kr = plain.rotate_half_split(proj[:, H * (d + rot) + R:], positions, f, rot)
    for i, j in ((T - 1, T - n), (T - 2, max(T - 2 - n, 0)), (100, 3)):
        # the plain part of the query is the key it should find, enlarged
        key = (c[j] @ uk.T).reshape(H, d)
        proj[i, :H * (d + rot)].reshape(H, d + rot)[:, :d] = key * (14.0 / scale / (key ** 2).sum(-1, keepdims=True))
    if dtype == torch.bfloat16:
        uk, uv = tu.bf16(uk), tu.bf16(uv)
    q = proj[:, :H * (d + rot)].reshape(T, H, d + rot)
    q = np.concatenate([q[..., :d], plain.rotate_half_split(q[..., d:], positions, f, rot)], axis=-1)
    keys = np.concatenate([(c @ uk.T).reshape(T, H, d), np.repeat(kr[:, None], H, axis=1)], axis=-1)
    values = (c @ uv.T).reshape(T, H, dv)
    want = attend(q, keys, values, scale, plain.window_mask(T, n))
    if window:
        assert np.abs(attend(q, keys, values, scale, plain.window_mask(T, n + 1)) - want).max() > 0.3
    pages = rng.permutation(20)[:-(-T // P)]
    table = torch.full((3, 64), -1, dtype=torch.int32, device=DEV)
    table[2, :len(pages)] = i32(pages)
    rows = torch.zeros((20, P, R + rot), dtype=dtype, device=DEV)
    uk_t = dev(uk.reshape(H, d, R).transpose(0, 2, 1), dtype)
    uv_d = dev(uv.reshape(H, dv, R), dtype)
    freq = dev(f, torch.float64)
    at = 0
    for cut in (3, 61, T - 67, 1, 1, 1):
        pos, seq = i32(range(at, at + cut)), i32([2] * cut)
        q_plain = torch.empty((cut, H, d), dtype=dtype, device=DEV)
        q_full = torch.empty((cut, H, R + rot), device=DEV)
        p = dev(proj[at:at + cut])
        ops.latent_prepare(p[:, :H * (d + rot)], p[:, H * (d + rot):], dev(cw), eps, freq, pos, seq, table, q_plain, q_full, rows,
                           True)
        ops.grouped_gemm(q_plain, uk_t, q_full, R, d, lda=H * d, ldo=H * (R + rot), groups=H, a_group_stride=d,
                         o_group_stride=R + rot, a_local=True, o_local=True, rows_per_group=cut)
        summed = torch.empty((cut, H, R), dtype=dtype, device=DEV)
        ops.paged_attention_ref(q_full, rows, table, seq, pos, summed, window, scale, latent=True)
        if ops.grouped_attention_ok(dtype, R + rot, R):
            again = torch.empty((cut, H, R), dtype=dtype, device=DEV)
            ops.grouped_attention(q_full, rows, table, seq, pos, again, window, scale, latent=True)
            assert np.abs(again.float().cpu().numpy() - summed.float().cpu().numpy()).max() < (1e-5 if dtype == torch.float32 else 2e-2)
        out = torch.empty((cut, H, dv), dtype=dtype, device=DEV)
        ops.grouped_gemm(summed, uv_d, out, dv, R, lda=H * R, ldo=H * dv, groups=H, a_group_stride=R,
                         o_group_stride=dv, a_local=True, o_local=True, rows_per_group=cut)
        tol = 3e-4 if dtype == torch.float32 else 0.1
        assert np.abs(out.float().cpu().numpy() - want[at:at + cut]).max() < tol, (at, cut)
        at += cut
    kept = rows.float().cpu().numpy()
    for t in (0, 15, 16, T - 1):
        row = kept[pages[t // P], t % P]
        tol = 2e-5 if dtype == torch.float32 else 3e-2
        assert np.abs(row[:R] - c[t]).max() < tol and np.abs(row[R:] - kr[t]).max() < tol


@pytest.mark.parametrize("mask", [("all", None), ("window", 70), ("window", 450), ("chunk", 200)])
@pytest.mark.parametrize("G,J,d,dv,latent,P", [(2, 5, 64, 48, False, 16), (1, 18, 128, 128, False, 64), (2, 16, 256, 200, False, 48),
                                                (1, 20, 576, 512, True, 16), (1, 3, 512, 512, False, 64), (1, 16, 640, 128, True, 32),
                                                (1, 17, 640, 600, True, 64)])
def test_grouped_attention_over_many_tiles_of_keys(G, J, d, dv, latent, P, mask):
    """Every shape of block (rows of up to 128, 256 and 640 numbers, one and two stages, values beyond 512), with so few splits
    that a block walks several tiles, and with more splits than tiles: against the 64-bit softmax, at positions around the edges
    of tiles; float32 and bfloat16 queries.  Keys that no query sees are NaN."""
    from air_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(d + J)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    kind, size = mask
    H, n, scale = G * J, 720, 2.5 * d ** -0.5
    k = rand(n, G, d).bfloat16()
    v = k[:, :, :dv] if latent else rand(n, G, dv).bfloat16()
    blocks = -(-n // P)
    table = torch.full((3, 64), -1, dtype=torch.int32, device="cuda")
    pages = torch.randperm(64, generator=g, device="cuda")[:blocks]
    table[2, :blocks] = pages.int()
    cache = torch.full((64, P, d) if latent else (64, G * P * (d + dv)), float("nan"), dtype=torch.bfloat16, device="cuda")
    at = torch.tensor([0, 63, 64, 127, 255, 384, 449, 450, 599, 600, 713], device="cuda")
    last = int(at.max())
    for t in range(last + 1):
        page = cache[pages[t // P]]
        if latent:
            page[t % P] = k[t, 0]
        else:
            page[:G * P * d].view(G, P, d)[:, t % P] = k[t]
            page[G * P * d:].view(G, P, dv)[:, t % P] = v[t]
    key = torch.arange(last + 1, device="cuda")[None]
    low = {"all": at * 0, "window": at - (size or 0) + 1, "chunk": at - at % (size or 1)}[kind]
    seen = (key <= at[:, None]) & (key >= low[:, None])
    sink = rand(H)
    for q in (rand(len(at), H, d), rand(len(at), H, d).bfloat16()):
        x = torch.einsum("tgjd,sgd->tgjs", q.double().view(len(at), G, J, d), k[:last + 1].double()) * scale
        x = torch.cat([x.masked_fill(~seen[:, None, None], -float("inf")), sink.double().view(1, G, J, 1).expand(len(at), G, J, 1)], dim=-1)
        want = torch.einsum("tgjs,sgv->tgjv", torch.softmax(x, dim=-1)[..., :-1], v[:last + 1].double()).reshape(len(at), H, dv)
        for splits in (1, 2, 3, 16):
            out = torch.empty((len(at), H, dv), dtype=torch.bfloat16, device="cuda")
            ops.grouped_attention(q, cache, table, i32([2] * len(at)), at.int(), out, size if kind == "window" else None, scale, kv_heads=G,
                                  page_tokens=P, chunk=size if kind == "chunk" else None, sink=sink, latent=latent, splits=splits)
            # (a result rounded to the 8 bits of bfloat16: 2^-8 of it at most; the 32-bit queries and weights enter as two bfloat16
            # numbers each, 2^-16 of them)
            assert ((out.double() - want).abs() - want.abs() / 256).max() <= 1e-4 * max(1.0, want.abs().max().item()), splits


@pytest.mark.parametrize("n,top,groups", [(31, 4, 1), (32, 32, 4), (33, 4, 3), (128, 8, 8), (129, 32, 3),
                                          (256, 8, 8), (257, 8, 1), (512, 8, 8)])
def test_router_at_the_edges_of_its_lanes(n, top, groups):
    """The numbers of experts at which a lane's room changes, with ties, with and without groups: the chosen experts are those
    of a stable sort; a weight is a sigmoid in 32 bits (a few roundings of a number below 1)."""
    from air_b200.csrc import ops
    rng = np.random.default_rng(n)
    T = 9
    z = np.round(rng.normal(size=(T, n)) * 8) / 8              # many equal scores
    z[2] = 0.5
    z[3, n - 1] = 9.0                                          # the last lane's last expert
    s = plain.sigmoid(z)
    expert = torch.empty((T, top), dtype=torch.int32, device=DEV)
    weight = torch.empty((T, top), device=DEV)
    keep = max(1, -(-top * groups // n), groups - 1)
    for g, k in ((1, 0), (groups, keep)):
        chosen = s.copy()
        if g > 1:
            marks = np.sort(s.reshape(T, g, n // g), axis=-1)[:, :, -1]
            out = np.argsort(-marks, axis=-1, kind="stable")[:, k:]
            for t in range(T):
                for group in out[t]:
                    chosen[t, group * (n // g):(group + 1) * (n // g)] = -1
        order = np.argsort(-chosen, axis=-1, kind="stable")[:, :top]
        more = dict(groups=g, keep=k, mark="best") if g > 1 else {}
        if top > (k * (n // g) if g > 1 else n):
            continue
        ops.moe_route(dev(z), n, top, expert, weight, None, **more)
        assert np.array_equal(expert.cpu().numpy(), order)
        assert np.abs(weight.cpu().numpy() - np.take_along_axis(s, order, -1)).max() < 1e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,top,E,F,T", [(5, 2, 64, 48, 150), (3, 3, 96, 40, 7), (8, 1, 72, 64, 65), (130, 6, 32, 20, 40)])
def test_router_and_experts(n, top, E, F, T, dtype):
    """The chosen experts and their weights against a sort; every (token, choice) once in its expert's slots; the two
    grouped products against the plain expert with the weight on its input."""
    from air_b200.csrc import ops
    rng = np.random.default_rng(n)
    x = rng.normal(size=(T, E))
    z = rng.normal(size=(T, n + 1)) * 2
    z[3, :n] = 0.7                                             # all equal: the lowest indices win
    if n > 2:
        z[5, 1], z[5, 2] = 1.5, 1.5
    expert = torch.empty((T, top), dtype=torch.int32, device=DEV)
    weight = torch.empty((T, top), device=DEV)
    gate = torch.empty((T,), device=DEV)
    ops.moe_route(dev(z), n, top, expert, weight, gate, has_gate=True)
    s = plain.sigmoid(z[:, :n].astype(np.float32).astype(np.float64))
    order = np.argsort(-s, axis=-1, kind="stable")[:, :top]
    assert np.array_equal(expert.cpu().numpy(), order)
    assert np.abs(weight.cpu().numpy() - np.take_along_axis(s, order, -1)).max() < 1e-6
    assert np.abs(gate.cpu().numpy() - plain.sigmoid(z[:, n])).max() < 1e-6
    soft = torch.empty((T, top), device=DEV)
    ops.moe_route(dev(z), n, top, expert, soft, None, score="softmax", renormalize=True)
    p = np.exp(z[:, :n] - z[:, :n].max(-1, keepdims=True))
    p = np.take_along_axis(p / p.sum(-1, keepdims=True), np.argsort(-p, axis=-1, kind="stable")[:, :top], -1)
    assert np.abs(soft.cpu().numpy() - p / p.sum(-1, keepdims=True)).max() < 1e-5
    ops.moe_route(dev(z), n, top, expert, weight, gate, has_gate=True)
    pairs = T * top
    start = torch.empty(n + 1, dtype=torch.int32, device=DEV)
    slots = torch.empty(pairs, dtype=torch.int32, device=DEV)
    tiles = torch.full((pairs // ops.GROUP_TILE + n, 2), -1, dtype=torch.int32, device=DEV)
    count = torch.empty(1, dtype=torch.int32, device=DEV)
    ops.moe_sort(expert, n, start, slots, tiles, count)
    st, sl = start.cpu().numpy(), slots.cpu().numpy()
    assert sorted(sl.tolist()) == list(range(pairs)) and st[0] == 0 and st[-1] == pairs
    for e in range(n):
        assert all(order.reshape(-1)[p] == e for p in sl[st[e]:st[e + 1]])
    listed = tiles.cpu().numpy()[:int(count)]
    assert sum(-(-(st[e + 1] - st[e]) // ops.GROUP_TILE) for e in range(n)) == len(listed)
    w = {}
    for e in range(n):
        w[f"e{e}.gate"], w[f"e{e}.up"] = rng.normal(size=(F, E)) / E ** 0.5, rng.normal(size=(F, E)) / E ** 0.5
        w[f"e{e}.down"] = rng.normal(size=(E, F)) / F ** 0.5
    if dtype == torch.bfloat16:
        w = {k: tu.bf16(a).astype(np.float64) for k, a in w.items()}
        x = tu.bf16(x).astype(np.float64)
    gate_up = dev(np.stack([np.concatenate([w[f"e{e}.gate"], w[f"e{e}.up"]]) for e in range(n)]), dtype)
    down = dev(np.stack([w[f"e{e}.down"] for e in range(n)]), dtype)
    act = torch.empty((pairs, F), dtype=dtype, device=DEV)
    ops.grouped_gemm(dev(x, dtype), gate_up, act, F, E, lda=E, ldo=F, groups=n, a_index=slots, a_div=top,
                     a_scale=weight.view(-1), start=start, tiles=tiles, num_tiles=count, silu_mul=True)
    y = torch.full((top, T, E), 9.0, device=DEV)
    ops.grouped_gemm(act, down, y, E, F, lda=F, ldo=E, groups=n, o_index=slots, o_div=top, o_part_stride=T * E,
                     start=start, tiles=tiles, num_tiles=count)
    want = np.zeros((T, E))
    sw = weight.cpu().numpy().astype(np.float64)
    for t in range(T):
        for j in range(top):
            u = sw[t, j] * x[t]
            want[t] += plain.expert(tu.bf16(u).astype(np.float64) if dtype == torch.bfloat16 else u, w, f"e{order[t, j]}.")
    tol = 1e-4 if dtype == torch.float32 else 3e-2
    assert np.abs(y.sum(0).cpu().numpy() - want).max() < tol * max(1.0, np.abs(want).max())


# ----------------------------------------------------------------------------- whole models
LENGTHS = {"A": (1, 7, 33, 97, 150), "B": (5, 40, 131, 64), "C": (2, 65, 150, 300)}


def streams_for(name, seed=0, lengths=None):
    return {f"{name}{i}": tu.tokens_for(name, n, seed + i) for i, n in enumerate(lengths or LENGTHS[name])}


def replay(name, dtype, steps, page_tokens=16, max_requests=4, peak_page=64):
    return util.replay(tu.model_folder(name), dtype, steps, max_tokens=util.peak_tokens(steps, page=peak_page),
                       page_tokens=page_tokens, max_requests=max_requests)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["A", "B", "C"])
def test_whole_prompts(name, dtype):
    streams = streams_for(name)
    got, _ = replay(name, dtype, util.trace_whole(streams))
    tu.check(got, name, streams, dtype)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["A", "B", "C"])
def test_prompt_then_token_by_token(name, dtype):
    """The tail is decoded one by one, long enough for windows and chunks to pass over decoded tokens."""
    streams = streams_for(name, 10)
    got, _ = replay(name, dtype, util.trace_bulk_tail(streams, tail=75))
    tu.check(got, name, streams, dtype)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["A", "B", "C"])
def test_portions_down_to_two_tokens(name, dtype):
    streams = streams_for(name, 20)
    got, _ = replay(name, dtype, util.trace_portions(streams))
    tu.check(got, name, streams, dtype)
    got, _ = replay(name, dtype, util.trace_portions(streams, sizes=(2, 2, 1, 3, 16, 15, 17, 64, 63, 65, 2)), page_tokens=64)
    tu.check(got, name, streams, dtype)


@pytest.mark.parametrize("page", [16, 64])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["A", "B", "C"])
def test_unequal_requests_together_with_pages_and_slots_used_again(name, dtype, page):
    """Ten requests through three slots and a pool that holds the peak only: every request must come out as it does
    alone (the oracle runs each alone), whatever shared its batches and whoever had its slot and pages before."""
    lengths = LENGTHS[name] + (120, 2, 77, 101, 64, 129)
    streams = streams_for(name, 50, lengths)
    steps = util.trace_mixed(streams, seed=3, live=3)
    got, engine = replay(name, dtype, steps, page_tokens=page, max_requests=3)
    tu.check(got, name, streams, dtype)
    for group in engine.cache.groups:
        assert group.pool.takes > group.pool.num_pages, "pages were used again"


@pytest.mark.parametrize("name", ["A", "B", "C"])
def test_experts_through_the_librarys_grouped_product(name, monkeypatch):
    """The road that steps of many rows per expert take through the experts, forced for short prompts too; experts that
    nobody chose, experts with one row, mixed batches."""
    from air_b200.parts.experts import RoutedExperts
    monkeypatch.setattr(RoutedExperts, "LIBRARY_ROWS", 0)
    streams = streams_for(name, 70, (3, 150, 41))
    got, _ = replay(name, "bfloat16", util.trace_whole(streams), page_tokens=64)
    tu.check(got, name, streams, "bfloat16")
    got, _ = replay(name, "bfloat16", util.trace_mixed(streams, seed=4, live=3), page_tokens=64, max_requests=3)
    tu.check(got, name, streams, "bfloat16")


@pytest.mark.parametrize("name", ["random1", "random2", "random3", "random5", "random8", "random13", "random21", "random34"])
def test_configurations_drawn_at_random(name):
    """Layer orders, sizes and constants that nobody chose (tomodra_util.random_config): whole prompts and a mixed
    schedule through three slots, in float32 within its tolerance; bfloat16 must be finite and agree with the oracle in
    the median (how far single rows lie depends on how a drawn model amplifies rounding)."""
    folder = tu.model_folder(name)
    streams = {f"{name}_{i}": tu.tokens_for(name, n, 80 + i) for i, n in enumerate((150, 3, 70, 1, 97))}
    margin = min(tu.plain_run(name, toks)[1] for toks in streams.values())
    whole = util.trace_whole(streams)
    mixed = util.trace_mixed(streams, seed=5, live=3, tail=20)
    got, _ = replay(name, "float32", whole, page_tokens=64)
    tu.check(got, name, streams, "float32")
    got, _ = replay(name, "float32", mixed, page_tokens=16, max_requests=3)
    tu.check(got, name, streams, "float32")
    for steps, page in ((whole, 16), (mixed, 64)):
        got, _ = replay(name, "bfloat16", steps, page_tokens=page, max_requests=3)
        means = []
        for (rid, p), row in got.items():
            ref = tu.plain_logits(name, streams[rid])[p]
            assert np.isfinite(row).all()
            means.append(np.abs(row - ref).mean() / max(1.0, np.abs(tu.plain_logits(name, streams[rid])).max()))
        if margin > 0.01:
            assert np.median(means) <= 2 * tu.BF16_MEDIAN_TOL, (name, float(np.median(means)))


@pytest.mark.parametrize("name", ["A", "C"])
def test_float32_does_not_depend_on_the_cut_or_the_batch(name):
    streams = streams_for(name, 30, (97, 40, 131))
    whole, _ = replay(name, "float32", util.trace_whole(streams))
    cut, _ = replay(name, "float32", util.trace_portions(streams, sizes=(2, 31, 1, 16, 5)))
    mixed, _ = replay(name, "float32", util.trace_mixed(streams, seed=1, live=3), max_requests=3)
    for key, row in whole.items():
        assert np.abs(cut[key] - row).max() < 2e-5
        assert np.abs(mixed[key] - row).max() < 2e-5


@pytest.mark.parametrize("name", ["A", "B", "C"])
def test_bfloat16_agrees_with_itself_across_schedules(name):
    """Rows of whole prompts against the same rows from portions and from mixed batches.  Long portions attend through
    matrix products over gathered keys, short ones and single tokens through the pages, so a row's rounding depends on
    the schedule; the rows must still agree as they agree with the oracle."""
    streams = streams_for(name, 30, (97, 40, 131))
    whole, _ = replay(name, "bfloat16", util.trace_whole(streams), page_tokens=64)
    cut, _ = replay(name, "bfloat16", util.trace_portions(streams, sizes=(2, 31, 1, 16, 5)), page_tokens=64)
    mixed, _ = replay(name, "bfloat16", util.trace_mixed(streams, seed=1, live=3), page_tokens=64, max_requests=3)
    for other in (cut, mixed):
        means = []
        for key, row in whole.items():
            scale = max(1.0, np.abs(row).max())
            diff = np.abs(other[key] - row)
            # (each is within the row limits of the oracle: together twice that)
            assert diff.max() <= 2 * tu.BF16_MAX_TOL * scale and diff.mean() <= 2 * tu.BF16_MEAN_TOL * scale, key
            means.append(diff.mean() / scale)
        assert np.median(means) <= tu.BF16_MEDIAN_TOL


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["A", "C"])
def test_page_borders_and_first_tokens(name, dtype):
    """Prompts that end just before, on and just behind a page's last place, then decoded across the border; and
    requests decoded from their very first token."""
    from air_b200.engine.batch import Entry
    from air_b200.engine.engine import Engine, EngineConfig
    engine = Engine.from_folder(tu.model_folder(name), EngineConfig(dtype=dtype, page_tokens=16, max_tokens=1024,
                                                                    max_requests=4))
    for n in (15, 16, 17, 31, 33):
        toks = tu.tokens_for(name, n + 4, n)
        got = [engine.step([Entry("r", toks[:n], range(n))]).cpu().numpy()]
        got += [engine.step([Entry("r", [t], [0])]).cpu().numpy() for t in toks[n:]]
        engine.finish("r")
        tu.check({("r", p): row for p, row in enumerate(np.concatenate(got))}, name, {"r": toks}, dtype)
    toks = tu.tokens_for(name, 6, 99)
    got = np.concatenate([engine.step([Entry("s", [t], [0])]).cpu().numpy() for t in toks])
    tu.check({("s", p): row for p, row in enumerate(got)}, name, {"s": toks}, dtype)
    got = [engine.step([Entry("t", toks[:2], [0, 1])]).cpu().numpy()]
    got += [engine.step([Entry("t", [t], [0])]).cpu().numpy() for t in toks[2:]]
    tu.check({("t", p): row for p, row in enumerate(np.concatenate(got))}, name, {"t": toks}, dtype)
    engine.check_status()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["A", "B"])
def test_long_decoding(name, dtype):
    """320 tokens one by one after a prompt of five, across twenty pages, windows and chunks (the decode steps replay
    a CUDA graph); pages that windows and chunks have left are back in the pool."""
    from air_b200.engine.batch import Entry
    from air_b200.engine.engine import Engine, EngineConfig
    toks = tu.tokens_for(name, 325, 7)
    engine = Engine.from_folder(tu.model_folder(name), EngineConfig(dtype=dtype, page_tokens=16, max_tokens=384,
                                                                    max_requests=2))
    got = [engine.step([Entry("r", toks[:5], range(5))]).cpu().numpy()]
    got += [engine.step([Entry("r", [t], [0])]).cpu().numpy() for t in toks[5:]]
    tu.check({("r", p): row for p, row in enumerate(np.concatenate(got))}, name, {"r": toks}, dtype)
    assert engine.graphs, "decode steps ran as a graph"
    held = [sum(p >= 0 for p in pages) for pages in engine.cache.sequences["r"].pages]
    assert min(held) < 21 and max(held) <= 21
    engine.check_status()


@pytest.mark.parametrize("name", ["A", "B"])
def test_greedy_generation_through_the_service(name):
    from air_b200 import GenerationConfig
    from air_b200.engine.engine import Engine, EngineConfig
    from air_b200.engine.service import InferenceService, SchedulerConfig
    engine = Engine.from_folder(tu.model_folder(name), EngineConfig(dtype="float32", page_tokens=16, max_tokens=1024,
                                                                    max_requests=4))
    svc = InferenceService(engine, SchedulerConfig(max_active_requests=4, prefill_quantum_tokens=5,
                                                   token_budget_per_cycle=12))
    prompts = [tu.tokens_for(name, n, 40 + n) for n in (1, 7, 33, 20, 3)]
    want = [tu.plain_greedy(name, p, 12) for p in prompts]
    got = svc.generate_cohort([(p, GenerationConfig(max_new_tokens=12, stop_on_eos=False)) for p in prompts])
    assert [r.tokens for r in got] == want
    assert engine.cache.free_pages() == engine.cache.num_pages
    engine.check_status()


@pytest.mark.parametrize("page", [16, 48, 64])
@pytest.mark.parametrize("W,reader_W,R", [(70, 100, 40), (200, 131, 64), (1000, 70, 512)])
def test_latent_layers_in_portions_over_expanded_keys(W, reader_W, R, page):
    """A latent layer with heads of 128 + 64 and values of 128 and one that reads its rows through another window, alone in a
    bfloat16 engine: two requests in steps of portions that are expanded, shorter ones and single tokens, against the plain
    function on each whole sequence.  Pages go back to the pool as the windows pass; what no token was written to is NaN."""
    from air_b200.cache.manager import CacheManager
    from air_b200.config import load_config
    from air_b200.engine.batch import Entry, build_context
    from air_b200.parts import registry
    from air_b200.parts.base import Runtime
    E, eps, H = 64, 1e-5, (2, 3)
    layers = [tu.with_mlp(tu.latent(H[0], 128, 64, 128, R, W, 0.08)),
              tu.with_mlp(tu.latent(H[1], 128, 64, 128, R, reader_W, 0.1, kv_from=0))]
    cfg = tu.config(20, E, eps, 1.0, layers)
    w = {n: a.astype(np.float64) for n, a in tu.draw_tensors(cfg, R + page).items()}
    spec = registry.architecture("Tomodra").build_spec(load_config(cfg))
    rt = Runtime(torch.device(DEV), torch.bfloat16, page, status=torch.zeros(1, dtype=torch.int32, device=DEV))
    parts = []
    for i in (0, 1):
        part = registry.MIXERS.get("latent_attention")(spec.layers[i].parts["mixer"], f"l{i}.mix.")
        part.load({n: dev(a, torch.float32 if n.endswith("norm") else torch.bfloat16) for n, a in w.items()}, rt)
        assert part.expands
        parts.append(part)
    rng = np.random.default_rng(R + W)
    streams = {"a": tu.bf16(rng.normal(size=(620, E))).astype(np.float64), "b": tu.bf16(rng.normal(size=(170, E))).astype(np.float64)}
    want = {}
    for r, x in streams.items():
        at = np.arange(len(x))
        kept = plain.latent_kv(x, w, "l0.mix.", layers[0]["mixer"], eps, at)
        want[r] = [plain.latent_attention(x, w, f"l{i}.mix.", layers[i]["mixer"], eps, at, kept) for i in (0, 1)]
    cache = CacheManager([parts[0].cache_needs()], page, 64, 3, dtype=torch.bfloat16, device=DEV)
    (view,) = cache.views(0)
    view.rows.fill_(float("nan"))
    for r in ("other", "a", "b"):
        cache.open(r)
    done, expanded = {"a": 0, "b": 0}, 0
    for step in ([("a", 200)], [("b", 1), ("a", 1)], [("a", 64), ("b", 65)], [("b", 1), ("a", 129)], [("a", 33), ("b", 2)], [("b", 64)],
                 [("a", 1), ("b", 36)], [("a", 115), ("b", 1)], [("a", 77)]):
        cache.reserve(step)
        x = np.concatenate([streams[r][done[r]:done[r] + n] for r, n in step])
        ctx = build_context([Entry(r, [0] * n, []) for r, n in step], cache, DEV, status=rt.status,
                            planners=list({p.plan_key(): p for p in parts}.values()))
        expanded += len(ctx.plans[parts[0].plan_key()].expanded)
        for i, part in enumerate(parts):
            y = part.forward(dev(x, torch.bfloat16), ctx, cache.views(0), i == 0)
            y = (y.sum(0) if y.dim() == 3 else y).cpu().numpy()
            at = 0
            for r, n in step:
                ref = want[r][i][done[r]:done[r] + n]
                assert np.abs(y[at:at + n] - ref).max() < 4e-2 * max(1.0, np.abs(want[r][i]).max()), (i, step, r)
                at += n
        for r, n in step:
            cache.commit(r, n)
            done[r] += n
    assert done == {"a": 620, "b": 170} and expanded == 7 and rt.status.item() == 0
    assert max(W, reader_W) > 600 or min(cache.sequences["a"].pages[0]) == -1, "pages were given back"


@pytest.mark.parametrize("page", [16, 48, 64])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_expanded_latents_and_wide_experts_in_every_schedule(dtype, page):
    """Configuration D whole, in portions and in mixed steps: latents expanded for portions of 64 tokens and more behind windows,
    gated experts as a stream of weights with planes per part of k through the norms, also in replayed decode steps."""
    lengths = (2, 65, 230, 420, 131)
    streams = streams_for("D", 90, lengths)
    for steps, requests in ((util.trace_whole(streams), 4), (util.trace_bulk_tail(streams, tail=40), 4),
                            (util.trace_portions(streams, sizes=(100, 1, 64, 65, 2, 33, 128)), 4),
                            (util.trace_mixed(streams, seed=6, live=3, portions=(2, 70, 100, 33, 128)), 3)):
        got, _ = replay("D", dtype, steps, page_tokens=page, max_requests=requests, peak_page=192)
        tu.check(got, "D", streams, dtype)


def test_trace_runner_program_and_command_line(capsys):
    """bin/trace_run as a program on a Tomodra folder (the class is chosen by config.json), and the command line."""
    name = "B"
    streams = streams_for(name, 60, (40, 9))
    steps = util.trace_mixed(streams, seed=2, live=2)
    with tempfile.TemporaryDirectory() as out:
        util.run_trace_program(tu.model_folder(name), "float32", steps, util.peak_tokens(steps), out)
        got = util.collect(steps, out, tu.CONFIGS[name]["vocab"])
    tu.check(got, name, streams, "float32")
    from air_b200 import cli
    prompt = tu.tokens_for(name, 9, 70)
    assert cli.main(["cuda", tu.model_folder(name), ",".join(map(str, prompt)), "--tokens", "6", "--dtype", "float32",
                     "--no-stop-on-eos"]) == 0
    assert capsys.readouterr().out.strip() == ",".join(map(str, tu.plain_greedy(name, prompt, 6)))


@pytest.mark.parametrize("T,top,n,E,F", [(1, 1, 3, 64, 128), (8, 2, 16, 200, 256), (16, 3, 5, 72, 384), (17, 2, 4, 136, 128),
                                         (33, 2, 7, 264, 128), (64, 1, 2, 64, 640), (150, 2, 9, 128, 256)])
@pytest.mark.parametrize("splits", [1, 2])
def test_expert_stream_against_64_bit_products(T, top, n, E, F, splits):
    """The experts' products as a stream of weights: one to more than 64 rows per expert, experts without rows, widths that are
    not whole tiles, parts of k in planes of their own, every epilogue."""
    from air_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(T + E)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    expert = torch.argsort(torch.rand(T, n - (n > 2), generator=g, device="cuda"), dim=1)[:, :top].int().contiguous()
    if T == 150:
        expert[:, 0], expert[:, 1] = 0, 1 + torch.arange(T, device="cuda") % 3      # 150 rows of one expert
    pairs = T * top
    i32 = lambda *s: torch.empty(s, dtype=torch.int32, device="cuda")
    start, slot_pair, tiles, count = i32(n + 1), i32(pairs), i32(pairs // 64 + n, 2), i32(1)
    ops.moe_sort(expert, n, start, slot_pair, tiles, count)
    x, weight = rand(T, E).bfloat16(), torch.rand(T, top, generator=g, device="cuda")
    up, down = (rand(n, 2 * F, E) * E ** -0.5).bfloat16(), (rand(n, E, F) * F ** -0.5).bfloat16()
    rows = ops.rows_by_index(x, slot_pair, top, weight.view(-1), torch.empty(pairs, E, dtype=torch.bfloat16, device="cuda"))
    lists = (start, tiles, count, T)
    act = torch.empty(pairs, F, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.expert_stream(rows, up, act, *lists, silu_mul=True, status=status)
    if splits > 1 and (-(-F // 64) % 2 or F < 128):
        splits = 1
    y = torch.full((splits * top, T, E), 9.0, device="cuda")
    ops.expert_stream(act, down, y, *lists, o_index=slot_pair, o_div=top, splits=splits, o_scale=weight.view(-1), lists_ready=True,
                      status=status)
    plain_up = torch.empty(pairs, 2 * F, dtype=torch.bfloat16, device="cuda")
    ops.expert_stream(rows, up, plain_up, *lists, relu2=True, status=status)
    assert status.item() == 0
    for s, p in enumerate(slot_pair.tolist()):
        t, c = divmod(p, top)
        e = int(expert[t, c])
        z = up[e].double() @ rows[s].double()
        assert (plain_up[s].double() - z.clamp(min=0) ** 2).abs().max() <= 0.005 * (z ** 2).max()      # (bfloat16: 2^-8)
        z = z.view(F // 128, 2, 128)
        want = (torch.nn.functional.silu(z[:, 0]) * z[:, 1]).flatten()
        assert (act[s].double() - want).abs().max() <= 0.005 * want.abs().max()
        want = down[e].double() @ act[s].double() * weight[t, c].double()
        got = y.view(splits, top, T, E)[:, c, t].double().sum(0)
        assert (got - want).abs().max() <= 3e-6 * (down[e].double().abs() @ act[s].double().abs()).max()


@pytest.mark.parametrize("T,top,n,E,F", [(70, 2, 3, 64, 128), (127, 1, 2, 136, 256), (128, 1, 1, 72, 128), (129, 2, 3, 264, 128),
                                         (300, 2, 4, 200, 640)])
def test_expert_stream_in_wide_tiles(T, top, n, E, F):
    """Tiles of 128 slots: experts with fewer rows, just as many, one more, and several tiles; the rows' results are those of
    tiles of 64, bit for bit, in every epilogue."""
    from air_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(T + E)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    expert = torch.argsort(torch.rand(T, n, generator=g, device="cuda"), dim=1)[:, :top].int().contiguous()
    expert[:, 0] = torch.where(torch.arange(T, device="cuda") < 65, 0, expert[:, 0]) if top == 1 else expert[:, 0]
    pairs = T * top
    i32 = lambda *s: torch.empty(s, dtype=torch.int32, device="cuda")
    x, weight = rand(T, E).bfloat16(), torch.rand(T, top, generator=g, device="cuda")
    up, down = (rand(n, 2 * F, E) * E ** -0.5).bfloat16(), (rand(n, E, F) * F ** -0.5).bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    outs = []
    for tile_rows in (ops.GROUP_TILE, ops.GROUP_WIDE):
        start, slot_pair, tiles, count = i32(n + 1), i32(pairs), i32(pairs // tile_rows + n, 2), i32(1)
        ops.moe_sort(expert, n, start, slot_pair, tiles, count, tile_rows=tile_rows)
        rows = ops.rows_by_index(x, slot_pair, top, None, torch.empty(pairs, E, dtype=torch.bfloat16, device="cuda"))
        lists, kw = (start, tiles, count, T), dict(status=status, tile_rows=tile_rows)
        act, square = (torch.empty(pairs, k * F, dtype=torch.bfloat16, device="cuda") for k in (1, 2))
        y = torch.full((top, T, E), 9.0, device="cuda")
        ops.expert_stream(rows, up, square, *lists, relu2=True, **kw)
        ops.expert_stream(rows, up, act, *lists, silu_mul=True, **kw)
        ops.expert_stream(act, down, y, *lists, o_index=slot_pair, o_div=top, o_scale=weight.view(-1), lists_ready=True, **kw)
        by_pair = torch.argsort(slot_pair)          # (the order of an expert's slots is not given)
        outs.append((act[by_pair], square[by_pair], y))
        sizes = (start[1:] - start[:-1]).tolist()
        assert int(count) == sum(-(-s // tile_rows) for s in sizes)
    assert status.item() == 0
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    for t in (0, T // 2, T - 1):
        for c in range(top):
            e = int(expert[t, c])
            z = (up[e].double() @ x[t].double()).view(F // 128, 2, 128)
            want = down[e].double() @ (torch.nn.functional.silu(z[:, 0]) * z[:, 1]).flatten() * weight[t, c].double()
            assert (outs[1][2][c, t].double() - want).abs().max() <= 0.01 * want.abs().max()


@pytest.mark.parametrize("T", [1, 7, 8, 9, 24, 25, 33, 64, 65])
@pytest.mark.parametrize("H,N,K", [(3, 512, 128), (5, 128, 512), (2, 33, 1024), (4, 72, 80), (1, 31, 16), (2, 64, 272)])
def test_products_per_head_of_few_rows(H, N, K, T):
    """Matrices that are read ahead of time, rows around eights and around the lines of the dispatch, rows of W that are not whole tiles, k
    that is no whole step of 32: the bits of the grouped product, and the 64-bit product's numbers; bands of wider rows, scales."""
    from air_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(T + N)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w, scale = rand(T, H * K + 8).bfloat16(), rand(H, N, K).bfloat16(), rand(T, H + 1)
    for dtype, kw in ((torch.float32, {}), (torch.bfloat16, dict(o_scale=scale, o_scale_ld=H + 1))):
        outs = []
        for ready in (False, True):
            out = torch.full((T, H * N + 3), 9.0, device="cuda", dtype=dtype)
            ops.grouped_gemm(x, w, out, N, K, lda=H * K + 8, ldo=H * N + 3, groups=H, a_group_stride=K, o_group_stride=N, a_local=True,
                             o_local=True, rows_per_group=T, w_ready=ready, **kw)
            outs.append(out)
        assert torch.equal(*outs) and (outs[1][:, H * N:] == 9.0).all()
        want = torch.einsum("thk,hnk->thn", x[:, :H * K].view(T, H, K).double(), w.double())
        want = want * scale[:, :H, None].double() if kw else want
        most = torch.einsum("thk,hnk->thn", x[:, :H * K].view(T, H, K).double().abs(), w.double().abs()) * (scale[:, :H, None].double().abs() if kw else 1)
        # (32-bit sums of exact products, and the output's rounding to 8 bits)
        bound = K * 2.0 ** -24 * most + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0)
        assert ((outs[1][:, :H * N].view(T, H, N).double() - want).abs() <= bound).all()


@pytest.mark.parametrize("H,N,K,rows", [(160, 128, 512, (32, 33)), (128, 128, 512, (32, 48, 49)), (32, 192, 1024, (16, 32, 33)), (96, 512, 64, (16, 17)),
                                        (128, 256, 256, (16, 24, 33))])
def test_products_of_many_heads_on_either_side_of_their_line(H, N, K, rows):
    """More blocks than the SMs take at once, on both sides of the rule's lines: the grouped product's bits."""
    from air_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(H + N)
    w = torch.randn(H, N, K, generator=g, device="cuda").bfloat16()
    assert len({ops.heads_at_once(T, H, N, K) for T in rows}) == 2
    for T in rows:
        x, outs = torch.randn(T, H * K, generator=g, device="cuda").bfloat16(), []
        for ready in (False, True):
            outs.append(torch.full((T, H * N), 9.0, device="cuda"))
            ops.grouped_gemm(x, w, outs[-1], N, K, lda=H * K, ldo=H * N, groups=H, a_group_stride=K, o_group_stride=N, a_local=True, o_local=True,
                             rows_per_group=T, w_ready=ready)
        assert torch.equal(*outs)


@pytest.mark.parametrize("ready", [False, True])
def test_products_per_head_refuse_what_they_do_not_read(ready):
    """A scale of A's rows without a list of them, and tiles without their starts, are refused whether or not W was there before."""
    from air_b200.csrc import ops
    H, N, K, T = 2, 64, 128, 4
    x, w = (torch.randn(*s, device="cuda").bfloat16() for s in ((T, H * K), (H, N, K)))
    out, scale, tiles = torch.zeros(T, H * N, device="cuda"), torch.ones(T, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    for more in (dict(a_scale=scale), dict(tiles=tiles, num_tiles=tiles)):
        with pytest.raises(ops.KernelError):
            ops.grouped_gemm(x, w, out, N, K, lda=H * K, ldo=H * N, groups=H, a_group_stride=K, o_group_stride=N, a_local=True, o_local=True,
                             rows_per_group=T, w_ready=ready, **more)
    assert (out == 0).all()


@pytest.mark.parametrize("H,d,dv,P", [(16, 576, 512, 64), (32, 576, 512, 64), (40, 576, 512, 16), (3, 320, 256, 128), (17, 128, 128, 32), (20, 192, 128, 8)])
@pytest.mark.parametrize("kind", ["plain", "window", "chunk", "cap", "sink", "rising"])
def test_single_tokens_over_latents_on_the_tensor_cores(H, d, dv, P, kind):
    """Contexts around a tile's edges, from one key to more tiles than there are parts, in one batch with a padded row: against 64-bit
    attention over the seen rows, with NaN in every row of the pages that no token sees, scores that rise from tile to tile (the reference
    maximum moves), and steps captured in a graph."""
    from air_b200.csrc import ops
    contexts = [0, 62, 63, 64, 127, 128, 700, 1700, 2600]
    T, rot, scale = len(contexts) + 1, d - dv, (dv + 32) ** -0.5
    g = torch.Generator(device="cuda").manual_seed(H + d)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    need = [-(-(c + 1) // P) for c in contexts]
    order = torch.randperm(sum(need) + 3, generator=torch.Generator().manual_seed(d))
    rows = torch.full((sum(need) + 3, P, d), float("nan"), device="cuda", dtype=torch.bfloat16)
    table = torch.full((T, max(need)), -1, dtype=torch.int32)
    q, past, at = rand(T, H, d) * 1.5, [], 0
    for i, (c, k) in enumerate(zip(contexts, need)):
        table[i, :k] = order[at:at + k].int()
        at += k
        x = rand(c + 1, d)
        if kind == "rising":            # keys along the first head's query, longer and longer
            x = x * 0.2 + q[i, 0] / q[i, 0].norm() * torch.linspace(0, 60, c + 1, device="cuda")[:, None]
        past.append(x.bfloat16())
        full = torch.full((k * P, d), float("nan"), device="cuda", dtype=torch.bfloat16)
        full[:c + 1] = past[-1]
        rows[table[i, :k].long().cuda()] = full.view(k, P, d)
    window, chunk = (100 if kind == "window" else None), (96 if kind == "chunk" else None)
    if window or chunk:                 # what no token sees may hold anything, ahead of the first key too
        for i, c in enumerate(contexts):
            lo = max(0, c - window + 1) if window else c - c % chunk
            for key in range(lo):
                rows[table[i, key // P], key % P] = float("nan")
    sink = rand(H) if kind == "sink" else None
    cap = 20.0 if kind == "cap" else 0.0
    seq = torch.tensor(list(range(len(contexts))) + [-1], dtype=torch.int32, device="cuda")
    pos = torch.tensor(contexts + [0], dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.full((T, H, dv), 7.0, device="cuda", dtype=torch.bfloat16)
    table = table.cuda()
    call = lambda: ops.grouped_attention(q, rows, table, seq, pos, out, window, scale, latent=True, chunk=chunk, sink=sink, softcap=cap,
                                         status=status)
    call()
    first = out.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    out.fill_(7.0)
    graph.replay()
    torch.cuda.synchronize()
    assert status.item() == 0 and torch.equal(out, first)
    assert (out[-1] == 7.0).all(), "a padded row is not touched"
    for i, c in enumerate(contexts):
        lo = max(0, c - window + 1) if window else c - c % chunk if chunk else 0
        keys = past[i][lo:].double()
        s = q[i].double() @ keys.t() * scale
        s = cap * torch.tanh(s / cap) if cap else s
        if sink is not None:
            s = torch.cat([s, sink.double()[:, None]], dim=1)
        p = torch.softmax(s, dim=1)[:, :keys.shape[0]]
        want = p @ keys[:, :dv]
        # (the output's rounding to 8 bits, 2^-8 of a number at most; queries and weights as two such halves each, to 2^-16 of what they are
        # multiplied with)
        bound = 2.0 ** -8 * want.abs() + 2.0 ** -16 * (p @ keys[:, :dv].abs()) + 2.0 ** -16 * (q[i].double().abs() @ keys.abs().t() * scale).max() * keys.abs().max()
        assert ((first[i].double() - want).abs() <= bound).all(), (i, float(((first[i].double() - want).abs() / bound).max()))


@pytest.mark.parametrize("H,d,dv", [(16, 576, 512), (3, 320, 256), (20, 128, 128), (8, 576, 512)])
@pytest.mark.parametrize("contexts", [[0, 70, 300], [0, 5, 63, 64, 65, 200, 299, 319]])
def test_latent_queries_on_any_boundary(contexts, H, d, dv):
    """Queries that do not begin on 16 bytes take the kernels that read them by less, a batch of no token takes none."""
    from air_b200.csrc import ops
    T, P = len(contexts), 64
    g = torch.Generator(device="cuda").manual_seed(d)
    rows = torch.randn(T * 5, P, d, generator=g, device="cuda").bfloat16()
    table = torch.arange(T * 5, dtype=torch.int32, device="cuda").view(T, 5)
    seq, pos = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in (list(range(T)), contexts))
    numbers = torch.randn(T, H, d, generator=g, device="cuda")
    outs = []
    for shift in (0, 2, 1):                     # (floats: boundaries of 16, 8 and 4 bytes)
        room = torch.empty(T * H * d + 4, device="cuda")
        q = room[shift:shift + T * H * d].view(T, H, d).copy_(numbers)
        assert q.data_ptr() % 16 == 4 * shift
        out = torch.full((T, H, dv), 7.0, device="cuda", dtype=torch.bfloat16)
        ops.grouped_attention(q, rows, table, seq, pos, out, None, d ** -0.5, latent=True)
        outs.append(out.double())
    for other in outs[1:]:                      # (two roundings to 8 bits, and as two halves of 8 bits what is multiplied)
        assert ((other - outs[0]).abs() <= 2.0 ** -7 * outs[0].abs() + 2.0 ** -12).all()
    none = torch.empty((0, H, dv), device="cuda", dtype=torch.bfloat16)
    ops.grouped_attention(numbers[:0], rows, table, seq[:0], pos[:0], none, None, d ** -0.5, latent=True)


def test_a_rows_experts_do_not_depend_on_the_rows_beside_it():
    """A mixture in bfloat16: a row's planes are the same, bit for bit, in every step of up to 64 rows, and in every longer one on
    the stream of weights; their sums are those of the 64-bit experts."""
    from types import SimpleNamespace
    from air_b200.parts.base import Runtime
    from air_b200.parts.experts import RoutedExperts
    from air_b200.parts.spec import PartSpec
    n, top, E, F = 16, 2, 4096, 1024
    g = torch.Generator(device="cuda").manual_seed(8)
    rand = lambda *s: (torch.randn(*s, generator=g, device="cuda") * s[-1] ** -0.5).bfloat16()
    w = {"m.router": rand(n, E) * 4}
    for e in range(n):
        w.update({f"m.e{e}.gate": rand(F, E) * 2, f"m.e{e}.up": rand(F, E), f"m.e{e}.down": rand(E, F)})
    part = RoutedExperts(PartSpec("routed_experts", dict(hidden=E, experts=n, top=top, intermediate=F, shared_intermediate=0,
                                                         weight_on="output")), "m.")
    part.load(w, Runtime(torch.device(DEV), torch.bfloat16, 64, status=torch.zeros(1, dtype=torch.int32, device=DEV)))
    x = torch.randn(300, E, generator=g, device="cuda").bfloat16()
    z = x.double() @ w["m.router"].double().T
    kept = {}
    for T in (64, 33, 17, 8, 3, 2, 1, 300, 130, 65):
        y = part.forward(x[:T].contiguous(), SimpleNamespace(residual=None)).clone()
        first = kept.setdefault(T <= 64, y)
        assert y.shape[0] == first.shape[0] and torch.equal(y, first[:, :T]), T
        for t in {0, T - 1}:
            s, chosen = torch.sigmoid(z[t]).topk(top)
            want = 0
            for weight, e in zip(s, chosen.tolist()):
                act = torch.nn.functional.silu(w[f"m.e{e}.gate"].double() @ x[t].double()) * (w[f"m.e{e}.up"].double() @ x[t].double())
                want = want + weight * (w[f"m.e{e}.down"].double() @ act)
            # (what the activation loses in bfloat16, 2^-8 of each of 1,024 numbers, averages out in the sum)
            assert (y[:, t].double().sum(0) - want).abs().max() < 0.01 * want.abs().max(), T


@pytest.mark.parametrize("H,rot,window,n,pos0,sink", [(3, 64, None, 64, 0, False), (2, 64, None, 300, 0, True), (1, 0, None, 257, 100, True),
                                                      (2, 64, 70, 200, 333, False), (4, 0, 130, 65, 0, False),
                                                      (2, 64, None, 70, 6000, True), (2, 64, 2000, 129, 5000, False)])
def test_attention_over_expanded_latents(H, rot, window, n, pos0, sink):
    """A portion's attention over keys and values expanded from latents: tiles with remainders, a prefix, windows, the keys'
    common part, sinks, and streams of keys that are cut into segments."""
    from air_b200.csrc import ops
    from air_b200.parts.attention import plan_segments, portion_tiles
    g = torch.Generator(device="cuda").manual_seed(n + pos0)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    lo = max(0, pos0 - window + 1) // 64 * 64 if window else 0
    keys, rank, row0 = pos0 + n - lo, 40, 5
    kv, rows, q = rand(keys, H * 256), rand(keys, rank + rot), rand(row0 + n + 3, H, 128)
    q_rot = rand(row0 + n + 3, H, rot) if rot else None
    sinks = torch.randn(H, generator=g, device="cuda") * 3 if sink else None
    tiles, key_tiles = portion_tiles(n, pos0, 0, row0, window)
    cut = plan_segments(key_tiles, H)
    assert (cut is not None) == (pos0 >= 5000), "the long prefixes are cut"
    on = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    more = {} if cut is None else dict(segments=on(cut[0]), items=on(cut[1]), slots=cut[2])
    out, status = torch.full((row0 + n + 3, H, 128), 7.0, device="cuda").bfloat16(), torch.zeros(1, dtype=torch.int32, device="cuda")
    scale = (128 + rot) ** -0.5
    ops.prefill_attention_expanded(q, q_rot, kv, rows, rank, lo, on(tiles), out, window, scale, status=status, sink=sinks, **more)
    assert status.item() == 0
    assert (out[:row0] == 7).all() and (out[row0 + n:] == 7).all(), "rows outside the portion are not touched"
    position = torch.arange(pos0, pos0 + n, device="cuda")[:, None]
    key = torch.arange(lo, pos0 + n, device="cuda")[None]
    seen = (key <= position) & (key > position - window if window else True)
    for h in range(H):
        k, v = kv[:, h * 256:h * 256 + 128].double(), kv[:, h * 256 + 128:(h + 1) * 256].double()
        s = q[row0:row0 + n, h].double() @ k.t()
        if rot:
            s += q_rot[row0:row0 + n, h].double() @ rows[:, rank:].double().t()
        s = (s * scale).masked_fill(~seen, -float("inf"))
        if sink:
            s = torch.cat([s, sinks[h].double().expand(n, 1)], dim=1)
            v = torch.cat([v, torch.zeros(1, 128, dtype=torch.float64, device="cuda")])
        want = torch.softmax(s, dim=1) @ v
        # (the weights are rounded to bfloat16 and so is the result: 2^-8 of sums of values of unit size)
        assert (out[row0:row0 + n, h].double() - want).abs().max() < 0.01 * max(1.0, want.abs().max().item()), h
