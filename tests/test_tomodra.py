"""Tomodra without a GPU: its configuration and description, the cache manager's handling of chunks and of a latent
that several layers read, and the plain implementation's mechanisms against closed forms written here."""
import json

import numpy as np
import pytest

import tomodra_util as tu
from plain import tomodra_plain as plain


def test_config_round_trip_and_description():
    from air_b200.config import load_config, ConfigError
    from air_b200.parts import registry
    from air_b200.engine.model import Model
    for name, cfg in tu.CONFIGS.items():
        c = load_config(cfg)
        assert c.architecture == "Tomodra" and c.width == cfg["width"] and len(c.layers) == len(cfg["layers"])
        assert load_config(c.to_dict()) == c
        model = Model(registry.architecture(c.architecture).build_spec(c))
        names = {t.name: tuple(t.shape) for t in model.tensor_specs() if not t.optional}
        assert {n: a.shape for n, a in tu.draw_tensors(cfg, 0).items()} == names
    with pytest.raises(ConfigError):
        load_config(dict(tu.CONFIGS["B"], layers=[dict(type="conv", mixer={})]))
    with pytest.raises(ConfigError):
        load_config({k: v for k, v in tu.CONFIGS["B"].items() if k != "postln_alpha"})
    bad = json.loads(json.dumps(tu.CONFIGS["A"]))
    bad["layers"][2]["mixer"]["kv_from"] = 1            # layer 1 is no latent layer
    with pytest.raises(ConfigError):
        load_config(bad)
    bad = json.loads(json.dumps(tu.CONFIGS["A"]))
    bad["layers"][2]["mixer"]["kv_rank"] = 48           # the reader's latent must have the owner's size
    with pytest.raises(ConfigError):
        load_config(bad)
    bad = json.loads(json.dumps(tu.CONFIGS["A"]))
    bad["layers"][0]["mlp"]["router"]["top"] = 6        # of five experts
    with pytest.raises(ConfigError):
        load_config(bad)


def test_runs_that_read_another_layers_latent_and_how_long_pages_live():
    from air_b200.config import load_config
    from air_b200.parts import registry
    from air_b200.engine.model import Model
    from air_b200.parts.base import PagedKV, PagedLatent
    c = load_config(tu.CONFIGS["A"])
    spec = registry.architecture(c.architecture).build_spec(c)
    assert [r.cache_from for r in spec.order] == [None, None, 0, None, None]
    needs = Model(spec).cache_needs()
    # layer 0 looks back 48 tokens, layer 2 reads the same rows through a window of 70: the rows live for 70
    assert needs[0] == (PagedLatent(48, 70),) and needs[2] == ()
    assert needs[1] == (PagedKV(2, 32, None, 16, 40),) and needs[3] == (PagedLatent(28, 17),)
    assert "feed_forward" not in spec.layers[2].parts and "feed_forward_norm" not in spec.layers[2].parts
    assert spec.layers[3].parts["feed_forward"]["shared_intermediate"] == 0
    # a chunk's pages go back once the request has left the chunk; a window's as it passes
    assert PagedKV(2, 32, None, 16, 40).first_live(79) == 40 and PagedKV(2, 32, None, 16, 40).first_live(80) == 80
    assert PagedLatent(48, 70).first_live(100) == 31 and PagedLatent(48, None).first_live(100) == 0


def test_cache_gives_back_the_pages_of_chunks_that_are_over():
    from air_b200.cache.manager import CacheManager
    from air_b200.parts.base import PagedKV, PagedLatent
    m = CacheManager([(PagedKV(1, 16, None, None, 40),), (PagedLatent(24, 20),)], 16, 12, 2, allocate=False)
    m.open("r")
    for n in (30, 9, 1, 45, 3):          # lengths 30, 39, 40, 85, 88
        m.reserve([("r", n)])
        m.commit("r", n)
        length = m.length("r")
        chunk_pages, window_pages = m.sequences["r"].pages
        first_chunk = (length - length % 40) // 16
        assert all((p < 0) == (b < first_chunk) for b, p in enumerate(chunk_pages)), (length, chunk_pages)
        first_window = max(0, length - 19) // 16
        assert all((p < 0) == (b < first_window) for b, p in enumerate(window_pages)), (length, window_pages)
        m.check()
    m.close("r")
    assert m.free_pages() == 12


def test_stretched_frequencies_match_the_plain_rule():
    from air_b200.parts.rope import bent_frequencies
    for dims, base, sc in ((64, 10000.0, (8.0, 1024, 32.0, 1.0)), (16, 5000.0, (4.0, 64, 16.0, 2.0)),
                           (8, 1e5, (16.0, 32, 8.0, 1.0)), (12, 1e4, None), (48, 500.0, (2.0, 4096, 1.0, 1.0))):
        scaling = dict(zip(("factor", "original", "fast", "slow"), sc)) if sc else None
        f, mag = bent_frequencies(dims, base, scaling)
        want, want_mag = plain.yarn_frequencies(dims, base, scaling)
        assert np.abs(f.numpy() - want).max() <= 1e-15 * want.max() and abs(mag - want_mag) < 1e-15
    f, _ = plain.yarn_frequencies(64, 10000.0, dict(factor=8.0, original=1024, fast=32.0, slow=1.0))
    g = plain.plain_frequencies(64, 10000.0)
    assert f[0] == g[0] and abs(f[-1] - g[-1] / 8.0) < 1e-18 and np.all(np.diff(f / g) <= 1e-12)


def test_plain_mechanisms_against_closed_forms():
    rng = np.random.default_rng(0)
    # a rotation by the key's angle and back: q.k depends on the distance only, for both pairings
    x, y = rng.normal(size=(1, 1, 8)), rng.normal(size=(1, 1, 8))
    f = plain.plain_frequencies(6, 100.0)
    for rotate in (plain.rotate_half_split, plain.rotate_neighbours):
        a = (rotate(x, np.array([7]), f, 6) * rotate(y, np.array([3]), f, 6)).sum()
        b = (rotate(x, np.array([104]), f, 6) * rotate(y, np.array([100]), f, 6)).sum()
        assert abs(a - b) < 1e-9
        assert np.array_equal(rotate(x, np.array([5]), f, 6)[..., 6:], x[..., 6:])        # the rest passes
    assert plain.rotate_neighbours(np.array([[[1.0, 0.0]]]), np.array([1]), np.array([np.pi / 2]), 2)[0, 0, 1] == pytest.approx(1.0)
    # masks
    w, c = plain.window_mask(10, 3), plain.chunk_mask(10, 4)
    assert w[5].tolist() == [False] * 3 + [True] * 3 + [False] * 4 and c[5].tolist() == [False] * 4 + [True] * 2 + [False] * 4
    assert c[4].sum() == 1 and c[7].sum() == 4 and w[0].sum() == 1
    # a sink as large as the only score takes half of the weight
    p = plain.masked_softmax(np.full((1, 1, 1), 2.0), np.ones((1, 1), dtype=bool), sink=np.array([2.0]))
    assert p[0, 0, 0] == pytest.approx(0.5)
    # the weight goes into the expert, not behind it
    w = {"e0.gate": rng.normal(size=(5, 4)), "e0.up": rng.normal(size=(5, 4)), "e0.down": rng.normal(size=(4, 5)),
         "router": np.array([[10.0, 0, 0, 0]])}
    u = np.array([[0.05, 1.0, -2.0, 0.5]])
    s = plain.sigmoid(0.5)
    y = plain.mixture(u, w, "", dict(router=dict(experts=1, top=1)))
    assert np.allclose(y, plain.expert(s * u, w, "e0.")) and not np.allclose(y, s * plain.expert(u, w, "e0."))


@pytest.mark.parametrize("page", [16, 32, 48, 64, 128])
@pytest.mark.parametrize("window", [70, 1000, 4096])
def test_an_expanded_portion_reads_pages_that_the_request_still_holds(window, page, monkeypatch):
    """Portions of latent layers with a window behind every remainder of a tile of 64 keys: what is gathered from the pages
    lies in blocks that the cache has not taken back, and the rows ahead of it are filled up to the tile."""
    from types import SimpleNamespace
    import torch
    from air_b200.cache.manager import CacheManager
    from air_b200.csrc import ops
    from air_b200.parts.base import HostBatch, Runtime
    from air_b200.parts.latent_attention import LatentAttention
    from air_b200.parts.spec import PartSpec
    n, R = 100, 8
    part = LatentAttention(PartSpec("latent_attention", {
        "hidden": 16, "heads": 1, "head_dim": 128, "rot_dim": 0, "v_dim": 128, "kv_rank": R, "scale": 0.1, "window": window}), "m.")
    part.rt, part.expansion = Runtime(device=torch.device("cpu"), dtype=torch.bfloat16, page_tokens=page), (torch.zeros(256, R).bfloat16(),)
    gathered = []
    monkeypatch.setattr(ops, "gather_keys", lambda cache, table, lo, count, rows, *a, ahead=0, **k: gathered.append((lo, ahead, count)))
    monkeypatch.setattr(ops, "prefill_attention_expanded", lambda *a, **k: None)
    cache = CacheManager([part.cache_needs()], page, 400, 1, allocate=False)
    seq = cache.open("r")
    for behind in (4990, 10) + (1,) * 66:
        cache.reserve([("r", behind)])
        cache.commit("r", behind)
        cache.reserve([("r", n)])                       # the portion's own pages
        pos0 = seq.length
        plan = part.plan(HostBatch(counts=[n], lengths=[pos0], slots=[0], q_start=[0, n]))
        assert len(plan.values["expanded"]) == 1
        part._attend_expanded(SimpleNamespace(**plan.values, **{k: None for k in plan.arrays}), torch.zeros(n, 1, 128), None,
                              SimpleNamespace(rows=None), [None], SimpleNamespace(status=None), None)
        lo, ahead, count = gathered.pop()
        first = max(0, pos0 - window + 1)
        assert lo % 64 == 0 and lo <= first < lo + 64 and lo + count == pos0 + n
        assert lo + ahead <= first, "every key that a query sees is gathered"
        assert all(seq.pages[0][key // page] >= 0 for key in range(lo + ahead, lo + count)), (pos0, lo, ahead)
        cache.trim("r")


@pytest.mark.parametrize("experts", [2, 16, 128])
def test_where_the_library_takes_the_experts_products(experts):
    """The stream of weights holds about as many rows per expert (in the mean) as a tile has slots; where it does not take the sizes, the
    library begins at half of that."""
    from air_b200.csrc import ops
    from air_b200.parts.experts import RoutedExperts
    from air_b200.parts.spec import PartSpec
    part = RoutedExperts(PartSpec("routed_experts", dict(hidden=64, experts=experts, top=2, intermediate=128)))
    at = ops.GROUP_WIDE * experts
    assert [part._for_the_library(p, True) for p in (1, at - 1, at, at + at // 32)] == [False, False, False, True]
    assert [part._for_the_library(p, False) for p in (1, at // 2 - 1, at // 2)] == [False, False, True]
