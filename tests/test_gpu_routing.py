"""Routing of decode-sized calls against the oracle where the selection can go wrong: expert counts at the edges of the lanes'
shares, every number of rows a CTA routes, ties, groups, selections made by the caller, and shapes the team form does not take."""
import numpy as np
import pytest

from helpers import near_tie_rows
from moe4all_b200 import MoeFfn, MoeGating
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
NE = 256


def route(be, x, router, k, *, bias=None, gating=0, groups=0, groups_used=0, norm_w=True, scale=1.0, given=None):
    rows, E = x.shape[0], router.shape[0]
    ids, wts = be.alloc(rows * k * 4), be.alloc(rows * k * 4)
    g = be.from_host(np.ascontiguousarray(given, np.int32)) if given is not None else None
    b = be.from_host(bias) if bias is not None else None
    be.moe_route(MoeFfn(x=be.from_host(x), router=be.from_host(router), gate_exps=None, up_exps=None, down_exps=None, dst=None, rows=rows, ne=x.shape[1],
                        n_expert=E, n_used=k, n_ff_exp=256, gating=MoeGating(gating), norm_w=norm_w, scale=scale, exp_probs_b=b,
                        n_expert_groups=groups, n_expert_groups_used=groups_used, ids_out=ids, wts_out=wts, expert_ids=g))
    be.sync()
    return be.download(ids, np.int32).reshape(rows, k), be.download(wts, np.float32).reshape(rows, k)


def reference(x, router, k, *, bias=None, gating=0, groups=0, groups_used=0, norm_w=True, scale=1.0, given=None):
    E = router.shape[0]
    ne = x.shape[1]
    z = np.zeros(E * ne * 144, np.uint8)  # expert blocks of zeros: only ids, weights and scores are looked at
    return orc.moe_ffn(x, router, z, z, np.zeros(E * ne * 210, np.uint8), n_expert=E, n_used=k, n_ff_exp=256, gating=gating, bias=bias, groups=groups,
                       groups_used=groups_used, norm_w=norm_w, scale=scale, expert_ids=given)


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 8, 9, 21])  # from nine on: a selecting CTA per row, or one per eight
@pytest.mark.parametrize("E,k,gating,groups,used,bias", [
    (4, 1, 0, 0, 0, False), (8, 8, 0, 0, 0, False), (36, 6, 1, 0, 0, True), (100, 8, 0, 0, 0, False), (128, 8, 0, 0, 0, False),
    (130, 8, 0, 0, 0, False),                                   # not a multiple of four: the general form
    (132, 8, 2, 0, 0, True), (256, 8, 0, 0, 0, False), (256, 9, 0, 0, 0, False), (256, 8, 1, 8, 4, True), (256, 8, 1, 2, 1, True),
    (128, 8, 1, 16, 5, True), (256, 2, 0, 32, 3, False), (64, 4, 1, 32, 7, True), (260, 8, 0, 0, 0, False), (252, 6, 1, 3, 2, True)])
def test_selection(backend, rows, E, k, gating, groups, used, bias):
    rng = np.random.default_rng(E * 31 + rows)
    x = rng.standard_normal((rows, NE)).astype(np.float32)
    router = (rng.standard_normal((E, NE)) * 0.1).astype(np.float32)
    kw = dict(bias=(rng.standard_normal(E) * 0.05).astype(np.float32) if bias else None, gating=gating, groups=groups, groups_used=used, scale=1.5)
    ids, wts = route(backend, x, router, k, **kw)
    ref = reference(x, router, k, **kw)
    tied = near_tie_rows(ref, k)
    same = (ids == ref.ids).all(axis=1)
    assert set(np.where(~same)[0]) <= set(tied), (ids, ref.ids)
    # the same operations on the same logits: only the last bit of exp can differ
    np.testing.assert_allclose(wts[same], ref.wts[same], rtol=1e-6)


@pytest.mark.parametrize("rows", [3, 4, 7])
@pytest.mark.parametrize("groups,used", [(0, 0), (2, 1), (4, 2)])
def test_groups_of_rows_of_unlike_sizes(backend, rows, groups, used):
    # three rows of 10240 fit a CTA, so four and seven leave one for the last group: teams of two warps and of four; with two expert
    # groups of 64 the larger team's lanes hold too few of them, and neither group of rows goes to teams
    rng = np.random.default_rng(rows * 7 + groups)
    x = rng.standard_normal((rows, 10240)).astype(np.float32)
    router = (rng.standard_normal((128, 10240)) * 0.02).astype(np.float32)
    kw = dict(gating=1, groups=groups, groups_used=used)
    ids, wts = route(backend, x, router, 8, **kw)
    ref = reference(x, router, 8, **kw)
    same = (ids == ref.ids).all(axis=1)
    assert set(np.where(~same)[0]) <= set(near_tie_rows(ref, 8)), (ids, ref.ids)
    np.testing.assert_allclose(wts[same], ref.wts[same], rtol=1e-6)


@pytest.mark.parametrize("rows", [1, 2, 4, 8])
@pytest.mark.parametrize("E", [32, 128, 256])
def test_ties_take_the_lower_index(backend, rows, E):
    rng = np.random.default_rng(E + rows)
    x = rng.standard_normal((rows, NE)).astype(np.float32)
    base = (rng.standard_normal((4, NE)) * 0.1).astype(np.float32)
    router = np.ascontiguousarray(base[np.arange(E) % 4])  # equal logits throughout: E / 4 experts share each score
    ids, _ = route(backend, x, router, 8)
    ref = reference(x, router, 8)
    assert np.array_equal(ids, ref.ids)


@pytest.mark.parametrize("rows", [1, 3])
def test_given_selection_and_plain_weights(backend, rows):
    rng = np.random.default_rng(rows)
    x = rng.standard_normal((rows, NE)).astype(np.float32)
    router = (rng.standard_normal((128, NE)) * 0.1).astype(np.float32)
    given = np.stack([rng.permutation(128)[:6] for _ in range(rows)]).astype(np.int32)
    for norm_w in (True, False):
        ids, wts = route(backend, x, router, 6, given=given, norm_w=norm_w, scale=0.5)
        ref = reference(x, router, 6, given=given, norm_w=norm_w, scale=0.5)
        assert np.array_equal(ids, given)
        np.testing.assert_allclose(wts, ref.wts, rtol=1e-6)


@pytest.mark.parametrize("ne,rows", [(256, 3), (768, 8), (1024, 8), (1280, 5), (2048, 1), (2048, 4), (2048, 5), (2304, 3), (4096, 2), (4096, 3),
                                     (4352, 2), (7168, 3)])
def test_rows_normed_in_the_router(backend, ne, rows):
    # every share of a row per thread and every remainder of rows per pass; the ids are those of the oracle on normed rows
    from helpers import assert_close
    from moe4all_b200 import synth
    L = synth.make_layer(ne + rows, ne, 16, 256, router_std=0.05)
    rng = np.random.default_rng(ne)
    x = (rng.standard_normal((rows, ne)) * rng.uniform(0.1, 10.0, (rows, 1))).astype(np.float32)
    nw = (1.0 + 0.1 * rng.standard_normal(ne)).astype(np.float32)
    b = {n: backend.from_host(getattr(L, n)) for n in ("router", "gate", "up", "down")}
    dst, ids = backend.alloc(rows * ne * 4), backend.alloc(rows * 4 * 4)
    backend.moe_ffn(MoeFfn(x=backend.from_host(x), dst=dst, norm_weight=backend.from_host(nw), norm_eps=1e-6, router=b["router"], gate_exps=b["gate"],
                           up_exps=b["up"], down_exps=b["down"], rows=rows, ne=ne, n_expert=16, n_used=4, n_ff_exp=256, ids_out=ids, path=1))
    backend.sync()
    ref = orc.moe_ffn(orc.rmsnorm(x, nw, 1e-6), L.router, L.gate, L.up, L.down, n_expert=16, n_used=4, n_ff_exp=256)
    keep = np.setdiff1d(np.arange(rows), near_tie_rows(ref, 4, ulps=64))  # the norm's own rounding moves a score by some ulps
    assert len(keep) >= rows - 1
    assert np.array_equal(backend.download(ids, np.int32).reshape(rows, 4)[keep], ref.ids[keep])
    assert_close(backend.download(dst, np.float32).reshape(rows, ne)[keep], ref.dst[keep])


@pytest.mark.parametrize("ne", [256, 768])
@pytest.mark.parametrize("rows,E", [(65, 40), (65, 256), (300, 256), (500, 256), (640, 256), (777, 256), (900, 250), (1024, 256), (1300, 256), (1700, 256),
                                    (2368, 256), (3000, 96), (3001, 130), (4100, 256)])
def test_tiles_of_batched_calls(backend, rows, E, ne):
    # every tile that prompts take (16 to 64 rows by 32 or 64 experts), ragged in rows and experts, four and twelve copies along k
    rng = np.random.default_rng(rows + E)
    x = rng.standard_normal((rows, ne)).astype(np.float32)
    router = (rng.standard_normal((E, ne)) * 0.1).astype(np.float32)
    ids, wts = route(backend, x, router, 8)
    at = np.unique(np.r_[0:16, rows // 2 : rows // 2 + 16, rows - 24 : rows])
    ref = reference(np.ascontiguousarray(x[at]), router, 8)
    same = (ids[at] == ref.ids).all(axis=1)
    assert set(np.where(~same)[0]) <= set(near_tie_rows(ref, 8))
    np.testing.assert_allclose(wts[at][same], ref.wts[same], rtol=1e-6)


@pytest.mark.parametrize("rows,E", [(4705, 160), (4705, 131)])
@pytest.mark.parametrize("ne", [256, 768])
def test_tile_of_32_rows_by_64_experts(backend, rows, E, ne):
    # the smallest of the wide tiles, which the counts above do not reach: whole and ragged in experts
    rng = np.random.default_rng(rows + E)
    x = rng.standard_normal((rows, ne)).astype(np.float32)
    router = (rng.standard_normal((E, ne)) * 0.1).astype(np.float32)
    ids, wts = route(backend, x, router, 8)
    at = np.unique(np.r_[0:16, rows // 2 : rows // 2 + 16, rows - 24 : rows])
    ref = reference(np.ascontiguousarray(x[at]), router, 8)
    same = (ids[at] == ref.ids).all(axis=1)
    assert set(np.where(~same)[0]) <= set(near_tie_rows(ref, 8))
    np.testing.assert_allclose(wts[at][same], ref.wts[same], rtol=1e-6)
