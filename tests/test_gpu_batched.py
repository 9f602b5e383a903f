"""GPU parity of the batched path (token permute + grouped GEMM + un-permute combine)."""
import numpy as np
import pytest

from moe4all_b200 import DType, MoeGating, synth
from oracle import oracle as orc

from helpers import GpuLayer, assert_close, near_tie_rows, oracle_layer

pytestmark = pytest.mark.gpu


def ids_match(ids, ref, n_used):
    ties = set(near_tie_rows(ref, n_used).tolist())
    bad = [r for r in range(ids.shape[0]) if r not in ties and ids[r].tolist() != ref.ids[r].tolist()]
    assert not bad, f"rows with different expert ids: {bad[:5]}"
    assert len(ties) <= max(2, ids.shape[0] // 50)
    return ties


# path 2 = tcgen05 tiles where the shape allows, path 3 = the legacy mma.sync tiles
@pytest.mark.parametrize("path", [2, 3])
@pytest.mark.parametrize("rows", [1, 5, 64, 200, 700])
def test_batched_small_layer(backend, rows, path):
    L = synth.make_layer(41, 512, 16, 256, sh_ff=256, router_std=0.05)
    x = synth.activations(rows, rows, 512)
    out, ids, wts = GpuLayer(backend, L).run(x, 4, path=path)
    ref = oracle_layer(L, x, 4)
    ties = ids_match(ids, ref, 4)
    keep = [r for r in range(rows) if r not in ties]
    np.testing.assert_allclose(wts[keep], ref.wts[keep], rtol=2e-6, atol=1e-9)
    assert_close(out[keep], ref.dst[keep])


def test_auto_path_switches_to_grouped_gemm(backend):
    # 48 tokens x 4 over 16 experts = 12 tokens per expert: past the small-m kernels' range (11 per expert)
    L = synth.make_layer(42, 512, 16, 256, router_std=0.05)
    x = synth.activations(1, 48, 512)
    g = GpuLayer(backend, L)
    n0 = backend.launch_count()
    out, ids, _ = g.run(x, 4)
    assert backend.launch_count() - n0 > 5  # neither the three per-pair kernels nor the five expert-major ones
    ref = oracle_layer(L, x, 4)
    ids_match(ids, ref, 4)
    assert_close(out, ref.dst)


@pytest.mark.parametrize("path", [2, 3])
def test_skewed_load_and_empty_experts(backend, path):
    # a router bias column (router_x differs from x, crates/infr-core/src/graph.rs:1261-1266) gives a
    # Zipf(1.1)-like load: a few experts get hundreds of rows, many get none
    ne, E, rows = 512, 64, 600
    L = synth.make_layer(43, ne, E, 256, sh_ff=256, router_std=0.02)
    rank = np.random.default_rng(0).permutation(E) + 1
    L.router[:, ne - 1] = (-1.1 * np.log(rank)).astype(np.float32)
    x = synth.activations(7, rows, ne)
    rx = x.copy()
    rx[:, ne - 1] = 1.0
    out, ids, wts = GpuLayer(backend, L).run(x, 4, router_x=rx, path=path)
    ref = oracle_layer(L, x, 4, router_x=rx)
    counts = np.bincount(ref.ids.reshape(-1), minlength=E)
    assert counts.max() > 300 and (counts == 0).sum() > 0, "the case must have a hot and an empty expert"
    ties = ids_match(ids, ref, 4)
    keep = [r for r in range(rows) if r not in ties]
    assert_close(out[keep], ref.dst[keep])


def test_grouped_sigmoid_bias_batched(backend):
    L = synth.make_layer(44, 512, 32, 256, sh_ff=256, gated_shared=False, bias_std=0.05, router_std=0.05)
    x = synth.activations(3, 96, 512)
    kw = dict(scale=2.5, gating=MoeGating.Sigmoid, groups=8, groups_used=4)
    out, ids, wts = GpuLayer(backend, L).run(x, 6, path=2, **kw)
    ref = oracle_layer(L, x, 6, **kw)
    ties = ids_match(ids, ref, 6)
    keep = [r for r in range(96) if r not in ties]
    assert_close(out[keep], ref.dst[keep])


def test_batched_ep_bands_sum_to_full(backend):
    L = synth.make_layer(45, 512, 32, 256, router_std=0.05)
    x = synth.activations(5, 100, 512)
    g = GpuLayer(backend, L)
    full, _, _ = g.run(x, 4, path=2)
    parts = [g.run(x, 4, path=2, ep_band=(lo, 8))[0] for lo in range(0, 32, 8)]
    assert_close(sum(parts), full, tol=1e-5)
    assert_close(parts[1], oracle_layer(L, x, 4, ep_band=(8, 8)).dst)


def test_q4k_down_banks_batched(backend):
    L = synth.make_layer(62, 1024, 16, 512, sh_ff=512, down_q4k=True, router_std=0.05)
    x = synth.activations(23, 300, 1024)
    out, ids, wts = GpuLayer(backend, L).run(x, 4, path=2)
    ref = oracle_layer(L, x, 4)
    ties = ids_match(ids, ref, 4)
    keep = [r for r in range(300) if r not in ties]
    assert_close(out[keep], ref.dst[keep])
    with pytest.raises(Exception):
        GpuLayer(backend, L).run(x, 4, path=3)  # the legacy tiles have no Q4_K down kernel


@pytest.mark.parametrize("path", [1, 2])
def test_deepseek_v3_dims(backend, path):
    # hidden 7168, expert intermediate 2048, sigmoid gating with 8 groups / 4 used, scale 2.5,
    # ungated shared expert; 16 experts keep the oracle quick.  64 rows is the decode batch of the
    # largest configuration, served by the small-m kernels (path 1) or the grouped GEMMs (path 2).
    L = synth.make_layer(51, 7168, 16, 2048, sh_ff=2048, gated_shared=False, bias_std=0.02)
    x = synth.activations(8, 64, 7168)
    kw = dict(scale=2.5, gating=MoeGating.Sigmoid, groups=8, groups_used=4)
    out, ids, wts = GpuLayer(backend, L).run(x, 4, path=path, **kw)
    ref = oracle_layer(L, x, 4, **kw)
    ties = ids_match(ids, ref, 4)
    keep = [r for r in range(64) if r not in ties]
    assert len(keep) > 56
    assert_close(out[keep], ref.dst[keep])


@pytest.mark.parametrize("rows,path", [(4, 1), (20, 1), (100, 2)])
def test_routing_from_outside_with_foreign_pairs(backend, rows, path):
    # what an expert-parallel rank runs: ids and weights are inputs (stages 2 + 4 + 8), pairs of
    # other ranks carry a negative id and contribute nothing
    from moe4all_b200 import MoeFfn
    L = synth.make_layer(47, 512, 32, 256, router_std=0.05)
    x = synth.activations(6, rows, 512)
    g = GpuLayer(backend, L)
    want, ids, wts = g.run(x, 4, path=path, ep_band=(8, 16))
    local = np.where((ids >= 8) & (ids < 24), ids, -1).astype(np.int32)
    be = backend
    dst = be.alloc(rows * 512 * 4)
    op = MoeFfn(x=be.from_host(x), router=g.router, gate_exps=g.gate, up_exps=g.up, down_exps=g.down, dst=dst, rows=rows, ne=512,
                n_expert=32, n_used=4, n_ff_exp=256, ids_out=be.from_host(local), wts_out=be.from_host(wts), stages=14, path=path)
    be.moe_ffn(op)
    be.sync()
    got = be.download(dst, np.float32).reshape(rows, 512)
    assert np.array_equal(got, want)
    assert_close(got, oracle_layer(L, x, 4, ep_band=(8, 16)).dst)


def test_config1_shape_512_rows(backend):
    # the Qwen3.6-35B-A3B layer shape with a 512-token chunk
    L = synth.make_layer(46, 2048, 256, 512, sh_ff=512)
    x = synth.activations(9, 512, 2048)
    out, ids, wts = GpuLayer(backend, L).run(x, 8, path=2)
    ref = oracle_layer(L, x, 8)
    ties = ids_match(ids, ref, 8)
    keep = [r for r in range(512) if r not in ties]
    assert_close(out[keep], ref.dst[keep])


def test_batched_rows_equal_decode_rows(backend):
    # size-independent property for the full 4096-token prefill: any row of the batched result
    # equals the same row pushed through the (oracle-checked) decode kernels alone
    L = synth.make_layer(47, 2048, 256, 512, sh_ff=512)
    x = synth.activations(10, 4096, 2048)
    g = GpuLayer(backend, L)
    out, ids, _ = g.run(x, 8, path=2)
    pick = np.random.default_rng(1).choice(4096, size=24, replace=False)
    for r0 in range(0, 24, 8):
        rows = pick[r0:r0 + 8]
        o2, i2, _ = g.run(x[rows], 8, path=1)
        assert np.array_equal(i2, ids[rows])
        assert_close(out[rows], o2, tol=1e-3)


def test_expert_rows_building_block(backend):
    # rows already grouped by local expert (what a rank runs between dispatch and combine)
    be = backend
    ne, nff, n_local = 512, 256, 4
    L = synth.make_layer(48, ne, n_local, nff)
    counts = [70, 0, 1, 130]
    seg = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    n_rows = int(seg[-1])
    x = synth.activations(11, n_rows, ne)
    yb = be.alloc(n_rows * ne * 4)
    gate, up, down = be.from_host(L.gate), be.from_host(L.up), be.from_host(L.down)
    be.moe_expert_rows(be.from_host(x), be.from_host(seg), gate, up, down, yb, n_rows, n_local, ne, nff)
    got = be.download(yb, np.float32).reshape(n_rows, ne)
    gb, db = nff * DType.Q4K.row_bytes(ne), ne * DType.Q6K.row_bytes(nff)
    want = np.zeros_like(got)
    for e in range(n_local):
        a, b = seg[e], seg[e + 1]
        if a == b:
            continue
        g_ = orc.linear(orc.DT_Q4K, L.gate[e * gb:(e + 1) * gb], x[a:b], nff)
        u_ = orc.linear(orc.DT_Q4K, L.up[e * gb:(e + 1) * gb], x[a:b], nff)
        want[a:b] = orc.linear(orc.DT_Q6K, L.down[e * db:(e + 1) * db], orc.gated_act_silu(g_, u_), ne)
    assert_close(got, want)


def test_many_pairs(backend):
    # past 65536 (token, expert) pairs the bucketing runs as count / scan / scatter kernels instead of
    # the single-CTA form
    L = synth.make_layer(43, 256, 16, 256, router_std=0.05)
    rows = 8300
    x = synth.activations(5, rows, 256)
    out, ids, wts = GpuLayer(backend, L).run(x, 8, path=2)
    ref = oracle_layer(L, x, 8)
    ties = ids_match(ids, ref, 8)
    keep = [r for r in range(rows) if r not in ties]
    assert_close(out[keep], ref.dst[keep])


@pytest.mark.parametrize("mix", [(12, 12, 14), (13, 13, 12), (8, 8, 8), (14, 12, 13)])
def test_phase_stamps_of_one_tile(backend, mix):
    # with a trace buffer set, the tcgen05 kernels stamp the phases of the chosen tile and compute what they do without
    be = backend
    L = synth.make_layer(63, 512, 8, 512, router_std=0.05, dtypes=mix)
    x = synth.activations(24, 400, 512)
    g = GpuLayer(be, L)
    want, _, _ = g.run(x, 2, path=2)
    for tile, there in ((0, True), (3, True), (4096, False)):
        buf = be.alloc(4096)
        be.set_trace(buf)
        be.set_config(trace_tile=tile)
        try:
            out, _, _ = g.run(x, 2, path=2)
        finally:
            be.set_trace(None)
            be.set_config(trace_tile=0)
        assert np.array_equal(out, want)
        ns = be.download(buf, np.uint64).reshape(256, 2)[:, 0].astype(np.int64)
        if not there:
            assert not ns[40:48].any() and not ns[64:192].any()
            continue
        assert (ns[40:48] > 0).all() and (np.diff(ns[40:44]) >= 0).all() and (np.diff(ns[44:48]) >= 0).all()
        # 512 inputs are eight K steps: four of the first producer warp, eight issued by the MMA warp
        for k in (64, 128):
            assert (ns[k : k + 16] > 0).all() and (np.diff(ns[k : k + 16]) >= 0).all() and not ns[k + 16 : k + 32].any()
            assert (ns[k + 32 : k + 48] > 0).all() and (np.diff(ns[k + 32 : k + 48]) >= 0).all() and not ns[k + 48 : k + 64].any()


@pytest.mark.parametrize("bits", [0x7C00, 0xFC00, 0x7E00, 0xFFFF], ids=["inf", "-inf", "nan", "-nan"])
@pytest.mark.parametrize("q4k", [False, True])
def test_outputs_that_are_not_finite_stay_so_between_down_and_combine(backend, bits, q4k):
    # a scale that is not finite in one block of the down banks: the rows packed for the combine kernel keep that, in that feature only
    L = synth.make_layer(46, 512, 8, 256, down_q4k=q4k, router_std=0.05)
    block, at = (144, 0) if q4k else (210, 208)
    bank = L.down.reshape(8, 512, block)
    bank[:, 77, at], bank[:, 77, at + 1] = bits & 0xFF, bits >> 8
    x = synth.activations(9, 96, 512)
    out, _, _ = GpuLayer(backend, L).run(x, 8, path=2)  # every expert serves every row
    assert not np.isfinite(out[:, 77]).any()
    assert np.isfinite(np.delete(out, 77, axis=1)).all()
