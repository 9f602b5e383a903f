"""Sizes at which the tiles of the batched and expert-major kernels begin, end and split, against the CPU oracle."""
import numpy as np
import pytest

from moe4all_b200 import synth

from helpers import GpuLayer, assert_close, near_tie_rows, oracle_layer

pytestmark = pytest.mark.gpu

Q8_0, Q4K, Q5K, Q6K = 8, 12, 13, 14


def ids_of(counts, seed):
    """One expert id per row, experts in mixed order, expert e chosen counts[e] times."""
    return np.random.default_rng(seed).permutation(np.repeat(np.arange(len(counts), dtype=np.int32), counts)).reshape(-1, 1)


@pytest.mark.parametrize("mix", [(Q4K, Q4K, Q6K), (Q5K, Q5K, Q4K), (Q8_0, Q8_0, Q8_0), (Q6K, Q4K, Q5K)])
@pytest.mark.parametrize("ne,nff", [(512, 256), (768, 768)])
def test_grouped_token_tiles(backend, mix, ne, nff):
    # an expert's tokens go in tiles of 160, the MMA's extent in steps of 16
    counts = [1, 15, 16, 17, 0, 33, 143, 144, 145, 159, 160, 161, 176, 321, 0, 2]
    L = synth.make_layer(51, ne, len(counts), nff, sh_ff=nff, router_std=0.05, dtypes=mix)
    ids = ids_of(counts, 3)
    x = synth.activations(81, len(ids), ne)
    out, _, _ = GpuLayer(backend, L).run(x, 1, path=2, expert_ids=ids)
    assert_close(out, oracle_layer(L, x, 1, expert_ids=ids).dst)


@pytest.mark.parametrize("raw_f32", [0, 1])
@pytest.mark.parametrize("ne,nff", [(256, 256), (768, 512), (256, 1024), (512, 1536), (256, 2048)])
def test_q6k_down_rows_by_offset(backend, ne, nff, raw_f32):
    # Q6_K down rows of 210 nff / 256 bytes go to the operand's lanes 8, 4, 2, 4 and 1 apart; the outputs come back in order, packed
    # or in f32, with the residual
    counts = [1, 16, 17, 0, 160, 161, 33]
    L = synth.make_layer(58, ne, len(counts), nff, sh_ff=nff, router_std=0.05)
    ids = ids_of(counts, 5)
    x, r = synth.activations(86, len(ids), ne), synth.activations(87, len(ids), ne)
    backend.set_config(raw_rows_f32=raw_f32)
    try:
        out, _, _ = GpuLayer(backend, L).run(x, 1, path=2, expert_ids=ids, residual=backend.from_host(r))
    finally:
        backend.set_config(raw_rows_f32=0)
    assert_close(out - r, oracle_layer(L, x, 1, expert_ids=ids).dst)


@pytest.mark.parametrize("rows", [8191, 8192, 8193, 16400])
def test_bucket_slices(backend, rows):
    # pairs are counted in slices over the CTAs of a cluster: just below, at and past 65536 and 131072 of them
    L = synth.make_layer(52, 256, 16, 256, router_std=0.05)
    x = synth.activations(82, rows, 256)
    out, ids, _ = GpuLayer(backend, L).run(x, 8)
    sel = np.unique(np.r_[0:8, rows // 2 : rows // 2 + 8, rows - 8 : rows])
    ref = oracle_layer(L, x[sel], 8)
    keep = [i for i in range(len(sel)) if i not in set(near_tie_rows(ref, 8).tolist())]
    assert np.array_equal(ids[sel[keep]], ref.ids[keep])
    assert_close(out[sel[keep]], ref.dst[keep])


@pytest.mark.parametrize("rows", [8, 9, 17, 63, 64, 65])
def test_router_of_wide_rows(backend, rows):
    # token rows stream through the router's stages from 9 rows on; 40 experts are not a whole tile
    L = synth.make_layer(53, 7168, 40, 256, router_std=0.05)
    x = synth.activations(83, rows, 7168)
    out, ids, _ = GpuLayer(backend, L).run(x, 4)
    ref = oracle_layer(L, x, 4)
    keep = [i for i in range(rows) if i not in set(near_tie_rows(ref, 4).tolist())]
    assert np.array_equal(ids[keep], ref.ids[keep])
    assert_close(out[keep], ref.dst[keep])


@pytest.mark.parametrize("down_q4k", [False, True])
@pytest.mark.parametrize("ne,nff", [(512, 256), (2048, 768), (4096, 512), (4352, 1024)])
def test_expert_major_segments(backend, ne, nff, down_q4k):
    # up to four tokens of a segment share one MMA with both limbs, more take one per limb; a segment holds eight
    counts = [1, 3, 4, 5, 0, 7, 8, 9, 12, 13]
    L = synth.make_layer(54, ne, len(counts), nff, sh_ff=nff, router_std=0.05, down_q4k=down_q4k)
    ids = ids_of(counts, 4)
    x = synth.activations(84, len(ids), ne)
    backend.set_config(expert_major=2)
    try:
        out, _, _ = GpuLayer(backend, L).run(x, 1, path=1, expert_ids=ids)
    finally:
        backend.set_config(expert_major=0)
    assert_close(out, oracle_layer(L, x, 1, expert_ids=ids).dst)


@pytest.mark.parametrize("down_q4k", [False, True])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_expert_major_largest_sums(backend, sign, down_q4k):
    # rows of one value: every fixed-point element is +-32639 and a sum of 32 is +-1044448, all three of its bytes in use; in the
    # last rows 24 elements of every 32 cancel or vanish (sums of any size, zero too)
    counts = [1, 4, 5, 8, 9]
    L = synth.make_layer(60, 1024, len(counts), 512, sh_ff=512, router_std=0.05, down_q4k=down_q4k)
    ids = ids_of(counts, 6)
    x = np.full((len(ids), 1024), 0.5 * sign, np.float32)
    x[-4:, 1::2] *= -1.0
    x[-2:].reshape(2, -1, 32)[:, :, 8:] = 0.0
    backend.set_config(expert_major=2)
    try:
        out, _, _ = GpuLayer(backend, L).run(x, 1, path=1, expert_ids=ids)
    finally:
        backend.set_config(expert_major=0)
    assert_close(out, oracle_layer(L, x, 1, expert_ids=ids).dst)


@pytest.mark.parametrize("ne,nff,sh_ff", [(256, 256, 0), (2048, 512, 512), (4096, 256, 768), (8192, 256, 0)])
@pytest.mark.parametrize("mix", [(Q5K, Q5K, Q6K), (Q5K, Q5K, Q8_0), (Q4K, Q5K, Q6K), (Q8_0, Q8_0, Q4K)])
def test_decode_stage_mixes(backend, mix, ne, nff, sh_ff):
    # per-pair decode: each stage takes the kernel of its own banks or the generic one
    L = synth.make_layer(55, ne, 8, nff, sh_ff=sh_ff, router_std=0.05, dtypes=mix)
    x = synth.activations(85, 3, ne)
    out, ids, _ = GpuLayer(backend, L).run(x, 4, path=1)
    ref = oracle_layer(L, x, 4)
    keep = [i for i in range(3) if i not in set(near_tie_rows(ref, 4).tolist())]
    assert np.array_equal(ids[keep], ref.ids[keep])
    assert_close(out[keep], ref.dst[keep])


@pytest.mark.parametrize("gated", [False, True])
def test_batched_calls_back_to_back(backend, gated):
    # the kernels of a call start beside their predecessors, those of the next call too: enqueued without a pause, with
    # other rows and other weights in the same scratch, calls give what they give alone
    from moe4all_b200 import MoeFfn
    be, calls = backend, []
    for i, rows in enumerate((300, 97, 641, 1200)):
        L = synth.make_layer(60 + i, 512, 32, 256, sh_ff=256, gated_shared=gated, router_std=0.05)
        g, x = GpuLayer(be, L), be.from_host(synth.activations(90 + i, rows, 512))
        norm = be.from_host(np.linspace(0.5, 1.5, 512).astype(np.float32)) if i % 2 else None
        dst = [be.alloc(rows * 512 * 4) for _ in range(2)]
        op = [MoeFfn(x=x, router=g.router, gate_exps=g.gate, up_exps=g.up, down_exps=g.down, dst=d, rows=rows, ne=512, n_expert=32, n_used=4,
                     n_ff_exp=256, sh_gate=g.sh_gate, sh_up=g.sh_up, sh_down=g.sh_down, sh_gate_inp=g.sh_gate_inp, sh_ff=256,
                     norm_weight=norm, path=2) for d in dst]
        calls.append((g, op, dst))
    for _, op, _ in calls:
        be.moe_ffn(op[0])
        be.sync()
    for rep in range(25):
        for _, op, _ in calls:
            be.moe_ffn(op[1])
        be.sync()
        for _, _, dst in calls:
            assert np.array_equal(be.download(dst[0], np.float32), be.download(dst[1], np.float32))


def scale_down_rows(L, scale_of_feature):
    """Multiplies the f16 scales (d, and dmin of Q4_K) of every expert's down rows, feature by feature."""
    nbytes, slots = synth.BLOCKS[L.down_dtype][1:]
    for name, n in (("down", L.n_expert), ("sh_down", 1)):
        if getattr(L, name) is None:
            continue
        blk = np.array(getattr(L, name), np.uint8).reshape(n, L.ne, -1, nbytes)
        for o in slots:
            d = np.ascontiguousarray(blk[..., o : o + 2]).view(np.float16).astype(np.float32) * scale_of_feature[None, :, None, None]
            blk[..., o : o + 2] = d.astype(np.float16).view(np.uint8)
        setattr(L, name, blk.reshape(-1))


@pytest.mark.parametrize("down_q4k", [False, True])
@pytest.mark.parametrize("with_nan", [False, True])
def test_raw_rows_keep_each_outputs_precision(backend, with_nan, down_q4k):
    # a few outputs a thousand times their neighbours (and two that are NaN): the others are as exact as alone
    ne, rows = 768, 150
    L = synth.make_layer(57, ne, 8, 256, sh_ff=256, router_std=0.05, down_q4k=down_q4k)
    big = np.random.default_rng(5).random(ne) < 0.1
    scale = np.where(big, 31.25, 0.03125).astype(np.float32)  # (the largest weights stay below 2^8, where f16 operands end)
    if with_nan:
        scale[[70, 401]] = np.nan
    scale_down_rows(L, scale)
    x = synth.activations(86, rows, ne)
    g, out = GpuLayer(backend, L), {}
    for f32 in (0, 1):
        backend.set_config(raw_rows_f32=f32)
        try:
            out[f32] = g.run(x, 4, path=2)[0], g.run(x, 1, path=2, shared=False)[0]
        finally:
            backend.set_config(raw_rows_f32=0)
    # one expert of weight 1 a row: an output is its raw value, rounded to 16 bits of mantissa (2^-16 of itself) at most
    got, want = out[0][1], out[1][1]
    finite = np.isfinite(want)
    assert np.array_equal(finite, ~np.isnan(got)) and finite.sum() == rows * (ne - 2 * with_nan)
    assert np.all(np.abs(got[finite] - want[finite]) <= 2.0**-16 * np.abs(want[finite]))
    # four experts and the shared one, feature by feature: at most 2^-16 of the sum of the five terms' magnitudes, which in
    # the 2-norm over the rows is about sqrt(5) times the sum's own; 2^-14 leaves 1.8 times that
    got, want = (out[i][0][:, np.isfinite(scale)].astype(np.float64) for i in (0, 1))
    assert np.all(np.linalg.norm(got - want, axis=0) <= 2.0**-14 * np.linalg.norm(want, axis=0))
    if not with_nan:
        ref = oracle_layer(L, x, 4)
        keep = [i for i in range(rows) if i not in set(near_tie_rows(ref, 4).tolist())]
        assert_close(out[0][0][keep], ref.dst[keep])


@pytest.mark.parametrize("recorded", [False, True])
def test_forms_in_turn_on_the_same_rows(backend, recorded):
    # every kernel family and format in turn, in place on the same rows and in the same scratch, each kernel starting beside
    # its predecessors: enqueued without a pause, or replayed as one plan, the rows end up as with a pause after every call
    from moe4all_b200 import DType, MoeFfn
    be, ne, calls = backend, 512, []
    forms = [((Q4K, Q4K, Q6K), 1200, 2, 0), ((Q4K, Q4K, Q6K), 4, 1, 1), ((Q5K, Q5K, Q6K), 300, 2, 0), ((Q5K, Q5K, Q6K), 2, 1, 0),
             ((Q8_0, Q8_0, Q8_0), 641, 2, 0), ((Q4K, Q4K, Q4K), 24, 1, 2), ((39, 39, 39), 97, 2, 0), ((39, 39, 39), 9, 1, 0),
             ((Q4K, Q4K, Q4K), 300, 2, 0), ((Q4K, Q4K, Q6K), 64, 1, 2), ((Q6K, Q4K, Q5K), 130, 2, 0), ((Q4K, Q4K, Q6K), 1, 1, 1)]
    hidden = be.alloc(1200 * ne * 4)
    for i, (mix, rows, path, em) in enumerate(forms):
        L = synth.make_layer(70 + i, ne, 16, 256, sh_ff=256, gated_shared=bool(i % 2), router_std=0.05, dtypes=mix)
        g, norm = GpuLayer(be, L), be.from_host(np.linspace(0.5, 1.5, ne).astype(np.float32))
        op = MoeFfn(x=hidden, router=g.router, gate_exps=g.gate, up_exps=g.up, down_exps=g.down, dst=hidden, rows=rows, ne=ne, n_expert=16,
                    n_used=4, n_ff_exp=256, sh_gate=g.sh_gate, sh_up=g.sh_up, sh_down=g.sh_down, sh_gate_inp=g.sh_gate_inp, sh_ff=256,
                    norm_weight=norm, residual=hidden, path=path, gate_dtype=DType(mix[0]), up_dtype=DType(mix[1]), down_dtype=DType(mix[2]))
        calls.append((op, em, g, norm))
    h0 = synth.activations(95, 1200, ne)

    def enqueue(pause=False):
        for op, em, *_ in calls:
            be.set_config(expert_major=em)
            be.moe_ffn(op)
            if pause:
                be.sync()

    try:
        be.upload(hidden, h0)
        enqueue(pause=True)
        want = be.download(hidden, np.float32)
        assert np.isfinite(want).all() and not np.array_equal(want, h0.reshape(-1))
        if recorded:
            be.graph_begin()
            enqueue()
            plan = be.graph_end()
        for rep in range(25):
            be.upload(hidden, h0)
            be.execute(plan) if recorded else enqueue()
            be.sync()
            assert np.array_equal(be.download(hidden, np.float32), want)
    finally:
        be.set_config(expert_major=0)


@pytest.mark.parametrize("ne,nff,used,shared,rows,mix", [
    (1024, 256, 4, False, 1, (Q4K, Q4K, Q6K)), (1024, 256, 4, False, 2, (Q4K, Q4K, Q6K)),       # gate/up 16 rows a role; 20 and 18 warps down
    (1024, 256, 4, False, 8, (Q4K, Q4K, Q6K)),                                                    # one task a warp, four CTAs to an SM
    (2048, 768, 8, False, 1, (Q4K, Q4K, Q6K)), (2048, 768, 8, False, 6, (Q4K, Q4K, Q6K)),        # 20 warps; past four waves, 12 of 16 tasks
    (2048, 512, 8, True, 3, (Q4K, Q4K, Q6K)), (2048, 512, 8, True, 4, (Q4K, Q4K, Q4K)),          # 12 warps, two rounds; nine
    (2560, 1536, 8, True, 1, (Q4K, Q4K, Q6K)),                                                    # 16 output rows in 217 KB, 24 warps
    (3072, 512, 6, False, 2, (Q4K, Q4K, Q4K)), (4096, 1024, 4, True, 1, (Q4K, Q4K, Q6K)),        # gate/up 8 x 2, two groups of x per lane
    (1536, 768, 2, True, 2, (Q5K, Q5K, Q6K)), (1536, 768, 2, True, 8, (Q5K, Q5K, Q6K)), (2048, 512, 8, True, 2, (Q5K, Q5K, Q6K))])
def test_per_pair_tiles_by_grid(backend, ne, nff, used, shared, rows, mix):
    # what a CTA takes follows from how many the grid has and an SM holds
    L = synth.make_layer(59, ne, 8, nff, sh_ff=nff if shared else 0, router_std=0.05, dtypes=mix)
    x = synth.activations(88, rows, ne)
    backend.set_config(expert_major=1)
    try:
        out, ids, _ = GpuLayer(backend, L).run(x, used, path=1)
    finally:
        backend.set_config(expert_major=0)
    ref = oracle_layer(L, x, used)
    keep = [i for i in range(rows) if i not in set(near_tie_rows(ref, used).tolist())]
    assert np.array_equal(ids[keep], ref.ids[keep])
    assert_close(out[keep], ref.dst[keep])


@pytest.mark.parametrize("mix", [(Q4K, Q4K, Q6K), (Q8_0, Q8_0, Q8_0)])
def test_both_halves_of_a_tiles_tokens_are_this_calls(backend, mix):
    # each CTA of a pair brings half of a tile's tokens (the second has none of its own up to 16), 64 steps through six stages, and the
    # MMAs of one read both: rows that change from call to call in the same buffers are those of the call, every time
    from moe4all_b200 import DType, MoeFfn
    be, counts = backend, [1, 16, 17, 32, 33, 100, 160, 161]
    L = synth.make_layer(61, 4096, len(counts), 512, sh_ff=512, router_std=0.05, dtypes=mix)
    g, ids = GpuLayer(be, L), ids_of(counts, 7)
    xs = [synth.activations(96 + i, len(ids), 4096) for i in range(2)]
    xb, dst = be.from_host(xs[0]), be.alloc(xs[0].nbytes)
    op = MoeFfn(x=xb, router=g.router, gate_exps=g.gate, up_exps=g.up, down_exps=g.down, dst=dst, rows=len(ids), ne=4096, n_expert=len(counts),
                n_used=1, n_ff_exp=512, sh_gate=g.sh_gate, sh_up=g.sh_up, sh_down=g.sh_down, sh_gate_inp=g.sh_gate_inp, sh_ff=512,
                expert_ids=be.from_host(ids), path=2, gate_dtype=DType(mix[0]), up_dtype=DType(mix[1]), down_dtype=DType(mix[2]))
    first = [None, None]
    for rep in range(40):
        i = rep & 1
        be.upload(xb, xs[i])
        be.moe_ffn(op)
        out = be.download(dst, np.float32).reshape(-1, 4096)
        if first[i] is None:
            first[i] = out
            assert_close(out, oracle_layer(L, xs[i], 1, expert_ids=ids).dst)
        assert np.array_equal(out, first[i])


@pytest.mark.parametrize("warps,chunks", [(0, 0), (0, 4), (16, 1), (3, 4)])
def test_gateup_shapes_by_config(backend, warps, chunks):
    # past four waves: the one-wave shape, a named one, and one that does not fit
    L = synth.make_layer(62, 2048, 8, 512, sh_ff=512, router_std=0.05)
    x = synth.activations(98, 6, 2048)
    backend.set_config(expert_major=1, gu_warps=warps, gu_chunks=chunks)
    try:
        out, ids, _ = GpuLayer(backend, L).run(x, 8, path=1)
    finally:
        backend.set_config(expert_major=0, gu_warps=4, gu_chunks=4)
    ref = oracle_layer(L, x, 8)
    keep = [i for i in range(6) if i not in set(near_tie_rows(ref, 8).tolist())]
    assert np.array_equal(ids[keep], ref.ids[keep])
    assert_close(out[keep], ref.dst[keep])


@pytest.mark.parametrize("mix,nff", [((Q4K, Q4K, Q6K), 256), ((Q4K, Q4K, Q6K), 512), ((Q4K, Q4K, Q6K), 1024), ((Q4K, Q4K, Q6K), 2048), ((Q4K, Q4K, Q4K), 512),
                                     ((Q5K, Q5K, Q5K), 512), ((Q8_0, Q8_0, Q8_0), 512), ((39, 39, 39), 512)])
@pytest.mark.parametrize("ne", [256, 1280])
@pytest.mark.parametrize("raw_f32", [0, 1])
def test_odd_widths(backend, mix, nff, ne, raw_f32):
    # 256-row blocks of an odd number: the last one of a tile goes half to each CTA of a pair, between jobs of whole blocks (1280) or alone
    # (256); Q6_K rows 8, 4, 2 and 1 apart, packed and f32 outputs
    counts = [1, 16, 17, 0, 33, 160, 161, 48]
    L = synth.make_layer(63, ne, len(counts), nff, sh_ff=nff, router_std=0.05, dtypes=mix)
    ids = ids_of(counts, 8)
    x = synth.activations(99, len(ids), ne)
    backend.set_config(raw_rows_f32=raw_f32)
    try:
        out, _, _ = GpuLayer(backend, L).run(x, 1, path=2, expert_ids=ids)
    finally:
        backend.set_config(raw_rows_f32=0)
    assert_close(out, oracle_layer(L, x, 1, expert_ids=ids).dst)
