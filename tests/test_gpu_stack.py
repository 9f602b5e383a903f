"""GPU: a stack of MoE sub-layers (RmsNorm -> MoeFfn + shared expert -> residual Add).

Parity is teacher-forced per layer: a 1e-3 drift in `hidden` can flip a near-tie top-k choice at
some layer, after which a free-running comparison diverges discretely; so every layer is fed the
oracle's hidden state and checked on its own, and the free-running drift is only reported."""
import numpy as np
import pytest
import torch

from moe4all_b200.devgen import DeviceLayer
from moe4all_b200.stack import MoeStack
from oracle import oracle as orc

from helpers import assert_close, near_tie_rows, rel_err

pytestmark = pytest.mark.gpu
NE, E, K, NFF, NL, ROWS = 512, 16, 4, 256, 6, 3


def oracle_sublayer(h, nw, L):
    hn = orc.rmsnorm(h, nw, 1e-6)
    res = orc.moe_layer(hn, L.router, L.gate, L.up, L.down, L.sh_gate, L.sh_up, L.sh_down, L.sh_gate_inp, NFF,
                        n_expert=E, n_used=K, n_ff_exp=NFF)
    return orc.add(h, res.dst), res


@pytest.mark.parametrize("fused", [False, True])
def test_stack_teacher_forced_and_replay(backend, fused):
    be = backend
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        be.set_stream(stream.cuda_stream)
        try:
            layers = [DeviceLayer(be, 300 + i, NE, E, NFF, sh_ff=NFF, router_std=0.05) for i in range(NL)]
            gen = torch.Generator(device="cuda")
            gen.manual_seed(1)
            nws = [1.0 + 0.1 * torch.randn(NE, generator=gen, device="cuda") for _ in range(NL)]
            st = MoeStack(be, layers, nws, ROWS, NE, E, K, NFF, sh_ff=NFF, fused=fused)
            hosts = [L.host() for L in layers]
            h0 = np.random.default_rng(2).normal(size=(ROWS, NE)).astype(np.float32)
            # teacher-forced: every layer starts from the oracle's hidden state
            h = h0
            for li in range(NL):
                st.hidden.copy_(torch.from_numpy(h))
                st.layer(li)
                be.sync()
                want, res = oracle_sublayer(h, nws[li].cpu().numpy(), hosts[li])
                ties = near_tie_rows(res, K)
                assert len(ties) == 0 and np.array_equal(st.ids[li].cpu().numpy(), res.ids), f"layer {li}: ids differ"
                assert_close(st.hidden.cpu().numpy(), want, what=f"layer {li}")
                h = want
            # free-running, eager vs recorded replay: bit-identical to each other
            st.hidden.copy_(torch.from_numpy(h0))
            st.step()
            be.sync()
            eager = st.hidden.cpu().numpy().copy()
            st.record()
            st.hidden.copy_(torch.from_numpy(h0))
            st.replay()
            be.sync()
            assert np.array_equal(st.hidden.cpu().numpy(), eager)
            rel, _ = rel_err(eager, h)
            print(f"free-running drift after {NL} layers: {rel:.2e}")
            assert rel < 5e-2
        finally:
            be.sync()
            be.set_stream(None)


@pytest.mark.parametrize("rows,k", [(1, 6), (5, 3), (25, 6)])
def test_ids_of_a_layer_may_end_anywhere(backend, rows, k):
    # rows x k ids that are no multiple of 16 bytes: every layer's are its own, and those of the layer alone
    be = backend
    # (norm weights of 0.04 with routers of 1 / 0.04: sub-layers that add a fraction of the stream, scores as far apart as without)
    layers = [DeviceLayer(be, 400 + i, NE, E, NFF, router_std=0.05 / 0.04) for i in range(3)]
    gen = torch.Generator(device="cuda").manual_seed(rows)
    nws = [0.04 * (1.0 + 0.1 * torch.randn(NE, generator=gen, device="cuda")) for _ in layers]
    torch.cuda.synchronize()
    st = MoeStack(be, layers, nws, rows, NE, E, k, NFF)
    assert tuple(st.ids.shape) == (3, rows, k)
    h = torch.randn(rows, NE, generator=gen, device="cuda")
    st.hidden.copy_(h)
    torch.cuda.synchronize()
    st.step()
    be.sync()
    h = h.cpu().numpy()
    for li, L in enumerate(layers):
        H = L.host()
        res = orc.moe_ffn(orc.rmsnorm(h, nws[li].cpu().numpy(), 1e-6), H.router, H.gate, H.up, H.down, n_expert=E, n_used=k, n_ff_exp=NFF)
        keep = np.setdiff1d(np.arange(rows), near_tie_rows(res, k, ulps=4096))  # the stream itself is the GPU's in the layers behind
        assert len(keep) >= rows - 2
        assert np.array_equal(st.ids[li].cpu().numpy()[keep], res.ids[keep])
        h = orc.add(h, res.dst)


@pytest.mark.parametrize("rows,path", [(2, 1), (40, 2)])
def test_fused_norm_and_residual_one_op(backend, rows, path):
    # RmsNorm -> MoeFfn -> Add folded into one call, in place on the hidden state, both paths
    from moe4all_b200 import MoeFfn, synth
    be = backend
    L = synth.make_layer(71, NE, E, NFF, sh_ff=NFF, router_std=0.05)
    rng = np.random.default_rng(3)
    h = rng.normal(size=(rows, NE)).astype(np.float32)
    nw = (1.0 + 0.1 * rng.normal(size=NE)).astype(np.float32)
    b = {k: be.from_host(getattr(L, k)) for k in ("router", "gate", "up", "down", "sh_gate", "sh_up", "sh_down", "sh_gate_inp")}
    hb, nwb = be.from_host(h), be.from_host(nw)
    ids = be.alloc(rows * K * 4)
    be.moe_ffn(MoeFfn(x=hb, dst=hb, residual=hb, norm_weight=nwb, norm_eps=1e-6, router=b["router"], gate_exps=b["gate"],
                      up_exps=b["up"], down_exps=b["down"], rows=rows, ne=NE, n_expert=E, n_used=K, n_ff_exp=NFF,
                      sh_gate=b["sh_gate"], sh_up=b["sh_up"], sh_down=b["sh_down"], sh_gate_inp=b["sh_gate_inp"], sh_ff=NFF,
                      ids_out=ids, path=path))
    got = be.download(hb, np.float32).reshape(rows, NE)
    want, res = oracle_sublayer(h, nw, L)
    ties = set(near_tie_rows(res, K).tolist())
    keep = [r for r in range(rows) if r not in ties]
    assert np.array_equal(be.download(ids, np.int32).reshape(rows, K)[keep], res.ids[keep])
    assert_close(got[keep], want[keep])


@pytest.mark.parametrize("seed", range(6))
def test_chain_of_layers_in_both_forms(backend, seed):
    # The per-pair and the expert-major kernels round a layer's activations differently, by less than 2e-4 of its result.  Down a chain
    # that may change which of two nearly equal experts a row takes, from where on the row is another one; the rows that take the same
    # experts throughout have to agree, and few may not.
    be, rows, n_expert, layers_n, small = backend, 24, 32, 8, 0.04  # a sub-layer adds a fraction of the stream, as in perf/cases.py
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        be.set_stream(stream.cuda_stream)
        try:
            layers = [DeviceLayer(be, 900 + 50 * seed + i, NE, n_expert, NFF, sh_ff=NFF, router_std=0.05 / small) for i in range(layers_n)]
            gen = torch.Generator(device="cuda").manual_seed(seed)
            nws = [small * (1.0 + 0.1 * torch.randn(NE, generator=gen, device="cuda")) for _ in layers]
            h0 = torch.randn(rows, NE, generator=gen, device="cuda")
            st = MoeStack(be, layers, nws, rows, NE, n_expert, K, NFF, sh_ff=NFF)
            got = []
            for form in (1, 2):
                be.set_config(expert_major=form)
                st.hidden.copy_(h0)
                st.step()
                be.sync()
                got.append((st.hidden.cpu().numpy().copy(), st.ids.cpu().numpy().copy()))
        finally:
            be.sync()
            be.set_config(expert_major=0)
            be.set_stream(None)
    (a, ids_a), (b, ids_b) = got
    same = (ids_a == ids_b).all(axis=(0, 2))
    assert same.sum() >= rows - 2
    assert not np.array_equal(a, b)  # two forms did run
    rel, _ = rel_err(b[same], a[same])
    print(f"{same.sum()} of {rows} rows, {rel:.2e}")
    assert rel <= layers_n * 2e-4
