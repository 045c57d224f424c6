"""Calls enqueued behind and beside one another without a wait in between: several attention + combine pairs in one
replayed graph, the attention kernel behind itself, layers' graphs on streams of their own, list and prefill calls in graphs."""
import numpy as np
import pytest

from conftest import check_close, make_decode_inputs
from gpu_util import to_dev

pytestmark = pytest.mark.gpu


def _capture(torch, calls):
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        with torch.cuda.graph(g, stream=side):
            for fn in calls:
                fn()
    torch.cuda.current_stream().wait_stream(side)
    return g


@pytest.mark.parametrize("n,T,H,d_qk", [(4096, 1, 20, 576), (32768, 2, 20, 576), (32768, 2, 32, 512), (4096, 1, 32, 512)])
def test_several_decodes_in_one_replayed_graph(pkg, cuda, oracle, n, T, H, d_qk):
    """One workspace, four caches, an output each; the records of a call are overwritten by the next one."""
    torch = cuda
    sets = [make_decode_inputs(100 + k, 1, T, H, n, d_qk=d_qk) for k in range(4)]
    dev = [(to_dev(torch, q), to_dev(torch, c), torch.full((1, T, H, 512), 7.0, device="cuda")) for q, c in sets]
    lens = to_dev(torch, np.array([n], np.int32))
    ws = pkg.new_workspace(1, T, H)

    def call(k, **kw):
        return lambda: pkg.mla_decode(dev[k][0], dev[k][1], lens, out=dev[k][2], workspace=ws, max_seq_len=n, impl=2, **kw)

    want = [oracle.mla_decode(q, c, [n], 1 / 16, key_splits=32) for q, c in sets]
    call(0)()
    torch.cuda.synchronize()
    assert pkg.decode_status(ws) == 0
    pairs = _capture(torch, [call(k) for k in (0, 1, 2, 3, 0, 1)])
    alone = _capture(torch, [call(k, no_combine=True) for k in (0, 1, 2, 3, 2, 1)] + [call(3)])
    for g in (pairs, alone, pairs):
        for _ in range(3):
            g.replay()
        torch.cuda.synchronize()
        assert pkg.decode_status(ws) == 0
    for k in range(4):
        check_close(dev[k][2].cpu().numpy(), want[k], f"cache {k}")


def test_decode_without_combine_behind_itself(pkg, cuda, oracle):
    torch = cuda
    n, T, H = 32768, 2, 20
    q, c = make_decode_inputs(7, 1, T, H, n)
    qd, cd, lens = to_dev(torch, q), to_dev(torch, c), to_dev(torch, np.array([n], np.int32))
    ws = pkg.new_workspace(1, T, H)
    for _ in range(20):
        pkg.mla_decode(qd, cd, lens, workspace=ws, max_seq_len=n, impl=2, no_combine=True)
    out = pkg.mla_decode(qd, cd, lens, workspace=ws, max_seq_len=n, impl=2)
    torch.cuda.synchronize()
    assert pkg.decode_status(ws) == 0
    check_close(out.cpu().numpy(), oracle.mla_decode(q, c, [n], 1 / 16, key_splits=32), "after launches without combine")


@pytest.mark.parametrize("n", [1024, 32768])
def test_layer_graphs_enqueued_without_waiting(pkg, cuda, oracle, n):
    """Steps of four layers, each on its layer's own stream, enqueued round after round and waited for once."""
    torch = cuda
    T, H = 2, 20
    rng = np.random.default_rng(n)
    q = rng.standard_normal((T, H, 576), dtype=np.float32).astype(np.float16)
    kv = (rng.standard_normal((T, 576), dtype=np.float32) * np.float32(0.5))
    qh, kvh = torch.from_numpy(q).pin_memory(), torch.from_numpy(kv).pin_memory()
    layers, caches = [], []
    for k in range(4):
        lay = pkg.MlaDecodeLayer(ctx=n, H=H, T_max=T, use_graph=True)
        c = (rng.standard_normal((n, 576), dtype=np.float32) * np.float32(0.5)).astype(np.float16)
        lay.cache.copy_(torch.from_numpy(c).cuda())
        layers.append(lay)
        caches.append(c)
    torch.cuda.synchronize()
    want = []
    for lay in layers:
        lay.pos = n - T
        want.append(lay.step(qh, kvh).numpy().copy())
    rows = layers[0].cache[n - T:].cpu().numpy()
    for c, w in zip(caches, want):
        c[n - T:] = rows  # the same new rows in every layer
        check_close(w[None], oracle.mla_decode(q[None], c, [n], 1 / 16, key_splits=32), "a step of its own")
    L = pkg._lib.load()
    for rounds in (1, 5):
        for lay in layers:
            lay._o_host.zero_()
        for _ in range(rounds):
            for lay in layers:
                h = lay._graphs[(qh.data_ptr(), kvh.data_ptr(), T)]
                assert L.gs_mla_layer_graph_step(h, n - T, lay._graph_stream_handle, 0) == 0
        torch.cuda.synchronize()
        for lay, w in zip(layers, want):
            assert pkg.decode_status(lay.workspace) == 0
            assert np.array_equal(lay._o_host[0].numpy(), w)


@pytest.mark.parametrize("q8", [False, True])
@pytest.mark.parametrize("T,splits", [(1, 16), (2, 4), (40, 1), (160, 1)])
def test_list_calls_in_one_replayed_graph(pkg, cuda, oracle, q8, T, splits):
    """Six calls over two caches behind one another: records with their combine, clusters, one CTA per list."""
    torch = cuda
    H, ctx, n = 64, 4000, 2052
    rng = np.random.default_rng(T)
    q = rng.standard_normal((T, H, 512), dtype=np.float32)
    sel = np.sort(np.stack([rng.permutation(ctx)[:n] for _ in range(T)]), 1).astype(np.int32)
    cnt = np.array([n - t % 4 for t in range(T)], np.int32)
    qd, sd, nd = to_dev(torch, q), to_dev(torch, sel), to_dev(torch, cnt)
    part = torch.empty(T * H * splits * 514, dtype=torch.float32, device="cuda") if splits > 1 else None
    calls, outs, want = [], [], []
    for k in range(2):
        c = (rng.standard_normal((ctx, 512), dtype=np.float32) * np.float32(0.5)).astype(np.float16)
        cq, cs = oracle.quant_q8_rows(c.astype(np.float32)) if q8 else (c, None)
        want.append(oracle.mla_attn_ref(q, oracle.dequant_q8(cq, cs) if q8 else c, sel, cnt, 1 / 16))
        cd, scd = to_dev(torch, cq), None if cs is None else to_dev(torch, cs)
        o = torch.full((T, H, 512), 7.0, device="cuda")
        outs.append(o)
        calls.append(lambda cd=cd, scd=scd, o=o: pkg.mla_attn(qd, cd, scd, sd, n, nd, 1 / 16, o, part, T, H, 512, splits))
    calls[0]()
    torch.cuda.synchronize()
    assert pkg.mla_attn_status() == 0
    g = _capture(torch, calls * 3)
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    assert pkg.mla_attn_status() == 0
    for o, w in zip(outs, want):
        check_close(o.cpu().numpy(), w, f"T={T}")


def test_prefill_behind_itself_in_a_graph(pkg, cuda):
    torch = cuda
    S, H = 2048, 20
    g = torch.Generator(device="cuda").manual_seed(4)
    sets = [tuple(torch.randn((S, H, 256), generator=g, device="cuda").half() for _ in range(3)) for _ in range(2)]
    outs = [torch.empty((S, H, 256), device="cuda") for _ in sets]
    want = [pkg.prefill_attn(*s).clone() for s in sets]
    calls = [lambda s=s, o=o: pkg.prefill_attn(*s, out=o) for s, o in zip(sets, outs)]
    graph = _capture(torch, calls * 3)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for o, w in zip(outs, want):
        assert torch.equal(o, w)


def test_calls_of_different_sizes_from_several_threads(pkg, cuda):
    """Two host threads on streams of their own, with calls of the same kernels that need different amounts of shared memory."""
    import threading
    torch = cuda
    n_big, H = 32768, 20
    cache = (torch.randn((n_big, 576), device="cuda") * 0.5).half()
    q = torch.randn((1, 1, H, 576), device="cuda").half()
    qs, ps = torch.randn((3, 96, 64), device="cuda"), torch.randn((500, 64), device="cuda")
    lens = {n: torch.full((1,), n, dtype=torch.int32, device="cuda") for n in (64, n_big)}
    want = {n: pkg.mla_decode(q, cache[:n].contiguous(), lens[n], max_seq_len=n) for n in lens}
    scores = {hq: torch.zeros((3, 500), device="cuda") for hq in (1, 96)}
    L = pkg._lib.load()
    torch.cuda.synchronize()
    errors = []

    def work(n, hq):
        try:
            torch.cuda.set_device(0)
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                c, ws, out = cache[:n].contiguous(), pkg.new_workspace(1, 1, H), torch.empty((1, 1, H, 512), device="cuda")
                w = torch.ones((3, hq), device="cuda")
                for _ in range(1500):
                    pkg.mla_decode(q, c, lens[n], workspace=ws, out=out, max_seq_len=n)
                    pkg._lib.check(L.gs_idx_score(qs.data_ptr(), w.data_ptr(), ps.data_ptr(), scores[hq].data_ptr(), 500, 1000, 3, 4, hq, 64, 0.1,
                                                  st.cuda_stream), "gs_idx_score")
                st.synchronize()
            assert pkg.decode_status(ws) == 0 and torch.equal(out, want[n])
        except Exception as exc:
            errors.append(exc)

    threads = [threading.Thread(target=work, args=a) for a in ((64, 1), (n_big, 96))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_first_calls_of_a_process_inside_a_capture(cuda):
    """Lists in clusters and split prefill items ask the device how many clusters it holds: also when a capture is the first to ask."""
    import os
    import subprocess
    import sys

    from conftest import ROOT
    code = """
import importlib, torch
pkg = importlib.import_module("glm-ssd_b200")
T, H, n = 2, 64, 2052
q, c = torch.randn((T, H, 512), device="cuda"), torch.randn((4000, 512), device="cuda").half()
sel = torch.arange(n, device="cuda").repeat(T, 1).int().contiguous()
cnt, o = torch.full((T,), n, dtype=torch.int32, device="cuda"), torch.zeros((T, H, 512), device="cuda")
Q, K, V = (torch.randn((s, 20, 256), device="cuda").half() for s in (100, 3100, 3100))
O = torch.zeros((100, 20, 256), device="cuda")
def calls():
    pkg.mla_attn(q, c, None, sel, n, cnt, 1 / 16, o, None, T, H, 512, 1)
    pkg.prefill_attn(Q, K, V, p0=3000, out=O)
s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
s.wait_stream(torch.cuda.current_stream())
with torch.cuda.stream(s):
    with torch.cuda.graph(g, stream=s):
        calls()
torch.cuda.synchronize()
g.replay()
torch.cuda.synchronize()
a, b = o.clone(), O.clone()
calls()
torch.cuda.synchronize()
assert pkg.mla_attn_status() == 0 and torch.equal(a, o) and torch.equal(b, O) and a.abs().max() > 0 and b.abs().max() > 0
"""
    subprocess.run([sys.executable, "-c", code], cwd=ROOT, check=True, timeout=120)
