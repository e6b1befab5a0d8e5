"""The decode step's CUDA graph: what orders its nodes, and that replays of one state give one result.

A step forks the LoRA products of a layer from its r / k / v products and joins them before the recurrence.  Kernels
start under the tail of the one before them (programmatic edges) and wait for it on the device, which orders them behind
ONE predecessor: a node that joins branches has to have full edges."""
import collections
import ctypes
import gc
import weakref

import pytest
import torch

import hf_adapter_b200 as hb

pytestmark = pytest.mark.gpu


class _Edge(ctypes.Structure):  # cudaGraphEdgeData
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte), ("reserved", ctypes.c_ubyte * 5)]


def _edges(graph):
    """[(to node, edge type)] of a captured graph (type 0: full, 1: programmatic)."""
    cu = ctypes.CDLL("libcuda.so.1")
    raw, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert cu.cuGraphGetEdges_v2(raw, None, None, None, ctypes.byref(n)) == 0
    a, b, e = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)(), (_Edge * n.value)()
    assert cu.cuGraphGetEdges_v2(raw, a, b, e, ctypes.byref(n)) == 0
    return [(b[i], e[i].type) for i in range(n.value)]


def _model(weights, D, layers, state=torch.float32, dtype=torch.float16):
    cfg = hb.NativeRWKV7Config(vocab_size=512, hidden_size=D, num_hidden_layers=layers, num_heads=D // 64, head_dim=64,
                               intermediate_size=4 * D, decay_low_rank_dim=64, a_low_rank_dim=64, v_low_rank_dim=32,
                               gate_low_rank_dim=128)
    old = torch.get_default_dtype()
    torch.set_default_dtype(dtype)
    try:
        with torch.device("cuda"):
            m = hb.RWKV7ForCausalLM(cfg, state_dtype=state).eval()
    finally:
        torch.set_default_dtype(old)
    gen = torch.Generator(device="cuda").manual_seed(D + layers)
    with torch.no_grad():
        for name, p in m.named_parameters():
            if p.dim() == 2:
                p.normal_(0.0, 1.0 if "embeddings" in name else 0.02, generator=gen)
            elif any(k in name for k in (".x_", "k_k", "k_a")):
                p.uniform_(0, 1, generator=gen)
    if weights != "dense":
        hb.quantize_model(m, weights, min_params=100_000, group_size=128, skip=("lm_head",))
    return m


@pytest.mark.parametrize("weights,batch,state", [("mm4", 64, torch.float32), ("w8", 64, torch.float16), ("dense", 16, torch.float32),
                                                 ("dense", 80, torch.float32), ("dense", 2, torch.float32)])
def test_joins_have_full_edges(weights, batch, state):
    m = _model(weights, 512, 3, state)
    cache, ids = m.new_cache(batch), torch.zeros(batch, device="cuda", dtype=torch.long)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        m._decode_step(ids, cache)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        m._decode_step(ids, cache)
    into = collections.defaultdict(list)
    for node, kind in _edges(graph):
        into[node].append(kind)
    assert any(kinds == [1] for kinds in into.values())  # chains are programmatic
    joins = [kinds for kinds in into.values() if len(kinds) > 1]
    assert bool(joins) == (batch > 8) and not any(any(kinds) for kinds in joins)


@pytest.mark.parametrize("weights,D,batch,state", [("mm4", 4096, b, torch.float32) for b in (1, 8, 9, 64, 128, 256)]
                         + [("w8", 2560, b, torch.float16) for b in (1, 9, 64, 256)]
                         + [("dense", 2560, b, torch.float32) for b in (1, 8, 9, 64, 256)])
def test_replays_of_a_state_agree(weights, D, batch, state):
    """Two states in turn, 25 replays of each: a value read too early or too late is the other state's."""
    m = _model(weights, D, 4, state)
    gen = torch.Generator(device="cuda").manual_seed(batch)
    cache = m.new_cache(batch)
    starts = []
    for _ in range(2):
        cache.reset()
        m.rwkv7_prefill_native(torch.randint(0, 512, (batch, 4), generator=gen, device="cuda"), cache)
        starts.append((torch.randint(0, 512, (batch,), generator=gen, device="cuda"), [t.clone() for t in cache._tensors()]))
    first = [None, None]
    for i in range(50):
        ids, tensors = starts[i % 2]
        for dst, src in zip(cache._tensors(), tensors):
            dst.copy_(src)
        got = [m.rwkv7_forward_token(ids, cache), *cache._tensors()]
        if first[i % 2] is None:
            first[i % 2] = [t.clone() for t in got]
        assert all(torch.equal(a, b) for a, b in zip(got, first[i % 2])), f"replay {i // 2} of state {i % 2}"
    assert not torch.equal(first[0][0], first[1][0])


@pytest.mark.parametrize("weights,D,batch", [("mm4", 4096, 128), ("w8", 2560, 256)])
def test_thousands_of_replays_agree(weights, D, batch):
    """A race between two roles of a kernel need not show in 25 replays: a stage of the weight ring that was given back while its loads were
    on their way showed once in 700 (int4) and 2600 (int8) steps of these."""
    m = _model(weights, D, 4, torch.float32 if weights == "mm4" else torch.float16)
    gen = torch.Generator(device="cuda").manual_seed(batch)
    cache, ids = m.new_cache(batch), torch.randint(0, 512, (batch,), generator=gen, device="cuda")
    m.rwkv7_prefill_native(torch.randint(0, 512, (batch, 4), generator=gen, device="cuda"), cache)
    start = [t.clone() for t in cache._tensors()]
    first, wrong = None, torch.zeros((), device="cuda", dtype=torch.int64)
    for _ in range(3000):
        for dst, src in zip(cache._tensors(), start):
            dst.copy_(src)
        logits = m.rwkv7_forward_token(ids, cache)
        first = logits.clone() if first is None else first
        wrong += (logits != first).any()
    assert int(wrong) == 0


def test_a_dropped_model_does_not_break_the_next_capture(monkeypatch):
    """A dropped model is a reference cycle that holds its graphs; the collector becomes due in the middle of a capture."""
    from hf_adapter_b200 import packing
    calls, real, threshold = [], packing.extract_graph_packs, gc.get_threshold()

    def due(*a, **k):
        calls.append(0)
        if len(calls) == 3:  # two warm-up steps, then the captured one
            gc.set_threshold(1)
            calls.extend([] for _ in range(1000))
        return real(*a, **k)

    ids = torch.zeros(1, device="cuda", dtype=torch.long)
    try:
        gc.set_threshold(10 ** 9)
        old = _model("dense", 256, 1)
        old.rwkv7_forward_token(ids, old.new_cache(1))
        del old
        m = _model("dense", 256, 1)
        monkeypatch.setattr(packing, "extract_graph_packs", due)
        out = m.rwkv7_forward_token(ids, m.new_cache(1))
        assert len(calls) > 1000 and gc.isenabled() and bool(torch.isfinite(out).all())
    finally:
        gc.set_threshold(*threshold)


def test_branch_results_outlive_their_use_on_the_main_stream():
    """Outside capture: memory of results that a branch allocated is not handed out again while the stream they were made for is
    still busy with them."""
    from hf_adapter_b200 import packing
    D, B, R = 256, 16, 32
    f = lambda *s: torch.randn(*s, device="cuda", dtype=torch.float16)
    ops, downs, ups = [f(D, D) for _ in range(3)], [f(R, D) for _ in range(4)], [f(D, R) for _ in range(4)]
    ctx, main = packing.StepContext(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(main):
        res = packing._wide_projections(ctx, f(B, D), ops, [f(B, D) for _ in range(3)], downs, ups, [f(B, D) for _ in range(4)])
        torch.cuda._sleep(200_000_000)  # a tenth of a second in which the results are "in use"
        used = {t.data_ptr() for t in res}
        del res
        for i in range(3):
            with torch.cuda.stream(ctx.side_stream(torch.device("cuda", torch.cuda.current_device()), i)):
                again = [torch.empty(B, D, device="cuda", dtype=torch.float16) for _ in range(8)]
            assert not main.query() and not used & {t.data_ptr() for t in again}
    torch.cuda.synchronize()


def test_a_dropped_pool_frees_its_graph_without_the_collector():
    """A graph that waits for the cyclic collector is destroyed at a moment nobody chose, a foreign capture among them.  A graph
    that is kept longer than its pool keeps the buffers it was captured over."""
    m = _model("dense", 256, 1)
    ids = torch.zeros(1, device="cuda", dtype=torch.long)
    on = gc.isenabled()
    gc.disable()
    try:
        pool = hb.RWKV7StatePool(m, 2)
        slots, gens = pool.allocate(["a"])
        pool.decode(ids, slots, gens)
        (graph,) = pool._graphs.values()
        assert graph.pool is pool
        gone, buffers = weakref.ref(pool), weakref.ref(pool.S_pool)
        del pool
        assert gone() is None and graph.pool is None and buffers() is not None
        graph, gone = None, weakref.ref(graph)
        assert gone() is None and buffers() is None
    finally:
        if on:
            gc.enable()


@pytest.mark.parametrize("weights,cls", [("mm4", "MM4Linear"), ("w8", "MM8Linear")])
def test_tiled_weights_are_built_on_the_stream_of_the_step(weights, cls, monkeypatch):
    """The tiled copy that a projection makes on first use outlives the step: its memory belongs to the stream that the program
    runs on, not to a branch of one step, whose later allocations would not wait for the readers of a copy that was dropped."""
    from hf_adapter_b200 import quant
    m = _model(weights, 512, 1)
    linear, seen = getattr(quant, cls), []
    real = linear.tiled_for

    def tiled_for(self, x):
        if self._tiled is None:
            seen.append(torch.cuda.current_stream())
        return real(self, x)

    monkeypatch.setattr(linear, "tiled_for", tiled_for)
    main = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(main), torch.no_grad():
        m._decode_step(torch.zeros(16, device="cuda", dtype=torch.long), m.new_cache(16))
    torch.cuda.synchronize()
    assert len(seen) >= 6 and all(s == main for s in seen)  # r, k, v, o and the two of the FFN


@pytest.mark.parametrize("weights,D,rows,leads", [("dense", 512, 16, True), ("dense", 2048, 16, False), ("dense", 512, 64, True),
                                                  ("dense", 1024, 64, False), ("mm8", 2048, 16, False), ("a8w8", 2048, 16, True),
                                                  ("mm4", 2048, 16, True)])
def test_longer_branch_of_a_layer_stays_on_the_stream_of_the_step(weights, D, rows, leads, monkeypatch):
    """Where r / k / v are three products of wide weights, r stays on the step's stream and the LoRA chain branches off, in its form
    with little shared memory; else the chain stays."""
    from hf_adapter_b200 import lora, packing
    m = _model(weights, D, 1)
    chain, products = [], []
    real_chain, real_linear = lora.small_gemm_group, packing.apply_linear
    monkeypatch.setattr(lora, "small_gemm_group", lambda *a, **k: (chain.append((torch.cuda.current_stream(), bool(k.get("lean")))), real_chain(*a, **k))[1])
    monkeypatch.setattr(packing, "apply_linear", lambda *a, **k: (products.append(torch.cuda.current_stream()), real_linear(*a, **k))[1])
    with torch.no_grad():
        m._decode_step(torch.zeros(rows, device="cuda", dtype=torch.long), m.new_cache(rows))
    torch.cuda.synchronize()
    main = torch.cuda.current_stream()
    assert [(s == main, lean) for s, lean in chain] == [(leads, not leads)] * 2
    if weights != "mm4":  # (one grouped launch)
        assert sum(s == main for s in products[:3]) == (0 if leads else 1)
