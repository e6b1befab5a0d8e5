"""The rows that pad a pool's batch to its graph's size: they name the scratch slot, are not computed, and change nothing."""
import pytest
import torch

import hf_adapter_b200 as hb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 3, 8])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
def test_rows_of_the_idle_slot(rows, dt):
    g = torch.Generator(device="cuda").manual_seed(rows)
    B, H, N, cap = 8, 3, 64, 11
    f = lambda *s: torch.randn(*s, generator=g, device="cuda")
    r, w, k, v, a, gate = (f(B, H * N).to(dt) for _ in range(6))
    par = [f(H * N).to(dt) for _ in range(5)]
    pool, vf, vg = f(cap, H, N, N), f(cap, H * N).to(dt), f(B, H * N).to(dt)
    slots = torch.tensor([5, 0, 9, 2, 7, 1, 3, 8][:rows] + [cap - 1] * (B - rows), device="cuda", dtype=torch.int32)
    results = []
    for idle in (-1, cap - 1):
        S = pool.clone()
        out, _ = hb.fused_recurrent_output_prepare_raw(r, w, k, v, a, S, gate, *par, eps=64e-5, v_first=vf, v_gate=vg, slot_ids=slots, idle_slot=idle)
        results.append((out, S))
    (all_out, all_S), (out, S) = results
    assert torch.equal(out[:rows], all_out[:rows]) and torch.equal(S[:cap - 1], all_S[:cap - 1])
    if rows < B:
        assert not bool(out[rows:].any()) and torch.equal(S[cap - 1], pool[cap - 1]) and not torch.equal(all_S[cap - 1], pool[cap - 1])


def test_entry_point_without_an_idle_slot():
    """The pool's recurrence as a C caller has it, without the argument for the idle row: that of none (-1)."""
    from hf_adapter_b200 import _lib
    from hf_adapter_b200._util import ptr, stream_ptr
    g = torch.Generator(device="cuda").manual_seed(1)
    B, H, N, cap = 4, 2, 64, 6
    f = lambda *s: torch.randn(*s, generator=g, device="cuda")
    r, w, k, v, a, gate = (f(B, H * N).half() for _ in range(6))
    par = [f(H * N).half() for _ in range(5)]
    pool, slots = f(cap, H, N, N), torch.tensor([3, 0, 5, 1], device="cuda", dtype=torch.int32)
    results = []
    for name, idle in (("rwkv7_wkv7_output_prepare_raw_pool", ()), ("rwkv7_wkv7_output_prepare_raw_pool_idle", (-1,))):
        S, out = pool.clone(), torch.empty_like(r)
        _lib.check(getattr(_lib.lib, name)(*(ptr(t) for t in (r, w, k, v, a, S, slots, gate, *par, out)), 0, 0, 0, 0, 0, 0, 0, 0, 0, *idle, B, H, N, 64e-5,
                                           _lib.F16, stream_ptr(r)), name)
        results.append((out, S))
    assert all(torch.equal(x, y) for x, y in zip(*results)) and not torch.equal(results[0][1], pool)


def test_padded_pool_step_is_the_unpadded_one():
    cfg = hb.NativeRWKV7Config(vocab_size=128, hidden_size=256, num_hidden_layers=2, num_heads=4, head_dim=64, intermediate_size=512,
                               decay_low_rank_dim=16, a_low_rank_dim=16, v_low_rank_dim=16, gate_low_rank_dim=32)
    torch.manual_seed(3)
    m = hb.RWKV7ForCausalLM(cfg).half().cuda().eval()
    ids = torch.randint(0, 128, (11,), device="cuda")
    outs = []
    for graph in (True, False):  # 16 rows, five of them padding, and 11
        pool = hb.RWKV7StatePool(m, 13)
        slots, gens = pool.allocate(range(13))
        for _ in range(3):
            out = pool.decode(ids, slots[:11], gens[:11], use_graph=graph)
        assert bool(torch.isfinite(out).all())
        outs.append((out, pool.S_pool[:, :13].clone()))
    for x, y in zip(*outs):  # other row counts take other product kernels: single roundings
        assert float((x.double() - y.double()).norm()) <= 4 * 2.0 ** -11 * float(y.double().norm())
