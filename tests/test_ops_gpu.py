"""GPU parity of the recurrence / norm-mix / LoRA / prep kernels, called through the C ABI via the
reference-signature wrappers, against (a) the golden outputs of the reference and (b) the pinned oracle on
fresh seeded inputs, including ragged and edge shapes."""
import numpy as np
import pytest
import torch

import hf_adapter_b200 as hb
from oracle import rwkv7_oracle as O
from tests.gpu_util import cu, golden, npf, rel_err, wkv_inputs

pytestmark = pytest.mark.gpu
H, N = 2, 64
EPS = N * 1e-5
TD = {"fp32": torch.float32, "fp16": torch.float16}


def tol(dt, k=1.0):
    return dict(rtol=3e-5 * k, atol=3e-5 * k) if dt == "fp32" else dict(rtol=4e-3 * k, atol=4e-3 * k)


@pytest.mark.parametrize("dt", ["fp32", "fp16"])
def test_step_against_golden(dt):
    g = golden(f"ops_{dt}.npz")
    t = {k: cu(v) for k, v in g.items() if k.startswith(("step_", "raw_"))}
    y, s = hb.fused_recurrent_update(t["step_r"], t["step_w"], t["step_k"], t["step_v"], t["step_kk"], t["step_a"], t["step_state"])
    st = dict(rtol=1e-4, atol=1e-4) if dt == "fp32" else dict(rtol=1e-2, atol=5e-3)
    np.testing.assert_allclose(npf(s), g["step_state_out"], **st)
    np.testing.assert_allclose(npf(y), g["step_y"].astype(np.float32), **tol(dt, 20))
    assert y.dtype == TD[dt] and s.dtype == torch.float32 and tuple(y.shape) == (2, H, N)
    # flat inputs -> flat output; the input state must be untouched
    s_before = t["step_state"].clone()
    y2, s2 = hb.fused_recurrent_update(*(t[f"step_{n}"].reshape(2, H * N) for n in ("r", "w", "k", "v", "kk", "a")), t["step_state"])
    assert tuple(y2.shape) == (2, H * N) and torch.equal(y2.reshape(2, H, N), y) and torch.equal(s2, s)
    assert torch.equal(t["step_state"], s_before)
    yp, sp = hb.fused_recurrent_output_prepare(t["step_r"], t["step_w"], t["step_k"], t["step_v"], t["step_kk"], t["step_a"],
                                               t["step_state"], t["step_g"], t["step_r_k"], t["step_gn_w"], t["step_gn_b"], eps=EPS)
    np.testing.assert_allclose(npf(yp), g["prep_y"].astype(np.float32), **tol(dt, 3))
    yr, sr = hb.fused_recurrent_output_prepare_raw(t["step_r"], t["raw_w"], t["raw_k"], t["step_v"], t["step_a"], t["step_state"],
                                                   t["step_g"], t["raw_k_k"], t["raw_k_a"], t["step_r_k"], t["step_gn_w"],
                                                   t["step_gn_b"], eps=EPS)
    np.testing.assert_allclose(npf(yr), g["raw_y"].astype(np.float32), **tol(dt, 3))
    np.testing.assert_allclose(npf(sr), g["raw_state_out"], **st)


@pytest.mark.parametrize("B,Hh", [(1, 1), (3, 5), (64, 8)])
def test_step_against_oracle_and_inplace(B, Hh):
    r, w, k, v, kk, a = (x[:, 0] for x in wkv_inputs(B, 1, Hh, N, seed=B * 31 + Hh))
    rng = np.random.default_rng(5)
    state = (0.3 * rng.standard_normal((B, Hh, N, N))).astype(np.float32)
    g = rng.standard_normal((B, Hh, N)).astype(np.float16)
    w_raw = rng.standard_normal((B, Hh, N)).astype(np.float16)
    k_k = (0.85 + 0.1 * rng.standard_normal(Hh * N)).astype(np.float16)
    k_a = (1 + 0.1 * rng.standard_normal(Hh * N)).astype(np.float16)
    r_k = (0.1 * rng.standard_normal((Hh, N))).astype(np.float16)
    gw = (1 + 0.1 * rng.standard_normal(Hh * N)).astype(np.float16)
    gb = (0.1 * rng.standard_normal(Hh * N)).astype(np.float16)
    yo, so = O.recurrent_output_prepare_raw(r, w_raw, k, v, a, state, g, k_k, k_a, r_k, gw, gb, EPS)
    args = [cu(x) for x in (r, w_raw, k, v, a)]
    st = cu(state)
    par = [cu(x) for x in (g, k_k, k_a, r_k, gw, gb)]
    y, s = hb.fused_recurrent_output_prepare_raw(*args, st, *par, eps=EPS)
    np.testing.assert_allclose(npf(s), so, rtol=2e-5, atol=2e-5)
    np.testing.assert_allclose(npf(y), yo.astype(np.float32), rtol=4e-3, atol=4e-3)
    # in-place variant gives bit-identical results
    st2 = st.clone()
    y2, s2 = hb.fused_recurrent_output_prepare_raw(*args, st2, *par, eps=EPS, new_state=st2)
    assert s2.data_ptr() == st2.data_ptr() and torch.equal(st2, s) and torch.equal(y2, y)
    # repeatability (no atomics, fixed reduction order)
    y3, s3 = hb.fused_recurrent_output_prepare_raw(*args, st, *par, eps=EPS)
    assert torch.equal(y3, y) and torch.equal(s3, s)


def test_back_to_back_steps_feed_each_other():
    """Twelve one-token updates launched back to back, each reading the state the previous launch wrote in place
    (the kernels are launched programmatically: a launch must wait for its predecessor before it loads the state),
    against the oracle's sequential scan."""
    B, T, Hh = 64, 12, 32
    r, w, k, v, kk, a = wkv_inputs(B, T, Hh, N, seed=77)
    state = (0.3 * np.random.default_rng(6).standard_normal((B, Hh, N, N))).astype(np.float32)
    yo, so = O.recurrent_scan(r, w, k, v, kk, a, state)
    dev = [cu(x) for x in (r, w, k, v, kk, a)]
    st = cu(state)
    steps = [[x[:, t].contiguous() for x in dev] for t in range(T)]  # sliced first: no other kernel between the launches
    outs = [hb.fused_recurrent_update(*steps[t], st, new_state=st)[0] for t in range(T)]
    np.testing.assert_allclose(npf(st), so, rtol=1e-4, atol=1e-4)
    np.testing.assert_allclose(npf(torch.stack(outs, 1)), yo.astype(np.float32), rtol=4e-3, atol=4e-3)


def test_step_fused_lora_epilogues():
    """w/a biases, sigmoids and the v_first interpolation folded into the step == doing them beforehand."""
    B, Hh = 4, 3
    rng = np.random.default_rng(11)
    f16 = lambda *s: rng.standard_normal(s).astype(np.float16)
    r, w_pre, k, v, a_pre, g, vg_pre, vf = (f16(B, Hh, N) for _ in range(8))
    wb, ab, vb = (0.5 * f16(Hh * N) for _ in range(3))
    k_k, k_a, r_k, gw, gb = (0.85 + 0.1 * f16(Hh * N)), (1 + 0.1 * f16(Hh * N)), 0.1 * f16(Hh, N), 1 + 0.1 * f16(Hh * N), 0.1 * f16(Hh * N)
    state = (0.3 * rng.standard_normal((B, Hh, N, N))).astype(np.float32)
    h = lambda x: np.asarray(x, np.float16)
    w_raw = h(w_pre.astype(np.float32) + wb.reshape(Hh, N).astype(np.float32))
    a = h(O.sigmoid(h(a_pre.astype(np.float32) + ab.reshape(Hh, N).astype(np.float32)).astype(np.float32)))
    gate = h(O.sigmoid(h(vg_pre.astype(np.float32) + vb.reshape(Hh, N).astype(np.float32)).astype(np.float32)))
    v_mix = h(v.astype(np.float32) + (vf.astype(np.float32) - v.astype(np.float32)) * gate.astype(np.float32))
    yo, so = O.recurrent_output_prepare_raw(r, w_raw, k, v_mix, a, state, g, h(k_k), h(k_a), h(r_k), h(gw), h(gb), EPS)
    v_out = torch.empty((B, Hh * N), device="cuda", dtype=torch.float16)
    y, s = hb.fused_recurrent_output_prepare_raw(
        cu(r), cu(w_pre), cu(k), cu(v), cu(a_pre), cu(state), cu(g), cu(h(k_k)), cu(h(k_a)), cu(h(r_k)), cu(h(gw)), cu(h(gb)),
        eps=EPS, w_bias=cu(h(wb)), a_bias=cu(h(ab)), a_is_raw=True, v_first=cu(vf), v_gate=cu(vg_pre),
        v_gate_bias=cu(h(vb)), v_gate_is_raw=True, v_out=v_out)
    np.testing.assert_allclose(npf(v_out).reshape(B, Hh, N), v_mix.astype(np.float32), rtol=2e-3, atol=2e-3)
    np.testing.assert_allclose(npf(s), so, rtol=1e-2, atol=3e-3)
    np.testing.assert_allclose(npf(y), yo.astype(np.float32), rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("dt", ["fp32", "fp16"])
def test_scan_against_golden(dt):
    g = golden(f"ops_{dt}.npz")
    a = [cu(g[f"scan_{n}"]) for n in ("r", "w", "k", "v", "kk", "a", "state")]
    y, s = hb.fused_recurrent_scan(*a)
    np.testing.assert_allclose(npf(s), g["scan_state_out"], rtol=1e-4, atol=1e-4 if dt == "fp32" else 5e-3)
    np.testing.assert_allclose(npf(y), g["scan_y"].astype(np.float32), rtol=1e-4 if dt == "fp32" else 1e-2, atol=2e-4 if dt == "fp32" else 3e-2)
    yp, sp = hb.fused_recurrent_scan_output_prepare(*a, cu(g["scan_g"]), cu(g["step_r_k"]), cu(g["step_gn_w"]), cu(g["step_gn_b"]), eps=EPS)
    np.testing.assert_allclose(npf(yp), g["scanprep_y"].astype(np.float32), rtol=1e-3 if dt == "fp32" else 2e-2, atol=1e-3 if dt == "fp32" else 3e-2)
    assert torch.equal(sp, s)


@pytest.mark.parametrize("B,T,Hh", [(1, 1, 1), (2, 17, 3), (3, 33, 2), (2, 130, 4)])
def test_scan_against_oracle_ragged(B, T, Hh):
    r, w, k, v, kk, a = wkv_inputs(B, T, Hh, N, seed=T)
    rng = np.random.default_rng(T + 1)
    s0 = (0.1 * rng.standard_normal((B, Hh, N, N))).astype(np.float32)
    yo, so = O.recurrent_scan(r, w, k, v, kk, a, s0)
    y, s = hb.fused_recurrent_scan(*(cu(x) for x in (r, w, k, v, kk, a, s0)))
    assert rel_err(npf(s), so) < 2e-5
    np.testing.assert_allclose(npf(y), yo.astype(np.float32), rtol=4e-3, atol=4e-3)
    # T single-step calls == scan (config-2 protocol), final state relative error <= 1e-3
    st = cu(s0)
    ys = []
    for t in range(T):
        yt, st = hb.fused_recurrent_update(*(cu(x[:, t]) for x in (r, w, k, v, kk, a)), st)
        ys.append(yt)
    assert rel_err(npf(st), so) < 1e-3
    np.testing.assert_allclose(npf(torch.stack(ys, 1)), npf(y), rtol=4e-3, atol=4e-3)
    # decay given in the activation dtype, and raw-w (clampw) variant
    y16, s16 = hb.fused_recurrent_scan(cu(r), cu(w.astype(np.float16)), *(cu(x) for x in (k, v, kk, a, s0)))
    yo16, so16 = O.recurrent_scan(r, w.astype(np.float16), k, v, kk, a, s0)
    assert rel_err(npf(s16), so16) < 2e-5
    w_raw = rng.standard_normal((B, T, Hh, N)).astype(np.float16)
    yc, sc = hb.fused_recurrent_scan_clampw(cu(r), cu(w_raw), *(cu(x) for x in (k, v, kk, a, s0)))
    wd = np.exp(-0.606531 * O.sigmoid(w_raw.astype(np.float32)))
    yoc, soc = O.recurrent_scan(r, wd, k, v, kk, a, s0)
    assert rel_err(npf(sc), soc) < 2e-5


@pytest.mark.parametrize("B,T,Hh", [(1, 9, 148), (1, 16, 149), (2, 7, 148), (3, 17, 99)])
def test_scan_tile_choice_by_grid(B, T, Hh):
    """148 / 149 / 296 / 297 CTAs are the edges between the register tiles; T around the block of 8 tokens.  Decays of
    zero and above one are legal operands.  fp32 sums of 64 terms: 2e-6 of the largest value is about 30 ulp."""
    r, w, k, v, kk, a = wkv_inputs(B, T, Hh, N, seed=T, dtype=np.float32)
    w[:, 1, 0], w[:, 2, -1] = 0.0, 1.5
    rng = np.random.default_rng(T)
    s0 = (0.1 * rng.standard_normal((B, Hh, N, N))).astype(np.float32)
    yo, so = O.recurrent_scan(r, w, k, v, kk, a, s0)
    y, s = hb.fused_recurrent_scan(*(cu(x) for x in (r, w, k, v, kk, a, s0)))
    assert rel_err(npf(s), so) < 2e-6
    assert rel_err(npf(y), yo.astype(np.float32)) < 2e-6
    f = lambda *sh: rng.standard_normal(sh).astype(np.float32)
    g, rk, gw, gb = f(B, T, Hh, N), 0.1 * f(Hh, N), 1 + 0.1 * f(Hh * N), 0.1 * f(Hh * N)
    yp, sp = hb.fused_recurrent_scan_output_prepare(*(cu(x) for x in (r, w, k, v, kk, a, s0, g, rk, gw, gb)), eps=EPS)
    assert torch.equal(sp, s)
    rows = lambda x: cu(x).reshape(B * T, Hh * N)
    want = hb.fused_attn_output_prepare(y.reshape(B * T, Hh * N), *(rows(x) for x in (r, k, v, g)), *(cu(x) for x in (rk, gw, gb)),
                                        num_heads=Hh, head_dim=N, head_v_dim=N, eps=EPS)
    assert rel_err(npf(yp).reshape(-1), npf(want).reshape(-1)) < 5e-6
    # a state in fp16: the same recurrence on the rounded state, rounded back once
    s16 = s0.astype(np.float16)
    yh, sh = hb.fused_recurrent_scan(*(cu(x.astype(np.float16)) for x in (r, w, k, v, kk, a, s16)))
    _, soh = O.recurrent_scan(*(x.astype(np.float16) for x in (r, w, k, v, kk, a)), s16.astype(np.float32))
    assert sh.dtype == torch.float16 and rel_err(npf(sh), soh) < 1e-3


@pytest.mark.parametrize("Hh", [2, 149])
@pytest.mark.parametrize("T", [8, 40, 41, 47, 48, 81])
def test_scan_in_pieces_is_the_scan(T, Hh):
    """Blocks of 8 tokens in a ring of five: a token's place in it is no part of its arithmetic (the same bits), whether its block
    is whole, the last one, or behind others.  Against the oracle as in the test above."""
    r, w, k, v, kk, a = wkv_inputs(1, T, Hh, N, seed=T, dtype=np.float32)
    rng = np.random.default_rng(T)
    f = lambda *sh: rng.standard_normal(sh).astype(np.float32)
    seq, s0 = [cu(x) for x in (r, w, k, v, kk, a)], 0.1 * f(1, Hh, N, N)
    g, rk, gw, gb = cu(f(1, T, Hh, N)), cu(0.1 * f(Hh, N)), cu(1 + 0.1 * f(Hh * N)), cu(0.1 * f(Hh * N))
    y, s = hb.fused_recurrent_scan_output_prepare(*seq, cu(s0), g, rk, gw, gb, eps=EPS)
    _, so = O.recurrent_scan(r, w, k, v, kk, a, s0)
    assert rel_err(npf(s), so) < 2e-6
    for cut in (1, 3, 7):
        state, ys = cu(s0), []
        for t0, t1 in ((0, cut), (cut, T)):
            yt, state = hb.fused_recurrent_scan_output_prepare(*(x[:, t0:t1].contiguous() for x in seq), state, g[:, t0:t1].contiguous(), rk, gw, gb, eps=EPS)
            ys.append(yt)
        assert torch.equal(torch.cat([x.reshape(-1) for x in ys]), y.reshape(-1)) and torch.equal(state, s)


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T", [193, 200, 201, 208, 264])
@pytest.mark.parametrize("Hh", [1, 148])
def test_scan_of_many_tokens_is_the_scan_of_few(dt, T, Hh):
    """Five blocks of operands in flight from 193 tokens on, three up to there: the bits of the same tokens in shorter calls, which the tests
    above compare with the oracle."""
    gen = torch.Generator(device="cuda").manual_seed(T)
    f = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    r, k, v, a, g = (f(1, T, Hh, N).to(dt) for _ in range(5))
    seq = (r, torch.sigmoid(f(1, T, Hh, N)), k, v, torch.nn.functional.normalize(k.float(), dim=-1).to(dt), torch.sigmoid(a.float()).to(dt))
    s0, par = 0.1 * f(1, Hh, N, N), [f(Hh, N).to(dt), f(Hh * N).to(dt), f(Hh * N).to(dt)]
    y, s = hb.fused_recurrent_scan_output_prepare(*seq, s0, g, *par, eps=EPS)
    assert bool(torch.isfinite(y).all()) and bool(torch.isfinite(s).all())
    state, ys = s0, []
    for t0, t1 in ((0, 1), (1, 100), (100, T)) if T > 193 else ((0, 1), (1, T)):
        yt, state = hb.fused_recurrent_scan_output_prepare(*(x[:, t0:t1].contiguous() for x in seq), state, g[:, t0:t1].contiguous(), *par, eps=EPS)
        ys.append(yt)
    assert torch.equal(torch.cat([x.reshape(-1) for x in ys]), y.reshape(-1)) and torch.equal(state, s)


@pytest.mark.parametrize("dt", ["fp16", "bf16", "fp32"])
@pytest.mark.parametrize("Hh", [3, 149, 297])
def test_scan_parameters_of_any_alignment(dt, Hh):
    """r_k and the GroupNorm parameters as views into one flat buffer at odd element offsets (3 / 149 / 297 CTAs: the
    three register tiles): the bits of the aligned call."""
    td = dict(TD, bf16=torch.bfloat16)[dt]
    gen = torch.Generator(device="cuda").manual_seed(Hh)
    f = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    T = 9
    r, k, v, g = (f(1, T, Hh, N).to(td) for _ in range(4))
    kk = torch.nn.functional.normalize(k.float(), dim=-1).to(td)
    w, a, s0 = torch.sigmoid(f(1, T, Hh, N)), torch.sigmoid(f(1, T, Hh, N)).to(td), f(1, Hh, N, N)
    size = Hh * N
    for off in (1, 3, 8):
        flat = f(3 * (size + 8) + off).to(td)
        views = [flat[off + i * (size + (1, 8, 2)[i]):][:size] for i in range(3)]
        assert off == 8 or any(p.data_ptr() % 16 for p in views)
        got = hb.fused_recurrent_scan_output_prepare(r, w, k, v, kk, a, s0, g, *views, eps=EPS)
        want = hb.fused_recurrent_scan_output_prepare(r, w, k, v, kk, a, s0, g, *(p.clone() for p in views), eps=EPS)
        assert all(torch.equal(x, y) for x, y in zip(got, want))


@pytest.mark.parametrize("Hh,sd", [(3, torch.float32), (149, torch.float16), (300, torch.float32)])
def test_scan_in_place_is_the_scan(Hh, sd):
    """The final state over the first one: the same bits as in a buffer of its own; a strided state is left alone."""
    from hf_adapter_b200.recurrent import scan_output_prepare_inplace
    T = 19
    rng = np.random.default_rng(Hh)
    f = lambda *sh: cu(rng.standard_normal(sh).astype(np.float16))
    seq = [cu(x) for x in wkv_inputs(1, T, Hh, N, seed=Hh)]
    seq[1] = seq[1].to(torch.float16)
    rest = f(1, T, Hh, N), 0.1 * f(Hh, N), f(Hh * N), f(Hh * N)
    s0 = (0.1 * f(2, Hh, N, N).float()).to(sd)
    want, final = hb.fused_recurrent_scan_output_prepare(*seq, s0[:1], *rest, eps=EPS)
    state = s0[:1].clone()
    got, same = scan_output_prepare_inplace(*seq, state, *rest, eps=EPS)
    assert same is state and torch.equal(got, want) and torch.equal(state, final)
    strided = s0[:1].transpose(2, 3).contiguous().transpose(2, 3)
    got, other = scan_output_prepare_inplace(*seq, strided, *rest, eps=EPS)
    assert other is not strided and torch.equal(got, want) and torch.equal(other, final) and torch.equal(strided, s0[:1])


def test_scan_in_place_is_a_change_of_the_state():
    """A backward pass through something that saved the state before a prefill moved it on is refused, not silently wrong."""
    from hf_adapter_b200.recurrent import scan_output_prepare_inplace
    T = 5
    f = lambda *sh: torch.randn(*sh, device="cuda", dtype=torch.float16)
    state, weight = torch.randn(1, 3, N, N, device="cuda"), torch.ones((), device="cuda", requires_grad=True)
    loss = (state * weight).sum()
    with torch.no_grad():
        _, same = scan_output_prepare_inplace(*(f(1, T, 3, N) for _ in range(6)), state, f(1, T, 3, N), f(3, N), f(3 * N), f(3 * N), eps=EPS)
    assert same is state
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        loss.backward()


def test_scan_empty_sequence_passes_state_through():
    s0 = torch.randn(2, 2, N, N, device="cuda")
    e = torch.empty(2, 0, 2, N, device="cuda", dtype=torch.float16)
    y, s = hb.fused_recurrent_scan(e, e.float(), e, e, e, e, s0)
    assert tuple(y.shape) == (2, 0, 2, N) and torch.equal(s, s0)


@pytest.mark.parametrize("dt", ["fp32", "fp16"])
def test_norm_mix_lora_prep_against_golden(dt):
    g = golden(f"ops_{dt}.npz")
    t = {k: cu(v) for k, v in g.items()}
    prev = t["mix_prev"].clone()
    outs = hb.fused_attn_norm_mix6_decode(t["mix_x"], prev, t["mix_nw"], t["mix_nb"], *t["mix_mixes"])
    np.testing.assert_allclose(npf(torch.stack(outs)), g["mix_outs"].astype(np.float32), **tol(dt))
    np.testing.assert_allclose(npf(prev), g["mix_prev_out"].astype(np.float32), **tol(dt))
    for kw in ({"stack_rkv": True}, {"stack_wav": True}, {"stack_rkv_wagv": True}):
        prev2 = t["mix_prev"].clone()
        outs2 = hb.fused_attn_norm_mix6_decode(t["mix_x"], prev2, t["mix_nw"], t["mix_nb"], *t["mix_mixes"], **kw)
        assert all(torch.equal(a, b) for a, b in zip(outs, outs2))
    prev = t["mix_prev"].clone()
    x, mixed = hb.fused_ffn_add_norm_mix_decode(t["mix_x"], t["ffnmix_attn"], prev, t["mix_nw"], t["mix_nb"], t["mix_mixes"][0])
    np.testing.assert_allclose(npf(x), g["ffnmix_res_out"].astype(np.float32), **tol(dt))
    np.testing.assert_allclose(npf(mixed), g["ffnmix_mixed"].astype(np.float32), **tol(dt, 3))
    np.testing.assert_allclose(npf(prev), g["ffnmix_prev_out"].astype(np.float32), **tol(dt, 3))
    seq = hb.fused_attn_sequence_shift_mix(t["seqmix_x"], t["seqmix_prev"], *t["mix_mixes"])
    np.testing.assert_allclose(npf(torch.stack(seq[:6])), g["seqmix_outs"].astype(np.float32), **tol(dt))
    assert torch.equal(seq[6], t["seqmix_next"])
    one, nxt = hb.fused_ffn_sequence_shift_mix(t["seqmix_x"], t["seqmix_prev"], t["mix_mixes"][2])
    assert torch.equal(one, seq[2]) and torch.equal(nxt, seq[6])
    w, a, gg, vg = hb.fused_wavg_lora(t["lora_xw"], t["lora_xa"], t["lora_xg"], t["lora_xv"], t["lora_wd"], t["lora_ad"],
                                      t["lora_gd"], t["lora_vd"], t["lora_wu"], t["lora_au"], t["lora_gu"], t["lora_vu"],
                                      t["lora_wb"], t["lora_ab"], None, t["lora_vb"])
    for mine, ref in ((w, "lora_w"), (a, "lora_a"), (gg, "lora_g"), (vg, "lora_vgate")):
        np.testing.assert_allclose(npf(mine), g[ref].astype(np.float32), **tol(dt, 2))
    pw, pk, pv, pkk = hb.fused_prefill_state_prep(t["sp_w_raw"], t["sp_k_raw"], t["sp_v_raw"], t["sp_a"], t["raw_k_k"], t["raw_k_a"],
                                                  v_first=t["sp_vf"], v_gate=t["sp_vg"], num_heads=H, head_dim=N)
    np.testing.assert_allclose(npf(pw), g["sp_w"], rtol=1e-5, atol=1e-6)
    for mine, ref in ((pk, "sp_k"), (pv, "sp_v"), (pkk, "sp_kk")):
        np.testing.assert_allclose(npf(mine), g[ref].astype(np.float32), **tol(dt))
    op = hb.fused_attn_output_prepare(t["op_rec"], t["op_r"], t["op_k"], t["op_v"], t["op_g"], t["step_r_k"], t["step_gn_w"],
                                      t["step_gn_b"], num_heads=H, head_dim=N, head_v_dim=N, eps=EPS)
    np.testing.assert_allclose(npf(op), g["op_out"].astype(np.float32), **tol(dt, 5))


@pytest.mark.parametrize("D", [64, 2048, 2056, 4104, 8192])
def test_norm_mix_rows_do_not_depend_on_their_number(D):
    """fp32 reads the shift state after the row statistics below 512 rows and with the row from there on: the same bits."""
    gen = torch.Generator(device="cuda").manual_seed(D)
    f = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x, attn, prev, w, b, mixes = f(512, D), f(512, D), f(512, D), f(D), f(D), [f(D) for _ in range(6)]
    got = []
    for n in (512, 511):
        p1, p2 = prev[:n].clone(), prev[:n].clone()
        got.append([*hb.fused_attn_norm_mix6_decode(x[:n], p1, w, b, *mixes),
                    *hb.fused_ffn_add_norm_mix_decode(x[:n], attn[:n], p2, w, b, mixes[0]), p1, p2])
    assert all(torch.equal(a[:511], c) for a, c in zip(*got))
    h = torch.nn.functional.layer_norm(x.double(), (D,), w.double(), b.double(), 1e-5)
    # fp32 sums of up to 8192 terms and a cancelling centre: 1e-5 of the largest value is some 80 ulp
    assert float((got[0][0].double() - (h + (prev - h) * mixes[0].double())).abs().max()) < 1e-5 * float(got[0][0].abs().max())


@pytest.mark.parametrize("rows,D", [(1, 8), (5, 768), (64, 4096), (3, 8192)])
def test_norm_mix_shapes(rows, D):
    rng = np.random.default_rng(D)
    f = lambda *s: rng.standard_normal(s).astype(np.float16)
    x, prev, attn = f(rows, D), f(rows, D), f(rows, D)
    nw, nb = (1 + 0.1 * f(D)).astype(np.float16), (0.1 * f(D)).astype(np.float16)
    mixes = [rng.random(D).astype(np.float16) for _ in range(6)]
    (outs_o, prev_o) = O.attn_norm_mix6_decode(x, prev, nw, nb, mixes)
    pv = cu(prev)
    outs = hb.fused_attn_norm_mix6_decode(cu(x), pv, cu(nw), cu(nb), *(cu(m) for m in mixes))
    np.testing.assert_allclose(npf(torch.stack(outs)), np.stack(outs_o).astype(np.float32), rtol=4e-3, atol=4e-3)
    np.testing.assert_allclose(npf(pv), prev_o.astype(np.float32), rtol=4e-3, atol=4e-3)
    xo, mo, po = O.ffn_add_norm_mix_decode(x, attn, prev, nw, nb, mixes[0])
    pv = cu(prev)
    xg, mg = hb.fused_ffn_add_norm_mix_decode(cu(x), cu(attn), pv, cu(nw), cu(nb), cu(mixes[0]))
    np.testing.assert_allclose(npf(xg), xo.astype(np.float32), rtol=2e-3, atol=2e-3)
    np.testing.assert_allclose(npf(mg), mo.astype(np.float32), rtol=4e-3, atol=6e-3)
    ln = hb.layer_norm(cu(x), cu(nw), cu(nb))
    np.testing.assert_allclose(npf(ln), O.layer_norm(x, nw, nb).astype(np.float32), rtol=4e-3, atol=4e-3)


@pytest.mark.parametrize("M", [1, 5, 64, 130])
def test_grouped_lora_gemm_against_oracle(M):
    """The one-launch grouped projection (tensor-core MMA, cluster split-K) for decode-size LoRA shapes."""
    from hf_adapter_b200.lora import small_gemm_group
    rng = np.random.default_rng(M)
    D, A = 4096, 512
    ranks = (64, 64, 128, 32)
    f = lambda *s, sc=1.0: (sc * rng.standard_normal(s)).astype(np.float16)
    xs = [f(M, D) for _ in ranks]
    downs = [f(r, D, sc=0.02) for r in ranks]
    ups = [f(A, r, sc=0.1) for r in ranks]
    biases = [f(A, sc=0.5), f(A, sc=0.5), None, f(A, sc=0.5)]
    wo, ao, go, vo = O.wavg_lora(xs[0], xs[1], xs[2], xs[3], downs, ups, biases)
    w, a, g, v = hb.fused_wavg_lora(*(cu(x) for x in xs), *(cu(d) for d in downs), *(cu(u) for u in ups),
                                    *(None if b is None else cu(b) for b in biases))
    for mine, ref in ((w, wo), (a, ao), (g, go), (v, vo)):
        np.testing.assert_allclose(npf(mine), ref.astype(np.float32), rtol=4e-3, atol=4e-3)
    again = hb.fused_wavg_lora(*(cu(x) for x in xs), *(cu(d) for d in downs), *(cu(u) for u in ups),
                               *(None if b is None else cu(b) for b in biases))
    assert all(torch.equal(p, q) for p, q in zip((w, a, g, v), again))
    # odd output width / K not a multiple of the 64-wide chunk
    x1, w1, b1 = f(M, 72), f(40, 72, sc=0.1), f(40)
    (y1,) = small_gemm_group((cu(x1),), (cu(w1),), (cu(b1),), acts=(1,))
    ref = np.tanh((x1.astype(np.float32) @ w1.astype(np.float32).T + b1.astype(np.float32)).astype(np.float16).astype(np.float32))
    np.testing.assert_allclose(npf(y1), ref, rtol=4e-3, atol=4e-3)


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M", [1, 65, 14300])  # (14300: more CTAs of a K above 128 than one wave, which take a ring of three)
@pytest.mark.parametrize("K,Nout", [((72,), (41,)), ((328, 328), (40, 1)), ((520,), (64,)), ((520, 520, 520), (66, 65, 2)),
                                    ((4104,), (41,)), ((4104, 72, 8), (40, 41, 1)), ((4104, 4096), (64, 32))])
def test_grouped_lora_gemm_odd_widths_and_ragged_k(dt, M, K, Nout):
    """Widths that are not pairs (one of a group makes all of it store by element), rows that end in the middle of a pair, K that
    ends in the middle of a chunk on the deep ring, with and without split K, and shares of K that are empty.  fp32 sums of exact
    products: K units of 2^-24 of the sum of magnitudes, then one rounding.  Nothing behind an output is written, nothing behind a
    bias counts."""
    from hf_adapter_b200.lora import small_gemm_group
    g = torch.Generator(device="cuda").manual_seed(M + sum(K) + sum(Nout))
    n = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dt)
    xs, ws = [n(M, k) for k in K], [n(o, k) for k, o in zip(K, Nout)]
    biases = [torch.cat([n(o), torch.full((8,), float("nan"), device="cuda", dtype=dt)])[:o] for o in Nout]
    flat = [torch.full((M * o + 8,), 7.0, device="cuda", dtype=dt) for o in Nout]
    small_gemm_group(xs, ws, biases, outs=[f[:M * o].view(M, o) for f, o in zip(flat, Nout)])
    for f, y in zip(flat, small_gemm_group(xs, ws, biases, lean=True)):  # the shallow ring: the same sums
        assert torch.equal(y.reshape(-1), f[:y.numel()])
    for x, w, b, f, k, o in zip(xs, ws, biases, flat, K, Nout):
        assert bool((f[M * o:] == 7.0).all())
        ref = x.double() @ w.double().T + b.double()
        room = torch.finfo(dt).eps * ref.abs() + k * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T + b.double().abs())
        assert bool(((f[:M * o].view(M, o).double() - ref).abs() <= room).all())


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,T,D", [(1, 1, 8), (2, 3, 264), (3, 37, 768), (2, 5, 4096), (1, 9, 4104), (2, 2, 8192), (1, 1537, 4096),
                                   (1, 768, 4096), (1, 769, 4096), (1, 128, 8192), (1, 129, 8192)])
def test_sequence_norm_mix(dt, B, T, D):
    """LayerNorm and token-shift mixes in one call, either side of the size at which one kernel becomes two and of the row
    width at which a thread takes two vectors, against 64 bits on the rounded rows.  The kernel's row may round the other way
    (one unit of this row and of the one before), and the mix rounds once."""
    from hf_adapter_b200 import norm_mix as NM
    g = torch.Generator(device="cuda").manual_seed(B * T + D)
    n = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dt)
    x, prev, w, b = n(B, T, D), n(B, D), n(D), n(D)
    mixes = [torch.rand(D, generator=g, device="cuda").to(dt) for _ in range(6)]
    xd = x.double()
    h = (xd - xd.mean(-1, keepdim=True)) * torch.rsqrt(xd.var(-1, unbiased=False, keepdim=True) + 1e-5) * w.double() + b.double()
    hr = h.to(dt).double()
    before = torch.cat([prev.double()[:, None], hr[:, :-1]], 1)
    eps = max(torch.finfo(dt).eps, 2e-6)  # fp32: the statistics of a row
    room = 2 * eps * (h.abs() + before.abs() + w.double().abs() + b.double().abs())
    for k in (6, 1):
        outs, nxt = NM.sequence_norm_mix(x, prev, w, b, mixes[:k])
        for o, m in zip(outs, mixes):
            assert ((o.double() - (hr + (before - hr) * m.double())).abs() <= room).all()
        assert ((nxt.double() - hr[:, -1]).abs() <= room[:, -1]).all()


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,T,D,piece", [(3, 148, 2560, 90), (3, 149, 2560, 91), (297, 3, 2560, 1), (1, 2963, 768, 100), (1, 297, 4096, 99), (2, 149, 3072, 61),
                                         (1, 8193, 4096, 256)])
def test_sequence_norm_mix_of_two_tokens_a_cta(dt, B, T, D, piece):
    """Either side of the row counts at which a CTA takes two tokens, odd lengths and sequences of three among them, and of the sizes at
    which one kernel becomes two: a long call gives the bits of short ones (one token a CTA) that carry the state."""
    from hf_adapter_b200 import norm_mix as NM
    g = torch.Generator(device="cuda").manual_seed(B * T + D)
    n = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dt)
    x, state, w, b = n(B, T, D), n(B, D), n(D), n(D)
    mixes = [torch.rand(D, generator=g, device="cuda").to(dt) for _ in range(6)]
    for k in (6, 1):
        one = NM._one_kernel(B * T, T, D, dt, k)
        outs, nxt = NM.sequence_norm_mix(x, state, w, b, mixes[:k])
        carried, parts = state, []
        for t in range(0, T, piece):
            got, carried = NM.sequence_norm_mix(x[:, t:t + piece].contiguous(), carried, w, b, mixes[:k])
            parts.append(got)
        whole = [torch.cat(p, 1) for p in zip(*parts)]
        if one:
            assert torch.equal(carried, nxt) and all(torch.equal(p.reshape(-1), q.reshape(-1)) for p, q in zip(whole, outs))
        else:  # two kernels: the row's statistics in another order, so a unit of the rounded rows, as in the test above
            eps = max(torch.finfo(dt).eps, 2e-6)
            assert all(((p.reshape(-1).float() - q.reshape(-1).float()).abs() <= 4 * eps * (8 + q.reshape(-1).float().abs())).all() for p, q in zip(whole, outs))


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,T,D,piece", [(1, 555, 2560, 222), (1, 556, 2560, 139), (1, 888, 2560, 222), (1, 889, 2560, 127), (1, 1333, 2560, 333), (1, 1777, 2560, 355),
                                         (149, 3, 2560, 1), (112, 5, 2560, 3), (280, 3, 4096, 1)])
def test_sequence_norm_mix_either_side_of_its_waves(dt, B, T, D, piece):
    """Six mixes in two tokens a CTA from 1.25 waves to two and from three on (fp32: four); sequences of 3 and 5, one token a CTA or two
    kernels: the bits of short calls that carry the state, as in the test above."""
    test_sequence_norm_mix_of_two_tokens_a_cta(dt, B, T, D, piece)


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,Hh", [(1, 1), (33, 1), (4095, 3), (12287, 1), (12288, 1), (4099, 3)])
def test_state_prep_either_side_of_its_two_forms(dt, rows, Hh):
    """8- and 16-byte pieces a lane (they change at 12288 heads) against 64 bits.  Each result is rounded once from fp32 arithmetic of a
    few steps: one unit of its type (below its smallest normal number the spacing stays tiny * eps), and in fp32 (gates and norms in
    two and more roundings) eight."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    n = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dt)
    w, k, v, a, vf, vg = (n(rows, Hh * N) for _ in range(6))
    ks, ka = n(Hh * N), n(Hh * N)
    got = hb.fused_prefill_state_prep(w, k, v, a, ks, ka, v_first=vf, v_gate=vg, num_heads=Hh, head_dim=N, a_is_raw=True, v_gate_is_raw=True)
    wd, kd, vd, ad, vfd, vgd, ksd, kad = (t.double() for t in (w, k, v, a, vf, vg, ks, ka))
    gate = torch.sigmoid(ad)
    kk = torch.nn.functional.normalize((kd * ksd).view(rows, Hh, N), dim=-1).view(rows, -1)
    ref = (torch.exp(-0.606531 * torch.sigmoid(wd)), kd * (1 + (gate - 1) * kad), vd + (vfd - vd) * torch.sigmoid(vgd), kk)
    size = (torch.ones_like(wd), kd.abs() * (1 + kad.abs()), vd.abs() + (vfd - vd).abs(), kk.abs())  # of the terms that are added
    for y, r, s in zip(got, ref, size):
        info = torch.finfo(y.dtype)
        assert bool(((y.double() - r).abs() <= (info.eps if y.dtype != torch.float32 else 8 * info.eps) * s + info.tiny * info.eps).all())


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,Hh", [(1, 1), (5, 3), (67, 12)])
def test_state_prep_returns_its_gate(dt, rows, Hh):
    """The fourth / fifth result of the prefill state prep is the gate it used: the sigmoid of raw ``a`` rounded once (one
    unit in the last place between two correct exponentials), ``a`` itself when it is no raw gate; the other results do not
    depend on whether it is asked for."""
    n = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dt)
    g = torch.Generator(device="cuda").manual_seed(rows)
    w, k, v, a, vf, vg = (n(rows, Hh * N) for _ in range(6))
    kk, ka = n(Hh * N), n(Hh * N)
    ulp = torch.finfo(dt).eps
    for first in (True, False):
        kw = dict(num_heads=Hh, head_dim=N, v_gate_is_raw=True, **({} if first else dict(v_first=vf, v_gate=vg)))
        for raw in (True, False):
            want = torch.sigmoid(a.float()).to(dt) if raw else a
            for fn, xs in ((hb.fused_prefill_kv_kk_prep, (k, v, a, kk, ka)), (hb.fused_prefill_state_prep, (w, k, v, a, kk, ka))):
                *rest, gate = fn(*xs, a_is_raw=raw, return_gate=True, **kw)
                assert ((gate.float() - want.float()).abs() <= ulp * want.float().abs()).all()
                assert all(torch.equal(p, q) for p, q in zip(rest, fn(*xs, a_is_raw=raw, **kw)))


@pytest.mark.parametrize("T", [16, 64, 80, 96, 112, 208])
def test_chunk_scan_ring_edges_with_raw_decay(T):
    """The chunked scan around the lengths of its pipeline (four warps prepare 16-token chunks in turn, six chunks in the ring),
    with the decay formed from raw logits in the kernel: against the sequential recurrence in 64 bits on the decay of those
    logits.  The bounds are the test below's: fp16 outputs, tf32 / fp16 operands of the products."""
    B, Hh = 2, 3
    r, w, k, v, kk, a = wkv_inputs(B, T, Hh, N, seed=T)
    rng = np.random.default_rng(T)
    w_raw = (2 * rng.standard_normal((B, T, Hh, N))).astype(np.float16)
    w = np.exp(-0.606531 / (1 + np.exp(-w_raw.astype(np.float64)))).astype(np.float32)
    s0 = (0.1 * rng.standard_normal((B, Hh, N, N))).astype(np.float32)
    yo, so = O.recurrent_scan(r, w, k, v, kk, a, s0, hi=True)
    y, s = hb.self_chunk_rwkv7(*[cu(x) for x in (r, w_raw, k, v, kk, a, s0)], chunk_size=16, w_is_raw=True)
    assert rel_err(npf(s), so) < 1e-3
    assert rel_err(npf(y), yo.astype(np.float32)) < 2e-3


@pytest.mark.parametrize("B,T,Hh,chunk", [(1, 64, 1, 64), (2, 128, 3, 16), (2, 192, 2, 32), (1, 1024, 2, 64)])
def test_chunk_scan_tensor_core_against_oracle(B, T, Hh, chunk):
    """Tensor-core chunked WY scan == the sequential recurrence (fp64 oracle on the same fp16 inputs):
    state relative error <= 1e-3, outputs within fp16 tolerance, no bounded wait gave up."""
    from hf_adapter_b200 import _lib
    r, w, k, v, kk, a = wkv_inputs(B, T, Hh, N, seed=T + chunk)
    rng = np.random.default_rng(T)
    s0 = (0.1 * rng.standard_normal((B, Hh, N, N))).astype(np.float32)
    yo, so = O.recurrent_scan(r, w, k, v, kk, a, s0, hi=True)
    _lib.kernel_status(True)
    args = [cu(x) for x in (r, w, k, v, kk, a, s0)]
    y, s = hb.self_chunk_rwkv7(*args, chunk_size=chunk)
    assert _lib.kernel_status(True) == 0
    assert rel_err(npf(s), so) < 1e-3
    scale = max(1.0, float(np.abs(yo.astype(np.float32)).max()))
    np.testing.assert_allclose(npf(y), yo.astype(np.float32), rtol=4e-3, atol=4e-3 * scale)
    assert rel_err(npf(y), yo.astype(np.float32)) < 2e-3
    y2, s2 = hb.dplr_chunk_scan(*args, chunk_size=chunk, algorithm="wy")
    assert torch.equal(y2, y) and torch.equal(s2, s)
    # the sequential kernel and the chunked kernel agree with each other as well
    y3, s3 = hb.fused_recurrent_scan(*args)
    assert rel_err(npf(s3), npf(s)) < 1e-3
    # decay in the activation dtype / raw w
    y16, s16 = hb.self_chunk_rwkv7(args[0], cu(w.astype(np.float16)), *args[2:], chunk_size=chunk)
    yo16, so16 = O.recurrent_scan(r, w.astype(np.float16), k, v, kk, a, s0, hi=True)
    assert rel_err(npf(s16), so16) < 1e-3
    with pytest.raises(ValueError):
        hb.self_chunk_rwkv7(*args, chunk_size=48)


def test_chunk_scan_single_chunk_error_against_64_bits():
    """One chunk of 16 tokens: the state no further from a float64 recurrence than with the 64-token tiles of the former kernel
    (1.5954e-4 over these inputs; 1.617e-4 with a chunk's operands scaled to its start, 1.581e-4 scaled to its end)."""
    errors = []
    for seed in range(8):
        g = torch.Generator(device="cuda").manual_seed(100 * seed + 16)
        n = lambda: torch.randn(4, 16, 40, N, generator=g, device="cuda")
        r, k, v = n().half(), n().half(), n().half()
        kk, a = torch.nn.functional.normalize(k.float(), dim=-1).half(), torch.sigmoid(n()).half()
        w = torch.exp(-0.606531 * torch.sigmoid(n().half().float()))
        s = torch.zeros(4, 40, N, N, device="cuda")
        _, got = hb.self_chunk_rwkv7(r, w, k, v, kk, a, s, chunk_size=16)
        s = s.double()
        for t in range(16):
            kd, vd, kkd, ad, wd = (x[:, t].double() for x in (k, v, kk, a, w))
            s = s * wd.unsqueeze(-2) - (s @ kkd.unsqueeze(-1)) * (kkd * ad).unsqueeze(-2) + vd.unsqueeze(-1) * kd.unsqueeze(-2)
        errors.append(float((got.double() - s).norm() / s.norm()))
    assert sum(errors) / len(errors) < 1.5955e-4


def test_chunk_scan_raw_decay_does_not_drift():
    """A state that is only decayed, by raw logits of about -6 over 8192 tokens.  A chunk's factor and its product with the state
    are rounded to nearest, half a unit each with either sign; allowed is a bias of a quarter unit for each of the 512 chunks."""
    g = torch.Generator(device="cuda").manual_seed(1)
    raw = (0.5 * torch.randn(1, 8192, 8, N, generator=g, device="cuda") - 6).half()
    s0 = torch.randn(1, 8, N, N, generator=g, device="cuda") + 2
    z = torch.zeros_like(raw)
    _, got = hb.self_chunk_rwkv7(z, raw, z, z, z, z, s0.clone(), chunk_size=16, w_is_raw=True)
    exact = s0.double() * torch.exp(-0.606531 * torch.sigmoid(raw.double()).sum(1)).unsqueeze(-2)
    assert abs(float(((got.double() - exact) / exact).mean())) < 512 * 2.0 ** -24 / 4


@pytest.mark.parametrize("f32", [False, True])
def test_chunk_scan_strong_decays(f32):
    """Decays down to the smallest that the chunked form admits (2^-6.85 for all 16 tokens of a chunk in some channels, anything
    above it in the others), against a float64 recurrence; the bounds of the other chunked tests."""
    g = torch.Generator(device="cuda").manual_seed(3)
    B, T, Hh = 2, 64, 3
    n = lambda: torch.randn(B, T, Hh, N, generator=g, device="cuda")
    r, k, v = n().half(), n().half(), n().half()
    kk, a = torch.nn.functional.normalize(k.float(), dim=-1).half(), torch.sigmoid(n()).half()
    log2 = -6.85 * torch.rand(B, T, Hh, N, generator=g, device="cuda")
    log2[..., ::8] = -6.85
    w = torch.exp2(log2) if f32 else torch.exp2(log2).half()
    s0 = torch.randn(B, Hh, N, N, generator=g, device="cuda")
    y, got = hb.self_chunk_rwkv7(r, w, k, v, kk, a, s0, chunk_size=16)
    s, ys = s0.double(), []
    for t in range(T):
        rd, kd, vd, kkd, ad, wd = (x[:, t].double() for x in (r, k, v, kk, a, w))
        s = s * wd.unsqueeze(-2) - (s @ kkd.unsqueeze(-1)) * (kkd * ad).unsqueeze(-2) + vd.unsqueeze(-1) * kd.unsqueeze(-2)
        ys.append((s @ rd.unsqueeze(-1)).squeeze(-1))
    assert rel_err(npf(got), npf(s)) < 1e-3
    assert rel_err(npf(y), npf(torch.stack(ys, 1))) < 2e-3


def test_scan_full_size_config2():
    """Isolated WKV-7 op at the benchmark's size (B8 T4096 H32 N64, zero state): chunked tensor-core scan vs the
    sequential kernel over all heads (state rel-err <= 1e-3, outputs <= 2e-3 relative), and both against the fp64
    oracle on a two-head slice (the oracle needs seconds per head at this length)."""
    B, T, Hh = 8, 4096, 32
    g = torch.Generator(device="cuda").manual_seed(0)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    r, k, v = (rn(B, T, Hh, N).half() for _ in range(3))
    kk = torch.nn.functional.normalize(k.float(), dim=-1).half()
    a = torch.sigmoid(rn(B, T, Hh, N)).half()
    w = torch.exp(-0.606531 * torch.sigmoid(rn(B, T, Hh, N)))
    s0 = torch.zeros(B, Hh, N, N, device="cuda")
    ys, ss = hb.fused_recurrent_scan(r, w, k, v, kk, a, s0)
    yc, sc = hb.self_chunk_rwkv7(r, w, k, v, kk, a, s0, chunk_size=64)
    assert rel_err(npf(sc), npf(ss)) < 1e-3
    assert rel_err(npf(yc), npf(ys)) < 2e-3
    sl = lambda t: t[:1, :, :2].contiguous().cpu().numpy()
    yo, so = O.recurrent_scan(sl(r), sl(w), sl(k), sl(v), sl(kk), sl(a), np.zeros((1, 2, N, N), np.float32), hi=True)
    for s_gpu, y_gpu in ((ss, ys), (sc, yc)):
        assert rel_err(npf(s_gpu[:1, :2]), so) < 1e-3
        assert rel_err(npf(y_gpu[:1, :, :2]), yo.astype(np.float32)) < 2e-3


def test_bf16_activations():
    """The CUDA-core kernels and the LoRA MMA kernel take bf16 storage as well (fp32 arithmetic inside)."""
    rng = np.random.default_rng(21)
    B, Hh, D = 3, 2, 256
    bf = lambda a: torch.from_numpy(np.asarray(a, np.float32)).cuda().to(torch.bfloat16)
    rt = lambda t: t.float().cpu().numpy()  # bf16-rounded values as fp32 for the oracle
    r, w_raw, k, v, g = (bf(rng.standard_normal((B, Hh, N))) for _ in range(5))
    a = bf(1 / (1 + np.exp(-rng.standard_normal((B, Hh, N)))))
    state = (0.3 * rng.standard_normal((B, Hh, N, N))).astype(np.float32)
    k_k, k_a = bf(0.85 + 0.1 * rng.standard_normal(Hh * N)), bf(1 + 0.1 * rng.standard_normal(Hh * N))
    r_k, gw, gb = bf(0.1 * rng.standard_normal((Hh, N))), bf(1 + 0.1 * rng.standard_normal(Hh * N)), bf(0.1 * rng.standard_normal(Hh * N))
    yo, so = O.recurrent_output_prepare_raw(rt(r), rt(w_raw), rt(k), rt(v), rt(a), state, rt(g), rt(k_k), rt(k_a), rt(r_k), rt(gw), rt(gb), EPS)
    y, s = hb.fused_recurrent_output_prepare_raw(r, w_raw, k, v, a, cu(state), g, k_k, k_a, r_k, gw, gb, eps=EPS)
    assert y.dtype == torch.bfloat16
    np.testing.assert_allclose(npf(s), so, rtol=2e-5, atol=2e-5)
    np.testing.assert_allclose(npf(y), yo, rtol=2e-2, atol=2e-2)
    x, prev = bf(rng.standard_normal((B, D))), bf(rng.standard_normal((B, D)))
    nw, nb = bf(1 + 0.1 * rng.standard_normal(D)), bf(0.1 * rng.standard_normal(D))
    mixes = [bf(rng.random(D)) for _ in range(6)]
    outs_o, prev_o = O.attn_norm_mix6_decode(rt(x), rt(prev), rt(nw), rt(nb), [rt(m) for m in mixes])
    pv = prev.clone()
    outs = hb.fused_attn_norm_mix6_decode(x, pv, nw, nb, *mixes)
    np.testing.assert_allclose(npf(torch.stack(outs)), np.stack(outs_o), rtol=2e-2, atol=2e-2)
    np.testing.assert_allclose(npf(pv), prev_o, rtol=2e-2, atol=2e-2)
    from hf_adapter_b200.lora import small_gemm_group
    W = bf(0.05 * rng.standard_normal((72, D)))
    (yl,) = small_gemm_group((x,), (W,), acts=(2,))
    ref = 1 / (1 + np.exp(-(rt(x) @ rt(W).T)))
    np.testing.assert_allclose(npf(yl), ref, rtol=2e-2, atol=2e-2)
    # scan in bf16 storage
    T = 20
    rs, ks, vs = (bf(rng.standard_normal((B, T, Hh, N))) for _ in range(3))
    kks = bf(rt(ks) / np.linalg.norm(rt(ks), axis=-1, keepdims=True))
    as_ = bf(1 / (1 + np.exp(-rng.standard_normal((B, T, Hh, N)))))
    ws = np.exp(-0.606531 / (1 + np.exp(-rng.standard_normal((B, T, Hh, N))))).astype(np.float32)
    yo2, so2 = O.recurrent_scan(rt(rs), ws, rt(ks), rt(vs), rt(kks), rt(as_), state)
    y2, s2 = hb.fused_recurrent_scan(rs, cu(ws), ks, vs, kks, as_, cu(state))
    assert rel_err(npf(s2), so2) < 2e-5
    np.testing.assert_allclose(npf(y2), yo2, rtol=2e-2, atol=3e-2)
