"""The few-row projection kernel against fp32 products of the same operands: edges of its channel tiles (16 / 32), of its K
units (64 dense, 128 quantised), of the warps and cluster ranks that split K, and of the 8 activation rows."""
import pytest
import torch

import hf_adapter_b200 as hb
from hf_adapter_b200 import _lib, rows
from hf_adapter_b200.packing import rows_projections

pytestmark = pytest.mark.gpu


def _close(got, want, dt, p=None):
    # one rounding of the product p to the storage type and one of the result, each half an ulp; the last term is the fp32
    # sum's own error and the type's smallest steps
    ulp = 2.0 ** -10 if dt == torch.float16 else 2.0 ** -7
    lim = 0.5 * ulp * (want.abs() + (want if p is None else p).abs()) * 1.01 + 1e-5
    assert bool(((got.float() - want).abs() <= lim).all()), float(((got.float() - want).abs() / lim).max())


@pytest.mark.parametrize("M", [1, 3, 8])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shapes", [[(8, 1), (32, 17), (72, 64), (520, 33), (1024, 130), (64, 2560), (128, 300)],
                                    [(10240, 48)], [(3080, 768), (768, 64)], [(768, 5000)]])
def test_dense_group_with_epilogues(M, dt, shapes):
    g = torch.Generator(device="cuda").manual_seed(M)
    epis = [0, 1, 2, 3, 4, 2, 0][:len(shapes)]
    xs = [torch.randn(M, K, generator=g, device="cuda").to(dt) for K, _ in shapes]
    ws = [(torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(dt) for K, N in shapes]
    res = [torch.randn(M, N, generator=g, device="cuda").to(dt) if e == 2 else None for (_, N), e in zip(shapes, epis)]
    for static in (False, True):
        outs = rows.rows_gemv(xs, ws, out_features=[N for _, N in shapes], fmts=[0] * len(xs), residuals=res, epilogues=epis,
                              static_weights=static)
        for x, w, r, e, y in zip(xs, ws, res, epis, outs):
            p = x.double() @ w.double().t()
            if e == 1:  # the product is rounded before it is squared, which doubles the relative size of that rounding
                ulp = 2.0 ** -10 if dt == torch.float16 else 2.0 ** -7
                torch.testing.assert_close(y.double(), torch.relu(p) ** 2, rtol=1.6 * ulp, atol=1e-5)
                continue
            want = p if e == 0 else p + r.double() if e == 2 else torch.tanh(p) if e == 3 else torch.sigmoid(p)
            _close(y, want.float(), dt, p.float())


@pytest.mark.parametrize("M", [1, 3, 8])
@pytest.mark.parametrize("K,N", [(128, 128), (256, 48), (1152, 200), (2560, 2560), (8192, 272)])
def test_quantised_formats(M, K, N):
    g = torch.Generator(device="cuda").manual_seed(K + M)
    x = torch.randn(M, K, generator=g, device="cuda").half()
    lin = torch.nn.Linear(K, N, bias=False, device="cuda", dtype=torch.float16)
    with torch.no_grad():
        lin.weight.normal_(0.0, K ** -0.5, generator=g)
    m4, m8 = hb.MM4Linear(lin), hb.MM8Linear(lin, rowwise=True)
    res = torch.randn(M, N, generator=g, device="cuda").half()
    p4 = (x.double() @ hb.w4_dequant(m4.packed_group, m4.group_scales, K).double().t()).float()
    p8 = (x.double() @ (m8.q_row.double() * m8.row_scale.double()[:, None]).t()).float()
    y4, y8 = rows.rows_gemv((x, x), (m4.tiled_for(x), m8.tiled_for(x)), out_features=(N, N), fmts=(1, 2), scales=(None, m8.row_scale),
                            residuals=(res, None), epilogues=(_lib.EPI_ADD, _lib.EPI_NONE))
    _close(y4, p4 + res.float(), torch.float16, p4)
    _close(y8, p8, torch.float16)
    # the modules give the same whichever kernel their row count and K select
    _close(m4.rwkv7_forward_add(x, res), p4 + res.float(), torch.float16, p4)
    _close(m8(x), p8, torch.float16)


def test_refusals():
    x, w = torch.zeros(9, 64, device="cuda").half(), torch.zeros(8, 64, device="cuda").half()
    with pytest.raises(ValueError):
        rows.rows_gemv((x,), (w,), out_features=(8,), fmts=(0,))
    with pytest.raises(ValueError):
        rows.rows_gemv((x[:1, :60].contiguous(),), (w,), out_features=(8,), fmts=(0,))
    assert not rows.takes_dense(x[:1].reshape(-1)[1:57].reshape(1, 56), torch.zeros(8, 56, device="cuda").half())  # misaligned


def test_operands_of_the_wrong_size_are_refused_on_the_host():
    """Each would be read or written out of range: the kernel has its sizes from x and out_features alone."""
    h = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.float16)
    u8 = lambda n: torch.zeros(n, device="cuda", dtype=torch.uint8)
    x, w = h(2, 128), h(16, 128)
    w4, w8 = int(_lib.lib.rwkv7_w4g_tiled_bytes(128, 16)), int(_lib.lib.rwkv7_w8_tiled_bytes(128, 16))
    ok = dict(out_features=(16,), fmts=(rows.DENSE,))
    for args, kw in [((h(15, 128),), {}), ((h(16, 64),), {}), ((w.float(),), {}), ((w.t().contiguous().t(),), {}),
                     ((u8(w4 - 1),), dict(fmts=(rows.INT4,))), ((u8(w8 - 1),), dict(fmts=(rows.INT8,), scales=(h(16),))),
                     ((u8(w8),), dict(fmts=(rows.INT8,), scales=(h(15),))), ((u8(w8),), dict(fmts=(rows.INT8,), scales=(h(16).float(),))),
                     ((u8(w8),), dict(fmts=(rows.INT8,))), ((u8(w4),), dict(fmts=(3,))),
                     ((w,), dict(residuals=(h(1, 16),), epilogues=(_lib.EPI_ADD,))),
                     ((w,), dict(residuals=(h(2, 16).float(),), epilogues=(_lib.EPI_ADD,))),
                     ((w,), dict(outs=(h(2, 15),))), ((w,), dict(outs=(h(2, 32)[:, ::2],))), ((w, w), {})]:
        with pytest.raises(ValueError):
            rows.rows_gemv((x,), args, **{**ok, **kw})
    assert rows.rows_gemv((x,), (w,), **ok)[0].shape == (2, 16)
    # a layer step does not hand the kernel activations of another width than the projection's
    m4 = hb.MM4Linear(torch.nn.Linear(128, 32, bias=False, device="cuda", dtype=torch.float16))
    assert rows_projections((m4,), (h(2, 256),)) is None and rows_projections((m4,), (h(2, 1, 128),)) is None
    assert rows_projections((m4,), (x,)) is not None
    with pytest.raises(ValueError):
        m4(h(2, 256))


@pytest.mark.parametrize("strided", [False, True])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_step_of_a_few_rows_is_the_step_of_many(strided, dt, monkeypatch):
    """Rows of a batch of 8 against the same rows in a batch of 9, which other kernels compute.  A layer with a strided LoRA "up"
    weight keeps the route of many rows, and nothing is launched for it and thrown away."""
    cfg = hb.NativeRWKV7Config(vocab_size=128, hidden_size=256, num_hidden_layers=2, num_heads=4, head_dim=64, intermediate_size=512,
                               decay_low_rank_dim=16, a_low_rank_dim=24, v_low_rank_dim=16, gate_low_rank_dim=32)
    torch.manual_seed(9)
    m = hb.RWKV7ForCausalLM(cfg).to(dt).cuda().eval()
    if strided:
        for layer in m.model.layers:
            up = layer.attn.a_lora.lora[2]
            up.weight = torch.nn.Parameter(up.weight.t().contiguous().t())
    launches = []
    real = rows.rows_gemv
    monkeypatch.setattr(rows, "rows_gemv", lambda xs, *a, **k: (launches.append(len(xs)), real(xs, *a, **k))[1])
    ids = torch.randint(0, 128, (9,), device="cuda")
    caches = [m.new_cache(b) for b in (8, 9)]
    for _ in range(3):
        few, many = (m.rwkv7_forward_token(ids[:b], c, use_graph=False) for b, c in zip((8, 9), caches))
    # r, k, v with the LoRA downs of a layer, then the ups
    assert [n for n in launches if n > 1] == ([] if strided else [6, 3, 7, 4] * 3)
    # two layers, three tokens: a few roundings to the activation type on either side
    ulp = 2.0 ** -11 if dt == torch.float16 else 2.0 ** -8
    for a, b in zip([few, *caches[0]._tensors()], [many, *caches[1]._tensors()]):
        a, b = a.float(), b[:8].float() if b.shape[0] == 9 else b.float()
        assert float((a - b).norm()) <= 4 * ulp * float(b.norm())


def test_products_that_something_follows_stay_visible():
    """Gradients, tangents, vmap and traces of a dense product of a few rows: those of the library GEMM, which it then is."""
    from torch.fx.experimental.proxy_tensor import make_fx
    from hf_adapter_b200.packing import apply_linear
    gen = torch.Generator(device="cuda").manual_seed(3)
    f = lambda *s: torch.randn(*s, generator=gen, device="cuda").half()
    x, w, res, t = f(4, 256), f(64, 256), f(4, 64), f(4, 256)
    plain = lambda a, b: torch.nn.functional.linear(a, b) + res
    ours = lambda a, b: apply_linear(b, a, residual=res)
    grads = []
    for fn in (plain, ours):
        a, b = x.clone().requires_grad_(), w.clone().requires_grad_()
        fn(a, b).float().square().sum().backward()
        grads.append((a.grad, b.grad))
    assert all(torch.equal(p, q) for p, q in zip(*grads))
    assert all(torch.equal(p, q) for p, q in zip(*(torch.func.jvp(lambda a: fn(a, w), (x,), (t,)) for fn in (plain, ours))))
    x3 = f(3, 4, 256)
    assert torch.equal(*(torch.func.vmap(lambda a: fn(a, w))(x3) for fn in (plain, ours)))
    g = make_fx(lambda a: ours(a, w))(x)
    assert torch.equal(g(t), plain(t, w))
    with torch.no_grad():  # nothing follows: one rounding of the product, one of the sum
        _close(ours(x, w), (x.double() @ w.double().t()).float() + res.float(), torch.float16, (x.double() @ w.double().t()).float())


@pytest.mark.parametrize("rows_,rank,dt", [(1, 24, torch.float16), (1024, 24, torch.bfloat16), (1025, 24, torch.float16), (8192, 24, torch.float16),
                                           (8193, 24, torch.bfloat16), (70, 20, torch.float16), (70, 24, torch.float32)])
@pytest.mark.parametrize("first", [False, True])
def test_prefill_lora_pairs(rows_, rank, dt, first):
    """Either side of the row counts up to which the pairs are grouped launches, a rank that those do not take, fp32."""
    from hf_adapter_b200.model import NativeRWKV7Attention, _prefill_lora
    cfg = hb.NativeRWKV7Config(vocab_size=16, hidden_size=128, num_hidden_layers=2, num_heads=2, head_dim=64, intermediate_size=256,
                               decay_low_rank_dim=64, a_low_rank_dim=rank, v_low_rank_dim=16, gate_low_rank_dim=72)
    torch.manual_seed(rows_ + rank)
    at = NativeRWKV7Attention(cfg, 1).cuda().to(dt)
    xs = [torch.randn(1, rows_, 128, device="cuda").to(dt) for _ in range(4)]
    with torch.no_grad():
        got = _prefill_lora(at, xs[0], xs[1], xs[2], None if first else xs[3])
        assert len(got) == 4 and (got[3] is None) == first
        same = lambda t: t
        for y, lora, x, act in zip(got, (at.w_lora, at.a_lora, at.g_lora, at.v_lora), xs, (torch.tanh, same, torch.sigmoid, same)):
            if y is None:
                continue
            l = lora.lora.double()
            want = l[2](act(l[0](x.double())))
            lora.to(dt)
            # the hidden value is rounded twice, the result once: each at most half an ulp of its size
            half_ulp = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -20}[dt]
            assert y.shape == want.shape and float((y.double() - want).norm()) <= 2 * half_ulp * float(want.norm())


@pytest.mark.parametrize("N", [9472, 9504, 18944, 18976, 28448])
@pytest.mark.parametrize("fmt", ["dense", "int8"])
def test_either_side_of_the_wave_limits(N, fmt):
    """CTAs of eight warps up to 296 tiles of 32 channels, of four up to 592 and from 889 on."""
    K, M = 512, 3
    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(M, K, generator=g, device="cuda").half()
    lin = torch.nn.Linear(K, N, bias=False, device="cuda", dtype=torch.float16)
    with torch.no_grad():
        lin.weight.normal_(0.0, K ** -0.5, generator=g)
    if fmt == "dense":
        y, = rows.rows_gemv((x,), (lin.weight,), out_features=(N,), fmts=(0,))
        p = x.double() @ lin.weight.double().t()
    else:
        m8 = hb.MM8Linear(lin, rowwise=True)
        y, = rows.rows_gemv((x,), (m8.tiled_for(x),), out_features=(N,), fmts=(2,), scales=(m8.row_scale,))
        p = x.double() @ (m8.q_row.double() * m8.row_scale.double()[:, None]).t()
    _close(y, p.float(), torch.float16)


@pytest.mark.parametrize("M", [1, 8])
def test_short_problems_beside_one_of_many_waves(M):
    """CTAs of four warps leave two partial sums each: of parts of one unit of K, of none, and of an odd number."""
    sizes = [(512, 9600), (64, 40), (72, 33), (136, 64), (704, 32)]
    g = torch.Generator(device="cuda").manual_seed(M)
    xs = [torch.randn(M, K, generator=g, device="cuda").half() for K, _ in sizes]
    ws = [(torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).half() for K, N in sizes]
    ys = rows.rows_gemv(xs, ws, out_features=[N for _, N in sizes], fmts=[0] * len(sizes))
    for x, w, y in zip(xs, ws, ys):
        _close(y, (x.double() @ w.double().t()).float(), torch.float16)
        alone, = rows.rows_gemv((x,), (w,), out_features=(int(w.shape[0]),), fmts=(0,))
        _close(alone, y.float(), torch.float16)


@pytest.mark.parametrize("M,epi", [(1, 0), (3, 1), (8, 2)])
@pytest.mark.parametrize("N,fewer", [(9504, 9472), (37920, 37888), (47392, 47360)])
@pytest.mark.parametrize("fmt", ["fp16", "bf16", "int4", "int8"])
def test_ctas_of_four_warps_give_the_bits_of_eight(M, epi, N, fewer, fmt):
    """Channels of a weight of N rows and of its first rows alone, either side of the limits at 296, 1184 and 1480 tiles of 32 channels (CTAs
    of eight warps up to 296, of four up to 592, of eight up to 888, of four up to 1184, of eight up to 1480, then of four): the same
    partial sums in the same order, whatever the warps of a CTA.  11 quantised units of K and 22 dense ones, so that halves are odd."""
    K = 1408
    g = torch.Generator(device="cuda").manual_seed(N + M)
    dt = torch.bfloat16 if fmt == "bf16" else torch.float16
    x = torch.randn(M, K, generator=g, device="cuda").to(dt)
    res = torch.randn(M, N, generator=g, device="cuda").to(dt) if epi == 2 else None
    if fmt == "int4":
        q = torch.randint(0, 256, (N, K // 2), generator=g, device="cuda", dtype=torch.uint8)
        sc = (torch.rand(N, K // 128, generator=g, device="cuda") * 0.01).half()
        weight, scale = (lambda n: hb.w4_repack_tiled(q[:n].contiguous(), sc[:n].contiguous(), K, 128)), None
    elif fmt == "int8":
        q = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
        weight, scale = (lambda n: hb.w8_repack_tiled(q[:n].contiguous())), (torch.rand(N, generator=g, device="cuda") * 0.01).half()
    else:
        w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(dt)
        weight, scale = (lambda n: w[:n].contiguous()), None
    outs = [rows.rows_gemv((x,), (weight(n),), out_features=(n,), fmts=({"int4": 1, "int8": 2}.get(fmt, 0),), epilogues=(epi,),
                           scales=(None if scale is None else scale[:n].contiguous(),),
                           residuals=(None if res is None else res[:, :n].contiguous(),))[0] for n in (N, fewer)]
    assert bool(torch.isfinite(outs[0]).all()) and torch.equal(outs[0][:, :fewer], outs[1])
