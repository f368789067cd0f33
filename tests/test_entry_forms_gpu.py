"""The launchers' vector forms have a general one behind them: widths, strides, addresses and counts that the wide accesses do not allow give
the same results (GPU only)."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _lib():
    from qwb200.ops import lib as qlib
    return qlib.load(True)


def P(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def S():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def gen(seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return lambda *s: torch.randn(*s, generator=g, device=DEV)


def shifted(t, by=1):
    """The same values `by` elements behind a 16-byte boundary (0: on it)."""
    flat = torch.zeros(t.numel() + 16, dtype=t.dtype, device=t.device)
    out = flat[by:by + t.numel()].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("SH,col0,ld,off", [(64, 0, 64, 0), (63, 0, 64, 0), (64, 1, 72, 0), (61, 2, 65, 0), (64, 0, 64, 1), (1030, 4, 1036, 3)])
def test_embedding_rows_of_any_width_and_address(SH, col0, ld, off):
    hc, vocab, M = 4, 50, 7
    table = shifted(gen(SH)(vocab, ld).to(torch.bfloat16), off)
    tok = i32([0, 49, 3, 3, 17, 48, 1])
    X = shifted(torch.zeros(M, hc, SH, device=DEV), off)
    assert _lib().qwk_embed_rows(P(tok), P(table), ld, col0, SH, hc, vocab, P(X), M, S()) == 0
    assert torch.equal(X, table[tok.long(), col0:col0 + SH].float().unsqueeze(1).expand(M, hc, SH))


@pytest.mark.parametrize("SH,ld,off", [(64, 64, 0), (63, 64, 0), (64, 65, 0), (64, 64, 1), (1030, 1031, 2)])
@pytest.mark.parametrize("pending", [True, False])
def test_deferred_combine_of_any_width_and_address(SH, ld, off, pending):
    """X += pending * gate, its bf16 rows and sums of squares, against 64 bits (fp32 sums of up to 1,030 squares: 1e-6; bf16 rows 2^-8)."""
    M, hc = 5, 4
    rn = gen(SH + ld)
    X, pend, inj, w1 = (shifted(t, off) for t in (rn(M, hc, SH), rn(M, ld), rn(M, hc), 1 + 0.1 * rn(hc, SH)))
    y, ssq = shifted(torch.zeros(M, hc, SH, dtype=torch.bfloat16, device=DEV), off), torch.zeros(M, hc, device=DEV)
    want = X.double() + (pend[:, None, :SH].double() * (2 * torch.sigmoid(inj.double() / hc))[..., None] if pending else 0)
    assert _lib().qwk_hc_pre(P(X), P(pend) if pending else None, ld, P(inj), hc, P(w1), SH, hc, P(y), P(ssq), hc, M, S()) == 0
    assert torch.allclose(X.double(), want, rtol=1e-6, atol=1e-6)
    assert torch.allclose(y.double(), X.double() * w1.double(), rtol=2 ** -8, atol=1e-30)
    assert torch.allclose(ssq.double(), X.double().pow(2).sum(-1), rtol=1e-6)


@pytest.mark.parametrize("H,hc,off", [(64, 4, 0), (63, 4, 0), (63, 1, 0), (61, 3, 0), (64, 4, 1), (1537, 3, 0)])
def test_mtp_norm_of_any_width_and_address(H, hc, off):
    """Both norms against 64 bits (one rounding to bf16: 2^-8, and the fp32 sum of squares)."""
    M, vocab, eps = 3, 20, 1e-6
    rn = gen(H)
    hidden, nh, ne = shifted(rn(M, hc, H), off), shifted(1 + 0.1 * rn(hc * H), off), 1 + 0.1 * rn(H)
    embed, tok = rn(vocab, H).to(torch.bfloat16), i32([3, 19, 0])
    hn, en = shifted(torch.zeros(M, hc, H, dtype=torch.bfloat16, device=DEV), off), torch.zeros(M, H, dtype=torch.bfloat16, device=DEV)
    assert _lib().qwk_mtp_norm(P(hidden), P(tok), P(embed), vocab, P(nh), P(ne), H, hc, C.c_float(eps), P(hn), P(en), M, S()) == 0
    h, e = hidden.double().view(M, -1), embed[tok.long()].double()
    h = h * torch.rsqrt(h.pow(2).mean(1, keepdim=True) + eps) * nh.double()
    e = e * torch.rsqrt(e.pow(2).mean(1, keepdim=True) + eps) * ne.double()
    assert torch.allclose(hn.double().view(M, -1), h, rtol=2 ** -8, atol=1e-30) and torch.allclose(en.double(), e, rtol=2 ** -8, atol=1e-30)


@pytest.mark.parametrize("SH,pad,taps,off,M", [(32, 0, 4, 0, 20), (32, 0, 4, 0, 300), (31, 0, 4, 0, 20), (32, 1, 4, 0, 20), (32, 0, 3, 0, 20),
                                               (32, 0, 5, 0, 300), (33, 3, 2, 0, 7), (32, 0, 4, 1, 20), (32, 0, 1, 2, 5)])
def test_ngram_layer_of_any_width_taps_and_address(SH, pad, taps, off, M):
    """Gate, dilated convolution over two runs of rows and their slots' rings, ring update: against the same formulas in 64 bits
    (fp32 throughout: 2e-5 of a value covers a dozen roundings)."""
    hc, H, eps, dil, RING = 4, 128, 1e-6, 3, 32
    xw = hc * SH
    rn = gen(SH * taps + M)
    kv, red, nc1, cw, X, ring = (shifted(t, off) for t in (rn(M, xw + SH + pad), rn(M, 16).abs() + 0.1, rn(xw), rn(xw, taps), rn(M, xw), rn(2, RING, xw)))
    first = M // 3
    runs = [(0, 0, first, 5), (1, first, M - first, 40)]                    # slot, first row, rows, position
    slot, pos, rs, rl = [], [], [], [0] * M
    for sl, r0, n, p0 in runs:
        slot += [sl] * n
        pos += [p0 + i for i in range(n)]
        rs += [r0] * n
        rl[r0] = n
    old, x0 = ring.double().clone(), X.double().clone()
    gv, nc = shifted(torch.zeros(M, xw, device=DEV), off), shifted(torch.zeros(M, xw, device=DEV), off)
    t = [i32(v) for v in (slot, pos, rs, rl)]
    assert _lib().qwk_ple_apply(P(kv), xw + SH + pad, P(red), 16, P(nc1), P(cw), SH, hc, H, C.c_float(eps), taps, dil, P(gv), P(nc), P(ring), P(X), M,
                                *[P(v) for v in t], S()) == 0
    r = red.double()[:, :3 * hc].view(M, hc, 3)
    gs = r[..., 2] * torch.rsqrt(r[..., 0] / H + eps) * torch.rsqrt(r[..., 1] / H + eps) / H ** 0.5
    gate = torch.sigmoid(torch.sign(gs) * gs.abs().clamp_min(1e-6).sqrt())
    rnorm = torch.rsqrt(gate ** 2 * red.double()[:, 3 * hc:3 * hc + 1] / H + eps)
    g = gate[..., None] * kv.double()[:, None, xw:xw + SH]
    n = (g * rnorm[..., None]).view(M, xw) * nc1.double()
    conv = torch.zeros(M, xw, dtype=torch.float64, device=DEV)
    for m in range(M):
        for k in range(taps):
            back = (taps - 1 - k) * dil
            q = pos[m] - back
            v = n[m - back] if m - back >= rs[m] else old[slot[m], q % RING] if q >= 0 else 0.0
            conv[m] += cw.double()[:, k] * v
    assert torch.allclose(X.double(), x0 + g.reshape(M, xw) + torch.nn.functional.silu(conv), rtol=2e-5, atol=2e-5)
    for m in range(M):
        if m - rs[m] >= rl[rs[m]] - RING:
            old[slot[m], pos[m] % RING] = n[m]
    assert torch.allclose(ring.double(), old, rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("pad,off", [(0, 0), (1, 0), (3, 0), (0, 1), (2, 3)])
def test_chunked_scan_takes_projections_of_any_stride_and_address(pad, off):
    """The output norm reads the gate z from the projection rows: the same bits wherever these rows start."""
    KL, VL, M = 1, 2, 70
    qkv_l = (2 * KL + VL) * 128
    ld0 = (qkv_l + VL * 128 + 2 * VL + 3) // 4 * 4
    rn = gen(5)
    qkv, beta, decay, proj0, S0, nw = rn(M, qkv_l) * 0.1, torch.sigmoid(rn(M, VL)), torch.sigmoid(rn(M, VL) + 3), rn(M, ld0), rn(1, VL, 128, 128) * 0.1, 1 + 0.1 * rn(128)
    need = 64 * 1024 * 1024

    def scan(pad, off):
        proj = shifted(torch.cat([proj0, torch.zeros(M, pad, device=DEV)], 1), off)
        st, o, scratch = S0.clone(), torch.zeros(M, VL * 128, dtype=torch.bfloat16, device=DEV), torch.zeros(need // 4, device=DEV)
        assert _lib().qwk_gdn_scan_chunked(P(qkv), P(decay), P(beta), P(proj), ld0 + pad, P(st), P(shifted(nw, off)), KL, VL, M, P(i32([0] * M)), P(scratch), P(o),
                                           C.c_float(1e-6), S()) == 0
        torch.cuda.synchronize()
        return st, o
    want, got = scan(0, 0), scan(pad, off)
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1]) and float(got[1].float().abs().max()) > 0


@pytest.mark.parametrize("runs", [[(0, 40, 3)], [(1, 13, 0), (0, 27, 6)], [(0, 1, 20), (1, 8, 2), (2, 30, 50)], [(2, 33, 1), (0, 33, 0), (1, 2, 9)]])
@pytest.mark.parametrize("off,pad", [(0, 0), (1, 0), (0, 1)])
def test_gdn_conv_of_many_rows_in_several_runs(runs, off, pad):
    """More than 32 rows: every run's taps come from its own rows and its own slot's ring, wherever the run begins within a block's
    eight rows.  Against 64 bits (four products, silu and a norm of 128 in fp32: 1e-5)."""
    KL, VL, RING = 1, 2, 16
    qkv_l = (2 * KL + VL) * 128
    ld = qkv_l + VL * 128 + 2 * VL + pad
    M = sum(n for _, n, _ in runs)
    rn = gen(M + off)
    proj, cw, ring = shifted(rn(M, ld), off), shifted(rn(qkv_l, 4) * 0.3, off), shifted(rn(3, RING, qkv_l), off)
    A, dt = rn(VL), rn(VL)
    slot, pos, rs, rl = [], [], [], [0] * M
    for sl, n, p0 in runs:
        rl[len(slot)] = n
        rs += [len(slot)] * n
        slot += [sl] * n
        pos += [p0 + i for i in range(n)]
    old = ring.double().clone()
    qkv, dec, beta = torch.zeros(M, qkv_l, device=DEV), torch.zeros(M, VL, device=DEV), torch.zeros(M, VL, device=DEV)
    t = [i32(v) for v in (slot, pos, rs, rl)]
    assert _lib().qwk_gdn_conv(P(proj), ld, P(ring), P(cw), P(A), P(dt), KL, VL, M, *[P(v) for v in t], P(qkv), P(dec), P(beta), C.c_float(1e-6), S()) == 0
    p, want = proj.double(), torch.zeros(M, qkv_l, dtype=torch.float64, device=DEV)
    for m in range(M):
        for k in range(4):
            back, q = 3 - k, pos[m] - 3 + k
            want[m] += cw.double()[:, k] * (p[m - back, :qkv_l] if m - back >= rs[m] else old[slot[m], q % RING] if q >= 0 else 0.0)
    want = torch.nn.functional.silu(want).view(M, -1, 128)
    norm = torch.rsqrt(want.pow(2).sum(-1, keepdim=True) + 1e-6)
    want[:, :KL] *= norm[:, :KL] / 128 ** 0.5
    want[:, KL:2 * KL] *= norm[:, KL:2 * KL]
    assert torch.allclose(qkv.double(), want.view(M, -1), rtol=1e-5, atol=1e-6)
    z = p[:, qkv_l + VL * 128:]
    assert torch.allclose(beta.double(), torch.sigmoid(z[:, :VL]), rtol=1e-5, atol=1e-6)
    assert torch.allclose(dec.double(), torch.exp(-torch.exp(A.double()) * torch.nn.functional.softplus(z[:, VL:2 * VL] + dt.double())), rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("D,off", [(1152, 0), (1153, 0), (1536, 0), (1540, 0), (2050, 0), (72, 1), (1152, 2)])
@pytest.mark.parametrize("add", [True, False])
def test_vision_norm_of_any_width_and_address(D, off, add):
    """x += y + bias, then the norm in bf16 (2^-8 of a value, and fp32 sums under a mean of near 0: 1e-5), against 64 bits."""
    L, eps = 9, 1e-6
    rn = gen(D)
    x, y, yb, w, b = (shifted(t, off) for t in (rn(L, D), rn(L, D), rn(D), 1 + 0.1 * rn(D), rn(D)))
    out = shifted(torch.zeros(L, D, dtype=torch.bfloat16, device=DEV), off)
    want = x.double() + (y.double() + yb.double() if add else 0)
    assert _lib().qwk_vit_layernorm(P(x), P(y) if add else None, P(yb) if add else None, P(w), P(b), L, D, C.c_float(eps), P(out), S()) == 0
    assert torch.allclose(x.double(), want, rtol=1e-6, atol=1e-6)
    ref = torch.nn.functional.layer_norm(x.double(), (D,), w.double(), b.double(), eps)
    assert torch.allclose(out.double(), ref, rtol=2 ** -8, atol=1e-5)


@pytest.mark.parametrize("heads,off", [(2, 0), (2, 1), (16, 4), (1, 2)])
def test_vision_rotary_at_any_address(heads, off):
    """The same bits from aligned and shifted rows, and against 64 bits (one rounding to bf16, relative to the pair's size)."""
    L, hd = 11, 72
    D = heads * hd
    rn = gen(heads)
    q0, bias, pos = rn(L, 3 * D).to(torch.bfloat16), rn(3 * D), torch.stack([torch.arange(L), torch.arange(L) % 4], 1).to(torch.int32).to(DEV)

    def rope(off):
        qkv, tab = shifted(q0, off), shifted(torch.zeros(L, 2, 36, device=DEV), off)
        assert _lib().qwk_vit_rope_table(P(pos), L, P(tab), S()) == 0
        assert _lib().qwk_vit_bias_rope(P(qkv), P(shifted(bias, off)), P(tab), L, heads, S()) == 0
        return qkv
    got = rope(off)
    assert torch.equal(got, rope(0))
    v = (q0.double() + bias.double()).view(L, 3, heads, 2, 36)
    ang = torch.cat([pos[:, :1].double(), pos[:, 1:].double()], 1).repeat_interleave(18, 1) * (10000.0 ** (-2.0 * torch.arange(18, device=DEV).double() / 36)).repeat(2)
    c, s = ang.cos()[:, None, None], ang.sin()[:, None, None]
    a, b = v[:, :2, :, 0], v[:, :2, :, 1]
    want = v.clone()
    want[:, :2, :, 0], want[:, :2, :, 1] = a * c - b * s, b * c + a * s
    assert torch.allclose(got.double().view(L, 3, heads, 2, 36), want, rtol=2 ** -8, atol=2e-5)


def test_vision_gelu_of_more_rows_than_a_grid_is_high():
    """600,000 rows of eight columns."""
    L, D = 600_000, 8
    rn = gen(1)
    y, bias = rn(L, D).to(torch.bfloat16), rn(D)
    want = torch.nn.functional.gelu(y.float() + bias, approximate="tanh")
    assert _lib().qwk_vit_bias_gelu(P(y), P(bias), L, D, 1, S()) == 0
    assert torch.allclose(y.float(), want, rtol=2 ** -8, atol=1e-6)


def test_logits_reduction_of_more_rows_than_a_grid_is_high():
    from qwb200.ops import kernels as K
    x = gen(2)(70_000, 9)
    val, idx, mx, sm = K.row_reduce(x)
    assert torch.equal(val, x.max(1).values) and torch.equal(idx.long(), x.argmax(1))
    assert torch.allclose(torch.log(sm) + mx, torch.logsumexp(x, 1), atol=1e-5)


@pytest.mark.parametrize("SH,R,n_inj,M", [(6400, 8, 4, 1), (6400, 8, 4, 9), (10240, 16, 0, 3), (32, 320, 300, 5), (32, 64, 500, 1)])
def test_mixers_with_long_rows_and_with_many_inject_rows(SH, R, n_inj, M):
    """Rows that leave no room for the tensor-core form's operands, and more low-rank and inject rows than a block has threads, against
    64 bits (fp32 sums of up to 10,240 exact products: 1e-5 of the result's size; the block input is rounded to bf16 once)."""
    L, hc, eps, H = _lib(), 4, 1e-6, SH
    down = R + n_inj
    ld = (hc + hc * down + 3) // 4 * 4
    rn = gen(SH + M)
    X, pend, ip, w1 = rn(M, hc, SH), rn(M, SH), rn(M, hc), 1 + 0.1 * rn(hc, SH)
    Wd, Wu = (rn(down, hc, SH) * 0.05).to(torch.bfloat16), (rn(SH, hc, R) * 0.1).to(torch.bfloat16)
    xo, send = torch.zeros_like(X), torch.zeros(M, ld, device=DEV)
    assert L.qwk_hc_down(P(X), P(xo), P(pend), SH, P(ip), P(w1), P(Wd), P(send), ld, SH, hc, down, M, S()) == 0
    x = X.double() + pend.double()[:, None] * (2 * torch.sigmoid(ip.double() / hc))[..., None]
    assert torch.allclose(xo.double(), x, rtol=1e-5, atol=1e-5)
    y = (xo * w1).to(torch.bfloat16).double()
    part = torch.einsum("msc,jsc->msj", y, Wd.double())
    got = send[:, hc:hc + hc * down].view(M, hc, down).double()
    assert float((got - part).norm() / part.norm()) < 1e-5
    assert torch.allclose(send[:, :hc].double(), xo.double().pow(2).sum(-1), rtol=1e-5)
    inj, out = torch.zeros(M, max(n_inj, 1), device=DEV), torch.zeros(M, SH, dtype=torch.bfloat16, device=DEV)
    assert L.qwk_hc_up_mix(P(send), ld, P(Wu), P(xo), P(w1), SH, hc, R, n_inj, H, C.c_float(eps), M, P(inj) if n_inj else None, max(n_inj, 1), P(out), SH, 0, S()) == 0
    r = torch.rsqrt(xo.double().pow(2).mean(-1) + eps)
    d = (r[..., None] * part).sum(1)
    if n_inj:
        assert float((inj.double() - d[:, R:]).norm() / d[:, R:].norm()) < 1e-5
    gate = torch.sigmoid(torch.einsum("csr,mr->msc", Wu.double(), torch.nn.functional.silu(d[:, :R] / hc)))
    want = (gate * y * r[..., None]).mean(1)
    assert float((out.double() - want).norm() / want.norm()) < 5e-3
