"""Kernels of a prefill chunk and of the vision tower at the edges of their forms (GPU only)."""
import ctypes as C

import pytest
import torch

from test_step_kernels_gpu import DEV, P, S, _lib, gen, i32

pytestmark = pytest.mark.gpu


@pytest.fixture
def exchange():
    """Sets the tokens of an exchanged tile (0: by cost, negative: the operands keep their roles) and puts the rule back."""
    L = _lib()
    word = torch.zeros(2, dtype=torch.int32, device=DEV)           # bounded waits that run out report here
    L.qwk_set_error_word(P(word))
    old = L.qwk_gemm_tc_exchange_nt(0)
    yield L.qwk_gemm_tc_exchange_nt
    torch.cuda.synchronize()
    L.qwk_gemm_tc_exchange_nt(old)
    L.qwk_set_error_word(None)
    assert word.tolist() == [0, 0]


def _product(T, N, K, dtype, off=0):
    from qwb200.ops import kernels as K_
    rn = gen(T + N + K)
    A, W = rn(T, K).bfloat16(), (rn(N, K) * 0.05).bfloat16()
    ld = (N + 7) // 8 * 8 + 8
    flat = torch.full((ld * (T + 2) + 8,), 768.0, dtype=dtype, device=DEV)
    out = flat[off:off + ld * (T + 2)].view(T + 2, ld)
    K_.gemm_bf16_tc(A, W, out=out[:T, :N])
    torch.cuda.synchronize()
    assert torch.all(out[:, N:].float() == 768.0) and torch.all(out[T:].float() == 768.0) and torch.all(flat[:off].float() == 768.0)
    return A, W, out[:T, :N]


@pytest.mark.parametrize("T,N,K,nt", [(257, 300, 72, 32), (300, 700, 192, 160), (777, 1793, 320, 208), (1021, 2560, 640, 256), (513, 257, 64, 48), (33, 40000, 64, 16),
                                      (1500, 4304, 136, 96), (3000, 5000, 64, 240)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("off", [0, 1])
def test_exchanged_operands_give_the_bits_of_the_other_forms(exchange, T, N, K, nt, dtype, off):
    """Weight rows as the pair's 256 rows, tokens as its columns: tiles that end inside the tokens and the columns, an odd number of columns
    (two of them leave in one word), outputs off 16 bytes; k is one chain in every form."""
    exchange(nt)
    assert _lib().qwk_gemm_tc_exchanged(T, N, K) == nt
    A, W, got = _product(T, N, K, dtype, off)
    exchange(-1)
    assert _lib().qwk_gemm_tc_exchanged(T, N, K) == 0
    assert torch.equal(got, _product(T, N, K, dtype)[2])
    ref = A.double() @ W.double().T
    assert float((got.double() - ref).norm() / ref.norm()) < (1e-5 if dtype == torch.float32 else 2 ** -8)


@pytest.mark.parametrize("T,N,K,form", [(520, 12800, 320, 1), (640, 12700, 72, 1), (300, 512, 64, 0), (777, 4352, 64, 2), (1111, 16480, 128, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_forms_that_keep_the_roles_match_64_bits(exchange, T, N, K, form, dtype):
    """What peers' products, and others where exchanging does not pay, go through."""
    exchange(-1)
    assert _lib().qwk_gemm_tc_form(T, N, K) == form
    A, W, got = _product(T, N, K, dtype)
    ref = A.double() @ W.double().T
    assert float((got.double() - ref).norm() / ref.norm()) < (1e-5 if dtype == torch.float32 else 2 ** -8)


@pytest.mark.parametrize("T,N,K,form", [(100, 256, 1024, 3), (300, 512, 64, 0), (520, 12800, 64, 1), (777, 10200, 320, 1), (777, 4352, 64, 2), (300, 10190, 136, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("off", [0, 1, 2, 4])
@pytest.mark.parametrize("stage", [1, 0])
def test_forms_that_keep_the_roles_at_any_address_with_and_without_staging(exchange, T, N, K, form, dtype, off, stage):
    """Each form that products between ranks take, told to run (none of these is exchanged): fp32 output through the staging buffers and straight from
    registers, outputs off 16 bytes, nothing beside them.  k is one chain in every form but the split one: the bits of an aligned output."""
    lib = _lib()
    exchange(-1)
    assert lib.qwk_gemm_tc_form(T, N, K) == form and lib.qwk_gemm_tc_exchanged(T, N, K) == 0
    old = lib.qwk_gemm_tc_stage_local(stage)
    try:
        A, W, got = _product(T, N, K, dtype, off)
    finally:
        lib.qwk_gemm_tc_stage_local(old)
    assert torch.equal(got, _product(T, N, K, dtype)[2])
    ref = A.double() @ W.double().T
    assert float((got.double() - ref).norm() / ref.norm()) < (1e-5 if dtype == torch.float32 else 2 ** -8)


@pytest.mark.parametrize("L,heads", [(128, 1), (129, 2), (600, 16), (2100, 3), (3520, 16)])
def test_vision_attention_with_its_keys_dealt_evenly(L, heads):
    """Runs that begin and end inside a unit's keys, units in two and more runs, a last key tile that is not whole: against 64 bits (weights and
    output rounded to bf16: 2^-8) and no further from them than 1.05 times what whole units give."""
    lib = _lib()
    rn = gen(L + heads)
    qkv = rn(L, 3 * heads * 72).bfloat16()
    need = lib.qwk_vit_attention_scratch(L, heads)
    parts = torch.full((max(need, 16),), 255, dtype=torch.uint8, device=DEV)          # NaN where nothing is written
    outs = [torch.zeros(L, heads * 72, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    assert lib.qwk_vit_attention_split(P(qkv), L, heads, P(outs[0]), P(parts) if need else None, S()) == 0
    assert lib.qwk_vit_attention(P(qkv), L, heads, P(outs[1]), S()) == 0
    q, k, v = (t.view(L, heads, 72).transpose(0, 1).double() for t in qkv.split(heads * 72, 1))
    want = torch.cat([(torch.softmax(q[h] @ k[h].T / 72 ** 0.5, -1) @ v[h]) for h in range(heads)], 1)
    err = [float((o.double() - want).norm() / want.norm()) for o in outs]
    assert err[0] < 2 ** -8 and err[0] < 1.05 * err[1] + 1e-6


@pytest.mark.parametrize("M", [33, 63, 65, 129])
@pytest.mark.parametrize("KL,VL", [(1, 2), (2, 6), (8, 16), (16, 48)])
def test_chunked_scan_of_ragged_runs_is_as_exact_as_its_operands(M, KL, VL):
    """Chunks that are not whole, against 64 bits.  The products' operands are tf32 (2^-12): outputs and states to 1.5e-3 of their size."""
    from qwb200.models.gdn_chunked import scan_sequential
    rn, D = gen(M + VL), 128
    q, k, v = torch.nn.functional.normalize(rn(M, KL, D), dim=-1) * D ** -0.5, torch.nn.functional.normalize(rn(M, KL, D), dim=-1), rn(M, VL, D)
    qkv = torch.cat([t.reshape(M, -1) for t in (q, k, v)], 1).contiguous()
    decay, beta = torch.exp(-rn(M, VL).abs() * 0.2).contiguous(), torch.sigmoid(rn(M, VL)).contiguous()
    qkv_l = qkv.shape[1]
    ld = qkv_l + VL * D + 2 * VL
    proj, S0, nw = rn(M, ld), rn(1, VL, D, D) * 0.1, 1 + 0.1 * rn(D)
    St, o = S0.clone(), torch.zeros(M, VL * D, dtype=torch.bfloat16, device=DEV)
    scratch = torch.full(((M + 63) // 64 * VL * (2 * 64 * 128 + 64 * 64 + 64) + M * VL * D,), float("nan"), device=DEV)
    assert _lib().qwk_gdn_scan_chunked(P(qkv), P(decay), P(beta), P(proj), ld, P(St), P(nw), KL, VL, M, P(i32([0] * M)), P(scratch), P(o), C.c_float(1e-6), S()) == 0
    raw = scratch[-M * VL * D:].view(M, VL, D)
    for h in range(VL):
        a = [t.double().cpu() for t in (q[:, h * KL // VL], k[:, h * KL // VL], v[:, h], decay[:, h], beta[:, h], S0[0, h])]
        want, Sw = scan_sequential(*a)
        assert float((raw[:, h].double().cpu() - want).norm() / want.norm()) < 1.5e-3
        assert float((St[0, h].double().cpu() - Sw).norm() / Sw.norm()) < 1.5e-3


@pytest.mark.parametrize("M,shared", [(64, 0), (130, 0), (130, 1)])
def test_chunked_scan_solves_its_systems_as_exactly_as_fp32_substitution(M, shared):
    """Keys in steps of 1/16 and a beta of 8 bits without decay: the matrix of a chunk is exact, so what is left is the solve.  Its result against 64
    bits, beside forward substitution in fp32 (each multiply-add rounded once): no further off than 1.05 times that (16,000 values)."""
    KL, VL, D = 1, 2, 128
    g = torch.Generator().manual_seed(M + shared)
    k = (torch.randint(-2, 3, (M, D), generator=g) if not shared else torch.randint(0, 3, (M, D), generator=g)).float() / 16
    v, beta = torch.randn(M, VL, D, generator=g), torch.randint(16, 256, (M, VL), generator=g).float() / 256
    qkv = torch.cat([k, k, v.reshape(M, -1)], 1).to(DEV).contiguous()
    ld, nch = qkv.shape[1] + VL * D + 2 * VL, (M + 63) // 64
    proj, St, o = torch.zeros(M, ld, device=DEV), torch.zeros(1, VL, D, D, device=DEV), torch.zeros(M, VL * D, dtype=torch.bfloat16, device=DEV)
    scratch = torch.zeros(nch * VL * (2 * 64 * 128 + 64 * 64 + 64) + M * VL * D, device=DEV)
    bd, dec, nw = beta.to(DEV), torch.ones(M, VL, device=DEV), torch.ones(D, device=DEV)
    assert _lib().qwk_gdn_scan_chunked(P(qkv), P(dec), P(bd), P(proj), ld, P(St), P(nw), KL, VL, M, P(i32([0] * M)), P(scratch), P(o), C.c_float(1e-6), S()) == 0
    got = scratch[nch * VL * 64 * D:2 * nch * VL * 64 * D].view(nch, VL, 64, D).cpu()
    here = there = 0.0
    for ch in range(nch):
        n = min(64, M - ch * 64)
        rows = slice(ch * 64, ch * 64 + n)
        for h in range(VL):
            A = torch.tril(beta[rows, h, None].double() * (k[rows].double() @ k[rows].double().T), -1)
            B = (beta[rows, h, None] * v[rows, h]).float()
            W, want = B.clone(), torch.linalg.solve_triangular(torch.eye(n).double() + A, B.double(), upper=False)
            for r in range(1, n):
                acc = torch.zeros(4, D)
                for s in range(r):
                    acc[s & 3] = (acc[s & 3].double() + A[r, s] * W[s].double()).float()
                W[r] -= (acc[0] + acc[1]) + (acc[2] + acc[3])
            here += float((got[ch, h, :n].double() - want).pow(2).sum())
            there += float((W.double() - want).pow(2).sum())
    assert here ** 0.5 < 1.05 * there ** 0.5, (here ** 0.5, there ** 0.5)


@pytest.mark.parametrize("bad", [20, 50, 63, 64 + 33, 64 + 50])
def test_chunked_scan_keeps_a_row_that_is_not_finite_from_the_tiles_before_it(bad):
    """Rows before the 16-row tile of a NaN row have the bits that they have without it; the row itself and the state show it."""
    KL, VL, M, D = 2, 4, 130, 128
    rn = gen(bad)
    qkv, decay, beta = rn(M, (2 * KL + VL) * D) * 0.1, torch.exp(-rn(M, VL).abs() * 0.2).contiguous(), torch.sigmoid(rn(M, VL)).contiguous()
    ld = qkv.shape[1] + VL * D + 2 * VL
    proj, S0, nw = rn(M, ld), rn(1, VL, D, D) * 0.1, 1 + 0.1 * rn(D)
    outs = []
    for poison in (False, True):
        x, St, o = qkv.clone(), S0.clone(), torch.zeros(M, VL * D, dtype=torch.bfloat16, device=DEV)
        if poison:
            x[bad] = float("nan")
        scratch = torch.zeros((M + 63) // 64 * VL * (2 * 64 * 128 + 64 * 64 + 64) + M * VL * D, device=DEV)
        assert _lib().qwk_gdn_scan_chunked(P(x), P(decay), P(beta), P(proj), ld, P(St), P(nw), KL, VL, M, P(i32([0] * M)), P(scratch), P(o), C.c_float(1e-6), S()) == 0
        torch.cuda.synchronize()
        outs.append((o, St))
    first = bad // 16 * 16
    assert torch.equal(outs[0][0][:first], outs[1][0][:first]) and torch.isfinite(outs[0][0]).all()
    assert torch.isnan(outs[1][0][bad:]).all() and torch.isnan(outs[1][1]).all()


@pytest.mark.parametrize("T,H,k,off,shared", [(3, 2560, 10, 0, True), (5, 516, 3, 0, True), (4, 510, 7, 0, False), (4, 512, 5, 1, True), (33, 8, 11, 0, False)])
def test_combined_experts_of_any_width_and_address(T, H, k, off, shared):
    """Four columns at a time or one, experts of other ranks left out: the sums of the same products in the same order."""
    rn = gen(T + H)
    flat = torch.zeros(T * k * H + 8, device=DEV)
    y = flat[off:off + T * k * H].view(T * k, H)
    y.copy_(rn(T * k, H))
    inv = torch.randperm(T * k, device=DEV).int().view(T, k)
    inv[0, 0] = -1
    w, sh, out = rn(T, k), rn(T, H), torch.zeros(T, H, device=DEV)
    assert _lib().qwk_moe_combine_T(P(y), H, P(inv), P(w), k, P(sh) if shared else None, H, P(out), T, S()) == 0
    rows = torch.where((inv >= 0)[..., None], y[inv.long().clamp(min=0)], torch.zeros((), device=DEV))
    want = (rows.double() * w[..., None].double()).sum(1) + (sh.double() if shared else 0)
    assert float((out.double() - want).norm() / want.norm()) < 1e-6


@pytest.mark.parametrize("base,M", [(0, 64), (3, 61), (257, 70)])
def test_attention_inputs_of_a_chunk_equal_the_step_kernels(base, M):
    """More than 32 rows take a block per row and a warp per head: queries, keys, values, indexer queries, compressed keys and the raw-key ring
    are those of the same rows in pieces of at most 32, bit for bit; behind the last row zeros up to the next multiple of 16."""
    lib = _lib()
    QL, KVL, IH, ratio, page, rope = 6, 2, 4, 4, 256, 64
    assert lib.qwk_rope_init(C.c_double(1e6), rope) == 0
    rn = gen(M + base)
    ld = QL * 512 + 2 * KVL * 256 + IH * 128 + 128
    proj = rn(M, ld)
    w = [1 + 0.1 * rn(n) for n in (256, 256, 128, 128)]
    pages = (base + M + page - 1) // page + 1
    table = torch.arange(pages, dtype=torch.int32, device=DEV)
    ring0 = rn(1, 16, 128)

    def run(pieces, entry):
        out = dict(k=torch.full((pages * page, KVL * 256), 3.0, dtype=torch.bfloat16, device=DEV), q=torch.zeros(M, QL, 256, device=DEV),
                   iq=torch.zeros(M, IH, 128, device=DEV), ring=ring0.clone(), ck=torch.zeros(1, (base + M) // ratio + 1, 128, dtype=torch.bfloat16, device=DEV))
        out["v"] = out["k"].clone()
        for m0, n in pieces:
            lens = [n] + [0] * (n - 1)
            t = [i32([0] * n), i32([base + m0 + i for i in range(n)]), i32([0] * n), i32(lens)]
            assert getattr(lib, entry)(P(proj[m0:]), ld, QL, KVL, IH, *map(P, w), n, *map(P, t), P(out["k"]), P(out["v"]), None, None, pages, P(table), pages,
                                       P(out["q"][m0:]), P(out["iq"][m0:]), P(out["ring"]), P(out["ck"]), out["ck"].shape[1], ratio, C.c_float(1e-6), S()) == 0
            torch.cuda.synchronize()
        return out

    a, b = run([(0, M)], "qwk_qsa_prep_run"), run([(m, min(32, M - m)) for m in range(0, M, 32)], "qwk_qsa_prep")
    end, tail = base + M, (base + M + 15) // 16 * 16
    for key in ("q", "iq", "ring", "ck"):
        assert torch.equal(a[key], b[key]), key
    for key in ("k", "v"):
        assert torch.equal(a[key][:end], b[key][:end]) and torch.equal(a[key][tail:], b[key][tail:]) and torch.all(a[key][end:tail] == 0), key


@pytest.mark.parametrize("T,SH,R", [(1200, 2560, 320), (1201, 264, 40), (1407, 8, 320), (2500, 520, 72), (40000, 40, 136)])
def test_mixer_up_projection_of_a_long_chunk_equals_its_pieces(T, SH, R):
    """The form that keeps its weights against the one for few rows: the same products and sums, so the same bits, and nothing beside them."""
    L, rn = _lib(), gen(T + SH)
    u, W, xn = rn(T, R).bfloat16(), (rn(4 * SH, R) * 0.1).bfloat16(), rn(T, 4, SH).bfloat16()
    u[T // 2, 0] = float("nan")
    W[:, 1] = 0
    W[4 * (SH // 2) + 1, 1] = 1.0
    u[5, 1], u[6, 1] = 300.0, -300.0                              # gates of 1 and 0
    word = torch.zeros(2, dtype=torch.int32, device=DEV)
    L.qwk_set_error_word(P(word))
    whole, parts = (torch.full((T + 2, SH + 8), 768.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    assert L.qwk_gemm_mix_tc(P(u), P(W), P(xn), SH, P(whole), SH + 8, T, R, R, R, S()) == 0
    for r in range(0, T, 640):
        n = min(640, T - r)
        assert L.qwk_gemm_mix_tc(P(u[r:]), P(W), P(xn[r:]), SH, P(parts[r:]), SH + 8, n, R, R, R, S()) == 0
    torch.cuda.synchronize()
    L.qwk_set_error_word(None)
    assert word.tolist() == [0, 0]
    assert torch.equal(whole.view(torch.int16), parts.view(torch.int16))
    assert torch.all(whole[T:].float() == 768.0) and torch.all(whole[:, SH:].float() == 768.0)
    assert torch.all(torch.isnan(whole[T // 2, :SH])) and torch.isfinite(torch.cat([whole[:T // 2, :SH], whole[T // 2 + 1:T, :SH]])).all()
    c = SH // 2
    gate = torch.sigmoid((u[5:7].double() @ W.double().T).view(2, SH, 4)[:, c])
    ref = (gate * xn[5:7, :, c].double()).mean(1)
    assert torch.allclose(whole[5:7, c].double(), ref, rtol=2 ** -8, atol=1e-5)      # bf16 result, fp32 logits
