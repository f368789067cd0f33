"""Kernels of a decode or verification step at the edges of their forms: streamed products, the delta-net step, flash-decode (GPU only)."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _lib():
    from qwb200.ops import lib as qlib
    return qlib.load(True)


def P(t):
    if t is None:
        return None
    p = C.c_void_p(t.data_ptr())
    p.tensor = t          # a tensor made inside a call lives until the launch: freed at once, its memory would be the next argument's
    return p


def S():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def gen(seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return lambda *s: torch.randn(*s, generator=g, device=DEV)


@pytest.mark.parametrize("N,K", [(40, 6000), (2600, 6144), (4800, 2560), (17, 64), (300, 8192), (33, 1296)])
def test_streamed_products_match_64_bits_at_every_row_count(N, K):
    """One and several tiles per group of warps, k in one, two and four passes, boxes of a whole stage (K a multiple of 64) and of 64
    columns with a ragged end; rows behind the weights' last, and an output with guard columns.  fp32 sums of exact products in eight
    chains of K / 128 tensor-core sums: 4e-10 K of the result's size; a row's bits do not depend on the rows beside it."""
    from qwb200.ops import kernels as K_
    rn = gen(N + K)
    W, x = (rn(N, K) * 0.05).bfloat16(), rn(32, K).bfloat16()
    ref = x.double() @ W.double().T
    one = None
    for M in (1, 7, 8, 9, 16, 17, 24, 25, 32):
        out = torch.full((M, N + 3), 777.0, device=DEV)
        K_.gemv_bf16(W, x[:M], out=out, N=N, ldy=N + 3)
        assert torch.all(out[:, N:] == 777.0)
        assert float((out[:, :N].double() - ref[:M]).norm() / ref[:M].norm()) < 4e-10 * max(K, 2560), M
        one = out[0, :N].clone() if one is None else one
        assert torch.equal(out[0, :N], one), M


@pytest.mark.parametrize("runs", [[1], [6, 6, 6, 6], [12], [13], [32], [3, 17, 1, 8]])
def test_delta_net_step_of_runs_equals_row_by_row(runs):
    """A run's rows in one launch - eight at a time, runs that end inside eight, runs longer than what the kernel stores into the ring itself
    - give what as many launches of single rows give: outputs, states, saved states and ring, bit for bit."""
    KL, VL, ring_rows, eps = 2, 6, 16, 1e-6
    D, slots = 128, len(runs)
    qkv_l = (2 * KL + VL) * D
    ld = qkv_l + VL * D + 2 * VL
    rn = gen(sum(runs))
    M = sum(runs)
    proj, cw = rn(M, ld), rn(qkv_l, 4) * 0.5
    a_log, dt, nw = rn(VL) * 0.1, rn(VL) * 0.1, 1 + 0.1 * rn(D)
    ring0, S0 = rn(slots, ring_rows, qkv_l), rn(slots, VL, D, D) * 0.1
    base = [0, 2, 40, 7][:slots]
    rows = [(s, base[s] + i, sum(runs[:s])) for s in range(slots) for i in range(runs[s])]

    def step(m0, n, starts, lens, ring, St, save, o):
        scratch = torch.empty(n * (qkv_l + 2 * VL), device=DEV)
        t = [i32([r[0] for r in rows[m0:m0 + n]]), i32([r[1] for r in rows[m0:m0 + n]]), i32(starts), i32(lens)]
        assert _lib().qwk_gdn_step(P(proj[m0:]), ld, P(ring), P(cw), P(a_log), P(dt), P(nw), KL, VL, n, *map(P, t), P(St), P(save), P(scratch),
                                   P(scratch[n * qkv_l:]), P(scratch[n * (qkv_l + VL):]), P(o), C.c_float(eps), S()) == 0
        torch.cuda.synchronize()

    outs = []
    for whole in (True, False):
        ring, St, o, save = ring0.clone(), S0.clone(), torch.zeros(M, VL * D, dtype=torch.bfloat16, device=DEV), torch.zeros(M, VL, D, D, device=DEV)
        if whole:
            lens = [0] * M
            for s in range(slots):
                lens[sum(runs[:s])] = runs[s]
            step(0, M, [r[2] for r in rows], lens, ring, St, save, o)
        else:
            for m in range(M):
                step(m, 1, [0], [1], ring, St, save[m:], o[m:])
        outs.append((ring, St, save, o))
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("runs", [[2], [1, 1], [3], [1, 2], [4], [5], [1, 1, 1, 1], [9, 3], [12], [13], [4, 4, 5]])
def test_delta_net_step_gives_the_same_with_and_without_saved_states(runs):
    """Few rows, and few rows whose states are kept, take a form of their own (four rows at a time): the bits of the form for many runs."""
    KL, VL, D, slots, M = 2, 6, 128, len(runs), sum(runs)
    qkv_l = (2 * KL + VL) * D
    ld = qkv_l + VL * D + 2 * VL
    rn = gen(M)
    proj, cw = rn(M + 2 * 8, ld), rn(qkv_l, 4) * 0.5
    a_log, dt, nw, ring0, S0 = rn(VL) * 0.1, rn(VL) * 0.1, 1 + 0.1 * rn(D), rn(slots + 2, 16, qkv_l), rn(slots + 2, VL, D, D) * 0.1
    outs = []
    for extra, saves in ((0, True), (0, False), (2, False)):          # two runs of eight rows more: always the form for many
        lens = list(runs) + [8] * extra
        n, starts = sum(lens), [sum(lens[:s]) for s in range(len(lens))]
        tables = [i32([s for s, k in enumerate(lens) for _ in range(k)]), i32([7 * s + i for s, k in enumerate(lens) for i in range(k)]),
                  i32([starts[s] for s, k in enumerate(lens) for _ in range(k)]), i32([k if i == 0 else 0 for k in lens for i in range(k)])]
        ring, St, o = ring0.clone(), S0.clone(), torch.zeros(n, VL * D, dtype=torch.bfloat16, device=DEV)
        save = torch.zeros(n, VL, D, D, device=DEV) if saves else None
        scratch = torch.empty(n * (qkv_l + 2 * VL), device=DEV)
        assert _lib().qwk_gdn_step(P(proj), ld, P(ring), P(cw), P(a_log), P(dt), P(nw), KL, VL, n, *map(P, tables), P(St), P(save), P(scratch),
                                   P(scratch[n * qkv_l:]), P(scratch[n * (qkv_l + VL):]), P(o), C.c_float(1e-6), S()) == 0
        torch.cuda.synchronize()
        if saves:
            for s in range(slots):
                assert torch.equal(save[starts[s] + runs[s] - 1], St[s])
        outs.append((ring[:slots], St[:slots], o[:M]))
    for other in outs[1:]:
        for a, b in zip(outs[0], other):
            assert torch.equal(a, b)


@pytest.mark.parametrize("QL,KVL,topk", [(24, 2, 512), (3, 1, 16), (32, 2, 4), (40, 2, 16)])
def test_flash_decode_parts_match_64_bits(QL, KVL, topk):
    """The partial softmaxes of 64 list entries against 64 bits: fp32 queries, scores and weights (three bf16 parts each), bf16 keys and values.
    A weight's relative error is the absolute one of its exponent: scores are sums of 256 products, the argument (up to 20) is rounded twice
    (2^-23 each) and __expf is good to two ulp: 6e-6.  More than 16 heads
    per KV head take the scalar kernel.  The merge of the parts against 64 bits: the output is rounded to bf16 (2^-9 of a value)."""
    ratio, page = 4, 256
    rn = gen(QL + topk)
    positions = [0, 1, 62, 63, 64, topk * ratio - 1, topk * ratio + 2, topk * ratio + 3, topk * ratio + 700]
    M, pages = len(positions), (positions[-1] + page) // page
    k, v = (rn(pages, page, KVL * 256).bfloat16() for _ in range(2))
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(3)).to(DEV, torch.int32)
    q, ldp = rn(M, QL, 256) * 2, QL * 512 + 8
    proj = rn(M, ldp)
    sel, sel_n, lists = torch.zeros(M, topk, dtype=torch.int32, device=DEV), torch.full((M,), -1, dtype=torch.int32, device=DEV), []
    for m, p in enumerate(positions):
        nb = (p + 1) // ratio
        toks = torch.arange(p + 1)
        if nb > topk:
            ch = torch.sort(torch.randperm(nb, generator=torch.Generator().manual_seed(m))[:topk]).values
            sel[m], sel_n[m] = ch.to(DEV, torch.int32), topk
            toks = torch.cat([(ch[:, None] * ratio + torch.arange(ratio)).reshape(-1), torch.arange(nb * ratio, p + 1)])
        lists.append(toks.to(DEV))
    nsplit = (topk * ratio + ratio + 63) // 64
    pm, pl = (torch.full((M, QL, nsplit), 7.0, device=DEV) for _ in range(2))
    pacc, o = torch.full((M, QL, nsplit, 256), float("nan"), device=DEV), torch.zeros(M, QL, 256, dtype=torch.bfloat16, device=DEV)
    assert _lib().qwk_qsa_attend(P(q), QL, KVL, M, P(i32([0] * M)), P(i32(positions)), P(k), P(v), None, None, pages, P(table), pages, P(sel), P(sel_n),
                                 topk, ratio, nsplit, P(pm), P(pl), P(pacc), P(proj), ldp, P(o), S()) == 0
    torch.cuda.synchronize()
    kf, vf = (x[table.long()].reshape(-1, KVL, 256).double() for x in (k, v))
    for m, toks in enumerate(lists):
        for h in range(QL):
            kv = h // (QL // KVL)
            s = kf[toks, kv] @ q[m, h].double() / 16
            for sp in range(nsplit):
                part = s[sp * 64:sp * 64 + 64]
                if len(part) == 0:
                    assert pm[m, h, sp] == float("-inf")
                    continue
                w = torch.exp(part - pm[m, h, sp].double())
                acc = w @ vf[toks[sp * 64:sp * 64 + 64], kv]
                assert abs(float(pm[m, h, sp]) - float(part.max())) < 1e-5
                assert abs(float(pl[m, h, sp]) / float(w.sum()) - 1) < 6e-6
                assert float((pacc[m, h, sp].double() - acc).norm() / acc.norm()) < 6e-6
            want = (torch.softmax(s, 0) @ vf[toks, kv]) * torch.sigmoid(proj[m, h * 512 + 256:h * 512 + 512].double())
            assert float((o[m, h].double() - want).norm() / want.norm()) < 2 ** -8


@pytest.mark.parametrize("heads", [12, 17])
def test_flash_decode_with_infinite_keys_and_values(heads):
    """Against 64 bits.  A key with one infinite value has a score of -inf for the queries of the other sign there: no weight, and no part of the list
    that holds nothing else counts.  A row that gives such a key a score of +inf is NaN; an infinite value is an infinite output where the key has weight.
    (The scalar kernel, which takes 17 heads a KV head, makes a part NaN whose warp meets such a key first: its lists have them later.)"""
    topk, ratio, page, KVL = 64, 4, 256, 2
    rn = gen(heads)
    lists = {70: [5], 65: [64], 64: list(range(64)), 200: list(range(64, 128)), 130: list(range(128, 131))} if heads == 12 else {70: [13], 200: [13, 100, 200]}
    positions = list(lists)
    M, QL = len(positions), heads * KVL
    k, v = (rn(M, page, KVL, 256).bfloat16() for _ in range(2))
    q = rn(M, KVL, heads, 256)
    for m, p in enumerate(positions):
        k[m, lists[p], :, 3] = float("inf")
        q[m, :, 1:, 3] = -q[m, :, 1:, 3].abs()
        q[m, 0, 0, 3] = 1.0                                # one head that the infinite keys win
        at = 64 if p == 64 else 35                          # a key with weight
        v[m, at, 1, 7], v[m, at, 0, 9] = float("inf"), float("-inf")
    table, sel, sel_n = torch.arange(M, dtype=torch.int32, device=DEV), torch.zeros(M, topk, dtype=torch.int32, device=DEV), torch.full((M,), -1, dtype=torch.int32, device=DEV)
    nsplit = (topk * ratio + ratio + 63) // 64
    pm, pl, pacc = torch.full((M, QL, nsplit), 7.0, device=DEV), torch.full((M, QL, nsplit), float("nan"), device=DEV), torch.full((M, QL, nsplit, 256), float("nan"), device=DEV)
    o, proj = torch.zeros(M, QL, 256, dtype=torch.bfloat16, device=DEV), torch.full((M, QL * 512), 30.0, device=DEV)          # gates of 1
    assert _lib().qwk_qsa_attend(P(q), QL, KVL, M, P(i32(range(M))), P(i32(positions)), P(k), P(v), None, None, M, P(table), 1, P(sel), P(sel_n),
                                 topk, ratio, nsplit, P(pm), P(pl), P(pacc), P(proj), QL * 512, P(o), S()) == 0
    torch.cuda.synchronize()
    got = o.view(M, KVL, heads, 256).double()
    for m, p in enumerate(positions):
        w = torch.softmax(torch.einsum("khd,tkd->kht", q[m].double(), k[m, :p + 1].double()) / 16, 2)
        # keys without weight have no part in the output, whatever their values are
        want = torch.where(w[..., None] > 0, w[..., None] * v[m, :p + 1].double().permute(1, 0, 2)[:, None], torch.where(w[..., None].isnan(), w[..., None], 0.0)).sum(2)
        assert bool(torch.isnan(want[0, 0]).all()) and bool(torch.isfinite(want).any())
        assert torch.equal(torch.isnan(got[m]), torch.isnan(want)), p
        inf = torch.isinf(want)
        assert torch.equal(got[m][inf], want[inf]) and torch.equal(torch.isinf(got[m]), inf)
        ok = torch.isfinite(want)
        assert float((got[m] - want)[ok].norm() / want[ok].norm()) < 2 ** -8


@pytest.mark.parametrize("off,nsplit", [(1, 6), (0, 6200)])
def test_flash_decode_with_scratch_at_any_address_and_many_splits(off, nsplit):
    """Sums that lie on 4 bytes, and more splits than a list needs (behind its end they hold nothing): what plain scratch gives, to the fp32 sums'
    order (the scalar kernel takes the first: 6e-6, and one rounding to bf16)."""
    QL, KVL, topk, positions = 4, 2, 64, [5, 200]
    rn, M = gen(3), len(positions)
    k, v = (rn(M, 256, KVL * 256).bfloat16() for _ in range(2))
    q, proj, table = rn(M, QL, 256), rn(M, QL * 512), i32(range(M))
    sel, sel_n = torch.zeros(M, topk, dtype=torch.int32, device=DEV), i32([-1] * M)
    outs = []
    for o_, n in ((0, 6), (off, nsplit)):
        pm, pl = (torch.full((M, QL, n), float("nan"), device=DEV) for _ in range(2))
        pacc = torch.full((M * QL * n * 256 + o_,), float("nan"), device=DEV)[o_:]
        o = torch.zeros(M, QL, 256, dtype=torch.bfloat16, device=DEV)
        assert _lib().qwk_qsa_attend(P(q), QL, KVL, M, P(i32(range(M))), P(i32(positions)), P(k), P(v), None, None, M, P(table), 1, P(sel), P(sel_n), topk, 4, n,
                                     P(pm), P(pl), P(pacc), P(proj), QL * 512, P(o), S()) == 0
        torch.cuda.synchronize()
        outs.append(o.float())
    assert bool(torch.isfinite(outs[0]).all())
    assert bool(((outs[1] - outs[0]).abs() <= outs[0].abs() * 2 ** -7 + 1e-5).all())


def test_router_rows_without_room_are_refused():
    """Rows so long that shared memory has no room for them in any plan: an error of the launcher, and nothing runs."""
    K_, nrs, M = 65536, 16, 8
    W, x = torch.zeros(nrs, K_, dtype=torch.bfloat16, device=DEV), torch.zeros(M, K_, dtype=torch.bfloat16, device=DEV)
    rs, pe, pw, ticket = torch.full((M, nrs), 7.0, device=DEV), torch.full((M, 2), -7, dtype=torch.int32, device=DEV), torch.full((M, 2), 7.0, device=DEV), i32([0])
    assert _lib().qwk_moe_router(P(W), P(x), P(rs), nrs, K_, M, K_, nrs, 2, 640, 0, nrs, P(pe), P(pw), None, P(ticket), None, None, 0, 0, S()) == -2
    torch.cuda.synchronize()
    assert bool((rs == 7.0).all()) and bool((pe == -7).all()) and bool((pw == 7.0).all()) and int(ticket) == 0


@pytest.mark.parametrize("size", [0.3, 1.0, 4.0])
def test_flash_decode_on_tensor_cores_is_as_exact_as_the_scalar_kernel(size):
    """The merged parts before bf16, against 64 bits, of both kernels: 17 heads per KV head take the scalar one, 12 of the same heads the tensor
    cores.  Bound: the scalar kernel's error and a tenth (420 rows of 256 values each: their mean error is known to a few percent)."""
    topk, ratio, page, KVL = 64, 4, 256, 2
    rn = gen(int(size * 10))
    positions = [3, 62, 64, 200, 255, 258, 300, 777, 1500, 3000]
    M, pages = len(positions), 12
    k, v = (rn(pages, page, KVL * 256).bfloat16() for _ in range(2))
    table, all_q = torch.arange(pages, dtype=torch.int32, device=DEV), rn(M, KVL, 17, 256) * size
    sel, sel_n = torch.zeros(M, topk, dtype=torch.int32, device=DEV), torch.full((M,), -1, dtype=torch.int32, device=DEV)
    lists = []
    for m, p in enumerate(positions):
        nb, toks = (p + 1) // ratio, torch.arange(p + 1, device=DEV)
        if nb > topk:
            ch = torch.sort(torch.randperm(nb, generator=torch.Generator().manual_seed(m))[:topk]).values.to(DEV)
            sel[m], sel_n[m] = ch.int(), topk
            toks = torch.cat([(ch[:, None] * ratio + torch.arange(ratio, device=DEV)).reshape(-1), toks[nb * ratio:]])
        lists.append(toks)
    nsplit, errs = (topk * ratio + ratio + 63) // 64, []
    for heads in (12, 17):
        QL, q = heads * KVL, all_q[:, :, :heads].contiguous()
        pm, pl = (torch.full((M, QL, nsplit), float("-inf"), device=DEV) for _ in range(2))
        pacc, o, proj = torch.zeros(M, QL, nsplit, 256, device=DEV), torch.zeros(M, QL, 256, dtype=torch.bfloat16, device=DEV), rn(M, QL * 512)
        assert _lib().qwk_qsa_attend(P(q), QL, KVL, M, P(i32([0] * M)), P(i32(positions)), P(k), P(v), None, None, pages, P(table), pages, P(sel), P(sel_n),
                                     topk, ratio, nsplit, P(pm), P(pl), P(pacc), P(proj), QL * 512, P(o), S()) == 0
        torch.cuda.synchronize()
        total = 0.0
        for m, toks in enumerate(lists):
            n = (len(toks) + 63) // 64
            for kv in range(KVL):
                kf, vf = (x.view(-1, KVL, 256)[toks, kv].double() for x in (k, v))
                want = torch.softmax(all_q[m, kv, :12].double() @ kf.T / 16, 1) @ vf
                at = slice(kv * heads, kv * heads + 12)
                w = torch.exp(pm[m, at, :n].double() - pm[m, at, :n].double().amax(1, keepdim=True))
                got = (w[..., None] * pacc[m, at, :n].double()).sum(1) / (w * pl[m, at, :n].double()).sum(1, keepdim=True)
                total += float(((got - want).norm(dim=1) / want.norm(dim=1)).pow(2).sum())
        errs.append((total / (M * KVL * 12)) ** 0.5)
    assert errs[0] < 1.1 * errs[1], errs


@pytest.mark.parametrize("pairs,layers,state", [([[0, 2], [2, 0], [1, -1]], 3, 48 * 128 * 128), ([[1, 1]], 1, 4), ([[0, 1], [1, 3]], 2, 4096 * 3 + 8)])
def test_accepted_states_are_copied_whole(pairs, layers, state):
    """Every value of an accepted row's state, whatever its size (pieces of 16 KB, a last one that is not whole); rejected slots stay."""
    rn = gen(state)
    rows, slots = 4, 3
    save, St = rn(layers, rows, state), rn(layers, slots, state)
    want = St.clone()
    for s, r in pairs:
        if r >= 0:
            want[:, s] = save[:, r]
    ptrs = torch.tensor([St[i].data_ptr() for i in range(layers)], dtype=torch.int64, device=DEV)
    assert _lib().qwk_gdn_accept(P(ptrs), P(save), layers, rows, C.c_longlong(state), P(i32(pairs)), len(pairs), S()) == 0
    assert torch.equal(St, want)


def test_logistic_function_against_64_bits():
    """The gates of a delta-net chunk, over all of fp32's range and most densely around 0.  e^-x: the rounding of x log2(e) and of that constant, |x| 2^-23
    together, and two units of the exponential, of which 1 / (1 + e^-x) keeps the share e^-x / (1 + e^-x); one rounding of the sum and one unit of the
    reciprocal.  Results below 2^-126 are values of their own, in steps of 2^-149; where e^-x is infinite (x < -88.7) the result is 0."""
    KL, VL, D = 1, 48, 128
    edges = torch.tensor([0.0, -0.0, 1e-30, -1e-30, -87.0, -87.3, -87.4, -88.0, -88.5, -88.7, -88.8, -104.0, 88.0, 104.0, 3e38, -3e38, float("inf"), float("-inf"), float("nan")])
    x = torch.cat([torch.linspace(-104, 104, 40001), torch.linspace(-4, 4, 20001), torch.linspace(-89, -86, 3001), edges])
    M = (len(x) + VL - 1) // VL
    x = torch.cat([x, torch.zeros(M * VL - len(x))]).to(DEV)
    qkv_l = (2 * KL + VL) * D
    ld = qkv_l + VL * D + 2 * VL
    proj = torch.zeros(M, ld, device=DEV)
    proj[:, qkv_l + VL * D:qkv_l + VL * D + VL] = x.view(M, VL)
    ring, cw, al, dt = torch.zeros(1, 16, qkv_l, device=DEV), torch.zeros(qkv_l, 4, device=DEV), torch.zeros(VL, device=DEV), torch.zeros(VL, device=DEV)
    qkv, decay, beta = torch.zeros(M, qkv_l, device=DEV), torch.zeros(M, VL, device=DEV), torch.zeros(M, VL, device=DEV)
    run_len = i32([M] + [0] * (M - 1))
    assert _lib().qwk_gdn_conv(P(proj), ld, P(ring), P(cw), P(al), P(dt), KL, VL, M, P(i32([0] * M)), P(i32(range(M))), P(i32([0] * M)), P(run_len), P(qkv),
                               P(decay), P(beta), C.c_float(1e-6), S()) == 0
    got, xd = beta.view(-1).double(), x.double()
    want = torch.sigmoid(xd)
    share = torch.sigmoid(-xd)
    tol = want * (share * (xd.abs().clamp(max=104) * 2 ** -23 + 2 ** -22) + 2 ** -24 + 2 ** -23) + 2 ** -149
    tol = torch.where(xd < -88.7, want + 2 ** -149, tol)
    ok = torch.where(torch.isnan(xd), torch.isnan(got), (got - want).abs() <= tol)
    assert bool(ok.all()), (x[~ok][:8].tolist(), got[~ok][:8].tolist())
