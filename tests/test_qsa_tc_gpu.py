"""Attention of a prefill chunk on the tcgen05 tensor cores (`ops/csrc/qsa_tc.cu`) against 64 bits and against the kernel that gathers
the chosen rows (`ops/csrc/qsa_mma.cuh`)."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _setup(QL, KVL, base, M, topk, seed, scale=1.0):
    """A run of M rows at `base` in slot 1 of two, its pages shuffled; the pool's rows behind the run are NaN."""
    dev = torch.device("cuda:0")
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=g, device=dev)
    ratio, page, D = 4, 256, 256
    pages = (base + M + page - 1) // page + 1
    k, v = (rn(2 * pages, page, KVL * D).bfloat16() for _ in range(2))
    table = torch.randperm(2 * pages, generator=torch.Generator().manual_seed(seed)).to(dev, torch.int32).view(2, pages)
    at = torch.arange(base + M, pages * page, device=dev)
    for pool in (k, v):
        pool[table[1][at // page].long(), at % page] = float("nan")
    ldp = QL * 2 * D + 40
    proj, q = rn(M, ldp), rn(M, QL, D) * scale
    pos = torch.arange(base, base + M, dtype=torch.int32, device=dev)
    sel, sel_n = torch.zeros(M, topk, dtype=torch.int32, device=dev), torch.full((M,), -1, dtype=torch.int32, device=dev)
    seen = torch.arange(base + M, device=dev)[None] <= pos[:, None]
    for m in range(M):
        nb = (base + m + 1) // ratio
        if nb > topk:
            ch = torch.sort(torch.randperm(nb, generator=torch.Generator().manual_seed(seed + m))[:topk]).values.to(dev)
            sel[m], sel_n[m] = ch.int(), topk
            chosen = torch.zeros(nb, dtype=torch.bool, device=dev)
            chosen[ch] = True
            seen[m, :nb * ratio] &= chosen.repeat_interleave(ratio)
    return dict(q=q, k=k, v=v, table=table, proj=proj, ldp=ldp, pos=pos, sel=sel, sel_n=sel_n, seen=seen, slot=torch.ones_like(pos), pages=pages)


def _exact(t, QL, KVL, base, M):
    rows = t["table"][1].long()
    kf, vf = (x[rows].reshape(-1, KVL, 256)[:base + M].double() for x in (t["k"], t["v"]))
    q = t["q"].bfloat16().double()
    out = torch.empty(M, QL, 256, dtype=torch.float64, device=q.device)
    for h in range(QL):
        kv = h // (QL // KVL)
        s = (q[:, h] @ kf[:, kv].T / 16).masked_fill(~t["seen"], float("-inf"))
        gate = t["proj"][:, h * 512 + 256:h * 512 + 512].double()
        out[:, h] = (torch.softmax(s, 1) @ vf[:, kv]) * torch.sigmoid(gate)
    return out


@pytest.mark.parametrize("QL,KVL,base,M,topk,scale", [
    (24, 2, 0, 1, 512, 1.0), (24, 2, 0, 70, 512, 1.0), (24, 2, 127, 2, 512, 1.0), (24, 2, 0, 300, 512, 3.0), (24, 2, 2040, 150, 512, 1.0),
    (24, 2, 1001, 129, 64, 3.0), (12, 1, 6000, 33, 512, 1.0), (3, 1, 250, 400, 32, 1.0), (8, 2, 5, 64, 4, 1.0), (16, 1, 383, 257, 16, 1.0)])
def test_matches_64_bits_and_the_gathering_kernel(QL, KVL, base, M, topk, scale):
    """Rows that see every key and rows with chosen groups, groups that are open or just closed, tiles that end with the context.  Bound:
    weights and the result rounded to bf16 (2^-9 each of a value), and no further from 64 bits than 1.1 times the gathering kernel."""
    from qwb200.ops import lib as qlib
    L = qlib.load(True)
    t = _setup(QL, KVL, base, M, topk, 7 * M + base, scale)
    P = lambda x: C.c_void_p(x.data_ptr())
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    want = _exact(t, QL, KVL, base, M)
    err = lambda o: float((o.double() - want).norm() / want.norm())
    gathered, o = (torch.zeros(M, QL, 256, dtype=torch.bfloat16, device="cuda:0") for _ in range(2))
    last, ld = base + M - 1, (base + M) // 4 + 8
    mask = torch.empty(M, ld, dtype=torch.int32, device="cuda:0")
    pool = [P(t["k"]), P(t["v"])]
    assert L.qwk_qsa_attend_mma(P(t["q"]), QL, KVL, M, P(t["slot"]), P(t["pos"]), *pool, None, None, 2 * t["pages"], P(t["table"]), t["pages"],
                                P(t["sel"]), P(t["sel_n"]), topk, 4, P(t["proj"]), t["ldp"], P(gathered), s) == 0
    for p in range(last + 1, (last + 16) // 16 * 16):          # as the prep kernel leaves them
        t["k"][t["table"][1][p // 256], p % 256] = t["v"][t["table"][1][p // 256], p % 256] = 0
    first_host = (last // 256 + 1) * 2 // 3                      # pages from here on also lie in a pool of their own, read as staged and as host rows
    moved = t["table"].clone()
    hk, hv = (torch.cat([x[t["table"][1, first_host:].long()], x[:1]]) for x in (t["k"], t["v"]))
    moved[1, first_host:] = 2 * t["pages"] + torch.arange(t["pages"] - first_host, device="cuda:0", dtype=torch.int32)
    for table, host, staged in ((t["table"], [None, None], 0), (moved, [P(hk), P(hv)], 1), (moved, [P(hk), P(hv)], 0)):
        before = o.clone()
        o.zero_()
        assert L.qwk_qsa_attend_tc(P(t["q"]), QL, KVL, M, last, P(t["slot"]), P(t["pos"]), *pool, *host, staged, 2 * t["pages"], P(table), t["pages"],
                                   P(t["sel"]), P(t["sel_n"]), topk, P(mask), ld, P(t["proj"]), t["ldp"], P(o), s) == 0
        torch.cuda.synchronize()
        assert host[0] is None or torch.equal(o, before)
    assert err(o) < 4e-3 and err(o) < 1.1 * err(gathered) + 1e-5


def _launch(L, t, QL, KVL, M, last, o, dev, host, staged, n_dev, topk, proj=None, q=None):
    P = lambda x: None if x is None else C.c_void_p(x.data_ptr())
    ld = last // 4 + 9
    mask = torch.empty(M, ld, dtype=torch.int32, device="cuda:0")
    rc = L.qwk_qsa_attend_tc(P(t["q"] if q is None else q), QL, KVL, M, last, P(t["slot"]), P(t["pos"]), *map(P, dev), *map(P, host), staged, n_dev, P(t["table"]),
                             t["pages"], P(t["sel"]), P(t["sel_n"]), topk, P(mask), ld, P(t["proj"] if proj is None else proj), t["ldp"], P(o),
                             C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return rc


def _gather(L, t, QL, KVL, M, o, topk, proj=None, q=None):
    P = lambda x: C.c_void_p(x.data_ptr())
    rc = L.qwk_qsa_attend_mma(P(t["q"] if q is None else q), QL, KVL, M, P(t["slot"]), P(t["pos"]), P(t["k"]), P(t["v"]), None, None, 2 * t["pages"], P(t["table"]),
                              t["pages"], P(t["sel"]), P(t["sel_n"]), topk, 4, P(t["proj"] if proj is None else proj), t["ldp"], P(o),
                              C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return rc


def _zero_tail(t, last):
    """The rows behind the last as the kernel before this one leaves them."""
    for p in range(last + 1, (last + 16) // 16 * 16):
        t["k"][t["table"][1][p // 256], p % 256] = t["v"][t["table"][1][p // 256], p % 256] = 0


@pytest.mark.parametrize("base,M,topk", [(0, 70, 512), (700, 130, 32)])
def test_a_pool_without_device_pages(base, M, topk):
    """Every page in the other pool, read as a staged copy and in place: the bits of the same pages in the first pool."""
    from qwb200.ops import lib as qlib
    L, QL, KVL, last = qlib.load(True), 12, 1, base + M - 1
    t = _setup(QL, KVL, base, M, topk, 11)
    _zero_tail(t, last)
    outs = [torch.zeros(M, QL, 256, dtype=torch.bfloat16, device="cuda:0") for _ in range(3)]
    assert _launch(L, t, QL, KVL, M, last, outs[0], [t["k"], t["v"]], [None, None], 0, 2 * t["pages"], topk) == 0
    for staged in (1, 0):
        assert _launch(L, t, QL, KVL, M, last, outs[1 + staged], [None, None], [t["k"], t["v"]], staged, 0, topk) == 0
        assert torch.equal(outs[0], outs[1 + staged])


@pytest.mark.parametrize("off_q,off_proj,off_o", [(2, 0, 0), (0, 2, 0), (0, 0, 2), (2, 2, 6)])
def test_addresses_off_16_bytes_are_gathered(off_q, off_proj, off_o):
    """Queries and gates on 8 bytes and an output on 4: what the rule accepts is served, by the kernel whose loads are that narrow."""
    from qwb200.ops import lib as qlib
    L, QL, KVL, base, M, topk = qlib.load(True), 12, 1, 300, 70, 32
    t, last = _setup(QL, KVL, base, M, topk, 5), base + M - 1
    _zero_tail(t, last)
    at = lambda x, off: torch.cat([x.new_zeros(off), x.reshape(-1)])[off:].view(x.shape)
    q, proj = at(t["q"], off_q), at(t["proj"], off_proj)
    got, want = (at(torch.zeros(M, QL, 256, dtype=torch.bfloat16, device="cuda:0"), off_o) for _ in range(2))
    assert q.data_ptr() % 16 == off_q * 4 and proj.data_ptr() % 16 == off_proj * 4 and got.data_ptr() % 16 == off_o * 2 % 16
    assert _launch(L, t, QL, KVL, M, last, got, [t["k"], t["v"]], [None, None], 0, 2 * t["pages"], topk, proj=proj, q=q) == 0
    assert _gather(L, t, QL, KVL, M, want, topk, proj=proj, q=q) == 0
    assert torch.equal(got, want)


@pytest.mark.parametrize("base,M,topk,host", [(0, 70, 512, False), (600, 90, 32, False), (600, 90, 32, True), (1500, 300, 64, False)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_values_that_are_not_finite_reach_only_rows_that_attend_to_them(base, M, topk, host, bad):
    """Single values of V that are not finite, at a key that some rows chose and at positions inside the chunk: the rows that attend to them show what the
    gathering kernel shows, every other row of the same tiles is as close to 64 bits as without them (weights and result rounded to bf16)."""
    from qwb200.ops import lib as qlib
    L, QL, KVL, last = qlib.load(True), 24, 2, base + M - 1
    t = _setup(QL, KVL, base, M, topk, base + M)
    _zero_tail(t, last)
    want = _exact(t, QL, KVL, base, M)
    cols = {base // 3: 5, base + M // 2: 256 + 77, last: 130}          # of K/V head 0, 1 and 0
    hit = torch.zeros(M, QL, 256, dtype=torch.bool, device="cuda:0")
    for at, c in cols.items():
        t["v"][t["table"][1][at // 256], at % 256, c] = bad
        hit[:, c // 256 * 12:c // 256 * 12 + 12, c % 256] |= t["seen"][:, at, None]
    got, gathered = (torch.zeros(M, QL, 256, dtype=torch.bfloat16, device="cuda:0") for _ in range(2))
    n_dev = 2 * t["pages"]
    assert _gather(L, t, QL, KVL, M, gathered, topk) == 0
    if host:
        pools, n_dev = ([None, None], [t["k"], t["v"]]), 0
    else:
        pools = ([t["k"], t["v"]], [None, None])
    assert _launch(L, t, QL, KVL, M, last, got, *pools, 0, n_dev, topk) == 0
    assert bool(hit.any()) and not bool(hit.all())
    assert torch.equal(torch.isfinite(gathered), ~hit) and torch.equal(torch.isfinite(got), ~hit)
    assert torch.equal(torch.isnan(got), torch.isnan(gathered))
    assert float((got.double() - want)[~hit].norm() / want[~hit].norm()) < 4e-3


def test_what_it_does_not_take():
    """Other group sizes, masks that do not fit, rows of the projection off 16 bytes are refused by the kernel; contexts that are long for
    their chunk, and chunks too small to matter, are the gathering kernel's."""
    from qwb200.ops import lib as qlib
    L = qlib.load(True)
    take = lambda **k: L.qwk_qsa_takes_tc(*{**dict(QL=24, KVL=2, M=100, last=4000, topk=512, ratio=4, ld=20000, ldp=13952), **k}.values())
    assert take() == 1 and take(M=1, last=1000) == 1 and take(M=4096, last=4095) == 1 and take(M=2048, last=16384 + 2047) == 1
    assert not any((take(ratio=8), take(last=40, M=100), take(ld=31), take(ldp=13953), take(QL=23), take(QL=0), take(KVL=0)))
    assert not any((take(last=1 << 20), take(M=100, last=99), take(M=1, last=9000), take(M=300, last=16684), take(M=2048, last=32000)))
    none = [None] * 4
    assert L.qwk_qsa_attend_tc(None, 23, 2, 4, 100, None, None, *none, 0, 1, None, 1, None, None, 512, None, 4, None, 13952, None, None) == -1
