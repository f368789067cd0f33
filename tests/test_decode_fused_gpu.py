"""Decode kernels with a collective inside them, ranks emulated on one GPU: the kernels of all ranks that send are launched before any that
receives, in one stream, so every word that a kernel waits for is there before it starts (GPU only)."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def P(t):
    return None if t is None else C.c_void_p(t.data_ptr())


class Ranks:
    """One region per rank with the receive slots of the three kinds of collective (0 all-reduce, 1 all-gather, 2 reduce-scatter)."""

    def __init__(self, R, rows, words):
        from qwb200.ops import structs as S
        self.R, self.rows, self.words = R, rows, words
        self.slot = [rows * n * 8 for n in words]
        self.off = [sum(2 * R * s for s in self.slot[:k]) for k in range(3)]
        self.region = [torch.zeros(sum(2 * R * s for s in self.slot), dtype=torch.uint8, device=DEV) for _ in range(R)]
        self.base = torch.full((1,), 4096, dtype=torch.int32, device=DEV)
        self.p = []
        for r in range(R):
            p = S.QwP2P()
            for d in range(R):
                p.peer[d] = self.region[d].data_ptr()
            p.ranks, p.rank, p.base = R, r, self.base.data_ptr()
            for k in range(3):
                p.off_recv[k], p.slot_bytes[k] = self.off[k], self.slot[k]
            self.p.append(p)

    def words_on(self, d, kind, k):
        """[sender][row][word] payloads that rank d holds of collective k; every word must carry its number."""
        at = self.off[kind] + (k & 1) * self.R * self.slot[kind]
        w = self.region[d][at:at + self.R * self.slot[kind]].view(torch.int32).view(self.R, self.rows, self.words[kind], 2)
        assert torch.all(w[..., 1] == 4096 + k)
        return w[..., 0].contiguous()


@pytest.mark.parametrize("R", [1, 2, 4])
@pytest.mark.parametrize("M", [1, 3, 9, 20])
def test_expert_output_to_block_input_through_the_fused_kernels(R, M):
    """Expert outputs of every rank (reduce-scatter) -> combine and down projection (all-reduce) -> up projection and mean (all-gather):
    against 64 bits on the same bf16 operands.  fp32 sums of exact products: 1e-5; the block input is rounded to bf16 once."""
    from qwb200.models.quant import dequantize_q4, quantize_q4, to_engine_order
    from qwb200.ops import lib as qlib
    L = qlib.load(True)
    s = lambda: C.c_void_p(torch.cuda.current_stream().cuda_stream)
    H, hc, rank_, n_inj, F, E, k_, eps = 512, 4, 32, 4, 128, 8, 4, 1e-6
    SH, SF, El, down = H // R, 64, E // R, rank_ + n_inj
    ld = hc + hc * down
    g = torch.Generator(device=DEV).manual_seed(R * 100 + M)
    rn = lambda *n: torch.randn(*n, generator=g, device=DEV)
    net = Ranks(R, M, [ld, SH, SH])
    err = torch.zeros(2, dtype=torch.int32, device=DEV)
    L.qwk_set_error_word(P(err))
    nxt = lambda r, *a: L.qwk_fuse_next(C.byref(net.p[r]), *a)

    # ---- experts: rank r holds E / R of them and a slice of the shared expert
    experts = torch.stack([torch.randperm(E, generator=g, device=DEV)[:k_] for _ in range(M)])
    weight = torch.rand(M, k_, generator=g, device=DEV)
    h = rn(M, k_, F).to(torch.bfloat16)
    total = torch.zeros(M, H, dtype=torch.float64, device=DEV)
    for r in range(R):
        packed, scale = quantize_q4(rn(El * H, F) * 0.05, scale_dtype=torch.bfloat16)
        W2 = dequantize_q4(packed, scale).double().view(El, H, F)
        words, sd, sh = to_engine_order(packed).contiguous(), (rn(H, SF) * 0.05).to(torch.bfloat16), rn(M, SF).to(torch.bfloat16)
        local = experts // El == r
        pe = torch.where(local, experts % El, -1).to(torch.int32).contiguous()
        assert nxt(r, -1, 0, 0, 2, 1, 2, SH) == 0
        assert L.qwk_moe_down_combine(P(words), P(scale), P(h), P(pe), P(weight), M, k_, F, H, P(sd), SF, P(sh), SF, None, H, s()) == 0
        total += sh.double() @ sd.double().T
        for m in range(M):
            for j in range(k_):
                if local[m, j]:
                    total[m] += float(weight[m, j]) * (W2[int(pe[m, j])] @ h[m, j].double())
    torch.cuda.synchronize()
    for d in range(R):
        got = net.words_on(d, 2, 1).view(torch.float32).double().sum(0)
        assert float((got - total[:, d * SH:(d + 1) * SH]).norm() / total.norm()) < 1e-5

    # ---- mixer: every rank its columns
    X, inj_prev, w1 = rn(M, hc, H), rn(M, hc), 1 + 0.1 * rn(hc, H)
    Wd, Wu = (rn(down, hc, H) * 0.05).to(torch.bfloat16), (rn(H, hc, rank_) * 0.1).to(torch.bfloat16)
    cols = [slice(r * SH, (r + 1) * SH) for r in range(R)]
    xs, ws, keep = [], [], []
    for r in range(R):
        x, xo, w, wd = X[..., cols[r]].contiguous(), torch.zeros(M, hc, SH, device=DEV), w1[:, cols[r]].contiguous(), Wd[..., cols[r]].contiguous()
        pend = torch.zeros(M, SH, device=DEV)                       # only its presence counts: the sums come out of the slots
        assert nxt(r, 2, 1, SH, 0, 2, 1, ld) == 0
        assert L.qwk_hc_down(P(x), P(xo), P(pend), SH, P(inj_prev), P(w), P(wd), None, ld, SH, hc, down, M, s()) == 0
        xs.append(xo)
        ws.append(w)
        keep += [x, wd, pend]
    inj = [torch.zeros(M, hc, device=DEV) for _ in range(R)]
    for r in range(R):
        wu = Wu[cols[r]].contiguous()
        assert nxt(r, 0, 2, ld, 1, 3, 1, SH) == 0
        assert L.qwk_hc_up_mix(None, ld, P(wu), P(xs[r]), P(ws[r]), SH, hc, rank_, n_inj, H, C.c_float(eps), M, P(inj[r]), hc, None, H, r * SH, s()) == 0
        keep.append(wu)
    torch.cuda.synchronize()
    assert err.tolist() == [0, 0]
    L.qwk_set_error_word(None)
    x64 = X.double() + total[:, None] * (2 * torch.sigmoid(inj_prev.double() / hc))[..., None]
    x = torch.cat(xs, 2)
    assert torch.allclose(x.double(), x64, rtol=1e-5, atol=1e-5)
    y = (x * w1).to(torch.bfloat16).double()
    part = torch.einsum("msc,jsc->msj", y, Wd.double())
    for d in range(R):
        got = net.words_on(d, 0, 2).view(torch.float32).double().sum(0)
        assert torch.allclose(got[:, :hc], x.double().pow(2).sum(-1), rtol=1e-5)
        assert float((got[:, hc:].view(M, hc, down) - part).norm() / part.norm()) < 1e-5
    rr = torch.rsqrt(x.double().pow(2).mean(-1) + eps)
    d64 = (rr[..., None] * part).sum(1)
    gate = torch.sigmoid(torch.einsum("csr,mr->msc", Wu.double(), torch.nn.functional.silu(d64[:, :rank_] / hc)))
    want = (gate * y * rr[..., None]).mean(1)
    for d in range(R):
        bits = net.words_on(d, 1, 3).to(torch.int16).view(torch.bfloat16)          # [sender][row][its columns]
        got = torch.cat(list(bits), 1).double()
        assert float((got - want).norm() / want.norm()) < 5e-3
        assert torch.equal(inj[d], inj[0]) and float((inj[d].double() - d64[:, rank_:]).norm() / d64[:, rank_:].norm()) < 1e-5
