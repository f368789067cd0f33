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
