"""Kernels of a prefill chunk and of the vision tower at the edges of their forms (GPU only)."""
import ctypes as C

import pytest
import torch

from test_step_kernels_gpu import DEV, P, S, _lib, gen, i32

pytestmark = pytest.mark.gpu


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
