"""tcgen05 GEMM numerics against a plain fp32 matmul (GPU only)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,N,K", [(128, 128, 64), (128, 128, 256), (256, 384, 2560), (200, 324, 2560), (4096, 512, 2560),
                                   (77, 130, 328),
                                   # products that run in CTA pairs, with ragged edges
                                   (1024, 2560, 320), (2000, 1536, 640), (4096, 1200, 128), (1111, 10240, 64)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_gemm_tc_matches_fp32(T, N, K, out_dtype):
    from qwb200.ops import kernels as K_
    g = torch.Generator(device="cuda").manual_seed(T + N + K)
    A = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    W = (torch.randn(N, K, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    ldc = (N + 7) // 8 * 8 + 8
    out = torch.full((T, ldc), 768.0, dtype=out_dtype, device="cuda")      # guard columns detect stray writes
    K_.gemm_bf16_tc(A, W, out=out[:, :N])
    torch.cuda.synchronize()
    ref = A.float() @ W.float().T
    assert torch.all(out[:, N:].float() == 768.0)
    tol = 2e-2 if out_dtype == torch.bfloat16 else 2e-3
    err = float((out[:, :N].float() - ref).abs().max() / ref.abs().max())
    assert err < tol, err


@pytest.mark.parametrize("T,N,K", [(1, 128, 512), (100, 2560, 6144), (100, 1793, 2560), (129, 324, 10240), (64, 100, 520), (200, 130, 4304),
                                   (300, 2560, 1024), (128, 128, 4096),
                                   # the line between the forms: 129-row and 257-row products in pairs, padded pairs
                                   (129, 10240, 1152), (777, 4304, 512), (257, 16480, 128)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_gemm_tc_split_and_padded_forms_match_64_bits(T, N, K, out_dtype):
    """Few tiles shared by clusters of 2, 4 and 8 CTAs (k blocks that do not divide evenly, ragged rows and columns) and the padded
    pair form: fp32 sums of exact products (1e-5 of the result's size for K <= 10240; bf16 output 2^-9 more), twice the
    same bits, and nothing outside the result written."""
    from qwb200.ops import kernels as K_
    g = torch.Generator(device="cuda").manual_seed(T + N + K)
    A = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    W = (torch.randn(N, K, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    ldc = (N + 7) // 8 * 8 + 8
    out = torch.full((T + 2, ldc), 768.0, dtype=out_dtype, device="cuda")
    K_.gemm_bf16_tc(A, W, out=out[:T, :N])
    again = torch.empty_like(out)
    K_.gemm_bf16_tc(A, W, out=again[:T, :N])
    torch.cuda.synchronize()
    ref = A.double() @ W.double().T
    assert torch.all(out[:, N:].float() == 768.0) and torch.all(out[T:].float() == 768.0)
    assert torch.equal(out[:T, :N], again[:T, :N])
    err = float((out[:T, :N].double() - ref).norm() / ref.norm())
    assert err < (1e-5 if out_dtype == torch.float32 else 2 ** -8), err


@pytest.mark.parametrize("Nw,K,counts", [(256, 256, [5, 0, 130, 128, 1, 300]), (1280, 2560, [80, 200, 0, 33]),
                                         (2560, 640, [77, 129, 64])])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_grouped_q4_gemm_matches_fp32(Nw, K, counts, out_dtype):
    """Grouped tcgen05 GEMM whose W operand is dequantised from q4 inside the kernel: every group's rows against
    A @ dequant(W_group)^T in fp32, rows of unused tile entries and guard rows untouched."""
    import ctypes as C
    from qwb200.models.quant import dequantize_q4, quantize_q4, to_engine_order
    from qwb200.ops import lib as qlib
    L = qlib.load(True)
    dev = torch.device("cuda:0")
    g = torch.Generator(device="cuda").manual_seed(Nw + K)
    E = len(counts)
    W = torch.randn(E * Nw, K, generator=g, device=dev) * 0.05
    packed, scale = quantize_q4(W, scale_dtype=torch.bfloat16)
    Wd = dequantize_q4(packed, scale).to(torch.bfloat16).float()       # the kernel rounds value * scale to bf16
    words = to_engine_order(packed).contiguous()
    rows = sum(counts)
    A = torch.randn(rows + 128, K, generator=g, device=dev).to(torch.bfloat16)
    tiles, r0 = [], 0
    for e, n in enumerate(counts):
        for t in range(0, n, 128):
            tiles.append([r0 + t, min(128, n - t), e * Nw, 0])
        r0 += n
    tiles.append([0, 0, 0, 0])                                   # an unused entry
    tt = torch.tensor(tiles, dtype=torch.int32, device=dev)
    out = torch.full((rows + 128, Nw), 768.0, dtype=out_dtype, device=dev)
    P = lambda t: C.c_void_p(t.data_ptr())
    rc = L.qwk_gemm_q4_tc_grouped(P(A), P(words), P(scale), P(out), P(tt), len(tiles), rows, E * Nw, Nw, K, K, Nw,
                                  1 if out_dtype == torch.bfloat16 else 0, C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    assert torch.all(out[rows:].float() == 768.0)
    r0 = 0
    tol = 2e-2 if out_dtype == torch.bfloat16 else 2e-3
    for e, n in enumerate(counts):
        if n:
            ref = A[r0:r0 + n].float() @ Wd[e * Nw:(e + 1) * Nw].float().T
            err = float((out[r0:r0 + n].float() - ref).abs().max() / ref.abs().max())
            assert err < tol, (e, err)
        r0 += n


@pytest.mark.parametrize("F,K,counts", [(128, 128, [1, 0, 16, 17, 64, 65, 128, 129, 2]), (640, 2560, [3, 70, 1, 64, 300, 0, 20]),
                                        (640, 256, [1] * 400 + [0] * 40 + [100] * 9)])      # the last: several units per block, both slot forms
def test_grouped_q4_swiglu_matches_fp32(F, K, counts):
    """Gate and up products with the activation in the epilogue: every row against silu(A @ gate^T) * (A @ up^T) in fp32 (bf16
    output: half a unit in the last place, 2^-9, plus the fp32 sums); rows behind the last one untouched."""
    import ctypes as C
    from qwb200.models.quant import dequantize_q4, quantize_q4, to_engine_order
    from qwb200.ops import lib as qlib
    L = qlib.load(True)
    g = torch.Generator(device="cuda").manual_seed(F + K)
    E = len(counts)
    W = torch.randn(E * 2 * F, K, generator=g, device="cuda") * 0.05
    packed, scale = quantize_q4(W, scale_dtype=torch.bfloat16)
    Wd = dequantize_q4(packed, scale).to(torch.bfloat16).float()
    words = to_engine_order(packed).contiguous()
    rows = sum(counts)
    A = torch.randn(rows, K, generator=g, device="cuda").to(torch.bfloat16)
    tiles, r0 = [], 0
    for e, n in enumerate(counts):
        tiles += [[r0 + t, min(128, n - t), e * 2 * F, 0] for t in range(0, n, 128)]
        r0 += n
    tiles += [[0, 0, 0, 0]] * 3
    tt = torch.tensor(tiles, dtype=torch.int32, device="cuda")
    out = torch.full((rows + 16, F + 8), 768.0, dtype=torch.bfloat16, device="cuda")
    P = lambda t: C.c_void_p(t.data_ptr())
    rc = L.qwk_gemm_q4_tc_swiglu(P(A), P(words), P(scale), P(out), P(tt), len(tiles), rows, E * 2 * F, F, K, K, F + 8,
                                 C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    assert torch.all(out[rows:].float() == 768.0) and torch.all(out[:, F:].float() == 768.0)
    r0 = 0
    for e, n in enumerate(counts):
        a, w = A[r0:r0 + n].float(), Wd[e * 2 * F:(e + 1) * 2 * F].float()
        ref = torch.nn.functional.silu(a @ w[:F].T) * (a @ w[F:].T)
        assert torch.allclose(out[r0:r0 + n, :F].float(), ref, rtol=2 ** -8, atol=1e-3), e
        r0 += n


@pytest.mark.parametrize("T,N,K,ks", [(200, 324, 10240, 3), (128, 128, 256, 2), (77, 40, 640, 1)])
def test_gemm_tc_split_k_partials_add_up(T, N, K, ks):
    """Split-K form: the partial products of the shares of K, added in order, equal the full product."""
    import ctypes as C
    from qwb200.ops import lib as qlib
    L = qlib.load(True)
    g = torch.Generator(device="cuda").manual_seed(T + N + K)
    A = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    W = (torch.randn(N, K, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    ldc = (N + 7) // 8 * 8
    out = torch.full((ks, T + 3, ldc), 768.0, device="cuda")
    P = lambda t: C.c_void_p(t.data_ptr())
    rc = L.qwk_gemm_bf16_tc_splitk(P(A), P(W), P(out), T, N, K, K, K, ldc, ks, (T + 3) * ldc,
                                   C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    assert torch.all(out[:, T:] == 768.0) and torch.all(out[:, :, N:] == 768.0)
    ref = A.float() @ W.float().T
    got = out[:, :T, :N].sum(0)
    err = float((got - ref).abs().max() / ref.abs().max())
    assert err < 2e-3, err


@pytest.mark.parametrize("T,N,K", [(1024, 2048, 256), (1500, 512, 192), (4096, 2560, 1536)])      # the last: the out projection of a chunk on 4 ranks (CTA-pair form)
def test_gemm_tc_reduce_scatter_epilogue_on_emulated_ranks(T, N, K):
    """The tensor-parallel forms of the product on four ranks emulated on one GPU: with the reduce-scatter epilogue every
    rank's tiles land in the column owner's receive buffer and the owners' rank-order sums equal the sum of the full
    products; with the all-reduce epilogue every rank receives every part.  (2048 columns: the 256-wide tile form.)"""
    import ctypes as C
    from qwb200.models.config import ModelConfig
    from qwb200.ops import lib as qlib, structs as S
    from qwb200.parallel import tp_channel
    L = qlib.load(True)
    dev = torch.device("cuda:0")
    R = 4
    cfg = ModelConfig.tiny(hidden=N)
    chans = tp_channel.make_emulated(cfg, R, T, dev, mtp=False)
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    P = lambda t: C.c_void_p(t.data_ptr())
    g = torch.Generator(device="cuda").manual_seed(N + K)
    A = [torch.randn(T, K, generator=g, device=dev).to(torch.bfloat16) for _ in range(R)]
    W = [(torch.randn(N, K, generator=g, device=dev) * 0.05).to(torch.bfloat16) for _ in range(R)]
    full = [a.float() @ w.float().T for a, w in zip(A, W)]
    for r in range(R):
        assert L.qwk_gemm_bf16_tc_tp(chans[r].ptr, P(A[r]), P(W[r]), None, T, N, K, K, K, N, 0, -1, 2, S.TP_RS, 0, s) == 0
    SH = N // R
    outs = [torch.zeros(T, SH, device=dev) for _ in range(R)]
    for r in range(R):
        assert L.qwk_tp_reduce(chans[r].ptr, S.TP_RS, P(outs[r]), T * SH, s) == 0
    torch.cuda.synchronize()
    want = sum(full)
    for r in range(R):
        err = float((outs[r] - want[:, r * SH:(r + 1) * SH]).abs().max() / want.abs().max())
        assert err < 2e-3, (r, err)


@pytest.fixture
def pair_form():
    """Switch the CTA-pair form of the dense kernel on for products at least 256 columns wide, and off again."""
    import ctypes as C
    from qwb200.ops import lib as qlib
    L = qlib.load(True)
    old = L.qwk_gemm_tc_pair_min_n(256)
    word = torch.zeros(2, dtype=torch.int32, device="cuda")           # bounded waits that run out report here
    L.qwk_set_error_word(C.c_void_p(word.data_ptr()))
    yield word
    torch.cuda.synchronize()
    L.qwk_set_error_word(None)
    L.qwk_gemm_tc_pair_min_n(old)


@pytest.mark.parametrize("T,N,K", [(256, 256, 64), (512, 512, 256), (4096, 2560, 640), (300, 700, 192), (1111, 1536, 128), (2048, 13952, 320)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_gemm_tc_pair_form_matches_fp32(pair_form, T, N, K, out_dtype):
    """256 x 256 tiles computed by two CTAs with tcgen05.mma.cta_group::2, ragged rows and columns included; a run whose
    barriers did not meet would end with the error word set, which is checked too."""
    from qwb200.ops import kernels as K_
    g = torch.Generator(device="cuda").manual_seed(T + N + K + 1)
    A = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    W = (torch.randn(N, K, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    ldc = (N + 7) // 8 * 8 + 8
    out = torch.full((T + 3, ldc), 768.0, dtype=out_dtype, device="cuda")      # guard columns and rows detect stray writes
    K_.gemm_bf16_tc(A, W, out=out[:T, :N])
    torch.cuda.synchronize()
    assert pair_form.tolist() == [0, 0]
    ref = A.float() @ W.float().T
    assert torch.all(out[:, N:].float() == 768.0) and torch.all(out[T:].float() == 768.0)
    tol = 2e-2 if out_dtype == torch.bfloat16 else 2e-3
    err = float((out[:T, :N].float() - ref).abs().max() / ref.abs().max())
    assert err < tol, err


def test_gemm_tc_pair_form_reduce_scatter_on_emulated_ranks(pair_form):
    test_gemm_tc_reduce_scatter_epilogue_on_emulated_ranks(1024, 2048, 256)


@pytest.mark.parametrize("T,SH,R", [(1, 32, 32), (100, 2560, 320), (129, 264, 40), (1500, 2560, 320), (300, 8, 320)])
def test_mixer_up_projection_with_the_mean_in_its_epilogue(T, SH, R):
    """Gate product, sigmoid, weighted mean over the streams in one kernel, against 64 bits (bf16 output: 2^-9, and fp32 logits) and
    with guard columns and rows."""
    import ctypes as C
    from qwb200.ops import lib as qlib
    L = qlib.load(True)
    g = torch.Generator(device="cuda").manual_seed(T + SH)
    u = torch.randn(T, R, generator=g, device="cuda").to(torch.bfloat16)
    W = (torch.randn(4 * SH, R, generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    xn = torch.randn(T, 4, SH, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((T + 2, SH + 8), 768.0, dtype=torch.bfloat16, device="cuda")
    P = lambda t: C.c_void_p(t.data_ptr())
    rc = L.qwk_gemm_mix_tc(P(u), P(W), P(xn), SH, P(out), SH + 8, T, R, R, R, C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    gate = torch.sigmoid((u.double() @ W.double().T).view(T, SH, 4).permute(0, 2, 1))
    ref = (gate * xn.double()).mean(1)
    assert torch.all(out[T:].float() == 768.0) and torch.all(out[:, SH:].float() == 768.0)
    assert float((out[:T, :SH].double() - ref).norm() / ref.norm()) < 2 ** -8


def _against_64_bits(T, N, K, out_dtype):
    """fp32 sums of exact products (1e-5 of the result's size for K <= 2560; bf16 output 2^-9 more), and nothing outside the result."""
    from qwb200.ops import kernels as K_
    g = torch.Generator(device="cuda").manual_seed(T + N + K + 2)
    A = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    W = (torch.randn(N, K, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    out = torch.full((T + 2, (N + 7) // 8 * 8 + 8), 768.0, dtype=out_dtype, device="cuda")
    K_.gemm_bf16_tc(A, W, out=out[:T, :N])
    ref = A.double() @ W.double().T
    assert torch.all(out[:, N:].float() == 768.0) and torch.all(out[T:].float() == 768.0)
    assert float((out[:T, :N].double() - ref).norm() / ref.norm()) < (1e-5 if out_dtype == torch.float32 else 2 ** -8)


@pytest.mark.parametrize("T,N,K", [(520, 12800, 2560), (640, 12700, 72), (777, 10200, 320), (300, 10190, 136)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("stage", [1, 0])
def test_gemm_tc_wide_tiles_match_64_bits(T, N, K, out_dtype, stage):
    """128 x 256 tiles, with the fp32 output through the staging buffers and straight from registers, ragged rows and columns."""
    from qwb200.ops import lib as qlib
    L = qlib.load(True)
    assert L.qwk_gemm_tc_form(T, N, K) == 1
    old = L.qwk_gemm_tc_stage_local(stage)
    try:
        _against_64_bits(T, N, K, out_dtype)
    finally:
        L.qwk_gemm_tc_stage_local(old)


@pytest.mark.parametrize("T,SH,R", [(300, 2560, 320), (3001, 2560, 320), (520, 3200, 40), (4096, 512, 64)])
def test_mixer_up_projection_of_many_tiles(T, SH, R):
    """Several tiles per block, ragged rows, and a width whose last column tile is not whole."""
    test_mixer_up_projection_with_the_mean_in_its_epilogue(T, SH, R)


@pytest.fixture
def only_pairs():
    """Every product of more than 128 rows and at least 256 columns that is not split runs in CTA pairs."""
    import ctypes as C
    from qwb200.ops import lib as qlib
    L = qlib.load(True)
    old = L.qwk_gemm_tc_pair_min_n(-256)
    word = torch.zeros(2, dtype=torch.int32, device="cuda")
    L.qwk_set_error_word(C.c_void_p(word.data_ptr()))
    yield word
    torch.cuda.synchronize()
    L.qwk_set_error_word(None)
    L.qwk_gemm_tc_pair_min_n(old)


@pytest.mark.parametrize("T,N,K", [(256, 256, 64), (512, 512, 256), (300, 700, 192), (1111, 1536, 128), (129, 300, 72), (257, 257, 320)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_gemm_tc_pairs_of_small_and_ragged_products_match_64_bits(only_pairs, T, N, K, out_dtype):
    from qwb200.ops import lib as qlib
    assert qlib.load(True).qwk_gemm_tc_form(T, N, K) == 2
    _against_64_bits(T, N, K, out_dtype)
    assert only_pairs.tolist() == [0, 0]


@pytest.mark.parametrize("T,N,K", [(1024, 2048, 256), (300, 512, 128), (129, 256, 64)])
def test_gemm_tc_pair_form_reduce_scatter_with_ragged_rows(only_pairs, T, N, K):
    test_gemm_tc_reduce_scatter_epilogue_on_emulated_ranks(T, N, K)


def test_gemm_tc_wide_form_reduce_scatter():
    from qwb200.ops import lib as qlib
    assert qlib.load(True).qwk_gemm_tc_form(520, 12800, 64) == 1
    test_gemm_tc_reduce_scatter_epilogue_on_emulated_ranks(520, 12800, 64)


@pytest.mark.parametrize("N,K", [(2560, 6144), (1793, 2560), (324, 4304), (12800, 640)])
def test_gemm_tc_rows_keep_their_bits_on_each_side_of_the_split_line(N, K):
    """Up to 256 rows, and from 257 on through single, wide and paired tiles: a row's result does not depend on the rows beside it.  Where
    few tiles are split over clusters the two sides differ by the rounding of the sum: each is within 1e-5 of 64 bits."""
    from qwb200.ops import kernels as K_, lib as qlib
    L = qlib.load(True)
    g = torch.Generator(device="cuda").manual_seed(N + K)
    A = torch.randn(4096, K, generator=g, device="cuda").to(torch.bfloat16)
    W = (torch.randn(N, K, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    whole, head = K_.gemm_bf16_tc(A, W), K_.gemm_bf16_tc(A[:256], W)
    tail = K_.gemm_bf16_tc(A[4096 - 256:], W)
    for T in (1, 33, 100, 128, 129, 200):
        assert torch.equal(K_.gemm_bf16_tc(A[:T], W), head[:T]) and torch.equal(K_.gemm_bf16_tc(A[4096 - T:], W), tail[256 - T:]), T
    for T in (257, 520, 777, 1021, 2048):
        assert torch.equal(K_.gemm_bf16_tc(A[:T], W), whole[:T]) and torch.equal(K_.gemm_bf16_tc(A[4096 - T:], W), whole[4096 - T:]), T
    if L.qwk_gemm_tc_form(256, N, K) != 3:
        assert torch.equal(head, whole[:256])
    else:
        assert float((head - whole[:256]).double().norm() / head.double().norm()) < 2e-5


@pytest.mark.parametrize("T,N,K,form", [(100, 256, 1024, 3), (300, 512, 64, 0), (520, 12800, 64, 1), (777, 4352, 64, 2)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("off", [1, 2, 4])
def test_gemm_tc_output_at_any_address(T, N, K, form, out_dtype, off):
    """Rows whose stride allows 16-byte stores but whose first element does not lie on 16 bytes: the same bits, nothing beside them."""
    from qwb200.ops import kernels as K_, lib as qlib
    assert qlib.load(True).qwk_gemm_tc_form(T, N, K) == form
    g = torch.Generator(device="cuda").manual_seed(T + off)
    A = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    W = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    flat = torch.full((T * (N + 8) + 16,), 768.0, dtype=out_dtype, device="cuda")
    out = flat[off:off + T * (N + 8)].view(T, N + 8)
    K_.gemm_bf16_tc(A, W, out=out[:, :N])
    assert torch.equal(out[:, :N], K_.gemm_bf16_tc(A, W, out_dtype=out_dtype))
    assert torch.all(out[:, N:].float() == 768.0) and torch.all(flat[:off].float() == 768.0) and torch.all(flat[off + T * (N + 8):].float() == 768.0)
