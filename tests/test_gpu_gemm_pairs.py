"""BF16 expert GEMMs on CTA pairs with the tokens as columns, and weight gradients that stop at an expert's last row."""
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


def _groups(rows, aligned):
    starts = [0]
    for n in rows:
        starts.append(starts[-1] + ((n + 127) // 128 * 128 if aligned else n))
    return starts, [starts[g] + n for g, n in enumerate(rows)]


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _close(out, ref):
    # fp32 sums of bf16 products, rounded once to bf16 (2^-9 relative of each value; the norm of the errors stays below 4e-3 of the norm)
    assert ((out.float() - ref).norm() / ref.norm().clamp(min=1e-20)).item() < 4e-3


def _check_columns(rows, K, N, sms, how, mn_major):
    from deepep_efa_b200 import _ext
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(K + N)
    starts, ends = _groups(rows, how != "ragged")
    if how == "zero_tail":  # a group of padding only
        starts, ends = starts + [starts[-1] + 128], ends + [starts[-1]]
        rows = rows + [0]
    G, M = len(rows), starts[-1]
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    if how == "zero_tail":
        for g in range(G):
            x[ends[g]:starts[g + 1]] = 0
    w = (torch.randn(G, N, K, device="cuda") * 0.1).to(torch.bfloat16)
    b = w.transpose(1, 2).contiguous() if mn_major else w
    out = torch.full((M, N), 7.0, dtype=torch.bfloat16, device="cuda")
    kw = {} if how in ("whole", "ragged") else dict(m_ends=_i32(ends), zero_tail=how == "zero_tail")
    C.grouped_gemm(x, b, _i32(starts), 0, False, None, None, out, sms, mn_major=mn_major, **kw)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    for g in range(G):
        end = starts[g + 1] if how == "whole" else ends[g]
        if end > starts[g]:
            _close(out[starts[g]:end], x[starts[g]:end].float() @ w[g].float().t())
        assert (out[end:starts[g + 1]] == (0.0 if how == "zero_tail" else 7.0)).all()
    return C.bf16_form(M, G, N, K, mn_major, bool(kw), how == "zero_tail", sms or 148)


@pytest.mark.parametrize("mn_major", [False, True])
@pytest.mark.parametrize("how", ["whole", "ragged", "masked", "zero_tail"])
@pytest.mark.parametrize("K,N,sms", [(64, 128, 0), (192, 384, 6), (512, 256, 0), (320, 1408, 0)])
def test_tokens_as_columns_on_pairs(monkeypatch, K, N, sms, how, mn_major):
    """Rows on both sides of the unit of 32, of a tile of 256 and of several equal tiles; odd counts of 128 features; empty groups."""
    monkeypatch.setenv("DEEPEP_GEMM_PAIR", "2")
    _check_columns([1, 0, 31, 32, 33, 255, 256, 257, 300, 513, 128], K, N, sms, how, mn_major)


@pytest.mark.parametrize("mn_major", [False, True])
@pytest.mark.parametrize("how", ["whole", "ragged", "masked", "zero_tail"])
@pytest.mark.parametrize("K,N,sms", [(64, 128, 2), (576, 384, 6), (1024, 256, 0), (1088, 384, 0)])
def test_tokens_as_columns_in_tiles_of_128(monkeypatch, K, N, sms, how, mn_major):
    """With up to 128 rows per group on average: rows on both sides of a unit and of a tile, K blocks fewer than, as many as and more than the eight
    stages, tiles enough on few SMs for both windows to go round. From K 1024 on this is what the product takes by itself."""
    if K < 1024:
        monkeypatch.setenv("DEEPEP_GEMM_PAIR", "2")
    else:
        monkeypatch.delenv("DEEPEP_GEMM_PAIR", raising=False)
    form = _check_columns([1, 0, 31, 0, 33, 64, 0, 65, 127, 128, 129, 257, 0, 0], K, N, sms, how, mn_major)
    assert K < 1024 or form == "columns 128"


def _launched(call):
    """Names of the kernels that a call launches."""
    from torch.profiler import ProfilerActivity, profile
    call()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
        call()
        torch.cuda.synchronize()
    names = " ".join(e.key for e in prof.key_averages())
    if "gemm_kernel" not in names:
        pytest.skip("the profiler records no kernels here")
    return names


@pytest.mark.parametrize("gradient", [False, True])
def test_forms_that_the_environment_asks_for(monkeypatch, gradient):
    """0: single CTAs, 1: pairs with tokens as rows, 2: tokens as columns; a product with a trace has the rows' forms only."""
    from deepep_efa_b200 import _ext
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(2)
    offs = _i32([0, 256, 512])
    x = torch.randn(512, 256, device="cuda").to(torch.bfloat16)
    w = (torch.randn(2, 256, 256, device="cuda") * 0.1).to(torch.bfloat16)
    ref = torch.cat([x[g * 256:(g + 1) * 256].float() @ (w[g].float() if gradient else w[g].float().t()) for g in range(2)])
    trace = torch.zeros(4, dtype=torch.int64, device="cuda")

    def run(**kw):
        return C.grouped_gemm(x, w, offs, 0, False, mn_major=gradient, **kw)

    for value, kw, kernel in (("0", {}, "grouped_gemm_kernel<256, false, false, false"), ("1", {}, "grouped_gemm_kernel<256, false, false, true"),
                              ("2", {}, "token_pairs_gemm_kernel"), (None, dict(trace=trace), "grouped_gemm_kernel<256, false, false, true")):
        monkeypatch.delenv("DEEPEP_GEMM_PAIR", raising=False)
        if value is not None:
            monkeypatch.setenv("DEEPEP_GEMM_PAIR", value)
        assert kernel in _launched(lambda: run(**kw)), (value, kw)
        _close(run(**kw), ref)
    assert C.gemm_error(0) == 0


@pytest.mark.parametrize("rows,K,N,forward,gradient", [
    ([100, 20, 128], 256, 384, "rows", "rows"),
    ([100, 20, 128], 1024, 768, "columns 128", "rows"),
    ([1, 0, 33, 128], 768, 1088, "rows", "columns 128"),
    ([300, 129, 200], 256, 384, "rows", "rows"),
    ([300, 129, 200], 1088, 1024, "columns 256", "columns 256"),
    ([500, 460, 430, 0], 256, 384, "rows", "rows"),
    ([500, 460, 430], 256, 384, "row pairs", "row pairs"),
])
def test_every_form_leaves_the_same_padding(rows, K, N, forward, gradient):
    """zero_tail on both sides of the lines between the forms: the same rows are zero, the same values are there."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import grouped_gemm, grouped_gemm_dgrad
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(5)
    starts, ends = _groups(rows, True)
    G, M = len(rows), starts[-1]
    n = N // 128 * 128  # (an output has a multiple of 128 columns, a reduction of 64)
    assert C.bf16_form(M, G, n, K, False, True, True) == forward and C.bf16_form(M, G, K // 128 * 128, N, True, True, True) == gradient
    for g_of, k, cols in (("forward", K, n), ("gradient", N, K // 128 * 128)):
        x = torch.randn(M, k, device="cuda").to(torch.bfloat16)
        for g in range(G):
            x[ends[g]:starts[g + 1]] = 0
        w = (torch.randn(G, cols, k, device="cuda") * 0.1).to(torch.bfloat16)
        y = grouped_gemm(x, w, _i32(starts), m_ends=_i32(ends), zero_tail=True) if g_of == "forward" else \
            grouped_gemm_dgrad(x, w.transpose(1, 2).contiguous(), _i32(starts), m_ends=_i32(ends))
        assert C.gemm_error(0) == 0
        for g in range(G):
            r = slice(starts[g], ends[g])
            if rows[g]:
                _close(y[r], x[r].float() @ w[g].float().t())
            assert (y[ends[g]:starts[g + 1]] == 0).all()
    with pytest.raises(ValueError):
        grouped_gemm(x, w, _i32(starts), zero_tail=True)


def test_padding_is_not_scattered():
    """Rows behind an expert's end have no destination, so zeros for them and the scatter epilogue do not go together."""
    from deepep_efa_b200 import _ext
    C = _ext.load()
    starts, ends = [0, 128, 256], [100, 256]
    x, w = torch.zeros(256, 128, device="cuda", dtype=torch.bfloat16), torch.zeros(2, 128, 128, device="cuda", dtype=torch.bfloat16)
    dst = torch.full((256, 128), 7.0, device="cuda", dtype=torch.bfloat16)
    info, bases = torch.arange(256, dtype=torch.int32, device="cuda"), torch.tensor([dst.data_ptr()], dtype=torch.int64, device="cuda")
    with pytest.raises(ValueError, match="zero_tail"):
        C.grouped_gemm(x, w, _i32(starts), 0, False, m_ends=_i32(ends), row_info=info, scatter_bases=bases, zero_tail=True)
    C.grouped_gemm(x, w, _i32(starts), 0, False, m_ends=_i32(ends), row_info=info, scatter_bases=bases)
    torch.cuda.synchronize()
    assert (dst[100:128] == 7.0).all() and (dst[:100] == 0).all() and (dst[128:] == 0).all()


@pytest.mark.parametrize("pair", ["0", "1"])
@pytest.mark.parametrize("N,K", [(128, 128), (256, 384), (384, 256)])
def test_weight_gradient_stops_at_the_last_row(monkeypatch, N, K, pair):
    """Rows that end inside every step of 16 of a K block, on its edges, and not at all; the rest of the group is zero."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import grouped_gemm_wgrad_inplace
    monkeypatch.setenv("DEEPEP_GEMM_PAIR", pair)
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(N)
    rows = [1, 0, 15, 16, 17, 47, 49, 63, 64, 65, 127, 128, 300]
    starts, ends = _groups(rows, True)
    starts, ends, rows = starts + [starts[-1] + 128], ends + [starts[-1]], rows + [0]  # (and a group of padding only)
    dy, x = (torch.randn(starts[-1], c, device="cuda").to(torch.bfloat16) for c in (N, K))
    for g in range(len(rows)):
        dy[ends[g]:starts[g + 1]] = x[ends[g]:starts[g + 1]] = 0
    dw = grouped_gemm_wgrad_inplace(dy, x, _i32(starts), m_ends=_i32(ends))
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    for g, n in enumerate(rows):
        r = slice(starts[g], ends[g])
        if n == 0:
            assert (dw[g] == 0).all()
        else:
            _close(dw[g], dy[r].float().t() @ x[r].float())


@pytest.mark.parametrize("pair", ["0", "1"])
@pytest.mark.parametrize("N,K", [(128, 128), (256, 384)])
def test_outputs_that_start_between_sectors_equal_aligned_ones(monkeypatch, N, K, pair):
    """Rows leave in pieces of 32 bytes where the output starts on such a boundary, and through a staging buffer elsewhere. Odd numbers of rows: the
    last row of a pair of lanes is not there."""
    from deepep_efa_b200 import _ext
    monkeypatch.setenv("DEEPEP_GEMM_PAIR", pair)
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(N + K)

    def outputs(shape):
        n = shape[0] * shape[1] * (shape[2] if len(shape) == 3 else 1)
        for shift in (0, 8):
            flat = torch.full((n + 32,), 7.0, device="cuda", dtype=torch.bfloat16)
            yield flat, flat[shift:shift + n].view(shape), shift

    rows = [1, 31, 33, 0, 129, 2]
    starts, _ = _groups(rows, False)
    x, w = (torch.randn(s, device="cuda").to(torch.bfloat16) for s in ((starts[-1], K), (len(rows), N, K)))
    forward = []
    for flat, out, shift in outputs((starts[-1], N)):
        C.grouped_gemm(x, w, _i32(starts), 0, False, None, None, out)
        assert (flat[:shift] == 7.0).all() and (flat[shift + out.numel():] == 7.0).all()
        forward.append(out)
    starts, _ = _groups([70, 0, 1, 128], True)
    dy, h = (torch.randn(starts[-1], c, device="cuda").to(torch.bfloat16) for c in (N, K))
    grads = []
    for flat, out, shift in outputs((4, N, K)):
        C.grouped_gemm(dy, h, _i32(starts), 1, False, None, None, out, mn_major=True)
        assert (flat[:shift] == 7.0).all() and (flat[shift + out.numel():] == 7.0).all()
        grads.append(out)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    assert torch.equal(*forward) and torch.equal(*grads)
    for g in range(4):
        r = slice(starts[g], starts[g + 1])
        if starts[g + 1] > starts[g]:
            _close(grads[0][g], dy[r].float().t() @ h[r].float())
        else:
            assert (grads[0][g] == 0).all()


def test_ends_of_weight_gradients_need_operands_in_place():
    from deepep_efa_b200 import _ext
    C = _ext.load()
    a = torch.zeros(128, 256, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="m_ends"):
        C.grouped_gemm(a, a, _i32([0, 128, 256]), 1, False, m_ends=_i32([100, 256]))


@pytest.mark.parametrize("swiglu,K,N,masked", [(True, 1152, 512, False), (False, 1280, 512, False), (True, 128, 256, True), (True, 640, 768, True),
                                               (False, 512, 256, True), (False, 1280, 512, True)])
def test_promotion_with_256_columns_equals_128(swiglu, K, N, masked):
    """FP8 with fp32 scales: few SMs make the wide tiles the better choice, all of them the narrow ones. Both add the K blocks in the same order
    with the same fused multiply-adds, so the results are the same bit for bit; rows on both sides of a warp's 32 and of a tile's 128."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import reference_grouped_gemm
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(N)
    rows = [1, 31, 33, 0, 127, 128, 129, 200]
    starts, ends = _groups(rows, True)
    G, M = len(rows), starts[-1]
    a = torch.randn(M, K, device="cuda").to(torch.float8_e4m3fn)
    b = torch.randn(G, N, K, device="cuda").to(torch.float8_e4m3fn)
    a_s, b_s = torch.rand(M, K // 128, device="cuda") + 0.1, torch.rand(G, N // 128, K // 128, device="cuda") * 0.1
    kw = dict(m_ends=_i32(ends), rows_hint=sum(rows)) if masked else {}
    assert [C.promotion_columns(M, G, N, K, swiglu, masked, kw.get("rows_hint", 0), sms) for sms in (1, 148)] == [256, 128]
    width = N // 2 if swiglu else N
    outs = []
    for sms in (1, 3, 0):
        out = torch.full((M, width), 7.0, dtype=torch.bfloat16, device="cuda")
        outs.append(C.grouped_gemm(a, b, _i32(starts), 0, swiglu, a_s, b_s, out, sms, **kw))
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1], outs[2])
    ref = reference_grouped_gemm(a, b, _i32(starts), swiglu=swiglu, a_scales=a_s, b_scales=b_s)
    for g in range(G):
        if rows[g]:
            # exact products of e4m3 values, fp32 sums and scales, one rounding to bf16
            _close(outs[0][starts[g]:ends[g]], ref[starts[g]:ends[g]])
        if masked:
            assert (outs[0][ends[g]:starts[g + 1]] == 7.0).all()


@pytest.mark.parametrize("N", [256, 768])
def test_promotion_with_256_columns_scatters_rows(N):
    from deepep_efa_b200 import _ext
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(3)
    rows, K = [40, 130, 0, 65], 512
    starts, ends = _groups(rows, True)
    M, valid = starts[-1], sum(rows)
    a = torch.randn(M, K, device="cuda").to(torch.float8_e4m3fn)
    b = torch.randn(len(rows), N, K, device="cuda").to(torch.float8_e4m3fn)
    a_s, b_s = torch.rand(M, K // 128, device="cuda") + 0.1, torch.rand(len(rows), N // 128, K // 128, device="cuda") * 0.1
    where, order = torch.full((M,), -1, dtype=torch.int32), torch.randperm(valid)
    at = torch.cat([torch.arange(starts[g], ends[g]) for g in range(len(rows))])
    where[at] = order.to(torch.int32)
    where[at[::7]] = -1  # dropped rows
    dst = torch.full((valid, N), 7.0, dtype=torch.bfloat16, device="cuda")
    bases = torch.tensor([dst.data_ptr()], dtype=torch.int64, device="cuda")
    plain = C.grouped_gemm(a, b, _i32(starts), 0, False, a_s, b_s)
    assert C.promotion_columns(M, len(rows), N, K, False, True, valid, 2) == 256
    C.grouped_gemm(a, b, _i32(starts), 0, False, a_s, b_s, None, 2, 2000.0, _i32(ends), row_info=where.cuda(), scatter_bases=bases, rows_hint=valid)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    want = torch.full_like(dst, 7.0)
    keep = where[at] >= 0
    want[where[at][keep].long().cuda()] = plain[at[keep].cuda()]
    assert torch.equal(dst, want)


@pytest.mark.parametrize("swiglu,N,K", [(True, 512, 384), (False, 256, 128)])
def test_promotion_with_256_columns_between_sectors(swiglu, N, K):
    """Outputs that start on a multiple of 16 bytes only are stored by other instructions, with the same values."""
    from deepep_efa_b200 import _ext
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(K)
    rows = [1, 0, 31, 129]
    starts, ends = _groups(rows, True)
    G, M, width = len(rows), starts[-1], N // 2 if swiglu else N
    a, b = torch.randn(M, K, device="cuda").to(torch.float8_e4m3fn), torch.randn(G, N, K, device="cuda").to(torch.float8_e4m3fn)
    a_s, b_s = torch.rand(M, K // 128, device="cuda") + 0.1, torch.rand(G, N // 128, K // 128, device="cuda") * 0.1
    assert C.promotion_columns(M, G, N, K, swiglu, True, sum(rows), 1) == 256
    outs = []
    for shift in (0, 8):
        flat = torch.full((M * width + 16,), 7.0, dtype=torch.bfloat16, device="cuda")
        out = flat[shift:shift + M * width].view(M, width)
        C.grouped_gemm(a, b, _i32(starts), 0, swiglu, a_s, b_s, out, 1, m_ends=_i32(ends), rows_hint=sum(rows))
        assert (flat[:shift] == 7.0).all() and (flat[shift + M * width:] == 7.0).all()
        outs.append(out)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    assert torch.equal(*outs)
    for g in range(G):
        assert (outs[0][ends[g]:starts[g + 1]] == 7.0).all()


@pytest.mark.parametrize("sms", [1, 148])  # tiles of 256 columns, which quantise their own output, and of 128 with a cast behind
@pytest.mark.parametrize("counts", [False, True])
def test_promotion_writes_quantised_output(sms, counts):
    """The same e4m3 rows and scales, byte for byte, as a cast of the BF16 output; nothing behind a group's last row where the tiles write them."""
    from deepep_efa_b200 import _ext
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(sms)
    rows, K, inter = [1, 0, 31, 33, 128, 97], 384, 256
    starts = list(range(0, 128 * len(rows) + 1, 128))
    G, M = len(rows), starts[-1]
    a, b = torch.randn(M, K, device="cuda").to(torch.float8_e4m3fn), torch.randn(G, 2 * inter, K, device="cuda").to(torch.float8_e4m3fn)
    a_s, b_s = torch.rand(M, K // 128, device="cuda") * 0.02, torch.rand(G, 2 * inter // 128, K // 128, device="cuda") * 0.1
    a.view(torch.uint8)[128 * 3 + 2] = 0  # a row of zeros: the smallest scale
    assert C.promotion_columns(M, G, 2 * inter, K, True, True, sum(rows), sms) == (256 if sms == 1 else 128)
    how = dict(m_ends=_i32(rows if counts else [s + n for s, n in zip(starts, rows)]), m_ends_are_counts=counts, rows_hint=sum(rows))
    plain = torch.zeros(M, inter, device="cuda", dtype=torch.bfloat16)
    C.grouped_gemm(a, b, _i32(starts), 0, True, a_s, b_s, plain, sms, **how)
    want_q, want_s = C.per_token_cast_to_fp8(plain, False, False)
    q, s = torch.full((M, inter), 7, device="cuda", dtype=torch.uint8), torch.full((M, inter // 128), 7.0, device="cuda")
    C.grouped_gemm(a, b, _i32(starts), 0, True, a_s, b_s, torch.zeros_like(plain), sms, out_fp8=q.view(torch.float8_e4m3fn), out_scales=s, **how)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    for g, n in enumerate(rows):
        r = slice(starts[g], starts[g] + n)
        assert torch.equal(q[r], want_q.view(torch.uint8)[r]) and torch.equal(s[r], want_s[r])
        if sms == 1:
            assert (q[starts[g] + n:starts[g + 1]] == 7).all() and (s[starts[g] + n:starts[g + 1]] == 7).all()


@pytest.mark.parametrize("H", [128, 1408, 4096, 7168])
@pytest.mark.parametrize("atoms", [False, True])
def test_gather_of_quantised_rows(H, atoms):
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import build_sf_atoms_a
    from deepep_efa_b200.ops.permute import gather_rows
    C = _ext.load()
    torch.manual_seed(H)
    N, M = 77, 384
    rows = torch.randint(0, 255, (N, H), device="cuda", dtype=torch.uint8).view(torch.float8_e4m3fn)
    scales = torch.exp2(torch.randint(-20, 20, (N, H // 128), device="cuda").float()) if atoms else torch.rand(N, H // 128, device="cuda")
    src = torch.randint(-1, N, (M,), device="cuda", dtype=torch.int32)
    sched = torch.full((2,), 9, device="cuda", dtype=torch.int32)
    got, got_s = C.gather_quantised(rows, scales, src, atoms, sched)
    want_s = gather_rows(scales, src)
    assert torch.equal(got.view(torch.uint8), gather_rows(rows, src).view(torch.uint8)) and sched.tolist() == [0, 0]
    assert torch.equal(got_s, build_sf_atoms_a(want_s) if atoms else want_s)
    assert C.gather_quantised(rows, scales, src[:0], atoms)[0].shape == (0, H)
