"""Grouped tcgen05 GEMM against a plain PyTorch fp32 reference of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _offsets(rows, device="cuda"):
    o = [0]
    for r in rows:
        o.append(o[-1] + r)
    return torch.tensor(o, dtype=torch.int32, device=device)


def _rel_err(x, ref):
    return ((x.float() - ref).norm() / ref.norm().clamp(min=1e-12)).item()


@pytest.mark.parametrize("rows,K,N", [([128], 64, 128), ([128, 256, 0, 384], 512, 256), ([256, 128], 1024, 384), ([128] * 5, 192, 512)])
def test_bf16_mgrouped(rows, K, N):
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import grouped_gemm, reference_grouped_gemm
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(0)
    G, M = len(rows), sum(rows)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = (torch.randn(G, N, K, device="cuda") * 0.1).to(torch.bfloat16)
    offs = _offsets(rows)
    c = grouped_gemm(a, b, offs)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    ref = reference_grouped_gemm(a, b, offs)
    assert _rel_err(c, ref) < 1e-2, _rel_err(c, ref)
    # a second launch on a smaller persistent grid walks several tiles per CTA
    c2 = grouped_gemm(a, b, offs, num_sms=3)
    assert torch.equal(c, c2)


def test_unaligned_and_masked_groups():
    """Group boundaries anywhere, and m_ends: only the first rows of every group are computed, the rest stay untouched."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import grouped_gemm, reference_grouped_gemm
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(5)
    rows, K, N = [40, 200, 0, 77, 3], 256, 256
    G, M = len(rows), sum(rows)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = (torch.randn(G, N, K, device="cuda") * 0.1).to(torch.bfloat16)
    offs = _offsets(rows)
    c = grouped_gemm(a, b, offs)
    ref = reference_grouped_gemm(a, b, offs)
    assert _rel_err(c, ref) < 1e-2, _rel_err(c, ref)
    # masked: fixed stride 64 per group (tiles of 128 rows overlap the next group), counts 0..64
    stride, counts = 64, [64, 0, 17, 33, 1]
    starts = torch.arange(G + 1, device="cuda", dtype=torch.int32) * stride
    ends = starts[:G] + torch.tensor(counts, device="cuda", dtype=torch.int32)
    a = torch.randn(G * stride, K, device="cuda").to(torch.bfloat16)
    out = torch.full((G * stride, N), 7.0, device="cuda", dtype=torch.bfloat16)
    grouped_gemm(a, b, starts, out=out, m_ends=ends)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    full = reference_grouped_gemm(a, b, starts)
    for g, n in enumerate(counts):
        lo = g * stride
        if n:
            assert _rel_err(out[lo:lo + n], full[lo:lo + n]) < 1e-2
        assert (out[lo + n:lo + stride] == 7.0).all()
    sw = torch.full((G * stride, N // 2), 7.0, device="cuda", dtype=torch.bfloat16)
    grouped_gemm(a, b, starts, swiglu=True, out=sw, m_ends=ends)
    fsw = reference_grouped_gemm(a, b, starts, swiglu=True)
    for g, n in enumerate(counts):
        lo = g * stride
        if n:
            assert _rel_err(sw[lo:lo + n], fsw[lo:lo + n]) < 1.5e-2
        assert (sw[lo + n:lo + stride] == 7.0).all()


@pytest.mark.parametrize("rows,K,I", [([128, 256], 256, 128), ([128, 128, 384], 512, 192)])
def test_bf16_swiglu(rows, K, I):
    from deepep_efa_b200.ops.grouped_gemm import grouped_gemm, reference_grouped_gemm
    torch.manual_seed(1)
    G, M = len(rows), sum(rows)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = (torch.randn(G, 2 * I, K, device="cuda") * 0.1).to(torch.bfloat16)
    offs = _offsets(rows)
    c = grouped_gemm(a, b, offs, swiglu=True)
    assert c.shape == (M, I)
    ref = reference_grouped_gemm(a, b, offs, swiglu=True)
    assert _rel_err(c, ref) < 1.5e-2, _rel_err(c, ref)


@pytest.mark.parametrize("swiglu", [False, True])
def test_fp8_blockscaled(swiglu):
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import grouped_gemm, reference_grouped_gemm
    from deepep_efa_b200.reference import oracle
    C = _ext.load()
    torch.manual_seed(2)
    rows, K, N = [128, 256, 128], 512, 256
    G, M = len(rows), sum(rows)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    a, a_s = C.per_token_cast_to_fp8(x, False, False)
    w = torch.randn(G, N, K, device="cuda") * 0.05
    wb = w.view(G, N // 128, 128, K // 128, 128)
    b_s = (wb.abs().amax(dim=(2, 4)).clamp(min=1e-4) / 448.0).contiguous()
    b = (wb / b_s.view(G, N // 128, 1, K // 128, 1)).view(G, N, K).to(torch.float8_e4m3fn)
    offs = _offsets(rows)
    c = grouped_gemm(a, b, offs, swiglu=swiglu, a_scales=a_s, b_scales=b_s)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    ref = reference_grouped_gemm(a, b, offs, swiglu=swiglu, a_scales=a_s, b_scales=b_s)
    assert _rel_err(c, ref) < 1e-2, _rel_err(c, ref)


def test_bf16_wgrad_kgrouped():
    from deepep_efa_b200.ops.grouped_gemm import grouped_gemm_wgrad
    torch.manual_seed(3)
    rows, n_out, k_out = [128, 0, 256], 256, 128
    M = sum(rows)
    dy = torch.randn(M, n_out, device="cuda").to(torch.bfloat16)
    x = torch.randn(M, k_out, device="cuda").to(torch.bfloat16)
    offs = _offsets(rows)
    dw = grouped_gemm_wgrad(dy.t().contiguous(), x.t().contiguous(), offs)
    assert dw.shape == (3, n_out, k_out)
    o = offs.tolist()
    for g in range(3):
        ref = dy[o[g]:o[g + 1]].float().t() @ x[o[g]:o[g + 1]].float()
        if rows[g] == 0:
            assert dw[g].float().abs().max().item() == 0
        else:
            assert _rel_err(dw[g], ref) < 1e-2


@pytest.mark.parametrize("shape", [(64, 64), (200, 72), (3, 136, 4096), (2, 1408, 264)])
def test_transpose_kernel(shape):
    from deepep_efa_b200.ops.grouped_gemm import transpose_last2
    torch.manual_seed(7)
    x = torch.randn(*shape, device="cuda").to(torch.bfloat16)
    assert torch.equal(transpose_last2(x), x.transpose(-1, -2).contiguous())


def test_swiglu_kernels_match_autograd():
    from deepep_efa_b200.ops.grouped_gemm import swiglu
    torch.manual_seed(8)
    M, I = 300, 1408
    h13 = torch.randn(M, 2 * I, device="cuda").to(torch.bfloat16).requires_grad_(True)
    dh = torch.randn(M, I, device="cuda").to(torch.bfloat16)
    h = swiglu(h13)
    h.backward(dh)
    ref_in = h13.detach().float().requires_grad_(True)
    ref = torch.nn.functional.silu(ref_in[:, :I]) * ref_in[:, I:]
    ref.backward(dh.float())
    assert _rel_err(h, ref.detach()) < 4e-3
    assert _rel_err(h13.grad, ref_in.grad) < 4e-3


def test_swiglu_of_zeros_infinities_and_the_far_ends():
    """Gates whose quotient x / (1 + e^-x) is a zero of either sign, infinite, not a number, or has a denominator near the end of the range."""
    from deepep_efa_b200.ops import grouped_gemm as gg
    inf, nan = float("inf"), float("nan")
    gates = [0.0, -0.0, inf, -inf, nan, 88.0, -87.0, -88.0, -89.0, -100.0, 3e38, -3e38, 1e-30, -1e-30, 20.0, -20.0]
    gate = torch.tensor([gates, [g / 8 for g in gates]], device="cuda").to(torch.bfloat16)
    h13 = torch.cat([gate, torch.ones_like(gate)], dim=1).requires_grad_(True)
    h = gg.swiglu(h13)
    h.backward(torch.ones_like(h))
    x = gate.double()
    sig = 1 / (1 + torch.exp(-x))
    want = torch.where(x == -inf, nan, x * sig)  # (-inf * 0)
    finite = torch.isfinite(x)

    def close(out, ref):
        # fp32 values with a few units of error, rounded to BF16 (2^-9); below 2^-126 only the magnitude counts
        assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-36).all()

    h = h.detach()
    close(h[finite], want[finite])
    close(h13.grad[:, 16:][finite], want[finite])
    close(h13.grad[:, :16][finite], (sig * (1 + x * (1 - sig)))[finite])
    assert torch.equal(torch.isnan(h), torch.isnan(want)) and torch.equal(torch.isinf(h), torch.isinf(want))
    assert torch.equal(torch.signbit(h[:, :2]), torch.signbit(gate[:, :2]))


@pytest.mark.parametrize("which", ["normal", "uniform", "wide", "tiny"])
def test_logistic_in_fp32_like_the_division(which):
    """The epilogues' silu and sigmoid, before they are rounded to BF16, against a division of the same fp32 denominator and against 64 bits. An estimate of 2^-23
    and one residual step leave 2^-44 in front of the last rounding, so all but one in 2^19 quotients are the division's and no other is further off than its
    neighbour; without the step every third would be. Numerators next to zero have the denominator 2 and come out exactly."""
    from deepep_efa_b200 import _ext
    n = 3_000_000
    gen = torch.Generator(device="cuda").manual_seed(7)
    if which == "normal":
        x = torch.randn(n, generator=gen, device="cuda")
    elif which == "uniform":
        x = torch.rand(n, generator=gen, device="cuda") * 40 - 20
    elif which == "wide":
        x = torch.rand(n, generator=gen, device="cuda") * 178 - 89
    else:  # all subnormal magnitudes' places, and from there to 2^-100
        bits = torch.randint(0, 27 << 23, (n,), generator=gen, device="cuda", dtype=torch.int32)
        x = bits.view(torch.float32) * torch.where(torch.rand(n, generator=gen, device="cuda") < 0.5, -1.0, 1.0)
    got = _ext.load().logistic(x)
    sig = torch.sigmoid(x.double())
    for ours, plain, exact in ((got[0], got[1], x.double() * sig), (got[2], got[3], sig)):
        places = (ours.view(torch.int32) - plain.view(torch.int32)).abs()
        assert places.max() <= 1 and (places != 0).double().mean() <= 2.0 ** -17
        if which == "tiny":
            assert (places == 0).all()
        elif which != "wide":
            off, off_plain = ((v.double() / exact - 1).abs() * 2 ** 24 for v in (ours, plain))
            print(which, [(float(o.square().mean().sqrt()), float(o.max())) for o in (off, off_plain)])
            assert off.square().mean() <= 1.0001 * off_plain.square().mean() and off.max() <= off_plain.max() + 2


@pytest.mark.parametrize("swiglu", [False, True])
def test_wide_promotion_has_its_registers(swiglu):
    """In this build the choice is free to take tiles of 256 columns."""
    from deepep_efa_b200 import _ext
    assert _ext.load().wide_promotion_fits(swiglu)


def test_rowdot_kernel():
    from deepep_efa_b200 import _ext
    torch.manual_seed(9)
    Mp, N, K, H = 500, 120, 6, 4096
    a = torch.randn(Mp, H, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, H, device="cuda").to(torch.bfloat16)
    pos = torch.randint(-1, Mp, (N, K), device="cuda", dtype=torch.int32)
    got = _ext.load().rowdot(a, b, pos)
    want = torch.where(pos >= 0, (a[pos.clamp(min=0).long()].float() * b.float().unsqueeze(1)).sum(-1), torch.zeros(N, K, device="cuda"))
    assert torch.allclose(got, want, rtol=1e-3, atol=1e-2)


@pytest.mark.parametrize("N,K,H,pad", [(1, 1, 8, 0), (37, 6, 1032, 5), (120, 8, 4096, 77)])
def test_unpermute_backward_kernel(N, K, H, pad):
    """Row gradients bit for bit (one product, rounded once), weight gradients against fp32 sums, padding rows cleared."""
    from deepep_efa_b200 import _ext
    torch.manual_seed(10)
    M = N * K + pad
    keep = torch.rand(N, K, device="cuda") < 0.8
    pos = torch.where(keep, torch.randperm(M, device="cuda")[:N * K].view(N, K), torch.full((N, K), -1, device="cuda")).int()
    src_row = torch.full((M,), -1, device="cuda", dtype=torch.int32)
    n_of = torch.arange(N, device="cuda").unsqueeze(1).expand(N, K)
    src_row[pos[keep].long()] = n_of[keep].int()
    a, g = (torch.randn(r, H, device="cuda").to(torch.bfloat16) for r in (M, N))
    w = torch.rand(N, K, device="cuda")
    da, dw = _ext.load().unpermute_bwd(a, g, w, pos, src_row)
    want = torch.zeros(M, H, device="cuda", dtype=torch.bfloat16)
    want[pos[keep].long()] = (w[keep].unsqueeze(1) * g[n_of[keep]].float()).to(torch.bfloat16)
    assert torch.equal(da, want)
    dot = torch.where(keep, (a[pos.clamp(min=0).long()].double() * g.double().unsqueeze(1)).sum(-1), torch.zeros(N, K, device="cuda", dtype=torch.double))
    # fp32 sum of H products of unit variance: error well below H * 2^-24 * max |partial sum|
    assert (dw.double() - dot).abs().max().item() < 1e-3


@pytest.mark.parametrize("swiglu,wide", [(False, True), (False, False), (True, True), (True, False)])
def test_fp8_native_block_scaling(swiglu, wide):
    """tcgen05 block-scaled MMA with UE8M0 scale atoms against the dequantised fp32 reference; the row scales differ by
    powers of two from row to row so that a wrong row-to-scale mapping cannot pass."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import build_sf_atoms_a, build_sf_atoms_b, grouped_gemm, reference_grouped_gemm
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(11)
    rows, K = [128, 256, 0, 384], 512
    N = 512
    G, M = len(rows), sum(rows)
    x = torch.randn(M, K, device="cuda") * torch.pow(2.0, (torch.arange(M, device="cuda") % 7).float()).unsqueeze(1)
    x = x * torch.pow(2.0, (torch.arange(K, device="cuda") // 128 % 3).float()).unsqueeze(0)
    a, a_s = C.per_token_cast_to_fp8(x.to(torch.bfloat16), True, False)  # power-of-two scales
    w = torch.randn(G, N, K, device="cuda") * 0.1 * torch.pow(2.0, (torch.arange(N, device="cuda") // 128 % 4).float()).view(1, N, 1)
    wb = w.view(G, N // 128, 128, K // 128, 128)
    b_s = torch.exp2(torch.ceil(torch.log2(wb.abs().amax(dim=(2, 4)).clamp(min=1e-4) / 448.0))).contiguous()
    b = (wb / b_s.view(G, N // 128, 1, K // 128, 1)).view(G, N, K).to(torch.float8_e4m3fn).contiguous()
    offs = _offsets(rows)
    c = grouped_gemm(a, b, offs, swiglu=swiglu, sfa_atoms=build_sf_atoms_a(a_s), sfb_atoms=build_sf_atoms_b(b_s, N, swiglu, wide))
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    ref = reference_grouped_gemm(a, b, offs, swiglu=swiglu, a_scales=a_s, b_scales=b_s)
    assert _rel_err(c, ref) < (1.5e-2 if swiglu else 1e-2), _rel_err(c, ref)


@pytest.mark.parametrize("rows,N_w,K_w", [([128, 256, 0, 384], 256, 512), ([40, 200, 77], 384, 128), ([256] * 3, 1408, 4096)])
def test_bf16_dgrad_reads_weight_in_place(rows, N_w, K_w):
    """dx = grad @ w[g] with the forward weight [G, N, K] consumed as an MN-major operand: no transposed copy."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import grouped_gemm_dgrad
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(11)
    G, M = len(rows), sum(rows)
    grad = torch.randn(M, N_w, device="cuda").to(torch.bfloat16)
    w = (torch.randn(G, N_w, K_w, device="cuda") * 0.1).to(torch.bfloat16)
    offs = _offsets(rows)
    dx = grouped_gemm_dgrad(grad, w, offs)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0 and dx.shape == (M, K_w)
    o = offs.tolist()
    for g in range(G):
        if rows[g]:
            ref = grad[o[g]:o[g + 1]].float() @ w[g].float()
            assert _rel_err(dx[o[g]:o[g + 1]], ref) < 1e-2, (g, _rel_err(dx[o[g]:o[g + 1]], ref))


@pytest.mark.parametrize("rows,n_out,k_out", [([128, 0, 256], 256, 128), ([64, 192, 128], 384, 256), ([512, 256], 1408, 4096)])
def test_bf16_wgrad_reads_gradient_and_activation_in_place(rows, n_out, k_out):
    """dw[g] = grad[rows of g].T @ x[rows of g] with both operands MN-major: no transposed copies."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import grouped_gemm_wgrad_inplace
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(12)
    M = sum(rows)
    dy = torch.randn(M, n_out, device="cuda").to(torch.bfloat16)
    x = torch.randn(M, k_out, device="cuda").to(torch.bfloat16)
    offs = _offsets(rows)
    dw = grouped_gemm_wgrad_inplace(dy, x, offs)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0 and dw.shape == (len(rows), n_out, k_out)
    o = offs.tolist()
    for g in range(len(rows)):
        ref = dy[o[g]:o[g + 1]].float().t() @ x[o[g]:o[g + 1]].float()
        if rows[g] == 0:
            assert dw[g].float().abs().max().item() == 0
        else:
            assert _rel_err(dw[g], ref) < 1e-2, (g, _rel_err(dw[g], ref))


@pytest.mark.parametrize("kind", ["bf16", "fp32_scales", "mx_narrow", "mx_wide", "mx_wide_swiglu"])
def test_partial_tiles_and_drawn_tiles(kind):
    """Masked groups whose last tile is cut at and around multiples of 32 rows, after full tiles, with NaN bytes in the rows that do
    not count; tiles drawn from a counter, which comes back zero, must give the same as tiles dealt out in strides."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import build_sf_atoms_a, build_sf_atoms_b, reference_grouped_gemm
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(17)
    counts, stride, K, N = [1, 31, 256, 32, 0, 33, 160, 64, 65, 129, 128, 161, 97, 96, 200], 256, 512, 512
    G, swiglu = len(counts), kind == "mx_wide_swiglu"
    cnt = torch.tensor(counts, device="cuda", dtype=torch.int32)
    starts = torch.arange(G + 1, device="cuda", dtype=torch.int32) * stride
    live = (torch.arange(stride, device="cuda").unsqueeze(0) < cnt.unsqueeze(1)).view(-1)
    x = torch.randn(G * stride, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(G, N, K, device="cuda") * 0.1).to(torch.bfloat16)
    a_s = b_s = sfa = sfb = None
    if kind == "bf16":
        a, b = x.clone(), w
    else:
        a, a_s = C.per_token_cast_to_fp8(x, kind != "fp32_scales", False)
        b_s = torch.full((G, N // 128, K // 128), 2.0 ** -9, device="cuda")
        b = (w.float() / 2.0 ** -9).to(torch.float8_e4m3fn)
        if kind.startswith("mx"):
            sfa, sfb = build_sf_atoms_a(a_s), build_sf_atoms_b(b_s, N, swiglu, kind != "mx_narrow")
    ref = reference_grouped_gemm(a, b, starts, swiglu=swiglu, a_scales=a_s, b_scales=b_s)
    a.view(torch.uint8)[~live] = 0xFF  # NaN in both types
    outs = []
    for sched in (None, torch.zeros(2, dtype=torch.int32, device="cuda")):
        for sms, columns in ((0, False), (2, False), (0, True), (2, True)):
            out = torch.full((G * stride, N // 2 if swiglu else N), 7.0, device="cuda", dtype=torch.bfloat16)
            scales = (None, None) if sfa is not None else (a_s, b_s)
            C.grouped_gemm(a, b, starts, 0, swiglu, *scales, out, sms, 2000.0, cnt, sfa, sfb, m_ends_are_counts=True, sched=sched, tokens_as_columns=columns)
            outs.append(out)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0 and sched.tolist() == [0, 0]
    assert _rel_err(outs[0][live], ref[live]) < (1.5e-2 if swiglu else 1e-2)
    assert (outs[0][~live] == 7.0).all()
    assert all(torch.equal(o, outs[0]) for o in outs)


def test_quantised_output_with_tokens_as_columns():
    """The kernel that takes the weights as M quantises like the row-wise one, bit for bit."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import build_sf_atoms_a, build_sf_atoms_b
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(19)
    counts, stride, K, I = [1, 15, 16, 17, 31, 32, 33, 0, 64, 65, 96, 97, 128, 129, 256, 200], 256, 384, 384
    G = len(counts)
    cnt = torch.tensor(counts, device="cuda", dtype=torch.int32)
    starts = torch.arange(G + 1, device="cuda", dtype=torch.int32) * stride
    live = (torch.arange(stride, device="cuda").unsqueeze(0) < cnt.unsqueeze(1)).view(-1)
    x = torch.randn(G * stride, K, device="cuda").to(torch.bfloat16)
    x[starts[4]:starts[5]] = 0  # a group whose maxima are all zero
    a, a_s = C.per_token_cast_to_fp8(x, True, False)
    b = torch.randn(G, 2 * I, K, device="cuda").to(torch.float8_e4m3fn)
    b_s = torch.exp2(torch.randint(-8, -4, (G, 2 * I // 128, K // 128), device="cuda").float())
    sfa, sfb = build_sf_atoms_a(a_s), build_sf_atoms_b(b_s, 2 * I, True, True)
    got = []
    for columns in (True, False):
        q = torch.zeros(G * stride, I, dtype=torch.uint8, device="cuda")
        atoms = torch.zeros(G * stride // 128, I // 128, 512, dtype=torch.uint8, device="cuda")
        C.grouped_gemm(a, b, starts, 0, True, None, None, None, 0, 2000.0, cnt, sfa, sfb, out_fp8=q.view(torch.float8_e4m3fn), out_atoms=atoms,
                       m_ends_are_counts=True, tokens_as_columns=columns)
        got.append((q, atoms))
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert (got[0][0][~live] == 0).all() and got[0][0][live].any()


@pytest.mark.parametrize("cap", [64, 128, 160, 192, 224])
@pytest.mark.parametrize("scatter", [False, True])
def test_token_columns_tile_sizes(cap, scatter):
    """Groups at and around every cut of the tiles that take tokens as columns, K blocks fewer than, as many as and more than the ring's
    stages: bit for bit the rows form, rows that do not count left alone, rows scattered to where their words say."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import build_sf_atoms_a, build_sf_atoms_b
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(cap)
    step = 64 if cap < 128 else 128 if cap < 192 else 192
    counts = [1, 0, 16, 17, step - 1, step, step + 1, cap - 16, cap - 15, cap, cap + 1, cap + 15, cap + 16, step + cap, step + cap + 1, 384, 385, 448]
    G, stride, I = len(counts), 512, 256
    cnt = torch.tensor(counts, device="cuda", dtype=torch.int32)
    starts = torch.arange(G + 1, device="cuda", dtype=torch.int32) * stride
    live = (torch.arange(stride, device="cuda").unsqueeze(0) < cnt.unsqueeze(1)).view(-1)
    for K in (128, 512, 1152):
        a, a_s = C.per_token_cast_to_fp8(torch.randn(G * stride, K, device="cuda").to(torch.bfloat16), True, False)
        a_s = a_s * torch.exp2(torch.randint(-3, 4, a_s.shape, device="cuda").float())  # another factor in every row and K block
        sfa = build_sf_atoms_a(a_s)
        a.view(torch.uint8)[~live] = 0xFF
        b = torch.randn(G, 2 * I, K, device="cuda").to(torch.float8_e4m3fn)
        b_s = torch.exp2(torch.randint(-8, -4, (G, 2 * I // 128, K // 128), device="cuda").float())
        info = torch.full((G * stride,), -1, dtype=torch.int32, device="cuda")
        info[live] = torch.randperm(sum(counts), device="cuda").int()
        got = []
        for columns in (cap, 0):
            how = dict(m_ends_are_counts=True, tokens_as_columns=columns)
            q = torch.zeros(G * stride, I, dtype=torch.uint8, device="cuda")
            atoms = torch.zeros(G * stride // 128, I // 128, 512, dtype=torch.uint8, device="cuda")
            if not scatter:
                C.grouped_gemm(a, b, starts, 0, True, None, None, None, 0, 2000.0, cnt, sfa, build_sf_atoms_b(b_s, 2 * I, True, True),
                               out_fp8=q.view(torch.float8_e4m3fn), out_atoms=atoms, **how)
            out = torch.full((sum(counts) if scatter else G * stride, 2 * I), 7.0, device="cuda", dtype=torch.bfloat16)
            extra = dict(row_info=info, scatter_bases=torch.tensor([out.data_ptr()], dtype=torch.int64, device="cuda")) if scatter else {}
            C.grouped_gemm(a, b, starts, 0, False, None, None, None if scatter else out, 3, 2000.0, cnt, sfa, build_sf_atoms_b(b_s, 2 * I, False, True),
                           **how, **extra)
            torch.cuda.synchronize()
            got.append((q, atoms, out))
        assert C.gemm_error(0) == 0
        assert all(torch.equal(x, y) for x, y in zip(*got))
        out = got[0][2]
        assert torch.isfinite(out.float()).all() and (scatter or ((out[~live] == 7.0).all() and got[0][0][live].any()))


def test_scale_atoms_of_counted_rows():
    from deepep_efa_b200 import _ext
    C = _ext.load()
    counts, stride, nkb = [0, 1, 31, 32, 33, 127, 128, 129, 256], 256, 5
    s = torch.exp2(torch.randint(-9, 9, (len(counts) * stride, nkb), device="cuda").float())
    full = C.build_sf_atoms_a(s).view(-1, nkb, 32, 4, 4)
    some = C.build_sf_atoms_a(s, torch.tensor(counts, dtype=torch.int32, device="cuda"), stride).view(-1, nkb, 32, 4, 4)
    for g, n in enumerate(counts):
        for r in range(n):
            tile, m0, m1 = (g * stride + r) // 128, r % 32, r % 128 // 32
            assert torch.equal(full[tile, :, m0, m1], some[tile, :, m0, m1])


@pytest.mark.parametrize("pair", ["0", "1"])
@pytest.mark.parametrize("n_out,k_out", [(128, 128), (128, 384), (384, 640), (256, 256)])
def test_bf16_mn_major_half_width_tiles_and_pairs(monkeypatch, pair, n_out, k_out):
    """Column counts that are odd multiples of 128 end in a half-width tile, alone or split over a CTA pair; empty and small groups."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import grouped_gemm_dgrad, grouped_gemm_wgrad_inplace
    monkeypatch.setenv("DEEPEP_GEMM_PAIR", pair)
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(13)
    rows = [128, 0, 384, 64, 640]
    dy = torch.randn(sum(rows), n_out, device="cuda").to(torch.bfloat16)
    x = torch.randn(sum(rows), k_out, device="cuda").to(torch.bfloat16)
    w = (torch.randn(len(rows), n_out, k_out, device="cuda") * 0.1).to(torch.bfloat16)
    offs = _offsets(rows)
    dx, dw = grouped_gemm_dgrad(dy, w, offs), grouped_gemm_wgrad_inplace(dy, x, offs)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    o = offs.tolist()
    for g, n in enumerate(rows):
        d, xx = dy[o[g]:o[g + 1]].float(), x[o[g]:o[g + 1]].float()
        if n == 0:
            assert dw[g].float().abs().max().item() == 0
            continue
        # fp32 sums of bf16 products, rounded once to bf16 (2^-9 relative)
        assert _rel_err(dx[o[g]:o[g + 1]], d @ w[g].float()) < 4e-3
        assert _rel_err(dw[g], d.t() @ xx) < 4e-3


def test_fp8_native_wide_swiglu_writes_quantised_output():
    """The wide natively block-scaled SwiGLU kernel can emit e4m3 rows plus UE8M0 scale atoms itself; both must equal what
    the standalone cast makes of the kernel's BF16 output, bit for bit (valid rows only; masked groups stay untouched)."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import build_sf_atoms_a, build_sf_atoms_b
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(21)
    rows, K, N = [128, 200, 0, 384], 512, 1024  # N/2 = 512 outputs = 4 scale blocks per row
    G = len(rows)
    starts = [0]
    for r in rows:
        starts.append(starts[-1] + (r + 127) // 128 * 128)
    M = starts[-1]
    offs = torch.tensor(starts, dtype=torch.int32, device="cuda")
    ends = torch.tensor([starts[g] + rows[g] for g in range(G)], dtype=torch.int32, device="cuda")
    x = torch.randn(M, K, device="cuda") * torch.pow(2.0, (torch.arange(M, device="cuda") % 5).float()).unsqueeze(1)
    a, a_s = C.per_token_cast_to_fp8(x.to(torch.bfloat16), True, False)
    w = torch.randn(G, N, K, device="cuda") * 0.1
    wb = w.view(G, N // 128, 128, K // 128, 128)
    b_s = torch.exp2(torch.ceil(torch.log2(wb.abs().amax(dim=(2, 4)).clamp(min=1e-4) / 448.0))).contiguous()
    b = (wb / b_s.view(G, N // 128, 1, K // 128, 1)).view(G, N, K).to(torch.float8_e4m3fn).contiguous()
    sfa, sfb = build_sf_atoms_a(a_s), build_sf_atoms_b(b_s, N, True, True)
    h = torch.zeros(M, N // 2, dtype=torch.bfloat16, device="cuda")
    C.grouped_gemm(a, b, offs, 0, True, None, None, h, 0, 2000.0, ends, sfa, sfb)
    hq_ref, atoms_ref = C.per_token_cast_to_fp8(h, True, False, None, 1, None, None, None, True)
    hq = torch.full((M, N // 2), 0x55, dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)
    atoms = torch.full(((M + 127) // 128, N // 2 // 128, 512), 0x55, dtype=torch.uint8, device="cuda")
    C.grouped_gemm(a, b, offs, 0, True, None, None, None, 0, 2000.0, ends, sfa, sfb, out_fp8=hq, out_atoms=atoms)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    rr = torch.arange(M, device="cuda")
    for g in range(G):
        lo, hi = starts[g], starts[g] + rows[g]
        assert torch.equal(hq.view(torch.uint8)[lo:hi], hq_ref.view(torch.uint8)[lo:hi]), g
        assert (hq.view(torch.uint8)[hi:starts[g + 1]] == 0x55).all()
        r = rr[lo:hi]
        for kb in range(N // 2 // 128):
            idx = (r % 32) * 16 + ((r // 32) % 4) * 4
            assert torch.equal(atoms[r // 128, kb, idx], atoms_ref[r // 128, kb, idx]), (g, kb)


def test_fp8_native_wide_swiglu_cta_pairs(monkeypatch):
    """The wide natively block-scaled SwiGLU tile on CTA pairs (one 256-row MMA per pair, each CTA staging its own rows of A,
    half of the B tile and its own copy of the scale atoms) gives the same numbers as the single-CTA kernel; rows carry
    different power-of-two scales, so scale atoms that reached the wrong CTA's TMEM cannot pass."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import build_sf_atoms_a, build_sf_atoms_b, grouped_gemm, reference_grouped_gemm
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(31)
    rows, K, N = [256, 512, 0, 384, 128], 1024, 1024
    G = len(rows)
    starts = [0]
    for r in rows:
        starts.append(starts[-1] + (r + 127) // 128 * 128)
    M = starts[-1]
    offs = torch.tensor(starts, dtype=torch.int32, device="cuda")
    x = torch.randn(M, K, device="cuda") * torch.pow(2.0, (torch.arange(M, device="cuda") % 7).float()).unsqueeze(1)
    x = x * torch.pow(2.0, (torch.arange(K, device="cuda") // 128 % 3).float()).unsqueeze(0)
    a, a_s = C.per_token_cast_to_fp8(x.to(torch.bfloat16), True, False)
    w = torch.randn(G, N, K, device="cuda") * 0.1 * torch.pow(2.0, (torch.arange(N, device="cuda") // 128 % 4).float()).view(1, N, 1)
    wb = w.view(G, N // 128, 128, K // 128, 128)
    b_s = torch.exp2(torch.ceil(torch.log2(wb.abs().amax(dim=(2, 4)).clamp(min=1e-4) / 448.0))).contiguous()
    b = (wb / b_s.view(G, N // 128, 1, K // 128, 1)).view(G, N, K).to(torch.float8_e4m3fn).contiguous()
    sfa, sfb = build_sf_atoms_a(a_s), build_sf_atoms_b(b_s, N, True, True)
    monkeypatch.setenv("DEEPEP_GEMM_PAIR", "0")
    single = grouped_gemm(a, b, offs, swiglu=True, sfa_atoms=sfa, sfb_atoms=sfb)
    monkeypatch.setenv("DEEPEP_GEMM_PAIR", "1")
    paired = grouped_gemm(a, b, offs, swiglu=True, sfa_atoms=sfa, sfb_atoms=sfb)
    paired_small_grid = grouped_gemm(a, b, offs, swiglu=True, sfa_atoms=sfa, sfb_atoms=sfb, num_sms=6)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    ref = reference_grouped_gemm(a, b, offs, swiglu=True, a_scales=a_s, b_scales=b_s)
    assert _rel_err(single, ref) < 1.5e-2
    assert _rel_err(paired, ref) < 1.5e-2, _rel_err(paired, ref)
    assert torch.equal(paired, single) and torch.equal(paired_small_grid, single)


def test_held_successor_leaves_the_free_sms_to_another_stream():
    """A GEMM on four SMs that holds its successor: the one behind it in the stream must not occupy the other SMs meanwhile, so a GEMM
    of another stream, launched last, ends before it begins."""
    from deepep_efa_b200 import _ext
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(23)
    big = torch.randn(8192, 4096, device="cuda").to(torch.bfloat16)
    big_w = (torch.randn(1, 4096, 4096, device="cuda") * 0.02).to(torch.bfloat16)
    small = torch.randn(148 * 128, 256, device="cuda").to(torch.bfloat16)
    small_w = torch.randn(1, 256, 256, device="cuda").to(torch.bfloat16)
    offs, offs_small = _offsets([8192]), _offsets([148 * 128])
    big_id = torch.iinfo(torch.int64).max
    stamps = [torch.tensor([big_id, 0, 0, 0], dtype=torch.int64, device="cuda") for _ in range(2)]
    side = torch.cuda.Stream()
    outs = []
    for warm in (True, False):  # (once without stamps, so that no allocation or module load falls between the launches)
        outs = [torch.empty(8192, 4096, dtype=torch.bfloat16, device="cuda")] + [torch.empty(148 * 128, 256, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        C.grouped_gemm(big, big_w, offs, 0, False, None, None, outs[0], 4, 2000.0, hold_successor=True)
        C.grouped_gemm(small, small_w, offs_small, 0, False, None, None, outs[1], 0, 2000.0, trace=None if warm else stamps[0])
        with torch.cuda.stream(side):
            C.grouped_gemm(small, small_w, offs_small, 0, False, None, None, outs[2], 100, 2000.0, trace=None if warm else stamps[1])
        torch.cuda.synchronize()
    assert C.gemm_error(0) == 0 and torch.equal(outs[1], outs[2])
    assert stamps[1][1].item() < stamps[0][0].item()


@pytest.mark.parametrize("L", [1, 3, 147, 149, 300, 1024, 1025, 2500])
@pytest.mark.parametrize("N,K", [(1, 1), (700, 3), (8200, 4), (10923, 6)])
def test_expert_plan_matches_the_cpu_plan(L, N, K):
    """More experts than CTAs, than a pass over the ids takes and than one launch takes; selections past a chunk of 32768."""
    import numpy as np
    from deepep_efa_b200.ops.permute import build_expert_plan
    if L * N * K > 70_000_000:
        pytest.skip("the CPU plan holds a word per selection and expert")
    g = torch.Generator().manual_seed(L + N)
    idx = torch.randint(-1, L + 1, (N, K), generator=g)
    idx[idx == L] = -1
    counts = (torch.bincount(idx[idx >= 0], minlength=L) + 127) // 128 * 128
    want = build_expert_plan(idx, counts.tolist())
    for given in (counts.tolist(), counts.double().numpy(), [np.int64(c) for c in counts.tolist()]):
        got = build_expert_plan(idx.cuda(), given)
        assert got.num_rows == want.num_rows and torch.equal(got.m_offsets.cpu(), want.m_offsets)
        assert torch.equal(got.pos.cpu(), want.pos) and torch.equal(got.src_row.cpu(), want.src_row)
        filled = want.src_row >= 0
        assert torch.equal(got.src_k.cpu()[filled], want.src_k[filled]) and bool((got.src_k.cpu()[~filled] == 0).all())
    beyond = idx.clone()
    beyond[idx < 0] = L  # an id past the last expert is as good as none
    assert torch.equal(build_expert_plan(beyond.cuda(), counts.tolist()).pos.cpu(), want.pos)


@pytest.mark.parametrize("N", [1, 31, 8191, 8192, 8193, 16385, 24577, 40961])
def test_expert_plan_where_parts_of_a_chunk_are_empty(N):
    """CTAs start at different quarters of 32768 selections, some of which have none."""
    from deepep_efa_b200.ops.permute import build_expert_plan
    L = 9
    idx = torch.randint(0, L, (N, 1), generator=torch.Generator().manual_seed(N))
    counts = ((torch.bincount(idx.view(-1), minlength=L) + 127) // 128 * 128).tolist()
    want, got = build_expert_plan(idx, counts), build_expert_plan(idx.cuda(), counts)
    assert torch.equal(got.pos.cpu(), want.pos) and torch.equal(got.src_row.cpu(), want.src_row)


def test_gathers_of_rows_without_columns():
    """Nothing to move, as with the scale rows of fewer than 128 channels: no launch, and no error from one."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.permute import gather_reduce_rows, gather_rows
    rows = torch.zeros(5, dtype=torch.int32, device="cuda")
    pos = torch.zeros(5, 2, dtype=torch.int32, device="cuda")
    empty = torch.empty(3, 0, dtype=torch.bfloat16, device="cuda")
    assert gather_rows(empty, rows).shape == (5, 0) and gather_reduce_rows(empty, pos).shape == (5, 0)
    out = torch.empty(5, 0, dtype=torch.bfloat16, device="cuda")
    _ext.load().stage_reduce(torch.empty(10, 0, dtype=torch.bfloat16, device="cuda"), out, pos.long(), torch.ones(5, 2, device="cuda"), 4)
    torch.cuda.synchronize()


@pytest.mark.parametrize("kind", ["bf16", "mx_wide"])
def test_tile_counter_after_a_launch_that_gave_up(kind):
    """An arrival gate that nobody opens ends in an error after its limit; the tile counter is zero again, and the next launch, whose
    table is built early, is right."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import build_sf_atoms_a, build_sf_atoms_b
    C = _ext.load()
    C.gemm_clear_error(0)
    torch.manual_seed(29)
    counts, stride, K, N = [200, 0, 33, 128], 256, 512, 512
    G = len(counts)
    cnt = torch.tensor(counts, device="cuda", dtype=torch.int32)
    starts = torch.arange(G + 1, device="cuda", dtype=torch.int32) * stride
    live = (torch.arange(stride, device="cuda").unsqueeze(0) < cnt.unsqueeze(1)).view(-1)
    x = torch.randn(G * stride, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(G, N, K, device="cuda") * 0.1).to(torch.bfloat16)
    scales = (None, None)
    if kind == "mx_wide":
        x, a_s = C.per_token_cast_to_fp8(x, True, False)
        w = (w.float() / 2.0 ** -9).to(torch.float8_e4m3fn)
        scales = (build_sf_atoms_a(a_s), build_sf_atoms_b(torch.full((G, N // 128, K // 128), 2.0 ** -9, device="cuda"), N, False, True))

    def run(timeout_ms, **how):
        out = torch.zeros(G * stride, N, device="cuda", dtype=torch.bfloat16)
        C.grouped_gemm(x, w, starts, 0, False, None, None, out, 0, timeout_ms, cnt, *scales, m_ends_are_counts=True, **how)
        return out

    want = run(2000.0)
    sched = torch.zeros(2, dtype=torch.int32, device="cuda")
    ready, expected = torch.zeros(G, dtype=torch.int64, device="cuda"), torch.tensor([0, 0, 0, 1], dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        run(20.0, sched=sched, ready=ready, expected=expected)
        torch.cuda.synchronize()
        assert C.gemm_error(0) == 1 and sched.tolist() == [0, 0]
        C.gemm_clear_error(0)
        run(2000.0, sched=sched)
        got = run(2000.0, sched=sched, early_table=True)
        torch.cuda.synchronize()
        assert C.gemm_error(0) == 0 and sched.tolist() == [0, 0]
        assert torch.equal(got[live], want[live])


@pytest.mark.parametrize("scatter", [False, True])
def test_token_columns_tile_of_96(scatter):
    """The one tile that is longer than the step of a cut group without being whole scale atoms."""
    test_token_columns_tile_sizes(96, scatter)


def _columns_case(counts, stride, K, I):
    """Both natively block-scaled products of an expert layer, as functions of the launch's options, on groups of `stride` rows of which
    `counts` count."""
    from deepep_efa_b200 import _ext
    from deepep_efa_b200.ops.grouped_gemm import build_sf_atoms_a, build_sf_atoms_b
    C, G = _ext.load(), len(counts)
    cnt = torch.tensor(counts, device="cuda", dtype=torch.int32)
    starts = torch.arange(G + 1, device="cuda", dtype=torch.int32) * stride
    a, a_s = C.per_token_cast_to_fp8(torch.randn(G * stride, K, device="cuda").to(torch.bfloat16), True, False)
    b = torch.randn(G, 2 * I, K, device="cuda").to(torch.float8_e4m3fn)
    b_s = torch.exp2(torch.randint(-8, -4, (G, 2 * I // 128, K // 128), device="cuda").float())
    sfa, sfb, sfb_swiglu = build_sf_atoms_a(a_s), build_sf_atoms_b(b_s, 2 * I, False, True), build_sf_atoms_b(b_s, 2 * I, True, True)

    def run(swiglu, timeout_ms=2000.0, sms=0, **how):
        if not swiglu:
            out = torch.zeros(G * stride, 2 * I, device="cuda", dtype=torch.bfloat16)
            C.grouped_gemm(a, b, starts, 0, False, None, None, out, sms, timeout_ms, cnt, sfa, sfb, m_ends_are_counts=True, **how)
            return (out,)
        q, qs = torch.zeros(G * stride, I, dtype=torch.uint8, device="cuda"), torch.zeros(G * stride // 128, I // 128, 512, dtype=torch.uint8, device="cuda")
        C.grouped_gemm(a, b, starts, 0, True, None, None, None, sms, timeout_ms, cnt, sfa, sfb_swiglu, out_fp8=q.view(torch.float8_e4m3fn), out_atoms=qs,
                       m_ends_are_counts=True, **how)
        return q, qs

    return C, run


@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("cap", [64, 160])
def test_token_columns_behind_an_arrival_gate(swiglu, cap):
    """Gates that are open, and one that nobody opens: an error after the limit, the tile counter zero again, and the next launch right."""
    torch.manual_seed(cap)
    C, run = _columns_case([200, 0, 33, 128, 1], 256, 512, 256)
    C.gemm_clear_error(0)
    want = run(swiglu)
    sched = torch.zeros(2, dtype=torch.int32, device="cuda")
    expected = torch.tensor([3, 0, 1, 7, 2], dtype=torch.int64, device="cuda")
    shut = expected.clone()
    shut[3] -= 1

    def check(got):
        torch.cuda.synchronize()
        assert C.gemm_error(0) == 0 and sched.tolist() == [0, 0]
        assert all(torch.equal(g, w) for g, w in zip(got, want))

    for _ in range(2):
        check(run(swiglu, sched=sched, ready=expected, expected=expected, tokens_as_columns=cap))
        run(swiglu, timeout_ms=20.0, sched=sched, ready=shut, expected=expected, tokens_as_columns=cap)
        torch.cuda.synchronize()
        assert C.gemm_error(0) == 1 and sched.tolist() == [0, 0]
        C.gemm_clear_error(0)
        for early in (False, True):
            check(run(swiglu, sched=sched, early_table=early, tokens_as_columns=cap))


def test_token_columns_hold_their_successor():
    """On four SMs with tokens as columns: the kernel behind it, which would fit on the others, begins when it has ended."""
    torch.manual_seed(31)
    C, run = _columns_case([128] * 64, 128, 2048, 512)
    C.gemm_clear_error(0)
    small = torch.randn(148 * 128, 256, device="cuda").to(torch.bfloat16)
    small_w = torch.randn(1, 256, 256, device="cuda").to(torch.bfloat16)
    offs, out = _offsets([148 * 128]), torch.empty(148 * 128, 256, dtype=torch.bfloat16, device="cuda")
    for _ in range(2):  # the first round loads both kernels (a product with a trace takes rows)
        stamps = [torch.tensor([torch.iinfo(torch.int64).max, 0, 0, 0], dtype=torch.int64, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        run(False, sms=4, tokens_as_columns=128, hold_successor=True, trace=stamps[0])
        C.grouped_gemm(small, small_w, offs, 0, False, None, None, out, 0, 2000.0, trace=stamps[1])
        torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    assert stamps[0][1].item() <= stamps[1][0].item()


@pytest.mark.parametrize("N,K,H", [(6300, 6, 4096), (6300, 1, 4096), (3600, 8, 7176), (700, 6, 1024)])
def test_permutation_by_changed_plans(N, K, H):
    """Above and below the size from which rows are spread instead of gathered: what src_row says decides, whatever was done to either map since."""
    import dataclasses
    from deepep_efa_b200.ops.permute import build_expert_plan, gather_rows, permute
    torch.manual_seed(3)
    idx = torch.rand(N, 16, device="cuda").topk(K, dim=1).indices
    idx[torch.rand(N, K, device="cuda") < 0.1] = -1
    counts = [(int((idx == e).sum()) + 127) // 128 * 128 for e in range(16)]
    plan, x = build_expert_plan(idx, counts), torch.randn(N, H, device="cuda").to(torch.bfloat16)
    M = plan.num_rows
    dropped, other, short = plan.src_row.clone(), plan.src_row.clone(), plan.pos.clone()
    dropped[torch.rand(M, device="cuda") < 0.2] = -1
    some = torch.rand(M, device="cuda") < 0.2
    other[some] = torch.randint(0, N, (M,), device="cuda", dtype=torch.int32)[some]
    short[torch.rand(N, K, device="cuda") < 0.2] = -1
    wild = torch.randint(-5, 2 * M, (N, K), device="cuda", dtype=torch.int32)
    for change in ({}, dict(src_row=dropped), dict(src_row=other), dict(pos=short), dict(pos=wild), dict(pos=plan.pos[:0]), dict(pos=plan.pos.long()), dict(pos=None),
                   dict(pos=plan.pos.t().contiguous().t()), dict(src_row=plan.src_row[: M - 77].contiguous()), dict(src_row=dropped, pos=wild)):
        changed = dataclasses.replace(plan, **change)
        dirt = torch.full((M, H), float("nan"), dtype=torch.bfloat16, device="cuda")
        del dirt
        assert torch.equal(permute(x, changed), gather_rows(x, changed.src_row)), change.keys()
