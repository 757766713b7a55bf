"""tcgen05 GEMM kernels against fp32 PyTorch references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel_err(got, want):
    return ((got.float() - want).norm() / want.norm().clamp_min(1e-6)).item()


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (128, 256, 512), (256, 512, 1024),
                                   (300, 520, 264), (1024, 3584, 2048), (77, 40, 72)])
def test_gemm_bf16_matches_fp32(m, n, k):
    from aboleth_b200.ops import check_gemm_status, gemm_bf16

    g = torch.Generator(device="cuda").manual_seed(m * 7 + n)
    a = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(n, k, generator=g, device="cuda").to(torch.bfloat16)
    out = gemm_bf16(a, b)
    torch.cuda.synchronize()
    check_gemm_status("cuda")
    want = a.float() @ b.float().t()
    assert _rel_err(out, want) < 5e-3
    # An exact case: small integers are exact in bf16 and in the fp32 accumulator.
    ai = torch.randint(-3, 4, (m, k), generator=g, device="cuda").to(torch.bfloat16)
    bi = torch.randint(-3, 4, (n, k), generator=g, device="cuda").to(torch.bfloat16)
    exact = (ai.float() @ bi.float().t())
    got = gemm_bf16(ai, bi).float()
    torch.cuda.synchronize()
    assert torch.equal(got, exact.to(torch.bfloat16).float())


def test_grouped_gemm_matches_loop_of_matmuls():
    from aboleth_b200.ops import check_gemm_status, grouped_gemm_bf16

    experts, n, k = 6, 512, 320
    counts = torch.tensor([0, 5, 128, 200, 1, 131], dtype=torch.int32, device="cuda")
    align = 8
    padded = (counts + align - 1) // align * align
    offsets = (torch.cumsum(padded, 0) - padded).to(torch.int32)
    rows = int(padded.sum())
    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(rows, k, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(experts, n, k, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((rows, n), 7.0, dtype=torch.bfloat16, device="cuda")
    grouped_gemm_bf16(a, w, counts, offsets, out)
    torch.cuda.synchronize()
    check_gemm_status("cuda")
    for e in range(experts):
        lo, cnt = int(offsets[e]), int(counts[e])
        want = a[lo:lo + cnt].float() @ w[e].float().t()
        if cnt:
            assert _rel_err(out[lo:lo + cnt], want) < 5e-3
        pad = out[lo + cnt:lo + int(padded[e])]
        assert bool((pad == 7.0).all())  # rows outside the expert are never written


def test_grouped_gemm_large_experts_use_wide_tiles():
    """Averages of >= 512 rows per expert take the 256-row tile path; ragged counts, many columns."""
    from aboleth_b200.ops import check_gemm_status, grouped_gemm_bf16

    experts, n, k = 4, 1288, 256  # 6 tile columns, the last one partial
    counts = torch.tensor([700, 0, 1031, 517], dtype=torch.int32, device="cuda")
    padded = (counts + 7) // 8 * 8
    offsets = (torch.cumsum(padded, 0) - padded).to(torch.int32)
    rows = int(padded.sum())
    g = torch.Generator(device="cuda").manual_seed(11)
    a = torch.randn(rows, k, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(experts, n, k, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((rows, n), 7.0, dtype=torch.bfloat16, device="cuda")
    grouped_gemm_bf16(a, w, counts, offsets, out)
    torch.cuda.synchronize()
    check_gemm_status("cuda")
    for e in range(experts):
        lo, cnt = int(offsets[e]), int(counts[e])
        if cnt:
            want = a[lo:lo + cnt].float() @ w[e].float().t()
            assert _rel_err(out[lo:lo + cnt], want) < 5e-3
        assert bool((out[lo + cnt:lo + int(padded[e])] == 7.0).all())


@pytest.mark.parametrize("m,n,k", [(512, 256, 256), (1000, 520, 384), (4096, 4096, 2048)])
def test_gemm_e4m3_matches_fp32(m, n, k):
    """e4m3 x e4m3 products are exact in fp32, so only the accumulation order and the final bf16
    rounding separate the kernel from an fp32 matmul of the dequantised operands."""
    from aboleth_b200.ops import check_gemm_status, gemm_e4m3

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g, device="cuda").to(torch.float8_e4m3fn)
    b = torch.randn(n, k, generator=g, device="cuda").to(torch.float8_e4m3fn)
    out = gemm_e4m3(a, b, alpha=0.5)
    torch.cuda.synchronize()
    check_gemm_status(a.device)
    want = 0.5 * (a.float() @ b.float().t())
    assert _rel_err(out, want) < 5e-3
    # small integers: every partial sum is exact
    ai = torch.randint(-2, 3, (m, k), generator=g, device="cuda").float().to(torch.float8_e4m3fn)
    bi = torch.randint(-2, 3, (n, k), generator=g, device="cuda").float().to(torch.float8_e4m3fn)
    got = gemm_e4m3(ai, bi).float()
    torch.cuda.synchronize()
    assert torch.equal(got, (ai.float() @ bi.float().t()).to(torch.bfloat16).float())


@pytest.mark.parametrize("m,n,k,pow2", [(256, 384, 512, True), (1000, 520, 384, False)])
def test_block_scaled_e4m3_gemm_matches_fp32(m, n, k, pow2):
    """1 x 128 activation scales and 128 x 128 weight scales: the expansion to bf16 is the fp32
    product rounded once (exact for power-of-two scales), and the GEMM over it matches an fp32
    matmul of the dequantised operands."""
    from aboleth_b200.ops import check_gemm_status
    from aboleth_b200.ops.gemm import dequant_block_scaled, gemm_e4m3_block_scaled
    from aboleth_b200.ops.moe_ops import quant_fp8

    g = torch.Generator(device="cuda").manual_seed(m * 7 + n)
    x = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    a_q, a_s = quant_fp8(x, round_scale=pow2)
    w = 0.02 * torch.randn(n, k, generator=g, device="cuda")
    rows_b, cols_b = -(-n // 128), k // 128
    padded = torch.zeros(rows_b * 128, k, device="cuda")
    padded[:n] = w
    amax = padded.view(rows_b, 128, cols_b, 128).abs().amax(dim=(1, 3)).clamp_min(1e-10)
    b_s = amax / 448.0
    if pow2:
        b_s = torch.exp2(torch.ceil(torch.log2(b_s)))
    b_full = b_s.repeat_interleave(128, dim=0)[:n].repeat_interleave(128, dim=1)
    b_q = (w / b_full).clamp(-448, 448).to(torch.float8_e4m3fn)
    a_full = a_s.repeat_interleave(128, dim=1)

    a_deq = dequant_block_scaled(a_q, a_s)
    b_deq = dequant_block_scaled(b_q, b_s.contiguous(), block=(128, 128))
    torch.cuda.synchronize()
    assert torch.equal(a_deq, (a_q.float() * a_full).to(torch.bfloat16))
    assert torch.equal(b_deq, (b_q.float() * b_full).to(torch.bfloat16))
    if pow2:  # nothing was rounded
        assert torch.equal(a_deq.float(), a_q.float() * a_full)

    # Power-of-two scales go to the tensor core as ue8m0 (no expansion); others take the expansion.
    out = gemm_e4m3_block_scaled(a_q, a_s, b_q, b_s.contiguous(), path="mx" if pow2 else "expand")
    torch.cuda.synchronize()
    check_gemm_status(out.device)
    want = (a_q.float() * a_full) @ (b_q.float() * b_full).t()
    assert _rel_err(out, want) < 5e-3
    if pow2:
        # fp32 accumulation of exact products of e4m3 values and power-of-two scales: the two paths
        # differ only in the order of additions
        other = gemm_e4m3_block_scaled(a_q, a_s, b_q, b_s.contiguous(), path="expand")
        torch.cuda.synchronize()
        assert _rel_err(out, other.float()) < 2e-3
    # A strided view (rows of a wider buffer) goes through the same kernel.
    wide = torch.zeros(m, k + 64, dtype=torch.float8_e4m3fn, device="cuda")
    wide[:, :k] = a_q
    assert torch.equal(dequant_block_scaled(wide[:, :k], a_s), a_deq)


@pytest.mark.parametrize("tile,m,n,k", [("1", 300, 640, 512),     # one CTA: partial rows, 2.5 column tiles
                                         ("2", 300, 640, 512),     # CTA pairs: a second row tile of 44 rows
                                         ("2", 700, 1000, 384),    # three row tiles, ragged last column tile
                                         ("1", 3000, 5000, 128),   # several tiles per CTA, one K step
                                         ("2", 3000, 5000, 128)])  # ... and per pair: both accumulators, in turn
def test_block_scaled_mx_gemm_is_exact_on_integers_and_flags_bad_scales(tile, m, n, k, monkeypatch):
    """Small integers and power-of-two scales: every product and partial sum is exact, so the
    tensor-core path must reproduce the fp32 result bit for bit (after the bf16 rounding of the
    output) - this pins the scale-factor layout: a wrong row or K segment changes the sum."""
    from aboleth_b200.ops import check_gemm_status, gemm_e4m3_block_scaled
    from aboleth_b200.ops.gemm import gemm_status

    monkeypatch.setenv("ABOLETH_GEMM_MX_TILE", tile)
    g = torch.Generator(device="cuda").manual_seed(11)
    a = torch.randint(-2, 3, (m, k), generator=g, device="cuda").float()
    b = torch.randint(-2, 3, (n, k), generator=g, device="cuda").float()
    a_s = torch.exp2(torch.randint(-3, 4, (m, k // 128), generator=g, device="cuda").float())
    b_s = torch.exp2(torch.randint(-3, 4, (-(-n // 128), k // 128), generator=g, device="cuda").float())
    a_q, b_q = a.to(torch.float8_e4m3fn), b.to(torch.float8_e4m3fn)
    out = gemm_e4m3_block_scaled(a_q, a_s, b_q, b_s)
    torch.cuda.synchronize()
    check_gemm_status(out.device)
    a_full = a_s.repeat_interleave(128, dim=1)
    b_full = b_s.repeat_interleave(128, dim=0)[:n].repeat_interleave(128, dim=1)
    want = ((a * a_full) @ (b * b_full).t()).to(torch.bfloat16)
    assert torch.equal(out, want)
    # a scale that is not a power of two cannot be carried as ue8m0: reported, not silently rounded
    bad = a_s.clone()
    bad[5, -1] = 0.3
    gemm_e4m3_block_scaled(a_q, bad, b_q, b_s)
    torch.cuda.synchronize()
    assert gemm_status(out.device)[:2].tolist() == [3, 0x3500]
    gemm_status(out.device).zero_()


@pytest.mark.parametrize("counts", [[0, 5, 128, 200, 1, 131],        # small experts: 128-row tiles
                                    [700, 0, 1031, 517, 300, 260]])   # 256-row tiles, ragged
def test_grouped_block_scaled_gemm_is_exact_on_integers(counts):
    """Expert-contiguous e4m3 rows (every expert on a 128-row boundary) times e4m3 expert weights, scales
    applied by the tensor core.  Small integers and power-of-two scales make the result exact."""
    from aboleth_b200.ops import check_gemm_status, grouped_gemm_e4m3_mx, pack_scales_mx

    experts, n, k = len(counts), 640, 384
    counts = torch.tensor(counts, dtype=torch.int32, device="cuda")
    padded = (counts + 127) // 128 * 128
    offsets = (torch.cumsum(padded, 0) - padded).to(torch.int32)
    rows = int(padded.sum())
    g = torch.Generator(device="cuda").manual_seed(17)
    a = torch.randint(-2, 3, (rows, k), generator=g, device="cuda").float()
    w = torch.randint(-2, 3, (experts, n, k), generator=g, device="cuda").float()
    a_s = torch.exp2(torch.randint(-2, 3, (rows, k // 128), generator=g, device="cuda").float())
    w_s = torch.exp2(torch.randint(-2, 3, (experts, n // 128, k // 128), generator=g, device="cuda").float())
    fp8 = torch.float8_e4m3fn
    out = torch.full((rows, n), 7.0, dtype=torch.bfloat16, device="cuda")
    grouped_gemm_e4m3_mx(a.to(fp8), pack_scales_mx(a_s, rows, k, weight=False), w.to(fp8),
                         pack_scales_mx(w_s.view(experts * n // 128, k // 128), experts * n, k, weight=True),
                         counts, offsets, out)
    torch.cuda.synchronize()
    check_gemm_status("cuda")
    a_full = a * a_s.repeat_interleave(128, dim=1)
    for e in range(experts):
        lo, cnt = int(offsets[e]), int(counts[e])
        w_full = w[e] * w_s[e].repeat_interleave(128, dim=0).repeat_interleave(128, dim=1)
        assert torch.equal(out[lo:lo + cnt], (a_full[lo:lo + cnt] @ w_full.t()).to(torch.bfloat16))
        assert bool((out[lo + cnt:lo + int(padded[e])] == 7.0).all())   # padding rows are never written


@pytest.mark.parametrize("counts,n,k", [([0, 5, 128, 200, 1, 131], 320, 264),    # 128-row tiles, 2.5 column tiles
                                        ([700, 0, 1031, 517], 1288, 192),       # 256-row tiles, ragged columns
                                        ([1000, 1281, 897, 640], 2048, 64)])    # 256 of them on 74 pairs, one K step
def test_grouped_swiglu_gemm_matches_fp32(counts, n, k):
    """silu(a gate^T) * (a up^T) per expert.  The oracle is fp32 over the same bf16 operands, so what differs
    is the one bf16 rounding of the result (2^-9 relative, 1.7e-3 in the mean) and the fast exponential (a few
    2^-22): 5e-3 as for the other products.  The up rows start at n, which is no multiple of the tile."""
    from aboleth_b200.ops import check_gemm_status, grouped_gemm_swiglu_bf16

    experts = len(counts)
    counts = torch.tensor(counts, dtype=torch.int32, device="cuda")
    padded = (counts + 7) // 8 * 8
    offsets = (torch.cumsum(padded, 0) - padded).to(torch.int32)
    rows = int(padded.sum())
    g = torch.Generator(device="cuda").manual_seed(29)
    a = torch.randn(rows, k, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(experts, 2 * n, k, generator=g, device="cuda") * 0.2).to(torch.bfloat16)
    out = torch.full((rows, n), 7.0, dtype=torch.bfloat16, device="cuda")
    grouped_gemm_swiglu_bf16(a, w, counts, offsets, out)
    torch.cuda.synchronize()
    check_gemm_status("cuda")
    for e in range(experts):
        lo, cnt = int(offsets[e]), int(counts[e])
        if cnt:
            h = a[lo:lo + cnt].float() @ w[e].float().t()
            assert _rel_err(out[lo:lo + cnt], torch.nn.functional.silu(h[:, :n]) * h[:, n:]) < 5e-3
        assert bool((out[lo + cnt:lo + int(padded[e])] == 7.0).all())  # rows outside the expert are never written


@pytest.mark.parametrize("counts,n,k", [([0, 5, 128, 200, 1, 131], 384, 384), ([700, 0, 300], 128, 128),
                                        ([700, 0, 500], 128, 128),              # pairs, as the next
                                        ([1000, 1281, 897, 640], 2048, 128)])   # 256 pair tiles on 74 pairs
def test_grouped_swiglu_block_scaled_gemm_is_its_parts(counts, n, k):
    """The fused gate / up product and its quantisation against the separate passes: block-scaled product, SiLU and
    multiply in bf16, ``quant_fp8``.  Both round to bf16 at the same three places; only the exponential differs, by a
    few 2^-22, which moves a bf16 rounding for one value in 2^11 at most and an e4m3 code for fewer."""
    from aboleth_b200.ops import (check_gemm_status, grouped_gemm_e4m3_mx, grouped_gemm_swiglu_e4m3_mx,
                                  pack_scales_mx, quant_fp8)

    experts, fp8 = len(counts), torch.float8_e4m3fn
    counts = torch.tensor(counts, dtype=torch.int32, device="cuda")
    padded = (counts + 127) // 128 * 128
    offsets = (torch.cumsum(padded, 0) - padded).to(torch.int32)
    rows = int(padded.sum())
    g = torch.Generator(device="cuda").manual_seed(31)
    a = torch.randn(rows, k, generator=g, device="cuda").to(fp8)
    w = torch.randn(experts, 2 * n, k, generator=g, device="cuda").to(fp8)
    a_s = torch.exp2(torch.randint(-3, 2, (rows, k // 128), generator=g, device="cuda").float())
    w_s = torch.exp2(torch.randint(-4, 0, (experts, 2 * n // 128, k // 128), generator=g, device="cuda").float())
    a_packed = pack_scales_mx(a_s, rows, k, weight=False)
    w_packed = pack_scales_mx(w_s.view(-1, k // 128), experts * 2 * n, k, weight=True)
    h = torch.zeros(rows, 2 * n, dtype=torch.bfloat16, device="cuda")
    grouped_gemm_e4m3_mx(a, a_packed, w, w_packed, counts, offsets, h)
    want, want_scales = quant_fp8((torch.nn.functional.silu(h[:, :n]) * h[:, n:]).contiguous(), round_scale=True)
    want_packed = pack_scales_mx(want_scales, rows, n, weight=False)
    q = torch.full((rows, n), 7.0, device="cuda").to(fp8)
    packed = torch.zeros_like(want_packed)
    grouped_gemm_swiglu_e4m3_mx(a, a_packed, w, w_packed, counts, offsets, out=(q, packed))
    torch.cuda.synchronize()
    check_gemm_status("cuda")
    # word (r % 32) * 4 + r / 32 of atom [row block][column block] is row r's scale
    by_row = lambda p: p.view(torch.int32).view(-1, n // 128, 32, 4)[: rows // 128].permute(0, 3, 2, 1).reshape(rows, -1)  # noqa: E731
    live = torch.zeros(rows, dtype=torch.bool, device="cuda")
    for e in range(experts):
        live[int(offsets[e]):int(offsets[e]) + int(counts[e])] = True
    assert bool((q[~live].float() == 7.0).all()) and bool((by_row(packed)[~live] == 0).all())
    assert torch.equal(by_row(packed)[live], by_row(want_packed)[live])
    assert float((q[live].float() != want[live].float()).double().mean()) <= 2.0 ** -11


def _dense(kind, a, b, out, g):
    """The public entry point of a kind on small integers; the fp32 operands that it stands for."""
    from aboleth_b200.ops import gemm_bf16, gemm_e4m3, gemm_e4m3_mx, pack_scales_mx

    (m, k), n = a.shape, b.shape[0]
    if kind == "bf16":
        gemm_bf16(a.bfloat16(), b.bfloat16(), out)
        return a, b
    fp8 = torch.float8_e4m3fn
    if kind == "e4m3":
        gemm_e4m3(a.to(fp8), b.to(fp8), out)
        return a, b
    a_s = torch.exp2(torch.randint(-2, 3, (m, k // 128), generator=g, device="cuda").float())
    b_s = torch.exp2(torch.randint(-2, 3, (-(-n // 128), k // 128), generator=g, device="cuda").float())
    gemm_e4m3_mx(a.to(fp8), pack_scales_mx(a_s, m, k, weight=False), b.to(fp8), pack_scales_mx(b_s, n, k, weight=True),
                 out)
    return (a * a_s.repeat_interleave(128, dim=1),
            b * b_s.repeat_interleave(128, dim=0)[:n].repeat_interleave(128, dim=1))


def _dense_case(kind, m, n, k):
    from aboleth_b200.ops import check_gemm_status

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randint(-2, 3, (m, k), generator=g, device="cuda").float()
    b = torch.randint(-2, 3, (n, k), generator=g, device="cuda").float()
    wide = torch.full((m + 1, n + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    a_full, b_full = _dense(kind, a, b, wide[:m, :n], g)
    torch.cuda.synchronize()
    check_gemm_status("cuda")
    assert torch.equal(wide[:m, :n], (a_full @ b_full.t()).to(torch.bfloat16))
    assert bool((wide[m] == 7.0).all()) and bool((wide[:, n:] == 7.0).all())


def _choice(kind, m, n, k):
    import ctypes

    from aboleth_b200.ops._kernels import call

    choice = (ctypes.c_int * 2)()
    call("ab_gemm_choice", ("bf16", "e4m3", "mx").index(kind), m, n, k, choice)
    return choice[0], choice[1]


# The kernels of the dispatch: a token tile of the split kernel; a loop with 256- (0) or 224-column (-1) pair tiles;
# for block-scaled operands the one-CTA loop (0, 1) and the pair loop (0, 2).
@pytest.mark.parametrize("kind,m,n,k,kernel", [
    ("bf16", 1, 312, 256, 32), ("bf16", 232, 2664, 256, 64), ("bf16", 132, 3872, 2048, 128),
    ("bf16", 2649, 1584, 1024, 256), ("bf16", 587, 5448, 384, 0), ("bf16", 227, 4840, 256, -1),
    ("e4m3", 1, 280, 256, 32), ("e4m3", 65, 6968, 256, 64), ("e4m3", 303, 1832, 3840, 128),
    ("e4m3", 783, 4624, 2176, 256), ("e4m3", 1920, 2112, 256, 0), ("e4m3", 1676, 704, 256, -1),
    ("mx", 1, 256, 256, 32), ("mx", 56, 288, 768, 64), ("mx", 129, 3296, 2304, 128), ("mx", 2721, 1544, 1024, 256),
    ("mx", 75, 360, 256, (0, 1)), ("mx", 905, 8136, 1024, (0, 2))])
def test_dense_gemm_through_every_kernel_of_its_dispatch(kind, m, n, k, kernel):
    """One size per outcome of the rule that picks the kernel, exact on integers, in a strided output."""
    choice = _choice(kind, m, n, k)
    assert (choice if isinstance(kernel, tuple) else choice[0]) == kernel
    _dense_case(kind, m, n, k)


@pytest.mark.parametrize("kind", ["bf16", "e4m3"])
@pytest.mark.parametrize("width", [256, 224])
@pytest.mark.parametrize("m,n,k", [(3000, 5000, 64), (3000, 5000, 320)])
def test_pair_loop_with_several_tiles_per_pair(kind, m, n, k, width, monkeypatch):
    """More than two tiles for every pair, so that both accumulators are used again, with one K step (the issuer
    runs ahead of the epilogue) and a few; the switch asks for pairs where the rule would not."""
    monkeypatch.setenv("ABOLETH_GEMM_PAIR", "1" if width == 256 else "2")
    assert _choice(kind, m, n, k) == (0 if width == 256 else -1, 2)
    assert -(-m // 256) * -(-n // width) > 2 * 74
    _dense_case(kind, m, n, k)
    monkeypatch.setenv("ABOLETH_GEMM_PAIR", "0")
    assert _choice(kind, m, n, k)[0] > 0
    _dense_case(kind, m, n, k)


@pytest.mark.parametrize("k", [128, 384])
def test_grouped_pair_loops_with_several_tiles_per_pair(k):
    """The same for the grouped products: 17 row tiles x 16 column tiles on 74 pairs, ragged last row tiles."""
    from aboleth_b200.ops import check_gemm_status, grouped_gemm_bf16, grouped_gemm_e4m3_mx, pack_scales_mx

    n, fp8 = 4096, torch.float8_e4m3fn
    counts = torch.tensor([1000, 1281, 897, 640], dtype=torch.int32, device="cuda")
    tiles = int(((counts + 255) // 256).sum()) * n // 256
    assert tiles > 3 * 74
    padded = (counts + 127) // 128 * 128
    offsets = (torch.cumsum(padded, 0) - padded).to(torch.int32)
    rows = int(padded.sum())
    g = torch.Generator(device="cuda").manual_seed(k)
    a = torch.randint(-2, 3, (rows, k), generator=g, device="cuda").float()
    w = torch.randint(-2, 3, (4, n, k), generator=g, device="cuda").float()
    a_s = torch.exp2(torch.randint(-2, 3, (rows, k // 128), generator=g, device="cuda").float())
    w_s = torch.exp2(torch.randint(-2, 3, (4, n // 128, k // 128), generator=g, device="cuda").float())
    plain = grouped_gemm_bf16(a.bfloat16(), w.bfloat16(), counts, offsets)
    scaled = torch.full((rows, n), 7.0, dtype=torch.bfloat16, device="cuda")
    grouped_gemm_e4m3_mx(a.to(fp8), pack_scales_mx(a_s, rows, k, weight=False), w.to(fp8),
                         pack_scales_mx(w_s.view(-1, k // 128), 4 * n, k, weight=True), counts, offsets, scaled)
    torch.cuda.synchronize()
    check_gemm_status("cuda")
    a_full = a * a_s.repeat_interleave(128, dim=1)
    for e in range(4):
        live = slice(int(offsets[e]), int(offsets[e]) + int(counts[e]))
        w_full = w[e] * w_s[e].repeat_interleave(128, dim=0).repeat_interleave(128, dim=1)
        assert torch.equal(plain[live], (a[live] @ w[e].t()).to(torch.bfloat16))
        assert torch.equal(scaled[live], (a_full[live] @ w_full.t()).to(torch.bfloat16))
        assert bool((scaled[live.stop:int(offsets[e]) + int(padded[e])] == 7.0).all())


def _split_case(kind, m, n, k, nt, split):
    """One product of small integers through the split kernel: every partial sum is exact, so the result is the fp32
    product rounded once, whatever the tile and however K is cut."""
    from aboleth_b200.ops import check_gemm_status, pack_scales_mx
    from aboleth_b200.ops._kernels import call, ptr, stream_ptr
    from aboleth_b200.ops.gemm import gemm_status

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randint(-2, 3, (m, k), generator=g, device="cuda").float()
    b = torch.randint(-2, 3, (n, k), generator=g, device="cuda").float()
    dtype = torch.bfloat16 if kind == 0 else torch.float8_e4m3fn
    a_full, b_full, packed_a, packed_b = a, b, None, None
    if kind == 2:
        a_s = torch.exp2(torch.randint(-2, 3, (m, k // 128), generator=g, device="cuda").float())
        b_s = torch.exp2(torch.randint(-2, 3, (-(-n // 128), k // 128), generator=g, device="cuda").float())
        a_full = a * a_s.repeat_interleave(128, dim=1)
        b_full = b * b_s.repeat_interleave(128, dim=0)[:n].repeat_interleave(128, dim=1)
        packed_a, packed_b = pack_scales_mx(a_s, m, k, weight=False), pack_scales_mx(b_s, n, k, weight=True)
    a, b = a.to(dtype), b.to(dtype)
    out = torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
    call("ab_gemm_split", kind, ptr(a), ptr(b), ptr(out), ptr(packed_a), ptr(packed_b), m, n, k, k, k, n, 0.5, nt,
         split, ptr(gemm_status(a.device)), stream_ptr())
    torch.cuda.synchronize()
    check_gemm_status("cuda")
    assert torch.equal(out[:m], (0.5 * (a_full @ b_full.t())).to(torch.bfloat16)), (kind, m, n, k, nt, split)
    assert bool((out[m] == 7.0).all())


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("m,n,k", [(1, 8, 128), (33, 1000, 640), (64, 136, 1152), (129, 520, 896), (300, 264, 2048)])
def test_split_gemm_is_exact_on_integers_for_every_tile_and_split(kind, m, n, k):
    """Token tiles with one row, one row over, ragged weight tiles, K steps that do not divide by the split."""
    for nt in (32, 64, 128, 256):
        if kind == 2 and nt < 128 and m > nt:
            continue
        for split in range(1, min(8, k // (64 if kind == 0 else 128)) + 1):
            _split_case(kind, m, n, k if kind else k + 8, nt, split)


@pytest.mark.parametrize("kind", ["bf16", "e4m3"])
@pytest.mark.parametrize("m", [1, 31, 32, 33, 64, 65, 128, 129, 256, 257, 700, 1500])
def test_dense_gemm_agrees_across_its_dispatch(kind, m):
    """Row counts around the edges of the token tiles, in a strided output."""
    from aboleth_b200.ops import check_gemm_status, gemm_bf16, gemm_e4m3

    n, k = 1160, 1040
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randint(-2, 3, (m, k), generator=g, device="cuda").float()
    b = torch.randint(-2, 3, (n, k), generator=g, device="cuda").float()
    dtype = torch.bfloat16 if kind == "bf16" else torch.float8_e4m3fn
    wide = torch.full((m, n + 64), 7.0, dtype=torch.bfloat16, device="cuda")
    (gemm_bf16 if kind == "bf16" else gemm_e4m3)(a.to(dtype), b.to(dtype), wide[:, :n])
    torch.cuda.synchronize()
    check_gemm_status("cuda")
    assert torch.equal(wide[:, :n], (a @ b.t()).to(torch.bfloat16)) and bool((wide[:, n:] == 7.0).all())


@pytest.mark.parametrize("counts", [[129, 0, 1, 1153], [256, 512, 255, 513], [129, 0, 1, 770], [256, 512, 255, 257]])
@pytest.mark.parametrize("n", [128, 640])
def test_grouped_pair_tiles_at_their_edges(counts, n):
    """Experts just over and under a 256-row pair tile, one with a single row, one column tile that is half full:
    small integers are exact in both operand types.  (At most one tile per pair here.)"""
    from aboleth_b200.ops import check_gemm_status, grouped_gemm_bf16, grouped_gemm_e4m3_mx, pack_scales_mx
    from aboleth_b200.ops._kernels import call_rc

    experts, k = len(counts), 256
    counts = torch.tensor(counts, dtype=torch.int32, device="cuda")
    padded = (counts + 127) // 128 * 128
    offsets = (torch.cumsum(padded, 0) - padded).to(torch.int32)
    rows = int(padded.sum())
    assert call_rc("ab_grouped_pairs", rows, experts) == (rows // experts > 384)   # the last two: the one-CTA loops
    g = torch.Generator(device="cuda").manual_seed(37)
    a = torch.randint(-2, 3, (rows, k), generator=g, device="cuda").float()
    w = torch.randint(-2, 3, (experts, n, k), generator=g, device="cuda").float()
    a_s = torch.exp2(torch.randint(-2, 3, (rows, k // 128), generator=g, device="cuda").float())
    w_s = torch.exp2(torch.randint(-2, 3, (experts, n // 128, k // 128), generator=g, device="cuda").float())
    fp8 = torch.float8_e4m3fn
    plain = torch.full((rows, n), 7.0, dtype=torch.bfloat16, device="cuda")
    scaled = plain.clone()
    for _ in range(3):
        grouped_gemm_bf16(a.bfloat16(), w.bfloat16(), counts, offsets, plain)
        grouped_gemm_e4m3_mx(a.to(fp8), pack_scales_mx(a_s, rows, k, weight=False), w.to(fp8),
                             pack_scales_mx(w_s.view(-1, k // 128), experts * n, k, weight=True), counts, offsets, scaled)
    torch.cuda.synchronize()
    check_gemm_status("cuda")
    a_full = a * a_s.repeat_interleave(128, dim=1)
    for e in range(experts):
        lo, cnt, end = int(offsets[e]), int(counts[e]), int(offsets[e]) + int(padded[e])
        w_full = w[e] * w_s[e].repeat_interleave(128, dim=0).repeat_interleave(128, dim=1)
        assert torch.equal(plain[lo:lo + cnt], (a[lo:lo + cnt] @ w[e].t()).to(torch.bfloat16))
        assert torch.equal(scaled[lo:lo + cnt], (a_full[lo:lo + cnt] @ w_full.t()).to(torch.bfloat16))
        assert bool((plain[lo + cnt:end] == 7.0).all()) and bool((scaled[lo + cnt:end] == 7.0).all())


@pytest.mark.parametrize("m,n,k", [(9472, 512, 200), (9400, 448, 200), (700, 4000, 72)])
def test_pair_tiles_of_both_widths_are_exact_on_integers(m, n, k):
    """37 x 2 tiles of 256 columns fill the device once where 224 columns need a second wave; 448 = 2 x 224; 4000
    columns end inside a narrow tile.  K ends inside a step."""
    from aboleth_b200.ops import check_gemm_status, gemm_bf16

    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randint(-2, 3, (m, k), generator=g, device="cuda").float()
    b = torch.randint(-2, 3, (n, k), generator=g, device="cuda").float()
    out = gemm_bf16(a.bfloat16(), b.bfloat16())
    torch.cuda.synchronize()
    check_gemm_status("cuda")
    assert torch.equal(out, (a @ b.t()).to(torch.bfloat16))


def test_chained_launches_see_what_the_kernels_before_them_wrote():
    """Quantise, pack and multiply in a row, with nothing waiting in between, over buffers that the next round
    overwrites: the results are those of the same calls with a synchronisation after each, also when the chain is captured
    in a graph and when another stream runs one at the same time."""
    from aboleth_b200.ops import gemm_bf16, gemm_e4m3_mx, pack_scales_mx, quant_fp8

    m, n, k = 257, 640, 512
    g = torch.Generator(device="cuda").manual_seed(41)
    w = torch.randn(n, k, generator=g, device="cuda").to(torch.float8_e4m3fn)
    back = (torch.randn(k, n, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    w_packed = pack_scales_mx(torch.full((n // 128, k // 128), 0.0625, device="cuda"), n, k, weight=True)
    x0 = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)

    def chain(x, y, wait):
        for _ in range(6):
            q, scales = quant_fp8(x, round_scale=True)
            wait()
            packed = pack_scales_mx(scales, m, k, weight=False)
            wait()
            gemm_e4m3_mx(q, packed, w, w_packed, y)
            wait()
            gemm_bf16(y, back, x)
            wait()

    def buffers():
        return x0.clone(), torch.zeros(m, n, dtype=torch.bfloat16, device="cuda")

    want, y = buffers()
    chain(want, y, torch.cuda.synchronize)
    got, y = buffers()
    chain(got, y, lambda: None)
    side = torch.cuda.Stream()
    other, y_other = buffers()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        chain(other, y_other, lambda: None)
    again, y_again = buffers()
    chain(again, y_again, lambda: None)
    torch.cuda.synchronize()
    graphed, y_graphed = buffers()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(graphed, y_graphed, lambda: None)
    graphed.copy_(x0)
    graph.replay()
    torch.cuda.synchronize()
    for result in (got, other, again, graphed):
        assert torch.equal(result, want)


@pytest.mark.parametrize("m,n", [(1000, 8192), (905, 8136)])
def test_block_scaled_pair_loop_back_to_back(m, n):
    """Quantise, pack and multiply on two input sets in turn, with no wait in between, at sizes whose product takes the
    CTA-pair loop with two tiles for most pairs (4 x 32 tiles on 74 pairs), ragged in both directions the second time.
    The activations are small integers and the weights' scales powers of two: the product is exact, so the outputs are
    the fp32 product rounded once."""
    from aboleth_b200.ops import check_gemm_status, gemm_e4m3_block_scaled, pack_scales_mx, quant_fp8

    k, fp8 = 1024, torch.float8_e4m3fn
    g = torch.Generator(device="cuda").manual_seed(m)
    b_s = torch.exp2(torch.randint(-2, 3, (-(-n // 128), k // 128), generator=g, device="cuda").float())
    b = torch.randint(-2, 3, (n, k), generator=g, device="cuda").float()
    packed = pack_scales_mx(b_s, n, k, weight=True)
    full = b * b_s.repeat_interleave(128, dim=0)[:n].repeat_interleave(128, dim=1)
    sets, want = [], []
    for _ in range(2):
        x = torch.randint(-7, 8, (m, k), generator=g, device="cuda").float()
        sets.append(x.to(torch.bfloat16))
        want.append((x @ full.t()).to(torch.bfloat16))
    b, got = b.to(fp8), []
    for i in range(40):
        q, scales = quant_fp8(sets[i % 2], round_scale=True)
        out = gemm_e4m3_block_scaled(q, scales, b, b_s, b_packed=packed)
        if i >= 36:
            got.append(out)
    torch.cuda.synchronize()
    check_gemm_status("cuda")
    for i, out in enumerate(got):
        assert torch.equal(out, want[i % 2])
