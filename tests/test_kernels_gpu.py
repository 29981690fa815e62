"""Numerics of every native sm_100a kernel against a plain PyTorch fp32 reference of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def native():
    from jaxpp_b200.ops import native as n

    n.load()  # fails loudly if the library was not built
    yield n
    torch.cuda.synchronize()
    assert n.read_status() == 0, "a kernel reported a bounded-wait time-out or a bad argument"


def rnd(*shape, dtype=torch.bfloat16, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32) * scale).to(dtype)


def close(got, ref, rtol, atol):
    torch.testing.assert_close(got.float(), ref.float(), rtol=rtol, atol=atol)


GEMM_SHAPES = [
    (128, 256, 64), (256, 512, 128), (384, 768, 192), (130, 264, 72),  # ragged M/N/K tails
    (1024, 1600, 6400), (512, 11008, 4096), (2048, 4096, 5504), (64, 8, 8),
]


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
def test_gemm_forward_layout(native, M, N, K):
    x, w = rnd(M, K, scale=0.5), rnd(N, K, scale=0.5, seed=1)
    bias = rnd(N, seed=2)
    got = native.linear(x, w, bias)
    ref = x.float() @ w.float().t() + bias.float()
    close(got, ref, rtol=2e-2, atol=2e-2 * (K ** 0.5) * 0.25)
    torch.cuda.synchronize()
    assert native.read_status(clear=False) == 0


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES[:6])
def test_gemm_dgrad_layout(native, M, N, K):
    dy, w = rnd(M, N, scale=0.5), rnd(N, K, scale=0.5, seed=1)
    got = native.linear_dgrad(dy, w)
    ref = dy.float() @ w.float()
    close(got, ref, rtol=2e-2, atol=2e-2 * (N ** 0.5) * 0.25)


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES[:6])
def test_gemm_wgrad_layout_and_accumulate(native, M, N, K):
    dy, x = rnd(M, N, scale=0.5), rnd(M, K, scale=0.5, seed=1)
    got = native.linear_wgrad(dy, x)
    ref = dy.float().t() @ x.float()
    close(got, ref, rtol=2e-2, atol=2e-2 * (M ** 0.5) * 0.25)
    acc = torch.ones(N, K, dtype=torch.float32, device="cuda")
    native.linear_wgrad(dy, x, out=acc, accumulate=True)
    native.linear_wgrad(dy, x, out=acc, accumulate=True)
    close(acc, 1.0 + 2.0 * ref, rtol=2e-2, atol=4e-2 * (M ** 0.5) * 0.25)


# remainders in every dimension (N % 64 != 0 takes the unblocked MN-major copies); the forms of the kernel by name are below
@pytest.mark.parametrize("M,N,K", [(2056, 5000, 136), (4104, 1096, 264), (776, 1032, 1032), (520, 264, 72), (264, 136, 2056), (72, 4088, 4104),
                                   (8, 64, 512), (136, 8, 1544)])
@pytest.mark.parametrize("layout", ["f", "d", "w"])
def test_gemm_forms_at_tile_edges(native, M, N, K, layout):
    a = rnd(*((K, M) if layout == "w" else (M, K)), seed=61)
    b = rnd(*((N, K) if layout == "f" else (K, N)), seed=62)
    A, B = a.double().t() if layout == "w" else a.double(), b.double().t() if layout == "f" else b.double()
    ref = A @ B
    slack = K * 2.0 ** -23 * (A.abs() @ B.abs())          # fp32 sums of K products in any order
    run = lambda out, **kw: native.gemm(a, b, M, N, K, layout == "w", layout != "f", out, **kw)

    def check(got, want, rounding):
        bad = (got.double() - want).abs() > slack + rounding * want.abs() + 2.0 ** -23 * want.abs()
        assert not bad.any(), f"{int(bad.sum())} of {bad.numel()} elements are out of bounds"

    check(run(torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")), ref, 2.0 ** -8)
    check(run(torch.full((M, N), 3.0, dtype=torch.float32, device="cuda"), accumulate=True), ref + 3, 0.0)
    bias = rnd(N, seed=63)
    wide = torch.full((M, N + 3), 7.0, dtype=torch.float32, device="cuda")   # rows that TMA cannot store; neighbours untouched
    check(run(wide[:, :N], bias=bias), ref + bias.double(), 0.0)
    assert (wide[:, N:] == 7.0).all()
    torch.cuda.synchronize()
    assert native.read_status(clear=False) == 0


PAIR256, PAIR128, ONE256, ONE128, ONE64 = range(5)


def _assert_form(native, form, split, batch, M, N, K, counted=False):
    """(the choice goes by the number of CTAs and clusters that are resident at once: the shapes are for 148 SMs)"""
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        for out_fp32 in (0, 1):
            assert native.load().jpb_gemm_form(batch, M, N, K, out_fp32, int(counted), 0, 0, 0) == form + 16 * split


@pytest.mark.parametrize("form,split,batch,M,N,K", [
    (PAIR256, 1, 1, 1032, 2056, 1544), (PAIR128, 1, 1, 776, 1352, 4104), (ONE256, 1, 1, 1032, 2056, 72), (ONE128, 1, 1, 776, 1352, 72),
    (ONE64, 1, 1, 72, 8, 72), (ONE64, 2, 1, 136, 1032, 2056), (ONE64, 4, 1, 72, 8, 2056),
    # several problems in one launch: tiles that end in the next problem's rows
    (PAIR256, 1, 5, 136, 2056, 2048), (PAIR256, 1, 5, 776, 2056, 1024), (PAIR128, 1, 8, 392, 1032, 4096), (ONE256, 1, 8, 136, 2056, 64),
    (ONE128, 1, 5, 136, 1032, 64), (ONE64, 1, 2, 72, 136, 64), (ONE64, 2, 2, 136, 520, 2048), (ONE64, 4, 2, 72, 136, 2048)])
@pytest.mark.parametrize("layout", ["f", "d", "w"])
def test_every_gemm_form(native, form, split, batch, M, N, K, layout):
    """Ragged shapes in each form of the kernel, all layouts, against 64 bits: bf16 and accumulated fp32 results through TMA,
    and a result whose rows TMA cannot store.  Errors as in the test above."""
    _assert_form(native, form, split, batch, M, N, K)
    a = rnd(batch, *((K, M) if layout == "w" else (M, K)), seed=61)
    b = rnd(batch, *((N, K) if layout == "f" else (K, N)), seed=62)
    A, B = a.double(), b.double()
    A, B = A.transpose(1, 2) if layout == "w" else A, B.transpose(1, 2) if layout == "f" else B
    ref = A @ B
    slack = K * 2.0 ** -23 * (A.abs() @ B.abs())

    def run(out, accumulate=False):
        if batch == 1:
            return native.gemm(a[0], b[0], M, N, K, layout == "w", layout != "f", out[0], accumulate=accumulate)
        return native._gemm_batched(a, b, out, batch, M, N, K, layout == "w", layout != "f", accumulate=accumulate)

    def check(out, want, rounding):
        bad = (out.double() - want).abs() > slack + rounding * want.abs() + 2.0 ** -23 * want.abs()
        assert not bad.any(), f"{int(bad.sum())} of {bad.numel()} elements are out of bounds"

    out = torch.full((batch, M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    run(out)
    check(out, ref, 2.0 ** -8)
    out = torch.full((batch, M, N), 3.0, device="cuda")
    run(out, accumulate=True)
    check(out, ref + 3, 0.0)
    wide = torch.full((batch, M, N + 3), 7.0, device="cuda")      # neighbours untouched
    run(wide[:, :, :N])
    check(wide[:, :, :N], ref, 0.0)
    assert (wide[:, :, N:] == 7.0).all()
    torch.cuda.synchronize()
    assert native.read_status(clear=False) == 0


@pytest.mark.parametrize("form,batch,M,N,K,segs", [(PAIR256, 5, 776, 2056, 1024, 2), (PAIR256, 5, 776, 2056, 1024, 8), (PAIR128, 8, 392, 1032, 4096, 2),
                                                   (ONE256, 8, 136, 2056, 64, 2), (ONE128, 5, 136, 1032, 64, 1), (ONE64, 3, 72, 136, 64, 1)])
@pytest.mark.parametrize("layout", ["f", "d", "w"])
def test_every_gemm_form_with_row_counts(native, form, batch, M, N, K, segs, layout):
    """Groups that fill only the first rows of each segment: empty tiles of every height are skipped and written as zeros, or
    left alone when the result is added, and so are empty blocks of a reduction (layout w)."""
    _assert_form(native, form, 1, batch, M, N, K, counted=True)
    over_k = layout == "w"
    if over_k:
        segs = max(1, segs // 2)
    seg = (K if over_k else M) // segs
    counts = torch.randint(0, seg + 1, (batch, segs), generator=torch.Generator().manual_seed(9), dtype=torch.int32)
    counts[0], counts[1], counts[2, 0] = seg, 0, 1
    live = (torch.arange(seg)[None, None] < counts[:, :, None]).reshape(batch, seg * segs, 1).cuda()
    a = rnd(batch, *((K, M) if over_k else (M, K)), seed=61) * live
    b = rnd(batch, *((N, K) if layout == "f" else (K, N)), seed=62)
    A, B = a.double(), b.double()
    A, B = A.transpose(1, 2) if over_k else A, B.transpose(1, 2) if layout == "f" else B
    ref = A @ B
    slack = K * 2.0 ** -23 * (A.abs() @ B.abs())
    run = lambda out, acc: native._gemm_batched(a, b, out, batch, M, N, K, over_k, layout != "f", counts.cuda(), seg, over_k, acc)
    out = run(torch.full((batch, M, N), float("nan"), dtype=torch.bfloat16, device="cuda"), False)
    assert ((out.double() - ref).abs() <= slack + 2.0 ** -8 * ref.abs()).all()
    out = run(torch.full((batch, M, N), 3.0, device="cuda"), True)
    assert ((out.double() - ref - 3).abs() <= slack + 2.0 ** -23 * (ref + 3).abs()).all()
    torch.cuda.synchronize()
    assert native.read_status(clear=False) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,H", [(37, 256), (128, 1600), (64, 4096), (16, 8192)])
def test_norms(native, dtype, rows, H):
    from jaxpp_b200.ops import core as ops

    tol = dict(rtol=1e-4, atol=1e-4) if dtype == torch.float32 else dict(rtol=2e-2, atol=2e-2)
    x, w, b, dy = rnd(rows, H, dtype=dtype), rnd(H, dtype=dtype, seed=1), rnd(H, dtype=dtype, seed=2), rnd(rows, H, dtype=dtype, seed=3)
    y, rstd = native.rmsnorm(x, w, 1e-5)
    ry, rr = ops._rmsnorm_ref(x.float(), w.float(), 1e-5)
    close(y, ry, **tol)
    close(rstd, rr, rtol=1e-4, atol=1e-4)
    dx, dw = native.rmsnorm_bwd(dy, x, w, rstd)
    rdx, rdw = ops._rmsnorm_bwd_ref(dy.float(), x.float(), w.float(), rr)
    close(dx, rdx, **tol)
    close(dw, rdw, rtol=tol["rtol"], atol=tol["atol"] * rows ** 0.5)
    y, mean, rstd = native.layernorm(x, w, b, 1e-5)
    ry, rm, rr = ops._layernorm_ref(x.float(), w.float(), b.float(), 1e-5)
    close(y, ry, **tol)
    close(mean, rm, rtol=1e-4, atol=1e-4)
    dx, dw, db = native.layernorm_bwd(dy, x, w, mean, rstd)
    rdx, rdw, rdb = ops._layernorm_bwd_ref(dy.float(), x.float(), w.float(), rm, rr)
    close(dx, rdx, **tol)
    close(dw, rdw, rtol=tol["rtol"], atol=tol["atol"] * rows ** 0.5)
    close(db, rdb, rtol=tol["rtol"], atol=tol["atol"] * rows ** 0.5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_activations_rope_colsum(native, dtype):
    from jaxpp_b200.ops import core as ops

    tol = dict(rtol=1e-4, atol=1e-4) if dtype == torch.float32 else dict(rtol=2e-2, atol=2e-2)
    x, dy = rnd(33, 1024, dtype=dtype), rnd(33, 1024, dtype=dtype, seed=1)
    close(native.gelu(x), ops._gelu_ref(x.float()), **tol)
    close(native.gelu_bwd(dy, x), ops._gelu_bwd_ref(dy.float(), x.float()), **tol)
    gu, d2 = rnd(33, 2048, dtype=dtype, seed=2), rnd(33, 1024, dtype=dtype, seed=3)
    close(native.swiglu(gu), ops._swiglu_ref(gu.float()), **tol)
    close(native.swiglu_bwd(d2, gu), ops._swiglu_bwd_ref(d2.float(), gu.float()), **tol)
    close(native.colsum(x), x.float().sum(0), rtol=tol["rtol"], atol=tol["atol"] * 6)
    q = rnd(2, 16, 4, 128, dtype=dtype, seed=4)
    ang = torch.rand(16, 64, device="cuda") * 6.28
    cos, sin = ang.cos(), ang.sin()
    r = native.rope(q, cos, sin, False)
    close(r, ops._rope_ref(q.float(), cos, sin, False), **tol)
    close(native.rope(r, cos, sin, True), q, rtol=tol["rtol"] * 2, atol=tol["atol"] * 2)
    # fused split of a packed qkv projection (+ RoPE on q, k) and its transpose
    for hq, hkv, rope_on in ((4, 2, True), (3, 3, False)):
        packed = rnd(2, 16, hq + 2 * hkv, 128, dtype=dtype, seed=5)
        c, s_ = (cos, sin) if rope_on else (None, None)
        got = native.qkv_split(packed, c, s_, hq, hkv)
        ref = ops._qkv_split_ref(packed.float(), c, s_, hq, hkv)
        for g, r_ in zip(got, ref):
            assert g.is_contiguous()
            close(g, r_, **tol)
        merged = native.qkv_merge(*got, c, s_)
        close(merged, packed, rtol=tol["rtol"] * 2, atol=tol["atol"] * 2)  # merge inverts split
        close(merged, ops._qkv_merge_ref(*[g.float() for g in got], c, s_), **tol)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norm_backward_with_residual_add_rounds_like_two_kernels(native, dtype):
    """dx + add from one kernel must equal norm_bwd followed by a separate add bit for bit."""
    rows, H = 77, 1024
    x, dy, add = rnd(rows, H, dtype=dtype, seed=51), rnd(rows, H, dtype=dtype, seed=52), rnd(rows, H, dtype=dtype, seed=53)
    w, b = rnd(H, dtype=dtype, seed=54), rnd(H, dtype=dtype, seed=55)
    _, rstd = native.rmsnorm(x, w, 1e-5)
    dx, dw = native.rmsnorm_bwd(dy, x, w, rstd)
    dx2, dw2 = native.rmsnorm_bwd_add(dy, x, w, rstd, add)
    assert torch.equal(dx2, dx + add) and torch.equal(dw2, dw)
    _, mean, rstd = native.layernorm(x, w, b, 1e-5)
    dx, dw, db = native.layernorm_bwd(dy, x, w, mean, rstd)
    dx2, dw2, db2 = native.layernorm_bwd_add(dy, x, w, mean, rstd, add)
    assert torch.equal(dx2, dx + add) and torch.equal(dw2, dw) and torch.equal(db2, db)


def test_narrow_linear_like_a_router(native):
    """A linear layer with 4 outputs (a small router): the narrow operands of its backward GEMMs are re-pitched."""
    x, w, dy = rnd(300, 256, seed=41), rnd(4, 256, scale=0.2, seed=42), rnd(300, 4, seed=43)
    close(native.linear(x, w, None), x.float() @ w.float().t(), rtol=2e-2, atol=0.1)
    close(native.linear_dgrad(dy, w), dy.float() @ w.float(), rtol=2e-2, atol=0.05)
    close(native.linear_wgrad(dy, x), dy.float().t() @ x.float(), rtol=2e-2, atol=0.5)
    acc = torch.ones(4, 256, dtype=torch.float32, device="cuda")
    native.linear_wgrad(dy, x, out=acc, accumulate=True)
    close(acc, 1 + dy.float().t() @ x.float(), rtol=2e-2, atol=0.5)


@pytest.mark.parametrize("E,M,N,K", [(3, 192, 320, 256), (2, 200, 264, 128), (4, 64, 128, 64)])
def test_grouped_gemm_equal_groups(native, E, M, N, K):
    """One launch over all groups against per-group fp32 matmuls, in the three linear-layer layouts.  Group sizes
    that are not multiples of the tile make tiles straddle two groups: the masked rows / columns must not leak."""
    x, w = rnd(E, M, K, seed=31), rnd(E, N, K, scale=0.2, seed=32)
    dy = rnd(E, M, N, seed=33)
    close(native.linear_batched(x, w), torch.bmm(x.float(), w.float().transpose(1, 2)), rtol=2e-2, atol=2e-2 * K ** 0.5 * 0.2)
    if N % 64 == 0:
        close(native.linear_dgrad_batched(dy, w), torch.bmm(dy.float(), w.float()), rtol=2e-2, atol=2e-2 * N ** 0.5 * 0.2)
    else:
        close(native.linear_dgrad_batched(dy, w), torch.bmm(dy.float(), w.float()), rtol=2e-2, atol=2e-2 * N ** 0.5 * 0.2)
    ref_w = torch.bmm(dy.float().transpose(1, 2), x.float())
    close(native.linear_wgrad_batched(dy, x, torch.float32), ref_w, rtol=2e-2, atol=2e-2 * M ** 0.5)
    close(native.linear_wgrad_batched(dy, x), ref_w, rtol=2e-2, atol=3e-2 * M ** 0.5)


@pytest.mark.parametrize("E,seg,segs,N,K", [(3, 200, 2, 320, 256), (2, 384, 1, 512, 128), (4, 80, 4, 256, 64)])
def test_grouped_gemm_unequal_groups(native, E, seg, segs, N, K):
    from jaxpp_b200.utils import config

    with config.moe_skip_empty_slots.set(2):   # row counts used by all three GEMMs
        _grouped_gemm_unequal_groups(native, E, seg, segs, N, K)


def _grouped_gemm_unequal_groups(native, E, seg, segs, N, K):
    """Groups of different sizes inside equal-sized storage: each group's rows are ``segs`` segments of ``seg`` rows
    with a filled prefix (given in ``counts``) and zeros behind it.  Skipping what holds no data must not change any
    of the three products; entirely empty groups and segments, full ones and ones that end inside a tile are covered,
    and the output of skipped tiles must be written (zeros), not left as it was."""
    M = seg * segs
    if M % 64:
        M = None
    g = torch.Generator().manual_seed(7)
    counts = torch.randint(0, seg + 1, (E, segs), generator=g, dtype=torch.int32)
    counts[0, 0] = seg          # a full segment
    counts[-1] = 0              # a group without any data
    if E > 2:
        counts[1, -1] = 1       # a single row
    live = (torch.arange(seg)[None, None, :] < counts[:, :, None]).reshape(E, seg * segs, 1).cuda()
    counts = counts.cuda()
    rows = seg * segs
    x = rnd(E, rows, K, seed=51) * live
    dy = rnd(E, rows, N, seed=52) * live
    w = rnd(E, N, K, scale=0.2, seed=53)
    # outputs are fresh allocations: leave NaNs in the block that the caching allocator hands out next
    junk = torch.full((E, rows, max(N, K)), float("nan"), dtype=torch.bfloat16, device="cuda")
    del junk
    y = native.linear_batched(x, w, counts, seg)
    assert torch.isfinite(y.float()).all()
    close(y, torch.bmm(x.float(), w.float().transpose(1, 2)), rtol=2e-2, atol=2e-2 * K ** 0.5 * 0.2)
    junk = torch.full((E, rows, max(N, K)), float("nan"), dtype=torch.bfloat16, device="cuda")
    del junk
    dx = native.linear_dgrad_batched(dy, w, counts, seg)
    assert torch.isfinite(dx.float()).all()
    close(dx, torch.bmm(dy.float(), w.float()), rtol=2e-2, atol=2e-2 * N ** 0.5 * 0.2)
    if M is not None:
        ref_w = torch.bmm(dy.float().transpose(1, 2), x.float())
        junk = torch.full((E, N, K), float("nan"), dtype=torch.float32, device="cuda")
        del junk
        dw = native.linear_wgrad_batched(dy, x, torch.float32, counts, seg)
        assert torch.isfinite(dw).all()
        close(dw, ref_w, rtol=2e-2, atol=2e-2 * rows ** 0.5)
        assert dw[-1].abs().max().item() == 0.0      # the empty group's gradient is exactly zero
        close(native.linear_wgrad_batched(dy, x, None, counts, seg), ref_w, rtol=2e-2, atol=3e-2 * rows ** 0.5)
        # as a gradient sink: added onto an fp32 accumulator in the epilogue (empty groups leave it alone)
        from jaxpp_b200.ops import sink

        acc = torch.ones(E, N, K, dtype=torch.float32, device="cuda")
        got = sink.accumulate(torch.ops.b200.linear_wgrad_batched.default, acc, dy, x, torch.float32, counts, seg)
        assert got is acc
        close(acc, 1.0 + ref_w, rtol=2e-2, atol=2e-2 * rows ** 0.5)
        assert (acc[-1] == 1.0).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_router_kernel(native, dtype):
    from jaxpp_b200.parallel import moe
    import jaxpp_b200 as jp

    for T, E, k in ((1000, 8, 2), (77, 16, 4)):
        logits = rnd(T, E, dtype=dtype, seed=21)
        with jp.MpmdMesh.create({"mpmd": 1, "data": 1, "model": 1}, kind="cuda", multi_process=False):
            top_i, w, probs, hits = torch.ops.b200moe.router(logits, k)
        r_i, r_w, r_p, r_h = moe._route_ref(logits, k)
        close(probs, r_p, rtol=1e-4, atol=1e-6)
        assert torch.equal(top_i.sort(-1).values, r_i.sort(-1).values)
        close(w.sort(-1).values, r_w.sort(-1).values, rtol=1e-4, atol=1e-6)
        assert torch.equal(hits, r_h)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,E,k,C,d", [(1000, 8, 2, 256, 512), (77, 16, 4, 8, 40), (3000, 64, 1, 40, 264), (1, 4, 2, 8, 8), (1025, 4, 3, 800, 4096)])
def test_moe_row_kernels_match_the_composition(native, T, E, k, C, d, dtype):
    """Slots, dispatch, combination and their gradients as kernels against the index ops they stand for: slots, copies and
    scaled copies are the same bits, sums over at most k (or d) fp32 products differ by their rounding."""
    from jaxpp_b200.parallel import moe

    g = torch.Generator().manual_seed(5)
    top_i = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)]).cuda()
    dest, _, counts = moe.slots_and_counts(top_i, E, C)
    d2, inv, c2 = torch.ops.b200moe.slots(top_i, E, C)
    assert torch.equal(dest, d2) and torch.equal(counts, c2)
    x, y, go = rnd(T, d, dtype=dtype, seed=81), rnd(E * C, d, dtype=dtype, seed=82), rnd(T, d, dtype=dtype, seed=83)
    w = torch.rand(T * k, generator=g).cuda()
    buf = torch.ops.b200moe.dispatch_rows(x, dest, inv, k)
    assert torch.equal(buf.view(E, C, d), moe.dispatch(x, dest, E, C, k))
    half = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22
    yd = torch.cat([y, y.new_zeros(1, d)]).double()
    want = (yd[dest].view(T, k, d) * w.double().view(T, k, 1)).sum(1)
    slack = (yd[dest].abs().view(T, k, d) * w.double().view(T, k, 1)).sum(1) * k * 2.0 ** -23
    assert ((torch.ops.b200moe.combine_rows(y, dest, inv, w, k).double() - want).abs() <= slack + half * want.abs()).all()
    dy, dw = torch.ops.b200moe.combine_rows_bwd(go, y, dest, inv, w, k)
    rows = (go.float().repeat_interleave(k, 0) * w[:, None]).to(dtype)
    ref = torch.zeros(E * C + 1, d, dtype=dtype, device="cuda")
    ref[dest] = rows
    assert torch.equal(dy, ref[:-1])
    prod = yd[dest] * go.double().repeat_interleave(k, 0)
    assert ((dw.double() - prod.sum(-1)).abs() <= d * 2.0 ** -23 * prod.abs().sum(-1)).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,E,k", [(1000, 8, 2), (65, 5, 1), (130, 17, 8), (33, 64, 3)])
def test_route_tokens_kernel_matches_the_composition(native, T, E, k, dtype):
    from jaxpp_b200.parallel import moe

    logits = rnd(T, E, dtype=dtype, seed=91)
    gw = torch.rand(T, k, device="cuda")
    ti, w, probs, hits, aux = torch.ops.b200moe.route_tokens(logits, k)
    lg = logits.double().requires_grad_(True)
    p = torch.softmax(lg, -1)
    pv = p.gather(1, ti)
    rw = pv / pv.sum(-1, keepdim=True)
    raux = E * (hits.double() / (T * k) * p.mean(0)).sum()
    assert torch.equal(ti.sort(-1).values, torch.topk(logits.float(), k).indices.sort(-1).values)
    assert torch.equal(hits, torch.bincount(ti.reshape(-1), minlength=E).float())
    close(w, rw.float(), rtol=1e-5, atol=1e-6)
    close(aux, raux.float(), rtol=1e-5, atol=1e-6)
    (want,) = torch.autograd.grad((rw * gw).sum() + 3.0 * raux, [lg])
    got = torch.ops.b200moe.route_tokens_bwd(ti, probs, hits, gw, None, torch.tensor(3.0, device="cuda"), logits)
    bound = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5
    assert (got.double() - want).norm() <= bound * want.norm()


@pytest.mark.parametrize("T,E,k", [(1, 3, 1), (8192, 8, 2), (12000, 16, 2), (40000, 64, 8)])
def test_load_balancing_loss_repeats_and_is_summed_in_trees(native, T, E, k):
    """The same bits on every run, and no long chain of additions: a CTA's 64 tokens in 6 steps, a thread's share of the CTAs'
    rows (2048 / E of them at a time, at most 4 x ceil(rows / (4 * 1024 / E')) with E' = E rounded up), 2 + 10 steps between
    threads, 3 roundings of the products; every term is positive, so each step adds at most 2^-24 of the result."""
    logits = rnd(T, E, seed=93)
    run = lambda: torch.ops.b200moe.route_tokens(logits, k)
    _, _, probs, hits, aux = run()
    for _ in range(30):
        assert torch.equal(run()[4], aux)
    want = E / (T * k * T) * (hits.double() * probs.double().sum(0)).sum()
    steps = 6 + -(-(-(-T // 64)) // (1024 // (1 << (E - 1).bit_length()))) + 2 + 10 + 3
    assert abs(aux.double() - want) <= steps * 2.0 ** -24 * want


@pytest.mark.parametrize("rows", [128, 250, 256])
def test_parameter_sums_are_added_in_trees(native, rows):
    """One large row among small ones, each row a partial sum of its own: at most 2 + 2 + 5 additions (within a thread, of its
    four sums, between 32 threads) have the large value as an operand, and each loses at most half a unit in its last place."""
    x = torch.full((rows, 64), 0.125, device="cuda")
    x[0] = 2.0 ** 24
    want = 2.0 ** 24 + (rows - 1) / 8
    assert ((native.colsum(x).double() - want).abs() <= 9 * 1.0).all()


@pytest.mark.parametrize("layer", [False, True])
@pytest.mark.parametrize("rows,H", [(2400, 1600), (9500, 256), (4737, 4096), (300, 8192)])
def test_norm_backward_over_many_rows(native, layer, rows, H):
    """More CTAs than two per SM, CTAs with unequal numbers of rows: against 64 bits, everything rounded once to bf16
    (2^-9) after fp32 arithmetic."""
    x, w, dy = rnd(rows, H, seed=1), rnd(H, seed=2), rnd(rows, H, seed=3)
    xd, g = x.double(), dy.double() * w.double()
    mean = xd.mean(-1, keepdim=True) if layer else torch.zeros(rows, 1, dtype=torch.float64, device="cuda")
    rstd = ((xd - mean).pow(2).mean(-1, keepdim=True) + 1e-5).rsqrt()
    xh = (xd - mean) * rstd
    want = [(g - (g.mean(-1, keepdim=True) if layer else 0) - xh * (g * xh).mean(-1, keepdim=True)) * rstd, (dy.double() * xh).sum(0)]
    m, r = mean.float().reshape(-1), rstd.float().reshape(-1)
    got = native.layernorm_bwd(dy, x, w, m, r) if layer else native.rmsnorm_bwd(dy, x, w, r)
    if layer:
        want.append(dy.double().sum(0))
    for a, b in zip(got, want):
        assert (a.double() - b).norm() <= 2.0 ** -8 * b.norm()


def test_embedding_gradient_into_any_accumulator(native):
    """Repeated tokens, and an accumulator that does not start on a 16-byte boundary (no vector reductions there)."""
    ids = torch.randint(0, 7, (500,), generator=torch.Generator().manual_seed(2)).cuda()
    dy = rnd(500, 24, seed=5)
    want = torch.zeros(7, 24, dtype=torch.float64, device="cuda").index_add_(0, ids, dy.double())
    slack = 500 * 2.0 ** -23 * torch.zeros_like(want).index_add_(0, ids, dy.double().abs())
    for offset in (0, 1):
        acc = torch.ones(7 * 24 + 4, device="cuda")[offset:offset + 7 * 24].view(7, 24)
        native.embedding_bwd(dy, ids, 7, torch.float32, out=acc, accumulate=True)
        assert ((acc.double() - 1 - want).abs() <= slack + 2.0 ** -20).all()


def test_sum_squares_over_many_tensors(native):
    """More tensors than one launch takes, of both types, single elements, chunk edges and an unaligned view."""
    ts = [rnd(n, dtype=dt, seed=n) for n in (1, 3, 32768, 32769, 100003) for dt in (torch.float32, torch.bfloat16)]
    ts += [rnd(1000, dtype=torch.float32, seed=7)[1:]] + [rnd(10 + i, dtype=torch.float32, seed=i) for i in range(50)]
    want = sum(t.double().pow(2).sum() for t in ts)
    assert abs(native.sum_squares(ts).double() - want) <= 1e-5 * want   # chains of fewer than 160 fp32 additions


@pytest.mark.parametrize("n,offset", [(1, 0), (3, 0), (1027, 0), (4096, 0), (1026, 1)])
@pytest.mark.parametrize("gdt", [torch.float32, torch.bfloat16])
def test_adamw_with_clip_coefficient(native, n, offset, gdt):
    """Whole and partial vectors, unaligned state, the clipping coefficient as a value on the device, in place or not."""
    from jaxpp_b200.ops import core as ops

    make = lambda seed: rnd(n + offset, dtype=torch.float32, seed=seed)[offset:]
    p, m, v, g = make(1), make(2), make(3).abs(), make(4).to(gdt)
    step, clip = torch.tensor(7, device="cuda"), torch.tensor(0.37, device="cuda")
    for c in (clip, None):
        args = (step, 1e-2, 0.9, 0.95, 1e-8, 0.1, 0.5, torch.bfloat16)
        want = ops._adamw_ref(p.double(), g.double(), m.double(), v.double(), *args, None, False, c)
        state = [t.clone() for t in (p, m, v)]
        got = native.adamw(state[0], g, state[1], state[2], *args, None, offset == 0, c)
        for a, b in zip(got[:3], want[:3]):
            close(a, b.float(), rtol=1e-5, atol=1e-6)
        assert torch.equal(got[3], got[0].to(torch.bfloat16))


@pytest.mark.parametrize("n", [(1 << 17) - 1, 1 << 17, (1 << 17) + 3])
def test_adamw_gives_the_same_bits_at_either_width(native, n):
    """Four elements per access from 2^17 elements on, one below and where a tensor is not on a 16-byte boundary."""
    args = (torch.tensor(7, device="cuda"), 1e-2, 0.9, 0.95, 1e-8, 0.1, 0.5, torch.bfloat16)
    results = []
    for offset in (0, 1):
        p, g, m, v = (torch.cat([torch.zeros(offset, device="cuda"), rnd(n, dtype=torch.float32, seed=s)])[offset:] for s in (1, 2, 3, 4))
        results.append(native.adamw(p, g, m, v.abs_(), *args, None, True))
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("vocab,d,n", [(8200, 1032, 700), (9000, 1024, 1), (70000, 128, 3000)])
def test_embedding_gradient_of_a_bf16_table(native, vocab, d, n):
    """Lists of tokens per id: ids that occur once, never and hundreds of times, more than one CTA per row, out of range;
    a table of its own and an accumulator.  One fp32 chain per element, rounded to bf16 (2^-9)."""
    g = torch.Generator().manual_seed(3)
    ids = torch.randint(0, vocab, (n,), generator=g)
    ids[: n // 2] = 17
    if n > 100:
        ids[5], ids[6] = -1, vocab
    ids, dy = ids.cuda(), rnd(n, d, seed=6)
    ok = (ids >= 0) & (ids < vocab)
    want = torch.zeros(vocab, d, dtype=torch.float64, device="cuda").index_add_(0, ids[ok], dy[ok].double())
    slack = n * 2.0 ** -23 * torch.zeros_like(want).index_add_(0, ids[ok], dy[ok].double().abs())
    got = native.embedding_bwd(dy, ids, vocab)
    assert got.dtype == torch.bfloat16 and ((got.double() - want).abs() <= slack + 2.0 ** -8 * want.abs()).all()
    acc = rnd(vocab, d, seed=7)
    expected = acc.float() + got.float()         # what adding the gradient as a tensor gives, but for the order of the sums
    native.embedding_bwd(dy, ids, vocab, out=acc, accumulate=True)
    assert ((acc.float() - expected).abs() <= 2.0 ** -7 * (expected.abs() + got.float().abs()) + 1e-6).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_dropout_matches_counter_based_reference(native, dtype):
    from jaxpp_b200.ops import core as ops

    x = rnd(37, 129, dtype=dtype, seed=11)   # odd element count: the last Philox block is partial
    seed = torch.tensor(0x1234567812345, dtype=torch.int64, device="cuda")
    for p_drop, offset in ((0.1, 0), (0.5, 3), (0.0, 9)):
        got = native.dropout(x, p_drop, seed, offset)
        ref = ops._dropout_ref(x, p_drop, seed, offset)
        assert torch.equal(got == 0, ref == 0), "mask differs from the Philox reference"
        close(got, ref.float(), rtol=1e-2 if dtype == torch.bfloat16 else 1e-6, atol=1e-6)
    drop = (native.dropout(torch.ones(1 << 20, device="cuda"), 0.3, seed, 1) == 0).float().mean().item()
    assert abs(drop - 0.3) < 5e-3


@pytest.mark.parametrize("n,d", [(127, 8200), (128, 8200), (129, 1000), (192, 1032), (20000, 520)])
def test_embedding_gradient_of_long_token_lists(native, n, d):
    """Lists at the edges of the segments that they are cut into, two long ones behind each other and short ones between."""
    vocab = 1100
    ids = torch.randint(0, 64, (n + 40,), generator=torch.Generator().manual_seed(4))
    ids[20:20 + n] = 70
    ids = torch.cat([ids, torch.full((150,), 71), torch.full((5,), -1), torch.full((300,), 72)]).cuda()
    dy = rnd(ids.numel(), d, seed=8)
    ok = ids >= 0
    want, size = (torch.zeros(vocab, d, dtype=torch.float64, device="cuda").index_add_(0, ids[ok], t) for t in (dy[ok].double(), dy[ok].double().abs()))
    for out in (torch.full((vocab, d), float("nan"), dtype=torch.bfloat16, device="cuda"), torch.ones(vocab, d, dtype=torch.bfloat16, device="cuda")):
        accumulate = not bool(out.isnan().any())
        native.embedding_bwd(dy, ids, vocab, out=out, accumulate=accumulate)
        # chains of at most 128 rows and n / 64 segments in fp32, rounded to bf16 (and once more where it is added to 1)
        slack = (128 + n / 64) * 2.0 ** -24 * size + 2.0 ** -8 * (want.abs() + accumulate * (1 + want).abs())
        assert ((out.double() - want - float(accumulate)).abs() <= slack).all()


def test_embedding_gradient_does_not_wait_for_a_dominant_token(native):
    """A batch that is 90 % padding costs about what a batch of different tokens does (measured 1.6 times that; as one
    chain of rows it took fifty times as long)."""
    vocab, d, n = 32000, 4096, 16384
    ids = torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(4)).cuda()
    padded = ids.clone()
    padded[n // 10:] = 3
    dy = rnd(n, d, seed=8)

    def best(tokens):
        times = []
        for _ in range(6):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            native.embedding_bwd(dy, tokens, vocab)
            end.record()
            end.synchronize()
            times.append(start.elapsed_time(end))
        return min(times[1:])

    assert best(padded) < 3 * best(ids)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_embedding_and_cross_entropy(native, dtype):
    from jaxpp_b200.ops import core as ops

    tol = dict(rtol=1e-4, atol=1e-4) if dtype == torch.float32 else dict(rtol=2e-2, atol=2e-2)
    vocab, d = 1000, 256
    table = rnd(vocab, d, dtype=dtype)
    ids = torch.randint(0, vocab, (4, 77), device="cuda")
    assert torch.equal(native.embedding(ids, table), table[ids])
    dy = rnd(4, 77, d, dtype=dtype, seed=1)
    close(native.embedding_bwd(dy, ids, vocab), ops._emb_bwd_ref(dy.float(), ids, vocab), **tol)
    # the fp32 form (no cast pass) and the accumulating form that a microbatch loop's gradient sink uses
    ref32 = ops._emb_bwd_ref(dy.float(), ids, vocab, torch.float32)
    got32 = native.embedding_bwd(dy, ids, vocab, torch.float32)
    assert got32.dtype == torch.float32
    close(got32, ref32, rtol=1e-5, atol=1e-5)
    acc = torch.full_like(ref32, 0.5)
    assert native.embedding_bwd(dy, ids, vocab, out=acc, accumulate=True) is acc
    native.embedding_bwd(dy, ids, vocab, out=acc, accumulate=True)
    close(acc, 0.5 + 2 * ref32, rtol=1e-5, atol=1e-5)
    for V in (32000, 50257, 1000):
        logits = rnd(19, V, dtype=dtype, scale=3.0, seed=2)
        labels = torch.randint(0, V, (19,), device="cuda")
        loss, lse = native.cross_entropy(logits, labels)
        rl, rlse = ops._ce_ref(logits.float(), labels)
        close(loss, rl, rtol=1e-4, atol=1e-3)
        close(lse, rlse, rtol=1e-4, atol=1e-3)
        dl = torch.rand(19, device="cuda")
        got = native.cross_entropy_bwd(dl, logits, labels, lse)
        close(got, ops._ce_bwd_ref(dl, logits.float(), labels, rlse), rtol=tol["rtol"], atol=1e-3)


@pytest.mark.parametrize("gdtype", [torch.float32, torch.bfloat16])
def test_adamw(native, gdtype):
    from jaxpp_b200.ops import core as ops

    n = 100003
    p, g = rnd(n, dtype=torch.float32), rnd(n, dtype=gdtype, seed=1)
    m, v = rnd(n, dtype=torch.float32, scale=0.1, seed=2), rnd(n, dtype=torch.float32, scale=0.1, seed=3).abs()
    step = torch.tensor(3, device="cuda")
    args = (1e-3, 0.9, 0.95, 1e-8, 0.1, 0.5)
    got = native.adamw(p, g, m, v, step, *args, torch.bfloat16)
    ref = ops._adamw_ref(p, g, m, v, step, *args, torch.bfloat16)
    for a, b in zip(got[:3], ref[:3]):
        close(a, b, rtol=1e-5, atol=1e-6)
    close(got[3], ref[3], rtol=1e-2, atol=1e-2)


def test_ops_dispatch_to_native_and_autograd(native):
    """The b200:: ops route CUDA tensors to the native kernels and differentiate through them."""
    from jaxpp_b200.ops import core as ops

    x = rnd(256, 512).requires_grad_()
    w = rnd(1024, 512, scale=0.05, seed=1).requires_grad_()
    g = rnd(512, seed=2).requires_grad_()
    h = ops.rmsnorm(x, g, 1e-5)[0]
    y = ops.swiglu(ops.linear(h, w, None))
    y.float().pow(2).mean().backward()
    xr, wr, gr = (t.detach().float().requires_grad_() for t in (x, w, g))
    hr = ops._rmsnorm_ref(xr, gr, 1e-5)[0]
    yr = ops._swiglu_ref(hr @ wr.t())
    yr.pow(2).mean().backward()
    close(y, yr, rtol=3e-2, atol=3e-2)
    close(x.grad, xr.grad, rtol=5e-2, atol=2e-3)
    close(w.grad, wr.grad, rtol=5e-2, atol=2e-3)
    close(g.grad, gr.grad, rtol=5e-2, atol=5e-3)


ATTN_CASES = [
    # B, Sq, Sk, H, Hkv, D, causal
    (2, 256, 256, 4, 4, 64, True),
    (1, 512, 512, 4, 2, 128, True),
    (2, 384, 384, 2, 2, 128, False),
    (1, 200, 200, 2, 1, 64, True),   # ragged sequence: masks past the end of K and padded query rows
    (1, 1024, 1024, 8, 2, 128, True),
    # different query and key lengths: what ring attention's zigzag layout and any cached-key use call
    (1, 512, 256, 4, 2, 128, False),   # all queries against half as many keys
    (2, 256, 512, 4, 4, 64, False),    # half the queries against all keys
    (1, 256, 640, 4, 2, 128, True),    # causal with an offset: query i sees keys up to i + (Sk - Sq)
    (1, 200, 328, 2, 2, 64, True),     # the same, ragged
]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Sq,Sk,H,Hkv,causal", [
    (1, 1, 513, 2, 2, True), (2, 10, 10, 4, 2, True), (1, 129, 129, 2, 1, True), (1, 257, 640, 2, 2, False),
    (1, 300, 100, 2, 2, True),      # the first 200 queries see no key at all
    (3, 100, 300, 6, 2, True), (1, 769, 769, 4, 1, True), (9, 128, 128, 3, 3, False)])
def test_flash_attention_at_block_edges(native, B, Sq, Sk, H, Hkv, causal, D):
    """Pairs of query tiles of which one is empty or short, single and odd numbers of blocks, fully hidden rows, against
    64 bits.  P and dS are rounded to bf16 before the second products (2^-9 each) and the results once more, so each
    result is within 3 * 2^-8 of its 2-norm; the log-sum-exp is all fp32."""
    _check_attention(native, B, Sq, Sk, H, Hkv, causal, D)


def _check_attention(native, B, Sq, Sk, H, Hkv, causal, D):
    q, k, v, do = rnd(B, Sq, H, D, seed=71), rnd(B, Sk, Hkv, D, seed=72), rnd(B, Sk, Hkv, D, seed=73), rnd(B, Sq, H, D, seed=74)
    scale, G = D ** -0.5, H // Hkv
    o, lse = native.attention(q, k, v, causal, scale)
    got = native.attention_bwd(do, q, k, v, o, lse, causal, scale)
    Q, K, V, dO = q.double(), k.double().repeat_interleave(G, 2), v.double().repeat_interleave(G, 2), do.double()
    s = torch.einsum("bqhd,bkhd->bhqk", Q, K) * scale
    if causal:
        s = s.masked_fill(torch.arange(Sk, device="cuda")[None, :] > torch.arange(Sq, device="cuda")[:, None] + (Sk - Sq), float("-inf"))
    rlse = torch.logsumexp(s, -1)
    p = torch.exp(s - rlse[..., None]).nan_to_num(0.0)
    ro = torch.einsum("bhqk,bkhd->bqhd", p, V)
    ds = p * (torch.einsum("bqhd,bkhd->bhqk", dO, V) - (dO * ro).sum(-1).transpose(1, 2)[..., None]) * scale
    fold = lambda t: t.view(B, Sk, Hkv, G, D).sum(3)
    want = (torch.einsum("bhqk,bkhd->bqhd", ds, K), fold(torch.einsum("bhqk,bqhd->bkhd", ds, Q)), fold(torch.einsum("bhqk,bqhd->bkhd", p, dO)))
    assert torch.equal(torch.isfinite(lse), torch.isfinite(rlse))
    close(lse[torch.isfinite(rlse)], rlse[torch.isfinite(rlse)].float(), rtol=1e-5, atol=1e-5)
    for a, b in ((o, ro), *zip(got, want)):
        assert (a.double() - b).norm() <= 3 * 2.0 ** -8 * b.norm()
    torch.cuda.synchronize()
    assert native.read_status(clear=False) == 0


# grids with more pairs of tiles than SMs take two tiles per CTA, smaller ones the two halves of one tile
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("halves,B,Sq,Sk,H,Hkv,causal", [
    (0, 70, 250, 506, 4, 2, True), (0, 80, 130, 391, 4, 4, False), (0, 100, 300, 100, 2, 2, True), (0, 2, 128, 128, 4, 4, True),
    (0, 72, 200, 3, 2, 1, False), (1, 1, 1025, 1025, 4, 2, True), (1, 3, 129, 1153, 2, 2, False), (1, 2, 257, 129, 2, 1, True),
    (1, 1, 64, 193, 2, 2, False), (1, 1, 300, 257, 4, 4, True), (1, 2, 300, 100, 2, 1, True)])
def test_flash_attention_in_both_forms(native, halves, B, Sq, Sk, H, Hkv, causal, D):
    """Odd and even numbers of blocks (the halves keep two blocks of scores), last blocks with nothing in the second half, tiles
    behind the last query, rows that see no key."""
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert native.load().jpb_attention_fwd_halves(B, Sq, Sk, H, D, int(causal)) == halves
    _check_attention(native, B, Sq, Sk, H, Hkv, causal, D)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("where", ["first", "second", "both", "apart"])
def test_flash_attention_halves_rescale(native, D, where):
    """Scores whose maximum grows block by block in one half of the keys, in the other, or in both, or that are far lower in
    one half everywhere: each half rescales its sums on its own, and the halves meet with maxima far apart."""
    B, S, H = 1, 1280, 2
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert native.load().jpb_attention_fwd_halves(B, S, S, H, D, 1) == 1
    col = torch.arange(S, device="cuda")
    first, ramp = ((col % 128) < 64).float(), (1 + col // 128).float()
    gain = {"first": first * ramp, "second": (1 - first) * ramp, "both": ramp, "apart": 20 * first - 10}[where]
    q, v = rnd(B, S, H, D, seed=75).abs(), rnd(B, S, H, D, seed=77)
    k = (rnd(B, S, H, D, seed=76).float() * 0.3 + 0.5 * gain[None, :, None, None]).to(torch.bfloat16)
    o, lse = native.attention(q, k, v, True, D ** -0.5)
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) * D ** -0.5
    s = s.masked_fill(col[None, :] > col[:, None], float("-inf"))
    rlse = torch.logsumexp(s, -1)
    ro = torch.einsum("bhqk,bkhd->bqhd", torch.exp(s - rlse[..., None]), v.double())
    assert float((s[0, 0, -1].max() - s[0, 0, -1].min())) > 20      # far more than the 8 steps of log2 that move a maximum
    close(lse, rlse.float(), rtol=1e-5, atol=1e-5)
    assert (o.double() - ro).norm() <= 3 * 2.0 ** -8 * ro.norm()


@pytest.mark.parametrize("rows,H,per_sm", [(3000, 2048, 2), (6000, 1024, 4), (7200, 1024, 8), (3600, 1600, 4), (9000, 4096, 2)])
def test_norm_backward_gives_every_cta_six_rows(native, rows, H, per_sm):
    """(the numbers of rows are for 148 SMs)  The grid shows in the scratch, 2 H sums per CTA; the sums against 64 bits, rounded
    to bf16 once."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms == 148:
        assert native.load().jpb_norm_bwd_scratch_elems(rows, H) == max(sms * per_sm, min(rows, sms * 2)) * 2 * H
    x, w, dy = rnd(rows, H, seed=1), rnd(H, seed=2), rnd(rows, H, seed=3)
    rstd = (x.double().pow(2).mean(-1) + 1e-5).rsqrt().float()
    want = (dy.double() * x.double() * rstd.double()[:, None]).sum(0)
    dw = native.rmsnorm_bwd(dy, x, w, rstd)[1]
    slack = rows * 2.0 ** -23 * (dy.double() * x.double() * rstd.double()[:, None]).abs().sum(0)
    assert ((dw.double() - want).abs() <= 2.0 ** -8 * want.abs() + slack).all()


@pytest.mark.parametrize("B,Sq,Sk,H,Hkv,D,causal", ATTN_CASES)
def test_flash_attention_forward_backward(native, B, Sq, Sk, H, Hkv, D, causal):
    from jaxpp_b200.ops import attention as att
    from jaxpp_b200.ops import core as ops

    q, k, v = rnd(B, Sq, H, D, seed=1), rnd(B, Sk, Hkv, D, seed=2), rnd(B, Sk, Hkv, D, seed=3)
    do = rnd(B, Sq, H, D, seed=4)
    scale = D ** -0.5
    o, lse = att.attention_fwd(q, k, v, causal, scale)
    ro, rlse = ops._attn_ref(q.float(), k.float(), v.float(), causal, scale)
    close(o, ro, rtol=2e-2, atol=2e-2)
    close(lse, rlse, rtol=1e-3, atol=2e-3)
    dq, dk, dv = att.attention_bwd(do, q, k, v, o, lse, causal, scale)
    rdq, rdk, rdv = ops._attn_bwd_ref(do.float(), q.float(), k.float(), v.float(), ro, rlse, causal, scale)
    close(dq, rdq, rtol=3e-2, atol=3e-2)
    close(dk, rdk, rtol=3e-2, atol=3e-2 * (H // Hkv) ** 0.5)
    close(dv, rdv, rtol=3e-2, atol=3e-2 * (H // Hkv) ** 0.5)
    torch.cuda.synchronize()
    assert native.read_status(clear=False) == 0
