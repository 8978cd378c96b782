"""GPU parity of the tcgen05 GEMM (eb_gemm) against an fp32 reference of the same product.

Tolerance: operands are fp16/bf16 and accumulation is fp32, so the only error against the
fp32 product of the same rounded operands is the final rounding of the output (half an ulp
of the output type, relative 2^-11 for fp16 and 2^-8 for bf16) plus fp32 summation-order
noise; the test allows 2x that."""
import pytest
import torch

pytestmark = pytest.mark.gpu

REL = {torch.float16: 2 ** -10, torch.bfloat16: 2 ** -7, torch.float32: 1e-5}


def reference(a, w, bias=None, act=None, residual=None):
    y = a.float() @ w.float().t()
    if bias is not None:
        y = y + bias.float()
    if act == "relu":
        y = torch.relu(y)
    elif act == "gelu_tanh":
        y = torch.nn.functional.gelu(y, approximate="tanh")
    elif act == "gelu":
        y = torch.nn.functional.gelu(y)
    if residual is not None:
        y = y + residual.float()
    return y


def check_close(out, ref, dtype):
    assert out.shape == ref.shape
    err = (out.float() - ref).abs()
    bound = REL[dtype] * ref.abs() + 2e-4 * ref.abs().max().clamp_min(1e-3)
    bad = err > bound
    assert not bad.any(), f"max err {err.max().item():.4g} at {int(bad.sum())} elements (ref max {ref.abs().max().item():.4g})"


def status_ok():
    from energonai_b200.gemm import device_status
    st = device_status()
    assert st[0] == 0, f"device status {st}"


SHAPES = [
    (256, 256, 64), (128 + 1, 8, 8), (300, 520, 200), (1024, 1024, 1024), (2048, 768, 3072), (640, 15360 // 8, 5120),
    (4096, 5120, 640), (1000, 2056, 264),
    # decode orientation (M <= 128): one weight pass split over all SMs
    (1, 256, 128), (16, 256, 64), (16, 5120, 5120), (16, 2560, 5120), (8, 1536, 12288), (64, 1152, 9216),
    (33, 520, 200), (100, 1024, 1024), (128, 384, 512), (16, 8, 8),
]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_plain(M, N, K, dtype):
    from energonai_b200.gemm import gemm
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(dtype)
    out = gemm(a, w)
    torch.cuda.synchronize()
    status_ok()
    check_close(out, reference(a, w), dtype)
    out2 = gemm(a, w)                  # deterministic
    assert torch.equal(out, out2)


@pytest.mark.parametrize("M", [16, 512])
@pytest.mark.parametrize("act", [None, "relu", "gelu_tanh", "gelu"])
def test_gemm_epilogue(M, act):
    from energonai_b200.gemm import gemm
    N, K, dtype = 1024, 512, torch.float16
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(dtype)
    bias = torch.randn(N, device="cuda", generator=g).to(dtype)
    res = torch.randn(M, N, device="cuda", generator=g).to(dtype)
    out = gemm(a, w, bias=bias, act=act, residual=res)
    check_close(out, reference(a, w, bias, act, res), dtype)
    out32 = gemm(a, w, bias=bias, act=act, out_dtype=torch.float32)
    assert out32.dtype == torch.float32
    check_close(out32, reference(a, w, bias, act), torch.float32)
    status_ok()


@pytest.mark.parametrize("rows", [1, 48])
def test_gemm_writes_into_a_cache_view(rows):
    """Row m of the result lands at [m // rows, pos + m % rows, col0:col0+N] of a
    [batch, max_len, width] cache, leaving everything else untouched."""
    from energonai_b200.gemm import gemm
    B, max_len, width, N, K, pos, col0 = 5, 64, 96, 64, 128, 7, 16
    dtype = torch.float16
    a = torch.randn(B * rows, K, device="cuda").to(dtype)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(dtype)
    cache = torch.full((B, max_len, width), 3.0, device="cuda", dtype=dtype)
    view = cache[:, pos:, col0:]
    gemm(a, w, out=view, out_rows_per_batch=rows, out_batch_stride=cache.stride(0), out_ld=cache.stride(1))
    ref = reference(a, w).view(B, rows, N)
    check_close(cache[:, pos:pos + rows, col0:col0 + N], ref, dtype)
    keep = torch.ones_like(cache, dtype=torch.bool)
    keep[:, pos:pos + rows, col0:col0 + N] = False
    assert (cache[keep] == 3.0).all()


def test_gemm_strided_operand_and_linear_api():
    from energonai_b200.gemm import gemm
    from energonai_b200.kernel import linear, find_algo
    big = torch.randn(300, 1024, device="cuda").half()
    a = big[:, 256:768]                            # row stride 1024, K = 512
    w = (torch.randn(264, 512, device="cuda") * 0.05).half()
    check_close(gemm(a, w), reference(a, w), torch.float16)
    x = torch.randn(4, 16, 512, device="cuda").half()
    y = linear(x, w, find_algo())
    assert y.shape == (4, 16, 264)
    check_close(y.view(-1, 264), reference(x.view(-1, 512), w), torch.float16)


def test_linear_reference_fixture_tolerance():
    """tests/test_kernel/test_linear_func.py:7-29: [16,64,12288] x [49152,12288] fp16 against
    F.linear with the reference's own pass criteria."""
    from energonai_b200.kernel import linear
    inputs = torch.randn(16, 64, 12288, device="cuda").half()
    params = torch.randn(49152, 12288, device="cuda").half()
    target = torch.nn.functional.linear(inputs, params)
    out = linear(inputs, params)
    diff = (out - target).abs()
    assert diff.mean() <= 0.5 and diff.max() <= 15 and diff.max() / target.max() <= 0.05


def test_gemm_rejects_bad_arguments():
    from energonai_b200.gemm import gemm
    a = torch.randn(16, 12, device="cuda").half()
    w = torch.randn(8, 12, device="cuda").half()
    with pytest.raises(RuntimeError, match="multiples of 8"):
        gemm(a, w)
    with pytest.raises(RuntimeError):
        gemm(a.float(), w.float())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("act", [None, "relu"])
@pytest.mark.parametrize("M,N,K", [(16, 5120, 5120), (1, 256, 128), (16, 1920, 5120), (32, 1024, 768), (5, 520, 200),
                                   (16, 8, 8), (20, 2560, 1024)])
def test_gemm_ln_fold(M, N, K, act, dtype):
    """LayerNorm folded into the GEMM (eb_gemm_ln) against LayerNorm -> projection in fp32.

    Tolerance: besides the rounding of the output, the folded weights W * gamma are rounded to
    the operand type once more (relative 2^-11 / 2^-8 per weight, averaging out over K), while the
    normalised activations are NOT rounded as they are on the two-kernel path; the bound is
    twice the plain GEMM's."""
    from energonai_b200.gemm import gemm, fold_layernorm
    from energonai_b200.kernel.cuda_native.layer_norm import layer_norm_forward
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + 7 * K)
    x = (torch.randn(M, K, device="cuda", generator=g) * 2.0 + 0.7).to(dtype)
    x[:, 0] += 6.0                                             # an outlier column, as residual streams have
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(dtype)
    b = torch.randn(N, device="cuda", generator=g).to(dtype)
    gamma = (1 + 0.2 * torch.randn(K, device="cuda", generator=g)).to(dtype)
    beta = (0.2 * torch.randn(K, device="cuda", generator=g)).to(dtype)
    r = torch.randn(M, N, device="cuda", generator=g).to(dtype)
    eps = 1e-5
    w_f, colsum, bias32 = fold_layernorm(w, b, gamma, beta)
    out = gemm(x, w_f, act=act, residual=r, static_weight=True, ln_fold=(colsum, bias32, eps))
    torch.cuda.synchronize()
    status_ok()
    xn = torch.nn.functional.layer_norm(x.float(), (K,), gamma.float(), beta.float(), eps)
    ref = xn @ w.float().t() + b.float()
    if act == "relu":
        ref = torch.relu(ref)
    ref = ref + r.float()
    err = (out.float() - ref).abs()
    bound = 2 * REL[dtype] * ref.abs() + 4e-4 * ref.abs().max().clamp_min(1e-3) + 2 * REL[dtype] * (xn.abs() @ w.float().abs().t()) / K ** 0.5
    assert not (err > bound).any(), f"max err {err.max().item():.4g} (ref max {ref.abs().max().item():.4g})"
    # and against the two-kernel path, which rounds the normalised activations
    two = gemm(layer_norm_forward(x, gamma, beta, eps), w, bias=b, act=act, residual=r)
    tol = {torch.float16: 4e-3, torch.bfloat16: 3e-2}[dtype]
    row_err = (out.float() - two.float()).abs().amax(-1)
    assert (row_err <= tol * two.float().abs().amax(-1).clamp_min(1e-3)).all(), row_err.max().item()
    assert torch.equal(out, gemm(x, w_f, act=act, residual=r, static_weight=True, ln_fold=(colsum, bias32, eps)))


def test_gemm_ln_fold_rejects_wide_batches():
    from energonai_b200.gemm import gemm, fold_layernorm
    x = torch.zeros(33, 64, device="cuda", dtype=torch.float16)
    w = torch.zeros(64, 64, device="cuda", dtype=torch.float16)
    ones = torch.ones(64, device="cuda", dtype=torch.float16)
    w_f, colsum, bias32 = fold_layernorm(w, None, ones, ones)
    with pytest.raises(RuntimeError):
        gemm(x, w_f, ln_fold=(colsum, bias32, 1e-5))


# Few rows against small weights (one CTA per 16 weight rows, its warps splitting K): batch rows around the
# multiples of 8, K below one slice, with an empty last slice and not a multiple of 32, N not a multiple of 16, more
# tiles than CTAs, and both sides of the sizes up to which that form is taken.
STEP_SHAPES = [(1, 8, 8), (7, 40, 40), (8, 5000, 264), (9, 768, 776), (16, 24, 3072), (17, 1000, 2056), (32, 520, 520), (31, 2048, 2048), (32, 2056, 2048),
               (1, 16392, 4096), (8, 4104, 4096), (16, 2048, 4096), (16, 4112, 2048), (3, 50257, 64)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", STEP_SHAPES)
def test_gemm_few_rows(M, N, K, dtype):
    """Every epilogue; the folded LayerNorm with a row mean of several standard deviations (its single-pass sums are
    fp32: 1e-5 of the row maximum, as REL has it, and the mean times the column sum on top, hence 1e-4)."""
    from energonai_b200.gemm import fold_layernorm, gemm, gemm_parts, project_unit
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w, b, res = rnd(M, K).to(dtype), (rnd(N, K) * K ** -0.5).to(dtype), rnd(N).to(dtype), rnd(M, N).to(dtype)
    plain = reference(x, w)
    check_close(gemm(x, w, bias=b, act="relu", residual=res, static_weight=True), reference(x, w, b, "relu", res), dtype)
    check_close(gemm(x, w, bias=b, out_dtype=torch.float32), plain + b.float(), torch.float32)
    # one row of a cache, its number on the device; nothing else is written, and nothing at all beyond the limit
    cache, row = torch.zeros(M, 3, N + 8, device="cuda", dtype=dtype), torch.tensor([1], dtype=torch.int32, device="cuda")
    where = dict(out=cache, out_rows_per_batch=1, out_batch_stride=cache.stride(0), out_ld=cache.stride(1), out_row_offset_device=row)
    gemm(x, w, out_row_limit=3, **where)
    check_close(cache[:, 1, :N], plain, dtype)
    assert not cache[:, [0, 2]].any() and not cache[:, 1, N:].any()
    status_ok()
    if N % 16 == 0:
        gate, up = plain.view(M, N // 16, 2, 8).unbind(2)
        check_close(project_unit(x, w, "geglu"), (torch.nn.functional.gelu(gate, approximate="tanh") * up).reshape(M, N // 2), dtype)
    if N % 8 == 0 and N > 16:
        out, tail = gemm_parts(x, w, bias=b, tail_col=N - 8)
        check_close(out, (plain + b.float())[:, :N - 8], dtype)
        check_close(tail, (plain + b.float())[:, N - 8:], torch.float32)
    shifted, gamma, beta = (x.float() + 3).to(dtype), (torch.rand(K, device="cuda", generator=g) + 0.5).to(dtype), rnd(K).to(dtype)
    folded, colsum, bias32 = fold_layernorm(w, b, gamma, beta)
    got = gemm(shifted, folded, ln_fold=(colsum, bias32, 1e-5), out_dtype=torch.float32, static_weight=True)
    want = torch.nn.functional.layer_norm(shifted.double(), (K,)) @ folded.double().t() + bias32.double()
    assert float((got - want).abs().max()) < 1e-4 * float(want.abs().max())
    status_ok()


# Tiles of 256 rows per pair of SMs: narrow and wide, few and many waves (16 and 8 epilogue warps); a last row tile of one row and with an
# empty second half, N ending inside a tile and a chunk, K below a k-block, with an odd number of k-blocks and not a multiple of 64.
PAIR_SHAPES = [(257, 8200, 72), (513, 2056, 776), (5000, 4112, 8), (700, 3088, 840), (6000, 2064, 136), (2300, 4112, 2120)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", PAIR_SHAPES)
def test_gemm_pair_tiles(M, N, K, dtype):
    from energonai_b200.gemm import gemm, gemm_parts, project_unit
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w, b, res = rnd(M, K).to(dtype), (rnd(N, K) * K ** -0.5).to(dtype), rnd(N).to(dtype), rnd(M, N).to(dtype)
    plain = reference(x, w)
    for act in ("relu", "gelu", "gelu_tanh"):
        check_close(gemm(x, w, bias=b, act=act), reference(x, w, b, act), dtype)
    # the result in place of the residual, as the blocks have it
    got = res.clone()
    gemm(x, w, bias=b, residual=got, out=got, static_weight=True)
    check_close(got, reference(x, w, b, None, res), dtype)
    check_close(gemm(x, w, bias=b, out_dtype=torch.float32), plain + b.float(), torch.float32)
    # batch rows of a cache, from a row on whose number is on the device; nothing else is written, and nothing at all beyond the limit
    batch = next(d for d in (4, 3, 2, 1) if M % d == 0)
    cache, row = torch.zeros(batch, M // batch + 2, N + 8, device="cuda", dtype=dtype), torch.tensor([1], dtype=torch.int32, device="cuda")
    gemm(x, w, out=cache, out_rows_per_batch=M // batch, out_batch_stride=cache.stride(0), out_ld=cache.stride(1), out_row_offset_device=row, out_row_limit=2)
    check_close(cache[:, 1:-1, :N].reshape(M, N), plain, dtype)
    assert not cache[:, [0, -1]].any() and not cache[:, :, N:].any()
    status_ok()
    if N % 16 == 0:
        gate, up = plain.view(M, N // 16, 2, 8).unbind(2)
        check_close(project_unit(x, w, "geglu"), (torch.nn.functional.gelu(gate, approximate="tanh") * up).reshape(M, N // 2), dtype)
    out, tail = gemm_parts(x, w, bias=b, tail_col=N - 24)
    check_close(out, (plain + b.float())[:, :N - 24], dtype)
    check_close(tail, (plain + b.float())[:, N - 24:], torch.float32)
    status_ok()


@pytest.mark.parametrize("M,N", [(1000, 4096), (3000, 6144)])
def test_gemm_pair_tiles_one_behind_the_other(M, N):
    """Launches that follow each other at once, with fewer k-blocks than the stages hold up to several rounds of them: whatever a stage's
    hand-back finds when a CTA has left, the next kernel's barriers would show."""
    from energonai_b200.gemm import gemm
    w, x = torch.randn(N, 840, device="cuda").half(), torch.randn(M, 840, device="cuda").half()
    for K in range(64, 841, 64):
        a, b = x[:, :K], w[:, :K]
        want = gemm(a, b, static_weight=True)
        check_close(want, reference(a, b), torch.float16)
        outs = [torch.empty_like(want) for _ in range(8)]
        for _ in range(4):
            for o in outs:
                gemm(a, b, out=o, static_weight=True)
        assert all(torch.equal(o, want) for o in outs)
        status_ok()


# A warp's slice of K above 256 columns: one column more, part of a second run, a whole one; rows in ones, eights, sixteens and thirty-twos.
@pytest.mark.parametrize("M,N,K", [(8, 520, 2056), (32, 520, 2304), (8, 1024, 3072), (2, 1024, 4096), (16, 1024, 4096)])
def test_gemm_few_rows_long_k(M, N, K):
    """No run of accumulations is longer than that of a K of 2048, so the sums are as close to 64 bits as those (3.5e-7, each
    accumulation truncating; 512 columns in one run: 6.4e-7).  And a row's sum does not depend on how many rows take this form."""
    from energonai_b200.gemm import gemm
    g = torch.Generator(device="cuda").manual_seed(K)
    x, w = torch.randn(M, K, device="cuda", generator=g).half(), (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).half()
    got, want = gemm(x, w, out_dtype=torch.float32), x.double() @ w.double().t()
    assert float((got - want).norm() / want.norm()) < 4e-7
    for m in (1, M // 2 + 1):
        assert torch.equal(gemm(x[-m:], w, out_dtype=torch.float32), got[-m:])
    status_ok()


# On the far side of the lines: 9 to 16 rows with more tiles than SMs and a K above 2048, up to 8 rows with many tiles of a short K.
@pytest.mark.parametrize("M,N,K", [(9, 2400, 2304), (16, 2720, 2816), (16, 2560, 3072), (8, 9488, 64), (1, 16384, 256), (8, 32768, 504)])
def test_gemm_few_rows_in_the_other_form(M, N, K):
    """These sizes are summed as the ones with 17 or more rows of as many weights are (in the tcgen05 form), bit for bit."""
    from energonai_b200.gemm import gemm
    g = torch.Generator(device="cuda").manual_seed(K)
    x, w = torch.randn(32, K, device="cuda", generator=g).half(), (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).half()
    both = gemm(x, w, out_dtype=torch.float32)
    assert torch.equal(gemm(x[:M], w, out_dtype=torch.float32), both[:M])
    check_close(both, reference(x, w), torch.float32)
    status_ok()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gemm_prompt_forms_agree(dtype):
    """The same rows in batches that take one-SM tiles of 32, 64, 128 and 256 columns and pair tiles of 128 and 256 with eight and sixteen epilogue
    warps: bit for bit the same results behind every epilogue, as the choice of a form claims."""
    from energonai_b200.gemm import gemm, project_unit
    for N, K, rows in ((1024, 4096, (64, 500, 1000, 2100, 4096, 9000)), (5120, 5120, (64, 333, 600, 777, 4100)), (50272, 768, (40, 130, 520, 1100)), (44912, 168, (65, 300, 900))):
        g = torch.Generator(device="cuda").manual_seed(N)
        rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
        w, b = (rnd(N, K) * K ** -0.5).to(dtype), rnd(N).to(dtype)
        x, res = rnd(max(rows), K).to(dtype), rnd(40, N).to(dtype)
        want = None
        for M in rows:
            a, r = x[:M], torch.zeros(M, N, device="cuda", dtype=dtype)
            r[:40] = res
            got = [gemm(a, w)[:40], gemm(a, w, bias=b, act="relu", residual=r)[:40], gemm(a, w, bias=b, act="gelu")[:40], gemm(a, w, bias=b, act="gelu_tanh")[:40],
                   gemm(a, w, bias=b, out_dtype=torch.float32)[:40], project_unit(a, w, "geglu")[:40]]
            want = got if want is None else want
            assert all(torch.equal(p, q) for p, q in zip(got, want)), (N, K, M)
    status_ok()
