"""The contraction kernels alone, against float64 matrix products of the same operands, at sizes
other than any model's (odd row counts, feature counts that are no multiple of the tile, a
reduction length that is no multiple of the K-block)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(M, N, K, dtype, seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    a = (torch.randn(M, K, generator=g) * 0.5).to(dtype).cuda()
    w = (torch.randn(N, K, generator=g) * 0.5).to(dtype).cuda()
    return a, w


def _check(got, a, w, want, out_is_bf16):
    bound = (a.double().abs() @ w.double().abs().T).max().item()
    err = (got.double() - want).abs().max().item()
    tol = 2e-6 * bound + (want.abs().max().item() * 2 ** -8 if out_is_bf16 else 0.0)
    assert err <= tol, (err, tol)


@pytest.mark.parametrize("adt,wdt", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16),
                                     (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("M,N,K", [(1, 7, 5), (3, 200, 72), (70, 130, 257), (129, 65, 64),
                                   (16, 333, 1100), (9, 1000, 4096), (2, 31, 516),        # few rows: the weight-streaming kernel
                                   (17, 64, 64), (24, 192, 64), (39, 64, 192), (64, 256, 1024), (33, 130, 516), (64, 512, 516),      # small matrices by 16 rows, and the first above
                                   (300, 260, 1000), (65, 128, 36), (200, 129, 130)])    # many rows: 128 x 128 tiles
def test_gemm_generic(M, N, K, adt, wdt):
    from fastgguf_b200 import ops
    a, _ = _operands(M, N, K, adt, 1)
    _, w = _operands(M, N, K, wdt, 1)
    want = a.double() @ w.double().T
    got = ops.gemm_generic(a, w, out_dtype=torch.float32)
    _check(got, a, w, want, False)
    res = torch.randn(M, N, device="cuda")
    acc = res.clone()
    ops.gemm_generic(a, w, out=acc, accumulate=True)
    _check(acc, a, w, want + res.double(), False)
    if adt == torch.bfloat16:
        _check(ops.gemm_generic(a, w), a, w, want, True)
    # a row's result does not depend on the other rows of the step: alone, it gives the same bits
    if M > 1:
        alone = ops.gemm_generic(a[M - 1:M].contiguous(), w, out_dtype=torch.float32)
        if (M <= 16) == (1 <= 16):                       # the same kernel serves both row counts
            assert torch.equal(alone[0], got[M - 1])
        else:
            assert (alone[0] - got[M - 1]).abs().max() <= 1e-5 * got.abs().max()


@pytest.mark.parametrize("M", [1, 5, 16, 33, 64, 100, 300, 700])
@pytest.mark.parametrize("N,K", [(200, 72), (384, 2048), (1000, 520)])
def test_gemm_tc_epilogues(M, N, K):
    from fastgguf_b200.ops import fast_gemm
    a, w = _operands(M, N, K, torch.bfloat16, 2)
    want = a.double() @ w.double().T
    got = fast_gemm.gemm_tc(a, w, out_dtype=torch.float32)
    assert got is not None
    _check(got, a, w, want, False)
    _check(fast_gemm.gemm_tc(a, w), a, w, want, True)
    res = torch.randn(M, N, device="cuda")
    acc = res.clone()
    fast_gemm.gemm_tc(a, w, out=acc, accumulate=True)
    _check(acc, a, w, want + res.double(), False)
    assert fast_gemm.pipeline_error() == 0


@pytest.mark.parametrize("splits", [2, 4, 8])
@pytest.mark.parametrize("M,N,K", [(1, 256, 2048), (8, 200, 1096), (64, 384, 8192)])
def test_gemm_tc_split_k(M, N, K, splits):
    from fastgguf_b200.ops import fast_gemm
    a, w = _operands(M, N, K, torch.bfloat16, 3)
    want = a.double() @ w.double().T
    for _ in range(2):
        got = fast_gemm.gemm_tc(a, w, out_dtype=torch.float32, force_splits=splits)
        _check(got, a, w, want, False)
    res = torch.randn(M, N, device="cuda")
    acc = res.clone()
    fast_gemm.gemm_tc(a, w, out=acc, accumulate=True, force_splits=splits)
    _check(acc, a, w, want + res.double(), False)
    assert fast_gemm.pipeline_error() == 0


@pytest.mark.parametrize("M", [1, 9, 64, 130, 513])
@pytest.mark.parametrize("F,K", [(192, 64), (320, 72), (640, 2048)])
def test_gemm_tc_silu(M, F, K):
    from fastgguf_b200.ops import fast_gemm
    a, w = _operands(M, 2 * F, K, torch.bfloat16, 4)
    g = a.double() @ w[:F].double().T
    u = a.double() @ w[F:].double().T
    want = g / (1 + torch.exp(-g)) * u
    got = fast_gemm.gemm_tc(a, fast_gemm.interleave_gate_up(w[:F], w[F:]), silu=True)
    assert got is not None and got.dtype == torch.bfloat16
    bound = (a.double().abs() @ w.double().abs().T).max().item()
    err = (got.double() - want).abs().max().item()
    assert err <= want.abs().max().item() * 2 ** -8 + 1e-5 * bound * bound
    assert fast_gemm.pipeline_error() == 0


@pytest.mark.parametrize("splits", [2, 4, 8])
@pytest.mark.parametrize("M,F,K", [(1, 192, 2048), (9, 320, 1096), (64, 640, 2048), (40, 64, 4096)])
def test_gemm_tc_silu_split_k(M, F, K, splits):
    """Gate and up partial sums of a cluster's CTAs meet in the owner of the token column before the activation."""
    from fastgguf_b200.ops import fast_gemm
    a, w = _operands(M, 2 * F, K, torch.bfloat16, 14)
    g = a.double() @ w[:F].double().T
    u = a.double() @ w[F:].double().T
    want = g / (1 + torch.exp(-g)) * u
    got = fast_gemm.gemm_tc(a, fast_gemm.interleave_gate_up(w[:F], w[F:]), silu=True, force_splits=splits)
    bound = (a.double().abs() @ w.double().abs().T).max().item()
    err = (got.double() - want).abs().max().item()
    assert err <= want.abs().max().item() * 2 ** -8 + 1e-5 * bound * bound
    assert fast_gemm.pipeline_error() == 0


def test_gemm_tc_refuses_unaligned():
    from fastgguf_b200.ops import fast_gemm
    a, w = _operands(4, 32, 36, torch.bfloat16, 5)      # K % 8 != 0: TMA cannot describe the rows
    assert fast_gemm.gemm_tc(a, w) is None
    assert fast_gemm.plan_for_weight(w) is None


@pytest.mark.parametrize("M,N,K", [(513, 3072, 256), (700, 3000, 136), (300, 1152, 2048), (129, 2048, 512)])
def test_gemm_tc_prefill_tile_widths_and_started_norm(M, N, K):
    """Prefill shapes that pick 192-wide tiles (3072, 3000 and 1152 features), whole and ragged, and 256-wide ones;
    plain, residual add through the shared-memory tiles (N % 32 == 0) and row-wise (3000), with the next norm started."""
    from fastgguf_b200.ops import fast_gemm
    a, w = _operands(M, N, K, torch.bfloat16, 6)
    want = a.double() @ w.double().T
    _check(fast_gemm.gemm_tc(a, w, out_dtype=torch.float32), a, w, want, False)
    _check(fast_gemm.gemm_tc(a, w), a, w, want, True)
    res = torch.randn(M, N, device="cuda")
    nw = (1 + 0.1 * torch.randn(N, device="cuda")).float()
    acc = res.clone()
    out, started = fast_gemm.gemm_tc(a, w, out=acc, accumulate=True, emit_norm_weight=nw, emit_eps=1e-5)
    x = want + res.double()
    _check(acc, a, w, x, False)
    assert (started.xw.double() - x * nw.double()).abs().max().item() <= 2 ** -7 * (x * nw.double()).abs().max().item()
    ss = started.ss[:started.tiles].double().sum(0)
    assert ((ss - (x * x).sum(1)).abs() / (x * x).sum(1)).max().item() < 1e-4
    assert fast_gemm.pipeline_error() == 0


@pytest.mark.parametrize("width", [-2, -4])
@pytest.mark.parametrize("M,N,K", [(512, 512, 256), (300, 384, 2048), (700, 1000, 520), (129, 256, 72), (2048, 2048, 512), (513, 3072, 264)])
def test_gemm_tc_prefill_pair_of_ctas(M, N, K, width):
    """The kernel that puts a pair of CTAs on a 256 x 256 tile (width -2) or a 256 x 192 tile (-4) (forced here; the
    engine picks it for large shapes): whole and ragged tiles in every direction, every epilogue, the next norm started."""
    from fastgguf_b200.ops import fast_gemm
    a, w = _operands(M, N, K, torch.bfloat16, 8)
    want = a.double() @ w.double().T
    _check(fast_gemm.gemm_tc(a, w, out_dtype=torch.float32, force_splits=width), a, w, want, False)
    _check(fast_gemm.gemm_tc(a, w, force_splits=width), a, w, want, True)
    res = torch.randn(M, N, device="cuda")
    nw = (1 + 0.1 * torch.randn(N, device="cuda")).float()
    acc = res.clone()
    out, started = fast_gemm.gemm_tc(a, w, out=acc, accumulate=True, emit_norm_weight=nw, emit_eps=1e-5, force_splits=width)
    x = want + res.double()
    _check(acc, a, w, x, False)
    assert (started.xw.double() - x * nw.double()).abs().max().item() <= 2 ** -7 * (x * nw.double()).abs().max().item()
    ss = started.ss[:started.tiles].double().sum(0)
    assert ((ss - (x * x).sum(1)).abs() / (x * x).sum(1)).max().item() < 1e-4
    if N % 128 == 0 and width == -2:
        F = N // 2
        gate, up = w[:F], w[F:]
        got = fast_gemm.gemm_tc(a, fast_gemm.interleave_gate_up(gate, up), silu=True, force_splits=-2)
        g, u = a.double() @ gate.double().T, a.double() @ up.double().T
        ref = g / (1 + torch.exp(-g)) * u
        bound = (a.double().abs() @ w.double().abs().T).max().item()
        assert (got.double() - ref).abs().max().item() <= ref.abs().max().item() * 2 ** -8 + 1e-5 * bound * bound
    assert fast_gemm.pipeline_error() == 0


@pytest.mark.parametrize("M,N,K", [(200, 2048, 8192), (256, 512, 4096), (384, 1000, 2048), (130, 264, 4096)])
def test_gemm_tc_prefill_split_along_k(M, N, K):
    """A few hundred rows through a projection of few output tiles: partial products over slices of K on all SMs and a
    second kernel that adds them in order and applies the epilogue - plain, bfloat16, residual add with the next norm
    started, and with a norm on the input side whose 1/rms that kernel applies (its row sums in 5 and in 40 parts)."""
    from fastgguf_b200.ops import fast_gemm
    for epi in (fast_gemm.EPI_BF16, fast_gemm.EPI_F32, fast_gemm.EPI_ADD_F32):
        assert fast_gemm.workspace_bytes(M, N, K, epi) > 0               # the shapes are ones that the split takes
    assert fast_gemm.workspace_bytes(64, N, K, fast_gemm.EPI_F32) == 0   # the decode kernel's range
    assert fast_gemm.workspace_bytes(4096, 4096, K, fast_gemm.EPI_F32) == 0      # enough tiles
    a, w = _operands(M, N, K, torch.bfloat16, 9)
    want = a.double() @ w.double().T
    got = fast_gemm.gemm_tc(a, w, out_dtype=torch.float32)
    _check(got, a, w, want, False)
    whole = fast_gemm.gemm_tc(a, w, out_dtype=torch.float32, split_k=False)
    assert (got - whole).abs().max().item() <= 2e-6 * (a.double().abs() @ w.double().abs().T).max().item()
    _check(fast_gemm.gemm_tc(a, w), a, w, want, True)
    res = torch.randn(M, N, device="cuda")
    nw = (1 + 0.1 * torch.randn(N, device="cuda")).float()
    acc = res.clone()
    out, started = fast_gemm.gemm_tc(a, w, out=acc, accumulate=True, emit_norm_weight=nw, emit_eps=1e-5)
    x = want + res.double()
    _check(acc, a, w, x, False)
    assert started.tiles == (N + 127) // 128
    assert (started.xw.double() - x * nw.double()).abs().max().item() <= 2 ** -7 * (x * nw.double()).abs().max().item()
    ss = started.ss[:started.tiles].double().sum(0)
    assert ((ss - (x * x).sum(1)).abs() / (x * x).sum(1)).max().item() < 1e-4
    # a norm on the input side: rows x (float32) arrive as bf16(x * weight) with the sums of squares of x in parts
    g = torch.Generator(device="cpu").manual_seed(10)
    xin = (torch.randn(M, K, generator=g) * torch.linspace(0.2, 3.0, M)[:, None]).cuda()
    wn = (1 + 0.1 * torch.randn(K, generator=g)).cuda()
    xw = (xin * wn).to(torch.bfloat16)
    for parts in (5, 40):
        edges = torch.linspace(0, K, parts + 1).long().tolist()
        ss_in = torch.stack([(xin[:, lo:hi].double() ** 2).sum(1).float() for lo, hi in zip(edges[:-1], edges[1:])])
        d = fast_gemm.DeferredNorm(xw, ss_in.contiguous(), parts, K, 1e-5, xin, wn)
        inv = 1.0 / torch.sqrt((xin.double() ** 2).mean(1) + 1e-5)
        want_n = (xw.double() * inv[:, None]) @ w.double().T
        got_n = fast_gemm.gemm_tc(xw, w, out_dtype=torch.float32, deferred=d)
        bound = ((xw.double().abs() * inv[:, None]) @ w.double().abs().T).max().item()
        assert (got_n.double() - want_n).abs().max().item() <= 4e-6 * bound
    assert fast_gemm.pipeline_error() == 0


@pytest.mark.parametrize("M,N,K", [(17, 516, 512), (64, 700, 520), (65, 256, 512), (129, 1000, 2048), (257, 512, 8192), (300, 257, 1000), (700, 3072, 2048),
                                   (513, 2048, 4096), (32, 90000, 512), (90000, 256, 512)])     # the last two: planes made in two portions
def test_gemm_f32_on_planes(M, N, K):
    """float32 by three bfloat16 planes: no further from float64 than the plain chain of fused multiply-adds is."""
    from fastgguf_b200 import ops
    from fastgguf_b200.ops import fast_gemm
    a, w = _operands(M, N, K, torch.float32, 5)
    wide = torch.cat([a, torch.full((M, 4), 7.0, device="cuda")], 1)[:, :K]             # rows further apart than they are long
    want = a.double() @ w.double().T
    got = fast_gemm.gemm_f32(wide, w)
    plain = ops.gemm_generic(a, w, out_dtype=torch.float32)
    _check(got, a, w, want, False)
    assert (got.double() - want).norm() <= (plain.double() - want).norm()
    res = torch.randn(M, N, device="cuda")
    acc = res.clone()
    fast_gemm.gemm_f32(a, w, out=acc, accumulate=True)
    assert torch.equal(acc, got + res)                     # one rounding more, of the same sum
    into = torch.full((M, N + 3), 9.0, device="cuda")      # rows of the output that no vector store may touch
    fast_gemm.gemm_f32(a, w, out=into[:, 1:N + 1])
    assert torch.equal(into[:, 1:N + 1], got) and (into[:, 0] == 9).all() and (into[:, N + 1:] == 9).all()


@pytest.mark.parametrize("M,N,K", [(40, 520, 512), (300, 2048, 2048)])
def test_gemm_f32_on_planes_keeps_what_the_split_does_not_carry(M, N, K):
    """Infinities, NaN, magnitudes above bfloat16's largest and sums that overflow on the way give what the plain kernel gives."""
    from fastgguf_b200 import ops
    from fastgguf_b200.ops import fast_gemm
    a, w = _operands(M, N, K, torch.float32, 6)
    a[3, 7] = float("inf")
    a[5, 9] = float("nan")
    a[8, 11] = 3.4e38
    w[8] *= 1e-3
    a[20, 0], a[20, 300], w[:, 300] = 3e38, 3e38, -w[:, 0]
    w[17, 2] = float("-inf")
    got, plain = fast_gemm.gemm_f32(a, w), ops.gemm_generic(a, w, out_dtype=torch.float32)
    assert torch.equal(got.isnan(), plain.isnan()) and torch.equal(got.isinf(), plain.isinf())
    ok = plain.isfinite()
    inf = plain.isinf()
    assert inf.any() and torch.equal(got[inf], plain[inf])           # their signs
    scale = a.double().nan_to_num(0, 0, 0).abs() @ w.double().nan_to_num(0, 0, 0).abs().T
    assert ((got - plain).double().abs()[ok] <= 4e-6 * scale[ok]).all()


@pytest.mark.parametrize("M,N,K", [(40, 1000, 2048), (300, 515, 1024), (1000, 8200, 2048)])      # with parts and without, ragged tiles
def test_gemm_f32_on_planes_without_a_finite_number(M, N, K):
    """Outputs that the plain chain has to give are computed side by side: operands full of NaN take no more than ten times the plain kernel,
    and everything beside them keeps its bits."""
    from fastgguf_b200 import ops
    from fastgguf_b200.ops import fast_gemm
    a, w = _operands(M, N, K, torch.float32, 16)
    clean, res = fast_gemm.gemm_f32(a, w), torch.randn(M, N, device="cuda")
    rows, cols = torch.randperm(M)[:3], torch.randperm(N)[:2]
    some, ws = a.clone(), w.clone()
    some[rows, 5], ws[cols, 9] = float("nan"), float("inf")
    got, acc = fast_gemm.gemm_f32(some, ws), res.clone()
    fast_gemm.gemm_f32(some, ws, out=acc, accumulate=True)
    plain = ops.gemm_generic(some, ws, out_dtype=torch.float32)
    ok = plain.isfinite()
    assert torch.equal(got[~ok].isnan(), plain[~ok].isnan()) and torch.equal(got[~ok].sign().nan_to_num(), plain[~ok].sign().nan_to_num())
    assert torch.equal(got[ok], clean[ok]) and torch.equal(acc[ok], clean[ok] + res[ok]) and not acc[~ok].isfinite().any()
    nothing = torch.full_like(a, float("nan"))
    assert fast_gemm.gemm_f32(nothing, w).isnan().all()

    def us(f):
        f()
        t = []
        for _ in range(3):
            one, two = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            one.record()
            f()
            two.record()
            torch.cuda.synchronize()
            t.append(one.elapsed_time(two) * 1e3)
        return min(t)

    assert us(lambda: fast_gemm.gemm_f32(nothing, w)) < 10 * us(lambda: ops.gemm_generic(nothing, w, out_dtype=torch.float32))
    assert fast_gemm.pipeline_error() == 0


@pytest.mark.parametrize("M,N,K", [(40, 1000, 2048), (300, 515, 1024), (130, 2100, 12288)])
def test_gemm_f32_on_planes_over_float32s_range(M, N, K):
    """Operands far below bfloat16's smallest number times operands far above one, rows whose numbers lie 2^105 apart, sums below float32's
    normal numbers and sums above its largest: no further from float64 than the plain chain is, which carries all of it."""
    from fastgguf_b200 import ops
    from fastgguf_b200.ops import fast_gemm
    a, w = _operands(M, N, K, torch.float32, 26)
    g = torch.Generator().manual_seed(3)
    mixed = torch.exp2(torch.randint(-115, -9, (K,), generator=g).float()).cuda()
    down, up = 2.0 ** -115, 2.0 ** 105
    for x, y in ((a * down, w * up), (a * up, w * down), (a * 2.0 ** -100 * 2.0 ** -22, w * 2.0 ** 100), (a * mixed, w / mixed)):
        want = x.double() @ y.double().T
        got, plain = fast_gemm.gemm_f32(x, y), ops.gemm_generic(x, y, out_dtype=torch.float32)
        assert (got.double() - want).norm() <= (plain.double() - want).norm()
    x, y = a * 2.0 ** -80, w * 2.0 ** -62                  # sums of a few units of float32's smallest number
    want = x.double() @ y.double().T
    assert want.abs().max() < 2.0 ** -126
    assert (fast_gemm.gemm_f32(x, y).double() - want).abs().max() <= 0.75 * 2.0 ** -149 + 2.0 ** -22 * want.abs().max()
    x, y = a * 2.0 ** 70, w * 2.0 ** 57                    # around float32's largest number: what overflows on the way there does so here
    got, plain = fast_gemm.gemm_f32(x, y), ops.gemm_generic(x, y, out_dtype=torch.float32)
    assert torch.equal(got, plain) or torch.equal(got.nan_to_num(7.0), plain.nan_to_num(7.0))
    assert plain.isinf().any() or plain.isnan().any()
    x, y, clean = a.clone(), w.clone(), fast_gemm.gemm_f32(a, w)     # a few such rows among ordinary ones, whose outputs keep their bits
    x[M // 3] *= down
    x[M - 1] *= 2.0 ** 60
    y[N // 2] *= 2.0 ** -118
    got, want, plain = fast_gemm.gemm_f32(x, y), x.double() @ y.double().T, ops.gemm_generic(x, y, out_dtype=torch.float32)
    rows, cols = torch.arange(M, device="cuda"), torch.arange(N, device="cuda")
    rows, cols = rows[(rows != M // 3) & (rows != M - 1)], cols[cols != N // 2]
    assert torch.equal(got[rows][:, cols], clean[rows][:, cols])
    for part in (got[M // 3], got[M - 1], got[rows, N // 2]):
        assert part.isfinite().all()
    for i in (M // 3, M - 1):
        assert (got[i, cols].double() - want[i, cols]).norm() <= (plain[i, cols].double() - want[i, cols]).norm()
    assert (got[rows, N // 2].double() - want[rows, N // 2]).norm() <= (plain[rows, N // 2].double() - want[rows, N // 2]).norm()
    zero = torch.zeros_like(a)
    assert not fast_gemm.gemm_f32(zero, w).any() and not fast_gemm.gemm_f32(a, torch.zeros_like(w)).any()


@pytest.mark.parametrize("M,N,K", [(32, 40000, 2048), (6000, 4100, 8192), (600, 2048, 8192)])
def test_gemm_f32_on_planes_with_less_scratch_memory(M, N, K):
    """Less scratch memory means more portions of the operands and the same bits; less than the least is refused."""
    import ctypes
    from fastgguf_b200.ops import fast_gemm
    from fastgguf_b200.ops.lib import lib, ptr, stream
    a, w = _operands(M, N, K, torch.float32, 36)
    want = fast_gemm.gemm_f32(a, w)
    most, least = lib("tc").fg_gemm_f32_tc_workspace_bytes, lib("tc").fg_gemm_f32_tc_least_bytes
    most.restype = least.restype = ctypes.c_longlong
    top, low = most(M, N, K), least(M, N, K)
    assert 0 < low <= top
    for size in (low, low + (top - low) // 4, low + (top - low) // 2, top - 1):
        if size < low:
            continue
        ws, out = torch.empty(size, dtype=torch.uint8, device="cuda"), torch.zeros(M, N, device="cuda")
        assert lib("tc").fg_gemm_f32_tc(ptr(a), K, ptr(w), K, ptr(out), N, 0, M, N, K, ptr(ws), size, stream()) == 0
        assert torch.equal(out, want)
    ws = torch.empty(low, dtype=torch.uint8, device="cuda")
    assert lib("tc").fg_gemm_f32_tc(ptr(a), K, ptr(w), K, ptr(want), N, 0, M, N, K, ptr(ws), low - 1, stream()) == 10002


def test_gemm_f32_on_planes_refuses_other_sizes():
    from fastgguf_b200.ops import fast_gemm
    for M, N, K in ((16, 512, 1024), (64, 256, 1024), (100, 128, 1024), (100, 512, 256), (100, 512, 1028)):
        a, w = _operands(M, N, K, torch.float32, 7)
        assert fast_gemm.gemm_f32(a, w) is None
    a, w = _operands(64, 512, 1025, torch.float32, 7)
    assert fast_gemm.gemm_f32(a[:, 1:], w[:, 1:]) is None  # rows that start off a 16-byte boundary


@pytest.mark.parametrize("M", [1, 2, 3, 5, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(512, 512), (1000, 2048), (2048, 8192), (16384, 520), (20011, 1000), (9473, 644)])
def test_gemm_f32_stream(M, N, K):
    """Against float64 and, where a tile is tall enough for its order of additions, bit for bit what gemv_rows_kernel gives."""
    from fastgguf_b200 import ops
    from fastgguf_b200.ops import fast_gemm
    a, w = _operands(M, N, K, torch.float32, 8)
    got = fast_gemm.gemm_f32_stream(a, w)
    _check(got, a, w, a.double() @ w.double().T, False)
    if N == 20011 or N == 16384:
        assert torch.equal(got, ops.gemm_generic(a, w, out_dtype=torch.float32))
    # a row's result does not depend on the other rows of the step
    assert torch.equal(fast_gemm.gemm_f32_stream(a[M - 1:].contiguous(), w)[0], got[M - 1])
    wide = torch.full((M, K + 8), 7.0, device="cuda")
    wide[:, 4:K + 4] = a
    into = torch.full((M, N + 3), 9.0, device="cuda")
    res = torch.randn(M, N, device="cuda")
    into[:, 1:N + 1] = res
    fast_gemm.gemm_f32_stream(wide[:, 4:K + 4], w, out=into[:, 1:N + 1], accumulate=True)
    assert torch.equal(into[:, 1:N + 1], got + res) and (into[:, 0] == 9).all() and (into[:, N + 1:] == 9).all()
    special = a.clone()
    special[0, 3], special[M - 1, 5] = float("inf"), float("nan")
    x, y = fast_gemm.gemm_f32_stream(special, w), ops.gemm_generic(special, w, out_dtype=torch.float32)
    assert torch.equal(x.isnan(), y.isnan()) and torch.equal(x.isinf(), y.isinf())


def test_gemm_f32_stream_refuses_other_sizes():
    from fastgguf_b200.ops import fast_gemm
    for M, N, K in ((17, 1024, 1024), (4, 500, 1024), (4, 1024, 508), (4, 1024, 1026)):
        a, w = _operands(M, N, K, torch.float32, 7)
        assert fast_gemm.gemm_f32_stream(a, w) is None
    a, w = _operands(4, 1024, 1025, torch.float32, 7)
    assert fast_gemm.gemm_f32_stream(a[:, 1:], w[:, 1:]) is None


def test_gemm_f32_stream_ring_belongs_to_the_same_warps():
    """Where boxes are dealt out over groups of warps, a stage of the ring always falls to the same group and a CTA has one tile:
    the wait for a stage by its parity rests on that.  (A race: with ring depths that are no such multiple, an early box of a later round
    now and then let a warp through; a wrong sum showed in one of a few runs.)"""
    import ctypes
    from fastgguf_b200.ops.lib import lib
    out = (ctypes.c_int * 6)()
    dealt = 0
    for M in (1, 2, 4, 8, 16):
        for N in list(range(512, 9000, 61)) + [16384, 28672, 128256]:
            lib("tc").fg_gemm_f32_stream_plan(ctypes.c_int(M), ctypes.c_int(N), out)
            rows, tiles, row_groups, k_groups, stages, bytes_ = out
            assert rows * tiles >= N > rows * (tiles - 1) and row_groups * 4 >= rows and row_groups * k_groups <= 7
            assert 2 <= stages <= 16 and stages >= k_groups and bytes_ <= 108 * 1024
            if k_groups > 1:
                dealt += 1
                assert stages % k_groups == 0 and tiles <= 2 * torch.cuda.get_device_properties(0).multi_processor_count
    assert dealt > 100


def test_gemm_f32_stream_repeats_bit_for_bit():
    from fastgguf_b200.ops import fast_gemm
    for M, N, K in ((9, 1000, 2048), (8, 2048, 8192), (3, 3072, 2048)):
        a, w = _operands(M, N, K, torch.float32, 9)
        first = fast_gemm.gemm_f32_stream(a, w)
        for _ in range(300):
            assert torch.equal(fast_gemm.gemm_f32_stream(a, w), first)
