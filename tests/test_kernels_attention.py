"""The attention kernels alone (any-size, tensor-core decode, tensor-core prefill) against a plain
float64 computation over the same paged cache, at sizes other than the engine's.  Pages are handed
out in a shuffled order so that a wrong page lookup shows, and one far key per sequence is scaled
up so that a missed or doubled key changes the result visibly."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

PAGE = 64


@pytest.fixture(params=[0, 3, 7], ids=["one-score-tile", "two-score-tiles", "two-score-tiles-two-softmax-sets"])
def tc_variant(request):
    """Both forms of the tcgen05 prefill kernel at both head sizes, whatever the step's shape would choose."""
    from fastgguf_b200.ops import fast_attention
    fast_attention.prefill_tc_variant(request.param)
    yield request.param
    fast_attention.prefill_tc_variant(-1)


def make_case(lens_before, new, H, KV, hd, dtype, seed, boost=True, ramp=0.0):
    """Sequences with `lens_before[i]` cached tokens that bring `new[i]` more.  Returns everything
    the kernels need plus dense per-sequence K, V (float64) for the plain computation."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    n_seq = len(new)
    total = [a + b for a, b in zip(lens_before, new)]
    n_pages = sum((t + PAGE - 1) // PAGE for t in total) + 1
    perm = (torch.randperm(n_pages - 1, generator=g) + 1).tolist()      # page 0 stays unused
    k_pool = torch.zeros(n_pages, KV, PAGE, hd)
    v_pool = torch.zeros(n_pages, KV, PAGE, hd)
    width = max((t + PAGE - 1) // PAGE for t in total)
    table = torch.zeros(n_seq, width, dtype=torch.int32)
    dense = []
    for s in range(n_seq):
        K = torch.randn(total[s], KV, hd, generator=g)
        V = torch.randn(total[s], KV, hd, generator=g)
        if boost and total[s] > 3:
            K[total[s] // 3] *= 4.0                                      # one key that stands out
        if ramp:
            # scores that keep growing with the key's position: the running maximum moves in every block of keys
            K += (torch.arange(total[s]) / 16.0)[:, None, None] * ramp / hd ** 0.5
        K, V = K.to(dtype).float(), V.to(dtype).float()
        dense.append((K.double(), V.double()))
        for p in range((total[s] + PAGE - 1) // PAGE):
            page = perm.pop()
            table[s, p] = page
            n = min(PAGE, total[s] - p * PAGE)
            k_pool[page, :, :n] = K[p * PAGE:p * PAGE + n].transpose(0, 1)
            v_pool[page, :, :n] = V[p * PAGE:p * PAGE + n].transpose(0, 1)
    M = sum(new)
    q = torch.randn(M, H * hd, generator=g)
    if ramp:
        q += hd ** 0.5
    q = q.to(dtype)
    positions = torch.tensor([lens_before[s] + i for s in range(n_seq) for i in range(new[s])], dtype=torch.int32)
    row_seq = torch.tensor([s for s in range(n_seq) for _ in range(new[s])], dtype=torch.int32)
    cu = torch.tensor([0] + list(torch.tensor(new).cumsum(0)), dtype=torch.int32)
    return dict(q=q.cuda(), positions=positions.cuda(), row_seq=row_seq.cuda(), cu_rows=cu.cuda(),
                seq_start=torch.tensor(lens_before, dtype=torch.int32).cuda(), table=table.cuda(),
                k_pool=k_pool.to(dtype).cuda(), v_pool=v_pool.to(dtype).cuda(), dense=dense, new=new,
                lens_before=lens_before)


def plain(case, H, KV, hd, scale, window):
    q = case["q"].double().cpu().reshape(-1, H, hd)
    out = torch.zeros_like(q)
    G, row = H // KV, 0
    for s, (K, V) in enumerate(case["dense"]):
        for i in range(case["new"][s]):
            pos = case["lens_before"][s] + i
            lo = max(0, pos - window + 1) if window else 0
            for h in range(H):
                sc = (K[lo:pos + 1, h // G] @ q[row, h]) * scale
                w = torch.softmax(sc, 0)
                out[row, h] = w @ V[lo:pos + 1, h // G]
            row += 1
    return out.reshape(-1, H * hd)


def _err(got, want):
    return (got.double().cpu() - want).abs().max().item() / want.abs().max().item()


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 1.5e-2)])
@pytest.mark.parametrize("H,KV,hd,window", [(4, 2, 16, 0), (6, 1, 24, 0), (3, 3, 40, 50), (2, 1, 160, 0)])
def test_attention_generic(H, KV, hd, window, dtype, tol):
    from fastgguf_b200 import ops
    case = make_case([0, 70, 1300, 5], [9, 1, 3, 130], H, KV, hd, dtype, 11)
    scale = 1.0 / math.sqrt(hd)
    got = ops.attention_generic(case["q"], case["positions"], case["row_seq"], case["table"], case["k_pool"],
                                case["v_pool"], H, KV, hd, scale, window)
    assert _err(got, plain(case, H, KV, hd, scale, window)) < tol


@pytest.mark.parametrize("H,KV,hd,window", [(8, 2, 64, 0), (3, 1, 128, 0), (24, 8, 128, 0), (20, 1, 64, 0), (4, 4, 64, 100), (4, 2, 64, 64),
                                            (8, 2, 64, 65), (6, 2, 128, 128), (4, 2, 64, -48), (3, 1, 128, -200)])
def test_attention_prefill_f32(H, KV, hd, window):
    """The tiled float32 kernel against float64, and - chunked masks too - against the any-size kernel.  A value that is no number in
    rows of the last page that no sequence has reached, or at a later token's place, reaches no other row."""
    from fastgguf_b200 import ops
    from fastgguf_b200.ops import fast_attention
    new = [200, 1, 67, 5, 130]
    case = make_case([0, 300, 60, 0, 700], new, H, KV, hd, torch.float32, 13)
    scale = 1.0 / math.sqrt(hd)

    def both():
        got = fast_attention.attention_prefill_f32(case["q"], case["cu_rows"], case["seq_start"], case["table"], case["k_pool"],
                                                   case["v_pool"], len(new), max(new), H, KV, hd, scale, window)
        return got, ops.attention_generic(case["q"], case["positions"], case["row_seq"], case["table"], case["k_pool"], case["v_pool"],
                                          H, KV, hd, scale, window)

    got, any_size = both()
    assert _err(got, any_size.double().cpu()) < 5e-6
    if window >= 0:
        want = plain(case, H, KV, hd, scale, window)
        assert _err(got, want) < 5e-6
        assert (got.double().cpu() - want).norm() <= 1.2 * (any_size.double().cpu() - want).norm()
    # the first sequence's key 150 and everything behind each sequence's end are no numbers
    page, off = int(case["table"][0, 150 // PAGE]), 150 % PAGE
    case["v_pool"][page, :, off] = float("nan")
    for s, (before, n) in enumerate(zip(case["lens_before"], new)):
        end = before + n
        if end % PAGE:
            last = int(case["table"][s, end // PAGE])
            case["v_pool"][last, :, end % PAGE:] = float("inf")
            case["k_pool"][last, :, end % PAGE:] = float("nan")
    bad, bad_any = both()
    assert torch.equal(bad.isnan(), bad_any.isnan())
    assert torch.equal(bad[:150], got[:150]) and torch.equal(bad[200:], got[200:])


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("what", ["large keys", "large queries", "large values", "small values", "a rare value alone", "infinite key", "infinite query",
                                  "no number among the values"])
def test_attention_prefill_f32_outside_the_range_of_the_planes(what, hd):
    """Numbers that three bfloat16 planes do not carry (or whose products overflow) come out as the any-size kernel has them, and a value that
    only a key of tiny probability has keeps its digits."""
    from fastgguf_b200 import ops
    from fastgguf_b200.ops import fast_attention
    H, KV, new = 8, 2, [130, 70]
    case = make_case([0, 100], new, H, KV, hd, torch.float32, 17, boost=False)
    k, v, q = case["k_pool"], case["v_pool"], case["q"]
    page = [int(p) for p in case["table"][0, :2]]
    if what == "large keys":
        k.mul_(2.0 ** 64); q.mul_(2.0 ** -64)
    elif what == "large queries":
        q.mul_(2.0 ** 70); k.mul_(2.0 ** -70)
    elif what == "large values":
        v.mul_(2.0 ** 100)
    elif what == "small values":
        v.mul_(2.0 ** -118)
    elif what == "a rare value alone":
        k[page[0], 0, 10] = -q[90, :hd] * (84.0 / float(q[90, :hd] @ q[90, :hd]) * hd ** 0.5)     # row 90, head 0: about e^-86
        v[:, 0, :, 3] = 0.0
        v[page[0], 0, 10, 3] = 1.2345678 * 2.0 ** 20
    elif what == "infinite key":
        k[page[1], 1, 5, 7] = float("inf")
    elif what == "infinite query":
        q[20, 3] = -float("inf")
    else:
        v[page[0], 0, 9, 2] = float("nan")
    scale = 1.0 / math.sqrt(hd)
    got = fast_attention.attention_prefill_f32(q, case["cu_rows"], case["seq_start"], case["table"], k, v, 2, 130, H, KV, hd, scale, 0)
    want = ops.attention_generic(q, case["positions"], case["row_seq"], case["table"], k, v, H, KV, hd, scale, 0)
    assert torch.equal(got.isnan(), want.isnan())
    got, want = got.double().nan_to_num(), want.double().nan_to_num()
    assert (got - want).abs().max() <= 5e-6 * want.abs().max()
    if what == "a rare value alone":
        # a score of -84 by a chain of hd additions is off by hd * 84 * 2^-24 at most, in either; a probability of 2^-124 in planes that end
        # at 2^-133 would be off by 2^-9
        x, y = got[90, 3], want[90, 3]
        assert y > 0 and abs(x - y) <= 2 * hd * 84 * 2.0 ** -24 * y


@pytest.mark.parametrize("hd,window,few", [(64, 0, "-x-x-xxx"), (64, 100, "-x-x-xxx"), (64, -256, "-x-x-xxx"), (128, 0, "-x-----x"), (128, 300, "-x-----x")])
def test_attention_prefill_f32_leaves_out_sequences_of_few_rows(hd, window, few):
    """With the engine's skip_few the rows of every sequence that the host's rule names keep what the output held, all others have their values:
    host and kernel agree on both sides of the line, behind a past of any length, under windows and chunks."""
    import ctypes
    from fastgguf_b200.ops import fast_attention
    from fastgguf_b200.ops.lib import lib, ptr, stream
    H, KV = 32, 8
    before, new = [0, 300, 2000, 0, 700, 64, 2000, 100], [200, 1, 70, 40, 130, 20, 20, 14]
    case = make_case(before, new, H, KV, hd, torch.float32, 14)
    left = [bool(lib("core").fg_attention_f32_left_out(n, p, H, hd, window)) for n, p in zip(new, before)]
    assert "".join("x" if x else "-" for x in left) == few
    q, scale = case["q"], 1.0 / math.sqrt(hd)
    want = fast_attention.attention_prefill_f32(q, case["cu_rows"], case["seq_start"], case["table"], case["k_pool"], case["v_pool"], len(new), max(new),
                                                H, KV, hd, scale, window)
    out = torch.full_like(want, 9.0)
    f = ctypes.c_float
    assert lib("core").fg_attention_prefill_f32_ext(ptr(q), q.stride(0), ptr(out), out.stride(0), ptr(case["cu_rows"]), ptr(case["seq_start"]),
                                                    ptr(case["table"]), case["table"].shape[1], ptr(case["k_pool"]), ptr(case["v_pool"]), len(new),
                                                    max(new), H, KV, hd, 64, f(scale), window, lib("core").fg_attention_f32_skip_few(hd), stream()) == 0
    at = 0
    for n, left_out in zip(new, left):
        rows = out[at:at + n]
        assert (rows == 9.0).all() if left_out else torch.equal(rows, want[at:at + n])
        at += n


@pytest.mark.parametrize("n_splits", [None, 1, 2, 3, 8, 16])
@pytest.mark.parametrize("H,KV,hd,window", [(8, 2, 64, 0), (3, 1, 128, 0), (24, 8, 128, 0), (20, 1, 64, 0),
                                            (4, 4, 64, 100), (4, 2, 64, 64), (4, 2, 64, 128), (8, 2, 64, 65),
                                            (6, 2, 128, 128), (3, 1, 128, 65)])
def test_attention_decode(H, KV, hd, window, n_splits):
    from fastgguf_b200.ops import fast_attention
    case = make_case([0, 63, 64, 700, 2047, 129], [1] * 6, H, KV, hd, torch.bfloat16, 12)
    scale = 1.0 / math.sqrt(hd)
    got = fast_attention.attention_decode(case["q"], case["positions"], case["table"], case["k_pool"], case["v_pool"],
                                          H, KV, hd, scale, window, n_splits=n_splits)
    want = plain(case, H, KV, hd, scale, window)
    assert _err(got, want) < 1.5e-2
    if n_splits in (2, 8):        # the same splits through scratch memory and the merge kernel
        got = fast_attention.attention_decode(case["q"], case["positions"], case["table"], case["k_pool"],
                                              case["v_pool"], H, KV, hd, scale, window, n_splits=n_splits,
                                              use_scratch=True)
        assert _err(got, want) < 1.5e-2


@pytest.mark.parametrize("H,KV,hd,window", [(8, 2, 64, 0), (3, 1, 128, 0), (24, 8, 128, 0), (20, 1, 64, 0),
                                            (4, 4, 64, 100), (4, 2, 64, 64), (4, 2, 64, 128), (8, 2, 64, 65),
                                            (6, 2, 128, 128), (3, 1, 128, 65)])
def test_attention_prefill(H, KV, hd, window):
    from fastgguf_b200.ops import fast_attention
    new = [200, 1, 67, 5]
    case = make_case([0, 300, 60, 0], new, H, KV, hd, torch.bfloat16, 13)
    scale = 1.0 / math.sqrt(hd)
    got = fast_attention.attention_prefill(case["q"], case["cu_rows"], case["seq_start"], case["table"], case["k_pool"],
                                           case["v_pool"], len(new), max(new), H, KV, hd, scale, window)
    assert _err(got, plain(case, H, KV, hd, scale, window)) < 1.5e-2


@pytest.mark.parametrize("H,KV,hd,window", [(8, 2, 64, 0), (3, 1, 128, 0), (24, 8, 128, 0), (20, 1, 64, 0),
                                            (4, 4, 64, 100), (4, 2, 64, 64), (4, 2, 64, 128), (8, 2, 64, 65),
                                            (6, 2, 128, 128), (3, 1, 128, 65)])
def test_attention_prefill_tcgen05(H, KV, hd, window, tc_variant):
    from fastgguf_b200.ops import fast_attention
    new = [200, 1, 67, 5, 300]
    case = make_case([0, 300, 60, 0, 129], new, H, KV, hd, torch.bfloat16, 14)
    scale = 1.0 / math.sqrt(hd)
    got = fast_attention.attention_prefill_tc(case["q"], case["cu_rows"], case["seq_start"], case["table"],
                                              case["k_pool"], case["v_pool"], len(new), max(new), H, KV, hd, scale, window)
    assert fast_attention.prefill_tc_error() == 0
    assert _err(got, plain(case, H, KV, hd, scale, window)) < 1.5e-2


@pytest.mark.parametrize("H,KV,hd", [(6, 2, 128), (8, 2, 64)])
def test_attention_prefill_tcgen05_batch_of_long_unequal_prompts(H, KV, hd, tc_variant):
    """Prompts of 64 to 2,048 tokens in one step: tiles of 1 to 32 iterations side by side, rows that finish long
    after the last MMA of their tile and rows that finish before it (every wait on a barrier has to name the right
    phase at either end)."""
    from fastgguf_b200.ops import fast_attention
    new = [1500, 64, 700, 2048, 300, 129]
    case = make_case([0, 0, 64, 0, 1000, 0], new, H, KV, hd, torch.bfloat16, 31)
    scale = 1.0 / math.sqrt(hd)
    got = fast_attention.attention_prefill_tc(case["q"], case["cu_rows"], case["seq_start"], case["table"],
                                              case["k_pool"], case["v_pool"], len(new), max(new), H, KV, hd, scale, 0)
    assert fast_attention.prefill_tc_error() == 0
    assert _err(got, plain(case, H, KV, hd, scale, 0)) < 1.5e-2


@pytest.mark.parametrize("n_splits", [None, 1, 4, 8])
@pytest.mark.parametrize("H,KV,hd,window", [(8, 2, 64, 0), (6, 2, 128, 0), (20, 1, 64, 0), (4, 4, 64, 100),
                                            (4, 2, 64, 64), (4, 2, 64, 128), (6, 2, 128, 65), (6, 2, 128, 128)])
def test_attention_decode_fused_with_rope_and_append(H, KV, hd, window, n_splits):
    """One kernel for RoPE, cache append and attention of a decode step, against the separate kernels."""
    from fastgguf_b200 import ops
    from fastgguf_b200.ops import fast_attention
    lens = [0, 63, 64, 700, 2047, 129]
    case = make_case(lens, [1] * 6, H, KV, hd, torch.bfloat16, 15)
    g = torch.Generator().manual_seed(16)
    qkv = torch.randn(6, (H + 2 * KV) * hd, generator=g).bfloat16().cuda()
    ang = torch.arange(2100, dtype=torch.float64)[:, None] * torch.pow(torch.tensor(10000.0, dtype=torch.float64),
                                                                       -2.0 * torch.arange(hd // 2) / hd)
    cos, sin = torch.cos(ang).float().cuda(), torch.sin(ang).float().cuda()
    scale = 1.0 / math.sqrt(hd)
    row_seq = torch.arange(6, dtype=torch.int32).cuda()
    # separate kernels on copies of the cache
    k1, v1, q1 = case["k_pool"].clone(), case["v_pool"].clone(), qkv.clone()
    ops.rope_append(q1, case["positions"], row_seq, case["table"], k1, v1, cos, sin, H, KV, hd)
    want = fast_attention.attention_decode(q1, case["positions"], case["table"], k1, v1, H, KV, hd, scale, window,
                                           n_splits=n_splits)
    k2, v2 = case["k_pool"].clone(), case["v_pool"].clone()
    got = fast_attention.attention_decode_fused(qkv, case["positions"], case["table"], k2, v2, cos, sin, H, KV, hd,
                                                scale, window, n_splits=n_splits)
    assert (got.float() - want.float()).abs().max() <= 2e-2 * want.float().abs().max()
    assert torch.equal(k2, k1) and torch.equal(v2, v1)          # the cache received the same rows


@pytest.mark.parametrize("n_splits", [1, 2, 4, 8])
@pytest.mark.parametrize("H,KV,hd,window", [(8, 2, 64, 0), (6, 2, 128, 0), (20, 1, 64, 0), (4, 4, 16, 0), (9, 3, 32, 0), (4, 4, 64, 100), (4, 2, 16, 64), (6, 2, 128, 65),
                                            (8, 1, 64, -200)])
def test_attention_decode_f32(H, KV, hd, window, n_splits):
    """One kernel for rotation, cache append and attention of a float32 decode step, against the separate kernels; places of a page that no
    token has reached hold what is no number."""
    import ctypes
    from fastgguf_b200 import ops
    from fastgguf_b200.ops.lib import lib, ptr, stream
    lens = [0, 63, 64, 700, 2047, 129]
    case = make_case(lens, [1] * 6, H, KV, hd, torch.float32, 15)
    for s, n in enumerate(lens):
        last = int(case["table"][s, n // PAGE])
        case["v_pool"][last, :, n % PAGE:] = float("nan")
        case["k_pool"][last, :, n % PAGE:] = float("inf")
    g = torch.Generator().manual_seed(16)
    qkv = torch.randn(6, (H + 2 * KV) * hd, generator=g).cuda()
    ang = torch.arange(2100, dtype=torch.float64)[:, None] * torch.pow(torch.tensor(10000.0, dtype=torch.float64), -2.0 * torch.arange(hd // 2) / hd)
    cos, sin = torch.cos(ang).float().cuda(), torch.sin(ang).float().cuda()
    scale = 1.0 / math.sqrt(hd)

    def both():
        k1, v1, q1 = case["k_pool"].clone(), case["v_pool"].clone(), qkv.clone()
        rows = torch.arange(6, dtype=torch.int32).cuda()
        ops.rope_append(q1, case["positions"], rows, case["table"], k1, v1, cos, sin, H, KV, hd)
        want = ops.attention_generic(q1, case["positions"], rows, case["table"], k1, v1, H, KV, hd, scale, window)
        torch.cuda.synchronize()
        k2, v2, out, f = case["k_pool"].clone(), case["v_pool"].clone(), torch.empty(6, H * hd, device="cuda"), ctypes.c_float
        torch.cuda.synchronize()
        assert lib("core").fg_attention_decode_f32(ptr(qkv), qkv.stride(0), ptr(out), out.stride(0), ptr(case["positions"]), ptr(case["table"]),
                                                   case["table"].shape[1], ptr(k2), ptr(v2), ptr(cos), ptr(sin), 6, H, KV, hd, 64,
                                                   f(scale), window, n_splits, stream()) == 0
        assert (k2 - k1).nan_to_num().abs().max() <= 2e-6 and torch.equal(v2.nan_to_num(7.0), v1.nan_to_num(7.0))
        return out, want

    out, want = both()
    assert _err(out, want.double().cpu()) < 5e-6
    # numbers that are none, or infinite, at places that tokens see
    case["k_pool"][int(case["table"][3, 10]), 0, 5, 1] = float("nan")
    case["k_pool"][int(case["table"][4, 30]), 0, 60, 1] = float("inf")
    case["v_pool"][int(case["table"][5, 1]), 0, 60, 1] = float("inf")
    bad, bad_want = both()
    assert torch.equal(bad.isfinite(), bad_want.isfinite()) and torch.equal(bad.isnan(), bad_want.isnan())
    assert torch.equal(bad[:3], out[:3])


@pytest.mark.parametrize("H,KV,hd", [(8, 2, 64), (4, 1, 128)])
def test_attention_prefill_tcgen05_growing_maximum(H, KV, hd):
    """Scores that grow by tens of binary orders every 128 keys: every iteration moves the running base, and
    the rows of the output accumulated so far are rescaled in tensor memory."""
    from fastgguf_b200.ops import fast_attention
    scale = 1.0 / math.sqrt(hd)
    case = make_case([0, 300], [600, 200], H, KV, hd, torch.bfloat16, 21, boost=False, ramp=2.0)
    got = fast_attention.attention_prefill_tc(case["q"], case["cu_rows"], case["seq_start"], case["table"], case["k_pool"],
                                              case["v_pool"], 2, 600, H, KV, hd, scale, 0)
    assert fast_attention.prefill_tc_error() == 0
    want = plain(case, H, KV, hd, scale, 0)
    assert (got.double().cpu() - want).abs().max().item() <= 2e-2 * want.abs().max().item()


def _decode_f32(case, qkv, cos, sin, H, KV, hd, window, n_splits, warps, rows=None, width=None):
    """fg_attention_decode_f32_ext over copies of the pools, for the sequences `rows` with a page table of `width` entries."""
    import ctypes
    from fastgguf_b200.ops.lib import lib, ptr, stream
    rows = list(range(qkv.shape[0])) if rows is None else rows
    table, pos, x = case["table"][rows], case["positions"][rows].contiguous(), qkv[rows].contiguous()
    table = torch.cat([table, torch.zeros(len(rows), (width or table.shape[1]) - table.shape[1], dtype=torch.int32, device="cuda")], 1).contiguous()
    k, v, out, f = case["k_pool"].clone(), case["v_pool"].clone(), torch.empty(len(rows), H * hd, device="cuda"), ctypes.c_float
    torch.cuda.synchronize()
    assert lib("core").fg_attention_decode_f32_ext(ptr(x), x.stride(0), ptr(out), out.stride(0), ptr(pos), ptr(table), table.shape[1], ptr(k), ptr(v), ptr(cos),
                                                   ptr(sin), len(rows), H, KV, hd, 64, f(1.0 / math.sqrt(hd)), window, n_splits, warps, stream()) == 0
    torch.cuda.synchronize()
    return out, k, v


def _decode_f32_case(lens, H, KV, hd, seed, turned=True):
    case = make_case(lens, [1] * len(lens), H, KV, hd, torch.float32, seed)
    qkv = torch.randn(len(lens), (H + 2 * KV) * hd, generator=torch.Generator().manual_seed(seed + 1)).cuda()
    ang = torch.arange(max(lens) + 1, dtype=torch.float64)[:, None] * torch.pow(torch.tensor(10000.0, dtype=torch.float64), -2.0 * torch.arange(hd // 2) / hd)
    return case, qkv, torch.cos(ang * turned).float().cuda(), torch.sin(ang * turned).float().cuda()


@pytest.mark.parametrize("H,KV,hd,window", [(8, 2, 64, 0), (4, 2, 64, 0), (2, 2, 64, 100), (6, 1, 128, 0), (2, 1, 128, 65), (1, 1, 128, 0), (8, 2, 32, 0), (3, 3, 32, -200),
                                            (4, 2, 16, 0), (6, 2, 16, 33), (5, 5, 16, 0)])
def test_attention_decode_f32_does_not_depend_on_the_step(H, KV, hd, window):
    """A row's bits follow from its own sequence: alone or beside others, with any number of CTAs and warps and any width of the page table.
    Lengths around the edges of units, of runs of one and two units, and of more than 64 runs."""
    lens = [0, 31, 32, 63, 64, 97, 129, 1023, 1024, 1055, 2047, 2048, 2100, 4200]
    case, qkv, cos, sin = _decode_f32_case(lens, H, KV, hd, 21)
    want, want_k, want_v = _decode_f32(case, qkv, cos, sin, H, KV, hd, window, 1, 2)
    assert want.isfinite().all()
    for n_splits in (1, 2, 4, 8):
        for warps in (0, 2, 4) + ((8,) if hd < 128 else ()):
            got, k, v = _decode_f32(case, qkv, cos, sin, H, KV, hd, window, n_splits, warps)
            assert torch.equal(got, want) and torch.equal(k, want_k) and torch.equal(v, want_v), (n_splits, warps)
    for i in (0, 2, 5, 8, 13):
        assert torch.equal(_decode_f32(case, qkv, cos, sin, H, KV, hd, window, 8, 0, rows=[i], width=90)[0][0], want[i])


@pytest.mark.parametrize("H,KV,hd", [(8, 2, 64), (4, 4, 64), (8, 2, 128), (4, 2, 32), (4, 2, 16)])
def test_attention_decode_f32_is_as_near_to_float64_as_the_any_size_kernel(H, KV, hd):
    """Without rotation (cosines of one), so that both kernels and float64 have the same queries, keys and scores.  The 2-norm of the error over
    sequences of three length classes: sums of 16 values added up in a tree against eight runs of up to 128 in a chain."""
    from fastgguf_b200 import ops
    errors, size = [0.0, 0.0], 0.0
    for seed in range(23, 35, 2):
        for lens in ([20 + 3 * i for i in range(48)], [150 + 9 * i for i in range(48)], [1100 + 20 * i for i in range(48)]):
            case, qkv, cos, sin = _decode_f32_case(lens, H, KV, hd, seed, turned=False)
            got, k, v = _decode_f32(case, qkv, cos, sin, H, KV, hd, 0, 1, 0)
            any_size = ops.attention_generic(qkv[:, :H * hd].contiguous(), case["positions"], torch.arange(48, dtype=torch.int32).cuda(), case["table"], k, v, H, KV,
                                             hd, 1.0 / math.sqrt(hd), 0)
            for b, n in enumerate(lens):
                pages = case["table"][b, :n // PAGE + 1].long()
                K, V = (x[pages].double().transpose(1, 2).reshape(-1, KV, hd)[:n + 1].repeat_interleave(H // KV, 1) for x in (k, v))
                p = torch.softmax(torch.einsum("hd,khd->hk", qkv[b, :H * hd].double().view(H, hd), K) / math.sqrt(hd), -1)
                want = torch.einsum("hk,khd->hd", p, V).flatten()
                errors = [e + (x[b].double() - want).square().sum() for e, x in zip(errors, (got, any_size))]
                size = size + want.square().sum()
    ours, other = (math.sqrt(float(e / size)) for e in errors)
    assert ours <= other, (ours, other)


@pytest.mark.parametrize("hd", [16, 128])
@pytest.mark.parametrize("power", [-140, -30, 12, 17, 18, 19, 30, 100])
def test_attention_decode_f32_over_the_range_of_scores(power, hd):
    """Scores of 2^-140 to 2^100, around 2^20 with both kinds of bases in one row, against the any-size kernel, which has the same scores: every
    weight is off by a few units in the last place (expf, its argument), so the output by less than 16 * 2^-24 of the largest value."""
    from fastgguf_b200 import ops
    H, KV, lens = 8, 2, [3, 40, 100, 500, 2200]
    case, qkv, cos, sin = _decode_f32_case(lens, H, KV, hd, 29, turned=False)
    qkv[:, :H * hd] *= 2.0 ** power
    got, k, v = _decode_f32(case, qkv, cos, sin, H, KV, hd, 0, 1, 0)
    want = ops.attention_generic(qkv[:, :H * hd].contiguous(), case["positions"], torch.arange(5, dtype=torch.int32).cuda(), case["table"], k, v, H, KV, hd,
                                 1.0 / math.sqrt(hd), 0)
    assert got.isfinite().all() and (got - want).abs().max() <= 16 * 2.0 ** -24 * v.abs().max()
    for n_splits, warps in ((8, 4), (2, 2)):
        assert torch.equal(_decode_f32(case, qkv, cos, sin, H, KV, hd, 0, n_splits, warps)[0], got)
