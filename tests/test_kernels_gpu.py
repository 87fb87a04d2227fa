"""Each kernel alone against a plain float32 reference of the same operation, at sizes other than the
engine's tiny models: ragged edges, widths that are no power of two, one row, many rows."""
import math

import numpy as np
import pytest
import torch

import plain_qwen3 as plain

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _bf16(t):
    return t.to(torch.bfloat16)


# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,width,vocab", [(1, 96, 50), (37, 100, 257), (300, 4096, 1000)])
def test_embed(dtype, rows, width, vocab):
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(1)
    table = torch.randn(vocab, width, generator=g).to(dtype).to(DEV)
    ids = torch.randint(0, vocab, (rows,), generator=g, dtype=torch.int32).to(DEV)
    out = torch.empty(rows, width, dtype=torch.float32, device=DEV)
    ops.embed(table, ids, out)
    assert torch.equal(out, table.float()[ids.long()])


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,width,eps", [(1, 16, 1e-6), (33, 100, 1e-5), (7, 4096, 1e-6), (5, 5000, 1e-3)])
def test_rmsnorm(out_dtype, rows, width, eps):
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(2)
    x = (torch.randn(rows, width, generator=g) * 3).to(DEV)
    w = (1 + 0.1 * torch.randn(width, generator=g)).to(DEV)
    out = torch.empty(rows, width, dtype=out_dtype, device=DEV)
    ops.rmsnorm(x, w, eps, out)
    ref = plain.rms_norm(x.cpu().numpy(), w.cpu().numpy(), eps)
    if out_dtype is torch.bfloat16:
        ref = plain.round_bf16(ref)
        assert np.abs(out.float().cpu().numpy() - ref).max() <= np.abs(ref).max() * 2 ** -7
    else:
        assert np.abs(out.cpu().numpy() - ref).max() <= 1e-5 * np.abs(ref).max()
    # Gathered rows: the head's pick of rows folded into the norm.
    idx = torch.tensor([rows - 1, 0], dtype=torch.int32, device=DEV)
    out2 = torch.empty(2, width, dtype=out_dtype, device=DEV)
    ops.rmsnorm(x, w, eps, out2, row_index=idx)
    assert torch.equal(out2, out[idx.long()])


@pytest.mark.parametrize("rows,width", [(1, 8), (19, 172), (64, 12288)])
def test_swiglu(rows, width):
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(3)
    gu = (torch.randn(rows, 2 * width, generator=g) * 4).to(DEV)
    out = torch.empty(rows, width, dtype=torch.float32, device=DEV)
    ops.swiglu(gu, out)
    a = gu.cpu().numpy()
    ref = plain.silu(a[:, :width]) * a[:, width:]
    assert np.abs(out.cpu().numpy() - ref).max() <= 1e-5 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,head_dim,rot,norm", [(4, 2, 16, 16, True), (6, 3, 32, 32, True), (3, 1, 48, 24, False),
                                                              (32, 8, 128, 128, True), (2, 2, 256, 64, True)])
@pytest.mark.parametrize("rows", [11, 70])
def test_head_norm_rope_kv(dtype, heads, kv_heads, head_dim, rot, norm, rows):
    """Per-head norm, rotation (whole or partial width) and the write into scattered cache slots
    (few rows and many: the kernel shares its work out differently)."""
    from llmx_b200 import ops
    page, pages = 8, 9
    g = torch.Generator().manual_seed(4)
    qkv = torch.randn(rows, (heads + 2 * kv_heads) * head_dim, generator=g).to(DEV)
    qw = (1 + 0.1 * torch.randn(head_dim, generator=g)).to(DEV) if norm else None
    kw = (1 + 0.1 * torch.randn(head_dim, generator=g)).to(DEV) if norm else None
    positions = torch.randint(0, 40, (rows,), generator=g, dtype=torch.int32)
    cos_np, sin_np = plain.rope_tables(40, rot, 10000.0)
    cos, sin = torch.from_numpy(cos_np).to(DEV), torch.from_numpy(sin_np).to(DEV)
    slots = torch.randperm(pages * page, generator=g)[:rows].to(torch.int32)
    slots[3] = -1                                                   # one row's write is skipped
    cache = torch.zeros(pages, 2, kv_heads, page, head_dim, dtype=dtype, device=DEV)
    q_out = torch.empty(rows, heads * head_dim, dtype=dtype, device=DEV)
    ops.head_norm_rope_kv(qkv, heads, kv_heads, head_dim, qw, kw, 1e-6, cos, sin, positions.to(DEV), slots.to(DEV),
                          q_out, cache)
    a = qkv.cpu().numpy()
    q = a[:, :heads * head_dim].reshape(rows, heads, head_dim)
    k = a[:, heads * head_dim:(heads + kv_heads) * head_dim].reshape(rows, kv_heads, head_dim)
    v = a[:, (heads + kv_heads) * head_dim:].reshape(rows, kv_heads, head_dim)
    if norm:
        q, k = plain.rms_norm(q, qw.cpu().numpy(), 1e-6), plain.rms_norm(k, kw.cpu().numpy(), 1e-6)
    c, s = cos_np[positions.numpy()], sin_np[positions.numpy()]

    def rotate(x):
        out = x.copy()
        out[..., :rot] = plain.rope_rotate(x[..., :rot], c, s)
        return out
    q, k = rotate(q), rotate(k)
    tol = 2 ** -7 if dtype is torch.bfloat16 else 1e-5
    got_q = q_out.float().cpu().numpy().reshape(rows, heads, head_dim)
    assert np.abs(got_q - q).max() <= tol * np.abs(q).max()
    cache_np = cache.float().cpu().numpy()
    for r in range(rows):
        sl = int(slots[r])
        if sl < 0:
            continue
        assert np.abs(cache_np[sl // page, 0, :, sl % page] - k[r]).max() <= tol * np.abs(k).max()
        assert np.abs(cache_np[sl // page, 1, :, sl % page] - v[r]).max() <= tol * np.abs(v).max()
    written = {int(s) for s in slots if s >= 0}
    for sl in range(pages * page):
        if sl not in written:
            assert not cache_np[sl // page, :, :, sl % page].any()


# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("m,n,k", [(1, 64, 16), (5, 100, 37), (70, 257, 100), (130, 384, 96)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gemm_plain(dtype, m, n, k):
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(5)
    a = torch.randn(m, k, generator=g).to(dtype).to(DEV)
    w = torch.randn(n, k, generator=g).to(dtype).to(DEV)
    base = torch.randn(m, n, generator=g).to(DEV)
    ref = a.float().cpu().double() @ w.float().cpu().double().T
    out = torch.empty(m, n, dtype=torch.float32, device=DEV)
    ops.gemm_plain(a, w, out)
    assert (out.cpu().double() - ref).abs().max() <= 1e-5 * ref.abs().max()
    acc = base.clone()
    ops.gemm_plain(a, w, acc, accumulate=True)
    assert (acc.cpu().double() - (ref + base.cpu().double())).abs().max() <= 1e-5 * ref.abs().max()


@pytest.mark.parametrize("m", [1, 3, 16, 17, 64, 65, 128, 200, 513])
@pytest.mark.parametrize("n,k", [(128, 64), (100, 72), (384, 96), (1000, 160), (6144, 1024)])
def test_gemm_tensor_core(m, n, k):
    """The tcgen05 product at ragged sizes: M, N beyond a tile's edge, K that is no multiple of 64."""
    from llmx_b200 import ops_tc
    g = torch.Generator().manual_seed(6)
    a = _bf16(torch.randn(m, k, generator=g)).to(DEV)
    w = _bf16(torch.randn(n, k, generator=g) * 0.1).to(DEV)
    ref = a.float().cpu().double() @ w.float().cpu().double().T
    guard = torch.full((m + 2, n), 7.0, device=DEV)             # rows around the output must stay untouched
    out = guard[1:m + 1]
    ops_tc.gemm_tc(a, w, out)
    torch.cuda.synchronize()
    ops_tc.check_errors()
    assert (out.cpu().double() - ref).abs().max() <= 2e-5 * max(1.0, ref.abs().max())
    assert torch.all(guard[0] == 7.0) and torch.all(guard[m + 1] == 7.0)
    base = torch.randn(m, n, generator=g).to(DEV)
    for splits in (1, 2, 5):
        acc = base.clone()
        ops_tc.gemm_tc(a, w, acc, accumulate=True, splits=splits)
        assert (acc.cpu().double() - (ref + base.cpu().double())).abs().max() <= 3e-5 * max(1.0, ref.abs().max())
    ops_tc.check_errors()


@pytest.mark.parametrize("tile", [16, 32, 64, 128, 256])
def test_gemm_tensor_core_every_token_tile(tile):
    from llmx_b200 import ops_tc
    g = torch.Generator().manual_seed(7)
    m, n, k = 300, 260, 200
    a = _bf16(torch.randn(m, k, generator=g)).to(DEV)
    w = _bf16(torch.randn(n, k, generator=g)).to(DEV)
    out = torch.empty(m, n, device=DEV)
    ops_tc.gemm_tc(a, w, out, token_tile=tile)
    ref = a.float().cpu().double() @ w.float().cpu().double().T
    ops_tc.check_errors()
    assert (out.cpu().double() - ref).abs().max() <= 2e-5 * ref.abs().max()


@pytest.mark.parametrize("m", [65, 130, 257, 600])
@pytest.mark.parametrize("n,k", [(100, 72), (384, 96), (1000, 160), (4096, 1024)])
def test_gemm_tensor_core_on_pairs_of_sms(m, n, k):
    """The two-block (tcgen05 `cta_group::2`) product at ragged sizes: a second block whose weight rows or token rows
    lie wholly or partly beyond the matrix, K that is no multiple of 64, both token tiles, K in ranges."""
    from llmx_b200 import ops_tc
    g = torch.Generator().manual_seed(16)
    a = _bf16(torch.randn(m, k, generator=g)).to(DEV)
    w = _bf16(torch.randn(n, k, generator=g) * 0.1).to(DEV)
    ref = a.float().cpu().double() @ w.float().cpu().double().T
    base = torch.randn(m, n, generator=g).to(DEV)
    for tile in (128, 256):
        guard = torch.full((m + 2, n), 7.0, device=DEV)
        out = guard[1:m + 1]
        ops_tc.gemm_tc_pair(a, w, out, token_tile=tile)
        torch.cuda.synchronize()
        ops_tc.check_errors()
        assert (out.cpu().double() - ref).abs().max() <= 2e-5 * max(1.0, ref.abs().max())
        assert torch.all(guard[0] == 7.0) and torch.all(guard[m + 1] == 7.0)
        for splits in (1, 2, 3, 0):
            acc = base.clone()
            ops_tc.gemm_tc_pair(a, w, acc, accumulate=True, splits=splits, token_tile=tile)
            assert (acc.cpu().double() - (ref + base.cpu().double())).abs().max() <= 3e-5 * max(1.0, ref.abs().max())
    ops_tc.check_errors()


@pytest.mark.parametrize("m,n,k", [(2300, 2100, 1104), (1100, 4100, 3000), (520, 1000, 64), (4100, 2300, 8200)])
def test_gemm_on_pairs_cuts_only_the_last_round(m, n, k):
    """`splits` 0: whole tiles for the full rounds of the 74 pairs, the remaining tiles' K in ranges.  Sizes with one
    or two full rounds and a ragged rest, fewer tiles than pairs, a single k block, and a K long enough that the
    rest is cut into many ranges; added to what the output holds, and stored."""
    from llmx_b200 import ops_tc
    g = torch.Generator().manual_seed(18)
    a = _bf16(torch.randn(m, k, generator=g)).to(DEV)
    w = _bf16(torch.randn(n, k, generator=g) * 0.1).to(DEV)
    ref = a.float().double() @ w.float().double().T
    base = torch.randn(m, n, generator=g).to(DEV)
    bound = 3e-5 * max(1.0, ref.abs().max().item())
    for tile in (128, 256):
        acc = base.clone()
        ops_tc.gemm_tc_pair(a, w, acc, accumulate=True, splits=0, token_tile=tile)
        assert (acc.double() - (ref + base.double())).abs().max() <= bound
        guard = torch.full((m + 2, n), 7.0, device=DEV)
        out = guard[1:m + 1]
        ops_tc.gemm_tc_pair(a, w, out, splits=0, token_tile=tile)
        assert (out.double() - ref).abs().max() <= bound
        assert torch.all(guard[0] == 7.0) and torch.all(guard[m + 1] == 7.0)
    ops_tc.check_errors()


def test_gemm_plan_may_choose_pairs_and_can_be_told_not_to():
    from llmx_b200 import ops_tc, runtime
    assert ops_tc.plan(2048, 4096, 4096, True)[0] == 2
    before = runtime.pair_products(False)
    try:
        assert ops_tc.plan(2048, 4096, 4096, True)[0] == 0
    finally:
        runtime.pair_products(before)
    assert ops_tc.plan(8, 4096, 4096, True)[0] == 1


def test_gemm_tensor_core_refuses_unaligned_width():
    from llmx_b200 import ops_tc
    from llmx_b200.ops import KernelError
    a = torch.zeros(4, 100, dtype=torch.bfloat16, device=DEV)
    w = torch.zeros(8, 100, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(KernelError):
        ops_tc.gemm_tc(a, w, torch.empty(4, 8, device=DEV))


# ---------------------------------------------------------------------------------------------
def _attention_case(dtype, heads, kv_heads, head_dim, page, layout, window, seed, spike=False):
    """A batch laid out as `layout` = [(history, new rows), ...] over a shuffled pool of pages.

    Returns everything the kernels need plus the plain result.  With `spike`, one far key of every
    request is made to stand out (its score dominates), so a kernel that drops or misplaces a page
    shows a large error instead of one that random values average away."""
    g = torch.Generator().manual_seed(seed)
    n_req = len(layout)
    lens = [h + n for h, n in layout]
    pages_needed = [-(-l // page) for l in lens]
    total_pages = sum(pages_needed) + 3
    perm = torch.randperm(total_pages, generator=g).tolist()
    cache = torch.randn(total_pages, 2, kv_heads, page, head_dim, generator=g)      # stale values everywhere
    tables = np.zeros((n_req, max(pages_needed)), dtype=np.int32)
    ks, vs, qs = [], [], []
    rows = sum(n for _, n in layout)
    row_start, at = [], 0
    for r, (h, n) in enumerate(layout):
        row_start.append(at)
        at += n
        k = torch.randn(lens[r], kv_heads, head_dim, generator=g)
        v = torch.randn(lens[r], kv_heads, head_dim, generator=g)
        q = torch.randn(n, heads, head_dim, generator=g)
        if spike and lens[r] > 3:
            far = max(0, lens[r] - (window or lens[r]) + 1) if window else 1
            far = min(far, lens[r] - 1)
            k[far] = q[-1, ::heads // kv_heads] * 4.0          # every group's key lines up with the last row's query
        ks.append(k); vs.append(v); qs.append(q)
        mine = [perm.pop() for _ in range(pages_needed[r])]
        tables[r, :len(mine)] = mine
        for t in range(lens[r]):
            cache[mine[t // page], 0, :, t % page] = k[t]
            cache[mine[t // page], 1, :, t % page] = v[t]
    cache = cache.to(dtype)
    q_all = torch.cat(qs).to(dtype)
    ref = np.zeros((rows, heads, head_dim), dtype=np.float32)
    for r, (h, n) in enumerate(layout):
        full_q = np.zeros((lens[r], heads, head_dim), dtype=np.float32)
        full_q[h:] = q_all[row_start[r]:row_start[r] + n].float().numpy()
        kk = ks[r].to(dtype).float().numpy()
        vv = vs[r].to(dtype).float().numpy()
        ref[row_start[r]:row_start[r] + n] = plain.attention(full_q, kk, vv, window=window)[h:]
    # The step (metadata on the device, launch plan of an attention of this shape) as the engine would make it.
    from llmx_b200 import ops_attn
    step = ops_attn.attention_step(DEV, layout, tables, heads, kv_heads, head_dim, window, page)
    group = step.groups[0]
    return q_all.reshape(rows, heads * head_dim).to(DEV).contiguous(), cache.to(DEV), step, group, ref.reshape(rows, -1)


LAYOUTS = {
    "decode": [(0, 1), (1, 1), (15, 1), (16, 1), (17, 1), (200, 1), (1027, 1)],
    "prefill": [(0, 1), (0, 2), (0, 17), (0, 130), (0, 300)],
    "mixed": [(40, 1), (0, 70), (128, 2), (63, 65), (5, 3), (300, 1), (16, 16)],
}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,head_dim,page", [(4, 2, 16, 8), (6, 3, 32, 16), (3, 1, 48, 4), (8, 8, 80, 16), (2, 1, 256, 32)])
@pytest.mark.parametrize("layout", ["decode", "prefill", "mixed"])
@pytest.mark.parametrize("window", [None, 19])
def test_attention_plain(dtype, heads, kv_heads, head_dim, page, layout, window):
    from llmx_b200 import ops
    q, cache, step, group, ref = _attention_case(dtype, heads, kv_heads, head_dim, page, LAYOUTS[layout], window, seed=8)
    out = torch.empty_like(q)
    ops.attention_plain(q, cache, out, step.row_request, step.positions, group.block_tables, heads, kv_heads, head_dim,
                        window, 1.0 / math.sqrt(head_dim))
    tol = 2e-2 if dtype is torch.bfloat16 else 2e-5
    assert np.abs(out.float().cpu().numpy() - ref).max() <= tol * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(32, 8, 128), (4, 4, 64), (16, 1, 128), (6, 2, 64), (8, 8, 128),
                                                     (40, 8, 128), (6, 2, 128), (12, 2, 128), (10, 2, 64), (7, 1, 128)])
@pytest.mark.parametrize("layout", ["decode", "prefill", "mixed"])
@pytest.mark.parametrize("window", [None, 100])
@pytest.mark.parametrize("spike", [False, True])
def test_attention_tiled_bf16(heads, kv_heads, head_dim, layout, window, spike):
    """The split-KV decode kernel and the tiled prefill kernel behind the one dispatch the mixer calls."""
    from llmx_b200 import ops_attn, ops_tc
    assert ops_attn.supported(heads, kv_heads, head_dim, 16)
    q, cache, step, group, ref = _attention_case(torch.bfloat16, heads, kv_heads, head_dim, 16, LAYOUTS[layout], window,
                                                 seed=9, spike=spike)
    out = torch.full_like(q, float("nan"))
    ops_attn.paged_attention_bf16(q, cache, out, step, group, heads, kv_heads, head_dim, window, 1.0 / math.sqrt(head_dim))
    torch.cuda.synchronize()
    ops_tc.check_errors()
    got = out.float().cpu().numpy()
    assert np.isfinite(got).all()
    assert np.abs(got - ref).max() <= 2e-2 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("item_tiles,key_splits", [(1, 1), (2, 1), (1, 2), (2, 2), (2, 3), (1, 5)])
@pytest.mark.parametrize("heads,kv_heads", [(32, 8), (16, 8), (8, 8), (40, 8), (6, 2), (14, 2)])
@pytest.mark.parametrize("window", [None, 300])
def test_attention_prefill_items_of_any_shape(item_tiles, key_splits, heads, kv_heads, window):
    """The tcgen05 prefill kernel's work items hold one row tile or two, and all of a block's keys or one of
    several ranges of them (a second kernel then adds the ranges up); the launcher chooses, here every
    combination is forced.  Short requests leave ranges without keys and rows that a range's keys do not reach."""
    from llmx_b200 import ops_attn, ops_tc
    layout = [(0, 300), (77, 130), (1500, 64), (3, 33), (40, 1), (700, 200)]
    q, cache, step, group, ref = _attention_case(torch.bfloat16, heads, kv_heads, 128, 16, layout, window, seed=23, spike=True)
    step.plan.native.plan.force_prefill_shape(item_tiles, key_splits)
    out = torch.full_like(q, float("nan"))
    ops_attn.paged_attention_bf16(q, cache, out, step, group, heads, kv_heads, 128, window, 1.0 / math.sqrt(128))
    torch.cuda.synchronize()
    ops_tc.check_errors()
    got = out.float().cpu().numpy()
    assert np.isfinite(got).all()
    assert np.abs(got - ref).max() <= 2e-2 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("history", [0, 320, 448])
def test_attention_prefill_blocks_walk_several_items(history):
    """More work items than SMs: a block of the tcgen05 prefill kernel then walks several (request, kv head, rows)
    items one after the other, its barriers' phases going on from item to item.  Forty requests of 64 new rows
    after the same history make 320 items of equal length, which is what once let a barrier complete twice
    before a waiting warp had looked."""
    from llmx_b200 import ops_attn, ops_tc
    heads, kv_heads, head_dim = 32, 8, 128
    layout = [(history, 64)] * 38 + [(history + 100, 33), (7, 130)]
    q, cache, step, group, ref = _attention_case(torch.bfloat16, heads, kv_heads, head_dim, 16, layout, None, seed=21, spike=True)
    for _ in range(3):                                   # the fault was one of timing: run it more than once
        out = torch.full_like(q, float("nan"))
        ops_attn.paged_attention_bf16(q, cache, out, step, group, heads, kv_heads, head_dim, None, 1.0 / math.sqrt(head_dim))
        torch.cuda.synchronize()
        ops_tc.check_errors()
        got = out.float().cpu().numpy()
        assert np.isfinite(got).all()
        assert np.abs(got - ref).max() <= 2e-2 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("window", [None, 5000])
def test_attention_over_long_histories(window):
    """Tens of thousands of keys behind a request: block tables of over a thousand pages, sixteen key ranges for the
    decoding rows, hundreds of key stages for a prompt portion.  One key near the start of every request (or of
    its window) is made to stand out for the last row, so a page that is dropped or misplaced anywhere shows."""
    from llmx_b200 import ops_attn, ops_tc
    heads, kv_heads, D, page = 32, 8, 128, 16
    layout = [(20000, 1), (9001, 3), (12345, 70), (33, 1)]
    g = torch.Generator().manual_seed(31)
    lens = [h + n for h, n in layout]
    pages_needed = [-(-l // page) for l in lens]
    total_pages = sum(pages_needed) + 5
    perm = torch.randperm(total_pages, generator=g).tolist()
    cache = torch.randn(total_pages, 2, kv_heads, page, D, generator=g).to(torch.bfloat16)
    tables = np.zeros((len(layout), max(pages_needed)), dtype=np.int32)
    qs, refs, row_start, at = [], [], [], 0
    for r, (h, n) in enumerate(layout):
        row_start.append(at)
        at += n
        k = torch.randn(lens[r], kv_heads, D, generator=g)
        v = torch.randn(lens[r], kv_heads, D, generator=g)
        q = torch.randn(n, heads, D, generator=g).to(torch.bfloat16)
        far = max(1, lens[r] - window + 1) if window else 1
        k[far] = q[-1, ::heads // kv_heads].float() * 4.0
        k, v = k.to(torch.bfloat16), v.to(torch.bfloat16)
        mine = [perm.pop() for _ in range(pages_needed[r])]
        tables[r, :len(mine)] = mine
        idx = torch.tensor(mine).repeat_interleave(page)[:lens[r]]
        off = torch.arange(lens[r]) % page
        cache[idx, 0, :, off] = k
        cache[idx, 1, :, off] = v
        # plain reference for the new rows alone: row at position p sees keys lo..p
        kk = k.double().repeat_interleave(heads // kv_heads, dim=1)      # [L, heads, D]
        vv = v.double().repeat_interleave(heads // kv_heads, dim=1)
        scores = torch.einsum("nhd,lhd->nhl", q.double(), kk) / math.sqrt(D)
        pos = torch.arange(h, h + n)[:, None, None]
        keys = torch.arange(lens[r])[None, None, :]
        seen = keys <= pos
        if window:
            seen &= keys > pos - window
        scores = scores.masked_fill(~seen, float("-inf"))
        refs.append(torch.einsum("nhl,lhd->nhd", torch.softmax(scores, dim=-1), vv))
        qs.append(q)
    rows = at
    ref = torch.cat(refs).reshape(rows, -1).numpy()
    q_all = torch.cat(qs).reshape(rows, heads * D).to(DEV).contiguous()

    step = ops_attn.attention_step(DEV, layout, tables, heads, kv_heads, D, window, page)
    group = step.groups[0]
    out = torch.full_like(q_all, float("nan"))
    ops_attn.paged_attention_bf16(q_all, cache.to(DEV), out, step, group, heads, kv_heads, D, window, 1.0 / math.sqrt(D))
    torch.cuda.synchronize()
    ops_tc.check_errors()
    got = out.float().cpu().numpy()
    assert np.isfinite(got).all()
    assert np.abs(got - ref).max() <= 2e-2 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("cluster", [True, False])
@pytest.mark.parametrize("splits", [1, 2, 3, 4, 7, 8, 12, 16, 20])
def test_attention_decode_any_number_of_key_ranges(splits, cluster):
    """Key ranges are combined through the shared memory of a thread-block cluster (up to sixteen ranges, unless
    turned off) or through memory by the block that finishes last; short requests leave ranges without keys."""
    from llmx_b200 import ops_attn, ops_tc
    before = ops_attn.cluster_merge(cluster)
    try:
        _decode_with_key_ranges(splits)
    finally:
        ops_attn.cluster_merge(before)


def _decode_with_key_ranges(splits):
    from llmx_b200 import ops_attn, ops_tc
    heads, kv_heads, head_dim = 8, 2, 128
    layout = [(1500, 1), (63, 1), (64, 1), (700, 2), (0, 1)]
    q, cache, step, group, ref = _attention_case(torch.bfloat16, heads, kv_heads, head_dim, 16, layout, None, seed=10, spike=True)
    chunk = -(-(-(-1501 // 64)) // splits) * 64
    step.plan.native.plan.force_decode(splits, chunk)
    out = torch.full_like(q, float("nan"))
    ops_attn.paged_attention_bf16(q, cache, out, step, group, heads, kv_heads, head_dim, None, 1.0 / math.sqrt(head_dim))
    torch.cuda.synchronize()
    ops_tc.check_errors()
    assert np.abs(out.float().cpu().numpy() - ref).max() <= 2e-2 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("heads,kv_heads", [(32, 8), (16, 1), (8, 8), (4, 2)])
@pytest.mark.parametrize("window", [None, 100])
@pytest.mark.parametrize("rotate,norm", [(True, True), (False, True), (True, False)])
@pytest.mark.parametrize("splits", [None, 3])
def test_attention_decode_from_the_products_output(heads, kv_heads, window, rotate, norm, splits):
    """The decode kernel that norms and rotates its own queries and new keys, against the separate kernel
    followed by the decode kernel: the same bits in the output and in the cache.  Histories put new rows at
    the first and last slot of a page, at the edge of a key range, and (with several new rows) across two pages;
    one request's write is skipped, as for a layer that reads another layer's cache."""
    from llmx_b200 import ops, ops_attn, ops_tc
    head_dim, page = 128, 16
    max_new = 16 // (heads // kv_heads)
    layout = [(0, 1), (15, 1), (16, 1), (63, min(2, max_new)), (64, 1), (127, min(3, max_new)), (700, max_new), (1500, 1)]
    _, cache, step, group, _ = _attention_case(torch.bfloat16, heads, kv_heads, head_dim, page, layout, window, seed=12)
    rows = step.rows
    g = torch.Generator().manual_seed(13)
    qkv = torch.randn(rows, (heads + 2 * kv_heads) * head_dim, generator=g).to(DEV)
    qw = (1 + 0.1 * torch.randn(head_dim, generator=g)).to(DEV) if norm else None
    kw = (1 + 0.1 * torch.randn(head_dim, generator=g)).to(DEV) if norm else None
    cos = sin = None
    if rotate:
        cos_np, sin_np = plain.rope_tables(1600, head_dim, 10000.0)
        cos, sin = torch.from_numpy(cos_np).to(DEV), torch.from_numpy(sin_np).to(DEV)
    slots = group.slots                                             # page * 16 + slot of every row's position
    slots[step.host_row_start[4]] = -1                              # this row's key and value are not written
    if splits:
        step.plan.native.plan.force_decode(splits, -(-(-(-1501 // 64)) // splits) * 64)
    scale = 1.0 / math.sqrt(head_dim)
    # the separate kernels
    cache_a = cache.clone()
    q = torch.empty(rows, heads * head_dim, dtype=torch.bfloat16, device=DEV)
    ops.head_norm_rope_kv(qkv, heads, kv_heads, head_dim, qw, kw, 1e-6, cos, sin, step.positions, slots, q, cache_a)
    out_a = torch.full_like(q, float("nan"))
    ops_attn.paged_attention_bf16(q, cache_a, out_a, step, group, heads, kv_heads, head_dim, window, scale)
    # the one kernel
    cache_b = cache.clone()
    out_b = torch.full_like(q, float("nan"))
    assert ops_attn.decode_from_qkv(qkv, qw, kw, 1e-6, cos, sin, out_b, step, 0, heads, kv_heads, head_dim, window, scale,
                                    cache=ops_attn.OneEntryCache(cache_b))
    torch.cuda.synchronize()
    ops_tc.check_errors()
    assert torch.isfinite(out_b.float()).all()
    assert torch.equal(cache_a, cache_b)
    assert torch.equal(out_a, out_b)


# ---------------------------------------------------------------------------------------------
def _sample_rows(logits, settings):
    from llmx_b200.sampling import RequestSampling, SamplingParams, sample
    states = []
    for s in settings:
        st = RequestSampling(SamplingParams(**{k: v for k, v in s.items() if k not in ("gen", "masked")}),
                             eos_id=s.get("masked", -1))
        st.masked = s.get("masked", -1)
        for t in s.get("gen", ()):
            st.saw(t)
        states.append(st)
    got = sample(torch.from_numpy(logits).to(DEV).contiguous(), states)
    return got, states


@pytest.mark.parametrize("vocab", [5, 257, 5000, 151936])
def test_sampling_against_the_plain_sampler(vocab):
    """Every mode of the device sampler against the plain one, the same uniform number for both."""
    rng = np.random.default_rng(vocab)
    settings = [
        dict(temp=0.0, top_k=0, top_p=1.0),
        dict(temp=0.0, top_k=0, top_p=1.0, masked=0),
        dict(temp=1.0, top_k=0, top_p=1.0, seed=3),
        dict(temp=0.7, top_k=40, top_p=1.0, seed=4),
        dict(temp=1.3, top_k=0, top_p=0.9, seed=5),
        dict(temp=0.8, top_k=40, top_p=0.95, seed=6),
        dict(temp=1.0, top_k=3, top_p=0.5, min_p=0.2, seed=7),
        dict(temp=2.0, top_k=0, top_p=1.0, min_p=0.05, seed=8),
        dict(temp=1.0, top_k=0, top_p=0.8, min_p=0.1, seed=9, masked=1),
        dict(temp=0.0, top_k=0, top_p=1.0, penalty=1.5, presence_penalty=0.2, frequency_penalty=0.1, gen=[1, 2, 2, 4]),
        dict(temp=0.9, top_k=10, top_p=0.9, penalty=1.2, seed=11, gen=[0, 3]),
    ]
    logits = (rng.standard_normal((len(settings), vocab)) * 3).astype(np.float32)
    logits[0, :] = 0.0
    logits[0, [2, 4]] = 5.0                                  # a tie: the lowest id wins
    logits[3, :min(vocab, 60)] = 2.0                         # ties across the top-k edge: lowest ids are kept
    expected = []
    for row, s in zip(logits, settings):
        r = 0.0 if s["temp"] <= 0 else plain.XorShift64(s.get("seed", 0)).unit()
        expected.append(plain.sample(row, s["temp"], s["top_k"], s["top_p"], s.get("min_p", 0.0), r,
                                     penalty=s.get("penalty", 1.0), presence=s.get("presence_penalty", 0.0),
                                     frequency=s.get("frequency_penalty", 0.0), gen=list(s.get("gen", ())),
                                     masked=s.get("masked", -1)))
    got, _ = _sample_rows(logits.copy(), settings)
    assert got == expected


@pytest.mark.parametrize("vocab", [9001, 40000, 151936])
@pytest.mark.parametrize("coarse", [False, True])
def test_sampling_settings_at_random_against_the_plain_sampler(vocab, coarse):
    """Vocabularies that two, four and eight blocks share (see the end); settings drawn at random (top-k beyond what is gathered into
    shared memory too); with `coarse`, scores on a grid of quarters, so that hundreds of tokens tie exactly at every
    threshold: ties go to the lowest ids, whichever block holds them."""
    rng = np.random.default_rng(vocab + int(coarse))
    settings = []
    for i in range(24):
        settings.append(dict(temp=float(rng.choice([0.3, 0.8, 1.0, 1.7])), top_k=int(rng.choice([0, 1, 7, 40, 300, 1024, 1025, 3000])),
                             top_p=float(rng.choice([1.0, 0.95, 0.6, 0.1])), min_p=float(rng.choice([0.0, 0.0, 0.05, 0.3])),
                             seed=int(rng.integers(1, 1 << 40))))
        if i % 5 == 0:
            settings[-1]["masked"] = int(rng.integers(0, vocab))
    logits = (rng.standard_normal((len(settings), vocab)) * 2.5).astype(np.float32)
    if coarse:
        logits = (np.round(logits * 4) / 4).astype(np.float32)
    expected = []
    for row, s in zip(logits, settings):
        r = plain.XorShift64(s["seed"]).unit()
        expected.append(plain.sample(row, s["temp"], s["top_k"], s["top_p"], s["min_p"], r, masked=s.get("masked", -1)))
    got, _ = _sample_rows(logits.copy(), settings)
    assert got == expected
    # The kernel gives a row fewer blocks when the rows are many (all rows run at one time): twelve rows a call still
    # get the most blocks their vocabulary allows, twenty-four at the largest vocabulary get half as many.
    halves = _sample_rows(logits[:12].copy(), settings[:12])[0] + _sample_rows(logits[12:].copy(), settings[12:])[0]
    assert halves == expected


@pytest.mark.parametrize("kind", ["one_binade", "wide", "two_values", "negative"])
def test_sampling_of_rows_whose_best_tokens_outnumber_a_blocks_list(kind):
    """Scores whose leading eight bits hardly tell them apart (all within a factor of two or four, of two values, a third of the row
    above the threshold's leading bits): a block's tokens do not fit its list (8,192) after the first round, after the second,
    or ever.  Against the plain sampler, with one row (eight blocks) and with sixteen (four)."""
    rng = np.random.default_rng(len(kind))
    vocab, rows = 151936, 16
    logits = {"one_binade": 8 + 8 * rng.random((rows, vocab)), "wide": 3 * rng.standard_normal((rows, vocab)),
              "two_values": 1.0 + 0.5 * (rng.random((rows, vocab)) < 0.4), "negative": -32 + 24 * rng.random((rows, vocab))}[kind].astype(np.float32)
    settings = [dict(temp=float(t), top_k=int(k), top_p=float(p), seed=r + 1, masked=7 if r % 3 == 0 else -1)
                for r, (t, k, p) in enumerate(zip(rng.choice([0.7, 1.0], rows), np.resize([1, 40, 1000, 1024, 1025, 3000, 100000, 62000], rows), rng.choice([1.0, 0.9], rows)))]
    expected = [plain.sample(row, s["temp"], s["top_k"], s["top_p"], 0.0, plain.XorShift64(s["seed"]).unit(), masked=s["masked"]) for row, s in zip(logits, settings)]
    assert _sample_rows(logits.copy(), settings)[0] == expected
    assert [_sample_rows(logits[r:r + 1].copy(), settings[r:r + 1])[0][0] for r in range(8)] == expected[:8]


def test_sampling_distribution_and_independence_of_the_batch():
    """Draws follow the softmax, and a request's draws do not depend on what shares its batch."""
    from llmx_b200.sampling import RequestSampling, SamplingParams, sample
    logits = torch.tensor([[0.0, 1.0, 2.0, -1.0]], device=DEV)
    st = RequestSampling(SamplingParams(temp=1.0, top_k=0, top_p=1.0, seed=99))
    counts = np.zeros(4)
    alone = []
    for _ in range(2000):
        t = sample(logits, [st])[0]
        alone.append(t)
        counts[t] += 1
    p = np.exp([0, 1, 2, -1.0]); p /= p.sum()
    assert np.abs(counts / counts.sum() - p).max() < 0.04
    st2 = RequestSampling(SamplingParams(temp=1.0, top_k=0, top_p=1.0, seed=99))
    other = RequestSampling(SamplingParams(temp=0.5, top_k=2, top_p=0.9, seed=5))
    both = torch.cat([torch.randn(1, 4, device=DEV), logits])
    batched = [sample(both, [other, st2])[1] for _ in range(200)]
    assert batched == alone[:200]


@pytest.mark.parametrize("m", [1, 8, 33, 64])
@pytest.mark.parametrize("n,k", [(128, 64), (100, 72), (1000, 160), (6144, 1024), (4096, 4096), (5000, 4104)])
def test_gemm_tensor_core_stream_k(m, n, k):
    """Few tokens: (tile, k block) units shared out over the blocks, pieces added with atomics.  The two largest
    weights stream long enough to get uneven shares (the second half of the blocks a shorter run each)."""
    from llmx_b200 import ops_tc
    g = torch.Generator().manual_seed(12)
    a = _bf16(torch.randn(m, k, generator=g)).to(DEV)
    w = _bf16(torch.randn(n, k, generator=g) * 0.1).to(DEV)
    ref = a.float().cpu().double() @ w.float().cpu().double().T
    out = torch.full((m, n), 5.0, device=DEV)
    ops_tc.gemm_tc(a, w, out, schedule=1)
    assert (out.cpu().double() - ref).abs().max() <= 3e-5 * max(1.0, ref.abs().max())
    base = torch.randn(m, n, generator=g).to(DEV)
    acc = base.clone()
    ops_tc.gemm_tc(a, w, acc, accumulate=True, schedule=1)
    ops_tc.check_errors()
    assert (acc.cpu().double() - (ref + base.cpu().double())).abs().max() <= 3e-5 * max(1.0, ref.abs().max())


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("m", [1, 16, 70, 128, 300])
@pytest.mark.parametrize("f,k", [(128, 64), (172, 104), (200, 128), (1536, 512)])
def test_gemm_tensor_core_gated(m, f, k, pair):
    """silu(gate) * up in the product's epilogue, for intermediate widths that are no multiple of a tile; on single
    blocks and on pairs of SMs."""
    from llmx_b200 import ops_tc
    g = torch.Generator().manual_seed(13)
    a = _bf16(torch.randn(m, k, generator=g)).to(DEV)
    w = _bf16(torch.randn(2 * f, k, generator=g) * 0.2).to(DEV)
    guard = torch.full((m + 2, f), 3.0, dtype=torch.bfloat16, device=DEV)
    out = guard[1:m + 1]
    ops_tc.gemm_tc_swiglu(a, w, out, pair=pair)
    ops_tc.check_errors()
    assert torch.all(guard[0] == 3.0) and torch.all(guard[m + 1] == 3.0)
    gu = (a.float().cpu().double() @ w.float().cpu().double().T).numpy()
    ref = plain.silu(gu[:, :f].astype(np.float32)) * gu[:, f:].astype(np.float32)
    assert np.abs(out.float().cpu().numpy() - ref).max() <= 2 ** -7 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("tile", [128, 256, "pair"])
@pytest.mark.parametrize("m,heads,kv_heads,k,rotate,norm", [(70, 4, 2, 64, True, True), (300, 3, 1, 200, True, True),
                                                            (129, 2, 2, 512, False, True), (1000, 5, 1, 136, True, False)])
def test_gemm_tensor_core_finishes_heads(tile, m, heads, kv_heads, k, rotate, norm):
    """The q/k/v product with the per-head norm, the rotation and the cache write in its epilogue: against the
    plain formulas, and bit for bit against the product followed by the per-head kernel (a prompt's keys must
    not depend on which of the two a portion's size chose).  Odd head counts leave half-empty 256-row tiles."""
    from llmx_b200 import ops, ops_tc
    D, page, pages = 128, 16, 80
    g = torch.Generator().manual_seed(21)
    a = _bf16(torch.randn(m, k, generator=g)).to(DEV)
    w = _bf16(torch.randn((heads + 2 * kv_heads) * D, k, generator=g) * 0.2).to(DEV)
    qw = (1 + 0.1 * torch.randn(D, generator=g)).to(DEV) if norm else None
    kw = (1 + 0.1 * torch.randn(D, generator=g)).to(DEV) if norm else None
    positions = torch.randint(0, 300, (m,), generator=g, dtype=torch.int32)
    cos_np, sin_np = plain.rope_tables(300, D, 10000.0)
    cos = torch.from_numpy(cos_np).to(DEV) if rotate else None
    sin = torch.from_numpy(sin_np).to(DEV) if rotate else None
    slots = torch.randperm(pages * page, generator=g)[:m].to(torch.int32)
    slots[5] = -1
    cache = torch.zeros(pages, 2, kv_heads, page, D, dtype=torch.bfloat16, device=DEV)
    q_out = torch.zeros(m, heads * D, dtype=torch.bfloat16, device=DEV)
    pair = tile == "pair"       # on pairs of SMs: 256 tokens x two heads a pair, each block loads one head
    ops_tc.gemm_tc_heads(a, ops_tc.WeightMap(w, 128 if pair else tile, heads=True), heads, kv_heads, qw, kw, 1e-6, cos, sin,
                         positions.to(DEV), slots.to(DEV), q_out, cache, pair=pair)
    ops_tc.check_errors()

    qkv = torch.empty(m, w.shape[0], device=DEV)
    ops_tc.gemm_tc(a, w, qkv, schedule=0, splits=1)
    cache2, q2 = torch.zeros_like(cache), torch.zeros_like(q_out)
    ops.head_norm_rope_kv(qkv, heads, kv_heads, D, qw, kw, 1e-6, cos, sin, positions.to(DEV), slots.to(DEV), q2, cache2)
    assert torch.equal(q_out, q2) and torch.equal(cache, cache2)

    full = (a.float().cpu().double() @ w.float().cpu().double().T).numpy().astype(np.float32)
    q = full[:, :heads * D].reshape(m, heads, D)
    kk = full[:, heads * D:(heads + kv_heads) * D].reshape(m, kv_heads, D)
    v = full[:, (heads + kv_heads) * D:].reshape(m, kv_heads, D)
    if norm:
        q, kk = plain.rms_norm(q, qw.cpu().numpy(), 1e-6), plain.rms_norm(kk, kw.cpu().numpy(), 1e-6)
    if rotate:
        c, s = cos_np[positions.numpy()], sin_np[positions.numpy()]
        q, kk = plain.rope_rotate(q, c, s), plain.rope_rotate(kk, c, s)
    tol = 2 ** -7
    assert np.abs(q_out.float().cpu().numpy().reshape(m, heads, D) - q).max() <= tol * np.abs(q).max()
    cache_np = cache.float().cpu().numpy()
    for r in range(m):
        sl = int(slots[r])
        if sl >= 0:
            assert np.abs(cache_np[sl // page, 0, :, sl % page] - kk[r]).max() <= tol * np.abs(kk).max()
            assert np.abs(cache_np[sl // page, 1, :, sl % page] - v[r]).max() <= tol * np.abs(v).max()


def test_a_wait_that_nothing_satisfies_gives_up_and_is_reported():
    """Every wait in the kernels is bounded; a wait that runs out records a code in the device's error word and the
    block goes on to its end.  The self-test kernel (csrc/selftest.cu) waits a millisecond on a barrier nobody
    arrives at: the kernel returns, the word holds the code, and `check_errors` raises (and clears the word)."""
    import ctypes
    from llmx_b200 import ops_tc, runtime
    from llmx_b200.csrc import build
    fn = build.load("selftest").llmx_wait_selftest
    fn.argtypes = [ctypes.c_ulonglong, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    fn.restype = ctypes.c_int
    torch.cuda.synchronize()
    ops_tc.check_errors()
    word = runtime.error_word(DEV)
    out = torch.zeros(2, dtype=torch.int32, device=DEV)
    assert fn(1_000_000, word.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()                                    # returns: nothing hangs
    assert out.tolist() == [2, 2]                               # the wait gave up; a later wait of the block returned at once
    with pytest.raises(runtime.KernelError, match="nobody arrives"):
        ops_tc.check_errors()
    ops_tc.check_errors()                                       # the word was cleared
    assert fn(10, word.data_ptr(), out.data_ptr(), None) == 10001          # limits outside 1 us .. 0.1 s are refused


def test_lanes_of_a_warps_wait_never_disagree():
    """Half of a warp's lanes wait on a barrier that has completed, half on one that nobody arrives at: all lanes get the same
    answer (csrc/selftest.cu), so that none is left waiting in the warp-wide instructions that follow such waits."""
    import ctypes
    from llmx_b200 import ops_tc, runtime
    from llmx_b200.csrc import build
    fn = build.load("selftest").llmx_warp_wait_selftest
    fn.argtypes = [ctypes.c_ulonglong, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    fn.restype = ctypes.c_int
    torch.cuda.synchronize()
    ops_tc.check_errors()
    word = runtime.error_word(DEV)
    out = torch.zeros(32, dtype=torch.int32, device=DEV)
    assert fn(1_000_000, word.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert out.tolist() == [2] * 32
    with pytest.raises(runtime.KernelError, match="nobody arrives"):
        ops_tc.check_errors()


def test_random_weights_are_the_same_on_the_device_and_on_the_host():
    """"Seed 0" names one model: the random-weights mode makes the same bits on the GPU (benchmarks, `Engine.from_config`)
    as on the CPU (model folders, the tests' plain implementation)."""
    from llmx_b200.weights.random_init import RandomSource
    from llmx_b200.weights.spec import TensorSpec
    specs = {"w.weight": TensorSpec((301, 257)), "n.weight": TensorSpec((129,), "vector", init="one_plus_normal", std=0.01)}
    for dtype in (torch.float32, torch.bfloat16):
        host, device = RandomSource(specs, 7, dtype=dtype, device="cpu"), RandomSource(specs, 7, dtype=dtype, device=DEV)
        for name in specs:
            assert torch.equal(host.tensor(name), device.tensor(name).cpu()), (name, dtype)


# ---- latent attention of requests with many rows: keys and values made once a step ----------------------------------------------
LATENT_STEPS = {
    "one_tile": ([32], [0]), "edges_of_a_tile": ([128, 127, 129], [0, 0, 0]), "odd_after_odd": ([65, 33], [63, 1]),
    "many_keys": ([40], [700]), "few_rows_between": ([3, 200, 1, 31, 64, 2], [50, 17, 130, 0, 64, 9]), "two_tiles_after_a_stage": ([256], [64]),
}


@pytest.mark.parametrize("name", list(LATENT_STEPS))
@pytest.mark.parametrize("heads,rot,latent,window,halves", [(3, 64, 512, 100, False), (5, 8, 64, None, True), (2, 0, 192, 1, False), (1, 48, 128, 64, True)])
def test_latent_prompt_equals_the_general_form(name, heads, rot, latent, window, halves):
    """Every row of a planned step against the same attention in 64 bits over the same queries, cache and maps, by the form for
    many rows and by the general one.  Both round the result to bfloat16 (2^-9 of it) after 32-bit sums of a few hundred to
    a thousand terms, whose error is relative to the values' size (about 2^-20 of it): the bound below is twice these."""
    from llmx_b200 import ops
    from llmx_b200.parts.base import Precision, StepShape
    from llmx_b200.parts.latent_attention import LatentAttention
    counts, histories = LATENT_STEPS[name]
    g = torch.Generator(device="cuda").manual_seed(7)
    page, rows, scale, mag = 16, sum(counts), 0.11, 1.25
    part = LatentAttention(64, heads, 128, rot, 128, None, latent, scale, 1e4, rot, 1e-6, window, pairing="halves" if halves else "neighbours")
    part.precision, part._sms = Precision.of("bfloat16"), 148
    part.w_uk, part.w_uv = (torch.randn(heads * 128, latent, device="cuda", generator=g).mul_(latent ** -0.5).bfloat16() for _ in range(2))
    freq = torch.from_numpy(part.frequencies()[0]).cuda()
    plan = part.plan_step(StepShape(counts, histories))
    assert plan.wide is not None and sum(r[1] for r in plan.runs) == sum(n for n in counts if n < 32)
    ints = torch.tensor(plan.values, device="cuda")
    needs = [-(-(h + n) // page) for h, n in zip(histories, counts)]
    order = torch.randperm(sum(needs), generator=torch.Generator().manual_seed(3)).tolist()
    tables, at = torch.full((len(counts), max(needs)), -1, dtype=torch.int32), 0
    for r, k in enumerate(needs):
        tables[r, :k] = torch.tensor(order[at:at + k])
        at += k
        if window is not None:                                   # pages below every row's window have been given back
            tables[r, :max(0, histories[r] - window + 1) // page] = -1
    cache = torch.randn(sum(needs), 1, 1, page, latent + rot, device="cuda", generator=g).bfloat16()
    q = torch.randn(rows, heads * (128 + rot), device="cuda", generator=g)
    request = torch.cat([torch.full((n,), r, dtype=torch.int32) for r, n in enumerate(counts)])
    position = torch.cat([torch.arange(h, h + n, dtype=torch.int32) for h, n in zip(histories, counts)])
    meta = request.cuda(), position.cuda(), tables.cuda()
    sizes = (heads, 128, rot, 128, latent, page, window, scale)
    out = torch.zeros(rows, heads * 128, device="cuda", dtype=torch.bfloat16)
    first, n_req, share, tiles_at, n_tiles, tokens, group = plan.wide
    ops.latent_attention_prompt(q, cache, part.w_uk, part.w_uv, out, freq, *meta, ints[first:], n_req, share, ints[tiles_at:], n_tiles, tokens,
                                max(1, min(group, heads - 1)), *sizes, halves=halves, magnitude=mag)
    for start, n, at, n_tiles, splits in plan.runs:
        s = slice(start, start + n)
        ops.latent_attention_tiled(q[s], cache, part.w_uk, part.w_uv, out[s], freq, meta[0][s], meta[1][s], meta[2], ints[at:], n_tiles, splits, *sizes,
                                   halves=halves, magnitude=mag)
    general = torch.zeros_like(out)
    ops.latent_attention(q, cache, part.w_uk, part.w_uv, general, freq, *meta, *sizes, halves=halves, magnitude=mag)
    from llmx_b200.runtime import check_errors
    check_errors()
    uk, uv = (w.double().view(heads, 128, latent) for w in (part.w_uk, part.w_uv))
    flat = cache.view(-1, latent + rot).double()
    for r in range(rows):
        p, table = int(position[r]), meta[2][int(request[r])].long()
        t = torch.arange(max(0, p - window + 1) if window else 0, p + 1, device="cuda")
        c = flat[table[t // page] * page + t % page]
        qh = q[r].double().view(heads, 128 + rot)
        x = qh[:, 128:].clone()
        a, b = (x[:, :rot // 2], x[:, rot // 2:]) if halves else (x[:, 0::2], x[:, 1::2])
        angle = (p * freq).double()                              # the angle is the 32-bit product
        turned = torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], 1)
        if not halves:
            turned = turned.view(heads, 2, rot // 2).transpose(1, 2).reshape(heads, rot)
        s = torch.einsum("hd,hdc,tc->ht", qh[:, :128], uk, c[:, :latent]) + mag * turned @ c[:, latent:].T
        values = torch.einsum("hvc,tc->htv", uv, c[:, :latent])
        want = torch.einsum("ht,htv->hv", torch.softmax(s * scale, 1), values).reshape(-1)
        bound = 2 * (2.0 ** -9 * want.abs() + 2.0 ** -20 * (1.0 + s.abs().max() * scale) * values.abs().max())
        for how, got in (("many rows", out), ("general", general)):
            worst = ((got[r].double() - want).abs() / bound).max()
            assert worst <= 1.0, (how, r, p, float(worst))


# ---- matrix-state recurrences over long runs of rows ----------------------------------------------------------------------------
@pytest.mark.parametrize("mode", ["constant", "delta", "scaled", "delta_channels", "channels"])
@pytest.mark.parametrize("heads,qk_heads,D,V,counts", [
    (2, 1, 4, 1, [9, 1]), (3, 3, 32, 17, [16, 23]), (4, 2, 36, 33, [40]), (2, 2, 64, 15, [31, 12, 64]), (40, 20, 64, 64, [17]), (1, 1, 66, 7, [25]),
    (2, 1, 128, 16, [33, 8]), (20, 10, 128, 130, [21, 48]), (1, 1, 130, 20, [18]), (2, 1, 256, 40, [35]), (1, 1, 512, 9, [20])])
def test_recurrence_over_many_rows(mode, heads, qk_heads, D, V, counts):
    """The wide form against the recurrence in 64 bits, from a state and from nothing: vector widths on both sides of every
    lane layout, columns that do not fill a block, 16 and 32 columns a block, runs that end within a chunk, a group of eight
    and a group of four rows.  32-bit sums of D terms and decays below one: an error of a few times sqrt(D) 2^-24 of the
    largest result."""
    import types
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(D + V)
    rows, R = sum(counts), len(counts)
    unit = lambda: torch.nn.functional.normalize(torch.randn(rows, qk_heads, D, generator=g), dim=-1)
    # q, k and v inside one wider matrix, as the projections hold them.
    wide = torch.cat([unit().reshape(rows, -1), unit().reshape(rows, -1), torch.randn(rows, heads * V, generator=g)], 1).to(DEV)
    qk = qk_heads * D
    q, k, v = wide[:, :qk], wide[:, qk:2 * qk], wide[:, 2 * qk:]
    per = D if mode in ("delta_channels", "channels") else 1
    gate = (0.7 + 0.3 * torch.rand(rows, heads * per, generator=g)).to(DEV)
    beta, skip = torch.rand(rows, heads, generator=g).to(DEV), torch.randn(heads, generator=g).to(DEV)
    decay = (0.9 + 0.1 * torch.rand(heads, generator=g)).to(DEV)
    state = torch.randn(2 * R + 1, heads, V, D, generator=g).to(DEV)
    history = [0 if r == 1 else 5 for r in range(R)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    step = types.SimpleNamespace(row_start=i32([sum(counts[:r]) for r in range(R)]), row_count=i32(counts), history=i32(history),
                                 state_slots=i32(list(range(R))), state_slots_out=i32([R + 1 + r for r in range(R)]), requests=R,
                                 max_row_count=max(counts), rows=rows)
    before = state.double().clone()
    out = torch.full((rows, heads * V), 7.0, device=DEV)
    code = ["constant", "delta", "scaled", "delta_channels", "channels"].index(mode)
    fn, P = ops._fn("recurrence", "llmx_linear_recurrence"), ops._ptr
    ops._check(fn(P(q), P(k), P(v), q.stride(0), k.stride(0), v.stride(0), code, P(decay), P(gate), P(beta), gate.stride(0), beta.stride(0),
                  P(skip) if mode == "scaled" else None, P(state), heads * V * D, P(step.row_start), P(step.row_count), P(step.history),
                  P(step.state_slots), P(step.state_slots_out), P(out), R, heads, qk_heads, D, V, max(counts), ops._stream()), "recurrence")
    share = heads // qk_heads
    at = 0
    for r, n in enumerate(counts):
        S = torch.zeros_like(before[r]) if history[r] == 0 else before[r].clone()          # [heads, V, D]
        want = []
        for t in range(at, at + n):
            kt, qt = (x[t].double().view(qk_heads, D).repeat_interleave(share, 0) for x in (k, q))
            vt, gt, bt = v[t].double().view(heads, V), gate[t].double().view(heads, 1, per), beta[t].double().view(heads, 1)
            S = S * (decay.double().view(heads, 1, 1) if mode == "constant" else gt)
            u = vt
            if mode in ("delta", "delta_channels"):
                u = bt * (vt - torch.einsum("hvd,hd->hv", S, kt))
            if mode == "scaled":
                u = bt * vt
            S = S + u[:, :, None] * kt[:, None, :]
            o = torch.einsum("hvd,hd->hv", S, qt)
            want.append((o + skip.double().view(heads, 1) * vt if mode == "scaled" else o).reshape(-1))
        want = torch.stack(want)
        bound = 8 * D ** 0.5 * 2.0 ** -24
        assert (out[at:at + n].double() - want).abs().max() <= bound * max(1.0, float(want.abs().max())), (r, "rows")
        assert (state[R + 1 + r].double() - S).abs().max() <= bound * max(1.0, float(S.abs().max())), (r, "state")
        at += n
    assert torch.equal(state[:R + 1].double(), before[:R + 1])


# ---- the experts' products on the tensor cores ----------------------------------------------------------------------------------
@pytest.mark.parametrize("counts", [[1, 0, 15, 16, 17], [255, 256, 257], [127, 128, 129, 512, 513], [272, 3]])
@pytest.mark.parametrize("K,N,clamp", [(32, 8, None), (160, 130, None), (96, 256, (1.5, 1.7))])
def test_expert_products_at_the_edges_of_their_tiles(counts, K, N, clamp):
    """Experts whose pairs end just below, at and above a tile, part of a tile or several equal ones, widths that end within a
    block of columns or a step of K: both products against the same in 64 bits.  The gated one is rounded to bfloat16 (2^-9),
    and 32-bit sums of K terms of about one are off by less than sqrt(K) 2^-22."""
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(K + N)
    experts, rows = len(counts), sum(counts)
    choice = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(counts)])[torch.randperm(rows, generator=g)].view(rows, 1).to(DEV)
    h = _bf16(torch.randn(rows, K, generator=g)).to(DEV)
    w_gu = _bf16(torch.randn(experts, 2 * N, K, generator=g) * K ** -0.5).to(DEV)
    w = _bf16(torch.randn(experts, N, K, generator=g) * K ** -0.5).to(DEV)
    lists = torch.empty((experts, rows), dtype=torch.int32, device=DEV)
    held = torch.empty((experts,), dtype=torch.int32, device=DEV)
    tiles = torch.empty((ops.moe_tiles_len(rows, experts),), dtype=torch.int32, device=DEV)
    ops.moe_route(None, choice, experts, lists, held, tiles, tensor_cores=True)
    assert held.tolist() == counts
    act = torch.full((rows, N), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.moe_product(h, 1, w_gu, lists, held, tiles, rows, act, gated=True, tensor_cores=True, clamp=clamp)
    y = torch.full((rows, N), 7.0, dtype=torch.float32, device=DEV)
    ops.moe_product(h, 1, w, lists, held, tiles, rows, y, gated=False, tensor_cores=True)
    e = choice[:, 0].long()
    both = torch.einsum("rk,rnk->rn", h.double(), w_gu.double()[e])
    gate, up = both[:, :N], both[:, N:]
    if clamp is None:
        want = gate * torch.sigmoid(gate) * up
    else:
        gate, up = gate.clamp(max=clamp[0]), up.clamp(-clamp[0], clamp[0])
        want = gate * torch.sigmoid(clamp[1] * gate) * (up + 1.0)
    slack = K ** 0.5 * 2.0 ** -22
    assert ((act.double() - want).abs() <= 2.0 ** -8 * want.abs() + 8 * slack).all()
    assert (y.double() - torch.einsum("rk,rnk->rn", h.double(), w.double()[e])).abs().max() <= 4 * slack


@pytest.mark.parametrize("tensor_cores", [False, True])
@pytest.mark.parametrize("rows,top,experts", [(1, 1, 2), (1023, 1, 3), (1365, 3, 5), (4095, 1, 4), (4097, 1, 4), (3001, 3, 6), (9001, 1, 3)])
def test_routing_of_pairs_over_several_chunks(rows, top, experts, tensor_cores):
    """Lists, counts and tiles exactly as the pairs' order gives them: a block looks up 4,096 pairs at a time (four turns of 1,024), so
    less than a turn, four turns but one pair, one chunk and a pair, three chunks; one expert takes most, the last gets none, some pairs
    name experts without weights."""
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(rows)
    pairs = rows * top
    choice = torch.randint(0, experts + 1, (rows, top), generator=g)
    choice[torch.rand(rows, top, generator=g) < 0.6] = 0
    choice[choice == experts - 1] = experts + 3
    table = choice.to(torch.int32).to(DEV)
    lists, counts = torch.full((experts, pairs), -1, dtype=torch.int32, device=DEV), torch.full((experts,), -1, dtype=torch.int32, device=DEV)
    tiles = torch.full((ops.moe_tiles_len(pairs, experts),), -1, dtype=torch.int32, device=DEV)
    ops.moe_route(None, table, experts, lists, counts, tiles, tensor_cores=tensor_cores)
    size, flat, want_tiles = 128 if tensor_cores else 32, choice.reshape(-1), []
    for e in range(experts):
        mine = torch.nonzero(flat == e).reshape(-1)
        assert counts[e].item() == mine.numel() and torch.equal(lists[e, :mine.numel()].cpu().long(), mine), e
        want_tiles += [x for at in range(0, mine.numel(), size) for x in (e, at)]
    assert tiles[:2].tolist() == [len(want_tiles) // 2, size] and tiles[2:2 + len(want_tiles)].tolist() == want_tiles


@pytest.mark.parametrize("rows,top,K,N,experts", [(1, 1, 8, 1, 3), (1, 8, 16, 7, 8), (8, 1, 1032, 300, 1), (3, 2, 4096, 333, 5), (4, 2, 12288, 95, 4), (9, 1, 264, 21, 2),
                                                  (2, 2, 12296, 5, 3), (7, 1, 2048, 2001, 4)])
def test_expert_products_of_a_few_pairs(rows, top, K, N, experts):
    """One to nine pairs (the stream of weight rows takes up to eight), one to all of them naming an expert, one pair naming none,
    rings of thirty-two places down to four, an odd column left over, more columns than blocks: both products against the same
    in 64 bits, with the bounds of the tiles' test."""
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(K + N)
    pairs = rows * top
    choice = torch.randint(0, experts, (rows, top), generator=g, dtype=torch.int32)
    if pairs > 2:
        choice.view(-1)[pairs // 2] = -1
    h = _bf16(torch.randn(rows, K, generator=g)).to(DEV)
    w_gu = _bf16(torch.randn(experts, 2 * N, K, generator=g) * K ** -0.5).to(DEV)
    act = torch.full((pairs, N), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.moe_product_few(h, top, w_gu, None, choice.to(DEV), pairs, act, gated=True)
    y = torch.full((pairs, N), 7.0, dtype=torch.float32, device=DEV)
    w = w_gu[:, :N].contiguous()
    ops.moe_product_few(h, top, w, None, choice.to(DEV), pairs, y, gated=False)
    for p in range(pairs):
        e = int(choice.view(-1)[p])
        if e < 0:
            assert (act[p] == 7.0).all() and (y[p] == 7.0).all()
            continue
        both = w_gu[e].double() @ h[p // top].double()
        want = both[:N] * torch.sigmoid(both[:N]) * both[N:]
        slack = K ** 0.5 * 2.0 ** -22
        assert ((act[p].double() - want).abs() <= 2.0 ** -8 * want.abs() + 8 * slack).all()
        assert (y[p].double() - both[:N]).abs().max() <= 4 * slack


# ---- small kernels of a few rows ---------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("kind", ["delta", "step", "delta_channel"])
@pytest.mark.parametrize("heads,D,taps,q_heads,more,counts", [
    (2, 4, 2, 1, 8, [1, 3]), (3, 64, 4, 2, 1100, [1] * 9), (2, 128, 3, 2, 260, [5, 1, 40]), (16, 128, 4, 8, 2048, [700, 3, 650]), (4, 12, 4, 0, 20, [33])])
def test_filter_of_channels_in_fours(kind, heads, D, taps, q_heads, more, counts):
    """The short filter, unit heads, gates and kept inputs against the same in 64 bits: one row a block and runs of rows that
    cross requests, first rows with and without a history, channels that end within a block.  32-bit throughout."""
    import types
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(D + taps)
    rows, R, q_ch, k_ch = sum(counts), len(counts), q_heads * D, q_heads * D
    channels, first = q_ch + k_ch + more, 4
    stride = first + channels + 2 * heads + (-(first + channels + 2 * heads)) % 4
    proj = torch.randn(rows, stride, generator=g).to(DEV)
    w, bias = (torch.randn(channels, taps, generator=g) * 0.4).to(DEV), (torch.randn(channels, generator=g) * 0.1).to(DEV)
    per = heads * D if kind == "delta_channel" else heads
    a_log, dt_bias = (torch.randn(heads, generator=g) * 0.5).to(DEV), (torch.randn(per, generator=g) * 0.5).to(DEV)
    decay_in = torch.randn(rows, per, generator=g).to(DEV) if kind == "delta_channel" else None
    state = torch.randn(2 * R, 8 + (taps - 1) * channels, generator=g)
    state = torch.cat([state, torch.zeros(2 * R, -state.shape[1] % 4)], 1).to(DEV)
    before, off = state.clone(), 8
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    history = [0 if r % 2 == 0 else 1 + r for r in range(R)]
    starts = [sum(counts[:r]) for r in range(R)]
    step = types.SimpleNamespace(row_request=i32([r for r, n in enumerate(counts) for _ in range(n)]), row_start=i32(starts), row_count=i32(counts),
                                 history=i32(history), state_slots=i32(list(range(R))), state_slots_out=i32([R + r for r in range(R)]), requests=R)
    ready = torch.full((rows, channels), 7.0, device=DEV)
    gates = torch.full((rows, heads + per), 7.0, device=DEV)
    b_off, a_off, q_factor = first + channels, first + channels + heads, 0.3
    ops.conv_prepare(proj, channels, q_ch, k_ch, w, ready, a_log, dt_bias, b_off, a_off, gates, heads, D, q_factor, state, off, step, first=first,
                     bias=bias, gate_kind=kind, decay_in=decay_in)
    for r, n in enumerate(counts):
        rows_r = slice(starts[r], starts[r] + n)
        u = proj[rows_r, first:first + channels].double()
        old = before[r, off:off + (taps - 1) * channels].double().view(taps - 1, channels).clone()
        for s in range(taps - 1):
            if history[r] - (taps - 1) + s < 0:
                old[s] = 0.0
        seen = torch.cat([old, u])
        y = bias.double() + sum(w[:, j].double() * seen[j:j + n] for j in range(taps))
        y = y * torch.sigmoid(y)
        for lo, factor in ((0, q_factor), (q_ch, 1.0)):
            if q_ch:
                part = y[:, lo:lo + q_ch].reshape(n, q_heads, D)
                y[:, lo:lo + q_ch] = (part * factor / (part.square().sum(-1, keepdim=True) + 1e-6).sqrt()).reshape(n, q_ch)
        assert (ready[rows_r].double() - y).abs().max() <= 2e-6 * max(1.0, float(y.abs().max())), r
        assert torch.equal(state[R + r, off:off + (taps - 1) * channels].view(taps - 1, channels).double(), seen[n:]), (r, "kept inputs")
        z = (decay_in[rows_r] if kind == "delta_channel" else proj[rows_r, a_off:a_off + heads]).double() + dt_bias.double()
        dt = torch.nn.functional.softplus(z, threshold=60.0)
        decay = torch.exp(-torch.exp(a_log.double()).repeat_interleave(per // heads) * dt)
        beta = torch.sigmoid(proj[rows_r, b_off:b_off + heads].double())
        want = {"delta": [decay, beta], "step": [decay, dt], "delta_channel": [beta, decay]}[kind]
        assert (gates[rows_r].double() - torch.cat(want, 1)).abs().max() <= 2e-6 * max(1.0, float(dt.abs().max())), r
    assert torch.equal(state[:R], before[:R])


@pytest.mark.parametrize("rows,heads,D,R,V,C,splits", [(1, 2, 40, 8, 50, 264, 1), (5, 3, 128, 64, 128, 512, 3), (64, 2, 136, 0, 33, 768, 5), (2, 1, 7, 4, 1, 8, 40)])
def test_latent_maps_of_a_few_rows(rows, heads, D, R, V, C, splits):
    """The query and merge steps with bfloat16 maps against the same in 64 bits; ranges without keys (maximum minus infinity, sums
    never made) among the merged ones.  32-bit sums of D or C terms, the merged result rounded to bfloat16 (2^-9)."""
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(C + rows)
    uk, uv = _bf16(torch.randn(heads * D, C, generator=g) * C ** -0.5).to(DEV), _bf16(torch.randn(heads * V, C, generator=g) * C ** -0.5).to(DEV)
    q = torch.randn(rows, heads * (D + R) + 3, generator=g).to(DEV)[:, :heads * (D + R)]
    freq = torch.rand(R // 2, generator=g).to(DEV)
    pos = torch.arange(3, 3 + rows, dtype=torch.int32, device=DEV)
    qk = torch.full((rows, heads, C + R), 7.0, device=DEV)
    P = ops._ptr
    ops._check(ops._fn("latent_attention", "llmx_latent_query")(P(q), q.stride(0), P(uk), 1, P(qk), P(freq), R // 2, 1, 1.5, P(pos), rows, heads, D, R, C,
                                                                0.25, ops._stream()), "query")
    qh = q.double().view(rows, heads, D + R)
    want = torch.einsum("rhd,hdc->rhc", qh[:, :, :D], uk.double().view(heads, D, C)) * 0.25
    assert (qk[:, :, :C].double() - want).abs().max() <= 2.0 ** -20 * D ** 0.5 * float(want.abs().max() + 1)
    angle = (pos[:, None].float() * freq).double()[:, None, :]
    a, b = qh[:, :, D:D + R // 2], qh[:, :, D + R // 2:]
    turned = torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], 2) * 1.5 * 0.25
    assert R == 0 or (qk[:, :, C:].double() - turned).abs().max() <= 1e-5
    part = torch.randn(rows, heads, splits, C + 2, generator=g).to(DEV)
    part[..., C + 1] = part[..., C + 1].abs() + 0.5
    if splits > 1:
        part[:, :, 1] = float("nan")
        part[:, :, 1, C] = -float("inf")
    out = torch.zeros(rows, heads * V, dtype=torch.bfloat16, device=DEV)
    ops._check(ops._fn("latent_attention", "llmx_latent_merge")(P(part), P(uv), 1, P(out), rows, heads, V, C, splits, ops._stream()), "merge")
    live = [s for s in range(splits) if s != 1 or splits == 1]
    p = part[:, :, live].double()
    e = torch.exp(p[..., C] - p[..., C].amax(2, keepdim=True))
    lat = (p[..., :C] * e[..., None]).sum(2) / (p[..., C + 1] * e).sum(2, keepdim=True)
    want = torch.einsum("rhc,hvc->rhv", lat, uv.double().view(heads, V, C)).reshape(rows, -1)
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * float(lat.abs().max())).all()


@pytest.mark.parametrize("rows,width", [(1, 4), (3, 100), (8, 2048), (70, 4096), (2, 8192), (2, 8196)])
def test_norms_of_rows_in_fours(rows, width):
    """Centred, gated and paired norms of rows that a block holds in groups of four (and one width beyond): against 64 bits, 32-bit
    results within a few roundings, bfloat16 ones within one."""
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(width)
    t = lambda *shape: torch.randn(*shape, generator=g).to(DEV)
    x, w, gate, wb = t(rows, width) + 0.5, 1 + 0.1 * t(width), t(rows, width + 4)[:, :width], 1 + 0.1 * t(width)
    rms = lambda v: v / (v.square().mean(-1, keepdim=True) + 1e-5).sqrt()
    for dtype, tol in ((torch.float32, 4e-6), (torch.bfloat16, 2.0 ** -8)):
        y, zero = torch.empty(rows, width, dtype=dtype, device=DEV), torch.full((4 * 700,), 3.0, device=DEV)
        ops.layernorm(x, w, 1e-5, y, zero=zero)
        d = x.double() - x.double().mean(-1, keepdim=True)
        want = rms(d) * w.double()
        assert ((y.double() - want).abs() <= tol * (want.abs() + 0.1)).all() and not zero.any()
        for kind in (0, 1):
            for gate_first in (0, 1):
                P = ops._ptr
                ops._check(ops._fn("rowwise", "llmx_gated_rmsnorm")(P(x), P(gate), gate.stride(0), P(w), width, P(y), ops._code(y), rows, 1, width, 1e-5, kind,
                                                                    gate_first, ops._stream()), "gated")
                a = torch.sigmoid(gate.double()) * (gate.double() if kind else 1.0)
                want = rms(x.double() * a) * w.double() if gate_first else rms(x.double()) * w.double() * a
                assert ((y.double() - want).abs() <= tol * (want.abs() + 0.1)).all(), (kind, gate_first)
    a, b, s = t(rows, width), t(rows, width), t(rows, width)
    want = s.double() + 0.5 * (rms(a.double()) * w.double() + rms(b.double()) * wb.double())
    P = ops._ptr
    ops._check(ops._fn("rowwise", "llmx_pair_norm_add")(P(a), P(b), P(w), P(wb), P(s), rows, width, 1e-5, 0.5, ops._stream()), "pair")
    assert (s.double() - want).abs().max() <= 4e-6 * float(want.abs().max())


@pytest.mark.parametrize("gate_first", [False, True])
@pytest.mark.parametrize("groups,group", [(1, 1000), (3, 100), (2, 600)])
def test_a_row_of_a_gated_norm_is_the_same_alone_and_among_others(groups, group, gate_first):
    """The gate lies in rows of a wider matrix whose width is no multiple of four: one row alone takes the form that several take,
    and gives the same bits."""
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(group)
    width, rows = groups * group, 40
    o, wide, w = torch.randn(rows, width, generator=g).to(DEV), torch.randn(rows, width + 3, generator=g).to(DEV), torch.randn(group, generator=g).to(DEV)
    make = lambda s: ops.gated_rmsnorm(o[s], wide[s, :width], w, 1e-6, group, "silu", torch.empty(s.stop - s.start, width, device=DEV), gate_first=gate_first)
    among = make(slice(0, rows))
    for r in range(rows):
        assert torch.equal(make(slice(r, r + 1))[0], among[r]), r


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (8, 65, 36), (4, 4096, 256), (3, 130, 1000), (8, 65, 512), (8, 33, 508), (2, 32768, 260), (3, 32769, 260), (3, 32769, 256)])
def test_plain_products_of_few_and_many_rows_are_the_tiled_one_bit_for_bit(dtype, M, N, K):
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(K)
    a, w, c = torch.randn(130, K, generator=g).to(dtype).to(DEV), torch.randn(N, K, generator=g).to(dtype).to(DEV), torch.randn(130, N, generator=g).to(DEV)
    for accumulate in (0, 1):
        tiled, few, many = c[:40].clone(), c[:M].clone(), c.clone()
        for out in (tiled, few, many):
            ops._check(ops._fn("gemm_plain", "llmx_gemm_plain")(ops._ptr(a), ops._code(a), ops._ptr(w), ops._code(w), ops._ptr(out), out.shape[0], N, K,
                                                                accumulate, ops._stream()), "plain")
        assert torch.equal(few, tiled[:M]) and torch.equal(tiled, many[:40])
        # K multiply-adds and at most one addition, each rounded once to 2^-24 of a partial sum: (K + 1) 2^-24 of the terms' sizes.
        start = c.double() if accumulate else torch.zeros_like(c, dtype=torch.float64)
        want, sizes = a.double() @ w.double().T + start, a.double().abs() @ w.double().abs().T + start.abs()
        assert ((many.double() - want).abs() <= (K + 1) * 2.0 ** -24 * sizes).all()


def _same_bits(got, want):
    return torch.equal(torch.where(torch.isnan(got), torch.full_like(got, 7.0), got).view(torch.int32),
                       torch.where(torch.isnan(want), torch.full_like(want, 7.0), want).view(torch.int32))


def test_division_without_a_branch_is_the_division():
    """`quotient` (csrc/common.cuh) against the IEEE division of the same numbers, bit for bit: x / (1 + exp(-x)) over every 251st
    float of both signs, all divisors of one binade, the divisor with all bits set under all dividends, and random pairs of any
    exponents from 2^-100 on; below that (subnormal remainders) one unit in the last place."""
    import ctypes
    from llmx_b200.csrc import build
    fn = build.load("selftest").llmx_quotient_selftest
    fn.argtypes, fn.restype = [ctypes.c_void_p] * 3 + [ctypes.c_longlong, ctypes.c_void_p], ctypes.c_int

    def quotient(a, b):
        out = torch.empty_like(a)
        assert fn(a.data_ptr(), b.data_ptr(), out.data_ptr(), a.numel(), torch.cuda.current_stream().cuda_stream) == 0
        return out

    g = torch.Generator(device=DEV).manual_seed(5)
    floats = lambda bits: bits.to(torch.int64).to(torch.int32).view(torch.float32).clone()
    signed = lambda bits: torch.where(bits >= 2 ** 31, bits - 2 ** 32, bits)
    x = floats(signed(torch.arange(0, 2 ** 32, 251, device=DEV, dtype=torch.int64)))
    x = torch.cat([x, torch.tensor([0.0, -0.0, float("inf"), float("-inf"), float("nan"), -69.4, -88.7, -88.8, -90.0, -104.0, 1e-45, -1e-45], device=DEV)])
    b = 1.0 + torch.exp(-x)
    assert _same_bits(quotient(x, b), x / b)
    assert _same_bits(quotient(torch.ones_like(b), b), torch.ones_like(b) / b)
    mantissa = torch.arange(2 ** 23, device=DEV, dtype=torch.int64)
    one = 127 << 23
    random = lambda: torch.randint(0, 2 ** 23, (2 ** 23,), device=DEV, generator=g)
    exponent = lambda lo, hi: torch.randint(lo, hi, (2 ** 23,), device=DEV, generator=g) << 23
    for a_bits, b_bits in ((one + random(), one + mantissa), (one + mantissa, exponent(127, 254) + 2 ** 23 - 1), (exponent(27, 255) + random(), exponent(127, 255) + random())):
        a, b = floats(a_bits), floats(b_bits)
        for a in (a, -a):
            assert _same_bits(quotient(a, b), a / b)
    a, b = floats(exponent(0, 27) + random()), floats(exponent(127, 255) + random())
    assert ((quotient(a, b).view(torch.int32) - (a / b).view(torch.int32)).abs() <= 1).all()


def test_silu_of_columns_has_one_result_wherever_the_columns_lie():
    """Runs of columns in fours and runs that are not take different kernels: the same bits from both, and silu's values at zeros of
    both signs, infinities and where the exponential leaves the normal numbers."""
    from llmx_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(2)
    x = torch.cat([torch.randn(5, 40, device=DEV, generator=g) * s for s in (1.0, 30.0, 1e-30, 1e30)])
    x[0, :12] = torch.tensor([0.0, -0.0, float("inf"), float("-inf"), float("nan"), -69.4, -88.7, -88.8, -90.0, -104.0, 1e-45, -3e38], device=DEV)
    fours, single = x.clone(), torch.cat([torch.zeros(20, 1, device=DEV), x], 1)
    ops.silu_columns_(fours, 0, 40)
    ops.silu_columns_(single, 1, 40)
    assert _same_bits(fours, single[:, 1:].contiguous()) and (single[:, 0] == 0).all()
    got = fours[0, :5].tolist()
    assert got[0] == 0.0 and math.copysign(1.0, got[0]) == 1.0 and got[1] == 0.0 and math.copysign(1.0, got[1]) == -1.0
    assert got[2] == math.inf and math.isnan(got[3]) and math.isnan(got[4])          # -inf / inf is no number
    want = x.double() / (1.0 + torch.exp(-x.double()))
    # exp within two units in the last place, the sum and the division half a unit each: below 2^-21 of the value where 1 + exp(-x) is finite.
    plain = torch.isfinite(want) & (x > -88.0) & (x.abs() > 1e-37)
    assert ((fours.double() - want).abs()[plain] <= 2.0 ** -21 * want.abs()[plain]).all()


def test_gated_unit_at_extreme_inputs():
    """silu(gate) * up of an expert over gates from subnormal exponentials to infinities, 32-bit output.  Gates that are numbers:
    exp within two units in the last place, the sum, the division and the product half a unit each, together below 2^-21 of the 64-bit value
    wherever that is a normal number.  A gate beyond the largest float (the product overflows, the up row's does not) gives its
    sign's limit: plus infinity, and no number for minus infinity over infinity."""
    from llmx_b200 import ops
    gates = torch.tensor([0.0, -0.0, 1e-3, -1.0, 1.0, -20.0, -69.0, -70.0, -86.0, -88.0, -88.5, -90.0, -104.0, -1e4, 60.0, 2e38, 5.5, 3e38, -3e38])
    n = gates.numel()
    h = torch.zeros(n, 32, dtype=torch.bfloat16)
    h[:, 0], h[:, 1] = gates.bfloat16(), 1.5
    gates = h[:, 0].double()
    choice = torch.zeros(n, 1, dtype=torch.int32, device=DEV)
    lists, held = torch.empty((1, n), dtype=torch.int32, device=DEV), torch.empty((1,), dtype=torch.int32, device=DEV)
    tiles = torch.empty((ops.moe_tiles_len(n, 1),), dtype=torch.int32, device=DEV)
    for factor, cores in ((1.0, True), (1.0, False), (2.0, False)):      # twice 2e38 and 3e38: beyond the largest float
        dtype = torch.bfloat16 if cores else torch.float32
        w = torch.zeros(1, 2 * 8, 32, dtype=dtype)
        w[0, :8, 0], w[0, 8:, 1] = factor, 1.0
        out = torch.zeros(n, 8, device=DEV)
        ops.moe_route(None, choice, 1, lists, held, tiles, tensor_cores=cores)
        ops.moe_product(h.to(dtype).to(DEV), 1, w.to(DEV), lists, held, tiles, n, out, gated=True, tensor_cores=cores)
        got = out[:, 0].cpu().double()
        z = factor * gates
        finite = z.abs() < 3.4e38
        want = 1.5 * z / (1.0 + torch.exp(-z))
        normal = finite & (want.abs() > 2e-37) & (want.abs() < 3.4e38)
        assert ((got - want).abs()[normal] <= 2.0 ** -21 * want.abs()[normal]).all() and (got[finite & (want.abs() <= 2e-37)].abs() <= 2.1e-37).all()
        assert (got[(z > 3.4e38) | (want > 3.4e38)] == math.inf).all() and torch.isnan(got[z < -3.4e38]).all()


@pytest.mark.parametrize("heads,kv_heads,page,window,chunk", [(4, 1, 16, None, None), (3, 1, 32, 70, None), (32, 2, 48, None, 96), (2, 2, 16, 1, None), (10, 2, 16, 64, 200)])
@pytest.mark.parametrize("counts,histories", [([5], [0]), ([128, 1, 33], [0, 63, 64]), ([65, 7], [700, 130]), ([300], [1]),
                                              ([1 + r % 3 for r in range(210)], [(37 * r) % 130 for r in range(210)])])
def test_attention_of_rows_that_share_their_keys(heads, kv_heads, page, window, chunk, counts, histories):
    """The tcgen05 form of the tiled attention against 64 bits: runs of rows below, at and above a tile, as many requests as give
    every SM a second tile and some a third (210 or 420 tiles on 148), padded head groups, windows and chunks that begin within a stage; every slot of the cache that no row may see holds NaN, pages below a window are
    given back.  Weights keep 24 bits, so the result's own rounding decides: twice its 2^-9 are allowed (how exactly the sums behind it
    are made, `test_attention_over_many_keys_rounds_as_the_exact_one` counts)."""
    import types
    from llmx_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(heads + page)
    rows, scale = sum(counts), 0.1
    needs = [-(-(h + n) // page) for h, n in zip(histories, counts)]
    order = torch.randperm(sum(needs), generator=torch.Generator().manual_seed(1)).tolist()
    tables, at = torch.full((len(counts), max(needs)), -1, dtype=torch.int32), 0
    cache = torch.full((sum(needs) + 1, 1, kv_heads, page, 256), float("nan"), device="cuda", dtype=torch.bfloat16)
    lowest = lambda p: max(max(0, p - window + 1) if window else 0, p // chunk * chunk if chunk else 0)
    kv = []
    for r, (n, h) in enumerate(zip(counts, histories)):
        mine = order[at:at + needs[r]]
        at += needs[r]
        tables[r, :needs[r]] = torch.tensor(mine)
        rows_r = torch.randn(h + n, kv_heads, 256, device="cuda", generator=g).bfloat16()
        kv.append(rows_r.double())
        lo = lowest(h)
        t = torch.arange(lo, h + n, device="cuda")
        cache[torch.tensor(mine, device="cuda")[t // page], 0, :, t % page] = rows_r[lo:]
        tables[r, :lo // page] = -1
    q = torch.randn(rows, heads * 128, device="cuda", generator=g).bfloat16()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    step = types.SimpleNamespace(row_start=i32([sum(counts[:r]) for r in range(len(counts))]), row_count=i32(counts), history=i32(histories), requests=len(counts),
                                 rows=rows)
    out = torch.zeros(rows, heads * 128, device="cuda", dtype=torch.bfloat16)
    ops.attention_tiled(q, cache, out, step, tables.cuda(), heads, kv_heads, 128, 128, window, chunk, scale)
    from llmx_b200.runtime import check_errors
    check_errors()
    row = 0
    for r, (n, h) in enumerate(zip(counts, histories)):
        k, v = (x.repeat_interleave(heads // kv_heads, 1) for x in kv[r].split(128, 2))
        for p in range(h, h + n):
            lo = lowest(p)
            s = torch.einsum("hd,thd->ht", q[row].double().view(heads, 128), k[lo:p + 1]) * scale
            want = torch.einsum("ht,thd->hd", torch.softmax(s, 1), v[lo:p + 1]).reshape(-1)
            bound = 2.0 ** -8 * want.abs() + 2.0 ** -19 * (1.0 + s.abs().max()) * v[lo:p + 1].abs().max()
            assert ((out[row].double() - want).abs() <= bound).all(), (r, p)
            row += 1


@pytest.mark.parametrize("bits", [3, 64, 120, 126.3, 128.5, 131])
def test_softmax_weights_below_the_normal_numbers_count(bits):
    """Two keys, the second 2^-bits of the first in weight, its value 2^120, the first's zero: the result is that product, also where
    the weight is no normal number any more (below 2^-126 it keeps what a bfloat16 holds of it, multiples of 2^-133), by the tcgen05
    forms over [key ; value] rows and over latents.  The score is a 32-bit product, its exponent's error below 2^-16 of the weight."""
    import types
    from llmx_b200 import ops
    from llmx_b200.runtime import check_errors
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    score = torch.tensor(-bits * math.log(2.0)).bfloat16().item()
    want = 2.0 ** 120 * math.exp(score) / (1.0 + math.exp(score))
    bound = 2.0 ** -8 * want + 2.0 ** -16 * want + (2.0 ** -133 * 2.0 ** 120 if bits > 125 else 0.0)
    cache = torch.zeros(1, 1, 1, 16, 256, device="cuda", dtype=torch.bfloat16)
    cache[0, 0, 0, 1, 0], cache[0, 0, 0, 1, 128:] = score, 2.0 ** 120
    q = torch.zeros(2, 128, device="cuda", dtype=torch.bfloat16)
    q[:, 0] = 1.0
    step = types.SimpleNamespace(row_start=i32([0]), row_count=i32([2]), history=i32([0]), requests=1, rows=2)
    rows = torch.zeros(2, 128, device="cuda", dtype=torch.bfloat16)
    ops.attention_tiled(q, cache, rows, step, i32([[0]]), 1, 1, 128, 128, None, None, 1.0)
    latent = torch.zeros(1, 1, 1, 16, 64 + 8, device="cuda", dtype=torch.bfloat16)
    latent[0, 0, 0, 1, 0], latent[0, 0, 0, 1, 64] = 2.0 ** 60, score
    w_uk, w_uv = torch.zeros(128, 64, device="cuda", dtype=torch.bfloat16), torch.zeros(128, 64, device="cuda", dtype=torch.bfloat16)
    w_uv[:, 0] = 2.0 ** 60
    ql = torch.zeros(2, 128 + 8, device="cuda")
    ql[:, 128] = 1.0
    made = torch.zeros(2, 128, device="cuda", dtype=torch.bfloat16)
    ops.latent_attention_prompt(ql, latent, w_uk, w_uv, made, torch.zeros(0, device="cuda"), i32([0, 0]), i32([0, 1]), i32([[0]]), i32([0, 2, 0, 128]), 1, 128,
                                i32([0, 2, 0, 0]), 1, 128, 1, 1, 128, 8, 128, 64, 16, None, 1.0)
    check_errors()
    for how, out in (("rows", rows), ("latents", made)):
        assert (out[0] == 0).all() and ((out[1].double() - want).abs() <= bound).all(), (how, out[1, 0].item(), want)


@pytest.mark.parametrize("mean", [0.0, 1.0])
@pytest.mark.parametrize("keys", [300, 2048, 8192])
def test_attention_over_many_keys_rounds_as_the_exact_one(keys, mean):
    """How many results round to another bfloat16 than the 64-bit ones, by the tcgen05 form and by the form on mma.sync (which the
    kernel's entry runs whatever the widths).  A stage of 64 keys is cut off at each of its twelve additions, the stages are
    joined by rounded ones, so with values of one sign the error stays below 12 x 2^-23 of the result however many keys there are:
    12 x 2^-23 / 2^-8 = 4e-4 of the results at most lie that close to a bfloat16's edge.  With values of both signs the sums are larger
    than the result: no more than the other form, whose accumulators run through all keys."""
    import types
    from llmx_b200 import ops
    from llmx_b200.runtime import check_errors
    g = torch.Generator(device="cuda").manual_seed(keys)
    rows, heads, kv_heads, scale = 64, 16, 4, 128 ** -0.5
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    cache = torch.randn(-(-keys // 16), 1, kv_heads, 16, 256, device="cuda", generator=g)
    cache[..., 128:] += mean
    cache = cache.bfloat16()
    q = torch.randn(rows, heads * 128, device="cuda", generator=g).bfloat16()
    tables = torch.arange(cache.shape[0], dtype=torch.int32, device="cuda")[None].contiguous()
    step = types.SimpleNamespace(row_start=i32([0]), row_count=i32([rows]), history=i32([keys - rows]), requests=1, rows=rows)
    out, other = (torch.zeros(rows, heads * 128, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    ops.attention_tiled(q, cache, out, step, tables, heads, kv_heads, 128, 128, None, None, scale)
    P = ops._ptr
    ops._check(ops._fn("attention_split", "llmx_attention_tiled")(
        P(q), P(cache), P(other), P(step.row_start), P(step.row_count), P(step.history), P(tables), tables.shape[1], rows, 1, heads, kv_heads, 128, 128, 16, 0, 0,
        scale, *ops.NO_EXTRAS.checked(heads, 128, rows), ops._stream()), "attention_tiled")
    check_errors()
    kv = cache[:, 0].transpose(1, 2).reshape(-1, kv_heads, 256)[:keys].double()
    unseen = torch.arange(keys, device="cuda")[None] > torch.arange(keys - rows, keys, device="cuda")[:, None]
    want = torch.empty(rows, heads, 128, device="cuda", dtype=torch.float64)
    for h in range(heads):
        k, v = kv[:, h // (heads // kv_heads)].split(128, 1)
        want[:, h] = torch.softmax((q.view(rows, heads, 128)[:, h].double() @ k.T * scale).masked_fill(unseen, -math.inf), 1) @ v
    nearest = want.float().bfloat16().view(rows, -1)
    share, before = ((x != nearest).double().mean().item() for x in (out, other))
    assert share <= (4e-4 if mean else max(before, 4e-4)), (share, before)


@pytest.mark.parametrize("mean,spread", [(0.5, 0.1), (0.5, 1.0), (0.0, 1.0)])
@pytest.mark.parametrize("history", [0, 512])
def test_latent_prompts_round_as_the_exact_ones(mean, spread, history):
    """How many results round to another bfloat16 than the 64-bit ones: no more in the form for many rows, whose keys, values, scores
    and outputs pass through the tensor cores' accumulators, than in the general form.  Latents of one sign and of both, even
    and peaked scores; a twentieth is left for chance (the counts are in the hundreds)."""
    from llmx_b200 import ops
    from llmx_b200.parts.base import Precision, StepShape
    from llmx_b200.parts.latent_attention import LatentAttention
    from llmx_b200.runtime import check_errors
    g = torch.Generator(device="cuda").manual_seed(history)
    rows, heads, latent, rot, page, scale = 512, 8, 512, 64, 16, 192 ** -0.5 * spread
    part = LatentAttention(64, heads, 128, rot, 128, None, latent, scale, 1e4, rot, 1e-6, None)
    part.precision, part._sms = Precision.of("bfloat16"), 148
    part.w_uk, part.w_uv = (torch.randn(heads * 128, latent, device="cuda", generator=g).mul_(latent ** -0.5).bfloat16() for _ in range(2))
    freq = torch.from_numpy(part.frequencies()[0]).cuda()
    plan = part.plan_step(StepShape([rows], [history]))
    ints = torch.tensor(plan.values, device="cuda")
    keys = rows + history
    cache = torch.randn(keys // page, 1, 1, page, latent + rot, device="cuda", generator=g)
    cache[..., :latent] += mean
    cache = cache.bfloat16()
    q = torch.randn(rows, heads * (128 + rot), device="cuda", generator=g)
    positions = torch.arange(history, keys, dtype=torch.int32, device="cuda")
    meta = torch.zeros(rows, dtype=torch.int32, device="cuda"), positions, torch.arange(keys // page, dtype=torch.int32, device="cuda")[None].contiguous()
    sizes = (heads, 128, rot, 128, latent, page, None, scale)
    out, general = (torch.zeros(rows, heads * 128, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    first, n_req, share, tiles_at, n_tiles, tokens, group = plan.wide
    ops.latent_attention_prompt(q, cache, part.w_uk, part.w_uv, out, freq, *meta, ints[first:], n_req, share, ints[tiles_at:], n_tiles, tokens, group, *sizes)
    _, _, at, n_tiles, splits = plan.whole
    ops.latent_attention_tiled(q, cache, part.w_uk, part.w_uv, general, freq, *meta, ints[at:], n_tiles, splits, *sizes)
    check_errors()
    c, pos = cache.view(-1, latent + rot).double(), positions.double()
    angle = (positions[:, None].float() * freq[None]).double()
    unseen = torch.arange(keys, device="cuda")[None] > positions[:, None]
    want = torch.empty(rows, heads, 128, device="cuda", dtype=torch.float64)
    for h in range(heads):
        x = q.view(rows, heads, -1)[:, h].double()
        a, b = x[:, 128::2], x[:, 129::2]
        turned = torch.stack([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], 2).reshape(rows, rot)
        uk, uv = (w[h * 128:(h + 1) * 128].double() for w in (part.w_uk, part.w_uv))
        s = (x[:, :128] @ (uk @ c[:, :latent].T) + turned @ c[:, latent:].T) * scale
        want[:, h] = torch.softmax(s.masked_fill(unseen, -math.inf), 1) @ (c[:, :latent] @ uv.T)
    nearest = want.float().bfloat16().view(rows, -1)
    made, before = ((o != nearest).double().mean().item() for o in (out, general))
    assert made <= 1.05 * before, (made, before)


@pytest.mark.parametrize("experts,top,rows,K,N", [(16, 2, 300, 576, 160), (1500, 1, 900, 32, 96), (6000, 2, 200, 96, 32), (3, 3, 700, 160, 416),
                                                  (128, 2, 300, 64, 96), (129, 2, 300, 64, 96), (8193, 1, 300, 32, 64), (9000, 2, 5000, 32, 32),
                                                  (8192, 1, 8300, 32, 32)])
def test_expert_products_in_sorted_rows(experts, top, rows, K, N):
    """The gated product leaves its rows in the lists' order and the plain one reads them there: every pair's result against 64 bits of
    the same bfloat16 steps, experts so many that fewer stages fit beside their numbers or that the numbers lie apart, the last number of
    experts that all have a place and the first that are listed, widths that end within a unit."""
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(experts + N)
    table = torch.rand(rows, experts, generator=g).argsort(1)[:, :top].to(torch.int32).contiguous().to(DEV)
    h = _bf16(torch.randn(rows, K, generator=g)).to(DEV)
    w_gu = _bf16(torch.randn(experts, 2 * N, K, generator=g) * K ** -0.5).to(DEV)
    w = _bf16(torch.randn(experts, K, N, generator=g) * N ** -0.5).to(DEV)
    pairs = rows * top
    lists = torch.empty((experts, pairs), dtype=torch.int32, device=DEV)
    counts = torch.empty((experts,), dtype=torch.int32, device=DEV)
    ops.moe_route(None, table, experts, lists, counts, None, tensor_cores=True)
    act = torch.full((pairs, N), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.moe_product_sorted(ops.moe_gather(h, top, lists, counts, pairs), w_gu, lists, counts, pairs, act, gated=True, out_sorted=True)
    y = torch.full((pairs, K), 7.0, device=DEV)
    ops.moe_product_sorted(act, w, lists, counts, pairs, y, gated=False)
    at = torch.cat([lists[e, :n] for e, n in enumerate(counts.tolist())]).long()
    expert = table.reshape(-1)[at].long()
    both = torch.einsum("pk,pnk->pn", h.double()[at // top], w_gu.double()[expert])
    want = both[:, :N] * torch.sigmoid(both[:, :N]) * both[:, N:]
    slack = K ** 0.5 * 2.0 ** -22
    assert ((act.double() - want).abs() <= 2.0 ** -8 * want.abs() + 8 * slack).all()
    want = torch.einsum("pn,pkn->pk", act.double(), w.double()[expert])
    assert (y[at].double() - want).abs().max() <= 4 * N ** 0.5 * 2.0 ** -22 * max(1.0, float(act.abs().max()))


@pytest.mark.parametrize("rows,n,k,offset", [(65, 128, 4, 0), (66, 2, 20, 1), (130, 200, 64, 3), (300, 4096, 256, 4), (777, 514, 132, 2)])
def test_product_in_parts(rows, n, k, offset):
    """A 32-bit product whose factors are cut into three bfloat16 parts, over strided rows at any offset, against 64 bits.  Bound, in
    2^-24 of the terms' absolute sum: 4 for the parts' products left out and the last parts' rounding; 8 for a group's additions on the
    tensor cores, which cut sums off (four whose sums are of full size and one between the runs, the smaller runs' a 256th of
    that); one for each group's addition.  (Leaving out a product of parts that counts is further off at every width here.)  Numbers that are not finite, and the largest one, come out as from the plain product."""
    from llmx_b200.parts.base import Precision
    from llmx_b200.parts.linear import SplitLinear
    g = torch.Generator().manual_seed(rows)
    wide = torch.randn(rows, k + 8, generator=g).to(DEV)
    w = (0.1 * torch.randn(n, k, generator=g)).to(DEV)
    lin = SplitLinear(w, Precision.of("bfloat16"))
    assert (lin.parts is not None) == (k >= 64)          # narrower ones run the plain product
    a = wide[:, offset:offset + k]
    got = lin.of_rows(a).double()
    want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    groups = -(-k // 64)
    assert bool(((got - want).abs() <= (12 + groups if lin.parts is not None else k + 1) * 2.0 ** -24 * size).all())
    wide[0, offset], wide[1, offset + 1], wide[2, offset + 2] = float("inf"), float("nan"), torch.finfo(torch.float32).max
    got, plain = lin.of_rows(a), lin(a.contiguous())
    assert torch.equal(torch.isnan(got), torch.isnan(plain)) and torch.equal(torch.isinf(got), torch.isinf(plain))
    assert torch.allclose(got[2], plain[2], rtol=1e-5)


@pytest.mark.parametrize("signs", ["both", "one", "mean"])
@pytest.mark.parametrize("k", [64, 68, 100, 128, 132, 192, 252, 256])
def test_product_in_parts_is_no_further_off_than_the_plain_one(k, signs):
    """Error norms against 64 bits: the product in parts' is at most the plain product's, for terms of both signs, of one sign and
    with a mean, at the narrowest width that it takes (one group of 64 values), with parts of groups and at the widest.  (Sums that the
    tensor cores cut off over the whole width are further off from 128 values of one sign on.)"""
    from llmx_b200.parts.base import Precision
    from llmx_b200.parts.linear import Linear, SplitLinear
    g = torch.Generator().manual_seed(k)
    a, w = torch.randn(300, k, generator=g), 0.1 * torch.randn(515, k, generator=g)
    if signs == "one":
        a, w = a.abs(), w.abs()
    if signs == "mean":
        a, w = a + 1.0, w + 0.1
    a, w = a.to(DEV), w.to(DEV)
    lin = SplitLinear(w, Precision.of("bfloat16"))
    assert lin.parts is not None
    got, plain, want = lin.of_rows(a), Linear.__call__(lin, a), a.double() @ w.double().T
    assert not torch.equal(got, plain)
    assert (got.double() - want).norm() <= (plain.double() - want).norm()
    assert torch.equal(got, lin.of_rows(a))              # one order of sums


@pytest.mark.parametrize("maps", [1, 2])
@pytest.mark.parametrize("value_dim", [40, 128, 192])
@pytest.mark.parametrize("splits", [1, 7, 9, 33, 64])
def test_ranges_without_keys_are_left_out_of_the_merge(maps, value_dim, splits):
    """More ranges than keys: rows of 1, 3, 40 and 200 keys against the same in one range, in both forms that leave ranges, over scratch
    memory full of NaN: what no range has written is not used.  Bound: 32-bit sums in another order, 64 terms of at most 4 each, with
    the difference's norm behind them."""
    from llmx_b200 import ops
    heads, kv_heads, key_dim, page = 4, 2, 64, 16
    g = torch.Generator().manual_seed(splits)
    lengths = [1, 3, 40, 200]
    pages = [(x + page - 1) // page for x in lengths]
    table = torch.zeros(4, max(pages), dtype=torch.int32)
    at = 0
    for r, p in enumerate(pages):
        table[r, :p] = torch.arange(at, at + p)
        at += p
    cache = torch.randn(at, 1, kv_heads, page, maps * key_dim + value_dim, generator=g).to(DEV)
    q = torch.randn(4, heads * maps * key_dim, generator=g).to(DEV)
    req, pos = torch.arange(4, dtype=torch.int32, device=DEV), torch.tensor([x - 1 for x in lengths], dtype=torch.int32, device=DEV)
    extras = ops.SoftmaxExtras(difference=(0.4, 0.8, 1e-6)) if maps == 2 else None
    want = torch.empty(4, heads * value_dim, device=DEV)
    ops.attention_split(q, cache, want, req, pos, table.to(DEV), heads, kv_heads, key_dim, value_dim, None, None, key_dim ** -0.5, extras=extras)
    table = table.to(DEV)
    x = (extras or ops.NO_EXTRAS).checked(heads, value_dim, 4)
    for form in ("llmx_attention_split", "llmx_attention_staged"):
        out = torch.empty(4, heads * value_dim, device=DEV)
        partial = torch.full((4, heads * maps, splits, value_dim + 2), float("nan"), device=DEV)
        ops._check(ops._fn("attention_split", form)(
            ops._ptr(q), ops._code(q), ops._ptr(cache), ops._code(cache), ops._ptr(out), ops._ptr(req), ops._ptr(pos), ops._ptr(table), table.shape[1], 4,
            heads * maps, kv_heads, key_dim, value_dim, page, 0, 0, key_dim ** -0.5, splits, ops._ptr(partial), *x, ops._stream()), form)
        assert bool(torch.isfinite(out).all()), form
        assert torch.allclose(out, want, rtol=2e-5, atol=2e-5), form


@pytest.mark.parametrize("splits", [1, 7])
def test_two_maps_of_a_row_without_keys_give_zeros(splits):
    """A position of -1 sees no key: both maps' sums are empty, and the row's output is zero, as is their difference's norm (the row
    beside it has keys)."""
    from llmx_b200 import ops
    heads, kv_heads, key_dim, value_dim, page = 4, 2, 64, 64, 16
    g = torch.Generator().manual_seed(5)
    cache = torch.randn(2, 1, kv_heads, page, 2 * key_dim + value_dim, generator=g).to(DEV)
    q = torch.randn(2, heads * 2 * key_dim, generator=g).to(DEV)
    req, table = torch.arange(2, dtype=torch.int32, device=DEV), torch.tensor([[0], [1]], dtype=torch.int32, device=DEV)
    out = torch.full((2, heads * value_dim), 7.0, device=DEV)
    ops.attention_split(q, cache, out, req, torch.tensor([-1, 11], dtype=torch.int32, device=DEV), table, heads, kv_heads, key_dim, value_dim,
                        None, None, key_dim ** -0.5, splits=splits, extras=ops.SoftmaxExtras(difference=(0.4, 0.8, 1e-6)))
    assert bool((out[0] == 0).all()) and bool(torch.isfinite(out[1]).all()) and bool((out[1] != 0).any())


def test_latent_scores_take_queries_at_any_offset():
    """Rows of queries at the start of an allocation and a float further (not on 16 bytes): the same partial states, bit for bit."""
    from llmx_b200 import ops
    rows, heads, C, R, page, keys = 3, 4, 128, 32, 16, 70
    g = torch.Generator().manual_seed(9)
    cache = _bf16(torch.randn(5, 1, 1, page, C + R, generator=g)).to(DEV)
    whole = torch.randn(rows * heads * (C + R) + 1, generator=g).to(DEV)
    further = whole[1:]
    start = further.clone()
    assert further.data_ptr() % 16 == 4 and start.data_ptr() % 16 == 0
    tiles = torch.tensor([[0, rows]], dtype=torch.int32, device=DEV)
    req, pos = torch.zeros(rows, dtype=torch.int32, device=DEV), torch.arange(keys - rows, keys, dtype=torch.int32, device=DEV)
    table = torch.arange(5, dtype=torch.int32, device=DEV).view(1, 5)
    parts = []
    for qk in (start, further):
        part = torch.zeros(rows, heads, 1, C + 2, device=DEV)
        ops._check(ops._fn("latent_attention", "llmx_latent_scores")(ops._ptr(qk), ops._ptr(cache), ops._code(cache), ops._ptr(part), ops._ptr(tiles), 1, 1,
                                                                     ops._ptr(req), ops._ptr(pos), ops._ptr(table), 5, heads, C, R, page, 0, 0,
                                                                     ops._stream()), "scores")
        parts.append(part)
    assert bool((parts[0] != 0).any()) and torch.equal(parts[0], parts[1])


def test_expert_products_of_a_few_pairs_wait_for_ids_that_a_draw_has_just_written():
    """Ids handed over straight from a draw (a kernel that lets its followers start early): without `settled` the product reads them only
    when they are there, and gives what it gives for the same ids once everything has ended; so does `settled` then."""
    from llmx_b200 import ops
    from llmx_b200.sampling import sampler
    rows, top, experts, vocab, K, N = 4, 2, 16, 32768, 64, 48
    g = torch.Generator().manual_seed(3)
    table = torch.rand(vocab, experts, generator=g).argsort(1)[:, :top].to(torch.int32).contiguous().to(DEV)
    h = _bf16(torch.randn(rows, K, generator=g)).to(DEV)
    w = _bf16(torch.randn(experts, 2 * N, K, generator=g)).to(DEV)
    settings = sampler._packer(rows).pack(*(rows * (0.0, 1.0, 0.0, 0.0, 0, -1)))
    ids, seen = torch.zeros(rows, dtype=torch.int32, device=DEV), set()
    product = lambda **kw: ops.moe_product_few(h, top, w, ids, table, rows * top, torch.full((rows * top, N), 7.0, dtype=torch.bfloat16, device=DEV), gated=True, **kw)
    first = product()
    for i in range(20):
        logits, out = torch.randn(rows, vocab, generator=g).to(DEV), torch.full_like(first, 7.0)
        torch.cuda.synchronize()
        ops._check(ops._fn("sampling", "llmx_sample_rows")(ops._ptr(logits), rows, vocab, settings, ops._ptr(ids), 1, ops._stream()), "sample")
        ops.moe_product_few(h, top, w, ids, table, rows * top, out, gated=True)
        torch.cuda.synchronize()
        assert torch.equal(ids.long(), logits.argmax(1)) and torch.equal(out, product()) and torch.equal(out, product(settled=True)), i
        seen.add(tuple(ids.tolist()))
    assert len(seen) > 1


@pytest.mark.parametrize("tensor_cores", [False, True])
def test_expert_products_read_the_counts_that_the_routing_wrote(tensor_cores):
    """A buffer of counts longer than the experts: what lies behind theirs is nobody's count."""
    from llmx_b200 import ops
    experts, rows, K, N = 3, 40, 64, 96
    g = torch.Generator().manual_seed(2)
    choice = torch.randint(0, experts, (rows, 1), generator=g, dtype=torch.int32)
    h, w = _bf16(torch.randn(rows, K, generator=g)).to(DEV), _bf16(torch.randn(experts, N, K, generator=g)).to(DEV)
    lists, tiles = torch.empty((experts, rows), dtype=torch.int32, device=DEV), torch.empty((ops.moe_tiles_len(rows, experts),), dtype=torch.int32, device=DEV)
    counts = torch.full((experts + 5,), 1 << 20, dtype=torch.int32, device=DEV)
    ops.moe_route(None, choice.to(DEV), experts, lists, counts, tiles, tensor_cores=tensor_cores)
    out = ops.moe_product(h, 1, w, lists, counts, tiles, rows, torch.zeros(rows, N, device=DEV), gated=False, tensor_cores=tensor_cores)
    want = torch.einsum("rk,rnk->rn", h.double(), w.double()[choice[:, 0].long().to(DEV)])
    assert (out.double() - want).abs().max() <= 4 * K ** 0.5 * 2.0 ** -22 * 8


def test_launches_of_a_routing_are_counted_as_they_are():
    """One kernel lists the pairs; the second one, which cuts tiles, runs only where tiles are wanted."""
    from llmx_b200 import ops
    choice = torch.zeros(5, 1, dtype=torch.int32, device=DEV)
    lists, counts = torch.empty((2, 5), dtype=torch.int32, device=DEV), torch.empty((2,), dtype=torch.int32, device=DEV)
    for tiles, launches in ((None, 1), (torch.empty((ops.moe_tiles_len(5, 2),), dtype=torch.int32, device=DEV), 2)):
        before = ops.launch_count()
        ops.moe_route(None, choice, 2, lists, counts, tiles, tensor_cores=True)
        assert ops.launch_count() - before == launches


@pytest.mark.parametrize("rows", [1, 64, 65])
@pytest.mark.parametrize("D,V,half", [(64, 64, 0), (64, 40, 32), (128, 128, 32), (128, 96, 64), (256, 256, 32), (256, 64, 96), (256, 128, 128), (128, 128, 24)])
def test_queries_and_keys_of_lanes_that_turn_their_own_pairs(rows, D, V, half):
    """Norm, rotation and write of heads of 64, 128 and 256 with nothing, a part and all of a head turned (a lane then holds both values of
    a pair; 24 pairs take the general kernel), steps on both sides of the line by rows, skipped slots, all types: against 64 bits of the
    same 32-bit angles.  Bound: sums of D squares and the norm's division, the sine's two units, a product and a sum: 2^-19 of the
    row's largest value (which the norm leaves below 16), and the type's rounding."""
    from llmx_b200 import ops
    heads, kv_heads, page = 5, 3, 16
    g = torch.Generator().manual_seed(D + V + half + rows)
    proj = torch.randn(rows, (heads + kv_heads) * D + kv_heads * V, generator=g)
    pos = torch.randint(0, 3000, (rows,), generator=g, dtype=torch.int32)
    slots = torch.randperm(6 * page, generator=g)[:rows].to(torch.int32)
    slots[rows // 2] = -1
    freq = torch.rand(half, generator=g) if half else None
    for norm in (False, True):
        qw, kw = (torch.rand(2, D, generator=g) + 0.5) if norm else (None, None)
        x = proj[:, :(heads + kv_heads) * D].double().view(rows, heads + kv_heads, D)
        if norm:
            x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6) * torch.cat([qw.expand(heads, D), kw.expand(kv_heads, D)]).double()
        want = x.clone()
        if half:
            angle = (pos.float()[:, None] * freq[None]).double()[:, None]
            lo, hi = x[..., :half], x[..., half:2 * half]
            want[..., :half], want[..., half:2 * half] = lo * angle.cos() - hi * angle.sin(), hi * angle.cos() + lo * angle.sin()
        values = proj[:, (heads + kv_heads) * D:].double().view(rows, kv_heads, V)
        for q_type in (torch.float32, torch.bfloat16):
            for c_type in (torch.float32, torch.bfloat16):
                q_out = torch.full((rows, heads * D), 7.0, dtype=q_type, device=DEV)
                cache = torch.full((6, 1, kv_heads, page, D + V), 7.0, dtype=c_type, device=DEV)
                ops.qk_norm_rope_write(proj.to(DEV), heads, kv_heads, D, V, None if qw is None else qw.to(DEV), None if kw is None else kw.to(DEV), 1e-6,
                                       None if freq is None else freq.to(DEV), pos.to(DEV), slots.to(DEV), q_out, cache)
                near = lambda got, ref, kind: bool(((got - ref).abs() <= 16 * 2.0 ** -19 + (2.0 ** -8 if kind is torch.bfloat16 else 0.0) * ref.abs()).all())
                assert near(q_out.cpu().double().view(rows, heads, D), want[:, :heads], q_type)
                held = cache.cpu().double()[:, 0].permute(0, 2, 1, 3).reshape(6 * page, kv_heads, D + V)
                kept = slots >= 0
                at = slots[kept].long()
                assert near(held[at][..., :D], want[kept][:, heads:], c_type) and near(held[at][..., D:], values[kept], c_type)
                rest = torch.ones(6 * page, dtype=torch.bool)
                rest[at] = False
                assert bool((held[rest] == 7.0).all())


@pytest.mark.parametrize("rows,width", [(1, 4), (3, 1020), (2, 1024), (5, 1028), (2, 4100), (3, 1022)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_clamped_unit_in_fours(rows, width, out_dtype):
    """Widths of one thread, below, at and above a block of 1,024 values, several blocks, and one that is not in fours: against 64 bits,
    values on both sides of the limits.  Bound: the exponential's two units, a sum, a division and two products, below 2^-20 of the
    result; its argument alpha g, rounded once from a rounded alpha, moves it by 2^-23 of alpha g; and the type's rounding."""
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(width)
    gu = 4 * torch.randn(rows, 2 * width, generator=g)
    gu[0, 0], gu[0, width] = -90.0, 50.0
    out = ops.clamped_glu(gu.to(DEV), torch.empty(rows, width, dtype=out_dtype, device=DEV), 1.5, 1.702).cpu().double()
    gate, up = gu[:, :width].double().clamp(max=1.5), gu[:, width:].double().clamp(-1.5, 1.5)
    want = gate / (1.0 + torch.exp(-1.702 * gate)) * (up + 1.0)
    bound = 2.0 ** -20 + 2.0 ** -23 * (1.702 * gate).abs() + (2.0 ** -8 if out_dtype is torch.bfloat16 else 0.0)
    assert bool(((out - want).abs() <= bound * want.abs() + 1e-30).all())


@pytest.mark.parametrize("rows", [128, 129, 200])
def test_sampling_of_more_rows_than_a_launch_carries(rows):
    """Up to 128 rows' settings travel with the launch, more in a buffer on the device, kept where all rows are greedy: both against the
    plain sampler, greedy rows twice with the same masked ids and once with others."""
    rng = np.random.default_rng(rows)
    vocab = 3001
    logits = (3 * rng.standard_normal((rows, vocab))).astype(np.float32)
    settings = [dict(temp=float(rng.choice([0.0, 0.7, 1.2])), top_k=int(rng.choice([0, 5, 40])), top_p=float(rng.choice([1.0, 0.9])), seed=r + 1,
                     masked=int(rng.integers(-1, 5))) for r in range(rows)]
    plainly = lambda some: [plain.sample(row, s["temp"], s["top_k"], s["top_p"], 0.0, 0.0 if s["temp"] <= 0 else plain.XorShift64(s["seed"]).unit(),
                                         masked=s["masked"]) for row, s in zip(logits, some)]
    assert _sample_rows(logits.copy(), settings)[0] == plainly(settings)
    greedy = [dict(s, temp=0.0) for s in settings]
    best = logits.argmax(1)
    other = [dict(s, masked=int(best[r])) for r, s in enumerate(greedy)]
    for some in (greedy, greedy, other, greedy):
        assert _sample_rows(logits.copy(), some)[0] == plainly(some)


@pytest.mark.parametrize("counts", [[1, 0, 15, 16, 17], [255, 256, 257], [127, 128, 129, 512, 513], [272, 3]])
@pytest.mark.parametrize("K,N,clamp", [(32, 32, None), (160, 96, (1.5, 1.7)), (96, 256, (1.5, 1.7))])
def test_expert_products_at_the_edges_of_their_parts_as_steps_run_them(counts, K, N, clamp):
    """Gathered rows, the gated product left in their order and the product back by pair: experts whose pairs end just below, at and
    above a part or in several equal ones, two pairs a row, every seventh row naming an expert without weights (its pairs lie past the
    lists and keep what they held).  Bounds as in the test of the tiles' edges."""
    from llmx_b200 import ops
    g = torch.Generator().manual_seed(K + N)
    experts, named = len(counts), sum(counts)
    lost = named // 7 + (named + named // 7) % 2
    pairs = named + lost
    choice = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(counts + [lost])])
    choice[choice == experts] = experts + 5
    choice = choice[torch.randperm(pairs, generator=g)]
    h = _bf16(torch.randn(pairs // 2, K, generator=g)).to(DEV)
    w_gu, w = (_bf16(torch.randn(experts, a, b, generator=g) * b ** -0.5).to(DEV) for a, b in ((2 * N, K), (K, N)))
    lists, held = torch.empty((experts, pairs), dtype=torch.int32, device=DEV), torch.empty((experts,), dtype=torch.int32, device=DEV)
    ops.moe_route(None, choice.view(-1, 2).to(DEV), experts, lists, held, None, tensor_cores=True)
    assert held.tolist() == counts
    act, y = torch.full((pairs, N), 7.0, dtype=torch.bfloat16, device=DEV), torch.full((pairs, K), 7.0, device=DEV)
    ops.moe_product_sorted(ops.moe_gather(h, 2, lists, held, pairs), w_gu, lists, held, pairs, act, gated=True, out_sorted=True, clamp=clamp)
    ops.moe_product_sorted(act, w, lists, held, pairs, y, gated=False)
    at = torch.cat([lists[e, :n] for e, n in enumerate(counts)]).long()
    e = choice.to(DEV)[at].long()
    both = torch.einsum("pk,pnk->pn", h.double()[at // 2], w_gu.double()[e])
    gate, up = both[:, :N], both[:, N:]
    if clamp is None:
        want = gate * torch.sigmoid(gate) * up
    else:
        gate, up = gate.clamp(max=clamp[0]), up.clamp(-clamp[0], clamp[0])
        want = gate * torch.sigmoid(clamp[1] * gate) * (up + 1.0)
    assert ((act[:named].double() - want).abs() <= 2.0 ** -8 * want.abs() + 8 * K ** 0.5 * 2.0 ** -22).all() and bool((act[named:] == 7.0).all())
    want = torch.einsum("pn,pkn->pk", act[:named].double(), w.double()[e])
    assert (y[at].double() - want).abs().max() <= 4 * N ** 0.5 * 2.0 ** -22 * max(1.0, float(act.abs().max()))
    gone = torch.ones(pairs, dtype=torch.bool, device=DEV)
    gone[at] = False
    assert int(gone.sum()) == lost and bool((y[gone] == 7.0).all())
