"""Kernels and dispatch branches at the sizes where they can go wrong: remainders of tiles and of a persistent grid's rounds,
the smallest and the largest of a range, ties and special values."""
import numpy as np
import pytest
import torch

from helpers import check_out, gen, make_paged, randn_bf16, random_blocks
from oracle import msa_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def i32(v, device=None):
    return torch.tensor(v, dtype=torch.int32, device=device)


# ---- page top-k: exact, whatever the ties ----
@pytest.mark.parametrize("h,t,nvp,topk,fb,fe", [
    (9, 33, 17, 16, 0, 0),          # one page more than topk, one token more than a warp
    (9, 33, 16 * 16 + 1, 16, 1, 2),
    (1, 1000, 769, 16, 0, 0),
    (2, 300, 33, 32, 0, 0), (2, 300, 2000, 32, 3, 0),
    (3, 257, 9, 8, 0, 0), (5, 64, 5, 4, 0, 1), (1, 31, 9000, 16, 0, 0),
    # either side of the line between a CTA and a thread per row, by rows and by pages, and with 4, 8 and 32 pages a thread
    (1, 32, 300, 16, 0, 0), (2, 32, 300, 16, 0, 0), (11, 33, 1024, 16, 0, 1), (11, 33, 1025, 16, 0, 0), (11, 33, 2048, 16, 0, 0),
    (11, 33, 2049, 16, 0, 0), (11, 33, 8192, 16, 0, 0), (5, 40, 900, 8, 1, 0), (40, 50, 8000, 4, 0, 0), (40, 50, 700, 4, 0, 0),
    (3, 33, 1100, 32, 0, 0), (3, 33, 900, 32, 0, 0), (2, 1100, 97, 32, 0, 0),
])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind", ["normal", "ties", "special"])
def test_topk_edges(h, t, nvp, topk, fb, fe, kind, dtype):
    import msa_for_sail as msa
    g = gen(h * 1000 + t + nvp)
    s = torch.randn(h, nvp + 3, t, generator=g)
    if kind == "ties":
        s = torch.randint(-2, 3, s.shape, generator=g).float()
        s[:, :, ::3] = -float("inf")
    elif kind == "special":
        pick = torch.randint(0, 12, s.shape, generator=g)
        for i, v in enumerate((float("nan"), float("inf"), -float("inf"), 0.0, -0.0, 3.402823466e38, -3.402823466e38, 1e-45)):
            s[pick == i] = v
        s[:, :, ::5] = float("nan")
    s = s.to(dtype)
    got = msa.sparse_topk_select(s.to(DEV), topk, num_valid_pages=nvp, force_begin_blocks=fb, force_end_blocks=fe)
    assert torch.equal(got.cpu(), orc.topk_select(s, topk, nvp, fb, fe))


# ---- proxy pass of decode ----
@pytest.mark.parametrize("heads,tokens", [(1, 1), (2, 1), (1, 3), (4, 1), (4, 2), (1, 7), (3, 1)])
@pytest.mark.parametrize("kv_dtype,q_dtype", [("bf16", "bf16"), ("e4m3", "e4m3"), ("e4m3", "bf16")])
@pytest.mark.parametrize("kv", [[1, 127, 128, 129, 3000], [9000], [40000] * 5])
def test_score_pass_edges(heads, tokens, kv_dtype, q_dtype, kv):
    """Ragged tails, a single long sequence, and enough pages for every warp of the grid."""
    import msa_for_sail as msa
    kv = [max(tokens, n) for n in kv]
    g = torch.Generator(device=DEV).manual_seed(heads * 10 + tokens)
    dt = torch.float8_e4m3fn if kv_dtype == "e4m3" else torch.bfloat16
    P = sum(-(-n // 128) for n in kv)
    k = torch.randn(P, 1, 128, 128, device=DEV, generator=g).to(dt)
    q = torch.randn(tokens * len(kv), heads, 128, device=DEV, generator=g).to(torch.float8_e4m3fn if q_dtype == "e4m3" else torch.bfloat16)
    table = torch.randperm(P, device=DEV, generator=g).to(torch.int32)
    plan = msa.fmha_sail_plan(i32([tokens] * len(kv)), i32(kv), heads, num_kv_heads=1, page_size=128, output_maxscore=True,
                              use_fp8_kvcache=kv_dtype == "e4m3")
    _, ms = msa.fmha_sail(q, k, k, plan, kv_indices=table, output_o=False)
    # fp32 sums of 128 products round by at most 128 * 2^-24 of the sum of their magnitudes; rounding a bf16 query to f16
    # adds 2^-11 of it (and nothing else: every other operand is exact)
    rel = 2.0 ** -17 + (2.0 ** -11 if kv_dtype != q_dtype else 0.0)
    p0 = 0
    for b, n in enumerate(kv):
        pages = -(-n // 128)
        kk = k[table[p0:p0 + pages].long(), 0].double().view(-1, 128)
        p0 += pages
        for t in range(tokens):
            qq = q[b * tokens + t].double()
            s, mag = qq @ kk.T, qq.abs() @ kk.abs().T
            s[:, n - tokens + t + 1:] = -float("inf")
            ref, bound = s.view(heads, pages, 128).amax(-1), rel * mag.view(heads, pages, 128).amax(-1)
            got = ms[:, :pages, b * tokens + t].double()
            fin = torch.isfinite(ref)
            assert torch.equal(torch.isfinite(got), fin)
            assert ((got - ref).abs()[fin] <= bound[fin]).all()
            assert torch.isinf(ms[:, pages:, b * tokens + t]).all()


def test_score_pass_many_items():
    """More work items than one scan of the kernel numbers (4 096), empty ones among them."""
    import msa_for_sail as msa
    g = torch.Generator(device=DEV).manual_seed(5)
    n = 4500
    kv = [1 + (i * 37) % 300 for i in range(n)]
    P = sum(-(-x // 128) for x in kv)
    k = torch.randn(P, 1, 128, 128, device=DEV, generator=g).to(torch.bfloat16)
    q = torch.randn(n, 1, 128, device=DEV, generator=g).to(torch.bfloat16)
    table = torch.randperm(P, device=DEV, generator=g).to(torch.int32)
    plan = msa.fmha_sail_plan(i32([1] * n), i32(kv), 1, num_kv_heads=1, page_size=128, output_maxscore=True)
    _, ms = msa.fmha_sail(q, k, k, plan, kv_indices=table, output_o=False)
    start = np.concatenate([[0], np.cumsum([-(-x // 128) for x in kv])])
    for b in list(range(0, n, 97)) + [4095, 4096, 4097, n - 1]:
        kk = k[table[start[b]:start[b + 1]].long(), 0].double().view(-1, 128)
        s = (kk @ q[b, 0].double())
        s[kv[b]:] = -float("inf")
        bound = 2.0 ** -17 * (kk.abs() @ q[b, 0].double().abs()).view(-1, 128).amax(-1)
        ref = s.view(-1, 128).amax(-1)
        assert ((ms[0, :len(ref), b].double() - ref).abs() <= bound).all()


def test_score_pass_long_runs():
    """More pages per warp than it looks up at a time (32): one sequence of 60 001 pages in e4m3."""
    import msa_for_sail as msa
    g = torch.Generator(device=DEV).manual_seed(6)
    P = 60001
    n = P * 128 - 100
    k = torch.empty(P, 1, 128, 128, device=DEV, dtype=torch.float8_e4m3fn)
    for i in range(0, P, 8192):
        k[i:i + 8192] = torch.randn(min(8192, P - i), 1, 128, 128, device=DEV, generator=g, dtype=torch.bfloat16).to(k.dtype)
    q = torch.randn(1, 1, 128, device=DEV, generator=g).to(k.dtype)
    table = torch.randperm(P, device=DEV, generator=g).to(torch.int32)
    plan = msa.fmha_sail_plan(i32([1]), i32([n]), 1, num_kv_heads=1, page_size=128, output_maxscore=True, use_fp8_kvcache=True)
    _, ms = msa.fmha_sail(q, k, k, plan, kv_indices=table, output_o=False)
    qq = q[0, 0].double()
    for i in range(0, P, 4096):
        kk = k[table[i:i + 4096].long(), 0].double()
        s = kk @ qq
        if i + 4096 >= P:
            s[-1, 28:] = -float("inf")
        bound = 2.0 ** -17 * (kk.abs() @ qq.abs()).amax(-1)
        assert ((ms[0, i:i + len(kk), 0].double() - s.amax(-1)).abs() <= bound).all()


# ---- dense prefill: CTAs that take several work items ----
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float8_e4m3fn])
@pytest.mark.parametrize("paged", [True, False])
def test_dense_prefill_items_per_cta(dtype, paged):
    """64 heads x 11 row tiles on 148 SMs: items of 0 to 5 tiles, with and without a second Q tile, and a sequence whose
    first rows see no key."""
    import msa_for_sail as msa
    g = gen(9)
    qo, kv, hq, hk = [257, 130, 1, 511, 200, 300, 256], [600, 130, 77, 511, 64, 300, 512], 64, 8
    off = [k - q for q, k in zip(qo, kv)]                    # 64 - 200 < 0: given below as an explicit offset
    q = randn_bf16(g, sum(qo), hq, 128).to(dtype)
    kp, vp, table = make_paged(g, kv, hk, 128, dtype=dtype)
    k = orc.paged_to_contiguous(kp, table, kv, 128); v = orc.paged_to_contiguous(vp, table, kv, 128)
    off[4] = 0
    plan = msa.fmha_sail_plan(i32(qo), i32(kv), hq, num_kv_heads=hk, page_size=128 if paged else -1, qo_offset=i32(off),
                              use_fp8_kvcache=dtype != torch.bfloat16)
    assert plan[3]["tc_preferred"] and plan[3]["num_work_tc"] > 2 * 148
    args = dict(kv_indices=table.to(DEV)) if paged else {}
    for _ in range(2):
        out, _ = msa.fmha_sail(q.to(DEV), (kp if paged else k).to(DEV), (vp if paged else v).to(DEV), plan, **args)
    ref = orc.attention(q.float(), k.float(), v.float(), qo, kv, hq, hk, qo_offset=off)
    check_out(out, ref, "dense items", **({} if dtype == torch.bfloat16 else dict(cos_min=0.999, max_abs=None)))


# ---- sparse prefill merge ----
@pytest.mark.parametrize("kbn,hq,hk,T", [(4, 2, 2, 300), (8, 16, 1, 257), (16, 16, 2, 301), (32, 32, 4, 260), (3, 8, 2, 1)])
def test_sparse_merge_edges(kbn, hq, hk, T):
    import msa_for_sail as msa
    from msa_for_sail import api
    g = gen(kbn * 100 + T)
    kv = [max(T, kbn * 128 + 50)]
    q = randn_bf16(g, T, hq, 128)
    kp, vp, table = make_paged(g, kv, hk, 128)
    bi = random_blocks(g, [T], kv, [kv[0] - T], hk, kbn)
    plan = msa.fmha_sail_plan(i32([T]), i32(kv), hq, num_kv_heads=hk, page_size=128, kv_block_num=kbn)
    lse = torch.empty(T, hq, dtype=torch.float32, device=DEV)
    api._FORCE_SPARSE_TC = True
    try:
        out, _ = msa.fmha_sail(q.to(DEV), kp.to(DEV), vp.to(DEV), plan, kv_indices=table.to(DEV), kv_block_indexes=bi.to(DEV), lse=lse)
    finally:
        api._FORCE_SPARSE_TC = False
    ref, ref_lse = orc.sparse_attention(q, kp, vp, [T], kv, table, bi, hq, return_lse=True)
    check_out(out, ref, "sparse merge")
    lse = lse.cpu()
    seen = torch.isfinite(ref_lse)                           # a token may have selected a page it cannot see, and no other
    assert torch.equal(torch.isfinite(lse), seen)
    # bf16 products are exact, fp32 sums round by 2^-17 of them at most, exp2 on the FMA pipe is good to 7.5e-5
    assert (lse - ref_lse)[seen].abs().max() <= 2e-3


@pytest.mark.parametrize("dtype", [torch.float8_e4m3fn, torch.bfloat16])
def test_sparse_prefill_partial_chunks(dtype):
    """Page lists whose last chunk has one token, so that two of the three loader warps have no row in it: a loader that
    waited for that chunk's buffer all the same could miss its phase and run into the limit of its wait."""
    import msa_for_sail as msa
    from msa_for_sail import api
    g = gen(77)
    hq, hk, pages, topk = 8, 1, 64, 4
    tpc = 128 * hk // hq                                     # a token is one unit: the last chunk has one
    per_page = 5 * tpc + 1
    # 16 tokens after another share out all 64 pages, so that each page is selected equally often
    bi = torch.cat([torch.randperm(pages, generator=g).view(pages // topk, topk) for _ in range(per_page)])
    T = bi.shape[0]
    kv = [pages * 128 + T]
    assert (torch.bincount(bi.view(-1), minlength=pages) == per_page).all() and per_page % tpc == 1
    bi = bi.sort(1).values.to(torch.int32).view(T, hk, topk)
    assert (bi[:, :, 1:] > bi[:, :, :-1]).all()
    q = randn_bf16(g, T, hq, 128).to(dtype).to(DEV)
    kp, vp, table = make_paged(g, kv, hk, 128, dtype=dtype)
    kp, vp, table, bi = kp.to(DEV), vp.to(DEV), table.to(DEV), bi.to(DEV)
    plan = msa.fmha_sail_plan(i32([T]), i32(kv), hq, num_kv_heads=hk, page_size=128, kv_block_num=4,
                              use_fp8_kvcache=dtype != torch.bfloat16)
    assert plan[3]["sparse_tc_preferred"]
    first, _ = msa.fmha_sail(q, kp, vp, plan, kv_indices=table, kv_block_indexes=bi)
    out = torch.empty_like(first)
    for _ in range(300):
        msa.fmha_sail(q, kp, vp, plan, kv_indices=table, kv_block_indexes=bi, out=out)
    assert api.last_status() == 0
    assert torch.equal(out, first)


# ---- planning on the device ----
@pytest.mark.parametrize("batch", [1, 31, 32, 33, 256, 257, 600])
def test_device_plan_prefix_sums(batch):
    import msa_for_sail as msa
    rng = np.random.default_rng(batch)
    kv = rng.integers(1, 5000, batch).astype(np.int32)
    qo = np.ones(batch, np.int32)
    ws = msa.allocate_graph_workspace(batch, 4, num_kv_heads=1, max_qo_len=1, page_size=128)
    plan = msa.fmha_sail_plan(torch.from_numpy(qo).to(DEV), torch.from_numpy(kv).to(DEV), 4, num_kv_heads=1, page_size=128,
                              given_workspace=ws, max_total_q=batch, graph_safe=True, max_qo_len_override=1,
                              qo_len_uniform_override=True, max_kv_len_override=5000)[3]
    for key, v in (("qo_segment_offsets", qo), ("kv_segment_offsets", kv), ("kv_page_indptr", -(-kv // 128))):
        assert plan[key].cpu().tolist() == [0] + np.cumsum(v).tolist(), key
    assert plan["qo_offset"].cpu().tolist() == (kv - qo).tolist()


# ---- kernels of one stream that come up before the one before them has ended ----
@pytest.mark.parametrize("tokens,kv", [(3, [2000, 700, 5000, 64]), (1100, [3000])])
def test_chained_passes_read_the_latest_data(tokens, kv):
    """Passes back to back into the same buffers, each on other inputs: bit for bit what a pass gives that nothing overlaps."""
    import msa_for_sail as msa
    g = torch.Generator(device=DEV).manual_seed(tokens)
    hq, hk, topk, T = 16, 2, 4, tokens * len(kv)
    P = sum(-(-n // 128) for n in kv)
    nvp = -(-max(kv) // 128)
    sets = [(torch.randn(T, hq, 128, device=DEV, generator=g).to(torch.bfloat16), torch.randn(T, hk, 128, device=DEV, generator=g).to(torch.bfloat16),
             torch.randn(P, 1, 128, 128, device=DEV, generator=g).to(torch.bfloat16), torch.randn(P, hk, 128, 128, device=DEV, generator=g).to(torch.bfloat16),
             torch.randn(P, hk, 128, 128, device=DEV, generator=g).to(torch.bfloat16)) for _ in range(3)]
    buf = [torch.empty_like(t) for t in sets[0]]
    q, iq, ik, k, v = buf
    table = torch.randperm(P, device=DEV, generator=g).to(torch.int32)
    lens = i32([tokens] * len(kv)), i32(kv)
    score = msa.fmha_sail_plan(*lens, hk, num_kv_heads=1, page_size=128, output_maxscore=True)
    sparse = msa.fmha_sail_plan(*lens, hq, num_kv_heads=hk, page_size=128, kv_block_num=topk, num_kv_splits=4)
    scores = torch.full((hk, -(-nvp // 128) * 128, T), -float("inf"), device=DEV)
    sel = torch.empty(T, hk, topk, dtype=torch.int32, device=DEV)

    def one(i, sync):
        for b, t in zip(buf, sets[i]):
            b.copy_(t)
        if sync:
            torch.cuda.synchronize()
        msa.fmha_sail(iq, ik, ik, score, kv_indices=table, output_o=False, max_score=scores)
        if sync:
            torch.cuda.synchronize()
        msa.sparse_topk_select(scores, topk, num_valid_pages=nvp, output=sel)
        if sync:
            torch.cuda.synchronize()
        return msa.fmha_sail(q, k, v, sparse, kv_indices=table, kv_block_indexes=sel)[0]

    want = [one(i, True) for i in range(3)]
    assert not torch.equal(want[0], want[1])
    got = [one(i % 3, False) for i in range(60)]
    for i, out in enumerate(got):
        assert torch.equal(out, want[i % 3]), i
