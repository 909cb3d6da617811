"""Each sm_100a kernel against the PyTorch fp32 statement of the same op."""
import math

import pytest
import torch

from stkernel_b200.ops import _lib
from stkernel_b200.ops import attention as A
from stkernel_b200.ops import cache as C
from stkernel_b200.ops import functional as Fn
from stkernel_b200.ops import moe as M
from stkernel_b200.ops import reference as R
from stkernel_b200.ops import sampling as S

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32


def dev():
    return torch.device("cuda:0")


def rel_err(a, b):
    a, b = a.float().cpu(), b.float().cpu()
    return ((a - b).norm() / b.norm().clamp(min=1e-12)).item()


@pytest.mark.parametrize("T", [1, 8, 64, 256, 1000])
@pytest.mark.parametrize("N,K", [(512, 1024), (2048, 4096), (384, 576)])
def test_gemm_bf16(T, N, K):
    torch.manual_seed(T + N)
    x = torch.randn(T, K, device=dev()).to(BF16)
    w = torch.randn(N, K, device=dev()).to(BF16)
    ref = x.float() @ w.float().t()
    out = Fn.linear(x, Fn.LinearWeight(w))
    assert rel_err(out, ref) < 1e-2
    out32 = Fn.linear(x, Fn.LinearWeight(w), out_dtype=F32)
    assert rel_err(out32, ref) < 2e-3


@pytest.mark.parametrize("T,N,K", [(512, 512, 256), (700, 1000, 1024), (1024, 4160, 4096), (4096, 2048, 8192)])
def test_gemm_bf16_wide_tile(T, N, K):
    """Large bf16 problems: one CTA per 256 weight rows x 256 tokens (two accumulators), ragged edges included."""
    torch.manual_seed(T + N + K)
    x = (torch.randn(T, K, device=dev()) * 0.5).to(BF16)
    w = (torch.randn(N, K, device=dev()) * 0.5).to(BF16)
    ref = x.float() @ w.float().t()
    out = Fn.linear(x, Fn.LinearWeight(w))
    assert rel_err(out, ref) < 1e-2
    out32 = Fn.linear(x, Fn.LinearWeight(w), out_dtype=F32)
    assert rel_err(out32, ref) < 2e-3
    # element-wise, not only in norm: a misplaced tile would hide in a relative norm of random data
    assert (out32 - ref).abs().max().item() < 0.05 * ref.abs().max().item()
    torch.cuda.synchronize()
    _lib.check_status()


@pytest.mark.parametrize("splits", [1, 2, 5])
def test_gemm_bf16_splitk_matches(splits):
    torch.manual_seed(1)
    x = torch.randn(8, 4096, device=dev()).to(BF16)
    w = torch.randn(256, 4096, device=dev()).to(BF16)
    ref = x.float() @ w.float().t()
    out = Fn.linear(x, Fn.LinearWeight(w), out_dtype=F32, splits=splits)
    assert rel_err(out, ref) < 2e-3


@pytest.mark.parametrize("T", [1, 6, 64, 128, 700])
@pytest.mark.parametrize("N,K", [(512, 1024), (2048, 4096), (1536, 7168)])
def test_gemm_fp8_block(T, N, K):
    torch.manual_seed(T)
    x = torch.randn(T, K, device=dev()).to(BF16)
    w = torch.randn(N, K, device=dev()) * 0.05
    lw = Fn.LinearWeight.from_master(w, "fp8", dev())
    xq, xs = R.quant_fp8_group128_act(x)
    ref = R.dequant_fp8_group128_act(xq, xs) @ lw.dequant().t()
    if T <= 4:                        # the CUDA-core weight-streaming kernel keeps the activations unquantised
        ref = x.float() @ lw.dequant().t()
    out = Fn.linear(x, lw, out_dtype=F32)
    assert rel_err(out, ref) < 2e-3
    # and against the unquantised product within fp8 error
    assert rel_err(out, x.float() @ w.t()) < 6e-2


def test_quant_act_matches_reference():
    x = (torch.randn(37, 640, device=dev()) * 3).to(BF16)
    qa = Fn.quant_act(x)
    q, s = R.quant_fp8_group128_act(x)
    assert torch.equal(qa.q.view(torch.uint8)[:37], q.view(torch.uint8))
    assert torch.allclose(qa.scale[:, :37].t(), s)


def test_rmsnorm_and_pair():
    x = torch.randn(9, 1536, device=dev()).to(BF16)
    w = (1 + 0.1 * torch.randn(1536, device=dev())).to(BF16)
    y = Fn.rms_norm(x, w, 1e-6)
    assert rel_err(y, R.rms_norm(x, w, 1e-6)) < 5e-3
    x1 = torch.randn(9, 512, device=dev()).to(BF16)
    w1 = torch.ones(512, device=dev()).to(BF16)
    a, b, qa = Fn.rms_norm_pair(x, w, x1, w1, 1e-6, quant0=True)
    assert rel_err(a, R.rms_norm(x, w, 1e-6)) < 5e-3
    assert rel_err(b, R.rms_norm(x1, w1, 1e-6)) < 5e-3
    deq = R.dequant_fp8_group128_act(qa.q[:9], qa.scale[:, :9].t())
    assert rel_err(deq, a) < 4e-2


def test_swiglu_clamp():
    gu = (torch.randn(5, 512, device=dev()) * 8).to(BF16)
    a = Fn.swiglu_clamp(gu, 10.0)
    assert rel_err(a, R.swiglu_clamp(gu[:, :256], gu[:, 256:], 10.0)) < 5e-3


@pytest.mark.parametrize("T,H", [(1, 4096), (7, 4096), (33, 256), (300, 4096), (700, 1024)])
def test_mhc_pre_post_head(T, H):
    torch.manual_seed(0)
    hc = 4
    res = torch.randn(T, hc, H, device=dev()).to(BF16)
    fn = torch.randn(24, hc * H, device=dev()) * 0.02
    base = torch.randn(24, device=dev()) * 0.1
    scale = torch.tensor([1.0, 0.7, 1.3], device=dev())
    nw = (1 + 0.1 * torch.randn(H, device=dev())).to(BF16)
    y, post, comb = Fn.mhc_pre(res, fn, base, scale, nw, 1e-6, 1e-6, 20)
    yr, pr, cr = R.mhc_pre(res, fn, base, scale, nw, 1e-6, 1e-6, 20, round_bf16=True)
    assert rel_err(y, yr) < 5e-3
    assert torch.allclose(post, pr, atol=1e-4, rtol=1e-4)
    assert torch.allclose(comb.view(T, hc, hc), cr, atol=1e-4, rtol=1e-3)
    # combine matrix is (nearly) doubly stochastic after Sinkhorn
    assert torch.allclose(comb.view(T, hc, hc).sum(1), torch.ones(T, hc, device=dev()), atol=1e-3)
    x = torch.randn(T, H, device=dev()).to(BF16)
    out = Fn.mhc_post(x, res, post, comb)
    assert rel_err(out, R.mhc_post(x, res, pr, cr)) < 5e-3
    hfn = torch.randn(hc, hc * H, device=dev()) * 0.02
    hb = torch.randn(hc, device=dev()) * 0.1
    hs = torch.tensor([0.9], device=dev())
    hh = Fn.hc_head(res, hfn, hb, hs, 1e-6, 1e-6)
    assert rel_err(hh, R.hc_head(res, hfn, hb, hs, 1e-6, 1e-6)) < 5e-3


@pytest.mark.parametrize("H", [272, 2064, 6144])
@pytest.mark.parametrize("norm", [True, False])
def test_mhc_pre_in_whole_rows(H, norm):
    """Widths that end inside a thread block's pass, and of one, two and four passes; without a norm behind the sum."""
    torch.manual_seed(2)
    T, hc = 259, 4
    res = torch.randn(T, hc, H, device=dev()).to(BF16)
    fn = torch.randn(24, hc * H, device=dev()) * 0.02
    base, scale = torch.randn(24, device=dev()) * 0.1, torch.tensor([1.0, 0.7, 1.3], device=dev())
    nw = (1 + 0.1 * torch.randn(H, device=dev())).to(BF16) if norm else None
    y, post, comb = Fn.mhc_pre(res, fn, base, scale, nw, 1e-6, 1e-6, 20)
    yr, pr, cr = R.mhc_pre(res, fn, base, scale, nw, 1e-6, 1e-6, 20, round_bf16=True)
    assert rel_err(y, yr) < 5e-3                          # two roundings to bf16
    assert torch.allclose(post, pr, atol=1e-4, rtol=1e-4) and torch.allclose(comb.view(T, hc, hc), cr, atol=1e-4, rtol=1e-3)
    x = torch.randn(T, H, device=dev()).to(BF16)
    assert rel_err(Fn.mhc_post(x, res, post, comb), R.mhc_post(x, res, pr, cr)) < 5e-3


@pytest.mark.parametrize("T", [5, 70, 300])
@pytest.mark.parametrize("iters", [0, 1, 2])
@pytest.mark.parametrize("H", [1024, 4608])
def test_mhc_pre_of_few_normalisations(T, iters, H):
    """Columns are normalised once whatever the number, in every kernel that serves a step: clusters, row dots, products of many tokens."""
    torch.manual_seed(2)
    hc = 4
    res = torch.randn(T, hc, H, device=dev()).to(BF16)
    fn = torch.randn(24, hc * H, device=dev()) * 0.02
    base, scale = torch.randn(24, device=dev()), torch.tensor([1.0, 0.7, 1.3], device=dev())
    _, _, comb = Fn.mhc_pre(res, fn, base, scale, None, 1e-6, 1e-6, iters)
    _, _, cr = R.mhc_pre(res, fn, base, scale, None, 1e-6, 1e-6, iters, round_bf16=True)
    assert torch.allclose(comb.view(T, hc, hc), cr, atol=1e-4, rtol=1e-3)


@pytest.mark.parametrize("n,e_local,start", [(2049, 300, 0), (5000, 37, 3), (24576, 256, 0)])
def test_moe_align_many_pairs(n, e_local, start):
    """Chunks and experts that fill neither a batch of counts nor a warp; pairs of other ranks' experts."""
    g = torch.Generator().manual_seed(n)
    ids = torch.randint(0, e_local + 5, (n,), generator=g, dtype=torch.int32)
    sorted_p, sorted_e, pair_row = (torch.full((n,), -7, dtype=torch.int32, device=dev()) for _ in range(3))
    offsets = torch.empty(e_local + 1, dtype=torch.int32, device=dev())
    counts = torch.empty((n + 255) // 256 * e_local, dtype=torch.int32, device=dev())
    _lib.call("stk_moe_align", ids.to(dev()), n, start, e_local, sorted_p, pair_row, offsets, sorted_e, counts, _lib.stream())
    local = ids - start
    mine = (local >= 0) & (local < e_local)
    order = torch.argsort(torch.where(mine, local, e_local), stable=True)[:int(mine.sum())]
    assert torch.equal(sorted_p.cpu()[:order.numel()], order.to(torch.int32))
    assert torch.equal(sorted_e.cpu()[:order.numel()], local[order])
    assert torch.equal(offsets.cpu()[1:], torch.bincount(local[mine].long(), minlength=e_local).cumsum(0).to(torch.int32))
    want = torch.full((n,), -1, dtype=torch.int32)
    want[order] = torch.arange(order.numel(), dtype=torch.int32)
    assert torch.equal(pair_row.cpu(), want)


@pytest.mark.parametrize("topk", [1, 8, 9, 16])
def test_moe_combine_places(topk):
    torch.manual_seed(topk)
    T, H = 70, 1096
    y, w = torch.randn(T * topk, H, device=dev()).to(BF16), torch.rand(T, topk, device=dev())
    rows = torch.randperm(T * topk).to(torch.int32).to(dev())
    rows[::5] = -1
    shared, out = torch.randn(T, H, device=dev()).to(BF16), torch.empty(T, H, dtype=BF16, device=dev())
    _lib.call("stk_moe_combine", y, w, rows, shared, out, T, H, topk, None, _lib.stream())
    picked = torch.where(rows[:, None] >= 0, y.double()[rows.clamp(min=0).long()], 0.0).view(T, topk, H)
    assert rel_err(out, (picked * w.double()[:, :, None]).sum(1) + shared.double()) < 2.5e-3      # rounded to bf16 once


@pytest.mark.parametrize("T,H", [(1, 4096), (5, 4096), (16, 1024), (40, 512)])
def test_mhc_post_pre_fused(T, H):
    """Post-mix of one sub-block fused into the next pre-mix (one cluster launch for T <= 16) against the two
    reference ops run back to back in fp32 (streams rounded to bf16 in between, as the unfused path stores them)."""
    torch.manual_seed(1)
    hc = 4
    res = torch.randn(T, hc, H, device=dev()).to(BF16)
    x = torch.randn(T, H, device=dev()).to(BF16)
    post_old = torch.rand(T, hc, device=dev()) * 2
    comb_old = torch.softmax(torch.randn(T, hc, hc, device=dev()), -1).reshape(T, hc * hc).contiguous()
    fn = torch.randn(24, hc * H, device=dev()) * 0.02
    base = torch.randn(24, device=dev()) * 0.1
    scale = torch.tensor([1.0, 0.7, 1.3], device=dev())
    nw = (1 + 0.1 * torch.randn(H, device=dev())).to(BF16)
    new_res, r = Fn.mhc_post_pre(x, res, post_old, comb_old, fn, base, scale, nw, 1e-6, 1e-6, 20)
    ref_res = R.mhc_post(x, res, post_old, comb_old.view(T, hc, hc)).to(BF16)
    assert rel_err(new_res, ref_res) < 5e-3
    yr, pr, cr = R.mhc_pre(ref_res, fn, base, scale, nw, 1e-6, 1e-6, 20, round_bf16=True)
    assert rel_err(r[0], yr) < 6e-3
    assert torch.allclose(r[1], pr, atol=2e-3, rtol=2e-3)
    assert torch.allclose(r[2].view(T, hc, hc), cr, atol=2e-3, rtol=2e-3)


def _rope_setup(T, R_):
    pos = torch.randint(0, 100000, (T,), device=dev(), dtype=torch.int64)
    inv = Fn.inv_freq(R_, 10000.0, dev())
    ang = pos.float()[:, None] * inv[None]
    return pos, inv, torch.cos(ang), torch.sin(ang)


def test_q_norm_rope():
    T, nh, D, R_ = 5, 8, 512, 64
    q = torch.randn(T, nh, D, device=dev()).to(BF16)
    pos, inv, cos, sin = _rope_setup(T, R_)
    ref = R.rms_norm(q, None, 1e-6)
    ref = torch.cat([ref[..., :D - R_], R.apply_rope_interleaved(ref[..., D - R_:], cos, sin)], -1)
    out = Fn.q_norm_rope(q.clone(), pos, inv, R_, 1e-6)
    assert rel_err(out, ref) < 6e-3


@pytest.mark.parametrize("fp8", [True, False])
def test_kv_insert_gather_roundtrip(fp8):
    T, D, R_ = 70, 512, 64
    kv = torch.randn(T, D, device=dev()).to(BF16)
    pos, inv, cos, sin = _rope_setup(T, R_)
    cache = C.PagedCache.allocate(4, D, R_, fp8, "latent", dev())
    slots = torch.randperm(4 * 64, device=dev())[:T].to(torch.int64)
    slots[3] = -1
    C.kv_rope_quant_insert(kv, pos, slots, inv, cache)
    rows = C.kv_gather_dequant(cache, slots)
    roped = torch.cat([kv.float()[:, :D - R_], R.apply_rope_interleaved(kv[:, D - R_:], cos, sin).to(BF16).float()], 1)
    ref = R.kv_fake_quant(roped, R_) if fp8 else roped.to(BF16).float()
    ref[3] = 0
    assert rel_err(rows, ref) < 4e-3
    # byte-exact against the CPU writer of the same format
    cpu = C.PagedCache.allocate(4, D, R_, fp8, "latent", "cpu")
    cpu.write_rows_cpu(slots.cpu(), roped.cpu())
    same = (cpu.buf == cache.buf.cpu()).float().mean().item()
    assert same > 0.999


@pytest.mark.parametrize("ratio,c,kind,fp8", [(4, 2, "latent", True), (4, 2, "indexer", True), (128, 1, "latent", False)])
def test_compress_windows_matches_cpu(ratio, c, kind, fp8):
    torch.manual_seed(3)
    D = 512 if kind == "latent" else 128
    R_ = 64
    ring = 2 * ratio if c == 2 else ratio
    # two requests: a 300-token prefill chunk starting at 0 and a decode token at position 2*ratio-1 with state
    lens = [300, 1]
    starts = [0, 2 * ratio - 1]
    T = sum(lens)
    kvs = torch.randn(T, 2 * c * D)
    ape = torch.randn(ratio, c * D) * 0.1
    nw = (1 + 0.1 * torch.randn(D)).to(BF16)
    inv = Fn.inv_freq(R_, 10000.0, "cpu")
    qs = torch.tensor([0, 300, 301], dtype=torch.int32)
    tok_req, positions, first, last = A.token_maps(qs, torch.tensor([0, 1], dtype=torch.int32),
                                                   torch.tensor(starts, dtype=torch.int32), 2, T)
    state = torch.randn(2, ring, 2 * c * D)
    bt = torch.tensor([[0, 1], [2, 3]], dtype=torch.int32)
    cpu_cache = C.PagedCache.allocate(4, D, R_, fp8, kind, "cpu")
    st_cpu = state.clone()
    C.compress_windows(kvs, ape, nw, inv, positions, tok_req, first, last, st_cpu, bt, cpu_cache, ratio, c, 1e-6)
    g = lambda t: t.to(dev())
    gpu_cache = C.PagedCache.allocate(4, D, R_, fp8, kind, dev())
    st_gpu = g(state.clone())
    C.compress_windows(g(kvs), g(ape), g(nw), g(inv), g(positions), g(tok_req), g(first), g(last), st_gpu, g(bt),
                       gpu_cache, ratio, c, 1e-6)
    n_win = 300 // ratio
    slots = torch.cat([torch.arange(n_win), torch.tensor([2 * 64 + 1])])
    a, sa = cpu_cache.read_rows_cpu(slots)
    gc = C.PagedCache(gpu_cache.buf.cpu(), D, R_, fp8, kind)
    b, sb = gc.read_rows_cpu(slots)
    if sa is not None:
        a, b = a * sa[:, None], b * sb[:, None]
    assert a.abs().sum() > 0
    assert rel_err(b, a) < 3e-2
    assert torch.allclose(st_gpu.cpu(), st_cpu)


def test_indexer_q_prep():
    T, ih, d, R_ = 6, 64, 128, 64
    q = torch.randn(T, ih, d, device=dev()).to(BF16)
    w = torch.randn(T, ih, device=dev())
    pos, inv, cos, sin = _rope_setup(T, R_)
    qq, wf = C.indexer_q_prep(q, w, pos, inv, R_, True)
    rq, rw = R.indexer_q_prepare(q, w, cos, sin, R_, True)
    # compare dequantised operands (scale folded into the weights)
    assert rel_err(qq.float() * wf[..., None], rq * rw[..., None]) < 2e-2


def _fill_indexer_cache(S, d, fp8):
    k = torch.randn(S, d, device=dev())
    cache = C.PagedCache.allocate((S + 63) // 64 + 1, d, 64, fp8, "indexer", "cpu")
    cache.write_rows_cpu(torch.arange(S), k.cpu())
    return k, C.PagedCache(cache.buf.to(dev()), d, 64, fp8, "indexer"), cache


@pytest.mark.parametrize("T", [3, 131, 300])
def test_indexer_scores_tensor_core_matches_cuda_core(T):
    """tcgen05 scorer (K block stationary, q tiles by TMA, head sum in the TMEM lane) against the CUDA-core scorer and
    the CPU reference: two requests with scattered pages, causal n_valid, a padded token (request -1)."""
    torch.manual_seed(17)
    ih, d, S = 64, 128, 1000
    n_pages = 2 * ((S + 63) // 64) + 3
    cache = C.PagedCache.allocate(n_pages, d, 64, True, "indexer", "cpu")
    perm = torch.randperm(n_pages - 1)[:2 * ((S + 63) // 64)] + 1
    bt_cpu = perm.view(2, -1).to(torch.int32)
    for req in range(2):
        k = torch.randn(S, d)
        slots = bt_cpu[req].long()[torch.arange(S) // 64] * 64 + torch.arange(S) % 64
        cache.write_rows_cpu(slots, k)
    gcache = C.PagedCache(cache.buf.to(dev()), d, 64, True, "indexer")
    bt = bt_cpu.to(dev()).contiguous()
    q = torch.randn(T, ih, d, device=dev()).to(BF16)
    w = torch.rand(T, ih, device=dev())
    split = T // 3                                          # request 0: first third, request 1: the rest
    tok_req = torch.cat([torch.zeros(split, dtype=torch.int32), torch.ones(T - split, dtype=torch.int32)]).to(dev())
    pos = torch.cat([torch.arange(split) + 900, torch.arange(T - split) * 9 + 5]).to(dev())
    tok_req[-1] = -1
    inv = Fn.inv_freq(64, 10000.0, dev())
    qq, wf = C.indexer_q_prep(q, w, pos, inv, 64, True)
    nv = A.compressed_valid(pos, 4)
    nv[-1] = 0
    assert int(nv.max()) <= S
    assert A.USE_TENSOR_CORE_INDEXER
    before = A.tc_indexer_calls
    tc = A.indexer_scores(qq, wf, gcache, bt, tok_req, nv, S, tag="idx_tc_test").clone()
    assert A.tc_indexer_calls == before + 1
    A.USE_TENSOR_CORE_INDEXER = False
    try:
        cc = A.indexer_scores(qq, wf, gcache, bt, tok_req, nv, S, tag="idx_cc_test").clone()
    finally:
        A.USE_TENSOR_CORE_INDEXER = True
    checked = 0
    for i in range(T):
        n = int(nv[i])
        if n:
            assert rel_err(tc[i, :n], cc[i, :n]) < 1e-3, i
            checked += 1
    assert checked >= T // 2
    sub = [0, max(0, split - 1), min(T - 2, split)]
    ref = A.indexer_scores(qq[sub].cpu(), wf[sub].cpu(), cache, bt_cpu, tok_req[sub].cpu(), nv[sub].cpu(), S)
    for j, i in enumerate(sub):
        n = int(nv[i])
        if n:
            assert rel_err(tc[i, :n], ref[j, :n]) < 2e-3


@pytest.mark.parametrize("fp8", [True, False])
def test_indexer_scores_and_topk(fp8):
    torch.manual_seed(5)
    T, ih, d, S, K = 5, 64, 128, 700, 64
    k, gcache, ccache = _fill_indexer_cache(S, d, fp8)
    q = torch.randn(T, ih, d, device=dev()).to(BF16)
    w = torch.rand(T, ih, device=dev())
    pos = torch.tensor([S * 4 - 1, 100, 3, 2000, 1023], device=dev(), dtype=torch.int64)
    inv = Fn.inv_freq(64, 10000.0, dev())
    qq, wf = C.indexer_q_prep(q, w, pos, inv, 64, fp8)
    bt = torch.arange(gcache.num_pages, dtype=torch.int32, device=dev())[None].contiguous()
    tok_req = torch.zeros(T, dtype=torch.int32, device=dev())
    nv = A.compressed_valid(pos, 4)
    scores = A.indexer_scores(qq, wf, gcache, bt, tok_req, nv, S)
    ref = A.indexer_scores(qq.cpu(), wf.cpu(), ccache, bt.cpu(), tok_req.cpu(), nv.cpu(), S)
    for i in range(T):
        n = int(nv[i])
        if n:
            assert rel_err(scores[i, :n], ref[i, :n]) < 2e-3
    top = A.topk_rows(scores, nv, K)
    for i in range(T):
        n = int(nv[i])
        got = top[i][top[i] >= 0].cpu()
        assert got.numel() == min(n, K)
        assert got.unique().numel() == got.numel()
        if n > K:
            thr = torch.topk(scores[i, :n], K).values.min()
            assert (scores[i, got.to(dev()).long()] >= thr).all()
        elif n > 0:
            assert torch.equal(got.sort().values, torch.arange(n, dtype=torch.int32))


def test_topk_large_with_ties():
    T, S, K = 3, 40000, 2048
    scores = torch.randn(T, S, device=dev())
    scores[1] = torch.randint(0, 50, (S,), device=dev()).float()      # heavy ties
    nv = torch.tensor([S, S, 5000], dtype=torch.int32, device=dev())
    top = A.topk_rows(scores, nv, K)
    for i in range(T):
        got = top[i].long()
        assert (got >= 0).all() and got.unique().numel() == K
        n = int(nv[i])
        assert (got < n).all()
        thr = torch.topk(scores[i, :n], K).values.min()
        assert (scores[i, got] >= thr).all()
        assert torch.isclose(scores[i, got].sum(), torch.topk(scores[i, :n], K).values.sum(), rtol=1e-4)


@pytest.mark.parametrize("nh,D,R_,fp8", [(64, 512, 64, True), (8, 512, 64, True), (4, 80, 16, False)])
def test_sparse_mla_matches_reference(nh, D, R_, fp8):
    torch.manual_seed(7)
    T, W, K = 4, 128, 512 if D == 512 else 16
    n_pages = 24
    rows = torch.randn(n_pages * 64, D)
    ccpu = C.PagedCache.allocate(n_pages, D, R_, fp8, "latent", "cpu")
    ccpu.write_rows_cpu(torch.arange(n_pages * 64), rows)
    cg = C.PagedCache(ccpu.buf.to(dev()), D, R_, fp8, "latent")
    q = torch.randn(T, nh, D, device=dev()).to(BF16)
    swa_slots = torch.randint(0, n_pages * 64, (T, W), dtype=torch.int32, device=dev())
    swa_lens = torch.tensor([W, 5, 1, 77], dtype=torch.int32, device=dev())
    topk_slots = torch.randint(0, n_pages * 64, (T, K), dtype=torch.int32, device=dev())
    topk_slots[0, 3] = -1
    topk_lens = torch.tensor([K, 0, K // 2, 9], dtype=torch.int32, device=dev())
    sink = torch.randn(nh, device=dev())
    out = A.sparse_mla(q, cg, swa_slots, swa_lens, cg, topk_slots, topk_lens, sink, D ** -0.5)
    ref = A.sparse_mla(q.cpu(), ccpu, swa_slots.cpu(), swa_lens.cpu(), ccpu, topk_slots.cpu(), topk_lens.cpu(),
                       sink.cpu(), D ** -0.5)
    assert rel_err(out, ref) < 1e-2
    out2 = A.sparse_mla(q, cg, swa_slots, swa_lens, None, None, None, sink, D ** -0.5)
    ref2 = A.sparse_mla(q.cpu(), ccpu, swa_slots.cpu(), swa_lens.cpu(), None, None, None, sink.cpu(), D ** -0.5)
    assert rel_err(out2, ref2) < 1e-2


@pytest.mark.parametrize("nh,T", [(8, 700), (32, 331), (64, 460)])
def test_sparse_mla_several_tokens_per_thread_block(nh, T):
    """More tokens than SMs, with lists of no rows, of one, of whole blocks and of parts of them next to one another, tokens without
    any at the beginning and the end of a thread block's share, slots of -1 inside; the second half of the lists from another cache."""
    D, R_, W, K, n = 512, 64, 128, 300, 1024
    g = torch.Generator().manual_seed(T)
    caches = []
    for _ in range(2):
        ccpu = C.PagedCache.allocate(n // 64, D, R_, True, "latent", "cpu")
        ccpu.write_rows_cpu(torch.arange(n), torch.randn(n, D, generator=g))
        caches.append((ccpu.read_rows_cpu(torch.arange(n))[0].double().to(dev()), C.PagedCache(ccpu.buf.to(dev()), D, R_, True, "latent")))
    q = torch.randn(T, nh, D, generator=g).to(dev()).to(BF16)
    slots = torch.randint(0, n, (T, W), generator=g, dtype=torch.int32).to(dev())
    tops = torch.randint(0, n, (T, K), generator=g, dtype=torch.int32).to(dev())
    tops[:, 7::31] = -1
    lens = torch.tensor([0, 1, 127, 128, 64, 0, 128])[torch.arange(T) % 7].to(torch.int32).to(dev())
    tlens = torch.tensor([0, 300, 129, 0, 128])[torch.arange(T) % 5].to(torch.int32).to(dev())
    lens[:150] = torch.where(torch.arange(150, device=dev()) % 3 == 0, 0, lens[:150])
    tlens[:150] = torch.where(torch.arange(150, device=dev()) % 3 == 0, 0, tlens[:150])
    lens[-20:], tlens[-20:] = 0, 0
    sink = torch.randn(nh, device=dev())
    out = A.sparse_mla(q, caches[0][1], slots, lens, caches[1][1], tops, tlens, sink, D ** -0.5)
    kv = torch.cat([caches[0][0][slots.long()], caches[1][0][tops.clamp(min=0).long()]], 1)
    at = torch.arange(W + K, device=dev())[None]
    there = torch.where(at < W, at < lens[:, None], at - W < tlens[:, None]) & torch.cat([slots >= 0, tops >= 0], 1)
    s = (q.double() @ kv.transpose(1, 2) * D ** -0.5).masked_fill(~there[:, None], -math.inf)
    p = torch.softmax(torch.cat([s, sink.double()[None, :, None].expand(T, -1, 1)], 2), 2)[:, :, :-1]
    ref = p @ kv
    assert rel_err(out, ref) < 3e-3                       # output rounded to bf16, weights to fp16
    none = (lens + tlens) == 0
    assert bool((out[none] == 0).all()) and rel_err(out[-21:], ref[-21:]) < 4e-3
    _lib.check_status()


@pytest.mark.parametrize("nh", [8, 64])
@pytest.mark.parametrize("off", [0, 4])
def test_sparse_mla_rows_beyond_fp16(nh, off):
    """Rows whose scales or rotated part pass fp16's range beside ordinary ones, maxima that first rise a little and then a lot, a
    list that ends inside a block, and an output that 16-byte copies cannot take (off).  Output rounded to bf16: 2^-9, 1.7e-3 in the
    2-norm; 3e-3 leaves as much again for fp16 weights."""
    D, R_, T, W, n = 512, 64, 150, 300, 512
    g = torch.Generator().manual_seed(3)
    rows = torch.randn(n, D, generator=g)
    size = torch.ones(n)
    size[1::4] = 3e4                                          # within the range, its products are not
    size[2::4] = 1e6                                          # scales up to 2^12, rotated values above 65504
    rows *= size[:, None]
    rows[3::8, D - R_:] *= 1e5                                # only the rotated part
    ccpu = C.PagedCache.allocate(n // 64, D, R_, True, "latent", "cpu")
    ccpu.write_rows_cpu(torch.arange(n), rows)
    kv = ccpu.read_rows_cpu(torch.arange(n))[0].double().to(dev())
    cg = C.PagedCache(ccpu.buf.to(dev()), D, R_, True, "latent")
    q = torch.randn(T, nh, D, generator=g).to(dev()).to(BF16)
    order = torch.argsort(size, stable=True).to(torch.int32)                # small rows first
    slots = order[torch.arange(W) * 512 // W].repeat(T, 1).to(dev())
    lens = torch.full((T,), W, dtype=torch.int32, device=dev())
    sink = torch.randn(nh, device=dev())
    scale = 2e-7
    buf = torch.zeros(T * nh * D + 8, dtype=BF16, device=dev())
    out = buf[off:off + T * nh * D].view(T, nh, D)
    _lib.call("stk_sparse_mla_tc_out", q, q.stride(0), cg.buf, cg.page_stride, cg.buf, cg.page_stride, slots, slots.stride(0), lens, None, 0,
              None, T, nh, D, R_, W, scale, out, out.stride(0), sink, None, None, _lib.status_buffer(), _lib.stream())
    k = kv[slots[0].long()]
    s = q.double() @ k.t() * scale
    p = torch.softmax(torch.cat([s, sink.double()[None, :, None].expand(T, -1, 1)], 2), 2)[:, :, :-1]
    assert rel_err(out, p @ k) < 3e-3
    assert float(buf[:off].abs().sum()) == 0 and float(buf[off + T * nh * D:].abs().sum()) == 0
    _lib.check_status()


@pytest.mark.parametrize("T", [12, 150])
@pytest.mark.parametrize("nh", [8, 32, 64])
@pytest.mark.parametrize("kind", ["small", "mixed", "far", "groups", "scales", "large queries", "small queries"])
def test_sparse_mla_magnitudes_that_fp16_does_not_hold(kind, nh, T):
    """Against 64 bits, per head: rows around 1e-6, alone and beside ordinary ones; a few rows of 1e12 beside ordinary ones that carry
    most of the weight; rows whose groups are 2^20 apart (every group of the output by itself); scales of 2^-67 as another writer may
    leave them; queries above 65504 and far below 2^-14 beside ordinary heads.  Partial rows and final ones.
    Output rounded to bf16, at most 2^-9 of a value (1.2e-3 in the 2-norm), weights to fp16 (2^-11); 3e-3 leaves half as much again."""
    D, R_, W, n = 512, 64, 300, 512
    g = torch.Generator().manual_seed(11)
    rows = torch.randn(n, D, generator=g)
    q = torch.randn(T, nh, D, generator=g)
    scale = D ** -0.5
    if kind == "small":
        rows, scale = rows * 1e-6, scale * 1e6
    elif kind == "mixed":
        rows[1::2] *= 1e-6
    elif kind == "far":
        rows[::30] *= 1e12
        scale *= 1e-12
    elif kind == "groups":
        rows *= (10.0 ** torch.tensor([3, 0, -3, 1, -2, 2, -1, -3])).repeat_interleave(64)
        scale *= 1e-3
    elif kind == "large queries":
        q[:, ::4] *= 2.0 ** 20
        scale *= 2.0 ** -20
    elif kind == "small queries":
        q *= 2.0 ** -30
        q[:, 0] = 0
        scale *= 2.0 ** 30
    ccpu = C.PagedCache.allocate(n // 64, D, R_, True, "latent", "cpu")
    ccpu.write_rows_cpu(torch.arange(n), rows)
    if kind == "scales":
        data = ccpu.buf[:, :64 * 576].view(-1, 64, 576)[:, :, D - R_:].contiguous().view(BF16)
        ccpu.buf[:, :64 * 576].view(-1, 64, 576)[:, :, D - R_:] = (data.float() * 2.0 ** -60).to(BF16).view(torch.uint8)
        ccpu.buf[:, 64 * 576:64 * 584].view(-1, 64, 8)[:, :, :7] -= 60
        scale *= 2.0 ** 60
    kv = ccpu.read_rows_cpu(torch.arange(n))[0].double().to(dev())
    cg = C.PagedCache(ccpu.buf.to(dev()), D, R_, True, "latent")
    q = q.to(dev()).to(BF16)
    slots = torch.arange(W, dtype=torch.int32, device=dev()).repeat(T, 1)
    lens = torch.full((T,), W, dtype=torch.int32, device=dev())
    sink = torch.randn(nh, generator=g).to(dev())
    out = A.sparse_mla(q, cg, slots, lens, None, None, None, sink, scale).double()
    s = q.double() @ kv[:W].t() * scale
    ref = torch.softmax(torch.cat([s, sink.double()[None, :, None].expand(T, -1, 1)], 2), 2)[:, :, :-1] @ kv[:W]
    cut = (T, nh, 8, 64) if kind == "groups" else (T, nh, 1, D)
    err = (out - ref).view(cut).pow(2).sum((0, 3)) / ref.view(cut).pow(2).sum((0, 3))
    assert float(err.sqrt().max()) < 3e-3
    _lib.check_status()


@pytest.mark.parametrize("nh", [8, 32, 64])
def test_sparse_mla_weights_relative_to_stale_maxima(nh):
    """A first block of rows 0 to 3 x log2(4 / 3) powers of two below two leading rows 3 x and -4 x of the last block, with weights 1
    and 3/4 of the largest: the maximum in use may stay (up to 2^1.5), so both weights are rounded to fp16.  Tolerance per element:
    2^-11 of each weight times what cancels, 3 + 4 * 3/4, over the sum of all weights; 1 % and 1e-5 for exponentials and output."""
    D, R_, T, W = 512, 64, 60, 128
    levels = [0, 1, 2, 3]
    rows = torch.zeros((1 + len(levels)) * 64, D)
    g = torch.Generator().manual_seed(0)
    x = torch.randint(0, 2, (D,), generator=g).float() * 2 - 1
    rows[0], rows[1] = 3 * x, -4 * x
    rows[0, 0], rows[1, 0] = 16, 15
    for i, n in enumerate(levels):
        rows[64 * (i + 1):64 * (i + 2), 0] = 16 - n
    ccpu = C.PagedCache.allocate(1 + len(levels), D, R_, True, "latent", "cpu")
    ccpu.write_rows_cpu(torch.arange(rows.shape[0]), rows)
    cg = C.PagedCache(ccpu.buf.to(dev()), D, R_, True, "latent")
    q = torch.zeros(T, nh, D, device=dev(), dtype=BF16)
    q[:, :, 0] = 1
    page = torch.arange(T) % len(levels) + 1
    slots = (page[:, None] * 64 + torch.arange(W)[None] % 64).to(torch.int32).to(dev())
    lens = torch.full((T,), W, dtype=torch.int32, device=dev())
    top = torch.tensor([[0, 1]], dtype=torch.int32, device=dev()).expand(T, -1).contiguous()
    top_lens = torch.full((T,), 2, dtype=torch.int32, device=dev())
    sink = torch.full((nh,), -1e30, device=dev())
    out = A.sparse_mla(q, cg, slots, lens, cg, top, top_lens, sink, math.log(4 / 3)).double().cpu()
    total = 1.75 + W * 0.75 ** torch.tensor(levels, dtype=torch.float64)[page - 1]
    assert bool((out[:, :, 1:].abs().amax((1, 2)) <= 6 * 2.0 ** -11 * 1.01 / total + 1e-5).all())


@pytest.mark.parametrize("nh", [8, 32, 64])
def test_sparse_mla_weights_are_relative_to_the_exact_maximum(nh):
    """Weights relative to the largest: 1 and 3/4 are bf16 numbers, so two leading rows 3 x and -4 x in the last block cancel whatever
    came before them -- a first block of rows 4 to 9 powers of two lower, a different distance per token, which a maximum taken from
    it would turn into weights that bf16 rounds.  Tolerance: 3/4 is met to the fp32 rounding of scores below 2^4 and of their
    difference (a few 2^-20 of a weight), times the 4 + 3 that are subtracted; 1e-4 is ten times that, and a tenth of what rounded weights leave."""
    D, R_, T, W = 512, 64, 60, 128
    levels = list(range(4, 14))
    rows = torch.zeros((1 + len(levels)) * 64, D)
    g = torch.Generator().manual_seed(0)
    x = torch.randint(0, 2, (D,), generator=g).float() * 2 - 1
    rows[0], rows[1] = 3 * x, -4 * x                          # leading rows
    rows[0, 0], rows[1, 0] = 16, 15
    for i, n in enumerate(levels):                            # a page of rows for each distance of the first block
        rows[64 * (i + 1):64 * (i + 2), 0] = 16 - n
    ccpu = C.PagedCache.allocate(1 + len(levels), D, R_, True, "latent", "cpu")
    ccpu.write_rows_cpu(torch.arange(rows.shape[0]), rows)
    assert torch.equal(ccpu.read_rows_cpu(torch.arange(rows.shape[0]))[0].float(), rows)
    cg = C.PagedCache(ccpu.buf.to(dev()), D, R_, True, "latent")
    q = torch.zeros(T, nh, D, device=dev(), dtype=BF16)
    q[:, :, 0] = 1
    page = torch.arange(T) % len(levels) + 1
    slots = (page[:, None] * 64 + torch.arange(W)[None] % 64).to(torch.int32).to(dev())
    lens = torch.full((T,), W, dtype=torch.int32, device=dev())
    top = torch.tensor([[0, 1]], dtype=torch.int32, device=dev()).expand(T, -1).contiguous()
    top_lens = torch.full((T,), 2, dtype=torch.int32, device=dev())
    sink = torch.full((nh,), -1e30, device=dev())
    scale = math.log(4 / 3)
    out = A.sparse_mla(q, cg, slots, lens, cg, top, top_lens, sink, scale).float()
    assert float(out[:, :, 1:].abs().max()) < 1e-4
    # the first value does not cancel: against the weights in 64 bits, one rounding of the weights and one of the result
    lead = torch.tensor([16 - n for n in levels], dtype=torch.float64)[page - 1]
    s = torch.stack([lead, torch.full_like(lead, 16), torch.full_like(lead, 15)], 1)
    w = torch.exp((s - 16) * scale) * torch.tensor([W, 1, 1], dtype=torch.float64)
    ref = (w * s).sum(1) / w.sum(1)
    assert float((out[:, :, 0].double().cpu() - ref[:, None]).abs().max()) < 2 ** -7 * 16


@pytest.mark.parametrize("T", [12, 40])
def test_sparse_mla_rotates_its_output_in_32_bits(T):
    """One rounding of the rotated dims, by the combine pass and by the kernel that writes final rows: every value within half a unit
    of bf16 (2^-8 of it) of the rotation in 64 bits.  1e-5 of the pair's length covers fp32: weights from exponentials good to 1e-6,
    angles up to 60 with 2^-24 of error each; a second rounding would add up to 4e-3 of it, also where the value itself is small."""
    D, R_, W, nh = 512, 64, 128, 8
    torch.manual_seed(T)
    ccpu = C.PagedCache.allocate(1, D, R_, True, "latent", "cpu")
    ccpu.write_rows_cpu(torch.arange(64), torch.randn(64, D))
    cg = C.PagedCache(ccpu.buf.to(dev()), D, R_, True, "latent")
    q = torch.randn(T, nh, D).to(BF16)
    slots = torch.arange(T * W).view(T, W).to(torch.int32) % 64
    lens = torch.ones(T, dtype=torch.int32)                       # one row and the sink: the weight in bf16 is 1, the rest fp32
    sink = torch.randn(nh)
    pos, inv = torch.arange(T, dtype=torch.int64) % 60, Fn.inv_freq(64, 10000.0, "cpu")
    out = A.sparse_mla(q.to(dev()), cg, slots.to(dev()), lens.to(dev()), None, None, None, sink.to(dev()), D ** -0.5,
                       inv_rope=(pos.to(dev()), inv.to(dev()))).cpu().double()[:, :, D - R_:]
    row = ccpu.read_rows_cpu(slots[:, 0].long())[0].double()
    s = torch.einsum("thd,td->th", q.double(), row) * D ** -0.5
    v = (torch.sigmoid(s - sink.double())[:, :, None] * row[:, None])[:, :, D - R_:]
    ang = (pos.double()[:, None] * inv.double())[:, None]
    x, y = v[:, :, 0::2], v[:, :, 1::2]
    ref = torch.stack([x * ang.cos() + y * ang.sin(), y * ang.cos() - x * ang.sin()], -1).flatten(2)
    length = (x * x + y * y).sqrt().repeat_interleave(2, 2)
    assert float(((out - ref).abs() / (2.0 ** -8 * ref.abs() + 1e-5 * length)).max()) < 1


@pytest.mark.parametrize("tokens", [9, 36, 37, 64, 148, 149])
@pytest.mark.parametrize("K", [0, 640])
@pytest.mark.parametrize("nh", [16, 64])
def test_sparse_mla_splits_rows_over_idle_sms(tokens, K, nh):
    """Both sides of each line of the split rule, with lists that fill their capacity, end in any split, or are empty; one and two
    softmax warps per quarter of the rows.
    Tolerance of the tests around it: fp8 rows against the fp32 reference of the same rows."""
    torch.manual_seed(tokens)
    D, R_, W, n_pages = 512, 64, 128, 24
    ccpu = C.PagedCache.allocate(n_pages, D, R_, True, "latent", "cpu")
    ccpu.write_rows_cpu(torch.arange(n_pages * 64), torch.randn(n_pages * 64, D))
    cg = C.PagedCache(ccpu.buf.to(dev()), D, R_, True, "latent")
    q = torch.randn(tokens, nh, D).to(BF16)
    swa_slots = torch.randint(0, n_pages * 64, (tokens, W), dtype=torch.int32)
    swa_lens = torch.randint(0, W + 1, (tokens,), dtype=torch.int32)
    top = torch.randint(0, n_pages * 64, (tokens, max(K, 1)), dtype=torch.int32) if K else None
    top_lens = torch.randint(0, K + 1, (tokens,), dtype=torch.int32) if K else None
    swa_lens[0], swa_lens[1] = W, 0
    if K:
        top_lens[0], top_lens[1], top_lens[2] = K, 0, 1
    sink = torch.randn(nh)
    out = A.sparse_mla(q.to(dev()), cg, swa_slots.to(dev()), swa_lens.to(dev()), cg if K else None, top.to(dev()) if K else None,
                       top_lens.to(dev()) if K else None, sink.to(dev()), D ** -0.5)
    sub = torch.tensor(sorted({0, 1, 2, tokens // 2, tokens - 1}))
    ref = A.sparse_mla(q[sub], ccpu, swa_slots[sub], swa_lens[sub], ccpu if K else None, top[sub] if K else None,
                       top_lens[sub] if K else None, sink, D ** -0.5)
    assert rel_err(out[sub.to(dev())], ref) < 1.2e-2
    assert float(out[1].float().abs().max()) == 0.0


@pytest.mark.parametrize("nh", [64, 8])
def test_sparse_mla_direct_output_matches_split_path(nh):
    """Steps with many tokens take the single-split kernel that writes the final rows itself (sink merge, normalisation,
    inverse RoPE in its epilogue); compare with the fp32 reference and with the partial + combine path."""
    torch.manual_seed(9)
    D, R_, T, W, K = 512, 64, 320, 128, 256
    n_pages = 24
    rows = torch.randn(n_pages * 64, D)
    ccpu = C.PagedCache.allocate(n_pages, D, R_, True, "latent", "cpu")
    ccpu.write_rows_cpu(torch.arange(n_pages * 64), rows)
    cg = C.PagedCache(ccpu.buf.to(dev()), D, R_, True, "latent")
    q = torch.randn(T, nh, D, device=dev()).to(BF16)
    swa_slots = torch.randint(0, n_pages * 64, (T, W), dtype=torch.int32, device=dev())
    swa_lens = torch.randint(0, W + 1, (T,), dtype=torch.int32, device=dev())
    topk_slots = torch.randint(0, n_pages * 64, (T, K), dtype=torch.int32, device=dev())
    topk_slots[0, 3] = -1
    topk_lens = torch.randint(0, K + 1, (T,), dtype=torch.int32, device=dev())
    swa_lens[1] = 0
    topk_lens[1] = 0                      # a token without any key: only the sink has mass, output zero
    sink = torch.randn(nh, device=dev())
    pos = torch.randint(0, 50000, (T,), device=dev(), dtype=torch.int64)
    inv = Fn.inv_freq(R_, 10000.0, dev())
    assert A.MLA_DIRECT_OUT
    out = A.sparse_mla(q, cg, swa_slots, swa_lens, cg, topk_slots, topk_lens, sink, D ** -0.5, inv_rope=(pos, inv))
    A.MLA_DIRECT_OUT = False
    try:
        split = A.sparse_mla(q, cg, swa_slots, swa_lens, cg, topk_slots, topk_lens, sink, D ** -0.5, inv_rope=(pos, inv))
    finally:
        A.MLA_DIRECT_OUT = True
    assert rel_err(out, split) < 4e-3
    assert float(out[1].float().abs().max()) == 0.0
    sub = slice(0, 6)
    ref = A.sparse_mla(q[sub].cpu(), ccpu, swa_slots[sub].cpu(), swa_lens[sub].cpu(), ccpu, topk_slots[sub].cpu(),
                       topk_lens[sub].cpu(), sink.cpu(), D ** -0.5, inv_rope=(pos[sub].cpu(), inv.cpu()))
    assert rel_err(out[sub], ref) < 1.2e-2


@pytest.mark.parametrize("nh,T,K", [(64, 300, 512), (64, 9, 1100), (40, 300, 130), (16, 300, 300)])
def test_sparse_mla_maxima_that_keep_growing(nh, T, K):
    """Keys whose scores grow along the list by far more than the factor a stale maximum may be off by (the accumulators are
    rescaled block after block), and lists that fall as steeply (they never are); ragged ends, gaps, whole blocks of gaps."""
    torch.manual_seed(21)
    D, R_, W = 512, 64, 128
    n_pages = 24
    n = n_pages * 64
    rows = torch.randn(n, D) * (0.2 + 6.0 * torch.arange(n)[:, None] / n)
    ccpu = C.PagedCache.allocate(n_pages, D, R_, True, "latent", "cpu")
    ccpu.write_rows_cpu(torch.arange(n), rows)
    cg = C.PagedCache(ccpu.buf.to(dev()), D, R_, True, "latent")
    q = (4 * torch.randn(T, nh, D, device=dev())).to(BF16)
    swa = torch.sort(torch.randint(0, n, (T, W), device=dev()), 1)[0].to(torch.int32)
    top = torch.sort(torch.randint(0, n, (T, K), device=dev()), 1)[0].to(torch.int32)
    top[::2], swa[::2] = top[::2].flip(1), swa[::2].flip(1)
    top[torch.rand(T, K, device=dev()) < 0.1] = -1
    swa[4], top[5, :K // 2] = -1, -1
    swa_lens = torch.randint(0, W + 1, (T,), dtype=torch.int32, device=dev())
    top_lens = torch.randint(0, K + 1, (T,), dtype=torch.int32, device=dev())
    swa_lens[:4], top_lens[:4] = W, torch.tensor([K, K, 0, 1], dtype=torch.int32)
    sink = torch.randn(nh, device=dev())
    out = A.sparse_mla(q, cg, swa, swa_lens, cg, top, top_lens, sink, D ** -0.5)
    sub = torch.arange(min(T, 9))
    ref = A.sparse_mla(q[:9].cpu(), ccpu, swa[:9].cpu(), swa_lens[:9].cpu(), ccpu, top[:9].cpu(), top_lens[:9].cpu(), sink.cpu(), D ** -0.5)
    # weights and results are rounded to bf16 (2^-9 each); scores of a few hundred carry fp32 rounding into the weights
    for i in sub.tolist():
        assert rel_err(out[i], ref[i]) < 1.2e-2 or float(ref[i].abs().max()) < 1e-6


@pytest.mark.parametrize("nh", [64, 16])
def test_sparse_mla_codes_and_scales(nh):
    """Every e4m3 code under ordinary and extreme scale bytes (0 counts as scale zero), rotated parts as they are; NaN codes reach
    the tokens that attend to them and no others."""
    torch.manual_seed(22)
    D, R_, T, W = 512, 64, 300, 128
    n_pages = 4
    buf = torch.zeros(n_pages, C.PagedCache.page_bytes(D, R_, True, "latent"), dtype=torch.uint8)
    codes = torch.randint(0, 256, (n_pages, 64, 448), dtype=torch.uint8)
    codes[(codes & 0x7f) == 0x7f] = 0x7e
    rope = torch.randn(n_pages, 64, R_).to(BF16).view(torch.uint8)
    scales = torch.zeros(n_pages, 64, 8, dtype=torch.uint8)
    scales[:, :, :7] = torch.tensor([0, 1, 60, 110, 119, 120, 121, 127, 133, 134, 135, 137], dtype=torch.uint8)[
        torch.randint(0, 12, (n_pages, 64, 7))]
    codes[1, 7, 100] = 0xff
    buf[:, :64 * 576] = torch.cat([codes, rope], 2).view(n_pages, -1)
    buf[:, 64 * 576:64 * 584] = scales.view(n_pages, -1)
    cg = C.PagedCache(buf.to(dev()), D, R_, True, "latent")
    value = torch.cat([(codes.view(torch.float8_e4m3fn).double().view(n_pages, 64, 7, 64)
                        * torch.where(scales[:, :, :7] == 0, 0.0, torch.exp2(scales[:, :, :7].double() - 127))[..., None]).view(n_pages * 64, 448),
                       rope.view(BF16).double().view(n_pages * 64, R_)], 1)
    q = (2.0 ** -19 * torch.randn(T, nh, D, device=dev())).to(BF16)
    slots = torch.randint(0, n_pages * 64, (T, W), dtype=torch.int32, device=dev())
    slots[slots == 71] = 70
    slots[3, 5] = 71
    lens = torch.full((T,), W, dtype=torch.int32, device=dev())
    sink = torch.zeros(nh, device=dev())
    out = A.sparse_mla(q, cg, slots, lens, None, None, None, sink, D ** -0.5)
    assert bool(out[3].isnan().all()) and int(out.isnan().any(2).any(1).sum()) == 1
    kv = value.to(dev())[slots.long()]
    p = torch.softmax(torch.cat([q.double() @ kv.transpose(1, 2) * D ** -0.5, torch.zeros(T, nh, 1, device=dev(), dtype=torch.float64)], 2), 2)
    ref = p[:, :, :-1] @ kv
    keep = torch.arange(T, device=dev()) != 3
    for part in (slice(0, 448), slice(448, 512)):           # weights and results are rounded to bf16
        assert rel_err(out[keep][:, :, part], ref[keep][:, :, part]) < 8e-3


@pytest.mark.parametrize("scoring", ["sigmoid", "sqrtsoftplus"])
def test_router(scoring):
    T, E, k = 33, 256, 6
    logits = torch.randn(T, E, device=dev())
    bias = (torch.rand(E, device=dev()) * 0.2 - 0.1)
    ids, w = M.router(logits, bias, k, scoring, True, 2.5)
    rid, rw = R.route(logits, bias, k, scoring, True, 2.5)
    assert torch.equal(ids.sort(-1).values, rid.sort(-1).values)
    assert torch.allclose(w.sum(-1), rw.sum(-1), rtol=1e-4)
    tid2eid = torch.randint(0, E, (1000, k), dtype=torch.int32, device=dev())
    toks = torch.randint(0, 1000, (T,), device=dev())
    ids2, w2 = M.router(logits, None, k, scoring, True, 1.0, tid2eid, toks)
    assert torch.equal(ids2, tid2eid[toks])
    rid2, rw2 = R.route(logits, None, k, scoring, True, 1.0, tid2eid[toks])
    assert torch.allclose(w2, rw2, rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("T,H,I,E", [(1, 4096, 2048, 16), (7, 4096, 2048, 16), (5, 256, 128, 8)])
def test_moe_experts_nvfp4(T, H, I, E):
    torch.manual_seed(11)
    k = 2 if E == 8 else 6
    w13 = torch.randn(E, 2 * I, H) * 0.02
    w2 = torch.randn(E, H, I) * 0.02
    ew = M.ExpertWeights.from_master(w13, w2, "nvfp4", dev())
    x = torch.randn(T, H, device=dev()).to(BF16)
    logits = torch.randn(T, E, device=dev())
    ids, w = M.router(logits, None, k, "sigmoid", True, 1.0)
    shared = torch.randn(T, H, device=dev()).to(BF16)
    out = M.moe_experts(x, ids, w, ew, 10.0, shared)
    d13, d2 = ew.dequant()
    ref = R.moe_experts(x, ids, w, d13, d2, 10.0) + shared.float()
    assert rel_err(out, ref) < 1.5e-2
    # expert-parallel slice: only experts [E/2, E) are local
    ew_hi = M.ExpertWeights(ew.w13[E // 2:], ew.w2[E // 2:], ew.s13[E // 2:], ew.s2[E // 2:], ew.g13[E // 2:],
                            ew.g2[E // 2:], E // 2)
    out_hi = M.moe_experts(x, ids, w, ew_hi, 10.0)
    ref_hi = R.moe_experts(x, ids, w, d13[E // 2:], d2[E // 2:], 10.0, E // 2)
    assert rel_err(out_hi, ref_hi) < 1.5e-2


def test_moe_experts_sliced_along_the_intermediate_dimension():
    """Decode steps under tensor parallelism: every rank holds 1/tp of every expert's intermediate rows; the ranks'
    partial results add up to the whole experts' output."""
    torch.manual_seed(12)
    T, H, I, E, k, tp = 2, 4096, 2048, 16, 6, 8
    w13 = torch.randn(E, 2 * I, H) * 0.02
    w2 = torch.randn(E, H, I) * 0.02
    x = torch.randn(T, H, device=dev()).to(BF16)
    ids, w = M.router(torch.randn(T, E, device=dev()), None, k, "sigmoid", True, 1.0)
    il = I // tp
    total = torch.zeros(T, H)
    ref = torch.zeros(T, H)
    for r in range(tp):
        sl = slice(r * il, (r + 1) * il)
        w13_r = torch.cat([w13[:, :I][:, sl], w13[:, I:][:, sl]], 1).contiguous()
        w2_r = w2[:, :, sl].contiguous()
        ew = M.ExpertWeights.from_master(w13_r, w2_r, "nvfp4", dev())
        out = M.moe_experts(x, ids, w, ew, 10.0, None, E)
        d13, d2 = ew.dequant()
        ref += R.moe_experts(x, ids, w, d13, d2, 10.0).float().cpu()
        total += out.float().cpu()
    assert rel_err(total, ref) < 1.5e-2
    full = R.moe_experts(x, ids, w, w13.to(dev()), w2.to(dev()), 10.0).float().cpu()
    assert rel_err(total, full) < 0.25          # NVFP4 quantisation of the weights
    torch.cuda.synchronize()
    _lib.check_status()


def test_gumbel_argmax_and_coupling():
    B, N, V = 3, 5, 129280
    logits = torch.randn(B * (N + 1), V, device=dev())
    temp = torch.tensor([0.6, 0.0, 1.0], device=dev())
    seed = torch.tensor([1, 2 ** 40 + 7, 3], device=dev(), dtype=torch.int64)
    pos = torch.tensor([10, 2000, 5], device=dev(), dtype=torch.int64)
    tok, proc = S.gumbel_argmax(logits, temp, seed, pos, rows_per_request=N + 1, want_processed=True)
    rtok, rproc = S.gumbel_argmax(logits.cpu(), temp.cpu(), seed.cpu(), pos.cpu(), rows_per_request=N + 1,
                                  want_processed=True)
    assert torch.equal(tok.cpu(), rtok)
    assert torch.allclose(proc.cpu(), rproc, rtol=1e-5, atol=1e-5)
    # same (seed, pos) => same noise: sampling identical logits twice gives identical tokens
    tok2, _ = S.gumbel_argmax(logits, temp, seed, pos, rows_per_request=N + 1)
    assert torch.equal(tok, tok2)
    ver = tok.view(B, N + 1)
    draft = ver[:, :N].clone()
    draft[0, 2] = (draft[0, 2] + 1) % V
    acc, em = S.coupled_accept(ver, draft)
    assert acc.tolist() == [2, N, N]
    assert em[0].tolist()[:3] == ver[0].tolist()[:3] and (em[0, 3:] == -1).all()


def test_markov_topk_bias():
    B, V, Rk = 2, 129280, 256
    base = torch.randn(B, V, device=dev()).to(BF16)
    w2 = (torch.randn(V, Rk, device=dev()) * 0.02).to(BF16)
    emb = torch.randn(B, Rk, device=dev()).to(BF16)
    out = S.markov_topk_bias(base, w2, emb, 512)
    ref = R.markov_bias_topk(base, w2, emb, 512)
    fin = torch.isfinite(ref)
    assert torch.equal(torch.isfinite(out), fin) or (torch.isfinite(out).sum(-1) == 512).all()
    assert (torch.isfinite(out).sum(-1) == 512).all()
    both = fin & torch.isfinite(out)
    assert torch.allclose(out[both], ref[both], rtol=1e-3, atol=1e-3)
    dense = S.markov_topk_bias(base, w2, emb, 0)
    assert torch.allclose(dense, R.markov_bias_topk(base, w2, emb, 0), rtol=1e-3, atol=1e-3)


def test_swa_indices_and_slots():
    pos = torch.tensor([0, 5, 200, -1], device=dev(), dtype=torch.int64)
    tok_req = torch.tensor([0, 1, 1, -1], dtype=torch.int32, device=dev())
    bt = torch.tensor([[3, 4, 5, 6], [7, 8, 9, 10]], dtype=torch.int32, device=dev())
    s, l = A.swa_indices(pos, tok_req, bt, 128)
    rs, rl = A.swa_indices(pos.cpu(), tok_req.cpu(), bt.cpu(), 128)
    assert torch.equal(s.cpu(), rs) and torch.equal(l.cpu(), rl)
    topk = torch.tensor([[0, 65, -1, 130], [1, 2, 3, 4]], dtype=torch.int32, device=dev())
    sl, ln = A.topk_to_slots(topk, bt, tok_req[:2].contiguous(), 256)
    rsl, rln = A.topk_to_slots(topk.cpu(), bt.cpu(), tok_req[:2].cpu(), 256)
    assert torch.equal(sl.cpu(), rsl) and torch.equal(ln.cpu(), rln)


@pytest.mark.parametrize("dtype", ["bf16", "fp8"])
@pytest.mark.parametrize("T", [1, 40, 300])
def test_gemm_grouped_block_diagonal(dtype, T):
    torch.manual_seed(2)
    G, Ng, K = 4, 256, 512
    x = torch.randn(T, G * K, device=dev()).to(BF16)
    ws = [torch.randn(Ng, K, device=dev()) * 0.05 for _ in range(G)]
    lws = [Fn.LinearWeight.from_master(w, dtype, dev()) for w in ws]
    stacked = Fn.LinearWeight(torch.cat([l.w for l in lws], 0).contiguous(),
                              torch.cat([l.scale for l in lws], 0).contiguous() if dtype == "fp8" else None)
    out = Fn.linear(x, stacked, out_dtype=F32, groups=G)
    for g in range(G):
        xg = x[:, g * K:(g + 1) * K]
        if dtype == "fp8" and T > 4:
            xq, xs = R.quant_fp8_group128_act(xg)
            ref = R.dequant_fp8_group128_act(xq, xs) @ lws[g].dequant().t()
        else:
            ref = xg.float() @ lws[g].dequant().t()
        assert rel_err(out[:, g * Ng:(g + 1) * Ng], ref) < 3e-3


@pytest.mark.parametrize("T,N,K", [(64, 4096, 8192), (100, 384, 1024), (128, 4096, 2048), (256, 4096, 8192), (300, 640, 2048)])
def test_gemm_splitk_wide_tiles(T, N, K):
    torch.manual_seed(3)
    x = torch.randn(T, K, device=dev()).to(BF16)
    w = torch.randn(N, K, device=dev()).to(BF16)
    ref = x.float() @ w.float().t()
    for splits in (2, 4):
        assert rel_err(Fn.linear(x, Fn.LinearWeight(w), splits=splits), ref) < 1e-2


@pytest.mark.parametrize("dtype", ["bf16", "fp8"])
@pytest.mark.parametrize("T", [1, 3, 4])
@pytest.mark.parametrize("N,K", [(2048, 4096), (40960, 1536), (4096, 8192), (176, 256)])
def test_skinny_linear(dtype, T, N, K):
    torch.manual_seed(T)
    x = torch.randn(T, K, device=dev()).to(BF16)
    w = torch.randn(N, K, device=dev()) * 0.05
    lw = Fn.LinearWeight.from_master(w, dtype, dev())
    ref = x.float() @ lw.dequant().t()
    out = Fn.linear(x, lw, out_dtype=F32)          # T <= 4 routes to the weight-streaming kernel
    assert rel_err(out, ref) < 2e-3
    out16 = Fn.linear(x, lw)
    assert rel_err(out16, ref) < 1e-2


@pytest.mark.parametrize("T", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K,groups", [(16, 128, 1), (48, 8192, 1), (4112, 384, 1), (64, 256, 4), (40, 256, 1), (48, 144, 1)])
def test_skinny_bf16_few_tokens(T, N, K, groups):
    """One to four tokens under bf16 weights: the smallest and largest K, rows and K of the other kernel (40 rows, K 144), groups, strided
    rows and values beyond fp16.  A sum in fp32 of K products with partial sums in any order is off by at most K x 2^-24 of the sum of
    magnitudes, a value of bf16 by 2^-8 of itself."""
    torch.manual_seed(T + N)
    x = (torch.randn(T, K * groups + 8, device=dev()) * 1e5).to(BF16)[:, :K * groups]
    w = (torch.randn(N, K, device=dev()) * 0.05).to(BF16)
    xd, wd = x.double().view(T, groups, K), w.double().view(groups, N // groups, K)
    ref = torch.einsum("tgk,gnk->tgn", xd, wd).reshape(T, N)
    slack = torch.einsum("tgk,gnk->tgn", xd.abs(), wd.abs()).reshape(T, N) * K * 2.0 ** -24
    if groups > 1 or (N % 16 == 0 and K % 128 == 0):
        lw = Fn.LinearWeight(w)
        assert bool(((Fn.linear(x, lw, out_dtype=F32, groups=groups).double() - ref).abs() <= slack).all())
        assert bool(((Fn.linear(x, lw, groups=groups).double() - ref).abs() <= slack + ref.abs() * 2.0 ** -8).all())
    else:                                          # fp16 activations: no larger than 65504
        small = (x * 1e-5).to(BF16)
        ref = small.double() @ w.double().t()
        assert rel_err(Fn.linear(small, Fn.LinearWeight(w), out_dtype=F32), ref.float()) < 2e-3


def test_skinny_linear_grouped():
    G, Ng, K, T = 8, 1024, 4096, 2
    x = torch.randn(T, G * K, device=dev()).to(BF16)
    w = torch.randn(G * Ng, K, device=dev()) * 0.05
    lw = Fn.LinearWeight.from_master(w, "fp8", dev())
    out = Fn.linear(x, lw, out_dtype=F32, groups=G)
    wd = lw.dequant().view(G, Ng, K)
    ref = torch.einsum("tgk,gnk->tgn", x.float().view(T, G, K), wd).reshape(T, G * Ng)
    assert rel_err(out, ref) < 2e-3


@pytest.mark.parametrize("dtype", ["bf16", "fp8"])
def test_skinny_swiglu(dtype):
    T, I, K = 2, 2048, 4096
    x = torch.randn(T, K, device=dev()).to(BF16)
    w = torch.randn(2 * I, K, device=dev()) * 0.03
    lw = Fn.LinearWeight.from_master(w, dtype, dev())
    act = Fn.linear_swiglu(x, lw, 10.0)
    gu = x.float() @ lw.dequant().t()
    ref = R.swiglu_clamp(gu[:, :I], gu[:, I:], 10.0)
    assert rel_err(act, ref) < 1e-2


@pytest.mark.parametrize("dtype", ["bf16", "fp8"])
@pytest.mark.parametrize("T", [5, 6, 8])
@pytest.mark.parametrize("N,K", [(2048, 4096), (16160, 1536), (4096, 8192), (176, 256), (576, 4096)])
def test_skinny_mma_linear_five_to_eight_tokens(dtype, T, N, K, monkeypatch):
    """Five to eight tokens: the warp-level tensor-core stream (fp8 activations quantised per 128 values inside the
    kernel, exactly like the GEMM path)."""
    monkeypatch.setattr(Fn, "SKINNY_MAX_T", 8)
    torch.manual_seed(T + N)
    buf = torch.randn(T, K + 256, device=dev()).to(BF16) * 2.0        # a strided view
    x = buf[:, :K]
    w = torch.randn(N, K, device=dev()) * 0.05
    lw = Fn.LinearWeight.from_master(w, dtype, dev())
    before = _lib.launch_count
    out = Fn.linear(x, lw, out_dtype=F32)
    if Fn._skinny_ok(x, T, K, dtype == "fp8", N):   # (the largest fp8 case at 8 tokens exceeds the staging area)
        assert _lib.launch_count == before + 1      # one kernel: no separate quantisation, no split-K reduction
    if dtype == "fp8":
        xq, xs = R.quant_fp8_group128_act(x.contiguous())
        ref = R.dequant_fp8_group128_act(xq, xs) @ lw.dequant().t()
    else:
        ref = x.float() @ lw.dequant().t()
    assert rel_err(out, ref) < 2e-3
    assert rel_err(Fn.linear(x, lw), ref) < 1e-2
    torch.cuda.synchronize()
    _lib.check_status()


@pytest.mark.parametrize("T", [9, 16, 33, 64])
@pytest.mark.parametrize("N,K", [(256, 4096), (512, 4096), (1024, 1536)])
def test_skinny_mma_narrow_weights_up_to_64_tokens(T, N, K, monkeypatch):
    """The router gate at decode batch sizes: the bf16 weight (<= 4 MB) is streamed once per group of eight tokens
    instead of through a mostly empty tensor-core tile with split-K (an option: STK_SKINNY_NARROW=1)."""
    monkeypatch.setattr(Fn, "SKINNY_NARROW", True)
    torch.manual_seed(T * 7 + N)
    x = torch.randn(T, K, device=dev()).to(BF16)
    lw = Fn.LinearWeight((torch.randn(N, K, device=dev()) * 0.05).to(BF16))
    assert Fn._skinny_ok(x, T, K, False, N, N)
    before = _lib.launch_count
    out = Fn.linear(x, lw, out_dtype=F32)
    assert _lib.launch_count == before + 1
    ref = x.float() @ lw.dequant().t()
    assert rel_err(out, ref) < 2e-3
    assert (out - ref).abs().max().item() < 0.02 * ref.abs().max().item()
    nw = (1 + 0.1 * torch.randn(K, device=dev())).to(BF16)
    xn = R.rms_norm(x, nw, 1e-6).to(BF16)
    assert rel_err(Fn.linear(x, lw, norm=(nw, 1e-6)), xn.float() @ lw.dequant().t()) < 1e-2
    # fp8 weights at these batch sizes stay on the tensor-core tile
    lw8 = Fn.LinearWeight.from_master(torch.randn(N, K, device=dev()) * 0.05, "fp8", dev())
    assert not Fn._skinny_ok(x, T, K, True, N, N)
    ref8 = R.dequant_fp8_group128_act(*R.quant_fp8_group128_act(x)) @ lw8.dequant().t()
    assert rel_err(Fn.linear(x, lw8, out_dtype=F32), ref8) < 2e-3
    torch.cuda.synchronize()
    _lib.check_status()


@pytest.mark.parametrize("dtype", ["bf16", "fp8"])
def test_skinny_mma_grouped_and_swiglu(dtype, monkeypatch):
    monkeypatch.setattr(Fn, "SKINNY_MAX_T", 8)
    torch.manual_seed(9)
    G, Ng, K, T = 8, 1024, 512, 6
    x = torch.randn(T, G * K, device=dev()).to(BF16)
    lw = Fn.LinearWeight.from_master(torch.randn(G * Ng, K, device=dev()) * 0.05, dtype, dev())
    out = Fn.linear(x, lw, out_dtype=F32, groups=G)
    wd = lw.dequant().view(G, Ng, K)
    if dtype == "fp8":
        xf = torch.cat([R.dequant_fp8_group128_act(*R.quant_fp8_group128_act(x[:, g * K:(g + 1) * K].contiguous()))
                        for g in range(G)], 1)
    else:
        xf = x.float()
    ref = torch.einsum("tgk,gnk->tgn", xf.view(T, G, K), wd).reshape(T, G * Ng)
    assert rel_err(out, ref) < 2e-3
    I, K2 = 2048, 4096
    x2 = torch.randn(T, K2, device=dev()).to(BF16)
    lw2 = Fn.LinearWeight.from_master(torch.randn(2 * I, K2, device=dev()) * 0.03, dtype, dev())
    act = Fn.linear_swiglu(x2, lw2, 10.0)
    assert act is not None
    x2f = R.dequant_fp8_group128_act(*R.quant_fp8_group128_act(x2)) if dtype == "fp8" else x2.float()
    gu = x2f @ lw2.dequant().t()
    assert rel_err(act, R.swiglu_clamp(gu[:, :I], gu[:, I:], 10.0)) < 1e-2
    torch.cuda.synchronize()
    _lib.check_status()


@pytest.mark.parametrize("T,E,k", [(64, 16, 6), (700, 16, 6), (300, 32, 2), (2048, 8, 2)])
def test_moe_grouped_gemm_nvfp4(T, E, k):
    """Batches beyond a handful of pairs go through the tcgen05 grouped GEMM."""
    torch.manual_seed(13)
    H, I = 1024, 512
    w13 = torch.randn(E, 2 * I, H) * 0.03
    w2 = torch.randn(E, H, I) * 0.03
    ew = M.ExpertWeights.from_master(w13, w2, "nvfp4", dev())
    x = torch.randn(T, H, device=dev()).to(BF16)
    logits = torch.randn(T, E, device=dev())
    logits[:, 0] -= 100.0                               # expert 0 never selected: an empty group
    ids, w = M.router(logits, None, k, "sigmoid", True, 1.0)
    out = M.moe_experts(x, ids, w, ew, 10.0, None, E)
    d13, d2 = ew.dequant()
    ref = R.moe_experts(x, ids, w, d13, d2, 10.0)
    assert rel_err(out, ref) < 1.5e-2
    M.USE_GROUPED_GEMM = False
    try:
        out2 = M.moe_experts(x, ids, w, ew, 10.0, None, E)
    finally:
        M.USE_GROUPED_GEMM = True
    assert rel_err(out, out2) < 1.5e-2


@pytest.mark.parametrize("T", [9, 47, 48, 100, 127, 128, 129, 300, 700])
@pytest.mark.parametrize("N,K", [(72, 192), (200, 512), (512, 2048), (2048, 4096), (20000, 1664)])
def test_gemm_fp8_token_tiles(T, N, K):
    """Ragged tiles of tokens and weight rows, a K that ends inside a block, K split over two and four CTAs of a cluster (with an
    uneven last part), several tiles per CTA, fp32 results and rows of a wider matrix."""
    torch.manual_seed(T + N)
    lw = Fn.LinearWeight.from_master(torch.randn(N, K, device=dev()) * 0.05, "fp8", dev())
    x = torch.randn(T, K, device=dev()).to(BF16)
    xq, xs = R.quant_fp8_group128_act(x)
    ref = R.dequant_fp8_group128_act(xq, xs).double() @ lw.dequant().double().t()
    out = Fn.linear(x, lw)
    assert rel_err(out, ref) < 3e-3                       # bf16 results; the activation's codes may differ at ties
    wide = torch.full((T, N + 24), 7.0, dtype=F32, device=dev())
    Fn.linear(x, lw, out=wide[:, 8:8 + N])
    assert rel_err(wide[:, 8:8 + N], ref) < 2.5e-3
    assert bool((wide[:, :8] == 7.0).all()) and bool((wide[:, 8 + N:] == 7.0).all())


@pytest.mark.parametrize("T,N,K", [(520, 6136, 272), (600, 6144, 1664), (2100, 2040, 1040), (700, 24600, 128)])
def test_gemm_fp8_pairs_of_ctas(T, N, K):
    """Products that pairs of CTAs take: ragged tiles of tokens and weight rows (a second CTA without tokens or weight rows of its
    own), a K that ends inside a block, one block only, several tiles per pair; rows of a wider matrix, in fp32."""
    torch.manual_seed(T + N)
    lw = Fn.LinearWeight.from_master(torch.randn(N, K, device=dev()) * 0.05, "fp8", dev())
    x = torch.randn(T, K, device=dev()).to(BF16)
    xq, xs = R.quant_fp8_group128_act(x)
    ref = R.dequant_fp8_group128_act(xq, xs).double() @ lw.dequant().double().t()
    assert rel_err(Fn.linear(x, lw), ref) < 3e-3          # bf16 results; the activation's codes may differ at ties
    wide = torch.full((T, N + 21), 7.0, dtype=F32, device=dev())
    Fn.linear(x, lw, out=wide[:, 8:8 + N])
    assert rel_err(wide[:, 8:8 + N], ref) < 2.5e-3
    assert bool((wide[:, :8] == 7.0).all()) and bool((wide[:, 8 + N:] == 7.0).all())
    _lib.check_status()


def test_gemm_fp8_workspace_serves_explicit_splits_only(monkeypatch):
    """By default the token tiles take these sizes and no workspace is reserved; an explicit split goes through it."""
    torch.manual_seed(3)
    asked = []
    scratch = Fn.scratch
    monkeypatch.setattr(Fn, "scratch", lambda name, *a, **k: asked.append(name) or scratch(name, *a, **k))
    for T, N, K in ((16, 2048, 4096), (40, 4096, 8192), (100, 1024, 4096)):
        lw = Fn.LinearWeight.from_master(torch.randn(N, K, device=dev()) * 0.05, "fp8", dev())
        x = torch.randn(T, K, device=dev()).to(BF16)
        xq, xs = R.quant_fp8_group128_act(x)
        ref = R.dequant_fp8_group128_act(xq, xs).double() @ lw.dequant().double().t()
        assert rel_err(Fn.linear(x, lw), ref) < 3e-3
        assert "gemm.splitk" not in asked
        ws = scratch("gemm.splitk", (4 * T * N,), F32, dev())
        ws.fill_(float("nan"))
        assert rel_err(Fn.linear(x, lw, splits=4), ref) < 3e-3
        assert "gemm.splitk" in asked and bool(ws.isfinite().all())
        asked.clear()


@pytest.mark.parametrize("T", [97, 128, 129, 255, 257, 520])
@pytest.mark.parametrize("N,K", [(16, 4096), (272, 1088), (1000, 64), (1030, 2048), (5000, 576)])
def test_gemm_bf16_wide_tiles_that_share_k(T, N, K):
    """256 x 256 tiles alone and split over two and four CTAs of a cluster: ragged edges, K of one block and of uneven parts.  Without
    workspace splits, which sizes up to 128 tokens would take by themselves."""
    torch.manual_seed(T + N)
    assert _lib.query("stk_gemm_token_tile_ctas", T, N, K, 0, _lib.sm_count()) == (4 if K >= 1024 else 2 if K >= 512 else 1)
    w = (torch.randn(N, K, device=dev()) * 0.05).to(BF16)
    x = torch.randn(T, K, device=dev()).to(BF16)
    ref = x.double() @ w.double().t()
    assert rel_err(Fn.linear(x, Fn.LinearWeight(w), splits=1), ref) < 2.5e-3
    wide = torch.full((T, N + 5), 7.0, dtype=F32, device=dev())
    Fn.linear(x, Fn.LinearWeight(w), out=wide[:, :N], splits=1)
    assert rel_err(wide[:, :N], ref) < 2e-5               # fp32 sums
    assert bool((wide[:, N:] == 7.0).all())


@pytest.mark.parametrize("T,N,K", [(64, 1030, 2048), (65, 1030, 2048), (96, 5000, 576), (600, 7500, 192), (1100, 6200, 1088), (2900, 3333, 64)])
def test_gemm_bf16_pairs_of_ctas(T, N, K):
    """Up to and from where `linear` leaves its workspace splits; pairs of CTAs with one tile and with several, a second CTA without
    tokens or weight rows, one K block; rows of a wider matrix in fp32."""
    torch.manual_seed(T + N)
    w = (torch.randn(N, K, device=dev()) * 0.05).to(BF16)
    x = torch.randn(T, K, device=dev()).to(BF16)
    ref = x.double() @ w.double().t()
    assert rel_err(Fn.linear(x, Fn.LinearWeight(w)), ref) < 2.5e-3
    wide = torch.full((T, N + 5), 7.0, dtype=F32, device=dev())
    Fn.linear(x, Fn.LinearWeight(w), out=wide[:, :N])
    assert rel_err(wide[:, :N], ref) < 2e-5               # fp32 sums
    assert bool((wide[:, N:] == 7.0).all())
    _lib.check_status()


@pytest.mark.parametrize("T", [9, 16, 17, 33, 64, 65, 128])
@pytest.mark.parametrize("N,K,groups", [(1024, 4096, 1), (1000, 2080, 1), (4096, 2048, 1), (9000, 576, 1), (1024, 1024, 8), (512, 2112, 2)])
def test_gemm_bf16_small_clusters(T, N, K, groups):
    """Two, four and eight CTAs per 128-row tile, parts of K that are uneven or empty, a last tile that is not whole, block-diagonal
    weights; every width of the token tile, results in rows of a wider matrix."""
    torch.manual_seed(T + N)
    assert _lib.query("stk_gemm_token_tile_ctas", T, N, K, 0, _lib.sm_count()) in (2, 4, 8)
    w = (torch.randn(N, K, device=dev()) * 0.05).to(BF16)
    x = torch.randn(T, K * groups, device=dev()).to(BF16)
    m = N // groups
    ref = torch.cat([x[:, g * K:(g + 1) * K].double() @ w[g * m:(g + 1) * m].double().t() for g in range(groups)], 1)
    assert rel_err(Fn.linear(x, Fn.LinearWeight(w), groups=groups), ref) < 2.5e-3
    wide = torch.full((T, N + 5), 7.0, dtype=F32, device=dev())
    Fn.linear(x, Fn.LinearWeight(w), out=wide[:, :N], groups=groups)
    assert rel_err(wide[:, :N], ref) < 2e-5               # fp32 sums
    assert bool((wide[:, N:] == 7.0).all())
    _lib.check_status()


@pytest.mark.parametrize("T", [130, 600])
@pytest.mark.parametrize("groups,n,K", [(2, 256, 128), (3, 512, 1024), (8, 128, 256)])
def test_gemm_bf16_wide_block_diagonal(T, groups, n, K):
    """Blocks of whole wide tiles (the last: blocks too narrow for them)."""
    torch.manual_seed(T)
    w = (torch.randn(groups * n, K, device=dev()) * 0.05).to(BF16)
    x = torch.randn(T, groups * K, device=dev()).to(BF16)
    ref = torch.cat([x[:, g * K:(g + 1) * K].double() @ w[g * n:(g + 1) * n].double().t() for g in range(groups)], 1)
    assert rel_err(Fn.linear(x, Fn.LinearWeight(w), groups=groups), ref) < 2.5e-3


@pytest.mark.parametrize("T,K", [(1, 128), (7, 640), (9, 512), (130, 2176)])
def test_quant_act_codes_and_scales(T, K):
    """Rows and groups that do not fill a thread block; a row of zeros, values at the ends of the range; equal to the plain
    statement up to ties of the scaled value."""
    torch.manual_seed(T)
    x = (torch.randn(T, K, device=dev()) * torch.exp(4 * torch.randn(T, 1, device=dev()))).to(BF16)
    x[T // 2] = 0
    x[0, :3] = torch.tensor([3e38, -3e38, 1e-30])
    big = torch.zeros(T, K + 64, dtype=BF16, device=dev())
    big[:, 8:8 + K] = x
    for src in (x, big[:, 8:8 + K], big[:, 4:4 + K]):        # the last: rows that 16-byte loads cannot take
        qa = Fn.quant_act(src)
        wq, ws = R.quant_fp8_group128_act(src)
        assert torch.equal(qa.scale[:, :T].t(), ws) or rel_err(qa.scale[:, :T].t(), ws) < 1e-6
        same = (qa.q.view(torch.uint8) == wq.view(torch.uint8)).float().mean()
        assert float(same) > 0.999


@pytest.mark.parametrize("H,I,E,counts", [
    (256, 128, 16, (0, 1, 15, 16, 17, 0, 31, 33)), (384, 256, 12, (127, 128, 129, 0, 300, 1)), (1024, 384, 9, (0, 0, 257, 2, 64, 65)),
    (128, 128, 2100, (3, 0, 40, 1))])
def test_moe_grouped_gemm_uneven_experts(H, I, E, counts):
    """Tiles of one row to several full ones, experts without rows between and behind them, feature counts that are no multiple of
    two weight tiles, K of a few blocks, more experts than one launch lists."""
    torch.manual_seed(14)
    chosen = torch.cat([torch.full((n,), (i * (E - 1)) // (len(counts) - 1), dtype=torch.int32) for i, n in enumerate(counts)])
    T = chosen.numel()
    ids = chosen[torch.randperm(T)][:, None].to(dev())
    w = torch.rand(T, 1, device=dev()) + 0.5
    scale = lambda *shape: (0.05 + torch.rand(*shape, device=dev())).to(torch.float8_e4m3fn).view(torch.uint8)
    code = lambda *shape: torch.randint(0, 256, shape, dtype=torch.uint8, device=dev())
    ew = M.ExpertWeights(code(E, 2 * I, H // 2), code(E, H, I // 2), scale(E, 2 * I, H // 16), scale(E, H, I // 16),
                         0.02 + 0.02 * torch.rand(E, device=dev()), 0.02 + 0.02 * torch.rand(E, device=dev()))
    x = torch.randn(T, H, device=dev()).to(BF16)
    old, M.DIRECT_MAX_PAIRS = M.DIRECT_MAX_PAIRS, 0
    try:
        out = M.moe_experts(x, ids, w, ew, 10.0, None, E)
    finally:
        M.DIRECT_MAX_PAIRS = old
    f8 = torch.float8_e4m3fn
    ref = torch.zeros(T, H, device=dev(), dtype=torch.float64)
    for e in ids.unique().tolist():
        rows = (ids[:, 0] == e).nonzero()[:, 0]
        h = x[rows].double() @ R.dequant_nvfp4(ew.w13[e], ew.s13[e].view(f8), ew.g13[e]).double().t()
        g, u = h[:, :I].clamp(max=10.0), h[:, I:].clamp(-10.0, 10.0)
        ref[rows] = (g * torch.sigmoid(g) * u) @ R.dequant_nvfp4(ew.w2[e], ew.s2[e].view(f8), ew.g2[e]).double().t() * w[rows].double()
    assert rel_err(out, ref) < 5e-3                     # activations rounded to fp16 in between, expert outputs and sums to bf16


@pytest.mark.parametrize("H,I,T,k,start,local", [(4096, 2048, 1, 6, 0, 32), (1024, 640, 8, 6, 8, 8), (160, 1056, 3, 2, 0, 16), (7168, 2112, 2, 4, 4, 5), (512, 1024, 5, 3, 16, 4)])
def test_moe_direct_pairs(H, I, T, k, start, local):
    """A handful of pairs without a sort: widths that end inside a warp's pass and of one to eight passes, outputs that the thread
    blocks do not divide, few, some or no pairs with local experts (the rest adds nothing)."""
    torch.manual_seed(H + T)
    E, f8 = 16, torch.float8_e4m3fn
    scale = lambda *shape: (0.05 + torch.rand(*shape, device=dev())).to(f8).view(torch.uint8)
    code = lambda *shape: torch.randint(0, 256, shape, dtype=torch.uint8, device=dev())
    ew = M.ExpertWeights(code(local, 2 * I, H // 2), code(local, H, I // 2), scale(local, 2 * I, H // 16), scale(local, H, I // 16),
                         0.02 + 0.02 * torch.rand(local, device=dev()), 0.02 + 0.02 * torch.rand(local, device=dev()), expert_start=start)
    x = torch.randn(T, H, device=dev()).to(BF16)
    ids = torch.stack([torch.randperm(E)[:k] for _ in range(T)]).to(torch.int32).to(dev())
    w = torch.rand(T, k, device=dev()) + 0.5
    shared = torch.randn(T, H, device=dev()).to(BF16)
    out = M.moe_experts(x, ids, w, ew, 10.0, shared, E)
    ref = shared.double()
    for t in range(T):
        for j in range(k):
            e = int(ids[t, j]) - start
            if not 0 <= e < local:
                continue
            h = x[t].double() @ R.dequant_nvfp4(ew.w13[e], ew.s13[e].view(f8), ew.g13[e]).double().t()
            g, u = h[:I].clamp(max=10.0), h[I:].clamp(-10.0, 10.0)
            ref[t] += (g * torch.sigmoid(g) * u) @ R.dequant_nvfp4(ew.w2[e], ew.s2[e].view(f8), ew.g2[e]).double().t() * w[t, j].double()
    assert rel_err(out, ref) < 6e-3                       # fp16 sums of sixteen products, activations in fp16, outputs in bf16
    _lib.check_status()


@pytest.mark.parametrize("H,I,E", [(512, 256, 6), (384, 128, 36), (128, 128, 6)])
def test_moe_grouped_gemm_scales_off_alignment(H, I, E):
    """Scales whose rows or base 16- and 4-byte copies cannot take, and K that ends inside a weight stage: the same bits as the
    aligned ones give."""
    torch.manual_seed(15)
    T = 90
    ids = torch.randint(0, E, (T, 2), dtype=torch.int32, device=dev())
    w = torch.rand(T, 2, device=dev()) + 0.5
    scale = lambda *shape: (0.05 + torch.rand(*shape, device=dev())).to(torch.float8_e4m3fn).view(torch.uint8)
    code = lambda *shape: torch.randint(0, 256, shape, dtype=torch.uint8, device=dev())
    g = torch.full((E,), 0.03, device=dev())
    w13, w2, s13, s2 = code(E, 2 * I, H // 2), code(E, H, I // 2), scale(E, 2 * I, H // 16), scale(E, H, I // 16)
    x = torch.randn(T, H, device=dev()).to(BF16)

    def moved(t, by):
        buf = torch.zeros(t.numel() + by, dtype=torch.uint8, device=dev())
        buf[by:] = t.reshape(-1)
        return buf[by:].view(t.shape)
    outs = [M.moe_experts(x, ids, w, M.ExpertWeights(w13, w2, moved(s13, by), moved(s2, by), g, g), 10.0, None, E) for by in (0, 4, 2)]
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    f8 = torch.float8_e4m3fn
    ref = torch.zeros(T, H, device=dev(), dtype=torch.float64)
    for e in range(E):
        rows, place = (ids == e).nonzero(as_tuple=True)
        h = x[rows].double() @ R.dequant_nvfp4(w13[e], s13[e].view(f8), g[e]).double().t()
        y = h[:, :I].clamp(max=10.0)
        y = y * torch.sigmoid(y) * h[:, I:].clamp(-10.0, 10.0)
        ref.index_add_(0, rows, y @ R.dequant_nvfp4(w2[e], s2[e].view(f8), g[e]).double().t() * w[rows, place].double()[:, None])
    assert rel_err(outs[0], ref) < 5e-3


@pytest.mark.parametrize("bt", [16, 128])
def test_moe_swiglu_against_64_bits(bt):
    """Rows of one value, so that gate and up products are exact whichever kernel forms them: SwiGLU of the grouped product and of a
    handful of pairs against 64 bits, down to gates whose exponential is infinite.  Tolerance: one rounding to fp16 (2^-11 of the
    value, 2^-25 where it is subnormal); in fp32 the exponential's 2 + 1.17 |g| units -- felt while the gate is above -17, below it the
    result is at most 2^-19 times the up value -- and a few of the quotient and the products: 30 x 2^-23."""
    H, I, T = 64, 1024, 960
    g = torch.Generator().manual_seed(5)
    w = torch.randint(0, 256, (1, 2 * I, H // 2), generator=g, dtype=torch.uint8).to(dev())
    s = (0.25 + 2 * torch.rand(1, 2 * I, H // 16, generator=g)).to(torch.float8_e4m3fn).view(torch.uint8).to(dev())
    gs = torch.ones(1, device=dev())
    x = torch.zeros(T, H)
    x[torch.arange(T), torch.arange(T) % H] = torch.randn(T, generator=g) * 4.0 ** (torch.arange(T) % 3).float()
    x = x.to(BF16).to(dev())
    ids = torch.zeros(T, 1, dtype=torch.int32, device=dev())
    few, grouped = (torch.empty(T + 128, I, dtype=torch.float16, device=dev()) for _ in range(2))
    for i in range(0, T, 48):
        _lib.call("stk_moe_expert_fc1", x[i:], x.stride(0), w, s, gs, None, None, None, 1, 1, few[i:], 48, H, I, 10.0, ids, 0, _lib.stream())
    rows = torch.zeros(T + 128, H, dtype=torch.float16, device=dev())
    rows[:T] = x.to(torch.float16)
    offsets = torch.tensor([0, T], dtype=torch.int32, device=dev())
    _lib.call("stk_moe_grouped", rows, T + 128, w, s, gs, offsets, 1, I, H, grouped, 1, 10.0, bt, _lib.status_buffer(), _lib.sm_count(),
              _lib.stream())
    h = x.double() @ R.dequant_nvfp4(w[0], s[0].view(torch.float8_e4m3fn), gs[0]).double().t()
    gate, up = h[:, :I].clamp(max=10.0), h[:, I:].clamp(-10.0, 10.0)
    assert float(gate.min()) < -100
    ref = gate * torch.sigmoid(gate) * up
    for out in (few[:T], grouped[:T]):
        assert float(((out.double() - ref).abs() - (2.0 ** -11 + 30 * 2.0 ** -23) * ref.abs()).max()) <= 2.0 ** -24


@pytest.mark.parametrize("I", [384, 640, 448])
@pytest.mark.parametrize("rows", [5, 40, 130])
def test_moe_grouped_gemm_steps_of_one_weight_tile(I, rows):
    """Single weight tiles (features no multiple of 256) with six, ten and seven K steps of 64, more tiles than thread blocks: operand
    places are taken in turn across tiles whose last stage is not whole."""
    H, E = 384, 64
    g = torch.Generator().manual_seed(I + rows)
    P = E * rows
    w = torch.randint(0, 256, (E, H, I // 2), generator=g, dtype=torch.uint8).to(dev())
    s = (0.05 + torch.rand(E, H, I // 16, generator=g)).to(torch.float8_e4m3fn).view(torch.uint8).to(dev())
    gs = torch.full((E,), 0.03, device=dev())
    x = torch.zeros(P + 128, I, dtype=torch.float16)
    x[:P] = torch.randn(P, I, generator=g)
    x = x.to(dev())
    offsets = (torch.arange(E + 1, dtype=torch.int32) * rows).to(dev())
    out = torch.empty(P, H, dtype=BF16, device=dev())
    _lib.call("stk_moe_grouped", x, P + 128, w, s, gs, offsets, E, H, I, out, 0, 0.0, 16 if rows < 16 else 64 if rows < 100 else 128,
              _lib.status_buffer(), _lib.sm_count(), _lib.stream())
    deq = torch.stack([R.dequant_nvfp4(w[e], s[e].view(torch.float8_e4m3fn), gs[e]) for e in range(E)]).double()
    ref = torch.bmm(x[:P].double().view(E, rows, I), deq.transpose(1, 2)).view(P, H)
    assert rel_err(out, ref) < 2.5e-3                     # rounded to bf16 once: 1.7e-3
    _lib.check_status()


@pytest.mark.parametrize("bt", [16, 64, 128])
def test_moe_grouped_gemm_of_rows_that_have_arrived(bt):
    """The expert-parallel first product with every row in place and every count at (or past) its expert's: the same bits as without."""
    H, I, E = 320, 256, 9
    g = torch.Generator().manual_seed(bt)
    counts = torch.tensor([3, 0, 70, 1, 0, 129, 16, 17, 0], dtype=torch.int32)
    offsets = torch.cat([torch.zeros(1, dtype=torch.int32), counts.cumsum(0).to(torch.int32)]).to(dev())
    P = int(counts.sum())
    w = torch.randint(0, 256, (E, 2 * I, H // 2), generator=g, dtype=torch.uint8).to(dev())
    s = (0.05 + torch.rand(E, 2 * I, H // 16, generator=g)).to(torch.float8_e4m3fn).view(torch.uint8).to(dev())
    gs = torch.full((E,), 0.03, device=dev())
    x = torch.zeros(P + 128, H, dtype=torch.float16)
    x[:P] = torch.randn(P, H, generator=g)
    x = x.to(dev())
    plain, ep = (torch.full((P + 128, I), 7.0, dtype=torch.float16, device=dev()) for _ in range(2))
    arrived = (counts + torch.tensor([0, 5, 0, 0, 0, 0, 1, 0, 0], dtype=torch.int32)).to(dev())
    _lib.call("stk_moe_grouped", x, P + 128, w, s, gs, offsets, E, I, H, plain, 1, 10.0, bt, _lib.status_buffer(), _lib.sm_count(), _lib.stream())
    _lib.call("stk_moe_grouped_ep", x, P + 128, w, s, gs, offsets, E, I, H, ep, 1, 10.0, bt, _lib.status_buffer(), _lib.sm_count(), arrived,
              1000, _lib.stream())
    assert torch.equal(plain.view(torch.int16), ep.view(torch.int16)) and bool((plain[P:] == 7.0).all())
    _lib.check_status()


@pytest.mark.parametrize("H,I", [(8704, 128), (128, 8704)])
def test_moe_experts_of_a_handful_of_pairs_beyond_8192(H, I):
    """Widths that the thread blocks that stay do not take: a thread block per part of a pair's rows, without a sort."""
    torch.manual_seed(15)
    E, T, k = 3, 5, 2
    assert _lib.query("stk_moe_direct_blocks", T * k, max(H, I), _lib.sm_count()) == 0
    ew = M.ExpertWeights.from_master(torch.randn(E, 2 * I, H, device=dev()) * 0.02, torch.randn(E, H, I, device=dev()) * 0.02, "nvfp4", dev())
    x = torch.randn(T, H, device=dev()).to(BF16)
    ids, w = M.router(torch.randn(T, E, device=dev()), None, k, "sigmoid", True, 1.0)
    d13, d2 = ew.dequant()
    assert rel_err(M.moe_experts(x, ids, w, ew, 10.0), R.moe_experts(x, ids, w, d13, d2, 10.0)) < 1.5e-2
    hi = M.ExpertWeights(ew.w13[1:], ew.w2[1:], ew.s13[1:], ew.s2[1:], ew.g13[1:], ew.g2[1:], 1)         # the first belongs to another rank
    assert rel_err(M.moe_experts(x, ids, w, hi, 10.0), R.moe_experts(x, ids, w, d13[1:], d2[1:], 10.0, 1)) < 1.5e-2


def test_topk_candidates_and_markov_chain_match_cpu():
    """The drafter's sampling path: two-level candidate selection over the full vocabulary and the one-launch
    sequential Markov sampling against their CPU statements."""
    torch.manual_seed(21)
    B, N, V, Rk, K = 3, 5, 129280, 256, 512
    base = (torch.randn(B * N, V, device=dev()) * 3).to(BF16)
    ci, cv = S.topk_candidates(base, K)
    ri, rv = S.topk_candidates(base.cpu(), K)
    assert ci.shape == (B * N, K) and int(ci.min()) >= 0 and int(ci.max()) < V
    # same value multiset (ties at the threshold may pick different ids of equal value)
    assert torch.equal(cv.sort(-1).values.cpu(), rv.sort(-1).values)
    assert torch.equal(base.float().gather(1, ci.long()), cv)
    w1 = (torch.randn(V, Rk, device=dev()) * 0.3).to(BF16)
    w2 = (torch.randn(V, Rk, device=dev()) * 0.3).to(BF16)
    anchors = torch.randint(0, V, (B,), device=dev())
    temp = torch.tensor([0.6, 0.0, 1.0], device=dev())
    seed = torch.tensor([11, 2 ** 41 + 5, 3], device=dev(), dtype=torch.int64)
    pos = torch.tensor([100, 32768, 7], device=dev(), dtype=torch.int64)
    got = S.markov_chain(ci.view(B, N, K), cv.view(B, N, K), anchors, w1, w2, temp, seed, pos)
    ref = S.markov_chain(ci.view(B, N, K).cpu(), cv.view(B, N, K).cpu(), anchors.cpu(), w1.cpu(), w2.cpu(), temp.cpu(),
                         seed.cpu(), pos.cpu())
    assert got.shape == (B, N)
    assert torch.equal(got[:, 0].cpu(), ref[:, 0])                       # first position: same inputs on both sides
    assert (got.cpu() == ref).float().mean().item() >= 0.8              # later ones depend on earlier draws
    # every drawn token is one of its position's candidates
    for b in range(B):
        for i in range(N):
            assert int(got[b, i]) in set(ci.view(B, N, K)[b, i].tolist())
