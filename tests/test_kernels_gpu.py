"""Numerics of every sm_100a kernel against the fp32 PyTorch statements in ops/reference.py."""
import math
import os
import subprocess
import sys

import pytest
import torch

from cosmos_rl_b200.ops import functional as F
from cosmos_rl_b200.ops import native, reference as R

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _bf16(*shape, scale=1.0):
    return (torch.randn(*shape, device=DEV) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (300, 1000, 520), (1024, 3584, 3584),
                                   (77, 128, 64), (4096, 152, 1024)])
def test_gemm_bf16_nt(M, N, K):
    torch.manual_seed(0)
    a, b = _bf16(M, K), _bf16(N, K)
    c = F.gemm_nt(a, b)
    native.read_status(a.device)
    ref = a.float() @ b.float().t()
    err = (c.float() - ref).abs().max().item()
    tol = 2e-2 * math.sqrt(K) + 1e-2 * ref.abs().max().item()
    assert err < tol, (err, tol)
    # tight check against a bf16-rounded fp32 result
    assert torch.allclose(c.float(), ref.to(torch.bfloat16).float(), rtol=2e-2, atol=1e-2 * math.sqrt(K))


def test_gemm_fp32_accumulate():
    torch.manual_seed(1)
    a, b = _bf16(256, 512), _bf16(384, 512)
    out = torch.ones(256, 384, dtype=torch.float32, device=DEV)
    F.gemm_nt(a, b, out=out, accumulate=True)
    native.read_status(a.device)
    ref = a.float() @ b.float().t() + 1.0
    assert torch.allclose(out, ref, rtol=1e-3, atol=1e-2)


@pytest.mark.parametrize("T,V,H,temp", [(100, 1000, 128, 1.0), (257, 5000, 256, 0.7), (1024, 32000, 512, 1.0)])
def test_fused_logprob_fwd_bwd(T, V, H, temp):
    torch.manual_seed(2)
    h = _bf16(T, H).requires_grad_(True)
    w = _bf16(V, H, scale=0.05).requires_grad_(True)
    labels = torch.randint(0, V, (T,), device=DEV)
    labels[::7] = -100
    lp, ent = F.fused_logprob(h, w, labels, temp)
    native.read_status(h.device)
    hr = h.detach().float().requires_grad_(True)
    wr = w.detach().float().requires_grad_(True)
    lpr, entr = R.logprob_entropy(hr, wr, labels, temp)
    assert torch.allclose(lp, lpr, rtol=1e-3, atol=2e-3), (lp - lpr).abs().max()
    assert torch.allclose(ent, entr, rtol=1e-3, atol=2e-3), (ent - entr).abs().max()
    g1 = torch.randn(T, device=DEV)
    g2 = torch.randn(T, device=DEV) * 0.1
    (lp * g1 + ent * g2).sum().backward()
    native.read_status(h.device)
    (lpr * g1 + entr * g2).sum().backward()
    assert torch.allclose(h.grad.float(), hr.grad, rtol=5e-2, atol=5e-2 * hr.grad.abs().max().item())
    assert torch.allclose(w.grad.float(), wr.grad, rtol=5e-2, atol=5e-2 * wr.grad.abs().max().item())


@pytest.mark.parametrize("T,V,H", [(128, 520, 64), (129, 264, 64), (255, 1000, 72), (385, 8, 128)])
def test_logit_gradient_tiles(T, V, H):
    torch.manual_seed(61)
    h, w = _bf16(T, H).requires_grad_(True), _bf16(V, H, scale=0.1).requires_grad_(True)
    labels = torch.randint(0, V, (T,), device=DEV)
    labels[::5] = -100
    g1, g2 = torch.randn(T, device=DEV), torch.randn(T, device=DEV)
    lp, ent = F.fused_logprob(h, w, labels, 0.9)
    (lp * g1 + ent * g2).sum().backward()
    native.read_status(h.device)
    hr, wr = h.detach().double(), w.detach().double()
    logits = (hr @ wr.t() / 0.9).requires_grad_(True)
    lsm = torch.log_softmax(logits, -1)
    picked = torch.where(labels >= 0, lsm.gather(1, labels.clamp_min(0)[:, None])[:, 0], 0.0)
    (picked * g1 - (lsm.exp() * lsm).sum(-1) * g2).sum().backward()
    d = logits.grad / 0.9   # kept as bf16: each entry is off by 2^-9 of itself, as is the result; fp32 sums: the floor
    for grad, ref, size in ((h.grad, d @ wr, d.abs() @ wr.abs()), (w.grad, d.t() @ hr, d.abs().t() @ hr.abs())):
        assert ((grad.double() - ref).abs() <= 2.0 ** -8 * (size + ref.abs()) + 1e-5).all()


@pytest.mark.parametrize("R_,C,off", [(1, 128, 0), (3, 200, 0), (17, 1032, 0), (5, 130, 1), (65, 4096, 0)])
def test_quant_fp8_rows_match_reference_bit_for_bit(R_, C, off):
    """Ragged last blocks, and rows that start off the 16-byte grid."""
    torch.manual_seed(37)
    w = _bf16(R_, C + off + 7)[:, off:off + C]
    q, s = F.quant_fp8_block(w, 1)
    nb = (C + 127) // 128
    pad = torch.zeros(R_, nb * 128, device=DEV)
    pad[:, :C] = w.float()
    scale = pad.view(R_, nb, 128).abs().amax(-1).clamp_min(1e-12) / torch.tensor(448.0, device=DEV)
    assert torch.equal(s, scale)
    want = (pad.view(R_, nb, 128) * (1.0 / scale)[:, :, None]).view(R_, -1)[:, :C].to(torch.float8_e4m3fn)
    assert torch.equal(q.view(torch.uint8), want.view(torch.uint8))


@pytest.mark.parametrize("T,H", [(33, 256), (1000, 3584), (64, 8192)])
@pytest.mark.parametrize("with_res", [False, True])
def test_rmsnorm(T, H, with_res):
    torch.manual_seed(3)
    x = _bf16(T, H).requires_grad_(True)
    w = (1 + 0.1 * torch.randn(H, device=DEV)).to(torch.bfloat16).requires_grad_(True)
    res = _bf16(T, H).requires_grad_(True) if with_res else None
    y, ro = F.rms_norm(x, w, 1e-6, res)
    xr = x.detach().float().requires_grad_(True)
    wr = w.detach().float().requires_grad_(True)
    rr = res.detach().float().requires_grad_(True) if with_res else None
    h = (xr + rr).to(torch.bfloat16).float() if with_res else xr
    if with_res:
        # straight-through for the bf16 rounding of the residual stream
        h = (xr + rr) + (h - (xr + rr)).detach()
    yr = h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-6) * wr
    assert torch.allclose(y.float(), yr, rtol=2e-2, atol=2e-2)
    gy = torch.randn_like(yr)
    loss = (y.float() * gy).sum()
    lossr = (yr * gy).sum()
    if with_res:
        gr = torch.randn_like(yr)
        loss = loss + (ro.float() * gr).sum()
        lossr = lossr + (h * gr).sum()
    loss.backward()
    lossr.backward()
    assert torch.allclose(x.grad.float(), xr.grad, rtol=3e-2, atol=3e-2)
    assert torch.allclose(w.grad.float(), wr.grad, rtol=3e-2, atol=3e-2 * wr.grad.abs().max().item())
    if with_res:
        assert torch.allclose(res.grad.float(), rr.grad, rtol=3e-2, atol=3e-2)


def test_rope_qkv_fwd_bwd():
    torch.manual_seed(4)
    T, hq, hkv, d = 50, 4, 2, 128
    base = _bf16(T, (hq + 2 * hkv) * d)
    pos = torch.randint(0, 4000, (T,), device=DEV)
    a = base.clone().requires_grad_(True)
    out = F.rope_qkv_(a * 1.0, pos, hq, hkv, d, 1e6)
    b = base.detach().cpu().float().requires_grad_(True)
    outr = F.rope_qkv_(b, pos.cpu(), hq, hkv, d, 1e6)
    assert torch.allclose(out.float().cpu(), outr, rtol=2e-2, atol=2e-2)
    g = torch.randn_like(outr)
    (out.float() * g.to(DEV)).sum().backward()
    (outr * g).sum().backward()
    assert torch.allclose(a.grad.float().cpu(), b.grad, rtol=2e-2, atol=2e-2)


def test_swiglu():
    torch.manual_seed(5)
    gu = _bf16(300, 2 * 1024).requires_grad_(True)
    y = F.swiglu(gu)
    gr = gu.detach().float().requires_grad_(True)
    yr = R.swiglu(gr)
    assert torch.allclose(y.float(), yr, rtol=2e-2, atol=2e-2)
    g = torch.randn_like(yr)
    (y.float() * g).sum().backward()
    (yr * g).sum().backward()
    assert torch.allclose(gu.grad.float(), gr.grad, rtol=3e-2, atol=3e-2)


def test_adamw_and_clip():
    from cosmos_rl_b200.ops import optim
    torch.manual_seed(6)
    n = 100003
    master = torch.randn(n, device=DEV)
    m = torch.zeros(n, device=DEV)
    v = torch.zeros(n, device=DEV)
    shadow = master.to(torch.bfloat16)
    mr, mm, vv = master.clone(), m.clone(), v.clone()
    for step in range(1, 4):
        grad = (torch.randn(n, device=DEV) * 0.1).to(torch.bfloat16)
        norm, coef = optim.grad_norm_and_clip([grad], 1.0)
        ref_norm = grad.float().norm()
        assert abs(norm.item() - ref_norm.item()) < 1e-2 * ref_norm.item()
        optim.adamw_flat(master, m, v, grad, shadow, lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=0.01,
                         step=step, grad_scale=coef)
        R.adamw_step(mr, mm, vv, grad, 1e-3, 0.9, 0.999, 1e-8, 0.01, step, grad_scale=min(1.0, 1.0 / (ref_norm.item() + 1e-6)))
    assert torch.allclose(master, mr, rtol=1e-4, atol=1e-5)
    assert torch.allclose(shadow.float(), mr.to(torch.bfloat16).float(), rtol=1e-2, atol=1e-2)


def test_sampling_distribution_and_logprob():
    torch.manual_seed(7)
    B, V = 64, 1000
    logits = torch.randn(1, V, device=DEV).repeat(B, 1) * 2
    temp = torch.full((B,), 0.8, device=DEV)
    counts = torch.zeros(V, device=DEV)
    n_rounds = 200
    for i in range(n_rounds):
        toks, lps = F.sample(logits, temp, None, None, seed=123, offset=i)
        counts.index_add_(0, toks, torch.ones(B, device=DEV))
    p = torch.softmax(logits[0] / 0.8, -1)
    emp = counts / counts.sum()
    assert (emp - p).abs().sum().item() < 0.15  # total variation small with 12800 draws
    lsm = torch.log_softmax(logits[0] / 0.8, -1)
    assert torch.allclose(lps, lsm[toks], rtol=1e-4, atol=1e-4)
    # greedy
    toks, _ = F.sample(logits, torch.zeros(B, device=DEV), None, None, seed=1, offset=0)
    assert (toks == logits[0].argmax()).all()
    # top-k / top-p restrict the support
    topk = torch.full((B,), 5, dtype=torch.int32, device=DEV)
    allowed = set(torch.topk(logits[0], 5).indices.tolist())
    for i in range(20):
        toks, _ = F.sample(logits, temp, None, topk, seed=5, offset=i)
        assert set(toks.tolist()) <= allowed
    topp = torch.full((B,), 0.5, device=DEV)
    sp, si = torch.sort(p, descending=True)
    ncut = int((sp.cumsum(0) < 0.5).sum()) + 1
    allowed = set(si[:ncut + 1].tolist())
    for i in range(20):
        toks, _ = F.sample(logits, temp, topp, None, seed=9, offset=i)
        assert set(toks.tolist()) <= allowed


@pytest.mark.parametrize("hq,hkv,d", [(28, 4, 128), (8, 8, 128), (16, 2, 64)])
def test_paged_decode_and_append(hq, hkv, d):
    torch.manual_seed(8)
    B, page_size, n_pages = 5, 16, 64
    cache = torch.zeros(n_pages, 2, hkv, page_size, d, dtype=torch.bfloat16, device=DEV)
    seq_lens = torch.tensor([1, 17, 100, 160, 33], dtype=torch.int32, device=DEV)
    max_pages = 12
    perm = torch.randperm(n_pages, device=DEV)[: B * max_pages].view(B, max_pages).to(torch.int32)
    # append all tokens through the kernel
    ks, vs, slots = [], [], []
    for b in range(B):
        L = int(seq_lens[b])
        ks.append(_bf16(L, hkv, d))
        vs.append(_bf16(L, hkv, d))
        t = torch.arange(L, device=DEV)
        slots.append(perm[b, t // page_size].long() * page_size + t % page_size)
    k, v, slot = torch.cat(ks), torch.cat(vs), torch.cat(slots).to(torch.int32)
    F.kv_append(k, v, cache, slot)
    cache_ref = torch.zeros_like(cache).cpu()
    R.kv_append(k.cpu(), v.cpu(), cache_ref, slot.cpu())
    assert torch.equal(cache.cpu(), cache_ref)
    q = _bf16(B, hq, d)
    ref = R.paged_decode(q.cpu(), cache_ref, perm.cpu(), seq_lens.cpu())
    for nsplit in (1, 4):
        out = F.paged_decode(q, cache, perm, seq_lens, nsplit=nsplit)
        assert torch.allclose(out.float().cpu(), ref.float(), rtol=2e-2, atol=2e-2), nsplit


@pytest.mark.parametrize("R_,C", [(256, 384), (300, 200), (128, 128)])
def test_quant_fp8(R_, C):
    torch.manual_seed(9)
    w = _bf16(R_, C)
    q, s = F.quant_fp8_block(w, 128)
    qr, sr = R.quant_fp8_block(w.cpu(), 128, 128)
    assert torch.allclose(s.cpu(), sr, rtol=1e-5)
    deq = R.dequant_fp8_block(q.cpu(), s.cpu())
    assert (deq - w.cpu().float()).abs().max() <= 0.07 * w.abs().max().item()
    assert (q.cpu().float() - qr.float()).abs().max() <= 32  # at most one e4m3 ulp at the top binade
    qa, sa = F.quant_fp8_block(w, 1)
    deqa = R.dequant_fp8_block(qa.cpu(), sa.cpu(), 1, 128)
    assert (deqa - w.cpu().float()).abs().max() <= 0.07 * w.abs().max().item()


@pytest.mark.parametrize("hq,hkv", [(28, 4), (8, 8), (64, 8), (4, 4)])
def test_paged_decode_tensor_core(hq, hkv):
    """tcgen05 decode kernel (V stored transposed, 128-token pages) against the fp32 statement."""
    torch.manual_seed(10)
    d, P, B, n_pages, max_pages = 128, 128, 7, 64, 6
    cache = torch.zeros(n_pages, 2, hkv, P, d, dtype=torch.bfloat16, device=DEV)
    seq_lens = torch.tensor([1, 127, 128, 129, 500, 768, 300], dtype=torch.int32, device=DEV)
    perm = torch.stack([torch.randperm(n_pages - 1, device=DEV)[:max_pages] + 1 for _ in range(B)]).to(torch.int32)
    ks, vs, slots = [], [], []
    for b in range(B):
        L = int(seq_lens[b])
        ks.append(_bf16(L, hkv, d))
        vs.append(_bf16(L, hkv, d))
        t = torch.arange(L, device=DEV)
        slots.append(perm[b, t // P].long() * P + t % P)
    k, v, slot = torch.cat(ks), torch.cat(vs), torch.cat(slots).to(torch.int32)
    F.kv_append(k, v, cache, slot, v_transposed=True)
    cache_ref = torch.zeros_like(cache).cpu()
    R.kv_append(k.cpu(), v.cpu(), cache_ref, slot.cpu(), v_transposed=True)
    assert torch.equal(cache.cpu(), cache_ref)
    q = _bf16(B, hq, d)
    ref = R.paged_decode(q.cpu(), cache_ref, perm.cpu(), seq_lens.cpu(), v_transposed=True)
    for nsplit in (1, 3):
        out = F.paged_decode(q, cache, perm, seq_lens, nsplit=nsplit, v_transposed=True)
        native.read_status(q.device)
        err = (out.float().cpu() - ref.float()).abs().max().item()
        assert err < 3e-2, (nsplit, err)


@pytest.mark.parametrize("a_mn,b_mn", [(False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K", [(256, 512, 384), (300, 200, 520), (1024, 3584, 2048)])
def test_gemm_operand_layouts(a_mn, b_mn, M, N, K):
    """dgrad (B stored [K, N]) and wgrad (both stored [K, *]) forms against fp32 matmul."""
    torch.manual_seed(11)
    K8 = K
    a = _bf16(K8, (M + 7) // 8 * 8)[:, :M] if a_mn else _bf16(M, K8)
    b = _bf16(K8, (N + 7) // 8 * 8)[:, :N] if b_mn else _bf16(N, K8)
    out = F.gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    native.read_status(a.device)
    af = a.float().t() if a_mn else a.float()
    bf_ = b.float().t() if b_mn else b.float()
    ref = af @ bf_.t()
    assert torch.allclose(out.float(), ref, rtol=2e-2, atol=1e-2 * math.sqrt(K)), (out.float() - ref).abs().max()


def test_linear_tc_matches_torch_linear():
    torch.manual_seed(12)
    x = _bf16(512, 1024).requires_grad_(True)
    w = _bf16(768, 1024, scale=0.05).requires_grad_(True)
    b = _bf16(768).requires_grad_(True)
    y = F.linear_tc(x, w, b)
    native.read_status(x.device)
    g = _bf16(512, 768)
    y.backward(g)
    native.read_status(x.device)
    xr, wr, br = (t.detach().float().requires_grad_(True) for t in (x, w, b))
    yr = torch.nn.functional.linear(xr, wr, br)
    yr.backward(g.float())
    assert torch.allclose(y.float(), yr, rtol=2e-2, atol=0.3)
    assert torch.allclose(x.grad.float(), xr.grad, rtol=2e-2, atol=0.3)
    assert torch.allclose(w.grad.float(), wr.grad, rtol=2e-2, atol=0.5)
    # second backward accumulates into the existing .grad inside the GEMM epilogue
    y2 = F.linear_tc(x.detach(), w, None)
    y2.backward(g)
    assert torch.allclose(w.grad.float(), 2 * wr.grad, rtol=3e-2, atol=1.0)


def test_moe_router_topk():
    from cosmos_rl_b200.ops import moe
    torch.manual_seed(13)
    T, E, k = 777, 128, 8
    logits = torch.randn(T, E, device=DEV) * 2
    counts = torch.zeros(E, dtype=torch.int32, device=DEV)
    p, i = moe.route_topk(logits, k, True, counts)
    pr, ir = moe.route_topk_reference(logits, k, True)
    assert torch.equal(i.long().sort(-1).values, ir.long().sort(-1).values)
    assert torch.allclose(p.sort(-1).values, pr.sort(-1).values, rtol=1e-4, atol=1e-6)
    assert torch.equal(counts.long(), torch.bincount(ir.flatten().long(), minlength=E))


@pytest.mark.parametrize("T,H,I,E,k", [(300, 256, 128, 8, 2), (1024, 2048, 768, 16, 8), (64, 512, 256, 32, 4)])
def test_moe_experts_fwd_bwd(T, H, I, E, k):
    from cosmos_rl_b200.ops import moe
    torch.manual_seed(14)
    x = _bf16(T, H).requires_grad_(True)
    wgu = _bf16(E, 2 * I, H, scale=0.05).requires_grad_(True)
    wd = _bf16(E, H, I, scale=0.05).requires_grad_(True)
    logits = torch.randn(T, E, device=DEV)
    probs, idx = moe.route_topk(logits, k, True)
    probs = probs.clone().requires_grad_(True)
    out = moe.moe_experts(x, probs, idx, wgu, wd)
    native.read_status(x.device)
    xr, pr, wgur, wdr = (t.detach().float().requires_grad_(True) for t in (x, probs, wgu, wd))
    ref = moe.moe_experts_reference(xr, pr, idx, wgur, wdr)
    scale = ref.abs().max().item()
    assert torch.allclose(out.float(), ref, rtol=3e-2, atol=3e-2 * scale), (out.float() - ref).abs().max()
    g = _bf16(T, H)
    out.backward(g)
    native.read_status(x.device)
    ref.backward(g.float())
    for name, a, b in (("dx", x.grad, xr.grad), ("dprob", probs.grad, pr.grad), ("dwgu", wgu.grad, wgur.grad),
                       ("dwd", wd.grad, wdr.grad)):
        s = b.abs().max().item()
        assert torch.allclose(a.float(), b, rtol=5e-2, atol=5e-2 * s), (name, (a.float() - b).abs().max().item(), s)


def test_rope_separate_qk_autograd_on_views():
    """q / k that are views of another tensor (the per-head-norm path of Qwen3) must work under autograd."""
    torch.manual_seed(15)
    T, hq, hkv, d = 40, 4, 2, 128
    qb = _bf16(T * hq, d).requires_grad_(True)
    kb = _bf16(T * hkv, d).requires_grad_(True)
    pos = torch.randint(0, 3000, (T,), device=DEV)
    q, k = F.apply_rope((qb * 1.0).view(T, hq, d), (kb * 1.0).view(T, hkv, d), pos, 1e6)
    qr = qb.detach().float().cpu().requires_grad_(True)
    kr = kb.detach().float().cpu().requires_grad_(True)
    qe, ke = R.apply_rope(qr.view(T, hq, d), kr.view(T, hkv, d), pos.cpu(), 1e6)
    assert torch.allclose(q.float().cpu(), qe, rtol=2e-2, atol=2e-2)
    (q.float().sum() + 2 * k.float().sum()).backward()
    (qe.sum() + 2 * ke.sum()).backward()
    assert torch.allclose(qb.grad.float().cpu(), qr.grad, rtol=2e-2, atol=2e-2)
    assert torch.allclose(kb.grad.float().cpu(), kr.grad, rtol=2e-2, atol=2e-2)


@pytest.mark.gpu
# more items than SMs, listed by length: the most sequences that are sorted and one more, equal and empty ones among them
@pytest.mark.parametrize("B,hq,hkv,nsplit", [(256, 7, 1, 1), (257, 4, 2, 1), (75, 8, 4, 2), (149, 2, 1, 1)])
def test_paged_decode_many_uneven_sequences(B, hq, hkv, nsplit):
    torch.manual_seed(B)
    lens = torch.randint(1, 500, (B,), dtype=torch.int32)
    lens[::9], lens[1::9], lens[B // 2] = 129, 128, 0
    lens[-1] = 1100
    per = (lens + 127) // 128
    pages, width = int(per.sum()) + 1, int(per.max()) + 1
    table = torch.zeros(B, width, dtype=torch.int32)
    order = torch.randperm(pages - 1).int() + 1
    at = 0
    for b in range(B):
        table[b, :per[b]] = order[at:at + per[b]]
        at += int(per[b])
    cache = torch.randn(pages, 2, hkv, 128, 128).to(torch.bfloat16).cuda()
    q = torch.randn(B, hq, 128).to(torch.bfloat16).cuda()
    out = F.paged_decode(q, cache, table.cuda(), lens.cuda(), nsplit=nsplit, v_transposed=True)
    torch.cuda.synchronize()
    assert native.read_status(q.device) == 0
    some = lens.nonzero().flatten()
    ref = R.paged_decode(q.cpu()[some], cache.cpu(), table[some], lens[some], v_transposed=True)
    # probabilities and the result are rounded to bf16 (2^-9 each)
    assert (out.cpu()[some].float() - ref.float()).norm() <= 2.0 ** -7 * ref.float().norm()
    assert (out.cpu()[some].float() - ref.float()).abs().max() <= 2.0 ** -6 * ref.float().abs().max()
    assert (out.cpu()[lens == 0] == 0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("over", [
    {}, {"kl_beta": 0.05}, {"kl_beta": 0.05, "unbiased_kl_estimate": True}, {"aipo_rho": 1.1},
    {"use_decoupled_loss": True, "behav_imp_weight_cap": 1.3, "kl_beta": 0.01},
    {"loss_type": "seq-mean-token-mean", "off_policy_masking_delta": 0.05},
    {"loss_type": "seq-mean-token-sum", "epsilon_high": 0.28, "lower_bound_ratio": 1.2},
])
def test_fused_grpo_loss_matches_op_by_op(over):
    from cosmos_rl_b200.policy import loss as L
    torch.manual_seed(3)
    n, n_seq = 5000, 37
    dev = torch.device("cuda")
    base = torch.randn(n, device=dev) - 2.0
    old = base + 0.25 * torch.randn(n, device=dev)
    old[::17] = base[::17]                               # exact ties: ratio == 1
    old[5] = base[5] + 30.0                              # clamp region
    ref = base + 0.1 * torch.randn(n, device=dev)
    roll = old + 0.2 * torch.randn(n, device=dev)
    seq_ids = torch.sort(torch.randint(0, n_seq, (n,), device=dev)).values
    A = torch.randn(n_seq, device=dev)[seq_ids]
    ent = torch.rand(n, device=dev)
    cfg = L.GrpoLossConfig(**over)
    res = {}
    for fused in (False, True):
        L.USE_FUSED_KERNEL = fused
        lp = base.clone().requires_grad_(True)
        loss, m = L.grpo_loss(lp, old, A, seq_ids, n_seq, cfg, ref_logprob=ref, rollout_logprob=roll, entropy=ent)
        loss.backward()
        res[fused] = (loss.detach(), lp.grad.clone(), {k: v.detach() for k, v in m.items()})
    L.USE_FUSED_KERNEL = True
    (l0, g0, m0), (l1, g1, m1) = res[False], res[True]
    assert torch.allclose(l0, l1, rtol=1e-4, atol=1e-6), (l0, l1)
    assert torch.allclose(g0, g1, rtol=1e-4, atol=1e-8), (g0 - g1).abs().max()
    for k in m0:
        assert torch.allclose(m0[k].float(), m1[k].float(), rtol=1e-4, atol=1e-6), k


@pytest.mark.gpu
@pytest.mark.parametrize("lens,hq,hkv", [([128], 2, 1), ([300, 17, 129, 1000], 4, 2), ([2048, 512], 28, 4),
                                         ([1, 1, 5], 8, 8)])
def test_flash_attention_forward_and_lse(lens, hq, hkv):
    from cosmos_rl_b200.ops import attention
    torch.manual_seed(11)
    d, T = 128, sum(lens)
    qkv = torch.randn(T, (hq + 2 * hkv) * d, device="cuda").to(torch.bfloat16)
    q, k, v = qkv.split([hq * d, hkv * d, hkv * d], dim=-1)         # strided views, as the model passes them
    q, k, v = q.unflatten(-1, (hq, d)), k.unflatten(-1, (hkv, d)), v.unflatten(-1, (hkv, d))
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device="cuda")
    scale = 1.0 / math.sqrt(d)
    out, lse = attention.flash_fwd(q, k, v, cu, cu, max(lens), scale)
    torch.cuda.synchronize()
    assert native.read_status(q.device) == 0
    ref = R.varlen_attention(q.float(), k.float(), v.float(), cu, scale)
    assert torch.allclose(out.float(), ref, atol=2e-2, rtol=2e-2), (out.float() - ref).abs().max()
    # log-sum-exp of the scaled scores per (head, token)
    g = hq // hkv
    for b in range(len(lens)):
        s0, s1 = int(cu[b]), int(cu[b + 1])
        qs, ks = q[s0:s1].float(), k[s0:s1].float().repeat_interleave(g, dim=1)
        sc = torch.einsum("qhd,khd->hqk", qs, ks) * scale
        sc = sc.masked_fill(torch.ones(s1 - s0, s1 - s0, device="cuda").triu(1).bool(), float("-inf"))
        assert torch.allclose(lse[:, s0:s1], torch.logsumexp(sc, -1), atol=2e-2, rtol=1e-3)


@pytest.mark.gpu
def test_flash_attention_prefix_aligned_queries():
    """Queries aligned to the end of a longer key sequence (prefill on top of cached keys, CP chunks)."""
    from cosmos_rl_b200.ops import attention
    torch.manual_seed(12)
    d, hq, hkv = 128, 4, 2
    lq, lk = [100, 256], [356, 300]
    q = torch.randn(sum(lq), hq, d, device="cuda").to(torch.bfloat16)
    k = torch.randn(sum(lk), hkv, d, device="cuda").to(torch.bfloat16)
    v = torch.randn(sum(lk), hkv, d, device="cuda").to(torch.bfloat16)
    cq = torch.tensor([0, 100, 356], dtype=torch.int32, device="cuda")
    ck = torch.tensor([0, 356, 656], dtype=torch.int32, device="cuda")
    scale = 1.0 / math.sqrt(d)
    out, _ = attention.flash_fwd(q, k, v, cq, ck, 256, scale)
    assert native.read_status(q.device) == 0
    for b in range(2):
        qs = q[int(cq[b]):int(cq[b + 1])].float()
        ks = k[int(ck[b]):int(ck[b + 1])].float().repeat_interleave(2, dim=1)
        vs = v[int(ck[b]):int(ck[b + 1])].float().repeat_interleave(2, dim=1)
        sc = torch.einsum("qhd,khd->hqk", qs, ks) * scale
        nq, nk = qs.shape[0], ks.shape[0]
        mask = torch.arange(nk, device="cuda")[None, :] > (torch.arange(nq, device="cuda")[:, None] + nk - nq)
        ref = torch.einsum("hqk,khd->qhd", torch.softmax(sc.masked_fill(mask, float("-inf")), -1), vs)
        got = out[int(cq[b]):int(cq[b + 1])].float()
        assert torch.allclose(got, ref, atol=2e-2, rtol=2e-2), (got - ref).abs().max()


@pytest.mark.gpu
@pytest.mark.parametrize("lens,hq,hkv", [([200, 56], 4, 2), ([128], 1, 1), ([300, 17, 129, 700], 14, 2),
                                         ([1, 5, 1500], 8, 8)])
def test_flash_attention_autograd_matches_reference(lens, hq, hkv):
    torch.manual_seed(13)
    d, T = 128, sum(lens)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device="cuda")
    qkv = torch.randn(T, (hq + 2 * hkv) * d, device="cuda").to(torch.bfloat16).requires_grad_(True)
    q, k, v = qkv.split([hq * d, hkv * d, hkv * d], dim=-1)         # strided views, as the model passes them
    go = torch.randn(T, hq, d, device="cuda").to(torch.bfloat16)
    F.varlen_attention(q.unflatten(-1, (hq, d)), k.unflatten(-1, (hkv, d)), v.unflatten(-1, (hkv, d)), cu,
                       max(lens)).backward(go)
    torch.cuda.synchronize()
    assert native.read_status(qkv.device) == 0
    ref = qkv.detach().float().requires_grad_(True)
    rq, rk, rv = ref.split([hq * d, hkv * d, hkv * d], dim=-1)
    R.varlen_attention(rq.unflatten(-1, (hq, d)), rk.unflatten(-1, (hkv, d)), rv.unflatten(-1, (hkv, d)), cu,
                       1.0 / math.sqrt(d)).backward(go.float())
    err = (qkv.grad.float() - ref.grad).abs().max().item()
    assert err <= 3e-2 * ref.grad.abs().max().item() + 2e-2, err


@pytest.mark.gpu
@pytest.mark.parametrize("lq,lk,hq,hkv", [([200, 56], None, 4, 2), ([300, 130], [77, 200], 4, 4), ([64], [333], 2, 1)])
def test_bidirectional_attention_self_and_cross(lq, lk, hq, hkv):
    """Non-causal mode of the attention kernels: every query sees all keys of its sequence, the key sequence may be
    shorter or longer than the query sequence (cross-attention)."""
    torch.manual_seed(14)
    d = 128
    cum = lambda l: torch.tensor([0] + list(torch.tensor(l).cumsum(0)), dtype=torch.int32, device="cuda")
    cq = cum(lq)
    ck = cq if lk is None else cum(lk)
    lk = lq if lk is None else lk
    q = torch.randn(sum(lq), hq, d, device="cuda").to(torch.bfloat16).requires_grad_(True)
    k = torch.randn(sum(lk), hkv, d, device="cuda").to(torch.bfloat16).requires_grad_(True)
    v = torch.randn(sum(lk), hkv, d, device="cuda").to(torch.bfloat16).requires_grad_(True)
    go = torch.randn(sum(lq), hq, d, device="cuda").to(torch.bfloat16)
    out = F.full_attention(q, k, v, cq, ck, max(lq), max(lk))
    out.backward(go)
    torch.cuda.synchronize()
    assert native.read_status(q.device) == 0
    rq, rk, rv = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    ref = R.varlen_attention(rq, rk, rv, cq, 1.0 / math.sqrt(d), causal=False, cu_k=ck)
    ref.backward(go.float())
    assert torch.allclose(out.float(), ref, atol=2e-2, rtol=2e-2), (out.float() - ref).abs().max()
    for got, want in ((q.grad, rq.grad), (k.grad, rk.grad), (v.grad, rv.grad)):
        err = (got.float() - want).abs().max().item()
        assert err <= 3e-2 * want.abs().max().item() + 2e-2, err


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(128, 128, 128), (300, 520, 1040), (1024, 3584, 3584), (17, 256, 4096)])
def test_gemm_fp8_block_scaled(M, N, K):
    torch.manual_seed(5)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    a[:, : K // 2] *= 8.0                                  # different scales along K: exercises the promotion
    b = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    aq, sa = F.quant_fp8_block(a, 1)
    bq, sb = F.quant_fp8_block(b, 128)
    got = F.gemm_fp8_block(aq, sa, bq, sb)
    torch.cuda.synchronize()
    assert native.read_status(a.device) == 0
    ref = R.dequant_fp8_block(aq, sa, 1, 128) @ R.dequant_fp8_block(bq, sb, 128, 128).t()   # same quantised inputs
    err = (got.float() - ref).abs().max().item()
    assert err <= 1e-2 * ref.abs().max().item() + 1e-3, err
    full = a.float() @ b.float().t()                       # and fp8 itself is close to the bf16 product
    assert (got.float() - full).abs().mean().item() <= 0.05 * full.abs().mean().item()
    y = F.fp8_linear(a, bq, sb)
    assert torch.equal(y, got)


@pytest.mark.gpu
# half a box of activation columns, one tile and eight columns, the layer's; a contraction of less than a block, and of a ragged
# number of them; enough rows for CTA pairs, and all other numbers that are not
@pytest.mark.parametrize("I,K,rows", [(8, 40, [1, 0, 130]), (136, 264, [128, 300, 0, 5]), (768, 512, [0, 257, 64]),
                                      (640, 512, [4500, 0, 4200])])
def test_grouped_gate_up_has_the_bits_of_two_passes(I, K, rows):
    E, lib, st = len(rows), native.lib(), native.status_word(torch.device("cuda"))
    padded = [(r + 127) // 128 * 128 for r in rows]
    Mp = sum(padded) + 128 * E
    sms = native.num_sms(0)
    assert lib.b200_grouped_gemm_pairs(Mp, 2 * I, K, E, 0, sms) == int(max(rows) > 4000)
    torch.manual_seed(I)
    first = torch.tensor([0] + padded, dtype=torch.int32).cumsum(0).to(torch.int32)
    x = torch.zeros(Mp, K, dtype=torch.bfloat16, device="cuda")
    for e, r in enumerate(rows):
        x[first[e]:first[e] + r] = torch.randn(r, K, device="cuda").to(torch.bfloat16)
    w = torch.randn(E, 2 * I, K, device="cuda").to(torch.bfloat16)
    w[0, :I] *= 40.0                                         # gates whose exponential overflows
    tiles = torch.repeat_interleave(torch.arange(E, dtype=torch.int32), torch.tensor(padded) // 128).cuda()
    n_tiles, offsets = torch.tensor([tiles.numel()], dtype=torch.int32, device="cuda"), first.cuda()
    h1, act = (torch.full((Mp, n), 7.0, dtype=torch.bfloat16, device="cuda") for n in (2 * I, I))
    native.check(native.host().b200_grouped_gate_up(x, w, h1, act, Mp, I, K, E, K, offsets, tiles, n_tiles, st, sms, native.stream()),
                 "grouped_gate_up")
    want_h1, want = torch.full_like(h1, 7.0), torch.full_like(act, 7.0)
    native.check(lib.b200_grouped_gemm(native.ptr(x), native.ptr(w), native.ptr(want_h1), Mp, 2 * I, K, E, K, 2 * I,
                                       native.ptr(tiles), native.ptr(n_tiles), 0, 0, native.ptr(st), sms, native.stream()),
                 "grouped_gemm")
    native.check(lib.b200_swiglu_fwd(native.ptr(want_h1), native.ptr(want), Mp, I, native.ptr(n_tiles), native.stream()), "swiglu_fwd")
    torch.cuda.synchronize()
    assert native.read_status(x.device) == 0
    assert torch.equal(h1, want_h1) and torch.equal(act.view(torch.int16), want.view(torch.int16))


@pytest.mark.gpu
# rows an expert: none, one, a whole pair of row blocks, one row more, the second block's last row; columns and contractions that
# end inside a tile; more row blocks than run side by side
@pytest.mark.parametrize("E,N,K,rows", [(40, 1032, 520, [0, 1, 256, 257, 511, 640, 129, 384]), (3, 1280, 512, [4500, 0, 4200]),
                                        (64, 512, 840, [255, 513, 300])])
@pytest.mark.parametrize("mode", [0, 1])
def test_grouped_gemm_on_pairs(E, N, K, rows, mode):
    rows = [rows[e % len(rows)] for e in range(E)]
    padded = [(r + 127) // 128 * 128 for r in rows]
    Mp = sum(padded) + 128 * E
    assert native.lib().b200_grouped_gemm_pairs(Mp, N, K, E, mode, native.num_sms(0)) == 1
    torch.manual_seed(E)
    offsets = torch.tensor([0] + padded, dtype=torch.int32).cumsum(0).to(torch.int32)
    x = torch.zeros(Mp, K, dtype=torch.bfloat16, device="cuda")
    for e, r in enumerate(rows):
        x[offsets[e]:offsets[e] + r] = torch.randn(r, K, device="cuda").to(torch.bfloat16)
    w = torch.randn((E, N, K) if mode == 0 else (E, K, N), device="cuda").to(torch.bfloat16)
    out = torch.full((Mp, N), 7.0, dtype=torch.bfloat16, device="cuda")
    tiles = torch.repeat_interleave(torch.arange(E, dtype=torch.int32), torch.tensor(padded) // 128).cuda()
    n_tiles, first = torch.tensor([tiles.numel()], dtype=torch.int32, device="cuda"), offsets.cuda()
    st = native.status_word(x.device)
    native.check(native.lib().b200_grouped_gemm_rows(native.ptr(x), native.ptr(w), native.ptr(out), Mp, N, K, E, K, N,
                                                     native.ptr(first), native.ptr(tiles), native.ptr(n_tiles), mode, 0,
                                                     native.ptr(st), native.num_sms(0), native.stream()), "grouped_gemm")
    torch.cuda.synchronize()
    assert native.read_status(x.device) == 0
    for e in range(E):
        lo, hi = int(offsets[e]), int(offsets[e + 1])
        a, b = x[lo:hi].double(), (w[e].t() if mode == 0 else w[e]).double()
        # one rounding to bf16 (2^-9) and fp32 sums of K products, which a 64-bit sum bounds by 2^-24 K |a| |b|
        bound = (a @ b).abs() * 2.0 ** -8 + 2.0 ** -24 * K * (a.abs() @ b.abs()) + 1e-30
        assert ((out[lo:hi].double() - a @ b).abs() <= bound).all()
    assert (out[offsets[E]:] == 7.0).all()


@pytest.mark.gpu
# ragged result rows and columns; experts without rows; fp32 sums; too few rows for CTA pairs; a round more than single CTAs have
@pytest.mark.parametrize("E,N,K,rows,pairs", [(10, 1000, 520, [256, 0, 1280, 768, 0, 512, 2048, 256, 1024, 1536], True),
                                              (6, 1536, 768, [768] * 6, True), (40, 256, 520, [128] * 40, False),
                                              (10, 1032, 520, [256, 0, 1280, 768, 0, 512, 2048, 256, 1024, 1536], False)])
@pytest.mark.parametrize("out_dtype,accumulate", [(torch.bfloat16, False), (torch.bfloat16, True), (torch.float32, True)])
def test_grouped_wgrad_forms(E, N, K, rows, pairs, out_dtype, accumulate):
    torch.manual_seed(E)
    fp32 = out_dtype == torch.float32
    assert native.lib().b200_grouped_wgrad_pairs(sum(rows), N, K, E, int(fp32), int(accumulate), native.num_sms(0)) == \
        (pairs and (fp32 or not accumulate))
    off = torch.tensor([0] + rows, device="cuda").cumsum(0).to(torch.int32)
    Mp = int(off[-1])
    dy, x = torch.randn(Mp, N, device="cuda").to(torch.bfloat16), torch.randn(Mp, K, device="cuda").to(torch.bfloat16)
    out = torch.randn(E, N, K, device="cuda").to(out_dtype)
    before = out.double()
    native.check(native.lib().b200_grouped_wgrad(native.ptr(dy), native.ptr(x), native.ptr(out), Mp, N, K, E, N, K,
                                                 native.ptr(off), int(out_dtype == torch.float32), int(accumulate),
                                                 native.ptr(native.status_word(x.device)), native.num_sms(0),
                                                 native.stream()), "grouped_wgrad")
    torch.cuda.synchronize()
    assert native.read_status(x.device) == 0
    for e in range(E):
        a, b = dy[off[e]:off[e + 1]].double(), x[off[e]:off[e + 1]].double()
        ref = a.t() @ b + (before[e] if accumulate else 0)
        bound = 2.0 ** -20 * a.norm(dim=0)[:, None] * b.norm(dim=0) + 1e-5      # fp32 sums
        if out_dtype == torch.bfloat16:
            bound = bound + 2.0 ** -8 * ref.abs()                              # and one rounding
        assert ((out[e].double() - ref).abs() <= bound).all(), e


@pytest.mark.gpu
# (rows, columns, contraction): one tile and few rows; ragged everything; tiles of 128 columns because there are no more of them;
# tiles of 128 columns, of which ten are left for a second round (not where A is stored transposed with rows that fill no box, as
# the first of the two has them); 256 columns and a second round; two shares of uneven length;
# columns that end inside 16 bytes; a contraction too short to be cut
@pytest.mark.parametrize("M,N,K", [(3, 256, 4096), (127, 1032, 4200), (129, 520, 8200), (300, 104, 4096), (700, 3584, 4104),
                                   (704, 3584, 4104), (1300, 3840, 4104), (900, 2304, 4160), (300, 1001, 4096), (256, 512, 512)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("out_dtype,accumulate", [(torch.bfloat16, False), (torch.float32, False), (torch.bfloat16, True),
                                                  (torch.float32, True)])
def test_gemm_cut_last_round(M, N, K, a_mn, b_mn, out_dtype, accumulate):
    torch.manual_seed(M + N)
    a, b = torch.randn(M, K, device="cuda").to(torch.bfloat16), torch.randn(N, K, device="cuda").to(torch.bfloat16)
    bv = None if accumulate else torch.randn(N, device="cuda").to(torch.bfloat16)
    sms, few = native.num_sms(0), M <= 128
    width = 128 if N <= 128 or (N == 3584 and not (a_mn and M % 64)) else 256
    left = -(-M // 256) * -(-N // width) % (sms // 2)
    scratch = F._gemm_scratch(M, N, K, a_mn, True, out_dtype == torch.float32, accumulate, bv is not None, False, 0, sms)
    shares = min(sms // 2 // left, 8)
    assert scratch == (0 if K == 512 or shares < 2 else left * shares * 256 * width)

    def stored(t):          # [K, rows], rows of whole 16 bytes
        buf = torch.zeros(K, (t.shape[0] + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")
        buf[:, :t.shape[0]] = t.t()
        return buf[:, :t.shape[0]]
    ops = stored(a) if a_mn else a, stored(b) if b_mn else b
    buf = torch.randn(M + 1, (N + 7) // 8 * 8, device="cuda").to(out_dtype)
    before = buf.clone()
    F.gemm(*ops, a_mn=a_mn, b_mn=b_mn, out=buf[:M, :N], accumulate=accumulate, bias=bv)
    torch.cuda.synchronize()
    assert native.read_status(a.device) == 0
    ref = a.double() @ b.double().t() + (0 if accumulate else bv.double())
    # fp32 sums of K products, and for bf16 one rounding of the product (not for few rows) and one of the sum with what was there
    bound = 2.0 ** -20 * a.double().norm(dim=1, keepdim=True) * b.double().norm(dim=1) + 1e-5
    if out_dtype == torch.bfloat16 and not (accumulate and few):
        bound = bound + 2.0 ** -8 * ref.abs()
    if accumulate:
        ref = ref + before[:M, :N].double()
        bound = bound + (2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -22) * ref.abs()
    assert ((buf[:M, :N].double() - ref).abs() <= bound).all()
    assert torch.equal(buf[M], before[M]) and torch.equal(buf[:M, N:], before[:M, N:])
    again = before.clone()
    F.gemm(*ops, a_mn=a_mn, b_mn=b_mn, out=again[:M, :N], accumulate=accumulate, bias=bv)
    assert torch.equal(again, buf)


@pytest.mark.gpu
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("n,hq,hkv", [(129, 4, 2), (700, 16, 4), (1200, 16, 16)])
def test_attention_far_apart_scores(n, hq, hkv, causal):
    """Scores that lie hundreds apart, so that most probabilities are below the smallest normal number, and a NaN key: it reaches
    every query that sees it and no other."""
    torch.manual_seed(n)
    d = 128
    q = (torch.randn(n, hq, d, device="cuda") * 6).to(torch.bfloat16).requires_grad_(True)
    k = (torch.randn(n, hkv, d, device="cuda") * 6).to(torch.bfloat16).requires_grad_(True)
    v = torch.randn(n, hkv, d, device="cuda").to(torch.bfloat16).requires_grad_(True)
    cu = torch.tensor([0, n], dtype=torch.int32, device="cuda")
    go = torch.randn(n, hq, d, device="cuda").to(torch.bfloat16)

    def run(q, k, v):
        return F.varlen_attention(q, k, v, cu, n) if causal else F.full_attention(q, k, v, cu, cu, n, n)
    out = run(q, k, v)
    out.backward(go)
    rq, rk, rv = (t.detach().double().requires_grad_(True) for t in (q, k, v))
    s = torch.einsum("qhd,khd->hqk", rq, rk.repeat_interleave(hq // hkv, 1)) / math.sqrt(d)
    if causal:
        s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    assert (s.detach()[:, -1].amax(-1) - s.detach()[:, -1].median(-1).values).min() > 64
    ref = torch.einsum("hqk,khd->qhd", s.softmax(-1), rv.repeat_interleave(hq // hkv, 1))
    ref.backward(go.double())
    # P, dS and the results are rounded to bf16 (2^-9 each); scores of 36 sqrt(d) carry 2^-24 of that into the exponent
    for got, want in ((out, ref), (q.grad, rq.grad), (k.grad, rk.grad), (v.grad, rv.grad)):
        assert (got.double() - want).norm() <= 2.0 ** -6 * want.norm()
    bad = k.detach().clone()
    bad[n // 2, 0, 5] = float("nan")
    with torch.no_grad():
        hit = run(q.detach(), bad, v.detach()).isnan().any(-1)      # [n, hq]
    want = torch.zeros_like(hit)
    want[n // 2 if causal else 0:, : hq // hkv] = True
    assert torch.equal(hit, want)
    assert native.read_status(q.device) == 0


@pytest.mark.gpu
# one row; K of one block, of less than one, of 4 n + 1 blocks; columns that end inside 16 bytes. CTA pairs: one block, an odd
# number of blocks, more of them than stages, with a second CTA that has one row or none and in one round of tiles and several
@pytest.mark.parametrize("M,N,K,pairs", [(1, 264, 128, False), (3, 5, 144, False), (1, 4096, 640, False), (127, 1001, 112, False),
                                         (129, 19000, 128, False), (257, 19197, 656, False), (129, 18900, 128, True),
                                         (129, 18901, 656, True), (384, 9470, 640, True), (2000, 12300, 400, True),
                                         (2000, 12300, 640, True), (1930, 12299, 1408, True)])
def test_gemm_fp8_block_forms(M, N, K, pairs):
    assert native.lib().b200_gemm_fp8_block_pairs(M, N, native.num_sms(0)) == pairs
    torch.manual_seed(M)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    aq, sa = F.quant_fp8_block(a, 1)
    bq, sb = F.quant_fp8_block(b, 128)
    out = torch.full((M + 1, (N + 7) // 8 * 8), 7.0, dtype=torch.bfloat16, device="cuda")
    F.gemm_fp8_block(aq, sa, bq, sb, out=out[:M, :N])
    torch.cuda.synchronize()
    assert native.read_status(a.device) == 0
    ref = R.dequant_fp8_block(aq, sa, 1, 128).double() @ R.dequant_fp8_block(bq, sb, 128, 128).double().t()
    # one rounding to bf16 (2^-9) and the fp32 sums of K products, which a 64-bit sum bounds by 2^-24 K |a| |b|
    bound = ref.abs() * 2.0 ** -8 + 2.0 ** -20 * K ** 0.5 * (a.double().norm(dim=1, keepdim=True) * b.double().norm(dim=1)) + 1e-6
    assert ((out[:M, :N].double() - ref).abs() <= bound).all()
    assert (out[M] == 7.0).all() and (out[:M, N:] == 7.0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 13, 33, 127, 129])
@pytest.mark.parametrize("inter,K", [(1536, 512), (14336, 256)])
def test_gate_up_rows_that_fill_no_box(M, inter, K):
    """Row counts between the sizes of the activation tiles: boxes of exactly those rows, and nothing of the accumulator's
    other rows reaches the result."""
    torch.manual_seed(M)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(2 * inter, K, device="cuda") * 0.05).to(torch.bfloat16)
    got = F.skinny_gate_up_swiglu(x, w)
    torch.cuda.synchronize()
    assert native.read_status(x.device) == 0
    h = x.double() @ w.double().t()
    ref = torch.nn.functional.silu(h[:, :inter]) * h[:, inter:]
    assert (got.double() - ref).abs().max() <= 2.0 ** -8 * ref.abs().max() + 1e-5   # one rounding, fp32 sums


@pytest.mark.gpu
@pytest.mark.parametrize("hq,hkv,n", [(28, 4, 4), (8, 8, 8), (64, 8, 3), (28, 4, 8)])
def test_paged_decode_shared_prefix_groups(hq, hkv, n):
    """Groups of n sequences share their first pages; the prefix pass + suffix pass + merge must equal plain
    attention over each sequence's whole block table."""
    torch.manual_seed(14)
    d, P, max_pages, max_shared = 128, 128, 8, 5
    groups = [(3, [400, 385, 500, 700, 384 + 1, 600, 900, 1000]), (0, [5, 100, 128, 129, 300, 1, 7, 64]),
              (5, [641, 700, 1024, 800, 650, 900, 1000, 777])]
    B = len(groups) * n
    n_pages = 1 + len(groups) * (5 + n * max_pages)
    cache = torch.zeros(n_pages, 2, hkv, P, d, dtype=torch.bfloat16, device=DEV)
    free = list(range(1, n_pages))
    bt = torch.zeros(B, max_pages, dtype=torch.int32)
    lens, pref = [], []
    for gi, (shared, ls) in enumerate(groups):
        shared_pages = [free.pop() for _ in range(shared)]
        for j in range(n):
            L = ls[j]
            own = [free.pop() for _ in range(max_pages - shared)]
            bt[gi * n + j] = torch.tensor(shared_pages + own)
            lens.append(L)
            pref.append(shared)
    # fill every page that any sequence can see with random K/V (shared pages hold the same data for the group)
    used = sorted(set(bt.flatten().tolist()))
    for pg in used:
        cache[pg, 0] = _bf16(hkv, P, d)
        cache[pg, 1] = _bf16(hkv, d, P)             # V slabs are stored transposed
    bt_d = bt.to(DEV)
    seq_lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    prefix = torch.tensor(pref, dtype=torch.int32, device=DEV)
    q = _bf16(B, hq, d)
    ref = R.paged_decode(q.cpu(), cache.cpu(), bt, seq_lens.cpu(), v_transposed=True)
    out = F.paged_decode(q, cache, bt_d, seq_lens, nsplit=1, v_transposed=True, prefix_pages=prefix, group=n,
                         max_shared=max_shared)
    torch.cuda.synchronize()
    assert native.read_status(q.device) == 0
    err = (out.float().cpu() - ref.float()).abs().max().item()
    assert err < 3e-2, err
    # a retired member (prefix 0) must not disturb the others
    prefix2 = prefix.clone()
    prefix2[0] = 0
    out2 = F.paged_decode(q, cache, bt_d, seq_lens, nsplit=1, v_transposed=True, prefix_pages=prefix2, group=n,
                          max_shared=max_shared)
    assert native.read_status(q.device) == 0
    assert (out2[1:].float().cpu() - ref[1:].float()).abs().max().item() < 3e-2


@pytest.mark.gpu
def test_dit_bf16_on_gpu_matches_fp32_reference():
    """Diffusion transformer with head_dim 128: self- and cross-attention run the non-causal tcgen05 kernels."""
    from cosmos_rl_b200.models.dit import DiT, DiTArgs
    torch.manual_seed(0)
    a = DiTArgs(in_channels=4, patch_size=(1, 2, 2), dim=256, n_layers=2, n_heads=2, head_dim=128, ffn_dim=512,
                text_dim=128, freq_dim=64)
    ref = DiT(a)
    ref.init_weights(0)
    with torch.no_grad():
        for n, p in ref.named_parameters():
            if "modulation" in n or n.startswith("patch_out"):
                p.normal_(0, 0.05)
    z, t, text = torch.randn(2, 4, 2, 16, 16), torch.tensor([0.2, 0.8]), torch.randn(2, 9, 128)
    mask = torch.tensor([[1] * 9, [1] * 4 + [0] * 5], dtype=torch.bool)
    want = ref(z, t, text, mask)
    want.square().mean().backward()
    import copy
    gpu = copy.deepcopy(ref).to("cuda", torch.bfloat16)
    gpu.zero_grad()
    got = gpu(z.cuda().to(torch.bfloat16), t.cuda(), text.cuda().to(torch.bfloat16), mask.cuda())
    got.square().mean().backward()
    torch.cuda.synchronize()
    assert native.read_status(torch.device("cuda")) == 0
    assert (got.float().cpu() - want).abs().max() < 0.05 * want.abs().max() + 0.02
    g_ref, g_gpu = ref.layers[0].qkv.weight.grad, gpu.layers[0].qkv.weight.grad.float().cpu()
    assert torch.nn.functional.cosine_similarity(g_ref.flatten(), g_gpu.flatten(), dim=0) > 0.98


@pytest.mark.gpu
@pytest.mark.parametrize("family", ["qwen2_5_vl", "internvl", "qwen3_vl_moe"])
def test_native_vision_language_models_bf16_on_gpu_match_fp32_reference(family):
    """The native vision-language families on the GPU in bf16 (decoder with head_dim 128 on the tcgen05 attention and
    GEMM kernels, vision towers with the head sizes of the public checkpoints) against the same weights in fp32 on the
    CPU: logits of a packed batch with two images, and the gradient that reaches the vision tower."""
    import copy
    torch.manual_seed(0)
    if family == "qwen2_5_vl":
        from cosmos_rl_b200.models.qwen2_5_vl import Qwen25VL, Qwen25VLArgs, VisionArgs
        a = Qwen25VLArgs(vocab_size=2048, dim=512, n_layers=2, n_heads=4, n_kv_heads=2, ffn_dim=1024, rope_theta=1e6,
                         qkv_bias=True, model_type="qwen2_5_vl", mrope_section=[16, 24, 24], image_token_id=2000)
        a.vision = VisionArgs(depth=3, hidden_size=160, num_heads=2, intermediate_size=216, out_hidden_size=512,
                              window_size=56, fullatt_block_indexes=[1])
        ref = Qwen25VL(a)
        grids = torch.tensor([[1, 6, 4], [1, 4, 8]])
        mm = {"pixel_values": torch.randn(56, 3 * 2 * 14 * 14), "image_grid_thw": grids}
        n_img, probe = (6, 8), lambda m: m.visual.blocks[0].qkv.weight
    elif family == "internvl":
        from cosmos_rl_b200.models.internvl import InternViTArgs, InternVL, InternVLArgs
        a = InternVLArgs(vocab_size=2048, dim=512, n_layers=2, n_heads=4, n_kv_heads=2, ffn_dim=1024, rope_theta=1e6,
                         qkv_bias=True, model_type="internvl", image_token_id=2000)
        a.vision = InternViTArgs(hidden_size=128, num_hidden_layers=2, num_attention_heads=2, intermediate_size=256,
                                 image_size=56, patch_size=14)
        ref = InternVL(a)
        mm = {"pixel_values": torch.randn(3, 3, 56, 56)}
        n_img, probe = (8, 4), lambda m: m.visual.blocks[0].q_proj.weight
    else:
        from cosmos_rl_b200.models.qwen3_vl_moe import Qwen3VisionArgs, Qwen3VLMoE, Qwen3VLMoEArgs
        a = Qwen3VLMoEArgs(vocab_size=2048, dim=512, n_layers=3, n_heads=4, n_kv_heads=2, head_dim=128, ffn_dim=512,
                           rope_theta=5e6, qkv_bias=False, qk_norm=True, model_type="qwen3_vl_moe", n_experts=8, top_k=2,
                           moe_ffn_dim=256, mrope_section=[24, 20, 20], image_token_id=2000)
        a.vision = Qwen3VisionArgs(depth=3, hidden_size=144, num_heads=2, intermediate_size=256, out_hidden_size=512,
                                   num_position_embeddings=64, deepstack_visual_indexes=[0, 2])
        ref = Qwen3VLMoE(a)
        grids = torch.tensor([[1, 6, 4], [1, 4, 8]])
        mm = {"pixel_values": torch.randn(56, 3 * 2 * 16 * 16), "image_grid_thw": grids}
        n_img, probe = (6, 8), lambda m: m.visual.blocks[0].qkv.weight
    ref = ref.float()
    with torch.no_grad():
        for n, p in ref.named_parameters():
            if p.dim() > 1:
                p.normal_(0, 0.05)
            else:                               # norm weights 1, layer scales 0.1, biases 0
                p.fill_(1.0 if "norm" in n and not n.endswith("_b") else (0.1 if "scale" in n else 0.0))
        for n, p in ref.named_parameters():
            if n.endswith("mlp.gate.weight"):   # decisive routing: bf16 rounding must not flip the chosen experts
                p.normal_(0, 1.0)
    g = torch.Generator().manual_seed(1)
    seq1 = torch.randint(0, 1900, (40,), generator=g).tolist()
    seq2 = torch.randint(0, 1900, (25,), generator=g).tolist()
    seq1[5:5] = [2000] * n_img[0]
    seq2[3:3] = [2000] * n_img[1]
    ids = torch.tensor(seq1 + seq2)
    cu = torch.tensor([0, len(seq1), len(seq1) + len(seq2)], dtype=torch.int32)
    ref.mm_inputs = mm
    want = ref.logits(ref(ids, ref.get_position_ids(cu, ids.numel()), cu, len(seq1)))
    want.square().mean().backward()
    gpu = copy.deepcopy(ref).to("cuda", torch.bfloat16)
    gpu.zero_grad()
    gpu.mm_inputs = {k: v.cuda() if k == "pixel_values" else v for k, v in mm.items()}
    cu_g = cu.cuda()
    got = gpu.logits(gpu(ids.cuda(), gpu.get_position_ids(cu_g, ids.numel()), cu_g, len(seq1)))
    got.square().mean().backward()
    torch.cuda.synchronize()
    assert native.read_status(torch.device("cuda")) == 0
    err = (got.float().cpu() - want).abs().amax(dim=1)              # per token
    tol = 0.06 * want.abs().max() + 0.03
    if family == "qwen3_vl_moe":       # a token whose second and third expert are nearly tied may still flip
        # the router's bf16 logits put the second and third expert of some tokens within rounding of each other in
        # at least one of the three blocks: those tokens take another expert than the fp32 model and differ by O(1)
        assert (err < tol).float().mean() > 0.7 and err.median() < tol / 3, (family, float(err.max()), float(err.median()))
    else:
        assert err.max() < tol, (family, err.max(), want.abs().max())
    g_ref, g_gpu = probe(ref).grad, probe(gpu).grad.float().cpu()
    cos = torch.nn.functional.cosine_similarity(g_ref.flatten(), g_gpu.flatten(), dim=0)
    assert cos > (0.6 if family == "qwen3_vl_moe" else 0.97), (family, float(cos))   # routing flips change which experts a token trains


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols,swizzle", [(128, 128, False), (300, 2880, True), (1, 32, True), (257, 96, False)])
def test_mxfp4_quant_matches_reference_bit_for_bit(rows, cols, swizzle):
    torch.manual_seed(9)
    w = (torch.randn(rows, cols, device="cuda") * torch.logspace(-3, 2, rows, device="cuda")[:, None]).to(torch.bfloat16)
    w[0, :32] = 0                                          # an all-zero block takes the smallest scale
    if rows > 2:
        w[2, :8] = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, -5.0], device="cuda") * 4   # ties, amax 20 -> scale 4
        w[2, 8:32] = 0
    q, sf = F.quant_mxfp4(w, swizzle)
    rq, rsf = R.quant_mxfp4(w, swizzle)
    assert torch.equal(q, rq) and torch.equal(sf, rsf)
    back = F.dequant_mxfp4(q, sf, swizzle)
    assert torch.equal(back.float(), R.dequant_mxfp4(rq, rsf, swizzle).to(torch.bfloat16).float())
    # error bound: the grid's largest gap is 2 scales (half of it when rounding), and a block maximum just under
    # 8 scales saturates at 6 scales
    blk = w.float().view(rows, cols // 32, 32)
    scale = torch.exp2(torch.floor(torch.log2(blk.abs().amax(-1).clamp_min(1e-30))) - 2)
    assert ((back.float().view(rows, cols // 32, 32) - blk).abs() <= scale[..., None] * 2.0 + 1e-30).all()


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(1024, 4608, 3584), (304, 256, 1040)])
def test_fp8_training_linear_on_gpu(M, N, K):
    """All three GEMMs of a projection on the block-scaled fp8 kernel against the exact fp32 products."""
    torch.manual_seed(6)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16).requires_grad_(True)
    w = (torch.randn(N, K, device="cuda") * 0.03).to(torch.bfloat16).requires_grad_(True)
    w._fp8_train = True
    go = torch.randn(M, N, device="cuda").to(torch.bfloat16)
    y = F.linear_maybe_fp8(x, w)
    y.backward(go)
    torch.cuda.synchronize()
    assert native.read_status(x.device) == 0
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    (xr @ wr.t()).backward(go.float())
    rel = lambda a, b: ((a.float() - b).norm() / b.norm()).item()
    assert rel(y.detach(), (xr @ wr.t()).detach()) < 0.05
    assert rel(x.grad, xr.grad) < 0.05 and rel(w.grad, wr.grad) < 0.05


# ---------------------------------------------------------------------------------------------------------
# CTA-pair GEMM (cta_group::2), its epilogues, and the decode-sized split-K GEMM with fused reductions
# ---------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("path", [1, 2])
@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (512, 768, 256), (300, 1000, 520), (77, 136, 64),
                                   (1024, 3584, 3584), (2048, 4608, 1024), (129, 128, 4096)])
def test_gemm_both_kernels(path, M, N, K):
    torch.manual_seed(20)
    a, b = _bf16(M, K), _bf16(N, K)
    c = F.gemm(a, b, path=path)
    native.read_status(a.device)
    ref = a.float() @ b.float().t()
    assert torch.allclose(c.float(), ref, rtol=2e-2, atol=1e-2 * math.sqrt(K)), (c.float() - ref).abs().max()


@pytest.mark.parametrize("a_mn,b_mn", [(False, True), (True, True), (True, False)])
def test_gemm_pair_kernel_operand_layouts(a_mn, b_mn):
    torch.manual_seed(21)
    M, N, K = 640, 904, 1096
    a = _bf16(K, M) if a_mn else _bf16(M, K)
    b = _bf16(K, N) if b_mn else _bf16(N, K)
    for out_dtype in (torch.bfloat16, torch.float32):
        out = F.gemm(a, b, a_mn=a_mn, b_mn=b_mn, path=2, out_dtype=out_dtype)
        native.read_status(a.device)
        ref = (a.float().t() if a_mn else a.float()) @ (b.float() if b_mn else b.float().t())
        assert torch.allclose(out.float(), ref, rtol=2e-2, atol=1e-2 * math.sqrt(K)), (out.float() - ref).abs().max()


def test_gemm_pair_kernel_bias_accumulate_and_swiglu():
    torch.manual_seed(22)
    M, N, K = 520, 1280, 768
    a, b = _bf16(M, K), _bf16(N, K, scale=0.05)
    bias = _bf16(N)
    ref = a.float() @ b.float().t()
    y = F.gemm(a, b, bias=bias, path=2)
    assert torch.allclose(y.float(), ref + bias.float(), rtol=2e-2, atol=0.1)
    # accumulate: C += A B^T by TMA reduce-add, fp32 and bf16
    acc = torch.full((M, N), 2.0, dtype=torch.float32, device=DEV)
    F.gemm(a, b, out=acc, accumulate=True, path=2)
    assert torch.allclose(acc, ref + 2.0, rtol=1e-3, atol=2e-2)
    acc16 = torch.full((M, N), 2.0, dtype=torch.bfloat16, device=DEV)
    F.gemm(a, b, out=acc16, accumulate=True, path=2)
    assert torch.allclose(acc16.float(), ref + 2.0, rtol=3e-2, atol=0.15)
    # SwiGLU epilogue on a fused gate/up weight
    I = N // 2
    g, u = ref[:, :I], ref[:, I:]
    z = F.gemm(a, b, swiglu=True)
    native.read_status(a.device)
    assert z.shape == (M, I)
    assert torch.allclose(z.float(), torch.nn.functional.silu(g) * u, rtol=3e-2, atol=0.05)


@pytest.mark.parametrize("M,N,K", [(128, 4608, 3584), (100, 3584, 3584), (8, 1024, 18944), (256, 3584, 1024),
                                   (200, 1000, 520), (128, 152064, 512)])
def test_gemm_skinny_matches_fp32(M, N, K):
    torch.manual_seed(23)
    x, w = _bf16(M, K), _bf16(N, K, scale=0.05)
    bias = _bf16(N)
    y = F.gemm_skinny(x, w, bias=bias)
    native.read_status(x.device)
    ref = x.float() @ w.float().t() + bias.float()
    assert torch.allclose(y.float(), ref, rtol=2e-2, atol=2e-2 * math.sqrt(K) * 0.05 + 0.05), (y.float() - ref).abs().max()


def test_skinny_fused_reductions():
    torch.manual_seed(24)
    M, H, I = 96, 1024, 2816
    hq, hkv, d, P = 6, 2, 128, 128
    x = _bf16(M, H)
    # o_proj / down_proj form: projection + residual + RMSNorm
    w = _bf16(H, I, scale=0.03)
    act = _bf16(M, I)
    res = _bf16(M, H)
    nw = (1.0 + 0.1 * torch.randn(H, device=DEV)).to(torch.bfloat16)
    y, res_out = F.skinny_linear_residual_rmsnorm(act, w, res, nw, 1e-6)
    native.read_status(x.device)
    r_ref = act.float() @ w.float().t() + res.float()
    assert torch.allclose(res_out.float(), r_ref, rtol=2e-2, atol=0.1)
    rr = res_out.float()
    y_ref = rr * torch.rsqrt(rr.pow(2).mean(-1, keepdim=True) + 1e-6) * nw.float()
    assert torch.allclose(y.float(), y_ref, rtol=2e-2, atol=2e-2)
    # gate/up form: SwiGLU in the GEMM epilogue
    wgu = _bf16(2 * I, H, scale=0.03)
    z = F.skinny_gate_up_swiglu(x, wgu)
    gu = x.float() @ wgu.float().t()
    assert torch.allclose(z.float(), torch.nn.functional.silu(gu[:, :I]) * gu[:, I:], rtol=3e-2, atol=0.05)
    # qkv form: bias + RoPE + cache append against the separate kernels
    wqkv = _bf16((hq + 2 * hkv) * d, H, scale=0.03)
    bqkv = _bf16((hq + 2 * hkv) * d)
    pos = torch.randint(0, 4000, (M,), device=DEV, dtype=torch.int64)
    n_pages = 8
    slots = torch.randperm(n_pages * P, device=DEV)[:M].to(torch.int32)
    slots[5] = -1
    for vt in (False, True):
        cache = torch.zeros(n_pages, 2, hkv, P, d, dtype=torch.bfloat16, device=DEV)
        q = F.skinny_qkv_rope_append(x, wqkv, bqkv, pos, slots, 1e6, hq, hkv, d, cache, vt)
        native.read_status(x.device)
        qkv_ref = (x.float() @ wqkv.float().t() + bqkv.float()).to(torch.bfloat16)
        q_ref, k_ref, v_ref = qkv_ref.split([hq * d, hkv * d, hkv * d], dim=-1)
        q_ref, k_ref = R.apply_rope(q_ref.reshape(M, hq, d).float(), k_ref.reshape(M, hkv, d).float(), pos, 1e6)
        assert torch.allclose(q.float(), q_ref.float(), rtol=2e-2, atol=3e-2), (q.float() - q_ref.float()).abs().max()
        cache_ref = torch.zeros_like(cache)
        R.kv_append(k_ref.to(torch.bfloat16), v_ref.reshape(M, hkv, d), cache_ref, slots, vt)
        assert torch.allclose(cache.float(), cache_ref.float(), rtol=2e-2, atol=3e-2)


def test_linear_product_path_runs_own_gemm():
    """The projection entry point of the models must reach this library's GEMM for bf16 CUDA tensors, in training
    (autograd) and inference (wide and decode-sized batches)."""
    torch.manual_seed(25)
    w = _bf16(768, 1024, scale=0.05).requires_grad_(True)
    b = _bf16(768).requires_grad_(True)
    for M in (64, 512):
        x = _bf16(M, 1024).requires_grad_(True)
        before = native.LAUNCHES[0]
        y = F.linear_maybe_fp8(x, w, b)
        assert native.LAUNCHES[0] > before
        y.float().sum().backward()
        ref = torch.nn.functional.linear(x.detach().float(), w.detach().float(), b.detach().float())
        assert torch.allclose(y.float(), ref, rtol=2e-2, atol=0.2)
        with torch.no_grad():
            before = native.LAUNCHES[0]
            y2 = F.linear_maybe_fp8(x, w, b)
            assert native.LAUNCHES[0] > before
            assert torch.allclose(y2.float(), ref, rtol=2e-2, atol=0.2)
    native.read_status(w.device)


def test_bounded_waits_run_out_report_status_and_release_tensor_memory():
    """Failure detection on the device, without a fault: a wait on a flag that nothing sets runs into its (short)
    limit, the kernel records ST_TIMEOUT_PEER_FLAG in the status word, frees what it holds and returns; the host
    reads the code, and the next tensor-core launch on the same context works (its TMEM allocation would block
    forever if the timed-out kernel had kept its columns)."""
    from cosmos_rl_b200.parallel import peer
    from cosmos_rl_b200.parallel.tp_fused import FusedTP
    dev = torch.device("cuda", torch.cuda.current_device())
    native.read_status(dev)
    # 1. the plain flag-wait kernel
    buf = peer.PeerBuffer(256, dev)
    peer.flag_wait(buf.ptr, 1, dev, limit_s=0.002)
    with pytest.raises(native.NativeError, match="peer flag"):
        native.read_status(dev)
    assert native.read_status(dev) == 0                      # reading the code re-arms the status word
    buf.free()
    # 2. the fused GEMM + all-reduce kernel (tcgen05 pipeline + side warps waiting for the other rank's arrivals)
    torch.manual_seed(30)
    M, N, K = 256, 512, 256
    a, w = _bf16(M, K), _bf16(N, K, scale=0.05)
    ctx = FusedTP.with_silent_peers(2, dev, M, N, wait_s=0.002)
    out = ctx.gemm_all_reduce(a, w)
    torch.cuda.synchronize()
    with pytest.raises(native.NativeError, match="peer flag"):
        native.read_status(dev)
    ctx.free_silent()
    del out
    # 3. the context is intact and no tensor memory leaked: ordinary GEMMs (both kernels) still run and are right
    ref = a.float() @ w.float().t()
    for path in (1, 2):
        c = F.gemm(a, w, path=path)
        assert torch.allclose(c.float(), ref, rtol=2e-2, atol=0.2)
    assert native.read_status(dev) == 0


def test_activation_offload_prefetches_and_keeps_gradients():
    """Saved activations go to pinned host memory in forward; in backward the copies of the tensors needed next are
    already enqueued when they are asked for (no host-side wait), and the gradients equal the resident run."""
    from torch import nn
    from cosmos_rl_b200.utils.activation_offloading import OffloadActivations
    torch.manual_seed(31)
    net = nn.Sequential(*[m for _ in range(6) for m in (nn.Linear(512, 512), nn.GELU())]).cuda()
    x = torch.randn(2048, 512, device=DEV, requires_grad=True)
    net(x).pow(2).sum().backward()
    ref = [p.grad.clone() for p in net.parameters()]
    gx = x.grad.clone()
    net.zero_grad()
    x.grad = None
    ctx = OffloadActivations(min_bytes=1 << 16, params={p.untyped_storage().data_ptr() for p in net.parameters()})
    with ctx:
        y = net(x).pow(2).sum()
    assert ctx.bytes_offloaded > 0 and len(ctx.stash) >= 6
    y.backward()
    torch.cuda.synchronize()
    assert ctx.n_prefetched >= len(ref) // 2 - 2, ctx.n_prefetched          # most fetches were issued ahead of their use
    assert not ctx.stash and not ctx.inflight
    for a, p in zip(ref, net.parameters()):
        assert torch.allclose(a, p.grad, rtol=1e-4, atol=1e-4)
    assert torch.allclose(gx, x.grad, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("fp32", [False, True])
def test_grouped_wgrad_accumulates(fp32):
    from cosmos_rl_b200.ops import moe
    torch.manual_seed(39)
    T, E, N, K = 200, 3, 136, 264
    idx = torch.randint(0, 2, (T, 1), device=DEV, dtype=torch.int32)                # the last expert has no rows
    disp = moe._Dispatch(idx, E)
    rows = [torch.zeros(disp.max_rows, n, dtype=torch.bfloat16, device=DEV) for n in (N, K)]
    off = disp.offsets.tolist()
    for r in rows:
        for e in range(E):
            r[off[e]:off[e + 1]] = _bf16(off[e + 1] - off[e], r.shape[1])
    out = _bf16(E, N, K).to(torch.float32 if fp32 else torch.bfloat16)
    want = out.double() + torch.stack([rows[0][off[e]:off[e + 1]].double().t() @ rows[1][off[e]:off[e + 1]].double() for e in range(E)])
    moe._grouped_wgrad(rows[0], rows[1], disp, out, True)
    native.read_status(out.device)
    assert torch.allclose(out.double(), want, rtol=1e-5 if fp32 else 2 ** -8, atol=1e-3)


@pytest.mark.parametrize("growth", [0.0, 60.0, -60.0])
def test_paged_decode_running_maximum(growth):
    """Scores that rise or fall by many powers of two from page to page; lengths around the page size."""
    torch.manual_seed(33)
    hq, hkv, d, P, B = 14, 2, 128, 128, 5
    lens = torch.tensor([1, 128, 129, 640, 1000], dtype=torch.int32, device=DEV)
    pages = 8
    table = (torch.arange(B * pages, device=DEV, dtype=torch.int32) + 1).view(B, pages)
    cache = torch.zeros(B * pages + 1, 2, hkv, P, d, dtype=torch.bfloat16, device=DEV)
    ramp = torch.linspace(0, growth, pages * P, device=DEV) / math.sqrt(d)
    for b in range(B):
        L = int(lens[b])
        t = torch.arange(L, device=DEV)
        k = (0.3 * torch.randn(L, hkv, d, device=DEV) + ramp[:L, None, None]).to(torch.bfloat16)
        F.kv_append(k, _bf16(L, hkv, d), cache, (table[b, t // P].long() * P + t % P).to(torch.int32), v_transposed=True)
    q = torch.ones(B, hq, d, device=DEV).to(torch.bfloat16)
    ref = R.paged_decode(q.cpu(), cache.cpu(), table.cpu(), lens.cpu(), v_transposed=True)
    for nsplit in (1, 3):
        out = F.paged_decode(q, cache, table, lens, nsplit=nsplit, v_transposed=True)
        native.read_status(q.device)
        assert (out.float().cpu() - ref.float()).abs().max() < 3e-2, nsplit


@pytest.mark.parametrize("T,H", [(1, 1032), (2, 2048), (3, 4096), (1185, 4104), (1184, 5120), (7, 128)])
def test_rmsnorm_row_groups(T, H):
    """One row, an odd number of rows, one and two vectors a thread, and more row groups than persistent blocks."""
    torch.manual_seed(34)
    x, w, res, gy, gr = _bf16(T, H), _bf16(H), _bf16(T, H), _bf16(T, H), _bf16(T, H)
    a = [t.clone().requires_grad_(True) for t in (x, w, res)]
    y, ro = F.rms_norm(a[0], a[1], 1e-6, a[2])
    got = torch.autograd.grad([y, ro], a, [gy, gr])
    assert torch.equal(ro, (x.float() + res.float()).to(torch.bfloat16))
    h = ro.double().requires_grad_(True)
    wd = w.double().requires_grad_(True)
    yr = h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-6) * wd
    dh, dw = torch.autograd.grad(yr, [h, wd], gy.double())
    # one bf16 rounding of the result is 2^-9 of it; the weight gradient sums T terms in fp32
    assert torch.allclose(y.double(), yr, rtol=2 ** -8, atol=1e-6)
    assert torch.allclose(got[0].double(), dh + gr.double(), rtol=2 ** -8, atol=1e-4)
    assert torch.equal(got[0], got[2])
    assert torch.allclose(got[1].double(), dw, rtol=2 ** -8, atol=1e-5 * T + 1e-5)


@pytest.mark.parametrize("T,H,I,E,k", [(5, 256, 128, 8, 1), (129, 264, 136, 4, 3), (260, 512, 256, 300, 9)])
def test_moe_experts_padding_and_many_choices(T, H, I, E, k):
    """Experts without tokens, tiles that are mostly padding, more experts than the scan's block, more choices than are
    summed at a time; whatever the permuted buffers held before must not show."""
    from cosmos_rl_b200.ops import moe
    torch.manual_seed(38)
    x, wgu, wd = (t.requires_grad_(True) for t in (_bf16(T, H), _bf16(E, 2 * I, H, scale=0.05), _bf16(E, H, I, scale=0.05)))
    idx = torch.stack([torch.randperm(max(k, E // 2), device=DEV)[:k] for _ in range(T)]).to(torch.int32)
    probs = torch.rand(T, k, device=DEV).requires_grad_(True)
    junk = [torch.full((1 << 24,), float("nan"), device=DEV) for _ in range(4)]     # freed blocks are handed out again
    del junk
    out = moe.moe_experts(x, probs, idx, wgu, wd)
    g = _bf16(T, H)
    got = torch.autograd.grad(out, (x, probs, wgu, wd), g)
    native.read_status(x.device)
    ref_in = [t.detach().float().requires_grad_(True) for t in (x, probs, wgu, wd)]
    ref = moe.moe_experts_reference(ref_in[0], ref_in[1], idx, ref_in[2], ref_in[3])
    want = torch.autograd.grad(ref, ref_in, g.float())
    assert torch.allclose(out.float(), ref, rtol=3e-2, atol=3e-2 * ref.abs().max().item())
    for a, b in zip(got, want):
        assert torch.allclose(a.float(), b, rtol=5e-2, atol=5e-2 * b.abs().max().item())


@pytest.mark.parametrize("M", [1, 16, 17, 64, 65, 129, 256])
@pytest.mark.parametrize("I,K", [(14336, 512), (18944, 128), (1000, 520), (64, 64)])
def test_skinny_swiglu_tile_widths(M, I, K):
    """Row counts around the kept A rows (16, 64, 128) and column counts that take both kinds of tiles."""
    torch.manual_seed(35)
    x, w = _bf16(M, K), _bf16(2 * I, K, scale=0.05)
    z = F.skinny_gate_up_swiglu(x, w)
    native.read_status(x.device)
    gu = x.float() @ w.float().t()
    ref = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
    # fp32 sums of K products, rounded once to bf16
    assert torch.allclose(z.float(), ref, rtol=2 ** -8, atol=1e-4 * math.sqrt(K)), (z.float() - ref).abs().max()


@pytest.mark.parametrize("M", [1, 16, 17, 64, 65])
@pytest.mark.parametrize("N,K", [(4096, 2048), (6144, 1032), (32000, 512), (72, 64)])
def test_skinny_kept_rows(M, N, K):
    torch.manual_seed(36)
    x, w, res = _bf16(M, K), _bf16(N, K, scale=0.05), _bf16(M, N)
    y = F.gemm_skinny(x, w)
    ref = x.float() @ w.float().t()
    assert torch.allclose(y.float(), ref, rtol=2 ** -8, atol=1e-4 * math.sqrt(K))
    if N <= 8192:
        _, r = F.skinny_linear_residual_rmsnorm(x, w, res, torch.ones(N, dtype=torch.bfloat16, device=DEV), 1e-6)
        assert torch.allclose(r.float(), ref + res.float(), rtol=2 ** -8, atol=1e-4 * math.sqrt(K))
    native.read_status(x.device)


# ------------------------------------------------------------------------------------------------ edges of tiles
@pytest.mark.parametrize("lens,hq,hkv,causal", [([127], 3, 1, True), ([128, 129], 2, 2, True), ([255, 256, 257, 1], 4, 2, True),
                                                ([385], 7, 1, True), ([127, 1, 130], 2, 1, False), ([513, 64], 2, 2, False)])
def test_flash_attention_tile_edges(lens, hq, hkv, causal):
    """Sequence lengths around one and two tiles of queries and keys: forward and gradients against fp32, the same bits on
    a second run, and a zero query gradient for tokens that belong to no sequence."""
    from cosmos_rl_b200.ops import attention
    torch.manual_seed(31)
    d, T = 128, sum(lens) + 3                                       # three tokens after the last sequence
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    q, k, v, go = _bf16(T, hq, d), _bf16(T, hkv, d), _bf16(T, hkv, d), _bf16(T, hq, d)
    scale, n = 1.0 / math.sqrt(d), sum(lens)
    out, lse = attention.flash_fwd(q, k, v, cu, cu, max(lens), scale, causal)
    grads = attention.flash_bwd(go, q, k, v, out, lse, cu, max(lens), scale, causal=causal)
    again = attention.flash_bwd(go, q, k, v, out, lse, cu, max(lens), scale, causal=causal)
    native.read_status(q.device)
    assert torch.equal(grads[0], again[0]) and all(torch.equal(a[:n], b[:n]) for a, b in zip(grads[1:], again[1:]))
    assert not grads[0][n:].any()
    rq, rk, rv = (t.float().requires_grad_(True) for t in (q, k, v))
    ref = R.varlen_attention(rq, rk, rv, cu, scale, causal=causal)
    ref.backward(go.float())
    # bf16 rounds the result (2^-9 of it) and P / dS on the way (2^-9 of sums of about unit terms)
    assert torch.allclose(out[:n].float(), ref[:n], atol=2e-2, rtol=2e-2)
    for got, want in zip(grads, (rq.grad, rk.grad, rv.grad)):
        assert (got[:n].float() - want[:n]).abs().max() <= 3e-2 * want.abs().max() + 2e-2


@pytest.mark.parametrize("causal,max_q", [(True, 299), (True, 700), (False, 700)])
def test_flash_attention_many_sequences(causal, max_q):
    """More items than SMs over more sequences than one warp-wide step of the work list covers, empty ones among them, and
    a bound on the length that no sequence reaches."""
    from cosmos_rl_b200.ops import attention
    torch.manual_seed(62)
    lens = [(37 * i) % 300 for i in range(70)]
    d, hq, hkv, T = 128, 16, 4, sum(lens) + 5
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    q, k, v, go = _bf16(T, hq, d), _bf16(T, hkv, d), _bf16(T, hkv, d), _bf16(T, hq, d)
    scale, n = 1.0 / math.sqrt(d), sum(lens)
    out, lse = attention.flash_fwd(q, k, v, cu, cu, max_q, scale, causal)
    grads = attention.flash_bwd(go, q, k, v, out, lse, cu, max_q, scale, causal=causal)
    native.read_status(q.device)
    assert not grads[0][n:].any()
    rq, rk, rv = (t.float().requires_grad_(True) for t in (q, k, v))
    ref = R.varlen_attention(rq, rk, rv, cu, scale, causal=causal)
    ref.backward(go.float())
    assert torch.allclose(out[:n].float(), ref[:n], atol=2e-2, rtol=2e-2)   # as in the test above
    for got, want in zip(grads, (rq.grad, rk.grad, rv.grad)):
        assert (got[:n].float() - want[:n]).abs().max() <= 3e-2 * want.abs().max() + 2e-2


def test_flash_attention_scores_that_grow_along_the_keys():
    """Running maximum that moves in every key block (the accumulator is rescaled) and probabilities that underflow."""
    from cosmos_rl_b200.ops import attention
    torch.manual_seed(32)
    L, h, d = 700, 2, 128
    q = torch.ones(L, h, d, device=DEV).to(torch.bfloat16)
    k = (torch.linspace(0, 40, L, device=DEV)[:, None, None] + torch.zeros(L, h, d, device=DEV)).to(torch.bfloat16)
    v = _bf16(L, h, d)
    cu = torch.tensor([0, L], dtype=torch.int32, device=DEV)
    out, _ = attention.flash_fwd(q, k, v, cu, cu, L, 1.0 / math.sqrt(d), True)
    native.read_status(q.device)
    ref = R.varlen_attention(q.float(), k.float(), v.float(), cu, 1.0 / math.sqrt(d))
    assert torch.allclose(out.float(), ref, atol=2e-2, rtol=2e-2), (out.float() - ref).abs().max()


# ------------------------------------------------------------------------------------------------ what memory held before
@pytest.fixture
def dirty_allocations(monkeypatch):
    """New tensors hold NaN, as memory that the allocator hands out again may."""
    for name in ("empty", "empty_like"):
        def dirty(*args, _plain=getattr(torch, name), **kw):
            t = _plain(*args, **kw)
            return t.fill_(float("nan")) if t.is_floating_point() else t
        monkeypatch.setattr(torch, name, dirty)


def _moe_case(T, H, I, E, k):
    return [t.requires_grad_(True) for t in (_bf16(T, H), torch.rand(T, k, device=DEV), _bf16(E, 2 * I, H, scale=0.05),
                                             _bf16(E, H, I, scale=0.05))]


def _check_moe(out, args, idx):
    from cosmos_rl_b200.ops import moe
    g = _bf16(*out.shape)
    got = torch.autograd.grad(out, args, g)
    native.read_status(out.device)
    ref_in = [t.detach().float().requires_grad_(True) for t in args]
    ref = moe.moe_experts_reference(ref_in[0], ref_in[1], idx, ref_in[2], ref_in[3])
    want = torch.autograd.grad(ref, ref_in, g.float())
    assert torch.allclose(out.float(), ref, rtol=3e-2, atol=3e-2 * ref.abs().max().item())
    for a, b in zip(got, want):
        assert torch.allclose(a.float(), b, rtol=5e-2, atol=5e-2 * b.abs().max().item())


def test_moe_experts_counts_buffer_used_again_before_backward(dirty_allocations):
    """One histogram buffer, cleared and filled again for the next call while the first call's backward is still to come."""
    from cosmos_rl_b200.ops import moe
    torch.manual_seed(71)
    T, E, k = 200, 6, 2
    counts, calls = torch.zeros(E, dtype=torch.int32, device=DEV), []
    for favoured in (0, 3):                                          # other experts are the long ones in the second call
        logits = torch.randn(T, E, device=DEV)
        logits[:, favoured] += 6.0
        counts.zero_()
        probs, idx = moe.route_topk(logits, k, counts=counts)
        args = _moe_case(T, 256, 128, E, k)
        args[1] = probs.requires_grad_(True)
        calls.append((moe.moe_experts(args[0], args[1], idx, args[2], args[3], counts), args, idx))
    for call in calls:
        _check_moe(*call)


@pytest.mark.parametrize("spare", [0, 5000])
def test_moe_experts_counts_above_what_the_choices_hold(dirty_allocations, spare):
    """An upper bound instead of the histogram: whole tiles, and for the last experts (which no token chooses) more rows than
    the permuted buffers have."""
    from cosmos_rl_b200.ops import moe
    torch.manual_seed(72)
    T, E, k = 150, 4, 1
    args = _moe_case(T, 256, 128, E, k)
    idx = torch.randint(0, 2, (T, k), device=DEV, dtype=torch.int32)
    counts = (torch.bincount(idx.flatten().long(), minlength=E) + 127) // 128 * 128
    counts[2:] = 64 + spare
    _check_moe(moe.moe_experts(args[0], args[1], idx, args[2], args[3], counts.to(torch.int32)), args, idx)


@pytest.mark.parametrize("nsplit", [1, 2])
def test_paged_decode_largest_probability_is_not_rounded(nsplit):
    """Only the key with the largest score has values (ones): the result is 1 / sum, rounded once, wherever that key lies."""
    torch.manual_seed(78)
    B, h, d, P, L = 32, 4, 128, 128, 700
    pages = (L + P - 1) // P
    table = (torch.arange(B * pages, device=DEV, dtype=torch.int32) + 1).view(B, pages)
    lens = torch.full((B,), L, dtype=torch.int32, device=DEV)
    cache = _bf16(B * pages + 1, 2, h, P, d)
    q = _bf16(B, h, d)
    k = cache[1:, 0].view(B, pages, h, P, d).transpose(1, 2).reshape(B, h, pages * P, d)[:, :, :L].double()
    s = torch.einsum("bhd,bhkd->bhk", q.double(), k) / math.sqrt(d)
    top = s.argmax(-1)
    cache[:, 1] = 0
    b, hh = torch.meshgrid(torch.arange(B, device=DEV), torch.arange(h, device=DEV), indexing="ij")
    cache[table.long().gather(1, (top // P)), 1, hh, :, top % P] = 1
    out = F.paged_decode(q, cache, table, lens, nsplit=nsplit, v_transposed=True)
    native.read_status(q.device)
    want = (s - s.amax(-1, keepdim=True)).exp().sum(-1).reciprocal().to(torch.bfloat16)
    # fp32 scores and sums are off by about 1e-6 of the result, a rounding step is 2^-8 of it: next to none may round otherwise
    assert (out != want[..., None]).any(-1).float().mean() <= 0.02


@pytest.mark.parametrize("scale", [0.0, -0.03, -1.0 / math.sqrt(128)])
@pytest.mark.parametrize("lens,causal", [([300, 17, 129, 256], True), ([300, 130], False)])
def test_flash_attention_scale_of_zero_or_less(scale, lens, causal):
    """Partly visible key blocks at a scale of zero (the mean of the visible values) and below it, forward and gradients."""
    from cosmos_rl_b200.ops import attention
    torch.manual_seed(73)
    d, hq, hkv, T = 128, 4, 2, sum(lens)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    q, k, v, go = _bf16(T, hq, d), _bf16(T, hkv, d), _bf16(T, hkv, d), _bf16(T, hq, d)
    out, lse = attention.flash_fwd(q, k, v, cu, cu, max(lens), scale, causal)
    grads = attention.flash_bwd(go, q, k, v, out, lse, cu, max(lens), scale, causal=causal)
    native.read_status(q.device)
    rq, rk, rv = (t.float().requires_grad_(True) for t in (q, k, v))
    ref, ref_lse = R.varlen_attention(rq, rk, rv, cu, scale, causal=causal, return_lse=True)
    ref.backward(go.float())
    # bf16 rounds the result (2^-9 of it) and P / dS on the way (2^-9 of sums of about unit terms); lse is fp32 throughout
    assert torch.allclose(out.float(), ref, atol=2e-2, rtol=2e-2)
    assert torch.allclose(lse, ref_lse, atol=1e-3, rtol=1e-4)
    for got, want in zip(grads, (rq.grad, rk.grad, rv.grad)):
        assert (got.float() - want).abs().max() <= 3e-2 * want.abs().max() + 2e-2


def test_flash_attention_gradients_with_nothing_to_attend_to(dirty_allocations):
    """No sequences, no keys, no queries: every gradient that has rows is zero."""
    from cosmos_rl_b200.ops import attention
    torch.manual_seed(74)
    d, hq, hkv, T = 128, 2, 1, 96
    q, k, out, go = _bf16(T, hq, d), _bf16(T, hkv, d), _bf16(T, hq, d), _bf16(T, hq, d)
    for nq, nk, cu, cu_k in ((T, T, [0], [0]), (T, 0, [0, T], [0, 0]), (0, T, [0, 0], [0, T])):
        cu, cu_k = (torch.tensor(c, dtype=torch.int32, device=DEV) for c in (cu, cu_k))
        grads = attention.flash_bwd(go[:nq], q[:nq], k[:nk], k[:nk], out[:nq], torch.zeros(hq, nq, device=DEV), cu, T, 0.1,
                                    cu_k=cu_k, max_k=T, causal=False)
        assert [len(g) for g in grads] == [nq, nk, nk]
        assert all(torch.equal(g, torch.zeros_like(g)) for g in grads)


@pytest.mark.parametrize("hkv,bound", [(1, 130), (4, 16384)])   # a key block shared by two CTAs, or by one
def test_flash_attention_gradients_of_tokens_outside_the_sequences(dirty_allocations, hkv, bound):
    """Tokens before the first and after the last sequence: zero gradients of queries, keys and values, as the one packed
    tensor that they are slices of needs them."""
    from cosmos_rl_b200.ops import attention
    torch.manual_seed(75)
    d, hq, head, lens, tail = 128, 4, 5, [130, 64], 140
    T = head + sum(lens) + tail
    cu = torch.tensor([head] + list(head + torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    q, k, v, go = _bf16(T, hq, d), _bf16(T, hkv, d), _bf16(T, hkv, d), _bf16(T, hq, d)
    out, lse = attention.flash_fwd(q, k, v, cu, cu, max(lens), 0.1)
    grads = attention.flash_bwd(go, q, k, v, out, lse, cu, bound, 0.1)
    native.read_status(q.device)
    for g in grads:
        assert not g[:head].any() and not g[T - tail:].any() and torch.isfinite(g.float()).all()


@pytest.mark.parametrize("R_,C,off", [(128, 128, 0), (130, 200, 0), (5, 130, 1), (257, 264, 3)])
def test_quant_fp8_weight_blocks_match_reference_bit_for_bit(R_, C, off):
    """Ragged last blocks, and rows that start off the 16-byte grid."""
    torch.manual_seed(77)
    w = _bf16(R_, C + off + 7)[:, off:off + C]
    q, s = F.quant_fp8_block(w, 128)
    nr, nc = (R_ + 127) // 128, (C + 127) // 128
    pad = torch.zeros(nr * 128, nc * 128, device=DEV)
    pad[:R_, :C] = w.float()
    blocks = pad.view(nr, 128, nc, 128)
    scale = blocks.abs().amax((1, 3)).clamp_min(1e-12) / torch.tensor(448.0, device=DEV)
    assert torch.equal(s, scale)
    want = (blocks * (1.0 / scale)[:, None, :, None]).view(nr * 128, -1)[:R_, :C].to(torch.float8_e4m3fn)
    assert torch.equal(q.view(torch.uint8), want.view(torch.uint8))


def test_skinny_workspace_only_where_there_is_a_split():
    torch.manual_seed(76)
    x, wide, x2, narrow = _bf16(3, 512), _bf16(32000, 512, scale=0.05), _bf16(3, 4096), _bf16(512, 4096, scale=0.05)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    key = (x.device.index, s.cuda_stream)
    F._skinny_ws.pop(key, None)
    with torch.cuda.stream(s):
        y = F.gemm_skinny(x, wide)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):                         # a first call inside a capture keeps nothing of its pool
            z = F.gemm_skinny(x, wide)
        assert key not in F._skinny_ws
        g.replay()
        t = F.gemm_skinny(x2, narrow)
        assert key in F._skinny_ws
    s.synchronize()
    native.read_status(x.device)
    assert torch.equal(y, z)
    for out, a, w in ((y, x, wide), (t, x2, narrow)):               # fp32 sums of K products, rounded once to bf16
        assert torch.allclose(out.float(), a.float() @ w.float().t(), rtol=2 ** -8, atol=1e-4 * math.sqrt(a.shape[1]))


@pytest.mark.parametrize("hq,hkv,causal", [(4, 2, True), (7, 1, True), (4, 4, False)])
def test_flash_attention_forward_forms_agree(hq, hkv, causal):
    """A sequence alone has an SM for each of its tiles, packed with others it has not: the two forms of the forward on the
    same rows, sliced out of one packed tensor, with as many keys as queries and with more."""
    from cosmos_rl_b200.ops import attention
    torch.manual_seed(79)
    d, scale = 128, 1.0 / math.sqrt(128)
    lens = [1, 64, 127, 128, 129, 255, 256, 257, 385, 40] * 3
    more = [0, 5, 128, 300, 0, 1, 255, 0, 127, 0] * 3               # keys before the first query
    lk = [a + b for a, b in zip(lens, more)]
    T, Tk = sum(lens), sum(lk)
    q = _bf16(T, (hq + 3) * d)[:, d:(hq + 1) * d].unflatten(-1, (hq, d))
    kv = _bf16(Tk, 2 * hkv * d)
    k, v = kv[:, :hkv * d].unflatten(-1, (hkv, d)), kv[:, hkv * d:].unflatten(-1, (hkv, d))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    cq, ck = i32([0] + list(torch.tensor(lens).cumsum(0))), i32([0] + list(torch.tensor(lk).cumsum(0)))
    assert sum((n + 127) // 128 for n in lens) * hq > native.num_sms(0) >= (max(lens) + 127) // 128 * hq
    out, lse = attention.flash_fwd(q, k, v, cq, ck, max(lens), scale, causal)
    ref, ref_lse = R.varlen_attention(q.float(), k.float(), v.float(), cq, scale, causal, ck, return_lse=True)
    for i, n in enumerate(lens):
        r, c = slice(int(cq[i]), int(cq[i + 1])), slice(int(ck[i]), int(ck[i + 1]))
        one, one_lse = attention.flash_fwd(q[r], k[c], v[c], i32([0, n]), i32([0, lk[i]]), n, scale, causal)
        for got, got_lse in ((out[r], lse[:, r]), (one, one_lse)):
            assert torch.allclose(got.float(), ref[r], atol=2e-2, rtol=2e-2)     # bf16 result and probabilities
            assert torch.allclose(got_lse, ref_lse[:, r], atol=1e-3, rtol=1e-4)
    native.read_status(q.device)


@pytest.mark.parametrize("n,hq,hkv", [(200, 4, 2), (1300, 16, 4)])     # the one-tile form; two tiles an item
def test_flash_attention_hidden_keys_have_no_weight(n, hq, hkv):
    """Values of later tokens and of the next sequence leave no trace, however large they are, and a query that sees no key
    has a zero row and an infinite log-sum-exp."""
    from cosmos_rl_b200.ops import attention
    torch.manual_seed(80)
    d, scale = 128, 1.0 / math.sqrt(128)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    cu = i32([0, n, n + 77])
    q, k, v = _bf16(n + 77, hq, d), _bf16(n + 77, hkv, d), _bf16(n + 77, hkv, d)
    assert ((n + 127) // 128 * hq * 2 > native.num_sms(0)) == (n > 1000)
    for causal in (True, False):
        want, want_lse = attention.flash_fwd(q, k, v, cu, cu, n, scale, causal)
        for first in (n // 3, n - 1, n) if causal else (n,):        # the first value that is changed
            big = v.clone()
            big[first:] = 3e38
            got, got_lse = attention.flash_fwd(q, k, big, cu, cu, n, scale, causal)
            assert torch.equal(got[:first], want[:first]) and torch.equal(got_lse, want_lse), (causal, first)
    more = 60                                                       # queries without a key, in front
    out, lse = attention.flash_fwd(q[:n], k[:n - more], v[:n - more], i32([0, n]), i32([0, n - more]), n, scale, True)
    native.read_status(q.device)
    assert (out[:more] == 0).all() and (lse[:, :more] == math.inf).all()
    ref = R.varlen_attention(q[more:n].float(), k[:n - more].float(), v[:n - more].float(), i32([0, n - more]), scale, True)
    assert torch.allclose(out[more:].float(), ref, atol=2e-2, rtol=2e-2)     # bf16 result and probabilities


@pytest.mark.parametrize("M", [256, 1024])      # the weight-streaming epilogue, that of the CTA pairs
def test_swiglu_gives_the_same_bits_wherever_it_is_formed(M):
    """Each weight row picks one input, so that the products give the gate and up values exactly: the epilogues and the kernel
    that takes them from memory round the same way, saturated and zero gates among them."""
    torch.manual_seed(81)
    n = 4096
    x = _bf16(M, n) * 4
    x[:, ::9], x[:, 1::9], x[:, 2::9] = 0, -100, 100
    eye = torch.eye(n, device=DEV, dtype=torch.bfloat16)
    w = torch.cat([eye, eye.roll(5, 0)])
    got = F.skinny_gate_up_swiglu(x, w) if M <= 256 else F.gemm(x, w, swiglu=True)
    native.read_status(x.device)
    assert torch.equal(got, F.swiglu(torch.cat([x, x.roll(5, 1)], 1)))


@pytest.mark.parametrize("hq,hkv,longest,copies", [(2, 2, 128, 1), (4, 2, 64, 1), (14, 2, 64, 5), (3, 3, 65, 1)])
@pytest.mark.parametrize("causal", [True, False])
def test_flash_attention_backward_forms_agree(dirty_allocations, hq, hkv, longest, copies, causal):
    """Sequences short enough for the one-kernel backward, and the same call with a longer bound, which takes the general one:
    strided inputs, tokens outside the sequences, more and fewer keys than queries, none of either."""
    from cosmos_rl_b200.ops import attention
    torch.manual_seed(80)
    d, scale = 128, 1.0 / math.sqrt(128)
    lens = [n for n in (1, 31, 32, 33, 63, 64, 65, 127, 128, 0, 20, 40, 17) if n <= longest] * copies
    lk = [128 if i % 4 == 1 else min(128, n + 9) if i % 4 == 2 else n for i, n in enumerate(lens)]
    lk[-1] = 0
    if not causal:
        lk[-2] = 3
    T, Tk = sum(lens) + 5, sum(lk) + 7
    qkv = _bf16(T, (hq + 2) * d)
    q, kv = qkv[:, d:(hq + 1) * d].unflatten(-1, (hq, d)), _bf16(Tk, 2 * hkv * d)
    k, v = kv[:, :hkv * d].unflatten(-1, (hkv, d)), kv[:, hkv * d:].unflatten(-1, (hkv, d))
    go = _bf16(T, hq, d)
    cq, ck = (torch.tensor([2] + list(2 + torch.tensor(x).cumsum(0)), dtype=torch.int32, device=DEV) for x in (lens, lk))
    out, lse = attention.flash_fwd(q, k, v, cq, ck, longest, scale, causal)
    rq, rk, rv = (t.float().requires_grad_(True) for t in (q, k, v))
    ref = R.varlen_attention(rq, rk, rv, cq, scale, causal, ck)
    ref.backward(go.float())
    for bound in (longest, 300):
        grads = attention.flash_bwd(go, q, k, v, out, lse, cq, bound, scale, cu_k=ck, max_k=max(bound, 128), causal=causal)
        native.read_status(q.device)
        for got, want in zip(grads, (rq.grad, rk.grad, rv.grad)):
            # bf16 rounds P, dS and the result; queries, keys and values of no sequence have a gradient of zero
            assert (got.float() - want).abs().max() <= 3e-2 * want.abs().max() + 2e-2


@pytest.mark.parametrize("T,I", [(1, 8), (57, 776), (1535, 8192), (1536, 8192)])
def test_swiglu_vectors_a_thread(T, I):
    """The smallest call, ragged last blocks, and both sides of the size from which a thread takes two vectors."""
    torch.manual_seed(81)
    gu, g = _bf16(T, 2 * I), _bf16(T, I)
    x = gu.clone().requires_grad_(True)
    y = F.swiglu(x)
    dx, = torch.autograd.grad(y, x, g)
    a, b = gu.double().chunk(2, -1)
    s = torch.sigmoid(a)
    # one bf16 rounding of the result; the exponential is good to 2^-21 of its argument
    assert torch.allclose(y.double(), a * s * b, rtol=2 ** -8, atol=1e-5)
    want = torch.cat([g.double() * b * (s + a * s * (1 - s)), g.double() * a * s], -1)
    assert torch.allclose(dx.double(), want, rtol=2 ** -8, atol=1e-5)


@pytest.mark.parametrize("M", [148, 149, 256])
@pytest.mark.parametrize("N,K", [(4096, 256), (4100, 320), (5120, 1032), (8192, 64)])
def test_skinny_residual_norm_rows_that_share_an_sm(M, N, K):
    torch.manual_seed(82)
    x, w, res, nw = _bf16(M, K), _bf16(N, K, scale=0.05), _bf16(M, N), _bf16(N)
    y, r = F.skinny_linear_residual_rmsnorm(x, w, res, nw, 1e-6)
    native.read_status(x.device)
    want = x.double() @ w.double().t() + res.double()
    assert torch.allclose(r.double(), want, rtol=2 ** -8, atol=1e-4 * math.sqrt(K))       # fp32 sums, rounded once to bf16
    h = r.double()                                                                        # the norm sees what is stored
    assert torch.allclose(y.double(), h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * nw.double(), rtol=2 ** -8,
                          atol=1e-6)


@pytest.mark.parametrize("h", [2, 40])                              # an SM for every tile of queries, and fewer
def test_flash_attention_running_maximum_in_both_forms(h):
    """Scores that grow along the keys by more than the maximum may lag, so the accumulator is rescaled in every key block."""
    from cosmos_rl_b200.ops import attention
    torch.manual_seed(83)
    L, d = 700, 128
    q = torch.ones(L, h, d, device=DEV).to(torch.bfloat16)
    k = (torch.linspace(0, 40, L, device=DEV)[:, None, None] + torch.zeros(L, h, d, device=DEV)).to(torch.bfloat16)
    v = _bf16(L, h, d)
    cu = torch.tensor([0, L], dtype=torch.int32, device=DEV)
    assert ((L + 127) // 128 * h <= native.num_sms(0)) == (h == 2)
    for causal in (True, False):
        out, lse = attention.flash_fwd(q, k, v, cu, cu, L, 1.0 / math.sqrt(d), causal)
        native.read_status(q.device)
        ref, ref_lse = R.varlen_attention(q.float(), k.float(), v.float(), cu, 1.0 / math.sqrt(d), causal, return_lse=True)
        assert torch.allclose(out.float(), ref, atol=2e-2, rtol=2e-2)      # bf16 result and probabilities
        assert torch.allclose(lse, ref_lse, atol=1e-2, rtol=1e-4)


def test_few_sms_in_the_first_call_do_not_bind_the_later_ones():
    """How many CTA pairs run at once is the device's affair: a process whose first product leaves SMs to other streams gets
    all of them in the next call, whose tiles then leave pairs idle and want scratch to be cut."""
    code = """
import torch
from cosmos_rl_b200.ops import native
L, st = native.lib(), native.status_word(torch.device("cuda", 0))
def call(M, N, K, sms):
    a, b = (torch.randn(n, K, device="cuda").to(torch.bfloat16) for n in (M, N))
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    return L.b200_gemm_bf16_ws(a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, K, K, N, 0, 0, 0, 0, None, 0, 0, 0, 0, 1, None, 0,
                               st.data_ptr(), sms, native.stream())
assert call(256, 2048, 512, 8) == 0
assert call(100, 4096, 8192, native.num_sms(0)) == native.NEED_WORKSPACE
torch.cuda.synchronize()
native.read_status(st.device)
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_gemm_scratch_is_what_the_call_uses(monkeypatch):
    """A call that is not cut takes no scratch, one that is takes the room of its shares, and where that cannot be had the
    tiles stay whole."""
    torch.manual_seed(84)
    N, K = 3840, 4104
    a, b, buf = _bf16(1300, K), _bf16(N, K), torch.empty(1300, N + 8, dtype=torch.bfloat16, device=DEV)
    ref = a.double() @ b.double().t()
    native.status_word(a.device)

    def check(out):
        native.read_status(a.device)
        # one rounding to bf16 and fp32 sums of K products
        assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -20 * a.double().norm(dim=1, keepdim=True)
                * b.double().norm(dim=1) + 1e-5).all()

    def taken(out, path):
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        F.gemm(a, b, out=out, path=path)
        return torch.cuda.max_memory_allocated() - before
    tiles, pairs = 6 * 15, native.num_sms(0) // 2
    shares = tiles % pairs * (pairs // (tiles % pairs))
    # four bytes a value of each share of 256 x 256; single CTAs; rows that do not start on 16-byte boundaries
    for out, path, want in ((buf[:, :N], 0, shares * 256 * 256 * 4), (buf[:, :N], 1, 0), (buf[:, 1:N + 1], 0, 0)):
        assert want <= taken(out, path) <= want * 17 // 16          # a kept block of up to 1 MB more is not split
        check(out)

    def no_room(*args, **kwargs):
        raise torch.cuda.OutOfMemoryError("no room for scratch")
    buf.zero_()
    monkeypatch.setattr(torch, "empty", no_room)
    F.gemm(a, b, out=buf[:, :N])
    monkeypatch.undo()
    check(buf[:, :N])


# all columns in one share, single CTAs (129 to 255 columns, not cut), several shares, tiles of 128 columns in several and in one
@pytest.mark.parametrize("M,N,K", [(100, 4096, 512), (128, 520, 256), (7, 184, 504), (77, 4096, 8192), (16, 104, 4096),
                                   (5, 72, 200)])
def test_gemm_few_rows_added_to_bf16_are_rounded_once(M, N, K):
    """Sums of whole numbers, which fp32 holds exactly: what was there and the product make one bf16 value with one rounding."""
    torch.manual_seed(85)
    a, b = (torch.randint(-3, 4, (n, K), device=DEV).to(torch.bfloat16) for n in (M, N))
    out = (torch.randn(M, N, device=DEV) * 16).to(torch.bfloat16)
    want = (out.float() + a.float() @ b.float().t()).to(torch.bfloat16)
    F.gemm(a, b, out=out, accumulate=True)
    native.read_status(a.device)
    assert torch.equal(out, want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N", [(300, 4096), (264, 1032)])
def test_gemm_cut_tiles_added_from_two_streams(dtype, M, N):
    """Products of small whole numbers that two streams add to one result at the same time: no addend is lost, in tiles that
    are cut as in those that are not, and every sum is exact in either type."""
    torch.manual_seed(86)
    K, times = 8192, 8
    a, b = ((torch.rand(n, K, device=DEV) < 1 / 64).to(torch.bfloat16) for n in (M, N))
    want = a.float() @ b.float().t()
    assert want.max() * 2 * times <= 256
    assert F._gemm_scratch(M, N, K, False, True, dtype == torch.float32, True, False, False, 0, native.num_sms(0)) > 0
    out = torch.zeros(M, N, dtype=dtype, device=DEV)
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(times):
        for s in streams:
            with torch.cuda.stream(s):
                F.gemm(a, b, out=out, accumulate=True)
    torch.cuda.synchronize()
    native.read_status(a.device)
    assert torch.equal(out.float(), 2 * times * want)


# columns that end inside 16 bytes: fewer than those; several tiles; one tile of 128 columns; few rows; tiles that are cut; SwiGLU,
# whose result has half of the columns
@pytest.mark.parametrize("M,N,K,swiglu", [(200, 5, 192, False), (300, 1001, 200, False), (130, 99, 128, False),
                                          (64, 1002, 128, False), (1300, 3843, 4104, False), (300, 2002, 200, True)])
@pytest.mark.parametrize("dtype,accumulate", [(torch.bfloat16, False), (torch.bfloat16, True), (torch.float32, False),
                                              (torch.float32, True)])
def test_gemm_leaves_the_values_beside_its_result(M, N, K, swiglu, dtype, accumulate):
    if swiglu and (accumulate or dtype == torch.float32):
        pytest.skip("the SwiGLU epilogue writes bf16 and does not add")
    torch.manual_seed(87)
    a, b = _bf16(M, K), _bf16(N, K)
    bias = None if swiglu else _bf16(N)                            # keeps few rows on the CTA pairs, too
    cols = N // 2 if swiglu else N
    buf = torch.randn(M + 1, (cols + 7) // 8 * 8 + 8, device=DEV).to(dtype)
    before = buf.clone()
    F.gemm(a, b, out=buf[:M, :cols], accumulate=accumulate, bias=bias, swiglu=swiglu)
    native.read_status(a.device)
    assert torch.equal(buf[:, cols:], before[:, cols:]) and torch.equal(buf[M], before[M])
    h = a.double() @ b.double().t()
    ref = torch.nn.functional.silu(h[:, :cols]) * h[:, cols:] if swiglu else h + bias.double()
    # fp32 sums of K products (through the gate's slope of at most 1.1, times the other factor), and for bf16 one rounding of
    # the product and one of the sum with what was there
    size = a.double().norm(dim=1, keepdim=True) * b.double().norm(dim=1)
    bound = 2.0 ** -20 * (size[:, :cols] * h[:, cols:].abs() * 1.1 + size[:, cols:] * h[:, :cols].abs() if swiglu else size) + 1e-5
    if dtype == torch.bfloat16:
        bound = bound + 2.0 ** -8 * ref.abs()
    if accumulate:
        ref = ref + before[:M, :cols].double()
        bound = bound + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22) * ref.abs()
    assert ((buf[:M, :cols].double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("M,N,K", [(1, 5, 64), (33, 1001, 256), (130, 4099, 128), (256, 20003, 64)])
def test_skinny_leaves_the_values_beside_its_result(M, N, K):
    """Columns that end inside 16 bytes, in rows with a stride of their own (too short a contraction to be split)."""
    torch.manual_seed(88)
    x, w, bias = _bf16(M, K), _bf16(N, K), _bf16(N)
    assert native.lib().b200_gemm_skinny_splits(M, N, K, 0, native.num_sms(0)) == 1
    buf = _bf16(M + 1, (N + 7) // 8 * 8 + 8)
    before = buf.clone()
    F.gemm_skinny(x, w, bias=bias, out=buf[:M, :N])
    native.read_status(x.device)
    assert torch.equal(buf[:, N:], before[:, N:]) and torch.equal(buf[M], before[M])
    ref = x.double() @ w.double().t() + bias.double()
    # one rounding to bf16 and fp32 sums of K products
    bound = 2.0 ** -8 * ref.abs() + 2.0 ** -20 * x.double().norm(dim=1, keepdim=True) * w.double().norm(dim=1) + 1e-5
    assert ((buf[:M, :N].double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("B,hq,hkv,length", [(256, 7, 1, 130), (40, 32, 8, 600), (80, 4, 2, 1)])
def test_paged_decode_many_equal_sequences(B, hq, hkv, length):
    """More items than SMs and nothing to sort: the items come in the order of the sequences."""
    torch.manual_seed(89)
    per = (length + 127) // 128
    table = torch.randperm(B * per).int().view(B, per)
    cache, q = _bf16(B * per, 2, hkv, 128, 128), _bf16(B, hq, 128)
    lens = torch.full((B,), length, dtype=torch.int32)
    out = F.paged_decode(q, cache, table.cuda(), lens.cuda(), v_transposed=True)
    native.read_status(q.device)
    ref = R.paged_decode(q.cpu(), cache.cpu(), table, lens, v_transposed=True)
    # probabilities and the result are rounded to bf16 (2^-9 each)
    assert (out.cpu().float() - ref.float()).norm() <= 2.0 ** -7 * ref.float().norm()
    assert (out.cpu().float() - ref.float()).abs().max() <= 2.0 ** -6 * ref.float().abs().max()


@pytest.mark.parametrize("I", [8, 248, 256, 264, 1536])
def test_moe_swiglu_bwd_rows(I):
    """The backward between the experts' projections: a vector less and more than a warp's 32, rows of padding, and tiles past the
    last one in use, which stay as they are."""
    torch.manual_seed(85)
    rows, used, k = 512, 256, 2
    h1, dact = _bf16(rows, 2 * I), _bf16(rows, I)
    probs = torch.rand(rows, device=DEV)
    live = torch.rand(rows, device=DEV) < 0.7
    src = torch.where(live, torch.randperm(rows, device=DEV), -1).to(torch.int32)
    info = torch.stack([src, torch.where(live, probs, 0.).view(torch.int32)], dim=1).contiguous()
    h1[:used][~live[:used]] = float("nan")                       # what padding holds must not show
    dh1, ap = (torch.full((rows, n), 7., dtype=torch.bfloat16, device=DEV) for n in (2 * I, I))
    dprob = torch.full((rows,), 7., device=DEV)
    n_tiles = torch.tensor([used // 128], dtype=torch.int32, device=DEV)
    native.check(native.lib().b200_moe_swiglu_bwd(native.ptr(dact), native.ptr(h1), native.ptr(info), native.ptr(n_tiles),
                                                  native.ptr(dh1), native.ptr(ap), native.ptr(dprob), rows, I,
                                                  native.stream()), "moe_swiglu_bwd")
    torch.cuda.synchronize()
    gu = h1[:used].double().requires_grad_(True)
    act = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
    p, d, on = probs[:used, None].double(), dact[:used].double(), live[:used, None]
    want, = torch.autograd.grad(torch.where(on, act, 0.), gu, p * d)
    want, act = torch.where(on, want, 0.), torch.where(on, act.detach(), 0.)
    # one rounding to bf16; the factors in fp32 with the fast exponential (2 ulp, and its argument's rounding)
    assert torch.allclose(dh1[:used].double(), want, rtol=2 ** -8, atol=1e-5)
    assert torch.allclose(ap[:used].double(), p * act, rtol=2 ** -8, atol=1e-5)
    at = src[:used][live[:used]].long()
    ref = (act * d).sum(-1)[live[:used]]
    # I fp32 products with a rounding of 2^-20 each at most
    assert ((dprob[at].double() - ref).abs() <= 2 ** -20 * (act * d).abs().sum(-1)[live[:used]] + 1e-6).all()
    assert (dh1[used:] == 7).all() and (ap[used:] == 7).all() and (dprob == 7).sum() == rows - at.numel()


@pytest.mark.parametrize("T,E,k", [(1, 2, 2), (16, 33, 1), (17, 256, 8), (4099, 16, 8)])
def test_moe_router_counts(T, E, k):
    """Choices counted a block at a time: one token, a full block, one more, and experts that every block has."""
    from cosmos_rl_b200.ops import moe
    torch.manual_seed(86)
    logits = torch.randn(T, E, device=DEV)
    counts = torch.full((E,), 5, dtype=torch.int32, device=DEV)      # added to
    p, i = moe.route_topk(logits, k, False, counts)
    pr, ir = torch.softmax(logits.double(), -1).topk(k, dim=-1)
    assert torch.equal(i.long(), ir)
    assert torch.allclose(p.double(), pr, rtol=2 ** -19, atol=1e-30)   # the exponential's argument is good to 2^-22 of up to 8
    assert torch.equal(counts.long() - 5, torch.bincount(ir.flatten(), minlength=E))


@pytest.mark.parametrize("counts", [(0, 1, 64, 65), (128, 63, 129, 320)])
@pytest.mark.parametrize("pairs", [False, True])
def test_expert_weight_gradients_of_filled_rows(counts, pairs):
    """Blocks of 64 rows past an expert's last one are not contracted over, whatever they hold, in both forms of the kernel."""
    torch.manual_seed(87)
    N, K, E = (2048, 2560, 4) if pairs else (136, 264, 4)
    off = [0]
    for c in counts:
        off.append(off[-1] + -(-c // 128) * 128)
    Mp = max(off[-1], 320 * E if pairs else 128)                     # the room decides which form it is
    dy, x = _bf16(Mp, N), _bf16(Mp, K)
    for e, c in enumerate(counts):
        last = off[e] + -(-c // 64) * 64
        dy[off[e] + c:last] = x[off[e] + c:last] = 0
        dy[last:off[e + 1]] = x[last:off[e + 1]] = float("nan")
    out = torch.full((E, N, K), 7., dtype=torch.bfloat16, device=DEV)
    offsets, filled = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in (off, counts))
    sms = native.num_sms(0)
    assert native.lib().b200_grouped_wgrad_pairs(Mp, N, K, E, 0, 0, sms) == int(pairs)
    native.check(native.lib().b200_grouped_wgrad_filled(native.ptr(dy), native.ptr(x), native.ptr(out), Mp, N, K, E, N, K,
                                                        native.ptr(offsets), native.ptr(filled), 0, 0,
                                                        native.ptr(native.status_word(dy.device)), sms, native.stream()),
                 "grouped_wgrad")
    native.read_status(dy.device)
    for e, c in enumerate(counts):
        a, b = dy[off[e]:off[e] + c].double(), x[off[e]:off[e] + c].double()
        # one rounding to bf16 and fp32 sums of c products
        bound = 2.0 ** -8 * (a.t() @ b).abs() + 2.0 ** -20 * a.norm(dim=0)[:, None] * b.norm(dim=0) + 1e-6
        assert ((out[e].double() - a.t() @ b).abs() <= bound).all(), e


def test_flash_attention_backward_items_without_keys_between_others():
    """CTAs take items one after the other and fetch the next one's rows early: items without a key block, of one and of several,
    last blocks of 2 and 60 rows, in one call of more items than there are SMs."""
    from cosmos_rl_b200.ops import attention
    torch.manual_seed(88)
    d, hq, hkv, lens_q, lens_k = 128, 28, 4, [300, 130, 700, 1], [200, 0, 64, 129]
    cu_q, cu_k = (torch.tensor([0] + n, dtype=torch.int32, device=DEV).cumsum(0).to(torch.int32) for n in (lens_q, lens_k))
    q, k, v = _bf16(sum(lens_q), hq, d), _bf16(sum(lens_k), hkv, d), _bf16(sum(lens_k), hkv, d)
    go, scale = _bf16(*q.shape), 1 / math.sqrt(d)
    out, lse = attention.flash_fwd(q, k, v, cu_q, cu_k, max(lens_q), scale, False)
    got = attention.flash_bwd(go, q, k, v, out, lse, cu_q, max(lens_q), scale, cu_k=cu_k, max_k=max(lens_k), causal=False)
    native.read_status(q.device)
    ref_in = [t.float().requires_grad_(True) for t in (q, k, v)]
    ref = R.varlen_attention(*ref_in, cu_q, scale, False, cu_k)
    want = torch.autograd.grad(ref, ref_in, go.float())
    for g, w in zip(got, want):   # P and dS are rounded to bf16 (2^-9 each) on the way, the result once more
        assert (g.float() - w).norm() <= 4 * 2 ** -9 * w.norm()
        assert (g.float() - w).abs().max() <= 2e-2 * w.abs().max()


@pytest.mark.parametrize("T,V,H", [(1, 40009, 64), (128, 1500, 136), (129, 257, 64), (256, 40009, 72), (300, 20001, 64), (777, 255, 64)])
def test_fused_logprob_ranges(T, V, H):
    """Rows around the tiles of both forms; a vocabulary with fewer tiles than CTAs, with more, and with a last tile of one column;
    a CTA pair whose ranges belong to two row blocks."""
    torch.manual_seed(89)
    h, w = _bf16(T, H), _bf16(V, H, scale=0.3)
    labels = torch.randint(0, V, (T,), device=DEV)
    labels[-1], labels[0] = V - 1, -100 if T > 1 else 0
    lp, ent = F.fused_logprob(h, w, labels, 0.8)
    native.read_status(h.device)
    logits = h.double() @ w.double().t() / 0.8
    lse = logits.logsumexp(-1)
    want = torch.where(labels >= 0, logits.gather(-1, labels.clamp_min(0)[:, None])[:, 0] - lse, 0.)
    want_ent = lse - ((logits - lse[:, None]).exp() * logits).sum(-1)
    # a logit is an fp32 sum of H products; the sums over the vocabulary are relative to their largest term
    logit = 2.0 ** -20 * (h.double().norm(dim=1) * w.double().norm(dim=1).max()) / 0.8
    assert ((lp.double() - want).abs() <= 2 * logit + 1e-5 * (1 + lse.abs())).all()
    assert ((ent.double() - want_ent).abs() <= (2 + logits.abs().amax(-1)) * (2 * logit + 1e-5)).all()


@pytest.mark.parametrize("H", [1032, 4096, 4104, 8192])
@pytest.mark.parametrize("T,residual", [(1, True), (2, False), (593, True), (1187, False), (2380, True)])
def test_rms_norm_backward_rows_through_a_ring(T, H, residual):
    """Fewer rows than stages, one row left of a pair, as many pairs as CTAs and one more, several times round the ring; a whole row
    of threads and one vector more."""
    torch.manual_seed(90)
    x, w = _bf16(T, H).requires_grad_(True), _bf16(H).requires_grad_(True)
    res = _bf16(T, H) if residual else None
    y, total = F.rms_norm(x, w, 1e-6, residual=res)
    dy, dres = _bf16(T, H), _bf16(T, H)
    dx, dw = torch.autograd.grad([y, total] if residual else [y], [x, w], [dy, dres] if residual else [dy])
    h = (total if residual else x).detach().double().requires_grad_(True)
    wd = w.detach().double().requires_grad_(True)
    ref = h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * wd
    want, want_w = torch.autograd.grad(ref, [h, wd], dy.double())
    if residual:
        want = want + dres.double()
    # one rounding to bf16; sums of H (rows: T) fp32 products in between
    assert ((dx.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -16 * dy.double().norm(dim=1, keepdim=True)).all()
    assert ((dw.double() - want_w).abs() <= 2 ** -8 * want_w.abs() + 2 ** -18 * T ** 0.5 * dy.double().norm(dim=0)).all()


@pytest.mark.parametrize("M", [1, 129])
@pytest.mark.parametrize("N,K,pad", [(136, 64, 0), (1032, 1024, 8), (1032, 1032, 0), (264, 1000, 4)])
def test_skinny_short_contractions(M, N, K, pad):
    """Up to 16 blocks in one kernel, one value more in two; rows that only the second kernel can write."""
    torch.manual_seed(91)
    x, w, bias = _bf16(M, K), _bf16(N, K, scale=0.1), _bf16(N)
    buf = torch.full((M, N + pad), 7., dtype=torch.bfloat16, device=DEV)
    F.gemm_skinny(x, w, bias=bias, out=buf[:, :N])
    native.read_status(x.device)
    ref = x.double() @ w.double().t() + bias.double()
    # one rounding to bf16, fp32 sums of K products
    bound = 2.0 ** -8 * ref.abs() + 2.0 ** -20 * x.double().norm(dim=1, keepdim=True) * w.double().norm(dim=1) + 1e-6
    assert ((buf[:, :N].double() - ref).abs() <= bound).all() and (buf[:, N:] == 7).all()


@pytest.mark.parametrize("M", [5, 100, 300])
def test_swiglu_epilogues_of_special_gates(M):
    """Gates whose exponential overflows, zeros, infinities and NaN beside ordinary ones, in the tiles of few, some and many rows."""
    special = torch.tensor([0., -0., 1., -1., 20., -20., -85.5, -86., -86.5, -88., -88.75, -100., -3e38, 3e38, 1e38, float("inf"),
                            float("-inf"), float("nan"), 1e-38, -1e-38], device=DEV)
    torch.manual_seed(92)
    I, K = 264, 64
    gates = torch.randn(I, device=DEV) * 8
    gates[:len(special)] = special
    gates[150:150 + len(special)] = special.flip(0)
    x, w = torch.zeros(M, K, dtype=torch.bfloat16, device=DEV), torch.zeros(2 * I, K, dtype=torch.bfloat16, device=DEV)
    x[:, 0], w[:I, 0], w[I:, 0] = 1., gates.to(torch.bfloat16), torch.randn(I, device=DEV).to(torch.bfloat16)
    got = F.skinny_gate_up_swiglu(x, w) if M <= 256 else F.gemm(x, w, swiglu=True)
    native.read_status(x.device)
    g, u = w[:I, 0].float(), w[I:, 0].float()
    want = (g / (1 + torch.exp(-g)) * u).to(torch.bfloat16)
    bad = torch.isnan(g) | torch.isinf(g)
    assert torch.equal(torch.isnan(got[:, bad]), torch.isnan(want[bad]).expand(M, -1))
    assert torch.equal(torch.isinf(got), torch.isinf(want).expand(M, -1))
    ok = torch.isfinite(want)
    # __expf is good to 2^-21 of a result of up to 2^6 in its exponent; one rounding to bf16
    assert torch.allclose(got[:, ok].float(), want[ok].float().expand(M, -1), rtol=2 ** -7, atol=1e-30)


@pytest.mark.parametrize("M,H,I", [(512, 64, 8), (513, 264, 136), (700, 256, 1000), (1100, 4104, 1160), (640, 3584, 2432)])
def test_gated_mlp_matches_its_separate_passes(M, H, I):
    """Blocks of 128 and 32 columns that end early, a last row block of one row, last rounds that are cut and that are not; gradients
    new and added to."""
    torch.manual_seed(93)
    x = _bf16(M, H).requires_grad_(True)
    wg, wd = _bf16(2 * I, H, scale=0.05).requires_grad_(True), _bf16(H, I, scale=0.05).requires_grad_(True)
    dy, before = _bf16(M, H), _bf16(2 * I, H)
    y = F.gated_mlp(x, wg, wd)
    assert "GatedMLP" in type(y.grad_fn).__name__
    wg.grad = before.clone()
    y.backward(dy)
    native.read_status(x.device)
    got = [y.detach(), x.grad, wg.grad, wd.grad]
    xs, ws, ds = (t.detach().clone().requires_grad_(True) for t in (x, wg, wd))
    ws.grad = before.clone()
    z = F.linear_tc(F.swiglu(F.linear_tc(xs, ws)), ds)
    z.backward(dy)
    native.read_status(x.device)
    for a, b in zip(got, (z.detach(), xs.grad, ws.grad, ds.grad)):
        # the same roundings; sums of cut tiles in another order turn some of them, and what follows sums over those
        assert (a.float() - b.float()).norm() <= 2 ** -8 * b.float().norm()
    # one side of the gradients at a time
    for needs in ((True, False, False), (False, True, False), (False, False, True)):
        ins = [t.detach().clone().requires_grad_(n) for t, n in zip((x, wg, wd), needs)]
        F.gated_mlp(*ins).backward(dy)
        for t, n, ref in zip(ins, needs, (xs.grad, None, ds.grad)):
            assert (t.grad is not None) == n
            if n and ref is not None:
                assert (t.grad.float() - ref.float()).norm() <= 2 ** -8 * ref.float().norm()
    native.read_status(x.device)


def test_gated_mlp_without_room_for_scratch(monkeypatch):
    """Shares of a last round need scratch; without it the round stays whole."""
    from cosmos_rl_b200.ops import functional
    torch.manual_seed(94)
    M, H, I = 600, 4096, 3840
    assert native.host().b200_gemm_gated_scratch(M, I, H, False, native.num_sms(0)) > 0
    x, wg, wd = _bf16(M, H).requires_grad_(True), _bf16(2 * I, H, scale=0.02), _bf16(H, I, scale=0.02)
    dy, outs = _bf16(M, H), []
    for room in (True, False):
        if not room:
            monkeypatch.setattr(functional, "_gated_workspace", lambda *a: (None, 0))
        y = F.gated_mlp(x, wg, wd)
        outs.append((y.detach(), torch.autograd.grad(y, x, dy)[0]))
        native.read_status(x.device)
    for a, b in zip(*outs):
        assert (a.float() - b.float()).norm() <= 2 ** -8 * b.float().norm()


@pytest.mark.parametrize("T,hq,hkv,d", [(1, 1, 1, 16), (7, 3, 1, 48), (593, 4, 2, 128), (1184, 62, 5, 128), (601, 2, 1, 512)])
def test_rope_rows_in_place_and_into_a_new_tensor(T, hq, hkv, d):
    """One token a CTA and two, a token left over, tokens of one part and of two; the backward's new tensor has the rotated columns of
    the in-place form and the values as they were."""
    torch.manual_seed(95)
    qkv, pos = _bf16(T, (hq + 2 * hkv) * d), torch.randint(0, 40000, (T,), device=DEV)
    for back in (False, True):
        inplace = qkv.clone()
        F._rope_qkv_native(inplace, pos, hq, hkv, d, 1e6, back)
        new = native.host().rope_qkv_new(qkv, pos, hq, hkv, d, 1e6, back, native.stream())
        assert torch.equal(new, inplace) and torch.equal(new[:, (hq + hkv) * d:], qkv[:, (hq + hkv) * d:])
        inv = 1e6 ** (-torch.arange(0, d, 2, device=DEV, dtype=torch.float64) / d)
        ang = pos.double()[:, None] * inv * (-1 if back else 1)
        x = qkv[:, :(hq + hkv) * d].double().view(T, hq + hkv, d)
        a, b, c, s = x[..., :d // 2], x[..., d // 2:], ang.cos()[:, None], ang.sin()[:, None]
        want = torch.cat([a * c - b * s, b * c + a * s], dim=-1)
        # angles of up to 40000 with an fp32 rounding and a power good to 2 ulp: 40000 * 2^-22; one rounding to bf16
        size = torch.cat([(a.square() + b.square()).sqrt()] * 2, dim=-1)
        assert ((new[:, :(hq + hkv) * d].double().view_as(want) - want).abs() <= 2 ** -8 * want.abs() + 40000 * 2.0 ** -22 * size).all()
    for bad in (qkv[:, ::2], qkv[:, :-1], qkv[:, 1:]):
        assert native.host().rope_qkv_new(bad, pos, hq, hkv, d, 1e6, True, native.stream()) is None


@pytest.mark.parametrize("T,E,k", [(1, 8, 8), (40, 16, 8), (17, 33, 2), (33, 128, 8), (16, 256, 1)])
@pytest.mark.parametrize("renorm", [False, True])
def test_moe_router_of_logits_that_are_not_numbers(T, E, k, renorm):
    """Rows that hold NaN or infinities, all over or here and there: k experts that exist, none twice, all of them counted, and
    weights that show it. What the other rows get does not change."""
    from cosmos_rl_b200.ops import moe
    torch.manual_seed(96)
    logits = torch.randn(T, E, device=DEV)
    plain_p, plain_i = moe.route_topk(logits, k, renorm)
    bad = torch.arange(T, device=DEV) % 5 != 4
    kinds = torch.arange(T, device=DEV) % 5
    logits[kinds == 0] = float("nan")
    logits[kinds == 1, E - 1] = float("nan")
    logits[kinds == 2] = float("-inf")
    logits[kinds == 3, 0] = float("inf")
    counts = torch.zeros(E, dtype=torch.int32, device=DEV)
    p, i = moe.route_topk(logits, k, renorm, counts)
    torch.cuda.synchronize()
    assert int(i.min()) >= 0 and int(i.max()) < E
    assert (i.sort(dim=-1).values.diff(dim=-1) > 0).all()
    assert torch.equal(counts.long(), torch.bincount(i.flatten().long(), minlength=E)) and int(counts.sum()) == T * k
    assert torch.isnan(p[bad]).all()
    assert torch.equal(p[~bad], plain_p[~bad]) and torch.equal(i[~bad], plain_i[~bad])


@pytest.mark.parametrize("M", [8, 511, 512, 1000])
def test_gated_mlp_refuses_a_contraction_of_two_lengths(M):
    """Activations that are wider or narrower than the weight raise, on either side of the rows that take the fused form."""
    w_gate_up, w_down = _bf16(96, 64).requires_grad_(True), _bf16(64, 48)
    for width in (56, 72):
        with pytest.raises(AssertionError):
            F.gated_mlp(_bf16(M, width), w_gate_up, w_down)


@pytest.mark.parametrize("shape", [(1, 600), (2, 3, 100), (600,)])
def test_gated_mlp_result_may_be_changed_in_place(shape):
    """Activations of any number of dimensions; what comes back is no view, which autograd would not let a caller change."""
    torch.manual_seed(97)
    x, wg, wd = _bf16(*shape, 64).requires_grad_(True), _bf16(96, 64, scale=0.1), _bf16(64, 48, scale=0.1)
    y = F.gated_mlp(x, wg, wd)
    assert "GatedMLP" in type(y.grad_fn).__name__ and y.shape == x.shape
    before = y.detach().clone()
    y.mul_(2.0)
    dx, = torch.autograd.grad(y, x, torch.ones_like(y))
    x2 = x.detach().reshape(-1, 64).requires_grad_(True)
    z = F.gated_mlp(x2, wg, wd)
    want, = torch.autograd.grad(z, x2, torch.full_like(z, 2.0))
    assert torch.equal(before.view_as(z), z) and torch.equal(dx.view_as(want), want)


def test_gated_mlp_backward_holds_no_more_than_its_separate_passes():
    """What the activation's gradient was formed from is given back before the gate/up projection's gradients are formed."""
    torch.manual_seed(98)
    M, H, I = 2048, 2048, 4096
    x, wg, wd = _bf16(M, H).requires_grad_(True), _bf16(2 * I, H, scale=0.02).requires_grad_(True), _bf16(H, I, scale=0.02).requires_grad_(True)
    dy = _bf16(M, H)

    def peak(fn):
        for _ in range(2):      # the second time with what the first keeps
            y = fn()
            torch.cuda.synchronize()
            before = torch.cuda.memory_allocated()
            torch.cuda.reset_peak_memory_stats()
            grads = torch.autograd.grad(y, (x, wg, wd), dy)
            most = torch.cuda.max_memory_allocated() - before
            del y, grads
        return most

    separate = peak(lambda: F.linear_tc(F.swiglu(F.linear_tc(x, wg)), wd))
    fused = peak(lambda: F.gated_mlp(x, wg, wd))
    scratch = 4 * native.host().b200_gemm_gated_scratch(M, I, H, True, native.num_sms(0))
    assert scratch < 2 * M * I and fused <= separate + scratch      # one row of I values more a token would show


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
@pytest.mark.parametrize("H", [3584, 8192])
def test_rms_norm_backward_on_a_second_gpu(H):
    grads = []
    torch.manual_seed(99)
    host = [torch.randn(n, H).to(torch.bfloat16) for n in (5, 1, 5)]
    for dev in (0, 1):
        with torch.cuda.device(dev):
            x, w, dy = (t.to(f"cuda:{dev}") for t in host)
            x, w = x.requires_grad_(True), w[0].requires_grad_(True)
            grads.append([g.cpu() for g in torch.autograd.grad(F.rms_norm(x, w)[0], [x, w], dy)])
    assert all(torch.equal(a, b) for a, b in zip(*grads))


@pytest.mark.parametrize("T,V,H", [(1, 20001, 64), (129, 20001, 136), (300, 65539, 64), (777, 16387, 72), (1100, 1031, 64)])
def test_fused_logprob_gradients_of_a_ragged_vocabulary(monkeypatch, T, V, H):
    """A vocabulary that is no multiple of 8: the logit gradients' rows start on 16 bytes all the same, so both products take this
    library's GEMM, in one chunk of few rows and in several of many."""
    calls, real = [], F.gemm

    def gemm(a, b, **kw):
        calls.append(a.stride(0))
        return real(a, b, **kw)

    monkeypatch.setattr(F, "gemm", gemm)
    torch.manual_seed(100)
    h, w = _bf16(T, H).requires_grad_(True), _bf16(V, H, scale=0.3).requires_grad_(True)
    labels, g, ge = torch.randint(0, V, (T,), device=DEV), torch.randn(T, device=DEV), torch.randn(T, device=DEV) * 0.1
    labels[0] = V - 1
    lp, ent = F.fused_logprob(h, w, labels, 1.0)
    got = torch.autograd.grad([lp, ent], [h, w], [g, ge])
    native.read_status(h.device)
    assert len(calls) == 2 * -(-V // F._dlogits_chunk(T, V)) and all(s % 8 == 0 for s in calls)
    hd, wd = h.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    logp = torch.log_softmax(hd @ wd.t(), -1)
    want = torch.autograd.grad([logp.gather(-1, labels[:, None])[:, 0], -(logp.exp() * logp).sum(-1)], [hd, wd], [g.double(), ge.double()])
    for a, b in zip(got, want):     # the logits' gradient is rounded to bf16 (2^-9), and the result once more
        assert (a.double() - b).norm() <= 2 ** -7 * b.norm()


@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("T,V,H,ranges", [(129, 40009, 64, 7), (300, 20001, 72, 79), (1153, 1025, 64, 5), (513, 3000, 136, 1), (2100, 9000, 64, 20)])
def test_fused_logprob_row_blocks_and_ranges(monkeypatch, pairs, T, V, H, ranges):
    """Both forms on several row blocks: ranges of unequal length, one range, a range a tile, more units than CTAs, and a last row
    block of one row."""
    monkeypatch.setattr(F, "_logprob_form", lambda *a: (ranges, pairs))
    torch.manual_seed(101)
    h, w = _bf16(T, H), _bf16(V, H, scale=0.3)
    labels = torch.randint(0, V, (T,), device=DEV)
    labels[-1], labels[0] = V - 1, -100
    lp, ent = F.fused_logprob(h, w, labels, 1.0)
    native.read_status(h.device)
    logits = h.double() @ w.double().t()
    lse = logits.logsumexp(-1)
    want = torch.where(labels >= 0, logits.gather(-1, labels.clamp_min(0)[:, None])[:, 0] - lse, 0.)
    want_ent = lse - ((logits - lse[:, None]).exp() * logits).sum(-1)
    # a logit is an fp32 sum of H products; the sums over the vocabulary are relative to their largest term
    logit = 2.0 ** -20 * (h.double().norm(dim=1) * w.double().norm(dim=1).max())
    assert ((lp.double() - want).abs() <= 2 * logit + 1e-5 * (1 + lse.abs())).all()
    assert ((ent.double() - want_ent).abs() <= (2 + logits.abs().amax(-1)) * (2 * logit + 1e-5)).all()


def _same_bits(a, b):
    nan = torch.isnan(b)
    return torch.equal(torch.isnan(a), nan) and torch.equal(a.view(torch.int16)[~nan], b.view(torch.int16)[~nan])


def _all_gates(M, H=64):
    """Activations and a fused weight whose gates are all the bf16 values there are, beside random ups, without a rounding."""
    torch.manual_seed(102)
    gates = torch.arange(1 << 16, device=DEV).to(torch.int32).to(torch.int16).view(torch.bfloat16)
    I = len(gates)
    x, w = torch.zeros(M, H, dtype=torch.bfloat16, device=DEV), torch.zeros(2 * I, H, dtype=torch.bfloat16, device=DEV)
    x[:, 0], w[:I, 0], w[I:, 0] = 1.0, gates, _bf16(I)
    return x, w, I


@pytest.mark.parametrize("M", [1, 5, 100, 200, 300])
def test_swiglu_epilogues_have_the_divisions_bits(M):
    """Every bf16 gate, infinities and NaN among them, in the epilogues of inference: what the pass over stored values makes of it,
    which divides. (A product's zeros have no sign.)"""
    x, w, I = _all_gates(M)
    want = F.swiglu(w[:, 0][None] + 0.0).expand(M, -1)
    got = F.skinny_gate_up_swiglu(x, w) if M <= 256 else F.gemm(x, w, swiglu=True)
    native.read_status(x.device)
    assert _same_bits(got, want.contiguous())


def test_gated_mlp_epilogues_have_the_bits_of_the_passes():
    """Every bf16 gate in training, and gates so small that they are stored as zeros of both signs, where nothing is cut: stored
    values, activation and gradients are those of the separate passes."""
    M = 300
    x, w, I = _all_gates(M)
    x[1::2, 0], w[:I][w[:I, 0].abs() < 2.0 ** -60] = 2.0 ** -70, -2.0 ** -66
    w_down, dy = _bf16(64, I), _bf16(M, 64)
    H, st, sms = native.host(), native.status_word(x.device), native.num_sms(0)
    assert not H.b200_gemm_gated_scratch(M, I, 64, False, sms) and not H.b200_gemm_gated_scratch(M, I, 64, True, sms)
    gu, act, dgu = (torch.empty(M, n, dtype=torch.bfloat16, device=DEV) for n in (2 * I, I, 2 * I))
    native.check(H.b200_gemm_gate_up(x, w, gu, act, M, I, 64, 64, 64, None, 0, st, sms, native.stream()), "gate_up")
    native.check(H.b200_gemm_dgate_up(dy, w_down, gu, dgu, M, I, 64, 64, I, None, 0, st, sms, native.stream()), "dgate_up")
    native.read_status(x.device)
    want_gu = F.gemm(x, w)
    assert ((want_gu[1, :I] == 0) & torch.signbit(want_gu[1, :I])).any()
    dact = F.gemm(dy, w_down, b_mn=True)
    want = native.tensors(H.swiglu_bwd(dact, want_gu, native.stream()), "swiglu_bwd")
    assert _same_bits(gu, want_gu) and _same_bits(act, F.swiglu(want_gu)) and _same_bits(dgu, want)


def test_expert_swiglu_backward_has_the_bits_of_its_pass():
    """Every bf16 gate between the experts' projections: with weights of one, the gradients of the pass that divides."""
    rows = 128
    _, w, I = _all_gates(1)
    h1, dact = w[:, 0][None].expand(rows, -1).contiguous(), _bf16(rows, I)
    info = torch.stack([torch.arange(rows, device=DEV, dtype=torch.int32), torch.ones(rows, device=DEV).view(torch.int32)], 1).contiguous()
    dh1, ap, dprob = torch.empty_like(h1), torch.empty_like(dact), torch.empty(rows, device=DEV)
    n_tiles = torch.ones(1, dtype=torch.int32, device=DEV)
    native.check(native.host().b200_moe_swiglu_bwd(dact, h1, info, n_tiles, dh1, ap, dprob, rows, I, native.stream()), "moe_swiglu_bwd")
    want = native.tensors(native.host().swiglu_bwd(dact, h1, native.stream()), "swiglu_bwd")
    torch.cuda.synchronize()
    assert _same_bits(dh1, want)


@pytest.mark.parametrize("T,hq,hkv,d", [(5, 2, 1, 128), (601, 4, 2, 64)])
def test_rope_gradients_in_rows_apart_and_expanded(T, hq, hkv, d):
    """The new tensor of the backward from rows that are further apart than they are long, that share one row's memory, or that start
    off the 16-byte grid or lie in columns, which are copied first."""
    torch.manual_seed(103)
    n, pos = (hq + 2 * hkv) * d, torch.arange(T, device=DEV) * 7
    qkv = _bf16(T, n).requires_grad_(True)
    wide, row = _bf16(T, n + 24), _bf16(1, n)
    for g in (wide[:, 8:8 + n], wide[:, 16:16 + n], row.expand(T, -1), wide[:, 3:3 + n], _bf16(n, T).t()):
        z = F.rope_qkv_(qkv * 1.0, pos, hq, hkv, d, 1e6)
        dx, = torch.autograd.grad(z, qkv, g)
        want = g.clone(memory_format=torch.contiguous_format)
        F._rope_qkv_native(want, pos, hq, hkv, d, 1e6, True)
        assert torch.equal(dx, want) and dx.is_contiguous()
    taken = [native.host().rope_qkv_new(g, pos, hq, hkv, d, 1e6, True, native.stream()) is not None
             for g in (wide[:, 8:8 + n], row.expand(T, -1), wide[:, 3:3 + n], _bf16(n, T).t())]
    assert taken == [True, True, False, False]
