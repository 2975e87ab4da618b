"""tcgen05 flash attention against the explicit fp32 attention of the oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(q, k, v, B, S, H, Hkv, hd):
    from parameter_golf_b200.ops.reference import causal_gqa_attention
    return causal_gqa_attention(q.float().reshape(B, S, H, hd), k.float().reshape(B, S, Hkv, hd), v.float().reshape(B, S, Hkv, hd)).reshape(B * S, H * hd)


def _ref_lse(q, k, B, S, H, Hkv, hd):
    qf = q.float().reshape(B, S, H, hd).permute(0, 2, 1, 3)
    kf = k.float().reshape(B, S, Hkv, hd).permute(0, 2, 1, 3).repeat_interleave(H // Hkv, 1)
    s = qf @ kf.transpose(-1, -2) / hd ** 0.5
    s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=q.device).tril(), float("-inf"))
    return torch.logsumexp(s, -1)


@pytest.mark.parametrize("B,S,H,Hkv", [(1, 128, 2, 1), (2, 256, 4, 2), (1, 640, 8, 4), (3, 384, 2, 2), (1, 1024, 4, 1)])
def test_attention_forward(B, S, H, Hkv):
    from parameter_golf_b200.ops import native as n
    hd = 64
    torch.manual_seed(S + H)
    qkv = (torch.randn(B * S, (H + 2 * Hkv) * hd, device="cuda") * 1.5).bfloat16()       # strided views of one packed buffer
    q, k, v = qkv[:, :H * hd], qkv[:, H * hd:(H + Hkv) * hd], qkv[:, (H + Hkv) * hd:]
    y = torch.zeros(B * S, H * hd, device="cuda", dtype=torch.bfloat16)
    lse = n.attn_fwd(q, k, v, y, B, S, H, Hkv, hd)
    torch.cuda.synchronize()
    n.check_status()
    ref = _ref(q, k, v, B, S, H, Hkv, hd)
    assert (y.float() - ref).abs().max() < 0.04, (y.float() - ref).abs().max()      # one bf16 ulp of an output in [4, 8) is 0.031
    lse_nat = -lse * 0.6931471805599453               # the kernel stores -(log2-domain lse), the form its backward consumes
    assert (lse_nat - _ref_lse(q, k, B, S, H, Hkv, hd)).abs().max().item() < 0.02


@pytest.mark.parametrize("B,S,H,Hkv", [(2, 256, 4, 2), (1, 640, 8, 4), (3, 128, 2, 2)])
def test_attention_forward_with_exclusive_self_attention_output(B, S, H, Hkv):
    """The optional second output: y with its component along the token's own value vector removed, from the same kernel."""
    from parameter_golf_b200.ops import native as n
    from parameter_golf_b200.ops import reference as R
    hd = 64
    torch.manual_seed(S + 7 * H)
    qkv = (torch.randn(B * S, (H + 2 * Hkv) * hd, device="cuda") * 1.5).bfloat16()
    q, k, v = qkv[:, :H * hd], qkv[:, H * hd:(H + Hkv) * hd], qkv[:, (H + Hkv) * hd:]
    y = torch.zeros(B * S, H * hd, device="cuda", dtype=torch.bfloat16)
    z = torch.zeros_like(y)
    n.attn_fwd(q, k, v, y, B, S, H, Hkv, hd, z=z, xsa_eps=1e-8)
    torch.cuda.synchronize()
    n.check_status()
    ref = _ref(q, k, v, B, S, H, Hkv, hd)
    assert (y.float() - ref).abs().max() < 0.04
    z_ref = R.xsa(ref.reshape(B, S, H, hd), v.float().reshape(B, S, Hkv, hd)).reshape(B * S, H * hd)
    assert (z.float() - z_ref).abs().max() < 0.04, (z.float() - z_ref).abs().max()
    # z is orthogonal to the value vector of its KV group
    zz = z.float().reshape(B * S, Hkv, H // Hkv, hd)
    vv = torch.nn.functional.normalize(v.float().reshape(B * S, Hkv, 1, hd), dim=-1)
    assert (zz * vv).sum(-1).abs().max() < 0.12


def test_attention_forward_large_scores_trigger_rescale():
    """Scores that keep growing along the sequence force the lazy rescale of the accumulator."""
    from parameter_golf_b200.ops import native as n
    B, S, H, Hkv, hd = 1, 512, 2, 1, 64
    torch.manual_seed(0)
    q = torch.randn(B * S, H * hd, device="cuda")
    k = torch.randn(B * S, Hkv * hd, device="cuda") * torch.linspace(0.5, 12.0, S, device="cuda")[:, None]
    v = torch.randn(B * S, Hkv * hd, device="cuda")
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    y = torch.empty(B * S, H * hd, device="cuda", dtype=torch.bfloat16)
    n.attn_fwd(q, k, v, y, B, S, H, Hkv, hd)
    torch.cuda.synchronize()
    n.check_status()
    assert (y.float() - _ref(q, k, v, B, S, H, Hkv, hd)).abs().max() < 0.05


@pytest.mark.parametrize("reproducible", [False, True])
@pytest.mark.parametrize("B,S,H,Hkv", [(1, 128, 2, 1), (2, 256, 4, 2), (1, 640, 8, 4), (2, 384, 2, 2), (1, 512, 4, 1), (3, 896, 4, 2)])
def test_attention_backward(B, S, H, Hkv, reproducible):
    from parameter_golf_b200.ops import native as n
    from parameter_golf_b200.ops.reference import causal_gqa_attention
    hd = 64
    torch.manual_seed(S * 3 + H)
    qkv = (torch.randn(B * S, (H + 2 * Hkv) * hd, device="cuda") * 1.2).bfloat16()
    q, k, v = qkv[:, :H * hd], qkv[:, H * hd:(H + Hkv) * hd], qkv[:, (H + Hkv) * hd:]
    dy = (torch.randn(B * S, H * hd, device="cuda") * 0.5).bfloat16()
    y = torch.empty(B * S, H * hd, device="cuda", dtype=torch.bfloat16)
    lse = n.attn_fwd(q, k, v, y, B, S, H, Hkv, hd)
    dqkv = torch.zeros_like(qkv)
    dq, dk, dv = dqkv[:, :H * hd], dqkv[:, H * hd:(H + Hkv) * hd], dqkv[:, (H + Hkv) * hd:]
    base = (torch.randn(B * S, Hkv * hd, device="cuda") * 0.1).bfloat16()
    dv.copy_(base)
    n.attn_bwd(q, k, v, y, dy, lse, dq, dk, dv, B, S, H, Hkv, hd, accumulate_dv=True, reproducible=reproducible)
    torch.cuda.synchronize()
    n.check_status()
    qf = q.float().reshape(B, S, H, hd).requires_grad_(True)
    kf = k.float().reshape(B, S, Hkv, hd).requires_grad_(True)
    vf = v.float().reshape(B, S, Hkv, hd).requires_grad_(True)
    out = causal_gqa_attention(qf, kf, vf)
    gq, gk, gv = torch.autograd.grad(out, (qf, kf, vf), dy.float().reshape(B, S, H, hd))
    for name, got, ref in (("dq", dq, gq.reshape(B * S, -1)), ("dk", dk, gk.reshape(B * S, -1)), ("dv", dv.float() - base.float(), gv.reshape(B * S, -1))):
        err = (got.float() - ref).abs().max().item()
        scale = ref.abs().max().item()
        assert err < 0.03 * scale + 0.02, (name, err, scale)


def test_attention_backward_single_pass_many_tiles_and_clean_scratch():
    """More CTA-level items than SMs (several items per persistent CTA, both K/V buffers and every Q/dO stage reused),
    checked against the two-kernel form; the shared accumulator must be left zero, and a second call must agree."""
    from parameter_golf_b200.ops import native as n
    B, S, H, Hkv, hd = 10, 1024, 8, 4, 64
    torch.manual_seed(7)
    qkv = torch.randn(B * S, (H + 2 * Hkv) * hd, device="cuda").bfloat16()
    q, k, v = qkv[:, :H * hd], qkv[:, H * hd:(H + Hkv) * hd], qkv[:, (H + Hkv) * hd:]
    dy = (torch.randn(B * S, H * hd, device="cuda") * 0.5).bfloat16()
    y = torch.empty(B * S, H * hd, device="cuda", dtype=torch.bfloat16)
    lse = n.attn_fwd(q, k, v, y, B, S, H, Hkv, hd)
    ref = [torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)]
    n.attn_bwd(q, k, v, y, dy, lse, *ref, B, S, H, Hkv, hd, reproducible=True)
    acc = n.attn_dq_scratch(q.device, B, S, H, hd)
    for _ in range(2):
        got = [torch.full_like(q, 7.0), torch.full_like(k, 7.0), torch.full_like(v, 7.0)]
        n.attn_bwd(q, k, v, y, dy, lse, *got, B, S, H, Hkv, hd)
        torch.cuda.synchronize()
        n.check_status()
        assert float(acc.abs().max()) == 0.0
        for g, r in zip(got, ref):
            err = (g.float() - r.float()).abs().max().item()
            assert err <= 0.01 * r.float().abs().max().item() + 1e-3, err


@pytest.mark.parametrize("B,S,H,Hkv,rope", [(1, 128, 2, 1, 16), (2, 2048, 8, 4, 16), (3, 1920, 8, 4, 0), (1, 640, 4, 1, 64), (9, 1024, 8, 4, 32), (5, 384, 3, 3, 16)])
def test_attention_backward_through_norm_and_rope_in_one_call(B, S, H, Hkv, rope):
    """The combined backward (fp32 query accumulator straight into the norm / rotation backward, last round of key tiles split over the
    SMs) against the two-kernel attention backward followed by the row kernel. The split's dK/dV sums are fp32 in CTA order, so two
    calls agree bit for bit in the value columns; bf16 intermediates of the reference path bound the difference (2^-8 of the largest)."""
    from parameter_golf_b200.ops import native as n, reference as R
    C = n.load()
    hd, T, eps = 64, B * S, 1e-6
    d, kv = H * hd, Hkv * hd
    torch.manual_seed(S + H + rope)
    pre = torch.randn(T, d + 2 * kv, device="cuda").bfloat16()
    post = torch.zeros_like(pre)
    gain = torch.rand(H, device="cuda") + 0.75
    cos = sin = None
    if rope:
        cos, sin = (t.contiguous() for t in R.rope_tables(S, rope, 10000.0, device="cuda"))
    C.qk_norm_rope_fwd(pre, post, cos, sin, gain, H, Hkv, hd, rope, S, eps)
    q, k, v = post[:, :d], post[:, d:d + kv], pre[:, d + kv:]
    y, dy = torch.empty(T, d, device="cuda", dtype=torch.bfloat16), (torch.randn(T, d, device="cuda") * 0.5).bfloat16()
    lse = n.attn_fwd(q, k, v, y, B, S, H, Hkv, hd)
    base = (torch.randn(T, kv, device="cuda") * 0.1).bfloat16()
    dsum = torch.empty(B, H, S, device="cuda")

    ref, ref_gain, tmp = torch.empty_like(pre), torch.zeros(H, device="cuda"), torch.zeros_like(pre)
    ref[:, d + kv:] = base
    n.attn_bwd(q, k, v, y, dy, lse, tmp[:, :d], tmp[:, d:d + kv], ref[:, d + kv:], B, S, H, Hkv, hd, accumulate_dv=True, reproducible=True)
    C.qk_norm_rope_bwd(tmp, pre, ref, cos, sin, gain, ref_gain, H, Hkv, hd, rope, S, eps)

    acc = torch.zeros(B * H * S * hd, device="cuda")
    outs = []
    for _ in range(2):
        got, d_gain, d_post = torch.full_like(pre, 7.0), torch.zeros(H, device="cuda"), torch.full_like(pre, 7.0)
        got[:, d + kv:] = base
        C.attn_bwd_qk(post, pre, y, dy, lse, dsum, acc, d_post, got, cos, sin, gain, d_gain, B, S, H, Hkv, rope, eps, True, n.status_word(pre.device),
                      False, n.attn_bwd_part(pre.device))
        torch.cuda.synchronize()
        n.check_status()
        assert float(acc.abs().max()) == 0.0
        outs.append(got)
        for lo, hi in ((0, d), (d, d + kv), (d + kv, d + 2 * kv)):
            r = ref[:, lo:hi].float()
            assert (got[:, lo:hi].float() - r).abs().max() <= 0.012 * r.abs().max() + 1e-3, (lo, hi)
        assert (d_gain - ref_gain).abs().max() <= 0.01 * ref_gain.abs().max() + 0.05
    assert torch.equal(outs[0][:, d:], outs[1][:, d:])


@pytest.mark.parametrize("B,S,H,Hkv", [(3, 128, 2, 1), (6, 1280, 2, 1), (9, 1920, 8, 4), (24, 2048, 8, 4)])
def test_a_sequence_has_the_same_attention_alone_and_in_a_batch(B, S, H, Hkv):
    """The forward of a sequence does not depend on how many are handed over beside it: outputs and log-sum-exp bit for bit."""
    from parameter_golf_b200.ops import native as n
    hd = 64
    torch.manual_seed(S + B)
    q = torch.randn(B * S, H * hd, device="cuda").bfloat16()
    k, v = (torch.randn(B * S, Hkv * hd, device="cuda").bfloat16() for _ in range(2))
    y, z = torch.full_like(q, 7.0), torch.full_like(q, 7.0)
    lse = n.attn_fwd(q, k, v, y, B, S, H, Hkv, hd, None, z)
    for b in (0, B - 1):
        r = slice(b * S, (b + 1) * S)
        y1, z1 = torch.full_like(q[r], 7.0), torch.full_like(q[r], 7.0)
        lse1 = n.attn_fwd(q[r], k[r], v[r], y1, 1, S, H, Hkv, hd, None, z1)
        torch.cuda.synchronize()
        n.check_status()
        assert torch.equal(y1, y[r]) and torch.equal(z1, z[r]) and torch.equal(lse1[0], lse[b]), b


@pytest.mark.parametrize("B,S,H,Hkv,merged", [(37, 128, 4, 4, False), (1, 512, 2, 1, True), (3, 1920, 8, 4, True)])
def test_launch_count_of_the_backward_is_the_number_of_its_kernels(B, S, H, Hkv, merged):
    """The single-pass backward launches its merge kernel only where a round of key tiles is split (148 items of one tile are a whole
    round): the count follows what ran, with and without the first kernel."""
    from torch.profiler import ProfilerActivity, profile
    from parameter_golf_b200.ops import native as n
    hd = 64
    torch.manual_seed(S)
    q, dy = (torch.randn(B * S, H * hd, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B * S, Hkv * hd, device="cuda").bfloat16() for _ in range(2))
    y, dq, dk, dv = torch.empty_like(q), torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    lse = n.attn_fwd(q, k, v, y, B, S, H, Hkv, hd)
    dsum = n.attn_bwd(q, k, v, y, dy, lse, dq, dk, dv, B, S, H, Hkv, hd)
    for ready in (False, True):
        torch.cuda.synchronize()
        before = n.launch_count()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            n.attn_bwd(q, k, v, y, dy, lse, dq, dk, dv, B, S, H, Hkv, hd, dsum=dsum, dsum_ready=ready)
            torch.cuda.synchronize()
        names = [e.name for e in prof.events() if "attn_bwd" in e.name]
        assert n.launch_count() - before == len(names), names
        assert any("merge" in x for x in names) == merged and any("prep" in x for x in names) != ready
