"""RMSNorm carried by the products around it: row sums of squares from one output stage, the row factor in the next."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,d,N,tile", [(1, 64, 64, 0), (130, 128, 96, 64), (300, 512, 160, 128), (257, 640, 320, 256), (5760, 512, 1536, 0)])
def test_norm_folded_into_products(M, d, N, tile):
    from parameter_golf_b200.ops import native as n
    C = n.load()
    torch.manual_seed(M + d)
    bf = lambda *s, k=1.0: (torch.randn(*s, device="cuda") * k).bfloat16()
    z, Wo, x, W, dy, Wd = bf(M, d), bf(d, d, k=d ** -0.5), bf(M, d), bf(N, d, k=d ** -0.5), bf(M, d), bf(d, N, k=d ** -0.5)
    mid, part, f = torch.empty(M, d, device="cuda", dtype=torch.bfloat16), torch.full((d // 64, M), float("nan"), device="cuda"), torch.empty(M, device="cuda")
    n.gemm(z, Wo, mid, epi=n.EPI_AXPBY_BF16, alpha=1.0, beta=1.0, aux=x, tile_n=tile, row_part=part)
    sums = mid.double().square().view(M, d // 64, 64).sum(2).t()
    assert ((part.double() - sums).abs() <= 64 * 2.0 ** -24 * sums).all()                       # 64 fp32 additions of non-negative terms
    a, h, a_ref = (torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    signs, st = torch.empty(N // 32, M, device="cuda", dtype=torch.int32), n.status_word(z.device)
    s, eps = 0.7, 1e-6
    C.gemm_act(mid, W, a, signs, 0.5, st, 0, tile, part, s, eps, f)
    want_f = s * (mid.double().square().mean(1) + eps).rsqrt()
    assert ((f.double() - want_f).abs() <= 1e-6 * want_f).all()
    h64 = (mid.double() * want_f[:, None]) @ W.double().t()
    a64 = torch.nn.functional.leaky_relu(h64, 0.5).square()
    n.gemm((mid.float() * f[:, None]).bfloat16(), W, h, epi=n.EPI_ACT_SQ, slope=0.5, D2=a_ref, tile_n=tile)      # the normed copy, rounded
    err = lambda y: (y.double() - a64).norm() / a64.norm()
    assert err(a) <= err(a_ref) + 1e-4                                  # one rounding less than with the copy
    d1, d0 = torch.empty_like(a), torch.empty_like(a)
    C.gemm_actgrad(dy, Wd, d1, a, signs, 0.5, st, 0, tile, f)
    C.gemm_actgrad(dy, Wd, d0, a, signs, 0.5, st, 0, tile)
    want = d0.double() * f.double()[:, None]
    # both are one value rounded to bf16 (at most 2^-8 relative each), one of them before the multiplication
    assert ((d1.double() - want).abs() <= 2.02 * 2.0 ** -8 * want.abs()).all()
    # norm backward from a gradient that carries the factor
    gx, gy = torch.empty_like(mid), torch.empty_like(mid)
    dn = bf(M, d)
    C.mix_norm_bwd(dn, None, mid, None, None, None, None, None, None, gx, None, None, None, None, False, s, eps)
    C.mix_norm_bwd((dn.float() * f[:, None]).bfloat16(), None, mid, None, None, None, None, None, None, gy, None, None, None, None, False, -1.0, eps)
    n.check_status()
    assert (gx.float() - gy.float()).norm() <= 0.01 * gx.float().norm()


def test_refused_forms():
    from parameter_golf_b200.ops import native as n
    C = n.load()
    z = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.bfloat16)
    part = torch.zeros(1, 64, device="cuda")
    for kw in (dict(epi=n.EPI_BF16), dict(epi=n.EPI_AXPBY_BF16, aux=z(64, 64), row=torch.zeros(2, 64, device="cuda"))):
        with pytest.raises(RuntimeError):
            n.gemm(z(64, 64), z(64, 64), z(64, 64), epi=kw["epi"], aux=kw.get("aux"), row_part=kw.get("row", part))
    with pytest.raises(RuntimeError):
        C.gemm_act(z(64, 64), z(64, 64), z(64, 64), None, 0.5, n.status_word("cuda:0"), 0, 0, torch.zeros(1, 63, device="cuda"))
