"""The MLP activation kept as its square and sign bits, against the form that keeps the pre-activation."""
import pytest
import torch


def test_activation_root():
    """Every bf16 value whose square stays in range is the root of that square rounded to bf16 (what `gemm_actgrad` relies on)."""
    t = torch.arange(0, 0x7F80, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    t = t[(t.float() > 2e-19) & (t.float() < 1.8e19)]
    assert t.numel() > 16000
    assert torch.equal((t.float() * t.float()).bfloat16().float().sqrt().bfloat16(), t)


def test_slopes_taken():
    from parameter_golf_b200.ops.native import act_root_supported
    assert all(map(act_root_supported, (0.0, 0.5, 0.25))) and not any(map(act_root_supported, (0.3, 1.0, 2.0, -0.5)))


@pytest.mark.gpu
@pytest.mark.parametrize("slope", [0.5, 0.0, 0.25])
@pytest.mark.parametrize("T,K,N,tile", [(1, 64, 64, 0), (127, 64, 96, 64), (300, 192, 160, 128), (257, 512, 1536, 256), (4096, 512, 1536, 0), (40000, 512, 1536, 128)])
def test_activation_and_gradient_equal_the_stored_preactivation(T, K, N, tile, slope):
    from parameter_golf_b200.ops import native as n
    C = n.load()
    torch.manual_seed(T + N)
    bf = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    x, W, dy, Wd = bf(T, K), bf(N, K) * 0.1, bf(T, K), bf(K, N) * 0.1
    h, a0, d0 = (torch.empty(T, N, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    n.gemm(x, W, h, epi=n.EPI_ACT_SQ, slope=slope, D2=a0, tile_n=tile)
    n.gemm(dy, Wd, d0, True, False, n.EPI_MUL_ACTGRAD, slope=slope, aux=h, tile_n=tile)
    a, d = torch.full_like(a0, float("nan")), torch.full_like(d0, float("nan"))
    signs = torch.zeros(N // 32, T, device="cuda", dtype=torch.int32)
    st = n.status_word(x.device)
    C.gemm_act(x, W, a, signs, slope, st, 0, tile)
    C.gemm_actgrad(dy, Wd, d, a, signs if slope else None, slope, st, 0, tile)
    no_signs = torch.empty_like(a)
    C.gemm_act(x, W, no_signs, None, slope, st, 0, tile)
    n.check_status()
    assert torch.equal(a, a0) and torch.equal(no_signs, a0)
    bits = (signs[:, :, None] >> torch.arange(32, device="cuda", dtype=torch.int32)) & 1
    assert torch.equal(bits.permute(1, 0, 2).reshape(T, N).bool(), torch.signbit(h))
    assert torch.equal(d, d0)


@pytest.mark.gpu
def test_refused_forms():
    from parameter_golf_b200.ops import native as n
    C = n.load()
    x, W, a = (torch.zeros(s, device="cuda", dtype=torch.bfloat16) for s in ((64, 64), (64, 64), (64, 64)))
    signs = torch.zeros(2, 64, device="cuda", dtype=torch.int32)
    for slope, sg in ((0.3, signs), (0.5, signs[:1]), (0.5, None)):
        with pytest.raises(RuntimeError):
            C.gemm_actgrad(x, W, torch.empty_like(a), a, sg, slope, n.status_word(x.device))
