"""GPTQ row kernel against the float32 restatement of the same algorithm."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(rows, cols, seed):
    torch.manual_seed(seed)
    X = torch.randn(4 * cols, cols, device="cuda") * torch.linspace(0.3, 2.0, cols, device="cuda")
    X = X + 0.5 * X.roll(1, dims=1)                                   # correlated inputs: off-diagonal Hessian mass
    H = X.t() @ X / X.shape[0]
    W = torch.randn(rows, cols, device="cuda") * 0.05
    W[:, 3] *= 6.0                                                    # a few heavy columns so that clipping matters
    return W, H


@pytest.mark.parametrize("rows,cols,bits", [(64, 512, 6), (37, 384, 6), (16, 1536, 5), (8, 200, 6)])
def test_gptq_rows_matches_reference(rows, cols, bits):
    from parameter_golf_b200.ops import native as n
    from parameter_golf_b200.quant.gptq import gptq_prepare, gptq_rows_torch
    W, H = _problem(rows, cols, rows + cols)
    perm, inv_perm, U = gptq_prepare(H)
    Wp = W[:, perm].contiguous()
    qmax = (1 << (bits - 1)) - 1
    scale = (Wp.abs().amax(1) / qmax).clamp_min(1e-8)
    want = gptq_rows_torch(Wp, U, scale, bits)
    got = n.gptq_rows(Wp, U, scale, bits)
    torch.cuda.synchronize()
    assert got.dtype == torch.int8 and got.shape == want.shape
    assert int(got.min()) >= -(qmax + 1) and int(got.max()) <= qmax
    diff = (got.int() - want.int()).abs()
    assert diff.max() <= 1                                              # only rounding-boundary flips from summation order
    assert (diff > 0).float().mean() < 0.01

    def loss(Q):                                                        # the objective GPTQ minimises: tr(E H E^T)
        E = (Wp - Q.float() * scale[:, None]).double()
        Hp = H[perm][:, perm].double()
        return torch.einsum("rc,cd,rd->", E, Hp, E).item()

    assert abs(loss(got) - loss(want)) <= 0.01 * loss(want)
    rtn = (Wp / scale[:, None]).round().clamp(-(qmax + 1), qmax)
    assert loss(got) < loss(rtn)                                        # error feedback beats round-to-nearest


def test_gptq_quantize_uses_the_kernel_on_cuda_tensors():
    from parameter_golf_b200.ops import native as n
    from parameter_golf_b200.quant.gptq import gptq_quantize, gptq_rows_torch
    W, H = _problem(48, 512, 5)
    before = n.launch_count()
    q, s = gptq_quantize(W, H, bits=6)
    assert n.launch_count() - before == 5                               # one launch per clip candidate
    q_ref, s_ref = gptq_quantize(W, H, bits=6, rows_fn=gptq_rows_torch)
    assert torch.allclose(s, s_ref)
    assert ((q.int() - q_ref.int()).abs() > 0).float().mean() < 0.01


@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 127), (5, 129), (4, 256), (6, 390), (9, 1288)])
def test_gptq_rows_at_the_edges_of_its_blocks(rows, cols):
    """Row counts around the four rows of a CTA and column counts around the 128-column blocks (one ragged block, a whole one, a
    one-column rest, widths off 16 bytes): the codes of the float32 statement up to rounding-boundary flips, which the summation
    order of the trailing update can cause and which then propagate through that row alone."""
    from parameter_golf_b200.ops import native as n
    from parameter_golf_b200.quant.gptq import gptq_prepare, gptq_rows_torch
    W, H = _problem(rows, cols, 7 * rows + cols)
    perm, _, U = gptq_prepare(H)
    Wp = W[:, perm].contiguous()
    scale = (Wp.abs().amax(1) / 31).clamp_min(1e-8)
    want, got = gptq_rows_torch(Wp, U, scale, 6), n.gptq_rows(Wp, U, scale, 6)
    diff = (got.int() - want.int()).abs()
    assert diff.max() <= 1 and int((diff > 0).sum()) <= max(2, rows * cols // 100)


def test_gptq_prepare_gives_the_upper_factor_of_the_inverse():
    from parameter_golf_b200.quant.gptq import damp_hessian, gptq_prepare
    _, H = _problem(4, 192, 11)
    perm, inv_perm, U = gptq_prepare(H)
    Hp = damp_hessian(H)[perm][:, perm].double()
    want = torch.linalg.cholesky(torch.cholesky_inverse(torch.linalg.cholesky(Hp)), upper=True)
    assert torch.equal(perm[inv_perm], torch.arange(192, device=perm.device)) and float(U.tril(-1).abs().max()) == 0.0
    assert float((U.double() - want).norm() / want.norm()) < 1e-6          # one rounding to fp32: 2^-24 per element


@pytest.mark.parametrize("rows,cols", [(7, 129), (150, 256), (700, 384), (1100, 200), (130, 2600)])
def test_gptq_rows_of_several_candidates_are_those_of_one_at_a_time(rows, cols):
    """One launch over (candidate, row) pairs, in the small form and in the large one (row counts around a CTA's 4 to 20 rows, one and
    two rounds, columns off 16 bytes), gives the codes of one launch per candidate: the arithmetic of a row is the same."""
    from parameter_golf_b200.ops import native as n
    from parameter_golf_b200.quant.gptq import gptq_prepare
    W, H = _problem(rows, cols, rows + cols)
    perm, _, U = gptq_prepare(H)
    Wp = W[:, perm].contiguous()
    scales = torch.stack([(Wp.abs().amax(1) * f / 31).clamp_min(1e-8) for f in (1.0, 0.9, 0.8, 0.7, 0.6)])
    got = n.gptq_rows(Wp, U, scales, 6)
    for k in range(5):
        want = torch.cat([n.gptq_rows(Wp[i:i + 500], U, scales[k, i:i + 500], 6) for i in range(0, rows, 500)])
        assert torch.equal(got[k], want), k


def test_gptq_rows_outside_the_range_of_the_short_division():
    """Infinite, overflowing, tiny and undefined quotients give the codes of the general division: the limits, zero, and the lowest code
    for NaN, in both divisions of a column (the second through a diagonal far from one)."""
    from parameter_golf_b200.ops import native as n
    inf, nan = float("inf"), float("nan")
    w = torch.tensor([inf, -inf, 3e38, -3e38, nan, 0.0, -0.0, 1e-45, 2.5, -2.5, 2.4999998], device="cuda")
    s = torch.tensor([1.0, 1.0, 6e-8, 6e-8, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0], device="cuda")
    for copies in (1, 80):                                                   # the small form and the large one
        got = n.gptq_rows(w.repeat(copies)[:, None], torch.ones(1, 1, device="cuda"), s.repeat(copies), 6)
        assert got[:, 0].reshape(copies, -1).eq(torch.tensor([31, -32, 31, -32, -32, 0, 0, 0, 3, -3, 2], dtype=torch.int8, device="cuda")).all()
    # column 2 receives -err * u with err = 0.25 / diagonal: exact powers of two, so the code is known
    for e in (-100, -70, -60, -59, 0, 59, 60, 61, 100):
        U = torch.tensor([[2.0 ** e, 2.0 ** (e + 6)], [0.0, 1.0]], device="cuda")
        got = n.gptq_rows(torch.tensor([[1.25, 0.0]], device="cuda"), U, torch.ones(1, device="cuda"), 6)
        assert got.tolist() == [[1, -16]], e


@pytest.mark.parametrize("bits", [5, 6, 8])
@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 127), (2000, 128), (500, 37)])
def test_gptq_codes_of_one_block_are_those_of_the_float32_statement(rows, cols, bits):
    """Without a trailing update there is no sum whose order could differ: every code equals the reference's, with weights on and
    next to the ties of the rounding (half-precision scales, as the export has them)."""
    from parameter_golf_b200.ops import native as n
    from parameter_golf_b200.quant.gptq import gptq_prepare, gptq_rows_torch
    W, H = _problem(rows, cols, rows + cols + bits)
    perm, _, U = gptq_prepare(H)
    Wp = W[:, perm].contiguous()
    scale = (Wp.abs().amax(1) / ((1 << (bits - 1)) - 1)).clamp_min(6e-8).half().float().clamp_min(6e-8)
    Wp[:, 0] = (torch.randint(-12, 12, (rows,), device="cuda") + 0.5) * scale          # a tie, and its two neighbours
    Wp[:, 0] = torch.where(torch.arange(rows, device="cuda") % 3 == 1, torch.nextafter(Wp[:, 0], torch.zeros_like(scale)), Wp[:, 0])
    Wp[:, 0] = torch.where(torch.arange(rows, device="cuda") % 3 == 2, torch.nextafter(Wp[:, 0], 9 * Wp[:, 0]), Wp[:, 0])
    assert torch.equal(n.gptq_rows(Wp, U, scale, bits), gptq_rows_torch(Wp, U, scale, bits))


@pytest.mark.parametrize("rows,cols", [(130, 200), (16000, 1100)])
def test_gptq_of_all_candidates_at_once_needs_no_more_memory_than_one_at_a_time(rows, cols):
    """The route with one launch (and its error pass, which takes a large matrix in pieces) picks the codes and scales of the route with
    a launch per candidate, and a large matrix does not need more memory by it."""
    from parameter_golf_b200.ops import native as n
    from parameter_golf_b200.quant.gptq import gptq_quantize
    W, H = _problem(rows, cols, rows + cols)
    out, peak = [], []
    for rows_fn in (n.gptq_rows, None):                       # a row function of the caller's: one candidate at a time
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        out.append(gptq_quantize(W, H, 6, rows_fn=rows_fn))
        torch.cuda.synchronize()
        peak.append(torch.cuda.max_memory_allocated() - before)
    (q0, s0), (q1, s1) = out
    same = s0 == s1                                           # two candidates' fp32 error sums can tie up to their order of summation
    assert same.float().mean() >= 0.999 and torch.equal(q0[same], q1[same])
    if rows > 1000:
        assert peak[1] <= peak[0], peak


@pytest.mark.parametrize("c", [1, 63, 64, 65, 130, 200, 513])
def test_gptq_factor_around_its_tiles(c):
    """The factor from the kernel against fp64 torch, at sizes around the 64-column tiles: both are fp64 sums rounded to fp32 once, so they
    may differ by an ulp where a rounding is close."""
    from parameter_golf_b200.quant.gptq import damp_hessian, gptq_prepare
    x = torch.randn(2 * c, c, device="cuda", generator=torch.Generator(device="cuda").manual_seed(c)) * torch.linspace(0.3, 2.0, c, device="cuda")
    H = x.t() @ x / (2 * c)
    perm, inv_perm, U = gptq_prepare(H)
    Hp = damp_hessian(H)[perm][:, perm].double()
    want = torch.linalg.cholesky(torch.linalg.inv(Hp), upper=True)
    assert (U.double() - want).norm() <= 1e-6 * want.norm()
    assert torch.equal(U, U.triu()) and torch.equal(perm[inv_perm], torch.arange(c, device="cuda"))


@pytest.mark.parametrize("c,bad", [(5, 2), (100, 70)])
def test_gptq_factor_refuses_what_is_not_positive_definite(c, bad):
    from parameter_golf_b200.quant.gptq import gptq_prepare, gptq_quantize
    for value in (-3.0, float("nan")):
        H = torch.eye(c, device="cuda")
        H[bad, bad] = value
        with pytest.raises(torch.linalg.LinAlgError, match="not positive-definite"):
            gptq_prepare(H)
        with pytest.raises(torch.linalg.LinAlgError, match="not positive-definite"):
            gptq_quantize(torch.randn(3, c, device="cuda"), H)
