"""Full-Hessian GPTQ with act-order, block error feedback and a per-row clip search.

Algorithm (``records/track_10min_16mb/2026-03-25_ValCalib_GPTQ_XSA_BigramHash3072/train_gpt.py:1104-1224``):
Hessians ``H = X^T X`` of every linear layer's input, averaged over calibration batches, 1 % mean-diagonal
damping; columns permuted by descending ``diag(H)``; ``U = chol(inv(H))`` upper; columns are quantised
left to right, the scaled error of column ``i`` is pushed into the not-yet-quantised columns through
``U[i, i:]``, block by block; five percentile clips are tried. Differences from the record, on purpose:
the integer range and rounding are the artifact's (``[-2^(b-1), 2^(b-1)-1]``, ties away from zero), and the
best clip is chosen per row (scales are per row) instead of per matrix.

Rows are independent given ``U``, which is what the CUDA kernel exploits (one warp per row and clip candidate); this file
is the torch statement of the same computation and its oracle.
"""
from __future__ import annotations

from typing import Callable, Dict, List, Optional, Tuple

import torch

from ..models.gpt import bank_views
from ..spec import RunSpec
from .quantize import CLIP_PERCENTILES, GROUPS, qrange, quantize_rows, round_half_away, scheme_bits


def damp_hessian(H: torch.Tensor, damping: float = 0.01) -> torch.Tensor:
    H = H.float().clone()
    d = torch.diagonal(H)
    dead = d == 0
    d[dead] = 1.0
    d += damping * d.mean().clamp_min(1e-6)
    return H


def gptq_prepare(H: torch.Tensor, damping: float = 0.01):
    """Return (perm, inv_perm, U) with ``U`` the upper Cholesky factor of ``inv(H[perm][:, perm])``."""
    perm, inv_perm, U, check = _prepare(H, damping)
    check()
    return perm, inv_perm, U


def _prepare(H: torch.Tensor, damping: float):
    """`gptq_prepare` and a function that raises if ``H`` was not positive definite: it waits for the device, so it is called last."""
    Hd = damp_hessian(H, damping).contiguous()
    perm = torch.argsort(torch.diagonal(Hd), descending=True)
    # inv(H) = U^T U with U upper means H = R R^T with R = inv(U) upper, and R is the Cholesky factor of H with its rows and
    # columns in reverse order, reversed back. So one factorisation and one triangular inverse give the (unique) factor; neither
    # inv(H) nor its own factorisation is needed.
    rev = perm.flip(0)
    if Hd.is_cuda:
        from ..ops import native
        U, info = native.gptq_factor(Hd, rev)
        inv_perm = torch.empty_like(perm).scatter_(0, perm, torch.arange(perm.numel(), device=perm.device))
        return perm, inv_perm, U, lambda: native.gptq_factor_check(info)
    L = torch.linalg.cholesky(Hd[rev][:, rev].double())
    eye = torch.eye(L.shape[0], dtype=L.dtype, device=L.device)
    U = torch.linalg.solve_triangular(L, eye, upper=False).flip(0, 1).float()
    return perm, torch.argsort(perm), U, lambda: None


def gptq_rows_torch(Wp: torch.Tensor, U: torch.Tensor, scales: torch.Tensor, bits: int, block: int = 128) -> torch.Tensor:
    """Quantise the (already permuted) rows ``Wp`` with fixed per-row ``scales``; returns int8 codes."""
    qmin, qmax = qrange(bits)
    rows, cols = Wp.shape
    W = Wp.clone()
    Q = torch.zeros_like(W, dtype=torch.int8)
    s = scales[:, None]
    for i1 in range(0, cols, block):
        i2 = min(i1 + block, cols)
        W1 = W[:, i1:i2].clone()
        Err = torch.zeros_like(W1)
        U1 = U[i1:i2, i1:i2]
        for i in range(i2 - i1):
            w = W1[:, i:i + 1]
            q = round_half_away(w / s).clamp_(qmin, qmax)
            Q[:, i1 + i] = q[:, 0].to(torch.int8)
            err = (w - q * s) / U1[i, i]
            W1[:, i:] -= err * U1[i:i + 1, i:]
            Err[:, i] = err[:, 0]
        if i2 < cols:
            W[:, i2:] -= Err @ U[i1:i2, i2:]
    return Q


def gptq_quantize(W: torch.Tensor, H: torch.Tensor, bits: int = 6, block: int = 128, damping: float = 0.01,
                  rows_fn: Optional[Callable] = None) -> Tuple[torch.Tensor, torch.Tensor]:
    """(q int8 [rows, cols], scale f32 [rows]). ``rows_fn`` substitutes the CUDA row kernel."""
    W = W.float()
    rows, cols = W.shape
    qmin, qmax = qrange(bits)
    perm, inv_perm, U, check = _prepare(H.to(W.device), damping)
    Wp = W[:, perm].contiguous()
    srt = W.abs().sort(dim=1).values
    native_rows = None
    if rows_fn is None:
        if W.is_cuda and block == 128:
            from ..ops import native                  # on a GPU the hand-written row kernel is the path; no silent fallback
            rows_fn = native_rows = native.gptq_rows
        else:
            rows_fn = gptq_rows_torch
    S = torch.stack([srt[:, min(int(cols * p), cols - 1)] for p in CLIP_PERCENTILES])
    S = (S.clamp_min(1e-8) / qmax).clamp_min(1e-8).half().float().clamp_min(6e-8)         # what de-quantisation will multiply by
    scales = list(S.unbind(0))
    best_err = torch.full((rows,), float("inf"), device=W.device)
    best_q = torch.zeros_like(Wp, dtype=torch.int8)
    best_s = torch.ones(rows, device=W.device)
    # All candidates from one launch once they are more rows than one round of the small kernel form holds (four per SM): 512 x 1536
    # takes 0.85 ms instead of five times 0.20. Fewer rows keep a launch per candidate, which is slower than one would be (five
    # chains one after the other): the number of launches of such a call is part of its tests. The first of the least errors wins.
    if native_rows is not None and rows * len(scales) > 4 * torch.cuda.get_device_properties(W.device).multi_processor_count:
        Q = native_rows(Wp, U, S, bits, block)
        err = torch.empty_like(S)
        step = max(1, (1 << 23) // (len(scales) * cols))      # the fp32 temporaries of the error pass stay at 100 MB
        for r0 in range(0, rows, step):
            r = slice(r0, r0 + step)
            err[:, r] = (Wp[r] - Q[:, r].float() * S[:, r, None]).pow(2).sum(2)
        err = torch.where(err < float("inf"), err, best_err)
        best_err = err.amin(0)
        order = torch.arange(len(scales), device=W.device)[:, None]
        k = torch.where(err == best_err, order, len(scales)).amin(0)
        found = best_err < float("inf")
        best_s = torch.where(found, S.gather(0, k[None])[0], best_s)
        best_q = torch.where(found[:, None], Q[k, torch.arange(rows, device=W.device)], best_q)
        check()
        return best_q[:, inv_perm].contiguous(), best_s
    for scale in scales:
        Q = rows_fn(Wp, U, scale, bits, block)
        err = (Wp - Q.float() * scale[:, None]).pow(2).sum(1)
        better = err < best_err
        best_err = torch.where(better, err, best_err)
        best_s = torch.where(better, scale, best_s)
        best_q = torch.where(better[:, None], Q, best_q)
    check()
    return best_q[:, inv_perm].contiguous(), best_s


class HessianTaps:
    """Accumulates ``X^T X`` of the inputs of every linear layer, keyed ``(layer, site)`` with site in
    ``qkv | o | up | down``; plugged into the oracle forward through ``block_forward(..., taps=...)``."""

    def __init__(self):
        self.H: Dict[Tuple[int, str], torch.Tensor] = {}
        self.batches = 0

    def add(self, layer: int, site: str, x: torch.Tensor):
        x = x.detach().reshape(-1, x.shape[-1]).float()
        h = x.t() @ x
        key = (layer, site)
        if key in self.H:
            self.H[key] += h
        else:
            self.H[key] = h

    def finish(self) -> Dict[Tuple[int, str], torch.Tensor]:
        n = max(self.batches, 1)
        return {k: v / n for k, v in self.H.items()}


GROUP_SITES = {"qo_bank.q": "qkv", "kv_bank.k": "qkv", "kv_bank.v": "qkv", "qo_bank.o": "o", "mlp_up_bank": "up", "mlp_down_bank": "down"}


def gptq_quantize_model(spec: RunSpec, params: Dict[str, torch.Tensor], hessians: Dict[Tuple[int, str], torch.Tensor],
                        rows_fn: Optional[Callable] = None, device=None) -> Dict[str, Tuple[torch.Tensor, torch.Tensor]]:
    """Quantise every bank group layer by layer with its Hessian; ``tok_emb`` uses the plain clip search.
    Returns the ``precomputed`` map accepted by `export_model`."""
    m, q = spec.model, spec.quant
    bits = scheme_bits(q.scheme, q.matrix_bits, q.embed_bits)
    views = bank_views(m, params)
    out = {}
    for g in GROUPS:
        W = views[g].detach().float()
        if device is not None:
            W = W.to(device)
        if g == "tok_emb":
            qq, ss = (W.half(), torch.ones(W.shape[0])) if bits[g] == 16 else quantize_rows(W, bits[g])     # 16: the table stays fp16
            out[g] = (qq.cpu(), ss.cpu())
            continue
        per = W.shape[0] // m.num_layers
        qs, ss = [], []
        for i in range(m.num_layers):
            H = hessians[(i, GROUP_SITES[g])]
            qi, si = gptq_quantize(W[i * per:(i + 1) * per], H.to(W.device), bits[g], q.gptq_block_size, q.gptq_damping, rows_fn)
            qs.append(qi.cpu())
            ss.append(si.cpu())
        out[g] = (torch.cat(qs), torch.cat(ss))
    return out
