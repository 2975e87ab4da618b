"""CUDA engine against the fp32 autograd oracle: row kernels, one-step loss/gradients, optimizer, short trajectory."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def small_spec(**ov):
    from parameter_golf_b200.spec import family_preset
    s = family_preset("record_11l")
    m = s.model
    m.num_layers, m.model_dim, m.num_heads, m.num_kv_heads, m.mlp_mult, m.vocab_size = 4, 128, 2, 1, 2.0, 256
    m.xsa_last_n, m.rope.dims = 2, 16
    m.bigram.vocab_size, m.bigram.dim = 96, 64
    m.train_seq_len = m.eval_seq_len = 128
    s.train.seq_len, s.train.batch_tokens, s.train.backend, s.train.world_size = 128, 4 * 128, "cuda_single", 1
    s.train.distributed_optimizer_backend = "all_reduce_replicated_muon"
    s.apply_overrides([f"{k}={v}" for k, v in ov.items()])
    return s.validate()


def oracle_grads(spec, params, ids, tgt):
    from parameter_golf_b200.models.runner import OracleRunner
    p = {k: v.double() for k, v in params.items()}
    return OracleRunner(spec.model, p).loss_and_grads(ids.long().cpu(), tgt.long().cpu())


def rel_err(a, b):
    return float((a.double().cpu() - b.double().cpu()).norm() / (b.double().cpu().norm() + 1e-12))


@pytest.mark.parametrize("variant", ["record", "baseline", "ve", "recurrence", "parallel", "attn_gate", "sparse_gate", "parallel_gate", "untied", "yarn",
                                     "full_rope"])
def test_one_step_loss_and_gradients_match_oracle(variant):
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import CudaEngine
    from parameter_golf_b200.ops import native
    ov = {}
    if variant == "baseline":
        ov = {"model.xsa_last_n": 0, "model.rope.dims": 0, "model.bigram.enabled": "false", "model.smear_gate": "false",
              "model.ln_scale": "false", "model.activation": "relu_sq"}
    if variant == "ve":
        ov = {"model.value_embedding.enabled": "true", "model.value_embedding.dim": 64, "model.value_embedding.layers": "[2,3]"}
    if variant == "recurrence":                  # layers 1 and 2 run twice; layer 1 is an encoder layer feeding a U-Net skip
        ov = {"model.recurrence.enabled": "true", "model.recurrence.start_layer": 1, "model.recurrence.repeat_layers": 2}
    if variant in ("parallel", "parallel_gate"):
        ov = {"model.parallel_residual.enabled": "true"}
    if variant == "attn_gate":
        ov = {"model.attn_out_gate.enabled": "true", "model.attn_out_gate.width": 12}
    if variant in ("sparse_gate", "parallel_gate"):
        ov.update({"model.sparse_attn_gate.enabled": "true", "model.sparse_attn_gate.width": 12, "model.sparse_attn_gate.scale": 1.5})
    if variant == "untied":
        ov = {"model.tie_embeddings": "false"}
    if variant == "yarn":                        # the frequency ramp only changes the tables the kernels are given
        ov = {"model.rope.mode": "yarn", "model.rope.yarn_max_len": 4096, "model.rope.base": 5000.0}
    if variant == "full_rope":                   # all 64 dims rotate: the widest rotary case of the QKV output stage
        ov = {"model.rope.dims": 64}
    spec = small_spec(**ov)
    params = gpt.fill_deterministic(spec.model)
    torch.manual_seed(0)
    ids = torch.randint(0, 256, (4, 128))
    tgt = torch.randint(0, 256, (4, 128))
    eng = CudaEngine(spec, params, "cuda", 4, 128)
    eng.zero_grads()
    eng.micro_step(ids.cuda().int(), tgt.cuda().int(), 1)
    torch.cuda.synchronize()
    native.check_status()
    loss = float(eng.loss_sum[0]) / eng.T
    ref_loss, ref = oracle_grads(spec, params, ids, tgt)
    assert abs(loss - float(ref_loss)) < 1e-3 * max(1.0, float(ref_loss)), (loss, float(ref_loss))       # bf16 activations: a relative bound
    worst = {}
    for k, g in ref.items():
        worst[k] = rel_err(eng.g[k], g)
    # bf16 activations/gradients vs an fp64 oracle; q_gain is one number per head summed over every token with heavy cancellation
    bad = {k: v for k, v in worst.items() if v > (0.15 if k == "q_gain" else 0.03)}
    assert not bad, worst


def test_one_step_at_the_record_width_matches_the_oracle():
    """The shapes the product runs: d = 512, 8 query / 4 KV heads, MLP 1536, vocabulary 1024, bigram table 3072 x 128,
    sequences of 2048 (three layers, two of them with XSA, two sequences). The oracle is the autograd model in fp32 on the
    GPU. This is where the 256-wide GEMM tiles with N = 1536, the two-vector row kernels and 8/4-head attention meet a
    reference; the small-shape tests select other template instances."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import CudaEngine
    from parameter_golf_b200.models.runner import OracleRunner
    from parameter_golf_b200.ops import native
    from parameter_golf_b200.spec import family_preset
    spec = family_preset("record_11l")
    spec.model.num_layers, spec.model.xsa_last_n = 3, 2
    spec.train.backend, spec.train.world_size, spec.train.seq_len, spec.train.batch_tokens = "cuda_single", 1, 2048, 2 * 2048
    spec.validate()
    params = gpt.fill_deterministic(spec.model)
    torch.manual_seed(0)
    ids = torch.randint(0, 1024, (2, 2048))
    tgt = torch.randint(0, 1024, (2, 2048))
    eng = CudaEngine(spec, params, "cuda", 2, 2048)
    eng.zero_grads()
    eng.micro_step(ids.cuda().int(), tgt.cuda().int(), 1)
    torch.cuda.synchronize()
    native.check_status()
    loss = float(eng.loss_sum[0]) / eng.T
    ref_loss, ref = OracleRunner(spec.model, {k: v.cuda().float() for k, v in params.items()}).loss_and_grads(ids.cuda(), tgt.cuda())
    assert abs(loss - float(ref_loss)) < 2e-3 * float(ref_loss), (loss, float(ref_loss))
    worst = {k: rel_err(eng.g[k], g) for k, g in ref.items()}
    assert max(worst.values()) < 0.05, worst


def test_forward_logits_and_nll_match_oracle():
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import EngineRunner
    from parameter_golf_b200.models.runner import OracleRunner
    spec = small_spec()
    params = gpt.fill_deterministic(spec.model)
    ids = torch.randint(0, 256, (3, 128))
    tgt = torch.randint(0, 256, (3, 128))
    r = EngineRunner(spec, params, "cuda", train=False)
    o = OracleRunner(spec.model, params)
    assert (r.logits(ids).cpu() - o.logits(ids)).abs().max() < 0.35
    assert (r.nll(ids, tgt).cpu() - o.nll(ids, tgt)).abs().mean().item() < 6e-2


def test_optimizer_step_matches_torch_optimizers():
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import CudaEngine
    from parameter_golf_b200.train import OracleBackend
    spec = small_spec(**{"train.grad_clip_norm": 0.3, "train.ema_decay": 0.9})
    params = gpt.fill_deterministic(spec.model)
    eng = CudaEngine(spec, params, "cuda", 4, 128)
    eng.enable_ema()
    cpu = OracleBackend(spec, {k: v.clone() for k, v in params.items()})
    torch.manual_seed(1)
    grads = {k: torch.randn_like(v) * 0.05 for k, v in params.items()}
    for k in grads:
        eng.g[k].copy_(grads[k])
    eng.set_hp(0.7, 0.93)
    eng.clip()
    eng.optimizer_step()
    torch.cuda.synchronize()
    from parameter_golf_b200.optim.muon import clip_grads_
    gl = {k: v.clone() for k, v in grads.items()}
    clip_grads_(list(gl.values()), 0.3)
    cpu.adam.step([[gl[k] for k in g["names"]] for g in cpu.adam_groups], 0.7)
    cpu.muon.step([gl[k] for k in cpu.bank_names], lr=spec.train.matrix_lr * 0.7, momentum=0.93)
    for k in params:
        upd_ref = cpu.params[k] - params[k]
        upd = eng.p[k].cpu() - params[k]
        tol = 0.08 if k in gpt.BANKS else 1e-3                  # bf16 Newton-Schulz vs fp32 Newton-Schulz
        assert rel_err(upd, upd_ref) < tol, (k, rel_err(upd, upd_ref))
    ema = eng.export_params(ema=True)
    for k in ("tok_emb", "qo_bank"):
        exp = 0.9 * params[k] + 0.1 * eng.p[k].cpu()
        assert (ema[k] - exp).abs().max() < 1e-5


def test_short_training_trajectory_tracks_oracle():
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import EngineBackend
    from parameter_golf_b200.train import OracleBackend
    spec = small_spec(**{"train.tied_embed_lr": 0.01, "train.ema_decay": 0.0})
    spec.mode = "record"
    spec.allow_unsupported_variants = True
    params = gpt.init_params(spec.model, 3)
    gpu = EngineBackend(spec, {k: v.clone() for k, v in params.items()})
    cpu = OracleBackend(spec, {k: v.clone() for k, v in params.items()})
    torch.manual_seed(2)
    lg, lc = [], []
    for step in range(6):
        ids = torch.randint(0, 256, (4, 128))
        tgt = (ids * 7 + 3) % 256                                # learnable mapping
        lg.append(gpu.train_step([(ids, tgt)], 1.0, 0.95, False))
        lc.append(cpu.train_step([(ids, tgt)], 1.0, 0.95, False))
    assert lg[-1] < lg[0] and all(abs(a - b) < 0.02 * max(1.0, abs(b)) for a, b in zip(lg, lc)), (lg, lc)


def test_cuda_graph_micro_step_matches_eager():
    """The captured forward+backward replays to the same losses and parameters as the eager launch sequence."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import EngineBackend
    res = {}
    for graph in (False, True):
        spec = small_spec(**{"train.cuda_graph": "true" if graph else "false", "train.ema_decay": 0.0})
        spec.mode = "record"
        spec.allow_unsupported_variants = True
        be = EngineBackend(spec, gpt.fill_deterministic(spec.model))
        T = be.engine.T
        gen = torch.Generator().manual_seed(5)
        losses = []
        for step in range(3):
            spans = [torch.randint(0, 256, (T + 1,), generator=gen).to(torch.int16) for _ in range(be.accum)]
            losses.append(be.train_step_spans(spans, 1.0, 0.95))
        res[graph] = (losses, {k: v.clone() for k, v in be.engine.p.items()})
    # split-K atomics make weight gradients order-dependent in their last bits and the bf16 Newton-Schulz iteration amplifies
    # that, so two eager runs differ by as much after the first update: the first loss is exact, the later ones agree loosely
    assert res[True][0][0] == pytest.approx(res[False][0][0], abs=1e-5), (res[True][0], res[False][0])
    assert res[True][0][1:] == pytest.approx(res[False][0][1:], abs=2e-2), (res[True][0], res[False][0])
    for k, v in res[False][1].items():            # Adam's normalised update flips sign on near-zero gradients: compare on average
        assert (res[True][1][k] - v).abs().mean().item() <= 2e-2 * (v.abs().mean().item() + 1e-6), k


def test_bounded_wait_times_out_and_reports():
    """A flag that nothing sets: the kernel gives up after its time limit, writes the status word and returns;
    the context stays usable."""
    from parameter_golf_b200.ops import native
    C = native.load()
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    native.status_word().zero_()
    C.comm_wait_flag(flag, 1, native.status_word())
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="wait_flag"):
        native.check_status()
    native.check_status()                                   # cleared
    flag.fill_(3)
    C.comm_wait_flag(flag, 1, native.status_word())
    torch.cuda.synchronize()
    native.check_status()
    assert float((torch.ones(4, device="cuda") * 2).sum()) == 8.0


def test_runner_shapes_share_weights_and_see_updates():
    """Two batch shapes of one runner alias the same parameters and bf16 weights: an in-place parameter change followed by
    `params_changed` is seen by both, and no engine is rebuilt when the shape alternates."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import EngineRunner
    spec = small_spec()
    params = gpt.fill_deterministic(spec.model)
    r = EngineRunner(spec, params, "cuda", train=True)
    torch.manual_seed(4)
    a_ids, a_tgt = torch.randint(0, 256, (3, 128)), torch.randint(0, 256, (3, 128))
    b_ids, b_tgt = torch.randint(0, 256, (2, 128)), torch.randint(0, 256, (2, 128))
    na0, nb0 = r.nll(a_ids, a_tgt), r.nll(b_ids, b_tgt)
    ea, eb = r.engines[(3, 128)], r.engines[(2, 128)]
    assert ea.p["tok_emb"].data_ptr() == eb.p["tok_emb"].data_ptr() and ea.Wqkv.data_ptr() == eb.Wqkv.data_ptr()
    assert torch.equal(r.nll(a_ids, a_tgt), na0) and r.engines[(3, 128)] is ea          # alternating shapes rebuilds nothing
    r.params["tok_emb"].mul_(1.5)
    r.params_changed()
    na1, nb1 = r.nll(a_ids, a_tgt), r.nll(b_ids, b_tgt)
    assert (na1 - na0).abs().max() > 1e-3 and (nb1 - nb0).abs().max() > 1e-3
    fresh = EngineRunner(spec, {k: v.clone() for k, v in r.params.items()}, "cuda", train=True)
    assert torch.allclose(fresh.nll(b_ids, b_tgt), nb1, atol=1e-5)


def test_complementary_token_weights_match_oracle():
    """Weighted-mean loss and its gradients with a [V, V] pair-weight table; scoring stays unweighted."""
    import numpy as np
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import CudaEngine
    from parameter_golf_b200.models.runner import OracleRunner
    from parameter_golf_b200.ops import complementary as comp
    from parameter_golf_b200.ops import native
    spec = small_spec()
    params = gpt.fill_deterministic(spec.model)
    torch.manual_seed(0)
    ids = torch.randint(0, 256, (4, 128))
    tgt = torch.randint(0, 256, (4, 128))
    st = comp.BigramStats(256)
    rng = np.random.default_rng(0)
    st.add_sequence(rng.integers(0, 256, 20000))
    seen = rng.random(ids.numel()) < 0.5                  # half of the (input, target) pairs of this batch are frequent bigrams
    a, b = ids.reshape(-1).numpy()[seen], tgt.reshape(-1).numpy()[seen]
    np.add.at(st.counts, (a, b), 2000)
    st.row_sums = st.counts.sum(axis=1, dtype=np.uint64)
    table = comp.weight_table(st, 0.9)
    tw = torch.from_numpy(table[ids.numpy(), tgt.numpy()])
    assert float(tw.min()) < 0.9 and float(tw.max()) == 1.0
    eng = CudaEngine(spec, params, "cuda", 4, 128)
    eng.set_token_weight_table(table)
    eng.zero_grads()
    eng.micro_step(ids.cuda().int(), tgt.cuda().int(), 1)
    torch.cuda.synchronize()
    native.check_status()
    np.testing.assert_allclose(eng.tok_w.cpu().numpy(), tw.reshape(-1).numpy(), rtol=1e-6)
    assert float(eng.w_total[0]) == pytest.approx(float(tw.sum()), rel=1e-5)
    loss = float(eng.loss_sum[0]) / eng.T
    p64 = {k: v.double() for k, v in params.items()}
    ref_loss, ref = OracleRunner(spec.model, p64).loss_and_grads(ids, tgt, token_weights=tw.double())
    assert abs(loss - float(ref_loss)) < 2e-2, (loss, float(ref_loss))
    worst = {k: rel_err(eng.g[k], g) for k, g in ref.items()}
    bad = {k: v for k, v in worst.items() if v > (0.2 if k == "q_gain" else 0.06)}
    assert not bad, worst
    # the same engine without gradients scores plain per-token losses
    eng.forward(ids.cuda().int(), tgt.cuda().int())
    plain = OracleRunner(spec.model, p64).nll(ids, tgt)
    assert float((eng.nll.view(4, 128).cpu().double() - plain).abs().mean()) < 6e-2
    eng.set_token_weight_table(None)
    eng.zero_grads()
    eng.micro_step(ids.cuda().int(), tgt.cuda().int(), 1)
    ref_loss2, _ = oracle_grads(spec, params, ids, tgt)
    assert abs(float(eng.loss_sum[0]) / eng.T - float(ref_loss2)) < 2e-2


@pytest.mark.parametrize("mode,variant", [("none", "record"), ("edges", "record"), ("recurrent", "recurrence"), ("none", "recurrence"),
                                          ("none", "parallel_gate"), ("inner", "ve")])
def test_activation_checkpointing_gives_the_same_gradients(mode, variant):
    """A block whose activations are not kept is run again inside the backward; every kernel is deterministic except the
    split-K fp32 atomics of the weight gradients, so the gradients agree with the keep-everything engine to rounding."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import CudaEngine
    from parameter_golf_b200.ops import native
    ov = {"model.num_layers": 6}
    if variant == "recurrence":
        ov.update({"model.recurrence.enabled": "true", "model.recurrence.start_layer": 1, "model.recurrence.repeat_layers": 2})
    if variant == "parallel_gate":
        ov.update({"model.parallel_residual.enabled": "true", "model.sparse_attn_gate.enabled": "true", "model.sparse_attn_gate.width": 12})
    if variant == "ve":
        ov.update({"model.value_embedding.enabled": "true", "model.value_embedding.dim": 64, "model.value_embedding.layers": "[3,5]"})
    torch.manual_seed(0)
    ids = torch.randint(0, 256, (4, 128)).cuda().int()
    tgt = torch.randint(0, 256, (4, 128)).cuda().int()
    out = {}
    for m_ in ("all", mode):
        spec = small_spec(**dict(ov, **{"train.save_layer_acts": m_}))
        params = gpt.fill_deterministic(spec.model)
        eng = CudaEngine(spec, params, "cuda", 4, 128)
        if m_ == "all":
            assert eng.nact == eng.nslots
        else:
            assert eng.nact < eng.nslots and not all(eng.saved)
        eng.zero_grads()
        eng.micro_step(ids, tgt, 1)
        torch.cuda.synchronize()
        native.check_status()
        out[m_] = (float(eng.loss_sum[0]), {k: v.clone() for k, v in eng.g.items()})
    assert out["all"][0] == pytest.approx(out[mode][0], rel=1e-6)
    worst = {k: rel_err(out[mode][1][k], g) for k, g in out["all"][1].items()}
    assert max(worst.values()) < 2e-3, worst


@pytest.mark.parametrize("mode", ["all", "none"])
def test_memory_estimate_tracks_engine_allocation(mode):
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import CudaEngine
    from parameter_golf_b200.plan import estimate_engine_memory
    spec = small_spec(**{"train.save_layer_acts": mode, "model.num_layers": 6})
    params = gpt.fill_deterministic(spec.model)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.memory_allocated()
    eng = CudaEngine(spec, params, "cuda", 16, 128)
    eng.enable_ema()
    used = torch.cuda.memory_allocated() - before
    est = estimate_engine_memory(spec, 16 * 128).total
    assert 0.7 * used < est < 1.3 * used, (est, used)


@pytest.mark.parametrize("V,weighted", [(4096, False), (8192, True)])
def test_wide_vocabulary_cross_entropy_matches_reference(V, weighted):
    """Vocabularies above 2048 take the one-CTA-per-row two-pass kernel; in place over the logits, as the engine calls it."""
    from parameter_golf_b200.ops import native, reference as R
    C = native.load()
    torch.manual_seed(0)
    rows, cap = 96, 30.0
    z = (torch.randn(rows, V, device="cuda") * 8).bfloat16()
    tgt = torch.randint(0, V, (rows,), device="cuda", dtype=torch.int32)
    tw = (torch.rand(rows, device="cuda") + 0.2) if weighted else None
    wt = tw.sum().reshape(1) if weighted else None
    zf = z.float().requires_grad_(True)
    per = R.softcap_cross_entropy(zf, tgt.long(), cap, reduction="none")
    loss = (per * tw).sum() / tw.sum() if weighted else per.mean()
    loss.backward()
    nll = torch.empty(rows, device="cuda")
    acc = torch.zeros(1, device="cuda")
    buf = z.clone()
    C.softcap_ce(buf, tgt, nll, buf, acc, cap, 1.0 / rows, tw, wt)
    torch.cuda.synchronize()
    native.check_status()
    assert torch.allclose(nll, per.detach(), atol=2e-3, rtol=1e-4)
    assert float(acc[0]) / rows == pytest.approx(float(loss.detach()), rel=1e-4)
    assert rel_err(buf.float(), zf.grad) < 1e-2
    C.softcap_ce(z, tgt, nll, None, None, cap, 0.0)            # scoring only: logits untouched
    torch.cuda.synchronize()
    assert torch.allclose(nll, per.detach(), atol=2e-3, rtol=1e-4)


def test_tall_embedding_table_scatter_and_vocab_8192_step():
    """8192-row tables do not fit the shared-memory scatter tile: the atomic form must give the same sums, and a whole
    engine step at vocabulary 8192 (the reference's sp8192 families) must match the oracle."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import CudaEngine
    from parameter_golf_b200.ops import native
    C = native.load()
    torch.manual_seed(1)
    ids = torch.randint(0, 8192, (1024,), device="cuda", dtype=torch.int32)
    g = torch.randn(1024, 128, device="cuda").bfloat16()
    table = torch.zeros(8192, 128, device="cuda")
    C.embed_scatter_add(ids, g, table, 0, 128)
    want = torch.zeros(8192, 128, device="cuda").index_add_(0, ids.long(), g.float())
    assert torch.allclose(table, want, atol=1e-4)
    spec = small_spec(**{"model.vocab_size": 8192})
    params = gpt.fill_deterministic(spec.model)
    ids2 = torch.randint(0, 8192, (4, 128))
    tgt2 = torch.randint(0, 8192, (4, 128))
    eng = CudaEngine(spec, params, "cuda", 4, 128)
    eng.zero_grads()
    eng.micro_step(ids2.cuda().int(), tgt2.cuda().int(), 1)
    torch.cuda.synchronize()
    native.check_status()
    ref_loss, ref = oracle_grads(spec, params, ids2, tgt2)
    assert abs(float(eng.loss_sum[0]) / eng.T - float(ref_loss)) < 2e-2
    worst = {k: rel_err(eng.g[k], v) for k, v in ref.items()}
    bad = {k: v for k, v in worst.items() if v > (0.2 if k == "q_gain" else 0.06)}
    assert not bad, worst


def test_backward_observer_sees_every_block_in_reverse_order():
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import CudaEngine
    spec = small_spec(**{"model.recurrence.enabled": "true", "model.recurrence.start_layer": 1, "model.recurrence.repeat_layers": 2})
    eng = CudaEngine(spec, gpt.fill_deterministic(spec.model), "cuda", 2, 128)
    seen = []
    done = {}
    def obs(layer, slot):
        seen.append((layer, slot))
        if slot == eng.first_slot[layer]:                  # last time this layer appears in the backward: its gradient is complete
            done[layer] = float(eng.g["mlp_up_bank"][layer].abs().sum())
    eng.backward_observer = obs
    ids = torch.randint(0, 256, (2, 128), device="cuda", dtype=torch.int32)
    eng.zero_grads()
    eng.micro_step(ids, ids.roll(-1, 1), 1)
    torch.cuda.synchronize()
    assert [s for _, s in seen] == list(range(eng.nslots - 1, -1, -1))
    assert [l for l, _ in seen] == [l for l, _ in reversed(eng.sched)]
    for layer, v in done.items():                          # nothing touched that layer's gradient after its last block
        assert v > 0 and v == float(eng.g["mlp_up_bank"][layer].abs().sum())


def test_checkpoint_state_round_trip_restores_ema_and_trajectory():
    """Optimizer state (momentum, Adam moments, EMA shadows) saved after two steps and loaded into a fresh backend gives the
    same EMA export and the same third step as the backend that kept running."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import EngineBackend
    spec = small_spec(**{"train.ema_decay": 0.9})
    spec.mode = "record"
    spec.allow_unsupported_variants = True
    gen = torch.Generator().manual_seed(11)
    batches = [[(torch.randint(0, 256, (4, 128), generator=gen), torch.randint(0, 256, (4, 128), generator=gen))] for _ in range(3)]
    a = EngineBackend(spec, gpt.init_params(spec.model, 3))
    for b in batches[:2]:
        a.train_step(b, 1.0, 0.95, False)
    params = {k: v.detach().cpu().clone() for k, v in a.sync_params().items()}
    state = a.state_dict()
    assert "ema_banks" in state and len(state["ema_groups"]) == len(a.engine.groups)
    fresh = EngineBackend(spec, gpt.init_params(spec.model, 99))          # different initial weights: nothing may survive from them
    for k, v in params.items():
        fresh.sync_params()[k].copy_(v)
    fresh.load_state_dict(state)
    fresh.params_changed()
    ea, ef = a.final_params(ema=True), fresh.final_params(ema=True)
    for k in ea:
        assert torch.equal(ea[k], ef[k]), k
    la, lf = a.train_step(batches[2], 1.0, 0.95, False), fresh.train_step(batches[2], 1.0, 0.95, False)
    assert lf == pytest.approx(la, abs=1e-5)
    state.pop("ema_banks")
    with pytest.raises(RuntimeError, match="no EMA state"):
        fresh.load_state_dict(state)


def test_training_step_raises_when_a_device_wait_ran_out():
    """A bounded wait that gave up (here: a flag nothing sets) must surface from the training backend's own step, not only
    from an explicit status check, and the context must stay usable afterwards."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import EngineBackend
    from parameter_golf_b200.ops import native
    spec = small_spec(**{"train.ema_decay": 0.0})
    spec.mode = "record"
    spec.allow_unsupported_variants = True
    be = EngineBackend(spec, gpt.init_params(spec.model, 3))
    ids = torch.randint(0, 256, (4, 128))
    be.train_step([(ids, ids)], 1.0, 0.95, False)
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    native.load().comm_wait_flag(flag, 1, native.status_word())             # runs out after its time limit and records it
    with pytest.raises(RuntimeError, match="timed out during the training step"):
        be.train_step([(ids, ids)], 1.0, 0.95, False)
    assert math.isfinite(be.train_step([(ids, ids)], 1.0, 0.95, False))     # status cleared, context alive


def test_token_ids_outside_the_vocabulary_are_rejected_not_dereferenced():
    """A span from a shard written with a larger vocabulary: the embedding kernels must not turn the id into an address. The
    gather writes a zero row and flags the status word, the scatter skips the row, the training step raises with a message
    that names the cause, and the next step on clean data runs."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import EngineBackend
    from parameter_golf_b200.ops import native
    C = native.load()
    table = torch.randn(256, 64, device="cuda").bfloat16()
    ids = torch.tensor([3, 255, 256, 70000, -1, 7], dtype=torch.int32, device="cuda")
    out = torch.full((6, 64), 9.0, device="cuda", dtype=torch.bfloat16)
    C.embed_gather(ids, table, out, 0, 6, native.status_word())
    torch.cuda.synchronize()
    assert torch.equal(out[0], table[3]) and torch.equal(out[1], table[255]) and torch.equal(out[5], table[7])
    assert float(out[2:5].abs().max()) == 0.0
    with pytest.raises(RuntimeError, match="outside its embedding table"):
        native.check_status()
    dtable = torch.zeros(256, 64, device="cuda")
    g = torch.ones(6, 64, device="cuda", dtype=torch.bfloat16)
    C.embed_scatter_add(ids, g, dtable, 0, 6)
    torch.cuda.synchronize()
    assert float(dtable.sum()) == 3 * 64 and float(dtable[3].sum()) == 64 and float(dtable[255].sum()) == 64
    big = torch.zeros(8192, 64, device="cuda")                  # the table too tall for the shared-memory form: the atomic kernel
    C.embed_scatter_add(ids, g, big, 0, 6)
    torch.cuda.synchronize()
    assert float(big.sum()) == 4 * 64                            # id 256 is a row of this taller table; 70000 and -1 are not
    spec = small_spec(**{"train.ema_decay": 0.0})
    spec.mode = "record"
    spec.allow_unsupported_variants = True
    be = EngineBackend(spec, gpt.init_params(spec.model, 3))
    good = torch.randint(0, 256, (4, 128))
    bad = good.clone()
    bad[1, 17] = 300
    with pytest.raises(RuntimeError, match="outside its embedding table"):
        be.train_step([(bad, good)], 1.0, 0.95, False)
    assert math.isfinite(be.train_step([(good, good)], 1.0, 0.95, False))


@pytest.mark.parametrize("rank", [16, 80])
def test_q_lora_forward_and_adapter_gradients_match_the_oracle(rank):
    """Q-LoRA on the CUDA engine (two skinny products in the forward, four in the backward) against the autograd model with the
    same adapter: loss, per-token NLL and the gradients of A and B."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import EngineRunner
    from parameter_golf_b200.models.runner import OracleRunner
    from parameter_golf_b200.ops import native
    spec = small_spec()
    m = spec.model
    params = gpt.fill_deterministic(m)
    g = torch.Generator().manual_seed(rank)
    lora = {"a": torch.randn(m.num_layers, rank, m.model_dim, generator=g) * 0.05, "b": torch.randn(m.num_layers, m.model_dim, rank, generator=g) * 0.05,
            "alpha": float(rank), "trainable": True}
    ids = torch.randint(0, 256, (4, 128), generator=g)
    tgt = torch.randint(0, 256, (4, 128), generator=g)
    oracle = OracleRunner(m, {k: v.double() for k, v in params.items()})
    oracle.lora = {"a": lora["a"].double(), "b": lora["b"].double(), "alpha": lora["alpha"], "trainable": True}
    ref_loss, ref = oracle.loss_and_grads(ids, tgt, names=[])
    ref_nll = oracle.nll(ids, tgt)
    eng = EngineRunner(spec, params, "cuda", batch=4)
    eng.lora = {"a": lora["a"].cuda(), "b": lora["b"].cuda(), "alpha": lora["alpha"], "trainable": True}
    loss, grads = eng.loss_and_grads(ids, tgt, names=[])
    torch.cuda.synchronize()
    native.check_status()
    assert abs(float(loss) - float(ref_loss)) < 1e-3 * max(1.0, float(ref_loss)), (float(loss), float(ref_loss))
    assert rel_err(grads["lora.a"], ref["lora.a"]) < 0.03 and rel_err(grads["lora.b"], ref["lora.b"]) < 0.03
    assert (eng.nll(ids, tgt).cpu().double() - ref_nll.double()).abs().mean().item() < 0.06          # per-token NLLs of 4-20 nats from bf16 activations
    base = EngineRunner(spec, params, "cuda", batch=4)                     # without the adapter the loss differs: the adapter is really applied
    assert abs(float(base.loss_and_grads(ids, tgt, names=[])[0]) - float(loss)) > 1e-3


def test_reproducible_backward_gives_bit_identical_bank_gradients():
    """With `train.reproducible_backward` the weight-gradient products go through per-chunk partials and a fixed-order
    reduction and the attention backward uses no fp32 atomics: the gradients of the four weight banks (97 % of the parameters)
    come out bit-identical from two runs, also at a shape with several chunks and several CTAs per product. (The small
    per-column reductions of the row kernels - mix, skip, gain, scale gradients - and the embedding scatter still use atomics.)"""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import CudaEngine
    from parameter_golf_b200.ops import native
    spec = small_spec(**{"train.reproducible_backward": "true"})
    params = gpt.fill_deterministic(spec.model)
    torch.manual_seed(3)
    ids = torch.randint(0, 256, (16, 128))
    tgt = torch.randint(0, 256, (16, 128))
    grads = []
    for run in range(2):
        eng = CudaEngine(spec, params, "cuda", 16, 128)
        eng.zero_grads()
        for _ in range(2):                                       # two micro-batches accumulate into the same gradient banks
            eng.micro_step(ids.cuda().int(), tgt.cuda().int(), 2)
        torch.cuda.synchronize()
        native.check_status()
        grads.append({k: eng.g[k].clone() for k in gpt.BANKS})
    for k in gpt.BANKS:
        assert torch.equal(grads[0][k], grads[1][k]), k
    ref_loss, ref = oracle_grads(spec, params, ids, tgt)         # and they are the right gradients
    for k in gpt.BANKS:
        assert rel_err(grads[0][k], ref[k]) < 0.03, k


def test_lora_phased_ttt_on_the_engine_tracks_the_oracle():
    """The whole phased Q-LoRA evaluation loop (score, guard, adapter gradients, SGD with weight decay, phase reset) on the
    CUDA engine and on the autograd model from the same start: the scores agree and the base weights are untouched."""
    import numpy as np
    from parameter_golf_b200.data.bpb import BpbLuts
    from parameter_golf_b200.eval import ttt as T
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import EngineRunner
    from parameter_golf_b200.models.runner import OracleRunner
    spec = small_spec()
    m, ev = spec.model, spec.eval
    ev.stride, ev.chunk_tokens, ev.lora_rank, ev.lora_alpha, ev.phased_ttt_phases = 64, 4 * 128, 16, 16.0, 2
    ev.ttt_lr, ev.ttt_batch_seqs, ev.batch_windows, ev.phased_ttt_weight_decay, ev.max_eval_seconds = 0.05, 4, 4, 0.01, 0.0
    params = gpt.init_params(m, 7)
    toks = np.random.default_rng(2).integers(0, 256, 128 * 12 + 1).astype(np.uint16)
    luts = BpbLuts.seeded(256)
    ref = T.eval_lora_phased_ttt(OracleRunner(m, {k: v.clone() for k, v in params.items()}), toks, m, ev, luts)
    runner = EngineRunner(spec, params, "cuda", batch=4)
    got = T.eval_lora_phased_ttt(runner, toks, m, ev, luts, device="cuda")
    assert abs(got[0] - ref[0]) < 2e-2 and abs(got[1] - ref[1]) < 2e-2, (got, ref)
    for k, v in params.items():
        assert torch.allclose(runner.params[k].cpu(), v), k
    assert runner.lora is None


def test_guard_zones_around_buffers_stay_intact_and_detect_an_overrun(monkeypatch):
    """`PGB_CANARY=1` places every activation and scratch buffer between guard zones: a full training micro-step (all
    kernels, odd and even tails) leaves them intact, and a byte written one past a buffer's end is reported."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import CudaEngine
    monkeypatch.setenv("PGB_CANARY", "1")
    spec = small_spec()
    eng = CudaEngine(spec, gpt.fill_deterministic(spec.model), "cuda", 3, 128)
    ids = torch.randint(0, 256, (3, 128))
    eng.zero_grads()
    eng.micro_step(ids.cuda().int(), ids.cuda().int(), 1)
    eng.check_canaries()
    assert len(eng._canaries) > 20
    name, raw, used = eng._canaries[5]
    raw[512 + used] = 0                                   # host-side store one byte past the end of the buffer
    with pytest.raises(RuntimeError, match="guard zone after"):
        eng.check_canaries()


@pytest.mark.parametrize("weighted", [False, True])
def test_chunked_output_head_matches_the_full_logits_path(weighted):
    """`train.logit_chunk_rows` makes the output projection, the cross-entropy and the two products that consume the logits
    gradient run per chunk of rows (the automatic setting for 8192-token vocabularies, where [T, V] would be gigabytes): loss,
    per-token NLL and every gradient must match the path that keeps all logits, with and without per-token loss weights."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import CudaEngine, EngineRunner
    from parameter_golf_b200.ops import native
    torch.manual_seed(1)
    ids = torch.randint(0, 256, (4, 128))
    tgt = torch.randint(0, 256, (4, 128))
    table = (torch.rand(256, 256) + 0.5) if weighted else None
    out = {}
    for rows in (0, 128):
        spec = small_spec(**{"train.logit_chunk_rows": rows})
        params = gpt.fill_deterministic(spec.model)
        eng = CudaEngine(spec, params, "cuda", 4, 128)
        assert eng.logit_rows == (512 if rows == 0 else 128) and eng.logits.shape[0] == eng.logit_rows
        if weighted:
            eng.set_token_weight_table(table)
        eng.zero_grads()
        eng.micro_step(ids.cuda().int(), tgt.cuda().int(), 1)
        torch.cuda.synchronize()
        native.check_status()
        out[rows] = (float(eng.loss_sum[0]), eng.nll.clone(), {k: v.clone() for k, v in eng.g.items()})
    assert out[128][0] == pytest.approx(out[0][0], rel=1e-5)
    assert torch.allclose(out[128][1], out[0][1], atol=1e-5)
    for k, g in out[0][2].items():
        assert rel_err(out[128][2][k], g) < 1e-3, k               # same products, summed in a different order
    spec = small_spec(**{"train.logit_chunk_rows": 128})
    r = EngineRunner(spec, gpt.fill_deterministic(spec.model), "cuda", batch=4, train=False)
    full = EngineRunner(small_spec(), gpt.fill_deterministic(spec.model), "cuda", batch=4, train=False)
    assert torch.allclose(r.logits(ids), full.logits(ids), atol=1e-3) and torch.allclose(r.nll(ids, tgt), full.nll(ids, tgt), atol=1e-5)


@pytest.mark.parametrize("names", [["mlp_up_bank", "q_gain"], ["bigram_proj", "attn_scale"], ["tok_emb"], ["kv_bank", "mlp_scale", "smear_gate"]])
def test_gradients_of_some_parameters_are_those_of_all(names):
    """`loss_and_grads(names=...)` leaves out the products that feed other gradients only; what it returns is what the full call
    returns, up to the order of the fp32 adds (relative 2-norm 1e-4: about sqrt(terms) 2^-24), also on the next full call."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import EngineRunner
    from parameter_golf_b200.ops import native
    spec = small_spec()
    params = gpt.fill_deterministic(spec.model)
    torch.manual_seed(5)
    ids, tgt = torch.randint(0, 256, (4, 128)), torch.randint(0, 256, (4, 128))
    eng = EngineRunner(spec, params, "cuda", batch=4)
    names = [k for k in names if k in params]
    full = {k: v.clone() for k, v in eng.loss_and_grads(ids, tgt)[1].items()}
    some = {k: v.clone() for k, v in eng.loss_and_grads(ids, tgt, names=names)[1].items()}
    again = eng.loss_and_grads(ids, tgt)[1]
    native.check_status()
    assert sorted(some) == sorted(names)
    for k in names:
        assert float((some[k] - full[k]).norm()) <= 1e-4 * float(full[k].norm()) + 1e-12, k
    for k in full:
        assert float((again[k] - full[k]).norm()) <= 1e-4 * float(full[k].norm()) + 1e-12, k


@pytest.mark.parametrize("S", [128, 1280])
def test_a_window_scores_the_same_alone_and_in_a_batch(S):
    """Scoring one window by itself, in a ragged last batch or among many gives the same bits: no sum over features, keys or
    vocabulary is cut by the number of sequences."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import EngineRunner
    spec = small_spec(**{"model.train_seq_len": S, "model.eval_seq_len": S, "train.seq_len": S, "train.batch_tokens": 4 * S})
    r = EngineRunner(spec, gpt.fill_deterministic(spec.model), "cuda", batch=12, train=False)
    torch.manual_seed(S)
    ids, tgt = torch.randint(0, 256, (12, S)), torch.randint(0, 256, (12, S))
    whole = r.nll(ids, tgt)
    for lo, hi in ((0, 1), (11, 12), (4, 7)):
        assert torch.equal(r.nll(ids[lo:hi], tgt[lo:hi]), whole[lo:hi]), (lo, hi)


@pytest.mark.parametrize("variant,names", [("ve", ["ve_proj"]), ("ve", ["ve_embed", "tok_emb"]), ("ve", ["ve_layer_scales", "kv_bank"]), ("ve_recurrence", ["ve_scale"]),
                                           ("ve_lora", []), ("untied", ["lm_head"]), ("untied", ["tok_emb", "bigram_scale"]),
                                           ("chunked", ["tok_emb"]), ("chunked", ["skip_weights", "qo_bank"]), ("chunked_untied", ["mlp_down_bank"]),
                                           ("recurrence", ["resid_mix", "mlp_up_bank"])])
def test_gradients_of_some_parameters_are_those_of_all_in_every_family(variant, names):
    """The products left out by `loss_and_grads(names=...)` with value embeddings, recurrent blocks, an untied and a row-chunked
    head, and for an adapter alone: the gradients of the full call (relative 2-norm 1e-4, the order of fp32 adds), before and after."""
    from parameter_golf_b200.eval.ttt import init_q_lora
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import EngineRunner
    from parameter_golf_b200.ops import native
    ov = {}
    if "ve" in variant:
        ov.update({"model.value_embedding.enabled": "true", "model.value_embedding.dim": 64, "model.value_embedding.layers": "[2,3]"})
    if "recurrence" in variant:
        ov.update({"model.recurrence.enabled": "true", "model.recurrence.start_layer": 1, "model.recurrence.repeat_layers": 2})
    if "untied" in variant:
        ov["model.tie_embeddings"] = "false"
    if "chunked" in variant:
        ov["train.logit_chunk_rows"] = 128
    spec = small_spec(**ov)
    params = gpt.fill_deterministic(spec.model)
    assert set(names) <= set(params)
    torch.manual_seed(7)
    ids, tgt = torch.randint(0, 256, (4, 128)), torch.randint(0, 256, (4, 128))
    eng = EngineRunner(spec, params, "cuda", batch=4)
    if "lora" in variant:
        eng.lora = init_q_lora(spec.model, 16, 32.0, "cuda")
        eng.lora["b"].normal_(0.0, 0.02)
        eng.lora["trainable"] = True
        names = names + ["lora.a", "lora.b"]
    full = {k: v.clone() for k, v in eng.loss_and_grads(ids, tgt)[1].items()}
    some = {k: v.clone() for k, v in eng.loss_and_grads(ids, tgt, names=[k for k in names if k in params])[1].items()}
    again = eng.loss_and_grads(ids, tgt)[1]
    native.check_status()
    assert sorted(some) == sorted(names) and all(float(full[k].norm()) > 0 for k in names)
    for k in names:
        assert float((some[k] - full[k]).norm()) <= 1e-4 * float(full[k].norm()), k
    for k in full:
        assert float((again[k] - full[k]).norm()) <= 1e-4 * float(full[k].norm()) + 1e-12, k


@pytest.mark.parametrize("which", ["fold_scaled_grad_bf16", "fold_scaled_grad"])
def test_a_backward_that_raised_leaves_no_product_behind(which):
    """The staging buffers of the scaled weights' gradients are zero between uses because the fold kernel leaves them so. A call that
    raises between the product and the fold must not add its product to the next call's gradients."""
    from parameter_golf_b200.models import gpt
    from parameter_golf_b200.models.engine import EngineRunner
    spec = small_spec()
    params = gpt.fill_deterministic(spec.model)
    torch.manual_seed(9)
    ids, tgt = torch.randint(0, 256, (4, 128)), torch.randint(0, 256, (4, 128))
    eng = EngineRunner(spec, params, "cuda", batch=4)
    full = {k: v.clone() for k, v in eng.loss_and_grads(ids, tgt)[1].items()}
    engine = next(iter(eng.engines.values()))
    ext = engine.C

    class Raising:
        def __getattr__(self, name):
            if name == which:
                def fold(*a):
                    raise KeyboardInterrupt
                return fold
            return getattr(ext, name)

    engine.C = Raising()
    with pytest.raises(KeyboardInterrupt):
        eng.loss_and_grads(ids, tgt)
    engine.C = ext
    assert float(sum(t.abs().sum() for t in (engine.Gd, engine.Go, engine.Gbp))) > 0           # the product is there
    again = eng.loss_and_grads(ids, tgt)[1]
    for k in full:
        assert float((again[k] - full[k]).norm()) <= 1e-4 * float(full[k].norm()) + 1e-12, k
