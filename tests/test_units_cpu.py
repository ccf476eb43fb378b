"""CPU unit tests of the model layer: config, compaction, mask, deciders, losses, sampler, data glue."""
import json
import os

import pytest
import torch

from tah_b200 import TaHConfig, TaHForCausalLM
from tah_b200.model.iter_decider import (IterLabelDecider, MLPIterDecider, load_iter_decider, save_iter_decider)
from tah_b200.model.loss import IterDeciderLoss, NextTokenPredLoss, fixed_cross_entropy
from tah_b200.model.tah_config import decode_config, encode_config, resolve_config, save_config
from tah_b200.model.tah_model import ActiveSet, gather_active, scatter_back, topk_softmax_input_update
from tah_b200.ops import torch_ref
from tests.helpers import tiny_tah


# ---- config -----------------------------------------------------------------------------------------
def test_config_json_sentinels_round_trip():
    cfg = {"iter_decider_kwargs": {"dtype": torch.bfloat16, "cls": torch.nn.Linear, "dims": [1, 2]}, "max_iter": 2}
    enc = encode_config(cfg)
    assert enc["iter_decider_kwargs"]["dtype"] == {"__dtype__": True, "__str__": "torch.bfloat16"}
    assert enc["iter_decider_kwargs"]["cls"]["__type__"] is True
    dec = decode_config(json.loads(json.dumps(enc)))
    assert dec["iter_decider_kwargs"]["dtype"] is torch.bfloat16
    assert dec["iter_decider_kwargs"]["cls"] is torch.nn.Linear


def test_config_merge_precedence(tmp_path):
    saved = TaHConfig(max_iter=2, iter_decider="MLPIterDecider", iter_decider_kwargs={"threshold": 0.8},
                      adapter_kwargs={"r": 32})
    save_config(saved, str(tmp_path))
    # unknown keys in an old file are ignored
    raw = json.load(open(tmp_path / "tah_config.json"))
    raw["iter_attention_mode"] = "duo"
    json.dump(raw, open(tmp_path / "tah_config.json", "w"))
    over = TaHConfig(iter_decider_kwargs={"threshold": 0.9}, max_iter=None, adapter_kwargs={})
    got = resolve_config(str(tmp_path), over)
    assert got.max_iter == 2 and got.iter_decider == "MLPIterDecider"
    assert got.iter_decider_kwargs == {"threshold": 0.9}          # non-empty override wins
    assert got.adapter_kwargs == {"r": 32}                         # {} means "use saved"
    assert resolve_config(str(tmp_path), None).iter_decider_kwargs == {"threshold": 0.8}


# ---- compaction -------------------------------------------------------------------------------------
def test_gather_scatter_round_trip():
    g = torch.Generator().manual_seed(0)
    for _ in range(20):
        B, S = int(torch.randint(1, 5, (1,), generator=g)), int(torch.randint(1, 12, (1,), generator=g))
        mask = torch.rand(B, S, generator=g) < 0.4
        x = torch.randn(B, S, 3, generator=g)
        ids = torch.randint(0, 50, (B, S), generator=g)
        pad, gx, gi, none = gather_active(mask, x, ids, None, pad_value=0)
        assert none is None and gx.shape[1] == int(mask.sum(1).max()) and pad.shape == gx.shape[:2]
        for b in range(B):
            n = int(mask[b].sum())
            assert torch.equal(gx[b, :n], x[b][mask[b]]) and torch.equal(gi[b, :n], ids[b][mask[b]])
            assert (gx[b, n:] == 0).all() and pad[b, n:].all() and not pad[b, :n].any()
        back = scatter_back(mask, gx, torch.full_like(x, -7.0))
        assert torch.equal(back[mask], x[mask]) and (back[~mask] == -7).all()
        sel = torch.rand(B, S, generator=g) < 0.5
        part = scatter_back(mask, gx, torch.zeros_like(x), assignment_mask=sel)
        assert torch.equal(part[mask & sel], x[mask & sel]) and (part[~(mask & sel)] == 0).all()


def test_active_set_empty():
    act = ActiveSet(torch.zeros(2, 5, dtype=torch.bool))
    assert act.n == 0 and act.width == 0


# ---- duo-causal predicate --------------------------------------------------------------------------
def test_duo_mask_matches_brute_force():
    g = torch.Generator().manual_seed(1)
    B, Tq, Tk = 2, 5, 9
    qp, kp = torch.randint(0, 6, (B, Tq), generator=g), torch.randint(0, 6, (B, Tk), generator=g)
    kvalid = (torch.rand(B, Tk, generator=g) < 0.8).long()
    qd, kd = torch.randint(0, 3, (B, Tq), generator=g), torch.randint(0, 3, (B, Tk), generator=g)
    m = torch_ref.duo_mask(qp, kp, kvalid, qd, kd)
    for b in range(B):
        for i in range(Tq):
            for j in range(Tk):
                want = bool(kp[b, j] <= qp[b, i] and kd[b, j] <= qd[b, i] and kvalid[b, j] == 1)
                assert bool(m[b, i, j]) == want


def test_depth0_queries_never_see_deeper_kv():
    model = tiny_tah().eval()
    ids = torch.randint(0, 1024, (1, 10))
    labels_hard = torch.ones(1, 10, dtype=torch.long)
    labels_hard[0, 3] = 2
    with torch.no_grad():
        # no `labels`: with labels the model forces one continuation when the decider stops everything
        a = model(ids, iter_count_labels=labels_hard)
        b = model(ids, iter_count_labels=torch.ones(1, 10, dtype=torch.long))
    # only the hard token's own logits change: depth-0 passes of later tokens ignore its depth-1 K/V
    same = torch.ones(10, dtype=torch.bool)
    same[3] = False
    torch.testing.assert_close(a.logits[0, same], b.logits[0, same])
    assert not torch.allclose(a.logits[0, 3], b.logits[0, 3])
    assert a.iter_count.tolist() == [[1, 1, 1, 2, 1, 1, 1, 1, 1, 1]]


# ---- soft embedding / deciders ----------------------------------------------------------------------
def test_topk_softmax_input_update():
    E = torch.randn(50, 8)
    logits = torch.randn(3, 50)
    out = topk_softmax_input_update(logits, E, 5)
    v, i = logits.topk(5, -1)
    ref = (torch.softmax(v, -1)[..., None] * E[i]).sum(-2)
    torch.testing.assert_close(out, ref)
    assert topk_softmax_input_update(logits, E, 500).shape == (3, 8)     # k is clipped to the vocabulary


def test_label_decider_rules():
    d = IterLabelDecider(max_iter=3)
    logits = torch.zeros(4, 7)
    labels = torch.tensor([1, 2, 3, -100])
    dec, z = d(logits, 1, iter_count_labels=labels)
    assert dec.tolist() == [False, True, True, False] and (z == 0).all()
    dec, z = d(logits, 3, iter_count_labels=labels)
    assert not dec.any() and (z == -10).all()
    dec, _ = d(logits, 1)
    assert not dec.any()


def test_mlp_decider_features_keys_and_persistence(tmp_path):
    torch.manual_seed(0)
    d = MLPIterDecider(topk=4, hidden_states_size=8, hidden_states_layer_nums=[0, 2], hidden_dims=[6, 6],
                       dropout_rate=0.0, threshold=0.8, max_iter=2, dtype=torch.float32).eval()
    keys = set(d.state_dict())
    assert {"threshold", "logits_projection.weight", "combined_projection.bias", "backbone.input_projection.weight",
            "backbone.blocks.0.layer_norm.weight", "backbone.blocks.0.mlp.0.weight", "backbone.blocks.0.mlp.3.bias",
            "backbone.output_layer.0.weight", "backbone.output_layer.1.weight"} <= keys
    logits, hs = torch.randn(5, 20), torch.randn(5, 3, 8)
    dec, z = d(logits, 1, all_hidden_states=hs)
    feats = torch.cat([hs[:, 0], hs[:, 2], d.logits_projection(logits.topk(4, -1).values)], -1)   # taps first, then logits
    torch.testing.assert_close(z, d.backbone(d.combined_projection(feats)).squeeze(-1))
    assert torch.equal(dec, torch.sigmoid(z) > 0.8)
    dec2, z2 = d(logits, 1, tapped_hidden_states=torch.cat([hs[:, 0], hs[:, 2]], -1))
    torch.testing.assert_close(z2, z)
    assert not d(logits, 2, all_hidden_states=hs)[0].any()
    with pytest.raises(ValueError):
        d(logits, 1, all_hidden_states=torch.randn(5, 2, 8))
    save_iter_decider(d, str(tmp_path))
    blob = torch.load(tmp_path / "iter_decider.bin", weights_only=False)
    assert blob["class"] == "MLPIterDecider" and blob["init_args"]["threshold"] == 0.8
    args = dict(blob["init_args"], threshold=0.9)
    d2 = load_iter_decider(str(tmp_path), class_name="MLPIterDecider", init_args=args).eval()
    assert abs(float(d2.threshold) - 0.9) < 1e-6                     # configured value beats the stored one
    torch.testing.assert_close(d2(logits, 1, all_hidden_states=hs)[1], z)


# ---- losses -----------------------------------------------------------------------------------------
def test_fixed_cross_entropy_normalisation():
    x, t = torch.randn(6, 9), torch.tensor([1, 2, -100, 4, -100, 0])
    ref_sum = torch.nn.functional.cross_entropy(x, t, ignore_index=-100, reduction="sum")
    torch.testing.assert_close(fixed_cross_entropy(x, t, num_items_in_batch=10), ref_sum / 10)
    torch.testing.assert_close(fixed_cross_entropy(x, t), ref_sum / 4)


def test_iter_decider_loss_scale_and_accuracy():
    loss = IterDeciderLoss(pos_weight=2.0, skip_last_iter=True, max_iter=2)
    B, T = 2, 4
    loss.prepare_loss(B, T, torch.device("cpu"), torch.float32)
    active_index = torch.arange(B * T)
    valid = torch.tensor([1, 1, 1, 0, 1, 1, 1, 1], dtype=torch.bool)
    labels = torch.tensor([1, 2, -100, 1, 2, 1, 1, 1])
    z = torch.tensor([-1.0, 2.0, 0.3, 0.5, -0.2, 0.1, -3.0])        # one per valid token
    loss.intra_iter_loss_func(active_index=active_index, active_valid=valid, continue_logits=z, iter_depth=1,
                              active_iter_count_labels=labels, iter_decider_threshold=0.5)
    lab_v = labels[valid]
    use = lab_v != -100
    bce = torch.nn.functional.binary_cross_entropy_with_logits(z[use], (lab_v[use] > 1).float(),
                                                               pos_weight=torch.tensor(2.0))
    iter_count = torch.ones(B, T, dtype=torch.long)
    full_labels = torch.tensor([[1, 2, 0, 1], [2, 1, 1, 1]])          # max-merged dense view: zeros, not -100
    out = loss.final_loss_func(torch.zeros(B, T, 3), None, iter_count, iter_count_labels=full_labels)
    # every processed position counts in the mean (the reference's scale quirk): the sum of the spread
    # per-token shares equals the mean BCE, divided by all B*T positions
    torch.testing.assert_close(out, bce / (B * T))
    loss.prepare_loss(B, T, torch.device("cpu"), torch.float32)
    loss.intra_iter_loss_func(active_index=active_index, active_valid=valid, continue_logits=z, iter_depth=2,
                              active_iter_count_labels=labels)
    assert float(loss.final_loss_func(torch.zeros(B, T, 3), None, iter_count, iter_count_labels=full_labels)) == 0.0
    with pytest.raises(ValueError):
        IterDeciderLoss(skip_last_iter=True)


def test_next_token_loss_matches_shifted_ce():
    model = tiny_tah(max_iter=1).eval()
    ids = torch.randint(0, 1024, (2, 12))
    labels = ids.clone()
    labels[:, :4] = -100
    with torch.no_grad():
        out = model(ids, labels=labels)
    ref = torch.nn.functional.cross_entropy(out.logits[:, :-1].reshape(-1, 1024).float(), labels[:, 1:].reshape(-1),
                                            ignore_index=-100)
    torch.testing.assert_close(out.loss, ref)
    assert isinstance(model.train_loss, NextTokenPredLoss)


# ---- sampler ----------------------------------------------------------------------------------------
def test_sampler_filters_in_order():
    logits = torch.log(torch.tensor([[0.5, 0.25, 0.15, 0.06, 0.04]]))
    g = torch.Generator().manual_seed(0)
    assert int(torch_ref.sample(logits, do_sample=False)) == 0
    draws = torch.stack([torch_ref.sample(logits, top_k=2, generator=g) for _ in range(200)])
    assert set(draws.flatten().tolist()) <= {0, 1}
    draws = torch.stack([torch_ref.sample(logits, top_p=0.7, generator=g) for _ in range(200)])
    assert set(draws.flatten().tolist()) <= {0, 1}                    # the token crossing top_p stays
    draws = torch.stack([torch_ref.sample(logits, min_p=0.4, generator=g) for _ in range(200)])
    assert set(draws.flatten().tolist()) <= {0, 1}
    draws = torch.stack([torch_ref.sample(logits, temperature=0.05, generator=g) for _ in range(50)])
    assert (draws == 0).all()


# ---- forward bookkeeping ----------------------------------------------------------------------------
def test_force_one_continuation_and_uniform_passes():
    model = tiny_tah(decider="MLPIterDecider",
                     decider_kwargs=dict(topk=10, hidden_states_size=256, hidden_states_layer_nums=[1, 4],
                                         hidden_dims=[32, 32], dropout_rate=0.0, threshold=0.999999, dtype=torch.float32),
                     train_loss="IterDeciderLoss", train_loss_kwargs=dict(pos_weight=5.4, skip_last_iter=True))
    model.train()
    ids = torch.randint(0, 1024, (2, 16))
    hard = torch.ones(2, 16, dtype=torch.long)
    out = model(ids, labels=ids, iter_count_labels=hard)
    assert int((out.iter_count == 2).sum()) == 1                      # exactly one forced continuation
    out.loss.backward()
    assert model.iter_decider.combined_projection.weight.grad.abs().sum() > 0
    model.eval()
    with torch.no_grad():
        out = model(ids)
    assert int(out.iter_count.max()) == 1
    model.uniform_passes = True
    with torch.no_grad():
        out2 = model(ids)
    torch.testing.assert_close(out2.logits, out.logits)


def test_padding_positions_count_one_pass():
    model = tiny_tah().eval()
    ids = torch.randint(0, 1024, (2, 8))
    attn = torch.ones(2, 8, dtype=torch.long)
    attn[0, :3] = 0
    hard = torch.full((2, 8), 2)
    with torch.no_grad():
        out = model(ids, attention_mask=attn, labels=ids, iter_count_labels=hard)
    assert out.iter_count[0, :3].tolist() == [1, 1, 1] and (out.iter_count[attn.bool()] == 2).all()


def test_segment_meta_matches_duo_mask_cpu():
    """The (base, count) prefixes handed to the tensor-core attention kernels describe exactly the keys
    that the duo-causal mask allows, for left-padded and right-padded batches and a sparse deeper pass."""
    import torch
    from tah_b200.ops.autograd_ops import SegmentMeta
    from tah_b200.ops.torch_ref import duo_mask
    B, T = 3, 11
    for pad_left in (True, False):
        lens = torch.tensor([11, 7, 3])
        valid0 = torch.zeros(B, T, dtype=torch.long)
        for b, n in enumerate(lens.tolist()):
            if pad_left:
                valid0[b, T - n:] = 1
            else:
                valid0[b, :n] = 1
        pos0 = (valid0.cumsum(-1) - 1).clamp(min=0)
        # deeper pass: a subset of the valid tokens, packed to the left of a narrower block
        g = torch.Generator().manual_seed(3)
        act = (torch.rand(B, T, generator=g) < 0.5) & valid0.bool()
        act[:, -1] |= valid0[:, -1].bool()
        width = int(act.sum(1).max())
        pos1 = torch.zeros(B, width, dtype=torch.long)
        valid1 = torch.zeros(B, width, dtype=torch.long)
        for b in range(B):
            idx = act[b].nonzero().flatten()
            pos1[b, :idx.numel()] = pos0[b, idx]
            valid1[b, :idx.numel()] = 1
        # queries of the deeper pass see depth-0 keys and depth-1 keys
        meta = SegmentMeta(pos1, [pos0, pos1], [valid0, valid1], q_valid=valid1)
        for s, (kp, kv, Ts) in enumerate(((pos0, valid0, T), (pos1, valid1, width))):
            mask = duo_mask(pos1, kp, kv)                               # [B, width, Ts]
            base = meta.bases[s].view(B, width)
            cnt = meta.counts[s].view(B, width)
            for b in range(B):
                for i in range(width):
                    if not valid1[b, i]:
                        continue
                    want = mask[b, i].nonzero().flatten() + b * Ts
                    got = torch.arange(int(base[b, i]), int(base[b, i]) + int(cnt[b, i]))
                    assert torch.equal(want, got), (pad_left, s, b, i)
            # padding queries see nothing; the tiling bound never decreases along a sample's rows and
            # is never below the count
            assert (cnt[valid1 == 0] == 0).all()
            bound = meta.bounds[s].view(B, width)
            assert (bound[:, 1:] >= bound[:, :-1]).all() and (bound >= cnt).all()
        row0, nkeys, kidx0, qa, qb = meta.items[0]
        assert int(nkeys.sum()) == int(valid0.sum()) and torch.equal(qb - qa, torch.full_like(qa, width))


def test_attention_tiling_helpers_cpu():
    """Query tiles and key-block work items of the packed attention kernels (pure index arithmetic)."""
    import torch
    from tah_b200.ops.cuda import attn_kv_items, attn_tiles
    q0, qn = attn_tiles(torch.tensor([300, 0, 128, 5]))
    assert q0.tolist() == [0, 128, 256, 300, 428] and qn.tolist() == [128, 128, 44, 128, 5]
    row0, nkeys, kidx0, qa, qb = attn_kv_items(torch.tensor([260, 3]), torch.tensor([10, 500]), torch.tensor([7, 9]))
    assert row0.tolist() == [10, 138, 266, 500] and nkeys.tolist() == [128, 128, 4, 3]
    assert kidx0.tolist() == [0, 128, 256, 0]
    assert qa.tolist() == [0, 0, 0, 7] and qb.tolist() == [7, 7, 7, 16]


def test_gemm_planner_choices_cpu():
    """The split-K / tile planner (pure host arithmetic): legal plans, split-K for small-M long-K shapes,
    none for shapes that already fill the GPU."""
    from tah_b200.ops.cuda import _fits, plan_gemm
    for (M, F, Kd, R, dual) in [(256, 4096, 2048, 192, False), (256, 2048, 6144, 64, False), (64, 2048, 2048, 0, False),
                                (256, 6144, 2048, 128, True), (8192, 4096, 2048, 0, False), (1, 128, 128, 0, False)]:
        bn, s = plan_gemm(M, F, Kd, R, dual)
        assert bn in (16, 32, 64, 128, 256) and s in (1, 2, 4)
        assert s == 1 or (bn % s == 0 and (bn // s) % 16 == 0 and _fits(bn, s, 2 if dual else 1))
    assert plan_gemm(256, 2048, 6144)[1] > 1            # few feature tiles, long K: split
    assert plan_gemm(8192, 4096, 2048)[1] == 1          # 1024 CTAs already
    assert plan_gemm(256, 151936, 2048)[1] == 1         # LM head


def test_reference_import_names_resolve_to_this_package():
    """``import tah`` (the reference's package name) serves the same module objects as ``tah_b200``."""
    import importlib
    import tah
    import tah_b200
    assert tah.TaHForCausalLM is tah_b200.TaHForCausalLM
    for sub in ("model", "model.tah_model", "model.iter_decider", "model.loss", "model.utils", "model.causal_cache",
                "model.tah_config", "train", "utils", "evaluate", "evaluate.backends", "evaluate.jobs",
                "evaluate.datasets", "evaluate.matheval", "evaluate.codeeval"):
        assert importlib.import_module("tah." + sub) is importlib.import_module("tah_b200." + sub)
    from tah.model.tah_model import additive_logits_update, gather_active, scatter_back, topk_softmax_input_update  # noqa: F401
    from tah.model.utils import TaHForCasualLM_generate, sample_next_token, set_all_seeds  # noqa: F401
    from tah.train import CustomTaHDataCollator, CustomTaHTrainer, LoggerCallback, fixed_cross_entropy  # noqa: F401
    from tah.utils import preprocess_dataset  # noqa: F401
    from tah.evaluate.backends import cleanup, setup_backend, setup_hf, setup_sglang, setup_tah, time_inference, warmup  # noqa: F401


def test_zero_adamw_no_decay_group_matches_torch_param_groups():
    """Parameters named as no-decay (norm gains, biases) take no weight decay, like the two parameter groups of the
    HuggingFace trainer the reference builds on."""
    from tah_b200.parallel.zero import ZeroAdamW
    torch.manual_seed(0)
    net = torch.nn.Sequential(torch.nn.Linear(6, 5), torch.nn.LayerNorm(5), torch.nn.Linear(5, 3))
    ref = torch.nn.Sequential(torch.nn.Linear(6, 5), torch.nn.LayerNorm(5), torch.nn.Linear(5, 3))
    ref.load_state_dict(net.state_dict())
    nd = [p for n, p in net.named_parameters() if p.dim() < 2]
    opt = ZeroAdamW(net.parameters(), lr=1e-2, weight_decay=0.1, no_decay=nd)
    rnd = {id(p) for n, p in ref.named_parameters() if p.dim() < 2}
    ropt = torch.optim.AdamW([{"params": [p for p in ref.parameters() if id(p) not in rnd], "weight_decay": 0.1},
                              {"params": [p for p in ref.parameters() if id(p) in rnd], "weight_decay": 0.0}], lr=1e-2)
    for step in range(3):
        x = torch.randn(4, 6, generator=torch.Generator().manual_seed(step))
        net(x).pow(2).mean().backward()
        ref(x).pow(2).mean().backward()
        opt.step()
        opt.zero_grad()
        ropt.step()
        ropt.zero_grad()
    for (n, a), b in zip(net.named_parameters(), ref.parameters()):
        torch.testing.assert_close(a, b, atol=1e-6, rtol=1e-5, msg=n)


def test_zero_adamw_accumulates_micro_batch_gradients_in_fp32():
    """``accumulate()`` after every backward: the window's gradient is summed in fp32 and rounded to bf16 once, so
    sixteen micro-batches whose gradients differ by orders of magnitude keep their small terms."""
    from tah_b200.parallel.zero import ZeroAdamW
    torch.manual_seed(0)
    n = 4096
    grads = [torch.randn(n) * (1.0 if i == 0 else 2e-3) for i in range(16)]
    exact = torch.stack(grads).sum(0)

    def run(use_acc):
        p = torch.nn.Parameter(torch.zeros(n, dtype=torch.bfloat16))
        opt = ZeroAdamW([p], lr=1e-3, weight_decay=0.0, max_grad_norm=0.0)
        for g in grads:
            p.grad.add_(g.to(torch.bfloat16))            # what autograd does: accumulate into the 16-bit buffer
            if use_acc:
                opt.accumulate()
        opt._collect_stray_grads()
        opt._flush_accumulator()
        return opt.flat_grad[:n].float().clone()

    err_plain = (run(False) - exact).abs().mean()
    err_acc = (run(True) - exact).abs().mean()
    assert err_acc < 0.5 * err_plain                      # one rounding instead of sixteen
    assert err_acc < 2.5e-3                                # bf16 rounding of values of order one


def test_kv_cache_guard_pages(monkeypatch):
    from tah_b200.engine.kv_cache import CacheGeometry, PagedKVCache
    monkeypatch.setenv("TAH_B200_CANARY", "2")
    kv = PagedKVCache(CacheGeometry(2, 2, 64, 16), 3, 40, 2, device="cpu")
    assert kv.pool[0].shape[1] == kv.n_pages[0] + 2 and kv.check_guards()
    slots = kv.assign_prefill(0, torch.tensor([5, 17, 33]))
    assert int(slots.max()) < kv.n_pages[0] * 16            # slots never reach into the guard pages
    kv.pool[1][0, kv.n_pages[1], 0, 0, 0, 0] = 1.0
    assert not kv.check_guards()
    monkeypatch.delenv("TAH_B200_CANARY")
    assert PagedKVCache(CacheGeometry(2, 2, 64, 16), 3, 40, 2, device="cpu").check_guards()


def test_adapter_factor_keeps_gradients_of_32_bit_factors():
    """The block-diagonal factor and its gradients are those of assigning each scaled block to its place, to the bit."""
    from tah_b200.ops.autograd_ops import _BlockDiag
    spans, F, r, scaling = ((0, 12), (12, 20)), 24, 8, 1.7
    g = torch.Generator().manual_seed(0)
    first = [torch.randn(hi - lo, r, generator=g) for lo, hi in spans]
    gy = torch.randn(F, len(spans) * r, generator=g).to(torch.bfloat16)
    got = []
    for assign in (False, True):
        blocks = [b.clone().requires_grad_() for b in first]
        if assign:
            out = torch.zeros(F, len(spans) * r, dtype=torch.bfloat16)
            for j, (lo, hi) in enumerate(spans):
                out[lo:hi, j * r:(j + 1) * r] = blocks[j] * scaling
        else:
            out = _BlockDiag.apply(F, spans, scaling, *blocks)
        out.backward(gy)
        got.append([out.detach()] + [b.grad for b in blocks])
    assert all(torch.equal(a, b) for a, b in zip(*got))


def test_native_pass_reads_the_tensors_that_the_layers_hold_now():
    from tah_b200.engine.weights import EngineWeights
    from tah_b200.ops import cuda
    w = EngineWeights(tiny_tah(max_iter=2, dtype=torch.bfloat16).simple_base_model)
    held = lambda: [[getattr(a, f) for f, _ in a._fields_] for a in w.native_pass()]
    want = lambda: [[0 if getattr(l, f) is None else getattr(l, f).data_ptr() for f, _ in w.native_pass()._type_._fields_] for l in w.layers]
    before = held()
    assert before == want() and w.native_pass() is w.native_pass()
    w.layers[1].w_o = w.layers[1].w_o.clone()
    assert held() == want() != before
    w.layers[0] = type(w.layers[0])(**{f: getattr(w.layers[1], f) for f, _ in w.native_pass()._type_._fields_})
    assert held() == want()
    ln1 = w.layers[1].ln1
    for other in (torch.zeros(ln1.numel() + 1, dtype=torch.bfloat16)[1:], ln1.float()):       # off the boundary, another type: launch by launch
        w.layers[1].ln1 = ln1
        w.pass_weights = w.pass_weights or cuda.pass_weights(w.layers)
        assert w.native_pass() is not None
        w.layers[1].ln1 = other
        assert w.native_pass() is None


def test_decode_attention_split_follows_the_warps_that_fit():
    """The split of the rows among CTAs is derived from how many the kernel keeps resident, which its geometry decides."""
    from tah_b200.ops import cuda
    if not os.path.exists(cuda._LIB_PATH):
        pytest.skip("the library is not built")
    split = lambda rows, nq, nkv, hd, pages: cuda.decode_attn_split(rows, nq, nkv, hd, pages)
    for nq, hd in ((8, 128), (16, 128), (32, 128), (8, 64), (16, 64), (32, 64)):
        at = [split(rows, nq, 8, hd, 70) for rows in range(1, 300)]
        assert at[0] == 4 and all(1 <= s <= 4 for s in at)          # one row of 70 pages is spread as far as it goes
        assert {split(rows, nq, 8, hd, 4) for rows in (1, 16, 64, 256)} == {1}      # four pages: a merge costs more than it gives
    # 64 rows of 8 KV heads and few pages: one wave holds them with three warps where 12 are resident, with two of eight, with four of 16
    warps = lambda nq, hd: cuda.lib().tahb_decode_attn_warps(64, nq, 8, hd, 6, 1)
    assert [warps(16, 128), warps(32, 128), warps(16, 64), warps(32, 64)] == [3, 2, 4, 3]


def test_tile_plan_counts_the_clusters_that_fit():
    """Clusters of four do not fill every SM: no plan counts on a wave of more than 132 of their CTAs; a narrow weight gets narrow tiles."""
    from tah_b200.ops import cuda
    for rows in (64, 192, 512, 1024, 1536, 2048, 2560, 4096):
        for K in (1024, 2048, 6144):
            for M in range(257, 3000, 31):
                pair, bn, splits = cuda.plan_tiles(M, rows, K, rows % 256 == 0, True)
                ctas = -(-rows // 128) * -(-M // bn) * splits
                assert splits < 4 or not 132 < ctas <= 148, (M, rows, K)
    assert cuda.plan_tiles(1536, 64, 2048, False, True) == (False, 64, 4)
    assert cuda.plan_tiles(450, 1536, 2048, True, True) == (False, 128, 2)


def test_persistent_tile_plan():
    """Tiles of the persistent product: narrow tiles where wide ones leave SMs idle, and none where few tiles with
    a long reduction want a split."""
    from tah_b200.ops import cuda
    for rows in (64, 512, 2048, 12288, 151936):
        for K in (64, 300, 2048, 12288):
            for M in (257, 700, 3072, 16000):
                assert cuda.plan_persist(M, rows, K) in (0, 64, 128, 192, 256)
                assert cuda.plan_persist(M, rows, K, 64, True) in (0, 64, 128, 192, 256)
    assert cuda.plan_persist(504, 2048, 2048) == 64 and cuda.plan_persist(16000, 2048, 2048) == 256
    assert cuda.plan_persist(264, 2048, 12288) == 0
    # one token tile: the wide SwiGLU and the head, which one tile per CTA does in an uneven wave or several
    assert cuda.plan_persist(256, 12288, 2048, 64, True) == 192 and cuda.plan_persist(256, 151936, 2048) in (192, 256)
    assert not any(cuda.plan_persist(M, rows, 2048) for M in (129, 192, 256) for rows in (1024, 2048, 4096))


def _launches(monkeypatch):
    """The products' entry points as fakes: what is called, in a list."""
    from tah_b200.ops import cuda
    called = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: called.append(name) or 0

    monkeypatch.setattr(cuda, "lib", Lib)
    monkeypatch.setattr(cuda, "_check_bf16_2d", lambda t, name: None)
    monkeypatch.setattr(cuda, "status_word", lambda device: None)
    monkeypatch.setattr(cuda, "_stream", lambda: None)
    monkeypatch.setattr(cuda, "_p", lambda t: None)
    return cuda, called


def test_one_tile_switch_turns_off_the_persistent_form(monkeypatch):
    """``TAH_B200_GEMM_PAIR=0``: one-tile forms only, whatever was planned before."""
    cuda, called = _launches(monkeypatch)
    t = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)
    x, w = t(1500, 2048), t(2048, 2048)

    def forms():
        called.clear()
        cuda.gemm(x, w)
        cuda.gemm_t(x, w, w_t=True)
        cuda.xielu_linear(x, w, 0.8, 0.5)
        return called[:]

    assert forms() == ["tahb_gemm_persist"] * 3
    monkeypatch.setattr(cuda, "PAIR_AUTO", False)
    assert forms() == ["tahb_gemm", "tahb_gemm_t", "tahb_gemm_xielu"]
    for M in (200, 600, 1504, 16000):
        assert cuda.plan_persist(M, 4096, 2048) == 0 and cuda.gemm_form(M, 4096, 2048)[0] == cuda.gemm_t_form(M, 4096, 2048, True, True)[0] == "tile"


def test_form_of_a_product_is_the_one_launched(monkeypatch):
    """What :func:`gemm_form` and :func:`gemm_t_form` name is what :func:`gemm` and :func:`gemm_t` launch."""
    cuda, called = _launches(monkeypatch)
    entry = {"few": "tahb_gemm_few", "persist": "tahb_gemm_persist", "pair": "tahb_gemm", "tile": "tahb_gemm"}
    t = lambda *s: torch.empty(*s, dtype=torch.bfloat16)
    for M in (1, 16, 40, 100, 130, 256, 257, 504, 1500, 5000):
        for rows, K in ((64, 256), (320, 448), (2048, 2048), (4096, 1024), (2048, 6144), (12288, 2048)):
            for how in ({}, dict(const_w=True), dict(swiglu=True), dict(swiglu_interleaved=True), dict(gelu=True)):
                called.clear()
                cuda.gemm(t(M, K), t(rows, K), **how)
                assert called == [entry[cuda.gemm_form(M, rows, K, **how)[0]]], (M, rows, K, how)
            for x_t, w_t in ((False, True), (True, True)):
                called.clear()
                cuda.gemm_t(t(K, M + -M % 8) if x_t else t(M, K), t(K, rows), x_t=x_t, w_t=w_t)
                form = cuda.gemm_t_form(M + -M % 8 if x_t else M, rows, K, x_t, w_t)[0]
                assert called == ["tahb_gemm_persist" if form == "persist" else "tahb_gemm_t"], (M, rows, K, x_t, w_t)


def test_weight_gradients_over_few_tokens_take_one_tile_or_pair_per_cta():
    """Reductions below those that the long ones' constants were fitted to: few output tiles stay off the persistent form, many take it."""
    from tah_b200.ops import cuda
    form = lambda F, K, T: cuda.gemm_t_form(F, K, T, True, True)
    assert [form(1000, 2048, T) for T in (8, 50, 128, 200)] == [("tile", 128, 1)] * 4
    assert [form(576, 1536, T) for T in (100, 200, 320)] == [("tile", 64, 1)] * 3
    assert form(2560, 2560, 8)[0] == form(2560, 2560, 64)[0] == "pair"
    assert form(12288, 2048, 50)[0] == form(2048, 6144, 200)[0] == form(12288, 2048, 3072)[0] == "persist"


def test_rules_of_ticks_of_few_rows():
    """Norms move into the products of ticks of few and narrow rows only; adapter inputs are gathered for many rows and large adapters."""
    from tah_b200.ops import cuda
    for K, most in ((256, 8), (1024, 8), (2048, 8), (2560, 5), (4096, 2), (8192, 0)):
        assert [M for M in range(1, 17) if cuda.few_fused_pays(M, K)] == list(range(1, most + 1))
    assert not cuda.lora_gated_pays(32, 2048, 192) and cuda.lora_gated_pays(33, 2048, 192) and cuda.lora_gated_pays(256, 6144, 64)
    assert not any(cuda.lora_gated_pays(M, K, R) for M in (64, 256) for K, R in ((2048, 64), (1024, 192), (512, 256), (16384, 64)))


def test_host_plan_of_a_prefill_is_the_device_one():
    """Query tiles and page assignment of a prefill worked out on the host: what the tensor operations give, over row counts and lengths
    (empty rows, whole pages, one past them), and the same refusal of a pool that is too small."""
    import numpy as np
    import torch
    from tah_b200.engine.kv_cache import CacheGeometry, PagedKVCache
    from tah_b200.ops import cuda
    gen = torch.Generator().manual_seed(0)
    for rows in (1, 2, 7, 40):
        counts = torch.randint(0, 400, (rows,), generator=gen)
        counts[0], counts[-1] = 128, 129
        want = cuda.attn_tiles(counts, by_work=True)
        got = cuda.attn_tiles_host(counts.numpy())
        assert all(torch.equal(a, torch.from_numpy(b).int()) for a, b in zip(want, got))
        kv = PagedKVCache(CacheGeometry(1, 1, 64, 16), rows, 400, 2, 0.5, "cpu")
        for depth in (0, 1):
            c = counts // (1 + 3 * depth)
            slots = kv.assign_prefill(depth, c)
            table, free = kv.page_table[depth].clone(), kv.free_count[depth].clone()
            kv.reset()
            t, s = kv.assign_fresh(depth, c.numpy())
            assert torch.equal(table, torch.from_numpy(t)) and torch.equal(slots, torch.from_numpy(s).int()) and torch.equal(free, kv.free_count[depth])
            kv.reset()
        for call in (lambda: kv.assign_prefill(0, counts * 50), lambda: kv.assign_fresh(0, counts.numpy() * 50)):
            try:
                call()
                raise AssertionError("accepted")
            except RuntimeError as e:
                assert "too small" in str(e)
        kv.reset()


def test_packed_tokens_of_masks_narrower_than_the_ids():
    """A mask's columns are the ids' first ones, whatever its pitch; the rows have to be the ids'."""
    import numpy as np
    import torch
    from tah_b200.engine.engine import packed_tokens
    gen = torch.Generator().manual_seed(0)
    ids = torch.randint(0, 1000, (3, 6), generator=gen)
    for width in (1, 4, 6):
        mask = torch.rand(3, width, generator=gen) < 0.7
        mask[:, 0] = True
        want = ids[mask.nonzero(as_tuple=True)]
        assert torch.equal(ids.reshape(-1)[torch.from_numpy(packed_tokens(mask.numpy(), 3, 6))], want)
    for bad in (np.ones((1, 6), bool), np.ones((4, 6), bool), np.ones(6, bool)):
        try:
            packed_tokens(bad, 3, 6)
            raise AssertionError("accepted")
        except ValueError as e:
            assert "attention mask" in str(e)


def test_reused_tick_state_clears_the_kernels_counters():
    """A cached tick state starts as a new one does: its scheduler tensors and the counters of its kernels are zero."""
    import types
    import torch
    from tah_b200.engine.base import DecodeEngine
    names = "tok depth pos finished n_out out_tokens iter_sum cur_iters slot gate tokens_done need_soft best sampled".split()
    s = types.SimpleNamespace(**{n: torch.ones(2, dtype=torch.int32) for n in names}, counters=[torch.tensor([5, 3], dtype=torch.int32)])
    eng = types.SimpleNamespace(hard_override=None, _states={(2, 8, None, None, None): s})
    assert DecodeEngine._tick_state(eng, 2, 8, None, None) is s
    assert all(not t.any() for t in [getattr(s, n) for n in names] + s.counters)


def test_host_arrays_keep_nothing_alive():
    """Arrays sent in one copy, with what runs behind it: the values arrive, and what the functions hold (an engine and its caches) is freed by
    the last reference, not by the cycle collector."""
    import gc
    import weakref
    import numpy as np
    import torch
    from tah_b200.engine.engine import HostArrays

    class Holder:
        pass

    def send(holder):
        up = HostArrays()
        a, b = up.put([1, 2, 3], np.int32), up.put(np.arange(5), np.int64)
        up.then(lambda: setattr(holder, "got", a() + 1))
        up.send("cpu")
        assert holder.got.tolist() == [2, 3, 4] and b().tolist() == [0, 1, 2, 3, 4] and b().dtype == torch.int64
        return weakref.ref(holder)

    gc.disable()
    try:
        alive = send(Holder())
        assert alive() is None
    finally:
        gc.enable()
