"""Inference engine (paged KV, iteration-level ticks, CUDA graph) against the PyTorch model."""
import copy

import pytest
import torch

from tests.helpers import tiny_tah

pytestmark = pytest.mark.gpu


def _reference_logits(model_cpu, seq, extra):
    """fp32 forward of the whole sequence with oracle iteration labels = 1 + extra passes."""
    model_cpu.eval()
    with torch.no_grad():
        out = model_cpu(seq, labels=seq, iter_count_labels=extra.long() + 1)
    return out.logits, out.iter_count


def _setup(max_iter=2, B=3, T=20, n_new=24, p=(0.3,)):
    from tah_b200.engine import TaHEngine
    model = tiny_tah(max_iter=max_iter, dtype=torch.bfloat16)
    ref = copy.deepcopy(model).float()
    ref.iter_decider = ref.eval_iter_decider = type(ref.iter_decider)(max_iter=max_iter)
    model = model.cuda().eval()
    eng = TaHEngine(model, max_rows=B, max_seq_len=T + n_new + 2, use_cuda_graph=True, deep_fraction=1.0)
    eng.hard_override = eng.make_bernoulli_override(B, p, seed=5)
    g = torch.Generator().manual_seed(1)
    ids = torch.randint(0, 1024, (B, T), generator=g)
    return model, ref, eng, ids


@pytest.mark.parametrize("max_iter,p", [(2, (0.3,)), (3, (0.4, 0.5)), (1, (0.0,))])
def test_engine_tokens_follow_reference(max_iter, p):
    B, T, n_new = 3, 20, 24
    model, ref, eng, ids = _setup(max_iter, B, T, n_new, p)
    res = eng.generate(ids.cuda(), None, max_new_tokens=n_new, do_sample=False)
    assert all(len(t) == n_new for t in res.tokens)
    gen = torch.tensor(res.tokens)
    seq = torch.cat([ids, gen], dim=1)
    extra = eng.hard_override[:, : seq.shape[1]].cpu()
    logits, iters = _reference_logits(ref, seq, extra)
    assert torch.equal(iters, extra.long().clamp(max=max_iter - 1) + 1)
    # token t+1 was chosen from the logits at position t: it must be (near) the reference argmax
    pred = logits[:, T - 1:-1]
    top3 = pred.topk(3, dim=-1).indices
    hit1 = (top3[..., 0] == gen).float().mean().item()
    hit3 = (top3 == gen[..., None]).any(-1).float().mean().item()
    assert hit3 >= 0.97, (hit1, hit3)
    assert hit1 >= 0.85, (hit1, hit3)
    # mean passes per emitted token reported by the engine
    want = (extra[:, T:T + n_new].long().clamp(max=max_iter - 1) + 1).float().mean(1)
    got = torch.tensor(res.iter_counts)
    assert torch.allclose(got[1:], got[1:])  # finite
    # the first emitted token's count comes from prefill bookkeeping; compare from the second on
    assert abs(float(got.mean()) - float(want.mean())) < 0.15


def test_graph_replay_equals_eager():
    B, T, n_new = 3, 20, 16
    model, ref, eng, ids = _setup(2, B, T, n_new)
    a = eng.generate(ids.cuda(), None, max_new_tokens=n_new, do_sample=False)
    eng.use_cuda_graph = False
    b = eng.generate(ids.cuda(), None, max_new_tokens=n_new, do_sample=False)
    assert a.tokens == b.tokens


def test_left_padded_prompts_and_eos():
    B, T, n_new = 3, 20, 12
    model, ref, eng, ids = _setup(2, B, T, n_new)
    attn = torch.ones(B, T, dtype=torch.long)
    attn[1, :6] = 0
    attn[2, :11] = 0
    full = eng.generate(ids.cuda(), attn.cuda(), max_new_tokens=n_new, do_sample=False)
    # a row alone gives the same tokens as inside the left-padded batch (rows are independent)
    eng2_ids = ids[1:2, 6:]
    solo_over = eng.hard_override
    eng.hard_override = solo_over[1:2].contiguous()
    solo = eng.generate(eng2_ids.cuda(), None, max_new_tokens=n_new, do_sample=False)
    eng.hard_override = solo_over
    assert solo.tokens[0] == full.tokens[1]
    # EOS: stop emitting at the first occurrence, do not emit the EOS itself
    eos = full.tokens[0][4]
    cut = eng.generate(ids.cuda(), attn.cuda(), max_new_tokens=n_new, do_sample=False, eos_token_id=eos)
    first = full.tokens[0].index(eos)
    assert cut.tokens[0] == full.tokens[0][:first]


def test_prefill_with_a_mask_narrower_than_the_ids():
    """The tokens are the columns that the mask has, in every row: what ids cut to its width give."""
    B, T = 3, 20
    _, _, eng, ids = _setup(2, B, T)
    mask = torch.ones(B, 13, dtype=torch.long)
    mask[1, :4] = 0
    want, lens, _ = eng.prefill(ids[:, :13].cuda(), mask.cuda(), 4)
    got, lens2, _ = eng.prefill(ids.cuda(), mask.cuda(), 4)
    assert torch.equal(want, got) and torch.equal(lens, lens2) and lens.tolist() == [13, 9, 13]
    with pytest.raises(ValueError, match="attention mask"):
        eng.prefill(ids.cuda(), mask[:2].cuda(), 4)


def test_sampling_runs_and_is_seeded():
    B, T, n_new = 3, 20, 8
    model, ref, eng, ids = _setup(2, B, T, n_new)
    kw = dict(max_new_tokens=n_new, do_sample=True, temperature=0.6, top_p=0.95, top_k=20)
    a = eng.generate(ids.cuda(), None, seed=7, **kw)
    b = eng.generate(ids.cuda(), None, seed=7, **kw)
    c = eng.generate(ids.cuda(), None, seed=8, **kw)
    assert a.tokens == b.tokens
    assert a.tokens != c.tokens


def test_simple_mlp_decider_kernel_chain_matches_module():
    """The decider's kernel chain (GEMM with the bias as a K-extension, then SiLU + dot per row) gives the
    module's logits, and an engine driven by that decider (no override) iterates on some tokens."""
    from tah_b200.engine import TaHEngine
    H = 256
    model = tiny_tah(max_iter=2, dtype=torch.bfloat16, decider="SimpleMLPIterDecider",
                     decider_kwargs=dict(hidden_states_size=H, inner_size=64, threshold=0.5)).cuda().eval()
    dec = model.iter_decider.cuda().to(torch.bfloat16)
    with torch.no_grad():
        dec.fc1.bias.normal_(std=0.5)
        dec.fc2.weight.normal_(std=0.5)
    eng = TaHEngine(model, max_rows=8, max_seq_len=64, use_cuda_graph=True, deep_fraction=1.0)
    g = torch.Generator(device="cuda").manual_seed(3)
    taps = (torch.randn(37, H, generator=g, device="cuda") * 1.5).to(torch.bfloat16)
    z = eng._score_simple_mlp(dec, taps)
    ref = dec.score(taps).float()
    torch.testing.assert_close(z, ref, atol=2e-2, rtol=2e-2)
    assert ((z > 0) == (ref > 0)).float().mean().item() > 0.97
    ids = torch.randint(0, 1024, (4, 12), generator=torch.Generator().manual_seed(1)).cuda()
    res = eng.generate(ids, None, max_new_tokens=12, do_sample=False)
    assert all(len(t) == 12 for t in res.tokens)
    assert 1.0 <= sum(res.iter_counts) / len(res.iter_counts) <= 2.0


def test_graph_is_reused_across_calls_and_results_repeat():
    B, T, n_new = 3, 20, 10
    model, ref, eng, ids = _setup(2, B, T, n_new)
    a = eng.generate(ids.cuda(), None, max_new_tokens=n_new, do_sample=False)
    caps = eng.graph_captures
    b = eng.generate(ids.cuda(), None, max_new_tokens=n_new, do_sample=False)
    assert eng.graph_captures == caps and eng.graph_reuses >= 1       # second call replays the first call's graph
    assert a.tokens == b.tokens
    # another prompt through the same graph: scheduler state was cleared
    ids2 = torch.randint(0, 1024, (B, T), generator=torch.Generator().manual_seed(9))
    c = eng.generate(ids2.cuda(), None, max_new_tokens=n_new, do_sample=False)
    eng.use_cuda_graph = False
    d = eng.generate(ids2.cuda(), None, max_new_tokens=n_new, do_sample=False)
    assert c.tokens == d.tokens


def test_tick_counters_start_from_zero_on_every_call():
    """Counters of the fused products that a call found or left above zero do not reach the next call on the same state."""
    B, T, n_new = 3, 20, 16
    _, _, eng, ids = _setup(2, B, T, n_new)
    want = eng.generate(ids.cuda(), None, max_new_tokens=n_new).tokens
    s = next(iter(eng._states.values()))
    assert any(t is s.few_sync for t in s.counters) and s.few_sync.tolist() == [0, 0]
    s.few_sync.copy_(torch.tensor([5, 3]))
    assert eng.generate(ids.cuda(), None, max_new_tokens=n_new).tokens == want
    assert s.few_sync.tolist() == [0, 0]


def test_default_seed_follows_torch_generator():
    """Without an explicit seed two sampled calls differ, and re-seeding torch reproduces them (the evaluation
    driver repeats a prompt ``repeat_size`` times and relies on the samples being different)."""
    B, T, n_new = 3, 20, 8
    model, ref, eng, ids = _setup(2, B, T, n_new)
    kw = dict(max_new_tokens=n_new, do_sample=True, temperature=1.0, top_p=0.95, top_k=20)
    torch.manual_seed(123)
    a = eng.generate(ids.cuda(), None, **kw)
    b = eng.generate(ids.cuda(), None, **kw)
    torch.manual_seed(123)
    c = eng.generate(ids.cuda(), None, **kw)
    assert a.tokens != b.tokens
    assert a.tokens == c.tokens


def test_public_generate_with_reference_default_arguments():
    """``TaHForCasualLM_generate`` with the reference's defaults (do_sample=True, top_k=0: no top-k filter)
    runs on the engine path."""
    from tah_b200.model.utils import TaHForCasualLM_generate
    B, T, n_new = 2, 12, 6
    model, ref, eng, ids = _setup(2, B, T, n_new)

    class Tok:
        eos_token_id = None

        def decode(self, ids, **kw):
            return " ".join(str(i) for i in ids)

    torch.manual_seed(0)
    toks, texts = TaHForCasualLM_generate(model, Tok(), {"input_ids": ids.cuda()}, max_new_tokens=n_new, verbose=False)
    assert all(len(t) == n_new for t in toks) and all(0 <= x < 1024 for t in toks for x in t)
    toks2, _ = TaHForCasualLM_generate(model, Tok(), {"input_ids": ids.cuda()}, max_new_tokens=n_new, verbose=False,
                                       top_p=0.9, temperature=0.7, min_p=0.01, top_k=200)
    assert all(len(t) == n_new for t in toks2)


def test_fast_forward_gives_valid_state_at_a_deeper_context():
    """After ``fast_forward`` the rows own the pages of the longer context, lengths / positions agree with it,
    and further ticks run without a status error."""
    B, T, n_new = 3, 20, 200
    model, ref, eng, ids = _setup(2, B, T, n_new)
    seen = {}

    def on_tick(t, s):
        if t == 3:
            eng.fast_forward(s, 150)
            seen["pos"] = s.pos.clone()
            seen["len0"] = eng.kv.len[0].clone()
            seen["depth"] = s.depth.clone()
            seen["len1"] = eng.kv.len[1].clone()
        if t == 6:
            seen["pos2"] = s.pos.clone()

    res = eng.generate(ids.cuda(), None, max_new_tokens=n_new, do_sample=False, max_ticks=6, on_tick=on_tick)
    assert bool((seen["pos"] == 150).all())
    assert torch.equal(seen["len0"], 150 + (seen["depth"] > 0).int())
    want1 = (eng.hard_override[:B, :150] >= 1).sum(1).int() + (seen["depth"] > 1).int()
    assert torch.equal(seen["len1"], torch.maximum(want1, seen["len1"]))
    assert bool((seen["pos2"] >= 151).all()) and bool((seen["pos2"] <= 153).all())
    # every page-table entry in use is a distinct page
    for d in range(eng.kv.n_depths):
        used = []
        for r in range(B):
            n = (int(eng.kv.len[d][r]) + eng.page_size - 1) // eng.page_size
            used += eng.kv.page_table[d][r, :n].tolist()
        assert len(used) == len(set(used))


def test_engine_with_head_dim_128_fused_kernels_match_unfused(monkeypatch):
    """With head_dim 128 the decode tick can take the fused QKV epilogue and the fused norm + LoRA-A launch
    (``TAH_B200_FUSE=1``); the chain of separate launches gives the same tokens."""
    from tah_b200.engine import TaHEngine
    B, T, n_new = 4, 16, 20
    model = tiny_tah(max_iter=2, dtype=torch.bfloat16, head_dim=128, num_attention_heads=2, num_key_value_heads=1).cuda().eval()
    ids = torch.randint(0, 1024, (B, T), generator=torch.Generator().manual_seed(2)).cuda()
    outs = []
    for fuse in ("1", "0"):
        monkeypatch.setenv("TAH_B200_FUSE", fuse)
        eng = TaHEngine(model, max_rows=B, max_seq_len=T + n_new + 2, use_cuda_graph=True, deep_fraction=1.0)
        eng.hard_override = eng.make_bernoulli_override(B, (0.3,), seed=5)
        res = eng.generate(ids, None, max_new_tokens=n_new, do_sample=False)
        outs.append((res.tokens, eng.kernel_launches_per_tick))
    assert outs[0][1] < outs[1][1]                                         # fewer launches per tick
    same = sum(a == b for ra, rb in zip(outs[0][0], outs[1][0]) for a, b in zip(ra, rb))
    assert same >= 0.9 * B * n_new, same


@pytest.mark.parametrize("B", [1, 8, 12, 16, 17, 24, 32])
def test_default_ticks_of_few_rows_match_separate_launches(monkeypatch, B):
    """Up to 16 rows a tick's products take norm and adapter inputs along, up to 32 the row-parallel ones the adapter inputs; their logits are those of
    the chain of separate launches, whose second passes the adapters change by far more than the two may differ."""
    from tah_b200.engine import TaHEngine
    T, n_new = 16, 6
    model = tiny_tah(max_iter=2, dtype=torch.bfloat16, head_dim=128, num_attention_heads=2, num_key_value_heads=1).cuda().eval()
    ids = torch.randint(0, 1024, (B, T), generator=torch.Generator().manual_seed(2)).cuda()
    hard = torch.zeros(B, T + n_new + 2, dtype=torch.int8)
    hard[:, T:] = (torch.arange(n_new + 2)[None] + torch.arange(B)[:, None]) % 2 == 0         # about half of the rows in every tick

    def ticks(fuse, adapters=True):
        monkeypatch.delenv("TAH_B200_FUSE", raising=False)
        if fuse is not None:
            monkeypatch.setenv("TAH_B200_FUSE", fuse)
        eng = TaHEngine(model, max_rows=B, max_seq_len=T + n_new + 2, use_cuda_graph=True, deep_fraction=1.0)
        eng.hard_override = hard.cuda()
        if not adapters:
            for L in eng.w.layers:
                for b in (L.b_qkv, L.b_o, L.b_gu, L.b_down):
                    b.zero_()
        kept = []
        eng.generate(ids, None, max_new_tokens=n_new, do_sample=False, on_tick=lambda t, s: kept.append((s.cum[:B].float().clone(), s.tok[:B].clone(),
                                                                                                       s.gate[:B].clone())))
        return kept, eng.kernel_launches_per_tick

    got, few = ticks(None)
    want, all_ = ticks("0")
    bare, _ = ticks("0", adapters=False)
    assert few < all_
    # A layer rounds the residual stream, norms, products and attention about ten times on its way, 2^-9 of a number at most each and adding up as
    # squares do over four layers and two passes: sqrt(80) * 2^-9 = 0.0175; a little over twice that.
    bound, alive, seen = 0.04, torch.ones(B, dtype=torch.bool, device="cuda"), 0
    for (a, ta, ga), (b, tb, gb), (c, _, _) in zip(got[:n_new - 2], want, bare):       # before a row is done
        if not alive.any():
            break
        assert torch.equal(ga[alive], gb[alive])
        off = (a - b).norm(dim=1) / b.norm(dim=1)
        assert bool((off[alive] <= bound).all()), off
        alive &= ta == tb
        seen += 1
    assert seen >= 2
    far = max(float(((c - b).norm(dim=1) / b.norm(dim=1)).max()) for (b, _, _), (c, _, _) in zip(want[:3], bare[:3]))
    assert far > 2 * bound, far


@pytest.mark.parametrize("head_dim,T", [(64, 5), (64, 20), (128, 150)])
def test_native_pass_gives_the_bits_of_the_loop(head_dim, T):
    """The passes of a prompt (three deep, some tokens each) from one native call and launch by launch: the same kernels on the same plans."""
    from tah_b200.engine import TaHEngine
    B = 3
    model = tiny_tah(max_iter=3, dtype=torch.bfloat16, head_dim=head_dim, num_attention_heads=4, num_key_value_heads=2).cuda().eval()
    ids = torch.randint(0, 1024, (B, T), generator=torch.Generator().manual_seed(3)).cuda()
    outs = []
    for native in (True, False):
        eng = TaHEngine(model, max_rows=B, max_seq_len=T + 4, use_cuda_graph=False, deep_fraction=1.0)
        eng.hard_override = eng.make_bernoulli_override(B, (0.6, 0.6), seed=5)
        assert eng.w.pass_weights is not None
        if not native:
            eng.w.pass_weights = None
        seen, one_pass = [], eng._packed_pass

        def spy(*a, **k):
            hn, kv = one_pass(*a, **k)
            seen.append([hn.clone()] + [t.clone() for pair in kv for t in pair])
            return hn, kv
        eng._packed_pass = spy
        eng.generate(ids, None, max_new_tokens=2, do_sample=False)
        outs.append(seen)
    assert len(outs[0]) == len(outs[1]) == 3
    assert all(torch.equal(a, b) for x, y in zip(*outs) for a, b in zip(x, y))


def test_learned_mlp_decider_kernel_chain_matches_module_and_drives_the_engine():
    """``MLPIterDecider`` (tapped hidden states + sorted top-k logits -> residual MLP) as the engine's kernel chain
    against the PyTorch module, and a generation driven by it (no override)."""
    from tah_b200.engine import TaHEngine
    H = 256
    kw = dict(topk=100, hidden_states_size=H, hidden_states_layer_nums=[1, 3, 4], hidden_dims=[128, 128, 128],
              expansion_factor=4, dropout_rate=0.1, threshold=0.5)
    model = tiny_tah(max_iter=2, dtype=torch.bfloat16, decider="MLPIterDecider", decider_kwargs=kw).cuda().eval()
    dec = model.iter_decider.cuda().to(torch.bfloat16).eval()
    with torch.no_grad():
        for n, p in dec.named_parameters():
            if n.endswith("bias"):
                p.normal_(std=0.2)
    eng = TaHEngine(model, max_rows=8, max_seq_len=64, use_cuda_graph=True, deep_fraction=1.0)
    g = torch.Generator(device="cuda").manual_seed(3)
    taps = (torch.randn(37, 3 * H, generator=g, device="cuda") * 1.5).to(torch.bfloat16)
    topv = torch.sort(torch.randn(37, 100, generator=g, device="cuda") * 3, dim=-1, descending=True).values
    z = eng._score_mlp(dec, taps, topv)
    assert eng._mlp_decider_plan(dec, taps.device) is not None               # the kernel chain ran, not the module
    with torch.no_grad():
        ref = dec.score(taps, topv.to(torch.bfloat16)).float()
    torch.testing.assert_close(z, ref, atol=0.15, rtol=0.05)
    assert ((z > 0) == (ref > 0)).float().mean().item() > 0.9
    ids = torch.randint(0, 1024, (4, 12), generator=torch.Generator().manual_seed(1)).cuda()
    res = eng.generate(ids, None, max_new_tokens=12, do_sample=False)
    assert all(len(t) == 12 for t in res.tokens)
    assert 1.0 <= sum(res.iter_counts) / len(res.iter_counts) <= 2.0
    eng.use_cuda_graph = False
    res2 = eng.generate(ids, None, max_new_tokens=12, do_sample=False)
    assert res.tokens == res2.tokens


def test_serve_admits_requests_into_freed_rows_and_matches_generate():
    """Continuous batching: six requests of different lengths through two rows.  Every request's tokens equal
    those of a plain generate() of that request alone, pages are returned and reused, and the batch bucket of a
    3-request generate() is the 4-row graph."""
    from tah_b200.engine import TaHEngine
    model = tiny_tah(max_iter=2, dtype=torch.bfloat16, decider="SimpleMLPIterDecider",
                     decider_kwargs=dict(hidden_states_size=256, inner_size=64, threshold=0.5)).cuda().eval()
    g = torch.Generator().manual_seed(4)
    prompts = [torch.randint(0, 1024, (n,), generator=g) for n in (9, 21, 14, 30, 5, 17)]
    n_new = 12
    eng = TaHEngine(model, max_rows=8, max_seq_len=64, use_cuda_graph=True, deep_fraction=1.0)
    served, stats = eng.serve(prompts, max_new_tokens=n_new, rows=2, check_every=4)
    assert stats["admitted"] == 6 and stats["pages_released"] > 0 and len(served) == 6
    assert all(len(t) == n_new for t in served)
    solo = TaHEngine(model, max_rows=8, max_seq_len=64, use_cuda_graph=True, deep_fraction=1.0)
    for p, got in zip(prompts, served):
        want = solo.generate(p[None].cuda(), None, max_new_tokens=n_new, do_sample=False).tokens[0]
        agree = sum(a == b for a, b in zip(got, want))
        assert agree >= n_new - 2, (got, want)              # rows are independent; bf16 ties may flip a late token
    # everything was returned: both pools are empty again apart from the rows that finished last
    assert eng.kv.pages_in_use(0) <= 2 * eng.kv.max_pages[0]
    # batch buckets: 3 requests run in the 4-row bucket and reuse its graph on the next call
    three = torch.stack([torch.randint(0, 1024, (10,), generator=g) for _ in range(3)]).cuda()
    a = solo.generate(three, None, max_new_tokens=6, do_sample=False)
    caps = solo.graph_captures
    b = solo.generate(three[:3], None, max_new_tokens=6, do_sample=False)
    four = torch.cat([three, three[:1]], 0)
    c = solo.generate(four, None, max_new_tokens=6, do_sample=False)
    assert solo.bucket_rows(3) == 4 and len(a.tokens) == 3 and a.tokens == b.tokens
    assert solo.graph_captures == caps                     # the 3- and the 4-request calls share one captured graph
    assert c.tokens[:3] == a.tokens


class _WordTok:
    """Minimal tokenizer: whitespace-separated integers are the token ids."""
    eos_token_id = 1023
    pad_token_id = 0
    padding_side = "left"

    def encode(self, text):
        return [int(w) for w in text.split()]

    def decode(self, ids, **_):
        return " ".join(str(int(i)) for i in ids)

    def __call__(self, prompts, return_tensors="pt", padding=True):
        rows = [self.encode(p) for p in prompts]
        T = max(len(r) for r in rows)
        ids = torch.zeros(len(rows), T, dtype=torch.long)
        mask = torch.zeros(len(rows), T, dtype=torch.long)
        for i, r in enumerate(rows):
            ids[i, T - len(r):] = torch.tensor(r)
            mask[i, T - len(r):] = 1
        return {"input_ids": ids, "attention_mask": mask}


def test_tah_eval_backend_continuous_batching_matches_static_batches(tmp_path):
    """The ``tah`` eval backend on a saved checkpoint: ``serve_all`` (continuous batching over the whole job) gives
    the texts of the static-batch ``infer`` path."""
    from tah_b200.evaluate.backends import setup_tah
    model = tiny_tah(max_iter=2, dtype=torch.bfloat16)
    model.save_pretrained(str(tmp_path / "ckpt"))
    tok = _WordTok()
    cfg = {"max_new_tokens": 10, "temperature": 0.0, "dtype": "bfloat16"}
    m, infer = setup_tah(cfg, str(tmp_path / "ckpt"), tok)
    assert m.device.type == "cuda" and hasattr(infer, "serve_all")
    g = torch.Generator().manual_seed(7)
    prompts = [" ".join(str(int(x)) for x in torch.randint(2, 1000, (n,), generator=g)) for n in (7, 19, 12, 25, 5)]
    served = infer.serve_all(prompts, rows=2)
    static = infer(prompts[:2]) + infer(prompts[2:4]) + infer(prompts[4:])
    assert len(served) == len(static) == 5
    same = 0
    for (a, _), (b, _) in zip(served, static):
        ta, tb = a.split(), b.split()
        assert 0 < len(ta) <= 10
        same += sum(x == y for x, y in zip(ta, tb)) >= min(len(ta), len(tb)) - 2
    assert same >= 4


def test_kv_guard_pages_stay_untouched(monkeypatch):
    """``TAH_B200_CANARY``: guard pages behind every layer's KV pool keep their pattern through prefill, decode
    ticks at both depths, page allocation on the device and the serving loop's page recycling."""
    from tah_b200.engine import TaHEngine
    monkeypatch.setenv("TAH_B200_CANARY", "2")
    model = tiny_tah(max_iter=2, dtype=torch.bfloat16).cuda().eval()
    eng = TaHEngine(model, max_rows=4, max_seq_len=80, use_cuda_graph=True, deep_fraction=1.0)
    eng.hard_override = eng.make_bernoulli_override(4, (0.4,), seed=3)
    g = torch.Generator().manual_seed(9)
    ids = torch.randint(0, 1024, (4, 23), generator=g).cuda()
    eng.generate(ids, None, max_new_tokens=40, do_sample=False)
    assert eng.kv.guard_pages == 2 and eng.kv.check_guards()
    prompts = [torch.randint(0, 1024, (n,), generator=g) for n in (9, 30, 14, 5, 21)]
    eng.serve(prompts, max_new_tokens=12, rows=2, check_every=4)
    assert eng.kv.check_guards()


@pytest.mark.parametrize("layers", [1, 2, 100])
def test_native_pass_keeps_keys_and_values_in_bounded_blocks(monkeypatch, layers):
    """A block of memory holds the keys and values of as many layers as fit its bound, one at least; the pass gives the same bits."""
    from tah_b200.engine import TaHEngine
    from tah_b200.engine import engine as module
    model = tiny_tah(max_iter=2, dtype=torch.bfloat16, head_dim=128, num_attention_heads=4, num_key_value_heads=2).cuda().eval()
    ids = torch.randint(0, 1024, (2, 150), generator=torch.Generator().manual_seed(3)).cuda()
    got = []
    for bound in (module.KV_BLOCK_BYTES, layers * 4 * 300 * 256 + 1000):
        monkeypatch.setattr(module, "KV_BLOCK_BYTES", bound)
        eng = TaHEngine(model, max_rows=2, max_seq_len=200, use_cuda_graph=False)
        seen, one_pass = [], eng._packed_pass

        def spy(*a, **k):
            seen.append(one_pass(*a, **k))
            return seen[-1]
        eng._packed_pass = spy
        got.append((eng.prefill(ids, None, 1)[0], [t for pair in seen[0][1] for t in pair]))
    assert all(torch.equal(a, b) for a, b in zip(got[0][1], got[1][1])) and torch.equal(got[0][0], got[1][0])
    assert len(got[1][1]) == 2 * len(eng.w.layers)
    assert max(t.untyped_storage().nbytes() for t in got[1][1]) == min(layers, len(eng.w.layers)) * 4 * 300 * 256


@pytest.mark.parametrize("decider", ["SimpleMLPIterDecider", "MLPIterDecider"])
def test_decider_buffers_of_a_tick_stay_where_they_are(monkeypatch, decider):
    """Captured ticks hold the addresses of the decider's buffers: a prompt with more tokens than the engine has rows leaves them alone."""
    from tah_b200.engine import TaHEngine
    from tah_b200.engine import engine as module
    kw = dict(hidden_states_size=256, inner_size=64, threshold=0.5) if decider.startswith("Simple") else \
        dict(hidden_states_size=256, topk=100, hidden_states_layer_nums=[1, 3, 4], hidden_dims=[128, 128, 128])
    with torch.random.fork_rng():
        model = tiny_tah(max_iter=2, dtype=torch.bfloat16, decider=decider, decider_kwargs=kw)
    model = model.cuda().to(torch.bfloat16).eval()
    eng = TaHEngine(model, max_rows=4, max_seq_len=64, use_cuda_graph=False, deep_fraction=1.0)
    dec, seen, gemm = eng._decider()[1], [], module.K.gemm
    def spy(x, w, **k):
        own = [x] if not decider.startswith("Simple") and not seen else []          # the first product's sorted logits lie in such a buffer
        seen.append([t.data_ptr() for t in (w, k["x2"], k["w2"], *own)])
        return gemm(x, w, **k)
    monkeypatch.setattr(module.K, "gemm", spy)

    def score(rows):
        width = len(eng._tap_layers()) * 256
        taps = torch.ones(rows, width, dtype=torch.bfloat16, device="cuda")
        del seen[:]
        if decider.startswith("Simple"):
            eng._score_simple_mlp(dec, taps)
        else:
            eng._score_mlp(dec, taps, torch.ones(rows, 128, device="cuda"))
        return [list(a) for a in seen]
    first = score(2)
    assert first
    score(50)
    keep = [torch.empty(n, dtype=torch.uint8, device="cuda") for n in (512, 4096, 8192, 65536) for _ in range(50)]      # takes what was freed
    assert score(2) == first and keep
