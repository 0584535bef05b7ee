"""Engine-level parity (GPU), through the C ABI: prefill + decode of the Qwen3 architecture against
the oracle (HF transformers Qwen3 on CPU and its pinned restatement), on identical weights and
inputs.  Tolerances: greedy token ids identical (tie-aware: a mismatch is only
tolerated where the oracle's own top-1/top-2 logit gap is within bf16 noise), logits and per-layer
hidden states within 1e-2 relative."""
import ctypes as C
import importlib
import json
import os

import numpy as np
import pytest
import torch

from _util import ROOT, bf16_ulp_of, engine_config_from_arch, pkg, record_parity, rel_err, rel_fro
from oracle.qwen3_oracle import (QWEN3_0_6B, QWEN3_TINY, KVState, Restated, attention_explicit, hf_model, hf_state_dict,
                                 make_prompts, perturb_norm_weights, random_weights, rope_inv_freq, top2_gap)

pytestmark = pytest.mark.gpu
GOLD = os.path.join(ROOT, "tests", "golden")
REL_TOL = 1e-2  # "per-layer bf16 logits must agree within 1e-2 relative"


@pytest.fixture(scope="module")
def P():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return pkg()


def bits_to_bf16(bits: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(bits.astype(np.int16)).view(torch.bfloat16)


@pytest.fixture(scope="module")
def tiny(P):
    model = hf_model(QWEN3_TINY, seed=0)
    sd = hf_state_dict(model)
    perturb_norm_weights(sd)
    model.load_state_dict(sd)
    return model, sd


def make_engine(P, arch, sd, **kw):
    cfg = engine_config_from_arch(P, arch, **kw)
    e = P.Engine(cfg, rope_inv_freq=rope_inv_freq(arch).numpy())
    e.load_state_dict(sd)
    return e


@pytest.mark.parametrize("graphs", [False, True])
def test_tiny_prefill_decode_matches_oracle(P, tiny, graphs):
    model, sd = tiny
    arch = QWEN3_TINY
    g = np.load(os.path.join(GOLD, "qwen3_tiny.npz"))
    prompts = g["prompt_ids"]  # [3][48]
    gold = g["greedy_ids"]     # [3][32] from HF generate
    e = make_engine(P, arch, sd, max_model_len=256, num_blocks=64, max_seqs=8, max_batch_tokens=512, use_cuda_graphs=graphs)
    if not graphs:
        e.set_debug(hidden=True, logits=True)
    sids = [e.seq_create(128) for _ in range(3)]
    first = e.prefill(sids, [p.tolist() for p in prompts])
    if not graphs:
        # per-layer residual stream of the prefill vs HF's output_hidden_states
        hid = g["hidden_bf16"]  # [L+1][3][80][H] (teacher-forced over prompt+generated)
        T = 3 * 48
        for layer in range(-1, arch.num_layers):
            got = bits_to_bf16(e.get_hidden(layer, T)).view(3, 48, arch.hidden)
            if layer == arch.num_layers - 1:
                continue  # HF reports the last layer post-norm; covered through the logits below
            ref = bits_to_bf16(hid[layer + 1][:, :48])
            assert rel_err(got, ref) < REL_TOL, "hidden after layer %d" % layer
        logits = torch.from_numpy(e.get_logits(3))
        ref_logits = bits_to_bf16(g["logits_bf16"])[:, 47].float()
        assert rel_err(logits, ref_logits) < REL_TOL
    toks = [first]
    for _ in range(gold.shape[1] - 1):
        toks.append(e.decode_step(sids))
    got = np.stack(toks, axis=1)
    # tie-aware comparison against HF greedy ids
    r = Restated(arch, sd)
    _, step_logits = r.greedy(torch.from_numpy(prompts).long(), gold.shape[1])
    gaps = top2_gap(step_logits)
    for b in range(3):
        for t in range(gold.shape[1]):
            if got[b, t] != gold[b, t]:
                assert gaps[b, t] <= 0.0625, "seq %d step %d: token %d != %d with oracle gap %.4f" % (
                    b, t, got[b, t], gold[b, t], gaps[b, t])
                break  # after a tie-flip the continuations legitimately differ
    assert (got[:, :8] == gold[:, :8]).mean() > 0.9
    for s in sids:
        e.seq_free(s)
    e.close()


def test_tiny_chain_path_matches_oracle(P, tiny, monkeypatch):
    """The persistent chain kernel (chain.cu, B2_CHAIN=1) is an alternative schedule of the same
    arithmetic: it must reproduce HF's greedy ids like the default path does."""
    monkeypatch.setenv("B2_CHAIN", "1")
    model, sd = tiny
    g = np.load(os.path.join(GOLD, "qwen3_tiny.npz"))
    prompts, gold = g["prompt_ids"], g["greedy_ids"]
    e = make_engine(P, QWEN3_TINY, sd, max_model_len=256, num_blocks=64, max_seqs=8, max_batch_tokens=512, use_cuda_graphs=True)
    sids = [e.seq_create(128) for _ in range(3)]
    first = e.prefill(sids, [p.tolist() for p in prompts])
    toks, _ = e.decode_run(sids, 31)
    got = np.concatenate([first[None, :], toks], axis=0).T   # [3][32]
    for i in range(3):
        n = 0
        while n < 32 and got[i, n] == gold[i, n]:
            n += 1
        assert n >= 16, "sequence %d: chain path agrees with HF on only %d leading tokens" % (i, n)
    e.close()


def test_tiny_batch_invariance_and_ragged(P, tiny):
    """Ragged prompts in one prefill + batched decode must equal each sequence run alone."""
    model, sd = tiny
    arch = QWEN3_TINY
    g = torch.Generator().manual_seed(5)
    lens = [1, 17, 64, 65, 130]
    prompts = [torch.randint(0, arch.vocab, (n,), generator=g).tolist() for n in lens]
    e = make_engine(P, arch, sd, max_model_len=512, num_blocks=128, max_seqs=8, max_batch_tokens=512, use_cuda_graphs=False)
    e.set_debug(logits=True)
    sids = [e.seq_create(200) for _ in lens]
    first = e.prefill(sids, prompts)
    batch_logits = e.get_logits(len(lens)).copy()
    steps = [first] + [e.decode_step(sids) for _ in range(6)]
    batched = np.stack(steps, axis=1)
    for s in sids:
        e.seq_free(s)
    r = Restated(arch, sd, attention=attention_explicit)
    for i, p in enumerate(prompts):
        sid = e.seq_create(200)
        f = e.prefill([sid], [p])
        solo_logits = e.get_logits(1)[0]
        # the batched prefill and the solo one take different projection tiles / K splits (fp32 sums in another order),
        # so activations round to the neighbouring bf16 here and there and two layers carry that into the logits: the bar is
        # the one the oracle comparison below uses, not bit equality (one bf16 ulp of the largest logit alone is 3.9e-3)
        assert rel_err(torch.from_numpy(batch_logits[i]), torch.from_numpy(solo_logits)) < REL_TOL
        ref_logits, _ = r.forward(torch.tensor([p]), torch.arange(len(p))[None], KVState(), last_only=True)
        assert rel_err(torch.from_numpy(solo_logits), ref_logits[0, 0].float()) < REL_TOL, "prompt len %d" % len(p)
        solo = [f] + [e.decode_step([sid]) for _ in range(6)]
        solo = np.concatenate(solo)
        if not np.array_equal(solo, batched[i]):
            # only a near-tie may differ between batch compositions (different split-K / tile shapes)
            k = int(np.argmax(solo != batched[i]))
            assert k > 0
        e.seq_free(sid)
    e.close()


def test_tiny_decode_run_equals_stepwise(P, tiny):
    """b2_decode_run (device-resident token feedback, CUDA graph) == b2_decode_step loop."""
    model, sd = tiny
    arch = QWEN3_TINY
    prompts = make_prompts(4, 33, arch.vocab, seed=3)
    outs = []
    for mode in ("step_eager", "step_graph", "run_graph"):
        e = make_engine(P, arch, sd, max_model_len=256, num_blocks=96, max_seqs=4, max_batch_tokens=256,
                        use_cuda_graphs=(mode != "step_eager"))
        sids = [e.seq_create(128) for _ in range(4)]
        e.prefill(sids, [p.tolist() for p in prompts])
        if mode == "run_graph":
            toks, ms = e.decode_run(sids, 40)
            assert ms > 0
        else:
            toks = np.stack([e.decode_step(sids) for _ in range(40)])
        assert e.seq_len(sids[0]) == 33 + 40
        outs.append(toks)
        e.close()
    assert np.array_equal(outs[0], outs[1]), "graph replay must equal eager launches"
    assert np.array_equal(outs[1], outs[2]), "device-side token feedback must equal host feedback"


def test_tiny_in_tokens_and_batch_change(P, tiny):
    """Teacher forcing through in_tokens, and a sequence leaving the batch mid-way."""
    model, sd = tiny
    arch = QWEN3_TINY
    gld = np.load(os.path.join(GOLD, "qwen3_tiny.npz"))
    prompts, gold = gld["prompt_ids"], gld["greedy_ids"]
    e = make_engine(P, arch, sd, max_model_len=256, num_blocks=64, max_seqs=8, max_batch_tokens=512, use_cuda_graphs=True)
    sids = [e.seq_create(128) for _ in range(3)]
    e.prefill(sids, [p.tolist() for p in prompts])
    agree = 0
    for t in range(10):  # feed HF's tokens: the engine's next-token must track HF's
        out = e.decode_step(sids, in_tokens=gold[:, t])
        agree += int((out == gold[:, t + 1]).sum())
    assert agree >= 27  # 30 comparisons; random-init logits have near-ties
    e.seq_free(sids[1])
    keep = [sids[0], sids[2]]
    out = e.decode_step(keep, in_tokens=gold[[0, 2], 10])
    assert out.shape == (2,)
    assert (out == gold[[0, 2], 11]).sum() >= 1
    e.close()


def test_sampling_modes(P, tiny):
    model, sd = tiny
    arch = QWEN3_TINY
    e = make_engine(P, arch, sd, max_model_len=128, num_blocks=32, max_seqs=4, max_batch_tokens=128, use_cuda_graphs=False)
    e.set_debug(logits=True)
    sid = e.seq_create(64)
    first = e.prefill([sid], [[1, 2, 3, 4, 5]])
    logits = e.get_logits(1)[0]
    assert int(first[0]) == int(np.argmax(logits))
    assert int(e.sample(1, temperature=0.0)[0]) == int(first[0])
    assert int(e.sample(1, temperature=1.0, top_k=1, seed=7)[0]) == int(first[0])
    top5 = set(np.argsort(-logits)[:5].tolist())
    draws = {int(e.sample(1, temperature=5.0, top_k=5, seed=s)[0]) for s in range(40)}
    assert draws <= top5 and len(draws) >= 2
    order = np.argsort(-logits)
    p = np.exp(logits - logits.max())
    p /= p.sum()
    nucleus = set(order[: int(np.searchsorted(np.cumsum(p[order]), 0.5)) + 1].tolist())
    draws = {int(e.sample(1, temperature=1.0, top_p=0.5, seed=s)[0]) for s in range(40)}
    assert draws <= nucleus
    e.close()


def test_errors_are_reported(P, tiny):
    model, sd = tiny
    e = make_engine(P, QWEN3_TINY, sd, max_model_len=64, num_blocks=8, max_seqs=2, max_batch_tokens=64, use_cuda_graphs=False)
    with pytest.raises(P.B2Error):
        e.seq_create(65)            # beyond max_model_len
    a = e.seq_create(64)
    with pytest.raises(P.B2Error):
        e.seq_create(64)            # pool exhausted (8 pages, page 0 is the null page)
    with pytest.raises(P.B2Error):
        e.decode_step([a])          # nothing prefilled
    with pytest.raises(P.B2Error):
        e.prefill([a], [list(range(65))])
    with pytest.raises(P.B2Error):
        e.seq_free(5)
    e.close()


def test_a_refused_engine_leaves_the_others_alone(P, tiny):
    """An engine that does not fit into memory is an error of its own call: prompts, sampling, new decode batches and new engines behind it work as before."""
    _, sd = tiny
    sizes = dict(max_model_len=64, num_blocks=16, max_seqs=2, max_batch_tokens=64)
    e = make_engine(P, QWEN3_TINY, sd, **sizes)
    e.set_debug(logits=True)
    prompt = [[3 + i for i in range(20)]]

    def refuse():
        with pytest.raises(P.B2Error, match="cudaMalloc"):
            make_engine(P, QWEN3_TINY, sd, **dict(sizes, num_blocks=1 << 28))   # terabytes

    a = e.seq_create(40)
    want = [e.prefill([a], prompt), e.decode_step([a]), e.sample(1, temperature=1.0, top_p=0.5, seed=7)]
    e.seq_free(a)
    refuse()
    b = e.seq_create(40)
    got = [e.prefill([b], prompt)]
    refuse()
    got.append(e.decode_step([b]))
    refuse()
    got.append(e.sample(1, temperature=1.0, top_p=0.5, seed=7))
    for x, y in zip(got, want):
        assert (x == y).all()
    refuse()
    other = make_engine(P, QWEN3_TINY, sd, **sizes)
    assert (other.prefill([other.seq_create(40)], prompt) == want[0]).all()
    other.close()
    e.close()


# ---------------------------------------------------------------------------------------------
# Full-size architecture: batch 1, 128-token prompt -> 128 tokens
# ---------------------------------------------------------------------------------------------
@pytest.fixture(scope="module")
def full(P):
    model = hf_model(QWEN3_0_6B, seed=0)
    return model, hf_state_dict(model)


def test_full_c1_greedy_and_logits(P, full):
    model, sd = full
    arch = QWEN3_0_6B
    fx = json.load(open(os.path.join(GOLD, "qwen3_0p6b_c1.json")))
    prompt = fx["prompt_ids"]
    gold = np.array(fx["greedy_ids"])
    e = make_engine(P, arch, sd, max_model_len=512, num_blocks=64, max_seqs=4, max_batch_tokens=512, use_cuda_graphs=False)
    e.set_debug(hidden=True, logits=True)
    sid = e.seq_create(300)
    # teacher-forced: prefill prompt + HF's generated tokens in one pass, compare every layer
    full_ids = prompt + gold.tolist()
    e.prefill([sid], [full_ids])
    T = len(full_ids)
    with torch.no_grad():
        out = model(torch.tensor([full_ids]), output_hidden_states=True)
        # HF's own second attention implementation on the same weights: the bf16 noise floor of the
        # oracle itself (measured: sdpa vs eager at 1.5e-2 on the last layers)
        model.set_attn_implementation("eager")
        out_e = model(torch.tensor([full_ids]), output_hidden_states=True)
        model.set_attn_implementation("sdpa")
    worst = 0.0
    for layer in range(-1, arch.num_layers - 1):
        got = bits_to_bf16(e.get_hidden(layer, T))
        ref = out.hidden_states[layer + 1][0]
        err, fro = rel_err(got, ref), rel_fro(got, ref)
        floor, floor_fro = rel_err(out_e.hidden_states[layer + 1][0], ref), rel_fro(out_e.hidden_states[layer + 1][0], ref)
        print("layer %2d: engine vs HF max-rel %.4g fro-rel %.4g | HF eager vs HF sdpa max-rel %.4g fro-rel %.4g" % (
            layer, err, fro, floor, floor_fro))
        worst = max(worst, err)
        # bar: 1e-2 relative, or -- where HF's own two attention paths already disagree by more than
        # that -- no worse than 1.5x the oracle's own disagreement at this layer
        assert err < max(REL_TOL, 1.5 * floor), "hidden after layer %d: rel err %.4g (oracle floor %.4g)" % (layer, err, floor)
        assert fro < max(REL_TOL, 1.5 * floor_fro), "hidden after layer %d: fro err %.4g (oracle floor %.4g)" % (layer, fro, floor_fro)
    lg = torch.from_numpy(e.get_logits(1))[0]
    lerr = rel_err(lg, out.logits[0, -1].float())
    lfloor = rel_err(out_e.logits[0, -1].float(), out.logits[0, -1].float())
    print("last-position logits: engine vs HF max-rel %.4g | HF eager vs sdpa %.4g" % (lerr, lfloor))
    assert lerr < max(REL_TOL, 1.5 * lfloor)
    e.seq_free(sid)

    # greedy decode from the prompt
    sid = e.seq_create(300)
    toks = [int(e.prefill([sid], [prompt])[0])]
    for _ in range(127):
        toks.append(int(e.decode_step([sid])[0]))
    toks = np.array(toks)
    top4 = np.array(fx["tf_top4_logits"])  # teacher-forced HF logits at positions 0..255
    mism = np.nonzero(toks != gold)[0]
    n_match = 128 if len(mism) == 0 else int(mism[0])
    print("C1 greedy: %d/128 leading tokens identical to HF; worst hidden rel err %.3g" % (n_match, worst))
    # the same 128 steps teacher-forced with HF's tokens: how many of the engine's tokens equal HF's when every step sees
    # HF's context (a free-running stream stops being comparable at its first tie flip)
    sid2 = e.seq_create(300)
    tf = [int(e.prefill([sid2], [prompt])[0])]
    for t in range(1, 128):
        tf.append(int(e.decode_step([sid2], in_tokens=[int(gold[t - 1])])[0]))
    tf = np.array(tf)
    tf_mism = np.nonzero(tf != gold)[0]
    for t in tf_mism:
        gap_t = float(top4[127 + t][0] - top4[127 + t][1])
        assert gap_t <= 2 * bf16_ulp_of(float(top4[127 + t][0])), "teacher-forced step %d differs from HF where its top-2 gap is %.4f" % (t, gap_t)
    rec = {"leading_match": n_match, "of": 128, "teacher_forced_equal": int(128 - len(tf_mism)), "teacher_forced_differing_steps": tf_mism.tolist(),
           "worst_hidden_rel_err": float(worst), "last_logits_rel_err": float(lerr), "last_logits_floor": float(lfloor)}
    if len(mism):
        # north_star: identical over the first 128 tokens; the only divergence tolerated is at a step where HF's own
        # top-2 gap is within 2 bf16 ulp of its top logit (HF's two attention paths flip such a step themselves)
        t = int(mism[0])
        gap = float(top4[127 + t][0] - top4[127 + t][1])
        ulp = bf16_ulp_of(float(top4[127 + t][0]))
        rec.update({"first_mismatch_step": t, "hf_top2_gap": gap, "gap_in_bf16_ulp_of_top1": gap / ulp})
        record_parity("c1_batch1_prompt128", rec)
        assert gap <= 2 * ulp, "first mismatch at step %d where the oracle's top-2 gap is %.4f = %.1f bf16 ulp (not a tie)" % (
            t, gap, gap / ulp)
    record_parity("c1_batch1_prompt128", rec)
    e.close()


@pytest.mark.parametrize("chain", ["1", "2"])
def test_full_alternative_decode_schedules(P, full, monkeypatch, chain):
    """The two experimental decode schedules -- chain.cu (B2_CHAIN=1: eight steps behind grid barriers) and
    chain_cluster.cu (B2_CHAIN=2: four fused steps, split-K reduced through distributed shared memory, RMSNorm
    folded into the next GEMM's operand) -- compute the same layer with other summation orders: they must
    reproduce HF's greedy ids on config 1 like the default path, and a batch of 64 must be deterministic."""
    monkeypatch.setenv("B2_CHAIN", chain)
    model, sd = full
    arch = QWEN3_0_6B
    fx = json.load(open(os.path.join(GOLD, "qwen3_0p6b_c1.json")))
    prompt, gold = fx["prompt_ids"], np.array(fx["greedy_ids"])
    e = make_engine(P, arch, sd, max_model_len=512, num_blocks=64 * 12 + 8, max_seqs=64, max_batch_tokens=2048, use_cuda_graphs=True)
    sid = e.seq_create(300)
    # teacher-forced with HF's tokens, so that every one of the 128 steps is compared (a free-running stream is only
    # comparable up to its first tie flip): the engine's token may differ from HF's only where HF's own top-2 logit gap
    # is within 2 bf16 ulp of the top logit
    got = [int(e.prefill([sid], [prompt])[0])]
    for t in range(1, 128):
        got.append(int(e.decode_step([sid], in_tokens=[int(gold[t - 1])])[0]))
    got = np.array(got)
    top4 = np.array(fx["tf_top4_logits"])
    mism = np.nonzero(got != gold)[0]
    print("B2_CHAIN=%s, C1 teacher-forced: %d/128 tokens identical to HF (differing steps: %s)" % (chain, 128 - len(mism), mism.tolist()))
    for t in mism:
        gap = float(top4[127 + t][0] - top4[127 + t][1])
        assert gap <= 2 * bf16_ulp_of(float(top4[127 + t][0])), "step %d differs from HF where its top-2 gap is %.4f (not a tie)" % (t, gap)
    assert len(mism) <= 6
    e.seq_free(sid)
    # batch 64 (the shape chain_cluster.cu is built for): same bits run after run
    p64 = make_prompts(64, 100, arch.vocab, seed=3)
    runs = []
    for rep in range(2):
        sids = [e.seq_create(150) for _ in range(64)]
        f = np.concatenate([e.prefill(sids[i:i + 16], [q.tolist() for q in p64[i:i + 16]]) for i in range(0, 64, 16)])
        t64, _ = e.decode_run(sids, 16)
        runs.append((f.copy(), t64.copy()))
        for s_ in sids:
            e.seq_free(s_)
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
    e.close()


def test_full_batch64_properties(P):
    """The served shapes (batch 64, paged KV) through size-independent properties.
    64 copies of one prompt: the prefill (one CTA per sequence tile) must give 64 identical first tokens;
    decode must be deterministic run to run.  Decode attention balances pages over its warps, so where
    a sequence's pages are cut depends on its position in the batch: copies may legitimately separate at
    a near-tie of the random-init logits, but never all of them and never at once."""
    arch = QWEN3_0_6B
    sd = random_weights(arch, seed=0)
    e = make_engine(P, arch, sd, max_model_len=1024, num_blocks=64 * 24 + 8, max_seqs=64, max_batch_tokens=8192,
                    use_cuda_graphs=True)
    prompt = make_prompts(1, 120, arch.vocab, seed=1)[0].tolist()
    runs = []
    for rep in range(2):
        sids = [e.seq_create(200) for _ in range(64)]
        first = e.prefill(sids, [prompt] * 64)
        toks, ms = e.decode_run(sids, 24)
        assert (first == first[0]).all()
        runs.append(toks.copy())
        for s in sids:
            e.seq_free(s)
    assert np.array_equal(runs[0], runs[1]), "decode is not deterministic run to run"
    toks = runs[0]
    same_as_first = (toks == toks[:, :1]).all(axis=0)          # per sequence: whole stream equals sequence 0's
    assert (toks[0] == toks[0, 0]).all(), "first decode step differs across identical sequences"
    assert same_as_first.mean() >= 0.5, "only %d/64 identical sequences stayed together" % int(same_as_first.sum())
    sid = e.seq_create(200)
    f1 = e.prefill([sid], [prompt])
    t1, _ = e.decode_run([sid], 24)
    agree = int((t1[:, 0] == toks[:, 0]).sum())
    assert int(f1[0]) == int(first[0])
    assert agree >= 12, "batch-64 stream vs batch-1 stream agree on %d/24 tokens" % agree
    assert e.info()["free_blocks"] > 0
    e.close()


def test_tiny_long_ragged_contexts(P, tiny):
    """Long and very ragged contexts (1 .. 1900 tokens, 40 sequences) on the tiny model: the page-balanced decode
    attention cuts such a batch into runs that start and end anywhere, empty and one-page sequences sit next to
    120-page ones, and decode crosses page boundaries while it runs.  Greedy ids against the restatement,
    tie-aware; logits of the last step within 1e-2."""
    model, sd = tiny
    arch = QWEN3_TINY
    g = torch.Generator().manual_seed(21)
    lens = [1, 2, 15, 16, 17, 31, 32, 33, 100, 255, 256, 257, 511, 777, 1023, 1024, 1025, 1500, 1900, 1899] + \
           [int(x) for x in torch.randint(1, 1900, (20,), generator=g)]
    steps = 20
    prompts = [torch.randint(0, arch.vocab, (n,), generator=g).tolist() for n in lens]
    e = make_engine(P, arch, sd, max_model_len=2048, num_blocks=sum((n + steps + 16) // 16 + 1 for n in lens) + 8, max_seqs=64,
                    max_batch_tokens=4096, use_cuda_graphs=True)
    e.set_debug(logits=True)
    sids = [e.seq_create(n + steps + 4) for n in lens]
    firsts = []
    i = 0
    while i < len(lens):  # prefill in chunks that respect max_batch_tokens
        j, tot = i, 0
        while j < len(lens) and tot + lens[j] <= 4096:
            tot += lens[j]
            j += 1
        firsts.append(e.prefill(sids[i:j], prompts[i:j]))
        i = j
    first = np.concatenate(firsts)
    toks = [first] + [e.decode_step(sids) for _ in range(steps - 1)]
    got = np.stack(toks, axis=1)
    last_logits = torch.from_numpy(e.get_logits(len(lens)).copy())
    r = Restated(arch, sd, attention=attention_explicit)
    checked_logits = 0
    for k, pr in enumerate(prompts):
        ref_ids, ref_logits = r.greedy(torch.tensor([pr]), steps)
        gaps = top2_gap(ref_logits)
        same = True
        for t in range(steps):
            if got[k, t] != int(ref_ids[0, t]):
                assert gaps[0, t] <= 0.0625, "sequence %d (prompt %d tokens) step %d: %d != %d with oracle gap %.4f" % (
                    k, lens[k], t, got[k, t], int(ref_ids[0, t]), gaps[0, t])
                same = False
                break
        if same:
            assert rel_err(last_logits[k], ref_logits[0, steps - 1].float()) < REL_TOL, "logits of sequence %d" % k
            checked_logits += 1
    assert checked_logits >= len(lens) // 2
    for s in sids:
        e.seq_free(s)
    assert e.info()["free_blocks"] == e.info()["num_blocks"] - 1  # everything returned (page 0 is the null page)
    e.close()


def test_sharded_checkpoint_and_dtypes(P, tiny, tmp_path):
    """A checkpoint split over two safetensors files, one stored in fp16 and one in fp32, loaded through
    b2_engine_load_safetensors: the engine must end up with exactly the weights (rounded to bf16, to nearest even)
    that a state dict of the same values gives -- identical greedy tokens."""
    weights = __import__("importlib").import_module("aws-k8s-ansible-provisioner_b200.weights")
    model, sd = tiny
    arch = QWEN3_TINY
    g = torch.Generator().manual_seed(5)
    wide = {k: (v.float() + 1e-3 * torch.randn(v.shape, generator=g)) for k, v in sd.items()}  # not bf16-representable
    names = list(wide)
    a = {k: wide[k].to(torch.float16) for k in names[: len(names) // 2]}
    b = {k: wide[k] for k in names[len(names) // 2:]}
    weights.write_safetensors(a, str(tmp_path / "model-00001-of-00002.safetensors"))
    weights.write_safetensors(b, str(tmp_path / "model-00002-of-00002.safetensors"))
    expect = {k: a[k].float().to(torch.bfloat16) for k in a}
    expect.update({k: b[k].to(torch.bfloat16) for k in b})
    prompts = make_prompts(2, 30, arch.vocab, seed=2)
    outs = []
    for mode in ("files", "dict"):
        cfg = engine_config_from_arch(P, arch, max_model_len=128, num_blocks=32, max_seqs=4, max_batch_tokens=128, use_cuda_graphs=False)
        e = P.Engine(cfg, rope_inv_freq=rope_inv_freq(arch).numpy())
        if mode == "files":
            e.load_safetensors([str(tmp_path / "model-00001-of-00002.safetensors"), str(tmp_path / "model-00002-of-00002.safetensors")])
        else:
            e.load_state_dict(expect)
        sids = [e.seq_create(64) for _ in range(2)]
        first = e.prefill(sids, [p.tolist() for p in prompts])
        toks, _ = e.decode_run(sids, 12)
        outs.append(np.concatenate([first[None, :], toks], axis=0))
        e.close()
    assert np.array_equal(outs[0], outs[1])


# The bench workload's shape (batch 64, 512-token prompts, graph decode) against HF over 128 tokens: test_parity_full_gpu.py


def test_prefix_cache_reuses_prompt_pages(P, tiny):
    """vLLM's --enable-prefix-caching in the engine (the router's prefix affinity needs it): a second
    prompt that shares a 448-token prefix with an earlier one prefills only its tail, gives the same greedy ids as the
    cold run, and pages are neither leaked nor rewritten while shared."""
    model, sd = tiny
    arch = QWEN3_TINY
    e = make_engine(P, arch, sd, max_model_len=640, num_blocks=200, max_seqs=8, max_batch_tokens=1024, use_cuda_graphs=True)
    g = torch.Generator().manual_seed(31)
    prefix = torch.randint(0, arch.vocab, (448,), generator=g).tolist()
    tails = [torch.randint(0, arch.vocab, (40,), generator=g).tolist() for _ in range(3)]

    def run(prompt, steps=12):
        sid = e.seq_create(len(prompt) + steps + 4)
        l0 = e.launch_count()
        first = int(e.prefill([sid], [prompt])[0])
        toks, _ = e.decode_run([sid], steps)
        return sid, [first] + toks[:, 0].tolist(), l0

    free0 = e.info()["free_blocks"]
    cold = []
    for t in tails:  # cache off: the reference streams
        sid, out, _ = run(prefix + t)
        cold.append(out)
        e.seq_free(sid)
    assert e.info()["free_blocks"] == free0
    e.set_tuning(prefix_cache=True)
    sid_a, out_a, _ = run(prefix + tails[0])
    st = e.prefix_cache_stats()
    assert out_a == cold[0] and st["hit_tokens"] == 0 and st["queried_tokens"] == 488 and st["cached_pages"] == 488 // 16
    # while A is alive: B shares A's 28 prefix pages, C too; both only compute their 40-token tails (+ nothing of the prefix)
    sid_b, out_b, _ = run(prefix + tails[1])
    st = e.prefix_cache_stats()
    assert st["hit_tokens"] == 448, st
    assert out_b == cold[1], "a prompt served from cached pages must give the cold run's tokens"
    e.seq_free(sid_a)  # B still holds the pages
    sid_c, out_c, _ = run(prefix + tails[2])
    assert out_c == cold[2] and e.prefix_cache_stats()["hit_tokens"] == 896
    # the very same prompt again: everything but the last page's worth is a hit, the result is the same
    sid_d, out_d, _ = run(prefix + tails[1])
    assert out_d == cold[1] and e.prefix_cache_stats()["hit_tokens"] == 896 + 480
    # truncating into the shared prefix un-shares those pages for this sequence only: B keeps decoding what it decoded
    e.seq_truncate(sid_d, 100)
    e.prefill([sid_d], [[7] * 20])  # rewrites positions 100..119 of D's private copies
    sid_e, out_e, _ = run(prefix + tails[1])
    assert out_e == cold[1], "pages shared with a truncated sequence were modified"
    for s in (sid_b, sid_c, sid_d, sid_e):
        e.seq_free(s)
    assert e.info()["free_blocks"] == free0, "pages leaked (cached pages nobody holds count as free)"
    # a pool too small to keep everything: old cached pages are evicted, nothing breaks
    many = [e.seq_create(600) for _ in range(5)]
    for s in many:
        e.prefill([s], [torch.randint(0, arch.vocab, (590,), generator=g).tolist()])
    for s in many:
        e.seq_free(s)
    sid_f, out_f, _ = run(prefix + tails[0])
    assert out_f == cold[0]
    e.seq_free(sid_f)
    e.set_tuning(prefix_cache=False)
    assert e.prefix_cache_stats()["cached_pages"] == 0 and e.info()["free_blocks"] == free0
    e.close()


@pytest.mark.parametrize("nseq", [1, 3, 40])
def test_logits_of_few_and_many_rows(P, nseq):
    """get_logits brings rows through staging in pieces, many rows by several threads: every row equals the same row read in another number of rows, and its
    largest entry is the greedy token."""
    cfg = P.EngineConfig(num_layers=1, hidden=256, num_q_heads=2, num_kv_heads=1, head_dim=128, intermediate=256, vocab=131 * 1001, max_model_len=32, num_blocks=2 * nseq + 4,
                         max_seqs=nseq, max_batch_tokens=64)
    eng = P.Engine(cfg)
    g = torch.Generator().manual_seed(3)
    eng.load_state_dict({k: (torch.randn(s, generator=g) * 0.05).to(torch.bfloat16) for k, s in importlib.import_module(P.__name__ + ".weights").tensor_shapes(cfg).items()})
    eng.set_debug(logits=True)
    sids = [eng.seq_create(16) for _ in range(nseq)]
    out = eng.prefill(sids, [[7 * i % 1000] for i in range(nseq)])
    full = eng.get_logits(nseq)
    assert (full.max(1) == full[np.arange(nseq), out]).all()
    one = eng.get_logits(1)
    assert (one[0] == full[0]).all()
    assert (eng.get_logits(nseq) == full).all()
    eng.close()


def test_page_locked_memory(P, tiny):
    """b2_host_alloc: too much is refused and leaves nothing behind; logits that are read into such a block are those of get_logits."""
    _, sd = tiny
    e = make_engine(P, QWEN3_TINY, sd, max_model_len=64, num_blocks=16, max_seqs=2, max_batch_tokens=64)
    e.set_debug(logits=True)
    p = C.c_void_p(1)
    assert e.lib.b2_host_alloc(1 << 55, C.byref(p)) == -12 and p.value is None and e.lib.b2_host_alloc(0, C.byref(p)) != 0
    e.prefill([e.seq_create(40)], [[3 + i for i in range(20)]])
    n = QWEN3_TINY.vocab
    assert e.lib.b2_host_alloc(4 * n, C.byref(p)) == 0
    assert e.lib.b2_get_logits(e.h, 1, C.cast(p, C.POINTER(C.c_float))) == 0
    assert (np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_float)), (n,)) == e.get_logits(1)[0]).all()
    e.lib.b2_host_free(p)
    e.lib.b2_host_free(None)
    e.close()


def test_a_copy_that_was_started_from_a_result_is_not_overtaken(P):
    """Logits on their way to a device while the array is dropped and the next ones are read: the copy has the values that it was started with."""
    cfg = P.EngineConfig(num_layers=1, hidden=256, num_q_heads=2, num_kv_heads=1, head_dim=128, intermediate=256, vocab=131 * 1001, max_model_len=32, num_blocks=16, max_seqs=2,
                         max_batch_tokens=64)
    eng = P.Engine(cfg)
    g = torch.Generator().manual_seed(3)
    eng.load_state_dict({k: (torch.randn(s, generator=g) * 0.05).to(torch.bfloat16) for k, s in importlib.import_module(P.__name__ + ".weights").tensor_shapes(cfg).items()})
    eng.set_debug(logits=True)
    sid = eng.seq_create(16)
    eng.prefill([sid], [[7, 9, 11]])
    side = torch.cuda.Stream()
    on_device = [torch.empty(1, cfg.vocab, device="cuda") for _ in range(5)]
    for cycles in (0, 400_000_000):   # (the first pass loads and captures what the second would wait for)
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            torch.cuda._sleep(cycles)   # what the copies wait behind
        want = []
        for d in on_device:
            logits = eng.get_logits(1)
            want.append(logits.copy())
            with torch.cuda.stream(side):
                d.copy_(torch.from_numpy(logits), non_blocking=True)
            del logits
            eng.decode_step([sid])
        torch.cuda.synchronize()
        for i, (d, w) in enumerate(zip(on_device, want)):
            assert (d.cpu().numpy() == w).all() and not (w == want[i - 1]).all(), i
    eng.close()


@pytest.mark.parametrize("n", [199, 700])
def test_prefill_reports_a_wait_that_ran_out(P, tiny, monkeypatch, n):
    """A prompt kernel whose waits run out (here: are given no time) makes the call an error; the caller's other engines are not touched by it.  Long prompts have their
    projections on pairs of CTAs."""
    _, sd = tiny
    prompt = [[1 + i % 300 for i in range(n)]]
    monkeypatch.setenv("B2_PREFILL_WAIT_MS", "0")
    bad = make_engine(P, QWEN3_TINY, sd, max_model_len=1024, num_blocks=140, max_seqs=2, max_batch_tokens=1024)
    monkeypatch.delenv("B2_PREFILL_WAIT_MS")
    good = make_engine(P, QWEN3_TINY, sd, max_model_len=1024, num_blocks=140, max_seqs=2, max_batch_tokens=1024)
    want = good.prefill([good.seq_create(n + 1)], prompt)
    sid = bad.seq_create(n + 1)
    with pytest.raises(P.B2Error, match="did not end within 0 ms"):
        bad.prefill([sid], prompt)
    bad.seq_free(sid)
    assert (good.prefill([good.seq_create(n + 1)], prompt) == want).all()
    bad.close()
    good.close()
