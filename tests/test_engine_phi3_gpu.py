"""Phi-3 variant of the hot path through the C ABI on the GPU, against HF
Phi3ForCausalLM's own outputs (tests/golden/phi3_tiny.npz) and against the pinned restatement
(oracle/phi3_oracle.py).  Same bars as the Qwen3 engine tests: hidden states and logits within 1e-2
relative, greedy ids identical except after a step whose oracle top-2 gap is within
bf16 noise.  The engine runs these models through its 128-wide, two-query-heads-per-kv-head kernels
with zero padding placed in the weights, so these tests are also the check that
the padding changes nothing."""
import os

import numpy as np
import pytest
import torch

from _util import ROOT, engine_config_from_arch, pkg, rel_err, rel_fro
from oracle.phi3_oracle import (PHI3_MINI_2L, PHI3_TINY, PHI3_TINY_PARTIAL, PHI3_TINY_WINDOW, RestatedPhi3, hf_phi3_model,
                                linear_fp32_order, phi3_inv_freq)
from oracle.qwen3_oracle import KVState, attention_explicit, hf_state_dict, make_prompts, perturb_norm_weights, top2_gap

pytestmark = pytest.mark.gpu
GOLD = os.path.join(ROOT, "tests", "golden")
REL_TOL = 1e-2


@pytest.fixture(scope="module")
def P():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return pkg()


def bits_to_bf16(bits: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(bits.astype(np.int16)).view(torch.bfloat16)


def make_engine(P, arch, sd, **kw):
    cfg = engine_config_from_arch(P, arch, **kw)
    e = P.Engine(cfg, rope_inv_freq=phi3_inv_freq(arch).numpy())
    e.load_state_dict(sd)
    return e


@pytest.mark.parametrize("tag", ["full", "partial", "window"])
@pytest.mark.parametrize("graphs", [False, True])
def test_phi3_tiny_matches_hf_golden(P, tag, graphs):
    arch = {"full": PHI3_TINY, "partial": PHI3_TINY_PARTIAL, "window": PHI3_TINY_WINDOW}[tag]
    model = hf_phi3_model(arch, seed=0)
    sd = hf_state_dict(model)
    perturb_norm_weights(sd)
    g = np.load(os.path.join(GOLD, "phi3_tiny.npz"))
    prompts, gold = g[tag + "_prompt_ids"], g[tag + "_greedy_ids"]   # [3][40], [3][24]
    e = make_engine(P, arch, sd, max_model_len=256, num_blocks=64, max_seqs=8, max_batch_tokens=512, use_cuda_graphs=graphs)
    if not graphs:
        e.set_debug(hidden=True, logits=True)
    sids = [e.seq_create(128) for _ in range(3)]
    first = e.prefill(sids, [p.tolist() for p in prompts])
    if not graphs:
        hid = g[tag + "_hidden_bf16"]  # [L+1][3][64][H], teacher-forced over prompt + generated
        T = 3 * 40
        for layer in range(-1, arch.num_layers - 1):  # the last entry is post-norm in HF; covered by the logits
            got = bits_to_bf16(e.get_hidden(layer, T)).view(3, 40, arch.hidden)
            ref = bits_to_bf16(hid[layer + 1][:, :40])
            assert rel_err(got, ref) < REL_TOL, "hidden after layer %d" % layer
        logits = torch.from_numpy(e.get_logits(3))
        ref_logits = bits_to_bf16(g[tag + "_logits_bf16"])[:, 39].float()
        assert rel_err(logits, ref_logits) < REL_TOL
    toks = [first] + [e.decode_step(sids) for _ in range(gold.shape[1] - 1)]
    got = np.stack(toks, axis=1)
    r = RestatedPhi3(arch, sd)
    _, step_logits = r.greedy(torch.from_numpy(prompts).long(), gold.shape[1])
    gaps = top2_gap(step_logits)
    for b in range(3):
        for t in range(gold.shape[1]):
            if got[b, t] != gold[b, t]:
                assert gaps[b, t] <= 0.0625, "seq %d step %d: token %d != %d with oracle gap %.4f" % (
                    b, t, got[b, t], gold[b, t], gaps[b, t])
                break
    assert (got[:, :8] == gold[:, :8]).mean() > 0.9
    e.close()


def test_phi3_mini_widths_two_layers(P):
    """Phi-3-mini's real widths (hidden 3072, 32 heads of 96, SwiGLU 8192, vocab 32064 untied) on two
    layers: ragged prefill + batched decode against the restatement, logits within 1e-2."""
    arch = PHI3_MINI_2L
    g = torch.Generator().manual_seed(11)

    def n(*shape):
        return (0.02 * torch.randn(*shape, generator=g)).to(torch.bfloat16)

    H, I, hd = arch.hidden, arch.intermediate, arch.head_dim
    sd = {"model.embed_tokens.weight": n(arch.vocab, H), "lm_head.weight": n(arch.vocab, H),
          "model.norm.weight": (1.0 + 0.25 * torch.randn(H, generator=g)).to(torch.bfloat16)}
    for l in range(arch.num_layers):
        p = "model.layers.%d." % l
        sd[p + "input_layernorm.weight"] = (1.0 + 0.25 * torch.randn(H, generator=g)).to(torch.bfloat16)
        sd[p + "post_attention_layernorm.weight"] = (1.0 + 0.25 * torch.randn(H, generator=g)).to(torch.bfloat16)
        sd[p + "self_attn.qkv_proj.weight"] = n(3 * arch.num_q_heads * hd, H)
        sd[p + "self_attn.o_proj.weight"] = n(H, arch.num_q_heads * hd)
        sd[p + "mlp.gate_up_proj.weight"] = n(2 * I, H)
        sd[p + "mlp.down_proj.weight"] = n(H, I)
    lens = [5, 33, 64]
    prompts = [torch.randint(0, arch.vocab, (k,), generator=g).tolist() for k in lens]
    e = make_engine(P, arch, sd, max_model_len=256, num_blocks=64, max_seqs=8, max_batch_tokens=256, use_cuda_graphs=True)
    e.set_debug(logits=True)
    sids = [e.seq_create(128) for _ in lens]
    first = e.prefill(sids, prompts)
    pre_logits = torch.from_numpy(e.get_logits(len(lens)).copy())
    steps = [first] + [e.decode_step(sids) for _ in range(5)]
    dec_logits = torch.from_numpy(e.get_logits(len(lens)).copy())
    got = np.stack(steps, axis=1)
    r = RestatedPhi3(arch, sd, attention=attention_explicit)
    # The same oracle with the fp32 additions of every Linear in another order (and the other attention
    # formulation): the distance between two equally valid evaluations is the bf16 noise floor of this
    # model -- measured ~0.8 % on the logits at these widths (K = 3072 / 8192, random weights), so the
    # 1e-2 bar alone would be a coin toss for ANY implementation.  Bars: Frobenius max(1e-2, 1.5 x floor);
    # max-norm max(1e-2, 2 x floor) -- the max-norm moves in whole bf16 ulps of the largest logit (0.7 % each
    # here), so the floor is 2 ulps and anything below 4 is the same measurement.
    r2 = RestatedPhi3(arch, sd, linear=linear_fp32_order)
    for i, pr in enumerate(prompts):
        ids = torch.tensor([pr])
        ref_ids, ref_logits = r.greedy(ids, 6)
        _, alt_logits = r2.greedy(ids, 1)
        ref0 = ref_logits[0, 0].float()
        floor, floor_fro = rel_err(alt_logits[0, 0].float(), ref0), rel_fro(alt_logits[0, 0].float(), ref0)
        err, fro = rel_err(pre_logits[i], ref0), rel_fro(pre_logits[i], ref0)
        print("sequence %d: prefill logits engine vs oracle max-rel %.4g fro %.4g | oracle vs its reordered self %.4g / %.4g" % (
            i, err, fro, floor, floor_fro))
        assert err <= max(REL_TOL, 2.0 * floor), "prefill logits, sequence %d" % i
        assert fro < max(REL_TOL, 1.5 * floor_fro), "prefill logits (Frobenius), sequence %d" % i
        gaps = top2_gap(ref_logits)
        same = True
        for t in range(6):
            if got[i, t] != int(ref_ids[0, t]):
                assert gaps[0, t] <= 0.0625, "seq %d step %d diverges with oracle gap %.4f" % (i, t, gaps[0, t])
                same = False
                break
        if same:
            assert rel_err(dec_logits[i], ref_logits[0, 5].float()) <= max(REL_TOL, 2.0 * floor), "decode logits, sequence %d" % i
    assert int(e.info()["free_blocks"]) > 0
    e.close()


def test_phi3_rejects_unsupported_shapes(P):
    from oracle.phi3_oracle import Phi3Arch
    bad = Phi3Arch(num_layers=1, hidden=512, num_q_heads=8, num_kv_heads=2, head_dim=64, intermediate=512, vocab=256,
                   tie_embeddings=False)  # 4 query heads per kv head
    cfg = engine_config_from_arch(P, bad, max_model_len=64, num_blocks=8, max_seqs=2, max_batch_tokens=64)
    with pytest.raises(Exception) as ei:
        P.Engine(cfg)
    assert "query heads per kv head" in str(ei.value)


@pytest.mark.parametrize("window", [24, 100])
def test_phi3_sliding_window_long_ragged(P, window):
    """Sliding-window attention at contexts many pages longer than the window: prompts of 5 .. 700 tokens, the
    window starting inside a page, at a page boundary and before the first token; prefill (window mask + skipped key
    tiles) and 12 decode steps (skipped pages + masked first page) against the restatement, tie-aware."""
    from dataclasses import replace
    arch = replace(PHI3_TINY_WINDOW, sliding_window=window, name="phi3-tiny-window-%d" % window)
    sd = hf_state_dict(hf_phi3_model(arch, seed=0))
    perturb_norm_weights(sd)
    g = torch.Generator().manual_seed(31)
    lens = [5, window - 1, window, window + 1, 40, 100, 333, 700, 16 * 9, 16 * 9 + window]
    steps = 12
    prompts = [torch.randint(0, arch.vocab, (n,), generator=g).tolist() for n in lens]
    e = make_engine(P, arch, sd, max_model_len=1024, num_blocks=sum((n + steps) // 16 + 2 for n in lens) + 8, max_seqs=16,
                    max_batch_tokens=2048, use_cuda_graphs=True)
    e.set_debug(logits=True)
    sids = [e.seq_create(n + steps + 2) for n in lens]
    first = e.prefill(sids, prompts)
    pre_logits = torch.from_numpy(e.get_logits(len(lens)).copy())
    toks = [first] + [e.decode_step(sids) for _ in range(steps - 1)]
    got = np.stack(toks, axis=1)
    last_logits = torch.from_numpy(e.get_logits(len(lens)).copy())
    r = RestatedPhi3(arch, sd)
    r2 = RestatedPhi3(arch, sd, linear=linear_fp32_order)  # the oracle's own bf16 noise floor (see the full-width test)
    full = RestatedPhi3(replace(arch, sliding_window=0), sd)  # no window: must differ once the context exceeds it
    for k, pr in enumerate(prompts):
        ref_ids, ref_logits = r.greedy(torch.tensor([pr]), steps)
        alt_ids, alt = r2.greedy(torch.tensor([pr]), steps)
        floor = rel_err(alt[0, 0].float(), ref_logits[0, 0].float())
        # the floor of the LAST step only means something if the reordered oracle decoded the same tokens
        floor_last = rel_err(alt[0, steps - 1].float(), ref_logits[0, steps - 1].float()) if torch.equal(alt_ids, ref_ids) else 1.0
        assert rel_err(pre_logits[k], ref_logits[0, 0].float()) <= max(REL_TOL, 2.0 * floor), "prefill logits, prompt of %d tokens" % lens[k]
        if lens[k] > 2 * window:
            _, nowin = full.greedy(torch.tensor([pr]), 1)
            assert rel_err(pre_logits[k], nowin[0, 0].float()) > REL_TOL, "the window had no effect at %d tokens" % lens[k]
        gaps = top2_gap(ref_logits)
        same = True
        for t in range(steps):
            if got[k, t] != int(ref_ids[0, t]):
                assert gaps[0, t] <= 0.0625, "prompt %d step %d: %d != %d, oracle gap %.4f" % (lens[k], t, got[k, t], int(ref_ids[0, t]), gaps[0, t])
                same = False
                break
        if same:
            assert rel_err(last_logits[k], ref_logits[0, steps - 1].float()) <= max(REL_TOL, 2.0 * floor_last), "decode logits, prompt of %d tokens" % lens[k]
    e.close()
