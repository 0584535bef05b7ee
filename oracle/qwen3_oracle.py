"""ORACLE (test infrastructure only -- never imported by the product path).

CPU restatement of the arithmetic the reference deployment implies for its one hot
path: the Qwen3-0.6B forward pass inside the model-server pod that
`llm-d-deploy.yaml:118,184` launches (model id `Qwen/Qwen3-0.6B`).  The reference
repository holds no arithmetic of its own; the arithmetic lives in a third-party
dependency, HF `transformers==5.5.0` over `torch==2.11.0` CPU kernels.  Both are
present in this image (here and on the GPU box), so this oracle is pinned two ways:

  * `hf_model()` builds the *real* HF `Qwen3ForCausalLM` from a hand-written config
    (no network) -- that object IS the graded oracle.
  * `Restated` is a plain-torch restatement of the same forward, one function per
    HF function, each citing the HF file:line it follows.  `tests/test_oracle.py`
    checks it bit-for-bit against `hf_model()` (same CPU kernels => identical bits)
    and against the committed golden fixtures in `tests/golden/`.

The reference's own tests pin nothing numeric at this boundary (only the model-id
substring, `llm-d-test.yaml:54-59`); parity is therefore pinned on outputs of HF
itself, generated by `oracle/make_golden.py` (committed with the fixtures).

Citations `HF:` are relative to site-packages/transformers/.
"""
from __future__ import annotations

import math
from dataclasses import dataclass, field

import torch
import torch.nn.functional as F


# --------------------------------------------------------------------------------------
# Model constants
# --------------------------------------------------------------------------------------
@dataclass
class ArchConfig:
    name: str = "Qwen/Qwen3-0.6B"
    num_layers: int = 28
    hidden: int = 1024
    num_q_heads: int = 16
    num_kv_heads: int = 8
    head_dim: int = 128
    intermediate: int = 3072
    vocab: int = 151936
    rms_eps: float = 1e-6
    rope_theta: float = 1e6
    max_position: int = 40960
    tie_embeddings: bool = True

    @property
    def q_size(self) -> int:
        return self.num_q_heads * self.head_dim

    @property
    def kv_size(self) -> int:
        return self.num_kv_heads * self.head_dim

    def kv_bytes_per_token(self) -> int:
        return 2 * self.num_layers * self.kv_size * 2

    def weight_bytes(self) -> int:
        per_layer = (
            (self.q_size + 2 * self.kv_size) * self.hidden
            + self.hidden * self.q_size
            + 3 * self.intermediate * self.hidden
            + 2 * self.hidden
            + 2 * self.head_dim
        )
        total = self.num_layers * per_layer + self.vocab * self.hidden + self.hidden
        if not self.tie_embeddings:
            total += self.vocab * self.hidden
        return 2 * total


QWEN3_0_6B = ArchConfig()

# A scaled-down architecture with the same structure (GQA 2:1, head_dim 128, QK-norm, tied
# head) for CPU-cheap tests.  Not a benchmark configuration.
QWEN3_TINY = ArchConfig(
    name="qwen3-tiny-test", num_layers=2, hidden=256, num_q_heads=4, num_kv_heads=2,
    head_dim=128, intermediate=512, vocab=1024, max_position=4096,
)


def hf_config(arch: ArchConfig):
    from transformers import Qwen3Config

    return Qwen3Config(
        vocab_size=arch.vocab,
        hidden_size=arch.hidden,
        intermediate_size=arch.intermediate,
        num_hidden_layers=arch.num_layers,
        num_attention_heads=arch.num_q_heads,
        num_key_value_heads=arch.num_kv_heads,
        head_dim=arch.head_dim,
        hidden_act="silu",
        max_position_embeddings=arch.max_position,
        rms_norm_eps=arch.rms_eps,
        rope_parameters={"rope_type": "default", "rope_theta": arch.rope_theta},
        tie_word_embeddings=arch.tie_embeddings,
        attention_bias=False,
        attention_dropout=0.0,
        use_sliding_window=False,
    )


def hf_model(arch: ArchConfig = QWEN3_0_6B, seed: int = 0, attn: str = "sdpa"):
    """The graded oracle: HF Qwen3ForCausalLM, default init under `torch.manual_seed(seed)`,
    cast to bf16, eval mode, on CPU."""
    from transformers import Qwen3ForCausalLM

    cfg = hf_config(arch)
    cfg._attn_implementation = attn
    torch.manual_seed(seed)
    model = Qwen3ForCausalLM(cfg)
    model = model.to(torch.bfloat16).eval()
    # `.to(bfloat16)` also rounds the non-persistent rotary `inv_freq` buffer to bf16, which a
    # deployed checkpoint never sees (`from_pretrained(dtype=bf16)` computes it in fp32,
    # HF:models/qwen3/modeling_qwen3.py:129-131).  Restore the fp32 table so the oracle is the
    # served model's arithmetic, not an artefact of how this script cast the weights.
    inv = rope_inv_freq(arch)
    model.model.rotary_emb.inv_freq = inv.clone()
    model.model.rotary_emb.original_inv_freq = inv.clone()
    return model


def random_weights(arch: ArchConfig, seed: int = 0, std: float = 0.02) -> dict[str, torch.Tensor]:
    """HF-named bf16 state dict drawn directly (no HF module construction) -- used by the
    bench and by GPU tests that do not need HF's exact init stream.  Same distribution as
    HF's default init (N(0, 0.02) for Linear/Embedding, ones for norms)."""
    g = torch.Generator().manual_seed(seed)

    def n(*shape):
        return (torch.randn(*shape, generator=g, dtype=torch.float32) * std).to(torch.bfloat16)

    sd: dict[str, torch.Tensor] = {}
    sd["model.embed_tokens.weight"] = n(arch.vocab, arch.hidden)
    for i in range(arch.num_layers):
        p = f"model.layers.{i}."
        sd[p + "input_layernorm.weight"] = torch.ones(arch.hidden, dtype=torch.bfloat16)
        sd[p + "self_attn.q_proj.weight"] = n(arch.q_size, arch.hidden)
        sd[p + "self_attn.k_proj.weight"] = n(arch.kv_size, arch.hidden)
        sd[p + "self_attn.v_proj.weight"] = n(arch.kv_size, arch.hidden)
        sd[p + "self_attn.o_proj.weight"] = n(arch.hidden, arch.q_size)
        sd[p + "self_attn.q_norm.weight"] = torch.ones(arch.head_dim, dtype=torch.bfloat16)
        sd[p + "self_attn.k_norm.weight"] = torch.ones(arch.head_dim, dtype=torch.bfloat16)
        sd[p + "post_attention_layernorm.weight"] = torch.ones(arch.hidden, dtype=torch.bfloat16)
        sd[p + "mlp.gate_proj.weight"] = n(arch.intermediate, arch.hidden)
        sd[p + "mlp.up_proj.weight"] = n(arch.intermediate, arch.hidden)
        sd[p + "mlp.down_proj.weight"] = n(arch.hidden, arch.intermediate)
    sd["model.norm.weight"] = torch.ones(arch.hidden, dtype=torch.bfloat16)
    if not arch.tie_embeddings:
        sd["lm_head.weight"] = n(arch.vocab, arch.hidden)
    return sd


def perturb_norm_weights(sd: dict[str, torch.Tensor], seed: int = 7) -> None:
    """HF initialises every norm weight to exactly 1, which would hide a kernel that
    forgot the weight multiply.  Tests call this to make the norm gains non-trivial."""
    g = torch.Generator().manual_seed(seed)
    for k, v in sd.items():
        if "norm" in k:
            sd[k] = (1.0 + 0.25 * torch.randn(v.shape, generator=g)).to(torch.bfloat16)


def make_prompts(batch: int, prompt_len: int, vocab: int, seed: int = 1) -> torch.Tensor:
    """Uniform random token ids, generator seed 1."""
    g = torch.Generator().manual_seed(seed)
    return torch.randint(0, vocab, (batch, prompt_len), generator=g, dtype=torch.int64)


# --------------------------------------------------------------------------------------
# Plain-torch restatement, one function per HF function
# --------------------------------------------------------------------------------------
def rms_norm(x: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    """HF:models/qwen3/modeling_qwen3.py:59-64  Qwen3RMSNorm.forward.
    fp32 variance, scale in fp32, ROUND TO bf16, then multiply by the bf16 weight (which
    rounds once more)."""
    dt = x.dtype
    xf = x.to(torch.float32)
    var = xf.pow(2).mean(-1, keepdim=True)
    xf = xf * torch.rsqrt(var + eps)
    return weight * xf.to(dt)


def rope_inv_freq(arch: ArchConfig) -> torch.Tensor:
    """HF:modeling_rope_utils / models/qwen3/modeling_qwen3.py:105-130 (default rope):
    inv_freq = 1 / theta^(2i/d), fp32."""
    d = arch.head_dim
    return 1.0 / (arch.rope_theta ** (torch.arange(0, d, 2, dtype=torch.int64).to(dtype=torch.float) / d))


def rope_cos_sin(arch: ArchConfig, positions: torch.Tensor, dtype=torch.bfloat16):
    """HF:models/qwen3/modeling_qwen3.py:132-148  Qwen3RotaryEmbedding.forward.
    freqs in fp32, emb = cat(freqs, freqs), cos/sin in fp32 then cast to the model dtype."""
    inv = rope_inv_freq(arch)
    pos = positions.to(torch.float32)
    freqs = pos[..., None] * inv  # [..., d/2]  (HF does inv[None,:,None] @ pos[:,None,:], same products)
    emb = torch.cat((freqs, freqs), dim=-1)
    return emb.cos().to(dtype), emb.sin().to(dtype)


def rotate_half(x: torch.Tensor) -> torch.Tensor:
    """HF:models/qwen3/modeling_qwen3.py:151-155."""
    x1 = x[..., : x.shape[-1] // 2]
    x2 = x[..., x.shape[-1] // 2:]
    return torch.cat((-x2, x1), dim=-1)


def apply_rope(q: torch.Tensor, k: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor):
    """HF:models/qwen3/modeling_qwen3.py:158-181  apply_rotary_pos_emb (bf16 elementwise;
    every product and the sum round to bf16).  q,k: [B, heads, T, d]; cos,sin: [B, T, d]."""
    cos = cos.unsqueeze(1)
    sin = sin.unsqueeze(1)
    q2 = (q * cos) + (rotate_half(q) * sin)
    k2 = (k * cos) + (rotate_half(k) * sin)
    return q2, k2


def attention_sdpa(q, k, v, scaling: float, causal: bool):
    """HF:integrations/sdpa_attention.py:40-104 with attention_mask=None: GQA handled by
    `enable_gqa=True`, `is_causal` only when T > 1."""
    return F.scaled_dot_product_attention(
        q, k, v, attn_mask=None, dropout_p=0.0, scale=scaling, is_causal=causal, enable_gqa=True
    )


def attention_explicit(q, k, v, scaling: float, causal: bool, p_dtype=torch.bfloat16):
    """The rounding points the CUDA kernels implement, written out: fp32 scores from bf16
    q,k; fp32 softmax statistics; un-normalised probabilities rounded to bf16 before the
    P.V product (as torch's CPU flash kernel does for reduced types); fp32 P.V accumulate;
    one division by the fp32 row sum; one rounding of the output to bf16.  Single KV block
    (global row max)."""
    B, Hq, T, d = q.shape
    Hk = k.shape[1]
    g = Hq // Hk
    kf = k.to(torch.float32).repeat_interleave(g, dim=1)
    vf = v.to(torch.float32).repeat_interleave(g, dim=1)
    s = torch.matmul(q.to(torch.float32), kf.transpose(-1, -2)) * scaling
    if causal:
        S = k.shape[2]
        mask = torch.ones(T, S, dtype=torch.bool).tril(diagonal=S - T)
        s = s.masked_fill(~mask, float("-inf"))
    m = s.max(dim=-1, keepdim=True).values
    p = torch.exp(s - m)
    l = p.sum(dim=-1, keepdim=True)
    p = p.to(p_dtype).to(torch.float32)
    o = torch.matmul(p, vf) / l
    return o.to(q.dtype)


def swiglu_mlp(x, gate_w, up_w, down_w):
    """HF:models/qwen3/modeling_qwen3.py:81-83  Qwen3MLP.forward: every Linear rounds to
    bf16; silu and the product are bf16 elementwise ops."""
    return F.linear(F.silu(F.linear(x, gate_w)) * F.linear(x, up_w), down_w)


@dataclass
class LayerTrace:
    attn_in: torch.Tensor | None = None
    q: torch.Tensor | None = None
    k: torch.Tensor | None = None
    v: torch.Tensor | None = None
    attn_out: torch.Tensor | None = None
    h_mid: torch.Tensor | None = None
    h_out: torch.Tensor | None = None


@dataclass
class KVState:
    k: list = field(default_factory=list)  # per layer [B, Hk, S, d]
    v: list = field(default_factory=list)


class Restated:
    """Plain-torch Qwen3 forward over an HF-named state dict."""

    def __init__(self, arch: ArchConfig, sd: dict[str, torch.Tensor], attention=attention_sdpa):
        self.arch = arch
        self.sd = sd
        self.attention = attention

    def w(self, name: str) -> torch.Tensor:
        return self.sd[name]

    def lm_head_weight(self) -> torch.Tensor:
        # HF:models/qwen3/modeling_qwen3.py:443,451 (tied to embed_tokens)
        if self.arch.tie_embeddings or "lm_head.weight" not in self.sd:
            return self.sd["model.embed_tokens.weight"]
        return self.sd["lm_head.weight"]

    def layer(self, i: int, h: torch.Tensor, positions: torch.Tensor, kv: KVState, trace: LayerTrace | None):
        """HF:models/qwen3/modeling_qwen3.py:305-334 Qwen3DecoderLayer.forward and
        :252-291 Qwen3Attention.forward."""
        a = self.arch
        p = f"model.layers.{i}."
        B, T, _ = h.shape
        residual = h
        x = rms_norm(h, self.w(p + "input_layernorm.weight"), a.rms_eps)
        q = F.linear(x, self.w(p + "self_attn.q_proj.weight")).view(B, T, a.num_q_heads, a.head_dim)
        k = F.linear(x, self.w(p + "self_attn.k_proj.weight")).view(B, T, a.num_kv_heads, a.head_dim)
        v = F.linear(x, self.w(p + "self_attn.v_proj.weight")).view(B, T, a.num_kv_heads, a.head_dim)
        q = rms_norm(q, self.w(p + "self_attn.q_norm.weight"), a.rms_eps).transpose(1, 2)
        k = rms_norm(k, self.w(p + "self_attn.k_norm.weight"), a.rms_eps).transpose(1, 2)
        v = v.transpose(1, 2)
        cos, sin = rope_cos_sin(a, positions)
        q, k = apply_rope(q, k, cos, sin)
        # HF:models/qwen3/modeling_qwen3.py:270-271 cache update (DynamicCache concatenation)
        if len(kv.k) <= i:
            kv.k.append(k)
            kv.v.append(v)
        else:
            kv.k[i] = torch.cat((kv.k[i], k), dim=2)
            kv.v[i] = torch.cat((kv.v[i], v), dim=2)
        ao = self.attention(q, kv.k[i], kv.v[i], a.head_dim ** -0.5, T > 1)
        ao = ao.transpose(1, 2).contiguous().reshape(B, T, a.q_size)
        o = F.linear(ao, self.w(p + "self_attn.o_proj.weight"))
        h = residual + o
        residual = h
        x2 = rms_norm(h, self.w(p + "post_attention_layernorm.weight"), a.rms_eps)
        m = swiglu_mlp(
            x2, self.w(p + "mlp.gate_proj.weight"), self.w(p + "mlp.up_proj.weight"), self.w(p + "mlp.down_proj.weight")
        )
        out = residual + m
        if trace is not None:
            trace.attn_in, trace.q, trace.k, trace.v = x, q, k, v
            trace.attn_out, trace.h_mid, trace.h_out = ao, h, out
        return out

    @torch.no_grad()
    def forward(self, ids: torch.Tensor, positions: torch.Tensor, kv: KVState, traces: list | None = None,
                last_only: bool = False):
        """HF:models/qwen3/modeling_qwen3.py:378-438 Qwen3Model.forward + :458-517 lm head.
        ids, positions: [B, T].  Returns (logits [B, T or 1, V], final hidden)."""
        a = self.arch
        h = F.embedding(ids, self.w("model.embed_tokens.weight"))
        for i in range(a.num_layers):
            tr = None
            if traces is not None:
                tr = LayerTrace()
                traces.append(tr)
            h = self.layer(i, h, positions, kv, tr)
        h = rms_norm(h, self.w("model.norm.weight"), a.rms_eps)
        hl = h[:, -1:, :] if last_only else h
        logits = F.linear(hl, self.lm_head_weight())
        return logits, h

    @torch.no_grad()
    def greedy(self, prompt: torch.Tensor, new_tokens: int):
        """generate(do_sample=False): argmax over the last position, lowest index on ties."""
        B, P = prompt.shape
        kv = KVState()
        pos = torch.arange(P)[None, :].expand(B, P)
        logits, _ = self.forward(prompt, pos, kv, last_only=True)
        out = []
        step_logits = []
        nxt = logits[:, -1, :].argmax(dim=-1)
        out.append(nxt)
        step_logits.append(logits[:, -1, :])
        for t in range(1, new_tokens):
            pos = torch.full((B, 1), P + t - 1, dtype=torch.int64)
            logits, _ = self.forward(nxt[:, None], pos, kv, last_only=True)
            nxt = logits[:, -1, :].argmax(dim=-1)
            out.append(nxt)
            step_logits.append(logits[:, -1, :])
        return torch.stack(out, dim=1), torch.stack(step_logits, dim=1)


def top2_gap(logits: torch.Tensor) -> torch.Tensor:
    """Gap between the best and second-best logit (tie-aware evidence)."""
    t = logits.to(torch.float32).topk(2, dim=-1).values
    return t[..., 0] - t[..., 1]


def hf_state_dict(model) -> dict[str, torch.Tensor]:
    sd = {k: v.detach() for k, v in model.state_dict().items()}
    return sd


def hf_cpu_decode_tok_s(arch: ArchConfig, batch: int, prompt_len: int, new_tokens: int, threads: int | None = None,
                        seed: int = 0):
    """CPU baseline leg of bench.py: HF `generate(do_sample=False)` wall time on host cores."""
    import time

    if threads:
        torch.set_num_threads(threads)
    model = hf_model(arch, seed=seed)
    ids = make_prompts(batch, prompt_len, arch.vocab)
    with torch.no_grad():
        t0 = time.perf_counter()
        model.generate(ids, attention_mask=torch.ones_like(ids), do_sample=False, max_new_tokens=1, min_new_tokens=1,
                       pad_token_id=0)
        t_prefill = time.perf_counter() - t0
        t0 = time.perf_counter()
        out = model.generate(ids, attention_mask=torch.ones_like(ids), do_sample=False, max_new_tokens=new_tokens,
                             min_new_tokens=new_tokens, pad_token_id=0)
        t_total = time.perf_counter() - t0
    decode_s = max(t_total - t_prefill, 1e-9)
    return {
        "tok_s": batch * (new_tokens - 1) / decode_s,
        "total_s": t_total,
        "prefill_s": t_prefill,
        "threads": torch.get_num_threads(),
        "tokens": out[:, prompt_len:],
    }
