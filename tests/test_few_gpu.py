"""The decode kernels of at most eight sequences (GPU), called through the C ABI: against the kernels that larger batches take (page writes bit for bit) and against
the same arithmetic in 64 bits between the bf16 roundings."""
import dataclasses

import numpy as np
import pytest
import torch

from _util import assert_bf16_close, cuda_stream_ptr, kv_swizzle, pkg, ptr

pytestmark = pytest.mark.gpu
HD, BS, EPS = 128, 16, 1e-6


@pytest.fixture(scope="module")
def lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return pkg().load_library()


def chk(lib, rc):
    assert rc == 0, lib.b2_last_error().decode()


def norm(x, gain):
    """bf16(gain * bf16(x * rstd)); the statistic in 64 bits"""
    rstd = (x.double().pow(2).mean(-1, keepdim=True) + EPS).rsqrt()
    return (gain.double() * (x.double() * rstd).to(torch.bfloat16).double()).to(torch.bfloat16)


@pytest.mark.parametrize("T", [1, 3, 8])
@pytest.mark.parametrize("N,K", [(8, 32), (40, 96), (72, 256), (264, 1024), (1024, 2048), (100, 3072), (48, 3360)])
def test_few_linear(lib, T, N, K):
    """Weight rows that fill no CTA, a K that is not the warps' multiple of 256 or takes several rounds; nothing behind row T.  The sums differ from 64 bits by fp32
    roundings, which move a bf16 result by one unit now and then (two where two roundings follow each other)."""
    g = torch.Generator().manual_seed(N * 10 + T)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16)
    gain = (1 + 0.2 * torch.randn(K, generator=g)).to(torch.bfloat16)
    for mode in (0, 1, 2):
        rows = 2 * N if mode == 2 else N
        w = (torch.randn(rows, K, generator=g) * K ** -0.5).to(torch.bfloat16)
        h = torch.randn(8, N, generator=g).to(torch.bfloat16)
        out = h.clone().cuda()
        dw, dx, dg = w.cuda(), x.cuda(), gain.cuda()
        chk(lib, lib.b2k_few_linear(ptr(dw), ptr(dx), ptr(dg), EPS, ptr(out), T, N, K, mode, cuda_stream_ptr()))
        torch.cuda.synchronize()
        y = ((x if mode == 1 else norm(x, gain)).double() @ w.double().T).to(torch.bfloat16)
        if mode == 1:
            ref = (h[:T].double() + y.double()).to(torch.bfloat16)
        elif mode == 2:
            gate, up = y[:, :N].double(), y[:, N:].double()
            ref = ((gate / (1 + torch.exp(-gate))).to(torch.bfloat16).double() * up).to(torch.bfloat16)
        else:
            ref = y
        assert_bf16_close(out[:T], ref, 3, 0.06, "mode %d" % mode, abs_floor=2.0 ** -8)
        assert torch.equal(out[T:].cpu(), h[T:])


@pytest.mark.parametrize("lens", [[1], [15, 16, 17, 2], [511, 512, 513, 0, 528], [1030, 33, 1024, 700, 1, 544, 496, 2000]])
def test_few_attn(lib, lens):
    """Contexts around a page, around the 32 pages of a cluster's first turn, several turns; a padding row.  Pages and rotated queries: those of b2k_qknorm_rope_kv."""
    nq, nkv, B = 8, 4, len(lens)
    g = torch.Generator().manual_seed(sum(lens))
    width = max(1, max((n + BS - 1) // BS for n in lens))
    blocks = B * width + 3
    bt = torch.randperm(blocks, generator=g)[:B * width].view(B, width).to(torch.int32)
    kp, vp = (torch.randn(blocks, nkv, BS, HD, generator=g).to(torch.bfloat16) for _ in range(2))
    qkv = torch.randn(B, (nq + 2 * nkv) * HD, generator=g).to(torch.bfloat16)
    qw, kw = ((1 + 0.25 * torch.randn(HD, generator=g)).to(torch.bfloat16) for _ in range(2))
    ang = torch.arange(2048)[:, None] * (1e4 ** (-torch.arange(64) / 64.0))[None, :]
    table = torch.cat([ang.cos(), ang.sin()], -1).to(torch.bfloat16)
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32)
    slots = torch.tensor([-1 if n == 0 else int(bt[b, (n - 1) // BS]) * BS + (n - 1) % BS for b, n in enumerate(lens)], dtype=torch.int32)
    d = [t.cuda() for t in (qkv, qw, kw, table, pos, slots, bt, torch.tensor(lens, dtype=torch.int32))]
    pages = [[t.cuda() for t in (kp, vp)] for _ in range(2)]
    q_out = torch.zeros(B, nq * HD, dtype=torch.bfloat16, device="cuda")
    chk(lib, lib.b2k_qknorm_rope_kv(ptr(d[0]), 0, 1, ptr(d[1]), ptr(d[2]), ptr(d[3]), ptr(d[4].clamp_min(0)), ptr(d[5]), ptr(q_out), ptr(pages[0][0]), ptr(pages[0][1]), B, nq, nkv,
                                    HD, BS, EPS, cuda_stream_ptr()))
    out = torch.full((B, nq * HD), float("nan"), dtype=torch.bfloat16, device="cuda")
    scale = HD ** -0.5
    run = lambda dst: chk(lib, lib.b2k_few_attn(ptr(d[0]), ptr(d[1]), ptr(d[2]), ptr(d[3]), ptr(d[4]), ptr(d[5]), ptr(pages[1][0]), ptr(pages[1][1]), ptr(d[6]), width, ptr(d[7]), ptr(dst),
                                                B, nq, nkv, EPS, scale, cuda_stream_ptr()))
    run(out)
    torch.cuda.synchronize()
    for a, b in zip(pages[0], pages[1]):
        assert torch.equal(a, b)
    k, v = (kv_swizzle(t.cpu()).double() for t in pages[1])
    for b, n in enumerate(lens):
        if n == 0:
            assert not out[b].any()
            continue
        idx = bt[b, :(n + BS - 1) // BS].long()
        ks, vs = (t[idx].permute(1, 0, 2, 3).reshape(nkv, -1, HD)[:, :n] for t in (k, v))
        q = q_out[b].cpu().double().view(nkv, 2, HD)
        ref = torch.softmax(torch.einsum("gqd,gkd->gqk", q, ks) * scale, -1) @ vs
        assert_bf16_close(out[b], ref.reshape(-1).to(torch.bfloat16), 2, 0.05, "sequence of %d" % n, abs_floor=2.0 ** -12)
    again = torch.empty_like(out)
    run(again)
    assert torch.equal(out, again)


@pytest.mark.parametrize("T", [1, 5, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(5, 32), (8, 1024), (9001, 96), (20003, 2048), (1189, 4096), (148 * 8 * 4 + 1, 256)])
def test_few_head(lib, T, N, K):
    """Fewer tiles than SMs, a last tile that is not whole, tiles under way behind the end, K that leaves warps without a chunk.  Sums of exact products in fp32: K
    roundings of 2^-24 of the sum of absolute values at most, and one of the scaling."""
    if T > 8 and K > 2048:
        assert lib.b2k_few_head(ptr(torch.zeros(1, device="cuda")), ptr(torch.zeros(1, device="cuda")), ptr(torch.zeros(1, device="cuda")), T, N, K, 1.0, cuda_stream_ptr()) != 0
        return
    g = torch.Generator().manual_seed(N + T)
    x, w = torch.randn(T, K, generator=g).to(torch.bfloat16).cuda(), torch.randn(N, K, generator=g).to(torch.bfloat16).cuda()
    out = torch.full((T + 1, N), 7.0, device="cuda")
    chk(lib, lib.b2k_few_head(ptr(w), ptr(x), ptr(out), T, N, K, 0.3, cuda_stream_ptr()))
    torch.cuda.synchronize()
    ref, mag = 0.3 * (x.double() @ w.double().T), 0.3 * (x.double().abs() @ w.double().abs().T)
    assert ((out[:T].double() - ref).abs() <= (K + 4) * 2.0 ** -24 * mag).all() and (out[T] == 7.0).all()


def small_model():
    P = pkg()
    torch.manual_seed(0)
    cfg = P.EngineConfig(num_layers=1, hidden=256, num_q_heads=4, num_kv_heads=2, head_dim=128, intermediate=512, vocab=20003, max_model_len=64, num_blocks=40, max_seqs=8,
                         max_batch_tokens=128)
    names = {"model.embed_tokens.weight": (20003, 256), "model.norm.weight": (256,), "model.layers.0.input_layernorm.weight": (256,),
             "model.layers.0.post_attention_layernorm.weight": (256,), "model.layers.0.self_attn.q_proj.weight": (512, 256), "model.layers.0.self_attn.k_proj.weight": (256, 256),
             "model.layers.0.self_attn.v_proj.weight": (256, 256), "model.layers.0.self_attn.o_proj.weight": (256, 512), "model.layers.0.self_attn.q_norm.weight": (128,),
             "model.layers.0.self_attn.k_norm.weight": (128,), "model.layers.0.mlp.gate_proj.weight": (512, 256), "model.layers.0.mlp.up_proj.weight": (512, 256),
             "model.layers.0.mlp.down_proj.weight": (256, 512)}
    sd = {n: (torch.ones(s) if len(s) == 1 else 0.05 * torch.randn(s)).to(torch.bfloat16) for n, s in names.items()}
    return P, cfg, sd


@pytest.mark.parametrize("n", [1, 5, 8, 9, 16])
def test_few_head_argmax(lib, n):
    """The lm head of at most sixteen rows through the engine's own entry, behind a prompt and behind decode steps: bf16 logits against 64-bit products of the final hidden
    rows (one rounding to eight bits, at most 2^-8 of the number, and fp32 sums of exact products), and the tokens."""
    P, cfg, sd = small_model()
    head = sd["model.embed_tokens.weight"].double().cuda()
    with P.Engine(dataclasses.replace(cfg, max_seqs=16, num_blocks=80, max_batch_tokens=512)) as e:
        e.load_state_dict(sd)
        e.set_debug(logits=True, hidden=True)
        sids = [e.seq_create(32) for _ in range(n)]
        toks = e.prefill(sids, [list(range(3 + i, 9 + 2 * i)) for i in range(n)])
        ends = np.cumsum([6 + i for i in range(n)]) - 1
        for step in range(3):
            logits = np.asarray(e.get_logits(n))
            rows = e.get_hidden(cfg.num_layers, ends[-1] + 1)[ends] if step == 0 else e.get_hidden(cfg.num_layers, n)
            x = torch.from_numpy(rows.astype(np.int32) << 16).view(torch.float32).double().cuda()
            ref, mag = x @ head.T, x.abs() @ head.abs().T
            got = torch.from_numpy(logits.astype(np.float64)).cuda()
            assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 2 * (256 + 4) * 2.0 ** -24 * mag).all()
            best = logits.max(1)
            for i in range(n):   # the lowest index of the largest bf16 value
                assert int(np.flatnonzero(logits[i] == best[i])[0]) == int(toks[i])
            toks = e.decode_step(sids, toks)


def test_decode_steps_whose_tokens_nobody_reads():
    """Steps with and without their tokens in turn, a batch that changes between them, given tokens and the engine's own, a run of several steps: the same tokens as from
    steps that are all read, one after the other."""
    P, cfg, sd = small_model()
    prompts = [list(range(3 + i, 9 + 2 * i)) for i in range(3)]
    with P.Engine(cfg) as e:
        e.load_state_dict(sd)
        sids = [e.seq_create(48) for _ in prompts]
        want = [list(map(int, e.prefill(sids, prompts)))]
        for _ in range(14):
            want.append(list(map(int, e.decode_step(sids))))
    with P.Engine(cfg) as e:
        e.load_state_dict(sd)
        sids = [e.seq_create(48) for _ in prompts]
        assert list(map(int, e.prefill(sids, prompts))) == want[0]
        e.decode_step(sids, want_output=False)
        e.decode_step(sids, want_output=False)
        assert list(map(int, e.decode_step(sids))) == want[3]
        assert list(map(int, e.decode_step(sids, want[3]))) == want[4]
        e.decode_step(sids, want[4], want_output=False)
        e.decode_step(sids, want[5], want_output=False)
        assert list(map(int, e.decode_step(sids, want[6]))) == want[7]
        for i in (2, 0, 1):                                   # each alone, then together again
            assert int(e.decode_step([sids[i]], [want[7][i]])[0]) == want[8][i]
        assert list(map(int, e.decode_step(sids, want[8]))) == want[9]
        toks, _ = e.decode_run(sids, 3)
        assert [list(map(int, r)) for r in np.asarray(toks)] == want[10:13]
        assert list(map(int, e.decode_step(sids))) == want[13]
        assert list(map(int, e.decode_step(sids))) == want[14]


def test_contexts_that_cross_the_line(monkeypatch):
    """Five sequences whose contexts pass the number of tokens from which the larger batches' kernels take their steps: logits of both sides of the line against an
    engine that takes those kernels always.  Two sequences hold most of it: the longest one times the bucket of eight is far beyond the line before."""
    P, cfg, sd = small_model()
    cfg = dataclasses.replace(cfg, max_model_len=12288, num_blocks=1600, max_batch_tokens=12288)
    g = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, 20003, (n,), generator=g).tolist() for n in (12150, 12151, 88, 88, 87)]   # 24564 in all: 24576 behind the second of five steps
    given = torch.randint(0, 20003, (5, 5), generator=g).tolist()

    def steps(few):
        monkeypatch.setenv("B2_FEW", few)
        with P.Engine(cfg) as e:
            e.load_state_dict(sd)
            e.set_debug(logits=True)
            sids = [e.seq_create(len(p) + 8) for p in prompts]
            for i, p in zip(sids, prompts):
                e.prefill([i], [p])
            out = []
            for toks in given:
                e.decode_step(sids, toks, want_output=False)
                out.append(np.asarray(e.get_logits(5)).astype(np.float32))
            return np.stack(out)
    a, b = steps("1"), steps("0")
    assert np.isfinite(a).all()
    # Below the line the attention's weights are rounded in one form only, and nothing behind them rounds alike: twelve bf16 roundings on either side (attention, projections,
    # residuals, norms, activation, logits), each at most 2^-8 / sqrt(3) of the number in the root mean square, independent: sqrt(24) of them are 2^-6.5.
    # Beyond it the kernels are the same, and only the keys and values of the two steps before it differ.
    apart = np.linalg.norm(a - b, axis=2) / np.linalg.norm(b, axis=2)
    assert apart[:2].max() <= 2.0 ** -6.5 and apart[:2].min() > 2.0 ** -10 and apart[2:].max() <= 2.0 ** -10, apart
