"""Kernels of the layer-list families (GPU), called through the C ABI (include/b2_engine.h, b2k_*) and compared with the same arithmetic in 64 bits."""
import pytest
import torch

from _util import cuda_stream_ptr, pkg, ptr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return pkg().load_library()


def chk(lib, rc):
    assert rc == 0, lib.b2_last_error().decode()


DECAY, DELTA, DELTA_HEAD, DECAY_HEAD, BONUS = range(5)


def scan_inputs(lengths, heads, kv, dim, vdim, rule, seed):
    g = torch.Generator().manual_seed(seed)
    T = sum(lengths)
    f = lambda *s: torch.randn(*s, generator=g)
    head = rule in (DELTA_HEAD, DECAY_HEAD)
    decay = torch.exp(-torch.exp(f(T, heads if head else heads * dim) - 2.0))
    decay[torch.rand(decay.shape, generator=g) < 0.02] = 0.0        # a memory that is gone at once
    decay[torch.rand(decay.shape, generator=g) < 0.02] = 1e-9
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    k = f(T, kv, dim)
    d = {"q": f(T, kv, dim), "k": unit(k) if rule in (DELTA, DELTA_HEAD) else k * dim ** -0.5, "v": f(T, heads, vdim), "decay": decay,
         "beta": torch.rand(T, heads, generator=g), "skip": f(heads), "bonus": f(heads, dim)}
    return {n: t.float() for n, t in d.items()}


def scan_reference(x, lengths, heads, kv, dim, vdim, rule, qscale, s0):
    """[T][heads][vdim] and the states behind the last tokens, in 64 bits."""
    d = {n: t.double().cuda() for n, t in x.items()}
    rep = heads // kv
    out, states, at = [], [], 0
    for i, n in enumerate(lengths):
        S = s0[i].double().cuda().clone()          # [heads][dim][vdim]
        for t in range(at, at + n):
            q, k = d["q"][t].repeat_interleave(rep, 0), d["k"][t].repeat_interleave(rep, 0)
            v, b = d["v"][t], d["beta"][t][:, None]
            a = d["decay"][t].view(heads, -1)[:, :, None]
            if rule == BONUS:
                o = torch.einsum("hd,hdv->hv", q, S) + (q * d["bonus"] * k).sum(1, keepdim=True) * v
                S = a * S + k[:, :, None] * v[:, None, :]
            else:
                S = a * S
                w = v if rule == DECAY else b * v if rule == DECAY_HEAD else b * (v - torch.einsum("hd,hdv->hv", k, S))
                S = S + k[:, :, None] * w[:, None, :]
                o = torch.einsum("hd,hdv->hv", q, S)
            o = o * qscale
            out.append(o + d["skip"][:, None] * v if rule == DECAY_HEAD else o)
        states.append(S)
        at += n
    return torch.stack(out), torch.stack(states)


def run_scan(lib, x, lengths, heads, kv, dim, vdim, rule, qscale, state, starts, single=False):
    """One launch over all portions; state [portions][2][heads][dim][vdim] on the GPU, updated in place."""
    T, n = sum(lengths), len(lengths)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    seq, first, end, pos, last, at = [], [], [], [], [], 0
    for i, m in enumerate(lengths):
        seq += [i] * m
        first += [at] * m
        end += [at + m] * m
        pos += list(range(starts[i], starts[i] + m))
        at += m
        last.append(at - 1)
    d = {name: t.cuda().contiguous() for name, t in x.items()}
    out = torch.full((T, heads * vdim), float("nan"), device="cuda")
    idx = [i32(v) for v in (last, seq, first, end, pos, list(range(T)))]
    chk(lib, lib.b2k_state_scan(ptr(d["q"]), kv * dim, ptr(d["k"]), kv * dim, ptr(d["v"]), heads * vdim, ptr(d["decay"]), ptr(d["beta"]), ptr(d["skip"]), ptr(d["bonus"]),
                                heads, kv, dim, vdim, rule, qscale, ptr(state), n, None if single else ptr(idx[0]), *[ptr(t) for t in idx[1:]], ptr(out), cuda_stream_ptr()))
    torch.cuda.synchronize()
    return out.view(T, heads, vdim)


def rel2(a, b):
    return ((a.double() - b).norm() / b.norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("rule", [DECAY, DELTA, DELTA_HEAD, DECAY_HEAD, BONUS])
@pytest.mark.parametrize("dim,vdim", [(128, 64), (64, 36), (96, 20), (20, 128), (18, 10), (160, 24)])
def test_state_scan(lib, rule, dim, vdim):
    """Portions around the chunk of eight tokens, a state to start from, decays down to zero; the sizes that the packed form does not hold ((18, 10): rows that are
    no multiples of 16 bytes, 160: wider keys) take the generic one.  Bound: a number of the result passes through at most dim + tokens roundings of 2^-24 each,
    of which the sums' random signs leave a few; an eighth of that count is allowed in the 2-norm."""
    heads, kv, lengths, starts, qscale = 4, 2, [1, 7, 8, 9, 33, 16], [0, 3, 0, 4, 6, 1], 0.37
    x = scan_inputs(lengths, heads, kv, dim, vdim, rule, seed=dim * 1000 + vdim * 10 + rule)
    g = torch.Generator().manual_seed(5)
    state = torch.zeros(len(lengths), 2, heads, dim, vdim)
    s0 = torch.zeros(len(lengths), heads, dim, vdim)
    for i, p in enumerate(starts):
        if p > 0:
            s0[i] = torch.randn(heads, dim, vdim, generator=g)
            state[i, (p - 1) & 1] = s0[i]
    ref, ref_s = scan_reference(x, lengths, heads, kv, dim, vdim, rule, qscale, s0)
    dev = state.cuda()
    got = run_scan(lib, x, lengths, heads, kv, dim, vdim, rule, qscale, dev, starts)
    got_s = torch.stack([dev[i, (p + n - 1) & 1] for i, (p, n) in enumerate(zip(starts, lengths))])
    tol = (dim + max(lengths)) / 8 * 2.0 ** -24
    assert rel2(got, ref) < tol and rel2(got_s, ref_s) < tol

    # one token per launch: the same, and the same bits where no factor is carried through a portion
    dev1 = state.cuda()
    at, per = 0, []
    for i, n in enumerate(lengths):
        per.append((at, n))
        at += n
    one = torch.empty_like(got)
    for step in range(max(lengths)):
        who = [i for i, n in enumerate(lengths) if step < n]
        sub = {name: t if name in ("skip", "bonus") else torch.stack([t[per[i][0] + step] for i in who]) for name, t in x.items()}
        sel = dev1[who].contiguous()
        o = run_scan(lib, sub, [1] * len(who), heads, kv, dim, vdim, rule, qscale, sel, [starts[i] + step for i in who], single=True)
        for j, i in enumerate(who):
            dev1[i] = sel[j]
            one[per[i][0] + step] = o[j]
    if rule in (DECAY, DELTA, BONUS):
        assert torch.equal(one, got)
    else:
        assert rel2(one, ref) < tol


@pytest.mark.parametrize("rule", [DECAY, DELTA, DELTA_HEAD, DECAY_HEAD, BONUS])
def test_state_scan_many_portions(lib, rule):
    """Enough portions for four columns per lane: the bits of a portion are those it has alone (two columns per lane)."""
    heads, kv, dim, vdim, n = 4, 4, 64, 128, 19
    one = scan_inputs([n], heads, kv, dim, vdim, rule, seed=rule)
    zero = lambda p: torch.zeros(p, 2, heads, dim, vdim, device="cuda")
    alone = run_scan(lib, one, [n], heads, kv, dim, vdim, rule, 1.0, zero(1), [0])
    many = 24   # 24 * 4 * 16 groups of eight columns
    x = {name: t if name in ("skip", "bonus") else torch.cat([t] * many) for name, t in one.items()}
    got = run_scan(lib, x, [n] * many, heads, kv, dim, vdim, rule, 1.0, zero(many), [0] * many)
    assert torch.equal(got, alone.repeat(many, 1, 1))


@pytest.mark.parametrize("tile", [128, 256, 0])
@pytest.mark.parametrize("N,K", [(128, 64), (64, 192), (704, 320), (256, 1024), (300, 128)])
def test_linear_sum_groups(lib, tile, N, K):
    """Ragged groups around the tiles of 128 and 256 rows, empty ones, weight rows that fill no pair of 256; nothing is written behind the last row.  Sums of K products
    of bf16 numbers, exact in fp32, in fp32: K roundings of 2^-24 of the sum of their absolute values at most (the activation squares the sum and rounds to bf16)."""
    sizes = [0, 1, 127, 128, 129, 255, 0, 256, 257, 300, 64]
    g = torch.Generator().manual_seed(N + K)
    rows, G = sum(sizes), len(sizes)
    x = torch.randn(rows, K, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(G, N, K, generator=g) * K ** -0.5).to(torch.bfloat16).cuda()
    off = torch.tensor([0] + list(torch.tensor(sizes).cumsum(0)), dtype=torch.int32, device="cuda")
    ref, mag = torch.empty(rows, N, dtype=torch.float64, device="cuda"), torch.empty(rows, N, dtype=torch.float64, device="cuda")
    for i in range(G):
        a, b = int(off[i]), int(off[i + 1])
        ref[a:b] = x[a:b].double() @ w[i].double().T
        mag[a:b] = x[a:b].double().abs() @ w[i].double().abs().T
    for epilogue, dtype in ((0, torch.float32), (1, torch.bfloat16)):
        out = torch.full((rows + 8, N), 7.0, dtype=dtype, device="cuda")
        chk(lib, lib.b2k_linear_sum(ptr(x), ptr(w), ptr(off), G, rows, ptr(out), N, K, epilogue, tile, cuda_stream_ptr()))
        torch.cuda.synchronize()
        assert (out[rows:] == 7.0).all()
        got = out[:rows].double()
        err = K * 2.0 ** -24 * mag
        if epilogue == 0:
            assert ((got - ref).abs() <= err).all()
        else:
            want = ref.clamp_min(0.0) ** 2
            assert ((got - want).abs() <= 2.0 ** -8 * want + 2.1 * err * (ref.abs() + err)).all()
    one = torch.full((rows, N), 7.0, device="cuda")   # one block
    chk(lib, lib.b2k_linear_sum(ptr(x), ptr(w[0]), None, 1, rows, ptr(one), N, K, 0, tile, cuda_stream_ptr()))
    torch.cuda.synchronize()
    want, mag = x.double() @ w[0].double().T, x.double().abs() @ w[0].double().abs().T
    assert ((one.double() - want).abs() <= K * 2.0 ** -24 * mag).all()
    # sums of 128, eight additions of sixteen products with at most a unit in the last place lost, joined by additions to nearest
    fine = torch.full((rows + 1, N), 7.0, device="cuda")
    chk(lib, lib.b2k_linear_sum(ptr(x), ptr(w[0]), None, 1, rows, ptr(fine), N, K, 2, tile, cuda_stream_ptr()))
    torch.cuda.synchronize()
    assert (fine[rows] == 7.0).all() and ((fine[:rows].double() - want).abs() <= (8 + K / 128) * 2.0 ** -23 * mag).all()


@pytest.mark.parametrize("tile", [128, 256, 0])
@pytest.mark.parametrize("rows,N,K", [(1, 64, 64), (5, 300, 128), (127, 128, 192), (129, 200, 320), (300, 704, 1024), (257, 256, 3072)])
def test_linear_split3(lib, tile, rows, N, K):
    """fp32 rows as three bf16 planes: numbers of all sizes, the largest ones, infinities and NaN.  Products are exact; every addition inside a chunk of 128 (three
    times 128 products, sixteen at a time, summed with at most one unit in the last place lost) and between chunks costs at most 2^-23 of the sum of absolute values."""
    g = torch.Generator().manual_seed(rows + N + K)
    x = torch.randn(rows, K, generator=g) * torch.exp2(torch.randint(-20, 20, (rows, K), generator=g).float())
    w = (torch.randn(N, K, generator=g) * K ** -0.5).to(torch.bfloat16)
    dx, dw, planes = x.cuda(), w.cuda(), torch.empty(3, rows, K, dtype=torch.bfloat16, device="cuda")
    def run(xs):
        out = torch.full((rows + 3, N), 7.0, device="cuda")
        chk(lib, lib.b2k_linear_split3(ptr(xs), ptr(planes), ptr(dw), ptr(out), rows, N, K, tile, cuda_stream_ptr()))
        torch.cuda.synchronize()
        assert (out[rows:] == 7.0).all()
        return out[:rows].double()
    got = run(dx)
    assert torch.equal(planes.double().sum(0), dx.double())
    ref, mag = dx.double() @ dw.double().T, dx.double().abs() @ dw.double().abs().T
    assert ((got - ref).abs() <= (24 + K / 128) * 2.0 ** -23 * mag).all()
    odd = x.clone()
    odd[0, :4] = torch.tensor([3.4028234e38, 1e-42, -3.4e38, 0.0])    # rounds to infinity in bf16; below bf16's normal numbers
    if rows > 4:
        odd[2, 1], odd[4, 2] = float("inf"), float("nan")
    got = run(odd.cuda())
    if rows > 4:
        fine = w[:, 1].float() != 0
        assert torch.equal(got[2].cpu()[fine], (w[:, 1].double() * float("inf"))[fine]) and torch.isnan(got[4]).all()
    keep = [r for r in range(rows) if r not in (0, 2, 4)]
    if keep:
        assert ((got[keep] - ref[keep]).abs() <= (24 + K / 128) * 2.0 ** -23 * mag[keep]).all()
    big, size = odd[0].double().cuda() @ dw.double().T, odd[0].double().abs().cuda() @ dw.double().abs().T
    sure = size < 1e38                                                # (else partial sums may pass the largest number on the way)
    assert sure.any() and torch.isfinite(planes[:, 0].float()).all() and ((got[0] - big).abs() <= 2.0 ** -15 * size)[sure].all()


@pytest.mark.parametrize("rows,N,K,rows_at_a_time,cols_at_a_time", [(1, 64, 64, 1, 64), (255, 300, 128, 255, 256), (300, 600, 320, 256, 256), (1030, 257, 64, 300, 600),
                                                                     (513, 1100, 192, 512, 511)])
def test_linear_split3_wide(lib, rows, N, K, rows_at_a_time, cols_at_a_time):
    """fp32 weights that are bf16 numbers, narrowed into the scratch: the bits of the product with bf16 weights, whole and in pieces of whole tiles, and nothing else written."""
    g = torch.Generator().manual_seed(rows + N + K)
    x = (torch.randn(rows, K, generator=g) * torch.exp2(torch.randint(-20, 20, (rows, K), generator=g).float())).cuda()
    w = (torch.randn(N, K, generator=g) * K ** -0.5).to(torch.bfloat16).cuda()
    w[0, 0], w[N - 1, K - 1] = float("inf"), -0.0
    whole, planes = torch.empty(rows, N, device="cuda"), torch.empty(3, rows, K, dtype=torch.bfloat16, device="cuda")
    chk(lib, lib.b2k_linear_split3(ptr(x), ptr(planes), ptr(w), ptr(whole), rows, N, K, 0, cuda_stream_ptr()))
    nx, nw = rows_at_a_time * K, cols_at_a_time * K
    planes, narrow = torch.full((3 * nx + 8,), 3.0, dtype=torch.bfloat16, device="cuda"), torch.full((nw + 8,), 3.0, dtype=torch.bfloat16, device="cuda")
    out, wide = torch.full((rows + 3, N), 7.0, device="cuda"), w.float()
    chk(lib, lib.b2k_linear_split3_wide(ptr(x), ptr(wide), ptr(planes), nx, ptr(narrow), nw, ptr(out), rows, N, K, cuda_stream_ptr()))
    torch.cuda.synchronize()
    assert torch.equal(out[:rows].view(torch.int32), whole.view(torch.int32)) and (out[rows:] == 7.0).all()
    assert (planes[3 * nx:] == 3.0).all() and (narrow[nw:] == 3.0).all()
    if rows > 256:   # no whole tile fits
        assert lib.b2k_linear_split3_wide(ptr(x), ptr(wide), ptr(planes), 255 * K, ptr(narrow), nw, ptr(out), rows, N, K, cuda_stream_ptr()) != 0


@pytest.mark.parametrize("rows,groups,N,K", [(1, 4, 64, 64), (65, 4, 320, 128), (300, 4, 2048, 192), (257, 3, 256, 64)])
def test_linear_sum_equal_groups(lib, rows, groups, N, K):
    """Groups of the same size without a table: the same bits as a launch for each."""
    g = torch.Generator().manual_seed(rows)
    x, w = (torch.randn(groups, n, K, generator=g).to(torch.bfloat16).cuda() for n in (rows, N))
    for tile in (128, 256):
        out, one = torch.full((groups * rows + 1, N), float("nan"), device="cuda"), torch.empty(groups, rows, N, device="cuda")
        chk(lib, lib.b2k_linear_sum(ptr(x), ptr(w), None, groups, groups * rows, ptr(out), N, K, 0, tile, cuda_stream_ptr()))
        for i in range(groups):
            chk(lib, lib.b2k_linear_sum(ptr(x[i]), ptr(w[i]), None, 1, rows, ptr(one[i]), N, K, 0, tile, cuda_stream_ptr()))
        assert torch.equal(out[:-1].view_as(one), one) and torch.isnan(out[-1]).all()
    assert lib.b2k_linear_sum(ptr(x), ptr(w), None, groups, groups * rows + 1, ptr(out), N, K, 0, 128, cuda_stream_ptr()) != 0


@pytest.mark.parametrize("rows,N,K,tile", [(129, 256, 64, 128), (300, 320, 192, 256), (700, 1024, 1024, 0)])
def test_linear_xielu(lib, rows, N, K, tile):
    """Against 64 bits: the activation's slope is at most 2 softplus(p) |z| + 1/2 and 1.2 below zero, its argument is an fp32 sum, the result one rounding to bf16."""
    g = torch.Generator().manual_seed(rows)
    x, w = torch.randn(rows, K, generator=g).to(torch.bfloat16), (torch.randn(N, K, generator=g) * K ** -0.5).to(torch.bfloat16)
    pq = torch.tensor([0.3, -0.2])
    act = torch.full((rows + 1, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    dx, dw, dp = x.cuda(), w.cuda(), pq.cuda()
    chk(lib, lib.b2k_linear_xielu(ptr(dx), ptr(dw), ptr(dp), ptr(act), rows, N, K, tile, cuda_stream_ptr()))
    z = x.double() @ w.double().t()
    ap, an = torch.nn.functional.softplus(pq.double())
    ref = torch.where(z > 0, ap * z * z + z / 2, (0.5 + an) * (torch.expm1(z) - z) + z / 2)
    assert torch.isnan(act[rows]).all()
    err = (act[:rows].cpu().double() - ref).abs()
    assert (err <= 2.0 ** -8 * ref.abs() + (2 * z.abs() + 1) * 2.0 ** -17).all(), err.max()


@pytest.mark.parametrize("T,I,K", [(256, 128, 256), (300, 384, 512), (513, 1024, 1024)])
def test_gateup_clamped(lib, T, I, K):
    """Against 64 bits: gate and up are fp32 sums (2^-17 of a few units), both factors are at most limit and limit + 1 wide, the result is one rounding to bf16."""
    g = torch.Generator().manual_seed(T)
    x, w = torch.randn(T, K, generator=g).to(torch.bfloat16), (torch.randn(2 * I, K, generator=g) * 3 * K ** -0.5).to(torch.bfloat16)
    act = torch.full((T + 1, I), float("nan"), dtype=torch.bfloat16, device="cuda")
    dx, dw = x.cuda(), w.cuda()
    limit, sharp = 5.0, 1.7
    chk(lib, lib.b2k_gateup_clamped(ptr(dx), ptr(dw), ptr(act), T, I, K, limit, sharp, cuda_stream_ptr()))
    z = x.double() @ w.double().t()
    gate, up = z[:, :I].clamp(max=limit), z[:, I:].clamp(-limit, limit)
    ref = gate * torch.sigmoid(sharp * gate) * (up + 1)
    assert torch.isnan(act[T]).all()
    err = (act[:T].cpu().double() - ref).abs()
    assert (err <= 2.0 ** -8 * ref.abs() + 2.0 ** -14).all(), err.max()


@pytest.mark.parametrize("heads,dim,rot,rank,rot_dims", [(16, 128, 64, 512, 64), (1, 4, 64, 4, 64), (16, 128, 0, 512, 0), (5, 12, 8, 1024, 6), (3, 132, 12, 36, 2), (1, 4, 4, 260, 4), (9, 64, 24, 132, 24)])
def test_latent_finish_forms_agree(lib, heads, dim, rot, rank, rot_dims):
    """The form that moves four numbers at a time against the general one (which rows off a 16-byte boundary take), bit for bit, and both against 64 bits.  (One head: tokens enough for
    roundings of the key's pairs that differ to fall on both sides of a bf16 edge, one in 50 000.)"""
    g = torch.Generator().manual_seed(rank + heads)
    T, kv0 = 40000 if heads == 1 and rot == 64 else 300, heads * (dim + rot)
    ld = kv0 + rank + rot + 4
    qd = torch.randn(T, ld, generator=g) * torch.exp(torch.randn(T, 1, generator=g))
    gain, pos = 1.0 + 0.1 * torch.randn(rank, generator=g), torch.randint(0, 5000, (T,), generator=g, dtype=torch.int32)
    slots = torch.randperm(T + 9, generator=g)[:T].to(torch.int32)
    slots[::7] = -1
    got = []
    for off in (0, 1):
        buf = torch.zeros(T * ld + 4, device="cuda")
        x = buf[off:off + T * ld]
        x.copy_(qd.view(-1))
        dg, dp, ds = gain.cuda(), pos.cuda(), slots.cuda()
        nope, qr = torch.full((T, heads * dim), float("nan"), dtype=torch.bfloat16, device="cuda"), torch.full((T, max(heads * rot, 1)), float("nan"), device="cuda")
        cache = torch.full((T + 9, rank + rot), 7.0, dtype=torch.bfloat16, device="cuda")
        chk(lib, lib.b2k_latent_finish(ptr(x), ld, heads, dim, rot, rank, rot_dims, 10000.0, 1e-6, 1, ptr(dg), ptr(dp), ptr(ds), ptr(nope), ptr(qr), ptr(cache), T, cuda_stream_ptr()))
        torch.cuda.synchronize()
        got.append((nope.cpu(), qr.cpu()[:, :heads * rot], cache.cpu()))
    for a, b in zip(*got):
        assert torch.equal(a, b), (a.float() - b.float()).abs().max()
    lat = qd[:, kv0:kv0 + rank].double()
    ref = lat / torch.sqrt((lat * lat).mean(1, keepdim=True) + 1e-6) * gain.double()
    seen = slots >= 0
    rows = got[0][2][slots[seen].long(), :rank].double()
    assert ((rows - ref[seen]).abs() <= 2.0 ** -8 * ref[seen].abs() + 1e-6).all()


@pytest.mark.parametrize("heads,softcap,turned,bs,pieces", [(32, 20.0, True, 16, False), (32, 0.0, False, 64, True), (16, 50.0, True, 32, True), (8, 3.0, False, 16, False)])
def test_heads_premix(lib, heads, softcap, turned, bs, pieces):
    """Portions around the tiles of 64, the units of 8 or 16 tokens and the blocks of 128 keys, some behind earlier tokens; `pieces`: a scratch that holds two tiles' units at most.
    Against 64 bits over the same queries (value + remainder), keys and values: scores and weights carry sixteen bits, so what is left is fp32 sums and the bf16 result, as in the
    test below."""
    g = torch.Generator().manual_seed(heads * 10 + bs)
    portions = [(0, 1), (0, 17), (100, 64), (3, 33), (200, 130), (0, 256), (121, 7), (127, 2)]            # (earlier tokens, tokens)
    kv, T, width = heads // 2, sum(n for _, n in portions), max((p + n + bs - 1) // bs for p, n in portions)
    pages = len(portions) * width + 2
    bt = torch.randperm(pages, generator=g)[:len(portions) * width].view(-1, width).to(torch.int32)
    q = torch.randn(T, heads, 128, generator=g)
    hi = q.to(torch.bfloat16)
    lo = (q - hi.float()).to(torch.bfloat16)
    planes = torch.stack([hi, lo], 2).view(T, kv, 2, 2, 128).permute(1, 0, 2, 3, 4).contiguous()
    kc, vc = (torch.randn(pages, bs, kv * 128, generator=g).to(torch.bfloat16) for _ in range(2))
    talk = torch.eye(heads) + 0.2 * torch.randn(heads, heads, generator=g)
    ang = torch.rand(T, 64, generator=g) * 6.0
    turn = torch.cat([torch.cos(ang), torch.sin(ang)], 1).contiguous()
    tiles, at = [], 0
    for b, (p, n) in enumerate(portions):
        tiles += [(at + i, p + i, min(64, n - i), b) for i in range(0, n, 64)]
        at += n
    host = torch.tensor(tiles, dtype=torch.int32)
    unit = heads * (8 if heads == 32 else 16) * 128
    units = [(r + 7 if heads == 32 else r + 15) // (8 if heads == 32 else 16) * ((p + r - 1) // 128 + 1) for _, p, r, _ in tiles]
    room = (2 * max(units) if pieces else sum(units)) * unit
    dev = [t.cuda() for t in (planes, kc, vc, bt, host, talk, turn)]
    scratch = torch.full((room,), float("nan"), device="cuda")
    out = torch.full((T + 1, heads * 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    scale = 128 ** -0.5
    call = lambda room: lib.b2k_heads_premix(ptr(dev[0]), ptr(dev[1]), ptr(dev[2]), pages * bs, heads, scale, softcap, ptr(talk), ptr(dev[6]) if turned else None, ptr(dev[3]), width, bs,
                                             ptr(dev[4]), ptr(host), len(tiles), ptr(out), T, ptr(scratch), room, cuda_stream_ptr())
    chk(lib, call(room))
    torch.cuda.synchronize()
    assert torch.isnan(out[T]).all() and call(unit) != 0   # (a tile that does not fit is refused)
    at = 0
    for b, (p, n) in enumerate(portions):
        idx, S = bt[b].long(), p + n
        k, v = (c[idx].reshape(-1, kv, 128)[:S].double().repeat_interleave(2, 1) for c in (kc, vc))
        s = torch.einsum("ihd,jhd->hij", (hi.double() + lo.double())[at:at + n], k) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = torch.einsum("ab,bij->aij", talk.double(), s)
        pr = torch.softmax(s.masked_fill(torch.arange(S)[None, :] > torch.arange(p, S)[:, None], float("-inf")), -1)
        ref, mag = (torch.einsum("hij,jhd->ihd", pr, x) for x in (v, v.abs()))
        if turned:
            c, sn = (x[at:at + n, None, :].double() for x in (turn[:, :64], turn[:, 64:]))
            ref = torch.cat([ref[..., :64] * c + ref[..., 64:] * sn, ref[..., 64:] * c - ref[..., :64] * sn], -1)
            mag = mag + mag.roll(64, -1)
        got = out[at:at + n].cpu().double().view(n, heads, 128)
        assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -14 * mag + 1e-6).all(), (b, (got - ref).abs().max())
        at += n


@pytest.mark.parametrize("heads,rot,factor,values,gains", [(32, 64, 4.0, True, True), (32, 0, 1.0, False, True), (16, 128, 1.0, True, True), (8, 128, 2.0, False, False), (8, 8, 0.0, True, True),
                                                           (16, 72, 3.0, False, True), (2, 64, 1.0, True, False)])
def test_heads_finish_planes(lib, heads, rot, factor, values, gains):
    """Against 64 bits: cosines and sines are rounded once (2^-24 of 1), a query is fp32 sums of a few roundings held in sixteen bits (value + remainder, 2^-17), keys and values are one
    rounding to bf16."""
    g = torch.Generator().manual_seed(heads + rot)
    T, kv = 131, heads // 2
    width = (heads + 2 * kv) * 128
    proj = torch.randn(T, width + 8, generator=g) * torch.exp(torch.randn(T, 1, generator=g))
    qg, kg = 1.0 + 0.2 * torch.randn(2, 128, generator=g)
    pos = torch.randint(0, 5000, (T,), generator=g, dtype=torch.int32)
    pos[:3] = torch.tensor([0, 1, 4999], dtype=torch.int32)
    slots = torch.randperm(T + 5, generator=g)[:T].to(torch.int32)
    slots[::6] = -1
    dev = [t.cuda() for t in (proj, qg, kg, pos, slots)]
    planes = torch.full((kv * T * 512 + 8,), float("nan"), dtype=torch.bfloat16, device="cuda")
    turn = torch.full((T + 1, 128), float("nan"), device="cuda")
    kc, vc = (torch.full((T + 5, kv * 128), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    base, eps = 3000.0, 1e-5
    chk(lib, lib.b2k_heads_finish_planes(ptr(dev[0]), width + 8, heads, rot, base, factor, int(values), eps, ptr(dev[1]) if gains else None, ptr(dev[2]) if gains else None, ptr(dev[3]),
                                         ptr(dev[4]), ptr(planes), ptr(turn) if values else None, ptr(kc), ptr(vc), T, cuda_stream_ptr()))
    torch.cuda.synchronize()

    def turned(x, dims, f):   # [T][heads][128]; pairs (m, m + dims / 2)
        m = torch.arange(dims // 2, dtype=torch.float64)
        ang = pos.double()[:, None] * base ** (-2.0 * m / dims) * f
        c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
        a, b = x[..., :dims // 2], x[..., dims // 2:dims]
        return torch.cat([a * c - b * s, b * c + a * s, x[..., dims:]], -1), torch.cat([torch.cos(ang), torch.sin(ang)], 1)

    x = proj[:, :width].double().view(T, -1, 128)
    q, k, v = x[:, :heads], x[:, heads:heads + kv], x[:, heads + kv:]
    norm = lambda y, w: y / torch.sqrt((y * y).mean(-1, keepdim=True) + eps) * w.double() if gains else y
    q, k = norm(q, qg), norm(k, kg)
    inv = 1.0 / factor if factor > 0 else 1.0
    if rot:
        q, k = turned(q, rot, inv)[0], turned(k, rot, inv)[0]
    near = lambda got, ref, bits: ((got - ref).abs() <= 2.0 ** -bits * ref.abs() + 2.0 ** -21 * ref.abs().amax(-1, keepdim=True)).all()
    assert torch.isnan(planes[-8:]).all()
    hi, lo = planes[:-8].view(kv, T, 2, 2, 128).cpu().double().unbind(3)
    assert near((hi + lo).permute(1, 0, 2, 3).reshape(T, heads, 128), q, 16) and (hi.permute(1, 0, 2, 3).reshape(T, heads, 128) - q).abs().max() > 0
    if values:
        v, cs = turned(v, 128, 1.0)
        assert (turn[:T].cpu().double() - cs).abs().max() <= 2.0 ** -23
    assert torch.isnan(turn[T if values else 0:]).all()
    seen = slots >= 0
    rows = slots[seen].long()
    for cache, ref in ((kc.cpu(), k), (vc.cpu(), v)):
        assert near(cache[rows].double().view(-1, kv, 128), ref[seen], 8)
        rest = torch.ones(T + 5, dtype=torch.bool)
        rest[rows] = False
        assert (cache[rest] == 7.0).all()


@pytest.mark.parametrize("heads", [32, 16, 8])
@pytest.mark.parametrize("before,n", [(0, 64), (0, 130), (37, 64), (101, 50), (64, 16)])
def test_heads_premix_reach_of_a_value(lib, heads, before, n):
    """A value that is not finite reaches the rows that see it and, of those that do not, only the ones in front of it among the same sixteen queries of a tile (0 times it is a NaN):
    the other rows have the bits that they have without it."""
    g = torch.Generator().manual_seed(heads + n)
    kv, S, bs = heads // 2, before + n, 16
    width = (S + bs - 1) // bs
    bt = torch.randperm(width + 1, generator=g)[:width].view(1, -1).to(torch.int32).cuda()
    planes = torch.randn(kv, n, 2, 2, 128, generator=g).to(torch.bfloat16)
    planes[:, :, :, 1] *= 2.0 ** -9
    planes = planes.cuda()
    kc, vc = (torch.randn((width + 1) * bs, kv, 128, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    talk = torch.eye(heads) + 0.2 * torch.randn(heads, heads, generator=g)
    host = torch.tensor([(i, before + i, min(64, n - i), 0) for i in range(0, n, 64)], dtype=torch.int32)
    tiles = host.cuda()
    room = len(host) * 64 * heads * 128 * ((S - 1) // 128 + 1)
    scratch = torch.empty(room, device="cuda")

    def call():
        out = torch.zeros(n, heads * 128, dtype=torch.bfloat16, device="cuda")
        chk(lib, lib.b2k_heads_premix(ptr(planes), ptr(kc), ptr(vc), (width + 1) * bs, heads, 128 ** -0.5, 0.0, ptr(talk), None, ptr(bt), width, bs, ptr(tiles), ptr(host), len(host), ptr(out),
                                      n, ptr(scratch), room, cuda_stream_ptr()))
        torch.cuda.synchronize()
        return out.cpu()

    clean = call()
    assert torch.isfinite(clean.float()).all()
    for i in sorted({0, 1, 15, 16, 33, n // 2, n - 2, n - 1} & set(range(n))):   # the token that is not finite
        p = before + i
        row = int(bt[0, p // bs]) * bs + p % bs
        kept = vc[row].clone()
        vc[row] = float("inf") if i % 2 else float("nan")
        got = call()
        vc[row] = kept
        free = i // 64 * 64 + i % 64 // 16 * 16   # rows in front of the sixteen that hold it
        assert torch.equal(got[:free], clean[:free]), (i, free)
        assert not torch.isfinite(got[i:].float()).any()


@pytest.mark.parametrize("heads,kv,dim,vdim,window,keep,bs", [(16, 8, 128, 128, 70, 9, 16), (16, 16, 64, 64, 0, 0, 32), (5, 1, 128, 64, 33, 0, 48), (8, 4, 64, 128, 16, 40, 16),
                                                              (1, 1, 128, 128, 1, 5, 16), (12, 4, 128, 128, 100, 16, 64)])
def test_heads_postmix(lib, heads, kv, dim, vdim, window, keep, bs):
    """Portions around the tiles of sixteen, some behind earlier tokens, windows and kept tokens around them, fewer heads than the mix's sixteen.  Against 64 bits over
    the same bf16 queries, keys and values: the weights carry sixteen bits into the products, so what is left is fp32 sums and the bf16 result (2^-9 of it).  A weight and
    a mixed one are off by 2^-17 of themselves, a score of a few units by as much: 2^-14 of the sum of absolute values holds them."""
    g = torch.Generator().manual_seed(heads * 100 + window)
    portions = [(0, 1), (0, 17), (100, 64), (3, 33), (200, 130), (0, 256)]            # (earlier tokens, tokens)
    T, width = sum(n for _, n in portions), max((p + n + bs - 1) // bs for p, n in portions)
    pages = len(portions) * width + 2
    bt = torch.randperm(pages, generator=g)[:len(portions) * width].view(-1, width).to(torch.int32)
    q = torch.randn(T, heads * dim, generator=g)
    kc, vc = (torch.randn(pages, bs, kv * d, generator=g).to(torch.bfloat16) for d in (dim, vdim))
    talk = torch.eye(heads) + 0.3 * torch.randn(heads, heads, generator=g)
    gate = torch.randn(T, heads + 3, generator=g)
    tiles, at = [], 0
    for b, (p, n) in enumerate(portions):
        tiles += [(at + i, p + i, min(64, n - i), b) for i in range(0, n, 64)]
        at += n
    scale, slope_exp = dim ** -0.5, 8.0
    dev = [t.cuda() for t in (q, kc, vc, bt, torch.tensor(tiles, dtype=torch.int32), talk, gate)]
    out = torch.full((T + 1, heads * vdim), float("nan"), dtype=torch.bfloat16, device="cuda")
    chk(lib, lib.b2k_heads_postmix(ptr(dev[0]), ptr(dev[1]), ptr(dev[2]), heads, kv, dim, vdim, scale, slope_exp, window, keep, ptr(dev[3]), width, bs, ptr(dev[4]), len(tiles),
                                   ptr(dev[5]), ptr(dev[6]), heads + 3, ptr(out), cuda_stream_ptr()))
    torch.cuda.synchronize()
    assert torch.isnan(out[T]).all()
    at, rep = 0, heads // kv
    slope = torch.tensor([2.0 ** (-slope_exp * (a + 1) / heads) for a in range(heads)], dtype=torch.float64)[:, None, None]
    for b, (p, n) in enumerate(portions):
        idx, S = bt[b].long(), p + n
        k = kc[idx].reshape(-1, kv, dim)[:S].double().repeat_interleave(rep, 1)
        v = vc[idx].reshape(-1, kv, vdim)[:S].double().repeat_interleave(rep, 1)
        qq = q[at:at + n].to(torch.bfloat16).double().view(n, heads, dim)
        i, j = torch.arange(p, S)[:, None], torch.arange(S)[None, :]
        seen = (j <= i) & ((i - j < window) | (j < keep)) if window else j <= i
        s = torch.einsum("ihd,jhd->hij", qq, k) * scale - slope * (i - j)
        pr = torch.softmax(s.masked_fill(~seen, float("-inf")), -1)
        w = torch.einsum("ab,bij->aij", talk.double(), pr)
        ref = torch.einsum("hij,jhd->ihd", w, v) * torch.sigmoid(gate[at:at + n, :heads].double())[:, :, None]
        got = out[at:at + n].cpu().double().view(n, heads, vdim)
        mag = torch.einsum("hij,jhd->ihd", torch.einsum("ab,bij->aij", talk.double().abs(), pr), v.abs())
        assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -14 * mag + 1e-6).all(), (b, (got - ref).abs().max())
        at += n
