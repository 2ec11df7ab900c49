"""Kernels of an engine step at the edges of their dispatch rules, against the CPU oracles."""
import pytest
import torch

from onecat_vllm.ops import ref

pytestmark = pytest.mark.gpu


def K():
    from onecat_vllm.ops import cuda
    return cuda


def _close(a, b, rtol, atol, what=""):
    a, b = a.float().cpu(), b.float().cpu()
    bad = ~((a - b).abs() <= atol + rtol * b.abs())   # NaN is a difference
    assert not bad.any(), f"{what}: {int(bad.sum())} of {bad.numel()} differ, largest by {float((a - b).abs().max())}"


@pytest.mark.parametrize("T,Hq,Hkv,D,rot,norm,fp8", [(1, 3, 1, 64, 64, False, False), (1300, 40, 8, 128, 128, True, False), (5, 7, 2, 256, 64, True, True),
                                                     (2100, 5, 1, 256, 32, False, False), (4099, 6, 3, 64, 48, True, True), (9, 2, 1, 128, 0, True, False)])
def test_rope_and_cache_in_wide_accesses(T, Hq, Hkv, D, rot, norm, fp8):
    """One and four heads per group, numbers of heads that four does not divide, rotary widths below the head, no slot for some tokens; one
    rounding to bf16 (2^-8) after the norm and one after the rotation."""
    g = torch.Generator().manual_seed(T)
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, generator=g).bfloat16()
    pos = torch.randint(0, 500, (T,), generator=g, dtype=torch.int32)
    cs = ref.build_cos_sin_cache(max(rot, 2), 512, 1e6, "cpu")[:, :rot]
    cache = torch.zeros(T // 16 + 2, 2, Hkv, 16, D).to(torch.float8_e4m3fn if fp8 else torch.bfloat16)
    slots = torch.randperm(cache.shape[0] * 16, generator=g)[:T].to(torch.int32)
    if T > 3:
        slots[3] = -1
    qn, kn = ((torch.randn(D, generator=g) * 0.2 + 1).bfloat16() for _ in range(2)) if norm else (None, None)
    dev = [t if t is None else t.cuda() for t in (qkv, pos, cs, cache, slots, qn, kn)]
    views = lambda x: (x[:, : Hq * D].view(T, Hq, D), x[:, Hq * D: (Hq + Hkv) * D].view(T, Hkv, D), x[:, (Hq + Hkv) * D:].view(T, Hkv, D))
    K().rope_and_cache(*views(dev[0]), dev[1], dev[2], dev[3], dev[4], rot, dev[5], dev[6], 1e-6, False)
    ref.rope_and_cache(*views(qkv), pos, cs, cache, slots, rot, qn, kn, 1e-6, False)
    _close(dev[0], qkv, 2 ** -7, 2 ** -6, "q and k")
    if fp8:   # a last bit of bf16 may cross a boundary between two codes
        a, b = dev[3].cpu().view(torch.uint8).int(), cache.view(torch.uint8).int()
        assert ((a - b).abs() <= 1).all() and (a != b).float().mean() < 0.01 and (a[:, 1] == b[:, 1]).all()
    else:
        _close(dev[3], cache, 2 ** -7, 2 ** -6, "cache")


@pytest.mark.parametrize("qlens,ctxs,H,rope,options", [([1, 1, 1], [0, 62, 63], 64, 64, False), ([1, 1], [16, 5000], 128, 64, True), ([1, 2, 5], [0, 127, 300], 64, 32, True),
                                                      ([3, 1, 0, 2], [77, 1, 9, 640], 24, 48, False), ([1] * 40, [130] * 40, 128, 64, False), ([1] * 80, [61, 63, 64, 5] * 20, 16, 64, True)])
def test_mla_decode_tiles_of_128_rows(qlens, ctxs, H, rope, options):
    """Contexts of one key to many tiles, tiles and pages that end with the context, rows that end inside a tile, several tokens a request, key
    parts below 64, and requests of 16 rows that stay with the 16-row kernel; the slots past a context hold NaN. Sinks and gates where asked. Weights and queries are bf16: 2^-8 each."""
    from onecat_vllm.worker.attn_metadata import AttentionMetadata
    lora, bs, R, T = 512, 16, len(qlens), sum(qlens)
    g = torch.Generator().manual_seed(T + H)
    seq = [c + q for q, c in zip(qlens, ctxs)]
    per = [-(-s // bs) for s in seq]
    bt = torch.zeros(R, max(per) + 1, dtype=torch.int32)
    order = torch.randperm(sum(per), generator=g).to(torch.int32) + 1
    cache = (torch.randn(sum(per) + 1, bs, lora + rope, generator=g) * 0.3).bfloat16()
    at = 0
    for r, n in enumerate(per):
        bt[r, :n] = order[at:at + n]
        at += n
        if seq[r] % bs:
            cache[bt[r, n - 1].long(), seq[r] % bs:] = float("nan")
    q_abs, q_pe = (torch.randn(T, H, lora, generator=g) * 0.5).bfloat16(), (torch.randn(T, H, rope, generator=g) * 0.5).bfloat16()
    sinks, gate = (torch.randn(H, generator=g), torch.randn(T, H, generator=g).bfloat16()) if options else (None, None)
    qsl = torch.tensor([0, *torch.tensor(qlens).cumsum(0).tolist()], dtype=torch.int32)
    sl = torch.tensor(seq, dtype=torch.int32)
    md = AttentionMetadata(R, T, qsl.cuda(), sl.cuda(), bt.cuda(), None, None, max(qlens), max(seq), query_lens_cpu=list(qlens), seq_lens_cpu=seq)
    dev = lambda t: None if t is None else t.cuda()
    want = ref.mla_decode(q_abs, q_pe, torch.nan_to_num(cache), bt, qsl, sl, 192 ** -0.5, lora, sinks, gate)
    for _ in range(2):
        out = K().mla_decode(q_abs.cuda(), q_pe.cuda(), cache.cuda(), md, 192 ** -0.5, lora, sinks=dev(sinks), gate=dev(gate))
        assert K().check_status() == 0
        _close(out, want, 2e-2, 5e-3)


def _mla_case(qlens, seq, H, g, q_pe, k_pe, lora=512, rope=64, bs=16):
    """(queries, rotated queries, cache in shuffled pages, block table, query starts, lengths, metadata): random latents beside given rotated parts."""
    from onecat_vllm.worker.attn_metadata import AttentionMetadata
    R, T = len(qlens), sum(qlens)
    per = [-(-s // bs) for s in seq]
    order = torch.randperm(sum(per), generator=g).to(torch.int32) + 1
    bt, at = torch.zeros(R, max(per), dtype=torch.int32), 0
    cache = (torch.randn(sum(per) + 1, bs, lora + rope, generator=g) * 0.3).bfloat16()
    for r, n in enumerate(per):
        bt[r, :n] = order[at:at + n]
        at += n
        rows = torch.zeros(n * bs, rope)
        rows[: seq[r]] = k_pe[r]
        cache[bt[r, :n].long(), :, lora:] = rows.view(n, bs, rope).bfloat16()
    q = (torch.randn(T, H, lora, generator=g) * 0.5).bfloat16()
    qsl, sl = torch.tensor([0, *torch.tensor(qlens).cumsum(0).tolist()], dtype=torch.int32), torch.tensor(seq, dtype=torch.int32)
    md = AttentionMetadata(R, T, qsl.cuda(), sl.cuda(), bt.cuda(), None, None, max(qlens), max(seq), query_lens_cpu=list(qlens), seq_lens_cpu=seq)
    return q, q_pe.bfloat16(), cache, bt, qsl, sl, md


def _in_splits(md, H, splits):
    md.static_ws, md.attn_plan = True, (("mla", H, 512), (md.max_query_len, 0, (splits, True)))
    return md


@pytest.mark.parametrize("splits", [2, 4])
def test_mla_decode_halves_of_the_columns_at_the_edge_of_a_new_reference(splits):
    """The CTAs of the two column halves sum a score in different orders. Where a row's maximum grows by 2^8 to within that difference, one of them
    may move its reference and the other not: each half is merged by its own. Parts of the scores that cancel widen the difference; the scale
    puts one head after another on the edge, between the first and the second tile of a split."""
    H, S, T = 128, 512, 1
    g = torch.Generator().manual_seed(splits)
    k_pe, q_pe = torch.zeros(1, S, 64), torch.zeros(T, H, 64)
    q_pe[..., 0] = 4
    k_pe[0, S // splits - 30, 0] = k_pe[0, -5, 0] = 10   # raw scores rise by 40, in the last tile of the first and of the last split
    q, q_pe, cache, bt, qsl, sl, md = _mla_case([1], [S], H, g, q_pe, k_pe)
    q[..., :32], q[..., 256:288], cache[..., :32], cache[..., 256:288] = 16, -16, 8, 8   # 4096 - 4096
    _in_splits(md, H, splits)
    dev = [t.cuda() for t in (q, q_pe, cache)]
    kv = cache[bt[0].long()].reshape(S, 576).double()
    raw = torch.cat([q, q_pe], -1)[0].double() @ kv.t()
    tiles = raw[:, : S // splits].view(H, -1, 64).amax(-1)
    growth = tiles[:, -1] - tiles[:, :-1].amax(-1)
    for h in range(0, H, 8):
        for off in (-1e-4, -3e-5, 0.0, 3e-5, 1e-4):
            scale = 8 / 1.4426950408889634 / float(growth[h]) * (1 + off)
            want = torch.softmax(raw * scale, -1) @ kv[:, :512]
            out = K().mla_decode(*dev, md, scale, 512)
            _close(out[0], want, 2e-2, 5e-2, f"head {h}, {off}")   # weights in bf16 (2^-8); results of up to 8
    assert K().check_status() == 0


@pytest.mark.parametrize("qlens,ctxs,H,step", [([1, 1], [700, 128], 128, 6.0), ([1, 3, 2], [320, 500, 63], 64, 25.0), ([5], [1000], 16, 60.0), ([1] * 3, [640, 65, 1], 128, -9.0)])
@pytest.mark.parametrize("splits", [1, 2, 3])
def test_mla_decode_rescales_its_results(qlens, ctxs, H, step, splits):
    """Maxima that grow (or fall) from tile to tile by 2^2 to 2^40, differently in every head: the results so far are rescaled in some rows of a warp
    and tiles, in one split and several, with several tokens a request. Weights and queries are bf16: 2^-8 each."""
    seq = [c + q for q, c in zip(qlens, ctxs)]
    g = torch.Generator().manual_seed(sum(seq) + splits)
    k_pe = [torch.zeros(s, 64) for s in seq]
    for k in k_pe:
        k[:, 0] = (torch.arange(len(k)) // 64) * step
    q_pe = torch.zeros(sum(qlens), H, 64)
    q_pe[..., 0] = torch.rand(sum(qlens), H, generator=g) * 8
    q, q_pe, cache, bt, qsl, sl, md = _mla_case(qlens, seq, H, g, q_pe, k_pe)
    out = K().mla_decode(q.cuda(), q_pe.cuda(), cache.cuda(), _in_splits(md, H, splits), 192 ** -0.5, 512)
    assert K().check_status() == 0
    _close(out, ref.mla_decode(q, q_pe, cache, bt, qsl, sl, 192 ** -0.5, 512), 2e-2, 1e-2)


def _packed(kind, N, Kd, g):
    """(packed tiles, scale table, padded rows, k tiles per group, weights in fp64) of random weights."""
    n = 64 if Kd % 128 else 128   # group
    if kind == 1:
        q, z = torch.randint(0, 16, (N, Kd), generator=g, dtype=torch.uint8, device=g.device), torch.randint(0, 16, (N, Kd // n), generator=g, dtype=torch.uint8, device=g.device)
        s = torch.rand(N, Kd // n, generator=g, device=g.device) * 0.01 + 0.001
        w = ((q.float() - z.float().repeat_interleave(n, 1)) * s.bfloat16().float().repeat_interleave(n, 1)).bfloat16().double()
        return (*K().pack_w4(q.cuda(), z.cuda(), s.cuda(), n), n // 64, w)
    if kind == 2:
        c = torch.randn(N, Kd, generator=g, device=g.device).to(torch.float8_e4m3fn)
        s = torch.rand(N, Kd // n, generator=g, device=g.device) * 0.02 + 0.001
        return (*K().pack_fp8(c.view(torch.uint8).cuda(), s.cuda(), n), n // 64, (c.float() * s.bfloat16().float().repeat_interleave(n, 1)).bfloat16().double())
    c = torch.randint(0, 256, (N, Kd // 2), generator=g, dtype=torch.uint8, device=g.device)
    values = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, 0, -.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64, device=g.device)[torch.stack([c & 15, c >> 4], -1).long().flatten(1)]
    if kind == 3:
        e = torch.randint(119, 123, (N, Kd // 32), generator=g, dtype=torch.uint8, device=g.device)
        return (*K().pack_mxfp4(c.cuda(), e.cuda()), 1, values * torch.exp2(e.double() - 127).repeat_interleave(32, 1))
    s = (torch.rand(N, Kd // 16, generator=g, device=g.device) * 4 + 0.5).to(torch.float8_e4m3fn)
    w = values * s.double().repeat_interleave(16, 1) * 0.25
    return (*K().pack_nvfp4(c.cuda(), s.cuda(), torch.tensor(0.25).cuda()), 1, w)


@pytest.mark.parametrize("kind", [1, 2, 3, 4])
@pytest.mark.parametrize("T,N,Kd,gated", [(1, 128, 128, False), (8, 160, 1152, True), (9, 96, 4224, False), (16, 5120, 704, True), (3, 224, 64, True), (13, 64, 8320, False), (13, 2080, 8320, False)])
def test_gemm_of_a_few_tokens(kind, T, N, Kd, gated):
    """One and two blocks of eight tokens, full and ragged, rows that end inside a tile, k ranges of an odd number of tiles, of fewer than the warps
    and of many, gated and plain (with a bias) epilogues, a strided activation. Weights are rounded to bf16 where they are widened; fp32 sums, one rounding at the end."""
    g = torch.Generator().manual_seed(kind * 100 + T)
    tiles, sz, npad, gk, w = _packed(kind, N, Kd, g)
    x = (torch.randn(T, Kd + 64, generator=g)).bfloat16()[:, :Kd]
    y = x.double() @ w.t()
    bias = None
    if gated:
        pair = y.view(T, -1, 2, 16)
        want = (torch.nn.functional.silu(pair[:, :, 0]) * pair[:, :, 1]).reshape(T, -1)
    else:
        bias = torch.randn(N, generator=g).bfloat16()
        want = y + bias.double()
    out = torch.full((T + 1, want.shape[1] + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    K()._gemm(x.cuda(), None, tiles, sz, out[:T, : want.shape[1]], None if bias is None else bias.cuda(), N, N, want.shape[1], npad, 1 if gated else 0, gk, wkind=kind)
    torch.cuda.synchronize()
    assert (out[T:] == 7).all() and (out[:, want.shape[1]:] == 7).all()
    _close(out[:T, : want.shape[1]], want, 2 ** -6, float(want.abs().mean()) * 2 ** -6, f"kind {kind}")


@pytest.mark.parametrize("D,Hq,Hkv,qlens,ctxs,options", [
    (128, 40, 8, [1, 1, 1], [0, 31, 5000], {}), (128, 8, 8, [1] * 5, [127, 128, 129, 15, 700], dict(softcap=20.0)), (128, 16, 1, [1, 1], [3000, 64], dict(sinks=True)),
    (128, 32, 4, [4, 1, 2], [95, 4000, 17], {}), (128, 6, 2, [3, 3], [600, 40], dict(window=100)), (256, 24, 4, [1, 2, 1], [0, 1000, 63], dict(window=70, softcap=30.0)),
    (256, 16, 2, [1, 1], [8000, 33], dict(sinks=True)), (256, 16, 4, [4, 3], [2000, 1], {})])
def test_decode_over_an_fp8_cache(D, Hq, Hkv, qlens, ctxs, options):
    """One and two blocks of 16 rows, turns that end with the context, in one and several splits, windows, caps and sinks; the bytes past a context
    are those of the largest codes. Queries and weights are bf16 (2^-8 each)."""
    from onecat_vllm.worker.attn_metadata import AttentionMetadata
    bs, R, T = 16, len(qlens), sum(qlens)
    g = torch.Generator().manual_seed(D + Hq)
    seq = [c + q for q, c in zip(qlens, ctxs)]
    per = [-(-s // bs) for s in seq]
    bt, at = torch.zeros(R, max(per) + 1, dtype=torch.int32), 1
    cache = torch.randn(sum(per) + 1, 2, Hkv, bs, D, generator=g).to(torch.float8_e4m3fn)
    for r, n in enumerate(per):
        bt[r, :n] = torch.arange(at, at + n, dtype=torch.int32).flip(0)
        at += n
        if seq[r] % bs:
            cache.view(torch.uint8)[bt[r, n - 1].long(), :, :, seq[r] % bs:] = 0x7e
    q = torch.randn(T, Hq, D, generator=g).bfloat16()
    window, softcap = options.get("window", 0), options.get("softcap", 0.0)
    sinks = torch.randn(Hq, generator=g) if options.get("sinks") else None
    qsl, sl = torch.tensor([0, *torch.tensor(qlens).cumsum(0).tolist()], dtype=torch.int32), torch.tensor(seq, dtype=torch.int32)
    want = ref.paged_attention(q, cache, bt, qsl, sl, D ** -0.5, window=window, softcap=softcap, sinks=sinks)
    for splits in (1, 3, None):
        md = AttentionMetadata(R, T, qsl.cuda(), sl.cuda(), bt.cuda(), None, None, max(qlens), max(seq), query_lens_cpu=list(qlens), seq_lens_cpu=seq)
        if splits:
            md.attn_plan = (K().attn_plan_key(Hq, Hkv, D, True), (max(qlens), 0, splits))
        out = K().paged_attention(q.cuda(), cache.cuda(), md, D ** -0.5, window=window, softcap=softcap, sinks=None if sinks is None else sinks.cuda())
        assert K().check_status() == 0
        _close(out, want, 2e-2, 1e-2, f"{splits} splits")


@pytest.mark.parametrize("qlens,ctxs,Hq,Hkv,scale", [([256, 257, 1, 128], [0, 1, 500, 128], 8, 2, 1.0), ([129, 640, 17], [127, 300, 2000], 4, 4, 1.0), ([700], [0], 2, 1, 30.0),
                                                        ([128, 17, 1, 100], [0, 239, 500, 256], 16, 2, 1.0), ([129, 400], [300, 0], 8, 2, 1.0), ([700], [60], 2, 1, 30.0)])
@pytest.mark.parametrize("pairs", [None, True, False])
def test_prompt_attention_in_pairs_of_query_tiles(qlens, ctxs, Hq, Hkv, scale, pairs, monkeypatch):
    """Portions that end inside the first or the second tile of a pair, one that fills both, tiles of unequal numbers of key tiles, a decoding request
    beside them, and scores that grow by far more than 2^8 along a row (the accumulator is rescaled). As planned, and each form
    (pairs, single tiles) for all of them. Weights are bf16 (2^-8)."""
    if pairs is not None:
        monkeypatch.setattr(K(), "prompt_tiles", lambda ql, sl, short, heads, sms: (pairs, sum(-(-n // (256 if pairs else 128)) for n in ql if n > short)))
    from onecat_vllm.worker.attn_metadata import AttentionMetadata
    D, bs, R, T = 128, 16, len(qlens), sum(qlens)
    g = torch.Generator().manual_seed(T)
    seq = [c + q for q, c in zip(qlens, ctxs)]
    per = [-(-s // bs) for s in seq]
    bt, at = torch.zeros(R, max(per), dtype=torch.int32), 1
    for r, n in enumerate(per):
        bt[r, :n] = torch.arange(at, at + n, dtype=torch.int32).flip(0)
        at += n
    cache = torch.randn(at, 2, Hkv, bs, D, generator=g)
    if scale != 1.0:   # keys grow with their position
        order = bt[0].long()
        cache[order, 0] *= torch.linspace(0.1, scale, len(order)).view(-1, 1, 1, 1)
    cache, q = cache.bfloat16(), torch.randn(T, Hq, D, generator=g).bfloat16()
    qsl, sl = torch.tensor([0, *torch.tensor(qlens).cumsum(0).tolist()], dtype=torch.int32), torch.tensor(seq, dtype=torch.int32)
    md = AttentionMetadata(R, T, qsl.cuda(), sl.cuda(), bt.cuda(), None, None, max(qlens), max(seq), query_lens_cpu=list(qlens), seq_lens_cpu=seq)
    lse = torch.zeros(T, Hq, device="cuda")
    out = K().paged_attention(q.cuda(), cache.cuda(), md, D ** -0.5, lse=lse)
    assert K().check_status() == 0
    _close(out, ref.paged_attention(q, cache, bt, qsl, sl, D ** -0.5), 2e-2, 1e-2)
    s = torch.einsum("hd,kd->hk", q[qsl[1] - 1, : Hq // Hkv].float(), cache[bt[0, :per[0]].long(), 0, 0].reshape(-1, D)[: seq[0]].float()) * D ** -0.5
    _close(lse[qsl[1] - 1, : Hq // Hkv], torch.logsumexp(s, -1), 1e-3, 1e-2, "lse")


@pytest.mark.parametrize("scale", [0.0, -0.1])
def test_prompt_attention_with_a_scale_of_zero_or_less(scale):
    """The tcgen05 kernel takes a row's maximum and masks keys ahead of the scale: such a scale stays with the kernel that scales first."""
    from onecat_vllm.worker.attn_metadata import AttentionMetadata
    Hq, Hkv, D, n = 4, 2, 128, 300
    g = torch.Generator().manual_seed(1)
    cache, q = torch.randn(20, 2, Hkv, 16, D, generator=g).bfloat16(), torch.randn(n, Hq, D, generator=g).bfloat16()
    bt, qsl, sl = torch.arange(1, 20, dtype=torch.int32).view(1, -1), torch.tensor([0, n], dtype=torch.int32), torch.tensor([n], dtype=torch.int32)
    md = AttentionMetadata(1, n, qsl.cuda(), sl.cuda(), bt.cuda(), None, None, n, n, query_lens_cpu=[n], seq_lens_cpu=[n])
    out = K().paged_attention(q.cuda(), cache.cuda(), md, scale)
    assert K().check_status() == 0
    _close(out, ref.paged_attention(q, cache, bt, qsl, sl, scale), 2e-2, 1e-2)


@pytest.mark.parametrize("T,N,Kd,epi,bias,f32", [(256, 9472, 64, 0, False, False), (300, 5120, 640, 0, True, False), (2500, 1000, 1088, 0, True, True), (129, 9600, 128, 1, False, False),
                                                 (1030, 2112, 448, 3, False, False), (515, 3336, 192, 2, True, False), (9000, 520, 256, 0, False, False),
                                                     (2500, 1096, 8256, 0, True, True), (700, 3300, 8192, 0, False, False)])
def test_gemm_over_pairs_of_sms(T, N, Kd, epi, bias, f32):
    """Ragged tokens and features, rings shorter and longer than the k tiles, several tiles per pair of SMs, a last group of fewer token tiles, long k (weights are
    brought to L2 ahead; halves of tiles past the rows); plain, gated
    and activated epilogues, fp32 and bf16 results. One rounding of an fp32 sum."""
    from onecat_vllm.ops import _C
    assert _C.gemm_route(T, N, Kd, 0, epi, f32, K()._sms(torch.device("cuda"))) == ("pair", 0)
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, Kd + 64, device="cuda", generator=g).bfloat16()[:, :Kd]
    w = (torch.randn(N, Kd, device="cuda", generator=g) * Kd ** -0.5).bfloat16()
    b = torch.randn(N, device="cuda", generator=g).bfloat16() if bias else None
    y = x.double() @ w.double().t()
    if epi in (1, 3):
        pair = y.view(T, -1, 2, 16)
        act = torch.nn.functional.silu(pair[:, :, 0]) if epi == 1 else torch.nn.functional.gelu(pair[:, :, 0], approximate="tanh")
        want = (act * pair[:, :, 1]).reshape(T, -1)
    else:
        want = y if b is None else y + b.double()
        want = torch.nn.functional.gelu(want, approximate="tanh") if epi == 2 else want
    n = want.shape[1]
    out = torch.full((T + 1, n + 8), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    before = K().check_status()
    K()._gemm(x, w, None, None, out[:T, :n], b, N, N, n, 0, epi, 1)
    torch.cuda.synchronize()
    assert before == 0 and K().check_status() == 0
    assert (out[T:] == 7).all() and (out[:, n:] == 7).all()
    _close(out[:T, :n], want, 1e-4 if f32 else 2 ** -7, 1e-4 if f32 else 2 ** -9)


@pytest.mark.parametrize("kind", [1, 2, 3, 4])
@pytest.mark.parametrize("T,N,Kd,gated,slabs", [(1100, 5120, 192, True, 1), (2048, 1312, 704, False, 1), (1024, 13096, 8256, False, 2), (2048, 24096, 4224, True, 2), (1024, 9984, 4224, False, 0)])
def test_packed_gemm_of_many_tokens(kind, T, N, Kd, gated, slabs):
    """One slab of widened weights and two, whose second ends with the rows (bias, plain and gated columns, the slab reused while the product before
    reads it), rows that end inside a tile, odd numbers of k tiles; none where tiles are the faster form. Weights are rounded to bf16 where they
    are widened; fp32 sums, one rounding at the end."""
    from onecat_vllm.ops import _C
    assert _C.gemm_route(T, N, Kd, kind, 1 if gated else 0, False, K()._sms(torch.device("cuda"))) == (("widen", slabs) if slabs else ("tiles", 0))
    g = torch.Generator(device="cuda").manual_seed(kind + T)
    tiles, sz, npad, gk, w = _packed(kind, N, Kd, g)
    x = torch.randn(T, Kd, generator=g, device="cuda").bfloat16()
    y = x.double() @ w.t()
    bias = None
    if gated:
        pair = y.view(T, -1, 2, 16)
        want = (torch.nn.functional.silu(pair[:, :, 0]) * pair[:, :, 1]).reshape(T, -1)
    else:
        bias = torch.randn(N, generator=g, device="cuda").bfloat16()
        want = y + bias.double()
    out = torch.full((T + 1, want.shape[1] + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    K()._gemm(x, None, tiles, sz, out[:T, : want.shape[1]], bias, N, N, want.shape[1], npad, 1 if gated else 0, gk, wkind=kind)
    torch.cuda.synchronize()
    assert K().check_status() == 0 and (out[T:] == 7).all() and (out[:, want.shape[1]:] == 7).all()
    _close(out[:T, : want.shape[1]], want, 2 ** -6, float(want.abs().mean()) * 2 ** -6, f"kind {kind}")


@pytest.mark.parametrize("qlens,fresh", [([1, 2, 3, 500, 5, 1], [0, 0, 1, 1, 0, 1]), ([515], [1]), ([300, 4, 1, 210], [0, 1, 0, 0])])
def test_causal_convolution_of_eight_tokens_a_thread(qlens, fresh):
    """Sequences that begin and end inside a tile of eight tokens, shorter than the taps, with and without a state, through the recurrent layer's step (its
    other kernels have tests of their own). Tolerances as there: bf16 products of normalised keys along the sequence."""
    from onecat_vllm.worker.attn_metadata import AttentionMetadata
    Hk, Hv, D, R, T = 1, 1, 128, len(qlens), sum(qlens)
    C = (2 * Hk + Hv) * D
    g = torch.Generator().manual_seed(T)
    x, w = (torch.randn(T, C, generator=g) * 0.5).bfloat16(), (torch.randn(C, 4, generator=g) * 0.3).bfloat16()
    ba, A_log, dt = torch.randn(T, 2 * Hv, generator=g).bfloat16(), torch.rand(Hv, generator=g) - 1.0, torch.rand(Hv, generator=g)
    conv, state = (torch.randn(R + 1, C, 3, generator=g) * 0.5).bfloat16(), torch.randn(R + 1, Hv, D, D, generator=g) * 0.1
    qsl = torch.tensor([0, *torch.tensor(qlens).cumsum(0).tolist()], dtype=torch.int32)
    slots, has = torch.randperm(R + 1, generator=g)[:R].to(torch.int32), 1 - torch.tensor(fresh, dtype=torch.int32)
    md = AttentionMetadata(R, T, qsl.cuda(), None, None, None, None, max(qlens), 0, state_slots=slots.cuda(), has_initial_state=has.cuda(), query_lens_cpu=list(qlens))
    dconv, dstate, dba = conv.cuda(), state.cuda(), ba.cuda()
    out = K().gdn_forward(x.cuda(), dba[:, :Hv], dba[:, Hv:], w.cuda(), A_log.cuda(), dt.cuda(), dconv, dstate, md, Hk, Hv, D, D)
    m = ref.causal_conv1d(x, w, None, conv, qsl, slots, has)
    gate, beta = ref.gdn_gating(ba[:, Hv:], ba[:, :Hv], A_log, dt)
    want = ref.gated_delta_rule(m[:, :D].reshape(T, 1, D), m[:, D:2 * D].reshape(T, 1, D), m[:, 2 * D:].reshape(T, 1, D), gate, beta, state, qsl, slots, has)
    _close(out.view(T, Hv, D), want, 4e-2, 4e-2)
    assert torch.equal(dconv.cpu(), conv)


@pytest.mark.parametrize("T,heads,D", [(1, 1, 64), (7, 3, 128), (33, 5, 256), (130, 48, 128)])
def test_gated_norm_in_wide_accesses(T, heads, D):
    """Odd numbers of rows (a group takes two), slices of wider rows; one rounding of fp32 arithmetic."""
    g = torch.Generator().manual_seed(T)
    x, wide, w = torch.randn(T, heads * D, generator=g).bfloat16(), torch.randn(T, 2 * heads * D, generator=g).bfloat16(), (1 + 0.1 * torch.randn(D, generator=g)).bfloat16()
    z = wide[:, heads * D:]
    y = K().rms_norm_gated(x.cuda(), wide.cuda()[:, heads * D:], w.cuda(), 1e-6, heads)
    _close(y.view(T, heads, D), ref.rms_norm_gated(x.view(T, heads, D), z.reshape(T, heads, D), w, 1e-6), 2 ** -6, 2 ** -8)


@pytest.mark.parametrize("kind,T,N,Kd,splits", [(1, 4, 1792, 1024, 0), (2, 12, 1792, 1024, 0), (1, 32, 1024, 1152, 1), (2, 200, 1024, 1024, 1), (0, 600, 20480, 1152, 0)])
def test_a_weight_row_sums_alike_in_a_layer_and_in_a_slice_of_it(kind, T, N, Kd, splits):
    """The order of a sum over k depends on no feature tile's number: the second half of the rows, as a layer of its own (a rank's slice), gives the same bits."""
    g = torch.Generator().manual_seed(N)
    x = torch.randn(T, Kd, generator=g).bfloat16().cuda()
    if kind == 0:
        w = (torch.randn(N, Kd, generator=g) * Kd ** -0.5).bfloat16().cuda()
        whole, half = (K().gemm_bf16(x, t, out_dtype=torch.float32) for t in (w, w[N // 2:]))
    else:
        c = torch.randint(0, 16, (N, Kd), generator=g, dtype=torch.uint8) if kind == 1 else torch.randn(N, Kd, generator=g).to(torch.float8_e4m3fn).view(torch.uint8)
        z, s = torch.randint(0, 16, (N, Kd // 128), generator=g, dtype=torch.uint8), torch.rand(N, Kd // 128, generator=g) * 0.02 + 0.001

        def product(lo):
            t = [v[lo:].contiguous().cuda() for v in (c, z, s)]
            tiles, sz, npad = K().pack_w4(*t, 128)[:3] if kind == 1 else K().pack_fp8(t[0], t[2], 128)[:3]
            out = torch.empty(T, N - lo, dtype=torch.bfloat16, device="cuda")
            return K()._gemm(x, None, tiles, sz, out, None, N - lo, N - lo, N - lo, npad, 0, 2, force_splits=splits, wkind=kind)
        whole, half = product(0), product(N // 2)
    assert torch.equal(whole[:, N // 2:], half)


@pytest.mark.parametrize("T,dtype,epi", [(40, torch.float32, 0), (1100, torch.float32, 0), (40, torch.bfloat16, 2), (1100, torch.bfloat16, 3)])
def test_packed_gemm_refuses_a_second_form_of_its_weight(T, dtype, epi):
    """fp32 results and GELU epilogues are those of bf16 weights; a bf16 weight beside the packed one does not open them."""
    N, Kd = 5120, 192
    tiles, sz, npad = K().pack_fp8(torch.zeros(N, Kd, dtype=torch.uint8, device="cuda"), torch.ones(N, Kd // 64, device="cuda"), 64)
    x, w = torch.zeros(T, Kd, device="cuda").bfloat16(), torch.zeros(N, Kd, device="cuda").bfloat16()
    n = N // 2 if epi == 3 else N
    with pytest.raises(RuntimeError, match="one form of the weight"):
        K()._gemm(x, w, tiles, sz, torch.empty(T, n, dtype=dtype, device="cuda"), None, N, N, n, npad, epi, 1, wkind=2)
