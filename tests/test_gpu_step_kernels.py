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
    bad = (a - b).abs() > atol + rtol * b.abs()
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
                                                      ([3, 1, 0, 2], [77, 1, 9, 640], 24, 48, False), ([1] * 40, [130] * 40, 128, 64, False)])
def test_mla_decode_tiles_of_128_rows(qlens, ctxs, H, rope, options):
    """Contexts of one key to many tiles, tiles and pages that end with the context, rows that end inside a tile, several tokens a request, key
    parts below 64; the slots past a context hold NaN. Sinks and gates where asked. Weights and queries are bf16: 2^-8 each."""
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
