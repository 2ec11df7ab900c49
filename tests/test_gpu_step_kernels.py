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
