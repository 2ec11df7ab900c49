"""Host-side choices of an engine step's kernels, on the CPU."""
import pytest
import torch


@pytest.mark.skipif(torch.cuda.is_available(), reason="a device answers")
def test_status_of_a_device_that_cannot_be_asked():
    """The worst status instead of an exception: failure detection reads a number."""
    from onecat_vllm.ops import _C
    assert _C.read_status(False) == 0x80000000 and _C.read_status(True) == 0x80000000


@pytest.mark.parametrize("form,wide", [(dict(), True), (dict(fine=True), False), (dict(page=8), False), (dict(rope_pad=128), False), (dict(lora=256), False), (dict(scale=-1.0), False)])
def test_latent_attention_is_split_for_the_kernel_that_runs(form, wide, monkeypatch):
    """The tcgen05 kernel's plan (one CTA an SM, 128 rows each) only for calls that it takes: the others keep the splits of 16-row tiles, in eager
    calls and in captured graphs."""
    from types import SimpleNamespace
    from onecat_vllm.ops import cuda as K
    from onecat_vllm.worker.cuda_graphs import DecodeGraphs
    f = dict(dict(lora=512, rope_pad=64, page=16, fine=False, scale=0.07), **form)
    assert K.mla_decode_wide(**f) == wide
    H, R, ctx = 16, 32, 4096
    per_sm = max(1, min(4, (227 << 10) // ((16 + 2 * 64) * (f["lora"] + 64) * 2 + 6144)))
    want = K.choose_decode_splits(2 * R, ctx, 148, 1, start=6.0, tile=1.3) if wide else K.choose_decode_splits(R, ctx, 148, per_sm)
    assert K.plan_mla(H, f["lora"], [1] * R, [ctx], 148, K.mla_decode_wide(**f)) == (want, wide)
    monkeypatch.setattr(K, "_sms", lambda device: 148)
    graphs = SimpleNamespace(eligible=True, sizes=[R], max_q=1, own_plans=False, geom=("mla", H, f["lora"]), mla_wide=wide, r=SimpleNamespace(device=None))
    assert DecodeGraphs.plan(graphs, R, 1, ctx) == (R, 1, (1 << (want - 1).bit_length(), wide))


@pytest.mark.parametrize("H,R,ctx,wide", [(16, 74, 16, True), (16, 75, 64, False), (16, 148, 190, False), (16, 149, 64, False), (16, 149, 100, True), (16, 256, 64, False),
                                          (16, 400, 400, True), (8, 128, 256, False), (8, 200, 190, True), (8, 256, 1000, True), (17, 256, 64, True), (128, 400, 64, True)])
def test_latent_rows_of_one_narrow_tile_and_short_contexts(H, R, ctx, wide):
    """Requests of at most 16 rows run in tiles of 16 where tiles of 128 (two CTAs each) are more waves and the contexts short: measured on either side of the line."""
    from onecat_vllm.ops import cuda as K
    splits, chosen = K.plan_mla(H, 512, [1] * R, [ctx], 148, True)
    assert chosen == wide and K.plan_mla(H, 512, [1] * R, [ctx], 148, False)[1] is False
    if not wide:
        assert splits == 1


@pytest.mark.parametrize("R,ctx,Hkv,D,best,slower", [(8, 1152, 8, 128, 4, 8), (16, 2000, 8, 128, 2, 4), (64, 1152, 8, 128, 1, 4), (128, 1152, 8, 128, 1, 2), (32, 4096, 8, 128, 1, 8), (64, 2300, 8, 128, 2, 4),
                                                     (8, 32768, 8, 128, 16, 8), (32, 500, 4, 128, 1, 2), (256, 1152, 4, 256, 1, 2), (8, 32768, 4, 256, 8, 4), (1, 4000, 8, 128, 16, 4)])
def test_captured_decoding_over_an_fp8_cache_is_split_for_its_kernel(R, ctx, Hkv, D, best, slower, monkeypatch):
    """Graphs and eager steps take their costs from one place; ``slower``: a number of splits that was measured slower than the chosen one."""
    from types import SimpleNamespace
    from onecat_vllm.ops import cuda as K
    from onecat_vllm.worker.cuda_graphs import DecodeGraphs
    monkeypatch.setattr(K, "_sms", lambda device: 148)
    graphs = lambda fp8: SimpleNamespace(eligible=True, sizes=[R], max_q=1, own_plans=False, geom=(5 * Hkv, Hkv, D), kv_fp8=fp8, r=SimpleNamespace(device=None))
    assert DecodeGraphs.plan(graphs(True), R, 1, ctx) == (R, 1, best) != (R, 1, slower)
    want = K.choose_decode_splits(R * Hkv, ctx, 148)
    assert DecodeGraphs.plan(graphs(False), R, 1, ctx) == (R, 1, min(32, 1 << (want - 1).bit_length()))
    assert K.plan_attention([1] * R, [ctx] * R, 5 * Hkv, Hkv, D, 148, fp8=True)[2] == K.choose_decode_splits(R * Hkv, ctx, 148, **K.decode_cost(D, 5, True))
    assert len({K.attn_plan_key(5 * Hkv, Hkv, D, f) for f in (True, False)}) == 2


@pytest.mark.parametrize("kind,N,Kd,T,skinny", [
    (1, 2048, 1024, 16, True), (1, 5120, 5120, 16, True), (1, 34816, 5120, 8, True), (1, 34816, 5120, 9, False), (1, 8192, 28672, 8, True), (1, 5120, 17408, 1, False),
    (1, 4800, 8192, 8, True), (1, 2048, 1024, 17, False), (2, 4096, 4096, 16, True), (2, 16384, 1536, 16, True), (2, 5120, 5120, 1, False), (2, 5120, 4096, 2, False),
    (2, 4096, 5120, 16, True), (2, 1024, 8192, 1, False), (2, 2048, 8192, 16, True), (2, 1536, 7168, 8, True), (2, 1536, 7168, 9, False), (2, 2112, 7168, 16, True),
    (2, 1024, 5120, 16, True), (3, 5120, 5120, 8, True), (3, 5120, 5120, 9, False), (4, 6144, 5120, 16, False), (4, 16384, 1536, 16, True), (3, 34816, 5120, 1, False)])
def test_packed_products_of_a_few_tokens(kind, N, Kd, T, skinny):
    """Either side of each line of the rule, as measured."""
    from onecat_vllm.ops import _C
    assert (_C.gemm_route(T, N, Kd, kind, 0, False, 148)[0] == "skinny") == skinny
    assert _C.gemm_route(T, N, Kd, 0, 0, False, 148)[0] == "tiles"


@pytest.mark.parametrize("n,q,ctx,heads,pairs", [
    (1, 64, 0, 40, False), (1, 256, 0, 16, False), (1, 300, 0, 40, False), (1, 512, 0, 16, False), (1, 512, 0, 40, True), (1, 1024, 0, 8, True), (1, 128, 400, 4, True),
    (16, 256, 0, 4, False), (16, 512, 0, 4, True), (32, 128, 0, 40, False), (8, 128, 200, 40, False), (32, 128, 500, 40, True), (128, 40, 0, 8, True), (32, 128, 0, 4, False),
    (4, 200, 0, 40, True), (1, 8192, 0, 40, True), (1, 64, 4000, 40, True)])
def test_prompt_attention_takes_single_tiles_for_short_contexts(n, q, ctx, heads, pairs):
    """Either side of the lines of the rule, as measured; decoding requests beside the portions do not count, and unknown lengths (a graph) take pairs."""
    from onecat_vllm.ops import cuda as K
    tiles = n * -(-q // (256 if pairs else 128))
    assert K.prompt_tiles([q] * n, [q + ctx] * n, 6, heads, 148) == (pairs, tiles)
    assert K.prompt_tiles([1, 6] + [q] * n, [9000, 9000] + [q + ctx] * n, 6, heads, 148) == (pairs, tiles)
    assert K.prompt_tiles([q] * n, [0] * n, 6, heads, 148) == (True, n * -(-q // 256))
