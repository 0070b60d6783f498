"""Prompts on the tensor-core path at the sizes where its tiling can go wrong, against the CPU oracle: several prompts per call
(more than one pair of launches takes, and shorter ones beside them that stay off it), lengths around the 64-token softmax step
and the 128-row tile, an odd number of q heads per kv head (a pair without its second head), more units of work than thread
blocks (q tiles staged ahead), rows that are not 16-byte aligned.  Bounds: those of assert_out_close for the output, bit equality
for the caches, 2 ulp for the roped rows."""
import numpy as np
import pytest
import torch

from oracle import attn_oracle as O

from gpu_util import (ROPE_MAX_ULP, assert_out_close, download_cache, make_desc, oracle_cfg, qkv_width, random_cache, ulp_distance,
                      upload_cache)

pytestmark = pytest.mark.gpu

EDGES = [2, 57, 63, 64, 65, 127, 128, 129, 191, 192, 193, 255, 256, 257, 260]


@pytest.mark.parametrize("H,G,rope,mask,V,lens,offset", [
    (6, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, EDGES, 0),         # three q heads per kv head, nine long prompts
    (4, 4, O.ROPE_CHATGLM, O.MASK_CHATGLM, 5, EDGES, 0),         # one q head per kv head, a P-Tuning prefix, v1 mask
    (5, 5, O.ROPE_DISABLED, O.MASK_CAUSAL, 0, [1000, 3, 641], 0),   # pairs of row tiles under the causal mask
    (32, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, [1410], 0),       # 192 units: more than thread blocks
    (4, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, [130, 170], 1),    # rows start on 4-byte boundaries only
])
def test_prompt_batches(H, G, rope, mask, V, lens, offset):
    from chatglm_cpp_b200 import _lib
    from chatglm_cpp_b200 import attention as A
    inter = rope == O.ROPE_CHATGLM
    desc = make_desc(H, G, 128, 1416, V, rope, 10000.0, mask)
    rng = np.random.default_rng(sum(lens))
    n, width = len(lens), qkv_width(desc, inter)
    arena, ws = A.KVArena(desc, n), A.Workspace(desc, n, max(lens))
    arr, caches, inputs, keep = (_lib.AttnSeq * n)(), [], [], []
    for i, S in enumerate(lens):
        k, v = random_cache(rng, desc, V)
        upload_cache(arena, i, k, v)
        x = rng.standard_normal((S, width)).astype(np.float32)
        flat = torch.zeros(S * width + offset, device="cuda")
        flat[offset:] = torch.from_numpy(x).reshape(-1)
        call = A.SeqCall(qkv=flat[offset:].view(S, width), slot=i, n_past=0, n_ctx=S, out=torch.zeros(S, H * 128, device="cuda"),
                         q_roped=torch.zeros(S, H, 128, device="cuda"), k_roped=torch.zeros(S, G, 128, device="cuda"))
        A.fill_seq(arr[i], desc, call, inter)
        caches.append((k, v))
        inputs.append(x)
        keep.append(call)
    before = _lib.lib().cglm_launch_count()
    _lib.check(_lib.lib().cglm_attn_forward(arena._h, arr, n, ws.ptr, ws.bytes, torch.cuda.current_stream().cuda_stream), "cglm_attn_forward")
    torch.cuda.synchronize()
    assert ws.status() == 0
    n_long = sum(S >= 128 for S in lens)
    # eight long prompts per pair of launches, two launches for the short ones
    assert _lib.lib().cglm_launch_count() - before == 2 * ((n_long + 7) // 8) + (2 if n_long < n else 0)
    for i, S in enumerate(lens):
        k, v = caches[i]
        want, qr, kr = O.attn_forward(oracle_cfg(desc, "f32"), inputs[i], inter, k, v, 0, n_ctx=S, want_roped=True)
        assert_out_close(keep[i].out.cpu().numpy(), want, f"prompt {i} of {S} tokens")
        assert ulp_distance(keep[i].q_roped.cpu().numpy(), qr).max() <= ROPE_MAX_ULP
        assert ulp_distance(keep[i].k_roped.cpu().numpy(), kr).max() <= ROPE_MAX_ULP
        gk, gv = download_cache(arena, i)
        np.testing.assert_array_equal(gk, k)
        np.testing.assert_array_equal(gv, v)
    arena.close()


@pytest.mark.parametrize("H,G,rope,mask,V,chunks,explicit_ids", [
    (8, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, [(0, 2), (0, 57), (0, 127), (61, 2), (127, 65), (1000, 5)], False),
    (8, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 5, [(200, 130), (0, 9), (1000, 300)], True),     # P-Tuning prefix, ids of the caller's
    (4, 4, O.ROPE_CHATGLM, O.MASK_CHATGLM, 0, [(0, 64), (61, 130), (127, 5), (200, 300)], False),   # one q head per kv head, 2-D RoPE
])
def test_short_prompts_and_chunks_keep_f32_operands(H, G, rope, mask, V, chunks, explicit_ids):
    """Prompts below 128 tokens and chunks at n_past > 0 (no mask, chatglm.cpp:689) multiply f32 q and f32 probabilities with the
    cached values.  Several of them in one call, at different positions, NaN in the cache rows behind the attended length.  Besides
    the oracle's gates, the output is compared with float64 over the same roped q and cached values.  Bound: sums of 128 and of T
    f32 products, 2^-24 * sqrt(128 + T) relative in the 2-norm with a factor of 8; operands rounded to f16 miss it by far (2^-12.2
    in the 2-norm for a uniform mantissa, 2e-4, against 2e-5 for the largest T here)."""
    from chatglm_cpp_b200 import _lib
    from chatglm_cpp_b200 import attention as A
    inter = rope == O.ROPE_CHATGLM
    desc = make_desc(H, G, 128, 1416, V, rope, 10000.0, mask)
    rng = np.random.default_rng(H + V)
    n, width, R = len(chunks), qkv_width(desc, inter), H // G
    arena, ws = A.KVArena(desc, n), A.Workspace(desc, n, max(S for _, S in chunks))
    arr, caches, inputs, keep = (_lib.AttnSeq * n)(), [], [], []
    for i, (P, S) in enumerate(chunks):
        k, v = random_cache(rng, desc, V + P)
        k[:, V + P + S:], v[:, :, V + P + S:] = 0x7E00, 0x7E00
        upload_cache(arena, i, k, v)
        x = rng.standard_normal((S, width)).astype(np.float32)
        ids = torch.arange(P, P + S, dtype=torch.int32, device="cuda") if explicit_ids else None
        call = A.SeqCall(qkv=torch.from_numpy(x).cuda(), slot=i, n_past=P, n_ctx=P + S, out=torch.zeros(S, H * 128, device="cuda"),
                         position_ids=ids, q_roped=torch.zeros(S, H, 128, device="cuda"), k_roped=torch.zeros(S, G, 128, device="cuda"))
        A.fill_seq(arr[i], desc, call, inter)
        caches.append((k, v))
        inputs.append(x)
        keep.append(call)
    _lib.check(_lib.lib().cglm_attn_forward(arena._h, arr, n, ws.ptr, ws.bytes, torch.cuda.current_stream().cuda_stream), "cglm_attn_forward")
    torch.cuda.synchronize()
    assert ws.status() == 0
    for i, (P, S) in enumerate(chunks):
        k, v = caches[i]
        want, qr, kr = O.attn_forward(oracle_cfg(desc, "f32"), inputs[i], inter, k, v, P, n_ctx=P + S, want_roped=True)
        got, T = keep[i].out.cpu().numpy(), V + P + S
        assert_out_close(got, want, f"{S} tokens at {P}")
        assert ulp_distance(keep[i].q_roped.cpu().numpy(), qr).max() <= ROPE_MAX_ULP
        assert ulp_distance(keep[i].k_roped.cpu().numpy(), kr).max() <= ROPE_MAX_ULP
        gk, gv = download_cache(arena, i)
        np.testing.assert_array_equal(gk, k)
        np.testing.assert_array_equal(gv, v)
        q = keep[i].q_roped.double().cpu().view(S, G, R, 128)
        kc, vc = (torch.from_numpy(c.view(np.float16)).double() for c in (k[:, :T], v[:, :, :T]))
        sc = torch.einsum("sgrd,gtd->sgrt", q, kc) / 128 ** 0.5
        if P == 0:
            rows, cols = torch.arange(S)[:, None], torch.arange(T)[None]
            hidden = cols > V + rows if mask == O.MASK_CAUSAL else (cols == T - 1) & (rows < S - 1)
            sc.masked_fill_(hidden[:, None, None], float("-inf"))
        exact = torch.einsum("sgrt,gdt->sgrd", torch.softmax(sc, -1), vc).reshape(S, H * 128)
        rel = float((torch.from_numpy(got).double() - exact).norm() / exact.norm())
        assert rel <= 8 * 2.0 ** -24 * (128 + T) ** 0.5, (P, S, rel)
    arena.close()


@pytest.mark.parametrize("H,G,S", [(6, 2, 300), (32, 2, 600), (5, 5, 400)])   # one q tile per CTA; two heads, two row tiles
def test_prompt_rows_whose_first_scores_are_minus_infinity(H, G, S):
    """Keys of the first 150 tokens overflow f16 (to -inf in a dimension that RoPE leaves alone, where every q is positive): their
    scores are -inf and their weights 0.  Rows from 150 on attend the tokens behind them; the reference is float64 over those."""
    from chatglm_cpp_b200 import _lib
    from chatglm_cpp_b200 import attention as A
    N, R = 150, H // G
    desc = make_desc(H, G, 128, 640)
    rng = np.random.default_rng(S)
    arena, ws = A.KVArena(desc, 1), A.Workspace(desc, 1, S)
    x = rng.standard_normal((S, qkv_width(desc, False))).astype(np.float32)
    x[:, 127:H * 128:128] = np.abs(x[:, 127:H * 128:128]) + 0.1
    x[:N, H * 128 + 127:(H + G) * 128:128] = -1e6
    before = _lib.lib().cglm_launch_count()
    out, qr, _ = A.BasicAttention(arena, 0, ws).forward(torch.from_numpy(x).cuda(), 0, want_roped=True)
    torch.cuda.synchronize()
    assert ws.status() == 0 and _lib.lib().cglm_launch_count() - before == 2
    k, v = arena.k_cache(0)[:, N:S].double().cpu(), arena.v_cache(0)[:, :, N:S].double().cpu()
    assert torch.isneginf(arena.k_cache(0)[:, :N, 127]).all()
    sc = torch.einsum("sgrd,gtd->sgrt", qr[N:].double().cpu().view(S - N, G, R, 128), k) / 128 ** 0.5
    sc.masked_fill_((torch.arange(S - N)[None] > torch.arange(S - N)[:, None])[:, None, None], float("-inf"))
    want = torch.einsum("sgrt,gdt->sgrd", torch.softmax(sc, -1), v).reshape(S - N, H * 128)
    assert_out_close(out[N:].cpu().numpy(), want.numpy().astype(np.float32), f"{S} tokens")
    arena.close()


@pytest.mark.parametrize("H,G,rope,mask", [(6, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL), (4, 4, O.ROPE_CHATGLM, O.MASK_CHATGLM)])
@pytest.mark.parametrize("offset", [4, 8, 16])   # f16 output rows on 8-, 16- and 32-byte boundaries only
def test_prompts_with_ids_of_their_own_and_f16_outputs(H, G, rope, mask, offset):
    """Three prompts in one call: ids derived, ids of the caller's that go beyond the cache's angle table, and the derived ids passed
    explicitly.  f16 in and out, the outputs at every alignment of their rows that the store distinguishes."""
    from chatglm_cpp_b200 import attention as A
    inter = rope == O.ROPE_CHATGLM
    desc = make_desc(H, G, 128, 328, 0, rope, 10000.0, mask)
    rng = np.random.default_rng(offset)
    lens, width, cfg = [190, 130, 257], qkv_width(desc, inter), oracle_cfg(desc, "f32")
    arena, ws = A.KVArena(desc, 3), A.Workspace(desc, 3, max(lens))
    calls, inputs, ids = [], [], []
    for i, S in enumerate(lens):
        x = rng.standard_normal((S, width)).astype(np.float16)
        own = O.position_ids(cfg, S, 0, S).astype(np.int32)
        if i == 1:
            own = rng.integers(0, 2000, own.shape).astype(np.int32)
        out = torch.zeros(offset + S * H * 128, device="cuda", dtype=torch.float16)[offset:].view(S, H * 128)
        assert out.data_ptr() % (2 * offset) == 0 and (offset == 16 or out.data_ptr() % (4 * offset) != 0)
        calls.append(A.SeqCall(qkv=torch.from_numpy(x).cuda(), slot=i, n_past=0, n_ctx=S, out=out,
                               position_ids=torch.from_numpy(own).cuda() if i else None))
        inputs.append(x.astype(np.float32))
        ids.append(own)
    A.forward_batch(arena, ws, calls, inter)
    torch.cuda.synchronize()
    assert ws.status() == 0
    for i, S in enumerate(lens):
        k, v = (np.zeros((G, 328, 128), np.uint16), np.zeros((G, 128, 328), np.uint16))
        want = O.attn_forward(cfg, inputs[i], inter, k, v, 0, n_ctx=S, ids=ids[i])
        assert_out_close(calls[i].out.float().cpu().numpy(), want.astype(np.float16).astype(np.float32), f"prompt {i} of {S} tokens")
        gk, gv = download_cache(arena, i)
        np.testing.assert_array_equal(gk, k)
        np.testing.assert_array_equal(gv, v)
    arena.close()
