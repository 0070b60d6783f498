"""Small decode launches (one thread-block cluster per sequence and kv head) against the CPU oracle, at the sizes where the split
of an item over the cluster's warps can go wrong: one token, around a warp's 32 and a thread block's 128 tokens, around a whole
round of the cluster (4 x 32 tokens per thread block), the capacity's last row; every cluster size the rule picks, and the lengths
on both sides of its line.  Bounds: those of run_decode_batch (output within assert_out_close, caches bit-exact, roped rows 2 ulp)."""
import numpy as np
import pytest
import torch

from oracle import attn_oracle as O

from gpu_util import assert_out_close, make_desc, oracle_cfg, qkv_width, random_cache, run_decode_batch, upload_cache

pytestmark = pytest.mark.gpu

ROUND = 1024   # tokens of one round of eight thread blocks
LENS8 = [0, 1, 30, 31, 32, 127, 128, 129]


@pytest.mark.parametrize("H,G,rope,mask,V,M,lens", [
    (32, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, 4160, [ROUND - 1]),                       # clusters of eight
    (32, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, 4160, [ROUND, 2 * ROUND + 33, 0, 4095]),   # the rule's line: 64 tiles of 64 tokens
    (32, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, 4160, [4096]),                             # just past it: the persistent kernel
    (32, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, 1096, LENS8 + [1095]),                     # clusters of four; the last cache row
    (6, 2, O.ROPE_DISABLED, O.MASK_CAUSAL, 0, 520, LENS8),                                # three q heads per kv head
    (32, 32, O.ROPE_CHATGLM, O.MASK_CHATGLM, 0, 1096, [700, 1023]),                       # clusters of two, one q head each
    (4, 4, O.ROPE_CHATGLM, O.MASK_CHATGLM, 5, 520, LENS8),                                # a P-Tuning prefix
    (4, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, 264, [7 * i % 256 for i in range(16)]),     # 32 items: clusters of four
    (4, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, 264, [7 * i % 256 for i in range(18)]),     # 36: more than are resident
    (4, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, 584, [512] * 37),                           # 74, two per SM: past its line
    (4, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, 584, [511] * 37),                           # and on it
])
@pytest.mark.parametrize("on_device", [False, True])
def test_small_decode(H, G, rope, mask, V, M, lens, on_device):
    inter = rope == O.ROPE_CHATGLM
    run_decode_batch(make_desc(H, G, 128, M, V, rope, 10000.0, mask), lens, seed=len(lens), interleaved=inter,
                     n_ctx_list=[max(2, p // 2) for p in lens] if inter else None, n_past_on_device=on_device, f16_io=len(lens) > 4)


def test_stale_cache_rows_behind_the_appended_token_do_not_reach_the_result():
    """NaN in every cache row past the attended length: what the last chunk loads beside the item's own tokens."""
    from chatglm_cpp_b200 import attention as A
    desc = make_desc(16, 1, 128, 264)
    rng = np.random.default_rng(5)
    for P in (0, 7, 31, 64, 200):
        arena, ws = A.KVArena(desc, 1), A.Workspace(desc, 1, 1)
        k, v = random_cache(rng, desc, P)
        k[:, P:], v[:, :, P:] = 0x7E00, 0x7E00
        upload_cache(arena, 0, k, v)
        qkv = rng.standard_normal((1, qkv_width(desc, False))).astype(np.float32)
        out = A.BasicAttention(arena, 0, ws).forward(torch.from_numpy(qkv).cuda(), P)
        torch.cuda.synchronize()
        k[:, P:], v[:, :, P:] = 0, 0
        assert_out_close(out.cpu().numpy(), O.attn_forward(oracle_cfg(desc, "f32"), qkv, False, k, v, P), f"n_past {P}")
        arena.close()


@pytest.mark.parametrize("G,P", [(1, 500), (2, 2047), (16, 700), (32, 300)])   # clusters of eight (twice), four, two
@pytest.mark.parametrize("lo,hi", [(0, 64), (96, 300)])
def test_tokens_whose_scores_are_minus_infinity(G, P, lo, hi):
    """Cached keys of tokens [lo, hi) are -inf in a dimension where every q is positive: the scores are -inf and the weights 0, also
    where everything that a warp sees at first is such a token.  The reference is float64 over the other tokens."""
    from chatglm_cpp_b200 import attention as A
    desc = make_desc(2 * G, G, 128, 2056)
    rng = np.random.default_rng(G + lo)
    arena, ws = A.KVArena(desc, 1), A.Workspace(desc, 1, 1)
    k, v = random_cache(rng, desc, P)
    k[:, lo:hi, 127] = 0xFC00
    upload_cache(arena, 0, k, v)
    x = rng.standard_normal((1, qkv_width(desc, False))).astype(np.float32)
    x[:, 127:2 * G * 128:128] = np.abs(x[:, 127:2 * G * 128:128]) + 0.1
    out, qr, _ = A.BasicAttention(arena, 0, ws).forward(torch.from_numpy(x).cuda(), P, want_roped=True)
    torch.cuda.synchronize()
    assert ws.status() == 0
    keep = [t for t in range(P + 1) if not lo <= t < hi]
    kk, vv = arena.k_cache(0)[:, keep].double().cpu(), arena.v_cache(0)[:, :, keep].double().cpu()
    w = torch.softmax(torch.einsum("grd,gtd->grt", qr.double().cpu().view(G, 2, 128), kk) / 128 ** 0.5, -1)
    assert_out_close(out.cpu().numpy(), torch.einsum("grt,gdt->grd", w, vv).reshape(1, -1).numpy().astype(np.float32), f"{G} kv heads")
    arena.close()


@pytest.mark.parametrize("R", [1, 2, 3, 15, 16])
@pytest.mark.parametrize("G", [2, 16, 32])   # clusters of eight, four and two
def test_rows_of_an_item_in_launches_back_to_back(R, G):
    """Items of fewer q heads than the sixteen rows that an MMA has, whole and as un-normalised partials, 100 launches each with
    nothing in between: every one gives the bits of the first, which the oracle holds."""
    from chatglm_cpp_b200 import _lib
    from chatglm_cpp_b200 import attention as A
    H, P = R * G, 190
    desc = make_desc(H, G, 128, 264)
    rng = np.random.default_rng(H)
    arena, ws = A.KVArena(desc, 1), A.Workspace(desc, 1, 1)
    k, v = random_cache(rng, desc, P)
    upload_cache(arena, 0, k, v)
    x = rng.standard_normal((1, qkv_width(desc, False))).astype(np.float32)
    qkv = torch.from_numpy(x).cuda()
    attn = A.BasicAttention(arena, 0, ws)
    outs = [attn.forward(qkv, P) for _ in range(100)]
    parts = [torch.zeros(H, 130, device="cuda") for _ in range(100)]
    for p in parts:
        A.forward_batch(arena, ws, [A.SeqCall(qkv=qkv, slot=0, n_past=P, n_ctx=0, partial=p, flags=_lib.SEQ_PARTIAL)], False)
    torch.cuda.synchronize()
    assert ws.status() == 0
    assert all(torch.equal(o, outs[0]) for o in outs) and all(torch.equal(p, parts[0]) for p in parts)
    want = O.attn_forward(oracle_cfg(desc, "f32"), x, False, k, v, P)
    assert_out_close(outs[0].cpu().numpy(), want, f"{H} q heads, {G} kv heads")
    whole = (parts[0][:, :128] / parts[0][:, 129:]).reshape(1, -1)
    assert_out_close(whole.cpu().numpy(), want, "partial")
    arena.close()


@pytest.mark.parametrize("G", [8, 10, 13, 16, 20])
def test_merge_of_items_cut_into_many_parts(G):
    """One sequence just past the clusters' line, cut over one thread block per SM: 7 to 18 parts per item, i.e. fewer than one
    batch of copies, both of its barriers, more parts than slots in the tile ring, and the two-level merge."""
    run_decode_batch(make_desc(2 * G, G, 128, 4168, 0, O.ROPE_CHATGLM2, 10000.0, O.MASK_CAUSAL), [4150], seed=G)


@pytest.mark.parametrize("G,P", [(8, 4150), (13, 4150), (2, 20000)])   # one and two rounds of copies, two levels of merging
def test_merged_parts_are_those_of_the_launch(G, P):
    """Launches with two inputs in turn through the same scratch: every result has the bits of the first launch with that input, so
    no part, group partial or slot of the tile ring is one that an earlier launch left behind."""
    from chatglm_cpp_b200 import attention as A
    desc = make_desc(2 * G, G, 128, P + 72)
    rng = np.random.default_rng(G)
    arena, ws = A.KVArena(desc, 2), A.Workspace(desc, 1, 1)
    attn, x = [], []
    for slot in range(2):
        k, v = random_cache(rng, desc, P)
        upload_cache(arena, slot, k, v)
        attn.append(A.BasicAttention(arena, slot, ws))
        x.append(torch.from_numpy(rng.standard_normal((1, qkv_width(desc, False))).astype(np.float32)).cuda())
    first = [attn[i].forward(x[i], P) for i in range(2)]
    outs = [attn[i % 2].forward(x[i % 2], P) for i in range(300)]
    torch.cuda.synchronize()
    assert ws.status() == 0 and not torch.equal(first[0], first[1])
    assert all(torch.equal(o, first[i % 2]) for i, o in enumerate(outs))
    arena.close()


@pytest.mark.parametrize("n_tok,n_in,n_out", [(128, 256, 128), (128, 512, 4096), (33, 4096, 4608), (1, 128, 128), (17, 4160, 256),
                                              (100, 8576, 256), (128, 8576, 4608), (128, 8448, 4096)])   # a whole SM each
def test_linear_k_split_over_a_cluster(n_tok, n_in, n_out):
    """Fewer weight blocks than the sums need room, one block per thread block, token counts that no CTA's share divides, a k that
    four does and does not split evenly, long slices of k by clusters of two and of four.  Bound: f32 sums of n_in products of f16 values, 2^-24 * sqrt(n_in) of the sum of their
    sizes with a factor of 8."""
    from chatglm_cpp_b200 import _lib
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n_tok + n_in)
    x = torch.randn(n_tok, n_in, device="cuda", generator=gen).half()
    w = torch.randn(n_out, n_in, device="cuda", generator=gen).half()
    b = torch.randn(n_out, device="cuda", generator=gen)
    L = _lib.lib()
    ws = torch.zeros(L.cglm_linear_workspace_bytes(), dtype=torch.uint8, device="cuda")
    out = torch.empty(n_tok, n_out, device="cuda")
    torch.cuda.synchronize()
    stream = torch.cuda.current_stream().cuda_stream
    _lib.check(L.cglm_linear_forward(x.data_ptr(), n_tok, n_in, w.data_ptr(), n_out, b.data_ptr(), out.data_ptr(), 0, ws.data_ptr(),
                                     ws.numel(), stream), "cglm_linear_forward")
    want = x.double() @ w.double().T + b.double()
    size = x.double().abs() @ w.double().abs().T + b.double().abs()
    assert ((out.double() - want).abs() <= 8 * 2.0 ** -24 * n_in ** 0.5 * size).all()
