"""Prompts on the tensor-core path at the sizes where its tiling can go wrong, against the CPU oracle: several prompts per call
(more than one pair of launches takes), lengths around the 64-token softmax step and the 128-row tile, an odd number of q heads
per kv head (a pair without its second head), more units of work than thread blocks (q tiles staged ahead), rows that are not
16-byte aligned.  Bounds: those of assert_out_close for the output, bit equality for the caches, 2 ulp for the roped rows."""
import numpy as np
import pytest
import torch

from oracle import attn_oracle as O

from gpu_util import (ROPE_MAX_ULP, assert_out_close, download_cache, make_desc, oracle_cfg, qkv_width, random_cache, ulp_distance,
                      upload_cache)

pytestmark = pytest.mark.gpu

EDGES = [2, 57, 63, 64, 65, 127, 128, 129, 191, 260]


@pytest.mark.parametrize("H,G,rope,mask,V,lens,offset", [
    (6, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, EDGES, 0),         # three q heads per kv head, ten prompts
    (4, 4, O.ROPE_CHATGLM, O.MASK_CHATGLM, 5, EDGES, 0),         # one q head per kv head, a P-Tuning prefix, v1 mask
    (5, 5, O.ROPE_DISABLED, O.MASK_CAUSAL, 0, [1000, 3, 641], 0),   # pairs of row tiles under the causal mask
    (32, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, [1410], 0),       # 192 units: more than thread blocks
    (4, 2, O.ROPE_CHATGLM2, O.MASK_CAUSAL, 0, [130, 70], 1),     # rows start on 4-byte boundaries only
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
    assert _lib.lib().cglm_launch_count() - before == 2 * ((n + 7) // 8)   # eight prompts per pair of launches
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
