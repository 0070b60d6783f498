"""The work a user of this framework has it do, as cases that can be timed and compared.

Everything goes through the public entry points: the Python module API (``KVArena``, ``Workspace``,
``BasicAttention.forward``) where one sequence is served, and the C ABI of include/cglm_attn.h with descriptor arrays
built once per sequence layout, as a host program calls it, where a batch or a whole attention block is.

Shapes are those of the model families the framework names: ChatGLM3-6B and GLM-4-9B (32 q heads, 2 kv heads, blocked
qkv, half-rotary RoPE) and ChatGLM-6B v1 (32 heads with their own K/V, interleaved qkv, 2-D RoPE, prefix mask); head_dim
128 and hidden 4096 throughout.  Synthetic data: activations and caches N(0, 1), weights N(0, 1) / sqrt(in_features).

The kinds of case:
  module   one sequence through BasicAttention.forward, one layer: a decode token (qlen 1 at n_past) or a prompt
           (qlen tokens into an empty cache)
  decode   one decode step of a batch through `layers` layers, attention only, inputs on the device
  host     the same step from pinned host buffers and back
  block    the step with both Linears around the attention (query_key_value, attention, dense), issued call by call
  graph    the step with both Linears captured once as a CUDA graph whose positions are device words, replayed per token
  prompt   a prompt through `layers` layers with both Linears
"""
import math

import numpy as np
import torch

from chatglm_cpp_b200 import _lib
from chatglm_cpp_b200 import attention as A

HIDDEN = 4096
MODELS = {
    # H, G, D, rope, theta, interleaved qkv, mask
    "glm3_6b": (32, 2, 128, _lib.ROPE_CHATGLM2, 1.0e4, False, _lib.MASK_CAUSAL),
    "glm4_9b": (32, 2, 128, _lib.ROPE_CHATGLM2, 5.0e6, False, _lib.MASK_CAUSAL),
    "glm1_6b": (32, 32, 128, _lib.ROPE_CHATGLM, 1.0e4, True, _lib.MASK_CHATGLM),
}


def _case(kind, model, seqs=1, layers=1, lo=0, hi=0, qlen=1, act="f32", virtual=0, capacity=8192, name=None):
    """lo, hi: range of the sequences' cached tokens (n_past) before the call; act: type of the activations that enter
    and leave the attention; virtual: tokens of a P-Tuning v2 prefix; capacity: max_length of the caches."""
    c = dict(kind=kind, model=model, seqs=seqs, layers=layers, lo=lo, hi=hi, qlen=qlen, act=act, virtual=virtual,
             capacity=capacity)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the reference's own CPU-runnable case: one token of one chat, one layer
        _case("module", "glm3_6b", lo=512, hi=512, capacity=2048, name="decode_1x512"),
        # a short question: most prompts of a chat are a few dozen tokens
        _case("module", "glm3_6b", qlen=57, capacity=2048, name="prompt_57"),
        # an ordinary prompt with the older family's mask, RoPE and qkv layout; ragged against every tile
        _case("module", "glm1_6b", qlen=777, capacity=2048, name="prompt_v1_777"),
        # a long document, half-precision hand-off: the contraction-bound end of the range
        _case("module", "glm3_6b", qlen=8192, act="f16", capacity=8192, name="prompt_8192"),
        # one very long context
        _case("module", "glm4_9b", lo=131072, hi=131072, capacity=131072 + 64, name="decode_1x131072"),
        # batched serving, attention only: the framework's headline step (a few of its layers)
        _case("decode", "glm4_9b", seqs=64, layers=4, lo=1024, hi=8191, name="decode_64"),
        # the older family, every head with its own cache
        _case("decode", "glm1_6b", seqs=4, layers=4, lo=2048, hi=2048, capacity=4096, name="decode_v1_4x2048"),
        # a host program that keeps its activations in pinned memory
        _case("host", "glm4_9b", seqs=64, layers=4, lo=1024, hi=8191, act="f16", name="host_decode_64"),
        # whole attention modules of a small and of a full batch
        _case("block", "glm4_9b", seqs=8, layers=4, lo=1024, hi=8191, act="f16", name="block_8"),
        _case("block", "glm4_9b", seqs=64, layers=4, lo=1024, hi=8191, act="f16", name="block_64"),
        # the reference's generation loop: one chat, every layer, one replayed graph per token
        _case("graph", "glm3_6b", layers=28, lo=512, hi=512, act="f16", capacity=2048, name="token_graph_28"),
        # an ordinary prompt through whole attention modules
        _case("prompt", "glm4_9b", layers=2, qlen=1024, act="f16", name="prompt_block_1024"),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["module", "module", "module", "decode", "decode", "host", "block", "block", "graph", "prompt"])
    if kind == "module":
        if rng.random() < 0.5:   # a prompt
            model = rng.choice(["glm3_6b", "glm4_9b", "glm1_6b"])
            virtual = rng.choice([0, 0, 0, 128]) if model != "glm4_9b" else 0
            qlen = _log(rng, 8, 2048 if model == "glm1_6b" else 8000)
            return _case(kind, model, qlen=qlen, act=rng.choice(["f32", "f16"]), virtual=virtual,
                         capacity=2048 if model == "glm1_6b" else 8192)
        model = rng.choice(["glm3_6b", "glm4_9b", "glm4_9b", "glm1_6b"])
        top = {"glm3_6b": 8191, "glm4_9b": 131072, "glm1_6b": 2047}[model]
        n = _log(rng, 16, top)
        return _case(kind, model, lo=n, hi=n, act=rng.choice(["f32", "f16"]),
                     virtual=rng.choice([0, 0, 0, 128]) if model == "glm3_6b" else 0,
                     capacity={"glm3_6b": 8192, "glm4_9b": 131072 + 64, "glm1_6b": 2048}[model])
    if kind == "prompt":
        return _case(kind, rng.choice(["glm3_6b", "glm4_9b"]), layers=rng.randint(1, 3), qlen=_log(rng, 8, 2048), act="f16")
    if kind == "graph":
        lo = _log(rng, 16, 1500)
        return _case(kind, rng.choice(["glm3_6b", "glm4_9b"]), seqs=rng.choice([1, 1, 1, 2, 4]), layers=rng.randint(8, 28),
                     lo=lo, hi=lo + rng.randint(0, 500), act="f16", capacity=2048)
    act = "f16" if kind in ("host", "block") else rng.choice(["f32", "f16"])
    if kind != "block" and rng.random() < 0.25:
        lo = _log(rng, 64, 1500)
        return _case(kind, "glm1_6b", seqs=_log(rng, 1, 8), layers=rng.randint(2, 4), lo=lo, hi=lo + rng.randint(0, 500), act=act,
                     capacity=2048)
    lo = _log(rng, 64, 4000)
    return _case(kind, "glm4_9b", seqs=_log(rng, 1, 64), layers=rng.randint(2, 4), lo=lo, hi=lo + rng.randint(0, 4000), act=act)


def _lengths(case):
    """Cached tokens of every sequence: a property of the case, so that its bytes are known."""
    return [int(p) for p in np.random.default_rng(1003 + case["seqs"]).integers(case["lo"], case["hi"] + 1, case["seqs"])]


def _dtype(case):
    return torch.float16 if case["act"] == "f16" else torch.float32


class _State:
    """One case's caches, activations, weights, descriptors and (graph) captured step."""

    def __init__(self, case, seed):
        H, G, D, rope, theta, interleaved, mask = MODELS[case["model"]]
        self.lib, self.kind, self.layers, self.n = _lib.lib(), case["kind"], case["layers"], case["seqs"]
        self.qlen, self.act = case["qlen"], _dtype(case)
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.H, self.G, self.D, self.interleaved, self.virtual = H, G, D, interleaved, case["virtual"]
        self.width, self.heads = (H + 2 * G) * D, H * D
        self.desc = _lib.AttnDesc(H, G, D, case["capacity"] + case["virtual"], case["virtual"], rope, theta, mask)
        self.arena = A.KVArena(self.desc, self.layers * self.n)
        self.k, self.v = self.arena.k_all(), self.arena.v_all()
        self.k.owner = self.v.owner = self.arena   # views of the arena's memory: whoever keeps them keeps it alive
        if self.qlen == 1:   # a cache that earlier tokens have filled; a prompt finds it empty
            self.k.normal_(generator=self.gen)
            self.v.normal_(generator=self.gen)
        elif self.virtual:
            prefix = self.randn(2, G, self.virtual, D)
            for slot in range(self.layers * self.n):
                self.arena.load_prefix(slot, prefix)
        self.ws = A.Workspace(self.desc, self.n, self.qlen)
        self.n_past = _lengths(case)
        # ChatGLM-6B v1 derives its two position ids from the prompt's length
        self.n_ctx = [self.qlen if self.qlen > 1 else max(2, p // 2) for p in self.n_past]
        getattr(self, "prepare_" + self.kind)()

    def randn(self, *shape, dtype=torch.float16, scale=1.0):
        x = torch.empty(*shape, device="cuda", dtype=dtype).normal_(generator=self.gen)
        return x.mul_(scale) if scale != 1.0 else x

    def descriptors(self, layer, qkv, out, flags=0, n_past_dev=None):
        """The descriptor array of one layer call: qkv [sequences * qlen, width], out [sequences * qlen, heads * head_dim]."""
        arr, q = (_lib.AttnSeq * self.n)(), self.qlen
        for i in range(self.n):
            A.fill_seq(arr[i], self.desc,
                       A.SeqCall(qkv=qkv[i * q:(i + 1) * q], slot=layer * self.n + i, n_past=self.n_past[i], n_ctx=self.n_ctx[i],
                                 out=out[i * q:(i + 1) * q], flags=flags,
                                 n_past_dev=None if n_past_dev is None else n_past_dev[i:i + 1]), self.interleaved)
        return arr

    # ---- one sequence, one layer, through the module -------------------------------------------------------------------
    def prepare_module(self):
        self.attn = A.BasicAttention(self.arena, 0, self.ws, self.interleaved)
        self.qkv = self.randn(self.qlen, self.width, dtype=self.act)

    def run_module(self):
        out = self.attn.forward(self.qkv, self.n_past[0], self.n_ctx[0], out_dtype=self.act)
        return {"out": out, "k": self.k, "v": self.v}

    # ---- a batch's decode step, attention only -----------------------------------------------------------------------------
    def prepare_decode(self):
        self.qkv = self.randn(self.layers, self.n, self.width, dtype=self.act)
        self.out = torch.empty(self.layers, self.n, self.heads, device="cuda", dtype=self.act)
        self.calls = [self.descriptors(l, self.qkv[l], self.out[l]) for l in range(self.layers)]

    def run_decode(self):
        stream = torch.cuda.current_stream().cuda_stream
        for arr in self.calls:
            _lib.check(self.lib.cglm_attn_forward(self.arena._h, arr, self.n, self.ws.ptr, self.ws.bytes, stream), "cglm_attn_forward")
        return {"out": self.out, "k": self.k, "v": self.v}

    # ---- the same step from and to pinned host memory ------------------------------------------------------------------------
    def prepare_host(self):
        dt = self.act
        self.qkv_host = self.randn(self.layers, self.n, self.width, dtype=dt).cpu().pin_memory()
        self.out_host = torch.empty(self.layers, self.n, self.heads, dtype=dt).pin_memory()
        self.stage = [(torch.empty(self.n, self.width, device="cuda", dtype=dt), torch.empty(self.n, self.heads, device="cuda", dtype=dt))
                      for _ in range(3)]
        self.calls = [self.descriptors(l, self.stage[l % 3][0], self.stage[l % 3][1]) for l in range(self.layers)]
        self.layout = (_lib.HOST_INTERLEAVED_QKV if self.interleaved else 0) | (_lib.HOST_F16 if dt == torch.float16 else 0)
        self.ptrs = [(self.qkv_host[l].data_ptr(), self.out_host[l].data_ptr(), self.stage[l % 3][0].data_ptr(),
                      self.stage[l % 3][1].data_ptr()) for l in range(self.layers)]

    def run_host(self):
        stream = torch.cuda.current_stream().cuda_stream
        for arr, (src, dst, dev_in, dev_out) in zip(self.calls, self.ptrs):
            _lib.check(self.lib.cglm_attn_forward_host(self.arena._h, arr, self.n, self.layout, src, dst, dev_in, dev_out, self.ws.ptr,
                                                       self.ws.bytes, stream), "cglm_attn_forward_host")
        # the step's results are read back here: the stream waits for the copies
        _lib.check(self.lib.cglm_attn_host_drain(self.arena._h, stream), "cglm_attn_host_drain")
        return {"out": self.out_host, "k": self.k, "v": self.v}

    # ---- with both Linears -----------------------------------------------------------------------------------------------------
    def prepare_linears(self):
        tokens = self.n * self.qlen
        self.w_qkv = self.randn(self.layers, self.width, HIDDEN, scale=HIDDEN ** -0.5)
        self.b_qkv = self.randn(self.layers, self.width, dtype=torch.float32, scale=0.1)
        self.w_dense = self.randn(self.layers, HIDDEN, self.heads, scale=self.heads ** -0.5)
        self.hidden = self.randn(self.layers, tokens, HIDDEN)
        self.qkv = torch.empty(tokens, self.width, device="cuda", dtype=torch.float16)
        self.context = torch.empty(tokens, self.heads, device="cuda", dtype=torch.float16)
        self.out = torch.empty(self.layers, tokens, HIDDEN, device="cuda", dtype=torch.float32)

    def issue_linears(self, calls):
        """Every layer: plain query_key_value GEMM (f16 row), attention with its own RoPE and append, dense GEMM."""
        lib, ws, n_bytes, tokens = self.lib, self.ws.ptr, self.ws.bytes, self.n * self.qlen
        stream = torch.cuda.current_stream().cuda_stream
        for l, arr in enumerate(calls):
            w_qkv, b_qkv, w_dense, x, y = self.layer_ptrs[l]
            _lib.check(lib.cglm_linear_forward(x, tokens, HIDDEN, w_qkv, self.width, b_qkv, self.qkv_ptr, 1, ws, n_bytes, stream),
                       "cglm_linear_forward")
            _lib.check(lib.cglm_attn_forward(self.arena._h, arr, self.n, ws, n_bytes, stream), "cglm_attn_forward")
            _lib.check(lib.cglm_linear_forward(self.context_ptr, tokens, self.heads, w_dense, HIDDEN, None, y, 0, ws, n_bytes, stream),
                       "cglm_linear_forward")

    def pointers(self):
        self.qkv_ptr, self.context_ptr = self.qkv.data_ptr(), self.context.data_ptr()
        self.layer_ptrs = [(self.w_qkv[l].data_ptr(), self.b_qkv[l].data_ptr(), self.w_dense[l].data_ptr(), self.hidden[l].data_ptr(),
                            self.out[l].data_ptr()) for l in range(self.layers)]

    def prepare_prompt(self):
        self.prepare_linears()
        self.calls = [self.descriptors(l, self.qkv, self.context) for l in range(self.layers)]
        self.pointers()

    def run_prompt(self):
        self.issue_linears(self.calls)
        return {"out": self.out, "k": self.k, "v": self.v}

    # Up to 32 sequences the query_key_value GEMM carries bias, RoPE and the cache append in its epilogue and hands roped q
    # to the attention, which is the route BasicAttention::forward of the C++ mirror takes for a decode token; a larger
    # batch takes the plain GEMM, as the framework's documentation says.
    def prepare_block(self):
        self.prepare_linears()
        self.fused = self.n <= 32
        if not self.fused:
            self.calls = [self.descriptors(l, self.qkv, self.context) for l in range(self.layers)]
            return self.pointers()
        self.q_roped = torch.empty(self.n, self.heads, device="cuda", dtype=torch.float32)
        self.lin_calls, self.calls = [], []
        flags = _lib.SEQ_Q_ROPED | _lib.SEQ_NO_APPEND | _lib.SEQ_USE_KV_LOCAL | _lib.SEQ_OUT_F16
        for l in range(self.layers):
            lin, att = (_lib.AttnSeq * self.n)(), (_lib.AttnSeq * self.n)()
            for i, p in enumerate(self.n_past):
                for a in (lin[i], att[i]):
                    a.slot, a.qlen, a.n_past = l * self.n + i, 1, p
                att[i].q = att[i].k = att[i].v = self.q_roped[i].data_ptr()   # k and v are not read
                att[i].q_tok_stride = att[i].kv_tok_stride = self.heads
                att[i].q_head_stride = att[i].kv_head_stride = self.D
                att[i].out, att[i].flags, att[i].kv_local = self.context[i].data_ptr(), flags, self.virtual + p + 1
            self.lin_calls.append(lin)
            self.calls.append(att)
        self.pointers()

    def run_block(self):
        if not self.fused:
            self.issue_linears(self.calls)
        else:
            lib, ws, n_bytes, n = self.lib, self.ws.ptr, self.ws.bytes, self.n
            stream, q_roped = torch.cuda.current_stream().cuda_stream, self.q_roped.data_ptr()
            for l in range(self.layers):
                w_qkv, b_qkv, w_dense, x, y = self.layer_ptrs[l]
                _lib.check(lib.cglm_qkv_linear_forward(self.arena._h, self.lin_calls[l], n, x, HIDDEN, w_qkv, b_qkv, q_roped, ws,
                                                       n_bytes, stream), "cglm_qkv_linear_forward")
                _lib.check(lib.cglm_attn_forward(self.arena._h, self.calls[l], n, ws, n_bytes, stream), "cglm_attn_forward")
                _lib.check(lib.cglm_linear_forward(self.context_ptr, n, self.heads, w_dense, HIDDEN, None, y, 0, ws, n_bytes, stream),
                           "cglm_linear_forward")
        return {"out": self.out, "k": self.k, "v": self.v}

    # What chatglm::DecodeStep does: the step's launches captured once, the positions read from device words that the
    # graph's last node advances.  Every pass here decodes the same token, so the words are set before each replay.
    def prepare_graph(self):
        self.prepare_linears()
        self.start = torch.tensor(self.n_past, dtype=torch.int32, device="cuda")
        self.position = self.start.clone()
        self.calls = [self.descriptors(l, self.qkv, self.context, _lib.SEQ_N_PAST_DEVICE, self.position) for l in range(self.layers)]
        for arr in self.calls:
            for i in range(self.n):   # an upper bound, as DecodeStep gives it: the capacity
                arr[i].n_past = self.desc.max_len - self.virtual - 1
        self.pointers()

        def step():
            self.issue_linears(self.calls)
            _lib.check(self.lib.cglm_seq_advance(self.position.data_ptr(), self.n, 1, torch.cuda.current_stream().cuda_stream),
                       "cglm_seq_advance")

        side = torch.cuda.Stream()   # one step issued eagerly, then captured
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            step()

    def run_graph(self):
        self.position.copy_(self.start)
        self.graph.replay()
        return {"out": self.out, "k": self.k, "v": self.v, "position": self.position}


def prepare(case, seed):
    return _State(case, seed)


def run(state):
    return getattr(state, "run_" + state.kind)()


def work(case):
    """Bytes: the cached K and V of every attended token (f16) once, the activations and weights in and out once.  Flops:
    two products of head_dim per q head and visible (token, token) pair, and the Linears."""
    H, G, D = MODELS[case["model"]][:3]
    esz = 2 if case["act"] == "f16" else 4
    q, n, V = case["qlen"], case["seqs"], case["virtual"]
    width, heads, tokens = (H + 2 * G) * D, H * D, n * q
    lengths = _lengths(case)
    kv = sum(4 * G * D * (V + p + q) for p in lengths)
    if q > 1:      # causal: row s sees V + s + 1 tokens; the v1 prefix mask hides one token from every row but the last
        pairs = q * V + (q * (q + 1) // 2 if case["model"] != "glm1_6b" else q * q - (q - 1))
    else:
        pairs = sum(V + p + 1 for p in lengths)
    n_bytes, flops = kv + tokens * (width + heads) * esz, 4 * H * D * pairs
    if case["kind"] in ("block", "graph", "prompt"):
        weights = width * HIDDEN + HIDDEN * heads
        n_bytes = kv + weights * 2 + width * 4 + tokens * HIDDEN * (2 + 4)
        flops += 2 * tokens * weights
    return {"bytes": n_bytes * case["layers"], "flops": flops * case["layers"]}


def tolerance(case):
    """q, the probabilities and the cached values enter the products in f16 (relative spacing 2^-11 each way); a block
    rounds the qkv row and the context to f16 as well, and values appended to the caches may be the neighbouring f16."""
    return {"rel": 3e-3 if case["kind"] in ("block", "graph", "prompt") else 2e-3}
