"""-m gpu: the attention of a chunk against 64 bits, from the very rows that lie in the cache.

The layer's projections only pick numbers of the normed row (one entry of a power of two in each row of a matrix), so that queries, keys and
values are the same bits whatever kernel forms the products: the rotated keys of a position are the rotated queries of its group's first
head, read back with the scratch hook from the token alone at that position, and the values are the same at position 0 (nothing rotates),
rolled by some dims."""
import ctypes as C
import math

import pytest
import torch

from oracle.llama_oracle import mlx_affine_quantize

pytestmark = pytest.mark.gpu

HD, H, ROLL = 128, 512, 37


def picks(rows, scale, g):
    """[rows * 128, H]: every output is one input times `scale`"""
    w = torch.zeros(rows * HD, H)
    w[torch.arange(rows * HD), torch.cat([torch.randperm(H, generator=g)[:HD] for _ in range(rows)])] = scale
    return w


class Layer:
    def __init__(self, lib, kv_heads, group, kv_bits=0, max_tokens=2560, seed=1):
        from dnet_b200.core.models.llama import LlamaRingModel

        self.lib, self.kv_heads, self.group, self.heads = lib, kv_heads, group, kv_heads * group
        g = torch.Generator().manual_seed(seed)
        k = picks(kv_heads, 1.0, g).view(kv_heads, 1, HD, H)
        q = picks(self.heads, 2.0, g).view(kv_heads, group, HD, H)
        q[:, 0] = k[:, 0]
        cfg = dict(hidden_size=H, num_attention_heads=self.heads, num_key_value_heads=kv_heads, head_dim=HD, intermediate_size=256, vocab_size=256,
                   num_hidden_layers=1, rms_norm_eps=1e-5, rope_theta=10000.0, model_type="llama", torch_dtype="bfloat16")
        p = "model.layers.0."
        w = {"self_attn.q_proj": q.reshape(-1, H), "self_attn.k_proj": k.reshape(-1, H), "self_attn.v_proj": k.roll(ROLL, 2).reshape(-1, H),
             "self_attn.o_proj": torch.randn(H, self.heads * HD, generator=g) * 0.01, "mlp.gate_proj": torch.randn(256, H, generator=g) * 0.01,
             "mlp.up_proj": torch.randn(256, H, generator=g) * 0.01, "mlp.down_proj": torch.randn(H, 256, generator=g) * 0.01,
             "input_layernorm": torch.ones(H), "post_attention_layernorm": torch.ones(H)}
        self.m = LlamaRingModel(cfg, [0], kv_pool_pages=max_tokens // 64 + 2, kv_bits=kv_bits)
        self.m.load_weights({f"{p}{n}.weight": t.to(torch.bfloat16).cuda() for n, t in w.items()})
        self.kv = self.m.make_cache(max_tokens=max_tokens)

    def close(self):
        self.kv.free()
        self.m.destroy()

    def run(self, x, at):
        self.kv.seek(at)
        return self.m.apply_single_layer(0, x.clone(), self.kv)

    def hook(self, which, T):
        out = torch.empty(T, self.heads, HD, dtype=torch.bfloat16)
        assert self.lib.dn_debug_scratch(self.m._h, which, out.data_ptr(), out.numel() * 2, 0) == 0
        return out

    def rows(self, x):
        """keys and values [tokens, kv heads, 128] as the cache is given them"""
        k, v = [], []
        for t in range(len(x)):
            self.run(x[t:t + 1], t)
            k.append(self.hook(0, 1)[0, ::self.group])
            self.run(x[t:t + 1], 0)
            v.append(self.hook(0, 1)[0, ::self.group].roll(ROLL, -1))
        return torch.stack(k), torch.stack(v)

    def attend(self, x, context):
        """queries and attention outputs [T, heads, 128] of the tokens behind `context`"""
        if context:
            self.run(x[:context], 0)
        self.run(x[context:], context)
        T = len(x) - context
        q, o = self.hook(0, T), self.hook(1, T)
        assert self.lib.dn_step_error(self.m._h, 0) == 0
        return q, o


def exact(q, k, v, context, group):
    """softmax attention in 64 bits; also the size of a sum whose terms are each off by their own share, and of one cut at every addition"""
    T, heads = q.shape[:2]
    out, spread, total = (torch.empty(T, heads, HD, dtype=torch.float64) for _ in range(3))
    seen = torch.arange(len(k))[None] <= context + torch.arange(T)[:, None]
    for h in range(heads):
        s = (q[:, h].double() @ k[:, h // group].double().T) * HD ** -0.5
        p = torch.softmax(s.masked_fill(~seen, -math.inf), -1)
        vv = v[:, h // group].double()
        out[:, h], spread[:, h], total[:, h] = p @ vv, ((p * p) @ (vv * vv)).sqrt(), p @ vv.abs()
    return out, spread, total


def beyond_rounding(got, ref):
    """how far a stored bf16 lies from the exact value beyond half a last place"""
    half = torch.exp2(torch.floor(torch.log2(ref.abs().clamp_min(1e-30))) - 8)
    return ((got.double() - ref).abs() - half).clamp_min(0)


# (groups of 5 and 7, chunks of fewer than 16 tokens and those of up to 32 rows a group, which k_attn_few takes, hold a weight's 24 bits; the others 16: a
# weight is off by 2^-18 of itself at most)
@pytest.mark.parametrize("group,context,T,eps", [(4, 300, 1, 2.0 ** -19), (4, 300, 3, 2.0 ** -19), (1, 500, 15, 2.0 ** -19), (5, 640, 8, 2.0 ** -19), (7, 63, 15, 2.0 ** -19), (8, 0, 2, 2.0 ** -19),
                                                 (8, 2200, 4, 2.0 ** -19), (2, 1100, 16, 2.0 ** -19), (1, 700, 32, 2.0 ** -19), (5, 127, 6, 2.0 ** -19), (7, 1900, 2, 2.0 ** -19),
                                                 (5, 2200, 64, 2.0 ** -18), (7, 300, 40, 2.0 ** -18), (5, 0, 300, 2.0 ** -18),
                                                 (4, 2200, 64, 2.0 ** -16), (8, 1000, 16, 2.0 ** -16), (2, 0, 300, 2.0 ** -16), (1, 129, 130, 2.0 ** -16)])
def test_attention_over_16_bit_pages(cuda_lib, group, context, T, eps):
    x = torch.randn(context + T, H, generator=torch.Generator().manual_seed(context + T)).to(torch.bfloat16).cuda()
    layer = Layer(cuda_lib, 2, group)
    try:
        k, v = layer.rows(x)
        q, got = layer.attend(x, context)
    finally:
        layer.close()
    ref, spread, total = exact(q, k, v, context, group)
    over = beyond_rounding(got, ref)
    print(f"G {group} context {context} T {T}: beyond rounding / spread {float((over / spread.clamp_min(1e-30)).max()):.2e}, misrounded {float((over > 0).double().mean()):.5f}")
    assert bool((over <= eps * spread + 2.0 ** -22 * total).all())


def exact_quantised(q, k, v, context, group, bits):
    """the quantised semantics in 64 bits: scores and probabilities rounded to bf16"""
    def deq(x):
        c, s, b = mlx_affine_quantize(x, bits)
        g = c.double().view(*x.shape[:-1], 2, 64)
        return (g * s.double()[..., None] + b.double()[..., None]).view(x.shape)

    def r16(x):      # nearest bf16 of a float64, ties to even
        m, e = torch.frexp(x)
        return torch.ldexp(torch.round(torch.ldexp(m, torch.tensor(8))), e - 8)

    kd, vd = deq(k), deq(v)
    T, heads = q.shape[:2]
    out = torch.empty(T, heads, HD, dtype=torch.float64)
    seen = torch.arange(len(k))[None] <= context + torch.arange(T)[:, None]
    for h in range(heads):
        qs = (q[:, h].float() * torch.tensor(0.08838834764831845)).to(torch.bfloat16).double()
        s = r16(qs @ kd[:, h // group].T).masked_fill(~seen, -math.inf)
        out[:, h] = r16(torch.softmax(s, -1)) @ vd[:, h // group]
    return out


@pytest.mark.parametrize("bits,group,context,T", [(8, 4, 300, 1), (8, 4, 2200, 3), (8, 1, 500, 128), (4, 8, 1500, 16), (8, 5, 2000, 64), (4, 7, 100, 40), (8, 2, 700, 512)])
def test_attention_over_quantised_pages(cuda_lib, bits, group, context, T):
    """Scores and probabilities are rounded to bf16, so that a fp32 sum near a rounding edge may land on its other side: how often is what a
    kernel's precision shows in.  The tensor-core kernel is held to the one of fp32 multiply-adds on the same pages."""
    x = torch.randn(context + T, H, generator=torch.Generator().manual_seed(context + T)).to(torch.bfloat16).cuda()
    layer, off = Layer(cuda_lib, 2, group, kv_bits=bits), {}
    try:
        k, v = layer.rows(x)
        for tc in (1, 0):
            cuda_lib.dn_set_option(b"tc_attn", tc)
            q, got = layer.attend(x, context)
            if tc:
                ref = exact_quantised(q, k, v, context, group, bits)
            over = beyond_rounding(got, ref)
            off[tc] = float((over > 0).double().mean())
    finally:
        cuda_lib.dn_set_option(b"tc_attn", 1)
        layer.close()
    print(f"bits {bits} G {group} context {context} T {T}: misrounded {off[1]:.5f}, multiply-adds {off[0]:.5f}")
    assert off[1] <= 2 * off[0] + 1e-3


@pytest.mark.parametrize("bits,group,T", [(0, 4, 1), (0, 5, 1), (0, 4, 3), (0, 7, 15), (0, 4, 16), (0, 5, 200), (8, 4, 1), (4, 1, 2), (8, 5, 64)])
def test_a_captured_chunk_gives_the_bits_of_an_eager_one(cuda_lib, bits, group, T):
    """a chunk captured once, for a cache of 4,096 tokens, and replayed at positions whose keys are shared out differently"""
    n = 2600
    x = torch.randn(n + T, H, generator=torch.Generator().manual_seed(n + T)).to(torch.bfloat16).cuda()
    layer, s, graph = Layer(cuda_lib, 2, group, kv_bits=bits, max_tokens=4096), torch.cuda.Stream(), C.c_void_p()
    try:
        layer.run(x, 0)      # the cache's rows
        torch.cuda.synchronize()
        buf, ids = torch.empty(T, H, dtype=torch.bfloat16, device="cuda"), (C.c_int32 * 1)(0)
        assert cuda_lib.dn_graph_begin(s.cuda_stream) == 0
        assert cuda_lib.dn_chunk_forward(layer.m._h, ids, 1, buf.data_ptr(), T, layer.kv._h, s.cuda_stream) == 0
        assert cuda_lib.dn_graph_end(s.cuda_stream, C.byref(graph)) == 0
        for at in (0, 300, 1100, n):
            with torch.cuda.stream(s):
                out = []
                for captured in (True, False):
                    buf.copy_(x[at:at + T])
                    layer.kv.seek(at, s.cuda_stream)
                    if captured:
                        assert cuda_lib.dn_graph_launch(graph, s.cuda_stream) == 0
                    else:
                        assert cuda_lib.dn_chunk_forward(layer.m._h, ids, 1, buf.data_ptr(), T, layer.kv._h, s.cuda_stream) == 0
                    out.append(buf.clone())
            torch.cuda.synchronize()
            assert torch.equal(*out), at
        assert cuda_lib.dn_step_error(layer.m._h, s.cuda_stream) == 0
    finally:
        if graph.value:
            cuda_lib.dn_graph_destroy(graph)
        layer.close()
