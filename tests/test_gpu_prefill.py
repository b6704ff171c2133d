"""-m gpu: the kernels of a prompt chunk's layer alone, at the sizes where they can go wrong: one decoder layer of a small model through
``apply_single_layer``, against another path of the library that forms the same sums in another order.

Bound: both paths store bf16 between a layer's operations and differ in the order of fp32 sums, so a stored value may differ by its last
rounding (2^-8 relative).  A flipped rounding of one operand of the following products moves their results by far less than their own
rounding, so results agree to a few last roundings of the largest value.  How many differ at all: the attention's sums differ by some
2^-16 of their terms, which flips about p = 1 in 100 of its roundings; a product of such rows is then off by sqrt(p) 2^-9 of its size,
a tenth of the distance of two roundings, which flips one result in ten, and the feed-forward does the same once more: below a quarter
(a wrong key, row or head changes all of them)."""
import ctypes as C

import pytest
import torch

from tests.helpers import rel_inf

pytestmark = pytest.mark.gpu


def _model(kv_heads, group, seed=0, pages=48, kv_bits=0, hidden=512, ffn=512):
    from dnet_b200.core.models.llama import LlamaRingModel

    cfg = dict(hidden_size=hidden, num_attention_heads=kv_heads * group, num_key_value_heads=kv_heads, head_dim=128, intermediate_size=ffn,
               vocab_size=256, num_hidden_layers=1, rms_norm_eps=1e-5, rope_theta=10000.0, model_type="llama", torch_dtype="bfloat16")
    g = torch.Generator().manual_seed(seed)
    p = "model.layers.0."
    rows = {"q": kv_heads * group * 128, "k": kv_heads * 128, "v": kv_heads * 128}

    def t(*shape, std):
        return (torch.randn(*shape, generator=g) * std).to(torch.bfloat16).cuda()

    w = {f"{p}self_attn.{c}_proj.weight": t(n, hidden, std=(2.0 if c in "qk" else 1.0) * hidden ** -0.5) for c, n in rows.items()}
    w.update({f"{p}self_attn.{c}_proj.bias": t(n, std=0.5) for c, n in rows.items()})
    w[p + "self_attn.o_proj.weight"] = t(hidden, rows["q"], std=rows["q"] ** -0.5)
    w[p + "mlp.gate_proj.weight"], w[p + "mlp.up_proj.weight"] = t(ffn, hidden, std=hidden ** -0.5), t(ffn, hidden, std=hidden ** -0.5)
    w[p + "mlp.down_proj.weight"] = t(hidden, ffn, std=ffn ** -0.5)
    for n in ("input_layernorm", "post_attention_layernorm"):
        w[f"{p}{n}.weight"] = torch.ones(hidden, dtype=torch.bfloat16).cuda()
    m = LlamaRingModel(cfg, [0], kv_pool_pages=pages, kv_bits=kv_bits)
    m.load_weights(w)
    return m


def _call(m, kv, x, context):
    """the layer's outputs of the tokens behind `context`"""
    kv.seek(0)
    if context:
        m.apply_single_layer(0, x[:context].clone(), kv)
        kv.seek(context)
    y = m.apply_single_layer(0, x[context:].clone(), kv)
    torch.cuda.synchronize()
    return y.float().cpu()


def _agree(a, b, differing=0.25):
    assert torch.isfinite(a).all()
    assert rel_inf(a, b) <= 3 * 2.0 ** -8, rel_inf(a, b)
    assert float((a != b).float().mean()) < differing


@pytest.mark.parametrize("group", [1, 2, 4, 5, 7, 8])
@pytest.mark.parametrize("context,T", [(0, 16), (0, 127), (129, 26), (1000, 300), (2490, 16)])
def test_prefill_attention_groups_and_key_shares(cuda_lib, group, context, T):
    """k_attn_prefill_tc against the CUDA-core kernel: groups that leave MMA rows empty (5, 7), row blocks with a remainder, one key tile
    (the second side has none), tiles cut by the causal edge, and contexts whose keys the CTAs of a cluster share (few tokens far back)."""
    m = _model(2, group, seed=group)
    kv = m.make_cache(max_tokens=2560)
    x = torch.randn(context + T, 512, generator=torch.Generator().manual_seed(T)).to(torch.bfloat16).cuda()
    out = {}
    try:
        for tc in (1, 0):
            cuda_lib.dn_set_option(b"tc_attn", tc)
            out[tc] = _call(m, kv, x, context)
        assert cuda_lib.dn_step_error(m._h, 0) == 0
    finally:
        cuda_lib.dn_set_option(b"tc_attn", 1)
        kv.free()
        m.destroy()
    _agree(out[1], out[0])


@pytest.mark.parametrize("group,context,T", [(1, 0, 1), (1, 63, 32), (2, 127, 8), (2, 128, 16), (4, 0, 3), (4, 2552, 8), (4, 500, 4), (5, 1300, 6), (7, 255, 2), (8, 2400, 4)])
def test_attention_of_a_few_tokens(cuda_lib, group, context, T):
    """k_attn_few against the CUDA-core kernel: one and two tiles of 16 rows, whole and ragged, one key tile (no partial outputs), page and tile edges
    inside the new tokens, more key tiles than CTAs of a key head."""
    m = _model(8 if context > 2500 else 2, group, seed=group)
    kv = m.make_cache(max_tokens=2560)
    x = torch.randn(context + T, 512, generator=torch.Generator().manual_seed(T)).to(torch.bfloat16).cuda()
    out = {}
    try:
        for tc in (1, 0):
            cuda_lib.dn_set_option(b"tc_attn", tc)
            out[tc] = _call(m, kv, x, context)
        assert cuda_lib.dn_step_error(m._h, 0) == 0
    finally:
        cuda_lib.dn_set_option(b"tc_attn", 1)
        kv.free()
        m.destroy()
    _agree(out[1], out[0])


@pytest.mark.parametrize("hidden,ffn,kv_heads,group,T", [(256, 8192, 2, 1, 17), (256, 8192, 2, 1, 45), (768, 1280, 1, 2, 65), (1024, 14336, 2, 4, 129),
                                                         (512, 2048, 2, 2, 300), (768, 27648, 1, 4, 512)])
def test_prefill_products_widths_splits_and_segments(cuda_lib, hidden, ffn, kv_heads, group, T):
    """k_gemm_tc (tiles of a CTA pair) against the row kernels: features and tokens that leave part of a tile empty, q, k and v in one launch
    with fewer rows than a tile, reductions shared by the pairs of a cluster, widths of 64 to 256 tokens, last tiles cut narrower."""
    x = torch.randn(T, hidden, generator=torch.Generator().manual_seed(T)).to(torch.bfloat16).cuda()
    out = {}
    try:
        for tc in (1, 0):
            cuda_lib.dn_set_option(b"tc_prefill", tc)
            m = _model(kv_heads, group, seed=T, hidden=hidden, ffn=ffn)
            assert m.max_prefill_chunk == (512 if tc else 0)
            kv = m.make_cache(max_tokens=576)
            out[tc] = _call(m, kv, x, 0)
            assert cuda_lib.dn_step_error(m._h, 0) == 0
            kv.free()
            m.destroy()
    finally:
        cuda_lib.dn_set_option(b"tc_prefill", 1)
    _agree(out[1], out[0])


@pytest.mark.parametrize("hidden,ffn,T", [(1024, 14336, 17), (2048, 8192, 33), (2048, 8192, 48), (1024, 14336, 64), (768, 8192, 129), (2048, 8192, 250)])
def test_prefill_products_of_single_ctas(cuda_lib, hidden, ffn, T):
    """k_gemm_tc where few tokens meet long reductions, against the row kernels: single CTAs and pairs as the plan takes them, one token tile to six."""
    x = torch.randn(T, hidden, generator=torch.Generator().manual_seed(T)).to(torch.bfloat16).cuda()
    out = {}
    try:
        for tc in (1, 0):
            cuda_lib.dn_set_option(b"tc_prefill", tc)
            m = _model(2, 2, seed=T, hidden=hidden, ffn=ffn)
            kv = m.make_cache(max_tokens=576)
            out[tc] = _call(m, kv, x, 0)
            assert cuda_lib.dn_step_error(m._h, 0) == 0
            kv.free()
            m.destroy()
    finally:
        cuda_lib.dn_set_option(b"tc_prefill", 1)
    _agree(out[1], out[0])


SINGLE = [("gate_up", 512, 2048, 2, 65, (48, 1)), ("o", 4864, 512, 1, 193, (80, 1)), ("down", 4352, 3072, 2, 97, (64, 2)), ("down", 2048, 2048, 2, 65, (48, 3)),
          ("down", 4096, 4096, 2, 17, (64, 4)), ("down", 4096, 8192, 2, 100, (128, 4))]


@pytest.mark.parametrize("product,hidden,ffn,kv_heads,T,plan", SINGLE)
def test_prefill_products_that_one_cta_a_tile_forms(cuda_lib, product, hidden, ffn, kv_heads, T, plan):
    """Every width and split that k_gemm_tc takes with one CTA a tile, by the plan that the library reports for the product (with the clusters that the plans
    rest on; a device that runs another number of them may plan otherwise), against the row kernels."""
    qd = 2 * kv_heads * 128
    rows, K = {"o": ([hidden], qd), "gate_up": ([ffn], hidden), "down": ([hidden], ffn)}[product]
    out = (C.c_int32 * 5)()
    assert cuda_lib.dn_debug_gemm_plan((C.c_int32 * len(rows))(*rows), len(rows), product == "gate_up", T, K, out) == 0
    assert list(out)[:3] == [1, *plan] or list(out)[3:] != [33, 15], list(out)
    x = torch.randn(T, hidden, generator=torch.Generator().manual_seed(T)).to(torch.bfloat16).cuda()
    got = {}
    try:
        for tc in (1, 0):
            cuda_lib.dn_set_option(b"tc_prefill", tc)
            m = _model(kv_heads, 2, seed=T, hidden=hidden, ffn=ffn)
            kv = m.make_cache(max_tokens=576)
            got[tc] = _call(m, kv, x, 0)
            assert cuda_lib.dn_step_error(m._h, 0) == 0
            kv.free()
            m.destroy()
    finally:
        cuda_lib.dn_set_option(b"tc_prefill", 1)
    _agree(got[1], got[0])


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("group,context,T", [(4, 0, 16), (1, 0, 130), (2, 100, 29), (5, 129, 64), (7, 1000, 40), (8, 2490, 16), (4, 1500, 512)])
def test_prefill_attention_over_quantised_pages(cuda_lib, bits, group, context, T):
    """k_attn_prefill_q against the CUDA-core kernel on the same pages: both widths of code, groups with empty rows, tiles cut by the causal
    edge, shares of a cluster.  Scores and probabilities are rounded to bf16 in both, so a score whose sum lies near an edge may flip: a
    weight is then off by 2^-8 of itself, less than what the stored outputs may be."""
    m = _model(2, group, seed=group + bits, kv_bits=bits)
    kv = m.make_cache(max_tokens=2560)
    x = torch.randn(context + T, 512, generator=torch.Generator().manual_seed(T)).to(torch.bfloat16).cuda()
    out = {}
    try:
        for tc in (1, 0):
            cuda_lib.dn_set_option(b"tc_attn", tc)
            out[tc] = _call(m, kv, x, context)
        assert cuda_lib.dn_step_error(m._h, 0) == 0
    finally:
        cuda_lib.dn_set_option(b"tc_attn", 1)
        kv.free()
        m.destroy()
    _agree(out[1], out[0])


@pytest.mark.parametrize("bits", [0, 8, 4])
@pytest.mark.parametrize("T", [2, 3, 7, 8, 9, 15, 16, 17])
@pytest.mark.parametrize("hidden,ffn,kv_heads,group,context", [(256, 512, 1, 2, 0), (768, 27648, 2, 5, 63), (4096, 1280, 2, 4, 700)])
def test_chunks_of_a_few_tokens(cuda_lib, hidden, ffn, kv_heads, group, context, T, bits):
    """A chunk of 2 .. 16 tokens in one pass over the weights (k_rows: one or two groups of eight tokens, warps with few columns and with
    many) against the same tokens one by one on the kernels of a model without tensor-core prompts (k_gemv, k_attn or k_attn_q); 17 tokens
    are the first that the GEMM takes.
    The row kernels form every product's sums in another order too, so that the flipped roundings start in q, k and v and grow from product
    to product.  Where every operand of the last one differs in its last place the result is off by 2^-9 / sqrt(3) of its size times sqrt(2),
    three quarters of a place at the most frequent sizes: about half of the results are stored differently.  Over quantised pages a
    score near a rounding edge flips by 2^-8 of itself, and its weight with it, which moves every result of its token by up to a rounding,
    half of them over an edge.  So below a half either way (a wrong weight, row or head changes nearly all, and by more)."""
    x = torch.randn(context + T, hidden, generator=torch.Generator().manual_seed(T)).to(torch.bfloat16).cuda()
    out = {}
    try:
        for tc in (1, 0):
            cuda_lib.dn_set_option(b"tc_prefill", tc)
            m = _model(kv_heads, group, seed=hidden, hidden=hidden, ffn=ffn, kv_bits=bits)
            kv = m.make_cache(max_tokens=768)
            if tc:
                out[tc] = _call(m, kv, x, context)
            else:
                assert cuda_lib.dn_model_max_chunk_forward(m._h) == 0      # (the row kernels)
                rows = []
                kv.seek(0)
                if context:
                    m.apply_single_layer(0, x[:context].clone(), kv)
                for t in range(context, context + T):
                    kv.seek(t)
                    rows.append(m.apply_single_layer(0, x[t:t + 1].clone(), kv))
                torch.cuda.synchronize()
                out[tc] = torch.cat(rows).float().cpu()
            assert cuda_lib.dn_step_error(m._h, 0) == 0
            kv.free()
            m.destroy()
    finally:
        cuda_lib.dn_set_option(b"tc_prefill", 1)
    _agree(out[1], out[0], 0.5)


@pytest.mark.parametrize("bits,group,hidden,ffn,T", [(0, 4, 512, 2048, 513), (8, 2, 512, 512, 1029), (0, 5, 768, 1280, 2048), (4, 1, 256, 512, 2050)])
def test_one_chunk_of_up_to_2048_tokens(cuda_lib, bits, group, hidden, ffn, T):
    """a prompt in chunks of 2,048 tokens and what is left over (more rows than a launch of 512, staging pages of a whole chunk, two tokens
    behind the last full one) against the same prompt in chunks of 512"""
    kv_heads = 2
    x = torch.randn(T, hidden, generator=torch.Generator().manual_seed(T)).to(torch.bfloat16).cuda()
    m = _model(kv_heads, group, seed=T, hidden=hidden, ffn=ffn, kv_bits=bits)
    kv = m.make_cache(max_tokens=2560)
    try:
        whole = _call(m, kv, x, 0)
        parts = []
        for t in range(0, T, 512):
            kv.seek(t)
            parts.append(m.apply_single_layer(0, x[t:t + 512].clone(), kv))
        torch.cuda.synchronize()
        assert cuda_lib.dn_step_error(m._h, 0) == 0
    finally:
        kv.free()
        m.destroy()
    _agree(whole, torch.cat(parts).float().cpu(), 0.5 if bits else 0.25)      # (quantised pages: as above)


@pytest.mark.parametrize("T", [1, 4])
def test_the_scratch_hook_reads_the_last_chunk(cuda_lib, T):
    """dn_debug_scratch after a chunk, whichever kernels it ran on: the rotated queries, the attention's output, the residual and the
    SwiGLU output of the chunk itself (a few last roundings of the row kernels')"""
    import torch as t

    hidden, ffn, heads = 512, 768, 4
    x = t.randn(70 + T, hidden, generator=t.Generator().manual_seed(T)).to(t.bfloat16).cuda()
    got = {}
    try:
        for tc in (1, 0):
            cuda_lib.dn_set_option(b"tc_prefill", tc)
            m = _model(2, 2, seed=5, hidden=hidden, ffn=ffn)
            kv = m.make_cache(max_tokens=128)
            _call(m, kv, x, 70)
            for which, n in enumerate((heads * 128, heads * 128, hidden, ffn)):
                host = t.empty(T, n, dtype=t.bfloat16)
                assert cuda_lib.dn_debug_scratch(m._h, which, host.data_ptr(), host.numel() * 2, 0) == 0
                got[tc, which] = host.float()
            kv.free()
            m.destroy()
    finally:
        cuda_lib.dn_set_option(b"tc_prefill", 1)
    for which in range(4):
        assert rel_inf(got[1, which], got[0, which]) <= 4 * 2.0 ** -8, which
