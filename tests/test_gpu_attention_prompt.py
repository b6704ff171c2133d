"""k_attn_prompt: items dealt out whole, one and several a CTA, and runs that cut items; against the CUDA-core kernel, 64 bits and the layer-list oracle."""
from __future__ import annotations

import ctypes as C

import pytest
import torch

from tests.test_gpu_attention_bits import H, Layer, beyond_rounding, exact
from tests.test_gpu_prefill import _agree, _call, _model
from tests.test_gpu_seqmix import FF, TOL, Rig, attn, config, delta, err, toks

pytestmark = pytest.mark.gpu


# (kv heads, query heads a key head): two parts of a weight for groups of 1, 2, 4 and 8, three for 5 and 7.  One item a CTA (the launch's last row block ragged); several a
# CTA; few long items, cut into runs (three pieces of an item and more); a row block whose last key tile is one page
@pytest.mark.parametrize("kv_heads,group,context,T", [(8, 4, 0, 300), (8, 1, 129, 1200), (3, 8, 0, 1111), (8, 2, 63, 900), (8, 4, 2100, 290), (6, 4, 2490, 513),
                                                      (8, 5, 0, 126), (8, 5, 64, 1000), (4, 7, 1000, 200), (8, 7, 2600, 100), (8, 5, 2000, 500)])
def test_against_the_cuda_core_kernel(cuda_lib, kv_heads, group, context, T):
    m = _model(kv_heads, group, seed=group)
    kv = m.make_cache(max_tokens=3072)
    x = torch.randn(context + T, 512, generator=torch.Generator().manual_seed(T)).to(torch.bfloat16).cuda()
    out = {}
    try:
        for tc in (1, 0):
            cuda_lib.dn_set_option(b"tc_attn", tc)
            out[tc] = _call(m, kv, x, context)
            if tc:      # the counts of finished pieces are zero again
                assert torch.equal(out[1], _call(m, kv, x, context))
        assert cuda_lib.dn_step_error(m._h, 0) == 0
    finally:
        cuda_lib.dn_set_option(b"tc_attn", 1)
        kv.free()
        m.destroy()
    _agree(out[1], out[0])


@pytest.mark.parametrize("kv_heads,group,context,T,eps", [(8, 4, 700, 290, 2.0 ** -16), (8, 5, 900, 130, 2.0 ** -18), (4, 7, 0, 400, 2.0 ** -18)])
def test_against_64_bits(cuda_lib, kv_heads, group, context, T, eps):
    """bounds as in test_attention_over_16_bit_pages"""
    x = torch.randn(context + T, H, generator=torch.Generator().manual_seed(context + T)).to(torch.bfloat16).cuda()
    layer = Layer(cuda_lib, kv_heads, group)
    try:
        k, v = layer.rows(x)
        q, got = layer.attend(x, context)
    finally:
        layer.close()
    ref, spread, total = exact(q, k, v, context, group)
    assert bool((beyond_rounding(got, ref) <= eps * spread + 2.0 ** -22 * total).all())


@pytest.mark.parametrize("kv_heads,group,T", [(8, 4, 300), (8, 5, 130)])
def test_a_captured_chunk_gives_the_bits_of_an_eager_one(cuda_lib, kv_heads, group, T):
    """replayed at positions whose items are dealt out whole and cut"""
    n = 2600
    x = torch.randn(n + T, H, generator=torch.Generator().manual_seed(n + T)).to(torch.bfloat16).cuda()
    layer, s, graph = Layer(cuda_lib, kv_heads, group, max_tokens=4096), torch.cuda.Stream(), C.c_void_p()
    try:
        for at in range(0, n + T, 1500):
            layer.run(x[at:at + 1500], at)
        torch.cuda.synchronize()
        buf, ids = torch.empty(T, H, dtype=torch.bfloat16, device="cuda"), (C.c_int32 * 1)(0)
        assert cuda_lib.dn_graph_begin(s.cuda_stream) == 0
        assert cuda_lib.dn_chunk_forward(layer.m._h, ids, 1, buf.data_ptr(), T, layer.kv._h, s.cuda_stream) == 0
        assert cuda_lib.dn_graph_end(s.cuda_stream, C.byref(graph)) == 0
        for at in (0, 1100, n):
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
    finally:
        if graph.value:
            cuda_lib.dn_graph_destroy(graph)
        layer.close()


BASE = {"dim": 128, "vdim": 128, "scale": 0.4}


@pytest.mark.parametrize("heads,kv_heads,mask", [(4, 1, None), (4, 2, 200), (3, 1, 64), (6, 6, 333), (14, 2, None)])
def test_layer_list_attention(heads, kv_heads, mask):
    """Ragged entries beside single tokens: block masks that cut tiles, keys of another layer, no mask; portions that start inside a page and inside a block; steps above
    and below the line from which the kernel is taken."""
    mx = {**BASE, "heads": heads, "kv_heads": kv_heads, "conv": 2, "rot": {"base": 500.0, "dims": 32}}
    if mask:
        mx["mask"] = {"size": mask}
    cfg = config([attn(mixer=mx, mlp=FF), attn(mixer={**mx, "kv_from": 0}), delta()], width=64)
    seqs = [toks(n, seed=500 + i) for i, n in enumerate((461, 300, 90, 215))]
    cuts = [[0, 161, 461], [0, 1, 300], [0, 89, 90], [0, 200, 215]]
    with Rig(cfg, "bfloat16", max_tokens=2048, max_batch_tokens=1024) as r:
        got = [[] for _ in seqs]
        for step in range(2):
            lg = r.eng.step([(f"s{i}", s[c[step]:c[step + 1]], list(range(c[step + 1] - c[step]))) for i, (s, c) in enumerate(zip(seqs, cuts))])
            at = 0
            for i, c in enumerate(cuts):
                got[i].append(lg[at:at + c[step + 1] - c[step]])
                at += c[step + 1] - c[step]
        r.model.check()
        for i, s in enumerate(seqs):
            assert err(torch.cat(got[i]), r.oracle(s)) < TOL["bfloat16"], f"request {i}"


# -- items that are cut, several a CTA, and more row blocks than are sorted ---------------------------------------------------------
def dealt_or_cut(entries, kv_heads, group, first_seen):
    """how a step's row blocks go over the SMs, from the rule as k_attn_prompt has it: "several" whole items a CTA, "cut" into runs (the most pieces an item comes to), or
    "unsorted" runs of more row blocks than are sorted"""
    sms, TB = torch.cuda.get_device_properties(0).multi_processor_count, 128 // group
    lens = []
    for pos, n in entries:
        for i in range(0, n, TB):
            end = pos + i + min(TB, n - i)
            lens.append(((end + 63) // 64 - first_seen(pos + i) // 64 + 1) // 2 + 1)
    items, total = kv_heads * len(lens), kv_heads * sum(lens)
    per = max(-(-total // sms), 4)
    if len(lens) > 256:
        return "unsorted"
    order = sorted(lens, reverse=True)
    load = [0] * sms
    for i in range(items):
        k, c = divmod(i, sms)
        load[sms - 1 - c if k & 1 else c] += order[i // kv_heads]
    return "cut" if max(load) > per + 6 else "several" if items > sms else "whole"


def twice(rig, steps):
    """the same steps two times over, with fresh sequences: the last one's logits"""
    runs = []
    for _ in range(2):
        runs.append([rig.eng.step(s) for s in steps][-1])
        rig.model.check()
        for rid in {e[0] for s in steps for e in s}:
            rig.eng.finish(rid)
    assert torch.equal(*runs)      # (the counts of finished pieces are zero again, too)
    return runs[0]


@pytest.mark.parametrize("how,heads,kv_heads,mask,first,portions", [
    ("cut", 4, 1, None, (0, 3, 333), (2000, 1, 40)), ("cut", 4, 1, 1500, (700, 0, 61), (1300, 90, 1)), ("several", 16, 8, None, (0, 100, 0), (1400, 17, 1)),
    ("unsorted", 16, 1, 700, (0, 0, 65), (2100, 33, 9))])
def test_layer_list_items_cut_and_joined(how, heads, kv_heads, mask, first, portions):
    """a long portion beside short ones: their tiles are on the line that runs are cut from, and a run may end in any of them"""
    mx = {**BASE, "heads": heads, "kv_heads": kv_heads, "conv": 2, "rot": {"base": 500.0, "dims": 32}}
    if mask:
        mx["mask"] = {"size": mask}
    assert dealt_or_cut(list(zip(first, portions)), kv_heads, heads // kv_heads, lambda p: p // mask * mask if mask else 0) == how
    seqs = [toks(a + n, seed=700 + i) for i, (a, n) in enumerate(zip(first, portions))]
    with Rig(config([attn(mixer=mx, mlp=FF)], width=64), "bfloat16", max_tokens=6144, max_batch_tokens=2304) as r:
        steps = [[(f"s{i}", s[:a], []) for i, (s, a) in enumerate(zip(seqs, first)) if a], [(f"s{i}", s[a:], list(range(len(s) - a))) for i, (s, a) in enumerate(zip(seqs, first))]]
        got, at = twice(r, [s for s in steps if s]), 0
        for i, (s, a) in enumerate(zip(seqs, first)):
            assert err(got[at:at + len(s) - a], r.oracle(s)[a:]) < TOL["bfloat16"], f"request {i}"
            at += len(s) - a


def test_layer_list_items_cut_under_a_sliding_window():
    """a window that starts inside pages: row blocks whose first page is not the sequence's, groups of three (126 of 128 rows), one key head"""
    from tests.test_gpu_bokenex import Rig as FamilyRig, made_up, random_for, rms1p

    size, heads, W = 1500, 3, 64
    cls = made_up("TestWindowSoftmax", {"norm": "rms", "qk_norm": False, "mask": "window"})
    cfg = {"architecture": "TestWindowSoftmax", "vocab": 96, "width": W, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
           "layers": [{"type": "attention", "mixer": {**BASE, "heads": heads, "kv_heads": 1, "mask": {"size": size}}, "mlp": {"kind": "dense", "ff": 80}}]}
    w = random_for(cls, cfg, 71)
    assert dealt_or_cut([(0, 2200), (0, 60)], 1, heads, lambda p: max(0, p - size + 1)) == "cut"
    t = toks(2200, seed=72)
    d = {k: v.double() for k, v in w.items()}
    x = d["embed"][t]
    h = rms1p(x, d["l0.norm1"], 1e-5)
    q, k, v = (h @ d[f"l0.mix.{c}"].T for c in "qkv")
    i = torch.arange(len(t))
    seen = (i[None] <= i[:, None]) & (i[None] > i[:, None] - size)
    s = torch.einsum("thd,nd->htn", q.view(-1, heads, 128), k) * BASE["scale"]
    a = torch.softmax(s.masked_fill(~seen, float("-inf")), -1) @ v
    x = x + a.transpose(0, 1).reshape(len(t), -1) @ d["l0.mix.o"].T
    h = rms1p(x, d["l0.norm2"], 1e-5)
    x = x + (torch.nn.functional.gelu(h @ d["l0.mlp.gate"].T, approximate="tanh") * (h @ d["l0.mlp.up"].T)) @ d["l0.mlp.down"].T
    ref = rms1p(x, d["final.norm"], 1e-5) @ d["head"].T
    with FamilyRig(cfg, "bfloat16", weights=w, max_tokens=4096, max_batch_tokens=2304) as r:
        got = twice(r, [[("a", t, list(range(len(t)))), ("b", t[:60], [59])]])
    assert err(got[:-1], ref) < TOL["bfloat16"]
    assert err(got[-1:], ref[59:60]) < TOL["bfloat16"]
