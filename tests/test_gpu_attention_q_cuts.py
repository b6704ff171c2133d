"""k_attn_prefill_q where key heads' longest row blocks are whole and the others shared: against the CUDA-core kernel, and captured."""
from __future__ import annotations

import ctypes as C

import pytest
import torch

from tests.test_gpu_attention_bits import H, Layer
from tests.test_gpu_prefill import _agree, _call, _model

pytestmark = pytest.mark.gpu


# (kv heads, query heads a key head): one round of whole blocks and two, the last row block ragged, an odd number of shared blocks; many key heads' shares of two without whole blocks
@pytest.mark.parametrize("bits,kv_heads,group,context,T", [(8, 8, 8, 1024, 305), (4, 8, 8, 1024, 400), (8, 8, 8, 1024, 650), (8, 6, 7, 1024, 577), (4, 8, 5, 1500, 650), (8, 2, 4, 0, 1500)])
def test_against_the_cuda_core_kernel(cuda_lib, bits, kv_heads, group, context, T):
    """bounds as in test_prefill_attention_over_quantised_pages"""
    m = _model(kv_heads, group, seed=group + bits, kv_bits=bits)
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


@pytest.mark.parametrize("bits,group,T", [(8, 8, 310), (4, 8, 650)])
def test_a_captured_chunk_gives_the_bits_of_an_eager_one(cuda_lib, bits, group, T):
    """replayed at positions whose blocks are all whole, whole and shared by two"""
    n = 2200
    x = torch.randn(n + T, H, generator=torch.Generator().manual_seed(n + T)).to(torch.bfloat16).cuda()
    layer, s, graph = Layer(cuda_lib, 8, group, kv_bits=bits, max_tokens=4096), torch.cuda.Stream(), C.c_void_p()
    try:
        for at in range(0, n + T, 1500):
            layer.run(x[at:at + 1500], at)      # the cache's rows
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
