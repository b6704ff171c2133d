"""-m gpu: layer-list models whose tensors lie at any address.  A checkpoint's tensors may be views into one flat buffer, where a scalar
in front leaves the next one on an odd element: the kernels then read them a number at a time, with the same results."""
from types import SimpleNamespace

import pytest
import torch

from tests import test_gpu_bokenex as bokenex
from tests import test_gpu_filinex as filinex
from tests import test_gpu_lutesun as lutesun
from tests import test_gpu_seqmix as moputar
from tests import test_gpu_tuguvik as tuguvik
from tests import test_gpu_vulanex as vulanex

pytestmark = pytest.mark.gpu

# latent attention with head sizes of the tensor-core products between heads and latent space, no routers
lutesun_dense = SimpleNamespace(**{**vars(lutesun), "FULL": lutesun.config([lutesun.lat(lutesun.DENSE), lutesun.lat(None, heads=2, dim=8, kv_rank=24)])})


def at_an_odd_element(t: torch.Tensor) -> torch.Tensor:
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:] = t.reshape(-1)
    return flat[1:].view(t.shape)


def move(model, names):
    model.load_weights({k: at_an_odd_element(model._bound[k]) for k in names})
    torch.cuda.synchronize()      # (the copies ran on torch's stream, the steps run on the engine's)


def logits(rig, tokens):
    """a prompt and a few single tokens behind it"""
    out = rig.eng.step([("r", tokens[:40], list(range(40)))])
    for t in tokens[40:]:
        out = torch.cat([out, rig.eng.step([("r", [t], [0])])])
    rig.eng.finish("r")
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("family,names", [(bokenex, ["embed"]), (bokenex, ["pos"]), (vulanex, ["embed"]), (vulanex, ["bigram"])])
def test_embedding_tables(cuda_lib, family, names, dtype):
    """the token, position and bigram tables: sums of single numbers, so the streams are the same bit for bit; a head that is the embedding
    table itself goes to another kernel, whose fp32 sums of 48 terms run in another order (48 x 2^-24 of the largest, and as much again)"""
    tokens = family.toks(44)
    with family.Rig(family.FULL, dtype) as rig:
        here = logits(rig, tokens)
        move(rig.model, names)
        there = logits(rig, tokens)
    assert torch.isfinite(there).all()
    assert float((here - there).abs().max()) <= 2 * 48 * 2.0 ** -24 * float(here.abs().max())


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("family", [moputar, bokenex, vulanex])
def test_query_and_key_norms(family, dtype):
    """weights of the q / k norms behind convolutions and rotations (over the whole projection and per head): products of single numbers,
    the same bit for bit, as the heads' kernels and the blocks' form them"""
    tokens = family.toks(44)
    with family.Rig(family.FULL, dtype) as rig:
        here = logits(rig, tokens)
        names = [k for k in rig.model._bound if k.endswith((".q.norm", ".k.norm"))]
        assert names
        move(rig.model, names)
        there = logits(rig, tokens)
    assert torch.isfinite(there).all()
    if family is moputar:
        assert torch.equal(here, there)
    else:      # (the kernel of single heads asks for aligned weights: another one forms the sums of squares in another order)
        assert family.err(there, here.cpu()) <= family.TOL[dtype]


@pytest.mark.parametrize("family,dtype", [(f, "float32") for f in (bokenex, filinex, lutesun, moputar, tuguvik, vulanex)] +
                         [(f, "bfloat16") for f in (moputar, tuguvik, vulanex)] + [(lutesun_dense, "bfloat16")])
def test_every_tensor(family, dtype):
    """all tensors on odd elements against the same ones where they were: no operand may go to TMA or to wide loads, so the products' sums
    run in another order (the bound of the families' own tests; 16-bit models without routers, whose choices could tip)"""
    tokens = family.toks(44)
    with family.Rig(family.FULL, dtype) as rig:
        here = logits(rig, tokens)
        move(rig.model, list(rig.model._bound))
        there = logits(rig, tokens)
    assert torch.isfinite(there).all()
    assert family.err(there, here.cpu()) <= family.TOL[dtype]
