"""The layer-list step's few-token kernels against the float64 oracle: products of up to eight rows on the tensor cores at the edges
of their tiles (dn_rows_mma.cuh), and what lies between two sublayers (k_turn, the mixers' convolutions).  Tolerances are those of the family's other tests: 4e-2 of the logits' spread in bf16 and 2e-4 in
fp32 (test_gpu_seqmix.py)."""
from __future__ import annotations

import pytest

from .test_gpu_seqmix import TOL, Rig, attn, config, delta, err, run_schedule, toks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width, ff, vocab", [
    (96, 224, 160),        # every product's columns in 32s
    (160, 176, 7121),      # the down product's columns are not (the row kernel); many features, 17 over a multiple of 32
    (2048, 4096, 7103),    # every warp of a block has columns; one feature below the wider blocks
])
def test_products_of_one_to_eight_tokens(width, ff, vocab):
    cfg = config([attn(mixer={"heads": 6, "kv_heads": 2, "dim": 16, "vdim": 16, "conv": 3}, mlp={"kind": "dense", "ff": ff}),
                  delta(mlp={"kind": "dense", "ff": ff})], streams=2, width=width, vocab=vocab)
    t = toks(39, vocab=vocab, seed=7)
    with Rig(cfg, "bfloat16") as rig:
        ref = rig.oracle(t)
        assert err(run_schedule(rig, t, [1, 2, 3, 4, 5, 6, 7, 8]), ref) < TOL["bfloat16"]
        assert rig.model.check() is None


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("streams, conv, width", [
    (0, 0, 48), (0, 4, 64), (1, 1, 128), (2, 2, 36), (4, 3, 264), (4, 4, 1024),
    (3, 4, 4096), (2, 3, 4100),      # the widest row of the joined kernel and the next one
    (5, 4, 64), (8, 5, 64),          # more streams and more taps than the joined kernels take
    (2, 3, 50),                      # rows that are not whole groups of four
])
def test_between_two_sublayers(dtype, streams, conv, width):
    """the write-back of one sublayer, the norm of the next and the mixers' convolutions: whole prompts and steps of one to three tokens"""
    mx = {"conv": conv, "rot": {"base": 50.0, "dims": 12}}
    cfg = config([attn(mixer={"heads": 4, "kv_heads": 2, "dim": 16, "vdim": 24, **mx}, mlp={"kind": "dense", "ff": 96}),
                  delta(mixer={"heads": 4, "kv_heads": 2, "dim": 16, "vdim": 16, "conv": conv}, mlp={"kind": "dense", "ff": 96}),
                  attn(mixer={"heads": 3, "kv_heads": 1, "dim": 10, "vdim": 7, "conv": conv, "rot": {"base": 50.0, "dims": 4}})],
                 streams=streams, width=width)
    t = toks(30, seed=11)
    with Rig(cfg, dtype) as rig:
        ref = rig.oracle(t)
        assert err(run_schedule(rig, t, [30]), ref) < TOL[dtype]
        assert err(run_schedule(rig, t, [17, 1, 3, 1, 2]), ref) < TOL[dtype]
        last = rig.eng.step([("w", t, [0, 29])])      # two rows wanted: the streams of the others end unread
        rig.eng.finish("w")
        assert err(last, ref[[0, 29]]) < TOL[dtype]
