"""The layer-list step's few-token kernels against the float64 oracle: products of up to eight rows on the tensor cores at the edges
of their tiles (dn_rows_mma.cuh).  Tolerances are those of the family's other tests: 4e-2 of the logits' spread in bf16 and 2e-4 in
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
