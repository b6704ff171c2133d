"""Prompt portions of the delta rule in chunks of 32 tokens (k_delta_chunk; entries of 80 tokens and more, key sizes 64 and 128) beside
token-by-token entries in the same step, against the float64 oracle and against the same tokens in portions that all go token by token."""
from __future__ import annotations

import pytest
import torch

from tests.test_gpu_seqmix import FF, TOL, Rig, config, delta, err, toks

pytestmark = pytest.mark.gpu

# key size, value size, heads, key heads: two blocks of columns with a ragged second one; one block, not full; more heads a key head than a block of the
# preparation takes at once; blocks of 64 columns (56 x 2 of them a step of one entry)
SHAPES = [(128, 96, 4, 2), (128, 40, 3, 3), (64, 128, 10, 1), (64, 20, 2, 1), (128, 128, 56, 4)]


@pytest.mark.parametrize("dk,dv,heads,groups", SHAPES)
def test_chunks_against_the_oracle_and_token_by_token(dk, dv, heads, groups):
    """First portions that end inside, on and behind the edge of a chunk; entries below the line beside them; second portions that start from the first's state."""
    cfg = config([delta(mixer={"heads": heads, "kv_heads": groups, "dim": dk, "vdim": dv, "conv": 3}, mlp=FF),
                  delta(mixer={"heads": heads, "kv_heads": groups, "dim": dk, "vdim": dv, "conv": 0})], width=64)
    seqs = [toks(n, seed=300 + i) for i, n in enumerate((161, 210, 86, 260))]
    first = [80, 97, 81, 79]
    with Rig(cfg, "bfloat16", max_tokens=1024, max_batch_tokens=512) as r:
        parts = [r.eng.step([(f"s{i}", s[a:b], list(range(b - a))) for i, (s, a, b) in enumerate(zip(seqs, lo, hi))])
                 for lo, hi in (([0] * 4, first), (first, [len(s) for s in seqs]))]
        r.model.check()
        for i in range(4):
            r.eng.finish(f"s{i}")
        at = [0, 0]
        for i, (s, n) in enumerate(zip(seqs, first)):
            mine = torch.cat([parts[0][at[0]:at[0] + n], parts[1][at[1]:at[1] + len(s) - n]])
            at = [at[0] + n, at[1] + len(s) - n]
            assert err(mine, r.oracle(s)) < TOL["bfloat16"], f"request {i}"
            # the recurrence's sums differ by a few 1e-8, which bf16 rounds away but for a place in a thousand
            small = torch.cat([r.eng.step([("c", s[a:a + 79], list(range(len(s[a:a + 79]))))]) for a in range(0, len(s), 79)])
            r.eng.finish("c")
            assert err(mine, small.cpu()) < 2e-2, f"request {i}"


def test_decays_of_zero_and_repeated_keys():
    """Decays that end a state at once (no quotient of decays may be formed) and one token over and over (keys that are all alike, so that (I + L) is full)."""
    cfg = config([delta(mixer={"heads": 2, "kv_heads": 1, "dim": 128, "vdim": 64, "conv": 0}, mlp=FF)], width=64)
    with Rig(cfg, "bfloat16", max_tokens=512) as r0:
        w = dict(r0.w)
    for A_log, tokens in ((8.0, toks(150, seed=7)), (-9.0, [5] * 150)):
        v = {k: t.clone() for k, t in w.items()}
        v["l0.mix.A_log"] = torch.full_like(v["l0.mix.A_log"], A_log)
        with Rig(cfg, "bfloat16", max_tokens=512, weights=v) as r:
            got = r.eng.step([("a", tokens, list(range(len(tokens))))])
            assert torch.isfinite(got).all()
            assert err(got, r.oracle(tokens)) < TOL["bfloat16"]
