"""k_router_scored with one and with several rows a warp: steps on both sides of the line, experts that do not fill a warp's rows."""
from __future__ import annotations

import pytest

from tests.test_gpu_bokenex import TOL, Rig, att, config, err, moe, toks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,experts,top,tokens", [("float32", 35, 3, 700), ("float32", 6, 2, 1380), ("bfloat16", 17, 16, 640)])
def test_steps_of_many_tokens_choose_as_portions_do(dtype, experts, top, tokens):
    cfg = config([att(moe(experts, top, 1.3, 16))])
    t = toks(tokens, seed=experts)
    wanted = [0, 1, tokens // 2, tokens - 2, tokens - 1]
    with Rig(cfg, dtype, max_tokens=1408, max_batch_tokens=1408) as rig:
        ref = rig.oracle(t)[wanted]
        assert err(rig.eng.step([("whole", t, wanted)]), ref) < TOL[dtype]      # more tokens than blocks of a row a warp run at once
        rig.eng.finish("whole")
        got = [rig.eng.step([("cut", t[a:b], [i - a for i in wanted if a <= i < b])]) for a, b in ((0, 250), (250, tokens - 1), (tokens - 1, tokens))]
        assert err(got[0], ref[:2]) < TOL[dtype]
        assert err(got[1], ref[2:4]) < TOL[dtype]
        assert err(got[2], ref[4:]) < TOL[dtype]
