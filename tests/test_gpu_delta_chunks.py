"""Prompt portions of the delta rule in chunks of 32 tokens (k_delta_chunk; entries of 96 tokens and more with keys of 128, of 128 with keys of 64) beside
token-by-token entries in the same step, against the float64 oracle and against the same tokens in portions that all go token by token."""
from __future__ import annotations

import ctypes as C

import pytest
import torch

from dnet_b200 import _seqabi
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
    seqs = [toks(n, seed=300 + i) for i, n in enumerate((260, 300, 210, 290))]
    first = [128, 145, 129, 95]
    with Rig(cfg, "bfloat16", max_tokens=1536, max_batch_tokens=640) as r:
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


# -- the recurrence alone ---------------------------------------------------------------------------------------------
def recurrence_inputs(kind, lens, heads, groups, dk, dv, seed=0):
    """fp32 q, k (of unit length), v, beta, decay and one state an entry"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    nd = lambda *s: torch.randn(*s, generator=g, device="cuda")      # noqa: E731
    silu, N = torch.nn.functional.silu, sum(lens)
    unit = lambda x: x / (x.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()      # noqa: E731
    q, k = unit(silu(nd(N, groups, dk))) * dk ** -0.5, nd(N, groups, dk)
    beta, decay = torch.sigmoid(nd(N, heads)), torch.exp(-torch.exp(0.5 * nd(N, heads) - 1) * torch.nn.functional.softplus(nd(N, heads)))
    if kind == "long memory, keys alike":
        k, beta, decay = nd(1, groups, dk) + 0.1 * k, torch.sigmoid(3 * nd(N, heads) + 3), 1 - 1e-4 * torch.rand(N, heads, generator=g, device="cuda")
    elif kind == "decays of 0, 1e-20 and 1":
        u = torch.rand(N, heads, generator=g, device="cuda")
        decay = torch.where(u < 0.1, 0.0, torch.where(u < 0.55, 1e-20, 1.0))
    return [x.float().contiguous() for x in (q, unit(silu(k)), silu(nd(N, heads, dv)), beta, decay, 0.3 * nd(len(lens), heads, dk, dv))]


def recurrence(chunked, lens, q, k, v, beta, decay, state):
    state, out = state.clone(), torch.full_like(v, float("nan"))
    _seqabi.init(0)
    _seqabi.check(_seqabi.load().dn_seq_debug_delta(chunked, len(lens), (C.c_int32 * len(lens))(*lens), v.shape[1], k.shape[1], k.shape[2], v.shape[2],
                                                    *(x.data_ptr() for x in (q, k, v, beta, decay, state, out)), torch.cuda.current_stream().cuda_stream))
    return out, state


def recurrence64(lens, q, k, v, beta, decay, state):
    r = v.shape[1] // k.shape[1]
    q, k = (x.double().repeat_interleave(r, 1) for x in (q, k))
    v, beta, decay, state = (x.double() for x in (v, beta, decay, state))
    out, states, at = torch.empty_like(v), [], 0
    for n, S in zip(lens, state):
        for t in range(at, at + n):
            S = S * decay[t, :, None, None]
            u = beta[t, :, None] * (v[t] - torch.einsum("hdj,hd->hj", S, k[t]))
            S = S + k[t, :, :, None] * u[:, None]
            out[t] = torch.einsum("hdj,hd->hj", S, q[t])
        states.append(S)
        at += n
    return out, torch.stack(states)


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("kind,bound", [("decays of about 0.8", 8e-8), ("long memory, keys alike", 4e-7), ("decays of 0, 1e-20 and 1", 8e-8)])
@pytest.mark.parametrize("lens,heads,groups,dk,dv", [([100, 97, 96, 127, 250], 8, 2, 128, 128), ([130, 191], 4, 2, 64, 96), ([98, 113], 2, 1, 128, 40), ([1500], 5, 5, 128, 128)])
def test_recurrence_is_as_close_to_64_bits_as_token_by_token(kind, bound, lens, heads, groups, dk, dv):
    """Outputs and states in fp32 against float64, 2-norm.  A rounding leaves 2.25e-8 (2^-23 / sqrt(12) over a mantissa of 1.53 rms).  Token by token a number takes two a token,
    of which a decay of about 0.8 leaves some three tokens' in all: 6e-8 to 7.5e-8, bound 8e-8; with a long memory and keys that are alike errors add up (9e-7 and 1.2e-6 over
    1,500 tokens).  Chunks are no further off than that, but for a twentieth, the spread of such a norm over inputs, or three roundings, 4e-8, which no order of the sums goes
    below (u = beta (v - ..), k u): states that a decay of 0 has left with a token or two.  Operands of two parts, 2^-17, are a hundred times off."""
    x = recurrence_inputs(kind, lens, heads, groups, dk, dv, seed=len(lens) + dk)
    ref = recurrence64(lens, *x)
    by_token, chunks = recurrence(0, lens, *x), recurrence(1, lens, *x)
    for name, a, c, r in zip(("outputs", "states"), by_token, chunks, ref):
        assert rel(c, r) < min(bound, max(1.05 * rel(a, r), 4e-8)), (name, rel(a, r))
    assert all(torch.equal(a, b) for a, b in zip(chunks, recurrence(1, lens, *x)))


def test_recurrence_hook_refuses_what_has_no_chunks():
    x = recurrence_inputs("decays of about 0.8", [90], 2, 1, 40, 20)
    assert all(torch.isfinite(a).all() for a in recurrence(0, [90], *x))
    with pytest.raises(_seqabi.DnError, match="no chunks"):
        recurrence(1, [90], *x)


@pytest.mark.parametrize("where,value", [(w, x) for w in ("q", "k", "v", "beta", "decay", "state") for x in (float("nan"), float("-inf"))] + [("v", 2e38)])
@pytest.mark.parametrize("token", [37, 64, 95, 152])      # inside, at the edges of and in the last, ragged chunk of an entry
def test_numbers_that_are_not_finite_touch_what_they_touch_token_by_token(where, value, token):
    """One such number in an entry's 153 tokens: outputs of earlier tokens, of other columns (values and states), heads and entries are what they are without it, and what is not
    finite is the same as token by token.  A value of 2e38 is finite and stays so."""
    lens, at = [90, 153], 90 + token
    x = recurrence_inputs("decays of about 0.8", lens, 4, 2, 64, 40, seed=3)
    clean = recurrence(1, lens, *x)
    tensor = x[["q", "k", "v", "beta", "decay", "state"].index(where)]
    {"q": lambda: tensor[at, 1, 7:8], "k": lambda: tensor[at, 1, 7:8], "v": lambda: tensor[at, 2, 13:14], "beta": lambda: tensor[at, 2:3], "decay": lambda: tensor[at, 2:3],
     "state": lambda: tensor[1, 2, 11, 13:14]}[where]().fill_(value)
    by_token, chunks = recurrence(0, lens, *x), recurrence(1, lens, *x)
    for name, a, c, w in zip(("outputs", "states"), by_token, chunks, clean):
        assert torch.equal(torch.isfinite(a), torch.isfinite(c)), name
        ok = torch.isfinite(a)
        assert not ok.all() or value == 2e38 or (where, name) == ("q", "states")
        assert torch.allclose(a[ok], c[ok], rtol=1e-5, atol=1e-6 * (2e38 if value == 2e38 else 1.0)), name
    if where != "state":
        assert torch.equal(chunks[0][:at], clean[0][:at])
