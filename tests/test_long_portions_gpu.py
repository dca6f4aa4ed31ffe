"""The recurrent mixers as parts in steps that hold long portions: those go through the kernels that take 64 tokens at a time, the
requests beside them are walked in order."""

import pytest
import torch

from tests import helpers as H
from tests.plain import koduzen_plain, makisun_plain, tebivik_plain, vofusun_plain
from tests.test_tebivik_gpu import _close, _ctx

pytestmark = pytest.mark.gpu
DEV = "cuda"
DTYPES = [("float32", torch.float32, 2e-5), ("bfloat16", torch.bfloat16, 3e-2)]  # the parts' own tests state the same


def _mixer(kind, dtype, Hh, dk, dv, D):
    """(part, its plain form for one sequence), with weights of their own."""
    from jax_llm_examples_b200.parts import HGRN2, GatedDeltaRule, GatedLinearAttention, RetentionMixer, TimeMixWKV, rotary_frequencies

    g = lambda *s: torch.randn(*s) * 0.3  # noqa: E731
    m, eps, F = {"heads": Hh, "dim": dk, "vdim": dv}, 1e-5, Hh * dk
    qkvg = {"q": g(F, D), "k": g(F, D), "v": g(Hh * dv, D), "g": g(Hh * dv, D), "norm": 1 + 0.2 * torch.randn(dv), "o": g(D, Hh * dv)}
    if kind == "gated":
        m["tau"] = 8.0
        w = {**qkvg, "a1": g(6, D), "a2": g(F, 6), "a2.b": g(F) + 2.0}
    elif kind == "time_mix":
        w = {**{"mu." + s: torch.rand(D) for s in "rkvgw"}, **{s: g(F, D) for s in "rkvg"}, "w1": g(6, D), "w2": g(F, 6), "w0": g(F) - 1.0,
             "u": g(Hh, dk), "norm": 1 + 0.2 * torch.randn(F), "o": g(D, F)}
    elif kind.startswith("retention"):
        m["decay"] = [0.99, 0.9, 1.0, 0.97][:Hh]
        if kind == "retention turned":
            m["rot"] = {"base": 10000.0, "dims": 64}
        w = {k: v for k, v in qkvg.items() if k != "norm"}
    elif kind == "hgrn2":
        w = {"q": g(F, D), "f": g(F, D), "v": g(Hh * dv, D), "f.b": g(F), "lower": torch.rand(F), "norm": 1 + 0.2 * torch.randn(dv), "o": g(D, Hh * dv)}
    else:
        G, taps = 1, 4
        m.update(kv_heads=G, conv=taps)
        w = {**qkvg, "q": g(G * dk, D), "k": g(G * dk, D), "b": g(Hh, D), "a": g(Hh, D), "q.conv": g(G * dk, taps), "k.conv": g(G * dk, taps),
             "v.conv": g(Hh * dv, taps), "A_log": g(Hh), "dt_bias": g(Hh)}
    w = {k: v.to(dtype) for k, v in w.items()}
    P, d = {"m." + k: v.double() for k, v in w.items()}, lambda k: w[k].to(DEV)  # noqa: E731
    if kind == "gated":
        return (GatedLinearAttention(torch.cat([d(s) for s in "qkvg"]), d("a1"), d("a2"), d("a2.b"), d("norm"), d("o"), Hh, dk, dv, m["tau"], eps),
                lambda s: makisun_plain.gated_linear_attention(s, P, "m.", m, eps))
    if kind == "time_mix":
        return (TimeMixWKV(torch.stack([d("mu." + s) for s in "rkvgw"]), torch.stack([d(s) for s in "rkvg"]), d("w1"), d("w2"), d("w0"), d("u"),
                           d("norm"), d("o"), Hh, dk, eps), lambda s: makisun_plain.wkv_mixer(s, P, "m.", m, eps))
    if kind.startswith("retention"):
        rot = m.get("rot")
        return (RetentionMixer(torch.cat([d(s) for s in "qkvg"]), d("o"), torch.tensor(m["decay"], device=DEV), Hh, dk, dv, eps, k_scale=dk ** -0.5,
                               inv_freq=rotary_frequencies(rot["base"], rot["dims"]).to(DEV) if rot else None, rot_dims=rot["dims"] if rot else 0),
                lambda s: koduzen_plain.retention_mixer(s, P, "m.", m, eps))
    if kind == "hgrn2":
        return (HGRN2(torch.cat([d("q"), d("f"), d("v")]), d("f.b"), d("lower"), d("norm"), d("o"), Hh, dk, dv, eps),
                lambda s: tebivik_plain.hgrn2(s, P, "m.", m, eps))
    return (GatedDeltaRule(torch.cat([d(s) for s in "qkvgba"]), torch.cat([d(s + ".conv") for s in "qkv"]), d("A_log"), d("dt_bias"), d("norm"), d("o"),
                           Hh, m["kv_heads"], dk, dv, eps), lambda s: vofusun_plain.delta_mixer(s, P, "m.", m, eps))


def _run(mixer, dtype, seqs, steps, slots, states, planners):
    """Feeds (request, first, end) portions step by step; the outputs per request."""
    from jax_llm_examples_b200.parts import LayerCache, Runtime

    rt, got = Runtime(dtype, torch.device(DEV)), [[] for _ in seqs]
    for step in steps:
        rows = torch.cat([seqs[r][lo:hi] for r, lo, hi in step]).to(DEV)
        ctx = _ctx(rt, [hi - lo for _, lo, hi in step], [lo for _, lo, _ in step], [slots[r] for r, _, _ in step], planners=planners)
        cache = LayerCache(None, None, False, states[0], states)
        f32_rows = mixer.needs_f32_input or type(mixer).__name__ == "HGRN2"
        out = H.as_rows_sum(mixer.forward(ctx, None, cache, h32=rows.float()) if f32_rows else mixer.forward(ctx, rows, cache))
        o = 0
        for r, lo, hi in step:
            got[r].append(out[o:o + hi - lo])
            o += hi - lo
    return [torch.cat(g) for g in got]


# a long portion alone; beside a single token and a portion one short of long; from a carried state beside others; two at once (the two
# heads of these parts are worth the chunk kernels from 1024 tokens on, or so far ahead of the rest)
STEPS = [[(0, 0, 1100)], [(0, 1100, 1101), (1, 0, 1430), (2, 0, 383)], [(2, 383, 384), (0, 1101, 1110), (1, 1430, 2500)], [(0, 1110, 2140), (1, 2500, 2884)]]
KINDS = ["gated", "time_mix", "retention", "retention turned", "hgrn2", "delta"]


@pytest.mark.parametrize("name, dtype, tol", DTYPES)
@pytest.mark.parametrize("kind, dk, dv", [(k, 128, 128) for k in KINDS] + [("gated", 70, 100), ("time_mix", 70, 70), ("retention turned", 72, 128),
                                                                        ("hgrn2", 70, 100), ("hgrn2", 127, 65), ("delta", 72, 100)])
def test_steps_with_long_portions_beside_others(kind, dk, dv, name, dtype, tol, monkeypatch):
    """Against the plain recurrence over the whole sequences, and against the same tokens walked in order (a step without the
    planner's lists); a slot of no request stays as it is."""
    from jax_llm_examples_b200.kernels import api as K

    torch.manual_seed(dk + len(kind))
    mixer, plain = _mixer(kind, dtype, 2, dk, dv, 40)
    seqs = [torch.randn(n, 40).to(dtype) for n in (2140, 2884, 384)]
    ref = [plain(s.double()) for s in seqs]
    got = {}
    ran = []
    for name_of in ("chunk_scan", "delta_chunk"):
        real = getattr(K, name_of)
        monkeypatch.setattr(K, name_of, lambda *a, real=real, **k: (ran.append(1), real(*a, **k)))
    for planned in (True, False):
        states = tuple(torch.zeros(5, *n.shape, device=DEV) for n in mixer.state_needs())
        for s in states:
            s[1] = 99.0
        got[planned] = _run(mixer, dtype, seqs, STEPS, [4, 0, 2], states, mixer.step_planners() if planned else ())
        assert len(ran) == 4  # every step, once
        for r in range(3):
            _close(got[planned][r], ref[r], tol, f"{name} request {r} planned={planned}")
        assert all(torch.equal(s[1], torch.full_like(s[1], 99.0)) for s in states)
    for r in range(3):
        _close(got[True][r], got[False][r], 1e-5 if dtype == torch.float32 else 2e-2, f"{name} request {r}: in chunks against in order")


@pytest.mark.parametrize("splits", [1, 2])
@pytest.mark.parametrize("dk, dv", [(128, 128), (70, 100)])
@pytest.mark.parametrize("lens", [[450], [64, 1, 450, 384]])
def test_hgrn2_kernels_with_chunks_from_partial_sums(splits, dk, dv, lens):
    """The projections in parts, or whole (then the values are read where they lie), alone and beside requests that are walked;
    the chunks against the walk over the same rows: two orders of sums over up to 450 tokens in float32, 1e-5."""
    from jax_llm_examples_b200.kernels import api as K
    from jax_llm_examples_b200.parts.base import StepShape
    from jax_llm_examples_b200.parts.recurrent import CHUNK_FROM_TOKENS, plan_scan_chunks

    torch.manual_seed(splits)
    Hh, N, R = 2, sum(lens), len(lens)
    i32 = lambda v: torch.tensor(v, device=DEV, dtype=torch.int32)  # noqa: E731
    qfv = torch.randn(splits, N, Hh * (2 * dk + dv), device=DEV)
    qfv = qfv if splits > 1 else qfv[0]
    bias, lower, norm = torch.randn(Hh * dk, device=DEV), torch.rand(Hh * dk, device=DEV), torch.rand(dv, device=DEV) + 0.5
    plan = {k: i32(v.reshape(-1).tolist()) for k, v in plan_scan_chunks(StepShape(tuple(lens), (0,) * R, 16, max(lens))).items()}
    long = [n for n in lens if n >= CHUNK_FROM_TOKENS]
    ch = K.Chunks(plan["scan_chunks"], plan["scan_chunk_requests"], plan["scan_chunks"].numel() // 3, len(long), CHUNK_FROM_TOKENS, len(long) < R)
    state = torch.randn(R + 1, Hh, dk, dv, device=DEV)
    walked, out, want = state.clone(), torch.empty(N, Hh * dv, device=DEV), torch.empty(N, Hh * dv, device=DEV)
    before = qfv.clone()
    common = (i32([sum(lens[:r]) for r in range(R + 1)]), i32(list(range(R, 0, -1))), norm, 1e-5)
    K.hgrn2_scan(qfv, splits, bias, lower, state, *common, out, Hh, dk, dv, chunks=ch,
                 chunk_scratch=torch.empty(K.chunk_scan_scratch(ch.n, Hh, dk, dv), device=DEV))
    K.hgrn2_scan(qfv, splits, bias, lower, walked, *common, want, Hh, dk, dv)
    _close(out, want, 1e-5, "outputs")
    _close(state, walked, 1e-5, "states")
    assert torch.equal(state[0], walked[0]) and torch.equal(qfv, before)


def _off(t):
    """The same numbers one entry behind a 16-byte boundary."""
    moved = torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view_as(t)
    assert moved.data_ptr() % 16
    return moved


def test_a_decays_bias_off_16_byte_boundaries():
    """Long portions of a gated linear attention take it as ever, whatever of q, k and v is left in place."""
    torch.manual_seed(7)
    mixer, _ = _mixer("gated", torch.float32, 2, 128, 128, 40)
    seqs, steps, outs = [torch.randn(1150, 40)], [[(0, 0, 1100)], [(0, 1100, 1150)]], []
    for bias in (mixer.a_bias, _off(mixer.a_bias)):
        mixer.a_bias = bias
        states = tuple(torch.zeros(2, *n.shape, device=DEV) for n in mixer.state_needs())
        outs.append(_run(mixer, torch.float32, seqs, steps, [1], states, mixer.step_planners())[0])
    _close(outs[1], outs[0], 1e-5)


def test_states_of_the_delta_rule_off_16_byte_boundaries():
    """The kernels for long portions read and write states entry by entry: slabs may start anywhere, as for the walk."""
    torch.manual_seed(7)
    mixer, _ = _mixer("delta", torch.float32, 2, 128, 128, 40)
    seqs, steps, outs = [torch.randn(1150, 40)], [[(0, 0, 1100)], [(0, 1100, 1150)]], []
    for place in (lambda s: s, _off):
        states = tuple(place(torch.zeros(2, *n.shape, device=DEV)) for n in mixer.state_needs())
        outs.append(_run(mixer, torch.float32, seqs, steps, [1], states, mixer.step_planners())[0])
    _close(outs[1], outs[0], 1e-5)
