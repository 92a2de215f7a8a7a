"""The device sampling chain against the oracle's restatement of the reference's decode crate
(crates/decode/src/processors.rs, sampler.rs, chain.rs), row by row, at the decoder vocabulary size.
Temperature, top-k and the repetition penalty are bit-exact; top-p, min-p and the multinomial walk sum
probabilities in a different order than the reference's sequential sums, so a token exactly at a cut
may differ: any difference must sit at the cut (checked on the probabilities in float64)."""
import numpy as np
import pytest
import torch

import oracle_lib as O
from gpu_util import DEV
from logismos_b200 import sampling as S
from logismos_b200.ops import InvalidOp

pytestmark = pytest.mark.gpu
V = 151936


def rows(seed, n_rows=5, n=V, scale=3.0):
    rng = np.random.default_rng(seed)
    x = (rng.standard_normal((n_rows, n)) * scale).astype(np.float32)
    x[1] = np.round(x[1] * 2) / 2          # a row full of ties
    x[2, : n // 2] = -np.inf               # a row half masked by an earlier processor
    return x


def probs64(row):
    r = row.astype(np.float64)
    e = np.where(np.isfinite(r), np.exp(r - r[np.isfinite(r)].max()), 0.0)
    return e / e.sum()


def run(proc, x):
    t = torch.from_numpy(x.copy()).to(DEV)
    proc.process(t)
    torch.cuda.synchronize()
    return t.cpu().numpy()


def test_temperature_top_k_and_repetition_penalty_are_bit_exact():
    x = rows(1)
    for t in (0.7, 1.0, 0.0, 2.5):
        got = run(S.TemperatureScale(t), x)
        for r in range(x.shape[0]):
            assert np.array_equal(got[r], O.temperature(x[r], t), equal_nan=True)
    xn = x.copy(); xn[0, 5] = np.nan; xn[3, 77] = np.nan
    for k in (1, 2, 50, 1000, V - 1, V, 0):
        got = run(S.TopK(k), xn)
        for r in range(x.shape[0]):
            assert np.array_equal(got[r], O.top_k(xn[r], k), equal_nan=True), (k, r)
    rng = np.random.default_rng(2)
    toks = rng.integers(0, V, (x.shape[0], 40)).astype(np.uint32)
    toks[0, 3] = toks[0, 2]; toks[1, 0] = V + 5   # listed twice; outside the vocabulary
    counts = np.array([40, 7, 0, 40, 13], np.int32)
    xr = x.copy(); xr[2] = np.abs(xr[4])  # finite rows
    got = run(S.RepetitionPenalty(torch.from_numpy(toks.view(np.int32)).to(DEV), torch.from_numpy(counts).to(DEV), 1.3), xr)
    for r in range(x.shape[0]):
        assert np.array_equal(got[r], O.repetition_penalty(xr[r], toks[r, : counts[r]], 1.3)), r


SUM_TOL = 1e-3  # the reference normalises by, and accumulates, SEQUENTIAL fp32 sums over up to 151936 terms: its own cut sits 1e-4..3e-4 (relative) off the exact one


@pytest.mark.parametrize("p", [0.05, 0.5, 0.9, 0.999, 1.0, 0.0])
def test_top_p_keeps_the_reference_nucleus(p):
    """Both nuclei are prefixes of the same order (descending probability, ties by index). They may differ
    in length only where the cumulative mass (float64) is within the reference's own summation error of p:
    its softmax divides by a sequential fp32 sum, the device sums pairwise."""
    x = rows(3)
    got = run(S.TopP(p), x)
    for r in range(x.shape[0]):
        ref = O.top_p(x[r], p)
        kg, kr = np.isfinite(got[r]), np.isfinite(ref)
        assert np.array_equal(got[r][kg], x[r][kg])  # kept logits are untouched
        if np.array_equal(kg, kr):
            continue
        pr = probs64(x[r])
        order = np.argsort(-pr, kind="stable")
        cum = np.cumsum(pr[order])
        ng, nr = int(kg.sum()), int(kr.sum())
        assert kg[order[:ng]].all() and kr[order[:nr]].all(), (p, r)   # both are prefixes of the order
        lo, hi = sorted((ng, nr))
        assert cum[lo - 1] >= p * (1 - SUM_TOL) and cum[hi - 2] <= p * (1 + SUM_TOL), (p, r, ng, nr, cum[lo - 1], cum[hi - 2])


@pytest.mark.parametrize("p", [0.001, 0.05, 0.5, 1.0, 0.0])
def test_min_p_masks_the_reference_tail(p):
    x = rows(4)
    got = run(S.MinP(p), x)
    for r in range(x.shape[0]):
        ref = O.min_p(x[r], p)
        diff = np.flatnonzero(np.isfinite(got[r]) != np.isfinite(ref))
        if diff.size:
            pr = probs64(x[r])
            thr = min(max(p, 0.0), 1.0) * pr.max()
            assert np.all(np.abs(pr[diff] - thr) <= 1e-5 * thr), (p, r, diff[:5])


def test_multinomial_returns_the_reference_token_for_the_same_draw():
    x = rows(5, n_rows=6)
    x[5] = -np.inf; x[5, 1234] = 0.5     # all the mass on one token
    x[4] = -np.inf                       # no mass at all: greedy, which returns index 0
    rng = np.random.default_rng(6)
    t = torch.from_numpy(x).to(DEV)
    sampler = S.MultinomialSampler(seed=1)
    for trial in range(6):
        u = rng.random(6).astype(np.float32)
        if trial == 0:
            u[:] = [0.0, 0.999999, 0.5, 1e-7, 0.3, 0.9]
        got = sampler.sample(t, uniforms=torch.from_numpy(u).to(DEV)).cpu().numpy().view(np.uint32)
        for r in range(6):
            ref = O.multinomial(x[r], float(u[r]))
            if got[r] != ref:
                cdf = np.cumsum(probs64(x[r]))
                lo, hi = sorted((int(got[r]), ref))
                assert cdf[hi - 1] - cdf[lo] <= SUM_TOL and abs(cdf[lo] - u[r]) <= SUM_TOL, (trial, r, got[r], ref)
    # seeded draws are reproducible (sampler.rs:72-82)
    a = S.MultinomialSampler(seed=42); b = S.MultinomialSampler(seed=42)
    for _ in range(4):
        assert torch.equal(a.sample(t), b.sample(t))


def test_chain_runs_processors_in_order_then_samples():  # chain.rs:33-76, :88-121
    x = rows(7)
    base = torch.from_numpy(x.copy()).to(DEV)
    chain = S.DecodeChain(S.GreedySampler()).push(S.TemperatureScale(0.8)).push(S.TopK(50)).push(S.TopP(0.95))
    assert len(chain) == 3 and not chain.is_empty()
    toks = chain.step(base).cpu().numpy().view(np.uint32)
    for r in range(x.shape[0]):
        ref = O.top_p(O.top_k(O.temperature(x[r], 0.8), 50), 0.95)
        assert toks[r] == O.greedy(ref)
        assert np.isfinite(base[r].cpu().numpy()).sum() <= 50 + (x[r] == np.sort(x[r])[-50]).sum()
    # a peaked small row, the reference's own example: cooling then top-p keeps only index 0
    small = torch.tensor([[3.0, 2.9, 2.8, 2.7]], dtype=torch.float32, device=DEV)
    c2 = S.DecodeChain(S.GreedySampler()).push(S.TemperatureScale(0.1)).push(S.TopP(0.5))
    assert int(c2.step(small)[0]) == 0 and torch.isinf(small[0, 1:]).all()
    with pytest.raises(InvalidOp):
        S.TopK(5).process(torch.zeros((2, 8)))  # CPU tensor: no CPU arm


@pytest.mark.parametrize("n", [1, 2, 31, 1000, 2047, 2048, 8195, 33000, 151937])
def test_edges_of_the_slices_of_a_row(n):
    """Rows below and above the length from which eight CTAs share one, lengths that leave rows unaligned and slices ragged or
    empty; survivors that fit the list of a CTA and that do not; ties at the cut in several slices; NaN and infinities.
    Top-k is bit-exact; the nucleus and the draw differ only where the mass (float64) lies within SUM_TOL of the cut."""
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((6, n)) * 3.0).astype(np.float32)
    x[1] = np.round(x[1]) + 0.0                   # ties everywhere (and one zero)
    x[2, rng.random(n) < 0.9] = -np.inf
    x[3] = 0.25                                   # one value: all of them tie
    x[4, n // 2] = np.nan
    x[5, -1] = np.inf
    for k in sorted({1, 2, 40, n // 2, n - 1}):
        got = run(S.TopK(k), x)
        for r in range(6):
            assert np.array_equal(got[r], O.top_k(x[r], k), equal_nan=True), (k, r)
    for p in (0.0, 0.3, 0.95):
        got = run(S.TopP(p), x)
        for r in range(6):
            if r == 3:  # equal probabilities: the first ceil(p n), give or take the one that fp32 rounding of 1 / n moves
                kept = np.flatnonzero(got[r] > -np.inf)
                assert abs(kept.size - max(np.ceil(p * n), 1)) <= 1 and kept[-1] == kept.size - 1, (p, kept.size)
                continue
            if r == 4 and n > 1:  # a NaN leaves the probabilities unnormalised: the maximum alone has mass one
                assert np.array_equal(np.flatnonzero(got[r] > -np.inf), [np.nanargmax(x[r])]), p
                continue
            if r >= 4:            # no probability that is a number: everything is kept
                assert np.array_equal(got[r], x[r], equal_nan=True), (p, r)
                continue
            ref = O.top_p(x[r], p)
            kg, kr = got[r] > -np.inf, ref > -np.inf
            pr = probs64(x[r]) if np.isfinite(x[r]).any() else np.zeros(n)
            order = np.argsort(-pr, kind="stable")
            ng, nr = int(kg.sum()), int(kr.sum())
            assert kg[order[:ng]].all() and kr[order[:nr]].all(), (p, r)
            if ng != nr:
                cum, (lo, hi) = np.cumsum(pr[order]), sorted((ng, nr))
                assert cum[lo - 1] >= p * (1 - SUM_TOL) and cum[max(hi - 2, 0)] <= p * (1 + SUM_TOL), (p, r, ng, nr)
    t = torch.from_numpy(x).to(DEV)
    for u in (0.0, 0.37, 0.999):
        got = S.MultinomialSampler(seed=1).sample(t, uniforms=torch.full((6,), u, device=DEV)).cpu().numpy().view(np.uint32)
        for r in range(6):
            ref = O.multinomial(x[r], u)
            if got[r] != ref:
                pr = np.where(np.isfinite(x[r]), probs64(x[r]), 0.0)
                cdf, (lo, hi) = np.cumsum(pr), sorted((int(got[r]), ref))
                assert cdf[hi - 1] - cdf[lo] <= SUM_TOL and abs(cdf[lo] - u) <= SUM_TOL, (u, r, got[r], ref)


@pytest.mark.parametrize("n,k", [(151936, 50), (151936, 3), (33000, 7), (1500, 4)])
def test_a_draw_never_falls_on_a_value_without_mass(n, k):
    """After a top-k nearly every value is -inf. Draws of zero, just above zero, on and just above every survivor's cumulative mass and just
    below one land on a survivor, and on the one whose interval holds the draw: bounds in float64, 1e-5 for fp32 sums of normalised masses
    (pairwise within a part, at most 64 parts)."""
    rng = np.random.default_rng(n + k)
    x = (rng.standard_normal(n) * 3.0).astype(np.float32)
    x[np.argsort(x)[:-k]] = -np.inf
    pr = probs64(x)
    cdf = np.cumsum(pr)
    edges = cdf[pr > 0]
    u = np.concatenate([[0.0, 1e-7, 1e-6, 2.0 ** -24, 1 - 2.0 ** -24, 1 - 2.0 ** -23, 1 - 1e-6]] + [edges[:-1] + d for d in (0.0, 6e-8, 3e-7, 1e-6, 1.9e-6, -3e-7)])
    u = np.clip(u, 0.0, 1 - 2.0 ** -24).astype(np.float32)
    t = torch.from_numpy(x).to(DEV).expand(u.size, n).contiguous()
    got = S.MultinomialSampler(seed=1).sample(t, uniforms=torch.from_numpy(u).to(DEV)).cpu().numpy().view(np.uint32).astype(np.int64)
    assert (pr[got] > 0).all(), [(float(a), int(b)) for a, b in zip(u[pr[got] == 0], got[pr[got] == 0])][:5]
    assert (u <= cdf[got] + 1e-5).all() and (u >= cdf[got] - pr[got] - 1e-5).all()


def test_results_do_not_change_between_runs():
    """Survivors of an earlier processor lie in lists whose order changes from run to run; sums over them must not. Min-p at the very bound:
    values whose probability equals p of the largest up to the rounding of exp and of the sum, beside 6000 others, in 64 rows."""
    rng = np.random.default_rng(3)
    x = np.full((64, V), -np.inf, np.float32)
    for r in range(64):
        at = rng.choice(V, 6000, replace=False)
        x[r, at] = rng.uniform(-9.0, -1.5, 6000)
        x[r, at[0]] = 0.0
        x[r, at[1:9]] = -1.0
    p = np.float32(np.exp(np.float32(-1.0)))
    t = torch.from_numpy(x).to(DEV)
    others = torch.empty(64 << 20, device=DEV)
    for ulps in range(-3, 5):
        q = (p.view(np.int32) + np.int32(ulps)).view(np.float32)
        first = None
        for i in range(30):
            y = t.clone()
            if i & 1:
                others.fill_(i)  # rows from memory, not from L2: other warps come first
            S.MinP(float(q)).process(y)
            first = y if first is None else first
            assert torch.equal(y, first)


@pytest.mark.parametrize("n", [262080, 262200, 600001, 4000003])
def test_top_p_of_long_rows_keeps_small_probabilities(n):
    """Rows of equal values, each of probability 1 / n: the nucleus is the first ceil(p n), within the rounding of 1 / n in fp32 (2^-24) and
    of the unit that masses are counted in (2^-41 n = 1.2e-7 at most); and rows of random values against float64 at the same bound."""
    t = torch.full((2, n), 0.25, device=DEV)
    rng = np.random.default_rng(n)
    x = (rng.standard_normal(n) * 2.0).astype(np.float32)
    t[1] = torch.from_numpy(x).to(DEV)
    for p in (0.3, 0.95):
        y = t.clone()
        S.TopP(p).process(y)
        kept = torch.isfinite(y[0]).sum().item()
        assert abs(kept - np.ceil(p * n)) <= 2e-7 * n + 1, (p, kept, p * n)
        keep = np.isfinite(y[1].cpu().numpy())
        pr = probs64(x)
        m = pr[keep].sum()
        assert p * (1 - 2e-6) <= m <= p * (1 + 2e-6) + pr[keep].min(), (p, m)


def _apart(chain, x, u):
    """The chain's processors one by one and the draw from the uniforms u."""
    t = torch.from_numpy(x.copy()).to(DEV)
    for p in chain.processors:
        p.process(t)
    return t, S.MultinomialSampler(seed=1).sample(t, uniforms=u)


@pytest.mark.parametrize("n", [2, 5, 255, 300, 1500, 2047, 2048, 2050, 8195, 33001, 151936, 262150])
@pytest.mark.parametrize("k", [1, 2, 50, 256, 257])
def test_a_chain_in_one_launch_leaves_what_its_processors_leave(n, k):
    """Temperature, top-k, top-p, min-p and draw as one launch against one launch each: the same survivors to the bit. Rows of random values, of few values (more ties
    at the cut than the launch lists), of one value, with fewer finite values than k, with NaN and infinities, with the largest values side by side, all -inf; rows that
    start off a 16-byte boundary (odd n). k below, at and above the largest that the launch takes. Draws may differ where both lie within 1e-5 of the draw
    in the survivors' cumulative mass (fp32 sums of at most 512 normalised masses in another order)."""
    rng = np.random.default_rng([n, k])
    x = (rng.standard_normal((9, n)) * 3.0).astype(np.float32)
    x[1] = np.round(x[1]) + 0.0
    x[2] = 0.25
    x[3, rng.random(n) < 0.995] = -np.inf
    x[4, :: 3] = np.nan
    x[5, n // 2] = np.inf
    x[5, -1] = np.inf
    x[6] = np.sort(x[6])
    x[7] = -np.inf
    x[8] *= 1e-3
    u = torch.from_numpy(rng.random(9).astype(np.float32)).to(DEV)
    for t, p, m in ((1.0, 1.0, 0.0), (0.8, 0.95, 0.0), (1.7, 0.3, 0.02), (1e-7, 0.0, 0.5), (0.7, 1.0, 0.1)):
        chain = S.DecodeChain(S.MultinomialSampler(seed=1)).push(S.TemperatureScale(t)).push(S.TopK(k)).push(S.TopP(p)).push(S.MinP(m))
        ref, ref_tokens = _apart(chain, x, u)
        got, tokens = torch.from_numpy(x.copy()).to(DEV), torch.empty(9, dtype=torch.int32, device=DEV)
        S.check(S.lib.logismos_launch_sample_chain_f32(S._p(got), 9, n, *chain._settings(), S._p(u), S._p(tokens), S._stream()), "sample_chain")
        assert torch.equal(got.view(torch.int32), ref.view(torch.int32)), (t, p, m, (got.view(torch.int32) != ref.view(torch.int32)).nonzero()[:5])
        for r in (tokens != ref_tokens).nonzero().flatten().tolist():
            row = got[r].double().cpu().numpy()
            cdf, (a, b) = np.cumsum(np.where(np.isfinite(row), probs64(row), 0.0)), sorted((int(tokens[r]), int(ref_tokens[r])))
            assert np.isfinite(row[a]) and np.isfinite(row[b]) and abs(cdf[a] - float(u[r])) <= 1e-5 and cdf[b - 1] - cdf[a] <= 1e-5, (t, p, m, r)
        chain.sampler = S.MultinomialSampler(seed=5)
        stepped = torch.from_numpy(x.copy()).to(DEV)
        drawn = chain.step(stepped)
        v = torch.rand(9, generator=S.MultinomialSampler(seed=5).gen, device=DEV, dtype=torch.float32)
        S.check(S.lib.logismos_launch_sample_chain_f32(S._p(got.copy_(torch.from_numpy(x))), 9, n, *chain._settings(), S._p(v), S._p(tokens), S._stream()), "sample_chain")
        assert torch.equal(stepped.view(torch.int32), ref.view(torch.int32)) and torch.equal(drawn, tokens)


def _apart_by_the_oracle(chain, x, u):
    """As _apart with top-k by the oracle: as a processor it would be the launch under test again where that takes its k."""
    t = torch.from_numpy(x.copy()).to(DEV)
    for p in chain.processors:
        if isinstance(p, S.TopK):
            t = torch.from_numpy(np.stack([O.top_k(row, p.k) for row in t.cpu().numpy()])).to(DEV)
        else:
            p.process(t)
    return t, S.MultinomialSampler(seed=1).sample(t, uniforms=u)


@pytest.mark.parametrize("n,k", [(n, k) for n in (2, 5, 255, 300, 1500, 2047, 2048, 2050, 8195, 33001, 151936, 262150) for k in (1, 2, 50, 256, 257)] +
                         # the largest k of the launch with top-p and without, and the next one
                         [(300, 28), (300, 29), (300, 42), (300, 43), (2047, 83), (2047, 84), (2047, 144), (2047, 145), (2048, 84), (2048, 85), (2048, 168), (2048, 169), (33001, 144), (33001, 145)])
def test_a_chain_in_one_launch_keeps_the_top_k_of_the_oracle(n, k, monkeypatch):
    """The test above, its rows and bounds, with the survivors of top-k from the oracle."""
    monkeypatch.setitem(globals(), "_apart", _apart_by_the_oracle)
    test_a_chain_in_one_launch_leaves_what_its_processors_leave(n, k)


def test_chains_of_another_shape_run_one_launch_per_processor():
    m = S.MultinomialSampler
    for chain in (S.DecodeChain(S.GreedySampler()).push(S.TopK(3)), S.DecodeChain(m(1)).push(S.TopP(0.9)), S.DecodeChain(m(1)).push(S.TopK(3)).push(S.TemperatureScale(0.5)),
                  S.DecodeChain(m(1)).push(S.TopK(3)).push(S.TopK(2)), S.DecodeChain(m(1)).push(S.TopK(-1)), S.DecodeChain(m(1)).push(S.TopK(3)).push(S.TypicalSampling(0.5)), S.DecodeChain(m(1))):
        assert chain._settings() is None
    assert S.DecodeChain(m(1)).push(S.TopK(3))._settings() == [1.0, 3, 1.0, 0.0]
