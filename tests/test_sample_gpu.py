"""The step after the LM head: greedy token choice on the device against Sampler::sample with temperature <= 0
(rusty-loader/src/tokenizer.rs:151-158: the last of equal maxima, 0 for an empty row)."""
import numpy as np
import pytest

from rusty_b200 import DType, UnifiedTensor

pytestmark = pytest.mark.gpu


def _run(ctx, engine, logits):
    M, N = logits.shape
    t = UnifiedTensor.new(ctx, logits, [M, N])
    idx = UnifiedTensor.from_bytes_with_dtype(ctx, np.full(M, 0xFFFFFFFF, np.uint32), [M * 4], DType.U8)
    val = UnifiedTensor.new(ctx, np.full(M, np.nan, np.float32), [M])
    engine.argmax_rows(ctx, t, idx, val)
    return idx.to_bytes(ctx).view(np.uint32), val.to_vec(ctx)


@pytest.mark.parametrize("M,N", [(1, 1), (1, 10), (3, 1000), (5, 1025), (32, 128256)])
def test_random_rows(ctx, engine, oracle, M, N):
    logits = np.random.default_rng(M * 31 + N).standard_normal((M, N)).astype(np.float32)
    idx, val = _run(ctx, engine, logits)
    want = np.array([oracle.greedy_sample(r) for r in logits], np.uint32)
    assert np.array_equal(idx, want)
    assert np.array_equal(val, logits[np.arange(M), want])


def test_ties_nan_and_infinities(ctx, engine, oracle):
    N = 5000
    rng = np.random.default_rng(0)
    rows = []
    r = rng.standard_normal(N).astype(np.float32)
    r[[7, 1500, 4999]] = 9.0                      # three equal maxima: the last wins
    rows.append(r)
    r = np.full(N, -np.inf, np.float32)            # all -inf: still "the last maximum"
    rows.append(r)
    r = rng.standard_normal(N).astype(np.float32)
    r[100] = np.nan
    r[200] = np.inf
    rows.append(r)
    rows.append(np.full(N, np.nan, np.float32))    # no candidate at all: 0
    r = np.zeros(N, np.float32)
    r[0] = 1.0                                      # maximum in the first column
    rows.append(r)
    logits = np.stack(rows)
    idx, val = _run(ctx, engine, logits)
    want = [oracle.greedy_sample(x) for x in logits]
    assert idx.tolist() == want == [4999, N - 1, 200, 0, 0]
    assert val[0] == 9.0 and val[1] == -np.inf and val[2] == np.inf and val[3] == -np.inf and val[4] == 1.0


def test_top_k_shader_differs_only_in_the_tie_rule(oracle):
    """k = 1 of the WGSL top_k takes the FIRST of equal maxima; the sampler takes the last (documented in the header)."""
    x = np.array([1.0, 5.0, 3.0, 5.0, 2.0], np.float32)
    assert oracle.top_k(x, 3).tolist() == [1, 3, 2] and oracle.greedy_sample(x) == 3


# ---- k > 1: WGSL `top_k` (rusty-backend/src/kernels.wgsl:168-188) for every row ----
def _topk(ctx, engine, logits, k):
    M, N = logits.shape
    t = UnifiedTensor.new(ctx, logits, [M, N])
    idx = UnifiedTensor.from_bytes_with_dtype(ctx, np.full(M * k, 0xFFFFFFFF, np.uint32), [M * k * 4], DType.U8)
    val = UnifiedTensor.new(ctx, np.full(M * k, np.nan, np.float32), [M, k])
    engine.top_k(ctx, t, idx, k, out_val=val)
    return idx.to_bytes(ctx).view(np.uint32).reshape(M, k), val.to_vec(ctx).reshape(M, k)


@pytest.mark.parametrize("M,N,k", [(1, 10, 3), (3, 1000, 50), (5, 1025, 1), (32, 128256, 50), (2, 2000, 1024), (4, 40, 64),
                                   (150, 333, 8)])
def test_top_k_random_rows_match_the_shader(ctx, engine, oracle, M, N, k):
    logits = np.random.default_rng(M * 31 + N + k).standard_normal((M, N)).astype(np.float32)
    idx, val = _topk(ctx, engine, logits, k)
    for m in range(M):
        want = oracle.top_k(logits[m], k)
        assert np.array_equal(idx[m], want), (m, idx[m][:8], want[:8])
        kk = min(k, N)
        assert np.array_equal(val[m, :kk], logits[m, want[:kk]])
        assert np.all(np.isneginf(val[m, kk:]))


def test_top_k_ties_nan_and_thresholds(ctx, engine, oracle):
    N, k = 6000, 40
    rng = np.random.default_rng(1)
    rows = []
    rows.append(np.round(rng.standard_normal(N) * 4).astype(np.float32))      # heavy ties: integers in about -16..16
    rows.append(np.full(N, 2.5, np.float32))                                  # all equal: the first k indices
    r = rng.standard_normal(N).astype(np.float32)
    r[::3] = np.nan
    r[5] = np.inf
    r[77] = -np.inf
    rows.append(r)
    r = np.full(N, -2e9, np.float32)                                          # nothing above the shader's -1e9 start value ...
    r[[10, 4000, 4001]] = [1.0, -5e8, 1.0]                                    # ... but three
    rows.append(r)
    r = rng.standard_normal(N).astype(np.float32)
    r[[3, 9]] = [0.0, -0.0]                                                   # the two zeros compare equal
    r[r > 0] = -r[r > 0]
    rows.append(r)
    rows.append(np.full(N, np.nan, np.float32))                               # no candidate at all
    logits = np.stack(rows)
    idx, val = _topk(ctx, engine, logits, k)
    for m in range(logits.shape[0]):
        assert np.array_equal(idx[m], oracle.top_k(logits[m], k)), m
    assert np.array_equal(idx[1], np.arange(k, dtype=np.uint32))
    assert np.array_equal(idx[3][:4], np.array([10, 4001, 4000, 0], np.uint32))
    assert np.all(idx[5] == 0) and np.all(np.isneginf(val[5]))


def test_top_k_argument_errors(ctx, engine):
    from rusty_b200 import BackendError
    t = UnifiedTensor.zeros(ctx, [2, 16])
    idx = UnifiedTensor.from_bytes_with_dtype(ctx, np.zeros(8, np.uint32), [32], DType.U8)
    for k in (0, 1025):
        with pytest.raises(BackendError) as e:
            engine.top_k(ctx, t, idx, k)
        assert e.value.kind == "InvalidDimensions"
    with pytest.raises(BackendError) as e:
        engine.top_k(ctx, t, idx, 8)          # 2 x 8 indices do not fit 32 bytes
    assert e.value.kind == "InvalidDimensions"


# ---- temperature / top-p with the device's top-k and soft-max statistics ----
def test_softmax_stats_rows(ctx, engine):
    rng = np.random.default_rng(5)
    M, N = 6, 50000
    logits = (rng.standard_normal((M, N)) * 3).astype(np.float32)
    logits[1, ::7] = np.nan
    logits[2, 100] = 40.0
    t = UnifiedTensor.new(ctx, logits, [M, N])
    mx, sm = UnifiedTensor.empty(ctx, [M]), UnifiedTensor.empty(ctx, [M])
    for temp in (0.7, 1.0, 2.5):
        engine.softmax_stats(ctx, t, temp, mx, sm)
        got_mx, got_sm = mx.to_vec(ctx), sm.to_vec(ctx)
        want_mx = np.nanmax(logits, axis=1)
        want_sm = np.nansum(np.exp((logits.astype(np.float64) - want_mx[:, None]) / temp), axis=1)
        assert np.array_equal(got_mx, want_mx)
        assert np.max(np.abs(got_sm - want_sm) / want_sm) < 2e-6
    from rusty_b200 import BackendError
    with pytest.raises(BackendError) as e:
        engine.softmax_stats(ctx, t, 0.0, mx, sm)
    assert e.value.kind == "InvalidOperation"


def test_device_assisted_nucleus_sampling_matches_the_host_sampler(ctx, engine):
    """Same draws, same tokens: k pairs and two floats per row leave the device instead of the whole vocabulary; a row
    whose nucleus is longer than k takes the host path over its logits."""
    from rusty_b200.sampler import Sampler
    rng = np.random.default_rng(9)
    M, N = 8, 32000
    logits = (rng.standard_normal((M, N)) * 4).astype(np.float32)
    logits[3] *= 0.02                       # nearly flat row: the nucleus holds thousands of tokens -> host path
    t = UnifiedTensor.new(ctx, logits, [M, N])
    for temp, top_p in ((0.7, 0.9), (1.0, 0.5), (0.0, 0.9)):
        draws = [float(v) for v in rng.random(M)]
        it = iter(draws)
        got = Sampler(temp, top_p, rand=lambda: next(it)).sample_rows_from_device(ctx, engine, t, k=64)
        it2 = iter(draws)
        host = Sampler(temp, top_p, rand=lambda: next(it2))
        want = [host.sample(logits[m]) for m in range(M)]
        assert got == want, (temp, top_p, got, want)


@pytest.mark.parametrize("M,N,k", [(1, 16384, 1), (2, 16387, 1024), (40, 4096, 64), (3, 70001, 200), (1, 2, 1)])
def test_rows_cut_over_a_cluster(ctx, engine, oracle, M, N, k):
    """Slices of a row on several blocks: edges of the slices, unaligned rows, more ties at the k-th value than the
    shortcut takes, all large logits side by side; arg-max, top-k and the host's candidates agree with the oracle."""
    rng = np.random.default_rng(M + N + k)
    logits = rng.standard_normal((M, N)).astype(np.float32)
    logits[0, [0, N - 1]] = 7.0                     # equal maxima in the first and the last slice
    if M > 1:
        logits[1] = np.float32(1.5)                 # one value only
    if M > 2:
        logits[2] = -np.sort(-logits[2])
    idx, val = _topk(ctx, engine, logits, k)
    want = np.stack([oracle.top_k(r, k) for r in logits])
    assert np.array_equal(idx, want) and np.array_equal(val, np.take_along_axis(logits, want.astype(np.int64), 1))
    am, _ = _run(ctx, engine, logits)
    assert am.tolist() == [oracle.greedy_sample(r) for r in logits]
    t = UnifiedTensor.new(ctx, logits, [M, N])
    mx, sm = UnifiedTensor.empty(ctx, [M]), UnifiedTensor.empty(ctx, [M])
    engine.softmax_stats(ctx, t, 0.7, mx, sm)
    c_idx, c_val, c_mx, c_sm = engine.sampler_candidates(ctx, t, k, 0.7)
    assert np.array_equal(c_idx, idx) and np.array_equal(c_val, val)
    assert np.array_equal(c_mx, mx.to_vec(ctx)) and np.array_equal(c_mx, logits.max(axis=1))
    assert np.array_equal(c_sm, sm.to_vec(ctx))
    want_sm = np.exp((logits.astype(np.float64) - c_mx[:, None]) / 0.7).sum(axis=1)
    assert np.max(np.abs(c_sm - want_sm) / want_sm) < 2e-6


@pytest.mark.parametrize("M,N,k", [(1, 1, 1), (3, 300, 7), (40, 4096, 64), (2, 70001, 1024), (5, 128256, 513)])
def test_top_p_draw_on_the_device(ctx, engine, M, N, k):
    """The nucleus walk on the device against the host's over the whole row: flat and peaked rows, one value only, NaN and
    infinities, the smallest draw; rows whose nucleus is longer than k are handed back."""
    from rusty_b200.sampler import Sampler
    rng = np.random.default_rng(M + N + k)
    logits = (rng.standard_normal((M, N)) * rng.uniform(0.5, 6.0, size=(M, 1))).astype(np.float32)
    if M > 2:
        logits[1, : N // 2] = np.nan
        logits[2] = np.float32(-3.0)
        logits[0, N // 3] = np.float32(-np.inf)
    t = UnifiedTensor.new(ctx, logits, [M, N])
    for temp, top_p in ((0.7, 0.9), (1.3, 0.4), (0.2, 0.98)):
        draws = rng.random(M).astype(np.float32)
        draws[0] = 0.0
        got = engine.sample_top_p(ctx, t, k, temp, top_p, draws)
        idx, val, mx, sm = engine.sampler_candidates(ctx, t, k, temp)
        for m in range(M):
            # exp differs by three units in the last place between here and there, and a sum of k terms rounds k times: a draw, or a
            # top_p, that close to a sum may fall to either side
            near = (4 + k) * 2.0**-24
            want = set()
            for dr in (0.0, -near, near):
                for dp in (0.0, -near, near):
                    w = Sampler(temp, top_p + dp, rand=lambda: np.float32(draws[m] + dr)).sample_from_candidates(idx[m], val[m], mx[m], sm[m])
                    want.add(0xFFFFFFFF if w is None else w)
            assert int(got[m]) in want, (temp, top_p, m)
            assert len(want) <= 3
    from rusty_b200 import BackendError
    with pytest.raises(BackendError) as e:
        engine.sample_top_p(ctx, t, k, 0.0, 0.9, draws)
    assert e.value.kind == "InvalidOperation"
    with pytest.raises(ValueError):
        engine.sample_top_p(ctx, t, k, 1.0, 0.9, draws[:-1] if M > 1 else np.zeros(2, np.float32))


def _winners(row, k, temp):
    """Of one row: indexes and values of its k largest logits in descending order (equal ones by ascending index; no NaN, nothing that is
    not above -1e9; index 0 and -inf where there are fewer), its largest number, and the sum of exp((x - max) / T) in 64 bits."""
    at = np.flatnonzero(row > np.float32(-1e9))
    at = at[np.argsort(-row[at].astype(np.float64), kind="stable")][:k]
    idx, val = np.zeros(k, np.uint32), np.full(k, -np.inf, np.float32)
    idx[:len(at)], val[:len(at)] = at, row[at]
    numbers = row[~np.isnan(row)]
    top = numbers.max() if numbers.size else np.float32(-np.inf)
    return idx, val, top, float(np.exp((numbers.astype(np.float64) - top) / temp).sum())


@pytest.mark.parametrize("M,N,k", [(1, 1, 1), (3, 300, 7), (40, 4096, 64), (2, 70001, 1024), (5, 128256, 513)])
def test_top_p_draw_from_the_logits(ctx, engine, M, N, k):
    """The same draw against the host's walk over candidates and sums that numpy takes from the logits: flat and peaked
    rows, one value only, NaN and infinities, the smallest draw; rows whose nucleus is longer than k are handed back."""
    from rusty_b200.sampler import Sampler
    rng = np.random.default_rng(M + N + k)
    logits = (rng.standard_normal((M, N)) * rng.uniform(0.5, 6.0, size=(M, 1))).astype(np.float32)
    if M > 2:
        logits[1, : N // 2] = np.nan
        logits[2] = np.float32(-3.0)
        logits[0, N // 3] = np.float32(-np.inf)
    t = UnifiedTensor.new(ctx, logits, [M, N])
    for temp, top_p in ((0.7, 0.9), (1.3, 0.4), (0.2, 0.98)):
        draws = rng.random(M).astype(np.float32)
        draws[0] = 0.0
        got = engine.sample_top_p(ctx, t, k, temp, top_p, draws)
        for m in range(M):
            idx, val, top, total = _winners(logits[m], k, np.float32(temp))
            # exp differs by three units in the last place between here and there, the device's sum over the row rounds 50 times (32 terms a
            # thread, then threads, warps and blocks), a sum of k terms k times: a draw, or a top_p, that close to a sum may fall to either side
            near = (56 + k) * 2.0**-24
            want = set()
            for dr in (0.0, -near, near):
                for dp in (0.0, -near, near):
                    w = Sampler(temp, top_p + dp, rand=lambda: np.float32(draws[m] + dr)).sample_from_candidates(idx, val, top, total)
                    want.add(0xFFFFFFFF if w is None else w)
            assert int(got[m]) in want, (temp, top_p, m)
            assert len(want) <= 3
