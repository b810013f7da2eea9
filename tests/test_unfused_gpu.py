"""GPU parity of the four unfused operators (and the buffer layer) against the
oracle, through the C ABI.  Written the way tests of rusty-backend's
ComputeEngine would read."""
import numpy as np
import pytest

from canary import GuardedOutput
from parity import TOL_FP32, assert_bits_equal, rel_err
from rusty_b200 import BackendError, DType, QLinear, UnifiedTensor

pytestmark = pytest.mark.gpu


def test_adapter_info(ctx):
    info = ctx.adapter_info()
    assert "CUDA sm_100" in info, info


def test_ops_test_matmul_identity(ctx, engine, kat):
    a = UnifiedTensor.new(ctx, [1.0, 2.0, 3.0, 4.0], [2, 2])
    b = UnifiedTensor.new(ctx, [1.0, 0.0, 0.0, 1.0], [2, 2])
    out = UnifiedTensor.empty(ctx, [2, 2])
    engine.matmul(ctx, a, b, out)
    assert out.to_vec(ctx).tolist() == [1.0, 2.0, 3.0, 4.0]


def test_matmul_tails_bit_exact_vs_fma_oracle(ctx, engine, kat):
    for i in range(int(kat["mm_count"])):
        a, b = kat[f"mm{i}_a"], kat[f"mm{i}_b"]
        M, K = a.shape
        N = b.shape[1]
        ta, tb = UnifiedTensor.new(ctx, a, [M, K]), UnifiedTensor.new(ctx, b, [K, N])
        out = UnifiedTensor.empty(ctx, [M, N])
        engine.matmul(ctx, ta, tb, out)
        got = out.to_vec(ctx).reshape(M, N)
        assert_bits_equal(got, kat[f"mm{i}_out_fma"])          # shader order under FMA contraction
        assert rel_err(got, kat[f"mm{i}_out"]) <= TOL_FP32     # and within tolerance of the uncontracted text
        tbt = UnifiedTensor.new(ctx, np.ascontiguousarray(b.T), [N, K])
        out2 = UnifiedTensor.empty(ctx, [M, N])
        engine.matmul_bt(ctx, ta, tbt, out2)
        assert_bits_equal(out2.to_vec(ctx).reshape(M, N), kat[f"mm{i}_bt_out_fma"])


@pytest.mark.parametrize("M,K,N", [(1, 4096, 4096), (33, 1000, 257), (128, 512, 640)])
def test_matmul_larger_vs_oracle(ctx, engine, oracle, M, K, N):
    rng = np.random.default_rng(M * 7 + N)
    a = rng.standard_normal((M, K)).astype(np.float32)
    b = rng.standard_normal((K, N)).astype(np.float32)
    ta, tb = UnifiedTensor.new(ctx, a, [M, K]), UnifiedTensor.new(ctx, b, [K, N])
    out = UnifiedTensor.empty(ctx, [M, N])
    engine.matmul(ctx, ta, tb, out)
    got = out.to_vec(ctx).reshape(M, N)
    rows = slice(0, min(M, 4))  # the scalar oracle on a few rows; all of them for M=1
    assert_bits_equal(got[rows], oracle.matmul_tiled(a[rows], b, fma=True))
    assert rel_err(got[rows], oracle.matmul_tiled(a[rows], b)) <= TOL_FP32
    assert rel_err(got, a.astype(np.float64) @ b.astype(np.float64)) <= TOL_FP32


def test_dequantize_kats(ctx, engine, kat):
    raw = kat["deq_in"]
    t_in = UnifiedTensor.from_bytes_with_dtype(ctx, raw, [raw.size], DType.U8)
    out = UnifiedTensor.empty(ctx, [raw.size])
    engine.dequantize(ctx, t_in, out)
    assert_bits_equal(out.to_vec(ctx), kat["deq_out"])
    big = kat["deq_big_in"]
    t_in = UnifiedTensor.from_bytes_with_dtype(ctx, big, [big.size], DType.U8)
    out = UnifiedTensor.empty(ctx, [big.size])
    engine.dequantize(ctx, t_in, out)
    assert_bits_equal(out.to_vec(ctx), kat["deq_big_out"])


def test_dequantize_ragged(ctx, engine, kat):
    raw = kat["deq_in"]
    # 7 outputs only: the shader's per-store guard drops the 8th value
    t_in = UnifiedTensor.from_bytes_with_dtype(ctx, raw[:8], [7], DType.U8)
    out = UnifiedTensor.new(ctx, np.full(7, -1.0, np.float32), [7])
    engine.dequantize(ctx, t_in, out)
    assert_bits_equal(out.to_vec(ctx), kat["deq_out_n7"])
    # input buffer holds 2 words but the shape claims 12 bytes: outputs past the input stay untouched
    t_in = UnifiedTensor.from_bytes_with_dtype(ctx, raw[:8], [12], DType.U8)
    out = UnifiedTensor.new(ctx, np.full(12, -1.0, np.float32), [12])
    engine.dequantize(ctx, t_in, out)
    assert_bits_equal(out.to_vec(ctx), kat["deq_out_short_in"])


def test_dequantize_config1_weight_exact(ctx, engine, oracle):
    """Every byte of the 4096x4096 weight unpacks bit-exactly (16.7 M values)."""
    rng = np.random.default_rng(0)
    raw = rng.integers(0, 256, size=4096 * 4096, dtype=np.uint8)
    t_in = UnifiedTensor.from_bytes_with_dtype(ctx, raw, [4096, 4096], DType.U8)
    out = UnifiedTensor.empty(ctx, [4096, 4096])
    engine.dequantize(ctx, t_in, out)
    got = out.to_vec(ctx)
    assert np.array_equal(got.view(np.uint32), raw.astype(np.float32).view(np.uint32))
    assert_bits_equal(got[:4096], oracle.dequantize(raw[:4096]))


def test_affine_dequantize_kat_bit_exact(ctx, engine, kat):
    u, s, b = kat["aff_u"], kat["aff_s"], kat["aff_b"]
    w = UnifiedTensor.from_bytes_with_dtype(ctx, np.concatenate([u, np.zeros(5, np.uint8)]), [u.size], DType.U8)
    out = UnifiedTensor.empty(ctx, [u.size])
    engine.affine_dequantize(ctx, w, UnifiedTensor.new(ctx, s, [s.size]), UnifiedTensor.new(ctx, b, [b.size]), out)
    assert_bits_equal(out.to_vec(ctx), kat["aff_out"])


def test_affine_dequantize_beyond_reference_dispatch_limit(ctx, engine, oracle):
    """n > 4 194 240: the reference's dispatch leaves the tail unwritten; this
    implementation writes every element with the intended arithmetic."""
    n = 4096 * 4096
    rng = np.random.default_rng(11)
    u = rng.integers(0, 256, size=n, dtype=np.uint8)
    s = rng.uniform(0.001, 0.02, size=n // 64).astype(np.float32)
    b = rng.uniform(-2, 2, size=n // 64).astype(np.float32)
    w = UnifiedTensor.from_bytes_with_dtype(ctx, u, [4096, 4096], DType.U8)
    out = UnifiedTensor.empty(ctx, [4096, 4096])
    engine.affine_dequantize(ctx, w, UnifiedTensor.new(ctx, s, [s.size]), UnifiedTensor.new(ctx, b, [b.size]), out)
    got = out.to_vec(ctx)
    assert_bits_equal(got, oracle.affine_dequantize(u, s, b, mt=True))


def test_add(ctx, engine):
    a = UnifiedTensor.new(ctx, [1.0, 2.0, 3.0, 4.0], [4])
    b = UnifiedTensor.new(ctx, [5.0, 6.0, 7.0, 8.0], [4])
    out = UnifiedTensor.empty(ctx, [4])
    engine.add(ctx, a, b, out)
    assert out.to_vec(ctx).tolist() == [6.0, 8.0, 10.0, 12.0]


# ---- buffer layer: pool bins, views, copy_tensor, errors ----

def test_pool_returns_exact_size_bins(ctx):
    ctx.pool_clear()
    nbytes = 12345 * 4
    t = UnifiedTensor.empty(ctx, [12345])
    p = t.device_ptr()
    assert ctx.pool_idle_count(nbytes) == 0
    del t
    assert ctx.pool_idle_count(nbytes) == 1
    t2 = UnifiedTensor.empty(ctx, [12345])           # same size: same buffer comes back
    assert t2.device_ptr() == p and ctx.pool_idle_count(nbytes) == 0
    t3 = UnifiedTensor.empty(ctx, [12346])           # other size: other bin
    assert t3.device_ptr() != p
    del t2, t3
    fresh = UnifiedTensor.new(ctx, np.zeros(12345, np.float32), [12345])  # `new` is not pooled
    del fresh
    assert ctx.pool_idle_count(nbytes) == 1
    ctx.pool_clear()
    assert ctx.pool_idle_count(nbytes) == 0


def test_reshaped_shares_storage(ctx):
    t = UnifiedTensor.new(ctx, np.arange(12, dtype=np.float32), [3, 4])
    v = t.reshaped([2, 6])
    assert v.device_ptr() == t.device_ptr() and v.shape == [2, 6]
    with pytest.raises(AssertionError):
        t.reshaped([5, 5])
    del t
    assert v.to_vec(ctx).tolist() == list(range(12))


def test_copy_tensor_with_offset(ctx, engine):
    src = UnifiedTensor.new(ctx, [1.0, 2.0], [2])
    dst = UnifiedTensor.zeros(ctx, [5])
    engine.copy_tensor(ctx, src, dst, 8)
    assert dst.to_vec(ctx).tolist() == [0.0, 0.0, 1.0, 2.0, 0.0]
    with pytest.raises(BackendError) as e:
        engine.copy_tensor(ctx, src, dst, 16)
    assert e.value.kind == "BufferOperation"


def test_shape_errors_are_status_codes(ctx, engine):
    a = UnifiedTensor.new(ctx, np.zeros(6, np.float32), [2, 3])
    b = UnifiedTensor.new(ctx, np.zeros(6, np.float32), [3, 2])
    small = UnifiedTensor.empty(ctx, [1, 2])
    with pytest.raises(BackendError) as e:
        engine.matmul(ctx, a, b, small)
    assert e.value.kind == "InvalidDimensions"
    ctx.sync()  # the context is still usable


def test_release_while_a_capture_is_open_is_deferred(ctx, engine):
    """A host-language destructor may run at any time, also between graph_begin and graph_end; freeing device memory
    or synchronising there would invalidate the capture, so the release is parked until the capture has ended."""
    from rusty_b200 import QLinear
    from rusty_b200.backend import Graph
    from rusty_b200.workloads import sym_row_linear
    rng = np.random.default_rng(3)
    a = rng.standard_normal(1000).astype(np.float32)
    b = rng.standard_normal(1000).astype(np.float32)
    ta, tb, out = UnifiedTensor.new(ctx, a, [1000]), UnifiedTensor.new(ctx, b, [1000]), UnifiedTensor.empty(ctx, [1000])
    victim = UnifiedTensor.new(ctx, a, [1000])          # not pooled: its release is a cudaFree
    x, q, s = sym_row_linear(0, 1, 256, 64)
    ql_victim = QLinear.from_host(ctx, q, s)             # a whole fused linear dies inside the capture as well
    old = Graph(ctx)
    with old:
        engine.add(ctx, ta, tb, out)
    g = Graph(ctx)
    with g:
        engine.add(ctx, ta, tb, out)
        del victim
        del ql_victim
        del old                                          # a graph destroyed while another capture is open
        engine.add(ctx, out, tb, out)
    g.launch()
    ctx.sync()
    assert np.array_equal(out.to_vec(ctx), (a + b) + b)
    # the context is fully usable afterwards (allocations, eager launches, another capture)
    t2 = UnifiedTensor.new(ctx, b, [1000])
    engine.add(ctx, t2, t2, out)
    assert np.array_equal(out.to_vec(ctx), b + b)
    g2 = Graph(ctx)
    with g2:
        engine.add(ctx, ta, ta, out)
    g2.launch()
    assert np.array_equal(out.to_vec(ctx), a + a)


@pytest.mark.parametrize("M,K,N", [(1, 257, 33), (3, 132, 70), (8, 64, 31), (9, 65, 4100), (17, 100, 4096), (33, 31, 5000), (70, 36, 5003),
                                   (130, 48, 9999)])
def test_matmul_tiles_bit_for_bit(ctx, engine, oracle, M, K, N):
    """Every tile of both matmuls at ragged edges: still one accumulator per output, k ascending, FMA."""
    rng = np.random.default_rng(M + K + N)
    a, b = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((K, N)).astype(np.float32)
    ta, tb, tbt = UnifiedTensor.new(ctx, a, [M, K]), UnifiedTensor.new(ctx, b, [K, N]), UnifiedTensor.new(ctx, np.ascontiguousarray(b.T), [N, K])
    want = oracle.matmul_tiled(a, b, fma=True)
    for run, t in ((engine.matmul, tb), (engine.matmul_bt, tbt)):
        out = GuardedOutput(ctx, [M, N], DType.FP32)
        run(ctx, ta, t, out.tensor)
        assert_bits_equal(out.read(), want)


@pytest.mark.parametrize("M,K,N,rank", [(1, 256, 64, 1), (5, 130, 96, 3), (40, 512, 260, 16), (300, 256, 128, 65)])
def test_linear_lora_call(ctx, engine, oracle, M, K, N, rank):
    """x . W + (x . A) . B in one call, over an f32 and over a quantised weight."""
    rng = np.random.default_rng(M + rank)
    x, w = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((K, N)).astype(np.float32)
    a, b = rng.standard_normal((K, rank)).astype(np.float32), rng.standard_normal((rank, N)).astype(np.float32)
    tx, ta, tb = UnifiedTensor.new(ctx, x, [M, K]), UnifiedTensor.new(ctx, a, [K, rank]), UnifiedTensor.new(ctx, b, [rank, N])
    branch = (x.astype(np.float64) @ a) @ b
    out = GuardedOutput(ctx, [M, N], DType.FP32)
    engine.linear_lora(ctx, tx, UnifiedTensor.new(ctx, w, [K, N]), ta, tb, out.tensor)
    assert rel_err(out.read(), x.astype(np.float64) @ w + branch) <= TOL_FP32
    if K % 16 == 0:
        q, s = rng.integers(-127, 128, size=(N, K), dtype=np.int8), rng.uniform(0.001, 0.02, size=N).astype(np.float32)
        out = GuardedOutput(ctx, [M, N], DType.FP32)
        engine.linear_lora(ctx, tx, QLinear.from_host(ctx, q, s), ta, tb, out.tensor)
        assert rel_err(out.read(), x.astype(np.float64) @ (q * s[:, None].astype(np.float64)).T + branch) <= TOL_FP32


@pytest.mark.parametrize("M,rank", [(262141, 4), (262150, 8), (3, 262141), (2, 262150)])
def test_linear_lora_of_many_rows_or_columns(ctx, engine, M, rank):
    """More rows than a launch holds row tiles of four, and a rank of more columns than a launch holds blocks of four: what the
    products one by one took.  Small whole numbers, so that every sum is exact."""
    K, N = 16, 64
    rng = np.random.default_rng(M + rank)
    x, w = rng.integers(-4, 5, size=(M, K)).astype(np.float32), rng.integers(-4, 5, size=(K, N)).astype(np.float32)
    a, b = rng.integers(-2, 3, size=(K, rank)).astype(np.float32), rng.integers(-1, 2, size=(rank, N)).astype(np.float32)
    tx, ta, tb = (UnifiedTensor.new(ctx, v, list(v.shape)) for v in (x, a, b))
    low = (x @ a) @ b
    out = GuardedOutput(ctx, [M, N])
    engine.linear_lora(ctx, tx, UnifiedTensor.new(ctx, w, [K, N]), ta, tb, out.tensor)
    assert_bits_equal(out.read(), x @ w + low)
    q = rng.integers(-4, 5, size=(N, K), dtype=np.int8)
    out = GuardedOutput(ctx, [M, N])
    engine.linear_lora(ctx, tx, QLinear.from_host(ctx, q, np.ones(N, np.float32)), ta, tb, out.tensor)
    assert_bits_equal(out.read(), x @ q.T.astype(np.float32) + low)


@pytest.mark.parametrize("M,rank", [(100, 16), (200, 32), (200, 30), (300, 64)])
def test_linear_lora_first_products_back_to_back(ctx, engine, M, rank):
    """The adapter's first product with four rows a block, with eight (16-byte and single loads of A) and as a matmul of its own,
    over an f32 and a quantised weight: calls back to back over an x that a kernel rewrites in between, against float64."""
    K, N, steps = 256, 192, 6
    rng = np.random.default_rng(M + rank)
    w, a, b = (rng.standard_normal(s).astype(np.float32) for s in ((K, N), (K, rank), (rank, N)))
    q, s = rng.integers(-127, 128, size=(N, K), dtype=np.int8), rng.uniform(0.001, 0.02, size=N).astype(np.float32)
    ta, tb = UnifiedTensor.new(ctx, a, [K, rank]), UnifiedTensor.new(ctx, b, [rank, N])
    weights = ((UnifiedTensor.new(ctx, w, [K, N]), w.astype(np.float64)), (QLinear.from_host(ctx, q, s), (q * s[:, None].astype(np.float64)).T))
    xs = [rng.standard_normal((M, K)).astype(np.float32) for _ in range(3)]
    src, zero = [UnifiedTensor.new(ctx, x, [M, K]) for x in xs], UnifiedTensor.zeros(ctx, [M, K])
    for tw, wf in weights:
        x, ys = UnifiedTensor.empty(ctx, [M, K]), [UnifiedTensor.empty(ctx, [M, N]) for _ in range(steps)]
        for i in range(steps):
            engine.add(ctx, src[i % 3], zero, x)
            engine.linear_lora(ctx, x, tw, ta, tb, ys[i])
        for i in range(steps):
            x64 = xs[i % 3].astype(np.float64)
            assert rel_err(ys[i].to_vec(ctx).reshape(M, N), x64 @ wf + (x64 @ a) @ b) <= TOL_FP32


@pytest.mark.parametrize("M,K,N,rank", [(1, 4096, 260, 2), (5, 1028, 1024, 8), (8, 1024, 1100, 3), (9, 2052, 516, 17), (16, 4096, 260, 64), (17, 1040, 1012, 1),
                                        (33, 1024, 4100, 30), (100, 8192, 132, 4)])
def test_linear_lora_with_k_cut(ctx, engine, M, K, N, rank):
    """The f32 weight's kernel that cuts K, at ragged rows, columns, units of k and ranks.  Bound: a product enters with the rounding of its
    addition alone, and at most 88 roundings of 2^-24 of the sum of magnitudes lie on an output's way (72 links of a chain, two halves, eight
    warps, eight ranges); half of that and more cancels, 52 are asked for."""
    rng = np.random.default_rng(M + K + N)
    x, w = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((K, N)).astype(np.float32)
    x[:, rng.integers(0, K, size=4)] *= 1000.0
    a, b = rng.standard_normal((K, rank)).astype(np.float32), rng.standard_normal((rank, N)).astype(np.float32)
    tx, tw = UnifiedTensor.new(ctx, x, [M, K]), UnifiedTensor.new(ctx, w, [K, N])
    ta, tb = UnifiedTensor.new(ctx, a, [K, rank]), UnifiedTensor.new(ctx, b, [rank, N])
    x64, t64 = x.astype(np.float64), x.astype(np.float64) @ a
    want = x64 @ w + t64 @ b
    sizes = np.abs(x64) @ np.abs(w) + (np.abs(x64) @ np.abs(a)) @ np.abs(b)
    out = GuardedOutput(ctx, [M, N], DType.FP32)
    engine.linear_lora(ctx, tx, tw, ta, tb, out.tensor)
    got = out.read()
    assert (np.abs(got - want) <= 52 * 2.0**-24 * sizes).all()
    # an infinity stays one, in its row (of x) or its column (of W)
    xi, wi = x.copy(), w.copy()
    xi[M // 2, 3], wi[K - 1, N // 2] = np.inf, -np.inf
    out = GuardedOutput(ctx, [M, N], DType.FP32)
    engine.linear_lora(ctx, UnifiedTensor.new(ctx, xi, [M, K]), UnifiedTensor.new(ctx, wi, [K, N]), ta, UnifiedTensor.zeros(ctx, [rank, N]), out.tensor)
    got = out.read()
    rows, cols = np.arange(M) != M // 2, np.arange(N) != N // 2
    assert np.isfinite(got[rows][:, cols]).all()
    assert np.array_equal(got[rows, N // 2], np.sign(xi[rows, K - 1]) * -np.inf)
    # the infinite x times A makes an infinite or undefined t, and that times a zero B is undefined, as in the products one by one
    assert np.isnan(got[M // 2]).all()


def _with_k_cut(ctx, engine, x, w, a=None, b=None):
    (M, K), N = x.shape, w.shape[1]
    a = np.zeros((K, 4), np.float32) if a is None else a
    b = np.zeros((4, N), np.float32) if b is None else b
    tensors = [UnifiedTensor.new(ctx, v, list(v.shape)) for v in (x, w, a, b)]
    out = GuardedOutput(ctx, [M, N], DType.FP32)
    engine.linear_lora(ctx, *tensors, out.tensor)
    return out.read()


@pytest.mark.parametrize("M", [1, 6, 16, 33])
@pytest.mark.parametrize("case", ["normal", "near_one", "tiny_x", "huge_x", "subnormal_products"])
def test_linear_lora_single_products(ctx, engine, M, case):
    """One activation of a row is not zero: every output is one product, and comes out as f32 rounds it, over the whole range of
    exponents (the zeros beside it add nothing)."""
    K, N = 2048, 1024
    rng = np.random.default_rng(M)
    v = {"normal": rng.standard_normal(M), "near_one": np.full(M, 1 + 2.0**-11 + 2.0**-23), "tiny_x": rng.standard_normal(M) * 2.0**-118,
         "huge_x": rng.standard_normal(M) * 2.0**121, "subnormal_products": rng.standard_normal(M) * 2.0**-100}[case].astype(np.float32)
    w = {"normal": rng.standard_normal((K, N)), "near_one": np.full((K, N), 1 + 2.0**-11 + 2.0**-22), "tiny_x": rng.standard_normal((K, N)) * 2.0**90,
         "huge_x": rng.standard_normal((K, N)), "subnormal_products": rng.standard_normal((K, N)) * 2.0**-30}[case].astype(np.float32)
    x = np.zeros((M, K), np.float32)
    at = rng.integers(0, K, size=M)
    x[np.arange(M), at] = v
    assert np.array_equal(_with_k_cut(ctx, engine, x, w), v[:, None] * w[at])


@pytest.mark.parametrize("K,N", [(4096, 1024), (1040, 4100), (8192, 132)])
def test_linear_lora_row_alone_and_in_a_batch(ctx, engine, K, N):
    """Up to 32 rows a row's bits do not depend on the rows beside it; an infinite weight changes its own column alone."""
    rng = np.random.default_rng(K + N)
    x, w = rng.standard_normal((32, K)).astype(np.float32), rng.standard_normal((K, N)).astype(np.float32)
    a, b = rng.standard_normal((K, 8)).astype(np.float32), rng.standard_normal((8, N)).astype(np.float32)
    want = _with_k_cut(ctx, engine, x, w, a, b)
    for first, rows in ((0, 1), (3, 4), (5, 7), (19, 13), (1, 17)):
        assert_bits_equal(_with_k_cut(ctx, engine, x[first:first + rows], w, a, b), want[first:first + rows])
    w[K // 3, N // 2] = np.inf
    got = _with_k_cut(ctx, engine, x, w, a, b)
    others = np.arange(N) != N // 2
    assert_bits_equal(got[:, others], want[:, others])
    assert np.array_equal(got[:, N // 2], np.sign(x[:, K // 3]) * np.inf)


def test_linear_lora_with_k_cut_back_to_back(ctx, engine):
    """Calls back to back over an x that a kernel rewrites in between, on one scratch for x . A: each sees its own."""
    M, K, N, rank, steps = 20, 2048, 1024, 30, 8
    rng = np.random.default_rng(5)
    w, a, b = (rng.standard_normal(s).astype(np.float32) for s in ((K, N), (K, rank), (rank, N)))
    xs = [rng.standard_normal((M, K)).astype(np.float32) for _ in range(3)]
    src, zero = [UnifiedTensor.new(ctx, x, [M, K]) for x in xs], UnifiedTensor.zeros(ctx, [M, K])
    tw, ta, tb = (UnifiedTensor.new(ctx, v, list(v.shape)) for v in (w, a, b))
    x, ys = UnifiedTensor.empty(ctx, [M, K]), [UnifiedTensor.empty(ctx, [M, N]) for _ in range(steps)]
    for i in range(steps):
        engine.add(ctx, src[i % 3], zero, x)
        engine.linear_lora(ctx, x, tw, ta, tb, ys[i])
    for i in range(steps):
        x64 = xs[i % 3].astype(np.float64)
        assert rel_err(ys[i].to_vec(ctx).reshape(M, N), x64 @ w + (x64 @ a) @ b) <= 1e-6


@pytest.mark.parametrize("M,K,N,rank", [(33, 640, 1640, 8), (47, 1040, 1000, 4), (48, 912, 2992, 1), (49, 2052, 1028, 17), (64, 1024, 1024, 8),
                                        (65, 4096, 260, 64), (200, 1552, 684, 12), (257, 512, 2052, 30)])
def test_linear_lora_with_k_cut_beyond_32_rows(ctx, engine, M, K, N, rank):
    """Tiles of 16 and of 32 rows, the last of each with a row, half of them or all; a last group of columns with 4 to 64.  Bound: what f32
    sums may be off, each addition by 2^-24 of the magnitudes before it: the links of half a warp's range, seventeen sums of ranges, and for
    the branch the K links of x . A before them."""
    rng = np.random.default_rng(M + K + N + rank)
    x, w, a, b = (rng.standard_normal(s).astype(np.float32) for s in ((M, K), (K, N), (K, rank), (rank, N)))
    got = _with_k_cut(ctx, engine, x, w, a, b).astype(np.float64)
    x64, w64, a64, b64 = (v.astype(np.float64) for v in (x, w, a, b))
    links = 8 * -(-(-(-K // 16) + -(-rank // 16)) // 8) + 18
    may = 2.0**-24 * (links * (abs(x64) @ abs(w64)) + (links + K) * (abs(x64) @ abs(a64) @ abs(b64)))
    assert (abs(got - (x64 @ w64 + (x64 @ a64) @ b64)) <= may).all()


def test_linear_lora_short_rows_alone_and_in_a_batch(ctx, engine):
    """The same bits for a row alone and in a batch of up to 32 where K is short and cut over a cluster."""
    K, N = 640, 1640
    rng = np.random.default_rng(6)
    x, w, a, b = (rng.standard_normal(s).astype(np.float32) for s in ((32, K), (K, N), (K, 12), (12, N)))
    want = _with_k_cut(ctx, engine, x, w, a, b)
    for first, rows in ((0, 1), (3, 4), (5, 8), (19, 13), (1, 17)):
        assert_bits_equal(_with_k_cut(ctx, engine, x[first:first + rows], w, a, b), want[first:first + rows])
