"""The arithmetic of the integer tensor-core kernels restated in numpy, checked on CPU: why feeding the tensor core integers
loses nothing against the reference's f32 dequantise-then-matmul.

One scale per output row, one or two activation rows (rusty_b200/csrc/gemv_mma.cu).  Per activation row and K slice (8 slices:
k-bytes [128 w, 128 w + 128) of every 1024) a power-of-two scale brings the slice's largest |a| into [64, 127];
T = round(a * scale * 2^24) is split EXACTLY into four balanced bytes; the integer dot products per digit plane are recombined in
64-bit integers and leave the slice as a double; the slices are added in a fixed order and rounded to f32 once, and the row's
scale multiplies the sum.

The reference's own format (u8 [in,out], one scale and bias per 64 consecutive outputs of an input row;
rusty_b200/csrc/gemm_gc_tc.cu).  The group's scales ride on the activations, a = fl32(x * s_g); q = round(a * 2^e) with the row's
largest |q| in [2^30, 2^31) and r = round(b_g / s_g * 2^j) with the group's largest below 2^31 are integers, q + 2^31 and
r + 2^31 four unsigned bytes each, and an output is 2^-e (sum q u + 2^-j sum q r), rounded once.

The same format along the contraction ([out,in] rows; rusty_b200/csrc/gemv_affine.cu).  Per activation row and 64 k four balanced
bytes below the chunk's own power of two; a chunk's share (upper planes' dot * s + upper part of sum(x) * b, and the same of the
lower parts) is an f32, gathered in f32 over up to 16 chunks and in double beyond."""
import numpy as np
import pytest

from parity import TOL_FP32, rel_err, rel_err_rows


def _balanced_bytes(t):
    """|t| <= 127 * 2^24 -> four signed bytes, most significant first: add 128 to the lower three, flip their top bits."""
    half = 0x808080
    w = ((t + half) ^ half) & 0xffffffff
    d = np.stack([((w >> s) & 0xff).astype(np.uint8).view(np.int8).astype(np.int64) for s in (24, 16, 8, 0)])
    assert np.array_equal(((d[0] * 256 + d[1]) * 256 + d[2]) * 256 + d[3], t)           # the split is exact
    return d


def _digits(a32: np.ndarray):
    """a32: one K slice of one activation row (f32).  Returns (digit planes int64 [4, n], most significant first; e2)."""
    v = float(np.max(np.abs(a32))) if a32.size else 0.0
    if v == 0.0:
        return np.zeros((4, a32.size), np.int64), 0
    e2 = 7 - int(np.frexp(v)[1])               # v * 2^e2 in [64, 128)
    if v * 2.0 ** e2 > 127.0:
        e2 -= 1
    t = np.rint(a32.astype(np.float64) * 2.0 ** (e2 + 24)).astype(np.int64)   # the device does this in f32: exact up to the rounding
    assert np.all(np.abs(t) <= 127 * 2 ** 24)
    return _balanced_bytes(t), e2


def _slices(K: int):
    for w in range(8):
        idx = np.concatenate([np.arange(c + 128 * w, min(c + 128 * w + 128, K)) for c in range(0, K, 1024)
                              if c + 128 * w < K]) if K > 128 * w else np.zeros(0, np.int64)
        yield idx.astype(np.int64)


def _model_row(a32: np.ndarray, wq: np.ndarray) -> np.ndarray:
    """One activation row a32 [K] against integer weights wq [N, K]."""
    N, K = wq.shape
    acc = np.zeros(N, np.float64)
    for idx in _slices(K):
        if idx.size == 0:
            continue
        d, e2 = _digits(a32[idx])
        w = wq[:, idx].astype(np.int64)
        hi = (w @ d[0]) * 256 + (w @ d[1])     # as the kernel folds its accumulator columns
        lo = (w @ d[2]) * 256 + (w @ d[3])
        acc += (hi * 65536 + lo).astype(np.float64) * 2.0 ** (-e2 - 24)       # exact: an integer times a power of two
    return acc.astype(np.float32)              # one rounding


def _unsigned_bytes(q):
    w = q + 2 ** 31
    assert np.all((w >= 0) & (w < 2 ** 32))
    return [(w >> s) & 0xff for s in (24, 16, 8, 0)]


def _native_group(x, s, b, u):
    """Activations x [M, K] f32 against one group: s, b [K] f32, u [64, K] bytes.  [M, 64] f32."""
    M, K = x.shape
    u = u.astype(np.int64)
    with np.errstate(divide="ignore", invalid="ignore"):
        ratio = np.where(b == 0, 0.0, b.astype(np.float64) / s.astype(np.float64))
    most = np.max(np.abs(ratio))
    has_r = bool(most <= 4096)                 # (a NaN has not)
    j = (30 - int(np.floor(np.log2(most))) if most > 2.0 ** -30 else 60) if has_r else 0
    r = np.clip(np.rint(ratio * 2.0 ** j), -2 ** 31, 2 ** 31 - 1).astype(np.int64) if has_r else np.zeros(K, np.int64)
    rb = np.stack(_unsigned_bytes(r) + [np.ones(K, np.int64)])                          # [5, K], the last a row of ones
    y = np.empty((M, u.shape[0]), np.float32)
    for m in range(M):
        a = (x[m] * s).astype(np.float32)                                               # the one rounding of an element
        top = np.max(np.abs(a))
        e = 30 - int(np.floor(np.log2(top))) if top else 0
        q = np.rint(a.astype(np.float64) * 2.0 ** e).astype(np.int64)
        planes = _unsigned_bytes(q)
        both = np.concatenate([u, rb])
        dots = [both @ p for p in planes]                                               # the MMA: int32 per plane
        assert max(int(np.max(np.abs(d))) for d in dots) < 2 ** 31
        t = ((dots[0] * 256 + dots[1]) * 256 + dots[2]) * 256 + dots[3]
        t = t - (both.sum(axis=1) << 31)                                                # q's offset: sum q u, sum q byte, sum q
        su, sr, sq = t[:u.shape[0]], t[u.shape[0]:-1], int(t[-1])
        qr = float(sr[0] - 128 * sq) * 2.0 ** 24 + (float(sr[1]) * 65536.0 + float(sr[2]) * 256.0 + float(sr[3]))   # r's offset off its top byte
        bias = 0.0 if has_r else float(x[m].astype(np.float64) @ b.astype(np.float64))
        y[m] = ((su.astype(np.float64) + (qr * 2.0 ** -j if has_r else 0.0)) * 2.0 ** -e + bias).astype(np.float32)
    return y


def _native_model(x, ukn, sg, bg):
    N = ukn.shape[1]
    return np.concatenate([_native_group(x, sg[:, g], bg[:, g], np.ascontiguousarray(ukn[:, 64 * g:64 * g + 64].T)) for g in range(N // 64)], axis=1)


def _along_k_model(x, u, sg, bg, run=16):
    """Activations x [M, K] f32, weights u [N, K] bytes with sg, bg [N, K / 64]: one range of all chunks."""
    f32 = np.float32
    M, K = x.shape
    total = np.zeros((M, u.shape[0]))
    acc = np.zeros((2, M, u.shape[0]), f32)
    for g in range(K // 64):
        xc, uc = x[:, 64 * g:64 * g + 64], u[:, 64 * g:64 * g + 64].astype(np.int64)
        e = np.maximum(np.frexp(np.max(np.abs(xc), axis=1))[1], -119)
        d = _balanced_bytes(np.rint(xc.astype(np.float64) * 2.0 ** (30 - e)[:, None]).astype(np.int64))
        sx = xc.astype(np.float64).sum(axis=1)
        upper = sx.astype(f32)
        for h, (hi, lo, unit, part) in enumerate(((d[0], d[1], 2.0 ** (e - 14), upper), (d[2], d[3], 2.0 ** (e - 30), (sx - upper).astype(f32)))):
            dots = hi @ uc.T * 256 + lo @ uc.T
            assert np.max(np.abs(dots)) < 2 ** 31
            dot = (dots.astype(f32) * unit.astype(f32)[:, None]).astype(f32)
            term = (part[:, None] * bg[None, :, g]).astype(f32)
            acc[h] += (dot.astype(np.float64) * sg[None, :, g] + term).astype(f32)
        if g % run == run - 1 or g == K // 64 - 1:
            total += (acc[0] + acc[1]).astype(np.float64)
            acc[:] = 0
    return total.astype(f32)


@pytest.mark.parametrize("K,N", [(1024, 48), (4096, 64), (1152, 33)])
def test_symmetric_weights_model_matches_the_oracle(oracle, K, N):
    from rusty_b200.workloads import sym_row_linear
    x, q, s = sym_row_linear(K + N, 2, K, N)
    x[0, ::97] *= 40.0
    got = np.stack([_model_row(x[m], q) * s for m in range(2)])
    wf = oracle.dequantize_rowscale(q, s)
    ref = oracle.matmul_bt(x, wf)
    assert rel_err(got, ref) <= TOL_FP32
    # and closer to the exact sums than the reference's own f32 accumulation is
    exact = oracle.matmul_bt_f64(x, wf)
    assert rel_err(got, exact) <= max(rel_err(ref, exact), 1e-7) * 1.5


@pytest.mark.parametrize("K,N", [(1024, 64), (4096, 128), (1152, 192)])
def test_reference_format_model_matches_the_oracle(oracle, K, N):
    from rusty_b200.workloads import sym_row_linear
    x, q, _ = sym_row_linear(3 * K + N, 2, K, N)
    x[1, ::61] *= 25.0
    rng = np.random.default_rng(K + N)
    ukn = (np.ascontiguousarray(q.T).astype(np.int16) + 128).astype(np.uint8)          # [K, N]
    sg = rng.uniform(0.001, 0.02, size=(K, N // 64)).astype(np.float32)
    bg = (-128.0 * sg + rng.uniform(-0.05, 0.05, size=sg.shape)).astype(np.float32)
    got = _native_model(x, ukn, sg, bg)
    ref = oracle.qlinear_affine(x, ukn, sg.ravel(), bg.ravel(), ukn.shape, layout_nk=False)
    assert rel_err(got, ref) <= TOL_FP32
    wf = np.ascontiguousarray(oracle.affine_dequantize(ukn, sg.ravel(), bg.ravel()).reshape(K, N).T)
    exact = oracle.matmul_bt_f64(x, wf)
    assert rel_err(got, exact) <= max(rel_err(ref, exact), 1e-6) * 1.5


def _native_case(K, G, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((3, K)).astype(np.float32)
    ukn = rng.integers(0, 256, size=(K, 64 * G), dtype=np.uint8)
    sg = rng.uniform(0.001, 0.02, size=(K, G)).astype(np.float32)
    bg = (-128.0 * sg * rng.uniform(0.8, 1.2, size=sg.shape)).astype(np.float32)
    return x, ukn, sg, bg


def _exact_kn(x, ukn, sg, bg):
    return x.astype(np.float64) @ (ukn * np.repeat(sg.astype(np.float64), 64, axis=1) + np.repeat(bg.astype(np.float64), 64, axis=1))


def test_reference_format_model_rounds_an_element_and_the_output_only():
    """2^-24 / sqrt(3) is the most a rounding to f32 has in the mean square; there are two."""
    x, ukn, sg, bg = _native_case(2048, 8, 1)
    exact = _exact_kn(x, ukn, sg, bg)
    assert np.linalg.norm(_native_model(x, ukn, sg, bg) - exact) / np.linalg.norm(exact) <= 2.0 ** 0.5 * 2.0 ** -24 / 3.0 ** 0.5


def test_reference_format_model_with_an_outlier_on_a_small_scale():
    """The unit follows the largest product: an input feature 10^6 times the others, on scales as much smaller, costs nothing."""
    x, ukn, sg, bg = _native_case(1024, 2, 2)
    x[:, 77] *= np.float32(1e6)
    sg[77] *= np.float32(1e-6)
    bg[77] *= np.float32(1e-6)
    assert rel_err_rows(_native_model(x, ukn, sg, bg), _exact_kn(x, ukn, sg, bg)) <= 1e-6


def test_reference_format_model_without_a_scale_to_measure_the_bias_by():
    x, ukn, sg, bg = _native_case(512, 3, 3)
    sg[:, 1], bg[5, 2] = 0.0, 1000.0                # a group of constants, and a bias of more than 4096 scales
    assert rel_err_rows(_native_model(x, ukn, sg, bg), _exact_kn(x, ukn, sg, bg)) <= 1e-6


@pytest.mark.parametrize("K", [64, 1024, 8192])
def test_scales_along_the_contraction_model(oracle, K):
    """The bound of the device test (roundings of a share at the size of its terms, of a run at the size it has gathered, and of
    the output), whatever the length of the contraction; rows of tiny values keep their bits."""
    rng = np.random.default_rng(K)
    M, N = 6, 96
    x = rng.standard_normal((M, K)).astype(np.float32)
    x[M - 1] *= np.float32(2.0 ** -100)
    u = rng.integers(0, 256, size=(N, K), dtype=np.uint8)
    sg = rng.uniform(0.001, 0.02, size=(N, K // 64)).astype(np.float32)
    bg = (-128.0 * sg * rng.uniform(0.9, 1.1, size=sg.shape)).astype(np.float32)
    got = _along_k_model(x, u, sg, bg)
    exact = x.astype(np.float64) @ (u * np.repeat(sg.astype(np.float64), 64, axis=1) + np.repeat(bg.astype(np.float64), 64, axis=1)).T
    err = np.linalg.norm(got - exact, axis=1) / np.linalg.norm(exact, axis=1)
    assert np.all(err <= 2.0 ** -24 * (17.0 / 3.0) ** 0.5 * 1.25)                        # (a row's sample of outputs)
    ref = oracle.qlinear_affine(x[:2], u, sg.ravel(), bg.ravel(), u.shape, layout_nk=True)
    assert rel_err(got[:2], ref) <= TOL_FP32
