"""GPU parity: the tcgen05 Gemm (mgpuMatmulEx16) and the reference entry point mgpuMatmul
against the CPU oracle.  Tolerance for 16-bit tensor-core math: max-rel <= 2e-2, where the
error of an element is divided by max(|ref|, 1e-2 * rms(ref))."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOL = 2e-2


@pytest.fixture(scope="module")
def m(mdc):
    mdc.init()
    return mdc


def _rm(m, dt):
    return oracle.ROUND_F16 if dt == m.F16 else oracle.ROUND_BF16


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (128, 256, 256), (256, 512, 64)])
def test_small_integers_are_exact(m, M, N, K):
    # products and sums of small integers are exact in fp16 x fp16 -> fp32, so any layout,
    # swizzle or descriptor mistake shows up as a hard mismatch
    rng = np.random.default_rng(0)
    a = rng.integers(-3, 4, (M, K)).astype(np.float32)
    w = rng.integers(-2, 3, (K, N)).astype(np.float32)
    got = m.matmul16(a, w, out_dtype=m.F32)
    assert np.array_equal(got, a @ w)


@pytest.mark.parametrize("M,N,K", [(37, 70, 129), (1, 8, 8), (130, 264, 72), (300, 40, 520), (129, 257, 65)])
@pytest.mark.parametrize("dtype_name", ["f16", "bf16"])
def test_ragged_shapes(m, M, N, K, dtype_name):
    dt = m.F16 if dtype_name == "f16" else m.BF16
    rng = np.random.default_rng(1)
    a = rng.standard_normal((M, K)).astype(np.float32)
    w = (0.05 * rng.standard_normal((K, N))).astype(np.float32)
    b = (0.05 * rng.standard_normal(N)).astype(np.float32)
    got = m.matmul16(a, w, bias=b, dtype=dt, out_dtype=m.F32)
    ref = oracle.matmul(a, w, b, round_mode=_rm(m, dt))
    assert oracle.max_rel_err(ref, got) <= TOL


@pytest.mark.parametrize("act", [0, 1, 2, 3])
def test_epilogues(m, act):
    rng = np.random.default_rng(2)
    M, N, K = 200, 328, 192
    a = rng.standard_normal((M, K)).astype(np.float32)
    w = (0.1 * rng.standard_normal((K, N))).astype(np.float32)
    b = (0.1 * rng.standard_normal(N)).astype(np.float32)
    r = rng.standard_normal((M, N)).astype(np.float32)
    got = m.matmul16(a, w, bias=b, residual=r, act=act)
    ref = oracle.matmul(a, w, b, residual=oracle.round_array(r, oracle.ROUND_F16), round_mode=oracle.ROUND_F16,
                        act=act, out_round=oracle.ROUND_F16)
    assert oracle.max_rel_err(ref, got) <= TOL


def test_layer_shapes(m):
    # the four Gemm shapes of one encoder layer at d=768, F=3072 (tokens reduced to 1024)
    rng = np.random.default_rng(3)
    T = 1024
    for K, N in ((768, 2304), (768, 768), (768, 3072), (3072, 768)):
        a = rng.standard_normal((T, K)).astype(np.float32)
        w = (0.02 * rng.standard_normal((K, N))).astype(np.float32)
        got = m.matmul16(a, w)
        ref = oracle.matmul(a, w, round_mode=oracle.ROUND_F16, out_round=oracle.ROUND_F16)
        assert oracle.max_rel_err(ref, got) <= TOL, (K, N)


def test_mgpu_matmul_config(m):
    # BASELINE config: A fp32 [2048,4096] N(0,1), W [4096,4096] N(0,0.02) passed as [K,N], bias N(0,0.02)
    rng = np.random.default_rng(4)
    a = rng.standard_normal((2048, 4096)).astype(np.float32)
    w = (0.02 * rng.standard_normal((4096, 4096))).astype(np.float32)
    b = (0.02 * rng.standard_normal(4096)).astype(np.float32)
    got = m.matmul(a, w, b)
    ref = oracle.matmul(a, w, b, round_mode=oracle.ROUND_F16)
    assert oracle.max_rel_err(ref, got) <= TOL
    t = oracle.diff_table(ref, got)
    assert t["gt_0.1"] == 0


def test_mgpu_matmul_reference_fixtures(m, golden):
    # benchmark/PyTorch/Models/Linear.py in the shape of test/End2End/GPU/linear.mlir
    y = m.activation(m.matmul(golden["lin_x"], golden["lin_w"], golden["lin_b"]), m.ACT_RELU)
    assert y.shape == golden["lin_y"].shape
    ref16 = oracle.matmul(golden["lin_x"], golden["lin_w"], golden["lin_b"], round_mode=oracle.ROUND_F16,
                          act=oracle.ACT_RELU)
    assert oracle.max_rel_err(ref16, y) <= TOL
    # against the fp32 model output the fp16 operand rounding shows: elements near zero are
    # judged against 5 % of the rms (as in tests/test_oracle_golden.py)
    assert oracle.max_rel_err(golden["lin_y"], y, floor_frac=5e-2) <= TOL
    # examples/genonnx.py:52-64: Gemm 20x10 . 10x20 (K not a multiple of 8)
    rng = np.random.default_rng(5)
    a, w = rng.standard_normal((20, 10)).astype(np.float32), rng.standard_normal((10, 20)).astype(np.float32)
    got = m.matmul(a, w, None)
    assert oracle.max_rel_err(oracle.matmul(a, w, round_mode=oracle.ROUND_F16), got) <= TOL


def test_linearity_at_full_size(m):
    # size-independent property: Gemm(a1 + a2) == Gemm(a1) + Gemm(a2) when a1, a2 have
    # disjoint supports (exact in fp16), checked at the full config size without the oracle
    rng = np.random.default_rng(6)
    M, K, N = 2048, 4096, 4096
    a = rng.standard_normal((M, K)).astype(np.float16).astype(np.float32)
    w = (0.02 * rng.standard_normal((K, N))).astype(np.float32)
    a1, a2 = a.copy(), a.copy()
    a1[:, K // 2:] = 0
    a2[:, :K // 2] = 0
    y = m.matmul16(a, w, out_dtype=m.F32)
    y12 = m.matmul16(a1, w, out_dtype=m.F32) + m.matmul16(a2, w, out_dtype=m.F32)
    # equal up to the order of the fp32 accumulation
    assert oracle.max_rel_err(y12, y) <= 5e-3
    assert np.max(np.abs(y12 - y)) <= 1e-4


@pytest.mark.parametrize("M,N,K", [(32768, 768, 64), (1024, 128, 64), (8192, 768, 192)])
def test_narrow_tiles_are_exact(m, M, N, K):
    # shapes for which the library picks 192- or 128-column tiles (fewer wasted tiles in the
    # last wave); small integers again, so the result must match exactly, with every epilogue
    # input in play (bias and residual are integers too)
    rng = np.random.default_rng(7)
    a = rng.integers(-3, 4, (M, K)).astype(np.float32)
    w = rng.integers(-2, 3, (K, N)).astype(np.float32)
    b = rng.integers(-4, 5, N).astype(np.float32)
    r = rng.integers(-8, 9, (M, N)).astype(np.float32)
    ref = a @ w + b + r
    assert np.array_equal(m.matmul16(a, w, bias=b, residual=r), ref)              # 16-bit output
    assert np.array_equal(m.matmul16(a, w, bias=b, residual=r, out_dtype=m.F32), ref)


@pytest.mark.parametrize("M,N,K", [
    (1, 16, 8), (33, 48, 64), (65, 2304, 768),     # rows around a box, one stage, whole K in the ring
    (99, 768, 3072), (250, 768, 4096), (640, 192, 1024),  # long K: the ring goes round
    (641, 1000, 1032), (5, 24, 72), (70, 40, 200), # ragged K: a box per k-block, the last stage partly past K
    (1024, 2304, 768), (2048, 768, 3072), (100, 77, 2048)])
def test_one_wave_tiles_are_exact(m, M, N, K):
    # small integers: fp16 products and fp32 sums are exact in any order of summation, so a wrong
    # tile or stage is a hard mismatch (|sum| <= 4096 * 6 < 2^24)
    rng = np.random.default_rng(11)
    a = rng.integers(-3, 4, (M, K)).astype(np.float32)
    w = rng.integers(-2, 3, (K, N)).astype(np.float32)
    b = rng.integers(-4, 5, N).astype(np.float32)
    r = rng.integers(-8, 9, (M, N)).astype(np.float32)
    ref = a @ w + b
    for _ in range(2):  # again with the plan kept from the first call
        assert np.array_equal(m.matmul16(a, w, bias=b, out_dtype=m.F32), ref)
    assert np.array_equal(m.matmul16(a, w, bias=b, residual=r, out_dtype=m.F32, act=m.ACT_RELU), np.maximum(ref, 0) + r)


@pytest.mark.parametrize("M,N,K", [
    (8, 64, 256), (17, 768, 264), (64, 768, 768), (71, 2304, 768), (129, 768, 3072), (200, 2304, 512),  # boxes of 8 to 64 rows, one tile or several
    (86, 1288, 520), (341, 424, 280), (456, 3136, 256), (1592, 704, 256),  # ragged K, 65 to 128 rows, less than half of the shared memory
    (1375, 1024, 1024), (1101, 1040, 1096)])  # CTA pairs
def test_one_wave_shares_of_rows_are_exact(m, M, N, K):
    # tiles of an equal share of the rows, with accumulators of 64 or 128 rows of which only the box's are stored: exact on
    # small integers, and nothing beside the result is written
    rng = np.random.default_rng(13)
    a, w = rng.integers(-3, 4, (M, K)).astype(np.float32), rng.integers(-2, 3, (K, N)).astype(np.float32)
    b, r = rng.integers(-4, 5, N).astype(np.float32), rng.integers(-8, 9, (M, N)).astype(np.float32)
    ref = np.maximum(a @ w + b, 0) + r
    assert np.array_equal(_matmul16_at(m, a, w, b, r, m.F32, m.ACT_RELU), ref)
    assert np.array_equal(_matmul16_at(m, a, w, b, r, m.F16, m.ACT_RELU), ref.astype(np.float16).astype(np.float32))


@pytest.mark.parametrize("bn", ["192", "128"])
def test_forced_tile_width(bn):
    # every shape of this file again with the tile width forced (read once per process)
    import os
    import subprocess
    import sys
    env = dict(os.environ, MDC_GEMM_BN=bn)
    r = subprocess.run([sys.executable, "-m", "pytest", __file__, "-q", "-m", "gpu", "-x",
                        "-k", "small_integers or ragged or epilogues or narrow"],
                       env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]


@pytest.mark.parametrize("N,K", [(768, 3072), (1000, 1000), (1024, 4096)])
def test_a_row_does_not_depend_on_the_number_of_rows(m, N, K):
    # from 1 row (narrow one-wave tiles) to 6000 (persistent CTA pairs): the same sum over K in the
    # same order, so equal bit for bit
    rng = np.random.default_rng(13)
    a = rng.standard_normal((6000, K)).astype(np.float32)
    w = (0.02 * rng.standard_normal((K, N))).astype(np.float32)
    whole = m.matmul16(a, w, out_dtype=m.F32)
    for M in (1, 16, 99, 128, 250, 512, 1000, 1024, 2048, 4096):
        assert np.array_equal(m.matmul16(a[:M], w, out_dtype=m.F32), whole[:M]), M


def _gelu64(v):
    from math import erf
    v = np.asarray(v, np.float64)
    return 0.5 * v * (1 + np.vectorize(erf)(v / np.sqrt(2.0)))


@pytest.mark.parametrize("M,N,bias_offset", [(70, 33, 0), (19200, 33, 0), (70, 64, 4), (19200, 64, 4)])
def test_gelu_of_ragged_rows_is_exact_to_fp32(m, M, N, bias_offset):
    # rows that cannot be accessed in vectors (an odd width, a bias off its 16-byte boundary) keep the
    # erf form: A . W is one fp16 value, so only the activation's own rounding is left.  erff and the
    # three products around it: 4 roundings of 2^-24 relative to 1 + erf <= 2, on values of rms 0.65:
    # 2-norm error below 1.5e-7 (measured 4e-8; the vector epilogue's fitted form has 7e-7)
    rng = np.random.default_rng(17)
    v = rng.standard_normal(M).astype(np.float16)
    a = np.zeros((M, 64), np.float16)
    a[:, 0] = v
    w = np.zeros((64, N), np.float32)
    w[0] = 1
    b = np.zeros(N + 1, np.float32)
    b[bias_offset // 4 + N - 1] = np.inf  # gelu(inf) is inf, not NaN
    da, dw, db, do = m.to_device(a), m.to_device(w), m.to_device(b), m.DeviceBuffer(M * N * 4)
    dwp = m.DeviceBuffer(N * 64 * 2)
    m.ops().mgpuPackWeight(dw.ptr, dwp.ptr, 64, N, m.F16, None)
    m.ops().mgpuMatmulEx16(da.ptr, dwp.ptr, db.ptr + bias_offset, None, do.ptr, M, N, 64, m.F16, m.F32, m.ACT_GELU_ERF, None)
    got = m.to_host(do, (M, N), np.float32)
    m.check("mgpuMatmulEx16")
    ref = np.repeat(_gelu64(v)[:, None], N - 1, axis=1)
    assert np.linalg.norm(got[:, :-1] - ref) <= 1.5e-7 * np.linalg.norm(ref)
    assert np.all(np.isposinf(got[:, -1]))


def _matmul16_at(m, a, w, b, r, out_dtype, act=0, out_off=0, res_off=0, bias_off=0, repeat=0):
    """mgpuMatmulEx16 with out / residual / bias that many bytes off their allocation; repeat > 0: the
    median time of that many calls in microseconds instead of the result."""
    M, K = a.shape
    N = w.shape[1]
    item = 4 if out_dtype == m.F32 else 2

    def at(arr, nbytes):
        return m.to_device(np.concatenate([np.zeros(nbytes, np.uint8), np.ascontiguousarray(arr).view(np.uint8).ravel()]))
    da, dw, db, dr = m.to_device(a.astype(np.float16)), m.to_device(w), at(b, bias_off), at(r.astype(np.float16), res_off)
    dwp, do = m.DeviceBuffer(N * K * 2), m.DeviceBuffer(M * N * item + 64)
    m.ops().mgpuPackWeight(dw.ptr, dwp.ptr, K, N, m.F16, None)

    def call(stream=None):
        m.ops().mgpuMatmulEx16(da.ptr, dwp.ptr, db.ptr + bias_off, dr.ptr + res_off, do.ptr + out_off, M, N, K, m.F16, out_dtype, act, stream)
    if repeat:
        import torch
        s = torch.cuda.Stream()
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(repeat + 4)]
        m.runtime().mgpuStreamSynchronize(None)
        for e in ev:
            e.record(s)
            call(s.cuda_stream)
        s.synchronize()
        return float(np.median([x.elapsed_time(y) * 1e3 for x, y in zip(ev[3:-1], ev[4:])]))
    rt = m.runtime()
    rt.mgpuMemset32(do.ptr, 0x7fc00000, (M * N * item + 64) // 4, None)
    call()
    raw = m.to_host(do, (M * N * item + 64,), np.uint8)
    assert m.ops().mgpuOpsCheckDeviceStatus(None) == 0
    m.check("mgpuMatmulEx16")
    fill = np.full(16 + M * N * item // 4 + 1, 0x7fc00000, np.uint32).view(np.uint8)
    end = out_off + M * N * item  # nothing beside the result was written
    assert np.array_equal(raw[:out_off], fill[:out_off]) and np.array_equal(raw[end:], fill[end:len(raw)])
    got = raw[out_off:end].view(np.float32 if out_dtype == m.F32 else np.float16).reshape(M, N)
    return got.astype(np.float32)


@pytest.mark.parametrize("offsets", [(0, 0, 0), (16, 0, 0), (0, 16, 0), (16, 16, 0), (0, 0, 4), (4, 2, 0)])
@pytest.mark.parametrize("M,N", [(70, 8), (70, 40), (200, 1000), (20000, 24), (19300, 128), (2500, 2056)])
def test_row_alignments_are_exact(m, M, N, offsets):
    # 32-byte, 16-byte and element-wise rows of both Gemm kernels (one-wave up to 200 rows here,
    # persistent above), with the tail columns of N = 8 mod 16; small integers, so equal bit for bit
    rng = np.random.default_rng(19)
    K = 64
    a = rng.integers(-3, 4, (M, K)).astype(np.float32)
    w = rng.integers(-2, 3, (K, N)).astype(np.float32)
    b = rng.integers(-4, 5, N).astype(np.float32)
    r = rng.integers(-8, 9, (M, N)).astype(np.float32)
    ref = np.maximum(a @ w + b, 0) + r
    oo, ro, bo = offsets
    for out_dtype in (m.F16, m.F32):
        assert np.array_equal(_matmul16_at(m, a, w, b, r, out_dtype, m.ACT_RELU, oo, ro, bo), ref)


@pytest.mark.parametrize("act", [0, 1, 2])
@pytest.mark.parametrize("M,N", [(19001, 16), (19001, 48), (6001, 400), (2499, 2064), (129, 19264)])
def test_rows_stored_in_pairs_are_exact(m, M, N, act):
    # whole-sector rows of the persistent kernel: two lanes store two rows, the last of which may be missing, in pieces of
    # 32 columns, the last of which may hold 16; the residual may be the output itself.  Small integers; GELU of values
    # from 10 is the value itself, and the residual shows what it was added to
    rng = np.random.default_rng(23)
    K = 64
    a, w = rng.integers(0, 4, (M, K)).astype(np.float32), rng.integers(0, 3, (K, N)).astype(np.float32)
    b, r = 10 + rng.integers(0, 5, N).astype(np.float32), rng.integers(-8, 9, (M, N)).astype(np.float32)
    ref = a @ w + b + r
    for out_dtype in (m.F16, m.F32):
        assert np.array_equal(_matmul16_at(m, a, w, b, r, out_dtype, act), ref)
    da, dw, db, do = m.to_device(a.astype(np.float16)), m.to_device(w), m.to_device(b), m.to_device(r.astype(np.float16))
    dwp = m.DeviceBuffer(N * K * 2)
    m.ops().mgpuPackWeight(dw.ptr, dwp.ptr, K, N, m.F16, None)
    m.ops().mgpuMatmulEx16(da.ptr, dwp.ptr, db.ptr, do.ptr, do.ptr, M, N, K, m.F16, m.F16, act, None)
    assert np.array_equal(m.to_host(do, (M, N), np.float16).astype(np.float32), ref)


@pytest.mark.parametrize("M", [70, 19200])
def test_gelu_of_vector_rows(m, M):
    # the fitted form, one wave and persistent: A . W is one fp16 value.  The fit is within 8e-7 absolute and 1.3e-5
    # relative (from -8 on; its exponent, up to 50 in 24 bits, brings another 2e-6 there, and ex2.approx 2^-22), and 6.6e-7
    # in the 2-norm of N(0, 1) arguments, to which fp32 rounding adds 1e-7
    from math import erfc
    gelu = np.vectorize(lambda t: 0.5 * t * erfc(-t / np.sqrt(2.0)))  # (1 + erf loses digits from -4 on)
    rng = np.random.default_rng(47)
    N = 64
    for v, whole in ((rng.standard_normal(M), True), (rng.uniform(-8, 12, M), False)):
        v = v.astype(np.float16)
        v[:3] = 0, -0.0, 6e4
        a, w = np.zeros((M, 64), np.float16), np.zeros((64, N), np.float32)
        a[:, 0], w[0] = v, 1
        a[5, 1], b = np.nan, np.zeros(N, np.float32)
        b[-1] = np.inf
        da, dw, db, do, dwp = m.to_device(a), m.to_device(w), m.to_device(b), m.DeviceBuffer(M * N * 4), m.DeviceBuffer(N * 64 * 2)
        m.ops().mgpuPackWeight(dw.ptr, dwp.ptr, 64, N, m.F16, None)
        m.ops().mgpuMatmulEx16(da.ptr, dwp.ptr, db.ptr, None, do.ptr, M, N, 64, m.F16, m.F32, m.ACT_GELU_ERF, None)
        got = m.to_host(do, (M, N), np.float32)
        m.check("mgpuMatmulEx16")
        assert np.isnan(got[5]).all()
        got, ref = np.delete(got, 5, 0), np.repeat(gelu(np.delete(v, 5).astype(np.float64))[:, None], N - 1, axis=1)
        assert np.all(np.isposinf(got[:, -1]))
        err = np.abs(got[:, :-1] - ref)
        assert np.all(err <= np.minimum(8e-7 + 1.2e-7 * np.abs(ref), 1.6e-5 * np.abs(ref)))
        if whole and M > 10000:  # (of 66 values it depends on which: at most 8e-7 over their rms of 0.6, which the line above says)
            assert np.linalg.norm(err[3:]) <= 7.6e-7 * np.linalg.norm(ref[3:])


@pytest.mark.parametrize("N,offsets", [(1000, (0, 0, 0)), (768, (16, 0, 0)), (768, (0, 16, 0))])
def test_rows_of_16_byte_multiples_are_not_slow(m, N, offsets):
    # against the next width of whole sectors: up to 1.3 times its time, 4 to 10 times when such rows
    # went one element at a time
    rng = np.random.default_rng(23)
    M, K, wide = 32768, 768, (N + 15) // 16 * 16
    a = rng.standard_normal((M, K)).astype(np.float32)
    for out_dtype in (m.F16, m.F32):
        t = []
        for n, off in ((N, offsets), (wide, (0, 0, 0))):
            w = (0.02 * rng.standard_normal((K, n))).astype(np.float32)
            t.append(_matmul16_at(m, a, w, np.zeros(n, np.float32), np.zeros((M, n), np.float32), out_dtype, 0, *off, repeat=20))
        assert t[0] <= 2.5 * t[1], t


def _exact_matmul(m, M, N, K, seed):
    # small integers, so any order of summation is exact and a wrong tile, stage or padding is a hard mismatch
    rng = np.random.default_rng(seed)
    a = rng.integers(-3, 4, (M, K)).astype(np.float32)
    w = rng.integers(-2, 3, (K, N)).astype(np.float32)
    b = rng.integers(-4, 5, N).astype(np.float32)
    assert np.array_equal(m.matmul(a, w, b), a @ w + b)
    assert np.array_equal(m.matmul(a, w, None), a @ w)


@pytest.mark.parametrize("M,N,K", [
    (65, 64, 8), (66, 63, 41), (130, 72, 129), (200, 1000, 136),   # packed rows of 16 k values, and of 8 more
    (128, 4104, 200), (641, 193, 1032), (5000, 264, 72),
    (700, 1000, 1100), (3000, 711, 1500)])                         # both operands in one launch
def test_packed_weights_are_exact(m, M, N, K):
    """Edges of the packing's tiles: 64 columns, 64 k in groups of 16, sectors and half sectors."""
    _exact_matmul(m, M, N, K, 19)


@pytest.mark.parametrize("offset", [0, 16])
@pytest.mark.parametrize("K,N", [(1, 1), (7, 5), (8, 64), (9, 65), (16, 3), (24, 130), (57, 66), (64, 64), (65, 1), (72, 129), (121, 64), (1000, 67)])
def test_packed_rows_on_and_off_sectors(m, K, N, offset):
    """Rows of an odd multiple of 16 bytes start alternately on and inside a 32-byte sector; a weight may be packed to
    any multiple of 16 bytes.  Every value once, zeros in the padding, the neighbours untouched."""
    rng = np.random.default_rng(K * 131 + N)
    w, Kp = rng.standard_normal((K, N)).astype(np.float32), (K + 7) // 8 * 8
    dw, out = m.to_device(w), m.to_device(np.full(N * Kp + 64, 0x5a5a, np.uint16))
    for dtype in (m.F16, m.BF16):
        m.ops().mgpuPackWeight(dw.ptr, out.ptr + 32 + offset, K, N, dtype, None)
        got = m.to_host(out, (N * Kp + 64,), np.uint16)
        m.check("mgpuPackWeight")
        first = 16 + offset // 2
        ref = np.zeros((N, Kp), np.uint16)
        ref[:, :K] = m.encode16(np.ascontiguousarray(w.T), dtype).view(np.uint16)
        assert np.array_equal(got[first:first + N * Kp].reshape(N, Kp), ref)
        assert (got[:first] == 0x5a5a).all() and (got[first + N * Kp:] == 0x5a5a).all()


@pytest.mark.parametrize("M,N,K", [
    (1, 8, 8), (1, 1, 1), (5, 17, 24), (32, 16, 128), (33, 15, 129),    # a stage, its edges, one column tile
    (16, 1000, 2048), (64, 2368, 200), (64, 2369, 200), (3, 4100, 63),  # 16 columns a CTA, 32, odd widths
    (7, 1100, 3210), (40, 2400, 3333), (7, 48, 6001),                   # the ring goes round; a long K that it leaves
    (7, 1760, 3210), (33, 4001, 1999), (2, 5000, 8100), (9, 7402, 130)])  # round with 16 columns, by value, in two waves
def test_few_rows_are_exact(m, M, N, K):
    """Up to 64 rows the weight is read in fp32 by the Gemm itself."""
    _exact_matmul(m, M, N, K, 23)


@pytest.mark.parametrize("offset", [4, 8])
def test_few_rows_off_their_boundaries(m, offset):
    M, N, K = 20, 64, 96
    rng = np.random.default_rng(29)
    a, w = rng.integers(-3, 4, (M, K)).astype(np.float32), rng.integers(-2, 3, (K, N)).astype(np.float32)
    b = rng.integers(-4, 5, N).astype(np.float32)
    pad = np.zeros(offset // 4, np.float32)
    da, dw, db = (m.to_device(np.concatenate([pad, t.ravel()])) for t in (a, w, b))
    do = m.DeviceBuffer(M * N * 4 + 64)
    m.ops().mgpuMatmul(da.ptr + offset, dw.ptr + offset, db.ptr + offset, do.ptr + offset, M, N, K, None)
    got = m.to_host(do, (M * N + 16,), np.float32)[offset // 4:][:M * N].reshape(M, N)
    m.check("mgpuMatmul")
    assert np.array_equal(got, a @ w + b)


@pytest.mark.parametrize("M,N,K", [(1, 1000, 2496), (8, 1000, 2500), (9, 2000, 6000), (17, 1000, 2333), (41, 2400, 7001), (57, 1000, 2499), (64, 2400, 7168),
                                   (8, 2400, 4096), (8, 2400, 5200)])
def test_few_rows_rings_are_exact(m, M, N, K):
    # boxes of 8 to 64 rows, rings of 8 stages to 18 with 16 columns a CTA and of 9 to 21 with 32 that go round, the deepest with
    # the input converted ahead and inside, the last stage partly past K
    rng = np.random.default_rng(53)
    a, w = rng.integers(-3, 4, (M, K)).astype(np.float32), rng.integers(-2, 3, (K, N)).astype(np.float32)
    b = rng.integers(-4, 5, N).astype(np.float32)
    assert np.array_equal(m.matmul(a, w, b), a @ w + b)


@pytest.mark.parametrize("M,N,K", [(2341, 768, 3072), (1711, 1024, 1400), (2399, 720, 1400), (300, 4090, 1408), (2976, 768, 1408), (2977, 768, 1392)])
def test_one_round_of_pairs_is_exact(m, M, N, K):
    # either side of the line between one-wave tiles of 128 columns and one round of the persistent kernel
    rng = np.random.default_rng(59)
    a, w = rng.integers(-3, 4, (M, K)).astype(np.float32), rng.integers(-2, 3, (K, N)).astype(np.float32)
    b, r = rng.integers(-4, 5, N).astype(np.float32), rng.integers(-8, 9, (M, N)).astype(np.float32)
    got = m.matmul16(a, w, bias=b, residual=r, out_dtype=m.F32, act=m.ACT_RELU)
    assert np.array_equal(got, np.maximum(a @ w + b, 0) + r)


@pytest.mark.parametrize("M,N,K", [(366, 337, 64), (1739, 59, 32), (2444, 46, 24), (653, 171, 64), (70, 405, 56), (130, 1, 8), (128, 9, 640)])
@pytest.mark.parametrize("residual", [False, True])
def test_one_wave_rows_stored_by_value_are_exact(m, M, N, K, residual):
    # tiles that are narrow because each value is a store of its own, 16 columns and boxes of 32 to 64 rows among them
    rng = np.random.default_rng(61)
    a, w = rng.integers(-3, 4, (M, K)).astype(np.float32), rng.integers(-2, 3, (K, N)).astype(np.float32)
    b, r = rng.integers(-4, 5, N).astype(np.float32), rng.integers(-8, 9, (M, N)).astype(np.float32)
    got = m.matmul16(a, w, bias=b, residual=r if residual else None, out_dtype=m.F32, act=m.ACT_RELU)
    assert np.array_equal(got, np.maximum(a @ w + b, 0) + (r if residual else 0))


@pytest.mark.parametrize("entry", ["mgpuMatmul", "mgpuMatmulNoAlloc"])
@pytest.mark.parametrize("M,N,K", [(16, 1000, 1024), (40, 2400, 500)])
def test_output_may_overlap_the_weight(m, entry, M, N, K):
    """The whole weight is read before the first store, with few rows too."""
    rng = np.random.default_rng(41)
    a, w = rng.integers(-3, 4, (M, K)).astype(np.float32), rng.integers(-2, 3, (K, N)).astype(np.float32)
    b = rng.integers(-4, 5, N).astype(np.float32)
    da, db, pad = m.to_device(a), m.to_device(b), M * N
    for at in (0, 1, K * N // 2, K * N - 4, -M * N + 4):  # of the output, in floats from the weight
        mem = m.to_device(np.concatenate([np.zeros(pad, np.float32), w.ravel(), np.zeros(pad, np.float32)]))
        first = mem.ptr + 4 * pad
        getattr(m.ops(), entry)(da.ptr, first, db.ptr, first + 4 * at, M, N, K, None)
        got = m.to_host(mem, (M, N), np.float32, offset_bytes=4 * (pad + at))
        assert m.ops().mgpuOpsCheckDeviceStatus(None) == 0
        m.check(entry)
        assert np.array_equal(got, a @ w + b), at


@pytest.mark.parametrize("entry", ["mgpuMatmul", "mgpuMatmulNoAlloc"])
@pytest.mark.parametrize("offset", [0, 4])  # bytes of the input from its boundary: vectors, value by value
@pytest.mark.parametrize("M,N,K", [(1, 17, 255), (1, 17, 257), (8, 1000, 2048), (9, 40, 259), (16, 2400, 768), (16, 2500, 1532), (17, 300, 300),
                                   (32, 2400, 508), (33, 16, 512), (48, 200, 500), (48, 2401, 512), (64, 64, 256)])
def test_few_rows_with_the_input_converted_inside(m, entry, offset, M, N, K):
    """Either side of the line to a launch that converts the input, with tails of rows, columns and K, and with the output
    over the input, which keeps that launch: exact on small integers."""
    rng = np.random.default_rng(M * N + K)
    a, w = rng.integers(-3, 4, (M, K)).astype(np.float32), rng.integers(-2, 3, (K, N)).astype(np.float32)
    b = rng.integers(-4, 5, N).astype(np.float32)
    ref, dw, db = a @ w + b, m.to_device(w), m.to_device(b)
    pad = np.zeros(offset // 4, np.float32)
    mem, out = m.to_device(np.concatenate([pad, a.ravel(), np.zeros(M * N, np.float32)])), m.DeviceBuffer(M * N * 4)
    for dst, at in ((out, 0), (mem, offset), (mem, offset + 4 * (M * K // 2))):
        getattr(m.ops(), entry)(mem.ptr + offset, dw.ptr, db.ptr, dst.ptr + at, M, N, K, None)
        got = m.to_host(dst, (M, N), np.float32, offset_bytes=at)
        assert m.ops().mgpuOpsCheckDeviceStatus(None) == 0
        m.check(entry)
        assert np.array_equal(got, ref)
        m.runtime().mgpuMemcpy(mem.ptr + offset, a.ctypes.data, a.nbytes, None)
        m.runtime().mgpuStreamSynchronize(None)


@pytest.mark.parametrize("entry", ["mgpuMatmul", "mgpuMatmulNoAlloc"])
@pytest.mark.parametrize("M,N,K", [(16, 1000, 1024), (40, 2400, 500)])  # 16 and 32 columns a CTA
def test_few_rows_read_what_is_queued_ahead(m, entry, M, N, K):
    """Nothing waits between the calls: the weight and the bias are written by kernels queued ahead of the Gemm (in
    either order, so that each is directly ahead once) and written again by those behind it."""
    rng = np.random.default_rng(43)
    rt, ops = m.runtime(), m.ops()
    ints = lambda lo, hi, *shape: rng.integers(lo, hi, shape).astype(np.float32)
    a, w0, b0 = ints(-3, 4, M, K), ints(-2, 3, K, N), ints(-4, 5, N)
    dw, db = [ints(-2, 3, K, N) for _ in range(3)], [ints(-4, 5, N) for _ in range(3)]
    da, dw0, db0 = m.to_device(a), m.to_device(w0), m.to_device(b0)
    ddw, ddb = [m.to_device(t) for t in dw], [m.to_device(t) for t in db]
    w, b = m.to_device(np.zeros_like(w0)), m.to_device(np.zeros_like(b0))
    outs = [m.to_device(np.zeros((M, N), np.float32)) for _ in range(12)]
    for stream in (None, rt.mgpuStreamCreate()):
        for i, out in enumerate(outs):
            writes = [(dw0.ptr, ddw[i % 3].ptr, w.ptr, K * N), (db0.ptr, ddb[i % 3].ptr, b.ptr, N)]
            for x, y, z, n in writes if i % 2 else reversed(writes):
                ops.mgpuAdd(x, y, z, n, stream)
            getattr(ops, entry)(da.ptr, w.ptr, b.ptr, out.ptr, M, N, K, stream)
        rt.mgpuStreamSynchronize(stream)
        m.check(entry)
        for i, out in enumerate(outs):
            got = m.to_host(out, (M, N), np.float32)
            assert np.array_equal(got, a @ (w0 + dw[i % 3]) + (b0 + db[i % 3])), i
        assert ops.mgpuOpsCheckDeviceStatus(stream) == 0
        if stream:
            rt.mgpuStreamDestroy(stream)
        for out in outs:
            rt.mgpuMemset32(out.ptr, 0, M * N, None)
        rt.mgpuStreamSynchronize(None)


def test_few_rows_keep_infinities_to_themselves(m):
    # a row or column with an infinity leaves the others alone
    rng = np.random.default_rng(31)
    a, w = rng.standard_normal((9, 300)).astype(np.float32), rng.standard_normal((300, 40)).astype(np.float32)
    clean = m.matmul(a, w, None)
    a2, w2 = a.copy(), w.copy()
    a2[4, 7], w2[200, 13] = np.inf, np.nan
    got = m.matmul(a2, w2, None)
    keep = np.ones_like(clean, bool)
    keep[4, :], keep[:, 13] = False, False
    assert np.array_equal(got[keep], clean[keep])
    assert not np.isfinite(got[4]).any() and np.isnan(got[:, 13]).all()


# 768 x 3072 is never read by the Gemm of a few rows; 1000 x 1000 and 1760 x 3210 are in its form with 16 columns,
# 2400 x 3000 in the one with 32, the latter two with more stages than its ring holds
@pytest.mark.parametrize("N,K", [(768, 3072), (1000, 1000), (72, 333), (1760, 3210), (2400, 3000)])
def test_matmul_rows_do_not_depend_on_their_number(m, N, K):
    # few rows, one wave, CTA pairs: the same sum over K in the same order
    rng = np.random.default_rng(37)
    a = rng.standard_normal((6000, K)).astype(np.float32)
    w = (0.02 * rng.standard_normal((K, N))).astype(np.float32)
    whole = m.matmul(a, w, None)
    for M in (1, 16, 33, 64, 65, 128, 250, 1000, 2048):
        assert np.array_equal(m.matmul(a[:M], w, None), whole[:M]), M
