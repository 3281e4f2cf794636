"""GPU parity of the INT4 / INT8 linear kernels against the CPU restatement of the reference's scalar
kernels (src/kernels/scalar.c:9-41,70-84), through the C ABI (ibcu_linear)."""
import ctypes as C

import numpy as np
import pytest

from libinferbit_b200 import Backend, LinearT, _ffi
from tests import _cpu

pytestmark = pytest.mark.gpu

RTOL, ATOL = 1e-3, 1e-4        # the float bar: |gpu - ref| <= 1e-4 + 1e-3 |ref|


def oracle_linear(libs, w, s16, x, bits):
    M = w.shape[0]; B, N = x.shape
    s = np.empty(M, np.float32); libs.oracle.ibo_fp16_array_to_fp32(s16, s, M)
    out = np.empty((B, M), np.float32)
    if bits == 8:
        libs.oracle.ibo_matmul_int8_batch(out, w, s, x, M, N, B, M)
    else:
        libs.oracle.ibo_matmul_int4_batch(out, w, s, x, M, N, B, M)
    return out


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("M,N,B", [
    (5632, 2048, 1),      # TinyLlama up_proj
    (1024, 4096, 1), (1024, 4096, 4), (1024, 4096, 16),     # k/v proj
    (4096, 4096, 4), (4096, 4096, 16),                      # q/o proj at the batch sizes of the attention configuration
    (512, 4096, 2), (512, 4096, 3), (512, 4096, 8), (256, 4096, 32),
    (4096, 14336, 1),     # down_proj shape
    (100, 320, 5),        # rows not a multiple of the tile, short rows
    (33, 96, 1), (1, 64, 1), (17, 4128, 7),
])
def test_linear_matches_scalar_reference(backend, cpu_libs, bits, M, N, B):
    rng = np.random.default_rng(bits * 7919 + M * 31 + N + B)
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, M, N, B)
    got = backend.linear(w, s16, x, bits)
    want = oracle_linear(cpu_libs, w, s16, x, bits)
    assert _cpu.close(got, want, RTOL, ATOL), float(np.max(np.abs(got - want)))


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("M,N,B", [(4096, 4096, 8), (4096, 4096, 16), (1000, 4096, 11), (130, 256, 8), (4096, 14336, 8), (2048, 14336, 16),
                                   (300, 1152, 9)])
def test_batched_tcgen05_path(backend, cpu_libs, bits, M, N, B):
    """The optional kernel for 8 to 16 activations on the tcgen05 tensor cores (accumulators in tensor memory): against
    the scalar restatement, and against the mma.sync kernel on the same inputs. Both sum exact
    integers; they can differ in the last place only where the columns were split into different numbers of slices."""
    rng = np.random.default_rng(bits * 13 + M + N + B)
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, M, N, B)
    init = rng.standard_normal((B, M)).astype(np.float32)
    want = oracle_linear(cpu_libs, w, s16, x, bits)
    backend.lib.ibcu_linear_use_tcgen05(backend.ctx, 2)
    try:
        before = backend.launches()
        got = backend.linear(w, s16, x, bits)
        assert backend.launches() - before >= (2 if N % 512 == 0 else 1)    # conversion kernel + tcgen05 kernel (+ recombination); other rows take the usual kernel
        assert _cpu.close(got, want, RTOL, ATOL), float(np.max(np.abs(got - want)))
        got_add = backend.linear(w, s16, x, bits, epilogue=1, out_init=init)
        assert np.allclose(got_add, init + got, rtol=1e-6, atol=1e-6 * float(np.abs(got).max()))    # the residual epilogue adds the same product
        backend.lib.ibcu_linear_use_tcgen05(backend.ctx, -1)
        other = backend.linear(w, s16, x, bits)
    finally:
        backend.lib.ibcu_linear_use_tcgen05(backend.ctx, 0)
    assert np.allclose(got, other, rtol=2e-6, atol=1e-6 * float(np.abs(other).max()))
    assert backend.lib.ibcu_sync(backend.ctx) == 0           # no wait inside the kernel ran out


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("M,N,B", [
    (1, 128, 5), (8, 96, 32),           # one row; a single block of columns, partly filled
    (129, 160, 32), (257, 2080, 31),    # one row more than a tile; columns that end inside a block of 128
    (37889, 256, 6), (40001, 128, 32),  # one row more than one pass of 256-row runs over all SMs: a block walks a second run
    (4096, 4096, 1), (1024, 14336, 17), # one activation; a cluster of eight blocks per run
])
def test_tcgen05_linear_edges(backend, cpu_libs, bits, M, N, B):
    """Edges of the tcgen05 kernel's tiles, runs and column parts against the product in double precision. Bound: an activation
    is rounded to half a unit of 2^-29 of its largest magnitude or finer, all sums are exact, the result is rounded to FP32
    twice (before and after the row scale). (The scalar FP32 restatement's own running sum is off by more at 14336 columns.)"""
    rng = np.random.default_rng(bits + M + N + B)
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, M, N, B)
    backend.lib.ibcu_linear_use_tcgen05(backend.ctx, 2)
    try:
        got = backend.linear(w, s16, x, bits)
    finally:
        backend.lib.ibcu_linear_use_tcgen05(backend.ctx, 0)
    v = w.astype(np.float64) if bits == 8 else np.stack([w & 15, w >> 4], axis=-1).reshape(M, N).astype(np.float64) - 8
    sc = s16.view(np.float16).astype(np.float64)
    want = (x.astype(np.float64) @ v.T) * sc
    bound = 2.0 ** -22 * np.abs(want) + 2.0 ** -30 * np.abs(x).max(axis=1, keepdims=True).astype(np.float64) * (np.abs(v).sum(axis=1) * sc)
    assert np.all(np.abs(got - want) <= bound), float(np.max(np.abs(got - want) / bound))


@pytest.mark.parametrize("bits,N", [(8, 1048576 - 128), (8, 1048576), (8, 1048704), (4, 1048576)])
def test_rows_longer_than_s32_sums_hold(backend, bits, N):
    """Weights of -128 times digits of -128 reach 2^31 at 131072 columns of one s32 sum, which eight blocks of a row meet at 1048576 columns.
    Every product is the same number, so the sum is N times it: exact up to the two roundings of the result."""
    M, B = 3, 5
    w = np.full((M, N), -128, np.int8) if bits == 8 else np.zeros((M, N // 2), np.uint8)
    digit = np.float32(64 * 2 ** 24 - 128 * 2 ** 16 - 128 * 2 ** 8)                  # digits 64, -128, -128, 0
    x = np.full((B, N), digit) * np.array([1, -1, 0.5, -0.5, 2], np.float32)[:, None]
    s16 = _cpu.fp16_bits(np.array([2.0 ** -10, 2.0 ** -11, 2.0 ** -12]))
    got = backend.linear(w, s16, x, bits)
    want = x[:, :1].astype(np.float64) * N * (-128 if bits == 8 else -8) * s16.view(np.float16).astype(np.float64)
    assert np.all(np.abs(got - want) <= 2.0 ** -23 * np.abs(want))


@pytest.mark.parametrize("bits", [8, 4])
def test_capture_without_room_for_the_digits(bits):
    """Under capture the digits of the tcgen05 kernel cannot be given more room: the call says so and launches nothing, it does not
    go on with another kernel under a context that holds an error. Afterwards the same call, run once outside, can be captured."""
    rng = np.random.default_rng(bits)
    M, N, B = 64, 2048, 5
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, M, N, B)
    with Backend(0) as be:
        lib = be.lib
        lib.ibcu_linear_use_tcgen05(be.ctx, -1)
        other = be.linear(w, s16, x, bits)                   # the other kernel has its room now, which is less
        lib.ibcu_linear_use_tcgen05(be.ctx, 2)
        dw, ds, dx, do = be.upload(w), be.upload(s16), be.upload(x), be.alloc(B * M * 4)
        t = LinearT(dw.ptr, ds.ptr, do.ptr, M, M, 0, 0)
        call = lambda: lib.ibcu_linear(be.ctx, C.byref(t), 1, dx.ptr, N, B, bits)
        g = C.c_int(-1)
        be._check(lib.ibcu_graph_begin(be.ctx))
        before = be.launches()
        rc, launched, message = call(), be.launches() - before, lib.ibcu_last_error(be.ctx)
        lib.ibcu_clear_error(be.ctx)
        be._check(lib.ibcu_graph_end(be.ctx, C.byref(g)))
        assert rc == -5 and launched == 0 and b"during graph capture" in message
        be._check(call()); be.sync()
        be._check(lib.ibcu_graph_begin(be.ctx))
        be._check(call())
        be._check(lib.ibcu_graph_end(be.ctx, C.byref(g)))
        be._check(lib.ibcu_memset(be.ctx, do.ptr, 0xFF, B * M * 4))
        be._check(lib.ibcu_graph_launch(be.ctx, g.value)); be.sync()
        assert np.allclose(be.download(do, np.float32, B * M).reshape(B, M), other, rtol=2e-6, atol=1e-6 * float(np.abs(other).max()))


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("N", [4096, 4224, 8192, 8320])
def test_row_lengths_converted_in_the_block(backend, cpu_libs, bits, N):
    """The last and first row lengths of the two instances that convert one activation in the block, and of the conversion kernel."""
    rng = np.random.default_rng(N + bits)
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, 70, N, 1)
    assert _cpu.close(backend.linear(w, s16, x, bits), oracle_linear(cpu_libs, w, s16, x, bits), RTOL, ATOL)


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("Ms,N,B", [([2048], 1024, 5), ([2049], 1024, 16), ([1520, 380, 380], 2048, 6), ([2639], 4224, 9)])
def test_tcgen05_rows_around_clusters_of_eight(backend, bits, Ms, N, B):
    """The last row count that clusters of eight blocks take with one tile each, and those that go to clusters of four: the sums of
    the mma.sync kernel, to the last place where that cuts a row into slices."""
    rng = np.random.default_rng(bits + sum(Ms) + N + B)
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, sum(Ms), N, B)
    be = backend
    dw, ds, dx = be.upload(w), be.upload(s16), be.upload(x)
    outs = []
    for mode in (2, -1):
        out, ts, row = be.alloc(B * sum(Ms) * 4), [], 0
        for M in Ms:
            ts.append(LinearT(dw.at(row * N * bits // 8), ds.at(2 * row), out.at(4 * B * row), M, M, 0, 0)); row += M
        be.lib.ibcu_linear_use_tcgen05(be.ctx, mode)
        try:
            be._check(be.lib.ibcu_linear(be.ctx, (LinearT * len(ts))(*ts), len(ts), dx.ptr, N, B, bits))
        finally:
            be.lib.ibcu_linear_use_tcgen05(be.ctx, 0)
        be.sync()
        outs.append(be.download(out, np.float32, B * sum(Ms)))
    assert np.allclose(outs[0], outs[1], rtol=2e-6, atol=1e-6 * float(np.abs(outs[1]).max()))


@pytest.mark.parametrize("M,N,B", [(38000, 1664, 6), (25000, 1920, 32), (3000, 4224, 24), (40000, 1152, 8)])
def test_tcgen05_int4_teams(backend, M, N, B):
    """Odd numbers of 128-column blocks through rings that are used again, over one and two runs of rows: the two teams of
    widening warps change places from run to run. Bound as above."""
    rng = np.random.default_rng(M + N + B)
    w, s16, x = _cpu.make_int4_case(rng, M, N, B)
    got = backend.linear(w, s16, x, 4)
    sc = s16.view(np.float16).astype(np.float64)
    want, mag = np.empty((B, M)), np.empty(M)
    for r in range(0, M, 4096):
        v = np.stack([w[r:r + 4096] & 15, w[r:r + 4096] >> 4], axis=-1).reshape(-1, N).astype(np.float64) - 8
        want[:, r:r + 4096], mag[r:r + 4096] = x.astype(np.float64) @ v.T, np.abs(v).sum(axis=1)
    want *= sc
    bound = 2.0 ** -22 * np.abs(want) + 2.0 ** -30 * np.abs(x).max(axis=1, keepdims=True).astype(np.float64) * (mag * sc)
    assert np.all(np.abs(got - want) <= bound), float(np.max(np.abs(got - want) / bound))


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("M,N,B", [(40, 66, 2), (9, 30, 1), (257, 1000, 3), (64, 4096, 4)])
def test_portable_kernel(backend, cpu_libs, bits, M, N, B):
    """Shapes the tensor-core path does not take (row bytes not a multiple of 16) and the forced
    portable kernel on a shape it does take."""
    rng = np.random.default_rng(M + N)
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, M, N, B)
    got = backend.linear(w, s16, x, bits, force_generic=True)
    want = oracle_linear(cpu_libs, w, s16, x, bits)
    assert _cpu.close(got, want, RTOL, ATOL)
    got2 = backend.linear(w, s16, x, bits)
    assert _cpu.close(got2, want, RTOL, ATOL)


@pytest.mark.parametrize("bits", [8, 4])
def test_unpack_is_exact(backend, bits):
    """One-hot activations read single weights back: out/scale must be the integer itself, for every
    column position modulo 128 and every nibble / byte value."""
    rng = np.random.default_rng(11)
    M, N = 64, 256
    if bits == 8:
        w = rng.integers(-128, 128, size=(M, N), dtype=np.int8)
        w[:, 0] = np.arange(M) - 128; w[:, 1] = np.arange(M) + 64
        vals = w.astype(np.float32)
    else:
        w = rng.integers(0, 256, size=(M, N // 2), dtype=np.uint8)
        w[:16, 0] = np.arange(16) | (np.arange(16)[::-1] << 4)
        vals = np.empty((M, N), np.float32)
        vals[:, 0::2] = (w & 15).astype(np.float32) - 8
        vals[:, 1::2] = (w >> 4).astype(np.float32) - 8
    ones = np.full(M, 0x3C00, np.uint16)                       # fp16 1.0
    for j0 in range(0, N, 32):
        x = np.zeros((32, N), np.float32)
        x[np.arange(32), j0 + np.arange(32)] = 1.0
        got = backend.linear(w, ones, x, bits)                 # [32, M]
        assert np.array_equal(got, vals[:, j0:j0 + 32].T)


@pytest.mark.parametrize("bits", [8, 4])
def test_scales_fp32_and_residual_epilogue(backend, cpu_libs, bits):
    rng = np.random.default_rng(5)
    M, N, B = 200, 512, 4
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, M, N, B)
    want = oracle_linear(cpu_libs, w, s16, x, bits)
    s32 = np.empty(M, np.float32); cpu_libs.oracle.ibo_fp16_array_to_fp32(s16, s32, M)
    assert _cpu.close(backend.linear(w, s32, x, bits), want, RTOL, ATOL)
    base = rng.standard_normal((B, M)).astype(np.float32)
    got = backend.linear(w, s16, x, bits, epilogue=1, out_init=base)
    assert _cpu.close(got, base + want, RTOL, ATOL)


def test_wide_dynamic_range_activations(backend, cpu_libs):
    """Activations spanning six orders of magnitude inside one vector, and huge and tiny vectors: the
    per-slice power-of-two scaling keeps the fixed-point limbs exact enough. The absolute term of the
    bar is scaled by the largest activation, which is what sets the reference's own rounding noise."""
    rng = np.random.default_rng(9)
    M, N = 128, 1024
    w, s16, _ = _cpu.make_int8_case(rng, M, N, 1)
    for scale in (1e-20, 1e-6, 1.0, 3e4, 1e12):
        x = (rng.standard_normal((2, N)) * scale * 10.0 ** rng.integers(-3, 3, (2, N))).astype(np.float32)
        got = backend.linear(w, s16, x, 8)
        want = oracle_linear(cpu_libs, w, s16, x, 8)
        assert _cpu.close(got, want, RTOL, ATOL * float(np.abs(x).max())), scale
    x = np.zeros((1, N), np.float32)
    assert np.array_equal(backend.linear(w, s16, x, 8), np.zeros((1, M), np.float32))


def test_three_tensors_one_launch_with_strided_output(backend, cpu_libs):
    """q, k, v share the activation: one launch, each tensor with its own rows, scales and output
    stride (the reference's M_stride, src/threading.c:373-380)."""
    rng = np.random.default_rng(21)
    N, B = 1024, 4
    Ms = [256, 64, 80]
    be = backend
    x = rng.standard_normal((B, N)).astype(np.float32)
    dx = be.upload(x)
    descs = (LinearT * 3)()
    keep, wants, outs = [], [], []
    for i, M in enumerate(Ms):
        w, s16, _ = _cpu.make_int8_case(rng, M, N, 1)
        wants.append(oracle_linear(cpu_libs, w, s16, x, 8))
        dw, ds = be.upload(w), be.upload(s16)
        stride = M + 8
        do = be.upload(np.full((B, stride), -7.0, np.float32))
        keep += [dw, ds]; outs.append((do, stride))
        descs[i] = LinearT(dw.ptr, ds.ptr, do.ptr, M, stride, 0, 0)
    be._check(be.lib.ibcu_linear(be.ctx, descs, 3, dx.ptr, N, B, 8))
    be.sync()
    for (do, stride), want, M in zip(outs, wants, Ms):
        got = be.download(do, np.float32, B * stride).reshape(B, stride)
        assert _cpu.close(got[:, :M], want, RTOL, ATOL)
        assert np.all(got[:, M:] == -7.0)                      # padding untouched


def test_gate_up_silu(backend, cpu_libs):
    rng = np.random.default_rng(22)
    M, N, B = 300, 512, 2
    be = backend
    x = rng.standard_normal((B, N)).astype(np.float32)
    wg, sg, _ = _cpu.make_int4_case(rng, M, N, 1)
    wu, su, _ = _cpu.make_int4_case(rng, M, N, 1)
    g = oracle_linear(cpu_libs, wg, sg, x, 4); u = oracle_linear(cpu_libs, wu, su, x, 4)
    want = np.empty_like(g)
    for b in range(B):
        cpu_libs.oracle.ibo_silu_mul(want[b], g[b], u[b], M)
    dx = be.upload(x)
    descs = (LinearT * 2)()
    og, ou = be.alloc(B * M * 4), be.alloc(B * M * 4)
    descs[0] = LinearT(be.upload(wg).ptr, be.upload(sg).ptr, og.ptr, M, M, 0, 0)
    descs[1] = LinearT(be.upload(wu).ptr, be.upload(su).ptr, ou.ptr, M, M, 0, 0)
    be._check(be.lib.ibcu_linear_gate_up_silu(be.ctx, descs, dx.ptr, N, B, 4))
    be.sync()
    got = be.download(og, np.float32, B * M).reshape(B, M)
    assert _cpu.close(got, want, 2e-3, 2e-4)


def test_bad_arguments_are_refused(backend):
    be = backend
    d = be.alloc(1024)
    t = LinearT(d.ptr, d.ptr, d.ptr, 4, 4, 0, 0)
    assert be.lib.ibcu_linear(be.ctx, C.byref(t), 1, d.ptr, 64, 1, 3) == -1       # bits
    assert b"bits" in be.lib.ibcu_last_error(be.ctx)
    assert be.lib.ibcu_status(be.ctx) == -1
    be.lib.ibcu_clear_error(be.ctx)
    assert be.lib.ibcu_linear(be.ctx, C.byref(t), 1, d.ptr, 64, 33, 8) == -1      # B > IB_BATCH_MAX
    be.lib.ibcu_clear_error(be.ctx)
    assert be.lib.ibcu_linear(be.ctx, C.byref(t), 1, d.ptr, 63, 1, 4) == -1       # odd N for nibbles
    be.lib.ibcu_clear_error(be.ctx)
    assert be.lib.ibcu_linear(be.ctx, C.byref(t), 0, d.ptr, 64, 1, 8) == -1
    be.lib.ibcu_clear_error(be.ctx)
    assert be.lib.ibcu_status(be.ctx) == 0


@pytest.mark.parametrize("N,B,M", [(128, 3, 70), (4096, 3, 70), (200, 3, 70), (14336, 1, 333), (4096, 8, 512), (2048, 11, 100),
                                   (4096, 1, 4096)])
def test_w4a8_route_bit_exact(backend, cpu_libs, N, B, M):
    """Activation quantiser (src/threading.c:401-432) and INT4 x INT8 kernel (src/kernels/scalar.c:43-124):
    integer work, so the bar is bit-exact, including the FP32 accumulation order. Whole groups of 128 columns
    take the tensor-core kernel (more than 8 activations in chunks of 8), N = 200 the row-per-warp kernel;
    both are also run against each other."""
    rng = np.random.default_rng(N + B)
    be = backend
    x = rng.standard_normal((B, N)).astype(np.float32)
    if B >= 3:
        x[1, :64] = 0; x[2, :] *= 1e-12
    groups = (N + 127) // 128
    q = np.empty((B, N), np.int8); sa = np.empty((B, groups), np.float32)
    for b in range(B):
        cpu_libs.oracle.ibo_quantize_input_int8_g128(x[b], q[b], sa[b], N)
    dx = be.upload(x); dq = be.alloc(B * N); dsa = be.alloc(B * groups * 4)
    be._check(be.lib.ibcu_quantize_input_int8_g128(be.ctx, dx.ptr, dq.ptr, dsa.ptr, N, B)); be.sync()
    assert np.array_equal(be.download(dq, np.int8, B * N).reshape(B, N), q)
    assert np.array_equal(be.download(dsa, np.float32, B * groups).reshape(B, groups), sa)
    w = rng.integers(0, 256, size=(M, N // 2), dtype=np.uint8)
    s16 = _cpu.fp16_bits(rng.uniform(0.002, 0.02, M))
    sw = np.empty(M, np.float32); cpu_libs.oracle.ibo_fp16_array_to_fp32(s16, sw, M)
    want = np.empty((B, M), np.float32)
    cpu_libs.oracle.ibo_matmul_w4a8_batch(want, w, sw, q, sa, M, N, B, M)
    do = be.alloc(B * M * 4)
    t = LinearT(be.upload(w).ptr, be.upload(s16).ptr, do.ptr, M, M, 0, 0)
    be._check(be.lib.ibcu_linear_w4a8(be.ctx, C.byref(t), dq.ptr, dsa.ptr, N, B)); be.sync()
    assert np.array_equal(be.download(do, np.float32, B * M).reshape(B, M), want)
    do3 = be.alloc(B * M * 4)                               # quantiser and matvec in one call from the FP32 activations
    t3 = LinearT(t.w, t.scales, do3.ptr, M, M, 0, 0)
    be._check(be.lib.ibcu_linear_w4a8_fp32(be.ctx, C.byref(t3), dx.ptr, N, B)); be.sync()
    assert np.array_equal(be.download(do3, np.float32, B * M).reshape(B, M), want)
    be.lib.ibcu_linear_force_generic(be.ctx, 1)             # the row-per-warp kernel on the same inputs
    try:
        do2 = be.alloc(B * M * 4)
        t2 = LinearT(t.w, t.scales, do2.ptr, M, M, 0, 0)
        be._check(be.lib.ibcu_linear_w4a8(be.ctx, C.byref(t2), dq.ptr, dsa.ptr, N, B)); be.sync()
        assert np.array_equal(be.download(do2, np.float32, B * M).reshape(B, M), want)
    finally:
        be.lib.ibcu_linear_force_generic(be.ctx, 0)


@pytest.mark.parametrize("bits,N", [(8, 1024), (4, 2048), (8, 200)])
def test_prologues_rmsnorm_and_silu_mul(backend, cpu_libs, bits, N):
    """RMSNorm (fp16 weights) and silu(x)*x2 folded into the call equal the separate scalar kernels
    (src/kernels/scalar.c:126-138,175-181) followed by the matvec; N = 200 takes the portable path."""
    from libinferbit_b200 import _ffi
    rng = np.random.default_rng(bits + N)
    be, o = backend, cpu_libs.oracle
    M, B = 96, 3
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, M, N, B)
    x *= 3.0
    x2 = rng.standard_normal((B, N)).astype(np.float32)
    nw16 = _cpu.fp16_bits(rng.uniform(0.9, 1.1, N)); nw = np.empty(N, np.float32); o.ibo_fp16_array_to_fp32(nw16, nw, N)
    dw, ds, dx, dx2, dn, do = be.upload(w), be.upload(s16), be.upload(x), be.upload(x2), be.upload(nw16), be.alloc(B * M * 4)
    t = LinearT(dw.ptr, ds.ptr, do.ptr, M, M, 0, 0)
    for op in (1, 2):
        xin = np.empty_like(x)
        for b in range(B):
            if op == 1:
                o.ibo_rmsnorm(xin[b], x[b], nw, 1e-5, N)
            else:
                o.ibo_silu_mul(xin[b], x[b], x2[b], N)
        want = oracle_linear(cpu_libs, w, s16, xin, bits)
        pro = _ffi.PrologueT(op, dx2.ptr, dn.ptr, 1e-5)
        be._check(be.lib.ibcu_linear_ex(be.ctx, C.byref(t), 1, dx.ptr, N, B, bits, C.byref(pro)))
        be.sync()
        got = be.download(do, np.float32, B * M).reshape(B, M)
        assert _cpu.close(got, want, 2e-3, 2e-4), op


@pytest.mark.parametrize("bits,M,N,B,parts", [(4, 96, 14336, 1, 28), (8, 80, 4096, 2, 7), (4, 64, 2048, 3, 5), (8, 48, 200, 2, 3), (8, 40, 40960, 1, 16)])
def test_silu_mul_amax_then_known_max_prologue(backend, cpu_libs, bits, M, N, B, parts):
    """ibcu_silu_mul_amax followed by a linear call told max|x| (IBCU_PRO_KNOWN_MAX) gives bit for bit what the
    silu(x)*x2 prologue gives: same activation values, same maximum, hence the same fixed-point operand.
    The pieces written by the element-wise step are checked against numpy."""
    from libinferbit_b200 import _ffi
    rng = np.random.default_rng(bits * 1000 + N + B)
    be, o = backend, cpu_libs.oracle
    w, s16, g = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, M, N, B)
    g *= 2.0
    u = rng.standard_normal((B, N)).astype(np.float32)
    dw, ds, dg, du = be.upload(w), be.upload(s16), be.upload(g), be.upload(u)
    dh, da, do1, do2 = be.alloc(B * N * 4), be.alloc(B * parts * 4), be.alloc(B * M * 4), be.alloc(B * M * 4)
    t1, t2 = LinearT(dw.ptr, ds.ptr, do1.ptr, M, M, 0, 0), LinearT(dw.ptr, ds.ptr, do2.ptr, M, M, 0, 0)
    p_silu = _ffi.PrologueT(2, du.ptr, None, 0.0, None, 0)
    be._check(be.lib.ibcu_linear_ex(be.ctx, C.byref(t1), 1, dg.ptr, N, B, bits, C.byref(p_silu)))
    be._check(be.lib.ibcu_silu_mul_amax(be.ctx, dh.ptr, dg.ptr, du.ptr, N, B, da.ptr, parts))
    p_known = _ffi.PrologueT(3, None, None, 0.0, da.ptr, parts)
    be._check(be.lib.ibcu_linear_ex(be.ctx, C.byref(t2), 1, dh.ptr, N, B, bits, C.byref(p_known)))
    be.sync()
    h = be.download(dh, np.float32, B * N).reshape(B, N)
    want_h = np.empty_like(h)
    for b in range(B):
        o.ibo_silu_mul(want_h[b], g[b], u[b], N)
    assert _cpu.close(h, want_h, 1e-5, 1e-6)
    am = be.download(da, np.float32, B * parts).reshape(B, parts)
    chunk = (N + parts - 1) // parts
    for b in range(B):
        for p in range(parts):
            seg = np.abs(h[b, p * chunk:(p + 1) * chunk])
            assert am[b, p] == (seg.max() if seg.size else 0.0)
    got1 = be.download(do1, np.float32, B * M).reshape(B, M)
    got2 = be.download(do2, np.float32, B * M).reshape(B, M)
    if N % 16 == 0:                       # the tensor-core path: identical fixed-point operands
        assert np.array_equal(got1, got2)
    assert _cpu.close(got2, oracle_linear(cpu_libs, w, s16, want_h, bits), 2e-3, 2e-4)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("M,N,parts", [(64, 128, 3), (300, 2048, 5), (96, 14336, 28)])
def test_known_max_of_two_activations(backend, bits, M, N, parts):
    """A block that converts two activations with a known maximum one after the other gives bit for bit what two calls with one
    give: the digit sums of the first are added up before the second overwrites their scratch."""
    from libinferbit_b200 import _ffi
    rng = np.random.default_rng(bits + M + N)
    be, B = backend, 2
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, M, N, B)
    am = np.stack([[np.abs(p).max() for p in np.array_split(row, parts)] for row in x]).astype(np.float32)
    dw, ds, dx, da = be.upload(w), be.upload(s16), be.upload(x), be.upload(am)
    both, one = be.alloc(B * M * 4), be.alloc(B * M * 4)
    for out, b0, n in ((both, 0, 2), (one, 0, 1), (one, 1, 1)):
        t = LinearT(dw.ptr, ds.ptr, out.at(4 * b0 * M), M, M, 0, 0)
        pro = _ffi.PrologueT(3, None, None, 0.0, da.at(4 * b0 * parts), parts)
        for _ in range(20 if n == 2 else 1):
            be._check(be.lib.ibcu_linear_ex(be.ctx, C.byref(t), 1, dx.at(4 * b0 * N), N, n, bits, C.byref(pro)))
    be.sync()
    assert np.array_equal(be.download(both, np.float32, B * M), be.download(one, np.float32, B * M))


@pytest.mark.parametrize("bits,Ms,N,B", [
    (8, [7, 250, 3], 512, 1),            # ragged tensors: runs of rows never cross a tensor, tiles shorter than 16 rows
    (4, [1, 2, 5000, 33], 1024, 2),      # four tensors, one of them larger than the whole grid's worth of 4-row runs
    (8, [4096, 1024, 1024], 4096, 1),    # the q,k,v launch of the headline step
    (4, [14336, 14336], 4096, 1),        # the gate,up launch of the 7B decode step
    (8, [0, 64, 0], 256, 3),             # empty shards (a rank that owns no rows of a tensor)
])
def test_several_tensors_with_ragged_rows(backend, cpu_libs, bits, Ms, N, B):
    rng = np.random.default_rng(bits + sum(Ms) + N)
    be = backend
    x = rng.standard_normal((B, N)).astype(np.float32)
    dx = be.upload(x)
    n = len(Ms)
    descs = (LinearT * n)()
    keep, wants, outs = [], [], []
    for i, M in enumerate(Ms):
        Mr = max(M, 1)
        w, s16, _ = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, Mr, N, 1)
        wants.append(oracle_linear(cpu_libs, w, s16, x, bits)[:, :M])
        dw, ds = be.upload(w), be.upload(s16)
        do = be.upload(np.full((B, Mr), -3.0, np.float32))
        keep += [dw, ds]; outs.append(do)
        descs[i] = LinearT(dw.ptr, ds.ptr, do.ptr, M, Mr, 0, 0)
    be._check(be.lib.ibcu_linear(be.ctx, descs, n, dx.ptr, N, B, bits))
    be.sync()
    for do, want, M in zip(outs, wants, Ms):
        Mr = max(M, 1)
        got = be.download(do, np.float32, B * Mr).reshape(B, Mr)
        assert _cpu.close(got[:, :M], want, RTOL, ATOL), (M, float(np.max(np.abs(got[:, :M] - want))) if M else 0)
        if M == 0:
            assert np.all(got == -3.0)


@pytest.mark.parametrize("bits,M,N,B", [(8, 32000, 4096, 1), (8, 48, 65536, 2), (4, 40, 131072, 1), (8, 200, 16384, 6)])
def test_full_size_head_and_rows_longer_than_shared_memory(backend, cpu_libs, bits, M, N, B):
    """The LM-head shape against the scalar restatement, and rows whose limbs do not fit one block's shared
    memory (columns split over several blocks, integer partial sums recombined by linear_finalize_kernel)."""
    rng = np.random.default_rng(bits * 13 + M + N + B)
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, M, N, B)
    got = backend.linear(w, s16, x, bits)
    want = oracle_linear(cpu_libs, w, s16, x, bits)
    assert _cpu.close(got, want, RTOL, ATOL * max(1.0, float(np.abs(want).max()))), float(np.max(np.abs(got - want)))


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,G,K_out,eps", [
    (4096, 4096, 128, 0, 0.0),        # attention projection of the 7B shape, groups of 128
    (5632, 2048, 64, 8, 0.0),         # TinyLlama up_proj shape with eight outlier columns per row
    (4099, 14336, 32, 0, 0.0),        # rows not a multiple of the four a warp carries; rows longer than one pass of the lanes
    (1000, 4096, 128, 16, 0.05),      # groups under 5 % of the largest activation are left out
    (33, 96, 32, 3, 0.0), (40, 48, 16, 2, 0.0), (17, 200, 8, 0, 0.2),   # small shapes; the last two take the generic kernel
])
def test_group_scaled_int4_rows(backend, cpu_libs, M, N, G, K_out, eps):
    """Group-scaled INT4 rows of the reference's session engine (src/pq_decode.c:3565-3651; skip rule :3854-3882) against
    their restatement (parity unpinned: static functions in the reference), within the float bar."""
    rng = np.random.default_rng(M + N + G + K_out)
    q, s, x, oi, ov = _cpu.make_int4g_case(rng, M, N, G, K_out)
    if eps:
        x[: N // 4] *= 1e-3                                   # a quarter of the groups fall under the threshold
    got = backend.int4g_matmul(q, s, G, x, oi, ov, eps)
    want = _cpu.oracle_int4g(cpu_libs.oracle, q, s, G, x, oi, ov, eps)
    assert _cpu.close(got, want, RTOL, ATOL), float(np.max(np.abs(got - want)))
    if eps:                                                   # the rule is visible: without it the result differs
        full = _cpu.oracle_int4g(cpu_libs.oracle, q, s, G, x, oi, ov, 0.0)
        assert not np.array_equal(full, want)
    assert np.array_equal(got, backend.int4g_matmul(q, s, G, x, oi, ov, eps))       # same bits again
    # linearity at full size: f(2x) = 2 f(x) exactly (every product and sum scales by a power of two)
    assert np.array_equal(backend.int4g_matmul(q, s, G, 2.0 * x, oi, ov, eps), 2.0 * got)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,G", [(17, 128, 128), (1, 14336, 128), (300, 160, 32), (4737, 1088, 64), (2000, 2112, 64), (9473, 1024, 32),
                                   (700, 4096, 512), (513, 3072, 1024), (65, 6144, 2048), (5000, 11008, 128), (641, 16384, 32), (33, 3232, 32)])
def test_group_scaled_int4_on_the_tensor_cores(backend, cpu_libs, M, N, G):
    """Tiles of 16 and 32 rows with a remainder, k-blocks that end inside a group or hold several, row scales that start in the middle of
    a word (an odd number of groups), groups of several k-blocks."""
    rng = np.random.default_rng(M * 7 + N + G)
    q, s, x, oi, ov = _cpu.make_int4g_case(rng, M, N, G, 0)
    got = backend.int4g_matmul(q, s, G, x, oi, ov, 0.0)
    want = _cpu.oracle_int4g(cpu_libs.oracle, q, s, G, x, oi, ov, 0.0)
    assert _cpu.close(got, want, RTOL, ATOL), float(np.max(np.abs(got - want)))
    assert np.array_equal(got, backend.int4g_matmul(q, s, G, x, oi, ov, 0.0))
    assert np.array_equal(backend.int4g_matmul(q, s, G, 2.0 * x, oi, ov, 0.0), 2.0 * got)


@pytest.mark.gpu
@pytest.mark.parametrize("N", [32, 2048, 2080, 8192, 8224, 16384, 16416])
def test_group_scaled_int4_row_lengths(backend, cpu_libs, N):
    """Where the kernels change how they hold the activation: one and several groups of eight columns per thread, the last length of each register
    instance and the first one of the next; 2048 columns and fewer, and 16416, by dp4a, the others on the tensor cores."""
    rng = np.random.default_rng(N)
    q, s, x, oi, ov = _cpu.make_int4g_case(rng, 50, N, 32, 0)
    got = backend.int4g_matmul(q, s, 32, x, oi, ov, 0.0)
    want = _cpu.oracle_int4g(cpu_libs.oracle, q, s, 32, x, oi, ov, 0.0)
    assert _cpu.close(got, want, RTOL, ATOL), float(np.max(np.abs(got - want)))


@pytest.mark.gpu
@pytest.mark.parametrize("K_out,eps,G", [(3, 0.0, 32), (0, 0.02, 32), (3, 0.02, 32), (0, 0.0, 96), (5, 0.0, 96)])
@pytest.mark.parametrize("N", [32, 2080, 8192, 8224, 12000, 16384, 16416])
def test_group_scaled_int4_row_lengths_of_the_dp4a_kernel(backend, cpu_libs, N, K_out, eps, G):
    """The same lengths with what keeps a call off the tensor cores: outlier columns, the skip rule, groups of 96."""
    N = -(-N // 96) * 96 if G == 96 else N
    rng = np.random.default_rng(N + K_out + G)
    q, s, x, oi, ov = _cpu.make_int4g_case(rng, 51, N, G, K_out)
    if eps:
        x[: N // 4] *= 1e-3
    got = backend.int4g_matmul(q, s, G, x, oi, ov, eps)
    want = _cpu.oracle_int4g(cpu_libs.oracle, q, s, G, x, oi, ov, eps)
    assert _cpu.close(got, want, RTOL, ATOL), float(np.max(np.abs(got - want)))
    assert np.array_equal(backend.int4g_matmul(q, s, G, 2.0 * x, oi, ov, eps), 2.0 * got)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,G", [(4736, 1024, 64), (4737, 1024, 64), (4750, 160, 32), (4737, 128, 128), (4800, 96, 32), (1184, 2048, 32), (1185, 2048, 32), (1184, 2080, 32),
                                   (14208, 12320, 32), (14209, 12320, 32), (14209, 12288, 32), (15, 4096, 128), (16, 4096, 64), (2369, 4096, 256), (4753, 4096, 32)])
def test_group_scaled_int4_kernel_by_size(backend, cpu_libs, M, N, G):
    """Both sides of the lines between the two kernels, short rows on the tensor cores, and runs of 16 rows a block with a remainder."""
    rng = np.random.default_rng(M + N + G)
    q, s, x, oi, ov = _cpu.make_int4g_case(rng, M, N, G, 0)
    got = backend.int4g_matmul(q, s, G, x, oi, ov, 0.0)
    want = _cpu.oracle_int4g(cpu_libs.oracle, q, s, G, x, oi, ov, 0.0)
    assert _cpu.close(got, want, RTOL, ATOL), float(np.max(np.abs(got - want)))
    assert np.array_equal(backend.int4g_matmul(q, s, G, 2.0 * x, oi, ov, 0.0), 2.0 * got)


@pytest.mark.parametrize("bits,Ms,N,B,tc", [
    (8, [1408] * 3, 1408, 7, False), (4, [1152, 128, 128], 1152, 6, False),      # few short rows: the preparation launch does not pay
    (8, [4096] * 3, 4096, 2, False), (8, [2048, 512, 512], 2048, 3, False),
    (8, [14336], 4096, 4, True), (4, [14336, 14336], 4096, 3, True), (8, [4096], 14336, 3, True), (8, [4096, 1024, 1024], 4096, 8, True),
    (8, [64], 512, 17, True), (8, [32000], 4096, 1, False),
])
def test_linear_kernel_by_cost(backend, bits, Ms, N, B, tc):
    """Which kernel a call takes by itself: the launches and the bits are those of the call that is told to."""
    rng = np.random.default_rng(bits + sum(Ms) + N + B)
    be = backend
    w = rng.integers(0, 256, sum(Ms) * N * bits // 8, dtype=np.uint8)
    s16, x = _cpu.fp16_bits(rng.uniform(0.001, 0.01, sum(Ms))), rng.standard_normal((B, N)).astype(np.float32)
    dw, ds, dx = be.upload(w), be.upload(s16), be.upload(x)

    def run(mode):
        out, ts, row = be.alloc(B * sum(Ms) * 4), [], 0
        for M in Ms:
            ts.append(LinearT(dw.at(row * N * bits // 8), ds.at(2 * row), out.at(4 * B * row), M, M, 0, 0)); row += M
        be.lib.ibcu_linear_use_tcgen05(be.ctx, mode)
        try:
            before = be.launches()
            be._check(be.lib.ibcu_linear(be.ctx, (LinearT * len(ts))(*ts), len(ts), dx.ptr, N, B, bits))
            n = be.launches() - before
        finally:
            be.lib.ibcu_linear_use_tcgen05(be.ctx, 0)
        be.sync()
        got = be.download(out, np.float32, B * sum(Ms)); out.free(); be._bufs.remove(out)
        return n, got

    n, got = run(0)
    want_n, want = run(2 if tc else -1)
    assert n == want_n and np.array_equal(got, want)
    if tc:
        assert n == 2


@pytest.mark.parametrize("M,N,B", [(130, 5 * 128, 2), (4096, 9 * 128, 7), (4000, 14336, 32), (2600, 6432, 12), (300, 23 * 128, 32), (40000, 11 * 128, 3),
                                   (16000, 2048, 4), (16000, 2048, 17), (9000, 15 * 128, 18), (9000, 15 * 128, 19), (6000, 1024, 8), (6000, 1024, 9), (4000, 14336, 3)])
def test_tcgen05_int4_four_teams(backend, M, N, B):
    """Runs of one tile: blocks of columns that are not a multiple of the two or four teams of widening warps, rings shorter than a part of the
    columns, clusters of one to eight blocks (40000 rows: two tiles, two teams, several runs a block); the last seven: both sides of the line between
    two teams and four. Bound as above."""
    rng = np.random.default_rng(M + N + B)
    w, s16, x = _cpu.make_int4_case(rng, M, N, B)
    backend.lib.ibcu_linear_use_tcgen05(backend.ctx, 2)
    try:
        got = backend.linear(w, s16, x, 4)
    finally:
        backend.lib.ibcu_linear_use_tcgen05(backend.ctx, 0)
    sc = s16.view(np.float16).astype(np.float64)
    v = np.stack([w & 15, w >> 4], axis=-1).reshape(M, N).astype(np.float32) - 8
    want = (x.astype(np.float64) @ v.T.astype(np.float64)) * sc
    bound = 2.0 ** -22 * np.abs(want) + 2.0 ** -30 * np.abs(x).max(axis=1, keepdims=True).astype(np.float64) * (np.abs(v).sum(axis=1, dtype=np.float64) * sc)
    assert np.all(np.abs(got - want) <= bound), float(np.max(np.abs(got - want) / bound))


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("op", ["plain", "norm", "silu"])
@pytest.mark.parametrize("N,B", [(32, 17), (2048, 32), (2080, 5), (4128, 17), (6176, 32), (8224, 18), (16384, 20), (16416, 17)])
def test_tcgen05_digits_prepared_by_clusters(backend, bits, op, N, B):
    """Digits by one to eight blocks per activation (the last length: one block): parts that end inside the last 128 columns or have none, every
    prologue; without one, as many rows as leave runs to clusters of less than eight, which the preparation by clusters needs there. Bound: the prologue rounds an activation to FP32 a few times (silu: exponential, division, product; the norm's sum of squares is a
    tree of at most 8 + 5 + 3 + 3 additions), 32 units in the last place hold all of it; the rest as above."""
    M, be = 70, backend
    if op == "plain":
        M, B = 2700, max(B, 21)
    rng = np.random.default_rng(N + B + bits)
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, M, N, B)
    x2 = rng.standard_normal((B, N)).astype(np.float32)
    nw = _cpu.fp16_bits(rng.uniform(0.2, 3.0, N))
    x64 = x.astype(np.float64)
    act = {"plain": x64, "silu": x64 / (1.0 + np.exp(-x64)) * x2,
           "norm": x64 / np.sqrt((x64 ** 2).mean(axis=1, keepdims=True) + float(np.float32(1e-5))) * nw.view(np.float16).astype(np.float64)}[op]
    dw, ds, dx, dx2, dn, do = be.upload(w), be.upload(s16), be.upload(x), be.upload(x2), be.upload(nw), be.upload(np.zeros((B, M), np.float32))
    t = LinearT(dw.ptr, ds.ptr, do.ptr, M, M, 0, 0)
    pro = _ffi.PrologueT()
    pro.op, pro.x2, pro.norm_w, pro.eps = {"plain": 0, "norm": 1, "silu": 2}[op], dx2.ptr, dn.ptr, 1e-5
    be.lib.ibcu_linear_use_tcgen05(be.ctx, 2)
    try:
        be._check(be.lib.ibcu_linear_ex(be.ctx, C.byref(t), 1, dx.ptr, N, B, bits, C.byref(pro)))
    finally:
        be.lib.ibcu_linear_use_tcgen05(be.ctx, 0)
    be.sync()
    got = be.download(do, np.float32, B * M).reshape(B, M)
    v = w.astype(np.float64) if bits == 8 else np.stack([w & 15, w >> 4], axis=-1).reshape(M, N).astype(np.float64) - 8
    sc = s16.view(np.float16).astype(np.float64)
    want = (act @ v.T) * sc
    bound = 2.0 ** -22 * np.abs(want) + 2.0 ** -30 * np.abs(act).max(axis=1, keepdims=True) * (np.abs(v).sum(axis=1) * sc) + 32 * 2.0 ** -24 * (np.abs(act) @ np.abs(v).T) * sc
    assert np.all(np.abs(got - want) <= bound), float(np.max(np.abs(got - want) / bound))


@pytest.mark.parametrize("bits,M,N,B", [(8, 1024, 3072, 5), (4, 1024, 4096, 5), (8, 1024, 1024, 2)])
def test_several_products_take_the_tcgen05_kernel(bits, M, N, B):
    """silu(x) * x2 of several activations, where an estimate without it takes the mma.sync kernel. The digits of the tcgen05 kernel take more room than
    those of the other: in a context that has run the other kernel, a capture of the call by itself has none and says so."""
    rng = np.random.default_rng(N + B)
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, M, N, B)
    with Backend(0) as be:
        dw, ds, dx, do = be.upload(w), be.upload(s16), be.upload(x), be.alloc(B * M * 4)
        t = LinearT(dw.ptr, ds.ptr, do.ptr, M, M, 0, 0)
        pro = _ffi.PrologueT(); pro.op, pro.x2 = 2, dx.ptr

        def captured(mode):
            be.lib.ibcu_linear_use_tcgen05(be.ctx, mode)
            gid = C.c_int(-1)
            be._check(be.lib.ibcu_graph_begin(be.ctx))
            rc = be.lib.ibcu_linear_ex(be.ctx, C.byref(t), 1, dx.ptr, N, B, bits, C.byref(pro))
            rc_end = be.lib.ibcu_graph_end(be.ctx, C.byref(gid))
            be.lib.ibcu_clear_error(be.ctx)
            return rc or rc_end

        be.lib.ibcu_linear_use_tcgen05(be.ctx, -1)
        be._check(be.lib.ibcu_linear_ex(be.ctx, C.byref(t), 1, dx.ptr, N, B, bits, C.byref(pro))); be.sync()
        assert captured(-1) == 0
        assert captured(0) != 0


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("op", ["plain", "norm", "silu"])
@pytest.mark.parametrize("N", [2048, 5152])
def test_rows_without_an_ordinary_maximum_through_clusters(backend, bits, op, N):
    """Activations of zeros, with Inf, with NaN, and with magnitudes whose squares overflow: digits by clusters give what the other kernel's conversion
    gives for them, to the bit (their maximum, scale and digits do not hang on the order of a sum; two activations a call, of which that kernel
    cuts no row into slices), and leave the other activations alone: 32 units in the last place of the largest result, as above."""
    M, B, be = 2700, 22, backend
    rng = np.random.default_rng(N + bits)
    w, s16, x = (_cpu.make_int8_case if bits == 8 else _cpu.make_int4_case)(rng, M, N, B)
    x2 = rng.standard_normal((B, N)).astype(np.float32)
    x[0] = 0.0
    x[3, N - 1] = np.inf; x[4, 0] = -np.inf; x[5, N // 2] = np.nan; x[6, 5] = np.nan; x[6, N - 3] = np.inf
    x[8] *= 1e25; x[9, 77] = 3e38; x[10] = np.nan; x[11] = np.inf
    x2[13, 3] = np.inf; x2[14, N - 2] = np.nan; x2[15] = 0.0
    odd = [0, 3, 4, 5, 6, 8, 9, 10, 11] + ([13, 14, 15] if op == "silu" else [])
    dw, ds, dx, dx2 = be.upload(w), be.upload(s16), be.upload(x), be.upload(x2)
    dn = be.upload(_cpu.fp16_bits(rng.uniform(0.2, 3.0, N)))
    got = {}
    for mode, group in ((-1, 2), (2, B)):
        do = be.upload(np.full((B, M), 7.0, np.float32))
        be.lib.ibcu_linear_use_tcgen05(be.ctx, mode)
        try:
            for b in range(0, B, group):
                t = LinearT(dw.ptr, ds.ptr, do.at(4 * b * M), M, M, 0, 0)
                pro = _ffi.PrologueT()
                pro.op, pro.x2, pro.norm_w, pro.eps = {"plain": 0, "norm": 1, "silu": 2}[op], dx2.at(4 * b * N), dn.ptr, 1e-5
                be._check(be.lib.ibcu_linear_ex(be.ctx, C.byref(t), 1, dx.at(4 * b * N), N, group, bits, C.byref(pro)))
        finally:
            be.lib.ibcu_linear_use_tcgen05(be.ctx, 0)
        be.sync()
        got[mode] = be.download(do, np.float32, B * M).reshape(B, M)
    assert np.array_equal(got[2][odd], got[-1][odd], equal_nan=True)
    rest = [b for b in range(B) if b not in odd]
    scale = np.abs(got[-1][rest]).max(axis=1, keepdims=True)
    assert np.all(np.abs(got[2][rest] - got[-1][rest]) <= 32 * 2.0 ** -24 * scale)
