"""The routes the automatic variant of the GEMM takes for small, narrow and long-k products: blocks on their own, operands
converted in registers, 192-column tiles, divided k-loops and their reduction — at the edges of tiles and divisions, with the
epilogue, for operands TMA can and cannot address, against the oracle at the bounds of the numeric modes."""
import ctypes as C
import math
import os
import subprocess
import sys

import numpy as np
import pytest

from spoc_b200 import Vector, _lib as L, dims1d, dims2d, run_vectors, sarek_ir
from tests import oracle_lib as O
from tests.gpu_util import CANARY, Dev, dev_from, gemm
from tests.test_gpu_gemm import tol

pytestmark = pytest.mark.gpu

MODES = [L.MODE_3XTF32, L.MODE_TF32, L.MODE_3XF16, L.MODE_F16]


def describe(mode, M, N, K, addressable):
    out = C.create_string_buffer(256)
    assert L.load().sb200_gemm_describe(mode, M, N, K, addressable, 148, out, 256) == 0
    return out.value.decode()


# (M, N, K): one row and the whole height of a block; k just at and beyond a division; ragged everything
SHAPES = [(1, 8, 1024), (64, 256, 1028), (65, 132, 1000), (128, 64, 2080), (17, 33, 1025), (300, 100, 4100), (129, 700, 513),
          (64, 64, 32), (63, 61, 31), (257, 191, 2049)]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("aligned", [True, False], ids=["aligned", "unaligned"])
def test_automatic_routes_match_the_oracle(backend, device, mode, shape, aligned):
    M, N, K = shape
    lda, ldb, ldd = ((x + 3) // 4 * 4 + 4 if aligned else x + 1 - x % 2 for x in (K, N, N))
    rng = np.random.default_rng(M + N + K)
    a, b, c = (rng.uniform(-1, 1, (r, ld)).astype(np.float32) for r, ld in ((M, lda), (K, ldb), (M, ldd)))
    bias = rng.uniform(-0.1, 0.1, N).astype(np.float32)
    A, B, Cm, Bi = (dev_from(backend, device, x.ravel()) for x in (a, b, c, bias))
    D = Dev(backend, device, M * ldd)
    try:
        gemm(backend, device, mode, M, N, K, A, B, D, alpha=1.5, C_=Cm, beta=0.5, bias=Bi, act=1, lda=lda, ldb=ldb, ldc=ldd, ldd=ldd)
        got = D.download().reshape(M, ldd)
        ref = O.gemm(np.ascontiguousarray(a[:, :K]).ravel(), np.ascontiguousarray(b[:, :N]).ravel(), M, N, K, 1.5, 0.5,
                     np.ascontiguousarray(c[:, :N]).ravel(), bias, 1)
        # the clamp halves the reference's mean square, alpha scales the error: as in the other epilogue tests
        assert O.gemm_rel_error(got[:, :N], ref) <= tol(mode, K) * 1.5 * math.sqrt(2), describe(mode, M, N, K, int(aligned))
        assert np.all(got[:, N:] == CANARY)
    finally:
        for x in (A, B, Cm, Bi, D):
            x.free()


@pytest.mark.parametrize("mode", [L.MODE_3XTF32, L.MODE_TF32])
@pytest.mark.parametrize("shape", [(64, 64, 64), (33, 100, 200), (64, 512, 480)])
def test_operands_converted_in_registers_give_the_bits_of_the_panels(backend, device, mode, shape):
    """The same parts summed in the same order (no k-loop here is divided): aligned quads, single elements, prepared panels."""
    M, N, K = shape
    a, b = O.fill(M * K, 61, 1), O.fill(K * N, 61, 2)
    a[5] = np.float32(3.4028234e38) if mode == L.MODE_TF32 else a[5]     # rounds to infinity: no low part may come of it
    A, B, D = dev_from(backend, device, a), dev_from(backend, device, b), Dev(backend, device, M * N)
    A1, B1 = dev_from(backend, device, a, offset=1), dev_from(backend, device, b, offset=1)
    try:
        backend.set_gemm_variant(3)
        gemm(backend, device, mode, M, N, K, A, B, D)
        want = D.download()
        backend.set_gemm_variant(0)
        assert "splits=1 " in describe(mode, M, N, K, 1) and "splits=1 " in describe(mode, M, N, K, 0)
        for x, y in ((A, B), (A1, B1)):
            D.clear()
            gemm(backend, device, mode, M, N, K, x, y, D)
            assert np.array_equal(D.download().view(np.uint32), want.view(np.uint32))
    finally:
        backend.set_gemm_variant(0)
        for x in (A, B, A1, B1, D):
            x.free()


def test_192_column_tiles_match_the_256_column_ones(backend, device):
    M, N, K = 1536, 2044, 256
    assert "tile=256x192" in describe(L.MODE_3XTF32, M, N, K, 1)
    a, b = O.fill(M * K, 62, 1), O.fill(K * N, 62, 2)
    A, B, D = dev_from(backend, device, a), dev_from(backend, device, b), Dev(backend, device, M * N)
    try:
        for mode in (L.MODE_3XTF32, L.MODE_3XF16):
            gemm(backend, device, mode, M, N, K, A, B, D)
            got = D.download()
            assert L.load().sb200_set_gemm_tile_n(256) == 0
            D.clear()
            gemm(backend, device, mode, M, N, K, A, B, D)
            assert L.load().sb200_set_gemm_tile_n(0) == 0
            assert np.array_equal(D.download(), got)
    finally:
        L.load().sb200_set_gemm_tile_n(0)
        for x in (A, B, D):
            x.free()


# (mode, M, N, K, aligned, splits): the blocks or pairs of one cluster share a k-loop; one row, rows and columns that end within
# a block's share, shares of unequal length, a last block with a shorter k-loop, two to eight items
CLUSTERS = [(L.MODE_TF32, 1, 8, 1024, True, 4), (L.MODE_TF32, 64, 256, 1028, True, 4), (L.MODE_TF32, 65, 132, 1000, True, 4),
            (L.MODE_3XTF32, 17, 33, 1025, False, 4), (L.MODE_3XTF32, 128, 64, 2080, False, 8), (L.MODE_3XTF32, 257, 191, 2049, True, 4),
            (L.MODE_3XTF32, 581, 118, 819, True, 3), (L.MODE_3XTF32, 71, 1411, 1414, True, 4), (L.MODE_TF32, 236, 3528, 4165, True, 4),
            (L.MODE_3XF16, 36, 3162, 1876, True, 2), (L.MODE_F16, 842, 98, 2240, True, 4)]


@pytest.mark.parametrize("mode,M,N,K,aligned,splits", CLUSTERS)
def test_k_loops_divided_within_a_cluster(backend, device, mode, M, N, K, aligned, splits):
    text = describe(mode, M, N, K, int(aligned))
    assert f"splits={splits} " in text
    a, b, c = O.fill(M * K, 63, 1), O.fill(K * N, 63, 2), O.fill(M * N, 63, 3)
    bias = O.fill(N, 63, 4, kind=1)
    off = 0 if aligned else 1
    pad = lambda x, cols: np.ascontiguousarray(np.pad(x.reshape(-1, cols), ((0, 0), (0, -cols % 4)))).ravel() if aligned else x   # noqa: E731
    A, B = dev_from(backend, device, pad(a, K), offset=off), dev_from(backend, device, pad(b, N), offset=off)
    lda, ldb = (K + -K % 4, N + -N % 4) if aligned else (K, N)
    Cm, Bi, D = dev_from(backend, device, c), dev_from(backend, device, bias), Dev(backend, device, M * N)
    try:
        first = None
        for _ in range(3):
            D.clear()
            gemm(backend, device, mode, M, N, K, A, B, D, alpha=1.5, C_=Cm, beta=0.5, bias=Bi, act=1, lda=lda, ldb=ldb, ldc=N, ldd=N)
            got = D.download()
            first = got.copy() if first is None else first
            assert np.array_equal(got.view(np.uint32), first.view(np.uint32))     # the order of the sums is fixed
        ref = O.gemm(a, b, M, N, K, 1.5, 0.5, c, bias, 1)
        assert O.gemm_rel_error(got.reshape(M, N), ref) <= tol(mode, K) * 1.5 * math.sqrt(2), text
    finally:
        for x in (A, B, Cm, Bi, D):
            x.free()


# the edges of a block's 64 rows, of the eight blocks' runs, of the 32-column strips, and of the range of K
@pytest.mark.parametrize("mode", [L.MODE_3XF16, L.MODE_F16])
@pytest.mark.parametrize("M,N,K", [(5, 1, 1), (40, 31, 64), (33, 36, 65), (64, 64, 513), (70, 97, 1000), (9, 32, 4095), (20, 100, 4096), (20, 100, 4097)])
@pytest.mark.parametrize("aligned", [True, False], ids=["aligned", "unaligned"])
def test_column_maxima_of_the_fp16_panels_are_found_wherever_they_lie(backend, device, mode, M, N, K, aligned):
    """Every column of B has one element 2^30 times the others, in a row of its own: with a scale from any smaller maximum its fp16
    part would be infinite."""
    rng = np.random.default_rng(K)
    lda, ldb = (((x + 3) // 4 * 4 if aligned else x + 1 - x % 2) for x in (K, N))
    a, b = rng.uniform(-1, 1, (M, lda)).astype(np.float32), rng.uniform(-1, 1, (K, ldb)).astype(np.float32)
    cols = np.arange(N)
    b[(cols * 37 + K - 1) % K, cols] = np.ldexp(1.5, 30).astype(np.float32)
    A, B, D = dev_from(backend, device, a.ravel()), dev_from(backend, device, b.ravel()), Dev(backend, device, M * N)
    try:
        gemm(backend, device, mode, M, N, K, A, B, D, lda=lda, ldb=ldb, ldd=N)
        got = D.download().reshape(M, N)
        ref = O.gemm(np.ascontiguousarray(a[:, :K]).ravel(), np.ascontiguousarray(b[:, :N]).ravel(), M, N, K)
        assert O.gemm_rel_error(got, ref) <= tol(mode, K)
    finally:
        for x in (A, B, D):
            x.free()


GROWING_SCRATCH = """
import ctypes as C
import numpy as np
from spoc_b200 import Backend, _lib as L
from tests import oracle_lib as O
from tests.gpu_util import Dev, dev_from, gemm
from tests.test_gpu_gemm import tol

M, N, K, mode = 455, 1149, 6946, L.MODE_TF32
backend = Backend()
backend.Device.init()
device, lib = backend.Device.get(0), L.load()
a, b = O.fill(M * K, 71, 1), O.fill(K * N, 71, 2)
# the scratch as large as the first block (256 rows, its k-loop divided within clusters) needs it, and no room behind it to grow into
A, B, D = dev_from(backend, device, a[:256 * K]), dev_from(backend, device, b), Dev(backend, device, 256 * N)
assert lib.sb200_set_gemm_tile_n(256) == 0
gemm(backend, device, mode, 256, N, K, A, B, D)
assert lib.sb200_set_gemm_tile_n(0) == 0
fence = [Dev(backend, device, 1 << 20) for _ in range(16)]
d = np.empty(M * N, np.float32)
ptr = lambda x: x.ctypes.data_as(C.c_void_p)
assert lib.sb200_gemm_f32_host(device.id, mode, M, N, K, ptr(a), K, ptr(b), N, ptr(d), N, 1.0, None, 0, 0.0, None, 0) == 0
err = O.gemm_rel_error(d.reshape(M, N), O.gemm(a, b, M, N, K))
assert err <= tol(mode, K), err
"""


def test_a_row_block_that_needs_more_scratch_still_finds_b():
    """The second of this product's row blocks (199 rows) keeps the sums of its divided k-loop in global memory, so it needs more
    scratch than the first, which left the copy of B there: growing the scratch loses the copy.  A process of its own: whatever
    ran before it here has grown the scratch already."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = subprocess.run([sys.executable, "-c", GROWING_SCRATCH], cwd=root, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]


CAPTURED_FIRST = """
import numpy as np
from cuda.bindings import runtime as rt
from spoc_b200 import Backend, _lib as L
from tests import oracle_lib as O
from tests.gpu_util import Dev, dev_from
from tests.test_gpu_gemm import tol

ok = rt.cudaError_t.cudaSuccess
backend = Backend()
backend.Device.init()
device, lib = backend.Device.get(0), L.load()
err, stream = rt.cudaStreamCreateWithFlags(rt.cudaStreamNonBlocking)
assert err == ok
captured = []
for mode in (L.MODE_TF32, L.MODE_3XTF32):
    for m, n, k in ((130, 130, 120), (449, 449, 449), (300, 300, 301)):     # the first one in front of the captures: kernels are loaded
        a, b = O.fill(m * k, 77, 1), O.fill(k * n, 77, 2)
        A, B, D = dev_from(backend, device, a, offset=1), dev_from(backend, device, b, offset=1), Dev(backend, device, m * n)
        args = (mode, m, n, k, A.ptr, k, B.ptr, n, D.ptr, n, 1.0, 0, 0, 0.0, 0, 0)
        if k != 120:
            assert rt.cudaStreamBeginCapture(stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)[0] == ok
        rc = lib.sb200_gemm_f32(device.id, int(stream), *args)
        assert rc == 0, lib.sb200_last_error_string()
        if k != 120:
            err, graph = rt.cudaStreamEndCapture(stream)
            assert err == ok
            err, run = rt.cudaGraphInstantiate(graph, 0)
            assert err == ok and rt.cudaGraphLaunch(run, stream)[0] == ok
        assert rt.cudaStreamSynchronize(stream)[0] == ok
        got = D.download()
        err = O.gemm_rel_error(got.reshape(m, n), O.gemm(a, b, m, n, k))
        assert err <= tol(mode, k), err
        captured.append((args, got, D, A, B))
for args, got, D, *_ in captured:       # with a scratch, by copies
    D.clear()
    assert lib.sb200_gemm_f32(device.id, 0, *args) == 0
    backend.Device.synchronize(device)
    assert np.array_equal(D.download().view(np.uint32), got.view(np.uint32))
"""


def test_unaligned_products_can_be_captured_before_there_is_any_scratch():
    """Copied where there is a scratch to copy into, converted in registers, with the same bits, where a capture keeps it from growing.  A
    process of its own, in which nothing has sized the scratch."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = subprocess.run([sys.executable, "-c", CAPTURED_FIRST], cwd=root, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]


# (form, grid, block, m, n, k): launches that compute the first rows (and part of the next one), or the first rows and columns, of a
# product whose k-loop is divided
PARTIAL = [("naive", (37 * 4096 + 100, 1), 1, 64, 4096, 4096), ("naive", (5 * 300 + 7, 1), 1, 40, 300, 2000), ("tiled", (75, 3), 16, 64, 4096, 4096),
           ("tiled", (2, 2), 16, 1024, 96, 3000), ("naive", (100 * 4096, 1), 1, 128, 4096, 4096), ("tiled", (11, 6), 16, 96, 1056, 4000)]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("form,grid,side,m,n,k", PARTIAL)
def test_a_partial_launch_has_the_bits_of_the_whole(backend, device, mode, form, grid, side, m, n, k):
    ir = (sarek_ir.matmul_tiled_ir if form == "tiled" else sarek_ir.matmul_naive_ir)()
    assert "splits=1 " not in describe(mode, m, n, k, 1)
    va, vb = Vector(backend, O.fill(m * k, 72, 1)), Vector(backend, O.fill(k * n, 72, 2))
    scalars = [("int32", m), ("int32", n), ("int32", k)]
    block = dims2d(side, side)
    whole = dims2d((n + 15) // 16, (m + 15) // 16) if form == "tiled" else dims1d(m * n)
    out = []
    backend.set_mode(mode)
    try:
        for g in (whole, dims2d(*grid)):
            vd = Vector.create(backend, m * n)
            run_vectors(backend, device=device, ir=ir, args=[va, vb, vd] + scalars, block=block, grid=g)
            out.append(vd.to_array().reshape(m, n).copy())
            vd.free()
    finally:
        backend.set_mode(L.MODE_3XTF32)
        va.free()
        vb.free()
    if form == "naive":
        covered = grid[0]
        assert np.array_equal(out[1].ravel()[:covered].view(np.uint32), out[0].ravel()[:covered].view(np.uint32))
        assert not out[1].ravel()[covered:].any()
    else:
        rows, cols = min(m, grid[1] * side), min(n, grid[0] * side)
        assert np.array_equal(out[1][:rows, :cols].view(np.uint32), out[0][:rows, :cols].view(np.uint32))
        assert not out[1][rows:].any() and not out[1][:, cols:].any()


# (mode, M, N, K, aligned, how the operands are read): converted, read in place, split on chip, copied, panels in one launch and in two, with
# the k-loop whole, divided within clusters and divided through global memory
KERNELS = [(L.MODE_3XTF32, 64, 64, 64, True, "converted"), (L.MODE_3XTF32, 64, 8192, 8192, True, "converted"), (L.MODE_3XTF32, 64, 4096, 4096, True, "split"), (L.MODE_TF32, 65, 33, 100, False, "converted"),
           (L.MODE_3XTF32, 512, 512, 512, True, "split"), (L.MODE_3XTF32, 8192, 4096, 512, True, "direct"), (L.MODE_3XTF32, 128, 4095, 1025, False, "copied+split"), (L.MODE_TF32, 512, 512, 512, True, "direct"), (L.MODE_TF32, 128, 96, 4096, True, "direct"),
           (L.MODE_3XTF32, 700, 900, 1000, False, "copied"), (L.MODE_TF32, 455, 1149, 6946, False, "copied"), (L.MODE_3XF16, 300, 200, 500, True, "panels"),
           (L.MODE_F16, 300, 200, 5000, False, "panels"), (L.MODE_3XMIXED, 512, 512, 512, True, "mixed")]


@pytest.mark.parametrize("mode,M,N,K,aligned,operands", KERNELS)
def test_the_described_kernels_are_the_ones_launched(backend, device, mode, M, N, K, aligned, operands):
    off = 0 if aligned else 1
    A, B, D = Dev(backend, device, M * K, offset=off), Dev(backend, device, K * N, offset=off), Dev(backend, device, M * N)
    lib = L.load()
    lib.sb200_set_mixed_min_macs(1 << 20)
    try:
        out = C.create_string_buffer(256)
        assert lib.sb200_gemm_describe(mode, M, N, K, int(aligned), device.sm_count, out, 256) == 0
        text = out.value.decode()
        before = backend.launch_count()
        gemm(backend, device, mode, M, N, K, A, B, D)
        assert f" operands={operands} " in text and text.endswith(f" kernels={backend.launch_count() - before}"), text
        backend.Device.synchronize(device)
    finally:
        lib.sb200_set_mixed_min_macs(0)
        for x in (A, B, D):
            x.free()


# (M, N, K): rows and columns at the edges of 64- and 128-row blocks and of every tile width, pairs whose second block has no rows, k-loops
# shorter than, as long as and one beyond the rings, k that ends within a k-block, more tiles than pairs, the last two with the ordinary
# epilogue, whose staging tiles lie where the loads of the next tile land
SPLIT = [(1, 4, 65), (64, 64, 96), (63, 68, 100), (65, 64, 96), (128, 128, 256), (129, 60, 257), (257, 516, 288), (300, 1000, 300), (512, 64, 512),
         (1536, 2044, 260), (2048, 2052, 68), (2304, 2304, 520), (3000, 2001, 1000), (2305, 2303, 776)]


@pytest.mark.parametrize("M,N,K", SPLIT)
@pytest.mark.parametrize("epilogue", [False, True], ids=["plain", "epilogue"])
def test_operands_split_on_chip_give_the_bits_of_the_panels(backend, device, M, N, K, epilogue):
    lda, ldb, ldd = ((x + 3) // 4 * 4 + 4 for x in (K, N, N))
    rng = np.random.default_rng(M + N + K)
    a, b, c = (rng.uniform(-1, 1, (r, ld)).astype(np.float32) for r, ld in ((M, lda), (K, ldb), (M, ldd)))
    a[0, 0], b[0, 0] = np.float32(2.0 ** -130), np.float32(2.0 ** 100)     # a subnormal element, and one that dwarfs the rest
    a[M - 1, 1] = np.float32(3.4028234e38)                                # rounds to infinity: no low part may come of it
    A, B, Cm, Bi = (dev_from(backend, device, x.ravel()) for x in (a, b, c, c[0, :N].copy()))
    D = Dev(backend, device, M * ldd)
    kw = dict(alpha=1.5, C_=Cm, beta=0.5, bias=Bi, act=1, ldc=ldd) if epilogue else {}
    out = []
    try:
        text = describe(L.MODE_3XTF32, M, N, K, 1)
        assert "splits=1 " in text and text.endswith("operands=split kernels=1")     # the k-loop is not divided; nothing is prepared
        for variant in (3, 0):
            backend.set_gemm_variant(variant)
            D.clear()
            gemm(backend, device, L.MODE_3XTF32, M, N, K, A, B, D, lda=lda, ldb=ldb, ldd=ldd, **kw)
            out.append(D.download().reshape(M, ldd))
        assert np.array_equal(out[0][:, :N].view(np.uint32), out[1][:, :N].view(np.uint32))
        assert np.all(out[1][:, N:] == CANARY)
    finally:
        backend.set_gemm_variant(0)
        for x in (A, B, Cm, Bi, D):
            x.free()


@pytest.mark.parametrize("M,N,K", [(64, 4096, 4096), (64, 4096, 1024), (128, 4096, 4096), (128, 1024, 4096), (1024, 1024, 1024), (256, 2048, 4096), (2304, 2304, 520)])
def test_operands_split_on_chip_give_the_same_bits_every_time(backend, device, M, N, K):
    """Stages that are written again while a warp still reads them show here: operands in L2 and not, launches alone and in a row."""
    a, b = O.fill(M * K, 74, 1), O.fill(K * N, 74, 2)
    A, B = dev_from(backend, device, a), dev_from(backend, device, b)
    D, other = Dev(backend, device, M * N), Dev(backend, device, 40 << 20)
    try:
        assert " operands=split " in describe(L.MODE_3XTF32, M, N, K, 1)
        first = None
        for i in range(12):
            if i % 3 == 1:
                other.clear()
            for _ in range(1 + i % 2):
                gemm(backend, device, L.MODE_3XTF32, M, N, K, A, B, D)
            got = D.download().view(np.uint32)
            first = got if first is None else first
            assert np.array_equal(got, first)
        assert O.gemm_rel_error(first.view(np.float32).reshape(M, N), O.gemm(a, b, M, N, K)) <= tol(L.MODE_3XTF32, K)
    finally:
        for x in (A, B, D, other):
            x.free()


# (M, N, K, offset, padding): the copies of unaligned operands split on chip, by single blocks of 64 and 128 rows and both tile widths
@pytest.mark.parametrize("M,N,K,off,pad", [(52, 5537, 331, 1, 0), (63, 70, 290, 0, 1), (114, 9, 259, 3, 0), (103, 2181, 711, 2, 3), (121, 10213, 577, 1, 0),
                                           (25, 9589, 439, 0, 2)])
def test_copies_split_on_chip_give_the_bits_of_the_panels(backend, device, M, N, K, off, pad):
    lda, ldb = K + pad, N + pad
    rng = np.random.default_rng(M + N + K)
    A, B = (dev_from(backend, device, rng.uniform(-1, 1, n).astype(np.float32), offset=off) for n in ((M - 1) * lda + K, (K - 1) * ldb + N))
    D, out = Dev(backend, device, M * N), []
    try:
        text = describe(L.MODE_3XTF32, M, N, K, 0)
        assert " operands=copied+split " in text and "splits=1 " in text
        for variant in (3, 0):
            backend.set_gemm_variant(variant)
            D.clear()
            gemm(backend, device, L.MODE_3XTF32, M, N, K, A, B, D, lda=lda, ldb=ldb)
            out.append(D.download())
        assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
    finally:
        backend.set_gemm_variant(0)
        for x in (A, B, D):
            x.free()


# copies of rows that start 1, 2 and 3 elements behind a 16-byte boundary and at all four in turn; a thread copies a quad of a row: lengths
# that end 0, 1, 2 and 3 elements into one; a matrix of which only one operand needs the copy
@pytest.mark.parametrize("mode", [L.MODE_3XTF32, L.MODE_TF32])
@pytest.mark.parametrize("M,N,K,off,pad", [(600, 513, 259, 1, 1), (1030, 1021, 513, 2, 0), (260, 1021, 516, 3, 2), (1025, 1030, 511, 3, 4), (1100, 514, 260, 0, 3)])
def test_copied_rows_give_the_bits_of_the_panels(backend, device, mode, M, N, K, off, pad):
    lda, ldb = K + pad, N + pad
    rng = np.random.default_rng(M + N + K)
    A, B = (dev_from(backend, device, rng.uniform(-1, 1, n).astype(np.float32), offset=off) for n in ((M - 1) * lda + K, (K - 1) * ldb + N))
    D, out = Dev(backend, device, M * N), []
    try:
        text = describe(mode, M, N, K, 0)
        assert " operands=copied " in text and "splits=1 " in text
        for variant in (3, 0):
            backend.set_gemm_variant(variant)
            D.clear()
            gemm(backend, device, mode, M, N, K, A, B, D, lda=lda, ldb=ldb)
            out.append(D.download())
        assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
    finally:
        backend.set_gemm_variant(0)
        for x in (A, B, D):
            x.free()


def test_tf32_up_to_128_rows_in_single_blocks_match_pairs(backend, device):
    for M, N, K in ((65, 2048, 1028), (100, 1024, 1024), (128, 4096, 4096), (128, 96, 16384)):
        A, B = (dev_from(backend, device, O.fill(n, 75, i)) for i, n in ((1, M * K), (2, K * N)))
        D = Dev(backend, device, M * N)
        try:
            text = describe(L.MODE_TF32, M, N, K, 1)
            assert text.startswith("single direct") and "workspace=0" in text
            gemm(backend, device, L.MODE_TF32, M, N, K, A, B, D)
            got = D.download()
            backend.set_gemm_variant(2)
            gemm(backend, device, L.MODE_TF32, M, N, K, A, B, D)
            want = D.download()
            # two float32 sums of the same rounded products in another order: 7e-9 of the result a term (the accumulator truncates)
            assert np.linalg.norm(got - want) <= (1e-5 + 1e-8 * K) * np.linalg.norm(want)
        finally:
            backend.set_gemm_variant(0)
            for x in (A, B, D):
                x.free()


@pytest.mark.parametrize("M,N,K", [(455, 1149, 6946), (600, 100, 3001), (700, 1001, 1003), (1100, 301, 2050), (390, 2001, 3003)])
def test_row_blocks_of_unaligned_host_operands_by_different_kernels(backend, device, M, N, K):
    """The blocks of one host-operand product may be split on chip over copies or read beside panels of low parts: what one leaves in the
    scratch is no preparation for the other."""
    a, b, d = O.fill(M * K, 76, 1), O.fill(K * N, 76, 2), np.empty(M * N, np.float32)
    ptr = lambda x: x.ctypes.data_as(C.c_void_p)   # noqa: E731
    lib = L.load()
    assert lib.sb200_gemm_f32_host(device.id, L.MODE_3XTF32, M, N, K, ptr(a), K, ptr(b), N, ptr(d), N, 1.0, None, 0, 0.0, None, 0) == 0
    assert O.gemm_rel_error(d.reshape(M, N), O.gemm(a, b, M, N, K)) <= tol(L.MODE_3XTF32, K)
