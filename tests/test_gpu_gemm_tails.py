"""Rows past the end of A, which have boxes of their own, and k-loops that the second choice divides within clusters."""
import ctypes as C
import math

import numpy as np
import pytest

from spoc_b200 import _lib as L
from spoc_b200.plugin import _check
from tests import oracle_lib as O
from tests import test_gpu_gemm_routes as routes
from tests.gpu_util import CANARY, Dev, dev_from, gemm
from tests.test_gpu_gemm import tol

pytestmark = pytest.mark.gpu

MODES = [L.MODE_3XTF32, L.MODE_TF32, L.MODE_3XF16, L.MODE_F16]


def describe(mode, M, N, K, addressable):
    out = C.create_string_buffer(256)
    assert L.load().sb200_gemm_describe(mode, M, N, K, addressable, 148, out, 256) == 0
    return out.value.decode()


def check(backend, device, mode, M, N, K, lda, ldb, ldd, ldc, noalloc=False):
    rng = np.random.default_rng(M + N + K)
    a, b, c = (rng.uniform(-1, 1, (r, ld)).astype(np.float32) for r, ld in ((M, lda), (K, ldb), (M, ldc)))
    bias = rng.uniform(-0.1, 0.1, N).astype(np.float32)
    A, B, Cm, Bi = (dev_from(backend, device, x.ravel()) for x in (a, b, c, bias))
    D = Dev(backend, device, (M + 1) * ldd)
    try:
        if noalloc:
            args = (M, N, K, A.ptr, lda, B.ptr, ldb, D.ptr, ldd, 1.5, Cm.ptr, ldc, 0.5, Bi.ptr, L.ACT_RELU)
            _check(L.load().sb200_gemm_f32_noalloc(device.id, 0, mode, *args))
        else:
            gemm(backend, device, mode, M, N, K, A, B, D, alpha=1.5, C_=Cm, beta=0.5, bias=Bi, act=1, lda=lda, ldb=ldb, ldc=ldc, ldd=ldd)
        got = D.download().reshape(M + 1, ldd)
        if noalloc and " splits=1 " in describe(mode, M, N, K, 1):     # it divides no k-loop: where the other entry does not either, the same bits
            gemm(backend, device, mode, M, N, K, A, B, D, alpha=1.5, C_=Cm, beta=0.5, bias=Bi, act=1, lda=lda, ldb=ldb, ldc=ldc, ldd=ldd)
            assert np.array_equal(D.download().view(np.uint32), got.ravel().view(np.uint32))
        ref = O.gemm(np.ascontiguousarray(a[:, :K]).ravel(), np.ascontiguousarray(b[:, :N]).ravel(), M, N, K, 1.5, 0.5,
                     np.ascontiguousarray(c[:, :N]).ravel(), bias, 1)
        # the clamp halves the reference's mean square, alpha scales the error: as in the other epilogue tests
        assert O.gemm_rel_error(got[:M, :N], ref) <= tol(mode, K) * 1.5 * math.sqrt(2), describe(mode, M, N, K, 1)
        assert np.all(got[:M, N:] == CANARY) and np.all(got[M] == CANARY)
    finally:
        for x in (A, B, Cm, Bi, D):
            x.free()


# One row, a multiple of 8 and one off it, whole 128 rows, and beside whole ones 1, 8, 9 and 127 more.
TAILS = [(1, 132, 260), (7, 260, 132), (8, 64, 96), (9, 516, 516), (64, 132, 260), (65, 256, 300), (127, 132, 1028), (128, 64, 260), (129, 1028, 516),
         (136, 2052, 260), (137, 1028, 516), (255, 516, 516), (257, 1028, 260), (393, 260, 700)]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("M,N,K", TAILS)
def test_rows_past_the_end(backend, device, mode, M, N, K):
    check(backend, device, mode, M, N, K, K, N, N, N)


# Whole 128 rows and boxes of the others side by side, which takes 2^26 multiply-adds; a pair's second block has some of the rows, or none.
BESIDE = [(138, 3472, 300, 16), (257, 1032, 260, 8), (393, 1028, 700, 16)]


@pytest.mark.parametrize("operands", ["read in place", "copied", "allocation-free"])
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("M,N,K,tail", BESIDE)
def test_rows_past_the_end_beside_whole_ones(backend, device, mode, M, N, K, tail, operands):
    noalloc, pad = operands == "allocation-free", 1 if operands == "copied" else 0
    if noalloc and mode not in (L.MODE_3XTF32, L.MODE_TF32):
        pytest.skip("the allocation-free entry has the TF32 modes")
    text = describe(mode, M, N, K, 1 - pad)
    assert f" a_tail={tail} " in text, text
    assert " splits=1 " in text or mode == L.MODE_3XTF32, text
    check(backend, device, mode, M, N, K, K + pad, N + pad, N, N, noalloc)


# (mode, M, N, K, splits): even and uneven shares of rows, rows and columns that end within a block's share, a last item that is shorter
SPREAD = [(L.MODE_3XTF32, 512, 512, 512, 2), (L.MODE_3XTF32, 509, 516, 1028, 3), (L.MODE_3XTF32, 768, 768, 768, 3), (L.MODE_3XTF32, 1000, 1020, 1000, 2),
          (L.MODE_TF32, 512, 512, 512, 2), (L.MODE_TF32, 1001, 1000, 2052, 2), (L.MODE_F16, 147, 56, 1700, 3), (L.MODE_3XF16, 300, 1020, 2052, 2)]


@pytest.mark.parametrize("mode,M,N,K,splits", SPREAD)
@pytest.mark.parametrize("ldd", ["quads", "single"])
def test_k_loops_divided_by_the_second_choice(backend, device, mode, M, N, K, splits, ldd):
    text = describe(mode, M, N, K, 1)
    assert f"splits={splits} " in text, text
    pad = 4 if ldd == "quads" else 1        # rows of the result on 16-byte boundaries, and not
    check(backend, device, mode, M, N, K, K, N, N + pad, N + pad)


# (mode, form, grid, block, M, N, K): parts of such products, by pairs and by blocks on their own, rows, columns and a last row that is cut short
PARTS = [(mode, *part, 509, 516, 1028) for mode in MODES for part in (("tiled", (33, 7), 16), ("tiled", (20, 20), 16), ("naive", (70 * 516 + 100, 1), 1))]
PARTS += [(L.MODE_3XTF32, "tiled", (64, 32), 16, 1024, 1024, 1024), (L.MODE_3XTF32, "tiled", (19, 48), 16, 768, 768, 768),
          (L.MODE_TF32, "tiled", (63, 8), 16, 1001, 1000, 2052), (L.MODE_3XF16, "tiled", (63, 8), 16, 1001, 1000, 2052)]


@pytest.mark.parametrize("mode,form,grid,side,M,N,K", PARTS)
def test_a_part_has_the_bits_of_a_whole_divided_by_the_second_choice(backend, device, mode, form, grid, side, M, N, K):
    routes.test_a_partial_launch_has_the_bits_of_the_whole(backend, device, mode, form, grid, side, M, N, K)


@pytest.mark.parametrize("M,N,K,tail", [(257, 1032, 260, 8), (1100, 1000, 300, 80), (1153, 1024, 64, 8), (511, 2052, 132, 128)])
def test_rows_past_the_end_behind_the_mixed_mode(backend, device, M, N, K, tail):
    """Operands the mixed mode declines go to a plain 3xTF32 launch behind it, which loads the last rows as other launches do."""
    lib = L.load()
    lib.sb200_set_mixed_min_macs(1 << 26)
    a, b = O.fill(M * K, 65, 1), O.fill(K * N, 65, 2)
    a, b = np.ldexp(a, 25), np.ldexp(b, 20)
    A, B, D = dev_from(backend, device, a), dev_from(backend, device, b), Dev(backend, device, (M + 1) * N)
    out = []
    try:
        text = describe(L.MODE_3XMIXED, M, N, K, 1)
        assert f" a_tail={tail} " in text and " operands=mixed " in text and " splits=1 " in describe(L.MODE_3XTF32, M, N, K, 1)
        for mode in (L.MODE_3XMIXED, L.MODE_3XTF32):
            D.clear()
            gemm(backend, device, mode, M, N, K, A, B, D)
            out.append(D.download())
        assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
        assert np.all(out[0][M * N:] == CANARY)
        assert O.gemm_rel_error(out[0][:M * N].reshape(M, N), O.gemm(a, b, M, N, K)) <= tol(L.MODE_3XTF32, K)
    finally:
        lib.sb200_set_mixed_min_macs(0)
        for x in (A, B, D):
            x.free()
