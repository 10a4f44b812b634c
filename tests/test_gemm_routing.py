"""How the library routes a product (kernel, tile, scratch, launches) — host logic, no GPU needed."""
import ctypes as C
import random

import pytest

from spoc_b200 import _lib as L

SMS = 148


def describe(mode, M, N, K, addressable=1, sms=SMS):
    out = C.create_string_buffer(256)
    assert L.load().sb200_gemm_describe(mode, M, N, K, addressable, sms, out, 256) == 0
    return dict(kv.split("=") for kv in out.value.decode().split()[2:]) | {"kernel": " ".join(out.value.decode().split()[:2])}


@pytest.mark.parametrize("mode", [L.MODE_3XTF32, L.MODE_TF32])
def test_benchmark_configurations_take_the_large_tile(mode):
    for shape in [(8192, 8192, 8192), (32768 // 8, 32768, 32768), (65536 // 8, 4096, 4096), (4096, 4096, 4096), (2048, 2048, 2048)]:
        d = describe(mode, *shape)
        assert d["kernel"] == "pair direct" and d["tile"] == "256x256", (shape, d)
        # 3xTF32 reads the largest ones beside panels of low parts, which are a launch of their own, and splits the others on chip
        assert (d["operands"], d["launches"], d["kernels"]) in ([("direct", "2", "2"), ("split", "1", "1")] if mode == L.MODE_3XTF32 else [("direct", "1", "1")])
    d = describe(L.MODE_TF32, 8192, 8192, 8192)
    assert d["stages"] == "6" and d["tiles"] == "1024" and d["waves"] == "14" and d["workspace"] == "0"
    d = describe(L.MODE_3XTF32, 8192, 8192, 8192)
    assert d["stages"] == "3" and d["workspace"] == str(2 * 8192 * 8192 * 4)     # the two low-part panels
    assert d["operands"] == "direct" and describe(L.MODE_3XTF32, 4096, 4096, 4096)["operands"] == "split"


def test_problems_with_few_tiles_take_narrower_tiles():
    assert describe(L.MODE_TF32, 1024, 1024, 1024)["tile"] == "256x64"
    assert describe(L.MODE_TF32, 256, 256, 256)["tile"] == "256x64"
    assert describe(L.MODE_3XTF32, 1536, 1536, 1536)["tile"] == "256x128"
    assert describe(L.MODE_TF32, 1792, 1792, 1792)["tile"] == "256x256"
    d = describe(L.MODE_TF32, 1024, 1024, 1024)
    assert d["stages"] == "8" and d["tiles"] == "64" and d["waves"] == "1"


def test_operands_tma_cannot_address_go_through_panels():
    d = describe(L.MODE_3XTF32, 700, 900, 1000, addressable=0)
    assert d["kernel"] == "pair panels" and d["launches"] == "3"
    kp = 1024
    assert int(d["workspace"]) == 2 * ((700 * kp * 4 + 1023) // 1024 * 1024 + (900 * kp * 4 + 1023) // 1024 * 1024)
    # at most 128 rows and a small product: converted in registers by single CTAs; a pair when it can read the operands directly
    assert describe(L.MODE_TF32, 100, 300, 500, addressable=0)["kernel"] == "single panels"
    assert describe(L.MODE_TF32, 100, 300, 500, addressable=1)["kernel"] == "pair direct"


def test_unaligned_operands_of_short_k_loops_are_converted():
    """In registers on their way: a copy in front of a few k-blocks takes longer than it saves (up to twice the time)."""
    for mode, shape in [(L.MODE_3XTF32, (97, 8712, 43)), (L.MODE_TF32, (114, 10433, 96)), (L.MODE_TF32, (854, 1182, 27)), (L.MODE_TF32, (77, 2794, 356)),
                        (L.MODE_3XTF32, (343, 3112, 9)), (L.MODE_3XTF32, (69, 1908, 149))]:
        d = describe(mode, *shape, addressable=0)
        assert d["operands"] == "converted" and d["workspace"] == "0", (mode, shape, d)
    for mode, shape in [(L.MODE_3XTF32, (255, 257, 259)), (L.MODE_3XTF32, (449, 449, 449)), (L.MODE_TF32, (449, 449, 449)), (L.MODE_3XTF32, (600, 513, 259)),
                        (L.MODE_TF32, (600, 513, 259))]:
        assert describe(mode, *shape, addressable=0)["operands"] == "copied", (mode, shape)


def test_many_rows_against_a_few_columns_are_converted_in_eight_warps():
    """And not by the splitting kernel, which waits for B's short rows."""
    for shape in [(9000, 4, 100), (14000, 4, 200), (9000, 8, 100), (14000, 16, 72)]:
        assert describe(L.MODE_3XTF32, *shape)["operands"] == "converted", shape
    for shape in [(4000, 16, 100), (6000, 16, 128), (9000, 32, 128)]:
        assert describe(L.MODE_3XTF32, *shape)["operands"] == "split", shape


def test_tf32_mode_reads_addressable_operands_without_scratch():
    """Long k-loops over few tiles among them: their partial sums stay within a cluster, so that calls on different streams, and
    graphs they were captured into, share nothing."""
    rng = random.Random(5)
    shapes = [(46, 1, 4640), (356, 329, 9218), (3420, 1398, 6654), (435, 1897, 8484), (128, 96, 16384), (1, 8, 16384)]
    shapes += [tuple(int(2 ** rng.uniform(0, 14)) for _ in range(3)) for _ in range(3000)]
    divided = 0
    for shape in shapes:
        d = describe(L.MODE_TF32, *shape)
        assert d["workspace"] == "0" and d["launches"] == "1", (shape, d)
        divided += d["splits"] != "1"
    assert divided > 100


def describe_part(mode, part, whole, K, addressable):
    out = C.create_string_buffer(256)
    assert L.load().sb200_gemm_describe_part(mode, *part, K, *whole, addressable, SMS, out, 256) == 0
    return dict(kv.split("=") for kv in out.value.decode().split()[2:])


@pytest.mark.parametrize("addressable", [1, 0])
@pytest.mark.parametrize("mode", [L.MODE_3XTF32, L.MODE_TF32, L.MODE_3XF16, L.MODE_F16])
def test_a_part_has_the_division_of_its_whole(mode, addressable):
    """Rows, columns or both of a product, as partial launches and row blocks compute them: a k-loop divided otherwise has other bits."""
    rng = random.Random(9)
    pairs = [((128, 4096), (100, 4096), 4096), ((128, 2048), (100, 2048), 4096), ((96, 1056), (96, 678), 1600), ((128, 4096), (65, 17), 4096),
             ((64, 4096), (37, 4096), 4096), ((128, 96), (128, 1), 16384)]
    while len(pairs) < 3000:
        M, N, K = (int(2 ** rng.uniform(0, 13.5)) for _ in range(3))
        if rng.random() < 0.3:
            M = rng.randint(65, 128)
        part = (rng.randint(1, M) if rng.random() < 0.7 else M, rng.randint(1, N) if rng.random() < 0.5 else N)
        pairs.append(((M, N), part, K))
    divided = 0
    for whole, part, K in pairs:
        w = describe(mode, *whole, K, addressable)
        p = describe_part(mode, part, whole, K, addressable)
        assert p["splits"] == w["splits"], (whole, part, K, w, p)
        assert mode != L.MODE_TF32 or not addressable or p["workspace"] == "0"
        divided += w["splits"] != "1"
    assert divided > 300


def test_degenerate_and_bad_arguments():
    out = C.create_string_buffer(64)
    lib = L.load()
    assert lib.sb200_gemm_describe(L.MODE_TF32, 0, 5, 5, 1, SMS, out, 64) == 0 and out.value == b"nothing to do"
    assert lib.sb200_gemm_describe(L.MODE_TF32, 5, 5, 0, 1, SMS, out, 64) == 0 and b"gemm_k0_kernel" in out.value
    assert lib.sb200_gemm_describe(7, 5, 5, 5, 1, SMS, out, 64) == L.ERR_INVALID_VALUE
    assert lib.sb200_gemm_describe(L.MODE_TF32, 5, 5, 5, 1, 0, out, 64) == L.ERR_INVALID_VALUE
    assert lib.sb200_set_gemm_tile_n(96) == L.ERR_INVALID_VALUE
    assert lib.sb200_set_gemm_tile_n(128) == 0
    assert describe(L.MODE_TF32, 8192, 8192, 8192)["tile"] == "256x128"
    assert lib.sb200_set_gemm_tile_n(0) == 0


@pytest.mark.parametrize("mode", [L.MODE_3XTF32, L.MODE_TF32, L.MODE_3XF16, L.MODE_F16, L.MODE_3XMIXED])
def test_the_last_rows_of_a_have_boxes_of_their_own(mode):
    """As high as there are rows, to the next multiple of 8; beside whole 128 rows only in larger products."""
    assert L.load().sb200_set_mixed_min_macs(1 << 26) == 0
    try:
        for M, N, K, rows in [(7, 4096, 4096, 8), (64, 4096, 4096, 64), (100, 4096, 4096, 104), (128, 4096, 4096, 128), (129, 4096, 4096, 8),
                              (257, 2064, 1024, 8), (1100, 2000, 640, 80), (2047, 2048, 2048, 128), (2048, 2048, 2048, 128), (137, 64, 260, 128),
                              (138, 3472, 256, 16), (135, 4028, 144, 8), (137, 3000, 160, 128)]:     # 2^26.9, 2^26.2 and 2^25.97 multiply-adds
            d = describe(mode, M, N, K)
            assert d["a_tail"] == (str(rows) if d["operands"] != "converted" else "0"), (M, N, K, d)
    finally:
        assert L.load().sb200_set_mixed_min_macs(0) == 0
