"""Rules by which launches are cut, asked on the host for devices of any size."""
import ctypes

import pytest


@pytest.fixture(scope="module")
def lib():
    import kirai_b200  # noqa: F401
    from kirai_b200.csrc import ops

    return ops.library()


@pytest.mark.parametrize("sms", [108, 132, 148, 160])
def test_32_bit_products_fill_whole_rounds_of_the_device_that_runs_them(lib, sms):
    cut = 0
    a_little_more = 128 * (2 * sms // 3 + 3)  # columns that make two rounds and about nine CTAs of three tiles of 192 rows
    for m, n, k in [(576, a_little_more, 2560), (515, 19456, 516), (515, 19456, 2560), (576, 6460, 1028), (128, 19200, 700), (30, 38404, 260), (800, 24576, 4096), (9, 151936, 2560)]:
        rows = ctypes.c_int(0)
        first = lib.kirai_gemm_f32_tc_first_columns(m, n, k, sms, ctypes.byref(rows))
        if first == 0:
            continue
        cut += 1
        assert first % 128 == 0 and 0 < first < n and rows.value in (32, 64, 128, 192)
        tiles, room = -(-m // rows.value), sms * (2 if rows.value <= 64 else 1)
        ctas = first // 128 * tiles
        assert ctas % room == 0 or room - ctas % room < tiles  # the last round lacks less than a column of tiles
    assert cut
    if sms == 148:  # 456 CTAs of 192 rows: three rounds, and 4 columns of tiles to the second launch
        assert (lib.kirai_gemm_f32_tc_first_columns(515, 19456, 2560, sms, ctypes.byref(rows)), rows.value) == (148 * 128, 192)
        # measured as two launches 119 and 379 us, as one 111 and 360
        for n in (6144, 19456):
            assert lib.kirai_gemm_f32_tc_first_columns(640, n, 2560, sms, ctypes.byref(rows)) == 0


def test_tiles_of_many_token_products_are_those_that_measured_faster(lib):
    """256 rows by fewer than 128 columns lost to 128 x 256 wherever they were picked; 128 x 256 is left for 8 % by the rule's count."""
    for n, k in [(2560, 4096), (2560, 9728), (4096, 4096), (4096, 8192), (4096, 12288), (5120, 8192), (5120, 25600), (3072, 3072), (6144, 4096)]:
        for m in range(129, 2049, 37):
            for form in (0, 1, 2):
                rows, width = divmod(lib.kirai_gemm_bf16_many_tile(m, n, k, form), 1000)
                assert rows == 1 and 48 <= width <= 256 or rows == 2 and 128 <= width <= 256, (m, n, k, form)
    # (on 148 SMs) measured 27.3, 56.1, 113.8, 86.0 and 214 us in 128 x 256, 30.7, 58.8, 118.8, 89.5 and 234 in what was picked before
    for m, n, k, form in [(1003, 4096, 4096, 0), (1003, 4096, 8192, 1), (1300, 12288, 4096, 1), (2048, 6144, 4096, 1), (256, 151936, 2560, 1)]:
        assert lib.kirai_gemm_bf16_many_tile(m, n, k, form) == 1256, (m, n, k, form)
