"""A factor's device bytes include the digit planes that its updates take while it is made: 8 bytes per row of a panel
and column in FP32 (up to 512 columns), 14 for each of 512 columns in FP64 where 64 divides nb."""


def test_factor_bytes_include_the_digit_planes(ooc):
    L = ooc.load()
    for n, nb in [(65536, 512), (4096, 256), (1001, 128)]:
        tiles = -(-n // nb) * nb * nb
        b32 = L.ooc_factor_bytes(n, nb, ooc.PREC_FP32)
        b64 = L.ooc_factor_bytes(n, nb, ooc.PREC_FP64)
        assert b32 >= 4 * n * n + 4 * tiles + 8 * n * min(nb, 512)
        assert b64 >= 8 * n * n + 8 * tiles + 8 * n * nb + 14 * 512 * n
    # 64 does not divide 100: FP64 updates without planes
    assert L.ooc_factor_bytes(5000, 100, ooc.PREC_FP64) < L.ooc_factor_bytes(5000, 128, ooc.PREC_FP64) - 14 * 512 * 5000 + 8 * 64 * 5000
