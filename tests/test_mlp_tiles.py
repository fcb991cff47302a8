"""The tiles of the MLP's layer products by batch size, from the library's rule (no
GPU needed): small batches have to give as many CTAs as 32 x 32 tiles did, or one to
every other SM."""
import pytest

from tailor_gb300 import _lib, build


@pytest.fixture(scope="module")
def lib():
    build.build()
    return _lib.load()


def ctas(lib, m, n, z=1, sms=152):
    g = lib.tlr_mlp_tile(m, n, z, sms)
    assert g in (16, 32, 64)
    return -(-m // g) * -(-n // g) * z, g


@pytest.mark.parametrize("rows", [1, 16, 24, 33, 64, 65, 192, 300, 512, 1000, 2048, 100000])
@pytest.mark.parametrize("width", [3, 80, 256])
def test_enough_ctas(lib, rows, width):
    for m, n in ((rows, width), (width, 256)):
        count, g = ctas(lib, m, n)
        assert g == 16 or 2 * count >= 152
        assert count >= min(76, -(-m // 32) * -(-n // 32))


def test_large_batches_keep_large_tiles(lib):
    assert ctas(lib, 2048, 256)[1] == 64 and ctas(lib, 256, 256, 16)[1] == 64
    assert ctas(lib, 24, 256)[1] == 16 and ctas(lib, 512, 256)[1] == 32
