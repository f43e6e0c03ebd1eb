"""The dealing of the streaming form's work (csrc/stream_deal.h), walked on the CPU as the kernel's CTAs walk it: every unit is dealt
once, a tile's contributors are as many as the count it waits for, and no two partial sums share a place."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("deal") / "libdeal.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + os.path.join(ROOT, "awesome_fusion_b200", "csrc"),
                           "-o", out, os.path.join(ROOT, "tests", "stream_deal_shim.cc")])
    lib = ctypes.CDLL(out)
    lib.check_deal.argtypes = [ctypes.c_uint32] * 3
    lib.fits.argtypes = [ctypes.c_uint32] * 3
    lib.check_waves.argtypes = [ctypes.c_uint32] * 4
    lib.tiles_past_the_end.argtypes = [ctypes.c_uint32] * 4 + [ctypes.c_int]
    lib.check_range.argtypes = [ctypes.c_uint32] * 3 + [ctypes.POINTER(ctypes.c_uint32)]
    return lib


@pytest.mark.parametrize("sms,tiles,blocks", [(148, 620, 14), (132, 420, 9), (7, 60, 12), (1, 5, 5)])
def test_every_number_of_tiles_and_blocks(shim, sms, tiles, blocks):
    """148 SMs: up to four waves of tiles with up to 13 units each (beyond one wave's rest the pattern repeats)."""
    where = (ctypes.c_uint32 * 2)()
    rc = shim.check_range(tiles, blocks, sms, where)
    assert rc == 0, f"rule {rc} broken at {where[0]} tiles of {where[1]} blocks on {sms} SMs"


@pytest.mark.parametrize("tiles,blocks", [(192, 2), (200, 2), (192, 3), (3300, 3), (1672, 3), (224, 64), (86, 32), (32, 512), (4928, 32)])
def test_sizes_of_calls(shim, tiles, blocks):
    """24576 x 512 and 25600 x 512 int4 at 17 to 32 rows, 24576 x 768, 2048 rows of 38400 x 768 and of 19456 x 768 (fewer units than
    CTAs next to whole waves: such tiles were lost), and sizes with more units than CTAs."""
    assert shim.check_deal(tiles, blocks, 148) == 0


@pytest.mark.parametrize("tiles,blocks,sms", [(300, 4, 148), (296, 4, 148), (40, 3, 148), (9, 5, 4)])
def test_a_wave_too_many_is_seen(shim, tiles, blocks, sms):
    """The streaming form's walk would take tiles past the end; the check walks as it does and says so.  (The pair form's walk stops there.)"""
    assert shim.check_waves(tiles, blocks, sms, 0) == 0 and shim.check_waves(tiles, blocks, sms, 1) != 0
    assert shim.tiles_past_the_end(tiles, blocks, sms, 1, 0) > 0 and shim.tiles_past_the_end(tiles, blocks, sms, 1, 1) == 0


def test_the_limit_of_the_32_bit_arithmetic(shim):
    """148 SMs, 200 tiles (52 shared): the largest number of blocks that is taken is dealt correctly, one more is refused (the launcher
    takes another form)."""
    most = (2 ** 32 - 1) // (52 * 149)
    assert shim.fits(200, most, 148) and not shim.fits(200, most + 1, 148)
    assert shim.check_deal(60, 40000, 148) == 0 and shim.check_deal(200, 300000, 148) == 0
