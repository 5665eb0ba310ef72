"""State rows that a caller writes in device memory, past the checks of the
calls that take whole states."""
import numpy as np
import pytest

import oracle
from fa_pkg import carts
from test_host_sim import assert_same
from test_host_warp import run_warps, warp  # noqa: F401  (the fixture)


@pytest.mark.parametrize("size", [4096, 8192, 16384, 32768])
def test_bank_outside_the_image(warp, size):  # noqa: F811
    """A 4K-bank cart's bank byte selects a bank of the image whatever it holds: its number modulo the banks."""
    rng = np.random.default_rng(size)
    nbanks = size // 4096
    rom = bytearray(rng.integers(0, 256, size, dtype=np.uint8).tobytes())
    for b in range(nbanks):
        rom[b * 4096 + 0xFFC:b * 4096 + 0xFFE] = bytes([0x00, 0xF0])
    rom = bytes(rom)
    banks = np.array([nbanks, nbanks + 1, 2 * nbanks - 1, 8, 13, 0x80, 0xFF], np.uint8)
    wild = np.array([oracle.reset_state(rom)] * len(banks), dtype=oracle.STATE_DTYPE)
    wild["pc"], wild["run_status"] = 0xF000 + rng.integers(0, 0x800, len(banks)), 0
    tame = wild.copy()
    wild["bank"], tame["bank"] = banks, banks % nbanks
    acts = carts.actions(seed=4, n=len(banks), frames=2)
    got = run_warps(warp, rom, wild, acts, 2, "lane", 20_000_000)
    ref = tame.copy()                                      # the oracle takes no bank outside the image
    oracle.run_batch(rom, ref, acts, 2)
    assert_same(got, ref, f"{size}-byte cart")
