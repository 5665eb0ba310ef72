"""Frames whose cycles are spent before their limit is looked at, against the oracle.

A frame waits for VSYNC to drop for up to 2,000,000 cycles and then ends at
the first instruction that finds more than 100,000 cycles spent
(src/atari.rs:584-598).  A program that holds VSYNC for longer than 100,000
cycles and then drops it has spent them before that second limit applies: its
frame ends at the next instruction boundary, whatever the timer, WSYNC or an
illegal opcode would do.  All compared values are integers: no tolerance.
"""
import numpy as np
import pytest

import oracle
from fa_pkg import carts, fa
from test_edge_programs import KINDS, program, states
from test_gpu_render import check
from test_host_sim import assert_same, run_both, sim  # noqa: F401  (the fixture)

ORG = 0xFC00                       # in the window that no scheme switches (E0, 3F), the same in every bank
DELAYS = {                         # what spends the cycles while VSYNC is held
    "loop": [0xA0, 100, 0xA2, 0, 0xCA, 0xD0, 0xFD, 0x88, 0xD0, 0xF8],                     # 128,000 cycles of DEX / BNE
    "wsync": [0xA0, 7, 0xA2, 0, 0x85, 0x02, 0xCA, 0xD0, 0xFB, 0x88, 0xD0, 0xF6],          # 1,792 lines of STA WSYNC
    "timer": [0xA9, 255, 0x8D, 0x97, 0x02,                                                # T1024T, then as "loop"
              0xA0, 100, 0xA2, 0, 0xCA, 0xD0, 0xFD, 0x88, 0xD0, 0xF8],
}
AFTER = {                          # what runs once VSYNC has dropped
    "jump": [0x4C],                                                                       # JMP to itself
    "rearm": [0xA9, 255, 0x8D, 0x97, 0x02, 0xE6, 0x90, 0x4C],                             # T1024T set over and over
    "wait": [0x85, 0x02, 0xE6, 0x90, 0x4C],                                               # a line at a time
    "illegal": [0xEA, 0xE6, 0x90, 0x02],                                                  # NOP, INC, an illegal opcode
}
# VSYNC dropped by a store, or by BRK's pushes with the stack pointer at 2:
# WSYNC, VBLANK and then VSYNC (P with Z clear), so that a wait begins in the
# same instruction.
DROPS = ["store", "brk"]


def hold_rom(size, delay, drop, after):
    """VSYNC raised, the delay, VSYNC dropped, `after`; the same code in every 4K (and last 1K)."""
    code = [0xA9, 2, 0x85, 0x00] + DELAYS[delay]
    code += [0xA9, 0, 0x85, 0x00] if drop == "store" else [0xA2, 2, 0x9A, 0xA9, 1, 0x00, 0x00]
    at = ORG + len(code)
    code += AFTER[after]
    if code[-1] == 0x4C:
        code += [at & 0xFF, at >> 8]
    bank = bytearray([0xEA]) * 4096
    bank[ORG & 0xFFF:(ORG & 0xFFF) + len(code)] = bytes(code)
    bank[0xFFC:] = bytes([ORG & 0xFF, ORG >> 8, at & 0xFF, at >> 8])
    return (bytes(bank) * 8)[:size]


class scheme_of:
    """The cart's scheme registered with the oracle and `registry` (the library or the host build)."""

    def __init__(self, rom, code, registry):
        self.rom, self.code, self.registry = rom, code, registry

    def __enter__(self):
        if self.code >= 0:
            self.registry(self.rom, self.code)
            oracle.set_rom_scheme(self.rom, self.code)

    def __exit__(self, *exc):
        if self.code >= 0:
            self.registry(self.rom, -1)
            oracle.set_rom_scheme(self.rom, "auto")


def on_host(L):
    def register(rom, code):
        r = np.frombuffer(rom, np.uint8).copy()
        L.fa_rom_set_scheme(r.ctypes.data, len(r), code)
    return register


@pytest.mark.parametrize("kind", KINDS)
def test_vsync_held_past_the_frame_cap(sim, kind):  # noqa: F811
    size, code = KINDS[kind]
    n, k = 2, 3
    for delay in DELAYS:
        for drop in DROPS:
            for after in AFTER:
                rom = hold_rom(size, delay, drop, after)
                with scheme_of(rom, code, on_host(sim)):
                    start = np.array([oracle.reset_state(rom)] * n, dtype=oracle.STATE_DTYPE)
                    got, ref = run_both(sim, rom, start, carts.actions(seed=5, n=n, frames=k), k)
                assert_same(got, ref, f"{kind}, {delay}, {drop}, {after}")


# Seeds 16, 13, 141 and 251 hold a console that drops VSYNC with the cap spent.
@pytest.mark.parametrize("kind,seed", [("fe", 16), ("8k", 13), ("4k", 141), ("dpc", 251)] +
                         [(kind, seed) for kind in KINDS for seed in (0, 1)])
def test_random_programs_that_start_in_vsync(sim, kind, seed):  # noqa: F811
    size, code = KINDS[kind]
    rng = np.random.default_rng(seed)
    rom = program(rng, size)
    with scheme_of(rom, code, on_host(sim)):
        start = states(rng, rom, 96)
        start["tia_vsync"] = rng.choice([0, 2, 2, 0xFF], 96)
        start["tia_wsync"] = rng.integers(0, 2, 96)
        got, ref = run_both(sim, rom, start, carts.actions(seed=seed, n=96, frames=2), 2)
    assert_same(got, ref, f"{kind} program {seed}")


RENDERED = ["4k", "8k", "32k", "e0", "3f"]


@pytest.mark.parametrize("kind", RENDERED)
def test_vsync_held_past_the_frame_cap_on_the_rendering_console(sim, kind):  # noqa: F811
    """Its frame loop looks at instruction cycles and counts a WSYNC wait cycle by cycle."""
    size, code = KINDS[kind]
    n, calls, k = 1, 2, 1
    acts = np.stack([carts.actions(seed=50 + i, n=n, frames=k) for i in range(calls)])
    for delay in ("loop", "wsync"):
        for drop in DROPS:
            for after in AFTER:
                rom = hold_rom(size, delay, drop, after)
                r = np.frombuffer(rom, np.uint8).copy()
                fb, ram = np.zeros((n, 192, 160), np.uint8), np.zeros((n, 128), np.uint8)
                st = np.zeros(n, fa.STATE_DTYPE)
                with scheme_of(rom, code, on_host(sim)):
                    assert sim.hs_render(r.ctypes.data, len(r), n, acts.ctypes.data, calls, k, fb.ctypes.data,
                                         st.ctypes.data, ram.ctypes.data) >= 0
                    consoles = oracle.render_reset(rom, n)
                    for i in range(calls):
                        oracle.render_steps(consoles, acts[i])
                check(fb, ram, st, consoles, f"{kind}, {delay}, {drop}, {after}")


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_vsync_held_past_the_frame_cap_on_the_gpu(kind):
    if fa.device_count() < 1:
        pytest.skip("no CUDA device")
    size, code = KINDS[kind]
    n, k = 33, 2
    for delay, drop, after in [("loop", "store", "jump"), ("wsync", "brk", "wait"), ("timer", "store", "rearm"),
                               ("wsync", "store", "illegal")]:
        rom = hold_rom(size, delay, drop, after)
        with scheme_of(rom, code, lambda r, c: fa.set_rom_scheme(r, c if c >= 0 else "auto")):
            ref = np.array([oracle.reset_state(rom)] * n, dtype=oracle.STATE_DTYPE)
            acts = carts.actions(seed=6, n=n, frames=k)
            with fa.BatchAtariGpu(rom, n) as g:
                g.upload_states(ref)
                g.step_multi(acts, k)
                got = g.download_states()
            oracle.run_batch(rom, ref, acts, k)
            assert_same(got, ref, f"{kind}, {delay}, {drop}, {after}")


@pytest.mark.gpu
@pytest.mark.parametrize("kind", RENDERED)
def test_vsync_held_past_the_frame_cap_on_the_rendering_console_on_the_gpu(kind):
    if fa.device_count() < 1:
        pytest.skip("no CUDA device")
    size, code = KINDS[kind]
    n, k = 33, 2
    acts = carts.actions(seed=50, n=n, frames=k)
    for delay, drop, after in [("wsync", "store", "jump"), ("wsync", "brk", "wait"), ("loop", "store", "illegal")]:
        rom = hold_rom(size, delay, drop, after)
        with scheme_of(rom, code, lambda r, c: fa.set_rom_scheme(r, c if c >= 0 else "auto")):
            consoles = oracle.render_reset(rom, n)
            oracle.render_steps(consoles, acts)
            with fa.AtariRender(rom, n) as g:
                g.reset()
                fb, ram = g.step_multi(acts, k)
                check(fb, ram, g.states(), consoles, f"{kind}, {delay}, {drop}, {after}")
