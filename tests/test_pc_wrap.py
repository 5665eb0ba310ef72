"""Calls that end on an instruction after which pc wraps past $FFFF, against the oracle.

Stored, pc is 16 bits beside P and the bank: what lies above must not reach
them.  pc wraps by an instruction that ends at $FFFF, by a forward branch and
by an RTS to $FFFF.  All compared values are integers: no tolerance.
"""
import numpy as np
import pytest

import oracle
from fa_pkg import carts, fa
from test_edge_programs import KINDS
from test_frame_limits import RENDERED, on_host, scheme_of
from test_gpu_render import check
from test_host_sim import assert_same, run_both, sim  # noqa: F401  (the fixture)

# At $FF90, through BRK at $0000 and back by the vector at $FFFE: 17 cycles
# with a branch to $0000, 25 with an RTS.  Nothing sets VSYNC: a frame ends
# at the cycle cap, and where in the loop follows from the start's place in a
# sled of NOPs.
LOOPS = {"branch": [0xA2, 0xFF, 0x9A, 0x18, 0x90, 0x6A],                # LDX #$FF, TXS, CLC, BCC $0000
         "rts": [0xA2, 0xFF, 0x9A, 0xA9, 0xFF, 0x18, 0x48, 0x48, 0x60]}  # .., CLC, PHA, PHA, RTS
SLED = 0xFF60


def loop_rom(size, loop, start=SLED):
    bank = bytearray([0xEA]) * 4096
    bank[0xF90:0xF90 + len(LOOPS[loop])] = bytes(LOOPS[loop])
    bank[0xFFC:] = bytes([start & 0xFF, start >> 8, 0x90, 0xFF])
    return (bytes(bank) * 8)[:size]


def loop_states(rom):
    st = np.array([oracle.reset_state(rom)] * 48, dtype=oracle.STATE_DTYPE)
    st["pc"] = SLED + np.arange(48)
    st["run_status"] = 0
    return st


def last_rom(size, op):
    """op $0000 at $FFFD (its bytes are the vectors' too), the same in every bank."""
    bank = bytearray([0xEA]) * 4096
    bank[0xFFD:] = bytes([op, 0x00, 0x00])
    return (bytes(bank) * 2)[:size]


def last_states(rom):
    """The store at $FFFD raises VSYNC and ends the frame; P with and without its carry."""
    st = np.array([oracle.reset_state(rom)] * 4, dtype=oracle.STATE_DTYPE)
    st["a"], st["y"], st["pc"] = 2, 0, 0xFFFD
    st["status"] = [0x20, 0x21, 0xE0, 0xE1]
    st["tia_vsync"], st["tia_wsync"], st["run_status"] = 0, 0, 0
    return st


def cases():
    for kind in KINDS:
        for loop in LOOPS:
            yield kind, loop, lambda size, loop=loop: loop_rom(size, loop), loop_states
    for kind in ("4k", "fe"):                                           # no hotspots at $FFF4-$FFFF
        for name, op in (("sta_abs", 0x8D), ("sta_absy", 0x99)):
            yield kind, name, lambda size, op=op: last_rom(size, op), last_states


CASES = [pytest.param(kind, rom, states, id=f"{kind}-{name}") for kind, name, rom, states in cases()]


@pytest.mark.parametrize("kind,rom_of,states_of", CASES)
def test_pc_wraps_at_the_end_of_a_call(sim, kind, rom_of, states_of):  # noqa: F811
    size, code = KINDS[kind]
    rom = rom_of(size)
    with scheme_of(rom, code, on_host(sim)):
        start = states_of(rom)
        got, ref = run_both(sim, rom, start, np.zeros((1, len(start)), np.uint8), 1)
        assert_same(got, ref, f"{kind}, the call's end")
        got, ref = run_both(sim, rom, got, np.zeros((1, len(start)), np.uint8), 1)
        assert_same(got, ref, f"{kind}, the next call's end")


@pytest.mark.parametrize("kind", RENDERED)
@pytest.mark.parametrize("loop", LOOPS)
def test_pc_wraps_at_the_end_of_a_call_of_the_rendering_console(sim, kind, loop):  # noqa: F811
    size, code = KINDS[kind]
    acts = np.zeros((1, 1, 1), np.uint8)
    for start in range(SLED, SLED + 26):
        rom = loop_rom(size, loop, start)
        r = np.frombuffer(rom, np.uint8).copy()
        fb, ram, st = np.zeros((1, 192, 160), np.uint8), np.zeros((1, 128), np.uint8), np.zeros(1, fa.STATE_DTYPE)
        with scheme_of(rom, code, on_host(sim)):
            assert sim.hs_render(r.ctypes.data, len(r), 1, acts.ctypes.data, 1, 1, fb.ctypes.data, st.ctypes.data,
                                 ram.ctypes.data) >= 0
            consoles = oracle.render_reset(rom, 1)
            oracle.render_steps(consoles, acts[0])
        check(fb, ram, st, consoles, f"{kind}, {loop} from {start:04x}")


@pytest.mark.gpu
@pytest.mark.parametrize("sched", ["pc", "lane"])
@pytest.mark.parametrize("kind,rom_of,states_of", CASES)
def test_pc_wraps_at_the_end_of_a_call_on_the_gpu(kind, rom_of, states_of, sched):
    if fa.device_count() < 1:
        pytest.skip("no CUDA device")
    size, code = KINDS[kind]
    rom = rom_of(size)
    with scheme_of(rom, code, lambda r, c: fa.set_rom_scheme(r, c if c >= 0 else "auto")):
        ref = states_of(rom)
        acts = carts.actions(seed=9, n=len(ref), frames=1)
        with fa.BatchAtariGpu(rom, len(ref)) as g:
            g.set_launch(128, sched, False)
            g.upload_states(ref)
            for call in range(2):
                g.step_multi(acts, 1)
                oracle.run_batch(rom, ref, acts, 1)
                assert_same(g.download_states(), ref, f"{kind} {sched}, call {call}")
