"""The warp scheduler (run_lanes) with the device core, 32 lanes at a time on the host.

tests/hostsim/warp_run.cpp runs each lane as a coroutine that a warp
intrinsic suspends until its mask's lanes have reached it, and gives up after
a number of such meetings: a schedule that makes no progress fails here
instead of hanging a GPU.  Results must equal the oracle's (integers).
"""
import ctypes
import os
import subprocess
import tempfile
from pathlib import Path

import numpy as np
import pytest

import oracle
from fa_pkg import ROOT, carts, fa
from test_edge_programs import KINDS, program, states
from test_frame_limits import scheme_of
from test_host_sim import assert_same

HERE = Path(__file__).resolve().parent / "hostsim"
SCHEDS = {"pc": 1, "line": 2, "lane": 0, "match": 3}


@pytest.fixture(scope="module")
def warp():
    out = Path(tempfile.mkdtemp(prefix="fa_hostwarp_")) / "libhostwarp.so"
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-fPIC", "-shared", "-I", str(HERE), "-I",
                    str(ROOT / "include"), str(HERE / "warp_run.cpp"), "-o", str(out)], check=True)
    L = ctypes.CDLL(str(out))
    L.hs_warps.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p,
                           ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_void_p]
    L.fa_rom_set_scheme.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int]
    return L


def run_warps(L, rom, start, acts, k, sched, limit):
    got, r = start.copy(), np.frombuffer(rom, np.uint8).copy()
    a, counters = np.ascontiguousarray(acts, dtype=np.uint8), np.zeros(2, np.uint64)
    rc = L.hs_warps(r.ctypes.data, len(r), got.ctypes.data, len(got), a.ctypes.data, k, SCHEDS[sched], limit,
                    counters.ctypes.data)
    assert rc == 0, {-1: "bad ROM", -2: "no end within the limit", -3: "lanes that wait for each other"}[rc]
    return got


@pytest.mark.parametrize("sched", SCHEDS)
@pytest.mark.parametrize("kind", ["4k", "8k", "3f", "fe"])
def test_warps_match_oracle(warp, kind, sched):
    size, code = KINDS[kind]
    rng = np.random.default_rng(size + code)
    rom = program(rng, size)

    def register(rom, code):
        r = np.frombuffer(rom, np.uint8).copy()
        warp.fa_rom_set_scheme(r.ctypes.data, len(r), code)
    with scheme_of(rom, code, register):
        start = states(rng, rom, 40)                         # a full warp and a part of one
        acts = carts.actions(seed=2, n=40, frames=2)
        got = run_warps(warp, rom, start, acts, 2, sched, 20_000_000)
        ref = start.copy()
        oracle.run_batch(rom, ref, acts, 2)
    assert_same(got, ref, f"{kind}, {sched}")


def last_key_rom():
    """8K, both banks alike.  From the 126th frame on (RAM $91), a frame makes
    512 hotspot accesses, then jumps to $FFFF, where CLD ends the address
    space, from two places by RAM $90; BRK at $0000 and the vector at $FFFE
    go on to the VSYNC."""
    code = [0xE6, 0x91, 0xA5, 0x91, 0xC9, 126, 0x90, 0x17,   # F000 INC $91, LDA $91, CMP #126, BCC F01F
            0xA0, 2, 0xA2, 0,                                # F008 LDY #2, LDX #0
            0x2C, 0xF8, 0x1F, 0xCA, 0xD0, 0xFA, 0x88, 0xD0, 0xF7,   # F00C BIT $1FF8, DEX, BNE, DEY, BNE
            0xA5, 0x90, 0xF0, 3,                             # F015 LDA $90, BEQ F01C
            0x4C, 0xFF, 0xFF, 0x4C, 0xFF, 0xFF,              # F019 JMP $FFFF, F01C JMP $FFFF
            0x4C, 0x00, 0xD8]                                # F01F JMP $D800
    vsync = [0xA2, 0xFF, 0x9A, 0xA9, 2, 0x85, 0, 0xA9, 0, 0x85, 0, 0x4C, 0x00, 0xF0]
    bank = bytearray([0xEA]) * 4096
    bank[:len(code)] = bytes(code)
    bank[0x800:0x800 + len(vsync)] = bytes(vsync)
    bank[0xFFC:] = bytes([0x00, 0xF0, 0x00, 0xD8])           # CLD is the vector's high byte: $D800, ROM offset $800
    return bytes(bank) * 2


def last_key_states(rom, n):
    """Lane 0 halted; the others part by RAM $90."""
    st = np.array([oracle.reset_state(rom)] * n, dtype=oracle.STATE_DTYPE)
    st["ram"][:, 0x10], st["ram"][:, 0x11] = np.arange(n) & 1, 0
    st["run_status"] = 0
    st["run_status"][0] = 1
    return st


def test_every_lane_at_the_last_scheduling_key(warp):
    """Past frame 127 of a call and 511 hotspot accesses, a lane at $FFFF has
    the greatest key there is, which lanes that do not run have too: the one
    that leads must run."""
    rom, n, k = last_key_rom(), 6, 130
    start = last_key_states(rom, n)
    acts = np.zeros((k, n), np.uint8)
    got = run_warps(warp, rom, start, acts, k, "pc", 400_000)
    ref = start.copy()
    oracle.run_batch(rom, ref, acts, k)
    assert (ref["frame_no"][1:] >= 130).all() and (ref["run_status"][1:] == 0).all()
    assert_same(got, ref, "last key")


@pytest.mark.gpu
def test_every_lane_at_the_last_scheduling_key_on_the_gpu():
    if fa.device_count() < 1:
        pytest.skip("no CUDA device")
    rom, n, k = last_key_rom(), 6, 130
    ref = last_key_states(rom, n)
    acts = np.zeros((k, n), np.uint8)
    with fa.BatchAtariGpu(rom, n) as g:
        g.upload_states(ref)
        g.step_multi(acts, k)
        got = g.download_states()
    oracle.run_batch(rom, ref, acts, k)
    assert_same(got, ref, "last key")
