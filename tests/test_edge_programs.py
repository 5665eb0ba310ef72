"""The table-driven interpreter at the edges of its straight path, against the oracle.

Programs whose operands sit where the straight path hands over: pages and
zero page ends, pointers and stacks at the RAM's borders, registers and their
mirrors (INTIM before and after its underflow), hotspots and the bytes around
them, $01FE, RMW on all of these, decimal mode on and off, branches near page
ends.  Every state and byte of RAM must equal the oracle's (integers: no
tolerance), on the host and on the GPU, in the build of the cart's own core
and in the one that holds every core.
"""
import numpy as np
import pytest

import oracle
from fa_pkg import carts, fa
from test_host_sim import assert_same, run_both, sim  # noqa: F401  (the fixture)

ZP = [0x00, 0x01, 0x02, 0x04, 0x08, 0x0C, 0x1B, 0x1C, 0x2A, 0x3F, 0x7E, 0x7F, 0x80, 0x81, 0xFD, 0xFE, 0xFF]
ABS = [0x0000, 0x003F, 0x0040, 0x007F, 0x0080, 0x00FF, 0x017F, 0x0180, 0x01FE, 0x01FF, 0x0200, 0x027F, 0x0280, 0x0282, 0x0284,
       0x0285, 0x0294, 0x0295, 0x0296, 0x0297, 0x02FF, 0x0480, 0x0F84, 0x0FFF, 0x1000, 0x1008, 0x103F, 0x1040, 0x107F, 0x10FF,
       0x1100, 0x1EFF, 0x1F00, 0x1FDF, 0x1FE0, 0x1FF3, 0x1FF4, 0x1FF8, 0x1FF9, 0x1FFA, 0x1FFF, 0x2084, 0xF0FF, 0xFFFE]
KINDS = {"4k": (4096, -1), "8k": (8192, -1), "16k": (16384, -1), "32k": (32768, -1), "e0": (8192, 4), "3f": (8192, 5),
         "dpc": (10240, -1), "fe": (8192, 7)}


def program(rng, size):
    """A ROM of random legal instructions with the operands above (every 4K bank its own)."""
    legal = carts.LEGAL_OPCODES
    size_of = {op: carts._SIZE[mode] for (_, mode), op in carts.OPCODES.items()}
    mode_of = {op: mode for (_, mode), op in carts.OPCODES.items()}
    rom = bytearray()
    while len(rom) < size:
        op = int(legal[rng.integers(len(legal))])
        if op in (0x00, 0x40, 0x4C, 0x6C) and rng.random() < 0.8:
            continue
        n, mode = size_of[op], mode_of[op]
        if n == 1:
            rom += bytes([op])
        elif mode == "rel":
            rom += bytes([op, int(rng.integers(0, 12)) if rng.random() < 0.9 else int(rng.integers(0, 256))])
        elif n == 2:
            rom += bytes([op, int(rng.choice(ZP)) if rng.random() < 0.7 else int(rng.integers(0, 256))])
        else:
            a = int(rng.choice(ABS)) if rng.random() < 0.8 else int(rng.integers(0, 65536))
            if op in (0x20, 0x4C):
                a = 0xF000 + int(rng.integers(0, 0xF00))
            rom += bytes([op, a & 0xFF, a >> 8])
    rom = rom[:size]
    for b in range(min(size, 32768) // 4096):
        rom[b * 4096 + 0xFFC:b * 4096 + 0xFFE] = bytes([0x00, 0xF0])
    return bytes(rom)


def states(rng, rom, n):
    st = np.array([oracle.reset_state(rom)] * n, dtype=oracle.STATE_DTYPE)
    for f in ("a", "x", "y"):
        st[f] = rng.integers(0, 256, n)
    st["sp"] = rng.choice([0x7E, 0x7F, 0x80, 0x81, 0x82, 0xFB, 0xFC, 0xFD, 0xFE, 0xFF, 0x00], n)
    st["status"] = rng.integers(0, 256, n) & 0xCF
    st["pc"] = rng.choice([0xF000, 0xF0FD, 0xF0FE, 0xF3FD, 0xF3FE, 0xF7FF, 0xFFE0, 0xFFF0, 0x1FF6, 0x0080, 0xF900], n)
    st["ram"] = rng.choice(np.array(ZP + [0x10, 0x1F, 0x02, 0xF0], dtype=np.uint8), (n, 128))
    st["timer_value"] = rng.integers(0, 4, n)
    st["timer_prescaler_select"] = rng.choice([1, 8, 64, 1024], n)
    st["timer_prescaler"] = 1
    st["timer_underflow"] = rng.integers(0, 2, n)
    for f in ("cxm0p", "cxppmm"):
        st[f] = rng.integers(0, 256, n)
    st["run_status"] = 0
    return st


@pytest.mark.parametrize("kind", KINDS)
def test_edges_on_the_host(sim, kind):  # noqa: F811
    size, code = KINDS[kind]
    rng = np.random.default_rng(len(kind) * 1000 + size + code)
    for t in range(6):
        rom = program(rng, size)
        r = np.frombuffer(rom, np.uint8).copy()
        if code >= 0:
            sim.fa_rom_set_scheme(r.ctypes.data, len(r), code)
            oracle.set_rom_scheme(rom, code)
        try:
            got, ref = run_both(sim, rom, states(rng, rom, 96), carts.actions(seed=t, n=96, frames=2), 2)
            assert_same(got, ref, f"{kind} program {t}")
        finally:
            if code >= 0:
                sim.fa_rom_set_scheme(r.ctypes.data, len(r), -1)
                oracle.set_rom_scheme(rom, "auto")


@pytest.mark.gpu
@pytest.mark.parametrize("sched", ["pc", "line", "lane"])
@pytest.mark.parametrize("kind", KINDS)
def test_edges_on_the_gpu(kind, sched):
    """Warps of lanes at different pcs; alone, and in a pool with a cart of another core."""
    if fa.device_count() < 1:
        pytest.skip("no CUDA device")
    size, code = KINDS[kind]
    rng = np.random.default_rng(len(kind) * 1000 + size + code + 7)
    n, k = 96, 2
    rom = program(rng, size)
    if code >= 0:
        fa.set_rom_scheme(rom, code)
        oracle.set_rom_scheme(rom, code)
    try:
        ref = states(rng, rom, n)
        start, acts = ref.copy(), carts.actions(seed=3, n=n, frames=k)
        oracle.run_batch(rom, ref, acts, k)
        with fa.BatchAtariGpu(rom, n) as g:
            g.set_launch(128, sched, False)
            g.upload_states(start)
            g.step_multi(acts, k)
            assert_same(g.download_states(), ref, f"{kind} {sched}")
        other = carts.plain_cart().rom if kind in ("e0", "3f", "dpc", "fe") else carts.dpc_cart().rom
        with fa.AtariPool() as p:
            p.add_cart(rom, n)
            p.add_cart(other, 33)
            p.set_group(0, sched)
            p.group(0).upload_states(start)
            p.step([acts, np.zeros((k, 33), np.uint8)], k)
            assert_same(p.group(0).download_states(), ref, f"{kind} {sched} in a mixed pool")
    finally:
        if code >= 0:
            fa.set_rom_scheme(rom, "auto")
            oracle.set_rom_scheme(rom, "auto")


@pytest.mark.parametrize("kind", ["4k", "8k", "32k", "e0", "3f"])
def test_edges_on_the_rendering_console(sim, kind):  # noqa: F811
    """The same programs from power-on on the rendering console (the reference's Atari + Tia restated)."""
    size, code = KINDS[kind]
    rng = np.random.default_rng(len(kind) * 1000 + size + code + 14)
    for t in range(4):
        rom = program(rng, size)
        r = np.frombuffer(rom, np.uint8).copy()
        if code >= 0:
            sim.fa_rom_set_scheme(r.ctypes.data, len(r), code)
            oracle.set_rom_scheme(rom, code)
        try:
            n, calls, k = 3, 2, 1
            acts = np.stack([carts.actions(seed=90 + i, n=n, frames=k) for i in range(calls)])
            fb, ram = np.zeros((n, 192, 160), np.uint8), np.zeros((n, 128), np.uint8)
            st = np.zeros(n, fa.STATE_DTYPE)
            a = np.ascontiguousarray(acts, dtype=np.uint8)
            assert sim.hs_render(r.ctypes.data, len(r), n, a.ctypes.data, calls, k, fb.ctypes.data, st.ctypes.data,
                                 ram.ctypes.data) >= 0
            consoles = oracle.render_reset(rom, n)
            for i in range(calls):
                oracle.render_steps(consoles, acts[i])
            for i, c in enumerate(consoles):
                what, s, v = f"{kind} program {t}, rendering console {i}", st[i], [int(x) for x in c.regs()]
                assert np.array_equal(fb[i], c.tia_record()["fb"]), what
                assert np.array_equal(ram[i], c.ram()), what
                # Not the frame number: a console may halt in its reset frame.
                assert [int(s["a"]) | int(s["x"]) << 8 | int(s["y"]) << 16 | int(s["sp"]) << 24,
                        int(s["pc"]) | int(s["status"]) << 16 | int(s["bank"]) << 24, int(s["cycles"]),
                        int(s["tia_clock"]) | int(s["tia_scanline"]) << 16, int(s["run_status"]),
                        int(s["timer_value"]) | int(s["timer_prescaler"]) << 16] == \
                       [v[0], v[1], v[2] | v[3] << 32, v[4], v[6], v[7]], what
        finally:
            if code >= 0:
                sim.fa_rom_set_scheme(r.ctypes.data, len(r), -1)
                oracle.set_rom_scheme(rom, "auto")
