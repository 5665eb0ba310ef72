"""The warps per CTA that a persistent launch picks by its carts and their
number: on both sides of every line of the rule, the same results as a launch
that names 8 warps per CTA (whose results the pool tests hold to the oracle)."""
import numpy as np
import pytest

from fa_pkg import carts, fa

pytestmark = pytest.mark.gpu

SMS = 148
FAMILIES = {
    "4k": lambda: [carts.plain_cart(), carts.mixed_carts()[2]],
    "sliced": lambda: [carts.e0_cart(), carts.f3_cart(6144)],
    "dpc": lambda: [carts.dpc_cart()],
    "fe": lambda: [carts.fe_cart()],
    "several": lambda: [carts.plain_cart(), carts.dpc_cart(), carts.fe_cart(), carts.e0_cart()],
}


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    if fa.device_count() < 1:
        pytest.skip("no CUDA device")


# Warps' worth of consoles per SM; the first cart holds all but 33 of each other.
@pytest.mark.parametrize("family,per_sm,extra", [
    ("4k", 0, 65), ("4k", 24, 0), ("4k", 24, 1), ("4k", 28, 0), ("4k", 28, 1),
    ("sliced", 0, 65), ("dpc", 0, 1), ("dpc", 16, 0), ("dpc", 16, 1), ("fe", 0, 1), ("fe", 16, 0), ("fe", 16, 1),
    ("several", 0, 130), ("several", 20, 1)])
def test_picked_warps_give_the_same_results(family, per_sm, extra):
    cs = FAMILIES[family]()
    total = per_sm * SMS * 32 + extra
    counts = [total - 33 * (len(cs) - 1)] + [33] * (len(cs) - 1)
    if family in ("4k", "several") and per_sm:
        counts[0] -= 31 * (len(cs) - 1)                  # the other carts' last warps are part-filled
    acts = [carts.actions(seed=7 + i, n=n, frames=1) for i, n in enumerate(counts)]
    got = []
    for warps in (0, 8):
        with fa.AtariPool() as pool:
            for c, n in zip(cs, counts):
                if c.scheme:
                    fa.set_rom_scheme(c.rom, c.scheme)
                pool.add_cart(c.rom, n)
            pool.set_launch(128, True, warps)
            obs = pool.step(acts, 1)
            got.append((obs, [pool.group(g).download_states() for g in range(len(cs))]))
    for g in range(len(cs)):
        assert np.array_equal(got[0][0][g], got[1][0][g])
        assert np.array_equal(np.asarray(got[0][1][g]), np.asarray(got[1][1][g]))


# Rendering consoles: the build for few consoles up to 8 warps per SM, and the
# other one past that, at every CTA size.
@pytest.mark.parametrize("n", [2 * SMS * 32, 4 * SMS * 32 - 1, 8 * SMS * 32, 8 * SMS * 32 + 1])
def test_rendering_builds_agree(n):
    c = carts.render_cart()
    acts = carts.actions(seed=11, n=n, frames=1)
    want = None
    for warps in (16, 8, 4):
        with fa.AtariRender(c.rom, n, cta_warps=warps) as r:
            r.reset()
            _, ram = r.step_multi(acts, 1, fb=False)
            got = (np.asarray(ram).copy(), r.states(), r.rgba(0, 32).copy(), r.rgba(n - 32, 32).copy())
        if want is None:
            want = got
        for a, b in zip(got, want):
            assert np.array_equal(a, b), f"{warps} warps"
