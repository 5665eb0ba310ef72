"""The emulator's work as its users have it done, as cases that can be timed.

Every case goes through the package's public entry points (BatchAtariGpu,
BatchAtariGpuEnv, AtariPool, AtariRender, AtariServer) on the seeded synthetic
carts of the package, at the sizes of the repository's benchmark and tests.
A pass steps consoles by K frames and returns what the caller reads: the
RAM observations (or the f32 observations, rewards and flags of the RL
environment, the framebuffers and RGBA of the rendering console) and, where a
handle exposes them, the consoles' state rows in device memory.

Consoles start from the carts' post-reset state advanced by a few frames of
the case's own random actions, so that their RAM and control flow differ as in
a running program.  All outputs are whole numbers except the environment's
b / 255 observations.
"""
import importlib.util
import math
import os
import random
import sys

import numpy as np
import torch

MASK = (1 << 31) - 1


def _package():
    if "fast_atari_b200" in sys.modules:
        return sys.modules["fast_atari_b200"]
    d = os.path.join(os.getcwd(), "fast-atari-rs_b200")
    spec = importlib.util.spec_from_file_location("fast_atari_b200", os.path.join(d, "__init__.py"),
                                                  submodule_search_locations=[d])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["fast_atari_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


_carts = {}


def _cart(name):
    """A cart of the package by the short name the cases use, its scheme registered."""
    if name not in _carts:
        fa = _package()
        from fast_atari_b200 import carts
        c = {"plain": carts.plain_cart, "divergence": carts.divergence_cart, "scale": carts.scale_cart,
             "mixed2k": lambda: carts.mixed_carts()[0], "mixed8k": lambda: carts.mixed_carts()[1],
             "mixed16k": lambda: carts.mixed_carts()[2], "mixed32k": lambda: carts.mixed_carts()[3],
             "e0": carts.e0_cart, "3f16": lambda: carts.f3_cart(16384), "3f6": lambda: carts.f3_cart(6144),
             "dpc": carts.dpc_cart, "dpctail": lambda: carts.dpc_cart(dump_tail=True), "fe": carts.fe_cart,
             "render": carts.render_cart}[name]()
        if c.scheme:
            fa.set_rom_scheme(c.rom, c.scheme)
        _carts[name] = c.rom
    return _carts[name]


def listed():
    return [
        # One console stepped a frame at a time from host buffers: an interactive or evaluation run.
        # Latency: one serial chain of 6502 instructions, one launch, the copies around it.
        {"name": "one_console", "kind": "handle", "cart": "plain", "n": 1, "k": 1, "host": True, "persistent": False,
         "episode": 0},
        # The benchmark's plain configuration: 1,000 consoles, one host-buffer step per frame.
        {"name": "plain_step_1000", "kind": "handle", "cart": "plain", "n": 1000, "k": 1, "host": True,
         "persistent": False, "episode": 0},
        # The batched RL environment: one action broadcast, frameskip 4, f32 observations, rewards from RAM.
        {"name": "env_1024", "kind": "env", "cart": "mixed8k", "n": 1024, "k": 4},
        # The divergence configuration: 50,000 consoles of a branchy 8K F8 cart, one launch per frame on device buffers.
        {"name": "divergence_50000", "kind": "handle", "cart": "divergence", "n": 50_000, "k": 1, "host": False,
         "persistent": False, "episode": 0},
        # The headline batch: four carts of different mappers in one persistent launch, K = 4.
        {"name": "mixed_pool", "kind": "pool", "carts": "mixed2k,mixed8k,mixed16k,mixed32k",
         "counts": "100000,30000,5000,500", "k": 4, "host": False},
        # The scale configuration's million F4 consoles with periodic episode resets, a frameskip of 4 per call.
        {"name": "scale_1m", "kind": "handle", "cart": "scale", "n": 1_000_000, "k": 4, "host": False,
         "persistent": True, "episode": 2000},
        # Parker Brothers E0 and Tigervision 3F carts in one pool (the benchmark's mappers workload).
        {"name": "mappers_pool", "kind": "pool", "carts": "e0,3f16,3f6", "counts": "40000,40000,20000", "k": 4,
         "host": False},
        # DPC carts, both dump lengths (the benchmark's dpc workload).
        {"name": "dpc_pool", "kind": "pool", "carts": "dpc,dpctail", "counts": "40000,40000", "k": 4, "host": False},
        # Activision FE carts (the benchmark's fe workload).
        {"name": "fe_pool", "kind": "pool", "carts": "fe", "counts": "80000", "k": 4, "host": False},
        # The rendering console, one full wave of the benchmark's render workload, framebuffers left on the device.
        {"name": "render_75776", "kind": "render", "cart": "render", "n": 75_776, "k": 4, "rgba": False},
        # Pixels for a learner or a viewer: 2,048 rendering consoles, four frames, then RGBA on the device.
        {"name": "render_rgba_2048", "kind": "render", "cart": "render", "n": 2048, "k": 4, "rgba": True},
        # The continuous-batching server: 60 sessions over the four mixed carts, one request each, lognormal batch
        # sizes (median 256) and K of 1 to 8, as the serving benchmark draws them.
        {"name": "serve_60", "kind": "serve", "sessions": 60, "median": 256, "most": 4096, "sizes": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["handle", "handle", "env", "pool", "pool", "render", "serve"])
    if kind == "handle":
        cart = rng.choice(["plain", "divergence", "scale", "mixed2k", "mixed8k", "mixed16k", "mixed32k", "e0", "dpc", "fe"])
        return {"kind": kind, "cart": cart, "n": _log_int(rng, 1, 60_000), "k": rng.choice([1, 1, 2, 4]),
                "host": rng.random() < 0.5, "persistent": rng.random() < 0.5, "episode": rng.choice([0, 0, 500])}
    if kind == "env":
        return {"kind": kind, "cart": rng.choice(["plain", "mixed8k", "mixed16k", "divergence"]),
                "n": _log_int(rng, 8, 8192), "k": rng.choice([1, 2, 4, 5])}
    if kind == "pool":
        family = rng.choice([["plain", "mixed2k", "mixed8k", "mixed16k", "mixed32k", "divergence"],
                             ["e0", "3f16", "3f6"], ["dpc", "dpctail"], ["fe"],
                             ["plain", "mixed8k", "e0", "3f16", "dpc", "fe"]])
        names = sorted(rng.sample(family, rng.randint(1, min(4, len(family)))))
        return {"kind": kind, "carts": ",".join(names), "counts": ",".join(str(_log_int(rng, 33, 25_000)) for _ in names),
                "k": rng.randint(1, 4), "host": rng.random() < 0.4}
    if kind == "render":
        rgba = rng.random() < 0.5
        return {"kind": kind, "cart": rng.choice(["render", "divergence", "mixed8k"]),
                "n": _log_int(rng, 16, 4096 if rgba else 20_000), "k": rng.choice([1, 2, 4]), "rgba": rgba}
    return {"kind": kind, "sessions": rng.randint(4, 60), "median": _log_int(rng, 64, 512), "most": 4096,
            "sizes": rng.randint(1, MASK)}


class _DeviceArray:
    """Device memory of the library as torch can wrap it (no copy).  The tensor keeps this object, and so the
    memory's owner, alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _rows(fa, g, owner):
    """The state rows of a handle: (rows, stride) 32-bit words in device memory."""
    import ctypes
    stride = ctypes.c_uint32()
    ptr = fa.lib().fa_device_state(g._h, ctypes.byref(stride))
    return torch.as_tensor(_DeviceArray(owner, ptr, (67, stride.value), "<i4"), device="cuda")


def _actions(rng, n, k):
    return torch.randint(0, 18, (k * n,), dtype=torch.uint8, device="cuda", generator=rng)


def prepare(case, seed):
    fa = _package()
    rng = torch.Generator(device="cuda").manual_seed((seed * 1_000_003 + 17) & MASK)
    kind = case["kind"]
    s = {"case": case, "fa": fa}
    if kind == "handle":
        n, k = case["n"], case["k"]
        g = s["g"] = fa.BatchAtariGpu(_cart(case["cart"]), n)
        g.set_launch(128, "pc", case["persistent"])
        g.reset()
        if case["episode"]:                                   # episodes end at different frames, as in a running job
            g.set_episode_frames(case["episode"])
            g.set_frame_numbers(np.random.RandomState(seed & MASK).randint(0, case["episode"], n).astype(np.uint32))
        warm = _actions(rng, n, 3)
        torch.cuda.synchronize()
        g.step_multi_async(warm.data_ptr(), 3)
        g.synchronize()
        s["rows"] = _rows(fa, g, g)
        a = _actions(rng, n, k)
        if case["host"]:
            s["actions"] = a.cpu().numpy()
        else:
            s["actions"] = a
            s["obs"] = torch.zeros(n, 128, dtype=torch.uint8, device="cuda")
    elif kind == "env":
        from fast_atari_b200.env import BatchAtariGpuEnv
        env = s["env"] = BatchAtariGpuEnv(_cart(case["cart"]), case["n"]).with_frameskip(case["k"])
        # Score, lives and an end flag at RAM bytes that the synthetic carts change.
        env.with_reward(fa.RewardSpec.make(score=(2, 3, 4), bcd=True, lives=(5, 0x70, 4), terminal=(6, 0x81, 0x81)))
        env.reset()
        s["todo"] = [int(v) for v in torch.randint(0, 18, (64,), generator=rng, device="cuda").cpu()]
        s["at"] = 0
        env.step(s["todo"][0])
    elif kind == "pool":
        k = case["k"]
        counts = [int(c) for c in case["counts"].split(",")]
        pool = s["pool"] = fa.AtariPool()
        for name, n in zip(case["carts"].split(","), counts):
            pool.add_cart(_cart(name), n)
        warm = [_actions(rng, n, 3) for n in counts]
        torch.cuda.synchronize()
        pool.step_async([w.data_ptr() for w in warm], 3)
        pool.synchronize()
        s["rows"] = [_rows(fa, pool.group(i), pool) for i in range(len(counts))]
        a = [_actions(rng, n, k) for n in counts]
        if case["host"]:
            s["actions"] = [x.cpu().numpy() for x in a]
            s["out"] = [np.zeros((n, 128), np.uint8) for n in counts]
        else:
            s["actions"] = a
            s["obs"] = [torch.zeros(n, 128, dtype=torch.uint8, device="cuda") for n in counts]
    elif kind == "render":
        n, k = case["n"], case["k"]
        r = s["r"] = fa.AtariRender(_cart(case["cart"]), n)
        fa._check(fa.lib().fa_render_reset(r._r, None, None))
        warm = _actions(rng, n, 2)
        torch.cuda.synchronize()
        r.step_multi_async(warm.data_ptr(), 2)
        r.synchronize()
        s["actions"] = _actions(rng, n, k)
        s["obs"] = torch.zeros(n, 128, dtype=torch.uint8, device="cuda")
        s["fb"] = torch.as_tensor(_DeviceArray(r, r.device_framebuffers(), (n, 192, 160), "|u1"), device="cuda")
        if case["rgba"]:
            s["rgba"] = torch.zeros(n, 192, 160, 4, dtype=torch.uint8, device="cuda")
    else:
        srv = s["srv"] = fa.AtariServer([_cart(c) for c in ("mixed2k", "mixed8k", "mixed16k", "mixed32k")])
        s["requests"] = []
        for i, (n, k) in enumerate(_request_sizes(case)):
            a = _actions(rng, n, k).cpu().numpy()
            sid = srv.open(i % 4)
            srv.step(sid, a[:n], n, 1)                          # admitted; its consoles have run a frame
            s["requests"].append((sid, a, n, k))
    torch.cuda.synchronize()
    return s


def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "handle":
        g = s["g"]
        if case["host"]:
            if case["k"] == 1:
                return {"ram": g.step(s["actions"]), "state": s["rows"]}
            return {"ram": g.step_multi(s["actions"], case["k"]), "state": s["rows"]}
        g.step_multi_async(s["actions"].data_ptr(), case["k"], s["obs"].data_ptr())
        return {"ram": s["obs"], "state": s["rows"]}
    if kind == "env":
        s["at"] = (s["at"] + 1) % len(s["todo"])
        st = s["env"].step(s["todo"][s["at"]])
        return {"observation": st.observation, "reward": st.reward, "terminated": st.terminated,
                "life_lost": st.life_lost}
    if kind == "pool":
        if case["host"]:
            return {"ram": s["pool"].step(s["actions"], case["k"], out=s["out"]), "state": s["rows"]}
        s["pool"].step_async([a.data_ptr() for a in s["actions"]], case["k"], [o.data_ptr() for o in s["obs"]])
        return {"ram": s["obs"], "state": s["rows"]}
    if kind == "render":
        r = s["r"]
        r.step_multi_async(s["actions"].data_ptr(), case["k"], s["obs"].data_ptr())
        if case["rgba"]:
            r.rgba_async(0, case["n"], s["rgba"].data_ptr())
            return {"framebuffers": s["fb"], "ram": s["obs"], "rgba": s["rgba"]}
        return {"framebuffers": s["fb"], "ram": s["obs"]}
    tickets = [s["srv"].submit(sid, a, n, k) for sid, a, n, k in s["requests"]]
    return [s["srv"].wait(t)[0] for t in tickets]


def _request_sizes(case):
    """(n, k) of the server case's requests: part of the case, so every seed's requests have the same sizes."""
    r = random.Random(case["sizes"])
    return [(min(case["most"], max(16, int(round(r.lognormvariate(math.log(case["median"]), 1.0))))), r.randint(1, 8))
            for _ in range(case["sessions"])]


def work(case):
    """Bytes only: the emulation itself is integer work on registers.  Per console: its 57 state words (the DPC
    rows too for DPC carts) read and written, K actions read, 128 bytes of RAM written."""
    kind = case["kind"]
    per = lambda cart, k: 2 * 4 * (67 if cart.startswith("dpc") else 57) + k + 128  # noqa: E731
    if kind == "handle":
        return {"bytes": case["n"] * per(case["cart"], case["k"])}
    if kind == "env":                                          # and the f32 observations, reward and flags
        return {"bytes": case["n"] * (per(case["cart"], case["k"]) + 512 + 4 + 2)}
    if kind == "pool":
        return {"bytes": sum(int(n) * per(c, case["k"]) for c, n in zip(case["carts"].split(","), case["counts"].split(",")))}
    if kind == "render":                                       # 63 state words; the framebuffer, and RGBA
        return {"bytes": case["n"] * (2 * 4 * 63 + case["k"] + 128 + 30_720 * (1 + 5 * bool(case["rgba"])))}
    return {"bytes": sum(n * per("", k) for n, k in _request_sizes(case))}


def exact(case, seed):
    """No output has a value in 64 bits that a formula gives: RAM, state, pixels and flags are whole numbers that only
    an emulator produces (the repository's tests compare them with one), and the f32 ones are made of them."""
    return None
