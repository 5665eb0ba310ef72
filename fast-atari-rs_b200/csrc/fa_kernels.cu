// fa_kernels.cu — launches of the batched Atari core on sm_100a.
//
// One kernel, fa_run (fa_core_kernels.cu), serves both launch forms of the
// library:
//   * plain:      one CTA per work unit (grid = number of units);
//   * persistent: grid sized to the SMs, each CTA pops work units from a
//                 device counter until the queue is empty.
// A work unit is up to BLOCK consecutive instances of one group (one cart's
// instance set).  Groups of different carts, instance counts, frame counts
// and scheduling policies share one launch.  When a CTA's next unit belongs
// to a different cart than the ROM it holds, it re-stages the ROM into shared
// memory with TMA bulk copies (cp.async.bulk, no multicast) on an mbarrier.
//
// Every wait is bounded; on expiry the kernel records FA_DEVERR_* in the
// launch's error word and leaves the unit untouched.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fa_internal.h"

namespace fa {

// Every instance column of `state` becomes a copy of `col` (FA_ROWS words).
__global__ void fa_broadcast(uint32_t* state, uint32_t stride, uint32_t n, const uint32_t* col)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        for (uint32_t w = 0; w < FA_ROWS; w++) state[(size_t)w * stride + i] = col[w];
}

}  // namespace fa

// ------------------------------------------------------------------ host launchers
// Lay out the ROM library (one copy per distinct ROM buffer); returns its size.
static uint32_t plan_romlib(FaLaunch& L)
{
    uint32_t bytes = 0;
    for (uint32_t g = 0; g < L.ngroups; g++) {
        L.g[g].rom_owner = 1;
        for (uint32_t h = 0; h < g; h++)
            if (L.g[h].rom == L.g[g].rom) { L.g[g].rom_off = L.g[h].rom_off; L.g[g].rom_owner = 0; break; }
        if (L.g[g].rom_owner) { L.g[g].rom_off = bytes; bytes += L.g[g].nbanks * 4096u; }
    }
    return bytes;
}

static void plan_units(FaLaunch& L, uint32_t unit)
{
    uint32_t units = 0;
    for (uint32_t g = 0; g < L.ngroups; g++) {
        L.g[g].unit_begin = units;
        units += (L.g[g].n + unit - 1) / unit;
    }
    L.nunits = units;
}

// The warps per CTA of a persistent launch that names none.  The build for
// more warps holds a thread to fewer registers (65,536 / (32 x warps)); the
// 32-warp one spills in the interpreter loop, and a lone warp is 16 % slower
// in it.  So:
// - 4K-bank carts: the smallest of 24, 28 and 32 that takes all units in one
//   wave (20,000 mixed consoles x 4 frames: 6.4 ms at 24, 7.2 at 32; 135,500:
//   17.2 at 28, two waves, 13.9 at 32).
// - E0 / 3F carts: 24 (100,000 consoles x 4 frames: 62 ms; 72 at 28, 69 at 32).
// - DPC, FE: CTAs of 4 (96 registers) while they can hold all units at once, up
//   to 16 units per SM (16,000 DPC consoles x 2 frames: 1.42 against 1.59 ms,
//   FE 2.57 against 2.81; at 21 per SM 3.38 against 2.72), then 24.
// - carts of several kinds: CTAs of 4.  Every kind's core is in use on every
//   SM, and fewer warps ask less of the instruction cache (100,000 consoles of
//   plain, DPC, FE and 8 KB carts x 2 frames: 7.7 ms at 4, 10.8 at 16, 8.9 at
//   24, 14.5 at 32; 600 consoles: 2.8, 3.0, 3.6, 4.1; nine carts, where the
//   library leaves room for one CTA of 4 or 8 warps: 28 and 44 ms).  Not the
//   best everywhere: from a library of 83 KB on one CTA of 4 is all that an SM
//   holds, which costs once there is more than a wave of them (with an E0
//   cart, x 2 frames, at 4, 8, 16 and 24 warps: 100,000 consoles and 32 KB of
//   library 16.6, 18.3, 17.9, 21.4 ms, 84 KB 28.3, 18.3, 17.5, 21.3, 124 KB
//   20.4, 17.9, 19.7, 20.3; 20,000 consoles and 84 KB 11.1, 11.0, 11.6, 12.8).
static int auto_warps(int maps, uint32_t units, uint32_t lib, uint32_t slab, int sms)
{
    const uint32_t per = sms > 0 ? (units + (uint32_t)sms - 1u) / (uint32_t)sms : units;
    if (maps == FA_MAPS_4K) return per <= 24u ? 24 : per <= 28u ? 28 : 32;
    if (maps == FA_MAPS_SLICED) return 24;
    if (maps == FA_MAPS_BOTH) return 4;
    // What 4-warp CTAs keep resident: by shared memory (9 KB of tables and 1 KB
    // of the system's per CTA), at most 20 warps of 96 registers.
    const uint32_t ctas = FA_SMEM_PER_SM / (lib + 4u * slab + 10240u);
    return per <= 16u && per <= 4u * ctas ? 4 : 24;
}

// The warp-granular layout of a launch: the ROM library, 32-instance work
// units and the warps per CTA.  False when the library leaves no room for
// block / 32 warp slabs (the launch is CTA-granular).
static bool warp_layout(FaLaunch& L, int block, bool persistent, int sms, int* warps)
{
    const uint32_t lib = plan_romlib(L);
    L.romlib_bytes = lib;
    const int maps = fa_maps_of(L.g, L.ngroups);
    const uint32_t slab = fa_slab_words(maps) * 32u * 4u;
    const int fit = (int)((FA_SMEM_PER_CTA_MAX - (int)lib) / (int)slab);
    if (fit < block / 32) return false;
    plan_units(L, 32u);
    int w = block / 32;
    if (persistent) {
        // As many as shared memory allows, up to the cap.
        const int cap = L.cta_warps ? (int)L.cta_warps : auto_warps(maps, L.nunits, lib, slab, sms);
        static const int sizes[] = { 32, 28, 24, 16, 8, 4, 2 };
        for (int x : sizes)
            if (x <= fit && x <= cap) { w = x; break; }
    }
    *warps = w;
    return true;
}

// sms: the device's; launch_sms: the same, or 0 to prepare the launch only.
static cudaError_t launch(const FaLaunch& L_in, int block, bool persistent, int sms, int launch_sms, cudaStream_t s)
{
    FaLaunch L = L_in;
    L.wait_ns = fa_wait_limit_ns();
    const int maps = fa_maps_of(L.g, L.ngroups);                       // which cores the carts need
    int warps = 0;
    if (warp_layout(L, block, persistent, sms, &warps)) {
        return maps == FA_MAPS_4K   ? FaCore<FA_MAPS_4K>::run_warps(warps, L, persistent, launch_sms, s)
             : maps == FA_MAPS_BOTH ? FaCore<FA_MAPS_BOTH>::run_warps(warps, L, persistent, launch_sms, s)
             : maps == FA_MAPS_DPC  ? FaCore<FA_MAPS_DPC>::run_warps(warps, L, persistent, launch_sms, s)
             : maps == FA_MAPS_FE   ? FaCore<FA_MAPS_FE>::run_warps(warps, L, persistent, launch_sms, s)
                                    : FaCore<FA_MAPS_SLICED>::run_warps(warps, L, persistent, launch_sms, s);
    }
    // ROM library too large for shared memory (with blocks of 128
    // over 200 KB, over 196 with DPC carts or several kinds):
    // CTA-granular units that re-stage one cart's ROM at a time.  100,000 4K-bank
    // consoles x 2 frames: 17.0 ms with 196 KB (resident), 7.3 with 204 (re-staged).
    plan_units(L, (uint32_t)block);
    return maps == FA_MAPS_4K   ? FaCore<FA_MAPS_4K>::run_block(block, L, persistent, launch_sms, s)
         : maps == FA_MAPS_BOTH ? FaCore<FA_MAPS_BOTH>::run_block(block, L, persistent, launch_sms, s)
         : maps == FA_MAPS_DPC  ? FaCore<FA_MAPS_DPC>::run_block(block, L, persistent, launch_sms, s)
         : maps == FA_MAPS_FE   ? FaCore<FA_MAPS_FE>::run_block(block, L, persistent, launch_sms, s)
                                : FaCore<FA_MAPS_SLICED>::run_block(block, L, persistent, launch_sms, s);
}

cudaError_t fa_launch_run(const FaLaunch& L, int block, bool persistent, int sms, cudaStream_t s)
{
    return launch(L, block, persistent, sms, sms, s);
}

bool fa_launch_warp_shape(const FaLaunch& L_in, int block, bool persistent, int sms, uint32_t* grid, uint32_t* warps,
                          int* per_sm)
{
    FaLaunch L = L_in;
    const int maps = fa_maps_of(L.g, L.ngroups);
    int w = 0;
    if (!warp_layout(L, block, persistent, sms, &w)) return false;
    *warps = (uint32_t)w;
    return maps == FA_MAPS_4K   ? FaCore<FA_MAPS_4K>::shape(w, L, persistent, sms, grid, per_sm)
         : maps == FA_MAPS_BOTH ? FaCore<FA_MAPS_BOTH>::shape(w, L, persistent, sms, grid, per_sm)
         : maps == FA_MAPS_DPC  ? FaCore<FA_MAPS_DPC>::shape(w, L, persistent, sms, grid, per_sm)
         : maps == FA_MAPS_FE   ? FaCore<FA_MAPS_FE>::shape(w, L, persistent, sms, grid, per_sm)
                                : FaCore<FA_MAPS_SLICED>::shape(w, L, persistent, sms, grid, per_sm);
}

cudaError_t fa_launch_prepare(const FaLaunch& L, int block, bool persistent, int sms)
{
    return launch(L, block, persistent, sms, 0, nullptr);
}

int fa_launch_occupancy(int block, uint32_t rom_bytes_max)
{
    const size_t base = (size_t)rom_bytes_max + (size_t)fa_slab_words(FA_MAPS_4K) * block * 4u;
    return FaCore<FA_MAPS_4K>::occupancy(block, base);
}

cudaError_t fa_launch_broadcast(uint32_t* state, uint32_t stride, uint32_t n, const uint32_t* col, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    uint32_t grid = (n + 255u) / 256u;
    if (grid > 4096u) grid = 4096u;
    fa::fa_broadcast<<<grid, 256, 0, s>>>(state, stride, n, col);
    return cudaGetLastError();
}
