// fa_render.cuh — one rendering console per lane: the frame loop, shared by
// the rendering kernel (fa_render.cu) and the host tests that run the same
// code on the CPU.  The kernel's start and end of a launch (the console's
// rows in and out of HBM) stay in the kernel body: moved into helpers here,
// the same steps ran 8 % slower on the render cart.
#pragma once

#include "fa_run.cuh"

namespace fa {

// One rendering console per lane: HeadlessAtari's frame loop with the
// rendering console's per-cycle run_one_cycle (src/atari.rs:284-318).
template <bool SLICED>
struct RRunner {
    Emu<32, true, SLICED> e;
    uint32_t f, phase;
    uint32_t fcyc;           // WSYNC wait cycles of the frame (Emu::cyc_acc has its instruction cycles)
    bool active;

    // set_action, then run_frame, which does nothing for a halted console
    // (src/atari.rs:250-270, 284-306): a halted console's inputs still take
    // the frame's action.
    __device__ __forceinline__ bool begin_frame()
    {
        const FaGroup* G = e.G;
        if (G->actions) e.apply_action(G->actions[(size_t)f * G->act_stride + e.i]);
        if (e.row(R_STATUS) & FA_STATUS_HALT_MASK) return false;
        e.tw &= ~TW_FCOMP;
        e.kb = (f < 0x7Fu ? f : 0x7Fu) << 25;
        fcyc = 0;
        phase = e.vsync_on() ? 0u : 1u;
        e.done = due();
        return true;
    }
    // The instruction cycles at which the frame loop must look: the VSYNC
    // budget's or the frame cap's, less the frame's WSYNC waits; after
    // attend's checks above cyc_acc.
    __device__ __forceinline__ uint32_t due() const { return (phase ? FA_FRAME_CYCLE_CAP : FA_VSYNC_BUDGET) + 1u - fcyc; }

    // After an instruction (ran), the frame-end checks of run_frame, then any
    // WSYNC wait it started, as a run_one_cycle of its own; until the frame
    // loop has nothing to do at an instruction boundary.
    __device__ __forceinline__ void attend(bool ran)
    {
#pragma unroll 1
        while (true) {
            if (ran) {
                const uint32_t fc = e.cyc_acc + fcyc;
                if (phase == 0u) {
                    if (fc > FA_VSYNC_BUDGET) {
                        e.fold_cycles();
                        e.set_status(FA_STATUS_VSYNC_BUDGET);
                        active = false;
                        return;
                    }
                    if (!e.vsync_on()) {
                        // VSYNC may drop with the (smaller) cap more than
                        // spent: spent to the cycle, it ends the frame after
                        // the next instruction or cycle of a wait too.
                        phase = 1u;
                        if (fc > FA_FRAME_CYCLE_CAP) fcyc = FA_FRAME_CYCLE_CAP - e.cyc_acc;
                    }
                } else {
                    const bool cap = fc > FA_FRAME_CYCLE_CAP;
                    if (cap || e.vsync_on()) {
                        if (cap) e.set_status(FA_STATUS_CYCLE_CAP);
                        e.fb_observe();                              // before the next frame's action moves the pins
                        e.fold_cycles();
                        e.row(R_FRAME) += 1u;
                        f++;
                        if (f >= e.G->k || !begin_frame()) { active = false; return; }
                    }
                }
            }
            if (!e.wsync()) break;
            e.settle();                                              // the wait starts where the beam is
            if (!e.wsync()) break;
            // The cycles of a WSYNC wait up to the end of the line, cut where
            // a per-cycle frame check would first fire: nothing else changes
            // from one cycle of the wait to the next.
            uint32_t n = (228u - e.clock + 2u) / 3u, lim = 1u;
            if (phase || e.vsync_on()) lim = due() - e.cyc_acc;
            n = n < lim ? n : lim;
            e.rcycles(n);
            fcyc += n;
            ran = true;
        }
        e.done = due();
    }

    __device__ __forceinline__ uint32_t key(uint32_t sched) const
    {
        if (sched != FA_SCHED_LINE) return e.kb | (e.pc & 0xFFFFu);
        return (e.kb & 0xFE000000u) | ((e.scanline < 0x1FEu ? e.scanline : 0x1FEu) << 16) | (e.pc & 0xFFFFu);
    }
    __device__ __forceinline__ uint32_t place() const { return (e.kb & 0x01FF0000u) | (e.bank << 13) | (e.pc & 0xFFFFu); }
    // Instructions of this lane up to one that may leave the lanes of its
    // group at different pcs, that reaches a waiting lane's key, or after
    // which the frame loop must look (and the WSYNC waits it started).
    __device__ __forceinline__ void burst(uint32_t wait_key)
    {
        if (e.wsync()) {
            attend(false);
            if (!active) return;
        }
        if (!e.run(wait_key, [this](uint32_t) { attend(true); return active; })) {
            // The reference's opcode fetch was a bus access (one cycle of TIA
            // and PIA) before it stopped (src/cpu.rs:1139-1141): the TIA and
            // PIA are owed up to the end of that cycle.
            e.lag += 1u;
            e.plag += 1u;
            e.fold_cycles();
            e.set_status(FA_STATUS_ILLEGAL_OPCODE);
            active = false;
            return;
        }
    }
    __device__ __forceinline__ void iterate() { burst(0xFFFFFFFFu); }
};

}  // namespace fa
