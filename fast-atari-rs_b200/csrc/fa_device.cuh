// fa_device.cuh — the per-thread Atari 2600 emulator for sm_100a.
//
// One thread emulates one console.  Its hot state lives in registers, its
// 128-byte PIA RAM in shared memory.  Headless consoles interleave the RAM by
// byte (byte o of thread t at o * BLOCK + t): one multiply to reach, up to
// four lanes at different offsets on a bank.  Their TIA registers that change
// only on a write stay in the HBM state rows; the DPC core's registers come
// into shared memory while a unit runs.  Rendering consoles keep RAM and
// graphics registers there, interleaved by 32-bit word (byte o of lane t in
// word (o/4)*32 + t), so that no two lanes meet on a bank.  ROM banks sit in
// shared memory, staged once per block.
//
// Semantics are those of the reference CPU emulator (RPP1011/fast-atari-rs):
//   src/cpu.rs            6502 step, including every phantom access whose
//                         side effect is visible on the Atari bus
//   src/atari.rs:460-552  HeadlessBus read/write decode and bank hotspots
//   src/atari.rs:584-614  run_frame / run_one_cycle
//   src/headless_tia.rs   HeadlessTia
//   src/pia.rs            Pia
// The interpreter (Emu::run) is driven by a table of eight words per opcode
// instead of a switch: most instructions run through one straight sequence of
// selects, so lanes at different opcodes share it too.
#pragma once
#include <stdint.h>

#include "fa_internal.h"
#include "fa_layout.h"

namespace fa {

// Instructions after which a converged group checks, at its next branch, that
// its lanes are still together (they check at once where a branch parts them,
// and after returns, indirect jumps and interrupts).
constexpr uint32_t FA_BURST = 32;

enum : uint32_t { F_C = 1, F_Z = 2, F_I = 4, F_D = 8, F_B = 16, F_U = 32, F_V = 64, F_N = 128 };

// Action -> (SWCHA | INPT4<<8 | paddle0<<16), src/atari.rs:34-81,571-582.
constexpr uint32_t act_word(int up, int down, int left, int right, int fire)
{
    return (0xFFu & ~(up ? 0x10u : 0u) & ~(down ? 0x20u : 0u) & ~(left ? 0x40u : 0u) & ~(right ? 0x80u : 0u))
         | ((fire ? 0u : 1u) << 8) | ((left ? 200u : right ? 50u : 128u) << 16);
}

// Action::decode order (src/atari.rs:59-80): up, down, left, right, fire.
static __constant__ uint32_t c_action_table[18] = {
    act_word(0, 0, 0, 0, 0), act_word(0, 0, 0, 0, 1), act_word(1, 0, 0, 0, 0), act_word(0, 0, 0, 1, 0),
    act_word(0, 0, 1, 0, 0), act_word(0, 1, 0, 0, 0), act_word(1, 0, 0, 1, 0), act_word(1, 0, 1, 0, 0),
    act_word(0, 1, 0, 1, 0), act_word(0, 1, 1, 0, 0), act_word(1, 0, 0, 0, 1), act_word(0, 0, 0, 1, 1),
    act_word(0, 0, 1, 0, 1), act_word(0, 1, 0, 0, 1), act_word(1, 0, 0, 1, 1), act_word(1, 0, 1, 0, 1),
    act_word(0, 1, 0, 1, 1), act_word(0, 1, 1, 0, 1),
};

// ---------------------------------------------------------------- opcode table
// What an opcode does, as eight words.  Emu::run executes most instructions
// from them without a branch: registers, operands, flags and destination are
// selected by byte permutes whose selectors are the words' low halves (so no
// field is extracted for them).  Lanes at different opcodes share its code too.
struct alignas(16) OpWord {
    uint32_t ix;   // over (registers, $80, 0): the index; high half: T_*
    uint32_t rs;   // over (registers, 0): the register operand; high half: cycles without the page-crossing and branch penalties
    uint32_t rd;   // over (registers, result): the new registers; high half: bytes
    uint32_t bs;   // over (operand bytes): the base address; high half: m of Emu::alu
    uint32_t qs;   // over (flags, 1, $FF, 0): what is added; high half: OP_* | T_IND, T_INDY
    uint32_t fs;   // over (flags, result and its flags): the new flags; high half: k of Emu::alu
    uint32_t am;   // address mask, $FF (wraps in zero page) or $FFFF; high half: what the operand is XORed with.  Branches: the flag tested
    uint32_t xs;   // over (memory operand, first operand byte): the operand
};
enum : uint32_t {                                                     // in ix
    T_CTRL = 1u << 16,    // not the straight path: branch, stack or jump; with T_MEM: through a zero-page pointer
    T_MEM = 1u << 17,     // has a memory operand
    T_WR = 1u << 31,      // writes it (stores, read-modify-write); the sign bit: run() clears ROM addresses' with it
    T_FIX = 1u << 20,     // the fix-up read of an indexed access is always made
    T_UV = 1u << 23,      // sets V; decimal mode applies (ADC, SBC)
    T_BR = 1u << 24,      // branch, taken when the flag is clear (T_BI) or set
    T_BI = 1u << 27,
    T_CTL = 1u << 28,     // may leave lanes of a converged group at different pcs
    T_ODD = 1u << 29,     // shifts, BIT, operations on I, D and V
};
enum : uint32_t { T_IND = 0x40u, T_INDY = 0x80u };                    // with the operation: through a zero-page pointer, (zp),Y
enum : uint32_t {
    // on a value read (memory or immediate)
    OP_ORA, OP_AND, OP_EOR, OP_ADC, OP_LDA, OP_CMP, OP_SBC, OP_LDX, OP_LDY, OP_CPX, OP_CPY, OP_BIT,
    // on a value read, written back
    OP_ASL, OP_ROL, OP_LSR, OP_ROR, OP_DEC, OP_INC,
    // stores
    OP_STA, OP_STX, OP_STY,
    // no operand
    OP_CLC, OP_SEC, OP_CLI, OP_SEI, OP_CLV, OP_CLD, OP_SED, OP_TAX, OP_TXA, OP_TAY, OP_TYA, OP_TSX, OP_TXS,
    OP_INX, OP_INY, OP_DEX, OP_DEY, OP_NOP,
    // branches, in opcode order
    OP_BPL, OP_BMI, OP_BVC, OP_BVS, OP_BCC, OP_BCS, OP_BNE, OP_BEQ,
    // stack and control
    OP_PHP, OP_PHA, OP_JSR, OP_BRK, OP_PLP, OP_PLA, OP_RTS, OP_RTI, OP_JMP, OP_JMPI,
    OP_ILL
};
struct OpTable { OpWord e[256]; };
// The 151 legal opcodes of src/cpu.rs:253-1141; the rest are OP_ILL.
constexpr OpTable make_op_table()
{
    OpTable t{};
    constexpr uint32_t A = 0, X = 1, Y = 2, S = 3, N = 4;            // registers; N: none
    constexpr uint32_t QC = 2, Q1 = 4, QF = 5, Q0 = 6;               // what is added: carry, 1, $FF, 0
    constexpr uint32_t ZP = 1, AB = 2, IM = 3, NO = 0;               // operand: zero page, absolute, immediate, none
    for (uint32_t op = 0; op < 256u; op++)
        t.e[op] = OpWord{ 0x5554u | T_CTRL | T_CTL, 0x4444u, 0x3210u | (1u << 16), 0x1111u, 0x6666u | (OP_ILL << 16), 0x3210u,
                          0xFFu, 0x1111u };
    auto set = [&](uint32_t op, uint32_t o, uint32_t mode, uint32_t idx, uint32_t flags, uint32_t ind, uint32_t len,
                   uint32_t cyc) {
        uint32_t src = N, dst = N, q = Q0, b = 0, m = 1, f = 0, kx = 1;
        bool nz = true, c = false, v = false, use = true;            // use: the operand enters the result
        switch (o) {
        case OP_ORA: src = dst = A; break;
        case OP_AND: src = dst = A; kx = 0; break;
        case OP_EOR: src = dst = A; m = 0; break;
        case OP_LDA: dst = A; break;
        case OP_LDX: dst = X; break;
        case OP_LDY: dst = Y; break;
        case OP_ADC: src = dst = A; m = 2; q = QC; c = v = true; f |= T_UV; break;
        case OP_SBC: src = dst = A; m = 2; q = QC; b = 0xFF; c = v = true; f |= T_UV; break;
        case OP_CMP: src = A; m = 2; q = Q1; b = 0xFF; c = true; break;
        case OP_CPX: src = X; m = 2; q = Q1; b = 0xFF; c = true; break;
        case OP_CPY: src = Y; m = 2; q = Q1; b = 0xFF; c = true; break;
        case OP_ASL: case OP_LSR: f |= T_ODD | (mode ? T_WR : 0u); break;
        case OP_ROL: case OP_ROR: q = QC; f |= T_ODD | (mode ? T_WR : 0u); break;
        case OP_INC: q = Q1; f |= T_WR; break;
        case OP_DEC: q = QF; f |= T_WR; break;
        case OP_STA: src = A; f |= T_WR; nz = use = false; break;
        case OP_STX: src = X; f |= T_WR; nz = use = false; break;
        case OP_STY: src = Y; f |= T_WR; nz = use = false; break;
        case OP_CLC: c = true; nz = false; break;
        case OP_SEC: b = 0x100; c = true; nz = false; break;
        case OP_TAX: src = A; dst = X; break;
        case OP_TXA: src = X; dst = A; break;
        case OP_TAY: src = A; dst = Y; break;
        case OP_TYA: src = Y; dst = A; break;
        case OP_TSX: src = S; dst = X; break;
        case OP_TXS: src = X; dst = S; nz = false; break;
        case OP_INX: src = dst = X; q = Q1; break;
        case OP_INY: src = dst = Y; q = Q1; break;
        case OP_DEX: src = dst = X; q = QF; break;
        case OP_DEY: src = dst = Y; q = QF; break;
        case OP_NOP: nz = false; break;
        case OP_BIT: case OP_CLI: case OP_SEI: case OP_CLV: case OP_CLD: case OP_SED: f |= T_ODD; nz = false; break;
        default: f |= T_CTRL; nz = false; break;
        }
        const bool mem = mode == ZP || mode == AB;
        if (mem) f |= T_MEM;
        if (ind) f |= T_CTRL;
        // Without a memory operand the address is $80: RAM, read and not used.
        const uint32_t i = !mem ? 4u : idx == N ? 5u : idx;
        const uint32_t d = dst == N ? 0x3210u : (0x3210u & ~(0xFu << (4u * dst))) | (4u << (4u * dst));
        const uint32_t fl = (nz ? 0x74u : 0x10u) | (c ? 0x500u : 0x200u) | (v ? 0x6000u : 0x3000u);
        t.e[op] = OpWord{ 0x5550u | i | f | flags, 0x4440u | src | (cyc << 16), d | (len << 16),
                          (mode == ZP ? 0x1110u : mode == AB ? 0x1140u : 0x1111u) | (m << 16), 0x6660u | q | ((o | ind) << 16), fl | (kx << 16),
                          (mode == AB ? 0xFFFFu : 0xFFu) | (b << 16),
                          !use ? 0x1111u : mem ? 0x1110u : mode == IM ? 0x1114u : 0x1111u };
    };
    // cc = 01: eight operations, eight modes.
    const uint32_t g1[8] = { OP_ORA, OP_AND, OP_EOR, OP_ADC, OP_STA, OP_LDA, OP_CMP, OP_SBC };
    for (uint32_t k = 0; k < 8u; k++) {
        const uint32_t b = (k << 5) | 1u, o = g1[k];
        const bool st = o == OP_STA;
        const uint32_t fix = st ? T_FIX : 0u, e = st ? 1u : 0u;
        set(b | 0x00u, o, AB, N, 0, T_IND, 2, 6);                                  // (zp,X)
        set(b | 0x04u, o, ZP, N, 0, 0, 2, 3);                                      // zp
        if (!st) set(b | 0x08u, o, IM, N, 0, 0, 2, 2);                             // #imm
        set(b | 0x0Cu, o, AB, N, 0, 0, 3, 4);                                      // abs
        set(b | 0x10u, o, AB, Y, fix, T_IND | T_INDY, 2, 5 + e);                   // (zp),Y
        set(b | 0x14u, o, ZP, X, 0, 0, 2, 4);                                      // zp,X
        set(b | 0x18u, o, AB, Y, fix, 0, 3, 4 + e);                                // abs,Y
        set(b | 0x1Cu, o, AB, X, fix, 0, 3, 4 + e);                                // abs,X
    }
    // cc = 10: shifts, INC, DEC; LDX, STX.
    const uint32_t g2[8] = { OP_ASL, OP_ROL, OP_LSR, OP_ROR, OP_STX, OP_LDX, OP_DEC, OP_INC };
    for (uint32_t k = 0; k < 8u; k++) {
        const uint32_t b = (k << 5) | 2u, o = g2[k];
        if (o == OP_STX || o == OP_LDX) {
            set(b | 0x04u, o, ZP, N, 0, 0, 2, 3);
            set(b | 0x0Cu, o, AB, N, 0, 0, 3, 4);
            set(b | 0x14u, o, ZP, Y, 0, 0, 2, 4);
            if (o == OP_LDX) {
                set(b | 0x00u, o, IM, N, 0, 0, 2, 2);
                set(b | 0x1Cu, o, AB, Y, 0, 0, 3, 4);
            }
            continue;
        }
        set(b | 0x04u, o, ZP, N, 0, 0, 2, 5);
        set(b | 0x0Cu, o, AB, N, 0, 0, 3, 6);
        set(b | 0x14u, o, ZP, X, 0, 0, 2, 6);
        set(b | 0x1Cu, o, AB, X, T_FIX, 0, 3, 7);
        if (k < 4u) set(b | 0x08u, o, NO, N, 0, 0, 1, 2);                          // of A
    }
    // cc = 00: BIT, STY, LDY, CPY, CPX.
    set(0x24, OP_BIT, ZP, N, 0, 0, 2, 3); set(0x2C, OP_BIT, AB, N, 0, 0, 3, 4);
    set(0x84, OP_STY, ZP, N, 0, 0, 2, 3); set(0x8C, OP_STY, AB, N, 0, 0, 3, 4); set(0x94, OP_STY, ZP, X, 0, 0, 2, 4);
    set(0xA0, OP_LDY, IM, N, 0, 0, 2, 2); set(0xA4, OP_LDY, ZP, N, 0, 0, 2, 3); set(0xAC, OP_LDY, AB, N, 0, 0, 3, 4);
    set(0xB4, OP_LDY, ZP, X, 0, 0, 2, 4); set(0xBC, OP_LDY, AB, X, 0, 0, 3, 4);
    set(0xC0, OP_CPY, IM, N, 0, 0, 2, 2); set(0xC4, OP_CPY, ZP, N, 0, 0, 2, 3); set(0xCC, OP_CPY, AB, N, 0, 0, 3, 4);
    set(0xE0, OP_CPX, IM, N, 0, 0, 2, 2); set(0xE4, OP_CPX, ZP, N, 0, 0, 2, 3); set(0xEC, OP_CPX, AB, N, 0, 0, 3, 4);
    // Implied.
    const uint32_t imp[18][2] = { { 0x18, OP_CLC }, { 0x38, OP_SEC }, { 0x58, OP_CLI }, { 0x78, OP_SEI }, { 0xB8, OP_CLV },
                                  { 0xD8, OP_CLD }, { 0xF8, OP_SED }, { 0xAA, OP_TAX }, { 0x8A, OP_TXA }, { 0xA8, OP_TAY },
                                  { 0x98, OP_TYA }, { 0xBA, OP_TSX }, { 0x9A, OP_TXS }, { 0xE8, OP_INX }, { 0xC8, OP_INY },
                                  { 0xCA, OP_DEX }, { 0x88, OP_DEY }, { 0xEA, OP_NOP } };
    for (uint32_t k = 0; k < 18u; k++) set(imp[k][0], imp[k][1], NO, N, 0, 0, 1, 2);
    // Branches by opcode bits 6-7 (N, V, C, Z) and 5 (clear, set); F holds Z as a byte that is 0 when Z is set.
    for (uint32_t k = 0; k < 8u; k++) {
        const uint32_t fl = k >> 1, on = k & 1u;
        set(0x10u | (k << 5), OP_BPL + k, NO, N, T_CTL | T_BR | (((fl == 3u) ? on : !on) ? T_BI : 0u), 0, 2, 2);
        t.e[0x10u | (k << 5)].am = fl == 0u ? 0x8080u : fl == 1u ? 0x80000000u : fl == 2u ? 0x10000u : 0xFFu;
    }
    // Stack, control.
    set(0x08, OP_PHP, NO, N, 0, 0, 1, 3); set(0x48, OP_PHA, NO, N, 0, 0, 1, 3); set(0x28, OP_PLP, NO, N, 0, 0, 1, 4);
    set(0x68, OP_PLA, NO, N, 0, 0, 1, 4); set(0x20, OP_JSR, NO, N, 0, 0, 2, 6); set(0x00, OP_BRK, NO, N, T_CTL, 0, 2, 7);
    set(0x60, OP_RTS, NO, N, T_CTL, 0, 1, 6); set(0x40, OP_RTI, NO, N, T_CTL, 0, 1, 6); set(0x4C, OP_JMP, NO, N, 0, 0, 3, 3);
    set(0x6C, OP_JMPI, NO, N, T_CTL, 0, 3, 5);
    return t;
}

// Headless TIA registers whose write only stores bits of the value
// (headless_tia.rs:225-298): private byte | shift << 8 | mask << 16; 0 for
// the others.
struct TiaTable { uint32_t w[64]; };
constexpr TiaTable make_tia_table()
{
    TiaTable t{};
    for (uint32_t r = 0; r < 64u; r++) t.w[r] = 0;
    auto set = [&](uint32_t r, uint32_t o, uint32_t sh, uint32_t m) { t.w[r] = o | (sh << 8) | (m << 16); };
    set(0x04, 164, 0, 0xFF); set(0x05, 165, 0, 0xFF);                 // NUSIZ
    for (uint32_t k = 0; k < 4u; k++) set(0x06u + k, 166u + k, 0, 0xFF);   // COLUx
    set(0x0A, 170, 0, 0xFF);                                          // CTRLPF
    set(0x0B, 171, 3, 1); set(0x0C, 172, 3, 1);                       // REFP
    for (uint32_t k = 0; k < 3u; k++) set(0x0Du + k, 173u + k, 0, 0xFF);   // PF
    for (uint32_t k = 0; k < 3u; k++) set(0x1Du + k, 155u + k, 1, 1);      // ENAM0 ENAM1 ENABL
    for (uint32_t k = 0; k < 5u; k++) set(0x20u + k, 146u + k, 0, 0xFF);   // HM
    for (uint32_t k = 0; k < 3u; k++) set(0x25u + k, 159u + k, 0, 1);      // VDEL
    set(0x28, 162, 1, 1); set(0x29, 163, 1, 1);                       // RESMP
    return t;
}

// v in a register of its own: not loaded or computed again from the launch's
// constants wherever it is used, which ptxas otherwise prefers to keeping it
// (4 constant loads and 12 more instructions per guest instruction).
template <class T>
__device__ __forceinline__ T kept(T v)
{
#ifdef __CUDA_ARCH__
    asm volatile("" : "+r"(v));
#endif
    return v;
}

// Bytes of shared memory by their 32-bit address there.  Pointers would do,
// but the interpreter's loop selects between two of them and keeps several:
// as generic pointers they cost 64-bit arithmetic.
#ifdef __CUDA_ARCH__
typedef uint32_t sptr;
__device__ __forceinline__ sptr to_sptr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t lds8(sptr p)
{
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ void sts8(sptr p, uint32_t v)
{
    asm volatile("st.shared.u8 [%0], %1;" ::"r"(p), "r"(v) : "memory");
}
#else
typedef uint8_t* sptr;
__device__ __forceinline__ sptr to_sptr(const void* p) { return (uint8_t*)p; }
__device__ __forceinline__ uint32_t lds8(const uint8_t* p) { return *p; }
__device__ __forceinline__ void sts8(uint8_t* p, uint32_t v) { *p = (uint8_t)v; }
#endif

// The kernels copy the table into shared memory (load_op_table): a constant
// load costs one pass per distinct index of the warp, a shared load does not.
#ifdef __CUDACC__
static __device__ const OpTable g_op = make_op_table();
static __device__ const TiaTable g_tia = make_tia_table();
__device__ __forceinline__ OpWord* op_table()
{
    __shared__ OpWord t[256];
    return t;
}
__device__ __forceinline__ uint32_t* tia_table()
{
    __shared__ uint32_t t[64];
    return t;
}
// Called by every thread of the CTA; a barrier must follow before the first
// instruction.
__device__ __forceinline__ void load_op_table()
{
    uint4* d = (uint4*)op_table();
    const uint4* s = (const uint4*)g_op.e;
    for (uint32_t k = threadIdx.x; k < 512u; k += blockDim.x) d[k] = s[k];
    for (uint32_t k = threadIdx.x; k < 64u; k += blockDim.x) tia_table()[k] = g_tia.w[k];
}
#else
inline const OpWord* op_table()
{
    static const OpTable t = make_op_table();
    return t.e;
}
inline const uint32_t* tia_table()
{
    static const TiaTable t = make_tia_table();
    return t.w;
}
#endif
// The high half of a table word w: loaded again rather than shifted out (the
// headless loop is bound by the ALU pipe, of which a shift is an instruction:
// 50 and 45 of them a guest instruction, the mixed batch 14.1 and 13.8 ms);
// the rendering loop is not, and shifts (load false).
enum : uint32_t { H_CYC = 6u, H_LEN = 10u, H_M = 14u, H_K = 22u, H_X = 26u };
template <bool LOAD>
__device__ __forceinline__ uint32_t high(sptr tab, uint32_t op, uint32_t h, uint32_t w)
{
    if constexpr (!LOAD) return w >> 16;
#ifdef __CUDA_ARCH__
    uint32_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(tab + op * 32u + h));
    return v;
#else
    return ((const uint32_t*)((const OpWord*)tab + op))[h / 4u] >> 16;
#endif
}
__device__ __forceinline__ OpWord ldw(sptr tab, uint32_t op)
{
#ifdef __CUDA_ARCH__
    OpWord w;
    const uint32_t a = tab + op * 32u;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w.ix), "=r"(w.rs), "=r"(w.rd), "=r"(w.bs) : "r"(a));
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4 + 16];" : "=r"(w.qs), "=r"(w.fs), "=r"(w.am), "=r"(w.xs) : "r"(a));
    return w;
#else
    return ((const OpWord*)tab)[op];
#endif
}

// Packed TIA flag word (Emu::tw).
enum : uint32_t { TW_WSYNC = 1u << 16, TW_FCOMP = 1u << 17, TW_PDUMP = 1u << 18,
                  TW_CX = 1u << 23,      // headless only: a collision latch may be set (only an upload sets them)
                  // rendering console only
                  TW_HMOVE = 1u << 19, TW_LATCH = 1u << 20, TW_L4 = 1u << 21, TW_L5 = 1u << 22 };

// NUSIZ copy offsets as a mask over {0, 16, 32, 64} (tia.rs:440-450, 480-488).
static __constant__ uint32_t c_copies[8] = { 0x1, 0x3, 0x5, 0x7, 0x9, 0x1, 0xD, 0x1 };


template <int BLOCK>
__device__ __forceinline__ uint32_t priv_off(uint32_t o) { return (o & ~3u) * BLOCK + (o & 3u); }

__device__ __forceinline__ uint32_t mod160(int v)
{
    int r = v % 160;
    return (uint32_t)(r < 0 ? r + 160 : r);
}

// Byte o (>= 128) of an instance's private bytes, in its HBM state rows:
// `col` is the instance's column base, stride4 the row stride in bytes.
__device__ __forceinline__ uint32_t cold_off(uint32_t o, uint32_t stride4) { return (o >> 2) * stride4 + (o & 3u); }

// TIA or PIA register read (HeadlessTia::read, src/headless_tia.rs:205-223;
// Pia::read I/O half, src/pia.rs:169-199), INTIM apart (pia_intim_io):
// sel_uf carries the timer's underflow flag in bits 16 and up.
static __device__ __forceinline__ uint32_t io_read(uint32_t a, uint32_t pcnt, uint32_t pins, uint32_t pads,
                                         uint32_t ports, uint32_t sel_uf, const uint8_t* col, uint32_t stride4)
{
    if (a & 0x80u) {                                                 // PIA: (a & 0x280) == 0x280
        switch (a & 7u) {
        case 0: return ((pins & ~(ports >> 8)) | (ports & (ports >> 8))) & 0xFFu;
        case 1: return (ports >> 8) & 0xFFu;
        case 2: return (((pins >> 8) & ~(ports >> 24)) | ((ports >> 16) & (ports >> 24))) & 0xFFu;
        case 3: return ports >> 24;
        case 5: return (sel_uf >> 16) ? 0x80u : 0u;
        default: return 0u;
        }
    }
    const uint32_t r = a & 0x0Fu;
    if (r < 8u) return col[cold_off(PB_CX + r, stride4)];
    switch (r) {
    case 0x8: return pcnt >= (pads & 0xFFu) ? 0x80u : 0u;
    case 0x9: return pcnt >= (pads >> 8) ? 0x80u : 0u;
    case 0xA: case 0xB: return 0x80u;
    case 0xC: return (pins >> 16) & 1u ? 0x80u : 0u;
    case 0xD: return (pins >> 17) & 1u ? 0x80u : 0u;
    default: return 0u;
    }
}

// HeadlessTia::write (src/headless_tia.rs:225-298).  tw is the packed flag
// word, lw = scanline | paddle_counter<<16; both come back updated.  The
// write-only registers live in the instance's HBM rows (col, stride4).
static __device__ __forceinline__ uint2 tia_write_io(uint32_t a, uint32_t v, uint32_t clock, uint32_t tw, uint32_t lw,
                                           uint8_t* col, uint32_t stride4)
{
    auto stp = [&](uint32_t o, uint32_t val) { col[cold_off(o, stride4)] = (uint8_t)val; };
    auto ldp = [&](uint32_t o) -> uint32_t { return col[cold_off(o, stride4)]; };
    auto stp16 = [&](uint32_t o, uint32_t val) { *(uint16_t*)(col + cold_off(o, stride4)) = (uint16_t)val; };
    auto ldp16 = [&](uint32_t o) -> uint32_t { return *(const uint16_t*)(col + cold_off(o, stride4)); };
    const uint32_t r = a & 0x3Fu;
    switch (r) {
    case 0x00:                                                        // VSYNC rising edge starts a frame
        if (!(tw & 2u) && (v & 2u)) { lw &= 0xFFFF0000u; tw |= TW_FCOMP; }
        tw = (tw & ~0xFFu) | v;
        break;
    case 0x01:                                                        // VBLANK bit 7 dumps the paddles
        if (v & 0x80u) { lw &= 0xFFFFu; tw |= TW_PDUMP; } else tw &= ~TW_PDUMP;
        tw = (tw & ~0xFF00u) | (v << 8);
        break;
    case 0x02: tw |= TW_WSYNC; break;
    case 0x04: stp(PB_NUSIZ0, v); break;
    case 0x05: stp(PB_NUSIZ1, v); break;
    case 0x06: case 0x07: case 0x08: case 0x09: stp(PB_COLUP0 + (r - 0x06u), v); break;
    case 0x0A: stp(PB_CTRLPF, v); break;
    case 0x0B: stp(PB_REFP0, (v >> 3) & 1u); break;
    case 0x0C: stp(PB_REFP1, (v >> 3) & 1u); break;
    case 0x0D: case 0x0E: case 0x0F: stp(PB_PF0 + (r - 0x0Du), v); break;
    case 0x10: case 0x11: case 0x12: case 0x13: case 0x14:
        // RESPx: (clock as i16 - 68 + 5).rem_euclid(160)
        stp16(PB_POS + 2u * (r - 0x10u), mod160((int16_t)(uint16_t)(clock - 63u)));
        break;
    case 0x1B: stp(PB_GRP0_OLD, ldp(PB_GRP0)); stp(PB_GRP0, v); break;
    case 0x1C:
        stp(PB_GRP1_OLD, ldp(PB_GRP1)); stp(PB_GRP1, v);
        stp(PB_ENABL_OLD, ldp(PB_ENABL)); break;
    case 0x1D: case 0x1E: case 0x1F: stp(PB_ENAM0 + (r - 0x1Du), (v >> 1) & 1u); break;
    case 0x20: case 0x21: case 0x22: case 0x23: case 0x24: stp(PB_HM + (r - 0x20u), v); break;
    case 0x25: case 0x26: case 0x27: stp(PB_VDELP0 + (r - 0x25u), v & 1u); break;
    case 0x28: case 0x29: stp(PB_RESMP0 + (r - 0x28u), (v >> 1) & 1u); break;
    case 0x2A:                                                        // HMOVE
        for (uint32_t k = 0; k < 5u; k++) {
            int off = ((int)(int8_t)(uint8_t)ldp(PB_HM + k)) >> 4;
            int16_t d = (int16_t)(uint16_t)(ldp16(PB_POS + 2u * k) - (uint32_t)off);
            stp16(PB_POS + 2u * k, mod160(d));
        }
        break;
    case 0x2B: for (uint32_t k = 0; k < 5u; k++) stp(PB_HM + k, 0); break;
    case 0x2C: for (uint32_t k = 0; k < 8u; k++) stp(PB_CX + k, 0); break;
    default: break;
    }
    return make_uint2(tw, lw);
}

// Pia::write, I/O half (src/pia.rs:202-228).  Returns (ports, timer value,
// prescaler, select | underflow<<16).
static __device__ __noinline__ uint4 pia_write_io(uint32_t a, uint32_t v, uint32_t ports, uint32_t tv, uint32_t ps,
                                           uint32_t sel_uf)
{
    if (a & 0x10u) {
        const uint32_t sel = 1u << ((0xA630u >> (4u * (a & 3u))) & 0xFu);   // 1, 8, 64, 1024
        return make_uint4(ports, v, sel, sel);
    }
    const uint32_t sh = 8u * (a & 3u);                                 // pa_out pa_ddr pb_out pb_ddr
    return make_uint4((ports & ~(0xFFu << sh)) | (v << sh), tv, ps, sel_uf);
}

// ---------------------------------------------------------------- rendering console
// The pixel-accurate Tia (src/tia.rs) and the per-cycle Pia::tick
// (src/pia.rs:80-103) of the reference's rendering console, as out-of-line
// functions on the state they touch.  The registers of the TIA are the
// console's private bytes in shared memory (PB_* graphics registers, RB_*
// extras), interleaved by lane in 32-lane slabs; the framebuffer is HBM.
struct RState {
    uint32_t clock, scanline, tw, pcnt, vtop;   // beam, TIA flags, paddle counter, visible_top | vblank_top << 16
    uint32_t rx;                                // the current line's pixels are drawn up to this clock
    uint32_t sc;                                // the framebuffer sector (32 pixels) whose pixels the sector buffer holds
    uint32_t zr;                                // rows written since the clear point | R_ZPEND (rows after them not yet zeroed)
};
constexpr uint32_t R_ZPEND = 0x100u;

static __device__ __forceinline__ uint32_t rp8(const uint8_t* pv, uint32_t o) { return pv[(o & ~3u) * 32u + (o & 3u)]; }
static __device__ __forceinline__ void wp8(uint8_t* pv, uint32_t o, uint32_t v) { pv[(o & ~3u) * 32u + (o & 3u)] = (uint8_t)v; }
static __device__ __forceinline__ uint32_t rp16(const uint8_t* pv, uint32_t o) { return *(const uint16_t*)(pv + (o & ~3u) * 32u + (o & 3u)); }
static __device__ __forceinline__ void wp16(uint8_t* pv, uint32_t o, uint32_t v) { *(uint16_t*)(pv + (o & ~3u) * 32u + (o & 3u)) = (uint16_t)v; }

// ---- framebuffer writes through a one-sector buffer
// Pixels of a line are drawn left to right, so a console stages the 32
// pixels of the framebuffer sector it is drawing (8 words after its private
// bytes in its shared-memory slab) and writes each sector whole, with two
// 16-byte stores, when the drawing moves past it: every sector of a visible
// row is written once, with zeros where nothing was drawn.  The reference
// clears the framebuffer where the visible area starts (tia.rs:349-351);
// here the rows are written as the beam completes them, and the rows the
// frame has not reached are zeroed when the framebuffer can next be seen
// (VSYNC, the end of a frame, the end of a call).
static __device__ __forceinline__ uint32_t* r_sbuf(uint8_t* pv, uint32_t k)
{
    return (uint32_t*)(pv + (FA_RPRIV_BYTES + 4u * k) * 32u);
}
static __device__ __forceinline__ void r_sec_write(uint8_t* pv, uint8_t* fbp, uint32_t sc)
{
    uint4* d = (uint4*)(fbp + (size_t)sc * 32u);
    d[0] = make_uint4(*r_sbuf(pv, 0), *r_sbuf(pv, 1), *r_sbuf(pv, 2), *r_sbuf(pv, 3));
    d[1] = make_uint4(*r_sbuf(pv, 4), *r_sbuf(pv, 5), *r_sbuf(pv, 6), *r_sbuf(pv, 7));
}
static __device__ __forceinline__ void r_sec_clear(uint8_t* pv)
{
#pragma unroll
    for (uint32_t k = 0; k < 8u; k++) *r_sbuf(pv, k) = 0u;
}
static __device__ __forceinline__ void r_zero_sectors(uint8_t* fbp, uint32_t from, uint32_t to)   // [from, to)
{
    uint4* d = (uint4*)fbp;
    for (uint32_t q = 2u * from; q < 2u * to; q++) d[q] = make_uint4(0u, 0u, 0u, 0u);
}
// The buffer moves on to sector t: the sector it held is written, the ones
// skipped between become zeros.
static __device__ void r_seek(uint32_t& sc, uint8_t* pv, uint8_t* fbp, uint32_t t)
{
    r_sec_write(pv, fbp, sc);
    if (t > sc) {
        r_zero_sectors(fbp, sc + 1u, t);
        r_sec_clear(pv);
    } else {                                                         // not reached by drawing order; kept exact
        const uint4* q = (const uint4*)(fbp + (size_t)t * 32u);
        const uint4 u0 = q[0], u1 = q[1];
        *r_sbuf(pv, 0) = u0.x; *r_sbuf(pv, 1) = u0.y; *r_sbuf(pv, 2) = u0.z; *r_sbuf(pv, 3) = u0.w;
        *r_sbuf(pv, 4) = u1.x; *r_sbuf(pv, 5) = u1.y; *r_sbuf(pv, 6) = u1.z; *r_sbuf(pv, 7) = u1.w;
    }
    sc = t;
}

// Bits 0..7 of b, each repeated over two bits.
static __device__ __forceinline__ uint32_t r_spread2(uint32_t b)
{
    uint32_t t = (b | (b << 4)) & 0x0F0Fu;
    t = (t | (t << 2)) & 0x3333u;
    t = (t | (t << 1)) & 0x5555u;
    return t * 3u;
}

// Bits 0..7 of b, each repeated over four bits.
static __device__ __forceinline__ uint32_t r_spread4(uint32_t b)
{
    uint32_t t = (b & 0x0Fu) | ((b & 0xF0u) << 12);
    t = (t | (t << 6)) & 0x03030303u;
    t = (t | (t << 3)) & 0x11111111u;
    return t * 0xFu;
}

// Bits 0..3 of n moved to bits 0, 4, 8, 12.
static __device__ __forceinline__ uint32_t r_nib(uint32_t n)
{
    const uint32_t t = (n | (n << 6)) & 0x303u;
    return (t | (t << 3)) & 0x1111u;
}

// Bits 0..3 of n as byte masks.
static __device__ __forceinline__ uint32_t r_bytes(uint32_t n)
{
    return (((n & 0xFu) * 0x00204081u) & 0x01010101u) * 0xFFu;
}

// Pixels [X, X + 32) of the 160-pixel line covered by an object of len <= 32
// pixels starting at pixel s < 160, whose graphics g hold pixel d from its
// left edge in bit d: bit i = pixel X + i.  An object wraps from pixel 159
// to pixel 0, as the position arithmetic of tia.rs:406-507 does mod 160.
static __device__ __forceinline__ uint32_t r_place(uint32_t g, uint32_t len, uint32_t s, uint32_t X)
{
    const uint32_t i0 = s >= X ? s - X : s + 160u - X;
    if (i0 < 32u) return g << i0;
    const uint32_t d0 = 160u - i0;
    return d0 < len ? g >> d0 : 0u;
}

static __device__ __forceinline__ uint32_t r_copies(uint32_t g, uint32_t len, uint32_t pos, uint32_t copies, uint32_t X)
{
    uint32_t m = r_place(g, len, pos, X);
#pragma unroll
    for (uint32_t c = 1; c < 4u; c++)
        if ((copies >> c) & 1u) {
            uint32_t st = pos + (8u << c);                            // copies at +16, +32, +64
            if (st >= 160u) st -= 160u;
            m |= r_place(g, len, st, X);
        }
    return m;
}

// Player n over pixels [X, X + 32) (tia.rs:423-465): NUSIZ copies and
// widths, REFP reflection, VDELP's old graphics.
static __device__ __forceinline__ uint32_t r_player_mask(const uint8_t* pv, uint32_t n, uint32_t X)
{
    const uint32_t grp = rp8(pv, n ? (rp8(pv, PB_VDELP1) ? PB_GRP1_OLD : PB_GRP1) : (rp8(pv, PB_VDELP0) ? PB_GRP0_OLD : PB_GRP0));
    if (grp == 0) return 0;
    const uint32_t mode = rp8(pv, n ? PB_NUSIZ1 : PB_NUSIZ0) & 7u;
    const uint32_t g8 = rp8(pv, n ? PB_REFP1 : PB_REFP0) ? grp : __brev(grp) >> 24;
    const uint32_t g = mode == 5u ? r_spread2(g8) : mode == 7u ? r_spread4(g8) : g8;
    const uint32_t len = mode == 5u ? 16u : mode == 7u ? 32u : 8u;
    return r_copies(g, len, rp16(pv, PB_POS + 2u * n), c_copies[mode], X);
}

// Missile n over pixels [X, X + 32) (tia.rs:468-497).
static __device__ __forceinline__ uint32_t r_missile_mask(const uint8_t* pv, uint32_t n, uint32_t X)
{
    if (!rp8(pv, n ? PB_ENAM1 : PB_ENAM0) || rp8(pv, n ? PB_RESMP1 : PB_RESMP0)) return 0;
    const uint32_t nusiz = rp8(pv, n ? PB_NUSIZ1 : PB_NUSIZ0);
    const uint32_t len = 1u << ((nusiz >> 4) & 3u);
    return r_copies((1u << len) - 1u, len, rp16(pv, PB_POS + 4u + 2u * n), c_copies[nusiz & 7u], X);
}

// Pixels [x0, x1) of visible line `vis` with the TIA registers as they are:
// Tia::tick's pixel stage (tia.rs:311-346) with compute_pixel (tia.rs:375-403)
// and the object tests (tia.rs:406-507), over a span in which no register
// changes.  Each object is a bit mask over 32 pixels at a time; the
// collision latches are the masks' intersections, and the priority of
// compute_pixel is the order in which the colors are laid down.  Each
// 32-pixel chunk is one framebuffer sector: its pixels go into the sector
// buffer four to a word, and the buffer is written out when the drawing
// moves to another sector (r_seek).
static __device__ __noinline__ RState r_span(RState s, uint8_t* pv, uint8_t* fbp, uint32_t vis, uint32_t x0, uint32_t x1)
{
    const uint32_t ctrlpf = rp8(pv, PB_CTRLPF);
    const uint32_t pfw = (rp8(pv, PB_PF0) >> 4) | (__brev(rp8(pv, PB_PF1)) >> 24 << 4) | (rp8(pv, PB_PF2) << 12);
    const uint32_t pfr = (ctrlpf & 1u) ? __brev(pfw) >> 12 : pfw;    // the right half, reflected or repeated
    const uint64_t line = (uint64_t)pfw | ((uint64_t)pfr << 20);     // bit g = playfield pixels 4g..4g+3
    const bool ben = rp8(pv, rp8(pv, PB_VDELBL) ? PB_ENABL_OLD : PB_ENABL) != 0;
    const uint32_t blen = 1u << ((ctrlpf >> 4) & 3u);
    uint32_t cx = 0;                                                 // bit 2r: 0x80 of CXr, bit 2r+1: 0x40
    for (uint32_t X = x0 & ~31u; X < x1; X += 32u) {
        const uint32_t lo = x0 > X ? x0 - X : 0u, hi = x1 < X + 32u ? x1 - X : 32u;
        const uint32_t in = (hi >= 32u ? 0xFFFFFFFFu : (1u << hi) - 1u) & ~((1u << lo) - 1u);
        const uint32_t pf = r_spread4((uint32_t)(line >> (X >> 2)) & 0xFFu) & in;
        const uint32_t p0 = r_player_mask(pv, 0, X) & in, p1 = r_player_mask(pv, 1, X) & in;
        const uint32_t m0 = r_missile_mask(pv, 0, X) & in, m1 = r_missile_mask(pv, 1, X) & in;
        const uint32_t bl = ben ? r_place((1u << blen) - 1u, blen, rp16(pv, PB_POS + 8u), X) & in : 0u;
        cx |= ((m0 & p1) ? 0x1u : 0u) | ((m0 & p0) ? 0x2u : 0u) | ((m1 & p0) ? 0x4u : 0u) | ((m1 & p1) ? 0x8u : 0u)
            | ((p0 & pf) ? 0x10u : 0u) | ((p0 & bl) ? 0x20u : 0u) | ((p1 & pf) ? 0x40u : 0u) | ((p1 & bl) ? 0x80u : 0u)
            | ((m0 & pf) ? 0x100u : 0u) | ((m0 & bl) ? 0x200u : 0u) | ((m1 & pf) ? 0x400u : 0u) | ((m1 & bl) ? 0x800u : 0u)
            | ((bl & pf) ? 0x1000u : 0u) | ((p0 & p1) ? 0x4000u : 0u) | ((m0 & m1) ? 0x8000u : 0u);
        uint32_t A = p0 | m0, B = p1 | m1, F = pf | bl;
        if ((s.tw & TW_HMOVE) && X == 0u) { A &= ~0xFFu; B &= ~0xFFu; F &= ~0xFFu; }   // HMOVE comb: background
        // compute_pixel's choice as a 2-bit index per pixel, for all 32 at once:
        // 0 background, 1 playfield/ball, 2 player 1, 3 player 0.
        const uint32_t I1 = (ctrlpf & 4u) ? (A | B) & ~F : A | B;    // playfield priority: F wins
        const uint32_t I0 = (ctrlpf & 4u) ? F | A : A | (F & ~B);
        const uint32_t c0 = rp8(pv, PB_COLUP0), c1 = rp8(pv, PB_COLUP1), cbk = rp8(pv, PB_COLUBK);
        const uint32_t cpf = rp8(pv, PB_COLUPF);
        const uint32_t tl = cbk | (((ctrlpf & 2u) ? c0 : cpf) << 8) | (c1 << 16) | (c0 << 24);   // x < 80 (score mode)
        const uint32_t tr = cbk | (((ctrlpf & 2u) ? c1 : cpf) << 8) | (c1 << 16) | (c0 << 24);
        const uint32_t t = vis * (FA_FB_W / 32u) + (X >> 5);            // the chunk is one framebuffer sector
        if (t != s.sc) r_seek(s.sc, pv, fbp, t);
        for (uint32_t q = lo >> 2; q < (hi + 3u) >> 2; q++) {
            const uint32_t x = X + 4u * q;
            // Four pixels' indices as a byte-permute selector, one nibble each.
            const uint32_t sel = r_nib((I0 >> (4u * q)) & 0xFu) | (r_nib((I1 >> (4u * q)) & 0xFu) << 1);
            const uint32_t w = __byte_perm(x < 80u ? tl : tr, 0u, sel);
            const uint32_t wl = lo > 4u * q ? lo - 4u * q : 0u, wh = hi < 4u * q + 4u ? hi - 4u * q : 4u;
            const uint32_t pm = ((1u << wh) - 1u) & ~((1u << wl) - 1u);
            uint32_t* bp = r_sbuf(pv, q);
            if (pm == 0xFu) {
                *bp = w;
            } else {
                const uint32_t bm = r_bytes(pm);
                *bp = (*bp & ~bm) | (w & bm);
            }
        }
    }
    if (cx) {                                                        // collision latches (tia.rs:329-343)
#pragma unroll
        for (uint32_t r = 0; r < 8u; r++) {
            const uint32_t b = (((cx >> (2u * r)) & 1u) ? 0x80u : 0u) | (((cx >> (2u * r + 1u)) & 1u) ? 0x40u : 0u);
            if (b) wp8(pv, PB_CX + r, rp8(pv, PB_CX + r) | b);
        }
    }
    return s;
}

// The pixels of the current line from clock s.rx up to clock `upto`, with
// the registers as they are: pixels are drawn only when something that
// affects them is about to change (a register write, a delayed playfield
// write, a collision read, the end of the line or of the call).
static __device__ __forceinline__ void r_pending(RState& s, uint8_t* pv, uint8_t* fbp, uint32_t upto)
{
    const uint32_t from = s.rx > 68u ? s.rx : 68u;
    s.rx = upto;
    if (upto <= from || (s.tw & 0x200u)) return;
    const uint32_t vis = (s.scanline - (s.vtop & 0xFFFFu)) & 0xFFFFu;
    if (vis < FA_FB_H) s = r_span(s, pv, fbp, vis, from - 68u, upto - 68u);
}

// The framebuffer as the reference would show it now (the pixels up to the
// beam are already drawn): the beam's row as far as drawn, with zeros after,
// and, once after each clear point, zeros in the rows the beam has not reached.
static __device__ __forceinline__ void r_observe(RState& s, uint8_t* pv, uint8_t* fbp)
{
    const uint32_t vis = (s.scanline - (s.vtop & 0xFFFFu)) & 0xFFFFu;
    constexpr uint32_t SPR = FA_FB_W / 32u, NSEC = FA_FB_H * SPR;   // sectors per row, in all
    if (vis < FA_FB_H) {
        r_sec_write(pv, fbp, s.sc);
        r_zero_sectors(fbp, s.sc + 1u, (vis + 1u) * SPR);
        if (s.zr & R_ZPEND) r_zero_sectors(fbp, (vis + 1u) * SPR, NSEC);
    } else if (s.zr & R_ZPEND) {
        r_zero_sectors(fbp, (s.zr & 0xFFu) * SPR, NSEC);
    }
    s.zr &= ~R_ZPEND;
}

// n TIA clocks, exactly as n calls of Tia::tick (tia.rs:271-372), advanced a
// line at a time: between register writes nothing but the pixels, the
// collision latches and the beam changes from one clock to the next (the
// input latches are idempotent, the resizer's candidate is the scanline
// itself, and a delayed playfield write fires on the first clock after it).
static __device__ __forceinline__ void r_advance(RState& s, uint32_t n, uint32_t pins, uint8_t* pv, uint8_t* fbp)
{
    if (n == 0) return;
    const uint32_t dlen = rp8(pv, RB_DLEN);
    if (dlen) {                                                      // every pending write has one clock left
        r_pending(s, pv, fbp, s.clock);
        for (uint32_t i = 0; i < dlen; i++) {
            const uint32_t reg = rp8(pv, RB_DQ + 3u * i + 1u), val = rp8(pv, RB_DQ + 3u * i + 2u);
            wp8(pv, reg == 0x0Du ? PB_PF0 : reg == 0x0Eu ? PB_PF1 : PB_PF2, val);
        }
        wp8(pv, RB_DLEN, 0u);
    }
    if (s.tw & TW_LATCH) {
        if (!(pins & 0x10000u)) s.tw &= ~TW_L4;
        if (!(pins & 0x20000u)) s.tw &= ~TW_L5;
    }
    while (n) {
        if (!(s.tw & 0x200u) && s.scanline >= 23u && s.scanline < (s.vtop >> 16))
            s.vtop = (s.vtop & 0xFFFFu) | (s.scanline << 16);
        const uint32_t seg = n < 228u - s.clock ? n : 228u - s.clock;
        s.clock += seg;
        n -= seg;
        if (s.clock >= 228u) {
            r_pending(s, pv, fbp, 228u);
            const uint32_t vis = (s.scanline - (s.vtop & 0xFFFFu)) & 0xFFFFu;
            if (vis < FA_FB_H) {                                     // the row is complete: written whole
                r_seek(s.sc, pv, fbp, (vis + 1u) * (FA_FB_W / 32u));
                s.zr = (s.zr & R_ZPEND) | (vis + 1u);
            }
            s.clock = 0;
            s.rx = 0;
            s.scanline = (s.scanline + 1u) & 0xFFFFu;
            s.tw &= ~(TW_WSYNC | TW_HMOVE);
            if (s.scanline == (s.vtop & 0xFFFFu)) {                  // framebuffer cleared (tia.rs:349-351)
                s.sc = 0;
                r_sec_clear(pv);
                s.zr = R_ZPEND;
            }
            if (!(s.tw & TW_PDUMP) && s.pcnt < 256u) s.pcnt++;
            if (s.scanline >= 262u) { s.scanline = 0; s.tw |= TW_FCOMP; }
        }
    }
}

// The pending pixels of the current line, up to the beam, then the
// framebuffer as it can be seen now.
static __device__ __noinline__ RState render_observe(RState s, uint8_t* pv, uint8_t* fbp)
{
    r_pending(s, pv, fbp, s.clock);
    r_observe(s, pv, fbp);
    return s;
}

// The PIA timer of the rendering console: value | prescaler << 16, interval |
// underflow << 16.
static __device__ __forceinline__ void r_pia_tick(uint32_t& tv, uint32_t& ps, uint32_t sel, uint32_t& uf)     // pia.rs:80-103
{
    if (tv == 0 && uf) { tv = 0xFFu; return; }
    ps = (ps - 1u) & 0xFFFFu;
    if (ps == 0) {
        ps = uf ? 1u : sel;
        if (tv == 0) { uf = 1; tv = 0xFFu; } else tv -= 1u;
    }
}

// m calls of Pia::tick (pia.rs:80-103), a prescaler period at a time.  Only
// the accesses that see or set the timer, and the state's store, need them:
// the TIA and the PIA do not interact.
static __device__ __noinline__ uint2 r_pia_ticks(uint32_t tp, uint32_t su, uint32_t m)
{
    uint32_t tv = tp & 0xFFFFu, ps = tp >> 16, sel = su & 0xFFFFu, uf = su >> 16;
    while (m) {
        if (ps == 0 || (uf && tv == 0)) { r_pia_tick(tv, ps, sel, uf); m--; continue; }
        if (uf && ps == 1u) { tv = (tv - m) & 0xFFu; break; }         // after underflow: one count per tick
        if (m < ps) { ps -= m; break; }
        m -= ps;                                                     // the tick that empties the prescaler
        ps = uf ? 1u : sel;
        if (tv == 0) { uf = 1; tv = 0xFFu; } else tv -= 1u;
    }
    return make_uint2(tv | (ps << 16), sel | (uf << 16));
}

// n TIA clocks.
static __device__ __noinline__ RState render_clocks(RState s, uint32_t n, uint32_t pins, uint8_t* pv, uint8_t* fbp)
{
    r_advance(s, n, pins, pv, fbp);
    return s;
}

static __device__ __forceinline__ uint32_t r_resp_player(uint32_t clk)       // tia.rs:512-520
{
    const uint32_t dc = (clk + (clk < 68u ? 3u : 4u) + 156u) % 228u;
    return dc >= 68u ? dc - 68u : dc + 160u - 68u;
}

static __device__ __forceinline__ void r_resize_commit(RState& s, uint8_t* pv)  // tia.rs:247-268
{
    const uint32_t vbt = s.vtop >> 16, top = s.vtop & 0xFFFFu;
    if (vbt > 262u) return;
    const uint32_t clamped = vbt < 23u ? 23u : vbt > 32u ? 32u : vbt;
    const uint32_t cand = clamped < top ? clamped : top;
    uint32_t ntop = top;
    const uint32_t ptop = rp16(pv, RB_PTOP), pfr = rp8(pv, RB_PFRAMES);
    if (cand != ptop) { wp16(pv, RB_PTOP, cand); wp8(pv, RB_PFRAMES, 3u); }
    else if (pfr > 0) { wp8(pv, RB_PFRAMES, pfr - 1u); if (pfr == 1u) ntop = ptop; }
    s.vtop = ntop | (ntop << 16);
}

// Tia::write (tia.rs:570-674) of register a & 0x3F.
// Registers whose write can change a pixel or a collision latch from the
// next clock on: VSYNC, VBLANK, NUSIZx-REFPx, RESPx-RESBL, GRPx-ENABL,
// VDELx-RESMPx, HMOVE and CXCLR.  The playfield registers reach the pixels
// through the delayed-write queue (flushed when it fires); WSYNC, RSYNC,
// audio, HMxx and HMCLR never do.
constexpr uint64_t R_PIXEL_REGS = 0x17E0F81F1FF3ull;

static __device__ __forceinline__ void r_write(uint32_t a, uint32_t v, RState& s, uint8_t* pv, uint8_t* fbp)
{
    if ((R_PIXEL_REGS >> (a & 0x3Fu)) & 1u) r_pending(s, pv, fbp, s.clock);   // the pixels drawn before the write
    switch (a & 0x3Fu) {
    case 0x00:
        if (!(s.tw & 2u) && (v & 2u)) { r_observe(s, pv, fbp); r_resize_commit(s, pv); s.scanline = 0; s.tw |= TW_FCOMP; }
        s.tw = (s.tw & ~0xFFu) | v;
        break;
    case 0x01:
        if (v & 0x40u) s.tw |= TW_LATCH | TW_L4 | TW_L5;
        else s.tw &= ~TW_LATCH;
        if (v & 0x80u) { s.pcnt = 0; s.tw |= TW_PDUMP; }
        else s.tw &= ~TW_PDUMP;
        s.tw = (s.tw & ~0xFF00u) | (v << 8);
        break;
    case 0x02: s.tw |= TW_WSYNC; break;
    case 0x04: wp8(pv, PB_NUSIZ0, v); break;
    case 0x05: wp8(pv, PB_NUSIZ1, v); break;
    case 0x06: wp8(pv, PB_COLUP0, v); break;
    case 0x07: wp8(pv, PB_COLUP1, v); break;
    case 0x08: wp8(pv, PB_COLUPF, v); break;
    case 0x09: wp8(pv, PB_COLUBK, v); break;
    case 0x0A: wp8(pv, PB_CTRLPF, v); break;
    case 0x0B: wp8(pv, PB_REFP0, (v & 8u) ? 1u : 0u); break;
    case 0x0C: wp8(pv, PB_REFP1, (v & 8u) ? 1u : 0u); break;
    case 0x0D: case 0x0E: case 0x0F: {                              // written after one TIA clock
        const uint32_t n = rp8(pv, RB_DLEN);
        if (n < 4u) {
            wp8(pv, RB_DQ + 3u * n, 1u);
            wp8(pv, RB_DQ + 3u * n + 1u, a & 0x3Fu);
            wp8(pv, RB_DQ + 3u * n + 2u, v);
            wp8(pv, RB_DLEN, n + 1u);
        } else {                                                    // queue full: written now
            r_pending(s, pv, fbp, s.clock);
            wp8(pv, (a & 0x3Fu) == 0x0Du ? PB_PF0 : (a & 0x3Fu) == 0x0Eu ? PB_PF1 : PB_PF2, v);
        }
        break;
    }
    case 0x10: wp16(pv, PB_POS + 0u, r_resp_player(s.clock)); break;
    case 0x11: wp16(pv, PB_POS + 2u, r_resp_player(s.clock)); break;
    case 0x12: wp16(pv, PB_POS + 4u, mod160((int)s.clock - 68 + 5)); break;
    case 0x13: wp16(pv, PB_POS + 6u, mod160((int)s.clock - 68 + 5)); break;
    case 0x14: wp16(pv, PB_POS + 8u, mod160((int)s.clock - 68 + 5)); break;
    case 0x1B: wp8(pv, PB_GRP0_OLD, rp8(pv, PB_GRP0)); wp8(pv, PB_GRP0, v); break;
    case 0x1C: wp8(pv, PB_GRP1_OLD, rp8(pv, PB_GRP1)); wp8(pv, PB_GRP1, v); wp8(pv, PB_ENABL_OLD, rp8(pv, PB_ENABL)); break;
    case 0x1D: wp8(pv, PB_ENAM0, (v & 2u) ? 1u : 0u); break;
    case 0x1E: wp8(pv, PB_ENAM1, (v & 2u) ? 1u : 0u); break;
    case 0x1F: wp8(pv, PB_ENABL, (v & 2u) ? 1u : 0u); break;
    case 0x20: case 0x21: case 0x22: case 0x23: case 0x24: wp8(pv, PB_HM + ((a & 0x3Fu) - 0x20u), v); break;
    case 0x25: wp8(pv, PB_VDELP0, v & 1u); break;
    case 0x26: wp8(pv, PB_VDELP1, v & 1u); break;
    case 0x27: wp8(pv, PB_VDELBL, v & 1u); break;
    case 0x28: wp8(pv, PB_RESMP0, (v & 2u) ? 1u : 0u); break;
    case 0x29: wp8(pv, PB_RESMP1, (v & 2u) ? 1u : 0u); break;
    case 0x2A:                                                      // HMOVE
        for (uint32_t o = 0; o < 5u; o++) {
            const int hm = (int)(int8_t)(uint8_t)rp8(pv, PB_HM + o) >> 4;
            wp16(pv, PB_POS + 2u * o, mod160((int)rp16(pv, PB_POS + 2u * o) - hm));
        }
        s.tw |= TW_HMOVE;
        break;
    case 0x2B: for (uint32_t o = 0; o < 5u; o++) wp8(pv, PB_HM + o, 0u); break;
    case 0x2C: for (uint32_t o = 0; o < 8u; o++) wp8(pv, PB_CX + o, 0u); break;
    default: break;                                                 // RSYNC, audio
    }
}

// `n` TIA clocks (those owed and the two of its own cycle before the write,
// src/atari.rs:207-222), then the write of a TIA register.  The clock after
// it is owed with the cycles that follow.
static __device__ __noinline__ RState render_write(uint32_t a, uint32_t v, uint32_t n, RState s, uint32_t pins, uint8_t* pv,
                                                   uint8_t* fbp)
{
    r_advance(s, n, pins, pv, fbp);
    r_write(a, v, s, pv, fbp);
    return s;
}

// Tia::read (tia.rs:533-566).
static __device__ __forceinline__ uint32_t r_read_tia(uint32_t a, const RState& s, uint32_t pins, uint32_t pads, const uint8_t* pv)
{
    const uint32_t r = a & 0x0Fu;
    if (r < 8u) return rp8(pv, PB_CX + r);
    switch (r) {
    case 0x8: return s.pcnt >= (pads & 0xFFu) ? 0x80u : 0u;
    case 0x9: return s.pcnt >= ((pads >> 8) & 0xFFu) ? 0x80u : 0u;
    case 0xA: case 0xB: return 0x80u;
    case 0xC: return (s.tw & TW_LATCH) ? ((s.tw & TW_L4) ? 0x80u : 0u) : ((pins & 0x10000u) ? 0x80u : 0u);
    case 0xD: return (s.tw & TW_LATCH) ? ((s.tw & TW_L5) ? 0x80u : 0u) : ((pins & 0x20000u) ? 0x80u : 0u);
    default: return 0u;
    }
}

struct RRead {
    RState s;
    uint32_t v;
};

// `n` owed TIA clocks, then the read of a TIA register (Bus::read,
// src/atari.rs:195-205), collisions drawn up to the beam.  The clocks of its
// own cycle are owed with those that follow.
static __device__ __noinline__ RRead render_read(uint32_t a, uint32_t n, RState s, uint32_t pins, uint32_t pads, uint8_t* pv,
                                                 uint8_t* fbp)
{
    r_advance(s, n, pins, pv, fbp);
    if ((a & 0x0Fu) < 8u) r_pending(s, pv, fbp, s.clock);            // collisions so far
    RRead out;
    out.v = r_read_tia(a, s, pins, pads, pv);
    out.s = s;
    return out;
}

// ---------------------------------------------------------------- DPC (Pitfall II)
// The DPC chip of FA_SCHEME_DPC carts (no counterpart in the reference),
// with the semantics the oracle's DPC section fixes: 8 data fetchers (11-bit
// counter, top, bottom, flag), an 8-bit random number generator and 3 music
// channels clocked at 20 kHz of Cpu::cycles.  The registers are the R_DPC_*
// rows from R_DPC_CNT on, register word k at d[k * S]: while a unit runs, in
// the console's shared-memory slab (as rows of HBM, changed in place one
// access at a time, they were 7 dependent loads, and the oscillator two 64-bit
// divisions, an access).  A read of $1000-$103F (wr 0; returns the value) or
// a write of v to $1040-$107F (wr 1).  now: the oscillator's clocks before the
// accessing instruction.  `disp` is the 2K of display data.
static __device__ __forceinline__ uint32_t dpc_byte(uint32_t w, uint32_t k) { return (w >> ((k & 3u) * 8u)) & 0xFFu; }

static __device__ __forceinline__ uint32_t dpc_io(uint32_t a, uint32_t v, uint32_t wr, uint32_t* d, uint32_t S, sptr disp,
                                                  uint32_t now)
{
    constexpr uint32_t CNT = 0u, TOP = R_DPC_TOP - R_DPC_CNT, BOT = R_DPC_BOT - R_DPC_CNT, MISC = R_DPC_MISC - R_DPC_CNT,
                       OSC = R_DPC_OSC - R_DPC_CNT;
    const uint32_t misc = d[MISC * S];
    uint32_t flags = misc & 0xFFu, music = (misc >> 8) & 7u, rnd = (misc >> 16) & 0xFFu;
    // The music channels up to the instruction's start: one clock of the
    // oscillator counts a channel's low byte down, the clock after 0 reloads
    // top; the flag is set while the low byte is above bottom.
    const uint32_t clocks = now - d[OSC * S];
    d[OSC * S] = now;
    if (clocks && music) {
#pragma unroll 1
        for (uint32_t f = 5u; f < 8u; f++) {
            if (!((music >> (f - 5u)) & 1u)) continue;
            uint32_t& cw = d[(CNT + (f >> 1)) * S];
            const uint32_t sh = (f & 1u) * 16u, cnt = (cw >> sh) & 0x7FFu;
            const uint32_t top = dpc_byte(d[(TOP + (f >> 2)) * S], f);
            const uint32_t bot = dpc_byte(d[(BOT + (f >> 2)) * S], f);
            uint32_t low = cnt & 0xFFu;
            low = clocks <= low ? low - clocks : top - (clocks - low - 1u) % (top + 1u);
            cw = (cw & ~(0xFFFFu << sh)) | (((cnt & 0x700u) | low) << sh);
            flags = low > bot ? flags | (1u << f) : flags & ~(1u << f);
        }
    }
    const uint32_t k = a & 7u, f = (a >> 3) & 7u, sh = (k & 1u) * 16u;
    uint32_t& cw = d[(CNT + (k >> 1)) * S];
    uint32_t& tw = d[(TOP + (k >> 2)) * S];
    uint32_t& bw = d[(BOT + (k >> 2)) * S];
    uint32_t cnt = (cw >> sh) & 0x7FFu, out = 0u;
    if (!wr) {
        const bool mus = k >= 5u && ((music >> (k - 5u)) & 1u);
        // The generator shifts left, taking in the XNOR of bits 7, 5, 4, 3.
        rnd = ((rnd << 1) | (~((rnd >> 7) ^ (rnd >> 5) ^ (rnd >> 4) ^ (rnd >> 3)) & 1u)) & 0xFFu;
        if (!mus) {
            const uint32_t low = cnt & 0xFFu;
            if (low == dpc_byte(tw, k)) flags |= 1u << k;
            else if (low == dpc_byte(bw, k)) flags &= ~(1u << k);
        }
        const uint32_t flag = ((flags >> k) & 1u) ? 0xFFu : 0u, data = lds8(disp + (2047u - cnt));
        switch (f) {
        case 0:
            if (k < 4u) out = rnd;
            else
                for (uint32_t m = 0; m < 3u; m++) out += (((music & (flags >> 5)) >> m) & 1u) ? 4u + m : 0u;
            break;
        case 1: out = data; break;
        case 2: out = data & flag; break;
        case 7: out = flag; break;
        default: break;
        }
        if (!mus) cw = (cw & ~(0xFFFFu << sh)) | (((cnt - 1u) & 0x7FFu) << sh);
    } else {
        const uint32_t bs = (k & 3u) * 8u;
        switch (f) {
        case 0: tw = (tw & ~(0xFFu << bs)) | (v << bs); flags &= ~(1u << k); break;
        case 1: bw = (bw & ~(0xFFu << bs)) | (v << bs); break;
        case 2: cw = (cw & ~(0xFFFFu << sh)) | (((cnt & 0x700u) | v) << sh); break;
        case 3:
            cw = (cw & ~(0xFFFFu << sh)) | ((((v & 7u) << 8) | (cnt & 0xFFu)) << sh);
            if (k >= 5u) music = (music & ~(1u << (k - 5u))) | (((v >> 4) & 1u) << (k - 5u));
            break;
        case 6: rnd = 1u; break;
        default: break;
        }
    }
    d[MISC * S] = flags | (music << 8) | (rnd << 16);
    return out;
}

// ---------------------------------------------------------------- PIA timer (pia.rs:107-166)
// Pia::tick_n on the unpacked timer: value, prescaler, interval, underflow.
static __device__ __forceinline__ void pia_tick_n(uint32_t& tv, uint32_t& ps, uint32_t sel, uint32_t& uf, uint32_t n)
{
    if (n == 0) return;
    if (tv == 0 && uf) { tv = (0xFFu - (n - 1u)) & 0xFFu; return; }
    uint32_t rem = n;
    if (ps > 0) {
        if (rem < ps) { ps -= rem; return; }
        rem -= ps;
        ps = 0;
        if (tv == 0) {
            uf = 1;
            tv = rem ? ((0xFFu - (rem - 1u)) & 0xFFu) : 0xFFu;
            return;
        }
        tv -= 1u;
    }
    if (rem == 0) { ps = sel; return; }
    uint32_t full, left;
    if ((sel & (sel - 1u)) == 0) {                    // 1, 8, 64, 1024
        uint32_t sh = __ffs(sel) - 1u;
        full = rem >> sh;
        left = rem & (sel - 1u);
    } else {
        full = rem / sel;
        left = rem % sel;
    }
    if (full >= tv) {
        rem = (rem - ((tv * sel) & 0xFFFFu)) & 0xFFFFu;   // u16 arithmetic as in the reference
        uf = 1;
        tv = rem ? ((0xFFu - (rem - 1u)) & 0xFFu) : 0xFFu;
    } else {
        tv -= full;
        ps = sel - left;
    }
}

// Headless timer bookkeeping (Emu::pia_count).  The window of a timer state
// is the run of cycles over which tick_n only counts.  With tv >= 1 it ends
// at the decrement that brings tv to zero: ps (a prescaler of 0, just after
// an underflow, counts as a whole interval: tick_n then decrements after sel
// cycles) plus tv - 1 intervals.  With tv = 0, no underflow flag and a
// prescaler left, it ends when the prescaler runs out (that decrement
// underflows).  Any other state, an interval that is not one of 1, 8, 64,
// 1024, or a prescaler above the interval (states only an upload makes)
// have no window: 0, every call exact.
static __device__ __forceinline__ uint32_t pia_span_of(uint32_t tv, uint32_t ps, uint32_t sel, uint32_t uf)
{
    if (sel == 0u || (sel & (sel - 1u)) != 0u || sel > 1024u || ps > sel) return 0u;
    if (tv == 0u) return uf ? 0u : ps;
    return (ps ? ps : sel) + ((tv - 1u) << (__ffs(sel) - 1u));
}
// (tv, ps) with the counted cycles (the window less tlim) applied: fewer
// cycles than the window, so tick_n's counting branches alone apply.
static __device__ __forceinline__ uint2 pia_now_of(uint32_t tv, uint32_t ps, uint32_t sel, uint32_t uf, uint32_t tlim)
{
    const uint32_t e = pia_span_of(tv, ps, sel, uf) - tlim;
    if (e == 0u) return make_uint2(tv, ps);
    const uint32_t p0 = ps ? ps : sel;
    if (e < p0) return make_uint2(tv, p0 - e);
    const uint32_t k = e - p0;
    return make_uint2(tv - 1u - (k >> (__ffs(sel) - 1u)), sel - (k & (sel - 1u)));
}
// An INTIM read (pia.rs:187-190): the counted cycles settled, the underflow
// flag cleared (tv = 0 with a prescaler left may gain a window by it).
// Packed (tv | ps << 16, sel | uf << 16, tlim); the value read is tv & 0xFF.
static __device__ __forceinline__ uint4 pia_intim_io(uint32_t tv_ps, uint32_t sel_uf, uint32_t tlim)
{
    const uint32_t sel = sel_uf & 0xFFFFu;
    const uint2 t = pia_now_of(tv_ps & 0xFFFFu, tv_ps >> 16, sel, sel_uf >> 16, tlim);
    return make_uint4(t.x | (t.y << 16), sel, pia_span_of(t.x, t.y, sel, 0u), 0u);
}
// Pia::write of an I/O register by the headless core (src/pia.rs:202-228):
// (ports, tv | ps << 16, sel | uf << 16, tlim) after it.  A port write
// leaves the timer and its counting alone; a timer write replaces value,
// prescaler, interval and flag, so the cycles counted so far no longer
// matter.
static __device__ __forceinline__ uint4 pia_store_io(uint32_t a, uint32_t v, uint32_t ports, uint32_t tp, uint32_t su,
                                                  uint32_t tlim)
{
    if (a & 0x10u) {
        const uint32_t sel = 1u << ((0xA630u >> (4u * (a & 3u))) & 0xFu);   // 1, 8, 64, 1024
        return make_uint4(ports, v | (sel << 16), sel, pia_span_of(v, sel, sel, 0u));
    }
    const uint32_t sh = 8u * (a & 3u);                                 // pa_out pa_ddr pb_out pb_ddr
    return make_uint4((ports & ~(0xFFu << sh)) | (v << sh), tp, su, tlim);
}
// Packed (tv | ps << 16, sel | uf << 16, tlim) after settling and one exact
// call of n cycles.
static __device__ __forceinline__ uint4 pia_sync_io(uint32_t tv_ps, uint32_t sel_uf, uint32_t tlim, uint32_t n)
{
    const uint32_t sel = sel_uf & 0xFFFFu;
    uint32_t uf = sel_uf >> 16;
    const uint2 t = pia_now_of(tv_ps & 0xFFFFu, tv_ps >> 16, sel, uf, tlim);
    uint32_t tv = t.x, ps = t.y;
    pia_tick_n(tv, ps, sel, uf, n);
    return make_uint4(tv | (ps << 16), sel | (uf << 16), pia_span_of(tv, ps, sel, uf), 0u);
}

// ---------------------------------------------------------------- decimal mode (cpu.rs:153-241)
// ADC and SBC with D set: (a, nz, carry, V in bit 7) as Emu keeps them.
static __device__ __forceinline__ uint4 decimal_op(bool sub, uint32_t a, uint32_t v, uint32_t c)
{
    if (sub) {
        const uint32_t b = c ^ 1u;
        const int bin = (int)a - (int)v - (int)b;
        const uint32_t r = (uint32_t)bin & 0xFFu;
        uint32_t lo = ((a & 0xFu) - (v & 0xFu) - b) & 0xFFu, lob = 0;
        if (lo & 0x80u) { lo = (lo - 6u) & 0xFFu; lob = 1; }
        uint32_t hi = ((a >> 4) - (v >> 4) - lob) & 0xFFu;
        if (hi & 0x80u) hi = (hi - 6u) & 0xFFu;
        return make_uint4(((hi & 0xFu) << 4) | (lo & 0xFu), r, bin >= 0 ? 1u : 0u, (a ^ v) & (a ^ r));
    }
    uint32_t lo = (a & 0xFu) + (v & 0xFu) + c;
    if (lo > 9u) lo += 6u;
    uint32_t hi = (a >> 4) + (v >> 4) + (lo > 0xFu ? 1u : 0u);
    const uint32_t bin = (a + v + c) & 0xFFu, res = ((hi << 4) | (lo & 0xFu)) & 0xFFu;
    const uint32_t nz = (bin ? 1u : 0u) | ((hi & 8u) << 12), vf = ~(a ^ v) & (a ^ res);
    if (hi > 9u) hi += 6u;
    return make_uint4(((hi & 0xFu) << 4) | (lo & 0xFu), nz, hi > 0xFu ? 1u : 0u, vf);
}

// The headless TIA's scanlines of a run of instruction ticks
// (headless_tia.rs:153-198) that brought the beam from below 228 to `clk`
// TIA clocks of the line it started on, no tick more than a line: what the
// ticks one by one leave.  lw = scanline (below 262) | paddle_counter << 16.
// Returns (clock, lw, tw).
static __device__ __forceinline__ uint4 tia_fold_io(uint32_t clk, uint32_t lw, uint32_t tw)
{
    const uint32_t lines = clk / 228u;
    uint32_t s = (lw & 0xFFFFu) + lines, pc = lw >> 16;
    if (s >= 262u) { s %= 262u; tw |= TW_FCOMP; }
    if (!(tw & TW_PDUMP) && pc < 256u) pc = pc + lines < 256u ? pc + lines : 256u;
    return make_uint4(clk - lines * 228u, s | (pc << 16), tw & ~TW_WSYNC, 0u);
}

// SLICED: the core of E0 and 3F carts (with DPC, of DPC carts alone; with
// FE, of FE carts alone).  The DPC and FE cores are their own builds so that
// the E0 / 3F core carries none of their bus decode.  The FE core issues
// every bus access the reference CPU makes, phantom ones included: any of
// them can select an FE cart's bank.
template <int BLOCK, bool RENDER = false, bool SLICED = false, bool DPC = false, bool FE = false>
struct Emu {
    static_assert(!DPC || (SLICED && !RENDER), "the DPC core is a headless sliced core");
    static_assert(!FE || (SLICED && !RENDER && !DPC), "the FE core is a headless sliced core");
    // ---- placement
    uint8_t* pv;             // this thread's RAM (shared memory, interleaved by thread)
    const FaGroup* G;        // the instance's group (HBM state rows, stride)
    uint32_t i;              // the instance's index in its group
    const uint8_t* rom;      // shared-memory ROM image, nbanks * 4 KiB
    uint32_t hot_lo, nbanks;
    int32_t lim;             // 4K-bank carts: ROM addresses << 19 below this, and the next two, are clear of the hotspots
    // ---- CPU (src/cpu.rs:96-105)
    // P is kept apart: what an instruction sets costs one move or none, and
    // PHP, BRK and the state rows assemble it (get_p / set_p).
    uint32_t R, pc;          // a | x << 8 | y << 16 | sp << 24 (packed, so a table word selects the register)
    uint32_t F;              // flags, by bytes: Z is set when byte 0 is 0; N is bit 7 of byte 0 or byte 1; C: byte 2
                             // (0 or 1); V: bit 7 of byte 3
    uint32_t p;              // P's I, B and unused bits
    uint32_t pd;             // T_UV in decimal mode, else 0
    uint32_t bank;           // 4K-bank carts: the bank's offset in the ROM image (index << 12)
    uint32_t kb;             // scheduling key above pc: frame << 25 | hotspot accesses this frame << 16, each saturating
    uint32_t slices;         // SLICED (E0, 3F carts): the 1K ROM slice of window k in byte k
    uint32_t cyc_acc;         // instruction cycles not yet added to Cpu::cycles in HBM (headless: up to the last sync)
    // Headless time.  An instruction only adds its cycles to `el` and compares
    // it with `dl`; the beam, the timer and the cycle counts are brought up to
    // date (sync) when something reads or changes them, or when el reaches dl:
    // the end of the timer's window, a frame limit, or an instruction that
    // wrote WSYNC or VSYNC (dl = 0).
    uint32_t el;             // cycles since the last sync
    uint32_t dl;             // cycles from the last sync at which the frame loop must look
    // ---- PIA (src/pia.rs:26-44): timer unpacked, ports and input pins packed
    //      (touched only by I/O accesses)
    uint32_t tp;             // timer value | prescaler << 16 (the R_TIMER row word)
    uint32_t su;             // interval (1, 8, 64, 1024) | underflow flag << 16
    uint32_t tlim;           // headless: cycles the timer may still count before an exact tick
                             // (tp lags by pia_span() - tlim counted cycles; see pia_count)
    uint32_t ports;          // pa_out | pa_ddr<<8 | pb_out<<16 | pb_ddr<<24
    uint32_t pins;           // pa_in | pb_in<<8 | inpt4<<16 | inpt5<<17
    uint32_t pads;           // paddle0 | paddle1<<8
    // ---- TIA (src/headless_tia.rs:16-45): beam position unpacked, flags packed
    uint32_t clock, scanline, pcnt;
    uint32_t tw;             // vsync | vblank<<8 | wsync<<16 | frame_complete<<17 | paddle_dumped<<18
    // ---- run bookkeeping
    uint32_t instr;           // instructions executed in this launch (statistics)

    // The instance's HBM rows.  Cpu::cycles, the frame counter and the run
    // status stay there and change only at frame boundaries.
    // The group through a pointer that the compiler cannot follow: the
    // descriptor lies in constant memory, and it would load the fields that
    // rare paths use ahead of the interpreter's loop and spill them.
    __device__ __forceinline__ const FaGroup* grp() const
    {
        const FaGroup* g = G;
#ifdef __CUDA_ARCH__
        asm volatile("" : "+l"(g));
#endif
        return g;
    }
    __device__ __forceinline__ uint32_t* column() const { return grp()->state + i; }
    __device__ __forceinline__ uint32_t& row(uint32_t w) const { return column()[(size_t)w * grp()->stride]; }
    __device__ __forceinline__ void fold_cycles()
    {
        uint32_t& lo = row(R_CYC_LO);
        const uint32_t v = lo + cyc_acc;
        if (v < cyc_acc) row(R_CYC_HI) += 1u;
        lo = v;
        cyc_acc = 0;
    }
    __device__ __forceinline__ void set_status(uint32_t bits) { row(R_STATUS) |= bits; }

    __device__ __forceinline__ bool vsync_on() const { return (tw & 2u) != 0; }
    __device__ __forceinline__ bool wsync() const { return (tw & TW_WSYNC) != 0; }

    // ------------------------------------------------------------ private bytes
    // Headless RAM: byte o of lane t at o * BLOCK + t, one multiply to reach;
    // lanes at one offset share 8 words, at different offsets at most 4 of
    // them meet in a bank.
    __device__ __forceinline__ uint32_t poff(uint32_t o) const { return RENDER ? priv_off<BLOCK>(o) : o * BLOCK; }
    __device__ __forceinline__ uint32_t ldp(uint32_t o) const { return pv[poff(o)]; }
    __device__ __forceinline__ void stp(uint32_t o, uint32_t v) { pv[poff(o)] = (uint8_t)v; }

    // ------------------------------------------------------------ flags
    __device__ __forceinline__ void set_nz(uint32_t v) { F = (F & 0xFFFF0000u) | v; }       // v: bytes 0 and 1
    __device__ __forceinline__ void setv(uint32_t v) { F = (F & 0x00FFFFFFu) | (v << 24); }
    __device__ __forceinline__ uint32_t get_p() const
    {
        return p | (pd ? F_D : 0u) | ((F >> 16) & F_C) | ((F & 0xFFu) ? 0u : F_Z) | ((F >> 25) & F_V) | ((F | (F >> 8)) & F_N);
    }
    __device__ __forceinline__ void set_p(uint32_t v)
    {
        p = v & (F_I | F_B | F_U);
        pd = (v & F_D) ? T_UV : 0u;
        F = ((v & F_Z) ? 0u : 1u) | ((v & F_N) << 8) | ((v & F_C) << 16) | ((v & F_V) << 25);
    }
    // One more hotspot access this frame (a scheduling key only, saturating;
    // at 510, so that no key is all ones).
    __device__ __forceinline__ void bump()
    {
        if ((kb & 0x01FF0000u) != 0x01FE0000u) kb += 0x10000u;
    }

    // ------------------------------------------------------------ bank switching
    // A hotspot access selects its bank (src/atari.rs:460-492) and counts one
    // more bank-switch point passed this frame.
    __device__ __forceinline__ void bsw(uint32_t a13)
    {
        const uint32_t d = a13 - hot_lo;
        if (d < nbanks) { bank = d << 12; bump(); }
    }
    // Sliced carts.  The ROM byte at a (A12 set): window (a >> 10) & 3 holds
    // slice `slices` byte k.  On the chain of every instruction's loads, so
    // the byte is taken by one permute, and DPC's and FE's four slices, which
    // lie in a row, by an offset (with code_ok's shorter tests, before and
    // now: DPC 5.19 and 4.78 ms, FE 8.99 and 8.31, 80,000 consoles x 4 frames;
    // E0 / 3F, 100,000 x 4: 63.3 and 61.8).
    __device__ __forceinline__ uint32_t srom(uint32_t a) const
    {
        if constexpr (DPC || FE) return (slices & 4u) * 1024u + (a & 0xFFFu);   // four slices in a row
        else return __byte_perm(slices, 0u, ((a >> 10) & 3u) | 0x4440u) * 1024u + (a & 0x3FFu);
    }
    // E0: any access to $1FE0-$1FF7 maps slice (a & 7) into window (a - $1FE0) >> 3.
    // DPC core: any access to $1FF8 / $1FF9 maps program bank 0 / 1 (slices 4b..4b+3).
    __device__ __forceinline__ void e0_hot(uint32_t a13)
    {
        if constexpr (DPC) {
            if ((a13 | 1u) == 0x1FF9u) {
                slices = (a13 & 1u) * 0x04040404u + 0x03020100u;
                bump();
            }
        } else {
            const uint32_t d = a13 - 0x1FE0u;
            if (d < 24u && fa_map_kind(hot_lo) == FA_MAP_E0) {
                const uint32_t sh = (d >> 3) * 8u;
                slices = (slices & ~(0xFFu << sh)) | ((a13 & 7u) << sh);
                bump();
            }
        }
    }
    // An access to ROM space: its hotspots.
    __device__ __forceinline__ void hot(uint32_t a13)
    {
        if constexpr (!SLICED) bsw(a13);
        else if constexpr (!FE) e0_hot(a13);
    }
    // The bank state (fa_state::mapper) to and from `slices`, for this core's
    // schemes only (fa_slices_from_mapper / fa_mapper_from_slices decode all
    // of them; a core carries only its own).
    __device__ __forceinline__ uint32_t slices_of(uint32_t m) const
    {
        if constexpr (DPC || FE) return fa_slices_4k_bank(m, FE);
        else return fa_slices_e0_3f(hot_lo, m);
    }
    __device__ __forceinline__ uint32_t mapper_of(uint32_t s) const
    {
        if constexpr (DPC || FE) return fa_mapper_4k_bank(s, FE);
        else return fa_mapper_e0_3f(hot_lo, s);
    }
    // FE core: the access after one to $01FE selects the 4K bank by bit 5 of
    // its data (set: bank 0, clear: bank 1); bit 7 of `slices` marks that the
    // last access was to $01FE.  v is the byte the access read or wrote.
    __device__ __forceinline__ void fe_note(uint32_t a13, uint32_t v)
    {
        if (slices & 0x80u) {
            slices = ((v & 0x20u) ? 0u : 0x04040404u) + 0x03020100u;
            bump();
        }
        if (a13 == 0x01FEu) slices |= 0x80u;
    }
    // DPC core: reads of $1000-$103F and writes of $1040-$107F reach the registers.
    __device__ __forceinline__ uint32_t dpc(uint32_t a13, uint32_t v, uint32_t wr)
    {
        return dpc_io(a13, v, wr, dpc_regs(), dpc_step(), to_sptr(rom) + 8192u, dpc_now());
    }
    // The DPC core's registers: FA_DPC_WORDS rows of BLOCK words after the
    // RAM in the console's slab (the host runs on the rows of the column).
    // The last two hold the oscillator at the frame's start: its clocks, and
    // the remainder of the division.
    __device__ __forceinline__ uint32_t* dpc_regs() const
    {
#ifdef __CUDA_ARCH__
        const uint32_t t = threadIdx.x & (BLOCK - 1u);
        return (uint32_t*)(pv - t + BLOCK * 128u) + t;
#else
        return &row(R_DPC_CNT);
#endif
    }
    __device__ __forceinline__ uint32_t dpc_step() const
    {
#ifdef __CUDA_ARCH__
        return BLOCK;
#else
        return G->stride;
#endif
    }
    // The oscillator's clocks at the instruction's start, 60000 per 3579545
    // of Cpu::cycles (as 12000 per 715909), exactly.
    __device__ __forceinline__ uint32_t dpc_now() const
    {
        const uint32_t n = cyc_acc + el;
#ifdef __CUDA_ARCH__
        const uint32_t* d = dpc_regs();
        const uint32_t q = d[(FA_DPC_WORDS - 2u) * BLOCK], r = d[(FA_DPC_WORDS - 1u) * BLOCK];
        if (n < 350000u) return q + (r + n * 12000u) / 715909u;       // r < 715909: within 32 bits
        return q + (uint32_t)((r + n * 12000ull) / 715909ull);
#else
        const uint2 b = dpc_clock();
        return b.x + (uint32_t)((b.y + n * 12000ull) / 715909ull);
#endif
    }
    __device__ __forceinline__ uint2 dpc_clock() const                // of the rows' Cpu::cycles
    {
        const unsigned long long t = ((unsigned long long)row(R_CYC_HI) << 32) | row(R_CYC_LO);
        const unsigned long long x = (t % 715909ull) * 12000ull;
        return make_uint2((uint32_t)(t / 715909ull * 12000ull + x / 715909ull), (uint32_t)(x % 715909ull));
    }
    // At a frame's start, after Cpu::cycles was brought up to date.
    __device__ __forceinline__ void dpc_frame()
    {
#ifdef __CUDA_ARCH__
        const uint2 b = dpc_clock();
        dpc_regs()[(FA_DPC_WORDS - 2u) * BLOCK] = b.x;
        dpc_regs()[(FA_DPC_WORDS - 1u) * BLOCK] = b.y;
#endif
    }
    __device__ __forceinline__ void load_dpc()
    {
#ifdef __CUDA_ARCH__
        for (uint32_t k = 0; k < FA_DPC_WORDS - 2u; k++) dpc_regs()[k * BLOCK] = row(R_DPC_CNT + k);
#endif
    }
    __device__ __forceinline__ void store_dpc() const
    {
#ifdef __CUDA_ARCH__
        for (uint32_t k = 0; k < FA_DPC_WORDS - 2u; k++) row(R_DPC_CNT + k) = dpc_regs()[k * BLOCK];
#endif
    }
    // 3F: a write of v to $0000-$003F maps 2K bank v mod n at $1000-$17FF.
    __device__ __forceinline__ void f3_write(uint32_t a13, uint32_t v)
    {
        if (a13 < 0x40u && fa_map_kind(hot_lo) == FA_MAP_3F) {
            const uint32_t b = v % (hot_lo & 0xFFu);
            slices = (slices & 0xFFFF0000u) | (2u * b) | ((2u * b + 1u) << 8);
            bump();
        }
    }

    // ------------------------------------------------------------ TIA (headless_tia.rs)
    __device__ __forceinline__ void end_scanline()                   // :183-198
    {
        clock = (clock - 228u) & 0xFFFFu;
        scanline = (scanline + 1u) & 0xFFFFu;
        tw &= ~TW_WSYNC;
        if (!(tw & TW_PDUMP) && pcnt < 256u) pcnt++;
        if (scanline >= 262u) { scanline = 0; tw |= TW_FCOMP; }
    }
    __device__ __forceinline__ void tia_tick(uint32_t n)            // :153-158
    {
        clock = (clock + 3u * n) & 0xFFFFu;
        if (clock >= 228u) end_scanline();
    }
    __device__ __forceinline__ uint32_t tia_skip()                   // :163-180
    {
        uint32_t rem = clock >= 228u ? 0u : 228u - clock;
        uint32_t c = (rem + 2u) / 3u;
        if (c) { clock = 228u; end_scanline(); }
        return c;
    }
    // Bring the beam, the timer's window and the cycle counter up to the d
    // cycles counted so far (at an instruction boundary).  Only instructions
    // that do not end the timer's window are counted, and only from a beam
    // position and scanline in range (due() keeps dl at 0 otherwise), so the
    // lines they complete fold together (tia_fold_io).
    __device__ __forceinline__ void fold(uint32_t d)
    {
        const uint32_t clk = clock + 3u * d;
        if (clk < 228u || d == 0u) {
            clock = clk;
        } else {
            const uint4 r = tia_fold_io(clk, scanline | (pcnt << 16), tw);
            clock = r.x; scanline = r.y & 0xFFFFu; pcnt = r.y >> 16; tw = r.z;
        }
        tlim -= d;
        cyc_acc += d;
    }
    __device__ __forceinline__ void sync()
    {
        fold(el);
        dl -= el;
        el = 0;
    }
    // The cycles that may be counted before the frame loop must look: the
    // timer's window, `lim` cycles to the frame limit, none while the beam is
    // out of range (states only an upload makes; ticked one by one).
    __device__ __forceinline__ uint32_t due(uint32_t lim) const
    {
        return (clock >= 228u || scanline >= 262u) ? 0u : tlim < lim ? tlim : lim;
    }

    // ------------------------------------------------------------ PIA timer (pia.rs:107-166)
    __device__ __forceinline__ void pia_tick(uint32_t n)
    {
        uint32_t tv = tp & 0xFFFFu, ps = tp >> 16, uf = su >> 16;
        pia_tick_n(tv, ps, su & 0xFFFFu, uf, n);
        tp = tv | (ps << 16);
        su = (su & 0xFFFFu) | (uf << 16);
    }

    // Headless consoles tick the timer once per instruction, with the
    // instruction's cycles (atari.rs:497-552).  Until a call makes the
    // decrement that brings the value to zero, or is made with the value at
    // zero, Pia::tick_n only counts, and consecutive calls add up: tick_n(a)
    // then tick_n(b) leaves what tick_n(a + b) leaves.  So an instruction
    // only takes its cycles off tlim, the cycles left before such a call;
    // the call that reaches it runs exactly through pia_tick, and the
    // counted cycles are folded into tp (pia_settle) before INTIM is
    // read, a PIA register is written or the state is stored.
    __device__ __forceinline__ uint32_t pia_span() const { return pia_span_of(tp & 0xFFFFu, tp >> 16, su & 0xFFFFu, su >> 16); }
    __device__ __forceinline__ uint2 pia_now() const { return pia_now_of(tp & 0xFFFFu, tp >> 16, su & 0xFFFFu, su >> 16, tlim); }
    // Fold the counted cycles in, run one exact call of n cycles (none for
    // n = 0), and open the next window.
    __device__ __forceinline__ void pia_sync(uint32_t n)
    {
        const uint4 r = pia_sync_io(tp, su, tlim, n);
        tp = r.x;
        su = r.y;
        tlim = r.z;
    }
    __device__ __forceinline__ void pia_settle() { pia_sync(0u); }
    // An INTIM read: the counted cycles settled, the underflow flag cleared.
    __device__ __forceinline__ void pia_intim()
    {
        const uint4 r = pia_intim_io(tp, su, tlim);
        tp = r.x; su = r.y; tlim = r.z;
    }
    __device__ __forceinline__ void pia_count(uint32_t n)
    {
        if (n < tlim) { tlim -= n; return; }
        // The call reaches the end of the window.  tick_n then underflows: uf
        // set, prescaler 0, and the o cycles past the window counted one per
        // cycle from $FF ($FF itself when o is 0).  That holds whatever the
        // state at the call when o > 0.  When o is 0 it needs a window that
        // began at tv = 0, or tv >= 2 at the call (with tv 1 and a prescaler
        // left, the call only empties the prescaler), which tlim > sel
        // guarantees.  Anything else runs exactly.
        const uint32_t sel = su & 0xFFFFu;
        if (tlim != 0u && (n > tlim || tlim > sel || (tp & 0xFFFFu) == 0u)) {
            const uint32_t o = n - tlim;
            const uint32_t tv = o ? (0u - o) & 0xFFu : 0xFFu;
            tp = tv;
            su = sel | 0x10000u;
            tlim = tv << (__ffs(sel) - 1u);
            return;
        }
        pia_sync(n);
    }

    // ------------------------------------------------------------ bus
    // Every access carries j, its cycle within the instruction: the
    // reference's CPU makes exactly one bus access per cycle (src/cpu.rs).
    // The headless console (atari.rs:497-552) ignores j: it ticks the TIA and
    // PIA once per instruction, after it.  The rendering console (RENDER,
    // atari.rs:195-222) ticks them up to cycle j before any access that
    // reaches a TIA or PIA register, whose state depends on the beam, and
    // gives writes the Bus's timing (two TIA clocks, the write, one TIA clock
    // and the PIA clock); accesses to ROM and RAM do not depend on the beam
    // and are ticked with the rest of the instruction.
    // Nothing here is a call in the headless console: a call costs some 50
    // cycles and, worse, makes ptxas spill values of the interpreter's loop.
    // The functions below serve exec(); run() has its own, narrower ones.
    __device__ __forceinline__ uint32_t io(uint32_t a, uint32_t j)   // TIA or PIA register read
    {
        if constexpr (RENDER) {
            if ((a & 0x1080u) == 0u) {
                const RRead r = render_read(a, 3u * (lag + j) + tl, rpack(), pins, pads, pv, fbp);
                runpack(r.s);
                lag = 0u - j;
                tl = 0;
                return r.v;
            }
            const uint32_t k = a & 7u;                                // Pia::read (pia.rs:169-199)
            if (k < 4u) {
                const uint32_t od = ports >> ((k & 2u) * 8u), ddr = (od >> 8) & 0xFFu, in = pins >> ((k & 2u) * 4u);
                return (k & 1u) ? ddr : ((in & ~ddr) | (od & ddr)) & 0xFFu;
            }
            if (k > 5u) return 0u;
            pia_to(j);
            if (k == 5u) return su >= 0x10000u ? 0x80u : 0u;
            su &= 0xFFFFu;                                            // an INTIM read clears the underflow flag
            return tp & 0xFFu;
        } else {
            if ((a & 0x87u) == 0x84u) {                             // INTIM: settles and clears the flag
                intim();
                return tp & 0xFFu;
            }
            if ((a & 0x8Eu) == 0x08u) sync();                       // INPT0, INPT1: the paddle counter
            return io_read(a, pcnt, pins, pads, ports, su, (const uint8_t*)column(), G->stride * 4u);
        }
    }
    __device__ __forceinline__ void io_write(uint32_t a, uint32_t v, uint32_t j)  // TIA or PIA register write
    {
        if constexpr (SLICED) f3_write(a, v);                       // the write still reaches the TIA
        if constexpr (RENDER) {
            if ((a & 0x1080u) != 0) {                                 // PIA register: rare, the general path
                pia_to(j);
                const uint4 q = pia_write_io(a, v, ports, tp & 0xFFFFu, tp >> 16, su);
                ports = q.x; tp = q.y | (q.z << 16); su = q.w;
            } else {
                const uint32_t t0 = tw;
                runpack(render_write(a, v, 3u * (lag + j) + tl + 2u, rpack(), pins, pv, fbp));
                lag = 0u - (j + 1u);
                tl = 1;
                if (((tw ^ t0) & 0xFFu) || wsync()) done = 0;         // VSYNC changed, or a wait: the frame loop looks
            }
        } else {
            sync();
            if (a & 0x200u) {
                const uint4 r = pia_store_io(a, v, ports, tp, su, tlim);
                ports = r.x; tp = r.y; su = r.z;
                rewindow(r.w);
            } else {
                const uint2 r = tia_write_io(a, v, clock, tw, scanline | (pcnt << 16), (uint8_t*)column(), G->stride * 4u);
                if ((r.x ^ tw) & (TW_WSYNC | 0xFFu)) dl = 0;          // a wait, or VSYNC changed: the frame loop looks
                tw = r.x; scanline = r.y & 0xFFFFu; pcnt = r.y >> 16;
            }
        }
    }
    // Headless, right after a sync: the timer has a new window.  A longer one
    // leaves dl early, which only makes the frame loop look once too often.
    __device__ __forceinline__ void rewindow(uint32_t w)
    {
        tlim = w;
        dl = w < dl ? w : dl;
    }
    __device__ __forceinline__ void intim()
    {
        sync();
        pia_intim();
        rewindow(tlim);
    }
    __device__ __forceinline__ uint32_t read_low(uint32_t a, uint32_t j)   // a < 0x1000
    {
        if ((a & 0x80u) && (a & 0x280u) != 0x280u) {                // RAM and its mirrors
            if constexpr (RENDER) return ldp(a & 0x7Fu);           // the rendering bus reads PIA RAM at every mirror
            else return a < 0x200u ? ldp(a & 0x7Fu) : 0u;           // other mirrors read the never-written flat array
        }
        return io(a, j);
    }
    __device__ __forceinline__ uint32_t read(uint32_t addr, uint32_t j)
    {
        uint32_t a = addr & 0x1FFFu;
        if (a & 0x1000u) {
            if constexpr (SLICED) {
                if constexpr (DPC) {
                    if (a < 0x1040u) return dpc(a, 0u, 0u);
                }
                e0_hot(a);
                if constexpr (FE) {
                    const uint32_t v = rom[srom(a)];
                    fe_note(a, v);
                    return v;
                }
                return rom[srom(a)];
            } else {
                bsw(a);
                return rom[bank | (a & 0xFFFu)];
            }
        }
        if constexpr (FE) {
            const uint32_t v = read_low(a, j);
            fe_note(a, v);
            return v;
        }
        return read_low(a, j);
    }
    __device__ __forceinline__ void write(uint32_t addr, uint32_t v, uint32_t j)
    {
        uint32_t a = addr & 0x1FFFu;
        if constexpr (FE) fe_note(a, v);
        if (a & 0x1000u) {
            if constexpr (SLICED) {
                if constexpr (DPC) {
                    if (a - 0x1040u < 0x40u) (void)dpc(a, v, 1u);
                }
                e0_hot(a);
            } else {
                bsw(a);
            }
            return;
        }
        if ((a & 0x280u) == 0x080u) { stp(a & 0x7Fu, v); return; }
        io_write(a, v, j);
    }
    // A phantom read: only its side effects (hotspot, INTIM) matter; in the FE
    // core its value too.
    __device__ __forceinline__ void dummy(uint32_t addr, uint32_t j)
    {
        if constexpr (FE) {
            (void)read(addr, j);
            return;
        }
        uint32_t a = addr & 0x1FFFu;
        if (a & 0x1000u) {
            if constexpr (SLICED) {
                if constexpr (DPC) {
                    if (a < 0x1040u) (void)dpc(a, 0u, 0u);
                }
                e0_hot(a);
            } else {
                bsw(a);
            }
        } else if ((a & 0x287u) == 0x284u) {
            if constexpr (RENDER) (void)io(a, j);
            else intim();
        }
    }
    __device__ __forceinline__ uint32_t zp_read(uint32_t z, uint32_t j)
    {
        if constexpr (FE) {
            const uint32_t v = (z & 0x80u) ? ldp(z & 0x7Fu) : io(z, j);
            fe_note(z, v);
            return v;
        }
        return (z & 0x80u) ? ldp(z & 0x7Fu) : io(z, j);
    }
    __device__ __forceinline__ void push(uint32_t sp, uint32_t v, uint32_t j)
    {
        if constexpr (FE) fe_note(0x100u | sp, v);
        if (sp & 0x80u) stp(sp & 0x7Fu, v); else io_write(0x100u | sp, v, j);
    }
    __device__ __forceinline__ uint32_t pull(uint32_t sp, uint32_t j)
    {
        const uint32_t v = (sp & 0x80u) ? ldp(sp & 0x7Fu) : io(0x100u | sp, j);   // page 1 below $180 is TIA
        if constexpr (FE) fe_note(0x100u | sp, v);
        return v;
    }
    // Read-modify-write's two writes, on cycles j and j+1; a RAM target only
    // needs the second.
    __device__ __forceinline__ void rmw_store(uint32_t ea, uint32_t oldv, uint32_t newv, uint32_t j)
    {
        uint32_t a = ea & 0x1FFFu;
        if constexpr (!FE) {                                          // FE: the first write is an access too
            if ((a & 0x1280u) == 0x080u) { stp(a & 0x7Fu, newv); return; }
        }
#pragma unroll 1
        for (uint32_t m = 0; m < 2u; m++) write(ea, m ? newv : oldv, j + m);
    }

    // ------------------------------------------------------------ instructions
    // Instruction bytes at a0..a0+2 (13-bit) can be read together (FE: once the
    // opcode is, which an access to $01FE before it lets select the bank): they lie in
    // the current bank (E0, 3F: in one window) and below every hotspot
    // (and, DPC, above its read registers at $1000-$103F), so reading them has
    // no side effect.  The few bytes past the hotspots hold vectors.
    __device__ __forceinline__ bool code_ok() const
    {
        const int32_t s = (int32_t)(pc << 19);                         // ROM addresses are negative, in order
        if constexpr (DPC) return (uint32_t)s - (0x1040u << 19) < ((0x1FF6u - 0x1040u) << 19);
        else if constexpr (FE) return s < (int32_t)(0x1FFEu << 19);
        else if constexpr (SLICED) return (s < (int32_t)(0x1FDEu << 19)) & ((pc & 0x3FEu) != 0x3FEu);
        else return s < lim;
    }
    // ROM data at ea, below every hotspot: a load without a side effect
    // (wr, T_WR or 0: and no write).
    __device__ __forceinline__ bool data_ok(uint32_t ea, uint32_t wr = 0u) const
    {
        const int32_t s = (int32_t)((ea << 19) & ~(wr & T_WR));         // ROM addresses are negative, in order
        if constexpr (DPC) return (uint32_t)s - (0x1040u << 19) < ((0x1FF8u - 0x1040u) << 19);
        else if constexpr (FE) return s < 0;
        else if constexpr (SLICED) return s < (int32_t)(0x1FE0u << 19);
        else return s < lim;
    }
    __device__ __forceinline__ uint32_t rom_at(uint32_t a) const { return SLICED ? srom(a) : bank | (a & 0xFFFu); }

    // Executes instructions until one that may leave the lanes of a group at
    // different pcs, one that reaches wait_key, or the end of the lane's
    // frames.  After an instruction that the frame loop must look at (el
    // reaches dl; RENDER: cyc_acc reaches done), look(cycles) does, and says
    // whether the lane goes on: in the loop, since lanes are due at different
    // times, and one that left would part from its group.  Returns 0 for an
    // illegal opcode (pc is then past it and nothing else changed: the
    // reference panics right after the opcode fetch, src/cpu.rs:1139-1141).
    //
    // What bounds it.  A lone warp on a scheduler: the dependent chain of
    // three shared loads (23 cycles each: opcode, table, data) and some 25
    // operations (5 each), and 11 cycles for every branch.  A full SM: the
    // issue of its instructions, as long as the code in use stays within the
    // 32 KB that the SM's instruction cache holds (2.5 times slower beyond).
    // So operations, registers and flags are selected by the table's words
    // instead of a switch (150 cycles for a lone warp), the loads are issued
    // whatever the opcode needs (always from this lane's RAM or the ROM
    // image), the frequent exceptions sit behind two tests, and the rest
    // (exec) apart.  Measured on one B200, before (a switch decoder with the
    // time kept per instruction) and now: 165 and 107 warp instructions, 1,290
    // and 450 cycles per guest instruction of a lone warp; a frame of one
    // plain cart 3.47 and 1.25 ms; the mixed batch of 135,500 consoles x 4
    // frames 22.4 and 13.2 ms; a frame of 50,000 divergence carts 7.2 and 3.1 ms.
    // Loading the next instruction's bytes and words while this one executes
    // gained nothing (1.24 and 1.26 ms): the warp waits on the operations.
    template <class LOOK>
    __device__ __forceinline__ uint32_t run(uint32_t wait_key, LOOK look)
    {
        const sptr tab = to_sptr(op_table()), rs = RENDER ? to_sptr(rom) : kept(to_sptr(rom)),
                   ps = RENDER ? to_sptr(pv) : kept(to_sptr(pv));
        uint32_t n;
        const uint32_t end = instr + FA_BURST;
#pragma unroll 1
        do {
            // Out of the window the loads stay inside the image: rom_at masks
            // the offset, and the image is followed by other shared memory.
            const bool ok = code_ok();
            sptr q = rs + rom_at(pc);
            const uint32_t op = lds8(q), slices0 = FE ? slices : 0u;
            if constexpr (FE) {
                if (ok & ((slices & 0x80u) != 0u)) { fe_note(pc & 0x1FFFu, op); q = rs + rom_at(pc); }
            }
            const uint32_t b1 = lds8(q + 1), b2 = lds8(q + 2);
            OpWord w = ldw(tab, op);
            const uint32_t f = w.ix;
            const uint32_t pc1 = pc + high<!RENDER>(tab, op, H_LEN, w.rd);            // may pass $FFFF: not ok then
            uint32_t base = __byte_perm(b1, b2, w.bs);
            n = high<!RENDER>(tab, op, H_CYC, w.rs);
            if (!ok | ((f & T_CTRL) != 0u)) {
                if (!ok) goto exec_;
                if (f & T_BR) {
                    const bool tk = ((F & w.am) != 0u) != ((f & T_BI) != 0u);
                    const uint32_t to = pc1 + (uint32_t)(int32_t)(int8_t)(uint8_t)b1;
                    if (tk) n = 3u;
                    if (tk & (((pc1 ^ to) & 0xFF00u) != 0u)) {        // the phantom read at the unfixed address
                        if (!data_ok((pc1 & 0xFF00u) | (to & 0xFFu))) goto exec_;
                        n = 4u;
                    }
                    pc = tk ? to : pc1;
                    if (parted(tk) | ((int32_t)(instr - end) >= 0)) wait_key = 0u;   // leaves the loop
                    goto done_;
                }
                if (f & T_MEM) {
                    // Through a zero-page pointer in RAM: its two bytes, then as
                    // the absolute forms ((zp,X): no index left).
                    const uint32_t z = (w.qs & (T_INDY << 16)) ? b1 : (b1 + ((R >> 8) & 0xFFu)) & 0xFFu;
                    if (z - 0x80u >= 0x7Fu) goto exec_;
                    base = lds8(ps + poff(z & 0x7Fu)) | (lds8(ps + poff((z + 1u) & 0x7Fu)) << 8);
                } else {
                    const uint32_t o = (w.qs >> 16) & 63u;
                    if (o == OP_JMP) { pc = b1 | (b2 << 8); goto done_; }
                    uint32_t sp = R >> 24;
                    if (o <= OP_JSR) {                                // PHP, PHA, JSR
                        if (sp < 0x81u) goto exec_;
                        const uint32_t u = o == OP_PHA ? R : o == OP_JSR ? (pc1 >> 8) : get_p() | F_B | F_U;
                        if constexpr (FE) {
                            if (o == OP_JSR) fe_note(0x100u | sp, lds8(ps + poff(sp & 0x7Fu)));   // JSR reads the stack first
                            fe_note(0x100u | sp, u & 0xFFu);
                        }
                        sts8(ps + poff(sp & 0x7Fu), u);
                        sp--;
                        pc = pc1;
                        if (o == OP_JSR) {
                            sts8(ps + poff(sp & 0x7Fu), pc1);
                            uint32_t hi = b2;
                            if constexpr (FE) {
                                fe_note(0x100u | sp, pc1 & 0xFFu);
                                hi = lds8(rs + rom_at(pc1));          // its high byte comes last
                                fe_note(pc1 & 0x1FFFu, hi);
                            }
                            sp--;
                            pc = b1 | (hi << 8);
                        }
                    } else if (o >= OP_PLP && o <= OP_RTS) {
                        if (sp - 0x7Fu >= (o == OP_RTS ? 0x7Fu : 0x80u) || (FE && sp < 0x80u)) goto exec_;
                        const uint32_t u = lds8(ps + poff((sp + 1u) & 0x7Fu));
                        if (o == OP_RTS) {
                            const uint32_t ra = u | (lds8(ps + poff((sp + 2u) & 0x7Fu)) << 8);
                            if (!data_ok(ra)) goto exec_;             // its phantom read
                            if constexpr (FE) {
                                fe_note(0x100u | sp, lds8(ps + poff(sp & 0x7Fu)));
                                fe_note(0x101u + sp, u);
                                fe_note(0x102u + sp, ra >> 8);
                                fe_note(ra & 0x1FFFu, lds8(rs + rom_at(ra)));
                            }
                            sp++;
                            pc = ra + 1u;
                            wait_key = 0u;
                        } else {
                            if constexpr (FE) {
                                fe_note(0x100u | sp, lds8(ps + poff(sp & 0x7Fu)));
                                fe_note(0x101u + sp, u);
                            }
                            pc = pc1;
                            if (o == OP_PLA) { R = (R & ~0xFFu) | u; set_nz(u); }
                            else set_p(u & ~(F_B | F_U));
                        }
                        sp++;
                    } else {
                        goto exec_;
                    }
                    R = (R & 0xFFFFFFu) | (sp << 24);
                    goto done_;
                }
            }
            {
                bool wr = (f & T_WR) != 0u;
                const uint32_t ea = (base + __byte_perm(R, 0x80u, f)) & w.am;
                const bool ram = ((ea & 0x1E80u) == 0x80u) & !(FE && (ea & 0x1FFFu) == 0x1FEu);
                const sptr pr = ps + poff(ea & 0x7Fu), po = rs + rom_at(ea);
                uint32_t ld = lds8(ram ? pr : po);
                uint32_t wm = high<!RENDER>(tab, op, H_M, w.bs), wk = high<!RENDER>(tab, op, H_K, w.fs),
                         wx = high<!RENDER>(tab, op, H_X, w.am);
                const bool plain = ram | data_ok(ea, f);
                const bool far = ((base ^ ea) & 0xFF00u) != 0u;       // a page crossed
                if (!plain | far | ((f & (pd | (T_ODD | T_FIX))) != 0u)) {
                    const uint32_t o = (w.qs >> 16) & 63u;
                    if (far | ((f & T_FIX) != 0u)) {
                        // A fix-up read, at the base's page.  With the access
                        // itself in plain ROM or RAM it is harmless unless that
                        // page is $0F (the PIA's mirror), $1F (hotspots; an access
                        // that wraps around) or, DPC, $10 (its registers).
                        if (((base & 0xF00u) == 0xF00u) | (DPC && ((base & 0x1F00u) | (ea & 0xFFu)) - 0x1000u < 0x40u)) goto exec_;
                        if (!plain & ((base & (FE ? 0x300u : 0x200u)) != 0u)) goto exec_;
                        if (!(f & T_FIX)) n++;
                    }
                    if (!plain) {
                        // ROM (a write, or a hotspot) or a register.
                        const uint32_t a = ea & 0x1FFFu;
                        const bool rmw = wr & (o < OP_STA);
                        if constexpr (FE) {
                            if (a == 0x1FEu) {                        // RAM, and the next access selects the bank
                                if (rmw | ((f & (pd | T_ODD)) != 0u)) goto exec_;
                                slices |= 0x80u;
                                ld = lds8(pr);
                                if (wr) sts8(pr, alu(w, ld, b1));
                                commit(w, alu(w, ld, b1));
                                pc = pc1;
                                goto done_;
                            }
                        }
                        if (!RENDER && (a & 0x1287u) == 0x284u && !intim_quick()) goto exec_;
                        // A DPC register: a read of $1000-$103F or a write to $1040-$107F.
                        if (DPC && rmw && a - 0x1000u < 0x80u) goto exec_;
                        const bool reg = DPC && a - 0x1000u - (wr ? 0x40u : 0u) < 0x40u;
                        if (reg) {
                            ld = dpc(a, __byte_perm(R, 0u, w.rs), wr ? 1u : 0u);
                            if (wr) { pc = pc1; goto done_; }
                        } else if (!wr | rmw) {
                            const uint32_t j = n - (rmw ? 3u : 1u);
                            if (a & 0x1000u) {
                                hot(a);
                                ld = lds8(rs + rom_at(ea));
                            } else {
                                ld = bus_read(a, j);
                            }
                        }
                        if (wr) {
                            uint32_t r = __byte_perm(R, 0u, w.rs);
                            if (rmw) {
                                r = (f & T_ODD) ? shift(w, o, ld) : alu(w, ld, b1);
                                F = __byte_perm(F, r, (f & T_ODD) ? 0x3574u : w.fs);
                            }
#pragma unroll 1
                            for (uint32_t m = rmw ? 0u : 1u; m < 2u; m++) {
                                const uint32_t u = (m ? r : ld) & 0xFFu;
                                if (a & 0x1000u) {
                                    hot(a);
                                } else {
                                    bus_write(a, u, n - 2u + m);
                                }
                            }
                            pc = pc1;
                            goto done_;
                        }
                    }
                    if constexpr (RENDER) {                           // not kept in registers across the pixel code's calls
                        w = ldw(tab, op);
                        wm = w.bs >> 16; wk = w.fs >> 16; wx = w.am >> 16;
                    }
                    if (f & (pd | T_ODD)) {
                        odd_op(w, o, ld, b1, pr, wr);
                        wr = false;
                        w.rd = w.fs = 0x3210u;                        // completed: nothing changes below
                    }
                }
                const uint32_t r = alu(w, ld, b1, wm, wk, wx);
                if (wr) sts8(pr, r);
                commit(w, r);
                pc = pc1;
                goto done_;
            }
        exec_:
            if constexpr (FE) slices = slices0;                       // as before the opcode fetch
            n = exec();
            if (n == 0u) return 0u;
            if (!ok | ((f & T_CTL) != 0u)) wait_key = 0u;
        done_:
            instr++;
            if constexpr (RENDER) {
                lag += n;
                plag += n;
                cyc_acc += n;
            } else {
                el += n;
            }
            if (RENDER ? cyc_acc >= done : el >= dl) {
                if (!look(n)) break;
            }
        } while ((kb | pc) < wait_key);
        return 1u;
    }

    // The result of a table word's operation (byte 0), its carry (byte 1) and
    // its V (bit 7 of byte 2): k (s ^ v) + m (s & v) + q.  k is 1 but for AND;
    // m = 2 adds (SBC and compares a v that x inverts), 1 ORs and ANDs, 0 XORs;
    // s = 0 loads, v = 0 moves.  Multiplies: the ALU pipe is the busy one.
    __device__ __forceinline__ uint32_t alu(const OpWord& w, uint32_t ld, uint32_t b1, uint32_t m, uint32_t k, uint32_t x) const
    {
        const uint32_t s = __byte_perm(R, 0u, w.rs), v = __byte_perm(ld, b1, w.xs) ^ x;
        const uint32_t q = __byte_perm(F, 0xFF01u, w.qs);
        const uint32_t r = (s & v) * m + ((s ^ v) * k + q);
        return __byte_perm(r, (s ^ r) & (v ^ r), 0x3410u);
    }
    __device__ __forceinline__ uint32_t alu(const OpWord& w, uint32_t ld, uint32_t b1) const
    {
        return alu(w, ld, b1, w.bs >> 16, w.fs >> 16, w.am >> 16);
    }
    __device__ __forceinline__ void commit(const OpWord& w, uint32_t r)
    {
        R = __byte_perm(R, r, w.rd);
        F = __byte_perm(F, r, w.fs);
    }

    // ASL, ROL, LSR, ROR of u: the result (byte 0) and its carry (byte 1).
    __device__ __forceinline__ uint32_t shift(const OpWord& w, uint32_t o, uint32_t u) const
    {
        const uint32_t q = __byte_perm(F, 0xFF01u, w.qs);
        return o <= OP_ROL ? (u << 1) | q : (u >> 1) | (q << 7) | ((u & 1u) << 8);
    }

    // Decimal ADC and SBC, and the T_ODD operations on A, RAM at pr (shifts
    // that write) or the operand.
    __device__ __forceinline__ void odd_op(const OpWord& w, uint32_t o, uint32_t ld, uint32_t b1, sptr pr, bool mem)
    {
        if (o == OP_ADC || o == OP_SBC) {
            const uint32_t v = __byte_perm(ld, b1, w.xs), c = (F >> 16) & 1u;
            const uint4 r = decimal_op(o == OP_SBC, R & 0xFFu, v, c);
            R = (R & ~0xFFu) | r.x;
            F = r.y | (r.z << 16) | ((r.w & 0x80u) << 24);
        } else if (o >= OP_ASL && o <= OP_ROR) {
            const uint32_t r = shift(w, o, mem ? ld : R & 0xFFu);
            F = __byte_perm(F, r, 0x3574u);
            if (mem) sts8(pr, r);
            else R = __byte_perm(R, r, 0x3214u);
        } else if (o == OP_BIT) {
            set_nz((R & ld & 0xFFu) | ((ld & 0x80u) << 8));
            setv(ld << 1);
        } else if (o == OP_CLV) {
            setv(0u);
        } else if (o <= OP_SEI) {
            p = o == OP_SEI ? p | F_I : p & ~F_I;
        } else {
            pd = o == OP_SED ? T_UV : 0u;
        }
    }

    // Whether the lanes running this branch together part on it.  The lanes
    // that read a mask are those it names, and each goes on to the vote with
    // it: one statement, so that nothing comes between and no lane of the mask
    // stays away.  Which lanes run together here is not promised: how soon the
    // scheduler is asked depends on it, never a result.
    __device__ __forceinline__ static bool parted(bool tk)
    {
#ifdef __CUDA_ARCH__
        uint32_t am, tb;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.u32 p, %2, 0;\n\t"
            "activemask.b32 %0;\n\t"
            "vote.sync.ballot.b32 %1, p, %0;\n\t}"
            : "=&r"(am), "=r"(tb)
            : "r"((uint32_t)tk));
        return (tb != 0u) & (tb != am);
#else
        (void)tk;
        return true;
#endif
    }

    // Headless: the timer is counting down with its underflow flag clear, so
    // that an INTIM read changes nothing.
    __device__ __forceinline__ bool intim_quick() const
    {
        return (su < 0x10000u) & (tlim != 0u) & ((tp & 0xFFFFu) != 0u);
    }
    // A read of a TIA or PIA register, or of a RAM mirror, at a < $1000
    // outside $80-$FF and $180-$1FF (headless INTIM only if intim_quick).
    __device__ __forceinline__ uint32_t bus_read(uint32_t a, uint32_t j)
    {
        if constexpr (RENDER) {
            return read_low(a, j);
        } else {
            if (a & 0x80u) {
                if (!(a & 0x200u)) return 0u;                        // never-written flat array
                const uint32_t k = a & 7u;
                // INTIM while the timer counts down: its value is that of the
                // cycles left in the window (whole intervals and the prescaler).
                if (k == 4u) return ((tlim - el - 1u) >> (__ffs(su) - 1)) + 1u;
                if (k >= 4u) return k == 5u && su >= 0x10000u ? 0x80u : 0u;   // INSTAT
                const uint32_t od = ports >> ((k & 2u) * 8u), ddr = (od >> 8) & 0xFFu;
                const uint32_t in = pins >> ((k & 2u) * 4u);
                return (k & 1u) ? ddr : ((in & ~ddr) | (od & ddr)) & 0xFFu;
            }
            const uint32_t r = a & 0x0Fu;
            if (r < 8u) return (tw & TW_CX) ? ((const uint8_t*)column())[cold_off(PB_CX + r, grp()->stride * 4u)] : 0u;
            if (r >= 12u) return ((pins >> (16u + (r & 1u))) & 1u) & (r < 14u ? 1u : 0u) ? 0x80u : 0u;
            if (r >= 10u) return 0x80u;
            sync();                                                  // INPT0, INPT1: the paddle counter
            return pcnt >= ((pads >> (8u * (r & 1u))) & 0xFFu) ? 0x80u : 0u;
        }
    }
    // A write at a < $1000 outside $80-$FF and $180-$1FF.
    __device__ __forceinline__ void bus_write(uint32_t a, uint32_t v, uint32_t j)
    {
        if ((a & 0x280u) == 0x80u) { stp(a & 0x7Fu, v); return; }     // RAM mirrors
        if constexpr (!RENDER) {
            if (!(a & 0x200u)) {
                const uint32_t r = a & 0x3Fu, e = tia_table()[r];
                if (r == 2u) {                                        // WSYNC: the frame loop looks
                    if constexpr (SLICED) f3_write(a, v);
                    tw |= TW_WSYNC;
                    dl = 0;
                    return;
                }
                if (e) {                                              // a register that only keeps bits of v
                    if constexpr (SLICED) f3_write(a, v);
                    ((uint8_t*)column())[cold_off(e & 0xFFu, grp()->stride * 4u)] = (uint8_t)((v >> ((e >> 8) & 0xFFu)) & (e >> 16));
                    return;
                }
            }
        }
        io_write(a, v, j);
    }

    // One instruction with every access on the bus, whatever it is.  What run()
    // needs it for is rare: code near a hotspot or outside ROM, stacks and
    // pointers that reach the TIA, phantom reads that may have side effects,
    // BRK, RTI, JMP (ind), illegal opcodes.  It is inlined: as a call it cost
    // the loop 30 registers' spills (a state in memory, and an ABI).
    __device__ __forceinline__ uint32_t exec()
    {
        pc &= 0xFFFFu;
        uint32_t b1, b2;
        OpWord w;
        if (code_ok() && !(FE && (slices & 0x80u))) {
            const uint8_t* q = rom + rom_at(pc);
            w = op_table()[q[0]];
            b1 = q[1];
            b2 = q[2];
        } else {
            fetch(b1, b2, w);
        }
        const uint32_t f = w.ix, o = (w.qs >> 16) & 63u;
        if ((f & T_CTRL) && !(f & T_MEM)) return control(w, o, b1, b2);
        pc = (pc + (w.rd >> 16)) & 0xFFFFu;
        uint32_t n = w.rs >> 16, ld = 0;
        if (f & T_MEM) {
            uint32_t base = __byte_perm(b1, b2, w.bs);
            if (w.qs & (T_IND << 16)) {
                // (zp,X): the pointer at zp b1 + X, read on cycles 3-4; (zp),Y: at
                // zp b1, on cycles 2-3.
                const bool iy = (w.qs & (T_INDY << 16)) != 0u;
                const uint32_t z = iy ? b1 : b1 + ((R >> 8) & 0xFFu), j0 = iy ? 2u : 3u;
                if constexpr (FE) {
                    if (!iy) dummy(b1, 2);                            // the base, before X is added
                }
                base = 0;
#pragma unroll 1
                for (uint32_t m = 0; m < 2u; m++) base |= zp_read((z + m) & 0xFFu, j0 + m) << (8u * m);
            }
            const uint32_t ea = (base + __byte_perm(R, 0x80u, f)) & w.am & 0xFFFFu;
            const bool far = ((base ^ ea) & 0xFF00u) != 0u;
            if (far && !(f & T_FIX)) n++;
            if constexpr (FE) {
                if (!(w.am & 0x100u) && (f & 7u) != 5u) dummy(b1, 2);   // zp,X / zp,Y: the base, before the index
            }
            const bool wr = (f & T_WR) != 0u, rmw = wr && o < OP_STA;
            const uint32_t j = n - (rmw ? 3u : 1u);                   // the access's cycle, the fix-up read before it
            if (far || (f & T_FIX)) dummy((base & 0xFF00u) | (ea & 0xFFu), j - 1u);
            if (wr && !rmw) {
                write(ea, __byte_perm(R, 0u, w.rs), j);
                return n;
            }
            ld = read(ea, j);
            if (rmw) {
                uint32_t r;
                r = (f & T_ODD) ? shift(w, o, ld) : alu(w, ld, b1);
                F = __byte_perm(F, r, (f & T_ODD) ? 0x3574u : w.fs);
                r &= 0xFFu;
                rmw_store(ea, ld, r, n - 2u);
                return n;
            }
        }
        if (f & (pd | T_ODD)) odd_op(w, o, ld, b1, sptr(), false);
        else commit(w, alu(w, ld, b1));
        return n;
    }

    // The instruction's bytes one bus access at a time: code near a hotspot,
    // outside ROM, or (FE) after an access to $01FE.
    __device__ __forceinline__ void fetch(uint32_t& b1, uint32_t& b2, OpWord& w)
    {
        uint32_t n = 1u, u = 0u;
#pragma unroll 1
        for (uint32_t k = 0; k < n; k++) {
            const uint32_t v = read((pc + k) & 0xFFFFu, k);
            if (k == 0u) {
                w = op_table()[v];
                if (((w.qs >> 16) & 63u) != OP_ILL) n = (w.rd >> 16) == 3u ? 3u : 2u;
            } else {
                u |= v << (8u * (k - 1u));
            }
        }
        b1 = u & 0xFFu;
        b2 = u >> 8;
        if (n != 3u) b2 |= 0x100u;                                    // JSR: not read yet
    }

    // Branches, stack and jumps.  Bus-access sites are shared (one push loop,
    // one pull loop, one read loop for the new pc's bytes): every site is
    // inlined code, and the code should fit the instruction cache.
    __device__ __forceinline__ uint32_t control(const OpWord& w, uint32_t o, uint32_t b1, uint32_t b2)
    {
        uint32_t n = w.rs >> 16;
        pc = (pc + (w.rd >> 16)) & 0xFFFFu;
        if (w.ix & T_BR) {
            if (((F & w.am) != 0u) == ((w.ix & T_BI) != 0u)) return n;   // not taken
            const uint32_t to = (pc + (uint32_t)(int32_t)(int8_t)(uint8_t)b1) & 0xFFFFu;
            n = 3;
            const bool far = ((pc ^ to) & 0xFF00u) != 0u;
            // The phantom read of the next opcode, and a far branch's at the
            // unfixed address; in plain ROM neither has a side effect.
            if (!code_ok()) dummy(pc, 2);
            if (far) { dummy((pc & 0xFF00u) | (to & 0xFFu), 3); n = 4; }
            pc = to;
            return n;
        }
        if (o == OP_ILL) return 0u;
        if (o == OP_JMP) { pc = (b1 | (b2 << 8)) & 0xFFFFu; return n; }
        uint32_t vb, vn, vs = 0u, vj, vv = 0u;
        if (o == OP_JMPI) {                                           // page-wrap bug
            vb = (b1 | (b2 << 8)) & 0xFFFFu; vn = 2u; vj = 3u;
        } else {
            uint32_t sp = R >> 24;
            if (o <= OP_BRK) {                                        // PHP, PHA, JSR, BRK
                // BRK (b1 is the padding byte) pushes pch, pcl, p on cycles 2-4;
                // JSR pushes pch, pcl on cycles 3-4, before it reads its high byte.
                const uint32_t u = o == OP_PHA ? R : o == OP_JSR ? pc : (pc << 8) | get_p() | F_B | F_U;
                const uint32_t m = o == OP_JSR ? 2u : o == OP_BRK ? 3u : 1u, j0 = o == OP_JSR ? 3u : 2u;
                if constexpr (FE) {
                    if (o == OP_JSR) dummy(0x100u | sp, 2);           // JSR reads the stack before its pushes
                }
#pragma unroll 1
                for (uint32_t k = m; k-- > 0u;) {
                    push(sp, (u >> (8u * k)) & 0xFFu, j0 + m - 1u - k);
                    sp = (sp - 1u) & 0xFFu;
                }
                R = (R & 0xFFFFFFu) | (sp << 24);
                if (o < OP_JSR) return n;
                if (o == OP_JSR) {
                    if (!FE && b2 < 0x100u) { pc = b1 | (b2 << 8); return n; }
                    vb = pc; vn = 1u; vs = 8u; vv = b1;
                } else {
                    p |= F_I;
                    vb = 0xFFFEu; vn = 2u;
                }
                vj = 5u;
            } else {                                                  // PLP, PLA, RTS, RTI
                const uint32_t m = o == OP_RTI ? 3u : o == OP_RTS ? 2u : 1u;
                uint32_t u = 0;
                if constexpr (FE) dummy(0x100u | sp, 2);              // the stack, before the pulls
#pragma unroll 1
                for (uint32_t k = 0; k < m; k++) {
                    sp = (sp + 1u) & 0xFFu;
                    u |= pull(sp, 3u + k) << (8u * k);
                }
                R = (R & 0xFFFFFFu) | (sp << 24);
                if (o == OP_PLA) {
                    R = (R & ~0xFFu) | u;
                    set_nz(u);
                } else if (o == OP_RTS) {
                    dummy(u, 5);
                    pc = (u + 1u) & 0xFFFFu;
                } else {
                    set_p(u & ~(F_B | F_U));
                    if (o == OP_RTI) pc = (u >> 8) & 0xFFFFu;
                }
                return n;
            }
        }
#pragma unroll 1
        for (uint32_t m = 0; m < vn; m++) vv |= read((vb & 0xFF00u) | ((vb + m) & 0xFFu), vj + m) << (vs + 8u * m);
        pc = vv;
        return n;
    }

    // ------------------------------------------------------------ rendering console
    // Used only by RENDER instantiations.  The pixel-accurate Tia of the
    // reference's rendering console (src/tia.rs) and Pia::tick run out of
    // line (render_clocks, render_write, render_read, render_observe and
    // r_pia_ticks, above), on the state they touch passed by value: one copy of
    // the pixel pipeline however many bus-access sites the interpreter has.
    uint32_t done;            // instruction cycles of the frame (cyc_acc) at which the frame loop must look
    uint32_t lag;             // CPU cycles not yet given to the TIA; within an instruction, up to its start
                             // (negative: they have reached cycle -lag of it)
    uint32_t tl;              // and TIA clocks (0 or 1: the one after a register write) before those
    uint32_t plag;            // CPU cycles not yet given to the PIA, likewise
    uint32_t vtop;            // visible_top | vblank_top << 16
    uint8_t* fbp;             // this instance's framebuffer, 160 x 192 palette indices
    uint32_t sc, zr;          // framebuffer sector in the sector buffer; rows written since the clear point | R_ZPEND
    uint32_t rx;              // the current line's pixels are drawn up to this TIA clock

    __device__ __forceinline__ RState rpack() const
    {
        RState r;
        r.clock = clock; r.scanline = scanline; r.tw = tw; r.pcnt = pcnt; r.vtop = vtop;
        r.sc = sc; r.zr = zr; r.rx = rx;
        return r;
    }
    __device__ __forceinline__ void runpack(const RState& r)
    {
        clock = r.clock; scanline = r.scanline; tw = r.tw; pcnt = r.pcnt; vtop = r.vtop;
        sc = r.sc; zr = r.zr; rx = r.rx;
    }
    // The TIA is advanced only before an access that observes or changes it:
    // the cycles of instructions that touch only ROM and RAM are owed (lag)
    // and given in one piece, with the clocks of the access before.  So is the
    // PIA, before the accesses that see or set its timer.
    __device__ __forceinline__ void rcycles(uint32_t n)              // of a WSYNC wait, nothing owed
    {
        runpack(render_clocks(rpack(), 3u * n, pins, pv, fbp));
        plag += n;
    }
    __device__ __forceinline__ void settle()
    {
        const uint32_t n = 3u * lag + tl;
        if (n) { runpack(render_clocks(rpack(), n, pins, pv, fbp)); lag = 0; tl = 0; }
    }
    __device__ __forceinline__ void pia_to(uint32_t j)               // the PIA up to cycle j of the instruction
    {
        const uint2 r = r_pia_ticks(tp, su, plag + j);
        tp = r.x; su = r.y;
        plag = 0u - j;
    }
    // The owed cycles, the pixels up to the beam, and the framebuffer as it
    // can be seen now (the end of a frame or of a call).
    __device__ __forceinline__ void fb_observe()
    {
        settle();
        pia_to(0u);
        runpack(render_observe(rpack(), pv, fbp));
    }
    // The sector buffer at the start of a call: the sector where the beam's
    // row has been drawn to, as the last call left it in the framebuffer.
    __device__ __forceinline__ void fb_resume()
    {
        const uint32_t vis = (scanline - (vtop & 0xFFFFu)) & 0xFFFFu;
        zr = vis < FA_FB_H ? vis : FA_FB_H;
        if (vis < FA_FB_H) {
            const uint32_t x = (rx > 68u ? rx : 68u) - 68u;
            sc = vis * (FA_FB_W / 32u) + ((x >> 5) < 4u ? (x >> 5) : 4u);
            const uint4* q = (const uint4*)(fbp + (size_t)sc * 32u);
            const uint4 u0 = q[0], u1 = q[1];
            *r_sbuf(pv, 0) = u0.x; *r_sbuf(pv, 1) = u0.y; *r_sbuf(pv, 2) = u0.z; *r_sbuf(pv, 3) = u0.w;
            *r_sbuf(pv, 4) = u1.x; *r_sbuf(pv, 5) = u1.y; *r_sbuf(pv, 6) = u1.z; *r_sbuf(pv, 7) = u1.w;
        } else {
            sc = 0;
            r_sec_clear(pv);
        }
    }

    // HeadlessAtari::set_action (src/atari.rs:571-582).
    __device__ __forceinline__ void apply_action(uint32_t act)
    {
        uint32_t t = c_action_table[act < 18u ? act : 0u];
        pins = (pins & ~0x100FFu) | (t & 0xFFu) | (((t >> 8) & 1u) << 16);
        pads = (pads & ~0xFFu) | ((t >> 16) & 0xFFu);
    }

    // ------------------------------------------------------------ state movement
    __device__ __forceinline__ void load_hot(const uint32_t* col, uint32_t stride)
    {
        uint32_t w;
        R = col[R_AXYS * stride];
        w = col[R_PC * stride];    pc = w & 0xFFFF; set_p((w >> 16) & 0xFF); bank = (w >> 24) << 12;
        cyc_acc = 0; el = 0; tl = 0; plag = 0;
        const uint32_t p0 = col[R_PIA0 * stride];                  // pa_out pa_ddr pa_in pb_out
        const uint32_t p1 = col[R_PIA1 * stride];                  // pb_ddr pb_in uf pdump
        ports = (p0 & 0xFFFFu) | ((p0 >> 24) << 16) | ((p1 & 0xFFu) << 24);
        tp = col[R_TIMER * stride];
        w = col[R_SELPC * stride]; su = (w & 0xFFFFu) | (((p1 >> 16) & 0xFFu) << 16); pcnt = w >> 16;
        tlim = RENDER ? 0u : pia_span();
        lim = kept((int32_t)((hot_lo - 2u) << 19));
        w = col[R_TIA0 * stride];  clock = w & 0xFFFF; scanline = w >> 16;
        w = col[R_TIA1 * stride];                                   // wsync fcomp vsync vblank
        tw = ((w >> 16) & 0xFFFFu) | ((w & 1u) << 16) | (((w >> 8) & 1u) << 17) | (((p1 >> 24) & 1u) << 18);
        if constexpr (!RENDER) {
            if (col[(PB_CX / 4u) * stride] | col[(PB_CX / 4u + 1u) * stride]) tw |= TW_CX;
        }
        if constexpr (SLICED) slices = slices_of(fa_tia1_mapper(w));
        w = col[R_TIA2 * stride];                                   // inpt4 inpt5 pad0 pad1
        pins = ((p0 >> 16) & 0xFFu) | (((p1 >> 8) & 0xFFu) << 8) | ((w & 1u) << 16) | (((w >> 8) & 1u) << 17);
        pads = w >> 16;
    }
    __device__ __forceinline__ void store_hot(uint32_t* col, uint32_t stride) const
    {
        col[R_AXYS * stride] = R;
        // pc is masked where an instruction starts: the last one may have left it past $FFFF.
        col[R_PC * stride] = (pc & 0xFFFFu) | (get_p() << 16) | ((bank >> 12) << 24);
        col[R_PIA0 * stride] = (ports & 0xFFFFu) | ((pins & 0xFFu) << 16) | (((ports >> 16) & 0xFFu) << 24);
        col[R_PIA1 * stride] = (ports >> 24) | (((pins >> 8) & 0xFFu) << 8) | ((su >> 16) << 16) | (((tw >> 18) & 1u) << 24);
        const uint2 t = RENDER ? make_uint2(tp & 0xFFFFu, tp >> 16) : pia_now();
        col[R_TIMER * stride] = t.x | (t.y << 16);
        col[R_SELPC * stride] = (su & 0xFFFFu) | (pcnt << 16);
        col[R_TIA0 * stride] = clock | (scanline << 16);
        uint32_t t1 = ((tw >> 16) & 1u) | (((tw >> 17) & 1u) << 8) | ((tw & 0xFFFFu) << 16);
        if constexpr (SLICED) t1 |= fa_mapper_tia1(mapper_of(slices));
        col[R_TIA1 * stride] = t1;
        col[R_TIA2 * stride] = ((pins >> 16) & 1u) | (((pins >> 17) & 1u) << 8) | (pads << 16);
    }
    // RAM words from the HBM rows into shared memory and back.
    __device__ __forceinline__ void load_ram(const uint32_t* c, uint32_t stride)
    {
#pragma unroll 4
        for (uint32_t k = 0; k < FA_SMEM_WORDS; k++) {
            const uint32_t v = c[k * stride];
#pragma unroll
            for (uint32_t j = 0; j < 4u; j++) pv[poff(4u * k + j)] = (uint8_t)(v >> (8u * j));
        }
    }
    __device__ __forceinline__ uint32_t ram_word(uint32_t k) const
    {
        uint32_t v = 0;
#pragma unroll
        for (uint32_t j = 0; j < 4u; j++) v |= (uint32_t)pv[poff(4u * k + j)] << (8u * j);
        return v;
    }
    __device__ __forceinline__ void store_ram(uint32_t* c, uint32_t stride) const
    {
#pragma unroll 4
        for (uint32_t k = 0; k < FA_SMEM_WORDS; k++) c[k * stride] = ram_word(k);
    }
};

}  // namespace fa
