// Test infrastructure: whole warps of the device core on the host.  32 lanes
// run run_unit_as (fa_run.cuh) with the scheduler of run_lanes as coroutines;
// a warp intrinsic suspends its lane until every lane of the mask has reached
// the same one.
#include "shim.h"
#include "../../fast-atari-rs_b200/csrc/fa_api.cu"
#include "../../fast-atari-rs_b200/csrc/fa_run.cuh"

#include <ucontext.h>

namespace {
enum Op { SHFL, XOR, BALLOT, ANY, ALL, MATCH, MIN };
struct Lane {
    ucontext_t ctx;
    bool done, waiting;
    uint32_t op, mask, val, src, out;
    std::vector<char> stack;
};
Lane lanes[32];
ucontext_t scheduler;
uint32_t cur;

uint32_t meet(Op op, uint32_t mask, uint32_t val, uint32_t src = 0)
{
    Lane& l = lanes[cur];
    l.waiting = true;
    l.op = op; l.mask = mask; l.val = val; l.src = src;
    swapcontext(&l.ctx, &scheduler);
    return l.out;
}

uint32_t result(const Lane& l)
{
    uint32_t ballot = 0, least = 0xFFFFFFFFu, same = 0;
    for (uint32_t j = 0; j < 32; j++)
        if (l.mask >> j & 1) {
            const Lane& o = lanes[j];
            if (o.val) ballot |= 1u << j;
            if (o.val < least) least = o.val;
            if (o.val == l.val) same |= 1u << j;
        }
    switch (l.op) {
    case SHFL: return lanes[l.src & 31u].val;
    case XOR: return lanes[(uint32_t)(&l - lanes) ^ l.src].val;
    case BALLOT: return ballot;
    case ANY: return ballot != 0;
    case ALL: return ballot == l.mask;
    case MATCH: return same;
    default: return least;
    }
}

struct Job {
    const FaGroup* G;
    uint32_t first, count;
    uint8_t* rom;
    uint32_t* priv;
    unsigned long long *instr, *rounds;
} job;

void lane_main()
{
    const FaGroup& G = *job.G;
    const uint32_t kind = fa_map_kind(G.hot_lo), t = cur;
    if (kind == FA_MAP_DPC) fa::run_unit_as<32, true, true>(G, job.first, job.count, job.rom, job.priv, t, job.instr, job.rounds);
    else if (kind == FA_MAP_FE) fa::run_unit_as<32, true, false, true>(G, job.first, job.count, job.rom, job.priv, t, job.instr, job.rounds);
    else if (kind) fa::run_unit_as<32, true>(G, job.first, job.count, job.rom, job.priv, t, job.instr, job.rounds);
    else fa::run_unit_as<32, false>(G, job.first, job.count, job.rom, job.priv, t, job.instr, job.rounds);
    lanes[t].done = true;
    swapcontext(&lanes[t].ctx, &scheduler);
}

// 0; -2: more than `limit` meetings; -3: lanes that wait for each other, or for one that has ended.
int run_warp(long long limit)
{
    for (uint32_t i = 0; i < 32; i++) {
        Lane& l = lanes[i];
        l.stack.resize(256 * 1024);
        l.done = l.waiting = false;
        getcontext(&l.ctx);
        l.ctx.uc_stack.ss_sp = l.stack.data();
        l.ctx.uc_stack.ss_size = l.stack.size();
        l.ctx.uc_link = &scheduler;
        makecontext(&l.ctx, lane_main, 0);
    }
    while (true) {
        uint32_t left = 0;
        for (cur = 0; cur < 32; cur++) {
            if (!lanes[cur].done && !lanes[cur].waiting) {
                threadIdx.x = cur;
                swapcontext(&scheduler, &lanes[cur].ctx);
            }
            left += !lanes[cur].done;
        }
        if (!left) return 0;
        bool met = false;
        for (uint32_t i = 0; i < 32; i++) {
            const uint32_t mask = lanes[i].mask, op = lanes[i].op;
            bool all = lanes[i].waiting;
            for (uint32_t j = 0; j < 32 && all; j++)
                if (mask >> j & 1) all = lanes[j].waiting && lanes[j].mask == mask && lanes[j].op == op;
            if (!all) continue;
            for (uint32_t j = 0; j < 32; j++)
                if (mask >> j & 1) lanes[j].out = result(lanes[j]);
            for (uint32_t j = 0; j < 32; j++)
                if (mask >> j & 1) lanes[j].waiting = false;
            met = true;
            if (--limit < 0) return -2;
        }
        if (!met) return -3;
    }
}
}  // namespace

uint32_t __shfl_sync(uint32_t m, uint32_t v, uint32_t s) { return meet(SHFL, m, v, s); }
uint32_t __shfl_xor_sync(uint32_t m, uint32_t v, uint32_t s) { return meet(XOR, m, v, s); }
uint32_t __ballot_sync(uint32_t m, bool v) { return meet(BALLOT, m, v); }
bool __any_sync(uint32_t m, bool v) { return meet(ANY, m, v) != 0; }
bool __all_sync(uint32_t m, bool v) { return meet(ALL, m, v) != 0; }
uint32_t __match_any_sync(uint32_t m, uint32_t v) { return meet(MATCH, m, v); }
uint32_t __reduce_min_sync(uint32_t m, uint32_t v) { return meet(MIN, m, v); }
unsigned long long atomicAdd(unsigned long long* p, unsigned long long v) { const unsigned long long o = *p; *p += v; return o; }

extern "C" int hs_warps(const uint8_t* rom, size_t len, fa_state* st, size_t n, const uint8_t* actions, int k, int sched,
                        long long limit, unsigned long long* counters)
{
    std::vector<uint8_t> img;
    int scheme = 0;
    uint32_t nbanks = 0, hot_lo = 0;
    if (fa_make_bank_image(rom, len, img, scheme, &nbanks, &hot_lo)) return -1;
    std::vector<uint8_t> simg(img.size() + 64, 0);
    memcpy(simg.data(), img.data(), img.size());
    std::vector<uint32_t> rows((size_t)FA_ROWS * n), priv(FA_SMEM_WORDS * 32);
    for (size_t i = 0; i < n; i++) fa_pack_column(st[i], rows.data() + i, n);
    FaGroup G;
    memset(&G, 0, sizeof(G));
    G.rom = simg.data(); G.state = rows.data(); G.stride = (uint32_t)n; G.n = (uint32_t)n;
    G.actions = actions; G.act_stride = (uint32_t)n; G.nbanks = nbanks; G.hot_lo = hot_lo; G.k = (uint32_t)k;
    G.sched = (uint32_t)sched;
    counters[0] = counters[1] = 0;
    for (uint32_t first = 0; first < n; first += 32) {
        job = Job{ &G, first, (uint32_t)(n - first < 32 ? n - first : 32), simg.data(), priv.data(), counters, counters + 1 };
        const int rc = run_warp(limit);
        if (rc) return rc;
    }
    for (size_t i = 0; i < n; i++) fa_unpack_column(rows.data() + i, n, scheme, st[i]);
    return 0;
}
