// Grouped multi-token MoE sublayer: every DISTINCT expert that the tokens of a step select is read once.
//
// The reference has no such kernel — its prefill runs token by token through the batch-1 path
// (src/runtime/engine.rs:1837-1838), so an expert chosen by 40 tokens is read 40 times.  Here the
// (token, expert) pairs of the step are bucketed by expert on the device, and per expert the projections
// are real matrix products on the 5th-generation tensor cores:
//
//   D[128 weight rows x N tokens] += A[128 x 256] . B[N x 256]^T      per 256-column slab of K
//
//   A  the INT4 page tile.  cp.async.bulk.tensor (one 3-D tensor map over the whole page pool: byte in
//      row, row in page, pool slot) brings 128 B of codes per row and slab, and the rows' group scales for four
//      slabs at a time (64 bytes of a row: a 16-byte piece per slab would cost half a memory sector and a row
//      segment of the TMA unit each), into shared memory (swizzled, so that lanes reading consecutive rows hit
//      different banks).  Converting warps turn the codes into the whole numbers n - 8 as fp16, exactly, and store
//      them with tcgen05.st into TENSOR MEMORY: the A operand never goes back through shared memory, whose
//      bandwidth could not carry 4x-expanded weights at the HBM rate.
//   B  the tokens of the expert: rows of a gathered fp16 activation matrix (pairs sorted by expert), loaded
//      by the same TMA unit as 128-byte-swizzled K-major tiles and read by the MMA through a shared-memory
//      descriptor.  Within every 8 columns the K order of both operands is (0,4,1,5,2,6,3,7): that is
//      the order in which one logic operation per two weights isolates the 4-bit codes, and a contraction
//      does not care about the order of K as long as both operands agree.
//   D  fp32 in tensor memory, one accumulator per scale group of 32 columns (two MMAs of 16): scaling warps read a
//      slab's accumulators with tcgen05.ld and add scale * D to their fp32 sums in registers, packed fp32 FMAs over
//      as many token columns as the expert has (2, 4, 8 or 16).  The scale costs one FMA per 32 weights and token
//      instead of one product per weight, and nothing is rounded between the codes and the fp32 sums.
//      At the end of a tile: gate/up SiLU product rounded to fp16 as the batch-1 path does; down fp16 per (pair, row),
//      combined per token in plan order by a last kernel, so that the result does not depend on scheduling.
//
// One elected thread per issuing warp issues MMAs; completion is tracked with tcgen05.commit on mbarriers.  Every wait is
// bounded (about four seconds): a thread that gives up sets VIB3_STATUS_TIMEOUT and the CTA drains and frees its tensor memory.
// No cluster launch, no multicast: every CTA fetches its own tiles.
//
// The path stays HBM-bound by construction: at 128 tokens the step has 90 GFLOP of tensor work (64 us at
// peak) against up to 7 GB of distinct expert weights (1 ms of HBM time); the figure of merit is bytes per
// second over the distinct experts, the tensor pipe's utilisation is reported beside it.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <new>

#include "int4_math.cuh"
#include "launch_common.h"
#include "pipe_common.cuh"

namespace vib3 {

// Warp roles: 0 weights' copies, 1 tokens' copies, 2.. MMA issuers, then scaling and converting warps.
constexpr int kGrpXWarp = 1, kGrpMmaWarp = 2;
constexpr int kGrpMmaWarps = 4;                 // an issuing warp takes every fourth scale group's MMAs
constexpr int kGrpFirstScaleWarp = kGrpMmaWarp + kGrpMmaWarps;   // two teams of four; TMEM lane quarter = warp & 3
constexpr int kGrpFirstConvWarp = kGrpFirstScaleWarp + 8;        // two teams of four
constexpr int kGrpThreads = (kGrpFirstConvWarp + 8) * 32;
constexpr int kGrpSlabK = 256;                  // columns of K per pipeline step
constexpr int kGrpMaxN = 16;                    // tokens of one expert per token group; a slab is converted once for up to two groups
constexpr int kGrpStages = 8;                   // code ring
constexpr int kGrpCodeBytes = 16 * 1024;        // codes of 128 rows x 256 columns
constexpr int kGrpXStages = 6;                  // token ring: one token group and slab per stage
constexpr int kGrpXBytes = kGrpMaxN * kGrpSlabK * 2;   // 16 tokens x 256 columns fp16
constexpr int kGrpChunkSlabs = 4;               // slabs whose scales travel together: 64 bytes of a row per copy
constexpr int kGrpScaleStages = 3;              // scale ring
constexpr int kGrpScaleBytes = 128 * kGrpChunkSlabs * 16;
constexpr int kGrpTmemCols = 512;
constexpr int kGrpACols = kGrpSlabK / 2;        // an A buffer: 256 fp16 per row
constexpr int kGrpDCols = 8 * kGrpMaxN;         // an accumulator buffer: 8 scale groups x 16 tokens
constexpr int kGrpDCol0 = 2 * kGrpACols;
static_assert(kGrpDCol0 + 2 * kGrpDCols <= kGrpTmemCols, "tensor memory budget");
static_assert(kGrpStages % 2 == 0, "the uses of a code stage belong to one converting team");
constexpr int kGrpMaxTokens = 128;
constexpr int kRouterMaxExpertsGrouped = 512;   // MAX_EXPERTS, src/core/types.rs:20

struct GroupedMaps {
    CUtensorMap gu_codes, gu_scales_full, gu_scales_last, dn_codes, dn_scales_full, dn_scales_last;
    CUtensorMap xg16, act16;
};

// Device-side description of the step, written by group_pairs_kernel.
struct GroupedWork {
    int n_active;            // distinct experts with at least one token (the shared expert counts as one)
    int n_pairs;
    int pad[2];
};

struct Unit;
// Trips over a unit's slabs: one per 32 tokens.
__host__ __device__ constexpr int grp_passes(int n_tok) { return (n_tok + 2 * kGrpMaxN - 1) / (2 * kGrpMaxN); }
struct GroupedArgs {
    const GroupedWork* work;
    __half* act;             // [pairs][I], K order permuted
    __half* y;               // [pairs][H]
    const Unit* units_gu;    // [n_active * tiles_gu]
    const Unit* units_dn;    // [n_active * tiles_dn]
    int tiles_gu, tiles_dn;
    int H, I;
    int* status;
};

// An mbarrier of this kernel by its 32-bit shared-memory address; `+ i` is the i-th of an array.
struct Bar {
    uint32_t addr;
    __device__ __forceinline__ Bar operator+(int i) const { return Bar{addr + 8u * (uint32_t)i}; }
};
// The waits of this kernel: one look that does not suspend the warp, then suspending tries without a time limit of their
// own.  A try with a suspend-time hint resumed later: with the hint the 32-token Kimi layer took 1025 us, without 983.
// Bounded: a try whose phase does not complete comes back after 3.95 us (200 tries in a row: 790 us), so a wait gives up,
// with false, after about four seconds.
constexpr unsigned kGrpWaitTries = 1u << 20;
__device__ __forceinline__ bool mbar_wait_grp(Bar bar, unsigned parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar.addr), "r"(parity) : "memory");
    for (unsigned it = 0; !ok && it < kGrpWaitTries; ++it)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar.addr), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void mbar_init(Bar bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar.addr), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(Bar bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar.addr), "r"(bytes) : "memory");
}
// one arrival for the warp (predicated, no branch)
__device__ __forceinline__ void mbar_arrive_lane0(Bar bar, int lane) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar.addr), "r"(lane) : "memory");
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, Bar bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar.addr) : "memory");
}
// One lane of the warp, the same one every time.  MMAs and tensor copies take their operands from uniform registers:
// behind elect.sync, with operands that are uniform by construction, they issue back to back; behind `lane == 0` each of
// their operands is moved over one by one.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ void umma_commit(Bar bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar.addr) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 codes (one scale group, word j = columns 8j .. 8j+7) -> 16 half2 of n - 8 in the K order
// (0,4),(1,5),(2,6),(3,7) per word.  (n + 1024) and (16 n + 1024) are exact fp16 numbers made by one logic
// operation per pair; subtracting 1032, or multiplying by 1/16 and subtracting 72, is exact as well.
__device__ __forceinline__ void codes_to_f16(const uint4& q, uint32_t* out) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t w8 = w[j] >> 8;
        const uint32_t a0 = lop3_and_or(w[j], 0x000F000Fu, 0x64006400u);
        const uint32_t a1 = lop3_and_or(w[j], 0x00F000F0u, 0x64006400u);
        const uint32_t a2 = lop3_and_or(w8, 0x000F000Fu, 0x64006400u);
        const uint32_t a3 = lop3_and_or(w8, 0x00F000F0u, 0x64006400u);
        asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(out[4 * j + 0]) : "r"(a0), "r"(0x64086408u));                       // (n + 1024) - 1032
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(out[4 * j + 1]) : "r"(a1), "r"(0x2C002C00u), "r"(0xD480D480u));  // / 16 - 72
        asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(out[4 * j + 2]) : "r"(a2), "r"(0x64086408u));
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(out[4 * j + 3]) : "r"(a3), "r"(0x2C002C00u), "r"(0xD480D480u));
    }
}

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
                 "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
                 "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
// N columns of this lane's row (N = 2, 4, 8, 16); the values are there after tmem_ld_wait.
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t* r) {
    if constexpr (N == 2)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr) : "memory");
    else if constexpr (N == 4)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
    else if constexpr (N == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                       "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                     : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// acc[t] += scale * D[group][t] for the eight groups of a slab and NE tokens (packed pairs of fp32 FMAs): the accumulators
// hold integer-weight sums over 32 columns, the scale of the group is applied here in fp32.  `release` is arrived on
// once the accumulators are in registers.
template <int NE>
__device__ __forceinline__ void scale_slab(uint32_t taddr, const uint4& sc, float2* acc, Bar release, int lane) {
    constexpr int kBatch = NE <= 4 ? 8 : NE == 8 ? 4 : 2;   // groups read together: up to 32 registers
    const uint32_t sw[4] = {sc.x, sc.y, sc.z, sc.w};
#pragma unroll
    for (int g0 = 0; g0 < 8; g0 += kBatch) {
        uint32_t d[kBatch][NE];
#pragma unroll
        for (int g = 0; g < kBatch; ++g) tmem_ld<NE>(taddr + (g0 + g) * kGrpMaxN, d[g]);
        tmem_ld_wait();
        if (g0 + kBatch == 8) {
            tc_fence_before();
            __syncwarp();
            mbar_arrive_lane0(release, lane);
        }
#pragma unroll
        for (int g = 0; g < kBatch; ++g) {
            const uint32_t pair = sw[(g0 + g) >> 1];
            const float s = __half2float(__ushort_as_half((unsigned short)((g0 + g) & 1 ? pair >> 16 : pair & 0xFFFFu)));
            uint64_t s2;
            asm("mov.b64 %0, {%1, %1};" : "=l"(s2) : "f"(s));
#pragma unroll
            for (int j = 0; j < NE / 2; ++j) {
                uint64_t dv, av;
                asm("mov.b64 %0, {%1, %2};" : "=l"(dv) : "r"(d[g][2 * j]), "r"(d[g][2 * j + 1]));
                asm("mov.b64 %0, {%1, %2};" : "=l"(av) : "f"(acc[j].x), "f"(acc[j].y));
                asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(av) : "l"(dv), "l"(s2));
                asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[j].x), "=f"(acc[j].y) : "l"(av));
            }
        }
    }
}

__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

// Position of row r (column of the down projection) in the permuted K order.
__device__ __forceinline__ int perm8(int r) {
    const int i = r & 7;
    return (r & ~7) | (i < 4 ? 2 * i : 2 * (i - 4) + 1);
}

// One work unit: a 128-row A tile of one expert (gate/up: 64 gate rows and the same 64 up rows; down: 128 rows).
// The units of a step are listed by build_units; unit u = (active expert u / tiles, tile u % tiles).
struct __align__(16) Unit {
    int slot_a, slot_b;      // pool slots of the page(s); -1: page absent
    short row0;              // first row of the tile inside the page
    short rows;              // valid rows of the tile (gate/up: of each half)
    short scales_last;       // 1: the page is a last (short) page, its scales start earlier
    short pad;
    int mrow0;               // first row inside the matrix
    int n_tok, pair_off;     // the expert's tokens: count and first sorted pair
    int pad2;
};
static_assert(sizeof(Unit) == 32, "a unit is two 16-byte loads");

struct UnitWalk {
    const Unit* units;
    int n_units, u;
    int ahead;   // a word of the next unit: loaded early, so that the unit itself is found in L1
    __device__ __forceinline__ void touch() {
        if (u < n_units) ahead = __ldg(reinterpret_cast<const int*>(units + u));
    }
    __device__ __forceinline__ UnitWalk(const Unit* units_, int n_units_) : units(units_), n_units(n_units_), u(blockIdx.x), ahead(0) { touch(); }
    // the next unit with work of this CTA
    __device__ __forceinline__ bool next(Unit& t) {
        while (u < n_units) {
            asm volatile("" ::"r"(ahead));
            const uint4* p = reinterpret_cast<const uint4*>(units + u);
            uint4* q = reinterpret_cast<uint4*>(&t);
            q[0] = __ldg(p);
            q[1] = __ldg(p + 1);
            u += gridDim.x;
            touch();
            if (t.rows > 0 && t.n_tok > 0) return true;
        }
        return false;
    }
};

// The halves of a token group's columns, as compile-time numbers.
struct First { static constexpr int value = 0; };
struct Second { static constexpr int value = 1; };

// DOWN = false: act[pair][perm(row)] = f16(silu(f16(Wg x)) * f16(Wu x)); DOWN = true: y[pair][row] = f16(Wd act).
//
// What bounds it: not memory (the same walk without conversion, MMAs and scaling runs at 6.2 TB/s) and not the tensor pipe, but
// the converting warps' instructions and the hand-overs between the roles.  Hence few warps (with 16 converting warps
// the waits of all of them took more issue slots than their arithmetic gained: 1210 us against 1140), a whole slab per
// hand-over (quarters: 1680 us), no scale product per weight, rolled conversion loops, operands that need no
// per-lane moves (elect_one).  Experts' launches alone, with one fp16 product with the scale per weight (26 warps) and now: Kimi
// layer, 32 tokens (177 distinct experts, 4.4 GB) 1201 -> 930 us = 4.7 TB/s; 8 tokens, even load, 430 -> 330 us; 128 tokens, skewed
// load, 1350 -> 1162 us; Mixtral shape, 50 tokens, 292 -> 259 us.
//
// Every role walks the same sequence: units blockIdx.x, + gridDim.x, ...; per unit ceil(n_tok / 32) passes of one or two
// token groups of 16; per pass nslab slabs of 256 columns; per slab a step for each token group.  `it` counts slabs (code
// stage it % 8, A buffer and converting team it & 1), `step` steps (accumulator buffer and scaling team step & 1).  With
// one token group the two scaling teams take alternate slabs of the same tokens and their sums meet at the end, with
// two groups each team has its own (so the order of a token's fp32 sums depends on whether its expert has more than 16
// tokens left, and on nothing else).  A barrier is only ever waited for by roles that have seen its previous phase
// complete (a wait names its phase by one parity bit).
template <bool DOWN>
__global__ void __launch_bounds__(kGrpThreads, 1) moe_grouped_kernel(const __grid_constant__ GroupedMaps maps, GroupedArgs a) {
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    const uint32_t wring = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    const uint32_t xring = wring + kGrpStages * kGrpCodeBytes;
    const uint32_t sring = xring + kGrpXStages * kGrpXBytes;
    const uint32_t exch_addr = sring + kGrpScaleStages * kGrpScaleBytes;
    float* exch = reinterpret_cast<float*>(smem_dyn + (exch_addr - smem_u32(smem_dyn)));               // [128][kGrpMaxN + 1]
    const Bar full{exch_addr + 128 * (kGrpMaxN + 1) * 4};
    const Bar empty = full + kGrpStages;
    const Bar xfull = empty + kGrpStages;
    const Bar xempty = xfull + kGrpXStages;
    const Bar sfull = xempty + kGrpXStages;
    const Bar sempty = sfull + kGrpScaleStages;
    const Bar a_full = sempty + kGrpScaleStages;   // [it & 1] the A operand is in tensor memory
    const Bar a_empty = a_full + 2;                // [it & 1] the MMAs that read it have completed
    const Bar d_full = a_empty + 2;                // [step & 1] the accumulators are complete
    const Bar d_empty = d_full + 2;                // [step & 1] the accumulators have been read
    const Bar part_full = d_empty + 2;             // [team] (one token group) the team's sums of the other's columns are in exch
    const Bar up_full = part_full + 2;             // [team] (gate/up) the up rows' sums are in exch
    const Bar exch_free = up_full + 2;             // every scaling warp is through with this pass's exchange
    const Bar mma_done = exch_free + 1;            // [issuer] (after a wait that ran out) all of the issuer's MMAs have completed
    const uint32_t tmem_slot = (mma_done + kGrpMmaWarps).addr;

    const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
    const int K = DOWN ? a.I : a.H;
    const int nslab = K / kGrpSlabK;
    if (tid == 0) {
        for (int s = 0; s < kGrpStages; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 4);
        }
        for (int s = 0; s < kGrpXStages; ++s) {
            mbar_init(xfull + s, 1);
            mbar_init(xempty + s, kGrpMmaWarps);
        }
        for (int s = 0; s < kGrpScaleStages; ++s) {
            mbar_init(sfull + s, 1);
            mbar_init(sempty + s, 8);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(a_full + s, 4);
            mbar_init(a_empty + s, kGrpMmaWarps);
            mbar_init(d_full + s, kGrpMmaWarps);
            mbar_init(d_empty + s, 4);
            mbar_init(up_full + s, 2);
            mbar_init(part_full + s, 4);
        }
        mbar_init(exch_free, 8);
        for (int s = 0; s < kGrpMmaWarps; ++s) mbar_init(mma_done + s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kGrpMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(kGrpTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    uint32_t tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot) : "memory");
    tmem = (uint32_t)uniform((int)tmem);
    pdl_wait();   // the work lists, the gathered tokens and (down) the intermediate are earlier kernels' outputs
    UnitWalk walk(DOWN ? a.units_dn : a.units_gu, a.work->n_active * (DOWN ? a.tiles_dn : a.tiles_gu));

    bool ok = true;
    if (warp == 0) {
        // ── TMA producer of the code and scale rings ──
        int it = 0, ss = 0, su = 0, nchunk = 0;   // scale stage, its use number, chunks issued
        Unit t;
        while (ok && walk.next(t)) {
            const CUtensorMap* codes = DOWN ? &maps.dn_codes : &maps.gu_codes;
            const CUtensorMap* scales = DOWN ? (t.scales_last ? &maps.dn_scales_last : &maps.dn_scales_full)
                                             : (t.scales_last ? &maps.gu_scales_last : &maps.gu_scales_full);
            const int row0 = uniform(t.row0), slot_a = uniform(t.slot_a), slot_b = uniform(t.slot_b);
            const int passes = grp_passes(t.n_tok);
            for (int p = 0; ok && p < passes; ++p) {
                for (int s = 0; s < nslab; ++s, ++it) {
                    const int st = it % kGrpStages;
                    const bool chunk = s % kGrpChunkSlabs == 0;
                    if (it >= kGrpStages) ok = mbar_wait_grp(empty + st, ((it / kGrpStages) - 1) & 1);
                    if (chunk && ok && su > 0) ok = mbar_wait_grp(sempty + ss, (su - 1) & 1);
                    if (!ok) break;
                    if (elect_one()) {
                        const uint32_t dst = wring + (uint32_t)st * kGrpCodeBytes;
                        mbar_expect_tx(full + st, kGrpCodeBytes);
                        tma_load_3d(dst, codes, s * 128, row0, slot_a, full + st);
                        if (!DOWN) tma_load_3d(dst + kGrpCodeBytes / 2, codes, s * 128, row0, slot_b, full + st);
                        if (chunk) {
                            const uint32_t sdst = sring + (uint32_t)ss * kGrpScaleBytes;
                            mbar_expect_tx(sfull + ss, kGrpScaleBytes);
                            tma_load_3d(sdst, scales, s * 16, row0, slot_a, sfull + ss);
                            if (!DOWN) tma_load_3d(sdst + kGrpScaleBytes / 2, scales, s * 16, row0, slot_b, sfull + ss);
                        }
                    }
                    __syncwarp();
                    if (chunk) {
                        ++nchunk;
                        if (++ss == kGrpScaleStages) {
                            ss = 0;
                            ++su;
                        }
                    }
                }
            }
        }
        if (!ok && lane == 0) flag(a.status, kStatusTimeout);
        // drain: every issued copy must have landed before the CTA's shared memory goes away (one wait that runs out ends
        // the drain: four more seconds at most)
        if (lane == 0) {
            bool landed = true;
            for (int k = max(0, it - kGrpStages); landed && k < it; ++k) landed = mbar_wait_grp(full + (k % kGrpStages), (k / kGrpStages) & 1);
            for (int k = max(0, nchunk - kGrpScaleStages); landed && k < nchunk; ++k)
                landed = mbar_wait_grp(sfull + (k % kGrpScaleStages), (k / kGrpScaleStages) & 1);
            if (!landed) flag(a.status, kStatusTimeout);
        }
    } else if (warp == kGrpXWarp) {
        // ── TMA producer of the token ring: one copy per step (four K-major tiles of 64 columns) ──
        int xs = 0, xu = 0, n = 0;   // stage, its use number, copies issued
        Unit t;
        const CUtensorMap* xmap = DOWN ? &maps.act16 : &maps.xg16;
        while (ok && walk.next(t)) {
            for (int p0 = 0; ok && p0 < t.n_tok; p0 += 2 * kGrpMaxN) {
                const int ng = t.n_tok - p0 > kGrpMaxN ? 2 : 1;
                const int row = uniform(t.pair_off + p0);
                for (int s = 0; ok && s < nslab; ++s) {
                    for (int g = 0; g < ng; ++g, ++n) {
                        if (xu > 0) ok = mbar_wait_grp(xempty + xs, (xu - 1) & 1);
                        if (!ok) break;
                        if (elect_one()) {
                            mbar_expect_tx(xfull + xs, kGrpXBytes);
                            tma_load_3d(xring + (uint32_t)xs * kGrpXBytes, xmap, 0, row + g * kGrpMaxN, s * (kGrpSlabK / 64), xfull + xs);
                        }
                        __syncwarp();
                        if (++xs == kGrpXStages) {
                            xs = 0;
                            ++xu;
                        }
                    }
                }
            }
        }
        if (!ok && lane == 0) flag(a.status, kStatusTimeout);
        if (lane == 0) {
            bool landed = true;
            for (int k = max(0, n - kGrpXStages); landed && k < n; ++k) landed = mbar_wait_grp(xfull + (k % kGrpXStages), (k / kGrpXStages) & 1);
            if (!landed) flag(a.status, kStatusTimeout);
        }
    } else if (warp < kGrpFirstScaleWarp) {
        // ── MMA issuers: per step and scale group (32 columns, an accumulator of its own) two MMAs; the issuers share the groups ──
        const int mw = warp - kGrpMmaWarp;
        int it = 0, step = 0, xs = 0, xu = 0;
        Unit t;
        constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(kGrpMaxN >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        while (ok && walk.next(t)) {
            for (int p0 = 0; ok && p0 < t.n_tok; p0 += 2 * kGrpMaxN) {
                const int ng = uniform(t.n_tok - p0 > kGrpMaxN ? 2 : 1);
                for (int s = 0; ok && s < nslab; ++s, ++it) {
                    const int ab = it & 1;
                    for (int g = 0; g < ng; ++g, ++step) {
                        const int db = step & 1;
                        if (step >= 2) ok = ok && mbar_wait_grp(d_empty + db, ((step >> 1) - 1) & 1);
                        ok = ok && mbar_wait_grp(xfull + xs, xu & 1);
                        const uint32_t xaddr = xring + (uint32_t)xs * kGrpXBytes;
                        const uint64_t xdesc = (uint64_t)((xaddr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
                                               ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
                        const uint32_t d0 = tmem + kGrpDCol0 + db * kGrpDCols, a0 = tmem + ab * kGrpACols;
                        // last, since it is the one that decides: a wait costs some 200 cycles also when its phase is over
                        if (g == 0) ok = ok && mbar_wait_grp(a_full + ab, (it >> 1) & 1);
                        if (!ok) break;
                        tc_fence_after();
                        if (elect_one()) {
#pragma unroll
                            for (int kk = 0; kk < 2; ++kk) {
#pragma unroll
                                for (int i = 0; i < 8 / kGrpMmaWarps; ++i) {
                                    const int gr = i * kGrpMmaWarps + mw;
                                    const uint64_t bdesc = xdesc + (uint64_t)(((gr >> 1) * kGrpMaxN * 128 + (gr & 1) * 64 + kk * 32) >> 4);
                                    umma_ts(d0 + gr * kGrpMaxN, a0 + 16 * gr + 8 * kk, bdesc, idesc, (uint32_t)kk);
                                }
                            }
                            umma_commit(d_full + db);
                            umma_commit(xempty + xs);
                            if (g == ng - 1) umma_commit(a_empty + ab);
                        }
                        __syncwarp();
                        if (++xs == kGrpXStages) {
                            xs = 0;
                            ++xu;
                        }
                    }
                }
            }
        }
        // Nothing may be owed to this CTA when it leaves.  The last commits' arrivals on xempty and a_empty have no other waiter;
        // after a wait that ran out, those phases may never complete, but this thread's own MMAs do, and until then they
        // read shared memory and use tensor memory.
        if (ok) {
            for (int k = max(0, step - kGrpXStages); ok && k < step; ++k) ok = mbar_wait_grp(xempty + k % kGrpXStages, (k / kGrpXStages) & 1);
            for (int k = max(0, it - 2); ok && k < it; ++k) ok = mbar_wait_grp(a_empty + (k & 1), (k >> 1) & 1);
        }
        if (!ok) {
            if (elect_one()) umma_commit(mma_done + mw);
            __syncwarp();
            mbar_wait_grp(mma_done + mw, 0);
            if (lane == 0) flag(a.status, kStatusTimeout);
        }
    } else if (warp >= kGrpFirstConvWarp) {
        // ── converting warps: two teams of four take alternate slabs.  Row m = 32 (warp % 4) + lane of the A tile ──
        const int team = (warp - kGrpFirstConvWarp) >> 2;
        const int q = warp & 3;
        const int m = 32 * q + lane;
        const uint32_t code_off = (uint32_t)m * 128u;         // (gate/up: the up tile follows the gate tile's 64 rows)
        const int first_row = DOWN ? 32 * q : 32 * (q & 1);   // first row (of the matrix half) among this warp's 32
        const uint32_t sw = (uint32_t)(m & 7);
        const uint32_t taddr = tmem + ((uint32_t)(32 * q) << 16) + team * kGrpACols;
        int it = 0;
        Unit t;
        while (ok && walk.next(t)) {
            const int end = it + grp_passes(t.n_tok) * nslab;
            // a warp whose 32 rows all lie beyond the tile's last row has nothing to convert: its lanes of the
            // accumulator are never read
            const bool work = first_row < t.rows;
            for (int i = it + ((it ^ team) & 1); i < end; i += 2) {
                const int st = i % kGrpStages, use = i >> 1;
                ok = mbar_wait_grp(full + st, (i / kGrpStages) & 1);
                if (!ok) break;
                const uint32_t cb = wring + (uint32_t)st * kGrpCodeBytes + code_off;
                uint4 n0 = make_uint4(0, 0, 0, 0), n1 = n0;   // the next two scale groups' codes
                if (work) {
                    n0 = lds128(cb + ((0u ^ sw) * 16u));
                    n1 = lds128(cb + ((1u ^ sw) * 16u));
                }
                if (use > 0) ok = mbar_wait_grp(a_empty + team, (use - 1) & 1);
                if (!ok) break;
                tc_fence_after();
                if (work) {
                    // (rolled: four trips through a short loop fetch fewer instructions than 320 of them in a row)
#pragma unroll 1
                    for (int j = 0; j < 8; j += 2) {
                        uint32_t g[32];
                        const uint4 c0 = n0, c1 = n1;
                        if (j < 6) {
                            n0 = lds128(cb + ((((uint32_t)j + 2) ^ sw) * 16u));
                            n1 = lds128(cb + ((((uint32_t)j + 3) ^ sw) * 16u));
                        }
                        codes_to_f16(c0, g);
                        codes_to_f16(c1, g + 16);
                        tmem_st32(taddr + 16 * j, g);
                    }
                }
                __syncwarp();
                mbar_arrive_lane0(empty + st, lane);   // the slab is in registers: the stage may be refilled
                if (work) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                mbar_arrive_lane0(a_full + team, lane);
            }
            it = end;
        }
        if (!ok && lane == 0) flag(a.status, kStatusTimeout);
    } else if (warp >= kGrpFirstScaleWarp) {
        // ── scaling warps: lane = row m of the tile ──
        const int team = (warp - kGrpFirstScaleWarp) >> 2;
        const int q = warp & 3;
        const int m = 32 * q + lane;
        const int first_row = DOWN ? 32 * q : 32 * (q & 1);
        // row m's scales in a stage: 64 bytes per row, 64-byte swizzle (the 16-byte unit number is XORed with row / 2)
        const uint32_t sbase = sring + (uint32_t)m * 64u;
        const uint32_t ssw = (uint32_t)(m >> 1) & 3u;
        const uint32_t taddr = tmem + ((uint32_t)(32 * q) << 16) + kGrpDCol0 + team * kGrpDCols;
        int step = 0, pc = 0, ss = 0, su = 0, n_part = 0, n_up = 0;
        Unit t;
        while (ok && walk.next(t)) {
            const bool work = first_row < t.rows;
            for (int p0 = 0; ok && p0 < t.n_tok; p0 += 2 * kGrpMaxN, ++pc) {
                const bool two = t.n_tok - p0 > kGrpMaxN;
                const int grp = two ? (team ^ step) & 1 : 0;      // this team's token group of the pass
                const int t0 = p0 + grp * kGrpMaxN;
                const int ntok = min(kGrpMaxN, t.n_tok - t0);
                float2 acc[kGrpMaxN / 2];
#pragma unroll
                for (int j = 0; j < kGrpMaxN / 2; ++j) acc[j] = make_float2(0.f, 0.f);
                for (int s = 0; s < nslab; ++s) {
                    const uint32_t sub = (uint32_t)s % kGrpChunkSlabs;
                    if (sub == 0) ok = ok && mbar_wait_grp(sfull + ss, su & 1);
                    // the step of this slab that belongs to this team, if any
                    const int mine = step + grp;
                    step += two ? 2 : 1;
                    if ((mine & 1) == team) {
                        uint4 sc = lds128(sbase + (uint32_t)ss * kGrpScaleBytes + ((sub ^ ssw) << 4));
                        ok = ok && mbar_wait_grp(d_full + team, (mine >> 1) & 1);
                        if (!ok) break;
                        tc_fence_after();
                        if (!work) {
                            __syncwarp();   // (a lane still on its way out of the wait could otherwise miss the phase)
                            mbar_arrive_lane0(d_empty + team, lane);
                        } else if (ntok <= 2) {
                            scale_slab<2>(taddr, sc, acc, d_empty + team, lane);
                        } else if (ntok <= 4) {
                            scale_slab<4>(taddr, sc, acc, d_empty + team, lane);
                        } else if (ntok <= 8) {
                            scale_slab<8>(taddr, sc, acc, d_empty + team, lane);
                        } else {
                            scale_slab<16>(taddr, sc, acc, d_empty + team, lane);
                        }
                    }
                    if (sub == kGrpChunkSlabs - 1 || s == nslab - 1) {
                        __syncwarp();
                        mbar_arrive_lane0(sempty + ss, lane);
                        if (++ss == kGrpScaleStages) {
                            ss = 0;
                            ++su;
                        }
                    }
                }
                if (pc > 0) ok = ok && mbar_wait_grp(exch_free, (pc - 1) & 1);
                if (!ok) break;
                // The ends of a pass, eight columns (a half) at a time.  With two token groups a team finishes both halves of its
                // own.  With one, the teams' sums meet in shared memory: team 0 finishes the first half and, if there are more
                // than eight tokens, team 1 the second.  While a team is busy here its accumulator buffer waits, which short units
                // feel: 64 experts of 1024 x 4096, 12 tokens each, 199 us with all sixteen columns left to team 0, 186 so;
                // Kimi layer, 8 tokens, 336 -> 330 us (loops of eight columns instead of sixteen).
                const bool wide = ntok > 8;
                float* ex = exch + m * (kGrpMaxN + 1);
                auto put = [&](float* to, auto half) {
                    constexpr int h = decltype(half)::value;
#pragma unroll
                    for (int j = 4 * h; j < 4 * h + 4; ++j) {
                        if (2 * j < ntok) {
                            to[2 * j] = acc[j].x;
                            to[2 * j + 1] = acc[j].y;
                        }
                    }
                };
                auto take = [&](auto half) {
                    constexpr int h = decltype(half)::value;
#pragma unroll
                    for (int j = 4 * h; j < 4 * h + 4; ++j) {
                        if (2 * j < ntok) {
                            acc[j].x += ex[2 * j];
                            acc[j].y += ex[2 * j + 1];
                        }
                    }
                };
                if (!two) {
                    if (team == 1) put(ex, First{});
                    else if (wide) put(ex, Second{});
                    if (team == 1 || wide) {
                        __syncwarp();
                        mbar_arrive_lane0(part_full + team, lane);
                    }
                    if (team == 0 || wide) ok = mbar_wait_grp(part_full + (team ^ 1), n_part++ & 1);
                    if (!ok) break;
                    if (team == 0) take(First{});
                    else if (wide) take(Second{});
                }
                const bool lo = two || team == 0, hi = wide && (two || team == 1);
                if (DOWN) {
                    if (m < t.rows) {
                        __half* y = a.y + (size_t)(t.pair_off + t0) * a.H + t.mrow0 + m;
                        auto store = [&](auto half) {
                            constexpr int h = decltype(half)::value;
#pragma unroll
                            for (int j = 8 * h; j < 8 * h + 8; ++j)
                                if (j < ntok) y[(size_t)j * a.H] = __float2half_rn(j & 1 ? acc[j >> 1].y : acc[j >> 1].x);
                        };
                        if (lo) store(First{});
                        if (hi) store(Second{});
                    }
                } else if (lo || hi) {
                    // the up half hands its values to the gate half of the same rows: through the second half of exch, or
                    // (two token groups) through the team's half
                    float* up = two ? exch + (team * 64 + (m & 63)) * (kGrpMaxN + 1) : exch + (64 + (m & 63)) * (kGrpMaxN + 1);
                    if (m >= 64) {
                        if (lo) put(up, First{});
                        if (hi) put(up, Second{});
                        __syncwarp();
                        mbar_arrive_lane0(up_full + team, lane);
                    } else {
                        ok = mbar_wait_grp(up_full + team, n_up & 1);
                        if (!ok) break;
                        if (m < t.rows) {
                            __half* act = a.act + (size_t)(t.pair_off + t0) * a.I + perm8(t.mrow0 + m);
                            auto store = [&](auto half) {
                                constexpr int h = decltype(half)::value;
#pragma unroll
                                for (int j = 8 * h; j < 8 * h + 8; ++j) {
                                    if (j < ntok) {
                                        const float g16 = __half2float(__float2half_rn(j & 1 ? acc[j >> 1].y : acc[j >> 1].x));
                                        const float u16 = __half2float(__float2half_rn(up[j]));
                                        act[(size_t)j * a.I] = __float2half_rn(silu_mul_f32(g16, u16));
                                    }
                                }
                            };
                            if (lo) store(First{});
                            if (hi) store(Second{});
                        }
                    }
                    ++n_up;
                }
                __syncwarp();
                mbar_arrive_lane0(exch_free, lane);
            }
        }
        if (!ok && lane == 0) flag(a.status, kStatusTimeout);
    }
    // Free the tensor memory once every role is done with it (a role that gave up has stopped touching it).
    tc_fence_before();
    __syncthreads();
    pdl_trigger();
    if (warp == kGrpMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kGrpTmemCols) : "memory");
    }
}

// ── bucketing ────────────────────────────────────────────────────────────────────────────────
// One CTA.  Pairs (token, slot) -> sorted by expert (stable in token order); the shared expert, if any, is
// expert E with every token.  Also the list of active experts, most tokens first (ties: lower id), so that
// the experts with several passes start first.
struct GroupPairsArgs {
    const unsigned short* ids;   // [T] rows of top_k, stride in bytes
    int ids_stride;
    int T, top_k, E, has_shared;
    int expert_lo, expert_hi;    // only pairs whose expert lies in [lo, hi) are taken (an expert-parallel rank's share)
    GroupedWork* work;
    int* active;
    int* counts;     // [E + 1]
    int* offsets;    // [E + 2]
    int* pos;        // [T][top_k + 1]: sorted position of (token, slot); slot top_k = the shared expert
    unsigned short* pair_token;  // [pairs]
    int* status;
};

__global__ void __launch_bounds__(1024) group_pairs_kernel(GroupPairsArgs g) {
    constexpr int kWords = kGrpMaxTokens / 32;
    __shared__ __align__(16) int cnt[kRouterMaxExpertsGrouped + 4];
    __shared__ int off[kRouterMaxExpertsGrouped + 2];
    __shared__ unsigned mask[kRouterMaxExpertsGrouped][kWords];   // bit t of expert e: token t chose e
    __shared__ int warp_total[32];
    __shared__ int nact;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int NE = g.E + 1;
    pdl_wait();
    for (int i = tid; i < g.E * kWords; i += blockDim.x) (&mask[0][0])[i] = 0;
    if (tid == 0) nact = 0;
    __syncthreads();
    const int total = g.T * g.top_k;
    for (int i = tid; i < total; i += blockDim.x) {
        const int t = i / g.top_k, s = i - t * g.top_k;
        const unsigned e = reinterpret_cast<const unsigned short*>(reinterpret_cast<const unsigned char*>(g.ids) + (size_t)t * g.ids_stride)[s];
        if (e >= (unsigned)g.E) flag(g.status, kStatusBadExpert);
        else if ((int)e >= g.expert_lo && (int)e < g.expert_hi) atomicOr(&mask[e][t >> 5], 1u << (t & 31));
    }
    __syncthreads();
    // counts, then their exclusive prefix sum (one value per thread: warp scans, then a scan of the warps' totals)
    int c = 0;
    if (tid < g.E) {
#pragma unroll
        for (int w = 0; w < kWords; ++w) c += __popc(mask[tid][w]);
    } else if (tid == g.E) {
        c = g.has_shared ? g.T : 0;
    }
    for (int e = tid; e < kRouterMaxExpertsGrouped + 4; e += blockDim.x) cnt[e] = e == tid ? c : 0;
    int incl = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
    }
    if (lane == 31) warp_total[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int v = warp_total[lane], iv = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, iv, d);
            if (lane >= d) iv += u;
        }
        warp_total[lane] = iv - v;
        if (lane == 31) g.work->n_pairs = iv;
    }
    __syncthreads();
    if (tid <= NE) off[tid] = warp_total[warp] + incl - c;   // (off[NE] = the total: the threads past NE hold zero counts)
    __syncthreads();
    if (tid < NE) {
        g.counts[tid] = c;
        g.offsets[tid] = off[tid];
        if (c > 0) {
            // position among the active experts, most tokens first (ties: lower id)
            int rank = 0;
            const int4* c4 = reinterpret_cast<const int4*>(cnt);
            for (int o4 = 0; o4 < (NE + 3) / 4; ++o4) {
                const int4 v = c4[o4];
                const int o = 4 * o4;
                rank += (v.x > c || (v.x == c && o < tid)) + (v.y > c || (v.y == c && o + 1 < tid)) + (v.z > c || (v.z == c && o + 2 < tid)) +
                        (v.w > c || (v.w == c && o + 3 < tid));
            }
            g.active[rank] = tid;
            atomicAdd(&nact, 1);
        }
    }
    // placement, stable in token order: a pair's position is its expert's offset plus the number of earlier tokens
    // that chose the expert
    for (int i = tid; i < total; i += blockDim.x) {
        const int t = i / g.top_k, s = i - t * g.top_k;
        const unsigned e = reinterpret_cast<const unsigned short*>(reinterpret_cast<const unsigned char*>(g.ids) + (size_t)t * g.ids_stride)[s];
        int p = -1;   // a pair of another rank's expert
        if (e < (unsigned)g.E && (int)e >= g.expert_lo && (int)e < g.expert_hi) {
            p = off[e] + __popc(mask[e][t >> 5] & ((1u << (t & 31)) - 1u));
            for (int w = 0; w < (t >> 5); ++w) p += __popc(mask[e][w]);
            g.pair_token[p] = (unsigned short)t;
        }
        g.pos[t * (g.top_k + 1) + s] = p;
    }
    for (int t = tid; t < g.T; t += blockDim.x) {
        if (g.has_shared) g.pair_token[off[g.E] + t] = (unsigned short)t;
        g.pos[t * (g.top_k + 1) + g.top_k] = g.has_shared ? off[g.E] + t : -1;
    }
    __syncthreads();
    if (tid == 0) g.work->n_active = nact;
    pdl_trigger();
}

// The unit tables of the step: one thread per (active expert, tile).
struct BuildUnitsArgs {
    const PageEntry* page_table;
    const PageEntry* shared_pages;
    const unsigned char* pool_base;
    const GroupedWork* work;
    const int* active;
    const int* counts;
    const int* offsets;
    Unit* units_gu;
    Unit* units_dn;
    int tiles_gu, tiles_dn, tiles_per_page_gu, tiles_per_page_dn;
    int E, P, rpp_gu, rpp_dn;
    int* status;
};

__device__ __forceinline__ void build_units(const BuildUnitsArgs& b, int block, int blocks) {
    const int per = b.tiles_gu + b.tiles_dn;
    const int total = b.work->n_active * per;
    for (int i = block * blockDim.x + threadIdx.x; i < total; i += blocks * blockDim.x) {
        const int ai = i / per, r = i - ai * per;
        const bool down = r >= b.tiles_gu;
        const int tile = down ? r - b.tiles_gu : r;
        const int tpp = down ? b.tiles_per_page_dn : b.tiles_per_page_gu;
        const int half_rows = down ? 128 : 64;
        const int page = tile / tpp, tp = tile - page * tpp;
        const int e = b.active[ai];
        const PageEntry* pg = e < b.E ? b.page_table + (size_t)e * 3 * b.P : b.shared_pages;
        const PageEntry ea = pg[(down ? kSegDown : kSegGate) * b.P + page];
        const PageEntry eb = down ? ea : pg[kSegUp * b.P + page];
        Unit u;
        const bool present = ea.ptr != 0 && eb.ptr != 0;
        if (!present) flag(b.status, kStatusMissingPage);
        u.slot_a = present ? (int)((ea.ptr - (unsigned long long)b.pool_base) >> 21) : -1;
        u.slot_b = present ? (int)((eb.ptr - (unsigned long long)b.pool_base) >> 21) : -1;
        u.row0 = (short)(tp * half_rows);
        u.rows = (short)(present ? max(0, min(half_rows, (int)ea.row_count - tp * half_rows)) : 0);
        u.scales_last = (short)(ea.row_count != (down ? b.rpp_dn : b.rpp_gu));
        u.pad = 0;
        u.mrow0 = ea.row_start + tp * half_rows;
        u.n_tok = b.counts[e];
        u.pair_off = b.offsets[e];
        u.pad2 = 0;
        (down ? b.units_dn : b.units_gu)[ai * (down ? b.tiles_dn : b.tiles_gu) + tile] = u;
    }
}

// xg[p][perm(k)] = fp16(x[token(p)][k]): the tokens gathered in pair order, K order permuted per 8 columns.
__device__ __forceinline__ void gather_tokens(const void* x, int x_dtype, int x_stride, const GroupedWork* work, const unsigned short* pair_token, __half* xg,
                                              int H, int block, int blocks) {
    const int n_pairs = work->n_pairs;
    const int items = H >> 3;
    for (int p = block; p < n_pairs; p += blocks) {
        const unsigned char* row = reinterpret_cast<const unsigned char*>(x) + (size_t)pair_token[p] * x_stride;
        for (int i = threadIdx.x; i < items; i += blockDim.x) {
            float v[8];
            load_x8(row, x_dtype, i, v);
            const __half2 h0 = __floats2half2_rn(fminf(fmaxf(v[0], -65504.f), 65504.f), fminf(fmaxf(v[4], -65504.f), 65504.f));
            const __half2 h1 = __floats2half2_rn(fminf(fmaxf(v[1], -65504.f), 65504.f), fminf(fmaxf(v[5], -65504.f), 65504.f));
            const __half2 h2 = __floats2half2_rn(fminf(fmaxf(v[2], -65504.f), 65504.f), fminf(fmaxf(v[6], -65504.f), 65504.f));
            const __half2 h3 = __floats2half2_rn(fminf(fmaxf(v[3], -65504.f), 65504.f), fminf(fmaxf(v[7], -65504.f), 65504.f));
            uint4 o;
            o.x = *reinterpret_cast<const uint32_t*>(&h0);
            o.y = *reinterpret_cast<const uint32_t*>(&h1);
            o.z = *reinterpret_cast<const uint32_t*>(&h2);
            o.w = *reinterpret_cast<const uint32_t*>(&h3);
            reinterpret_cast<uint4*>(xg + (size_t)p * H)[i] = o;
        }
    }
}

// The two things that follow from the bucketing, in one launch: the first kUnitBlocks blocks list the units, the others
// gather the tokens.  (One launch after the other they cost the chain of small kernels 3 us more.)
constexpr int kUnitBlocks = 64;
__global__ void __launch_bounds__(256) prepare_step_kernel(BuildUnitsArgs b, const void* x, int x_dtype, int x_stride, const unsigned short* pair_token, __half* xg, int H) {
    pdl_wait();
    if (blockIdx.x < kUnitBlocks) build_units(b, blockIdx.x, kUnitBlocks);
    else gather_tokens(x, x_dtype, x_stride, b.work, pair_token, xg, H, blockIdx.x - kUnitBlocks, gridDim.x - kUnitBlocks);
    pdl_trigger();
}

// out[t][r] = sum over the token's slots in plan order of w * y[pair][r], then the shared expert (fp32 FMAs,
// cuda/src/kernels.cu:803-813).
__global__ void __launch_bounds__(256) combine_pairs_kernel(const __half* y, const int* pos, const float* weights, int w_stride,
                                                            int T, int top_k, int has_shared, float shared_weight, float* out,
                                                            int out_stride, int out_accumulate, int H) {
    __shared__ int sp[17];
    __shared__ float sw[17];
    pdl_wait();
    const int t = blockIdx.y;
    if ((int)threadIdx.x <= top_k) {
        const int s = threadIdx.x;
        const float* wrow = reinterpret_cast<const float*>(reinterpret_cast<const unsigned char*>(weights) + (size_t)t * w_stride);
        sp[s] = (s < top_k || has_shared) ? pos[t * (top_k + 1) + s] : -1;
        sw[s] = s < top_k ? wrow[s] : shared_weight;
    }
    __syncthreads();
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) * 2;
    if (r < H) {
        // all loads first, then the sum in plan order (the shared expert last)
        __half2 v[17];
#pragma unroll
        for (int s = 0; s < 17; ++s)
            if (s <= top_k && sp[s] >= 0) v[s] = *reinterpret_cast<const __half2*>(y + (size_t)sp[s] * H + r);
        float o0 = 0.f, o1 = 0.f;
#pragma unroll
        for (int s = 0; s < 17; ++s)
            if (s <= top_k && sp[s] >= 0) {
                o0 = fmaf(sw[s], __low2float(v[s]), o0);
                o1 = fmaf(sw[s], __high2float(v[s]), o1);
            }
        float* o = out + (size_t)t * out_stride + r;
        if (out_accumulate) {
            o[0] += o0;
            o[1] += o1;
        } else {
            o[0] = o0;
            o[1] = o1;
        }
    }
    pdl_trigger();
}

}  // namespace vib3

using namespace vib3;

extern "C" int vib3_launch_moe_layer_int4_paged(const void* x, int x_dtype, const void* page_table, int num_experts,
                                                const void* shared_pages, const unsigned short* expert_ids,
                                                const float* expert_weights, int top_k, float shared_weight,
                                                void* act_scratch, float* out, int out_accumulate, int hidden_dim,
                                                int expert_hidden_dim, int pages_per_segment,
                                                int rows_per_page_gate_up, int rows_per_page_down, int group_size,
                                                int* status, void* stream);

// ── host side ────────────────────────────────────────────────────────────────────────────────

namespace {

struct GroupedHandle {
    GroupedMaps maps;
    unsigned char* pool_base;
    size_t capacity_pages;
    int H, I, rpp_gu, rpp_dn, max_tokens, top_k, E;
    // workspace carve-up (device pointers)
    GroupedWork* work;
    int *active, *counts, *offsets, *pos;
    unsigned short* pair_token;
    __half *xg, *act, *y;
    Unit *units_gu, *units_dn;
    int tiles_gu, tiles_dn, tiles_per_page_gu, tiles_per_page_dn;
    int max_pairs;
};

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess) p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// 3-D map over the pool: x = byte in a row (row_bytes), y = row in the page (rows), z = pool slot.
int make_pool_map(CUtensorMap* m, void* base, size_t row_bytes, int rows, size_t slots, int box_x, int box_y, CUtensorMapSwizzle swizzle) {
    const cuuint64_t dims[3] = {(cuuint64_t)row_bytes, (cuuint64_t)rows, (cuuint64_t)slots};
    const cuuint64_t strides[2] = {(cuuint64_t)row_bytes, (cuuint64_t)(2u << 20)};
    const cuuint32_t box[3] = {(cuuint32_t)box_x, (cuuint32_t)box_y, 1};
    const cuuint32_t es[3] = {1, 1, 1};
    CUresult r = encode_fn()(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : VIB3_ERR_STATE;
}

// fp16 rows [rows][cols] seen as x = column within a block of 64, y = row, z = block of 64 columns; a box is 64 columns x
// box_rows x 4 blocks, 128-byte swizzle: one copy brings a slab of 256 columns as four K-major operand tiles
// [box_rows][128 bytes].
int make_rows_map(CUtensorMap* m, void* base, int cols, int rows, int box_rows) {
    const cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)(cols / 64)};
    const cuuint64_t strides[2] = {(cuuint64_t)cols * 2, 128};
    const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, (cuuint32_t)(kGrpSlabK / 64)};
    const cuuint32_t es[3] = {1, 1, 1};
    CUresult r = encode_fn()(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : VIB3_ERR_STATE;
}

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct Carve {
    size_t work, active, counts, offsets, pos, pair_token, units_gu, units_dn, xg, act, y, total;
    int tiles_gu, tiles_dn, tpp_gu, tpp_dn;
};

// tiles of a matrix of `rows` rows cut into pages of `rpp` rows, in tiles of `tile_rows`
int tiles_of(int rows, int rpp, int tile_rows, int* per_page) {
    *per_page = (rpp + tile_rows - 1) / tile_rows;
    return ((rows + rpp - 1) / rpp) * *per_page;
}

Carve carve(int max_tokens, int top_k, int E, int H, int I, int rpp_gu, int rpp_dn) {
    Carve c;
    const size_t pairs = (size_t)max_tokens * (top_k + 1);
    c.tiles_gu = tiles_of(I, rpp_gu, 64, &c.tpp_gu);
    c.tiles_dn = tiles_of(H, rpp_dn, 128, &c.tpp_dn);
    const size_t max_active = (size_t)(max_tokens * top_k < E ? max_tokens * top_k : E) + 1;
    size_t o = 0;
    c.work = o; o = align_up(o + sizeof(GroupedWork), 256);
    c.active = o; o = align_up(o + (E + 1) * sizeof(int), 256);
    c.counts = o; o = align_up(o + (E + 1) * sizeof(int), 256);
    c.offsets = o; o = align_up(o + (E + 2) * sizeof(int), 256);
    c.pos = o; o = align_up(o + pairs * sizeof(int), 256);
    c.pair_token = o; o = align_up(o + pairs * sizeof(unsigned short), 256);
    c.units_gu = o; o = align_up(o + max_active * c.tiles_gu * sizeof(Unit), 256);
    c.units_dn = o; o = align_up(o + max_active * c.tiles_dn * sizeof(Unit), 256);
    c.xg = o; o = align_up(o + pairs * (size_t)H * 2, 1024);
    c.act = o; o = align_up(o + pairs * (size_t)I * 2, 1024);
    c.y = o; o = align_up(o + pairs * (size_t)H * 2, 1024);
    c.total = o;
    return c;
}

template <class K, class... Args>
int launch_pdl(K kernel, dim3 grid, int threads, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kernel, args...);
}

constexpr int kGrpBarriers = 2 * kGrpStages + 2 * kGrpXStages + 2 * kGrpScaleStages + 8 + 5 + kGrpMmaWarps + 1;   // (+ the tensor memory address)
constexpr size_t kGrpSmem = 1024 + (size_t)kGrpStages * kGrpCodeBytes + (size_t)kGrpXStages * kGrpXBytes + (size_t)kGrpScaleStages * kGrpScaleBytes +
                            128 * (kGrpMaxN + 1) * sizeof(float) + kGrpBarriers * sizeof(uint64_t);
static_assert(kGrpSmem <= kSmemBudget, "shared memory of a CTA");

}  // namespace

extern "C" size_t vib3_moe_grouped_workspace_bytes(int max_tokens, int top_k, int num_experts, int hidden_dim, int expert_hidden_dim,
                                                   int rows_per_page_gate_up, int rows_per_page_down) {
    if (max_tokens <= 0 || top_k <= 0 || num_experts <= 0 || hidden_dim <= 0 || expert_hidden_dim <= 0 || rows_per_page_gate_up <= 0 ||
        rows_per_page_down <= 0)
        return 0;
    return carve(max_tokens, top_k, num_experts, hidden_dim, expert_hidden_dim, rows_per_page_gate_up, rows_per_page_down).total;
}

extern "C" int vib3_moe_grouped_prewarm(void* pool_base, size_t capacity_pages, int num_experts, int top_k, int hidden_dim,
                                        int expert_hidden_dim, int rows_per_page_gate_up, int rows_per_page_down,
                                        int last_page_rows_gate_up, int last_page_rows_down, int max_tokens, void* workspace,
                                        size_t workspace_bytes, void** handle_out) {
    if (!pool_base || !workspace || !handle_out) return VIB3_ERR_NULL;
    if (num_experts <= 0 || num_experts > kRouterMaxExpertsGrouped || top_k <= 0 || top_k > 16) return VIB3_ERR_COUNT;
    if (max_tokens <= 0 || max_tokens > kGrpMaxTokens) return VIB3_ERR_COUNT;
    if (hidden_dim % kGrpSlabK || expert_hidden_dim % kGrpSlabK) return VIB3_ERR_UNSUPPORTED;
    if (((uintptr_t)pool_base & 15) || ((uintptr_t)workspace & 1023)) return VIB3_ERR_ALIGN;
    if (rows_per_page_gate_up <= 0 || rows_per_page_down <= 0 || rows_per_page_gate_up > 32767 || rows_per_page_down > 32767) return VIB3_ERR_SHAPE;
    const Carve c = carve(max_tokens, top_k, num_experts, hidden_dim, expert_hidden_dim, rows_per_page_gate_up, rows_per_page_down);
    if (workspace_bytes < c.total) return VIB3_ERR_CAPACITY;
    if (!encode_fn()) return VIB3_ERR_UNSUPPORTED;
    GroupedHandle* h = new (std::nothrow) GroupedHandle();
    if (!h) return VIB3_ERR_STATE;
    unsigned char* pb = static_cast<unsigned char*>(pool_base);
    unsigned char* ws = static_cast<unsigned char*>(workspace);
    h->pool_base = pb; h->capacity_pages = capacity_pages;
    h->H = hidden_dim; h->I = expert_hidden_dim; h->rpp_gu = rows_per_page_gate_up; h->rpp_dn = rows_per_page_down;
    h->max_tokens = max_tokens; h->top_k = top_k; h->E = num_experts;
    h->work = reinterpret_cast<GroupedWork*>(ws + c.work);
    h->active = reinterpret_cast<int*>(ws + c.active);
    h->counts = reinterpret_cast<int*>(ws + c.counts);
    h->offsets = reinterpret_cast<int*>(ws + c.offsets);
    h->pos = reinterpret_cast<int*>(ws + c.pos);
    h->pair_token = reinterpret_cast<unsigned short*>(ws + c.pair_token);
    h->xg = reinterpret_cast<__half*>(ws + c.xg);
    h->act = reinterpret_cast<__half*>(ws + c.act);
    h->y = reinterpret_cast<__half*>(ws + c.y);
    h->units_gu = reinterpret_cast<Unit*>(ws + c.units_gu);
    h->units_dn = reinterpret_cast<Unit*>(ws + c.units_dn);
    h->tiles_gu = c.tiles_gu; h->tiles_dn = c.tiles_dn; h->tiles_per_page_gu = c.tpp_gu; h->tiles_per_page_dn = c.tpp_dn;
    h->max_pairs = max_tokens * (top_k + 1);
    const size_t gu_code_row = hidden_dim / 2, gu_scale_row = hidden_dim / 16;
    const size_t dn_code_row = expert_hidden_dim / 2, dn_scale_row = expert_hidden_dim / 16;
    const CUtensorMapSwizzle sw128 = CU_TENSOR_MAP_SWIZZLE_128B, sw64 = CU_TENSOR_MAP_SWIZZLE_64B;
    constexpr int kScaleBox = kGrpChunkSlabs * 16;
    int e = 0;
    e |= make_pool_map(&h->maps.gu_codes, pb, gu_code_row, rows_per_page_gate_up, capacity_pages, 128, 64, sw128);
    e |= make_pool_map(&h->maps.gu_scales_full, pb + (size_t)rows_per_page_gate_up * gu_code_row, gu_scale_row, rows_per_page_gate_up,
                       capacity_pages, kScaleBox, 64, sw64);
    e |= make_pool_map(&h->maps.gu_scales_last, pb + (size_t)last_page_rows_gate_up * gu_code_row, gu_scale_row, last_page_rows_gate_up,
                       capacity_pages, kScaleBox, 64, sw64);
    e |= make_pool_map(&h->maps.dn_codes, pb, dn_code_row, rows_per_page_down, capacity_pages, 128, 128, sw128);
    e |= make_pool_map(&h->maps.dn_scales_full, pb + (size_t)rows_per_page_down * dn_code_row, dn_scale_row, rows_per_page_down,
                       capacity_pages, kScaleBox, 128, sw64);
    e |= make_pool_map(&h->maps.dn_scales_last, pb + (size_t)last_page_rows_down * dn_code_row, dn_scale_row, last_page_rows_down,
                       capacity_pages, kScaleBox, 128, sw64);
    e |= make_rows_map(&h->maps.xg16, h->xg, hidden_dim, h->max_pairs, 16);
    e |= make_rows_map(&h->maps.act16, h->act, expert_hidden_dim, h->max_pairs, 16);
    if (e) {
        delete h;
        return VIB3_ERR_STATE;
    }
    cudaError_t ce = cudaFuncSetAttribute(moe_grouped_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGrpSmem);
    if (ce == cudaSuccess) ce = cudaFuncSetAttribute(moe_grouped_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGrpSmem);
    if (ce != cudaSuccess) {
        delete h;
        return (int)ce;
    }
    *handle_out = h;
    return VIB3_OK;
}

extern "C" void vib3_moe_grouped_destroy(void* handle) { delete static_cast<GroupedHandle*>(handle); }

extern "C" int vib3_launch_moe_grouped_int4(void* handle, const void* x, int x_dtype, int x_stride_bytes, int n_tokens,
                                            const unsigned short* ids, int ids_stride_bytes, const float* weights,
                                            int weights_stride_bytes, const void* page_table, const void* shared_pages,
                                            float shared_weight, int pages_per_segment, int expert_lo, int expert_hi, float* out,
                                            int out_stride, int out_accumulate, int* status, void* stream) {
    GroupedHandle* h = static_cast<GroupedHandle*>(handle);
    if (!h || !x || !ids || !weights || !page_table || !out) return VIB3_ERR_NULL;
    if (n_tokens <= 0 || n_tokens > h->max_tokens) return VIB3_ERR_COUNT;
    if (expert_lo < 0 || expert_hi < expert_lo || expert_hi > h->E) return VIB3_ERR_COUNT;
    if (x_dtype < X_F32 || x_dtype > X_BF16) return VIB3_ERR_UNSUPPORTED;
    if (pages_per_segment <= 0 || pages_per_segment > kMaxPages) return VIB3_ERR_COUNT;
    if (pages_per_segment * h->tiles_per_page_gu < h->tiles_gu || pages_per_segment * h->tiles_per_page_dn < h->tiles_dn) return VIB3_ERR_SHAPE;
    if (((uintptr_t)x & 15) || (x_stride_bytes & 15) || (ids_stride_bytes & 1) || (weights_stride_bytes & 3) || ((uintptr_t)out & 7) ||
        (out_stride & 1) || out_stride < h->H)
        return VIB3_ERR_ALIGN;
    cudaStream_t st = (cudaStream_t)stream;
    const int has_shared = shared_pages ? 1 : 0;
    // One token with all of its experts here: the batch-1 kernels stream the nine experts faster than tensor-core
    // tiles that are fifteen sixteenths padding.
    if (n_tokens == 1 && expert_lo == 0 && expert_hi == h->E) {
        const int e = vib3_launch_moe_layer_int4_paged(x, x_dtype, page_table, h->E, shared_pages, ids, weights, h->top_k, shared_weight,
                                                       h->act, out, out_accumulate, h->H, h->I, pages_per_segment, h->rpp_gu, h->rpp_dn,
                                                       kGroupSize, status, stream);
        if (e != VIB3_ERR_UNSUPPORTED && e != VIB3_ERR_ALIGN) return e;
    }

    GroupPairsArgs g;
    g.ids = ids; g.ids_stride = ids_stride_bytes; g.T = n_tokens; g.top_k = h->top_k; g.E = h->E; g.has_shared = has_shared;
    g.expert_lo = expert_lo; g.expert_hi = expert_hi;
    g.work = h->work; g.active = h->active; g.counts = h->counts; g.offsets = h->offsets; g.pos = h->pos;
    g.pair_token = h->pair_token; g.status = status;
    int err = launch_pdl(group_pairs_kernel, dim3(1), 1024, 0, st, g);
    if (err) return err;
    BuildUnitsArgs bu;
    bu.page_table = (const PageEntry*)page_table; bu.shared_pages = (const PageEntry*)shared_pages; bu.pool_base = h->pool_base;
    bu.work = h->work; bu.active = h->active; bu.counts = h->counts; bu.offsets = h->offsets; bu.units_gu = h->units_gu;
    bu.units_dn = h->units_dn; bu.tiles_gu = h->tiles_gu; bu.tiles_dn = h->tiles_dn; bu.tiles_per_page_gu = h->tiles_per_page_gu;
    bu.tiles_per_page_dn = h->tiles_per_page_dn; bu.E = h->E; bu.P = pages_per_segment; bu.rpp_gu = h->rpp_gu; bu.rpp_dn = h->rpp_dn;
    bu.status = status;
    err = launch_pdl(prepare_step_kernel, dim3(kUnitBlocks + min(h->max_pairs, 2 * sm_count())), 256, 0, st, bu, x, x_dtype, x_stride_bytes,
                     (const unsigned short*)h->pair_token, h->xg, h->H);
    if (err) return err;

    GroupedArgs a;
    a.work = h->work; a.act = h->act; a.y = h->y; a.units_gu = h->units_gu; a.units_dn = h->units_dn;
    a.tiles_gu = h->tiles_gu; a.tiles_dn = h->tiles_dn; a.H = h->H; a.I = h->I; a.status = status;
    err = launch_pdl(moe_grouped_kernel<false>, dim3(sm_count()), kGrpThreads, kGrpSmem, st, h->maps, a);
    if (err) return err;
    err = launch_pdl(moe_grouped_kernel<true>, dim3(sm_count()), kGrpThreads, kGrpSmem, st, h->maps, a);
    if (err) return err;
    return launch_pdl(combine_pairs_kernel, dim3((h->H / 2 + 255) / 256, n_tokens), 256, 0, st, (const __half*)h->y, (const int*)h->pos, weights,
                      weights_stride_bytes, n_tokens, h->top_k, has_shared, shared_weight, out, out_stride, out_accumulate, h->H);
}
