// Affine-Q4 GEMM on the 5th-generation tensor cores (tcgen05 + TMEM, CTA pairs), sm_100a: 17 activation rows and more.
//
// Replaces the reference's prompt path: qwen38_q4_affine_matmul_simdgroup / _simdgroup_wide
// (shaders/qwen38.metal:3769-3966), and the dequantise-whole-matrix + MPS FP16 GEMM route
// (qwen38_q4_affine_dequantize_f16, shaders/qwen38.metal:4102-4164; src/mps.rs:93-104;
// src/metal_runtime.rs:3897-4047). Arithmetic is that path's: w = 16bit(q*scale + bias), products of
// 16-bit operands, fp32 accumulation -- with bf16 where the reference uses half. No dequantised copy of the
// matrix is ever written to HBM or to shared memory: packed words go straight into tensor memory as the A operand.
//
// What bounds it, and why this shape. With both operands in shared memory a 128 x 256 x 64 stage costs 104 KB of
// shared-memory traffic (dequantised A written and read, B written and read, packed words written and read) against
// 512 cycles of MMA: 1.6 times what 128 B/clk allow, and 32 KB of activations per stage and SM from L2. Here
//   * A lives in TMEM: the dequantising warps store bf16 with tcgen05.st, one weight row per lane, and the MMA reads
//     it from there -- no shared-memory traffic at all for A;
//   * two SMs share a tile (cta_group::2): 256 weight rows x BN activation rows, each SM brings and holds half of the
//     activation tile, so shared memory and L2 see 16 KB per stage and SM instead of 32.
// A 256 x 256 x 64 stage of a pair then costs 43 KB of shared-memory traffic per SM in 512 cycles.
//
// Orientation: weights are the MMA's A operand (one weight row per TMEM lane), activations the B operand, so D[n][m]
// lands with one weight row per lane and the epilogue writes out[m][n] with the lanes of a warp on consecutive n.
// K advances 128 per stage = two affine groups (one, in the last stage of an odd number of groups).
//
// Work: all projections of a call form one list of tiles (256 weight rows x BN activation rows). A worker (CTA pair)
// takes `full_rounds` whole tiles, strided; what is left is cut along K into equal runs of stages over all workers. A
// tile cut between workers is summed, in worker order, by the one that finishes last (partial tiles in scratch, one
// counter per warp's share; nobody waits), so results do not depend on timing.
//
// Warps of a block (28):
//   0       one thread: TMA loads of this SM's half of the activation tile (bf16, 128-byte swizzle)
//   1       allocates TMEM; in the pair's first block one thread issues tcgen05.mma for both and commits
//   2       one thread: TMA loads of packed weights (two boxes of 64 rows x two groups)
//   3       idle
//   4-7     epilogue: tcgen05.ld of the accumulators, sum of a cut tile's parts, SwiGLU in pair mode, stores
//   8-23    dequantise: four groups of four warps, group g takes stages g, g+4, ...; a thread expands the 128 weights
//           of its row, 64 at a time into 32 registers that one tcgen05.st moves into TMEM
//   24-27   scales and biases: a lane reads 16 bytes of its row's parameters (four stages, any byte alignment) one
//           period ahead and lays them out in shared memory as {scale, bias} words, stage by row by group
// The instruction streams are what limits it once memory does not: a warp advances one instruction in about five
// cycles, so the MMA warp has to get along with some fifty per stage (one barrier to wait for, one commit, ring
// position and descriptors in uniform registers) and an SM's sixteen expanding warps with some 150 per group and row.
// Every wait is bounded: a wait that runs out sets an error flag, the block drains and frees its TMEM.
#include <cuda.h>

#include <algorithm>
#include <cstring>

#include "q4_decomp.h"
#include "q4_kernels.h"

#include "q4_device.cuh"

namespace q4 {

constexpr uint32_t kEpilogueWarp = 4, kDequantWarp = 8, kParamWarp = 24;
constexpr uint32_t kGemmThreads = 28 * 32;
constexpr uint32_t kGroup = 64;              // inputs of an affine group: 128 bytes of bf16, one row of a swizzled tile
constexpr uint32_t kGroupsPerStage = 2;
constexpr unsigned long long kWaitLimitNs = 2000000000ull;  // a wait gives up after two seconds
// Packed weights are staged one K stage of 128 rows at a time:
//   16-byte aligned tensors: 64-byte rows, 64-byte swizzle, so the 16-byte reads of eight lanes cover all banks;
//   any other alignment:     the tensor map starts at the address rounded down to 16 bytes and a row is an 80-byte
//                            window, unswizzled (eight lanes at a pitch of 80 cover all banks too); readers take five
//                            16-byte pieces and funnel-shift.
// The ring's length is a multiple of the four groups that read it, so a slot always belongs to the same group: a group
// that runs ahead can never wait on a slot whose previous use it has not read itself (a parity wait that is two uses
// early would succeed at once).
constexpr uint32_t kWBufs = 8, kWBoxRows = 64;
constexpr uint32_t kWAlignedPitch = 64, kWWindowPitch = 80;
constexpr uint32_t kWBufBytes = 128 * kWWindowPitch;  // 10 KB, a multiple of 1024
constexpr uint32_t kParamStages = 4;         // K stages whose scales (or biases) one 16-byte read covers
constexpr uint32_t kParamSlots = 4, kParamSlotBytes = kParamStages * 128 * 8;
constexpr uint32_t kMaxStages = 8;
constexpr uint32_t kGemmSmemBytes = 227 * 1024;  // all of an SM: one block per SM

struct GemmTensor {  // one projection (pair mode: gate and up)
    const uint8_t *s[2], *b[2];  // scales, biases per side; both sides the same tensor unless in pair mode
    float *out;                  // [m][n]
    uint32_t n;
    uint32_t row_tile;           // first row tile of this projection in the launch
    uint32_t w_misalign;         // weight address & 15
    uint32_t pad;
};

struct GemmParams {
    CUtensorMap map_x;
    CUtensorMap map_w[kMaxJobs];  // in pair mode: [0] gate, [1] up
    GemmTensor t[kMaxJobs];
    uint32_t n_jobs;
    uint32_t m, groups, k_stages;
    uint32_t bn;                 // activation rows per tile: a multiple of 32, at most 256
    uint32_t accs, stages;       // TMEM columns: accs * bn accumulators, then stages * 64 of A
    uint32_t tiles, tiles_m;     // output tiles (activation tiles innermost)
    uint32_t full_rounds, workers;   // worker w takes tiles w, w + workers, ... for full_rounds rounds
    uint32_t tail_workers;       // workers that share the K stages of the remaining tiles
    uint32_t accumulate;         // out += result
    // Pair mode (fused MLP front half, src/metal_runtime.rs:4267-4474): a tile holds 128 gate rows and the same 128 up
    // rows, interleaved over the TMEM lanes; the epilogue exchanges them between lanes and stores
    // bf16(silu(gate) * up) (qwen38_swiglu_rows, shaders/qwen38.metal:4188-4198) as h_out[m][h_stride], in the element
    // order of a prepared activation, i.e. ready to be the B operand of the down projection's GEMM.
    uint32_t pair;
    uint16_t *h_out;
    uint32_t h_stride;
    float *partials;             // [2 * tail_workers slots][2 blocks][4 warps][bn / 4][32 lanes][4]
    unsigned int *counters;      // [tail tiles][2 blocks][4 warps], zero between launches
    int *error_flag;             // set non-zero when a bounded wait runs out
};

// ---- PTX wrappers ---------------------------------------------------------------------------------

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// on a barrier of either block of the pair (address from map_to_leader)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait. Returns false (and raises the block's abort flag) when the limit is reached or another
// role has already given up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    if (mbar_try_wait(bar, parity)) return true;
    unsigned long long begin = 0;
    for (uint32_t spin = 1; spin != 0; ++spin) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((spin & 255u) == 0) {
            if (*abort_flag) return false;
            unsigned long long now;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (begin == 0) begin = now;
            if (now - begin > kWaitLimitNs) break;
        }
    }
    *abort_flag = 1;
    return false;
}
// The same for a whole warp: its lanes agree on the outcome.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag)) != 0;
}
// ... for a warp that is usually ahead of whoever it waits for: it sleeps between its polls, which leaves the issue slots
// and the barrier unit to the warps that work (twenty polling warps slowed the one that issues the MMAs by half)
__device__ __forceinline__ bool mbar_wait_idle(uint32_t bar, uint32_t parity, uint32_t ns, volatile int *abort_flag) {
    bool ok = mbar_try_wait(bar, parity);
    unsigned long long begin = 0;
    for (uint32_t spin = 1; !__all_sync(0xffffffffu, ok); ++spin) {
        __nanosleep(ns);
        ok = ok || mbar_try_wait(bar, parity);
        if ((spin & 63u) == 0) {
            unsigned long long now;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (begin == 0) begin = now;
            const bool late = now - begin > kWaitLimitNs || *abort_flag;
            if (__any_sync(0xffffffffu, late)) {
                *abort_flag = 1;
                return false;
            }
        }
    }
    return true;
}
// one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
    uint32_t on;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(on));
    return on != 0;
}
// shared::cluster address of the same shared-memory location in the pair's first block
__device__ __forceinline__ uint32_t map_to_leader(uint32_t addr) {
    uint32_t out;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(out) : "r"(addr));
    return out;
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t x, int32_t y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
        : "memory");
}
// into this block's shared memory, completion counted on a barrier of either block of the pair
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, uint32_t cluster_bar, int32_t x, int32_t y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(cluster_bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void prefetch_map(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_result, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_result), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}

// D[tmem] (+)= A[tmem] * B[smem], 256 x N x 16 over the pair, bf16 inputs, fp32 accumulate; bdesc_lo: see smem_desc_lo
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint32_t tmem_a, uint32_t bdesc_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 desc;\n\tmov.b64 desc, {%2, %5};\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], desc, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "r"(bdesc_lo), "r"(idesc), "r"(accumulate), "n"((1024u >> 4) | (1u << 14) | (2u << 29))
        : "memory");
}
// arrive on the barrier at this offset in both blocks once every MMA issued so far by this thread has completed
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .b16 both;\n\tmov.b16 both, 3;\n\t"
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], both;\n\t}" ::"r"(bar)
        : "memory");
}

// 32 lanes x 16 consecutive fp32 columns of TMEM -> 16 registers per thread
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// (the registers pass through the wait, so that nothing computes on them before it)
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                   "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}
// 32 registers per thread -> 32 lanes x 32 consecutive columns
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};" ::"r"(r[0]),
        "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
        "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major bf16 tile with 128-byte swizzle: rows are 128 bytes, groups of 8 rows (1024
// bytes) follow each other (stride byte offset 1024), descriptor version 1 (Blackwell). The low word holds the address
// (and a leading byte offset that swizzled K-major layouts do not use).
__device__ __forceinline__ uint32_t smem_desc_lo(uint32_t smem_addr) { return ((smem_addr & 0x3ffffu) >> 4) | (1u << 16); }

// two nibbles -> bf16x2 of q*scale + bias (one rounding): 0x4300|q is bf16 128+q, minus 128 is exact. The constants come in
// registers, so that mask-and-or is one three-input logic instruction.
struct DequantConstants {
    uint32_t mask, k128, one, neg128;
};
__device__ __forceinline__ DequantConstants dequant_constants() {
    DequantConstants c;
    asm volatile("mov.b32 %0, 0x000f000f;\n\tmov.b32 %1, 0x43004300;\n\tmov.b32 %2, 0x3f803f80;\n\tmov.b32 %3, 0xc300c300;"
                 : "=r"(c.mask), "=r"(c.k128), "=r"(c.one), "=r"(c.neg128));
    return c;
}
__device__ __forceinline__ uint32_t dequant_pair(uint32_t v, uint32_t scale2, uint32_t bias2, const DequantConstants &c) {
    uint32_t biased, q, out;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(biased) : "r"(v), "r"(c.mask), "r"(c.k128));  // (v & mask) | 128.0
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(q) : "r"(biased), "r"(c.one), "r"(c.neg128));
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(out) : "r"(q), "r"(scale2), "r"(bias2));
    return out;
}

// predicated 16-byte load that stays where it is written (it is issued well ahead of its use); zeros when not wanted
__device__ __forceinline__ uint4 ldg_v4_ahead(const uint8_t *p, bool pred) {
    uint4 v;
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
        "@q ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p), "r"((uint32_t)pred));
    return v;
}

// 16 bytes that start `off` (0..15) bytes into the 32 bytes {lo, hi}; unlike realign_16 the offset may differ per lane
__device__ __forceinline__ uint4 window_16(uint4 lo, uint4 hi, uint32_t off) {
    uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i] = (off & 8u) ? w[i + 2] : w[i];
#pragma unroll
    for (int i = 0; i < 5; ++i) w[i] = (off & 4u) ? w[i + 1] : w[i];
    const uint32_t sh = (off & 3u) * 8u;
    uint4 out;
    out.x = __funnelshift_r(w[0], w[1], sh);
    out.y = __funnelshift_r(w[1], w[2], sh);
    out.z = __funnelshift_r(w[2], w[3], sh);
    out.w = __funnelshift_r(w[3], w[4], sh);
    return out;
}

// ---- activation preparation: bf16, each block of 8 inputs reordered k0,k4,k1,k5,k2,k6,k3,k7 (the order the
// nibble extraction yields), so weights and activations agree on k inside every MMA ----------------------------
// (A programmatic dependent: x is read by ordinary loads after the wait. A read-only load of a pointer that promises not to alias
// may be moved up, or hit a line cached before it; loads that bypass L1 fetch every fp32 sector twice: 333 rows x 5120 57.4 -> 58.5 us
// with the GEMM behind it.)
__global__ void __launch_bounds__(256) q4_gemm_prepare_x_kernel(const void *x, int x_is_f32, uint64_t blocks, uint16_t *xp) {
    grid_dependency_wait();
    grid_dependents_launch();
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= blocks) return;
    uint32_t bits[8];
    if (x_is_f32) {
        const float4 *src = reinterpret_cast<const float4 *>(static_cast<const float *>(x) + i * 8);
        float4 lo = src[0], hi = src[1];
        const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) bits[j] = float_to_bf16_bits(v[j]);
    } else {
        uint4 raw = *reinterpret_cast<const uint4 *>(static_cast<const uint16_t *>(x) + i * 8);
        const uint32_t r[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            bits[2 * j] = r[j] & 0xffffu;
            bits[2 * j + 1] = r[j] >> 16;
        }
    }
    uint4 out;
    out.x = bits[0] | (bits[4] << 16);
    out.y = bits[1] | (bits[5] << 16);
    out.z = bits[2] | (bits[6] << 16);
    out.w = bits[3] | (bits[7] << 16);
    *reinterpret_cast<uint4 *>(xp + i * 8) = out;
}

// ---- the GEMM ------------------------------------------------------------------------------------------------

// The work items of one worker, in the order every role walks them.
struct GemmWalk {
    uint32_t worker, round, u, u_end;
    uint32_t tile, ks0, ksn;  // the current item: output tile, first K stage, number of K stages

    __device__ __forceinline__ GemmWalk(const GemmParams &p, uint32_t w) : worker(w), round(0), u(0), u_end(0) {
        const uint32_t done = p.full_rounds * p.workers;
        if (p.tiles > done && w < p.tail_workers) {
            const Q4Split split{(uint64_t)(p.tiles - done) * p.k_stages, p.k_stages, p.tail_workers};
            u = (uint32_t)q4_split_begin(split, w);
            u_end = (uint32_t)q4_split_begin(split, w + 1);
        }
    }
    __device__ __forceinline__ bool next(const GemmParams &p) {
        while (round < p.full_rounds) {
            tile = worker + round * p.workers;
            ++round;
            if (tile < p.tiles) {
                ks0 = 0;
                ksn = p.k_stages;
                return true;
            }
        }
        if (u >= u_end) return false;
        const uint32_t tt = u / p.k_stages;
        ks0 = u - tt * p.k_stages;
        ksn = min(p.k_stages - ks0, u_end - u);
        tile = p.full_rounds * p.workers + tt;
        u += ksn;
        return true;
    }
    // the projection of the current item, its first weight row in this block, and its first activation row
    __device__ __forceinline__ void locate(const GemmParams &p, uint32_t rank, uint32_t &job, uint32_t &row0, uint32_t &m0) const {
        const uint32_t rt = tile / p.tiles_m;
        m0 = (tile - rt * p.tiles_m) * p.bn;
        job = 0;
        while (job + 1 < p.n_jobs && rt >= p.t[job + 1].row_tile) ++job;
        const uint32_t local = rt - p.t[job].row_tile;
        row0 = p.pair ? local * 128u + rank * 64u : local * 256u + rank * 128u;
    }
};

// position in a ring of `size` slots and the parity of its current use
struct Ring {
    uint32_t slot, parity;
    __device__ __forceinline__ Ring() : slot(0), parity(0) {}
    __device__ __forceinline__ Ring(uint32_t count, uint32_t size) : slot(count % size), parity((count / size) & 1u) {}
    __device__ __forceinline__ void advance(uint32_t by, uint32_t size) {  // by <= size
        slot += by;
        if (slot >= size) {
            slot -= size;
            parity ^= 1u;
        }
    }
};

// TMEM lane r (0..127) of a block holds staged row `row_of_lane(r)`: the identity, or in pair mode, where staged rows 0..63
// are gate rows and 64..127 the same up rows, lanes in fours of a gate, b up, b gate, a up of eight rows (a: rows 0-3, b:
// rows 4-7), so that gate and up of a row are 12 lanes apart (xor) and eight consecutive lanes read staged rows that
// differ modulo 8 (no bank conflict in the swizzled layout).
__device__ __forceinline__ uint32_t pair_row(uint32_t r) {  // row 0..63 of either side
    const uint32_t l = r & 15u;
    const uint32_t in8 = l < 8u ? l : (l < 12u ? l - 4u : l - 12u);
    return (r >> 4) * 8u + in8;
}
__device__ __forceinline__ uint32_t pair_side(uint32_t r) { return (r >> 2) & 1u; }  // 0 gate, 1 up

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1) q4_gemm_tc_kernel(const __grid_constant__ GemmParams p) {
    extern __shared__ uint8_t gemm_smem_raw[];
    const uint32_t smem_base = ((uint32_t)__cvta_generic_to_shared(gemm_smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_generic = gemm_smem_raw + (smem_base - (uint32_t)__cvta_generic_to_shared(gemm_smem_raw));
    // barriers and flags (1 KB) | parameter ring | packed-weight ring | activation ring
    const uint32_t bars = smem_base;
    auto full = [&](uint32_t s) { return bars + 8u * s; };           // activations and A of both blocks are there (first block)
    auto empty = [&](uint32_t s) { return bars + 64u + 8u * s; };    // the MMAs have read them
    auto full_w = [&](uint32_t b) { return bars + 128u + 8u * b; };  // packed words
    auto empty_w = [&](uint32_t b) { return bars + 192u + 8u * b; };
    auto full_p = [&](uint32_t b) { return bars + 256u + 8u * b; };  // scales and biases
    auto empty_p = [&](uint32_t b) { return bars + 288u + 8u * b; };
    auto acc_full = [&](uint32_t a) { return bars + 320u + 8u * a; };
    auto acc_empty = [&](uint32_t a) { return bars + 336u + 8u * a; };  // (first block)
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem_generic + 352);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem_generic + 360);
    const uint32_t param_ring = smem_base + 1024u;
    const uint32_t w_ring = param_ring + kParamSlots * kParamSlotBytes;
    const uint32_t x_ring = w_ring + kWBufs * kWBufBytes;  // kWBufBytes is a multiple of 1024
    const uint32_t x_group_bytes = p.bn * 64u;               // this block's half of one group: bn / 2 rows of 128 bytes

    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31u;  // (uniform register)
    const uint32_t rank = cluster_rank(), worker = blockIdx.x >> 1;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kMaxStages; ++s) {
            mbar_init(full(s), 9);   // four warps of either block; the first block's expect_tx for the bytes of both
            mbar_init(empty(s), 1);  // tcgen05.commit
        }
        for (uint32_t s = 0; s < kWBufs; ++s) {
            mbar_init(full_w(s), 1);
            mbar_init(empty_w(s), 4);  // the warps of the group that reads the stage
        }
        for (uint32_t s = 0; s < kParamSlots; ++s) {
            mbar_init(full_p(s), 4);
            mbar_init(empty_p(s), 16);
        }
        for (uint32_t a = 0; a < 2; ++a) {
            mbar_init(acc_full(a), 1);
            mbar_init(acc_empty(a), 8);  // four epilogue warps of either block
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc_pair(bars + 352u, 512);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_a = tmem_base + p.accs * p.bn;
    const uint32_t leader_bars = map_to_leader(bars);  // the first block's barriers, as cluster addresses

    GemmWalk walk(p, worker);
    uint32_t job, row0, m0;

    if (warp == 0) {
        // ---- TMA producer: activations ----
        grid_dependency_wait();
        grid_dependents_launch();
        Ring ring;
        bool ok = true;
        while (ok && walk.next(p)) {
            walk.locate(p, rank, job, row0, m0);
            const int32_t y = (int32_t)(m0 + rank * (p.bn / 2u));
            for (uint32_t i = 0; i < walk.ksn; ++i) {
                if (!mbar_wait_warp(empty(ring.slot), ring.parity ^ 1u, abort_flag)) { ok = false; break; }
                const uint32_t g0 = (walk.ks0 + i) * kGroupsPerStage;
                const bool two = g0 + 1u < p.groups;
                const uint32_t dst = x_ring + ring.slot * kGroupsPerStage * x_group_bytes, bar = leader_bars + 8u * ring.slot;
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(full(ring.slot), (two ? 4u : 2u) * x_group_bytes);
                    tma_load_2d_pair(dst, &p.map_x, bar, (int32_t)(g0 * kGroup), y);
                    if (two) tma_load_2d_pair(dst + x_group_bytes, &p.map_x, bar, (int32_t)((g0 + 1u) * kGroup), y);
                }
                __syncwarp();
                ring.advance(1, p.stages);
            }
        }
        // every signal that is still on its way to this block's barriers arrives before the block leaves
        for (uint32_t i = 0; i < p.stages && ok; ++i) {
            ok = mbar_wait_warp(empty(ring.slot), ring.parity ^ 1u, abort_flag);
            ring.advance(1, p.stages);
        }
        if (!ok) __nanosleep(50000);  // copies in flight land in shared memory first
    } else if (warp == 1) {
        // ---- MMA issuer: the warp stays converged, so that ring positions and descriptors live in uniform registers ----
        if (rank == 0) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((p.bn >> 3) << 17) | (16u << 24);  // f32 += bf16 x bf16, N = bn, M = 256
            const uint32_t x_desc = smem_desc_lo(x_ring), group_step = x_group_bytes >> 4;
            Ring ring, accr;
            bool ok = true;
            while (ok && walk.next(p)) {
                if (!mbar_wait_warp(acc_empty(accr.slot), accr.parity ^ 1u, abort_flag)) break;
                tc_fence_after();
                const uint32_t d = tmem_base + accr.slot * p.bn;
                for (uint32_t i = 0; i < walk.ksn; ++i) {
                    const bool two = (walk.ks0 + i) * kGroupsPerStage + 1u < p.groups;
                    const uint32_t a = tmem_a + ring.slot * 64u, b = x_desc + ring.slot * kGroupsPerStage * group_step;
                    if (!mbar_wait_warp(full(ring.slot), ring.parity, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (uint32_t k16 = 0; k16 < kGroup / 16; ++k16)  // 16 inputs: 8 columns of A, 32 bytes of the B rows
                            umma_bf16_pair(d, a + 8u * k16, b + 2u * k16, idesc, k16 == 0 ? i : 1u);
                        if (two) {
#pragma unroll
                            for (uint32_t k16 = 0; k16 < kGroup / 16; ++k16)
                                umma_bf16_pair(d, a + 32u + 8u * k16, b + group_step + 2u * k16, idesc, 1u);
                        }
                        umma_commit_pair(empty(ring.slot));
                    }
                    __syncwarp();
                    ring.advance(1, p.stages);
                }
                if (ok && elect_one()) umma_commit_pair(acc_full(accr.slot));
                __syncwarp();
                accr.advance(1, p.accs);
            }
        }
    } else if (warp == 2) {
        // ---- TMA producer: packed weights. They are requested (and parameters read) before this kernel's wait: the kernel in
        // front is always the preparation or another GEMM of the same call, which writes no weights and lets this one start
        // only after its own wait, when everything before the call is complete ----
        Ring ring;
        bool ok = true;
        while (ok && walk.next(p)) {
            walk.locate(p, rank, job, row0, m0);
            const CUtensorMap *map0 = &p.map_w[job], *map1 = p.pair ? &p.map_w[1] : map0;
            const uint32_t half = kWBoxRows * (p.t[job].w_misalign ? kWWindowPitch : kWAlignedPitch);
            const int32_t row1 = (int32_t)(p.pair ? row0 : row0 + kWBoxRows);
            for (uint32_t i = 0; i < walk.ksn; ++i) {
                if (!mbar_wait_warp(empty_w(ring.slot), ring.parity ^ 1u, abort_flag)) { ok = false; break; }
                // x is a byte offset from the (rounded-down) tensor base: a multiple of 64
                const int32_t x = (int32_t)((walk.ks0 + i) * 64u);
                const uint32_t dst = w_ring + ring.slot * kWBufBytes;
                if (elect_one()) {
                    mbar_expect_tx(full_w(ring.slot), 2u * half);
                    tma_load_2d(dst, map0, full_w(ring.slot), x, (int32_t)row0);
                    tma_load_2d(dst + half, map1, full_w(ring.slot), x, row1);
                }
                __syncwarp();
                ring.advance(1, kWBufs);
            }
        }
        if (!ok) __nanosleep(50000);
    } else if (warp >= kEpilogueWarp && warp < kDequantWarp) {
        // ---- epilogue ----
        grid_dependency_wait();
        const uint32_t quarter = warp & 3u;  // a warp may touch TMEM lanes 32 * (warp % 4) .. + 31
        const uint32_t r = quarter * 32u + lane;
        const uint32_t done = p.full_rounds * p.workers;
        const Q4Split split{(uint64_t)(p.tiles > done ? p.tiles - done : 1u) * p.k_stages, p.k_stages, p.tail_workers ? p.tail_workers : 1u};
        Ring accr;
        while (walk.next(p)) {
            walk.locate(p, rank, job, row0, m0);
            if (!mbar_wait_idle(acc_full(accr.slot), accr.parity, 200, abort_flag)) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((quarter * 32u) << 16) + accr.slot * p.bn;
            const uint32_t cols = min(p.bn, p.m - m0);
            const GemmTensor &T = p.t[job];
            const bool cut = walk.ksn != p.k_stages;
            uint32_t first = 0, last = 0;
            bool store = true;
            const size_t slot_floats = (size_t)p.bn * 256u;  // both blocks' rows of a slot
            float *const mine = p.partials + (size_t)rank * p.bn * 128u + (size_t)quarter * p.bn * 32u + lane * 4u;
            const uint32_t tt = walk.tile - done;
            if (cut) {
                // this worker's part of the tile goes to scratch; whoever counts last adds all parts in worker order
                q4_split_contributors(split, tt, &first, &last);
                float *dst = mine + q4_split_slot(split, worker, tt) * slot_floats;
#pragma unroll 1
                for (uint32_t c0 = 0; c0 < cols; c0 += 16, dst += 16 * 32) {
                    uint32_t v[16];
                    tmem_ld_32x16(taddr + c0, v);
                    tmem_ld_wait(v);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        __stcg(reinterpret_cast<uint4 *>(dst + i * 128), make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
                }
                __threadfence();
                __syncwarp();
                unsigned int before = 0;
                unsigned int *counter = p.counters + tt * 8u + rank * 4u + quarter;
                if (lane == 0) before = atomicAdd(counter, 1u);
                before = __shfl_sync(0xffffffffu, before, 0);
                store = before == last - first;
                if (store) {
                    __threadfence();
                    if (lane == 0) *counter = 0;  // ready for the next launch
                }
            }
            // 16 columns of a cut tile: the sum of its parts
            auto summed = [&](uint32_t c0, uint32_t (&v)[16]) {
                float f[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) f[i] = 0.f;
                for (uint32_t w = first; w <= last; ++w) {
                    const float *src = mine + q4_split_slot(split, w, tt) * slot_floats + (size_t)c0 * 32u;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4 q = __ldcg(reinterpret_cast<const float4 *>(src + i * 128));
                        f[4 * i] += q.x;
                        f[4 * i + 1] += q.y;
                        f[4 * i + 2] += q.z;
                        f[4 * i + 3] += q.w;
                    }
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(f[i]);
            };
            // all columns, 16 at a time; the next 16 are on their way from TMEM while `emit` works
            auto each16 = [&](auto &&emit) {
                uint32_t v0[16], v1[16];
                if (cut) {
#pragma unroll 1
                    for (uint32_t c0 = 0; c0 < cols; c0 += 16) {
                        summed(c0, v0);
                        emit(c0, v0);
                    }
                    return;
                }
                tmem_ld_32x16(taddr, v0);
#pragma unroll 1
                for (uint32_t c0 = 0; c0 < cols; c0 += 32) {
                    __syncwarp();
                    tmem_ld_wait(v0);
                    tmem_ld_32x16(taddr + c0 + 16u, v1);  // (bn is a multiple of 32)
                    emit(c0, v0);
                    __syncwarp();
                    tmem_ld_wait(v1);
                    if (c0 + 32u < cols) tmem_ld_32x16(taddr + c0 + 32u, v0);
                    emit(c0 + 16u, v1);
                }
            };
            if (store && p.pair) {
                // two columns at a time: a gate lane takes up of column i from its partner, an up lane gate of column i + 1
                const bool gate_lane = pair_side(r) == 0;
                const uint32_t n = row0 + pair_row(r);
                // inside each block of 8 inputs of a prepared activation the order is k0,k4,k1,k5,k2,k6,k3,k7
                const uint32_t pos = (n & ~7u) | ((n & 3u) << 1) | ((n >> 2) & 1u);
                uint16_t *dst = p.h_out + (size_t)(m0 + (gate_lane ? 0u : 1u)) * p.h_stride + pos;
                const uint32_t mine_cols = n < T.n ? (cols + (gate_lane ? 1u : 0u)) / 2u : 0u;  // columns of this lane's parity
                each16([&](uint32_t c0, const uint32_t (&v)[16]) {
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        const float other = __uint_as_float(__shfl_xor_sync(0xffffffffu, gate_lane ? v[i + 1] : v[i], 12));
                        const float g = gate_lane ? __uint_as_float(v[i]) : other, u = gate_lane ? other : __uint_as_float(v[i + 1]);
                        // hardware exponential and reciprocal (as Metal's fast math in the reference's kernel): their
                        // error is far below the bf16 rounding that follows
                        const float h = __fdividef(g, 1.0f + __expf(-g)) * u;
                        if (c0 / 2u + i / 2u < mine_cols) *dst = (uint16_t)float_to_bf16_bits(h);
                        dst += 2u * (size_t)p.h_stride;
                    }
                });
            } else if (store) {
                const uint32_t n = row0 + r;
                float *dst = T.out + (size_t)m0 * T.n + n;
                const size_t step = T.n;
                const uint32_t mine_cols = n < T.n ? cols : 0u;
                each16([&](uint32_t c0, const uint32_t (&v)[16]) {
                    if (p.accumulate) {
                        float old[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) old[i] = c0 + i < mine_cols ? dst[i * step] : 0.f;
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (c0 + i < mine_cols) dst[i * step] = __uint_as_float(v[i]) + old[i];
                    } else if (c0 + 16u <= mine_cols) {
                        float *q = dst;
#pragma unroll
                        for (int i = 0; i < 16; ++i, q += step) *q = __uint_as_float(v[i]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (c0 + i < mine_cols) dst[i * step] = __uint_as_float(v[i]);
                    }
                    dst += 16 * step;
                });
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(leader_bars + 336u + 8u * accr.slot);
            accr.advance(1, p.accs);
        }
    } else if (warp >= kDequantWarp && warp < kParamWarp) {
        // ---- dequantise ----
        const uint32_t group = (warp - kDequantWarp) >> 2;
        const uint32_t r = (warp & 3u) * 32u + lane;  // TMEM lane
        const uint32_t row = p.pair ? pair_side(r) * 64u + pair_row(r) : r;  // staged row
        const uint32_t a_addr = tmem_a + (((warp & 3u) * 32u) << 16);
        const DequantConstants magic = dequant_constants();
        uint32_t count = 0;  // stages of the items so far; this group takes those whose overall number is `group` modulo 4
        Ring pr, wr(group, kWBufs), sr(group, p.stages);
        bool ok = true;
        while (ok && walk.next(p)) {
            walk.locate(p, rank, job, row0, m0);
            const uint32_t mis = p.t[job].w_misalign;
            const uint32_t row_at = w_ring + row * (mis ? kWWindowPitch : kWAlignedPitch);
            uint32_t i = (group - count) & 3u;  // local number of the group's first stage
            const uint32_t param_at = param_ring + (i * 128u + r) * 8u;
            count += walk.ksn;
            for (; i < walk.ksn; i += 4u) {
                if (!mbar_wait_warp(full_w(wr.slot), wr.parity, abort_flag)) { ok = false; break; }
                const uint32_t at = row_at + wr.slot * kWBufBytes;
                uint4 q[4];  // 32 weights each
                if (mis == 0) {
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) q[j] = lds_v4(at + ((j ^ ((row >> 1) & 3u)) << 4));
                } else {
                    const uint4 w0 = lds_v4(at), w1 = lds_v4(at + 16u), w2 = lds_v4(at + 32u), w3 = lds_v4(at + 48u), w4 = lds_v4(at + 64u);
                    q[0] = realign_16(w0, w1, mis);
                    q[1] = realign_16(w1, w2, mis);
                    q[2] = realign_16(w2, w3, mis);
                    q[3] = realign_16(w3, w4, mis);
                }
                if (!mbar_wait_warp(full_p(pr.slot), pr.parity, abort_flag)) { ok = false; break; }
                const uint2 pv = lds_v2(param_at + pr.slot * kParamSlotBytes);
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(empty_w(wr.slot));
                    mbar_arrive(empty_p(pr.slot));
                }
                wr.advance(4u, kWBufs);
                pr.advance(1u, kParamSlots);
                const bool two = (walk.ks0 + i) * kGroupsPerStage + 1u < p.groups;
#pragma unroll
                for (uint32_t half = 0; half < 2; ++half) {
                    const uint32_t sc = __byte_perm(half ? pv.y : pv.x, 0u, 0x1010u), bi = __byte_perm(half ? pv.y : pv.x, 0u, 0x3232u);
                    const uint4 &lo = q[2 * half], &hi = q[2 * half + 1];
                    const uint32_t words[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                    uint32_t o[32];
#pragma unroll
                    for (int w = 0; w < 8; ++w) {
                        o[4 * w] = dequant_pair(words[w], sc, bi, magic);
                        o[4 * w + 1] = dequant_pair(words[w] >> 4, sc, bi, magic);
                        o[4 * w + 2] = dequant_pair(words[w] >> 8, sc, bi, magic);
                        o[4 * w + 3] = dequant_pair(words[w] >> 12, sc, bi, magic);
                    }
                    if (half == 0) {
                        if (!mbar_wait_idle(empty(sr.slot), sr.parity ^ 1u, 40, abort_flag)) { ok = false; break; }
                        tc_fence_after();
                    }
                    if (half == 0 || two) tmem_st_32x32(a_addr + sr.slot * 64u + half * 32u, o);
                }
                if (!ok) break;
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(leader_bars + 8u * sr.slot);
                sr.advance(4u, p.stages);
            }
            // a stage that the item's last parameter period does not have is counted as read
            if (ok && i / kParamStages < (walk.ksn + kParamStages - 1u) / kParamStages) {
                ok = mbar_wait_warp(full_p(pr.slot), pr.parity, abort_flag);
                if (ok && lane == 0) mbar_arrive(empty_p(pr.slot));
                pr.advance(1u, kParamSlots);
            }
        }
    } else if (warp >= kParamWarp) {
        // ---- scales and biases ----
        const uint32_t r = (warp - kParamWarp) * 32u + lane;
        const uint32_t side = p.pair ? pair_side(r) : 0u;
        const uint32_t row_in = p.pair ? pair_row(r) : r;
        struct Fetched {
            uint4 s_lo, s_hi, b_lo, b_hi;
        };
        Ring pr;
        bool ok = true;
        while (ok && walk.next(p)) {
            walk.locate(p, rank, job, row0, m0);
            const GemmTensor &T = p.t[job];
            const uint32_t row = min(row0 + row_in, T.n - 1u);  // rows past n take a valid row's parameters and are never stored
            const size_t at = ((size_t)row * p.groups + walk.ks0 * kGroupsPerStage) * 2u;
            const uint8_t *sp = T.s[side] + at, *bp = T.b[side] + at;
            const uint32_t s_off = (uint32_t)(uintptr_t)sp & 15u, b_off = (uint32_t)(uintptr_t)bp & 15u;
            sp -= s_off;
            bp -= b_off;
            const uint32_t periods = (walk.ksn + kParamStages - 1u) / kParamStages;
            // (reads at most 31 bytes past the parameters of the item's last stage: shards are padded for that)
            auto fetch = [&](Fetched &f, uint32_t t) {
                const bool in = t < periods;
                f.s_lo = ldg_v4_ahead(sp + t * 16u, in);
                f.s_hi = ldg_v4_ahead(sp + t * 16u + 16u, in && s_off != 0);
                f.b_lo = ldg_v4_ahead(bp + t * 16u, in);
                f.b_hi = ldg_v4_ahead(bp + t * 16u + 16u, in && b_off != 0);
            };
            auto deliver = [&](const Fetched &f) {
                const uint4 s4 = window_16(f.s_lo, f.s_hi, s_off), b4 = window_16(f.b_lo, f.b_hi, b_off);
                if (!mbar_wait_idle(empty_p(pr.slot), pr.parity ^ 1u, 200, abort_flag)) return false;
                const uint32_t dst = param_ring + pr.slot * kParamSlotBytes + r * 8u;
                const uint32_t sw[4] = {s4.x, s4.y, s4.z, s4.w}, bw[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                for (int j = 0; j < 4; ++j)  // a stage: {scale, bias} of its two groups
                    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(dst + j * 1024u), "r"(__byte_perm(sw[j], bw[j], 0x5410u)),
                                 "r"(__byte_perm(sw[j], bw[j], 0x7632u))
                                 : "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(full_p(pr.slot));
                pr.advance(1u, kParamSlots);
                return true;
            };
            Fetched f0, f1;
            fetch(f0, 0);
            for (uint32_t t = 0; t < periods && ok; t += 2) {
                fetch(f1, t + 1);
                ok = deliver(f0);
                if (ok && t + 1 < periods) {
                    fetch(f0, t + 2);
                    ok = deliver(f1);
                }
            }
        }
    }

    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // neither block leaves while the other may still signal its barriers or read its shared memory
    tc_fence_after();
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
    if (threadIdx.x == 0 && *abort_flag && p.error_flag) *p.error_flag = 1;
}

}  // namespace q4

// ---------------------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------------------

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
    static const EncodeTiledFn fn = [] {
        void *sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            return reinterpret_cast<EncodeTiledFn>(sym);
        return static_cast<EncodeTiledFn>(nullptr);
    }();
    return fn;
}

// packed weights as a byte matrix [n][k/2] from the tensor's address rounded down to 16 bytes (TMA needs that;
// the row pitch k/2 is a multiple of 32): 64-byte swizzled rows when the tensor is aligned, 80-byte windows else.
// The matrix is declared 16 bytes wider than k/2 in the window form so the last window of a row is in range; the
// extra bytes are the next row's first bytes or, after the last row, the padding every shard carries.
bool encode_weight_map(EncodeTiledFn encode, CUtensorMap *wmap, const uint8_t *w, uint32_t n, uint32_t k) {
    const uint32_t w_mis = (uint32_t)((uintptr_t)w & 15u);
    const cuuint64_t wdims[2] = {(cuuint64_t)k / 2 + (w_mis ? 16u : 0u), n};
    const cuuint64_t wstrides[1] = {(cuuint64_t)k / 2};
    const cuuint32_t wbox[2] = {w_mis ? q4::kWWindowPitch : q4::kWAlignedPitch, (cuuint32_t)q4::kWBoxRows};
    const cuuint32_t estr[2] = {1, 1};
    return encode(wmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t *>(w - w_mis), wdims, wstrides, wbox, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, w_mis ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_64B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool encode_activation_map(EncodeTiledFn encode, CUtensorMap *map, const uint16_t *xp, uint32_t m, uint32_t k, uint32_t box_rows) {
    const cuuint64_t dims[2] = {k, m};
    const cuuint64_t strides[1] = {(cuuint64_t)k * 2};
    const cuuint32_t box[2] = {(cuuint32_t)q4::kGroup, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t *>(xp), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

extern "C" cudaError_t q4k_gemm_prepare_x(const void *x, int x_is_f32, uint64_t elements, uint16_t *xp, cudaStream_t stream) {
    const uint64_t blocks = elements / 8;
    return q4::launch_dependent(q4::q4_gemm_prepare_x_kernel, dim3((uint32_t)((blocks + 255) / 256)), 256, 0, stream, x, x_is_f32, blocks, xp);
}

// xp: prepared activations [m][k] bf16 (q4k_gemm_prepare_x), 16-byte aligned. Up to kMaxJobs projections in one launch,
// planned by q4_gemm_plan for their row tiles. With `h_out` the two jobs are gate and up of a fused MLP (equal n, equal
// weight offset from a 16-byte boundary): h[m][n] = bf16(silu(x gate^T) * (x up^T)) in the element order of a prepared
// activation, rows h_stride elements apart (16-byte aligned). partials / counters: scratch of the plan's sizes.
extern "C" cudaError_t q4k_gemm_tc(const Q4GemmPlan *plan, const uint16_t *xp, uint32_t m, uint32_t k, const q4::GemmJob *jobs,
                                   uint32_t n_jobs, uint16_t *h_out, uint32_t h_stride, int accumulate, int *error_flag,
                                   float *partials, unsigned int *counters, cudaStream_t stream) {
    EncodeTiledFn encode = encode_tiled_fn();
    if (!encode) return cudaErrorNotSupported;
    if (n_jobs == 0 || n_jobs > (uint32_t)q4::kMaxJobs) return cudaErrorInvalidValue;
    q4::GemmParams p;
    memset(&p, 0, sizeof p);
    if (!encode_activation_map(encode, &p.map_x, xp, m, k, plan->bn / 2)) return cudaErrorInvalidValue;
    for (uint32_t i = 0; i < n_jobs; ++i)
        if (!encode_weight_map(encode, &p.map_w[i], jobs[i].w, jobs[i].n, k)) return cudaErrorInvalidValue;
    uint32_t row_tiles = 0;
    if (h_out) {
        if (n_jobs != 2 || jobs[0].n != jobs[1].n || !q4k_gemm_pair_supported(jobs[0].w, jobs[1].w)) return cudaErrorInvalidValue;
        p.pair = 1;
        p.h_out = h_out;
        p.h_stride = h_stride;
        p.n_jobs = 1;
    } else {
        p.n_jobs = n_jobs;
    }
    for (uint32_t i = 0; i < p.n_jobs; ++i) {
        q4::GemmTensor &t = p.t[i];
        const q4::GemmJob &other = p.pair ? jobs[1] : jobs[i];
        t.s[0] = jobs[i].s;
        t.b[0] = jobs[i].b;
        t.s[1] = other.s;
        t.b[1] = other.b;
        t.out = jobs[i].out;
        t.n = jobs[i].n;
        t.row_tile = row_tiles;
        t.w_misalign = (uint32_t)((uintptr_t)jobs[i].w & 15u);
        row_tiles += q4_gemm_row_tiles(jobs[i].n, p.pair);
    }
    if (row_tiles * plan->tiles_m != plan->tiles) return cudaErrorInvalidValue;
    p.m = m;
    p.groups = k / 64;
    p.k_stages = q4_gemm_k_stages(k);
    p.bn = plan->bn;
    p.accs = plan->accs;
    p.stages = plan->stages;
    p.tiles = plan->tiles;
    p.tiles_m = plan->tiles_m;
    p.full_rounds = plan->full_rounds;
    p.workers = plan->workers;
    p.tail_workers = plan->tail_workers;
    p.accumulate = accumulate ? 1u : 0u;
    p.partials = partials;
    p.counters = counters;
    p.error_flag = error_flag;
    static_assert(1024u + 1024u + q4::kParamSlots * q4::kParamSlotBytes + q4::kWBufs * q4::kWBufBytes + 4u * 256u * 128u <= q4::kGemmSmemBytes, "shared memory");
    if (p.stages > q4::kMaxStages || p.stages * p.bn > 1024u) return cudaErrorInvalidValue;  // (activation ring: at most four stages of 256 rows)
    const cudaError_t e = cudaFuncSetAttribute(q4::q4_gemm_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)q4::kGemmSmemBytes);
    if (e != cudaSuccess) return e;
    return q4::launch_dependent(q4::q4_gemm_tc_kernel, dim3(2u * p.workers), q4::kGemmThreads, q4::kGemmSmemBytes, stream, p);
}

// 1 when the gate and up tensors can share one pair launch: the staged weight tiles of a projection have one geometry, so
// both tensors must sit at the same offset from a 16-byte boundary
extern "C" int q4k_gemm_pair_supported(const uint8_t *w_gate, const uint8_t *w_up) {
    return (((uintptr_t)w_gate ^ (uintptr_t)w_up) & 15u) == 0 ? 1 : 0;
}
