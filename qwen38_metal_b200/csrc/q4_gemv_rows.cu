// Short batches (2..16 activation rows) of MLX affine-Q4 projections on the integer tensor-core path: the shape of the
// reference's batched kernels (qwen38_q4_affine_matvec_batch2/4/8, shaders/qwen38.metal:213-246 applied per row),
// HBM-bound on B200 because every packed weight is read once for all rows.
//
// Arithmetic. Every affine group (64 inputs) of an activation row is held as 23-bit fixed point after an exact
// power-of-two scaling by the group's own largest magnitude, x' = d0 + 256 d1 + 65536 d2 with signed 8-bit digits. A
// packed weight word becomes two byte registers (even and odd nibbles) and is the A operand of mma.sync.m16n8k32.s32.u8.s8 as it is; the B operand holds one digit of eight
// activation rows, so one MMA returns, for 16 weight rows and 8 activation rows, the exact integer sum of
// q * digit over 32 inputs. An affine group (64 inputs) is two MMAs per digit; its three integer sums are
// put together (q0 + 256 q1 + 65536 q2, the group's exact integer dot product, rounded to fp32 once), the power of two is
// undone and the sum is scaled with the group's bf16 scale in fp32; the bias term is bias * (sum of x' over the group).
// Products and group sums are exact; the approximations are the fixed-point step of the activation (2^-22 of the largest
// of 64 neighbours, the last bit of an fp32 number of that size) and fp32 rounding of the per-group terms, as in the
// reference. A group that holds an infinity or a NaN makes every result of its row NaN.
//
// Up to four rows (DC) the three digits of two rows share one B operand -- columns 0..2 hold the digits of the first row,
// 4..6 those of the second -- instead of one digit of eight rows each: 2 MMAs per group and pair of rows where the form
// above takes 6 for up to eight.
//
// Work. The K range is cut into `parts` runs of 128-input chunks. A block holds the digits of ONE part for all rows
// in shared memory (converted by the block itself from the caller's bf16 or fp32 rows). A part's work is the list of its
// 16-row tiles (pairs of them when TW = 2) times its quads of four chunks; every warp of the part's blocks takes the same
// number of consecutive quads, wherever in a tile that begins and ends, so no warp has a round more than another one.
// A warp's quads run through ONE private ring of cp.async stages that never drains between tiles. A tile that several
// warps share goes through scratch; the LAST of them (one counter per tile, put back to zero by that warp) adds all
// contributions in K order -- the result does not depend on which one came last -- and stores the tile. No block
// ever waits for another one.
//
// Tensors at any byte offset (MIS). A shard's tensors start where its header put them, so the weights of a launch may miss
// a 16-byte boundary (all rows of a tensor by the same amount: a row is a multiple of 32 bytes) and so may the scales and
// biases (every row by its own amount when the number of groups is not a multiple of eight). The copies then fetch the
// aligned 16-byte windows that hold bytes of the row: a lane's 8 bytes come out of two neighbouring 8-byte words and a
// funnel shift, and the last words of a chunk lie in the first window of the next one, which is the next ring stage.
// The instance without MIS keeps the shorter loop for launches whose tensors are all aligned.
//
// Launches are programmatic dependents of whatever runs in front of them: a block requests its first weights -- which no
// kernel that lets a dependent start early ever writes -- and only then waits for the kernel before it.
// What bounds it and what was measured (B200, calls back to back, before -> after the byte-addressed instance, the shared
// B operands, the ring that does not drain and the dependent launch): 8 fp32 rows x 8192 x 5120 at a byte offset 131 -> 18.9 us
// (was: four launch pairs of the fp16 kernel), 4 rows x 34816 x 5120 35.0 -> 27.5 us (3.6 TB/s), 4 rows x 248320 x 5120 with
// the argmax 205 -> 173 us (4.1 TB/s), one accumulating fp32 row x 5120 x 17408 at a byte offset 47.1 -> 21.5 us. Small
// calls are bound by launch, conversion and the first round trips, long ones by the warps' instruction issue.
#include "q4_decomp.h"
#include "q4_device.cuh"
#include "q4_kernels.h"

namespace q4 {

constexpr int kRowsWarps = 16;
constexpr int kRowsStageBytes = 1024;  // one chunk of one tile: 16 weight rows x 64 packed bytes
constexpr int kRowsPerThread = 8;      // blocks of 8 inputs a thread converts at most (bounds a part: rows x chunks <= 256)
constexpr uint32_t kRowsPairColumns = 4;  // up to this many rows share B operands in pairs

// A warp walks TW tiles at a time (1 or 2): with two, the B fragments (activation digits) are read from shared memory
// once for 32 weight rows. The ring of a warp is 8 KB either way: 8 stages of one chunk, or 4 stages of a chunk of both
// tiles. Scales and biases travel per four chunks (16 rows x 2 arrays x 16 bytes per tile): three such stages cover
// the 7 chunks a one-tile warp is ahead, two the 3 chunks of a two-tile warp.
__host__ __device__ constexpr uint32_t rows_stages(uint32_t tw) { return 8u / tw; }
__host__ __device__ constexpr uint32_t rows_param_stages(uint32_t tw) { return tw == 1u ? 3u : 2u; }
// parameters of one tile and four chunks: a 16-byte window per row and array, two of them when they may start anywhere
__host__ __device__ constexpr uint32_t rows_param_bytes(bool mis) { return mis ? 1024u : 512u; }
__host__ __device__ constexpr uint32_t rows_ring_bytes(uint32_t tw, bool mis) { return 8u * kRowsStageBytes + rows_param_stages(tw) * rows_param_bytes(mis) * tw; }

__host__ __device__ constexpr bool rows_dc(uint32_t m) { return m <= kRowsPairColumns; }
__host__ __device__ constexpr uint32_t rows_padded(uint32_t m) { return rows_dc(m) ? (m + 1u) & ~1u : (m + 7u) & ~7u; }

// Shared memory of one chunk's digits: [group 2][digit 3][activation row MP][64 bytes], DC: [group 2][row MP][digit 3][64 bytes]. The 64 bytes of a (group, digit,
// row) hold the 64 inputs of the group in the order lane t of a quad wants them as B registers of the group's two MMAs:
// byte 16 t + 8 j + 4 odd + i  <->  input 16 t + 8 j + 2 i + odd   (t: quad lane, j: MMA of the group, i: byte).
__host__ __device__ constexpr uint32_t rows_chunk_bytes(uint32_t mp) { return 2u * 3u * mp * 64u; }

// beside the digits: {sum of x', 2^-e} of every group and row, rows in pairs: {sum, sum, 2^-e, 2^-e}; DC: what a lane
// multiplies digits 0 and 1 with and what digit 2: {sum, 2^-e, 0, 2^(16-e)}
__host__ __device__ constexpr uint32_t rows_scale_bytes(bool dc) { return dc ? 16u : 8u; }
__host__ __device__ inline size_t rows_smem_bytes(uint32_t mp, uint32_t part_chunks, uint32_t tw, bool mis, bool dc) {
    return (size_t)kRowsWarps * rows_ring_bytes(tw, mis) + (size_t)part_chunks * (rows_chunk_bytes(mp) + 2u * mp * rows_scale_bytes(dc));
}

// Sums are carried 2^12 too small: a group's sum over 64 inputs times 0..15 of the largest fp32 numbers stays finite.
constexpr float kRowsSumScale = 1.0f / 4096.0f;

// 16 bytes starting `mis` (0..15, any value per lane) bytes into the 32-byte window {lo, hi}
__device__ __forceinline__ uint4 realign_16_any(const uint4 &lo, const uint4 &hi, uint32_t mis) {
    const bool by8 = (mis & 8u) != 0, by4 = (mis & 4u) != 0;
    const uint32_t w[6] = {by8 ? lo.z : lo.x, by8 ? lo.w : lo.y, by8 ? hi.x : lo.z, by8 ? hi.y : lo.w, by8 ? hi.z : hi.x, by8 ? hi.w : hi.y};
    uint32_t v[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) v[i] = by4 ? w[i + 1] : w[i];
    const uint32_t sh = (mis & 3u) * 8u;
    return make_uint4(__funnelshift_r(v[0], v[1], sh), __funnelshift_r(v[1], v[2], sh), __funnelshift_r(v[2], v[3], sh), __funnelshift_r(v[3], v[4], sh));
}

// exponent that puts a group's largest magnitude into [2^21, 2^22); both 2^e and 2^-e are normal numbers. Magnitudes
// below 2^-105 keep an absolute step of 2^-126.
__device__ __forceinline__ int rows_group_exponent(uint32_t amax_bits) { return min(126, 148 - (int)(amax_bits >> 23)); }

__device__ __forceinline__ unsigned long long rows_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

template <int NB, bool DC, int TW, bool MIS>
__global__ void __launch_bounds__(kRowsWarps * 32, 1) q4_rows_kernel(const __grid_constant__ RowsParams p) {
    constexpr uint32_t MP = (DC ? 2 : 8) * NB;
    constexpr uint32_t T = kRowsWarps * 32;
    constexpr uint32_t S = rows_stages(TW), PS = rows_param_stages(TW);
    constexpr uint32_t kParamTile = rows_param_bytes(MIS);
    constexpr uint32_t kStage = kRowsStageBytes * TW, kParamStage = kParamTile * TW;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint32_t part = blockIdx.x % p.parts, gi = blockIdx.x / p.parts;
    // parts begin at multiples of four chunks: parameters are copied in 16-byte pieces of eight groups
    const uint32_t c_lo = q4_rows_part_begin(p.cpt, p.parts, part), c_hi = q4_rows_part_begin(p.cpt, p.parts, part + 1u), nch = c_hi - c_lo;
    uint8_t *xdig = smem + kRowsWarps * rows_ring_bytes(TW, MIS);
    float *xscale = reinterpret_cast<float *>(xdig + (size_t)p.part_chunks * rows_chunk_bytes(MP));
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem) + warp * rows_ring_bytes(TW, MIS);
    const uint32_t pring = ring + S * kStage;

    // ---- an item's weights (TW tiles): lane l copies 16 bytes of row l >> 2 (and of the row eight further down) per
    // chunk and tile. The four 16-byte quarters of a row are stored with quarter q at q ^ (2 * bit 1 of the row), so
    // that the 8-byte reads below (lane (g, t): bytes 8 t.. of a group) touch every bank once per half-warp.
    const uint32_t cr = lane >> 2, cq = lane & 3u;
    const uint32_t copy_off = 16u * (cr * 4u + (cq ^ (2u * ((cr >> 1) & 1u))));
    const uint64_t row_bytes = (uint64_t)p.k >> 1;
    // item i of a part = tiles TW * i .. TW * i + TW - 1 (a tile past the last one repeats the last: computed, never stored)
    const uint32_t items = (p.tiles + TW - 1) / TW, quads = (nch + 3u) / 4u;
    const uint32_t worker = gi * kRowsWarps + warp;
    const uint32_t u0 = min(worker * p.run, items * quads), u1 = min(u0 + p.run, items * quads);  // this warp's quads of the part
    auto find_tile = [&](uint32_t it, int w, bool &live, const RowsJob *&job, uint32_t &row0) {
        const uint32_t want = it * TW + w;
        live = want < p.tiles;
        const uint32_t tile = live ? want : p.tiles - 1u;
        uint32_t ji = 0;
        while (ji + 1 < p.n_jobs && tile >= p.jobs[ji + 1].tile_begin) ++ji;
        job = &p.jobs[ji];
        row0 = (tile - job->tile_begin) * 16u;
    };
    // A run of n chunks of one item takes this many ring stages: the byte-addressed form needs one more, for the window
    // that completes its last chunk, and keeps its quads apart (two quads never share the parameter stages' period).
    auto stages_of = [](uint32_t n) { return !MIS ? n : (n & 3u) ? (n + 3u) & ~3u : n + 1u; };

    // what is requested next: cursors of the run that is being requested, at chunk pc
    const uint8_t *wa[TW], *wb[TW], *pw[TW];
    uint32_t wmis[TW];  // bytes by which the tile's weight rows miss a 16-byte boundary
    uint32_t pown[TW];  // the same for the parameter row that this lane copies
#pragma unroll
    for (int w = 0; w < TW; ++w) {
        wa[w] = wb[w] = pw[w] = nullptr;
        wmis[w] = pown[w] = 0;
    }
    uint32_t pu = u0, pc = 0, pc_end = 0, pc_stop = 0;  // next quad to open; chunks [pc, pc_end) are left, stages up to pc_stop
    uint32_t req_stage = 0, req_param = 0;
    auto open_run = [&]() {
        const uint32_t it = pu / quads, q = pu - it * quads, q_end = min(quads, q + (u1 - pu));
        pc = c_lo + 4u * q;
        pc_end = min(c_lo + 4u * q_end, c_hi);
        pc_stop = pc + stages_of(pc_end - pc);
        pu += q_end - q;
#pragma unroll
        for (int w = 0; w < TW; ++w) {
            bool live;
            const RowsJob *job;
            uint32_t row0;
            find_tile(it, w, live, job, row0);
            const uint32_t last = job->n - 1u;
            const uint32_t ra = min(row0 + cr, last), rb = min(row0 + 8u + cr, last);  // rows past n: read a valid row
            const uint32_t rp = min(row0 + (lane & 15u), last);
            if (MIS) wmis[w] = (uint32_t)((uintptr_t)job->w & 15u);
            wa[w] = job->w + (uint64_t)ra * row_bytes + cq * 16u + (size_t)pc * 64u - wmis[w];
            wb[w] = job->w + (uint64_t)rb * row_bytes + cq * 16u + (size_t)pc * 64u - wmis[w];
            pw[w] = ((lane >> 4) ? job->b : job->s) + ((size_t)rp * p.groups) * 2u + (size_t)pc * 4u;
            if (MIS) {
                pown[w] = (uint32_t)((uintptr_t)pw[w] & 15u);
                pw[w] -= pown[w];
            }
        }
    };
    auto request_stage = [&]() {  // the next ring stage of this warp
        if (pc == pc_stop && pu < u1) open_run();
        if (pc != pc_stop) {
            const uint32_t stage = ring + req_stage * kStage;
            const bool in = !MIS || pc < pc_end;
            if (!MIS || (in && 2u * pc + 1u < p.groups)) {
#pragma unroll
                for (int w = 0; w < TW; ++w) {
                    cp_async_16(stage + w * kRowsStageBytes + copy_off, wa[w]);
                    cp_async_16(stage + w * kRowsStageBytes + 512u + copy_off, wb[w]);
                }
            } else {
                // at the end of a row or run only windows that hold bytes of the row (q4_decomp.h); the stage after the run's
                // last chunk holds the window that completes that chunk
#pragma unroll
                for (int w = 0; w < TW; ++w) {
                    const bool pred = in ? q4_window_wanted(cq, wmis[w], false) : pc == pc_end && cq == 0 && q4_fifth_window_wanted(wmis[w], 2u * pc - 1u < p.groups);
                    cp_async_16_pred(stage + w * kRowsStageBytes + copy_off, wa[w], pred);
                    cp_async_16_pred(stage + w * kRowsStageBytes + 512u + copy_off, wb[w], pred);
                }
            }
#pragma unroll
            for (int w = 0; w < TW; ++w) {
                wa[w] += 64;
                wb[w] += 64;
            }
            // every quad: lane l copies the scales (l < 16) or biases of row l & 15 for the next eight groups
            if ((pc & 3u) == 0 && in) {
#pragma unroll
                for (int w = 0; w < TW; ++w) {
                    const uint32_t dst = pring + req_param * kParamStage + w * kParamTile + lane * 16u;
                    cp_async_16(dst, pw[w]);
                    if (MIS) cp_async_16_pred(dst + 512u, pw[w] + 16, pown[w] + 2u * min(8u, p.groups - 2u * pc) > 16u);
                    pw[w] += 16;
                }
                req_param = req_param + 1u == PS ? 0u : req_param + 1u;
            }
            ++pc;
        }
        cp_async_commit();
        req_stage = (req_stage + 1u) & (S - 1u);
    };
    unsigned long long *tr = (p.trace && lane == 0) ? p.trace + ((size_t)blockIdx.x * kRowsWarps + warp) * 4 : nullptr;
    if (tr) tr[0] = rows_ns();
    bool first_run = true;

    // weights do not depend on the kernel in front of this one, activation, output and scratch do
#pragma unroll 1
    for (uint32_t i = 0; i < S - 1u; ++i) request_stage();
    grid_dependency_wait();
    grid_dependents_launch();

    // ---- the part's digits for every row ----
    // Every thread holds its blocks of 8 inputs (at most kRowsPerThread) in registers, so that all of its loads are in
    // flight at once: one round trip to L2 instead of one per block.
    const uint32_t span8 = nch * 16u;  // blocks of 8 inputs per row in this part
    uint4 raw[kRowsPerThread][2];
    const uint32_t total8 = p.m * span8, padded8 = MP * span8;  // rows past m are zero-filled
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) {
        const uint32_t idx = threadIdx.x + i * T;
        raw[i][0] = raw[i][1] = make_uint4(0, 0, 0, 0);
        if (idx < total8) {
            const uint32_t mrow = idx / span8, b8 = idx - mrow * span8;
            const size_t at = (size_t)mrow * p.k + (size_t)c_lo * 128u + (size_t)b8 * 8u;
            if (!MIS || c_lo * 128u + b8 * 8u < p.k) {  // (the last group of an odd number of groups: zeros)
                if (p.x_is_f32) {
                    const uint4 *src = reinterpret_cast<const uint4 *>(static_cast<const float *>(p.x) + at);
                    raw[i][0] = __ldcg(src);
                    raw[i][1] = __ldcg(src + 1);
                } else {
                    raw[i][0] = __ldcg(reinterpret_cast<const uint4 *>(static_cast<const uint16_t *>(p.x) + at));
                }
            }
        }
    }
    auto unpack8 = [&](const uint4 (&r)[2], float (&v)[8]) {
        if (p.x_is_f32) {
            v[0] = __uint_as_float(r[0].x); v[1] = __uint_as_float(r[0].y); v[2] = __uint_as_float(r[0].z); v[3] = __uint_as_float(r[0].w);
            v[4] = __uint_as_float(r[1].x); v[5] = __uint_as_float(r[1].y); v[6] = __uint_as_float(r[1].z); v[7] = __uint_as_float(r[1].w);
        } else {
            const uint32_t w[4] = {r[0].x, r[0].y, r[0].z, r[0].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[2 * j] = bf16_bits_to_float(w[j] & 0xffffu);
                v[2 * j + 1] = bf16_bits_to_float(w[j] >> 16);
            }
        }
    };
    auto digits_at = [&](uint32_t chunk, uint32_t grp, uint32_t mrow) {
        return xdig + (size_t)chunk * rows_chunk_bytes(MP) + (size_t)grp * 3u * MP * 64u + (size_t)mrow * (DC ? 192u : 64u);
    };
    auto store_scale = [&](uint32_t chunk, uint32_t grp, uint32_t mrow, float sum, float inv) {
        if (DC) {
            *reinterpret_cast<float4 *>(xscale + ((size_t)(chunk * 2u + grp) * MP + mrow) * 4u) = make_float4(sum, inv, 0.f, inv * 65536.f);
        } else {
            float *dst = xscale + ((size_t)(chunk * 2u + grp) * (MP / 2u) + (mrow >> 1)) * 4u + (mrow & 1u);
            dst[0] = sum;
            dst[2] = inv;
        }
    };
    // the eight threads of a group agree on its scale (span8 is a multiple of 16: a group never leaves its half-warp)
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) {
        if ((uint32_t)i * T >= padded8) continue;  // (uniform)
        const uint32_t idx = threadIdx.x + i * T;
        const bool live = idx < padded8;
        const uint32_t mrow = live ? idx / span8 : 0u, b8 = live ? idx - mrow * span8 : 0u;
        float v[8];
        unpack8(raw[i], v);
        uint32_t mx = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) mx = max(mx, __float_as_uint(v[j]) & 0x7fffffffu);
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        const int e = rows_group_exponent(mx);
        const float scale = __uint_as_float((uint32_t)(e + 127) << 23), inv = __uint_as_float((uint32_t)(127 - e) << 23) * kRowsSumScale;
        int sum = 0;
        uint32_t z[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int xi = __float2int_rn(v[j] * scale);
            sum += xi;
            z[j] = ((uint32_t)xi + 0x00808080u) ^ 0x00808080u;  // bytes 0..2: the signed digits
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        if (live) {
            const uint32_t chunk = b8 >> 4, grp = (b8 >> 3) & 1u, b = b8 & 7u;  // block b of the group: inputs 8 b .. 8 b + 7
            uint8_t *dst = digits_at(chunk, grp, mrow) + 16u * (b >> 1) + 8u * (b & 1u);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const uint32_t sel = (uint32_t)d | ((4u + (uint32_t)d) << 4);
                uint2 w;
                w.x = __byte_perm(__byte_perm(z[0], z[2], sel), __byte_perm(z[4], z[6], sel), 0x5410u);  // even inputs
                w.y = __byte_perm(__byte_perm(z[1], z[3], sel), __byte_perm(z[5], z[7], sel), 0x5410u);  // odd inputs
                *reinterpret_cast<uint2 *>(dst + (size_t)d * (DC ? 64u : MP * 64u)) = w;
            }
            // infinity or NaN: poison the row
            if (b == 0) store_scale(chunk, grp, mrow, mx >= 0x7f800000u ? __uint_as_float(0x7fc00000u) : (float)sum * inv, inv);
        }
    }
    __syncthreads();

    if (tr) tr[1] = rows_ns();

    // ---- tiles ----
    // B operands: digit d of row g of a block of eight (16 bytes from lane t); DC: digit g & 3 of row g >> 2 of a pair, zeros
    // in columns 3 and 7
    const bool has_x = !DC || (g & 3u) < 3u;
    const uint32_t xdig_addr = (uint32_t)__cvta_generic_to_shared(xdig) + (DC ? (g >> 2) * 192u + (g & 3u) * 64u : g * 64u) + t * 16u;
    const uint32_t xscale_addr = (uint32_t)__cvta_generic_to_shared(xscale) + (DC ? (t >> 1) * 16u + (t & 1u) * 8u : t * 16u);
    constexpr int XD = DC ? 1 : 3;  // B operands of a group and block of rows
    uint4 xf[2][NB][XD];
#pragma unroll
    for (int i = 0; i < 2 * NB * XD; ++i) (&xf[0][0][0])[i] = make_uint4(0, 0, 0, 0);
    // this lane's 8 bytes of group G of row g in a stage: word j = 4 G + t of the row's eight 8-byte words, in quarter
    // j >> 1, swizzled as above; words 8 and 9 (MIS) are the first two of the next stage
    const uint32_t rd_swz = 2u * ((g >> 1) & 1u);
    auto word_off = [&](uint32_t j) { return 16u * (g * 4u + (((j >> 1) & 3u) ^ rd_swz)) + 8u * (j & 1u); };
    const uint32_t rd0 = word_off(t), rd1 = word_off(4u + t);
    constexpr int AV = DC ? 2 : 4;  // sums a lane holds per tile and block of rows
    uint32_t stage_i = 0, param_i = 0;
    for (uint32_t u = u0; u < u1;) {
        const uint32_t item = u / quads, q0 = u - item * quads, q1 = min(quads, q0 + (u1 - u));
        const uint32_t c_begin = c_lo + 4u * q0, c_stop = min(c_lo + 4u * q1, c_hi);
        u += q1 - q0;
        const RowsJob *job[TW];
        uint32_t row0[TW], wm[TW], pmis[TW];  // pmis: of the parameter row this lane copied (and realigns)
        uint32_t rlo[TW][2], rhi[TW][2];      // where this lane's two 8-byte words of each group are in a stage ...
        bool nlo[TW], nhi[TW];                // ... and whether those of the second group are in the next stage
        bool tile_live[TW];
#pragma unroll
        for (int w = 0; w < TW; ++w) {
            find_tile(item, w, tile_live[w], job[w], row0[w]);
            wm[w] = pmis[w] = 0;
            if (MIS) {
                wm[w] = (uint32_t)((uintptr_t)job[w]->w & 15u);
                const uint32_t j = t + (wm[w] >> 3);
                rlo[w][0] = word_off(j);
                rhi[w][0] = word_off(j + 1u);
                rlo[w][1] = word_off(j + 4u);
                rhi[w][1] = word_off(j + 5u);
                nlo[w] = j + 4u >= 8u;
                nhi[w] = j + 5u >= 8u;
                const uint32_t rp = min(row0[w] + (lane & 15u), job[w]->n - 1u);
                pmis[w] = ((uint32_t)(uintptr_t)((lane >> 4) ? job[w]->b : job[w]->s) + rp * p.groups * 2u) & 15u;  // (runs begin at multiples of 16 bytes)
            }
        }
        float acc[TW][NB][AV];
#pragma unroll
        for (int i = 0; i < TW * NB * AV; ++i) (&acc[0][0][0])[i] = 0.f;
        for (uint32_t c = c_begin; c < c_stop; ++c) {
            request_stage();
            cp_async_wait<S - (MIS ? 2 : 1)>();  // (MIS: the next chunk's first window too)
            __syncwarp();
            const uint32_t stage = ring + stage_i * kStage, next_stage = ring + ((stage_i + 1u) & (S - 1u)) * kStage;
            const uint32_t pst = pring + param_i * kParamStage;
            const uint32_t xc = xdig_addr + (c - c_lo) * rows_chunk_bytes(MP);
            const uint32_t xs = xscale_addr + (c - c_lo) * (2u * MP * rows_scale_bytes(DC));
            if (MIS && (c & 3u) == 0) {
                // a new quad: lane l shifts the parameter row it copied to the boundary, groups past the last one become zero
                const uint32_t left = p.groups - 2u * c;
#pragma unroll
                for (int w = 0; w < TW; ++w) {
                    const uint32_t at = pst + w * kParamTile + lane * 16u;
                    uint4 v = realign_16_any(lds_v4(at), lds_v4(at + 512u), pmis[w]);
                    if (left < 8u) {
                        uint32_t *r = &v.x;
#pragma unroll
                        for (uint32_t i = 0; i < 4u; ++i) r[i] = 2u * i >= left ? 0u : 2u * i + 1u >= left ? r[i] & 0xffffu : r[i];
                    }
                    sts_v4(at, v);
                }
                __syncwarp();
            }
            // scales and biases of the chunk's two groups, rows g and g + 8
            uint32_t prm[TW][4];
#pragma unroll
            for (int w = 0; w < TW; ++w)
#pragma unroll
                for (int i = 0; i < 4; ++i) prm[w][i] = lds_u32(pst + w * kParamTile + (i >> 1) * 256u + (g + 8u * (i & 1)) * 16u + (c & 3u) * 4u);
#pragma unroll
            for (int grp = 0; grp < 2; ++grp) {
                // the activation's digits of this group: read once, used by every tile of the item
                uint4 xv[NB];  // {sum, sum, 2^-e, 2^-e} of rows 2 t, 2 t + 1 of this block of 8; DC: {sum, factor} of this lane
#pragma unroll
                for (int nb = 0; nb < NB; ++nb) {
                    if constexpr (DC) {
                        lds_v4_keep(xf[grp][nb][0], xc + (uint32_t)(grp * 3 * MP * 64 + nb * 384), has_x);
                        const uint2 f = lds_v2(xs + (uint32_t)((grp * MP + nb * 2) * 16));
                        xv[nb] = make_uint4(f.x, f.y, 0, 0);
                    } else {
#pragma unroll
                        for (int d = 0; d < XD; ++d) xf[grp][nb][d] = lds_v4(xc + (uint32_t)((grp * 3 + d) * MP + nb * 8) * 64u);
                        xv[nb] = lds_v4(xs + (uint32_t)(grp * MP + nb * 8) * 8u);
                    }
                }
#pragma unroll
                for (int w = 0; w < TW; ++w) {
                    const uint32_t wst = stage + w * kRowsStageBytes;
                    uint2 wA, wB;
                    if (!MIS || wm[w] == 0) {
                        wA = lds_v2(wst + (grp ? rd1 : rd0));
                        wB = lds_v2(wst + 512u + (grp ? rd1 : rd0));
                    } else {
                        const uint32_t nst = next_stage + w * kRowsStageBytes;
                        const uint32_t a0 = (grp && nlo[w] ? nst : wst) + rlo[w][grp], a1 = (grp && nhi[w] ? nst : wst) + rhi[w][grp];
                        const uint2 loA = lds_v2(a0), hiA = lds_v2(a1), loB = lds_v2(a0 + 512u), hiB = lds_v2(a1 + 512u);
                        const uint32_t sh = (wm[w] & 3u) * 8u;
                        const bool by4 = (wm[w] & 4u) != 0;
                        wA.x = __funnelshift_r(by4 ? loA.y : loA.x, by4 ? hiA.x : loA.y, sh);
                        wA.y = __funnelshift_r(by4 ? hiA.x : loA.y, by4 ? hiA.y : hiA.x, sh);
                        wB.x = __funnelshift_r(by4 ? loB.y : loB.x, by4 ? hiB.x : loB.y, sh);
                        wB.y = __funnelshift_r(by4 ? hiB.x : loB.y, by4 ? hiB.y : hiB.x, sh);
                    }
                    const uint32_t m4 = 0x0f0f0f0fu;
                    const uint32_t a_lo0 = wA.x & m4, a_hi0 = (wA.x >> 4) & m4, a_lo1 = wA.y & m4, a_hi1 = (wA.y >> 4) & m4;
                    const uint32_t b_lo0 = wB.x & m4, b_hi0 = (wB.x >> 4) & m4, b_lo1 = wB.y & m4, b_hi1 = (wB.y >> 4) & m4;
                    const float sa = bf16_bits_to_float(grp ? (prm[w][0] >> 16) : (prm[w][0] & 0xffffu));
                    const float sb = bf16_bits_to_float(grp ? (prm[w][1] >> 16) : (prm[w][1] & 0xffffu));
                    const float ba = bf16_bits_to_float(grp ? (prm[w][2] >> 16) : (prm[w][2] & 0xffffu));
                    const float bb = bf16_bits_to_float(grp ? (prm[w][3] >> 16) : (prm[w][3] & 0xffffu));
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) {
                        int q[XD][4];
#pragma unroll
                        for (int d = 0; d < XD; ++d) {
                            const uint4 &x = xf[grp][nb][d];
                            q[d][0] = q[d][1] = q[d][2] = q[d][3] = 0;
                            mma_u8s8_16832(q[d], a_lo0, b_lo0, a_hi0, b_hi0, x.x, x.y);
                            mma_u8s8_16832(q[d], a_lo1, b_lo1, a_hi1, b_hi1, x.z, x.w);
                        }
                        if constexpr (DC) {
                            // even lanes hold digits 0 and 1 of a row, odd ones digit 2 (and a zero); the two sums meet at
                            // the end of the tile
                            const float sum = __uint_as_float(xv[nb].x), f = __uint_as_float(xv[nb].y);
                            acc[w][nb][0] = fmaf(__int2float_rn(q[0][0] + (q[0][1] << 8)) * f, sa, fmaf(sum, ba, acc[w][nb][0]));
                            acc[w][nb][1] = fmaf(__int2float_rn(q[0][2] + (q[0][3] << 8)) * f, sb, fmaf(sum, bb, acc[w][nb][1]));
                        } else {
                            // the group's integer dot product q0 + 256 q1 + 65536 q2 (exact; |q0 + 256 q1| < 2^25 is rounded to fp32 once)
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const float dot = fmaf(__int2float_rn(q[XD - 1][i]), 65536.f, __int2float_rn(q[0][i] + (q[XD / 2][i] << 8))) *
                                                  __uint_as_float((i & 1) ? xv[nb].w : xv[nb].z);
                                acc[w][nb][i] = fmaf(dot, i < 2 ? sa : sb, acc[w][nb][i]);
                            }
                            const float x0 = __uint_as_float(xv[nb].x), x1 = __uint_as_float(xv[nb].y);
                            acc[w][nb][0] = fmaf(x0, ba, acc[w][nb][0]);
                            acc[w][nb][1] = fmaf(x1, ba, acc[w][nb][1]);
                            acc[w][nb][AV - 2] = fmaf(x0, bb, acc[w][nb][AV - 2]);
                            acc[w][nb][AV - 1] = fmaf(x1, bb, acc[w][nb][AV - 1]);
                        }
                    }
                }
            }
            __syncwarp();  // every lane is done with the stage before the next iteration refills it
            stage_i = (stage_i + 1u) & (S - 1u);
            if ((c & 3u) == 3u || c + 1u == c_stop) param_i = param_i + 1u == PS ? 0u : param_i + 1u;
        }
        if (MIS) {
            for (uint32_t n = c_stop - c_begin, pad = stages_of(n) - n; pad; --pad) {
                request_stage();
                stage_i = (stage_i + 1u) & (S - 1u);
            }
        }
        if (tr && first_run) tr[2] = rows_ns();
        first_run = false;

        // ---- the tile's contributions meet ----
        if constexpr (DC) {
#pragma unroll
            for (int i = 0; i < TW * NB * AV; ++i) (&acc[0][0][0])[i] += __shfl_xor_sync(0xffffffffu, (&acc[0][0][0])[i], 1);
        }
#pragma unroll
        for (int i = 0; i < TW * NB * AV; ++i) (&acc[0][0][0])[i] *= 1.0f / kRowsSumScale;
        // value i of a block of rows: activation row and weight row of the tile (DC: only even lanes store)
        auto act_row = [&](int nb, int i) { return DC ? nb * 2u + (t >> 1) : nb * 8u + 2u * t + (uint32_t)(i & 1); };
        auto weight_row = [&](int i) { return g + 8u * (uint32_t)(DC ? i : i >> 1); };
        const bool mine = !DC || (t & 1u) == 0;
        const uint32_t rows_total = items * TW * 16u;
        const bool whole = p.parts == 1u && q0 == 0 && q1 == quads;
        uint32_t shares = 0;  // lane l: contributions of part l to this item
        bool last = true;
        if (!whole) {
            const size_t slot = (size_t)part * p.part_slots + (worker - item * quads / p.run);
#pragma unroll
            for (int w = 0; w < TW; ++w)
#pragma unroll
                for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                    for (int i = 0; i < AV; ++i)
                        if (mine) p.partials[(slot * MP + act_row(nb, i)) * rows_total + (size_t)(item * TW + w) * 16u + weight_row(i)] = acc[w][nb][i];
            fence_gpu();
            __syncwarp();
            unsigned int before = 0;
            if (lane == 0) before = atomicAdd(p.counters + item, 1u);
            if (lane < p.parts) {
                const uint32_t ql = (q4_rows_part_begin(p.cpt, p.parts, lane + 1u) - q4_rows_part_begin(p.cpt, p.parts, lane) + 3u) / 4u;
                shares = q4_rows_shares(item, ql, p.run);
            }
            before = __shfl_sync(0xffffffffu, before, 0);
            last = before + 1u == __reduce_add_sync(0xffffffffu, shares);
            if (last) {
                fence_gpu();
                if (lane == 0) p.counters[item] = 0;  // ready for the next launch
            }
        }
        if (last) {
            if (!whole) {
                // all contributions in K order, whoever came last; four at a time, so that a round trip to L2 fetches four
#pragma unroll
                for (int i = 0; i < TW * NB * AV; ++i) (&acc[0][0][0])[i] = 0.f;
                uint32_t pp = 0, jj = 0, n = __shfl_sync(0xffffffffu, shares, 0);
                while (pp < p.parts) {
                    constexpr int B = 4;
                    float got[B][TW * NB * AV];
#pragma unroll
                    for (int b = 0; b < B; ++b) {
                        const bool have = pp < p.parts;  // (uniform)
                        const float *src = p.partials + ((size_t)pp * p.part_slots + jj) * MP * rows_total + (size_t)item * TW * 16u;
#pragma unroll
                        for (int v = 0; v < TW * NB * AV; ++v) {
                            const int i = v % AV, nb = v / AV % NB, w = v / (AV * NB);
                            got[b][v] = have ? __ldcg(src + (size_t)act_row(nb, i) * rows_total + w * 16u + weight_row(i)) : 0.f;
                        }
                        if (have && ++jj == n) {
                            jj = 0;
                            n = __shfl_sync(0xffffffffu, shares, ++pp & 31u);
                        }
                    }
#pragma unroll
                    for (int b = 0; b < B; ++b)
#pragma unroll
                        for (int v = 0; v < TW * NB * AV; ++v) (&acc[0][0][0])[v] += got[b][v];
                }
            }
#pragma unroll
            for (int w = 0; w < TW; ++w)
#pragma unroll
                for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                    for (int i = 0; i < AV; ++i) {
                        const uint32_t mcol = act_row(nb, i), r = weight_row(i);
                        if (!mine || !tile_live[w] || mcol >= p.m || row0[w] + r >= job[w]->n) continue;
                        float *dst = job[w]->out + (size_t)mcol * job[w]->out_stride + row0[w] + r;
                        *dst = p.accumulate ? *dst + acc[w][nb][i] : acc[w][nb][i];
                    }
        }
    }
    cp_async_wait<0>();
    if (tr) tr[3] = rows_ns();
}

}  // namespace q4

// Largest part (in chunks) a block can hold for `mp` padded activation rows and `tw` tiles per warp, 0 if not even
// four chunks fit.
static uint32_t rows_part_capacity(uint32_t mp, uint32_t tw, bool mis, bool dc) {
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    uint32_t chunks = 0;
    while (q4::rows_smem_bytes(mp, chunks + 1, tw, mis, dc) <= (size_t)optin && (chunks + 1) * mp <= 256u) ++chunks;
    return chunks >= 4 ? chunks : 0;
}

// How the K range of a launch is cut: the number of parts (0: the shape is not supported), the longest part, and how
// many tiles a warp walks at a time (two share the activation's fragments; up to 8 rows only). `mis`: the byte-addressed
// instance, which any K % 64 == 0 and any byte offset may use; the other one wants K % 512 == 0 and 16-byte alignment.
extern "C" uint32_t q4k_rows_plan(uint32_t m, uint32_t k, uint32_t tiles, uint32_t sm_count, int mis, uint32_t *part_chunks, uint32_t *tiles_per_warp) {
    if (m < 1 || m > 16 || k == 0 || k % (mis ? 64u : 512u) != 0 || tiles == 0) return 0;
    const uint32_t mp = q4::rows_padded(m);
    const bool dc = q4::rows_dc(m);
    uint32_t best = 0;
    double best_cost = 0.0;
    for (uint32_t tw = 1; tw <= (mp == 8 ? 2u : 1u); ++tw) {
        const uint32_t cap = rows_part_capacity(mp, tw, mis != 0, dc);
        if (cap == 0) continue;
        uint32_t chunks = 0;
        double cost = 0.0;
        const uint32_t parts = q4_rows_plan((k / 64u + 1u) / 2u, tiles, sm_count, cap, tw, mp, &chunks, &cost);
        if (parts && (best == 0 || cost < best_cost * 0.98)) {
            best = parts;
            best_cost = cost;
            *part_chunks = chunks;
            *tiles_per_warp = tw;
        }
    }
    return best;
}

extern "C" uint32_t q4k_rows_padded(uint32_t m) { return q4::rows_padded(m); }

template <int NB, bool DC, int TW, bool MIS>
static cudaError_t rows_launch(const q4::RowsParams &p, uint32_t grid, size_t smem, cudaStream_t stream) {
    const cudaError_t e = cudaFuncSetAttribute(q4::q4_rows_kernel<NB, DC, TW, MIS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(q4::kRowsWarps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, q4::q4_rows_kernel<NB, DC, TW, MIS>, p);
}

extern "C" cudaError_t q4k_rows(const q4::RowsParams *params, uint32_t sm_count, cudaStream_t stream) {
    const q4::RowsParams &p = *params;
    const uint32_t mp = q4::rows_padded(p.m);
    const bool mis = p.byte_addressed != 0, dc = q4::rows_dc(p.m);
    if (p.tiles_per_warp != 1u && !(p.tiles_per_warp == 2u && mp == 8u)) return cudaErrorInvalidValue;
    const size_t smem = q4::rows_smem_bytes(mp, p.part_chunks, p.tiles_per_warp, mis, dc);
    const uint32_t grid = (sm_count / p.parts) * p.parts;
    if (grid == 0 || p.run == 0) return cudaErrorInvalidValue;
    if (mp == 2) return mis ? rows_launch<1, true, 1, true>(p, grid, smem, stream) : rows_launch<1, true, 1, false>(p, grid, smem, stream);
    if (mp == 4) return mis ? rows_launch<2, true, 1, true>(p, grid, smem, stream) : rows_launch<2, true, 1, false>(p, grid, smem, stream);
    if (mp == 16) return mis ? rows_launch<2, false, 1, true>(p, grid, smem, stream) : rows_launch<2, false, 1, false>(p, grid, smem, stream);
    if (p.tiles_per_warp == 2u) return mis ? rows_launch<1, false, 2, true>(p, grid, smem, stream) : rows_launch<1, false, 2, false>(p, grid, smem, stream);
    return mis ? rows_launch<1, false, 1, true>(p, grid, smem, stream) : rows_launch<1, false, 1, false>(p, grid, smem, stream);
}
