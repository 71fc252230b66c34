// Single rows and short batches (up to 16 activation rows) of MLX affine-Q4 projections on the integer tensor-core path: the shape of the
// reference's matvec and batched kernels (qwen38_q4_affine_matvec_batch2/4/8, shaders/qwen38.metal:213-246 applied per row),
// HBM-bound on B200 because every packed weight is read once for all rows.
//
// Arithmetic. Every affine group (64 inputs) of an activation row is held as fixed point after an exact power-of-two
// scaling by the group's own largest magnitude, x' = d0 + 256 d1 + 65536 d2 (+ 2^24 d3) with D signed 8-bit digits. A packed
// weight word becomes two byte registers (even and odd nibbles): a nibble in the upper half of a byte with its top bit
// flipped is the signed byte 16 (q - 8), so the A operand of mma.sync.m16n8k32.s32.s8.s8 takes two logic instructions
// and a shift for eight weights, and the weights are centred: y = scale * sum x (q - 8) + (bias + 8 scale) * sum x, whose two
// terms do not cancel one another as those of the uncentred form do. The B operand holds one digit of eight activation
// rows; an affine group is two MMAs per digit, and its integer sums are exact, put together with one rounding to fp32, and
// scaled in fp32. The approximations are the fixed-point step of the activation and the fp32 rounding of the per-group terms.
// Relative error (2-norm) of a result against 64 bits, normal inputs, K = 5120: 1.0e-7 with four digits or bf16 inputs, 3.0e-7 with three
// digits of fp32 inputs (uncentred: 1.1e-7 to 2.2e-7, and 1.3e-7 through fp16 terms; 3.3e-7 with three digits of fp32 inputs).
// D = 4 leaves the step at 2^-30 of the largest of 64 neighbours (bf16 within 2^22 of it is exact, fp32 within 2^6): single rows,
// byte-addressed launches, fp32 inputs of up to four rows. D = 3, at 2^-22 (bf16 exact within 2^14), the others: 2 to 16 rows
// of aligned tensors, where a fourth digit would cost four rows 15 % (34816 x 5120, 26.8 -> 30.8 us: a quarter more digits to
// read). What a step costs shows when an input far above its 63 neighbours meets a weight of zero: results are off by 1e-4 (D = 3)
// or 5e-7 (D = 4) at 10^4 times its neighbours, 1e-3 or 5e-6 at 10^5. A group that holds an infinity or a NaN makes every result of its
// row NaN. Byte-addressed bf16 launches had three digits (and 16 rows); the fourth costs 8 rows x 34816 x 5120 47.7 -> 55.8 us, 8192 x 5120
// 16.7 -> 17.7, 12 rows in two launches 79.6 -> 99.9 and 35.6 -> 34.2.
//
// Up to four rows (DC) the digits of two rows share one B operand -- columns 0..3 hold the digits of the first row,
// 4..7 those of the second (three digits leave the last of the four zero) -- instead of one digit of eight rows each: 2 MMAs
// per group and pair of rows where the form above takes 6 or 8 for up to eight.
//
// Work. The K range is cut into `parts` runs of 128-input chunks. A block holds the digits of ONE part for all rows
// in shared memory (converted by the block itself from the caller's bf16 or fp32 rows). A part's work is the list of its
// 16-row tiles times its quads of four chunks; every warp of the part's blocks takes the same
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
// Launches are programmatic dependents of whatever runs in front of them: a block requests its first weights and only then waits
// for the kernel before it, unless that kernel may write them (weights_ahead: the caller holds the address of a shard).
// Measured (B200, weights from HBM; in a row of calls, and in brackets with a small kernel of the caller's between them, which cannot let this one
// start early): 1 row x 5120 x 5120 7.8 us (12.6), 1 x 34816 x 5120 19.5 (24.8), at a byte offset 26.8 (33.4), 4 rows 26.8 (32.9), 8 rows
// 32.6 = 3.1 TB/s (38.1), 16 rows 63.2 (68.4), 1 fp32 row x 5120 x 17408 at a byte offset 18.1 (24.1), 8 fp32 rows x 8192 x 5120 at a
// byte offset 17.8 (23.1), 4 rows x 248320 x 5120 141 = 5.1 TB/s (138).
// What bounds it: 8 rows x 34816 x 5120 issue 205 warp instructions per 1 KB chunk (fixed part included), at 54 % of the issue slots
// and 40 % of the ALU of sixteen warps an SM, none of which is waiting for memory much: instruction issue and its
// dependencies. In a call that starts by itself the digits are ready after 7 to 9 us, although they take 2 without weights in flight:
// the warps stand at their own requests until the memory has taken them. Requesting the second half of the ring after the
// conversion gives 0.5 to 1.8 us there and costs 0.4 to 1.3 us in a row of calls, requesting nothing before the wait 2 to 3. Two tiles at a
// time (units of two chunks of two tiles) take 41.9 us for the 8 rows above. Contributions of parts meet in 2 to 3 us.
#include "q4_decomp.h"
#include "q4_device.cuh"
#include "q4_kernels.h"

namespace q4 {

constexpr int kRowsWarps = 16;
constexpr int kRowsStageBytes = 1024;  // one chunk of one tile: 16 weight rows x 64 packed bytes
constexpr int kRowsPerThread = 8;      // blocks of 8 inputs a thread converts at most (bounds a part: rows x chunks <= 256)
constexpr uint32_t kRowsPairColumns = 4;  // up to this many rows share B operands in pairs

// A warp's ring has two halves of a quad each: four 1 KB chunks of one tile and the scales and biases of their eight groups
// (a 16-byte window per row and array). Byte-addressed, a fifth stage follows the four: the first quarter of its rows
// holds the window that completes the fourth chunk, where a following chunk would have it, and the second and third
// quarters the second windows of the parameters. One half is consumed while the other one is on its way; the loop
// over a quad is unrolled, so that every address in it is a constant from the half's base.
__host__ __device__ constexpr uint32_t rows_weight_bytes(bool mis) { return (mis ? 5u : 4u) * kRowsStageBytes; }
__host__ __device__ constexpr uint32_t rows_half_bytes(bool mis) { return rows_weight_bytes(mis) + 512u; }

__host__ __device__ constexpr bool rows_dc(uint32_t m) { return m <= kRowsPairColumns; }
__host__ __device__ constexpr uint32_t rows_padded(uint32_t m) { return rows_dc(m) ? (m + 1u) & ~1u : (m + 7u) & ~7u; }

// Shared memory of one chunk's digits: [group 2][digit D][activation row MP][64 bytes], DC: [group 2][row MP][digit D][64 bytes]. The 64 bytes of a (group, digit,
// row) hold the 64 inputs of the group in the order lane t of a quad wants them as B registers of the group's two MMAs:
// byte 16 t + 8 j + 4 odd + i  <->  input 16 t + 8 j + 2 i + odd   (t: quad lane, j: MMA of the group, i: byte).
__host__ __device__ constexpr uint32_t rows_chunk_bytes(uint32_t mp, uint32_t digits) { return 2u * digits * mp * 64u; }
__host__ __device__ constexpr uint32_t rows_digits(uint32_t m, bool mis, bool f32) { return m == 1u || mis || (f32 && rows_dc(m)) ? 4u : 3u; }

// beside the digits: {sum of x', 2^-e} of every group and row, rows in pairs: {sum, sum, 2^-e, 2^-e}; DC: what a lane
// multiplies digits 0 and 1 with and what digits 2 and 3: {0, 2^-e, sum, 2^(16-e)} -- the sum beside the digits that weigh
__host__ __device__ constexpr uint32_t rows_scale_bytes(bool dc) { return dc ? 16u : 8u; }
__host__ __device__ inline size_t rows_smem_bytes(uint32_t mp, uint32_t part_chunks, bool mis, bool dc, uint32_t digits) {
    return (size_t)kRowsWarps * 2u * rows_half_bytes(mis) + (size_t)part_chunks * (rows_chunk_bytes(mp, digits) + 2u * mp * rows_scale_bytes(dc));
}

// Sums are carried 2^16 too small (2^12 with the weights' 16): a group's sum over 64 of the largest fp32 numbers stays finite.
constexpr float kRowsSumScale = 1.0f / 65536.0f;

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

// Exponent that puts a group's largest magnitude into [2^21, 2^22), or with four digits into [2^29, 2^30); both 2^e and 2^-e
// are normal numbers. Magnitudes below 2^-105 (2^-97) keep an absolute step of 2^-126.
__device__ __forceinline__ int rows_group_exponent(uint32_t amax_bits, int digits) { return min(126, (digits == 4 ? 156 : 148) - (int)(amax_bits >> 23)); }

__device__ __forceinline__ unsigned long long rows_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

template <int F>
struct Form {
    static constexpr int value = F;
};

template <int NB, bool DC, bool MIS, int D>
__global__ void __launch_bounds__(kRowsWarps * 32, 1) q4_rows_kernel(const __grid_constant__ RowsParams p) {
    constexpr uint32_t MP = (DC ? 2 : 8) * NB;
    constexpr uint32_t T = kRowsWarps * 32;
    constexpr uint32_t kHalf = rows_half_bytes(MIS), kTail = 4u * kRowsStageBytes, kParams = rows_weight_bytes(MIS);
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint32_t part = blockIdx.x % p.parts, gi = blockIdx.x / p.parts;
    // parts begin at multiples of four chunks: parameters are copied in 16-byte pieces of eight groups
    const uint32_t c_lo = q4_rows_part_begin(p.cpt, p.parts, part), c_hi = q4_rows_part_begin(p.cpt, p.parts, part + 1u), nch = c_hi - c_lo;
    uint8_t *xdig = smem + kRowsWarps * 2u * kHalf;
    float *xscale = reinterpret_cast<float *>(xdig + (size_t)p.part_chunks * rows_chunk_bytes(MP, D));
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem) + warp * 2u * kHalf;

    // ---- a tile's weights: lane l copies 16 bytes of row l >> 2 (and of the row eight further down) per chunk. The four 16-byte quarters of a row are stored with quarter q at q ^ (2 * bit 1 of the row), so
    // that the 8-byte reads below (lane (g, t): bytes 8 t.. of a group) touch every bank once per half-warp.
    const uint32_t cr = lane >> 2, cq = lane & 3u;
    const uint32_t copy_off = 16u * (cr * 4u + (cq ^ (2u * ((cr >> 1) & 1u))));
    // second window of the parameter row that lane l copies: row l & 15 of the fifth stage, quarter 1 (scales) or 2 (biases)
    const uint32_t second_off = kTail + 64u * (lane & 15u) + 16u * ((1u + (lane >> 4)) ^ (2u * ((lane >> 1) & 1u)));
    const uint64_t row_bytes = (uint64_t)p.k >> 1;
    const uint32_t quads = (nch + 3u) / 4u;
    const uint32_t worker = gi * kRowsWarps + warp;
    const uint32_t u0 = min(worker * p.run, p.tiles * quads), u1 = min(u0 + p.run, p.tiles * quads);  // this warp's quads of the part
    auto find_tile = [&](uint32_t tile, const RowsJob *&job, uint32_t &row0) {
        uint32_t ji = 0;
        while (ji + 1 < p.n_jobs && tile >= p.jobs[ji + 1].tile_begin) ++ji;
        job = &p.jobs[ji];
        row0 = (tile - job->tile_begin) * 16u;
    };

    // what is requested next: cursors at chunk pc of the run (chunks of one tile, up to pc_end) that is being requested
    const uint8_t *wa = nullptr, *wb = nullptr, *pw = nullptr;
    uint32_t wmis = 0;  // bytes by which the tile's weight rows miss a 16-byte boundary
    uint32_t pown = 0;  // the same for the parameter row that this lane copies
    uint32_t pu = u0, pc = 0, pc_end = 0;
    auto open_run = [&]() {
        const uint32_t tile = pu / quads, q = pu - tile * quads, q_end = min(quads, q + (u1 - pu));
        pc = c_lo + 4u * q;
        pc_end = min(c_lo + 4u * q_end, c_hi);
        pu += q_end - q;
        const RowsJob *job;
        uint32_t row0;
        find_tile(tile, job, row0);
        const uint32_t end = job->n - 1u;
        const uint32_t ra = min(row0 + cr, end), rb = min(row0 + 8u + cr, end);  // rows past n: read a valid row
        const uint32_t rp = min(row0 + (lane & 15u), end);
        if (MIS) wmis = (uint32_t)((uintptr_t)job->w & 15u);
        wa = job->w + (uint64_t)ra * row_bytes + cq * 16u + (size_t)pc * 64u - wmis;
        wb = job->w + (uint64_t)rb * row_bytes + cq * 16u + (size_t)pc * 64u - wmis;
        pw = ((lane >> 4) ? job->b : job->s) + ((size_t)rp * p.groups) * 2u + (size_t)pc * 4u;
        if (MIS) {
            pown = (uint32_t)((uintptr_t)pw & 15u);
            pw -= pown;
        }
    };
    auto request_quad = [&](uint32_t half) {  // the next quad of this warp's list
        if (pc >= pc_end && pu < u1) open_run();
        if (pc < pc_end) {
            const uint32_t base = ring + half * kHalf;
            if (!MIS || (pc + 4u <= pc_end && 2u * pc + 8u <= p.groups)) {
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    cp_async_16(base + s * kRowsStageBytes + copy_off, wa + s * 64);
                    cp_async_16(base + s * kRowsStageBytes + 512u + copy_off, wb + s * 64);
                }
                if (MIS) {
                    const bool pred = cq == 0 && q4_fifth_window_wanted(wmis, true);
                    cp_async_16_pred(base + kTail + copy_off, wa + 256, pred);
                    cp_async_16_pred(base + kTail + 512u + copy_off, wb + 256, pred);
                }
            } else {
                // at the end of a row only windows that hold bytes of the row (q4_decomp.h); the stage after the last chunk holds
                // the window that completes it
#pragma unroll
                for (int s = 0; s < 5; ++s) {
                    const uint32_t c = pc + s;
                    const bool fifth = cq == 0 && c == pc_end && q4_fifth_window_wanted(wmis, 2u * c - 1u < p.groups);
                    const bool pred = (s < 4 && c < pc_end) ? q4_window_wanted(cq, wmis, 2u * c + 1u < p.groups) : fifth;
                    cp_async_16_pred(base + s * kRowsStageBytes + copy_off, wa + s * 64, pred);
                    cp_async_16_pred(base + s * kRowsStageBytes + 512u + copy_off, wb + s * 64, pred);
                }
            }
            // lane l copies the scales (l < 16) or biases of row l & 15 for the quad's eight groups
            cp_async_16(base + kParams + lane * 16u, pw);
            if (MIS) cp_async_16_pred(base + second_off, pw + 16, pown + 2u * min(8u, p.groups - 2u * pc) > 16u);
            wa += 256;
            wb += 256;
            pw += 16;
            pc += 4u;
        }
        cp_async_commit();
    };
    unsigned long long *tr = (p.trace && lane == 0) ? p.trace + ((size_t)blockIdx.x * kRowsWarps + warp) * 4 : nullptr;
    if (tr) tr[0] = rows_ns();
    bool first_run = true;

    // activation, output and scratch depend on the kernel in front of this one, and weights the caller may write
    if (!p.weights_ahead) grid_dependency_wait();
    request_quad(0);
    request_quad(1);
    grid_dependency_wait();
    grid_dependents_launch();

    // ---- the part's digits for every row ----
    // Every thread holds its blocks of 8 inputs (at most kRowsPerThread) in registers, so that all of its loads are in
    // flight at once: one round trip to L2 instead of one per block.
    const uint32_t span8 = nch * 16u;  // blocks of 8 inputs per row in this part
    uint4 raw[kRowsPerThread][2];
    const uint32_t total8 = p.m * span8, todo8 = DC ? total8 : MP * span8;  // rows past m: zeros (DC: their columns stay zero)
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
        return xdig + (size_t)chunk * rows_chunk_bytes(MP, D) + (size_t)grp * D * MP * 64u + (size_t)mrow * (DC ? D * 64u : 64u);
    };
    auto store_scale = [&](uint32_t chunk, uint32_t grp, uint32_t mrow, float sum, float inv) {
        if (DC) {
            *reinterpret_cast<float4 *>(xscale + ((size_t)(chunk * 2u + grp) * MP + mrow) * 4u) = make_float4(0.f, inv, sum, inv * 65536.f);
        } else {
            float *dst = xscale + ((size_t)(chunk * 2u + grp) * (MP / 2u) + (mrow >> 1)) * 4u + (mrow & 1u);
            dst[0] = sum;
            dst[2] = inv;
        }
    };
    // the eight threads of a group agree on its scale (span8 is a multiple of 16: a group never leaves its half-warp)
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) {
        if ((uint32_t)i * T >= todo8) continue;  // (uniform)
        const uint32_t idx = threadIdx.x + i * T;
        const bool live = idx < todo8;
        const uint32_t mrow = live ? idx / span8 : 0u, b8 = live ? idx - mrow * span8 : 0u;
        float v[8];
        unpack8(raw[i], v);
        uint32_t mx = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) mx = max(mx, __float_as_uint(v[j]) & 0x7fffffffu);
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        const int e = rows_group_exponent(mx, D);
        const float scale = __uint_as_float((uint32_t)(e + 127) << 23), inv = __uint_as_float((uint32_t)(127 - e) << 23) * kRowsSumScale;
        int sum = 0, low = 0;  // (low: the lowest byte apart where 64 inputs of 30 bits would not fit)
        uint32_t z[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int xi = __float2int_rn(v[j] * scale);
            sum += D == 4 ? xi >> 8 : xi;
            if (D == 4) low += xi & 0xff;
            z[j] = ((uint32_t)xi + 0x00808080u) ^ 0x00808080u;  // bytes 0..2 (and 3): the signed digits
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        if (D == 4) {
            low += __shfl_xor_sync(0xffffffffu, low, 1);
            low += __shfl_xor_sync(0xffffffffu, low, 2);
            low += __shfl_xor_sync(0xffffffffu, low, 4);
        }
        const float total = D == 4 ? fmaf((float)sum, 256.f, (float)low) : (float)sum;
        if (live) {
            const uint32_t chunk = b8 >> 4, grp = (b8 >> 3) & 1u, b = b8 & 7u;  // block b of the group: inputs 8 b .. 8 b + 7
            uint8_t *dst = digits_at(chunk, grp, mrow) + 16u * (b >> 1) + 8u * (b & 1u);
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const uint32_t sel = (uint32_t)d | ((4u + (uint32_t)d) << 4);
                uint2 w;
                w.x = __byte_perm(__byte_perm(z[0], z[2], sel), __byte_perm(z[4], z[6], sel), 0x5410u);  // even inputs
                w.y = __byte_perm(__byte_perm(z[1], z[3], sel), __byte_perm(z[5], z[7], sel), 0x5410u);  // odd inputs
                *reinterpret_cast<uint2 *>(dst + (size_t)d * (DC ? 64u : MP * 64u)) = w;
            }
            // infinity or NaN: poison the row
            if (b == 0) store_scale(chunk, grp, mrow, mx >= 0x7f800000u ? __uint_as_float(0x7fc00000u) : total * inv, inv);
        }
    }
    __syncthreads();

    if (tr) tr[1] = rows_ns();

    // ---- tiles ----
    // B operands: digit d of row g of a block of eight (16 bytes from lane t); DC: digit g & 3 of row g >> 2 of a pair, zeros
    // in the columns of a fourth digit that there is not and of a row past m
    auto has_x = [&](int nb) { return (g & 3u) < (uint32_t)D && nb * 2u + (g >> 2) < p.m; };
    const uint32_t xdig_addr = (uint32_t)__cvta_generic_to_shared(xdig) + (DC ? (g >> 2) * (D * 64u) + (g & 3u) * 64u : g * 64u) + t * 16u;
    const uint32_t xscale_addr = (uint32_t)__cvta_generic_to_shared(xscale) + (DC ? (t >> 1) * 16u + (t & 1u) * 8u : t * 16u);
    constexpr int XD = DC ? 1 : D;  // B operands of a group and block of rows
    uint4 xf[2][NB][XD];
#pragma unroll
    for (int i = 0; i < 2 * NB * XD; ++i) (&xf[0][0][0])[i] = make_uint4(0, 0, 0, 0);
    // this lane's 8 bytes of group G of row g in a stage: word j = 4 G + t of the row's eight 8-byte words, in quarter
    // j >> 1, swizzled as above; words 8 and 9 (MIS) are the first two of the next stage
    const uint32_t rd_swz = 2u * ((g >> 1) & 1u);
    auto word_off = [&](uint32_t j) { return (j >> 3) * kRowsStageBytes + 16u * (g * 4u + (((j >> 1) & 3u) ^ rd_swz)) + 8u * (j & 1u); };
    const uint32_t rd0 = word_off(t), rd1 = word_off(4u + t);
    constexpr int AV = DC ? 2 : 4;  // sums a lane holds per tile and block of rows
    uint32_t half = 0;
    for (uint32_t u = u0; u < u1;) {
        const uint32_t tile = u / quads, q0 = u - tile * quads, q1 = min(quads, q0 + (u1 - u));
        const uint32_t c_begin = c_lo + 4u * q0, c_stop = min(c_lo + 4u * q1, c_hi);
        u += q1 - q0;
        const RowsJob *job;
        uint32_t row0;
        find_tile(tile, job, row0);
        uint32_t wm = 0, pmis = 0;  // pmis: of the parameter row this lane copied (and realigns)
        uint32_t rlo[2] = {0, 0}, rhi[2] = {0, 0};  // where this lane's two 8-byte words of each group are, from a chunk's stage
        if (MIS) {
            wm = (uint32_t)((uintptr_t)job->w & 15u);
            const uint32_t j = t + (wm >> 3);
            rlo[0] = word_off(j);
            rhi[0] = word_off(j + 1u);
            rlo[1] = word_off(j + 4u);
            rhi[1] = word_off(j + 5u);
            const uint32_t rp = min(row0 + (lane & 15u), job->n - 1u);
            pmis = ((uint32_t)(uintptr_t)((lane >> 4) ? job->b : job->s) + rp * p.groups * 2u) & 15u;  // (runs begin at multiples of 16 bytes)
        }
        float acc[NB][AV];
#pragma unroll
        for (int i = 0; i < NB * AV; ++i) (&acc[0][0])[i] = 0.f;
        uint32_t xc = xdig_addr + (c_begin - c_lo) * rows_chunk_bytes(MP, D);
        uint32_t xs = xscale_addr + (c_begin - c_lo) * (2u * MP * rows_scale_bytes(DC));
        for (uint32_t c = c_begin; c < c_stop; c += 4u) {
            cp_async_wait<1>();
            __syncwarp();
            const uint32_t base = ring + half * kHalf, pst = base + kParams;
            if (MIS) {
                // lane l shifts the parameter row it copied to the boundary, groups past the last one become zero
                const uint32_t left = p.groups - 2u * c;
                uint4 v = realign_16_any(lds_v4(pst + lane * 16u), lds_v4(base + second_off), pmis);
                if (left < 8u) {
                    uint32_t *r = &v.x;
#pragma unroll
                    for (uint32_t i = 0; i < 4u; ++i) r[i] = 2u * i >= left ? 0u : 2u * i + 1u >= left ? r[i] & 0xffffu : r[i];
                }
                sts_v4(pst + lane * 16u, v);
                __syncwarp();
            }
            // scales and biases of the quad's eight groups, rows g and g + 8
            uint4 prm[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) prm[i] = lds_v4(pst + (i >> 1) * 256u + (g + 8u * (i & 1)) * 16u);
            // One chunk. `form`: the weights are aligned (0), miss a boundary by less than four bytes of every eight (1) or by four
            // or more (2), or whatever wm says (3): a branch inside the chunk would keep the loads of one group from
            // overlapping the arithmetic of the one before it (one row x 248320 x 5120 at a byte offset: 164 -> 151 us).
            auto chunk = [&](auto form, int s) {
                constexpr int F = decltype(form)::value;
                const uint32_t stage = base + s * kRowsStageBytes;
                uint32_t pr[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) pr[i] = s == 0 ? prm[i].x : s == 1 ? prm[i].y : s == 2 ? prm[i].z : prm[i].w;
#pragma unroll
                for (int grp = 0; grp < 2; ++grp) {
                    uint4 xv[NB];  // {sum, sum, 2^-e, 2^-e} of rows 2 t, 2 t + 1 of this block of 8; DC: {sum, factor} of this lane
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) {
                        const uint32_t xcs = xc + s * rows_chunk_bytes(MP, D), xss = xs + s * (2u * MP * rows_scale_bytes(DC));
                        if constexpr (DC) {
                            lds_v4_keep(xf[grp][nb][0], xcs + (uint32_t)(grp * D * MP * 64 + nb * 2 * D * 64), has_x(nb));
                            const uint2 f = lds_v2(xss + (uint32_t)((grp * MP + nb * 2) * 16));
                            xv[nb] = make_uint4(f.x, f.y, 0, 0);
                        } else {
#pragma unroll
                            for (int d = 0; d < XD; ++d) xf[grp][nb][d] = lds_v4(xcs + (uint32_t)((grp * D + d) * MP + nb * 8) * 64u);
                            xv[nb] = lds_v4(xss + (uint32_t)(grp * MP + nb * 8) * 8u);
                        }
                    }
                    uint2 wA, wB;
                    if (F == 0 || (F == 3 && wm == 0)) {
                        wA = lds_v2(stage + (grp ? rd1 : rd0));
                        wB = lds_v2(stage + 512u + (grp ? rd1 : rd0));
                    } else {
                        // the word the lane's bytes begin in and the two after it: a 64-bit and a 32-bit read
                        const uint32_t a0 = stage + rlo[grp], a1 = stage + rhi[grp], sh = (wm & 3u) * 8u;
                        uint32_t va[3], vb[3];
                        if (F == 2 || (F == 3 && (wm & 4u))) {
                            const uint2 hiA = lds_v2(a1), hiB = lds_v2(a1 + 512u);
                            va[0] = lds_u32(a0 + 4u);
                            vb[0] = lds_u32(a0 + 516u);
                            va[1] = hiA.x;
                            va[2] = hiA.y;
                            vb[1] = hiB.x;
                            vb[2] = hiB.y;
                        } else {
                            const uint2 loA = lds_v2(a0), loB = lds_v2(a0 + 512u);
                            va[2] = lds_u32(a1);
                            vb[2] = lds_u32(a1 + 512u);
                            va[0] = loA.x;
                            va[1] = loA.y;
                            vb[0] = loB.x;
                            vb[1] = loB.y;
                        }
                        wA.x = __funnelshift_r(va[0], va[1], sh);
                        wA.y = __funnelshift_r(va[1], va[2], sh);
                        wB.x = __funnelshift_r(vb[0], vb[1], sh);
                        wB.y = __funnelshift_r(vb[1], vb[2], sh);
                    }
                    const uint32_t up = 0xf0f0f0f0u, flip = 0x80808080u;
                    const uint32_t a_lo0 = ((wA.x << 4) & up) ^ flip, a_hi0 = (wA.x & up) ^ flip, a_lo1 = ((wA.y << 4) & up) ^ flip, a_hi1 = (wA.y & up) ^ flip;
                    const uint32_t b_lo0 = ((wB.x << 4) & up) ^ flip, b_hi0 = (wB.x & up) ^ flip, b_lo1 = ((wB.y << 4) & up) ^ flip, b_hi1 = (wB.y & up) ^ flip;
                    const float sa = __uint_as_float(grp ? pr[0] & 0xffff0000u : pr[0] << 16), sb = __uint_as_float(grp ? pr[1] & 0xffff0000u : pr[1] << 16);
                    // (the MMAs' weights are 16 (q - 8): everything is carried 16 times too large until the end of the tile)
                    const float ba = fmaf(8.f, sa, __uint_as_float(grp ? pr[2] & 0xffff0000u : pr[2] << 16)) * 16.f;
                    const float bb = fmaf(8.f, sb, __uint_as_float(grp ? pr[3] & 0xffff0000u : pr[3] << 16)) * 16.f;
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) {
                        int q[XD][4];
#pragma unroll
                        for (int d = 0; d < XD; ++d) {
                            const uint4 &x = xf[grp][nb][d];
                            q[d][0] = q[d][1] = q[d][2] = q[d][3] = 0;
                            mma_s8s8_16832(q[d], a_lo0, b_lo0, a_hi0, b_hi0, x.x, x.y);
                            mma_s8s8_16832(q[d], a_lo1, b_lo1, a_hi1, b_hi1, x.z, x.w);
                        }
                        if constexpr (DC) {
                            // even lanes hold digits 0 and 1 of a row, odd ones digits 2 and 3; the two sums meet at the
                            // end of the tile
                            const float sum = __uint_as_float(xv[nb].x), f = __uint_as_float(xv[nb].y);
                            acc[nb][0] = fmaf(__int2float_rn(q[0][0] + (q[0][1] << 8)) * f, sa, fmaf(sum, ba, acc[nb][0]));
                            acc[nb][1] = fmaf(__int2float_rn(q[0][2] + (q[0][3] << 8)) * f, sb, fmaf(sum, bb, acc[nb][1]));
                        } else {
                            // the group's integer dot product: two exact sums of two digits (|q0 + 256 q1| < 2^29), put together
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const int hi = D == 4 ? q[XD / 2][i] + (q[XD - 1][i] << 8) : q[XD - 1][i];
                                const float dot = fmaf(__int2float_rn(hi), 65536.f, __int2float_rn(q[0][i] + (q[DC ? 0 : 1][i] << 8))) *
                                                  __uint_as_float((i & 1) ? xv[nb].w : xv[nb].z);
                                acc[nb][i] = fmaf(dot, i < 2 ? sa : sb, acc[nb][i]);
                            }
                            const float x0 = __uint_as_float(xv[nb].x), x1 = __uint_as_float(xv[nb].y);
                            acc[nb][0] = fmaf(x0, ba, acc[nb][0]);
                            acc[nb][1] = fmaf(x1, ba, acc[nb][1]);
                            acc[nb][AV - 2] = fmaf(x0, bb, acc[nb][AV - 2]);
                            acc[nb][AV - 1] = fmaf(x1, bb, acc[nb][AV - 1]);
                        }
                    }
                }
            };
            if (!MIS) {
#pragma unroll
                for (int s = 0; s < 4; ++s) chunk(Form<0>{}, s);
            } else if (c + 4u <= c_stop) {
                if (wm == 0) {
#pragma unroll
                    for (int s = 0; s < 4; ++s) chunk(Form<0>{}, s);
                } else if (!(wm & 4u)) {
#pragma unroll
                    for (int s = 0; s < 4; ++s) chunk(Form<MIS ? 1 : 0>{}, s);
                } else {
#pragma unroll
                    for (int s = 0; s < 4; ++s) chunk(Form<MIS ? 2 : 0>{}, s);
                }
            } else {
#pragma unroll
                for (int s = 0; s < 3; ++s)
                    if (c + s < c_stop) chunk(Form<MIS ? 3 : 0>{}, s);
            }
            __syncwarp();  // every lane is done with the half before it is refilled
            request_quad(half);
            half ^= 1u;
            xc += 4u * rows_chunk_bytes(MP, D);
            xs += 4u * (2u * MP * rows_scale_bytes(DC));
        }
        if (tr && first_run) tr[2] = rows_ns();
        first_run = false;

        // ---- the tile's contributions meet ----
        if constexpr (DC) {
#pragma unroll
            for (int i = 0; i < NB * AV; ++i) (&acc[0][0])[i] += __shfl_xor_sync(0xffffffffu, (&acc[0][0])[i], 1);
        }
#pragma unroll
        for (int i = 0; i < NB * AV; ++i) (&acc[0][0])[i] *= 1.0f / (16.0f * kRowsSumScale);
        // value i of a block of rows: activation row and weight row of the tile (DC: only even lanes store)
        auto act_row = [&](int nb, int i) { return DC ? nb * 2u + (t >> 1) : nb * 8u + 2u * t + (uint32_t)(i & 1); };
        auto weight_row = [&](int i) { return g + 8u * (uint32_t)(DC ? i : i >> 1); };
        const bool mine = !DC || (t & 1u) == 0;
        const uint32_t rows_total = p.tiles * 16u;
        const bool whole = p.parts == 1u && q0 == 0 && q1 == quads;
        uint32_t shares = 0;  // lane l: contributions of part l to this tile
        bool last = true;
        if (!whole) {
            const size_t slot = (size_t)part * p.part_slots + (worker - tile * quads / p.run);
#pragma unroll
                for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                    for (int i = 0; i < AV; ++i)
                        if (mine) p.partials[(slot * MP + act_row(nb, i)) * rows_total + (size_t)tile * 16u + weight_row(i)] = acc[nb][i];
            fence_gpu();
            __syncwarp();
            unsigned int before = 0;
            if (lane == 0) before = atomicAdd(p.counters + tile, 1u);
            if (lane < p.parts) {
                const uint32_t ql = (q4_rows_part_begin(p.cpt, p.parts, lane + 1u) - q4_rows_part_begin(p.cpt, p.parts, lane) + 3u) / 4u;
                shares = q4_rows_shares(tile, ql, p.run);
            }
            before = __shfl_sync(0xffffffffu, before, 0);
            last = before + 1u == __reduce_add_sync(0xffffffffu, shares);
            if (last) {
                fence_gpu();
                __syncwarp();
                if (lane == 0) p.counters[tile] = 0;  // ready for the next launch
            }
        }
        if (last) {
            if (!whole) {
                // all contributions in K order, whoever came last; four at a time, so that a round trip to L2 fetches four
#pragma unroll
                for (int i = 0; i < NB * AV; ++i) (&acc[0][0])[i] = 0.f;
                uint32_t pp = 0, jj = 0, n = __shfl_sync(0xffffffffu, shares, 0);
                while (pp < p.parts) {
                    constexpr int B = 4;
                    float got[B][NB * AV];
#pragma unroll
                    for (int b = 0; b < B; ++b) {
                        const bool have = pp < p.parts;  // (uniform)
                        const float *src = p.partials + ((size_t)pp * p.part_slots + jj) * MP * rows_total + (size_t)tile * 16u;
#pragma unroll
                        for (int v = 0; v < NB * AV; ++v) {
                            const int i = v % AV, nb = v / AV;
                            got[b][v] = have ? __ldcg(src + (size_t)act_row(nb, i) * rows_total + weight_row(i)) : 0.f;
                        }
                        if (have && ++jj == n) {
                            jj = 0;
                            n = __shfl_sync(0xffffffffu, shares, ++pp & 31u);
                        }
                    }
#pragma unroll
                    for (int b = 0; b < B; ++b)
#pragma unroll
                        for (int v = 0; v < NB * AV; ++v) (&acc[0][0])[v] += got[b][v];
                }
            }
#pragma unroll
                for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                    for (int i = 0; i < AV; ++i) {
                        const uint32_t mcol = act_row(nb, i), r = weight_row(i);
                        if (!mine || mcol >= p.m || row0 + r >= job->n) continue;
                        float *dst = job->out + (size_t)mcol * job->out_stride + row0 + r;
                        *dst = p.accumulate ? *dst + acc[nb][i] : acc[nb][i];
                    }
        }
    }
    cp_async_wait<0>();
    if (tr) tr[3] = rows_ns();
}

}  // namespace q4

// Largest part (in chunks) a block can hold for `mp` padded activation rows, 0 if not even
// four chunks fit.
static uint32_t rows_part_capacity(uint32_t mp, bool mis, bool dc, uint32_t digits) {
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    uint32_t chunks = 0;
    while (q4::rows_smem_bytes(mp, chunks + 1, mis, dc, digits) <= (size_t)optin && (chunks + 1) * mp <= 256u) ++chunks;
    return chunks >= 4 ? chunks : 0;
}

// Activation rows a launch takes: 16, or 8 where they are held with four digits.
extern "C" uint32_t q4k_rows_per_launch(int mis) { return mis ? 8u : 16u; }

// How the K range of a launch is cut: the number of parts (0: the shape is not supported) and the longest part. `mis`: the
// byte-addressed instance, which any K % 64 == 0 and any byte offset may use; the other one wants K % 512 == 0 and
// 16-byte alignment.
extern "C" uint32_t q4k_rows_plan(uint32_t m, uint32_t k, uint32_t tiles, uint32_t sm_count, int mis, int f32, uint32_t *part_chunks) {
    if (m < 1 || m > q4k_rows_per_launch(mis) || k == 0 || k % (mis ? 64u : 512u) != 0 || tiles == 0) return 0;
    const uint32_t mp = q4::rows_padded(m);
    const uint32_t cap = rows_part_capacity(mp, mis != 0, q4::rows_dc(m), q4::rows_digits(m, mis != 0, f32 != 0));
    return cap ? q4_rows_plan((k / 64u + 1u) / 2u, tiles, sm_count, cap, mp, part_chunks, nullptr) : 0u;
}

extern "C" uint32_t q4k_rows_padded(uint32_t m) { return q4::rows_padded(m); }

template <int NB, bool DC, bool MIS, int D>
static cudaError_t rows_launch(const q4::RowsParams &p, uint32_t grid, size_t smem, cudaStream_t stream) {
    const cudaError_t e = cudaFuncSetAttribute(q4::q4_rows_kernel<NB, DC, MIS, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return q4::launch_dependent(q4::q4_rows_kernel<NB, DC, MIS, D>, dim3(grid), q4::kRowsWarps * 32, smem, stream, p);
}

extern "C" cudaError_t q4k_rows(const q4::RowsParams *params, uint32_t sm_count, cudaStream_t stream) {
    const q4::RowsParams &p = *params;
    const uint32_t mp = q4::rows_padded(p.m);
    const bool mis = p.byte_addressed != 0, dc = q4::rows_dc(p.m);
    const uint32_t digits = q4::rows_digits(p.m, mis, p.x_is_f32 != 0);
    const size_t smem = q4::rows_smem_bytes(mp, p.part_chunks, mis, dc, digits);
    const uint32_t grid = (sm_count / p.parts) * p.parts;
    if (grid == 0 || p.run == 0 || p.m > q4k_rows_per_launch(mis)) return cudaErrorInvalidValue;
    if (mis) {
        if (mp == 2) return rows_launch<1, true, true, 4>(p, grid, smem, stream);
        if (mp == 4) return rows_launch<2, true, true, 4>(p, grid, smem, stream);
        return rows_launch<1, false, true, 4>(p, grid, smem, stream);
    }
    if (mp == 2) return digits == 4 ? rows_launch<1, true, false, 4>(p, grid, smem, stream) : rows_launch<1, true, false, 3>(p, grid, smem, stream);
    if (mp == 4) return digits == 4 ? rows_launch<2, true, false, 4>(p, grid, smem, stream) : rows_launch<2, true, false, 3>(p, grid, smem, stream);
    return mp == 8 ? rows_launch<1, false, false, 3>(p, grid, smem, stream) : rows_launch<2, false, false, 3>(p, grid, smem, stream);
}
