// Kernel-side parameter blocks and launcher prototypes shared between the .cu files and the
// host runtime (q4_runtime.cu). Plain C structs: no CUDA types beyond cudaStream_t/cudaError_t.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "q4_decomp.h"

namespace q4 {

constexpr int kMaxJobs = 12;

// One projection of a grouped launch (the device image of a MappedQ4AffineJob,
// src/metal_runtime.rs:155-192 of the reference, with shard ids resolved to pointers).
struct GemvJob {
    const uint8_t *w;      // packed weights, [n][k/8] u32, any byte alignment
    const uint8_t *s;      // scales, [n][k/64] bf16
    const uint8_t *b;      // biases, [n][k/64] bf16
    float *out;            // [m][out_stride] fp32
    uint32_t n;            // output rows
    uint32_t out_stride;   // elements between activation rows of `out`
    uint32_t tile_begin;   // first 16-row tile of this job in the launch
    uint32_t w_misalign;   // (uintptr_t)w & 15
    // persistent decode kernel only: a tile of this job counts as `vcpt` >= cpt units when the launch's work is cut
    // into equal ranges -- the units past cpt are empty, so projections whose chunks cost more (weights at a byte
    // offset) get proportionally fewer real chunks per warp; unit_begin = first unit of the job
    uint32_t vcpt;
    uint32_t unit_begin;
};

struct GemvParams {
    GemvJob jobs[kMaxJobs];
    uint32_t n_jobs;
    const uint16_t *xp;    // prepared activation columns, [v_cols][kp] fp16 in fragment order, row-scaled
    const float *xsum;     // [kp/64][vpad] per-group column sums
    const float *row_inv;  // [m_rows] inverse of the power-of-two row scaling
    uint32_t v_cols;       // activation columns in use (m_rows, or 3*m_rows for fp32 input)
    uint32_t vpad;         // 4 * column tiles
    uint32_t m_rows;       // activation rows
    uint32_t x_is_f32;     // columns are hi/mid/lo splits of fp32 rows
    uint32_t accumulate;   // out += projection (residual form) instead of out = projection
    uint32_t k;            // input elements
    uint32_t kp;           // k rounded up to 128 (row stride of xp)
    uint32_t groups;       // k / 64
    uint32_t cpt;          // K-chunks (128 inputs) per tile = ceil(groups / 2)
    uint32_t workers;      // warps (= blocks) in the grid
    uint64_t units;        // tiles * cpt
    float *partials;       // [workers][2][column tiles][32][4] fp32 scratch for split tiles
    unsigned int *counters;  // [workers], zero between launches
    unsigned long long *trace;  // optional [workers][4] globaltimer stamps (start, first data, loop end, done); may be null
    // Row-sharded multi-GPU runs: mirror[job * kMaxPeers + r] is where rank r keeps the same output rows
    // (peer memory), or null; every result is stored there too. Null table on one GPU.
    float *const *mirror;
    uint32_t world, rank;
};

constexpr int kMaxPeers = 8;

// Short-batch kernel (q4_gemv_rows.cu): up to 16 activation rows.
struct RowsJob {
    const uint8_t *w, *s, *b;
    float *out;            // [m][out_stride] fp32
    uint32_t n;            // output rows
    uint32_t out_stride;
    uint32_t tile_begin;   // first 16-row tile of this job in the launch
    uint32_t pad;
};

struct RowsParams {
    RowsJob jobs[kMaxJobs];
    uint32_t n_jobs;
    uint32_t m;            // activation rows, 1..16
    const void *x;         // [m][k] bf16 or fp32, 16-byte aligned
    uint32_t x_is_f32;
    uint32_t k, groups, cpt;  // inputs, k / 64, chunks of 128 inputs (the last may hold one group)
    uint32_t parts;        // runs the K range is cut into (q4k_rows_plan)
    uint32_t part_chunks;  // chunks of the longest run
    uint32_t tiles;        // 16-row tiles of all jobs
    uint32_t run;          // quads of chunks per warp (q4_rows_run)
    uint32_t part_slots;   // most contributions a part makes to one tile (q4_rows_part_slots)
    uint32_t accumulate;
    uint32_t weights_ahead;  // weights may be requested before the kernel in front has finished
    uint32_t byte_addressed;  // some tensor misses a 16-byte boundary, or K % 512 != 0
    float *partials;       // [parts][part_slots][padded rows][tiles * 16] fp32, for tiles with several contributions
    unsigned int *counters;  // [tiles], zero between launches
    unsigned long long *trace;  // optional [warps of the grid][4] globaltimer stamps (start, digits ready, first tile streamed, done)
};

// One projection of a tensor-core launch (q4_gemm_tc.cu): any byte alignment.
struct GemmJob {
    const uint8_t *w, *s, *b;
    float *out;            // [m][n] fp32
    uint32_t n;            // output rows
};

}  // namespace q4

extern "C" {
cudaError_t q4k_prepare_x(const void *x, int x_is_f32, uint32_t m_rows, uint32_t k, uint32_t kp, uint32_t vpad,
                          uint16_t *xp, float *xsum, float *row_inv, cudaStream_t stream);
cudaError_t q4k_gemv(const q4::GemvParams *params, int column_tiles, int aligned, cudaStream_t stream);  // one warp per block
uint32_t q4k_gemv_occupancy(int column_tiles, int aligned);  // resident warps per SM, 0 on error

uint32_t q4k_rows_plan(uint32_t m, uint32_t k, uint32_t tiles, uint32_t sm_count, int mis, int f32, uint32_t *part_chunks);  // parts, 0: unsupported
uint32_t q4k_rows_per_launch(int mis);  // most rows of a launch
uint32_t q4k_rows_padded(uint32_t m);  // activation rows a launch of m rows holds
cudaError_t q4k_rows(const q4::RowsParams *params, uint32_t sm_count, cudaStream_t stream);

cudaError_t q4k_swiglu(const float *gate, const float *up, uint64_t count, float *out_f32, uint16_t *out_bf16,
                       cudaStream_t stream);
cudaError_t q4k_f32_to_bf16(const float *in, uint64_t count, uint16_t *out, cudaStream_t stream);
uint32_t q4k_argmax_parts(uint32_t n);
cudaError_t q4k_argmax_rows(const float *logits, uint32_t m, uint32_t n, uint32_t index_base, float *pv, uint32_t *pi,
                            uint32_t *tokens, float *values, cudaStream_t stream);
cudaError_t q4k_rms_unit_bf16(const float *in, uint32_t rows, uint32_t n, float eps, uint16_t *out, cudaStream_t stream);
cudaError_t q4k_dequantize_row(const uint8_t *w, const uint8_t *s, const uint8_t *b, uint32_t k, uint32_t row, float *out,
                               cudaStream_t stream);

cudaError_t q4k_gemm_prepare_x(const void *x, int x_is_f32, uint64_t elements, uint16_t *xp, cudaStream_t stream);
cudaError_t q4k_gemm_tc(const Q4GemmPlan *plan, const uint16_t *xp, uint32_t m, uint32_t k, const q4::GemmJob *jobs, uint32_t n_jobs,
                        uint16_t *h_out, uint32_t h_stride, int accumulate, int *error_flag, float *partials, unsigned int *counters,
                        cudaStream_t stream);
int q4k_gemm_pair_supported(const uint8_t *w_gate, const uint8_t *w_up);

cudaError_t q4k_synth_q4(uint64_t seed, uint64_t tensor, float sigma, uint64_t row0, uint64_t rows, uint32_t k,
                         uint8_t *w, uint8_t *s, uint8_t *b, cudaStream_t stream);
cudaError_t q4k_synth_bf16(uint64_t seed, uint64_t tensor, uint64_t count, uint16_t *out, cudaStream_t stream);
}
