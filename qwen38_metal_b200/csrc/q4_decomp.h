// Work decomposition of the streaming (decode) projection kernel, shared by device and host
// code so the index arithmetic can be unit-tested on a CPU.
//
// A launch covers `tiles` row tiles (16 output rows each, over all jobs of the launch) times
// `cpt` K-chunks per tile (a chunk is 128 inputs = two affine groups = 64 packed bytes per
// row). The tiles*cpt units are numbered tile-major and cut into `workers` contiguous,
// near-equal ranges, one per warp. A tile whose units fall into more than one range is
// summed through per-warp partial slots by the last warp to arrive, in worker order.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define Q4_HD __host__ __device__ __forceinline__
#else
#define Q4_HD inline
#endif

struct Q4Split {
    uint64_t units;    // tiles * cpt
    uint32_t cpt;      // chunks per tile
    uint32_t workers;  // warps in the grid
};

// first unit of worker w (w may equal workers: one past the last unit)
Q4_HD uint64_t q4_split_begin(const Q4Split &s, uint32_t w) {
    return (s.units * (uint64_t)w) / s.workers;
}

// the worker whose range holds unit u
Q4_HD uint32_t q4_split_owner(const Q4Split &s, uint64_t u) {
    return (uint32_t)((((u + 1) * (uint64_t)s.workers) - 1) / s.units);
}

// workers contributing to the units [u0, u0 + span): [first, last]
Q4_HD void q4_split_span_contributors(const Q4Split &s, uint64_t u0, uint32_t span, uint32_t *first, uint32_t *last) {
    *first = q4_split_owner(s, u0);
    *last = q4_split_owner(s, u0 + span - 1);
}

// workers contributing to tile t when every tile has s.cpt units: [first, last]
Q4_HD void q4_split_contributors(const Q4Split &s, uint32_t tile, uint32_t *first, uint32_t *last) {
    q4_split_span_contributors(s, (uint64_t)tile * s.cpt, s.cpt, first, last);
}

// partial slot worker w uses for tile t: slot 0 when t is the tile its range starts in, else 1
Q4_HD uint32_t q4_split_slot(const Q4Split &s, uint32_t w, uint32_t tile) {
    uint32_t head_tile = (uint32_t)(q4_split_begin(s, w) / s.cpt);
    return 2u * w + (tile == head_tile ? 0u : 1u);
}

// Byte-addressed variant of the streaming kernel: which aligned 16-byte windows it asks for. A chunk is 64 packed
// bytes of a row: lanes t = 0,1 of a quad hold affine group A (bytes 0..31), lanes 2,3 group B (bytes 32..63), and
// the lane's window is the aligned 16 bytes that start `mis` bytes before its share ([16t - mis, 16t - mis + 16)); a
// lane completes its 16 bytes from the window after its own, so the quad needs a fifth window when mis != 0. Every
// window the kernel asks for holds at least one byte of the row, so nothing outside the 16-byte blocks that the
// tensor itself touches is ever read. `has_b`: group B of this chunk exists (the last chunk of a row with an odd
// number of groups has only group A).
Q4_HD bool q4_window_wanted(uint32_t t, uint32_t mis, bool has_b) {
    if (t < 2u) return true;
    if (t == 2u) return has_b || mis != 0u;  // its first `mis` bytes complete lane 1's share
    return has_b;
}
Q4_HD bool q4_fifth_window_wanted(uint32_t mis, bool has_b) { return has_b && mis != 0u; }
// chunks of a row in which lane t (0..3) of a quad has an affine group: group 2*chunk + (t >> 1) < groups
Q4_HD uint32_t q4_lane_chunks(uint32_t groups, uint32_t t) { return (groups + 1u - (t >> 1)) >> 1; }

// Short-batch kernel: the K range (cpt chunks of 128 inputs) is cut into `parts` runs that begin at multiples of four
// chunks (parameters travel in 16-byte pieces of eight groups). First chunk of `part`; part may equal parts (one past
// the last chunk).
Q4_HD uint32_t q4_rows_part_begin(uint32_t cpt, uint32_t parts, uint32_t part) {
    const uint32_t c = (((cpt + 3u) / 4u) * part / parts) * 4u;
    return c < cpt ? c : cpt;
}

// Inside a part the quads (four chunks) of all 16-row tiles are numbered tile-major and every warp of the part's blocks
// takes `run` consecutive ones. Contributions (warps) of a part with `quads` quads per tile to tile `tile`; warp
// tile * quads / run makes the first.
Q4_HD uint32_t q4_rows_shares(uint32_t tile, uint32_t quads, uint32_t run) { return (tile * quads + quads - 1u) / run - tile * quads / run + 1u; }

// quads a warp takes: the longest part's, spread over its warps
Q4_HD uint32_t q4_rows_run(uint32_t tiles, uint32_t part_chunks, uint32_t parts, uint32_t sm_count) {
    const uint32_t warps = sm_count / parts * 16u;
    return (tiles * ((part_chunks + 3u) / 4u) + warps - 1u) / warps;
}

// the most contributions any part makes to one tile
inline uint32_t q4_rows_part_slots(uint32_t cpt, uint32_t parts, uint32_t run) {
    uint32_t most = 1;
    for (uint32_t p = 0; p < parts; ++p) {
        const uint32_t quads = (q4_rows_part_begin(cpt, parts, p + 1u) - q4_rows_part_begin(cpt, parts, p) + 3u) / 4u;
        const uint32_t n = run % quads == 0 ? 1u : quads % run == 0 ? quads / run : (quads - 1u + run - 1u) / run + 1u;
        most = n > most ? n : most;
    }
    return most;
}

// How many parts to cut K into for `tiles` 16-row tiles on `sm_count` SMs of 16 warps, when a block can hold at most `cap`
// chunks of activation digits of `mp` rows; 0 when no split fits.
// *part_chunks: chunks of the longest part; *cost_out: the estimate the choice was made by.
// Cost of a split in chunk times: the chunks of a warp's run, about three more for a tile it finishes alone and six for one
// whose sums meet in scratch, and the conversion of the part's activation before the first chunk.
Q4_HD uint32_t q4_rows_plan(uint32_t cpt, uint32_t tiles, uint32_t sm_count, uint32_t cap, uint32_t mp, uint32_t *part_chunks, double *cost_out) {
    if (cpt == 0 || tiles == 0 || sm_count == 0) return 0;
    const uint32_t all = (cpt + 3u) / 4u;
    if ((uint64_t)tiles * all + (uint64_t)all * 65536u > 0xffffffffull) return 0;  // quads are counted in 32 bits
    uint32_t best = 0;
    double best_cost = 0.0;
    for (uint32_t parts = 1; parts <= all && parts <= sm_count && parts <= 32u; ++parts) {
        const uint32_t quads = (all + parts - 1u) / parts;
        if (quads * 4u > cap && !(parts == 1u && cpt <= cap)) continue;
        const uint32_t run = q4_rows_run(tiles, quads * 4u, parts, sm_count);
        const bool split = run % quads != 0;
        const uint32_t pieces = (run + quads - 1u) / quads + (split && quads % run != 0 ? 1u : 0u);
        const double piece = parts == 1u ? 3.0 : 6.0;
        const double cost = 4.0 * run + pieces * piece + (split ? 6.0 : 0.0) + 0.02 * mp * quads * 4.0 + 0.3 * parts;
        if (best == 0 || cost < best_cost * 0.98) {
            best_cost = cost;
            best = parts;
        }
    }
    if (best == 0) return 0;
    *part_chunks = ((all + best - 1u) / best) * 4u;
    if (*part_chunks > cpt) *part_chunks = cpt;
    if (cost_out) *cost_out = best_cost;
    return best;
}

// ---- tensor-core GEMM (q4_gemm_tc.cu): how a launch is cut ----

struct Q4GemmPlan {
    uint32_t bn;            // activation rows per tile: a multiple of 32, at most 256
    uint32_t accs, stages;  // accumulators and A stages in TMEM: accs * bn + 64 * stages <= 512 columns
    uint32_t tiles, tiles_m;  // output tiles of 256 weight rows x bn activation rows; tiles along m
    uint32_t workers;       // CTA pairs
    uint32_t full_rounds;   // whole tiles per worker ...
    uint32_t tail_workers;  // ... and workers that share the K stages of the tiles left over
    uint64_t partial_floats;  // scratch for the parts of tiles that are cut between workers
    uint32_t counters;
};

// The most scratch any plan asks for: two parts of a 256 x 256 tile per worker, and a counter per warp's share of the tiles left
// over after the whole rounds, of which there are fewer than two per worker.
inline uint64_t q4_gemm_most_partial_floats(uint32_t pairs) { return (uint64_t)pairs * 2u * 256u * 256u; }
inline uint32_t q4_gemm_most_counters(uint32_t pairs) { return (2u * pairs - 1u) * 8u; }

// row tiles of an n-row projection: 256 weight rows of one tensor, or (pair mode) 128 gate rows and the same up rows
Q4_HD uint32_t q4_gemm_row_tiles(uint32_t n, uint32_t pair) { return pair ? (n + 127u) / 128u : (n + 255u) / 256u; }

// K stages of 128 inputs (two affine groups)
Q4_HD uint32_t q4_gemm_k_stages(uint32_t k) { return (k / 64u + 1u) / 2u; }

// The plan with the smallest estimate, in SM cycles. A stage of bn activation rows takes 4 bn cycles of MMA, but no
// less than the ~600 in which an SM's warps expand 128 x 128 weights; a tile's epilogue takes about 20 cycles a column
// and is hidden when there are two accumulators (bn <= 128); every part of a tile that is cut costs another pass over
// bn columns, and the last one adds them all up.
// Candidates: the fewest activation tiles and up to two more (narrower tiles waste less on ragged m); whole tiles for
// everybody, or all but the last one or two rounds whole and the rest cut along K over all workers, or over fewer
// workers when there is little to cut.
inline void q4_gemm_plan(uint32_t m, uint32_t k, uint32_t row_tiles, uint32_t pairs, Q4GemmPlan *plan) {
    const uint32_t ks = q4_gemm_k_stages(k);
    double best = 0.0;
    bool have = false;
    for (uint32_t tm = (m + 255u) / 256u, tries = 0; tries < 3u; ++tm, ++tries) {
        const uint32_t bn = (((m + tm - 1u) / tm) + 31u) & ~31u;
        if (tries > 0 && bn < 96u) break;
        const uint32_t tiles_m = (m + bn - 1u) / bn, tiles = row_tiles * tiles_m;
        const uint32_t accs = bn <= 128u ? 2u : 1u;
        const uint32_t stages = (512u - accs * bn) / 64u < 8u ? (512u - accs * bn) / 64u : 8u;
        const double stage = 4.0 * bn > 600.0 ? 4.0 * bn : 600.0, epilogue = 20.0 * bn + 1000.0, shown = accs == 2u ? 0.0 : epilogue;
        auto consider = [&](uint32_t workers, uint32_t rounds, uint32_t tail_workers) {
            const uint32_t whole = rounds * workers < tiles ? rounds * workers : tiles, rest = tiles - whole;
            double cost = rounds * (ks * stage + shown) + epilogue;
            if (rest) {
                const uint64_t units = (uint64_t)rest * ks;
                const double run = (double)((units + tail_workers - 1u) / tail_workers);
                const double parts = ks / run < 1.0 ? 2.0 : ks / run + 1.0;  // contributors of a tile
                cost += run * stage + 2000.0 + epilogue + parts * bn * 10.0;
            }
            if (have && cost >= best) return;
            have = true;
            best = cost;
            plan->bn = bn;
            plan->accs = accs;
            plan->stages = stages;
            plan->tiles = tiles;
            plan->tiles_m = tiles_m;
            plan->workers = workers;
            plan->full_rounds = rounds;
            plan->tail_workers = rest ? tail_workers : 0u;
            plan->partial_floats = rest ? (uint64_t)tail_workers * 2u * bn * 256u : 0u;
            plan->counters = rest * 8u;
        };
        if (tiles <= pairs) {
            consider(tiles, 1u, 0u);
            for (uint32_t parts = 2; tiles * (parts - 1u) < pairs && parts <= ks; ++parts) {
                const uint32_t w = tiles * parts < pairs ? tiles * parts : pairs;
                if ((uint64_t)w <= (uint64_t)tiles * ks) consider(w, 0u, w);
            }
        } else {
            consider(pairs, (tiles + pairs - 1u) / pairs, 0u);
            if (tiles % pairs) consider(pairs, tiles / pairs - 1u, pairs);
        }
    }
}
