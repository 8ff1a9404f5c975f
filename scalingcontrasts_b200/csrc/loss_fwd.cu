// Forward tile kernel of the streamed Matryoshka sigmoid loss: scores a block of candidates against this rank's rows at
// every prefix, applies the sigmoid loss cell by cell, and leaves per band the suffix-summed gradient with respect to
// the raw dot product (bfloat16) plus per-row partial sums. Optionally the same launch pulls the NEXT peer's block
// from that peer's memory into local staging, so the NVLink transfer hides under this block's tensor-core work.
//
// Shape of the work. A tile is 128 query rows x 64 candidates, scored by one CTA, or 128 x 128, scored by a pair of CTAs (a cluster of
// two): each loads half the rows and half the candidates, the UMMAs of the pair read both, and each CTA scores its 64 rows
// against all 128 candidates, so that a cell costs a third fewer operand bytes. The hidden axis streams through shared memory in
// stages of 64 channels (TMA, 128-byte swizzle), widest channels first. Every band of the ladder owns one 64-column
// slot of tensor memory and the UMMAs of a 16-channel step accumulate into the slot of the band that contains the
// step, so each channel is multiplied exactly once (depth H per cell, where a sweep-and-subtract scheme spends up to
// 2H). The eight slots form a ring: while the epilogue warps drain the K slots of tile t, the issuing thread already
// fills the widest bands of tile t+1. A thread of the epilogue takes its columns eight at a time and holds all bands' values
// of a chunk in registers: the segment dots come in, the prefix dots run up the ladder, the raw-dot gradients (without the
// factor beta / |q_k| that the row and band share) replace the dots, and the suffix sums that go to the gradient cube run
// down the ladder. A tile's slots go back to the issuer when its last chunk has been loaded. Ladders of five and more bands
// keep some or all of their gradients in the tensor-memory slots the dots came from until the suffix sums reach them
// (fwd_parked_bands_for, fwd_rolled_for).
//
// Warp roles (640 threads): warps 0-15 epilogue (warp w owns tensor-memory lanes 32*(w%4).. and the 16 columns w/4 of
// the tile; four warps per scheduler keep the issue slots busy), warp 16 TMA producer (and the candidates' norms), warp 17
// UMMA issuer and tensor-memory owner (each loop run by one elected lane), warp 18 peer pull (plain 16-byte loads from the
// peer's replica, plain stores to local staging; never a TMA load from another GPU's memory), warp 19 the fused kernel's second issuer. The epilogue's four warpgroups run with 104
// registers a thread, the helpers' with 64.
//
// What bounds it (B200, one block of 4096 rows, H=768, K=5, off the diagonal: 75 us): the epilogue, which by itself takes about 60 (cells
// 6.4 k of a tile's 9 k cycles: a warp's instructions wait for one another, and four warps to a scheduler do not hide all of it).
// A single CTA's operands and UMMAs by themselves took 41. One block of 16384 rows (1.13 ms): the memory side as well; a single CTA's loads and
// the cube's stores without any arithmetic took 1.05 ms, and the GPU runs at its power limit.
//
// A CTA or pair walks work items (row strip, run of consecutive candidate tiles) in a fixed round-robin order and writes one
// partial record per (run, column quarter, row); the fold over records happens in a fixed order elsewhere, so the loss
// summands do not depend on scheduling.
//
// Parity: forward_tile_cuda_ and score_forward_row_ (scalingcontrasts.cuh:688-1040) and fold of its row partials;
// the staging copy of streamed_loss_t::score (scalingcontrasts.cuh:1262-1265) is what the pull warps replace.
#include <stdexcept>
#include <string>

#include "api.h"
#include "common.cuh"
#include "driver.h"
#include "launch.h"

namespace sc {

namespace {

constexpr uint32_t fwd_rows = 128; // of a strip: one CTA's, or a pair's
constexpr uint32_t fwd_depth = 64;
constexpr uint32_t fwd_max_stages = 8;
// The kernel's forms. A CTA scores tiles of 128 rows x 64 candidates by itself (`form_single`, and `form_fused`, which also runs the
// gradient GEMM), or two CTAs, a cluster, score tiles of 128 x 128 together (`form_pair`, and `form_pair_apart` for blocks that
// hold no row's own copy or partner: nothing of what those need is in it). See forward_form for which is taken when.
enum form_t { form_single, form_pair, form_pair_apart, form_fused };
__host__ __device__ constexpr bool fwd_paired(form_t form) { return form == form_pair || form == form_pair_apart; }
__host__ __device__ constexpr uint32_t fwd_cols_for(form_t form) { return fwd_paired(form) ? 128u : 64u; }
__host__ __device__ constexpr uint32_t fwd_ctas_for(form_t form) { return fwd_paired(form) ? 2u : 1u; }
constexpr uint32_t fwd_max_slots = 8;
// Tensor-memory slots of the score accumulators: all eight 64-column slots, or six when the last 128 columns hold the
// gradient GEMM's accumulator.
__host__ __device__ constexpr uint32_t fwd_slots_for(form_t form) { return form == form_fused ? 6u : 8u; }
constexpr uint32_t fwd_slot_columns = 64;
constexpr uint32_t fwd_tmem_columns = 512;
// The gradient GEMM that the fused kernel runs beside the scoring: 128 rows x up to 128 channels per accumulator, the
// candidate index as the K dimension in stages of 64, two stages of [128 rows of the gradient patch | 128 channels of
// the transposed candidates].
constexpr uint32_t fz_max_prefixes = 6;
constexpr uint32_t fz_depth = 64;
constexpr uint32_t fz_max_width = 128;
constexpr uint32_t fz_a_bytes = 128 * fz_depth * 2;
constexpr uint32_t fz_b_bytes = fz_max_width * fz_depth * 2;
constexpr uint32_t fz_stage_bytes = fz_a_bytes + fz_b_bytes;
constexpr uint32_t fz_stages = 2;
constexpr uint32_t fz_accumulator_column = 6 * fwd_slot_columns;
constexpr uint32_t fz_max_tiles = 48;
constexpr uint32_t fz_candidate_maps = 4; // boxes of 16, 32, 64 and 128 channels
constexpr uint32_t fz_max_tiles_per_run = 16;
constexpr uint32_t fwd_epilogue_warps = 16; // four per scheduler
constexpr uint32_t fwd_epilogue_threads = fwd_epilogue_warps * 32;
constexpr uint32_t fwd_column_groups = fwd_epilogue_warps / 4;             // warps that share a lane quadrant
constexpr uint32_t fwd_warp_columns = fwd_slot_columns / fwd_column_groups; // columns of a tile that one warp owns
// Columns a thread takes at a time: all bands' values of a chunk are held in registers together.
// Ladders of seven and eight bands go band by band instead (`rolled`), sixteen columns at a time: their values do not fit the
// registers, and eight bands times three forms of the cell math are more code than the instruction cache likes. One block
// of 4096 rows, H=1024, K=8: 215 us with half the bands parked, 190 us band by band; at six bands 150 us either way, and 153
// against 161 us where every cell takes the general form, so six stay with two bands parked.
__host__ __device__ constexpr bool fwd_rolled_for(int prefixes) { return prefixes >= 7; }
__host__ __device__ constexpr int fwd_chunk_columns_for(int prefixes) { return prefixes <= 1 || fwd_rolled_for(prefixes) ? 16 : 8; }
// The narrowest bands, where the registers have no room for them beside four others: their gradients are parked in the tensor
// memory their dots came from until the suffix sums reach them, and their slots are released later than the others'. With all
// five bands of K=5 in registers the kernel spilled 72 bytes each way: one block of 4096 rows, H=768, took 90.7 us and, with every
// cell in the general form, 133.9 us; with one band parked it takes 87.9 and 125.0; two blocks of 16384 rows as a
// whole step 4.06 and 5.22 ms against 4.06 and 5.14 (at that size the GPU runs at its power limit).
__host__ __device__ constexpr int fwd_parked_bands_for(int prefixes) {
    return fwd_rolled_for(prefixes) ? prefixes - 2 : (prefixes > 4 ? prefixes - 4 : 0);
}
static_assert(fwd_warp_columns == 16, "a warp's store patch of a band is 32 rows x 16 columns");
constexpr uint32_t fwd_producer_warp = fwd_epilogue_warps;
constexpr uint32_t fwd_mma_warp = fwd_epilogue_warps + 1;
constexpr uint32_t fwd_first_pull_warp = fwd_epilogue_warps + 2;
constexpr uint32_t fwd_pull_warps = 1;
constexpr uint32_t fz_mma_warp = fwd_epilogue_warps + 3; // fused kernel only; the pull warp doubles as its producer
// Twenty warps, five warpgroups: four of epilogue warps, one of helpers (the last helper works in the fused kernel only).
// Launched with 96 registers a thread, of which the helpers' warpgroup hands most on: 512 x 104 + 128 x 64 = 640 x 96.
constexpr uint32_t fwd_threads = 32 * (fwd_epilogue_warps + 4);
constexpr uint32_t fwd_epilogue_registers = 104, fwd_helper_registers = 64, fwd_launch_registers = 96;
static_assert(fwd_epilogue_threads * fwd_epilogue_registers + (fwd_threads - fwd_epilogue_threads) * fwd_helper_registers <=
                  fwd_threads * fwd_launch_registers,
              "the register split must not exceed what the block is launched with");
// A CTA's share of a stage: its rows of the strip and its part of the tile's candidates.
__host__ __device__ constexpr uint32_t fwd_own_rows(form_t form) { return fwd_rows / fwd_ctas_for(form); }
__host__ __device__ constexpr uint32_t fwd_own_cols(form_t form) { return fwd_cols_for(form) / fwd_ctas_for(form); }
__host__ __device__ constexpr uint32_t fwd_q_bytes(form_t form) { return fwd_own_rows(form) * fwd_depth * 2; }
__host__ __device__ constexpr uint32_t fwd_stage_bytes(form_t form) { return fwd_q_bytes(form) + fwd_own_cols(form) * fwd_depth * 2; }
constexpr uint32_t fwd_tile_barriers = 8;
constexpr float log2_e = 1.4426950408889634f;
// (logit + bias) * log2(e) below these: the series may be cut. At e < 2^-8 three terms leave out e^3 / 4 of log1p(e) (1.5e-8
// relative) and e^3 of e / (1 + e) (6e-8, half a float32 step); at e < 2^-5 five terms leave out e^5 / 6 (5e-9) and e^5 (3e-8).
constexpr float easy_negative_limit = -8.0f;
constexpr float near_negative_limit = -5.0f;
constexpr float left_out_logit = -1000.0f; // a base-two exponential of zero

constexpr uint32_t fwd_norm_slots = 4;

struct fwd_tail {
    uint64_t stage_full[fwd_max_stages];
    uint64_t stage_empty[fwd_max_stages];
    // Tile t's accumulators have been read by every epilogue warp (index t % fwd_slots): all bands', or, where the narrowest
    // bands are parked, the others' (`tile_taken`, with a third of the tile's work still to come) and the parked ones'.
    uint64_t tile_taken[fwd_max_slots];
    uint64_t tile_parked_taken[fwd_max_slots];
    uint64_t tile_full[fwd_tile_barriers];
    // The candidate norms of tile t are in ring entry t % fwd_norm_slots / have been read by every epilogue warp.
    uint64_t norms_full[fwd_norm_slots];
    uint64_t norms_empty[fwd_norm_slots];
    // Fused kernel: the gradient GEMM's stage ring, "this item's gradient patches are in memory" (one per scratch
    // buffer, an arrival per epilogue warp), and the hand-over of its single accumulator.
    uint64_t fz_stage_full[fz_stages];
    uint64_t fz_stage_empty[fz_stages];
    uint64_t fz_item_stored[2];
    uint64_t fz_accumulator_full;
    uint64_t fz_accumulator_empty;
    uint32_t tmem_base;
    uint32_t abort_flag;
};
constexpr uint32_t fwd_tail_bytes = (sizeof(fwd_tail) + 127) / 128 * 128;
// Ring of candidate norms, one entry per tile in flight: [prefixes][columns] inverse norms, then [8] maxima per 64 columns.
__host__ __device__ constexpr uint32_t fwd_norm_floats(uint32_t prefixes, form_t form) {
    return prefixes * fwd_cols_for(form) + 8 * (fwd_cols_for(form) / 64);
}
__host__ __device__ constexpr uint32_t fwd_norm_bytes(uint32_t prefixes, form_t form) { return fwd_norm_slots * fwd_norm_floats(prefixes, form) * 4; }
// Per epilogue thread and band the row factor beta / |q_k|: in shared memory where the bands' values leave no registers for
// it (chunks of eight columns times four or more bands), in registers otherwise. Band by band, the row's loss and
// coefficient as well.
__host__ __device__ constexpr bool fwd_factors_in_shared(uint32_t prefixes, form_t form) { return form != form_fused && prefixes >= 4; }
__host__ __device__ constexpr uint32_t fwd_factor_bytes(uint32_t prefixes, form_t form) {
    return (fwd_rolled_for(prefixes) ? 3u : (fwd_factors_in_shared(prefixes, form) ? 1u : 0u)) * prefixes * fwd_epilogue_threads * 4;
}
// Per epilogue warp and band (four in rotation when the bands go one by one) a patch of [32 rows][16 columns] bfloat16, from
// which the gradient cube is written by TMA stores.
constexpr uint32_t fwd_store_patch_bytes = 32 * fwd_warp_columns * 2;
__host__ __device__ constexpr uint32_t fwd_store_patches(uint32_t prefixes) { return fwd_rolled_for(prefixes) ? 4u : prefixes; }
__host__ __device__ constexpr uint32_t fwd_store_bytes(uint32_t prefixes) {
    return fwd_epilogue_warps * fwd_store_patches(prefixes) * fwd_store_patch_bytes;
}
// Stages of the score operands: as many as the rest of the shared memory leaves room for. The fused kernel keeps room for
// the gradient GEMM's stages and runs the scores on what is left (three at five prefixes, two at six).
constexpr uint32_t fwd_shared_limit = 227 * 1024;
__host__ __device__ constexpr uint32_t fwd_stages_for(uint32_t prefixes, form_t form) {
    uint32_t const rest = 1024 + (form == form_fused ? fz_stages * fz_stage_bytes : 0u) + fwd_store_bytes(prefixes) + fwd_tail_bytes +
                          fwd_norm_bytes(prefixes, form) + fwd_factor_bytes(prefixes, form);
    uint32_t const fit = (fwd_shared_limit - rest) / fwd_stage_bytes(form);
    return fit < fwd_max_stages ? fit : fwd_max_stages;
}
static_assert(fwd_stages_for(8, form_pair) >= 3 && fwd_stages_for(fz_max_prefixes, form_fused) >= 2, "the score operands need a ring of stages");
__host__ __device__ constexpr uint32_t fwd_stage_region_bytes(uint32_t prefixes, form_t form) {
    return fwd_stages_for(prefixes, form) * fwd_stage_bytes(form) + (form == form_fused ? fz_stages * fz_stage_bytes : 0u);
}
__host__ __device__ constexpr uint32_t fwd_shared_bytes(uint32_t prefixes, form_t form) {
    return 1024 + fwd_stage_region_bytes(prefixes, form) + fwd_store_bytes(prefixes) + fwd_tail_bytes + fwd_norm_bytes(prefixes, form) +
           fwd_factor_bytes(prefixes, form);
}

struct fwd_params {
    float const* q_inv;
    float const* c_inv;
    float const* c_tile_max;
    __nv_bfloat16* cube;
    float* partials;
    uint32_t* status;
    uint32_t rows_q, rows_c, hidden;
    ladder_t ladder;
    uint32_t tiles_per_run, tiles_per_strip, runs_per_strip, items; // a strip's last run may be shorter
    float beta, bias, weight;
    float const* scalars; // optional device copy of {beta, bias}: learnable values never visit the host
    uint64_t query_base, candidate_base;
    uint32_t spec_code;
    uint64_t budget_ns;
    pull_request pull;
    unsigned long long* trace; // optional: phase cycle counters of CTA 0 (see forward_trace_slots in api.h)
    // One word per 64-channel chunk, one byte per 16-channel step of the chunk: non-zero when, walking the channels
    // downwards, the step is the first of a band (the topmost step, or the step just below a band's first channel).
    // Kept in the kernel's parameters: the issuer's lane has them without a load from global memory. hidden <= 4096.
    uint32_t band_starts[64];
    // Fused kernel only. The gradient GEMM's channel tiles, one word each: band | first channel / 16 << 4 | width / 16
    // << 16; a tile never crosses a band edge, so its A operand is one band's patch.
    float* gradient;       // [rows_q, hidden] float32, accumulated with vector reductions
    float gradient_scale;  // the loss's 2 / live, applied as the accumulator leaves tensor memory
    uint32_t tile_count;
    uint32_t tiles[fz_max_tiles];
};

// The tensor maps only the fused kernel uses: one over the per-CTA scratch of gradient patches (box of 128 rows x 64
// candidates, 128-byte swizzle: the GEMM's A operand) and the transposed candidates under boxes of 16 << index channels.
struct fz_maps {
    CUtensorMap patches;
    CUtensorMap candidates[fz_candidate_maps];
};

// Phase timers, compiled in only with -DSC_FWD_TRACE=1 (a diagnostic build: the clock reads and their branches cost the
// epilogue a few percent of its issue slots). A role keeps its cycle counters in registers and adds them to the trace
// array once, when it is done, so that timing a phase costs a clock read and not a round trip to memory. Only CTA 0
// records. Without the flag the type is empty and the `trace` argument is ignored.
#ifndef SC_FWD_TRACE
#define SC_FWD_TRACE 0
#endif
#if SC_FWD_TRACE
struct phase_timer {
    long long since;
    unsigned long long cycles[4];
    bool on;
    __device__ __forceinline__ explicit phase_timer(fwd_params const& p) : since(0), cycles{0, 0, 0, 0}, on(false) {
#ifdef __CUDA_ARCH__
        on = p.trace != nullptr && blockIdx.x == 0;
        since = clock64();
#endif
    }
    __device__ __forceinline__ void only_if(bool keep) { on = on && keep; }
    // Adds the cycles since the last call to counter `which` (0..3 of this role) and restarts the clock.
    __device__ __forceinline__ void lap(int which) {
#ifdef __CUDA_ARCH__
        if (on) {
            long long const now = clock64();
            cycles[which] += static_cast<unsigned long long>(now - since);
            since = now;
        }
#endif
    }
    __device__ __forceinline__ void flush(fwd_params const& p, int first_slot, int count) {
        if (on)
            for (int i = 0; i < count; ++i) p.trace[first_slot + i] += cycles[i];
    }
};
#else
struct phase_timer {
    __device__ __forceinline__ explicit phase_timer(fwd_params const&) {}
    __device__ __forceinline__ void only_if(bool) {}
    __device__ __forceinline__ void lap(int) {}
    __device__ __forceinline__ void flush(fwd_params const&, int, int) {}
};
#endif

// ---- the cell math ----------------------------------------------------------------------------------------------
// Accumulators are kept without the 1/N weight: `g` sums -mask*z*(1-sigmoid(s)), `loss` sums mask*softplus(-s),
// `coefficient` sums raw gradient * dot; the weight is applied once when the partial record is written.
// The cell pass forms each band's raw-dot gradients without the factor beta / |q_k| that is common to the row and the
// band; the suffix pass multiplies it in while it sums the bands. The norms kernel writes an inverse
// norm of 0 for a row of zero norm (factor 0, and its cosines are floored anyway); the cap only keeps a huge inverse
// norm of a tiny row from turning 0 * factor into a NaN.
__device__ __forceinline__ float row_factor(float beta, float inv_q) { return beta * fminf(inv_q, 1e30f); }

// Any cell: positives, the diagonal, floored cosines. Returns what the cell adds to each of the row's sums.
struct cell_outcome {
    float raw, loss, cell;
};
__device__ __forceinline__ cell_outcome cell_general(float prefix_dot, float inv_q, float inv_c, float beta, float bias,
                                                     bool own, bool partner, uint32_t spec_code) {
    uint32_t const diagonal = (spec_code >> 1) & 3u; // 0 own, 1 negative, 2 skip
    float z = partner ? 1.0f : -1.0f;
    float mask = 1.0f;
    if (own) {
        if (diagonal == 0u) z = 1.0f;
        if (diagonal == 2u) mask = 0.0f;
    }
    float const inverse_denominator = fminf(inv_q * inv_c, 100.0f);
    bool const floored = inverse_denominator >= 100.0f;
    float const cosine = floored ? 0.0f : prefix_dot * inverse_denominator;
    float const s = z * (beta * (own ? 1.0f : cosine) + bias);
    float const d = fast_ex2(-fabsf(s) * log2_e);
    float const complement = (s >= 0.0f ? d : 1.0f) * fast_rcp(1.0f + d);
    float const cell = -mask * z * complement;
    float const raw = (own || floored) ? 0.0f : cell * inverse_denominator * beta;
    return cell_outcome{raw, mask * (fmaxf(-s, 0.0f) + log1p_unit(d)), cell};
}

template <int columns_> __device__ __forceinline__ void tmem_load(uint32_t taddr, uint32_t (&r)[columns_]) {
    static_assert(columns_ == 8 || columns_ == 16, "tensor-memory loads of 8 or 16 columns");
    if constexpr (columns_ == 16) {
        tmem_load_16(taddr, r);
    } else {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr)
                     : "memory");
    }
}
__device__ __forceinline__ void tmem_store_16(uint32_t taddr, uint32_t const (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_store_8(uint32_t taddr, uint32_t const (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- roles ------------------------------------------------------------------------------------------------------
// The producer and UMMA roles' loops are run by one elected lane: a chunk of the issue loop costs 228 cycles (192 of them its four
// UMMAs), where the whole warp walking it, with only the TMA / UMMA / commit instructions under the elected lane's predicate,
// took 379 (votes over the waits' answers, reconvergence after every predicated block). One block of 4096 rows, H=768, K=5:
// 88.9 -> 81 us, H=1024, K=1: 72.6 -> 58 us. They wait on their barriers without sleeping in between (the suspended wait takes
// no issue slots worth counting; with naps of 200 and 20 ns the same blocks take 82.4 and 60.4 us).
// (The timed part of the epilogue's wait is a function of its own: one function cannot serve both sides of the register split.)
__device__ __forceinline__ bool mbar_wait_lane(uint32_t bar, uint32_t parity, wait_context const& ctx, uint32_t site, uint32_t detail) {
#pragma unroll 1
    for (int spin = 0; spin < 16; ++spin)
        if (mbar_try_wait(bar, parity)) return true;
    return mbar_wait_sleeping(bar, parity, ctx.status, ctx.budget_ns, ctx.abort_flag, site, detail, 0u);
}
// The same for tensor-memory slots that both CTAs of a pair give back.
__device__ __forceinline__ bool mbar_wait_lane_cluster(uint32_t bar, uint32_t parity, wait_context const& ctx, uint32_t site, uint32_t detail) {
#pragma unroll 1
    for (int spin = 0; spin < 16; ++spin)
        if (mbar_try_wait_cluster(bar, parity)) return true;
    return mbar_wait_sleeping(bar, parity, ctx.status, ctx.budget_ns, ctx.abort_flag, site, detail, 0u) && mbar_try_wait_cluster(bar, parity);
}
constexpr uint32_t sleep_gemm_ns = 500; // the fused kernel's gradient GEMM runs a whole item behind

// The items of a CTA or pair: every so many-th of the list.
template <form_t form_> __device__ __forceinline__ uint32_t item_count(uint32_t items) {
    uint32_t const walkers = gridDim.x / fwd_ctas_for(form_), walker = blockIdx.x / fwd_ctas_for(form_);
    return (items + walkers - 1 - walker) / walkers;
}
template <form_t form_> __device__ __forceinline__ uint32_t item_at(uint32_t n) {
    return blockIdx.x / fwd_ctas_for(form_) + n * (gridDim.x / fwd_ctas_for(form_));
}

// Tiles of a strip's run: a divisor of the tiles of 64, but not always of those of 128.
template <form_t form_> __device__ __forceinline__ uint32_t run_length(fwd_params const& p, uint32_t run) {
    if constexpr (!fwd_paired(form_)) return p.tiles_per_run;
    else return min(p.tiles_per_run, p.tiles_per_strip - run * p.tiles_per_run);
}

// The producer also brings the candidates' inverse norms of a tile (and their maxima) into the ring the epilogue warps read
// them from: plain loads at the start of the tile, stored once the tile's operand loads have been issued.
template <int prefixes_, form_t form_>
__device__ __forceinline__ void producer_role(CUtensorMap const* q_map, CUtensorMap const* c_map, fwd_params const& p,
                                              uint32_t stages_base, float* norm_ring, fwd_tail* tail,
                                              wait_context const& ctx, uint32_t const rank) {
    constexpr uint32_t stages = fwd_stages_for(prefixes_, form_), columns = fwd_cols_for(form_), halves = columns / 32;
    bool const elected = elect_one();
    uint32_t const lane = threadIdx.x % 32;
    uint32_t stage = 0, phase = 0, tile_local = 0;
    uint32_t const chunks = p.hidden / fwd_depth;
    uint32_t const maxima = p.rows_c / 64;
    phase_timer timer(p);
    timer.only_if(elected);
    for (uint32_t n = 0, count = item_count<form_>(p.items); n < count; ++n) {
        uint32_t const item = item_at<form_>(n);
        uint32_t const strip = item / p.runs_per_strip, run = item % p.runs_per_strip;
        for (uint32_t t = 0, length = run_length<form_>(p, run); t < length; ++t, ++tile_local) {
            uint32_t const first_column = (run * p.tiles_per_run + t) * columns;
            float norms[halves * prefixes_], largest = 0.0f;
#pragma unroll
            for (int j = 0; j < static_cast<int>(halves) * prefixes_; ++j) {
                size_t const at = static_cast<size_t>(j / halves) * p.rows_c + first_column + (j % halves) * 32u + lane;
                norms[j] = SC_IN_BOUNDS(at, static_cast<size_t>(prefixes_) * p.rows_c) ? *(p.c_inv + at) : 0.0f;
            }
            // Lane 8 h + k: band k's largest inverse norm among the tile's h-th 64 columns.
            uint32_t const maximum = first_column / 64 + lane / 8;
            if (lane % 8 < prefixes_ && lane / 8 < columns / 64 &&
                SC_IN_BOUNDS(static_cast<size_t>(lane % 8) * maxima + maximum, static_cast<size_t>(prefixes_) * maxima))
                largest = *(p.c_tile_max + static_cast<size_t>(lane % 8) * maxima + maximum);
            bool ok = true;
            if (elected) {
                for (int chunk = static_cast<int>(chunks) - 1; chunk >= 0; --chunk) {
                    timer.lap(0);
                    ok = mbar_wait_lane(smem_u32(&tail->stage_empty[stage]), phase ^ 1u, ctx, site_fwd_stage_empty, item);
                    if (!ok) break;
                    timer.lap(1);
                    uint32_t const full = smem_u32(&tail->stage_full[stage]);
                    uint32_t const destination = stages_base + stage * fwd_stage_bytes(form_);
                    int const x = chunk * static_cast<int>(fwd_depth);
                    int const q_row = static_cast<int>(strip * fwd_rows + rank * fwd_own_rows(form_));
                    int const c_row = static_cast<int>(first_column + rank * fwd_own_cols(form_));
                    if constexpr (fwd_paired(form_)) {
                        // The first CTA's barrier counts both CTAs' bytes, whichever arrive first.
                        uint32_t const counted = smem_of(full, 0);
                        if (rank == 0) mbar_arrive_expect_tx(full, 2 * fwd_stage_bytes(form_));
                        tma_load_2d_pair(destination, q_map, counted, x, q_row);
                        tma_load_2d_pair(destination + fwd_q_bytes(form_), c_map, counted, x, c_row);
                    } else {
                        mbar_arrive_expect_tx(full, fwd_stage_bytes(form_));
                        tma_load_2d(destination, q_map, full, x, q_row);
                        tma_load_2d(destination + fwd_q_bytes(form_), c_map, full, x, c_row);
                    }
                    if (++stage == stages) stage = 0, phase ^= 1u;
                }
            }
            if (!__all_sync(0xFFFFFFFFu, ok)) return;
            uint32_t const entry = tile_local % fwd_norm_slots;
            if (!__all_sync(0xFFFFFFFFu, mbar_wait_lane(smem_u32(&tail->norms_empty[entry]), ((tile_local / fwd_norm_slots) & 1u) ^ 1u,
                                                        ctx, site_fwd_norms_empty, item)))
                return;
            float* const into = norm_ring + entry * fwd_norm_floats(prefixes_, form_);
#pragma unroll
            for (int j = 0; j < static_cast<int>(halves) * prefixes_; ++j) into[(j / halves) * columns + (j % halves) * 32u + lane] = norms[j];
            if (lane < columns / 8) into[prefixes_ * columns + lane] = largest;
            __syncwarp();
            if (elected) mbar_arrive(smem_u32(&tail->norms_full[entry]));
        }
    }
    timer.flush(p, 0, 2);
}

template <int prefixes_, form_t form_>
__device__ __forceinline__ void mma_role(fwd_params const& p, uint32_t stages_base, fwd_tail* tail, uint32_t tmem_base,
                                         wait_context const& ctx) {
    constexpr uint32_t fwd_slots = fwd_slots_for(form_);
    constexpr uint32_t idesc = umma_idesc_bf16(fwd_rows, fwd_cols_for(form_));
    constexpr uint32_t parked = fwd_parked_bands_for(prefixes_);
    constexpr uint32_t descriptor_high = (1024u >> 4) | (1u << 14) | (2u << 29); // stride 1024 B, version 1, 128-byte swizzle
    if (!elect_one()) return;
    uint32_t const chunks = p.hidden / fwd_depth;
    uint32_t const low_base = ((stages_base & 0x3FFFFu) >> 4) | (1u << 16);
    uint32_t stage = 0, phase = 0, unit = 0, tile_local = 0, seen = 0, seen_parked = 0;
    phase_timer timer(p);
    auto multiply = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
        if constexpr (fwd_paired(form_)) umma_bf16_pair(d, a, b, idesc, accumulate);
        else umma_bf16(d, a, b, idesc, accumulate);
    };
    auto commit = [&](uint32_t bar) { // to both CTAs of a pair
        if constexpr (fwd_paired(form_)) umma_commit_pair(smem_of(bar, 0)), umma_commit_pair(smem_of(bar, 1));
        else umma_commit(bar);
    };
    // The next band's slot, once it is free. The slot's last user was unit - fwd_slots, a band of tile `needed`; the
    // epilogue must have read it out. Releases are observed here strictly in tile order, per barrier array, so a barrier's
    // parity can never be a full turn ahead of the one waited for: tile X + fwd_slots cannot even be issued before tile X's release has been
    // seen.
    uint32_t slot_address = 0;
    auto take_slot = [&]() -> bool {
        if (unit >= fwd_slots) {
            uint32_t const needed = (unit - fwd_slots) / prefixes_;
            bool const was_parked = parked > 0 && (unit - fwd_slots) % prefixes_ >= prefixes_ - parked; // ranks run from the widest
            uint64_t* const barriers = was_parked ? tail->tile_parked_taken : tail->tile_taken;
            uint32_t& observed = was_parked ? seen_parked : seen;
            timer.lap(0);
            while (observed <= needed) {
                uint32_t const given_back = smem_u32(&barriers[observed % fwd_slots]), parity = (observed / fwd_slots) & 1u;
                if (!(fwd_paired(form_) ? mbar_wait_lane_cluster(given_back, parity, ctx, site_fwd_slot_empty, unit)
                                        : mbar_wait_lane(given_back, parity, ctx, site_fwd_slot_empty, unit)))
                    return false;
                ++observed;
            }
            timer.lap(2);
            tcgen05_fence_after();
        }
        slot_address = tmem_base + unit % fwd_slots * fwd_slot_columns;
        ++unit;
        return true;
    };
    for (uint32_t n = 0, count = item_count<form_>(p.items); n < count; ++n) {
        for (uint32_t t = 0, length = run_length<form_>(p, item_at<form_>(n) % p.runs_per_strip); t < length; ++t) {
            for (int chunk = static_cast<int>(chunks) - 1; chunk >= 0; --chunk) {
                uint32_t const starts = p.band_starts[chunk];
                timer.lap(0);
                if (!mbar_wait_lane(smem_u32(&tail->stage_full[stage]), phase, ctx, site_fwd_stage_full, tile_local))
                    return;
                timer.lap(1);
                tcgen05_fence_after();
                uint32_t const low = low_base + stage * (fwd_stage_bytes(form_) >> 4);
                uint64_t q_descriptor, c_descriptor;
                asm("mov.b64 %0, {%1, %2};" : "=l"(q_descriptor) : "r"(low), "r"(descriptor_high));
                asm("mov.b64 %0, {%1, %2};" : "=l"(c_descriptor) : "r"(low + (fwd_q_bytes(form_) >> 4)), "r"(descriptor_high));
                uint32_t const empty = smem_u32(&tail->stage_empty[stage]);
                // A step of 16 channels advances both descriptors by 32 bytes. Steps run from the chunk's top down; a band
                // that starts inside the chunk (its edge is not a multiple of 64) takes the step-by-step way.
                if ((starts & 0x00FFFFFFu) == 0u) {
                    if (starts != 0u && !take_slot()) return;
                    multiply(slot_address, q_descriptor + 6, c_descriptor + 6, starts != 0u ? 0u : 1u);
                    multiply(slot_address, q_descriptor + 4, c_descriptor + 4, 1u);
                    multiply(slot_address, q_descriptor + 2, c_descriptor + 2, 1u);
                    multiply(slot_address, q_descriptor, c_descriptor, 1u);
                } else {
#pragma unroll 1
                    for (int sub = 3; sub >= 0; --sub) {
                        bool const begins = ((starts >> (8 * sub)) & 0xFFu) != 0u;
                        if (begins && !take_slot()) return;
                        multiply(slot_address, q_descriptor + 2u * sub, c_descriptor + 2u * sub, begins ? 0u : 1u);
                    }
                }
                commit(empty);
                if (++stage == fwd_stages_for(prefixes_, form_)) stage = 0, phase ^= 1u;
            }
            commit(smem_u32(&tail->tile_full[tile_local % fwd_tile_barriers]));
            ++tile_local;
        }
    }
    timer.flush(p, 2, 3);
}

// Position of a CTA in its walk over (work item, tile of the run).
template <form_t form_> struct tile_cursor {
    uint32_t n, t, strip, run;
    __device__ __forceinline__ void go_to(fwd_params const& p, uint32_t to) {
        uint32_t const item = item_at<form_>(to);
        n = to, t = 0, strip = item / p.runs_per_strip, run = item % p.runs_per_strip;
    }
    __device__ __forceinline__ void advance(fwd_params const& p) {
        if (++t == run_length<form_>(p, run)) go_to(p, n + 1);
    }
    __device__ __forceinline__ uint32_t column_tile(fwd_params const& p) const { return run * p.tiles_per_run + t; }
};

// Fused kernel: one warp's share of a finished accumulator of the gradient GEMM, added to the owner's rows. The
// accumulator is [128 rows x width channels]; the warp owns the 32 rows of its lane quadrant and every fourth 16-column
// chunk, starting at its column group. A real call: the code exists once and the hot loops keep their registers.
__device__ __noinline__ void fz_drain_chunks(float* destination, uint32_t chunks, uint32_t accumulator, uint32_t group,
                                             float scale) {
    for (uint32_t chunk = group; chunk < chunks; chunk += fwd_column_groups) {
        uint32_t values[16];
        tmem_load_16(accumulator + chunk * 16u, values);
        tmem_load_wait();
#pragma unroll
        for (int v = 0; v < 4; ++v)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(destination + chunk * 16u + 4 * v),
                         "f"(scale * __uint_as_float(values[4 * v])), "f"(scale * __uint_as_float(values[4 * v + 1])),
                         "f"(scale * __uint_as_float(values[4 * v + 2])), "f"(scale * __uint_as_float(values[4 * v + 3]))
                         : "memory");
    }
}

// Where band `band` of the tile whose widest band is unit `first_unit` of the ring has its slot.
template <int prefixes_, form_t form_> __device__ __forceinline__ uint32_t band_slot(uint32_t first_unit, uint32_t band) {
    return ((first_unit + (prefixes_ - 1 - band)) % fwd_slots_for(form_)) * fwd_slot_columns;
}

// In a patch that the diagonal crosses, a row's own copy and its pair partner: each thread scores its two cells (where the
// patch has them) band by band in their general form, and leaves the band's loss, coefficient and the partner's raw-dot
// gradient (without the row factor; a row's own copy has none) in 16 bytes of shared memory per lane and band: the second half
// of the lane's row in the warp's own store patches, which is idle until the last chunk is stored. The common path then
// takes the patch with those cells left out. A real call with a rolled loop over the bands, so that the common path keeps its
// registers. (Sending all of such a patch's cells through the general form, and the gradients back to the common path through
// tensor memory, made a launch whose block holds the diagonal 28 us longer at 4096 rows.)
struct special_sums {
    float cell, own_logit;
};
__device__ __forceinline__ float pick_column(uint32_t const (&d)[16], uint32_t column) {
    uint32_t eight[8], four[4], two[2];
#pragma unroll
    for (int c = 0; c < 8; ++c) eight[c] = (column & 8u) ? d[c + 8] : d[c];
#pragma unroll
    for (int c = 0; c < 4; ++c) four[c] = (column & 4u) ? eight[c + 4] : eight[c];
#pragma unroll
    for (int c = 0; c < 2; ++c) two[c] = (column & 2u) ? four[c + 2] : four[c];
    return __uint_as_float((column & 1u) ? two[1] : two[0]);
}
template <int prefixes_, form_t form_>
__device__ __noinline__ special_sums special_cells(uint32_t lane_base, uint32_t first_unit, float const* norms,
                                                   float const* q_inv, uint32_t rows_q, float beta, float bias,
                                                   int own_column, int partner_column, uint32_t spec_code, uint32_t sums,
                                                   uint32_t sums_stride) {
    static_assert(fwd_warp_columns == 16, "a patch is sixteen columns wide");
    special_sums total{0.0f, 0.0f};
    float own_dot = 0.0f, partner_dot = 0.0f;
#pragma unroll 1
    for (int k = 0; k < prefixes_; ++k) {
        uint32_t d[16];
        tmem_load<16>(lane_base + band_slot<prefixes_, form_>(first_unit, k), d);
        float const inv_q = *(q_inv + static_cast<size_t>(k) * rows_q);
        float const row_beta = row_factor(beta, inv_q);
        float const without_row_factor = row_beta != 0.0f ? __fdividef(1.0f, row_beta) : 0.0f;
        float loss = 0.0f, coefficient = 0.0f, partner_raw = 0.0f;
        tmem_load_wait();
        own_dot += pick_column(d, static_cast<uint32_t>(own_column));
        partner_dot += pick_column(d, static_cast<uint32_t>(partner_column));
        if (own_column >= 0) {
            cell_outcome const cell = cell_general(own_dot, inv_q, norms[k * fwd_cols_for(form_) + own_column], beta, bias, true, false, spec_code);
            loss += cell.loss;
            total.cell += cell.cell, total.own_logit += cell.cell * beta;
        }
        if (partner_column >= 0) {
            cell_outcome const cell =
                cell_general(partner_dot, inv_q, norms[k * fwd_cols_for(form_) + partner_column], beta, bias, false, true, spec_code);
            loss += cell.loss;
            total.cell += cell.cell;
            partner_raw = cell.raw * without_row_factor;
            coefficient = partner_raw * partner_dot;
        }
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(sums + k * sums_stride), "f"(loss),
                     "f"(coefficient), "f"(partner_raw), "f"(0.0f) : "memory");
    }
    return total;
}

// Epilogue warps: warp w owns tensor-memory lanes 32*(w%4).. (a quarter of the tile's rows) and the column group w/4 of
// the tile (16 columns each with sixteen warps). A thread takes its columns in chunks; of a chunk it holds every band's
// values in registers from the tensor-memory load to the store: segment dots come in, the prefix dots run up the ladder,
// raw-dot gradients replace the dots, and the suffix sums run down the ladder straight from the same registers. Up to four
// bands nothing is parked in tensor memory in between, so a tile's slots go back to the issuer as soon as its last chunk has been
// loaded, about half a tile before the epilogue is done with it; above that the narrowest bands' gradients wait in their
// slots, which go back later than the others'.
//
// What it costs: eleven packed float32 instructions per pair of cells and prefix, two cycles each, and one exponential per
// cell, eight cycles; about 5000 cycles of a tile's 9700 at K=5 are bound by these. One block of 4096 rows, H=768, K=5: 98 ->
// 88 us off the diagonal, 123 -> 89 us on it, against the form that parked every band in tensor memory.
template <int prefixes_, form_t form_>
__device__ __forceinline__ void epilogue_role(CUtensorMap const* cube_map, fwd_params const& p, fwd_tail* tail,
                                              uint32_t store_base, float const* norm_ring, float* row_factors, uint32_t tmem_base,
                                              wait_context const& ctx, uint32_t warp, uint32_t lane, uint32_t rank) {
    constexpr uint32_t fwd_slots = fwd_slots_for(form_);
    constexpr int columns = fwd_chunk_columns_for(prefixes_);
    constexpr int parked = fwd_parked_bands_for(prefixes_);
    constexpr bool rolled = fwd_rolled_for(prefixes_);
    constexpr int warp_columns = fwd_warp_columns;
    uint32_t const quadrant = warp % 4, group = warp / 4;
    // Where the warp's patch lies in the strip and in the tile. A CTA of a pair has half the strip's rows; the upper half of its
    // tensor-memory lanes holds the same rows' products with the tile's second 64 candidates.
    uint32_t const patch_row = fwd_paired(form_) ? rank * fwd_own_rows(form_) + quadrant % 2 * 32 : quadrant * 32;
    uint32_t const column_half = fwd_paired(form_) ? quadrant / 2 : 0u;
    uint32_t const patch_column = column_half * 64 + group * fwd_warp_columns;
    uint32_t const row_local = patch_row + lane;
    uint32_t const lane_base = tmem_base + ((quadrant * 32u) << 16) + group * warp_columns;
    uint32_t const quantities = 2 + 2 * prefixes_;
    float const beta = p.scalars != nullptr ? *p.scalars : p.beta;
    float const bias = p.scalars != nullptr ? *(p.scalars + 1) : p.bias;
    uint32_t tile_local = 0;
    uint32_t const warp_store_base = store_base + warp * fwd_store_patches(prefixes_) * fwd_store_patch_bytes;

    tile_cursor<form_> cursor;
    cursor.go_to(p, 0);
    uint32_t const items = item_count<form_>(p.items);
    // Per-row sums of the item, in registers or in the thread's own words of shared memory; `coefficient` is kept without the
    // row factor beta / |q_k|. Lane k of a warp holds the largest inverse norm of the warp's rows at band k (`rows_max`).
    constexpr bool shared_factors = fwd_factors_in_shared(prefixes_, form_);
    constexpr int factor_stride = shared_factors ? fwd_epilogue_threads : 1;
    float own_factors[shared_factors ? 1 : prefixes_];
    float* const row_beta = shared_factors ? row_factors + threadIdx.x : own_factors;
    constexpr int sums_kept = rolled ? 1 : prefixes_;
    float loss[sums_kept] = {}, coefficient[sums_kept] = {};
    float* const band_sums = row_factors + threadIdx.x + prefixes_ * fwd_epilogue_threads; // rolled: [2 * prefixes_] strided
    auto add_sums = [&](int k, float to_loss, float to_coefficient) {
        if constexpr (rolled) {
            band_sums[k * fwd_epilogue_threads] += to_loss;
            band_sums[(prefixes_ + k) * fwd_epilogue_threads] += to_coefficient;
        } else {
            loss[k] += to_loss, coefficient[k] += to_coefficient;
        }
    };
    float g = 0.0f, own_logit = 0.0f, rows_max = 0.0f;
    auto give_back = [&](uint64_t* barrier) { // slots, to the issuer: in a pair the first CTA's
        if constexpr (fwd_paired(form_)) mbar_arrive_cluster(smem_of(smem_u32(barrier), 0));
        else mbar_arrive(smem_u32(barrier));
    };
    uint32_t row = 0;
    phase_timer timer(p);
    timer.only_if(threadIdx.x == 0);

    // Fused kernel: the gradient GEMM of a finished item runs on the tensor cores while these warps score the next
    // item. Its accumulators (one per channel tile, `tile_count` per item, in item order) are drained here: whichever
    // are ready at the top of a tile, and, before the scratch buffer of item n - 1 is written again by item n + 1,
    // everything up to item n - 1 (by then long done). `drained` counts the accumulators this warp has taken; the
    // GEMM does not start accumulator u + 1 before all sixteen warps have taken u, so the barrier's parity is exact.
    uint32_t items_done = 0, drained = 0;
    auto drain = [&](uint32_t limit, bool blocking) -> bool {
        while (drained < limit) {
            uint32_t const full = smem_u32(&tail->fz_accumulator_full);
            if (blocking) {
                if (!mbar_wait(full, drained & 1u, ctx, site_fz_accumulator_full, drained)) return false;
            } else if (__shfl_sync(0xFFFFFFFFu, mbar_test_wait(full, drained & 1u) ? 1 : 0, 0) == 0) {
                break;
            }
            tcgen05_fence_after();
            uint32_t const item = item_at<form_>(drained / p.tile_count);
            uint32_t const word = p.tiles[drained % p.tile_count];
            float* const destination = p.gradient +
                                       (static_cast<size_t>(item / p.runs_per_strip) * fwd_rows + row_local) * p.hidden +
                                       ((word >> 4) & 0xFFFu) * 16u;
            if (SC_WARP_IN_BOUNDS((static_cast<size_t>(item / p.runs_per_strip) * fwd_rows + row_local) * p.hidden +
                                      ((word >> 4) & 0xFFFu) * 16u + (word >> 16) * 16u - 1,
                                  static_cast<size_t>(p.rows_q) * p.hidden))
                fz_drain_chunks(destination, word >> 16, tmem_base + ((quadrant * 32u) << 16) + fz_accumulator_column, group,
                            p.gradient_scale);
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&tail->fz_accumulator_empty));
            ++drained;
        }
        return true;
    };

    uint32_t strip_now = 0xFFFFFFFFu;
    while (cursor.n < items) {
        if constexpr (form_ == form_fused) drain(items_done * p.tile_count, false);
        uint32_t const strip = cursor.strip, run = cursor.run;
        if (strip != strip_now) {
            strip_now = strip;
            row = strip * fwd_rows + row_local;
#pragma unroll
            for (int k = 0; k < prefixes_; ++k) {
                float const inv_q = *(p.q_inv + static_cast<size_t>(k) * p.rows_q + row);
                // inverse norms are not negative, so their bits order as they do
                float const band_max = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(inv_q)));
                rows_max = lane == static_cast<uint32_t>(k) ? band_max : rows_max;
                row_beta[k * factor_stride] = row_factor(beta, inv_q);
            }
        }
        if (cursor.t == 0) {
#pragma unroll
            for (int k = 0; k < prefixes_; ++k) {
                if constexpr (rolled) band_sums[k * fwd_epilogue_threads] = 0.0f, band_sums[(prefixes_ + k) * fwd_epilogue_threads] = 0.0f;
                else loss[k] = 0.0f, coefficient[k] = 0.0f;
            }
            g = 0.0f, own_logit = 0.0f;
        }
        uint32_t const column = cursor.column_tile(p) * fwd_cols_for(form_) + patch_column;
        uint32_t const entry = tile_local % fwd_norm_slots;
        float const* const norms_now = norm_ring + entry * fwd_norm_floats(prefixes_, form_) + patch_column;
        // Does the diagonal cross this warp's patch? It does when the patch's columns come within one of its rows (a row's
        // own copy, or its pair partner next to it); then each row's own and partner cells are scored apart, and the others
        // as everywhere. Decided per warp, so that of a tile on the diagonal only the patches it crosses pay for that.
        uint64_t const first_row = p.query_base + static_cast<uint64_t>(strip) * fwd_rows + patch_row;
        uint64_t const first_column = p.candidate_base + column;
        uint64_t const odd = first_row & 1u; // then the first row's partner lies a row before, the last one's a row behind the patch's
        bool const special = form_ != form_pair_apart &&
                             first_column - first_row + (warp_columns - 1) + odd < 32u + (warp_columns - 1) + 2 * odd;

        timer.lap(0);
        if (!mbar_wait(smem_u32(&tail->tile_full[tile_local % fwd_tile_barriers]), (tile_local / fwd_tile_barriers) & 1u, ctx,
                       site_fwd_tile_full, tile_local))
            return;
        tcgen05_fence_after();
        if (!mbar_wait(smem_u32(&tail->norms_full[entry]), (tile_local / fwd_norm_slots) & 1u, ctx, site_fwd_norms_full, tile_local))
            return;
        timer.lap(1);
        // Bands in which some cosine of the patch may sit on the floor (one bit each).
        uint32_t floors = 0;
        {
            bool const may = lane < prefixes_ &&
                             rows_max * norm_ring[entry * fwd_norm_floats(prefixes_, form_) + prefixes_ * fwd_cols_for(form_) +
                                                  column_half * 8u + lane % 8u] >= 100.0f;
            floors = __ballot_sync(0xFFFFFFFFu, may);
        }

        // The staging patches are rewritten below: the stores of the tile before must have finished reading them.
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
        uint32_t const first_unit = tile_local * prefixes_;
        // Which of this warp's columns, if any, is the row's own copy or its pair partner: bit c for a cell scored apart, bit
        // 16 + c for the partner's.
        uint32_t apart = 0;
        uint32_t const sums = warp_store_base + (rolled ? lane * 16u : lane * 32u + (((lane >> 2) & 1u) ^ 1u) * 16u);
        constexpr uint32_t sums_stride = rolled ? 512u : fwd_store_patch_bytes;
        if (special) {
            uint64_t const global_row = p.query_base + row;
            int64_t const first = static_cast<int64_t>(p.candidate_base + column);
            int64_t const own_at = static_cast<int64_t>(global_row) - first;
            int64_t const partner_at = static_cast<int64_t>(global_row ^ 1ull) - first;
            int own_column = -1, partner_column = -1;
            if (own_at >= 0 && own_at < warp_columns) own_column = static_cast<int>(own_at);
            if ((p.spec_code & 1u) != 0u && partner_at >= 0 && partner_at < warp_columns) partner_column = static_cast<int>(partner_at);
            special_sums const total =
                special_cells<prefixes_, form_>(lane_base, first_unit, norms_now, p.q_inv + row, p.rows_q, beta, bias, own_column,
                                                 partner_column, p.spec_code, sums, sums_stride);
            g += total.cell, own_logit += total.own_logit;
            apart = (own_column >= 0 ? 1u << own_column : 0u) | (partner_column >= 0 ? 0x10001u << partner_column : 0u);
#pragma unroll
            for (int k = 0; k < prefixes_; ++k) {
                float band_loss, band_coefficient;
                asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(band_loss), "=f"(band_coefficient)
                             : "r"(sums + k * sums_stride) : "memory");
                add_sums(k, band_loss, band_coefficient);
            }
        }
        // Stores the patches from `patch` on to bands `band` and up (one band when they go one by one, else all) of the block's
        // gradient cube at the tile's place, or (fused kernel) of this CTA's scratch buffer of the item,
        // [band][128 rows][tiles_per_run * 64 candidates], at the tile's place in the run.
        auto store_patches = [&](int patch, int band) {
            uint32_t const store_x = form_ == form_fused ? cursor.t * fwd_cols_for(form_) + patch_column : column;
            uint32_t const store_y = form_ == form_fused ? patch_row : strip * fwd_rows + patch_row;
            uint32_t const store_z = form_ == form_fused ? (blockIdx.x * 2u + (items_done & 1u)) * prefixes_ : 0u;
            asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                             reinterpret_cast<uint64_t>(cube_map)),
                         "r"(warp_store_base + patch * fwd_store_patch_bytes), "r"(store_x), "r"(store_y), "r"(store_z + band)
                         : "memory");
        };
        // A cell scored apart takes no part: its decay, and with it all that the cell adds, becomes zero.
        auto without_special = [&](pair_t a, int at) {
            a.x = apart & (1u << at) ? left_out_logit : a.x;
            a.y = apart & (2u << at) ? left_out_logit : a.y;
            return a;
        };
#pragma unroll 1
        for (int first = 0; first < warp_columns; first += columns) {
            pair_t prefix[columns / 2], running[columns / 2];
            if constexpr (rolled) {
#pragma unroll
                for (int c = 0; c < columns / 2; ++c) prefix[c] = running[c] = pack2(0.0f, 0.0f);
            }
            pair_t const bias2_binary = pack2(bias * log2_e, bias * log2_e);
            // One band of the chunk: the dots in `dk` become raw-dot gradients.
            auto score_band = [&](int const k, uint32_t (&dk)[columns]) {
                // The candidates' inverse norms (broadcast shared loads). A cell on the cosine floor has cosine and
                // gradient zero, which is what an inverse norm of zero gives it.
                pair_t inv_c[columns / 2];
#pragma unroll
                for (int c = 0; c < columns / 2; c += 2) {
                    float4 const quad = *reinterpret_cast<float4 const*>(norms_now + k * fwd_cols_for(form_) + first + 2 * c);
                    inv_c[c] = pack2(quad.x, quad.y), inv_c[c + 1] = pack2(quad.z, quad.w);
                }
                if ((floors >> k) & 1u) {
                    float const inv_q = *(p.q_inv + static_cast<size_t>(k) * p.rows_q + row);
#pragma unroll
                    for (int c = 0; c < columns / 2; ++c) {
                        inv_c[c].x = inv_q * inv_c[c].x >= 100.0f ? 0.0f : inv_c[c].x;
                        inv_c[c].y = inv_q * inv_c[c].y >= 100.0f ? 0.0f : inv_c[c].y;
                    }
                }
                // First every cell's logit + bias, in base two (the scale and the bias carry log2(e), so that an
                // exponential is a single MUFU), and the largest of the thread's cells. Where the warp's cells are all
                // easy negatives (every logit + bias below the limit, which is all but the hardest cells) the rest is
                // the exponential e and a few packed multiply-adds: log1p(e) = e - e^2/2 + e^3/3 and 1 - sigmoid =
                // e / (1 + e) = e - e^2 + e^3, to float32 rounding below the limit. Up to the second limit two more terms
                // of both series do. Otherwise the general form runs: the decay with the absolute value, reciprocal,
                // select by sign, the full log1p polynomial, the hinge.
                float const row_beta_binary = row_beta[k * factor_stride] * log2_e;
                pair_t const row_beta2_binary = pack2(row_beta_binary, row_beta_binary);
                pair_t logits[columns / 2];
                float largest = -INFINITY;
#pragma unroll
                for (int c = 0; c < columns / 2; ++c) {
                    pair_t const dots = pack2(__uint_as_float(dk[2 * c]), __uint_as_float(dk[2 * c + 1]));
                    prefix[c] = !rolled && k == 0 ? dots : add2(prefix[c], dots);
                    logits[c] = fma2(prefix[c], mul2(inv_c[c], row_beta2_binary), bias2_binary);
                }
                if (special) {
#pragma unroll
                    for (int c = 0; c < columns / 2; ++c) logits[c] = without_special(logits[c], 2 * c);
                }
#pragma unroll
                for (int c = 0; c < columns / 2; ++c) largest = fmaxf(fmaxf(largest, logits[c].x), logits[c].y);
                pair_t complements = pack2(0.0f, 0.0f), coefficient2 = pack2(0.0f, 0.0f);
                float band_loss, band_g;
                if (__all_sync(0xFFFFFFFFu, largest < easy_negative_limit)) {
                    // With u = e^2 - e the complement is c = e + e u, and e^2 and e^3 = c + u are combinations of the two:
                    // the loss's sum is that of e / 2 - u / 6 + c / 3, so three sums serve both.
                    pair_t singles, lower;
#pragma unroll
                    for (int c = 0; c < columns / 2; ++c) {
                        pair_t const e = pack2(fast_ex2(logits[c].x), fast_ex2(logits[c].y));
                        pair_t const u = fma2(e, e, pack2(-e.x, -e.y));
                        pair_t const complement = fma2(e, u, e);
                        singles = c == 0 ? e : add2(singles, e);
                        lower = c == 0 ? u : add2(lower, u);
                        complements = c == 0 ? complement : add2(complements, complement);
                        pair_t const raw = mul2(complement, inv_c[c]);
                        coefficient2 = c == 0 ? mul2(raw, prefix[c]) : fma2(raw, prefix[c], coefficient2);
                        dk[2 * c] = __float_as_uint(raw.x), dk[2 * c + 1] = __float_as_uint(raw.y);
                    }
                    band_g = complements.x + complements.y;
                    band_loss = fmaf(0.5f, singles.x + singles.y, fmaf(-1.0f / 6.0f, lower.x + lower.y, (1.0f / 3.0f) * band_g));
                } else if (__all_sync(0xFFFFFFFFu, largest < near_negative_limit)) {
                    pair_t const minus_one = pack2(-1.0f, -1.0f);
                    pair_t loss2 = pack2(0.0f, 0.0f);
#pragma unroll
                    for (int c = 0; c < columns / 2; ++c) {
                        pair_t const e = pack2(fast_ex2(logits[c].x), fast_ex2(logits[c].y));
                        pair_t s = fma2(e, pack2(-0.2f, -0.2f), pack2(0.25f, 0.25f)); // minus the series of log1p(e) / e
                        pair_t h = add2(e, minus_one);                                // minus that of 1 / (1 + e)
                        h = fma2(e, h, pack2(1.0f, 1.0f)), s = fma2(e, s, pack2(-1.0f / 3.0f, -1.0f / 3.0f));
                        h = fma2(e, h, minus_one), s = fma2(e, s, pack2(0.5f, 0.5f));
                        h = fma2(e, h, pack2(1.0f, 1.0f)), s = fma2(e, s, minus_one);
                        loss2 = fma2(e, s, loss2);
                        pair_t const complement = mul2(e, h);
                        complements = add2(complements, complement);
                        pair_t const raw = mul2(complement, inv_c[c]);
                        coefficient2 = fma2(raw, prefix[c], coefficient2);
                        dk[2 * c] = __float_as_uint(raw.x), dk[2 * c + 1] = __float_as_uint(raw.y);
                    }
                    band_g = complements.x + complements.y;
                    band_loss = -(loss2.x + loss2.y);
                } else {
                    pair_t hinges = pack2(0.0f, 0.0f), loss2 = pack2(0.0f, 0.0f);
                    float const factor = row_beta[k * factor_stride];
                    pair_t const row_beta2 = pack2(factor, factor);
                    // In natural units: a hard cell's gradient is large, and is rounded as the special cells' are. The cells
                    // scored apart are looked for only in patches that have any: for every patch it cost 2 % at four bands,
                    // 3 % at five and 6 % at six. Up to four bands there are registers to look ahead of the loop, which then
                    // has no branch in it (K=4, 4096 rows, H=768: 101.4 -> 98.7 us; in the fused form and with more bands it costs spills).
                    constexpr bool ahead = form_ != form_fused && prefixes_ <= 4;
                    auto natural = [&](int const c) { return fma2(prefix[c], mul2(inv_c[c], row_beta2), pack2(bias, bias)); };
                    if constexpr (ahead) {
#pragma unroll
                        for (int c = 0; c < columns / 2; ++c) logits[c] = natural(c);
                        if (special) {
#pragma unroll
                            for (int c = 0; c < columns / 2; ++c) logits[c] = without_special(logits[c], 2 * c);
                        }
                    }
#pragma unroll
                    for (int c = 0; c < columns / 2; ++c) {
                        pair_t a = ahead ? logits[c] : natural(c);
                        if (!ahead && special) a = without_special(a, 2 * c);
                        pair_t const e = pack2(fast_ex2(-fabsf(a.x) * log2_e), fast_ex2(-fabsf(a.y) * log2_e));
                        pair_t const whole = add2(e, pack2(1.0f, 1.0f));
                        pair_t const complement = mul2(pack2(a.x >= 0.0f ? 1.0f : e.x, a.y >= 0.0f ? 1.0f : e.y),
                                                       pack2(fast_rcp(whole.x), fast_rcp(whole.y)));
                        loss2 = fma2(log1p_ratio2(e), e, loss2);
                        hinges = add2(hinges, pack2(fmaxf(a.x, 0.0f), fmaxf(a.y, 0.0f)));
                        complements = add2(complements, complement);
                        pair_t const raw = mul2(complement, inv_c[c]);
                        coefficient2 = fma2(raw, prefix[c], coefficient2);
                        dk[2 * c] = __float_as_uint(raw.x), dk[2 * c + 1] = __float_as_uint(raw.y);
                    }
                    band_g = complements.x + complements.y;
                    band_loss = (hinges.x + hinges.y) + (loss2.x + loss2.y);
                }
                if (special) {
                    float raw;
                    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(raw) : "r"(sums + k * sums_stride + 8u) : "memory");
#pragma unroll
                    for (int c = 0; c < columns; ++c) dk[c] = apart & (0x10000u << c) ? __float_as_uint(raw) : dk[c];
                }
                add_sums(k, band_loss, coefficient2.x + coefficient2.y);
                g += band_g;
            };
            // Suffix sums, widest band first: band k's gradient cube holds the sum over bands >= k, each with its row
            // factor beta / |q_k|. A warp's patch of a band is [32 rows x 16 columns] bfloat16, 32 bytes per row, under the
            // 32-byte swizzle (the two 16-byte halves of a row change places in every second group of four rows), so that
            // the eight lanes of a store phase cover all banks: unswizzled, every phase had two lanes on each bank.
            auto sum_band = [&](int const k, uint32_t const (&dk)[columns], int const patch) {
                float const factor = row_beta[k * factor_stride];
                pair_t const factor2 = pack2(factor, factor);
                uint32_t packed[columns / 2];
#pragma unroll
                for (int c = 0; c < columns / 2; ++c) {
                    pair_t const raw = pack2(__uint_as_float(dk[2 * c]), __uint_as_float(dk[2 * c + 1]));
                    running[c] = !rolled && k == prefixes_ - 1 ? mul2(raw, factor2) : fma2(raw, factor2, running[c]);
                    packed[c] = pack_bf16x2(running[c].x, running[c].y);
                }
#pragma unroll
                for (int part = 0; part < columns; part += 8) {
                    uint32_t const half = static_cast<uint32_t>(first + part) / 8u;
                    uint32_t const at = warp_store_base + patch * fwd_store_patch_bytes + lane * 32u + (((half & 1u) ^ ((lane >> 2) & 1u)) * 16u);
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(packed[part / 2]),
                                 "r"(packed[part / 2 + 1]), "r"(packed[part / 2 + 2]), "r"(packed[part / 2 + 3]) : "memory");
                }
            };
            auto load_bands = [&](auto& d, int const from, int const to) {
#pragma unroll
                for (int k = from; k < to; ++k) tmem_load<columns>(lane_base + band_slot<prefixes_, form_>(first_unit, k) + first, d[k - from]);
                tmem_load_wait();
            };
            auto release_slots = [&](uint64_t* barriers) { // this warp is done with the tile's slots (or one kind of them)
                if (first + columns != warp_columns) return;
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) give_back(&barriers[tile_local % fwd_slots]);
            };
            if constexpr (rolled) {
#pragma unroll 1
                for (int k = 0; k < prefixes_; ++k) {
                    uint32_t const address = lane_base + band_slot<prefixes_, form_>(first_unit, k);
                    uint32_t d[columns];
                    tmem_load<columns>(address, d);
                    tmem_load_wait();
                    score_band(k, d);
                    tmem_store_16(address, d);
                }
                tmem_store_wait();
                // Two bands at a time, widest first: both loads in flight, both patches behind one proxy fence and in one bulk
                // group; a pair's patches are rewritten two pairs later, once their stores have read them.
#pragma unroll 1
                for (int k = prefixes_ - 1; k >= 0; k -= 2) {
                    int const below = k > 0 ? k - 1 : 0, patch = ((prefixes_ - 1 - k) / 2 % 2) * 2;
                    uint32_t upper[columns], lower[columns];
                    tmem_load<columns>(lane_base + band_slot<prefixes_, form_>(first_unit, k), upper);
                    tmem_load<columns>(lane_base + band_slot<prefixes_, form_>(first_unit, below), lower);
                    tmem_load_wait();
                    if (k == prefixes_ - 1) release_slots(tail->tile_taken);
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    __syncwarp();
                    sum_band(k, upper, patch);
                    if (k > 0) sum_band(below, lower, patch + 1);
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        store_patches(patch, k);
                        if (k > 0) store_patches(patch + 1, below);
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                }
                release_slots(tail->tile_parked_taken);
            } else {
                if constexpr (parked > 0) {
                    uint32_t d[parked][columns];
                    load_bands(d, 0, parked);
#pragma unroll
                    for (int k = 0; k < parked; ++k) {
                        score_band(k, d[k]);
                        tmem_store_8(lane_base + band_slot<prefixes_, form_>(first_unit, k) + first, d[k]);
                    }
                }
                {
                    uint32_t d[prefixes_ - parked][columns];
                    load_bands(d, parked, prefixes_);
                    release_slots(tail->tile_taken);
#pragma unroll
                    for (int k = parked; k < prefixes_; ++k) score_band(k, d[k - parked]);
#pragma unroll
                    for (int k = prefixes_ - 1; k >= parked; --k) sum_band(k, d[k - parked], k);
                }
                if constexpr (parked > 0) {
                    uint32_t d[parked][columns];
                    tmem_store_wait();
                    load_bands(d, 0, parked);
                    release_slots(tail->tile_parked_taken);
#pragma unroll
                    for (int k = parked - 1; k >= 0; --k) sum_band(k, d[k], k);
                }
            }
            apart >>= columns; // the next chunk's cells
        }
        timer.lap(2);
        if constexpr (!rolled) {
            // The tile's patches, all bands of them, leave as one TMA store issued by one lane.
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                store_patches(0, 0);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
        }
        if (lane == 0) mbar_arrive(smem_u32(&tail->norms_empty[entry])); // every lane's reads are behind a __syncwarp above
        timer.lap(3);
        if (cursor.t + 1 == run_length<form_>(p, run)) {
            // One partial record per (run, column group, row); the 1/N weight and the mirror cell's factor two go in here.
            uint32_t const slot = (run * (fwd_cols_for(form_) / 64) + column_half) * fwd_column_groups + group;
            float* record = p.partials + static_cast<size_t>(slot) * quantities * p.rows_q + row;
            if (SC_IN_BOUNDS((static_cast<size_t>(slot) * quantities + quantities - 1) * p.rows_q + row,
                             static_cast<size_t>(p.runs_per_strip) * (fwd_cols_for(form_) / 64) * fwd_column_groups * quantities * p.rows_q)) {
                auto put = [&](uint32_t quantity, float value) { record[static_cast<size_t>(quantity) * p.rows_q] = value; };
                // sum of cell gradient * logit: the coefficients are exactly that, except for a row's own copy, whose logit
                // is the scale itself and which moves no dot product
                float logits = own_logit;
#pragma unroll
                for (int k = 0; k < prefixes_; ++k) {
                    float const band_loss = rolled ? band_sums[k * fwd_epilogue_threads] : loss[rolled ? 0 : k];
                    float const band_coefficient = rolled ? band_sums[(prefixes_ + k) * fwd_epilogue_threads] : coefficient[rolled ? 0 : k];
                    float const whole = row_beta[k * factor_stride] * band_coefficient;
                    logits += whole;
                    put(2 + k, p.weight * band_loss);
                    put(2 + prefixes_ + k, 2.0f * p.weight * whole);
                }
                put(0, p.weight * g);
                put(1, p.weight * logits);
            }
            if constexpr (form_ == form_fused) {
                // The item's patches of this warp are in memory once its bulk stores have completed (not merely been
                // read out of the staging buffers); then the gradient GEMM's producer may load them.
                if (lane == 0) {
                    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
                    fence_proxy_async_all();
                    mbar_arrive(smem_u32(&tail->fz_item_stored[items_done & 1u]));
                }
                __syncwarp();
                ++items_done;
                // The next item writes the other scratch buffer, whose last reader was the GEMM of item items_done - 2.
                if (!drain((items_done - 1) * p.tile_count, true)) return;
            }
        }
        cursor.advance(p);
        ++tile_local;
    }
    timer.flush(p, 5, 4);
    // The staging buffers must outlive the stores that read them.
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    if constexpr (form_ == form_fused) drain(items_done * p.tile_count, true);
}

// ---- fused kernel: the gradient GEMM's two roles ------------------------------------------------------------------
// For every item this CTA has scored (in the same order), for every channel tile, the K loop over the item's candidates:
// A = the band's gradient patch [128 rows x 64 candidates] from this CTA's scratch buffer, B = the transposed candidates
// [width channels x 64 candidates]. Both K-major under the 128-byte swizzle.
__device__ __forceinline__ void fz_producer_role(fz_maps const* maps, fwd_params const& p, uint32_t stages_base,
                                                 fwd_tail* tail, wait_context const& ctx, uint32_t const prefixes) {
    if (!elect_one()) return;
    uint32_t stage = 0, phase = 0, local = 0;
    phase_timer timer(p);
    for (uint32_t count = item_count<form_fused>(p.items); local < count; ++local) {
        uint32_t const item = item_at<form_fused>(local);
        uint32_t const buffer = local & 1u;
        timer.lap(0);
        if (!mbar_wait_relaxed(smem_u32(&tail->fz_item_stored[buffer]), (local >> 1) & 1u, ctx, site_fz_item_stored, item, sleep_gemm_ns))
            return;
        timer.lap(1);
        fence_proxy_async_all();
        uint32_t const first_candidate = (item % p.runs_per_strip) * p.tiles_per_run * fwd_cols_for(form_fused);
        for (uint32_t which = 0; which < p.tile_count; ++which) {
            uint32_t const word = p.tiles[which];
            uint32_t const band = word & 0xFu, channel0 = ((word >> 4) & 0xFFFu) * 16u, width = (word >> 16) * 16u;
            for (uint32_t block = 0; block < p.tiles_per_run; ++block) {
                timer.lap(0);
                if (!mbar_wait_lane(smem_u32(&tail->fz_stage_empty[stage]), phase ^ 1u, ctx, site_fz_stage_empty, which))
                    return;
                timer.lap(2);
                uint32_t const full = smem_u32(&tail->fz_stage_full[stage]);
                uint32_t const destination = stages_base + stage * fz_stage_bytes;
                mbar_arrive_expect_tx(full, fz_a_bytes + width * fz_depth * 2u);
                tma_load_3d(destination, &maps->patches, full, static_cast<int>(block * fz_depth), 0,
                            static_cast<int>((blockIdx.x * 2u + buffer) * prefixes + band));
                // Largest boxes first; 16 channels are 2048 bytes of the stage (rows of 128 bytes under the swizzle).
                uint32_t done = 0;
#pragma unroll
                for (int index = static_cast<int>(fz_candidate_maps) - 1; index >= 0; --index) {
                    uint32_t const box = 16u << index;
                    if (width - done >= box) {
                        tma_load_2d(destination + fz_a_bytes + done * 128u, &maps->candidates[index], full,
                                    static_cast<int>(first_candidate + block * fz_depth), static_cast<int>(channel0 + done));
                        done += box;
                    }
                }
                if (++stage == fz_stages) stage = 0, phase ^= 1u;
            }
        }
    }
    timer.flush(p, 9, 3);
}

__device__ __forceinline__ void fz_mma_role(fwd_params const& p, uint32_t stages_base, fwd_tail* tail, uint32_t tmem_base,
                                            wait_context const& ctx) {
    constexpr uint32_t descriptor_high = (1024u >> 4) | (1u << 14) | (2u << 29); // stride 1024 B, version 1, 128-byte swizzle
    if (!elect_one()) return;
    uint32_t const low_base = ((stages_base & 0x3FFFFu) >> 4) | (1u << 16);
    uint32_t const accumulator = tmem_base + fz_accumulator_column;
    uint32_t stage = 0, phase = 0, unit = 0;
    phase_timer timer(p);
    for (uint32_t n = 0, count = item_count<form_fused>(p.items); n < count; ++n) {
        for (uint32_t which = 0; which < p.tile_count; ++which, ++unit) {
            uint32_t const idesc = umma_idesc_bf16(128, (p.tiles[which] >> 16) * 16u);
            // The accumulator's previous contents must have left tensor memory (an arrival per epilogue warp).
            timer.lap(0);
            if (unit != 0 &&
                !mbar_wait_relaxed(smem_u32(&tail->fz_accumulator_empty), (unit - 1) & 1u, ctx, site_fz_accumulator_empty, unit, sleep_gemm_ns))
                return;
            timer.lap(1);
            tcgen05_fence_after();
            for (uint32_t block = 0; block < p.tiles_per_run; ++block) {
                if (!mbar_wait_lane(smem_u32(&tail->fz_stage_full[stage]), phase, ctx, site_fz_stage_full, unit)) return;
                timer.lap(2);
                tcgen05_fence_after();
                uint32_t const a_low = low_base + stage * (fz_stage_bytes >> 4);
                uint32_t const b_low = a_low + (fz_a_bytes >> 4);
#pragma unroll
                for (uint32_t step = 0; step < fz_depth / 16; ++step) {
                    uint64_t a_descriptor, b_descriptor;
                    asm("mov.b64 %0, {%1, %2};" : "=l"(a_descriptor) : "r"(a_low + step * 2u), "r"(descriptor_high));
                    asm("mov.b64 %0, {%1, %2};" : "=l"(b_descriptor) : "r"(b_low + step * 2u), "r"(descriptor_high));
                    umma_bf16(accumulator, a_descriptor, b_descriptor, idesc, (block | step) != 0u ? 1u : 0u);
                }
                umma_commit(smem_u32(&tail->fz_stage_empty[stage]));
                if (++stage == fz_stages) stage = 0, phase ^= 1u;
            }
            umma_commit(smem_u32(&tail->fz_accumulator_full));
        }
    }
    timer.flush(p, 12, 3);
}

__device__ __forceinline__ void pull_role(pull_request const& request, uint32_t thread_in_role) {
    size_t const thread = static_cast<size_t>(blockIdx.x) * (fwd_pull_warps * 32) + thread_in_role;
    size_t const threads = static_cast<size_t>(gridDim.x) * (fwd_pull_warps * 32);
    for (int part = 0; part < 2; ++part) {
        size_t const vectors = request.bytes[part] / 16;
        if (vectors == 0) continue;
        uint4 const* src = static_cast<uint4 const*>(request.src[part]);
        uint4* dst = static_cast<uint4*>(request.dst[part]);
        size_t index = thread;
        for (; index + 7 * threads < vectors; index += 8 * threads) {
            uint4 held[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) held[u] = src[index + u * threads];
#pragma unroll
            for (int u = 0; u < 8; ++u) dst[index + u * threads] = held[u];
        }
        for (; index < vectors; index += threads) dst[index] = src[index];
    }
}

template <int prefixes_, form_t form_>
__global__ void __launch_bounds__(fwd_threads, 1)
    forward_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap c_map,
                   const __grid_constant__ CUtensorMap cube_map, const __grid_constant__ fz_maps gemm_maps,
                   const fwd_params p) {
    constexpr uint32_t fwd_slots = fwd_slots_for(form_);
    constexpr uint32_t stages = fwd_stages_for(prefixes_, form_);
    extern __shared__ uint8_t raw_shared[];
    uint32_t const raw_address = smem_u32(raw_shared);
    uint32_t const stages_base = (raw_address + 1023u) & ~1023u;
    uint32_t const gemm_stages_base = stages_base + stages * fwd_stage_bytes(form_);
    uint32_t const store_base = stages_base + fwd_stage_region_bytes(prefixes_, form_);
    fwd_tail* tail = reinterpret_cast<fwd_tail*>(raw_shared + (store_base - raw_address) + fwd_store_bytes(prefixes_));
    uint32_t const warp = threadIdx.x / 32, lane = threadIdx.x % 32;

    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < fwd_max_stages; ++i) {
            mbar_init(smem_u32(&tail->stage_full[i]), 1);
            mbar_init(smem_u32(&tail->stage_empty[i]), 1);
        }
        for (uint32_t i = 0; i < fwd_slots; ++i) {
            mbar_init(smem_u32(&tail->tile_taken[i]), fwd_ctas_for(form_) * fwd_epilogue_warps);
            mbar_init(smem_u32(&tail->tile_parked_taken[i]), fwd_ctas_for(form_) * fwd_epilogue_warps);
        }
        for (uint32_t i = 0; i < fwd_tile_barriers; ++i) mbar_init(smem_u32(&tail->tile_full[i]), 1);
        for (uint32_t i = 0; i < fwd_norm_slots; ++i) {
            mbar_init(smem_u32(&tail->norms_full[i]), 1);
            mbar_init(smem_u32(&tail->norms_empty[i]), fwd_epilogue_warps);
        }
        if constexpr (form_ == form_fused) {
            for (uint32_t i = 0; i < fz_stages; ++i) {
                mbar_init(smem_u32(&tail->fz_stage_full[i]), 1);
                mbar_init(smem_u32(&tail->fz_stage_empty[i]), 1);
            }
            mbar_init(smem_u32(&tail->fz_item_stored[0]), fwd_epilogue_warps);
            mbar_init(smem_u32(&tail->fz_item_stored[1]), fwd_epilogue_warps);
            mbar_init(smem_u32(&tail->fz_accumulator_full), 1);
            mbar_init(smem_u32(&tail->fz_accumulator_empty), fwd_epilogue_warps);
        }
        fence_barrier_init();
    }
    if (warp == fwd_mma_warp) {
        if constexpr (fwd_paired(form_)) {
            tmem_alloc_pair(smem_u32(&tail->tmem_base), fwd_tmem_columns);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(smem_u32(&tail->tmem_base), fwd_tmem_columns);
            tmem_relinquish();
        }
    }
    if (warp == fwd_producer_warp && lane == 0) {
        tma_prefetch_descriptor(&q_map);
        tma_prefetch_descriptor(&c_map);
    }
    if constexpr (form_ == form_fused) {
        if (warp == fwd_first_pull_warp && lane == 0) {
            tma_prefetch_descriptor(&gemm_maps.patches);
            for (uint32_t i = 0; i < fz_candidate_maps; ++i) tma_prefetch_descriptor(&gemm_maps.candidates[i]);
        }
    }
    let_dependents_start();
    uint32_t rank = 0;
    if constexpr (fwd_paired(form_)) {
        rank = cluster_rank();
        cluster_sync(); // the other CTA's barriers are set up
    }
    // Everything up to here may run beside the end of the kernel before.
    wait_for_kernels_before();
    // (Both CTAs of a pair read the same: only kernels before this one have written it, or waits of this one that ran out, long after
    // its CTAs have started; should they ever disagree, the other's waits run out too.)
    if (threadIdx.x == 0) tail->abort_flag = status_poisoned(p.status) ? 1u : 0u;
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    uint32_t const tmem_base = tail->tmem_base;
    wait_context const ctx{p.status, p.budget_ns, &tail->abort_flag};

    float* const norm_ring = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(tail) + fwd_tail_bytes);
    bool const poisoned = tail->abort_flag != 0u; // by an earlier kernel: nothing is scored
    if (poisoned) {
    } else if (warp < fwd_epilogue_warps) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(fwd_epilogue_registers));
        epilogue_role<prefixes_, form_>(&cube_map, p, tail, store_base, norm_ring, norm_ring + fwd_norm_bytes(prefixes_, form_) / 4,
                                        tmem_base, ctx, warp, lane, rank);
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(fwd_helper_registers));
        if (warp == fwd_producer_warp) {
            producer_role<prefixes_, form_>(&q_map, &c_map, p, stages_base, norm_ring, tail, ctx, rank);
        } else if (warp == fwd_mma_warp) {
            if (rank == 0) mma_role<prefixes_, form_>(p, stages_base, tail, tmem_base, ctx);
        } else if (warp == fwd_first_pull_warp) {
            // The pull is a short copy at the start of the launch; the gradient GEMM's first item is not ready before the
            // epilogue warps have scored a whole item, so the same warp serves both.
            pull_role(p.pull, threadIdx.x - fwd_first_pull_warp * 32);
            if constexpr (form_ == form_fused) fz_producer_role(&gemm_maps, p, gemm_stages_base, tail, ctx, prefixes_);
        } else if (warp == fz_mma_warp) {
            if constexpr (form_ == form_fused) fz_mma_role(p, gemm_stages_base, tail, tmem_base, ctx);
        }
    }

    tcgen05_fence_before();
    __syncthreads();
    if (!poisoned && tail->abort_flag != 0u) {
        // Something gave up. Give copies and UMMAs that are still in flight a bounded time to land before the tensor
        // memory goes back.
        uint64_t const start = global_timer_ns();
        while (global_timer_ns() - start < 200000ull) __nanosleep(1000);
    }
    // A pair's barriers and operands are used by both CTAs until both are done.
    if constexpr (fwd_paired(form_)) cluster_sync();
    else __syncthreads();
    if (warp == fwd_mma_warp) {
        tcgen05_fence_after();
        if constexpr (fwd_paired(form_)) tmem_dealloc_pair(tmem_base, fwd_tmem_columns);
        else tmem_dealloc(tmem_base, fwd_tmem_columns);
    }
}

// ---- host side --------------------------------------------------------------------------------------------------
template <int prefixes_, form_t form_>
void launch_instance(CUtensorMap const& q_map, CUtensorMap const& c_map, CUtensorMap const& cube_map, fz_maps const& gemm_maps,
                     fwd_params const& p, int blocks, cudaStream_t stream, bool overlap) {
    // The attribute is per device; a process drives one GPU, but a second one costs only the repeat of a cheap call.
    static int prepared_device = -1, resident = 0;
    int device = 0;
    cudaGetDevice(&device);
    if (prepared_device != device) {
        require(cudaFuncSetAttribute(forward_kernel<prefixes_, form_>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     fwd_shared_bytes(prefixes_, form_)),
                "raising the forward kernel's shared memory");
        resident = 1 << 30;
        if constexpr (fwd_paired(form_)) {
            // How many pairs the device holds at a time: the walk over the items assumes that all of them run.
            cudaLaunchAttribute attribute{};
            attribute.id = cudaLaunchAttributeClusterDimension;
            attribute.val.clusterDim.x = 2, attribute.val.clusterDim.y = 1, attribute.val.clusterDim.z = 1;
            cudaLaunchConfig_t config{};
            config.gridDim = 2, config.blockDim = fwd_threads, config.dynamicSmemBytes = fwd_shared_bytes(prefixes_, form_);
            config.attrs = &attribute, config.numAttrs = 1;
            require(cudaOccupancyMaxActiveClusters(&resident, forward_kernel<prefixes_, form_>, &config), "asking for the resident pairs");
            if (resident < 1) throw std::runtime_error("forward: the device holds no pair of CTAs");
            resident *= 2;
        }
        prepared_device = device;
    }
    launch_dependent_clusters(overlap, fwd_ctas_for(form_), forward_kernel<prefixes_, form_>, blocks < resident ? blocks : resident, fwd_threads,
                              fwd_shared_bytes(prefixes_, form_), stream, q_map, c_map, cube_map, gemm_maps, p);
}

template <form_t form_>
void launch_for_count(uint32_t count, CUtensorMap const& q_map, CUtensorMap const& c_map, CUtensorMap const& cube_map,
                      fz_maps const& gemm_maps, fwd_params const& p, int blocks, cudaStream_t stream, bool overlap) {
    switch (count) {
    case 1: launch_instance<1, form_>(q_map, c_map, cube_map, gemm_maps, p, blocks, stream, overlap); break;
    case 2: launch_instance<2, form_>(q_map, c_map, cube_map, gemm_maps, p, blocks, stream, overlap); break;
    case 3: launch_instance<3, form_>(q_map, c_map, cube_map, gemm_maps, p, blocks, stream, overlap); break;
    case 4: launch_instance<4, form_>(q_map, c_map, cube_map, gemm_maps, p, blocks, stream, overlap); break;
    case 5: launch_instance<5, form_>(q_map, c_map, cube_map, gemm_maps, p, blocks, stream, overlap); break;
    case 6: launch_instance<6, form_>(q_map, c_map, cube_map, gemm_maps, p, blocks, stream, overlap); break;
    default:
        if constexpr (form_ != form_fused) {
            if (count == 7) launch_instance<7, form_>(q_map, c_map, cube_map, gemm_maps, p, blocks, stream, overlap);
            else launch_instance<8, form_>(q_map, c_map, cube_map, gemm_maps, p, blocks, stream, overlap);
        }
        break;
    }
}

template <int prefixes_> void preload_count(bool fused) {
    cudaFuncAttributes attributes;
    if (!fused) {
        require(cudaFuncGetAttributes(&attributes, forward_kernel<prefixes_, form_single>), "preload forward (single)");
        require(cudaFuncGetAttributes(&attributes, forward_kernel<prefixes_, form_pair>), "preload forward (pair)");
        require(cudaFuncGetAttributes(&attributes, forward_kernel<prefixes_, form_pair_apart>), "preload forward (pair, apart)");
    } else if constexpr (prefixes_ <= static_cast<int>(fz_max_prefixes)) {
        require(cudaFuncGetAttributes(&attributes, forward_kernel<prefixes_, form_fused>), "preload forward (fused)");
    }
}

} // namespace

// Which form a launch takes; by sizes and numbers alone, so that a block takes the same one however much of the GPU it gets.
// - Every tile of 64 at once on the GPU, or an odd number of them (a pair's tile is two): a single CTA each. A pair's barriers and
//   commits across CTAs cost a launch 0.7 us (128 rows, H=768, K=5: 11.6 against 12.4 us; 1024 rows 12.2 against 13.0).
// - A block without the rows' own copies: the pair's form that has nothing of the diagonal in it (one block of 4096 rows, H=768, K=5: 74.7
//   us against 80.7 with a single CTA and 82.3 with a pair that can score the diagonal; 2944 rows, H=832, K=4: 44.8, 49.3, 50.8;
//   16384 rows, H=768, K=5: 1130, 1248, 1215; every cell in the general form, 8192 rows, H=512, K=4: 328, 359, 371).
// - A block with them: a pair loads a third fewer operand bytes per cell but carries the diagonal's code beside two CTAs' hand-overs, and
//   spills a little more (4 to 36 bytes from K = 4 on; alone 12 at K = 4). Measured for 256 to 2048 channels, one to eight bands, 2048 to 16384 rows,
//   in turn, single CTA against pair in us:
//   1536 channels and more, a pair everywhere (1 to 19 %): K=5 4096 rows 110.4 against 104.0, K=6 16384 rows 2363 against 2209.
//   Seven and eight bands, from 512 channels on: H=512, K=7 4096 rows 134.3 against 132.1, K=8 16384 rows 2307 against 2075; at
//   H=256, K=8 a pair takes 1 % more. Six bands, from 768 channels on: H=768 4096 rows 101.8 against 99.8, H=1024 125.0 against 114.2.
//   Fewer bands, where the operands weigh more than the cells: H=768, K=2 4096 rows 45.5 against 43.8, H=1024, K=1 45.1 against 43.4; not at
//   256 channels a band and less: H=768, K=3 54.7 against 56.4, H=1024, K=4 2048 rows 23.5 against 24.2, 4096 rows 74.0 against 74.4,
//   H=512, K=4 63.5 against 67.8. Large launches, which run at the GPU's power limit, gain from 768 channels on: 16384 rows, H=768, K=3
//   979 against 900, K=5 1332 against 1320, H=1024, K=5 1488 against 1394, but H=512, K=3 772 against 813.
static form_t forward_form(forward_arguments const& a) {
    if (a.fused) return form_fused;
    uint32_t const column_tiles = a.rows_c / 64, bands = a.ladder.count;
    uint64_t const singles = static_cast<uint64_t>(a.rows_q / fwd_rows) * column_tiles;
    if (column_tiles % 2 || singles <= static_cast<uint64_t>(a.device_multiprocessors)) return form_single;
    // A row's own copy is the candidate of the same number, its partner the other of the pair 2m, 2m + 1.
    uint64_t const first = a.query_base & ~1ull, behind = (a.query_base + a.rows_q + 1) & ~1ull;
    bool const apart = a.candidate_base >= behind || a.candidate_base + a.rows_c <= first;
    if (apart) return form_pair_apart;
    bool const large = static_cast<uint64_t>(a.rows_q) * a.rows_c >= (1ull << 26);
    bool const pair = a.hidden >= 1536 || (bands >= 7 && a.hidden >= 512) || (bands == 6 && a.hidden >= 768) || a.hidden >= 320 * bands ||
                      (large && a.hidden >= 768 && a.hidden >= 144 * bands);
    return pair ? form_pair : form_single;
}
// A run is `tiles_per_run` tiles, of 64 candidates or, in a pair, of 128, and has one record per 64 columns of a tile and column group. A
// pair's last run may be shorter.
static uint32_t runs_of(form_t form, uint32_t rows_c, uint32_t tiles_per_run) {
    return (rows_c / fwd_cols_for(form) + tiles_per_run - 1) / tiles_per_run;
}
static uint32_t slots_of(form_t form, uint32_t rows_c, uint32_t tiles_per_run) {
    return fwd_column_groups * (fwd_cols_for(form) / 64) * runs_of(form, rows_c, tiles_per_run);
}
uint32_t forward_partial_slots(uint32_t rows_c, uint32_t tiles_per_run) {
    uint32_t const single = slots_of(form_single, rows_c, tiles_per_run), pair = slots_of(form_pair, rows_c, tiles_per_run);
    return single > pair ? single : pair;
}
uint32_t forward_filled_slots(forward_arguments const& a) { return slots_of(forward_form(a), a.rows_c, a.tiles_per_run); }
uint32_t forward_quantities(uint32_t prefixes) { return 2 + 2 * prefixes; }

// The run length (a power of two that divides the tiles of 64) after which the busiest pair is done first: its tiles, and an eighth of a
// tile for every run's record, which the epilogue writes and the backward launch folds. With at least six runs to a walker
// instead (2944 and 3072 rows: runs of one tile, 184 and 192 records to a row) the fold took longer than the gradient GEMM that
// hides it: three blocks of 2944 rows, H=832, K=4, took 274 us, with runs of two tiles 237.
uint32_t forward_choose_tiles_per_run(uint32_t rows_q, uint32_t rows_c, int multiprocessors) {
    uint64_t const strips = rows_q / fwd_rows, column_tiles = rows_c / 64, tiles = (column_tiles + 1) / 2; // of 128
    uint64_t const walkers = multiprocessors > 1 ? static_cast<uint64_t>(multiprocessors) / 2 : 1;
    uint32_t best = 1;
    uint64_t least = ~0ull;
    for (uint32_t t = 1; t <= 32 && column_tiles % t == 0 && (t == 1 || t <= tiles); t *= 2) {
        uint64_t const runs = (strips * ((tiles + t - 1) / t) + walkers - 1) / walkers; // of the busiest pair
        if (runs * (8 * t + 1) < least) least = runs * (8 * t + 1), best = t;
    }
    return best;
}

bool forward_fused_supported(uint32_t hidden, uint32_t prefixes) { return prefixes <= fz_max_prefixes && hidden <= 4096; }

// A fused item is a run of tiles whose gradient patches one GEMM pass folds, adding a [128, hidden] float32 tile to the
// gradient once per item: runs of at least four tiles keep those additions rare, longer runs are taken while enough
// items remain to balance the GPU.
uint32_t forward_choose_tiles_per_run_fused(uint32_t rows_q, uint32_t rows_c, int multiprocessors) {
    uint32_t const strips = rows_q / fwd_rows, column_tiles = rows_c / fwd_cols_for(form_fused);
    uint32_t best = 1;
    for (uint32_t t = 1; t <= fz_max_tiles_per_run && column_tiles % t == 0; t *= 2)
        if (t <= 4 || static_cast<uint64_t>(strips) * (column_tiles / t) >= 6ull * static_cast<uint64_t>(multiprocessors)) best = t;
    return best;
}

// Two buffers per CTA of [prefixes][128 rows][tiles_per_run * 64 candidates] bfloat16.
size_t forward_fused_scratch_bytes(uint32_t prefixes, uint32_t tiles_per_run, int multiprocessors) {
    return static_cast<size_t>(multiprocessors) * 2 * prefixes * fwd_rows * tiles_per_run * fwd_cols_for(form_fused) * 2;
}

void launch_forward(forward_arguments const& a, cudaStream_t stream) {
    if (a.rows_q % fwd_rows || a.rows_c % 64 || a.hidden % fwd_depth || a.hidden > 4096)
        throw std::runtime_error("forward: rows must be multiples of 128 (queries) and 64 (candidates), hidden of 64 up to 4096");
    if (a.ladder.count < 1 || a.ladder.count > 8 || a.ladder.ends[a.ladder.count - 1] != a.hidden)
        throw std::runtime_error("forward: the ladder's widest prefix must equal hidden");
    for (uint32_t band = 0, begin = 0; band < a.ladder.count; begin = a.ladder.ends[band++])
        if (a.ladder.ends[band] % 16 || a.ladder.ends[band] <= begin)
            throw std::runtime_error("forward: band edges must ascend in multiples of 16");
    uint32_t const column_tiles = a.rows_c / 64;
    if (a.tiles_per_run == 0 || column_tiles % a.tiles_per_run)
        throw std::runtime_error("forward: tiles_per_run must divide the number of candidate tiles");
    if (a.pull.bytes[0] % 16 || a.pull.bytes[1] % 16) throw std::runtime_error("forward: pull sizes must be multiples of 16");
    if (a.multiprocessors < 1 || a.multiprocessors > a.device_multiprocessors)
        throw std::runtime_error("forward: the multiprocessor count must be positive and the device's at most");

    fwd_params p{};
    p.q_inv = a.query_inverse_norms, p.c_inv = a.candidate_inverse_norms, p.c_tile_max = a.candidate_tile_max;
    p.cube = static_cast<__nv_bfloat16*>(a.gradient_cube_bf16);
    p.partials = a.partials, p.status = a.status;
    p.rows_q = a.rows_q, p.rows_c = a.rows_c, p.hidden = a.hidden;
    p.ladder.count = a.ladder.count;
    for (int i = 0; i < 8; ++i) p.ladder.ends[i] = a.ladder.ends[i];
    form_t const form = forward_form(a);
    p.tiles_per_run = a.tiles_per_run;
    p.tiles_per_strip = a.rows_c / fwd_cols_for(form);
    p.runs_per_strip = runs_of(form, a.rows_c, a.tiles_per_run);
    p.items = (a.rows_q / fwd_rows) * p.runs_per_strip;
    p.beta = a.beta, p.bias = a.bias, p.weight = a.weight;
    p.scalars = a.scalars;
    p.query_base = a.query_base, p.candidate_base = a.candidate_base, p.spec_code = a.spec_code;
    p.budget_ns = a.budget_ns;
    p.pull = a.pull;
    p.trace = a.trace;
    for (uint32_t chunk = 0; chunk < a.hidden / fwd_depth; ++chunk) {
        uint32_t word = 0;
        for (uint32_t sub = 0; sub < 4; ++sub) {
            uint32_t const above = (chunk * 4 + sub + 1) * 16; // first channel above this step
            bool starts = above == a.hidden;
            for (uint32_t band = 0; band + 1 < a.ladder.count; ++band) starts |= a.ladder.ends[band] == above;
            word |= (starts ? 1u : 0u) << (8 * sub);
        }
        p.band_starts[chunk] = word;
    }
    int const ctas = static_cast<int>(fwd_ctas_for(form)), walkers = a.multiprocessors / ctas;
    int blocks = static_cast<int>(p.items < static_cast<uint32_t>(walkers) ? p.items : walkers);
    if ((a.pull.bytes[0] | a.pull.bytes[1]) != 0 && blocks < walkers / 2) blocks = walkers / 2;
    blocks = (blocks < 1 ? 1 : blocks) * ctas;

    if (a.fused) {
        if (!forward_fused_supported(a.hidden, a.ladder.count))
            throw std::runtime_error("forward: the fused kernel takes ladders of at most six prefixes");
        if (a.tiles_per_run > fz_max_tiles_per_run) throw std::runtime_error("forward: a fused run holds at most 16 tiles");
        if (a.fused_scratch_bytes < forward_fused_scratch_bytes(a.ladder.count, a.tiles_per_run, blocks))
            throw std::runtime_error("forward: the fused kernel's scratch is too small");
        if (a.fused_scratch_bf16 == nullptr || a.transposed_candidates == nullptr || a.query_gradient == nullptr)
            throw std::runtime_error("forward: the fused kernel needs its scratch, the transposed candidates and the gradient");
    }
    // Everything above is checked before the first driver or runtime call.
    CUtensorMap const q_map = cached_operand_map(a.queries_bf16, a.hidden, a.rows_q, fwd_depth, fwd_own_rows(form));
    CUtensorMap const c_map = cached_operand_map(a.candidates_bf16, a.hidden, a.rows_c, fwd_depth, fwd_own_cols(form));
    fz_maps gemm_maps{};
    if (!a.fused) {
        // The warps' patches of the gradient cube [K, rows_q, rows_c]: boxes of all bands x 32 rows x 16 candidates, staged under the
        // 32-byte swizzle.
        cuuint64_t const dims[3] = {a.rows_c, a.rows_q, a.ladder.count};
        cuuint64_t const strides[2] = {static_cast<cuuint64_t>(a.rows_c) * 2, static_cast<cuuint64_t>(a.rows_c) * a.rows_q * 2};
        cuuint32_t const box[3] = {fwd_warp_columns, 32, fwd_rolled_for(static_cast<int>(a.ladder.count)) ? 1u : a.ladder.count};
        CUtensorMap const cube_map =
            cached_map(a.gradient_cube_bf16, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_NONE);
        switch (form) {
        case form_single:
            launch_for_count<form_single>(a.ladder.count, q_map, c_map, cube_map, gemm_maps, p, blocks, stream, !a.ordinary_launch);
            break;
        case form_pair:
            launch_for_count<form_pair>(a.ladder.count, q_map, c_map, cube_map, gemm_maps, p, blocks, stream, !a.ordinary_launch);
            break;
        default:
            launch_for_count<form_pair_apart>(a.ladder.count, q_map, c_map, cube_map, gemm_maps, p, blocks, stream, !a.ordinary_launch);
            break;
        }
    } else {
        p.gradient = a.query_gradient, p.gradient_scale = a.gradient_scale;
        for (uint32_t band = 0, begin = 0; band < a.ladder.count; begin = a.ladder.ends[band++])
            for (uint32_t channel = begin; channel < a.ladder.ends[band]; channel += fz_max_width) {
                if (p.tile_count == fz_max_tiles) throw std::runtime_error("forward: too many channel tiles for the fused kernel");
                uint32_t const left = a.ladder.ends[band] - channel;
                p.tiles[p.tile_count++] = band | ((channel / 16) << 4) | (((left < fz_max_width ? left : fz_max_width) / 16) << 16);
            }
        // Scratch of gradient patches: [CTA and buffer][band][128 rows][run of candidates], written in the warps' boxes
        // (under the 32-byte swizzle), read back as the GEMM's A operand (128 rows x 64 candidates, swizzled).
        uint64_t const run = static_cast<uint64_t>(a.tiles_per_run) * fwd_cols_for(form_fused);
        cuuint64_t const dims[3] = {run, fwd_rows, static_cast<cuuint64_t>(blocks) * 2 * a.ladder.count};
        cuuint64_t const strides[2] = {run * 2, run * fwd_rows * 2};
        cuuint32_t const store_box[3] = {fwd_warp_columns, 32, a.ladder.count};
        cuuint32_t const load_box[3] = {fz_depth, fwd_rows, 1};
        CUtensorMap const store_map =
            cached_map(a.fused_scratch_bf16, 3, dims, strides, store_box, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_NONE);
        gemm_maps.patches =
            cached_map(a.fused_scratch_bf16, 3, dims, strides, load_box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
        for (uint32_t index = 0; index < fz_candidate_maps; ++index) {
            // A box may not be taller than the tensor; such a box is never asked for either (tiles are at most `hidden` wide).
            uint32_t const channels = 16u << index;
            gemm_maps.candidates[index] =
                cached_operand_map(a.transposed_candidates, a.rows_c, a.hidden, fz_depth, channels <= a.hidden ? channels : 16u);
        }
        launch_for_count<form_fused>(a.ladder.count, q_map, c_map, store_map, gemm_maps, p, blocks, stream, !a.ordinary_launch);
    }
    cudaError_t const error = cudaGetLastError();
    if (error != cudaSuccess) throw std::runtime_error(std::string("forward launch failed: ") + cudaGetErrorString(error));
    note_launch();
}

SC_DEFINE_BOUNDS_READER(bounds_record_forward)

void preload_forward_kernels(uint32_t prefixes, bool fused) {
    switch (prefixes) {
    case 1: preload_count<1>(fused); break;
    case 2: preload_count<2>(fused); break;
    case 3: preload_count<3>(fused); break;
    case 4: preload_count<4>(fused); break;
    case 5: preload_count<5>(fused); break;
    case 6: preload_count<6>(fused); break;
    case 7: preload_count<7>(fused); break;
    case 8: preload_count<8>(fused); break;
    default: throw std::runtime_error("preload: a ladder holds one to eight prefixes");
    }
}

} // namespace sc
