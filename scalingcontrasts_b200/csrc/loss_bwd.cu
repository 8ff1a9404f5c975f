// Backward tile kernel of the streamed loss: folds a block's per-band gradient cubes into the owner's rows,
//   query_gradient[i, h] += sum_j G_band(h)[i, j] * candidate[j, h],
// as tcgen05 GEMM tiles of 128 rows x up to 256 channels, the candidate index as the K dimension in stages of 64.
// A channel tile never crosses a band edge (edges are multiples of 16 channels and a tile is a multiple of 16 wide),
// so its A operand is a single band's cube, read through a three-dimensional TMA map. The candidates are the B operand
// in one of two layouts: as they are, [R, H] row-major, read in boxes of 64 channels x 64 candidates and handed to the
// tensor cores as an MN-major operand (the channels, the GEMM's N, are the contiguous dimension), which needs no copy of
// the block; or transposed, [H, R], K-major, for callers that hold them that way.
//
// A CTA owns one or two 128-row blocks of a strip and up to 512 tensor-memory columns of accumulators: two blocks x up to
// 256 channels (both blocks use the same candidate stage, which halves the candidate refills from L2), or, for a band of
// 257 to 384 channels, one block x the whole band, so that the band's cube, the traffic this kernel is bound by, is read
// from DRAM once instead of once per 256-channel tile.
//
// Where it pays, two CTAs with consecutive row blocks of a tile, a cluster, run their UMMAs together (256 rows) and load half of the
// tile's candidates each.
//
// Warp roles (192 threads): warps 0-3 epilogue (tensor-memory lanes 32*w..; before that the fold of the forward launch's
// partial records, if asked for), warp 4 TMA producer, warp 5 UMMA issuer and tensor-memory owner. The producer's
// and the issuer's loops are run by one elected lane each. The epilogue adds its scaled accumulators with
// vector reductions (fire and forget: no read of the old value comes back to the SM). With `split == 1` each output
// element receives exactly one addition per launch, so the sum's order is the launches' stream order and the result
// is deterministic; with a larger split the candidate range is divided and the order of a launch's partial sums is not.
//
// Parity: backward_tile_cuda_ (scalingcontrasts.cuh:1042-1136).
#include <array>
#include <stdexcept>
#include <string>
#include <vector>

#include "api.h"
#include "common.cuh"
#include "driver.h"
#include "launch.h"

namespace sc {

namespace {

constexpr uint32_t bwd_rows = 128;
constexpr uint32_t bwd_depth = 64;        // candidates per stage
constexpr uint32_t bwd_max_width = 256;   // channels per UMMA and per tile of a two-block CTA
constexpr uint32_t bwd_wide_width = 384;  // channels of a one-block CTA that takes a whole band
constexpr uint32_t bwd_stages = 6;                                  // at most
constexpr uint32_t bwd_a_bytes = bwd_rows * bwd_depth * 2;        // one 128-row block of the cube
constexpr uint32_t bwd_b_bytes = bwd_max_width * bwd_depth * 2;
constexpr uint32_t bwd_stage_bytes = 2 * bwd_a_bytes + bwd_b_bytes; // two row blocks share one candidate tile
static_assert(bwd_a_bytes + bwd_wide_width * bwd_depth * 2 <= bwd_stage_bytes, "a wide one-block stage must fit a stage");
constexpr uint32_t bwd_tmem_columns = 512;
constexpr uint32_t bwd_block_columns = 256;                         // tensor-memory columns between the two accumulators
constexpr uint32_t bwd_threads = 192;
constexpr uint32_t bwd_max_tiles = 32;

struct bwd_tail {
    uint64_t stage_full[bwd_stages];
    uint64_t stage_empty[bwd_stages];
    uint64_t accumulated;
    uint32_t tmem_base;
    uint32_t abort_flag;
};
// The ring of stages: 208 KB; a stage is the CTA's row blocks of the cube plus the candidates of the tile's own width.
constexpr uint32_t bwd_ring_bytes = 208 * 1024;
// Shared launches (two CTAs on a multiprocessor, see plan_tiles) have half the ring and half the tensor memory.
constexpr uint32_t bwd_shared_width = 128;
constexpr uint32_t bwd_half_ring_bytes = 104 * 1024;
constexpr uint32_t bwd_shared_bytes_for(uint32_t ring) { return 1024 + ring + sizeof(bwd_tail); }
constexpr uint32_t bwd_shared_bytes = bwd_shared_bytes_for(bwd_ring_bytes);
static_assert(2 * (bwd_shared_bytes_for(bwd_half_ring_bytes) + 1024) <= 228 * 1024, "two CTAs of a shared launch must fit one multiprocessor");
static_assert(3 * (bwd_a_bytes + bwd_shared_width * bwd_depth * 2) <= bwd_half_ring_bytes, "three stages of a shared launch's widest tile must fit");
static_assert(3 * bwd_stage_bytes <= bwd_ring_bytes, "three of the largest stages must fit the ring");
static_assert(bwd_shared_bytes <= 227 * 1024, "the kernel's shared memory must fit one CTA's maximum");
constexpr uint32_t bwd_candidate_maps = 5;                          // boxes of 16, 32, 64, 128 and 256 channels

struct bwd_tile {
    uint32_t band, channel0, width;
    uint32_t blocks;    // row blocks per CTA of this tile: 1 or 2
    uint32_t first_cta; // first CTA of the tile's group; a group's CTAs walk its tiles fastest, then the row blocks
    uint32_t group;     // tiles in the group: the tiles of one band (they read the same rows of the cube)
};

// The transposed candidates under five tensor maps that differ only in the box's channel count (16 << index): a tile's
// channels are fetched greedily with the largest boxes that fit, so a stage takes one to three candidate loads.
struct bwd_candidate_boxes {
    CUtensorMap maps[bwd_candidate_maps];
};


struct bwd_params {
    float* query_gradient;
    uint32_t* status;
    uint32_t rows_q, rows_c, hidden;
    uint32_t tile_count, split;
    uint32_t ring_bytes, tmem_columns; // of one CTA
    float scale; // applied to every product before it is added: the loss's 2/N (mirror cell and weight)
    uint64_t budget_ns;
    float const* partials; // optional: the block's partial records and the sums they are folded into
    float* row_accumulators;
    uint32_t partial_slots, quantities;
    bwd_tile tiles[bwd_max_tiles];
};

// Shared-memory descriptor words of the B operand. K-major (transposed candidates): rows of 64 candidates, eight rows
// per 1024-byte swizzle atom, atoms 1024 bytes apart along N; a step of 16 candidates adds 32 bytes. MN-major (row-major
// candidates): a box is 64 candidates (K) x 64 channels (N, contiguous, one 128-byte row per candidate); eight
// candidates make one atom, atoms follow each other every 1024 bytes along K (the stride offset), boxes of 64 channels
// every 8192 bytes along N (the leading offset); a step of 16 candidates is two atoms, 2048 bytes.
constexpr uint32_t bwd_mn_box_bytes = 64 * bwd_depth * 2;

// The fold of the forward launch's partial records into the row accumulators, by the epilogue warps before their accumulators
// are ready. A warp takes sixteen rows of one quantity: a lane four rows (one 16-byte load per record) of every eighth record,
// eight of them in flight. The eight lanes' sums are then added in order, which gives bit for bit what the fold's own kernel
// gives. Bound by the latency of its loads, which the GEMM beside it hides: as a launch of its own between the two tile kernels
// the fold took 4.7 us a block of 4096 rows (72 blocks 11.52 -> 11.19 ms) and 9 us one of 2944 (three blocks 337 -> 310 us).
// With 128 rows of a quantity to a warp and all its records in eight chains of one lane, the latter took 329 us.
__device__ __forceinline__ void fold_share(bwd_params const& p, uint32_t warp, uint32_t lane) {
    constexpr uint32_t chains = 8, rows = 16;
    uint32_t const groups = p.rows_q / rows, units = groups * p.quantities;
    size_t const stride = static_cast<size_t>(p.quantities) * p.rows_q;
    for (uint32_t unit = blockIdx.x + warp * gridDim.x; unit < units; unit += 4 * gridDim.x) {
        size_t const at = static_cast<size_t>(unit / groups) * p.rows_q + unit % groups * rows + lane % 4 * 4;
        float4 total = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
        for (uint32_t slot = lane / 4; slot < p.partial_slots; slot += chains)
            if (SC_IN_BOUNDS(slot * stride + at + 3, p.partial_slots * stride)) {
                float4 const record = *reinterpret_cast<float4 const*>(p.partials + slot * stride + at);
                total.x += record.x, total.y += record.y, total.z += record.z, total.w += record.w;
            }
        __syncwarp();
        float4 const own = total;
#pragma unroll
        for (uint32_t c = 1; c < chains; ++c) {
            uint32_t const from = c * 4 + lane % 4;
            total.x += __shfl_sync(0xFFFFFFFFu, own.x, from), total.y += __shfl_sync(0xFFFFFFFFu, own.y, from);
            total.z += __shfl_sync(0xFFFFFFFFu, own.z, from), total.w += __shfl_sync(0xFFFFFFFFu, own.w, from);
        }
        if (lane < 4 && SC_IN_BOUNDS(at + 3, stride)) { // these lanes began with the first sums
            float4* const into = reinterpret_cast<float4*>(p.row_accumulators + at);
            float4 const before = *into;
            *into = make_float4(before.x + total.x, before.y + total.y, before.z + total.z, before.w + total.w);
        }
    }
}

template <bool mn_major_, bool pair_>
__global__ void __launch_bounds__(bwd_threads, 1)
    backward_kernel(const __grid_constant__ CUtensorMap cube_map, const __grid_constant__ bwd_candidate_boxes candidates,
                    const bwd_params p) {
    extern __shared__ uint8_t raw_shared[];
    uint32_t const raw_address = smem_u32(raw_shared);
    uint32_t const stages_base = (raw_address + 1023u) & ~1023u;
    bwd_tail* tail = reinterpret_cast<bwd_tail*>(raw_shared + (stages_base - raw_address) + p.ring_bytes);
    uint32_t const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    uint32_t tile_index = 0; // the first tile of the group this CTA falls into, then the CTA's own tile within it
    while (tile_index + p.tiles[tile_index].group < p.tile_count &&
           blockIdx.x >= p.tiles[tile_index + p.tiles[tile_index].group].first_cta)
        tile_index += p.tiles[tile_index].group;
    uint32_t const group = p.tiles[tile_index].group, rank = pair_ ? cluster_rank() : 0u;
    uint32_t within = blockIdx.x - p.tiles[tile_index].first_cta;
    // A pair takes one tile of the group for the rows of two CTAs, one after the other.
    if constexpr (pair_) within = (within / 2 / group * 2 + rank) * group + within / 2 % group;
    tile_index += within % group;
    bwd_tile const tile = p.tiles[tile_index];
    // Stage geometry: [row blocks of the cube, 16 KB each][candidate tile of the tile's width]. MN-major candidates come in
    // whole boxes of 64 channels (8 KB), K-major ones in rows of 128 bytes per channel; either way a stage is a multiple of
    // 1 KB, so every stage starts on a swizzle atom.
    bool const wide = tile.width > bwd_max_width;
    // A pair's UMMAs take N in steps of 32 channels (what the last one has beyond the tile is never read), half of them from
    // either CTA.
    uint32_t const pair_width = (tile.width + 31u) / 32u * 32u;
    uint32_t const boxes = ((pair_ ? pair_width / 2 : tile.width) + 63u) / 64u; // MN-major: whole boxes of 64 channels, the last one partly used
    uint32_t const candidate_bytes = mn_major_ ? boxes * bwd_mn_box_bytes : tile.width * bwd_depth * 2u;
    uint32_t const stage_bytes = tile.blocks * bwd_a_bytes + candidate_bytes;
    // One-block tiles (small launches) take as deep a ring as fits: 0.187 -> 0.181 ms per 4096-row block. Two-block tiles
    // stay at three stages: deeper rings for the narrow, DRAM-bound ones made a 16384-row launch slower (1.82 -> 1.85 ms per
    // block), their CTAs then take bandwidth from the wide ones that finish last.
    uint32_t const stages = tile.blocks == 2 ? 3u : min(bwd_stages, p.ring_bytes / stage_bytes);
    uint32_t const b_offset = tile.blocks * bwd_a_bytes;
    uint32_t const first_block = within / group * tile.blocks;
    uint32_t const blocks = min(tile.blocks, p.rows_q / bwd_rows - first_block);
    uint32_t const chunks_total = p.rows_c / bwd_depth;
    uint32_t const chunks_per_split = (chunks_total + p.split - 1) / p.split;
    uint32_t const chunk_begin = min(blockIdx.y * chunks_per_split, chunks_total);
    uint32_t const chunk_end = min(chunk_begin + chunks_per_split, chunks_total);

    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < bwd_stages; ++i) {
            mbar_init(smem_u32(&tail->stage_full[i]), 1);
            mbar_init(smem_u32(&tail->stage_empty[i]), 1);
        }
        mbar_init(smem_u32(&tail->accumulated), 1);
        fence_barrier_init();
    }
    let_dependents_start();
    if (chunk_begin >= chunk_end) { // a split with nothing left
        wait_for_kernels_before();
        return;
    }
    if (warp == 5) {
        if constexpr (pair_) {
            tmem_alloc_pair(smem_u32(&tail->tmem_base), p.tmem_columns);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(smem_u32(&tail->tmem_base), p.tmem_columns);
            tmem_relinquish();
        }
    }
    if (warp == 4 && lane == 0) {
        tma_prefetch_descriptor(&cube_map);
        for (uint32_t i = 0; i < (mn_major_ ? 1u : bwd_candidate_maps); ++i) tma_prefetch_descriptor(&candidates.maps[i]);
    }
    if constexpr (pair_) cluster_sync(); // the other CTA's barriers are set up
    // Everything up to here may run beside the end of the kernel before.
    wait_for_kernels_before();
    if (threadIdx.x == 0) tail->abort_flag = status_poisoned(p.status) ? 1u : 0u;
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    uint32_t const tmem_base = tail->tmem_base;
    wait_context const ctx{p.status, p.budget_ns, &tail->abort_flag};

    // The producer's and the issuer's loops are run by one elected lane each, as in the forward kernel (walked by the whole warp a
    // launch of 2944 rows, H=832, K=4 took 31 us instead of 29, one of 2048 rows, H=2048, K=8 41 instead of 36).
    bool const poisoned = tail->abort_flag != 0u; // by an earlier kernel: nothing is added
    if (poisoned) {
    } else if (warp == 4) {
        if (elect_one()) {
            uint32_t stage = 0, phase = 0;
            uint32_t const bytes = blocks * bwd_a_bytes + candidate_bytes;
            for (uint32_t chunk = chunk_begin; chunk < chunk_end; ++chunk) {
                if (!mbar_wait(smem_u32(&tail->stage_empty[stage]), phase ^ 1u, ctx, site_bwd_stage_empty, chunk)) break;
                uint32_t const full = smem_u32(&tail->stage_full[stage]);
                uint32_t const destination = stages_base + stage * stage_bytes;
                if constexpr (pair_) {
                    // The first CTA's barrier counts both CTAs' bytes, whichever arrive first.
                    uint32_t const counted = smem_of(full, 0);
                    if (rank == 0) mbar_arrive_expect_tx(full, 2 * bytes);
                    tma_load_3d_pair(destination, &cube_map, counted, static_cast<int>(chunk * bwd_depth), static_cast<int>(first_block * bwd_rows),
                                     static_cast<int>(tile.band));
                    for (uint32_t box = 0; box < boxes; ++box)
                        tma_load_2d_pair(destination + b_offset + box * bwd_mn_box_bytes, &candidates.maps[0], counted,
                                         static_cast<int>(tile.channel0 + rank * (pair_width / 2) + box * 64u), static_cast<int>(chunk * bwd_depth));
                    if (++stage == stages) stage = 0, phase ^= 1u;
                    continue;
                }
                mbar_arrive_expect_tx(full, bytes);
                for (uint32_t block = 0; block < blocks; ++block)
                    tma_load_3d(destination + block * bwd_a_bytes, &cube_map, full, static_cast<int>(chunk * bwd_depth),
                                static_cast<int>((first_block + block) * bwd_rows), static_cast<int>(tile.band));
                if constexpr (mn_major_) {
                    // Boxes of 64 channels x 64 candidates straight from the row-major block; channels past the tile (or
                    // past the tensor, which the load fills with zeros) are carried along and never multiplied.
                    for (uint32_t box = 0; box < boxes; ++box)
                        tma_load_2d(destination + b_offset + box * bwd_mn_box_bytes, &candidates.maps[0], full,
                                    static_cast<int>(tile.channel0 + box * 64u), static_cast<int>(chunk * bwd_depth));
                } else {
                    // Largest boxes first; 16 channels are 2048 bytes of the stage (rows of 128 bytes under the swizzle).
                    uint32_t done = 0;
#pragma unroll
                    for (int index = static_cast<int>(bwd_candidate_maps) - 1; index >= 0; --index) {
                        uint32_t const box = 16u << index;
                        if (tile.width - done >= box) {
                            tma_load_2d(destination + b_offset + done * 128u, &candidates.maps[index], full,
                                        static_cast<int>(chunk * bwd_depth), static_cast<int>(tile.channel0 + done));
                            done += box;
                        }
                    }
                }
                if (++stage == stages) stage = 0, phase ^= 1u;
            }
        }
    } else if (warp == 5) {
        if (rank == 0 && elect_one()) {
            // A tile wider than one UMMA's 256 columns is issued in two pieces; the second starts 256 channels on, which is
            // 32 KB into the candidate stage in either layout (four 8 KB boxes, or 256 rows of 128 bytes).
            uint32_t const major = mn_major_ ? umma_idesc_b_mn_major : 0u;
            uint32_t const width0 = wide ? bwd_max_width : tile.width;
            uint32_t const idesc0 = (pair_ ? umma_idesc_bf16(2 * bwd_rows, pair_width) : umma_idesc_bf16(bwd_rows, width0)) | major;
            uint32_t const idesc1 = wide ? (umma_idesc_bf16(bwd_rows, tile.width - bwd_max_width) | major) : 0u;
            auto multiply = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
                if constexpr (pair_) umma_bf16_pair(d, a, b, idesc, accumulate);
                else umma_bf16(d, a, b, idesc, accumulate);
            };
            auto commit = [&](uint32_t bar) {
                if constexpr (pair_) umma_commit_pair(smem_of(bar, 0)), umma_commit_pair(smem_of(bar, 1));
                else umma_commit(bar);
            };
            constexpr uint32_t descriptor_high = (1024u >> 4) | (1u << 14) | (2u << 29); // stride 1024 B, version 1, 128-byte swizzle
            uint32_t const low_base = ((stages_base & 0x3FFFFu) >> 4) | (1u << 16);
            // The B operand's leading offset (bits 16-29 of the low word) and its advance per 16 candidates.
            constexpr uint32_t b_leading = mn_major_ ? ((bwd_mn_box_bytes >> 4) << 16) : (1u << 16);
            constexpr uint32_t b_step = mn_major_ ? (2048u >> 4) : 2u;
            uint32_t stage = 0, phase = 0, accumulate = 0;
            bool ok = true;
            for (uint32_t chunk = chunk_begin; chunk < chunk_end; ++chunk) {
                ok = mbar_wait(smem_u32(&tail->stage_full[stage]), phase, ctx, site_bwd_stage_full, chunk);
                if (!ok) break;
                tcgen05_fence_after();
                uint32_t const a_low = low_base + ((stage * stage_bytes) >> 4);
                uint64_t a_descriptor, b_descriptor;
                asm("mov.b64 %0, {%1, %2};" : "=l"(a_descriptor) : "r"(a_low), "r"(descriptor_high));
                asm("mov.b64 %0, {%1, %2};" : "=l"(b_descriptor) : "r"((a_low & 0xFFFFu) + (b_offset >> 4) + b_leading), "r"(descriptor_high));
                // Straight-line runs of four: with a loop over the row blocks around them and the wide tile's test between them, a
                // chunk took 457 cycles to issue (64 channels, nothing to load) and 730 (256 channels), now 255 and 540.
                auto four_steps = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t idesc) {
                    multiply(d, a, b, idesc, accumulate);
                    multiply(d, a + 2u, b + b_step, idesc, 1u);
                    multiply(d, a + 4u, b + 2u * b_step, idesc, 1u);
                    multiply(d, a + 6u, b + 3u * b_step, idesc, 1u);
                };
                four_steps(tmem_base, a_descriptor, b_descriptor, idesc0);
                if (!pair_ && blocks == 2) four_steps(tmem_base + bwd_block_columns, a_descriptor + (bwd_a_bytes >> 4), b_descriptor, idesc0);
                if (!pair_ && wide) four_steps(tmem_base + bwd_max_width, a_descriptor, b_descriptor + ((bwd_max_width * bwd_depth * 2u) >> 4), idesc1);
                accumulate = 1;
                commit(smem_u32(&tail->stage_empty[stage]));
                if (++stage == stages) stage = 0, phase ^= 1u;
            }
            if (ok) commit(smem_u32(&tail->accumulated));
        }
    } else {
        if (p.partials != nullptr) fold_share(p, warp, lane);
        if (mbar_wait(smem_u32(&tail->accumulated), 0u, ctx, site_bwd_accumulated, tile_index)) {
            tcgen05_fence_after();
            for (uint32_t block = 0; block < blocks; ++block) {
                uint32_t const row = (first_block + block) * bwd_rows + warp * 32 + lane;
                float* destination = p.query_gradient + static_cast<size_t>(row) * p.hidden + tile.channel0;
                uint32_t const lane_base = tmem_base + ((warp * 32u) << 16) + block * bwd_block_columns;
                for (uint32_t column = 0; column < tile.width; column += 16) {
                    if (!SC_WARP_IN_BOUNDS(static_cast<size_t>(row) * p.hidden + tile.channel0 + column + 15,
                                           static_cast<size_t>(p.rows_q) * p.hidden))
                        break;
                    uint32_t values[16];
                    tmem_load_16(lane_base + column, values);
                    tmem_load_wait();
#pragma unroll
                    for (int v = 0; v < 4; ++v)
                        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(destination + column + 4 * v),
                                     "f"(p.scale * __uint_as_float(values[4 * v])), "f"(p.scale * __uint_as_float(values[4 * v + 1])),
                                     "f"(p.scale * __uint_as_float(values[4 * v + 2])), "f"(p.scale * __uint_as_float(values[4 * v + 3]))
                                     : "memory");
                }
            }
        }
    }

    tcgen05_fence_before();
    __syncthreads();
    if (!poisoned && tail->abort_flag != 0u) {
        uint64_t const start = global_timer_ns();
        while (global_timer_ns() - start < 200000ull) __nanosleep(1000);
    }
    // A pair's barriers and operands are used by both CTAs until both are done.
    if constexpr (pair_) cluster_sync();
    else __syncthreads();
    if (warp == 5) {
        tcgen05_fence_after();
        if constexpr (pair_) tmem_dealloc_pair(tmem_base, p.tmem_columns);
        else tmem_dealloc(tmem_base, p.tmem_columns);
    }
}

// The launch's tile table: which (band, channels, row blocks per CTA) tiles there are and which CTAs of the
// one-dimensional grid belong to each. Pure arithmetic on the shape, so that it can be checked without a GPU.
uint32_t plan_tiles(uint32_t rows_q, ladder_host const& ladder, uint32_t split, int multiprocessors, bwd_tile* tiles,
                    uint32_t& tile_count, bool& shared) {
    tile_count = 0;
    // Two row blocks per CTA once that still leaves at least two CTAs per multiprocessor with tiles of 256 channels. Only
    // then (a launch bound by the cube's bytes, not by its tail) does a band of 257..384 channels go to one-block CTAs
    // that take it whole; a small launch prefers more and shorter CTAs.
    uint32_t const row_blocks = rows_q / bwd_rows;
    uint32_t plain_tiles = 0, narrow_tiles = 0, begin = 0;
    for (uint32_t band = 0; band < ladder.count; ++band) {
        uint32_t const end = ladder.ends[band];
        if (end % 16 || end <= begin) throw std::runtime_error("backward: band edges must ascend in multiples of 16");
        plain_tiles += (end - begin + bwd_max_width - 1) / bwd_max_width;
        narrow_tiles += (end - begin + bwd_shared_width - 1) / bwd_shared_width;
        begin = end;
    }
    bool const two_blocks = static_cast<uint64_t>(row_blocks / 2) * plain_tiles * split >= 2ull * static_cast<uint64_t>(multiprocessors);
    // One-block tiles that make a little more than one CTA per multiprocessor leave most of the chip idle in a second round
    // (4096 rows, H=768, K=5: 192 CTAs on 148, 58 us). Cut to 128 channels they run two to a multiprocessor, each with half
    // the ring and half the tensor memory, as long as all of them are resident at once: 47 us. One with more CTAs than two per
    // multiprocessor, which would start a third round, stays with 256 channels.
    uint64_t const rounds_of = static_cast<uint64_t>(row_blocks) * split;
    shared = !two_blocks && rounds_of * plain_tiles > static_cast<uint64_t>(multiprocessors) && narrow_tiles <= bwd_max_tiles &&
             rounds_of * narrow_tiles <= 2ull * static_cast<uint64_t>(multiprocessors);
    uint32_t widest = shared ? bwd_shared_width : bwd_max_width;
    // A launch of one round takes as long as its longest CTA: the narrowest width with which all tiles still run at once. With tiles of 256
    // channels wherever a band has them: 1024 rows, H=768, K=5 13.9 us in 48 CTAs, now 7.9 in 128; 3072 rows, H=512, K=4 26.7 -> 19.8;
    // 2944 rows, H=832, K=4 26.5 -> 22.8. Tiles narrower than a box of 64 channels still load whole ones, but 512 rows take 5.2 us
    // with 32 channels against 5.9 with 64.
    bool const one_round = !two_blocks && rounds_of * plain_tiles <= static_cast<uint64_t>(multiprocessors);
    if (one_round)
        for (uint32_t width = 32; width < bwd_max_width; width += 16) {
            uint64_t tiles_of = 0;
            for (uint32_t band = 0, from = 0; band < ladder.count; from = ladder.ends[band++]) tiles_of += (ladder.ends[band] - from + width - 1) / width;
            if (rounds_of * tiles_of > static_cast<uint64_t>(multiprocessors) || tiles_of > bwd_max_tiles) continue;
            widest = width;
            break;
        }
    begin = 0;
    for (uint32_t band = 0; band < ladder.count; ++band) {
        uint32_t const end = ladder.ends[band];
        // A band's tiles are as equal as multiples of 16 can be, where one of them is the last to end.
        uint32_t const pieces = (end - begin + widest - 1) / widest;
        uint32_t const equal = one_round ? ((end - begin + pieces - 1) / pieces + 15) / 16 * 16 : widest;
        for (uint32_t channel = begin; channel < end;) {
            if (tile_count == bwd_max_tiles) throw std::runtime_error("backward: too many channel tiles for one launch");
            uint32_t const left = end - channel;
            bool const whole_band = two_blocks && left == end - begin && left > bwd_max_width && left <= bwd_wide_width;
            uint32_t const width = whole_band || left <= equal ? left : equal;
            tiles[tile_count++] = bwd_tile{band, channel, width, two_blocks && !whole_band ? 2u : 1u, 0u, 1u};
            channel += width;
        }
        begin = end;
    }
    // CTAs go band by band in the order the hardware hands them out: two-block tiles before one-block tiles and wider
    // bands before narrower. In a large launch the two-block CTAs of the narrow bands wait for DRAM
    // while the one-block CTAs of a whole wide band are busy with their UMMAs; measured, the launch is fastest with the
    // latter last (1.832 ms per 16384-row block against 1.861 with them first and 1.860 with both kinds mixed pair of
    // row blocks by pair).
    auto band_width = [&](uint32_t band) { return ladder.ends[band] - (band ? ladder.ends[band - 1] : 0u); };
    auto before = [&](bwd_tile const& x, bwd_tile const& y) { // does x go ahead of y?
        if (x.blocks != y.blocks) return x.blocks > y.blocks;
        if (x.band != y.band) return band_width(x.band) != band_width(y.band) ? band_width(x.band) > band_width(y.band) : x.band > y.band;
        return x.width > y.width;
    };
    for (uint32_t i = 1; i < tile_count; ++i)
        for (uint32_t j = i; j > 0 && before(tiles[j], tiles[j - 1]); --j) {
            bwd_tile const held = tiles[j - 1];
            tiles[j - 1] = tiles[j], tiles[j] = held;
        }
    // The tiles of one band read the same rows of the cube. Their CTAs for a row block are handed out one after the
    // other, so that they run side by side at the pace of the slower one and the second read of a row is served by L2.
    uint32_t ctas = 0;
    for (uint32_t i = 0; i < tile_count;) {
        uint32_t members = 1;
        while (i + members < tile_count && tiles[i + members].band == tiles[i].band &&
               tiles[i + members].blocks == tiles[i].blocks)
            ++members;
        for (uint32_t m = 0; m < members; ++m) tiles[i + m].first_cta = ctas, tiles[i + m].group = members;
        ctas += members * ((row_blocks + tiles[i].blocks - 1) / tiles[i].blocks);
        i += members;
    }
    return ctas;
}

} // namespace

void launch_backward(backward_arguments const& a, cudaStream_t stream) {
    if (a.rows_q % bwd_rows || a.rows_c % bwd_depth || a.hidden % 16)
        throw std::runtime_error("backward: rows must be multiples of 128 (queries) and 64 (candidates)");
    if (a.split < 1) throw std::runtime_error("backward: split must be at least 1");
    bwd_params p{};
    p.query_gradient = a.query_gradient, p.status = a.status;
    p.rows_q = a.rows_q, p.rows_c = a.rows_c, p.hidden = a.hidden;
    p.split = a.split, p.budget_ns = a.budget_ns, p.scale = a.scale;
    if (a.partials != nullptr && (a.split != 1 || a.row_accumulators == nullptr))
        throw std::runtime_error("backward: the partial records are folded by launches without split, into row accumulators");
    p.partials = a.partials, p.row_accumulators = a.row_accumulators;
    p.partial_slots = a.partial_slots, p.quantities = a.quantities;
    // Per device, once: the multiprocessor count (a runtime query that needs no context of its own).
    static int counted_device = -1, multiprocessors = 148;
    int device = 0;
    cudaGetDevice(&device);
    if (counted_device != device) {
        if (cudaDeviceGetAttribute(&multiprocessors, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) multiprocessors = 148;
        counted_device = device;
    }
    bool shared = false;
    uint32_t const ctas = plan_tiles(a.rows_q, a.ladder, a.split, multiprocessors, p.tiles, p.tile_count, shared);
    p.ring_bytes = shared ? bwd_half_ring_bytes : bwd_ring_bytes;
    p.tmem_columns = shared ? bwd_tmem_columns / 2 : bwd_tmem_columns;
    uint32_t const shared_bytes = bwd_shared_bytes_for(p.ring_bytes);
    bool const mn_major = a.candidates_row_major != nullptr && a.hidden >= 64;
    if (!mn_major && a.transposed_candidates == nullptr) throw std::runtime_error("backward: no candidates given");
    // Everything above is checked before the first driver or runtime call.
    cuuint64_t const cube_dims[3] = {a.rows_c, a.rows_q, a.ladder.count};
    cuuint64_t const cube_strides[2] = {static_cast<cuuint64_t>(a.rows_c) * 2, static_cast<cuuint64_t>(a.rows_c) * a.rows_q * 2};
    cuuint32_t const cube_box[3] = {bwd_depth, bwd_rows, 1};
    CUtensorMap const cube_map = cached_map(a.gradient_cube_bf16, 3, cube_dims, cube_strides, cube_box, CU_TENSOR_MAP_SWIZZLE_128B,
                                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    bwd_candidate_boxes candidates;
    for (uint32_t index = 0; index < bwd_candidate_maps; ++index) {
        if (mn_major) {
            // One map over the block as it lies in memory: boxes of 64 channels (the contiguous dimension) x 64 candidates.
            candidates.maps[index] = cached_operand_map(a.candidates_row_major, a.hidden, a.rows_c, 64, bwd_depth);
            continue;
        }
        // A box may not be taller than the tensor; such a box is never asked for either (tiles are at most `hidden` wide).
        uint32_t const channels = 16u << index;
        candidates.maps[index] =
            cached_operand_map(a.transposed_candidates, a.rows_c, a.hidden, bwd_depth, channels <= a.hidden ? channels : 16u);
    }

    // Per device, once: the shared-memory limit of the kernel.
    static int prepared_device = -1;
    if (prepared_device != device) {
        for (auto* kernel : {backward_kernel<false, false>, backward_kernel<true, false>, backward_kernel<true, true>})
            require(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bwd_shared_bytes),
                    "raising the backward kernel's shared memory");
        prepared_device = device;
    }
    dim3 const grid(ctas, a.split, 1);
    // Pairs of CTAs, each with one row block of a tile, load half of its candidates each: where a launch of one-block tiles is more than one
    // round (4096 rows, H=768, K=5 44.5 -> 40.8 us, 6144 rows, H=1024, K=2 85 -> 78). In one round the barriers across CTAs cost more
    // than that (1024 rows 7.6 -> 9 us), as with bands narrower than a pair's UMMA (2048 rows, H=2048, K=8 28 -> 30); in a large launch, whose
    // two-block CTAs share their candidates already, it changed nothing (16384 rows, H=1024, K=5, a whole step 2.09 ms either way).
    bool pair = mn_major && a.rows_q / bwd_rows % 2 == 0 && static_cast<uint64_t>(ctas) * a.split > static_cast<uint64_t>(multiprocessors);
    for (uint32_t i = 0; i < p.tile_count; ++i)
        pair = pair && p.tiles[i].blocks == 1 && p.tiles[i].width >= 32 && p.tiles[i].width <= bwd_max_width;
    if (pair)
        launch_dependent_clusters(!a.ordinary_launch, 2, backward_kernel<true, true>, grid, bwd_threads, shared_bytes, stream, cube_map,
                                  candidates, p);
    else
        launch_dependent(!a.ordinary_launch, mn_major ? backward_kernel<true, false> : backward_kernel<false, false>, grid, bwd_threads, shared_bytes,
                         stream, cube_map, candidates, p);
    cudaError_t const error = cudaGetLastError();
    if (error != cudaSuccess) throw std::runtime_error(std::string("backward launch failed: ") + cudaGetErrorString(error));
    note_launch();
}

std::vector<std::array<uint32_t, 6>> backward_plan(uint32_t rows_q, ladder_host const& ladder, uint32_t split,
                                                    int multiprocessors, uint32_t* ctas) {
    if (rows_q % bwd_rows || split < 1) throw std::runtime_error("backward_plan: rows must be a multiple of 128 and split positive");
    bwd_tile tiles[bwd_max_tiles];
    uint32_t count = 0;
    bool shared = false;
    uint32_t const total = plan_tiles(rows_q, ladder, split, multiprocessors, tiles, count, shared);
    if (ctas) *ctas = total;
    std::vector<std::array<uint32_t, 6>> out;
    for (uint32_t i = 0; i < count; ++i)
        out.push_back({tiles[i].band, tiles[i].channel0, tiles[i].width, tiles[i].blocks, tiles[i].first_cta, tiles[i].group});
    return out;
}

SC_DEFINE_BOUNDS_READER(bounds_record_backward)

void preload_backward_kernels() {
    cudaFuncAttributes attributes;
    require(cudaFuncGetAttributes(&attributes, backward_kernel<false, false>), "preload backward");
    require(cudaFuncGetAttributes(&attributes, backward_kernel<true, false>), "preload backward (row-major candidates)");
    require(cudaFuncGetAttributes(&attributes, backward_kernel<true, true>), "preload backward (pairs)");
}

} // namespace sc
