// The memory-bound kernels around the two tile kernels of the streamed loss, and the keyed generators / validators.
//
//   prefix_norms      per row, the inverse norm of every prefix (and optionally a copy of the row into symmetric
//                     memory, so that publishing a block to the peers costs no extra pass), then per 64 rows the
//                     largest inverse norm, which lets a tile prove that no cosine of it sits on the floor
//   transpose         [R, H] -> [H, R] so that the gradient tiles read candidates K-major
//   pull              peer block -> local staging by plain 16-byte loads and stores
//   fold_partials     per row, adds the forward kernel's per-run partials in a fixed order (deterministic)
//   finish            folds the L2-normalisation's self term into the query gradient and casts to bfloat16; fixed-tree sums
//                     of the row accumulators into the loss summands
//
// Parity: transpose_cuda_, prefix_inverse_norms_cuda_, fold_partials_cuda_, finalize_cuda_, sum_summands_cuda_
// (scalingcontrasts.cuh:660-686, 1138-1177); keyed_* and count_* (scalingcontrasts.cu:48-105). The staging pull
// replaces the reference's cudaMemcpyAsync (scalingcontrasts.cuh:1262-1265).
#include <algorithm>
#include <stdexcept>
#include <string>

#include "api.h"
#include "common.cuh"
#include "launch.h"

namespace sc {

namespace {

void check_launch(char const* what) {
    cudaError_t const error = cudaGetLastError();
    if (error != cudaSuccess) throw std::runtime_error(std::string(what) + " launch failed: " + cudaGetErrorString(error));
    note_launch();
}

ladder_t to_device(ladder_host const& host) {
    ladder_t ladder{};
    ladder.count = host.count;
    for (int i = 0; i < 8; ++i) ladder.ends[i] = host.ends[i];
    return ladder;
}

// A block takes 64 rows, a warp two of them with the loads of both in flight; the block then has the rows' largest inverse
// norm per band at hand, which had a launch of its own before (2.9 us). Each lane reads 16-byte vectors (8 channels); band
// edges are multiples of 16 channels, so a vector never straddles two bands.
constexpr uint32_t norm_rows = 64, norm_warps = 32;
__global__ void __launch_bounds__(norm_warps * 32)
    prefix_norms_kernel(uint4 const* rows, uint4* copy, float* inverse_norms, float* tile_max, uint32_t row_count, uint32_t hidden,
                        ladder_t ladder, float4* clear, size_t clear_vectors, learned_scalars learned) {
    constexpr uint32_t each = norm_rows / norm_warps;
    __shared__ float largest[norm_warps][8];
    uint32_t const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    uint32_t const first = blockIdx.x * norm_rows + warp * each;
    uint32_t const vectors = hidden / 8;
    let_dependents_start();
    wait_for_kernels_before();
    for (size_t v = blockIdx.x * blockDim.x + threadIdx.x; v < clear_vectors; v += static_cast<size_t>(gridDim.x) * blockDim.x)
        clear[v] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (learned.out != nullptr && blockIdx.x == 0 && threadIdx.x == 0) {
        learned.out[0] = expf(*learned.log_scale);
        learned.out[1] = *learned.bias;
    }
    if (blockIdx.x * norm_rows >= row_count) return; // a block that only clears
    float sums[each][8];
#pragma unroll
    for (uint32_t r = 0; r < each; ++r)
#pragma unroll
        for (int band = 0; band < 8; ++band) sums[r][band] = 0.0f;
    // Three vectors of both rows are under way before the first is used (stores to `copy` stand between the trips).
    constexpr uint32_t ahead = 3;
    for (uint32_t base = lane; base < vectors; base += 32 * ahead) {
        uint4 packed[ahead][each];
#pragma unroll
        for (uint32_t a = 0; a < ahead; ++a)
#pragma unroll
            for (uint32_t r = 0; r < each; ++r) {
                uint32_t const v = base + 32 * a;
                packed[a][r] = make_uint4(0u, 0u, 0u, 0u);
                if (v < vectors && first + r < row_count &&
                    SC_IN_BOUNDS(static_cast<size_t>(first + r) * vectors + v, static_cast<size_t>(row_count) * vectors))
                    packed[a][r] = rows[static_cast<size_t>(first + r) * vectors + v];
            }
#pragma unroll
        for (uint32_t a = 0; a < ahead; ++a) {
            uint32_t const v = base + 32 * a, channel = v * 8;
            if (v >= vectors) break;
#pragma unroll
            for (uint32_t r = 0; r < each; ++r) {
                if (copy != nullptr && first + r < row_count &&
                    SC_IN_BOUNDS(static_cast<size_t>(first + r) * vectors + v, static_cast<size_t>(row_count) * vectors))
                    copy[static_cast<size_t>(first + r) * vectors + v] = packed[a][r];
                uint32_t const words[4] = {packed[a][r].x, packed[a][r].y, packed[a][r].z, packed[a][r].w};
                float square = 0;
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    float const lo = __uint_as_float(words[w] << 16), hi = __uint_as_float(words[w] & 0xFFFF0000u);
                    square = fmaf(lo, lo, square);
                    square = fmaf(hi, hi, square);
                }
#pragma unroll
                for (int band = 0; band < 8; ++band)
                    if (band < ladder.count && channel >= ladder.begin(band) && channel < ladder.ends[band]) sums[r][band] += square;
            }
        }
    }
    float running[each];
#pragma unroll
    for (uint32_t r = 0; r < each; ++r) running[r] = 0.0f;
#pragma unroll
    for (int band = 0; band < 8; ++band) {
        if (band >= ladder.count) break;
        float warp_max = 0.0f;
#pragma unroll
        for (uint32_t r = 0; r < each; ++r) {
            float total = sums[r][band];
#pragma unroll
            for (int offset = 16; offset > 0; offset >>= 1) total += __shfl_xor_sync(0xFFFFFFFFu, total, offset);
            running[r] += total;
            float const inverse = running[r] > 0.0f ? rsqrtf(running[r]) : 0.0f;
            if (lane == 0 && first + r < row_count &&
                SC_IN_BOUNDS(static_cast<size_t>(band) * row_count + first + r, static_cast<size_t>(ladder.count) * row_count))
                inverse_norms[static_cast<size_t>(band) * row_count + first + r] = inverse;
            warp_max = fmaxf(warp_max, inverse);
        }
        if (lane == 0) largest[warp][band] = warp_max;
    }
    if (tile_max == nullptr) return;
    __syncthreads();
    // tile_max[band, t] = max over rows [64 t, 64 t + 64) of inverse_norms[band, row]; warp b takes band b.
    if (warp < ladder.count) {
        float value = largest[lane][warp];
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) value = fmaxf(value, __shfl_xor_sync(0xFFFFFFFFu, value, offset));
        size_t const tiles = row_count / norm_rows;
        if (lane == 0 && SC_IN_BOUNDS(warp * tiles + blockIdx.x, ladder.count * tiles)) tile_max[warp * tiles + blockIdx.x] = value;
    }
}

__global__ void __launch_bounds__(256)
    transpose_kernel(__nv_bfloat16 const* in, __nv_bfloat16* out, uint32_t rows, uint32_t hidden) {
    __shared__ __nv_bfloat16 tile[32][33];
    let_dependents_start();
    wait_for_kernels_before();
    uint32_t const column = blockIdx.x * 32 + threadIdx.x;
    for (uint32_t r = threadIdx.y; r < 32; r += 8) {
        uint32_t const row = blockIdx.y * 32 + r;
        if (row < rows && column < hidden && SC_IN_BOUNDS(static_cast<size_t>(row) * hidden + column, static_cast<size_t>(rows) * hidden))
            tile[r][threadIdx.x] = in[static_cast<size_t>(row) * hidden + column];
    }
    __syncthreads();
    uint32_t const out_column = blockIdx.y * 32 + threadIdx.x;
    for (uint32_t r = threadIdx.y; r < 32; r += 8) {
        uint32_t const out_row = blockIdx.x * 32 + r;
        if (out_row < hidden && out_column < rows &&
            SC_IN_BOUNDS(static_cast<size_t>(out_row) * rows + out_column, static_cast<size_t>(rows) * hidden))
            out[static_cast<size_t>(out_row) * rows + out_column] = tile[threadIdx.x][r];
    }
}

__device__ __forceinline__ void copy_vectors(uint4 const* src, uint4* dst, size_t vectors, size_t thread, size_t threads) {
    size_t index = thread;
    for (; index + 3 * threads < vectors; index += 4 * threads) {
        uint4 a = src[index], b = src[index + threads], c = src[index + 2 * threads], d = src[index + 3 * threads];
        dst[index] = a, dst[index + threads] = b, dst[index + 2 * threads] = c, dst[index + 3 * threads] = d;
    }
    for (; index < vectors; index += threads) dst[index] = src[index];
}

__global__ void __launch_bounds__(256) pull_kernel(pull_request request) {
    let_dependents_start();
    wait_for_kernels_before();
    size_t const thread = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    size_t const threads = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (int part = 0; part < 2; ++part)
        if (request.bytes[part] != 0)
            copy_vectors(static_cast<uint4 const*>(request.src[part]), static_cast<uint4*>(request.dst[part]),
                         request.bytes[part] / 16, thread, threads);
}

// A block takes 128 rows of one quantity: a lane four rows (one 16-byte load per record), a warp every eighth record, four
// of them in flight; the warps' sums are then added in warp order, so the result is the same from run to run. Bound by the
// latency of its loads: with a thread per row and all records in one chain, 128 records of 4096 rows took 20 us.
constexpr uint32_t fold_warps = 8;
// Four rows from `row` on; without `vector_` (rows or pointers that are no whole, aligned vectors) word by word.
template <bool vector_> __device__ __forceinline__ float4 load_rows(float const* quantity, uint32_t row, uint32_t rows) {
    if constexpr (vector_) {
        return row < rows ? *reinterpret_cast<float4 const*>(quantity + row) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    } else {
        return make_float4(row < rows ? quantity[row] : 0.0f, row + 1 < rows ? quantity[row + 1] : 0.0f,
                           row + 2 < rows ? quantity[row + 2] : 0.0f, row + 3 < rows ? quantity[row + 3] : 0.0f);
    }
}
template <bool vector_>
__global__ void __launch_bounds__(fold_warps * 32)
    fold_partials_kernel(float const* partials, float* accumulators, uint32_t rows, uint32_t slots,
                         uint32_t quantities) {
    __shared__ float4 sums[fold_warps][32];
    uint32_t const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    uint32_t const row = blockIdx.x * 128 + lane * 4;
    uint32_t const quantity = blockIdx.y;
    float4 total = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    size_t const stride = static_cast<size_t>(quantities) * rows;
    let_dependents_start();
    wait_for_kernels_before();
    float const* const first = partials + static_cast<size_t>(quantity) * rows;
#pragma unroll 4
    for (uint32_t slot = warp; slot < slots; slot += fold_warps)
        if (SC_IN_BOUNDS(slot * stride + static_cast<size_t>(quantity) * rows + rows - 1, static_cast<size_t>(slots) * stride)) {
            float4 const record = load_rows<vector_>(first + slot * stride, row, rows);
            total.x += record.x, total.y += record.y, total.z += record.z, total.w += record.w;
        }
    sums[warp][lane] = total;
    __syncthreads();
    if (warp != 0) return;
#pragma unroll
    for (uint32_t w = 1; w < fold_warps; ++w) {
        float4 const other = sums[w][lane];
        total.x += other.x, total.y += other.y, total.z += other.z, total.w += other.w;
    }
    float* const into = accumulators + static_cast<size_t>(quantity) * rows;
    float4 const before = load_rows<vector_>(into, row, rows);
    float4 const after = make_float4(before.x + total.x, before.y + total.y, before.z + total.z, before.w + total.w);
    if constexpr (vector_) {
        if (row < rows) *reinterpret_cast<float4*>(into + row) = after;
    } else {
        if (row < rows) into[row] = after.x;
        if (row + 1 < rows) into[row + 1] = after.y;
        if (row + 2 < rows) into[row + 2] = after.z;
        if (row + 3 < rows) into[row + 3] = after.w;
    }
}

// The end of a step, one launch. Row accumulators are laid out [quantity, row] with quantities: 0 bias grad, 1 log-beta
// grad, 2..2+K prefix losses, 2+K..2+2K self coefficients. Block 0 reduces the first 2 + K of them to the summands; it is
// the first to start and done before the others (a launch of its own with one pass per quantity took 9 us at 4096 rows).
// Every other block takes eight rows, a warp each: the self term of the normalisation is folded into the gradient, which
// leaves as bfloat16. Bound by memory.
constexpr uint32_t finish_warps = 8;

// A fixed reduction tree, so the bits do not depend on anything but the inputs. All quantities go in one pass: a thread has
// a 16-byte load of every quantity in flight at once, and the block meets twice instead of twice per quantity.
template <uint32_t prefixes_>
__device__ __forceinline__ void sum_summands(float const* accumulators, float* summands, uint32_t rows) {
    constexpr uint32_t quantities = 2 + prefixes_, prefixes = prefixes_, warps = finish_warps;
    __shared__ float scratch[quantities][warps];
    __shared__ float totals[quantities];
    uint32_t const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    float partial[quantities];
#pragma unroll
    for (uint32_t quantity = 0; quantity < quantities; ++quantity) partial[quantity] = 0.0f;
    uint32_t const count = rows / 4; // rows are a multiple of 4, so a quantity's rows are whole, aligned vectors
#pragma unroll 2
    for (uint32_t index = threadIdx.x; index < count; index += warps * 32) {
        float4 held[quantities];
#pragma unroll
        for (uint32_t quantity = 0; quantity < quantities; ++quantity)
            held[quantity] = reinterpret_cast<float4 const*>(accumulators + static_cast<size_t>(quantity) * rows)[index];
#pragma unroll
        for (uint32_t quantity = 0; quantity < quantities; ++quantity)
            partial[quantity] += (held[quantity].x + held[quantity].y) + (held[quantity].z + held[quantity].w);
    }
#pragma unroll
    for (uint32_t quantity = 0; quantity < quantities; ++quantity) {
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) partial[quantity] += __shfl_xor_sync(0xFFFFFFFFu, partial[quantity], offset);
        if (lane == 0) scratch[quantity][warp] = partial[quantity];
    }
    __syncthreads();
    if (threadIdx.x < quantities) {
        float value = 0.0f;
#pragma unroll
        for (uint32_t w = 0; w < warps; ++w) value += scratch[threadIdx.x][w];
        totals[threadIdx.x] = value;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float loss = 0;
        for (uint32_t band = 0; band < prefixes; ++band) loss += totals[2 + band];
        summands[0] = loss;
        summands[1] = totals[0];
        summands[2] = totals[1];
        summands[3] = 0.0f;
        for (uint32_t band = 0; band < 8; ++band) summands[4 + band] = band < prefixes ? totals[2 + band] : 0.0f;
    }
}

template <uint32_t prefixes_>
__global__ void __launch_bounds__(finish_warps * 32)
    finish_kernel(uint4 const* queries, float const* inverse_norms, float const* accumulators, float const* query_gradient,
                  uint4* gradient_out, float* summands, uint32_t rows, uint32_t hidden, ladder_t ladder) {
    let_dependents_start();
    wait_for_kernels_before();
    if (blockIdx.x == 0) {
        sum_summands<prefixes_>(accumulators, summands, rows);
        return;
    }
    __shared__ float folds[finish_warps][8]; // per row, [b] = sum over bands k >= b of coefficient_k * inverse_norm_k^2
    uint32_t const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    uint32_t const row = (blockIdx.x - 1) * finish_warps + warp;
    if (row >= rows) return;
    if (lane == 0) {
        float inverse[prefixes_], coefficient[prefixes_], running = 0;
#pragma unroll
        for (uint32_t band = 0; band < prefixes_; ++band) {
            inverse[band] = inverse_norms[static_cast<size_t>(band) * rows + row];
            coefficient[band] = accumulators[static_cast<size_t>(2 + prefixes_ + band) * rows + row];
        }
#pragma unroll
        for (int band = static_cast<int>(prefixes_) - 1; band >= 0; --band) {
            running += coefficient[band] * inverse[band] * inverse[band];
            folds[warp][band] = running;
        }
    }
    __syncwarp();
    uint32_t const vectors = hidden / 8;
    constexpr uint32_t ahead = 3; // vectors under way before the first is used
    for (uint32_t base = lane; base < vectors; base += 32 * ahead) {
        uint4 packed[ahead];
        float4 g0[ahead], g1[ahead];
#pragma unroll
        for (uint32_t a = 0; a < ahead; ++a) {
            uint32_t const v = base + 32 * a, channel = v * 8;
            if (v >= vectors || !SC_IN_BOUNDS(static_cast<size_t>(row) * hidden + channel + 7, static_cast<size_t>(rows) * hidden)) continue;
            packed[a] = queries[static_cast<size_t>(row) * vectors + v];
            g0[a] = *reinterpret_cast<float4 const*>(query_gradient + static_cast<size_t>(row) * hidden + channel);
            g1[a] = *reinterpret_cast<float4 const*>(query_gradient + static_cast<size_t>(row) * hidden + channel + 4);
        }
#pragma unroll
        for (uint32_t a = 0; a < ahead; ++a) {
            uint32_t const v = base + 32 * a, channel = v * 8;
            if (v >= vectors || !SC_IN_BOUNDS(static_cast<size_t>(row) * hidden + channel + 7, static_cast<size_t>(rows) * hidden)) continue;
            uint32_t band = 0;
#pragma unroll
            for (uint32_t b = 0; b + 1 < prefixes_; ++b) band += channel >= ladder.ends[b] ? 1u : 0u;
            float const fold = folds[warp][band];
            uint32_t const words[4] = {packed[a].x, packed[a].y, packed[a].z, packed[a].w};
            float const g[8] = {g0[a].x, g0[a].y, g0[a].z, g0[a].w, g1[a].x, g1[a].y, g1[a].z, g1[a].w};
            uint32_t out[4];
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                float const lo = __uint_as_float(words[w] << 16), hi = __uint_as_float(words[w] & 0xFFFF0000u);
                out[w] = pack_bf16x2(fmaf(-fold, lo, g[2 * w]), fmaf(-fold, hi, g[2 * w + 1]));
            }
            gradient_out[static_cast<size_t>(row) * vectors + v] = make_uint4(out[0], out[1], out[2], out[3]);
        }
    }
}

// A step's summands for whoever differentiates the loss later (the span they were summed in is rewritten by the next step),
// and the loss by itself.
__global__ void keep_summands_kernel(float const* summands, float* kept, float* loss, uint32_t count) {
    let_dependents_start();
    wait_for_kernels_before();
    if (threadIdx.x < count) kept[threadIdx.x] = summands[threadIdx.x];
    if (threadIdx.x == 0) *loss = summands[0];
}

// The row gradients and the two scalar gradients times the upstream gradient (a device scalar), in one pass. The row gradients
// are bfloat16 and so is their product with the upstream gradient's nearest bfloat16; it leaves in the embeddings' type.
template <typename out_t>
__global__ void __launch_bounds__(256)
    scale_gradients_kernel(uint4 const* gradient, float const* upstream, float const* summands, out_t* out, float* scale_gradient,
                           float* bias_gradient, size_t scalars) {
    let_dependents_start();
    wait_for_kernels_before();
    float const whole = *upstream, factor = __bfloat162float(__float2bfloat16(whole));
    if (blockIdx.x == 0 && threadIdx.x == 0) *scale_gradient = summands[2] * whole, *bias_gradient = summands[1] * whole;
    size_t const threads = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t v = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < scalars / 8; v += threads) {
        if (!SC_IN_BOUNDS(v * 8 + 7, scalars)) continue;
        uint4 const packed = gradient[v];
        uint32_t const words[4] = {packed.x, packed.y, packed.z, packed.w};
        uint32_t scaled[4];
#pragma unroll
        for (int w = 0; w < 4; ++w)
            scaled[w] = pack_bf16x2(__uint_as_float(words[w] << 16) * factor, __uint_as_float(words[w] & 0xFFFF0000u) * factor);
        if constexpr (sizeof(out_t) == 2) {
            reinterpret_cast<uint4*>(out)[v] = make_uint4(scaled[0], scaled[1], scaled[2], scaled[3]);
        } else {
            float4* const into = reinterpret_cast<float4*>(out) + 2 * v;
            into[0] = make_float4(__uint_as_float(scaled[0] << 16), __uint_as_float(scaled[0] & 0xFFFF0000u),
                                  __uint_as_float(scaled[1] << 16), __uint_as_float(scaled[1] & 0xFFFF0000u));
            into[1] = make_float4(__uint_as_float(scaled[2] << 16), __uint_as_float(scaled[2] & 0xFFFF0000u),
                                  __uint_as_float(scaled[3] << 16), __uint_as_float(scaled[3] & 0xFFFF0000u));
        }
    }
}

__device__ __forceinline__ uint64_t splitmix64(uint64_t value) {
    value = (value ^ (value >> 30)) * 0xBF58476D1CE4E5B9ull;
    value = (value ^ (value >> 27)) * 0x94D049BB133111EBull;
    return value ^ (value >> 31);
}

__global__ void keyed_embeddings_kernel(__nv_bfloat16* rows, uint32_t row_count, uint32_t hidden, uint64_t salt, float scale) {
    uint64_t const row = blockIdx.x;
    for (uint32_t channel = threadIdx.x; channel < hidden; channel += blockDim.x) {
        uint64_t const bits = splitmix64((salt * row_count + row) * hidden + channel);
        rows[row * hidden + channel] = __float2bfloat16((static_cast<float>(bits >> 40) * 0x1.0p-24f - 0.5f) * scale);
    }
}

__global__ void keyed_integers_kernel(float* out, size_t scalars, size_t first, uint32_t members, uint32_t member) {
    size_t const index = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (index >= scalars) return;
    out[index] = static_cast<float>(splitmix64((first + index) * members + member) >> 52);
}

__global__ void keyed_fractions_kernel(float* out, size_t scalars, size_t first, uint32_t members, uint32_t member) {
    size_t const index = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (index >= scalars) return;
    out[index] = static_cast<float>(splitmix64((first + index) * members + member) >> 40) * 0x1.0p-24f - 0.5f;
}

__global__ void count_wrong_sums_kernel(float const* values, size_t scalars, size_t first, uint32_t members,
                                        unsigned long long* counter) {
    size_t const index = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (index >= scalars) return;
    float expected = 0;
    for (uint32_t member = 0; member < members; ++member)
        expected += static_cast<float>(splitmix64((first + index) * members + member) >> 52);
    if (values[index] != expected) atomicAdd(counter, 1ull);
}

__global__ void count_differences_kernel(uint32_t const* values, uint32_t const* expected, size_t scalars,
                                         unsigned long long* counter) {
    size_t const index = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (index >= scalars) return;
    if (values[index] != expected[index]) atomicAdd(counter, 1ull);
}

__global__ void scale_cast_kernel(float const* __restrict__ src, __nv_bfloat16* __restrict__ dst, size_t scalars, float scale) {
    size_t const index = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (index < scalars) dst[index] = __float2bfloat16(src[index] * scale);
}

int blocks_of(size_t items, int per_block) { return static_cast<int>((items + per_block - 1) / per_block); }

} // namespace

// How far passes over memory spread; no result depends on it.
constexpr size_t b200_multiprocessors = 148;

bool bounds_build() { return SC_BOUNDS != 0; }
SC_DEFINE_BOUNDS_READER(bounds_record_small)

void launch_prefix_norms(void const* rows_bf16, void* copy_bf16, float* inverse_norms, float* tile_max, uint32_t rows,
                         uint32_t hidden, ladder_host const& ladder, cudaStream_t stream, float* clear, size_t clear_floats,
                         learned_scalars learned) {
    if (hidden % 8) throw std::runtime_error("prefix_norms: hidden must be a multiple of 8");
    if (tile_max != nullptr && rows % norm_rows) throw std::runtime_error("prefix_norms: rows must be a multiple of 64 for tile maxima");
    if (clear_floats % 4 || reinterpret_cast<uintptr_t>(clear) % 16)
        throw std::runtime_error("prefix_norms: the span to clear must be whole, aligned vectors");
    // A few rows make a few blocks, which would clear a wide gradient slowly: up to one block per multiprocessor helps them.
    size_t const clearing = (clear_floats / 4 + norm_warps * 32 - 1) / (norm_warps * 32);
    int const blocks = std::max(blocks_of(rows, norm_rows), static_cast<int>(std::min<size_t>(clearing, b200_multiprocessors)));
    launch_dependent(true, prefix_norms_kernel, blocks, norm_warps * 32, 0, stream, static_cast<uint4 const*>(rows_bf16),
                     static_cast<uint4*>(copy_bf16), inverse_norms, tile_max, rows, hidden, to_device(ladder),
                     reinterpret_cast<float4*>(clear), clear_floats / 4, learned);
    check_launch("prefix_norms");
}

void launch_transpose(void const* rows_bf16, void* transposed_bf16, uint32_t rows, uint32_t hidden, cudaStream_t stream) {
    dim3 const grid((hidden + 31) / 32, (rows + 31) / 32), block(32, 8);
    launch_dependent(true, transpose_kernel, grid, block, 0, stream, static_cast<__nv_bfloat16 const*>(rows_bf16),
                     static_cast<__nv_bfloat16*>(transposed_bf16), rows, hidden);
    check_launch("transpose");
}

void launch_pull(void const* src0, void* dst0, size_t bytes0, void const* src1, void* dst1, size_t bytes1, int blocks,
                 cudaStream_t stream) {
    if (bytes0 % 16 || bytes1 % 16) throw std::runtime_error("pull: sizes must be multiples of 16 bytes");
    pull_request request{};
    request.src[0] = src0, request.dst[0] = dst0, request.bytes[0] = bytes0;
    request.src[1] = src1, request.dst[1] = dst1, request.bytes[1] = bytes1;
    launch_dependent(true, pull_kernel, blocks < 1 ? 1 : blocks, 256, 0, stream, request);
    check_launch("pull");
}

void launch_fold_partials(float const* partials, float* row_accumulators, uint32_t rows, uint32_t slots,
                          uint32_t quantities, cudaStream_t stream, bool ordinary_launch) {
    bool const vectors = rows % 4 == 0 && reinterpret_cast<uintptr_t>(partials) % 16 == 0 &&
                         reinterpret_cast<uintptr_t>(row_accumulators) % 16 == 0;
    dim3 const grid(blocks_of(rows, 128), quantities);
    launch_dependent(!ordinary_launch, vectors ? fold_partials_kernel<true> : fold_partials_kernel<false>, grid, fold_warps * 32, 0, stream, partials,
                     row_accumulators, rows, slots, quantities);
    check_launch("fold_partials");
}

void launch_finish(void const* queries_bf16, float const* inverse_norms, float const* row_accumulators,
                   float const* query_gradient, void* gradient_out_bf16, float* summands, uint32_t rows, uint32_t hidden,
                   ladder_host const& ladder, cudaStream_t stream) {
    if (rows % 4 || hidden % 8 || reinterpret_cast<uintptr_t>(row_accumulators) % 16)
        throw std::runtime_error("finish: rows must be a multiple of 4, hidden of 8 and the accumulators 16-byte aligned");
    auto launch = [&](auto kernel) {
        launch_dependent(true, kernel, 1 + blocks_of(rows, finish_warps), finish_warps * 32, 0, stream,
                         static_cast<uint4 const*>(queries_bf16), inverse_norms, row_accumulators, query_gradient,
                         static_cast<uint4*>(gradient_out_bf16), summands, rows, hidden, to_device(ladder));
    };
    switch (ladder.count) {
    case 1: launch(finish_kernel<1>); break;
    case 2: launch(finish_kernel<2>); break;
    case 3: launch(finish_kernel<3>); break;
    case 4: launch(finish_kernel<4>); break;
    case 5: launch(finish_kernel<5>); break;
    case 6: launch(finish_kernel<6>); break;
    case 7: launch(finish_kernel<7>); break;
    case 8: launch(finish_kernel<8>); break;
    default: throw std::runtime_error("finish: a ladder holds one to eight prefixes");
    }
    check_launch("finish");
}

void launch_keep_summands(float const* summands, float* kept, float* loss, uint32_t count, cudaStream_t stream) {
    if (count == 0 || count > 32) throw std::runtime_error("keep_summands: one to 32 summands");
    launch_dependent(true, keep_summands_kernel, 1, 32, 0, stream, summands, kept, loss, count);
    check_launch("keep_summands");
}

void launch_scale_gradients(void const* gradient_bf16, float const* upstream, float const* summands, void* out, bool out_f32,
                            float* scale_gradient, float* bias_gradient, size_t scalars, cudaStream_t stream) {
    if (scalars % 8 || reinterpret_cast<uintptr_t>(gradient_bf16) % 16 || reinterpret_cast<uintptr_t>(out) % 16)
        throw std::runtime_error("scale_gradients: whole, aligned vectors of eight");
    uint32_t const blocks = static_cast<uint32_t>(std::min<size_t>((scalars / 8 + 255) / 256, b200_multiprocessors * 8));
    uint4 const* const gradient = static_cast<uint4 const*>(gradient_bf16);
    if (out_f32)
        launch_dependent(true, scale_gradients_kernel<float>, blocks < 1 ? 1 : blocks, 256, 0, stream, gradient, upstream, summands,
                         static_cast<float*>(out), scale_gradient, bias_gradient, scalars);
    else
        launch_dependent(true, scale_gradients_kernel<__nv_bfloat16>, blocks < 1 ? 1 : blocks, 256, 0, stream, gradient, upstream,
                         summands, static_cast<__nv_bfloat16*>(out), scale_gradient, bias_gradient, scalars);
    check_launch("scale_gradients");
}

void launch_keyed_embeddings(void* rows_bf16, uint32_t rows, uint32_t hidden, uint64_t salt, float scale,
                             cudaStream_t stream) {
    keyed_embeddings_kernel<<<rows, 256, 0, stream>>>(static_cast<__nv_bfloat16*>(rows_bf16), rows, hidden, salt, scale);
    check_launch("keyed_embeddings");
}

void launch_keyed_integers(float* out, size_t scalars, size_t first, uint32_t members, uint32_t member,
                           cudaStream_t stream) {
    keyed_integers_kernel<<<blocks_of(scalars, 256), 256, 0, stream>>>(out, scalars, first, members, member);
    check_launch("keyed_integers");
}

void launch_keyed_fractions(float* out, size_t scalars, size_t first, uint32_t members, uint32_t member,
                            cudaStream_t stream) {
    keyed_fractions_kernel<<<blocks_of(scalars, 256), 256, 0, stream>>>(out, scalars, first, members, member);
    check_launch("keyed_fractions");
}

void launch_count_wrong_sums(float const* values, size_t scalars, size_t first, uint32_t members,
                             unsigned long long* counter, cudaStream_t stream) {
    count_wrong_sums_kernel<<<blocks_of(scalars, 256), 256, 0, stream>>>(values, scalars, first, members, counter);
    check_launch("count_wrong_sums");
}

void launch_count_differences(float const* values, float const* expected, size_t scalars, unsigned long long* counter,
                              cudaStream_t stream) {
    count_differences_kernel<<<blocks_of(scalars, 256), 256, 0, stream>>>(reinterpret_cast<uint32_t const*>(values),
                                                                       reinterpret_cast<uint32_t const*>(expected), scalars,
                                                                       counter);
    check_launch("count_differences");
}

void launch_scale_cast(float const* src, void* dst_bf16, size_t scalars, float scale, cudaStream_t stream) {
    scale_cast_kernel<<<blocks_of(scalars, 256), 256, 0, stream>>>(src, static_cast<__nv_bfloat16*>(dst_bf16), scalars, scale);
    check_launch("scale_cast");
}

} // namespace sc
