// axis.cu -- reductions along one axis (libsci's roadmap, README.md:151: "sum(a, axis) and the
// rest"): sum, minimum, maximum and mean of a row-major array over one of its axes.
//
// The whole-array reductions set the rules (include/operations/reduce.hpp:16-42, dispatch.cpp:
// 106-165): values fold in double whatever the element type, a NaN anywhere in a fold gives NaN,
// the result is cast to the element type once, and mean is that sum divided by the count in the
// element type (sum / static_cast<element>(count), reduce.hpp:27). An empty axis gives 0 for sum
// and mean and NaN for minimum and maximum.
//
// The array is viewed as (outer, extent, inner): out[o][j] = fold over k of in[o][k][j].
//   - inner == 1 (the last axis): a warp per (row, piece of the row); lanes stride the piece
//     (coalesced) and fold with shuffles in a fixed order;
//   - inner > 1: a thread per (o, piece, j), j fastest, so a warp reads 32 consecutive elements
//     per k -- or, when inner is a whole number of 16-byte vectors, a thread per (o, piece, vector
//     of j) reading 512 bytes per warp per k (rows shorter than 64 take this form, a thread
//     per row).
// Each lane keeps 4 to 16 loads in flight ahead of its ordered fold, and the kind of fold is a template
// argument. Sum over axis 0 and mean over axis 1 of 16384 x 16384 floats (one call, events around
// it): 233 -> 189 us (5.7 TB/s) and 199 -> 184; of 5001 x 7003: 54 -> 47 and 45 -> 38. A block per 128
// columns, its warps' folds combined in shared memory, took 370 us for the first (512 bytes of a row
// at a time instead of 4 KB).
// Short outputs over long axes split the axis
// into pieces so the grid fills the GPU; pieces write
// double partials that one more pass folds in piece order. The order of every fold is fixed by the
// shape, the input's 16-byte alignment (vectors or single columns) and the GPU (the pieces fill its
// waves), so results are deterministic. HBM bound: the input is read once.
#include "context.hpp"
#include "workspace.hpp"

#include <cuda_runtime.h>

#include <algorithm>
#include <limits>

using namespace sci_cuda;

namespace sci_cuda {
    namespace {

        // `fold` is a constant in the wide forms, so that their inner loops do not choose.
        __device__ __forceinline__ double fold_pair(unsigned fold, double a, double b) {
            if (fold == SCI_FOLD_SUM) return __dadd_rn(a, b);
            if (a != a) return a;
            if (b != b) return b;
            if (fold == SCI_FOLD_MINIMUM) return b < a ? b : a;
            return b > a ? b : a;
        }

        __device__ __forceinline__ double fold_start(unsigned fold) {
            if (fold == SCI_FOLD_SUM) return 0.0;
            return fold == SCI_FOLD_MINIMUM ? __longlong_as_double(0x7ff0000000000000ll)    // +inf
                                            : __longlong_as_double(0xfff0000000000000ll);  // -inf
        }

        // fold 3 is mean: the sum, then divided by the count in the element type.
        template <typename T> __device__ __forceinline__ T finish(unsigned fold, double value, unsigned long long extent);
        template <> __device__ __forceinline__ float finish<float>(unsigned fold, double value, unsigned long long extent) {
            const float narrow = __double2float_rn(value);
            return fold == 3 ? __fdiv_rn(narrow, __ull2float_rn(extent)) : narrow;
        }
        template <> __device__ __forceinline__ double finish<double>(unsigned fold, double value, unsigned long long extent) {
            return fold == 3 ? __ddiv_rn(value, __ull2double_rn(extent)) : value;
        }

        struct AxisShape {
            unsigned long long outer, extent, inner, pieces, span;  // span: k per piece
            unsigned fold;    // SCI_FOLD_* or 3 (mean)
            unsigned folded;  // the fold applied to values (mean folds as a sum)
        };

        template <typename T, unsigned FOLD, int U>
        __global__ void __launch_bounds__(256) axis_rows(const T *in, AxisShape s, double *partial, T *out) {
            const unsigned lane = threadIdx.x & 31;
            const unsigned long long warps = 1ull * gridDim.x * (blockDim.x >> 5);
            const unsigned long long units = s.outer * s.pieces;
            for (unsigned long long unit = 1ull * blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); unit < units; unit += warps) {
                const unsigned long long row = unit / s.pieces, piece = unit - row * s.pieces;
                const unsigned long long k0 = piece * s.span, k1 = k0 + s.span < s.extent ? k0 + s.span : s.extent;
                const T *line = in + row * s.extent;
                double acc = fold_start(FOLD);
                unsigned long long k = k0 + lane;
                for (; k + 32ull * (U - 1) < k1; k += 32ull * U) {
                    T v[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) v[u] = line[k + 32ull * u];
#pragma unroll
                    for (int u = 0; u < U; ++u) acc = fold_pair(FOLD, acc, static_cast<double>(v[u]));
                }
                // the rest: the same loads, each where there is an element
                T v[U];
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (k + 32ull * u < k1) v[u] = line[k + 32ull * u];
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (k + 32ull * u < k1) acc = fold_pair(FOLD, acc, static_cast<double>(v[u]));
#pragma unroll
                for (int offset = 16; offset > 0; offset >>= 1)
                    acc = fold_pair(FOLD, acc, __shfl_xor_sync(0xffffffffu, acc, offset));
                if (lane == 0) {
                    if (s.pieces == 1) out[row] = finish<T>(s.fold, acc, s.extent);
                    else partial[unit] = acc;
                }
            }
        }

        // Columns: a thread per (o, piece, group of C adjacent columns), each folding its columns in the order of k. C is a
        // 16-byte vector's width when inner is a whole number of vectors and the input 16-byte aligned, else 1.
        template <typename T, unsigned FOLD, int C>
        __global__ void __launch_bounds__(256) axis_columns(const T *in, AxisShape s, double *partial, T *out) {
            constexpr int U = 16 / C < 8 ? 8 : 16 / C;  // loads in flight
            const unsigned long long threads = 1ull * gridDim.x * blockDim.x;
            const unsigned long long groups = s.inner / C;
            const unsigned long long units = s.outer * s.pieces * groups;
            for (unsigned long long unit = 1ull * blockIdx.x * blockDim.x + threadIdx.x; unit < units; unit += threads) {
                const unsigned long long rest = unit / groups, g = unit - rest * groups;
                const unsigned long long o = rest / s.pieces, piece = rest - o * s.pieces;
                const unsigned long long k0 = piece * s.span, k1 = k0 + s.span < s.extent ? k0 + s.span : s.extent;
                const T *column = in + o * s.extent * s.inner + g * C;
                double acc[C];
#pragma unroll
                for (int e = 0; e < C; ++e) acc[e] = fold_start(FOLD);
                auto read = [&](unsigned long long k, T *v) {
                    if constexpr (C > 1) load16(column + k * s.inner, v);
                    else v[0] = column[k * s.inner];
                };
                unsigned long long k = k0;
                for (; k + U <= k1; k += U) {
                    T v[U][C];
#pragma unroll
                    for (int u = 0; u < U; ++u) read(k + u, v[u]);
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int e = 0; e < C; ++e) acc[e] = fold_pair(FOLD, acc[e], static_cast<double>(v[u][e]));
                }
                for (; k < k1; ++k) {
                    T v[C];
                    read(k, v);
#pragma unroll
                    for (int e = 0; e < C; ++e) acc[e] = fold_pair(FOLD, acc[e], static_cast<double>(v[e]));
                }
#pragma unroll
                for (int e = 0; e < C; ++e) {
                    const unsigned long long j = g * C + e;
                    if (s.pieces == 1) out[o * s.inner + j] = finish<T>(s.fold, acc[e], s.extent);
                    else partial[(o * s.pieces + piece) * s.inner + j] = acc[e];
                }
            }
        }

        // Folds the pieces of every output in piece order: partial[(o * pieces + p) * inner + j].
        template <typename T, unsigned FOLD>
        __global__ void __launch_bounds__(256) axis_pieces(const double *partial, AxisShape s, T *out) {
            const unsigned long long outputs = s.outer * s.inner, step = 1ull * gridDim.x * blockDim.x;
            for (unsigned long long i = 1ull * blockIdx.x * blockDim.x + threadIdx.x; i < outputs; i += step) {
                const unsigned long long o = i / s.inner, j = i - o * s.inner;
                double acc = fold_start(FOLD);
                const double *from = partial + o * s.pieces * s.inner + j;
                constexpr int U = 16;  // loads in flight ahead of the (ordered) fold
                unsigned long long p = 0;
                for (; p + U <= s.pieces; p += U) {
                    double v[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) v[u] = from[(p + u) * s.inner];
#pragma unroll
                    for (int u = 0; u < U; ++u) acc = fold_pair(FOLD, acc, v[u]);
                }
                for (; p < s.pieces; ++p) acc = fold_pair(FOLD, acc, from[p * s.inner]);
                out[i] = finish<T>(s.fold, acc, s.extent);
            }
        }

        template <typename T, unsigned FOLD> int launch_axis(Context &ctx, const T *in, T *out, AxisShape s) {
            // Work units for several resident waves, run by one persistent wave, so the last units do not leave most of the
            // GPU idle.
            constexpr int V = 16 / sizeof(T);
            const bool rows = s.inner == 1 && s.extent >= 64;  // shorter rows go a thread per row
            const bool vectors = !rows && s.inner % V == 0 && (reinterpret_cast<uintptr_t>(in) & 15u) == 0;
            // Loads in flight per lane of a row: 16, but a row of few steps takes the registers for more warps (sums of 1000000
            // x 65 floats: 198 us with 4, 257 with 8, 410 with 16; of 50000 x 700: 32, 28 and 31; of 30000 x 1500: 40,
            // 35 and 33).
            const void *by_rows = s.extent < 512    ? reinterpret_cast<const void *>(&axis_rows<T, FOLD, 4>)
                                  : s.extent < 1500 ? reinterpret_cast<const void *>(&axis_rows<T, FOLD, 8>)
                                                    : reinterpret_cast<const void *>(&axis_rows<T, FOLD, 16>);
            const void *kernel = rows      ? by_rows
                                 : vectors ? reinterpret_cast<const void *>(&axis_columns<T, FOLD, V>)
                                           : reinterpret_cast<const void *>(&axis_columns<T, FOLD, 1>);
            const unsigned long long most = 1ull * ctx.sms * ctx.blocks_per_sm(kernel, 256, 0);  // blocks of 256
            unsigned long long want, cap;
            if (rows) {
                // a warp per (row, piece): a wave of warps in pieces of at least 2048 values, and four waves in pieces of at
                // least 4096 (600 x 100000 floats: 57 -> 52 us)
                const unsigned long long wave = 8 * most;
                want = std::max(std::min((wave + s.outer - 1) / s.outer, (s.extent + 2047) / 2048),
                                std::min((4 * wave + s.outer - 1) / s.outer, s.extent / 4096));
                // a row per warp fills two thirds of a wave: no pieces, and no pass to fold them (5001 rows
                // of 7003 floats: 35 + 4 us in pieces, 33 without) -- unless the rows beyond the last full wave
                // are less than a quarter of one and long, and would run alone (5001 x 100000: 389 us whole, 310 in
                // four pieces; 7200 x 30000 doubles, 96 rows above two waves: 302 and 266)
                if (s.outer * 3 >= wave * 2) {
                    const bool alone = s.outer > wave && s.outer < 8 * wave && s.outer % wave * 4 < wave;
                    want = alone ? std::min<unsigned long long>(4, s.extent / 4096) : 1;
                }
                cap = s.extent;
            } else {
                // a thread per (o, piece, group of columns): four waves, in pieces of at least 64 values, at most 4096 of
                // them, which one thread per output folds (1000000 x 65 floats: 9327 pieces 827 us, 4663 439)
                const unsigned long long groups = s.outer * (vectors ? s.inner / V : s.inner);
                want = std::min<unsigned long long>((4 * most * 256 + groups - 1) / groups, 4096);
                cap = (s.extent + 63) / 64;
            }
            s.pieces = want < cap ? want : cap;
            if (s.pieces < 1) s.pieces = 1;
            s.span = (s.extent + s.pieces - 1) / s.pieces;
            s.pieces = (s.extent + s.span - 1) / s.span;
            double *partial = nullptr;
            if (s.pieces > 1) {
                if (int code = ctx.check(ctx.workspace->reserve(s.outer * s.pieces * s.inner * sizeof(double)),
                                         "reserving axis partials"))
                    return code;
                partial = static_cast<double *>(ctx.workspace->memory);
            }
            auto grid = [&](unsigned long long blocks) { return static_cast<unsigned>(blocks < most ? blocks : most); };
            if (rows) {
                void *args[] = {&in, &s, &partial, &out};
                if (int code = ctx.check(cudaLaunchKernel(kernel, dim3(grid((s.outer * s.pieces + 7) / 8)), dim3(256), args, 0, ctx.stream),
                                         "launching an axis reduction"))
                    return code;
            } else if (vectors) {
                axis_columns<T, FOLD, V><<<grid((s.outer * s.pieces * (s.inner / V) + 255) / 256), 256, 0, ctx.stream>>>(in, s, partial, out);
            } else {
                axis_columns<T, FOLD, 1><<<grid((s.outer * s.pieces * s.inner + 255) / 256), 256, 0, ctx.stream>>>(in, s, partial, out);
            }
            if (int code = ctx.check(cudaGetLastError(), "launching an axis reduction")) return code;
            if (s.pieces > 1) {
                axis_pieces<T, FOLD><<<grid((s.outer * s.inner + 255) / 256), 256, 0, ctx.stream>>>(partial, s, out);
                if (int code = ctx.check(cudaGetLastError(), "launching the axis piece fold")) return code;
            }
            return SCI_CUDA_OK;
        }

        template <typename T> int launch_fold(Context &ctx, const void *in, void *out, const AxisShape &s) {
            const T *from = static_cast<const T *>(in);
            T *to = static_cast<T *>(out);
            if (s.folded == SCI_FOLD_MINIMUM) return launch_axis<T, SCI_FOLD_MINIMUM>(ctx, from, to, s);
            if (s.folded == SCI_FOLD_MAXIMUM) return launch_axis<T, SCI_FOLD_MAXIMUM>(ctx, from, to, s);
            return launch_axis<T, SCI_FOLD_SUM>(ctx, from, to, s);
        }

    } // namespace
} // namespace sci_cuda

extern "C" int sci_cuda_reduce_axis(sci_cuda_context *context, uint32_t precision, uint32_t fold, const void *input,
                                    uint32_t rank, const uint64_t *shape, uint32_t axis, void *output) {
    if (!context) return SCI_CUDA_ERROR_INVALID;
    std::lock_guard<std::recursive_mutex> lock(context->guard);
    if (precision > SCI_PRECISION_WIDE) return context->fail(SCI_CUDA_ERROR_INVALID, "unknown precision %u", precision);
    if (fold > SCI_AXIS_MEAN) return context->fail(SCI_CUDA_ERROR_INVALID, "unknown axis fold %u", fold);
    if (rank < 1 || rank > 8 || !shape || axis >= rank)
        return context->fail(SCI_CUDA_ERROR_INVALID, "reduce_axis: axis %u of rank %u (1 to 8, with its shape)", axis, rank);
    AxisShape s{1, shape[axis], 1, 1, 0, fold, fold == SCI_AXIS_MEAN ? static_cast<unsigned>(SCI_FOLD_SUM) : fold};
    unsigned long long total = 1;
    for (uint32_t a = 0; a < rank; ++a) {
        if (shape[a] != 0 && total > ~0ull / shape[a]) return context->fail(SCI_CUDA_ERROR_INVALID, "reduce_axis: shape overflows");
        total *= shape[a];
        if (a < axis) s.outer *= shape[a];
        if (a > axis) s.inner *= shape[a];
    }
    const unsigned long long outputs = s.outer * s.inner;
    if (outputs == 0) return SCI_CUDA_OK;
    if (!output || !reachable(*context, output)) return context->fail(SCI_CUDA_ERROR_INVALID, "reduce_axis: the output is not memory of this device");
    if (s.extent == 0) {
        // an empty axis: 0 for sum and mean, NaN for minimum and maximum
        const double empty = (fold == SCI_FOLD_SUM || fold == SCI_AXIS_MEAN) ? 0.0 : std::numeric_limits<double>::quiet_NaN();
        return sci_cuda_fill(context, precision, output, outputs, empty);
    }
    if (!input || !reachable(*context, input)) return context->fail(SCI_CUDA_ERROR_INVALID, "reduce_axis: the input is not memory of this device");
    if (input == output) return context->fail(SCI_CUDA_ERROR_INVALID, "reduce_axis: the output must not be the input");
    cudaSetDevice(context->device);
    if (precision == SCI_PRECISION_WIDE) return launch_fold<double>(*context, input, output, s);
    return launch_fold<float>(*context, input, output, s);
}
