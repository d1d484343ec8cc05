// broadcast.cu -- elementwise operations over operands of different shapes, and the elementwise
// functions libsci lists as next on its roadmap (README.md:149-152: broadcasting, "so (3, 1) and
// (1, 4) arrays combine into (3, 4)"; power, floor, ceil, round, clip and where).
//
// libsci has none of these yet, so the rules are numpy's, which its operations are named after
// (include/operations/reduce.hpp:8-9):
//   - shapes: every operand has the output's rank (the caller prepends 1s), and each of its extents
//     equals the output's or is 1 (a broadcast axis, read with stride 0);
//   - add / subtract / multiply / divide: one IEEE operation, rounded once;
//   - minimum / maximum: numpy.minimum / maximum, a NaN in either operand gives NaN, and of two
//     equal values (+0 and -0) the second;
//   - floor, ceil: exact; round: numpy.round, halves to even;
//   - power: C pow; a float is raised in double and rounded once (within 1 ulp of powf);
//   - clip(x, lo, hi) = minimum(maximum(x, lo), hi), as numpy.clip;
//   - where(condition, x, y) = condition != 0 ? x : y (NaN counts as true, as in numpy).
//
// Kernels: the host merges adjacent axes that every operand reads alike (both broadcast or both
// full), so most calls reduce to one or two axes (a same-shape or scalar operation to one). When
// the last merged axis is long, blocks walk (row, piece of the last axis) pairs: the row's offsets
// are computed once per piece and the piece is read and written contiguously (stride 0 or 1 per
// operand), in 16-byte vectors, two per thread, or element by element. Short last axes map each
// thread's flat index to every operand's offset (launch_apply says where the lines lie). HBM bound:
// bytes = the output written + each operand read once (a broadcast operand mostly from L2).
#include "context.hpp"

#include <cuda_runtime.h>

#include <cmath>

using namespace sci_cuda;

namespace sci_cuda {
    namespace {

        constexpr int kMaxAxes = 8;
        constexpr unsigned kPiece = 1024;
        constexpr int kVectorsPerThread = 2;  // 16-byte vectors per thread per piece (vector form)

        template <typename T> struct ApplyLaunch {
            int code;
            int rank;                                       // merged axes
            unsigned long long extent[kMaxAxes];            // merged output extents
            unsigned long long stride[3][kMaxAxes];         // element strides (0 on broadcast axes)
            const T *input[3];
            T *output;
            unsigned long long count;
        };

        // numpy's minimum / maximum: the first operand if it is NaN or strictly smaller (larger),
        // else the second (so a NaN second operand, and the second of two equal values, win).
        template <typename T> __device__ __forceinline__ T nan_minimum(T a, T b) { return (a < b || a != a) ? a : b; }
        template <typename T> __device__ __forceinline__ T nan_maximum(T a, T b) { return (a > b || a != a) ? a : b; }

        __device__ __forceinline__ float quotient(float a, float b) { return __fdiv_rn(a, b); }
        __device__ __forceinline__ double quotient(double a, double b) { return __ddiv_rn(a, b); }
        __device__ __forceinline__ float raise(float a, float b) {
            return __double2float_rn(pow(static_cast<double>(a), static_cast<double>(b)));
        }
        __device__ __forceinline__ double raise(double a, double b) { return pow(a, b); }

        template <typename T> __device__ __forceinline__ T apply_shaped(int code, T a, T b, T c) {
            switch (code) {  // with a constant code (the vector kernel) the switch folds away
            case SCI_CODE_COPY: return a;
            case SCI_CODE_ADD: return add(a, b);
            case SCI_CODE_SUBTRACT: return sub(a, b);
            case SCI_CODE_MULTIPLY: return mul(a, b);
            case SCI_CODE_DIVIDE: return quotient(a, b);
            case SCI_CODE_MINIMUM: return nan_minimum(a, b);
            case SCI_CODE_MAXIMUM: return nan_maximum(a, b);
            case SCI_EXTRA_FLOOR: return floor(a);
            case SCI_EXTRA_CEIL: return ceil(a);
            case SCI_EXTRA_ROUND: return rint(a);
            case SCI_EXTRA_POWER: return raise(a, b);
            case SCI_EXTRA_CLIP: return nan_minimum(nan_maximum(a, b), c);
            default: return a != T(0) ? b : c;  // SCI_EXTRA_WHERE
            }
        }

        template <typename T> __device__ __forceinline__ T operand(const ApplyLaunch<T> &L, int k, unsigned long long offset) {
            return L.input[k] ? L.input[k][offset] : T(0);
        }

        // Flat: one element per thread per step, offsets from the flat index.
        template <typename T> __global__ void __launch_bounds__(256) apply_flat(const __grid_constant__ ApplyLaunch<T> L) {
            const unsigned long long step = 1ull * gridDim.x * blockDim.x;
            for (unsigned long long i = 1ull * blockIdx.x * blockDim.x + threadIdx.x; i < L.count; i += step) {
                unsigned long long rest = i, offset[3] = {0, 0, 0};
                for (int axis = L.rank - 1; axis >= 0; --axis) {
                    const unsigned long long coordinate = rest % L.extent[axis];
                    rest /= L.extent[axis];
#pragma unroll
                    for (int k = 0; k < 3; ++k) offset[k] += coordinate * L.stride[k][axis];
                }
                L.output[i] = apply_shaped<T>(L.code, operand(L, 0, offset[0]), operand(L, 1, offset[1]), operand(L, 2, offset[2]));
            }
        }

        // Rows: (row, piece of the last axis) per block step; the last axis is read with stride 0
        // or 1 per operand.
        template <typename T> __global__ void __launch_bounds__(256) apply_rows(const __grid_constant__ ApplyLaunch<T> L) {
            const int last = L.rank - 1;
            const unsigned long long columns = L.extent[last];
            const unsigned long long chunks = (columns + kPiece - 1) / kPiece;
            const unsigned long long rows = L.count / columns, pieces = rows * chunks;
            for (unsigned long long piece = blockIdx.x; piece < pieces; piece += gridDim.x) {
                const unsigned long long row = piece / chunks, c0 = (piece - row * chunks) * kPiece;
                unsigned long long rest = row, base[3] = {0, 0, 0};
                for (int axis = last - 1; axis >= 0; --axis) {
                    const unsigned long long coordinate = rest % L.extent[axis];
                    rest /= L.extent[axis];
#pragma unroll
                    for (int k = 0; k < 3; ++k) base[k] += coordinate * L.stride[k][axis];
                }
                T *out = L.output + row * columns;
                for (unsigned long long c = c0 + threadIdx.x; c < c0 + kPiece && c < columns; c += blockDim.x) {
                    out[c] = apply_shaped<T>(L.code, operand(L, 0, base[0] + c * L.stride[0][last]),
                                             operand(L, 1, base[1] + c * L.stride[1][last]),
                                             operand(L, 2, base[2] + c * L.stride[2][last]));
                }
            }
        }

        // Rows in 16-byte vectors, two per thread per piece, whatever the row length and the arrays'
        // alignment: a row's vectors start at the first element that lies on a 16-byte boundary of
        // the output, and the few elements before and after them are done one by one. An
        // operand read along the last axis is loaded as a vector where its row lies on the same
        // boundary (every operand of the output's shape does, in arrays that are 16-byte aligned),
        // else by elements, which a warp still reads as whole lines; an operand broadcast
        // along the last axis is one value per row. The code is a template argument, and so is EVEN: rows of
        // whole vectors in aligned arrays, whose kernel has no ends to look for. A block steps from
        // piece to piece by adding, not dividing (the 64-bit division, once per two vectors, was a
        // fifth of the time of the operations that only write). Bound by HBM; at 5001 x 7003 floats, where
        // rows that are not whole vectors went element by element, and at 16384 x 16384 (one call, events
        // around it): where((r, 1), x, y) 202 -> 104 us and 493 -> 468, x - (r, 1) 184 -> 73 and
        // 400 -> 359, (r, 1) + (1, c) 131 -> 56 and 264 -> 211.
        template <typename T, int CODE, bool EVEN>
        __global__ void __launch_bounds__(256) apply_vectors(const __grid_constant__ ApplyLaunch<T> L) {
            constexpr unsigned V = 16 / sizeof(T), U = kVectorsPerThread;
            const int last = L.rank - 1;
            const unsigned long long columns = L.extent[last], span = 256ull * V * U;
            const unsigned long long chunks = (columns + span - 1) / span;  // at most columns / V vectors after the row's first boundary
            const unsigned long long rows = L.count / columns;
            const unsigned long long row_step = gridDim.x / chunks, chunk_step = gridDim.x - row_step * chunks;
            unsigned long long row = blockIdx.x / chunks, chunk = blockIdx.x - row * chunks;
            for (; row < rows; row += row_step, chunk += chunk_step, row += chunk >= chunks, chunk -= chunk >= chunks ? chunks : 0) {
                unsigned long long rest = row, base[3] = {0, 0, 0};
                for (int axis = last - 1; axis >= 0; --axis) {
                    const unsigned long long above = axis > 0 ? rest / L.extent[axis] : 0;
                    const unsigned long long coordinate = rest - above * L.extent[axis];
                    rest = above;
#pragma unroll
                    for (int k = 0; k < 3; ++k) base[k] += coordinate * L.stride[k][axis];
                }
                T *out = L.output + row * columns;
                // elements before the first boundary of the output
                const unsigned offset = static_cast<unsigned>(reinterpret_cast<uintptr_t>(out) / sizeof(T)) % V;
                const unsigned long long head = EVEN || offset == 0 ? 0 : (V - offset < columns ? V - offset : columns);
                const unsigned long long vectors = (columns - head) / V;
                const unsigned long long first = chunk * (256 * U) + threadIdx.x;
                T v[3][U][V];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const T *from = L.input[k] + base[k];
                    const bool along = L.stride[k][last] != 0;
                    const bool whole = EVEN || reinterpret_cast<uintptr_t>(from + head) % 16 == 0;
                    const T single = (L.input[k] && !along) ? *from : T(0);
#pragma unroll
                    for (unsigned u = 0; u < U; ++u) {
                        const unsigned long long at = first + 256 * u;
                        if (along && at < vectors) {
                            if (whole) {
                                load16(from + head + at * V, v[k][u]);
                            } else {
#pragma unroll
                                for (unsigned e = 0; e < V; ++e) v[k][u][e] = from[head + at * V + e];
                            }
                        } else {
#pragma unroll
                            for (unsigned e = 0; e < V; ++e) v[k][u][e] = single;
                        }
                    }
                }
#pragma unroll
                for (unsigned u = 0; u < U; ++u) {
                    const unsigned long long at = first + 256 * u;
                    if (at >= vectors) continue;
                    T r[V];
#pragma unroll
                    for (unsigned e = 0; e < V; ++e) r[e] = apply_shaped<T>(CODE, v[0][u][e], v[1][u][e], v[2][u][e]);
                    store16(out + head + at * V, r);
                }
                if constexpr (EVEN) continue;
                // the elements before and after the vectors: fewer than 2 V
                const unsigned long long after = columns - head - vectors * V;
                if (chunk == 0 && threadIdx.x < head + after) {
                    const unsigned long long c = threadIdx.x < head ? threadIdx.x : columns - after + (threadIdx.x - head);
                    out[c] = apply_shaped<T>(CODE, operand(L, 0, base[0] + c * L.stride[0][last]),
                                             operand(L, 1, base[1] + c * L.stride[1][last]),
                                             operand(L, 2, base[2] + c * L.stride[2][last]));
                }
            }
        }

        template <typename T, int CODE, bool EVEN> void launch_vectors(Context &ctx, const ApplyLaunch<T> &L) {
            constexpr int V = 16 / sizeof(T);
            const unsigned long long columns = L.extent[L.rank - 1], span = 256ull * V * kVectorsPerThread;
            const unsigned long long pieces = (L.count / columns) * ((columns + span - 1) / span);
            // one wave: as many blocks as stay resident
            const unsigned long long most =
                    1ull * ctx.sms * ctx.blocks_per_sm(reinterpret_cast<const void *>(&apply_vectors<T, CODE, EVEN>), 256, 0);
            apply_vectors<T, CODE, EVEN><<<static_cast<unsigned>(pieces < most ? pieces : most), 256, 0, ctx.stream>>>(L);
        }
        // Rows of whole vectors in aligned arrays: every row starts on a vector.
        template <typename T> bool even(const ApplyLaunch<T> &L) {
            auto aligned = [](const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
            return L.extent[L.rank - 1] % (16 / sizeof(T)) == 0 && aligned(L.output) && aligned(L.input[0]) && aligned(L.input[1]) &&
                   aligned(L.input[2]);
        }
        template <typename T, int CODE> void launch_vectors(Context &ctx, const ApplyLaunch<T> &L) {
            if (even(L)) launch_vectors<T, CODE, true>(ctx, L);
            else launch_vectors<T, CODE, false>(ctx, L);
        }

        template <typename T> void launch_vector_code(Context &ctx, const ApplyLaunch<T> &L) {
            switch (L.code) {
            case SCI_CODE_COPY: launch_vectors<T, SCI_CODE_COPY>(ctx, L); return;
            case SCI_CODE_ADD: launch_vectors<T, SCI_CODE_ADD>(ctx, L); return;
            case SCI_CODE_SUBTRACT: launch_vectors<T, SCI_CODE_SUBTRACT>(ctx, L); return;
            case SCI_CODE_MULTIPLY: launch_vectors<T, SCI_CODE_MULTIPLY>(ctx, L); return;
            case SCI_CODE_DIVIDE: launch_vectors<T, SCI_CODE_DIVIDE>(ctx, L); return;
            case SCI_CODE_MINIMUM: launch_vectors<T, SCI_CODE_MINIMUM>(ctx, L); return;
            case SCI_CODE_MAXIMUM: launch_vectors<T, SCI_CODE_MAXIMUM>(ctx, L); return;
            case SCI_EXTRA_FLOOR: launch_vectors<T, SCI_EXTRA_FLOOR>(ctx, L); return;
            case SCI_EXTRA_CEIL: launch_vectors<T, SCI_EXTRA_CEIL>(ctx, L); return;
            case SCI_EXTRA_ROUND: launch_vectors<T, SCI_EXTRA_ROUND>(ctx, L); return;
            case SCI_EXTRA_POWER: launch_vectors<T, SCI_EXTRA_POWER>(ctx, L); return;
            case SCI_EXTRA_CLIP: launch_vectors<T, SCI_EXTRA_CLIP>(ctx, L); return;
            default: launch_vectors<T, SCI_EXTRA_WHERE>(ctx, L);
            }
        }

        int arity(uint32_t code) {
            switch (code) {
            case SCI_CODE_COPY: case SCI_EXTRA_FLOOR: case SCI_EXTRA_CEIL: case SCI_EXTRA_ROUND: return 1;
            case SCI_CODE_ADD: case SCI_CODE_SUBTRACT: case SCI_CODE_MULTIPLY: case SCI_CODE_DIVIDE:
            case SCI_CODE_MINIMUM: case SCI_CODE_MAXIMUM: case SCI_EXTRA_POWER: return 2;
            case SCI_EXTRA_CLIP: case SCI_EXTRA_WHERE: return 3;
            default: return 0;
            }
        }

        template <typename T>
        int launch_apply(Context &ctx, uint32_t code, int rank, const unsigned long long *extent,
                         const unsigned long long (*stride)[kMaxAxes], const void *const *inputs, int operands, void *output,
                         unsigned long long count) {
            ApplyLaunch<T> L{};
            L.code = static_cast<int>(code);
            L.rank = rank;
            for (int a = 0; a < rank; ++a) L.extent[a] = extent[a];
            for (int k = 0; k < operands; ++k) {
                L.input[k] = static_cast<const T *>(inputs[k]);
                for (int a = 0; a < rank; ++a) L.stride[k][a] = stride[k][a];
            }
            L.output = static_cast<T *>(output);
            L.count = count;
            // A block of the row forms steps from row to row, so short rows leave most of it idle. Rows of whole vectors go by
            // vectors from 64 elements on. Ragged ones by a flat index below 288 (where((r, 1), x, y) of 500000 x 127
            // floats: 480 us flat, 970 by rows, 1903 by vectors), from there by vectors (100000 x 385, (r, 1) + (1, c): 185,
            // 256 flat, 213 by rows) -- but three operands by rows below 576 (the same size: 307 by rows, 294 flat, 359
            // by vectors; 40000 x 1023: 150 by vectors, 221 by rows), and powers, which are bound by their arithmetic,
            // by rows below 16384 (20000 x 2049 floats: 497 by rows, 912 by vectors; 30 x 2000003: 695 and 632).
            const unsigned long long columns = extent[rank - 1];
            const unsigned long long most = 8ull * ctx.sms;
            const unsigned long long vectors_from = code == SCI_EXTRA_POWER ? 16384 : (operands == 3 ? 576 : 288);
            if (columns >= 64 && (even(L) || columns >= vectors_from)) {
                launch_vector_code<T>(ctx, L);
            } else if (columns >= 288) {
                const unsigned long long pieces = (count / columns) * ((columns + kPiece - 1) / kPiece);
                apply_rows<T><<<static_cast<unsigned>(pieces < most ? pieces : most), 256, 0, ctx.stream>>>(L);
            } else {
                const unsigned long long wanted = (count + 255) / 256;
                apply_flat<T><<<static_cast<unsigned>(wanted < most ? wanted : most), 256, 0, ctx.stream>>>(L);
            }
            return ctx.check(cudaGetLastError(), "launching a broadcast operation");
        }

    } // namespace
} // namespace sci_cuda

extern "C" int sci_cuda_broadcast(sci_cuda_context *context, uint32_t precision, uint32_t code, uint32_t rank,
                                  const uint64_t *shape, uint32_t operands, const void *const *inputs,
                                  const uint64_t *input_shapes, void *output) {
    if (!context) return SCI_CUDA_ERROR_INVALID;
    std::lock_guard<std::recursive_mutex> lock(context->guard);
    if (precision > SCI_PRECISION_WIDE) return context->fail(SCI_CUDA_ERROR_INVALID, "unknown precision %u", precision);
    if (arity(code) == 0) return context->fail(SCI_CUDA_ERROR_INVALID, "broadcast: unknown code %u", code);
    if (static_cast<int>(operands) != arity(code))
        return context->fail(SCI_CUDA_ERROR_INVALID, "broadcast: code %u takes %d operands, not %u", code, arity(code), operands);
    if (rank < 1 || rank > static_cast<uint32_t>(kMaxAxes) || !shape || !inputs || !input_shapes)
        return context->fail(SCI_CUDA_ERROR_INVALID, "broadcast: rank %u (1 to %d, with shapes)", rank, kMaxAxes);
    unsigned long long count = 1;
    for (uint32_t a = 0; a < rank; ++a) {
        if (shape[a] != 0 && count > ~0ull / shape[a]) return context->fail(SCI_CUDA_ERROR_INVALID, "broadcast: shape overflows");
        count *= shape[a];
    }
    for (uint32_t k = 0; k < operands; ++k)
        for (uint32_t a = 0; a < rank; ++a) {
            const uint64_t e = input_shapes[k * rank + a];
            if (e != shape[a] && e != 1)
                return context->fail(SCI_CUDA_ERROR_INVALID, "broadcast: operand %u axis %u has %llu, not 1 or %llu", k, a,
                                     static_cast<unsigned long long>(e), static_cast<unsigned long long>(shape[a]));
        }
    if (count == 0) return SCI_CUDA_OK;
    if (!output || !reachable(*context, output)) return context->fail(SCI_CUDA_ERROR_INVALID, "broadcast: the output is not memory of this device");
    for (uint32_t k = 0; k < operands; ++k) {
        if (!inputs[k] || !reachable(*context, inputs[k]))
            return context->fail(SCI_CUDA_ERROR_INVALID, "broadcast: operand %u is not memory of this device", k);
        if (inputs[k] == output) {
            // in place only when the operand is read exactly where it is written
            for (uint32_t a = 0; a < rank; ++a)
                if (input_shapes[k * rank + a] != shape[a])
                    return context->fail(SCI_CUDA_ERROR_INVALID, "broadcast: a broadcast operand cannot be the output");
        }
    }
    // Merge adjacent axes that every operand reads alike; drop axes of extent 1.
    unsigned long long extent[kMaxAxes], stride[3][kMaxAxes] = {};
    bool full[3][kMaxAxes];
    int merged = 0;
    for (uint32_t a = 0; a < rank; ++a) {
        if (shape[a] == 1) continue;
        bool same = merged > 0;
        for (uint32_t k = 0; k < operands && same; ++k) same = full[k][merged - 1] == (input_shapes[k * rank + a] != 1);
        if (same) {
            extent[merged - 1] *= shape[a];
        } else {
            extent[merged] = shape[a];
            for (uint32_t k = 0; k < operands; ++k) full[k][merged] = input_shapes[k * rank + a] != 1;
            ++merged;
        }
    }
    if (merged == 0) {
        extent[0] = 1;
        for (uint32_t k = 0; k < operands; ++k) full[k][0] = true;
        merged = 1;
    }
    for (uint32_t k = 0; k < operands; ++k) {
        unsigned long long s = 1;
        for (int a = merged - 1; a >= 0; --a) {
            stride[k][a] = full[k][a] ? s : 0;
            if (full[k][a]) s *= extent[a];
        }
    }
    cudaSetDevice(context->device);
    if (precision == SCI_PRECISION_WIDE)
        return launch_apply<double>(*context, code, merged, extent, stride, inputs, static_cast<int>(operands), output, count);
    return launch_apply<float>(*context, code, merged, extent, stride, inputs, static_cast<int>(operands), output, count);
}
