// small_solve.cuh -- systems of order 256 or less, one CTA per system (and group of right-hand sides).
//
// A system (double operands) is factored in FP32 and refined in FP64 inside one CTA; nothing but its
// matrix, right-hand sides and solution is in global memory. The CTA has a thread per row (32 threads
// for each 32 rows), and a row stays where it was loaded, in its own row of shared memory, from the
// load to the last substitution: a pivot exchange only changes the row's `place` (its position under
// the reference's row exchanges), no value moves. The rows' pitch is an odd multiple of 16 bytes, so
// eight rows' 16-byte pieces fall on all 32 banks. A system of more than kSmallWhole rows does not
// fit; the entries of its last two 32-column blocks stay in the registers of the rows' threads.
//
// Factorisation, by 32-column blocks, left-looking: every earlier block K is applied to the block, and
// the block is factored column by column.
//  - applying block K: the 32 rows placed in it are published (shared memory); U_K = L_KK^-1 W_K by
//    substitution, a column per lane of one warp; every row below subtracts L[row, K] U_K. A warp holds its 32
//    rows' entries of the block as tiles of 4 rows x 8 columns per lane through all K (a row per
//    lane reads 33 values for 32 multiplications, and shared memory returns a quarter of what the
//    multipliers consume: 6.3 thousand cycles a step at order 256; the tile reads 12 for 32), a pair of columns per FMA
//    instruction. Two barriers.
//  - a column: two rows per thread, their entries of the block in registers. Each warp finds its largest
//    |value| (the lowest place among equals: the first row with the strictly largest |a|,
//    include/linear/decompose.hpp:29-72; a zero pivot skips the column's elimination); after a barrier
//    every warp knows the pivot, its thread publishes the row, and after another every thread eliminates.
// Inverses of the blocks' triangles in place of the substitutions, here and in the refinement, lost accuracy:
// systems of order 48 and condition 1e6 took 4.9 corrections instead of 4.0.
// Refinement: x = 0, r = b; repeat { d = U^-1 L^-1 P r in FP32; x += d; r = b - A x in FP64 } until the
// normwise backward error |r|_inf / (|A|_inf |x|_inf + |b|_inf) is at most `target` or stops halving
// (at most 30 corrections): the rule of sci_cuda_solve's refinement (a column of zeros counts as solved). A
// substitution step is a block's triangle by one warp and an update of the other rows from their own L or U.
//
// What bounds it: the chain of columns (700 cycles each at order 128, 790 at 256: two barriers, a
// warp-wide maximum and vote, four trips through shared memory) and of barriers; systems of order 152
// or less run several to an SM and fill each other's gaps. 4096 systems with orders uniform in
// [8, 256]: 2.94 ms, where a column by column elimination in shared memory (about 3900 cycles a
// column at 256) took 11.8 ms. One wave of 148 systems of order 64 / 128 / 256: 41 / 101 / 254 us.
#pragma once

#include "chunk_kernel.cuh"  // static_for

namespace sci_cuda {

    struct SmallSystem {
        const double *a;  // n x n, row-major
        const double *b;  // n rows of right-hand sides, `pitch` apart
        double *x;        // laid out as b
        unsigned n;
        unsigned pitch;
        unsigned columns;     // right-hand sides from b on that this CTA solves (at most the kernel's NR)
        unsigned transposed;  // solve A^T x = b
    };

    constexpr int kSmallMax = 256;        // largest order
    constexpr int kSmallWhole = 224;      // largest order whose factors lie in shared memory whole
    constexpr int kSmallShared = 192;     // columns kept in shared memory beyond it (the other two blocks in registers)
    constexpr int kSmallPitch = 36;       // floats between the rows of a 32 x 32 block apart from the matrix

    // Floats between the matrix's rows: its columns, up to an odd number of 16-byte pieces.
    __host__ __device__ inline int small_pitch(int n, int register_blocks) {
        return 4 * (((register_blocks > 0 ? kSmallShared : n) + 3) / 4 | 1);
    }

    // Dynamic shared memory of one launch for systems up to order `most`.
    inline unsigned long long small_shared_bytes(int most, int right_sides, int register_blocks) {
        unsigned long long bytes = 4ull * most * small_pitch(most, register_blocks);  // factors
        bytes += 2ull * 32 * kSmallPitch * 4;                    // published blocks (later: products with x)
        bytes += 4ull * register_blocks * 32 * kSmallPitch;      // triangles of register blocks
        bytes += 8ull * most * right_sides;                      // x
        bytes += 2ull * 2 * most;                                // rows by position, positions by row
        return (bytes + 15) / 16 * 16;
    }

    __device__ __forceinline__ unsigned long long small_pair(float lo, float hi) {
        unsigned long long out;
        asm("mov.b64 %0, {%1, %2};" : "=l"(out) : "f"(lo), "f"(hi));
        return out;
    }
    __device__ __forceinline__ void small_unpair(unsigned long long v, float &lo, float &hi) {
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    }
    // (lo, hi) += f * (u, v), each lane rounded once
    __device__ __forceinline__ void small_fma_pair(float &lo, float &hi, unsigned long long f, float u, float v) {
        unsigned long long out;
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(out) : "l"(f), "l"(small_pair(u, v)), "l"(small_pair(lo, hi)));
        small_unpair(out, lo, hi);
    }

    // Predicated stores to shared memory (two words, a 16-byte piece): no branch around them.
    __device__ __forceinline__ void small_store_if(bool yes, void *to, unsigned a, unsigned b) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.v2.u32 [%1], {%2, %3};\n\t}" ::"r"(yes ? 1u : 0u),
                     "r"(smem_address(to)), "r"(a), "r"(b)
                     : "memory");
    }
    __device__ __forceinline__ void small_store_if(bool yes, void *to, float a, float b, float c, float d) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.v4.f32 [%1], {%2, %3, %4, %5};\n\t}" ::"r"(
                             yes ? 1u : 0u),
                     "r"(smem_address(to)), "f"(a), "f"(b), "f"(c), "f"(d)
                     : "memory");
    }

    __device__ __forceinline__ double small_larger(double v, double m) { return (v > m || v != v) ? v : m; }  // NaN wins

    // Division by a value that is known before the dividends: its reciprocal by a step of Newton's iteration on the approximate
    // one, and the quotient corrected by its remainder (Markstein, Computation of elementary functions on the IBM RISC
    // System/6000, 1990): equal to the rounded division in 2^33 random trials without denormal intermediates.
    // `scale` keeps these in range; an infinite value divides by 1 and multiplies by 0. The division itself
    // waits for the pivot's row: 291 us instead of 247 for 4096 systems of order 33 to 64 (238 uncorrected).
    struct Divisor {
        float scale, reciprocal, scaled;
    };
    __device__ __forceinline__ Divisor divisor_of(float value) {
        const float size = fabsf(value);
        const float scale = size < 0x1p-96f ? 0x1p96f : (size > 0x1p96f ? 0x1p-96f : 1.0f);
        const float scaled = value * scale, guess = __fdividef(1.0f, scaled);
        const bool infinite = size == INFINITY;
        return Divisor{scale, infinite || size == 0.0f ? guess : fmaf(guess, fmaf(-scaled, guess, 1.0f), guess), infinite ? 1.0f : scaled};
    }
    __device__ __forceinline__ float quotient_of(float dividend, const Divisor &d) {
        const float x = dividend * d.scale, about = x * d.reciprocal;
        return fmaf(fmaf(-about, d.scaled, x), d.reciprocal, about);
    }

    // Sums M values of every lane over the warp, M a power of two up to 8: lanes exchange halves of the
    // values while they can, so value m's sum ends in the lanes whose top bits spell m.
    template <int M> __device__ __forceinline__ double small_warp_sums(double (&s)[M], int lane, int &which) {
        which = 0;
        int offset = 16;
#pragma unroll
        for (int half = M / 2; half > 0; half /= 2, offset /= 2) {
            const bool upper = (lane & offset) != 0;
#pragma unroll
            for (int m = 0; m < half; ++m) {
                const double send = upper ? s[m] : s[m + half];
                const double keep = upper ? s[m + half] : s[m];
                s[m] = keep + __shfl_xor_sync(0xffffffffu, send, offset);
            }
            which += upper ? half : 0;
        }
        double total = s[0];
#pragma unroll
        for (; offset > 0; offset /= 2) total += __shfl_xor_sync(0xffffffffu, total, offset);
        return total;
    }

    // One call's right-hand sides, `group` of them per CTA: CTAs [0, groups) solve A x = b, and with
    // `b_transposed` CTAs [groups, 2 groups) solve A^T x = b_transposed.
    struct SmallCall {
        const double *a, *b, *b_transposed;
        double *x, *x_transposed;
        unsigned n, width, group, groups;
        const int *status;  // the context's error word, and where the first CTA copies it for the host (or null)
        int *host_status;
        __device__ __forceinline__ SmallSystem system(unsigned block) const {
            const bool flip = block >= groups;
            const unsigned first = (flip ? block - groups : block) * group;
            return SmallSystem{a, (flip ? b_transposed : b) + first, (flip ? x_transposed : x) + first, n, width,
                               width - first < group ? width - first : group, flip ? 1u : 0u};
        }
    };

    // NR: right-hand sides of a CTA. RB: 32-column blocks in registers (0, or 2 for n > kSmallWhole). The systems
    // come from a table in device memory, the CTA's by `order`, or from `call` when there is no table.
    template <int NR, int RB>
    __global__ void __maxnreg__(RB > 0 ? 255 : 168)
            small_solve(const SmallSystem *systems, const unsigned *order, const __grid_constant__ SmallCall call,
                        double target, double *errors, int *iterations) {
        constexpr int kWarps = kSmallMax / 32;
        constexpr unsigned kAll = 0xffffffffu;
        __shared__ __align__(16) float pivot_rows[2][32];      // the pivot's row of the block, by column parity
        __shared__ __align__(16) float4 divisors[2];           // the pivot as a Divisor
        __shared__ __align__(16) uint2 best[kWarps];           // each warp's largest key (0: no row left) and its place
        __shared__ __align__(16) float to_solve[32 * NR], solved[32 * NR];  // a substitution step's block, in and out
        __shared__ double maxima[kWarps][2 * NR];
        extern __shared__ __align__(16) unsigned char small_shared[];

        const unsigned id = order ? order[blockIdx.x] : blockIdx.x;
        const SmallSystem sys = systems ? systems[id] : call.system(blockIdx.x);
        const int n = static_cast<int>(sys.n), nb = (n + 31) / 32, P = small_pitch(n, RB);
        const int SB = RB > 0 ? kSmallShared / 32 : nb;        // blocks in shared memory
        const int columns = RB > 0 ? kSmallShared : (n + 3) / 4 * 4;  // columns there, zeros beyond n
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
        const bool row = tid < n;
        const double *a = sys.a;

        float *A = reinterpret_cast<float *>(small_shared);
        unsigned char *cursor = small_shared + 4ull * n * P;
        float *published = reinterpret_cast<float *>(cursor);  // the block's rows as they were
        float *u_block = published + 32 * kSmallPitch;         // and as rows of U
        double *sums = reinterpret_cast<double *>(cursor);     // the rows' products with x, once the factors are done
        cursor += 2ull * 32 * kSmallPitch * 4;
        float *triangles = reinterpret_cast<float *>(cursor);
        cursor += 4ull * RB * 32 * kSmallPitch;
        double *x = reinterpret_cast<double *>(cursor);
        unsigned short *rows = reinterpret_cast<unsigned short *>(x + n * NR);  // the row at each position
        unsigned short *places = rows + n;                                      // each row's place
        float *own = A + tid * P;
        auto vector = [](float *p) -> float4 & { return *reinterpret_cast<float4 *>(p); };

        // ---- load A in FP32, with |A|_inf
        float held[RB > 0 ? RB : 1][32];
        double norm = 0.0;  // the largest row sum this thread saw
        if (sys.transposed) {
            // row t of A^T is column t of A: a thread's loads are a warp's consecutive columns
            if (row) {
                const int stored = RB > 0 ? kSmallShared : n;
#pragma unroll 16
                for (int c = 0; c < stored; ++c) {
                    const double v = a[1ll * c * n + tid];
                    own[c] = static_cast<float>(v);
                    norm += fabs(v);
                }
                for (int c = stored; c < columns; ++c) own[c] = 0.0f;
                if constexpr (RB > 0) {
#pragma unroll
                    for (int q = 0; q < RB; ++q)
#pragma unroll
                        for (int c = 0; c < 32; ++c) {
                            const int at = kSmallShared + 32 * q + c;
                            const double v = at < n ? a[1ll * at * n + tid] : 0.0;
                            held[q][c] = static_cast<float>(v);
                            norm += fabs(v);
                        }
                }
            }
        } else {
            // a warp per row, the loads of several rows in flight: G pieces of 32 columns each
            auto load = [&](auto g_c) {
                constexpr int G = decltype(g_c)::value, R = G <= 4 ? 8 : 4;
                for (int row0 = warp; row0 < n; row0 += R * warps) {
                    double v[R][G], sum[R];
#pragma unroll
                    for (int u = 0; u < R; ++u)
#pragma unroll
                        for (int g = 0; g < G; ++g) {
                            const int at = row0 + u * warps, c = lane + 32 * g;
                            v[u][g] = at < n && c < n ? a[1ll * at * n + c] : 0.0;
                        }
#pragma unroll
                    for (int u = 0; u < R; ++u) {
                        const int at = row0 + u * warps;
                        sum[u] = 0.0;
#pragma unroll
                        for (int g = 0; g < G; ++g) {
                            const int c = lane + 32 * g;
                            if (at < n && c < columns) A[at * P + c] = static_cast<float>(v[u][g]);
                            sum[u] += fabs(v[u][g]);
                        }
                    }
                    int which;
                    norm = small_larger(small_warp_sums<R>(sum, lane, which), norm);
                }
            };
            if (nb == 1) load(Int<1>{});
            else if (nb == 2) load(Int<2>{});
            else if (nb <= 4) load(Int<4>{});
            else load(Int<8>{});
            if constexpr (RB > 0) {
#pragma unroll
                for (int q = 0; q < RB; ++q)
#pragma unroll
                    for (int c = 0; c < 32; ++c) {
                        const int at = kSmallShared + 32 * q + c;
                        held[q][c] = row && at < n ? static_cast<float>(a[1ll * tid * n + at]) : 0.0f;
                    }
            }
        }
        double rhs[NR], b_norm[NR], a_norm = 0.0;  // this thread's row of b, then |b_q|_inf and |A|_inf
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            rhs[q] = row && q < static_cast<int>(sys.columns) ? sys.b[1ull * tid * sys.pitch + q] : 0.0;
            b_norm[q] = fabs(rhs[q]);
        }
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) {
            norm = small_larger(__shfl_xor_sync(kAll, norm, offset), norm);
#pragma unroll
            for (int q = 0; q < NR; ++q) b_norm[q] = small_larger(__shfl_xor_sync(kAll, b_norm[q], offset), b_norm[q]);
        }
        if (lane == 0) {
            maxima[warp][0] = norm;
#pragma unroll
            for (int q = 0; q < NR; ++q) maxima[warp][NR + q] = b_norm[q];
        }
        if (row) {
            places[tid] = static_cast<unsigned short>(tid);
#pragma unroll
            for (int q = 0; q < NR; ++q) x[tid * NR + q] = 0.0;
        }
        for (int i = tid; i < 32 * NR; i += blockDim.x) to_solve[i] = 0.0f;
        if (tid < kWarps) best[tid] = make_uint2(0u, ~0u);
        __syncthreads();
        for (int w = 0; w < warps; ++w) {
            a_norm = small_larger(maxima[w][0], a_norm);
#pragma unroll
            for (int q = 0; q < NR; ++q) b_norm[q] = small_larger(maxima[w][NR + q], b_norm[q]);
        }

        // ---- LU with partial pivoting
        int place = row ? tid : kSmallMax;
        // row i of block K's triangles: L's strictly below the diagonal, U's on and above it
        auto triangle_row = [&](int K, int i) -> float * {
            if (RB > 0 && K >= SB) return triangles + ((K - SB) * 32 + i) * kSmallPitch;
            return A + rows[32 * K + i] * P + 32 * K;
        };
        // U_K = L_KK^-1 W_K by substitution, a column per lane of one warp
        auto substitute = [&](int K) {
            if (warp == 0) {
                float v[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = published[i * kSmallPitch + lane];
                static_for<32>([&](auto i_c) {
                    constexpr int i = decltype(i_c)::value;
                    float *l = triangle_row(K, i);
#pragma unroll
                    for (int k = 0; k < i; k += 4) {
                        const float4 q = vector(l + k);
                        v[i] = fmaf(-q.x, v[k], v[i]);
                        if (k + 1 < i) v[i] = fmaf(-q.y, v[k + 1], v[i]);
                        if (k + 2 < i) v[i] = fmaf(-q.z, v[k + 2], v[i]);
                        if (k + 3 < i) v[i] = fmaf(-q.w, v[k + 3], v[i]);
                    }
                });
#pragma unroll
                for (int i = 0; i < 32; ++i) u_block[i * kSmallPitch + lane] = v[i];
            }
        };
        // The columns of a block, R rows per thread of `crew` warps: w[h][0] is the next column, and the registers move
        // down by one as it is eliminated (zeros come in at the top, so a row's registers beyond its
        // columns are zeros). `home(h, column, entry)` takes the column's own entry, a multiplier or an
        // entry of U. To keep the chain short
        //  - only the pivot's row is published (a 16-byte store takes shared memory about six cycles however few
        //    lanes store: eight warps' candidate rows took 385), and two rows per thread halve the readers;
        //  - nothing but the loop branches (10 to 20 cycles each): selects and predicated stores, and the number
        //    of 16-byte pieces a row still has is a constant for eight columns at a time. With branches a column
        //    took 1030 cycles at order 128; all 32 columns unrolled took 840, waiting for instructions.
        auto columns_of = [&](auto rows_c, auto alone_c, auto &w, auto &line, auto &spot, int crew, int j0, int bw, auto home) {
            constexpr int R = decltype(rows_c)::value, kCrew = kWarps / R;
            constexpr bool alone = decltype(alone_c)::value != 0;  // a crew of one warp: its maximum is the pivot
            auto meet = [&] {
                if constexpr (alone) __syncwarp();
                else asm volatile("bar.sync 1, %0;" ::"r"(32 * crew) : "memory");
            };
            static_for<4>([&](auto segment_c) {
                constexpr int segment = decltype(segment_c)::value, V = 8 - 2 * segment;
#pragma unroll 1
                for (int j = 8 * segment; j < (bw < 8 * segment + 8 ? bw : 8 * segment + 8); ++j) {
                    const int column = j0 + j;
                    unsigned key[R];
                    bool live[R];
#pragma unroll
                    for (int h = 0; h < R; ++h) {
                        live[h] = line[h] < n && spot[h] >= column;
                        const unsigned bits = __float_as_uint(w[h][0]) & 0x7fffffffu;
                        // |value| + 1; a NaN only stands at the pivot position, where every comparison fails
                        const unsigned ordinary = bits <= 0x7f800000u ? bits + 1u : (spot[h] == column ? ~0u : 0u);
                        key[h] = live[h] ? ordinary : 0u;
                    }
                    const bool second = R > 1 && (key[R - 1] > key[0] || (key[R - 1] == key[0] && spot[R - 1] < spot[0]));
                    const unsigned own_key = second ? key[R - 1] : key[0];
                    const unsigned own_place = static_cast<unsigned>(second ? spot[R - 1] : spot[0]);
                    const float own_value = second ? w[R - 1][0] : w[0][0];
                    const unsigned most = __reduce_max_sync(kAll, own_key);
                    const Divisor own = divisor_of(own_value);  // of use if this row is the pivot's
                    unsigned mine = __ballot_sync(kAll, own_key == most);
                    if (mine & (mine - 1)) {  // equals: the lowest place
                        const unsigned lowest = __reduce_min_sync(kAll, own_key == most ? own_place : ~0u);
                        mine = __ballot_sync(kAll, own_key == most && own_place == lowest);
                    }
                    const bool leads = lane == __ffs(mine) - 1;
                    uint2 top;
                    int from = 0;
                    if constexpr (alone) {
                        top = make_uint2(most, __shfl_sync(kAll, own_place, __ffs(mine) - 1));
                    } else {
                        small_store_if(leads, &best[warp], most, own_place);
                        meet();
                        top = best[0];
#pragma unroll
                        for (int v = 1; v < kCrew; ++v) {
                            const uint2 other = best[v];
                            const bool better = other.x > top.x || (other.x == top.x && other.y < top.y);
                            top.x = better ? other.x : top.x, top.y = better ? other.y : top.y, from = better ? v : from;
                        }
                    }
                    const bool winner = leads && (alone || warp == from);
                    float *pivot = pivot_rows[j & 1];
#pragma unroll
                    for (int h = 0; h < R; ++h) {
                        const bool publishes = winner && second == (h > 0);
#pragma unroll
                        for (int v = 0; v < V; ++v) small_store_if(publishes, pivot + 4 * v, w[h][4 * v], w[h][4 * v + 1], w[h][4 * v + 2], w[h][4 * v + 3]);
                    }
                    small_store_if(winner, &divisors[j & 1], own.scale, own.reciprocal, own.scaled, 0.0f);
                    meet();
                    float4 u[V + 1];
                    u[V] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    const float4 stored = divisors[j & 1];
                    const Divisor divisor{stored.x, stored.y, stored.z};
#pragma unroll
                    for (int v = 0; v < V; ++v) u[v] = vector(pivot + 4 * v);
#pragma unroll
                    for (int h = 0; h < R; ++h) {
                        const bool chosen = winner && second == (h > 0);
                        const bool act = live[h] && !chosen && u[0].x != 0.0f;
                        const float quotient = quotient_of(w[h][0], divisor);
                        const float l = act ? quotient : 0.0f;  // a row that is done multiplies by zero
                        home(h, column, act ? quotient : w[h][0]);
                        spot[h] = chosen ? column : (spot[h] == column ? static_cast<int>(top.y) : spot[h]);
#pragma unroll
                        for (int v = 0; v < V; ++v) {
                            w[h][4 * v] = fmaf(-l, u[v].y, w[h][4 * v + 1]);
                            w[h][4 * v + 1] = fmaf(-l, u[v].z, w[h][4 * v + 2]);
                            w[h][4 * v + 2] = fmaf(-l, u[v].w, w[h][4 * v + 3]);
                            w[h][4 * v + 3] = v < V - 1 ? fmaf(-l, u[v + 1].x, w[h][4 * v + 4 < 32 ? 4 * v + 4 : 0]) : 0.0f;
                        }
                    }
                }
            });
        };
        for (int J = 0; J < nb; ++J) {
            const int j0 = 32 * J, bw = n - j0 < 32 ? n - j0 : 32;
            if (RB > 0 && J >= SB) {
                // a register block: a row per thread
                float held_rows[1][32], (&w)[32] = held_rows[0];
#pragma unroll
                for (int c = 0; c < 32; ++c) w[c] = J == SB ? held[0][c] : held[RB > 1 ? 1 : 0][c];
                for (int K = 0; K < J; ++K) {
                    const int q = place - 32 * K;
                    if (q >= 0 && q < 32) {
#pragma unroll
                        for (int c = 0; c < 32; c += 4) vector(published + q * kSmallPitch + c) = make_float4(w[c], w[c + 1], w[c + 2], w[c + 3]);
                    }
                    __syncthreads();
                    substitute(K);
                    __syncthreads();
                    auto subtract_row = [&](int k, float l) {
                        const unsigned long long f = small_pair(-l, -l);
#pragma unroll
                        for (int c = 0; c < 32; c += 4) {
                            const float4 u = vector(u_block + k * kSmallPitch + c);
                            small_fma_pair(w[c], w[c + 1], f, u.x, u.y);
                            small_fma_pair(w[c + 2], w[c + 3], f, u.z, u.w);
                        }
                    };
                    if (q >= 0 && q < 32) {
#pragma unroll
                        for (int c = 0; c < 32; c += 4) {
                            const float4 u = vector(u_block + q * kSmallPitch + c);
                            w[c] = u.x, w[c + 1] = u.y, w[c + 2] = u.z, w[c + 3] = u.w;
                        }
                    } else if (row && q >= 32) {
                        if (K >= SB) {
#pragma unroll
                            for (int k = 0; k < 32; ++k) subtract_row(k, held[0][k]);  // only the first register block precedes another
                        } else {
#pragma unroll 1
                            for (int k = 0; k < 32; k += 4) {
                                const float4 l = vector(own + 32 * K + k);
                                subtract_row(k, l.x), subtract_row(k + 1, l.y), subtract_row(k + 2, l.z), subtract_row(k + 3, l.w);
                            }
                        }
                    }
                }
                float kept[32];
                const int line[1] = {tid};
                int spot[1] = {place};
                columns_of(Int<1>{}, Int<0>{}, held_rows, line, spot, warps, j0, bw, [&](int, int, float entry) {
#pragma unroll
                    for (int c = 0; c < 31; ++c) kept[c] = kept[c + 1];
                    kept[31] = entry;
                });
                place = spot[0];
                if (row && place >= j0 && place < j0 + bw) rows[place] = static_cast<unsigned short>(tid);
#pragma unroll 1
                for (int j = bw; j < 32; ++j) {
#pragma unroll
                    for (int c = 0; c < 31; ++c) kept[c] = kept[c + 1];
                    kept[31] = 0.0f;
                }
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    if (J == SB) held[0][c] = kept[c];
                    else held[RB > 1 ? 1 : 0][c] = kept[c];
                }
                if (row && place >= j0 && place < j0 + bw) {
#pragma unroll
                    for (int c = 0; c < 32; c += 4)
                        vector(triangle_row(J, place - j0) + c) = make_float4(kept[c], kept[c + 1], kept[c + 2], kept[c + 3]);
                }
            } else {
                if (J > 0) {
                    // tiles of 4 rows (eight apart) x 8 columns per lane
                    const int first = 32 * warp + (lane >> 2), c0 = (lane & 3) * 8;
                    float t[4][8];
                    int at[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int line = first + 8 * i;
                        at[i] = line < n ? places[line] : -1;
#pragma unroll
                        for (int h = 0; h < 8; h += 4) {
                            const float4 v = line < n && j0 + c0 + h < columns ? vector(A + line * P + j0 + c0 + h)
                                                                               : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                            t[i][h] = v.x, t[i][h + 1] = v.y, t[i][h + 2] = v.z, t[i][h + 3] = v.w;
                        }
                    }
                    for (int K = 0; K < J; ++K) {
                        bool below = false;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int q = at[i] - 32 * K;
                            below = below || q >= 32;
                            if (q >= 0 && q < 32) {
#pragma unroll
                                for (int h = 0; h < 8; h += 4)
                                    vector(published + q * kSmallPitch + c0 + h) = make_float4(t[i][h], t[i][h + 1], t[i][h + 2], t[i][h + 3]);
                            }
                        }
                        __syncthreads();
                        substitute(K);
                        __syncthreads();
                        if (__any_sync(kAll, below)) {
#pragma unroll 2
                            for (int k0 = 0; k0 < 32; k0 += 4) {
                                float l[4][4];
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const bool live = at[i] >= 32 * K + 32;  // rows placed in or above the block keep theirs
                                    const float4 v = live ? vector(A + (first + 8 * i) * P + 32 * K + k0)
                                                          : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                                    l[i][0] = -v.x, l[i][1] = -v.y, l[i][2] = -v.z, l[i][3] = -v.w;
                                }
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    const float4 u = vector(u_block + (k0 + e) * kSmallPitch + c0);
                                    const float4 v = vector(u_block + (k0 + e) * kSmallPitch + c0 + 4);
#pragma unroll
                                    for (int i = 0; i < 4; ++i) {
                                        const unsigned long long f = small_pair(l[i][e], l[i][e]);
                                        small_fma_pair(t[i][0], t[i][1], f, u.x, u.y);
                                        small_fma_pair(t[i][2], t[i][3], f, u.z, u.w);
                                        small_fma_pair(t[i][4], t[i][5], f, v.x, v.y);
                                        small_fma_pair(t[i][6], t[i][7], f, v.z, v.w);
                                    }
                                }
                            }
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int q = at[i] - 32 * K;
                            if (q >= 0 && q < 32) {
#pragma unroll
                                for (int h = 0; h < 8; h += 4) {
                                    const float4 u = vector(u_block + q * kSmallPitch + c0 + h);
                                    t[i][h] = u.x, t[i][h + 1] = u.y, t[i][h + 2] = u.z, t[i][h + 3] = u.w;
                                }
                            }
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int h = 0; h < 8; h += 4)
                            if (first + 8 * i < n && j0 + c0 + h < columns)
                                vector(A + (first + 8 * i) * P + j0 + c0 + h) = make_float4(t[i][h], t[i][h + 1], t[i][h + 2], t[i][h + 3]);
                    __syncthreads();
                }
                const int crew = (n + 63) / 64;
                if (warp < crew) {
                    float w[2][32];
                    int line[2], spot[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        line[h] = 64 * warp + 32 * h + lane;
                        spot[h] = line[h] < n ? places[line[h]] : kSmallMax;
#pragma unroll
                        for (int c = 0; c < 32; c += 4) {
                            const float4 v = line[h] < n && j0 + c < columns ? vector(A + line[h] * P + j0 + c)
                                                                             : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                            w[h][c] = v.x, w[h][c + 1] = v.y, w[h][c + 2] = v.z, w[h][c + 3] = v.w;
                        }
                    }
                    auto home = [&](int h, int column, float entry) {
                        if (line[h] < n) A[line[h] * P + column] = entry;
                    };
                    if (crew == 1) columns_of(Int<2>{}, Int<1>{}, w, line, spot, crew, j0, bw, home);
                    else columns_of(Int<2>{}, Int<0>{}, w, line, spot, crew, j0, bw, home);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (line[h] < n) {
                            places[line[h]] = static_cast<unsigned short>(spot[h]);
                            if (spot[h] >= j0 && spot[h] < j0 + bw) rows[spot[h]] = static_cast<unsigned short>(line[h]);
                        }
                }
                __syncthreads();
                if (row) place = places[tid];
            }
        }
        __syncthreads();

        // ---- refinement
        double berr = INFINITY, previous = INFINITY;
        int count = 0;
        float c[NR];
#pragma unroll
        for (int q = 0; q < NR; ++q) c[q] = static_cast<float>(rhs[q]);
        // this row's entries of block K, read ahead of the values they multiply
        auto entries = [&](int K, float (&l)[32]) {
            if (RB > 0 && K >= SB) {
#pragma unroll
                for (int k = 0; k < 32; ++k) l[k] = K == SB ? held[0][k] : held[RB > 1 ? 1 : 0][k];
            } else {
#pragma unroll
                for (int k = 0; k < 32; k += 4) {
                    const float4 v = 32 * K + k < columns ? vector(own + 32 * K + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    l[k] = v.x, l[k + 1] = v.y, l[k + 2] = v.z, l[k + 3] = v.w;
                }
            }
        };
        auto subtract = [&](const float (&l)[32]) {
            if constexpr (NR == 1) {
                float s[2] = {0.0f, 0.0f};
#pragma unroll
                for (int k = 0; k < 32; k += 4) {
                    const float4 v = vector(solved + k);
                    s[0] = fmaf(l[k], v.x, s[0]), s[1] = fmaf(l[k + 1], v.y, s[1]);
                    s[0] = fmaf(l[k + 2], v.z, s[0]), s[1] = fmaf(l[k + 3], v.w, s[1]);
                }
                c[0] -= s[0] + s[1];
            } else {
                static_assert(NR == 1 || NR == 4, "right-hand sides in 16-byte pieces");
#pragma unroll
                for (int k = 0; k < 32; ++k) {
                    const float4 v = vector(solved + k * NR);
                    c[0] = fmaf(-l[k], v.x, c[0]), c[1 % NR] = fmaf(-l[k], v.y, c[1 % NR]);
                    c[2 % NR] = fmaf(-l[k], v.z, c[2 % NR]), c[3 % NR] = fmaf(-l[k], v.w, c[3 % NR]);
                }
            }
        };
        // Block K's right-hand sides by substitution, a row per lane of one warp: four columns at a time, whose own
        // 4 x 4 triangle every lane solves for itself, so that the chain crosses the lanes eight times, not 32. U's rows
        // are divided by their diagonals first. Zeros for lanes beyond the block.
        auto solve_block = [&](int K, int bw, auto lower_c, float (&y)[NR]) {
            constexpr bool lower = decltype(lower_c)::value != 0;
            float *own_line = triangle_row(K, lane < bw ? lane : 0);
            Divisor own{};
            if constexpr (!lower) own = divisor_of(own_line[lane < bw ? lane : 0]);
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                y[q] = lane < bw ? to_solve[lane * NR + q] : 0.0f;
                if constexpr (!lower) y[q] = lane < bw ? quotient_of(y[q], own) : 0.0f;
            }
            const int groups = (bw + 3) / 4;
            float4 next = vector(own_line + (lower ? 0 : 4 * groups - 4));
#pragma unroll 2
            for (int step = 0; step < groups; ++step) {
                const int g = lower ? step : groups - 1 - step;
                float pieces[4] = {next.x, next.y, next.z, next.w};
                if (step + 1 < groups) next = vector(own_line + 4 * (lower ? g + 1 : g - 1));
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    // what lies beyond the triangle, or the block's columns (another row's, or nothing's), counts as zero
                    const int k = 4 * g + e;
                    const bool inside = lower ? k < lane && lane < bw : k > lane && k < bw;
                    if constexpr (lower) pieces[e] = inside ? -pieces[e] : 0.0f;
                    else pieces[e] = inside ? -quotient_of(pieces[e], own) : 0.0f;
                }
                float t[4][NR];
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int q = 0; q < NR; ++q) t[e][q] = __shfl_sync(kAll, y[q], 4 * g + e);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int e = lower ? u : 3 - u;
#pragma unroll
                    for (int f = 0; f < 4; ++f) {
                        if (lower ? f <= e : f >= e) continue;
                        const float entry = __shfl_sync(kAll, pieces[e], 4 * g + f);
#pragma unroll
                        for (int q = 0; q < NR; ++q) t[f][q] = fmaf(entry, t[e][q], t[f][q]);
                    }
#pragma unroll
                    for (int q = 0; q < NR; ++q) y[q] = fmaf(pieces[e], t[e][q], y[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < NR; ++q) y[q] = lane < bw ? y[q] : 0.0f;
        };
        while (true) {
#pragma unroll 1
            for (int K = 0; K < nb; ++K) {
                const int at = place - 32 * K, bw = n - 32 * K < 32 ? n - 32 * K : 32;
                const bool below = row && at >= 32;
                float l[32];
                if (at >= 0 && at < 32) {
#pragma unroll
                    for (int q = 0; q < NR; ++q) to_solve[at * NR + q] = c[q];
                }
                __syncthreads();
                if (below) entries(K, l);
                if (warp == 0) {
                    float y[NR];
                    solve_block(K, bw, Int<1>{}, y);
#pragma unroll
                    for (int q = 0; q < NR; ++q) solved[lane * NR + q] = y[q];
                }
                __syncthreads();
                if (at >= 0 && at < 32) {
#pragma unroll
                    for (int q = 0; q < NR; ++q) c[q] = solved[at * NR + q];
                } else if (below) {
                    subtract(l);
                }
            }
#pragma unroll 1
            for (int K = nb - 1; K >= 0; --K) {
                const int at = place - 32 * K, bw = n - 32 * K < 32 ? n - 32 * K : 32;
                float l[32];
                if (at >= 0 && at < 32) {
#pragma unroll
                    for (int q = 0; q < NR; ++q) to_solve[at * NR + q] = c[q];
                }
                __syncthreads();
                if (at < 0) entries(K, l);  // the rows placed above the block
                if (warp == 0) {
                    float y[NR];
                    solve_block(K, bw, Int<0>{}, y);
#pragma unroll
                    for (int q = 0; q < NR; ++q) {
                        solved[lane * NR + q] = y[q];
                        if (lane < bw) x[(32 * K + lane) * NR + q] += static_cast<double>(y[q]);
                    }
                }
                __syncthreads();
                if (at < 0) subtract(l);
            }
            // r = b - A x in FP64, with |r_q|_inf and |x_q|_inf. The diagonal's term is subtracted from b first, by the row's
            // thread: in diagonally dominant systems they nearly cancel, and what is added to them rounds at the
            // remainder's size (orders 16 to 256, A = G + nI: a mean backward error of 4.8e-17 to 9.6e-17 with
            // the term in the row's sum, 2.1e-17 to 2.4e-17 here).
            double left[NR], r_max[NR], x_max[NR];  // this row's residuals
            const double diagonal = row ? a[1ll * tid * n + tid] : 0.0;
#pragma unroll
            for (int q = 0; q < NR; ++q) left[q] = row ? fma(-diagonal, x[tid * NR + q], rhs[q]) : 0.0;
            if (sys.transposed) {
                // A thread per row, in parts of 16 terms whose sums are added to the total: a rounding error for every 16
                // terms or less, as in the blocked residual (one chain over all terms doubled the error at order 256).
                if (row) {
                    auto part = [&](int k0, auto whole_c) {
                        constexpr bool whole = decltype(whole_c)::value != 0;
                        double v[16], s[NR][2];
#pragma unroll
                        for (int k = 0; k < 16; ++k) v[k] = (whole || k0 + k < n) && k0 + k != tid ? a[1ll * (k0 + k) * n + tid] : 0.0;
#pragma unroll
                        for (int q = 0; q < NR; ++q) s[q][0] = s[q][1] = 0.0;
#pragma unroll
                        for (int k = 0; k < 16; ++k)
#pragma unroll
                            for (int q = 0; q < NR; ++q)
                                s[q][k & 1] = fma(v[k], whole || k0 + k < n ? x[(k0 + k) * NR + q] : 0.0, s[q][k & 1]);
#pragma unroll
                        for (int q = 0; q < NR; ++q) left[q] -= s[q][0] + s[q][1];
                    };
                    int k0 = 0;
#pragma unroll 2
                    for (; k0 + 16 <= n; k0 += 16) part(k0, Int<1>{});
                    if (k0 < n) part(k0, Int<0>{});
                }
            } else {
                // a warp per row, several rows' loads in flight (as the load); R rows' sums of every right-hand side
                auto residual = [&](auto g_c) {
                    constexpr int G = decltype(g_c)::value, R = NR == 1 ? (G <= 4 ? 8 : 4) : 2, M = R * NR;
                    double v[R][G];
                    auto fetch = [&](int row0) {
#pragma unroll
                        for (int u = 0; u < R; ++u)
#pragma unroll
                            for (int g = 0; g < G; ++g) {
                                const int at = row0 + u * warps, col = lane + 32 * g;
                                v[u][g] = at < n && col < n && col != at ? a[1ll * at * n + col] : 0.0;
                            }
                    };
                    fetch(warp);
                    for (int row0 = warp; row0 < n; row0 += R * warps) {
                        double s[M];
#pragma unroll
                        for (int m = 0; m < M; ++m) s[m] = 0.0;
#pragma unroll
                        for (int g = 0; g < G; ++g) {
                            const int col = lane + 32 * g;
#pragma unroll
                            for (int q = 0; q < NR; ++q) {
                                const double value = col < n ? x[col * NR + q] : 0.0;
#pragma unroll
                                for (int u = 0; u < R; ++u) s[u * NR + q] = fma(v[u][g], value, s[u * NR + q]);
                            }
                        }
                        fetch(row0 + R * warps);  // the next rows' loads, in flight during the sums
                        int which;
                        const double total = small_warp_sums<M>(s, lane, which);
                        const int at = row0 + which / NR * warps, q = which % NR;
                        if (at < n && lane % (32 / M) == 0) sums[at * NR + q] = total;
                    }
                };
                if (nb == 1) residual(Int<1>{});
                else if (nb == 2) residual(Int<2>{});
                else if (nb <= 4) residual(Int<4>{});
                else residual(Int<8>{});
                __syncthreads();
                if (row) {
#pragma unroll
                    for (int q = 0; q < NR; ++q) left[q] -= sums[tid * NR + q];
                }
            }
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                r_max[q] = fabs(left[q]);
                x_max[q] = row ? fabs(x[tid * NR + q]) : 0.0;
#pragma unroll
                for (int offset = 16; offset > 0; offset >>= 1) {
                    x_max[q] = small_larger(__shfl_xor_sync(kAll, x_max[q], offset), x_max[q]);
                    r_max[q] = small_larger(__shfl_xor_sync(kAll, r_max[q], offset), r_max[q]);
                }
            }
            if (lane == 0) {
#pragma unroll
                for (int q = 0; q < NR; ++q) maxima[warp][q] = r_max[q], maxima[warp][NR + q] = x_max[q];
            }
            __syncthreads();
            berr = 0.0;
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                double rm = 0.0, xm = 0.0;
                for (int v = 0; v < warps; ++v) rm = small_larger(maxima[v][q], rm), xm = small_larger(maxima[v][NR + q], xm);
                // zero over zero: a right-hand side of zeros with its exact solution, not a NaN that would end
                // the refinement of the other columns
                const double scale = a_norm * xm + b_norm[q];
                const double error = rm == 0.0 && scale == 0.0 ? 0.0 : rm / scale;
                if (q < static_cast<int>(sys.columns)) berr = small_larger(error, berr);
            }
            ++count;
            if (count >= 30 || !(berr > target) || !(berr < 0.5 * previous)) break;
            previous = berr;
#pragma unroll
            for (int q = 0; q < NR; ++q) c[q] = static_cast<float>(left[q]);
        }
        if (row) {
#pragma unroll
            for (int q = 0; q < NR; ++q)
                if (q < static_cast<int>(sys.columns)) sys.x[1ull * tid * sys.pitch + q] = x[tid * NR + q];
        }
        if (call.host_status != nullptr) {
            // the host polls `iterations`: the solution, the error and the status come before it
            __threadfence();
            __syncthreads();
            if (tid == 0 && blockIdx.x == 0) *call.host_status = __ldcg(call.status);
        }
        if (tid == 0) {
            if (errors) errors[id] = berr;
            if (call.host_status != nullptr) __threadfence_system();
            if (iterations) *static_cast<volatile int *>(iterations + id) = count;
        }
    }

} // namespace sci_cuda
