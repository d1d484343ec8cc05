// small_solve.hpp -- launching the one-CTA solves of order 256 or less (small_solve.cuh).
#pragma once

#include "context.hpp"

namespace sci_cuda {

    struct SmallSystem;
    struct SmallCall;

    constexpr unsigned long long kSmallOrder = 256;  // the largest order they take
    constexpr unsigned kSmallGroup = 4;              // right-hand sides of one CTA of a call

    // A table of systems with one right-hand side each (device memory), the CTAs' by `order`; none of
    // them larger than `most`.
    int small_solve_table(Context &ctx, cudaStream_t stream, const SmallSystem *systems, const unsigned *order,
                          unsigned count, unsigned most, double target, double *errors, int *iterations);
    // One call's right-hand sides: X of A X = B (n x width) and, with `b_transposed`, of A^T X = B. Queued on the
    // context's stream; errors / iterations: an entry per CTA (small_solve_blocks), pinned host memory. A CTA's iteration
    // count is written last, after its part of X and, by the first, the status word in host_status.
    unsigned small_solve_blocks(unsigned long long width, bool transposed);
    int small_solve_call(Context &ctx, const double *a, const double *b, double *x, const double *b_transposed,
                         double *x_transposed, unsigned long long n, unsigned long long width, double target,
                         double *errors, int *iterations);

} // namespace sci_cuda
