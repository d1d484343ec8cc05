// small_solve.cu -- the launches of small_solve.cuh.
#include "small_solve.cuh"
#include "small_solve.hpp"

namespace sci_cuda {

    namespace {

        const void *kernel_for(bool single, bool registers) {
            if (single)
                return registers ? reinterpret_cast<const void *>(&small_solve<1, 2>) : reinterpret_cast<const void *>(&small_solve<1, 0>);
            return registers ? reinterpret_cast<const void *>(&small_solve<kSmallGroup, 2>)
                             : reinterpret_cast<const void *>(&small_solve<kSmallGroup, 0>);
        }

        int launch(Context &ctx, cudaStream_t stream, bool single, unsigned most, unsigned blocks, void **args) {
            const bool registers = most > static_cast<unsigned>(kSmallWhole);
            const void *kernel = kernel_for(single, registers);
            const unsigned long long smem =
                    small_shared_bytes(static_cast<int>(most), single ? 1 : static_cast<int>(kSmallGroup), registers ? 2 : 0);
            if (smem > ctx.shared_limit)
                return ctx.fail(SCI_CUDA_ERROR_UNSUPPORTED, "order %u needs %llu bytes of shared memory", most, smem);
            // set on every launch, to the device's limit: other contexts launch the same kernel with other sizes
            if (int code = ctx.check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                          static_cast<int>(small_shared_bytes(
                                                                  registers ? kSmallMax : kSmallWhole,
                                                                  single ? 1 : static_cast<int>(kSmallGroup), registers ? 2 : 0))),
                                     "raising the small solve's shared memory"))
                return code;
            return ctx.check(cudaLaunchKernel(kernel, dim3(blocks), dim3((most + 31) / 32 * 32), args, smem, stream),
                             "launching small solves");
        }

    } // namespace

    int small_solve_table(Context &ctx, cudaStream_t stream, const SmallSystem *systems, const unsigned *order,
                          unsigned count, unsigned most, double target, double *errors, int *iterations) {
        SmallCall none{};
        void *args[] = {&systems, &order, &none, &target, &errors, &iterations};
        return launch(ctx, stream, true, most, count, args);
    }

    unsigned small_solve_blocks(unsigned long long width, bool transposed) {
        const unsigned long long group = width == 1 ? 1 : kSmallGroup;
        return static_cast<unsigned>((width + group - 1) / group * (transposed ? 2 : 1));
    }

    int small_solve_call(Context &ctx, const double *a, const double *b, double *x, const double *b_transposed,
                         double *x_transposed, unsigned long long n, unsigned long long width, double target,
                         double *errors, int *iterations) {
        const unsigned blocks = small_solve_blocks(width, b_transposed != nullptr);
        SmallCall call{a, b, b_transposed, x, x_transposed, static_cast<unsigned>(n), static_cast<unsigned>(width),
                       width == 1 ? 1u : kSmallGroup, small_solve_blocks(width, false), ctx.status, ctx.host_status};
        const SmallSystem *systems = nullptr;
        const unsigned *order = nullptr;
        void *args[] = {&systems, &order, &call, &target, &errors, &iterations};
        return launch(ctx, ctx.stream, width == 1, static_cast<unsigned>(n), blocks, args);
    }

} // namespace sci_cuda
