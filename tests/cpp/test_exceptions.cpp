// An allocation of the host that fails within a call on a batch of uneven orders
// (operator new throws, the k-th time it is asked for 4 KB or more): the exception
// leaves the context as it was before the call.  Its later calls run on its own
// stream, report an expired wait, and give the results of a context that saw none.
//
// Prints "ok <calls that threw>", or what went wrong.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "zest_gpu.h"

static bool armed = false;
static long seen = 0, fail_at = 0;

void* operator new(std::size_t n) {
    if (armed && n >= 4096 && ++seen == fail_at) throw std::bad_alloc();
    void* p = std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

namespace {

const std::vector<int> orders{24, 24, 24, 40, 40, 40};
std::vector<double> coeffs, euler;
std::size_t grid_size = 0;
double *dc = nullptr, *de = nullptr, *dg = nullptr;

void check(bool ok, const char* what, long k) {
    if (ok) return;
    std::printf("%s (failing allocation %ld): %s\n", what, k, zest_gpu_last_error());
    std::exit(1);
}

int call(zest_gpu_context* ctx) {
    cudaMemcpy(dc, coeffs.data(), coeffs.size() * sizeof(double), cudaMemcpyHostToDevice);
    return zest_gpu_zt_rotate_backward_ragged(ctx, 0, 0, 0, orders.size(), orders.data(), dc, de, 0, dg);
}

std::vector<double> grids(zest_gpu_context* ctx) {
    std::vector<double> g(grid_size);
    zest_gpu_synchronize(ctx);
    cudaMemcpy(g.data(), dg, grid_size * sizeof(double), cudaMemcpyDeviceToHost);
    return g;
}

zest_gpu_context* context(int precision, cudaStream_t s) {
    zest_gpu_context* ctx = nullptr;
    check(zest_gpu_ctx_create(&ctx, 0, s) == 0 && zest_gpu_set_precision(ctx, precision, 0) == 0 &&
              zest_gpu_set_autotune(ctx, 0) == 0,
          "context", 0);
    return ctx;
}

}  // namespace

int main() {
    std::size_t nc = 0;
    for (int L : orders) {
        nc += 2 * zest_gpu_zt_coeff_size(L);
        grid_size += zest_gpu_zt_grid_size(L);
    }
    unsigned x = 1;
    auto next = [&] { return double((x = x * 1664525u + 1013904223u) >> 8) / (1 << 24) - 0.5; };
    for (std::size_t i = 0; i < nc; ++i) coeffs.push_back(next());
    for (std::size_t i = 0; i < 3 * orders.size(); ++i) euler.push_back(next());
    check(cudaMalloc(&dc, nc * sizeof(double)) == cudaSuccess && cudaMalloc(&de, euler.size() * sizeof(double)) == cudaSuccess &&
              cudaMalloc(&dg, grid_size * sizeof(double)) == cudaSuccess,
          "device memory", 0);
    cudaMemcpy(de, euler.data(), euler.size() * sizeof(double), cudaMemcpyHostToDevice);
    cudaStream_t s;
    check(cudaStreamCreate(&s) == cudaSuccess, "stream", 0);
    long thrown = 0;
    for (int precision = 0; precision < 2; ++precision) {
        zest_gpu_context* first = context(precision, s);
        check(call(first) == 0, "the call", 0);
        const std::vector<double> want = grids(first);
        zest_gpu_ctx_destroy(first);
        for (long k = 1;; ++k) {
            zest_gpu_context* ctx = context(precision, s);
            cudaDeviceSynchronize();
            bool threw = false;
            int rc = 0;
            seen = 0;
            fail_at = k;
            armed = true;
            try {
                rc = call(ctx);
            } catch (const std::bad_alloc&) {
                threw = true;
            }
            armed = false;
            check(rc == 0, "the call", k);
            if (threw) {
                ++thrown;
                check(zest_gpu_selftest_wait_timeout(ctx, 0.001) == ZEST_GPU_ERR_TIMEOUT, "an expired wait is not reported", k);
                for (int again = 0; again < 2; ++again) {
                    check(call(ctx) == 0, "a later call", k);
                    check(cudaStreamSynchronize(s) == cudaSuccess, "the stream", k);
                    check(grids(ctx) == want, "a later call's results", k);
                }
            }
            zest_gpu_ctx_destroy(ctx);
            if (!threw) break;
        }
    }
    std::printf("ok %ld\n", thrown);
    return 0;
}
