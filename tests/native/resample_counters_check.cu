// The systematic resampler's block counters after calls that overlapped: whatever
// they hold, the first call may be wrong (as the overlapping ones are), but it leaves
// them at zero, so the next call is right.  Uses the launcher behind the C ABI, with
// counters of its own.
#include <stdio.h>
#include <string.h>

#include <random>
#include <vector>

#include "tsdfl_internal.h"

using namespace tsdfl;

static int fails = 0;
#define CUDA(x)                                                              \
    do {                                                                     \
        const cudaError_t e_ = (x);                                          \
        if (e_ != cudaSuccess) {                                             \
            printf("%s: %s\n", #x, cudaGetErrorString(e_));                  \
            return 2;                                                        \
        }                                                                    \
    } while (0)

int main()
{
    const size_t most = 70'000, cap = 2 * most;
    std::mt19937 g(3);
    for (int tiny = 0; tiny < 2; ++tiny)   // the exact path, and the serial sums' path
        for (size_t M : {(size_t)5, (size_t)257, (size_t)2049, most}) {
            std::vector<float> w(M);
            double sum = 0;
            for (float& v : w) sum += v = (float)(1 + g() % 1000);
            for (float& v : w) v = (float)(v / sum);
            if (tiny) w[M / 2] = 1e-25f;
            const size_t bytes = resample_workspace_bytes(M);
            float* d_w;
            char* d_ws;
            uint32_t *d_idx, *d_count, *d_done;
            int32_t* d_status;
            CUDA(cudaMalloc(&d_w, 4 * M));
            CUDA(cudaMalloc(&d_ws, bytes));
            CUDA(cudaMalloc(&d_idx, 4 * cap));
            CUDA(cudaMalloc(&d_count, 4));
            CUDA(cudaMalloc(&d_done, 8));
            CUDA(cudaMalloc(&d_status, 4));
            CUDA(cudaMemcpy(d_w, w.data(), 4 * M, cudaMemcpyHostToDevice));
            std::vector<uint32_t> want(cap), got(cap);
            uint32_t n_want = 0, n_got = 0;
            auto call = [&](std::vector<uint32_t>& idx, uint32_t& n) {
                CUDA(cudaMemset(d_ws, 0, bytes));
                CUDA(cudaMemset(d_idx, 0xff, 4 * cap));
                CUDA(cudaMemset(d_status, 0, 4));
                if (launch_resample_impl(nullptr, d_w, 1, M, 0.3f / (float)M, nullptr, d_idx, cap, d_count, d_ws,
                                         d_done, d_status, nullptr)) {
                    printf("launch failed\n");
                    return 2;
                }
                CUDA(cudaDeviceSynchronize());
                CUDA(cudaMemcpy(idx.data(), d_idx, 4 * cap, cudaMemcpyDeviceToHost));
                CUDA(cudaMemcpy(&n, d_count, 4, cudaMemcpyDeviceToHost));
                return 0;
            };
            CUDA(cudaMemset(d_done, 0, 8));
            if (call(want, n_want)) return 2;
            if (n_want < M - M / 8 - 1 || n_want > M + M / 8 + 1) ++fails;
            for (uint32_t left : {1u, 2u, 77u}) {
                const uint32_t set[2] = {left, left + 1};
                CUDA(cudaMemcpy(d_done, set, 8, cudaMemcpyHostToDevice));
                if (call(got, n_got)) return 2;   // may be wrong
                uint32_t now[2];
                CUDA(cudaMemcpy(now, d_done, 8, cudaMemcpyDeviceToHost));
                if (now[0] || now[1]) {
                    printf("M %zu tiny %d: counters %u %u after the call\n", M, tiny, now[0], now[1]);
                    ++fails;
                }
                if (call(got, n_got)) return 2;
                if (n_got != n_want || memcmp(got.data(), want.data(), 4 * cap)) {
                    printf("M %zu tiny %d: %u indices, not %u\n", M, tiny, n_got, n_want);
                    ++fails;
                }
            }
            for (void* p : {(void*)d_w, (void*)d_ws, (void*)d_idx, (void*)d_count, (void*)d_done, (void*)d_status})
                cudaFree(p);
        }
    printf("fails %d\n", fails);
    return fails != 0;
}
