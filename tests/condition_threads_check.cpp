// Trace conditioning by several engines at once, a thread each (see
// tests/test_gpu_condition_threads.py): every call must launch, and the last
// one of each thread must leave the samples of its first, made alone.  Prints
// the calls that failed and the threads whose samples differ.
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "psdm_rtm.h"

int main(int argc, char** argv) {
    // shared memory above the default limit of 48 KB, up to the form's 96 KB
    const int sizes[] = {2049, 4095, 2600, 3700, 2100, 4000, 3000, 3500}, nthreads = 8, calls = atoi(argv[1]);
    std::atomic<int> failed{0}, differ{0}, ready{0};
    auto work = [&](int k) {
        const int n = sizes[k], m = 4 * n, zero = 0, lens[4] = {m, m, 10, 0};
        std::vector<float> f(n), first(m), last(m);
        for (int i = 0; i < n; ++i) f[i] = std::sin(0.01f * i * (k + 1));
        psdm_engine* e = nullptr;
        float *d_f = nullptr, *d_o = nullptr;
        psdm_conditioning c{};
        bool ok = psdm_engine_create(0, &e) == PSDM_OK && cudaMalloc(&d_f, n * 4) == cudaSuccess &&
                  cudaMalloc(&d_o, m * 4) == cudaSuccess &&
                  cudaMemcpy(d_f, f.data(), n * 4, cudaMemcpyHostToDevice) == cudaSuccess;
        auto call = [&] {
            return psdm_condition_traces_device(e, &c, 1, d_f, n, 2e-3f, 5e-4f, &m, &zero, lens, d_o) == PSDM_OK;
        };
        auto fetch = [&](std::vector<float>& to) {
            return cudaDeviceSynchronize() == cudaSuccess &&
                   cudaMemcpy(to.data(), d_o, m * 4, cudaMemcpyDeviceToHost) == cudaSuccess;
        };
        while (ready.load() != k) std::this_thread::yield();  // the first calls one after another
        ok = ok && call() && fetch(first);
        ++ready;
        if (!ok) ++failed;
        while (ready.load() < nthreads) std::this_thread::yield();
        for (int i = 0; ok && i < calls; ++i)
            if (!call()) {
                if (failed++ == 0) printf("%d samples: %s\n", n, psdm_last_error());
            }
        if (ok && (!fetch(last) || std::memcmp(first.data(), last.data(), m * 4) != 0)) ++differ;
        psdm_engine_destroy(e);
        cudaFree(d_f);
        cudaFree(d_o);
    };
    std::vector<std::thread> threads;
    for (int k = 0; k < nthreads; ++k) threads.emplace_back(work, k);
    for (auto& t : threads) t.join();
    printf("%d %d\n", failed.load(), differ.load());
    return 0;
}
