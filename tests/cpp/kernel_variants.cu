// Internal launches of the engine on prepared inputs: `kernel_variants SECTION` prints one
// line per check, "ok ..." or "FAIL ...".
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <string>
#include <vector>

#include "qk_kernels.h"

static int g_failed = 0;

static void check(bool ok, const std::string &what) {
    std::printf("%s %s\n", ok ? "ok" : "FAIL", what.c_str());
    g_failed += !ok;
}

#define CUDA(call)                                                                    \
    do {                                                                              \
        const cudaError_t e_ = (call);                                                \
        if (e_ != cudaSuccess) {                                                      \
            std::printf("FAIL %s: %s\n", #call, cudaGetErrorString(e_));              \
            std::exit(1);                                                             \
        }                                                                             \
    } while (0)

template <class T>
struct Dev {
    T *p = nullptr;
    explicit Dev(size_t n) { CUDA(cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T))); }
    Dev(const std::vector<T> &v) : Dev(v.size()) { CUDA(cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice)); }
    ~Dev() { cudaFree(p); }
    std::vector<T> host(size_t n) const {
        std::vector<T> v(n);
        CUDA(cudaMemcpy(v.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost));
        return v;
    }
};

// ---------------------------------------------------------------- order statistics
// Sixteen ranks, neighbours among them, so that many share their prefix down to the last
// digit and a rank's reduced value falls among other lanes' bins.
static void section_select() {
    std::mt19937_64 g(5);
    for (const int64_t n : {1, 2, 16, 255, 256, 257, 4096, 70001, 200000}) {
        for (int kind = 0; kind < 4; ++kind) {
            std::vector<double> x(n);
            for (int64_t i = 0; i < n; ++i) {
                const double u = std::uniform_real_distribution<double>(-1.0, 1.0)(g);
                switch (kind) {
                    case 0: x[i] = u * std::exp2(200.0 * u); break;                            // every exponent and sign
                    case 1: x[i] = std::floor(4.0 * u); break;                                  // few values
                    case 2: x[i] = std::ldexp(4503599627370496.0 + static_cast<double>(g() % 700), -52); break;  // neighbouring bit patterns
                    default:
                        x[i] = g() % 3 ? 5e-324 * static_cast<double>(g() % 300)
                                       : (u > 0 ? HUGE_VAL : -HUGE_VAL);                        // subnormals, infinities
                }
            }
            qk::SelectRanks ranks = {};
            for (int r = 0; r < qk::kSelectRanks; ++r)
                ranks.r[r] = static_cast<unsigned long long>(r < 8 ? std::min<int64_t>(n - 1, n / 3 + r) : (n - 1) * (r - 7) / 8);
            std::sort(ranks.r, ranks.r + qk::kSelectRanks);
            Dev<double> dx(x), out(qk::kSelectRanks);
            Dev<char> scratch(qk::select_scratch_bytes());
            CUDA(qk::launch_select(nullptr, 148, dx.p, n, ranks, qk::kSelectRanks, scratch.p, out.p));
            CUDA(cudaDeviceSynchronize());
            const std::vector<double> got = out.host(qk::kSelectRanks);
            std::sort(x.begin(), x.end());
            bool same = true;
            for (int r = 0; r < qk::kSelectRanks; ++r) same &= got[r] == x[ranks.r[r]];
            check(same, "select n " + std::to_string(n) + " kind " + std::to_string(kind));
        }
    }
}

int main(int argc, char **argv) {
    const std::string section = argc > 1 ? argv[1] : "";
    if (section == "select") section_select();
    else check(false, "unknown section " + section);
    return g_failed != 0;
}
