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

#include "qk_engine.h"
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

// ---------------------------------------------------------------- contracts
static qk_payoff leg(int type, int right, double K, double B = 0.0) {
    qk_payoff p{};
    p.type = type;
    p.right = right;
    p.strike = K;
    p.barrier = B;
    return p;
}

static qk_contract contract(int precision, int model, int scheme, int64_t n_paths, int n_steps, std::vector<qk_payoff> legs) {
    qk_contract c{};
    c.S0 = 100.0;
    c.v0 = 0.04;
    c.r = 0.03;
    c.model = model;
    c.scheme = scheme;
    c.kappa = 2.0;
    c.theta = 0.04;
    c.sigma = 0.3;
    c.rho = -0.7;
    c.lambda_j = model == QK_BATES ? 0.4 : 0.0;
    c.mu_j = -0.05;
    c.sigma_j = 0.1;
    c.psi_c = 1.5;
    c.T = n_steps / 252.0;
    c.n_steps = n_steps;
    c.n_paths = n_paths;
    c.seed = 0x1234567890ABull;
    c.precision = precision;
    c.normalize = 1;
    c.n_payoffs = static_cast<int>(legs.size());
    for (size_t i = 0; i < legs.size(); ++i) c.payoffs[i] = legs[i];
    return c;
}

static bool same_legs(const qk_result &a, const qk_result &b, int n) {
    bool same = a.n_payoffs == b.n_payoffs;
    for (int k = 0; k < n; ++k)
        same &= a.p[k].price == b.p[k].price && a.p[k].std_error == b.p[k].std_error && a.p[k].prob_itm == b.p[k].prob_itm;
    return same;
}

// ---------------------------------------------------------------- price beside a distribution
// One leg: priced from the stored payoffs, the same bits as without; several legs: not
// answered from them, and the prices are those without.
static void section_distribution() {
    qk_handle *h = nullptr;
    if (qk_create(0, &h) != QK_OK) {
        check(false, std::string("qk_create: ") + qk_last_error());
        return;
    }
    for (int precision : {QK_FP32, QK_FP64})
        for (int64_t n : {1, 33, 65, 4097, 100003})
            for (int legs = 1; legs <= 2; ++legs) {
                std::vector<qk_payoff> l{leg(QK_ASIAN, QK_CALL, 100.0)};
                if (legs == 2) l.push_back(leg(QK_EUROPEAN, QK_PUT, 105.0));
                const qk_contract c = contract(precision, QK_BATES, QK_ANDERSEN_QE, n, 20, l);
                qk_result alone{}, beside{};
                double order[3];
                qk::PayoffRanks dist;
                dist.ranks.r[1] = static_cast<unsigned long long>(n) / 2;
                dist.ranks.r[2] = static_cast<unsigned long long>(n) - 1;
                dist.n_ranks = 3;
                dist.out = order;
                bool ok = qk::price_contracts(h, &c, 1, nullptr, &alone, false) == QK_OK &&
                          qk::price_contracts(h, &c, 1, nullptr, &beside, false, &dist) == QK_OK;
                ok = ok && same_legs(alone, beside, legs) && dist.done == (legs == 1);
                check(ok, "distribution precision " + std::to_string(precision) + " paths " + std::to_string(n) + " legs " +
                              std::to_string(legs));
            }
    qk_destroy(h);
}

int main(int argc, char **argv) {
    const std::string section = argc > 1 ? argv[1] : "";
    if (section == "select") section_select();
    else if (section == "distribution") section_distribution();
    else check(false, "unknown section " + section);
    return g_failed != 0;
}
