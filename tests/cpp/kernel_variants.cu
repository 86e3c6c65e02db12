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
#include "qk_math64.cuh"

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

// ---------------------------------------------------------------- one task, every launch shape
struct DeviceTask {
    qk::TaskDev t;
    Dev<qk::TaskDev> task;
    Dev<int64_t> prefix;
    Dev<unsigned long long> cursor;
    Dev<qk::Moments> partials;
    size_t records;
    DeviceTask(const qk::TaskDev &t_)
        : t(t_), task(std::vector<qk::TaskDev>{t_}), prefix(std::vector<int64_t>{0}), cursor(1),
          partials(static_cast<size_t>(t_.n_tiles) * t_.n_payoffs), records(static_cast<size_t>(t_.n_tiles) * t_.n_payoffs) {}
    // The tile records of one launch.
    std::vector<qk::Moments> run(int grid, int block, bool table) {
        CUDA(cudaMemset(cursor.p, 0, sizeof(unsigned long long)));
        CUDA(cudaMemset(partials.p, 0xFF, records * sizeof(qk::Moments)));
        const uint64_t seed = static_cast<uint64_t>(t.key0) | (static_cast<uint64_t>(t.key1) << 32);
        CUDA(qk::launch_price_tiles(t.precision, t.model, t.scheme, grid, nullptr, task.p, prefix.p, 1, 0, t.n_tiles,
                                    cursor.p, partials.p, true, seed, t.lane_mode, t.track, block, table));
        CUDA(cudaDeviceSynchronize());
        return partials.host(records);
    }
};

static bool same_bytes(const std::vector<qk::Moments> &a, const std::vector<qk::Moments> &b) {
    return a.size() == b.size() && std::memcmp(a.data(), b.data(), a.size() * sizeof(qk::Moments)) == 0;
}

// A launch whose every tile has a warp of its own against persistent launches of each block
// size, and those with a term table: the same records.
static void section_shapes() {
    qk_handle *h = nullptr;  // loads the kernels
    if (qk_create(0, &h) != QK_OK) return check(false, std::string("qk_create: ") + qk_last_error());
    int tables = 0;
    for (int precision : {QK_FP32, QK_FP64})
        for (int model : {QK_HESTON, QK_BATES})
            for (int lanes : {qk::kLaneOne, qk::kLaneTwo})
                for (int64_t n : {1, 33, 4096, 151553})
                    for (double rho : {-0.7, 0.6}) {
                        qk_contract c = contract(precision, model, QK_ANDERSEN_QE, n, 25,
                                                 {leg(QK_EUROPEAN, QK_CALL, 100.0), leg(QK_ASIAN, QK_PUT, 100.0)});
                        c.rho = rho;
                        double scale = 1.0;
                        DeviceTask d(qk::make_task(qk::normalised(c, &scale), n > 100000 ? 3 : 1, lanes));
                        const auto want = d.run((d.t.n_tiles + 3) / 4, 128, false);
                        bool same = true;
                        for (int block : {128, 256, 512}) {
                            if (!qk::price_tiles_block_ok(precision, block)) continue;
                            for (int grid : {1, 37}) same &= same_bytes(want, d.run(grid, block, false));
                            if (!qk::price_tiles_takes_table(d.t, block)) continue;
                            ++tables;
                            for (int grid : {1, 37}) same &= same_bytes(want, d.run(grid, block, true));
                        }
                        check(same, "shapes precision " + std::to_string(precision) + " model " + std::to_string(model) + " lanes " +
                                        std::to_string(lanes) + " paths " + std::to_string(n) + " rho " + std::to_string(rho));
                    }
    check(tables == 16, "shapes: FP32 with two paths per lane takes a table");
    qk_destroy(h);
}

// The American forward slabs with a term table, without, and one path per thread.
static void section_slabs() {
    qk_handle *h = nullptr;
    if (qk_create(0, &h) != QK_OK) return check(false, std::string("qk_create: ") + qk_last_error());
    const int sms = 148, stride = 5, rows = 5;
    int tables = 0;
    for (int model : {QK_HESTON, QK_BATES})
        for (double rho : {-0.7, 0.0, 0.6})
            for (double sigma : {0.3, 0.9}) {
                const int64_t n = 400003;  // above the line from which the slab kernel takes the table
                qk_contract c = contract(QK_FP32, model, QK_ANDERSEN_QE, n, stride * rows, {leg(QK_AMERICAN, QK_PUT, 100.0)});
                c.rho = rho;
                c.sigma = sigma;
                double scale = 1.0;
                const qk::TaskDev t = qk::make_task(qk::normalised(c, &scale), 1);
                Dev<qk::TaskDev> task(std::vector<qk::TaskDev>{t});
                Dev<float> S(n * rows), v(n * rows);
                std::vector<float> got[3][2];
                // a range of too many floats has no table (sigma 0.9 with rho)
                const int launches = t.term_lo > 0 ? 3 : 2;
                tables += t.term_lo > 0;
                for (int k = 0; k < launches; ++k) {
                    CUDA(cudaMemset(S.p, 0xFF, n * rows * sizeof(float)));
                    CUDA(cudaMemset(v.p, 0xFF, n * rows * sizeof(float)));
                    CUDA(qk::launch_slab_paths(QK_FP32, model, QK_ANDERSEN_QE, c.seed, nullptr, task.p, 0, n, stride, S.p, v.p, n,
                                               sms, k == 0 ? 1 : 2, k == 2));
                    CUDA(cudaDeviceSynchronize());
                    got[k][0] = S.host(n * rows);
                    got[k][1] = v.host(n * rows);
                }
                bool same = true;
                for (int k = 1; k < launches; ++k)
                    for (int a = 0; a < 2; ++a)
                        same &= std::memcmp(got[0][a].data(), got[k][a].data(), n * rows * sizeof(float)) == 0;
                check(same, "slabs model " + std::to_string(model) + " rho " + std::to_string(rho) + " sigma " + std::to_string(sigma));
            }
    check(tables == 8, "slabs: eight of the contracts take a table");
    qk_destroy(h);
}

// ---------------------------------------------------------------- FP64 functions
enum Fn { kNeg2LogWord, kNeg2Log, kExp2, kRcp, kRsqrt, kSqrt, kSqrtPos, kMax0, kNormals };

__global__ void eval_kernel(int fn, const double *x, const uint32_t *w1, const uint32_t *w2, int n, double *y, double *y2) {
    __shared__ qk::Tab64 tab;
    qk::fill_tab64(tab);
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        switch (fn) {
            case kNeg2LogWord: y[i] = qk::neg2_log64(tab, x[i], 32); break;
            case kNeg2Log: y[i] = qk::neg2_log64(tab, x[i], 0); break;
            case kExp2: y[i] = qk::exp2_64(tab, x[i]); break;
            case kRcp: y[i] = qk::rcp64(x[i]); break;
            case kRsqrt: y[i] = qk::rsqrt64(x[i]); break;
            case kSqrt: y[i] = qk::sqrt64(x[i]); break;
            case kSqrtPos: y[i] = qk::sqrt_pos64(x[i]); break;
            case kMax0: y[i] = qk::max0_64(x[i]); break;
            default: qk::box_muller64(tab, w1[i], w2[i], y[i], y2[i]);
        }
    }
}

static std::vector<double> evaluate(Fn fn, const std::vector<double> &x) {
    Dev<double> dx(x), dy(x.size());
    eval_kernel<<<148, 256>>>(fn, dx.p, nullptr, nullptr, static_cast<int>(x.size()), dy.p, nullptr);
    CUDA(cudaGetLastError());
    CUDA(cudaDeviceSynchronize());
    return dy.host(x.size());
}

// Largest relative error against long double values (an exact zero has to be met exactly).
template <class F>
static void check_function(const char *name, Fn fn, const std::vector<double> &x, double bound, F exact) {
    const std::vector<double> y = evaluate(fn, x);
    double worst = 0.0, at = 0.0;
    for (size_t i = 0; i < x.size(); ++i) {
        const long double e = exact(static_cast<long double>(x[i]));
        const double r = e == 0.0L ? (y[i] == 0.0 ? 0.0 : HUGE_VAL) : static_cast<double>(fabsl((y[i] - e) / e));
        if (!(r <= worst)) worst = r, at = x[i];
    }
    char text[160];
    std::snprintf(text, sizeof(text), "%s: largest relative error %.3g (at %.17g), bound %.3g, %zu arguments", name, worst, at,
                  bound, x.size());
    check(worst <= bound, text);
}

// Bounds: two units in the last place (2^-51) for the table-driven functions (a rounded table
// entry, its product, the final sum), one (2^-52) for the reciprocal and the roots, three of
// the radius for a normal.
static void section_functions() {
    const double ulp = 2.220446049250313e-16;
    std::mt19937_64 g(11);
    auto u = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(g); };
    const std::vector<uint32_t> edges = {0u, 1u, 2u, 255u, (1u << 22) - 1, 1u << 22, (1u << 23) - 1, 1u << 23, (1u << 23) + 1,
                                         0x7FFFFFFFu, 0x80000000u, 0x80000001u, 0xFFFFFFFDu, 0xFFFFFFFEu, 0xFFFFFFFFu};
    std::vector<double> x;
    for (uint32_t w : edges) x.push_back(w + 0.5);
    for (int i = 0; i < (1 << 20); ++i) x.push_back(static_cast<uint32_t>(i & 1 ? g() : 0xFFFFFFFFull - (g() >> (32 + i % 32))) + 0.5);
    check_function("-2 ln of a word", kNeg2LogWord, x, 2 * ulp, [](long double t) { return -2 * logl(t / 4294967296.0L); });
    x = {1.0, 0.25, 4.0, 0.7002, 1.4004, 1e-150, 1e190};
    for (int k = 1; k < 4000; ++k) x.insert(x.end(), {1.0 + k * ulp, 1.0 - k * ulp / 2});
    for (int i = 0; i < (1 << 20); ++i) x.push_back(std::exp2(u(-3.0, 3.0) * (i % 16 == 0 ? 100.0 : 1.0)));
    check_function("-2 ln of a product", kNeg2Log, x, 2 * ulp, [](long double t) { return -2 * logl(t); });
    x = {0.0, -0.0, 1e-300, -1e-300, 1.0, -1.0, 999.99, -999.99, std::nextafter(1000.0, 0.0), -std::nextafter(1000.0, 0.0), 1000.0, -1000.0};
    for (int k = -512; k <= 512; ++k) x.insert(x.end(), {k / 512.0, std::nextafter(k / 512.0, 9.0), std::nextafter(k / 512.0, -9.0)});
    for (int i = 0; i < (1 << 20); ++i) x.push_back(i % 4 ? u(-8.0, 8.0) : u(-1000.0, 1000.0));
    check_function("2^x", kExp2, x, 2 * ulp, [](long double t) { return exp2l(t); });
    x.clear();
    for (int i = 0; i < (1 << 20); ++i) x.push_back(std::exp2(u(-60.0, 60.0) * (i % 16 == 0 ? 8.0 : 1.0)) * (i % 5 ? 1.0 : -1.0));
    check_function("1/x", kRcp, x, ulp, [](long double t) { return 1 / t; });
    for (double &t : x) t = std::fabs(t);
    x.insert(x.end(), {1.0, 2.0, 4.0, 0.25, 2.2250738585072014e-308, 1e300});
    check_function("1/sqrt x", kRsqrt, x, ulp, [](long double t) { return 1 / sqrtl(t); });
    check_function("sqrt x > 0", kSqrtPos, x, ulp, [](long double t) { return sqrtl(t); });
    x.push_back(0.0);
    check_function("sqrt x >= 0", kSqrt, x, ulp, [](long double t) { return sqrtl(t); });

    const std::vector<double> tiny = evaluate(kSqrt, {5e-324, 1e-310, 2.2e-308});
    check(tiny[0] >= 0 && tiny[0] < 1.5e-154 && tiny[1] >= 0 && tiny[1] < 1.5e-154 && tiny[2] >= 0 && tiny[2] < 1.6e-154,
          "sqrt of subnormal numbers stays below that of the least normal one");
    const double inf = HUGE_VAL, nan = std::nan("");
    const std::vector<double> far = evaluate(kExp2, {1000.5, 1023.5, 1024.0, 1e300, inf, -1000.5, -1073.5, -1080.0, -inf, nan});
    bool ok = far[2] == inf && far[3] == inf && far[4] == inf && far[7] == 0.0 && far[8] == 0.0 && std::isnan(far[9]);
    ok = ok && std::fabs(far[0] / std::exp2(1000.5) - 1) <= 2 * ulp && std::fabs(far[1] / std::exp2(1023.5) - 1) <= 2 * ulp &&
         std::fabs(far[5] / std::exp2(-1000.5) - 1) <= 2 * ulp && far[6] >= 0.0 && far[6] <= 1e-322;
    check(ok, "2^x beyond 1000, infinities and NaN");
    const std::vector<double> m0 = evaluate(kMax0, {0.0, -0.0, 5e-324, -5e-324, 1.5, -1.5, inf, -inf, nan, -nan});
    check(m0[0] == 0 && m0[1] == 0 && m0[2] == 5e-324 && m0[3] == 0 && m0[4] == 1.5 && m0[5] == 0 && m0[6] == inf && m0[7] == 0 &&
              m0[8] == 0 && m0[9] == 0,
          "max(x, 0)");

    std::vector<uint32_t> w1, w2;
    for (uint32_t a : edges)
        for (uint32_t b : edges) w1.push_back(a), w2.push_back(b);
    for (int i = 0; i < (1 << 20); ++i) w1.push_back(static_cast<uint32_t>(g())), w2.push_back(static_cast<uint32_t>(g()));
    Dev<uint32_t> d1(w1), d2(w2);
    Dev<double> z1(w1.size()), z2(w1.size());
    eval_kernel<<<148, 256>>>(kNormals, nullptr, d1.p, d2.p, static_cast<int>(w1.size()), z1.p, z2.p);
    CUDA(cudaGetLastError());
    CUDA(cudaDeviceSynchronize());
    const auto g1 = z1.host(w1.size()), g2 = z2.host(w1.size());
    double worst = 0.0;
    for (size_t i = 0; i < w1.size(); ++i) {
        const long double r = sqrtl(-2 * logl((w1[i] + 0.5L) / 4294967296.0L));
        const long double a = 2 * 3.14159265358979323846264338327950288L * ((w2[i] + 0.5L) / 4294967296.0L - 0.5L);
        worst = std::max(worst, static_cast<double>(std::max(fabsl(g1[i] - r * cosl(a)), fabsl(g2[i] - r * sinl(a))) / r));
    }
    char text[120];
    std::snprintf(text, sizeof(text), "normals: largest error %.3g of the radius, %zu pairs", worst, w1.size());
    check(worst <= 3 * ulp, text);
}

int main(int argc, char **argv) {
    const std::string section = argc > 1 ? argv[1] : "";
    if (section == "select") section_select();
    else if (section == "distribution") section_distribution();
    else if (section == "shapes") section_shapes();
    else if (section == "slabs") section_slabs();
    else if (section == "functions") section_functions();
    else check(false, "unknown section " + section);
    return g_failed != 0;
}
