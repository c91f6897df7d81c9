// host_check.cpp -- the product's per-root secular state machine
// (brdc_secular.cuh) compiled for the host, so the CPU test suite can check
// its numerics against LAPACK DLAED4 without a GPU.  Not used by the solver.
#include <atomic>
#include <cfloat>
#include <chrono>
#include <thread>
#include <vector>

#include "brdc_device_cache.h"
#include "brdc_leaf.cuh"
#include "brdc_secular.cuh"

extern "C" int brdc_host_secular_root(int K, const double *d, const double *z,
                                      double rho, double znorm2, int i,
                                      int *org, double *tau, int *failed) {
    return brdc::sec_solve_serial(K, d, z, rho, znorm2, i, org, tau, failed,
                                  DBL_EPSILON);
}

// The same with an iteration cap of its own (the failure path).
extern "C" int brdc_host_secular_root_capped(int K, const double *d, const double *z,
                                             double rho, double znorm2, int i, int max_iter,
                                             int *org, double *tau, int *failed) {
    return brdc::sec_solve_serial(K, d, z, rho, znorm2, i, org, tau, failed,
                                  DBL_EPSILON, max_iter);
}

// The same root by sweeps of sec_accum_any (both sides in one loop), dealt to
// `lanes` lanes and combined as the kernels' butterfly does.
extern "C" int brdc_host_secular_root_any(int K, const double *d, const double *z, double rho,
                                          double znorm2, int i, int lanes, int *org, double *tau,
                                          int *failed) {
    brdc::SecRoot r;
    brdc::sec_init(r, i, K, d, z, rho, znorm2);
    int sweeps = 0;
    while (r.stage != 2) {
        brdc::SecTot t[32] = {};
        for (int j = 0; j < K; ++j) {
            brdc::sec_accum_any(t[j % lanes], r, j, d[j], z[j]);
        }
        for (int o = lanes >> 1; o > 0; o >>= 1) {
            for (int l = 0; l < o; ++l) {
                brdc::sec_combine(t[l], t[l + o]);
            }
        }
        ++sweeps;
        brdc::sec_bound(t[0], (K + lanes - 1) / lanes);
        brdc::sec_after_sweep(r, t[0], DBL_EPSILON);
    }
    *org = r.org;
    *tau = r.tau;
    *failed = r.failed;
    return sweeps;
}

// One leaf of s rows (d, e >= 0, scaled to a norm in [0.5, 1)) as
// leaf_pairs solves it, its lanes in turn: eigenvalues, vectors (s x s,
// vector i in row i), the largest residual, |F| and evaluations of a lane.
// Returns 1 where the kernel would keep the result.
extern "C" int brdc_host_leaf(int s, const double *d, const double *e, double *lam, double *vec,
                              double *stats) {
    using namespace brdc;
    LeafScratch B;
    double hi = -8.0, nlo = -8.0;
    for (int k = 0; k < kLeafN; ++k) {
        const double ek = k + 1 < s ? e[k] : 0.0, ep = k > 0 && k < s ? e[k - 1] : 0.0;
        B.v[k][kLeafN] = k < s ? d[k] : kLeafPad;
        B.v[k][kLeafN + 1] = ek * ek;
        B.e[k] = ek;
        if (k < s) {
            hi = std::fmax(hi, d[k] + (ek + ep));
            nlo = std::fmax(nlo, (ek + ep) - d[k]);
        }
    }
    const double wide = fma(0x1p-5, hi + nlo, 0x1p-48);
    const double lo = -nlo - wide;
    hi += wide;
    const double w = (hi - lo) * (1.0 / 17.0);
    int cnt[16];
    for (int x = 0; x < 16; ++x) {
        double p, q;
        cnt[x] = leaf_minors(B, fma(w, (double)(x + 1), lo), &p, &q);
    }
    int evals = 0;
    bool ok = true;
    for (int x = 0; x < s; ++x) {
        LeafRoot r;
        int below = 0;
        r.ca = 0;
        r.cb = s;
        for (int j = 0; j < 16; ++j) {
            if (cnt[j] <= x) {
                ++below;
                r.ca = cnt[j];
            } else {
                r.cb = r.cb < cnt[j] ? r.cb : cnt[j];
            }
        }
        r.a = fma(w, (double)below, lo);
        r.b = fma(w, (double)(below + 1), lo);
        r.x = 0.5 * (r.a + r.b);
        r.state = 0;
        int it = 0;
        for (; it < kLeafMaxEval && r.state == 0; ++it) {
            double p, q;
            const int c = leaf_minors(B, r.x, &p, &q);
            leaf_advance(r, x, c, p, q);
        }
        evals = evals > it ? evals : it;
        ok = ok && r.state == 1;
        lam[x] = r.x;
    }
    for (int x = 0; x + 1 < s; ++x) {
        ok = ok && lam[x + 1] - lam[x] > kLeafGap;
    }
    stats[2] = evals;
    stats[0] = stats[1] = INFINITY;
    if (!ok) {
        return 0;
    }
    double V[16][16], res = 0.0, orth = 0.0;
    for (int x = 0; x < s; ++x) {
        const double r = leaf_vector(B, x, s, &lam[x], V[x]);
        res = r <= res ? res : r;
    }
    for (int x = 0; x < s; ++x) {
        double acc[16] = {};
        for (int i = 0; i < s; ++i) {
            double F = i == x ? -1.0 : 0.0;
            for (int k = 0; k < s; ++k) {
                F = fma(V[i][k], V[x][k], F);
            }
            orth = std::fabs(F) <= orth ? orth : std::fabs(F);
            for (int k = 0; k < s; ++k) {
                acc[k] = fma(F, V[i][k], acc[k]);
            }
        }
        for (int k = 0; k < s; ++k) {
            vec[x * s + k] = fma(-0.5, acc[k], V[x][k]);
        }
    }
    stats[0] = res;
    stats[1] = orth;
    return res <= kLeafResid && orth <= kLeafOrth;
}

// `threads` threads ask a device's cache at once; how often the (slow) query
// ran, or -1 if a thread got another answer than the query's.
extern "C" int brdc_host_cache_queries(int threads, int device) {
    brdc::DeviceCache<int> cache;
    std::atomic<int> queries{0}, wrong{0}, ready{0};
    std::vector<std::thread> pool;
    for (int t = 0; t < threads; ++t) {
        pool.emplace_back([&]() {
            ++ready;
            while (ready.load() < threads) {
            }
            const int got = cache.get(device, [&](int dev) {
                std::this_thread::sleep_for(std::chrono::milliseconds(20));
                ++queries;
                return 100 + dev;
            });
            const bool known = device >= 0 && device < brdc::kMaxDevices;
            wrong += got != (known ? 100 + device : 0);
        });
    }
    for (std::thread &t : pool) {
        t.join();
    }
    return wrong.load() != 0 ? -1 : queries.load();
}
