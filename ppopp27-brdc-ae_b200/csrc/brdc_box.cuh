// brdc_box.cuh -- the large merges k_level leaves (KArgs::big_k): roots,
// Loewner weights and boundary rows by sums of which most terms come from an
// interpolant.
//
// Every sum of a merge has the form F(x) = sum_j c_j / (d_j - x)^(1 or 2), or
// is the product of (x - lambda_j) / (x - d_j), at x inside one pole's
// neighbourhood.  The poles are dealt into boxes of b consecutive ones.  On
// a box's interval [mid - h, mid + h] the part of F from the poles at least
// h * 2 away from the interval is analytic well beyond it (a Bernstein
// ellipse of parameter 3 + sqrt(8) = 5.83), so its interpolant at p = 24
// Chebyshev points is off by at most 2.5e-18 of it (one pole at the edge of
// the far part, evaluated in extended precision; the squared sums, whose poles
// are double, 3.1e-17), below rounding.  A box's interpolants cost p K terms once, and each of its b poles or roots
// then takes the near poles (3 b where they lie evenly) and one polynomial
// per sum and sweep instead of K terms: at K = 4096, b = 64, 1536 terms a
// root once and 200 a sweep.  Differences are taken from mid, which
// is exact to the rounding of the difference, so nothing is lost where a box
// is narrow.  A box whose far part would be less than half of the poles
// (clusters straddled by its interval) sums all of them directly.  Boxes with
// many near poles are listed, and their roots get more lanes (box_runs).  The
// last root, whose bracket leaves the poles' range, is summed directly by a
// whole block.
//
// Bound: FP64 arithmetic.  Measured on B200 against sweeps over all poles
// (k_sweeps, which still serves levels with the fused kernel off): Toeplitz
// 16,384 2.31 -> 1.05 ms, 65,536 20.3 -> 3.6 ms, the mixed batch of 4096
// matrices 66 -> 37 ms; largest error of Toeplitz 16,384 against its closed
// form 1.3e-16 -> 0.9e-16 of the norm.
#pragma once

#include "brdc_kernels.cuh"

namespace brdc {

constexpr int kBoxP = 24;        // Chebyshev points of an interpolant
// Points a warp sums over its share of the poles: 6 points keep a pole's two
// loads hidden behind 42 FP64 instructions; the block's 8 warps are 4 groups
// of points by 2 halves of the poles.
constexpr int kBoxNodes = 6;
constexpr int kBoxHalves = (kSweepThreads / 32) * kBoxNodes / kBoxP;
static_assert(kBoxHalves * kBoxP == (kSweepThreads / 32) * kBoxNodes, "points and halves");
constexpr double kBoxFar = 3.0;  // far: at least this many h from mid
constexpr int kBoxLong = 6;      // listed: more near poles than this many boxes'

// A box's scratch lies in the node's slices of the next level's arrays,
// which the placement fills last: 64 doubles of each from the box's first
// pole on (a box has at least 64 poles).
//   nd  0 psi, 24 dpsi, 48 mid, 49 1/h, 50 nlo, 51 nhi, 52 h,
//       53 (of the level's i-th box) the i-th listed box
//   nf  0 phi, 24 dphi; for the rows 0 sum l u
//   nl  0 Loewner product; for the rows 0 sum u^2, 24 sum f u
struct BoxHdr {
    double mid, ih, h;
    int nlo, nhi; // near poles [nlo, nhi)
    __device__ bool far(int K) const { return nlo > 0 || nhi < K; }
    // the Loewner product pairs pole j with root j in (d_j, d_{j+1}): the
    // root of the last far pole below may be near
    __device__ int low() const { return nlo > 0 ? nlo - 1 : 0; }
    __device__ bool listed(int b) const { return nhi - nlo > kBoxLong * b; }
};

// Where box `item` of the level keeps its scratch.
__device__ inline long long box_slice(const KArgs &a, int item) {
    const Ws &w = a.w;
    const int g = w.items_c[item];
    return node_geom(a.F, a.k, g).gstart +
           (long long)(item - w.pref_c[g]) * w.hdr->lvl[a.k].box;
}

__device__ inline BoxHdr box_header(const Ws &w, long long sb) {
    BoxHdr H;
    H.mid = __ldcg(w.nd + sb + 48);
    H.ih = __ldcg(w.nd + sb + 49);
    H.nlo = (int)__ldcg(w.nd + sb + 50);
    H.nhi = (int)__ldcg(w.nd + sb + 51);
    H.h = __ldcg(w.nd + sb + 52);
    return H;
}

// sum_m c_m T_m(t), Clenshaw.
__device__ __forceinline__ double box_eval(const double *c, double t) {
    const double t2 = t + t;
    double b1 = 0.0, b2 = 0.0;
#pragma unroll 8
    for (int m = kBoxP - 1; m > 0; --m) {
        const double b = fma(t2, b1, c[m] - b2);
        b2 = b1;
        b1 = b;
    }
    return fma(t, b1, c[0] - b2);
}

enum BoxSum { kBoxSecular, kBoxLowner, kBoxRows };

struct BoxSmem {
    double cosv[4 * kBoxP];               // cos(pi i / 48)
    double val[kBoxHalves][4][kBoxP];     // sums at the points
    double coef[kSweepThreads / 32][4 * kBoxP]; // a warp's box
    double red[32];
};

// Poles of node list d[0, K) with d - mid < v (or <= v), by all threads.
__device__ inline int box_count(const double *d, int K, double mid, double v, bool closed) {
    int lo = 0, hi = K;
    while (lo < hi) {
        const int step = (hi - lo + kSweepThreads - 1) / kSweepThreads;
        const int i = lo + (int)threadIdx.x * step;
        bool in = false;
        if (i < hi) {
            const double x = __ldg(d + i) - mid;
            in = closed ? x <= v : x < v;
        }
        const int n = __syncthreads_count(in);
        if (n == 0) {
            hi = lo;
        } else {
            hi = min(hi, lo + n * step);
            lo = lo + (n - 1) * step + 1;
        }
    }
    return lo;
}

// Far sums of every box at its Chebyshev points, and their coefficients.
template <BoxSum WHAT>
__device__ void box_far(const KArgs &a, BoxSmem &S) {
    const Ws &w = a.w;
    LevelCtl *ctl = &w.hdr->lvl[a.k];
    const int boxes = ctl->items_c, b = ctl->box;
    const int warp = threadIdx.x >> 5;
    const int node0 = (warp / kBoxHalves) * kBoxNodes, half = warp % kBoxHalves;
    // the warp's lanes among those that stride over the poles
    const int lane = half * 32 + (threadIdx.x & 31);
    constexpr int kStep = 32 * kBoxHalves;
    constexpr int NF = WHAT == kBoxSecular ? 4 : WHAT == kBoxLowner ? 1 : 3;
    for (int item = blockIdx.x; item < boxes; item += gridDim.x) {
        const int g = w.items_c[item];
        const NodeGeom G = node_geom(a.F, a.k, g);
        if (WHAT != kBoxSecular && G.depth == 0) {
            continue;
        }
        const int K = w.nK[g], q = item - w.pref_c[g], nb = K / b;
        const long long po = G.poff, sb = G.gstart + (long long)q * b;
        const double *pd = w.pd + po;
        BoxHdr H;
        if (WHAT == kBoxSecular) {
            const int B0 = q * b;
            const double lo = __ldg(pd + B0), hi = __ldg(pd + (q == nb - 1 ? K - 1 : B0 + b));
            H.h = 0.5 * (hi - lo);
            H.mid = lo + H.h;
            H.ih = 1.0 / H.h;
            H.nlo = box_count(pd, K, H.mid, -kBoxFar * H.h, false);
            H.nhi = box_count(pd, K, H.mid, kBoxFar * H.h, true);
            if (!(H.h > 0.0) || !isfinite(H.ih) || 2 * (H.nhi - H.nlo) > K) {
                H.nlo = 0;
                H.nhi = K;
            }
            if (threadIdx.x == 0) {
                w.nd[sb + 48] = H.mid;
                w.nd[sb + 49] = H.ih;
                w.nd[sb + 50] = (double)H.nlo;
                w.nd[sb + 51] = (double)H.nhi;
                w.nd[sb + 52] = H.h;
                if (H.listed(b)) {
                    w.nd[box_slice(a, atomicAdd(&ctl->citem, 1)) + 53] = (double)item;
                }
            }
        } else {
            H = box_header(w, sb);
        }
        if (!H.far(K)) {
            continue;
        }
        double x[kBoxNodes], f[NF][kBoxNodes];
#pragma unroll
        for (int u = 0; u < kBoxNodes; ++u) {
            x[u] = H.h * S.cosv[2 * (node0 + u) + 1];
#pragma unroll
            for (int i = 0; i < NF; ++i) {
                f[i][u] = WHAT == kBoxLowner ? 1.0 : 0.0;
            }
        }
        if constexpr (WHAT == kBoxSecular) {
            const double *pz = w.pz + po;
#pragma unroll 4
            for (int j = lane; j < H.nlo; j += kStep) {
                const double d = __ldg(pd + j) - H.mid, z = __ldg(pz + j);
#pragma unroll
                for (int u = 0; u < kBoxNodes; ++u) {
                    const double t = z * brdc_rcp(d - x[u]);
                    f[0][u] = fma(z, t, f[0][u]);
                    f[1][u] = fma(t, t, f[1][u]);
                }
            }
#pragma unroll 4
            for (int j = H.nhi + lane; j < K; j += kStep) {
                const double d = __ldg(pd + j) - H.mid, z = __ldg(pz + j);
#pragma unroll
                for (int u = 0; u < kBoxNodes; ++u) {
                    const double t = z * brdc_rcp(d - x[u]);
                    f[2][u] = fma(z, t, f[2][u]);
                    f[3][u] = fma(t, t, f[3][u]);
                }
            }
        } else if constexpr (WHAT == kBoxLowner) {
            const double *rdo = w.rdo + po, *rtau = w.rtau + po;
            // far poles by number: [0, low) and then [nhi, K)
            const int nl = H.low(), nf = nl + (K - H.nhi);
            auto at = [&](int i, double *n, double *d) {
                const int j = i < nl ? i : H.nhi + (i - nl);
                *n = (H.mid - __ldcg(rdo + j)) - __ldcg(rtau + j);
                *d = H.mid - __ldg(pd + j);
            };
            int i = lane;
            for (; i + kStep < nf; i += 2 * kStep) {
                double n1, d1, n2, d2;
                at(i, &n1, &d1);
                at(i + kStep, &n2, &d2);
#pragma unroll
                for (int u = 0; u < kBoxNodes; ++u) {
                    f[0][u] *= lowner_pair(n1 + x[u], d1 + x[u], n2 + x[u], d2 + x[u]);
                }
            }
            if (i < nf) {
                double n1, d1;
                at(i, &n1, &d1);
#pragma unroll
                for (int u = 0; u < kBoxNodes; ++u) {
                    f[0][u] *= (n1 + x[u]) * brdc_rcp(d1 + x[u]);
                }
            }
        } else {
            const double *pw = w.pw + po, *pf = w.pf + po, *pl = w.pl + po;
            const int nf = H.nlo + (K - H.nhi);
#pragma unroll 4
            for (int i = lane; i < nf; i += kStep) {
                const int j = i < H.nlo ? i : H.nhi + (i - H.nlo);
                const double d = __ldg(pd + j) - H.mid, wj = __ldcg(pw + j);
                const double fj = __ldg(pf + j), lj = __ldg(pl + j);
#pragma unroll
                for (int u = 0; u < kBoxNodes; ++u) {
                    const double t = wj * brdc_rcp(d - x[u]);
                    f[0][u] = fma(t, t, f[0][u]);
                    f[1][u] = fma(fj, t, f[1][u]);
                    f[2][u] = fma(lj, t, f[2][u]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NF; ++i) {
#pragma unroll
            for (int u = 0; u < kBoxNodes; ++u) {
                const double v = WHAT == kBoxLowner ? group_prod(f[i][u], 32)
                                                    : group_sum(f[i][u], 32);
                if ((threadIdx.x & 31) == 0) {
                    S.val[half][i][node0 + u] = v;
                }
            }
        }
        __syncthreads();
        // c_m = (2/p) sum_k f_k cos(pi m (2k+1) / (2p)), c_0 half of that
        if (threadIdx.x < NF * kBoxP) {
            const int i = threadIdx.x / kBoxP, m = threadIdx.x % kBoxP;
            double c = 0.0;
#pragma unroll 4
            for (int k = 0; k < kBoxP; ++k) {
                double v = S.val[0][i][k];
#pragma unroll
                for (int h = 1; h < kBoxHalves; ++h) {
                    v = WHAT == kBoxLowner ? v * S.val[h][i][k] : v + S.val[h][i][k];
                }
                c = fma(v, S.cosv[(m * (2 * k + 1)) % (4 * kBoxP)], c);
            }
            c *= (m == 0 ? 1.0 : 2.0) / kBoxP;
            double *to = WHAT == kBoxSecular ? (i < 2 ? w.nd : w.nf) + sb + kBoxP * (i & 1)
                         : WHAT == kBoxLowner ? w.nl + sb
                                              : (i < 2 ? w.nl + kBoxP * i : w.nf) + sb;
            to[m] = c;
        }
        __syncthreads();
    }
}

// A warp's share of the near phases: runs of 32 / tpr consecutive poles or
// roots of one box.  body(G, g, K, first root, roots, tpr, slice, box header).
//
// The listed boxes have runs of their own, with as many lanes per root as the
// grid has threads for them, up to a warp a root: with the level's lanes, one
// box whose interval straddles two clusters held up the level, its warps at K
// terms a sweep for many roots each and the rest of the GPU idle.  Measured on
// B200 (whole solves, without -> with): poles in two clusters, n = 3000 661 ->
// 568 us, 40,000 18.5 -> 3.6 ms; in 16 clusters, 9001 1816 -> 1480 us.
template <class Body>
__device__ inline void box_runs(const KArgs &a, bool inner_only, Body body) {
    const Ws &w = a.w;
    const LevelCtl *ctl = &w.hdr->lvl[a.k];
    const int listed = __ldcg(&ctl->citem), b = ctl->box;
    const int warp = threadIdx.x >> 5;
    int tpr = ctl->tpr_w, Rw = 32 / tpr;
    const int items = ctl->items_w;
    // the last blocks first: the merges' last roots are with the first ones
    // (Toeplitz 2049 326 -> 306 us, 4096 437 -> 417)
    const int back = (int)(gridDim.x - 1 - blockIdx.x);
    for (int it = back * kWarpsPerBlock + warp; it < items;
         it += (int)gridDim.x * kWarpsPerBlock) {
        const int item = items - 1 - it;
        const int g = w.items_w[item];
        const NodeGeom G = node_geom(a.F, a.k, g);
        if (inner_only && G.depth == 0) {
            continue;
        }
        const int K = w.nK[g], r0 = (item - w.pref_w[g]) * Rw;
        const long long sb = G.gstart + (long long)min(r0 / b, K / b - 1) * b;
        const BoxHdr H = box_header(w, sb);
        if (!H.listed(b)) {
            body(G, g, K, r0, Rw, tpr, sb, H);
        }
    }
    if (listed == 0) {
        return;
    }
    while (tpr < 32 && 2LL * tpr * listed * b <= (long long)gridDim.x * kSweepThreads) {
        tpr <<= 1;
    }
    // a merge's last box has up to 2 b - 1 poles; the first blocks, which had
    // the fewest runs above, come first, and block 0 last
    Rw = 32 / tpr;
    const int per = 2 * b / Rw;
    const int turn = (int)(blockIdx.x > 0 ? blockIdx.x : gridDim.x) - 1;
    for (int it = turn * kWarpsPerBlock + warp; it < listed * per;
         it += (int)gridDim.x * kWarpsPerBlock) {
        const int item = (int)__ldcg(w.nd + box_slice(a, it / per) + 53);
        const int g = w.items_c[item];
        const NodeGeom G = node_geom(a.F, a.k, g);
        const int K = w.nK[g], q = item - w.pref_c[g];
        const int r0 = q * b + it % per * Rw;
        if ((inner_only && G.depth == 0) || r0 >= (q == K / b - 1 ? K : (q + 1) * b)) {
            continue;
        }
        const long long sb = G.gstart + (long long)q * b;
        body(G, g, K, r0, Rw, tpr, sb, box_header(w, sb));
    }
}

// A warp's copy of 24 coefficients.
__device__ inline void box_coef(double *dst, const double *src) {
    const int lane = threadIdx.x & 31;
    if (lane < kBoxP) {
        dst[lane] = __ldcg(src + lane);
    }
}

// body(G, g, K) for every merge of the level, one block each (the merges are
// found by their first boxes).
template <class Body>
__device__ inline void box_merges(const KArgs &a, bool inner_only, Body body) {
    const Ws &w = a.w;
    const int boxes = w.hdr->lvl[a.k].items_c;
    for (int item = blockIdx.x; item < boxes; item += gridDim.x) {
        const int g = w.items_c[item];
        if (item != w.pref_c[g]) {
            continue;
        }
        const NodeGeom G = node_geom(a.F, a.k, g);
        if (!(inner_only && G.depth == 0)) {
            body(G, g, w.nK[g]);
        }
    }
}

// The last roots, each over all poles of its merge by a whole block (one
// warp took 28 us for 8192 poles, longer than all other roots of the level).
__device__ void box_last_root(const KArgs &a, BoxSmem &S) {
    const Ws &w = a.w;
    const double eps = DBL_EPSILON;
    const int max_iter = w.hdr->max_iter;
    box_merges(a, false, [&](const NodeGeom &G, int g, int K) {
        const long long po = G.poff;
        const double *pd = w.pd + po, *pz = w.pz + po;
        SecRoot st;
        sec_init(st, K - 1, K, pd, pz, w.nrho[g], w.nzn[g]);
        while (st.stage != 2) {
            SecSums sum;
            sec_zero(sum);
            secular_span(sum, st, 0, K, threadIdx.x, kSweepThreads, K - 2, K,
                         [&](int j, double *d, double *z) {
                             *d = __ldg(pd + j);
                             *z = __ldg(pz + j);
                         });
            SecTot tot = sec_total(sum);
            // every thread ends with the same totals, and so the same state
            tot.sum = block_sum<kSweepThreads>(tot.sum, S.red);
            tot.mag = block_sum<kSweepThreads>(tot.mag, S.red);
            tot.dpsi = block_sum<kSweepThreads>(tot.dpsi, S.red);
            tot.dphi = block_sum<kSweepThreads>(tot.dphi, S.red);
            sec_bound(tot, K / kSweepThreads);
            sec_after_sweep(st, tot, eps, max_iter);
        }
        if (threadIdx.x < 32) {
            if (threadIdx.x == 0) {
                secular_store(w, a, po, K - 1, st);
            }
            secular_diag_warp(w, a.k, threadIdx.x == 0, st);
        }
    });
}

__device__ void box_secular(const KArgs &a, BoxSmem &S) {
    const Ws &w = a.w;
    const double eps = DBL_EPSILON;
    const int max_iter = w.hdr->max_iter;
    const int lane = threadIdx.x & 31;
    double *cf = S.coef[threadIdx.x >> 5];
    box_runs(a, false, [&](const NodeGeom &G, int g, int K, int r0, int Rw, int tpr, long long sb,
                           const BoxHdr &H) {
        const long long po = G.poff;
        const double *pd = w.pd + po, *pz = w.pz + po;
        const double rho = w.nrho[g], zn = w.nzn[g];
        const int l = lane & (tpr - 1), r = r0 + lane / tpr;
        const int r1 = min(r0 + Rw, K);
        const bool far = H.far(K);
        auto ld = [&](int j, double *d, double *z) {
            *d = __ldg(pd + j);
            *z = __ldg(pz + j);
        };
        if (far) {
            __syncwarp();
            box_coef(cf, w.nd + sb);
            box_coef(cf + kBoxP, w.nd + sb + kBoxP);
            box_coef(cf + 2 * kBoxP, w.nf + sb);
            box_coef(cf + 3 * kBoxP, w.nf + sb + kBoxP);
            __syncwarp();
        }
        const bool active = r < K - 1;
        SecRoot st;
        if (active) {
            sec_init(st, r, K, pd, pz, rho, zn);
        } else {
            st.stage = 2;
        }
        while (__any_sync(kFull, st.stage != 2)) {
            SecTot tot{};
            if (st.stage != 2) {
                SecSums near;
                sec_zero(near);
                secular_span(near, st, H.nlo, H.nhi - H.nlo, l, tpr, min(r0, K - 2), r1,
                             [&](int jj, double *d, double *z) { ld(H.nlo + jj, d, z); });
                tot = sec_total(near);
                if (far) {
                    const double t = ((st.eorg_d - H.mid) + st.etau) * H.ih;
                    for (int q = l; q < 4; q += tpr) {
                        const double v = box_eval(cf + q * kBoxP, t);
                        const double m = q == 0 ? -v : q == 2 ? v : 0.0; // modulus
                        tot.sum += (q & 1) == 0 ? v : 0.0;
                        tot.mag += m;
                        tot.err += m;
                        tot.dpsi += q == 1 ? v : 0.0;
                        tot.dphi += q == 3 ? v : 0.0;
                    }
                }
            }
            sums_reduce(tot, tpr);
            if (st.stage != 2) {
                sec_after_sweep(st, tot, eps, max_iter);
            }
        }
        if (active && l == 0) {
            secular_store(w, a, po, r, st);
        }
        secular_diag_warp(w, a.k, active && l == 0, st);
    });
}

__device__ void box_lowner(const KArgs &a, BoxSmem &S) {
    const Ws &w = a.w;
    const int lane = threadIdx.x & 31;
    double *cf = S.coef[threadIdx.x >> 5];
    box_runs(a, true, [&](const NodeGeom &G, int g, int K, int r0, int Rw, int tpr, long long sb,
                          const BoxHdr &H) {
        const long long po = G.poff;
        const double *pd = w.pd + po, *rdo = w.rdo + po, *rtau = w.rtau + po;
        const int l = lane & (tpr - 1), i = r0 + lane / tpr;
        const bool far = H.far(K), active = i < K;
        if (far) {
            __syncwarp();
            box_coef(cf, w.nl + sb);
            __syncwarp();
        }
        double prod = 1.0;
        if (active) {
            const double di = __ldg(pd + i);
            int j = H.low() + l;
#pragma unroll 4
            for (; j + tpr < H.nhi; j += 2 * tpr) {
                const int j2 = j + tpr;
                const double dl = (di - __ldcg(rdo + j)) - __ldcg(rtau + j);
                const double dl2 = (di - __ldcg(rdo + j2)) - __ldcg(rtau + j2);
                prod *= lowner_pair(dl, j == i ? 1.0 : di - __ldg(pd + j), dl2,
                                    j2 == i ? 1.0 : di - __ldg(pd + j2));
            }
            if (j < H.nhi) {
                const double dl = (di - __ldcg(rdo + j)) - __ldcg(rtau + j);
                prod *= dl * brdc_rcp(j == i ? 1.0 : di - __ldg(pd + j));
            }
            if (far && l == 0) {
                prod *= box_eval(cf, (di - H.mid) * H.ih);
            }
        }
        prod = group_prod(prod, tpr);
        if (active && l == 0) {
            w.pw[po + i] = lowner_value(w, po, i, prod, w.nrho[g]);
        }
    });
}

// sum u^2, sum f u, sum l u of the root at (dorg, tau) over poles i, i + n,
// ... below hi.
__device__ __forceinline__ void rows_span(const Ws &w, long long po, double dorg, double tau,
                                          int i, int hi, int n, double (&f)[3]) {
    const double *pd = w.pd + po, *pw = w.pw + po, *pf = w.pf + po, *pl = w.pl + po;
    auto add = [&](int j, double u) {
        f[0] += u * u;
        f[1] += __ldg(pf + j) * u;
        f[2] += __ldg(pl + j) * u;
    };
#pragma unroll 4
    for (; i + n < hi; i += 2 * n) {
        double u, u2;
        row_pair(__ldcg(pw + i), (__ldg(pd + i) - dorg) - tau, __ldcg(pw + i + n),
                 (__ldg(pd + i + n) - dorg) - tau, &u, &u2);
        add(i, u);
        add(i + n, u2);
    }
    if (i < hi) {
        const double dl = (__ldg(pd + i) - dorg) - tau;
        add(i, dl != 0.0 ? __ldcg(pw + i) * brdc_rcp(dl) : 0.0);
    }
}

__device__ __forceinline__ void rows_store(const Ws &w, long long po, int s,
                                           const double (&f)[3]) {
    const double nrm = sqrt(f[0]);
    w.rf[po + s] = nrm > 0.0 ? f[1] / nrm : 0.0;
    w.rl[po + s] = nrm > 0.0 ? f[2] / nrm : 0.0;
}

__device__ void box_rows(const KArgs &a, BoxSmem &S) {
    const Ws &w = a.w;
    const int lane = threadIdx.x & 31;
    double *cf = S.coef[threadIdx.x >> 5];
    // the last roots by whole blocks
    box_merges(a, true, [&](const NodeGeom &G, int g, int K) {
        const long long po = G.poff;
        double f[3] = {0.0, 0.0, 0.0};
        rows_span(w, po, __ldcg(w.rdo + po + K - 1), __ldcg(w.rtau + po + K - 1), threadIdx.x, K,
                  kSweepThreads, f);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            f[c] = block_sum<kSweepThreads>(f[c], S.red);
        }
        if (threadIdx.x == 0) {
            rows_store(w, po, K - 1, f);
        }
    });
    box_runs(a, true, [&](const NodeGeom &G, int g, int K, int r0, int Rw, int tpr, long long sb,
                          const BoxHdr &H) {
        const long long po = G.poff;
        const bool far = H.far(K);
        if (far) {
            __syncwarp();
            box_coef(cf, w.nl + sb);
            box_coef(cf + kBoxP, w.nl + sb + kBoxP);
            box_coef(cf + 2 * kBoxP, w.nf + sb);
            __syncwarp();
        }
        const int s = r0 + lane / tpr, l = lane & (tpr - 1);
        const bool active = s < K - 1;
        double f[3] = {0.0, 0.0, 0.0};
        if (active) {
            const double dorg = __ldcg(w.rdo + po + s), tau = __ldcg(w.rtau + po + s);
            rows_span(w, po, dorg, tau, H.nlo + l, H.nhi, tpr, f);
            if (far) {
                const double t = ((dorg - H.mid) + tau) * H.ih;
                for (int q = l; q < 3; q += tpr) {
                    const double v = box_eval(cf + q * kBoxP, t);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        f[c] += c == q ? v : 0.0;
                    }
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            f[c] = group_sum(f[c], tpr);
        }
        if (active && l == 0) {
            rows_store(w, po, s, f);
        }
    });
}

// The merges of level a.k with more than a.big_k poles, in one cooperative
// launch; it returns at once when the level plan has none.  rows = 0: every
// merge is an instance root.
__global__ void __launch_bounds__(kSweepThreads, 2) k_box(KArgs a, int rows, long long total_n) {
    pdl_begin();
    if (halted(a.w.hdr)) {
        return;
    }
    WsHeader *h = a.w.hdr;
    LevelCtl *ctl = &h->lvl[a.k];
    if (__ldcg(&ctl->items_w) == 0) {
        return;
    }
    __shared__ BoxSmem S;
    for (int i = threadIdx.x; i < 4 * kBoxP; i += kSweepThreads) {
        S.cosv[i] = cospi(i / (2.0 * kBoxP));
    }
    __syncthreads();
    box_far<kBoxSecular>(a, S);
    if (!grid_barrier(h, ctl)) {
        return;
    }
    box_last_root(a, S);
    box_secular(a, S);
    if (!grid_barrier(h, ctl)) {
        return;
    }
    if (rows) {
        box_far<kBoxLowner>(a, S);
        if (!grid_barrier(h, ctl)) {
            return;
        }
        box_lowner(a, S);
        if (!grid_barrier(h, ctl)) {
            return;
        }
        box_far<kBoxRows>(a, S);
        if (!grid_barrier(h, ctl)) {
            return;
        }
        box_rows(a, S);
        if (!grid_barrier(h, ctl)) {
            return;
        }
    }
    place_rows(a, total_n);
}

} // namespace brdc
