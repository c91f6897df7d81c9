// brdc_leaf.cuh -- one eigenpair of a leaf (at most 16 rows) per thread.
//
// A leaf of the merge tree needs its eigenvalues and the first and last
// rows of its eigenvector matrix.  The leaf is tridiagonal, so thread i of a
// half-warp finds eigenpair i by itself, with no exchange of columns:
//   * eigenvalue i inside a bracket kept by Sturm counts (sign changes of
//     the leading principal minors of T - x, W. Givens), by Newton steps on
//     det(T - x) once the bracket holds one eigenvalue, by bisection until
//     then;
//   * its eigenvector from the twisted factorisation of T - lambda at the
//     index of the smallest pivot (K. V. Fernando, "On computing an
//     eigenvector of a tridiagonal matrix", SIAM J. Matrix Anal. Appl. 18,
//     1997), with the Rayleigh-quotient correction of lambda that the
//     factorisation yields.
// Such vectors have residuals of rounding size, but are orthogonal only to
// rounding / gap.  The half-warp therefore forms F = V^T V - I and corrects
// V to V (I - F/2) (the first terms of P.-O. Loewdin's symmetric
// orthogonalisation V (I + F)^(-1/2)), which leaves |F|^2.  The result is
// checked: a leaf whose residual, gap or |F| is outside the bounds below,
// or that is nearly diagonal, is left to the Jacobi solver.
#pragma once

#include "brdc_secular.cuh"

namespace brdc {

constexpr int kLeafN = 16;           // rows of a leaf, padded
constexpr int kLeafStride = 18;      // doubles per row of the scratch (below)
constexpr double kLeafPad = 64.0;    // diagonal of the padding rows (the scaled leaf is <= 1)
constexpr int kLeafMaxEval = 40;     // evaluations of det(T - x) before a leaf is given up
constexpr double kLeafNewton = 1e-11;   // a Newton step this short ends the iteration: the
                                        // error left is its square over the gap
constexpr double kLeafSlack = 1e-13;    // a Newton point this far past its bracket is taken
constexpr double kLeafGap = 0x1p-23;    // smallest gap (1.2e-7) the vectors are taken at
constexpr double kLeafResid = 0x1p-47;  // largest |T v - lambda v| (7e-15; the norm is ~1)
constexpr double kLeafOrth = 0x1p-27;   // largest |F| the correction takes (F^2 < 6e-17)
constexpr double kLeafOffDiag = 0x1p-10; // a leaf whose couplings are all below this share of
                                         // its norm is nearly diagonal: Jacobi needs two or
                                         // three sweeps, and gaps may be as small as e^2
constexpr double kLeafTiny = 1e-30;     // pivots are moved away from zero by this much

// The scratch of one leaf: row k holds eigenvector k (16 entries), d_k and
// e_k^2 (e_k couples rows k and k+1); the scaled leaf, rows past its end
// decoupled (e = 0) with diagonal kLeafPad.
struct LeafScratch {
    double v[kLeafN][kLeafStride];
    double e[kLeafN];
};

// det(T - x), its derivative and the number of eigenvalues below x, by the
// three-term recurrence of the leading minors.  Written with explicit FMAs,
// so every kernel that calls it gets the same bits.
__host__ __device__ inline int leaf_minors(const LeafScratch &B, double x, double *det,
                                           double *ddet) {
    double p0 = 1.0, q0 = 0.0;
    double p1 = B.v[0][kLeafN] - x, q1 = -1.0;
    int count = p1 < 0.0 ? 1 : 0;
#pragma unroll
    for (int k = 1; k < kLeafN; ++k) {
        const double t = B.v[k][kLeafN] - x, e2 = B.v[k - 1][kLeafN + 1];
        const double p = fma(t, p1, -(e2 * p0));
        const double q = fma(t, q1, -fma(e2, q0, p1));
        count += (p < 0.0) != (p1 < 0.0);
        p0 = p1;
        q0 = q1;
        p1 = p;
        q1 = q;
    }
    *det = p1;
    *ddet = q1;
    return count;
}

// The bracket (a, b] of eigenvalue i: ca and cb eigenvalues lie below a and
// b, ca <= i < cb.
struct LeafRoot {
    double a, b, x;
    int ca, cb;
    int state; // 0 iterating, 1 found (x), 2 given up
};

// Take the counts and minors at r.x and choose the next point.
__host__ __device__ inline void leaf_advance(LeafRoot &r, int i, int count, double det,
                                             double ddet) {
    if (count <= i) {
        r.a = r.x;
        r.ca = count;
    } else {
        r.b = r.x;
        r.cb = count;
    }
    double next = 0.5 * (r.a + r.b);
    const bool alone = r.cb - r.ca == 1;
    if (alone) {
        const double step = det * brdc_rcp(ddet);
        const double cand = r.x - step;
        if (fabs(step) <= kLeafNewton) {
            r.x = cand;
            r.state = 1;
            return;
        }
        // (an eigenvalue may sit on the end of its bracket)
        if (cand > r.a - kLeafSlack && cand < r.b + kLeafSlack) {
            next = cand;
        }
    }
    if (r.b - r.a <= (alone ? 0x1p-51 : kLeafGap)) {
        r.x = next;
        r.state = alone ? 1 : 2; // a pair closer than the vectors allow
        return;
    }
    r.x = next;
}

__host__ __device__ inline double leaf_pivot(double t) {
    return fabs(t) < kLeafTiny ? kLeafTiny : t;
}

// Eigenvector of the eigenvalue nearest *lambda (a simple one), with the
// corrected eigenvalue; returns the largest residual entry.  s = rows of
// the leaf (the padding rows get 0); the 16 entries of row x of the scratch
// are this lane's own (they keep a 16-row array out of its registers).
__host__ __device__ inline double leaf_vector(LeafScratch &B, int x, int s, double *lambda,
                                              double (&v)[kLeafN]) {
    const double lam = *lambda;
    // ratios of neighbouring entries from the bottom (U, in the scratch) and
    // the top (L): v_{k+1} = -U_k v_k below the twist, v_k = -L_k v_{k+1}
    // above it
    double L[kLeafN];
    {
        double t = B.v[kLeafN - 1][kLeafN] - lam;
#pragma unroll
        for (int k = kLeafN - 2; k >= 0; --k) {
            const double u = B.e[k] * brdc_rcp(leaf_pivot(t));
            B.v[x][k] = u;
            t = fma(-B.e[k], u, B.v[k][kLeafN] - lam);
        }
    }
    // the pivot of a twist at k: d_k - lambda less what both sides eliminate
    double gam = 1e300;
    int tw = 0;
    {
        double t = B.v[0][kLeafN] - lam;
#pragma unroll
        for (int k = 0; k < kLeafN; ++k) {
            const double g = k + 1 < kLeafN ? fma(-B.e[k], B.v[x][k], t) : t;
            if (k < s && fabs(g) < fabs(gam)) {
                gam = g;
                tw = k;
            }
            if (k + 1 < kLeafN) {
                L[k] = B.e[k] * brdc_rcp(leaf_pivot(t));
                t = fma(-B.e[k], L[k], B.v[k + 1][kLeafN] - lam);
            }
        }
        L[kLeafN - 1] = 0.0;
    }
#pragma unroll
    for (int k = 0; k + 1 < kLeafN; ++k) {
        L[k] = k < tw ? L[k] : B.v[x][k];
    }
    double ss = 0.0, t = 0.0;
#pragma unroll
    for (int k = kLeafN - 1; k >= 0; --k) {
        t = k == tw ? 1.0 : k < tw ? -L[k] * t : 0.0;
        v[k] = t;
    }
    t = 0.0;
#pragma unroll
    for (int k = 1; k < kLeafN; ++k) {
        t = k - 1 < tw ? 0.0 : -L[k - 1] * (k - 1 == tw ? 1.0 : t);
        v[k] = k > tw ? t : v[k];
    }
#pragma unroll
    for (int k = 0; k < kLeafN; ++k) {
        ss = fma(v[k], v[k], ss);
    }
    const double inv = brdc_rcp(sqrt(ss));
#pragma unroll
    for (int k = 0; k < kLeafN; ++k) {
        v[k] = v[k] * inv;
    }
    const double lam2 = fma(gam * inv, inv, lam);
    double res = 0.0;
#pragma unroll
    for (int k = 0; k < kLeafN; ++k) {
        double r = (B.v[k][kLeafN] - lam2) * v[k];
        if (k > 0) {
            r = fma(B.e[k - 1], v[k - 1], r);
        }
        if (k + 1 < kLeafN) {
            r = fma(B.e[k], v[k + 1], r);
        }
        // a NaN fails the caller's test too
        res = fabs(r) <= res ? res : fabs(r);
    }
    *lambda = lam2;
    return res;
}

#if defined(__CUDACC__)

__device__ __forceinline__ double half_max(double v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    }
    return v;
}

// The leaf (d, e) of s rows by the half-warp whose lane x passes d_x and
// e_x = |coupling of rows x and x+1| (0 where there is none).  Both halves
// of a warp call it, each with its own leaf and scratch.  Returns whether
// this half's leaf was solved: lane x < s then holds eigenvalue x
// (ascending) and row entries 0 and s-1 of its eigenvector, or with FULL
// the whole vector in vf.  The result depends on the leaf alone.
template <bool FULL>
__device__ inline bool leaf_pairs(LeafScratch &B, double dx, double ex, int s, int x,
                                  double *key, double *v0, double *v1,
                                  double (&vf)[kLeafN]) {
    constexpr unsigned full = 0xffffffffu;
    const unsigned half = 0xffffu << (threadIdx.x & 16);
    const double amax = half_max(fmax(fabs(dx), ex));
    const double emax = half_max(ex);
    bool ok = s >= 2 && emax > kLeafOffDiag * amax && amax > 1e-280 && amax < 1e280;
    if (!__any_sync(full, ok)) {
        return false;
    }
    // scaled by a power of two to a norm in [0.5, 1): no minor over- or
    // underflows, and the bounds above are absolute
    const int eb = ok ? (__double2hiint(amax) >> 20) & 0x7ff : 1022;
    const double sc = __hiloint2double((2045 - eb) << 20, 0);
    const double un = __hiloint2double((eb + 1) << 20, 0);
    const double d = dx * sc, e = ex * sc;
    const double ep = __shfl_up_sync(full, e, 1, 16);
    const bool row = x < s;
    const double rad = e + (x > 0 ? ep : 0.0);
    // Gershgorin's bounds, widened so that Newton steps may pass an
    // eigenvalue that lies on one (Toeplitz leaves have it)
    const double gh = half_max(row ? d + rad : -8.0);
    const double gl = -half_max(row ? rad - d : -8.0);
    const double wide = fma(0x1p-5, gh - gl, 0x1p-48);
    const double hi = gh + wide, lo = gl - wide;
    __syncwarp();
    B.v[x][kLeafN] = row ? d : kLeafPad;
    B.v[x][kLeafN + 1] = e * e;
    B.e[x] = e;
    __syncwarp();

    // 16 equidistant points give every lane its first bracket
    const double w = (hi - lo) * (1.0 / 17.0);
    LeafRoot r;
    {
        double p, q;
        const int c = leaf_minors(B, fma(w, (double)(x + 1), lo), &p, &q);
        int below = 0;
        r.ca = 0;
        r.cb = s;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int cj = __shfl_sync(full, c, j, 16);
            if (cj <= x) {
                ++below;
                r.ca = cj;
            } else {
                r.cb = min(r.cb, cj);
            }
        }
        r.a = fma(w, (double)below, lo);
        r.b = fma(w, (double)(below + 1), lo);
        r.x = 0.5 * (r.a + r.b);
        r.state = ok && row ? 0 : 1;
    }
    for (int it = 0; it < kLeafMaxEval && __any_sync(full, r.state == 0); ++it) {
        double p, q;
        // the leaf is read again at every point: kept in registers across
        // the loop it would take half of them
        asm volatile("" ::: "memory");
        const int c = leaf_minors(B, r.x, &p, &q);
        if (r.state == 0) {
            leaf_advance(r, x, c, p, q);
        }
    }
    double lam = r.x;
    {
        const double up = __shfl_down_sync(full, lam, 1, 16);
        const bool bad = row && (r.state != 1 || (x + 1 < s && !(up - lam > kLeafGap)));
        const unsigned bb = __ballot_sync(full, bad); // by all lanes, whatever their ok
        ok = ok && (bb & half) == 0u;
    }
    if (!__any_sync(full, ok)) {
        return false;
    }
    double v[kLeafN];
    const double res = leaf_vector(B, x, s, &lam, v);
    bool bad = !(res <= kLeafResid);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kLeafN; k += 2) {
        *reinterpret_cast<double2 *>(&B.v[x][k]) =
            row ? make_double2(v[k], v[k + 1]) : make_double2(0.0, 0.0);
    }
    __syncwarp();
    double a0 = 0.0, a1 = 0.0, acc[kLeafN];
#pragma unroll
    for (int k = 0; k < kLeafN; ++k) {
        acc[k] = 0.0;
    }
    const int last = s > 0 ? s - 1 : 0;
    double vl = 0.0;
#pragma unroll
    for (int k = 0; k < kLeafN; ++k) {
        vl = k == last ? v[k] : vl;
    }
#pragma unroll 2
    for (int i = 0; i < kLeafN; ++i) {
        double u[kLeafN];
#pragma unroll
        for (int k = 0; k < kLeafN; k += 2) {
            const double2 t = *reinterpret_cast<const double2 *>(&B.v[i][k]);
            u[k] = t.x;
            u[k + 1] = t.y;
        }
        double f0 = i == x ? -1.0 : 0.0, f1 = 0.0;
#pragma unroll
        for (int k = 0; k < kLeafN; k += 2) {
            f0 = fma(u[k], v[k], f0);
            f1 = fma(u[k + 1], v[k + 1], f1);
        }
        const double F = __dadd_rn(f0, f1);
        bad |= i < s && !(fabs(F) <= kLeafOrth);
        if (FULL) {
#pragma unroll
            for (int k = 0; k < kLeafN; ++k) {
                acc[k] = fma(F, u[k], acc[k]);
            }
        } else {
            a0 = fma(F, u[0], a0);
            a1 = fma(F, B.v[i][last], a1);
        }
    }
    if (FULL) {
#pragma unroll
        for (int k = 0; k < kLeafN; ++k) {
            vf[k] = fma(-0.5, acc[k], v[k]);
        }
    } else {
        *v0 = fma(-0.5, a0, v[0]);
        *v1 = fma(-0.5, a1, vl);
    }
    *key = lam * un;
    const unsigned bb = __ballot_sync(full, row && bad);
    return ok && (bb & half) == 0u;
}

#endif

} // namespace brdc
