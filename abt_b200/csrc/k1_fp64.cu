// k1_fp64.cu -- FP64 far-field sum in the reference's arithmetic (the plain drop-in).
//
// One thread per far-field bin; each thread walks a run of the facet list in order and
// adds every facet's 2x2 complex amplitude to its bin.  Within a run the order is the
// reference's, ((0 + c_1) + c_2) + ... (src/diff_mod.f90:744-766), in fused
// multiply-adds and the circular basis; a list is one run on large grids and up to 64 on
// small ones (k1_launch), whose sums are added in run order.
//
// The rounding of a few quantities decides the result far above 1e-16 and they
// are formed operation by operation as the reference forms them: the rotated
// bin (x3, y3, z3), its distance and the phase bvs = k |x3| ~ 1e7 rad
// (src/diff_mod.f90:576-618, 357-360), the aperture wave vector (kxx, kyy), the
// field-of-view test next to its threshold, and the whole contour integral
// (:357-428) in bins where its terms cancel.  Everything else of a facet x bin
// takes the shortest form of the same value, which differs by a few ulp:
// * Away from the cancellation the contour sum of a triangle equals
//   2 i A e^{i bvs} sum_j e^{i d_j} / prod_{k != j} (d_j - d_k), d_j the vertex
//   phases: one sincos a vertex and one reciprocal, where the contour takes
//   three sincos and two reciprocals an edge.  A polygon takes its edges with
//   one sincos and one reciprocal each.
// * The reference's noise in an edge's term is about ulp(d) L / (min(|kxx|,
//   |kyy|) |omega|), omega the phase step along the edge, L the edge's extent.
//   A lane with omega_min * min(|kxx|, |kyy|) below the facet's `cond`
//   (K1Facet; ulp(max(|d|, 1)), since cosines near 1 are known to 1.1e-16 only) has a
//   noise above 5e-11 of the facet's area and takes the contour itself, so both agree to
//   5e-11 of the area everywhere.  Facets with a clamped edge slope (:379-382) always
//   take it.
// * The polarisation block (karczewski :124-198 and the scattering-plane
//   rotation :628-658) reduces, away from the clamp of ky, to A = sc (P d + Q e),
//   B = sc (P e - Q d) with d = -(Kz t + kz), e = -kx ky, t = kx^2 + kz^2, h = (b, -a, 0) the incidence direction times the unit
//   direction (a, b, c) from the facet, P = y . h, Q = y_z |h|^2 - c (y_x a + y_y b)
//   (y the aperture frame's second axis) and sc = 1 / (2 |h| t); in the forward bodge
//   (:630-633) with h from another bin, not normal to (a, b, c).
// * [[A, B], [-B, A]] is diagonal in the columns' circular basis u+- = a1 +- i a2,
//   in which the sums are kept; the basis change and the rotation T(phi), which
//   depends on the bin alone, are applied once at the end.
//
// Bound: FP64 pipe (66 % of cycles; 351 instructions a triangle and bin, 191 of them FP64,
// and 331 and 185 on 2,000 triangles x 259,560 bins, where fewer lanes take the contour;
// 1,813 with every operation of the reference).  A triangle list of
// 2,582 x 32,580 bins takes 1.42 ms (5.9e10 facet-bin/s), the operation-by-operation
// kernel took 6.92 ms (1.59 ms with quadrant polynomials in place of the table of
// roots, 1.51 ms with the forward bodge in the aperture frame).  The facet records go
// through shared memory, three stages of 16 and one barrier a stage: read from global
// memory they cost 38 % of the issue slots in load waits; a private stage per warp,
// without barriers, measured 3 % slower.
//
// The file is built with -fmad=false: a multiply-add is fused only where fma()
// is written.  Facet frames come from the host (host_setup.cpp); the bin grid
// and cos/sin(phi) are libm values.
#include <float.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <mutex>

#include "frame.h"
#include "k1_math.cuh"
#include "pbt_internal.h"

namespace pbt {

namespace {

struct Z {
    double re, im;
};
__device__ __forceinline__ Z zmul(Z a, Z b) {
    return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}

__device__ __forceinline__ void cross_n(const double a[3], const double b[3], double c[3]) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
    double nf = sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
    c[0] = c[0] / nf;
    c[1] = c[1] / nf;
    c[2] = c[2] / nf;
}
__device__ __forceinline__ double dot_3(const double a[3], const double b[3]) {
    double s = 0.0;
    s = s + a[0] * b[0];
    s = s + a[1] * b[1];
    s = s + a[2] * b[2];
    return s;
}

// contour_integral for one bin (src/diff_mod.f90:357-428), operation by operation
__device__ __noinline__ void contour_ref(const K1Facet *__restrict__ F, const K1Edge *__restrict__ E,
                                         double waveno, double lambda, double x3, double y3,
                                         double bvs, Z *out) {
    const int nv = (int)F->nv;
    double kxx = F->kinc0 - waveno * waveno * x3 / bvs;
    double kyy = F->kinc1 - waveno * waveno * y3 / bvs;
    Z eK;
    sincos(bvs, &eK.im, &eK.re);
    if (fabs(kxx) < kLit1em6) kxx = kLit1em6;
    if (fabs(kyy) < kLit1em6) kyy = kLit1em6;
    Z area = {0, 0};
    for (int j = 0; j < nv; j++) {
        const double xj = E[j].xj, yj = E[j].yj, mj = E[j].mj, nj = E[j].nj;
        const double dx = E[j].dx, dy = E[j].dy;
        const double delta = kxx * xj + kyy * yj;
        const double delta1 = kyy * mj + kxx;
        const double delta2 = kxx * nj + kyy;
        const double omega1 = dx * delta1;
        const double omega2 = dy * delta2;
        const double alpha = 1 / (2 * kyy * delta1);
        const double beta = 1 / (2 * kxx * delta2);
        double s0, c0d, s1, c1d, s2, c2d;
        sincos(delta, &s0, &c0d);
        sincos(delta + omega1, &s1, &c1d);
        sincos(delta + omega2, &s2, &c2d);
        const double sumim = alpha * (c0d - c1d) - beta * (c0d - c2d);
        const double sumre = -(alpha * (s0 - s1)) + beta * (s0 - s2);
        Z t = zmul(eK, Z{sumre, sumim});
        t.re = t.re / lambda;
        t.im = t.im / lambda;
        area.re = area.re + t.re;
        area.im = area.im + t.im;
    }
    *out = area;
}

// The polarisation block where the clamp of ky or the forward bodge applies
// (src/diff_mod.f90:124-198, 628-658): A and B of rot4 . D = [[A, B], [-B, A]].
// h: the direction from the facet to the bodge's bin, aperture frame.
__device__ __noinline__ void polar_ref(const K1Facet *__restrict__ F, double kx, double ky, double kz,
                                       double hx, double hy, double hz, double *A, double *B) {
    double k[3] = {kx, ky, kz};
    const double inc2[3] = {F->inc2[0], F->inc2[1], F->inc2[2]};
    if (fabs(k[1]) > kLit0_999999) k[1] = copysign(kLit0_999999, k[1]);
    const double Kx = F->Kx, Ky = F->Ky, Kz = F->Kz;
    const double sq = sqrt(1 - k[1] * k[1]);
    const double m[3] = {-(k[0] * k[1] / sq), sq, -(k[1] * k[2] / sq)};
    const double frac = sqrt((1 - k[1] * k[1]) / (1 - Ky * Ky));
    const double d = 0.5 * (-Kz * frac + -k[2] / frac);
    const double e = 0.5 * (-(k[0] * k[1] / frac) + Kx * Ky * frac);
    double hc[3], evo2[3];
    if (fabs(dot_3(inc2, k)) < kLit0_999) {
        cross_n(inc2, k, hc);
    } else {
        const double hk[3] = {hx, hy, hz};
        cross_n(inc2, hk, hc);
    }
    cross_n(k, m, evo2);
    const double p = dot_3(hc, m), r = dot_3(hc, evo2);
    *A = p * d + r * e;
    *B = p * e - r * d;
}

constexpr int K1_THREADS = 128;
constexpr int K1_CH = 16;   // facets per shared-memory stage
constexpr int K1_NST = 3;   // stages
// 96 registers for five CTAs an SM: 1.64 ms against 1.72 at four (128 registers) and
// 2.01 at six (80, spilling) on 1,700 + 882 triangles x 32,580 bins
constexpr int K1_MINB = 5;
constexpr int K1_WAVES = 32;  // CTAs per resident slot that the runs of a small grid aim at

struct K1Args {
    const K1Facet *fac;
    const K1Edge *edges;
    const double *xyz, *phitab;
    int64_t nphi, nb, theta_i;
    double waveno, lambda;
    // list k: facets [first[k], first[k] + n[k]) in `split[k]` runs of `run[k]` facets
    int64_t first[2], n[2], run[2];
    int split[2];
    double *grid[2];  // output grid of each list
    double *part;     // partial grids of the runs of a list with more than one
};

// facets [f0, f0 + n) into a stage, 16 bytes a thread and step
__device__ __forceinline__ void k1_stage(K1Facet *dst, const K1Facet *src, int n) {
    const char *s = reinterpret_cast<const char *>(src);
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    for (int b = threadIdx.x * 16; b < n * (int)sizeof(K1Facet); b += K1_THREADS * 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + b), "l"(s + b) : "memory");
}

// One thread per bin; blockIdx.y selects a run of one list's facets, walked in
// order and written to the list's grid, or to its partial grid for k1_sum_kernel.
template <bool FAST>
__global__ void __launch_bounds__(K1_THREADS, K1_MINB) k1_kernel(const K1Args P) {
    __shared__ K1Facet sfac[K1_NST][K1_CH];
    __shared__ double2 s_root[kRoots];  // see sincos_n; the first stage's barrier publishes it
    static_assert(K1_THREADS == kRoots, "one root a thread");
    sincospi(threadIdx.x * (2.0 / kRoots), &s_root[threadIdx.x].y, &s_root[threadIdx.x].x);
    const int kind = (int)blockIdx.y >= P.split[0];
    const int run = (int)blockIdx.y - (kind ? P.split[0] : 0);
    const int64_t fb = P.first[kind] + run * P.run[kind];
    const int64_t nf = max((int64_t)0, min(P.run[kind], P.first[kind] + P.n[kind] - fb));
    const int64_t nb = P.nb;
    // tiles from both ends of the grid inwards: the poles' rows, whose polarisation
    // takes the longer form, go first and not into the launch's tail
    const int64_t tile = blockIdx.x & 1 ? gridDim.x - 1 - (blockIdx.x >> 1) : blockIdx.x >> 1;
    const int64_t o_ = tile * K1_THREADS + threadIdx.x;
    const bool in = o_ < nb;
    const int64_t o = in ? o_ : nb - 1;
    const int64_t i = o % P.nphi;
    const double X = P.xyz[o], Y = P.xyz[nb + o], Zc = P.xyz[2 * nb + o];
    const double waveno = P.waveno, lambda = P.lambda;
    // u+- of column b: acc[b], acc[2 + b]
    Z acc[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
    // two stages in flight; the one barrier of a stage also frees the stage before it
    for (int c = 0; c < 2; c++) {
        if (c * K1_CH < nf)
            k1_stage(sfac[c], P.fac + fb + c * K1_CH, (int)min((int64_t)K1_CH, nf - c * K1_CH));
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int st = 0;
    for (int64_t f0 = 0; f0 < nf; f0 += K1_CH) {
        const int cnt = (int)min((int64_t)K1_CH, nf - f0);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const int64_t f2 = f0 + 2 * K1_CH;
        if (f2 < nf)
            k1_stage(sfac[st == 0 ? 2 : st - 1], P.fac + fb + f2, (int)min((int64_t)K1_CH, nf - f2));
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (int j = 0; j < cnt; j++) {
            const K1Facet *F = &sfac[st][j];
            const double2 *v = reinterpret_cast<const double2 *>(F);
            const double2 v0 = v[0], v1 = v[1];  // com, kinc0
            const double x1 = X - v0.x, y1 = Y - v0.y, z1 = Zc - v1.x;
            if (FAST) {
                // the field-of-view test (src/diff_mod.f90:593-603); within 1e-12 of the
                // threshold with the reference's roundings
                const double p0[3] = {F->prop0[0], F->prop0[1], F->prop0[2]};
                const double q1 = x1 * x1 + y1 * y1 + z1 * z1;
                const double d = fma(z1, p0[2], fma(y1, p0[1], x1 * p0[0])) * rsqrt_n(q1) - F->cos_fov;
                if (d < -1e-12) continue;  // outside the field of view
                if (!(d > 1e-12)) {
                    const double r1 = sqrt(q1);
                    const double vec[3] = {x1 / r1, y1 / r1, z1 / r1};
                    if (dot_3(vec, p0) < F->cos_fov) continue;
                }
            }
            // R: v2..v5 and half of v6
            const double2 v2 = v[2], v3 = v[3], v4 = v[4], v5 = v[5], v6 = v[6], v7 = v[7];
            const double x3 = v2.x * x1 + v2.y * y1 + v3.x * z1;
            const double R3 = v3.y, R4 = v4.x, R5 = v4.y;
            const double y3 = R3 * x1 + R4 * y1 + R5 * z1;
            const double z3 = v5.x * x1 + v5.y * y1 + v6.x * z1;
            // |x3| rounded once and its reciprocal; the phase; the aperture wave vector
            const double q3 = x3 * x3 + y3 * y3 + z3 * z3;
            const double ir = rsqrt_n(q3);
            double rr = q3 * ir;
            rr = fma(fma(-rr, rr, q3), 0.5 * ir, rr);
            const double bvs = waveno * rr;
            // polarisation
            const double kx = x3 * ir, ky = y3 * ir, kz = z3 * ir;
            const double a = x1 * ir, b = y1 * ir, c = z1 * ir;
            double A, B;
            const double fc = fabs(c);
            // the reference's roundings decide next to the bodge's limit (:630)
            if (fabs(fc - kLit0_999) > 1e-9 && fabs(ky) < kLit0_999999) {
                const double tt = fma(kx, kx, kz * kz);
                double hn2, Pp, Q;
                if (fc < kLit0_999) {
                    hn2 = fma(a, a, b * b);
                    Pp = fma(R3, b, -(R4 * a));
                    Q = fma(R5, hn2, -(c * fma(R4, b, R3 * a)));
                } else {
                    // forward bodge: h = (p, q, 0) from the bin at the same phi and theta
                    // index theta_i, no longer normal to k:
                    // P = y . h - ky (h . k), Q = -y . (k x h)
                    const int64_t oh = i + P.nphi * P.theta_i;
                    const double xh = P.xyz[oh] - v0.x, yh = P.xyz[nb + oh] - v0.y,
                                 zh = P.xyz[2 * nb + oh] - v1.x;
                    const double ih = rsqrt_n(fma(zh, zh, fma(yh, yh, xh * xh)));
                    const double p = yh * ih, q = -(xh * ih);
                    hn2 = fma(p, p, q * q);
                    Pp = fma(R4, q, R3 * p) - ky * fma(q, b, p * a);
                    Q = fma(c, fma(R3, q, -(R4 * p)), -(R5 * fma(a, q, -(b * p))));
                }
                const double d = -fma(v7.x, tt, kz), e = -(kx * ky);
                const double sc = 0.5 * rsqrt_n((hn2 * tt) * tt);
                A = sc * fma(Pp, d, Q * e);
                B = sc * fma(Pp, e, -(Q * d));
            } else {
                const int64_t oh = i + P.nphi * P.theta_i;
                const double xh = P.xyz[oh] - F->com[0], yh = P.xyz[nb + oh] - F->com[1],
                             zh = P.xyz[2 * nb + oh] - F->com[2];
                const double rh = sqrt(xh * xh + yh * yh + zh * zh);
                const double x3h = v2.x * xh + v2.y * yh + v3.x * zh;
                const double y3h = R3 * xh + R4 * yh + R5 * zh;
                const double z3h = v5.x * xh + v5.y * yh + v6.x * zh;
                polar_ref(F, kx, ky, kz, x3h / rh, y3h / rh, z3h / rh, &A, &B);
            }
            // aperture integral; the phase bvs = nK h + rK joins each vertex phase
            const int nv = (int)F->nv;
            const double kxx = fma(-waveno, kx, v1.y), kyy = fma(-waveno, ky, v6.y);
            int nK;
            const double rK = reduce_n(bvs, &nK);
            Z g;
            // a lower bound of min |omega| * min(|kxx|, |kyy|) from the high words; the
            // contour also takes the reference's floor of 1e-6 under |kxx| and |kyy|
            auto top = [](double x) { return __double2hiint(x) & 0x7fffffff; };
            const int kmin = min(top(kxx), top(kyy));
            const double kfloor = kmin > top(kLit1em6) ? __hiloint2double(kmin, 0) : 0.0;
            bool contour;
            if (nv == 3) {
                // xy: v12..v14, dxy: v15, v16
                const double2 e0 = v[15], e1 = v[16];
                const double w0 = fma(kyy, e0.y, kxx * e0.x), w1 = fma(kyy, e1.y, kxx * e1.x);
                const double wl = -(w0 + w1);
                const int wmin = min(min(top(w0), top(w1)), top(wl));
                contour = !(__hiloint2double(wmin, 0) * kfloor >= F->cond);
                if (!contour) {
                    const double2 p0 = v[12], p1 = v[13], p2 = v[14];
                    double s0, c0, s1, c1, s2, c2;
                    sincos_n(fma(kyy, p0.y, fma(kxx, p0.x, rK)), nK, s_root, &s0, &c0);
                    sincos_n(fma(kyy, p1.y, fma(kxx, p1.x, rK)), nK, s_root, &s1, &c1);
                    sincos_n(fma(kyy, p2.y, fma(kxx, p2.x, rK)), nK, s_root, &s2, &c2);
                    // i sum_j e_j / prod (d_j - d_k) = -i (e_0 w1 + e_1 w2 + e_2 w0) / (w0 w1 w2)
                    const double t = v7.y * rcp_n(w0 * w1 * wl);
                    g.re = fma(s2, w0, fma(s1, wl, s0 * w1)) * t;
                    g.im = fma(c2, w0, fma(c1, wl, c0 * w1)) * -t;
                }
            } else {
                // edges: (1 / (2 kxx kyy)) sum_j (kxx dx - kyy dy) / omega_j (e_j - e_{j+1})
                const K1Edge *E = P.edges + F->edge_off;
                int wmin = 0x7fffffff;
                for (int q = 0; q < nv; q++)
                    wmin = min(wmin, top(fma(kyy, E[q].dy, kxx * E[q].dx)));
                contour = !(__hiloint2double(wmin, 0) * kfloor >= F->cond);
                if (!contour) {
                    double s0, c0, sp, cp;
                    g = {0, 0};
                    sincos_n(fma(kyy, E[0].yj, fma(kxx, E[0].xj, rK)), nK, s_root, &s0, &c0);
                    sp = s0;
                    cp = c0;
                    for (int q = 0; q < nv; q++) {
                        const double kdx = kxx * E[q].dx;
                        const double w = fma(-kyy, E[q].dy, kdx) * rcp_n(fma(kyy, E[q].dy, kdx));
                        double sn = s0, cn = c0;
                        if (q + 1 < nv)
                            sincos_n(fma(kyy, E[q + 1].yj, fma(kxx, E[q + 1].xj, rK)), nK, s_root, &sn, &cn);
                        g.re = fma(w, sn - sp, g.re);
                        g.im = fma(w, cp - cn, g.im);
                        sp = sn;
                        cp = cn;
                    }
                    const double t = rcp_n(2.0 * lambda * kxx * kyy);
                    g.re *= t;
                    g.im *= t;
                }
            }
            if (contour) contour_ref(F, P.edges + F->edge_off, waveno, lambda, x3, y3, bvs, &g);
            // u+- take g (A -+ i B)
            const double gxB = g.re * B, gyB = g.im * B;
            const Z qp = {fma(g.re, A, gyB), fma(g.im, A, -gxB)},
                    qm = {fma(g.re, A, -gyB), fma(g.im, A, gxB)};
#pragma unroll
            for (int col = 0; col < 4; col++) {
                const Z q = col < 2 ? qp : qm;
                const double2 u = v[8 + col];
                acc[col].re = fma(q.re, u.x, fma(-q.im, u.y, acc[col].re));
                acc[col].im = fma(q.re, u.y, fma(q.im, u.x, acc[col].im));
            }
        }
        st = st == 2 ? 0 : st + 1;
    }
    if (!in) return;
    double *out = P.split[kind] > 1 ? P.part + (int64_t)blockIdx.y * 8 * nb : P.grid[kind];
    // back from the circular basis, a1 = (u+ + u-)/2, a2 = -i (u+ - u-)/2, then
    // T(phi) = [[-s, -c], [c, -s]] (src/diff_mod.f90:646-650)
    const double cp = P.phitab[i], sp = P.phitab[P.nphi + i];
    Z S[2][2];
#pragma unroll
    for (int col = 0; col < 2; col++) {
        const Z p = acc[col], m = acc[2 + col];
        S[0][col] = {0.5 * (p.re + m.re), 0.5 * (p.im + m.im)};
        S[1][col] = {0.5 * (p.im - m.im), 0.5 * (m.re - p.re)};
    }
#pragma unroll
    for (int row = 0; row < 2; row++) {
        const Z u = S[row][0], v = S[row][1];
        const Z t0 = {v.re * cp - u.re * sp, v.im * cp - u.im * sp};
        const Z t1 = {-(u.re * cp + v.re * sp), -(u.im * cp + v.im * sp)};
        out[2 * (o + nb * row)] = t0.re;
        out[2 * (o + nb * row) + 1] = t0.im;
        out[2 * (o + nb * (2 + row))] = t1.re;
        out[2 * (o + nb * (2 + row)) + 1] = t1.im;
    }
}

// The grid of list blockIdx.y from its runs' partial grids, in run order.
__global__ void k1_sum_kernel(const double *__restrict__ part, int s0, int s1, int64_t n,
                              double *__restrict__ grid0, double *__restrict__ grid1) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int ns = blockIdx.y ? s1 : s0;
    if (t >= n || ns <= 1) return;
    const double *p = part + (blockIdx.y ? (int64_t)s0 * n : 0) + t;
    double s = p[0];
    for (int k = 1; k < ns; k++) s = s + p[k * n];
    (blockIdx.y ? grid1 : grid0)[t] = s;
}

}  // namespace

int k1_launch(pbt_ctx *ctx, cudaStream_t st, const K1Facet *d_fac, int64_t n0, int64_t n1,
              const K1Edge *d_edges, double lambda, int fast_diff, double *d_grid0, double *d_grid1) {
    pbt::NvtxRange nvtx_("pbt: far-field sum (FP64)");
    const GridCache &g = ctx->grid;
    const int64_t blocks = (g.nb + K1_THREADS - 1) / K1_THREADS;
    K1Args A{};
    A.fac = d_fac;
    A.edges = d_edges;
    A.xyz = g.xyz.as<double>();
    A.phitab = g.phitab.as<double>();
    A.nphi = (int64_t)g.phi.size();
    A.nb = g.nb;
    A.theta_i = g.theta_i;
    A.waveno = 2.0 * kPiRef / lambda;
    A.lambda = lambda;
    A.grid[0] = d_grid0;
    A.grid[1] = d_grid1;
    const int64_t n[2] = {n0, n1}, first[2] = {0, n0};
    // A grid with fewer bins than K1_WAVES waves of CTAs leaves SMs idle or its last
    // waves uneven (tiles at the poles and on the contour take longer): the facets go in
    // runs of at least 16 over blockIdx.y (at most 64 runs a list), both lists in one
    // launch, each run into a partial grid of its own.  They are summed in run order, so
    // the result is deterministic; it differs from the one-run order by rounding.
    // Measured on 1,700 + 882 triangles x 32,580 bins: 10 waves 1.48 ms, 14 1.45, 18 1.43,
    // 24 1.42, 32 1.41 with the sum of the partial grids, which takes 37 us of it.
    // The partial grids take 64 B a bin and run, 195 MB on grids of up to 200,000 bins and
    // 600 MB at most (near 3 million); a device without room for them gets fewer runs, at
    // last one a list, which needs none.
    const int64_t resident = (int64_t)ctx->sm_count * K1_MINB;
    const int64_t all = std::max<int64_t>(n0 + n1, 1);
    int ysum = 0;
    bool parts = false;
    for (int64_t waves = K1_WAVES;; waves /= 2) {
        const int64_t runs = (waves * resident + blocks - 1) / blocks;
        for (int k = 0; k < 2; k++) {
            int64_t s = std::min<int64_t>(std::min<int64_t>(runs * n[k] / all, n[k] / 16), 64);
            s = std::max<int64_t>(s, 1);
            A.n[k] = n[k];
            A.first[k] = first[k];
            A.run[k] = std::max<int64_t>((n[k] + s - 1) / s, 1);
            A.split[k] = n[k] > 0 ? (int)((n[k] + A.run[k] - 1) / A.run[k]) : 1;
        }
        if (!d_grid1) A.split[1] = 0;
        ysum = A.split[0] + A.split[1];
        parts = A.split[0] > 1 || A.split[1] > 1;
        if (!parts || ctx->d_k1part.ensure((size_t)ysum * 8 * g.nb * sizeof(double)) == PBT_OK) break;
        clear_error();
    }
    if (parts) A.part = ctx->d_k1part.as<double>();
    timing_begin(ctx, st);
    const dim3 grid((unsigned)blocks, (unsigned)ysum);
    if (fast_diff)
        k1_kernel<true><<<grid, K1_THREADS, 0, st>>>(A);
    else
        k1_kernel<false><<<grid, K1_THREADS, 0, st>>>(A);
    ctx->launches++;
    if (parts) {
        const int64_t n8 = 8 * g.nb;
        k1_sum_kernel<<<dim3((unsigned)((n8 + 255) / 256), d_grid1 ? 2 : 1), 256, 0, st>>>(
            A.part, A.split[0], A.split[1], n8, d_grid0, d_grid1);
        ctx->launches++;
    }
    timing_end(ctx, st);
    PBT_CUDA_TRY(cudaGetLastError());
    return PBT_OK;
}

}  // namespace pbt

// ---------------------------------------------------------------------------
// pbt_diffraction_noalloc_c: pbt_diffraction_c without any allocation.
//
// Some host programs cannot let a library allocate device memory: programs
// whose device memory is reserved up front by their own pool allocator (a
// cudaMalloc from inside the library would fail, or fragment that pool), and
// programs run under a rule that nothing is allocated after start-up.  This
// variant computes the same FP64 far-field amplitude of one outbeam as
// pbt_diffraction_c, but keeps its device scratch (bin grid, facet record,
// edges, result grid) in one fixed array compiled into the library and its
// host staging in static storage, so it calls no cudaMalloc, cudaFree,
// cudaMallocHost or other allocating routine, and needs no context.
//
// Limits: ntheta * nphi <= PBT_NOALLOC_MAX_BINS (65,536 bins), nphi <=
// PBT_NOALLOC_MAX_PHI (4,096), faces of at most PBT_NOALLOC_MAX_VERTS (64)
// vertices; larger inputs are rejected with PBT_EINVAL.  The array takes
// about 5.6 MB on every GPU that loads the library, until the process exits.
//
// Set-up: every call looks up the array's device address on the current
// device with cudaGetSymbolAddress (cheap once the library's device code is
// loaded, and correct again after a cudaDeviceReset).  The first call on a
// device loads that code and commits the array there, which makes the CUDA
// runtime allocate device memory (and may create the device's primary
// context): make that first call at start-up, before a pool reserves the
// device's memory and outside any stream capture, or run with
// CUDA_MODULE_LOADING=EAGER so that the array is committed when the program
// initialises CUDA.  Each call enqueues its copies and its kernel on the
// calling thread's per-thread default stream (cudaStreamPerThread, not the
// legacy default stream) and waits for them.  Every call on a device shares the
// one array and overwrites what the previous call left there; the result grid
// is written in full, so nothing has to start at zero.  Calls in one process
// are serialised by a host lock and finish before they return; calls that
// overlapped on the GPU would race on the shared array.
namespace pbt {
namespace {

constexpr int64_t kNaMaxBins = 65536;
constexpr int64_t kNaMaxPhi = 4096;
constexpr int kNaMaxVerts = 64;
constexpr size_t kNaOffXyz = 0;
constexpr size_t kNaOffPhi = kNaOffXyz + (size_t)3 * kNaMaxBins * sizeof(double);
constexpr size_t kNaOffFacet = kNaOffPhi + (size_t)2 * kNaMaxPhi * sizeof(double);
constexpr size_t kNaOffEdges = kNaOffFacet + 512;
constexpr size_t kNaOffOut = kNaOffEdges + (((size_t)kNaMaxVerts * sizeof(K1Edge) + 255) & ~(size_t)255);
constexpr size_t kNaBytes = kNaOffOut + (size_t)8 * kNaMaxBins * sizeof(double);
static_assert(sizeof(K1Facet) <= 512, "facet slot");

// the device scratch of pbt_diffraction_noalloc_c
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

static std::mutex g_na_mu;
static double g_na_host[3 * kNaMaxBins + 2 * kNaMaxPhi];  // host staging of the bin grid
// The grid in g_na_host was built from these theta / phi values (g_na_nt < 0: none
// yet); g_na_gen counts the grids built.  A device's scratch holds that grid when
// the 64-bit tag at kNaOffTag (in the facet slot's unused tail) reads
// kNaTagBase ^ g_na_gen, so a call with the same theta and phi as the last one
// builds and uploads nothing; a reset device, or one whose scratch last held
// another grid, gets the grid again.
static double g_na_theta[kNaMaxBins], g_na_phi[kNaMaxPhi];
static int64_t g_na_nt = -1, g_na_np = -1;
static uint64_t g_na_gen = 0;
constexpr uint64_t kNaTagBase = 0x6e61677269645f31ull;
constexpr size_t kNaOffTag = kNaOffFacet + 504;
static_assert(sizeof(K1Facet) <= 504, "the grid tag follows the facet record in its slot");

int na_fail(int status, const char *msg) {
    set_error("%s", msg);
    return status;
}

}  // namespace
}  // namespace pbt

extern "C" int pbt_diffraction_noalloc_c(const pbt_outbeam *outbeam, const double *verts,
                                         int64_t nverts, const int64_t *face_off,
                                         const int64_t *face_vi, int64_t nfaces,
                                         const double *theta, int64_t ntheta, const double *phi,
                                         int64_t nphi, double lambda, int32_t is_fast_diff,
                                         double *amplC) {
    using namespace pbt;
    clear_error();
    if (!outbeam || !amplC) return na_fail(PBT_EINVAL, "outbeam and amplC must not be NULL");
    if (!(lambda > 0) || !isfinite(lambda)) return na_fail(PBT_EINVAL, "lambda must be positive and finite");
    PBT_TRY(validate_angles(theta, ntheta, phi, nphi));
    if (ntheta * nphi > kNaMaxBins || nphi > kNaMaxPhi) {
        set_error("pbt_diffraction_noalloc_c: grid %lld x %lld exceeds its fixed scratch "
                  "(at most %lld bins and %lld phi values); use pbt_diffraction_c",
                  (long long)ntheta, (long long)nphi, (long long)kNaMaxBins, (long long)kNaMaxPhi);
        return PBT_EINVAL;
    }
    PBT_TRY(validate_geometry(verts, nverts, face_off, face_vi, nfaces));
    PBT_TRY(validate_outbeams(outbeam, 1, nfaces, "outbeam"));
    const int64_t fb = face_off[outbeam->fi - 1];
    const int nv = (int)(face_off[outbeam->fi] - fb);
    if (nv > kNaMaxVerts) {
        set_error("pbt_diffraction_noalloc_c: face of %d vertices exceeds its limit of %d", nv,
                  kNaMaxVerts);
        return PBT_EINVAL;
    }
    int64_t theta_i = -1;
    for (int64_t i = 0; i < ntheta; i++)
        if (theta[i] > 1 * kPiRef / 180) {
            theta_i = i;
            break;
        }
    if (theta_i < 0) return na_fail(PBT_EINVAL, "no theta value above 1 degree");

    std::lock_guard<std::mutex> lock(g_na_mu);
    // the array's address on the current device (host code cannot name it directly)
    void *sym = nullptr;
    {
        const cudaError_t e = cudaGetSymbolAddress(&sym, g_noalloc_scratch);
        if (e != cudaSuccess || !sym) {
            (void)cudaGetLastError();
            set_error("cudaGetSymbolAddress(g_noalloc_scratch) failed: %s", cudaGetErrorString(e));
            return PBT_ECUDA;
        }
    }
    unsigned char *base = static_cast<unsigned char *>(sym);

    // bin grid (make_far_field_bins, phi fastest) and cos/sin(phi), libm values;
    // kept from the last call when theta and phi are the same, bit for bit
    const int64_t nb = ntheta * nphi;
    double *hx = g_na_host, *hp = g_na_host + 3 * nb;
    const bool same_grid = ntheta == g_na_nt && nphi == g_na_np &&
                           memcmp(theta, g_na_theta, (size_t)ntheta * sizeof(double)) == 0 &&
                           memcmp(phi, g_na_phi, (size_t)nphi * sizeof(double)) == 0;
    if (!same_grid) {
        for (int64_t j = 0; j < ntheta; j++)
            for (int64_t i = 0; i < nphi; i++) {
                const int64_t o = i + nphi * j;
                hx[o] = kFarR * sin(theta[j]) * cos(phi[i]);
                hx[nb + o] = kFarR * sin(theta[j]) * sin(phi[i]);
                hx[2 * nb + o] = -(kFarR * cos(theta[j]));
            }
        for (int64_t i = 0; i < nphi; i++) {
            hp[i] = cos(phi[i]);
            hp[nphi + i] = sin(phi[i]);
        }
        memcpy(g_na_theta, theta, (size_t)ntheta * sizeof(double));
        memcpy(g_na_phi, phi, (size_t)nphi * sizeof(double));
        g_na_nt = ntheta;
        g_na_np = nphi;
        g_na_gen++;
    }

    // the facet record and its edges (src/diff_mod.f90:515-574, :334-393), on the stack
    const double waveno = 2.0 * kPiRef / lambda;
    double vx[kNaMaxVerts], vy[kNaMaxVerts], vz[kNaMaxVerts];
    double rx[kNaMaxVerts], ry[kNaMaxVerts], rz[kNaMaxVerts];
    double xs[kNaMaxVerts], ys[kNaMaxVerts], ms[kNaMaxVerts];
    for (int i = 0; i < nv; i++) {
        const int64_t vi = face_vi[fb + i] - 1;
        vx[i] = verts[vi];
        vy[i] = verts[vi + nverts];
        vz[i] = verts[vi + 2 * nverts];
    }
    FacetFrame fr;
    fr.sign = 1.0;
    facet_frame(vx, vy, vz, nv, outbeam->prop_out, outbeam->vk7, fr, rx, ry, rz);
    K1Facet F;
    K1Edge E[kNaMaxVerts];
    k1_facet(fr, *outbeam, outbeam->fov, nv, rx, ry, rz, xs, ys, ms, waveno, lambda, 0, F, E);

    // stage into the fixed array, run, copy the grid out (per-thread default stream)
    const cudaStream_t st = cudaStreamPerThread;
    double *d_xyz = reinterpret_cast<double *>(base + kNaOffXyz);
    double *d_phi = reinterpret_cast<double *>(base + kNaOffPhi);
    K1Facet *d_fac = reinterpret_cast<K1Facet *>(base + kNaOffFacet);
    K1Edge *d_edges = reinterpret_cast<K1Edge *>(base + kNaOffEdges);
    double *d_out = reinterpret_cast<double *>(base + kNaOffOut);
    uint64_t *d_tag = reinterpret_cast<uint64_t *>(base + kNaOffTag);
    const uint64_t tag = kNaTagBase ^ g_na_gen;
    uint64_t have = 0;
    PBT_CUDA_TRY(cudaMemcpyAsync(&have, d_tag, sizeof(have), cudaMemcpyDeviceToHost, st));
    PBT_CUDA_TRY(cudaStreamSynchronize(st));
    if (have != tag) {
        // the grid, then its tag (stream order: the tag lands after the grid)
        PBT_CUDA_TRY(cudaMemcpyAsync(d_xyz, hx, 3 * nb * sizeof(double), cudaMemcpyHostToDevice, st));
        PBT_CUDA_TRY(cudaMemcpyAsync(d_phi, hp, 2 * nphi * sizeof(double), cudaMemcpyHostToDevice, st));
        PBT_CUDA_TRY(cudaMemcpyAsync(d_tag, &tag, sizeof(tag), cudaMemcpyHostToDevice, st));
    }
    PBT_CUDA_TRY(cudaMemcpyAsync(d_fac, &F, sizeof(K1Facet), cudaMemcpyHostToDevice, st));
    PBT_CUDA_TRY(cudaMemcpyAsync(d_edges, E, nv * sizeof(K1Edge), cudaMemcpyHostToDevice, st));
    K1Args A{};
    A.fac = d_fac;
    A.edges = d_edges;
    A.xyz = d_xyz;
    A.phitab = d_phi;
    A.nphi = nphi;
    A.nb = nb;
    A.theta_i = theta_i;
    A.waveno = waveno;
    A.lambda = lambda;
    A.n[0] = A.run[0] = 1;
    A.split[0] = 1;
    A.grid[0] = d_out;
    const unsigned blocks = (unsigned)((nb + K1_THREADS - 1) / K1_THREADS);
    if (is_fast_diff)
        k1_kernel<true><<<blocks, K1_THREADS, 0, st>>>(A);
    else
        k1_kernel<false><<<blocks, K1_THREADS, 0, st>>>(A);
    PBT_CUDA_TRY(cudaGetLastError());
    PBT_CUDA_TRY(cudaMemcpyAsync(amplC, d_out, 8 * nb * sizeof(double), cudaMemcpyDeviceToHost, st));
    PBT_CUDA_TRY(cudaStreamSynchronize(st));
    return PBT_OK;
}
