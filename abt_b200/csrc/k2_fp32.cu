// k2_fp32.cu -- batched far-field sum in FP32 with the phase formed in FP64.
//
// Pipeline for a batch of orientations (all on the GPU, no host round trip):
//   1. k2_setup: one thread per outgoing facet forms the facet's aperture frame in
//      FP64 (frame.h, the reference's set-up of src/diff_mod.f90:515-574) and writes
//      nv-2 triangle records, or one polygon record.  Fans of mixed faces count their
//      records first (k2_count, CUB scan); large calls with the field-of-view test
//      take each list in order of direction (k2_order, CUB sort).
//   2. k2_plan: per (orientation, beam|external) segment, the number of
//      work items = facet splits x bin tiles.
//   3. k2_main: a persistent kernel; each CTA claims work items with an
//      atomic counter, streams the item's facet records through shared memory
//      with 1-D bulk copies (cp.async.bulk + mbarrier, bounded waits), and
//      accumulates for each of its bins the 2x2 complex amplitude in FP32
//      (chunk sums carried in FP64), then adds it to the orientation's
//      amplitude workspace.
//   4. k2_epi: FP64 epilogue per bin over the orientations of the batch:
//      T(phi) rotation, Mueller matrix (ampl_to_mueller, src/outputs_mod.f90:
//      473-549), running orientation sum, and per-orientation weighted sums
//      that equal the reference's simpne phi/theta integrals of M11.
//   5. k2_final: per-orientation parameters (finalise,
//      src/outputs_mod.f90:133-245) and the orientation average
//      (summation + divide_by_num_orientations); k2_avg: its Mueller matrix.
//
// Per facet x bin arithmetic.  The reference evaluates, per edge, a contour
// term with a 1/(kxx kyy) coordinate singularity (src/diff_mod.f90:408-420).
// Summed over a triangle's edges it equals (-i/lambda) e^{iK} times the
// aperture integral, which for a triangle is -2A g[d1,d2,d3]: the second
// divided difference of e^{ix} at the three vertex phases.  That form has no
// coordinate singularity; it is evaluated from edge-midpoint phases and
// sinc((d_b - d_a)/2) (stable for every pair gap), with a Taylor series when
// all three phases lie within 0.25 rad.  The far-field phase
// k(|X - c| - |X|) = -k u.c + k(|c|^2 - (u.c)^2)(1 + u.c/R)/(2R) is formed
// with k u.c in FP64 and reduced (as a fixed-point fraction of a turn) before the
// FP32 work; the common
// e^{ik|X|} is applied per bin only when amplitudes are returned.
#include <stdio.h>
#include <stdlib.h>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <algorithm>
#include <type_traits>

#include "frame.h"
#include "k2_common.cuh"
#include "pbt_internal.h"

namespace pbt {

namespace {

constexpr int K2_THREADS = 128;
constexpr int K2_CH = 32;   // records per shared-memory stage
constexpr int K2_NST = 3;   // stages
constexpr double kTwoPi = 6.283185307179586;
constexpr double kInv2Pi = 0.15915494309189535;
constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52, round-to-integer constant
constexpr double kFracMagic = 1572864.0;  // 1.5 * 2^20: an FP64 unit of 2^-32
constexpr double kPi = 3.141592653589793;
constexpr double kInvPi = 0.3183098861837907;
// 1 - c^2 for the reference's clamp c = 0.999999 (a float literal)
constexpr float kOneMinusClampSq = (float)(1.0 - (double)0.999999f * (double)0.999999f);

struct BinDev {
    double ux, uy, uz;  // unit bin direction, FP64
    float fx, fy, fz;   // same, FP32
    float sz, sg;       // s = u + sg z: sz = uz + sg (rounded once from FP64), sg = +-1
    float hx, hy, hsz;  // the (phi_i, theta_i) bin of the forward bodge in the same form
    int64_t bin;        // bin index
};

// The field-of-view test of the FP64 drop-in for bin `bin` (src/diff_mod.f90:593-603):
// x1 = X - com, dot(x1/r1, prop0) >= cos(fov), each operation rounded once.
__device__ __forceinline__ bool fov_exact(const K2FovExact &f, const double *__restrict__ xyz, int64_t nb,
                                       int64_t bin) {
    const double x1 = __dadd_rn(xyz[bin], -f.com[0]);
    const double y1 = __dadd_rn(xyz[nb + bin], -f.com[1]);
    const double z1 = __dadd_rn(xyz[2 * nb + bin], -f.com[2]);
    const double r1 =
        __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(x1, x1), __dmul_rn(y1, y1)), __dmul_rn(z1, z1)));
    const double v0 = __ddiv_rn(x1, r1), v1 = __ddiv_rn(y1, r1), v2 = __ddiv_rn(z1, r1);
    const double d = __dadd_rn(__dadd_rn(__dmul_rn(v0, f.p0[0]), __dmul_rn(v1, f.p0[1])),
                               __dmul_rn(v2, f.p0[2]));
    return !(d < f.cos_fov);
}

// ---------------------------------------------------------------- set-up

struct RefSrc {
    const pbt_outbeam *beam;
    const pbt_outbeam *ext;
    const int64_t *beam_off;  // device copies, norient+1
    const int64_t *ext_off;
    const int64_t *refbase;   // beam_off[o] + ext_off[o]
    int64_t norient;
    // records before outbeam g: start[g] (k2_count and its scan), or g * per where every
    // face has per + 2 vertices (start NULL): nothing to count then
    const int64_t *start;
    int64_t per;
    // outbeam at position g of the call's list, NULL: g itself (k2_order_kernel)
    const int *order;
    __device__ __forceinline__ int64_t first(int64_t g) const { return start ? start[g] : g * per; }
};

__device__ __forceinline__ int64_t find_orient(const int64_t *base, int64_t n, int64_t g) {
    int64_t lo = 0, hi = n;  // largest o in [0, n) with base[o] <= g
    while (hi - lo > 1) {
        int64_t mid = (lo + hi) >> 1;
        if (base[mid] <= g)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

__device__ __forceinline__ const pbt_outbeam *ref_lookup(const RefSrc &S, int64_t g, int64_t &o,
                                                         int &kind) {
    if (S.order) g = S.order[g];
    o = find_orient(S.refbase, S.norient, g);
    const int64_t local = g - S.refbase[o];
    const int64_t nb = S.beam_off[o + 1] - S.beam_off[o];
    if (local < nb) {
        kind = 0;
        return S.beam + S.beam_off[o] + local;
    }
    kind = 1;
    return S.ext + S.ext_off[o] + (local - nb);
}

// Sort keys of the field-of-view sum's order: the list (orientation, kind), then the
// outbeam's direction in the 32 x 32 cells of an octahedral map, in Z order.  A record
// pair is visited where either record's field of view meets a warp's bins, so partners,
// and a stage's records, should look the same way.  `alike` counts the pairs that do.
constexpr int kOrderBits = 5;
__global__ void k2_order_kernel(RefSrc S, int64_t nrefs, unsigned *__restrict__ keys, int *__restrict__ pos,
                                int *__restrict__ alike) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned lanes = __ballot_sync(0xffffffffu, g < nrefs);
    if (g >= nrefs) return;
    int64_t o;
    int kind;
    const pbt_outbeam *ob = ref_lookup(S, g, o, kind);
    const float x = (float)ob->prop_out[0], y = (float)ob->prop_out[1], z = (float)ob->prop_out[2];
    const float s = 1.0f / (fabsf(x) + fabsf(y) + fabsf(z));
    float u = x * s, v = y * s;
    if (z < 0.0f) {
        const float t = (1.0f - fabsf(v)) * (u < 0.0f ? -1.0f : 1.0f);
        v = (1.0f - fabsf(u)) * (v < 0.0f ? -1.0f : 1.0f);
        u = t;
    }
    constexpr int n = 1 << kOrderBits;
    auto cell = [](float w) { return min(max((int)((0.5f * w + 0.5f) * n), 0), n - 1); };
    const int cu = cell(u), cv = cell(v);
    unsigned code = 0;
    for (int b = 0; b < kOrderBits; b++)
        code |= ((unsigned)(cu >> b) & 1u) << (2 * b) | ((unsigned)(cv >> b) & 1u) << (2 * b + 1);
    const unsigned key = (unsigned)(2 * o + kind) << (2 * kOrderBits) | code;
    keys[g] = key;
    pos[g] = (int)g;
    const unsigned next = __shfl_down_sync(lanes, key, 1);
    const unsigned same = __ballot_sync(lanes, !(g & 1) && g + 1 < nrefs && next == key);
    if ((threadIdx.x & 31) == 0 && same) atomicAdd(alike, __popc(same));
}

// Lists in which three of four pairs look the same way already (a beam's outbeams one
// after the other) keep their order: sorting whole beams gains nothing.
__global__ void k2_keep_order_kernel(int64_t nrefs, unsigned *__restrict__ keys, const int *__restrict__ alike) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g < nrefs && 4 * (int64_t)*alike >= 3 * (nrefs / 2)) keys[g] &= ~0u << (2 * kOrderBits);
}

__global__ void k2_count_kernel(RefSrc S, int64_t nrefs, const int64_t *__restrict__ face_off,
                                int64_t nfaces, int64_t *__restrict__ cnt, int *__restrict__ err) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g > nrefs) return;
    if (g == nrefs) {
        cnt[g] = 0;
        return;
    }
    int64_t o;
    int kind;
    const pbt_outbeam *ob = ref_lookup(S, g, o, kind);
    const int64_t fi = ob->fi;
    if (fi < 1 || fi > nfaces) {
        atomicOr(err, 1);
        cnt[g] = 0;
        return;
    }
    cnt[g] = face_off[fi] - face_off[fi - 1] - 2;
}

// Write record r into half r % 2 of pair r / 2 (K2Pair's half-phase and
// scaled forms): kzc = -Kz / (1 - Ky^2), the circular-basis amplitudes uc
// times sqrt(1 - Ky^2) / 4 and the vertices times -k/2, all formed in FP64 by the
// caller.
__device__ __forceinline__ void store_pair_half(K2Pair *pairs, int64_t r, const K2Rec &rec,
                                                double kzc, const double (&uc)[8],
                                                double Kx, const double (&xa)[3],
                                                const double (&ya)[3], double nkh) {
    K2Pair &P = pairs[r >> 1];
    const int h = (int)(r & 1);
    auto put = [h](float2 &dst, float v) {
        if (h)
            dst.y = v;
        else
            dst.x = v;
    };
    for (int c = 0; c < 3; c++) {
        P.kc[c][h] = 0.5 * kInvPi * rec.kc[c];
        put(P.eps[c], rec.eps[c]);
        put(P.vx[c], (float)(nkh * xa[c]));
        put(P.vy[c], (float)(nkh * ya[c]));
    }
    put(P.b, rec.b);
    for (int q = 0; q < 9; q++) put(P.R[q], rec.R[q]);
    put(P.nKx, (float)-Kx);
    put(P.kzc, (float)kzc);
    for (int q = 0; q < 8; q++) put(P.amp[q], (float)uc[q]);
}

// A record's field-of-view data: prop0, fov and the facet centre.
__device__ __forceinline__ void make_fov(const double *prop0, double fov, const double *com, K2Fov &fv,
                                         K2FovExact &fx) {
    fv.p0[0] = (float)prop0[0];
    fv.p0[1] = (float)prop0[1];
    fv.p0[2] = (float)prop0[2];
    fv.cos_fov = (float)cos(fov);
    // the per-bin test uses the direction from the facet centre: it is
    // within |c|/R of the direction from the origin; 2|c|/R + 1e-5 rad
    // also covers the FP32 rounding of both tests
    const double cn = sqrt(com[0] * com[0] + com[1] * com[1] + com[2] * com[2]);
    const double fovm = fov + 2.0 * cn / kFarR + 1e-5;
    fv.fovm = (float)fovm;
    fv.cos_fovm = (float)cos(fovm);
    fv.sin_fovm = (float)sin(fovm);
    // FP32 test error: second-order parallax (< 3 |c/R|^2) and rounding (< 8e-7)
    const double e2 = (cn / kFarR) * (cn / kFarR);
    fv.tol = (float)(3.0 * e2 + 8e-7);
    for (int c = 0; c < 3; c++) {
        fx.com[c] = com[c];
        fx.p0[c] = prop0[c];
    }
    fx.cos_fov = cos(fov);
    fx.pad = 0.0;
}

__global__ void k2_setup_kernel(RefSrc S, int64_t nrefs, const double *__restrict__ verts,
                                int64_t nverts, const int64_t *__restrict__ face_off,
                                int64_t nfaces, const int64_t *__restrict__ face_vi, double waveno, double lambda, int fast_diff,
                                K2Rec *__restrict__ recs, K2Pair *__restrict__ pairs,
                                K2Fov *__restrict__ fovs, K2FovExact *__restrict__ fovx,
                                float2 *__restrict__ rlo, int *__restrict__ err,
                                unsigned *__restrict__ epsmax) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nrefs) return;
    int64_t o;
    int kind;
    const pbt_outbeam *ob = ref_lookup(S, g, o, kind);
    const int64_t fi = ob->fi;
    if (fi < 1 || fi > nfaces) {
        atomicOr(err, 1);
        if (!S.start) {
            // the outbeam's records exist all the same: empty ones
            K2Rec rec{};
            rec.R[0] = rec.R[4] = rec.R[8] = 1.0f;
            const double uc[8] = {}, z[3] = {};
            for (int64_t r = g * S.per; r < (g + 1) * S.per; r++) {
                if (pairs)
                    store_pair_half(pairs, r, rec, 0.0, uc, 0.0, z, z, 0.0);
                else
                    recs[r] = rec;
                for (int i = 0; i < 3; i++) {
                    float2 &l = rlo[(r >> 1) * 3 + i];
                    (r & 1 ? l.y : l.x) = 0.0f;
                }
                if (fast_diff) {
                    fovs[r] = K2Fov{};
                    fovx[r] = K2FovExact{};
                }
            }
        }
        return;
    }
    const int64_t fb = face_off[fi - 1];
    const int nv = (int)(face_off[fi] - fb);
    const double *V = verts + o * 3 * nverts;
    constexpr int NVS = 16;  // vertices held in registers; larger faces re-read
    double vx[NVS], vy[NVS], vz[NVS];
    double prop0[3] = {ob->prop_out[0], ob->prop_out[1], ob->prop_out[2]};
    double perp0[3] = {ob->vk7[0], ob->vk7[1], ob->vk7[2]};
    if (nv > NVS) {
        atomicOr(err, 2);  // faces above 16 vertices are not supported in FP32
        return;
    }
    for (int i = 0; i < nv; i++) {
        const int64_t vi = face_vi[fb + i] - 1;
        vx[i] = V[vi];
        vy[i] = V[vi + nverts];
        vz[i] = V[vi + 2 * nverts];
    }
    FacetFrame fr;
    facet_frame(vx, vy, vz, nv, prop0, perp0, fr, nullptr, nullptr, nullptr);
    const double sign = fr.sign;
    const double *com = fr.com;
    const double R = kFarR;
    if (epsmax) {
        // an upper bound of |com| / R over the records (positive floats order as
        // unsigned integers)
        const double e = sqrt(com[0] * com[0] + com[1] * com[1] + com[2] * com[2]) / R;
        atomicMax(epsmax, __float_as_uint((float)(e * (1.0 + 1e-6)) + 1e-30f));
    }
    const double Ky = fr.prop2[1];
    const double cf = 1.0 / sqrt(1.0 - Ky * Ky);
    double ea[3];
    mv33(fr.R, com, ea);
    const int64_t r0 = S.first(g);
    // an odd record count: the low parts of the last pair's unused half
    if (g == nrefs - 1 && ((r0 + nv - 2) & 1))
        for (int i = 0; i < 3; i++) rlo[((r0 + nv - 2) >> 1) * 3 + i].y = 0.0f;
    for (int t = 0; t < nv - 2; t++) {
        const int iv[3] = {0, t + 1, t + 2};
        double xa[3], ya[3];
        for (int q = 0; q < 3; q++) {
            const double d[3] = {vx[iv[q]] - com[0], vy[iv[q]] - com[1], vz[iv[q]] - com[2]};
            double rr[3];
            mv33(fr.R, d, rr);
            xa[q] = rr[0];
            ya[q] = rr[1];
        }
        const double As = 0.5 * ((xa[1] - xa[0]) * (ya[2] - ya[0]) - (xa[2] - xa[0]) * (ya[1] - ya[0]));
        const double cpre = 2.0 * As / lambda * sign;  // amp' = i * cpre * ampl
        K2Rec rec;
        for (int c = 0; c < 3; c++) {
            rec.kc[c] = waveno * com[c];
            rec.eps[c] = (float)(com[c] / R);
            rec.ea[c] = (float)(ea[c] / R);
            rec.inc[c] = (float)fr.inc2[c];
            rec.vx[c] = (float)xa[c];
            rec.vy[c] = (float)ya[c];
        }
        rec.b = (float)((com[0] * com[0] + com[1] * com[1] + com[2] * com[2]) / (R * R));
        for (int q = 0; q < 9; q++) rec.R[q] = (float)fr.R.m[q / 3][q % 3];
        for (int i = 0; i < 3; i++) {
            // the low part of the y row, read only by lanes on the ky clamp
            float2 &l = rlo[((r0 + t) >> 1) * 3 + i];
            const float lo = (float)(fr.R.m[1][i] - (double)rec.R[3 + i]);
            if ((r0 + t) & 1)
                l.y = lo;
            else
                l.x = lo;
        }
        rec.kp[0] = (float)(waveno * fr.prop2[0]);
        rec.kp[1] = (float)(waveno * fr.prop2[1]);
        rec.hkz_cf = (float)(-0.5 * fr.prop2[2] * cf);
        rec.hicf = (float)(0.5 / cf);
        rec.hkxky_cf = (float)(0.5 * fr.prop2[0] * Ky * cf);
        double am[8];  // (2 i A / lambda) sign ampl: (1,1),(2,1),(1,2),(2,2) re/im
        for (int q = 0; q < 4; q++) {
            am[2 * q] = -cpre * ob->ampl[2 * q + 1];
            am[2 * q + 1] = cpre * ob->ampl[2 * q];
        }
        for (int q = 0; q < 8; q++) rec.amp[q] = (float)am[q];
        if (pairs) {
            // the packed kernel works on the columns in the circular basis
            // u+ = a1c + i a2c, u- = a1c - i a2c (formed in FP64), scaled by the
            // Karczewski-Wolf factor sqrt(1 - Ky^2) / 2 and the 1/2 of the
            // half-phase divided difference
            const double sk = 0.25 / cf;
            const double uc[8] = {sk * (am[0] - am[3]), sk * (am[1] + am[2]), sk * (am[0] + am[3]),
                                  sk * (am[1] - am[2]), sk * (am[4] - am[7]), sk * (am[5] + am[6]),
                                  sk * (am[4] + am[7]), sk * (am[5] - am[6])};
            store_pair_half(pairs, r0 + t, rec, -fr.prop2[2] * cf * cf, uc, fr.prop2[0], xa, ya,
                            -0.5 * waveno);
        } else {
            recs[r0 + t] = rec;
        }
        if (fast_diff) {
            make_fov(prop0, kind ? kPiRef / 2.0 : ob->fov, fr.com, fovs[r0 + t], fovx[r0 + t]);
        }
    }
}

// Thread per outbeam g: its half of facet pair g / 2 (K2Poly and its vertices, `stride`
// bytes a pair).  Both threads of a pair look up both faces for the fans' common length.
__global__ void k2_setup_poly_kernel(RefSrc S, int64_t nrefs, const double *__restrict__ verts,
                                     int64_t nverts, const int64_t *__restrict__ face_off,
                                     int64_t nfaces, const int64_t *__restrict__ face_vi, double waveno,
                                     double lambda, int fast_diff, int nvmax, char *__restrict__ polys,
                                     int64_t stride, K2Fov *__restrict__ fovs,
                                     K2FovExact *__restrict__ fovx, float2 *__restrict__ rlo,
                                     int *__restrict__ err, unsigned *__restrict__ epsmax) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nrefs) return;
    int64_t o, o2;
    int kind, kind2;
    const pbt_outbeam *ob = ref_lookup(S, g, o, kind);
    auto corners = [&](const pbt_outbeam *b) {
        return b->fi < 1 || b->fi > nfaces ? 0 : (int)(face_off[b->fi] - face_off[b->fi - 1]);
    };
    int nv = corners(ob);
    if (nv == 0) atomicOr(err, 1);
    if (nv > kMaxPolyVerts) atomicOr(err, 2);  // larger faces are not supported in FP32
    if (nv > nvmax) nv = 0;
    const int64_t g2 = g ^ 1;
    const int nv2 = g2 < nrefs ? corners(ref_lookup(S, g2, o2, kind2)) : 0;
    const int m = max(max(nv, nv2 > nvmax ? 0 : nv2), 3) - 2;
    K2Poly &P = *reinterpret_cast<K2Poly *>(polys + (g >> 1) * stride);
    K2PolyVertex *pv = reinterpret_cast<K2PolyVertex *>(&P + 1);
    const int h = (int)(g & 1);
    auto put = [h](float2 &dst, double v) {
        if (h)
            dst.y = (float)v;
        else
            dst.x = (float)v;
    };
    P.m = m;  // the same value from both threads
    FacetFrame fr;
    double vx[kMaxPolyVerts], vy[kMaxPolyVerts], vz[kMaxPolyVerts], sign = 1.0;
    if (nv > 0) {
        const int64_t fb = face_off[ob->fi - 1];
        const double *V = verts + o * 3 * nverts;
        for (int i = 0; i < nv; i++) {
            const int64_t vi = face_vi[fb + i] - 1;
            vx[i] = V[vi];
            vy[i] = V[vi + nverts];
            vz[i] = V[vi + 2 * nverts];
        }
        facet_frame(vx, vy, vz, nv, ob->prop_out, ob->vk7, fr, nullptr, nullptr, nullptr);
        sign = fr.sign;
    } else {
        // no face: a record that adds nothing
        fr = FacetFrame{};
        fr.R.m[0][0] = fr.R.m[1][1] = fr.R.m[2][2] = 1.0;
    }
    const double *com = fr.com;
    const double R = kFarR, c2 = com[0] * com[0] + com[1] * com[1] + com[2] * com[2];
    atomicMax(epsmax, __float_as_uint((float)(sqrt(c2) / R * (1.0 + 1e-6)) + 1e-30f));
    const double Ky = fr.prop2[1], cf2 = 1.0 / (1.0 - Ky * Ky);
    for (int c = 0; c < 3; c++) {
        P.kc[c][h] = 0.5 * kInvPi * waveno * com[c];
        put(P.eps[c], com[c] / R);
    }
    put(P.b, c2 / (R * R));
    for (int q = 0; q < 9; q++) put(P.R[q], fr.R.m[q / 3][q % 3]);
    put(P.nKx, -fr.prop2[0]);
    put(P.kzc, -fr.prop2[2] * cf2);
    for (int i = 0; i < 3; i++) {
        put(rlo[(g >> 1) * 3 + i], fr.R.m[1][i] - (double)(float)fr.R.m[1][i]);
        // an odd list: the last pair's unused half
        if (g == nrefs - 1 && !h) rlo[(g >> 1) * 3 + i].y = 0.0f;
    }
    // amplitude (2 i / lambda) sign ampl in the circular basis, times sqrt(1 - Ky^2) / 4
    const double cpre = nv > 0 ? 2.0 / lambda * sign : 0.0, sk = 0.25 / sqrt(cf2);
    for (int b = 0; b < 2; b++) {
        double am[4];  // (1,b), (2,b) re/im
        for (int q = 0; q < 2; q++) {
            am[2 * q] = -cpre * ob->ampl[4 * b + 2 * q + 1];
            am[2 * q + 1] = cpre * ob->ampl[4 * b + 2 * q];
        }
        put(P.amp[4 * b], sk * (am[0] - am[3]));
        put(P.amp[4 * b + 1], sk * (am[1] + am[2]));
        put(P.amp[4 * b + 2], sk * (am[0] + am[3]));
        put(P.amp[4 * b + 3], sk * (am[1] - am[2]));
    }
    double x0 = 0, y0 = 0, xp = 0, yp = 0;
    for (int j = 0; j < m + 2; j++) {
        double x = xp, y = yp, w = 0.0;
        if (j < nv) {
            const double d[3] = {vx[j] - com[0], vy[j] - com[1], vz[j] - com[2]};
            double r[3];
            mv33(fr.R, d, r);
            x = r[0];
            y = r[1];
            if (j == 0) {
                x0 = x;
                y0 = y;
            }
            if (j >= 2) w = 0.5 * ((xp - x0) * (y - y0) - (x - x0) * (yp - y0));
        }
        put(pv[j].vx, -0.5 * waveno * x);
        put(pv[j].vy, -0.5 * waveno * y);
        put(pv[j].w, w);
        xp = x;
        yp = y;
    }
    if (fast_diff) make_fov(ob->prop_out, kind ? kPiRef / 2.0 : ob->fov, com, fovs[g], fovx[g]);
}

// Per orientation chunk [o0, o0+no): segment records and work-item prefix (block 0, a
// scan over the segments), and the split tickets set to zero (the other blocks).
constexpr int K2_PLAN_THREADS = 256;
__global__ void k2_plan_kernel(RefSrc S, int64_t o0, int64_t no, int64_t rpi, int64_t ntiles,
                               int64_t *__restrict__ seg_rec, int64_t *__restrict__ item_pre,
                               unsigned long long *__restrict__ counter, unsigned *__restrict__ tickets) {
    const int t = threadIdx.x;
    if (blockIdx.x > 0) {
        const int64_t n = 2 * no * ntiles, step = (int64_t)(gridDim.x - 1) * K2_PLAN_THREADS;
        for (int64_t i = (int64_t)(blockIdx.x - 1) * K2_PLAN_THREADS + t; i < n; i += step) tickets[i] = 0u;
        return;
    }
    __shared__ int64_t sum[K2_PLAN_THREADS];
    // thread t takes segments [s0, s1)
    const int64_t nseg = 2 * no, each = (nseg + K2_PLAN_THREADS - 1) / K2_PLAN_THREADS;
    const int64_t s0 = min(t * each, nseg), s1 = min(s0 + each, nseg);
    auto rec_of = [&](int64_t s) {
        const int64_t o = o0 + (s >> 1);
        return S.first(S.refbase[o] + (s & 1 ? S.beam_off[o + 1] - S.beam_off[o] : 0));
    };
    int64_t items = 0, r = s0 < s1 ? rec_of(s0) : 0;
    for (int64_t s = s0; s < s1; s++) {
        const int64_t r1 = rec_of(s + 1);
        seg_rec[s] = r;
        if (s + 1 == nseg) seg_rec[nseg] = r1;
        item_pre[s] = items;  // from the thread's first segment; its base is added below
        items += ((r1 - r + rpi - 1) / rpi) * ntiles;
        r = r1;
    }
    sum[t] = items;
    __syncthreads();
    for (int d = 1; d < K2_PLAN_THREADS; d <<= 1) {
        const int64_t v = t >= d ? sum[t - d] : 0;
        __syncthreads();
        sum[t] += v;
        __syncthreads();
    }
    const int64_t base = sum[t] - items;
    for (int64_t s = s0; s < s1; s++) item_pre[s] += base;
    if (t == K2_PLAN_THREADS - 1) {
        item_pre[nseg] = sum[t];
        *counter = 0ull;
    }
}

// ------------------------------------------------------------ main kernel

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// sin(h)/h for h >= 0: Taylor series below 0.5, MUFU sine above
__device__ __forceinline__ float sinc_pos(float h) {
    const float h2 = h * h;
    const float p = fmaf(h2, fmaf(h2, fmaf(h2, fmaf(h2, 2.7557319e-6f, -1.9841270e-4f), 8.3333333e-3f),
                                  -1.6666667e-1f),
                         1.0f);
    const float q = __sinf(h) * rcp_approx(h);
    return h < 0.5f ? p : q;
}

// Second divided difference of e^{ix} at t1, t2, t3 (symmetric in its arguments).
__device__ __forceinline__ float2 tri_dd(float t1, float t2, float t3) {
    float lo = fminf(t1, t2), hi = fmaxf(t1, t2);
    const float mid = fmaxf(lo, fminf(hi, t3));
    lo = fminf(lo, t3);
    hi = fmaxf(hi, t3);
    const float D = hi - lo;
    float2 g;
    if (D >= 0.25f) {
        const float h1 = 0.5f * (mid - lo), h2 = 0.5f * (hi - mid);
        float s1, c1, s2, c2;
        __sincosf(lo + h1, &s1, &c1);
        __sincosf(mid + h2, &s2, &c2);
        const float sc1 = sinc_pos(h1), sc2 = sinc_pos(h2);
        const float iD = rcp_approx(D);
        g.x = (sc1 * s1 - sc2 * s2) * iD;
        g.y = (sc2 * c2 - sc1 * c1) * iD;
    } else {
        // e^{i mid} * sum_n i^(n+2)/(n+2)! h_n(ya, yc), h_n complete homogeneous
        const float ya = lo - mid, yc = hi - mid;
        const float h1 = ya + yc;
        const float ya2 = ya * ya;
        const float h2 = fmaf(yc, h1, ya2);
        const float ya3 = ya2 * ya;
        const float h3 = fmaf(yc, h2, ya3);
        const float ya4 = ya3 * ya;
        const float h4 = fmaf(yc, h3, ya4);
        const float h5 = fmaf(yc, h4, ya4 * ya);
        const float h6 = fmaf(yc, h5, ya4 * ya2);
        const float re = -0.5f + h2 * (1.0f / 24.0f) - h4 * (1.0f / 720.0f) + h6 * (1.0f / 40320.0f);
        const float im = -h1 * (1.0f / 6.0f) + h3 * (1.0f / 120.0f) - h5 * (1.0f / 5040.0f);
        float sm, cm;
        __sincosf(mid, &sm, &cm);
        g.x = cm * re - sm * im;
        g.y = cm * im + sm * re;
    }
    return g;
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint64_t gtimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    mbar_expect(bar, bytes);
    bulk_copy(dst, src, bytes, bar);
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait on an mbarrier phase: false after limit_ns of global time or
// 2^26 polls, whichever comes first.
constexpr uint64_t kWaitLimitNs = 2000000000ull;
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity,
                                          uint64_t limit_ns = kWaitLimitNs) {
    uint64_t t0 = 0;
    for (uint32_t it = 0; it < (1u << 26); ++it) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if (it == 0) t0 = gtimer();
        else if ((it & 255) == 0 && gtimer() - t0 > limit_ns) return false;
    }
    return false;
}

// Work items of one (segment, bin tile) are facet splits.  Each adds its FP64
// sums into the workspace after the previous split of the same tile: ticket
// tk counts the splits added so far (split s waits for tk >= s, adds, and sets
// tk = s + 1), so the sum over splits is in split order and the result is the
// same from run to run.  The item of split s - 1 has the lower item index, so
// it was claimed earlier by a running CTA and never waits on split s.  A wait
// that gives up (2 s of global time or 2^26 polls), or a CTA whose bulk copy
// timed out, sets the ticket to kTicketPoison: later splits of the tile then
// skip their add at once and the call reports PBT_ETIMEOUT.
constexpr unsigned kTicketPoison = 0xffffffffu;
__device__ __forceinline__ bool ticket_wait(const unsigned *tk, unsigned s) {
    uint64_t t0 = 0;
    for (uint32_t it = 0; it < (1u << 26); ++it) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(tk) : "memory");
        if (v >= s) return v != kTicketPoison;
        if (it == 0) t0 = gtimer();
        else if ((it & 255) == 0 && gtimer() - t0 > kWaitLimitNs) return false;
    }
    return false;
}

// The item's sums (lin[bin][8], FP64) into the workspace in split order (see
// ticket_wait); every thread of the CTA calls this.
template <int BPT>
__device__ __forceinline__ void ordered_add(double *__restrict__ out, int64_t nb, unsigned *tk,
                                            unsigned split, const bool (&valid)[BPT],
                                            const int64_t (&bin)[BPT], const double (&lin)[BPT][8],
                                            int *s_ok, int *err) {
    if (threadIdx.x == 0) *s_ok = ticket_wait(tk, split);
    __syncthreads();
    const bool go = *s_ok != 0;
    if (go) {
        __threadfence();
#pragma unroll
        for (int q = 0; q < BPT; q++)
            if (valid[q])
#pragma unroll
                for (int cc = 0; cc < 8; cc++) {
                    // the first split of a tile stores: the workspace needs no clearing
                    double *o = out + cc * nb + bin[q];
                    *o = split ? __ldcg(o) + lin[q][cc] : lin[q][cc];
                }
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (go) {
            atomicMax(tk, split + 1u);
        } else {
            atomicOr(err, 4);
            atomicMax(tk, kTicketPoison);
        }
    }
}

struct K2MainArgs {
    const K2Rec *recs;
    const K2Fov *fovs;
    const K2FovExact *fovx;
    const float2 *rlo;  // R_1 - (float)R_1, pair layout (3 per pair)
    const int64_t *seg_rec;
    const int64_t *item_pre;
    int64_t nseg;
    int64_t rpi;
    int64_t ntiles;
    const double *xyz;
    int64_t nb, nphi;
    int64_t theta_i;
    float k;      // wavenumber
    float hkR;    // k R / 2
    float sgh;    // +1 when the bodge row theta_i lies in the hemisphere of (0,0,-1), else -1
    double *ws;   // [seg][8][nb]
    unsigned *tickets;  // [seg][tile], splits added so far
    unsigned long long *counter;
    int *err;
};

// For a lane on the ky clamp: one component of v = u - sigma R_1, sigma the sign of
// ky and R_1 the aperture frame's y axis (rounded row hi, low part lo), formed from
// the FP64 bin direction.  On the clamp the reference divides kx and kz by
// s = sqrt(1 - 0.999999^2) = 1.4e-3 (m = (-kx ky / s, s, -kz ky / s),
// src/diff_mod.f90:151-158); formed in FP32 from u they are differences of O(1)
// terms with an absolute error near 1e-7, which that division makes 1e-4.  With
// R_0 . R_1 = 0, kx = R_0 . v opa2 + nea_0 opa and kz = R_2 . v opa2 + nea_2 opa,
// where v is small and known to FP32 precision (absolute error near 1e-10).
__device__ __forceinline__ float clamp_v(float hi, float lo, double u, float sigma) {
    return fmaf(-sigma, lo, (float)fma(-(double)sigma, (double)hi, u));
}

template <int BPT, bool FAST>
__device__ __forceinline__ void k2_record(const K2Rec &r, const K2Fov *fv, const K2FovExact *fx,
                                          const BinDev (&bd)[BPT],
                                          const bool (&valid)[BPT], float (&acc)[BPT][8], float k,
                                          float hkR, float sgh, const double *__restrict__ xyz,
                                          int64_t nb, const float2 *__restrict__ rl, int half) {
    const double kc0 = r.kc[0], kc1 = r.kc[1], kc2 = r.kc[2];
#pragma unroll
    for (int q = 0; q < BPT; q++) {
        const BinDev &B = bd[q];
        // far-field phase: FP64 k u.c, reduced mod 2 pi
        const double ka = fma(B.uz, kc2, fma(B.uy, kc1, B.ux * kc0));
        const double nq = fma(ka, kInv2Pi, kMagic) - kMagic;
        const float rf = (float)fma(-nq, kTwoPi, ka);
        const float a = fmaf(B.fz, r.eps[2], fmaf(B.fy, r.eps[1], B.fx * r.eps[0]));
        const float ph = fmaf(hkR * fmaf(-a, a, r.b), 1.0f + a, -rf);
        // bin direction from the facet centre, in the aperture frame:
        // (u - e)/|u - e| = u (1 + a + 3a^2/2 - b/2) - e (1 + a) + O(|e|^3), e = c/R.
        // The second-order terms matter: near k ~ +-y the polarisation matrix
        // depends on 1 - ky^2 and amplifies direction errors by 1/(1 - ky^2).
        // With s = u + sg z and inc = -R z: k = ks + sg opa2 inc, ks = R s opa2 - ea opa,
        // and h = inc x k = inc x ks is formed from small vectors near the poles.
        const float opa = 1.0f + a;
        const float opa2 = fmaf(a, fmaf(1.5f, a, 1.0f), fmaf(-0.5f, r.b, 1.0f));
        const float w0 = fmaf(r.R[2], B.sz, fmaf(r.R[1], B.fy, r.R[0] * B.fx));
        const float w1 = fmaf(r.R[5], B.sz, fmaf(r.R[4], B.fy, r.R[3] * B.fx));
        const float w2 = fmaf(r.R[8], B.sz, fmaf(r.R[7], B.fy, r.R[6] * B.fx));
        const float ks0 = fmaf(w0, opa2, -r.ea[0] * opa);
        const float ks1 = fmaf(w1, opa2, -r.ea[1] * opa);
        const float ks2 = fmaf(w2, opa2, -r.ea[2] * opa);
        const float so = B.sg * opa2;
        const float kx = fmaf(so, r.inc[0], ks0);
        const float ky = fmaf(so, r.inc[1], ks1);
        const float kz = fmaf(so, r.inc[2], ks2);
        bool use = valid[q];
        if (FAST) {
            // lab-frame direction from the centre: u - eps + u a
            const float dx = fmaf(B.fx, opa, -r.eps[0]);
            const float dy = fmaf(B.fy, opa, -r.eps[1]);
            const float dz = fmaf(B.fz, opa, -r.eps[2]);
            const float dp = fmaf(dz, fv->p0[2], fmaf(dy, fv->p0[1], dx * fv->p0[0]));
            bool in = !(dp < fv->cos_fov);
            if (use && fabsf(dp - fv->cos_fov) < fv->tol) in = fov_exact(*fx, xyz, nb, B.bin);
            use = use && in;
        }
        // aperture integral
        const float kxx = fmaf(-k, kx, r.kp[0]);
        const float kyy = fmaf(-k, ky, r.kp[1]);
        const float t1 = fmaf(kyy, r.vy[0], fmaf(kxx, r.vx[0], ph));
        const float t2 = fmaf(kyy, r.vy[1], fmaf(kxx, r.vx[1], ph));
        const float t3 = fmaf(kyy, r.vy[2], fmaf(kxx, r.vx[2], ph));
        const float2 g = tri_dd(t1, t2, t3);
        // Karczewski-Wolf polarisation matrix [[d, e], [-e, d]].  1 - ky^2 is
        // formed as kx^2 + kz^2 (equal for a unit vector, without the
        // cancellation near |ky| = 1); the floor is the reference's clamp
        // |ky| <= 0.999999 (src/diff_mod.f90:151).
        const float kyc = fminf(fmaxf(ky, -0.999999f), 0.999999f);
        const float tr = fmaf(kx, kx, kz * kz);
        float kxv = kx, kzv = kz;  // kx, kz of the polarisation block
        if (tr <= kOneMinusClampSq) {
            auto lo = [&](int i) { return half ? rl[i].y : rl[i].x; };
            const float sig = ky < 0.0f ? -1.0f : 1.0f;
            const float v0 = clamp_v(r.R[3], lo(0), B.ux, sig), v1 = clamp_v(r.R[4], lo(1), B.uy, sig),
                        v2 = clamp_v(r.R[5], lo(2), B.uz, sig);
            kxv = fmaf(fmaf(r.R[2], v2, fmaf(r.R[1], v1, r.R[0] * v0)), opa2, -r.ea[0] * opa);
            kzv = fmaf(fmaf(r.R[8], v2, fmaf(r.R[7], v1, r.R[6] * v0)), opa2, -r.ea[2] * opa);
        }
        const float tt = fmaxf(tr, kOneMinusClampSq);
        const float rs = rsqrtf(tt);
        const float s = tt * rs;
        const float kyrs = kyc * rs;
        const float m0 = -kxv * kyrs, m1 = s, m2 = -kzv * kyrs;
        const float d = fmaf(r.hkz_cf, s, -(kzv * rs) * r.hicf);
        const float e = fmaf(r.hkxky_cf, s, -(kxv * kyrs) * r.hicf);
        // vector perpendicular to the scattering plane (forward bodge near the poles)
        // h = inc x (kx, kyc, kz) = inc x (ks0, ks1 + kyc - ky, ks2)
        float qx = ks0, qy = ks1 + (kyc - ky), qz = ks2;
        const float dinc = fmaf(r.inc[2], kzv, fmaf(r.inc[1], kyc, r.inc[0] * kxv));
        if (!(fabsf(dinc) < 0.999f)) {
            // bodge direction in the s form: uh . eps = hs . eps - sgh eps_z
            const float ah = fmaf(-sgh, r.eps[2],
                                  fmaf(B.hsz, r.eps[2], fmaf(B.hy, r.eps[1], B.hx * r.eps[0])));
            const float oh = 1.0f + ah;
            const float oh2 = fmaf(ah, fmaf(1.5f, ah, 1.0f), fmaf(-0.5f, r.b, 1.0f));
            qx = fmaf(fmaf(r.R[2], B.hsz, fmaf(r.R[1], B.hy, r.R[0] * B.hx)), oh2, -r.ea[0] * oh);
            qy = fmaf(fmaf(r.R[5], B.hsz, fmaf(r.R[4], B.hy, r.R[3] * B.hx)), oh2, -r.ea[1] * oh);
            qz = fmaf(fmaf(r.R[8], B.hsz, fmaf(r.R[7], B.hy, r.R[6] * B.hx)), oh2, -r.ea[2] * oh);
        }
        float hx = fmaf(r.inc[1], qz, -r.inc[2] * qy);
        float hy = fmaf(r.inc[2], qx, -r.inc[0] * qz);
        float hz = fmaf(r.inc[0], qy, -r.inc[1] * qx);
        const float hn = rsqrtf(fmaf(hz, hz, fmaf(hy, hy, hx * hx)));
        hx *= hn;
        hy *= hn;
        hz *= hn;
        float ex = fmaf(kyc, m2, -kzv * m1);
        float ey = fmaf(kzv, m0, -kxv * m2);
        float ez = fmaf(kxv, m1, -kyc * m0);
        if (tt <= kOneMinusClampSq) {
            // inside the clamp cone k and m are not unit vectors and the
            // reference's normalisation of k x m (src/diff_mod.f90:637) matters
            const float ne = rsqrtf(fmaf(ez, ez, fmaf(ey, ey, ex * ex)));
            ex *= ne;
            ey *= ne;
            ez *= ne;
        }
        const float p = fmaf(hz, m2, fmaf(hy, m1, hx * m0));
        const float rr = fmaf(hz, ez, fmaf(hy, ey, hx * ex));
        const float A = fmaf(p, d, rr * e);
        const float Bc = fmaf(p, e, -rr * d);
        // G = [[A, B], [-B, A]] . amp ; acc += g * G
        const float gx = use ? g.x : 0.0f, gy = use ? g.y : 0.0f;
        float G[8];
        G[0] = fmaf(A, r.amp[0], Bc * r.amp[2]);
        G[1] = fmaf(A, r.amp[1], Bc * r.amp[3]);
        G[2] = fmaf(A, r.amp[2], -Bc * r.amp[0]);
        G[3] = fmaf(A, r.amp[3], -Bc * r.amp[1]);
        G[4] = fmaf(A, r.amp[4], Bc * r.amp[6]);
        G[5] = fmaf(A, r.amp[5], Bc * r.amp[7]);
        G[6] = fmaf(A, r.amp[6], -Bc * r.amp[4]);
        G[7] = fmaf(A, r.amp[7], -Bc * r.amp[5]);
#pragma unroll
        for (int c = 0; c < 4; c++) {
            acc[q][2 * c] = fmaf(gx, G[2 * c], fmaf(-gy, G[2 * c + 1], acc[q][2 * c]));
            acc[q][2 * c + 1] = fmaf(gx, G[2 * c + 1], fmaf(gy, G[2 * c], acc[q][2 * c + 1]));
        }
    }
}

template <int BPT, bool FAST>
__global__ void __launch_bounds__(K2_THREADS, 2) k2_main_kernel(K2MainArgs P) {
    __shared__ __align__(128) K2Rec sbuf[K2_NST][K2_CH];
    __shared__ __align__(8) uint64_t bars[K2_NST];
    __shared__ long long s_item;
    __shared__ int s_ok;
    const int tid = threadIdx.x;
    if (tid == 0) {
        for (int s = 0; s < K2_NST; s++) mbar_init(smem_u32(&bars[s]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    uint32_t parity[K2_NST] = {0, 0, 0};
    const int64_t total = P.item_pre[P.nseg];
    constexpr int64_t TILE = (int64_t)K2_THREADS * BPT;
    for (;;) {
        if (tid == 0) s_item = (long long)atomicAdd(P.counter, 1ull);
        __syncthreads();
        const int64_t item = s_item;
        if (item >= total) break;
        // decode item -> (segment, split, tile)
        int64_t lo = 0, hi = P.nseg;
        while (hi - lo > 1) {
            const int64_t m = (lo + hi) >> 1;
            if (P.item_pre[m] <= item)
                lo = m;
            else
                hi = m;
        }
        const int64_t seg = lo;
        const int64_t local = item - P.item_pre[seg];
        const int64_t split = local / P.ntiles, tile = local % P.ntiles;
        const int64_t rbeg = P.seg_rec[seg] + split * P.rpi;
        const int64_t rend = min(rbeg + P.rpi, P.seg_rec[seg + 1]);
        // bins of this thread
        BinDev bd[BPT];
        bool valid[BPT];
        int64_t bin[BPT];
#pragma unroll
        for (int q = 0; q < BPT; q++) {
            bin[q] = tile * TILE + q * K2_THREADS + tid;
            valid[q] = bin[q] < P.nb;
            const int64_t o = valid[q] ? bin[q] : 0;
            const double X = P.xyz[o], Y = P.xyz[P.nb + o], Zc = P.xyz[2 * P.nb + o];
            const double ir = 1.0 / sqrt(X * X + Y * Y + Zc * Zc);
            bd[q].bin = o;
            bd[q].ux = X * ir;
            bd[q].uy = Y * ir;
            bd[q].uz = Zc * ir;
            bd[q].fx = (float)bd[q].ux;
            bd[q].fy = (float)bd[q].uy;
            bd[q].fz = (float)bd[q].uz;
            const double sg = bd[q].uz <= 0.0 ? 1.0 : -1.0;
            bd[q].sz = (float)(bd[q].uz + sg);
            bd[q].sg = (float)sg;
            const int64_t oh = (o % P.nphi) + P.nphi * P.theta_i;
            const double Xh = P.xyz[oh], Yh = P.xyz[P.nb + oh], Zh = P.xyz[2 * P.nb + oh];
            const double irh = 1.0 / sqrt(Xh * Xh + Yh * Yh + Zh * Zh);
            bd[q].hx = (float)(Xh * irh);
            bd[q].hy = (float)(Yh * irh);
            bd[q].hsz = (float)(Zh * irh + (double)P.sgh);
        }
        double acc64[BPT][8];
#pragma unroll
        for (int q = 0; q < BPT; q++)
#pragma unroll
            for (int c = 0; c < 8; c++) acc64[q][c] = 0.0;
        const int64_t nrec = rend - rbeg;
        const int64_t nchunk = (nrec + K2_CH - 1) / K2_CH;
        if (tid == 0) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            for (int64_t c = 0; c < nchunk && c < K2_NST; c++) {
                const int64_t n = min((int64_t)K2_CH, nrec - c * K2_CH);
                bulk_load(smem_u32(&sbuf[c][0]), P.recs + rbeg + c * K2_CH,
                          (uint32_t)(n * sizeof(K2Rec)), smem_u32(&bars[c]));
            }
        }
        bool timed_out = false;
        int64_t c_out = 0;
        for (int64_t c = 0; c < nchunk; c++) {
            const int st = (int)(c % K2_NST);
            const bool ok = mbar_wait(smem_u32(&bars[st]), parity[st]);
            parity[st] ^= 1u;
            if (__syncthreads_or(!ok)) {
                timed_out = true;
                c_out = c;
                break;
            }
            const int n = (int)min((int64_t)K2_CH, nrec - c * K2_CH);
            float acc[BPT][8];
#pragma unroll
            for (int q = 0; q < BPT; q++)
#pragma unroll
                for (int cc = 0; cc < 8; cc++) acc[q][cc] = 0.0f;
            const K2Fov *fv = FAST ? P.fovs + rbeg + c * K2_CH : nullptr;
            for (int j = 0; j < n; j++) {
                const int64_t ri = rbeg + c * K2_CH + j;
                k2_record<BPT, FAST>(sbuf[st][j], FAST ? fv + j : nullptr,
                                     FAST ? P.fovx + ri : nullptr, bd, valid, acc, P.k,
                                     P.hkR, P.sgh, P.xyz, P.nb, P.rlo + (ri >> 1) * 3, (int)(ri & 1));
            }
#pragma unroll
            for (int q = 0; q < BPT; q++)
#pragma unroll
                for (int cc = 0; cc < 8; cc++) acc64[q][cc] += (double)acc[q][cc];
            __syncthreads();  // every thread is done with stage st
            if (tid == 0 && c + K2_NST < nchunk) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                const int64_t c2 = c + K2_NST;
                const int64_t n2 = min((int64_t)K2_CH, nrec - c2 * K2_CH);
                bulk_load(smem_u32(&sbuf[st][0]), P.recs + rbeg + c2 * K2_CH,
                          (uint32_t)(n2 * sizeof(K2Rec)), smem_u32(&bars[st]));
            }
        }
        unsigned *tk = P.tickets + seg * P.ntiles + tile;
        if (timed_out) {
            if (tid == 0) {
                atomicOr(P.err, 4);
                atomicMax(tk, kTicketPoison);
                // bounded wait for this CTA's bulk copies still in flight
                for (int64_t c2 = c_out; c2 < min(nchunk, c_out + K2_NST); c2++) {
                    const int s2 = (int)(c2 % K2_NST);
                    mbar_wait(smem_u32(&bars[s2]), c2 == c_out ? parity[s2] ^ 1u : parity[s2]);
                }
            }
            return;
        }
        ordered_add<BPT>(P.ws + seg * 8 * P.nb, P.nb, tk, (unsigned)split, valid, bin, acc64, &s_ok,
                         P.err);
    }
}

// ---------------------------------------------- packed two-facet main kernel
//
// Same arithmetic as k2_record, evaluated for two facets at once with packed
// FP32x2 instructions (FFMA2/FMUL2/FADD2 of sm_100): the x lane carries the
// even record of a K2Pair, the y lane the odd one.  The bin's data are
// loop-invariant broadcast pairs.  Special-function calls, the sort of the
// three phases and the FP64 phase stay per facet.
//
// Bound: issue.  Over the pair loop the FMA pipe's cycles (an FFMA2 holds it two)
// and the other instructions add up to 88 % of the cycles, at 16 and 20 warps per SM
// alike, so only fewer operations help.  200,000 triangles x 259,560 bins take
// 213.0 ms: 244.8 before the lab-frame normal (no R s + R e, no h in the aperture
// frame; 227.8), the sinc series formed by every lane instead of behind a vote
// (224.1), the fixed-point phase with the item's state and sums in shared memory
// (215.9; with CTA barriers between the stages or the sums in registers 224-226, five
// CTAs per SM with 96 registers 228), and the steps of their own for warps away from
// the incidence axis, at it, and on the clamp of ky (213.0; 24 lists of 3,300 facets
// within 13 um x 64,980 bins 22.0 -> 21.1 ms, 1 % of it by Near, 2 % by the Pole step
// in place of Full).  One operation less in the second-order terms ((u - eps) opa2, no
// 1 + al) came out of the compiler slower, 221.7 ms.

__device__ __forceinline__ float2 bc2(float v) { return make_float2(v, v); }
// the special-function unit's approximations with subnormal inputs flushed
// to zero (the arguments here are phases and squared norms, never subnormal)
__device__ __forceinline__ float sin_fz(float x) {
    float r;
    asm("sin.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float cos_fz(float x) {
    float r;
    asm("cos.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_fz(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 sel2(bool px, bool py, float2 a, float2 b) {
    return make_float2(px ? a.x : b.x, py ? a.y : b.y);
}

// A bin of the packed kernel: the unit direction in FP64 and as FP32 broadcast
// pairs.  The forward-bodge bin direction, used near the poles only, is kept in
// shared memory.
struct BinPk {
    double ux, uy, uz;     // unit bin direction, FP64
    float2 fx, fy, fz;     // broadcast FP32 pairs
    bool pole;             // within reach of the forward bodge (|uz| near 1) for some record
    int bin;               // bin index, -1: none
};

// sin(h)/(2h) below h = 0.5, where the MUFU sine's absolute error would be a large
// relative one: half of 1 + c1 h^2 + c2 h^4 with c1, c2 the minimax fit to the
// relative error on [0, 0.5] (Lawson's iteration: 1.2e-7, 1.6e-7 evaluated in FP32)
__device__ __forceinline__ float2 half_sinc_series(float2 h) {
    const float2 hh = mul2(h, h);
    return fma2(hh, fma2(hh, bc2(0.5f * 8.264339e-3f), bc2(0.5f * -1.6666131e-1f)), bc2(0.5f));
}

// 2 sc g for each lane, g the second divided difference of e^{ix} at the full
// phases 2 t1, 2 t2, 2 t3, from the half phases t, and sc = 1 / (|h| tt) =
// rsqrt(hn2 tt^2) the normalisation of the polarisation block.  With the half
// phases sorted (lo <= mid <= hi) the edge midpoints of the full phases are
// lo + mid and mid + hi and the half gaps mid - lo and hi - mid, each one
// operation.  Formed in two halves: tri_front from the three half phases alone,
// tri_back with the polarisation block's |h|^2 and tt (for the shared reciprocal
// square root below).
struct TriF {
    float2 lo, mid, hi, Dh, s1, k1, s2, k2, p12, S1, S2;
};
__device__ __forceinline__ TriF tri_front(float2 t1, float2 t2, float2 t3) {
    TriF F;
    float2 lo, hi, mid;
    lo.x = fminf(t1.x, t2.x);
    hi.x = fmaxf(t1.x, t2.x);
    mid.x = fmaxf(lo.x, fminf(hi.x, t3.x));
    lo.x = fminf(lo.x, t3.x);
    hi.x = fmaxf(hi.x, t3.x);
    lo.y = fminf(t1.y, t2.y);
    hi.y = fmaxf(t1.y, t2.y);
    mid.y = fmaxf(lo.y, fminf(hi.y, t3.y));
    lo.y = fminf(lo.y, t3.y);
    hi.y = fmaxf(hi.y, t3.y);
    const float2 Dh = add2(hi, neg2(lo));  // half of the largest gap D
    const float2 h1 = add2(mid, neg2(lo));
    const float2 h2 = add2(hi, neg2(mid));
    const float2 c1 = add2(lo, mid), c2 = add2(mid, hi);
    F.s1 = make_float2(sin_fz(c1.x), sin_fz(c1.y));
    F.k1 = make_float2(cos_fz(c1.x), cos_fz(c1.y));
    F.s2 = make_float2(sin_fz(c2.x), sin_fz(c2.y));
    F.k2 = make_float2(cos_fz(c2.x), cos_fz(c2.y));
    // With a1 = max(h1, .5) and a2 = max(h2, .5), 2 sc g = scr (S1 e^{i c1} -
    // S2 e^{i c2}) (imaginary unit and sign aside), S1 = sinc(h1) a1 a2,
    // S2 = sinc(h2) a1 a2 and scr = sc / (a1 a2 Dh): one reciprocal square root,
    // rsqrt(hn2 (tt a1 a2 Dh)^2), gives the polarisation block's normalisation,
    // 1/a1, 1/a2 and 2/D.  sinc(h1) a1 is sin(h1) where h1 >= 0.5 and half of the
    // sinc series below.  Some lane of a warp nearly always needs the series (two of
    // a triangle's phases within 1 rad), so every lane forms it, without a vote.
    const float2 a1 = make_float2(fmaxf(h1.x, 0.5f), fmaxf(h1.y, 0.5f));
    const float2 a2 = make_float2(fmaxf(h2.x, 0.5f), fmaxf(h2.y, 0.5f));
    F.lo = lo; F.mid = mid; F.hi = hi; F.Dh = Dh;
    F.p12 = mul2(a1, a2);
    F.S1 = mul2(sel2(h1.x < 0.5f, h1.y < 0.5f, half_sinc_series(h1),
                     make_float2(sin_fz(h1.x), sin_fz(h1.y))), a2);
    F.S2 = mul2(sel2(h2.x < 0.5f, h2.y < 0.5f, half_sinc_series(h2),
                     make_float2(sin_fz(h2.x), sin_fz(h2.y))), a1);
    return F;
}

// scr = sc / (p12 Dh); twice_sc() is formed only where the Taylor series needs it.
template <class Sc>
__device__ __forceinline__ void tri_back(const TriF &F, float2 scr, Sc twice_sc, float2 &gx, float2 &gy) {
    const float2 Dh = F.Dh;
    gx = mul2(fma2(F.S1, F.s1, neg2(mul2(F.S2, F.s2))), scr);
    gy = mul2(fma2(F.S2, F.k2, neg2(mul2(F.S1, F.k1))), scr);
    // (uniform over the warp: the lanes that need it select)
    if (__any_sync(0xffffffffu, Dh.x < 0.125f || Dh.y < 0.125f)) {
        // all three full phases within 0.25 rad: Taylor series about the middle
        // phase, g = e^{2i mid} sum_n i^(n+2)/(n+2)! q_n(ya, yc) with the complete
        // homogeneous q_n of the full-phase offsets 2 ya, 2 yc (2^n folded into
        // the coefficients)
        const float2 ya = add2(F.lo, neg2(F.mid)), yc = add2(F.hi, neg2(F.mid));
        const float2 q1 = add2(ya, yc);
        const float2 ya2 = mul2(ya, ya);
        const float2 q2 = fma2(yc, q1, ya2);
        const float2 ya3 = mul2(ya2, ya);
        const float2 q3 = fma2(yc, q2, ya3);
        const float2 ya4 = mul2(ya3, ya);
        const float2 q4 = fma2(yc, q3, ya4);
        const float2 q5 = fma2(yc, q4, mul2(ya4, ya));
        const float2 q6 = fma2(yc, q5, mul2(ya4, ya2));
        const float2 tsc = twice_sc();
        const float2 re = mul2(tsc, fma2(q6, bc2(1.0f / 630.0f),
                                         fma2(q4, bc2(-1.0f / 45.0f), fma2(q2, bc2(1.0f / 6.0f), bc2(-0.5f)))));
        const float2 im = mul2(tsc, fma2(q5, bc2(-2.0f / 315.0f),
                                         fma2(q3, bc2(1.0f / 15.0f), mul2(q1, bc2(-1.0f / 3.0f)))));
        const float2 m2 = add2(F.mid, F.mid);
        const float2 sm = make_float2(sin_fz(m2.x), sin_fz(m2.y));
        const float2 cm = make_float2(cos_fz(m2.x), cos_fz(m2.y));
        const float2 sx = fma2(cm, re, neg2(mul2(sm, im)));
        const float2 sy = fma2(cm, im, mul2(sm, re));
        gx = sel2(Dh.x < 0.125f, Dh.y < 0.125f, sx, gx);
        gy = sel2(Dh.x < 0.125f, Dh.y < 0.125f, sy, gy);
    }
}

// 2 g for each lane, g the second divided difference alone
__device__ __forceinline__ void tri_poly(float2 t1, float2 t2, float2 t3, float2 &gx, float2 &gy) {
    const TriF F = tri_front(t1, t2, t3);
    const float2 q = mul2(F.p12, F.Dh);
    tri_back(F, make_float2(rcp_approx(q.x), rcp_approx(q.y)), [] { return make_float2(2.0f, 2.0f); }, gx, gy);
}

// Two adjacent float2 fields of a record pair from one 16-byte shared-memory load
// (every such field pair of K2Pair starts on a 16-byte boundary).
__device__ __forceinline__ void ld22(const float2 *p, float2 &a, float2 &b) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    a = make_float2(v.x, v.y);
    b = make_float2(v.z, v.w);
}

// How far a launch's facet centres lie from the origin.  Near: |com| / R up to 2^-14
// (61 um); the second order of the direction from a facet centre, below 1.5 |com|^2 / R^2
// = 5.6e-9, is then under a tenth of FP32's half ulp and left out.  Wide: half phases
// k |com| / 2 from 2^18 pi on, beyond the fixed-point form of the far-field phase.
enum class Reach { Near, Mid, Wide };
__device__ __forceinline__ Reach k2_reach(float epsmax, float turns) {
    if (!(turns * epsmax < 262144.0f)) return Reach::Wide;
    return epsmax <= 6.1035156e-5f ? Reach::Near : Reach::Mid;
}

// Main: the step without the forward bodge and the clamp of ky; Pole: with the bodge, for
// warps with a bin near the incidence axis; both lower tmin to the smallest kx^2 + kz^2:
// at or below the clamp's the caller takes the Full step, with a branch for either.
enum class Step { Main, Pole, Full };
template <bool FAST, Step STEP, Reach REACH, class PairT>
__device__ __forceinline__ void k2_pair(const PairT &P, const K2Fov *fv, const K2FovExact *fx, const BinPk &B,
                                        float2 (&acc)[8], float2 hkRh, float &tmin,
                                        const float4 &hb, bool lo_ok, bool hi_ok,
                                        const double *__restrict__ xyz, int64_t nb,
                                        const float2 *__restrict__ rl) {
    // far-field half phase per facet, k u.c / 2 modulo pi, as a fixed-point fraction of
    // pi (2^-32 units): added to 1.5 * 2^20 the FP64 sum's low word is that fraction, so
    // the reduction costs no operation of its own (each of the three steps rounds to
    // 2^-32 pi = 7e-10 rad).  The fraction is then rounded to FP32 and multiplied by a
    // rounded constant: 4.0e-8 rad rms and 1.5e-7 at most over a half phase, where one
    // rounding of an FP64 remainder makes 2.3e-8 and 6.0e-8.  The sum's error against 64
    // bits is set by the vertex phases and did not grow: over 48 sets of 150 facets (0.1 to
    // 10 um, up to 200 um from the origin) 0.85 to 1.01 of that with the FP64 remainder.
    // The fixed point holds up to 2^19 half turns; records beyond (Wide) subtract the
    // nearest integer.
    float2 fr;
    {
        const double2 k0 = *reinterpret_cast<const double2 *>(&P.kc[0][0]);
        const double2 k1 = *reinterpret_cast<const double2 *>(&P.kc[1][0]);
        const double2 k2 = *reinterpret_cast<const double2 *>(&P.kc[2][0]);
        if (REACH != Reach::Wide) {
            fr.x = (float)__double2loint(fma(B.uz, k2.x, fma(B.uy, k1.x, fma(B.ux, k0.x, kFracMagic))));
            fr.y = (float)__double2loint(fma(B.uz, k2.y, fma(B.uy, k1.y, fma(B.ux, k0.y, kFracMagic))));
        } else {
            const double ka = fma(B.uz, k2.x, fma(B.uy, k1.x, B.ux * k0.x));
            const double kb = fma(B.uz, k2.y, fma(B.uy, k1.y, B.ux * k0.y));
            fr.x = (float)((ka - ((ka + kMagic) - kMagic)) * 4294967296.0);
            fr.y = (float)((kb - ((kb + kMagic) - kMagic)) * 4294967296.0);
        }
    }
    const float2 one = bc2(1.0f);
    float2 eps0, eps1, eps2, pb;
    ld22(&P.eps[0], eps0, eps1);
    ld22(&P.eps[2], eps2, pb);
    const float2 al = fma2(B.fz, eps2, fma2(B.fy, eps1, mul2(B.fx, eps0)));  // u . eps
    // with y = b - al^2: half phase hkRh y (1 + al) - pi 2^-32 fr
    const float2 opa = add2(one, al);
    const float2 y = fma2(neg2(al), al, pb);
    const float2 ph = fma2(fr, bc2((float)(-kPi / 4294967296.0)), mul2(mul2(hkRh, y), opa));
    const float2 opa2 = fma2(al, al, fma2(bc2(-0.5f), y, opa));
    // The unit direction from the facet centre in the lab frame, (a, b, c) = u opa2 -
    // eps opa with opa2 = 1 + al + 1.5 al^2 - 0.5 b = (1 + al) - 0.5 y + al^2, or u opa -
    // eps for Near, and k = R (a, b, c) in the aperture frame.  The normal of the
    // scattering plane, h = inc x k with inc = (0, 0, -1), is (b, -a, 0): formed from
    // the lab components it has no cancellation of nearly parallel unit vectors near
    // the forward and backward directions, where a and b are small and known to full
    // FP32 precision.
    float2 a, b, c;
    if (REACH == Reach::Near) {
        a = fma2(B.fx, opa, neg2(eps0));
        b = fma2(B.fy, opa, neg2(eps1));
        c = fma2(B.fz, opa, neg2(eps2));
    } else {
        a = fma2(B.fx, opa2, neg2(mul2(eps0, opa)));
        b = fma2(B.fy, opa2, neg2(mul2(eps1, opa)));
        c = fma2(B.fz, opa2, neg2(mul2(eps2, opa)));
    }
    float2 r3, r4, r5, nKx, kx, ky, kz, u;
    {
        float2 r0, r1, r2, r6, r7, r8;
        ld22(&P.R[0], r0, r1);
        ld22(&P.R[2], r2, r3);
        ld22(&P.R[4], r4, r5);
        ld22(&P.R[6], r6, r7);
        ld22(&P.R[8], r8, nKx);
        kx = fma2(r2, c, fma2(r1, b, mul2(r0, a)));
        u = fma2(r4, b, mul2(r3, a));
        ky = fma2(r5, c, u);
        kz = fma2(r8, c, fma2(r7, b, mul2(r6, a)));
    }
    // the divided difference's phases, sort, sines and cosines: independent of
    // the polarisation block and its rare branch, so formed ahead of the branch
    // (one basic block with the direction arithmetic for the scheduler)
    constexpr bool POLY = std::is_same<PairT, K2Poly>::value;
    const float2 dx = add2(kx, nKx);
    [[maybe_unused]] TriF tf;
    if constexpr (!POLY) {
        float2 vx0, vx1, vx2, vy0, vy1, vy2;
        ld22(&P.vx[0], vx0, vx1);
        ld22(&P.vx[2], vx2, vy0);
        ld22(&P.vy[1], vy1, vy2);
        const float2 t1 = fma2(ky, vy0, fma2(dx, vx0, ph));
        const float2 t2 = fma2(ky, vy1, fma2(dx, vx1, ph));
        const float2 t3 = fma2(ky, vy2, fma2(dx, vx2, ph));
        tf = tri_front(t1, t2, t3);
    }
    // Polarisation matrix [[d, e], [-e, d]] (see k2_record for the forms) and
    // the rotation into the scattering plane, with their normalisations folded
    // into one factor: with s = sqrt(tt) and hc = h / |h|,
    //   d = d1 / s, e = e1 / s, p = P1 / (|h| s), rr = R1 / (|h| s),
    // so A = p d + rr e = sc (P1 d1 + R1 e1) and B = sc (P1 e1 - R1 d1) with
    // sc = 1 / (|h| tt) = rsqrt(|h|^2 tt^2).  The in-plane rotation of the set-up
    // puts prop2 in the x-z plane (src/diff_mod.f90:540-559), so Ky = 0 up to
    // rounding and d1 = (sqrt(1 - Ky^2)/2) (kzc tt - kz), e1 = (sqrt(1 - Ky^2)/2)(-kx kyc)
    // (the Kx Ky term is below 1e-16 and left out); the common factor is in the
    // record's amplitudes and sc in the divided difference.
    // Main path: |ky| < 0.999999 (no clamp) and no forward bodge, so kyc = ky,
    // tt = kx^2 + kz^2 and h is normal to k.  Then P1 = p |h| s = hy tt - kyc (hx kx +
    // hz kz) is hy |k|^2 = hy (|k| = 1 up to rounding) and R1 = rr |h| s =
    // hz kx - hx kz = -y . (k x h), with k x h = (c a, c b, -|h|^2) in the lab frame
    // and y = (r3, r4, r5) the frame's second axis: neither needs h in the aperture
    // frame.
    const float2 tr = fma2(kx, kx, mul2(kz, kz));
    float2 tt = tr;
    float2 d1, e1;
    float2 hn2 = fma2(a, a, mul2(b, b));
    float2 P1 = fma2(r3, b, neg2(mul2(r4, a)));
    float2 R1 = fma2(r5, hn2, neg2(mul2(c, u)));
    float2 kzc = P.kzc;
    constexpr bool FULL = STEP == Step::Full;
    const bool cx = FULL && tr.x <= kOneMinusClampSq, cy = FULL && tr.y <= kOneMinusClampSq;
    if (!FULL) tmin = fminf(tmin, fminf(tr.x, tr.y));
    if (STEP == Step::Pole) {
        // the forward bodge (src/diff_mod.f90:630-633): h = (bb, -ba, 0) from the direction
        // (ba, bb, .) to the bodge's bin, no longer normal to k: P1 = y . h - ky (h . k),
        // R1 = -y . (k x h)
        const bool bx = !(fabsf(c.x) < 0.999f), by = !(fabsf(c.y) < 0.999f);
        const float2 ux = bc2(hb.x), uy = bc2(hb.y), uz = bc2(hb.z);
        const float2 ah = fma2(uz, eps2, fma2(uy, eps1, mul2(ux, eps0)));
        const float2 oh = add2(one, ah);
        const float2 oh2 = fma2(ah, fma2(bc2(1.5f), ah, one), fma2(bc2(-0.5f), pb, one));
        const float2 ba = fma2(ux, oh2, neg2(mul2(eps0, oh)));
        const float2 bb = fma2(uy, oh2, neg2(mul2(eps1, oh)));
        const float2 hk = fma2(bb, a, neg2(mul2(ba, b)));
        P1 = sel2(bx, by, fma2(r3, bb, neg2(fma2(r4, ba, mul2(ky, hk)))), P1);
        R1 = sel2(bx, by, fma2(r5, fma2(a, ba, mul2(b, bb)), neg2(mul2(c, fma2(r4, bb, mul2(r3, ba))))), R1);
        hn2 = sel2(bx, by, fma2(ba, ba, mul2(bb, bb)), hn2);
    }
    if (FULL && (B.pole || cx || cy)) {
        float2 r0, r1, r2, r6, r7, r8, q3, q4, q5, q9;
        ld22(&P.R[0], r0, r1);
        ld22(&P.R[2], r2, q3);
        ld22(&P.R[4], q4, q5);
        ld22(&P.R[6], r6, r7);
        ld22(&P.R[8], r8, q9);
        // h in the aperture frame, R (b, -a, 0)
        float2 hx = fma2(r0, b, neg2(mul2(r1, a)));
        float2 hz = fma2(r6, b, neg2(mul2(r7, a)));
        float2 hy = P1;
        if (cx || cy) {
            // on the clamp: kx and kz from v = u - sigma R_1 (see clamp_v)
            const float2 l0 = rl[0], l1 = rl[1], l2 = rl[2];
            const float sx = ky.x < 0.0f ? -1.0f : 1.0f, sy = ky.y < 0.0f ? -1.0f : 1.0f;
            const float2 v0 = make_float2(clamp_v(r3.x, l0.x, B.ux, sx), clamp_v(r3.y, l0.y, B.ux, sy));
            const float2 v1 = make_float2(clamp_v(r4.x, l1.x, B.uy, sx), clamp_v(r4.y, l1.y, B.uy, sy));
            const float2 v2 = make_float2(clamp_v(r5.x, l2.x, B.uz, sx), clamp_v(r5.y, l2.y, B.uz, sy));
            const float2 e0 = fma2(r2, eps2, fma2(r1, eps1, mul2(r0, eps0)));
            const float2 e2 = fma2(r8, eps2, fma2(r7, eps1, mul2(r6, eps0)));
            const float2 kxa = fma2(fma2(r2, v2, fma2(r1, v1, mul2(r0, v0))), opa2, neg2(mul2(e0, opa)));
            const float2 kza = fma2(fma2(r8, v2, fma2(r7, v1, mul2(r6, v0))), opa2, neg2(mul2(e2, opa)));
            kx = sel2(cx, cy, kxa, kx);
            kz = sel2(cx, cy, kza, kz);
        }
        // near the poles (the forward bodge) or on the clamp: ky clamped to
        // +-0.999999 and tt to 1 - 0.999999^2 as in src/diff_mod.f90
        const float2 kyc = make_float2(fminf(fmaxf(ky.x, -0.999999f), 0.999999f),
                                       fminf(fmaxf(ky.y, -0.999999f), 0.999999f));
        tt = make_float2(fmaxf(tr.x, kOneMinusClampSq), fmaxf(tr.y, kOneMinusClampSq));
        d1 = fma2(kzc, tt, neg2(kz));
        e1 = mul2(neg2(kx), kyc);
        bool bx = false, by = false;
        if (B.pole) {
            // the forward bodge (src/diff_mod.f90:630-633) can apply only in bins near
            // the poles; dinc = z . (kx, kyc, kz) = -inc . (kx, kyc, kz)
            const float2 dinc = fma2(r8, kz, fma2(r5, kyc, mul2(r2, kx)));
            bx = !(fabsf(dinc.x) < 0.999f);
            by = !(fabsf(dinc.y) < 0.999f);
            if (bx || by) {
                // h from the direction (ba, bb, .) from the facet to the bodge's bin
                const float2 ux = bc2(hb.x), uy = bc2(hb.y), uz = bc2(hb.z);
                const float2 ah = fma2(uz, eps2, fma2(uy, eps1, mul2(ux, eps0)));
                const float2 oh = add2(one, ah);
                const float2 oh2 = fma2(ah, fma2(bc2(1.5f), ah, one), fma2(bc2(-0.5f), pb, one));
                const float2 ba = fma2(ux, oh2, neg2(mul2(eps0, oh)));
                const float2 bb = fma2(uy, oh2, neg2(mul2(eps1, oh)));
                const float2 gx = fma2(r0, bb, neg2(mul2(r1, ba)));
                const float2 gy = fma2(r3, bb, neg2(mul2(r4, ba)));
                const float2 gz = fma2(r6, bb, neg2(mul2(r7, ba)));
                const float2 gP = fma2(gy, tt, neg2(mul2(kyc, fma2(gx, kx, mul2(gz, kz)))));
                hx = sel2(bx, by, gx, hx);
                hy = sel2(bx, by, gy, hy);
                hz = sel2(bx, by, gz, hz);
                P1 = sel2(bx, by, gP, P1);
            }
        }
        float2 Rq = fma2(hz, kx, neg2(mul2(hx, kz)));
        if (cx || cy) {
            // a lane on the clamp: outside the bodge, h = inc x (kx, kyc, kz) takes the
            // clamped ky; evo2 = normalise(k x m) with the clamped ky, R1 = s (h . evo2)
            const float2 dk = add2(kyc, neg2(ky));
            const bool ux = cx && !bx, uy = cy && !by;
            hx = sel2(ux, uy, fma2(r8, dk, hx), hx);
            hz = sel2(ux, uy, fma2(neg2(r2), dk, hz), hz);
            const float2 rs = make_float2(rsqrtf(tt.x), rsqrtf(tt.y));
            const float2 s = mul2(tt, rs), kyrs = mul2(kyc, rs);
            const float2 m0 = neg2(mul2(kx, kyrs)), m1 = s, m2 = neg2(mul2(kz, kyrs));
            float2 ex = fma2(kyc, m2, neg2(mul2(kz, m1)));
            float2 ey = fma2(kz, m0, neg2(mul2(kx, m2)));
            float2 ez = fma2(kx, m1, neg2(mul2(kyc, m0)));
            const float2 en2 = fma2(ez, ez, fma2(ey, ey, mul2(ex, ex)));
            const float2 ne = make_float2(cx ? rsqrtf(en2.x) : 1.0f, cy ? rsqrtf(en2.y) : 1.0f);
            const float2 rc = mul2(mul2(s, ne), fma2(hz, ez, fma2(hy, ey, mul2(hx, ex))));
            Rq = sel2(cx, cy, rc, fma2(hz, kx, neg2(mul2(hx, kz))));
        }
        // lanes of the main form (an ordinary bin beside a clamped one) keep it
        const bool gx_ = bx || cx, gy_ = by || cy;
        R1 = sel2(gx_, gy_, Rq, R1);
        hn2 = sel2(gx_, gy_, fma2(hz, hz, fma2(hy, hy, mul2(hx, hx))), hn2);
    } else {
        d1 = fma2(kzc, tr, neg2(kz));
        e1 = mul2(neg2(kx), ky);
    }
    const float2 A = fma2(P1, d1, mul2(R1, e1));
    const float2 Bc = fma2(P1, e1, neg2(mul2(R1, d1)));
    // aperture integral on the half phases, its second half (the normalisation
    // sc needs the polarisation block's |h| and tt): 2 sc g
    float2 gx, gy;
    if constexpr (!POLY) {
        const float2 q = mul2(mul2(tf.p12, tf.Dh), tt);
        const float2 hq = mul2(hn2, mul2(q, q));
        tri_back(tf, make_float2(rsqrt_fz(hq.x), rsqrt_fz(hq.y)), [&] {
            const float2 ht = mul2(mul2(hn2, tt), tt);
            return make_float2(2.0f * rsqrt_fz(ht.x), 2.0f * rsqrt_fz(ht.y));
        }, gx, gy);
    } else {
        // the fan's triangles share all of the above; their areas weight them
        const float4 *v = reinterpret_cast<const float4 *>(&P + 1);  // vx, vy | w, pad
        auto phase = [&](int j) {
            const float4 q = v[2 * j];
            return fma2(ky, make_float2(q.z, q.w), fma2(dx, make_float2(q.x, q.y), ph));
        };
        const float2 t0 = phase(0);
        float2 tp = phase(1);
        gx = gy = bc2(0.0f);
        const int m = P.m;
#pragma unroll 1
        for (int j = 2; j < m + 2; j++) {
            const float2 tn = phase(j), w = *reinterpret_cast<const float2 *>(&v[2 * j + 1]);
            float2 ax, ay;
            tri_poly(t0, tp, tn, ax, ay);
            gx = fma2(w, ax, gx);
            gy = fma2(w, ay, gy);
            tp = tn;
        }
        const float2 ht = mul2(mul2(hn2, tt), tt);
        const float2 sc = make_float2(rsqrt_fz(ht.x), rsqrt_fz(ht.y));
        gx = mul2(gx, sc);
        gy = mul2(gy, sc);
    }
    // [[A, B], [-B, A]] is diagonal in the circular basis: with z = A - iB the
    // columns' u+ take z, their u- take conj(z).  q+ = g z, q- = g conj(z).
    const float2 gyB = mul2(gy, Bc), gxB = mul2(gx, Bc);
    float2 qpr = fma2(gx, A, gyB), qmr = fma2(gx, A, neg2(gyB));
    float2 qpi = fma2(gy, A, neg2(gxB)), qmi = fma2(gy, A, gxB);
    bool ok_x = lo_ok, ok_y = hi_ok;
    if (FAST) {
        // the field-of-view test (direction from the facet centre, lab frame)
        const K2Fov &fa = fv[0], &fb = fv[1];
        const float dpx = fmaf(c.x, fa.p0[2], fmaf(b.x, fa.p0[1], a.x * fa.p0[0]));
        const float dpy = fmaf(c.y, fb.p0[2], fmaf(b.y, fb.p0[1], a.y * fb.p0[0]));
        bool in_x = !(dpx < fa.cos_fov), in_y = !(dpy < fb.cos_fov);
        if (ok_x && fabsf(dpx - fa.cos_fov) < fa.tol) in_x = fov_exact(fx[0], xyz, nb, B.bin);
        if (ok_y && fabsf(dpy - fb.cos_fov) < fb.tol) in_y = fov_exact(fx[1], xyz, nb, B.bin);
        ok_x = ok_x && in_x;
        ok_y = ok_y && in_y;
    }
    if (FAST || !lo_ok || !hi_ok) {
        // a lane outside the item or outside the field of view adds nothing
        qpr = sel2(ok_x, ok_y, qpr, bc2(0.0f));
        qmr = sel2(ok_x, ok_y, qmr, bc2(0.0f));
        qpi = sel2(ok_x, ok_y, qpi, bc2(0.0f));
        qmi = sel2(ok_x, ok_y, qmi, bc2(0.0f));
    }
    // acc: (U+ col 1, U- col 1, U+ col 2, U- col 2), re/im
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const float2 qr = (q & 1) ? qmr : qpr, qi = (q & 1) ? qmi : qpi;
        float2 ur, ui;
        ld22(&P.amp[2 * q], ur, ui);
        acc[2 * q] = fma2(qr, ur, fma2(neg2(qi), ui, acc[2 * q]));
        acc[2 * q + 1] = fma2(qr, ui, fma2(qi, ur, acc[2 * q + 1]));
    }
}

using MainC = std::integral_constant<Step, Step::Main>;
using PoleC = std::integral_constant<Step, Step::Pole>;
using FullC = std::integral_constant<Step, Step::Full>;
using NearC = std::integral_constant<Reach, Reach::Near>;
using MidC = std::integral_constant<Reach, Reach::Mid>;
using WideC = std::integral_constant<Reach, Reach::Wide>;

// Record pairs per shared-memory stage: 44 for the full sum (three stages, 44 KB,
// four CTAs per SM); 32 with the field-of-view cull, whose per-stage keep masks are
// two 32-bit ballot words of the stage's 64 records.
constexpr int K2P_CH_FULL = 44, K2P_CH_FOV = 32;
// bytes a stage of polygons: 29 pairs of up to 6 vertices, 24 beside the field-of-view data
constexpr int poly_stage(bool fast) { return (fast ? 37 : 44) * 288; }

// The record's per-bin test passes no bin of the tile when the angle between
// prop0 and the tile centre exceeds fovm + psi (fovm includes the parallax
// and rounding margin); compared through cosines with a further 1e-6 margin.
__device__ __forceinline__ bool cone_culled(const K2Fov &f, const K2Cone &t) {
    if (!(f.fovm + t.psi < 3.14159f)) return false;
    const float d = fmaf(f.p0[2], t.c[2], fmaf(f.p0[1], t.c[1], f.p0[0] * t.c[0]));
    return d < fmaf(f.cos_fovm, t.cos_psi, -f.sin_fovm * t.sin_psi) - 1e-6f;
}

struct K2PkArgs {
    const float2 *rlo;  // R_1 - (float)R_1, pair layout (3 per pair)
    const K2Pair *pairs;
    const char *polys;  // polygons: K2Poly and vertices, stride bytes a pair
    int stride, chunk;  // and pairs per shared-memory stage
    const K2Fov *fovs;
    const K2FovExact *fovx;
    const int *perm;        // is_fast_diff: tile-major bin order (-1: padding)
    const K2Cone *cones;    // is_fast_diff: cone of each warp's 32 bins
    const int64_t *seg_rec;
    const int64_t *item_pre;
    int64_t nseg;
    int64_t rpi;
    int64_t ntiles;
    const double *xyz;
    int64_t nb, nphi;
    int64_t theta_i;
    float hkR;
    float turns;  // k R / (2 pi): half turns of the far-field phase per unit of |com| / R
    const unsigned *epsmax;  // float bits of a bound of |com| / R over the records
    double *ws;         // [seg][8][nb]
    unsigned *tickets;  // [seg][tile], splits added so far
    unsigned long long *counter;
    int *err;
};

// The record pairs go through K2_NST shared-memory stages.  `full` of a stage
// completes when its bulk copy has landed, `empty` when all four warps are done with
// it; thread 0 refills the stage of chunk c - 1 after its own chunk c, so a warp runs
// up to a chunk ahead of or behind the others and no CTA barrier stands between the
// chunks.
// With the field-of-view test each warp culls the stage's records against the cone of
// its own 4 x 8 bins (13.3 ms; 14.9 with one 8 x 16 cone for the CTA, on 16 lists of
// 3,500 polygons x 64,979 bins).  The records' field-of-view data come through the
// stages too and the warp's cones lie in shared memory: read from global memory they held
// 2.0 of the 7.7 stalled cycles an issue (200,000 triangles x 259,560 bins, 13 % of the
// pairs kept: 49.0 -> 45.6 ms).
// POLY: facets of up to 16 vertices as one record each (K2Poly): the direction, the
// polarisation block and the phase once a facet, a divided difference for each triangle
// of its fan.  16 lists of 3,500 facets of 3-6 vertices with the field-of-view test: 9.85
// ms against 12.75 as fans (8.37 now).
template <int BPT, bool FAST, bool POLY>
__global__ void __launch_bounds__(K2_THREADS, BPT == 1 ? 4 : 0) k2_main_pk_kernel(K2PkArgs P) {
    using PairT = std::conditional_t<POLY, K2Poly, K2Pair>;
    constexpr int CHT = FAST ? K2P_CH_FOV : K2P_CH_FULL;
    const int CH = POLY ? P.chunk : CHT;
    constexpr int NW = K2_THREADS / 32;
    __shared__ __align__(128) char sbuf[K2_NST][POLY ? poly_stage(FAST) : CHT * sizeof(K2Pair)];
    __shared__ __align__(128) K2Fov sfov[FAST ? K2_NST : 1][FAST ? 2 * CHT : 1];
    const int stride = POLY ? P.stride : (int)sizeof(K2Pair);
    auto pair_at = [&](int s, int j) -> PairT & { return *reinterpret_cast<PairT *>(sbuf[s] + j * stride); };
    __shared__ __align__(8) uint64_t full[K2_NST], empty[K2_NST];
    __shared__ K2Cone s_cone[FAST ? BPT : 1][NW];  // cones of each warp's bins, written by the warp itself
    __shared__ float4 s_hb[BPT][K2_THREADS];  // forward-bodge bin directions of this CTA's bins
    // the item's FP64 sums, a column per thread: in registers (two bins a thread) they
    // made the compiler spill inside the pair loop
    constexpr bool ACCS = BPT == 1;
    __shared__ double s_acc[ACCS ? 8 : 1][ACCS ? K2_THREADS : 1];
    // the current item, decoded by thread 0: in shared memory, so that its state takes
    // no registers across the pair loop
    __shared__ struct {
        int64_t seg, p0;          // segment; first record pair
        int npair, nchunk, tile, split;
        int edge;                 // bit 0 / 1: the first / last pair is half the item's
        int st0, ph0, issued;     // first stage and its parity, chunks asked for
    } I;
    __shared__ int s_ok;
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < K2_NST; s++) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), NW);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    int st = 0;             // stage of the next chunk
    uint32_t phase = 0;     // its parity: the number of rounds over the stages, modulo 2
    const int64_t total = P.item_pre[P.nseg];
    constexpr int64_t TILE = (int64_t)K2_THREADS * BPT;
    // half phases: k R / 4
    const float2 hkRh = bc2(0.5f * P.hkR);
    // bins with |uz| below pole_cos are out of reach of the forward bodge for every
    // record: |inc . k - (-uz)| <= 2 |com| / R for the direction k from a facet centre
    const float pole_cos = 0.999f - 2.0f * __uint_as_float(*P.epsmax) - 1e-5f;
    const Reach reach = k2_reach(__uint_as_float(*P.epsmax), P.turns);
    for (;;) {
        auto after = [](int s, int n) { return s + n >= K2_NST ? s + n - K2_NST : s + n; };
        // chunk c of the item into its stage (s its index); thread 0 only
        auto load = [&](int c, int s) {
            const int n = min(CH, I.npair - c * CH);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            const char *src = POLY ? P.polys : reinterpret_cast<const char *>(P.pairs);
            const uint32_t bytes = (uint32_t)(n * stride), fbytes = FAST ? (uint32_t)(2 * n * sizeof(K2Fov)) : 0;
            mbar_expect(smem_u32(&full[s]), bytes + fbytes);
            bulk_copy(smem_u32(sbuf[s]), src + (I.p0 + c * CH) * stride, bytes, smem_u32(&full[s]));
            if (FAST) bulk_copy(smem_u32(sfov[s]), P.fovs + 2 * (I.p0 + c * CH), fbytes, smem_u32(&full[s]));
        };
        if (tid == 0) {
            const int64_t item = (int64_t)atomicAdd(P.counter, 1ull);
            I.seg = -1;
            if (item < total) {
                int64_t lo = 0, hi = P.nseg;
                while (hi - lo > 1) {
                    const int64_t m = (lo + hi) >> 1;
                    if (P.item_pre[m] <= item)
                        lo = m;
                    else
                        hi = m;
                }
                const int64_t local = item - P.item_pre[lo];
                const int64_t split = local / P.ntiles;
                const int64_t rbeg = P.seg_rec[lo] + split * P.rpi;
                const int64_t rend = min(rbeg + P.rpi, P.seg_rec[lo + 1]);
                // record pairs [p0, p0 + npair) cover records [rbeg, rend)
                I.seg = lo;
                I.p0 = rbeg >> 1;
                I.npair = (int)(((rend + 1) >> 1) - (rbeg >> 1));
                I.nchunk = (I.npair + CH - 1) / CH;
                I.tile = (int)(local - split * P.ntiles);
                I.split = (int)split;
                I.edge = (int)(rbeg & 1) | (int)(rend & 1) << 1;
                I.st0 = st;
                I.ph0 = (int)phase;
                I.issued = min(I.nchunk, K2_NST);
                // every stage is free: the previous item's chunks were consumed by all warps
                for (int c = 0; c < I.issued; c++) load(c, after(st, c));
            }
        }
        __syncthreads();
        if (I.seg < 0) break;
        // the bin of this thread's slot q in the item's tile, -1: none
        auto bin_of = [&](int q) {
            const int64_t li = I.tile * TILE + q * K2_THREADS + tid;
            return FAST ? P.perm[li] : li < P.nb ? (int)li : -1;
        };
        BinPk bd[BPT];
#pragma unroll
        for (int q = 0; q < BPT; q++) {
            bd[q].bin = bin_of(q);
            const int64_t o = bd[q].bin >= 0 ? bd[q].bin : 0;
            const double X = P.xyz[o], Y = P.xyz[P.nb + o], Zc = P.xyz[2 * P.nb + o];
            const double ir = 1.0 / sqrt(X * X + Y * Y + Zc * Zc);
            bd[q].ux = X * ir;
            bd[q].uy = Y * ir;
            bd[q].uz = Zc * ir;
            bd[q].fx = bc2((float)bd[q].ux);
            bd[q].fy = bc2((float)bd[q].uy);
            bd[q].fz = bc2((float)bd[q].uz);
            bd[q].pole = !(fabs(bd[q].uz) < (double)pole_cos);
            const int64_t oh = (o % P.nphi) + P.nphi * P.theta_i;
            const double Xh = P.xyz[oh], Yh = P.xyz[P.nb + oh], Zh = P.xyz[2 * P.nb + oh];
            const double irh = 1.0 / sqrt(Xh * Xh + Yh * Yh + Zh * Zh);
            s_hb[q][tid] = make_float4((float)(Xh * irh), (float)(Yh * irh), (float)(Zh * irh), 0.0f);
        }
        double acc64[BPT][8];
        auto sum = [&](int q, int c) -> double & {
            if constexpr (ACCS)
                return s_acc[c][tid];
            else
                return acc64[q][c];
        };
#pragma unroll
        for (int q = 0; q < BPT; q++)
#pragma unroll
            for (int c = 0; c < 8; c++) sum(q, c) = 0.0;
        if (FAST) {
#pragma unroll
            for (int q = 0; q < BPT; q++)
                if (lane < 8)
                    reinterpret_cast<float *>(&s_cone[q][tid >> 5])[lane] = reinterpret_cast<const float *>(
                        &P.cones[((int64_t)I.tile * BPT + q) * NW + (tid >> 5)])[lane];
            __syncwarp();
        }
        bool pole = false;
#pragma unroll
        for (int q = 0; q < BPT; q++) pole = pole || bd[q].pole;
        pole = __any_sync(0xffffffffu, pole);
        bool failed = false;
        for (int c = 0; c < I.nchunk; c++) {
            if (__any_sync(0xffffffffu, !mbar_wait(smem_u32(&full[st]), phase))) {
                failed = true;
                break;
            }
            const int n = min(CH, I.npair - c * CH);
            // The item's first pair (odd rbeg) and last pair (odd rend) hold a record of another
            // item or, at the end of an odd list, one that was never written: that half takes a
            // copy of the pair's other record with zero amplitude.  A stranger's infinite or
            // NaN amplitude cannot reach the sums then (0 times it is NaN), nor its kx^2 + kz^2
            // the choice of the step, and without the field-of-view test the pair loop
            // needs no per-pair range test.  Every warp writes the same values for itself:
            // 3 FP64 phases, then the float2 fields from eps on (8 of them the amplitudes; a
            // polygon's length m belongs to both halves, its vertices follow).
            auto patch = [&](int j, int src, int dst) {
                PairT &Q = pair_at(st, j);
                float2 *f = &Q.eps[0];
                const int amp0 = (int)(&Q.amp[0] - f);
                const int nf = (stride - (int)((char *)f - (char *)&Q)) / 8;
                for (int t = lane; t < 3 + nf; t += 32) {
                    if (t < 3) {
                        Q.kc[t][dst] = Q.kc[t][src];
                    } else if (!POLY || t - 3 != amp0 - 1) {
                        const int i = t - 3;
                        const float v = i >= amp0 && i < amp0 + 8 ? 0.0f : (src ? f[i].y : f[i].x);
                        if (dst)
                            f[i].y = v;
                        else
                            f[i].x = v;
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
            };
            if (c == 0 && (I.edge & 1)) patch(0, 1, 0);
            if (c == I.nchunk - 1 && (I.edge & 2)) patch(n - 1, 0, 1);
            float2 acc[BPT][8];
            [[maybe_unused]] unsigned pm0 = 0, keep[2] = {0, 0};
            if (FAST) {
                // the tile cull of the stage's 2n records, two per lane: a record
                // whose field of view misses the warp's bins adds nothing
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int r = h * 32 + lane;
                    bool k = false;
                    if (r < 2 * n) {
                        const K2Fov &f = sfov[st][r];
#pragma unroll
                        for (int q = 0; q < BPT; q++)
                            k = k || !cone_culled(f, s_cone[q][tid >> 5]);
                    }
                    keep[h] = __ballot_sync(0xffffffffu, k);
                }
                if (c == 0 && (I.edge & 1)) keep[0] &= ~1u;
                if (c == I.nchunk - 1 && (I.edge & 2)) keep[(2 * n - 1) >> 5] &= ~(1u << ((2 * n - 1) & 31));
                // visit only the pairs with a record the cull kept: bit j of pm is
                // set when record 2j or 2j+1 is (the two ballot words compacted)
                auto pairs_of = [](unsigned x) {
                    x = (x | (x >> 1)) & 0x55555555u;
                    x = (x | (x >> 1)) & 0x33333333u;
                    x = (x | (x >> 2)) & 0x0F0F0F0Fu;
                    x = (x | (x >> 4)) & 0x00FF00FFu;
                    x = (x | (x >> 8)) & 0x0000FFFFu;
                    return x;
                };
                pm0 = pairs_of(keep[0]) | (pairs_of(keep[1]) << 16);
            }
            // Without the field-of-view test every lane adds (the edge pairs are patched
            // above; a bin beyond nb is never written out).
            float tmin = 1.0f;
            auto pairs = [&](auto step_, auto reach_) {
                constexpr Step ST = decltype(step_)::value;
                constexpr Reach RE = decltype(reach_)::value;
#pragma unroll
                for (int q = 0; q < BPT; q++)
#pragma unroll
                    for (int cc = 0; cc < 8; cc++) acc[q][cc] = bc2(0.0f);
                if constexpr (FAST) {
                    for (unsigned pm = pm0; pm; pm &= pm - 1u) {
                        const int j = __ffs(pm) - 1;
                        const unsigned m = (j & 16 ? keep[1] : keep[0]) >> (2 * (j & 15));
                        const K2FovExact *fx = P.fovx + 2 * (I.p0 + c * CH + j);
#pragma unroll
                        for (int q = 0; q < BPT; q++)
                            k2_pair<true, ST, RE>(pair_at(st, j), &sfov[st][2 * j], fx, bd[q], acc[q], hkRh, tmin, s_hb[q][tid],
                                                 (m & 1u) && bd[q].bin >= 0, (m & 2u) && bd[q].bin >= 0,
                                                 P.xyz, P.nb, P.rlo + (I.p0 + c * CH + j) * 3);
                    }
                } else {
                    for (int j = 0; j < n; j++)
#pragma unroll
                        for (int q = 0; q < BPT; q++)
                            k2_pair<false, ST, RE>(pair_at(st, j), nullptr, nullptr, bd[q], acc[q], hkRh, tmin,
                                                  s_hb[q][tid], true, true, P.xyz, P.nb,
                                                  P.rlo + (I.p0 + c * CH + j) * 3);
                }
            };
            // A warp that meets the clamp of ky (a 0.08 degree cone around a facet's second
            // axis) does the chunk again.
            bool again = reach == Reach::Wide;
            if (!again) {
                if (pole)
                    pairs(PoleC(), MidC());
                else if (reach == Reach::Near)
                    pairs(MainC(), NearC());
                else
                    pairs(MainC(), MidC());
                again = __any_sync(0xffffffffu, tmin <= kOneMinusClampSq);
            }
            if (again) pairs(FullC(), WideC());
#pragma unroll
            for (int q = 0; q < BPT; q++)
#pragma unroll
                for (int cc = 0; cc < 8; cc++)
                    sum(q, cc) += (double)acc[q][cc].x + (double)acc[q][cc].y;
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&empty[st]));
            // the stage before this one (chunk c - 1) takes chunk c - 1 + K2_NST once
            // every warp has left it; its parity is this stage's, or the round before
            if (tid == 0 && c > 0 && c - 1 + K2_NST < I.nchunk) {
                const int sp = st == 0 ? K2_NST - 1 : st - 1;
                if (mbar_wait(smem_u32(&empty[sp]), st == 0 ? phase ^ 1u : phase)) {
                    load(c - 1 + K2_NST, sp);
                    I.issued = c + K2_NST;
                } else {
                    failed = true;  // the other warps' waits for its chunk run out too
                }
            }
            st = after(st, 1);
            if (st == 0) phase ^= 1u;
            if (__any_sync(0xffffffffu, failed)) break;
        }
        unsigned *tk = P.tickets + I.seg * P.ntiles + I.tile;
        if (__syncthreads_or(failed)) {
            if (tid == 0) {
                atomicOr(P.err, 4);
                atomicMax(tk, kTicketPoison);
                // bounded wait for this CTA's bulk copies still in flight: the latest
                // copy of every stage
                for (int c = max(0, I.issued - K2_NST); c < I.issued; c++)
                    mbar_wait(smem_u32(&full[(I.st0 + c) % K2_NST]),
                              (uint32_t)(I.ph0 ^ (((I.st0 + c) / K2_NST) & 1)));
            }
            return;
        }
        // back from the circular basis: a1 = (U+ + U-)/2, a2 = -i (U+ - U-)/2
        double lin[BPT][8];
#pragma unroll
        for (int q = 0; q < BPT; q++) {
            double u[8];
#pragma unroll
            for (int c = 0; c < 8; c++) u[c] = sum(q, c);
            lin[q][0] = 0.5 * (u[0] + u[2]);
            lin[q][1] = 0.5 * (u[1] + u[3]);
            lin[q][2] = 0.5 * (u[1] - u[3]);
            lin[q][3] = 0.5 * (u[2] - u[0]);
            lin[q][4] = 0.5 * (u[4] + u[6]);
            lin[q][5] = 0.5 * (u[5] + u[7]);
            lin[q][6] = 0.5 * (u[5] - u[7]);
            lin[q][7] = 0.5 * (u[6] - u[4]);
        }
        bool valid[BPT];
        int64_t bin[BPT];
#pragma unroll
        for (int q = 0; q < BPT; q++) {
            bin[q] = bin_of(q);
            valid[q] = bin[q] >= 0;
        }
        ordered_add<BPT>(P.ws + I.seg * 8 * P.nb, P.nb, tk, (unsigned)I.split, valid, bin, lin, &s_ok,
                         P.err);
    }
}

// --------------------------------------------------------------- epilogue

struct Zd {
    double re, im;
};
__device__ __forceinline__ double re_mc(Zd a, Zd b) { return a.re * b.re + a.im * b.im; }
__device__ __forceinline__ double im_mc(Zd a, Zd b) { return a.im * b.re - a.re * b.im; }

__device__ __forceinline__ void mueller16d(const Zd *S, double mu[16]) {
    const Zd a11 = S[0], a21 = S[1], a12 = S[2], a22 = S[3];
    const double p11 = re_mc(a11, a11), p12 = re_mc(a12, a12), p21 = re_mc(a21, a21),
                 p22 = re_mc(a22, a22);
    mu[0] = 0.5 * (p11 + p12 + p21 + p22);
    mu[1] = 0.5 * (p11 - p12 + p21 - p22);
    mu[2] = re_mc(a11, a12) + re_mc(a22, a21);
    mu[3] = im_mc(a11, a12) - im_mc(a22, a21);
    mu[4] = 0.5 * (p11 + p12 - p21 - p22);
    mu[5] = 0.5 * (p11 - p12 - p21 + p22);
    mu[6] = re_mc(a11, a12) - re_mc(a22, a21);
    mu[7] = im_mc(a11, a12) + im_mc(a22, a21);
    mu[8] = re_mc(a11, a21) + re_mc(a22, a12);
    mu[9] = re_mc(a11, a21) - re_mc(a22, a12);
    mu[10] = re_mc(a11, a22) + re_mc(a12, a21);
    mu[11] = im_mc(a11, a22) + im_mc(a21, a12);
    mu[12] = im_mc(a21, a11) + im_mc(a22, a12);
    mu[13] = im_mc(a21, a11) - im_mc(a22, a12);
    mu[14] = im_mc(a22, a11) - im_mc(a12, a21);
    mu[15] = re_mc(a22, a11) - re_mc(a12, a21);
}

// Amplitude of segment seg at bin o as reference-layout complex 2x2 (with
// T(phi) applied and scaled by sc), common phase e^{ik|X|} omitted.  A segment
// without records has no work items and nothing in the workspace: zero.
__device__ __forceinline__ void ws_ampl(const double *ws, const int64_t *seg_rec, int64_t seg, int64_t nb,
                                        int64_t o, double cp, double sp, double sc, Zd S[4]) {
    const double *w = ws + seg * 8 * nb + o;
    Zd a[4];
    const bool some = seg_rec[seg + 1] > seg_rec[seg];
#pragma unroll
    for (int c = 0; c < 4; c++) {
        a[c].re = some ? w[(2 * c) * nb] : 0.0;
        a[c].im = some ? w[(2 * c + 1) * nb] : 0.0;
    }
    // (S T)(a,b) = S(a,1) T(1,b) + S(a,2) T(2,b); T = [[-s, -c], [c, -s]]
    // order (1,1),(2,1),(1,2),(2,2): a[0]=S11 a[1]=S21 a[2]=S12 a[3]=S22
    const double T11 = -sp, T12 = -cp, T21 = cp, T22 = -sp;
    S[0] = {(a[0].re * T11 + a[2].re * T21) * sc, (a[0].im * T11 + a[2].im * T21) * sc};
    S[1] = {(a[1].re * T11 + a[3].re * T21) * sc, (a[1].im * T11 + a[3].im * T21) * sc};
    S[2] = {(a[0].re * T12 + a[2].re * T22) * sc, (a[0].im * T12 + a[2].im * T22) * sc};
    S[3] = {(a[1].re * T12 + a[3].re * T22) * sc, (a[1].im * T12 + a[3].im * T22) * sc};
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

constexpr int K2_EPI_THREADS = 256;

// Per-orientation sums over the bins are reduced in two fixed-order steps (a warp's
// sum into part[(q K + k) nwarp + warp], then k2_part_sum_kernel over the warps in
// order), so they are the same from run to run and no block waits for its warps.
// Pre-pass of -scaling: per-orientation scatt_beam / scatt_ext sums; blockIdx.y takes
// every gridDim.y-th orientation.
__global__ void k2_scatt_be_kernel(const double *__restrict__ ws, const int64_t *__restrict__ seg_rec,
                                   int64_t no, int64_t nb, int64_t nphi,
                                   const double *__restrict__ phitab, double waveno,
                                   const double *__restrict__ wbin, double *__restrict__ part) {
    const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = o < nb;
    const int64_t oo = in ? o : 0;
    const double cp = phitab[oo % nphi], sp = phitab[nphi + oo % nphi];
    const double W = in ? wbin[oo] / (waveno * waveno) : 0.0;
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5), w = o >> 5;
    for (int64_t q = blockIdx.y; q < no; q += gridDim.y) {
        Zd S[4];
        double m[16];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            ws_ampl(ws, seg_rec, 2 * q + k, nb, oo, cp, sp, waveno, S);
            mueller16d(S, m);
            const double v = warp_sum(W * m[0]);
            if ((threadIdx.x & 31) == 0) part[(2 * q + k) * nw + w] = v;
        }
    }
}
// out[r] = sum over b of part[r n + b] (a block per row: each thread its stride in
// order, then a fixed tree).
__global__ void k2_part_sum_kernel(const double *__restrict__ part, int64_t n, double *__restrict__ out) {
    __shared__ double red[8];
    const double *p = part + blockIdx.x * n;
    double v = 0.0;
    for (int64_t b = threadIdx.x; b < n; b += blockDim.x) v += p[b];
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = red[0];
        for (int i = 1; i < (int)(blockDim.x >> 5); i++) t += red[i];
        out[blockIdx.x] = t;
    }
}

// sqrt(scatt_part / energy_part) per orientation (src/outputs_mod.f90:151,154)
__global__ void k2_scale_kernel(double *__restrict__ scale, const pbt_output_params *__restrict__ pin,
                                int64_t o0, int64_t no) {
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= no) return;
    const int64_t o = o0 + q;
    scale[2 * o] = sqrt(scale[2 * o] / pin[o].beam_energy_out);
    scale[2 * o + 1] = sqrt(scale[2 * o + 1] / pin[o].ext_energy_out);
}

// Main epilogue: Mueller sum over the chunk's orientations and per-orientation
// weighted sums  red[o] = {scatt, scatt_beam, scatt_ext, g_num, g_num_beam, g_num_ext}.
// blockIdx.y takes every gridDim.y-th orientation; with more than one, each leaves its
// own Mueller sum in dst + blockIdx.y * 16 nb (k2_fold_kernel adds them), otherwise dst
// is the running sum, stored (first) or added to.
// Bound: HBM (128 B a bin and orientation).  A small grid has too few bins to fill the
// SMs and walked its orientations one after another, twelve block barriers each: 256
// orientations x 6,552 bins took 745 us, 86 us with the orientations over
// blockIdx.y and warp sums.
__global__ void __launch_bounds__(K2_EPI_THREADS)
    k2_epi_kernel(const double *__restrict__ ws, const int64_t *__restrict__ seg_rec, int64_t no, int64_t o0,
                  int64_t nb, int64_t nphi, const double *__restrict__ phitab, const double *__restrict__ cth,
                  double waveno, const double *__restrict__ wbin, int64_t back_bin,
                  const double *__restrict__ scale, double *__restrict__ dst, int first,
                  double *__restrict__ part, double *__restrict__ bs) {
    const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = o < nb;
    const int64_t oo = in ? o : 0;
    const int64_t i = oo % nphi, j = oo / nphi;
    const double cp = phitab[i], sp = phitab[nphi + i];
    const double W = in ? wbin[oo] / (waveno * waveno) : 0.0;
    const double ct = cth[j];
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5), w = o >> 5;
    double acc[16];
#pragma unroll
    for (int e = 0; e < 16; e++) acc[e] = 0.0;
    for (int64_t q = blockIdx.y; q < no; q += gridDim.y) {
        const int64_t og = o0 + q;
        const double sb = scale ? 1.0 / scale[2 * og] : 1.0;
        const double se = scale ? 1.0 / scale[2 * og + 1] : 1.0;
        Zd Sb[4], Se[4], St[4];
        ws_ampl(ws, seg_rec, 2 * q, nb, oo, cp, sp, waveno * sb, Sb);
        ws_ampl(ws, seg_rec, 2 * q + 1, nb, oo, cp, sp, waveno * se, Se);
#pragma unroll
        for (int c = 0; c < 4; c++) St[c] = {Sb[c].re + Se[c].re, Sb[c].im + Se[c].im};
        double m[16];
        mueller16d(St, m);
#pragma unroll
        for (int e = 0; e < 16; e++) acc[e] += m[e];
        const double mb = 0.5 * (re_mc(Sb[0], Sb[0]) + re_mc(Sb[2], Sb[2]) + re_mc(Sb[1], Sb[1]) +
                                 re_mc(Sb[3], Sb[3]));
        const double me = 0.5 * (re_mc(Se[0], Se[0]) + re_mc(Se[2], Se[2]) + re_mc(Se[1], Se[1]) +
                                 re_mc(Se[3], Se[3]));
        const double v[6] = {W * m[0], W * mb, W * me, W * ct * m[0], W * ct * mb, W * ct * me};
#pragma unroll
        for (int k = 0; k < 6; k++) {
            const double t = warp_sum(v[k]);
            if ((threadIdx.x & 31) == 0) part[(6 * q + k) * nw + w] = t;
        }
        if (in && o == back_bin) bs[og] = m[0] * 4.0 * kPiRef / (waveno * waveno);
    }
    if (!in) return;
    if (gridDim.y > 1) dst += (int64_t)blockIdx.y * 16 * nb;
#pragma unroll
    for (int e = 0; e < 16; e++) {
        double *d = dst + e * nb + o;
        *d = gridDim.y > 1 || first ? acc[e] : *d + acc[e];
    }
}

// mu_sum (stored when first, else added to) = the ny partial Mueller sums in order
__global__ void k2_fold_kernel(const double *__restrict__ part, int ny, int64_t n, int first,
                               double *__restrict__ mu_sum) {
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    double s = first ? 0.0 : mu_sum[q];
    for (int y = 0; y < ny; y++) s += part[y * n + q];
    mu_sum[q] = s;
}

// Per-orientation parameters (finalise, src/outputs_mod.f90:133-245), then their
// orientation average (summation and divide): one block, a warp per field for the
// average.
__global__ void __launch_bounds__(608)
    k2_final_kernel(const double *__restrict__ redo, const double *__restrict__ bs,
                    const pbt_output_params *__restrict__ pin, int64_t norient,
                    pbt_output_params *__restrict__ pout, pbt_output_params *__restrict__ avg) {
    for (int64_t o = threadIdx.x; o < norient; o += blockDim.x) {
        const double *r = redo + 6 * o;
        pbt_output_params p = pin[o];
        const double scatt = r[0], scatt_b = r[1], scatt_e = r[2];
        p.scatt = scatt;
        p.ext = p.abs + scatt;
        p.albedo = 1 - (p.ext - scatt) / p.ext;
        p.asymmetry = r[3] / scatt;
        p.abs_eff = p.abs / p.geo_cross_sec;
        p.scatt_eff = scatt / p.geo_cross_sec;
        p.ext_eff = p.ext / p.geo_cross_sec;
        p.back_scatt = bs[o];
        p.scatt_beam = scatt_b;
        p.scatt_ext_diff = scatt_e;
        p.asymmetry_beam = r[4] / scatt_b;
        p.asymmetry_ext_diff = r[5] / scatt_e;
        p.scatt_eff_beam = scatt_b / p.geo_cross_sec;
        p.scatt_eff_ext_diff = scatt_e / p.geo_cross_sec;
        pout[o] = p;
    }
    __threadfence_block();
    __syncthreads();
    const int f = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (f >= 18) return;
    const double *src = reinterpret_cast<const double *>(pout);
    double s = 0.0;
    for (int64_t o = lane; o < norient; o += 32) s += src[18 * o + f];
    s = warp_sum(s);
    // beam_energy_out / ext_energy_out are not summed by the reference
    if (lane == 0) reinterpret_cast<double *>(avg)[f] = (f == 10 || f == 11) ? 0.0 : s / (double)norient;
}

// The orientation average of the Mueller sums and its phi integral: a warp per theta
// row and element.
__global__ void k2_avg_kernel(const double *__restrict__ mu_sum, const double *__restrict__ wphi,
                              int64_t nphi, int64_t ntheta, double norient, double *__restrict__ mu_avg,
                              double *__restrict__ m1d) {
    const int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= 16 * ntheta) return;
    const int64_t j = t % ntheta, e = t / ntheta, row = (e * ntheta + j) * nphi;
    double s = 0.0;
    for (int64_t i = lane; i < nphi; i += 32) {
        const double v = mu_sum[row + i] / norient;
        mu_avg[row + i] = v;
        s += wphi[i] * v;
    }
    s = warp_sum(s);
    if (lane == 0) m1d[j + ntheta * e] = s;
}

// FP32 diff_main output: reference-layout complex(8) grids, e^{ik|X|} S' T(phi).
__global__ void k2_ampl_out_kernel(const double *__restrict__ ws, const int64_t *__restrict__ seg_rec,
                                   int64_t nb, int64_t nphi,
                                   const double *__restrict__ phitab, const double *__restrict__ xyz,
                                   double waveno, double *__restrict__ afb, double *__restrict__ afe) {
    const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= nb) return;
    const double cp = phitab[o % nphi], sp = phitab[nphi + o % nphi];
    const double X = xyz[o], Y = xyz[nb + o], Zc = xyz[2 * nb + o];
    double sK, cK;
    sincos(waveno * sqrt(X * X + Y * Y + Zc * Zc), &sK, &cK);
    for (int kind = 0; kind < 2; kind++) {
        Zd S[4];
        ws_ampl(ws, seg_rec, kind, nb, o, cp, sp, 1.0, S);
        double *dst = kind ? afe : afb;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            dst[2 * (o + nb * c)] = S[c].re * cK - S[c].im * sK;
            dst[2 * (o + nb * c) + 1] = S[c].re * sK + S[c].im * cK;
        }
    }
}

}  // namespace

// --------------------------------------------------------------- host side

namespace {

// Launch shape of the main kernel.  variant 1 = packed two-facet kernel over
// K2Pair records, 0 = one facet per step over K2Rec records.  bpt = bins per
// thread, rpi = facet records per work item.  PBT_K2_PLAN="variant,bpt,rpi"
// overrides the default (used by the tuner).
K2Plan k2_plan_for(const pbt_ctx *ctx) {
    K2Plan p;
    if (ctx->plan_variant >= 0) {
        p.variant = ctx->plan_variant;
        p.bpt = ctx->plan_bpt;
        p.rpi = ctx->plan_rpi;
        p.auto_rpi = false;
        return p;
    }
    if (const char *e = getenv("PBT_K2_PLAN")) {
        int v = 0, b = 0;
        long long r = 0;
        if (sscanf(e, "%d,%d,%lld", &v, &b, &r) == 3 && (v == 0 || v == 1) && (b == 1 || b == 2) &&
            r >= 32 && r <= (1 << 22)) {
            p.variant = v;
            p.bpt = b;
            p.rpi = r;
            p.auto_rpi = false;
        }
    }
    return p;
}

// Device-side set-up shared by the batched and single-orientation entry points.
struct K2Setup {
    K2Rec *recs = nullptr;
    K2Pair *pairs = nullptr;
    char *polys = nullptr;  // facet pairs of polygons, poly_stride bytes each
    int64_t poly_stride = 0;
    K2Fov *fovs = nullptr;
    K2FovExact *fovx = nullptr;
    float2 *rlo = nullptr;  // R_1 - (float)R_1 per record (the y row), pair layout (3 per pair)
    RefSrc src{};
};

// Error flags of a call (or of all its runs) and a bound of |com| / R over the
// records, set to zero before the first set-up.
struct K2Flags {
    int err, pad;
    unsigned epsmax, pad2;  // float bits
};

size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

// Smallest and largest vertex count of the faces.
struct FaceRange {
    int64_t lo, hi;
};
FaceRange face_range(const int64_t *h_face_off, int64_t nfaces) {
    FaceRange r{h_face_off[1] - h_face_off[0], 3};
    for (int64_t f = 0; f < nfaces; f++) {
        const int64_t nv = h_face_off[f + 1] - h_face_off[f];
        r.lo = std::min(r.lo, nv);
        r.hi = std::max(r.hi, nv);
    }
    return r;
}

int k2_prepare(pbt_ctx *ctx, cudaStream_t st, int64_t norient, const pbt_outbeam *d_beam,
               const int64_t *h_beam_off, const pbt_outbeam *d_ext, const int64_t *h_ext_off,
               const double *d_verts, int64_t nverts, const int64_t *h_face_off,
               const int64_t *d_face_off, const int64_t *d_face_vi, int64_t nfaces, double lambda,
               int fast_diff, const K2Plan &plan, K2Flags *flags, K2Setup &S) {
    pbt::NvtxRange nvtx_("pbt: set-up (records)");
    const int64_t nrefs = h_beam_off[norient] + h_ext_off[norient];
    const FaceRange nv = face_range(h_face_off, nfaces);
    const int variant = plan.variant;
    // One record a facet (k2_main_pk_kernel's POLY) from 1.2 triangles a face on, one a
    // triangle of the fan below and with the other plans.  Measured on 6 lists of 3,500
    // facets, 361 x 180 bins, quads among triangles: 10 % quads 6.97 ms (facets) against
    // 6.71 (fans), 20 % 7.49 against 7.51, all quads 9.31 against 12.08.
    const bool poly = variant == 1 && plan.bpt == 1 && nv.hi > 3 && 5 * h_face_off[nfaces] >= 16 * nfaces;
    const int64_t nvp = std::min<int64_t>(nv.hi, kMaxPolyVerts);
    const int64_t max_recs = std::max<int64_t>(1, nrefs * (poly ? 1 : std::max<int64_t>(1, nv.hi - 2)));
    // Faces of one vertex count (triangles nearly always): outbeam g's records start at
    // g (nv - 2), so the count and its scan (three launches) are for mixed fans only.
    const bool uniform = poly || nv.lo == nv.hi;
    size_t scan_tmp = 0;
    if (!uniform)
        cub::DeviceScan::ExclusiveSum(nullptr, scan_tmp, (int64_t *)nullptr, (int64_t *)nullptr,
                                      (int)(nrefs + 1), st);
    // With the field-of-view test the outbeams of each list are put in order of direction,
    // where the sum is large enough to pay for the sort (40 us): 16 lists of 3,500 polygons
    // of random directions x 64,979 bins, kernel 9.44 -> 8.37 ms; one list of 4,800
    // triangles x 259,560 bins, a pass 2.18 -> 1.96 ms; 2,000 beams of 100 outbeams x
    // 259,560 bins, which keep their order, 44.55 ms (45.3 sorted).  The sort is stable, so
    // the order depends on the lists alone.  An explicit plan fixes the order of summation
    // whatever the call's size and sorts nothing.
    int sort_bits = 2 * kOrderBits;
    while (sort_bits < 40 && ((int64_t)1 << (sort_bits - 2 * kOrderBits)) < 2 * norient) sort_bits++;
    const bool sorted = fast_diff && variant == 1 && plan.auto_rpi && sort_bits <= 32 && nrefs < INT32_MAX &&
                        (double)nrefs * (double)ctx->grid.nb >= 1e9;
    size_t sort_tmp = 0;
    if (sorted)
        cub::DeviceRadixSort::SortPairs(nullptr, sort_tmp, (const unsigned *)nullptr, (unsigned *)nullptr,
                                        (const int *)nullptr, (int *)nullptr, (int)nrefs, 0, sort_bits, st);
    // d_scan: refbase, beam_off, ext_off | cnt | start | scan tmp | sort keys, positions, tmp
    const size_t nc = uniform ? 0 : (size_t)(nrefs + 1) * 8;
    const size_t o_rb = 0, o_cnt = align_up(o_rb + 3 * (norient + 1) * 8), o_start = align_up(o_cnt + nc),
                 o_tmp = align_up(o_start + nc), o_key = align_up(o_tmp + scan_tmp);
    const size_t n4 = sorted ? align_up((size_t)nrefs * 4) : 0;
    const size_t o_alike = o_key + 4 * n4, o_stmp = o_alike + (sorted ? 256 : 0), o_end = align_up(o_stmp + sort_tmp);
    PBT_TRY(ctx->d_scan.ensure(o_end));
    char *base = ctx->d_scan.as<char>();
    int64_t *rb = (int64_t *)(base + o_rb), *cnt = (int64_t *)(base + o_cnt);
    RefSrc &src = S.src;
    src.beam = d_beam;
    src.ext = d_ext;
    src.refbase = rb;
    src.beam_off = rb + (norient + 1);
    src.ext_off = rb + 2 * (norient + 1);
    src.norient = norient;
    src.start = uniform ? nullptr : (int64_t *)(base + o_start);
    src.per = poly ? 1 : nv.lo - 2;
    src.order = nullptr;
    S.poly_stride = poly ? (int64_t)(sizeof(K2Poly) + nvp * sizeof(K2PolyVertex)) : 0;
    // records (or record pairs; an even count so the last pair is whole)
    const int64_t nrec2 = (max_recs + 1) & ~(int64_t)1;
    const size_t rec_bytes = poly      ? (size_t)(nrec2 / 2) * S.poly_stride
                             : variant ? (size_t)(nrec2 / 2) * sizeof(K2Pair)
                                       : (size_t)max_recs * sizeof(K2Rec);
    const size_t fov_head = fast_diff ? align_up(nrec2 * sizeof(K2Fov)) : 0;
    const size_t fov_bytes = fast_diff ? fov_head + align_up(nrec2 * sizeof(K2FovExact)) : 0;
    PBT_TRY(ctx->d_rec.ensure(align_up(rec_bytes) + fov_bytes + (size_t)(nrec2 / 2) * 3 * sizeof(float2)));
    S.recs = variant ? nullptr : ctx->d_rec.as<K2Rec>();
    S.pairs = variant && !poly ? ctx->d_rec.as<K2Pair>() : nullptr;
    S.polys = poly ? ctx->d_rec.as<char>() : nullptr;
    S.fovs = fast_diff ? (K2Fov *)(ctx->d_rec.as<char>() + align_up(rec_bytes)) : nullptr;
    S.fovx = fast_diff ? (K2FovExact *)(ctx->d_rec.as<char>() + align_up(rec_bytes) + fov_head) : nullptr;
    S.rlo = (float2 *)(ctx->d_rec.as<char>() + align_up(rec_bytes) + fov_bytes);
    // host-side offsets -> device (pinned staging; the previous call's copy
    // out of the staging buffer must have run before it is overwritten)
    if (ctx->stage_pending && !ctx->capturing) {
        PBT_CUDA_TRY(cudaEventSynchronize(ctx->stage_ev));
        ctx->stage_pending = false;
    }
    if (!ctx->stage_ev) PBT_CUDA_TRY(cudaEventCreateWithFlags(&ctx->stage_ev, cudaEventDisableTiming));
    PBT_TRY(ctx->h_stage.ensure(3 * (norient + 1) * 8));
    int64_t *hs = ctx->h_stage.as<int64_t>();
    for (int64_t o = 0; o <= norient; o++) {
        hs[o] = h_beam_off[o] + h_ext_off[o];
        hs[norient + 1 + o] = h_beam_off[o];
        hs[2 * (norient + 1) + o] = h_ext_off[o];
    }
    PBT_CUDA_TRY(cudaMemcpyAsync(rb, hs, 3 * (norient + 1) * 8, cudaMemcpyHostToDevice, st));
    if (!ctx->capturing) {
        PBT_CUDA_TRY(cudaEventRecord(ctx->stage_ev, st));
        ctx->stage_pending = true;
    }
    if (sorted) {
        unsigned *keys = (unsigned *)(base + o_key);
        int *pos = (int *)(base + o_key + 2 * n4), *order = (int *)(base + o_key + 3 * n4);
        int *alike = (int *)(base + o_alike);
        const unsigned blocks = (unsigned)((nrefs + 127) / 128);
        PBT_CUDA_TRY(cudaMemsetAsync(alike, 0, sizeof(int), st));
        k2_order_kernel<<<blocks, 128, 0, st>>>(src, nrefs, keys, pos, alike);
        k2_keep_order_kernel<<<blocks, 128, 0, st>>>(nrefs, keys, alike);
        PBT_CUDA_TRY(cub::DeviceRadixSort::SortPairs(base + o_stmp, sort_tmp, (const unsigned *)keys,
                                                     (unsigned *)(base + o_key + n4), (const int *)pos, order,
                                                     (int)nrefs, 0, sort_bits, st));
        ctx->launches += 3;
        src.order = order;
    }
    if (!uniform) {
        const int th = 256;
        k2_count_kernel<<<(unsigned)((nrefs + 1 + th - 1) / th), th, 0, st>>>(src, nrefs, d_face_off,
                                                                              nfaces, cnt, &flags->err);
        PBT_CUDA_TRY(cub::DeviceScan::ExclusiveSum(base + o_tmp, scan_tmp, cnt, (int64_t *)(base + o_start),
                                                   (int)(nrefs + 1), st));
        ctx->launches += 2;
    }
    const double waveno = 2.0 * kPiRef / lambda;
    // 64 threads: a short list's set-up is one chain of FP64 steps a thread, spread over
    // the SMs
    const int th = 64;
    if (nrefs > 0 && poly)
        k2_setup_poly_kernel<<<(unsigned)((nrefs + th - 1) / th), th, 0, st>>>(
            src, nrefs, d_verts, nverts, d_face_off, nfaces, d_face_vi, waveno, lambda, fast_diff, (int)nvp,
            S.polys, S.poly_stride, S.fovs, S.fovx, S.rlo, &flags->err, &flags->epsmax);
    else if (nrefs > 0)
        k2_setup_kernel<<<(unsigned)((nrefs + th - 1) / th), th, 0, st>>>(
            src, nrefs, d_verts, nverts, d_face_off, nfaces, d_face_vi, waveno, lambda, fast_diff,
            S.recs, S.pairs, S.fovs, S.fovx, S.rlo, &flags->err, &flags->epsmax);
    ctx->launches++;
    PBT_CUDA_TRY(cudaGetLastError());
    return PBT_OK;
}

template <int BPT, bool FAST>
int k2_launch_main(pbt_ctx *ctx, cudaStream_t st, const K2MainArgs &A) {
    // resident CTAs per SM, computed once (thread-safe static initialisation)
    static const int occ = [] {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k2_main_kernel<BPT, FAST>, K2_THREADS, 0) !=
            cudaSuccess)
            (void)cudaGetLastError();
        return n > 0 ? n : 1;
    }();
    const int grid = ctx->sm_count * occ;
    timing_begin(ctx, st);
    k2_main_kernel<BPT, FAST><<<grid, K2_THREADS, 0, st>>>(A);
    timing_end(ctx, st);
    ctx->launches++;
    PBT_CUDA_TRY(cudaGetLastError());
    return PBT_OK;
}

template <int BPT, bool FAST, bool POLY>
int k2_launch_pk(pbt_ctx *ctx, cudaStream_t st, const K2PkArgs &A) {
    static const int occ = [] {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k2_main_pk_kernel<BPT, FAST, POLY>, K2_THREADS,
                                                          0) != cudaSuccess)
            (void)cudaGetLastError();
        return n > 0 ? n : 1;
    }();
    const int grid = ctx->sm_count * occ;
    timing_begin(ctx, st);
    k2_main_pk_kernel<BPT, FAST, POLY><<<grid, K2_THREADS, 0, st>>>(A);
    timing_end(ctx, st);
    ctx->launches++;
    PBT_CUDA_TRY(cudaGetLastError());
    return PBT_OK;
}

// One warp per group of `tile` bins: unit centre of their directions and the
// largest angle of a bin from it (FP64).
__global__ void k2_cone_kernel(const int *__restrict__ perm, int64_t ntiles, int64_t tile,
                               const double *__restrict__ xyz, int64_t nb, K2Cone *__restrict__ cones) {
    const int64_t t = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= ntiles) return;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    int n = 0;
    for (int64_t i = lane; i < tile; i += 32) {
        const int o = perm[t * tile + i];
        if (o < 0) continue;
        n++;
        const double X = xyz[o], Y = xyz[nb + o], Z = xyz[2 * nb + o];
        const double ir = 1.0 / sqrt(X * X + Y * Y + Z * Z);
        sx += X * ir;
        sy += Y * ir;
        sz += Z * ir;
    }
    for (int off = 16; off > 0; off >>= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, off);
        sy += __shfl_xor_sync(0xffffffffu, sy, off);
        sz += __shfl_xor_sync(0xffffffffu, sz, off);
    }
    const double sn = sqrt(sx * sx + sy * sy + sz * sz);
    // a tile whose directions cancel gets psi > pi: never culled
    const bool ok = sn > 1e-9;
    const double cx = ok ? sx / sn : 0.0, cy = ok ? sy / sn : 0.0, cz = ok ? sz / sn : 1.0;
    double dmin = 1.0;
    for (int64_t i = lane; i < tile; i += 32) {
        const int o = perm[t * tile + i];
        if (o < 0) continue;
        const double X = xyz[o], Y = xyz[nb + o], Z = xyz[2 * nb + o];
        const double ir = 1.0 / sqrt(X * X + Y * Y + Z * Z);
        dmin = fmin(dmin, (X * cx + Y * cy + Z * cz) * ir);
    }
    for (int off = 16; off > 0; off >>= 1) dmin = fmin(dmin, __shfl_xor_sync(0xffffffffu, dmin, off));
    const bool some = __any_sync(0xffffffffu, n > 0);
    if (lane == 0) {
        const double psi = ok ? acos(fmax(-1.0, fmin(1.0, dmin))) + 1e-6 : 4.0;
        K2Cone c;
        c.c[0] = (float)cx;
        c.c[1] = (float)cy;
        c.c[2] = (float)cz;
        // a group of padding only: culled for every record (cone_culled's bound is +inf)
        c.psi = some ? (float)psi : 0.0f;
        c.cos_psi = some ? (float)cos(psi) : 0.0f;
        c.sin_psi = some ? (float)sin(psi) : -INFINITY;
        c.pad[0] = c.pad[1] = 0.0f;
        cones[t] = c;
    }
}

// is_fast_diff tiles of `tile` bins: blocks of (tile/16) theta x 16 phi bins, each
// warp's 32 bins a block of 4 theta x 8 phi within it, so that a warp spans a small
// solid angle; cached with the bin grid, a cone per warp.
int k2_fast_tiles(pbt_ctx *ctx, cudaStream_t st, int64_t tile) {
    GridCache &g = ctx->grid;
    if (g.fast_tile == tile) return PBT_OK;
    const int64_t nphi = (int64_t)g.phi.size(), ntheta = (int64_t)g.theta.size();
    const int64_t bp = 16, bt = tile / bp;
    const int64_t ntb = (ntheta + bt - 1) / bt, npb = (nphi + bp - 1) / bp;
    const int64_t ntiles = ntb * npb;
    std::vector<int> perm((size_t)(ntiles * tile), -1);
    for (int64_t a = 0; a < ntb; a++)
        for (int64_t b = 0; b < npb; b++)
            for (int64_t i = 0; i < tile; i++) {
                const int64_t w = (i % 128) / 32, l = i % 32;
                const int64_t j = a * bt + (i / 128) * 8 + (w >> 1) * 4 + (l >> 3);
                const int64_t q = b * bp + (w & 1) * 8 + (l & 7);
                if (j < ntheta && q < nphi) perm[(size_t)((a * npb + b) * tile + i)] = (int)(q + nphi * j);
            }
    const int64_t ncones = ntiles * tile / 32;
    PBT_TRY(g.fast_perm.ensure(perm.size() * sizeof(int)));
    PBT_TRY(g.fast_cone.ensure((size_t)ncones * sizeof(K2Cone)));
    PBT_CUDA_TRY(cudaMemcpyAsync(g.fast_perm.p, perm.data(), perm.size() * sizeof(int),
                                 cudaMemcpyHostToDevice, st));
    k2_cone_kernel<<<(unsigned)((ncones + 3) / 4), 128, 0, st>>>(
        g.fast_perm.as<int>(), ncones, 32, g.xyz.as<double>(), g.nb, g.fast_cone.as<K2Cone>());
    ctx->launches++;
    PBT_CUDA_TRY(cudaGetLastError());
    PBT_CUDA_TRY(cudaStreamSynchronize(st));  // perm (pageable) and cones ready before caching
    g.fast_tile = tile;
    g.fast_ntiles = ntiles;
    return PBT_OK;
}

// Records per work item of the default plan, in multiples of 32.  Fewer, larger items
// cost less per item; too few leave SMs short of work at the end of the launch.  About
// eight items per resident CTA (four per SM) up to 2,048 records, and from there twelve
// up to 8,192:
// * 24 lists of 3,300 on 64,980 bins, which 5,600 leaves whole: 20.84 ms against 21.09 at
//   2,048; 60,000 records on 259,560 bins with the field-of-view test 13.72 against 14.04
//   (without: 63.9 and 63.8); 7,000 records 7.58 at 2,048, 7.88 at 8,192.
// * Not below 160 records for one list, where the items' number decides how even the
//   launch ends (eleven lists of 600 to 5,000 on 8,000 to 65,000 bins: 1.5 % above each
//   one's best on average at 160, 5.1 % at 256, 4 % at 96), and 256 for several, whose
//   shorter lists split less (60 lists of 200: 0.42 ms, 0.46 at 160).
// * A call that does not give every resident CTA an item of that takes smaller ones, down
//   to 64 (528 outbeams on 6,552 bins, a pass: 147 us at 64, 164 at 128, 205 at 256, 157
//   at 32).
int64_t k2_auto_rpi(int64_t nrec, int64_t ntiles, int64_t norient, int nsm) {
    const int64_t per_slot = nrec * ntiles / ((int64_t)4 * std::max(nsm, 1));
    const int64_t least = norient > 1 ? 256 : 160;
    const int64_t r = std::max<int64_t>(std::min<int64_t>(2048, std::max(least, per_slot / 8)),
                                        std::min<int64_t>(8192, per_slot / 12));
    return std::min(r, std::max<int64_t>(64, per_slot)) / 32 * 32;
}

int k2_run_chunk(pbt_ctx *ctx, cudaStream_t st, const K2Setup &S, K2Flags *flags, int64_t o0, int64_t no,
                 int64_t nrefs, double lambda, int fast_diff, K2Plan plan, double *ws,
                 int64_t *seg_rec, int64_t *item_pre, unsigned long long *counter) {
    pbt::NvtxRange nvtx_("pbt: far-field sum (FP32)");
    const GridCache &g = ctx->grid;
    const int64_t tile = (int64_t)K2_THREADS * plan.bpt;
    int64_t ntiles = (g.nb + tile - 1) / tile;
    const bool cull = fast_diff && plan.variant == 1;
    if (cull) {
        PBT_TRY(k2_fast_tiles(ctx, st, tile));
        ntiles = g.fast_ntiles;
    }
    if (plan.auto_rpi) plan.rpi = k2_auto_rpi(nrefs, ntiles, S.src.norient, ctx->sm_count);
    // split tickets of every (segment, tile)
    const int64_t ntk = 2 * no * ntiles;
    PBT_TRY(ctx->d_tk.ensure((size_t)ntk * sizeof(unsigned)));
    const int64_t zb = std::min<int64_t>((ntk + 8 * K2_PLAN_THREADS - 1) / (8 * K2_PLAN_THREADS), 256);
    k2_plan_kernel<<<(unsigned)(1 + zb), K2_PLAN_THREADS, 0, st>>>(S.src, o0, no, plan.rpi, ntiles, seg_rec,
                                                                   item_pre, counter,
                                                                   ctx->d_tk.as<unsigned>());
    ctx->launches++;
    const double waveno = 2.0 * kPiRef / lambda;
    K2MainArgs A;
    A.recs = S.recs;
    A.fovs = S.fovs;
    A.fovx = S.fovx;
    A.rlo = S.rlo;
    A.seg_rec = seg_rec;
    A.item_pre = item_pre;
    A.nseg = 2 * no;
    A.rpi = plan.rpi;
    A.ntiles = ntiles;
    A.xyz = g.xyz.as<double>();
    A.nb = g.nb;
    A.nphi = (int64_t)g.phi.size();
    A.theta_i = g.theta_i;
    A.k = (float)waveno;
    A.hkR = (float)(0.5 * waveno * kFarR);
    A.sgh = -cos(g.theta[g.theta_i]) <= 0.0 ? 1.0f : -1.0f;  // sign rule of the bin set-up
    A.ws = ws;
    A.tickets = ctx->d_tk.as<unsigned>();
    A.counter = counter;
    A.err = &flags->err;
    if (plan.variant == 1) {
        K2PkArgs B;
        B.pairs = S.pairs;
        B.polys = S.polys;
        B.stride = (int)S.poly_stride;
        B.chunk = S.polys ? std::min(fast_diff ? K2P_CH_FOV : K2P_CH_FULL, (int)(poly_stage(fast_diff) / S.poly_stride)) : 0;
        B.rlo = S.rlo;
        B.fovs = S.fovs;
        B.fovx = S.fovx;
        B.perm = cull ? g.fast_perm.as<int>() : nullptr;
        B.cones = cull ? g.fast_cone.as<K2Cone>() : nullptr;
        B.seg_rec = seg_rec;
        B.item_pre = item_pre;
        B.nseg = A.nseg;
        B.rpi = plan.rpi;
        B.ntiles = ntiles;
        B.xyz = A.xyz;
        B.nb = A.nb;
        B.nphi = A.nphi;
        B.theta_i = A.theta_i;
        B.hkR = A.hkR;
        B.turns = (float)(0.5 * waveno * kFarR * kInvPi);
        B.epsmax = &flags->epsmax;
        B.ws = ws;
        B.tickets = A.tickets;
        B.counter = counter;
        B.err = &flags->err;
        if (S.polys)
            return fast_diff ? k2_launch_pk<1, true, true>(ctx, st, B) : k2_launch_pk<1, false, true>(ctx, st, B);
        if (plan.bpt == 1)
            return fast_diff ? k2_launch_pk<1, true, false>(ctx, st, B) : k2_launch_pk<1, false, false>(ctx, st, B);
        return fast_diff ? k2_launch_pk<2, true, false>(ctx, st, B) : k2_launch_pk<2, false, false>(ctx, st, B);
    }
    if (plan.bpt == 1)
        return fast_diff ? k2_launch_main<1, true>(ctx, st, A) : k2_launch_main<1, false>(ctx, st, A);
    return fast_diff ? k2_launch_main<2, true>(ctx, st, A) : k2_launch_main<2, false>(ctx, st, A);
}

}  // namespace

namespace {
// One CTA waits on an mbarrier that nothing arrives at: the bounded wait must
// give up after limit_ns and raise the timeout flag.
__global__ void k2_wait_selftest_kernel(uint64_t limit_ns, int *__restrict__ err) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const bool ok = mbar_wait(smem_u32(&bar), 0u, limit_ns);
    if (threadIdx.x == 0 && !ok) atomicOr(err, 4);
}
}  // namespace

int k2_wait_selftest(pbt_ctx *ctx, cudaStream_t st, uint64_t limit_ns) {
    PBT_TRY(ctx->d_misc.ensure(64));
    int *d_err = ctx->d_misc.as<int>();
    PBT_CUDA_TRY(cudaMemsetAsync(d_err, 0, sizeof(int), st));
    k2_wait_selftest_kernel<<<1, 32, 0, st>>>(limit_ns, d_err);
    ctx->launches = 1;
    PBT_CUDA_TRY(cudaGetLastError());
    return k2_check_err(ctx, st, d_err);
}

int k2_check_err(pbt_ctx *ctx, cudaStream_t st, const int *d_err) {
    (void)ctx;
    int h = 0;
    PBT_CUDA_TRY(cudaMemcpyAsync(&h, d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
    PBT_CUDA_TRY(cudaStreamSynchronize(st));
    if (h & 1) {
        set_error("an outbeam face index fi is out of range");
        return PBT_EINVAL;
    }
    if (h & 2) {
        set_error("the FP32 path supports faces of up to 16 vertices");
        return PBT_EINVAL;
    }
    if (h & 4) {
        set_error("a bounded device wait timed out in the far-field kernel");
        return PBT_ETIMEOUT;
    }
    return PBT_OK;
}

// Batched FP32 orientation average in three steps: begin (the orientation
// sums and per-orientation results for norient orientations), add (a run of
// orientations [o0, o0+no): record set-up, the far-field sum and the
// epilogue into the sums), finish (averages and phi integrals).
// h_beam_off / h_ext_off (relative to the run) and h_face_off are host arrays;
// every other array is device memory.
int k2_batch_begin(pbt_ctx *ctx, cudaStream_t st, int64_t norient, int64_t max_run,
                   const pbt_output_params *d_params_per, K2Batch &B) {
    const GridCache &g = ctx->grid;
    const int64_t nb = g.nb;
    B.norient = norient;
    B.plan = k2_plan_for(ctx);
    // orientation chunks of the FP64 workspace, capped at 16 GiB
    const size_t per_orient = (size_t)2 * 8 * nb * sizeof(double);
    const size_t cap = (size_t)16 << 30;
    B.wchunk = std::max<int64_t>(1, std::min<int64_t>(max_run, (int64_t)(cap / per_orient)));
    const int64_t chunk = B.wchunk;
    // A grid with too few bins for the SMs spreads the epilogue's orientations over
    // blockIdx.y, up to 32 ways, each with a Mueller sum of its own.
    const int64_t eblk = (nb + K2_EPI_THREADS - 1) / K2_EPI_THREADS;
    B.ny = (int)std::max<int64_t>(1, std::min<int64_t>({(8 * ctx->sm_count + eblk - 1) / eblk, chunk, 32}));
    // d_ws: workspace | mu_sum | partial sums of it | per-orient red (6) | bs | scale (2) |
    // per-orient params | seg/items | counter | flags | warps' partial sums
    const size_t o_ws = 0, o_mu = align_up(o_ws + chunk * per_orient), o_mp = align_up(o_mu + 16 * nb * 8),
                 o_red = align_up(o_mp + (B.ny > 1 ? (size_t)B.ny * 16 * nb * 8 : 0)),
                 o_bs = align_up(o_red + 6 * norient * 8),
                 o_sc = align_up(o_bs + norient * 8), o_pp = align_up(o_sc + 2 * norient * 8),
                 o_seg = align_up(o_pp + norient * sizeof(pbt_output_params)),
                 o_it = align_up(o_seg + (2 * chunk + 1) * 8), o_cnt = align_up(o_it + (2 * chunk + 1) * 8),
                 o_flags = align_up(o_cnt + 64),
                 o_part = align_up(o_flags + sizeof(K2Flags)),
                 o_end = align_up(o_part + (size_t)6 * chunk * eblk * (K2_EPI_THREADS / 32) * 8);
    PBT_TRY(ctx->d_ws.ensure(o_end));
    char *base = ctx->d_ws.as<char>();
    B.flags = base + o_flags;
    B.part = (double *)(base + o_part);
    B.mu_part = (double *)(base + o_mp);
    PBT_CUDA_TRY(cudaMemsetAsync(B.flags, 0, sizeof(K2Flags), st));
    B.ws = (double *)(base + o_ws);
    B.mu_sum = (double *)(base + o_mu);
    B.redo = (double *)(base + o_red);
    B.bs = (double *)(base + o_bs);
    B.scale = (double *)(base + o_sc);
    B.pp = d_params_per ? const_cast<pbt_output_params *>(d_params_per) : (pbt_output_params *)(base + o_pp);
    B.seg_rec = (int64_t *)(base + o_seg);
    B.item_pre = (int64_t *)(base + o_it);
    B.counter = (unsigned long long *)(base + o_cnt);
    B.first = true;
    return PBT_OK;
}

int k2_batch_add(pbt_ctx *ctx, cudaStream_t st, K2Batch &B, int64_t o0, int64_t no,
                 const pbt_outbeam *d_beam, const int64_t *h_beam_off, const pbt_outbeam *d_ext,
                 const int64_t *h_ext_off, const double *d_verts, int64_t nverts,
                 const int64_t *h_face_off, const int64_t *d_face_off, const int64_t *d_face_vi,
                 int64_t nfaces, double lambda, int fast_diff, int scaling,
                 const pbt_output_params *d_params_in) {
    const GridCache &g = ctx->grid;
    const int64_t nb = g.nb, nphi = (int64_t)g.phi.size(), ntheta = (int64_t)g.theta.size();
    K2Flags *flags = (K2Flags *)B.flags;
    K2Setup S;
    PBT_TRY(k2_prepare(ctx, st, no, d_beam, h_beam_off, d_ext, h_ext_off, d_verts, nverts, h_face_off,
                       d_face_off, d_face_vi, nfaces, lambda, fast_diff, B.plan, flags, S));
    const double waveno = 2.0 * kPiRef / lambda;
    const double *phitab = g.phitab.as<double>(), *cth = g.thtab.as<double>() + ntheta;
    const int64_t back_bin = 0 + nphi * g.back_i;
    const int eb = K2_EPI_THREADS;
    const unsigned egrid = (unsigned)((nb + eb - 1) / eb);
    const int64_t nw = (int64_t)egrid * (eb / 32);
    for (int64_t l0 = 0; l0 < no; l0 += B.wchunk) {
        const int64_t n = std::min(B.wchunk, no - l0);
        const int64_t nrefs =
            (h_beam_off[l0 + n] - h_beam_off[l0]) + (h_ext_off[l0 + n] - h_ext_off[l0]);
        PBT_TRY(k2_run_chunk(ctx, st, S, flags, l0, n, nrefs, lambda, fast_diff, B.plan, B.ws, B.seg_rec,
                             B.item_pre, B.counter));
        const int64_t og = o0 + l0;  // global orientation of the workspace's first slot
        pbt::NvtxRange nvtx_epi("pbt: epilogue (Mueller, orientation sums)");
        const int ny = (int)std::min<int64_t>(B.ny, n);
        const dim3 grid(egrid, (unsigned)ny);
        if (scaling) {
            k2_scatt_be_kernel<<<grid, eb, 0, st>>>(B.ws, B.seg_rec, n, nb, nphi, phitab, waveno,
                                                    g.wbin.as<double>(), B.part);
            k2_part_sum_kernel<<<(unsigned)(2 * n), 256, 0, st>>>(B.part, nw, B.scale + 2 * og);
            k2_scale_kernel<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(B.scale, d_params_in, og, n);
            ctx->launches += 3;
        }
        k2_epi_kernel<<<grid, eb, 0, st>>>(B.ws, B.seg_rec, n, og, nb, nphi, phitab, cth, waveno,
                                           g.wbin.as<double>(), back_bin, scaling ? B.scale : nullptr,
                                           ny > 1 ? B.mu_part : B.mu_sum, B.first ? 1 : 0, B.part, B.bs);
        k2_part_sum_kernel<<<(unsigned)(6 * n), 256, 0, st>>>(B.part, nw, B.redo + 6 * og);
        ctx->launches += 2;
        if (ny > 1) {
            k2_fold_kernel<<<(unsigned)((16 * nb + 255) / 256), 256, 0, st>>>(B.mu_part, ny, 16 * nb,
                                                                              B.first ? 1 : 0, B.mu_sum);
            ctx->launches++;
        }
        B.first = false;
        PBT_CUDA_TRY(cudaGetLastError());
    }
    return PBT_OK;
}

int k2_batch_finish(pbt_ctx *ctx, cudaStream_t st, K2Batch &B, const pbt_output_params *d_params_in,
                    double *d_mueller_avg, double *d_m1d_avg, pbt_output_params *d_params_avg,
                    int check_errors) {
    pbt::NvtxRange nvtx_("pbt: orientation average");
    const GridCache &g = ctx->grid;
    const int64_t nphi = (int64_t)g.phi.size(), ntheta = (int64_t)g.theta.size();
    k2_final_kernel<<<1, 608, 0, st>>>(B.redo, B.bs, d_params_in, B.norient, B.pp, d_params_avg);
    k2_avg_kernel<<<(unsigned)((16 * ntheta + 7) / 8), 256, 0, st>>>(
        B.mu_sum, g.wphi.as<double>(), nphi, ntheta, (double)B.norient, d_mueller_avg, d_m1d_avg);
    ctx->launches += 2;
    PBT_CUDA_TRY(cudaGetLastError());
    if (check_errors) PBT_TRY(k2_check_err(ctx, st, &((K2Flags *)B.flags)->err));
    return PBT_OK;
}

int k2_batch_impl(pbt_ctx *ctx, cudaStream_t st, int64_t norient, const pbt_outbeam *d_beam,
                  const int64_t *h_beam_off, const pbt_outbeam *d_ext, const int64_t *h_ext_off,
                  const double *d_verts, int64_t nverts, const int64_t *h_face_off,
                  const int64_t *d_face_off, const int64_t *d_face_vi, int64_t nfaces,
                  double lambda, int fast_diff, int scaling, const pbt_output_params *d_params_in,
                  double *d_mueller_avg, double *d_m1d_avg, pbt_output_params *d_params_avg,
                  pbt_output_params *d_params_per, int check_errors) {
    K2Batch B;
    PBT_TRY(k2_batch_begin(ctx, st, norient, norient, d_params_per, B));
    PBT_TRY(k2_batch_add(ctx, st, B, 0, norient, d_beam, h_beam_off, d_ext, h_ext_off, d_verts,
                         nverts, h_face_off, d_face_off, d_face_vi, nfaces, lambda, fast_diff,
                         scaling, d_params_in));
    return k2_batch_finish(ctx, st, B, d_params_in, d_mueller_avg, d_m1d_avg, d_params_avg,
                           check_errors);
}

// FP32 diff_main: one orientation, amplitude grids in the reference layout.
int k2_diff_main_impl(pbt_ctx *ctx, cudaStream_t st, const pbt_outbeam *d_beam, int64_t nbeam,
                      const pbt_outbeam *d_ext, int64_t next, const double *d_verts, int64_t nverts,
                      const int64_t *h_face_off, const int64_t *d_face_off,
                      const int64_t *d_face_vi, int64_t nfaces, double lambda, int fast_diff,
                      double *d_afb, double *d_afe) {
    const GridCache &g = ctx->grid;
    const int64_t nb = g.nb;
    const K2Plan plan = k2_plan_for(ctx);
    K2Setup S;
    const int64_t hbo[2] = {0, nbeam}, heo[2] = {0, next};
    const size_t o_ws = 0, o_seg = align_up(o_ws + (size_t)2 * 8 * nb * sizeof(double)),
                 o_it = align_up(o_seg + 3 * 8), o_cnt = align_up(o_it + 3 * 8),
                 o_flags = align_up(o_cnt + 64), o_end = align_up(o_flags + sizeof(K2Flags));
    PBT_TRY(ctx->d_ws.ensure(o_end));
    char *base = ctx->d_ws.as<char>();
    double *ws = (double *)(base + o_ws);
    int64_t *seg_rec = (int64_t *)(base + o_seg);
    K2Flags *flags = (K2Flags *)(base + o_flags);
    PBT_CUDA_TRY(cudaMemsetAsync(flags, 0, sizeof(K2Flags), st));
    PBT_TRY(k2_prepare(ctx, st, 1, d_beam, hbo, d_ext, heo, d_verts, nverts, h_face_off, d_face_off,
                       d_face_vi, nfaces, lambda, fast_diff, plan, flags, S));
    PBT_TRY(k2_run_chunk(ctx, st, S, flags, 0, 1, nbeam + next, lambda, fast_diff, plan, ws, seg_rec,
                         (int64_t *)(base + o_it), (unsigned long long *)(base + o_cnt)));
    const double waveno = 2.0 * kPiRef / lambda;
    k2_ampl_out_kernel<<<(unsigned)((nb + 127) / 128), 128, 0, st>>>(
        ws, seg_rec, nb, (int64_t)g.phi.size(), g.phitab.as<double>(), g.xyz.as<double>(), waveno, d_afb,
        d_afe);
    ctx->launches++;
    PBT_CUDA_TRY(cudaGetLastError());
    return k2_check_err(ctx, st, &flags->err);
}

}  // namespace pbt
