// compact.cu -- FP32 compact-slot stepper (throughput tier).
//
// A time step does what the reference does in three dense launches
// (src/gpu_kernels_3d.py:462-486 APT rebuild, :530-680 phase update, :833-838
// cooling).  A sweep writes the cells whose neighbourhood holds one phase and
// queues the rest on work lists; the list kernels then rebuild each queued
// cell's active-phase list from the stored lists of the cell and its 6 face
// neighbours, evaluate the anisotropic interface, torque and kinetic terms and
// the pair sums, clip, renormalise and write only the phases that stay positive.
// Small domains have one list kernel (octet_kernel: eight lanes per cell, or one thread
// where the lists are long), large ones one per kind of cell: pair_kernel, trio_kernel,
// general_kernel and, for what those leave, rest_kernel (isotropic_kernel alone without
// anisotropy).
//
// State layout in HBM (x fastest, so a warp of 32 threads along x reads
// 32 consecutive entries of each array and an interface -- normal to z --
// keeps a warp convergent):
//   head uint32[cells]     bits 0-6 number n of stored phases (phi > 0),
//                          bit 7 "single value stored explicitly",
//                          bits 8-23 id of the first (smallest) stored phase
//   idx  uint16[S][cells]  ids of stored phases 1..n-1 (ascending; slot 0 unused)
//   val  float [S][cells]  fractions of stored phases 0..n-1
// A cell holding one phase at exactly 1 -- about nine cells in ten in a
// directional-solidification run -- costs 4 bytes: its value is implicit.
// Temperature is T0[z] - (accumulated cooling) with the accumulator in
// float64 on the host; the per-cell sum-to-one uses a compensated float
// pair (TwoSum), which keeps GB300's slow float64 pipe out of the loop.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <string.h>

#include <mutex>
#include <unordered_map>
#include <utility>

#include "compact_state.cuh"
#include "mpf3d.h"
#include "mpf3d_internal.h"

namespace mpf3d {
namespace compact {

// the reference's pi approximation in the driving-force prefactor (:651)
constexpr float FORCE_PREF = (float)(8.0 / 3.1415926535);

struct Params {
    int nx, ny, nz, N;
    int64_t cells;
    uint32_t cells32;
    float e2_flat, b_flat;  // eps^2 and b for a liquid gradient below the floor
    float inv_dx2, inv_2dx, half_over_dx, inv_dx, dt;
    float eps0, eps0sq, w0, mu_a, delta_a, mu_da, pp, tan_a0, g2_floor, ksi, theta_c, cos_theta_lo, Sf;
    double Tmc;  // T_melt + accumulated cooling (float64)
    // Device step clock (null: Tmc above).  The sweep reads the step's index
    // s = clock->step[parity], writes clock->tmc[parity] = clock_T_melt +
    // s * clock_rate (rounded operation by operation, like the host's
    // float64 expression) for the work-list kernels and clock->step[parity ^
    // 1] = s + 1 for the next step, so a CUDA graph of steps keeps cooling
    // when it is replayed.
    mpf3d_step_clock *clock;
    double clock_T_melt, clock_rate;
    int parity;
    int use_aniso, use_torque;
    int sym_normals;  // every grain's n111 rows 4..7 are -(rows 3..0)
    // per-domain view (a batch of instances shares the state arrays)
    uint32_t base;    // index of the domain's first cell in the state arrays
    int n111_base;    // first n111 row of the domain's phases
    int t_uniform;    // temperature uniform in the domain ...
    float dT_uniform; // ... with T - T_melt = dT_uniform
};


// max |cos| between a gradient and the grain's 8 rotated {111} normals, with
// the signed cosine and the winning normal (best_cos_from_grad_3d :110-134,
// facet_cos_and_nxyz_from_grad :251-301)
struct Facet {
    bool valid;
    float cabs, cs, nx, ny, nz, q;
};

// a * b - c * d with one rounding error at most (Kahan's difference of
// products); the _rn intrinsics keep the compiler from contracting the
// error-free steps into other FMAs
__device__ __forceinline__ float diff_of_products(float a, float b, float c, float d) {
    const float w = __fmul_rn(c, d);
    const float e = fmaf(-c, d, w);
    const float f = fmaf(a, b, -w);
    return __fadd_rn(f, e);
}

// theta = acos(c) for the facet's best |cos| c = |g . n| / |g| against the
// float32 normal n, accurate where c is near 1.  There FP32 acos of a
// rounded c loses most of theta (an absolute error of 1e-7 in c is a
// relative error of 1e-7 / theta^2 in 1 - c), and b(theta) is steep.  The
// reference evaluates c in float64 from the same float32 normals, whose
// length differs from 1 by their rounding, so
//   1 - c = (1 - |n|) + |n| (1 - cos t),  t the angle between g and n,
// with 1 - |n|^2 from compensated squares (TwoProduct, TwoSum) and
//   1 - cos t = |g x n|^2 / (|g|^2 |n|^2 (1 + cos t))
// from accurate cross-product components; theta = 2 asin(sqrt((1 - c)/2)).
// |theta - acos(c)| stays within a few 1e-6 rad against float64 (c > 1,
// possible when |n| > 1, gives theta = 0 as the reference's clamp does).
__device__ __forceinline__ float facet_angle(float3 g, const Facet &f) {
    const float nx = f.nx, ny = f.ny, nz = f.nz;
    const float p1 = __fmul_rn(nx, nx), e1 = fmaf(nx, nx, -p1);
    const float p2 = __fmul_rn(ny, ny), e2 = fmaf(ny, ny, -p2);
    const float p3 = __fmul_rn(nz, nz), e3 = fmaf(nz, nz, -p3);
    const float s1 = __fadd_rn(p1, p2);
    const float t1 = __fsub_rn(s1, p1);
    float err = __fadd_rn(__fsub_rn(p1, __fsub_rn(s1, t1)), __fsub_rn(p2, t1));
    const float s2 = __fadd_rn(s1, p3);
    const float t2 = __fsub_rn(s2, s1);
    err = __fadd_rn(err, __fadd_rn(__fsub_rn(s1, __fsub_rn(s2, t2)), __fsub_rn(p3, t2)));
    const float dn2 = __fsub_rn(__fsub_rn(1.0f, s2), __fadd_rn(err, __fadd_rn(e1, __fadd_rn(e2, e3))));  // 1 - |n|^2
    const float cx = diff_of_products(g.y, nz, g.z, ny);
    const float cy = diff_of_products(g.z, nx, g.x, nz);
    const float cz = diff_of_products(g.x, ny, g.y, nx);
    const float sin2 = (cx * cx + cy * cy + cz * cz) / (f.q * (1.0f - dn2));
    const float omc = fmaxf(0.5f * dn2 + sin2 / (1.0f + f.cabs), 0.0f);  // 1 - c
    return 2.0f * asinf(sqrtf(0.5f * omc));
}

// b(theta) (calc_b_from_cos :33-55) for the facet of the liquid gradient g
// at the cell; below the gradient floor the best cos is 0 and b is 1
__device__ __forceinline__ float calc_b(const Params &P, float3 g, const Facet &f) {
    if (!f.valid || f.cabs <= P.cos_theta_lo) return 1.0f;  // theta >= theta_c: outside the cusp
    const float theta = facet_angle(g, f);
    if (theta >= P.theta_c) return 1.0f;
    const float hp = 1.57079632679489662f;
    float y = hp * (theta / P.theta_c);
    y = fminf(fmaxf(y, 1.0e-6f), hp - 1.0e-6f);
    float t = tanf(y);
    return P.ksi + (1.0f - P.ksi) * t * tanhf(1.0f / t);
}

// Work lists of a step (scratch memory owned by the caller): items holds
// x-fastest cell indices -- cells needing the general update from the front,
// solid-liquid interface cells from items[cells - 1] down; count[4] holds the two
// list lengths for even and odd steps (count[2*parity + 0/1]), so the sweep
// of one step can clear the other parity's counters without a memset.
struct Queue {
    uint32_t *__restrict__ items;
    uint32_t *__restrict__ count;
    // With split set, interface cells whose active list holds two or more
    // solids go to a third list at items[cells + ...] (counters count[4 +
    // parity]): the second list is then pair_kernel's.
    int split;
};

struct Mats {
    const double *__restrict__ T0z;
    const float *__restrict__ wij;
    const float *__restrict__ a2ij;
    const float *__restrict__ mij;
    const float *__restrict__ n111;
};

__device__ __forceinline__ uint32_t cidx(const Params &P, int l, int m, int k) {
    return P.base + ((uint32_t)k * (uint32_t)P.ny + (uint32_t)m) * (uint32_t)P.nx + (uint32_t)l;
}

// place of slot s of cell c in the idx and val arrays.  Slots beyond the second may lie
// past 2^32 entries in states that the step accepts (2^31 cells).
__device__ __forceinline__ size_t slot_at(uint32_t s, uint32_t cells, uint32_t c) { return (size_t)s * cells + c; }

// liquid fraction of cell q; the head and the first value are loaded
// together (the value is ignored where the head says it is not needed), so
// the liquid stencil costs one round of loads rather than two
__device__ __forceinline__ float liquid32(const In &in, uint32_t q) {
    const uint32_t h = __ldg(in.head + q);
    const float v = __ldg(in.val + q);
    // a head with liquid is 1..255, alone and implicit 1
    return h - 1u < 255u ? (h == 1u ? 1.0f : v) : 0.0f;
}

// 7-point Laplacian of one phase, rounded operation by operation
__device__ __forceinline__ float lap7(const Params &P, const float (&v)[7]) {
    float s = __fadd_rn(v[1], v[2]);
    s = __fadd_rn(s, v[3]);
    s = __fadd_rn(s, v[4]);
    s = __fadd_rn(s, v[5]);
    s = __fadd_rn(s, v[6]);
    return __fmul_rn(__fsub_rn(s, __fmul_rn(6.0f, v[0])), P.inv_dx2);
}

// a b c . x y z with the roundings fixed.  The solid-liquid terms are written
// with explicit roundings throughout, so that every kernel that inlines them, and
// all forms of the interface update, give the same bits.  The order is part of the
// results: the two faces of an axis are differenced first, then the axes added, with
// products fused into the sums.  Other orders change the last bits of lap_sl, and with
// them now and then which phases of a cell are clipped: with the six faces summed one
// after the other, one of 24 bicrystals differed by 2.5e-3 in a fraction after 20 steps.
__device__ __forceinline__ float dot3(float a, float b, float c, float x, float y, float z) {
    return fmaf(c, z, fmaf(a, x, __fmul_rn(b, y)));
}

// sqrtf as this file is compiled (-prec-sqrt=false) and the reciprocal of
// __fdividef, for normal numbers: without the scaling of subnormal ones
__device__ __forceinline__ float root(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float recip(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The liquid gradient (or the dominant solid's) at a stencil point.
struct Grad {
    float3 g;
    float q, ig;  // squared length; 1 / length, 0 below the floor
    bool valid;
    __device__ __forceinline__ Grad(const Params &P, float3 g_) : g(g_) {
        q = dot3(g.x, g.y, g.z, g.x, g.y, g.z);
        valid = !(q < P.g2_floor);
        ig = valid ? rsqrtf(q) : 0.0f;
    }
};

// What one grain's facet gives at a stencil point: the best normal (first
// maximum of |cos|; below the gradient floor cosine 0), a(theta)
// (calc_a_from_cos :24-30), eps^2 = (eps0 a)^2 and the factor of
// d a / d(grad phi) (da_dphixyz_A12 :304-341).  With 8 normals that are 4 exact
// antipodal pairs, one of each pair among the first four (checked on the
// host), |cos| ties exactly within a pair and 4 normals give the same search.
struct PointTerms {
    float cabs, cs, nx, ny, nz, a, e2, coef;
};
template <int NT>
__device__ __forceinline__ PointTerms point_terms(const Params &P, const Grad &G, const float (&un)[3 * NT]) {
    PointTerms t;
    t.cs = 0.0f; t.nx = 1.0f; t.ny = 0.0f; t.nz = 0.0f;
    const float x = G.g.x * G.ig, y = G.g.y * G.ig, z = G.g.z * G.ig;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        const float d = dot3(x, y, z, un[3 * i], un[3 * i + 1], un[3 * i + 2]);
        if (fabsf(d) > fabsf(t.cs)) {
            t.cs = d; t.nx = un[3 * i]; t.ny = un[3 * i + 1]; t.nz = un[3 * i + 2];
        }
    }
    t.cabs = fminf(fabsf(t.cs), 1.0f);
    t.cs = fminf(fmaxf(t.cs, -1.0f), 1.0f);
    const float C = root(fmaf(t.cs, t.cs, P.pp)), Sn = root(fmaxf(fmaf(-t.cs, t.cs, 1.0f), 0.0f) + P.pp);
    t.a = P.mu_a * fmaf(P.delta_a, fmaf(P.tan_a0, Sn, C), 1.0f);
    const float e = P.eps0 * t.a;
    t.e2 = G.valid ? e * e : P.e2_flat;
    t.coef = P.mu_da * fmaf(t.cs, recip(C), -__fmul_rn(P.tan_a0, __fmul_rn(t.cs, recip(Sn))));
    return t;
}
// d cos / d(grad phi); 0 below the floor
__device__ __forceinline__ float3 dcos(const Grad &G, const PointTerms &t) {
    const float ud = dot3(G.g.x, G.g.y, G.g.z, t.nx, t.ny, t.nz), ig3 = __fmul_rn(__fmul_rn(G.ig, G.ig), G.ig);
    return make_float3(fmaf(t.nx, G.ig, -__fmul_rn(__fmul_rn(ud, G.g.x), ig3)),
                       fmaf(t.ny, G.ig, -__fmul_rn(__fmul_rn(ud, G.g.y), ig3)),
                       fmaf(t.nz, G.ig, -__fmul_rn(__fmul_rn(ud, G.g.z), ig3)));
}

// The flux through the + face of an axis less that through its - face: wp, wm are
// eps^2 at the cell + at the neighbour, dp, dm phi_L there - at the cell.
__device__ __forceinline__ float face_difference(float wp, float dp, float wm, float dm) {
    return fmaf(wp, dp, __fmul_rn(wm, dm));
}

// lap_sl and b_sl of one solid at a cell from its facet there and, per axis, the
// difference of the two faces' fluxes (flux) and of the neighbours' da/d(grad phi)
// components along the axis, + side minus - side (div) (aniso_term1_solid_3d
// :149-204, torque_A11_3d :386-441 with A13_divergence_3d :344-383,
// calc_b_from_cos :33-55).  L: liquid at the 7 points; hxy, hxz, hyz: its mixed
// differences.
__device__ __forceinline__ float flux_sum(const Params &P, const float (&flux)[3]) {
    const float h = P.inv_2dx * P.inv_dx;
    return fmaf(flux[2], h, fmaf(flux[0], h, __fmul_rn(flux[1], h)));
}
__device__ __forceinline__ void center_terms(const Params &P, const Grad &G, const PointTerms &t, const float (&L)[7],
                                             float hxy, float hxz, float hyz, const float (&flux)[3],
                                             const float (&div)[3], float &lap_sl, float &b_sl) {
    lap_sl = flux_sum(P, flux);
    if (!G.valid) return;
    if (P.use_torque) {
        const float qq = 0.25f * P.inv_dx2;
        const float pxx = __fadd_rn(fmaf(-2.0f, L[0], L[1]), L[2]) * P.inv_dx2;
        const float pyy = __fadd_rn(fmaf(-2.0f, L[0], L[3]), L[4]) * P.inv_dx2;
        const float pzz = __fadd_rn(fmaf(-2.0f, L[0], L[5]), L[6]) * P.inv_dx2;
        const float pxy = hxy * qq, pxz = hxz * qq, pyz = hyz * qq;
        const float qx = 2.0f * dot3(G.g.x, G.g.y, G.g.z, pxx, pxy, pxz);
        const float qy = 2.0f * dot3(G.g.x, G.g.y, G.g.z, pxy, pyy, pyz);
        const float qz = 2.0f * dot3(G.g.x, G.g.y, G.g.z, pxz, pyz, pzz);
        const float3 dc = dcos(G, t);
        const float cxx = dot3(dc.x, dc.y, dc.z, pxx, pxy, pxz);
        const float cyy = dot3(dc.x, dc.y, dc.z, pxy, pyy, pyz);
        const float czz = dot3(dc.x, dc.y, dc.z, pxz, pyz, pzz);
        // per axis da/dx da/d(phi_x) q + a d(da/d(phi_x))/dx q + a da/d(phi_x) dq/dx
        auto axis = [&](float c, float d_cos, float d, float dq) {
            const float da = __fmul_rn(t.coef, d_cos), dd = __fmul_rn(d, P.half_over_dx);
            const float e = fmaf(__fmul_rn(t.a, dd), G.q, __fmul_rn(__fmul_rn(__fmul_rn(t.coef, c), da), G.q));
            return fmaf(__fmul_rn(t.a, da), dq, e);
        };
        const float Ex = axis(cxx, dc.x, div[0], qx), Ey = axis(cyy, dc.y, div[1], qy), Ez = axis(czz, dc.z, div[2], qz);
        lap_sl = fmaf(P.eps0sq, __fadd_rn(__fadd_rn(Ex, Ey), Ez), lap_sl);
    }
    Facet f;
    f.valid = true;
    f.cabs = t.cabs; f.cs = t.cs; f.nx = t.nx; f.ny = t.ny; f.nz = t.nz; f.q = G.q;
    b_sl = calc_b(P, G.g, f);
}

// Cell (l, m, k) and the steps to its neighbours in cell indices, modulo 2^32
// (x and y periodic, z clamped): one step each way, and two.
struct Offsets {
    uint32_t c, xp, xm, yp, ym, zp, zm, x2p, x2m, y2p, y2m, z2p, z2m;
    __device__ __forceinline__ Offsets(const Params &P, int l, int m, int k) {
        c = cidx(P, l, m, k);
        const uint32_t nx = (uint32_t)P.nx, plane = nx * (uint32_t)P.ny;
        const int lp = wrap_p(l, P.nx), lm = wrap_m(l, P.nx), mp = wrap_p(m, P.ny), mm = wrap_m(m, P.ny);
        xp = (uint32_t)(lp - l), xm = (uint32_t)(lm - l);
        x2p = (uint32_t)(wrap_p(lp, P.nx) - l), x2m = (uint32_t)(wrap_m(lm, P.nx) - l);
        yp = (uint32_t)(mp - m) * nx, ym = (uint32_t)(mm - m) * nx;
        y2p = (uint32_t)(wrap_p(mp, P.ny) - m) * nx, y2m = (uint32_t)(wrap_m(mm, P.ny) - m) * nx;
        zp = k < P.nz - 1 ? plane : 0u, zm = k > 0 ? 0u - plane : 0u;
        z2p = k < P.nz - 2 ? 2u * plane : zp, z2m = k > 1 ? 0u - 2u * plane : zm;
    }
};

// Liquid gradients at the 7 points and mixed second differences at the cell,
// from the liquid vL there and at the 18 further points of the 25-point stencil
// (offsets with |dx|+|dy|+|dz| <= 2).
struct Stencil {
    float3 G[7];
    float hxy, hxz, hyz;
    __device__ __forceinline__ Stencil(const In &in, const Params &P, const Offsets &o, const float (&vL)[7]) {
        const float Lxpyp = liquid32(in, o.c + o.xp + o.yp), Lxpym = liquid32(in, o.c + o.xp + o.ym);
        const float Lxmyp = liquid32(in, o.c + o.xm + o.yp), Lxmym = liquid32(in, o.c + o.xm + o.ym);
        const float Lxpzp = liquid32(in, o.c + o.xp + o.zp), Lxpzm = liquid32(in, o.c + o.xp + o.zm);
        const float Lxmzp = liquid32(in, o.c + o.xm + o.zp), Lxmzm = liquid32(in, o.c + o.xm + o.zm);
        const float Lypzp = liquid32(in, o.c + o.yp + o.zp), Lypzm = liquid32(in, o.c + o.yp + o.zm);
        const float Lymzp = liquid32(in, o.c + o.ym + o.zp), Lymzm = liquid32(in, o.c + o.ym + o.zm);
        const float Lx2p = liquid32(in, o.c + o.x2p), Lx2m = liquid32(in, o.c + o.x2m);
        const float Ly2p = liquid32(in, o.c + o.y2p), Ly2m = liquid32(in, o.c + o.y2m);
        const float Lz2p = liquid32(in, o.c + o.z2p), Lz2m = liquid32(in, o.c + o.z2m);
        const bool top = o.zp == 0, bottom = o.zm == 0;
        const float g2 = P.inv_2dx;
        G[0] = make_float3((vL[1] - vL[2]) * g2, (vL[3] - vL[4]) * g2, (vL[5] - vL[6]) * g2);
        G[1] = make_float3((Lx2p - vL[0]) * g2, (Lxpyp - Lxpym) * g2, (Lxpzp - Lxpzm) * g2);
        G[2] = make_float3((vL[0] - Lx2m) * g2, (Lxmyp - Lxmym) * g2, (Lxmzp - Lxmzm) * g2);
        G[3] = make_float3((Lxpyp - Lxmyp) * g2, (Ly2p - vL[0]) * g2, (Lypzp - Lypzm) * g2);
        G[4] = make_float3((Lxpym - Lxmym) * g2, (vL[0] - Ly2m) * g2, (Lymzp - Lymzm) * g2);
        // z neighbours sit on the clamped rows: at the top/bottom row the
        // neighbour is the cell itself
        G[5] = (top) ? G[0] : make_float3((Lxpzp - Lxmzp) * g2, (Lypzp - Lymzp) * g2, (Lz2p - vL[0]) * g2);
        G[6] = (bottom) ? G[0] : make_float3((Lxpzm - Lxmzm) * g2, (Lypzm - Lymzm) * g2, (vL[0] - Lz2m) * g2);
        if (top) G[5].z = (vL[5] - vL[6]) * g2;
        if (bottom) G[6].z = (vL[5] - vL[6]) * g2;
        hxy = Lxpyp - Lxpym - Lxmyp + Lxmym;
        hxz = Lxpzp - Lxpzm - Lxmzp + Lxmzm;
        hyz = Lypzp - Lypzm - Lymzp + Lymzm;
    }
};

// lap_sl and b_sl of one solid with the liquid gradient at the 7 points in
// one thread.
template <int NT>
__device__ __forceinline__ void interface_terms(const Params &P, const Stencil &st, const float (&L)[7],
                                                const float (&un)[3 * NT], float &lap_sl, float &b_sl) {
    const float3 (&G)[7] = st.G;
    const Grad g0(P, G[0]);
    bool any = g0.valid;
#pragma unroll
    for (int p = 1; p < 7; ++p)
        any = any || !(dot3(G[p].x, G[p].y, G[p].z, G[p].x, G[p].y, G[p].z) < P.g2_floor);
    float flux[3], div[3];
    if (!any) {  // flat liquid everywhere: eps^2 = (eps0 a(0))^2 at all 7 points, no torque
        const float w = P.e2_flat + P.e2_flat;
#pragma unroll
        for (int x = 0; x < 3; ++x) flux[x] = face_difference(w, L[1 + 2 * x] - L[0], w, L[2 + 2 * x] - L[0]);
        lap_sl = flux_sum(P, flux);
        b_sl = P.b_flat;
        return;
    }
    const PointTerms t0 = point_terms<NT>(P, g0, un);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        float w[2], da[2];
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const Grad g(P, G[1 + 2 * x + side]);
            const PointTerms t = point_terms<NT>(P, g, un);
            const float3 dc = dcos(g, t);
            w[side] = t0.e2 + t.e2;
            da[side] = g.valid ? __fmul_rn(t.coef, x == 0 ? dc.x : (x == 1 ? dc.y : dc.z)) : 0.0f;
        }
        flux[x] = face_difference(w[0], L[1 + 2 * x] - L[0], w[1], L[2 + 2 * x] - L[0]);
        div[x] = __fsub_rn(da[0], da[1]);
    }
    b_sl = 1.0f;
    center_terms(P, g0, t0, L, st.hxy, st.hxz, st.hyz, flux, div, lap_sl, b_sl);
}

// Four forms of the update of a queued cell give the same bits:
//   pair_cell   one thread, a neighbourhood of the liquid and one solid
//   trio_cell   one thread, a neighbourhood of up to three phases
//   octet_cell  eight lanes, any neighbourhood
//   any_cell    one thread, any neighbourhood, its phases in local memory
// The first two take most cells of a large domain: no per-phase arrays in local
// memory, and the records in one or two rounds of loads.  What they leave, and
// everything on small domains, where a step is one cell's latency, goes to the
// third, or to the fourth where that is many cells.  A 256^3 step with 64 grains (0.57
// M general cells, 0.30 M pairs, 73 k others, 13 k of them beyond three phases), each
// kernel by itself with cold caches: pairs 24 us, general 24, trios 23, rest 25; by
// any_cell alone the two list kernels took 150 us, by octets alone the lists take 292.

// Update of an interface cell whose neighbourhood holds the liquid and one
// solid, as the sweep's list 1 does where it split the lists: no merge, and only
// the pair's terms.
template <int NT>
__device__ __forceinline__ void pair_cell(const In &in, const Out &out, const Mats &M, const Params &P, int l, int m,
                                          int k) {
    const uint32_t cells = P.cells32;
    const Offsets at(P, l, m, k);
    const uint32_t pt[7] = {at.c, at.c + at.xp, at.c + at.xm, at.c + at.yp, at.c + at.ym, at.c + at.zp, at.c + at.zm};
    uint32_t h[7];
    float v0[7], v1[7];
    int i1[7];
#pragma unroll
    for (int p = 0; p < 7; ++p) {
        h[p] = __ldg(in.head + pt[p]);
        v0[p] = __ldg(in.val + pt[p]);
        i1[p] = (int)__ldg(in.idx + cells + pt[p]);
        v1[p] = __ldg(in.val + cells + pt[p]);
    }
    // heads: none 0; liquid 1 or explicit 0x81; liquid and solid 2; solid id << 8
    // | 1 or explicit
    float vL[7], vS[7];
    int sid = 0;
#pragma unroll
    for (int p = 0; p < 7; ++p) {
        const float v = (h[p] & 0xffu) == 1u ? 1.0f : v0[p];
        vL[p] = h[p] - 1u < 255u ? v : 0.0f;
        vS[p] = h[p] == 2u ? v1[p] : (h[p] > 255u ? v : 0.0f);
        sid = max(sid, h[p] == 2u ? i1[p] : hid0(h[p]));
    }
    const Stencil st(in, P, at, vL);
    const float *ug = M.n111 + (size_t)(P.n111_base + sid) * 24;
    float un[3 * NT], lap_sl, b_sl;
#pragma unroll
    for (int q = 0; q < 3 * NT; ++q) un[q] = __ldg(ug + q);
    interface_terms<NT>(P, st, vL, un, lap_sl, b_sl);
    const float3 gs = make_float3((vS[1] - vS[2]) * P.inv_2dx, (vS[3] - vS[4]) * P.inv_2dx, (vS[5] - vS[6]) * P.inv_2dx);
    const float al = point_terms<NT>(P, Grad(P, gs), un).a;
    const float w_sl = P.w0 * (al * al);

    // the pair (solid, liquid) of trio_cell's sums; (liquid, solid) negates it
    const int N = P.N;
    const float WL = fmaf(__ldg(M.wij + sid), vS[0], __fmul_rn(__ldg(M.wij), vL[0]));
    const float WS = fmaf(__ldg(M.wij + sid * N + sid), vS[0], __fmul_rn(w_sl, vL[0]));
    const double Tmc = P.clock ? P.clock->tmc[P.parity] : P.Tmc;
    const float dT = P.t_uniform ? P.dT_uniform : (float)(M.T0z[k] - Tmc);
    const float ppp = __fadd_rn(__fsub_rn(WS, WL), 0.5f * lap_sl);
    const float tf = __fmul_rn(__fmul_rn(FORCE_PREF, sqrtf(fmaxf(__fmul_rn(vS[0], vL[0]), 0.0f))), -P.Sf * dT);
    const float drive = __fsub_rn(ppp, tf);
    const float mS = __ldg(M.mij + sid * N) * b_sl, mL = __ldg(M.mij + sid) * b_sl;
    const float dS = -__fmul_rn(__fmul_rn(__fmul_rn(2.0f, mS), 0.5f), drive);
    const float dL = __fmul_rn(__fmul_rn(__fmul_rn(2.0f, mL), 0.5f), drive);
    const float oL = fminf(fmaxf(fmaf(P.dt, dL, vL[0]), 0.0f), 1.0f);
    const float oS = fminf(fmaxf(fmaf(P.dt, dS, vS[0]), 0.0f), 1.0f);
    // compensated sum of the two, as the loop over phases forms it
    const float s2 = oL + oS, bb = s2 - oL;
    const float low = (oL - (s2 - bb)) + (oS - bb);
    const bool normal = s2 + low > 1e-20f;
    float inv = 1.0f / s2;
    inv = fmaf(-__fmul_rn(inv, inv), low, inv);
    const float rL = normal ? oL * inv : 1.0f, rS = normal ? oS * inv : oS;
    const uint32_t c = pt[0];
    const bool keepL = rL > 0.0f, keepS = rS > 0.0f;
    out.val[c] = keepL ? rL : rS;
    if (keepL && keepS) {
        out.idx[cells + c] = (uint16_t)sid;
        out.val[cells + c] = rS;
    }
    out.head[c] = mkhead(keepL || !keepS ? LIQ : sid, (keepL ? 1 : 0) + (keepS ? 1 : 0), false);
}

// Update of a cell whose neighbourhood holds up to three phases, in registers:
// HEAVY the multi-solid interface cells (list 2), otherwise list 0 (grain
// boundaries, and everything of the isotropic model).  Returns false, with
// nothing written, where the neighbourhood holds more.
template <int S, bool HEAVY, int NT>
__device__ __forceinline__ bool trio_cell(const In &in, const Out &out, const Mats &M, const Params &P, int l, int m,
                                          int k) {
    constexpr int NONE = 0x7fffffff;
    const uint32_t cells = P.cells32;
    const int lp = wrap_p(l, P.nx), lm = wrap_m(l, P.nx), mp = wrap_p(m, P.ny), mm = wrap_m(m, P.ny);
    const int kp = clamp_p(k, P.nz), km = clamp_m(k, P.nz);
    const uint32_t pt[7] = {cidx(P, l, m, k), cidx(P, lp, m, k), cidx(P, lm, m, k), cidx(P, l, mp, k),
                            cidx(P, l, mm, k), cidx(P, l, m, kp), cidx(P, l, m, km)};
    // each point's list, and its merge by shifting the lists
    int ia[7], ib[7], ic[7];
    float va[7], vb[7], vd[7];
    bool fits = true;
#pragma unroll
    for (int p = 0; p < 7; ++p) {
        const uint32_t h = __ldg(in.head + pt[p]);
        const float v = __ldg(in.val + pt[p]);
        const int i1 = (int)__ldg(in.idx + cells + pt[p]);
        vb[p] = __ldg(in.val + cells + pt[p]);
        const int n = min(hcount(h), S);
        ia[p] = n > 0 ? hid0(h) : NONE;
        va[p] = hcount(h) >= 2 || hexplicit(h) ? v : 1.0f;
        ib[p] = n > 1 ? i1 : NONE;
        ic[p] = NONE;
        vd[p] = 0.0f;
        if (n > 2) {
            ic[p] = (int)__ldg(in.idx + slot_at(2, cells, pt[p]));
            vd[p] = __ldg(in.val + slot_at(2, cells, pt[p]));
        }
        fits = fits && n <= 3;
    }
    int ids[3];
    float V[3][7];
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        int id = ia[0];
#pragma unroll
        for (int p = 1; p < 7; ++p) id = min(id, ia[p]);
        ids[t] = id;
#pragma unroll
        for (int p = 0; p < 7; ++p) {
            const bool hit = ia[p] == id && id != NONE;
            V[t][p] = hit ? va[p] : 0.0f;
            ia[p] = hit ? ib[p] : ia[p];
            va[p] = hit ? vb[p] : va[p];
            ib[p] = hit ? ic[p] : ib[p];
            vb[p] = hit ? vd[p] : vb[p];
            ic[p] = hit ? NONE : ic[p];
        }
    }
#pragma unroll
    for (int p = 0; p < 7; ++p) fits = fits && ia[p] == NONE;
    if (!fits || ids[0] == NONE) return false;
    const int n = ids[1] == NONE ? 1 : (ids[2] == NONE ? 2 : 3);
    float lap[3], lap_sl[3] = {0.0f, 0.0f, 0.0f}, b_sl[3] = {1.0f, 1.0f, 1.0f};
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        lap[t] = lap7(P, V[t]);
        if (t >= n) ids[t] = LIQ;  // a valid index; never used
    }
    float w_sl = P.w0;
    if (ids[0] == LIQ && n > 1) {
        if (HEAVY) {
            const Stencil st(in, P, Offsets(P, l, m, k), V[0]);
            // dominant solid
            const bool last = n == 3 && V[2][0] > V[1][0];
            const float3 gs = last ? make_float3((V[2][1] - V[2][2]) * P.inv_2dx, (V[2][3] - V[2][4]) * P.inv_2dx,
                                                 (V[2][5] - V[2][6]) * P.inv_2dx)
                                   : make_float3((V[1][1] - V[1][2]) * P.inv_2dx, (V[1][3] - V[1][4]) * P.inv_2dx,
                                                 (V[1][5] - V[1][6]) * P.inv_2dx);
#pragma unroll 1
            for (int t = 1; t < n; ++t) {
                const float *ug = M.n111 + (size_t)(P.n111_base + (t == 1 ? ids[1] : ids[2])) * 24;
                float un[3 * NT], lv, b;
#pragma unroll
                for (int q = 0; q < 3 * NT; ++q) un[q] = __ldg(ug + q);
                interface_terms<NT>(P, st, V[0], un, lv, b);
                if (t == 1) { lap_sl[1] = lv; b_sl[1] = b; }
                else { lap_sl[2] = lv; b_sl[2] = b; }
                if ((t == 2) == last) {
                    const float al = point_terms<NT>(P, Grad(P, gs), un).a;
                    w_sl = P.w0 * (al * al);
                }
            }
        } else {
            // isotropic branch of the switchable kernel (:729-731)
            lap_sl[1] = lap_sl[2] = P.eps0sq * lap[0];
        }
    }

    // Pair sums (:600-661) in O(n^2): for a pair (i, j) the t3 sum of the
    // reference splits into W_i - W_j (potential) plus either the
    // solid-liquid term of lap_sl or (A_i - A_j)/2 (gradient energy).
    const int N = P.N;
    float W[3], Ag[3], o[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        W[i] = Ag[i] = o[i] = 0.0f;
        if (i >= n) continue;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            if (q >= n) continue;
            const float w = (ids[q] == LIQ && ids[i] != LIQ) ? w_sl : __ldg(M.wij + ids[i] * N + ids[q]);
            W[i] = fmaf(w, V[q][0], W[i]);
            Ag[i] = fmaf(__ldg(M.a2ij + ids[i] * N + ids[q]), lap[q], Ag[i]);
        }
    }
    const double Tmc = P.clock ? P.clock->tmc[P.parity] : P.Tmc;
    const float dT = P.t_uniform ? P.dT_uniform : (float)(M.T0z[k] - Tmc);
    const float inv_n = 1.0f / (float)n;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if (i >= n) continue;
        float dpi = 0.0f;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            if (j == i || j >= n) continue;
            const bool sl = ids[i] != LIQ && ids[j] == LIQ, ls = ids[i] == LIQ && ids[j] != LIQ;
            const float T = sl ? 0.5f * lap_sl[i] : (ls ? -0.5f * lap_sl[j] : 0.5f * __fsub_rn(Ag[i], Ag[j]));
            const float ppp = __fadd_rn(__fsub_rn(W[i], W[j]), T);
            const float df = sl ? -P.Sf * dT : (ls ? P.Sf * dT : 0.0f);
            const float tf = __fmul_rn(__fmul_rn(FORCE_PREF, sqrtf(fmaxf(__fmul_rn(V[i][0], V[j][0]), 0.0f))), df);
            float me = __ldg(M.mij + ids[i] * N + ids[j]);
            if (HEAVY) {
                if (sl) me *= b_sl[i];
                else if (ls) me *= b_sl[j];
            }
            dpi = __fsub_rn(dpi, __fmul_rn(__fmul_rn(__fmul_rn(2.0f, me), inv_n), __fsub_rn(ppp, tf)));
        }
        o[i] = fminf(fmaxf(fmaf(P.dt, dpi, V[i][0]), 0.0f), 1.0f);
    }
    // renormalise with a compensated (TwoSum) float accumulation (:663-680)
    float sum = 0.0f, low = 0.0f;
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        if (t >= n) continue;
        const float s2 = sum + o[t], bb = s2 - sum;
        low += (sum - (s2 - bb)) + (o[t] - bb);
        sum = s2;
    }
    const bool normal = sum + low > 1e-20f;
    float inv = 1.0f / sum;
    inv = fmaf(-__fmul_rn(inv, inv), low, inv);
    // stored list: the phases that stay positive, ascending; all clipped to
    // ~0: the liquid takes the cell (:679-680)
    const uint32_t c = pt[0];
    int stored = normal ? 0 : 1, first = LIQ;
    if (!normal) out.val[c] = 1.0f;
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        const float v = normal ? o[t] * inv : o[t];
        if (t >= n || !(v > 0.0f) || (!normal && ids[t] == LIQ)) continue;
        if (stored == 0) first = ids[t];
        else out.idx[slot_at(stored, cells, c)] = (uint16_t)ids[t];
        out.val[slot_at(stored, cells, c)] = v;
        ++stored;
    }
    // one stored phase: its renormalised value is 1 and is left implicit
    out.head[c] = mkhead(first, stored, false);
    return true;
}

// ---------------------------------------------------------------------------
// Any queued cell, eight lanes per cell.
//
// Lanes 0..6 of an octet stand for the cell and its x+, x-, y+, y-, z+, z-
// neighbours.  Each loads its own point's records, takes part in the merge of
// the 7 ascending lists (an octet-wide minimum per phase), loads the three
// liquid values its gradient needs beyond those the octet holds, and evaluates
// the facet of every solid at its own point; lane 7 evaluates the dominant
// solid's facet for w_sl.  After the merge lane t (and t - 8, ...) holds phase t
// for the pair sums, the renormalisation and the stores.
//
// The isotropic model (P.use_aniso 0) and cells without liquid or solid skip
// the facets.
// a lane's place in its octet: offsets of its point (d), of the next axis (a)
struct OctetLane {
    int p, axis;
    bool plus;       // on the + side
    int dl, dm, dk;  // the point's offset from the cell
    int al, am, ak;  // unit offset along the axis after the point's own
    __device__ __forceinline__ OctetLane() {
        p = threadIdx.x & 7;
        const bool arm = p >= 1 && p <= 6;
        axis = arm ? (p - 1) >> 1 : 3;
        plus = (p & 1) != 0;
        const int s = plus ? 1 : -1;
        dl = axis == 0 ? s : 0; dm = axis == 1 ? s : 0; dk = axis == 2 ? s : 0;
        al = axis == 2 ? 1 : 0; am = axis == 0 ? 1 : 0; ak = axis == 1 ? 1 : 0;
    }
};

// v of lane src of the octet
template <typename T>
__device__ __forceinline__ T from_lane(T v, int src) {
    return __shfl_sync(0xffffffffu, v, src, 8);
}
// phase t of the octet (t the same for the whole warp)
template <int NH, typename T>
__device__ __forceinline__ T phase_of(const T (&a)[NH], int t) {
    T x = a[0];
#pragma unroll
    for (int h = 1; h < NH; ++h)
        if ((t >> 3) == h) x = a[h];
    return from_lane(x, t & 7);
}

template <int S, int AMAX, int NT, bool LAST>
__device__ __forceinline__ bool octet_phases(const In &in, const Out &out, const Mats &M, const Params &P,
                                           int32_t *__restrict__ err, const OctetLane &O, bool active, int l, int m,
                                           int k) {
    constexpr unsigned ALL = 0xffffffffu;
    constexpr int NH = AMAX / 8;  // phases per lane
    constexpr int NONE = 0x7fffffff;
    const uint32_t cells = P.cells32;
    const int p = O.p, oct = (threadIdx.x & 31) >> 3;
    auto wrap = [](int a, int n) { return a < 0 ? n - 1 : (a >= n ? 0 : a); };
    auto clamp = [&](int a) { return min(max(a, 0), P.nz - 1); };
    const uint32_t c = cidx(P, l, m, k);
    const int lo = wrap(l + O.dl, P.nx), mo = wrap(m + O.dm, P.ny), ko = clamp(k + O.dk);
    const uint32_t pt = cidx(P, lo, mo, ko);

    // ---- merge of the 7 lists
    const uint32_t hw = __ldg(in.head + pt);
    float cur = __ldg(in.val + pt);
    // liquid beyond the octet's points: the next point along the lane's axis
    // and the two beside its own point along the next axis
    const float L2 = liquid32(in, cidx(P, wrap(lo + O.dl, P.nx), wrap(mo + O.dm, P.ny), clamp(ko + O.dk)));
    const float LA = liquid32(in, cidx(P, wrap(lo + O.al, P.nx), wrap(mo + O.am, P.ny), clamp(ko + O.ak)));
    const float LB = liquid32(in, cidx(P, wrap(lo - O.al, P.nx), wrap(mo - O.am, P.ny), clamp(ko - O.ak)));
    if (!(hcount(hw) >= 2 || hexplicit(hw))) cur = 1.0f;
    const int cnt = p < 7 ? min(hcount(hw), S) : 0;
    int next = cnt > 0 ? hid0(hw) : NONE, pos = 0, nid = NONE;
    float nval = 0.0f;
    if (cnt >= 2) {
        nid = (int)__ldg(in.idx + cells + pt);
        nval = __ldg(in.val + cells + pt);
    }
    int ids[NH];
    float vc[NH], lap[NH];
#pragma unroll
    for (int h = 0; h < NH; ++h) {
        ids[h] = 0;
        vc[h] = lap[h] = 0.0f;
    }
    int n = 0, ts = -1, first = NONE;
    bool ovf = false;
    float vL = 0.0f, maxv = -1.0f;
    float3 g = make_float3(0.f, 0.f, 0.f);  // gradient of the dominant solid, later of the lane's point
    while (true) {
        int id = min(next, __shfl_xor_sync(ALL, next, 1));
        id = min(id, __shfl_xor_sync(ALL, id, 2));
        id = min(id, __shfl_xor_sync(ALL, id, 4));
        const bool live = id != NONE;
        if (!__any_sync(ALL, live)) break;
        float own = 0.0f;
        if (live && next == id) {
            own = cur;
            cur = nval;
            next = nid;
            ++pos;
            nid = NONE;
            if (pos + 1 < cnt) {
                nid = (int)__ldg(in.idx + slot_at(pos + 1, cells, pt));
                nval = __ldg(in.val + slot_at(pos + 1, cells, pt));
            }
        }
        const float v[7] = {from_lane(own, 0), from_lane(own, 1), from_lane(own, 2), from_lane(own, 3), from_lane(own, 4), from_lane(own, 5), from_lane(own, 6)};
        if (live && n == AMAX) {
            ovf = true;
            next = NONE;
        } else if (live) {
            if (n == 0) first = id;
#pragma unroll
            for (int h = 0; h < NH; ++h)
                if (n == 8 * h + p) {
                    ids[h] = id;
                    vc[h] = v[0];
                    lap[h] = lap7(P, v);
                }
            if (id == LIQ) {
                vL = own;
            } else if (v[0] > maxv) {
                maxv = v[0];
                ts = n;
                g = make_float3((v[1] - v[2]) * P.inv_2dx, (v[3] - v[4]) * P.inv_2dx, (v[5] - v[6]) * P.inv_2dx);
            }
            ++n;
        }
    }
    if (!LAST && __any_sync(ALL, ovf)) return false;
    const int n_most = __reduce_max_sync(ALL, n);

    // ---- solid-liquid terms
    float lap_sl[NH], b_sl[NH];
#pragma unroll
    for (int h = 0; h < NH; ++h) {
        lap_sl[h] = 0.0f;
        b_sl[h] = 1.0f;
    }
    const bool heavy = n > 1 && first == LIQ;  // solids beside liquid
    float w_sl = P.w0;
    if (!P.use_aniso) {
        // isotropic branch of the switchable kernel (:729-731)
        const float lap_liq = from_lane(lap[0], 0);
#pragma unroll
        for (int h = 0; h < NH; ++h)
            if (heavy) lap_sl[h] = P.eps0sq * lap_liq;
    } else if (__any_sync(ALL, heavy)) {
        const float L[7] = {from_lane(vL, 0), from_lane(vL, 1), from_lane(vL, 2), from_lane(vL, 3), from_lane(vL, 4), from_lane(vL, 5), from_lane(vL, 6)};
        // the point's gradient: along its own axis, the next one, the third
        float along = O.plus ? L2 - L[0] : L[0] - L2;
        // a z neighbour beyond the domain is the cell itself
        if (O.axis == 2 && ko == k) along = L[5] - L[6];
        const float beside = LA - LB;
        const int q0 = O.axis == 0 ? 5 : (O.axis == 1 ? 1 : 3);
        const float Ap = from_lane(LA, q0), Am = from_lane(LA, q0 + 1), Bp = from_lane(LB, q0), Bm = from_lane(LB, q0 + 1);
        const float across = O.plus ? Ap - Am : Bp - Bm;
        const float hxy = from_lane(beside, 1) - from_lane(LA, 2) + from_lane(LB, 2);
        const float hxz = from_lane(across, 1) - from_lane(LB, 5) + from_lane(LB, 6);
        const float hyz = from_lane(beside, 3) - from_lane(LA, 4) + from_lane(LB, 4);
        const float3 g0 = make_float3((L[1] - L[2]) * P.inv_2dx, (L[3] - L[4]) * P.inv_2dx, (L[5] - L[6]) * P.inv_2dx);
        if (O.axis < 3) {
            const float u = along * P.inv_2dx, v = beside * P.inv_2dx, w = across * P.inv_2dx;
            g = O.axis == 0 ? make_float3(u, v, w) : (O.axis == 1 ? make_float3(w, u, v) : make_float3(v, w, u));
        } else if (p == 0) {
            g = g0;
        }
        const Grad G(P, g);
        const bool any = (__ballot_sync(ALL, G.valid && p < 7) >> (8 * oct) & 0x7fu) != 0u;
        const float dL = vL - L[0];
        float al = 0.0f;
#pragma unroll 1
        for (int t = 1; t < n_most; ++t) {
            const bool solid = heavy && t < n;
            const int id = phase_of(ids, t);
            const float *u = M.n111 + (size_t)(P.n111_base + (solid ? id : 0)) * 24;
            float un[3 * NT];
#pragma unroll
            for (int i = 0; i < 3 * NT; ++i) un[i] = __ldg(u + i);
            const PointTerms T = point_terms<NT>(P, G, un);
            if (t == ts) al = T.a;  // used from lane 7
            const float3 dc = dcos(G, T);
            const float e2_0 = from_lane(T.e2, 0);
            const float da = G.valid ? __fmul_rn(T.coef, O.axis == 0 ? dc.x : (O.axis == 1 ? dc.y : dc.z)) : 0.0f;
            // face_difference of each axis on its + lane, whose neighbour holds the - side
            const float w = e2_0 + T.e2;
            const float face = fmaf(w, dL, from_lane(__fmul_rn(w, dL), p + 1)), side = __fsub_rn(da, from_lane(da, p + 1));
            const float flux[3] = {from_lane(face, 1), from_lane(face, 3), from_lane(face, 5)};
            const float div[3] = {from_lane(side, 1), from_lane(side, 3), from_lane(side, 5)};
            float lv = 0.0f, b = any ? 1.0f : P.b_flat;
            if (p == 0 && solid) center_terms(P, G, T, L, hxy, hxz, hyz, flux, div, lv, b);
            __syncwarp();
            lv = from_lane(lv, 0);
            b = from_lane(b, 0);
#pragma unroll
            for (int h = 0; h < NH; ++h)
                if (solid && t == 8 * h + p) {
                    lap_sl[h] = lv;
                    b_sl[h] = b;
                }
        }
        al = from_lane(al, 7);
        if (heavy && ts > 0) w_sl = P.w0 * (al * al);
    }

    // ---- pair sums (trio_cell), lane t on phase t
    const int N = P.N;
    float W[NH], Ag[NH], dpi[NH], outv[NH];
#pragma unroll
    for (int h = 0; h < NH; ++h) W[h] = Ag[h] = dpi[h] = outv[h] = 0.0f;
    // (no branch on t < n: the loads of two phases are in flight together)
#pragma unroll 2
    for (int t = 0; t < n_most; ++t) {
        const int id = phase_of(ids, t);
        const float v = phase_of(vc, t), lp = phase_of(lap, t);
        const bool has = t < n;
#pragma unroll
        for (int h = 0; h < NH; ++h) {
            if (h > 0 && 8 * h >= n_most) break;
            const float w0 = __ldg(M.wij + ids[h] * N + id), a2 = __ldg(M.a2ij + ids[h] * N + id);
            const float w = (id == LIQ && ids[h] != LIQ) ? w_sl : w0;
            W[h] = has ? fmaf(w, v, W[h]) : W[h];
            Ag[h] = has ? fmaf(a2, lp, Ag[h]) : Ag[h];
        }
    }
    const double Tmc = P.clock ? P.clock->tmc[P.parity] : P.Tmc;
    const float dT = P.t_uniform ? P.dT_uniform : (float)(M.T0z[k] - Tmc);
    const float inv_n = 1.0f / (float)(n > 0 ? n : 1);
#pragma unroll 2
    for (int t = 0; t < n_most; ++t) {
        const int j = phase_of(ids, t);
        const float v2 = phase_of(vc, t), W2 = phase_of(W, t), A2 = phase_of(Ag, t), l2 = phase_of(lap_sl, t), b2 = phase_of(b_sl, t);
#pragma unroll
        for (int h = 0; h < NH; ++h) {
            if (h > 0 && 8 * h >= n_most) break;
            const bool has = t < n && t != 8 * h + p;
            const int i = ids[h];
            const bool sl = (i != LIQ && j == LIQ), ls = (i == LIQ && j != LIQ);
            float me = __ldg(M.mij + i * N + j);
            const float T = sl ? 0.5f * lap_sl[h] : (ls ? -0.5f * l2 : 0.5f * __fsub_rn(Ag[h], A2));
            const float ppp = __fadd_rn(__fsub_rn(W[h], W2), T);
            const float df = sl ? -P.Sf * dT : (ls ? P.Sf * dT : 0.0f);
            const float tf = __fmul_rn(__fmul_rn(FORCE_PREF, sqrtf(fmaxf(__fmul_rn(vc[h], v2), 0.0f))), df);
            me = sl ? me * b_sl[h] : (ls ? me * b2 : me);
            const float d = __fsub_rn(dpi[h], __fmul_rn(__fmul_rn(__fmul_rn(2.0f, me), inv_n), __fsub_rn(ppp, tf)));
            dpi[h] = has ? d : dpi[h];
        }
    }
#pragma unroll
    for (int h = 0; h < NH; ++h)
        if (8 * h + p < n) outv[h] = fminf(fmaxf(fmaf(P.dt, dpi[h], vc[h]), 0.0f), 1.0f);
    // renormalise with a compensated (TwoSum) float accumulation (:663-680)
    float sum = 0.0f, low = 0.0f;
#pragma unroll 1
    for (int t = 0; t < n_most; ++t) {
        const float b = phase_of(outv, t);
        const float s2 = sum + b;
        const float bb = s2 - sum;
        low = t < n ? low + ((sum - (s2 - bb)) + (b - bb)) : low;
        sum = t < n ? s2 : sum;
    }
    // stored list: the phases that stay positive, ascending; all clipped to
    // ~0: the liquid takes the cell (:679-680)
    const bool normal = sum + low > 1e-20f;
    float inv = 1.0f / sum;
    inv = fmaf(-__fmul_rn(inv, inv), low, inv);
    int stored = normal ? 0 : 1, id_first = LIQ;
    const bool writes = active && !ovf;
#pragma unroll
    for (int h = 0; h < NH; ++h) {
        const float v = normal ? outv[h] * inv : outv[h];
        const bool keep = 8 * h + p < n && v > 0.0f && (normal || ids[h] != LIQ);
        const uint32_t mask = __ballot_sync(ALL, keep) >> (8 * oct) & 0xffu;
        const int at = stored + __popc(mask & ((1u << p) - 1u));
        const int id = from_lane(ids[h], max(__ffs(mask) - 1, 0));
        if (stored == 0 && mask) id_first = id;
        if (writes && keep && at < S) {
            if (at > 0) out.idx[slot_at(at, cells, c)] = (uint16_t)ids[h];
            out.val[slot_at(at, cells, c)] = v;
        }
        stored += __popc(mask);
    }
    if (p == 0 && active) {
        if (ovf) {
            // leave the cell as it was and report; the host re-runs the step
            // with a wider template
            atomicOr(err, MPF3D_DEV_SLOT_OVERFLOW);
            const int c0 = min(hcount(hw), S);
            out.head[c] = hw;
            for (int s = 0; s < c0; ++s) {
                out.idx[slot_at(s, cells, c)] = __ldg(in.idx + slot_at(s, cells, c));
                out.val[slot_at(s, cells, c)] = __ldg(in.val + slot_at(s, cells, c));
            }
        } else {
            if (!normal) out.val[c] = 1.0f;
            // one stored phase: its renormalised value is 1 and is left implicit
            out.head[c] = mkhead(id_first, min(stored, S), false);
            if (stored > S) atomicOr(err, MPF3D_DEV_SLOT_OVERFLOW);
        }
    }
    return true;
}

// the cells of a warp by up to 8 phases, one per lane; where one has more, by AMAX (whose
// arrays cost rest_kernel with 16 slots about 300 bytes of spills)
template <int S, int AMAX, int NT>
__device__ __forceinline__ void octet_many(const In &in, const Out &out, const Mats &M, const Params &P,
                                        int32_t *__restrict__ err, const OctetLane &O, bool active, int l, int m,
                                        int k) {
    octet_phases<S, AMAX, NT, true>(in, out, M, P, err, O, active, l, m, k);
}

template <int S, int AMAX, int NT>
__device__ __forceinline__ void octet_cell(const In &in, const Out &out, const Mats &M, const Params &P,
                                           int32_t *__restrict__ err, const OctetLane &O, bool active, int l, int m,
                                           int k) {
    if (!octet_phases<S, 8, NT, AMAX == 8>(in, out, M, P, err, O, active, l, m, k))
        octet_many<S, AMAX, NT>(in, out, M, P, err, O, active, l, m, k);
}

// ---------------------------------------------------------------------------
// Any queued cell, one thread: the lists merged and the pair sums formed in arrays of
// local memory, a phase at a time.  A cell takes several times as long as by an octet,
// but 32 of them share a warp where octets have four: the better form where the cells
// are many (see Lists::are_long, EVERYWHERE and MANY_LEFT).
// FACETS: the anisotropic solid-liquid terms, for cells that have them.
template <int S, int AMAX, bool FACETS, int NT>
__device__ __forceinline__ void any_cell(const In &in, const Out &out, const Mats &M, const Params &P,
                                         int32_t *__restrict__ err, int l, int m, int k) {
    constexpr int NONE = 0x7fffffff;
    const uint32_t cells = P.cells32;
    const Offsets o(P, l, m, k);
    const uint32_t c = o.c, pt[7] = {c, c + o.xp, c + o.xm, c + o.yp, c + o.ym, c + o.zp, c + o.zm};
    int n = 0, ts = -1, ids[AMAX];
    float vc[AMAX], lap[AMAX], vL[7], maxv = -1.0f;
    float3 gs = make_float3(0.f, 0.f, 0.f);
    bool ovf = false;
    uint32_t hw[7];
    int pos[7], next[7];
#pragma unroll
    for (int p = 0; p < 7; ++p) {
        hw[p] = __ldg(in.head + pt[p]);
        pos[p] = 0;
        next[p] = hcount(hw[p]) > 0 ? hid0(hw[p]) : NONE;
        vL[p] = 0.0f;
    }
    while (true) {
        int id = next[0];
#pragma unroll
        for (int p = 1; p < 7; ++p) id = min(id, next[p]);
        if (id == NONE) break;
        float v[7];
#pragma unroll
        for (int p = 0; p < 7; ++p) {
            v[p] = 0.0f;
            if (next[p] != id) continue;
            v[p] = pos[p] == 0 ? value0(in, hw[p], pt[p]) : __ldg(in.val + slot_at(pos[p], cells, pt[p]));
            ++pos[p];
            next[p] = pos[p] < min(hcount(hw[p]), S) ? (int)__ldg(in.idx + slot_at(pos[p], cells, pt[p])) : NONE;
        }
        if (n == AMAX) {
            ovf = true;
            break;
        }
        ids[n] = id;
        vc[n] = v[0];
        lap[n] = lap7(P, v);
        if (id == LIQ) {
#pragma unroll
            for (int p = 0; p < 7; ++p) vL[p] = v[p];
        } else if (v[0] > maxv) {
            maxv = v[0];
            ts = n;
            gs = make_float3((v[1] - v[2]) * P.inv_2dx, (v[3] - v[4]) * P.inv_2dx, (v[5] - v[6]) * P.inv_2dx);
        }
        ++n;
    }
    if (ovf) {
        // leave the cell as it was and report; the host re-runs the step with a
        // wider template
        atomicOr(err, MPF3D_DEV_SLOT_OVERFLOW);
        out.head[c] = hw[0];
        for (int t = 0; t < min(hcount(hw[0]), S); ++t) {
            out.idx[slot_at(t, cells, c)] = __ldg(in.idx + slot_at(t, cells, c));
            out.val[slot_at(t, cells, c)] = __ldg(in.val + slot_at(t, cells, c));
        }
        return;
    }
    // solid-liquid terms
    const bool heavy = n > 1 && ids[0] == LIQ, facets = FACETS && heavy && P.use_aniso;
    const float lap_iso = heavy ? P.eps0sq * lap[0] : 0.0f;  // isotropic branch of the switchable kernel (:729-731)
    float lap_sl[AMAX], b_sl[AMAX], w_sl = P.w0;
    if (facets) {
        const Stencil st(in, P, o, vL);
        lap_sl[0] = 0.0f;
        b_sl[0] = 1.0f;
#pragma unroll 1
        for (int t = 1; t < n; ++t) {
            const float *ug = M.n111 + (size_t)(P.n111_base + ids[t]) * 24;
            float un[3 * NT], lv, b;
#pragma unroll
            for (int q = 0; q < 3 * NT; ++q) un[q] = __ldg(ug + q);
            interface_terms<NT>(P, st, vL, un, lv, b);
            lap_sl[t] = lv;
            b_sl[t] = b;
            if (t == ts) {
                const float al = point_terms<NT>(P, Grad(P, gs), un).a;
                w_sl = P.w0 * (al * al);
            }
        }
    }
    // pair sums (trio_cell)
    const int N = P.N;
    float W[AMAX], Ag[AMAX], outv[AMAX];
#pragma unroll 1
    for (int t = 0; t < n; ++t) {
        const int i = ids[t];
        float w = 0.0f, a = 0.0f;
#pragma unroll 1
        for (int q = 0; q < n; ++q) {
            const float wik = ids[q] == LIQ && i != LIQ ? w_sl : __ldg(M.wij + i * N + ids[q]);
            w = fmaf(wik, vc[q], w);
            a = fmaf(__ldg(M.a2ij + i * N + ids[q]), lap[q], a);
        }
        W[t] = w;
        Ag[t] = a;
    }
    const double Tmc = P.clock ? P.clock->tmc[P.parity] : P.Tmc;
    const float dT = P.t_uniform ? P.dT_uniform : (float)(M.T0z[k] - Tmc);
    const float inv_n = 1.0f / (float)(n > 0 ? n : 1);
    float sum = 0.0f, low = 0.0f;
#pragma unroll 1
    for (int t = 0; t < n; ++t) {
        const int i = ids[t];
        float dpi = 0.0f;
#pragma unroll 1
        for (int q = 0; q < n; ++q) {
            if (q == t) continue;
            const int j = ids[q];
            const bool sl = i != LIQ && j == LIQ, ls = i == LIQ && j != LIQ;
            const float l1 = sl && facets ? lap_sl[t] : lap_iso, l2 = ls && facets ? lap_sl[q] : lap_iso;
            const float T = sl ? 0.5f * l1 : (ls ? -0.5f * l2 : 0.5f * __fsub_rn(Ag[t], Ag[q]));
            const float ppp = __fadd_rn(__fsub_rn(W[t], W[q]), T);
            const float df = sl ? -P.Sf * dT : (ls ? P.Sf * dT : 0.0f);
            const float tf = __fmul_rn(__fmul_rn(FORCE_PREF, sqrtf(fmaxf(__fmul_rn(vc[t], vc[q]), 0.0f))), df);
            float me = __ldg(M.mij + i * N + j);
            if (facets) me = sl ? me * b_sl[t] : (ls ? me * b_sl[q] : me);
            dpi = __fsub_rn(dpi, __fmul_rn(__fmul_rn(__fmul_rn(2.0f, me), inv_n), __fsub_rn(ppp, tf)));
        }
        outv[t] = fminf(fmaxf(fmaf(P.dt, dpi, vc[t]), 0.0f), 1.0f);
        // compensated (TwoSum) float accumulation (:663-680)
        const float s2 = sum + outv[t], bb = s2 - sum;
        low += (sum - (s2 - bb)) + (outv[t] - bb);
        sum = s2;
    }
    // stored list: the phases that stay positive, ascending; all clipped to
    // ~0: the liquid takes the cell (:679-680)
    const bool normal = sum + low > 1e-20f;
    float inv = 1.0f / sum;
    inv = fmaf(-__fmul_rn(inv, inv), low, inv);
    int stored = normal ? 0 : 1, first = LIQ;
    if (!normal) out.val[c] = 1.0f;
#pragma unroll 1
    for (int t = 0; t < n; ++t) {
        const float v = normal ? outv[t] * inv : outv[t];
        if (!(v > 0.0f) || (!normal && ids[t] == LIQ)) continue;
        if (stored < S) {
            if (stored == 0) first = ids[t];
            else out.idx[slot_at(stored, cells, c)] = (uint16_t)ids[t];
            out.val[slot_at(stored, cells, c)] = v;
        }
        ++stored;
    }
    // one stored phase: its renormalised value is 1 and is left implicit
    out.head[c] = mkhead(first, min(stored, S), false);
    if (stored > S) atomicOr(err, MPF3D_DEV_SLOT_OVERFLOW);
}

// Kernel 1 of a step: every cell.  Uniform neighbourhoods (the cell and its
// 6 neighbours hold one and the same phase: active list of one phase, empty
// pair sums, renormalised fraction exactly 1) are written directly; every
// other cell is appended to a work list -- solid-liquid interface cells
// (liquid and a solid in the neighbourhood, anisotropy on) to the back,
// the rest (grain boundaries, junctions without liquid, the isotropic model)
// to the front -- so that the general update runs with converged warps.
constexpr int SWEEP_ZB = 4;  // cells per thread along z (default; batches always use it)

// Where the sweep sends its cells: 0 for one it wrote itself, else 1 + the
// list (0 general, 1 interface, 2 interface with several solids), two bits per
// cell of a thread's column.  BlockSink counts a block's cells per list in
// shared memory (one shared atomic per warp and list, over the warp's whole
// column) and keeps each cell's offset in registers; the block then reserves
// its segments with one global atomic per list and writes the cell indices
// (flush).  The counters are one address each, and per-warp global atomics
// from every SM queued up at the L2 slice that holds them.  Cells are
// independent, so the order within a list changes no result.

template <int ZB>
struct BlockSink {
    uint32_t *cnt;     // shared: cells of the block per list
    uint32_t off[ZB];  // cell j's position in its list's block segment
    uint32_t codes;
    uint32_t cell, plane;  // cell j is cell + j * plane

    __device__ __forceinline__ explicit BlockSink(uint32_t *c) : cnt(c), codes(0) {}
    // by all lanes of a warp
    __device__ __forceinline__ void add(uint32_t column, uint32_t cell0, uint32_t stride) {
        codes = column;
        cell = cell0;
        plane = stride;
        if (!__any_sync(0xffffffffu, column)) return;
        const unsigned before = (1u << (threadIdx.x & 31)) - 1u;
#pragma unroll
        for (uint32_t L = 1; L <= 3; ++L) {
            uint32_t total = 0, at[ZB];
#pragma unroll
            for (int j = 0; j < ZB; ++j) {
                const unsigned bm = __ballot_sync(0xffffffffu, (column >> (2 * j) & 3u) == L);
                at[j] = total + __popc(bm & before);
                total += __popc(bm);
            }
            if (!total) continue;
            uint32_t base = 0;
            if ((threadIdx.x & 31) == 0) base = atomicAdd(cnt + L - 1, total);
            base = __shfl_sync(0xffffffffu, base, 0);
#pragma unroll
            for (int j = 0; j < ZB; ++j)
                if ((column >> (2 * j) & 3u) == L) off[j] = base + at[j];
        }
    }
    // after the block's adds and a barrier: base[L] is the block's first
    // position in list L
    __device__ __forceinline__ void flush(const Queue &Q, uint32_t cells, const uint32_t *base) const {
#pragma unroll
        for (int j = 0; j < ZB; ++j) {
            const uint32_t code = codes >> (2 * j) & 3u;
            if (!code) continue;
            const uint32_t pos = base[code - 1] + off[j];
            const uint32_t c = cell + (uint32_t)j * plane;
            Q.items[code == 1 ? pos : (code == 2 ? cells - 1u - pos : cells + pos)] = c;
        }
    }
};

// Classification of a cell c from its head h0 and its 6 neighbours' heads hn =
// {x+, x-, y+, y-, z+, z-} at qn (z clamped: a neighbour beyond the domain is the
// cell itself): a uniform neighbourhood is written directly, any other cell goes
// to a work list.  Returns the cell's code.
__device__ __forceinline__ uint32_t sweep_cell(const In &in, const Out &out, const Params &P, bool split, uint32_t c,
                                               uint32_t h0, const uint32_t (&hn)[6], const uint32_t (&qn)[6]) {
    const uint32_t h[7] = {h0, hn[0], hn[1], hn[2], hn[3], hn[4], hn[5]};
    uint32_t differ = 0, any = 0, least = 0xffffffffu;
#pragma unroll
    for (int p = 0; p < 7; ++p) {
        differ |= h[p] ^ h0;
        any |= h[p];
        least = min(least, h[p] - 1u);
    }
    if (differ == 0 && (h0 & 0xffu) == 1u) {
        // the one phase of the neighbourhood keeps the cell at exactly 1
        out.head[c] = h0;
        return 0;
    }
    // Liquid somewhere: a head with phases and first id 0 is 1..255 (an empty one
    // is 0).  A solid somewhere: a first id beyond 0, or a count beyond 1.
    const bool heavy = P.use_aniso && least < 0xffu && (any & ~0x81u) != 0u;
    if (!heavy) return 1;
    if (!split) return 2;
    // Several solids: more than one in a cell (3 phases, or 2 without liquid), or
    // different ones in two; the solid beside the liquid of a two-phase cell is
    // its second id (head 2: first id 0, count 2).
    uint32_t second[7], most = 0, hi = 0, lo = 0xffffffffu;
#pragma unroll
    for (int p = 0; p < 7; ++p)
        second[p] = h[p] == 2u ? (uint32_t)__ldg(in.idx + P.cells32 + (p == 0 ? c : qn[p == 0 ? 0 : p - 1])) : h[p] >> 8;
#pragma unroll
    for (int p = 0; p < 7; ++p) {
        most = max(most, (h[p] & 0x7fu) + (h[p] >> 8 ? 1u : 0u));
        hi = max(hi, second[p]);
        lo = min(lo, second[p] - 1u);
    }
    return most > 2u || hi != lo + 1u ? 3 : 2;
}

// The sweep of one column of ZB cells (l, m, k0..k0+ZB-1) of a domain;
// returns their codes (cells past the top count as written).
template <int ZB = SWEEP_ZB>
__device__ __forceinline__ uint32_t sweep_column(const In &in, const Out &out, const Params &P, bool split, int l,
                                                 int m, int k0) {
    const uint32_t plane = (uint32_t)P.nx * (uint32_t)P.ny;
    const uint32_t col = P.base + (uint32_t)m * (uint32_t)P.nx + (uint32_t)l;
    const uint32_t dxp = (l < P.nx - 1) ? 1u : (uint32_t)(1 - P.nx);
    const uint32_t dxm = (l > 0) ? (uint32_t)-1 : (uint32_t)(P.nx - 1);
    const uint32_t dyp = (m < P.ny - 1) ? (uint32_t)P.nx : (uint32_t)(-(P.ny - 1) * P.nx);
    const uint32_t dym = (m > 0) ? (uint32_t)(-P.nx) : (uint32_t)((P.ny - 1) * P.nx);
    // heads of the column k0-1 .. k0+ZB (z clamped)
    uint32_t hz[ZB + 2];
    uint32_t codes = 0;
#pragma unroll
    for (int j = 0; j < ZB + 2; ++j) {
        const int kk = min(max(k0 - 1 + j, 0), P.nz - 1);
        hz[j] = __ldg(in.head + (uint32_t)kk * plane + col);
    }
#pragma unroll
    for (int j = 0; j < ZB; ++j) {
        const int k = k0 + j;
        if (k >= P.nz) break;
        const uint32_t c = (uint32_t)k * plane + col;
        const uint32_t h0 = hz[j + 1];
        // neighbour indices wrap in 32-bit cell-index arithmetic; the offsets
        // must be added to the index, never to the pointer
        const uint32_t qxp = c + dxp, qxm = c + dxm, qyp = c + dyp, qym = c + dym;
        uint32_t hn[6] = {__ldg(in.head + qxp), __ldg(in.head + qxm), __ldg(in.head + qyp),
                          __ldg(in.head + qym), hz[j + 2], hz[j]};
        // a z neighbour beyond the domain is the cell itself (clamped index)
        if (k == P.nz - 1) hn[4] = h0;
        if (k == 0) hn[5] = h0;
        const uint32_t qn[6] = {qxp, qxm, qyp, qym, k < P.nz - 1 ? c + plane : c, k > 0 ? c - plane : c};
        codes |= sweep_cell(in, out, P, split, c, h0, hn, qn) << (2 * j);
    }
    return codes;
}

// The same sweep reading the heads from a shared-memory tile: the block's
// 32 x by x ZB cells plus a one-cell halo, staged by the Tensor Memory
// Accelerator (TMA_X columns from l0 - 4, by + 2 rows from m0 - 1, ZB + 2
// layers from k0 - 1; the periodic x and y halos patched in after the copy).
constexpr int TMA_X = 40;

template <int ZB>
__device__ __forceinline__ uint32_t sweep_column_tile(const uint32_t *tile, int rows, const In &in, const Out &out,
                                                      const Params &P, bool split, int l, int m, int k0, int l0,
                                                      int m0) {
    const uint32_t plane = (uint32_t)P.nx * (uint32_t)P.ny;
    const uint32_t col = (uint32_t)m * (uint32_t)P.nx + (uint32_t)l;
    const int xi = l - l0 + 4, yi = m - m0 + 1;
    auto at = [&](int x, int y, int z) { return tile[(z * rows + y) * TMA_X + x]; };
    uint32_t codes = 0;
#pragma unroll
    for (int j = 0; j < ZB; ++j) {
        const int k = k0 + j;
        if (k >= P.nz) break;
        const int zi = j + 1;
        const uint32_t c = (uint32_t)k * plane + col;
        const uint32_t h0 = at(xi, yi, zi);
        uint32_t hn[6] = {at(xi + 1, yi, zi), at(xi - 1, yi, zi), at(xi, yi + 1, zi),
                          at(xi, yi - 1, zi), at(xi, yi, zi + 1), at(xi, yi, zi - 1)};
        if (k == P.nz - 1) hn[4] = h0;
        if (k == 0) hn[5] = h0;
        const uint32_t row = (uint32_t)k * plane;
        const uint32_t qn[6] = {row + (uint32_t)m * (uint32_t)P.nx + (uint32_t)wrap_p(l, P.nx),
                                row + (uint32_t)m * (uint32_t)P.nx + (uint32_t)wrap_m(l, P.nx),
                                row + (uint32_t)wrap_p(m, P.ny) * (uint32_t)P.nx + (uint32_t)l,
                                row + (uint32_t)wrap_m(m, P.ny) * (uint32_t)P.nx + (uint32_t)l,
                                k < P.nz - 1 ? c + plane : c, k > 0 ? c - plane : c};
        codes |= sweep_cell(in, out, P, split, c, h0, hn, qn) << (2 * j);
    }
    return codes;
}

// Quiet tiles.  A tile is the 32 x 1 x ZB cells one warp of the sweep
// covers.  When every cell of a tile is uniform in step n, step n leaves the
// tile unchanged (S(n+1) = S(n) there).  If the tile and its 6 face
// neighbours were all uniform in step n-1, the neighbourhoods of the tile's
// cells are unchanged in step n, so the tile is uniform again, and its
// content in the output buffer -- written by step n-2, i.e. S(n-1) -- already
// equals S(n+1): the warp writes nothing and queues nothing.  flags[2][tiles]
// (one byte per tile, uniform = 1) alternate with the step parity; both
// halves must be zero after the state buffers are written from outside the
// step (the first step then visits every tile).
struct Tiles {
    uint8_t *__restrict__ flags;
    int ntx, nkb;
    uint32_t n;  // tiles per parity half
};

template <int ZB>
__host__ __device__ __forceinline__ uint32_t tiles_of(int nx, int ny, int nz) {
    return (uint32_t)((nz + ZB - 1) / ZB) * (uint32_t)ny * (uint32_t)((nx + 31) / 32);
}

// One thread of the sweep advances the device step clock (Params::clock):
// the step's T_melt + cooling for the work-list kernels, the next index.
__device__ __forceinline__ void advance_clock(const Params &P) {
    if (!P.clock) return;
    const int64_t s = P.clock->step[P.parity];
    P.clock->tmc[P.parity] = __dadd_rn(P.clock_T_melt, __dmul_rn((double)s, P.clock_rate));
    P.clock->step[P.parity ^ 1] = s + 1;
}

// The sweep's tiles in chunks of blockDim.y rows; a block takes every
// gridDim.x-th chunk, at most SWEEP_TILES tiles (distant ones: the tiles that are
// not quiet lie together).  A lane per tile reads its flags (quiet), then the warps
// share the others, one per warp and round; visit fills the warp's sink, flag_of
// is a tile's place in fout, domain_of its instance, or -1 for the rows of a chunk
// beyond the domain's last: they are no tiles, are not listed, and have no flag (the
// place that flag_of computes for one belongs to another tile).  A warp of its own for each of the 79 % quiet tiles of
// a 256^3 step with 64 grains spent the time on starting blocks; us per step with a
// block per chunk / with up to 128 tiles per block: 256^3 41 / 23, 512 x 512 x 256
// 155 / 63 (64 tiles: 69, 32: 78), 24 bicrystals 92 / 79.  With consecutive chunks
// per block, 256^3 took 43: blocks whose tiles are all visited came last.
constexpr uint32_t SWEEP_TILES = 128;  // blocks have at least as many threads

template <int ZB, class Domain, class Flag, class Quiet, class Visit>
__device__ __forceinline__ void sweep_tiles(const Queue &Q, uint32_t cells, int parity, uint32_t chunks,
                                            uint8_t *__restrict__ fout, Domain &&domain_of, Flag &&flag_of,
                                            Quiet &&quiet, Visit &&visit) {
    __shared__ uint32_t s_cnt[3], s_base[3], s_tile[SWEEP_TILES], s_n;
    __shared__ int s_of[SWEEP_TILES];
    const uint32_t lane = threadIdx.x, tlin = lane + 32u * threadIdx.y, rows = blockDim.y;
    if (tlin < 3) s_cnt[tlin] = 0;
    if (tlin == 3) s_n = 0;
    __syncthreads();
    if (32u * threadIdx.y < SWEEP_TILES) {
        const uint32_t chunk = blockIdx.x + tlin / rows * gridDim.x, row = tlin % rows;
        const int of = chunk < chunks ? domain_of(chunk, row) : -1;
        const bool in = of >= 0;
        const bool skip = in && quiet(of, chunk, row);
        if (skip && fout) fout[flag_of(chunk, row)] = 1;
        const unsigned mask = __ballot_sync(0xffffffffu, in && !skip);
        uint32_t at = 0;
        if (lane == 0 && mask) at = atomicAdd(&s_n, (uint32_t)__popc(mask));
        at = __shfl_sync(0xffffffffu, at, 0);
        at += __popc(mask & ((1u << lane) - 1u));
        if (mask >> lane & 1u) {
            s_tile[at] = chunk * rows + row;
            s_of[at] = of;
        }
    }
    __syncthreads();
    const uint32_t n = s_n;
    for (uint32_t r = 0; r < n; r += rows) {
        BlockSink<ZB> sink(s_cnt);
        if (r + threadIdx.y < n) {
            const uint32_t t = s_tile[r + threadIdx.y], chunk = t / rows, row = t - chunk * rows;
            visit(s_of[r + threadIdx.y], chunk, row, sink);
            if (fout) {
                const bool all = __all_sync(0xffffffffu, sink.codes == 0u);
                if (lane == 0) fout[flag_of(chunk, row)] = all ? 1 : 0;
            }
        }
        __syncthreads();
        if (tlin < 3) {
            const uint32_t k = s_cnt[tlin];
            uint32_t *ctr = tlin == 2 ? Q.count + 4 + parity : Q.count + 2 * parity + tlin;
            s_base[tlin] = k ? atomicAdd(ctr, k) : 0u;
            s_cnt[tlin] = 0;
        }
        __syncthreads();
        sink.flush(Q, cells, s_base);
    }
}

// First statements of a kernel that launch_early starts: its blocks may be
// resident before the stream's previous kernel is complete, and wait here until
// it is and its writes are visible; the next such kernel may do the same.
__device__ __forceinline__ void wait_for_previous() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// the other parity's counters, which the previous step's kernels are done with
__device__ __forceinline__ void clear_counters(const Queue &Q, int parity, uint32_t t) {
    if (t < 2) Q.count[2 * (parity ^ 1) + t] = 0;
    if (t == 2 && Q.split) Q.count[4 + (parity ^ 1)] = 0;
}

// 40 registers (3 blocks of 512 per SM): more resident warps beat keeping
// ZB = 8 columns in registers; the tuner then prefers ZB = 4
template <int ZB>
__global__ void __launch_bounds__(512, 3) sweep_kernel(In in, Out out, Params P, Queue Q, int parity, Tiles T,
                                                       uint32_t chunks) {
    wait_for_previous();
    if (blockIdx.x == 0) {
        const uint32_t t = threadIdx.x + 32u * threadIdx.y;
        clear_counters(Q, parity, t);
        if (t == 3) advance_clock(P);
    }
    const uint8_t *fin = T.flags + (size_t)(parity ^ 1) * T.n;
    uint8_t *fout = T.flags ? T.flags + (size_t)parity * T.n : nullptr;
    const uint32_t ntx = (uint32_t)T.ntx, bands = ((uint32_t)P.ny + blockDim.y - 1u) / blockDim.y;
    struct Tile {
        int tx, m, kb;
    };
    auto tile_of = [&](uint32_t chunk, uint32_t row) {  // chunks: x first, then bands of rows, then z
        const uint32_t q = chunk / ntx, kb = q / bands;
        return Tile{(int)(chunk - q * ntx), (int)((q - kb * bands) * blockDim.y + row), (int)kb};
    };
    auto at = [&](int a, int b, int c) { return ((uint32_t)c * (uint32_t)P.ny + (uint32_t)b) * ntx + (uint32_t)a; };
    sweep_tiles<ZB>(
        Q, P.cells32, parity, chunks, fout,
        [&](uint32_t chunk, uint32_t row) { return tile_of(chunk, row).m < P.ny ? 0 : -1; },
        [&](uint32_t chunk, uint32_t row) {
            const Tile t = tile_of(chunk, row);
            return at(t.tx, t.m, t.kb);
        },
        [&](int, uint32_t chunk, uint32_t row) {
            const auto [tx, m, kb] = tile_of(chunk, row);
            if (!T.flags) return false;
            // the 7 flags are loaded together (no short-circuit chain of loads)
            const uint32_t f0 = fin[at(tx, m, kb)];
            const uint32_t f1 = fin[at(tx + 1 < T.ntx ? tx + 1 : 0, m, kb)];
            const uint32_t f2 = fin[at(tx > 0 ? tx - 1 : T.ntx - 1, m, kb)];
            const uint32_t f3 = fin[at(tx, m + 1 < P.ny ? m + 1 : 0, kb)];
            const uint32_t f4 = fin[at(tx, m > 0 ? m - 1 : P.ny - 1, kb)];
            const uint32_t f5 = fin[at(tx, m, kb + 1 < T.nkb ? kb + 1 : kb)];
            const uint32_t f6 = fin[at(tx, m, kb > 0 ? kb - 1 : kb)];
            return (f0 & f1 & f2 & f3 & f4 & f5 & f6) != 0u;
        },
        [&](int, uint32_t chunk, uint32_t row, BlockSink<ZB> &sink) {
            const Tile t = tile_of(chunk, row);
            const uint32_t plane = (uint32_t)P.nx * (uint32_t)P.ny;
            const int l = t.tx * 32 + (int)threadIdx.x;
            sink.add(l < P.nx ? sweep_column<ZB>(in, out, P, Q.split, l, t.m, t.kb * ZB) : 0u,
                     P.base + (uint32_t)(t.kb * ZB) * plane + (uint32_t)t.m * (uint32_t)P.nx + (uint32_t)l, plane);
        });
}

// Bounded wait on phase `parity` of a shared-memory mbarrier (nanoseconds
// of %globaltimer); false if it did not complete in time.
__device__ __forceinline__ bool mbar_wait_ns(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
    uint64_t t0;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    while (true) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.b32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        uint64_t t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 > limit_ns) return false;
    }
}

// Kernel 1 with its heads staged in shared memory by one TMA copy per block
// (cp.async.bulk.tensor.3d of the block's cells plus a one-cell halo from
// the head array, which the tensor map describes as nx x ny x nz uint32).
// Blocks whose warps are all quiet copy nothing.  The x and y halos at the
// domain's periodic edges lie outside the copied box (TMA fills them with
// zeros) and are patched in with plain loads; z halo layers outside the
// domain are never read (the clamped neighbour is the cell itself).  A copy
// that does not land within 1 s sets MPF3D_DEV_STAGING_TIMEOUT and the block
// waits once more before it leaves.  Same results as sweep_kernel.
template <int ZB>
__global__ void __launch_bounds__(512, 3) sweep_kernel_tma(const __grid_constant__ CUtensorMap map, In in, Out out,
                                                         Params P, Queue Q, int parity, Tiles T,
                                                         int32_t *__restrict__ err) {
    constexpr int MAX_ROWS = 16 + 2;
    __shared__ __align__(128) uint32_t tile[TMA_X * MAX_ROWS * (ZB + 2)];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t s_cnt[3], s_base[3];
    __shared__ int s_need;
    const int by = (int)blockDim.y, rows = by + 2;
    const int l0 = blockIdx.x * 32, m0 = blockIdx.y * by;
    const int l = l0 + threadIdx.x, m = m0 + threadIdx.y;
    const int k0 = blockIdx.z * ZB;
    const int tlin = threadIdx.x + 32 * threadIdx.y;
    const uint32_t bar_a = (uint32_t)__cvta_generic_to_shared(&bar);
    if (tlin < 3) s_cnt[tlin] = 0;
    if (tlin == 0) {
        s_need = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar_a) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.y == 0 && threadIdx.x < 2)
        Q.count[2 * (parity ^ 1) + threadIdx.x] = 0;  // the previous step's kernels are done with them
    if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.y == 0 && threadIdx.x == 2 && Q.split)
        Q.count[4 + (parity ^ 1)] = 0;
    if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.y == 0 && threadIdx.x == 3)
        advance_clock(P);
    // quiet flags of this warp's tile (as sweep_kernel)
    const bool row_ok = m < P.ny && k0 < P.nz;
    bool quiet = false;
    uint32_t t = 0;
    const uint8_t *fin = nullptr;
    uint8_t *fout = nullptr;
    if (row_ok && T.flags) {
        const int tx = (int)blockIdx.x, kb = k0 / ZB;
        fin = T.flags + (size_t)(parity ^ 1) * T.n;
        fout = T.flags + (size_t)parity * T.n;
        auto tid = [&](int a, int b, int c) {
            return ((uint32_t)c * (uint32_t)P.ny + (uint32_t)b) * (uint32_t)T.ntx + a;
        };
        t = tid(tx, m, kb);
        const uint32_t f0 = fin[t];
        const uint32_t f1 = fin[tid(tx + 1 < T.ntx ? tx + 1 : 0, m, kb)];
        const uint32_t f2 = fin[tid(tx > 0 ? tx - 1 : T.ntx - 1, m, kb)];
        const uint32_t f3 = fin[tid(tx, m + 1 < P.ny ? m + 1 : 0, kb)];
        const uint32_t f4 = fin[tid(tx, m > 0 ? m - 1 : P.ny - 1, kb)];
        const uint32_t f5 = fin[tid(tx, m, kb + 1 < T.nkb ? kb + 1 : kb)];
        const uint32_t f6 = fin[tid(tx, m, kb > 0 ? kb - 1 : kb)];
        quiet = (f0 & f1 & f2 & f3 & f4 & f5 & f6) != 0u;
    }
    __syncthreads();
    if (row_ok && !quiet && threadIdx.x == 0) s_need = 1;
    __syncthreads();
    const bool need = s_need != 0;
    bool staged = false;
    if (need) {
        if (tlin == 0) {
            const uint32_t bytes = (uint32_t)(TMA_X * rows * (ZB + 2) * 4);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar_a), "r"(bytes)
                         : "memory");
            asm volatile(
                "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
                "[%5];\n" ::"r"((uint32_t)__cvta_generic_to_shared(tile)),
                "l"(reinterpret_cast<uint64_t>(&map)), "r"(l0 - 4), "r"(m0 - 1), "r"(k0 - 1), "r"(bar_a)
                : "memory");
        }
        staged = mbar_wait_ns(bar_a, 0, 1000000000ull);
        if (!staged) {
            if (threadIdx.x == 0) atomicOr(err, MPF3D_DEV_STAGING_TIMEOUT);
            mbar_wait_ns(bar_a, 0, 1000000000ull);  // the copy may still land: let it, before leaving
        }
        staged = __syncthreads_and(staged) != 0;
        if (staged) {
            // periodic halos outside the copied box
            const uint32_t plane = (uint32_t)P.nx * (uint32_t)P.ny;
            const int nz_box = ZB + 2;
            if (l0 == 0 || l0 + 32 >= P.nx) {
                for (int e = tlin; e < 2 * rows * nz_box; e += 32 * by) {
                    const int side = e / (rows * nz_box), r = e % (rows * nz_box);
                    const int yi = r % rows, zi = r / rows;
                    const int gy = m0 - 1 + yi, gz = k0 - 1 + zi;
                    if (gy < 0 || gy >= P.ny || gz < 0 || gz >= P.nz) continue;
                    if (side == 0 && l0 == 0)
                        tile[(zi * rows + yi) * TMA_X + 3] = __ldg(in.head + (uint32_t)gz * plane + (uint32_t)gy * P.nx + (P.nx - 1));
                    if (side == 1 && l0 + 32 >= P.nx)
                        tile[(zi * rows + yi) * TMA_X + (P.nx - l0 + 4)] = __ldg(in.head + (uint32_t)gz * plane + (uint32_t)gy * P.nx);
                }
            }
            if (m0 == 0 || m0 + by >= P.ny) {
                for (int e = tlin; e < 2 * 32 * nz_box; e += 32 * by) {
                    const int side = e / (32 * nz_box), r = e % (32 * nz_box);
                    const int xo = r % 32, zi = r / 32;
                    const int gx = l0 + xo, gz = k0 - 1 + zi;
                    if (gx >= P.nx || gz < 0 || gz >= P.nz) continue;
                    if (side == 0 && m0 == 0)
                        tile[(zi * rows + 0) * TMA_X + xo + 4] = __ldg(in.head + (uint32_t)gz * plane + (uint32_t)(P.ny - 1) * P.nx + gx);
                    if (side == 1 && m0 + by >= P.ny)
                        tile[(zi * rows + (P.ny - m0 + 1)) * TMA_X + xo + 4] = __ldg(in.head + (uint32_t)gz * plane + gx);
                }
            }
            __syncthreads();
        }
    }
    BlockSink<ZB> sink(s_cnt);
    const uint32_t plane = (uint32_t)P.nx * (uint32_t)P.ny;
    const uint32_t cell0 = (uint32_t)k0 * plane + (uint32_t)m * (uint32_t)P.nx + (uint32_t)l;
    if (row_ok && staged) {
        if (!T.flags) {
            sink.add(l < P.nx ? sweep_column_tile<ZB>(tile, rows, in, out, P, Q.split, l, m, k0, l0, m0) : 0u,
                     cell0, plane);
        } else if (quiet) {
            if (threadIdx.x == 0) fout[t] = 1;
        } else {
            sink.add(l < P.nx ? sweep_column_tile<ZB>(tile, rows, in, out, P, Q.split, l, m, k0, l0, m0) : 0u,
                     cell0, plane);
            const bool all = __all_sync(0xffffffffu, sink.codes == 0u);
            if (threadIdx.x == 0) fout[t] = all ? 1 : 0;
        }
    } else if (row_ok && quiet && threadIdx.x == 0) {
        fout[t] = 1;
    }
    __syncthreads();
    if (tlin < 3) {
        const uint32_t n = s_cnt[tlin];
        uint32_t *ctr = tlin == 2 ? Q.count + 4 + parity : Q.count + 2 * parity + tlin;
        s_base[tlin] = n ? atomicAdd(ctr, n) : 0u;
    }
    __syncthreads();
    sink.flush(Q, P.cells32, s_base);
}

// Lists so long that a thread per cell gets through them sooner than eight lanes: us a
// step by octets / by threads, 64 x 64 x 64 with two grains and 61 k cells listed 29.5 /
// 23.2, with 8 grains and 70 k 37.9 / 42.4, 113 k 47.3 / 40.8; 32 x 32 x 64 isotropic,
// 44 k 25.8 / 25.5, 58 k 31.5 / 27.0, with 20 k 16.2 / 19.5.  Cells with several solids, the
// costly ones, weigh more: 48 x 40 x 56 with 54 k of them 134 / 66.
constexpr uint32_t LONG_LISTS = 49152, LONG_SEVERAL = 16384;

// The work lists: 0 at items[0..), 1 at items[cells-1..] downwards, 2 at
// items[cells..).
struct Lists {
    uint32_t n[3];
    __device__ __forceinline__ Lists(const Queue &Q, int parity) {
        n[0] = *(volatile uint32_t *)(Q.count + 2 * parity);
        n[1] = *(volatile uint32_t *)(Q.count + 2 * parity + 1);
        n[2] = Q.split ? *(volatile uint32_t *)(Q.count + 4 + parity) : 0u;
    }
    __device__ __forceinline__ bool are_long() const {
        return n[2] > LONG_SEVERAL || n[0] + n[1] + n[2] > LONG_LISTS;
    }
    // index in items of entry i of the lists one after the other
    __device__ __forceinline__ uint32_t item(uint32_t i, uint32_t cells) const {
        if (i < n[0]) return i;
        i -= n[0];
        return i < n[1] ? cells - 1u - i : cells + (i - n[1]);
    }
};

// resident blocks of 128 threads per SM of octet_kernel: registers for any_cell, and
// still a wave for 12 k cells
constexpr int OCTET_BLOCKS = 5;

// calls cell(c, active) for the cells of all lists, four per warp and call, or where
// they are long each(c, of list 0?), one per thread
template <class Cell, class Each>
__device__ __forceinline__ void for_octets(const Queue &Q, uint32_t cells, int parity, Cell &&cell, Each &&each) {
    const Lists L(Q, parity);
    const uint32_t n = L.n[0] + L.n[1] + L.n[2], oct = (threadIdx.x & 31u) >> 3;
    if (L.are_long()) {
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
            each(Q.items[L.item(i, cells)], i < L.n[0]);
        return;
    }
    const uint32_t warps = gridDim.x * (blockDim.x >> 5), warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    for (uint32_t w = warp; w * 4u < n; w += warps) {
        const uint32_t i = w * 4u + oct;
        cell(Q.items[L.item(min(i, n - 1u), cells)], i < n);
    }
}

// Items get(0..n) one per thread, by take(item); those it refuses by
// rest(item, active), eight lanes each, shared out over the block's warps: they
// lie in clusters, and a warp that kept its own would take several, at 8-10 us
// each, one after the other.  For the same reason a block takes runs of RUN
// items from distant parts of the range; PER: items that make another block
// worth starting.
// With EACH, a block that is left with more than MANY_LEFT of them, and more than a third
// of its items, does them by each(item), one per thread.  isotropic_kernel, us a step, by
// octets / threads with a block for every 256 items, 96 and half of them / as it is: 64^3 with
// 146 k cells of 9 phases 380 / 130 / 108, 80^3 with 40 grains and 143 k cells listed 219 / 199 /
// 128, with a front, 8 grains and 35 k 21 / 21 / 17; a block for every 64 items 298, 148, 17.
constexpr uint32_t LEFT_CELLS = 1024, MANY_LEFT = 48;

template <uint32_t RUN, uint32_t PER, bool EACH, class Get, class Take, class Rest, class Each>
__device__ __forceinline__ void for_items(uint32_t n, Get &&get, Take &&take, Rest &&rest, Each &&each) {
    __shared__ uint32_t left[LEFT_CELLS], n_left;
    const uint32_t blocks = min(gridDim.x, (n + PER - 1u) / PER);
    if (blockIdx.x >= blocks) return;
    const uint32_t warp = threadIdx.x >> 5, oct = (threadIdx.x & 31u) >> 3;
    const uint32_t step = blocks * blockDim.x, passes = LEFT_CELLS / blockDim.x;
    if (threadIdx.x == 0) n_left = 0;
    __syncthreads();
    for (uint32_t at0 = 0; at0 < n;) {
        const uint32_t first = at0;
        for (uint32_t pass = 0; pass < passes && at0 < n; ++pass, at0 += step) {
            const uint32_t i = at0 + (threadIdx.x / RUN * blocks + blockIdx.x) * RUN + threadIdx.x % RUN;
            if (i >= n) continue;
            const uint32_t c = get(i);
            if (!take(c)) left[atomicAdd(&n_left, 1u)] = c;
        }
        __syncthreads();
        const uint32_t m = n_left;
        if (EACH && m > MANY_LEFT && 3u * m > (min(at0, n) - first) / blocks) {
            for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) each(left[i]);
        } else {
            for (uint32_t w = warp; w * 4u < m; w += blockDim.x >> 5)
                rest(left[min(w * 4u + oct, m - 1u)], w * 4u + oct < m);
        }
        __syncthreads();
        if (threadIdx.x == 0) n_left = 0;
        __syncthreads();
    }
}

// Set in the items that trio_cell left to the octets of a kernel of their own
// (lists 0 and 2; list 1 instead of 2 where the sweep kept all interface cells
// there).
constexpr uint32_t LEFT = 0x80000000u;

struct Place {
    int l, m, k;
    __device__ __forceinline__ Place(uint32_t r0, int nx, int ny) {
        const uint32_t plane = (uint32_t)nx * (uint32_t)ny;
        k = (int)(r0 / plane);
        const uint32_t r = r0 - (uint32_t)k * plane;
        m = (int)(r / (uint32_t)nx);
        l = (int)(r - (uint32_t)m * (uint32_t)nx);
    }
};

// Kernel 2 of a step on small domains: eight lanes per cell, or one thread where the
// lists are long.  NT: normals per grain (4 or 8, from P.sym_normals).
template <int S, int AMAX, int NT>
__global__ void __launch_bounds__(128, OCTET_BLOCKS) octet_kernel(In in, Out out, Mats M, Params P, Queue Q, int parity,
                                                       int32_t *__restrict__ err) {
    wait_for_previous();
    const OctetLane O;
    for_octets(Q, P.cells32, parity, [&](uint32_t c, bool active) {
        const Place at(c, P.nx, P.ny);
        octet_cell<S, AMAX, NT>(in, out, M, P, err, O, active, at.l, at.m, at.k);
    }, [&](uint32_t c, bool general) {
        const Place at(c, P.nx, P.ny);
        if (!general || !trio_cell<S, false, 4>(in, out, M, P, at.l, at.m, at.k))
            any_cell<S, AMAX, true, NT>(in, out, M, P, err, at.l, at.m, at.k);
    });
}

// The work-list kernels on large domains: list 1 by pair_cell, where the sweep
// kept it to pairs, on a second stream beside lists 2 and 0 by trio_cell.
template <int NT>
__global__ void __launch_bounds__(128, 5) pair_kernel(In in, Out out, Mats M, Params P, Queue Q, int parity) {
    const uint32_t n = *(volatile uint32_t *)(Q.count + 2 * parity + 1);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const Place at(Q.items[P.cells32 - 1u - i], P.nx, P.ny);
        pair_cell<NT>(in, out, M, P, at.l, at.m, at.k);
    }
}

// list 2: multi-solid interface cells.  Where there are far more of them than one-solid
// cells, a melt solidifies everywhere at once and its cells hold a phase of most grains:
// they go to any_cell instead of trio_cell in vain and then the octets (160 x 160 x 32 with
// 229 k of them 512 / 241 us a step, 128 x 128 x 64 with 500 grains and 205 k 243 / 205; with
// 50 k of them 75 / 85).  With a front, list 2 is at most 1.5 times as long as list 1.
constexpr uint32_t EVERYWHERE = 60000;
template <int S, int AMAX, int NT>
__global__ void __launch_bounds__(128, 4) trio_kernel(In in, Out out, Mats M, Params P, Queue Q, int parity,
                                                      int32_t *__restrict__ err) {
    wait_for_previous();
    // loads that are in flight together
    const uint32_t one = __ldcg(Q.count + 2 * parity + 1), several = __ldcg(Q.count + (Q.split ? 4 : 2) + parity);
    const uint32_t n = Q.split ? several : one;
    if (Q.split && several > EVERYWHERE && several / 8u > one) {
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
            const Place at(Q.items[P.cells32 + i], P.nx, P.ny);
            any_cell<S, AMAX, true, NT>(in, out, M, P, err, at.l, at.m, at.k);
        }
        return;
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t &item = Q.items[Q.split ? P.cells32 + i : P.cells32 - 1u - i];
        const uint32_t c = item;
        const Place at(c, P.nx, P.ny);
        if (!trio_cell<S, true, NT>(in, out, M, P, at.l, at.m, at.k)) item = c | LEFT;
    }
}

// list 0: grain boundaries and junctions, after trio_kernel on its stream
template <int S>
__global__ void __launch_bounds__(256, 4) general_kernel(In in, Out out, Mats M, Params P, Queue Q, int parity) {
    wait_for_previous();
    const uint32_t n = *(volatile uint32_t *)(Q.count + 2 * parity);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t c = Q.items[i];
        const Place at(c, P.nx, P.ny);
        if (!trio_cell<S, false, 4>(in, out, M, P, at.l, at.m, at.k)) Q.items[i] = c | LEFT;
    }
}

// what the two left
template <int S, int AMAX, int NT>
__global__ void __launch_bounds__(128, 8)
    rest_kernel(In in, Out out, Mats M, Params P, Queue Q, int parity, int32_t *__restrict__ err) {
    wait_for_previous();
    const OctetLane O;
    Lists L(Q, parity);
    if (Q.split) L.n[1] = 0;
    for_items<8, 32, false>(
        L.n[0] + L.n[1] + L.n[2], [&](uint32_t i) { return Q.items[L.item(i, P.cells32)]; },
        [](uint32_t c) { return (c & LEFT) == 0u; },
        [&](uint32_t marked, bool active) {
            const uint32_t c = marked & ~LEFT;
            const Place at(c, P.nx, P.ny);
            octet_cell<S, AMAX, NT>(in, out, M, P, err, O, active, at.l, at.m, at.k);
        },
        [](uint32_t) {});
}

// list 0 of the isotropic model, which has no other: what trio_cell leaves is
// done by the same block
template <int S, int AMAX>
__global__ void __launch_bounds__(256, 3)
    isotropic_kernel(In in, Out out, Mats M, Params P, Queue Q, int parity, int32_t *__restrict__ err) {
    wait_for_previous();
    const OctetLane O;
    for_items<32, 128, true>(
        *(volatile uint32_t *)(Q.count + 2 * parity), [&](uint32_t i) { return Q.items[i]; },
        [&](uint32_t c) {
            const Place at(c, P.nx, P.ny);
            return trio_cell<S, false, 4>(in, out, M, P, at.l, at.m, at.k);
        },
        [&](uint32_t c, bool active) {
            const Place at(c, P.nx, P.ny);
            octet_cell<S, AMAX, 4>(in, out, M, P, err, O, active, at.l, at.m, at.k);
        },
        [&](uint32_t c) {
            const Place at(c, P.nx, P.ny);
            any_cell<S, AMAX, false, 4>(in, out, M, P, err, at.l, at.m, at.k);
        });
}

// ---------------------------------------------------------------------------
// dense [N][nx][ny][nz] (z fastest) -> compact (x fastest)
template <typename T, int S>
__global__ void from_dense_kernel(const T *__restrict__ phi, int N, int nx, int ny, int nz, Out out,
                                  int32_t *__restrict__ err) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int m = blockIdx.y * blockDim.y + threadIdx.y;
    const int l = blockIdx.z * blockDim.z + threadIdx.z;
    if (k >= nz || m >= ny || l >= nx) return;
    const int64_t plane = (int64_t)nx * ny * nz;
    const int64_t src = ((int64_t)l * ny + m) * nz + k;
    const int64_t cells = plane;
    const int64_t dst = ((int64_t)k * ny + m) * nx + l;
    int c = 0, id0 = 0;
    float v0 = 0.0f;
    bool bad = false, ovf = false;
    for (int g = 0; g < N; ++g) {
        const T v = phi[(int64_t)g * plane + src];
        if (!(v >= (T)0)) { bad = true; continue; }
        if (v > (T)0) {
            if (c < S) {
                if (c == 0) { id0 = g; v0 = (float)v; }
                else out.idx[c * cells + dst] = (uint16_t)g;
                out.val[c * cells + dst] = (float)v;
            } else {
                ovf = true;
            }
            ++c;
        }
    }
    const int n = c < S ? c : S;
    out.head[dst] = mkhead(id0, n, n == 1 && v0 != 1.0f);
    if (bad) atomicOr(err, MPF3D_DEV_BAD_INPUT);
    if (ovf) atomicOr(err, MPF3D_DEV_SLOT_OVERFLOW);
}

// compact -> dense float32 [N][nx][ny][nz], four cells along z per thread, for nz a
// multiple of 4, aligned fields and the cases of by_four_cells.  Bound by the N planes
// it writes, to HBM or over the CPU-GPU link: each is written once, phase by phase beside
// the cells' ascending lists, 16 bytes per store, past the caches.  256^3 with 65 phases:
// 671 us (6.5 TB/s), with cached stores 727, by the kernel below 743.
template <int S>
__global__ void to_dense_kernel(In in, int N, int nx, int ny, int nz, uint32_t stride, uint32_t base,
                                float *__restrict__ phi) {
    constexpr int V = 4;
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    const int m = blockIdx.y * blockDim.y + threadIdx.y;
    const int l = blockIdx.z * blockDim.z + threadIdx.z;
    if (k >= nz || m >= ny || l >= nx) return;
    constexpr int NONE = 0x7fffffff;
    const int64_t plane = (int64_t)nx * ny * nz;
    uint32_t q[V];
    int left[V], id[V], next[V];  // entries beyond the next one; the current and the next entry
    float cur[V], val[V];
#pragma unroll
    for (int j = 0; j < V; ++j) {
        q[j] = base + ((uint32_t)(k + j) * (uint32_t)ny + (uint32_t)m) * (uint32_t)nx + (uint32_t)l;
        const uint32_t h = __ldg(in.head + q[j]);
        const int c = min(hcount(h), S);
        id[j] = c > 0 ? hid0(h) : NONE;
        cur[j] = value0(in, h, q[j]);
        next[j] = c > 1 ? (int)__ldg(in.idx + stride + q[j]) : NONE;
        val[j] = c > 1 ? __ldg(in.val + stride + q[j]) : 0.0f;
        left[j] = c - 2;
    }
    float *dst = phi + ((int64_t)l * ny + m) * nz + k;
    for (int g = 0; g < N; ++g, dst += plane) {
        float v[V];
        bool hit = false;
#pragma unroll
        for (int j = 0; j < V; ++j) {
            v[j] = id[j] == g ? cur[j] : 0.0f;
            hit = hit || id[j] == g;
        }
        __stcs((float4 *)dst, make_float4(v[0], v[1], v[2], v[3]));
        if (!hit) continue;
#pragma unroll
        for (int j = 0; j < V; ++j) {
            if (id[j] != g) continue;
            id[j] = next[j];
            cur[j] = val[j];
            next[j] = NONE;
            if (left[j] > 0) {
                const int64_t at = (int64_t)(min(hcount(__ldg(in.head + q[j])), S) - left[j]) * stride + q[j];
                next[j] = (int)__ldg(in.idx + at);
                val[j] = __ldg(in.val + at);
                --left[j];
            }
        }
    }
}

// One cell per thread, for the others: the planes zeroed, then the few stored phases
// written over them.
template <typename T, int S>
__global__ void to_dense_each_kernel(In in, int N, int nx, int ny, int nz, uint32_t stride, uint32_t base,
                                     T *__restrict__ phi) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int m = blockIdx.y * blockDim.y + threadIdx.y;
    const int l = blockIdx.z * blockDim.z + threadIdx.z;
    if (k >= nz || m >= ny || l >= nx) return;
    const int64_t plane = (int64_t)nx * ny * nz;
    const int64_t dstc = ((int64_t)l * ny + m) * nz + k;
    const uint32_t srcc = base + ((uint32_t)k * (uint32_t)ny + (uint32_t)m) * (uint32_t)nx + (uint32_t)l;
    for (int g = 0; g < N; ++g) phi[(int64_t)g * plane + dstc] = (T)0;
    const uint32_t h = in.head[srcc];
    const int c = min(hcount(h), S);
    for (int s = 0; s < c; ++s) {
        const int g = s == 0 ? hid0(h) : (int)in.idx[(size_t)s * stride + srcc];
        const float v = s == 0 ? value0(in, h, srcc) : in.val[(size_t)s * stride + srcc];
        if (g < N) phi[(int64_t)g * plane + dstc] = (T)v;
    }
}

// number of active phases per cell (the APT's nf), dense z-fastest output
template <int S>
__global__ void active_count_kernel(In in, int nx, int ny, int nz, int32_t *__restrict__ nf) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int m = blockIdx.y * blockDim.y + threadIdx.y;
    const int l = blockIdx.z * blockDim.z + threadIdx.z;
    if (k >= nz || m >= ny || l >= nx) return;
    nf[((int64_t)l * ny + m) * nz + k] = active_count_at<S>(in, nx, ny, nz, l, m, k);
}

// ---------------------------------------------------------------------------
// Batches of independent domains ("instances") sharing one set of state
// arrays: instance i owns cells [offset, offset + nx*ny*nz) of every array.
// One launch of each step kernel covers all instances; tiles and queued
// cells find their instance by binary search over the instance table.

__device__ __forceinline__ int find_instance_by_tile(const mpf3d_instance *__restrict__ inst, int n, int tile) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&inst[mid].tile_start) <= tile) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ int find_instance_by_cell(const mpf3d_instance *__restrict__ inst, int n, uint32_t c) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&inst[mid].offset) <= c) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ Params instance_params(const Params &P0, const mpf3d_instance &I) {
    Params P = P0;
    P.nx = I.nx; P.ny = I.ny; P.nz = I.nz;
    P.base = I.offset;
    P.n111_base = I.n111_base;
    P.delta_a = I.delta_a;
    P.mu_da = I.mu_da;
    P.e2_flat = I.e2_flat;
    P.t_uniform = 1;
    P.dT_uniform = -I.undercooling;
    return P;
}

// The batched sweep.  An instance is cut into tiles of 32 x 8 x SWEEP_ZB cells
// (tile_start) and each of those into 8 warp tiles of 32 x 1 x SWEEP_ZB, numbered
// 8 * tile + row.  With `flags` (2 x 8 x n_tiles bytes, halves alternating with
// the step parity; NULL: every tile visited) a warp tile that was uniform in the
// previous step together with its 6 face neighbours in the same instance
// (periodic x and y, clamped z) is quiet and skipped, by the argument of the
// single-domain sweep's quiet tiles.
struct WarpTile {
    int tile_start, tx, ty, tz, bx, m, kb;
    __device__ __forceinline__ WarpTile(const mpf3d_instance &I, uint32_t tile, uint32_t row) {
        tile_start = I.tile_start;
        tx = (I.nx + 31) / 32, ty = (I.ny + 7) / 8, tz = (I.nz + SWEEP_ZB - 1) / SWEEP_ZB;
        const int t = (int)tile - tile_start, q = t / tx;
        bx = t - q * tx, kb = q / ty, m = (q - kb * ty) * 8 + (int)row;
    }
    // the number of (x tile, row, z tile) in this instance
    __device__ __forceinline__ uint32_t at(int a, int mm, int c) const {
        return (uint32_t)(tile_start + (c * ty + mm / 8) * tx + a) * 8u + (uint32_t)(mm % 8);
    }
};

__global__ void __launch_bounds__(256, 8) batched_sweep_kernel(In in, Out out, Params P0,
                                                               const mpf3d_instance *__restrict__ inst, int n_inst,
                                                               Queue Q, int parity, uint8_t *__restrict__ flags,
                                                               uint32_t n_tiles) {
    wait_for_previous();
    if (blockIdx.x == 0) clear_counters(Q, parity, threadIdx.x + 32u * threadIdx.y);
    const uint8_t *fin = flags + (size_t)(parity ^ 1) * 8 * n_tiles;
    uint8_t *fout = flags ? flags + (size_t)parity * 8 * n_tiles : nullptr;
    sweep_tiles<SWEEP_ZB>(
        Q, P0.cells32, parity, n_tiles, fout,
        [&](uint32_t tile, uint32_t) { return find_instance_by_tile(inst, n_inst, (int)tile); },
        [](uint32_t tile, uint32_t row) { return tile * 8u + row; },
        [&](int i, uint32_t tile, uint32_t row) {
            if (!flags) return false;
            const mpf3d_instance &I = inst[i];
            const WarpTile t(I, tile, row);
            const int bx = t.bx, m = t.m, kb = t.kb;
            if (m >= I.ny) return true;  // a row past the instance's top: its flag has a place of its own
            // the 7 flags are loaded together (no short-circuit chain of loads)
            const uint32_t f0 = fin[tile * 8u + row];
            const uint32_t f1 = fin[t.at(bx + 1 < t.tx ? bx + 1 : 0, m, kb)];
            const uint32_t f2 = fin[t.at(bx > 0 ? bx - 1 : t.tx - 1, m, kb)];
            const uint32_t f3 = fin[t.at(bx, m + 1 < I.ny ? m + 1 : 0, kb)];
            const uint32_t f4 = fin[t.at(bx, m > 0 ? m - 1 : I.ny - 1, kb)];
            const uint32_t f5 = fin[t.at(bx, m, kb + 1 < t.tz ? kb + 1 : kb)];
            const uint32_t f6 = fin[t.at(bx, m, kb > 0 ? kb - 1 : kb)];
            return (f0 & f1 & f2 & f3 & f4 & f5 & f6) != 0u;
        },
        [&](int i, uint32_t tile, uint32_t row, BlockSink<SWEEP_ZB> &sink) {
            const mpf3d_instance I = inst[i];
            const WarpTile t(I, tile, row);
            const Params P = instance_params(P0, I);
            const uint32_t plane = (uint32_t)I.nx * (uint32_t)I.ny;
            const int l = t.bx * 32 + (int)threadIdx.x, k0 = t.kb * SWEEP_ZB;
            sink.add(l < I.nx && t.m < I.ny ? sweep_column(in, out, P, Q.split, l, t.m, k0) : 0u,
                     P.base + (uint32_t)k0 * plane + (uint32_t)t.m * (uint32_t)I.nx + (uint32_t)l, plane);
        });
}

// The work-list kernels of a batch: as the single domain's, on the instance of
// each cell.
template <int S, int AMAX, int NT>
__global__ void __launch_bounds__(128, OCTET_BLOCKS) batched_octet_kernel(In in, Out out, Mats M, Params P0,
                                                               const mpf3d_instance *__restrict__ inst, int n_inst,
                                                               Queue Q, int parity, int32_t *__restrict__ err) {
    wait_for_previous();
    const OctetLane O;
    for_octets(Q, P0.cells32, parity, [&](uint32_t c, bool active) {
        const mpf3d_instance I = inst[find_instance_by_cell(inst, n_inst, c)];
        const Place at(c - I.offset, I.nx, I.ny);
        octet_cell<S, AMAX, NT>(in, out, M, instance_params(P0, I), err, O, active, at.l, at.m, at.k);
    }, [&](uint32_t c, bool general) {
        const mpf3d_instance I = inst[find_instance_by_cell(inst, n_inst, c)];
        const Place at(c - I.offset, I.nx, I.ny);
        const Params P = instance_params(P0, I);
        if (!general || !trio_cell<S, false, 4>(in, out, M, P, at.l, at.m, at.k))
            any_cell<S, AMAX, true, NT>(in, out, M, P, err, at.l, at.m, at.k);
    });
}

template <int NT>
__global__ void __launch_bounds__(128, 5) batched_pair_kernel(In in, Out out, Mats M, Params P0,
                                                              const mpf3d_instance *__restrict__ inst, int n_inst,
                                                              Queue Q, int parity) {
    wait_for_previous();
    const uint32_t n = *(volatile uint32_t *)(Q.count + 2 * parity + 1);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t c = Q.items[P0.cells32 - 1u - i];
        const mpf3d_instance I = inst[find_instance_by_cell(inst, n_inst, c)];
        const Place at(c - I.offset, I.nx, I.ny);
        pair_cell<NT>(in, out, M, instance_params(P0, I), at.l, at.m, at.k);
    }
}

// list 2: multi-solid interface cells
template <int S, int NT>
__global__ void __launch_bounds__(128, 4) batched_trio_kernel(In in, Out out, Mats M, Params P0, const mpf3d_instance *__restrict__ inst, int n_inst, Queue Q, int parity) {
    wait_for_previous();  // two grains and the liquid: trio_cell takes every cell of a batch's bicrystals
    const uint32_t n = *(volatile uint32_t *)(Q.count + (Q.split ? 4 + parity : 2 * parity + 1));
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t &item = Q.items[Q.split ? P0.cells32 + i : P0.cells32 - 1u - i];
        const uint32_t c = item;
        const mpf3d_instance I = inst[find_instance_by_cell(inst, n_inst, c)];
        const Place at(c - I.offset, I.nx, I.ny);
        if (!trio_cell<S, true, NT>(in, out, M, instance_params(P0, I), at.l, at.m, at.k)) item = c | LEFT;
    }
}

// list 0: grain boundaries and junctions
template <int S>
__global__ void __launch_bounds__(256, 4) batched_general_kernel(In in, Out out, Mats M, Params P0, const mpf3d_instance *__restrict__ inst, int n_inst, Queue Q, int parity) {
    wait_for_previous();
    const uint32_t n = *(volatile uint32_t *)(Q.count + 2 * parity);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t c = Q.items[i];
        const mpf3d_instance I = inst[find_instance_by_cell(inst, n_inst, c)];
        const Place at(c - I.offset, I.nx, I.ny);
        if (!trio_cell<S, false, 4>(in, out, M, instance_params(P0, I), at.l, at.m, at.k)) Q.items[i] = c | LEFT;
    }
}

// what the two left
template <int S, int AMAX, int NT>
__global__ void __launch_bounds__(128, 8)
    batched_rest_kernel(In in, Out out, Mats M, Params P0, const mpf3d_instance *__restrict__ inst, int n_inst, Queue Q, int parity, int32_t *__restrict__ err) {
    wait_for_previous();
    const OctetLane O;
    Lists L(Q, parity);
    if (Q.split) L.n[1] = 0;
    for_items<8, 32, false>(
        L.n[0] + L.n[1] + L.n[2], [&](uint32_t i) { return Q.items[L.item(i, P0.cells32)]; },
        [](uint32_t c) { return (c & LEFT) == 0u; },
        [&](uint32_t marked, bool active) {
            const uint32_t c = marked & ~LEFT;
            const mpf3d_instance I = inst[find_instance_by_cell(inst, n_inst, c)];
            const Place at(c - I.offset, I.nx, I.ny);
            octet_cell<S, AMAX, NT>(in, out, M, instance_params(P0, I), err, O, active, at.l, at.m, at.k);
        },
        [](uint32_t) {});
}

// list 0 of the isotropic model, which has no other: what trio_cell leaves is
// done by the same block
template <int S, int AMAX>
__global__ void __launch_bounds__(256, 3)
    batched_isotropic_kernel(In in, Out out, Mats M, Params P0, const mpf3d_instance *__restrict__ inst, int n_inst, Queue Q, int parity, int32_t *__restrict__ err) {
    wait_for_previous();
    const OctetLane O;
    for_items<32, 128, true>(
        *(volatile uint32_t *)(Q.count + 2 * parity), [&](uint32_t i) { return Q.items[i]; },
        [&](uint32_t c) {
            const mpf3d_instance I = inst[find_instance_by_cell(inst, n_inst, c)];
            const Place at(c - I.offset, I.nx, I.ny);
            return trio_cell<S, false, 4>(in, out, M, instance_params(P0, I), at.l, at.m, at.k);
        },
        [&](uint32_t c, bool active) {
            const mpf3d_instance I = inst[find_instance_by_cell(inst, n_inst, c)];
            const Place at(c - I.offset, I.nx, I.ny);
            octet_cell<S, AMAX, 4>(in, out, M, instance_params(P0, I), err, O, active, at.l, at.m, at.k);
        },
        [&](uint32_t c) {
            const mpf3d_instance I = inst[find_instance_by_cell(inst, n_inst, c)];
            const Place at(c - I.offset, I.nx, I.ny);
            any_cell<S, AMAX, false, 4>(in, out, M, instance_params(P0, I), err, at.l, at.m, at.k);
        });
}

// Initial bicrystal: a solid base of height base_height (tanh profile
// 0.5*(1 - tanh(2.2/delta*(k - h)*dz)), as src/seed_modes_3d.py:46-56), grain
// 1 for x < split and grain 2 for x >= split, liquid = clip(1 - solid).
__global__ void batched_init_bicrystal_kernel(Out out, const mpf3d_instance *__restrict__ inst, int n_inst,
                                              uint32_t stride, float factor_dz, int32_t *__restrict__ err) {
    const int i = blockIdx.y;
    if (i >= n_inst) return;
    const mpf3d_instance I = inst[i];
    const uint32_t cells = (uint32_t)I.nx * I.ny * I.nz;
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < cells; r += gridDim.x * blockDim.x) {
        const uint32_t plane = (uint32_t)I.nx * I.ny;
        const int k = (int)(r / plane);
        const int l = (int)((r - (uint32_t)k * plane) % (uint32_t)I.nx);
        const float s = (float)(0.5 * (1.0 - tanh((double)factor_dz * ((double)k - (double)I.base_height))));
        const float liq = fminf(fmaxf(1.0f - s, 0.0f), 1.0f);
        const int g = l < I.split ? 1 : 2;
        const uint32_t c = I.offset + r;
        int n = 0, id0 = 0;
        float v0 = 0.0f;
        if (liq > 0.0f) { id0 = LIQ; v0 = liq; out.val[c] = liq; n = 1; }
        if (s > 0.0f) {
            if (n == 0) { id0 = g; v0 = s; out.val[c] = s; }
            else { out.idx[(size_t)stride + c] = (uint16_t)g; out.val[(size_t)stride + c] = s; }
            ++n;
        }
        out.head[c] = mkhead(id0, n, n == 1 && v0 != 1.0f);
    }
}

// Per instance: mean front height of each grain half (highest z with solid
// fraction > 0.5 per column, interface_positions_3d of
// tests/verification_3d.py:409-416) and the total fraction of grains 1, 2.
// acc[6*i + ...] = {sum h left, columns left, sum h right, columns right, V1, V2}
template <int S>
__global__ void batched_fronts_kernel(In in, const mpf3d_instance *__restrict__ inst, int n_inst, uint32_t stride,
                                      double *__restrict__ acc) {
    const int i = blockIdx.y;
    const mpf3d_instance I = inst[i];
    const int cols = I.nx * I.ny;
    const uint32_t plane = (uint32_t)cols;
    double hl = 0.0, nl = 0.0, hr = 0.0, nr = 0.0, v1 = 0.0, v2 = 0.0;
    for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < cols; col += gridDim.x * blockDim.x) {
        const int l = col % I.nx;
        int front = -1;
        for (int k = I.nz - 1; k >= 0; --k) {
            const uint32_t c = I.offset + (uint32_t)k * plane + (uint32_t)col;
            const float solid = 1.0f - phase_at<S>(in, stride, c, LIQ);
            if (front < 0 && solid > 0.5f) front = k;
            v1 += phase_at<S>(in, stride, c, 1);
            v2 += phase_at<S>(in, stride, c, 2);
        }
        if (front >= 0) {
            if (l < I.split) { hl += front; nl += 1.0; }
            else { hr += front; nr += 1.0; }
        }
    }
    double vals[6] = {hl, nl, hr, nr, v1, v2};
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        double v = vals[q];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) atomicAdd(acc + 6 * i + q, v);
    }
}

// Per instance and z row: the phi1 = phi2 crossing along x nearest the
// initial split, averaged over y, for rows whose solid fraction is >= 0.15
// (the grain-boundary locator of measure_gb_inclination,
// tests/run_paper_verification.py:658-723, with a linear root between the
// two cells of the sign change).  gb[2*(row_base + k) + {0,1}] = {sum x, rows}.
template <int S>
__global__ void batched_gb_rows_kernel(In in, const mpf3d_instance *__restrict__ inst, int n_inst, uint32_t stride,
                                       const int *__restrict__ row_base, double *__restrict__ gb) {
    const int i = blockIdx.y;
    const mpf3d_instance I = inst[i];
    const int rows = I.ny * I.nz;
    const uint32_t plane = (uint32_t)I.nx * I.ny;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        const int m = r % I.ny, k = r / I.ny;
        const uint32_t row0 = I.offset + (uint32_t)k * plane + (uint32_t)m * I.nx;
        float solid = 0.0f, best_x = 0.0f, best_d = 1e30f;
        bool found = false;
        float dprev = phase_at<S>(in, stride, row0, 1) - phase_at<S>(in, stride, row0, 2);
        solid += 1.0f - phase_at<S>(in, stride, row0, LIQ);
        for (int l = 1; l < I.nx; ++l) {
            const uint32_t c = row0 + (uint32_t)l;
            const float d = phase_at<S>(in, stride, c, 1) - phase_at<S>(in, stride, c, 2);
            solid += 1.0f - phase_at<S>(in, stride, c, LIQ);
            if ((dprev > 0.0f && d <= 0.0f) || (dprev < 0.0f && d >= 0.0f)) {
                const float x = (float)(l - 1) + dprev / (dprev - d);
                const float dist = fabsf(x - (float)I.split);
                if (dist < best_d) { best_d = dist; best_x = x; found = true; }
            }
            dprev = d;
        }
        if (found && solid >= 0.15f * I.nx) {
            atomicAdd(gb + 2 * (row_base[i] + k), (double)best_x);
            atomicAdd(gb + 2 * (row_base[i] + k) + 1, 1.0);
        }
    }
}


// Initial state from a grain-owner map and a z profile: owner[k][m][l]
// (x fastest) holds the grain of the first `slab` layers; rows above the slab
// repeat the top layer.  The grain holds prof[k], the liquid
// clip(1 - prof[k], 0, 1) (init_phi_from_grain_map_3d,
// src/seed_modes_3d.py:38-57, with a 3-D owner map).
__global__ void init_owner_kernel(Out out, const int32_t *__restrict__ owner, int slab, const float *__restrict__ prof,
                                  int nx, int ny, int nz, uint32_t cells) {
    const uint32_t plane = (uint32_t)nx * (uint32_t)ny;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < cells; c += gridDim.x * blockDim.x) {
        const int k = (int)(c / plane);
        const uint32_t col = c - (uint32_t)k * plane;
        const int g = owner[(uint32_t)min(k, slab - 1) * plane + col];
        const float s = prof[k];
        const float liq = fminf(fmaxf(1.0f - s, 0.0f), 1.0f);
        int n = 0, id0 = 0;
        float v0 = 0.0f;
        if (liq > 0.0f) { id0 = LIQ; v0 = liq; out.val[c] = liq; n = 1; }
        if (s > 0.0f) {
            if (n == 0) { id0 = g; v0 = s; out.val[c] = s; }
            else { out.idx[(size_t)cells + c] = (uint16_t)g; out.val[(size_t)cells + c] = s; }
            ++n;
        }
        out.head[c] = mkhead(id0, n, n == 1 && v0 != 1.0f);
    }
}

}  // namespace compact
}  // namespace mpf3d

using namespace mpf3d;
using namespace mpf3d::compact;

namespace {

dim3 zfast_grid(int nx, int ny, int nz, dim3 b) {
    return dim3((nz + b.x - 1) / b.x, (ny + b.y - 1) / b.y, (nx + b.z - 1) / b.z);
}


// Whether to_dense_kernel writes a float32 field, four cells a thread.  Over the CPU-GPU
// link its wide stores win at every size (us, a cell / four cells a thread: 32^3 with 9
// phases 15 / 13, 512 x 512 x 8 with 9 736 / 435, 128^3 with 33 1500 / 1436).  In device memory
// it wants many planes and whole rows of threads along z (32^3 with 9 phases 6.8 / 8.8, 512 x
// 512 x 8 with 9 58 / 64, 128 x 128 x 64 with 33 31 / 36, 64^3 with 301 62 / 58, 128^3 with 33
// 52 / 49).  Float64 is not for it: a warp's stores of four cells leave gaps (128^3 with 33 in
// device memory 93 / 163, over the link 2975 / 7211).
bool by_four_cells(int64_t values, int nz, const void *phi) {
    cudaPointerAttributes at{};
    const bool known = cudaPointerGetAttributes(&at, phi) == cudaSuccess;
    if (!known) cudaGetLastError();
    if (known && at.type == cudaMemoryTypeHost) return true;
    return values >= (int64_t)1 << 26 && nz >= 64;
}

template <typename T, int S>
void launch_to_dense(const In &in, int N, int nx, int ny, int nz, uint32_t stride, uint32_t base, T *phi,
                     cudaStream_t s) {
    const dim3 b(16, 4, 4), each(32, 4, 2);
    if (sizeof(T) == 4 && nz % 4 == 0 && (uintptr_t)phi % 16 == 0 && by_four_cells((int64_t)nx * ny * nz * N, nz, phi))
        to_dense_kernel<S><<<zfast_grid(nx, ny, nz / 4, b), b, 0, s>>>(in, N, nx, ny, nz, stride, base, (float *)phi);
    else
        to_dense_each_kernel<T, S><<<zfast_grid(nx, ny, nz, each), each, 0, s>>>(in, N, nx, ny, nz, stride, base, phi);
}

int to_dense(const In &in, int slots, int N, int nx, int ny, int nz, uint32_t stride, uint32_t base, void *phi,
             int phi_dtype, cudaStream_t s) {
#define TD(T)                                                                                              \
    do {                                                                                                   \
        if (slots == 4) launch_to_dense<T, 4>(in, N, nx, ny, nz, stride, base, (T *)phi, s);               \
        else if (slots == 8) launch_to_dense<T, 8>(in, N, nx, ny, nz, stride, base, (T *)phi, s);          \
        else if (slots == 16) launch_to_dense<T, 16>(in, N, nx, ny, nz, stride, base, (T *)phi, s);        \
        else return MPF3D_ERR_ARG;                                                                         \
    } while (0)
    if (phi_dtype == MPF3D_F32) TD(float);
    else if (phi_dtype == MPF3D_F64) TD(double);
    else return MPF3D_ERR_DTYPE;
#undef TD
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}

// A second stream of one device, on which pair_kernel runs beside trio_kernel and then
// general_kernel on the caller's.  They read only what the sweep wrote and write disjoint
// cells, and fill each other's idle issue slots.  Created on first use outside a
// stream capture; the fork/join is enqueued under the mutex so that callers
// on other host threads cannot interleave their event records with it.
// The second stream of a step and its fork/join events, one set per
// (device, caller stream): steps that callers issue on independent streams
// stay independent of each other.
struct SideStream {
    bool ready = false;
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};

struct SideTable {
    std::mutex mu;
    std::unordered_map<cudaStream_t, SideStream> by_caller;  // element references survive rehashing
};

SideTable &side_table_of(int dev) {
    static SideTable all[64];
    return all[dev & 63];
}

// Creates the side stream and its events once, outside any capture of s.
bool side_ready(SideStream &side, cudaStream_t s) {
    if (!side.ready) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone &&
            cudaStreamCreateWithFlags(&side.stream, cudaStreamNonBlocking) == cudaSuccess &&
            cudaEventCreateWithFlags(&side.fork, cudaEventDisableTiming) == cudaSuccess &&
            cudaEventCreateWithFlags(&side.join, cudaEventDisableTiming) == cudaSuccess)
            side.ready = true;
    }
    return side.ready;
}

// Blocks of the sweep of `chunks` chunks of `rows` tiles, a warp per row, 48 warps
// resident per SM: a block per chunk up to SWEEP_WAVES waves of blocks, then up to
// SWEEP_TILES tiles per block.  (256^3: 23.5 us with 1 wave, 22.7 with 4, 28.4 with
// 8.)
constexpr uint32_t SWEEP_WAVES = 4;
uint32_t sweep_blocks(uint32_t chunks, int rows, int sms) {
    const uint32_t each = chunks / (SWEEP_WAVES * (uint32_t)sms * 48u / (uint32_t)rows);
    const uint32_t n = min(max(each, 1u), SWEEP_TILES / (uint32_t)rows);
    return (chunks + n - 1u) / n;
}

// Whether a step's lists go to the kernels by kind of cell (isotropic_kernel, or
// pair_kernel, trio_kernel, general_kernel and rest_kernel) or all to octet_kernel,
// which takes short lists by octets and long ones by threads.  Five kernels a step pay
// where many cells are listed, which the host does not know: it follows the size.  us a
// step, octet_kernel / by kind, after 20, 200 and 1000 steps: 80 x 80 x 80 33 / 40, 34 /
// 41, 47 / 48; 300 x 60 x 28 45 / 47, 47 / 50, 62 / 61; 160 x 160 x 32 46 / 49, 49 / 52,
// 68 / 66; 150 x 117 x 90 45 / 47, 47 / 50, 68 / 61; 128 x 128 x 128 46 / 49, 50 / 52, 69 /
// 63.  Batches of 32 x 32 x 64, after 20 and 800 steps: 3 of them 23 / 36, 16 / 39, 12 of
// them 39 / 44, 34 / 42.  Isotropic, one kernel either way, 10 steps with dense output: 45 x
// 45 x 90 361 / 344, 64 x 64 x 64 425 / 356; a batch of 4 335 / 207.
constexpr int64_t KIND_CELLS = 7 << 17, KIND_CELLS_ISOTROPIC = 1 << 19, KIND_PLANE_ISOTROPIC = 2000,
                  KIND_CELLS_BATCH = 1 << 20;
bool by_kind(const Params &P) {
    return P.use_aniso ? P.cells >= KIND_CELLS
                       : P.cells >= KIND_CELLS_ISOTROPIC || (int64_t)P.nx * P.ny >= KIND_PLANE_ISOTROPIC;
}
bool by_kind_batch(const Params &P) { return P.cells >= KIND_CELLS_BATCH || !P.use_aniso; }

// general(stream) and interface(stream) launch the work-list kernels of a step;
// interface's go to the caller stream's side stream, forked from s after the
// sweep and joined back before s continues.
template <class General, class Interface>
void launch_side_by_side(cudaStream_t s, General &&general, Interface &&interface) {
    int dev = 0;
    cudaGetDevice(&dev);
    SideTable &tab = side_table_of(dev);
    std::lock_guard<std::mutex> lock(tab.mu);
    SideStream &side = tab.by_caller[s];
    if (!side_ready(side, s)) {  // first call inside a capture: both kernels on the caller's stream
        general(s);
        interface(s);
        return;
    }
    cudaEventRecord(side.fork, s);
    cudaStreamWaitEvent(side.stream, side.fork, 0);
    interface(side.stream);
    general(s);
    cudaEventRecord(side.join, side.stream);
    cudaStreamWaitEvent(s, side.join, 0);  // the caller's stream sees the whole step
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// dependency on libcuda)
PFN_cuTensorMapEncodeTiled_v12000 encode_tiled() {
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// Tensor map of a head array (uint32 nx x ny x nz, x fastest) with boxes of
// TMA_X x (by + 2) x (zb + 2); out-of-range elements read as zero.  Needs
// nx a multiple of 4 (16-byte row pitch) and a 16-byte aligned base.
bool head_map(CUtensorMap *map, const uint32_t *head, int nx, int ny, int nz, int by, int zb) {
    PFN_cuTensorMapEncodeTiled_v12000 fn = encode_tiled();
    if (!fn || nx % 4 != 0 || ((uintptr_t)head & 15u) != 0) return false;
    cuuint64_t dims[3] = {(cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz};
    cuuint64_t strides[2] = {(cuuint64_t)nx * 4, (cuuint64_t)nx * ny * 4};
    cuuint32_t box[3] = {(cuuint32_t)TMA_X, (cuuint32_t)(by + 2), (cuuint32_t)(zb + 2)};
    cuuint32_t estr[3] = {1u, 1u, 1u};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<uint32_t *>(head), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Launch of a kernel that begins with wait_for_previous, without waiting for the
// kernel before it in the stream to drain.
template <class... K, class... A>
void launch_early(void (*kernel)(K...), unsigned grid, dim3 block, cudaStream_t s, A &&...args) {
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = block;
    cfg.stream = s;
    cfg.attrs = &early;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

template <int S, int AMAX>
void launch_step(const In &in, const Out &out, const Mats &M, const Params &P, const Queue &Q, int parity,
                 uint8_t *tile_flags, int32_t *err, cudaStream_t s, const mpf3d_tuning &T, bool sweep_tma) {
    const int by = T.sweep_by, sms = sms_of_current_device();
    dim3 blk(32, by, 1);
    CUtensorMap map;
    const bool tma = sweep_tma && P.base == 0 && head_map(&map, in.head, P.nx, P.ny, P.nz, by, T.sweep_zb);
#define SWEEP_LAUNCH(ZB)                                                                                           \
    do {                                                                                                           \
        const dim3 grid((P.nx + 31) / 32, (P.ny + by - 1) / by, (P.nz + ZB - 1) / ZB);                             \
        const Tiles tl{tile_flags, (P.nx + 31) / 32, (P.nz + ZB - 1) / ZB, tiles_of<ZB>(P.nx, P.ny, P.nz)};       \
        if (tma) sweep_kernel_tma<ZB><<<grid, blk, 0, s>>>(map, in, out, P, Q, parity, tl, err);          \
        else {                                                                                                     \
            const uint32_t chunks = grid.x * grid.y * grid.z;                                                      \
            launch_early(sweep_kernel<ZB>, sweep_blocks(chunks, by, sms), blk, s, in, out, P, Q, parity, tl,       \
                         chunks);                                                                                  \
        }                                                                                                          \
    } while (0)
    if (T.sweep_zb == 2) SWEEP_LAUNCH(2);
    else if (T.sweep_zb == 8) SWEEP_LAUNCH(8);
    else SWEEP_LAUNCH(4);
#undef SWEEP_LAUNCH
    if (!by_kind(P)) {
        launch_early(P.sym_normals ? octet_kernel<S, AMAX, 4> : octet_kernel<S, AMAX, 8>, sms * OCTET_BLOCKS, dim3(128), s, in,
                     out, M, P, Q, parity, err);
        return;
    }
    const int g_general = sms * T.general_blocks_per_sm, g_iface = sms * T.iface_blocks_per_sm;
    if (!P.use_aniso) {
        launch_early(isotropic_kernel<S, AMAX>, g_general, dim3(T.general_threads), s, in, out, M, P, Q, parity, err);
        return;
    }
    launch_side_by_side(
        s,
        [&](cudaStream_t st) {
            launch_early(P.sym_normals ? trio_kernel<S, AMAX, 4> : trio_kernel<S, AMAX, 8>, g_iface, dim3(T.iface_threads),
                         st, in, out, M, P, Q, parity, err);
            launch_early(general_kernel<S>, g_general, dim3(T.general_threads), st, in, out, M, P, Q, parity);
        },
        [&](cudaStream_t st) {
            if (!Q.split) return;
            if (P.sym_normals) pair_kernel<4><<<g_iface, T.iface_threads, 0, st>>>(in, out, M, P, Q, parity);
            else pair_kernel<8><<<g_iface, T.iface_threads, 0, st>>>(in, out, M, P, Q, parity);
        });
    if (P.sym_normals) rest_kernel<S, AMAX, 4><<<sms * 8, 128, 0, s>>>(in, out, M, P, Q, parity, err);
    else rest_kernel<S, AMAX, 8><<<sms * 8, 128, 0, s>>>(in, out, M, P, Q, parity, err);
}

bool tuning_ok(const mpf3d_tuning &T) {
    return (T.sweep_zb == 2 || T.sweep_zb == 4 || T.sweep_zb == 8) &&
           (T.sweep_by == 4 || T.sweep_by == 8 || T.sweep_by == 16) && T.general_blocks_per_sm >= 1 &&
           T.general_blocks_per_sm <= 64 && (T.general_threads == 128 || T.general_threads == 256) &&
           T.iface_blocks_per_sm >= 1 && T.iface_blocks_per_sm <= 64 &&
           (T.iface_threads == 64 || T.iface_threads == 128);
}

// Launch shape of a step (single or batched) without mpf3d_tuning: blocks of 128 threads, all of
// them resident in one or two waves.  (us per step at 256^3 / 512 x 512 x 256 /
// 128^3 with general and interface grids of 16 x 128 threads per SM: 147 / 343 /
// 57; with 8 x 256 and 64 x 64: 153 / 347 / 60; with 8 x 256 and 8 x 128: 148 /
// 349 / 58.)
constexpr mpf3d_tuning DEFAULT_TUNING = {4, 8, 16, 128, 16, 128};

}  // namespace

extern "C" int mpf3d_compact_from_dense(const void *phi, int phi_dtype, int N, int nx, int ny, int nz, int slots,
                                        uint32_t *cnt, uint16_t *idx, float *val, int32_t *err, void *stream) {
    if (!phi || !cnt || !idx || !val || !err || N <= 0 || N > 65535 || !dims_ok(nx, ny, nz)) return MPF3D_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    dim3 b(32, 4, 2);
    dim3 g = zfast_grid(nx, ny, nz, b);
    Out o{cnt, idx, val};
#define FD(T, SS) from_dense_kernel<T, SS><<<g, b, 0, s>>>((const T *)phi, N, nx, ny, nz, o, err)
    if (phi_dtype == MPF3D_F32) {
        if (slots == 4) FD(float, 4); else if (slots == 8) FD(float, 8); else if (slots == 16) FD(float, 16);
        else return MPF3D_ERR_ARG;
    } else if (phi_dtype == MPF3D_F64) {
        if (slots == 4) FD(double, 4); else if (slots == 8) FD(double, 8); else if (slots == 16) FD(double, 16);
        else return MPF3D_ERR_ARG;
    } else {
        return MPF3D_ERR_DTYPE;
    }
#undef FD
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}

extern "C" int mpf3d_compact_to_dense(const uint32_t *cnt, const uint16_t *idx, const float *val, int slots, int N,
                                      int nx, int ny, int nz, void *phi, int phi_dtype, void *stream) {
    if (!phi || !cnt || !idx || !val || N <= 0 || N > 65535 || !dims_ok(nx, ny, nz)) return MPF3D_ERR_ARG;
    return to_dense({cnt, idx, val}, slots, N, nx, ny, nz, (uint32_t)((int64_t)nx * ny * nz), 0u, phi, phi_dtype,
                    (cudaStream_t)stream);
}

extern "C" int mpf3d_host_device_pointer(const void *host, void **device) {
    if (!host || !device) return MPF3D_ERR_ARG;
    *device = nullptr;
    void *d = nullptr;
    if (cudaHostGetDevicePointer(&d, const_cast<void *>(host), 0) != cudaSuccess) {
        cudaGetLastError();  // not page-locked host memory: clear the error, report it
        return MPF3D_ERR_ARG;
    }
    *device = d;
    return MPF3D_OK;
}

extern "C" int mpf3d_compact_active_count(const uint32_t *cnt, const uint16_t *idx, int slots, int nx, int ny, int nz,
                                          int32_t *nf, void *stream) {
    if (!cnt || !idx || !nf || !dims_ok(nx, ny, nz)) return MPF3D_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    dim3 b(32, 4, 2);
    dim3 g = zfast_grid(nx, ny, nz, b);
    In in{cnt, idx, nullptr};
    if (slots == 4) active_count_kernel<4><<<g, b, 0, s>>>(in, nx, ny, nz, nf);
    else if (slots == 8) active_count_kernel<8><<<g, b, 0, s>>>(in, nx, ny, nz, nf);
    else if (slots == 16) active_count_kernel<16><<<g, b, 0, s>>>(in, nx, ny, nz, nf);
    else return MPF3D_ERR_ARG;
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}

namespace {

// physics shared by every cell of a step, from the 13 kernel scalars
Params shared_params(const mpf3d_scalars *sc, int enable_anisotropy, int enable_torque, int symmetric_normals) {
    const double *v = sc->v;
    Params P;
    memset(&P, 0, sizeof P);
    const double dx = v[MPF3D_S_DX];
    P.inv_dx2 = (float)(1.0 / (dx * dx));
    P.inv_2dx = (float)(1.0 / (2.0 * dx));
    P.half_over_dx = (float)(0.5 / dx);
    P.inv_dx = (float)(1.0 / dx);
    P.dt = (float)v[MPF3D_S_DT];
    P.eps0 = (float)v[MPF3D_S_EPS0_SL];
    P.eps0sq = (float)(v[MPF3D_S_EPS0_SL] * v[MPF3D_S_EPS0_SL]);
    P.w0 = (float)v[MPF3D_S_W0_SL];
    P.mu_a = (float)v[MPF3D_S_MU_A];
    P.delta_a = (float)v[MPF3D_S_DELTA_A];
    P.mu_da = (float)(v[MPF3D_S_MU_A] * v[MPF3D_S_DELTA_A]);
    P.pp = (float)(v[MPF3D_S_P_ROUND] * v[MPF3D_S_P_ROUND]);
    P.tan_a0 = (float)tan(v[MPF3D_S_A0]);
    P.g2_floor = (float)v[MPF3D_S_G2_FLOOR];
    P.ksi = (float)v[MPF3D_S_KSI];
    P.theta_c = (float)v[MPF3D_S_THETA_C_RAD];
    // below this best |cos| the facet angle is >= theta_c with a margin far
    // above the FP32 error of c (~1e-7), so b = 1 without computing the angle
    P.cos_theta_lo = (float)(cos(v[MPF3D_S_THETA_C_RAD]) - 1.0e-5);
    P.Sf = (float)v[MPF3D_S_SF];
    P.Tmc = v[MPF3D_S_T_MELT];
    P.use_aniso = enable_anisotropy != 0;
    P.use_torque = enable_anisotropy != 0 && enable_torque != 0;
    P.sym_normals = symmetric_normals != 0;
    const double pp = v[MPF3D_S_P_ROUND] * v[MPF3D_S_P_ROUND];
    const double th = acos(0.0), thc = v[MPF3D_S_THETA_C_RAD];
    double b = 1.0;
    if (th < thc) {
        double y = 0.5 * 3.14159265358979323846 * (th / thc);
        y = fmin(fmax(y, 1e-6), 0.5 * 3.14159265358979323846 - 1e-6);
        const double t = tan(y);
        b = v[MPF3D_S_KSI] + (1.0 - v[MPF3D_S_KSI]) * t * tanh(1.0 / t);
    }
    P.b_flat = (float)b;
    const double a_flat =
        v[MPF3D_S_MU_A] * (1.0 + v[MPF3D_S_DELTA_A] * (sqrt(pp) + tan(v[MPF3D_S_A0]) * sqrt(1.0 + pp)));
    const double e = v[MPF3D_S_EPS0_SL] * a_flat;
    P.e2_flat = (float)(e * e);
    return P;
}


template <int S, int AMAX>
void launch_batched(const In &in, const Out &out, const Mats &M, const Params &P0, const mpf3d_instance *inst,
                    int n_inst, int n_tiles, const Queue &Q, int parity, int32_t *err, cudaStream_t s,
                    const mpf3d_tuning &T, uint8_t *tile_flags) {
    const int sms = sms_of_current_device();
    launch_early(batched_sweep_kernel, sweep_blocks((uint32_t)n_tiles, 8, sms), dim3(32, 8), s, in, out, P0, inst,
                 n_inst, Q, parity, tile_flags, (uint32_t)n_tiles);
    // one stream: the side-by-side launch of the compact step measured no gain here when
    // there were two list kernels (not measured with these); the work-list grids come from
    // T (the sweep's 32 x 8 x 4 tiles are fixed by the instance table)
    const int g_iface = sms * T.iface_blocks_per_sm, g_general = sms * T.general_blocks_per_sm;
    const dim3 b_iface(T.iface_threads), b_general(T.general_threads);
    const bool sym = P0.sym_normals;
    if (!by_kind_batch(P0)) {
        launch_early(sym ? batched_octet_kernel<S, AMAX, 4> : batched_octet_kernel<S, AMAX, 8>, sms * OCTET_BLOCKS, dim3(128), s,
                     in, out, M, P0, inst, n_inst, Q, parity, err);
        return;
    }
    if (!P0.use_aniso) {
        launch_early(batched_isotropic_kernel<S, AMAX>, g_general, b_general, s, in, out, M, P0, inst, n_inst, Q,
                     parity, err);
        return;
    }
    if (Q.split)
        launch_early(sym ? batched_pair_kernel<4> : batched_pair_kernel<8>, g_iface, b_iface, s, in, out, M, P0, inst,
                     n_inst, Q, parity);
    launch_early(sym ? batched_trio_kernel<S, 4> : batched_trio_kernel<S, 8>, g_iface, b_iface, s, in, out, M, P0,
                 inst, n_inst, Q, parity);
    launch_early(batched_general_kernel<S>, g_general, b_general, s, in, out, M, P0, inst, n_inst, Q, parity);
    launch_early(sym ? batched_rest_kernel<S, AMAX, 4> : batched_rest_kernel<S, AMAX, 8>, sms * 8, dim3(128), s, in,
                 out, M, P0, inst, n_inst, Q, parity, err);
}

}  // namespace

extern "C" int mpf3d_streams_prepare(void *stream) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return MPF3D_ERR_CUDA;
    SideTable &tab = side_table_of(dev);
    std::lock_guard<std::mutex> lock(tab.mu);
    return side_ready(tab.by_caller[(cudaStream_t)stream], (cudaStream_t)stream) ? MPF3D_OK : MPF3D_ERR_CUDA;
}

// The body of mpf3d_compact_step_tuned and mpf3d_compact_step_clocked
// (clock: null, or the device step clock with T_melt and the cooling rate).
static int compact_step_impl(const uint32_t *cnt, const uint16_t *idx, const float *val, uint32_t *cnt_out,
                             uint16_t *idx_out, float *val_out, int slots, int amax, const double *T0z,
                             double Tm_plus_cool, const float *wij, const float *a2ij, const float *mij,
                             const float *n111, int N, int nx, int ny, int nz, const mpf3d_scalars *sc,
                             int enable_anisotropy, int enable_torque, int symmetric_normals, uint32_t *work_items,
                             uint32_t *work_count, int parity, int32_t *err, void *stream,
                             const mpf3d_tuning *tuning, uint8_t *tile_flags, int options, mpf3d_step_clock *clock,
                             double clock_T_melt, double clock_rate) {
    const mpf3d_tuning T = tuning ? *tuning : DEFAULT_TUNING;
    if (!tuning_ok(T)) return MPF3D_ERR_ARG;
    if (!cnt || !idx || !val || !cnt_out || !idx_out || !val_out || !T0z || !wij || !a2ij || !mij || !n111 || !sc ||
        !err || !work_items || !work_count)
        return MPF3D_ERR_ARG;
    if (N <= 0 || N > 65535 || !dims_ok(nx, ny, nz)) return MPF3D_ERR_ARG;
    if ((int64_t)nx * ny * nz >= ((int64_t)1 << 31)) return MPF3D_ERR_TOO_LARGE;
    if (cnt == cnt_out || idx == idx_out || val == val_out) return MPF3D_ERR_ARG;
    Params P = shared_params(sc, enable_anisotropy, enable_torque, symmetric_normals);
    P.nx = nx; P.ny = ny; P.nz = nz; P.N = N;
    P.cells = (int64_t)nx * ny * nz;
    P.cells32 = (uint32_t)P.cells;
    P.Tmc = Tm_plus_cool;
    parity &= 1;
    P.clock = clock;
    P.clock_T_melt = clock_T_melt;
    P.clock_rate = clock_rate;
    P.parity = parity;
    In in{cnt, idx, val};
    Out out{cnt_out, idx_out, val_out};
    Mats M{T0z, wij, a2ij, mij, n111};
    Queue Q{work_items, work_count, (options & MPF3D_STEP_MULTI_LIST) ? 1 : 0};
    cudaStream_t s = (cudaStream_t)stream;
    const bool tma = (options & MPF3D_STEP_SWEEP_TMA) != 0;
    if (slots == 4 && amax == 8) launch_step<4, 8>(in, out, M, P, Q, parity, tile_flags, err, s, T, tma);
    else if (slots == 8 && amax == 16) launch_step<8, 16>(in, out, M, P, Q, parity, tile_flags, err, s, T, tma);
    else if (slots == 16 && amax == 32) launch_step<16, 32>(in, out, M, P, Q, parity, tile_flags, err, s, T, tma);
    else return MPF3D_ERR_ARG;
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}

extern "C" int mpf3d_compact_step_tuned(const uint32_t *cnt, const uint16_t *idx, const float *val,
                                        uint32_t *cnt_out, uint16_t *idx_out, float *val_out, int slots, int amax,
                                        const double *T0z, double Tm_plus_cool, const float *wij, const float *a2ij,
                                        const float *mij, const float *n111, int N, int nx, int ny, int nz,
                                        const mpf3d_scalars *sc, int enable_anisotropy, int enable_torque,
                                        int symmetric_normals, uint32_t *work_items, uint32_t *work_count,
                                        int parity, int32_t *err, void *stream, const mpf3d_tuning *tuning,
                                        uint8_t *tile_flags, int options) {
    return compact_step_impl(cnt, idx, val, cnt_out, idx_out, val_out, slots, amax, T0z, Tm_plus_cool, wij, a2ij,
                             mij, n111, N, nx, ny, nz, sc, enable_anisotropy, enable_torque, symmetric_normals,
                             work_items, work_count, parity, err, stream, tuning, tile_flags, options, nullptr, 0.0,
                             0.0);
}

extern "C" int mpf3d_compact_step_clocked(const uint32_t *cnt, const uint16_t *idx, const float *val,
                                          uint32_t *cnt_out, uint16_t *idx_out, float *val_out, int slots,
                                          int amax, const double *T0z, mpf3d_step_clock *clock, double T_melt,
                                          double cooling_rate, const float *wij, const float *a2ij,
                                          const float *mij, const float *n111, int N, int nx, int ny, int nz,
                                          const mpf3d_scalars *sc, int enable_anisotropy, int enable_torque,
                                          int symmetric_normals, uint32_t *work_items, uint32_t *work_count,
                                          int parity, int32_t *err, void *stream, const mpf3d_tuning *tuning,
                                          uint8_t *tile_flags, int options) {
    if (!clock) return MPF3D_ERR_ARG;
    return compact_step_impl(cnt, idx, val, cnt_out, idx_out, val_out, slots, amax, T0z, T_melt, wij, a2ij, mij,
                             n111, N, nx, ny, nz, sc, enable_anisotropy, enable_torque, symmetric_normals,
                             work_items, work_count, parity, err, stream, tuning, tile_flags, options, clock, T_melt,
                             cooling_rate);
}

extern "C" int mpf3d_compact_step(const uint32_t *cnt, const uint16_t *idx, const float *val, uint32_t *cnt_out,
                                  uint16_t *idx_out, float *val_out, int slots, int amax, const double *T0z,
                                  double Tm_plus_cool, const float *wij, const float *a2ij, const float *mij,
                                  const float *n111, int N, int nx, int ny, int nz, const mpf3d_scalars *sc,
                                  int enable_anisotropy, int enable_torque, int symmetric_normals,
                                  uint32_t *work_items, uint32_t *work_count, int parity, int32_t *err,
                                  void *stream) {
    return mpf3d_compact_step_tuned(cnt, idx, val, cnt_out, idx_out, val_out, slots, amax, T0z, Tm_plus_cool, wij,
                                    a2ij, mij, n111, N, nx, ny, nz, sc, enable_anisotropy, enable_torque,
                                    symmetric_normals, work_items, work_count, parity, err, stream, nullptr,
                                    nullptr, 0);
}

extern "C" int mpf3d_compact_step_by_kind(int nx, int ny, int nz, int enable_anisotropy) {
    if (!dims_ok(nx, ny, nz)) return 0;
    Params P;
    memset(&P, 0, sizeof P);
    P.nx = nx; P.ny = ny; P.nz = nz;
    P.cells = (int64_t)nx * ny * nz;
    P.use_aniso = enable_anisotropy != 0;
    return by_kind(P) ? 1 : 0;
}

extern "C" int mpf3d_batched_step_by_kind(uint32_t total_cells, int enable_anisotropy) {
    Params P;
    memset(&P, 0, sizeof P);
    P.cells = total_cells;
    P.use_aniso = enable_anisotropy != 0;
    return by_kind_batch(P) ? 1 : 0;
}

extern "C" int64_t mpf3d_compact_tile_flags_len(int nx, int ny, int nz) {
    if (!dims_ok(nx, ny, nz)) return 0;
    return 2 * (int64_t)tiles_of<2>(nx, ny, nz);
}

extern "C" int mpf3d_compact_to_dense_view(const uint32_t *head, const uint16_t *idx, const float *val, int slots,
                                           uint32_t stride, uint32_t base, int N, int nx, int ny, int nz, void *phi,
                                           int phi_dtype, void *stream) {
    if (!phi || !head || !idx || !val || N <= 0 || N > 65535 || !dims_ok(nx, ny, nz)) return MPF3D_ERR_ARG;
    if ((uint64_t)base + (uint64_t)nx * ny * nz > (uint64_t)stride) return MPF3D_ERR_ARG;
    return to_dense({head, idx, val}, slots, N, nx, ny, nz, stride, base, phi, phi_dtype, (cudaStream_t)stream);
}


extern "C" int mpf3d_batched_init_bicrystal(const mpf3d_instance *inst, int n_inst, uint32_t total_cells, double dx,
                                            double delta, uint32_t *head, uint16_t *idx, float *val, int32_t *err,
                                            void *stream) {
    if (!inst || n_inst <= 0 || n_inst > 65535 || !head || !idx || !val || !err || total_cells == 0)
        return MPF3D_ERR_ARG;
    const float factor_dz = (float)((double)(float)(2.2 / delta) * dx);
    Out o{head, idx, val};
    batched_init_bicrystal_kernel<<<dim3(64, n_inst), 256, 0, (cudaStream_t)stream>>>(o, inst, n_inst, total_cells,
                                                                                      factor_dz, err);
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}

extern "C" int mpf3d_batched_step_tuned(const uint32_t *head, const uint16_t *idx, const float *val,
                                        uint32_t *head_out, uint16_t *idx_out, float *val_out, int slots, int amax,
                                        const mpf3d_instance *inst, int n_inst, int n_tiles, uint32_t total_cells,
                                        const float *wij, const float *a2ij, const float *mij, const float *n111, int N,
                                        const mpf3d_scalars *sc, int enable_anisotropy, int enable_torque,
                                        int symmetric_normals, uint32_t *work_items, uint32_t *work_count, int parity,
                                        int32_t *err, void *stream, int options, const mpf3d_tuning *tuning,
                                        uint8_t *tile_flags) {
    const mpf3d_tuning T = tuning ? *tuning : DEFAULT_TUNING;
    if (!tuning_ok(T)) return MPF3D_ERR_ARG;
    if (!head || !idx || !val || !head_out || !idx_out || !val_out || !inst || !wij || !a2ij || !mij || !n111 ||
        !sc || !err || !work_items || !work_count || n_inst <= 0 || n_tiles <= 0 || total_cells == 0 || N <= 0 ||
        N > 65535)
        return MPF3D_ERR_ARG;
    if (total_cells >= (1u << 31)) return MPF3D_ERR_TOO_LARGE;
    if (head == head_out || idx == idx_out || val == val_out) return MPF3D_ERR_ARG;
    Params P0 = shared_params(sc, enable_anisotropy, enable_torque, symmetric_normals);
    P0.cells = total_cells;
    P0.cells32 = total_cells;
    P0.N = N;
    In in{head, idx, val};
    Out out{head_out, idx_out, val_out};
    Mats M{nullptr, wij, a2ij, mij, n111};
    Queue Q{work_items, work_count, (options & MPF3D_STEP_MULTI_LIST) ? 1 : 0};
    cudaStream_t s = (cudaStream_t)stream;
    parity &= 1;
    uint8_t *F = tile_flags;
    if (slots == 4 && amax == 8) launch_batched<4, 8>(in, out, M, P0, inst, n_inst, n_tiles, Q, parity, err, s, T, F);
    else if (slots == 8 && amax == 16) launch_batched<8, 16>(in, out, M, P0, inst, n_inst, n_tiles, Q, parity, err, s, T, F);
    else if (slots == 16 && amax == 32) launch_batched<16, 32>(in, out, M, P0, inst, n_inst, n_tiles, Q, parity, err, s, T, F);
    else return MPF3D_ERR_ARG;
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}

extern "C" int64_t mpf3d_batched_tile_flags_len(int n_tiles) {
    return n_tiles > 0 ? 16 * (int64_t)n_tiles : 0;
}

extern "C" int mpf3d_batched_step(const uint32_t *head, const uint16_t *idx, const float *val, uint32_t *head_out,
                                  uint16_t *idx_out, float *val_out, int slots, int amax, const mpf3d_instance *inst,
                                  int n_inst, int n_tiles, uint32_t total_cells, const float *wij, const float *a2ij,
                                  const float *mij, const float *n111, int N, const mpf3d_scalars *sc,
                                  int enable_anisotropy, int enable_torque, int symmetric_normals,
                                  uint32_t *work_items, uint32_t *work_count, int parity, int32_t *err,
                                  void *stream, int options) {
    return mpf3d_batched_step_tuned(head, idx, val, head_out, idx_out, val_out, slots, amax, inst, n_inst, n_tiles,
                                    total_cells, wij, a2ij, mij, n111, N, sc, enable_anisotropy, enable_torque,
                                    symmetric_normals, work_items, work_count, parity, err, stream, options,
                                    nullptr, nullptr);
}

extern "C" int mpf3d_batched_fronts(const uint32_t *head, const uint16_t *idx, const float *val, int slots,
                                    const mpf3d_instance *inst, int n_inst, uint32_t total_cells, double *acc,
                                    void *stream) {
    if (!head || !idx || !val || !inst || !acc || n_inst <= 0 || n_inst > 65535) return MPF3D_ERR_ARG;
    In in{head, idx, val};
    dim3 g(16, n_inst);
    cudaStream_t s = (cudaStream_t)stream;
    if (slots == 4) batched_fronts_kernel<4><<<g, 256, 0, s>>>(in, inst, n_inst, total_cells, acc);
    else if (slots == 8) batched_fronts_kernel<8><<<g, 256, 0, s>>>(in, inst, n_inst, total_cells, acc);
    else if (slots == 16) batched_fronts_kernel<16><<<g, 256, 0, s>>>(in, inst, n_inst, total_cells, acc);
    else return MPF3D_ERR_ARG;
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}

extern "C" int mpf3d_batched_gb_rows(const uint32_t *head, const uint16_t *idx, const float *val, int slots,
                                     const mpf3d_instance *inst, int n_inst, uint32_t total_cells,
                                     const int32_t *row_base, double *gb, void *stream) {
    if (!head || !idx || !val || !inst || !row_base || !gb || n_inst <= 0 || n_inst > 65535) return MPF3D_ERR_ARG;
    In in{head, idx, val};
    dim3 g(16, n_inst);
    cudaStream_t s = (cudaStream_t)stream;
    if (slots == 4) batched_gb_rows_kernel<4><<<g, 128, 0, s>>>(in, inst, n_inst, total_cells, row_base, gb);
    else if (slots == 8) batched_gb_rows_kernel<8><<<g, 128, 0, s>>>(in, inst, n_inst, total_cells, row_base, gb);
    else if (slots == 16) batched_gb_rows_kernel<16><<<g, 128, 0, s>>>(in, inst, n_inst, total_cells, row_base, gb);
    else return MPF3D_ERR_ARG;
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}

extern "C" int mpf3d_compact_init_owner(const int32_t *owner, int slab, const float *prof, int nx, int ny, int nz,
                                        int slots, uint32_t *head, uint16_t *idx, float *val, void *stream) {
    if (!owner || !prof || !head || !idx || !val || slab <= 0 || slab > nz || slots < 2 || !dims_ok(nx, ny, nz))
        return MPF3D_ERR_ARG;
    const int64_t cells = (int64_t)nx * ny * nz;
    if (cells >= ((int64_t)1 << 32)) return MPF3D_ERR_TOO_LARGE;
    Out o{head, idx, val};
    init_owner_kernel<<<sms_of_current_device() * 16, 256, 0, (cudaStream_t)stream>>>(o, owner, slab, prof, nx, ny, nz,
                                                                                       (uint32_t)cells);
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// Step without device allocation.
//
// Some hosts cannot let this library allocate device memory: applications
// that reserve the whole GPU memory budget up front for their own pool and
// give plugins none, or real-time loops where a cudaMalloc -- which may
// synchronise the device -- is not acceptable.  For them the work list of
// the step lives in a file-scope device array instead of caller scratch.
// Every GPU that loads the library holds the array until the process exits.
namespace {

constexpr uint32_t kNoAllocMaxCells = MPF3D_NOALLOC_MAX_CELLS;
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) uint32_t g_noalloc_items[kNoAllocMaxCells];
static __device__ __align__(256) uint32_t g_noalloc_count[4];

struct NoAllocScratch {
    uint32_t *items = nullptr;
    uint32_t *count = nullptr;
    bool ready = false;
};
NoAllocScratch g_noalloc_dev[kNoAllocMaxDevices];
std::mutex g_noalloc_mu;

// Device addresses of the array on the current device.  In host code the
// array's name is only a host-side stand-in, so the address is looked up
// once per device, with that device current.
int noalloc_scratch(uint32_t **items, uint32_t **count) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return MPF3D_ERR_CUDA;
    if (dev < 0 || dev >= kNoAllocMaxDevices) return MPF3D_ERR_ARG;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    NoAllocScratch &s = g_noalloc_dev[dev];
    if (!s.ready) {
        void *pi = nullptr, *pc = nullptr;
        if (cudaGetSymbolAddress(&pi, g_noalloc_items) != cudaSuccess) return MPF3D_ERR_CUDA;
        if (cudaGetSymbolAddress(&pc, g_noalloc_count) != cudaSuccess) return MPF3D_ERR_CUDA;
        s.items = (uint32_t *)pi;
        s.count = (uint32_t *)pc;
        s.ready = true;
    }
    *items = s.items;
    *count = s.count;
    return MPF3D_OK;
}

}  // namespace

extern "C" int mpf3d_compact_step_noalloc(const uint32_t *head, const uint16_t *idx, const float *val,
                                          uint32_t *head_out, uint16_t *idx_out, float *val_out, int slots,
                                          int amax, const double *T0z, double Tm_plus_cool, const float *wij,
                                          const float *a2ij, const float *mij, const float *n111, int N, int nx,
                                          int ny, int nz, const mpf3d_scalars *sc, int enable_anisotropy,
                                          int enable_torque, int symmetric_normals, int32_t *err, void *stream) {
    if (nx <= 0 || ny <= 0 || nz <= 0) return MPF3D_ERR_ARG;
    if ((int64_t)nx * ny * nz > (int64_t)kNoAllocMaxCells) return MPF3D_ERR_TOO_LARGE;
    uint32_t *items = nullptr, *count = nullptr;
    const int rc = noalloc_scratch(&items, &count);
    if (rc != MPF3D_OK) return rc;
    // the counters must start at zero; the previous call left its totals there
    if (cudaMemsetAsync(count, 0, 4 * sizeof(uint32_t), (cudaStream_t)stream) != cudaSuccess) return MPF3D_ERR_CUDA;
    return mpf3d_compact_step(head, idx, val, head_out, idx_out, val_out, slots, amax, T0z, Tm_plus_cool, wij,
                              a2ij, mij, n111, N, nx, ny, nz, sc, enable_anisotropy, enable_torque,
                              symmetric_normals, items, count, 0, err, stream);
}
