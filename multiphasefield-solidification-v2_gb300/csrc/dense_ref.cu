// dense_ref.cu -- dense drop-in tier: the reference's 3D kernels with the
// reference's numerics, on the reference's dense [N][nx][ny][nz] arrays.
//
// Replaces src/gpu_kernels_3d.py:462-838 (kernel_update_nfmf_3d[_checked],
// kernel_update_phasefield_active_3d[_switchable], kernel_update_temp_3d).
//
// Numerics: arithmetic types follow compiled Numba (float literals are
// float64, float32 op float64 -> float64, float32(...) casts, float32 local
// arrays lap_sl/b_sl).  This translation unit is compiled with -fmad=false
// because the reference's NVVM pipeline does not contract a*b+c without
// fastmath; with that, results match the reference up to the last-bit
// differences of libm transcendentals.
//
// GB300 layout choices (not the reference's): a warp's lanes run along z, the
// contiguous axis, so every phi/mf/nf row is a 128-byte coalesced segment;
// blocks take tiles of such rows, find the active cells with bit masks (APT)
// and do the float64 arithmetic of the update on compacted cells only.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "float64.cuh"
#include "mpf3d.h"
#include "mpf3d_internal.h"

namespace mpf3d {
namespace dense {

constexpr int KMAX = MPF3D_KMAX;
constexpr int LIQ = 0;

struct Params {
    int N, nx, ny, nz, depth;
    double dx, dt, T_melt, Sf, eps0, w0, a0, delta_a, mu_a, p_round, g2_floor, ksi, theta_c;
    double two_dx, half_over_dx, inv_dx2, pp, mu_da, eps0sq;
    double r_dx, r_two_dx;  // reciprocals for div_const
    float floor_lo;         // squared differences below this are below g2_floor
    double cos_lo;          // acos of a cosine below this is above theta_c
    int a0_32, p32, dT32, df32;
    int use_aniso, use_torque, switchable;
};

__device__ __forceinline__ int ixp(int l, int n) { return l < n - 1 ? l + 1 : 0; }
__device__ __forceinline__ int ixm(int l, int n) { return l > 0 ? l - 1 : n - 1; }
__device__ __forceinline__ int izp(int k, int n) { return k < n - 1 ? k + 1 : n - 1; }
__device__ __forceinline__ int izm(int k, int n) { return k > 0 ? k - 1 : 0; }

template <typename T>
struct Field {
    const T *__restrict__ p;
    int nx, ny, nz;
    size_t plane;
    __device__ __forceinline__ T at(int g, int l, int m, int k) const {
        return __ldg(p + (size_t)g * plane + ((size_t)l * ny + m) * nz + k);
    }
};

struct Vec3 {
    double x, y, z;
};

// grad_phi_xyz (:94-107) of phase g at cell (l,m,k)
template <typename T>
__device__ __forceinline__ Vec3 grad_at(const Field<T> &f, int g, int l, int m, int k, double two_dx) {
    int lp = ixp(l, f.nx), lm = ixm(l, f.nx), mp = ixp(m, f.ny), mm = ixm(m, f.ny);
    int kp = izp(k, f.nz), km = izm(k, f.nz);
    Vec3 r;
    r.x = (double)(T)(f.at(g, lp, m, k) - f.at(g, lm, m, k)) / two_dx;
    r.y = (double)(T)(f.at(g, l, mp, k) - f.at(g, l, mm, k)) / two_dx;
    r.z = (double)(T)(f.at(g, l, m, kp) - f.at(g, l, m, km)) / two_dx;
    return r;
}

// Float64 roots and quotients out of line: inlined at every use they made the
// update wait on instruction fetch.
__device__ __noinline__ double root(double x) { return sqrt(x); }
__device__ __noinline__ double quotient(double x, double y) { return x / y; }
__device__ __noinline__ double reciprocal(double x) { return 1.0 / x; }

// 1/c for div_const, or 0 (plain division) where c is far from 1
inline double safe_reciprocal(double c) { return fabs(c) > 1e-100 && fabs(c) < 1e100 ? 1.0 / c : 0.0; }

// x / c for a constant c with rc = RN(1/c): Markstein's division with the
// reciprocal known (P. Markstein, IBM J. Res. Dev. 34(1), 1990) -- quotient
// estimate, exact FMA remainder, corrected quotient: 3 float64 operations
// where a division takes about 7.  Exponents near the ends of the range,
// infinities and NaN take the division.
__device__ __forceinline__ double div_const(double x, double c, double rc) {
    const uint32_t e = (uint32_t)__double2hiint(x) & 0x7fffffffu;
    if (__double_as_longlong(rc) == 0 || (e - 0x10000000u > 0x60000000u && (e | (uint32_t)__double2loint(x)) != 0u))
        return quotient(x, c);
    const double q = x * rc;
    return fma(fma(-q, c, x), rc, q);
}

// A gradient of squared length q >= g2_floor with its best {111} normal:
// best_cos_from_grad_3d (:110-134, float64 result) and
// facet_cos_and_nxyz_from_grad (:251-301, float32 results), which evaluate
// the same dot products in the same order.  s = sqrt(q), ig = 1 / s.
struct Facet {
    double q, s, ig, best64;
    float cs, ca, nx, ny, nz;
};

// The first maximum of |g . u| over the 8 normals.  d is proportional to g
// in float32: a normal whose float32 |d . u| lies more than the float32
// error bound below the largest one cannot win, and only the others are
// evaluated in float64 (one of an exact antipodal pair, which ties).
__device__ __forceinline__ Facet facet(const Vec3 &g, double q, float dx, float dy, float dz,
                                       const float *__restrict__ u) {
    Facet f;
    f.q = q;
    f.s = root(q);
    f.ig = reciprocal(f.s);
    const double gx = g.x * f.ig, gy = g.y * f.ig, gz = g.z * f.ig;
    float a[8], top = 0.0f, mag = 0.0f;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const float px = dx * __ldg(u + 3 * t), py = dy * __ldg(u + 3 * t + 1), pz = dz * __ldg(u + 3 * t + 2);
        a[t] = fabsf(px + py + pz);
        top = fmaxf(top, a[t]);
        mag = fmaxf(mag, fabsf(px) + fabsf(py) + fabsf(pz));
    }
    const float least = mag > 1e-30f ? top - 2e-6f * mag : -1.0f;
    uint32_t left = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) left |= a[t] < least ? 0u : 1u << t;
    double best_abs = 0.0, best_signed = 0.0;
    f.nx = 1.0f; f.ny = 0.0f; f.nz = 0.0f;
    while (left) {
        const int t = __ffs(left) - 1;
        left &= left - 1;
        const float ux = __ldg(u + 3 * t), uy = __ldg(u + 3 * t + 1), uz = __ldg(u + 3 * t + 2);
        if (best_abs > 0.0 && ux == -f.nx && uy == -f.ny && uz == -f.nz) continue;
        const double dot = gx * wide(ux) + gy * wide(uy) + gz * wide(uz);
        const double ad = fabs(dot);
        if (above(ad, best_abs)) {
            best_abs = ad; best_signed = dot; f.nx = ux; f.ny = uy; f.nz = uz;
        }
    }
    if (above(best_abs, 1.0)) best_abs = 1.0;
    if (above(best_signed, 1.0)) best_signed = 1.0;
    if (above(-best_signed, 1.0)) best_signed = -1.0;
    f.best64 = best_abs;
    f.cs = narrow<float>(best_signed); f.ca = narrow<float>(best_abs);
    return f;
}

// calc_a_from_cos (:24-30) with a float64 cosine
__device__ __forceinline__ double calc_a64(const Params &P, double tan_a0, double cost) {
    double c2 = cost * cost;
    double C = root(c2 + P.pp);
    double S = root(at_least_zero(1.0 - c2) + P.pp);
    return P.mu_a * (1.0 + P.delta_a * (C + tan_a0 * S));
}

// calc_a_from_cos with a float32 cosine (the f32-cast facet value)
__device__ __forceinline__ double calc_a32(const Params &P, double tan_a0, float cost) {
    float c2f = cost * cost;
    double c2 = wide(c2f);
    double C = P.p32 ? wide(sqrtf(c2f + (float)P.pp)) : root(c2 + P.pp);
    double S = root(at_least_zero(1.0 - c2) + P.pp);
    return P.mu_a * (1.0 + P.delta_a * (C + tan_a0 * S));
}

// calc_b_from_cos (:33-55); a cosine surely outside the cusp needs no angle
__device__ __forceinline__ double calc_b(const Params &P, double c) {
    if (c < P.cos_lo) return 1.0;
    if (c > 1.0) c = 1.0;
    else if (c < -1.0) c = -1.0;
    double theta = acos(c);
    if (theta >= P.theta_c) return 1.0;
    double x = theta / P.theta_c;
    const double eps = 1.0e-6;
    const double hp = 0.5 * 3.14159265358979323846;
    double y = hp * x;
    if (y > hp - eps) y = hp - eps;
    if (y < eps) y = eps;
    double t = tan(y);
    return P.ksi + (1.0 - P.ksi) * t * tanh(1.0 / t);
}

// coef = (c/C) - tan(a0)*(c/S) of da_dphixyz_A12 / torque_A11_3d (:327-330, :423-426)
__device__ __forceinline__ double dadc_coef(const Params &P, double tan_a0, float cs) {
    float ccf = cs * cs;
    double S = root(at_least_zero(1.0 - wide(ccf)) + P.pp);
    if (P.p32) {
        float Cf = sqrtf(ccf + (float)P.pp);
        return wide(cs / Cf) - tan_a0 * quotient(wide(cs), S);
    }
    double C = root(wide(ccf) + P.pp);
    return quotient(wide(cs), C) - tan_a0 * quotient(wide(cs), S);
}

// d cos / d(grad phi) of the facet (da_dphixyz_A12 :304-341): component
// g_p, n_p with the shared u = g . n and 1/|g|^3
__device__ __forceinline__ double dcos(const Facet &f, double g_p, float n_p, double udotg, double ig3) {
    return wide(n_p) * f.ig - udotg * g_p * ig3;
}

// First cell of a block's tile of RX x RY rows of 32 cells along z.  BY_ROW:
// the chunks of one row tile are neighbours in the launch order; otherwise the
// row tiles of one layer of chunks are.
template <int RX, int RY, bool BY_ROW>
__device__ __forceinline__ void tile_origin(int nx, int ny, int nz, int &l0, int &m0, int &k0) {
    const unsigned chunks = (unsigned)(nz + 31) / 32, ty = (unsigned)(ny + RY - 1) / RY;
    const unsigned rows = (unsigned)(nx + RX - 1) / RX * ty;
    const unsigned c = BY_ROW ? blockIdx.x % chunks : blockIdx.x / rows;
    const unsigned t = BY_ROW ? blockIdx.x / chunks : blockIdx.x % rows;
    l0 = (int)(t / ty) * RX;
    m0 = (int)(t % ty) * RY;
    k0 = (int)c * 32;
}

// ---------------------------------------------------------------------------
// APT (:462-527)
//
// A block takes a tile of AX x AY rows of 32 cells along z.  For
// APT_PHASES phases at a time its warps load each row of the tile and of its
// one-row halo once and keep two 32-bit masks of it, "positive" and "zero"
// (plus the two cells beyond its ends), lane p those of phase p; the six-neighbour test of 32 cells is
// then a handful of bit operations, and most (row, phase) pairs end there
// with no active cell.  What is left is memory: each value is read once from
// DRAM.  The chunks of a row follow one another in the launch order, so that
// the cells beyond a row's ends are still in L2 (row tiles first: 2.3 ms).
// Against one thread per cell that loads up to seven values per phase in
// turn, on GB300: 256^3 float32, 65 phases: 8.7 -> 1.86 ms (4.4 GB, 0.65 ms at
// the copy rate); 101 x 90 x 77 float64, 17 phases: 223 -> 67 us.
constexpr int APT_PHASES = 8;

// sign tests on the bit patterns (float64 comparisons would occupy the slow
// float64 pipe); NaN is neither
__device__ __forceinline__ bool positive(float v) { return v > 0.0f; }
__device__ __forceinline__ bool positive(double v) { return above(v, 0.0); }
__device__ __forceinline__ bool is_zero(float v) { return v == 0.0f; }
__device__ __forceinline__ bool is_zero(double v) { return (__double_as_longlong(v) << 1) == 0; }

// nonzero bits in any of the values
__device__ __forceinline__ bool any_bit(const float (&v)[APT_PHASES]) {
    uint32_t b = 0;
#pragma unroll
    for (int p = 0; p < APT_PHASES; ++p) b |= __float_as_uint(v[p]);
    return b != 0u;
}
__device__ __forceinline__ bool any_bit(const double (&v)[APT_PHASES]) {
    uint64_t b = 0;
#pragma unroll
    for (int p = 0; p < APT_PHASES; ++p) b |= (uint64_t)__double_as_longlong(v[p]);
    return b != 0u;
}

template <typename T, int AX, int AY, int THREADS>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) apt_kernel(Field<T> phi, int N, int32_t *__restrict__ mf, int depth,
                                                      int32_t *__restrict__ nf, int32_t *__restrict__ status,
                                                      int checked, int32_t *__restrict__ err) {
    constexpr int HX = AX + 2, HY = AY + 2, WARPS = THREADS / 32, OWN = AX * AY / WARPS, HALO = 2 * (AX + AY),
                  HALO_OWN = (HALO + WARPS - 1) / WARPS;
    __shared__ uint32_t pos[APT_PHASES][HX * HY];  // positive cells of each row
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int l0, m0, k0;
    tile_origin<AX, AY, true>(phi.nx, phi.ny, phi.nz, l0, m0, k0);
    const int k = k0 + lane;
    const bool in_z = k < phi.nz;
    const int zl = min(lane, phi.nz - 1 - k0);  // lanes past the top load the top cell, outside `cells`
    const uint32_t cells = phi.nz - k0 >= 32 ? 0xffffffffu : (1u << (phi.nz - k0)) - 1u;
    // rows of the warp: its own and its share of the halo (periodic images; a
    // row past the domain stands for the image beside it)
    size_t row[OWN + HALO_OWN];
    int at[OWN + HALO_OWN];  // the row's entry in pos, -1 for none
#pragma unroll
    for (int o = 0; o < OWN + HALO_OWN; ++o) {
        int hx, hy;
        const int r = warp * OWN + o, q = warp + (o - OWN) * WARPS;
        if (o < OWN) {
            hx = r / AY + 1;
            hy = r % AY + 1;
        } else {
            const int side = q < 2 * AY ? q / AY : 2 + (q - 2 * AY) / AX;
            const int along = q < 2 * AY ? q % AY : (q - 2 * AY) % AX;
            hx = side == 0 ? 0 : (side == 1 ? HX - 1 : along + 1);
            hy = side == 2 ? 0 : (side == 3 ? HY - 1 : along + 1);
        }
        at[o] = o < OWN || q < HALO ? hx * HY + hy : -1;
        int l = l0 - 1 + hx, m = m0 - 1 + hy;
        l = l < 0 ? phi.nx - 1 : (l >= phi.nx ? 0 : l);
        m = m < 0 ? phi.ny - 1 : (m >= phi.ny ? 0 : m);
        row[o] = ((size_t)l * phi.ny + m) * phi.nz + k0;
    }
    // active phases so far of this lane's cell in each of the warp's rows
    int count[OWN];
#pragma unroll
    for (int o = 0; o < OWN; ++o) count[o] = 0;
    bool deep = false;
    for (int g0 = 0; g0 < N; g0 += APT_PHASES) {
        const int phases = min(APT_PHASES, N - g0);
        const T *block = phi.p + (size_t)g0 * phi.plane;
        const uint32_t keep = lane < phases ? cells : 0u;
        bool some_here = false;
        // lane p keeps phase g0 + p: positive cells, zero cells, and in bits
        // 0 and 31 whether the cells below and above the row are positive
        uint32_t mp[OWN], mz[OWN], me[OWN];
        auto load = [&](size_t row, T (&v)[APT_PHASES]) {
            const T *src = block + row + zl;
#pragma unroll
            for (int p = 0; p < APT_PHASES; ++p) v[p] = __ldg(src + (size_t)min(p, phases - 1) * phi.plane);
        };
        auto masks = [&](const T (&v)[APT_PHASES], uint32_t &p_mask, uint32_t &z_mask) {
            p_mask = 0u;
            z_mask = keep;
            if (!__any_sync(0xffffffffu, any_bit(v))) return;  // most rows: none of these phases
            some_here = true;
#pragma unroll
            for (int p = 0; p < APT_PHASES; ++p) {
                const uint32_t b = __ballot_sync(0xffffffffu, positive(v[p]));
                const uint32_t z = __ballot_sync(0xffffffffu, is_zero(v[p]));
                p_mask = lane == p ? b & keep : p_mask;
                z_mask = lane == p ? z & keep : z_mask;
            }
        };
        // the cells beyond the ends: lane p below, lane 8 + p above
        const int pe = lane & (APT_PHASES - 1);
        const bool up = lane >= APT_PHASES;
        const bool end = lane < 2 * APT_PHASES && pe < phases && (up ? k0 + 32 < phi.nz : k0 > 0);
        T v[2][APT_PHASES], e[OWN];
#pragma unroll
        for (int o = 0; o < OWN; ++o)
            e[o] = end ? __ldg(block + row[o] + (size_t)pe * phi.plane + (up ? 32 : -1)) : (T)0;
        load(row[0], v[0]);
#pragma unroll
        for (int o = 0; o < OWN + HALO_OWN; ++o) {  // the next row's loads run under this row's masks
            if (o + 1 < OWN + HALO_OWN) load(row[o + 1], v[(o + 1) & 1]);
            uint32_t p_mask, z_mask;
            masks(v[o & 1], p_mask, z_mask);
            if (o < OWN) {
                mp[o] = p_mask;
                mz[o] = z_mask;
                const uint32_t b = __ballot_sync(0xffffffffu, positive(e[o]));
                some_here = some_here || b != 0u;
                me[o] = ((b >> pe) & 1u) | ((b >> (APT_PHASES + pe)) << 31);
            }
            if (lane < APT_PHASES && at[o] >= 0) pos[lane][at[o]] = p_mask;
        }
        // none of these phases in the tile or beside it: nothing is active
        if (!__syncthreads_or(some_here)) continue;
#pragma unroll
        for (int o = 0; o < OWN; ++o) {
            const int r = warp * OWN + o, l = l0 + r / AY, m = m0 + r % AY;
            // lane p forms the active mask of phase g0 + p, for all 32 cells of the row
            uint32_t act = 0;
            if (lane < phases && l < phi.nx && m < phi.ny) {
                const uint32_t *c = &pos[lane][(r / AY + 1) * HY + r % AY + 1];
                const uint32_t near = c[-HY] | c[HY] | c[-1] | c[1] | (mp[o] << 1) | (mp[o] >> 1) | me[o];
                act = mp[o] | (mz[o] & near);
            }
            const size_t cell = ((size_t)l * phi.ny + m) * phi.nz + k;
            uint32_t some = __ballot_sync(0xffffffffu, act != 0u);
            while (some) {
                const int p = __ffs(some) - 1;
                some &= some - 1;
                if ((__shfl_sync(0xffffffffu, act, p) >> lane) & 1u) {
                    const int n = ++count[o];
                    if (n <= (checked ? KMAX : depth) && n <= depth) mf[(size_t)(n - 1) * phi.plane + cell] = g0 + p;
                    else if (!checked) deep = true;
                }
            }
        }
        __syncthreads();
    }
    bool ovf = false;
    int most = 0;
#pragma unroll
    for (int o = 0; o < OWN; ++o) {
        const int r = warp * OWN + o, l = l0 + r / AY, m = m0 + r % AY, n = count[o];
        if (l >= phi.nx || m >= phi.ny || !in_z) continue;
        ovf = ovf || n > KMAX;
        most = max(most, n);
        const int lim = checked ? KMAX : depth;
        nf[((size_t)l * phi.ny + m) * phi.nz + k] = n > lim ? lim : n;
    }
    if (checked) {
        // warp-aggregated atomic max: same final values as one atomic per cell
        for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
        const unsigned any_ovf = __ballot_sync(0xffffffffu, ovf);
        if (lane == 0) {
            if (any_ovf) atomicMax(status + 0, 1);
            if (most > *(volatile int32_t *)(status + 1)) atomicMax(status + 1, most);
        }
    }
    if (deep && err) atomicOr(err, MPF3D_DEV_MF_DEPTH);
}

// ---------------------------------------------------------------------------
// Phase update (:530-830)
//
// Float64 arithmetic bounds this kernel: an SM retires about 2 float64 lanes a
// clock, 1/64 of its float32 rate, so the time is the number of warp-wide
// float64 instructions.  Three things keep it down, without changing a result
// (each expression keeps the reference's rounding, see div_const, facet and
// solid_terms):
//  - only cells with two or more active phases do arithmetic.  A block takes a
//    tile of ROWS (x, y) rows of 32 cells along z, writes the zeros and the
//    one-phase cells with coalesced rows, and collects the other cells, z by z,
//    in a shared-memory list: the lanes of a warp then hold cells of one layer
//    of a front, which need the same terms;
//  - solid-liquid terms only for cells whose list holds the liquid, Laplacians
//    only where two solids meet, and each pair (i, j) once: the (j, i) terms
//    are its exact negatives;
//  - float32 tests first: gradients surely below the floor, and normals that
//    surely do not win, cost no float64.
// The liquid's 25-point stencils read a shared-memory tile with a two-cell
// halo.  Against one thread per cell of the whole grid, per step on GB300:
// 256^3 float32, 64 grains: 38.2 -> 3.1 ms (of which the 4.4 GB of zeros alone
// would take 0.65); 101 x 90 x 77 float64, 16 grains: 3.06 -> 0.64 ms; 32^3
// float32, 8 grains: 0.78 -> 0.22 ms.
constexpr int UPD_PITCH = 37;  // 32 cells along z, two halo cells on both sides, an odd pitch for the banks

// values of one launch that every cell shares (computed once per block, by
// the device's own functions)
struct Shared {
    double tan_a0, e2_flat, w_flat;  // ... for a gradient below the floor (facet cosine 0)
    float b_flat;
    double inv_n[KMAX + 1];
};

// the liquid around a cell, read from the block's tile
template <typename T, int RY>
struct Liquid {
    const T *c;      // the cell's entry
    int k, nz;
    static constexpr int SX = (RY + 4) * UPD_PITCH, SY = UPD_PITCH;
    // entry at (dx, dy) in the layer kk (a clamped z index)
    __device__ __forceinline__ T at(int dx, int dy, int kk) const { return c[dx * SX + dy * SY + (kk - k)]; }
    // central differences (before the division by 2 dx) at (dx, dy, kk)
    __device__ __forceinline__ void diffs(int dx, int dy, int kk, T &x, T &y, T &z) const {
        x = at(dx + 1, dy, kk) - at(dx - 1, dy, kk);
        y = at(dx, dy + 1, kk) - at(dx, dy - 1, kk);
        z = at(dx, dy, izp(kk, nz)) - at(dx, dy, izm(kk, nz));
    }
};

// a gradient from its differences; false if its squared length lies below
// the floor.  The float32 test settles gradients clearly below it.
template <typename T>
__device__ __forceinline__ bool gradient(const Params &P, T x, T y, T z, Vec3 &g, double &q) {
    const float fx = to_float(x), fy = to_float(y), fz = to_float(z);
    if (fx * fx + fy * fy + fz * fz < P.floor_lo) return false;
    g.x = div_const(wide(x), P.two_dx, P.r_two_dx);
    g.y = div_const(wide(y), P.two_dx, P.r_two_dx);
    g.z = div_const(wide(z), P.two_dx, P.r_two_dx);
    q = g.x * g.x + g.y * g.y + g.z * g.z;
    return !below(q, P.g2_floor);
}

// lap_sl and b_sl of one solid at a cell: aniso_term1_solid_3d (:149-204),
// torque_A11_3d (:386-441) with A13_divergence_3d (:344-383), and
// calc_b_from_cos of the cell's facet.  The stencil points are visited in
// turn (cell, x+, x-, y+, y-, z+, z-), each with one facet search.
template <typename T, int RY>
__device__ __forceinline__ void solid_terms(const Params &P, const Shared &S, const Liquid<T, RY> &L,
                                            const float *__restrict__ u, float &lap_sl, float &b_sl) {
    const int kp = izp(L.k, L.nz), km = izm(L.k, L.nz);
    const T pc = L.at(0, 0, L.k);
    double e2_0 = 0.0, flux = 0.0, lap_val = 0.0;
    float da_plus = 0.0f, dd[3] = {0.0f, 0.0f, 0.0f};
    Vec3 g0 = {0.0, 0.0, 0.0};
    Facet f0;
    bool tq = false;
    b_sl = S.b_flat;
#pragma unroll 1
    for (int p = 0; p < 7; ++p) {
        const int axis = (p - 1) >> 1;
        const int step = p == 0 ? 0 : ((p & 1) ? 1 : -1);
        const int ox = axis == 0 ? step : 0, oy = axis == 1 ? step : 0;
        const int kk = axis == 2 ? (step > 0 ? kp : km) : L.k;
        T x, y, z;
        L.diffs(ox, oy, kk, x, y, z);
        Vec3 g;
        double q, e2 = S.e2_flat;
        float da = 0.0f;
        if (gradient(P, x, y, z, g, q)) {
            const Facet f = facet(g, q, to_float(x), to_float(y), to_float(z), u);
            const double e = P.eps0 * calc_a64(P, S.tan_a0, f.best64);
            e2 = e * e;
            if (p == 0) {
                tq = P.use_torque;
                g0 = g;
                f0 = f;
                b_sl = narrow<float>(calc_b(P, f.best64));
            } else if (tq) {
                // the da/d(grad phi) component along the point's own axis
                const double udotg = g.x * wide(f.nx) + g.y * wide(f.ny) + g.z * wide(f.nz);
                const double g_p = axis == 0 ? g.x : (axis == 1 ? g.y : g.z);
                const float n_p = axis == 0 ? f.nx : (axis == 1 ? f.ny : f.nz);
                const double dc = dcos(f, g_p, n_p, udotg, reciprocal(f.q * f.s));
                da = narrow<float>(P.mu_da * dadc_coef(P, S.tan_a0, f.cs) * dc);
            }
        }
        if (p == 0) {
            e2_0 = e2;
            continue;
        }
        const T pv = L.at(ox, oy, kk);
        const T d = (p & 1) ? pv - pc : pc - pv;
        const double F = div_const((e2_0 + e2) * wide(d), P.two_dx, P.r_two_dx);
        if (p & 1) {
            flux = F;
            da_plus = da;
        } else {
            const double t = div_const(flux - F, P.dx, P.r_dx);
            lap_val = axis == 0 ? t : lap_val + t;
            const float v = narrow<float>(wide(da_plus - da) * P.half_over_dx);
            if (axis == 0) dd[0] = v;
            else if (axis == 1) dd[1] = v;
            else dd[2] = v;
        }
    }
    if (tq) {
        const double q = f0.q;
        // d2_phi_xyz (:207-248) of the liquid
        const double two_pc = 2.0 * wide(pc);
        const double pxx = (wide(L.at(1, 0, L.k)) - two_pc + wide(L.at(-1, 0, L.k))) * P.inv_dx2;
        const double pyy = (wide(L.at(0, 1, L.k)) - two_pc + wide(L.at(0, -1, L.k))) * P.inv_dx2;
        const double pzz = (wide(L.at(0, 0, kp)) - two_pc + wide(L.at(0, 0, km))) * P.inv_dx2;
        const double qq = 0.25 * P.inv_dx2;
        const double pxy =
            wide((T)(((T)(L.at(1, 1, L.k) - L.at(1, -1, L.k)) - L.at(-1, 1, L.k)) + L.at(-1, -1, L.k))) * qq;
        const double pxz = wide((T)(((T)(L.at(1, 0, kp) - L.at(1, 0, km)) - L.at(-1, 0, kp)) + L.at(-1, 0, km))) * qq;
        const double pyz = wide((T)(((T)(L.at(0, 1, kp) - L.at(0, 1, km)) - L.at(0, -1, kp)) + L.at(0, -1, km))) * qq;
        const double q_x = 2.0 * (g0.x * pxx + g0.y * pxy + g0.z * pxz);
        const double q_y = 2.0 * (g0.x * pxy + g0.y * pyy + g0.z * pyz);
        const double q_z = 2.0 * (g0.x * pxz + g0.y * pyz + g0.z * pzz);
        const double ig3 = reciprocal(q * f0.s);
        const double udotg = g0.x * wide(f0.nx) + g0.y * wide(f0.ny) + g0.z * wide(f0.nz);
        const double dcx = dcos(f0, g0.x, f0.nx, udotg, ig3);
        const double dcy = dcos(f0, g0.y, f0.ny, udotg, ig3);
        const double dcz = dcos(f0, g0.z, f0.nz, udotg, ig3);
        const double mc = P.mu_da * dadc_coef(P, S.tan_a0, f0.cs);
        const float d0x = narrow<float>(mc * dcx), d0y = narrow<float>(mc * dcy), d0z = narrow<float>(mc * dcz);
        const double da_dx = mc * (dcx * pxx + dcy * pxy + dcz * pxz);
        const double da_dy = mc * (dcx * pxy + dcy * pyy + dcz * pyz);
        const double da_dz = mc * (dcx * pxz + dcy * pyz + dcz * pzz);
        const float a = narrow<float>(calc_a32(P, S.tan_a0, f0.ca));
        const double Ex = (da_dx * wide(d0x) * q) + (wide(a * dd[0]) * q) + (wide(a * d0x) * q_x);
        const double Ey = (da_dy * wide(d0y) * q) + (wide(a * dd[1]) * q) + (wide(a * d0y) * q_y);
        const double Ez = (da_dz * wide(d0z) * q) + (wide(a * dd[2]) * q) + (wide(a * d0z) * q_z);
        lap_val += P.eps0sq * (Ex + Ey + Ez);
    }
    lap_sl = narrow<float>(lap_val);
}

// clip and renormalise (:663-680) the n unclipped fractions and store them
template <typename T>
__device__ __forceinline__ void store_cell(T *__restrict__ phi_new, size_t plane, size_t cell, int n, const int *ids,
                                           T *outv) {
    double ssum = 0.0;
    for (int t = 0; t < n; ++t) {
        double v = wide(outv[t]);
        if (below_zero(v)) v = 0.0;
        if (above(v, 1.0)) v = 1.0;
        outv[t] = narrow<T>(v);
        ssum += v;
    }
    if (above(ssum, 1e-20)) {
        const double invs = reciprocal(ssum);
        for (int t = 0; t < n; ++t) phi_new[(size_t)ids[t] * plane + cell] = narrow<T>(wide(outv[t]) * invs);
    } else {
        for (int t = 0; t < n; ++t) phi_new[(size_t)ids[t] * plane + cell] = outv[t];
        phi_new[cell] = (T)1;
    }
}

// One cell with n >= 2 active phases (ids checked).
template <typename T, typename TT, int RY>
__device__ __forceinline__ void update_cell(const Field<T> &phi, T *__restrict__ phi_new, const TT *__restrict__ temp,
                                            const int32_t *__restrict__ mf, int n, const float *__restrict__ wij,
                                            const float *__restrict__ aij, const float *__restrict__ mij,
                                            const float *__restrict__ n111, const Params &P, const Shared &S,
                                            const Liquid<T, RY> &L, int l, int m) {
    const int N = P.N, k = L.k;
    const size_t plane = phi.plane;
    const size_t cell = ((size_t)l * P.ny + m) * P.nz + k;
    int ids[KMAX];
    T phc[KMAX];
    bool liq = false;
    int solids = 0;
    for (int t = 0; t < n; ++t) {
        ids[t] = __ldg(mf + (size_t)t * plane + cell);
        phc[t] = __ldg(phi.p + (size_t)ids[t] * plane + cell);
        liq |= ids[t] == LIQ;
        solids += ids[t] != LIQ;
    }
    const int lp = ixp(l, P.nx), lm = ixm(l, P.nx), mp = ixp(m, P.ny), mm = ixm(m, P.ny);
    const int kp = izp(k, P.nz), km = izm(k, P.nz);

    // solid-liquid terms; only pairs with the liquid use them
    float lap_sl[KMAX], b_sl[KMAX];
    double w_sl = P.w0;
    if (liq && solids) {
        float lap_iso = 0.0f;
        if (!P.use_aniso) {
            T s = L.at(1, 0, k) + L.at(-1, 0, k);
            s = s + L.at(0, 1, k);
            s = s + L.at(0, -1, k);
            s = s + L.at(0, 0, kp);
            s = s + L.at(0, 0, km);
            const double lap_liq = (wide(s) - 6.0 * wide(L.at(0, 0, k))) * P.inv_dx2;
            lap_iso = narrow<float>(P.eps0sq * lap_liq);
        }
        // dominant solid (:579-589)
        int i_s = -1;
        T maxv = (T)-1;
        for (int t = 0; t < n; ++t) {
            if (ids[t] == LIQ) continue;
            lap_sl[t] = lap_iso;
            b_sl[t] = 1.0f;
            if (P.use_aniso) solid_terms(P, S, L, n111 + (size_t)ids[t] * 24, lap_sl[t], b_sl[t]);
            if (phc[t] > maxv) {
                maxv = phc[t];
                i_s = ids[t];
            }
        }
        if (P.use_aniso && i_s != -1) {
            // anisotropic w_sl of its gradient (:590-595)
            const T x = phi.at(i_s, lp, m, k) - phi.at(i_s, lm, m, k);
            const T y = phi.at(i_s, l, mp, k) - phi.at(i_s, l, mm, k);
            const T z = phi.at(i_s, l, m, kp) - phi.at(i_s, l, m, km);
            Vec3 g;
            double q;
            w_sl = S.w_flat;
            if (gradient(P, x, y, z, g, q)) {
                const Facet f = facet(g, q, to_float(x), to_float(y), to_float(z), n111 + (size_t)i_s * 24);
                const double al = calc_a64(P, S.tan_a0, f.best64);
                w_sl = P.w0 * (al * al);
            }
        }
    }
    // Laplacians (laplacian_3d :444-459); only pairs of solids use them
    double lapk[KMAX];
    if (solids >= 2) {
        for (int t = 0; t < n; ++t) {
            const int g = ids[t];
            T s = phi.at(g, lp, m, k) + phi.at(g, lm, m, k);
            s = s + phi.at(g, l, mp, k);
            s = s + phi.at(g, l, mm, k);
            s = s + phi.at(g, l, m, kp);
            s = s + phi.at(g, l, m, km);
            lapk[t] = (wide(s) - 6.0 * wide(phc[t])) * P.inv_dx2;
        }
    }
    const double Tcur = wide(temp[cell]);
    const double dTv = P.dT32 ? (double)((float)Tcur - (float)P.T_melt) : Tcur - P.T_melt;
    const double force = liq ? (P.df32 ? (double)((float)P.Sf * (float)dTv) : P.Sf * dTv) : 0.0;
    const double inv_n = S.inv_n[n];
    const bool n_pow2 = (n & (n - 1)) == 0;
    double dpi[KMAX];
    for (int t = 0; t < n; ++t) dpi[t] = 0.0;
    for (int t1 = 0; t1 < n; ++t1) {
        const int i = ids[t1];
        for (int t2 = t1 + 1; t2 < n; ++t2) {
            const int j = ids[t2];
            if (i == j) continue;
            // with the liquid: the solid's terms, the sign of the pair's order
            const bool sl = j == LIQ, with_liq = sl || i == LIQ;
            const int ts = sl ? t1 : t2;
            double ppp = 0.0;
            for (int t3 = 0; t3 < n; ++t3) {
                const int pk3 = ids[t3];
                double wik = wide(__ldg(wij + i * N + pk3)), wjk = wide(__ldg(wij + j * N + pk3));
                if (pk3 == LIQ) {
                    if (i != LIQ) wik = w_sl;
                    if (j != LIQ) wjk = w_sl;
                }
                double term = (wik - wjk) * wide(phc[t3]);
                if (!with_liq) {
                    const float ai = __ldg(aij + i * N + pk3), aj = __ldg(aij + j * N + pk3);
                    const float e2i = ai * ai, e2j = aj * aj;
                    term += 0.5 * wide(e2i - e2j) * lapk[t3];
                } else if (pk3 == ids[ts]) {
                    term += (sl ? 0.5 : -0.5) * wide(lap_sl[ts]);
                }
                ppp = t3 == 0 ? term : ppp + term;
            }
            float m_ij = __ldg(mij + i * N + j), m_ji = __ldg(mij + j * N + i);
            if (with_liq) {
                const T pij = phc[t1] * phc[t2];
                const double pijd = wide(pij);
                ppp -= (8.0 / 3.1415926535) * root(above(pijd, 0.0) ? pijd : 0.0) * (sl ? -force : force);
                m_ij = m_ij * b_sl[ts];
                m_ji = m_ji * b_sl[ts];
            }
            auto over_n = [&](float me) {
                const double x = 2.0 * wide(me);
                return n_pow2 ? x * inv_n : div_const(x, (double)n, inv_n);
            };
            const double c_ij = over_n(m_ij);
            const double c_ji = m_ji == m_ij ? c_ij : over_n(m_ji);
            dpi[t1] -= c_ij * ppp;
            dpi[t2] += c_ji * ppp;
        }
    }
    T outv[KMAX];
    for (int t = 0; t < n; ++t) outv[t] = narrow<T>(wide(phc[t]) + P.dt * dpi[t]);
    store_cell(phi_new, plane, cell, n, ids, outv);
}

// One block per tile of RX x RY rows of 32 cells along z.
template <typename T, typename TT, int RX, int RY, int THREADS, int PER_SM>
__global__ void __launch_bounds__(THREADS, PER_SM) update_kernel(Field<T> phi, T *__restrict__ phi_new,
                                                             const TT *__restrict__ temp,
                                                             const int32_t *__restrict__ mf,
                                                             const int32_t *__restrict__ nf,
                                                             const float *__restrict__ wij,
                                                             const float *__restrict__ aij,
                                                             const float *__restrict__ mij,
                                                             const float *__restrict__ n111, Params P,
                                                             int32_t *__restrict__ err) {
    constexpr int ROWS = RX * RY;
    static_assert(ROWS <= 32, "one lane per row builds the list");
    __shared__ T tile[(RX + 4) * (RY + 4) * UPD_PITCH];
    __shared__ Shared S;
    __shared__ uint32_t row_mask[3][ROWS];  // three and more phases; two, with a gradient; two, flat
    __shared__ uint16_t list[ROWS * 32];
    __shared__ int list_n;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t plane = phi.plane;
    const int N = P.N;
    int l0, m0, k0;
    tile_origin<RX, RY, false>(P.nx, P.ny, P.nz, l0, m0, k0);
    const int k = k0 + lane;
    bool listed = false;
    // zeros, one-phase cells, and each row's mask of the others
    for (int r = warp; r < ROWS; r += THREADS / 32) {
        const int l = l0 + r / RY, m = m0 + r % RY;
        const bool inside = l < P.nx && m < P.ny && k < P.nz;
        const size_t cell = ((size_t)l * P.ny + m) * P.nz + k;
        int n = -1, id0 = LIQ;
        if (inside) {
            n = nf[cell];
            if (n < 0 || n > KMAX) {
                if (err) atomicOr(err, MPF3D_DEV_NF_GT_KMAX);
                n = -1;
            } else if (n > P.depth) {  // mf holds fewer rows than nf claims
                if (err) atomicOr(err, MPF3D_DEV_MF_DEPTH);
                n = -1;
            }
            for (int q = 0; q < n; ++q) {
                const int g = mf[(size_t)q * plane + cell];
                if (g < 0 || g >= N) {
                    if (err) atomicOr(err, MPF3D_DEV_BAD_ID);
                    n = -1;
                    break;
                }
                if (q == 0) id0 = g;
            }
        }
        const uint32_t many = __ballot_sync(0xffffffffu, n >= 3), two = __ballot_sync(0xffffffffu, n == 2);
        if (lane == 0) {
            row_mask[0][r] = many;
            row_mask[1][r] = two;
        }
        listed = listed || (many | two) != 0u;
        if (n >= 0) {
            T *out = phi_new + cell;
            for (int g = 0; g < N; ++g) out[(size_t)g * plane] = (T)0;
            if (n < 2) {
                T v = n == 1 ? __ldg(phi.p + (size_t)id0 * plane + cell) : (T)0;
                if (v == (T)1) out[(size_t)id0 * plane] = v;
                else store_cell(phi_new, plane, cell, n, &id0, &v);
            }
        }
    }
    // one answer for the block: the crew below changes row_mask, which a late warp
    // must not read to decide whether to stay
    if (!__syncthreads_or(listed)) return;
    // the last warp evaluates the shared values, the others collect the cells
    constexpr int CREW = THREADS - 32;
    if (threadIdx.x >= CREW) {
        if (lane == 0) {
            S.tan_a0 = P.a0_32 ? (double)tanf((float)P.a0) : tan(P.a0);
            const double al = calc_a64(P, S.tan_a0, 0.0), e = P.eps0 * al;
            S.e2_flat = e * e;
            S.w_flat = P.w0 * (al * al);
            S.b_flat = (float)calc_b(P, 0.0);
        } else {
            for (int n = lane; n <= KMAX; n += 31) S.inv_n[n] = 1.0 / (double)n;
        }
    } else {
        auto crew_barrier = [] { asm volatile("bar.sync 1, %0;\n" ::"n"(CREW) : "memory"); };
        // the liquid of the tile and its halo (periodic x and y, clamped z)
        for (int e = warp; e < (RX + 4) * (RY + 4); e += CREW / 32) {
            int l = (l0 - 2 + e / (RY + 4)) % P.nx, m = (m0 - 2 + e % (RY + 4)) % P.ny;
            l += l < 0 ? P.nx : 0;
            m += m < 0 ? P.ny : 0;
            for (int z = lane; z < 36; z += 32) {
                const int kk = min(max(k0 - 2 + z, 0), P.nz - 1);
                tile[e * UPD_PITCH + z] = phi.at(LIQ, l, m, kk);
            }
        }
        crew_barrier();
        // two-phase cells with no gradient above the floor on their stencil
        // are cheap: they go to warps of their own
        for (int r = warp; r < ROWS; r += CREW / 32) {
            const uint32_t two = row_mask[1][r];
            bool steep = false;
            if ((two >> lane) & 1u) {
                const Liquid<T, RY> L{tile + ((r / RY + 2) * (RY + 4) + r % RY + 2) * UPD_PITCH + lane + 2, k, P.nz};
                const int kp = izp(k, P.nz), km = izm(k, P.nz);
                auto over = [&](int dx, int dy, int kk) {
                    T x, y, z;
                    L.diffs(dx, dy, kk, x, y, z);
                    const float fx = to_float(x), fy = to_float(y), fz = to_float(z);
                    return !(fx * fx + fy * fy + fz * fz < P.floor_lo);
                };
                steep = over(0, 0, k) || over(1, 0, k) || over(-1, 0, k) || over(0, 1, k) || over(0, -1, k) ||
                        over(0, 0, kp) || over(0, 0, km);
            }
            const uint32_t b = __ballot_sync(0xffffffffu, steep);
            if (lane == 0) {
                row_mask[1][r] = b;
                row_mask[2][r] = two & ~b;
            }
        }
        crew_barrier();
        if (warp == 0) {  // the list: the costly classes first, each layer by layer
            int at = 0;
            for (int c = 0; c < 3; ++c) {
                const uint32_t mine = lane < ROWS ? row_mask[c][lane] : 0u;
                uint32_t layers = __reduce_or_sync(0xffffffffu, mine);
                while (layers) {
                    const int z = __ffs(layers) - 1;
                    layers &= layers - 1;
                    const uint32_t b = __ballot_sync(0xffffffffu, (mine >> z) & 1u);
                    if ((mine >> z) & 1u) list[at + __popc(b & ((1u << lane) - 1u))] = (uint16_t)(lane * 32 + z);
                    at += __popc(b);
                }
            }
            if (lane == 0) list_n = at;
        }
    }
    __syncthreads();
    const int todo = list_n;
    for (int i = threadIdx.x; i < todo; i += THREADS) {
        const int r = list[i] >> 5, z = list[i] & 31, kk = k0 + z;
        const int l = l0 + r / RY, m = m0 + r % RY;
        const size_t cell = ((size_t)l * P.ny + m) * P.nz + kk;
        const Liquid<T, RY> L{tile + ((r / RY + 2) * (RY + 4) + r % RY + 2) * UPD_PITCH + z + 2, kk, P.nz};
        update_cell<T, TT, RY>(phi, phi_new, temp, mf, nf[cell], wij, aij, mij, n111, P, S, L, l, m);
    }
}

// kernel_update_temp_3d (:833-838)
template <typename TT>
__global__ void temp_kernel(TT *__restrict__ temp, double rate, int rate32, int64_t n) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) {
        if (sizeof(TT) == 4 && rate32)
            temp[i] = (TT)((float)temp[i] - (float)rate);
        else
            temp[i] = (TT)((double)temp[i] - rate);
    }
}

}  // namespace dense
}  // namespace mpf3d

using namespace mpf3d;
using namespace mpf3d::dense;

static inline int bitset(uint32_t m, int i) { return (int)((m >> i) & 1u); }

// cells below (and from) which the launches take smaller (and larger) tiles
constexpr int64_t SMALL_GRID = 1 << 18, LARGE_GRID = 1 << 21;

// blocks of tiles of rx x ry rows of 32 cells along z (see tile_origin)
static unsigned tile_blocks(int nx, int ny, int nz, int rx, int ry) {
    return (unsigned)((nx + rx - 1) / rx) * (unsigned)((ny + ry - 1) / ry) * (unsigned)((nz + 31) / 32);
}

static bool grid_ok(int nx, int ny, int nz) {
    return nx > 0 && ny > 0 && nz > 0 && ny <= 65535 * 4 && nx <= 65535;
}

template <typename T>
static void launch_apt(const void *phi, int N, int nx, int ny, int nz, int32_t *mf, int depth, int32_t *nf,
                       int32_t *status, int checked, int32_t *err, cudaStream_t s) {
    const Field<T> f{(const T *)phi, nx, ny, nz, (size_t)nx * ny * nz};
    // small grids: smaller tiles, so that more SMs take part
    if ((int64_t)nx * ny * nz < SMALL_GRID)
        apt_kernel<T, 2, 4, 128><<<tile_blocks(nx, ny, nz, 2, 4), 128, 0, s>>>(f, N, mf, depth, nf, status, checked, err);
    else
        apt_kernel<T, 4, 8, 512><<<tile_blocks(nx, ny, nz, 4, 8), 512, 0, s>>>(f, N, mf, depth, nf, status, checked, err);
}

extern "C" int mpf3d_version(void) { return MPF3D_VERSION; }

extern "C" int mpf3d_dense_apt(const void *phi, int phi_dtype, int N, int nx, int ny, int nz, int32_t *mf,
                               int depth, int32_t *nf, int32_t *status, int checked, int32_t *err,
                               void *stream) {
    if (!phi || !mf || !nf || N <= 0 || depth <= 0 || !grid_ok(nx, ny, nz)) return MPF3D_ERR_ARG;
    if (checked && !status) return MPF3D_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    if (phi_dtype == MPF3D_F32) launch_apt<float>(phi, N, nx, ny, nz, mf, depth, nf, status, checked, err, s);
    else if (phi_dtype == MPF3D_F64) launch_apt<double>(phi, N, nx, ny, nz, mf, depth, nf, status, checked, err, s);
    else return MPF3D_ERR_DTYPE;
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}

template <typename T, typename TT>
static void launch_update(const void *phi, void *phi_new, const void *temp, const int32_t *mf, const int32_t *nf,
                          const float *wij, const float *aij, const float *mij, const float *n111, const Params &P,
                          int32_t *err, cudaStream_t s) {
    Field<T> f{(const T *)phi, P.nx, P.ny, P.nz, (size_t)P.nx * P.ny * P.nz};
#define UPDATE(RX, RY, THREADS, PER_SM)                                                                          \
    update_kernel<T, TT, RX, RY, THREADS, PER_SM><<<tile_blocks(P.nx, P.ny, P.nz, RX, RY), THREADS, 0, s>>>(     \
        f, (T *)phi_new, (const TT *)temp, mf, nf, wij, aij, mij, n111, P, err)
    // Large tiles fill the warps of a class better, small ones leave fewer
    // SMs idle at the end (float32, 256^3: 3.1 ms with 4 x 8 rows and 3 blocks
    // per SM, 4.3 ms with 4 x 4 rows and 2; float64, 101 x 90 x 77: 0.77 and
    // 0.64 ms; float32, 32^3: 0.22 ms with 1 x 4 rows, 0.27 ms with 2 x 4)
    const int64_t cells = (int64_t)P.nx * P.ny * P.nz;
    if (cells < SMALL_GRID) UPDATE(1, 4, 128, 1);
    else if (cells < LARGE_GRID) UPDATE(4, 4, 256, 2);
    else UPDATE(4, 8, 256, 3);
#undef UPDATE
}

extern "C" int mpf3d_dense_update(const void *phi, void *phi_new, int phi_dtype, const void *temp, int temp_dtype,
                                  const int32_t *mf, int depth, const int32_t *nf, const float *wij,
                                  const float *aij, const float *mij, const float *n111, int N, int nx, int ny,
                                  int nz, const mpf3d_scalars *sc, int switchable, int enable_anisotropy,
                                  int enable_torque, int32_t *err, void *stream) {
    if (!phi || !phi_new || !temp || !mf || !nf || !wij || !aij || !mij || !n111 || !sc) return MPF3D_ERR_ARG;
    if (N <= 0 || N > 65535 || depth <= 0 || !grid_ok(nx, ny, nz)) return MPF3D_ERR_ARG;
    if ((phi_dtype != MPF3D_F32 && phi_dtype != MPF3D_F64) || (temp_dtype != MPF3D_F32 && temp_dtype != MPF3D_F64))
        return MPF3D_ERR_DTYPE;
    Params P;
    P.N = N; P.nx = nx; P.ny = ny; P.nz = nz; P.depth = depth;
    const double *v = sc->v;
    const uint32_t fm = sc->f32mask;
    P.dx = v[MPF3D_S_DX]; P.dt = v[MPF3D_S_DT]; P.T_melt = v[MPF3D_S_T_MELT]; P.Sf = v[MPF3D_S_SF];
    P.eps0 = v[MPF3D_S_EPS0_SL]; P.w0 = v[MPF3D_S_W0_SL]; P.a0 = v[MPF3D_S_A0]; P.delta_a = v[MPF3D_S_DELTA_A];
    P.mu_a = v[MPF3D_S_MU_A]; P.p_round = v[MPF3D_S_P_ROUND]; P.g2_floor = v[MPF3D_S_G2_FLOOR];
    P.ksi = v[MPF3D_S_KSI]; P.theta_c = v[MPF3D_S_THETA_C_RAD];
    P.two_dx = 2.0 * P.dx;
    P.half_over_dx = 0.5 / P.dx;
    if (bitset(fm, MPF3D_S_DX)) {
        float d = (float)P.dx;
        P.inv_dx2 = 1.0 / (double)(d * d);
    } else {
        P.inv_dx2 = 1.0 / (P.dx * P.dx);
    }
    P.p32 = bitset(fm, MPF3D_S_P_ROUND);
    P.pp = P.p32 ? (double)((float)P.p_round * (float)P.p_round) : P.p_round * P.p_round;
    P.mu_da = (bitset(fm, MPF3D_S_MU_A) && bitset(fm, MPF3D_S_DELTA_A))
                  ? (double)((float)P.mu_a * (float)P.delta_a)
                  : P.mu_a * P.delta_a;
    P.eps0sq = bitset(fm, MPF3D_S_EPS0_SL) ? (double)((float)P.eps0 * (float)P.eps0) : P.eps0 * P.eps0;
    P.r_dx = safe_reciprocal(P.dx);
    P.r_two_dx = safe_reciprocal(P.two_dx);
    // float32 squares of differences are within 1e-6 of exact; a threshold
    // outside float32's normal range settles nothing
    const double lo = P.g2_floor * P.two_dx * P.two_dx * (1.0 - 1.0e-5);
    P.floor_lo = lo > 1e-30 && lo < 1e30 ? (float)lo : 0.0f;
    P.cos_lo = P.theta_c > 0.0 && P.theta_c < 3.0 ? cos(P.theta_c) - 1.0e-9 : -2.0;
    P.a0_32 = bitset(fm, MPF3D_S_A0);
    P.dT32 = (temp_dtype == MPF3D_F32) && bitset(fm, MPF3D_S_T_MELT);
    P.df32 = P.dT32 && bitset(fm, MPF3D_S_SF);
    P.switchable = switchable;
    P.use_aniso = switchable ? (enable_anisotropy != 0) : 1;
    P.use_torque = switchable ? (enable_anisotropy != 0 && enable_torque != 0) : 1;
    cudaStream_t s = (cudaStream_t)stream;
    if (phi_dtype == MPF3D_F32 && temp_dtype == MPF3D_F32)
        launch_update<float, float>(phi, phi_new, temp, mf, nf, wij, aij, mij, n111, P, err, s);
    else if (phi_dtype == MPF3D_F32)
        launch_update<float, double>(phi, phi_new, temp, mf, nf, wij, aij, mij, n111, P, err, s);
    else if (temp_dtype == MPF3D_F32)
        launch_update<double, float>(phi, phi_new, temp, mf, nf, wij, aij, mij, n111, P, err, s);
    else
        launch_update<double, double>(phi, phi_new, temp, mf, nf, wij, aij, mij, n111, P, err, s);
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}

extern "C" int mpf3d_dense_temp(void *temp, int temp_dtype, double rate, int rate_is_f32, int64_t n, void *stream) {
    if (!temp || n < 0) return MPF3D_ERR_ARG;
    if (n == 0) return MPF3D_OK;
    if (rate_is_f32) rate = (double)(float)rate;
    cudaStream_t s = (cudaStream_t)stream;
    int blocks = (int)((n + 255) / 256);
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (temp_dtype == MPF3D_F32)
        temp_kernel<float><<<blocks, 256, 0, s>>>((float *)temp, rate, rate_is_f32, n);
    else if (temp_dtype == MPF3D_F64)
        temp_kernel<double><<<blocks, 256, 0, s>>>((double *)temp, rate, rate_is_f32, n);
    else
        return MPF3D_ERR_DTYPE;
    return cudaGetLastError() == cudaSuccess ? MPF3D_OK : MPF3D_ERR_CUDA;
}
