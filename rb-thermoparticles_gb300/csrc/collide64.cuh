// collide64.cuh — moments and collision of one FP64 node on the integer units (fixed64.cuh).
#pragma once

#include "fixed64.cuh"
#include "rbtp_internal.cuh"

namespace rbtp {

// Place p = 9 (cy + 1) + 3 (cx + 1) + (cz + 1) of a direction: three slabs of equal cy, whose code is
// shared by a loop; the opposite direction sits at 26 - p.
__host__ __device__ constexpr int place_cx(int p) { return p / 3 % 3 - 1; }
__host__ __device__ constexpr int place_cy(int p) { return p / 9 - 1; }
__host__ __device__ constexpr int place_cz(int p) { return p % 3 - 1; }
__host__ __device__ constexpr int place_dir(int p)
{
    for (int i = 0; i < 27; ++i)
        if (dcx(i) == place_cx(p) && dcy(i) == place_cy(p) && dcz(i) == place_cz(p)) return i;
    return -1;
}
// direction index of (cx, cy, cz)
__host__ __device__ constexpr int dir_at(int cx, int cy, int cz)
{
    return place_dir(9 * (cy + 1) + 3 * (cx + 1) + cz + 1);
}
// number of nonzero components of (cx, cz) at place q of a slab
__host__ __device__ constexpr int slab_class(int q) { return (q / 3 != 1) + (q % 3 != 1); }

// times two: the exponent one up.  A zero becomes 2^-1022, which vanishes on any grid; infinities and NaN stay what
// they are (the plain path has to spread them as FP64 formulas do), and what overflows becomes one of them.
// A selection: an FP64 addition for such values alone cost 1.5 % of the step, as a branch too.
__host__ __device__ __forceinline__ double fx_twice(double d)
{
    const uint32_t hi = fx_hi(d);
    return fx_double(hi + ((hi & 0x7fffffffu) < 0x7ff00000u ? 1u << 20 : 0u), fx_lo(d));
}

// Weights in units of 1/108: exponent of class c (number of nonzero components).
__host__ __device__ constexpr int up64(int c) { return 5 - 2 * c; }

// The largest fx_mag of the 27 values at val[p * stride], as they are and over 2^up64 of their class.
struct Tops64 {
    uint32_t all, weighted;
};
__host__ __device__ __forceinline__ Tops64 tops64(const double *val, int stride)
{
    Tops64 r{FX_TOP_MIN, FX_TOP_MIN};
#pragma unroll 1
    for (int s = 0; s < 3; ++s, val += 9 * stride) {
        uint32_t t[3] = {0u, 0u, 0u};
        t[0] = fx_mag(val[4 * stride]);
        fx_cover(t[1], val[stride], val[3 * stride]);
        fx_cover(t[1], val[5 * stride], val[7 * stride]);
        fx_cover(t[2], val[0], val[2 * stride]);
        fx_cover(t[2], val[6 * stride], val[8 * stride]);
        const uint32_t up = (s == 1 ? 5u : 3u) << 20;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (t[c] < FX_TOP_MIN) t[c] = FX_TOP_MIN;
            const uint32_t w = t[c] - up + ((uint32_t)(2 * c) << 20);
            r.all = t[c] > r.all ? t[c] : r.all;
            r.weighted = w > r.weighted ? w : r.weighted;
        }
    }
    return r;
}

// Zeroth and first moments of the 27 values on one grid: exact sums along z, then x, then y.
__host__ __device__ __forceinline__ void moments64(const double *val, int stride, uint32_t grid, double &m0, double &mx,
                                                   double &my, double &mz)
{
    int64_t i0 = 0, ix = 0, iy = 0, iz = 0;
#pragma unroll 1
    for (int s = 0; s < 3; ++s, val += 9 * stride) {
        int64_t t[3], d[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int64_t n = fx_from(val[3 * k * stride], grid), p = fx_from(val[(3 * k + 2) * stride], grid);
            t[k] = n + p + fx_from(val[(3 * k + 1) * stride], grid);
            d[k] = p - n;
        }
        const int64_t all = t[0] + t[1] + t[2];
        i0 += all;
        ix += t[2] - t[0];
        iz += d[0] + d[1] + d[2];
        if (s == 0) iy = -all;
        if (s == 2) iy += all;
    }
    m0 = fx_to(i0, grid);
    mx = fx_to(ix, grid);
    my = fx_to(iy, grid);
    mz = fx_to(iz, grid);
}

// Both BGK collisions (collision.cu:3-89).  With v = 3u, P_i = c_i.v + (c_i.v)^2 / 2 - v^2 / 6 they are
//   f*_i = om  f_i + w_i [ rho/tau - G u_x + k1 P_i + c_ix G (1 + P_i) ],  k1 = 1/tau - G u_x
//   g*_i = omc g_i + w_i [ p (1 + rho + P_i) + c_i.V ],  p = phi/tauc  (i = 0: less p rho in all),
// polynomials in c_i whose coefficients are computed in FP64 once per node, over 108 (coef64_f,
// coef64_g); relax64 evaluates them by integer additions on the coefficients' grid; the weight
// w_i = {32, 8, 2, 1/2} / 108 is an exponent, and so are the factors 2 of the coefficients.
// om f_i joins the sum on the same grid, and the result is rounded once.
//
// 1/tau and the weights enter as the products of their rounded values, as in the reference's
// formulas: a constant that folds both would shift mass and heat by its own rounding in every step.
constexpr double W108 = 1.0 / 108.0;

// v, its products and v^2 / 6.  The sixth is taken in two parts: 1/6 rounded to a double is 5.5e-17 too small, and
// the mass that sum_i w_i ((c_i.v)^2 / 2 - v^2 / 6) = 0 leaves unchanged would grow by that much of v^2 in every
// step (a closed 16x12x8 cavity, Ra 1e5, 20,000 steps: +1.1e-12, and 6e-15 with both parts).
constexpr double SIXTH = 1.0 / 6.0, SIXTH_REST = 0x1.5555555555555p-57;
struct Vel64 {
    double x, y, z, xx, yy, zz, xy, xz, yz, s;
};
__host__ __device__ __forceinline__ Vel64 vel64(double ux, double uy, double uz)
{
    Vel64 v;
    v.x = 3.0 * ux; v.y = 3.0 * uy; v.z = 3.0 * uz;
    v.xx = v.x * v.x; v.yy = v.y * v.y; v.zz = v.z * v.z;
    v.xy = v.x * v.y; v.xz = v.x * v.z; v.yz = v.y * v.z;
    const double t = v.xx + v.yy + v.zz;
    v.s = fma(t, SIXTH, t * SIXTH_REST);
    return v;
}
// Coefficients: rest, constant, xx, yy, zz, xy, xz, yz (even), x, y, z (odd), and for f the odd xyy, xzz, xxy,
// xxz, xyz.
constexpr int NCOEF64 = 16;
__host__ __device__ __forceinline__ void coef64_f(double (&c)[NCOEF64], double rho, double ux, double Fx, const Vel64 &v,
                                                  const StepK<double> &K)
{
    const double G = K.Gcw * Fx, G2 = fx_twice(G), Gux = G * ux;
    const double k1 = fma(K.tinv, 0.5 * W108, -Gux), k2 = fx_twice(k1);
    c[0] = c[1] = fx_twice(fma(-v.s, k1, fma(rho * K.tinv, 0.5 * W108, -Gux)));
    c[2] = fma(k1, v.xx, G2 * v.x);
    c[3] = k1 * v.yy;
    c[4] = k1 * v.zz;
    c[5] = fma(k2, v.xy, G2 * v.y);
    c[6] = fma(k2, v.xz, G2 * v.z);
    c[7] = k2 * v.yz;
    c[8] = fma(G2, fma(0.5, v.xx, 1.0 - v.s), k2 * v.x);
    c[9] = k2 * v.y;
    c[10] = k2 * v.z;
    c[11] = G * v.yy;
    c[12] = G * v.zz;
    c[13] = G2 * v.xy;
    c[14] = G2 * v.xz;
    c[15] = G2 * v.yz;
}
// What g's coefficients take before the velocity products: p, p (1 + rho), p rho / 32 and the vector V.
struct Src64 {
    double p, pr, rest, x, y, z;
};
__host__ __device__ __forceinline__ Src64 src64(double rho, double ux, double uy, double uz, double phi, double Fx,
                                                double kx, double ky, double kz, const StepK<double> &K)
{
    Src64 s;
    const double pt = phi * K.tcinv;
    s.p = pt * (0.5 * W108);
    s.pr = fma(s.p, rho, s.p);
    s.rest = pt * rho;
    const double rgd = rho / fma(rho, 1.0 / 3.0, K.gd0), c2 = rgd * K.Rcw2;
    s.x = fma(c2, fma(-phi, ux, kx), K.Rcw * Fx * phi * (3.0 - rgd));
    s.y = c2 * fma(-phi, uy, ky);
    s.z = c2 * fma(-phi, uz, kz);
    return s;
}
__host__ __device__ __forceinline__ void coef64_g(double (&c)[NCOEF64], const Src64 &s, const Vel64 &v)
{
    const double p = s.p, p2 = fx_twice(p);
    c[1] = fx_twice(fma(-v.s, p, s.pr));
    c[0] = fma(s.rest, -1.0 / 32.0, c[1]);
    c[2] = p * v.xx;
    c[3] = p * v.yy;
    c[4] = p * v.zz;
    c[5] = p2 * v.xy;
    c[6] = p2 * v.xz;
    c[7] = p2 * v.yz;
    c[8] = fma(p2, v.x, s.x);
    c[9] = fma(p2, v.y, s.y);
    c[10] = fma(p2, v.z, s.z);
    c[11] = c[12] = c[13] = c[14] = c[15] = 0.0;
}

// The collided population om val + w X of every place 9 s + q, handed to out(s, r[9]) slab by slab
// (s = cy + 1; UNROLL slabs per round of the loop).  `weighted` is that of tops64.  False, with nothing
// handed out, where a coefficient is too large for the grids (or not finite).
template <int UNROLL, class Out>
__host__ __device__ __forceinline__ bool relax64(const double *val, int stride, double omega, uint32_t weighted,
                                                 const double (&c)[NCOEF64], Out &&out)
{
    // the grid also holds om f_i over the weights, which stay below 2^62 units from 3 exponents above
    // the coefficients'
    uint32_t top = weighted - (3u << 20);
#pragma unroll
    for (int k = 0; k < NCOEF64; k += 2) fx_cover(top, c[k], c[k + 1]);
    if (top >= FX_TOP_MAX) return false;
    const uint32_t grid = fx_grid(top);
    int64_t a[NCOEF64];
#pragma unroll
    for (int k = 0; k < NCOEF64; ++k) a[k] = fx_from(c[k], grid);
    const FxFactor om = fx_factor(omega);
#pragma unroll UNROLL
    for (int s = 0; s < 3; ++s, val += 9 * stride) {
        // the polynomial of this slab: cy = s - 1
        int64_t k0 = a[1], kx = a[8], kz = a[10], kxx = a[2], kxz = a[6];
        if (s == 0) {
            k0 += a[3] - a[9]; kx += a[11] - a[5]; kz -= a[7]; kxx -= a[13]; kxz -= a[15];
        }
        if (s == 2) {
            k0 += a[3] + a[9]; kx += a[11] + a[5]; kz += a[7]; kxx += a[13]; kxz += a[15];
        }
        int64_t x[9];
        const int64_t e = k0 + kxx;
        x[1] = e - kx;
        x[4] = k0;
        x[7] = e + kx;
        const int64_t zp = kz + a[14], ep = x[7] + a[4] + a[12], em = x[1] + a[4] - a[12];
        x[3] = k0 + a[4] - kz;
        x[5] = k0 + a[4] + kz;
        x[6] = ep - zp - kxz;
        x[8] = ep + zp + kxz;
        x[0] = em - zp + kxz;
        x[2] = em + zp - kxz;
        if (s == 1) x[4] = a[0];
        // weights of the slab: up64 of class slab_class + (cy != 0)
        const uint32_t slab = grid - (s == 1 ? 0u : 2u << 20);
        double r[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) r[q] = val[q * stride];
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const int up = up64(slab_class(q));
            r[q] = fx_to(fx_times(om, r[q], fx_places(om, slab, up)) + x[q], slab, up);
        }
        out(s, r);
    }
    return true;
}

}  // namespace rbtp
