// diagnostics.cu — on-device reductions for the reference's statistics and Nusselt outputs.
//
// output/output_statis.cu copies whole fields to the host every NDIAG/NNUOUT steps and loops over
// them serially.  Here one coalesced pass produces, for every x plane, the ten sums the three
// diagnostics need; the host then applies the reference's formulas to lx*10 numbers.  Partial sums
// are combined in a fixed order, so results are deterministic run to run.
//   q0  sum over fluid nodes of ux*phi           (output_nu, output_statis.cu:128-153)
//   q1  number of fluid nodes
//   q2  sum over solid nodes of ux*phi
//   q3  number of solid nodes
//   q4  wall sum: (T_HOT - phi)/0.5 at x = 0, (phi - T_COLD)/0.5 at x = LX-1, fluid nodes only
//   q5  wall count
//   q6..q9  sums of ux, uy, uz, phi with solid nodes replaced by the rigid-body velocity and the
//           particle temperature (overwrite_particle_nodes, output_statis.cu:5-60)
#include "collide64.cuh"
#include "rbtp_internal.cuh"

namespace rbtp {

namespace {

constexpr int PLANE_TX = 128;

// Sums of plane ix over row chunk `chunk` of nchunks (rows = (y, z) pairs in z-major order), in row order.
// The rows are loaded PLANE_ROWS at a time ahead of their sums, node counts are integers, and
// the row's (y, z) is carried along (a 64-bit division per row and one row in flight took 620 us
// at 320x320x160 instead of the 90 us that memory needs; the FP64 additions take 140).
constexpr int PLANE_ROWS = 4;
__device__ __forceinline__ void plane_partial_body(const Geo &geo, const Phys &ph, const double *ux,
                                                   const double *uy, const double *uz, const double *phi,
                                                   const int *owner, const double *pst, int np,
                                                   double *partials, int nchunks, int ix, int chunk)
{
    const long long rows = (long long)geo.ly * geo.lz;
    const long long r0 = rows * chunk / nchunks;
    const int nrows = (int)(rows * (chunk + 1) / nchunks - r0);
    double q[NPLANEQ];
#pragma unroll
    for (int k = 0; k < NPLANEQ; ++k) q[k] = 0.0;
    int nfluid = 0, nsolid = 0;
    int iz = (int)(r0 / geo.ly), iy = (int)(r0 - (long long)iz * geo.ly);
    const long long base = r0 * geo.lx + ix;   // rows of all planes follow one another
    for (int r = 0; r < nrows; r += PLANE_ROWS) {
        double us[PLANE_ROWS], vs[PLANE_ROWS], ws[PLANE_ROWS], Ts[PLANE_ROWS];
        int owns[PLANE_ROWS];
#pragma unroll
        for (int k = 0; k < PLANE_ROWS; ++k) {
            const long long idx = base + (long long)min(r + k, nrows - 1) * geo.lx;
            us[k] = ux[idx]; vs[k] = uy[idx]; ws[k] = uz[idx]; Ts[k] = phi[idx];
            owns[k] = owner ? owner[idx] : -1;
        }
#pragma unroll
        for (int k = 0; k < PLANE_ROWS; ++k) {
            if (r + k >= nrows) break;
            const double u = us[k], v = vs[k], w = ws[k], T = Ts[k];
            const int own = owns[k];
            if (own < 0) {
                q[0] += u * T;
                ++nfluid;
                if (ix == 0) q[4] += (ph.thot - T) / 0.5;
                else if (ix == geo.lx - 1) q[4] += (T - ph.tcold) / 0.5;
                q[6] += u; q[7] += v; q[8] += w; q[9] += T;
            } else {
                q[2] += u * T;
                ++nsolid;
                if (own < np) {
                    const double relx = ((double)ix + 0.5) - pst[0 * (long long)np + own];
                    const double rely = ((double)iy + 0.5) - pst[1 * (long long)np + own];
                    const double relz = ((double)iz + 0.5) - pst[2 * (long long)np + own];
                    const double wx = pst[18 * (long long)np + own], wy = pst[19 * (long long)np + own],
                                 wz = pst[20 * (long long)np + own];
                    q[6] += pst[3 * (long long)np + own] + (relz * wy - rely * wz);
                    q[7] += pst[4 * (long long)np + own] + (relx * wz - relz * wx);
                    q[8] += pst[5 * (long long)np + own] + (rely * wx - relx * wy);
                    q[9] += pst[30 * (long long)np + own];
                } else {
                    q[6] += u; q[7] += v; q[8] += w; q[9] += T;
                }
            }
            if (++iy == geo.ly) { iy = 0; ++iz; }
        }
    }
    q[1] = (double)nfluid;
    q[3] = (double)nsolid;
    q[5] = ix == 0 || ix == geo.lx - 1 ? (double)nfluid : 0.0;
#pragma unroll
    for (int k = 0; k < NPLANEQ; ++k) partials[((long long)chunk * NPLANEQ + k) * geo.lx + ix] = q[k];
}

__global__ void __launch_bounds__(PLANE_TX) k_plane_partial(const Geo geo, const Phys ph,
                                                            const double *ux, const double *uy,
                                                            const double *uz, const double *phi,
                                                            const int *owner, const double *pst,
                                                            int np, double *partials, int nchunks)
{
    const int ix = blockIdx.x * PLANE_TX + threadIdx.x;
    if (ix >= geo.lx) return;
    plane_partial_body(geo, ph, ux, uy, uz, phi, owner, pst, np, partials, nchunks, ix, blockIdx.y);
}

// Sum of output t over the chunks, deterministic and the same in the single-cavity and the batched
// reductions: FINAL_PARTS threads each add a contiguous part of the chunks in ascending order, and the
// parts' sums are added in order (512 chunks in one chain of additions took 68 us).  Called by all
// threads of a (FINAL_OUTS, FINAL_PARTS) block; the result is valid in the threads with y = 0.
constexpr int FINAL_OUTS = 32, FINAL_PARTS = 16;
__device__ __forceinline__ double plane_final_body(const double *partials, int nchunks, int lx, int t,
                                                   double (&sh)[FINAL_PARTS][FINAL_OUTS])
{
    const int part = threadIdx.y, c0 = nchunks * part / FINAL_PARTS, c1 = nchunks * (part + 1) / FINAL_PARTS;
    double s = 0.0;
    if (t < NPLANEQ * lx) {
#pragma unroll 4
        for (int c = c0; c < c1; ++c) s += partials[(long long)c * NPLANEQ * lx + t];
    }
    sh[part][threadIdx.x] = s;
    __syncthreads();
    if (part == 0)
        for (int k = 1; k < FINAL_PARTS; ++k) s += sh[k][threadIdx.x];
    __syncthreads();
    return s;
}

__global__ void __launch_bounds__(FINAL_OUTS * FINAL_PARTS) k_plane_final(const Geo geo, const double *partials,
                                                                          int nchunks, double *plane)
{
    __shared__ double sh[FINAL_PARTS][FINAL_OUTS];
    const int t = blockIdx.x * FINAL_OUTS + threadIdx.x;
    const double s = plane_final_body(partials, nchunks, geo.lx, t, sh);
    if (threadIdx.y == 0 && t < NPLANEQ * geo.lx) plane[t] = s;
}

// Batched sampling, after the step's advance: cavities with samp_now set reduce their current
// macroscopic fields (owners of the new solid flags, particle state after the update) exactly as
// the single-cavity reduction does; the first pass also counts the sample, and the final pass writes
// (step, plane sums) into its slot of the cavity's sample ring.
__global__ void __launch_bounds__(PLANE_TX) k_batch_sample_partial(const CavDesc *desc)
{
    pdl_wait();
    pdl_trigger();
    const CavDesc &d = desc[blockIdx.y];
    if (!d.samp_now) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) d.status->nsamp += 1;
    const int *owner = d.pb.np > 0 ? d.owner[d.ocur] : nullptr;
    for (int chunk = blockIdx.x; chunk < d.nchunks; chunk += gridDim.x)
        for (int ix = threadIdx.x; ix < d.geo.lx; ix += PLANE_TX)
            plane_partial_body(d.geo, d.ph, d.ux, d.uy, d.uz, d.phi, owner, d.pb.state, d.pb.np, d.partials,
                               d.nchunks, ix, chunk);
}

__global__ void __launch_bounds__(FINAL_OUTS * FINAL_PARTS) k_batch_sample_final(const CavDesc *desc)
{
    pdl_wait();
    pdl_trigger();
    __shared__ double sh[FINAL_PARTS][FINAL_OUTS];
    const CavDesc &d = desc[blockIdx.y];
    if (!d.samp_now) return;
    const int lx = d.geo.lx;
    const int slot = (d.status->nsamp - 1) % d.samp_cap;
    double *dst = d.samp + (long long)slot * (1 + NPLANEQ * lx);
    for (int t0 = blockIdx.x * FINAL_OUTS; t0 < NPLANEQ * lx; t0 += gridDim.x * FINAL_OUTS) {
        const int t = t0 + threadIdx.x;
        const double s = plane_final_body(d.partials, d.nchunks, lx, t, sh);
        if (threadIdx.y == 0 && t < NPLANEQ * lx) dst[1 + t] = s;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && threadIdx.y == 0) dst[0] = (double)d.istep;
}

// Second moments of f and first moments of g at one node, sums over the columns of equal (cx, cy); T is
// int64_t (exact sums on the values' grid, fixed64.cuh) or double.
template <class T>
struct NodeSums {
    T xx, yy, zz, xy, xz, yz, gx, gy, gz;
};
template <class T, class F, class G>
__device__ __forceinline__ NodeSums<T> node_sums(F &&f, G &&g)
{
    NodeSums<T> s{};
    unroll<9>([&](auto C) {
        constexpr int cx = decltype(C)::value / 3 - 1, cy = decltype(C)::value % 3 - 1;
        constexpr std::integral_constant<int, dir_at(cx, cy, 0)> O{};
        constexpr std::integral_constant<int, dir_at(cx, cy, 1)> P{};
        constexpr std::integral_constant<int, dir_at(cx, cy, -1)> N{};
        const T p = f(P), n = f(N), tzz = p + n, tz = p - n, t0 = tzz + f(O);
        if constexpr (cx != 0) s.xx += t0;
        if constexpr (cy != 0) s.yy += t0;
        s.zz += tzz;
        if constexpr (cx * cy == 1) s.xy += t0;
        if constexpr (cx * cy == -1) s.xy -= t0;
        if constexpr (cx == 1) s.xz += tz;
        if constexpr (cx == -1) s.xz -= tz;
        if constexpr (cy == 1) s.yz += tz;
        if constexpr (cy == -1) s.yz -= tz;
        const T gp = g(P), gn = g(N);
        s.gz += gp - gn;
        if constexpr (cx != 0 || cy != 0) {
            const T g0 = gp + gn + g(O);
            if constexpr (cx == 1) s.gx += g0;
            if constexpr (cx == -1) s.gx -= g0;
            if constexpr (cy == 1) s.gy += g0;
            if constexpr (cy == -1) s.gy -= g0;
        }
    });
    return s;
}

// compute_Ked (collision.cu:91-152) and compute_ted (collision.cu:154-198) on the FP64 copy of
// the step's post-collision populations; solid nodes are then zeroed as output_flow does.  The
// reference subtracts the equilibrium direction by direction; its second and third moments are
// known (sum c_a c_b feq = r d_ab / 3 + u_a u_b, sum c_a c_b c_k feq F_k = (u_a F_b + u_b F_a +
// u.F d_ab) / 3, sum c_a geqnew = phi u_a), so only the moments of the populations are summed, on the
// integer units (160x160x80: 4.25 -> 0.32 ms; the differences of large and nearly equal terms are fewer,
// so the result is also closer to the exact one).
__global__ void __launch_bounds__(128) k_dissipation(const Geo geo, const Phys ph, const double *fcol, const double *gcol,
                              const double *rho, const double *ux, const double *uy,
                              const double *uz, const double *phi, const void *faux, bool aux32,
                              const int *owner, double *ted, double *ked)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= geo.L) return;
    const long long L = geo.L;
    double f[27], g[27];
    unroll<27>([&](auto I) {
        f[I] = fcol[(long long)I * L + idx];
        g[I] = gcol[(long long)I * L + idx];
    });
    const double fx = aux32 ? (double)static_cast<const float *>(faux)[idx] : static_cast<const double *>(faux)[idx];
    const double r = rho[idx], ph_ = phi[idx];
    const double u = ux[idx], v = uy[idx], w = uz[idx];
    uint32_t tf = FX_TOP_MIN, tg = FX_TOP_MIN;
    unroll<13>([&](auto K) {
        fx_cover(tf, f[2 * K + 1], f[2 * K + 2]);
        fx_cover(tg, g[2 * K + 1], g[2 * K + 2]);
    });
    fx_cover(tf, f[0], f[0]);
    fx_cover(tg, g[0], g[0]);
    NodeSums<double> s;
    if (max(tf, tg) < FX_TOP_MAX) {
        const uint32_t gf = fx_grid(tf), gg = fx_grid(tg);
        const NodeSums<int64_t> i = node_sums<int64_t>([&](auto I) { return fx_from(f[I], gf); },
                                                       [&](auto I) { return fx_from(g[I], gg); });
        s = {fx_to(i.xx, gf), fx_to(i.yy, gf), fx_to(i.zz, gf), fx_to(i.xy, gf), fx_to(i.xz, gf), fx_to(i.yz, gf),
             fx_to(i.gx, gg), fx_to(i.gy, gg), fx_to(i.gz, gg)};
    } else {
        s = node_sums<double>([&](auto I) { return f[I]; }, [&](auto I) { return g[I]; });
    }
    // F = (fx, 0, 0); the force term is 3/2 (sum c_a c_b c.F feq - (F.u) sum c_a c_b feq)
    const double bu = fx * u, r3 = r * (1.0 / 3.0);
    const double txx = (s.xx - (r3 + u * u)) + 1.5 * (bu - bu * (r3 + u * u));
    const double tyy = (s.yy - (r3 + v * v)) + 1.5 * (bu * (1.0 / 3.0) - bu * (r3 + v * v));
    const double tzz = (s.zz - (r3 + w * w)) + 1.5 * (bu * (1.0 / 3.0) - bu * (r3 + w * w));
    const double txy = (s.xy - u * v) + 0.5 * v * fx - 1.5 * bu * (u * v);
    const double txz = (s.xz - u * w) + 0.5 * w * fx - 1.5 * bu * (u * w);
    const double tyz = (s.yz - v * w) - 1.5 * bu * (v * w);
    // S_ab = -(1 - 1/(2 tau)) t_ab / (2 visc)
    const double k = (1.0 - 0.5 / ph.tau) / (2.0 * ph.visc);
    double kv = 0.5 * ph.visc * (k * k) *
                (4.0 * (txx * txx + tyy * tyy + tzz * tzz) + 8.0 * (txy * txy + txz * txz + tyz * tyz));
    const double inv = 1.0 / (2.0 * ph.tauc * (1.0 / 3.0) + r3);
    const double tx = (2.0 * (s.gx - ph_ * u) + ph_ * fx) * inv;
    const double ty = 2.0 * (s.gy - ph_ * v) * inv;
    const double tz = 2.0 * (s.gz - ph_ * w) * inv;
    double tv = (ph.diff > 0.0) ? ph.diff * (tx * tx + ty * ty + tz * tz) : 0.0;
    if (owner && owner[idx] >= 0) { kv = 0.0; tv = 0.0; }
    ked[idx] = kv;
    ted[idx] = tv;
}

}  // namespace

cudaError_t launch_batch_sample(const CavDesc *desc, int n, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    cudaError_t e = pdl_launch(k_batch_sample_partial, dim3(64, n), dim3(PLANE_TX), st, desc);
    if (e != cudaSuccess) return e;
    return pdl_launch(k_batch_sample_final, dim3(16, n), dim3(FINAL_OUTS, FINAL_PARTS), st, desc);
}

cudaError_t launch_plane_sums(const Geo &geo, const Phys &ph, const double *ux, const double *uy,
                              const double *uz, const double *phi, const int *owner,
                              const double *pstate, int np, double *partials, int nchunks,
                              double *plane, cudaStream_t st)
{
    const dim3 grd((geo.lx + PLANE_TX - 1) / PLANE_TX, nchunks, 1);
    k_plane_partial<<<grd, PLANE_TX, 0, st>>>(geo, ph, ux, uy, uz, phi, owner, pstate, np, partials, nchunks);
    const int n = NPLANEQ * geo.lx;
    k_plane_final<<<(n + FINAL_OUTS - 1) / FINAL_OUTS, dim3(FINAL_OUTS, FINAL_PARTS), 0, st>>>(geo, partials, nchunks, plane);
    return cudaGetLastError();
}

cudaError_t launch_dissipation(int mode, const Geo &geo, const Phys &ph, const double *fcol,
                               const double *gcol, const double *rho, const double *ux,
                               const double *uy, const double *uz, const double *phi,
                               const void *faux, const int *owner, double *ted, double *ked,
                               cudaStream_t st)
{
    k_dissipation<<<(unsigned)((geo.L + 127) / 128), 128, 0, st>>>(geo, ph, fcol, gcol, rho, ux, uy, uz, phi, faux,
                                                                   mode != RBTP_STORE_F64, owner, ted, ked);
    return cudaGetLastError();
}

}  // namespace rbtp
