// step_node64.cuh — the per-node body of the fused step for FP64 storage (slots, walls and parities as
// in step_node.cuh, which covers the float modes).
#pragma once

#include "collide64.cuh"
#include "step_node.cuh"

namespace rbtp {

// An FP64 step block (32, 1, 2): 32 consecutive nodes of a row or plane, two threads each, one for f
// (threadIdx.z = 0) and one for g, so that a warp of f works beside its partner warp of g.  Shared
// memory: the 27 populations of thread t at [place][t] (places of collide64.cuh), and what the two
// threads of a node exchange.  A block is one warp pair, whose shared memory is free again when its
// slower warp is done (four pairs: 4.65 against 4.45 ms per step at 320x320x160, and 1.41 against
// 1.35 ms for a batch of 32 members of 32 to 96 nodes across).
constexpr int STEP64_NODES = 32;
constexpr int STEP64_SWAP = 16;      // doubles exchanged per node
constexpr int STEP64_DOUBLES = (27 * 2 + STEP64_SWAP) * STEP64_NODES;
// Resident blocks per SM that the kernels ask registers for: 9 (up to 112 per thread), the best of 8 to 12 where a
// grid has several waves (320x320x160 at 12 | 11 | 10 | 9 | 8: 4.66 | 4.64 | 4.42 | 4.38 | 4.90 ms per step;
// 113x97x59 212 | 211 | 190 | 191 | 205 us), 12 (80 per thread, all that shared memory allows) for some
// short grids (lbm_step.cu), and 8 batched (12 | 11 | 10 | 9 | 8 | 7: 1.44 | 1.44 | 1.33 | 1.33 | 1.30 | 1.31 ms
// for 32 members of 32 to 96 nodes across).
constexpr int STEP64_BLOCKS = 9, STEP64_BLOCKS_MOST = 12, STEP64_BLOCKS_BATCHED = 8;

// Variant of the single-cavity kernel for a grid of `blocks` on a GPU of `sms` multiprocessors.
struct Step64Choice {
    bool unrolled, most;
};
// A grid of up to four waves of resident blocks runs at the latency of a block's chain of instructions,
// which unrolled slabs and fixed outputs shorten; a longer one is bound by throughput, and then the
// code with the loop stays in the instruction caches and the longer one without does not.  Within the
// short ones more resident blocks with fewer registers where that saves a wave that is more than a
// quarter full.  Measured figures in lbm_step.cu.
constexpr Step64Choice step64_choice(long long blocks, long long sms)
{
    const long long wave = sms * STEP64_BLOCKS, wave_most = sms * STEP64_BLOCKS_MOST;
    const bool unrolled = blocks <= 4 * wave;
    return {unrolled, unrolled && (blocks + wave_most - 1) / wave_most < (blocks - wave / 4 + wave - 1) / wave};
}

// eight times the direction index of a place, for loops that are not unrolled, and dir_mask by places
static __constant__ int c_place_dir8[27] = {200, 72, 168, 144, 32, 112, 208, 80, 176, 136, 24, 104, 48, 0, 40, 120, 8, 88, 192, 64, 160, 128, 16, 96, 184, 56, 152};
__host__ __device__ constexpr unsigned place_mask(int axis, int sign)
{
    unsigned m = 0;
    for (int p = 0; p < 27; ++p) {
        const int c = axis == 0 ? place_cx(p) : (axis == 1 ? place_cy(p) : place_cz(p));
        if (c == sign) m |= 1u << p;
    }
    return m;
}

__device__ __forceinline__ void copy_async8(uint32_t dst, const double *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copy_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

// Moments and collision in plain FP64 operations for the values that the grids do not take (beyond
// 2^16, infinite, not a number).
static __device__ __noinline__ void moments64_plain(const double *val, int stride, double *m)
{
    m[0] = m[1] = m[2] = m[3] = 0.0;
#pragma unroll 1
    for (int p = 0; p < 27; ++p) {
        const double v = val[p * stride];
        m[0] += v;
        if (place_cx(p)) m[1] += place_cx(p) * v;
        if (place_cy(p)) m[2] += place_cy(p) * v;
        if (place_cz(p)) m[3] += place_cz(p) * v;
    }
}
// in place; c: the coefficients over 108 of relax64
static __device__ __noinline__ void relax64_plain(double *val, int stride, double omega, const double *c)
{
#pragma unroll 1
    for (int p = 0; p < 27; ++p) {
        const int x = place_cx(p), y = place_cy(p), z = place_cz(p);
        double s = p == 13 ? c[0] : c[1];
        if (x) s += c[2];
        if (y) s += c[3];
        if (z) s += c[4];
        if (x && y) s += x * y * c[5];
        if (x && z) s += x * z * c[6];
        if (y && z) s += y * z * c[7];
        if (x) s += x * c[8];
        if (y) s += y * c[9];
        if (z) s += z * c[10];
        if (x && y) s += x * c[11] + y * c[13];
        if (x && z) s += x * c[12] + z * c[14];
        if (x && y && z) s += x * y * z * c[15];
        val[p * stride] = omega * val[p * stride] + 108.0 * dweight_rt(c_place_dir8[p] / 8) * s;
    }
}

// base + bytes of slot (i, x + off) relative to slot (0, x), for i8 = 8 i: two multiply-adds of the
// FMA pipe (the other integer instructions share the pipe that bounds the step).
__device__ __forceinline__ double *slot_at(double *base, unsigned i8, unsigned L, int off)
{
    char *const p = reinterpret_cast<char *>(base) + (unsigned long long)i8 * L;
    return reinterpret_cast<double *>(p + (long long)off * 8);
}

// One distribution of one node of the fused FP64 step.  An FP64 instruction of a warp takes 64 cycles
// of its scheduler on GB300, so the sums run on the integer units (collide64.cuh), and a step is as
// fast as enough warps keep both busy.  With the 54 populations of a node in registers (255) only two
// warps fit a scheduler; the populations therefore go from global to shared memory by cp.async, without
// passing through registers, and are read from there where they are used, and f and g of a node
// belong to two threads, which exchange the moments: four and a half warps per scheduler.  The code loops over the
// three slabs of directions: unrolled, it did not stay in the instruction caches (4.90 ms).  Measured
// at 320x320x160: 4.38 ms per step, 13.1 ms with every sum on the FP64 pipe (424 FP64 instructions
// per node there, 77.4 here; 880 B per node at the copy bandwidth would take 2.2 ms); at 64x64x32 44
// against 118 us.  What bounds it now is the latency of the chain load - integer sums - FP64
// coefficients - integer sums with the warps that fit (issue slots 60 %, integer pipe 70 %, FP64 pipe 46 % busy).  `out`
// selects the outputs (StepOut; COL: also the post-collision copies; a kernel for each value had the
// compiler unroll some, see the choice of UNROLL, the slabs per round of the collision's loop, in
// lbm_step.cu), `smem` is the block's shared memory.  Threads that are not `active` only take part in
// the barriers; they read the slots of the node they are given (which must exist).
template <bool ODD, bool COL, int UNROLL>
__device__ __forceinline__ void step_node64(const Geo &geo, const StepK<double> &K, const StepBuffers &b, int out,
                                            int ix, int iy, int iz, bool active, double *smem)
{
    constexpr int NODES = STEP64_NODES, T = 2 * NODES;
    const bool is_g = threadIdx.z != 0;
    const int tn = threadIdx.y * blockDim.x + threadIdx.x;
    double *const pop = smem + (is_g ? NODES : 0) + tn;
    double *const swap = smem + 27 * T + tn;
    const unsigned L = (unsigned)geo.L;   // below 2^31
    const int lx = geo.lx, lxy = (int)geo.lxy;
    const long long node = (long long)iz * geo.lxy + (long long)iy * geo.lx + ix;
    double *const N = static_cast<double *>(is_g ? b.g : b.f) + node;
    const bool xlo = ix == 0, xhi = ix == geo.lx - 1;
    const long long wall_slot = (xhi ? (long long)geo.lz * geo.ly : 0) + (long long)iz * geo.ly + iy;
    // Bit p of out_x / out_yz: x - c_p lies outside the box through an x face / a y or z face; the
    // scatter's neighbour x + c_p is tested as the opposite direction, bit 26 - p.
    const unsigned out_x = (xlo ? place_mask(0, 1) : 0u) | (xhi ? place_mask(0, -1) : 0u);
    const unsigned out_yz = (iy == 0 ? place_mask(1, 1) : 0u) | (iy == geo.ly - 1 ? place_mask(1, -1) : 0u) |
                            (iz == 0 ? place_mask(2, 1) : 0u) | (iz == geo.lz - 1 ? place_mask(2, -1) : 0u);
    const unsigned out_any = out_x | out_yz;

    // even step: the post-streaming f_i(x) in slot (i, x); odd step: f_i(x) = f*_i(x - c_i), swapped
    // into slot (opp(i), x - c_i), or f*_opp(i)(x) in slot (i, x) where x - c_i is outside the box
    {
        uint32_t col = (uint32_t)__cvta_generic_to_shared(pop);
        unsigned outside = out_any;
#pragma unroll 1
        for (int s = 0; s < 3; ++s, col += 9 * T * 8, outside >>= 9) {
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                const int p = 9 * s + q;
                unsigned i8 = c_place_dir8[p];
                int off = 0;
                if (ODD && !(outside >> q & 1u)) {
                    i8 = c_place_dir8[26 - p];
                    off = -(place_cx(q) + (s - 1) * lx + place_cz(q) * lxy);
                }
                copy_async8(col + q * T * 8, slot_at(N, i8, L, off));
            }
        }
        copy_async_commit();
    }
    const double fold = is_g ? 0.0 : __ldg(static_cast<const double *>(b.faux) + node);
    copy_async_wait<0>();
    // At the x walls a direction that leaves only through x takes the Dirichlet anti-bounce-back, y/z
    // exits stay adiabatic (streaming.cu:45-61).  Few nodes of a warp lie there (two where rows are longer
    // than 32), so the lanes share their images, one (node, direction) each: with every lane doing its
    // own node's nine, an odd step of such a warp had 18 rounds with FP64 instructions (32x32x16: 11.4
    // against 10.6 us per step, 64x64x32: 46.2 against 43.0, 320x320x160: 4.47 against 4.44 ms).
    // `sign`: the populations that come from outside (-1) or leave (1) along their place's direction;
    // put(the node's lane and index, place, image).
    unsigned walls = 0u;
    if constexpr (ODD) walls = is_g ? __ballot_sync(~0u, out_x != 0u && active) : 0u;
    auto images = [&](int sign, auto &&density, auto &&put) {
        const unsigned mine = (sign < 0 ? out_x & ~out_yz : __brev(out_x & ~out_yz) >> 5) | (xlo ? 1u << 27 : 0u);
        const int lane = tn & 31, items = 9 * __popc(walls);
        __syncwarp();
#pragma unroll 1
        for (int first = 0; first < items; first += 32) {
            const int j = first + lane, k = j % 9;
            unsigned rest = walls;
#pragma unroll 1
            for (int n = j / 9; n; --n) rest &= rest - 1;
            const int at = j < items ? __ffs((int)rest) - 1 : lane;
            const unsigned m = __shfl_sync(~0u, mine, at);
            const bool lo = m >> 27;
            const int p = k / 3 * 9 + k % 3 + (lo == (sign < 0) ? 6 : 0);
            const double rho_w = density(at);
            const int wall_node = __shfl_sync(~0u, (int)node, at);
            if (j < items && (m >> p & 1u))
                put(at, wall_node, p,
                    wall_image(pop[p * T + at - lane], dweight_rt(c_place_dir8[p] / 8), lo ? K.thot : K.tcold, rho_w));
        }
        __syncwarp();
    };
    // the even step's output, with the node's density of that step
    if (walls)
        images(-1, [&](int at) { return b.rho_wall[__shfl_sync(~0u, wall_slot, at)]; },
               [&](int at, int, int p, double v) { pop[p * T + at - (tn & 31)] = v; });

    // ---- moments (macrovar.cu:3-34) and forcing, F_x = g0 beta (phi - T0) ----
    const Tops64 tops = tops64(pop, T);
    double m0, mx, my, mz;
    if (tops.all < FX_TOP_MAX) {
        moments64(pop, T, fx_grid(tops.all), m0, mx, my, mz);
    } else {
        double m[4];
        moments64_plain(pop, T, m);
        m0 = m[0]; mx = m[1]; my = m[2]; mz = m[3];
        if (active && !(fabs(m0) < 1e30)) atomicOr(&b.status->nonfinite, 1);
    }
    enum { RHO, UX, UY, UZ, PHI, FX, VEL };
    if (is_g) {
        swap[PHI * NODES] = m0;
        swap[FX * NODES] = K.g0b * (m0 - K.t0);
    } else {
        swap[RHO * NODES] = m0;
        swap[UX * NODES] = fma(0.5, fold, mx);
        swap[UY * NODES] = my;
        swap[UZ * NODES] = mz;
    }
    __syncthreads();
    const double rho = swap[RHO * NODES], ux = swap[UX * NODES], Fx = swap[FX * NODES];
    if (active) {
        if (is_g) static_cast<double *>(b.faux)[node] = Fx;
        else if (out >= OUT_RHO) b.rho[node] = rho;
        if (out >= OUT_MACROS) {
            if (is_g) {
                b.phi[node] = m0;
            } else {
                b.ux[node] = ux;
                b.uy[node] = my;
                b.uz[node] = mz;
            }
        }
        // the wall densities the next (odd) step's gather and the stream export apply
        if (!ODD && !is_g && (xlo || xhi)) b.rho_wall[wall_slot] = rho;
    }

    // ---- collision: f's thread forms the velocity products, g's meanwhile its source vector ----
    double c[NCOEF64];
    Vel64 v;
    if (is_g) {
        const Src64 src = src64(rho, ux, swap[UY * NODES], swap[UZ * NODES], m0, Fx, mx, my, mz, K);
        __syncthreads();
        double *const vv = &v.x;
#pragma unroll
        for (int k = 0; k < 10; ++k) vv[k] = swap[(VEL + k) * NODES];
        coef64_g(c, src, v);
    } else {
        v = vel64(ux, my, mz);
        const double *const vv = &v.x;
#pragma unroll
        for (int k = 0; k < 10; ++k) swap[(VEL + k) * NODES] = vv[k];
        __syncthreads();
        coef64_f(c, rho, ux, Fx, v, K);
    }

    // even step: f*_i(x) swapped into the node's own slot (opp(i), x); odd step: f*_i(x) streams to
    // slot (i, x + c_i), or leaving the box becomes the next step's f_opp(i)(x) in slot (opp(i), x),
    // bounced back (and see below)
    auto scatter = [&](int s, int q, double r) {
        const int p = 9 * s + q;
        if constexpr (COL) (is_g ? b.gcol : b.fcol)[(long long)(c_place_dir8[p] / 8) * L + node] = r;
        unsigned i8 = c_place_dir8[26 - p];
        int off = 0;
        if (ODD && !(out_any >> (26 - p) & 1u)) {
            i8 = c_place_dir8[p];
            off = place_cx(q) + (s - 1) * lx + place_cz(q) * lxy;
        }
        *slot_at(N, i8, L, off) = r;
        if (ODD && is_g && out_x != 0u) pop[p * T] = r;
    };
    const double omega = is_g ? K.omc : K.om;
    if (!relax64<UNROLL>(pop, T, omega, tops.weighted, c, [&](int s, const double(&r)[9]) {
            if (active) {
#pragma unroll
                for (int q = 0; q < 9; ++q) scatter(s, q, r[q]);
            }
        })) {
        relax64_plain(pop, T, omega, c);
        if (active) {
#pragma unroll 1
            for (int p = 0; p < 27; ++p) scatter(p / 9, p % 9, pop[p * T]);
        }
    }
    // this step's output at the x walls, with this step's density: the population that left along p is
    // the next step's incoming one at 26 - p
    if (walls)
        images(1, [&](int at) { return __shfl_sync(~0u, rho, at); },
               [&](int, int n, int p, double v) {
                   *slot_at(static_cast<double *>(b.g) + n, c_place_dir8[26 - p], L, 0) = v;
               });
}

}  // namespace rbtp
