// The host side of fixed64.cuh, collide64.cuh and step_node64.cuh behind C functions, for test_fx_host.py.
#include "step_node64.cuh"

using namespace rbtp;

extern "C" {
// v^2 / 6 and the three squares of v = 3 u
void fxh_vel(const double *u, double *out)
{
    const Vel64 v = vel64(u[0], u[1], u[2]);
    out[0] = v.s;
    out[1] = v.xx;
    out[2] = v.yy;
    out[3] = v.zz;
}
unsigned fxh_grid(double largest) { return fx_grid(fx_mag(largest)); }
long long fxh_from(double d, unsigned grid) { return fx_from(d, grid); }
double fxh_to(long long v, unsigned grid, int up) { return fx_to(v, grid, up); }
long long fxh_times(double k, double d, unsigned grid, int up)
{
    const FxFactor f = fx_factor(k);
    return fx_times(f, d, fx_places(f, grid, up));
}
// bit 0: unrolled, bit 1: more resident blocks
int fxh_choice(long long blocks, long long sms)
{
    const Step64Choice c = step64_choice(blocks, sms);
    return (c.unrolled ? 1 : 0) | (c.most ? 2 : 0);
}
}
