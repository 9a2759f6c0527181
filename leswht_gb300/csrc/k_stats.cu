// Running time averages of field_avg (misc_hist.f90:287-527): after each step
// with time > AVG_TST, dt-weighted sums of the cell-centre velocity, pressure,
// temperature, their products, the vorticity and S:S are added to
// LESGPU_NAVG accumulators.  One thread per cell reads the staggered
// neighbours once and updates the 21 (23 with temperature) sums in place.
// 90x81x96: 287 us with the gradients written out, 128 with the 1-D weights
// and the time step multiplied into one factor of each product.
#include "k_grad64.cuh"

namespace lg {

__global__ void __launch_bounds__(kThreads) k_field_avg(KP p, Box b, double *avg) {
    chained();
    const DGrid &g = p.g;
    const DScal *S = p.S;
    if (!(S->time > p.c.avg_tst)) return;          // field_avg returns while time <= AVG_TST
    const double dt = S->dt;
    const double *u = p.f.u, *v = p.f.v, *w = p.f.w, *pp = p.f.p, *t = p.f.t;
    const long long n = b.count(), nt = g.nt, sx = g.sx, sxy = g.sxy;
    if (blockIdx.x == 0 && threadIdx.x == 0) p.S->avg_count += 1;
    for (long long tt = (long long)blockIdx.x * blockDim.x + threadIdx.x; tt < n; tt += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        b.at(tt, i, j, k);
        const long long q = g.ix(i, j, k);
        double *A = avg + q;
        auto acc = [&](int a, double x, double y) { A[a * nt] = fma(x, y, A[a * nt]); };
        const double ucc = 0.5 * (u[q] + u[q + 1]);
        const double vcc = 0.5 * (v[q] + v[q + sx]);
        const double wcc = 0.5 * (w[q] + w[q + sxy]);
        const double ud = ucc * dt, vd = vcc * dt, wd = wcc * dt, pd = pp[q] * dt;
        acc(0, ucc, dt);
        acc(1, vcc, dt);
        acc(2, wcc, dt);
        acc(3, ucc, ud);
        acc(4, vcc, ud);
        acc(5, wcc, ud);
        acc(6, vcc, vd);
        acc(7, wcc, vd);
        acc(8, wcc, wd);
        acc(9, pp[q], dt);
        acc(10, pp[q], pd);
        if (p.c.ihtrans == 1) {
            acc(21, t[q], dt);
            acc(22, t[q], t[q] * dt);
        }
        // velocity gradients at the cell centre (misc_hist.f90:379-455)
        double a[9];
        velgrad64<false>(p, i, j, k, u, v, w, a);
        const double s2 = 0.5 * (a[3] + a[1]), s3 = 0.5 * (a[6] + a[2]), s5 = 0.5 * (a[7] + a[5]);
        const double wx = a[5] - a[7], wy = a[6] - a[2], wz = a[1] - a[3];
        const double xd = wx * dt, yd = wy * dt, zd = wz * dt;
        acc(11, wx, dt);
        acc(12, wy, dt);
        acc(13, wz, dt);
        acc(14, wx, xd);
        acc(15, wy, xd);
        acc(16, wz, xd);
        acc(17, wy, yd);
        acc(18, wz, yd);
        acc(19, wz, zd);
        const double srsr = fma(2.0, s2 * s2 + s3 * s3 + s5 * s5, a[0] * a[0] + a[4] * a[4] + a[8] * a[8]);
        acc(20, srsr, dt);
    }
}

void launch_field_avg(lesgpu_case *c) {
    const DGrid &g = c->kp.g;
    Box b{1, 1, 1, g.n1m, g.n2m, g.n3m};
    chain(k_field_avg, blocks_for(b.count()), kThreads, 0, c->stream)(c->kp, b, c->kp.f.avg);
}

}  // namespace lg
