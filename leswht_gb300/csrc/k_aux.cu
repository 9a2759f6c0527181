// Step/substep bookkeeping, global reductions, projection and pressure
// update: the routines of 02_solver/f90/lib/slv_auxi.f90, meanpg of
// slv_mmtm.f90:2-177 and the checks of misc_init.f90:1047-1104.
//
// Every global sum is a two-stage deterministic reduction: a grid whose size
// depends on the box alone strides over the cells in a fixed order, each block
// writes its partials, and the last block folds them in a fixed tree and
// applies the scalar logic of the reference routine.  The result is the same
// bit pattern on every run.
#include "lesgpu_internal.cuh"

namespace lg {

static Box interior(const DGrid &g) { return Box{1, 1, 1, g.n1m, g.n2m, g.n3m}; }

// ------------------------------------------------------------ stepinit/cfl
// cfl, slv_auxi.f90:53-102: max over cells of the cell-centre |u|/dx sum.
// The reference multiplies each cell's sum by dt before the max; dt > 0 so
// max(s)*dt is the same rounded value.
struct CflTerm {
    static constexpr int kLoads = 1;
    __device__ void load(const KP &p, int i, int j, int k, double *x) const {
        const DGrid &g = p.g;
        const long long q = g.ix(i, j, k);
        const double c1 = abs_bits(p.f.u[q] + p.f.u[q + 1]), c2 = abs_bits(p.f.v[q] + p.f.v[q + g.sx]);
        const double c3 = abs_bits(p.f.w[q] + p.f.w[q + g.sxy]);
        // in the order c1 + c2 + c3 has always been contracted: the time step's bits
        x[0] = fma(c3, p.st.hz[k], fma(c1, p.st.hx[i], c2 * p.st.hy[j]));
    }
    __device__ void add(const KP &, int, int, int, const double *x, double *v) const {
        take_max(v[0], x[0]);
    }
};

// stepinit, slv_auxi.f90:2-50
__device__ void stepinit_pre(KP p);
// The last block of the CFL reduction first does stepinit's scalar updates
// (k_stepinit_pre's work; the per-cell terms read none of them), saving a
// launch per step.
struct StepinitFinal {
    __device__ void operator()(const KP &p, const double *out) const {
        stepinit_pre(p);
        DScal *S = p.S;
        const DCfg &c = p.c;
        double cflm = out[0] * S->dt;
        if (cflm < 0.0) cflm = 0.0;
        S->cflmax = cflm;
        if (c.idtopt != 0 && cflm != 0.0) {
            double a = S->dt * c.cflfac / cflm;
            double b = S->dt * (0.80 + 0.20 * c.cflfac / cflm);
            double dtcfl = a < b ? a : b;
            if (c.idtopt == 1) S->dt = dtcfl;
        }
        double at = fabs(S->time);
        double eps_t = 1.0e-12 * (at > 1.0 ? at : 1.0);
        double dt_evt = S->dt;
        if (c.ptb_tst > S->time + eps_t) dt_evt = fmin(dt_evt, c.ptb_tst - S->time);
        if (c.avg_tst > S->time + eps_t) dt_evt = fmin(dt_evt, c.avg_tst - S->time);
        if (c.tend > S->time + eps_t) dt_evt = fmin(dt_evt, c.tend - S->time);
        if (dt_evt < S->dt) S->dt = dt_evt;
        if (!(S->dt > 0.0) || !isfinite(S->dt)) S->err |= 1;
    }
};

__device__ void stepinit_pre(KP p) {
    DScal *S = p.S;
    S->ntime += 1;
    S->m = S->ntime;
    S->poisson_unconv = 0;
    S->heat_body = 0.0;
    if (p.c.ich != 0) S->pmiavg = 0.0;
    if (p.c.idtopt == 0) S->dt = p.c.dt_size;
    S->subdt = 0.0;
}

__global__ void k_zero_fcvavg(KP p) {
    chained();
    for (int l = 0; l < 4; l++) {
        int n = p.c.nbody[l];
        for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
            p.f.fcvavg[l][t + 1] = 0.0;
    }
}

void launch_stepinit(lesgpu_case *c) {
    if (c->kp.c.ibmon == 1) chain(k_zero_fcvavg, 64, kThreads, 0, c->stream)(c->kp);
    reduce<1, 1u>(c, interior(c->kp.g), CflTerm{}, StepinitFinal{});
}

// substepinit, slv_auxi.f90:105-123 (RK3 coefficients of rk3coefinit,
// misc_init.f90:1031-1044)
__global__ void k_substepinit(KP p, int s, int carry) {
    chained();
    const double gam[4] = {0.0, 8.0 / 15.0, 5.0 / 12.0, 3.0 / 4.0};
    const double ro[4] = {0.0, 0.0, -17.0 / 60.0, -5.0 / 12.0};
    DScal *S = p.S;
    // the metric factors of the projection with flow rates (UcalcQvolTerm), a
    // multiplication per line and not one per cell
    const double dtc = S->dt * (gam[s] + ro[s]);
    const DGrid &g = p.g;
    for (int i = threadIdx.x; i <= g.n1; i += blockDim.x) p.st.px[i] = dtc * g.c2cxi[i];
    for (int j = threadIdx.x; j <= g.n2; j += blockDim.x) p.st.py[j] = dtc * g.c2cyi[j];
    for (int k = threadIdx.x; k <= g.n3; k += blockDim.x) p.st.pz[k] = dtc * g.c2czi[k];
    if (threadIdx.x != 0) return;
    S->alpha = 0.5 * (gam[s] + ro[s]);
    S->dtconst = dtc;
    S->dtconsti = 1.0 / S->dtconst;
    S->test1 = p.c.resid1 * S->dtconsti;
    S->acoef = S->alpha * S->dt / p.c.re;
    S->acoefi = 1.0 / S->acoef;
    S->pmiavg = S->pmiavg + S->pmi[0] * 2.0 * S->alpha;
    S->subdt = S->subdt + S->dtconst;
    if (carry) S->qvol[1] = S->qvol[0];
}

void launch_substepinit(lesgpu_case *c, int msub, bool carry) {
    chain(k_substepinit, 1, kThreads, 0, c->stream)(c->kp, msub, carry ? 1 : 0);
}

// ------------------------------------------------------------ qvol / tvol
struct QvolTerm {   // qvolcalc, slv_auxi.f90:126-149
    static constexpr int kLoads = 2;
    __device__ void load(const KP &p, int i, int j, int k, double *x) const {
        const long long q = p.g.ix(i, j, k);
        x[0] = p.f.u[q];
        x[1] = p.f.wq[q];                // c2cx f2fy f2fz over the fluid u points
    }
    __device__ void add(const KP &p, int i, int j, int k, const double *x, double *v) const { v[0] = fma(x[0], x[1], v[0]); }
};
struct QvolFinal {
    int slot;
    __device__ void operator()(const KP &p, const double *out) const { p.S->qvol[slot] = out[0]; }
};
void launch_qvolcalc(lesgpu_case *c, int slot) { reduce<1, 0u>(c, interior(c->kp.g), QvolTerm{}, QvolFinal{slot}); }

struct TvolTerm {   // tvolcalc, slv_auxi.f90:152-173
    static constexpr int kLoads = 2;
    __device__ void load(const KP &p, int i, int j, int k, double *x) const {
        const long long q = p.g.ix(i, j, k);
        x[0] = p.f.t[q];
        x[1] = p.f.wt[q];                // f2fx f2fy f2fz / c*
    }
    __device__ void add(const KP &p, int i, int j, int k, const double *x, double *v) const { v[0] = fma(x[0], x[1], v[0]); }
};
struct TvolFinal {
    int slot;
    __device__ void operator()(const KP &p, const double *out) const { p.S->tvol[slot] = out[0]; }
};
void launch_tvolcalc(lesgpu_case *c, int slot) { reduce<1, 0u>(c, interior(c->kp.g), TvolTerm{}, TvolFinal{slot}); }

// Weights of the volume reductions: the cell-volume products and fluid masks
// of qvolcalc / meanpg (fb_u), the bulk velocity (fb_c) and tvolcalc (1/c*),
// formed once so each reduction does one multiply per cell.
__global__ void k_red_weights(KP p, Box b) {
    chained();
    const DGrid &g = p.g;
    const long long n = b.count();
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        b.at(t, i, j, k);
        const long long q = g.ix(i, j, k);
        const double cv = g.c2cx[i] * g.f2fy[j] * g.f2fz[k];
        p.f.wq[q] = p.f.fb_u[q] >= 1.0e-10 ? cv : 0.0;
        p.f.wb[q] = p.f.fb_c[q] >= 1.0e-10 ? cv : 0.0;
        p.f.wt[q] = g.f2fx[i] * g.f2fy[j] * g.f2fz[k] / p.f.cstar[q];
    }
}
// The volumes those weights sum to, which meanpg, the bulk velocity, the bulk
// temperature and the mean eddy viscosity divide by: constant, so summed here
// and not with every reduction.
struct VolumeTerm {
    __device__ void operator()(const KP &p, int i, int j, int k, double *w) const {
        const long long q = p.g.ix(i, j, k);
        w[0] = p.f.wq[q];
        w[1] = p.f.wb[q];
        w[2] = p.f.fb_c[q] >= 1.0e-10 ? p.g.f2fx[i] * p.g.f2fy[j] * p.g.f2fz[k] : 0.0;
    }
};
struct VolumeFinal {
    __device__ void operator()(const KP &p, const double *o) const {
        p.S->flowvol = o[0];
        p.S->cellvol = o[1];
        p.S->fluidvol = o[2];
    }
};
void launch_red_weights(lesgpu_case *c) {
    Box b = interior(c->kp.g);
    chain(k_red_weights, blocks_for(b.count()), kThreads, 0, c->stream)(c->kp, b);
    reduce<3, 0u>(c, b, VolumeTerm{}, VolumeFinal{});
}

// tvolcorr, slv_auxi.f90:206-230.  The volume integral of 1/c* does not
// change in time; it is reduced once (lesgpu_start) into S->cvol.
struct CvolTerm {
    __device__ void operator()(const KP &p, int i, int j, int k, double *w) const {
        long long q = p.g.ix(i, j, k);
        w[0] = p.f.wt[q];                // 1 / c* f2fx f2fy f2fz
    }
};
struct CvolFinal {
    __device__ void operator()(const KP &p, const double *out) const { p.S->cvol = out[0]; }
};
// tvolcalc(tvol(2)) followed by tvolcorr in one launch: the reduction's last
// block stores tvol(2) and forms thcap from it
// (slot0: tcalc leaves t unchanged, so the following tvolcalc(tvol(0)) is the
// same sum and is stored here too)
struct TvolCorrFinal {
    int slot0;
    __device__ void operator()(const KP &p, const double *out) const {
        p.S->tvol[2] = out[0];
        p.S->thcap = (p.S->tvol[2] - p.S->tvol[1]) / p.S->cvol;
        if (slot0) p.S->tvol[0] = out[0];
    }
};
// the same with the fluid cells' temperature sum of writehistory
struct TvolBulkTerm {
    static constexpr int kLoads = 3;
    __device__ void load(const KP &p, int i, int j, int k, double *x) const {
        const long long q = p.g.ix(i, j, k);
        x[0] = p.f.t[q];
        x[1] = p.f.wt[q];
        x[2] = p.f.wb[q];
    }
    __device__ void add(const KP &p, int i, int j, int k, const double *x, double *v) const {
        v[0] = fma(x[0], x[1], v[0]);
        v[1] = fma(x[0], x[2], v[1]);
    }
};
struct TvolBulkFinal {
    int slot0;
    __device__ void operator()(const KP &p, const double *out) const {
        TvolCorrFinal{slot0}(p, out);
        p.S->tbulk_sum = out[1];
    }
};
void launch_tvolcalc_corr(lesgpu_case *c, bool slot0, bool bulk) {
    if (bulk) reduce<2, 0u>(c, interior(c->kp.g), TvolBulkTerm{}, TvolBulkFinal{slot0 ? 1 : 0});
    else reduce<1, 0u>(c, interior(c->kp.g), TvolTerm{}, TvolCorrFinal{slot0 ? 1 : 0});
}
void launch_cvol(lesgpu_case *c) { reduce<1, 0u>(c, interior(c->kp.g), CvolTerm{}, CvolFinal{}); }

// tcalc, slv_auxi.f90:496-516
__global__ void k_tcalc(KP p, Box b) {
    chained();
    long long n = b.count();
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        b.at(t, i, j, k);
        p.f.t[p.g.ix(i, j, k)] -= p.S->thcap;
    }
}
void launch_tcalc(lesgpu_case *c) {
    if (c->kp.c.ich == 1 && c->kp.c.xprdic == 0) {
        Box b = interior(c->kp.g);
        chain(k_tcalc, blocks_for(b.count()), kThreads, 0, c->stream)(c->kp, b);
    }
}

// ------------------------------------------------------------------ meanpg
// The flow rate -- the projection's where it has just formed it with qvol(0)
// (ICH = 1), else a pass of its own; only ICH = 1 reads it -- and the four
// wall-shear sums over the planes next to no-slip walls only.  The wall pass
// runs last and finishes the update.
// Box (i, plane, c): plane 0 / 1 = the y-bottom / top wall (j = 1 / n2m,
// k = c), 2 / 3 = the z-bottom / top wall (k = 1 / n3m, j = c); c beyond the
// plane's extent contributes nothing.  A cell on two walls is visited once
// per wall, as the one-pass form tested each wall for every cell.
struct MeanpgWallTerm {
    __device__ void operator()(const KP &p, int i, int plane, int cc, double *w) const {
        const DGrid &g = p.g;
        const DCfg &c = p.c;
        const double *u = p.f.u;
        w[0] = w[1] = w[2] = w[3] = 0.0;
        int j, k;
        if (plane <= 1) {
            j = plane == 0 ? 1 : g.n2m;
            k = cc;
            if (k > g.n3m || (plane == 0 && c.bc_ybtm != 0) || (plane == 1 && c.bc_ytop != 0)) return;
        } else {
            k = plane == 2 ? 1 : g.n3m;
            j = cc;
            if (j > g.n2m || (plane == 2 && c.bc_zbtm != 0) || (plane == 3 && c.bc_ztop != 0)) return;
        }
        const long long q = g.ix(i, j, k);
        if (!fluid(p.f.fb_u[q])) return;
        // the one-sided second-order wall gradient over re, its two weights
        // formed once on the host (per cell they cost four divisions)
        const long long in = plane == 0 ? g.sx : plane == 1 ? -g.sx : plane == 2 ? g.sxy : -g.sxy;
        const double gu = c.wall_a[plane] * u[q] - c.wall_b[plane] * u[q + in];
        w[plane] = gu * (g.c2cx[i] * (plane <= 1 ? g.f2fz[k] : g.f2fy[j]));
    }
};

// IB streamwise forcing term of meanpg (slv_mmtm.f90:141-146)
__global__ void k_meanpg_ibm(KP p) {
    chained();
    double v[1] = {0.0};
    int n = p.c.nbody[0];
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        int m = t + 1;
        v[0] += p.f.fcv[0][m] * p.g.c2cx[p.f.ifc[0][m]] * p.g.f2fy[p.f.jfc[0][m]] * p.g.f2fz[p.f.kfc[0][m]];
    }
    block_totals<1, 0u>(v);
    if (threadIdx.x == 0) p.f.part[(size_t)kRedBlocks * kMaxRed] = v[0];
}

struct FlowFinal {
    __device__ void operator()(const KP &p, const double *o) const { p.S->qcur = o[0]; }
};
struct MeanpgFinal {
    __device__ void operator()(const KP &p, const double *o) const {
        DScal *S = p.S;
        const DCfg &c = p.c;
        for (int q = 0; q < 4; q++) S->pmiw[q] = o[q];
        const double qcur = S->qcur;
        double ubulk = S->flowvol > 0.0 ? qcur / S->flowvol : 0.0;
        double pm[5] = {0.0, c.bc_ybtm == 0 ? o[0] : 0.0, c.bc_ytop == 0 ? o[1] : 0.0, c.bc_zbtm == 0 ? o[2] : 0.0,
                        c.bc_ztop == 0 ? o[3] : 0.0};
        pm[0] = pm[1] + pm[2] + pm[3] + pm[4];
        double ibm = (c.nbody[0] > 0) ? p.f.part[(size_t)kRedBlocks * kMaxRed] : 0.0;
        pm[0] = pm[0] + ibm;
        for (int q = 0; q < 5; q++) S->pmi[q] = pm[q] * c.ivol;
        if (c.ich == 0) {
            S->pmi[0] = 0.0;
        } else if (c.ich == 1) {
            if (S->ntime > 0 && S->dt > 0.0) {
                double err = c.udrv_i - ubulk;
                S->err_integral = S->err_integral + err * S->dtconst;
                S->pmi[0] = S->pmi[0] - (1.0 * err + 0.1 * S->err_integral);
            }
        } else if (c.ich == 2) {
            S->pmi[0] = -c.udrv_i;
        }
    }
};

void launch_meanpg(lesgpu_case *c, bool have_q) {
    const DGrid &g = c->kp.g;
    if (c->kp.c.nbody[0] > 0) chain(k_meanpg_ibm, 1, kThreads, 0, c->stream)(c->kp);
    if (!have_q && c->kp.c.ich == 1) reduce<1, 0u>(c, interior(g), QvolTerm{}, FlowFinal{});
    reduce<4, 0u>(c, Box{1, 0, 1, g.n1m, 4, g.n2m > g.n3m ? g.n2m : g.n3m}, MeanpgWallTerm{}, MeanpgFinal{});
}

// ------------------------------------------------------------------- ucalc
// ucalc, slv_auxi.f90:233-416 (interior update; ghosts by launch_ghost_*)
__global__ void __launch_bounds__(kThreads) k_ucalc(KP p, Box b) {
    chained();
    long long n = b.count();
    const DGrid &g = p.g;
    const double dtc = p.S->dtconst;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        b.at(t, i, j, k);
        long long q = g.ix(i, j, k);
        const double *phi = p.f.phi;
        double ph = phi[q];
        if (i >= g.i_bgpx) p.f.u[q] = p.f.u[q] - dtc * (ph - phi[g.ix(g.imv[i], j, k)]) * g.c2cxi[i];
        if (j >= 2) p.f.v[q] = p.f.v[q] - dtc * (ph - phi[q - g.sx]) * g.c2cyi[j];
        if (k >= g.k_bgpz) p.f.w[q] = p.f.w[q] - dtc * (ph - phi[g.ix(i, j, g.kmv[k])]) * g.c2czi[k];
    }
}

// Periodic ghost copy of one plane pair for up to 4 arrays.
//  dir 0: a(0,j,k) = a(n1m,j,k), a(n1,j,k) = a(1,j,k) over j in [j0,j1], k in [k0,k1]
//  dir 1: a(i,0,k) = a(i,n2m,k), a(i,n2,k) = a(i,1,k) over i, k
//  dir 2: a(i,j,0) = a(i,j,n3m), a(i,j,n3) = a(i,j,1) over i, j

__global__ void k_ghost(KP p, int dir, GhostSpec s0, GhostSpec s1, GhostSpec s2, GhostSpec s3, int na) {
    chained();
    const DGrid &g = p.g;
    GhostSpec ss[4] = {s0, s1, s2, s3};
    for (int a = 0; a < na; a++) {
        const GhostSpec &s = ss[a];
        int n0 = s.hi0 - s.lo0 + 1, n1 = s.hi1 - s.lo1 + 1;
        long long n = (long long)n0 * n1;
        for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
            int x0 = s.lo0 + (int)(t % n0), x1 = s.lo1 + (int)(t / n0);
            if (dir == 0) {
                s.a[g.ix(0, x0, x1)] = s.a[g.ix(g.n1m, x0, x1)];
                s.a[g.ix(g.n1, x0, x1)] = s.a[g.ix(1, x0, x1)];
            } else if (dir == 1) {
                s.a[g.ix(x0, 0, x1)] = s.a[g.ix(x0, g.n2m, x1)];
                s.a[g.ix(x0, g.n2, x1)] = s.a[g.ix(x0, 1, x1)];
            } else {
                s.a[g.ix(x0, x1, 0)] = s.a[g.ix(x0, x1, g.n3m)];
                s.a[g.ix(x0, x1, g.n3)] = s.a[g.ix(x0, x1, 1)];
            }
        }
    }
}

void ghost(lesgpu_case *c, int dir, GhostSpec *s, int na) {
    GhostSpec z{nullptr, 0, -1, 0, -1};
    GhostSpec a0 = na > 0 ? s[0] : z, a1 = na > 1 ? s[1] : z, a2 = na > 2 ? s[2] : z, a3 = na > 3 ? s[3] : z;
    long long mx = 0;
    for (int q = 0; q < na; q++) {
        long long n = (long long)(s[q].hi0 - s[q].lo0 + 1) * (s[q].hi1 - s[q].lo1 + 1);
        if (n > mx) mx = n;
    }
    chain(k_ghost, blocks_for(mx), kThreads, 0, c->stream)(c->kp, dir, a0, a1, a2, a3, na);
}

// qvolcalc(qvol(2)), ucalc and qvolcalc(qvol(0)) in one pass: per cell the
// flow-rate term of the predicted u, the projection of u, v, w (which reads
// only phi's neighbours), then the flow-rate term of the projected u.  The
// sums run in the reduction kernel's own order, so qvol(2) and qvol(0) are
// bitwise those of two separate qvolcalc launches.  Eight FP64 operations a
// cell (16 with dtconst multiplied in per cell and the sums unfused):
// 384x256x384 922 us -> 559.
struct UcalcQvolTerm {
    static constexpr int kLoads = 8;
    __device__ void load(const KP &p, int i, int j, int k, double *x) const {
        const DGrid &g = p.g;
        const long long q = g.ix(i, j, k);
        const double *phi = p.f.phi;
        x[0] = p.f.u[q];
        x[1] = p.f.v[q];
        x[2] = p.f.w[q];
        x[3] = phi[q];
        x[4] = phi[g.ix(g.imv[i], j, k)];
        x[5] = phi[q - g.sx];
        x[6] = phi[g.ix(i, j, g.kmv[k])];
        x[7] = p.f.wq[q];
    }
    __device__ void add(const KP &p, int i, int j, int k, const double *x, double *v) const {
        const DGrid &g = p.g;
        const long long q = g.ix(i, j, k);
        double u = x[0];
        if (i >= g.i_bgpx) p.f.u[q] = u = fma(x[4] - x[3], p.st.px[i], u);
        if (j >= 2) p.f.v[q] = fma(x[5] - x[3], p.st.py[j], x[1]);
        if (k >= g.k_bgpz) p.f.w[q] = fma(x[6] - x[3], p.st.pz[k], x[2]);
        v[0] = fma(x[0], x[7], v[0]);
        v[1] = fma(u, x[7], v[1]);
    }
};
struct UcalcQvolFinal {
    __device__ void operator()(const KP &p, const double *o) const {
        p.S->qvol[2] = o[0];
        p.S->qvol[0] = p.S->qcur = o[1];
    }
};

static void ucalc_interior(lesgpu_case *c, bool with_qvol) {
    Box b = interior(c->kp.g);
    if (with_qvol) reduce<2, 0u>(c, b, UcalcQvolTerm{}, UcalcQvolFinal{});
    else chain(k_ucalc, blocks_for(b.count()), kThreads, 0, c->stream)(c->kp, b);
}

// prdic_adj_uvw(0), slv_mmtm.f90:1746-1857: x, then y, then z
void launch_ghost_uvw(lesgpu_case *c) {
    const DGrid &g = c->kp.g;
    DFields &f = c->kp.f;
    if (c->kp.c.xprdic == 1) {
        GhostSpec s[3] = {{f.u, 0, g.n2, 0, g.n3}, {f.v, 1, g.n2, 0, g.n3}, {f.w, 0, g.n2, 1, g.n3}};
        ghost(c, 0, s, 3);
    }
    if (c->kp.c.yprdic == 1) {
        GhostSpec s[3] = {{f.u, 0, g.n1, 1, g.n3}, {f.v, 0, g.n1, 0, g.n3}, {f.w, 1, g.n1, 0, g.n3}};
        ghost(c, 1, s, 3);
    }
    if (c->kp.c.zprdic == 1) {
        GhostSpec s[3] = {{f.u, 1, g.n1, 0, g.n2}, {f.v, 0, g.n1, 1, g.n2}, {f.w, 0, g.n1, 0, g.n2}};
        ghost(c, 2, s, 3);
    }
}

// ------------------------------------------------------------------- pcalc
// pcalc, slv_auxi.f90:419-493
struct PhirefTerm {
    __device__ void operator()(const KP &p, int i, int j, int k, double *w) const {
        w[0] = p.f.phi[p.g.ix(p.g.n1m, j, k)] * p.g.f2fy[j] * p.g.f2fz[k];
    }
};
struct PhirefFinal {
    __device__ void operator()(const KP &p, const double *o) const { p.S->phiref = o[0] / (p.g.yl * p.g.zl); }
};

__global__ void __launch_bounds__(kThreads) k_pcalc(KP p, Box b) {
    chained();
    long long n = b.count();
    const DGrid &g = p.g;
    // in the order the pressure has always been summed: the mixed form's
    // momentum kernel differences p in FP32, so its last bits show in w
    // (kFineSpan).  A thread takes several cells: 384x256x384 368 us with one, 307 so
    const double dtc = p.S->dtconst, phiref = p.S->phiref, rei = p.c.rei_d;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        b.at(t, i, j, k);
        long long q = g.ix(i, j, k);
        const double pn = p.f.p[q] + p.f.phi[q] - 0.5 * dtc * p.f.divgsum[q] * rei;
        p.f.p[q] = pn - phiref;
    }
}

// ucalc then pcalc.  pcalc reads p, phi and divgsum but no velocity ghost,
// so the periodic ghost copies of u, v, w (ucalc, slv_auxi.f90:360-412) and of
// p (pcalc, :470-490) run after both interiors, the four arrays sharing one
// launch per direction; each array still gets z first, then x.
void launch_ucalc_pcalc(lesgpu_case *c, bool with_qvol) {
    const DGrid &g = c->kp.g;
    ucalc_interior(c, with_qvol);
    reduce<1, 0u>(c, Box{1, 1, 1, 1, g.n2m, g.n3m}, PhirefTerm{}, PhirefFinal{});
    Box b = interior(g);
    const int nb = blocks_for(b.count());
    chain(k_pcalc, nb < 2 * kRedBlocks ? nb : 2 * kRedBlocks, kThreads, 0, c->stream)(c->kp, b);
    DFields &f = c->kp.f;
    if (c->kp.c.zprdic == 1) {
        GhostSpec s[4] = {{f.u, 1, g.n1, 0, g.n2}, {f.v, 0, g.n1, 1, g.n2}, {f.w, 0, g.n1, 0, g.n2}, {f.p, 1, g.n1m, 1, g.n2m}};
        ghost(c, 2, s, 4);
    }
    if (c->kp.c.xprdic == 1) {
        GhostSpec s[4] = {{f.u, 0, g.n2, 0, g.n3}, {f.v, 1, g.n2, 0, g.n3}, {f.w, 0, g.n2, 1, g.n3}, {f.p, 1, g.n2m, 1, g.n3m}};
        ghost(c, 0, s, 4);
    }
}

// ------------------------------------------------------- end-of-step checks
struct DivTerm {   // convergence_check, misc_init.f90:1047-1077
    static constexpr int kLoads = 3;
    __device__ void load(const KP &p, int i, int j, int k, double *x) const {
        const DGrid &g = p.g;
        const long long q = g.ix(i, j, k);
        const double u = p.f.u[q], v = p.f.v[q], z = p.f.w[q], r = p.f.p[q];
        const double d1 = (p.f.u[q + 1] - u) * g.f2fxi[i];
        const double d2 = (p.f.v[q + g.sx] - v) * g.f2fyi[j];
        const double d3 = (p.f.w[q + g.sxy] - z) * g.f2fzi[k];
        x[0] = d1 + d2 + d3;
        x[1] = p.f.qmass[q];
        // u + v + w + p finite, on the exponents: FP64 operations are this
        // pass's time and a compiled fabs or maximum is some
        // (384x256x384 1429 us so, 434 on the bits)
        auto inf = [](double a) { return (__double2hiint(a) & 0x7ff00000) == 0x7ff00000; };
        x[2] = inf(u) | inf(v) | inf(z) | inf(r) ? 1.0 : 0.0;
    }
    __device__ void add(const KP &p, int, int, int, const double *x, double *v) const {
        take_max(v[0], abs_bits(p.c.masson == 1 ? x[0] - x[1] : x[0]));
        take_max(v[1], abs_bits(x[1]));
        take_max(v[2], x[2]);
    }
};
// the last block also advances time (k_time_advance's work; the divergence
// terms do not read it), one launch fewer per step
struct DivFinal {
    __device__ void operator()(const KP &p, const double *o) const {
        p.S->time = p.S->time + p.S->dt;
        p.S->dvmax = o[0];
        if (p.c.ibmon == 1 && p.c.masson == 1) p.S->qmmax = o[1];
        if (o[2] > 0.0 || !isfinite(o[0])) p.S->err |= 2;
    }
};
void launch_advance_and_convergence(lesgpu_case *c) { reduce<3, 7u>(c, interior(c->kp.g), DivTerm{}, DivFinal{}); }

// writehistory's bulk quantities, misc_hist.f90:73-181: the flow rate and the
// fluid cells' temperature sum where the step has not formed them already (the
// volumes are constants), then the scalars; the solid cells' sums
// (temperature inside bodies) in a pass of their own only when some cell
// centre lies inside a body.
struct BulkTerm {
    __device__ void operator()(const KP &p, int i, int j, int k, double *w) const {
        const long long q = p.g.ix(i, j, k);
        w[0] = p.f.u[q] * p.f.wq[q];
        w[1] = p.c.ihtrans == 1 ? p.f.t[q] * p.f.wb[q] : 0.0;
    }
};
struct BulkTTerm {
    __device__ void operator()(const KP &p, int i, int j, int k, double *w) const {
        const long long q = p.g.ix(i, j, k);
        w[0] = p.f.t[q] * p.f.wb[q];
    }
};
__device__ __forceinline__ void bulk_scalars(const KP &p, double q, double t, int solid) {
    DScal *S = p.S;
    S->ubulk = S->flowvol > 0.0 ? q / S->flowvol : 0.0;
    S->qflux = q / p.g.xl;
    S->tbulk_fluid = p.c.ihtrans == 1 && S->cellvol > 0.0 ? t / S->cellvol : 0.0;
    if (!solid) S->tbulk_solid = 0.0;
}
struct BulkSolidTerm {
    __device__ void operator()(const KP &p, int i, int j, int k, double *w) const {
        const DGrid &g = p.g;
        long long q = g.ix(i, j, k);
        w[0] = w[1] = 0.0;
        if (p.f.fb_c[q] < 1.0e-10) {
            double cv = g.c2cx[i] * g.f2fy[j] * g.f2fz[k];
            w[0] = cv;
            w[1] = p.f.t[q] * cv;
        }
    }
};
struct BulkFinal {
    int solid;      // the solid pass follows (else the solid bulk temperature is 0)
    __device__ void operator()(const KP &p, const double *o) const { bulk_scalars(p, o[0], o[1], solid); }
};
struct BulkTFinal {
    int solid;
    __device__ void operator()(const KP &p, const double *o) const { bulk_scalars(p, p.S->qcur, o[0], solid); }
};
__global__ void k_bulk_scalars(KP p, int solid) {
    chained();
    bulk_scalars(p, p.S->qcur, p.S->tbulk_sum, solid);
}
struct BulkSolidFinal {
    __device__ void operator()(const KP &p, const double *o) const {
        p.S->tbulk_solid = o[0] > 0.0 ? o[1] / o[0] : 0.0;
    }
};
void launch_bulk_diag(lesgpu_case *c, bool have_q, bool have_t) {
    const bool solid = c->kp.c.ihtrans == 1 && c->bulk_solid;
    const int sl = solid ? 1 : 0;
    if (have_q && (have_t || c->kp.c.ihtrans != 1)) chain(k_bulk_scalars, 1, 1, 0, c->stream)(c->kp, sl);
    else if (have_q) reduce<1, 0u>(c, interior(c->kp.g), BulkTTerm{}, BulkTFinal{sl});
    else reduce<2, 0u>(c, interior(c->kp.g), BulkTerm{}, BulkFinal{sl});
    if (solid) reduce<2, 0u>(c, interior(c->kp.g), BulkSolidTerm{}, BulkSolidFinal{});
}


}  // namespace lg
