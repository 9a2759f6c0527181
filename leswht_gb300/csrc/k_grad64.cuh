// Velocity gradients of the FP64 form from 1-D weights.
//
// On GB300 an FP64 instruction holds its sub-partition's pipe for 64 clocks a
// warp, so an FP64 stencil's time is its FP64 instruction count, and what
// depends on one index only is formed once per case (Stn, lesgpu_create): the
// face interpolation's metric products with the wall flags folded in, and the
// three-point derivative of the interpolated values.  The nine gradients of a
// cell then take 39 operations where the written-out form took some 120.
#pragma once
#include "lesgpu_internal.cuh"

namespace lg {

// a[0..8] = du/dx dv/dx dw/dx du/dy dv/dy dw/dy du/dz dv/dz dw/dz at the
// centre of (i, j, k).  WRAP: neighbours by the periodic index tables (velgrad,
// sgs.f90:772-875), else by the ghost layers (misc_hist.f90:379-455).
template <bool WRAP>
__device__ __forceinline__ void velgrad64(const KP &p, int i, int j, int k, const double *u, const double *v,
                                          const double *w, double a[9]) {
    const DGrid &g = p.g;
    const Stn &T = p.st;
    const long long q = g.ix(i, j, k);
    const long long ip = WRAP ? g.ipv[i] - i : 1, im = WRAP ? g.imv[i] - i : -1;
    const long long jp = WRAP ? (g.jpv[j] - j) * g.sx : g.sx, jm = WRAP ? (g.jmv[j] - j) * g.sx : -g.sx;
    const long long kp = WRAP ? (g.kpv[k] - k) * g.sxy : g.sxy, km = WRAP ? (g.kmv[k] - k) * g.sxy : -g.sxy;
    const double4 X = (WRAP ? T.dwx : T.dgx)[i], Y = (WRAP ? T.dwy : T.dgy)[j], Z = (WRAP ? T.dwz : T.dgz)[k];
    const double us = u[q] + u[q + ip], vs = v[q] + v[q + jp], ws = w[q] + w[q + kp];
    a[0] = g.f2fxi[i] * (u[q + ip] - u[q]);
    a[4] = g.f2fyi[j] * (v[q + jp] - v[q]);
    a[8] = g.f2fzi[k] * (w[q + kp] - w[q]);
    a[3] = Y.x * (u[q + jm] + u[q + ip + jm]) + Y.y * us + Y.z * (u[q + jp] + u[q + ip + jp]);
    a[6] = Z.x * (u[q + km] + u[q + ip + km]) + Z.y * us + Z.z * (u[q + kp] + u[q + ip + kp]);
    a[1] = X.x * (v[q + im] + v[q + jp + im]) + X.y * vs + X.z * (v[q + ip] + v[q + jp + ip]);
    a[7] = Z.x * (v[q + km] + v[q + jp + km]) + Z.y * vs + Z.z * (v[q + kp] + v[q + jp + kp]);
    a[2] = X.x * (w[q + im] + w[q + kp + im]) + X.y * ws + X.z * (w[q + ip] + w[q + kp + ip]);
    a[5] = Y.x * (w[q + jm] + w[q + kp + jm]) + Y.y * ws + Y.z * (w[q + jp] + w[q + kp + jp]);
}

}  // namespace lg
