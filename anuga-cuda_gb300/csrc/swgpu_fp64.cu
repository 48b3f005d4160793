// swgpu_fp64.cu -- FP64 evolve kernels (the parity path).
//
// Every floating-point operation is performed in the order of the
// reference's ANUGA C kernels so that the results agree bit for bit with
// them on the same mesh (the file is compiled with --fmad=false: no
// contraction into FMA).  On GB300 this path is bound by the FP64 pipe, not
// by HBM, so what the pipe is not needed for runs elsewhere: quotients, roots
// and comparisons on the integer pipe (swgpu_soft64.cuh, the same bits),
// constants of the geometry from a table, each edge's flux once.
//
// One Euler step of the device-resident loop is three kernels:
//   flux_fp64       central-upwind flux of each edge (one thread per edge),
//                   CFL timestep -> block min -> atomicMin into Ctrl
//   update_fp64     the edge fluxes of each triangle summed in ANUGA's order,
//                   gravity_wb, the step's update_timestep (evaluated here or
//                   once by the flux kernel's last block), Manning
//                   friction, the semi-implicit conserved update, protect,
//                   centroid velocities for the next extrapolation
//   distribute_fp64 second-order limited extrapolation, balance_deep_and_
//                   shallow, boundary conditions of the triangle's boundary
//                   edges; vertex and edge values stored; the scenario's
//                   first block commits the step (time, counters, a stop)
#include <cstdio>

#include "swgpu_device.cuh"
#include "swgpu_soft64.cuh"

namespace swgpu {

// ---------------------------------------------------------------- flux ---

// src/anuga_HMPP/shallow_water_ext.c:214-242 (_compute_speed).
__device__ __forceinline__ double limited_speed(double &uh, double &h, double eps, double h0,
                                                double lim) {
    double u;
    if (h < lim) {
        if (h < eps) {
            h = 0.0;
            u = 0.0;
        } else {
            u = uh / (h + h0 / h);
        }
        uh = u * h;
    } else {
        u = uh / h;
    }
    return u;
}

// The two states of an edge in its own frame's order: stage and momentum
// left and right, bed left and right, the left side's outward normal.
struct EdgeState {
    double wl, uhl, vhl, wr, uhr, vhr, zl, zr, n1, n2;
};
struct EdgeFlux {
    double f0, f1, f2, ms;
    double t;  // the edge's bound of the timestep
    bool bad;  // discontinuous bed
};

// src/anuga_HMPP/shallow_water_ext.c:302-441 (_flux_function_central) in
// plain FP64 arithmetic, with the dry test of :4581-4587: for states that
// are not finite or huge, and for parameters that are not positive.
static __device__ __noinline__ EdgeFlux central_flux_any(const EdgeState &s, const DevParams &P,
                                                         double rad) {
    const double h0 = P.h0, lim = P.lim;
    EdgeFlux r;
    r.f0 = r.f1 = r.f2 = r.ms = 0.0;
    r.t = P.evolve_max_timestep;
    r.bad = false;
    if (P.optimise_dry_cells && fabs(s.wl - s.zl) < P.epsilon && fabs(s.wr - s.zr) < P.epsilon)
        return r;
    // rotate into the edge frame (_rotate, :36-53)
    const double al = s.n1 * s.uhl + s.n2 * s.vhl;
    const double bl = -s.n2 * s.uhl + s.n1 * s.vhl;
    const double ar = s.n1 * s.uhr + s.n2 * s.vhr;
    const double br = -s.n2 * s.uhr + s.n1 * s.vhr;
    if (fabs(s.zl - s.zr) > 1.0e-10) {
        r.bad = true;
        return r;
    }
    const double z = 0.5 * (s.zl + s.zr);
    const double g = P.g, eps = P.epsilon;

    double hl = s.wl - z, uhl = al;
    const double ul = limited_speed(uhl, hl, eps, h0, lim);
    double hr = s.wr - z, uhr = ar;
    const double ur = limited_speed(uhr, hr, eps, h0, lim);
    double vhl = bl, vhr = br;
    limited_speed(vhl, hl, eps, h0, lim);
    limited_speed(vhr, hr, eps, h0, lim);

    const double cl = sqrt(g * hl);
    const double cr = sqrt(g * hr);
    double smax = omax(ul + cl, ur + cr);
    if (smax < 0.0) smax = 0.0;
    double smin = omin(ul - cl, ur - cr);
    if (smin > 0.0) smin = 0.0;

    const double fl0 = ul * hl;
    const double fl1 = ul * uhl + 0.5 * g * hl * hl;
    const double fl2 = ul * vhl;
    const double fr0 = ur * hr;
    const double fr1 = ur * uhr + 0.5 * g * hr * hr;
    const double fr2 = ur * vhr;

    const double denom = smax - smin;
    if (denom < eps) return r;
    const double inv = 1.0 / denom;
    const double ss = smax * smin;
    double e0 = smax * fl0 - smin * fr0;
    e0 += ss * (s.wr - s.wl);
    e0 *= inv;
    double e1 = smax * fl1 - smin * fr1;
    e1 += ss * (ar - al);
    e1 *= inv;
    double e2 = smax * fl2 - smin * fr2;
    e2 += ss * (br - bl);
    e2 *= inv;
    r.ms = omax(fabs(smax), fabs(smin));
    if (r.ms > eps) r.t = omin(r.t, rad / r.ms);
    // rotate back: _rotate(edgeflux, n1, -n2)
    r.f0 = e0;
    r.f1 = s.n1 * e1 + (-s.n2) * e2;
    r.f2 = -(-s.n2) * e1 + s.n1 * e2;
    return r;
}

// x small enough that nothing computed from it overflows (and not NaN)
__device__ __forceinline__ bool tame(double x) {
    return (hi32(x) & 0x7fffffffu) < 0x52b00000u;  // below 2^300
}

// central_flux_any with the same operations in the same order, its
// comparisons, quotients and roots on the integer pipe: 62 FP64
// instructions where the plain form executes about 165.
__device__ __forceinline__ EdgeFlux central_flux(const EdgeState &s, const DevParams &P,
                                                 double rad) {
    if (!(P.plain_positive && tame(s.wl) && tame(s.uhl) && tame(s.vhl) && tame(s.wr) &&
          tame(s.uhr) && tame(s.vhr) && tame(s.zl) && tame(s.zr)))
        return central_flux_any(s, P, rad);
    const double h0 = P.h0, lim = P.lim;
    EdgeFlux r;
    r.f0 = r.f1 = r.f2 = r.ms = 0.0;
    r.t = P.evolve_max_timestep;
    r.bad = false;
    const double g = P.g, eps = P.epsilon;
    double hl = s.wl - s.zl, hr = s.wr - s.zr;
    if (P.optimise_dry_cells && mag_lt(hl, eps) && mag_lt(hr, eps)) return r;
    if (bits64(s.zl) != bits64(s.zr)) {
        // a continuous bed gives both sides the same z, which is then z_l
        if (mag_lt(1.0e-10, s.zl - s.zr)) {
            r.bad = true;
            return r;
        }
        const double z = 0.5 * (s.zl + s.zr);
        hl = s.wl - z;
        hr = s.wr - z;
    }
    const double al = s.n1 * s.uhl + s.n2 * s.vhl;
    const double bl = -s.n2 * s.uhl + s.n1 * s.vhl;
    const double ar = s.n1 * s.uhr + s.n2 * s.vhr;
    const double br = -s.n2 * s.uhr + s.n1 * s.vhr;
    double uhl = al, vhl = bl, uhr = ar, vhr = br;
    // limited_speed for both momentum components of both sides (its second
    // call sees the depth that the first one left; a zero over a positive
    // depth is a zero).  Epsilon may lie above lim: it cuts a side below both.
    double dl = hl, dr = hr;
    const bool sl = lt_pos(hl, lim), sr = lt_pos(hr, lim);
    if (sl || sr) {
        const bool zl = sl && lt_pos(hl, eps), zr = sr && lt_pos(hr, eps);
        if (zl) hl = uhl = vhl = 0.0;
        if (zr) hr = uhr = vhr = 0.0;
        dl = zl ? 1.0 : hl;
        dr = zr ? 1.0 : hr;
        const Two r = div2(h0, dl, h0, dr);
        if (sl && !zl) dl = hl + r.a;
        if (sr && !zr) dr = hr + r.b;
    }
    const Two u = div2(uhl, dl, uhr, dr);
    const double ul = u.a, ur = u.b;
    if (sl || sr) {
        const Two v = div2(vhl, dl, vhr, dr);
        if (sl) {
            uhl = ul * hl;
            vhl = v.a * hl;
        }
        if (sr) {
            uhr = ur * hr;
            vhr = v.b * hr;
        }
    }
    const double ghl = g * hl, ghr = g * hr;
    const Two c = sqrt2(ghl, ghr);
    const double cl = c.a, cr = c.b;
    double smax = imax(ul + cl, ur + cr);
    if (lt_zero(smax)) smax = 0.0;
    double smin = imin(ul - cl, ur - cr);
    if (gt_zero(smin)) smin = 0.0;
    const double denom = smax - smin;
    if (lt_pos(denom, eps)) return r;
    const double fl0 = ul * hl;
    const double fl1 = ul * uhl + half_of(ghl) * hl;  // (0.5 g) h = (g h) / 2
    const double fl2 = ul * vhl;
    const double fr0 = ur * hr;
    const double fr1 = ur * uhr + half_of(ghr) * hr;
    const double fr2 = ur * vhr;
    r.ms = fabs(mag_lt(smin, smax) ? smax : smin);
    const bool fast = lt_pos(eps, r.ms);
    const Two iq = div2(1.0, denom, rad, fast ? r.ms : 1.0);
    const double inv = iq.a;
    if (fast) r.t = iq.b;
    const double ss = smax * smin;
    double e0 = smax * fl0 - smin * fr0;
    e0 += ss * (s.wr - s.wl);
    e0 *= inv;
    double e1 = smax * fl1 - smin * fr1;
    e1 += ss * (ar - al);
    e1 *= inv;
    double e2 = smax * fl2 - smin * fr2;
    e2 += ss * (br - bl);
    e2 *= inv;
    r.f0 = e0;
    r.f1 = s.n1 * e1 + (-s.n2) * e2;
    r.f2 = s.n2 * e1 + s.n1 * e2;
    return r;
}

// compute_fluxes: the central flux of every edge, once, as its owner (the
// triangle with the lower index, which is the one that ANUGA's loop computes
// it for) sees it, times the edge's length; the update subtracts it from the
// owner and adds it to the neighbour.  One thread per edge: 1.5 fluxes per
// triangle instead of three, and equal work for every lane.
//
// PER_SM: blocks of 256 that the registers leave room for, here and in the
// distribute.  With three, at 80 registers (24 and 58 words spilled, which L1
// holds), the FP64 pipe of a large mesh finds a ready warp more often than with
// two at 97 and 127 (a million triangles: flux 224 -> 205 us, distribute 318 ->
// 304; four: 202 and 310); a mesh without that many warps only has the spills
// (2,132 triangles: 26.7 -> 27.7 us a stage).
//
// CFL: min(r_k, r_n) / ms is the smaller of r_k / ms and r_n / ms, since a
// correctly rounded quotient does not fall when its numerator grows; the
// radius is infinite for an edge that does not count (owner not full).
template <int PER_SM>
__global__ void __launch_bounds__(kBlock, PER_SM) flux_fp64(DevMesh M, DevState S, DevParams P,
                                                    Ctrl *ctrl, int flags) {
    const DevEdges &F = M.edges;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (F.blk_scen) ctrl += F.blk_scen[(blockIdx.x * blockDim.x) >> 8];
    int left = -1, right = 0;
    EdgeState s;
    double len = 0.0, rad = 0.0;
    if (e < F.E) {
        left = F.left[e];
        right = F.right[e];
        s.n1 = F.n1[e];
        s.n2 = F.n2[e];
        len = F.len[e];
        rad = F.rad[e];
    }
    pdl_wait();
    if ((flags & kFused) && ctrl_halted(ctrl)) return;
    double t = P.evolve_max_timestep;
    int bad = 0;
    if (left >= 0) {
        const int N = M.N;
        const int k = (left & 3) * N + (left >> 2);
        s.wl = S.we[k];
        s.uhl = S.uhe[k];
        s.vhl = S.vhe[k];
        s.zl = S.ze[k];
        if (right >= 0) {
            const int n = (right & 3) * N + (right >> 2);
            s.wr = S.we[n];
            s.uhr = S.uhe[n];
            s.vhr = S.vhe[n];
            s.zr = S.ze[n];
        } else {
            const int mb = -right - 1;
            s.wr = S.wb[mb];
            s.uhr = S.uhb[mb];
            s.vhr = S.vhb[mb];
            s.zr = s.zl;
        }
        const EdgeFlux r = central_flux(s, P, rad);
        F.f[e] = r.f0 * len;
        F.f[F.E + e] = r.f1 * len;
        F.f[2 * F.E + e] = r.f2 * len;
        if (flags & kWriteMaxSpeed) F.ms[e] = r.ms;
        bad = r.bad;
        t = lt64(t, r.t) ? t : r.t;
    }
    if (bad) set_status(ctrl, SWGPU_EBED);
    if (flags & kNoTimestep) return;  // later Runge-Kutta stage: the step's dt is set
    pdl_launch_dependents();
    block_min_timestep<kBlock>(t, ctrl);
    if ((flags & (kFused | kClock)) == (kFused | kClock) && threadIdx.x == 0 &&
        last_block_done(&ctrl->done_flux, ctrl->blocks_flux))
        publish_step_clock(ctrl, P);
}

// The explicit update of triangle k: the sum of its edges' fluxes in ANUGA's
// order (edges to lower-index neighbours first, by neighbour index, then its
// remaining edges by edge index), over the area, and gravity_wb ('wb_2',
// src/anuga_HMPP/shallow_water_ext.c:1942-2036).
__device__ __forceinline__ void explicit_update(const DevMesh &M, const DevState &S,
                                                const DevParams &P, int k, double w, double zc,
                                                double &a0, double &a1, double &a2) {
    const int N = M.N;
    const DevEdges &F = M.edges;
    double f0[3], f1[3], f2[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int te = F.te[i * N + k];
        const u64 flip = (u64)(te & 1) << 63;  // the neighbour's side: the flux enters
        const int e = te >> 1;
        f0[i] = from64(bits64(F.f[e]) ^ flip);
        f1[i] = from64(bits64(F.f[F.E + e]) ^ flip);
        f2[i] = from64(bits64(F.f[2 * F.E + e]) ^ flip);
    }
    const int code = M.order[k];
    a0 = a1 = a2 = 0.0;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const int i = (code >> (2 * j)) & 3;
        a0 -= i == 0 ? f0[0] : (i == 1 ? f0[1] : f0[2]);
        a1 -= i == 0 ? f1[0] : (i == 1 ? f1[1] : f1[2]);
        a2 -= i == 0 ? f2[0] : (i == 1 ? f2[1] : f2[2]);
    }
    const double *G = M.geo64 + k;
    const double inv_area = G[kGeoInvArea * (size_t)N];
    a0 *= inv_area;
    a1 *= inv_area;
    a2 *= inv_area;
    const double g = P.g;
    const double x10 = G[kGeoX10 * (size_t)N], y10 = G[kGeoY10 * (size_t)N];
    const double x20 = G[kGeoX20 * (size_t)N], y20 = G[kGeoY20 * (size_t)N];
    const double det = G[kGeoDet * (size_t)N];
    const double w0 = S.wv[k], d1 = S.wv[N + k] - w0, d2 = S.wv[2 * N + k] - w0;
    const double avg_h = w - zc;
    double sidex = 0.0, sidey = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double hh = S.we[i * N + k] - S.ze[i * N + k];
        const double fact = P.minus_half_g * hh * hh * M.len[i * N + k];
        const double sx = fact * M.normals[(2 * i) * N + k];
        const double sy = fact * M.normals[(2 * i + 1) * N + k];
        // (0 + s is s: the sign of a zero is lost in the sum with a1 below)
        sidex = i == 0 ? sx : sidex + sx;
        sidey = i == 0 ? sy : sidey + sy;
    }
    const double area = M.areas[k];
    const Two w_xy = div2(y20 * d1 - y10 * d2, det, x10 * d2 - x20 * d1, det);
    const Two side = div2(-sidex, area, -sidey, area);
    a1 += -g * w_xy.a * avg_h;
    a2 += -g * w_xy.b * avg_h;
    a1 += side.a;
    a2 += side.b;
}

// compute_fluxes as the stand-alone method: the explicit updates, and
// max_speed (the largest speed of the edges that triangle k owns).
__global__ void __launch_bounds__(kBlock) explicit_fp64(DevMesh M, DevState S, DevParams P) {
    pdl_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int N = M.N;
    if (k >= N) return;
    double a0, a1, a2;
    explicit_update(M, S, P, k, S.w[k], S.zc[k], a0, a1, a2);
    S.ew[k] = a0;
    S.euh[k] = a1;
    S.evh[k] = a2;
    double ms = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int pk = M.nbr[i * N + k];
        if (pk < 0 || (pk >> 2) > k) ms = omax(ms, M.edges.ms[M.edges.te[i * N + k] >> 1]);
    }
    S.max_speed[k] = ms;
}

// The per-triangle constants of the FP64 path (DevMesh::geo64), with the
// operations and the order in which ANUGA's kernels compute them on each
// call: 1 / area and the vertex differences and determinant of gravity_wb
// (shallow_water_ext.c:1990-2006), and the auxiliary triangle of the
// extrapolation (:2850-2930).
__global__ void __launch_bounds__(kBlock) geometry_fp64(DevMesh M, double *geo) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int N = M.N;
    if (k >= N) return;
    double *G = geo + k;
    const auto put = [&](int plane, double v) { G[plane * (size_t)N] = v; };
    put(kGeoInvArea, 1.0 / M.areas[k]);
    double vx[3], vy[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        vx[i] = M.vxy[(2 * i) * N + k];
        vy[i] = M.vxy[(2 * i + 1) * N + k];
    }
    put(kGeoX10, vx[1] - vx[0]);
    put(kGeoY10, vy[1] - vy[0]);
    put(kGeoX20, vx[2] - vx[0]);
    put(kGeoY20, vy[2] - vy[0]);
    put(kGeoDet, (vy[2] - vy[0]) * (vx[1] - vx[0]) - (vy[1] - vy[0]) * (vx[2] - vx[0]));
    const double x = M.cxy[k], y = M.cxy[N + k];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        put(kGeoDxv + i, vx[i] - x);
        put(kGeoDyv + i, vy[i] - y);
    }
    const int nbk = M.nb[k];
    double dx1 = 0.0, dy1 = 0.0, dx2 = 0.0, dy2 = 0.0, inv = 0.0;  // inv 0: zero gradient
    if (nbk <= 1) {
        const int k0 = M.surr[k], k1 = M.surr[N + k], k2 = M.surr[2 * N + k];
        const double x0 = M.cxy[k0], y0 = M.cxy[N + k0];
        dx1 = M.cxy[k1] - x0;
        dx2 = M.cxy[k2] - x0;
        dy1 = M.cxy[N + k1] - y0;
        dy2 = M.cxy[N + k2] - y0;
        const double area2 = dy2 * dx1 - dy1 * dx2;
        if (!(area2 <= 0)) inv = 1.0 / area2;
    } else if (nbk == 2) {
        int k1 = -1;  // the one interior neighbour: first surrogate that is not k
#pragma unroll
        for (int i = 2; i >= 0; i--) {
            const int sn = M.surr[i * N + k];
            if (sn != k) k1 = sn;
        }
        if (k1 >= 0) {
            dx1 = M.cxy[k1] - x;
            dy1 = M.cxy[N + k1] - y;
            const double area2 = dx1 * dx1 + dy1 * dy1;
            dx2 = 1.0 / area2;
            dy2 = dx2 * dy1;
            dx2 *= dx1;
        }
    }
    put(kGeoDx1, dx1);
    put(kGeoDy1, dy1);
    put(kGeoDx2, dx2);
    put(kGeoDy2, dy2);
    put(kGeoInvArea2, inv);
}

// ------------------------------------------------------------- update ---

// src/anuga_HMPP/shallow_water_ext.c:1238-1317: Manning friction
// coefficient S of triangle k (0 when it does not apply).
__device__ __forceinline__ double manning_S(const DevMesh &M, const DevState &S,
                                            const DevParams &P, int k, double w, double uh,
                                            double vh, bool &applied) {
    const int N = M.N;
    const double eta = S.fric[k];
    const double eps = P.minimum_allowed_height;
    applied = false;
    if (!gt64_nan(eta, eps)) return 0.0;  // (a triangle without a value, NaN, has none)
    const double z0 = S.zv[k], z1 = S.zv[N + k], z2 = S.zv[2 * N + k];
    double zs = 1.0;
    if (P.use_sloped_mannings) {
        const double x0 = M.vxy[0 * N + k], y0 = M.vxy[1 * N + k];
        const double x1 = M.vxy[2 * N + k], y1 = M.vxy[3 * N + k];
        const double x2 = M.vxy[4 * N + k], y2 = M.vxy[5 * N + k];
        const double det = (y2 - y0) * (x1 - x0) - (y1 - y0) * (x2 - x0);
        double zx = (y2 - y0) * (z1 - z0) - (y1 - y0) * (z2 - z0);
        zx = fdiv64(zx, det);
        double zy = (x1 - x0) * (z2 - z0) - (x2 - x0) * (z1 - z0);
        zy = fdiv64(zy, det);
        zs = fsqrt64(1.0 + zx * zx + zy * zy);
    }
    const double z = fdiv64(z0 + z1 + z2, 3.0);
    const double h = w - z;
    if (lt64(h, eps) || nan64(h)) return 0.0;
    double Sf;
    if (P.use_sloped_mannings)
        Sf = -P.g * eta * eta * zs * fsqrt64(uh * uh + vh * vh);
    else
        Sf = -P.g * eta * eta * fsqrt64(uh * uh + vh * vh);
    Sf = fdiv64(Sf, pow_seven_thirds(h));
    applied = true;
    return Sf;
}

// compute_forcing_terms for the per-method API: semi_implicit_update += S*q
// (manning_friction_implicit, gpu_domain_advanced.py:1255-1324), or with
// explicit_target explicit_update += S*q (manning_friction_explicit, :1330-1388:
// the same _manning_friction_flat / _sloped kernels given the explicit arrays).
__global__ void __launch_bounds__(kBlock) forcing_fp64(DevMesh M, DevState S, DevParams P,
                                                       int explicit_target) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M.N) return;
    bool applied;
    const double uh = S.uh[k], vh = S.vh[k];
    const double Sf = manning_S(M, S, P, k, S.w[k], uh, vh, applied);
    if (applied) {
        double *xu = explicit_target ? S.euh : S.suh;
        double *yu = explicit_target ? S.evh : S.svh;
        xu[k] += Sf * uh;
        yu[k] += Sf * vh;
    }
}

// src/anuga_HMPP/shallow_water_ext.c:1638-1705 (_protect) on one triangle.
// The 'tsunami' protection (src/anuga_cuda/protect/protect.cu:64-131) of
// triangle k: below max(0.1 (max bed edge - bed centroid), mah) momentum is
// zeroed; a non-positive depth lifts stage to the lowest bed vertex minus
// mah.  Returns the lifted stage floor bmin (or -inf) for the vertex clamp.
__device__ __forceinline__ double protect_swb2_one(const DevParams &P, double zc,
                                                   const double (&zv)[3], double &w, double &uh,
                                                   double &vh) {
    const double mah = P.minimum_allowed_height;
    const double hc = w - zc;
    const double bmax = 0.5 * fmax(zv[0] + zv[1], fmax(zv[1] + zv[2], zv[2] + zv[0]));
    double floor_w = -pos_inf();
    if (hc < fmax(0.1 * (bmax - zc), mah)) {
        uh = 0.0;
        vh = 0.0;
        if (hc <= 0.0) {
            const double bmin = fmin(zv[0], fmin(zv[1], zv[2])) - mah;
            if (w < bmin) {
                w = fmax(w, bmin);
                floor_w = bmin;
            }
        }
    }
    return floor_w;
}

__device__ __forceinline__ void protect_one(const DevParams &P, double zc, double &w, double &uh,
                                            double &vh) {
    const double hc = w - zc;
    if (!lt64_nan(hc, P.minimum_allowed_height)) return;
    if (P.maximum_allowed_speed < P.epsilon) {
        uh = 0.0;
        vh = 0.0;
        if (!gt_zero(hc)) w = zc;
    } else if (!gt_zero(hc)) {
        w = zc;
        uh = 0.0;
        vh = 0.0;
    } else {
        const double u = uh / hc, v = vh / hc;
        if (fabs(u) > P.maximum_allowed_speed) uh = (P.maximum_allowed_speed * u / fabs(u)) * hc;
        if (fabs(v) > P.maximum_allowed_speed) vh = (P.maximum_allowed_speed * v / fabs(v)) * hc;
    }
}

// src/anuga_HMPP/quantity.c:769-820 (_update) on both momenta with nonzero
// semi-implicit terms; returns false if a denominator is not positive.
__device__ __forceinline__ bool semi_update(double &u, double &v, double eu, double ev, double su,
                                            double sv, double dt) {
    const bool zu = (bits64(u) & kMag64) == 0, zv = (bits64(v) & kMag64) == 0;
    Two s = div2(su, zu ? 1.0 : u, sv, zv ? 1.0 : v);
    if (zu) s.a = 0.0;
    if (zv) s.b = 0.0;
    u += dt * eu;
    v += dt * ev;
    const double du = 1.0 - dt * s.a, dv = 1.0 - dt * s.b;
    if (!(gt_zero(du) && gt_zero(dv)) &&
        (lt64_nan(du, 0.0) || lt64_nan(dv, 0.0) || (bits64(du) & kMag64) == 0 ||
         (bits64(dv) & kMag64) == 0))
        return false;
    const Two q = div2(u, du, v, dv);
    u = q.a;
    v = q.b;
    return true;
}

// update_conserved_quantities (gpu_domain_advanced.py:1412-1442).  Fused:
// the explicit update gathered here from the edge fluxes (and stored, for
// downloads), dt from the device update_timestep, Manning friction computed
// here, then protect (the first step of the next distribute, moved here:
// nothing reads the centroids in between) and the centroid velocities the
// next extrapolation reads.  API: dt given, explicit and semi-implicit terms
// from compute_fluxes and compute_forcing_terms, no protect.
template <int BS, bool FUSED>
__global__ void __launch_bounds__(BS) update_fp64(DevMesh M, DevState S, DevParams P,
                                                      Ctrl *ctrl, double dt_api, int flags,
                                                      Stage stg) {
    ctrl = block_ctrl(ctrl, M);
    pdl_wait();
    if (FUSED && ctrl_halted(ctrl)) {
        if (threadIdx.x == 0 && first_of_scenario(M) && ctrl->halt == 2)
            ctrl->halt = 1;  // the last step's distribute has run
        return;
    }
    __shared__ double block_dt;
    const bool own_clock = FUSED && (flags & kClock);
    if (own_clock && threadIdx.x == 0) {
        const StepClock c = device_update_timestep(ctrl, P);
        block_dt = c.dt;
        if (first_of_scenario(M)) publish_step_clock(ctrl, c);
    }
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    int bad = 0, nonfinite = 0;
    if (own_clock) __syncthreads();
    const double dt = own_clock ? block_dt : (FUSED ? ctrl->clk_dt : dt_api);
    if (k < M.N) {
        double w = S.w[k], uh = S.uh[k], vh = S.vh[k];
        const double zc = S.zc[k];
        double ew, euh, evh;
        if (FUSED) {
            explicit_update(M, S, P, k, w, zc, ew, euh, evh);
            S.ew[k] = ew;
            S.euh[k] = euh;
            S.evh[k] = evh;
        } else {
            ew = S.ew[k];
            euh = S.euh[k];
            evh = S.evh[k];
        }
        if (stg.kind == kStageFirst) {  // backup_conserved_quantities
            S.bw[k] = w;
            S.buh[k] = uh;
            S.bvh[k] = vh;
        }
        double su, sv;
        bool applied;
        if (FUSED) {
            const double Sf = manning_S(M, S, P, k, w, uh, vh, applied);
            su = applied ? Sf * uh : 0.0;
            sv = applied ? Sf * vh : 0.0;
        } else {
            su = S.suh[k];
            sv = S.svh[k];
            applied = (su != 0.0) || (sv != 0.0);
            S.suh[k] = 0.0;
            S.svh[k] = 0.0;
        }
        // stage has no semi-implicit term: its denominator is exactly 1
        w += dt * ew;
        if (applied) {
            if (!semi_update(uh, vh, euh, evh, su, sv, dt)) bad = 1;
        } else {
            uh += dt * euh;
            vh += dt * evh;
        }
        if (stg.kind == kStageMid || stg.kind == kStageLast) {
            // saxpy_conserved_quantities (quantity.c:749-765)
            w = stg.a * w + stg.b * S.bw[k];
            uh = stg.a * uh + stg.b * S.buh[k];
            vh = stg.a * vh + stg.b * S.bvh[k];
        }
        if (FUSED) {
            if (P.flow_algorithm) {
                // the stage vertex clamp of protect_swb2 is overwritten by the
                // extrapolation that follows in the same step
                const double zv[3] = {S.zv[k], S.zv[M.N + k], S.zv[2 * M.N + k]};
                protect_swb2_one(P, zc, zv, w, uh, vh);
            } else {
                protect_one(P, zc, w, uh, vh);
            }
            if (P.extrapolate_velocity_second_order == 1) {
                const double dw = w - zc, mah = P.minimum_allowed_height;
                const double dk = gt64_nan(dw, mah) ? dw : mah;
                const Two vel = div2(uh, dk, vh, dk);
                S.uvel[k] = vel.a;
                S.vvel[k] = vel.b;
            }
        }
        // NaN / Inf anywhere in the new state stops the run: beyond 1e308 in
        // magnitude, on the integer pipe
        const u64 big = 0x7fe1ccf385ebc8a0ull;  // the bits of 1e308
        if ((bits64(w) & kMag64) > big || (bits64(uh) & kMag64) > big ||
            (bits64(vh) & kMag64) > big)
            nonfinite = 1;
        S.w[k] = w;
        S.uh[k] = uh;
        S.vh[k] = vh;
        if (FUSED && (flags & kTrack) &&
            (stg.kind == kStageEuler || stg.kind == kStageLast))
            track_depth(S, k, w - zc, step_end_time(ctrl, dt, stg), P.track_threshold);
    }
    if (bad) set_status(ctrl, SWGPU_EDENOMINATOR);
    if (nonfinite) set_status(ctrl, SWGPU_ENONFINITE);
    // the stage is committed by the distribute (its scenario's first block)
    if (FUSED) pdl_launch_dependents();
}

__global__ void __launch_bounds__(kBlock) track_reset(int N, float *hmax, float *tarr) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= N) return;
    hmax[k] = 0.0f;
    tarr[k] = -1.0f;
}
void launch_track_reset(const DevMesh &M, const DevState &S, cudaStream_t st) {
    track_reset<<<grid_for(M.N), kBlock, 0, st>>>(M.N, S.hmax, S.tarr);
}

// saxpy_conserved_quantities (src/anuga_cuda/saxpy_centroid_values/
// saxpy_centroid_values.cu:1-12, src/anuga_HMPP/quantity.c:749-765) on the
// three conserved quantities: Q = a*Q + b*backup, products then sum, no
// contraction (this unit is built with --fmad=false).
__global__ void __launch_bounds__(kBlock) saxpy_fp64(int N, double a, double b, double *w,
                                                     double *uh, double *vh,
                                                     const double *bw, const double *buh,
                                                     const double *bvh) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= N) return;
    w[k] = a * w[k] + b * bw[k];
    uh[k] = a * uh[k] + b * buh[k];
    vh[k] = a * vh[k] + b * bvh[k];
}

// protect plus the centroid velocities: the head of a stand-alone
// distribute (gpu_domain_advanced.py:1003-1055 and
// extrapolate_velocity_second_order_true, extrapolate_second_order_sw.cu:77-104).
__global__ void __launch_bounds__(kBlock) prepare_fp64(DevMesh M, DevState S, DevParams P) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int N = M.N;
    if (k >= N) return;
    double w = S.w[k], uh = S.uh[k], vh = S.vh[k];
    const double zc = S.zc[k];
    if (P.flow_algorithm) {
        const double zv[3] = {S.zv[k], S.zv[N + k], S.zv[2 * N + k]};
        const double floor_w = protect_swb2_one(P, zc, zv, w, uh, vh);
        if (floor_w > -pos_inf()) {
#pragma unroll
            for (int i = 0; i < 3; i++) S.wv[i * N + k] = fmax(S.wv[i * N + k], floor_w);
        }
    } else {
        protect_one(P, zc, w, uh, vh);
    }
    S.w[k] = w;
    S.uh[k] = uh;
    S.vh[k] = vh;
    const double dk = omax(w - zc, P.minimum_allowed_height);
    const Two vel = div2(uh, dk, vh, dk);
    S.uvel[k] = vel.a;
    S.vvel[k] = vel.b;
}

// The centroid velocities alone: extrapolate_velocity_second_order_true
// (extrapolate_second_order_sw.cu:77-104) as the stand-alone
// extrapolate_second_order_sw runs it, on the state as it is (no protect).
__global__ void __launch_bounds__(kBlock) velocities_fp64(DevMesh M, DevState S, DevParams P) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M.N) return;
    const double dk = omax(S.w[k] - S.zc[k], P.minimum_allowed_height);
    const Two vel = div2(S.uh[k], dk, S.vh[k], dk);
    S.uvel[k] = vel.a;
    S.vvel[k] = vel.b;
}

// --------------------------------------------------------- distribute ---

// The limiter in plain FP64 arithmetic (find_qmin_and_qmax and limit_gradient,
// src/anuga_HMPP/shallow_water_ext.c:98-181): for a gradient with an infinity or
// a NaN, whose comparisons the integer forms below do not have.
__device__ __forceinline__ Three limit_plain(double d0, double d1, double d2, double qmin,
                                             double qmax, double beta) {
    const double TINY = 1.0e-100, d[3] = {d0, d1, d2};
    double r = 1000.0, r0 = 1.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        if (d[i] < -TINY) r0 = qmin / d[i];
        if (d[i] > TINY) r0 = qmax / d[i];
        r = omin(r0, r);
    }
    const double phi = omin(r * beta, 1.0);
    return Three{d0 * phi, d1 * phi, d2 * phi};
}
static __device__ __noinline__ Three aux_limit_any(double d0, double d1, double d2, double dq0,
                                                   double dq1, double dq2, double beta) {
    const double s1 = dq0 + dq1, s2 = dq0 + dq2;
    double qmin, qmax;
    if (dq0 >= 0.0) {
        qmax = dq1 >= dq2 ? (dq1 >= 0.0 ? s1 : dq0) : (dq2 > 0.0 ? s2 : dq0);
        qmin = dq1 >= dq2 ? s2 : s1;
        if (qmin >= 0.0) qmin = 0.0;
    } else {
        qmin = dq1 <= dq2 ? (dq1 < 0.0 ? s1 : dq0) : (dq2 < 0.0 ? s2 : dq0);
        qmax = dq1 <= dq2 ? s2 : s1;
        if (qmax <= 0.0) qmax = 0.0;
    }
    return limit_plain(d0, d1, d2, qmin, qmax, beta);
}
static __device__ __noinline__ Three one_limit_any(double d0, double d1, double d2, double dq1,
                                                   double beta) {
    const bool up = dq1 >= 0.0;
    return limit_plain(d0, d1, d2, up ? 0.0 : dq1, up ? dq1 : 0.0, beta);
}

// src/anuga_HMPP/shallow_water_ext.c:98-148 (find_qmin_and_qmax); branches
// and comparisons on the integer pipe.
__device__ __forceinline__ void qmin_qmax(double dq0, double dq1, double dq2, double &qmin,
                                          double &qmax) {
    const double s1 = dq0 + dq1, s2 = dq0 + dq2;
    const bool above = !lt64(dq1, dq2);  // dq1 >= dq2
    if (ge_zero(dq0)) {
        qmax = above ? (ge_zero(dq1) ? s1 : dq0) : (gt_zero(dq2) ? s2 : dq0);
        qmin = above ? s2 : s1;
        if (ge_zero(qmin)) qmin = 0.0;
    } else {
        const bool below = !lt64(dq2, dq1);  // dq1 <= dq2
        qmin = below ? (lt_zero(dq1) ? s1 : dq0) : (lt_zero(dq2) ? s2 : dq0);
        qmax = below ? s2 : s1;
        if (!gt_zero(qmax)) qmax = 0.0;
    }
}

// src/anuga_HMPP/shallow_water_ext.c:151-181 (limit_gradient): r0 is the
// quotient by the last jump that is not tiny, never below zero.
__device__ __forceinline__ void limit_jumps(double (&d)[3], double qmin, double qmax,
                                            double beta) {
    const u64 tiny = 0x2b2bff2ee48e0530ull;  // the bits of 1e-100
    bool on[3];
    double top[3], low[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        on[i] = (bits64(d[i]) & kMag64) > tiny;
        top[i] = lt_zero(d[i]) ? qmin : qmax;
        low[i] = on[i] ? d[i] : 1.0;
    }
    const Three q3 = div3(top[0], low[0], top[1], low[1], top[2], low[2]);
    const double q[3] = {q3.a, q3.b, q3.c};
    double r = 1000.0, r0 = 1.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        if (on[i]) r0 = q[i];
        r = mag_lt(r0, r) ? r0 : r;
    }
    const double rb = r * beta;
    const double phi = lt_pos(rb, 1.0) ? rb : 1.0;
#pragma unroll
    for (int i = 0; i < 3; i++) d[i] = d[i] * phi;
}

// Auxiliary-triangle reconstruction of one quantity
// (src/anuga_HMPP/shallow_water_ext.c:2942-3055).
__device__ __forceinline__ void aux_jumps(double qk, double q0, double q1, double q2, double dx1,
                                          double dy1, double dx2, double dy2, double inv_area2,
                                          const double (&dxv)[3], const double (&dyv)[3],
                                          double beta, double (&out)[3]) {
    const double dq0 = q0 - qk, dq1 = q1 - q0, dq2 = q2 - q0;
    double a = dy2 * dq1 - dy1 * dq2;
    a *= inv_area2;
    double b = dx1 * dq2 - dx2 * dq1;
    b *= inv_area2;
    double d[3];
#pragma unroll
    for (int i = 0; i < 3; i++) d[i] = a * dxv[i] + b * dyv[i];
    if (finite64(a, b)) {
        double qmin, qmax;
        qmin_qmax(dq0, dq1, dq2, qmin, qmax);
        limit_jumps(d, qmin, qmax, beta);
    } else {
        const Three t = aux_limit_any(d[0], d[1], d[2], dq0, dq1, dq2, beta);
        d[0] = t.a;
        d[1] = t.b;
        d[2] = t.c;
    }
#pragma unroll
    for (int i = 0; i < 3; i++) out[i] = qk + d[i];
}

// Single interior neighbour (src/anuga_HMPP/shallow_water_ext.c:3058-3205).
__device__ __forceinline__ void one_nbr_jumps(double qk, double q1, double dx2, double dy2,
                                              const double (&dxv)[3], const double (&dyv)[3],
                                              double beta, double (&out)[3]) {
    const double dq1 = q1 - qk;
    const double a = dq1 * dx2, b = dq1 * dy2;
    double d[3];
#pragma unroll
    for (int i = 0; i < 3; i++) d[i] = a * dxv[i] + b * dyv[i];
    if (finite64(a, b)) {
        const bool up = ge_zero(dq1);
        limit_jumps(d, up ? 0.0 : dq1, up ? dq1 : 0.0, beta);
    } else {
        const Three t = one_limit_any(d[0], d[1], d[2], dq1, beta);
        d[0] = t.a;
        d[1] = t.b;
        d[2] = t.c;
    }
#pragma unroll
    for (int i = 0; i < 3; i++) out[i] = qk + d[i];
}

// omax(h0, omax(h1, h2)) < epsilon of the surrogate neighbours' depths: a NaN
// gives way to the other operand, unless it is the last.
__device__ __forceinline__ bool dry_neighbours(double h0, double h1, double h2, double eps) {
    return (lt64(h0, eps) || nan64(h0)) && (lt64(h1, eps) || nan64(h1)) && lt64_nan(h2, eps);
}
// omin(omin(h0, omin(h1, h2)), hc): the depth that the limiter's factors follow
__device__ __forceinline__ double least_depth(double h0, double h1, double h2, double hc) {
    return imin_nan(imin_nan(h0, imin_nan(h1, h2)), hc);
}

// the limiter's factor of each quantity: beta_dry + (beta - beta_dry) * hfactor
// (the same number whatever hfactor where the two are equal)
__device__ __forceinline__ void limiter_betas(const DevParams &P, double hfactor,
                                              double (&beta)[3]) {
    beta[0] = P.beta_w_dry;
    beta[1] = P.beta_uh_dry;
    beta[2] = P.beta_vh_dry;
    if (P.betas_differ) {
        beta[0] += P.rise_w * hfactor;
        beta[1] += P.rise_uh * hfactor;
        beta[2] += P.rise_vh * hfactor;
    }
}

// The 'tsunami' distribute (gpu_domain_advanced.py:1755-1812): the edge
// extrapolation of src/anuga_HMPP/shallow_water_ext.c:3328-3964
// (_extrapolate_second_order_edge_sw) after protect_swb2 (applied by the
// update kernel or prepare_fp64): limited auxiliary-triangle gradients
// evaluated at the edge midpoints, dry surrogate neighbours replaced by the
// triangle itself, beta fully wet or dry, vertex values from the edge values
// (v_i = e_j + e_k - e_i), momenta back from velocities with the edge and
// vertex depths; cells skipped as dry keep their previous edge values.  Edge
// values are always stored (the flux reads them), then the boundary values.
template <int BS, int PER_SM>
__global__ void __launch_bounds__(BS, PER_SM * 256 / BS) distribute_de_fp64(DevMesh M, DevState S, DevParams P,
                                                         const BcTag *tags, Ctrl *ctrl,
                                                         int flags, Stage stg) {
    const bool fused = flags & kFused;
    ctrl = block_ctrl(ctrl, M);
    pdl_wait();
    if (fused && ctrl_halt_settled(ctrl) == 1) return;
    if (fused && threadIdx.x == 0 && first_of_scenario(M, blockIdx.x * blockDim.x)) {
        commit_stage(ctrl, published_step_clock(ctrl), P, stg);
        announce_halt(ctrl);
    }
    const int N = M.N;
    const double time = fused ? committed_time(ctrl, stg) : ctrl->time;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    int bad_bc = 0, no_nbr = 0;
    if (k < N) {
        const bool vel = P.extrapolate_velocity_second_order == 1;
        const double *U = vel ? S.uvel : S.uh;  // extrapolated centroid values
        const double *V = vel ? S.vvel : S.vh;
        const double wk = S.w[k], uk = U[k], vk = V[k];
        const int nbk = M.nb[k];
        double ed[3][3];  // edge values of stage and the momenta (or velocities)
        double (&ew)[3] = ed[0], (&eu)[3] = ed[1], (&ev)[3] = ed[2];
        const double own[3] = {wk, uk, vk};
        bool flat = false, keep = false;
        if (nbk == 3) {
            flat = true;
        } else {
            const double x = M.cxy[k], y = M.cxy[N + k];
            double vx[3], vy[3], dxv[3], dyv[3];
#pragma unroll
            for (int i = 0; i < 3; i++) {
                vx[i] = M.vxy[(2 * i) * N + k];
                vy[i] = M.vxy[(2 * i + 1) * N + k];
            }
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const int a = (i + 1) % 3, b = (i + 2) % 3;
                dxv[i] = 0.5 * (vx[a] + vx[b]) - x;  // edge midpoint offsets
                dyv[i] = 0.5 * (vy[a] + vy[b]) - y;
            }
            if (nbk <= 1) {
                int k0 = M.surr[k], k1 = M.surr[N + k], k2 = M.surr[2 * N + k];
                if (le64_nan(S.w[k2], S.zc[k2])) k2 = k;
                if (le64_nan(S.w[k0], S.zc[k0])) k0 = k;
                if (le64_nan(S.w[k1], S.zc[k1])) k1 = k;
                const double x0 = M.cxy[k0], y0 = M.cxy[N + k0];
                const double dx1 = M.cxy[k1] - x0, dx2 = M.cxy[k2] - x0;
                const double dy1 = M.cxy[N + k1] - y0, dy2 = M.cxy[N + k2] - y0;
                const double area2 = dy2 * dx1 - dy1 * dx2;
                if (!gt_zero(area2)) {
                    flat = true;
                } else {
                    const double hc = wk - S.zc[k];
                    const double h0 = S.w[k0] - S.zc[k0];
                    const double h1 = S.w[k1] - S.zc[k1];
                    const double h2 = S.w[k2] - S.zc[k2];
                    double hfactor = 0.0;
                    if (P.betas_differ && gt64_nan(least_depth(h0, h1, h2, hc), 0.0))
                        hfactor = 1.0;
                    if (P.optimise_dry_cells && dry_neighbours(h0, h1, h2, P.epsilon)) {
                        keep = true;
                    } else {
                        const double q0[3] = {S.w[k0], U[k0], V[k0]};
                        const double q1[3] = {S.w[k1], U[k1], V[k1]};
                        const double q2[3] = {S.w[k2], U[k2], V[k2]};
                        double beta[3];
                        limiter_betas(P, hfactor, beta);
                        const double inv_area2 = fdiv64(1.0, area2);
#pragma unroll
                        for (int v = 0; v < 3; v++)
                            aux_jumps(own[v], q0[v], q1[v], q2[v], dx1, dy1, dx2, dy2, inv_area2,
                                      dxv, dyv, beta[v], ed[v]);
                    }
                }
            } else {
                int k1 = -1;
#pragma unroll
                for (int i = 2; i >= 0; i--) {
                    const int sn = M.surr[i * N + k];
                    if (sn != k) k1 = sn;
                }
                if (k1 < 0) {
                    no_nbr = 1;
                    flat = true;
                } else {
                    const double dx1 = M.cxy[k1] - x, dy1 = M.cxy[N + k1] - y;
                    const double area2 = dx1 * dx1 + dy1 * dy1;
                    double dx2 = fdiv64(1.0, area2);
                    const double dy2 = dx2 * dy1;
                    dx2 *= dx1;
                    const double q1[3] = {S.w[k1], U[k1], V[k1]};
#pragma unroll
                    for (int v = 0; v < 3; v++)
                        one_nbr_jumps(own[v], q1[v], dx2, dy2, dxv, dyv, P.beta_w, ed[v]);
                }
            }
        }
        if (flat) {
#pragma unroll
            for (int i = 0; i < 3; i++) {
                ew[i] = wk;
                eu[i] = uk;
                ev[i] = vk;
            }
        } else if (keep) {
#pragma unroll
            for (int i = 0; i < 3; i++) {
                ew[i] = S.we[i * N + k];
                eu[i] = S.uhe[i * N + k];
                ev[i] = S.vhe[i * N + k];
            }
        }
        double ow[3], ou[3], ov[3];
        ow[0] = ew[1] + ew[2] - ew[0];
        ow[1] = ew[0] + ew[2] - ew[1];
        ow[2] = ew[0] + ew[1] - ew[2];
        ou[0] = eu[1] + eu[2] - eu[0];
        ou[1] = eu[0] + eu[2] - eu[1];
        ou[2] = eu[0] + eu[1] - eu[2];
        ov[0] = ev[1] + ev[2] - ev[0];
        ov[1] = ev[0] + ev[2] - ev[1];
        ov[2] = ev[0] + ev[1] - ev[2];
        if (vel) {
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const double de = above_zero(ew[i] - S.ze[i * N + k]);
                eu[i] = eu[i] * de;
                ev[i] = ev[i] * de;
                const double dv = above_zero(ow[i] - S.zv[i * N + k]);
                ou[i] = ou[i] * dv;
                ov[i] = ov[i] * dv;
            }
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
            S.we[i * N + k] = ew[i];
            S.uhe[i * N + k] = eu[i];
            S.vhe[i * N + k] = ev[i];
            S.wv[i * N + k] = ow[i];
            S.uhv[i * N + k] = ou[i];
            S.vhv[i * N + k] = ov[i];
        }
        if ((flags & kWriteBoundary) && nbk > 0) {
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const int pk = M.nbr[i * N + k];
                if (pk < 0) {
                    const int mb = -pk - 1;
                    const double ze = S.ze[i * N + k];
                    double wb, uhb, vhb;
                    if (!eval_boundary(tags[M.btag[mb]], time, ew[i], eu[i], ev[i],
                                       M.normals[(2 * i) * N + k],
                                       M.normals[(2 * i + 1) * N + k], ze, P.g, wb, uhb, vhb)) {
                        bad_bc = 1;
                        wb = uhb = vhb = 0.0;
                    }
                    S.wb[mb] = wb;
                    S.uhb[mb] = uhb;
                    S.vhb[mb] = vhb;
                    S.zb[mb] = ze;
                }
            }
        }
    }
    if (bad_bc) set_status(ctrl, SWGPU_EBOUNDARY);
    if (no_nbr) set_status(ctrl, SWGPU_EMESH);
    if (fused) pdl_launch_dependents();
}

// distribute_to_vertices_and_edges for triangle k: extrapolation of the
// current order (src/anuga_HMPP/shallow_water_ext.c:2717-3324 or
// extrapolate_first_order.cu:3-30), balance_deep_and_shallow
// (shallow_water_ext.c:1462-1636), vertex values stored; optionally the edge
// values (quantity.c:687-706) and the boundary values of k's boundary edges.
// Quantity.extrapolate_second_order_and_limit_by_vertex / _by_edge for one
// quantity q of triangle k, vertex values to out: the centroid gradient from
// the surrogate neighbours (src/anuga_HMPP/quantity.c:24-95 with the plane
// gradients of util_ext.h:66-162; no true neighbour leaves it zero),
// extrapolation to vertices and edge midpoints (quantity.c:130-172), then
// one limiter phi over the three vertices (:298-361) or the three edges
// (:363-447) against the min/max of the true neighbours' centroids.
// Returns false where the surrogate neighbours repeat (the reference's
// _compute_gradients gives up there).
__device__ __forceinline__ bool limit_by_neighbours(const DevMesh &M, const double *q, int k,
                                                    double beta, bool by_edge, double out[3]) {
    const int N = M.N;
    const int nbk = M.nb[k];
    const double qk = q[k];
    const double x = M.cxy[k], y = M.cxy[N + k];
    double a = 0.0, b = 0.0;
    bool ok = true;
    if (nbk < 2) {
        const int k0 = M.surr[k], k1 = M.surr[N + k], k2 = M.surr[2 * N + k];
        if (k0 == k1 || k1 == k2) {
            ok = false;
        } else {
            const double x0 = M.cxy[k0], y0 = M.cxy[N + k0];
            const double x1 = M.cxy[k1], y1 = M.cxy[N + k1];
            const double x2 = M.cxy[k2], y2 = M.cxy[N + k2];
            const double q0 = q[k0], q1 = q[k1], q2 = q[k2];
            const double det = (y2 - y0) * (x1 - x0) - (y1 - y0) * (x2 - x0);
            a = (y2 - y0) * (q1 - q0) - (y1 - y0) * (q2 - q0);
            a /= det;
            b = (x1 - x0) * (q2 - q0) - (x2 - x0) * (q1 - q0);
            b /= det;
        }
    } else if (nbk == 2) {
        int k0 = k;
        for (int i = 0; i < 3 && k0 == k; i++) k0 = M.surr[i * N + k];
        if (k0 == k) {
            ok = false;
        } else {
            const double xx = x - M.cxy[k0], yy = y - M.cxy[N + k0], qq = qk - q[k0];
            const double det = xx * xx + yy * yy;
            a = xx * qq / det;
            b = yy * qq / det;
        }
    }
    double v[3], e[3], dqa[3];
#pragma unroll
    for (int i = 0; i < 3; i++)
        v[i] = qk + a * (M.vxy[(2 * i) * N + k] - x) + b * (M.vxy[(2 * i + 1) * N + k] - y);
    e[0] = 0.5 * (v[1] + v[2]);
    e[1] = 0.5 * (v[2] + v[0]);
    e[2] = 0.5 * (v[0] + v[1]);
    double qmin = qk, qmax = qk;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int pk = M.nbr[i * N + k];
        if (pk >= 0) {
            const double qn = q[pk >> 2];
            qmin = omin(qmin, qn);
            qmax = omax(qmax, qn);
        }
    }
    double phi = 1.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        double r = 1.0;
        const double dq = (by_edge ? e[i] : v[i]) - qk;
        dqa[i] = dq;
        if (dq > 0.0) r = (qmax - qk) / dq;
        if (dq < 0.0) r = (qmin - qk) / dq;
        phi = omin(omin(r * beta, 1.0), phi);
    }
    if (by_edge) {
#pragma unroll
        for (int i = 0; i < 3; i++) e[i] = qk + phi * dqa[i];
        out[0] = e[1] + e[2] - e[0];
        out[1] = e[2] + e[0] - e[1];
        out[2] = e[0] + e[1] - e[2];
    } else {
#pragma unroll
        for (int i = 0; i < 3; i++) out[i] = qk + phi * dqa[i];
    }
    return ok;
}

// balance_deep_and_shallow (src/anuga_HMPP/shallow_water_ext.c:1462-1636)
// of one triangle: centroid stage wk, bed zk, momentum uk, vk; bed vertex
// values zvk; stage / momentum vertex values ow, ou, ov blended in place.
// hv: the vertex depths ow - zvk.
struct Balance {
    double alpha, hc, uc, vc;  // blend, centroid depth and velocities (alpha below 1 only)
};
__device__ __forceinline__ Balance balance_of(const DevParams &P, double wk, double zk, double uk,
                                              double vk, const double (&zvk)[3],
                                              const double (&hv)[3]) {
    const double eps = 1.0e-6;
    double dz = 0.0;
    if (P.tight_slope_limiters == 0) {
#pragma unroll
        for (int i = 0; i < 3; i++) dz = omax(dz, fabs(zvk[i] - zk));
    }
    // (comparisons as the reference's have it where a depth is NaN)
    double alpha = 1.0, hc = 0.0;
    if (P.tight_slope_limiters == 0) {
        const double hmin = imin_nan(hv[0], imin_nan(hv[1], hv[2]));
        if (dz > 0.0) {
            // omax(omin(q, 1), 0), which the compiler, given so, makes 0 of a NaN q
            const double q = fdiv64(P.alpha_balance * hmin, dz);
            alpha = above_zero(lt64_nan(q, 1.0) ? q : 1.0);
        }
    } else if ((lt64_nan(hv[0], P.H0) || lt64_nan(hv[1], P.H0) || lt64(hv[2], P.H0)) &&
               !nan64(hv[2])) {  // omin(hv[0], omin(hv[1], hv[2])) < H0
        hc = wk - zk;
        const double head = hc - P.H0;
        double hd[3];
        bool on[3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            hd[i] = hc - hv[i];
            on[i] = gt_zero(hd[i]) || nan64(hd[i]);
            if (!on[i]) hd[i] = 1.0;
        }
        const Three q3 = div3(head, hd[0], head, hd[1], head, hd[2]);
        const double q[3] = {q3.a, q3.b, q3.c};
#pragma unroll
        for (int i = 0; i < 3; i++)
            if (on[i]) alpha = imin_nan(alpha, q[i]);
        if (nan64(alpha)) alpha = 1.0;  // no blend
        if (lt_zero(alpha)) alpha = 0.0;
    }
    double uc = 0.0, vc = 0.0;
    if (lt64(alpha, 1.0)) {
        if (P.tight_slope_limiters == 0) hc = wk - zk;
        if (P.use_centroid_velocities == 1 && gt64_nan(hc, eps)) {
            const Two c = div2(uk, hc, vk, hc);
            uc = c.a;
            vc = c.b;
        }
    }
    return Balance{alpha, hc, uc, vc};
}
// One vertex of it (alpha below 1).
__device__ __forceinline__ void balance_vertex(const DevParams &P, const Balance &B, double uk,
                                               double vk, double zv, double hv, double &ow,
                                               double &ou, double &ov) {
    ow = zv + (1 - B.alpha) * B.hc + B.alpha * hv;
    if (P.use_centroid_velocities == 1) {
        const double h = ow - zv;
        ou = B.uc * h;
        ov = B.vc * h;
    } else {
        ou = (1 - B.alpha) * uk + B.alpha * ou;
        ov = (1 - B.alpha) * vk + B.alpha * ov;
    }
}
__device__ __forceinline__ void balance_one(const DevParams &P, double wk, double zk, double uk,
                                            double vk, const double (&zvk)[3],
                                            const double (&hv)[3], double (&ow)[3],
                                            double (&ou)[3], double (&ov)[3]) {
    const Balance B = balance_of(P, wk, zk, uk, vk, zvk, hv);
    if (lt64(B.alpha, 1.0)) {
#pragma unroll
        for (int i = 0; i < 3; i++)
            balance_vertex(P, B, uk, vk, zvk[i], hv[i], ow[i], ou[i], ov[i]);
    }
}

// balance_deep_and_shallow as the stand-alone method
// (gpu_domain_advanced.py:957-995): reads the stored vertex values.
__global__ void __launch_bounds__(kBlock) balance_fp64(DevMesh M, DevState S, DevParams P) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int N = M.N;
    if (k >= N) return;
    double zvk[3], hv[3], ow[3], ou[3], ov[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        zvk[i] = S.zv[i * N + k];
        ow[i] = S.wv[i * N + k];
        ou[i] = S.uhv[i * N + k];
        ov[i] = S.vhv[i * N + k];
        hv[i] = ow[i] - zvk[i];
    }
    balance_one(P, S.w[k], S.zc[k], S.uh[k], S.vh[k], zvk, hv, ow, ou, ov);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        S.wv[i * N + k] = ow[i];
        S.uhv[i * N + k] = ou[i];
        S.vhv[i * N + k] = ov[i];
    }
}

template <int BS, int PER_SM>
__global__ void __launch_bounds__(BS, PER_SM * 256 / BS) distribute_fp64(DevMesh M, DevState S, DevParams P,
                                                          const BcTag *tags, Ctrl *ctrl,
                                                          int flags, Stage stg) {
    const bool fused = flags & kFused;
    ctrl = block_ctrl(ctrl, M);
    pdl_wait();
    if (fused && ctrl_halt_settled(ctrl) == 1) return;
    if (fused && threadIdx.x == 0 && first_of_scenario(M, blockIdx.x * blockDim.x)) {
        commit_stage(ctrl, published_step_clock(ctrl), P, stg);
        announce_halt(ctrl);
    }
    const int N = M.N;
    const int order = (int)(fused ? ctrl->clk_order : ctrl->order);
    const double time = fused ? committed_time(ctrl, stg) : ctrl->time;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    int bad_bc = 0, no_nbr = 0;
    if (k < N) {
        const double wk = S.w[k], zk = S.zc[k], uk = S.uh[k], vk = S.vh[k];
        double zvk[3];
#pragma unroll
        for (int i = 0; i < 3; i++) zvk[i] = S.zv[i * N + k];
        double vert[3][3];  // vertex values of stage and the momenta
        double (&ow)[3] = vert[0], (&ou)[3] = vert[1], (&ov)[3] = vert[2];
        // the stand-alone extrapolate_second_order_sw is second order with
        // the optimised limiter whatever the domain's order and limiter
        const bool extrapolate_only = flags & kExtrapolateOnly;
        bool to_momentum = false;
        if (order == 1 && !extrapolate_only) {
#pragma unroll
            for (int i = 0; i < 3; i++) {
                ow[i] = wk;
                ou[i] = uk;
                ov[i] = vk;
            }
        } else if (P.limiter != kLimiterOptimised && !extrapolate_only) {
            const bool by_edge = P.limiter == kLimiterEdge;
            bool ok = limit_by_neighbours(M, S.w, k, P.beta_w, by_edge, ow);
            ok &= limit_by_neighbours(M, S.uh, k, P.beta_uh, by_edge, ou);
            ok &= limit_by_neighbours(M, S.vh, k, P.beta_vh, by_edge, ov);
            if (!ok) no_nbr = 1;
        } else {
            const bool vel = P.extrapolate_velocity_second_order == 1;
            // centroid values being extrapolated (velocity or momentum)
            const double *U = vel ? S.uvel : S.uh, *V = vel ? S.vvel : S.vh;
            const double qu = vel ? U[k] : uk;
            const double qv = vel ? V[k] : vk;
            const double own[3] = {wk, qu, qv};
            const int nbk = M.nb[k];
            bool keep = false;  // dry: previous vertex values stay
            bool flat = nbk == 3;  // zero gradient: centroid values at vertices
            if (!flat) {
                const double *G = M.geo64 + k;
                const size_t n = N;
                const double inv_area2 = G[kGeoInvArea2 * n];
                double dxv[3], dyv[3];
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    dxv[i] = G[(kGeoDxv + i) * n];
                    dyv[i] = G[(kGeoDyv + i) * n];
                }
                const double dx2 = G[kGeoDx2 * n], dy2 = G[kGeoDy2 * n];
                if (nbk <= 1) {
                    if ((bits64(inv_area2) & kMag64) == 0) {
                        flat = true;
                    } else {
                        const int k0 = M.surr[k], k1 = M.surr[N + k], k2 = M.surr[2 * N + k];
                        const double dx1 = G[kGeoDx1 * n], dy1 = G[kGeoDy1 * n];
                        const double w0 = S.w[k0], w1 = S.w[k1], w2 = S.w[k2];
                        const double h0 = w0 - S.zc[k0];
                        const double h1 = w1 - S.zc[k1];
                        const double h2 = w2 - S.zc[k2];
                        if (P.optimise_dry_cells && dry_neighbours(h0, h1, h2, P.epsilon)) {
                            keep = true;
                        } else {
                            double hfactor = 0.0;
                            if (P.betas_differ) {
                                const double hmin = least_depth(h0, h1, h2, wk - zk);
                                if (gt64_nan(hmin, 0.001))
                                    hfactor = fdiv64(hmin - 0.001, hmin + 0.004);
                            }
                            const double q0[3] = {w0, U[k0], V[k0]};
                            const double q1[3] = {w1, U[k1], V[k1]};
                            const double q2[3] = {w2, U[k2], V[k2]};
                            double beta[3];
                            limiter_betas(P, hfactor, beta);
#pragma unroll
                            for (int v = 0; v < 3; v++)
                                aux_jumps(own[v], q0[v], q1[v], q2[v], dx1, dy1, dx2, dy2,
                                          inv_area2, dxv, dyv, beta[v], vert[v]);
                        }
                    }
                } else {
                    // the one interior neighbour: first surrogate that is not k
                    int k1 = -1;
#pragma unroll
                    for (int i = 2; i >= 0; i--) {
                        const int s = M.surr[i * N + k];
                        if (s != k) k1 = s;
                    }
                    if (k1 < 0) {
                        no_nbr = 1;
                        flat = true;
                    } else {
                        const double q1[3] = {S.w[k1], U[k1], V[k1]};
#pragma unroll
                        for (int v = 0; v < 3; v++)
                            one_nbr_jumps(own[v], q1[v], dx2, dy2, dxv, dyv, P.beta_w, vert[v]);
                    }
                }
            }
            if (flat) {
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    ow[i] = wk;
                    ou[i] = qu;
                    ov[i] = qv;
                }
            } else if (keep) {
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    ow[i] = S.wv[i * N + k];
                    ou[i] = S.uhv[i * N + k];
                    ov[i] = S.vhv[i * N + k];
                }
            }
            to_momentum = vel;
        }
        double hv[3];
#pragma unroll
        for (int i = 0; i < 3; i++) hv[i] = ow[i] - zvk[i];
        if (to_momentum) {
            // back from velocity to momentum with the vertex depth
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const double dv = above_zero(hv[i]);
                ou[i] = ou[i] * dv;
                ov[i] = ov[i] * dv;
            }
        }

        if (!(flags & kExtrapolateOnly)) balance_one(P, wk, zk, uk, vk, zvk, hv, ow, ou, ov);

#pragma unroll
        for (int i = 0; i < 3; i++) {
            S.wv[i * N + k] = ow[i];
            S.uhv[i * N + k] = ou[i];
            S.vhv[i * N + k] = ov[i];
        }
        // interpolated edge values (quantity.c:687-706)
        double ew[3], eu[3], ev[3];
        if (flags & kWriteEdges) {
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const int a = (i == 0) ? 1 : 0, b = (i == 2) ? 1 : 2;
                S.we[i * N + k] = ew[i] = half_of(ow[a] + ow[b]);
                S.uhe[i * N + k] = eu[i] = half_of(ou[a] + ou[b]);
                S.vhe[i * N + k] = ev[i] = half_of(ov[a] + ov[b]);
            }
        }
        if ((flags & kWriteBoundary) && M.nb[k] > 0) {
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const int pk = M.nbr[i * N + k];
                if (pk < 0) {
                    const int mb = -pk - 1;
                    double wb, uhb, vhb;
                    if (!eval_boundary(tags[M.btag[mb]], time, ew[i], eu[i], ev[i],
                                       M.normals[(2 * i) * N + k],
                                       M.normals[(2 * i + 1) * N + k], S.ze[i * N + k], P.g,
                                       wb, uhb, vhb)) {
                        bad_bc = 1;
                        wb = uhb = vhb = 0.0;
                    }
                    S.wb[mb] = wb;
                    S.uhb[mb] = uhb;
                    S.vhb[mb] = vhb;
                    S.zb[mb] = S.ze[i * N + k];
                }
            }
        }
    }
    if (bad_bc) set_status(ctrl, SWGPU_EBOUNDARY);
    if (no_nbr) set_status(ctrl, SWGPU_EMESH);
    if (fused) pdl_launch_dependents();
}

// Boundary values of boundary edge mb, edge i of triangle k, from its edge
// values; returns 1 where they could not be evaluated.
__device__ __forceinline__ int boundary_edge(const DevMesh &M, const DevState &S,
                                             const DevParams &P, const BcTag *tags, double time,
                                             int k, int i, int mb, double we, double uhe,
                                             double vhe) {
    const int N = M.N;
    const double ze = S.ze[i * N + k];
    double wb, uhb, vhb;
    int bad = 0;
    if (!eval_boundary(tags[M.btag[mb]], time, we, uhe, vhe, M.normals[(2 * i) * N + k],
                       M.normals[(2 * i + 1) * N + k], ze, P.g, wb, uhb, vhb)) {
        bad = 1;
        wb = uhb = vhb = 0.0;
    }
    S.wb[mb] = wb;
    S.uhb[mb] = uhb;
    S.vhb[mb] = vhb;
    S.zb[mb] = ze;
    return bad;
}

// distribute_fp64 and distribute_de_fp64 with three threads per triangle, one
// for each quantity in the reconstruction and for each vertex and edge after
// it, in three warps that meet through shared memory.  A mesh that leaves the
// SMs few warps is bound by the chain of FP64 operations and quotients of one
// triangle (an operation that a warp waits for takes about 100 clocks, its
// pipe 16): a third of the operations per thread, three times the warps.  The
// depths and the balance's blend are computed by all three, so a mesh that
// fills the FP64 pipe is better off with a thread per triangle (distribute_split;
// microseconds per step, three threads / one: 1,024 triangles 28.9 / 35.9, 4,096
// 28.8 / 36.1, 14,400 32.5 / 36.9, 20,164 37.4 / 39.5, 28,900 43.0 / 42.4, 40,000
// 54.8 / 50.7, 160,000 164 / 152).
__global__ void __launch_bounds__(3 * kSplitTile) distribute_split_fp64(DevMesh M, DevState S,
                                                                        DevParams P,
                                                                        const BcTag *tags,
                                                                        Ctrl *ctrl, int flags, Stage stg) {
    const bool fused = flags & kFused;
    const int k0 = blockIdx.x * kSplitTile;
    if (M.blk_scen) ctrl += M.blk_scen[k0 >> 8];
    pdl_wait();
    if (fused && ctrl_halt_settled(ctrl) == 1) return;
    if (fused && threadIdx.x == 0 && first_of_scenario(M, blockIdx.x * kSplitTile)) {
        commit_stage(ctrl, published_step_clock(ctrl), P, stg);
        announce_halt(ctrl);
    }
    const int N = M.N;
    const int role = threadIdx.x / kSplitTile, t = threadIdx.x % kSplitTile, k = k0 + t;
    __shared__ double vert[3][3][kSplitTile];  // [quantity][vertex], then balanced
    const bool in = k < N;
    int bad_bc = 0, no_nbr = 0;
    bool to_momentum = false;
    double wk = 0.0, zk = 0.0, zvk[3] = {0.0, 0.0, 0.0};
    if (in) {
        const int order = (int)(fused ? ctrl->clk_order : ctrl->order);
        wk = S.w[k];
        zk = S.zc[k];
#pragma unroll
        for (int i = 0; i < 3; i++) zvk[i] = S.zv[i * N + k];
        const bool extrapolate_only = flags & kExtrapolateOnly;
        const bool vel = P.extrapolate_velocity_second_order == 1;
        const double *mom = role == 1 ? S.uh : S.vh;
        double out[3];
        if (order == 1 && !extrapolate_only) {
            const double q = role == 0 ? wk : mom[k];
#pragma unroll
            for (int i = 0; i < 3; i++) out[i] = q;
        } else if (P.limiter != kLimiterOptimised && !extrapolate_only) {
            if (!limit_by_neighbours(M, role == 0 ? S.w : mom, k,
                                     role == 0 ? P.beta_w : (role == 1 ? P.beta_uh : P.beta_vh),
                                     P.limiter == kLimiterEdge, out))
                no_nbr = 1;
        } else {
            const double *Q = role == 0 ? S.w : (!vel ? mom : (role == 1 ? S.uvel : S.vvel));
            const double own = Q[k];
            const int nbk = M.nb[k];
            bool keep = false;
            bool flat = nbk == 3;
            if (!flat) {
                const double *G = M.geo64 + k;
                const size_t n = N;
                const double inv_area2 = G[kGeoInvArea2 * n];
                double dxv[3], dyv[3];
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    dxv[i] = G[(kGeoDxv + i) * n];
                    dyv[i] = G[(kGeoDyv + i) * n];
                }
                const double dx2 = G[kGeoDx2 * n], dy2 = G[kGeoDy2 * n];
                if (nbk <= 1) {
                    if ((bits64(inv_area2) & kMag64) == 0) {
                        flat = true;
                    } else {
                        const int k0n = M.surr[k], k1n = M.surr[N + k], k2n = M.surr[2 * N + k];
                        const double dx1 = G[kGeoDx1 * n], dy1 = G[kGeoDy1 * n];
                        const double q0 = Q[k0n], q1 = Q[k1n], q2 = Q[k2n];
                        const double h0 = S.w[k0n] - S.zc[k0n];
                        const double h1 = S.w[k1n] - S.zc[k1n];
                        const double h2 = S.w[k2n] - S.zc[k2n];
                        if (P.optimise_dry_cells && dry_neighbours(h0, h1, h2, P.epsilon)) {
                            keep = true;
                        } else {
                            double hfactor = 0.0;
                            if (P.betas_differ) {
                                const double hmin = least_depth(h0, h1, h2, wk - zk);
                                if (gt64_nan(hmin, 0.001))
                                    hfactor = fdiv64(hmin - 0.001, hmin + 0.004);
                            }
                            double beta[3];
                            limiter_betas(P, hfactor, beta);
                            aux_jumps(own, q0, q1, q2, dx1, dy1, dx2, dy2, inv_area2, dxv, dyv,
                                      role == 0 ? beta[0] : (role == 1 ? beta[1] : beta[2]), out);
                        }
                    }
                } else {
                    int k1 = -1;
#pragma unroll
                    for (int i = 2; i >= 0; i--) {
                        const int sn = M.surr[i * N + k];
                        if (sn != k) k1 = sn;
                    }
                    if (k1 < 0) {
                        no_nbr = 1;
                        flat = true;
                    } else {
                        one_nbr_jumps(own, Q[k1], dx2, dy2, dxv, dyv, P.beta_w, out);
                    }
                }
            }
            if (flat) {
#pragma unroll
                for (int i = 0; i < 3; i++) out[i] = own;
            } else if (keep) {
                const double *before = role == 0 ? S.wv : (role == 1 ? S.uhv : S.vhv);
#pragma unroll
                for (int i = 0; i < 3; i++) out[i] = before[i * N + k];
            }
            to_momentum = vel;
        }
#pragma unroll
        for (int i = 0; i < 3; i++) vert[role][i][t] = out[i];
    }
    __syncthreads();
    // vertex `role`
    double ow = 0.0, ou = 0.0, ov = 0.0;
    if (in) {
        double hv[3];
#pragma unroll
        for (int i = 0; i < 3; i++) hv[i] = vert[0][i][t] - zvk[i];
        const double h = role == 0 ? hv[0] : (role == 1 ? hv[1] : hv[2]);
        const double zv = role == 0 ? zvk[0] : (role == 1 ? zvk[1] : zvk[2]);
        ow = vert[0][role][t];
        ou = vert[1][role][t];
        ov = vert[2][role][t];
        if (to_momentum) {
            const double dv = above_zero(h);
            ou = ou * dv;
            ov = ov * dv;
        }
        if (!(flags & kExtrapolateOnly)) {
            const double uk = S.uh[k], vk = S.vh[k];
            const Balance B = balance_of(P, wk, zk, uk, vk, zvk, hv);
            if (lt64(B.alpha, 1.0)) balance_vertex(P, B, uk, vk, zv, h, ow, ou, ov);
        }
        S.wv[role * N + k] = ow;
        S.uhv[role * N + k] = ou;
        S.vhv[role * N + k] = ov;
    }
    if (flags & kWriteEdges) {
        __syncthreads();
        vert[0][role][t] = ow;
        vert[1][role][t] = ou;
        vert[2][role][t] = ov;
        __syncthreads();
        if (in) {
            // edge `role`
            const int a = role == 0 ? 1 : 0, b = role == 2 ? 1 : 2;
            const double we = half_of(vert[0][a][t] + vert[0][b][t]);
            const double uhe = half_of(vert[1][a][t] + vert[1][b][t]);
            const double vhe = half_of(vert[2][a][t] + vert[2][b][t]);
            S.we[role * N + k] = we;
            S.uhe[role * N + k] = uhe;
            S.vhe[role * N + k] = vhe;
            if (flags & kWriteBoundary) {
                const int pk = M.nbr[role * N + k];
                if (pk < 0)
                    bad_bc = boundary_edge(M, S, P, tags,
                                       fused ? committed_time(ctrl, stg) : ctrl->time, k, role, -pk - 1, we, uhe,
                                           vhe);
            }
        }
    }
    if (bad_bc) set_status(ctrl, SWGPU_EBOUNDARY);
    if (no_nbr) set_status(ctrl, SWGPU_EMESH);
    if (fused) pdl_launch_dependents();
}

__global__ void __launch_bounds__(3 * kSplitTile) distribute_de_split_fp64(DevMesh M, DevState S,
                                                                           DevParams P,
                                                                           const BcTag *tags,
                                                                           Ctrl *ctrl, int flags, Stage stg) {
    const bool fused = flags & kFused;
    const int first = blockIdx.x * kSplitTile;
    if (M.blk_scen) ctrl += M.blk_scen[first >> 8];
    pdl_wait();
    if (fused && ctrl_halt_settled(ctrl) == 1) return;
    if (fused && threadIdx.x == 0 && first_of_scenario(M, blockIdx.x * kSplitTile)) {
        commit_stage(ctrl, published_step_clock(ctrl), P, stg);
        announce_halt(ctrl);
    }
    const int N = M.N;
    const int role = threadIdx.x / kSplitTile, t = threadIdx.x % kSplitTile, k = first + t;
    __shared__ double edge[3][3][kSplitTile];  // [quantity][edge]
    const bool in = k < N;
    const bool vel = P.extrapolate_velocity_second_order == 1;
    int bad_bc = 0, no_nbr = 0;
    if (in) {
        const double *mom = role == 1 ? (vel ? S.uvel : S.uh) : (vel ? S.vvel : S.vh);
        const double *Q = role == 0 ? S.w : mom;
        const double own = Q[k];
        const int nbk = M.nb[k];
        double out[3];
        bool flat = false, keep = false;
        if (nbk == 3) {
            flat = true;
        } else {
            const double x = M.cxy[k], y = M.cxy[N + k];
            double vx[3], vy[3], dxv[3], dyv[3];
#pragma unroll
            for (int i = 0; i < 3; i++) {
                vx[i] = M.vxy[(2 * i) * N + k];
                vy[i] = M.vxy[(2 * i + 1) * N + k];
            }
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const int a = (i + 1) % 3, b = (i + 2) % 3;
                dxv[i] = half_of(vx[a] + vx[b]) - x;  // edge midpoint offsets
                dyv[i] = half_of(vy[a] + vy[b]) - y;
            }
            if (nbk <= 1) {
                int k0 = M.surr[k], k1 = M.surr[N + k], k2 = M.surr[2 * N + k];
                if (le64_nan(S.w[k2], S.zc[k2])) k2 = k;
                if (le64_nan(S.w[k0], S.zc[k0])) k0 = k;
                if (le64_nan(S.w[k1], S.zc[k1])) k1 = k;
                const double x0 = M.cxy[k0], y0 = M.cxy[N + k0];
                const double dx1 = M.cxy[k1] - x0, dx2 = M.cxy[k2] - x0;
                const double dy1 = M.cxy[N + k1] - y0, dy2 = M.cxy[N + k2] - y0;
                const double area2 = dy2 * dx1 - dy1 * dx2;
                if (!gt_zero(area2)) {
                    flat = true;
                } else {
                    const double hc = S.w[k] - S.zc[k];
                    const double h0 = S.w[k0] - S.zc[k0];
                    const double h1 = S.w[k1] - S.zc[k1];
                    const double h2 = S.w[k2] - S.zc[k2];
                    double hfactor = 0.0;
                    if (P.betas_differ && gt64_nan(least_depth(h0, h1, h2, hc), 0.0))
                        hfactor = 1.0;
                    if (P.optimise_dry_cells && dry_neighbours(h0, h1, h2, P.epsilon)) {
                        keep = true;
                    } else {
                        double beta[3];
                        limiter_betas(P, hfactor, beta);
                        const double inv_area2 = fdiv64(1.0, area2);
                        aux_jumps(own, Q[k0], Q[k1], Q[k2], dx1, dy1, dx2, dy2, inv_area2, dxv,
                                  dyv, role == 0 ? beta[0] : (role == 1 ? beta[1] : beta[2]), out);
                    }
                }
            } else {
                int k1 = -1;
#pragma unroll
                for (int i = 2; i >= 0; i--) {
                    const int sn = M.surr[i * N + k];
                    if (sn != k) k1 = sn;
                }
                if (k1 < 0) {
                    no_nbr = 1;
                    flat = true;
                } else {
                    const double dx1 = M.cxy[k1] - x, dy1 = M.cxy[N + k1] - y;
                    const double area2 = dx1 * dx1 + dy1 * dy1;
                    double dx2 = fdiv64(1.0, area2);
                    const double dy2 = dx2 * dy1;
                    dx2 *= dx1;
                    one_nbr_jumps(own, Q[k1], dx2, dy2, dxv, dyv, P.beta_w, out);
                }
            }
        }
        if (flat) {
#pragma unroll
            for (int i = 0; i < 3; i++) out[i] = own;
        } else if (keep) {
            const double *before = role == 0 ? S.we : (role == 1 ? S.uhe : S.vhe);
#pragma unroll
            for (int i = 0; i < 3; i++) out[i] = before[i * N + k];
        }
#pragma unroll
        for (int i = 0; i < 3; i++) edge[role][i][t] = out[i];
    }
    __syncthreads();
    if (in) {
        // edge and vertex `role`
        const int a = role == 0 ? 1 : 0, b = role == 2 ? 1 : 2;
        const double we = edge[0][role][t];
        double ue = edge[1][role][t], ve = edge[2][role][t];
        const double ow = edge[0][a][t] + edge[0][b][t] - we;
        double ou = edge[1][a][t] + edge[1][b][t] - ue;
        double ov = edge[2][a][t] + edge[2][b][t] - ve;
        if (vel) {
            const double de = above_zero(we - S.ze[role * N + k]);
            ue = ue * de;
            ve = ve * de;
            const double dv = above_zero(ow - S.zv[role * N + k]);
            ou = ou * dv;
            ov = ov * dv;
        }
        S.we[role * N + k] = we;
        S.uhe[role * N + k] = ue;
        S.vhe[role * N + k] = ve;
        S.wv[role * N + k] = ow;
        S.uhv[role * N + k] = ou;
        S.vhv[role * N + k] = ov;
        if (flags & kWriteBoundary) {
            const int pk = M.nbr[role * N + k];
            if (pk < 0)
                bad_bc = boundary_edge(M, S, P, tags,
                                       fused ? committed_time(ctrl, stg) : ctrl->time, k, role, -pk - 1, we, ue, ve);
        }
    }
    if (bad_bc) set_status(ctrl, SWGPU_EBOUNDARY);
    if (no_nbr) set_status(ctrl, SWGPU_EMESH);
    if (fused) pdl_launch_dependents();
}

// update_boundary as a stand-alone pass over boundary slots, from the
// stored vertex values (gpu_domain_advanced.py:2006-2108).
__global__ void __launch_bounds__(kBlock) boundary_fp64(DevMesh M, DevState S, DevParams P,
                                                        const BcTag *tags, Ctrl *ctrl) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M.Nb) return;
    const int N = M.N;
    const int k = M.bcell[m], i = M.bedge[m];
    if (M.blk_scen) ctrl += M.blk_scen[k >> 8];  // the owning scenario's time
    const int a = (i == 0) ? 1 : 0, b = (i == 2) ? 1 : 2;
    // the 'tsunami' distribute stores its edge values; otherwise they are the
    // interpolation of the vertex values
    const double we = P.flow_algorithm ? S.we[i * N + k]
                                       : 0.5 * (S.wv[a * N + k] + S.wv[b * N + k]);
    const double uhe = P.flow_algorithm ? S.uhe[i * N + k]
                                        : 0.5 * (S.uhv[a * N + k] + S.uhv[b * N + k]);
    const double vhe = P.flow_algorithm ? S.vhe[i * N + k]
                                        : 0.5 * (S.vhv[a * N + k] + S.vhv[b * N + k]);
    double wb, uhb, vhb;
    if (!eval_boundary(tags[M.btag[m]], ctrl->time, we, uhe, vhe, M.normals[(2 * i) * N + k],
                       M.normals[(2 * i + 1) * N + k], S.ze[i * N + k], P.g, wb, uhb, vhb)) {
        set_status(ctrl, SWGPU_EBOUNDARY);
        wb = uhb = vhb = 0.0;
    }
    S.wb[m] = wb;
    S.uhb[m] = uhb;
    S.vhb[m] = vhb;
    S.zb[m] = S.ze[i * N + k];
}

// interpolate_from_vertices_to_edges for stage, xmom, ymom (quantity.c:687-706).
__global__ void __launch_bounds__(kBlock) interpolate_fp64(DevMesh M, DevState S) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int N = M.N;
    if (k >= N) return;
    const double *V[3] = {S.wv, S.uhv, S.vhv};
    double *E[3] = {S.we, S.uhe, S.vhe};
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const double q0 = V[q][k], q1 = V[q][N + k], q2 = V[q][2 * N + k];
        E[q][k] = half_of(q1 + q2);
        E[q][N + k] = half_of(q0 + q2);
        E[q][2 * N + k] = half_of(q0 + q1);
    }
}

// update_centroids_of_velocities_and_height
// (update_centroids_of_velocities_and_height.cu:1-52), centroids and
// boundary slots.
__global__ void __launch_bounds__(kBlock) other_quantities(DevMesh M, DevState S) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const double H0 = 1.0e-8;
    if (k < M.N) {
        double h = S.w[k] - S.zc[k];
        if (h < 0) h = 0;
        const double f = h / (h * h + H0);
        S.hc[k] = h;
        S.uc[k] = S.uh[k] * f;
        S.vc[k] = S.vh[k] * f;
    }
    if (k < M.Nb) {
        double h = S.wb[k] - S.zb[k];
        if (h < 0) h = 0;
        const double f = h / (h * h + H0);
        S.hb[k] = h;
        S.ub[k] = S.uhb[k] * f;
        S.vb[k] = S.vhb[k] * f;
    }
}

// Water volume: per-block partial sums in a fixed order, then one block adds
// the partials in index order (deterministic).
__global__ void __launch_bounds__(kBlock) mass_partials(DevMesh M, DevState S) {
    __shared__ double sh[kBlock];
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    sh[threadIdx.x] = k < M.N ? M.areas[k] * (S.w[k] - S.zc[k]) : 0.0;
    __syncthreads();
    for (int s = kBlock / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) S.partials[blockIdx.x] = sh[0];
}

__global__ void __launch_bounds__(kBlock) mass_final(const double *partials, int n, double *out) {
    __shared__ double sh[kBlock];
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += partials[i];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int t = kBlock / 2; t > 0; t >>= 1) {
        if ((int)threadIdx.x < t) sh[threadIdx.x] += sh[threadIdx.x + t];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = sh[0];
}

// ------------------------------------------------------------ launches ---

void launch_prepare_fp64(const DevMesh &M, const DevState &S, const DevParams &P, Ctrl *,
                         cudaStream_t st) {
    prepare_fp64<<<grid_for(M.N), kBlock, 0, st>>>(M, S, P);
}
// Block sizes of the fused-step kernels come from M.shape (fp64_block).
void launch_distribute_fp64(const DevMesh &M, const DevState &S, const DevParams &P,
                            const BcTag *tags, Ctrl *ctrl, int flags, const Stage &stage,
                            cudaStream_t st) {
    const int tile = distribute_tile_fp64(M.shape.distribute, M.N, M.shape.sms);
    const int g = (M.n_launch + tile - 1) / tile;
    const bool pdl = M.shape.pdl && (flags & kFused) && overlap_fp64(M.n_launch, M.shape.sms);
    if (distribute_split(M.N, M.shape.sms)) {
        launch_k(P.flow_algorithm ? distribute_de_split_fp64 : distribute_split_fp64, g, 3 * tile,
                 st, pdl, M, S, P, tags, ctrl, flags, stage);
        return;
    }
    const bool dense = dense_fp64(M.N, M.shape.sms);
    if (P.flow_algorithm)
        launch_k(tile > 256 ? distribute_de_fp64<512, 2>
                            : (dense ? distribute_de_fp64<256, 3> : distribute_de_fp64<256, 2>),
                 g, tile, st, pdl, M, S, P, tags, ctrl, flags, stage);
    else
        launch_k(tile > 256 ? distribute_fp64<512, 2>
                            : (dense ? distribute_fp64<256, 3> : distribute_fp64<256, 2>),
                 g, tile, st, pdl, M, S, P, tags, ctrl, flags, stage);
}
void launch_boundary_fp64(const DevMesh &M, const DevState &S, const DevParams &P,
                          const BcTag *tags, Ctrl *ctrl,
                          cudaStream_t st) {
    if (M.Nb > 0) boundary_fp64<<<grid_for(M.Nb), kBlock, 0, st>>>(M, S, P, tags, ctrl);
}
void launch_flux_fp64(const DevMesh &M, const DevState &S, const DevParams &P, Ctrl *ctrl,
                      int flags, cudaStream_t st) {
    const int bs = fp64_block(M.shape.flux, M.edges.E, M.shape.sms);
    const bool pdl = M.shape.pdl && (flags & kFused) && overlap_fp64(M.n_launch, M.shape.sms);
    if (!update_clock_fp64(M.N, M.shape.sms)) flags |= kClock;
    launch_k(dense_fp64(M.N, M.shape.sms) ? flux_fp64<3> : flux_fp64<1>,
             (M.edges.launch + bs - 1) / bs, bs, st, pdl, M, S, P, ctrl, flags);
}
void launch_explicit_fp64(const DevMesh &M, const DevState &S, const DevParams &P,
                          cudaStream_t st) {
    const int bs = fp64_block(kBlock, M.N, M.shape.sms);
    explicit_fp64<<<(M.N + bs - 1) / bs, bs, 0, st>>>(M, S, P);
}
void launch_geometry_fp64(const DevMesh &M, double *geo, cudaStream_t st) {
    geometry_fp64<<<grid_for(M.N), kBlock, 0, st>>>(M, geo);
}
void launch_forcing_fp64(const DevMesh &M, const DevState &S, const DevParams &P,
                         bool explicit_target, cudaStream_t st) {
    forcing_fp64<<<grid_for(M.N), kBlock, 0, st>>>(M, S, P, explicit_target ? 1 : 0);
}
void launch_velocities_fp64(const DevMesh &M, const DevState &S, const DevParams &P,
                            cudaStream_t st) {
    velocities_fp64<<<grid_for(M.N), kBlock, 0, st>>>(M, S, P);
}
void launch_balance_fp64(const DevMesh &M, const DevState &S, const DevParams &P,
                         cudaStream_t st) {
    balance_fp64<<<grid_for(M.N), kBlock, 0, st>>>(M, S, P);
}
void launch_update_fp64(const DevMesh &M, const DevState &S, const DevParams &P, Ctrl *ctrl,
                        double dt, int flags, const Stage &stage, cudaStream_t st) {
    const int bs = fp64_block(M.shape.update, M.N, M.shape.sms);
    const int g = (M.n_launch + bs - 1) / bs;
    // (a later Runge-Kutta stage has the step's clock)
    if ((stage.kind == kStageEuler || stage.kind == kStageFirst) &&
        update_clock_fp64(M.N, M.shape.sms))
        flags |= kClock;
    if (flags & kFused)
        launch_k(bs > 256 ? update_fp64<512, true> : update_fp64<256, true>, g, bs, st,
                 M.shape.pdl && overlap_fp64(M.n_launch, M.shape.sms), M, S, P, ctrl, dt, flags,
                 stage);
    else
        launch_k(bs > 256 ? update_fp64<512, false> : update_fp64<256, false>, g, bs, st, false,
                 M, S, P, ctrl, dt, flags, stage);
}
void launch_saxpy_fp64(const DevMesh &M, const DevState &S, double a, double b,
                       cudaStream_t st) {
    saxpy_fp64<<<grid_for(M.N), kBlock, 0, st>>>(M.N, a, b, S.w, S.uh, S.vh, S.bw, S.buh,
                                                 S.bvh);
}
void launch_interpolate_fp64(const DevMesh &M, const DevState &S, cudaStream_t st) {
    interpolate_fp64<<<grid_for(M.N), kBlock, 0, st>>>(M, S);
}
void launch_other_quantities(const DevMesh &M, const DevState &S, cudaStream_t st) {
    const int n = M.N > M.Nb ? M.N : M.Nb;
    other_quantities<<<grid_for(n), kBlock, 0, st>>>(M, S);
}
void launch_mass_partials(const DevMesh &M, const DevState &S, cudaStream_t st) {
    mass_partials<<<grid_for(M.N), kBlock, 0, st>>>(M, S);
}
void launch_mass(const DevMesh &M, const DevState &S, double *out, cudaStream_t st) {
    const int g = grid_for(M.N);
    mass_partials<<<g, kBlock, 0, st>>>(M, S);
    mass_final<<<1, kBlock, 0, st>>>(S.partials, g, out);
}

}  // namespace swgpu
