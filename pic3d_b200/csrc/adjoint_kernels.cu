// Hand-written adjoint of the per-timestep loop (no counterpart in the
// reference), for gradients of a final-state objective with respect to the
// particle weights (hence a density profile) and the laser's transverse
// amplitude coefficients.
//
// Forward step n (absorbing faces):  BC(t_n) -> E half -> B half -> clear J ->
// push+deposit -> removal -> B half -> E half.  The adjoint runs the
// transposes in reverse order.  The field updates are linear, so their
// transposes need no stored values; the push needs the particles before the
// push and the fields it gathered (after the first half-update), which a
// tape records while a checkpointed segment is recomputed.
//
//   * Yee transposes: one thread per buffer point in gather form (each
//     thread writes only its own point, no atomics).
//   * BC transpose: one thread per face row; adds into neighbours with
//     atomics and accumulates d objective / d(profile coefficient).
//   * push adjoint: one thread per particle; recomputes the gather with
//     shape-derivative weights, contracts the current adjoint with the
//     Esirkepov factors to get the derivatives of the deposit with respect
//     to the old and new positions and the weight, applies the transpose of
//     the Boris rotation and scatters the gathered-field adjoints back to
//     the grid.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "pic_kernels.cuh"
#include "push_core.cuh"
#include "tile_common.cuh"

namespace pic {

// ---------------------------------------------------------------------------
// Boris rotation and move (particle.cpp:271-315) of one particle, and its
// transpose.  (The Jacobian by forward-mode dual numbers, three passes of three
// tangents, took about 2000 instructions per particle; the transpose takes
// some 130 beside the values.)
template <typename T>
struct Boris {
    T e[3], b[3], p1[3], t[3], s[3], p2[3], pn[3];
    T ig1, f, ig;   // 1 / gamma of p1, 2 / (1 + t^2), 1 / gamma of pn
};

template <typename T>
__device__ __forceinline__ void cross_add(const T (&a)[3], const T (&b)[3], T (&r)[3]) {
    r[0] += a[1] * b[2] - a[2] * b[1];
    r[1] += a[2] * b[0] - a[0] * b[2];
    r[2] += a[0] * b[1] - a[1] * b[0];
}

// inputs p, fields e, b (unscaled)
template <typename T>
__device__ __forceinline__ void boris_values(const T (&p)[3], const T *e, const T *b, T qm, Boris<T> &v) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        v.e[d] = e[d] * qm;
        v.b[d] = b[d] * qm;
        v.p1[d] = p[d] + v.e[d];
    }
    v.ig1 = T(1) / sqrt(T(1) + (v.p1[0] * v.p1[0] + v.p1[1] * v.p1[1] + v.p1[2] * v.p1[2]));
#pragma unroll
    for (int d = 0; d < 3; ++d) v.t[d] = v.b[d] * v.ig1;
    v.f = T(2) / (T(1) + v.t[0] * v.t[0] + v.t[1] * v.t[1] + v.t[2] * v.t[2]);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        v.s[d] = v.t[d] * v.f;
        v.p2[d] = v.p1[d];
        v.pn[d] = v.p1[d] + v.e[d];
    }
    cross_add(v.p1, v.t, v.p2);
    cross_add(v.p2, v.s, v.pn);
    v.ig = T(1) / sqrt(T(1) + (v.pn[0] * v.pn[0] + v.pn[1] * v.pn[1] + v.pn[2] * v.pn[2]));
}

// lin = J^T (lp, lx), J = d(p', displacement in cells) / d(p, e, b); the
// displacement is pn ig dtd.  Uses grad_a a x b . l = b x l and
// grad_b a x b . l = l x a.
template <typename T>
__device__ __forceinline__ void boris_transpose(const Boris<T> &v, T qm, const T (&dtd)[3], const T (&lp)[3],
                                                const T (&lx)[3], T (&lin)[9]) {
    T l[3], li = 0;   // adjoints of pn and ig
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const T q = lx[d] * dtd[d];
        l[d] = lp[d] + q * v.ig;
        li += q * v.pn[d];
    }
    li *= v.ig * v.ig * v.ig;
#pragma unroll
    for (int d = 0; d < 3; ++d) l[d] -= li * v.pn[d];
    // pn = p1 + p2 x s + e
    T l1[3] = {l[0], l[1], l[2]}, l2[3] = {0, 0, 0}, ls[3] = {0, 0, 0}, lt[3] = {0, 0, 0};
    cross_add(v.s, l, l2);
    cross_add(l, v.p2, ls);
    // p2 = p1 + p1 x t
#pragma unroll
    for (int d = 0; d < 3; ++d) l1[d] += l2[d];
    cross_add(v.t, l2, l1);
    cross_add(l2, v.p1, lt);
    // s = t f, f = 2 / (1 + t^2)
    const T k = v.f * v.f * (ls[0] * v.t[0] + ls[1] * v.t[1] + ls[2] * v.t[2]);
#pragma unroll
    for (int d = 0; d < 3; ++d) lt[d] += v.f * ls[d] - k * v.t[d];
    // t = b ig1
    const T k1 = v.ig1 * v.ig1 * v.ig1 * (lt[0] * v.b[0] + lt[1] * v.b[1] + lt[2] * v.b[2]);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        l1[d] -= k1 * v.p1[d];
        lin[d] = l1[d];
        lin[3 + d] = qm * (l[d] + l1[d]);
        lin[6 + d] = qm * v.ig1 * lt[d];
    }
}

// derivatives of the shape weights with respect to the position
template <typename real>
__device__ __forceinline__ void shape_derivs(real d, real (&w)[3]) {
    const real h = real(0.5);
    w[0] = -(h - d);
    w[1] = real(-2) * d;
    w[2] = h + d;
}
template <typename real>
__device__ __forceinline__ void shape_derivs(real d, real (&w)[5]) {
    real u, u2;
    u = d - real(0.5);
    u2 = u * u;
    w[0] = u2 * u * real(1.0 / 6.0);
    u = d + real(1.0);
    u2 = u * u;
    w[1] = -u2 * u * real(4.0 / 6.0) + u2 * real(15.0 / 6.0) - u * real(10.0 / 4.0) + real(5.0 / 24.0);
    u = d;
    u2 = u * u;
    w[2] = u2 * u - u * real(5.0 / 4.0);
    u = d - real(1.0);
    u2 = u * u;
    w[3] = -u2 * u * real(4.0 / 6.0) - u2 * real(15.0 / 6.0) - u * real(10.0 / 4.0) - real(5.0 / 24.0);
    u = d + real(0.5);
    u2 = u * u;
    w[4] = u2 * u * real(1.0 / 6.0);
}

// gather of one component with its gradient with respect to the position
template <typename real, int P, bool LDG>
__device__ __forceinline__ void gather_grad(const View<const real> &f, int i0, int j0, int k0,
                                            const real (&wx)[P], const real (&wy)[P], const real (&wz)[P],
                                            const real (&dx)[P], const real (&dy)[P], const real (&dz)[P], real &e,
                                            real (&gr)[3]) {
    e = 0;
    gr[0] = gr[1] = gr[2] = 0;
    for (int k = 0; k < P; ++k) {
        real a = 0, ax = 0, ay = 0;
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const real *row = f.at(k0 + k, j0 + j, i0);
            real s = 0, sd = 0;
#pragma unroll
            for (int i = 0; i < P; ++i) {
                real v = LDG ? __ldg(row + i) : row[i];
                s += wx[i] * v;
                sd += dx[i] * v;
            }
            a += wy[j] * s;
            ax += wy[j] * sd;
            ay += dy[j] * s;
        }
        const real wzk = pick(wz, k), dzk = pick(dz, k);
        e += wzk * a;
        gr[0] += wzk * ax;
        gr[1] += wzk * ay;
        gr[2] += dzk * a;
    }
}

template <typename real, int P>
__device__ __forceinline__ void scatter_adj(real *f, const Geom &g, int i0, int j0, int k0, const real (&wx)[P],
                                            const real (&wy)[P], const real (&wz)[P], real lam) {
    if (lam == real(0)) return;
    for (int k = 0; k < P; ++k) {
        const real lk = lam * pick(wz, k);
#pragma unroll
        for (int j = 0; j < P; ++j) {
            real *row = f + g.fi(k0 + k, j0 + j, i0);
            const real lj = lk * wy[j];
#pragma unroll
            for (int i = 0; i < P; ++i) atomic_add(row + i, lj * wx[i]);
        }
    }
}

// union-span arrays of a quantity of the old (a0 at centre i1) and new (a1
// at centre i2) positions, as span1d does for the weights
template <typename T, int P>
__device__ __forceinline__ void span_pair(int i1, const T (&a0)[P], int i2, const T (&a1)[P], T (&u0)[P + 1],
                                          T (&u1)[P + 1]) {
    const int lo = min(i1, i2);
    const bool o0 = i1 != lo, o1 = i2 != lo;
#pragma unroll
    for (int a = 0; a <= P; ++a) {
        u0[a] = o0 ? (a >= 1 ? a0[a - 1] : T(0)) : (a < P ? a0[a] : T(0));
        u1[a] = o1 ? (a >= 1 ? a1[a - 1] : T(0)) : (a < P ? a1[a] : T(0));
    }
}

// Adjoint of one Esirkepov component in the factors s = (s0 + s1)/2 and
// d = (s1 - s0)/sqrt(12) of each axis.  Axis `c` carries the running sum of
// ds = sqrt(12) d, axes `u` and `v` the weight W = s_u s_v + d_u d_v (two
// products where the four of the old and new shapes took six).  Returns
// G1 = sum(lam * J) / w and adds dG1/ds, dG1/dd into gs, gd.
template <int P, bool LDG, typename LT>
__device__ __forceinline__ double esirkepov_adj(const LT *lam, int sc, int su, int sv, int lc, int lu, int lv,
                                                double coef, const double (&dc)[P + 1], const double (&s_u)[P + 1],
                                                const double (&d_u)[P + 1], const double (&s_v)[P + 1],
                                                const double (&d_v)[P + 1], double (&gdc)[P + 1],
                                                double (&gsu)[P + 1], double (&gdu)[P + 1], double (&gsv)[P + 1],
                                                double (&gdv)[P + 1]) {
    constexpr double kSqrt12 = 3.4641016151377546;
    double C[P], M[P];
    double acc = 0.0;
#pragma unroll
    for (int a = 0; a < P; ++a) {
        acc += dc[a];
        C[a] = (a < lc - 1) ? coef * kSqrt12 * acc : 0.0;   // the last running-sum point is not deposited
        M[a] = 0.0;
    }
#pragma unroll 1
    for (int b = 0; b < lv; ++b) {
        const double sb = pick(s_v, b), db = pick(d_v, b);
        double ts = 0.0, td = 0.0;
#pragma unroll
        for (int a = 0; a <= P; ++a) {
            if (a >= lu) break;
            const double W = s_u[a] * sb + d_u[a] * db;
            double T = 0.0;
            const LT *row = lam + b * sv + a * su;
#pragma unroll
            for (int q = 0; q < P; ++q) {
                if (q >= lc - 1) break;
                const double l = (double)(LDG ? __ldg(row + q * sc) : row[q * sc]);
                T += C[q] * l;
                M[q] += l * W;
            }
            gsu[a] += T * sb;
            gdu[a] += T * db;
            ts += T * s_u[a];
            td += T * d_u[a];
        }
        // add into gsv[b], gdv[b] for a run-time b
#pragma unroll
        for (int q = 0; q <= P; ++q)
            if (q == b) {
                gsv[q] += ts;
                gdv[q] += td;
            }
    }
    // dG/dds(q') = coef * sum_{q >= q'} M(q)
    double suf = 0.0, G = 0.0;
#pragma unroll
    for (int q = P - 1; q >= 0; --q) {
        G += C[q] * M[q];
        suf += M[q];
        gdc[q] += coef * kSqrt12 * suf;
    }
    return G;
}

template <typename real>
struct AdjPushArgs {
    Geom g;
    CellPack cp;
    long long n;
    // tape: particles before the push, fields after the first half-update
    const double *x, *y, *z;
    const int *cell;
    const float *ox, *oy, *oz;
    const real *px, *py, *pz;
    const unsigned char *dead;
    const real *f[6];
    const real *w;
    // adjoints
    const real *lj[3];         // d objective / dJ (ring buffers)
    real *lf[6];               // d objective / d(E, B) after the first half-update (field buffers)
    real *lx, *ly, *lz, *lpx, *lpy, *lpz;   // per particle, in: after the push, out: before it
    double *lw;                // per particle, accumulated
    real qm, charge;
    real dt_d[3];
    double d_dt[3];
    int scatter_fields;        // 0 for the t = 0 push (fields identically zero there)
    unsigned *status;
    const int *idx;            // optional particle list (count *nidx); null: all n particles
    const unsigned long long *nidx;
};

// One particle's push adjoint (everything but the scatter of the gathered
// field adjoints): per-particle adjoints updated in place, the weight
// adjoint accumulated, and lin[3..8] = d objective / d(gathered E, B) left
// for the caller to scatter with the gather weights.  fv: the tape's six
// field components; lj: the three J adjoints (ring layout or a shared box),
// both addressed in buffer coordinates.  Returns false if the particle is
// skipped (its stencil leaves the buffers).
template <typename real, int P, bool LDG>
__device__ __forceinline__ bool adj_particle(const AdjPushArgs<real> &a, long long p, const View<const real> (&fv)[6],
                                             const View<const real> (&lj)[3], real (&lin)[9]) {
    constexpr bool F64 = sizeof(real) == 8;
    constexpr int H = P / 2;
    const Geom &g = a.g;
    {
        // ---- old position --------------------------------------------------
        int ip[3], id[3], cc[3] = {0, 0, 0};
        real dp[3], dd[3];
        double xd[3] = {0, 0, 0};
        real oo[3] = {0, 0, 0};
        if constexpr (F64) {
            xd[0] = a.x[p];
            xd[1] = a.y[p];
            xd[2] = a.z[p];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                double xc = xd[d] - (double)(1 - g.mem);
                ip[d] = (int)(xc + 0.5);
                dp[d] = xc - (double)ip[d];
                id[d] = (int)xc;
                dd[d] = (xc - 0.5) - (double)id[d];
            }
        } else {
            a.cp.unpack(a.cell[p], cc[0], cc[1], cc[2]);
            oo[0] = a.ox[p];
            oo[1] = a.oy[p];
            oo[2] = a.oz[p];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                int b = cc[d] + g.mem - 1;
                bool up = oo[d] >= 0.5f;
                ip[d] = b + (up ? 1 : 0);
                dp[d] = up ? oo[d] - 1.0f : oo[d];
                id[d] = b;
                dd[d] = oo[d] - 0.5f;
            }
        }
        bool ok = true;
#pragma unroll
        for (int d = 0; d < 3; ++d) ok = ok && id[d] >= H && ip[d] <= g.f[d] - 1 - H;
        if (!ok) {
            set_status(a.status, ST_OOB);
            return false;
        }
        // ---- gather with gradients (Yee staggering, particle.cpp:207-259) -
        real ev[6], eg[6][3];
        {
        real wp[3][P], wd[3][P], gp[3][P], gd[3][P];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            shape_weights(dp[d], wp[d]);
            shape_weights(dd[d], wd[d]);
            shape_derivs(dp[d], gp[d]);
            shape_derivs(dd[d], gd[d]);
        }
        gather_grad<real, P, LDG>(fv[0], id[0] - H, ip[1] - H, ip[2] - H, wd[0], wp[1], wp[2], gd[0], gp[1], gp[2], ev[0], eg[0]);
        gather_grad<real, P, LDG>(fv[1], ip[0] - H, id[1] - H, ip[2] - H, wp[0], wd[1], wp[2], gp[0], gd[1], gp[2], ev[1], eg[1]);
        gather_grad<real, P, LDG>(fv[2], ip[0] - H, ip[1] - H, id[2] - H, wp[0], wp[1], wd[2], gp[0], gp[1], gd[2], ev[2], eg[2]);
        gather_grad<real, P, LDG>(fv[3], ip[0] - H, id[1] - H, id[2] - H, wp[0], wd[1], wd[2], gp[0], gd[1], gd[2], ev[3], eg[3]);
        gather_grad<real, P, LDG>(fv[4], id[0] - H, ip[1] - H, id[2] - H, wd[0], wp[1], wd[2], gd[0], gp[1], gd[2], ev[4], eg[4]);
        gather_grad<real, P, LDG>(fv[5], id[0] - H, id[1] - H, ip[2] - H, wd[0], wd[1], wp[2], gd[0], gd[1], gp[2], ev[5], eg[5]);
        }
        // ---- Boris: values only here (the displacement fixes the new
        // position); they are formed again for the transpose, after the deposit
        // adjoint ------------------------------------------------------------
        const real pin[3] = {a.px[p], a.py[p], a.pz[p]};
        real disp_v[3];
        {
            Boris<real> v;
            boris_values<real>(pin, ev, ev + 3, a.qm, v);
#pragma unroll
            for (int o = 0; o < 3; ++o) disp_v[o] = v.pn[o] * v.ig * a.dt_d[o];
        }
        // ---- new position, as the forward deposit forms it ----------------
        int i2[3];
        double d2[3], d0[3];
        if constexpr (F64) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                double xc = (xd[d] + (double)disp_v[d]) - (double)(1 - g.mem);
                i2[d] = (int)(xc + 0.5);
                d2[d] = xc - (double)i2[d];
                d0[d] = dp[d];
            }
        } else {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                double u = (double)oo[d] + (double)disp_v[d];
                double f = floor(u + 0.5);
                i2[d] = cc[d] + g.mem - 1 + (int)f;
                d2[d] = u - f;
                d0[d] = (double)dp[d];
            }
        }
        bool cfl = abs(i2[0] - ip[0]) <= 1 && abs(i2[1] - ip[1]) <= 1 && abs(i2[2] - ip[2]) <= 1;
        if (!cfl) {
            set_status(a.status, ST_CFL);
            return false;
        }
        // ---- deposit adjoint ----------------------------------------------
        constexpr double kInvSqrt12 = 0.28867513459481287;
        double ss[3][P + 1], sd[3][P + 1];   // s and d of each axis on the common span
        double gs[3][P + 1], gd[3][P + 1];   // dG1 / d(s, d)
        int base[3], len[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            double w0[P], w1[P], u0[P + 1], u1[P + 1];
            shape_weights(d0[d], w0);
            shape_weights(d2[d], w1);
            span_pair<double, P>(ip[d], w0, i2[d], w1, u0, u1);
            base[d] = min(ip[d], i2[d]) - H;
            len[d] = P + abs(i2[d] - ip[d]);
#pragma unroll
            for (int q = 0; q <= P; ++q) {
                ss[d][q] = 0.5 * (u0[q] + u1[q]);
                sd[d][q] = kInvSqrt12 * (u1[q] - u0[q]);
                gs[d][q] = gd[d][q] = 0.0;
            }
        }
        const double qd = (double)a.charge;
        double G1 = 0.0;
        // Jx: running sum along x, weight from y and z (particle.cpp:427-450);
        // the J adjoints are read in place from the ring buffers
#pragma unroll 1
        for (int comp = 0; comp < 3; ++comp) {
            const real *lbuf = lj[comp].at(base[2], base[1], base[0]);
            const int sX = 1, sY = lj[comp].sy, sZ = lj[comp].sz;
            if (comp == 0)
                G1 += esirkepov_adj<P, LDG>(lbuf, sX, sY, sZ, len[0], len[1], len[2], -qd * a.d_dt[0], sd[0], ss[1], sd[1],
                                            ss[2], sd[2], gd[0], gs[1], gd[1], gs[2], gd[2]);
            else if (comp == 1)
                G1 += esirkepov_adj<P, LDG>(lbuf, sY, sX, sZ, len[1], len[0], len[2], -qd * a.d_dt[1], sd[1], ss[0], sd[0],
                                            ss[2], sd[2], gd[1], gs[0], gd[0], gs[2], gd[2]);
            else
                G1 += esirkepov_adj<P, LDG>(lbuf, sZ, sX, sY, len[2], len[0], len[1], -qd * a.d_dt[2], sd[2], ss[0], sd[0],
                                            ss[1], sd[1], gd[2], gs[0], gd[0], gs[1], gd[1]);
        }
        const double wgt = (double)a.w[p];
        a.lw[p] += G1;
        double dGx0[3], dGx1[3];   // d G / d x_old, d G / d x_new
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            double v0[P], v1[P], t0[P + 1], t1[P + 1];   // weight derivatives on the span
            shape_derivs(d0[d], v0);
            shape_derivs(d2[d], v1);
            span_pair<double, P>(ip[d], v0, i2[d], v1, t0, t1);
            double s_0 = 0.0, s_1 = 0.0;
#pragma unroll
            for (int q = 0; q <= P; ++q) {
                const double hs = 0.5 * gs[d][q], hd = kInvSqrt12 * gd[d][q];
                s_0 += (hs - hd) * t0[q];
                s_1 += (hs + hd) * t1[q];
            }
            dGx0[d] = wgt * s_0;
            dGx1[d] = wgt * s_1;
        }
        // ---- chain rule: lin = J^T (lp', lx') ----------------------------
        const real lxn[3] = {a.lx[p] + (real)dGx1[0], a.ly[p] + (real)dGx1[1], a.lz[p] + (real)dGx1[2]};
        const real lpn[3] = {a.lpx[p], a.lpy[p], a.lpz[p]};
        {
            Boris<real> v;
            boris_values<real>(pin, ev, ev + 3, a.qm, v);
            boris_transpose<real>(v, a.qm, a.dt_d, lpn, lxn, lin);
        }
        real lxo[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            real s = lxn[d] + (real)dGx0[d];
#pragma unroll
            for (int c = 0; c < 6; ++c) s += lin[3 + c] * eg[c][d];
            lxo[d] = s;
        }
        a.lx[p] = lxo[0];
        a.ly[p] = lxo[1];
        a.lz[p] = lxo[2];
        a.lpx[p] = lin[0];
        a.lpy[p] = lin[1];
        a.lpz[p] = lin[2];
        return true;
    }
}

// The gather weights of the six staggered components of a particle at its
// tape position (primal/dual index and offset per axis), for the scatter.
template <typename real, int P>
__device__ __forceinline__ void gather_stencils(const AdjPushArgs<real> &a, long long p, int (&ip)[3], int (&id)[3],
                                                real (&wp)[3][P], real (&wd)[3][P]) {
    const Geom &g = a.g;
    if constexpr (sizeof(real) == 8) {
        const double xd[3] = {a.x[p], a.y[p], a.z[p]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            double xc = xd[d] - (double)(1 - g.mem);
            ip[d] = (int)(xc + 0.5);
            id[d] = (int)xc;
            shape_weights((real)(xc - (double)ip[d]), wp[d]);
            shape_weights((real)((xc - 0.5) - (double)id[d]), wd[d]);
        }
    } else {
        int cc[3];
        a.cp.unpack(a.cell[p], cc[0], cc[1], cc[2]);
        const real oo[3] = {a.ox[p], a.oy[p], a.oz[p]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int b = cc[d] + g.mem - 1;
            const bool up = oo[d] >= 0.5f;
            ip[d] = b + (up ? 1 : 0);
            id[d] = b;
            shape_weights(up ? oo[d] - 1.0f : oo[d], wp[d]);
            shape_weights(oo[d] - 0.5f, wd[d]);
        }
    }
}

template <typename real, int P>
__global__ void __launch_bounds__(128) adj_push_kernel(AdjPushArgs<real> a) {
    constexpr int H = P / 2;
    const Geom &g = a.g;
    View<const real> fv[6], lj[3];
#pragma unroll
    for (int c = 0; c < 6; ++c) fv[c] = View<const real>{a.f[c], g.f[0], g.fxy, 0};
#pragma unroll
    for (int c = 0; c < 3; ++c) lj[c] = View<const real>{a.lj[c], g.r[0], g.rxy, g.rxy + g.r[0] + 1};
    const long long n = a.idx ? (long long)*a.nidx : a.n;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
        const long long p = a.idx ? (long long)a.idx[t] : t;
        if (a.dead && a.dead[p]) continue;
        real lin[9];
        if (!adj_particle<real, P, true>(a, p, fv, lj, lin)) continue;
        if (a.scatter_fields) {
            int ip[3], id[3];
            real wp[3][P], wd[3][P];   // the gather weights again (cheaper than keeping them live)
            gather_stencils<real, P>(a, p, ip, id, wp, wd);
            scatter_adj<real, P>(a.lf[0], g, id[0] - H, ip[1] - H, ip[2] - H, wd[0], wp[1], wp[2], lin[3]);
            scatter_adj<real, P>(a.lf[1], g, ip[0] - H, id[1] - H, ip[2] - H, wp[0], wd[1], wp[2], lin[4]);
            scatter_adj<real, P>(a.lf[2], g, ip[0] - H, ip[1] - H, id[2] - H, wp[0], wp[1], wd[2], lin[5]);
            scatter_adj<real, P>(a.lf[3], g, ip[0] - H, id[1] - H, id[2] - H, wp[0], wd[1], wd[2], lin[6]);
            scatter_adj<real, P>(a.lf[4], g, id[0] - H, ip[1] - H, id[2] - H, wd[0], wp[1], wd[2], lin[7]);
            scatter_adj<real, P>(a.lf[5], g, id[0] - H, id[1] - H, ip[2] - H, wd[0], wd[1], wp[2], lin[8]);
        }
    }
}

// ---------------------------------------------------------------------------
// Tiled push adjoint.  The tape holds the particles in the order of the
// forward push, i.e. sorted by tile at the last sort; with each sort the tape
// also keeps the tile boundaries of that order.  One CTA per tile:
//   1. stages the tape's six field components over the tile's gather box
//      and the three J adjoints over its deposit box in shared memory; then,
//      for as many particles at a time as the scratch holds,
//   2. runs each particle's push adjoint from shared memory, keeping the
//      adjoints of its gathered E and B (six values) and their largest
//      magnitude per component;
//   3. adds every particle's field adjoint times its gather weights into
//      fixed-point shared accumulators (20-bit limbs, scaled so that the
//      largest value fits), then flushes them with one pass of global atomics.
// Particles that left their tile since the sort go to the global kernel
// afterwards.
//
// What bounds it: latency.  About 15 k instructions per 32 particles (scatter
// 30 %, Esirkepov transpose in FP64 27 %, gather with gradients 20 %) issue at
// 0.34 of the rate, two warps per scheduler at 255 registers.  384 or 512
// threads spill and are no faster (FP32 592 and 618 against 593 us, FP64 352
// and 423 against 339 us, 48 x 32 x 32 and 32 x 24 x 24 cells with 8 per cell),
// nor are two FP32 CTAs of 128 threads (565 against 559 us).

struct AdjTileGeom {
    int T, nt[3];
    int nodes;               // 1: tiles of nodes, 0: tiles of cells
    int GE, DE;
    int gsy, gsz, gsize, dsy, dsz, dsize;
    int cap;                 // particles the shared scratch holds
};

template <typename real>
constexpr int adj_limbs() { return sizeof(real) == 8 ? 3 : 2; }

// Zeros are added like any value: a per-point zero test measured 9 % slower
// on the whole reverse sweep (as on the forward deposit).
template <typename real, int NL>
__device__ __forceinline__ void fixed_add(unsigned *a, int lstride, real q) {
    if constexpr (NL == 3) {
        const long long qi = __double_as_longlong((double)q + 6755399441055744.0) - 0x4338000000000000LL;
        atomicAdd(a, (unsigned)(qi & 0xFFFFF));
        atomicAdd(a + lstride, (unsigned)((qi >> 20) & 0xFFFFF));
        atomicAdd(a + 2 * lstride, (unsigned)(int)(qi >> 40));
    } else {
        const int qi = __float2int_rn((float)q);
        atomicAdd(a, (unsigned)qi & 0xFFFFFu);
        atomicAdd(a + lstride, (unsigned)(qi >> 20));
    }
}

// TT: the tile edge as a compile-time constant (0: from tg), which makes
// every shared-box stride a constant.
constexpr int kAdjThreads = 256;
template <typename real, int P, int TT>
__global__ void __launch_bounds__(kAdjThreads, 1) adj_tile_kernel(const __grid_constant__ AdjPushArgs<real> a, AdjTileGeom tg,
                                                          const unsigned *toffs, int *strag, unsigned long long *nstrag) {
    AdjTileGeom t = tg;
    if constexpr (TT > 0) {
        constexpr int ge = TT + 2 * (P / 2) + 1, de = TT + 2 * (P / 2) + 3;
        constexpr int gy = padded_row(ge, TT), gz = padded_plane(ge, TT);
        constexpr int dy = padded_row(de, TT), dz = padded_plane(de, TT);
        t.T = TT; t.GE = ge; t.DE = de;
        t.gsy = gy; t.gsz = gz; t.gsize = ge * gz;
        t.dsy = dy; t.dsz = dz; t.dsize = de * dz;
    }
    constexpr int H = P / 2, NL = adj_limbs<real>(), NT = kAdjThreads;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Geom &g = a.g;
    const int T = t.T, GE = t.GE, DE = t.DE, GS = t.gsize, DS = t.dsize;
    real *sf = reinterpret_cast<real *>(smem_raw);              // 6 x GS
    real *sl = sf + 6 * GS;                                       // 3 x DS
    real *slin = sl + 3 * DS;                                     // cap x 6
    unsigned *acc = reinterpret_cast<unsigned *>(slin + 6 * t.cap);   // 6 x NL x GS
    unsigned *smax = acc + 6 * NL * GS;                           // 6 (bits of non-negative values)
    unsigned char *flag = reinterpret_cast<unsigned char *>(smax + 8);   // cap
    const int tile = blockIdx.x;
    const int tx = tile % t.nt[0], ty = (tile / t.nt[0]) % t.nt[1], tz = tile / (t.nt[0] * t.nt[1]);
    const int t0[3] = {tx * T, ty * T, tz * T};
    int gO[3], dO[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        // the lowest dual stencil starts a point lower where tiles hold nodes
        gO[d] = t0[d] + g.mem - 1 - H - t.nodes;
        dO[d] = t0[d] + g.mem - 2 - H;
    }
    long long pa = toffs[tile], pb = toffs[tile + 1];
    pb = pb < a.n ? pb : a.n;
    if (pa >= pb) return;
    const int m_all = (int)(pb - pa);
    const int G2 = GE * GE, G3 = G2 * GE, D2 = DE * DE, D3 = D2 * DE;
    for (int l = threadIdx.x; l < G3; l += NT) {
        const int lz = l / G2, r = l - lz * G2, ly = r / GE, lx = r - ly * GE;
        const int x = gO[0] + lx, y = gO[1] + ly, z = gO[2] + lz;
        const bool in = x >= 0 && x < g.f[0] && y >= 0 && y < g.f[1] && z >= 0 && z < g.f[2];
        const int src = in ? g.fi(z, y, x) : 0;
        real *dst = sf + lz * t.gsz + ly * t.gsy + lx;
#pragma unroll
        for (int c = 0; c < 6; ++c) cp_async<sizeof(real)>(dst + c * GS, a.f[c] + src, in ? (int)sizeof(real) : 0);
    }
    for (int l = threadIdx.x; l < D3; l += NT) {
        const int lz = l / D2, r = l - lz * D2, ly = r / DE, lx = r - ly * DE;
        const int x = dO[0] + lx, y = dO[1] + ly, z = dO[2] + lz;
        const bool in = x >= -1 && x <= g.f[0] && y >= -1 && y <= g.f[1] && z >= -1 && z <= g.f[2];
        const int src = in ? g.ri(z, y, x) : 0;
        real *dst = sl + lz * t.dsz + ly * t.dsy + lx;
#pragma unroll
        for (int c = 0; c < 3; ++c) cp_async<sizeof(real)>(dst + c * DS, a.lj[c] + src, in ? (int)sizeof(real) : 0);
    }
    cp_async_commit();
    for (int e = threadIdx.x; e < 6 * NL * GS; e += NT) acc[e] = 0u;
    if (threadIdx.x < 6) smax[threadIdx.x] = 0u;
    cp_async_wait_all();
    __syncthreads();
    View<const real> fv[6], lj[3];
#pragma unroll
    for (int c = 0; c < 6; ++c) fv[c] = View<const real>{sf + c * GS, t.gsy, t.gsz, -(gO[2] * t.gsz + gO[1] * t.gsy + gO[0])};
#pragma unroll
    for (int c = 0; c < 3; ++c) lj[c] = View<const real>{sl + c * DS, t.dsy, t.dsz, -(dO[2] * t.dsz + dO[1] * t.dsy + dO[0])};
#pragma unroll 1
    for (int first = 0; first < m_all; first += t.cap, pa += t.cap) {
        const int m = min(t.cap, m_all - first);
        // 2. the particles' push adjoints
#pragma unroll 1
        for (int i = threadIdx.x; i < m; i += NT) {
            const long long p = pa + i;
            flag[i] = 0;
            if (a.dead && a.dead[p]) continue;
            // dual index (the cell's lower primal point), or the node, per axis
            int at[3];
            if constexpr (sizeof(real) == 8) {
                const double half = t.nodes ? 0.5 : 0.0;
                at[0] = (int)(a.x[p] - (double)(1 - g.mem) + half);
                at[1] = (int)(a.y[p] - (double)(1 - g.mem) + half);
                at[2] = (int)(a.z[p] - (double)(1 - g.mem) + half);
            } else {
                int cc[3];
                a.cp.unpack(a.cell[p], cc[0], cc[1], cc[2]);
                const float o[3] = {a.ox[p], a.oy[p], a.oz[p]};
#pragma unroll
                for (int d = 0; d < 3; ++d) at[d] = cc[d] + g.mem - 1 + (t.nodes && o[d] >= 0.5f ? 1 : 0);
            }
            bool inside = true;
#pragma unroll
            for (int d = 0; d < 3; ++d) inside = inside && at[d] >= t0[d] + g.mem - 1 && at[d] < t0[d] + g.mem - 1 + T;
            if (!inside) {
                strag[atomicAdd(nstrag, 1ull)] = (int)p;
                continue;
            }
            real lin[9];
            if (!adj_particle<real, P, false>(a, p, fv, lj, lin)) continue;
            if (!a.scatter_fields) continue;
            flag[i] = 1;
            // per component the largest magnitude of the tile: reduced over the
            // warp's active lanes first, one shared atomic per warp
            const unsigned am = __activemask();
            const bool leader = (threadIdx.x & 31) == __ffs(am) - 1;
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                slin[c * t.cap + i] = lin[3 + c];
                const unsigned mag = __reduce_max_sync(am, __float_as_uint((float)fabs(lin[3 + c])));
                if (leader) atomicMax(smax + c, mag);
            }
        }
        if (!a.scatter_fields) continue;
        __syncthreads();
        // 3. field adjoints into fixed point, then one flush
        const double lim = sizeof(real) == 8 ? 2251799813685248.0 /* 2^51 */ : 2147483648.0 /* 2^31 */;
        real scale[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            const double mx = (double)__uint_as_float(smax[c]);
            scale[c] = mx > 0.0 ? (real)(lim / (1.01 * mx)) : real(0);
        }
        // Sorted by node, neighbouring particles add to the same points: the
        // lanes of a warp take particles m / 32 apart.
        const int step = t.nodes ? (m + 31) >> 5 : 1;
        const int lane = threadIdx.x & 31, nb = (m + 31) >> 5;
#pragma unroll 1
        for (int b = threadIdx.x >> 5; b < nb; b += NT / 32) {
            const int i = t.nodes ? lane * step + b : b * 32 + lane;
            if (i >= m || !flag[i]) continue;
            int ip[3], id[3];
            real wp[3][P], wd[3][P];
            gather_stencils<real, P>(a, pa + i, ip, id, wp, wd);
#pragma unroll 1
            for (int c = 0; c < 6; ++c) {
                const real q = slin[c * t.cap + i] * (c == 0 ? scale[0] : c == 1 ? scale[1] : c == 2 ? scale[2] : c == 3 ? scale[3]
                                                      : c == 4 ? scale[4] : scale[5]);
                if (q == real(0)) continue;
                // dual axes (Yee staggering as in the gather): Ex x; Ey y; Ez z; Bx y, z; By x, z; Bz x, y
                const bool dx_ = c == 0 || c == 4 || c == 5, dy_ = c == 1 || c == 3 || c == 5,
                           dz_ = c == 2 || c == 3 || c == 4;
                real wx[P], wy[P], wz[P];
#pragma unroll
                for (int q2 = 0; q2 < P; ++q2) {
                    wx[q2] = dx_ ? wd[0][q2] : wp[0][q2];
                    wy[q2] = dy_ ? wd[1][q2] : wp[1][q2];
                    wz[q2] = dz_ ? wd[2][q2] : wp[2][q2];
                }
                unsigned *ac = acc + c * NL * GS;
                const int b0 = ((dz_ ? id[2] : ip[2]) - H - gO[2]) * t.gsz + ((dy_ ? id[1] : ip[1]) - H - gO[1]) * t.gsy +
                               ((dx_ ? id[0] : ip[0]) - H - gO[0]);
#pragma unroll 1
                for (int k = 0; k < P; ++k) {
                    const real qk = q * pick(wz, k);
#pragma unroll
                    for (int j = 0; j < P; ++j) {
                        const real qj = qk * wy[j];
#pragma unroll
                        for (int ii = 0; ii < P; ++ii)
                            fixed_add<real, NL>(ac + b0 + k * t.gsz + j * t.gsy + ii, GS, qj * wx[ii]);
                    }
                }
            }
        }
        __syncthreads();
        const bool more = first + t.cap < m_all;
        double inv[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) inv[c] = scale[c] > real(0) ? 1.0 / (double)scale[c] : 0.0;
        if (threadIdx.x < 6) smax[threadIdx.x] = 0u;
        for (int l = threadIdx.x; l < G3; l += NT) {
            const int lz = l / G2, r = l - lz * G2, ly = r / GE, lx = r - ly * GE;
            const int x = gO[0] + lx, y = gO[1] + ly, z = gO[2] + lz;
            const bool in = x >= 0 && x < g.f[0] && y >= 0 && y < g.f[1] && z >= 0 && z < g.f[2];
            const int dst = in ? g.fi(z, y, x) : 0;
            unsigned *q = acc + lz * t.gsz + ly * t.gsy + lx;
#pragma unroll
            for (int c = 0; c < 6; ++c, q += NL * GS) {
                long long tot;
                if constexpr (NL == 2) tot = ((long long)(int)q[GS] << 20) + (long long)q[0];
                else tot = ((long long)(int)q[2 * GS] << 40) + ((long long)q[GS] << 20) + (long long)q[0];
                if (tot == 0) continue;
                if (more) {
#pragma unroll
                    for (int n = 0; n < NL; ++n) q[n * GS] = 0u;
                }
                if (in) atomic_add(a.lf[c] + dst, (real)((double)tot * inv[c]));
            }
        }
        __syncthreads();
    }
}

__global__ void tile_bounds_kernel(const unsigned *offs, long long keys_per_tile, int ntiles, unsigned *out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t <= ntiles) out[t] = offs[(long long)t * keys_per_tile];
}

// ---------------------------------------------------------------------------
// transposes of the Yee half-updates (physical cells only, absorbing faces)

__device__ __forceinline__ bool physical(const Geom &g, int k, int j, int i) {
    return i >= g.mem && i < g.n[0] + g.mem && j >= g.mem && j < g.n[1] + g.mem && k >= g.mem && k < g.n[2] + g.mem;
}

// transpose of E += h (curl B - J): lamB += h curl^T lamE, lamJ -= h lamE
template <typename real>
__global__ void adj_update_e_kernel(Geom g, const real *lex, const real *ley, const real *lez, real *lbx, real *lby,
                                    real *lbz, real *ljx, real *ljy, real *ljz, real h, real idx, real idy, real idz) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.fsz) return;
    int i = (int)(t % g.f[0]), j = (int)((t / g.f[0]) % g.f[1]), k = (int)(t / g.fxy);
    const int q = (int)t;
    auto L = [&](const real *a, int kk, int jj, int ii) -> real {
        return (ii < g.f[0] && jj < g.f[1] && kk < g.f[2] && physical(g, kk, jj, ii)) ? a[g.fi(kk, jj, ii)] : real(0);
    };
    real ex0 = L(lex, k, j, i), ey0 = L(ley, k, j, i), ez0 = L(lez, k, j, i);
    lbz[q] += h * idy * (ex0 - L(lex, k, j + 1, i)) - h * idx * (ey0 - L(ley, k, j, i + 1));
    lby[q] += -h * idz * (ex0 - L(lex, k + 1, j, i)) + h * idx * (ez0 - L(lez, k, j, i + 1));
    lbx[q] += h * idz * (ey0 - L(ley, k + 1, j, i)) - h * idy * (ez0 - L(lez, k, j + 1, i));
    if (physical(g, k, j, i)) {
        const int r = g.ri(k, j, i);
        ljx[r] -= h * ex0;
        ljy[r] -= h * ey0;
        ljz[r] -= h * ez0;
    }
}

// transpose of B -= h curl E: lamE -= h curl^T lamB
template <typename real>
__global__ void adj_update_b_kernel(Geom g, real *lex, real *ley, real *lez, const real *lbx, const real *lby,
                                    const real *lbz, real h, real idx, real idy, real idz) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.fsz) return;
    int i = (int)(t % g.f[0]), j = (int)((t / g.f[0]) % g.f[1]), k = (int)(t / g.fxy);
    const int q = (int)t;
    auto L = [&](const real *a, int kk, int jj, int ii) -> real {
        return (ii >= 0 && jj >= 0 && kk >= 0 && physical(g, kk, jj, ii)) ? a[g.fi(kk, jj, ii)] : real(0);
    };
    real bx0 = L(lbx, k, j, i), by0 = L(lby, k, j, i), bz0 = L(lbz, k, j, i);
    lez[q] += -h * idy * L(lbx, k, j - 1, i) + h * idy * bx0 + h * idx * L(lby, k, j, i - 1) - h * idx * by0;
    ley[q] += h * idz * L(lbx, k - 1, j, i) - h * idz * bx0 - h * idx * L(lbz, k, j, i - 1) + h * idx * bz0;
    lex[q] += -h * idz * L(lby, k - 1, j, i) + h * idz * by0 + h * idy * L(lbz, k, j - 1, i) - h * idy * bz0;
}

// transpose of radiating_boundary (boundary.cpp:42-99) at time t: the two
// B columns it overwrites hand their adjoint to the inputs of the formula
// and to the laser source; d source / d coefficient accumulates in lprof.
struct AdjBcArgs {
    Geom g;
    double dt, dx, dy, dz;
    double Pi, omega, l0, amp, dur, start, waist, xfocus, yfocus, zfocus, phase, time;
    int pol, envelope, profile_n;
    double *lprof;
};

__device__ double adj_envelope(const AdjBcArgs &L, double t) {
    t = t - L.start;
    if (L.envelope == 1) {
        if (t < 0.0 || t > 3.0 * L.dur) return 0.0;
        double r = (t - 1.5 * L.dur) / L.dur;
        return L.amp * exp(-2.0 * log(2.0) * r * r);
    }
    return (t >= 0.0 && t <= L.dur) ? L.amp * sin(L.Pi * t / L.dur) : 0.0;
}

template <typename real>
__global__ void adj_bc_kernel(AdjBcArgs A, real *lex, real *ley, real *lez, real *lbx, real *lby, real *lbz,
                              real *ljy, real *ljz) {
    (void)lex;
    const Geom &g = A.g;
    int iy = blockIdx.x * blockDim.x + threadIdx.x;
    int iz = blockIdx.y * blockDim.y + threadIdx.y;
    if (iy >= g.n[1] || iz >= g.n[2]) return;
    iy += g.mem;
    iz += g.mem;
    const double alpha = 1 / (1 + A.dt / A.dx), beta = 1 - A.dt / A.dx;
    const int m = g.mem, L = g.n[0];
    double lsrc = 0.0;
    for (int side = 0; side < 2; ++side) {
        const int col = side == 0 ? m : L, out = side == 0 ? m - 1 : L + 1;
        const int c = g.fi(iz, iy, col), o = g.fi(iz, iy, out), rc = g.ri(iz, iy, col);
        const double Lz = lbz[o], Ly = lby[o];
        lbz[o] = 0;
        lby[o] = 0;
        const double sg = side == 0 ? 1.0 : -1.0;   // right column: signs of the E and J terms flip
        atomic_add(ley + c, (real)(-2 * alpha * sg * Lz));
        atomic_add(lbx + c, (real)(-alpha * A.dt / A.dz * Lz + alpha * A.dt / A.dy * Ly));
        atomic_add(lbx + c - g.fxy, (real)(alpha * A.dt / A.dz * Lz));
        atomic_add(lbx + c - g.f[0], (real)(-alpha * A.dt / A.dy * Ly));
        atomic_add(lbz + c, (real)(-alpha * beta * Lz));
        atomic_add(ljy + rc, (real)(-alpha * A.dt * sg * Lz));
        atomic_add(lez + c, (real)(2 * alpha * sg * Ly));
        atomic_add(lby + c, (real)(-alpha * beta * Ly));
        atomic_add(ljz + rc, (real)(alpha * A.dt * sg * Ly));
        if (side == 0) {
            if (A.pol == 1 || A.pol == 3) lsrc += 4 * alpha * Lz;
            if (A.pol == 2 || A.pol == 3) lsrc += -4 * alpha * Ly;
        }
    }
    if (!A.lprof || lsrc == 0.0) return;
    // d source / d coefficient (laser_profile = 1): -env * B_c(u) B_b(v) * cos(PHI + phase)
    const double k = 2.0 * A.Pi / A.l0, rl = 0.5 * k * A.waist * A.waist, xe = 0.0 - A.xfocus;
    const double y = iy * A.dy - A.yfocus, z = iz * A.dz - A.zfocus;
    const double q = xe / rl, w = A.waist * sqrt(1 + q * q);
    const double PHI = (xe / rl) * (y * y + z * z) / w / w - atan(xe / rl) + k * xe - A.omega * A.time;
    const double f = -1.0 * adj_envelope(A, A.time) * cos(PHI + A.phase);
    if (f == 0.0) return;
    const int nc = A.profile_n;
    const double u = ((double)(iy - g.mem) + 0.5) / (double)g.n[1] * (double)(nc - 1);
    const double v = ((double)(iz - g.mem) + 0.5) / (double)g.n[2] * (double)(nc - 1);
    // the coefficients within two knots (the others' basis is zero)
    const int b0 = max((int)floor(v) - 1, 0), b1 = min((int)floor(v) + 2, nc - 1);
    const int c0 = max((int)floor(u) - 1, 0), c1 = min((int)floor(u) + 2, nc - 1);
    for (int b = b0; b <= b1; ++b) {
        double wv = cubic_bspline(v - b);
        if (wv == 0.0) continue;
        for (int cidx = c0; cidx <= c1; ++cidx) {
            double wu = cubic_bspline(u - cidx);
            if (wu == 0.0) continue;
            atomicAdd(A.lprof + b * nc + cidx, lsrc * f * wu * wv);
        }
    }
}

// smooth window over [xlo, xhi): 0 outside, 1 inside, sin^2 ramps of width
// `ramp` cells at both ends (ramp = 0: a hard window); returns s(x), ds/dx
__device__ inline void window_weight(double x, double xlo, double xhi, double ramp, double &s, double &ds) {
    s = 0.0;
    ds = 0.0;
    if (!(x >= xlo && x < xhi)) return;
    const double half_pi = 1.5707963267948966;
    s = 1.0;
    if (ramp > 0.0) {
        const double up = (x - xlo) / ramp, down = (xhi - x) / ramp;
        if (up < 1.0) {
            double sn = sin(half_pi * up), cs = cos(half_pi * up);
            s = sn * sn;
            ds = 2.0 * sn * cs * half_pi / ramp;
        }
        if (down < 1.0) {
            double sn = sin(half_pi * down), cs = cos(half_pi * down);
            double s2 = sn * sn, d2 = -2.0 * sn * cs * half_pi / ramp;
            ds = ds * s2 + s * d2;
            s *= s2;
        }
    }
}

// objective: kinetic energy sum s(x) w m (gamma - 1) of the alive particles
// of a species, s the window weight above; seeds d objective / d (x, p, w)
template <typename real>
__global__ void adj_seed_kinetic_kernel(Geom g, CellPack cp, int fp32, long long n, const double *x, const int *cell,
                                        const float *ox, const real *px, const real *py, const real *pz,
                                        const real *w, const unsigned char *dead, double mass, double xlo,
                                        double xhi, double ramp, real *lx, real *lpx, real *lpy, real *lpz,
                                        double *lw, double *loss) {
    long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double contrib = 0.0;
    if (p < n && !(dead && dead[p])) {
        double xp;
        if (fp32) {
            int cx, cy, cz;
            cp.unpack(cell[p], cx, cy, cz);
            xp = (double)cx + (double)ox[p];
        } else {
            xp = x[p];
        }
        double sw, dsw;
        window_weight(xp, xlo, xhi, ramp, sw, dsw);
        if (sw != 0.0) {
            double a = px[p], b = py[p], c = pz[p];
            double u2 = a * a + b * b + c * c, gam = sqrt(1.0 + u2);
            double gm1 = u2 / (gam + 1.0);
            double wt = w[p];
            contrib = sw * wt * mass * gm1;
            lx[p] += (real)(dsw * wt * mass * gm1);
            lpx[p] += (real)(sw * wt * mass * a / gam);
            lpy[p] += (real)(sw * wt * mass * b / gam);
            lpz[p] += (real)(sw * wt * mass * c / gam);
            lw[p] += sw * mass * gm1;
        }
    }
    // warp reduction of the loss
    for (int o = 16; o > 0; o >>= 1) contrib += __shfl_down_sync(0xffffffffu, contrib, o);
    if ((threadIdx.x & 31) == 0 && contrib != 0.0) atomicAdd(loss, contrib);
}

}  // namespace pic

// Several device arrays of 16-byte aligned addresses copied in one launch
// (blockIdx.y: the array).  A tape slot has 16 or more of them and is saved
// before every push: one by one, 1.9 us and a launch each, they took a tenth
// of a small differentiable run.
struct CopyList {
    static constexpr int kMax = 24;
    const void *src[kMax];
    void *dst[kMax];
    unsigned long long bytes[kMax];
};

__global__ void __launch_bounds__(256) copy_arrays_kernel(const __grid_constant__ CopyList l) {
    const int a = blockIdx.y;
    const unsigned long long words = l.bytes[a] / 16, nt = (unsigned long long)gridDim.x * 256;
    const uint4 *src = (const uint4 *)l.src[a];
    uint4 *dst = (uint4 *)l.dst[a];
    for (unsigned long long i = (unsigned long long)blockIdx.x * 256 + threadIdx.x; i < words; i += nt) dst[i] = src[i];
    const unsigned tail = (unsigned)(l.bytes[a] & 15);
    if (blockIdx.x == 0 && threadIdx.x < tail)
        ((unsigned char *)dst)[words * 16 + threadIdx.x] = ((const unsigned char *)src)[words * 16 + threadIdx.x];
}

// The same permutation of several per-particle arrays in one launch (bit
// copies between orders):
// out[map[i]] = in[i], or (GATHER) out[i] = in[map[i]].
struct PermuteList {
    const unsigned long long *ds[8];
    unsigned long long *dd[8];
    int nd;
    const unsigned *fs[8];
    unsigned *fd[8];
    int nf;
};

template <bool GATHER>
__global__ void __launch_bounds__(256) permute_kernel(const __grid_constant__ PermuteList l, const int *map, long long n) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const long long j = map[i], from = GATHER ? j : i, to = GATHER ? i : j;
    pic::move_words(l.ds, l.dd, l.nd, from, to);
    pic::move_words(l.fs, l.fd, l.nf, from, to);
}

// ===========================================================================
// host side: checkpoints, tape and the C ABI
// ===========================================================================

using namespace pic;

struct Blob {
    std::vector<std::pair<void *, size_t>> parts;   // (device pointer, bytes) at save time
    void *buf = nullptr;
    size_t bytes = 0;
    int step = 0;
    int cur[2] = {0, 0};
    long long count[2] = {0, 0};
    int field_part = 0;          // tape: index of the first of the six field parts
    int perm_part[2] = {-1, -1}; // tape: the sort permutation run right before this push, per species
    int toff_part[2] = {-1, -1}; // tape: tile boundaries of the particle order of this push, per species
};

struct AdjState {
    std::vector<Blob> ckpt;
    std::vector<Blob> tape;
    int tape_len = 0;
    bool recording = false;
    // adjoint arrays
    void *lf[6] = {};        // field-buffer adjoints (E, B)
    void *lj[3] = {};        // ring-buffer adjoints (J)
    void *lpart[2][6] = {};  // per species: lx, ly, lz, lpx, lpy, lpz
    double *lw[2] = {};
    double *lprof = nullptr;
    double *loss = nullptr;
    int nprof = 0;
    // tiled contexts: upload index of each particle in the order the
    // per-particle adjoints are held in (valid once seeded), and scratch
    int *lam_orig[2] = {};
    bool lam_valid = false;
    unsigned *toffs[2] = {};   // tiled contexts: tile boundaries extracted for the tape
    // second set of the per-particle arrays: where a permutation goes
    void *lpart_b[2][6] = {};
    double *lw_b[2] = {};
};

static std::vector<std::pair<pic_ctx *, AdjState *>> g_adj;

static AdjState *adj_of(pic_ctx *c, bool create) {
    for (auto &e : g_adj)
        if (e.first == c) return e.second;
    if (!create) return nullptr;
    g_adj.push_back({c, new AdjState()});
    return g_adj.back().second;
}

static size_t rsize(const pic_ctx *c) { return c->fp32 ? 4 : 8; }

// pieces of the particle state (current positions, momenta, dead flags)
static void particle_parts(pic_ctx *c, std::vector<std::pair<void *, size_t>> &v) {
    for (int k = 0; k < 2; ++k) {
        Species &s = c->sp[k];
        size_t n = (size_t)s.n_host;
        if (n == 0) continue;
        if (c->fp32) {
            v.push_back({s.a.cell[s.cur], n * 4});
            v.push_back({s.a.ox[s.cur], n * 4});
            v.push_back({s.a.oy[s.cur], n * 4});
            v.push_back({s.a.oz[s.cur], n * 4});
        } else {
            v.push_back({s.a.x[s.cur], n * 8});
            v.push_back({s.a.y[s.cur], n * 8});
            v.push_back({s.a.z[s.cur], n * 8});
        }
        v.push_back({s.a.px, n * rsize(c)});
        v.push_back({s.a.py, n * rsize(c)});
        v.push_back({s.a.pz, n * rsize(c)});
        if (s.dead) v.push_back({s.dead, n});
    }
}

// a checkpoint additionally holds what a sort moves but the tape need not:
// weights, ids and upload indices (tiled contexts)
static void checkpoint_parts(pic_ctx *c, std::vector<std::pair<void *, size_t>> &v) {
    particle_parts(c, v);
    for (int k = 0; k < 2; ++k) {
        Species &s = c->sp[k];
        size_t n = (size_t)s.n_host;
        if (n == 0 || !s.orig) continue;
        v.push_back({s.a.w, n * rsize(c)});
        v.push_back({s.a.id, n * sizeof(int)});
        v.push_back({s.orig, n * sizeof(int)});
    }
    for (int f = 0; f < 6; ++f) v.push_back({c->field[f], (size_t)c->g.fsz * rsize(c)});
    for (int f = 0; f < 5; ++f) v.push_back({c->ring[f], (size_t)c->g.rsz * rsize(c)});
}

// between the parts and their places in the blob, as many arrays per launch
// as a list holds
static void copy_parts(pic_ctx *c, const Blob &b, const std::vector<std::pair<void *, size_t>> &parts, bool save) {
    size_t off = 0;
    for (size_t i = 0; i < parts.size();) {
        CopyList l{};
        int m = 0;
        size_t most = 0;
        for (; i < parts.size() && m < CopyList::kMax; ++i, ++m) {
            void *in_blob = (char *)b.buf + off;
            l.src[m] = save ? parts[i].first : in_blob;
            l.dst[m] = save ? in_blob : parts[i].first;
            l.bytes[m] = parts[i].second;
            most = std::max(most, parts[i].second);
            off += (parts[i].second + 255) & ~(size_t)255;
        }
        // four words per thread, at most 4 blocks per SM for one array
        const unsigned grid = (unsigned)std::min<size_t>(most / 16 / 1024 + 1, 148 * 4);
        copy_arrays_kernel<<<dim3(grid, (unsigned)m), 256, 0, c->stream>>>(l);
    }
}

static int blob_save(pic_ctx *c, Blob &b, const std::vector<std::pair<void *, size_t>> &parts) {
    size_t total = 0;
    for (auto &p : parts) total += (p.second + 255) & ~(size_t)255;
    if (b.bytes < total) {
        if (b.buf) cudaFree(b.buf);
        b.buf = nullptr;
        b.bytes = 0;
        if (cudaMalloc(&b.buf, total) != cudaSuccess) {
            c->err = "adjoint: out of device memory for a checkpoint / tape slot";
            return PIC_ENOMEM;
        }
        b.bytes = total;
    }
    b.parts = parts;
    copy_parts(c, b, parts, true);
    b.step = c->step;
    for (int k = 0; k < 2; ++k) {
        b.cur[k] = c->sp[k].cur;
        b.count[k] = c->sp[k].n_host;
    }
    return PIC_OK;
}

// the tape slot's device pointer of part `idx`
static void *blob_part(const Blob &b, int idx) {
    size_t off = 0;
    for (int i = 0; i < idx; ++i) off += (b.parts[i].second + 255) & ~(size_t)255;
    return (char *)b.buf + off;
}

namespace pic {
// called by the step orchestration right before each push while recording
void adjoint_record_hook(pic_ctx *c) {
    AdjState *A = adj_of(c, false);
    if (!A || !A->recording) return;
    if (A->tape_len >= (int)A->tape.size()) {
        c->err = "adjoint tape full";
        return;
    }
    std::vector<std::pair<void *, size_t>> parts;
    particle_parts(c, parts);
    const int field_part = (int)parts.size();
    for (int f = 0; f < 6; ++f) parts.push_back({c->field[f], (size_t)c->g.fsz * rsize(c)});
    int perm_part[2] = {-1, -1}, toff_part[2] = {-1, -1};
    for (int k = 0; k < 2; ++k) {
        Species &s = c->sp[k];
        if (!s.perm_fresh || s.n_host == 0) continue;
        perm_part[k] = (int)parts.size();
        parts.push_back({s.perm, (size_t)s.n_host * sizeof(int)});
        s.perm_fresh = false;
    }
    const int ntiles = c->ntile[0] * c->ntile[1] * c->ntile[2];
    for (int k = 0; k < 2; ++k) {
        Species &s = c->sp[k];
        if (c->tile <= 0 || s.n_host == 0 || !s.sorted || !A->toffs[k]) continue;
        const long long kpt = c->keys_per_tile;
        tile_bounds_kernel<<<(ntiles + 256) / 256, 256, 0, c->stream>>>(s.offs, kpt, ntiles, A->toffs[k]);
        toff_part[k] = (int)parts.size();
        parts.push_back({A->toffs[k], (size_t)(ntiles + 1) * sizeof(unsigned)});
    }
    prof_begin(c, "adjoint_tape_record");
    Blob &b = A->tape[A->tape_len];
    if (blob_save(c, b, parts) == PIC_OK) {
        b.field_part = field_part;
        b.perm_part[0] = perm_part[0];
        b.perm_part[1] = perm_part[1];
        b.toff_part[0] = toff_part[0];
        b.toff_part[1] = toff_part[1];
        A->tape_len++;
    }
    prof_end(c);
}
}  // namespace pic

static int ensure_adj_arrays(pic_ctx *c, AdjState *A) {
    const size_t rs = rsize(c);
    auto alloc = [&](void **p, size_t bytes) -> bool {
        if (*p) return true;
        if (cudaMalloc(p, bytes) != cudaSuccess) return false;
        return true;
    };
    bool ok = true;
    for (int f = 0; f < 6; ++f) ok = ok && alloc(&A->lf[f], (size_t)c->g.fsz * rs);
    // the three J adjoints in one block: cleared by one memset
    ok = ok && alloc(&A->lj[0], 3 * (size_t)c->g.rsz * rs);
    for (int f = 1; f < 3 && ok; ++f) A->lj[f] = (char *)A->lj[0] + (size_t)f * c->g.rsz * rs;
    for (int k = 0; k < 2; ++k) {
        size_t n = (size_t)std::max<int64_t>(c->sp[k].cap, 1);
        for (int q = 0; q < 6; ++q) ok = ok && alloc(&A->lpart[k][q], n * rs);
        ok = ok && alloc((void **)&A->lw[k], n * sizeof(double));
    }
    ok = ok && alloc((void **)&A->loss, sizeof(double));
    if (c->sp[0].orig || c->sp[1].orig) {
        size_t n = (size_t)std::max<int64_t>(std::max(c->sp[0].cap, c->sp[1].cap), 1);
        for (int k = 0; k < 2; ++k) {
            ok = ok && alloc((void **)&A->lam_orig[k], n * sizeof(int));
            size_t nk = (size_t)std::max<int64_t>(c->sp[k].cap, 1);
            for (int q = 0; q < 6; ++q) ok = ok && alloc(&A->lpart_b[k][q], nk * rs);
            ok = ok && alloc((void **)&A->lw_b[k], nk * sizeof(double));
        }
    }
    int np = std::max(c->profile_n * c->profile_n, 1);
    if (A->nprof != np && A->lprof) {
        cudaFree(A->lprof);
        A->lprof = nullptr;
    }
    ok = ok && alloc((void **)&A->lprof, (size_t)np * sizeof(double));
    A->nprof = np;
    if (!ok) {
        c->err = "adjoint: out of device memory";
        return PIC_ENOMEM;
    }
    return PIC_OK;
}

// The per-particle arrays a sort moves that the reverse sweep reads: the
// adjoints (position, momentum, weight) and, if `all`, weights and upload
// index; between the first and the second set of arrays.
static PermuteList moved_arrays(pic_ctx *c, AdjState *A, int k, bool all, bool back) {
    PermuteList l{};
    auto add = [&](void *a, void *b, size_t es) {
        if (back) std::swap(a, b);
        if (es == 8) {
            l.ds[l.nd] = (const unsigned long long *)a;
            l.dd[l.nd++] = (unsigned long long *)b;
        } else {
            l.fs[l.nf] = (const unsigned *)a;
            l.fd[l.nf++] = (unsigned *)b;
        }
    };
    Species &s = c->sp[k];
    for (int q = 0; q < 6; ++q) add(A->lpart[k][q], A->lpart_b[k][q], rsize(c));
    add(A->lw[k], A->lw_b[k], sizeof(double));
    if (all) {
        add(s.a.w, s.b.w, rsize(c));
        add(s.orig, s.orig_b, sizeof(int));
    }
    return l;
}

static void permute(pic_ctx *c, const PermuteList &l, const int *map, long long n, bool gather) {
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (gather) permute_kernel<true><<<blocks, 256, 0, c->stream>>>(l, map, n);
    else permute_kernel<false><<<blocks, 256, 0, c->stream>>>(l, map, n);
}

// undo one recorded sort of species k (perm[new] = old): every moved array
// goes back to the order before that sort, into the other set, which becomes
// the first
static void unsort_species(pic_ctx *c, AdjState *A, int k, const int *perm, long long n) {
    permute(c, moved_arrays(c, A, k, true, false), perm, n, false);
    Species &s = c->sp[k];
    for (int q = 0; q < 6; ++q) std::swap(A->lpart[k][q], A->lpart_b[k][q]);
    std::swap(A->lw[k], A->lw_b[k]);
    std::swap(s.a.w, s.b.w);
    std::swap(s.orig, s.orig_b);
}

// the adjoints are held in the order given by lam_orig (upload indices);
// bring them into the context's current order (its orig array): a segment
// recomputed from a checkpoint sorts again and need not end in the order
// the later segment's reverse sweep started from
static void remap_adjoints(pic_ctx *c, AdjState *A) {
    if (!A->lam_valid) return;
    for (int k = 0; k < 2; ++k) {
        Species &s = c->sp[k];
        const long long n = s.n_host;
        if (!s.orig || n == 0) continue;
        permute(c, moved_arrays(c, A, k, false, false), A->lam_orig[k], n, false);
        permute(c, moved_arrays(c, A, k, false, true), s.orig, n, true);
    }
}

static void note_adjoint_order(pic_ctx *c, AdjState *A) {
    for (int k = 0; k < 2; ++k) {
        Species &s = c->sp[k];
        if (s.orig && s.n_host > 0)
            cudaMemcpyAsync(A->lam_orig[k], s.orig, (size_t)s.n_host * sizeof(int), cudaMemcpyDeviceToDevice,
                            c->stream);
    }
    A->lam_valid = c->sp[0].orig || c->sp[1].orig;
}

template <typename real, int P>
static void adj_push_launch(pic_ctx *c, AdjState *A, const Blob &b, int kind, int part_base, int scatter) {
    Species &s = c->sp[kind];
    AdjPushArgs<real> a{};
    a.g = c->g;
    a.cp = c->cp;
    a.n = b.count[kind];
    int idx = part_base;
    if (c->fp32) {
        a.cell = (const int *)blob_part(b, idx++);
        a.ox = (const float *)blob_part(b, idx++);
        a.oy = (const float *)blob_part(b, idx++);
        a.oz = (const float *)blob_part(b, idx++);
    } else {
        a.x = (const double *)blob_part(b, idx++);
        a.y = (const double *)blob_part(b, idx++);
        a.z = (const double *)blob_part(b, idx++);
    }
    a.px = (const real *)blob_part(b, idx++);
    a.py = (const real *)blob_part(b, idx++);
    a.pz = (const real *)blob_part(b, idx++);
    a.dead = s.dead ? (const unsigned char *)blob_part(b, idx++) : nullptr;
    for (int f = 0; f < 6; ++f) a.f[f] = (const real *)blob_part(b, b.field_part + f);
    a.w = (const real *)s.a.w;
    for (int f = 0; f < 3; ++f) a.lj[f] = (const real *)A->lj[f];
    for (int f = 0; f < 6; ++f) a.lf[f] = (real *)A->lf[f];
    real **lp = (real **)A->lpart[kind];
    a.lx = lp[0]; a.ly = lp[1]; a.lz = lp[2]; a.lpx = lp[3]; a.lpy = lp[4]; a.lpz = lp[5];
    a.lw = A->lw[kind];
    const PicParams &p = c->p;
    a.qm = (real)(p.charge[kind] / p.mass[kind] * p.dt_half);
    a.charge = (real)p.charge[kind];
    a.dt_d[0] = (real)(p.dt / p.dx); a.dt_d[1] = (real)(p.dt / p.dy); a.dt_d[2] = (real)(p.dt / p.dz);
    a.d_dt[0] = p.dx / p.dt; a.d_dt[1] = p.dy / p.dt; a.d_dt[2] = p.dz / p.dt;
    a.scatter_fields = scatter;
    a.status = c->d_status;
    long long blocks = (a.n + 127) / 128;
    if (c->tile > 0 && b.toff_part[kind] >= 0) {
        // one CTA per tile, then the particles it handed back
        const TileBoxes bx = tile_boxes(c);
        AdjTileGeom tg{};
        tg.T = c->tile;
        for (int d = 0; d < 3; ++d) tg.nt[d] = c->ntile[d];
        tg.nodes = c->node_tiles ? 1 : 0;
        tg.GE = bx.GE; tg.DE = bx.DE;
        tg.gsy = bx.gsy; tg.gsz = bx.gsz; tg.gsize = bx.gsize;
        tg.dsy = bx.dsy; tg.dsz = bx.dsz; tg.dsize = bx.dsize;
        // scratch for 10 (FP64) or 18 (FP32) particles per cell of the default
        // tile, at most 4095 (the limbs): beyond, the tile takes several rounds
        const size_t rs = sizeof(real), nl = adj_limbs<real>();
        const size_t fixed = (6 * (size_t)bx.gsize + 3 * (size_t)bx.dsize) * rs + (6 * nl * bx.gsize + 8) * 4;
        const size_t budget = 227 * 1024;
        tg.cap = fixed + 64 < budget ? (int)std::min<size_t>(rs == 8 ? 640 : 1152, (budget - fixed - 64) / (6 * rs + 1)) : 0;
        const size_t smem = fixed + (size_t)tg.cap * (6 * rs + 1);
        const int ntiles = c->ntile[0] * c->ntile[1] * c->ntile[2];
        cudaMemsetAsync(c->d_nstrag + kind, 0, sizeof(unsigned long long), c->stream);
        prof_begin(c, "adjoint_tile_push_deposit");
        if (tg.cap > 0) {
            const unsigned *toffs = (const unsigned *)blob_part(b, b.toff_part[kind]);
            if (c->tile == 4) {   // the default edge: strides as constants
                cudaFuncSetAttribute(adj_tile_kernel<real, P, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
                adj_tile_kernel<real, P, 4><<<ntiles, kAdjThreads, smem, c->stream>>>(a, tg, toffs, s.strag, c->d_nstrag + kind);
            } else {
                cudaFuncSetAttribute(adj_tile_kernel<real, P, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
                adj_tile_kernel<real, P, 0><<<ntiles, kAdjThreads, smem, c->stream>>>(a, tg, toffs, s.strag, c->d_nstrag + kind);
            }
            a.idx = s.strag;
            a.nidx = c->d_nstrag + kind;
        }
        prof_end(c);
    }
    prof_begin(c, "adjoint_push_deposit");
    adj_push_kernel<real, P><<<(unsigned)std::min<long long>(blocks, 148 * 16), 128, 0, c->stream>>>(a);
    prof_end(c);
}

template <typename real>
static void adj_fields_e(pic_ctx *c, AdjState *A) {
    const Geom &g = c->g;
    real **F = (real **)A->lf;
    real **J = (real **)A->lj;
    prof_begin(c, "adjoint_yee_e");
    adj_update_e_kernel<real><<<(unsigned)((g.fsz + 255) / 256), 256, 0, c->stream>>>(
        g, F[0], F[1], F[2], F[3], F[4], F[5], J[0], J[1], J[2], (real)c->p.dt_half, (real)(1.0 / c->p.dx),
        (real)(1.0 / c->p.dy), (real)(1.0 / c->p.dz));
    prof_end(c);
}

template <typename real>
static void adj_fields_b(pic_ctx *c, AdjState *A) {
    const Geom &g = c->g;
    real **F = (real **)A->lf;
    prof_begin(c, "adjoint_yee_b");
    adj_update_b_kernel<real><<<(unsigned)((g.fsz + 255) / 256), 256, 0, c->stream>>>(
        g, F[0], F[1], F[2], F[3], F[4], F[5], (real)c->p.dt_half, (real)(1.0 / c->p.dx), (real)(1.0 / c->p.dy),
        (real)(1.0 / c->p.dz));
    prof_end(c);
}

template <typename real>
static void adj_bc(pic_ctx *c, AdjState *A, int step) {
    const Geom &g = c->g;
    const PicParams &p = c->p;
    AdjBcArgs B{};
    B.g = g;
    B.dt = p.dt; B.dx = p.dx; B.dy = p.dy; B.dz = p.dz;
    B.Pi = p.Pi; B.omega = p.omega; B.l0 = p.l0; B.amp = p.laser_amplitude; B.dur = p.laser_pulse_duration;
    B.start = p.laser_start_time; B.waist = p.waist; B.xfocus = p.xfocus; B.yfocus = p.yfocus; B.zfocus = p.zfocus;
    B.phase = p.phase; B.time = step * p.dt; B.pol = p.laser_polarization; B.envelope = p.laser_envelope;
    B.profile_n = c->profile_n;
    B.lprof = (p.laser_profile == 1 && c->d_profile) ? A->lprof : nullptr;
    real **F = (real **)A->lf;
    real **J = (real **)A->lj;
    dim3 blk(32, 8), grd((g.n[1] + 31) / 32, (g.n[2] + 7) / 8);
    prof_begin(c, "adjoint_boundary");
    adj_bc_kernel<real><<<grd, blk, 0, c->stream>>>(B, F[0], F[1], F[2], F[3], F[4], F[5], J[1], J[2]);
    prof_end(c);
}

template <typename real>
static int adj_backward_t(pic_ctx *c, AdjState *A, int nsteps) {
    for (int t = 0; t < nsteps; ++t) {
        if (A->tape_len == 0) {
            c->err = "adjoint: tape exhausted";
            return PIC_EINVAL;
        }
        const Blob &b = A->tape[--A->tape_len];
        const int step = b.step;   // 0: the t = 0 push; n >= 1: loop iteration n
        const bool loop = step >= 1;
        if (loop) {
            // second half (field.cpp:88-117): B then E forward, so E then B here
            adj_fields_e<real>(c, A);
            adj_fields_b<real>(c, A);
        }
        // push + deposit of both species, in reverse species order
        int base[2] = {0, 0};
        {
            int idx = 0;
            for (int k = 0; k < 2; ++k) {
                base[k] = idx;
                if (b.count[k] == 0) continue;
                idx += (c->fp32 ? 4 : 3) + 3 + (c->sp[k].dead ? 1 : 0);
            }
        }
        for (int k = 1; k >= 0; --k) {
            if (b.count[k] == 0) continue;
            if (c->order == 2) adj_push_launch<real, 3>(c, A, b, k, base[k], loop);
            else adj_push_launch<real, 5>(c, A, b, k, base[k], loop);
        }
        // the push ran right after a sort: back to the order before it
        for (int k = 0; k < 2; ++k)
            if (b.perm_part[k] >= 0) unsort_species(c, A, k, (const int *)blob_part(b, b.perm_part[k]), b.count[k]);
        // clear_currents: J before the clear does not reach the deposit
        prof_begin(c, "adjoint_clear");
        cudaMemsetAsync(A->lj[0], 0, 3 * (size_t)c->g.rsz * rsize(c), c->stream);
        prof_end(c);
        if (loop) {
            // first half (field.cpp:56-86): E then B forward
            adj_fields_b<real>(c, A);
            adj_fields_e<real>(c, A);
            adj_bc<real>(c, A, step);
        }
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        c->err = std::string("adjoint: ") + cudaGetErrorString(e);
        return PIC_ECUDA;
    }
    return PIC_OK;
}

extern "C" {

int pic_checkpoint_save(pic_ctx *c, int slot) {
    if (!c || slot < 0) return PIC_EINVAL;
    AdjState *A = adj_of(c, true);
    if ((int)A->ckpt.size() <= slot) A->ckpt.resize(slot + 1);
    std::vector<std::pair<void *, size_t>> parts;
    checkpoint_parts(c, parts);
    return blob_save(c, A->ckpt[slot], parts);
}

int pic_checkpoint_restore(pic_ctx *c, int slot) {
    if (!c || slot < 0) return PIC_EINVAL;
    AdjState *A = adj_of(c, false);
    if (!A || slot >= (int)A->ckpt.size() || !A->ckpt[slot].buf) {
        c->err = "no such checkpoint";
        return PIC_EINVAL;
    }
    Blob &b = A->ckpt[slot];
    for (int k = 0; k < 2; ++k) {
        if (c->sp[k].n_host != b.count[k]) {
            c->err = "checkpoint particle count differs from the context's";
            return PIC_EINVAL;
        }
        c->sp[k].cur = b.cur[k];
    }
    // the arrays' current buffers (a sort since the save may have swapped them)
    std::vector<std::pair<void *, size_t>> parts;
    checkpoint_parts(c, parts);
    if (parts.size() != b.parts.size()) {
        c->err = "checkpoint layout differs from the context's";
        return PIC_EINVAL;
    }
    copy_parts(c, b, parts, false);
    for (int k = 0; k < 2; ++k) {
        c->sp[k].sorted = false;   // the next push sorts (and the tape records that permutation)
        c->sp[k].perm_fresh = false;
    }
    c->step = b.step;
    return PIC_OK;
}

int pic_adjoint_tape(pic_ctx *c, int nsteps) {
    if (!c || nsteps < 0) return PIC_EINVAL;
    if (!c->p.adjoint) {
        c->err = "the context was not created with adjoint = 1";
        return PIC_EINVAL;
    }
    AdjState *A = adj_of(c, true);
    if ((int)A->tape.size() < nsteps) A->tape.resize(nsteps);
    A->tape_len = 0;
    if (c->tile > 0) {
        const size_t nt = (size_t)c->ntile[0] * c->ntile[1] * c->ntile[2] + 1;
        for (int k = 0; k < 2; ++k)
            if (!A->toffs[k] && cudaMalloc((void **)&A->toffs[k], nt * sizeof(unsigned)) != cudaSuccess) {
                A->toffs[k] = nullptr;
                c->err = "adjoint: out of device memory for the tile boundaries";
                return PIC_ENOMEM;
            }
    }
    return PIC_OK;
}

int pic_adjoint_record(pic_ctx *c, int on) {
    if (!c) return PIC_EINVAL;
    AdjState *A = adj_of(c, true);
    A->recording = on != 0;
    return PIC_OK;
}

int pic_adjoint_seed_kinetic(pic_ctx *c, int kind, double xlo, double xhi, double ramp, double *loss) {
    if (!c || kind < 0 || kind > 1 || !(ramp >= 0.0) || !(xhi >= xlo) || 2.0 * ramp > xhi - xlo) {
        if (c) c->err = "adjoint: window needs xlo <= xhi and 0 <= 2 ramp <= xhi - xlo";
        return PIC_EINVAL;
    }
    if (!c->p.adjoint) {
        c->err = "the context was not created with adjoint = 1";
        return PIC_EINVAL;
    }
    AdjState *A = adj_of(c, true);
    int r = ensure_adj_arrays(c, A);
    if (r) return r;
    const size_t rs = rsize(c);
    for (int f = 0; f < 6; ++f) cudaMemsetAsync(A->lf[f], 0, (size_t)c->g.fsz * rs, c->stream);
    cudaMemsetAsync(A->lj[0], 0, 3 * (size_t)c->g.rsz * rs, c->stream);
    for (int k = 0; k < 2; ++k) {
        size_t n = (size_t)std::max<int64_t>(c->sp[k].cap, 1);
        for (int q = 0; q < 6; ++q) cudaMemsetAsync(A->lpart[k][q], 0, n * rs, c->stream);
        cudaMemsetAsync(A->lw[k], 0, n * sizeof(double), c->stream);
    }
    cudaMemsetAsync(A->lprof, 0, (size_t)A->nprof * sizeof(double), c->stream);
    cudaMemsetAsync(A->loss, 0, sizeof(double), c->stream);
    Species &s = c->sp[kind];
    long long n = s.n_host;
    if (n > 0) {
        unsigned blocks = (unsigned)((n + 255) / 256);
        if (c->fp32)
            adj_seed_kinetic_kernel<float><<<blocks, 256, 0, c->stream>>>(
                c->g, c->cp, 1, n, nullptr, s.a.cell[s.cur], s.a.ox[s.cur], (float *)s.a.px, (float *)s.a.py,
                (float *)s.a.pz, (float *)s.a.w, s.dead, c->p.mass[kind], xlo, xhi, ramp, (float *)A->lpart[kind][0], (float *)A->lpart[kind][3],
                (float *)A->lpart[kind][4], (float *)A->lpart[kind][5], A->lw[kind], A->loss);
        else
            adj_seed_kinetic_kernel<double><<<blocks, 256, 0, c->stream>>>(
                c->g, c->cp, 0, n, s.a.x[s.cur], nullptr, nullptr, (double *)s.a.px, (double *)s.a.py,
                (double *)s.a.pz, (double *)s.a.w, s.dead, c->p.mass[kind], xlo, xhi, ramp, (double *)A->lpart[kind][0], (double *)A->lpart[kind][3],
                (double *)A->lpart[kind][4], (double *)A->lpart[kind][5], A->lw[kind], A->loss);
    }
    note_adjoint_order(c, A);
    double l = 0.0;
    cudaMemcpyAsync(&l, A->loss, sizeof(double), cudaMemcpyDeviceToHost, c->stream);
    if (cudaStreamSynchronize(c->stream) != cudaSuccess) return PIC_ECUDA;
    if (loss) *loss = l;
    return PIC_OK;
}

int pic_adjoint_backward(pic_ctx *c, int nsteps) {
    if (!c || nsteps < 0) return PIC_EINVAL;
    AdjState *A = adj_of(c, false);
    if (!A || !A->lf[0]) {
        c->err = "adjoint: seed the objective first";
        return PIC_EINVAL;
    }
    remap_adjoints(c, A);
    int r = c->fp32 ? adj_backward_t<float>(c, A, nsteps) : adj_backward_t<double>(c, A, nsteps);
    note_adjoint_order(c, A);
    return r;
}

int pic_adjoint_weight_grad(pic_ctx *c, int kind, double *out, int64_t n) {
    if (!c || kind < 0 || kind > 1 || !out) return PIC_EINVAL;
    AdjState *A = adj_of(c, false);
    if (!A || !A->lw[kind]) return PIC_EINVAL;
    if (n > c->sp[kind].n_host) n = c->sp[kind].n_host;
    const double *src = A->lw[kind];
    Species &s = c->sp[kind];
    if (s.orig && n > 0 && s.n_host > 0) {   // sorted context: back to upload order
        PermuteList l{};
        l.ds[0] = (const unsigned long long *)A->lw[kind];
        l.dd[0] = (unsigned long long *)A->lw_b[kind];
        l.nd = 1;
        permute(c, l, s.orig, s.n_host, false);
        src = A->lw_b[kind];
    }
    cudaMemcpyAsync(out, src, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
    return cudaStreamSynchronize(c->stream) == cudaSuccess ? PIC_OK : PIC_ECUDA;
}

int pic_adjoint_profile_grad(pic_ctx *c, double *out, int n) {
    if (!c || !out) return PIC_EINVAL;
    AdjState *A = adj_of(c, false);
    if (!A || !A->lprof) return PIC_EINVAL;
    n = std::min(n, A->nprof);
    cudaMemcpyAsync(out, A->lprof, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
    return cudaStreamSynchronize(c->stream) == cudaSuccess ? PIC_OK : PIC_ECUDA;
}

int pic_adjoint_release(pic_ctx *c) {
    if (!c) return PIC_EINVAL;
    for (size_t i = 0; i < g_adj.size(); ++i) {
        if (g_adj[i].first != c) continue;
        AdjState *A = g_adj[i].second;
        for (auto &b : A->ckpt)
            if (b.buf) cudaFree(b.buf);
        for (auto &b : A->tape)
            if (b.buf) cudaFree(b.buf);
        for (void *p : A->lf) if (p) cudaFree(p);
        if (A->lj[0]) cudaFree(A->lj[0]);
        for (auto &sp : A->lpart) for (void *p : sp) if (p) cudaFree(p);
        for (double *p : A->lw) if (p) cudaFree(p);
        if (A->lprof) cudaFree(A->lprof);
        if (A->loss) cudaFree(A->loss);
        for (int *p : A->lam_orig) if (p) cudaFree(p);
        for (unsigned *p : A->toffs) if (p) cudaFree(p);
        for (auto &sp : A->lpart_b) for (void *p : sp) if (p) cudaFree(p);
        for (double *p : A->lw_b) if (p) cudaFree(p);
        delete A;
        g_adj.erase(g_adj.begin() + (long)i);
        return PIC_OK;
    }
    return PIC_OK;
}

}  // extern "C"
