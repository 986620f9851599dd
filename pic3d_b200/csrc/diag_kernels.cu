// FP64 diagnostics: field energy, kinetic energy and charge per species,
// and the largest Gauss-law residual |div E - rho| over physical nodes.
// The reference has no diagnostics; these run in FP64 in both precisions.
#include "pic_kernels.cuh"

namespace pic {

// Everything runs in one launch: blockIdx.y 0 takes the fields, 1 and 2 the
// species.  What bounds it: HBM on large states (32 B per particle in FP64);
// on 64^3 cells the reductions: with one atomic maximum per thread the fields
// took 102 us, with one per block they take their share of about 15 us.
struct DiagArgs {
    Geom g;
    const void *f[6], *rho[2];   // ex .. bz; rho0, rho1
    const void *p[2][4];         // px, py, pz, w per species (null: none)
    const long long *count[2];
    double mass[2], dV, inv[3];
    double *out;
};

constexpr int kDiagThreads = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// the block's sums of v[0 .. N-1], each added to its output
template <int N>
__device__ __forceinline__ void block_add(double (&v)[N], double *const (&out)[N]) {
    __shared__ double part[N][kDiagThreads / 32];
    const int t = threadIdx.y * 32 + threadIdx.x, lane = t & 31, wid = t >> 5;
#pragma unroll
    for (int n = 0; n < N; ++n) {
        v[n] = warp_sum(v[n]);
        if (lane == 0) part[n][wid] = v[n];
    }
    __syncthreads();
    if (t < N) {
        double s = 0.0;
        for (int w = 0; w < kDiagThreads / 32; ++w) s += part[t][w];
        double *o = out[0];
#pragma unroll
        for (int n = 1; n < N; ++n)
            if (t == n) o = out[n];
        atomicAdd(o, s);
    }
}

template <typename real>
__device__ __forceinline__ void field_part(const DiagArgs &a) {
    const Geom &g = a.g;
    const real *ex = (const real *)a.f[0], *ey = (const real *)a.f[1], *ez = (const real *)a.f[2];
    const real *bx = (const real *)a.f[3], *by = (const real *)a.f[4], *bz = (const real *)a.f[5];
    const real *r0 = (const real *)a.rho[0], *r1 = (const real *)a.rho[1];
    double e = 0.0, q0 = 0.0, q1 = 0.0, gmax = 0.0;
    const unsigned rows = (unsigned)g.n[1] * (unsigned)g.n[2];
    for (unsigned row = blockIdx.x * blockDim.y + threadIdx.y; row < rows; row += gridDim.x * blockDim.y) {
        const int k = (int)(row / (unsigned)g.n[1]), j = (int)(row - (unsigned)k * (unsigned)g.n[1]);
        for (int i = threadIdx.x; i < g.n[0]; i += 32) {
            const int c = g.fi(k + g.mem, j + g.mem, i + g.mem), rc = g.ri(k + g.mem, j + g.mem, i + g.mem);
            const double x = ex[c], y = ey[c], z = ez[c], u = bx[c], v = by[c], w = bz[c];
            e += x * x + y * y + z * z + u * u + v * v + w * w;
            const double rho0 = r0 ? (double)r0[rc] : 0.0, rho1 = r1 ? (double)r1[rc] : 0.0;
            q0 += rho0;
            q1 += rho1;
            const double div = (x - (double)ex[c - 1]) * a.inv[0] + (y - (double)ey[c - g.f[0]]) * a.inv[1] +
                               (z - (double)ez[c - g.fxy]) * a.inv[2];
            const double res = fabs(div - rho0 - rho1);
            gmax = (res != res || res > gmax) ? res : gmax;   // a NaN residual wins and stays
        }
    }
    // max of non-negative doubles through their ordered bit patterns (a
    // positive NaN orders above every finite value and +inf)
    unsigned long long m = (unsigned long long)__double_as_longlong(gmax);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long v = __shfl_xor_sync(0xffffffffu, m, o);
        m = v > m ? v : m;
    }
    __shared__ unsigned long long mpart[kDiagThreads / 32];
    if (threadIdx.x == 0) mpart[threadIdx.y] = m;
    double v[3] = {0.5 * e * a.dV, q0 * a.dV, q1 * a.dV};
    double *const out[3] = {a.out, a.out + 3, a.out + 4};
    block_add(v, out);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        for (int w = 1; w < kDiagThreads / 32; ++w) m = mpart[w] > m ? mpart[w] : m;
        atomicMax((unsigned long long *)(a.out + 5), m);
    }
}

template <typename real>
__global__ void __launch_bounds__(kDiagThreads) diag_kernel(const __grid_constant__ DiagArgs a) {
    if (blockIdx.y == 0) {
        field_part<real>(a);
        return;
    }
    const int k = (int)blockIdx.y - 1;
    const real *px = (const real *)a.p[k][0], *py = (const real *)a.p[k][1], *pz = (const real *)a.p[k][2],
               *w = (const real *)a.p[k][3];
    if (!px) return;
    const long long n = *a.count[k], nt = (long long)gridDim.x * kDiagThreads;
    const double mass = a.mass[k];
    double s[1] = {0.0};
    for (long long i = (long long)blockIdx.x * kDiagThreads + threadIdx.y * 32 + threadIdx.x; i < n; i += nt) {
        const double x = px[i], y = py[i], z = pz[i];
        const double u2 = x * x + y * y + z * z;
        // gamma - 1 without cancellation
        s[0] += (double)w[i] * mass * (u2 / (sqrt(1.0 + u2) + 1.0));
    }
    double *const out[1] = {a.out + 1 + k};
    block_add(s, out);
}

void launch_diagnostics(pic_ctx *c, double *d_out) {
    const PicParams &p = c->p;
    DiagArgs a{};
    a.g = c->g;
    for (int f = 0; f < 6; ++f) a.f[f] = c->field[f];
    for (int k = 0; k < 2; ++k) {
        a.rho[k] = c->ring[3 + k];
        const Species &s = c->sp[k];
        if (!s.a.px || s.n_host == 0) continue;
        const void *q[4] = {s.a.px, s.a.py, s.a.pz, s.a.w};
        for (int n = 0; n < 4; ++n) a.p[k][n] = q[n];
        a.count[k] = s.d_count;
        a.mass[k] = p.mass[k];
    }
    a.dV = p.dx * p.dy * p.dz;
    a.inv[0] = 1.0 / p.dx;
    a.inv[1] = 1.0 / p.dy;
    a.inv[2] = 1.0 / p.dz;
    a.out = d_out;
    cudaMemsetAsync(d_out, 0, PIC_NDIAG * sizeof(double), c->stream);
    const dim3 grid(148 * 4, 3), blk(32, kDiagThreads / 32);
    if (c->fp32) diag_kernel<float><<<grid, blk, 0, c->stream>>>(a);
    else diag_kernel<double><<<grid, blk, 0, c->stream>>>(a);
}

}  // namespace pic
