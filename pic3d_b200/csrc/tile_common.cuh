// What the tile kernels share: tile geometry, launch arguments, asynchronous
// copies and the fixed-point accumulators' limits.
#pragma once

#include <algorithm>
#include <cmath>

#include "pic_kernels.cuh"
#include "push_core.cuh"

namespace pic {

struct TileGeom {
    int T, nt[3];
    long long nkeys;
    int nodes;               // 1: tiles of nodes, 0: tiles of cells (pic_ctx::node_tiles)
    int GE, DE, nacc;
    // padded shared-memory strides: row gsy/dsy, plane gsz/dsz, array gsize/dsize
    int gsy, gsz, gsize, dsy, dsz, dsize;
};

template <int P>
__host__ __device__ constexpr int gather_extent(int T) { return T + 2 * (P / 2) + 1; }
template <int P>
__host__ __device__ constexpr int deposit_extent(int T) { return T + 2 * (P / 2) + 3; }

// limbs of the shared-memory fixed-point accumulators
template <typename real>
constexpr int limbs() { return sizeof(real) == 8 ? 3 : 2; }
// |value * scale| stays below 2^fixed_bits: with at most kMaxTileParticles
// additions per point the limb sums fit in 32 bits and the reassembled
// total in 64 bits (FixedAcc)
constexpr int kMaxTileParticles = 16383;

// Asynchronous global -> shared copies (cp.async): a CTA issues every copy
// of a batch without waiting on any, then waits once.  src_bytes 0 fills the
// destination with zeros and reads nothing.
template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src, int src_bytes = BYTES) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(src), "n"(BYTES), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// moves element i of n arrays to dst, the loads of eight arrays before their
// stores (the compiler must assume that a store changes the next source)
template <typename T, int N>
__device__ __forceinline__ void move_words(const T *const (&src)[N], T *const (&to)[N], int n, long long i, long long dst) {
#pragma unroll
    for (int k0 = 0; k0 < N; k0 += 8) {
        if (k0 >= n) break;
        T v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (k0 + k < N && k0 + k < n) v[k] = src[k0 + k][i];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (k0 + k < N && k0 + k < n) to[k0 + k][dst] = v[k];
    }
}

// word offset (from the accumulators) of the particle input buffers: after
// the five accumulators, rounded up to 16 bytes
__host__ __device__ constexpr int particle_buffer_offset(int acc_words) { return (acc_words + 3) & ~3; }

template <typename real>
struct TileArgs {
    PushArgs<real> sp[2];
    const unsigned *offs[2];
    int active[2];
    TileGeom t;
    real *ring[5];
    const real *field[6];
    real scale[4];          // jx, jy, jz, rho
    double inv_scale[4];
    int *strag[2];          // (index, home tile) of particles left for the global kernel
    unsigned long long *nstrag;
    // visitor lists of this push (vis_off null: none) and the recording of
    // the next push's (vsink.raw null: off)
    const int *vis[2];
    const uint2 *vis_off[2];
    const VisState *vs[2];
    VisSink vsink[2];
};

// arguments of a tile launch over the species of `mask` (host side)
template <typename real, int P>
inline TileArgs<real> make_tile_args(pic_ctx *c, int mask, const TileGeom &t) {
    TileArgs<real> ta{};
    double qw_max = 0.0;
    for (int k = 0; k < 2; ++k) {
        ta.sp[k] = make_push_args<real>(c, k);
        ta.offs[k] = c->sp[k].offs;
        ta.active[k] = ((mask >> k) & 1) && c->sp[k].n_host > 0;
        if (ta.active[k]) qw_max = std::max(qw_max, std::fabs(c->p.charge[k]) * c->sp[k].max_abs_w);
    }
    ta.t = t;
    for (int k = 0; k < 5; ++k) ta.ring[k] = (real *)c->ring[k];
    for (int k = 0; k < 6; ++k) ta.field[k] = (const real *)c->field[k];
    // one contribution is at most |q w| d/dt (J: the running sum of ds and the
    // Esirkepov weight are both within [-1, 1]) or |q w| smax^3 (rho, smax the
    // largest shape weight: 3/4 at 2nd order, 115/192 at 4th)
    const double dmax = std::max(c->p.dx, std::max(c->p.dy, c->p.dz));
    const double lim = std::ldexp(1.0, fixed_bits<real>());
    const double smax = P == 3 ? 0.75 : 115.0 / 192.0;
    const double bj = 1.01 * qw_max * dmax / c->p.dt, br = 1.01 * qw_max * smax * smax * smax;
    for (int k = 0; k < 4; ++k) {
        double b = k < 3 ? bj : br;
        double s = b > 0.0 ? lim / b : 1.0;
        ta.scale[k] = (real)s;
        ta.inv_scale[k] = 1.0 / (double)ta.scale[k];
    }
    for (int k = 0; k < 2; ++k) {
        Species &s = c->sp[k];
        ta.strag[k] = s.strag;
        ta.vis[k] = s.vis;
        ta.vis_off[k] = s.vis_off;
        ta.vs[k] = s.vs;
        ta.vsink[k] = vis_sink_of(c, s);
    }
    ta.nstrag = c->d_nstrag;
    return ta;
}

}  // namespace pic
