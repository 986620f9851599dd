// The sort and the visitor lists of every tiled context, and the tiled gather +
// push + deposit over tiles of cells: tile edges other than the default one,
// which has tiles of nodes (tile_node_kernels.cu, tile_mma_kernels.cu).
//
// Particles of each species are kept in counting-sort order by tile (T^3
// cells), then by half-cell octant of the position (which side of the cell
// centre on each axis: it fixes the primal stencil index relative to the
// cell), then by cell.  One CTA owns one tile:
//   1. it stages the six field components of the tile plus the gather halo
//      (T + 2H + 1 points per axis) in shared memory,
//   2. clears shared-memory accumulators for jx, jy, jz, rho0, rho1 over the
//      deposit footprint (T + 2H + 3 points per axis),
//   3. pushes the tile's particles, both species, gathering from and
//      depositing into shared memory: those whose sort key fell in it and that
//      are still in it, and its visitor list, which names those that have come
//      into it since the sort (without valid lists a particle away from home is
//      left to the global kernel, which runs after this one),
//   4. flushes the accumulators with one coalesced pass of global atomics
//      (zero entries skipped); halos of neighbouring tiles overlap, hence the
//      atomics.
// A warp takes 32 consecutive particles of the sorted list: mostly one
// octant and consecutive cells, so at a common stencil point their
// shared-memory addresses fall in different banks.
//
// The counting sort (key histogram, exclusive scan, scatter into the second
// set of arrays) runs every `sort_interval` pushes and after an upload; one
// set of launches sorts both species.
#include "tile_common.cuh"

namespace pic {

// Row and plane strides of a shared-memory box of extent e for tile edge T.
// Lanes of a warp take 32 consecutive cells of the tile (cell index
// x + T*y + T*T*z); with row stride = T (mod 2T) and plane stride = T*T
// (mod 2T*T) those 32 cells start in 32 different banks, so a warp's loads
// and atomics at a common stencil offset are conflict-free (2 wavefronts
// per 8-byte access, the minimum).
static inline void padded_strides(int e, int T, int &sy, int &sz) {
    sy = padded_row(e, T);
    sz = padded_plane(e, T);
}

// Sort key of a particle.  Tiles of cells: tile, then half-cell octant `oct`
// (bit d set: the particle's node is its cell's plus one along d), then cell
// within the tile; `at` is the cell.  Tiles of nodes: tile, then node within
// the tile, x fastest, so that consecutive particles share the y and z of
// their stencils; `at` is the node.
__device__ __forceinline__ int tile_key(const TileGeom &t, const int (&at)[3], int oct) {
    const int T = t.T;
    int q[3], l[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        q[d] = at[d] / T;
        l[d] = at[d] - q[d] * T;
    }
    const int tile = (q[2] * t.nt[1] + q[1]) * t.nt[0] + q[0];
    return ((t.nodes ? tile : tile * kOctants + oct) * T + l[2]) * T * T + l[1] * T + l[0];
}

// Sort key of particle i: cell and node as the next push will decode them,
// clamped to cells 0 .. n - 1, or nodes 0 .. n.
__device__ __forceinline__ int particle_key(const Geom &g, const TileGeom &t, const CellPack &cp, int fp32,
                                            const double *x, const double *y, const double *z, const int *cell,
                                            const float *ox, const float *oy, const float *oz, long long i) {
    int c[3], nd[3];
    if (fp32) {
        cp.unpack(cell[i], c[0], c[1], c[2]);
        const float o[3] = {ox[i], oy[i], oz[i]};
#pragma unroll
        for (int d = 0; d < 3; ++d) nd[d] = c[d] + (o[d] >= 0.5f ? 1 : 0);
    } else {
        const double v[3] = {x[i], y[i], z[i]};
#pragma unroll
        for (int d = 0; d < 3; ++d) bin_of(g, d, v[d], c[d], nd[d]);
    }
    int oct = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        oct |= (nd[d] > c[d] ? 1 : 0) << d;
        c[d] = t.nodes ? min(max(nd[d], 0), g.n[d]) : min(max(c[d], 0), g.n[d] - 1);
    }
    return tile_key(t, c, oct);
}

// ---------------------------------------------------------------------------
// counting sort.  One launch of each kernel serves up to two species
// (blockIdx.y): a 32^3 step is bound by launches and the gaps between them,
// about 2.3 us each.

constexpr int kSortKeysPerBlock = 4096;   // of the scan, 4 per thread

struct SortArgs {
    Geom g;
    TileGeom t;
    CellPack cp;
    int fp32;
    unsigned *done;              // blocks of the scan that have finished, per species (zero between sorts)
    int ntiles;
    struct One {
        const long long *count;
        const double *x, *y, *z;
        const int *cell;
        const float *ox, *oy, *oz;
        int *keys;
        unsigned *hist, *sums, *offs;
        // visitor lists (null: none) and the straggler count, reset here
        VisState *vs;
        int par;
        uint2 *vis_off;
        unsigned *vis_cnt;
        unsigned long long *nstrag;
    } s[2];
};

__global__ void sort_keys_kernel(const __grid_constant__ SortArgs sa) {
    const SortArgs::One &a = sa.s[blockIdx.y];
    long long n = *a.count;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned act = __ballot_sync(0xffffffffu, i < n);
    if (i >= n) return;
    int key = particle_key(sa.g, sa.t, sa.cp, sa.fp32, a.x, a.y, a.z, a.cell, a.ox, a.oy, a.oz, i);
    a.keys[i] = key;
    unsigned peers = __match_any_sync(act, key);
    int lane = threadIdx.x & 31;
    if (lane == __ffs(peers) - 1) atomicAdd(&a.hist[key], (unsigned)__popc(peers));
}

// exclusive sum over the block (1024 threads) of one value per thread;
// `total` gets the block's sum
__device__ __forceinline__ unsigned block_exclusive(unsigned s, unsigned &total) {
    __shared__ unsigned warp_tot[33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        const unsigned t = lane < nw ? warp_tot[lane] : 0u;
        unsigned ti = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, ti, o);
            if (lane >= o) ti += u;
        }
        if (lane < nw) warp_tot[lane] = ti - t;
        if (lane == nw - 1) warp_tot[32] = ti;
    }
    __syncthreads();
    const unsigned excl = warp_tot[w] + incl - s;
    total = warp_tot[32];
    __syncthreads();
    return excl;
}

// Sums of the histogram's blocks of kSortKeysPerBlock keys; the last block to
// finish turns them into exclusive offsets (sums[nb]: the total), so that the
// scan takes two launches.  The visitor lists and the straggler count are
// emptied.  After the sort every particle is at home, except one whose cell was
// clamped into the grid (x = n on a periodic axis where tiles hold cells, a
// position outside the domain): no list names it, so the lists do not count
// as valid for the push that follows and it goes to the global kernel.
__global__ void __launch_bounds__(1024) sort_sums_kernel(const __grid_constant__ SortArgs sa, int nb) {
    const SortArgs::One &a = sa.s[blockIdx.y];
    __shared__ bool last;
    const long long base = (long long)blockIdx.x * kSortKeysPerBlock + (long long)threadIdx.x * 4;
    unsigned s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) s += base + k < sa.t.nkeys ? a.hist[base + k] : 0u;
    unsigned total;
    block_exclusive(s, total);
    if (threadIdx.x == 0) {
        a.sums[blockIdx.x] = total;
        __threadfence();
        last = atomicAdd(sa.done + blockIdx.y, 1u) == gridDim.x - 1;
    }
    if (a.vs) {
        for (int q = blockIdx.x * 1024 + threadIdx.x; q < sa.ntiles; q += gridDim.x * 1024) {
            a.vis_off[q] = make_uint2(0u, 0u);
            a.vis_cnt[q] = 0u;
        }
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    unsigned carry = 0;
    for (int off = 0; off < nb; off += 1024) {
        const int i = off + threadIdx.x;
        const unsigned v = i < nb ? __ldcg(a.sums + i) : 0u;
        const unsigned e = block_exclusive(v, total);
        if (i < nb) a.sums[i] = carry + e;
        carry += total;
    }
    if (threadIdx.x == 0) {
        a.sums[nb] = carry;
        sa.done[blockIdx.y] = 0u;
        *a.nstrag = 0ull;
        if (a.vs) {
            a.vs->nraw[a.par] = 0ull;
            a.vs->valid_next[a.par] = 1u;
            a.vs->valid_cur = 0u;   // a home particle found away from its tile: the global kernel
            a.vs->total = 0u;
            a.vs->nvis = 0ull;
        }
    }
}

__global__ void __launch_bounds__(1024) sort_offsets_kernel(const __grid_constant__ SortArgs sa, int nb) {
    const SortArgs::One &a = sa.s[blockIdx.y];
    const long long base = (long long)blockIdx.x * kSortKeysPerBlock + (long long)threadIdx.x * 4;
    unsigned loc[4], s = 0, total;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        loc[k] = base + k < sa.t.nkeys ? a.hist[base + k] : 0u;
        s += loc[k];
    }
    unsigned run = block_exclusive(s, total) + a.sums[blockIdx.x];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (base + k < sa.t.nkeys) a.offs[base + k] = run;
        run += loc[k];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.offs[sa.t.nkeys] = a.sums[nb];
}

struct ScatterArgs {
    unsigned *status;
    struct One {
        const long long *count;
        long long cap;
        const int *keys;
        const unsigned *offs;
        unsigned *hist;            // counted down to zero: the next sort's histogram
        // arrays moved src -> dst: at most 13 of 8 bytes (two position buffers,
        // momenta, weight, spins) and 17 of 4 (the same in FP32, id, upload index)
        const double *ds[13];
        double *dd[13];
        int nd;
        const unsigned *fs[17];
        unsigned *fd[17];
        int nf;
        const unsigned char *bs;   // one byte array (adjoint mode: dead flags), or null
        unsigned char *bd;
        int *perm;                 // adjoint mode: perm[dst] = src, the gather form of this sort
    } s[2];
};

__global__ void __launch_bounds__(256) scatter_kernel(const __grid_constant__ ScatterArgs sa) {
    const ScatterArgs::One &a = sa.s[blockIdx.y];
    long long n = *a.count;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned act = __ballot_sync(0xffffffffu, i < n);
    if (i >= n) return;
    int key = a.keys[i];
    unsigned peers = __match_any_sync(act, key);
    int lane = threadIdx.x & 31;
    int leader = __ffs(peers) - 1;
    unsigned base = 0;
    if (lane == leader) {
        const unsigned k = (unsigned)__popc(peers);
        base = a.offs[key] + atomicSub(&a.hist[key], k) - k;
    }
    base = __shfl_sync(peers, base, leader);
    unsigned dst = base + __popc(peers & ((1u << lane) - 1u));
    if ((long long)dst >= a.cap) {  // cannot happen with a consistent histogram; never write past the arrays
        atomicOr(sa.status, ST_OVERFLOW);
        return;
    }
    move_words(a.ds, a.dd, a.nd, i, (long long)dst);
    move_words(a.fs, a.fd, a.nf, i, (long long)dst);
    if (a.bs) a.bd[dst] = a.bs[i];
    if (a.perm) a.perm[dst] = (int)i;
}

// ---------------------------------------------------------------------------
// visitor lists: a counting sort by tile of the (index, home, tile) entries
// the last push recorded (and counted under their tiles), in two launches:
// each tile is given a range of the list, in no particular order of the
// tiles, then the entries are scattered.

// The lists are used however few particles are away from home (FP64 pushes
// used them from 3 % on, when a tile's few visitors added a partial round to a
// CTA that took the species one after the other).  Now, with 1.4 % away on the
// thermal plasma, ms per step of the tile kernel and the global kernel for the
// rest, lists against no lists: FP64 2nd order, 256 x 128 x 128 cells 10.52 +
// 0.00 against 10.34 + 0.50; 4th order, 128 x 64 x 64 cells 4.26 against 4.01 +
// 0.25; laser run 1.57 against 1.56 + 0.06.
struct VisArgs {
    int ntiles;
    struct One {
        const int *raw;
        int *vis;
        uint2 *off;
        unsigned *cnt;
        VisState *vs;
        int par;                 // the counter the last push recorded under
        long long cap;
        unsigned long long *nstrag;
    } s[2];
};

// The lists become the ones the coming push reads; it records under the
// other counter.
__global__ void __launch_bounds__(1024) vis_ranges_kernel(const __grid_constant__ VisArgs va) {
    const VisArgs::One &a = va.s[blockIdx.y];
    __shared__ unsigned first;
    const int base = (int)(blockIdx.x * 4096 + threadIdx.x * 4);
    unsigned loc[4], s = 0, total;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        loc[k] = base + k < va.ntiles ? a.cnt[base + k] : 0u;
        s += loc[k];
    }
    unsigned run = block_exclusive(s, total);
    if (threadIdx.x == 0) first = atomicAdd(&a.vs->total, total);
    __syncthreads();
    run += first;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (base + k < va.ntiles) a.off[base + k] = make_uint2(run, run + loc[k]);
        run += loc[k];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        VisState &v = *a.vs;
        v.nvis = min((long long)v.nraw[a.par], a.cap);
        v.valid_cur = v.valid_next[a.par];
        v.nraw[a.par ^ 1] = 0ull;
        v.valid_next[a.par ^ 1] = 1u;
        *a.nstrag = 0ull;
    }
}

// entries with tile -1 were dropped by the removal compaction
__global__ void __launch_bounds__(256) vis_scatter_kernel(const __grid_constant__ VisArgs va) {
    const VisArgs::One &a = va.s[blockIdx.y];
    const long long n = min((long long)a.vs->nraw[a.par], a.cap);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int p = a.raw[3 * i], home = a.raw[3 * i + 1], t = a.raw[3 * i + 2];
        if (t < 0) continue;
        const unsigned slot = a.off[t].x + atomicSub(a.cnt + t, 1u) - 1u;
        reinterpret_cast<int2 *>(a.vis)[slot] = make_int2(p, home);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.vs->total = 0u;
}

static void launch_vis_build(pic_ctx *c, int mask) {
    VisArgs va{};
    va.ntiles = c->ntile[0] * c->ntile[1] * c->ntile[2];
    unsigned ns = 0;
    long long n = 0;
    for (int k = 0; k < 2; ++k) {
        if (!((mask >> k) & 1)) continue;
        Species &s = c->sp[k];
        va.s[ns++] = VisArgs::One{s.vraw, s.vis, s.vis_off, s.vis_cnt, s.vs, s.vis_par, s.vcap, c->d_nstrag + k};
        s.vis_par ^= 1;
        s.strag_zero = true;
        n = std::max<long long>(n, s.vcap);
    }
    vis_ranges_kernel<<<dim3((unsigned)((va.ntiles + 4095) / 4096), ns), 1024, 0, c->stream>>>(va);
    const unsigned grid = (unsigned)std::min<long long>((n + 255) / 256, 148 * 4);
    vis_scatter_kernel<<<dim3(grid, ns), 256, 0, c->stream>>>(va);
}

static TileGeom tile_geom(const pic_ctx *c) {
    TileGeom t{};
    t.T = c->tile;
    for (int d = 0; d < 3; ++d) t.nt[d] = c->ntile[d];
    t.nkeys = c->nkeys;
    t.nodes = c->node_tiles ? 1 : 0;
    return t;
}

int sort_slots(long long nkeys) { return nkeys <= (1ll << 24) ? 2 : 1; }
size_t sort_hist_bytes(const pic_ctx *c) { return (size_t)c->sort_slots * c->nkeys * sizeof(unsigned); }
static int scan_blocks(const pic_ctx *c) { return (int)((c->nkeys + kSortKeysPerBlock - 1) / kSortKeysPerBlock); }
size_t sort_sums_bytes(const pic_ctx *c) {
    return ((size_t)c->sort_slots * (scan_blocks(c) + 1) + 2) * sizeof(unsigned);
}

// the species of `mask` (all with particles), in one set of launches
static void sort_together(pic_ctx *c, int mask) {
    const int sb = scan_blocks(c);
    SortArgs a{};
    ScatterArgs sa{};
    a.g = c->g;
    a.t = tile_geom(c);
    a.cp = c->cp;
    a.fp32 = c->fp32;
    a.ntiles = c->ntile[0] * c->ntile[1] * c->ntile[2];
    a.done = c->d_blocksums + (size_t)c->sort_slots * (sb + 1);
    sa.status = c->d_status;
    unsigned ns = 0;
    long long nmax = 0;
    for (int kind = 0; kind < 2; ++kind) {
        if (!((mask >> kind) & 1)) continue;
        Species &s = c->sp[kind];
        SortArgs::One &o = a.s[ns];
        o.count = s.d_count;
        o.x = s.a.x[s.cur]; o.y = s.a.y[s.cur]; o.z = s.a.z[s.cur];
        o.cell = s.a.cell[s.cur];
        o.ox = s.a.ox[s.cur]; o.oy = s.a.oy[s.cur]; o.oz = s.a.oz[s.cur];
        o.keys = s.keys;
        o.hist = c->d_hist + (size_t)ns * c->nkeys;
        o.sums = c->d_blocksums + (size_t)ns * (sb + 1);
        o.offs = s.offs;
        o.vs = s.vs;
        o.par = s.vis_par;
        o.vis_off = s.vis_off;
        o.vis_cnt = s.vis_cnt;
        o.nstrag = c->d_nstrag + kind;
        ScatterArgs::One &m = sa.s[ns++];
        m.count = s.d_count;
        m.cap = s.cap;
        m.keys = s.keys;
        m.offs = s.offs;
        m.hist = o.hist;
        auto word = [&](const void *src, void *dst) {
            m.fs[m.nf] = (const unsigned *)src;
            m.fd[m.nf++] = (unsigned *)dst;
        };
        auto dbl = [&](const void *src, void *dst) {
            m.ds[m.nd] = (const double *)src;
            m.dd[m.nd++] = (double *)dst;
        };
        // The sort runs right before a push, which overwrites the previous-position
        // buffer: only the current one moves (the adjoint's tape keeps both).
        for (int b = 0; b < 2; ++b) {
            if (b != s.cur && !c->p.adjoint) continue;
            if (c->fp32) {
                word(s.a.ox[b], s.b.ox[b]);
                word(s.a.oy[b], s.b.oy[b]);
                word(s.a.oz[b], s.b.oz[b]);
                word(s.a.cell[b], s.b.cell[b]);
            } else {
                dbl(s.a.x[b], s.b.x[b]);
                dbl(s.a.y[b], s.b.y[b]);
                dbl(s.a.z[b], s.b.z[b]);
            }
        }
        void *src[7] = {s.a.px, s.a.py, s.a.pz, s.a.w, s.a.sx, s.a.sy, s.a.sz};
        void *dst[7] = {s.b.px, s.b.py, s.b.pz, s.b.w, s.b.sx, s.b.sy, s.b.sz};
        for (int k = 0; k < 7; ++k) {
            if (!src[k]) continue;
            if (c->fp32) word(src[k], dst[k]);
            else dbl(src[k], dst[k]);
        }
        word(s.a.id, s.b.id);
        if (s.orig) {   // adjoint mode: upload index, dead flags, and the permutation for the tape
            word(s.orig, s.orig_b);
            m.bs = s.dead;
            m.bd = s.dead_b;
            m.perm = s.perm;
        }
        nmax = std::max<long long>(nmax, s.n_host);
    }
    const unsigned nb = (unsigned)((nmax + 255) / 256);
    sort_keys_kernel<<<dim3(nb, ns), 256, 0, c->stream>>>(a);
    sort_sums_kernel<<<dim3((unsigned)sb, ns), 1024, 0, c->stream>>>(a, sb);
    sort_offsets_kernel<<<dim3((unsigned)sb, ns), 1024, 0, c->stream>>>(a, sb);
    scatter_kernel<<<dim3(nb, ns), 256, 0, c->stream>>>(sa);
    for (int kind = 0; kind < 2; ++kind) {
        if (!((mask >> kind) & 1)) continue;
        Species &s = c->sp[kind];
        std::swap(s.a, s.b);
        if (s.orig) {
            std::swap(s.orig, s.orig_b);
            std::swap(s.dead, s.dead_b);
            s.perm_fresh = true;
        }
        s.sorted = true;
        s.pushes_since_sort = 0;
        s.vis_built_for = 0;
        s.strag_zero = true;
    }
}

// the species of `mask` whose sort is due before their next push
static int sorts_due(const pic_ctx *c, int mask) {
    int due = 0;
    for (int k = 0; k < 2; ++k) {
        const Species &s = c->sp[k];
        if (((mask >> k) & 1) && s.n_host > 0 && (!s.sorted || s.pushes_since_sort >= c->sort_interval)) due |= 1 << k;
    }
    return due;
}

void launch_sort_due(pic_ctx *c, int mask) {
    if (c->tile <= 0) return;
    const int due = sorts_due(c, mask);
    if (!due) return;
    prof_begin(c, "sort_particles");
    if (c->sort_slots == 2) {
        sort_together(c, due);
    } else {
        for (int k = 0; k < 2; ++k)
            if ((due >> k) & 1) sort_together(c, 1 << k);
    }
    prof_end(c);
}

// Before a push: a full sort when due, else this push's visitor lists from
// what the last push recorded (once per push: pushes_since_sort counts them).
static void prepare_push(pic_ctx *c, int mask) {
    if (c->tile <= 0) return;
    launch_sort_due(c, mask);
    int build = 0;
    for (int k = 0; k < 2; ++k) {
        Species &s = c->sp[k];
        if (!((mask >> k) & 1) || s.n_host <= 0) continue;
        if (s.vs && s.vis_built_for != s.pushes_since_sort) build |= 1 << k;
        s.vis_built_for = s.pushes_since_sort;
    }
    if (build) {
        prof_begin(c, "visitor_lists");
        launch_vis_build(c, build);
        prof_end(c);
    }
    for (int k = 0; k < 2; ++k) {
        Species &s = c->sp[k];
        if (!((mask >> k) & 1) || s.n_host <= 0) continue;
        if (!s.strag_zero) cudaMemsetAsync(c->d_nstrag + k, 0, sizeof(unsigned long long), c->stream);
        s.strag_zero = false;
    }
}

// ---------------------------------------------------------------------------
// the tile kernel

// (The figures here were taken at the default edge, when it had tiles of
// cells.)  Threads per CTA of an ordinary step (the kernel's launch bounds ask for
// two CTAs per SM at 256 threads, one at 512: 128 registers either way).
// Two CTAs of 256 threads (128 registers) where the shared memory of two
// fits: FP32 (measured 1.46x faster at 4th order than one CTA with more
// registers) and FP64 at 2nd order (107 KB per CTA on a step without rho;
// 15.6 vs 19.4 ms per launch on the 256x128x128 thermal plasma against one
// CTA of 512), while one CTA of the other overlaps its staging and flush.
// FP64 at 4th order (160 KB) allows one CTA per SM: 512 threads at 128
// registers (a few spills) measured 12 % faster on the laser workload than
// 256 at 237 registers, while 384 lost (a tile's 512 particles per species
// then leave a third of the second round idle).  Three FP32 CTAs per SM at
// 2nd order measured slower than two.
template <typename real, int P>
constexpr int tile_threads() { return sizeof(real) == 4 || P == 3 ? 256 : 512; }

// NT: threads per CTA of this instantiation (512: one CTA per SM)
template <typename real, int P, bool SPIN, int NT>
__global__ void __launch_bounds__(NT, (NT >= 512 ? 1 : 2)) tile_push_kernel(TileArgs<real> ta) {
    constexpr int H = P / 2;
    constexpr int NL = limbs<real>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    real *sf = reinterpret_cast<real *>(smem_raw);
    const Geom &g = ta.sp[0].g;
    const int T = ta.t.T;
    const int GE = gather_extent<P>(T), DE = deposit_extent<P>(T);
    const int gsy = ta.t.gsy, gsz = ta.t.gsz, GS = ta.t.gsize, dsy = ta.t.dsy, dsz = ta.t.dsz, DS = ta.t.dsize;
    const int G2 = GE * GE, G3 = G2 * GE, D2 = DE * DE, D3 = D2 * DE;
    unsigned *sa = reinterpret_cast<unsigned *>(sf + 6 * GS);   // [component][limb][DS]
    // per warp, two slots of one batch of particle inputs, [word][lane],
    // and the (index, home tile) of each lane's particle per slot
    using PWord = typename PartIn<real>::word;
    constexpr int KW = PartIn<real>::kWords;
    PWord *sp_in = reinterpret_cast<PWord *>(sa + particle_buffer_offset(ta.t.nacc * NL * DS)) + (threadIdx.x >> 5) * 2 * KW * 32;
    int2 *sp_loc = reinterpret_cast<int2 *>(reinterpret_cast<PWord *>(sa + particle_buffer_offset(ta.t.nacc * NL * DS)) +
                                            (blockDim.x >> 5) * 2 * KW * 32) + (threadIdx.x >> 5) * 2 * 32;
    const int nacc = ta.t.nacc;
    const int tile = blockIdx.x;
    const int tx = tile % ta.t.nt[0], ty = (tile / ta.t.nt[0]) % ta.t.nt[1], tz = tile / (ta.t.nt[0] * ta.t.nt[1]);
    const int t0[3] = {tx * T, ty * T, tz * T};
    int gO[3], dO[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        gO[d] = t0[d] + g.mem - 1 - H;   // field buffer coordinate of the first staged point
        dO[d] = t0[d] + g.mem - 2 - H;   // buffer coordinate of the first accumulator point
    }
    // particle ranges of this tile: its slice of the sorted arrays (home
    // particles) and its visitor list
    const long long T3 = (long long)T * T * T * kOctants;   // keys per tile
    long long pa[2] = {0, 0}, pb[2] = {0, 0}, va[2] = {0, 0}, vb[2] = {0, 0};
    bool vvalid[2] = {false, false};
    long long mtot = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (!ta.active[k]) continue;
        const long long n = *ta.sp[k].count;
        pa[k] = ta.offs[k][tile * T3];
        pb[k] = ta.offs[k][(tile + 1) * T3];
        pb[k] = pb[k] < n ? pb[k] : n;
        if (pa[k] > pb[k]) pa[k] = pb[k];
        vvalid[k] = ta.vs[k] && ta.vs[k]->valid_cur;
        if (vvalid[k] && ta.vis_off[k]) {
            const uint2 r = ta.vis_off[k][tile];
            va[k] = r.x;
            vb[k] = r.y;
        }
        mtot += pb[k] - pa[k] + vb[k] - va[k];
    }
    if (mtot == 0) return;
    const bool use_smem = mtot <= kMaxTileParticles;
    // 1. stage fields (asynchronous copies; points outside the buffers read
    // as zero), 2. clear accumulators
    if (use_smem) {
        for (int e = threadIdx.x; e < 6 * G3; e += blockDim.x) {
            int c = e / G3, l = e - c * G3;
            int lz = l / G2, r = l - lz * G2, ly = r / GE, lx = r - ly * GE;
            int x = gO[0] + lx, y = gO[1] + ly, z = gO[2] + lz;
            const bool in = x >= 0 && x < g.f[0] && y >= 0 && y < g.f[1] && z >= 0 && z < g.f[2];
            cp_async<sizeof(real)>(sf + c * GS + lz * gsz + ly * gsy + lx,
                                   ta.field[c] + (in ? g.fi(z, y, x) : 0), in ? (int)sizeof(real) : 0);
        }
        cp_async_commit();
        for (int e = threadIdx.x; e < nacc * NL * DS; e += blockDim.x) sa[e] = 0u;
    }
    cp_async_wait_all();
    __syncthreads();

    View<const real> fs[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) fs[c] = View<const real>{sf + c * GS, gsy, gsz, -(gO[2] * gsz + gO[1] * gsy + gO[0])};
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    // a warp takes 32 consecutive particles of the tile's list: mostly one
    // octant, so the lanes' primal stencils sit at the same offset from
    // their cells and their shared-memory accesses at a common stencil point
    // fall in different banks (the padded strides)
    const int lo_id[3] = {t0[0] + g.mem - 1, t0[1] + g.mem - 1, t0[2] + g.mem - 1};

    // 3. particles of both species
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
        const long long mh = pb[k] - pa[k];         // home particles, then visitors
        const long long m = mh + vb[k] - va[k];
        if (m <= 0) continue;
        const PushArgs<real> &a = ta.sp[k];
        FixedAcc<real, NL> af;
#pragma unroll
        for (int c = 0; c < 3; ++c) af.p[c] = sa + c * NL * DS;
        af.p[3] = (a.rho && nacc == 5) ? sa + (3 + k) * NL * DS : nullptr;
        af.lstride = DS;
        af.sy = dsy;
        af.sz = dsz;
        af.o = -(dO[2] * dsz + dO[1] * dsy + dO[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) af.scale[c] = ta.scale[c];
        // The particle of list position i: a home particle, or an entry of
        // the visitor list.  Its inputs are copied asynchronously into slot
        // `slot` of this warp's buffer one batch ahead of its push.
        const long long pak = pa[k];
        const int2 *visk = reinterpret_cast<const int2 *>(ta.vis[k]) + va[k];
        auto prefetch = [&](long long i, int slot) {
            if (i >= m) return;
            int2 e = make_int2((int)(pak + i), tile);
            if (i >= mh) e = visk[i - mh];
            sp_loc[slot * 32 + lane] = e;
            PWord *dst = sp_in + slot * KW * 32 + lane;
#pragma unroll
            for (int w = 0; w < KW; ++w) cp_async<sizeof(PWord)>(dst + w * 32, particle_word_src(a, (long long)e.x, w));
        };
        long long idx = (long long)warp * 32 + lane;
        int slot = 0;
        prefetch(idx, 0);
        cp_async_commit();
#pragma unroll 1
        for (long long base = (long long)warp * 32; base < m; base += (long long)nwarp * 32) {
            cp_async_wait_all();
            const int2 loc = sp_loc[slot * 32 + lane];
            const long long p = loc.x;
            const int home = loc.y;
            const bool dead = idx < m && a.dead && a.dead[p];   // adjoint mode: removed particles stay, dead
            // the next batch into the other slot
            prefetch(idx + (long long)nwarp * 32, slot ^ 1);
            cp_async_commit();
            const PWord *row = sp_in + slot * KW * 32 + lane;
            if (idx < m && !dead) {
                PartIn<real> in;
#pragma unroll
                for (int w = 0; w < PartIn<real>::kPos; ++w) in.v[w] = row[w * 32];
                OldPos<real> o;
                decode_old(a, p, in, o);
                bool inside = true;
#pragma unroll
                for (int d = 0; d < 3; ++d) inside = inside && o.id[d] >= lo_id[d] && o.id[d] < lo_id[d] + T;
                if (!in_buffers(g, o, H)) {
                    set_status(a.status, ST_OOB);
                } else if (inside && use_smem) {
                    constexpr int mo = PartIn<real>::kPos;   // momenta, then weight
                    const real *pr = reinterpret_cast<const real *>(sp_in + slot * KW * 32);
                    const PmSrc<real> pm{pr + mo * 32, pr + (mo + 1) * 32, pr + (mo + 2) * 32, pr + (mo + 3) * 32, lane};
                    push_body<real, P, SPIN, false>(a, p, o, pm, fs, af, [&](const int (&cn)[3], const int (&nn)[3]) {
                        vis_note(ta.vsink[k], g, (int)p, home, cn, nn, tile, t0);
                    });
                } else if (!inside && idx < mh && vvalid[k]) {
                    // away from home: pushed from the visitor list of the tile it is in
                } else {
                    // a crowded tile, or away from home without valid visitor
                    // lists: pushed by the global kernel after this one
                    const unsigned long long q = atomicAdd(ta.nstrag + k, 1ull);
                    ta.strag[k][2 * q] = (int)p;
                    ta.strag[k][2 * q + 1] = home;
                }
            }
            idx += (long long)nwarp * 32;
            slot ^= 1;
        }
        cp_async_wait_all();
    }
    if (!use_smem) return;
    __syncthreads();
    // 4. reassemble the limbs and flush with one pass of global atomics
    for (int e = threadIdx.x; e < nacc * D3; e += blockDim.x) {
        int c = e / D3, l = e - c * D3;
        int lz = l / D2, r = l - lz * D2, ly = r / DE, lx = r - ly * DE;
        const unsigned *q = sa + c * NL * DS + lz * dsz + ly * dsy + lx;
        long long tot;
        if constexpr (NL == 2) tot = ((long long)(int)q[DS] << kLimbBits) + (long long)q[0];
        else
            tot = ((long long)(int)q[2 * DS] << (2 * kLimbBits)) + ((long long)q[DS] << kLimbBits) + (long long)q[0];
        if (tot == 0) continue;
        int x = dO[0] + lx, y = dO[1] + ly, z = dO[2] + lz;
        // FP32: single-precision arithmetic (the sum rounded to 24 bits)
        const real v = (real)tot * (real)ta.inv_scale[c < 3 ? c : 3];
        if (x >= -1 && x <= g.f[0] && y >= -1 && y <= g.f[1] && z >= -1 && z <= g.f[2])
            atomic_add(ta.ring[c] + g.ri(z, y, x), v);
        else
            set_status(ta.sp[0].status, ST_OOB);
    }
}

static TileGeom tile_layout(const pic_ctx *c) {
    TileGeom t = tile_geom(c);
    const int P = c->order == 2 ? 3 : 5;
    t.GE = t.T + 2 * (P / 2) + 1;
    t.DE = t.T + 2 * (P / 2) + 3;
    padded_strides(t.GE, t.T, t.gsy, t.gsz);
    padded_strides(t.DE, t.T, t.dsy, t.dsz);
    t.gsize = t.GE * t.gsz;
    t.dsize = t.DE * t.dsz;
    t.nacc = (c->p.deposit_rho && !c->rho_skip) ? 5 : 3;
    return t;
}

TileBoxes tile_boxes(const pic_ctx *c) {
    const TileGeom t = tile_layout(c);
    return TileBoxes{t.GE, t.DE, t.gsy, t.gsz, t.gsize, t.dsy, t.dsz, t.dsize};
}

// Threads per CTA of a launch.  FP64 at 2nd order on a step whose rho is
// observed: its five accumulators (131 KB per CTA) leave room for one CTA
// per SM, so that CTA takes 512 threads instead of 256.
static int tile_launch_threads(const pic_ctx *c) {
    const bool o2 = c->order == 2;
    if (!c->fp32 && o2 && tile_layout(c).nacc == 5) return 512;
    return c->fp32 ? (o2 ? tile_threads<float, 3>() : tile_threads<float, 5>())
                   : (o2 ? tile_threads<double, 3>() : tile_threads<double, 5>());
}

size_t tile_smem_bytes(const pic_ctx *c) {
    const TileGeom t = tile_layout(c);
    const size_t rs = c->fp32 ? 4 : 8, nl = c->fp32 ? 2 : 3;
    const size_t warps = (size_t)tile_launch_threads(c) / 32;
    const size_t words = c->fp32 ? PartIn<float>::kWords : PartIn<double>::kWords;
    // the accumulators of this launch: jx, jy, jz, and rho0, rho1 on a step whose rho is observed
    return 6 * (size_t)t.gsize * rs + 4 * (size_t)particle_buffer_offset((int)(t.nacc * nl * t.dsize)) +
           warps * 2 * 32 * (words * rs + sizeof(int2));
}

VisSink vis_sink_of(const pic_ctx *c, const Species &s) {
    VisSink v{};
    if (!s.vs) return v;
    v.raw = s.vraw;
    v.nraw = &s.vs->nraw[s.vis_par];
    v.valid = &s.vs->valid_next[s.vis_par];
    v.cnt = s.vis_cnt;
    v.cap = s.vcap;
    v.T = c->tile;
    v.nodes = c->node_tiles ? 1 : 0;
    for (int d = 0; d < 3; ++d) v.nt[d] = c->ntile[d];
    return v;
}

template <typename real, int P, bool SPIN>
static void tile_push_t(pic_ctx *c, int mask) {
    const TileArgs<real> ta = make_tile_args<real, P>(c, mask, tile_layout(c));
    size_t smem = tile_smem_bytes(c);
    const int ntiles = c->ntile[0] * c->ntile[1] * c->ntile[2];
    constexpr int NT = tile_threads<real, P>();
    auto launch = [&](auto kernel, int threads) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kernel<<<ntiles, threads, smem, c->stream>>>(ta);
    };
    const bool wide = tile_launch_threads(c) != NT;
    if constexpr (sizeof(real) == 8 && NT != 512) {
        if (wide) {
            launch(tile_push_kernel<real, P, SPIN, 512>, 512);
            return;
        }
    }
    launch(tile_push_kernel<real, P, SPIN, NT>, NT);
}

// the counts pic_particle_order_stats reports (host side, synchronising)
int tile_order_stats(pic_ctx *c, int kind, long long (&out)[4]) {
    Species &s = c->sp[kind];
    out[0] = out[1] = out[3] = 0;
    out[2] = s.pushes_since_sort;
    if (cudaStreamSynchronize(c->stream) != cudaSuccess) return PIC_ECUDA;
    if (s.vs && s.sorted) {
        // the lists the next push will read: built from what the last push
        // recorded unless a full sort comes first
        VisState v{};
        if (cudaMemcpy(&v, s.vs, sizeof v, cudaMemcpyDeviceToHost) != cudaSuccess) return PIC_ECUDA;
        const bool built = s.vis_built_for == s.pushes_since_sort;
        out[0] = built ? (long long)v.nvis : std::min<long long>((long long)v.nraw[s.vis_par], s.vcap);
        out[1] = built ? v.valid_cur : v.valid_next[s.vis_par];
    }
    if (c->d_nstrag) {
        unsigned long long ns[2] = {0, 0};
        if (cudaMemcpy(ns, c->d_nstrag, sizeof ns, cudaMemcpyDeviceToHost) != cudaSuccess) return PIC_ECUDA;
        out[3] = (long long)ns[kind];
    }
    return PIC_OK;
}

void launch_tile_push(pic_ctx *c, int mask) {
    prepare_push(c, mask);
    bool spin = ((mask & 1) && spin_active(c, 0)) || ((mask & 2) && spin_active(c, 1));
    prof_begin(c, "tile_push_gather_deposit");
    if (c->node_tiles) {
        launch_node_tile_kernel(c, mask, spin);
    } else if (c->fp32) {
        if (c->order == 2) spin ? tile_push_t<float, 3, true>(c, mask) : tile_push_t<float, 3, false>(c, mask);
        else spin ? tile_push_t<float, 5, true>(c, mask) : tile_push_t<float, 5, false>(c, mask);
    } else {
        if (c->order == 2) spin ? tile_push_t<double, 3, true>(c, mask) : tile_push_t<double, 3, false>(c, mask);
        else spin ? tile_push_t<double, 5, true>(c, mask) : tile_push_t<double, 5, false>(c, mask);
    }
    prof_end(c);
    prof_begin(c, "straggler_push");
    launch_push_stragglers(c, mask);
    prof_end(c);
    for (int k = 0; k < 2; ++k) {
        Species &s = c->sp[k];
        if (!((mask >> k) & 1) || s.n_host <= 0) continue;
        s.cur = 1 - s.cur;
        s.pushes_since_sort += 1;
    }
}

}  // namespace pic
