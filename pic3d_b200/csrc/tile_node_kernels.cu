// Tiled gather + push + deposit over tiles of nodes at 2nd order.
//
// As at 4th order (tile_mma_kernels.cu) a tile holds 4 x 4 x 4 nodes (a
// particle's node is its primal stencil index), the particles are sorted by
// tile, then node, and one CTA owns one tile: it stages the six field
// components in shared memory, pushes the tile's particles one per lane, and
// deposits into shared fixed-point accumulators flushed by one pass of global
// atomics.
//
// The deposit.  Particles of a node that stay in it cover the same 3 x 3 x 3
// points, 54 currents.  With the averages s = s_old + ds/2 and
// d = ds/sqrt(12) of each axis the Esirkepov weight of two axes is
// W(u, v) = s(u) s(v) + d(u) d(v).  Each lane leaves its particle's factors
// (9 pairs (s, d), 6 scaled fluxes) in shared memory; then nine lanes per
// node, three nodes at a time, go through the node's particles, a lane
// summing the six currents of its pair of points (two fluxes of each
// component) in registers, and add the sums to the accumulators once per node
// and batch.  A scatter per particle adds 108 (FP32) or 162 (FP64) words by
// shared atomics, 3.3 wavefronts each: the particles of a cell hit the same
// address, and sorted so that they do not, the gather's loads conflict.  Node
// order makes the gather's loads broadcasts and leaves 12 (18) atomics per
// lane, node and batch.
// What bounds it (128 x 64 x 64 cells, 8 + 8 per cell): in FP32 issue (65 % of
// the slots) and the shared-memory pipe (75 %) together, 850 us against 993 us
// with the scatter; in FP64 the shared-memory pipe (83 %), on 256 x 128 x 128
// cells 10.3 against 11.5 ms, with rho 13.5 against 17.0 ms.  About half of the
// pipe's time goes to the gather's 162 loads.
// A particle that changes its node goes into its warp's queue; the general
// deposit runs on 32 queued particles at a time, and on the rest of the tile's
// at the end.  An entry is the particle's index: its move is read back from
// where the push stored it.
#include "tile_common.cuh"

namespace pic {

namespace {

template <typename real>
struct alignas(2 * sizeof(real)) Pair {
    real s, d;
};

template <typename real, bool RHO>
struct NodeTile2 {
    static constexpr bool F64 = sizeof(real) == 8;
    static constexpr int T = 4, P = 3, H = 1, NL = limbs<real>(), NACC = RHO ? 5 : 3;
    // Gather box.  Lanes hold about five neighbouring nodes of a row with
    // either dual index: {0 .. 4} + {0, 1} gsy + {0, 1} gsz fall into
    // different banks (FP64: those of a half-warp's two or three nodes).
    static constexpr int GE = T + 2 * H + 1, gsy = GE, gsz = F64 ? 52 : 49, GS = GE * gsz;
    // Accumulators: three neighbouring nodes' pairs of points {0, 1, 2} +
    // {0, 1, 2} dsy + {0, 1, 2} dsz, one bank shared.
    static constexpr int DE = T + 2 * H + 2, dsy = DE, dsz = DE * DE + 3, DS = DE * dsz;
    // One particle's factors: 6 fluxes, charge, pad, then (s, d) of x, y, z,
    // then (rho) the new shapes of z, a zero, those of x and y; a stride that
    // spreads the lanes' stores over the banks
    static constexpr int kPairs = 8, kNew = kPairs + 6 * P, TS = RHO ? kNew + 12 : F64 ? kNew : kNew + 2;
    static constexpr int KW = PartIn<real>::kWords;
    // CTAs of 4 warps, as many per SM as shared memory (FP64) or registers
    // (FP32) allow: the others cover one's staging, flush and last partial
    // round.  FP64 with two CTAs of 8 warps: 11.1 against 10.3 ms (256 x 128 x
    // 128 cells), with rho one of 16 against two of 4 warps: 17.2 and 13.5 ms.
    // FP32 with five CTAs (96 registers): the same as four.
    static constexpr int kThreads = 128, kWarps = kThreads / 32, kCtas = F64 ? (RHO ? 2 : 3) : 4;
    static constexpr int kQueue = 64;
    // Per warp: slot 0, rest, slot 1.  A slot holds a batch of particle inputs;
    // the table of factors takes the place of the batch it belongs to and
    // of the rest, whichever side of it the slot is on.
    static constexpr int kSlot = 32 * KW * sizeof(real), kTable = 32 * TS * sizeof(real);
    static constexpr int kWarpBytes = kTable + kSlot + 2 * 32 * (int)sizeof(int2) + kQueue * (int)sizeof(int);
    static constexpr int kFieldBytes = (6 * GS * sizeof(real) + 15) / 16 * 16;
    static constexpr int kAccBytes = (NACC * NL * DS * 4 + 15) / 16 * 16;
    static constexpr int kZeroBytes = (TS * sizeof(real) + 15) / 16 * 16;   // a row of zeros
    static constexpr int kBytes = kFieldBytes + kAccBytes + kWarps * kWarpBytes + kZeroBytes;
    static_assert(kSlot % 16 == 0 && kTable > kSlot, "");
    static_assert(kCtas * (kBytes + 1024 + 128) <= 228 * 1024, "the CTAs of an SM share 228 KB");
};

// The sums over some particles (at most 32) of the contributions f w to two
// points, in steps of the accumulators, and their addition to the points.
// FP64: the steps are 2^-49 of the largest contribution, far above the
// rounding of a sum in double.
template <typename real>
struct PairSum {
    double v[2] = {0.0, 0.0};
    __device__ __forceinline__ void add(Pair<double> f, double w0, double w1) {
        v[0] = fma(f.s, w0, v[0]);
        v[1] = fma(f.d, w1, v[1]);
    }
    template <int I>
    __device__ __forceinline__ void to(unsigned *a, int lstride) const {
        const long long q = __double2ll_rn(v[I]);
        atomicAdd(a, (unsigned)q & kLimbMask);
        atomicAdd(a + lstride, (unsigned)(q >> kLimbBits) & kLimbMask);
        atomicAdd(a + 2 * lstride, (unsigned)(int)(q >> (2 * kLimbBits)));
    }
};

// FP32: a sum in one register loses what the accumulators would have kept (64
// particles per node, 0.3 c thermal: currents 12 % less accurate than with
// an addition per particle).  It is kept in two: `hi` starts at 1.5 2^41, where
// a float's last bit is 2^18 (one step of the upper limb), so that it takes
// the multiple of 2^18 nearest to each contribution (up to 2^31), without
// error; `lo` takes the rest, up to 2^17 each, rounded to a fraction of a step.
// Two points per instruction (FP32 pairs).  128 x 64 x 64 cells, 8 + 8 particles
// per cell: 850 us against 796 with one register; sums in FP64, whose operands
// have to be converted, 893, two registers without pairs 881.
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
template <>
struct PairSum<float> {
    static constexpr float kStart = 3298534883328.0f;
    unsigned long long hi = pack2(kStart, kStart), lo = 0ull;
    __device__ __forceinline__ void add(Pair<float> f, float w0, float w1) {
        const unsigned long long ff = pack2(f.s, f.d), ww = pack2(w0, w1), t = fma2(ff, ww, hi);
        lo = add2(lo, fma2(ff, ww, sub2(hi, t)));   // f w - (t - hi)
        hi = t;
    }
    template <int I>
    __device__ __forceinline__ void to(unsigned *a, int lstride) const {
        static_assert(kLimbBits == 18, "the last bit of hi is one step of the upper limb");
        const int upper = (int)(unsigned)(hi >> (32 * I)) - __float_as_int(kStart);
        const int rest = __float2int_rn(__uint_as_float((unsigned)(lo >> (32 * I))));
        atomicAdd(a, (unsigned)rest & kLimbMask);
        atomicAdd(a + lstride, (unsigned)(upper + (rest >> kLimbBits)));
    }
};

template <typename real, bool SPIN, bool RHO>
__global__ void __launch_bounds__(NodeTile2<real, RHO>::kThreads, NodeTile2<real, RHO>::kCtas)
    node_sum_kernel(const __grid_constant__ TileArgs<real> ta) {
    using L = NodeTile2<real, RHO>;
    constexpr int P = L::P, H = L::H, NL = L::NL, T = L::T, NACC = L::NACC, NT = L::kThreads, NW = L::kWarps, KW = L::KW;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int left[NW];
    real *sf = reinterpret_cast<real *>(smem_raw);
    unsigned *sa = reinterpret_cast<unsigned *>(smem_raw + L::kFieldBytes);   // [component][limb][DS]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    using PWord = typename PartIn<real>::word;
    unsigned char *wbase = smem_raw + L::kFieldBytes + L::kAccBytes;
    unsigned char *wb = wbase + warp * L::kWarpBytes;
    int2 *sp_loc = reinterpret_cast<int2 *>(wb + L::kTable + L::kSlot);
    constexpr int kQueueAt = L::kTable + L::kSlot + 2 * 32 * (int)sizeof(int2);
    int *queue = reinterpret_cast<int *>(wb + kQueueAt);

    constexpr int zero_at = (L::kBytes - L::kZeroBytes) / (int)sizeof(real);

    const Geom &g = ta.sp[0].g;
    const int tile = blockIdx.x;
    const int tx = tile % ta.t.nt[0], ty = (tile / ta.t.nt[0]) % ta.t.nt[1], tz = tile / (ta.t.nt[0] * ta.t.nt[1]);
    const int t0[3] = {tx * T, ty * T, tz * T};
    // particle ranges: this tile's slice of the sorted arrays (home
    // particles) and its visitor list
    constexpr int kKeys = T * T * T;
    int pa[2] = {0, 0}, va[2] = {0, 0}, mh[2] = {0, 0}, m[2] = {0, 0};
    bool vvalid[2] = {false, false};
    long long mtot = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (!ta.active[k]) continue;
        const long long n = *ta.sp[k].count;
        long long b = ta.offs[k][(long long)(tile + 1) * kKeys];
        const long long a = ta.offs[k][(long long)tile * kKeys];
        b = b < n ? b : n;
        const long long home = b > a ? b - a : 0;
        vvalid[k] = ta.vs[k] && ta.vs[k]->valid_cur;
        long long vis = 0;
        if (vvalid[k] && ta.vis_off[k]) {
            const uint2 r = ta.vis_off[k][tile];
            va[k] = (int)r.x;
            vis = r.y - r.x;
        }
        mtot += home + vis;
        pa[k] = (int)a;
        mh[k] = (int)home;
        m[k] = (int)(home + vis);
    }
    if (mtot == 0) return;
    const bool use_smem = mtot <= kMaxTileParticles;
    // The batches of both species in one list: a warp takes every NW-th, its
    // inputs copied asynchronously one batch ahead.
    const int nb0 = (m[0] + 31) >> 5, nb = nb0 + ((m[1] + 31) >> 5);
    auto slot_of = [&](int slot) { return reinterpret_cast<PWord *>(wb + (slot ? L::kTable : 0)); };
    auto prefetch = [&](int b, int slot) {
        if (b >= nb) return;
        const int k = b >= nb0;
        const int i = (b - (k ? nb0 : 0)) * 32 + lane, home = k ? mh[1] : mh[0];
        if (i >= (k ? m[1] : m[0])) return;
        int2 e = make_int2((k ? pa[1] : pa[0]) + i, tile);
        if (i >= home) e = (reinterpret_cast<const int2 *>(ta.vis[k]) + (k ? va[1] : va[0]))[i - home];
        sp_loc[slot * 32 + lane] = e;
        PWord *dst = slot_of(slot) + lane;
        const PushArgs<real> &a = ta.sp[k];
#pragma unroll
        for (int w = 0; w < KW; ++w) cp_async<sizeof(PWord)>(dst + w * 32, particle_word_src(a, (long long)e.x, w));
    };
    // buffer coordinates of the first staged field point and of the first
    // accumulator point
    const int gO[3] = {t0[0] + g.mem - 2 - H, t0[1] + g.mem - 2 - H, t0[2] + g.mem - 2 - H};
    if (use_smem) {
        // stage the fields (asynchronous copies; points outside the buffers
        // read as zero) and clear the accumulators
        constexpr int G2 = L::GE * L::GE, G3 = G2 * L::GE;
        for (int l = threadIdx.x; l < G3; l += NT) {
            const int lz = l / G2, r = l - lz * G2, ly = r / L::GE, lx = r - ly * L::GE;
            const int x = gO[0] + lx, y = gO[1] + ly, z = gO[2] + lz;
            const bool in = x >= 0 && x < g.f[0] && y >= 0 && y < g.f[1] && z >= 0 && z < g.f[2];
            const int src = in ? g.fi(z, y, x) : 0;
            real *dst = sf + lz * L::gsz + ly * L::gsy + lx;
#pragma unroll
            for (int c = 0; c < 6; ++c)
                cp_async<sizeof(real)>(dst + c * L::GS, ta.field[c] + src, in ? (int)sizeof(real) : 0);
        }
    }
    int slot = 0;
    prefetch(warp, 0);   // the first batch arrives with the fields
    cp_async_commit();
    if (use_smem)
        for (int e = threadIdx.x; e < L::kAccBytes / 16; e += NT) reinterpret_cast<uint4 *>(sa)[e] = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x < L::TS) sf[zero_at + threadIdx.x] = real(0);
    cp_async_wait_all();
    __syncthreads();

    View<const real> fs[6];
#pragma unroll
    for (int c = 0; c < 6; ++c)
        fs[c] = View<const real>{sf + c * L::GS, L::gsy, L::gsz, -(gO[2] * L::gsz + gO[1] * L::gsy + gO[0])};
    const int lo[3] = {t0[0] + g.mem - 1, t0[1] + g.mem - 1, t0[2] + g.mem - 1};   // buffer index of the first node
    // this lane's part in the sums: which of three nodes, which pair of points
    const int grp = lane / 9, u = (lane - 9 * grp) % 3, v = (lane - 9 * grp) / 3;

    int queued = 0;
#pragma unroll 1
    for (int b = warp;; b += NW) {
        const bool more = b < nb;
        if (more) {
            const int k = b >= nb0;
            const int i = (b - (k ? nb0 : 0)) * 32 + lane;
            const PushArgs<real> &a = ta.sp[k];
            cp_async_wait_all();
            const int2 loc = sp_loc[slot * 32 + lane];
            prefetch(b + NW, slot ^ 1);
            cp_async_commit();
            const PWord *row_in = slot_of(slot) + lane;

            // ---- push, one particle per lane --------------------------------
            bool dep = false;
            Moved<real> mv;
            // (adjoint contexts: removed particles stay, dead)
            if (i < (k ? m[1] : m[0]) && !(a.dead && a.dead[loc.x])) {
                const long long p = loc.x;
                PartIn<real> in;
#pragma unroll
                for (int w = 0; w < PartIn<real>::kPos; ++w) in.v[w] = row_in[w * 32];
                OldPos<real> o;
                decode_old(a, p, in, o);
                bool inside = true;
#pragma unroll
                for (int d = 0; d < 3; ++d) inside = inside && o.ip[d] >= lo[d] && o.ip[d] < lo[d] + T;
                if (!in_buffers(g, o, H)) {
                    set_status(a.status, ST_OOB);
                } else if (inside && use_smem) {
                    constexpr int mo = PartIn<real>::kPos;   // momenta, then weight
                    const real *pr = reinterpret_cast<const real *>(row_in - lane);
                    const PmSrc<real> pm{pr + mo * 32, pr + (mo + 1) * 32, pr + (mo + 2) * 32, pr + (mo + 3) * 32, lane};
                    dep = push_move<real, P, SPIN, false>(
                        a, p, o, pm, fs,
                        [&](const int (&cn)[3], const int (&nn)[3]) {
                            vis_note(ta.vsink[k], g, (int)p, loc.y, cn, nn, tile, t0);
                        },
                        mv);
                } else if (!inside && i < (k ? mh[1] : mh[0]) && (k ? vvalid[1] : vvalid[0])) {
                    // away from home: pushed from the visitor list of the tile it is in
                } else {
                    // a crowded tile, or away from home without valid visitor
                    // lists: pushed by the global kernel after this one
                    const unsigned long long q = atomicAdd(ta.nstrag + k, 1ull);
                    ta.strag[k][2 * q] = (int)p;
                    ta.strag[k][2 * q + 1] = loc.y;
                }
            }
            // ---- the factors of the particles that keep their node ----------
            const bool moves = dep && (mv.i1[0] != mv.i2[0] || mv.i1[1] != mv.i2[1] || mv.i1[2] != mv.i2[2]);
            const bool sums = dep && !moves && (RHO || mv.moved);
            // The table takes the place of the batch's inputs: every lane has read
            // its own (the weight last) before another stores there.
            __syncwarp();
            const unsigned changes = __ballot_sync(0xffffffffu, moves);
            real *tab = reinterpret_cast<real *>(slot ? wb + L::kSlot : wb);
            const int tab_at = (int)(tab - sf);
            int node = -1;
            if (sums) {
                node = (mv.i1[0] - lo[0]) + T * ((mv.i1[1] - lo[1]) + T * (mv.i1[2] - lo[2]));
                real *row = tab + lane * L::TS;
                Pair<real> f[4];   // (x, y) of the first flux, of the second, z, charge
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    real w0[P], ds[P], w1[P];
                    shape_weights(mv.d0[d], w0);
                    if constexpr (sizeof(real) == 8) {
                        shape_weights(mv.dm[d], w1);
#pragma unroll
                        for (int q = 0; q < P; ++q) ds[q] = w1[q] - w0[q];
                    } else {
                        shape_diff(mv.d0[d], mv.dm[d], ds);
                        if constexpr (RHO) shape_weights(mv.d0[d] + mv.dm[d], w1);
                    }
                    const real q0 = -(mv.qw * a.d_dt[d] * ta.scale[d]);
                    (d == 0 ? f[0].s : d == 1 ? f[0].d : f[2].s) = q0 * ds[0];
                    (d == 0 ? f[1].s : d == 1 ? f[1].d : f[2].d) = q0 * (ds[0] + ds[1]);
#pragma unroll
                    for (int q = 0; q < P; ++q) {
                        reinterpret_cast<Pair<real> *>(row + L::kPairs)[3 * d + q] =
                            Pair<real>{w0[q] + real(0.5) * ds[q], ds[q] * real(0.28867513459481287)};
                        if constexpr (RHO) row[L::kNew + (d == 2 ? 0 : 4 + 3 * d) + q] = w1[q];
                    }
                }
                if constexpr (RHO) row[L::kNew + 3] = real(0);
                f[3] = Pair<real>{RHO ? mv.qw * ta.scale[3] : real(0), real(0)};
#pragma unroll
                for (int q = 0; q < 4; ++q) reinterpret_cast<Pair<real> *>(row)[q] = f[q];
            }
            if (moves) queue[queued + __popc(changes & ((1u << lane) - 1u))] = loc.x | (k << 31);
            queued += __popc(changes);
            const unsigned same = __match_any_sync(0xffffffffu, node);
            unsigned first = __ballot_sync(0xffffffffu, sums && lane == __ffs(same) - 1);
            __syncwarp();

            // ---- sums over the particles of three nodes at a time -----------
#pragma unroll 1
            while (first) {
                int mine = -1, n = 0, at = 0;
                unsigned todo = 0;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const int l = __ffs(first) - 1;   // -1: no node left
                    const unsigned s = l < 0 ? 0u : __shfl_sync(0xffffffffu, same, l & 31);
                    const int nd = __shfl_sync(0xffffffffu, node, l & 31);
                    first &= first - 1;
                    n = max(n, __popc(s));
                    if (grp == q) {
                        mine = l;
                        todo = s;
                        at = nd;
                    }
                }
                // (jx, jy) of the first points, of the second, (jz, jz); rho
                PairSum<real> j[3], r[RHO ? 2 : 1];
                // lanes whose node has no more particles read zeros (their last
                // row again, with zeros for its fluxes only: 2 % slower)
#pragma unroll 2
                for (int it = 0; it < n; ++it) {
                    const real *row = sf + (todo ? tab_at + (__ffs(todo) - 1) * L::TS : zero_at);
                    todo &= todo - 1;
                    const Pair<real> *fl = reinterpret_cast<const Pair<real> *>(row),
                                     *xyz = reinterpret_cast<const Pair<real> *>(row + L::kPairs);
                    const Pair<real> xu = xyz[u], yu = xyz[3 + u], yv = xyz[3 + v], zv = xyz[6 + v];
                    const real wx = yu.s * zv.s + yu.d * zv.d, wy = xu.s * zv.s + xu.d * zv.d,
                               wz = xu.s * yv.s + xu.d * yv.d;
                    j[0].add(fl[0], wx, wy);
                    j[1].add(fl[1], wx, wy);
                    j[2].add(fl[2], wz, wz);
                    if constexpr (RHO) {
                        const real w = row[6] * (row[L::kNew + 4 + u] * row[L::kNew + 7 + v]);
                        const Pair<real> *z = reinterpret_cast<const Pair<real> *>(row + L::kNew);
                        r[0].add(z[0], w, w);
                        r[1].add(z[1], w, w);
                    }
                }
                if (mine >= 0) {
                    unsigned *q0 = sa + ((at & 3) + 1) + (((at >> 2) & 3) + 1) * L::dsy + ((at >> 4) + 1) * L::dsz;
                    unsigned *qx = q0 + u * L::dsy + v * L::dsz, *qy = q0 + NL * L::DS + u + v * L::dsz,
                             *qz = q0 + 2 * NL * L::DS + u + v * L::dsy;
                    j[0].template to<0>(qx, L::DS);
                    j[1].template to<0>(qx + 1, L::DS);
                    j[0].template to<1>(qy, L::DS);
                    j[1].template to<1>(qy + L::dsy, L::DS);
                    j[2].template to<0>(qz, L::DS);
                    j[2].template to<1>(qz + L::dsz, L::DS);
                    if constexpr (RHO) {
                        unsigned *qr = q0 + (3 + k) * NL * L::DS + u + v * L::dsy;
                        r[0].template to<0>(qr, L::DS);
                        r[0].template to<1>(qr + L::dsz, L::DS);
                        r[1].template to<0>(qr + 2 * L::dsz, L::DS);
                    }
                }
            }
            __syncwarp();
            slot ^= 1;
        }
        // ---- the particles that changed their node ---------------------------
        int total = 32, step = 32, i = lane;
        unsigned parts = RHO ? 15u : 7u;
        if (more) {
            if (queued < 32) continue;
            queued -= 32;
        } else {
            // the rest of all warps' (fewer than 32 of each): 32 particles and
            // one array per warp, so that the CTA does not wait for a single one
            if (lane == 0) left[warp] = queued;
            __syncthreads();
            total = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) total += left[w];
            constexpr int NP = RHO ? 4 : 3, NS = NW / NP;
            if (warp >= NS * NP) total = 0;
            step = 32 * NS;
            i += 32 * (warp / NP);
            parts = 1u << (warp % NP);
        }
#pragma unroll 1
        for (; i < total; i += step) {
            int w = warp, q = queued + i;
            if (!more) {
                for (w = 0, q = i; q >= left[w]; ++w) q -= left[w];
            }
            const int e = reinterpret_cast<const int *>(wbase + w * L::kWarpBytes + kQueueAt)[q];
            const int k = (unsigned)e >> 31;
            FixedAcc<real, NL> af;
#pragma unroll
            for (int c = 0; c < 3; ++c) af.p[c] = sa + c * NL * L::DS;
            af.p[3] = RHO ? sa + (3 + k) * NL * L::DS : nullptr;
            af.lstride = L::DS;
            af.sy = L::dsy;
            af.sz = L::dsz;
            af.o = -(gO[2] * L::dsz + gO[1] * L::dsy + gO[0]);
#pragma unroll
            for (int c = 0; c < 4; ++c) af.scale[c] = ta.scale[c];
            deposit_stored<real, P>(af, ta.sp[k], e & 0x7fffffff, parts);
        }
        __syncwarp();
        if (!more) break;
    }
    cp_async_wait_all();
    if (!use_smem) return;
    __syncthreads();
    // reassemble the limbs and flush with one pass of global atomics
    constexpr int D2 = L::DE * L::DE, D3 = D2 * L::DE;
    for (int l = threadIdx.x; l < D3; l += NT) {
        const int lz = l / D2, r = l - lz * D2, ly = r / L::DE, lx = r - ly * L::DE;
        const int x = gO[0] + lx, y = gO[1] + ly, z = gO[2] + lz;
        const bool in = x >= -1 && x <= g.f[0] && y >= -1 && y <= g.f[1] && z >= -1 && z <= g.f[2];
        const int dst = in ? g.ri(z, y, x) : 0;
        const unsigned *q = sa + lz * L::dsz + ly * L::dsy + lx;
#pragma unroll
        for (int c = 0; c < NACC; ++c, q += NL * L::DS) {
            long long tot;
            if constexpr (NL == 2) tot = ((long long)(int)q[L::DS] << kLimbBits) + (long long)q[0];
            else
                tot = ((long long)(int)q[2 * L::DS] << (2 * kLimbBits)) + ((long long)q[L::DS] << kLimbBits) + (long long)q[0];
            if (tot == 0) continue;
            // FP32: single-precision arithmetic (the sum rounded to 24 bits)
            const real val = (real)tot * (real)ta.inv_scale[c < 3 ? c : 3];
            if (in) atomic_add(ta.ring[c] + dst, val);
            else set_status(ta.sp[0].status, ST_OOB);
        }
    }
}

template <typename real, bool SPIN>
void node_sum_push(pic_ctx *c, int mask) {
    TileGeom t{};
    t.T = c->tile;
    for (int d = 0; d < 3; ++d) t.nt[d] = c->ntile[d];
    t.nkeys = c->nkeys;
    t.nodes = 1;
    t.nacc = (c->p.deposit_rho && !c->rho_skip) ? 5 : 3;
    const TileArgs<real> ta = make_tile_args<real, 3>(c, mask, t);
    const int ntiles = c->ntile[0] * c->ntile[1] * c->ntile[2];
    auto launch = [&](auto kernel, int threads, int smem) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        kernel<<<ntiles, threads, smem, c->stream>>>(ta);
    };
    if (t.nacc == 5) launch(node_sum_kernel<real, SPIN, true>, NodeTile2<real, true>::kThreads, NodeTile2<real, true>::kBytes);
    else launch(node_sum_kernel<real, SPIN, false>, NodeTile2<real, false>::kThreads, NodeTile2<real, false>::kBytes);
}

}  // namespace

size_t node_sum_smem_bytes(const pic_ctx *c) {
    return c->fp32 ? NodeTile2<float, true>::kBytes : NodeTile2<double, true>::kBytes;
}

void launch_node_sum_kernel(pic_ctx *c, int mask, bool spin) {
    if (c->fp32) spin ? node_sum_push<float, true>(c, mask) : node_sum_push<float, false>(c, mask);
    else spin ? node_sum_push<double, true>(c, mask) : node_sum_push<double, false>(c, mask);
}

}  // namespace pic
