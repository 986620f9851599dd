// Tiled gather + push + deposit over tiles of nodes, with the deposit as
// small matrix products.
//
// A particle's node is its primal stencil index (the grid point nearest to
// it).  A tile holds 4 x 4 x 4 nodes; the particles of each species are kept
// in counting-sort order by tile, then node, x fastest.  One CTA owns one
// tile: it stages the six field components of the tile plus the gather halo
// in shared memory, pushes the tile's particles one per lane, and deposits
// their currents into shared fixed-point accumulators that one pass of
// global atomics flushes at the end.
//
// The deposit.  All particles of a row (the nodes of one y and z) that keep
// their y and z node cover the same 5 x 5 points in y and z, and at most
// eight points in x.  With the averages s = s_old + ds/2 and d = ds/sqrt(12)
// the Esirkepov weight of two axes is the sum of two products,
//     W(j, k) = s(j) s(k) + d(j) d(k),
// so the currents of a row are sums over its particles of outer products,
//     Jx(x; j, k) = sum_p Cx_p(x) W_p(j, k)
//     Jy(j, k; x) = sum_p [Cy_p(j) s_p(k)] s_p(x) + [Cy_p(j) d_p(k)] d_p(x)
//     Jz(k, j; x) = sum_p [Cz_p(k) s_p(j)] s_p(x) + [Cz_p(k) d_p(j)] d_p(x)
// (C the running sum of ds along the component's axis), i.e. matrix products
// whose inner dimension is the particle.  A warp forms them with FP64
// m8n8k4 matrix instructions, four particles per instruction, in both
// precisions (FP32 has no matrix unit of its own accuracy; the products of its
// FP32 factors are then exact, their sums rounded at 53 bits), and adds each
// row's sum to the shared accumulators once.  The scatter by particle this replaces spent
// 300 x 3 (FP64) shared atomics per particle, 3.2 cycles of the shared-memory
// pipe for each warp's worth.
// Particles that change their y or z node, leave the row's eight columns, or
// are alone in their row within a batch are added point by point, one
// particle by the whole warp (a lane per column).
//
// What bounds it (128 x 64 x 64 cells, 8 + 8 particles per cell): FP64 takes
// 141 cycles of an SM per particle, of which the gather's 8-byte shared loads
// need 55 and all shared accesses 95; FP32 81 cycles, 190 warp instructions
// per particle at 0.54 of the issue rate.  The push alone takes 84 and 38.
#include "tile_common.cuh"

namespace pic {

namespace {

// D += A B, 8 x 4 by 4 x 8: A(row = lane / 4, k = lane % 4),
// B(k = lane % 4, col = lane / 4), D(row = lane / 4, cols 2 (lane % 4) + {0, 1})
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
        : "+d"(d[0]), "+d"(d[1])
        : "d"(a), "d"(b));
}

template <typename real>
struct alignas(2 * sizeof(real)) Pair {
    real s, d;
};

// Compile-time layout of a tile of 4 x 4 x 4 nodes.  Strides: consecutive
// lanes hold neighbouring nodes of a row with either dual index, so a
// gather's addresses are {0..4} + {0, 1} gsy + {0, 1} gsz; these strides put
// them (for FP64, those of a half-warp) into different banks.
template <typename real, int P>
struct NodeTile {
    static_assert(P == 5, "a row of 4 nodes has 8 columns at 4th order");
    static constexpr bool F64 = sizeof(real) == 8;
    static constexpr int T = 4, H = P / 2, NL = limbs<real>();
    static constexpr int GE = T + 2 * H + 1;   // dual stencils start at node -1 - H
    static constexpr int gsy = GE, gsz = F64 ? 85 : 82, GS = GE * gsz;
    static constexpr int DE = T + 2 * H + 2;   // a move by one node to either side
    static constexpr int dsy = F64 ? 10 : 12, dsz = dsy * DE, DS = DE * dsz;
    // per-warp table of 8 particles: (s, d) pairs of the P + 1 points of each
    // axis, running sums C of the P fluxes of each axis (then the rho weight);
    // strides per particle chosen against bank conflicts
    static constexpr int Q = P + 1;
    static constexpr int PS = F64 ? 18 : 20, CS = F64 ? 20 : 24;
    static constexpr int kTableReals = 8 * (2 * PS + CS);
    static constexpr int KW = PartIn<real>::kWords;
    // FP64: one CTA per SM (195 KB), 4 warps per scheduler at 128 registers;
    // FP32: two CTAs of 8 warps, one of which stages and flushes while the
    // other pushes.  12 or 11 warps (168 registers) lost 3-7 % in FP64, two
    // CTAs of 7 or 10 warps 5-28 % in FP32.
    static constexpr int kThreads = F64 ? 512 : 256;
    static constexpr int kCtas = F64 ? 1 : 2;
    static constexpr int kWarps = kThreads / 32;
    static constexpr size_t warp_bytes() { return 2 * 32 * (KW * sizeof(real) + sizeof(int2)) + kTableReals * sizeof(real); }
    __host__ __device__ static constexpr size_t acc_bytes(int nacc) { return ((size_t)nacc * NL * DS * 4 + 15) & ~(size_t)15; }
    static constexpr size_t field_bytes() { return (6 * (size_t)GS * sizeof(real) + 15) & ~(size_t)15; }
    static size_t smem(int nacc) { return field_bytes() + acc_bytes(nacc) + kWarps * warp_bytes(); }
};

// s = s_old + ds/2 and d = ds/sqrt(12) of one axis of a move on its P + 1
// points from the lower node, and the running sums of ds
template <typename real, int P>
__device__ __forceinline__ void axis_factors(real d0, real dm, int cross, real (&s)[P + 1], real (&ds)[P + 1]) {
    Axis1D<real, P> ax;
    if constexpr (sizeof(real) == 8) axis_from_offsets<real, P>(0, d0, cross, dm, ax);
    else axis_from_move<P>(0, d0, dm, cross, ax);
#pragma unroll
    for (int q = 0; q <= P; ++q) {
        ds[q] = ax.ds[q];
        s[q] = ax.s0[q] + real(0.5) * ax.ds[q];
    }
}

constexpr double kInvSqrt12 = 0.28867513459481287, kSqrt3 = 1.7320508075688772;

// one value, already an integer, into the limbs of a point
template <int NL>
__device__ __forceinline__ void add_limbs(unsigned *a, int lstride, double v) {
    const long long q = __double2ll_rn(v);
    atomicAdd(a, (unsigned)q & kLimbMask);
    if constexpr (NL == 3) {
        atomicAdd(a + lstride, (unsigned)(q >> kLimbBits) & kLimbMask);
        atomicAdd(a + 2 * lstride, (unsigned)(int)(q >> (2 * kLimbBits)));
    } else {
        atomicAdd(a + lstride, (unsigned)(int)(q >> kLimbBits));
    }
}

// RHO: rho0 and rho1 are deposited too (steps whose rho is observed)
template <typename real, int P, bool SPIN, bool RHO>
__global__ void __launch_bounds__(NodeTile<real, P>::kThreads, NodeTile<real, P>::kCtas)
    node_tile_kernel(const __grid_constant__ TileArgs<real> ta) {
    using L = NodeTile<real, P>;
    constexpr int H = P / 2, NL = L::NL, Q = L::Q, T = L::T;
    constexpr int NACC = RHO ? 5 : 3, NT = L::kThreads, NW = L::kWarps;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    real *sf = reinterpret_cast<real *>(smem_raw);
    unsigned *sa = reinterpret_cast<unsigned *>(smem_raw + L::field_bytes());   // [component][limb][DS]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    using PWord = typename PartIn<real>::word;
    constexpr int KW = L::KW;
    unsigned char *wb = smem_raw + L::field_bytes() + L::acc_bytes(NACC) + warp * L::warp_bytes();
    // per warp: two slots of one batch of particle inputs, [word][lane], the
    // (index, home tile) of each lane's particle per slot, and the table
    PWord *sp_in = reinterpret_cast<PWord *>(wb);
    int2 *sp_loc = reinterpret_cast<int2 *>(wb + 2 * 32 * KW * sizeof(real));
    real *tab = reinterpret_cast<real *>(wb + 2 * 32 * (KW * sizeof(real) + sizeof(int2)));
    Pair<real> *tp = reinterpret_cast<Pair<real> *>(tab);
    real *tc = tab + 8 * 2 * L::PS;

    const Geom &g = ta.sp[0].g;
    const int tile = blockIdx.x;
    const int tx = tile % ta.t.nt[0], ty = (tile / ta.t.nt[0]) % ta.t.nt[1], tz = tile / (ta.t.nt[0] * ta.t.nt[1]);
    const int t0[3] = {tx * T, ty * T, tz * T};
    // particle ranges: this tile's slice of the sorted arrays (home
    // particles) and its visitor list
    constexpr int kKeys = T * T * T;
    long long pa[2] = {0, 0}, va[2] = {0, 0};
    int mh[2] = {0, 0}, m[2] = {0, 0};
    bool vvalid[2] = {false, false};
    long long mtot = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (!ta.active[k]) continue;
        const long long n = *ta.sp[k].count;
        long long b = ta.offs[k][(long long)(tile + 1) * kKeys];
        pa[k] = ta.offs[k][(long long)tile * kKeys];
        b = b < n ? b : n;
        const long long home = b > pa[k] ? b - pa[k] : 0;
        vvalid[k] = ta.vs[k] && ta.vs[k]->valid_cur;
        long long vis = 0;
        if (vvalid[k] && ta.vis_off[k]) {
            const uint2 r = ta.vis_off[k][tile];
            va[k] = r.x;
            vis = r.y - r.x;
        }
        mtot += home + vis;
        mh[k] = (int)home;
        m[k] = (int)(home + vis);
    }
    if (mtot == 0) return;
    const bool use_smem = mtot <= kMaxTileParticles;
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
        cp_async_commit();
        uint4 *z4 = reinterpret_cast<uint4 *>(sa);
        for (int e = threadIdx.x; e < (int)(L::acc_bytes(NACC) / 16); e += NT) z4[e] = make_uint4(0u, 0u, 0u, 0u);
    }
    cp_async_wait_all();
    __syncthreads();

    View<const real> fs[6];
#pragma unroll
    for (int c = 0; c < 6; ++c)
        fs[c] = View<const real>{sf + c * L::GS, L::gsy, L::gsz, -(gO[2] * L::gsz + gO[1] * L::gsy + gO[0])};
    const int lo[3] = {t0[0] + g.mem - 1, t0[1] + g.mem - 1, t0[2] + g.mem - 1};   // buffer index of the first node

    // the batches of both species in one list: a warp takes every NW-th
    const int nb0 = (m[0] + 31) >> 5, nb = nb0 + ((m[1] + 31) >> 5);
    auto prefetch = [&](int b, int slot) {
        if (b >= nb) return;
        const int k = b >= nb0;
        const int i = (b - (k ? nb0 : 0)) * 32 + lane;
        if (i >= m[k]) return;
        int2 e = make_int2((int)(pa[k] + i), tile);
        if (i >= mh[k]) e = (reinterpret_cast<const int2 *>(ta.vis[k]) + va[k])[i - mh[k]];
        sp_loc[slot * 32 + lane] = e;
        PWord *dst = sp_in + slot * KW * 32 + lane;
        const PushArgs<real> &a = ta.sp[k];
#pragma unroll
        for (int w = 0; w < KW; ++w) cp_async<sizeof(PWord)>(dst + w * 32, particle_word_src(a, (long long)e.x, w));
    };
    int slot = 0;
    prefetch(warp, 0);
    cp_async_commit();
#pragma unroll 1
    for (int b = warp; b < nb; b += NW) {
        const int k = b >= nb0;
        const int i = (b - (k ? nb0 : 0)) * 32 + lane;
        const PushArgs<real> &a = ta.sp[k];
        cp_async_wait_all();
        const int2 loc = sp_loc[slot * 32 + lane];
        prefetch(b + NW, slot ^ 1);
        cp_async_commit();
        PWord *row_in = sp_in + slot * KW * 32 + lane;

        // ---- push, one particle per lane ------------------------------------
        bool dep = false;      // the particle deposits
        // its row (y + 4 z of the node) if it takes part in the matrix products,
        // -2: at rest, it adds no current
        int row = -1;
        int geo = 0;           // lower node + 1 per axis (3 bits each), move in nodes + 1 per axis (2 bits each)
        Moved<real> mv;
        // (adjoint contexts: removed particles stay, dead)
        if (i < m[k] && !(a.dead && a.dead[loc.x])) {
            const long long p = loc.x;
            const int home = loc.y;
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
                const real *pr = reinterpret_cast<const real *>(sp_in + slot * KW * 32);
                const PmSrc<real> pm{pr + mo * 32, pr + (mo + 1) * 32, pr + (mo + 2) * 32, pr + (mo + 3) * 32, lane};
                dep = push_move<real, P, SPIN, false>(
                    a, p, o, pm, fs,
                    [&](const int (&cn)[3], const int (&nn)[3]) {
                        vis_note(ta.vsink[k], g, (int)p, home, cn, nn, tile, t0);
                    },
                    mv);
                if (dep) {
                    int mn[3], cr[3];
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        cr[d] = mv.i2[d] - mv.i1[d];
                        mn[d] = min(mv.i1[d], mv.i2[d]) - lo[d];
                        geo |= (mn[d] + 1) << (3 * d) | (cr[d] + 1) << (9 + 2 * d);
                    }
                    // at rest (as Moved::moved, which costs FP64 2 % here): dm is
                    // the new offset (FP64) or the move (FP32)
                    bool rest = !RHO && cr[0] == 0 && cr[1] == 0 && cr[2] == 0;
#pragma unroll
                    for (int d = 0; d < 3; ++d) rest = rest && mv.dm[d] == (L::F64 ? mv.d0[d] : real(0));
                    if (rest) row = -2;
                    else if (cr[1] == 0 && cr[2] == 0 && mn[0] >= 0 && mn[0] + abs(cr[0]) < T) row = mn[1] + T * mn[2];
                }
            } else if (!inside && i < mh[k] && vvalid[k]) {
                // away from home: pushed from the visitor list of the tile it is in
            } else {
                // a crowded tile, or away from home without valid visitor
                // lists: pushed by the global kernel after this one
                const unsigned long long q = atomicAdd(ta.nstrag + k, 1ull);
                ta.strag[k][2 * q] = (int)p;
                ta.strag[k][2 * q + 1] = home;
            }
        }
        // the deposit's inputs replace the particle's inputs: d0, dm, q w
        // (zeros where nothing is deposited, so that every factor is finite)
        real *fin = reinterpret_cast<real *>(row_in);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            fin[d * 32] = dep ? mv.d0[d] : real(0);
            fin[(3 + d) * 32] = dep ? mv.dm[d] : real(0);
        }
        fin[6 * 32] = dep ? mv.qw : real(0);
        if (!dep) geo = 1 << 9 | 1 << 11 | 1 << 13;

        // ---- deposit ------------------------------------------------------------
        const real *fw = reinterpret_cast<const real *>(sp_in + slot * KW * 32);
        const int p4 = lane & 3, n8 = lane >> 2;
        double Dx[P][2], Dv[P][2], Dr[RHO ? P : 1][2];
        // Jy and Jz share the matrices Dv: 4 fluxes x 5 points each, 40 rows in
        // five matrices.  Second factor of row n8 of the t-th: the z point v of
        // a Jy row (v < P), else the y point v - P of a Jz row.
        auto yz_row = [](int t, int n) { return 2 * t + (n >> 2); };
        unsigned reg = __ballot_sync(0xffffffffu, row >= 0);      // not yet summed
        const unsigned irr = __ballot_sync(0xffffffffu, dep && row == -1);
        unsigned todo = 0, sc = 0;   // of the current group of 8: to sum, to scatter
        int cur = -1, grp = -1;
#pragma unroll 1
        for (;;) {
            int next = -1;
            // the particles of row `cur`, group after group, until another row takes over
#pragma unroll 1
            for (;;) {
                if (todo == 0) {
                    // one by one: a lane per column of each component
#pragma unroll 1
                    for (; sc; sc &= sc - 1) {
                        const int l = __ffs(sc) - 1;
                        const int ge = __shfl_sync(0xffffffffu, geo, l);
                        const Pair<real> *pr = tp + (l & 7) * L::PS;
                        const real *pc = tc + (l & 7) * L::CS;
                        const int st[3] = {1, L::dsy, L::dsz};
                        const int base = (ge & 7) + ((ge >> 3) & 7) * L::dsy + ((ge >> 6) & 7) * L::dsz;
                        int len[3];
#pragma unroll
                        for (int d = 0; d < 3; ++d) len[d] = P + (((ge >> (9 + 2 * d)) & 3) != 1 ? 1 : 0);
                        FixedAcc<real, NL> af;
                        af.lstride = L::DS;
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const int u = c == 0 ? 1 : 0, v = c == 2 ? 1 : 2;
                            af.p[0] = sa + c * NL * L::DS;
#pragma unroll 1
                            for (int q = lane; q < len[u] * len[v]; q += 32) {
                                const int qv = len[u] == P ? q / P : q / Q, qu = q - qv * len[u];
                                const Pair<real> fu = pr[u * Q + qu], fv = pr[v * Q + qv];
                                const real W = fu.s * fv.s + fu.d * fv.d;
                                const int at = base + qu * st[u] + qv * st[v];
#pragma unroll
                                for (int e = 0; e < P; ++e) {
                                    if (e >= len[c] - 1) break;
                                    af.add(0, at + e * st[c], pc[c * P + e] * W);
                                }
                            }
                        }
                        if constexpr (RHO) {
                            af.p[0] = sa + (3 + k) * NL * L::DS;
#pragma unroll 1
                            for (int q = lane; q < len[1] * len[2]; q += 32) {
                                const int qv = len[1] == P ? q / P : q / Q, qu = q - qv * len[1];
                                const Pair<real> fu = pr[Q + qu], fv = pr[2 * Q + qv];
                                const real W = pc[3 * P] * (fu.s + real(kSqrt3) * fu.d) * (fv.s + real(kSqrt3) * fv.d);
                                const int at = base + qu * L::dsy + qv * L::dsz;
                                for (int e = 0; e < len[0]; ++e)
                                    af.add(0, at + e, W * (pr[e].s + real(kSqrt3) * pr[e].d));
                            }
                        }
                    }
                    do ++grp;
                    while (grp < 4 && !((reg | irr) >> (8 * grp) & 0xffu));
                    if (grp >= 4) break;
                    // the table of the next 8 particles: lane = (particle, axis)
                    __syncwarp();
                    {
                        const int src = 8 * grp + n8, axis = p4 < 3 ? p4 : 2;
                        const int cr = ((__shfl_sync(0xffffffffu, geo, src) >> (9 + 2 * axis)) & 3) - 1;
                        real s[Q], ds[Q];
                        axis_factors<real, P>(fw[axis * 32 + src], fw[(3 + axis) * 32 + src], cr, s, ds);
                        const real qw = fw[6 * 32 + src];
                        const real f = -qw * (axis == 0 ? a.d_dt[0] * ta.scale[0] : axis == 1 ? a.d_dt[1] * ta.scale[1]
                                                                                                : a.d_dt[2] * ta.scale[2]);
                        if (p4 < 3) {
                            Pair<real> *pr = tp + n8 * L::PS + axis * Q;
                            real *pc = tc + n8 * L::CS + axis * P;
                            real run = 0;
#pragma unroll
                            for (int q = 0; q <= P; ++q) pr[q] = Pair<real>{s[q], ds[q] * real(kInvSqrt12)};
#pragma unroll
                            for (int q = 0; q < P; ++q) {
                                run += ds[q];
                                // the last point of the sum of all ds (zero) is not a flux
                                pc[q] = q < P - 1 || cr != 0 ? f * run : real(0);
                            }
                        } else if (RHO) {
                            tc[n8 * L::CS + 3 * P] = qw * ta.scale[3];
                        }
                    }
                    __syncwarp();
                    todo = reg & (0xffu << (8 * grp));
                    sc = irr & (0xffu << (8 * grp));
                    continue;
                }
                unsigned sel = __ballot_sync(0xffffffffu, row == cur) & todo;
                if (!sel) {
                    const int r = __shfl_sync(0xffffffffu, row, __ffs(todo) - 1);
                    const unsigned rest = __ballot_sync(0xffffffffu, row == r) & reg;
                    const unsigned left = cur >= 0 ? __ballot_sync(0xffffffffu, row == cur) & reg : 0u;
                    const unsigned mine = rest & todo;
                    if (__popc(rest) >= 2 && __popc(rest) > __popc(left)) {
                        next = r;
                        break;
                    }
                    sc |= mine;   // alone, or a stray among another row's particles
                    todo &= ~mine;
                    reg &= ~mine;
                    continue;
                }
                todo &= ~sel;
                reg &= ~sel;
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    const unsigned s4 = sel >> (8 * grp + 4 * h) & 0xfu;
                    if (!s4) continue;
                    const bool act = s4 >> p4 & 1u;
                    const int off = (__shfl_sync(0xffffffffu, geo, 8 * grp + 4 * h + p4) & 7) - 1;
                    const Pair<real> *pr = tp + (4 * h + p4) * L::PS;
                    const real *pc = tc + (4 * h + p4) * L::CS;
                    const int ix = n8 - off;
                    Pair<real> xb{real(0), real(0)};
                    if (ix >= 0 && ix <= P) xb = pr[ix];
                    const double ax = act && ix >= 0 && ix < P ? (double)pc[ix] : 0.0;
                    // Jx: rows x, columns (j, k); rho: rows (j, k) of the same tiles, columns x
                    Pair<real> yj{real(0), real(0)};
                    if (n8 <= P) yj = pr[Q + n8];
                    real wyr = real(0), wxr = real(0);
                    if constexpr (RHO) {
                        wyr = act ? pc[3 * P] * (yj.s + real(kSqrt3) * yj.d) : real(0);
                        wxr = xb.s + real(kSqrt3) * xb.d;
                    }
#pragma unroll
                    for (int t = 0; t < P; ++t) {
                        const Pair<real> zk = pr[2 * Q + t];
                        dmma(Dx[t], ax, (double)(yj.s * zk.s + yj.d * zk.d));
                        if constexpr (RHO) dmma(Dr[t], (double)(wyr * (zk.s + real(kSqrt3) * zk.d)), (double)wxr);
                    }
                    // Jy and Jz: rows (j, k) and (k, j), columns x
                    const int f1 = n8 & 3;
                    const real cy = act ? pc[P + f1] : real(0), cz = act ? pc[2 * P + f1] : real(0);
                    const double xs = (double)xb.s, xd = (double)xb.d;
                    Pair<real> o[P];
                    real c[P];
#pragma unroll
                    for (int t = 0; t < P; ++t) {
                        const int v = yz_row(t, n8);
                        const bool z = v >= P;
                        o[t] = pr[z ? Q + v - P : 2 * Q + v];
                        c[t] = z ? cz : cy;
                        dmma(Dv[t], (double)(c[t] * o[t].s), xs);
                    }
#pragma unroll
                    for (int t = 0; t < P; ++t) dmma(Dv[t], (double)(c[t] * o[t].d), xd);
                }
            }
            // the row's sums into the shared accumulators
            if (cur >= 0) {
                const int ry = cur % T, rz = cur / T;
                unsigned *at = sa + (rz + 1) * L::dsz + (ry + 1) * L::dsy + 1;
#pragma unroll
                for (int t = 0; t < P; ++t)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        if (2 * p4 + e < P) add_limbs<NL>(at + t * L::dsz + (2 * p4 + e) * L::dsy + n8, L::DS, Dx[t][e]);
                const int f1 = n8 & 3;
#pragma unroll
                for (int t = 0; t < P; ++t) {
                    const int v = yz_row(t, n8);
                    const bool z = v >= P;
                    const int f2 = z ? v - P : v;
                    unsigned *av = at + 2 * p4 + (z ? 2 * NL * L::DS + f1 * L::dsz + f2 * L::dsy
                                                    : NL * L::DS + f2 * L::dsz + f1 * L::dsy);
                    add_limbs<NL>(av, L::DS, Dv[t][0]);
                    add_limbs<NL>(av + 1, L::DS, Dv[t][1]);
                }
                if constexpr (RHO) {
                    at += (3 + k) * NL * L::DS;
#pragma unroll
                    for (int t = 0; t < P; ++t) {
                        if (n8 >= P) break;
                        add_limbs<NL>(at + t * L::dsz + n8 * L::dsy + 2 * p4, L::DS, Dr[t][0]);
                        add_limbs<NL>(at + t * L::dsz + n8 * L::dsy + 2 * p4 + 1, L::DS, Dr[t][1]);
                    }
                }
            }
            if (next < 0) break;
            cur = next;
#pragma unroll
            for (int t = 0; t < P; ++t) {
                Dx[t][0] = Dx[t][1] = Dv[t][0] = Dv[t][1] = 0.0;
                if constexpr (RHO) Dr[t][0] = Dr[t][1] = 0.0;
            }
        }
        __syncwarp();
        slot ^= 1;
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
            const real v = (real)tot * (real)ta.inv_scale[c < 3 ? c : 3];
            if (in) atomic_add(ta.ring[c] + dst, v);
            else set_status(ta.sp[0].status, ST_OOB);
        }
    }
}

template <typename real, int P, bool SPIN>
void node_tile_push(pic_ctx *c, int mask) {
    using L = NodeTile<real, P>;
    TileGeom t{};
    t.T = c->tile;
    for (int d = 0; d < 3; ++d) t.nt[d] = c->ntile[d];
    t.nkeys = c->nkeys;
    t.nodes = 1;
    t.nacc = (c->p.deposit_rho && !c->rho_skip) ? 5 : 3;
    const TileArgs<real> ta = make_tile_args<real, P>(c, mask, t);
    const int ntiles = c->ntile[0] * c->ntile[1] * c->ntile[2];
    auto launch = [&](auto kernel) {
        const size_t smem = L::smem(t.nacc);
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kernel<<<ntiles, L::kThreads, smem, c->stream>>>(ta);
    };
    if (t.nacc == 5) launch(node_tile_kernel<real, P, SPIN, true>);
    else launch(node_tile_kernel<real, P, SPIN, false>);
}

}  // namespace

// Tiles of nodes: both orders at the default tile edge.  The matrix deposit
// here is for 4th order; measured per launch on 128 x 64 x 64 cells, 8 + 8
// particles per cell (tiles of cells with a scatter per particle first): FP64
// 7.08 -> 4.07 ms, FP32 3.72 -> 2.42 ms (in FP64 without the 1.4 % away from
// home, now in the tiles' lists: 0.25 ms).  At 2nd order the factors of its
// products cost more to make (FP32 1.23 ms) than a particle's 54 points to
// scatter (1.01 ms): tile_node_kernels.cu sums them per node instead.  Other
// edges keep the tiles of cells of tile_kernels.cu.
bool node_tiles_for(int tile, int order) { return tile == 4 && (order == 2 || order == 4); }

size_t node_tile_smem_bytes(const pic_ctx *c) {
    if (c->order == 2) return node_sum_smem_bytes(c);
    return c->fp32 ? NodeTile<float, 5>::smem(5) : NodeTile<double, 5>::smem(5);
}

void launch_node_tile_kernel(pic_ctx *c, int mask, bool spin) {
    if (c->order == 2) return launch_node_sum_kernel(c, mask, spin);
    if (c->fp32) spin ? node_tile_push<float, 5, true>(c, mask) : node_tile_push<float, 5, false>(c, mask);
    else spin ? node_tile_push<double, 5, true>(c, mask) : node_tile_push<double, 5, false>(c, mask);
}

}  // namespace pic
