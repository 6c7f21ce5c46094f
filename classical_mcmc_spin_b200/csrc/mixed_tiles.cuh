// mixed_tiles.cuh -- the mixed SU(2) / SU(3) integrator (mixed.cuh: same fields, equations
// of motion and steps) as FP64 matrix products over tiles of eight like sites, with every
// RK vector on chip.
//
// mixed_integrate_kernel gives each site one thread, which walks ~400 couplings in a
// chain, and keeps the RK vectors in global memory.  Here a warp owns a tile: eight sites
// of one kind with the same couplings in every slot (the atoms of one sublattice).  The
// field of a tile is a sum over slots of (coupling matrix) x (partners' components, one
// column per site), which is the shape of mma.m8n8k4.f64: 8x8 matrices are two, 8x3 and
// 3x3 ones one, 3x8 two instructions (SU(2) rows fill three of eight).  Matrices sit in
// shared memory in fragment order (32 doubles per k-step, lane by lane), partners are read
// straight from the stage vector.
//   * Lane l owns component l / 4 of sites 2 (l % 4) and 2 (l % 4) + 1 (the accumulator
//     layout): y, the stage derivatives and stage inputs are registers (rk_fixed.cuh's
//     steps over two elements per tile).
//   * A stage input is published in its CTA's stage vector in shared memory; after the
//     cluster barrier each CTA gathers the partners it lacks (its halo, a list made on the
//     host) through distributed shared memory.  Stage vectors alternate between two
//     buffers: one cluster barrier and one CTA barrier per stage.  SU(3) vectors lie 12
//     doubles apart, SU(2) ones 4: the 32-byte pieces four sites of a half warp read fall
//     in different banks.
//   * f_abc H_b S_c: component a takes its (at most four) pairs (b, c); H and S of the tile pass
//     through a [component][site] block of the warp, both sites of a lane in one load.
//   * Drive factors come from a table filled before the launch (mixed_factor_kernel):
//     evaluated in the kernel, their exp and cos cost each warp more than its field sums.
//
// Bound: a stage's exchange and matrix products, in turn.  864 + 864 sites on a 16-CTA cluster: the halo (about 1200
// 16-byte pieces a CTA; the network takes a warp's request in ~17 cycles whatever its width, so pieces of 8 bytes
// cost twice) and the cluster barrier ~1700 cycles, 20 products of 16 cycles for each of a scheduler's four tiles
// 1300.  B200: 2.7 us per SSPRK53 stage (12.3 with one thread per site; 3.4 with 8-byte pieces, 4.1 exchanging
// through L2, 4.7 with eight lanes per site and plain FMAs): 400 steps 5.47 ms instead of 24.7.
#pragma once

#include "mixed.cuh"

namespace cmd {

constexpr int kTileSites = 8;
constexpr int kTileStride2 = 4, kTileStride3 = 12;   // doubles between the sites of a kind in the stage vector

struct MixedTilesDev {
    const double* tab;         // [fragments][32] coupling fragments, then the field vectors; copied to shared memory
    int tab_doubles;
    const int* ints;           // [cs][int_stride] int block of each CTA, copied to shared memory
    int int_stride;
    int tiles;                 // per CTA; tile w + q * warps belongs to warp w
    int slots;                 // records per tile
    int vec;                   // doubles of the stage vector (own sites, halo, a zero vector)
    int halo_max;
    int N2, N3, NA2, NA3;
    int driven2, driven3;
    const double* drive2;      // [2][NA2][3]
    const double* drive3;      // [2][NA3][8]
    const double2* factors;    // [n_steps * stages][2]: (pulse 1, pulse 2) of SU(2), of SU(3)
};
constexpr int kTileRegs = 8;                         // records of each sort a one-tile warp keeps in registers
constexpr int kHaloRegs = 3;                         // halo entries a thread keeps in registers

// Int block of a CTA: {halo entries, 0}; per tile {kind, slots with 8-component partners, slots with 3-component
// partners, field offset}; sites [tiles][8] (-1: none); own stage-vector offsets [tiles][8]; records
// [slots][tiles][8] (fragment / 32) << 16 | partner's stage-vector offset; {owner << 16 | its offset, offset here} of
// the halo's 16-byte pieces.
struct MixedTilesLayout {
    int tile, site, own, part, halo, total;
};
__host__ __device__ inline MixedTilesLayout mixed_tiles_layout(int tiles, int slots, int halo_max) {
    MixedTilesLayout l{};
    l.tile = 2;
    l.site = l.tile + 4 * tiles;
    l.own = l.site + 8 * tiles;
    l.part = l.own + 8 * tiles;
    l.halo = (l.part + 8 * slots * tiles + 1) / 2 * 2;
    l.total = (l.halo + 2 * halo_max + 3) / 4 * 4;
    return l;
}
__host__ __device__ inline long long mixed_tiles_smem(const MixedTilesDev& m) {
    return ((long long)m.tab_doubles + 2LL * m.vec + 16 * 128) * 8 + (long long)m.int_stride * 4;
}

// Stage times c_j of each method in call order (rk_fixed.cuh); the drive table holds t_n + c_j dt.
__host__ __device__ constexpr int mixed_stages(int mode) {
    return mode == kModeEuler ? 1 : mode == kModeMidpoint ? 2 : mode == kModeRK4 ? 4 : mode == kModeSSPRK53 ? 5
         : mode == kModeRK78 ? 11 : 6;
}
struct MixedStageTimes {
    int n;
    double c[11];
};

// out[(n * stages + j)][4]: drive factors (SU(2) pulse 1, 2, SU(3) pulse 1, 2) at times[n] + c_j dt.
static __global__ void mixed_factor_kernel(const __grid_constant__ MixedDev m, const double* __restrict__ times,
                                           long long n_steps, double dt, const __grid_constant__ MixedStageTimes s,
                                           double* __restrict__ out) {
    const long long total = n_steps * s.n * 4;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int q = (int)(e & 3);
        const long long st = e >> 2, n = st / s.n;
        const double ts = times[n] + s.c[st - n * s.n] * dt;
        out[e] = q == 0   ? drive_factor(m.amp2, ts - m.t1_2, m.width2, m.freq2)
                 : q == 1 ? drive_factor(m.amp2, ts - m.t2_2, m.width2, m.freq2)
                 : q == 2 ? drive_factor(m.amp3, ts - m.t1_3, m.width3, m.freq3)
                          : drive_factor(m.amp3, ts - m.t2_3, m.width3, m.freq3);
    }
}

// Component a's pairs (b, c) with f_abc (from su3_cross's nine constants, cyclic): b, c, and the coefficient.
struct Su3Pairs {
    unsigned char b[8][4], c[8][4];
    double f[8][4];
};
constexpr Su3Pairs make_su3_pairs() {
    constexpr double h = 0.5, q = 0.86602540378443864676;
    constexpr int T[9][3] = {{0, 1, 2}, {0, 3, 6}, {0, 4, 5}, {1, 3, 5}, {1, 4, 6},
                             {2, 3, 4}, {2, 5, 6}, {3, 4, 7}, {5, 6, 7}};
    constexpr double F[9] = {1.0, h, -h, h, h, h, -h, q, q};
    Su3Pairs p{};
    int n[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int t = 0; t < 9; ++t)
        for (int r = 0; r < 3; ++r) {
            const int a = T[t][r], k = n[a]++;
            p.b[a][k] = (unsigned char)T[t][(r + 1) % 3];
            p.c[a][k] = (unsigned char)T[t][(r + 2) % 3];
            p.f[a][k] = F[t];
        }
    return p;
}
static __constant__ Su3Pairs kSu3Pairs = make_su3_pairs();

// d += a b: one k-step of an 8x8 product (row-major a, lane (row l / 4, k l % 4); b (k l % 4, column l / 4);
// d (row l / 4, columns 2 (l % 4), + 1)).
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ double ld_shared(uint32_t addr) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ double2 ld_shared2(uint32_t addr) {
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_shared2(uint32_t addr, double x, double y) {
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(x), "d"(y) : "memory");
}
__device__ __forceinline__ double2 ld_cluster2(uint32_t addr) {
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(addr) : "memory");
    return v;
}

// The elements a lane owns: two per tile.
template <class R, int NE>
struct TilesStepCtx {
    const R& rhs_f;
    __device__ __forceinline__ void rhs(double* Y, double* K, double) const { rhs_f(Y, K); }
    template <class F>
    __device__ __forceinline__ void each(F&& f) const {
#pragma unroll
        for (int q = 0; q < NE; ++q) f(q);
    }
    __device__ __forceinline__ void sync() const {}      // every vector is private; rhs synchronises the stage input
};

// MODE: rk_fixed.cuh mode (not Bulirsch-Stoer).  TPW: tiles per warp.
template <int MODE, int TPW>
__global__ void __launch_bounds__(512, 1)
mixed_tiles_kernel(const __grid_constant__ MixedTilesDev m, const __grid_constant__ MixedRun r) {
    constexpr int NE = 2 * TPW;
    extern __shared__ double2 tiles_smem[];
    double* tab = reinterpret_cast<double*>(tiles_smem);
    double* vecs = tab + m.tab_doubles;                               // [2][vec]
    double* hs_all = vecs + 2 * m.vec;                                // [16 warps][2][8][8]: a tile's H and S
    int* ib = reinterpret_cast<int*>(hs_all + 16 * 128);
    const MixedTilesLayout L = mixed_tiles_layout(m.tiles, m.slots, m.halo_max);
    unsigned rank, cs;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(cs));
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int a = lane >> 2, kc = lane & 3;                           // component owned (also column read); k-step row
    for (int i = tid; i < m.tab_doubles; i += nt) tab[i] = m.tab[i];
    for (int i = tid; i < 2 * m.vec; i += nt) vecs[i] = 0.0;
    for (int i = tid; i < m.int_stride; i += nt) ib[i] = m.ints[(long long)rank * m.int_stride + i];
    __syncthreads();
    const int n_halo = ib[0];
    const int2* halo = reinterpret_cast<const int2*>(ib + L.halo);
    const long long V = 3LL * m.N2 + 8LL * m.N3;

    int own[NE], vi[NE];                             // stage-vector offset of the element's site; state index
    bool live[NE], su3[TPW];
    double d1[TPW], d2[TPW];
#pragma unroll
    for (int q = 0; q < TPW; ++q) {
        const int t = warp + q * (nt / 32);
        su3[q] = t < m.tiles && ib[L.tile + 4 * t] == 3;
        d1[q] = d2[q] = 0.0;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int n = 2 * kc + e;                // site of the tile
            const int s = t < m.tiles ? ib[L.site + 8 * t + n] : -1;
            own[2 * q + e] = t < m.tiles ? ib[L.own + 8 * t + n] : m.vec - kTileStride3;
            live[2 * q + e] = s >= 0 && (su3[q] || a < 3);
            vi[2 * q + e] = su3[q] ? 3 * m.N2 + 8 * s + a : 3 * s + a;
            if (live[2 * q + e]) {                   // the tile's sites are one atom of the cell
                if (su3[q] && m.driven3) {
                    d1[q] = m.drive3[8 * (s % m.NA3) + a];
                    d2[q] = m.drive3[8 * (m.NA3 + s % m.NA3) + a];
                } else if (!su3[q] && m.driven2) {
                    d1[q] = m.drive2[3 * (s % m.NA2) + a];
                    d2[q] = m.drive2[3 * (m.NA2 + s % m.NA2) + a];
                }
            }
        }
        d1[q] = __shfl_sync(0xffffffffu, d1[q], a * 4);               // column 0 is never padding
        d2[q] = __shfl_sync(0xffffffffu, d2[q], a * 4);
    }
    const bool driven = m.driven2 || m.driven3;
    int buf = 0;
    long long stage = 0;
    // shared-memory addresses of the tile's first records, 8-component and 3-component partners apart: fragment
    // (this lane's word) and partner (this lane's k-step row, buffer 0); and this thread's first halo entries
    // (shared::cluster source, local destination)
    constexpr int RR = TPW == 1 ? kTileRegs : 0;
    uint32_t ra[2][RR > 0 ? RR : 1], rp[2][RR > 0 ? RR : 1];
    const uint32_t tab0 = (uint32_t)__cvta_generic_to_shared(tab);
    const uint32_t vec0 = (uint32_t)__cvta_generic_to_shared(vecs);
    auto record = [&](int n, int t, uint32_t& fa, uint32_t& pa) {
        const int w = ib[L.part + 8 * (n * m.tiles + t) + a];
        fa = tab0 + 8u * (32 * (w >> 16) + lane);
        pa = vec0 + 8u * ((w & 0xffff) + kc);
    };
#pragma unroll
    for (int n = 0; n < RR; ++n) {
        ra[0][n] = ra[1][n] = tab0 + 8u * (m.tab_doubles - 64 + lane);    // none: a zero fragment, the zero vector
        rp[0][n] = rp[1][n] = vec0 + 8u * (m.vec - kTileStride3 + kc);
        if (warp < m.tiles) {
            const int n8 = ib[L.tile + 4 * warp + 1], n3 = ib[L.tile + 4 * warp + 2];
            if (n < n8) record(n, warp, ra[0][n], rp[0][n]);
            if (n < n3) record(n8 + n, warp, ra[1][n], rp[1][n]);
        }
    }
    // f_abc H_b S_c: byte offsets of H_b and H_c (both of this lane's sites) in the warp's [8][8] block; S follows it
    const uint32_t blk = (uint32_t)__cvta_generic_to_shared(hs_all + 128 * warp);
    uint32_t ob[TPW][4], oc[TPW][4];
    double fc[TPW][4];
#pragma unroll
    for (int q = 0; q < TPW; ++q)
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const int b = su3[q] ? kSu3Pairs.b[a][p] : (a + 1) % 3, c = su3[q] ? kSu3Pairs.c[a][p] : (a + 2) % 3;
            ob[q][p] = blk + 64 * b + 16 * kc;
            oc[q][p] = blk + 64 * c + 16 * kc;
            fc[q][p] = su3[q] ? kSu3Pairs.f[a][p] : 1.0;
        }
    auto halo_at = [&](int e, uint32_t& src, int& dst) {
        const int2 h = halo[e];
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(src) : "r"(vec0 + 8u * (h.x & 0xffff)), "r"(h.x >> 16));
        dst = h.y;
    };
    uint32_t hs[kHaloRegs];
    int hd[kHaloRegs];
#pragma unroll
    for (int i = 0; i < kHaloRegs; ++i) {
        hs[i] = vec0 + 8u * (m.vec - kTileStride3);
        asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(hs[i]) : "r"(rank));
        hd[i] = m.vec - kTileStride3;
        if (tid + i * nt < n_halo) halo_at(tid + i * nt, hs[i], hd[i]);
    }
    if (cs > 1)                                      // every CTA of the cluster runs before its memory is read
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");

    auto rhs = [&](const double* Y, double* K) __attribute__((always_inline)) {
        double* vec = vecs + buf * m.vec;
        const uint32_t shift = 8u * (uint32_t)(buf * m.vec);
        buf ^= 1;
        double2 f[TPW];
#pragma unroll
        for (int q = 0; q < TPW; ++q)
            f[q] = driven ? m.factors[2 * stage + (su3[q] ? 1 : 0)] : make_double2(0.0, 0.0);
        ++stage;
#pragma unroll
        for (int i = 0; i < NE; ++i)
            if (live[i]) vec[own[i] + a] = Y[i];
        if (cs > 1) {
            asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
            double2 v[kHaloRegs];
#pragma unroll
            for (int i = 0; i < kHaloRegs; ++i) v[i] = ld_cluster2(hs[i] + shift);    // none: own zero vector, onto itself
#pragma unroll
            for (int i = 0; i < kHaloRegs; ++i) *reinterpret_cast<double2*>(vec + hd[i]) = v[i];
            for (int e = tid + kHaloRegs * nt; e < n_halo; e += nt) {
                uint32_t src;
                int dst;
                halo_at(e, src, dst);
                *reinterpret_cast<double2*>(vec + dst) = ld_cluster2(src + shift);
            }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < TPW; ++q) {
            const int t = warp + q * (nt / 32);
            if (t >= m.tiles) {
                K[2 * q] = K[2 * q + 1] = 0.0;
                continue;
            }
            const int n8 = ib[L.tile + 4 * t + 1], n3 = ib[L.tile + 4 * t + 2];
            const double c0 = su3[q] || a < 3 ? -tab[ib[L.tile + 4 * t + 3] + a] : 0.0;
            double acc[2][2] = {{c0, c0}, {0.0, 0.0}};
            // four records at a time: their loads first, then the products
#pragma unroll
            for (int n = 0; n < RR; n += 4) {
                if (n >= n8) break;
                double fa[4][2], pv[4][2];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t pa = rp[0][n + i] + shift;
                    fa[i][0] = ld_shared(ra[0][n + i]);
                    pv[i][0] = ld_shared(pa);
                    fa[i][1] = ld_shared(ra[0][n + i] + 256);
                    pv[i][1] = ld_shared(pa + 32);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    mma_f64(acc[0], fa[i][0], pv[i][0]);
                    mma_f64(acc[1], fa[i][1], pv[i][1]);
                }
            }
#pragma unroll
            for (int n = 0; n < RR; n += 4) {
                if (n >= n3) break;
                double fa[4], pv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    fa[i] = ld_shared(ra[1][n + i]);
                    pv[i] = ld_shared(rp[1][n + i] + shift);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) mma_f64(acc[i & 1], fa[i], pv[i]);
            }
            for (int n = RR; n < n8; ++n) {
                uint32_t fa, pa;
                record(n, t, fa, pa);
                mma_f64(acc[0], ld_shared(fa), ld_shared(pa + shift));
                mma_f64(acc[1], ld_shared(fa + 256), ld_shared(pa + shift + 32));
            }
            for (int n = n8 + RR; n < n8 + n3; ++n) {
                uint32_t fa, pa;
                record(n, t, fa, pa);
                mma_f64(acc[0], ld_shared(fa), ld_shared(pa + shift));
            }
            const double d = f[q].x * d1[q] + f[q].y * d2[q];
            // H and S of the tile, [component][site], for the products below
            __syncwarp();
            st_shared2(blk + 64 * a + 16 * kc, acc[0][0] + acc[1][0] - d, acc[0][1] + acc[1][1] - d);
            st_shared2(blk + 512 + 64 * a + 16 * kc, Y[2 * q], Y[2 * q + 1]);
            __syncwarp();
            double k0 = 0.0, k1 = 0.0;
            auto pair = [&](int p) __attribute__((always_inline)) {
                const double2 hb = ld_shared2(ob[q][p]), hc = ld_shared2(oc[q][p]);
                const double2 sb = ld_shared2(ob[q][p] + 512), sc = ld_shared2(oc[q][p] + 512);
                k0 = fma(fc[q][p], hb.x * sc.x - hc.x * sb.x, k0);
                k1 = fma(fc[q][p], hb.y * sc.y - hc.y * sb.y, k1);
            };
            pair(0);
            if (su3[q]) {
                pair(1);
                pair(2);
                pair(3);
            }
            K[2 * q] = k0;
            K[2 * q + 1] = k1;
        }
    };
    const TilesStepCtx<decltype(rhs), NE> ctx{rhs};

    double y[NE], kk[7][NE], Ya[NE], Yb[NE], yn[NE];
    double* k[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) k[i] = kk[i];
#pragma unroll
    for (int i = 0; i < NE; ++i) y[i] = live[i] ? r.y0[vi[i]] : 0.0;
    long long row = 0, save_left = 0;
    auto save = [&]() {
        if (r.rows && row < r.max_rows)
#pragma unroll
            for (int i = 0; i < NE; ++i)
                if (live[i]) r.rows[row * V + vi[i]] = y[i];
        ++row;
    };
    for (long long step = 0; step < r.n_steps; ++step) {
        const bool obs = save_left == 0;
        save_left = obs ? r.save_every - 1 : save_left - 1;
        if (obs) save();
        rhs(y, k[0]);
        fixed_step<true>(MODE, ctx, y, k, Ya, Yb, yn, 0.0, r.dt);
    }
    save();
#pragma unroll
    for (int i = 0; i < NE; ++i)
        if (live[i]) r.y_out[vi[i]] = y[i];
    if (cs > 1)                                      // no CTA leaves while others may read its stage vector
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace cmd
