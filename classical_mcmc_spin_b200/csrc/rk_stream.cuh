// rk_stream.cuh -- RK4 and its discrete adjoint for lattices too large for a
// resident CTA (e.g. the 65536-spin conventional-cubic pyrochlore), with state
// streamed through L2 / HBM.
//
// Every RK4 stage is ONE launch over a (cell tile, trajectory) grid; each
// thread advances one site (cell, atom) with rk4_stage_site, the atom uniform
// per warp, so all SMs work on every trajectory and the kernel boundary is the
// only barrier between stages (no device-side waits anywhere).  The adjoint
// uses the same launches for its segment recompute and one stream_vjp_kernel
// launch per stage for the reverse sweep (one site per thread).
//
// Vectors are blocked by tiles of CP = 256 / NAT cells, v[((g / CP)*NAT*3 + atom*3 + c)*CP
// + g % CP] (soff), the last tile padded, trajectory b at p + b*stride (SVec): a site's
// components and its in-cell partners lie at compile-time distances, which takes most of
// the index arithmetic out of the stages (with one row of G cells per component, 140 of a
// warp's 410 instructions), and a tile is one contiguous piece.  Per stage a cell reads its
// stage input (own and partners'), y and the RK4 sum, and writes the sum and the next stage
// input: per spin 72 B (stage 0: y in, sum and next input out), 120 B (stages 1, 2) and
// 96 B (stage 3: y written in place), 408 B per spin-step when the partners' reads hit in
// cache.
//
// Bound: latency of a short-lived CTA (partner offset, partner spins, store: two dependent
// trips to L2) at 32 warps an SM; DRAM carries little once a group of trajectories fits L2.
// B200, 65536-spin pyrochlore: 32 trajectories x 300 steps 46.7-47.4 ms (70.8 with rows of G cells,
// one launch group, cell-major offsets and one kernel for all stages) = 5.4-5.5 TB/s of those
// 408 B; groups of a share of L2: 0.3 75.6, 0.4 69.3, 0.55-0.7 64.4, 0.9 68.4, all at once
// 70.0 ms (before the blocked layout).  Adjoint of 8 x 100 steps 24.1 ms (34.3: a cell per
// thread, each partner's Hbar formed per bond from three vectors, couplings indexed at run
// time); a VJP stage takes about 36 us.
//
// Observables, in a fixed summation order without atomics: the stage-0 launch
// of step n leaves one partial per (trajectory, tile) (spin sums per atom class
// and the energy), and the first CTA of each trajectory in the stage-1 launch
// of the same step sums them over the tiles in a fixed order.  That CTA writes the
// raw row (as rk4_resident's rows: finished by finish_rows_kernel) and/or the
// M_local loss terms.  The state after the last step is summed by
// stream_obs_kernel + stream_reduce_kernel.
#pragma once

#include "rk_adjoint.cuh"

namespace cmd {

constexpr int kStreamTile = 256;     // threads of a CTA (one site each)
constexpr int kPart = 16;            // doubles per partial slot

struct SVec {
    double* p;
    long long stride;                // doubles between trajectories
    __device__ __forceinline__ double* at(int b) const { return p ? p + (long long)b * stride : nullptr; }
};

struct StreamArgs {
    int G;                           // cells per trajectory
    int tiles;                       // ceil(G / stream_cells<NAT>())
    int B;
    const int* nbr;                  // [NAT][Z-LZ][G] partner offsets, cell-minor: a warp's loads are consecutive
    double dt;
    long long n_steps;
    const double* times;             // [n_steps + 1] accumulated t_n
    const double* drive;             // [B][n_steps][6] envelope factors (drive_table_kernel) or null
    double* part;                    // [B][tiles][kPart]
    // raw rows [B][rows][raw_stride] (3*NAT spin sums + energy), or null
    double* raw;
    long long raw_stride, save_every, rows;
    // M_local loss: target / mloc [B][n_steps+1][3], loss [B], or null
    const double* target;
    double* mloc;
    double* loss;
    double n_sites;
    // checkpoints [B][n_ckpt][V] every ckpt_every steps, or null
    double* ckpt;
    long long ckpt_every, n_ckpt, V;
    // step base added to every stage launch's step argument, or null (base 0):
    // a replayed launch sequence (CUDA graph) advances it on the device
    const long long* nbase;
    int b0;                          // first trajectory of the launch (blockIdx.y counts from it)
};

// Threads of a CTA: NAT groups of kStreamTile/NAT consecutive threads, group
// a advancing atom a of the CTA's kStreamTile/NAT cells (the atom is uniform
// per warp for NAT in {1, 2, 4, 8}).
template <int NAT>
constexpr int stream_cells() { return kStreamTile / NAT; }

// Offset of component 0 of site (cell g, atom at) in a vector; component c is c * stream_cells<NAT>() further.
template <int NAT>
__host__ __device__ __forceinline__ int soff(int g, int at) {
    constexpr int CP = stream_cells<NAT>();
    return g / CP * (NAT * 3 * CP) + at * 3 * CP + g % CP;
}

template <int NAT>
__device__ __forceinline__ void stream_site(int& at, int& g) {
    constexpr int CPT = stream_cells<NAT>();
    at = (int)threadIdx.x / CPT;
    g = (int)blockIdx.x * CPT + ((int)threadIdx.x - at * CPT);
}

// rk4_stage_cell for site (cell g, atom AT) alone.  Every load comes before
// the first store (acc / Ynext may alias y), so a thread's loads are all in
// flight together.
// PAIR: bonds are paired (Layout::paired; nbr in that order), so J_n (S_local + S_far) stands for both.
template <int NAT, int Z, int LZ, int AT, int OBS, bool PAIR>
__device__ __forceinline__ void rk4_stage_site(const Couplings<NAT, Z>& cp, const int* __restrict__ nbr, int G,
                                               int g, double dt, int s, const double* __restrict__ Yin,
                                               const double* y, double* acc, double* Ynext, double f1, double f2,
                                               bool drive, double* obs) {
    constexpr int NL = Z - LZ;
    constexpr int CP = stream_cells<NAT>();
    const int i0 = soff<NAT>(g, AT);
    double S[3], yv[3], av[3], H[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) S[c] = Yin[i0 + c * CP];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        yv[c] = s == 0 ? S[c] : y[i0 + c * CP];
        av[c] = (s == 0 || !acc) ? 0.0 : acc[i0 + c * CP];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) H[d] = cp.has_field ? -cp.field[AT][d] : 0.0;
    if (cp.has_onsite) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            bond_acc(H[d], 2.0 * cp.onsite[AT][3 * d], 2.0 * cp.onsite[AT][3 * d + 1], 2.0 * cp.onsite[AT][3 * d + 2], S[0], S[1], S[2]);
        }
    }
#pragma unroll
    for (int n = 0; n < LZ; ++n) {
        const int ip = i0 + ((AT + 1 + n) % NAT - AT) * 3 * CP;
        double P0 = Yin[ip], P1 = Yin[ip + CP], P2 = Yin[ip + 2 * CP];
        if constexpr (PAIR) {
            const int p = nbr[(AT * NL + n) * G + g];
            P0 += Yin[p];
            P1 += Yin[p + CP];
            P2 += Yin[p + 2 * CP];
        }
#pragma unroll
        for (int d = 0; d < 3; ++d)
            bond_acc(H[d], cp.J[AT][n][3 * d], cp.J[AT][n][3 * d + 1], cp.J[AT][n][3 * d + 2], P0, P1, P2);
    }
#pragma unroll
    for (int m = 0; m < (PAIR ? 0 : NL); ++m) {
        const int n = LZ + m;
        if (n < cp.zc[AT]) {
            const int p = nbr[(AT * NL + m) * G + g];
            const double P0 = Yin[p], P1 = Yin[p + CP], P2 = Yin[p + 2 * CP];
#pragma unroll
            for (int d = 0; d < 3; ++d)
                bond_acc(H[d], cp.J[AT][n][3 * d], cp.J[AT][n][3 * d + 1], cp.J[AT][n][3 * d + 2], P0, P1, P2);
        }
    }
    if (OBS == 2) {
#pragma unroll
        for (int c = 0; c < 3; ++c) obs[c] = S[c];
#pragma unroll
        for (int d = 0; d < 3; ++d) obs[3] += S[d] * (H[d] - (cp.has_field ? cp.field[AT][d] : 0.0));
    }
    if (drive) {
#pragma unroll
        for (int d = 0; d < 3; ++d) drive_acc(H[d], cp.d1[AT][d], cp.d2[AT][d], f1, f2);
    }
    const double k[3] = {H[1] * S[2] - H[2] * S[1], H[2] * S[0] - H[0] * S[2], H[0] * S[1] - H[1] * S[0]};
    const double cy = s == 2 ? dt : 0.5 * dt;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int i = i0 + c * CP;
        if (s == 0) {
            acc[i] = k[c];
            Ynext[i] = 1.0 * yv[c] + cy * k[c];
        } else if (s < 3) {
            acc[i] = av[c] + 2.0 * k[c];
            Ynext[i] = 1.0 * yv[c] + cy * k[c];
        } else if (Ynext) {
            Ynext[i] = yv[c] + (dt / 6.0) * (av[c] + k[c]);
        }
    }
}

// Envelope factors of trajectory b for stage s of step n.
__device__ __forceinline__ void stream_drive(const StreamArgs& a, int b, long long n, int s, double& f1,
                                             double& f2) {
    if (!a.drive) {
        f1 = f2 = 0.0;
        return;
    }
    const int q = s == 0 ? 0 : (s < 3 ? 2 : 4);
    const double* d = a.drive + ((long long)b * a.n_steps + n) * 6 + q;
    f1 = d[0];
    f2 = d[1];
}

// Sums the tile partials of step n of trajectory b and writes its raw row
// and / or loss terms.  Called by a whole CTA: warp w sums values w, w+nwarps,
// ...; lane l adds tiles l, l+32, ... in order, then a fixed butterfly adds
// the lanes, so the order never depends on timing.
template <int NAT>
__device__ void stream_reduce(const StreamArgs& a, int b, long long n, double* sh) {
    constexpr int NR = 3 * NAT + 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const double* p = a.part + (long long)b * a.tiles * kPart;
    for (int q = warp; q < NR; q += nw) {
        double s = 0.0;
        for (int t = lane; t < a.tiles; t += 32) s += p[(long long)t * kPart + q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) sh[q] = s;
    }
    __syncthreads();
    if (a.raw && tid < NR) {
        long long r = -1;
        if (n % a.save_every == 0) r = n / a.save_every;
        else if (n == a.n_steps) r = a.rows - 1;
        if (r >= 0) a.raw[((long long)b * a.rows + r) * a.raw_stride + tid] = sh[tid];
    }
    if (a.mloc && tid == 0) {
        double l = 0.0;
        for (int c = 0; c < 3; ++c) {
            double m = 0.0;
            for (int at = 0; at < NAT; ++at) m += sh[3 * at + c];
            m /= a.n_sites;
            const long long i = ((long long)b * (a.n_steps + 1) + n) * 3 + c;
            a.mloc[i] = m;
            const double r = m - a.target[i];
            l += r * r;
        }
        a.loss[b] = (n == 0 ? 0.0 : a.loss[b]) + l;
    }
    __syncthreads();
}

// Block sum of v[0..used) in a fixed order (lanes by the butterfly, then the
// warps in order), finished in parallel: thread q < used gets the total of
// value q and returns it in *out (other threads: false).
template <int NV>
__device__ __forceinline__ bool block_sum_par(double (&v)[NV], double* red, int used, double* out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const double r = warp_reduce_many<NV>(v);
    constexpr int span = 32 / NV;
    if ((lane % span) == 0) red[warp * kRedStride + lane / span] = r;
    __syncthreads();
    if ((int)threadIdx.x >= used) return false;
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += red[w * kRedStride + threadIdx.x];
    *out = s;
    return true;
}

// Block sums of a site's spin and energy term o[4] (zeros past the last cell), stored in the tile's slot: a warp's
// sites are one atom, so four values are reduced per warp; value q < 3 NAT adds the warps of its atom, the last one
// all of them, in warp order.
template <int NAT>
__device__ __forceinline__ void stream_store_partial(const StreamArgs& a, int b, double (&o)[4], double* red) {
    constexpr int NW = kStreamTile / 32, WA = NW / NAT;
    static_assert(WA >= 1, "an atom fills a warp");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double r = warp_reduce_many<4>(o);
    if ((lane & 7) == 0) red[warp * 4 + (lane >> 3)] = r;
    __syncthreads();
    if (tid > 3 * NAT) return;
    double t = 0.0;
    if (tid < 3 * NAT) {
#pragma unroll
        for (int w = 0; w < WA; ++w) t += red[(tid / 3 * WA + w) * 4 + tid % 3];
    } else {
#pragma unroll
        for (int w = 0; w < NW; ++w) t += red[w * 4 + 3];
    }
    a.part[((long long)b * a.tiles + blockIdx.x) * kPart + tid] = t;
}

// One RK4 stage s of step n for every (tile, trajectory).  Stage 0 also leaves
// the observables' partials of Yin (= y_n) and the checkpoint of y_n; the
// first tile of stage 1 finishes step n's observables.
// The stage is a template parameter: one kernel for all four carries their code for every
// atom, and waits for instructions (1.8 of 17 cycles an issue).
template <int NAT, int Z, int LZ, bool PAIR, int s, bool with_obs>
__global__ void __launch_bounds__(kStreamTile, 4)
stream_stage_kernel(const __grid_constant__ Couplings<NAT, Z> cp, const __grid_constant__ StreamArgs a, long long n_arg,
                    SVec Yin, SVec y, SVec acc, SVec Ynext) {
    const long long n = (a.nbase ? *a.nbase : 0) + n_arg;
    __shared__ double red[kStreamTile / 8];
    __shared__ double tot[16];
    const int b = a.b0 + blockIdx.y;
    int at, g;
    stream_site<NAT>(at, g);
    if (s == 1 && with_obs && blockIdx.x == 0) stream_reduce<NAT>(a, b, n, tot);
    double f1, f2;
    stream_drive(a, b, n, s, f1, f2);
    const bool drive = a.drive != nullptr && (f1 != 0.0 || f2 != 0.0);
    double o[4] = {0.0, 0.0, 0.0, 0.0};
    if (g < a.G) {
        const double* yin = Yin.at(b);
        with_atom<NAT>(at, [&](auto tag) {
            constexpr int AT = decltype(tag)::value;
            if (s == 0 && with_obs)
                rk4_stage_site<NAT, Z, LZ, AT, 2, PAIR>(cp, a.nbr, a.G, g, a.dt, s, yin, y.at(b), acc.at(b), Ynext.at(b),
                                                  f1, f2, drive, o);
            else
                rk4_stage_site<NAT, Z, LZ, AT, 0, PAIR>(cp, a.nbr, a.G, g, a.dt, s, yin, y.at(b), acc.at(b), Ynext.at(b),
                                                  f1, f2, drive, nullptr);
            if (s == 0 && a.ckpt && n % a.ckpt_every == 0) {
                double* dst = a.ckpt + ((long long)b * a.n_ckpt + n / a.ckpt_every) * a.V;
#pragma unroll
                for (int c = 0; c < 3; ++c) dst[soff<NAT>(g, AT) + c * stream_cells<NAT>()] = yin[soff<NAT>(g, AT) + c * stream_cells<NAT>()];
            }
        });
    }
    if (s == 0 && with_obs) stream_store_partial<NAT>(a, b, o, red);
}

// Advances the step base of a replayed launch sequence by k steps.
static __global__ void stream_advance_kernel(long long* nbase, long long k) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *nbase += k;
}

// Sets the step base of a replayed launch sequence.
static __global__ void stream_set_base_kernel(long long* nbase, long long v) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *nbase = v;
}

// Observables' partials of y (the state after the last step).
template <int NAT, int Z, int LZ, bool PAIR>
__global__ void __launch_bounds__(kStreamTile)
stream_obs_kernel(const __grid_constant__ Couplings<NAT, Z> cp, const __grid_constant__ StreamArgs a, SVec y) {
    __shared__ double red[kStreamTile / 8];
    const int b = a.b0 + blockIdx.y;
    int at, g;
    stream_site<NAT>(at, g);
    double o[4] = {0.0, 0.0, 0.0, 0.0};
    if (g < a.G) {
        // a stage-3 pass with no output: only the observables of y are kept
        with_atom<NAT>(at, [&](auto tag) {
            rk4_stage_site<NAT, Z, LZ, decltype(tag)::value, 2, PAIR>(cp, a.nbr, a.G, g, a.dt, 3, y.at(b), y.at(b), nullptr,
                                                                nullptr, 0.0, 0.0, false, o);
        });
    }
    stream_store_partial<NAT>(a, b, o, red);
}

// Finishes step n's observables (one CTA per trajectory).
template <int NAT>
__global__ void __launch_bounds__(kStreamTile) stream_reduce_kernel(const __grid_constant__ StreamArgs a, long long n) {
    __shared__ double sh[16];
    stream_reduce<NAT>(a, blockIdx.x, n, sh);
}

// AoS state [B][N][3] (site = cell*NAT + atom; y0_stride doubles between
// trajectories, 0 = shared) -> SoA vector, and back.
template <int NAT>
__global__ void stream_load_kernel(const double* __restrict__ y0, long long y0_stride, int G, SVec y) {
    const int b = blockIdx.y;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G) return;
    const double* src = y0 + (long long)b * y0_stride;
    double* dst = y.at(b);
#pragma unroll
    for (int at = 0; at < NAT; ++at)
#pragma unroll
        for (int c = 0; c < 3; ++c) dst[soff<NAT>(g, at) + c * stream_cells<NAT>()] = src[((long long)g * NAT + at) * 3 + c];
}

template <int NAT>
__global__ void stream_store_kernel(SVec y, int G, double* __restrict__ out) {
    const int b = blockIdx.y;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G) return;
    const double* src = y.at(b);
    double* dst = out + (long long)b * G * NAT * 3;
#pragma unroll
    for (int at = 0; at < NAT; ++at)
#pragma unroll
        for (int c = 0; c < 3; ++c) dst[((long long)g * NAT + at) * 3 + c] = src[soff<NAT>(g, at) + c * stream_cells<NAT>()];
}

// ---------------------------------------------------------------------------
// Adjoint sweep.

struct StreamVjpArgs {
    int G, tiles;                    // as StreamArgs
    const int* nbr;
    double dt;
    long long n_steps;
    const double* drive;             // as StreamArgs::drive
    const double* target;            // [B][n_steps+1][3]
    const double* mloc;              // [B][n_steps+1][3]
    double n_sites;
    double* gpart;                   // [B][tiles][kPart] gradient partials (accumulated)
    const long long* nbase;          // step base of a replayed launch sequence (step = *nbase + n), or nullptr
};

// lam_b = dl_S (the loss cotangent of the last state) on every site.
template <int NAT>
__global__ void stream_lam_init_kernel(const __grid_constant__ StreamVjpArgs a, SVec lam) {
    const int b = blockIdx.y;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= a.G) return;
    const long long i = ((long long)b * (a.n_steps + 1) + a.n_steps) * 3;
    double* l = lam.at(b);
#pragma unroll
    for (int at = 0; at < NAT; ++at)
#pragma unroll
        for (int c = 0; c < 3; ++c)
            l[soff<NAT>(g, at) + c * stream_cells<NAT>()] = 2.0 * (a.mloc[i + c] - a.target[i + c]) / a.n_sites;
}

// Hbar of the first VJP stage of a segment: hb = Y x (c lam) of every site.
template <int NAT>
__global__ void __launch_bounds__(kStreamTile)
stream_hbar_kernel(int G, double c, SVec Y, SVec lam, SVec hb) {
    const int b = blockIdx.y;
    int at, g;
    stream_site<NAT>(at, g);
    if (g >= G) return;
    constexpr int CP = stream_cells<NAT>();
    const int i = soff<NAT>(g, at);
    const double *y = Y.at(b) + i, *l = lam.at(b) + i;
    double* o = hb.at(b) + i;
    const double y0 = y[0], y1 = y[CP], y2 = y[2 * CP], v0 = c * l[0], v1 = c * l[CP], v2 = c * l[2 * CP];
    o[0] = y1 * v2 - y2 * v1;
    o[CP] = y2 * v0 - y0 * v2;
    o[2 * CP] = y0 * v1 - y1 * v0;
}

// Coefficients and outputs of one stage VJP: v = ca lam + cb S of this stage (cb 0 for kind 0); kind 0 (RK stage 3): S = sbar, acc = lam
// + sbar; 1 (stages 2, 1): S = sbar, acc += sbar; 2 (stage 0): lam = acc + sbar + dl.  Then the next VJP stage's
// Hbar = Ynext x (ca2 lam + cb2 S), unless Ynext is null.
struct VjpStage {
    int s;
    double ca, cb, ca2, cb2;
};

// Stage VJP of site (cell g, atom AT).  Y and hb (Hbar = Y x v, formed by the previous VJP stage or
// stream_hbar_kernel) are read of the partners too, every other vector only at the own site, so lam, S and acc change
// in place.  Sum over bonds as in vjp_cell; with PAIR (bonds and their parameter derivatives paired) the two partners
// of a pair are added first.
template <int NAT, int Z, int LZ, int NQ, int AT, bool PAIR, int kind>
__device__ __forceinline__ void stream_vjp_site(const Couplings<NAT, Z>& cp, const ParamDerivs<NAT, Z, NQ>& pd,
                                                const int* __restrict__ nbr, int G, int g, const VjpStage& st,
                                                const double* __restrict__ Y, const double* __restrict__ hb,
                                                double* lam, double* S, double* acc, const double* Ynext, double* hb_out,
                                                double f1, double f2, bool drive, const double (&dl)[3],
                                                double (&gq)[NQ]) {
    constexpr int NL = Z - LZ;
    constexpr int CP = stream_cells<NAT>();
    const int i0 = soff<NAT>(g, AT);
    double Yo[3], ho[3], lo[3], so[3], ao[3], yn[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int i = i0 + c * CP;
        Yo[c] = Y[i];
        ho[c] = hb[i];
        lo[c] = lam[i];
        so[c] = kind == 0 ? 0.0 : S[i];
        ao[c] = kind == 0 ? lo[c] : acc[i];
        yn[c] = Ynext ? Ynext[i] : 0.0;
    }
    double H[3], sb[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int d = 0; d < 3; ++d) H[d] = cp.has_field ? -cp.field[AT][d] : 0.0;
    if (cp.has_onsite) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            bond_acc(H[d], 2.0 * cp.onsite[AT][3 * d], 2.0 * cp.onsite[AT][3 * d + 1], 2.0 * cp.onsite[AT][3 * d + 2],
                     Yo[0], Yo[1], Yo[2]);
            sb[d] += 2.0 * (cp.onsite[AT][d] * ho[0] + cp.onsite[AT][3 + d] * ho[1] + cp.onsite[AT][6 + d] * ho[2]);
        }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        double t = -(ho[0] * pd.DB[q][AT][0] + ho[1] * pd.DB[q][AT][1] + ho[2] * pd.DB[q][AT][2]);
        if (pd.has_DA) {
#pragma unroll
            for (int d = 0; d < 3; ++d)
                t += 2.0 * ho[d] * (pd.DA[q][AT][3 * d] * Yo[0] + pd.DA[q][AT][3 * d + 1] * Yo[1] +
                                    pd.DA[q][AT][3 * d + 2] * Yo[2]);
        }
        gq[q] += t;
    }
    auto bond = [&](int n, const double (&P)[3], const double (&Q)[3]) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            bond_acc(H[d], cp.J[AT][n][3 * d], cp.J[AT][n][3 * d + 1], cp.J[AT][n][3 * d + 2], P[0], P[1], P[2]);
            bond_acc(sb[d], cp.J[AT][n][3 * d], cp.J[AT][n][3 * d + 1], cp.J[AT][n][3 * d + 2], Q[0], Q[1], Q[2]);
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (!pd.dj_any[q]) continue;             // e.g. a field parameter
            const double* D = pd.DJ[q][AT][n];
            gq[q] += Yo[0] * (D[0] * Q[0] + D[1] * Q[1] + D[2] * Q[2]) +
                     Yo[1] * (D[3] * Q[0] + D[4] * Q[1] + D[5] * Q[2]) +
                     Yo[2] * (D[6] * Q[0] + D[7] * Q[1] + D[8] * Q[2]);
        }
    };
#pragma unroll
    for (int n = 0; n < LZ; ++n) {
        const int ip = i0 + ((AT + 1 + n) % NAT - AT) * 3 * CP;
        double P[3] = {Y[ip], Y[ip + CP], Y[ip + 2 * CP]}, Q[3] = {hb[ip], hb[ip + CP], hb[ip + 2 * CP]};
        if constexpr (PAIR) {
            const int p = nbr[(AT * NL + n) * G + g];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                P[c] += Y[p + c * CP];
                Q[c] += hb[p + c * CP];
            }
        }
        bond(n, P, Q);
    }
#pragma unroll
    for (int m = 0; m < (PAIR ? 0 : NL); ++m)
        if (LZ + m < cp.zc[AT]) {
            const int p = nbr[(AT * NL + m) * G + g];
            const double P[3] = {Y[p], Y[p + CP], Y[p + 2 * CP]}, Q[3] = {hb[p], hb[p + CP], hb[p + 2 * CP]};
            bond(LZ + m, P, Q);
        }
    if (drive) {
#pragma unroll
        for (int d = 0; d < 3; ++d) drive_acc(H[d], cp.d1[AT][d], cp.d2[AT][d], f1, f2);
    }
    double v[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        v[c] = st.ca * lo[c];
        if (kind != 0) v[c] = v[c] + st.cb * so[c];
    }
    sb[0] += v[1] * H[2] - v[2] * H[1];
    sb[1] += v[2] * H[0] - v[0] * H[2];
    sb[2] += v[0] * H[1] - v[1] * H[0];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int i = i0 + c * CP;
        if (kind == 2) {
            lo[c] = ao[c] + sb[c] + dl[c];
            lam[i] = lo[c];
        } else {
            S[i] = sb[c];
            acc[i] = ao[c] + sb[c];
        }
        v[c] = st.ca2 * lo[c];
        if (kind != 2) v[c] = v[c] + st.cb2 * sb[c];
    }
    if (Ynext) {
        hb_out[i0] = yn[1] * v[2] - yn[2] * v[1];
        hb_out[i0 + CP] = yn[2] * v[0] - yn[0] * v[2];
        hb_out[i0 + 2 * CP] = yn[0] * v[1] - yn[1] * v[0];
    }
}

// One stage VJP of step n for every (tile, trajectory), one site per thread (atom uniform per warp, so couplings and
// derivatives are constant-bank operands); the tile's parameter cotangents are added to its slot.
template <int NAT, int Z, int LZ, int NQ, bool PAIR, int kind>
__global__ void __launch_bounds__(kStreamTile, 3)
stream_vjp_kernel(const __grid_constant__ Couplings<NAT, Z> cp, const __grid_constant__ ParamDerivs<NAT, Z, NQ> pd,
                  const __grid_constant__ StreamVjpArgs a, const __grid_constant__ VjpStage st, long long n_arg, SVec Y,
                  SVec hb, SVec lam, SVec S, SVec acc, SVec Ynext, SVec hb_out) {
    constexpr int NQV = NQ <= 4 ? 4 : 8;
    const long long n = (a.nbase ? *a.nbase : 0) + n_arg;
    __shared__ double red[32 * kRedStride];
    const int b = blockIdx.y;
    int at, g;
    stream_site<NAT>(at, g);
    double f1 = 0.0, f2 = 0.0;
    if (a.drive) {
        const int q = st.s == 0 ? 0 : (st.s < 3 ? 2 : 4);
        const double* d = a.drive + ((long long)b * a.n_steps + n) * 6 + q;
        f1 = d[0];
        f2 = d[1];
    }
    const bool drive = a.drive != nullptr && (f1 != 0.0 || f2 != 0.0);
    double dl[3] = {0.0, 0.0, 0.0};
    if (kind == 2) {
        const long long i = ((long long)b * (a.n_steps + 1) + n) * 3;
#pragma unroll
        for (int c = 0; c < 3; ++c) dl[c] = 2.0 * (a.mloc[i + c] - a.target[i + c]) / a.n_sites;
    }
    double gq[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) gq[q] = 0.0;
    if (g < a.G)
        with_atom<NAT>(at, [&](auto tag) {
            stream_vjp_site<NAT, Z, LZ, NQ, decltype(tag)::value, PAIR, kind>(
                cp, pd, a.nbr, a.G, g, st, Y.at(b), hb.at(b), lam.at(b), S.at(b), acc.at(b), Ynext.at(b), hb_out.at(b),
                f1, f2, drive, dl, gq);
        });
    double v[NQV];
#pragma unroll
    for (int q = 0; q < NQV; ++q) v[q] = q < NQ ? gq[q] : 0.0;
    double t;
    // one CTA per slot and launch: a reduction without a result is as ordered as a load and a store, and not waited for
    if (block_sum_par<NQV>(v, red, NQ, &t))
        atomicAdd(&a.gpart[((long long)b * a.tiles + blockIdx.x) * kPart + threadIdx.x], t);
}

// grad[b][q] = sum over tiles of the partials, in a fixed order (lane l adds tiles l, l + 32, ..., then a butterfly);
// one CTA per trajectory, one warp per parameter.
static __global__ void stream_grad_kernel(const double* __restrict__ gpart, int tiles, int nq, double* __restrict__ out,
                                   long long out_stride) {
    const int b = blockIdx.x, q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (q >= nq) return;
    double s = 0.0;
    for (int t = lane; t < tiles; t += 32) s += gpart[((long long)b * tiles + t) * kPart + q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[(long long)b * out_stride + q] = s;
}

}  // namespace cmd
