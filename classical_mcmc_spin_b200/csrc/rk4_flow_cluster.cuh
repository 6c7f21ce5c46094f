// rk4_flow_cluster.cuh -- rk4_flow.cuh with one trajectory over a thread-block cluster of CS
// CTAs (CS SMs), for lattices one CTA cannot hold (48x48 honeycomb: 4 x 576 cells).
//
// CTA `rank` owns cells [rank*Gc, rank*Gc + Gc).  A site that other CTAs read is stored into
// their halo columns too (each stage-buffer row is MAXT own columns, then HMAX halo columns;
// tables as of the RK45 halo tilings), so every partner read is a plain shared-memory load.
// The warps that exchange spins wait on one another as in rk4_flow.cuh, across CTAs through
// remote arrives on the same input barriers (cluster-scope release / acquire); there is no
// cluster barrier inside the run, so only the few warps at a slab's edge see the 200-cycle
// distance to the next SM, and they hide it by running ahead or behind.  rk4_cluster_kernel
// pays a cluster barrier (~490 cycles) per stage in every warp, and a remote load per
// component of a remote partner.
//
// B200, 48x48 honeycomb on 4 CTAs: 0.87 us a stage (1.54 with a cluster barrier per stage, 0.68
// for one 24x24 CTA of the same size); 198 warp instructions per warp and stage, 82 of them FP64;
// 64 trajectories x 1000 steps 6.91 ms, sliced (11.98; 6.81 without the look at FlowWait::dead once
// a step, 7.03 with it in the middle of a stage).  Pyrochlore, 1372 cells: 2.7 us a stage against 4.2.
//
// Rows: each CTA's helper warp sums its warps' partials and stores them in CTA 0's totals
// ring; CTA 0's helper adds them in rank order and writes the raw row.
#pragma once

#include "rk4_cluster.cuh"
#include "rk4_flow.cuh"

namespace cmd {

constexpr int kFlowPeers = 32;                // peers of a warp, itself included (one lane each)

struct FlowClusterArgs {
    int Gc;                    // cells per CTA
    const int* pw;             // [G][NAT][Z-LZ] partner offsets in this CTA's stage buffer 0 (own or halo column)
    const int* push;           // [G][NAT][Z-LZ] (rank << 24) | halo slot this site is stored to in that CTA, or -1
    const int* peers;          // [CS][warps][kFlowPeers] (rank << 8) | warp, or -1
};

__host__ __device__ constexpr int flow_halo(int nat) { return nat <= 2 ? 128 : 256; }
__host__ __device__ constexpr long long flow_cluster_smem_doubles(int nat, int maxt, int cs) {
    return 2LL * nat * 3 * (maxt + flow_halo(nat)) + flow_ring_doubles(nat, maxt) + kFlowRows * cs * flow_nv(nat) +
           2LL * (maxt / 32) + 4 * kFlowRows + (long long)sizeof(FlowWait) / 8;
}

__device__ __forceinline__ uint32_t flow_map(uint32_t local, int rank) {
    uint32_t out;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(local), "r"(rank));
    return out;
}
__device__ __forceinline__ void flow_st_cluster(uint32_t addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
// Arrives on a barrier of any CTA of the cluster in the lanes where `on` is set.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr, bool on) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t"
        "@p mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n\t}" ::"r"(addr), "r"((unsigned)on)
        : "memory");
}
__device__ __forceinline__ void flow_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// mbar_wait with cluster-scope acquire.
__device__ __forceinline__ void mbar_wait_cluster(uint32_t bar, uint32_t parity, uint32_t words, int* fault) {
    CMD_MBAR_WAIT("cluster", offsetof(FlowWait, ns));
}

template <int NAT, int Z, int LZ, int CS, int MAXT, bool STAT, bool DRIVE, bool PAIR>
__global__ void __launch_bounds__(MAXT, 1)
rk4_flow_cluster_kernel(const __grid_constant__ Couplings<NAT, Z> cp, const __grid_constant__ ResidentArgs a,
                        const __grid_constant__ FlowClusterArgs fc) {
    constexpr int NS = 4;
    constexpr int NL = Z - LZ;                       // non-local slots per atom
    constexpr int NR = NVals<NAT>::used;
    constexpr int NV = flow_nv(NAT);
    constexpr int NW = MAXT / 32;
    constexpr int GS = MAXT + flow_halo(NAT);        // component stride in shared memory
    constexpr int SB = NAT * 3 * GS;                 // one stage buffer
    constexpr int span = 32 / NV;
    extern __shared__ double smem[];
    double* red = smem + 2 * SB;                     // [kFlowRows][NW][NV] observable partials of the warps
    double* tot = red + flow_ring_doubles(NAT, MAXT);               // [kFlowRows][CS][NV] the CTAs' totals (CTA 0)
    double* bars = tot + kFlowRows * CS * NV;        // [2][NW] inputs, [kFlowRows] full, free, totals, totals free
    unsigned rank_u;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank_u));
    const int rank = (int)rank_u;
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int ncw = nwarps - 1;                      // warps with cells; the last one is the helper
    const uint32_t bar_in = (uint32_t)__cvta_generic_to_shared(bars);
    const uint32_t bar_full = bar_in + 16 * NW, bar_free = bar_full + 8 * kFlowRows;
    const uint32_t bar_tot = bar_free + 8 * kFlowRows, bar_tfree = bar_tot + 8 * kFlowRows;
    FlowWait* fw = reinterpret_cast<FlowWait*>(bars + 2 * NW + 4 * kFlowRows);
    const uint32_t wait_words = (uint32_t)__cvta_generic_to_shared(fw);

    // this CTA's trajectory and steps [n0, n1): items are (slice, trajectory), trajectories fastest
    const long long item = a.item0 + blockIdx.x / CS;
    const long long slice = item / a.B, b = item - slice * a.B;
    const long long n0 = a.n_steps * slice / a.slices, n1 = a.n_steps * (slice + 1) / a.slices;
    const int G = a.G;
    const int g = rank * fc.Gc + tid;                // global cell of this thread
    const bool own = tid < fc.Gc && g < G;
    const long long N3 = (long long)G * NAT * 3;

    double y[NAT][3], acc[NAT][3], yc[NAT][3];
    int pb[NAT][NL > 0 ? NL : 1];                    // word offset of each partner's component 0 in buffer 0
    const double* y0 = slice == 0 ? a.y0 + b * a.y0_stride : a.y_mid + b * N3;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
#pragma unroll
    for (int at = 0; at < NAT; ++at)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            y[at][c] = own ? y0[((long long)g * NAT + at) * 3 + c] : 0.0;
            acc[at][c] = 0.0;
        }
    uint32_t pd[NAT][NL > 0 ? NL : 1];               // shared::cluster addresses of the halo slots to store to (~0: none)
    bool pushes = false;
#pragma unroll
    for (int at = 0; at < NAT; ++at)
#pragma unroll
        for (int m = 0; m < NL; ++m) {
            const long long i = ((long long)g * NAT + at) * NL + m;
            pb[at][m] = own ? fc.pw[i] : at * 3 * GS + tid;
            const int w = own ? fc.push[i] : -1;
            pd[at][m] = ~0u;
            if (w >= 0) pd[at][m] = flow_map(sbase + 8u * (uint32_t)(w & kClusterOffsetMask), w >> kClusterRankShift);
            pushes |= w >= 0;
        }
    pushes = __any_sync(0xffffffffu, pushes);
    // lane l serves peer l of this warp
    const int pw = warp < ncw ? fc.peers[(rank * ncw + warp) * kFlowPeers + lane] : -1;
    const bool peer = pw >= 0;
    const unsigned n_peers = __popc(__ballot_sync(0xffffffffu, peer));
    const bool remote = __any_sync(0xffffffffu, peer && (pw >> 8) != rank);     // some peer is in another CTA
    const double dt = a.dt, half = 0.5 * dt;
    // envelope factors of the current step: lane e < NE holds factor e (drive_table_kernel, drive_stages_kernel)
    constexpr int NE = 6;
    const bool stager = DRIVE && lane < NE;
    const double* dtab = stager ? a.drive + b * a.n_steps * NE + lane : nullptr;
    double cur_f = stager && n0 < n1 ? dtab[n0 * NE] : 0.0;
    if (lane == 0 && warp < ncw)
        for (int p = 0; p < 2; ++p) mbar_init(bar_in + 8 * (NW * p + warp), n_peers);
    if (tid < kFlowRows) {
        mbar_init(bar_full + 8 * tid, ncw);
        mbar_init(bar_free + 8 * tid, 1);
        mbar_init(bar_tot + 8 * tid, CS);
        mbar_init(bar_tfree + 8 * tid, 1);
    }
    flow_wait_init(fw, tid, a.wait_ns, a.row_ns);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    flow_cluster_sync();                             // every CTA's barriers exist
    const uint32_t my_in = bar_in + 8 * warp;
    const bool far = peer && (pw >> 8) != rank;
    const uint32_t near_in = bar_in + 8 * (peer ? pw & 255 : 0), far_in = flow_map(near_in, peer ? pw >> 8 : rank);
    // stores v as component c of own atom `at` of buffer buf (0 / 1), and into the halo columns of its readers
    auto store = [&](int buf, int at, int c, double v) __attribute__((always_inline)) {
        smem[buf * SB + (at * 3 + c) * GS + tid] = v;
    };
    auto push_all = [&](int buf, const double (&v)[NAT][3]) __attribute__((always_inline)) {
        if (!pushes) return;
#pragma unroll
        for (int at = 0; at < NAT; ++at)
#pragma unroll
            for (int m = 0; m < NL; ++m)
                if (pd[at][m] != ~0u)
#pragma unroll
                    for (int c = 0; c < 3; ++c) flow_st_cluster(pd[at][m] + 8u * (uint32_t)(buf * SB + c * GS), v[at][c]);
    };
#pragma unroll
    for (int at = 0; at < NAT; ++at)
#pragma unroll
        for (int c = 0; c < 3; ++c) store(0, at, c, y[at][c]);
    push_all(0, y);
    // Stage k (counted over the run) waits for phase k / 2 of input barrier k % 2.
    auto wait_in = [&](int k) {
        if (remote) mbar_wait_cluster(my_in + 8 * NW * (k & 1), (k >> 1) & 1, wait_words, a.fault);
        else mbar_wait(my_in + 8 * NW * (k & 1), (k >> 1) & 1, wait_words, a.fault);
    };
    auto publish = [&](int k) {                      // the input of stage k is stored
        __syncwarp();
        mbar_arrive(near_in + 8 * NW * (k & 1), peer && !far);
        if (remote) mbar_arrive_cluster(far_in + 8 * NW * (k & 1), far);
    };
    // H = field of the thread's atoms at the stage input S (own atoms) / buffer buf (partners)
    auto field_at = [&](int buf, const double (&S)[NAT][3], double (&H)[NAT][3]) {
        double P[NAT][NL > 0 ? NL : 1][3];
#pragma unroll
        for (int at = 0; at < NAT; ++at)
#pragma unroll
            for (int m = 0; m < NL; ++m)
#pragma unroll
                for (int c = 0; c < 3; ++c) P[at][m][c] = smem[pb[at][m] + buf * SB + c * GS];
#pragma unroll
        for (int at = 0; at < NAT; ++at)
#pragma unroll
            for (int d = 0; d < 3; ++d) H[at][d] = STAT ? opaque_zero() - cp.field[at][d] : 0.0;
        if (STAT && cp.has_onsite) {
#pragma unroll
            for (int at = 0; at < NAT; ++at) {
                const double s0 = 2.0 * S[at][0], s1 = 2.0 * S[at][1], s2 = 2.0 * S[at][2];
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    bond_acc(H[at][d], cp.onsite[at][3 * d], cp.onsite[at][3 * d + 1], cp.onsite[at][3 * d + 2], s0,
                             s1, s2);
            }
        }
#pragma unroll
        for (int n = 0; n < LZ; ++n)
#pragma unroll
            for (int at = 0; at < NAT; ++at) {
                const int pa = (at + 1 + n) % NAT;
                // PAIR: slot LZ + n has the same coupling, so J_n (S + P) stands for both bonds
                double T[3] = {S[pa][0], S[pa][1], S[pa][2]};
                if constexpr (PAIR) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) T[c] += P[at][n][c];
                }
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    bond_acc(H[at][d], cp.J[at][n][3 * d], cp.J[at][n][3 * d + 1], cp.J[at][n][3 * d + 2], T[0], T[1],
                             T[2]);
            }
        if constexpr (PAIR) return;
#pragma unroll
        for (int m = 0; m < NL; ++m)
#pragma unroll
            for (int at = 0; at < NAT; ++at)
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    bond_acc(H[at][d], cp.J[at][LZ + m][3 * d], cp.J[at][LZ + m][3 * d + 1],
                             cp.J[at][LZ + m][3 * d + 2], P[at][m][0], P[at][m][1], P[at][m][2]);
    };
    auto add_obs = [&](double (&part)[NV], const double (&S)[NAT][3], const double (&H)[NAT][3]) {
#pragma unroll
        for (int q = 0; q < NV; ++q) part[q] = 0.0;
#pragma unroll
        for (int at = 0; at < NAT; ++at) {
#pragma unroll
            for (int c = 0; c < 3; ++c) part[3 * at + c] = S[at][c];
#pragma unroll
            for (int c = 0; c < 3; ++c)
                part[3 * NAT] = fma(S[at][c], STAT ? H[at][c] - cp.field[at][c] : H[at][c], part[3 * NAT]);
        }
    };
    auto store_partials = [&](double (&part)[NV], int slot) {
        const double r = warp_reduce_many<NV>(part);
        if ((lane % span) == 0) red[(slot * NW + warp) * NV + lane / span] = r;
        __syncwarp();
        mbar_arrive(bar_full + 8 * slot, lane == 0);
    };
    // helper: all warps' partials of the row are in the slot; this CTA's totals go to CTA 0, whose helper adds the CTAs
    // in rank order and writes the raw row
    auto cta_total = [&](int slot) {
        double v[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) v[q] = lane < ncw ? red[(slot * NW + lane) * NV + q] : 0.0;
        return warp_reduce_many<NV>(v);
    };
    const uint32_t tot0 = flow_map((uint32_t)__cvta_generic_to_shared(tot), 0);
    auto write_row = [&](int slot, long long row) {
        if (!a.raw || lane >= NR) return;
        double s = 0.0;
#pragma unroll
        for (int r = 0; r < CS; ++r) s += tot[(slot * CS + r) * NV + lane];
        a.raw[(b * a.rows + row) * a.raw_stride + lane] = s;
    };
    auto finish_row = [&](int slot, long long row, int phase) {
        const double r = cta_total(slot);
        __syncwarp();
        mbar_arrive(bar_free + 8 * slot, lane == 0);
        mbar_wait_cluster(bar_tfree + 8 * slot, phase ^ 1, wait_words, a.fault);
        if ((lane % span) == 0) flow_st_cluster(tot0 + 8u * ((slot * CS + rank) * NV + lane / span), r);
        __syncwarp();
        mbar_arrive_cluster(flow_map(bar_tot + 8 * slot, 0), lane == 0);
        if (rank != 0) return;
        mbar_wait_cluster(bar_tot + 8 * slot, phase, wait_words, a.fault);
        write_row(slot, row);
        __syncwarp();
        mbar_arrive_cluster(flow_map(bar_tfree + 8 * slot, lane < CS ? lane : 0), lane < CS);
    };
    auto write_state = [&](double* dst) {
#pragma unroll
        for (int at = 0; at < NAT; ++at)
#pragma unroll
            for (int c = 0; c < 3; ++c) dst[((long long)g * NAT + at) * 3 + c] = y[at][c];
    };

    const long long row0 = (n0 + a.save_every - 1) / a.save_every;   // rows before this slice
    long long save_left = row0 * a.save_every - n0;
    int row = 0;                                     // rows begun here; ring slot row % kFlowRows
    double part[NV];
    if (warp == ncw) {
        for (long long n = n0 + save_left; n < n1; n += a.save_every, ++row) {
            mbar_wait_row(bar_full + 8 * (row % kFlowRows), (row / kFlowRows) & 1, wait_words, a.fault);
            if (gave_up(wait_words)) break;
            finish_row(row % kFlowRows, row0 + row, (row / kFlowRows) & 1);
            if (gave_up(wait_words)) break;
        }
    } else {
        publish(0);
        for (long long step = n0; step < n1; ++step) {
            const bool observe = save_left == 0;
            save_left = observe ? a.save_every - 1 : save_left - 1;
            const bool driven = DRIVE && __any_sync(0xffffffffu, cur_f != 0.0);   // 0*d adds exactly 0
            double next_f = 0.0;
            bool leave = false;
            if (stager && step + 1 < n1) next_f = dtab[(step + 1) * NE];
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                const int rb = s & 1;                // buffer read in this stage; the other one is written
                const int ti = s == 0 ? 0 : (s == 3 ? 2 : 1);
                if (s == 1 && observe) {
                    mbar_wait(bar_free + 8 * (row % kFlowRows), ((row / kFlowRows) & 1) ^ 1, wait_words, a.fault);
                    store_partials(part, row % kFlowRows);
                }
                const double(&S)[NAT][3] = s == 0 ? y : yc;
                double H[NAT][3];
                wait_in(s);
                field_at(rb, S, H);
                if (s == 0 && observe) add_obs(part, S, H);
                if (driven) {
                    const double f1 = -__shfl_sync(0xffffffffu, cur_f, 2 * ti);
                    const double f2 = -__shfl_sync(0xffffffffu, cur_f, 2 * ti + 1);
#pragma unroll
                    for (int at = 0; at < NAT; ++at)
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            H[at][d] = fma(cp.d1[at][d], f1, H[at][d]);
                            H[at][d] = fma(cp.d2[at][d], f2, H[at][d]);
                        }
                }
                double K[NAT][3];
#pragma unroll
                for (int at = 0; at < NAT; ++at) {
                    K[at][0] = H[at][1] * S[at][2] - H[at][2] * S[at][1];
                    K[at][1] = H[at][2] * S[at][0] - H[at][0] * S[at][2];
                    K[at][2] = H[at][0] * S[at][1] - H[at][1] * S[at][0];
                }
                if (s == 0 && observe && a.traj && own) write_state(a.traj + (b * a.rows + row0 + row) * N3);
#pragma unroll
                for (int at = 0; at < NAT; ++at)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        if (s == 3) {
                            y[at][c] += (dt / 6.0) * (acc[at][c] + K[at][c]);
                        } else {
                            acc[at][c] = s == 0 ? K[at][c] : acc[at][c] + 2.0 * K[at][c];
                            yc[at][c] = 1.0 * y[at][c] + (s == 2 ? dt : half) * K[at][c];
                        }
                        store(rb ^ 1, at, c, s == NS - 1 ? y[at][c] : yc[at][c]);
                    }
                push_all(rb ^ 1, s == NS - 1 ? y : yc);
                publish(s + 1);
                if (s == NS - 2) leave = gave_up(wait_words);      // here, where the wait and the field sums hide it
            }
            cur_f = next_f;
            if (observe) ++row;
            if (leave) break;
        }
    }
    // every store into this CTA has landed, every row is written; and where a wait gave up, no CTA leaves while others
    // (whose own waits for it then run out) may still store into it
    flow_cluster_sync();
    if (slice + 1 < a.slices) {
        if (own) write_state(a.y_mid + b * N3);
        return;
    }
    // Final observation of y(t_end): one more static-field evaluation for E.
    if (warp < ncw) {
        double H[NAT][3];
        field_at(0, y, H);
        add_obs(part, y, H);
        if (a.traj && own) write_state(a.traj + (b * a.rows + a.rows - 1) * N3);
        const double r = warp_reduce_many<NV>(part);
        if ((lane % span) == 0) red[warp * NV + lane / span] = r;
    }
    __syncthreads();
    if (warp == 0) {
        const double r = cta_total(0);
        if ((lane % span) == 0) flow_st_cluster(tot0 + 8u * (rank * NV + lane / span), r);
    }
    flow_cluster_sync();
    if (rank == 0 && warp == 0) write_row(0, a.rows - 1);
    if (a.y_out && own) write_state(a.y_out + b * N3);
}

}  // namespace cmd
