// rk4_flow.cuh -- resident RK4, one CTA per trajectory and one unit cell per thread,
// with waits between the warps that exchange spins in place of a stage barrier.
//
// State on chip as in rk4_resident.cuh: y_n, the RK4 sum and the own stage input in
// registers, the stage input neighbours read double-buffered in shared memory at the
// compile-time component stride MAXT (buf[(atom*3 + comp)*MAXT + cell]), couplings as
// constant-bank operands, no memory traffic per step but the observable row.
//
//   * A warp needs only the stage inputs of the few warps its bonds reach.  When it has
//     stored its part of a stage input it arrives at the input barrier (mbarrier) of each
//     of those warps, one lane per peer, and it starts a stage when all of its own peers
//     have arrived.  Warps then drift apart by up to a stage per hop, so partner loads of
//     some overlap the field sums of others; under a CTA barrier all warps load, add and
//     wait together, and the FP64 pipe stands still meanwhile.
//   * Peers are symmetric (built from both ends of every bond), so a peer's arrival for
//     stage k+1 also says that it no longer reads the buffer of stage k, which is the one
//     written next.  Two barriers per warp alternate: a peer may arrive for stage k+1
//     while another still misses for k, but not for k+2.
//   * Observables leave through a ring of kFlowRows rows: every warp stores its partial
//     sums and goes on; a helper warp without cells (HELP; else the warps in turn) adds
//     them over the warps, writes the raw row and frees the slot.
//   * The field sums of a cell's atoms are interleaved (3 NAT independent chains); -B and
//     2 A S are formed from values the compiler cannot hoist, which keeps every coupling a
//     constant-bank operand without a branch per atom.
// Waits are bounded (mbar_wait); a run whose wait gave up skips its remaining steps and reports CMD_ERR_WATCHDOG.
//
// Bound: issue slots and the FP64 pipe.  24x24 honeycomb, one step's observables every step: 183 warp instructions
// per warp and stage, 82 of them FP64 (209 and 92 with the drive); 18 warps put 5 on two of the SM's four schedulers,
// so the pipe needs 820 and the issue port 915 of the stage's 1330 cycles there (0.68 us; 0.88 us with a CTA barrier
// per stage and 205 instructions).  B200, 1965 MHz: 768 driven trajectories x 2000 steps 31.7 ms (45.5 ms with the
// barrier and whole waves); one trajectory 2.78 us per step (3.61); 40 trajectories of 8x8 x 500 steps 0.94 ms (1.35);
// 200 of the 1024-spin pyrochlore x 800 driven steps 4.26 ms (11.6 with the atoms in sequence); one 24x24 SSPRK53
// trajectory x 400 steps, 11 states saved, 1.60 ms (7.05 in global memory, where every RK vector is read and written
// each stage).  Polling progress words instead of waiting on mbarriers: 256 instructions, 0.83 us.  The look at
// FlowWait::dead once a step stands after the publish of the last but one stage: 31.7 ms (32.1 with a flag in a
// register that only the cold path sets and a vote, 31.9 in the middle of the last stage); lone undriven warps lose
// 1-5 % to it.
#pragma once

#include "flow_wait.h"
#include "rk4_resident.cuh"

namespace cmd {

constexpr int kFlowRows = 2;                  // observable rows in flight (ring slots, a power of two)
constexpr int kFlowMaxWarps = 20;             // warps with cells

__host__ __device__ constexpr int flow_nv(int nat) { return nat <= 2 ? 8 : 16; }

// Shared memory of a CTA in doubles: two stage buffers of stride MAXT, and room for the ring
// [kFlowRows][warps][values], two input barriers per warp, the ring's barriers, peer masks.
__host__ __device__ constexpr long long flow_smem_doubles(int nat, int maxt) {
    return 2LL * nat * 3 * maxt + 32 * kRedStride + 12;
}
__host__ __device__ constexpr long long flow_ring_doubles(int nat, int maxt) {
    return (long long)kFlowRows * (maxt / 32) * flow_nv(nat);
}

// +0 the compiler cannot see through.
__device__ __forceinline__ double opaque_zero() {
    double z;
    asm volatile("mov.f64 %0, 0d0000000000000000;" : "=d"(z));
    return z;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// Arrives (release) in the lanes where `on` is set; predicated, so the warp does not branch.
__device__ __forceinline__ void mbar_arrive(uint32_t bar, bool on) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t"
        "@p mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar), "r"((unsigned)on) : "memory");
}
// Waits until the phase of `parity` of the mbarrier completes (acquire, at the named scope).  Bounded: a thread that
// has tried kWaitTries times and for longer than its limit in FlowWait (the tries too, so that time in which the GPU runs another
// process does not count) sets FlowWait::dead and *fault (host) and goes on, as does one that finds `dead` set; every
// warp of the CTA looks at `dead` once a step and leaves the step loop (gave_up).  No thread ends early: a CTA of a
// cluster stays while others may store into it, and every thread meets the barriers after the loop.  One block of
// inline PTX: as a call, or as C++ after a failed first try, the cold path costs the hot one spills.
constexpr unsigned kWaitTries = 4096;
#define CMD_MBAR_WAIT(SCOPE, LIMIT)                                                                          \
    asm volatile(                                                                                            \
        "{\n\t.reg .pred p;\n\t.reg .u64 t0, t1, lim;\n\t.reg .u32 d, n;\n\t"                               \
        "mbarrier.try_wait.parity.acquire." SCOPE ".shared::cta.b64 p, [%0], %1;\n\t"                        \
        "@p bra DONE;\n\t"                                                                                   \
        "mov.u64 t0, %%globaltimer;\n\t"                                                                     \
        "mov.u32 n, 0;\n"                                                                                    \
        "AGAIN:\n\t"                                                                                         \
        "ld.volatile.shared::cta.u32 d, [%2];\n\t"                                                           \
        "setp.ne.u32 p, d, 0;\n\t"                                                                           \
        "@p bra DONE;\n\t"                                                                                   \
        "mbarrier.try_wait.parity.acquire." SCOPE ".shared::cta.b64 p, [%0], %1, 2000;\n\t"                  \
        "@p bra DONE;\n\t"                                                                                   \
        "add.u32 n, n, 1;\n\t"                                                                               \
        "mov.u64 t1, %%globaltimer;\n\t"                                                                     \
        "sub.u64 t1, t1, t0;\n\t"                                                                            \
        "ld.shared::cta.u64 lim, [%2+%5];\n\t"                                                               \
        "setp.le.u64 p, t1, lim;\n\t"                                                                        \
        "@p bra AGAIN;\n\t"                                                                                  \
        "setp.lt.u32 p, n, %4;\n\t"                                                                          \
        "@p bra AGAIN;\n\t"                                                                                  \
        "mov.u32 d, 1;\n\t"                                                                                  \
        "st.volatile.shared::cta.u32 [%2], d;\n\t"                                                           \
        "st.volatile.global.u32 [%3], d;\n"                                                                  \
        "DONE:\n\t}"                                                                                         \
        :                                                                                                    \
        : "r"(bar), "r"(parity), "r"(words), "l"(fault), "n"(kWaitTries), "n"(LIMIT)                         \
        : "memory")

__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, uint32_t words, int* fault) {
    CMD_MBAR_WAIT("cta", offsetof(FlowWait, ns));
}
// The helper warp's wait for a row, which is as many steps away as the caller saves rows apart.
__device__ __forceinline__ void mbar_wait_row(uint32_t bar, uint32_t parity, uint32_t words, int* fault) {
    CMD_MBAR_WAIT("cta", offsetof(FlowWait, row_ns));
}
// Whether a wait of the CTA gave up, the same answer in every lane of the warp.
__device__ __forceinline__ bool gave_up(uint32_t words) {
    unsigned d;
    asm volatile("ld.volatile.shared::cta.u32 %0, [%1];" : "=r"(d) : "r"(words));
    return __any_sync(0xffffffffu, d != 0);
}

// Stages per step: classic RK4, or the reference GPU's default method SSPRK(5,3) (integrator.cuh:406-448).
constexpr int kFlowRK4 = 4, kFlowSSPRK53 = 5;

// PAIR: the layout's bonds are paired (Layout::paired; a.nbr in that order).  NS = stages per step (kFlow*).  Registers hold y, the stage input and one more vector: the RK4 sum, or the second
// SSPRK(5,3) stage input.
template <int NAT, int Z, int LZ, int MAXT, int MINB, bool STAT, bool DRIVE, bool HELP, int NS, bool PAIR>
__global__ void __launch_bounds__(MAXT, MINB)
rk4_flow_kernel(const __grid_constant__ Couplings<NAT, Z> cp, const __grid_constant__ ResidentArgs a) {
    constexpr int NL = Z - LZ;                       // non-local slots per atom
    constexpr int NR = NVals<NAT>::used;
    constexpr int NV = flow_nv(NAT);
    constexpr int NW = MAXT / 32;
    constexpr int GS = MAXT;                         // component stride in shared memory
    constexpr int SB = NAT * 3 * GS;                 // one stage buffer
    constexpr int span = 32 / NV;
    static_assert(flow_ring_doubles(NAT, MAXT) + 2 * NW + 2 * kFlowRows + 16 + sizeof(FlowWait) / 8 <= 32 * kRedStride + 12,
                  "ring, barriers, peer masks and wait words fit");
    extern __shared__ double smem[];
    double* red = smem + 2 * SB;                     // [kFlowRows][NW][NV] observable partials of the warps
    double* bars = red + flow_ring_doubles(NAT, MAXT);              // [2][NW] inputs, [kFlowRows] full, free
    int* dep = reinterpret_cast<int*>(bars + 2 * NW + 2 * kFlowRows);  // [32] warps a warp exchanges spins with
    FlowWait* fw = reinterpret_cast<FlowWait*>(dep + 32);
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int ncw = HELP ? nwarps - 1 : nwarps;      // warps with cells
    const uint32_t bar_in = (uint32_t)__cvta_generic_to_shared(bars);
    const uint32_t bar_full = bar_in + 16 * NW, bar_free = bar_full + 8 * kFlowRows;
    const uint32_t wait_words = (uint32_t)__cvta_generic_to_shared(fw);

    // this CTA's trajectory and steps [n0, n1): items are (slice, trajectory), trajectories fastest
    const long long item = a.item0 + blockIdx.x;
    const long long slice = item / a.B, b = item - slice * a.B;
    const long long n0 = a.n_steps * slice / a.slices, n1 = a.n_steps * (slice + 1) / a.slices;
    const int G = a.G;
    const int g = tid;
    const bool own = g < G;
    const long long N3 = (long long)G * NAT * 3;

    double y[NAT][3], acc[NAT][3], yc[NAT][3];
    int pb[NAT][NL > 0 ? NL : 1];                    // word offset of each partner's component 0 in buffer 0
    const double* y0 = slice == 0 ? a.y0 + b * a.y0_stride : a.y_mid + b * N3;
    if (tid < 32) dep[tid] = 0;
    flow_wait_init(fw, tid, a.wait_ns, a.row_ns);
#pragma unroll
    for (int at = 0; at < NAT; ++at)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double v = own ? y0[((long long)g * NAT + at) * 3 + c] : 0.0;
            y[at][c] = v;
            acc[at][c] = 0.0;
            smem[(at * 3 + c) * GS + g] = v;
        }
    __syncthreads();
#pragma unroll
    for (int at = 0; at < NAT; ++at)
#pragma unroll
        for (int m = 0; m < NL; ++m) {
            int w = at * 3 * GS + g;
            if (own) {
                // resident-layout offset (atom*3)*G + cell -> (atom*3)*GS + cell
                const int off = a.nbr[((long long)g * NAT + at) * NL + m];
                const int pat3 = off / G, cell = off - pat3 * G;
                w = pat3 * GS + cell;
                atomicOr(&dep[warp], 1 << (cell >> 5));
                atomicOr(&dep[cell >> 5], 1 << warp);
            }
            pb[at][m] = w;
        }
    const double dt = a.dt, half = 0.5 * dt;
    // envelope factors of the current step: lane e < NE holds factor e (drive_table_kernel, drive_stages_kernel)
    constexpr int NE = NS == kFlowRK4 ? 6 : 2 * NS;
    const bool stager = DRIVE && lane < NE;
    const double* dtab = stager ? a.drive + b * a.n_steps * NE + lane : nullptr;
    double cur_f = stager && n0 < n1 ? dtab[n0 * NE] : 0.0;
    __syncthreads();
    // a warp is its own peer too, so that every input barrier completes
    if (tid < ncw)
        for (int p = 0; p < 2; ++p) mbar_init(bar_in + 8 * (NW * p + tid), __popc(dep[tid] | (1 << tid)));
    if (tid < kFlowRows) {
        mbar_init(bar_full + 8 * tid, ncw);
        mbar_init(bar_free + 8 * tid, 1);
    }
    __syncthreads();
    const bool peer = lane < ncw && warp < ncw && (((dep[warp] | (1 << warp)) >> lane) & 1);
    const uint32_t my_in = bar_in + 8 * warp, peer_in = bar_in + 8 * lane;
    // Stage k (counted over the run) waits for phase k / 2 of input barrier k % 2.
    auto wait_in = [&](int k) { mbar_wait(my_in + 8 * NW * (k & 1), (k >> 1) & 1, wait_words, a.fault); };
    auto publish = [&](int k) {                      // the input of stage k is stored
        __syncwarp();
        mbar_arrive(peer_in + 8 * NW * (k & 1), peer);
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
    // all warps' partials of the row are in the slot: add them, write the raw row, free the slot
    auto finish_row = [&](int slot, long long row) {
        double v[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) v[q] = lane < ncw ? red[(slot * NW + lane) * NV + q] : 0.0;
        const double r = warp_reduce_many<NV>(v);
        if (a.raw && (lane % span) == 0 && lane / span < NR) a.raw[(b * a.rows + row) * a.raw_stride + lane / span] = r;
        __syncwarp();
        mbar_arrive(bar_free + 8 * slot, lane == 0);
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
    int finisher = 0;                                // warp that finishes the current row (no helper)
    int k0 = 0;                                      // first stage of the step, mod 4 (0 when a step has 4 stages)
    double part[NV];
    if (HELP && warp == ncw) {
        for (long long n = n0 + save_left; n < n1; n += a.save_every, ++row) {
            mbar_wait_row(bar_full + 8 * (row % kFlowRows), (row / kFlowRows) & 1, wait_words, a.fault);
            if (gave_up(wait_words)) break;
            finish_row(row % kFlowRows, row0 + row);
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
                const int k = NS == 4 ? s : k0 + s;
                const int rb = k & 1;                // buffer read in this stage; the other one is written
                const int ti = NS == kFlowSSPRK53 ? s : (s == 0 ? 0 : (s == 3 ? 2 : 1));
                if (s == 1 && observe) {
                    mbar_wait(bar_free + 8 * (row % kFlowRows), ((row / kFlowRows) & 1) ^ 1, wait_words, a.fault);
                    store_partials(part, row % kFlowRows);
                }
                const double(&S)[NAT][3] = s == 0 ? y : yc;
                double H[NAT][3];
                wait_in(k);
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
                double* wbuf = smem + (rb ^ 1) * SB;
#pragma unroll
                for (int at = 0; at < NAT; ++at)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        if constexpr (NS == kFlowSSPRK53) {          // the reference's 15-digit coefficients
                            if (s == 0) {
                                yc[at][c] = 1.0 * y[at][c] + (0.377268915331368 * dt) * K[at][c];
                            } else if (s == 1) {
                                yc[at][c] = 1.0 * yc[at][c] + (0.377268915331368 * dt) * K[at][c];
                                acc[at][c] = yc[at][c];
                            } else if (s == 2) {
                                yc[at][c] = 0.355909775063327 * y[at][c] + 0.644090224936674 * acc[at][c] +
                                            (0.242995220537396 * dt) * K[at][c];
                            } else if (s == 3) {
                                yc[at][c] = 0.367933791638137 * y[at][c] + 0.632066208361863 * yc[at][c] +
                                            (0.238458932846290 * dt) * K[at][c];
                            } else {
                                y[at][c] = 0.237593836598569 * acc[at][c] + 0.762406163401431 * yc[at][c] +
                                           (0.287632146308408 * dt) * K[at][c];
                            }
                        } else if (s == 3) {
                            y[at][c] += (dt / 6.0) * (acc[at][c] + K[at][c]);
                        } else {
                            acc[at][c] = s == 0 ? K[at][c] : acc[at][c] + 2.0 * K[at][c];
                            yc[at][c] = 1.0 * y[at][c] + (s == 2 ? dt : half) * K[at][c];
                        }
                        wbuf[(at * 3 + c) * GS + g] = s == NS - 1 ? y[at][c] : yc[at][c];
                    }
                publish(k + 1);
                if (s == NS - 2) leave = gave_up(wait_words);      // here, where the next wait hides it
            }
            cur_f = next_f;
            if (NS % 4 != 0) k0 = (k0 + NS) & 3;
            if (observe) {
                if (!HELP) {
                    if (warp == finisher) {
                        mbar_wait(bar_full + 8 * (row % kFlowRows), (row / kFlowRows) & 1, wait_words, a.fault);
                        finish_row(row % kFlowRows, row0 + row);
                    }
                    finisher = finisher + 1 == ncw ? 0 : finisher + 1;
                }
                ++row;
            }
            if (leave) break;
        }
    }
    __syncthreads();
    if (slice + 1 < a.slices) {
        if (own) write_state(a.y_mid + b * N3);
        return;
    }
    // Final observation of y(t_end): one more static-field evaluation for E.
    if (warp < ncw) {
        double H[NAT][3];
        field_at(NS % 2 == 0 ? 0 : k0 & 1, y, H);
        add_obs(part, y, H);
        if (a.traj && own) write_state(a.traj + (b * a.rows + a.rows - 1) * N3);
        const double r = warp_reduce_many<NV>(part);
        if ((lane % span) == 0) red[warp * NV + lane / span] = r;
    }
    __syncthreads();
    if (warp == 0) finish_row(0, a.rows - 1);
    if (a.y_out && own) write_state(a.y_out + b * N3);
}

}  // namespace cmd
