// resident.cu -- resident RK4 launches: one CTA, or one thread-block cluster of
// 2 or 4 CTAs, per trajectory (rk4_resident.cuh, rk4_cluster.cuh), the variant
// table the autotuner chooses from, and the partner tables of the cluster
// layouts.
#include "cmd_core.h"
#include "rk4_cluster.cuh"
#include "rk4_flow.cuh"
#include "rk4_flow_cluster.cuh"

namespace cmd {
namespace {

template <int NAT, int Z, int LZ, int CPT, int MAXT, int MINB, bool YREG, int TPC>
int launch_one(const cmd_handle* h, const cmd::ResidentArgs& args, const double* d1, const double* d2,
               int64_t B, cudaStream_t st) {
    auto kern = cmd::rk4_resident_kernel<NAT, Z, LZ, CPT, MAXT, MINB, YREG, TPC>;
    const int64_t G = h->lay.G;
    int threads = (int)((G + CPT - 1) / CPT);
    threads = ((threads + 31) / 32) * 32;
    if (threads > MAXT) return fail(CMD_ERR_UNSUPPORTED, "lattice too large for this kernel variant");
    const size_t smem = resident_smem(NAT, G, TPC);
    if (smem > kMaxSmem) return fail(CMD_ERR_UNSUPPORTED, "stage buffers exceed shared memory");
    // Function attributes belong to the current device's context: set on every
    // launch (a host-side call of about a microsecond), so handles on several
    // devices, several host threads and a re-created context all see it.
    CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem));
    cmd::Couplings<NAT, Z> cp;
    fill_couplings<NAT, Z>(h, d1, d2, cp);
    cmd::ResidentArgs a = args;
    a.B = B;
    kern<<<(unsigned)((B + TPC - 1) / TPC), threads, smem, st>>>(cp, a);
    CUDA_TRY(cudaGetLastError());
    return CMD_OK;
}

template <int NAT, int Z, int LZ, int MAXT, int MINB, bool HELP, int NS, bool PAIR>
auto flow_kernel_of(bool stat, bool drive) {
    return stat ? (drive ? rk4_flow_kernel<NAT, Z, LZ, MAXT, MINB, true, true, HELP, NS, PAIR>
                         : rk4_flow_kernel<NAT, Z, LZ, MAXT, MINB, true, false, HELP, NS, PAIR>)
                : (drive ? rk4_flow_kernel<NAT, Z, LZ, MAXT, MINB, false, true, HELP, NS, PAIR>
                         : rk4_flow_kernel<NAT, Z, LZ, MAXT, MINB, false, false, HELP, NS, PAIR>);
}

template <int NAT, int Z, int LZ, int MAXT, int MINB, bool HELP>
auto flow_kernel(const cmd_handle* h, bool drive, int method = CMD_RK4) {
    const bool stat = h->has_field || h->has_onsite;
    if constexpr (Z == 2 * LZ) {
        if (h->lay.paired)
            return method == CMD_SSPRK53 ? flow_kernel_of<NAT, Z, LZ, MAXT, MINB, HELP, kFlowSSPRK53, true>(stat, drive)
                                         : flow_kernel_of<NAT, Z, LZ, MAXT, MINB, HELP, kFlowRK4, true>(stat, drive);
    }
    return method == CMD_SSPRK53 ? flow_kernel_of<NAT, Z, LZ, MAXT, MINB, HELP, kFlowSSPRK53, false>(stat, drive)
                                 : flow_kernel_of<NAT, Z, LZ, MAXT, MINB, HELP, kFlowRK4, false>(stat, drive);
}

// Trajectories the GPU runs at a time.
template <int NAT, int Z, int LZ, int MAXT, int MINB, bool HELP>
int64_t flow_slots(const cmd_handle* h, bool drive) {
    auto kern = flow_kernel<NAT, Z, LZ, MAXT, MINB, HELP>(h, drive);
    const int threads = (int)((h->lay.G + 31) / 32 * 32) + (HELP ? 32 : 0);
    const size_t smem = (size_t)flow_smem_doubles(NAT, MAXT) * sizeof(double);
    int sms = 0, per = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, smem) != cudaSuccess)
        return 0;
    return (int64_t)sms * per;
}

template <int NAT, int Z, int LZ, int MAXT, int MINB, bool HELP>
int launch_flow(const cmd_handle* h, const cmd::ResidentArgs& args, const double* d1, const double* d2,
                int64_t B, cudaStream_t st) {
    auto kern = flow_kernel<NAT, Z, LZ, MAXT, MINB, HELP>(h, args.drive != nullptr, args.method);
    const int64_t G = h->lay.G;
    const int threads = (int)((G + 31) / 32 * 32) + (HELP ? 32 : 0);
    if (threads > MAXT) return fail(CMD_ERR_UNSUPPORTED, "lattice too large for this kernel variant");
    const size_t smem = (size_t)cmd::flow_smem_doubles(NAT, MAXT) * sizeof(double);
    CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem));
    cmd::Couplings<NAT, Z> cp;
    fill_couplings<NAT, Z>(h, d1, d2, cp);
    cmd::ResidentArgs a = args;
    a.B = B;
    a.fault = h->hfault.as<int>();
    a.wait_ns = (unsigned long long)h->wait_ns;
    a.row_ns = flow_row_ns(a.wait_ns, (unsigned long long)std::min<int64_t>(a.save_every, a.n_steps));
    if (h->lay.paired) a.nbr = h->nbrp.as<int>();
    // items are (slice, trajectory), trajectories fastest: the earlier slice of an item ran in an earlier launch
    // (slots <= B), so stream order is the only dependence
    const int64_t items = B * a.slices, per = a.slices > 1 ? a.slots : items;
    for (int64_t i = 0; i < items; i += per) {
        a.item0 = i;
        kern<<<(unsigned)std::min(per, items - i), threads, smem, st>>>(cp, a);
        CUDA_TRY(cudaGetLastError());
    }
    return CMD_OK;
}

template <int NAT, int Z, int LZ, int CS, int MAXT>
auto flow_cluster_kernel(const cmd_handle* h, bool drive) {
    const bool stat = h->has_field || h->has_onsite;
    auto of = [&](auto pair) {
        constexpr bool P = decltype(pair)::value != 0;
        return stat ? (drive ? rk4_flow_cluster_kernel<NAT, Z, LZ, CS, MAXT, true, true, P>
                             : rk4_flow_cluster_kernel<NAT, Z, LZ, CS, MAXT, true, false, P>)
                    : (drive ? rk4_flow_cluster_kernel<NAT, Z, LZ, CS, MAXT, false, true, P>
                             : rk4_flow_cluster_kernel<NAT, Z, LZ, CS, MAXT, false, false, P>);
    };
    if constexpr (Z == 2 * LZ) {
        if (h->lay.paired) return of(AtomTag<1>{});
    }
    return of(AtomTag<0>{});
}

template <int NAT, int CS, int MAXT>
cudaLaunchConfig_t flow_cluster_config(const cmd_handle* h, int64_t clusters, cudaStream_t st, cudaLaunchAttribute* attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * CS));
    cfg.blockDim = dim3((unsigned)((cluster_cells(h->lay.G, CS) + 31) / 32 * 32 + 32));
    cfg.dynamicSmemBytes = (size_t)flow_cluster_smem_doubles(NAT, MAXT, CS) * sizeof(double);
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

template <int NAT, int Z, int LZ, int CS, int MAXT>
int64_t flow_cluster_slots(const cmd_handle* h, bool drive) {
    auto kern = flow_cluster_kernel<NAT, Z, LZ, CS, MAXT>(h, drive);
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = flow_cluster_config<NAT, CS, MAXT>(h, 1, nullptr, attr);
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, (const void*)kern, &cfg) != cudaSuccess)
        return 0;
    return n;
}

template <int NAT, int Z, int LZ, int CS, int MAXT>
int launch_flow_cluster(const cmd_handle* h, const cmd::ResidentArgs& args, const double* d1, const double* d2,
                        int64_t B, cudaStream_t st) {
    auto kern = flow_cluster_kernel<NAT, Z, LZ, CS, MAXT>(h, args.drive != nullptr);
    CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem));
    cmd::Couplings<NAT, Z> cp;
    fill_couplings<NAT, Z>(h, d1, d2, cp);
    cmd::ResidentArgs a = args;
    a.B = B;
    a.fault = h->hfault.as<int>();
    a.wait_ns = (unsigned long long)h->wait_ns;
    a.row_ns = flow_row_ns(a.wait_ns, (unsigned long long)std::min<int64_t>(a.save_every, a.n_steps));
    FlowClusterArgs fc{};
    const Layout::FlowCluster& t = h->lay.flow_cluster[CS];
    fc.Gc = (int)cluster_cells(h->lay.G, CS);
    fc.pw = h->fctab[CS].as<int>();
    fc.push = fc.pw + t.pw.size();
    fc.peers = fc.push + t.push.size();
    const int64_t items = B * a.slices, per = a.slices > 1 ? a.slots : items;   // as launch_flow
    for (int64_t i = 0; i < items; i += per) {
        a.item0 = i;
        cudaLaunchAttribute attr[1];
        cudaLaunchConfig_t cfg = flow_cluster_config<NAT, CS, MAXT>(h, std::min(per, items - i), st, attr);
        CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, cp, a, fc));
    }
    return CMD_OK;
}

template <int NAT, int Z, int LZ, int CS, int MAXT>
int launch_cluster(const cmd_handle* h, const cmd::ResidentArgs& args, const double* d1, const double* d2,
                   int64_t B, cudaStream_t st) {
    auto kern = cmd::rk4_cluster_kernel<NAT, Z, LZ, CS, MAXT>;
    const int64_t G = h->lay.G, Gc = cluster_cells(G, CS);
    const int threads = (int)((Gc + 31) / 32 * 32);
    if (threads > MAXT) return fail(CMD_ERR_UNSUPPORTED, "lattice too large for this cluster variant");
    const size_t smem = cluster_smem(NAT, G, CS);
    if (smem > kMaxSmem) return fail(CMD_ERR_UNSUPPORTED, "stage buffers exceed shared memory");
    const DevBuf& tab = CS == 2 ? h->cnbr2 : h->cnbr4;
    if (!tab.p) return fail(CMD_ERR_UNSUPPORTED, "no cluster neighbour table for this lattice");
    // Function attributes belong to the current device's context: set on every
    // launch (a host-side call of about a microsecond), so handles on several
    // devices, several host threads and a re-created context all see it.
    CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem));
    cmd::Couplings<NAT, Z> cp;
    fill_couplings<NAT, Z>(h, d1, d2, cp);
    cmd::ResidentArgs a = args;
    a.B = B;
    a.nbr = static_cast<const int*>(tab.p);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(B * CS));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, cp, a, (int)Gc));
    return CMD_OK;
}

const StageTimes kSSPRK53Times = {
    5, {0.0, 0.377268915331368, 0.754537830662736, 0.728985661612188, 0.699226135931670, 0.0, 0.0, 0.0}};

#define CMD_VARIANT(NAT, Z, LZ, CPT, MAXT, MINB, YREG, TPC) \
    Variant{NAT, Z, LZ, CPT, MAXT, MINB, YREG, TPC, 1, false, &launch_one<NAT, Z, LZ, CPT, MAXT, MINB, YREG, TPC>, \
            "rk4_resident<" #NAT "," #Z "," #LZ "> cpt=" #CPT " maxt=" #MAXT " minb=" #MINB " yreg=" #YREG \
            " tpc=" #TPC}
#define CMD_FLOW(NAT, Z, LZ, MAXT, MINB, HELP) \
    Variant{NAT, Z, LZ, 1, MAXT, MINB, true, 1, 1, true, &launch_flow<NAT, Z, LZ, MAXT, MINB, HELP>, \
            "rk4_flow<" #NAT "," #Z "," #LZ "> maxt=" #MAXT " minb=" #MINB " help=" #HELP, HELP, \
            &flow_slots<NAT, Z, LZ, MAXT, MINB, HELP>}
#define CMD_FLOW_CLUSTER(NAT, Z, LZ, CS, MAXT) \
    Variant{NAT, Z, LZ, 1, MAXT, 1, true, 1, CS, true, &launch_flow_cluster<NAT, Z, LZ, CS, MAXT>, \
            "rk4_cluster_flow<" #NAT "," #Z "," #LZ "> cs=" #CS " maxt=" #MAXT, true, \
            &flow_cluster_slots<NAT, Z, LZ, CS, MAXT>}
#define CMD_CLUSTER(NAT, Z, LZ, CS, MAXT) \
    Variant{NAT, Z, LZ, 1, MAXT, 1, true, 1, CS, false, &launch_cluster<NAT, Z, LZ, CS, MAXT>, \
            "rk4_cluster<" #NAT "," #Z "," #LZ "> cs=" #CS " maxt=" #MAXT}

const Variant kVariants[] = {
    // 2-atom cells with 3 bonds per site (Kitaev / Heisenberg honeycomb)
    // shorter rows for small lattices: more CTAs per SM
    CMD_FLOW(2, 3, 1, 160, 4, true),
    CMD_FLOW(2, 3, 1, 288, 2, true),
    CMD_FLOW(2, 3, 1, 640, 1, true),
    CMD_FLOW(2, 3, 1, 640, 1, false),
    CMD_VARIANT(2, 3, 1, 1, 640, 1, true, 1),
    CMD_VARIANT(2, 3, 1, 2, 320, 2, false, 1),
    CMD_VARIANT(2, 3, 1, 3, 192, 3, false, 1),
    CMD_VARIANT(2, 3, 1, 4, 160, 3, false, 1),
    CMD_VARIANT(2, 3, 1, 4, 160, 3, true, 1),
    CMD_VARIANT(2, 3, 1, 6, 96, 3, true, 1),
    CMD_VARIANT(2, 3, 1, 2, 512, 1, true, 1),
    CMD_VARIANT(2, 3, 1, 4, 256, 2, false, 1),
    // two trajectories per CTA: twice the independent work between barriers
    CMD_VARIANT(2, 3, 1, 1, 640, 1, false, 2),
    CMD_VARIANT(2, 3, 1, 1, 640, 1, true, 2),
    CMD_VARIANT(2, 3, 1, 2, 320, 1, false, 2),
    // one trajectory over a cluster of 2 or 4 CTAs (distributed shared memory)
    CMD_FLOW_CLUSTER(2, 3, 1, 2, 640),
    CMD_FLOW_CLUSTER(2, 3, 1, 4, 640),
    CMD_CLUSTER(2, 3, 1, 2, 640),
    CMD_CLUSTER(2, 3, 1, 4, 640),
    // 4-atom cells with 6 bonds per site (nearest-neighbour pyrochlore)
    CMD_FLOW(4, 6, 3, 256, 1, false),
    CMD_VARIANT(4, 6, 3, 1, 512, 1, true, 1),
    CMD_VARIANT(4, 6, 3, 2, 256, 2, false, 1),
    CMD_VARIANT(4, 6, 3, 2, 512, 1, false, 1),
    CMD_FLOW_CLUSTER(4, 6, 3, 2, 512),
    CMD_FLOW_CLUSTER(4, 6, 3, 4, 512),
    CMD_CLUSTER(4, 6, 3, 2, 512),
    CMD_CLUSTER(4, 6, 3, 4, 512),
};
constexpr int kNumVariants = (int)(sizeof(kVariants) / sizeof(kVariants[0]));

}  // namespace

const Variant* variant_table() { return kVariants; }
int variant_count() { return kNumVariants; }

// Partner table of the CS-CTA cluster kernel: the resident table's offsets
// (atom*3)*G + cell become (rank << 24) | ((atom*3)*Gc + cell - rank*Gc) with
// Gc = ceil(G / CS) cells per CTA.  Built once per handle.
int upload_cluster_table(cmd_handle* h, int cs) {
    DevBuf& d = cs == 2 ? h->cnbr2 : h->cnbr4;
    if (d.p) return CMD_OK;
    const Layout& L = h->lay;
    const int64_t G = L.G, Gc = cluster_cells(G, cs);
    if ((int64_t)L.NA * 3 * Gc >= (1 << cmd::kClusterRankShift)) return CMD_OK;   // never launched
    std::vector<int> t(L.nbr.size(), 0);
    for (size_t i = 0; i < L.nbr.size(); ++i) {
        const int64_t off = L.nbr[i];
        const int64_t at = off / (3 * G), c = off - at * 3 * G;     // partner atom*3 block and cell
        const int64_t gp = c % G, comp = c / G;                     // comp is 0 for the offsets stored
        const int64_t r = gp / Gc, l = gp - r * Gc;
        t[i] = (int)((r << cmd::kClusterRankShift) | ((at * 3 + comp) * Gc + l));
    }
    return upload_once(d, t.data(), t.size() * sizeof(int), "cluster neighbour table");
}

// Partner words of the cluster layout with CS CTAs (CS = 1: the global offsets, rank 0).
const int* cluster_table(const cmd_handle* h, int cs) {
    return cs == 1 ? h->nbr.as<int>() : static_cast<const int*>((cs == 2 ? h->cnbr2 : h->cnbr4).p);
}

// Tables of rk4_flow_cluster_kernel for clusters of cs CTAs of up to maxt - 32 cells: partner offsets (own or halo
// column), push words, and the peers of every warp.  False when a row needs more halo columns than flow_halo, or a
// warp has more than kFlowPeers peers.
bool flow_cluster_plan(const Layout& L, int cs, int maxt) {
    Layout::FlowCluster& F = L.flow_cluster[cs];
    if (F.fits >= 0) return F.fits == 1;
    F.fits = 0;
    const int NA = L.NA, NL = L.Z - L.LZ;
    const int64_t G = L.G, Gc = cluster_cells(G, cs), row = maxt + flow_halo(NA), nw = (Gc + 31) / 32;
    std::vector<int> col;
    if (NL == 0 || halo_columns(L, cs, Gc, &col) > flow_halo(NA)) return false;
    const std::vector<int>& nbr = L.paired ? L.nbr_pair : L.nbr;
    std::vector<int> pw(nbr.size(), 0), push(nbr.size(), -1);
    std::vector<std::vector<int>> peers((size_t)cs * nw);
    auto join = [&](int64_t a, int64_t b) {          // warps (rank * nw + warp), both ways
        for (int k = 0; k < 2; ++k, std::swap(a, b)) {
            const int w = (int)((b / nw) << 8 | b % nw);
            std::vector<int>& p = peers[a];
            if (std::find(p.begin(), p.end(), w) == p.end()) p.push_back(w);
        }
    };
    for (int64_t i = 0; i < (int64_t)peers.size(); ++i) join(i, i);
    for (size_t i = 0; i < nbr.size(); ++i) {
        const int64_t site = (int64_t)(i / NL), g = site / NA, r = g / Gc;
        const int64_t pat = nbr[i] / (3 * G), gp = nbr[i] - pat * 3 * G, rp = gp / Gc;
        join(r * nw + (g - r * Gc) / 32, rp * nw + (gp - rp * Gc) / 32);
        if (rp == r) {
            pw[i] = (int)(pat * 3 * row + gp - r * Gc);
            continue;
        }
        const int64_t slot = pat * 3 * row + maxt + col[((size_t)r * G + gp) * NA + pat];
        pw[i] = (int)slot;
        int* to = &push[((size_t)gp * NA + pat) * NL];
        const int word = (int)(r << kClusterRankShift | slot);
        int k = 0;
        while (k < NL && to[k] >= 0 && to[k] != word) ++k;
        if (k == NL) return false;                   // read by more CTAs than it has bonds
        to[k] = word;
    }
    F.peers.assign(peers.size() * kFlowPeers, -1);
    for (size_t i = 0; i < peers.size(); ++i) {
        if (peers[i].size() > (size_t)kFlowPeers) return false;
        std::copy(peers[i].begin(), peers[i].end(), F.peers.begin() + i * kFlowPeers);
    }
    F.pw = std::move(pw);
    F.push = std::move(push);
    F.fits = 1;
    return true;
}

int prepare_variant(cmd_handle* h, int vi) {
    const Variant& V = kVariants[vi];
    if (V.CS == 1) return CMD_OK;
    if (!V.flow) return upload_cluster_table(h, V.CS);
    DevBuf& d = h->fctab[V.CS];
    if (d.p) return CMD_OK;
    const Layout::FlowCluster& t = h->lay.flow_cluster[V.CS];
    std::vector<int> all(t.pw);
    all.insert(all.end(), t.push.begin(), t.push.end());
    all.insert(all.end(), t.peers.begin(), t.peers.end());
    return upload_once(d, all.data(), all.size() * sizeof(int), "cluster flow table");
}

bool variant_fits(const Variant& v, const Layout& L) {
    if (!L.uniform || v.NAT != L.NA || v.Z != L.Z || v.LZ != L.LZ) return false;
    if (v.flow) {
        for (int a = 0; a < L.NA; ++a)
            if (L.zc[a] != L.Z) return false;
        if (v.CS > 1) {
            const int64_t Gc = cluster_cells(L.G, v.CS);
            return Gc >= 32 && (Gc + 31) / 32 * 32 + 32 <= v.MAXT &&
                   (size_t)flow_cluster_smem_doubles(v.NAT, v.MAXT, v.CS) * sizeof(double) <= kMaxSmem &&
                   flow_cluster_plan(L, v.CS, v.MAXT);
        }
        return (L.G + 31) / 32 * 32 + (v.help ? 32 : 0) <= v.MAXT &&
               (size_t)flow_smem_doubles(v.NAT, v.MAXT) * sizeof(double) <= kMaxSmem;
    }
    if (v.CS > 1) {
        const int64_t Gc = cluster_cells(L.G, v.CS);
        return Gc >= 32 && (Gc + 31) / 32 * 32 <= v.MAXT && cluster_smem(v.NAT, L.G, v.CS) <= kMaxSmem &&
               (int64_t)v.NAT * 3 * Gc < (1 << cmd::kClusterRankShift);
    }
    const int64_t threads = ((L.G + v.CPT - 1) / v.CPT + 31) / 32 * 32;
    if (threads > v.MAXT) return false;
    const size_t smem = resident_smem(v.NAT, L.G, v.TPC);
    if (smem > kMaxSmem) return false;
    return true;
}

// Variant used when the caller did not pick one: the first fitting entry of
// the table (entries are ordered by preference for a lone trajectory).
int default_variant(const Layout& L) {
    for (int i = 0; i < kNumVariants; ++i)
        if (variant_fits(kVariants[i], L)) return i;
    return -1;
}

// The fixed-step methods other than RK4 that run resident (SSPRK53) use the first flow variant that fits.
int flow_variant(const Layout& L) {
    for (int i = 0; i < kNumVariants; ++i)
        if (kVariants[i].flow && kVariants[i].CS == 1 && variant_fits(kVariants[i], L)) return i;
    return -1;
}

int no_instance(const Layout& L) {
    if (!L.uniform) return fail(CMD_ERR_UNSUPPORTED, "lattice layout not supported: " + L.why);
    char buf[200];
    std::snprintf(buf, sizeof(buf),
                  "no resident kernel for %d atoms/cell, %d bonds/site, %d local, %lld cells",
                  L.NA, L.Z, L.LZ, (long long)L.G);
    return fail(CMD_ERR_UNSUPPORTED, buf);
}

int pick_variant(const cmd_handle* h) {
    if (h->variant >= 0 && h->variant < kNumVariants && variant_fits(kVariants[h->variant], h->lay))
        return h->variant;
    return default_variant(h->lay);
}

// Steps split into slices so that the last, partly filled wave of a batch costs less.  A run of B trajectories on
// `slots` resident CTAs takes ceil(B / slots) times its steps; cut into K slices, every slots (slice, trajectory)
// items one launch, ceil(B K / slots) times a K-th of them, plus the start of each launch (kSliceSteps steps' time:
// launch gap, state, peer masks).  K is the cheapest up to kMaxSlices; one slice unless that saves over 2 %.
// 768 trajectories of the 24x24 honeycomb on 148 SMs, 2000 steps: 6 waves become 5.2 (figures at rk4_flow.cuh).
void plan_slices(const cmd_handle* h, const Variant& V, int64_t B, int64_t n_steps, ResidentArgs& a) {
    constexpr int64_t kSliceSteps = 5, kMaxSlices = 32;
    a.slices = 1;
    a.slots = V.slots ? V.slots(h, a.drive != nullptr) : 0;
    if (a.slots <= 0 || B <= a.slots) return;
    auto cost = [&](int64_t k) { return (B * k + a.slots - 1) / a.slots * ((n_steps + k - 1) / k + kSliceSteps); };
    int64_t best = 1;
    for (int64_t k = 2; k <= kMaxSlices && k <= n_steps; ++k)
        if (cost(k) < cost(best)) best = k;
    if (cost(best) * 50 < cost(1) * 49) a.slices = best;
}

// Slices need the final states' memory, and that memory must not hold the one initial state that every trajectory's
// first slice reads.
bool may_slice(const RunSpec& r, int64_t n3) {
    if (!r.y_out) return false;
    return r.y0_stride != 0 || r.y0 + n3 <= r.y_out || r.y_out + r.B * n3 <= r.y0;
}

int64_t resident_launches(const ResidentArgs& a, int64_t B) {
    return a.slices > 1 ? (B * a.slices + a.slots - 1) / a.slots : 1;
}

// The cluster flow kernel that batch_variant may choose in place of default variant vi, or -1.
static int cluster_alternative(const Layout& L, int vi) {
    if (vi < 0 || kVariants[vi].CS > 1 || kVariants[vi].flow) return -1;
    for (int i = 0; i < kNumVariants; ++i)
        if (kVariants[i].flow && kVariants[i].CS > 1 && variant_fits(kVariants[i], L)) return i;
    return -1;
}

// The variant of a batch of B trajectories: the handle's, but where nothing was pinned and the default is a
// one-CTA kernel with a stage barrier, the cluster flow kernel if every trajectory's cluster is resident at once (SMs
// would idle otherwise), or always where that CTA would hold two 4-atom cells per thread.  B200, per stage and
// trajectory, one CTA against clusters of 2: honeycomb 27x31 1.63 us on one SM, 0.94 us on two; pyrochlore 500 cells
// 2.47 / 1.93 us, 864 cells (two per thread, spills) 8.66 / 2.84 us.  The line does not count what slices give the
// clusters of a larger batch: by these figures they would lead a little further (to about 1.7 waves of clusters).
// The two kernels add in different orders, so a trajectory's last bits depend on B there (cmd_batch_variant).
int batch_variant(const cmd_handle* h, int64_t B, bool drive) {
    const int vi = pick_variant(h);
    if (vi < 0 || vi == h->variant || kVariants[vi].CS > 1) return vi;
    if (kVariants[vi].flow) {
        // a helper warp can cost a CTA per SM: batches that need the CTA more go without
        const int64_t slots = kVariants[vi].slots(h, drive);
        for (int i = vi + 1; i < kNumVariants && kVariants[vi].help && B > slots; ++i) {
            const Variant& v = kVariants[i];
            if (v.flow && v.CS == 1 && !v.help && variant_fits(v, h->lay)) return v.slots(h, drive) > slots ? i : vi;
        }
        return vi;
    }
    const int alt = cluster_alternative(h->lay, vi);
    if (alt < 0) return vi;
    return (kVariants[vi].NAT == 4 && kVariants[vi].CPT > 1) || B <= kVariants[alt].slots(h, drive) ? alt : vi;
}

// Uploads the tables of every variant that batches of h may run without a pin.
int prepare_defaults(cmd_handle* h) {
    const int vi = default_variant(h->lay);
    if (vi < 0) return CMD_OK;
    if (int rc = prepare_variant(h, vi)) return rc;
    const int alt = cluster_alternative(h->lay, vi);
    return alt >= 0 ? prepare_variant(h, alt) : CMD_OK;
}

// Room for the envelope table of n_steps driven SSPRK53 steps.
bool stages_room(cmd_handle* h, int64_t n_steps) {
    if (h->amp == 0.0 || n_steps <= 0) return true;
    if (h->times.ensure((size_t)n_steps * sizeof(double)) == CMD_OK &&
        h->drive.ensure((size_t)n_steps * 2 * kSSPRK53Times.n * sizeof(double)) == CMD_OK)
        return true;
    cudaGetLastError();
    clear_error();
    return false;
}

// Launches drive-table pre-pass (when driven), the resident kernel and the
// row-finishing post-pass on `st`.  Asynchronous; returns the launch count.
int run_resident(cmd_handle* h, const RunSpec& r, cudaStream_t st, int32_t* launches) {
    int32_t nl = 0;
    const int vi = r.method != CMD_RK4 ? flow_variant(h->lay)
                   : r.variant >= 0    ? r.variant
                                       : batch_variant(h, r.B, r.pulses && r.n_steps > 0);
    if (vi < 0 || !variant_fits(kVariants[vi], h->lay)) return no_instance(h->lay);
    const Variant& V = kVariants[vi];
    if (int rc = prepare_variant(h, vi)) return rc;
    const int64_t rows = rows_for(r.n_steps, r.save);
    const int NR = 3 * V.NAT + 1;
    cmd::ResidentArgs a{};
    a.method = r.method;
    a.G = (int)h->lay.G;
    a.n_steps = r.n_steps;
    a.save_every = r.save;
    a.T0 = r.T0;
    a.dt = r.dt;
    a.nbr = h->nbr.as<int>();
    a.y0 = r.y0;
    a.y0_stride = r.y0_stride;
    a.y_out = r.y_out;
    a.rows = rows;
    a.traj = r.traj;
    a.drive = nullptr;
    if (r.obs) {
        if (NR <= 10) {
            a.raw = r.obs;
            a.raw_stride = 10;
        } else {
            if (int rc = h->raw.ensure((size_t)r.B * rows * NR * sizeof(double))) return rc;
            a.raw = h->raw.as<double>();
            a.raw_stride = NR;
        }
    }
    if (r.pulses && r.n_steps > 0) {
        std::vector<double> grid;
        grid.reserve(r.n_steps + 1);
        double t = r.T0;
        for (int64_t k = 0; k < r.n_steps; ++k) {     // t_k of the reference loop (t += dt)
            grid.push_back(t);
            t += r.dt;
        }
        if (int rc = h->times.ensure(grid.size() * sizeof(double))) return rc;
        const int ne = r.method == CMD_SSPRK53 ? 2 * kSSPRK53Times.n : 6;
        if (int rc = h->drive.ensure((size_t)r.B * r.n_steps * ne * sizeof(double))) return rc;
        CUDA_TRY(cudaMemcpyAsync(h->times.p, grid.data(), grid.size() * sizeof(double), cudaMemcpyHostToDevice, st));
        a.drive = h->drive.as<double>();
    }
    if (r.obs && V.NAT != 2 && V.NAT != 4) return fail(CMD_ERR_UNSUPPORTED, "no row finisher for this cell size");
    // slices keep their states in the caller's final states (nothing of the handle's: calls without a drive may
    // overlap on several streams)
    a.slices = 1;
    if (may_slice(r, h->N * 3)) plan_slices(h, V, r.B, r.n_steps, a);
    a.y_mid = r.y_out;
    static const std::vector<double> zeros(3 * 64, 0.0);
    const double* d1 = r.d1 ? r.d1 : zeros.data();
    const double* d2 = r.d2 ? r.d2 : zeros.data();
    // drive table, the resident kernel and the row finisher: one graph
    const int rc = graph_call(h, kGraphResident, st, [&]() -> int {
        if (a.drive) {
            const int64_t total = r.B * r.n_steps * 6;
            const int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 32);
            if (r.method == CMD_SSPRK53)
                cmd::drive_stages_kernel<<<blocks, 256, 0, st>>>(r.pulses, h->times.as<double>(), r.n_steps, r.dt,
                                                                r.width, r.freq, kSSPRK53Times, h->drive.as<double>());
            else
                cmd::drive_table_kernel<<<blocks, 256, 0, st>>>(r.pulses, h->times.as<double>(), r.n_steps, r.dt,
                                                               r.width, r.freq, r.B, h->drive.as<double>());
            CUDA_TRY(cudaGetLastError());
            ++nl;
        }
        if (int rc2 = V.fn(h, a, d1, d2, r.B, st)) return rc2;
        nl += (int32_t)resident_launches(a, r.B);
        if (r.obs) {
            const int64_t n = r.B * rows;
            const double* fr = r.frames ? r.frames : h->dframes.as<double>();
            const double* af = r.afm ? r.afm : h->dafm.as<double>();
            if (V.NAT == 2) launch_finish<2>(a.raw, a.raw_stride, n, fr, af, r.n_sites, r.obs, st);
            else launch_finish<4>(a.raw, a.raw_stride, n, fr, af, r.n_sites, r.obs, st);
            CUDA_TRY(cudaGetLastError());
            ++nl;
        }
        return CMD_OK;
    });
    if (rc != CMD_OK) return rc;
    if (launches) *launches = nl;
    return CMD_OK;
}

void variant_shape(const Variant& V, const Layout& L, int64_t* threads, int64_t* smem) {
    if (V.flow && V.CS == 1) {
        *threads = (L.G + 31) / 32 * 32;             // threads with cells
        *smem = (int64_t)flow_smem_doubles(V.NAT, V.MAXT) * (int64_t)sizeof(double);
    } else if (V.CS > 1) {
        *threads = (cluster_cells(L.G, V.CS) + 31) / 32 * 32;   // threads with cells; own cells' shared memory
        *smem = (int64_t)cluster_smem(L.NA, L.G, V.CS);
    } else {
        *threads = ((L.G + V.CPT - 1) / V.CPT + 31) / 32 * 32;
        *smem = (int64_t)resident_smem(L.NA, L.G, V.TPC);
    }
}

}  // namespace cmd
