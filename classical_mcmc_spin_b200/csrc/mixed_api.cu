// mixed_api.cu -- C ABI of the mixed SU(2) / SU(3) path (cmd_mixed.h): the
// handle owns the device copies of the lattice tables, the state and the
// integrator workspace; every call runs on the handle's stream.
#include "cmd.h"
#include "cmd_mixed.h"
#include "cmd_internal.h"
#include "mixed_tiles.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <map>
#include <string>
#include <vector>

using cmd::fail;

#define MIX_TRY(x)                                                                               \
    do {                                                                                         \
        cudaError_t e_ = (x);                                                                    \
        if (e_ != cudaSuccess) return fail(CMD_ERR_CUDA, std::string(#x ": ") + cudaGetErrorString(e_)); \
    } while (0)

struct cmd_mixed {
    cmd::MixedDev m{};
    int64_t V = 0;
    cmd::DevBuf tables;        // distinct couplings and index arrays, one allocation
    cmd::DevBuf drive2, drive3;
    cmd::DevBuf state, work, rows, mag;
    // tiles of like sites, state on chip (mixed_tiles.cuh), where the lattice fits; tcs = 0: it does not
    cmd::MixedTilesDev td{};
    int tcs = 0, tthreads = 0, tpw = 1;
    cmd::DevBuf ttab, tints, tfact, ttimes;
    bool has_state = false;
    cudaStream_t stream = nullptr;
    ~cmd_mixed() {
        for (cmd::DevBuf* b : {&tables, &drive2, &drive3, &state, &work, &rows, &mag, &ttab, &tints, &tfact, &ttimes})
            b->release();
    }
};

namespace {

size_t pad(size_t bytes) { return (bytes + 255) / 256 * 256; }

constexpr size_t kMixedSmemMax = 200 * 1024;   // distinct couplings copied to shared memory up to this size

// Distinct blocks of w doubles in first-seen order, and the index of each block added.
struct Distinct {
    int w;
    std::vector<double> vals;
    std::map<std::vector<double>, int> seen;
    explicit Distinct(int w_) : w(w_) {}
    // `hint`: the block that the same slot of an earlier like atom had, tried first (and updated)
    int add(const double* p, int& hint) {
        if (hint >= 0 && std::memcmp(p, &vals[(size_t)hint * w], w * sizeof(double)) == 0) return hint;
        return hint = add(p);
    }
    int add(const double* p) {
        std::vector<double> k(p, p + w);
        auto it = seen.find(k);
        if (it != seen.end()) return it->second;
        const int id = (int)(vals.size() / w);
        vals.insert(vals.end(), k.begin(), k.end());
        seen.emplace(std::move(k), id);
        return id;
    }
};

// One kind of site: distinct field / on-site / bond / mixed-bond blocks, and the
// per-site and per-(slot, site) indices (slot-major: index n * N + s).
struct KindTables {
    std::vector<int> fi, oi, bi, part, cnt, mi, mpart, mcnt;
};

void build_kind(int64_t N, int NA, int z, int zm, int dim, const double* field, const double* onsite,
                const double* bil, const int64_t* partners, const int64_t* counts, int64_t limit_same,
                const double* mix, const int64_t* mpartners, const int64_t* mcounts, int64_t limit_other,
                Distinct& F, Distinct& O, Distinct& B, Distinct& M, KindTables& t) {
    t.fi.assign(N, 0); t.oi.assign(N, 0); t.cnt.assign(N, 0); t.mcnt.assign(N, 0);
    t.bi.assign((size_t)N * z, 0); t.part.assign((size_t)N * z, -1);
    t.mi.assign((size_t)N * zm, 0); t.mpart.assign((size_t)N * zm, -1);
    std::vector<int> hints((size_t)NA * (2 + z + zm), -1);
    for (int64_t s = 0; s < N; ++s) {
        int* hint = &hints[(size_t)(s % NA) * (2 + z + zm)];
        t.fi[s] = F.add(field + (size_t)s * dim, hint[0]);
        t.oi[s] = O.add(onsite + (size_t)s * dim * dim, hint[1]);
        t.cnt[s] = (int)std::max<int64_t>(0, std::min<int64_t>(counts[s], z));
        for (int n = 0; n < t.cnt[s]; ++n) {
            const int64_t p = partners[(size_t)s * z + n];
            if (p < 0 || p >= limit_same) continue;
            t.part[(size_t)n * N + s] = (int)p;
            t.bi[(size_t)n * N + s] = B.add(bil + ((size_t)s * z + n) * dim * dim, hint[2 + n]);
        }
        t.mcnt[s] = zm > 0 ? (int)std::max<int64_t>(0, std::min<int64_t>(mcounts[s], zm)) : 0;
        for (int n = 0; n < t.mcnt[s]; ++n) {
            const int64_t p = mpartners[(size_t)s * zm + n];
            if (p < 0 || p >= limit_other) continue;
            t.mpart[(size_t)n * N + s] = (int)p;
            t.mi[(size_t)n * N + s] = M.add(mix + ((size_t)s * zm + n) * 24, hint[2 + z + n]);
        }
    }
}

int method_mode(int method) {
    switch (method) {
        case CMD_RK4: return cmd::kModeRK4;
        case CMD_DOPRI5_FIXED: return cmd::kModeDopri5Fixed;
        case CMD_CASH_KARP_FIXED: return cmd::kModeCashKarpFixed;
        case CMD_EULER: return cmd::kModeEuler;
        case CMD_MIDPOINT: return cmd::kModeMidpoint;
        case CMD_SSPRK53: return cmd::kModeSSPRK53;
        case CMD_RK78: return cmd::kModeRK78;
        case CMD_BULIRSCH_STOER: return cmd::kModeBulirschStoer;
        default: return -1;
    }
}

// Reference loop (integrator.cuh:470-488): steps taken and the times of the saved rows.
int64_t loop_steps(double T0, double T1, double dt, std::vector<double>* grid) {
    int64_t n = 0;
    double t = T0;
    if (grid) grid->clear();
    while (t < T1) {
        if (grid) grid->push_back(t);
        t += dt;
        ++n;
    }
    if (grid) grid->push_back(t);
    return n;
}

template <int CS>
cudaLaunchConfig_t config(cmd_mixed* h, int threads, cudaLaunchAttribute* attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CS);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = h->m.tab_in_smem ? (size_t)h->m.tab_doubles * sizeof(double) : 0;
    cfg.stream = h->stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Function attributes belong to the current device's context, so they are set
// before every launch (a host-side call of about a microsecond): handles on
// several devices, several host threads and a re-created context all see them.
template <int CS>
int set_attributes() {
    auto kern = cmd::mixed_integrate_kernel<CS>;
    MIX_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMixedSmemMax));
    if (CS > 8) MIX_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    return CMD_OK;
}

template <int CS>
int launch_cs(cmd_mixed* h, const cmd::MixedRun& r, int threads) {
    if (int rc = set_attributes<CS>()) return rc;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = config<CS>(h, threads, attr);
    MIX_TRY(cudaLaunchKernelEx(&cfg, cmd::mixed_integrate_kernel<CS>, h->m, r));
    return CMD_OK;
}

// ---- tiles of eight like sites (mixed_tiles.cuh)

constexpr size_t kTilesSmemMax = 232448;       // 227 KB dynamic shared memory per CTA on sm_100
constexpr int kTilesWarps = 16;                // warps per CTA, one or two tiles each

using TilesKernel = void (*)(const cmd::MixedTilesDev, const cmd::MixedRun);

template <int MODE>
TilesKernel tiles_kernel_of(int tpw) {
    return tpw == 1 ? (TilesKernel)cmd::mixed_tiles_kernel<MODE, 1> : (TilesKernel)cmd::mixed_tiles_kernel<MODE, 2>;
}

TilesKernel tiles_kernel(int mode, int tpw) {
    switch (mode) {
        case cmd::kModeRK4: return tiles_kernel_of<cmd::kModeRK4>(tpw);
        case cmd::kModeDopri5Fixed: return tiles_kernel_of<cmd::kModeDopri5Fixed>(tpw);
        case cmd::kModeCashKarpFixed: return tiles_kernel_of<cmd::kModeCashKarpFixed>(tpw);
        case cmd::kModeEuler: return tiles_kernel_of<cmd::kModeEuler>(tpw);
        case cmd::kModeMidpoint: return tiles_kernel_of<cmd::kModeMidpoint>(tpw);
        case cmd::kModeSSPRK53: return tiles_kernel_of<cmd::kModeSSPRK53>(tpw);
        case cmd::kModeRK78: return tiles_kernel_of<cmd::kModeRK78>(tpw);
        default: return nullptr;
    }
}

cmd::MixedStageTimes tiles_stage_times(int mode) {
    using cmd::MixedStageTimes;
    switch (mode) {
        case cmd::kModeEuler: return MixedStageTimes{1, {0.0}};
        case cmd::kModeMidpoint: return MixedStageTimes{2, {0.0, 0.5}};
        case cmd::kModeRK4: return MixedStageTimes{4, {0.0, 0.5, 0.5, 1.0}};
        case cmd::kModeSSPRK53:
            return MixedStageTimes{5, {0.0, 0.377268915331368, 0.754537830662736, 0.728985661612188, 0.699226135931670}};
        case cmd::kModeDopri5Fixed: return MixedStageTimes{6, {0.0, 1.0 / 5.0, 3.0 / 10.0, 4.0 / 5.0, 8.0 / 9.0, 1.0}};
        case cmd::kModeCashKarpFixed: return MixedStageTimes{6, {0.0, 1.0 / 5.0, 3.0 / 10.0, 3.0 / 5.0, 1.0, 7.0 / 8.0}};
        default:
            return MixedStageTimes{11, {0.0, 2.0 / 27.0, 1.0 / 9.0, 1.0 / 6.0, 5.0 / 12.0, 1.0 / 2.0, 5.0 / 6.0, 1.0 / 6.0,
                                        2.0 / 3.0, 1.0 / 3.0, 1.0}};
    }
}

int tiles_launch(cmd_mixed* h, TilesKernel kern, const cmd::MixedRun* r, int* clusters) {
    MIX_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTilesSmemMax));
    if (h->tcs > 8) MIX_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)h->tcs);
    cfg.blockDim = dim3((unsigned)h->tthreads);
    cfg.dynamicSmemBytes = (size_t)cmd::mixed_tiles_smem(h->td);
    cfg.stream = h->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)h->tcs;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (clusters) {
        MIX_TRY(cudaOccupancyMaxActiveClusters(clusters, (const void*)kern, &cfg));
        return CMD_OK;
    }
    MIX_TRY(cudaLaunchKernelEx(&cfg, kern, h->td, *r));
    return CMD_OK;
}

// The tables of mixed_tiles.cuh for a cluster of cs CTAs: CTA c owns the c-th share of each kind's sites (consecutive
// sites are consecutive cells); its sites of one atom and with equal couplings in every slot are cut into tiles.
// False when a CTA needs more than two tiles per warp, or its tables and stage vectors exceed shared memory.
bool plan_tiles(cmd_mixed* h, int cs, const KindTables& k2, const KindTables& k3, const Distinct& F2, const Distinct& O2,
                const Distinct& B2, const Distinct& M2, const Distinct& F3, const Distinct& O3, const Distinct& B3,
                const Distinct& M3, std::vector<double>& tab, std::vector<int>& ints) {
    const int N2 = h->m.N2, N3 = h->m.N3;
    h->tcs = 0;
    // fragments of a rows x cols block, zero-padded: k-step by k-step, lane (row l / 4, column 4 step + l % 4)
    auto fragments = [&](const Distinct& D, int rows, int cols, double scale) {
        const int off = (int)tab.size(), steps = (cols + 3) / 4;
        const size_t nb = D.vals.size() / D.w;
        tab.resize(tab.size() + nb * steps * 32, 0.0);
        for (size_t b = 0; b < nb; ++b)
            for (int i = 0; i < rows; ++i)
                for (int c = 0; c < cols; ++c)
                    tab[off + (b * steps + c / 4) * 32 + 4 * i + c % 4] = scale * D.vals[b * D.w + i * cols + c];
        return off;
    };
    tab.clear();
    const int o3 = fragments(O3, 8, 8, 2.0), b3 = fragments(B3, 8, 8, 1.0), m3 = fragments(M3, 8, 3, 1.0);
    const int o2 = fragments(O2, 3, 3, 2.0), b2 = fragments(B2, 3, 3, 1.0), m2 = fragments(M2, 3, 8, 1.0);
    const int f3 = (int)tab.size();
    tab.insert(tab.end(), F3.vals.begin(), F3.vals.end());
    const int f2 = (int)tab.size();
    tab.insert(tab.end(), F2.vals.begin(), F2.vals.end());
    tab.resize((tab.size() + 1) / 2 * 2 + 64, 0.0);       // a zero fragment of two k-steps at the end
    if (tab.size() * sizeof(double) > kTilesSmemMax) return false;

    // couplings of a site: {kind, atom, field, 8-component slots, 3-component slots, fragment of each slot}
    struct Slot { int kind, site, frag; };                // partner
    auto slots_of = [&](int kind, int s, std::vector<Slot>& eight, std::vector<Slot>& three) {
        const KindTables& k = kind == 3 ? k3 : k2;
        const int N = kind == 3 ? N3 : N2;
        std::vector<Slot>& like = kind == 3 ? eight : three;
        std::vector<Slot>& other = kind == 3 ? three : eight;
        like.push_back({kind, s, kind == 3 ? o3 + 64 * k.oi[s] : o2 + 32 * k.oi[s]});
        for (int n = 0; n < k.cnt[s]; ++n) {
            const int p = k.part[(size_t)n * N + s], b = k.bi[(size_t)n * N + s];
            if (p >= 0) like.push_back({kind, p, kind == 3 ? b3 + 64 * b : b2 + 32 * b});
        }
        for (int n = 0; n < k.mcnt[s]; ++n) {
            const int p = k.mpart[(size_t)n * N + s], b = k.mi[(size_t)n * N + s];
            if (p >= 0) other.push_back({5 - kind, p, kind == 3 ? m3 + 32 * b : m2 + 64 * b});
        }
    };
    struct Tile {
        int kind, field, n8, n3;
        std::vector<int> frag;
        std::vector<int> sites;
        std::vector<std::vector<Slot>> slots;             // [site][slot]
    };
    struct Cta {
        std::vector<Tile> tiles;
        std::vector<std::array<int, 4>> halo;             // kind, site, component, offset here
        std::vector<int> loc2, loc3;                      // offsets of the sites held (-1: not)
    };
    std::vector<Cta> ctas(cs);
    int tiles = 0, slots = 0, vec = 0, halo = 0;
    for (int c = 0; c < cs; ++c) {
        Cta& C = ctas[c];
        int first[2], last[2];
        for (int kind : {3, 2}) {
            const int N = kind == 3 ? N3 : N2, NA = kind == 3 ? h->m.NA3 : h->m.NA2;
            const int lo = (int)((int64_t)N * c / cs), hi = (int)((int64_t)N * (c + 1) / cs);
            first[kind - 2] = lo;
            last[kind - 2] = hi;
            std::map<std::vector<int>, int> open;         // couplings -> tile being filled
            for (int s = lo; s < hi; ++s) {
                std::vector<Slot> sl, three;
                slots_of(kind, s, sl, three);
                // by coupling, so that sites whose tables list the same bonds in another order share tiles (two-pulse
                // drive, bonds listed in varying order: 3.99 -> 2.60 us an RK4 stage, 4.48 -> 2.67 an SSPRK53 stage)
                auto by_frag = [](const Slot& x, const Slot& y) { return x.frag < y.frag; };
                for (auto* v : {&sl, &three})
                    if (!std::is_sorted(v->begin(), v->end(), by_frag)) std::stable_sort(v->begin(), v->end(), by_frag);
                const int n8 = (int)sl.size();
                sl.insert(sl.end(), three.begin(), three.end());
                std::vector<int> key{s % NA, kind == 3 ? f3 + 8 * k3.fi[s] : f2 + 3 * k2.fi[s], n8};
                for (const Slot& p : sl) key.push_back(p.frag);
                auto it = open.find(key);
                if (it == open.end() || C.tiles[it->second].sites.size() == cmd::kTileSites) {
                    Tile t{kind, key[1], n8, (int)sl.size() - n8, {key.begin() + 3, key.end()}, {}, {}};
                    open[key] = (int)C.tiles.size();
                    C.tiles.push_back(t);
                    if ((int)C.tiles.size() > 2 * kTilesWarps) return false;
                    it = open.find(key);
                }
                C.tiles[it->second].sites.push_back(s);
                slots = std::max(slots, (int)sl.size());
                C.tiles[it->second].slots.push_back(std::move(sl));
            }
        }
        // stage vector: own sites tile by tile, then the partners of other CTAs
        C.loc2.assign(N2, -1);
        C.loc3.assign(N3, -1);
        int at = 0;
        std::vector<std::pair<int, int>> remote;          // kind, site
        auto hold = [&](int kind, int s) {
            int& l = kind == 3 ? C.loc3[s] : C.loc2[s];
            if (l >= 0) return;
            l = at;
            at += kind == 3 ? cmd::kTileStride3 : cmd::kTileStride2;
            if (s < first[kind - 2] || s >= last[kind - 2]) remote.push_back({kind, s});
        };
        for (const Tile& t : C.tiles)
            for (int s : t.sites) hold(t.kind, s);
        for (const Tile& t : C.tiles)
            for (size_t n = 0; n < t.frag.size(); ++n)
                for (const auto& sl : t.slots) hold(sl[n].kind, sl[n].site);
        std::sort(remote.begin(), remote.end());          // neighbouring lanes, neighbouring words
        for (const auto& [kind, s] : remote)
            for (int d = 0; d < (kind == 3 ? 8 : 4); d += 2)          // SU(2): the fourth double is zero
                C.halo.push_back({kind, s, d, (kind == 3 ? C.loc3 : C.loc2)[s] + d});
        tiles = std::max(tiles, (int)C.tiles.size());
        vec = std::max(vec, at + cmd::kTileStride3);
        halo = std::max(halo, (int)C.halo.size());
    }
    cmd::MixedTilesDev& m = h->td;
    m.tab_doubles = (int)tab.size();
    m.tiles = tiles;
    m.slots = slots;
    m.vec = (vec + 1) / 2 * 2;
    m.halo_max = halo;
    const cmd::MixedTilesLayout L = cmd::mixed_tiles_layout(tiles, slots, halo);
    m.int_stride = L.total;
    m.N2 = N2;
    m.N3 = N3;
    m.NA2 = h->m.NA2;
    m.NA3 = h->m.NA3;
    if ((size_t)cmd::mixed_tiles_smem(m) > kTilesSmemMax) return false;
    h->tcs = cs;
    h->tpw = tiles <= kTilesWarps ? 1 : 2;
    h->tthreads = 32 * (h->tpw == 1 ? tiles : (tiles + 1) / 2);
    ints.assign((size_t)cs * L.total, 0);
    for (int c = 0; c < cs; ++c) {
        const Cta& C = ctas[c];
        int* b = &ints[(size_t)c * L.total];
        b[0] = (int)C.halo.size();
        for (int t = 0; t < tiles; ++t) {
            for (int n = 0; n < 8; ++n) {
                b[L.site + 8 * t + n] = -1;
                b[L.own + 8 * t + n] = m.vec - cmd::kTileStride3;       // the zero vector
                for (int e = 0; e < slots; ++e)
                    b[L.part + 8 * (e * tiles + t) + n] =
                        (t < (int)C.tiles.size() && e < (int)C.tiles[t].frag.size() ? C.tiles[t].frag[e] / 32 : 0) << 16 |
                        (m.vec - cmd::kTileStride3);
            }
            if (t >= (int)C.tiles.size()) continue;                     // no site: kind 0, no slots
            const Tile& T = C.tiles[t];
            b[L.tile + 4 * t] = T.kind;
            b[L.tile + 4 * t + 1] = T.n8;
            b[L.tile + 4 * t + 2] = T.n3;
            b[L.tile + 4 * t + 3] = T.field;
            for (size_t n = 0; n < T.sites.size(); ++n) {
                b[L.site + 8 * t + n] = T.sites[n];
                b[L.own + 8 * t + n] = (T.kind == 3 ? C.loc3 : C.loc2)[T.sites[n]];
                for (size_t e = 0; e < T.frag.size(); ++e) {
                    const Slot& p = T.slots[n][e];
                    b[L.part + 8 * (e * tiles + t) + n] = (p.frag / 32) << 16 | (p.kind == 3 ? C.loc3 : C.loc2)[p.site];
                }
            }
        }
        for (size_t e = 0; e < C.halo.size(); ++e) {
            const auto& x = C.halo[e];
            const int64_t N = x[0] == 3 ? N3 : N2;
            int o = (int)((int64_t)x[1] * cs / N);        // the owner: the largest CTA that starts at or before the site
            while (o + 1 < cs && N * (o + 1) / cs <= x[1]) ++o;
            while (N * o / cs > x[1]) --o;
            b[L.halo + 2 * e] = o << 16 | ((x[0] == 3 ? ctas[o].loc3 : ctas[o].loc2)[x[1]] + x[2]);
            b[L.halo + 2 * e + 1] = x[3];
        }
    }
    return true;
}

int run_tiles(cmd_mixed* h, int mode, cmd::MixedRun& r) {
    const cmd::MixedStageTimes st = tiles_stage_times(mode);
    cmd::MixedTilesDev& d = h->td;
    d.driven2 = h->m.amp2 != 0.0 && h->m.N2 > 0;
    d.driven3 = h->m.amp3 != 0.0 && h->m.N3 > 0;
    d.drive2 = h->m.drive2;
    d.drive3 = h->m.drive3;
    if ((d.driven2 || d.driven3) && r.n_steps > 0) {
        std::vector<double> grid;
        grid.reserve(r.n_steps);
        double t = r.T0;
        for (int64_t n = 0; n < r.n_steps; ++n, t += r.dt) grid.push_back(t);
        if (int rc = h->ttimes.ensure(grid.size() * sizeof(double))) return rc;
        if (int rc = h->tfact.ensure((size_t)r.n_steps * st.n * 4 * sizeof(double))) return rc;
        MIX_TRY(cudaMemcpyAsync(h->ttimes.p, grid.data(), grid.size() * sizeof(double), cudaMemcpyHostToDevice, h->stream));
        const int64_t total = r.n_steps * st.n * 4;
        const int blocks = (int)std::min<int64_t>((total + 127) / 128, 148 * 16);
        cmd::mixed_factor_kernel<<<blocks, 128, 0, h->stream>>>(h->m, h->ttimes.as<double>(), r.n_steps, r.dt, st,
                                                               h->tfact.as<double>());
        MIX_TRY(cudaGetLastError());
        d.factors = h->tfact.as<double2>();
    }
    return tiles_launch(h, tiles_kernel(mode, h->tpw), &r, nullptr);
}

// The smallest cluster (1, 2, 4, 8, 16 CTAs) that holds the lattice with one tile per warp, else with two.  A 16-CTA
// cluster is a non-portable size: only where it can be resident.
bool choose_tiles(cmd_mixed* h, const KindTables& k2, const KindTables& k3, const Distinct& F2, const Distinct& O2,
                  const Distinct& B2, const Distinct& M2, const Distinct& F3, const Distinct& O3, const Distinct& B3,
                  const Distinct& M3, std::vector<double>& tab, std::vector<int>& ints) {
    const int64_t sites = (int64_t)h->m.N2 + h->m.N3;
    auto plan = [&](int cs) { return plan_tiles(h, cs, k2, k3, F2, O2, B2, M2, F3, O3, B3, M3, tab, ints); };
    auto resident = [&]() {
        int n = 0;
        return h->tcs <= 8 || (tiles_launch(h, tiles_kernel(cmd::kModeRK78, h->tpw), nullptr, &n) == CMD_OK && n >= 1);
    };
    for (int want : {1, 2})
        for (int cs : {1, 2, 4, 8, 16}) {
            if (sites > (int64_t)cs * want * kTilesWarps * cmd::kTileSites) continue;
            if (plan(cs) && h->tpw <= want && resident()) return true;
        }
    h->tcs = 0;
    return false;
}

// Whether a 16-CTA cluster (a non-portable size) of this shape can be resident.
bool cluster16_fits(cmd_mixed* h, int threads) {
    if (set_attributes<16>() != CMD_OK) return false;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = config<16>(h, threads, attr);
    int n = 0;
    return cudaOccupancyMaxActiveClusters(&n, cmd::mixed_integrate_kernel<16>, &cfg) == cudaSuccess && n >= 1;
}

// One persistent launch over a cluster sized to the lattice: one site per thread up
// to 16 CTAs, the threads loop beyond that (at most kMixedThreads per CTA).
int run(cmd_mixed* h, int method, double T0, double dt, int64_t n_steps, int64_t save_every, int64_t max_rows) {
    const int mode = method_mode(method);
    if (mode < 0) return fail(CMD_ERR_INVALID_ARG, "the mixed path takes a fixed-step method (any CMD_* but CMD_RK45)");
    const bool tiles = h->tcs > 0 && mode != cmd::kModeBulirschStoer;         // whose stage vectors rotate at run time
    if (max_rows > 0)
        if (int rc = h->rows.ensure((size_t)max_rows * h->V * sizeof(double))) return rc;
    cmd::MixedRun r{};
    r.y0 = h->state.as<double>();
    r.y_out = h->state.as<double>();
    r.rows = max_rows > 0 ? h->rows.as<double>() : nullptr;
    r.max_rows = max_rows;
    r.T0 = T0;
    r.dt = dt;
    r.n_steps = n_steps;
    r.save_every = save_every;
    r.mode = mode;
    if (tiles) {
        // the envelope table grows with the steps: where it finds no room, the kernel that needs none
        const int rc = run_tiles(h, mode, r);
        if (rc != CMD_ERR_OOM) return rc;
        cudaGetLastError();
        cmd::clear_error();
    }
    if (int rc = h->work.ensure((size_t)11 * h->V * sizeof(double))) return rc;
    r.work = h->work.as<double>();
    // Up to 128 sites per CTA before the cluster grows (more SMs per trajectory beat
    // more warps per SM here: the stages are latency-bound), up to 16 CTAs.
    const int64_t sites = (int64_t)h->m.N2 + h->m.N3;
    const int64_t per = (sites + 127) / 128;
    int cs = per <= 1 ? 1 : per <= 2 ? 2 : per <= 4 ? 4 : per <= 8 ? 8 : 16;
    auto threads_for = [&](int c) {
        return (int)std::min<int64_t>(cmd::kMixedThreads, std::max<int64_t>(32, ((sites + c - 1) / c + 31) / 32 * 32));
    };
    if (cs == 16 && !cluster16_fits(h, threads_for(16))) cs = 8;
    const int threads = threads_for(cs);
    int rc = cs == 1 ? launch_cs<1>(h, r, threads)
           : cs == 2 ? launch_cs<2>(h, r, threads)
           : cs == 4 ? launch_cs<4>(h, r, threads)
           : cs == 8 ? launch_cs<8>(h, r, threads)
                     : launch_cs<16>(h, r, threads);
    if (rc) return rc;
    MIX_TRY(cudaGetLastError());
    return CMD_OK;
}

int check(cmd_mixed* h, bool need_state) {
    if (!h) return fail(CMD_ERR_INVALID_ARG, "NULL handle");
    if (need_state && !h->has_state) return fail(CMD_ERR_STATE, "spins not set (call cmd_mixed_set_spins first)");
    return CMD_OK;
}

}  // namespace

extern "C" {

int cmd_mixed_create(const cmd_mixed_desc* d, cmd_mixed** out) {
    cmd::clear_error();
    if (!d || !out) return fail(CMD_ERR_INVALID_ARG, "NULL argument");
    *out = nullptr;
    if (d->spin_dim_su2 != 3 || d->spin_dim_su3 != 8)
        return fail(CMD_ERR_INVALID_ARG, "spin dimensions must be 3 (SU(2)) and 8 (SU(3))");
    if (d->n_su2 < 0 || d->n_su3 < 0 || d->n_su2 + d->n_su3 <= 0 || d->n_su2 + d->n_su3 >= (1LL << 30))
        return fail(CMD_ERR_INVALID_ARG, "bad site counts");
    if ((d->n_su2 > 0 && d->n_atoms_su2 <= 0) || (d->n_su3 > 0 && d->n_atoms_su3 <= 0))
        return fail(CMD_ERR_INVALID_ARG, "n_atoms must be positive for a non-empty sublattice");
    if (d->max_bilinear_su2 < 0 || d->max_bilinear_su3 < 0 || d->max_mixed_su2 < 0 || d->max_mixed_su3 < 0)
        return fail(CMD_ERR_INVALID_ARG, "negative ELL width");
    const int64_t N2 = d->n_su2, N3 = d->n_su3;
    const int z2 = d->max_bilinear_su2, z3 = d->max_bilinear_su3, zm2 = d->max_mixed_su2, zm3 = d->max_mixed_su3;
    auto need = [](const void* p, int64_t n) { return n == 0 || p != nullptr; };
    if (!need(d->field_su2, N2) || !need(d->onsite_su2, N2) || !need(d->counts_su2, N2) ||
        !need(d->field_su3, N3) || !need(d->onsite_su3, N3) || !need(d->counts_su3, N3) ||
        !need(d->bilinear_su2, N2 * z2) || !need(d->partners_su2, N2 * z2) || !need(d->bilinear_su3, N3 * z3) ||
        !need(d->partners_su3, N3 * z3) || !need(d->mixed_su2, N2 * zm2) || !need(d->mixed_partners_su3, N2 * zm2) ||
        !need(d->mixed_counts_su2, N2 * (zm2 > 0)) || !need(d->mixed_su3, N3 * zm3) ||
        !need(d->mixed_partners_su2, N3 * zm3) || !need(d->mixed_counts_su3, N3 * (zm3 > 0)))
        return fail(CMD_ERR_INVALID_ARG, "missing table");
    cmd_mixed* h = new cmd_mixed;
    auto bail = [&](int rc) {
        if (h->stream) cudaStreamDestroy(h->stream);
        delete h;
        return rc;
    };
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess)
        return bail(fail(CMD_ERR_CUDA, "no CUDA device (cudaStreamCreate failed)"));
    Distinct F2(3), O2(9), B2(9), M2(24), F3(8), O3(64), B3(64), M3(24);
    KindTables k2, k3;
    build_kind(N2, std::max(1, d->n_atoms_su2), z2, zm2, 3, d->field_su2, d->onsite_su2, d->bilinear_su2, d->partners_su2, d->counts_su2, N2,
               d->mixed_su2, d->mixed_partners_su3, d->mixed_counts_su2, N3, F2, O2, B2, M2, k2);
    build_kind(N3, std::max(1, d->n_atoms_su3), z3, zm3, 8, d->field_su3, d->onsite_su3, d->bilinear_su3, d->partners_su3, d->counts_su3, N3,
               d->mixed_su3, d->mixed_partners_su2, d->mixed_counts_su3, N2, F3, O3, B3, M3, k3);
    std::vector<double> tab;
    cmd::MixedDev& m = h->m;
    // each distinct block at the kernel's odd stride (mixed.cuh kStride*)
    auto append = [&](const Distinct& D, int stride, int& off) {
        off = (int)tab.size();
        const size_t nb = D.vals.size() / D.w;
        tab.resize(tab.size() + nb * stride, 0.0);
        for (size_t b = 0; b < nb; ++b)
            std::copy(D.vals.begin() + b * D.w, D.vals.begin() + (b + 1) * D.w, tab.begin() + off + b * stride);
    };
    append(F2, cmd::kStrideF2, m.off_f2); append(O2, cmd::kStrideO2, m.off_o2);
    append(B2, cmd::kStrideB2, m.off_b2); append(M2, cmd::kStrideM, m.off_m2);
    append(F3, cmd::kStrideF3, m.off_f3); append(O3, cmd::kStrideO3, m.off_o3);
    append(B3, cmd::kStrideB3, m.off_b3); append(M3, cmd::kStrideM, m.off_m3);
    // work slots: warp-sized runs of SU(2) and SU(3) sites in turn, so every CTA gets both kinds
    std::vector<int> order;
    order.reserve(N2 + N3);
    for (int64_t a = 0, b = 0; a < N2 || b < N3;) {
        for (int k = 0; k < 32 && a < N2; ++k) order.push_back((int)a++);
        for (int k = 0; k < 32 && b < N3; ++k) order.push_back((int)(N2 + b++));
    }
    const std::vector<int>* ints[17] = {&k2.fi, &k2.oi, &k2.bi, &k2.part, &k2.cnt, &k2.mi, &k2.mpart, &k2.mcnt,
                                        &k3.fi, &k3.oi, &k3.bi, &k3.part, &k3.cnt, &k3.mi, &k3.mpart, &k3.mcnt,
                                        &order};
    size_t total = pad(tab.size() * sizeof(double));
    for (const auto* v : ints) total += pad(v->size() * sizeof(int));
    if (int rc = h->tables.ensure(total)) return bail(rc);
    char* cur = h->tables.as<char>();
    int rc = CMD_OK;
    auto put = [&](const void* src, size_t bytes) {
        char* at = cur;
        if (rc == CMD_OK && bytes) {
            if (cudaMemcpyAsync(cur, src, bytes, cudaMemcpyHostToDevice, h->stream) != cudaSuccess)
                rc = fail(CMD_ERR_CUDA, "upload of the mixed lattice tables failed");
        }
        cur += pad(bytes);
        return at;
    };
    m.N2 = (int)N2; m.N3 = (int)N3;
    m.NA2 = std::max(1, d->n_atoms_su2); m.NA3 = std::max(1, d->n_atoms_su3);
    m.z2 = z2; m.z3 = z3; m.zm2 = zm2; m.zm3 = zm3;
    m.tab = (const double*)put(tab.data(), tab.size() * sizeof(double));
    m.tab_doubles = (int)tab.size();
    m.tab_in_smem = tab.size() * sizeof(double) <= kMixedSmemMax;
    const int* dev[17];
    for (int i = 0; i < 17; ++i) dev[i] = (const int*)put(ints[i]->data(), ints[i]->size() * sizeof(int));
    m.order = dev[16];
    m.f2i = dev[0]; m.o2i = dev[1]; m.b2i = dev[2]; m.part2 = dev[3]; m.cnt2 = dev[4]; m.m2i = dev[5];
    m.mpart2 = dev[6]; m.mcnt2 = dev[7];
    m.f3i = dev[8]; m.o3i = dev[9]; m.b3i = dev[10]; m.part3 = dev[11]; m.cnt3 = dev[12]; m.m3i = dev[13];
    m.mpart3 = dev[14]; m.mcnt3 = dev[15];
    if (rc) return bail(rc);
    // the host vectors above must outlive the copies
    if (cudaStreamSynchronize(h->stream) != cudaSuccess) return bail(fail(CMD_ERR_CUDA, "upload failed"));
    // drives start at zero, width 1 (the reference's defaults)
    const size_t bd2 = 2 * (size_t)m.NA2 * 3 * 8, bd3 = 2 * (size_t)m.NA3 * 8 * 8;
    if ((rc = h->drive2.ensure(bd2)) || (rc = h->drive3.ensure(bd3))) return bail(rc);
    if (cudaMemsetAsync(h->drive2.p, 0, bd2, h->stream) != cudaSuccess ||
        cudaMemsetAsync(h->drive3.p, 0, bd3, h->stream) != cudaSuccess)
        return bail(fail(CMD_ERR_CUDA, "cudaMemsetAsync failed"));
    m.drive2 = h->drive2.as<double>();
    m.drive3 = h->drive3.as<double>();
    m.width2 = m.width3 = 1.0;
    h->V = 3 * N2 + 8 * N3;
    {
        std::vector<double> tab_t;
        std::vector<int> ints_t;
        const bool fits = choose_tiles(h, k2, k3, F2, O2, B2, M2, F3, O3, B3, M3, tab_t, ints_t);
        cmd::clear_error();
        if (fits) {
            if ((rc = h->ttab.ensure(tab_t.size() * sizeof(double))) || (rc = h->tints.ensure(ints_t.size() * sizeof(int))))
                return bail(rc);
            if (cudaMemcpyAsync(h->ttab.p, tab_t.data(), tab_t.size() * sizeof(double), cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
                cudaMemcpyAsync(h->tints.p, ints_t.data(), ints_t.size() * sizeof(int), cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
                cudaStreamSynchronize(h->stream) != cudaSuccess)
                return bail(fail(CMD_ERR_CUDA, "upload of the mixed lattice tables failed"));
            h->td.tab = h->ttab.as<double>();
            h->td.ints = h->tints.as<int>();
        }
    }
    if ((rc = h->state.ensure((size_t)h->V * sizeof(double)))) return bail(rc);
    if (cudaStreamSynchronize(h->stream) != cudaSuccess) return bail(fail(CMD_ERR_CUDA, "upload failed"));
    *out = h;
    return CMD_OK;
}

int cmd_mixed_destroy(cmd_mixed* h) {
    cmd::clear_error();
    if (!h) return CMD_OK;
    cudaStreamSynchronize(h->stream);
    cudaStreamDestroy(h->stream);
    delete h;
    return CMD_OK;
}

int cmd_mixed_set_pulse(cmd_mixed* h, int32_t sub, const double* fd, double amp, double width, double freq,
                        double t1, double t2) {
    cmd::clear_error();
    if (int rc = check(h, false)) return rc;
    if (sub != 2 && sub != 3) return fail(CMD_ERR_INVALID_ARG, "sublattice must be 2 (SU(2)) or 3 (SU(3))");
    if (!fd) return fail(CMD_ERR_INVALID_ARG, "NULL field_drive");
    if (!std::isfinite(amp) || !std::isfinite(width) || !std::isfinite(freq) || !std::isfinite(t1) || !std::isfinite(t2))
        return fail(CMD_ERR_INVALID_ARG, "non-finite pulse parameter");
    cmd::MixedDev& m = h->m;
    const size_t n = sub == 2 ? 2 * (size_t)m.NA2 * 3 : 2 * (size_t)m.NA3 * 8;
    MIX_TRY(cudaMemcpyAsync(sub == 2 ? h->drive2.p : h->drive3.p, fd, n * sizeof(double), cudaMemcpyHostToDevice,
                            h->stream));
    MIX_TRY(cudaStreamSynchronize(h->stream));
    if (sub == 2) { m.amp2 = amp; m.width2 = width; m.freq2 = freq; m.t1_2 = t1; m.t2_2 = t2; }
    else { m.amp3 = amp; m.width3 = width; m.freq3 = freq; m.t1_3 = t1; m.t2_3 = t2; }
    return CMD_OK;
}

int cmd_mixed_set_spins(cmd_mixed* h, const double* s, int64_t n) {
    cmd::clear_error();
    if (int rc = check(h, false)) return rc;
    if (!s || n != h->V) return fail(CMD_ERR_INVALID_ARG, "spins must hold n_su2*3 + n_su3*8 values");
    for (int64_t i = 0; i < n; ++i)
        if (!std::isfinite(s[i])) return fail(CMD_ERR_NONFINITE, "non-finite spin component");
    MIX_TRY(cudaMemcpyAsync(h->state.p, s, n * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    MIX_TRY(cudaStreamSynchronize(h->stream));
    h->has_state = true;
    return CMD_OK;
}

int cmd_mixed_get_spins(cmd_mixed* h, double* s, int64_t n) {
    cmd::clear_error();
    if (int rc = check(h, true)) return rc;
    if (!s || n != h->V) return fail(CMD_ERR_INVALID_ARG, "spins must hold n_su2*3 + n_su3*8 values");
    MIX_TRY(cudaMemcpyAsync(s, h->state.p, n * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    MIX_TRY(cudaStreamSynchronize(h->stream));
    return CMD_OK;
}

int cmd_mixed_step(cmd_mixed* h, double t, double dt, int method) {
    cmd::clear_error();
    if (int rc = check(h, true)) return rc;
    if (!std::isfinite(t) || !std::isfinite(dt)) return fail(CMD_ERR_INVALID_ARG, "non-finite t or dt");
    if (int rc = run(h, method, t, dt, 1, 1, 0)) return rc;
    MIX_TRY(cudaStreamSynchronize(h->stream));
    return CMD_OK;
}

int cmd_mixed_integrate(cmd_mixed* h, double T0, double T1, double dt, int64_t save_interval, int method,
                        double* times, double* states, int64_t max_rows, int64_t* rows_out) {
    cmd::clear_error();
    if (int rc = check(h, true)) return rc;
    if (save_interval <= 0 || !(dt > 0.0) || !std::isfinite(T0) || !std::isfinite(T1))
        return fail(CMD_ERR_INVALID_ARG, "bad integration window");
    if (method_mode(method) < 0)
        return fail(CMD_ERR_INVALID_ARG, "the mixed path takes a fixed-step method (any CMD_* but CMD_RK45)");
    std::vector<double> grid;
    const int64_t n = loop_steps(T0, T1, dt, &grid);
    const int64_t rows = (n + save_interval - 1) / save_interval + 1;
    if (rows_out) *rows_out = rows;
    if (max_rows < rows) return fail(CMD_ERR_INVALID_ARG, "max_rows too small");
    if (int rc = run(h, method, T0, dt, n, save_interval, states ? rows : 0)) return rc;
    if (states)
        MIX_TRY(cudaMemcpyAsync(states, h->rows.p, (size_t)rows * h->V * sizeof(double), cudaMemcpyDeviceToHost,
                                h->stream));
    MIX_TRY(cudaStreamSynchronize(h->stream));
    if (times) {
        int64_t r = 0;
        for (int64_t k = 0; k < n; k += save_interval) times[r++] = grid[k];
        times[r] = grid[n];
    }
    return CMD_OK;
}

int cmd_mixed_magnetization(cmd_mixed* h, double* m2, double* ms2, double* m3, double* ms3) {
    cmd::clear_error();
    if (int rc = check(h, true)) return rc;
    if (!m2 || !ms2 || !m3 || !ms3) return fail(CMD_ERR_INVALID_ARG, "NULL output");
    if (int rc = h->mag.ensure(22 * sizeof(double))) return rc;
    cmd::mixed_magnetization_kernel<<<11, 256, 0, h->stream>>>(h->state.as<double>(), h->m.N2, h->m.N3, h->m.NA2,
                                                              h->m.NA3, h->mag.as<double>());
    MIX_TRY(cudaGetLastError());
    double out[22];
    MIX_TRY(cudaMemcpyAsync(out, h->mag.p, sizeof(out), cudaMemcpyDeviceToHost, h->stream));
    MIX_TRY(cudaStreamSynchronize(h->stream));
    for (int i = 0; i < 3; ++i) { m2[i] = out[i]; ms2[i] = out[3 + i]; }
    for (int i = 0; i < 8; ++i) { m3[i] = out[6 + i]; ms3[i] = out[14 + i]; }
    return CMD_OK;
}

int cmd_mixed_normalize(cmd_mixed* h, double l2, double l3) {
    cmd::clear_error();
    if (int rc = check(h, true)) return rc;
    const int sites = h->m.N2 + h->m.N3;
    cmd::mixed_normalize_kernel<<<(sites + 255) / 256, 256, 0, h->stream>>>(h->state.as<double>(), h->m.N2, h->m.N3,
                                                                           l2, l3);
    MIX_TRY(cudaGetLastError());
    MIX_TRY(cudaStreamSynchronize(h->stream));
    return CMD_OK;
}

int cmd_mixed_dims(cmd_mixed* h, int64_t* dims) {
    cmd::clear_error();
    if (int rc = check(h, false)) return rc;
    if (!dims) return fail(CMD_ERR_INVALID_ARG, "NULL output");
    dims[0] = h->m.N2; dims[1] = 3; dims[2] = h->m.NA2;
    dims[3] = h->m.N3; dims[4] = 8; dims[5] = h->m.NA3;
    return CMD_OK;
}

}  // extern "C"
