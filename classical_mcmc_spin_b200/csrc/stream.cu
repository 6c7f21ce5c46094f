// stream.cu -- streamed RK4 and the streamed discrete adjoint (rk_stream.cuh):
// lattices no resident or cluster variant holds, one launch per RK stage over
// (cell tile, trajectory).
#include "cmd_core.h"
#include "rk_stream.cuh"

namespace cmd {
namespace {

// Steps of the streamed RK4 loop: enqueue(g, k) launches the four stages of step
// base + k of trajectory group g, base read by the kernels from h->snbase.  A
// chunk of steps runs group by group, so a group's vectors stay in L2 from stage
// to stage.  With graphs on and at least two chunks of work, one chunk of
// kChunk / groups steps (4 kChunk stage launches and a base advance) is captured
// once per distinct set of launch parameters (`key`), kept in the handle and
// replayed; the remaining steps are launched directly.  The kernels see the same
// step numbers either way.
constexpr int64_t kChunk = 128;

template <class F>
int run_steps(cmd_handle* h, cudaStream_t st, int64_t S, int64_t groups, const std::vector<unsigned char>& key,
              F&& enqueue, int32_t* nl) {
    CUDA_TRY(cudaMemsetAsync(h->snbase.p, 0, sizeof(long long), st));
    int64_t done = 0;
    const int64_t chunk = std::max<int64_t>(kChunk / groups, 16);
    if (h->graphs && S >= 2 * kChunk) {
        if (!h->stream_graph || h->stream_graph_key != key) {
            release_stream_graph(h);
            cudaGraph_t g = nullptr;
            CUDA_TRY(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
            for (int64_t i = 0; i < groups; ++i)
                for (int64_t k = 0; k < chunk; ++k) enqueue(i, k);
            stream_advance_kernel<<<1, 32, 0, st>>>(h->snbase.as<long long>(), chunk);
            const cudaError_t e = cudaStreamEndCapture(st, &g);
            if (e != cudaSuccess || !g) return fail(CMD_ERR_CUDA, std::string("stream capture: ") + cudaGetErrorString(e));
            const cudaError_t e2 = cudaGraphInstantiate(&h->stream_graph, g, 0);
            cudaGraphDestroy(g);
            if (e2 != cudaSuccess) {
                h->stream_graph = nullptr;
                return fail(CMD_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e2));
            }
            h->stream_graph_key = key;
        }
        for (; done + chunk <= S; done += chunk) {
            CUDA_TRY(cudaGraphLaunch(h->stream_graph, st));
            *nl += (int32_t)(4 * groups * chunk) + 1;
        }
    }
    const int64_t rest = S - done;
    for (int64_t k0 = 0; k0 < rest; k0 += chunk)
        for (int64_t i = 0; i < groups; ++i) {
            const int64_t k1 = std::min(k0 + chunk, rest);
            for (int64_t k = k0; k < k1; ++k) enqueue(i, k);
            *nl += (int32_t)(4 * (k1 - k0));
            CUDA_TRY(cudaGetLastError());
        }
    return CMD_OK;
}

// Partner offsets (soff) of the streamed kernels, [NAT][Z-LZ][G], from Layout::nbr or, when `pair`, nbr_pair; built
// on first use.
template <int NAT>
int stream_table(cmd_handle* h, bool pair) {
    DevBuf& d = h->nbrt[pair];
    if (d.p) return CMD_OK;
    const Layout& L = h->lay;
    const std::vector<int>& src = pair ? L.nbr_pair : L.nbr;
    const int NL = L.Z - L.LZ;
    std::vector<int> t(std::max<size_t>(src.size(), 1));
    for (int64_t g = 0; g < L.G; ++g)
        for (int a = 0; a < L.NA; ++a)
            for (int m = 0; m < NL; ++m)
            {
                const int64_t off = src[((size_t)g * L.NA + a) * NL + m], at = off / (3 * L.G);
                t[((size_t)a * NL + m) * L.G + g] = soff<NAT>((int)(off - at * 3 * L.G), (int)at);
            }
    return upload_once(d, t.data(), t.size() * sizeof(int), "streamed partner table");
}

// One launch of RK stage s.
template <int NAT, int Z, int LZ, bool PAIR>
void stage(int s, dim3 grid, cudaStream_t st, const Couplings<NAT, Z>& cp, const StreamArgs& a, int64_t n, SVec Yin, SVec y,
           SVec acc, SVec Ynext, int obs) {
    auto kern = s == 0   ? (obs ? stream_stage_kernel<NAT, Z, LZ, PAIR, 0, true> : stream_stage_kernel<NAT, Z, LZ, PAIR, 0, false>)
                : s == 1 ? (obs ? stream_stage_kernel<NAT, Z, LZ, PAIR, 1, true> : stream_stage_kernel<NAT, Z, LZ, PAIR, 1, false>)
                : s == 2 ? stream_stage_kernel<NAT, Z, LZ, PAIR, 2, false>
                         : stream_stage_kernel<NAT, Z, LZ, PAIR, 3, false>;
    kern<<<grid, kStreamTile, 0, st>>>(cp, a, n, Yin, y, acc, Ynext);
}

// Trajectories per group of a streamed run with `vectors` vectors of V doubles each: as many as keep the group's
// vectors within kL2Share of L2 (measured on the 65536-spin pyrochlore, 32 trajectories, before the blocked layout: see rk_stream.cuh), in
// groups of equal size.
int64_t stream_group(const cmd_handle* h, int64_t B, int64_t V, int vectors) {
    int l2 = 0;
    if (cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, h->device) != cudaSuccess || l2 <= 0) return B;
    constexpr double kL2Share = 0.6;
    const int64_t fit = std::max<int64_t>(1, (int64_t)(kL2Share * l2 / ((double)vectors * V * sizeof(double))));
    const int64_t groups = (B + fit - 1) / fit;
    return (B + groups - 1) / groups;
}

template <class T>
void key_add(std::vector<unsigned char>& k, const T& v) {
    const unsigned char* p = reinterpret_cast<const unsigned char*>(&v);
    k.insert(k.end(), p, p + sizeof(T));
}

// ---------------------------------------------------------------------------
// Streamed RK4 (rk_stream.cuh): lattices no resident variant holds.  One launch
// per stage over (cell tile, trajectory); same RunSpec contract and outputs as
// run_resident.

template <int NAT, int Z, int LZ, bool PAIR>
int stream_forward(cmd_handle* h, const RunSpec& r, cudaStream_t st, int32_t* launches) {
    constexpr int NR = 3 * NAT + 1;
    int32_t nl = 0;
    const int G = (int)h->lay.G;
    const int tiles = (G + cmd::stream_cells<NAT>() - 1) / cmd::stream_cells<NAT>();
    const int64_t V = (int64_t)NAT * 3 * tiles * cmd::stream_cells<NAT>();      // padded to whole tiles
    const int64_t B = r.B;
    if (B > 65535) return fail(CMD_ERR_UNSUPPORTED, "streamed batches are limited to 65535 trajectories");
    if (r.traj && B != 1) return fail(CMD_ERR_UNSUPPORTED, "streamed state saving is for single trajectories");
    const int64_t rows = rows_for(r.n_steps, r.save);
    if (int rc = h->sbuf.ensure((size_t)4 * B * V * sizeof(double))) return rc;
    if (int rc = h->spart.ensure((size_t)B * tiles * cmd::kPart * sizeof(double))) return rc;
    double* base = h->sbuf.as<double>();
    const cmd::SVec y{base, V}, acc{base + B * V, V}, Ya{base + 2 * B * V, V}, Yb{base + 3 * B * V, V};
    cmd::StreamArgs a{};
    a.G = G;
    a.tiles = tiles;
    a.B = (int)B;
    if (int rc = stream_table<NAT>(h, PAIR)) return rc;
    a.nbr = h->nbrt[PAIR].as<int>();
    a.dt = r.dt;
    a.n_steps = r.n_steps;
    a.part = h->spart.as<double>();
    a.n_sites = r.n_sites;
    a.save_every = r.save;
    a.rows = rows;
    a.V = V;
    if (r.obs) {
        if (NR <= 10) {
            a.raw = r.obs;
            a.raw_stride = 10;
        } else {
            if (int rc = h->raw.ensure((size_t)B * rows * NR * sizeof(double))) return rc;
            a.raw = h->raw.as<double>();
            a.raw_stride = NR;
        }
    }
    if (r.pulses && r.n_steps > 0) {
        std::vector<double> grid;
        grid.reserve(r.n_steps);
        double t = r.T0;
        for (int64_t k = 0; k < r.n_steps; ++k) {     // t_k of the reference loop (t += dt)
            grid.push_back(t);
            t += r.dt;
        }
        if (int rc = h->times.ensure(grid.size() * sizeof(double))) return rc;
        if (int rc = h->drive.ensure((size_t)B * r.n_steps * 6 * sizeof(double))) return rc;
        CUDA_TRY(cudaMemcpyAsync(h->times.p, grid.data(), grid.size() * sizeof(double), cudaMemcpyHostToDevice, st));
        const int64_t total = B * r.n_steps * 6;
        const int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 32);
        cmd::drive_table_kernel<<<blocks, 256, 0, st>>>(r.pulses, h->times.as<double>(), r.n_steps, r.dt, r.width,
                                                       r.freq, B, h->drive.as<double>());
        CUDA_TRY(cudaGetLastError());
        ++nl;
        a.times = h->times.as<double>();
        a.drive = h->drive.as<double>();
    }
    static const std::vector<double> zeros(3 * 64, 0.0);
    cmd::Couplings<NAT, Z> cp;
    fill_couplings<NAT, Z>(h, r.d1 ? r.d1 : zeros.data(), r.d2 ? r.d2 : zeros.data(), cp);
    const dim3 grid(tiles, (unsigned)B), gridc((G + 255) / 256, (unsigned)B);
    const int64_t N3 = (int64_t)G * NAT * 3;
    auto save_traj = [&](int64_t row) {
        const cmd::SVec src = y;
        cmd::stream_store_kernel<NAT><<<gridc, 256, 0, st>>>(src, G, r.traj + row * N3);
        ++nl;
    };
    cmd::stream_load_kernel<NAT><<<gridc, 256, 0, st>>>(r.y0, r.y0_stride, G, y);
    CUDA_TRY(cudaGetLastError());
    ++nl;
    const int with_obs = r.obs ? 1 : 0;
    if (r.traj) {                                    // states saved between steps: direct launches
        for (int64_t n = 0; n < r.n_steps; ++n) {
            if (n % r.save == 0) save_traj(n / r.save);
            stage<NAT, Z, LZ, PAIR>(0, grid, st, cp, a, n, y, y, acc, Ya, with_obs);
            stage<NAT, Z, LZ, PAIR>(1, grid, st, cp, a, n, Ya, y, acc, Yb, with_obs);
            stage<NAT, Z, LZ, PAIR>(2, grid, st, cp, a, n, Yb, y, acc, Ya, with_obs);
            stage<NAT, Z, LZ, PAIR>(3, grid, st, cp, a, n, Ya, y, acc, y, with_obs);
            nl += 4;
            if ((n & 1023) == 0) CUDA_TRY(cudaGetLastError());
        }
        CUDA_TRY(cudaGetLastError());
    } else {
        if (int rc = h->snbase.ensure(sizeof(long long))) return rc;
        a.nbase = h->snbase.as<long long>();
        std::vector<unsigned char> key;
        key_add(key, 1);                             // forward stages of this NAT/Z/LZ
        key_add(key, NAT * 100 + Z * 10 + LZ);
        key_add(key, cp);
        key_add(key, a);
        key_add(key, y);
        key_add(key, acc);
        key_add(key, Ya);
        key_add(key, Yb);
        key_add(key, with_obs);
        key_add(key, grid);
        const int64_t per = stream_group(h, B, V, 4), groups = (B + per - 1) / per;
        key_add(key, per);
        auto enqueue = [&](int64_t i, int64_t k) {
            cmd::StreamArgs ag = a;
            ag.b0 = (int)(i * per);
            const dim3 gg(tiles, (unsigned)std::min(per, B - i * per));
            stage<NAT, Z, LZ, PAIR>(0, gg, st, cp, ag, k, y, y, acc, Ya, with_obs);
            stage<NAT, Z, LZ, PAIR>(1, gg, st, cp, ag, k, Ya, y, acc, Yb, with_obs);
            stage<NAT, Z, LZ, PAIR>(2, gg, st, cp, ag, k, Yb, y, acc, Ya, with_obs);
            stage<NAT, Z, LZ, PAIR>(3, gg, st, cp, ag, k, Ya, y, acc, y, with_obs);
        };
        if (int rc = run_steps(h, st, r.n_steps, groups, key, enqueue, &nl)) return rc;
        a.nbase = nullptr;                           // the final observation below uses absolute steps
    }
    if (r.traj) save_traj(rows - 1);
    if (r.obs) {
        cmd::stream_obs_kernel<NAT, Z, LZ, PAIR><<<grid, cmd::kStreamTile, 0, st>>>(cp, a, y);
        cmd::stream_reduce_kernel<NAT><<<(unsigned)B, cmd::kStreamTile, 0, st>>>(a, r.n_steps);
        CUDA_TRY(cudaGetLastError());
        nl += 2;
    }
    if (r.y_out) {
        cmd::stream_store_kernel<NAT><<<gridc, 256, 0, st>>>(y, G, r.y_out);
        CUDA_TRY(cudaGetLastError());
        ++nl;
    }
    if (r.obs) {
        const double* fr = r.frames ? r.frames : h->dframes.as<double>();
        const double* af = r.afm ? r.afm : h->dafm.as<double>();
        launch_finish<NAT>(a.raw, a.raw_stride, B * rows, fr, af, r.n_sites, r.obs, st);
        CUDA_TRY(cudaGetLastError());
        ++nl;
    }
    if (launches) *launches = nl;
    return CMD_OK;
}

template <int NAT, int Z, int LZ, int NQ, bool PAIR>
int stream_adjoint(cmd_handle* h, const StreamAdjJob& j, const std::vector<double>& DJ, const std::vector<double>& DB,
                   const std::vector<double>& DA, bool has_DA) {
    cudaStream_t st = h->stream;
    const int G = (int)h->lay.G;
    const int tiles = (G + cmd::stream_cells<NAT>() - 1) / cmd::stream_cells<NAT>();
    const int64_t V = (int64_t)NAT * 3 * tiles * cmd::stream_cells<NAT>(), B = j.B, S = j.S, C = j.C, K = j.K;
    if (int rc = h->sbuf.ensure((size_t)5 * B * V * sizeof(double))) return rc;
    if (int rc = h->spart.ensure(((size_t)B * tiles * cmd::kPart + B) * sizeof(double))) return rc;
    if (int rc = h->sgpart.ensure((size_t)B * tiles * cmd::kPart * sizeof(double))) return rc;
    double* base = h->sbuf.as<double>();
    double* d_loss = h->spart.as<double>() + (size_t)B * tiles * cmd::kPart;
    const bool driven = h->amp != 0.0;
    if (driven) {
        std::vector<cmd::Pulse> pl((size_t)B, cmd::Pulse{h->t1, h->t2, h->amp, h->amp});
        if (int rc = h->pulses.ensure((size_t)B * sizeof(cmd::Pulse))) return rc;
        if (int rc = h->drive.ensure((size_t)B * S * 6 * sizeof(double))) return rc;
        CUDA_TRY(cudaMemcpyAsync(h->pulses.p, pl.data(), pl.size() * sizeof(cmd::Pulse), cudaMemcpyHostToDevice, st));
        const int64_t total = B * S * 6;
        const int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 32);
        cmd::drive_table_kernel<<<blocks, 256, 0, st>>>(h->pulses.as<cmd::Pulse>(), j.times, S, j.dt, h->width,
                                                       h->freq, B, h->drive.as<double>());
        CUDA_TRY(cudaGetLastError());
    }
    cmd::Couplings<NAT, Z> cp;
    fill_couplings<NAT, Z>(h, h->fd.data(), h->fd.data() + 3 * h->NA, cp);
    cmd::StreamArgs a{};
    a.G = G;
    a.tiles = tiles;
    a.B = (int)B;
    if (int rc = stream_table<NAT>(h, PAIR)) return rc;
    a.nbr = h->nbrt[PAIR].as<int>();
    a.dt = j.dt;
    a.n_steps = S;
    a.times = j.times;
    a.drive = driven ? h->drive.as<double>() : nullptr;
    a.part = h->spart.as<double>();
    a.save_every = 1;
    a.rows = S + 1;
    a.target = j.target;
    a.mloc = j.mloc;
    a.loss = d_loss;
    a.n_sites = (double)h->N;
    a.ckpt = j.fwd_only ? nullptr : h->ackpt.as<double>();
    a.ckpt_every = C;
    a.n_ckpt = K;
    a.V = V;
    const dim3 grid(tiles, (unsigned)B), gridc((G + 255) / 256, (unsigned)B);
    const cmd::SVec none{nullptr, 0};
    // forward: loss terms every step, checkpoints every C steps
    {
        const cmd::SVec y{base, V}, acc{base + B * V, V}, Ya{base + 2 * B * V, V}, Yb{base + 3 * B * V, V};
        cmd::stream_load_kernel<NAT><<<gridc, 256, 0, st>>>(j.y0, (long long)G * NAT * 3, G, y);
        if (int rc = h->snbase.ensure(sizeof(long long))) return rc;
        cmd::StreamArgs af = a;                      // steps relative to the device step base
        af.nbase = h->snbase.as<long long>();
        std::vector<unsigned char> key;
        key_add(key, 2);                             // adjoint forward stages of this NAT/Z/LZ
        key_add(key, NAT * 100 + Z * 10 + LZ);
        key_add(key, cp);
        key_add(key, af);
        key_add(key, y);
        key_add(key, acc);
        key_add(key, Ya);
        key_add(key, Yb);
        key_add(key, grid);
        const int64_t per = stream_group(h, B, V, 4), groups = (B + per - 1) / per;
        key_add(key, per);
        auto enqueue = [&](int64_t i, int64_t k) {
            cmd::StreamArgs ag = af;
            ag.b0 = (int)(i * per);
            const dim3 gg(tiles, (unsigned)std::min(per, B - i * per));
            stage<NAT, Z, LZ, PAIR>(0, gg, st, cp, ag, k, y, y, acc, Ya, 1);
            stage<NAT, Z, LZ, PAIR>(1, gg, st, cp, ag, k, Ya, y, acc, Yb, 1);
            stage<NAT, Z, LZ, PAIR>(2, gg, st, cp, ag, k, Yb, y, acc, Ya, 1);
            stage<NAT, Z, LZ, PAIR>(3, gg, st, cp, ag, k, Ya, y, acc, y, 1);
        };
        int32_t nl = 0;
        if (int rc = run_steps(h, st, S, groups, key, enqueue, &nl)) return rc;
        cmd::stream_obs_kernel<NAT, Z, LZ, PAIR><<<grid, cmd::kStreamTile, 0, st>>>(cp, a, y);
        cmd::stream_reduce_kernel<NAT><<<(unsigned)B, cmd::kStreamTile, 0, st>>>(a, S);
        CUDA_TRY(cudaGetLastError());
        CUDA_TRY(cudaMemcpy2DAsync(j.out, (1 + kAdjParams) * sizeof(double), d_loss, sizeof(double), sizeof(double),
                                   (size_t)B, cudaMemcpyDeviceToDevice, st));
    }
    if (j.fwd_only) return CMD_OK;
    cmd::ParamDerivs<NAT, Z, NQ> pd;
    std::memset(&pd, 0, sizeof(pd));
    for (int q = 0; q < NQ; ++q)
        for (int at = 0; at < NAT; ++at) {
            for (int sl = 0; sl < Z; ++sl)
                std::memcpy(pd.DJ[q][at][sl], &DJ[(((size_t)q * NAT + at) * Z + sl) * 9], 9 * sizeof(double));
            std::memcpy(pd.DB[q][at], &DB[((size_t)q * NAT + at) * 3], 3 * sizeof(double));
            std::memcpy(pd.DA[q][at], &DA[((size_t)q * NAT + at) * 9], 9 * sizeof(double));
        }
    pd.has_DA = has_DA;
    for (int q = 0; q < NQ; ++q)
        for (int at = 0; at < NAT; ++at)
            for (int sl = 0; sl < Z; ++sl)
                for (int e = 0; e < 9; ++e) pd.dj_any[q] |= pd.DJ[q][at][sl][e] != 0.0;
    cmd::StreamVjpArgs v{};
    v.G = G;
    v.tiles = tiles;
    v.nbr = a.nbr;
    v.dt = j.dt;
    v.n_steps = S;
    v.drive = a.drive;
    v.target = j.target;
    v.mloc = j.mloc;
    v.n_sites = a.n_sites;
    v.gpart = h->sgpart.as<double>();
    cmd::StreamArgs ar = a;              // recompute: no observables, no checkpoints
    ar.ckpt = nullptr;
    CUDA_TRY(cudaMemsetAsync(v.gpart, 0, (size_t)B * tiles * cmd::kPart * sizeof(double), st));
    const cmd::SVec lam{base, V}, acc{base + B * V, V}, Sv{base + 2 * B * V, V};
    const cmd::SVec hb[2] = {{base + 3 * B * V, V}, {base + 4 * B * V, V}};
    cmd::stream_lam_init_kernel<NAT><<<gridc, 256, 0, st>>>(v, lam);
    double* seg = h->aseg.as<double>();
    auto slot = [&](int64_t jj, int q) { return cmd::SVec{seg + (jj * 4 + q) * V, C * 4 * V}; };
    const double dt = j.dt;
    // One checkpoint segment of len steps: the recompute that stores every
    // stage input, then the reverse sweep; kernel step arguments are nb + jj.
    auto segment = [&](int64_t len, int64_t nb, const cmd::StreamArgs& sa, const cmd::StreamVjpArgs& sv) {
        for (int64_t jj = 0; jj < len; ++jj) {
            const int64_t n = nb + jj;
            const cmd::SVec y = slot(jj, 0);
            const cmd::SVec last = jj + 1 < len ? slot(jj + 1, 0) : none;
            stage<NAT, Z, LZ, PAIR>(0, grid, st, cp, sa, n, y, y, acc,
                                                                                   slot(jj, 1), 0);
            stage<NAT, Z, LZ, PAIR>(1, grid, st, cp, sa, n, slot(jj, 1), y, acc,
                                                                                   slot(jj, 2), 0);
            stage<NAT, Z, LZ, PAIR>(2, grid, st, cp, sa, n, slot(jj, 2), y, acc,
                                                                                   slot(jj, 3), 0);
            stage<NAT, Z, LZ, PAIR>(3, grid, st, cp, sa, n, slot(jj, 3), y, acc,
                                                                                   last, 0);
        }
        cmd::stream_hbar_kernel<NAT><<<grid, cmd::kStreamTile, 0, st>>>(G, dt / 6.0, slot(len - 1, 3), lam, hb[0]);
        for (int64_t jj = len - 1; jj >= 0; --jj) {
            const int64_t n = nb + jj;
            auto vjp0 = cmd::stream_vjp_kernel<NAT, Z, LZ, NQ, PAIR, 0>;
            auto vjp1 = cmd::stream_vjp_kernel<NAT, Z, LZ, NQ, PAIR, 1>;
            auto vjp2 = cmd::stream_vjp_kernel<NAT, Z, LZ, NQ, PAIR, 2>;
            const double c6 = dt / 6.0, c3 = dt / 3.0;
            const cmd::VjpStage s3{3, c6, 0.0, c3, dt}, s2{2, c3, dt, c3, 0.5 * dt};
            const cmd::VjpStage s1{1, c3, 0.5 * dt, c6, 0.5 * dt}, s0{0, c6, 0.5 * dt, c6, 0.0};
            vjp0<<<grid, cmd::kStreamTile, 0, st>>>(cp, pd, sv, s3, n, slot(jj, 3), hb[0], lam, Sv, acc, slot(jj, 2), hb[1]);
            vjp1<<<grid, cmd::kStreamTile, 0, st>>>(cp, pd, sv, s2, n, slot(jj, 2), hb[1], lam, Sv, acc, slot(jj, 1), hb[0]);
            vjp1<<<grid, cmd::kStreamTile, 0, st>>>(cp, pd, sv, s1, n, slot(jj, 1), hb[0], lam, Sv, acc, slot(jj, 0), hb[1]);
            vjp2<<<grid, cmd::kStreamTile, 0, st>>>(cp, pd, sv, s0, n, slot(jj, 0), hb[1], lam, Sv, acc,
                                                  jj > 0 ? slot(jj - 1, 3) : none, hb[0]);
        }
    };
    // Full-length segments replay a captured graph of the segment with the
    // kernels' steps relative to the device step base (set to the segment's
    // first step before each replay).  The partial segment (processed first)
    // and, with graphs off, every segment launch directly.
    if (int rc = h->snbase.ensure(sizeof(long long))) return rc;
    cmd::StreamArgs ar_rel = ar;
    ar_rel.nbase = h->snbase.as<long long>();
    cmd::StreamVjpArgs v_rel = v;
    v_rel.nbase = h->snbase.as<long long>();
    for (int64_t sg = K - 1; sg >= 0; --sg) {
        const int64_t n0 = sg * C, n1 = std::min(n0 + C, S);
        CUDA_TRY(cudaMemcpy2DAsync(seg, (size_t)C * 4 * V * sizeof(double), h->ackpt.as<double>() + sg * V,
                                   (size_t)K * V * sizeof(double), (size_t)V * sizeof(double), (size_t)B,
                                   cudaMemcpyDeviceToDevice, st));
        const int64_t len = n1 - n0;
        if (!h->graphs || len != C || K < 3) {
            segment(len, n0, ar, v);
            CUDA_TRY(cudaGetLastError());
            continue;
        }
        std::vector<unsigned char> key;
        key_add(key, 3);                             // adjoint segment of this NAT/Z/LZ/NQ
        key_add(key, NAT * 10000 + Z * 1000 + LZ * 100 + NQ * 10 + PAIR);
        key_add(key, cp);
        key_add(key, pd);
        key_add(key, ar_rel);
        key_add(key, v_rel);
        key_add(key, lam);
        key_add(key, seg);
        key_add(key, C);
        key_add(key, grid);
        key_add(key, dt);
        cmd::stream_set_base_kernel<<<1, 32, 0, st>>>(h->snbase.as<long long>(), n0);
        CUDA_TRY(cudaGetLastError());
        cudaGraphExec_t& ex = h->adj_graph;
        if (!ex || h->adj_graph_key != key) {
            if (ex) {
                cudaStreamSynchronize(st);
                cudaGraphExecDestroy(ex);
                ex = nullptr;
            }
            h->adj_graph_key.clear();
            cudaGraph_t g = nullptr;
            CUDA_TRY(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
            segment(len, 0, ar_rel, v_rel);
            const cudaError_t e = cudaStreamEndCapture(st, &g);
            if (e != cudaSuccess || !g) {
                if (g) cudaGraphDestroy(g);
                return fail(CMD_ERR_CUDA, std::string("stream capture: ") + cudaGetErrorString(e));
            }
            const cudaError_t e2 = cudaGraphInstantiate(&ex, g, 0);
            cudaGraphDestroy(g);
            if (e2 != cudaSuccess) {
                ex = nullptr;
                return fail(CMD_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e2));
            }
            h->adj_graph_key = key;
        }
        CUDA_TRY(cudaGraphLaunch(ex, st));
    }
    cmd::stream_grad_kernel<<<(unsigned)B, 32 * NQ, 0, st>>>(v.gpart, tiles, NQ, j.out + 1, 1 + kAdjParams);
    CUDA_TRY(cudaGetLastError());
    return CMD_OK;
}

// Threads per CTA and shared memory per CTA of variant V on layout L.
}  // namespace

void release_stream_graph(cmd_handle* h) {
    if (h->stream) cudaStreamSynchronize(h->stream);
    if (h->stream_graph) cudaGraphExecDestroy(h->stream_graph);
    h->stream_graph = nullptr;
    h->stream_graph_key.clear();
    for (int i = 0; i < 2; ++i) {
        if (h->call_graph[i]) cudaGraphExecDestroy(h->call_graph[i]);
        h->call_graph[i] = nullptr;
        h->call_sig[i].clear();
    }
    if (h->adj_graph) cudaGraphExecDestroy(h->adj_graph);
    h->adj_graph = nullptr;
    h->adj_graph_key.clear();
}

namespace {

// The node types in order and, per kernel node, its function, grid, block,
// dynamic shared memory and cluster shape: what an in-place update of an
// executable graph may not change.  False when a query fails.
bool graph_signature(cudaGraph_t g, std::vector<unsigned char>& sig) {
    size_t n = 0;
    if (cudaGraphGetNodes(g, nullptr, &n) != cudaSuccess) return false;
    std::vector<cudaGraphNode_t> nodes(n);
    if (n && cudaGraphGetNodes(g, nodes.data(), &n) != cudaSuccess) return false;
    sig.clear();
    key_add(sig, n);
    for (cudaGraphNode_t nd : nodes) {
        cudaGraphNodeType t;
        if (cudaGraphNodeGetType(nd, &t) != cudaSuccess) return false;
        key_add(sig, (int)t);
        if (t != cudaGraphNodeTypeKernel) continue;
        cudaKernelNodeParams p{};
        if (cudaGraphKernelNodeGetParams(nd, &p) != cudaSuccess) return false;
        key_add(sig, p.func);
        key_add(sig, p.gridDim);
        key_add(sig, p.blockDim);
        key_add(sig, p.sharedMemBytes);
        cudaLaunchAttributeValue v{};                  // zeros where the node has no cluster shape
        if (cudaGraphKernelNodeGetAttribute(nd, cudaLaunchAttributeClusterDimension, &v) != cudaSuccess) {
            (void)cudaGetLastError();
            v = cudaLaunchAttributeValue{};
        }
        key_add(sig, v.clusterDim.x);
        key_add(sig, v.clusterDim.y);
        key_add(sig, v.clusterDim.z);
    }
    return true;
}

}  // namespace

int graph_call(cmd_handle* h, int slot, cudaStream_t st, const std::function<int()>& enqueue) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    const bool capture = h->graphs && st != nullptr && st != cudaStreamLegacy && st != cudaStreamPerThread &&
                         cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone;
    if (!capture) return enqueue();
    // relaxed: the launch helpers set kernel attributes, which is not stream work
    CUDA_TRY(cudaStreamBeginCapture(st, cudaStreamCaptureModeRelaxed));
    const int rc = enqueue();
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(st, &g);
    if (rc != CMD_OK || e != cudaSuccess || !g) {
        if (g) cudaGraphDestroy(g);
        (void)cudaGetLastError();
        if (rc != CMD_OK) return rc;
        return fail(CMD_ERR_CUDA, std::string("stream capture: ") + cudaGetErrorString(e));
    }
    // Same kernels and launch shapes as the kept graph: update its arguments in
    // place; otherwise (or when the update is refused) build a new one.
    std::vector<unsigned char> sig;
    const bool have_sig = graph_signature(g, sig);
    (void)cudaGetLastError();
    cudaGraphExec_t& ex = h->call_graph[slot];
    bool updated = false;
    if (ex && have_sig && sig == h->call_sig[slot]) {
        cudaGraphExecUpdateResultInfo info{};
        updated = cudaGraphExecUpdate(ex, g, &info) == cudaSuccess;
        (void)cudaGetLastError();
    }
    if (ex && !updated) {
        cudaStreamSynchronize(st);                    // the old graph's last launch is done
        cudaGraphExecDestroy(ex);
        ex = nullptr;
    }
    h->call_sig[slot] = have_sig ? sig : std::vector<unsigned char>();
    if (!ex) {
        const cudaError_t e2 = cudaGraphInstantiate(&ex, g, 0);
        if (e2 != cudaSuccess) {
            ex = nullptr;
            cudaGraphDestroy(g);
            return fail(CMD_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e2));
        }
    }
    cudaGraphDestroy(g);
    CUDA_TRY(cudaGraphLaunch(ex, st));
    return CMD_OK;
}

int run_streamed(cmd_handle* h, const RunSpec& r, cudaStream_t st, int32_t* launches) {
    switch (global_type(h->lay)) {
        case 0: return stream_forward<2, 3, 1, false>(h, r, st, launches);
        case 1:
            return h->lay.paired ? stream_forward<4, 6, 3, true>(h, r, st, launches)
                                 : stream_forward<4, 6, 3, false>(h, r, st, launches);
        default: return no_instance(h->lay);
    }
}

int run_stream_adjoint(cmd_handle* h, const StreamAdjJob& j, int n_params, const std::vector<double>& DJ,
                       const std::vector<double>& DB, const std::vector<double>& DA, bool has_DA) {
    const int ty = global_type(h->lay);
    if (ty < 0) return no_instance(h->lay);
    // paired bonds: their parameter derivatives must be too
    const Layout& L = h->lay;
    bool pair = L.paired;
    const int nq = n_params <= 4 ? 4 : 5;
    for (int q = 0; q < nq && pair; ++q)
        for (int at = 0; at < L.NA && pair; ++at)
            for (int n = 0; n < L.LZ && pair; ++n) {
                const double* D = &DJ[((size_t)q * L.NA + at) * L.Z * 9];
                pair = std::memcmp(D + 9 * n, D + 9 * (L.LZ + L.pair[at * L.LZ + n]), 9 * sizeof(double)) == 0;
            }
    // the VJP carries as many parameter cotangents as requested (4 or 5)
    if (ty == 0)
        return nq == 4 ? stream_adjoint<2, 3, 1, 4, false>(h, j, DJ, DB, DA, has_DA)
                       : stream_adjoint<2, 3, 1, 5, false>(h, j, DJ, DB, DA, has_DA);
    if (pair)
        return nq == 4 ? stream_adjoint<4, 6, 3, 4, true>(h, j, DJ, DB, DA, has_DA)
                       : stream_adjoint<4, 6, 3, 5, true>(h, j, DJ, DB, DA, has_DA);
    return nq == 4 ? stream_adjoint<4, 6, 3, 4, false>(h, j, DJ, DB, DA, has_DA)
                   : stream_adjoint<4, 6, 3, 5, false>(h, j, DJ, DB, DA, has_DA);
}

}  // namespace cmd
