// Work-tile shapes and their autotuner (include/rh3t.h rh3t_set_tile_shapes,
// rh3t_autotune). A shape is per instance and travels in every Tile record,
// so one launch mixes instances tuned to different shapes; the arithmetic of
// a face or a cell does not depend on the shape.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "context.h"
#include "kernels.cuh"

using namespace rh3t;

namespace {

struct ClassKey {
    int nx, ny, diffusion;
    bool operator<(const ClassKey& o) const {
        return std::tie(nx, ny, diffusion) < std::tie(o.nx, o.ny, o.diffusion);
    }
};

std::mutex g_mu;
std::map<ClassKey, Shape> g_cache; // process-wide tuning results

bool shape_ok(int lgx, int lgy, int lgr) {
    return lgx >= FX_LG_MIN && lgx <= FX_LG_MAX && lgy >= FY_LG_MIN && lgy <= FY_LG_MAX && lgr >= RHS_LG_MIN &&
           lgr <= RHS_LG_MAX;
}

// cache file: kCacheHead, then one "nx ny diffusion lg_fx lg_fy lg_rhs" line per class. A
// file with another first line holds shapes that were timed on other kernels (before
// the heading, x and y faces apart): it is not read, and rewritten.
const char* const kCacheHead = "rh3t tile shapes 2\n";

void load_cache(const char* path) {
    FILE* f = std::fopen(path, "r");
    if (!f) return;
    char head[64] = {0};
    int nx, ny, df, a, b, r;
    if (std::fgets(head, sizeof(head), f) && std::strcmp(head, kCacheHead) == 0)
        while (std::fscanf(f, "%d %d %d %d %d %d", &nx, &ny, &df, &a, &b, &r) == 6)
            if (shape_ok(a, b, r)) g_cache[ClassKey{nx, ny, df}] = Shape{a, b, r};
    std::fclose(f);
}

bool save_cache(const char* path) {
    std::string tmp = std::string(path) + ".tmp";
    FILE* f = std::fopen(tmp.c_str(), "w");
    if (!f) return false;
    std::fputs(kCacheHead, f);
    for (const auto& kv : g_cache)
        std::fprintf(f, "%d %d %d %d %d %d\n", kv.first.nx, kv.first.ny, kv.first.diffusion, kv.second.lgx,
                     kv.second.lgy, kv.second.lgr);
    bool ok = std::fclose(f) == 0;
    return ok && std::rename(tmp.c_str(), path) == 0;
}

enum Kind { KX = 0, KY = 1, KR = 2 };

// Tiles of one kind of every instance, kept per instance so that a trial rebuilds its class's alone
using Tiles = std::vector<std::vector<Tile>>;
void build_tiles(const rh3t_ctx* c, const std::vector<int>& of, Kind kind, const Shape& sh, Tiles& t) {
    for (int k : of) {
        t[k].clear();
        instance_tiles(c->hi[k], sh, k, kind == KX ? &t[k] : nullptr, kind == KY ? &t[k] : nullptr,
                       kind == KR ? &t[k] : nullptr);
    }
}
int upload_tiles(rh3t_ctx* c, const Tiles& t, Tile** d, int* n) {
    std::vector<Tile> all;
    for (const auto& v : t) all.insert(all.end(), v.begin(), v.end());
    *n = (int)all.size();
    CK(c, cudaMalloc(d, std::max<size_t>(all.size(), 1) * sizeof(Tile)));
    CK(c, cudaMemcpyAsync(*d, all.data(), all.size() * sizeof(Tile), cudaMemcpyHostToDevice, c->stream));
    CK(c, cudaStreamSynchronize(c->stream));
    return RH3T_OK;
}

// Minimum over `reps` of the launch that a step makes, with these shapes: the fluxes of
// both directions of all instances (kind KX or KY; tx and ty), or the cell update (KR; tx).
// Timed alone, a direction or a class runs with another number of thread groups a
// tile and another shared memory than in the step, and a shape's cost to the
// others does not show: ensembles of 24 and 96 took 4 x 16 x faces for a third of their
// instances, and a flux block a SM less for all of them (0.6% slower than untuned).
int time_launch(rh3t_ctx* c, Kind kind, const std::vector<Shape>& shapes, const Tiles& tx, const Tiles& ty, int reps,
                double* ms_out) {
    *ms_out = 0.0;
    cudaStream_t s = c->stream;
    Tile *dx = nullptr, *dy = nullptr;
    int nx = 0, ny = 0, smem = 0;
    FluxSize z{0, 0, false};
    for (int k = 0; k < c->n_inst; ++k) {
        z.npx = std::max(z.npx, flux_points(0, shapes[k].lgx));
        z.npy = std::max(z.npy, flux_points(1, shapes[k].lgy));
        z.diffusion = z.diffusion || c->hi[k].diffusion;
        smem = std::max(smem, rhs_smem(shapes[k].lgr));
    }
    int rc = upload_tiles(c, tx, &dx, &nx);
    if (!rc && kind != KR) rc = upload_tiles(c, ty, &dy, &ny);
    if (rc || nx + ny == 0) {
        cudaFree(dx);
        cudaFree(dy);
        return rc;
    }
    cudaEvent_t a = nullptr, b = nullptr;
    cudaError_t e = cudaEventCreate(&a);
    if (e == cudaSuccess) e = cudaEventCreate(&b);
    auto launch = [&]() {
        if (kind == KR) launch_rhs_stage(s, c->d_inst, dx, nx, 0, 0, c->d_io2, smem);
        else launch_flux(s, c->d_inst, dx, nx, dy, ny, 0, z);
        c->launches += 1;
    };
    double best = 1e30;
    if (e == cudaSuccess) {
        for (int r = 0; r < 3; ++r) launch(); // warm-up
        for (int r = 0; r < reps && e == cudaSuccess; ++r) {
            cudaEventRecord(a, s);
            launch();
            cudaEventRecord(b, s);
            e = cudaEventSynchronize(b);
            float ms = 0.f;
            if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, a, b);
            best = std::min(best, (double)ms);
        }
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (a) cudaEventDestroy(a);
    if (b) cudaEventDestroy(b);
    cudaStreamSynchronize(s);
    cudaFree(dx);
    cudaFree(dy);
    CK(c, e);
    *ms_out = best;
    return RH3T_OK;
}

// a shape replaces the default where it takes this much less: minima of one shape's
// launches repeat to about 0.5% in an ensemble, to 4% at 13 us
constexpr double TUNE_GAIN = 0.97;

} // namespace

extern "C" int rh3t_set_tile_shapes(rh3t_ctx* c, int32_t k, int32_t lg_fx, int32_t lg_fy, int32_t lg_rhs) {
    if (!c) return RH3T_ERR_INVALID_ARGUMENT;
    if (k < -1 || k >= c->n_inst || !shape_ok(lg_fx, lg_fy, lg_rhs))
        return set_error(c, RH3T_ERR_INVALID_ARGUMENT, "tile shape or instance out of range");
    CK(c, cudaSetDevice(c->device));
    for (int q = 0; q < c->n_inst; ++q)
        if (k < 0 || q == k) c->hi[q].shape = Shape{lg_fx, lg_fy, lg_rhs};
    return make_tiles(c);
}

extern "C" int rh3t_get_tile_shapes(const rh3t_ctx* c, int32_t k, int32_t* lg3) {
    if (!c || !lg3 || k < 0 || k >= c->n_inst) return RH3T_ERR_INVALID_ARGUMENT;
    const Shape& s = c->hi[k].shape;
    lg3[0] = s.lgx;
    lg3[1] = s.lgy;
    lg3[2] = s.lgr;
    return RH3T_OK;
}

extern "C" int rh3t_autotune(rh3t_ctx* c, const char* cache_path, int32_t reps, rh3t_tune_entry* out,
                             int32_t max_out, int32_t* n_out) {
    if (!c) return RH3T_ERR_INVALID_ARGUMENT;
    CK(c, cudaSetDevice(c->device));
    reps = std::max(1, std::min(reps, 100));
    std::lock_guard<std::mutex> lock(g_mu);
    if (cache_path) load_cache(cache_path);
    std::map<ClassKey, std::vector<int>> classes;
    for (int k = 0; k < c->n_inst; ++k)
        classes[ClassKey{(int)c->hi[k].nx, (int)c->hi[k].ny, c->hi[k].diffusion}].push_back(k);
    // every class at its cached shape, or the default of its grid
    std::vector<Shape> shapes((size_t)c->n_inst);
    bool measure = false;
    for (const auto& kv : classes) {
        const auto hit = g_cache.find(kv.first);
        measure = measure || hit == g_cache.end();
        for (int k : kv.second)
            shapes[k] = hit != g_cache.end() ? hit->second : default_shape(kv.first.nx, kv.first.ny);
    }
    Tiles t[3];
    double ms_now[3] = {0.0, 0.0, 0.0}; // of the launch with `shapes` (KX and KY: the same)
    if (measure) {
        for (int kind = 0; kind < 3; ++kind) {
            t[kind].resize((size_t)c->n_inst);
            for (int k = 0; k < c->n_inst; ++k) build_tiles(c, {k}, (Kind)kind, shapes[k], t[kind]);
        }
        int rc = time_launch(c, KX, shapes, t[KX], t[KY], reps, &ms_now[KX]);
        if (!rc) rc = time_launch(c, KR, shapes, t[KR], t[KR], reps, &ms_now[KR]);
        if (rc) return rc;
    }
    std::vector<rh3t_tune_entry> entries;
    for (const auto& kv : classes) {
        const std::vector<int>& of = kv.second;
        rh3t_tune_entry E{};
        E.nx = kv.first.nx;
        E.ny = kv.first.ny;
        E.diffusion = kv.first.diffusion;
        E.n_instances = (int)of.size();
        if (g_cache.count(kv.first)) {
            E.from_cache = 1;
        } else {
            const int lo[3] = {FX_LG_MIN, FY_LG_MIN, RHS_LG_MIN}, hi[3] = {FX_LG_MAX, FY_LG_MAX, RHS_LG_MAX};
            double* ms[3] = {E.ms_fx, E.ms_fy, E.ms_rhs};
            for (int kind = 0; kind < 3; ++kind) {
                const Shape base = shapes[of[0]];
                auto lg = [kind](Shape& s) -> int& { return kind == KX ? s.lgx : (kind == KY ? s.lgy : s.lgr); };
                Shape now = base;
                const int lg0 = lg(now);
                double& current = ms_now[kind == KR ? KR : KX];
                double tbest = TUNE_GAIN * current;
                int pick = lg0;
                for (int q = lo[kind]; q <= hi[kind]; ++q) {
                    double time = current;
                    if (q != lg0) {
                        Shape sh = base;
                        lg(sh) = q;
                        for (int k : of) shapes[k] = sh;
                        build_tiles(c, of, (Kind)kind, sh, t[kind]);
                        int rc = kind == KR ? time_launch(c, KR, shapes, t[KR], t[KR], reps, &time)
                                            : time_launch(c, (Kind)kind, shapes, t[KX], t[KY], reps, &time);
                        if (rc) return rc;
                        if (time < tbest) {
                            tbest = time;
                            pick = q;
                        }
                    }
                    ms[kind][q - lo[kind]] = time;
                }
                lg(now) = pick;
                for (int k : of) shapes[k] = now;
                build_tiles(c, of, (Kind)kind, now, t[kind]);
                if (pick != lg0) current = tbest;
            }
            g_cache[kv.first] = shapes[of[0]];
        }
        E.lg_fx = shapes[of[0]].lgx;
        E.lg_fy = shapes[of[0]].lgy;
        E.lg_rhs = shapes[of[0]].lgr;
        entries.push_back(E);
    }
    for (int k = 0; k < c->n_inst; ++k) c->hi[k].shape = shapes[k];
    int rc = make_tiles(c);
    if (rc) return rc;
    if (cache_path && !save_cache(cache_path))
        return set_error(c, RH3T_ERR_INVALID_ARGUMENT, "cannot write the tuning cache file");
    if (out)
        for (int q = 0; q < (int)entries.size() && q < max_out; ++q) out[q] = entries[q];
    if (n_out) *n_out = (int)entries.size();
    return RH3T_OK;
}
