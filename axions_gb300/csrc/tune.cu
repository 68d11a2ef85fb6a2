// Autotuning of the tiled FP32 step: the number of x-planes each CTA marches
// through ("chunk").  Short chunks give small lattices enough CTAs to fill the
// 152 SMs; long chunks spend less on each CTA's prologue (one extra plane of
// link data and the pipeline fill).  lat_autotune() times candidates, every default
// among them, on a
// scratch lattice of the caller's shape (device-generated IC, the caller's
// state is not touched), applies the fastest to the handle and remembers it
// per shape; new handles of a tuned shape start with the remembered value and
// untuned ones with the cheapest chunk of a fitted cost model.  The cache can
// be saved to and loaded from a small JSON file.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <fstream>
#include <map>
#include <mutex>
#include <set>
#include <sstream>
#include <string>
#include <tuple>
#include <vector>

#include "lattice_handle.hpp"

using namespace lat;

namespace {

using Key = std::tuple<int, int, int, int64_t, int64_t, int64_t>;  // model, precision, bc, nx, ny, nz

struct Entry {
    int chunk;
    double ms;
};

std::mutex g_tune_mu;
std::map<Key, Entry> g_tune;

Key key_of(const lat_params& p) { return Key(p.model, p.precision, p.bc, p.nx, p.ny, p.nz); }

// Timed by lat_autotune: the long ones, then the others default_chunk may pick.
const int kLong[] = {4, 8, 16, 32, 64, 128};
const int kOthers[] = {1, 2, 6, 12, 24};

}  // namespace

namespace lat {

// Time of an x-marching FP32 step, in arbitrary units, with `ctas` CTAs of
// `chunk` planes each: a CTA's prologue costs about 1.7 planes; a plane takes
// 0.4, and 0.41 for each of the SM's CTAs (latency and throughput).  Fitted to
// chunks of 1..128 on 32^3 .. 384^3, both models; the chunk it picks is within
// 5 % of the best one measured, where the rule before it (the largest chunk
// with four CTAs per SM) lost 5 % at 384^3 (645 -> 614 us), 14 % at 201x199x203
// (169 -> 146) and 28 % at 40x36x33 (8.7 -> 6.3).
static double march_cost(int chunk, double ctas)
{
    return (chunk + 1.7) * (0.4 + 0.41 * std::ceil(ctas / 152));
}

static double march_ctas(const lat_params& p, int chunk)
{
    const Geom g = make_geom(p);
    return (double)march_tiles(g, p.model == LAT_MODEL_MOORE) * ((g.hix - g.lox - 1) / chunk + 1);
}

// The cheapest chunk by march_cost.
static int model_chunk(const lat_params& p)
{
    int best = 1;
    double cost = 1e300;
    for (int c : {1, 2, 4, 6, 8, 12, 16, 24, 32}) {
        const double t = march_cost(c, march_ctas(p, c));
        if (t < cost) {
            cost = t;
            best = c;
        }
    }
    return best;
}

// Default chunk for a handle: the tuned value of its shape, else the model's.
int default_chunk(const lat_params& p)
{
    {
        std::lock_guard<std::mutex> lock(g_tune_mu);
        auto it = g_tune.find(key_of(p));
        if (it != g_tune.end()) return it->second.chunk;
    }
    return model_chunk(p);
}

// Sets a handle's chunk and the one its steps are launched with: the same, except
// that one longer than the model's choice gives way to it where it leaves SMs
// without a CTA or is more than 10 % dearer by the model, twice what that is off by.
// Files tuned to longer chunks and chunks set for another shape leave a small
// lattice with too few CTAs otherwise: 32^3 with 4 planes takes 5.3 us a step, with 1
// 2.5; 64x48x40 6.5 with 4 and 5.1 with 2; 40x36x33 6.4 with 4 and 4.0 with 1.
void set_chunk(lat_handle* h, int chunk)
{
    const int model = model_chunk(h->p);
    const double ctas = march_ctas(h->p, chunk), best = march_ctas(h->p, model);
    h->chunk = chunk;
    h->launch_chunk =
        chunk > model && (ctas < 152 || march_cost(chunk, ctas) > 1.1 * march_cost(model, best)) ? model : chunk;
}

}  // namespace lat

extern "C" {

int lat_get_tuning(const lat_handle* h, lat_tuning* out)
{
    if (!h || !out) {
        set_error("lat_get_tuning: null argument");
        return LAT_ERR_INVALID;
    }
    out->chunk = h->chunk;
    out->candidates = 0;
    out->ms_per_step = 0;
    std::lock_guard<std::mutex> lock(g_tune_mu);
    auto it = g_tune.find(key_of(h->p));
    if (it != g_tune.end() && it->second.chunk == h->chunk) out->ms_per_step = it->second.ms;
    return LAT_OK;
}

int lat_set_tuning(lat_handle* h, const lat_tuning* t)
{
    if (!h || !t || t->chunk < 1) {
        set_error("lat_set_tuning: bad argument");
        return LAT_ERR_INVALID;
    }
    set_chunk(h, t->chunk);
    return LAT_OK;
}

int lat_autotune(lat_handle* h, int32_t trial_steps, lat_tuning* out)
{
    if (!h || trial_steps < 1) {
        set_error("lat_autotune: bad argument");
        return LAT_ERR_INVALID;
    }
    if (h->elem != 4 || h->p.kernel_variant == 1) {  // only the tiled FP32 step has a chunk
        if (out) {
            out->chunk = h->chunk;
            out->candidates = 0;
            out->ms_per_step = 0;
        }
        return LAT_OK;
    }
    lat_handle* t = nullptr;
    int rc = lat_create(&h->p, &t);
    if (rc) return rc;
    rc = lat_random_phase_ic_device(t, 12345, 1);
    if (rc) {
        lat_destroy(t);
        return rc;
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const Geom& g = h->geom;
    double best_ms = 1e300;
    int best = h->chunk, tried = 0;
    std::set<int> launched;   // the chunks timed, as launched
    auto time = [&](int c) {   // the fastest of three runs
        launched.insert(t->launch_chunk);
        ++tried;
        for (int run = 0; run < 3; ++run) {
            if ((rc = lat_step(t, 1))) return;  // warm-up
            cudaEventRecord(e0, t->stream);
            if ((rc = lat_step(t, trial_steps))) return;
            cudaEventRecord(e1, t->stream);
            cudaEventSynchronize(e1);
            float ms = 0;
            cudaEventElapsedTime(&ms, e0, e1);
            if (ms / trial_steps < best_ms) {
                best_ms = ms / trial_steps;
                best = c;
            }
        }
    };
    for (int c : kLong) {
        if (rc || (c > 2 * (g.hix - g.lox) && c != kLong[0])) continue;  // beyond the lattice: same as a shorter one
        set_chunk(t, c);
        time(c);
    }
    for (int c : kOthers) {
        set_chunk(t, c);
        if (!rc && !launched.count(t->launch_chunk)) time(c);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    lat_destroy(t);
    if (rc) return rc;
    set_chunk(h, best);
    {
        std::lock_guard<std::mutex> lock(g_tune_mu);
        g_tune[key_of(h->p)] = {best, best_ms};
    }
    if (out) {
        out->chunk = best;
        out->candidates = tried;
        out->ms_per_step = best_ms;
    }
    return LAT_OK;
}

int lat_tune_cache_save(const char* path)
{
    if (!path) {
        set_error("lat_tune_cache_save: null path");
        return LAT_ERR_INVALID;
    }
    std::ofstream o(path);
    if (!o) {
        set_error(std::string("lat_tune_cache_save: cannot write ") + path);
        return LAT_ERR_INVALID;
    }
    std::lock_guard<std::mutex> lock(g_tune_mu);
    o << "{\"chunk\": [";
    bool first = true;
    for (auto& kv : g_tune) {
        const Key& k = kv.first;
        o << (first ? "" : ",") << "\n  {\"model\": " << std::get<0>(k) << ", \"precision\": " << std::get<1>(k)
          << ", \"bc\": " << std::get<2>(k) << ", \"nx\": " << std::get<3>(k) << ", \"ny\": " << std::get<4>(k)
          << ", \"nz\": " << std::get<5>(k) << ", \"chunk\": " << kv.second.chunk << ", \"ms\": " << kv.second.ms
          << "}";
        first = false;
    }
    o << "\n]}\n";
    return o.good() ? LAT_OK : LAT_ERR_INVALID;
}

// Reads files written by lat_tune_cache_save: one entry per line.
int lat_tune_cache_load(const char* path)
{
    if (!path) {
        set_error("lat_tune_cache_load: null path");
        return LAT_ERR_INVALID;
    }
    std::ifstream in(path);
    if (!in) {
        set_error(std::string("lat_tune_cache_load: cannot read ") + path);
        return LAT_ERR_INVALID;
    }
    std::string line;
    int loaded = 0;
    auto field = [](const std::string& l, const char* name, double& v) {
        const std::string pat = std::string("\"") + name + "\": ";
        const size_t at = l.find(pat);
        if (at == std::string::npos) return false;
        v = std::strtod(l.c_str() + at + pat.size(), nullptr);
        return true;
    };
    while (std::getline(in, line)) {
        double m, pr, bc, nx, ny, nz, ch, ms;
        if (field(line, "model", m) && field(line, "precision", pr) && field(line, "bc", bc) && field(line, "nx", nx) &&
            field(line, "ny", ny) && field(line, "nz", nz) && field(line, "chunk", ch) && field(line, "ms", ms) &&
            ch >= 1) {
            std::lock_guard<std::mutex> lock(g_tune_mu);
            g_tune[Key((int)m, (int)pr, (int)bc, (int64_t)nx, (int64_t)ny, (int64_t)nz)] = {(int)ch, ms};
            ++loaded;
        }
    }
    return loaded;
}

}  // extern "C"
