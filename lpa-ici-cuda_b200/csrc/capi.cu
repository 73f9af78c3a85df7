// capi.cu -- C ABI entry points for the forward path, the reference-shaped host engine and the
// tile-configuration table.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "configs.h"
#include "internal.h"

using namespace lpaici;

namespace lpaici {

int default_config(const lpaici_kernelset *ks) {
    int dev = 0, max_optin = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) {
        std::lock_guard<std::mutex> lock(ks->mu);
        if (dev < static_cast<int>(ks->tuned_config.size()) && ks->tuned_config[dev] >= 0)
            return ks->tuned_config[dev];
    }
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    static const int order[] = LPAICI_TILE_PREFERENCE;
    static_assert(sizeof(order) / sizeof(order[0]) == LPAICI_NUM_TILE_CONFIGS, "one preference per configuration");
    for (const int c : order)
        if (config_smem(c, ks->layout.total_words, ks->D * ks->S, ks->radius) + kStaticShared <= static_cast<size_t>(max_optin))
            return c;
    return LPAICI_DEFAULT_TILE_CONFIG;  // nothing fits: the launch reports LPAICI_ERR_UNSUPPORTED
}

// Time of one tile of configuration c on one SM of a B200 (1,965 MHz), for kernel sets that were not tuned:
//   base + per_work * W * (directions a round takes, rounded up) / D,   W = taps + 1.4 runs + 5 kernels,
// fitted to 4096^2 launches (time / waves) of the 16 x 7 symmetric set (W = 8,041) and the 8 x 4 set
// (W = 545); the tapered set (W = 14,552) is 4 % above its estimate.  A run costs about 1.4 taps beside its
// taps, a kernel's interval update about 5 (measured with synthetic kernel sets of one run length).  The last entry (64 x
// 16) stands to the 64 x 32 one a little above their measured times (61 x 61 64 and 89 us, 85 x 85 119 and 164; both are
// sets of one direction, whose 64 x 32 tiles take less than this table says).
struct TileCost {
    float base_us, ns_per_work;
    int ctas = 1;  // CTAs per SM of the fit
};
static const TileCost kTileCost[LPAICI_NUM_TILE_CONFIGS] = {{8.7f, 59.7f}, {8.1f, 31.2f}, {7.3f, 25.0f}, {4.2f, 15.8f},
                                                            {2.9f, 8.35f}, {0.6f, 4.58f}, {1.2f, 2.60f, 2}, {0.5f, 26.1f},
                                                            {9.0f, 47.3f}, {9.8f, 36.9f}, {4.8f, 19.5f}, {0.5f, 22.0f}};

static int groups_of(int c) {
#define LPAICI_GROUPS_CASE(idx, WX, WY, Q, DS) \
    case idx: return DS;
    switch (c) {
        LPAICI_TILE_CONFIGS(LPAICI_GROUPS_CASE)
        default: return 1;
    }
#undef LPAICI_GROUPS_CASE
}

// The same for a tile that a cluster shares, alone on its SMs (LPAICI_CLUSTERS; back to back in a graph 97 x 64 takes 12.8 us
// with the symmetric set and 17.3 us with the tapered one, 128 x 128 17.0 and 24.1 us, 150 x 120 22.7 and 36.2 us,
// 200 x 150 25.1 and 40.7 us).
static const TileCost kClusterCost[LPAICI_NUM_CLUSTERS] = {{5.3f, 0.72f}, {6.4f, 1.12f}, {4.2f, 2.1f}, {3.8f, 2.45f}};

static float estimated_ms(const lpaici_kernelset *ks, const TileCost &cost, int ds) {
    const int nk = ks->D * ks->S;
    const float work = static_cast<float>(ks->run_w.size()) + 1.4f * ks->layout.n_runs + 5.0f * nk;
    const float rounded = static_cast<float>((ks->D + ds - 1) / ds * ds) / ks->D;
    return 1e-3f * cost.base_us + 1e-6f * cost.ns_per_work * work * rounded;
}

// (one CTA an SM where the fit had two: 1.5 tile times, as for a lone one in choose_plan)
static float estimated_tile_ms(const lpaici_kernelset *ks, int c, int bps) {
    return estimated_ms(ks, kTileCost[c], groups_of(c)) * (bps < kTileCost[c].ctas ? 1.5f : 1.0f);
}

// CTAs per SM of configuration c for ks on device dev (cached; 0 when it does not fit every kernel of it).
static int cached_bps(const lpaici_kernelset *ks, int dev, int c, int max_optin) {
    {
        std::lock_guard<std::mutex> lock(ks->mu);
        if (dev < static_cast<int>(ks->blocks_per_sm.size()) && !ks->blocks_per_sm[dev].empty() &&
            ks->blocks_per_sm[dev][c] >= 0)
            return ks->blocks_per_sm[dev][c];
    }
    const size_t smem = config_smem(c, ks->layout.total_words, ks->D * ks->S, ks->radius);
    const int n = smem + kStaticShared <= static_cast<size_t>(max_optin) ? config_blocks_per_sm(c, smem) : 0;
    std::lock_guard<std::mutex> lock(ks->mu);
    if (static_cast<int>(ks->blocks_per_sm.size()) <= dev) ks->blocks_per_sm.resize(dev + 1);
    if (ks->blocks_per_sm[dev].empty()) ks->blocks_per_sm[dev].assign(LPAICI_NUM_TILE_CONFIGS, -1);
    ks->blocks_per_sm[dev][c] = n;
    return n;
}

static long tiles_of(int c, int width, int rows) {
    int tw = 1, th = 1;
    config_tile(c, &tw, &th);
    return static_cast<long>((width + tw - 1) / tw) * ((rows + th - 1) / th);
}

// Time until the last of n_small tiles of t is done, handed out as SMs get free after n_big tiles of big_t.
static double mixed_makespan(long n_big, double big_t, long n_small, double t, int sms) {
    const long waves = n_big / sms, rem = n_big % sms;  // rem SMs sweep one big tile more
    const double early = waves * big_t, late = early + (rem > 0 ? big_t : 0.0);
    const auto done = [&](double at) {  // small tiles finished by then
        const long a = static_cast<long>((at - early) / t + 1e-6), b = at > late ? static_cast<long>((at - late) / t + 1e-6) : 0;
        return a * (sms - rem) + b * rem;
    };
    const long before = done(late);  // the SMs of the last wave's gap
    if (before >= n_small) return std::max(late, early + t * ((n_small + sms - rem - 1) / (sms - rem)));
    const double by_late = late + t * ((n_small - before + sms - 1) / sms);
    const double by_early = early + t * static_cast<long>((by_late - early) / t + 1e-6);  // the early SMs' last end before it
    return by_early > late && done(by_early) >= n_small ? by_early : by_late;
}

// What a plan is chosen with: the tile times of a kernel set on the current device.
struct PlanCosts {
    int sms = 0, max_smem = 0;
    bool forced = false, tuned = false;
    int forced_config = 0;
    float tile_ms[LPAICI_NUM_TILE_CONFIGS];  // <= 0: does not fit
    int bps[LPAICI_NUM_TILE_CONFIGS];
};

static bool plan_costs(const lpaici_kernelset *ks, PlanCosts *pc) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    // the last configuration is for sets of one or two directions: others need not ask what fits of it (3 us of a new
    // set's first call)
    const int n = ks->D > 2 ? LPAICI_NUM_TILE_CONFIGS - 1 : LPAICI_NUM_TILE_CONFIGS;
    pc->bps[LPAICI_NUM_TILE_CONFIGS - 1] = 0;
    bool known = false;  // CTAs per SM of every configuration
    {
        std::lock_guard<std::mutex> lock(ks->mu);
        const bool have = dev < static_cast<int>(ks->tuned_config.size()) && ks->tuned_config[dev] >= 0;
        pc->tuned = dev < static_cast<int>(ks->tuned_tile_ms.size()) && !ks->tuned_tile_ms[dev].empty();
        if (have && !pc->tuned) {  // forced by lpaici_set_tile_config
            pc->forced = true;
            pc->forced_config = ks->tuned_config[dev];
            return true;
        }
        if (pc->tuned) std::copy_n(ks->tuned_tile_ms[dev].begin(), LPAICI_NUM_TILE_CONFIGS, pc->tile_ms);
        if (dev < static_cast<int>(ks->blocks_per_sm.size()) && !ks->blocks_per_sm[dev].empty()) {
            std::copy_n(ks->blocks_per_sm[dev].begin(), n, pc->bps);
            known = std::all_of(pc->bps, pc->bps + n, [](int b) { return b >= 0; });
        }
    }
    cudaDeviceGetAttribute(&pc->sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&pc->max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    for (int c = 0; c < LPAICI_NUM_TILE_CONFIGS; c++) {
        if (!known && c < n) pc->bps[c] = cached_bps(ks, dev, c, pc->max_smem);
        if (pc->bps[c] <= 0)
            pc->tile_ms[c] = 0.0f;
        else if (!pc->tuned)
            pc->tile_ms[c] = estimated_tile_ms(ks, c, pc->bps[c]);
    }
    return true;
}

static constexpr int kMixes[][2] = LPAICI_TILE_MIXES;

// by_rows: the images are one size and a mix's big tiles are whole tile rows of every image.
static TilePlan choose_plan(const lpaici_kernelset *ks, const int *widths, const int *rows, int n, bool by_rows) {
    TilePlan plan;
    PlanCosts pc;
    if (!plan_costs(ks, &pc)) return TilePlan::one(default_config(ks));
    if (pc.forced) return TilePlan::one(pc.forced_config);
    double best_ms = -1.0;
    for (int c = 0; c < LPAICI_NUM_TILE_CONFIGS; c++) {
        const float tile_ms = pc.tile_ms[c];
        const int bps = pc.bps[c];
        if (!(tile_ms > 0.0f)) continue;
        long tiles = 0;
        for (int i = 0; i < n; i++) tiles += tiles_of(c, widths[i], rows[i]);
        const long slots = static_cast<long>(pc.sms) * bps;
        // a lone CTA of a configuration that two fit on an SM takes 1.5 tile times, not 2 (97 x 64 as 28
        // tiles of 16 x 16: 36.9 us against 24 us for one more tile per SM at full occupancy)
        const double waves = tiles <= pc.sms ? 0.5 * (1 + bps) / bps : static_cast<double>((tiles + slots - 1) / slots);
        const double est = tile_ms * bps * waves;
        if (best_ms < 0.0 || est < best_ms) {
            plan = TilePlan::one(c);
            best_ms = est;
        }
    }
    if (best_ms < 0.0) return TilePlan::one(default_config(ks));
    // one image of a few tiles: clusters, as long as they all run at once.  The autotuner times no clusters: of a tuned
    // set they are taken to be off their estimates as the one configuration of the same tile is (33 x 20 and 97 x 64 take
    // 2.4 and 2.3 times as long without, 200 x 150 1.3 times).
    if (by_rows && n == 1) {
        for (int c = 0; c < LPAICI_NUM_CLUSTERS; c++) {
            int tw = 1, th = 1, ctas = 1, groups = 1;
            size_t smem = 0;
            cluster_config(c, ks->radius, ks->layout.total_words, ks->D * ks->S, &tw, &th, &ctas, &groups, &smem);
            const long tiles = static_cast<long>((widths[0] + tw - 1) / tw) * ((rows[0] + th - 1) / th);
            const long slots = ctas == 1 ? pc.sms : (pc.sms - 4 - 3 * ctas) / ctas;  // a cluster's CTAs run in one GPC
            double est = estimated_ms(ks, kClusterCost[c], groups);
            const int like = tw == 16 ? 6 : 5;
            if (pc.tuned && pc.tile_ms[like] > 0.0f) est *= pc.tile_ms[like] / estimated_tile_ms(ks, like, pc.bps[like]);
            if (tiles <= slots && smem <= static_cast<size_t>(pc.max_smem) && est < best_ms) {
                best_ms = est;
                plan = TilePlan::clusters(c);
            }
        }
    }
    // a mix: whole waves of big tiles, or one wave fewer, the rest in small ones
    for (const auto &mix : kMixes) {
        const int a = mix[0], b = mix[1];
        if (!(pc.tile_ms[a] > 0.0f) || !(pc.tile_ms[b] > 0.0f)) continue;
        int aw = 1, ah = 1, bw = 1, bh = 1;
        config_tile(a, &aw, &ah);
        config_tile(b, &bw, &bh);
        long whole = 0, all = 0;  // whole big tiles; small tiles if everything were cut small
        for (int i = 0; i < n; i++) {
            whole += static_cast<long>(widths[i] / aw) * (rows[i] / ah);
            all += static_cast<long>((widths[i] + bw - 1) / bw) * ((rows[i] + bh - 1) / bh);
        }
        const long per = static_cast<long>(aw / bw) * (ah / bh);
        const long row = by_rows ? static_cast<long>(widths[0] / aw) * n : 1;  // big tiles of one tile row
        auto consider = [&](long rows_or_tiles) {
            const long big = rows_or_tiles * row;
            const long small = all - big * per;
            if (big <= 0 || small <= 0) return;
            const double est = mixed_makespan(big, pc.tile_ms[a], small, pc.tile_ms[b], pc.sms);
            if (est < best_ms) {
                best_ms = est;
                plan = by_rows ? TilePlan::mix_rows(a, b, static_cast<int>(rows_or_tiles)) : TilePlan::mix_tiles(a, b, big);
            }
        };
        if (row <= 0 || whole <= 0) continue;
        const long full = whole / row, w0 = whole / pc.sms;
        for (long r : {full, std::min(full, w0 * pc.sms / row), std::min(full, (w0 - 1) * pc.sms / row)})
            consider(r);
    }
    return plan;
}

TilePlan plan_for(const lpaici_kernelset *ks, int width, int rows, int n) {
    if (n == 1) return choose_plan(ks, &width, &rows, 1, true);
    const std::vector<int> w(n, width), h(n, rows);
    return choose_plan(ks, w.data(), h.data(), n, true);
}

TilePlan plan_for_images(const lpaici_kernelset *ks, const int *widths, const int *rows, int n) {
    return choose_plan(ks, widths, rows, n, false);
}

static int check_params(float sigma_or_one, float gamma) {
    if (!(sigma_or_one > 0.0f) || !std::isfinite(sigma_or_one))
        return set_error(LPAICI_ERR_INVALID_ARG, "sigma needs a positive number, got %g", sigma_or_one);
    if (!(gamma > 0.0f) || !std::isfinite(gamma))
        return set_error(LPAICI_ERR_INVALID_ARG, "gamma needs a positive number, got %g", gamma);
    return LPAICI_OK;
}

// Checks a forward call and fills its launch arguments.
static int forward_args(const lpaici_kernelset *ks, const float *d_in, int in_pitch, int width, int in_height,
                        int row_begin, int row_count, float *d_out, int out_pitch, const float *host_var, float sigma,
                        float gamma, uint8_t *d_smap, int step, ImageArgs *args, KernelTables *tables) {
    if (!ks || !d_in || !d_out) return set_error(LPAICI_ERR_INVALID_ARG, "forward: null kernel set or image pointer");
    if (width <= 0 || in_height <= 0 || row_count <= 0)
        return set_error(LPAICI_ERR_INVALID_ARG, "forward: non-positive size %d x %d", width, row_count);
    const long row_floats = static_cast<long>(width - 1) * step + 1;
    if (in_pitch < row_floats || out_pitch < row_floats)
        return set_error(LPAICI_ERR_INVALID_ARG, "forward: pitch smaller than width");
    if (row_begin < 0 || row_begin + row_count > in_height)
        return set_error(LPAICI_ERR_INVALID_ARG, "forward: output rows [%d, %d) outside the %d input rows", row_begin,
                         row_begin + row_count, in_height);
    int rc = check_params(host_var ? 1.0f : sigma, gamma);
    if (rc != LPAICI_OK) return rc;
    if (host_var)
        for (int k = 0; k < ks->D * ks->S; k++)
            if (!(host_var[k] >= 0.0f))
                return set_error(LPAICI_ERR_INVALID_ARG, "forward: variance %d is %g", k, host_var[k]);
    const int *blob = nullptr;
    rc = device_blob(ks, &blob);
    if (rc != LPAICI_OK) return rc;
    ImageArgs &img = *args;
    img = ImageArgs{};
    img.in = d_in;
    img.out = d_out;
    img.smap = d_smap;
    img.W = width;
    img.in_h = in_height;
    img.in_pitch = in_pitch;
    img.out_pitch = out_pitch;
    img.row_begin = row_begin;
    img.rows_out = row_count;
    img.step = step;
    fill_tables(ks, host_var, sigma, gamma, tables);
    tables->blob = blob;
    return LPAICI_OK;
}

// Shared body of the forward entry points.
static int forward_common(const lpaici_kernelset *ks, const float *d_in, int in_pitch, int width, int in_height,
                          int row_begin, int row_count, float *d_out, int out_pitch, const float *host_var,
                          float sigma, float gamma, uint8_t *d_smap, cudaStream_t stream,
                          const TilePlan *plan = nullptr, bool fused = false) {
    ImageArgs img{};
    KernelTables tab;
    const int rc = forward_args(ks, d_in, in_pitch, width, in_height, row_begin, row_count, d_out, out_pitch, host_var,
                                sigma, gamma, d_smap, 1, &img, &tab);
    if (rc != LPAICI_OK) return rc;
    return launch_forward(img, tab, plan ? *plan : plan_for(ks, width, row_count), stream, fused);
}

// Every channel of an interleaved image (pixel (x, y), channel c at row y, float x * channels + c) as
// its own image, in place with element stride `channels`: one launch over all of them.
static int forward_channels(const lpaici_kernelset *ks, const float *d_in, int in_pitch, float *d_out, int out_pitch,
                            int width, int height, int channels, const float *host_var, float sigma, float gamma,
                            cudaStream_t stream) {
    if (channels <= 0 || channels > kMaxMultiImages)
        return set_error(LPAICI_ERR_INVALID_ARG, "channels must be 1 .. %d, got %d", kMaxMultiImages, channels);
    ImageArgs img{};
    KernelTables tab;
    const int rc = forward_args(ks, d_in, in_pitch, width, height, 0, height, d_out, out_pitch, host_var, sigma, gamma,
                                nullptr, channels, &img, &tab);
    if (rc != LPAICI_OK) return rc;
    if (channels == 1) return launch_forward(img, tab, plan_for(ks, width, height), stream);
    MultiImages mi{};
    for (int c = 0; c < channels; c++) {
        mi.in[c] = d_in + c;
        mi.out[c] = d_out + c;
    }
    return launch_forward_multi(img, tab, mi, channels, plan_for(ks, width, height, channels), stream);
}

}  // namespace lpaici

extern "C" {

int lpaici_forward(const lpaici_kernelset *ks, const float *d_noisy, int noisy_pitch, float *d_denoised,
                   int out_pitch, int width, int height, float sigma, float gamma, uint8_t *d_scale_map,
                   lpaici_stream_t stream) {
    return forward_common(ks, d_noisy, noisy_pitch, width, height, 0, height, d_denoised, out_pitch, nullptr, sigma,
                          gamma, d_scale_map, reinterpret_cast<cudaStream_t>(stream));
}

int lpaici_forward_ffma(const lpaici_kernelset *ks, const float *d_noisy, int noisy_pitch, float *d_denoised,
                        int out_pitch, int width, int height, float sigma, float gamma, uint8_t *d_scale_map,
                        lpaici_stream_t stream) {
    return forward_common(ks, d_noisy, noisy_pitch, width, height, 0, height, d_denoised, out_pitch, nullptr, sigma,
                          gamma, d_scale_map, reinterpret_cast<cudaStream_t>(stream), nullptr, true);
}

int lpaici_forward_var(const lpaici_kernelset *ks, const float *d_noisy, int noisy_pitch, float *d_denoised,
                       int out_pitch, int width, int height, const float *host_var, float gamma,
                       uint8_t *d_scale_map, lpaici_stream_t stream) {
    if (!host_var) return set_error(LPAICI_ERR_INVALID_ARG, "lpaici_forward_var: null variances");
    return forward_common(ks, d_noisy, noisy_pitch, width, height, 0, height, d_denoised, out_pitch, host_var, 1.0f,
                          gamma, d_scale_map, reinterpret_cast<cudaStream_t>(stream));
}

int lpaici_forward_rows(const lpaici_kernelset *ks, const float *d_in, int in_pitch, int width, int in_height,
                        int row_begin, int row_count, float *d_out, int out_pitch, float sigma, float gamma,
                        uint8_t *d_scale_map, lpaici_stream_t stream) {
    return forward_common(ks, d_in, in_pitch, width, in_height, row_begin, row_count, d_out, out_pitch, nullptr, sigma,
                          gamma, d_scale_map, reinterpret_cast<cudaStream_t>(stream));
}

int lpaici_forward_channels(const lpaici_kernelset *ks, const float *d_noisy, int noisy_pitch, float *d_denoised,
                            int out_pitch, int width, int height, int channels, float sigma, float gamma,
                            lpaici_stream_t stream) {
    return forward_channels(ks, d_noisy, noisy_pitch, d_denoised, out_pitch, width, height, channels, nullptr, sigma,
                            gamma, reinterpret_cast<cudaStream_t>(stream));
}

int lpaici_num_tile_configs(void) { return LPAICI_NUM_TILE_CONFIGS; }

int lpaici_tile_config_desc(int index, int *tile_w, int *tile_h, int *threads, int *pixels_per_thread) {
#define LPAICI_DESC_CASE(idx, WX, WY, Q, DS)              \
    case idx:                                             \
        if (tile_w) *tile_w = (WX) * 4 * (Q);             \
        if (tile_h) *tile_h = (WY) * 16;                  \
        if (threads) *threads = 32 * (WX) * (WY) * (DS);  \
        if (pixels_per_thread) *pixels_per_thread = 2 * (Q) / (DS); \
        return LPAICI_OK;
    switch (index) {
        LPAICI_TILE_CONFIGS(LPAICI_DESC_CASE)
        default: return set_error(LPAICI_ERR_INVALID_ARG, "tile config %d out of range", index);
    }
#undef LPAICI_DESC_CASE
}

// ---- host-pointer engines ---------------------------------------------------------------------

namespace {
// Device buffers and the copy/compute pipeline of lpaici_denoise_host, per host thread and device.
constexpr int kMaxBands = 64;
// Bands in flight: one of fewer tiles than SMs would otherwise hold back the next one on its stream for a tile's time.
constexpr int kBandStreams = 8;
struct HostBuffers {
    int dev = -1;
    float *in = nullptr, *out = nullptr;
    size_t cap = 0;
    cudaStream_t s_in = nullptr, s_out = nullptr, s_comp[kBandStreams] = {};
    cudaEvent_t ev_start = nullptr, ev_done = nullptr, ev_in[kMaxBands] = {}, ev_comp[kMaxBands] = {};
    ~HostBuffers() { release(); }
    void release() {
        if (dev >= 0) {
            int cur = -1;
            cudaGetDevice(&cur);
            cudaSetDevice(dev);
            cudaFree(in);
            cudaFree(out);
            for (cudaStream_t st : {s_in, s_out})
                if (st) cudaStreamDestroy(st);
            for (cudaStream_t st : s_comp)
                if (st) cudaStreamDestroy(st);
            for (cudaEvent_t ev : {ev_start, ev_done})
                if (ev) cudaEventDestroy(ev);
            for (int i = 0; i < kMaxBands; i++) {
                if (ev_in[i]) cudaEventDestroy(ev_in[i]);
                if (ev_comp[i]) cudaEventDestroy(ev_comp[i]);
                ev_in[i] = ev_comp[i] = nullptr;
            }
            if (cur >= 0) cudaSetDevice(cur);
        }
        in = out = nullptr;
        s_in = s_out = nullptr;
        for (cudaStream_t &st : s_comp) st = nullptr;
        ev_start = ev_done = nullptr;
        cap = 0;
        dev = -1;
    }
    cudaError_t make_pipeline() {
        cudaError_t e = cudaSuccess;
        for (cudaStream_t *st : {&s_in, &s_out})
            if (e == cudaSuccess) e = cudaStreamCreateWithFlags(st, cudaStreamNonBlocking);
        for (cudaStream_t &st : s_comp)
            if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
        for (cudaEvent_t *ev : {&ev_start, &ev_done})
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
        for (int i = 0; i < kMaxBands && e == cudaSuccess; i++) {
            e = cudaEventCreateWithFlags(&ev_in[i], cudaEventDisableTiming);
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev_comp[i], cudaEventDisableTiming);
        }
        return e;
    }
};
thread_local HostBuffers t_bufs;
}  // namespace

int lpaici_denoise_host(const lpaici_kernelset *ks, const float *host_noisy, float *host_denoised, int width,
                        int height, float sigma, float gamma, lpaici_stream_t stream_) {
    if (!ks || !host_noisy || !host_denoised || width <= 0 || height <= 0)
        return set_error(LPAICI_ERR_INVALID_ARG, "lpaici_denoise_host: bad argument");
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_error(e, "cudaGetDevice");
    int rc = check_params(sigma, gamma);
    if (rc != LPAICI_OK) return rc;
    const size_t n = static_cast<size_t>(width) * height;
    if (t_bufs.dev != dev || t_bufs.cap < n) {
        t_bufs.release();
        t_bufs.dev = dev;
        e = cudaMalloc(&t_bufs.in, n * sizeof(float));
        if (e == cudaSuccess) e = cudaMalloc(&t_bufs.out, n * sizeof(float));
        if (e == cudaSuccess) e = t_bufs.make_pipeline();
        if (e != cudaSuccess) {
            t_bufs.release();
            return cuda_error(e, "host-pointer buffers");
        }
        t_bufs.cap = n;
    }
    // Row bands, pipelined: the upload of the rows band b needs (its rows + R below) on s_in, its
    // forward on one of the compute streams (the next bands' CTAs fill the SMs that this band leaves
    // idle), its download on s_out.  With pinned host buffers the copies overlap the kernels.
    // The bands' launches overlap, so the GPU sees one stream of tiles: they take the whole
    // image's plan, big tiles in the upper bands and the plan's small ones in the lower (2048^2: 2.45 ms with
    // one configuration in ten bands on two streams, 1.95 ms so).
    // Bands hide the copies behind the kernels at about 6 us of host calls each: as many as make (copies / bands)
    // + 6 us * bands least, six at most.  Six bands or more: the first is one tile row, so that the first forward
    // starts after a short upload, the last one at most two rows of small tiles, so that the download after the
    // last forward is short.  us from pinned arrays, five to eleven bands at every size and so: 8 directions of one
    // scale 200x150 58 and 37, 512^2 95 and 64; 16x7 symmetric set 256^2 132 and 73, 512^2 252 and 196; the same from
    // about 1.35 Mpx on.  An image that clusters sweep is one band too (under 150 KB, one wave of tiles).
    const TilePlan plan = plan_for(ks, width, height);
    const bool mixed = plan.kind == TilePlan::kMix;
    const int low_config = mixed ? plan.rest : plan.config;
    int big_h = height, low_h = height;
    if (plan.kind != TilePlan::kCluster) {
        lpaici_tile_config_desc(plan.config, nullptr, &big_h, nullptr, nullptr);
        lpaici_tile_config_desc(low_config, nullptr, &low_h, nullptr, nullptr);
    }
    const int R = ks->radius;
    // band i covers rows [edge[i], edge[i + 1]); bands from `low` on use low_config
    int edge[kMaxBands + 1];
    int nb = 0, low = 0;
    edge[0] = 0;
    constexpr int kMostBands = 6;
    const double copies_us = 2.0 * sizeof(float) * static_cast<double>(n) / 50e3;  // PCIe 5 x16, about 50 GB/s
    const int bands = std::clamp(static_cast<int>(std::sqrt(copies_us / 6.0)), 1, kMostBands);
    if (plan.kind == TilePlan::kCluster || bands == 1) {
        edge[++nb] = height;
        low = nb;
    } else {
        const bool thin_ends = bands == kMostBands;
        const int rows = (height + bands - 1) / bands;
        const int upper = mixed ? std::min(plan.big_rows * big_h, height) : 0;
        auto cut = [&](int to, int tile, int rows) {  // bands of about `rows` rows, whole tile rows, up to row `to`
            int band = std::max(1, (rows + tile - 1) / tile) * tile;
            while (edge[nb] < to && nb < kMaxBands - 8) {
                edge[nb + 1] = std::min(to, edge[nb] + band);
                nb++;
            }
            if (edge[nb] < to) edge[++nb] = to;
        };
        if (upper > 0) {
            if (thin_ends) cut(big_h, big_h, big_h);
            cut(upper, big_h, rows);
        }
        low = nb;
        if (thin_ends) {
            if (nb == 0) cut(low_h, low_h, low_h);
            const int last = std::max(edge[nb], height - 2 * low_h - (height - edge[nb]) % low_h);
            cut(last, low_h, rows);
            cut(height, height, height);
        } else {
            cut(height, low_h, rows);
        }
        if (!mixed) low = 0;
    }
    HostBuffers &b = t_bufs;
    e = cudaEventRecord(b.ev_start, stream);
    for (cudaStream_t st : {b.s_in, b.s_out})
        if (e == cudaSuccess) e = cudaStreamWaitEvent(st, b.ev_start, 0);
    if (e != cudaSuccess) return cuda_error(e, "lpaici_denoise_host: stream order");
    int copied = 0;  // input rows [0, copied) uploaded
    for (int i = 0; i < nb && rc == LPAICI_OK; i++) {
        const int r0 = edge[i], r1 = edge[i + 1], need = std::min(height, r1 + R);
        if (need > copied) {
            e = cudaMemcpyAsync(b.in + static_cast<size_t>(copied) * width, host_noisy + static_cast<size_t>(copied) * width,
                                sizeof(float) * width * static_cast<size_t>(need - copied), cudaMemcpyHostToDevice, b.s_in);
            copied = need;
        }
        if (e == cudaSuccess) e = cudaEventRecord(b.ev_in[i], b.s_in);
        cudaStream_t sc = b.s_comp[i % kBandStreams];
        if (e == cudaSuccess) e = cudaStreamWaitEvent(sc, b.ev_in[i], 0);
        if (e != cudaSuccess) {
            rc = cuda_error(e, "lpaici_denoise_host: upload");
            break;
        }
        const TilePlan band = nb == 1 ? plan : i < low ? TilePlan::mix_rows(plan.config, plan.rest, (r1 - r0) / big_h)
                                               : TilePlan::one(low_config);
        rc = forward_common(ks, b.in, width, width, height, r0, r1 - r0, b.out + static_cast<size_t>(r0) * width, width,
                            nullptr, sigma, gamma, nullptr, sc, &band);
        if (rc != LPAICI_OK) break;
        e = cudaEventRecord(b.ev_comp[i], sc);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(b.s_out, b.ev_comp[i], 0);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(host_denoised + static_cast<size_t>(r0) * width, b.out + static_cast<size_t>(r0) * width,
                                sizeof(float) * width * static_cast<size_t>(r1 - r0), cudaMemcpyDeviceToHost, b.s_out);
        if (e != cudaSuccess) rc = cuda_error(e, "lpaici_denoise_host: download");
    }
    // every band's download waited for its forward, every forward for its upload: s_out covers all
    e = cudaEventRecord(b.ev_done, b.s_out);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(stream, b.ev_done, 0);
    const cudaError_t es = cudaStreamSynchronize(b.s_out);
    if (rc != LPAICI_OK) return rc;
    if (e != cudaSuccess) return cuda_error(e, "lpaici_denoise_host: join");
    if (es != cudaSuccess) return cuda_error(es, "cudaStreamSynchronize");
    return LPAICI_OK;
}

int lpaici_release_host_buffers(void) {
    t_bufs.release();
    return LPAICI_OK;
}

int lpaici_anisotropic_gpu_fused(float *host_img_noisy, float *host_img_denoised, int width, int height, int channels,
                                 float *host_global_weights_buffer, int num_dirs, int num_scales,
                                 float *host_kernel_weights, int host_kernel_weights_size, int *host_offsets,
                                 int *host_rows, int *host_cols, float *host_kernel_variances, float ici_gamma,
                                 double *seconds) {
    (void)host_global_weights_buffer;
    if (channels <= 0 || channels > 64)
        return set_error(LPAICI_ERR_INVALID_ARG, "channels must be 1 .. 64, got %d", channels);
    if (!host_img_noisy || !host_img_denoised || !host_kernel_weights || !host_offsets || !host_rows || !host_cols ||
        !host_kernel_variances || width <= 0 || height <= 0)
        return set_error(LPAICI_ERR_INVALID_ARG, "lpaici_anisotropic_gpu_fused: bad argument");
    const long nk = static_cast<long>(num_dirs) * num_scales;
    for (long k = 0; k < nk; k++)
        if (host_offsets[k] < 0 || static_cast<long>(host_offsets[k]) + static_cast<long>(host_rows[k]) * host_cols[k] >
                                       host_kernel_weights_size)
            return set_error(LPAICI_ERR_KERNEL_FORMAT, "kernel %ld lies outside the %d weights", k,
                             host_kernel_weights_size);
    lpaici_kernelset *ks = nullptr;
    int rc = lpaici_kernelset_create(host_kernel_weights, host_offsets, host_rows, host_cols, num_dirs, num_scales, &ks);
    if (rc != LPAICI_OK) return rc;
    const size_t n = static_cast<size_t>(width) * height * channels;
    float *d_in = nullptr, *d_out = nullptr;
    cudaError_t e = cudaMalloc(&d_in, n * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&d_out, n * sizeof(float));
    if (e == cudaSuccess) e = cudaMemcpy(d_in, host_img_noisy, n * sizeof(float), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        rc = cuda_error(e, "lpaici_anisotropic_gpu_fused setup");
    } else {
        cudaDeviceSynchronize();
        const auto t0 = std::chrono::steady_clock::now();  // the reference's window starts here (:1216)
        rc = forward_channels(ks, d_in, width * channels, d_out, width * channels, width, height, channels,
                              host_kernel_variances, 1.0f, ici_gamma, nullptr);
        if (rc == LPAICI_OK) {
            e = cudaMemcpy(host_img_denoised, d_out, n * sizeof(float), cudaMemcpyDeviceToHost);
            if (e != cudaSuccess) rc = cuda_error(e, "cudaMemcpy(D2H)");
        }
        const auto t1 = std::chrono::steady_clock::now();  // ... and ends after the copy back (:1240)
        if (seconds) *seconds = std::chrono::duration<double>(t1 - t0).count();
    }
    cudaFree(d_in);
    cudaFree(d_out);
    lpaici_kernelset_destroy(ks);
    return rc;
}

}  // extern "C"

// ---- autotuner ----------------------------------------------------------------------------------

namespace {

// Built-in tuning image: a smooth ramp, a stripe texture and blocks, plus hash noise of 0.08.
__global__ void synth_tuning_image(float *img, int W, int H, int pitch) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= W || y >= H) return;
    unsigned h = static_cast<unsigned>(x) * 0x9E3779B1u ^ static_cast<unsigned>(y) * 0x85EBCA77u;
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 12;
    const float u = (h & 0xFFFFFF) * (1.0f / 16777216.0f) - 0.5f;
    const float ramp = 0.3f * x / W + 0.2f * y / H;
    const float stripes = 0.2f * sinf(0.7f * x + 0.4f * y);
    const float block = (((x >> 7) ^ (y >> 7)) & 1) ? 0.3f : 0.0f;
    img[static_cast<size_t>(y) * pitch + x] = ramp + stripes + block + 0.28f * u;
}

}  // namespace

extern "C" int lpaici_autotune(lpaici_kernelset *ks, const float *d_sample, int width, int height, int pitch,
                               float sigma, float gamma, int reps, int *best_config, float *ms_out,
                               lpaici_stream_t stream_) {
    if (!ks || width <= 0 || height <= 0 || (d_sample && pitch < width) || reps <= 0)
        return set_error(LPAICI_ERR_INVALID_ARG, "lpaici_autotune: bad argument");
    int rc = check_params(sigma, gamma);
    if (rc != LPAICI_OK) return rc;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    const size_t n = static_cast<size_t>(width) * height;
    float *in = nullptr, *out = nullptr;
    cudaError_t e = cudaSuccess;
    if (!d_sample) {
        e = cudaMalloc(&in, n * sizeof(float));
        if (e != cudaSuccess) return cuda_error(e, "cudaMalloc(autotune)");
        synth_tuning_image<<<dim3((width + 255) / 256, height), 256, 0, stream>>>(in, width, height, width);
        pitch = width;
    }
    e = cudaMalloc(&out, n * sizeof(float));
    if (e != cudaSuccess) {
        cudaFree(in);
        return cuda_error(e, "cudaMalloc(autotune)");
    }
    const float *src = d_sample ? d_sample : in;
    const int *blob = nullptr;
    rc = device_blob(ks, &blob);
    ImageArgs img{};
    img.in = src;
    img.out = out;
    img.W = width;
    img.in_h = height;
    img.in_pitch = pitch;
    img.out_pitch = width;
    img.rows_out = height;
    KernelTables tab;
    fill_tables(ks, nullptr, sigma, gamma, &tab);
    tab.blob = blob;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    float best_ms = 0.0f;
    int best = -1;
    std::vector<float> config_ms(LPAICI_NUM_TILE_CONFIGS, -1.0f);
    for (int c = 0; rc == LPAICI_OK && c < LPAICI_NUM_TILE_CONFIGS; c++) {
        int crc = launch_forward(img, tab, TilePlan::one(c), stream);  // warm-up
        if (crc != LPAICI_OK) {
            if (ms_out) ms_out[c] = -1.0f;
            if (crc == LPAICI_ERR_UNSUPPORTED) continue;  // this tile does not fit for this kernel set
            rc = crc;
            break;
        }
        cudaEventRecord(e0, stream);
        for (int r = 0; r < reps && crc == LPAICI_OK; r++) crc = launch_forward(img, tab, TilePlan::one(c), stream);
        cudaEventRecord(e1, stream);
        e = cudaEventSynchronize(e1);
        if (e != cudaSuccess) {
            rc = cuda_error(e, "autotune");
            break;
        }
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, e0, e1);
        ms /= reps;
        if (ms_out) ms_out[c] = ms;
        config_ms[c] = ms;
        if (best < 0 || ms < best_ms) {
            best = c;
            best_ms = ms;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(in);
    cudaFree(out);
    if (rc != LPAICI_OK) return rc;
    if (best < 0) return set_error(LPAICI_ERR_UNSUPPORTED, "no tile configuration fits this kernel set");
    if (best_config) *best_config = best;
    rc = lpaici_set_tile_config(ks, best);
    if (rc != LPAICI_OK) return rc;
    // per-tile times, for picking the plan of other image sizes (plan_for)
    int dev = 0, sms = 0, max_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    std::vector<float> tile_ms(LPAICI_NUM_TILE_CONFIGS, -1.0f);
    for (int c = 0; c < LPAICI_NUM_TILE_CONFIGS; c++) {
        const int bps = cached_bps(ks, dev, c, max_optin);
        if (!(config_ms[c] > 0.0f) || bps <= 0) continue;
        const long slots = static_cast<long>(sms) * bps;
        tile_ms[c] = config_ms[c] / (bps * static_cast<float>((tiles_of(c, width, height) + slots - 1) / slots));
    }
    std::lock_guard<std::mutex> lock(ks->mu);
    if (static_cast<int>(ks->tuned_tile_ms.size()) <= dev) ks->tuned_tile_ms.resize(dev + 1);
    ks->tuned_tile_ms[dev] = tile_ms;
    return LPAICI_OK;
}

extern "C" int lpaici_set_tile_config(lpaici_kernelset *ks, int config) {
    if (!ks || config < -1 || config >= LPAICI_NUM_TILE_CONFIGS)
        return set_error(LPAICI_ERR_INVALID_ARG, "lpaici_set_tile_config: bad argument");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_error(e, "cudaGetDevice");
    std::lock_guard<std::mutex> lock(ks->mu);
    if (static_cast<int>(ks->tuned_config.size()) <= dev) {
        ks->dev_blob.resize(dev + 1, nullptr);
        ks->tuned_config.resize(dev + 1, -1);
    }
    ks->tuned_config[dev] = config;
    if (dev < static_cast<int>(ks->tuned_tile_ms.size())) ks->tuned_tile_ms[dev].clear();  // forced
    return LPAICI_OK;
}
