// batched.cu -- many images of uneven sizes, sigmas and gammas, planned together.
//
// The plan (plan_for_images) takes one tile configuration, or a mix: big tiles where whole ones fit, in
// whole waves, and small tiles for the rest, as a second launch that starts while the first one's last
// tiles run (programmatic dependent launch; the two write different tiles).  Each launch has one CTA per
// item {image, x0, y0}, full tiles of the largest images first and partial edge tiles last: the hardware
// dispatches blocks in index order as SMs free up, so the queue order is the execution order without a
// persistent loop (a persistent grid pulling items from an atomic counter ran 2-2.5 % slower).  Ten mixed
// images of 4.9 Mpx in all: one configuration 2.51 ms, both tiles in one kernel 2.19, two launches 2.12.
// No CTA waits for another.  With use_graph the launches are captured once into a CUDA graph and replayed
// by lpaici_batch_run.  A plan of one image launches the single-image kernel instead (image and tables as
// launch parameters): there are no small-image tails to fill, and the item's decode would cost a little
// per CTA.  A plan of up to kMaxMultiImages images of one size, pitch, sigma and gamma launches that
// kernel with a grid layer per image (lpaici_forward_multi_kernel).
// No reference counterpart: the reference denoises one image per process
// (src/v4_1_lpa_ici_2D_sparse_shared.cu:365-530).
#include <algorithm>
#include <cstring>
#include <vector>

#include "configs.h"
#include "tile_core.cuh"

namespace lpaici {

// Per-image descriptor in device memory.
struct BatchImage {
    const float *in;
    float *out;       // null: no estimate (the adjoint's selection pass)
    uint8_t *smap;
    float *rden;      // optional 1/den map (the adjoint's selection pass)
    const float *g;   // optional cotangent: rden is g / den
    int W, H, in_pitch, out_pitch, g_pitch;
    int tab_offset;  // float index of var[nk] (thr[nk] follows) in the plan's table array
};

struct BatchArgs {
    const BatchImage *images;
    const float *tables;    // per image var[nk], thr[nk]
    const int4 *items;      // (image, x0, y0, unused)
    int rest_follows;       // a launch over the plan's small tiles follows
    int D, S, R;
    const int *blob;
    int blob_words, mask_word, stream_word;
    float neg_zero;  // -0.0f, read at run time (see prod2 in tile_core.cuh)
    // every image of the plan has the same sigma and gamma (always so for one image): its var and thr
    // travel here, as in the single-image launch, instead of being read per CTA from `tables`
    int shared_tables;
    float var[kMaxKernels];
    float thr[kMaxKernels];
};

// One tile: stages the kernel set, the image's tables and the tile, and sweeps it.
template <int WX, int WY, int Q, int DS>
__device__ __forceinline__ void batched_tile(int *smem, const BatchArgs &a, const ImageArgs &img, int image, int x0, int y0) {
    const int nk = a.D * a.S;
    const SweepCta<WX, WY, Q, DS> cta(smem, a.blob_words, nk, a.R);
    load_tile(cta.tile, img, x0, y0, cta.g);
    stage_blob<Q>(cta.blob, a.blob, a.blob_words, a.mask_word, a.stream_word, cta.g.pitch2);
    if (a.shared_tables) {
        stage_tables(cta.tab, a.var, a.thr, nk);
    } else {
        const float *t = a.tables + a.images[image].tab_offset;
        stage_tables(cta.tab, t, t + nk, nk);
    }
    tile_wait();
    __syncthreads();
    sweep_tile<WX, WY, Q, DS, false>(img, x0, y0, a.D, a.S, cta.g, cta.blob, cta.tab, cta.tile, cta.xch, a.neg_zero);
}

// The CTA's image arguments live in shared memory: in registers they would stay live across the whole sweep,
// beside the run loop's (the single-image kernel reads them from its parameters).
__device__ __forceinline__ void batched_image(const BatchArgs &a, int image, ImageArgs *out) {
    if (threadIdx.x == 0) {
        const BatchImage bi = a.images[image];
        ImageArgs img{};
        img.in = bi.in;
        img.out = bi.out;
        img.smap = bi.smap;
        img.rden = bi.rden;
        img.g = bi.g;
        img.g_pitch = bi.g_pitch;
        img.W = bi.W;
        img.in_h = bi.H;
        img.in_pitch = bi.in_pitch;
        img.out_pitch = bi.out_pitch;
        img.row_begin = 0;
        img.rows_out = bi.H;
        *out = img;
    }
    __syncthreads();
}

// One CTA per queue item, dispatched in queue order.
template <int WX, int WY, int Q, int DS>
__global__ void __launch_bounds__(32 * WX * WY * DS, 1)
    lpaici_batched_kernel(const __grid_constant__ BatchArgs a) {
    extern __shared__ __align__(16) int smem[];
    __shared__ __align__(16) unsigned char s_img[sizeof(ImageArgs)];
    ImageArgs &img = *reinterpret_cast<ImageArgs *>(s_img);
    // a plan's big tiles let the launch over its small ones start as they end; the last small tile waits for the
    // big ones, so that what follows in the stream follows both (lpaici_forward_rest_kernel)
    if (a.rest_follows) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int4 item = __ldg(a.items + blockIdx.x);
    batched_image(a, item.x, &img);
    batched_tile<WX, WY, Q, DS>(smem, a, img, item.x, item.y, item.z);
    if (blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
}

namespace {

struct KernelInfo {
    const void *fn;
    int tile_w, tile_h, threads;
    size_t smem;
};

template <int WX, int WY, int Q, int DS>
int batched_info(const KernelTables &tab, KernelInfo *info) {
    using Shape = TileShape<WX, WY, Q, DS>;
    info->fn = reinterpret_cast<const void *>(lpaici_batched_kernel<WX, WY, Q, DS>);
    info->tile_w = Shape::kTileW;
    info->tile_h = Shape::kTileH;
    info->threads = Shape::kThreads;
    info->smem = sweep_smem<Shape, Q>(tab.blob_words, tab.D * tab.S, tab.R);
    return LPAICI_OK;
}

int get_info(int config, const KernelTables &tab, KernelInfo *info) {
#define LPAICI_BATCH_CASE(idx, WX, WY, Q, DS) \
    case idx: return batched_info<WX, WY, Q, DS>(tab, info);
    switch (config) {
        LPAICI_TILE_CONFIGS(LPAICI_BATCH_CASE)
        default: return set_error(LPAICI_ERR_INVALID_ARG, "tile config %d out of range", config);
    }
#undef LPAICI_BATCH_CASE
}

}  // namespace
}  // namespace lpaici

using namespace lpaici;

struct lpaici_batch {
    int device = -1;
    KernelInfo info{}, rest{};  // rest: of a plan's small tiles
    BatchArgs args{};
    int grid = 0, rest_grid = 0;
    void *dev_mem = nullptr;  // images | tables | items
    bool use_graph = false;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    // a plan of one image runs the single-image kernel (image and tables as launch parameters, no queue
    // to decode): one image has no small-image tails for the queue to fill
    bool single = false;
    // a plan of 2 .. kMaxMultiImages images of one size, pitch, sigma and gamma runs the single-image kernel
    // once with a grid layer per image (lpaici_forward_multi_kernel): no queue to decode, and each image's
    // CTAs fill the SMs the previous image's last wave leaves idle
    bool multi = false;
    int n_multi = 0;
    MultiImages mi{};
    ImageArgs img{};
    KernelTables tab{};
    TilePlan plan;
};

namespace lpaici {

int batch_plan_enqueue(lpaici_batch *b, cudaStream_t stream) {
    if (b->single) return launch_forward(b->img, b->tab, b->plan, stream);
    if (b->multi) return launch_forward_multi(b->img, b->tab, b->mi, b->n_multi, b->plan, stream);
    void *params[] = {&b->args};
    cudaError_t e = b->grid > 0
                        ? cudaLaunchKernel(b->info.fn, dim3(b->grid), dim3(b->info.threads), params, b->info.smem, stream)
                        : cudaSuccess;
    if (e != cudaSuccess) return cuda_error(e, "batched launch");
    if (b->rest_grid > 0) {
        BatchArgs rest = b->args;
        rest.items += b->grid;
        rest.rest_follows = 0;
        void *rest_params[] = {&rest};
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(b->rest_grid);
        cfg.blockDim = dim3(b->rest.threads);
        cfg.dynamicSmemBytes = b->rest.smem;
        cfg.stream = stream;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelExC(&cfg, b->rest.fn, rest_params);
        if (e != cudaSuccess) return cuda_error(e, "batched launch (small tiles)");
    }
    return LPAICI_OK;
}

void batch_plan_free(lpaici_batch *b) {
    if (!b) return;
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    if (b->dev_mem) cudaFree(b->dev_mem);
    delete b;
}

// The tile configurations of a plan that is not a cluster's, and whether they fit.
static int check_tiles(lpaici_batch *b, const KernelTables &tab) {
    int rc = get_info(b->plan.config, tab, &b->info);
    if (rc == LPAICI_OK && b->plan.kind == TilePlan::kMix) rc = get_info(b->plan.rest, tab, &b->rest);
    if (rc != LPAICI_OK) return rc;
    int max_optin = 0;
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, b->device);
    if (b->info.smem + kStaticShared > static_cast<size_t>(max_optin))
        return set_error(LPAICI_ERR_UNSUPPORTED, "batched tile needs %zu B of shared memory, device allows %d",
                         b->info.smem + kStaticShared, max_optin);
    return LPAICI_OK;
}

// The queue of a plan over images of several sizes, sigmas or gammas: descriptors, tables and ordered items in
// device memory.
static int build_queue(lpaici_batch *b, const lpaici_kernelset *ks, const BatchSpec *specs, int n, const KernelTables &tab) {
    const int nk = ks->D * ks->S;
    std::vector<BatchImage> imgs(n);
    std::vector<float> tables(static_cast<size_t>(n) * 2 * nk);
    struct Item {
        int image, x, y;
        long key;
    };
    std::vector<Item> items, small;
    auto push = [&](std::vector<Item> &to, int i, int x, int y, int tw, int th) {
        const int w = std::min(tw, specs[i].width - x), h = std::min(th, specs[i].height - y);
        // full tiles first, then by image size (largest first), then raster order
        const long area = static_cast<long>(specs[i].width) * specs[i].height;
        if (w > 0 && h > 0) to.push_back({i, x, y, static_cast<long>(w) * h * (1L << 40) + area});
    };
    for (int i = 0; i < n; i++) {
        const BatchSpec &im = specs[i];
        KernelTables t;
        fill_tables(ks, nullptr, im.sigma, im.gamma, &t);
        std::memcpy(&tables[static_cast<size_t>(i) * 2 * nk], t.var, sizeof(float) * nk);
        std::memcpy(&tables[static_cast<size_t>(i) * 2 * nk + nk], t.thr, sizeof(float) * nk);
        imgs[i] = BatchImage{im.noisy, im.out, im.smap, im.rden, im.g, im.width, im.height, im.noisy_pitch, im.out_pitch,
                             im.g_pitch, i * 2 * nk};
        for (int y = 0; y < im.height; y += b->info.tile_h)
            for (int x = 0; x < im.width; x += b->info.tile_w) push(items, i, x, y, b->info.tile_w, b->info.tile_h);
    }
    const auto by_key = [](const Item &p, const Item &q) { return p.key > q.key; };
    std::stable_sort(items.begin(), items.end(), by_key);
    if (b->plan.kind == TilePlan::kMix) {  // all tiles past the plan's big ones are cut small
        const size_t big = std::min(items.size(), static_cast<size_t>(b->plan.big_tiles));
        for (size_t j = big; j < items.size(); j++)
            for (int y = 0; y < b->info.tile_h; y += b->rest.tile_h)
                for (int x = 0; x < b->info.tile_w; x += b->rest.tile_w)
                    push(small, items[j].image, items[j].x + x, items[j].y + y, b->rest.tile_w, b->rest.tile_h);
        items.resize(big);
        std::stable_sort(small.begin(), small.end(), by_key);
    }
    std::vector<int4> qitems;
    qitems.reserve(items.size() + small.size());
    for (const Item &it : items) qitems.push_back(make_int4(it.image, it.x, it.y, 0));
    for (const Item &it : small) qitems.push_back(make_int4(it.image, it.x, it.y, 0));

    const size_t img_bytes = sizeof(BatchImage) * n;
    const size_t tab_off = (img_bytes + 255) & ~size_t(255);
    const size_t tab_bytes = sizeof(float) * tables.size();
    const size_t item_off = (tab_off + tab_bytes + 255) & ~size_t(255);
    const size_t item_bytes = sizeof(int4) * qitems.size();
    cudaError_t e = cudaMalloc(&b->dev_mem, item_off + item_bytes);
    if (e != cudaSuccess) return cuda_error(e, "cudaMalloc(batch plan)");
    char *base = static_cast<char *>(b->dev_mem);
    e = cudaMemcpy(base, imgs.data(), img_bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(base + tab_off, tables.data(), tab_bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(base + item_off, qitems.data(), item_bytes, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_error(e, "cudaMemcpy(batch plan)");
    b->args.images = reinterpret_cast<const BatchImage *>(base);
    b->args.tables = reinterpret_cast<const float *>(base + tab_off);
    b->args.items = reinterpret_cast<const int4 *>(base + item_off);
    b->args.D = ks->D;
    b->args.S = ks->S;
    b->args.R = ks->radius;
    b->args.blob = tab.blob;
    b->args.blob_words = tab.blob_words;
    b->args.mask_word = tab.mask_word;
    b->args.stream_word = tab.stream_word;
    b->args.neg_zero = -0.0f;
    bool same = true;
    for (int i = 1; i < n; i++) same = same && specs[i].sigma == specs[0].sigma && specs[i].gamma == specs[0].gamma;
    b->args.shared_tables = same ? 1 : 0;
    if (same) {
        std::memcpy(b->args.var, tables.data(), sizeof(float) * nk);
        std::memcpy(b->args.thr, tables.data() + nk, sizeof(float) * nk);
    }
    b->grid = static_cast<int>(items.size());  // one CTA per queue item
    b->rest_grid = static_cast<int>(small.size());
    b->args.rest_follows = b->rest_grid > 0 ? 1 : 0;

    int per_sm = 0;
    e = allow_shared_memory(b->info.fn, kStaticShared);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, b->info.fn, b->info.threads, b->info.smem);
    if (e != cudaSuccess) return cuda_error(e, "batched occupancy");
    if (per_sm <= 0) return set_error(LPAICI_ERR_UNSUPPORTED, "batched kernel does not fit on an SM");
    if (b->rest_grid > 0) e = allow_shared_memory(b->rest.fn, kStaticShared);
    return e == cudaSuccess ? LPAICI_OK : cuda_error(e, "batched attributes");
}

// The plan of lpaici_batch_create for already validated images (specs); the adjoint's batched
// selection pass uses it with out = null and smap/rden set.
int batch_plan_create(const lpaici_kernelset *ks, const BatchSpec *specs, int n, int config, bool use_graph,
                      cudaStream_t stream, lpaici_batch **out) {
    *out = nullptr;
    if (ks->S > kMaxScales)
        return set_error(LPAICI_ERR_UNSUPPORTED, "%d scales per direction; the kernels support at most %d", ks->S,
                         kMaxScales);
    const int *blob = nullptr;
    int rc = device_blob(ks, &blob);
    if (rc != LPAICI_OK) return rc;

    auto *b = new lpaici_batch();
    cudaGetDevice(&b->device);
    KernelTables tab;
    fill_tables(ks, nullptr, 1.0f, 1.0f, &tab);
    tab.blob = blob;
    bool one_size = n >= 2 && n <= kMaxMultiImages;
    for (int i = 1; one_size && i < n; i++) {
        const BatchSpec &a0 = specs[0], &ai = specs[i];
        one_size = ai.width == a0.width && ai.height == a0.height && ai.noisy_pitch == a0.noisy_pitch &&
                   ai.out_pitch == a0.out_pitch && ai.sigma == a0.sigma && ai.gamma == a0.gamma &&
                   (ai.out == nullptr) == (a0.out == nullptr) && (ai.smap == nullptr) == (a0.smap == nullptr) &&
                   (ai.rden == nullptr) == (a0.rden == nullptr) && (ai.g == nullptr) == (a0.g == nullptr) &&
                   ai.g_pitch == a0.g_pitch;
    }
    if (config >= 0) {
        b->plan = TilePlan::one(config);
    } else if (n == 1 || one_size) {
        b->plan = plan_for(ks, specs[0].width, specs[0].height, n);
    } else {
        std::vector<int> w(n), h(n);
        for (int i = 0; i < n; i++) {
            w[i] = specs[i].width;
            h[i] = specs[i].height;
        }
        b->plan = plan_for_images(ks, w.data(), h.data(), n);
    }
    rc = check_forward_limit(tab);
    if (rc == LPAICI_OK && b->plan.kind != TilePlan::kCluster) rc = check_tiles(b, tab);  // (clusters are chosen among those that fit)
    if (rc == LPAICI_OK && n != 1 && !one_size) rc = build_queue(b, ks, specs, n, tab);
    if (rc != LPAICI_OK) {
        batch_plan_free(b);
        return rc;
    }
    if (n == 1 || one_size) {
        const BatchSpec &im = specs[0];
        b->single = n == 1;
        b->multi = one_size;
        b->n_multi = one_size ? n : 0;
        for (int i = 0; one_size && i < n; i++) {
            b->mi.in[i] = specs[i].noisy;
            b->mi.out[i] = specs[i].out;
            b->mi.smap[i] = specs[i].smap;
            b->mi.rden[i] = specs[i].rden;
            b->mi.g[i] = specs[i].g;
        }
        b->img.in = im.noisy;
        b->img.out = im.out;
        b->img.smap = im.smap;
        b->img.rden = im.rden;
        b->img.g = im.g;
        b->img.g_pitch = im.g_pitch;
        b->img.W = im.width;
        b->img.in_h = im.height;
        b->img.in_pitch = im.noisy_pitch;
        b->img.out_pitch = im.out_pitch;
        b->img.row_begin = 0;
        b->img.rows_out = im.height;
        fill_tables(ks, nullptr, im.sigma, im.gamma, &b->tab);
        b->tab.blob = blob;
    }

    b->use_graph = use_graph;
    if (b->use_graph) {
        cudaStream_t cap = nullptr;
        cudaError_t e = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            rc = batch_plan_enqueue(b, cap);
            cudaError_t e2 = cudaStreamEndCapture(cap, &b->graph);
            if (rc == LPAICI_OK && e2 != cudaSuccess) rc = cuda_error(e2, "cudaStreamEndCapture");
            if (rc == LPAICI_OK) {
                e = cudaGraphInstantiate(&b->exec, b->graph, 0);
                if (e != cudaSuccess) rc = cuda_error(e, "cudaGraphInstantiate");
            }
        } else {
            rc = cuda_error(e, "graph capture");
        }
        if (cap) cudaStreamDestroy(cap);
        if (rc != LPAICI_OK) {
            batch_plan_free(b);
            return rc;
        }
        e = cudaGraphUpload(b->exec, stream);
        if (e != cudaSuccess) {
            batch_plan_free(b);
            return cuda_error(e, "cudaGraphUpload");
        }
    }
    *out = b;
    return LPAICI_OK;
}

}  // namespace lpaici

extern "C" {

int lpaici_batch_create(const lpaici_kernelset *ks, const lpaici_image *images, int n, const lpaici_batch_options *opts,
                        lpaici_stream_t stream_, lpaici_batch **out) {
    if (!ks || !images || n <= 0 || !out) return set_error(LPAICI_ERR_INVALID_ARG, "lpaici_batch_create: bad argument");
    *out = nullptr;
    std::vector<BatchSpec> specs(n);
    for (int i = 0; i < n; i++) {
        const lpaici_image &im = images[i];
        if (!im.noisy || !im.denoised || im.width <= 0 || im.height <= 0 || im.noisy_pitch < im.width ||
            im.out_pitch < im.width)
            return set_error(LPAICI_ERR_INVALID_ARG, "batch image %d: bad pointer or size", i);
        if (!(im.sigma > 0.0f) || !(im.gamma > 0.0f))
            return set_error(LPAICI_ERR_INVALID_ARG, "batch image %d: sigma and gamma need positive numbers", i);
        specs[i] = BatchSpec{im.noisy, im.denoised, im.scale_map, nullptr, im.width, im.height, im.noisy_pitch,
                             im.out_pitch, im.sigma, im.gamma};
    }
    const int config = opts ? opts->tile_config : -1;
    return batch_plan_create(ks, specs.data(), n, config, opts && opts->use_graph,
                             reinterpret_cast<cudaStream_t>(stream_), out);
}

int lpaici_batch_run(lpaici_batch *b, lpaici_stream_t stream_) {
    if (!b) return set_error(LPAICI_ERR_INVALID_ARG, "lpaici_batch_run: null plan");
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    int dev = -1;
    cudaGetDevice(&dev);
    if (dev != b->device)
        return set_error(LPAICI_ERR_INVALID_ARG, "batch planned on device %d, current device is %d", b->device, dev);
    if (b->use_graph) {
        cudaError_t e = cudaGraphLaunch(b->exec, stream);
        if (e != cudaSuccess) return cuda_error(e, "cudaGraphLaunch");
        return LPAICI_OK;
    }
    return batch_plan_enqueue(b, stream);
}

int lpaici_batch_destroy(lpaici_batch *b) {
    if (b) {
        int cur = -1;
        cudaGetDevice(&cur);
        cudaSetDevice(b->device);
        cudaDeviceSynchronize();
        batch_plan_free(b);
        if (cur >= 0) cudaSetDevice(cur);
    }
    return LPAICI_OK;
}

int lpaici_forward_batched(const lpaici_kernelset *ks, const lpaici_image *images, int n, lpaici_stream_t stream) {
    lpaici_batch *b = nullptr;
    lpaici_batch_options opts{0, -1};
    int rc = lpaici_batch_create(ks, images, n, &opts, stream, &b);
    if (rc != LPAICI_OK) return rc;
    rc = lpaici_batch_run(b, stream);
    cudaError_t e = cudaStreamSynchronize(reinterpret_cast<cudaStream_t>(stream));
    if (rc == LPAICI_OK && e != cudaSuccess) rc = cuda_error(e, "cudaStreamSynchronize");
    batch_plan_free(b);
    return rc;
}

}  // extern "C"
