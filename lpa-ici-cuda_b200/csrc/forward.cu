// forward.cu -- LPA-ICI forward of one image, or of several of one size: a CTA (a cluster of CTAs for images of a few
// tiles) sweeps all directions and scales of an output tile and aggregates them; one launch, or two for images whose
// last wave small tiles take (launch_rest).
//
// Replaces the directional loop of anisotropic_lpa_ici_gpu_fused
// (src/v4_1_lpa_ici_2D_sparse_shared.cu:1216-1235), i.e. 16 launches of
// process_direction_fused_kernel (:1007-1092) + accumulate_direction_kernel (:1104-1111) and one
// normalize_estimate_kernel (:1113-1120), with the kernel set read from global memory (staged in
// shared memory per CTA) instead of capacity-limited constant memory.
#include "tile_core.cuh"
#include "configs.h"

namespace lpaici {

// A launch over part of the tiles may be followed by one over the rest (launch_rest), whose CTAs the hardware
// hands out once every CTA of this one has started.
__device__ __forceinline__ void let_rest_start(const KernelTables &tab) {
    if (tab.rest_follows) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Stages the kernel set, the tables and the tile at (x0, y0) of img, and sweeps it.
// Fused = false: every tap's product and sum rounded on their own (bit-exact with the reference);
// true: each tap one fused multiply-add (lpaici_forward_ffma).
template <int WX, int WY, int Q, int DS, bool Fused>
__device__ __forceinline__ void forward_tile(int *smem, const ImageArgs &img, const KernelTables &tab, int x0, int y0) {
    const int nk = tab.D * tab.S;
    const SweepCta<WX, WY, Q, DS> cta(smem, tab.blob_words, nk, tab.R);
    load_tile(cta.tile, img, x0, y0, cta.g);
    stage_blob<Q>(cta.blob, tab.blob, tab.blob_words, tab.mask_word, tab.stream_word, cta.g.pitch2);
    stage_tables(cta.tab, tab.var, tab.thr, nk);
    tile_wait();
    __syncthreads();
    sweep_tile<WX, WY, Q, DS, Fused>(img, x0, y0, tab.D, tab.S, cta.g, cta.blob, cta.tab, cta.tile, cta.xch, tab.neg_zero);
}

template <int WX, int WY, int Q, int DS, bool Fused>
__global__ void __launch_bounds__(32 * WX * WY * DS, 1)
    lpaici_forward_kernel(const __grid_constant__ ImageArgs img, const __grid_constant__ KernelTables tab) {
    extern __shared__ __align__(16) int smem[];
    using Shape = TileShape<WX, WY, Q, DS>;
    let_rest_start(tab);
    forward_tile<WX, WY, Q, DS, Fused>(smem, img, tab, blockIdx.x * Shape::kTileW, blockIdx.y * Shape::kTileH);
}

// Image z of a launch over several images (mi; img itself of a launch over one), in shared memory: kept in
// registers its pointers would stay live across the sweep (the single-image kernel reads its parameters).
struct SharedImage {
    __align__(16) unsigned char raw[sizeof(ImageArgs)];
    static_assert(sizeof(ImageArgs) + 16 <= kStaticShared, "static shared memory of the kernels that hold one");
    __device__ __forceinline__ const ImageArgs &fill(const ImageArgs &img, const MultiImages &mi, int images, int z) {
        ImageArgs &im = *reinterpret_cast<ImageArgs *>(raw);
        if (threadIdx.x == 0) {
            im = img;
            if (images > 1) {
                im.in = mi.in[z];
                im.out = mi.out[z];
                im.smap = mi.smap[z];
                im.rden = mi.rden[z];
                im.g = mi.g[z];
            }
        }
        __syncthreads();
        return im;
    }
};

// Several images of one size, pitch, sigma and gamma in one launch (a batched plan of such images, the channels
// of an interleaved image): grid layer z is image z, whose buffers replace img's; everything else is the
// single-image kernel.  The CTAs of image z + 1 fill the SMs image z's last wave leaves idle.  No counterpart
// in the reference.
template <int WX, int WY, int Q, int DS>
__global__ void __launch_bounds__(32 * WX * WY * DS, 1)
    lpaici_forward_multi_kernel(const __grid_constant__ ImageArgs img, const __grid_constant__ KernelTables tab,
                                const __grid_constant__ MultiImages mi) {
    extern __shared__ __align__(16) int smem[];
    __shared__ SharedImage s_img;
    using Shape = TileShape<WX, WY, Q, DS>;
    let_rest_start(tab);
    forward_tile<WX, WY, Q, DS, false>(smem, s_img.fill(img, mi, 2, blockIdx.z), tab, blockIdx.x * Shape::kTileW,
                                       blockIdx.y * Shape::kTileH);
}

// How a mix cuts each image: big tiles over [0, wb) x [0, hb), small ones over the strip to their right and over
// the rows below.
struct MixGrid {
    int images;
    int wb, hb;
    int right_x, n_right, bottom_x, n_small;  // n_small: both strips
};

// The small tiles of a mix.  Big tiles sweep a pixel in the least time, but an image of a few waves of them
// leaves SMs idle in the last one: the first launch takes whole waves of big tiles, this one cuts the rest into
// tiles of 8 or 16 direction groups, an eighth or a sixteenth of a big one's time, which fill the SMs as the big
// tiles end (programmatic dependent launch).  It depends on nothing of the first launch; its last CTA waits for
// that one, so that what follows in the stream follows both.
// us, gaussian 16 x 7 set with scale maps, 1535 x 1021 (192 big tiles are 1.3 waves): 787 with one configuration,
// 698 so; 768 x 513 x 3 channels 642 and 526.  (Both kinds of tiles in one kernel cost the big ones 2 to 5 %: the
// compiler allocates registers for both sweeps together.)
template <int WX, int WY, int Q, int DS, bool Fused>
__global__ void __launch_bounds__(32 * WX * WY * DS, 1)
    lpaici_forward_rest_kernel(const __grid_constant__ ImageArgs img, const __grid_constant__ KernelTables tab,
                               const __grid_constant__ MultiImages mi, const __grid_constant__ MixGrid g) {
    extern __shared__ __align__(16) int smem[];
    __shared__ SharedImage s_img;
    using Shape = TileShape<WX, WY, Q, DS>;
    const int z = blockIdx.x / g.n_small, t = blockIdx.x - z * g.n_small;
    // (the strips' tiles end where the big tiles do: a big tile is whole small ones high and wide)
    int x0, y0;
    if (t < g.n_right) {
        x0 = g.wb + (t % g.right_x) * Shape::kTileW;
        y0 = (t / g.right_x) * Shape::kTileH;
    } else {
        x0 = ((t - g.n_right) % g.bottom_x) * Shape::kTileW;
        y0 = g.hb + ((t - g.n_right) / g.bottom_x) * Shape::kTileH;
    }
    forward_tile<WX, WY, Q, DS, Fused>(smem, s_img.fill(img, mi, g.images, z), tab, x0, y0);
    if (blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// An image of a few tiles: C CTAs of a cluster share each tile's directions, as the groups of a CTA do.  Each
// stages only the runs of its directions if one round covers them all.  A group is one warp and its helper
// (SweepSplit).  97 x 64, 16 x 7 symmetric set, calls in a stream one after the other: 36.9 us with one CTA per 16 x 16
// tile, 22.6 us with four, 14.4 us with helpers (12.9 us of it the kernel, back to back in a graph).
template <int WX, int WY, int Q, int DS, int C, bool Fused>
__global__ void __launch_bounds__((C > 1 ? 2 : 1) * 32 * WX * WY * DS, 1)
    lpaici_forward_cluster_kernel(const __grid_constant__ ImageArgs img, const __grid_constant__ KernelTables tab) {
    extern __shared__ __align__(16) int smem[];
    using Shape = TileShape<WX, WY, Q, DS>;
    const int nk = tab.D * tab.S, tile = blockIdx.x / C, rank = blockIdx.x % C;
    const int across = (img.W + Shape::kTileW - 1) / Shape::kTileW;
    const int x0 = (tile % across) * Shape::kTileW, y0 = (tile / across) * Shape::kTileH;
    const SweepCta<WX, WY, Q, DS> cta(smem, tab.blob_words, nk, tab.R);
    int from = 0, to = 1 << 30;
    if (tab.D <= DS * C) {
        from = __ldg(tab.blob + min(tab.D, rank * DS) * tab.S);
        to = __ldg(tab.blob + min(tab.D, (rank + 1) * DS) * tab.S);
    }
    if (C > 1 && threadIdx.x < DS)  // no direction stopped yet
        reinterpret_cast<unsigned *>(reinterpret_cast<char *>(cta.xch) + Shape::kXchBytes +
                                     sizeof(float2) * kHelperScales * Q * Shape::kRegion * DS)[threadIdx.x] = 0;
    load_tile(cta.tile, img, x0, y0, cta.g);
    stage_blob<Q>(cta.blob, tab.blob, tab.blob_words, tab.mask_word, tab.stream_word, cta.g.pitch2, from, to);
    stage_tables(cta.tab, tab.var, tab.thr, nk);
    tile_wait();
    __syncthreads();
    sweep_tile<WX, WY, Q, DS, Fused, C>(img, x0, y0, tab.D, tab.S, cta.g, cta.blob, cta.tab, cta.tile, cta.xch,
                                        tab.neg_zero);
}

namespace {

// The helpers' sums and stop words follow the exchange; a cluster of one CTA has no helpers.
template <class Shape, int Q, int DS, int C>
size_t cluster_smem(int blob_words, int nk, int radius) {
    constexpr size_t helpers = sizeof(float2) * kHelperScales * Q * Shape::kRegion * DS + sizeof(int) * DS;
    return sweep_smem<Shape, Q>(blob_words, nk, radius) + (C > 1 ? helpers : 0);
}

template <int WX, int WY, int Q, int DS, int C, bool Fused>
int launch_cluster(const ImageArgs &img, const KernelTables &tab, cudaStream_t stream) {
    using Shape = TileShape<WX, WY, Q, DS>;
    static_assert(Shape::kRegion == 32, "a group is one warp and its helper");
    const size_t smem = cluster_smem<Shape, Q, DS, C>(tab.blob_words, tab.D * tab.S, tab.R);
    auto kern = lpaici_forward_cluster_kernel<WX, WY, Q, DS, C, Fused>;
    cudaError_t e = allow_shared_memory(reinterpret_cast<const void *>(kern));
    if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(forward, clusters)");
    const int tiles = ((img.W + Shape::kTileW - 1) / Shape::kTileW) * ((img.rows_out + Shape::kTileH - 1) / Shape::kTileH);
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = C;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(tiles) * C);
    cfg.blockDim = dim3((C > 1 ? 2 : 1) * Shape::kThreads);  // every warp has a helper
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kern, img, tab);
    return e == cudaSuccess ? LPAICI_OK : cuda_error(e, "forward launch (clusters)");
}

// across x down tiles from the image's origin (0: as many as cover it)
template <int WX, int WY, int Q, int DS>
int launch_multi_cfg(const ImageArgs &img, const KernelTables &tab, const MultiImages &mi, int n, int across, int down,
                     cudaStream_t stream) {
    using Shape = TileShape<WX, WY, Q, DS>;
    const size_t smem = sweep_smem<Shape, Q>(tab.blob_words, tab.D * tab.S, tab.R);
    auto kern = lpaici_forward_multi_kernel<WX, WY, Q, DS>;
    int dev = 0, max_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (smem + kStaticShared > static_cast<size_t>(max_optin))
        return set_error(LPAICI_ERR_UNSUPPORTED, "forward tile needs %zu B of shared memory, device allows %d",
                         smem + kStaticShared, max_optin);
    cudaError_t e = allow_shared_memory(reinterpret_cast<const void *>(kern), kStaticShared);
    if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(forward, several images)");
    const dim3 grid(across > 0 ? across : (img.W + Shape::kTileW - 1) / Shape::kTileW,
                    across > 0 ? down : (img.rows_out + Shape::kTileH - 1) / Shape::kTileH, n);
    kern<<<grid, Shape::kThreads, smem, stream>>>(img, tab, mi);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(e, "forward launch (several images)");
    return LPAICI_OK;
}

template <int WX, int WY, int Q, int DS, bool Fused>
int launch_cfg(const ImageArgs &img, const KernelTables &tab, int across, int down, cudaStream_t stream) {
    using Shape = TileShape<WX, WY, Q, DS>;
    const size_t smem = sweep_smem<Shape, Q>(tab.blob_words, tab.D * tab.S, tab.R);
    auto kern = lpaici_forward_kernel<WX, WY, Q, DS, Fused>;
    int dev = 0, max_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (smem > static_cast<size_t>(max_optin))
        return set_error(LPAICI_ERR_UNSUPPORTED, "forward tile needs %zu B of shared memory, device allows %d", smem,
                         max_optin);
    cudaError_t e = allow_shared_memory(reinterpret_cast<const void *>(kern));
    if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(forward)");
    const dim3 grid(across > 0 ? across : (img.W + Shape::kTileW - 1) / Shape::kTileW,
                    across > 0 ? down : (img.rows_out + Shape::kTileH - 1) / Shape::kTileH);
    kern<<<grid, Shape::kThreads, smem, stream>>>(img, tab);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(e, "forward launch");
    return LPAICI_OK;
}

template <int WX, int WY, int Q, int DS, bool Fused>
int launch_rest(const ImageArgs &img, const KernelTables &tab, const MultiImages &mi, const MixGrid &grid, cudaStream_t stream) {
    using Shape = TileShape<WX, WY, Q, DS>;
    const size_t smem = sweep_smem<Shape, Q>(tab.blob_words, tab.D * tab.S, tab.R);
    auto kern = lpaici_forward_rest_kernel<WX, WY, Q, DS, Fused>;
    cudaError_t e = allow_shared_memory(reinterpret_cast<const void *>(kern), kStaticShared);
    if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(forward, rest)");
    MixGrid g = grid;
    g.right_x = (img.W - g.wb + Shape::kTileW - 1) / Shape::kTileW;
    g.n_right = g.right_x * ((g.hb + Shape::kTileH - 1) / Shape::kTileH);
    g.bottom_x = (img.W + Shape::kTileW - 1) / Shape::kTileW;
    g.n_small = g.n_right + g.bottom_x * ((img.rows_out - g.hb + Shape::kTileH - 1) / Shape::kTileH);
    const long ctas = static_cast<long>(g.images) * g.n_small;
    if (ctas > 0x7fffffffL) return set_error(LPAICI_ERR_UNSUPPORTED, "image too large: %d x %d", img.W, img.rows_out);
    if (ctas == 0) return LPAICI_OK;
    const bool follows = g.wb > 0 && g.hb > 0;  // a launch over the big tiles; else this one has the whole image
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(ctas));
    cfg.blockDim = dim3(Shape::kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = follows ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, kern, img, tab, mi, g);
    return e == cudaSuccess ? LPAICI_OK : cuda_error(e, "forward launch (rest)");
}

}  // namespace

cudaError_t allow_shared_memory(const void *fn, size_t static_bytes) {
    int dev = 0, max_optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, max_optin - static_cast<int>(static_bytes));
}

#define LPAICI_FWD_CASE(idx, WX, WY, Q, DS)                                      \
    case idx:                                                                    \
        return fused ? launch_cfg<WX, WY, Q, DS, true>(img, tab, across, down, stream) \
                     : launch_cfg<WX, WY, Q, DS, false>(img, tab, across, down, stream);

template <int WX, int WY, int Q, int DS>
int blocks_per_sm(size_t smem) {
    auto kern = lpaici_forward_kernel<WX, WY, Q, DS, false>;
    if (allow_shared_memory(reinterpret_cast<const void *>(kern)) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, TileShape<WX, WY, Q, DS>::kThreads, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

int config_blocks_per_sm(int config, size_t smem) {
#define LPAICI_BPS_CASE(idx, WX, WY, Q, DS) \
    case idx: return blocks_per_sm<WX, WY, Q, DS>(smem);
    switch (config) {
        LPAICI_TILE_CONFIGS(LPAICI_BPS_CASE)
        default: return 0;
    }
#undef LPAICI_BPS_CASE
}

void config_tile(int config, int *tile_w, int *tile_h) {
#define LPAICI_TILE_CASE(idx, WX, WY, Q, DS) \
    case idx:                            \
        *tile_w = 4 * (Q) * (WX);        \
        *tile_h = 16 * (WY);             \
        return;
    switch (config) {
        LPAICI_TILE_CONFIGS(LPAICI_TILE_CASE)
        default: *tile_w = *tile_h = 1;
    }
#undef LPAICI_TILE_CASE
}

// Shared memory a tile configuration needs for a kernel set: blob + tables + the tile + the exchange.
size_t config_smem(int config, int blob_words, int nk, int R) {
#define LPAICI_SMEM_CASE(idx, WX, WY, Q, DS)                                                   \
    case idx:                                             \
        return sweep_smem<TileShape<WX, WY, Q, DS>, Q>(blob_words, nk, R);
    switch (config) {
        LPAICI_TILE_CONFIGS(LPAICI_SMEM_CASE)
        default: return ~size_t(0);
    }
#undef LPAICI_SMEM_CASE
}

int check_forward_limit(const KernelTables &tab) {
    int dev = 0, max_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const size_t need = sizeof(int) * (tab.limit_words + table_words(tab.D * tab.S)) +
                        sizeof(float2) * static_cast<size_t>(tile_pitch2(64 + 2 * tab.R + 4)) * (24 + 2 * tab.R);
    if (need <= static_cast<size_t>(max_optin)) return LPAICI_OK;
    return set_error(LPAICI_ERR_UNSUPPORTED, "forward tile needs %zu B of shared memory, device allows %d", need, max_optin);
}

static int launch_config(const ImageArgs &img, const KernelTables &tab, int config, int across, int down, bool fused,
                         cudaStream_t stream) {
    switch (config) {
        LPAICI_TILE_CONFIGS(LPAICI_FWD_CASE)
        default: return set_error(LPAICI_ERR_INVALID_ARG, "tile config %d out of range", config);
    }
}

static int launch_multi_config(const ImageArgs &img, const KernelTables &tab, const MultiImages &mi, int n, int config,
                               int across, int down, cudaStream_t stream) {
#define LPAICI_MULTI_CASE(idx, WX, WY, Q, DS) \
    case idx: return launch_multi_cfg<WX, WY, Q, DS>(img, tab, mi, n, across, down, stream);
    switch (config) {
        LPAICI_TILE_CONFIGS(LPAICI_MULTI_CASE)
        default: return set_error(LPAICI_ERR_INVALID_ARG, "tile config %d out of range", config);
    }
#undef LPAICI_MULTI_CASE
}

static int launch_rest_config(const ImageArgs &img, const KernelTables &tab, const MultiImages &mi, const MixGrid &g,
                              int config, bool fused, cudaStream_t stream) {
#define LPAICI_REST_CASE(idx, WX, WY, Q, DS)                                          \
    case idx:                                                                         \
        return fused ? launch_rest<WX, WY, Q, DS, true>(img, tab, mi, g, stream)      \
                     : launch_rest<WX, WY, Q, DS, false>(img, tab, mi, g, stream);
    switch (config) {
        LPAICI_REST_CONFIGS(LPAICI_REST_CASE)
        default: return set_error(LPAICI_ERR_INVALID_ARG, "tile config %d takes no rest", config);
    }
#undef LPAICI_REST_CASE
}

static int launch_cluster_config(const ImageArgs &img, const KernelTables &tab, int index, bool fused, cudaStream_t stream) {
#define LPAICI_CLUSTER_CASE(idx, WX, WY, Q, DS, C)                                        \
    case idx:                                                                             \
        return fused ? launch_cluster<WX, WY, Q, DS, C, true>(img, tab, stream)           \
                     : launch_cluster<WX, WY, Q, DS, C, false>(img, tab, stream);
    switch (index) {
        LPAICI_CLUSTERS(LPAICI_CLUSTER_CASE)
        default: return set_error(LPAICI_ERR_INVALID_ARG, "cluster configuration %d out of range", index);
    }
#undef LPAICI_CLUSTER_CASE
}

void cluster_config(int index, int radius, int blob_words, int nk, int *tile_w, int *tile_h, int *ctas, int *groups, size_t *smem) {
#define LPAICI_CLUSTER_CASE(idx, WX, WY, Q, DS, C)                                 \
    case idx:                                                                      \
        *tile_w = 4 * (Q) * (WX);                                                  \
        *tile_h = 16 * (WY);                                                       \
        *ctas = C;                                                                 \
        *groups = (DS) * (C);                                                      \
        *smem = cluster_smem<TileShape<WX, WY, Q, DS>, Q, DS, C>(blob_words, nk, radius); \
        return;
    switch (index) { LPAICI_CLUSTERS(LPAICI_CLUSTER_CASE) }
#undef LPAICI_CLUSTER_CASE
}

// Images of more tile rows than a grid has (16-row tiles: 1,048,560 rows) are swept as a rest without big tiles,
// whose tiles are all in blockIdx.x; taller than 65,535 of the tallest tiles there have been (128 rows), they are
// refused.  64-row tiles in grid layers were possible too, but the layer's row cost the other images 1.4 to 2.7 % (768
// x 513 x 3 channels 527 us and 541).
constexpr int kMaxGridRows = 65535;
constexpr int kMaxRows = 128 * kMaxGridRows;
static bool too_tall(const ImageArgs &img, const TilePlan &plan) {
    int tw = 1, th = 1;
    if (plan.kind == TilePlan::kCluster) return false;
    config_tile(plan.config, &tw, &th);
    return (plan.kind == TilePlan::kMix ? plan.big_rows : (img.rows_out + th - 1) / th) > kMaxGridRows;
}
static int launch_tall(const ImageArgs &img, const KernelTables &tab, const MultiImages &mi, int n, bool fused,
                       cudaStream_t stream) {
    if (img.rows_out > kMaxRows) return set_error(LPAICI_ERR_UNSUPPORTED, "image too tall: %d rows", img.rows_out);
    int dev = 0, max_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    MixGrid g{};
    g.images = n;
    static const int order[] = LPAICI_TALL_CONFIGS;
    for (const int c : order)
        if (config_smem(c, tab.blob_words, tab.D * tab.S, tab.R) + kStaticShared <= static_cast<size_t>(max_optin))
            return launch_rest_config(img, tab, mi, g, c, fused, stream);
    return set_error(LPAICI_ERR_UNSUPPORTED, "no tile for images of %d rows fits", img.rows_out);
}

// The strips of a plan's mix, for images of img's size.
static MixGrid mix_grid(const ImageArgs &img, const TilePlan &plan, int n, int *across) {
    int tw = 1, th = 1;
    config_tile(plan.config, &tw, &th);
    *across = img.W / tw;
    MixGrid g{};
    g.images = n;
    g.wb = *across * tw;
    g.hb = plan.big_rows * th;
    return g;
}

int launch_forward_multi(const ImageArgs &img, const KernelTables &tab, const MultiImages &mi, int n,
                         const TilePlan &plan, cudaStream_t stream) {
    if (tab.S > kMaxScales)
        return set_error(LPAICI_ERR_UNSUPPORTED, "%d scales per direction; the kernels support at most %d", tab.S,
                         kMaxScales);
    int rc = check_forward_limit(tab);
    if (rc != LPAICI_OK) return rc;
    if (n < 1 || n > kMaxMultiImages)
        return set_error(LPAICI_ERR_INVALID_ARG, "%d images in one launch; at most %d", n, kMaxMultiImages);
    if (too_tall(img, plan)) return launch_tall(img, tab, mi, n, false, stream);
    if (plan.kind == TilePlan::kOne) return launch_multi_config(img, tab, mi, n, plan.config, 0, 0, stream);
    int across = 0;
    const MixGrid g = mix_grid(img, plan, n, &across);
    KernelTables first = tab;
    first.rest_follows = 1;
    rc = launch_multi_config(img, first, mi, n, plan.config, across, plan.big_rows, stream);
    return rc == LPAICI_OK ? launch_rest_config(img, tab, mi, g, plan.rest, false, stream) : rc;
}

int launch_forward(const ImageArgs &img, const KernelTables &tab, const TilePlan &plan, cudaStream_t stream, bool fused) {
    if (tab.S > kMaxScales)
        return set_error(LPAICI_ERR_UNSUPPORTED, "%d scales per direction; the kernels support at most %d", tab.S,
                         kMaxScales);
    int rc = check_forward_limit(tab);
    if (rc != LPAICI_OK) return rc;
    if (too_tall(img, plan)) return launch_tall(img, tab, MultiImages{}, 1, fused, stream);
    if (plan.kind == TilePlan::kCluster) return launch_cluster_config(img, tab, plan.cluster, fused, stream);
    if (plan.kind == TilePlan::kOne) return launch_config(img, tab, plan.config, 0, 0, fused, stream);
    int across = 0;
    const MixGrid g = mix_grid(img, plan, 1, &across);
    KernelTables first = tab;
    first.rest_follows = 1;
    rc = launch_config(img, first, plan.config, across, plan.big_rows, fused, stream);
    return rc == LPAICI_OK ? launch_rest_config(img, tab, MultiImages{}, g, plan.rest, fused, stream) : rc;
}

}  // namespace lpaici
