// forward.cu -- single-image LPA-ICI forward: one launch, one CTA per output tile, all directions
// and scales of the tile inside the CTA, aggregation in registers.
//
// Replaces the directional loop of anisotropic_lpa_ici_gpu_fused
// (src/v4_1_lpa_ici_2D_sparse_shared.cu:1216-1235), i.e. 16 launches of
// process_direction_fused_kernel (:1007-1092) + accumulate_direction_kernel (:1104-1111) and one
// normalize_estimate_kernel (:1113-1120), with the kernel set read from global memory (staged in
// shared memory per CTA) instead of capacity-limited constant memory.
#include "tile_core.cuh"
#include "configs.h"

namespace lpaici {

// Stages the kernel set, the tables and the tile at (x0, y0) of img, and sweeps it.
// Fused = false: every tap's product and sum rounded on their own (bit-exact with the reference);
// true: each tap one fused multiply-add (lpaici_forward_ffma).
template <int WX, int WY, int Q, int DS, bool Fused>
__device__ __forceinline__ void forward_tile(int *smem, const ImageArgs &img, const KernelTables &tab, int x0, int y0) {
    const int nk = tab.D * tab.S;
    const SweepCta<WX, WY, Q, DS> cta(smem, tab.blob_words, nk, tab.R);
    load_tile(cta.tile, img, x0, y0, cta.g);
    stage_blob<Q>(cta.blob, tab.blob, tab.blob_words, tab.run_word, tab.weight_word, cta.g.pitch2);
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
    forward_tile<WX, WY, Q, DS, Fused>(smem, img, tab, blockIdx.x * Shape::kTileW, blockIdx.y * Shape::kTileH);
}

__device__ __forceinline__ ImageArgs image_of(const ImageArgs &img, const MultiImages &mi, int z) {
    ImageArgs im = img;
    im.in = mi.in[z];
    im.out = mi.out[z];
    im.smap = mi.smap[z];
    im.rden = mi.rden[z];
    return im;
}

// Several images of one size, pitch, sigma and gamma in one launch (a batched plan of such images, the channels
// of an interleaved image): grid layer z is image z, whose buffers replace img's; everything else is the
// single-image kernel.  The CTAs of image z + 1 fill the SMs image z's last wave leaves idle.  No counterpart
// in the reference.
template <int WX, int WY, int Q, int DS>
__global__ void __launch_bounds__(32 * WX * WY * DS, 1)
    lpaici_forward_multi_kernel(const __grid_constant__ ImageArgs img, const __grid_constant__ KernelTables tab,
                                const __grid_constant__ MultiImages mi) {
    extern __shared__ __align__(16) int smem[];
    using Shape = TileShape<WX, WY, Q, DS>;
    forward_tile<WX, WY, Q, DS, false>(smem, image_of(img, mi, blockIdx.z), tab, blockIdx.x * Shape::kTileW,
                                       blockIdx.y * Shape::kTileH);
}

// How a mixed launch cuts each image: big tiles over [0, wb) x [0, hb), small ones over the strip to their right
// and over the rows below.  CTAs: the big tiles of all images, then the small ones.
struct MixGrid {
    int images;
    int wb, hb, big_x, n_big;
    int right_x, n_right, bottom_x, n_small;  // n_small: both strips
};

// Big tiles sweep a pixel in the least time, but an image of a few waves of them leaves SMs idle in the last
// one: the launch takes whole waves of big tiles and cuts the rest into tiles of 8 or 16 direction groups, an
// eighth or a sixteenth of a big one's time, which fill the SMs as the big tiles end.  1535 x 1021 (192 big
// tiles are 1.3 waves): 817 us with one configuration, 736 us mixed; 1600 x 1200 contracted 738 and 641 us; a
// 10-image plan 2506 and 2173 us.
template <int AX, int AY, int AQ, int AD, int BX, int BY, int BQ, int BD, bool Fused>
__global__ void __launch_bounds__(32 * AX * AY * AD, 1)
    lpaici_forward_mixed_kernel(const __grid_constant__ ImageArgs img, const __grid_constant__ KernelTables tab,
                                const __grid_constant__ MultiImages mi, const __grid_constant__ MixGrid g) {
    static_assert(AX * AY * AD == BX * BY * BD, "both tiles have the CTA's threads");
    static_assert(AY % BY == 0 && AX * AQ % (BX * BQ) == 0, "a big tile is whole small ones");
    extern __shared__ __align__(16) int smem[];
    using Big = TileShape<AX, AY, AQ, AD>;
    using Small = TileShape<BX, BY, BQ, BD>;
    int b = blockIdx.x;
    const int all_big = g.images * g.n_big;
    if (b < all_big) {
        const int z = b / g.n_big, t = b - z * g.n_big;
        const int x0 = (t % g.big_x) * Big::kTileW, y0 = (t / g.big_x) * Big::kTileH;
        if (g.images == 1)
            forward_tile<AX, AY, AQ, AD, Fused>(smem, img, tab, x0, y0);
        else
            forward_tile<AX, AY, AQ, AD, Fused>(smem, image_of(img, mi, z), tab, x0, y0);
        return;
    }
    b -= all_big;
    const int z = b / g.n_small;
    int t = b - z * g.n_small, x0, y0;
    if (t < g.n_right) {
        x0 = g.wb + (t % g.right_x) * Small::kTileW;
        y0 = (t / g.right_x) * Small::kTileH;
    } else {
        t -= g.n_right;
        x0 = (t % g.bottom_x) * Small::kTileW;
        y0 = g.hb + (t / g.bottom_x) * Small::kTileH;
    }
    // (the strips' tiles end where the big tiles do: a big tile is whole small ones high and wide)
    if (g.images == 1)
        forward_tile<BX, BY, BQ, BD, Fused>(smem, img, tab, x0, y0);
    else
        forward_tile<BX, BY, BQ, BD, Fused>(smem, image_of(img, mi, z), tab, x0, y0);
}

namespace {

template <int WX, int WY, int Q, int DS>
int launch_multi_cfg(const ImageArgs &img, const KernelTables &tab, const MultiImages &mi, int n,
                     cudaStream_t stream) {
    using Shape = TileShape<WX, WY, Q, DS>;
    const size_t smem = sweep_smem<Shape, Q>(tab.blob_words, tab.D * tab.S, tab.R);
    auto kern = lpaici_forward_multi_kernel<WX, WY, Q, DS>;
    int dev = 0, max_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (smem > static_cast<size_t>(max_optin))
        return set_error(LPAICI_ERR_UNSUPPORTED, "forward tile needs %zu B of shared memory, device allows %d", smem,
                         max_optin);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(forward, several images)");
    const dim3 grid((img.W + Shape::kTileW - 1) / Shape::kTileW, (img.rows_out + Shape::kTileH - 1) / Shape::kTileH,
                    n);
    if (grid.y > 65535u) return set_error(LPAICI_ERR_UNSUPPORTED, "image too tall: %d rows", img.rows_out);
    kern<<<grid, Shape::kThreads, smem, stream>>>(img, tab, mi);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(e, "forward launch (several images)");
    return LPAICI_OK;
}

template <int WX, int WY, int Q, int DS, bool Fused>
int launch_cfg(const ImageArgs &img, const KernelTables &tab, cudaStream_t stream) {
    using Shape = TileShape<WX, WY, Q, DS>;
    const size_t smem = sweep_smem<Shape, Q>(tab.blob_words, tab.D * tab.S, tab.R);
    auto kern = lpaici_forward_kernel<WX, WY, Q, DS, Fused>;
    int dev = 0, max_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (smem > static_cast<size_t>(max_optin))
        return set_error(LPAICI_ERR_UNSUPPORTED, "forward tile needs %zu B of shared memory, device allows %d", smem,
                         max_optin);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(forward)");
    const dim3 grid((img.W + Shape::kTileW - 1) / Shape::kTileW, (img.rows_out + Shape::kTileH - 1) / Shape::kTileH);
    if (grid.y > 65535u) return set_error(LPAICI_ERR_UNSUPPORTED, "image too tall: %d rows", img.rows_out);
    kern<<<grid, Shape::kThreads, smem, stream>>>(img, tab);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(e, "forward launch");
    return LPAICI_OK;
}

template <int AX, int AY, int AQ, int AD, int BX, int BY, int BQ, int BD, bool Fused>
int launch_mixed(const ImageArgs &img, const KernelTables &tab, const MultiImages &mi, int n, int big_rows,
                 cudaStream_t stream) {
    using Big = TileShape<AX, AY, AQ, AD>;
    using Small = TileShape<BX, BY, BQ, BD>;
    const size_t sa = sweep_smem<Big, AQ>(tab.blob_words, tab.D * tab.S, tab.R);
    const size_t sb = sweep_smem<Small, BQ>(tab.blob_words, tab.D * tab.S, tab.R);
    const size_t smem = sa > sb ? sa : sb;
    auto kern = lpaici_forward_mixed_kernel<AX, AY, AQ, AD, BX, BY, BQ, BD, Fused>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(forward, mixed tiles)");
    MixGrid g{};
    g.images = n;
    g.big_x = img.W / Big::kTileW;
    g.wb = g.big_x * Big::kTileW;
    g.hb = big_rows * Big::kTileH;
    g.n_big = g.big_x * big_rows;
    g.right_x = (img.W - g.wb + Small::kTileW - 1) / Small::kTileW;
    g.n_right = g.right_x * ((g.hb + Small::kTileH - 1) / Small::kTileH);
    g.bottom_x = (img.W + Small::kTileW - 1) / Small::kTileW;
    g.n_small = g.n_right + g.bottom_x * ((img.rows_out - g.hb + Small::kTileH - 1) / Small::kTileH);
    const long ctas = static_cast<long>(n) * (g.n_big + g.n_small);
    if (ctas > 0x7fffffffL) return set_error(LPAICI_ERR_UNSUPPORTED, "image too large: %d x %d", img.W, img.rows_out);
    kern<<<static_cast<unsigned>(ctas), Big::kThreads, smem, stream>>>(img, tab, mi, g);
    e = cudaGetLastError();
    return e == cudaSuccess ? LPAICI_OK : cuda_error(e, "forward launch (mixed tiles)");
}

int forward_mixed(const ImageArgs &img, const KernelTables &tab, const MultiImages &mi, int n, const TilePlan &plan,
                  bool fused, cudaStream_t stream) {
#define LPAICI_MIX_CASE(idx, A, AX, AY, AQ, AD, B, BX, BY, BQ, BD)                                                     \
    case idx:                                                                                                          \
        return fused ? launch_mixed<AX, AY, AQ, AD, BX, BY, BQ, BD, true>(img, tab, mi, n, plan.big_rows, stream)     \
                     : launch_mixed<AX, AY, AQ, AD, BX, BY, BQ, BD, false>(img, tab, mi, n, plan.big_rows, stream);
    switch (plan.mix) {
        LPAICI_TILE_MIXES(LPAICI_MIX_CASE)
        default: return set_error(LPAICI_ERR_INVALID_ARG, "tile mix %d out of range", plan.mix);
    }
#undef LPAICI_MIX_CASE
}

}  // namespace

#define LPAICI_FWD_CASE(idx, WX, WY, Q, DS) \
    case idx: return fused ? launch_cfg<WX, WY, Q, DS, true>(img, tab, stream) : launch_cfg<WX, WY, Q, DS, false>(img, tab, stream);

template <int WX, int WY, int Q, int DS>
int blocks_per_sm(size_t smem) {
    auto kern = lpaici_forward_kernel<WX, WY, Q, DS, false>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess) {
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

// Shared memory a tile configuration needs for a kernel set: blob + tables + the T8 tile.
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

int launch_forward_multi(const ImageArgs &img, const KernelTables &tab, const MultiImages &mi, int n,
                         const TilePlan &plan, cudaStream_t stream) {
    if (tab.S > kMaxScales)
        return set_error(LPAICI_ERR_UNSUPPORTED, "%d scales per direction; the kernels support at most %d", tab.S,
                         kMaxScales);
    const int rc = check_forward_limit(tab);
    if (rc != LPAICI_OK) return rc;
    if (n < 1 || n > kMaxMultiImages)
        return set_error(LPAICI_ERR_INVALID_ARG, "%d images in one launch; at most %d", n, kMaxMultiImages);
    if (plan.mix >= 0) return forward_mixed(img, tab, mi, n, plan, false, stream);
#define LPAICI_MULTI_CASE(idx, WX, WY, Q, DS) \
    case idx: return launch_multi_cfg<WX, WY, Q, DS>(img, tab, mi, n, stream);
    switch (plan.config) {
        LPAICI_TILE_CONFIGS(LPAICI_MULTI_CASE)
        default: return set_error(LPAICI_ERR_INVALID_ARG, "tile config %d out of range", plan.config);
    }
#undef LPAICI_MULTI_CASE
}

int launch_forward(const ImageArgs &img, const KernelTables &tab, const TilePlan &plan, cudaStream_t stream, bool fused) {
    if (tab.S > kMaxScales)
        return set_error(LPAICI_ERR_UNSUPPORTED, "%d scales per direction; the kernels support at most %d", tab.S,
                         kMaxScales);
    const int rc = check_forward_limit(tab);
    if (rc != LPAICI_OK) return rc;
    if (plan.mix >= 0) return forward_mixed(img, tab, MultiImages{}, 1, plan, fused, stream);
    switch (plan.config) {
        LPAICI_TILE_CONFIGS(LPAICI_FWD_CASE)
        default: return set_error(LPAICI_ERR_INVALID_ARG, "tile config %d out of range", plan.config);
    }
}

}  // namespace lpaici
