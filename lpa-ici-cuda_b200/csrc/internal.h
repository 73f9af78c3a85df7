// internal.h -- shared declarations of the LPA-ICI library (not part of the C ABI).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "lpaici.h"

namespace lpaici {

// Limits of this library.  The per-kernel variance and threshold tables travel as kernel
// parameters (2 * 4 B * kMaxKernels), so D*S is capped; the radius bounds the shared-memory halo.
constexpr int kMaxKernels = 256;
constexpr int kMaxRadius = 127;
// The sweeps keep each pixel's selected scale in 4 bits.
constexpr int kMaxScales = 16;

// Device image of a kernel set, one contiguous block of 32-bit words, every part 16-byte aligned.
// A row run of a kernel is the taps (dy, dx0 + j), j < L, offsets from the output pixel (row - rows/2,
// col - cols/2), in row-major order.  The forward's blob:
//   [0, nk+1)               per kernel k the byte offset of its runs in the stream; they end where kernel
//                           k + 1's begin
//   [mask_word, ...)        one bit per 16-byte group of the stream: set for a run's first group
//   [stream_word, ...)      the stream: per run {dy, dx0, L % 4, L / 4}, its first L % 4 weights padded to a
//                           group of 4 (none if L % 4 is 0), the other weights in groups of 4
struct BlobLayout {
    int nk = 0, n_runs = 0;
    int mask_word = 0, stream_word = 0, total_words = 0;  // total a multiple of 4
    // the forward's support limit (check_forward_limit): words of the set with every weight stored twice
    int limit_words = 0;
};

// Device image of the adjoint's kernels (mirrored and telescoped, kernelset.cpp) for the gather's tile of
// 32*wx x 32*wy outputs and its field of two row planes (backward.cu), in bytes:
//   table          per piece entry_words(groups) words: {its block's byte offset | its scale, then 16 bits for each group's
//                  end of its stream, in 8-byte pairs from the block's start}, and one more entry; a block ends where the
//                  next one begins
//   blocks, 16-byte aligned: the stream of the first group of warps (every groups-th unit), then the next one's
// A piece is a kernel, or some units of one whose block is too large for two of them in shared memory.  A unit is
// {field byte offset, its bytes | flags | L % 4} and the weights of L taps, in one of two forms (a set has one):
//   pairs   a field row j of a kernel and the columns [a, a + L) where kernel row j (the tap of the lane's first output
//           row) or kernel row j - 1 (of its second) has taps; the weights are {D(j, t), D(j - 1, t)}, -0 where a row has
//           no tap;
//   single  a row j of a kernel, which the lane's second output row meets a field row further down; the weights are
//           D(j, t), the first L % 4 padded to an even number; flag 4: field row R + j is odd.
// The field offset is that of (row R + j, column R + a + L % 4).
struct AdjointLayout {
    int wx = 0, wy = 0;       // warps of one group across and down a tile
    bool single = false;      // the units' form
    // Groups of warps that share a tile's units.  Four where two are few warps for an SM (64 x 32 tiles: one to a
    // scheduler; 1024^2 from kept state, a 75 x 75 kernel in three scales 488 and 394 us), but not for 128 x 32 tiles of
    // pairs, which the two more groups' sums would leave no room (4 x 4 kernels of radius 45 529 and 642 us).
    static constexpr int groups(int wx, int wy, bool single) { return wx == 2 || (single && wy == 1) ? 4 : 2; }
    static constexpr int entry_words(int groups) { return groups > 2 ? 4 : 2; }
    int pitch = 0, plane = 0; // floats of a field row and of a row plane
    int block_bytes = 0;      // the largest block
    int pieces = 0;
    std::vector<int> first_piece;  // per direction, and past the last one
    int units = 0, taps = 0;  // of all kernels (weight pairs, or single weights)
    size_t limit_bytes = 0;   // shared memory the support limit counts (gather_setup)
    size_t limit_words = 0;   // of these the kernels, every weight stored twice; also the least size of the blob
    std::vector<int> box;     // per kernel: first and last row, first and last column of its taps (empty: 0, -1)
};

// Per-launch arguments shared by the forward and backward kernels (passed by value as a
// __grid_constant__ parameter; the tables are read with uniform indices from the constant bank).
struct ImageArgs {
    const float *in;  // input rows [0, in_h), width W, pitch in_pitch
    float *out;       // optional output rows [0, rows_out), pitch out_pitch
    uint8_t *smap;    // optional D x rows_out x W scale map
    float *rden;      // optional rows_out x W map of 1 / sum_d 1/v_d (pitch W; the adjoint's selection pass)
    const float *g;   // optional, with rden: the map is g * (1 / sum_d 1/v_d) (pitch g_pitch)
    int W, in_h, in_pitch, out_pitch, g_pitch;
    int row_begin;    // output row r is input row row_begin + r
    int rows_out;
    int step = 1;     // floats between neighbouring pixels of a row, in and out (channels of an interleaved image)
};

struct KernelTables {
    int D, S, R;
    float neg_zero;  // -0.0f, read at run time (see prod2 in tile_core.cuh)
    const int *blob;  // device blob (BlobLayout)
    int blob_words, mask_word, stream_word;
    int limit_words;
    int rest_follows = 0;  // a launch over the tiles that this one leaves follows (TilePlan::rest)
    float var[kMaxKernels];
    float thr[kMaxKernels];
};

// How a launch cuts its images into tiles.  Fields that a kind does not have are -1.
struct TilePlan {
    enum Kind {
        kOne,      // configuration `config` everywhere
        kMix,      // `config` over whole tiles, configuration `rest` over what they leave
        kCluster,  // one image, its tiles shared by clusters: entry `cluster` of LPAICI_CLUSTERS
    };
    Kind kind = kOne;
    int config = -1, rest = -1, cluster = -1;
    int big_rows = -1;   // mix over images of one size: whole tile rows of `config`, over their whole tile columns
    long big_tiles = -1; // mix over images of any sizes: whole tiles of `config`, largest images first
    static TilePlan one(int config) { return TilePlan{kOne, config, -1, -1, -1, -1}; }
    static TilePlan mix_rows(int config, int rest, int rows) { return TilePlan{kMix, config, rest, -1, rows, -1}; }
    static TilePlan mix_tiles(int config, int rest, long tiles) { return TilePlan{kMix, config, rest, -1, -1, tiles}; }
    static TilePlan clusters(int entry) { return TilePlan{kCluster, -1, -1, entry, -1, -1}; }
};

// Buffers of the images of a one-size batched plan (lpaici_forward_multi_kernel): image z's input,
// output, scale maps, 1/den (with a cotangent g/den) and cotangent (the last four may be null, as in ImageArgs).
constexpr int kMaxMultiImages = 64;
struct MultiImages {
    const float *in[kMaxMultiImages];
    float *out[kMaxMultiImages];
    uint8_t *smap[kMaxMultiImages];
    float *rden[kMaxMultiImages];
    const float *g[kMaxMultiImages];
};

int set_error(int code, const char *fmt, ...);
int cuda_error(cudaError_t e, const char *what);
// The checks every adjoint entry point makes before any copy or launch: sigma and gamma finite and
// positive (gamma only when the caller passes one), at most kMaxScales scales per direction (the
// selection sweep keeps each pixel's scale in 4 bits).  `who` names the entry point in the message.
int check_adjoint_params(const lpaici_kernelset *ks, float sigma, const float *gamma, const char *who);

}  // namespace lpaici

// The opaque kernel set of the C ABI.
struct lpaici_kernelset {
    int D = 0, S = 0;
    // the loader's dense output (load_LPA_kernels_standardized)
    std::vector<float> dense_w;
    std::vector<int> off, rows, cols;
    // the reference-layout run packing (build_sparse_kernels)
    std::vector<float> run_w;
    std::vector<int> run_row, run_col, run_len, k_first_run, k_num_runs, k_first_weight;
    // sum of squared weights per kernel, float, dense row-major order (compute_kernel_variances)
    std::vector<float> norm2;
    // nonzero taps per kernel (algorithmic work accounting)
    std::vector<int> nnz;
    int radius = 0;
    lpaici::BlobLayout layout;
    std::vector<int32_t> blob;  // host copy of the device blob
    // the adjoint gather's kernels, mirrored through their centre (taps (-dy, -dx)): scale 0 as it is, every
    // later scale as the difference from the scale before it (kernelset.cpp, build_adjoint_blob)
    lpaici::AdjointLayout adj_layout;
    std::vector<int32_t> adj_blob;
    // device copies, one per CUDA device, created on first use
    mutable std::mutex mu;
    mutable std::vector<int *> dev_blob;
    mutable std::vector<int *> dev_adj_blob;
    mutable std::vector<int> tuned_config;  // per device, -1 = not tuned
    // per device: ms one SM spends on one tile of each configuration, from lpaici_autotune (empty: not
    // tuned, or a configuration forced by lpaici_set_tile_config); and CTAs per SM of each (-1: unknown)
    mutable std::vector<std::vector<float>> tuned_tile_ms;
    mutable std::vector<std::vector<int>> blocks_per_sm;
};

namespace lpaici {

// Device blob of ks on the current device (uploaded on first use).  Returns an LPAICI_* code.
int device_blob(const lpaici_kernelset *ks, const int **out);
// The adjoint's flipped-kernel blob on the current device (uploaded on first use).
int device_adj_blob(const lpaici_kernelset *ks, const int **out);

// Fills var/thr exactly as the reference: var = (sigma*sigma)*norm2, thr = gamma*sqrt(var).
void fill_tables(const lpaici_kernelset *ks, const float *var_or_null, float sigma, float gamma, KernelTables *t);

// Forward / backward launchers (forward.cu, backward.cu).
// fused: each tap one fused multiply-add instead of a rounded product and a rounded sum (faster, not
// bit-exact with the reference: lpaici_forward_ffma).
int launch_forward(const ImageArgs &img, const KernelTables &tab, const TilePlan &plan, cudaStream_t stream,
                   bool fused = false);
// n images of img's size, pitches and tables (tab) in one launch, their buffers in mi.
int launch_forward_multi(const ImageArgs &img, const KernelTables &tab, const MultiImages &mi, int n, const TilePlan &plan,
                         cudaStream_t stream);
// Static shared memory of the kernels over several images and of the rest (their image arguments), rounded up.
constexpr size_t kStaticShared = 128;
// Lets kernel fn launch with all the dynamic shared memory that the current device has beside `static_bytes`.  The
// value never depends on the kernel set: the attribute belongs to the function, so that a smaller set's size would be
// in the way of a plan made before with a larger one, and of another thread's launch.
cudaError_t allow_shared_memory(const void *fn, size_t static_bytes = 0);
// Bytes of shared memory tile configuration `config` needs for a kernel set.
size_t config_smem(int config, int blob_words, int nk, int R);
// The autotuned configuration of ks on the current device, else the first one that fits.
int default_config(const lpaici_kernelset *ks);
// The plan expected to be fastest for one launch over n images of width x rows pixels: per-tile time (tuned,
// else a B200 cost model) times the waves of CTAs the images need.  A forced configuration wins.
TilePlan plan_for(const lpaici_kernelset *ks, int width, int rows, int n = 1);
// The same for one launch over n images of any sizes (a batched plan's tile queue): the images' tiles add up.
TilePlan plan_for_images(const lpaici_kernelset *ks, const int *widths, const int *rows, int n);
// Kernel sets are supported up to what a 64 x 32 tile with 24 + 2R pair rows takes in shared memory beside
// the set with duplicated weights: the bound on radius and taps that callers have always met, kept as it is
// (LPAICI_ERR_UNSUPPORTED beyond it) although today's tiles and weights take less.
int check_forward_limit(const KernelTables &tab);
// CTAs of the forward kernel of `config` that fit on one SM with `smem` bytes of shared memory.
int config_blocks_per_sm(int config, size_t smem);
// Tile, CTAs, direction groups (of all CTAs) and shared memory per CTA of entry `index` of LPAICI_CLUSTERS.
void cluster_config(int index, int radius, int blob_words, int nk, int *tile_w, int *tile_h, int *ctas, int *groups, size_t *smem);
// Tile width and height of a configuration.
void config_tile(int config, int *tile_w, int *tile_h);
// One image of a batch plan (batched.cu): out may be null (no estimate), smap, rden and g optional.
struct BatchSpec {
    const float *noisy;
    float *out;
    uint8_t *smap;
    float *rden;
    int width, height, noisy_pitch, out_pitch;
    float sigma, gamma;
    const float *g = nullptr;  // with rden: the map is g / den
    int g_pitch = 0;
};
// config < 0: chosen for the images (plan_for, plan_for_images).
int batch_plan_create(const lpaici_kernelset *ks, const BatchSpec *specs, int n, int config, bool use_graph,
                      cudaStream_t stream, lpaici_batch **out);
int batch_plan_enqueue(lpaici_batch *b, cudaStream_t stream);  // the launch, or the launch and the rest's
void batch_plan_free(lpaici_batch *b);

// The adjoint's two passes over storage the caller provides: device copies of ks->blob and ks->adj_blob,
// D*width*height selection bytes and width*height floats of g/den.  Allocates nothing.
int adjoint_passes(const lpaici_kernelset *ks, const int *blob, const int *adj_blob, uint8_t *smap, float *rden,
                   const float *d_noisy, int noisy_pitch, const float *d_grad_out, int gout_pitch, float *d_grad_in,
                   int gin_pitch, int width, int height, float sigma, float gamma, cudaStream_t stream);

}  // namespace lpaici
