// configs.h -- the tile configurations the kernels are instantiated for: region warps across WX and down WY,
// column pairs per thread Q (4 or 8), direction groups DS.  A region warp covers 16 rows x 4Q columns (2Q
// pixels per thread), so a CTA covers (4Q*WX) x (16*WY) pixels with 32*WX*WY*DS threads: DS groups of warps
// share the tile and split the directions (sweep_tile in tile_core.cuh).  Each launch takes the
// configuration with the least estimated time for its image (plan_for in capi.cu); configurations whose
// shared memory does not fit a kernel set are skipped.  The adjoint's selection pass runs the configuration
// the forward uses.  The last one is for sets of one or two directions, which groups do not divide, on images of few
// rows or few tiles: half of a 64 x 32 tile's time (85 x 85 in three scales, us: 4000 x 16 164 as 64 x 32 tiles, 118 as
// 64 x 16; 200 x 150 164 and 119).
#pragma once

// X(index, WX, WY, Q, DS)
#define LPAICI_TILE_CONFIGS(X) \
    X(0, 4, 4, 8, 1)           \
    X(1, 2, 4, 8, 2)           \
    X(2, 3, 2, 8, 2)           \
    X(3, 2, 2, 8, 4)           \
    X(4, 1, 2, 8, 8)           \
    X(5, 1, 1, 8, 16)          \
    X(6, 1, 1, 4, 8)           \
    X(7, 4, 2, 4, 1)           \
    X(8, 3, 4, 8, 1)           \
    X(9, 2, 4, 8, 1)           \
    X(10, 2, 4, 4, 2)          \
    X(11, 4, 1, 4, 1)

#define LPAICI_NUM_TILE_CONFIGS 12
#define LPAICI_DEFAULT_TILE_CONFIG 0

// The configurations that can take what whole waves of bigger tiles leave of an image (launch_rest in
// forward.cu), the mixes {big, rest} that a plan considers, and, in order of preference, the configurations for
// images of more tile rows than a grid has (the last one fits every supported kernel set).
#define LPAICI_REST_CONFIGS(X) \
    X(4, 1, 2, 8, 8)           \
    X(5, 1, 1, 8, 16)          \
    X(7, 4, 2, 4, 1)
#define LPAICI_TALL_CONFIGS {4, 7}
#define LPAICI_TILE_MIXES {{0, 4}, {0, 5}, {1, 5}, {3, 5}}

// Tiles that the C CTAs of a cluster share (images of a few tiles; lpaici_forward_cluster_kernel): each CTA has
// DS direction groups.  C = 1 takes the images that have more tiles than pairs of CTAs run at once, but no more
// than there are SMs: a tile's 16 directions in one round (200 x 150: 33.5 us as entry 6 above, 25.1 us so; tapered
// set 51.4 and 40.7 us).
// X(index, WX, WY, Q, DS, C)
#define LPAICI_CLUSTERS(X) \
    X(0, 1, 1, 4, 4, 4)    \
    X(1, 1, 1, 8, 4, 4)    \
    X(2, 1, 1, 8, 8, 2)    \
    X(3, 1, 1, 4, 16, 1)
#define LPAICI_NUM_CLUSTERS 4

// Without a device to estimate on, the first of these whose shared memory fits is used: the configurations
// in order of their B200 time on the 4096^2 benchmark image (16x7 symmetric kernels), fastest first.
#define LPAICI_TILE_PREFERENCE {0, 8, 1, 3, 2, 4, 9, 5, 10, 6, 7, 11}
