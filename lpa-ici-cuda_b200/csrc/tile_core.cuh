// tile_core.cuh -- the per-tile LPA-ICI sweep shared by the single-image, batched and adjoint kernels.
//
// Shared memory of one CTA:
//   blob   the packed kernel set (BlobLayout): kernel table, runs, weights
//   tab    var[nk], thr[nk], rvar[nk] = 1/var of the image being processed
//   tile   T[j][c] = {x(j, c), x(j + TH/2, c)}: the input window of the TW x TH output tile as pairs of
//          rows TH/2 apart, j < TH/2 + 2R, c < pitch2 (odd); input row j is output row j - R of the tile,
//          input column c is output column c - R; zero outside the input
//   xch    (direction groups only) the groups' estimates of one round, see sweep_tile
//
// Thread mapping (Q = column pairs per thread, 4 or 8): a region warp covers 8 + 8 rows x 4Q columns; the
// lane with row index a (0..7) and column group b (0..3) owns the 2Q pixels of rows (a, a + TH/2) and
// columns Qb .. Qb + Q - 1, held as Q float2 pairs {row a, row a + TH/2}.  Every window value is then a
// natural register pair, so one packed product and one packed add do two pixels' taps.  The 16 lanes of a
// half-warp hit 16 different bank pairs with 8-byte loads (pitch2 odd): Q = 4 puts 4 rows x 4 groups in a
// half-warp (rows give the residues mod 4, groups the multiples of 4), Q = 8 puts 8 rows x 2 groups (rows
// give 8 distinct values mod 16 that never differ by 8, groups add 0 or 8).  Pairing rows half a tile
// apart instead of 8 stores TH/2 + 2R pair rows instead of TH - 8 + 2R (128 x 64 tiles at R = 31: 146 KB
// instead of 184 KB).
//
// What bounds the sweep, and why it looks as it does.  The work is FP32 arithmetic, two packed
// instructions per tap and pixel pair; on sm_100a each takes two cycles of its SM quarter's FP32 pipe, and
// an ALU instruction beside them costs 0.2 to 0.9 cycles more (its register reads compete with the packed
// instructions' 64-bit operands; measured with chains of packed instructions and one other instruction
// type), a shared load next to nothing.  So:
//   - 16 pixels per thread (Q = 8) where the image fills the chip: a run's descriptor, branches and
//     addresses serve twice the pixels of Q = 4;
//   - weights are single floats, four taps per 16-byte load: the packed product takes the weight as one
//     broadcast register, a {w, w} pair costs a second operand read and twice the shared memory;
//   - a run of L taps is a head of L % 4 taps (one dispatch to straight-line code) followed by L / 4
//     blocks of 4 taps over a sliding register window, with the four descriptor words ready to use; descriptor
//     and weights lie in one stream, so one pointer walks a direction's runs and ends every loop;
//   - shared memory is read by 32-bit shared addresses (ld.shared in PTX): generic pointers cost a third
//     of the uniform instructions per run.
// 4096^2, 16 x 7 symmetric kernels: 8.15 ms before (Q = 4, 64 x 96 tiles, 103 warp instructions per run of
// a 256-pixel warp), 6.84 ms now (128 x 64 tiles, 144 per run of a 512-pixel warp; with descriptors and
// weights behind pointers of their own 7.04 ms); the packed arithmetic alone would take 5.3 ms.  Per tile of
// 8,192 pixels and 16 warps: 32 cycles a tap (the packed arithmetic's own), about 45 a run and 150 an
// interval update.
//
// Arithmetic (bit-identical to src/v1_0_lpa_ici_2D_fused.cpp:803-930 for finite inputs):
//   conv  = sum over the kernel's taps in row-major order of w*x (rounded), added one by one with
//           round-to-nearest, starting from +0.0f -- packed f32x2 instructions round each half on its
//           own; zero-filled halo taps and zero weights add +-0, which changes nothing (a running sum
//           started at +0 never becomes -0);
//   lb/ub = conv -+ thr;  lo = max(lo, lb); hi = min(hi, ub); accept while hi >= lo, else stop;
//   num  += est * (1/var); den += 1/var (in direction order, 1/var correctly rounded);  out = num / den.
#pragma once

#include "internal.h"

namespace lpaici {

// Packed FP32 arithmetic, two lanes per instruction, each half rounded to nearest on its own.
//
// ptxas contracts a packed multiply feeding a packed add (mul.rn.f32x2 -> add.rn.f32x2) into one
// fused multiply-add even with .rn and --fmad=false, which changes the rounding of the sums.  The
// product is therefore formed as fma.rn.f32x2(w, x, nz) with nz = {-0, -0} passed in at run time
// (so it cannot be folded away): w*x + (-0) is w*x exactly before the single rounding, hence the
// correctly rounded product with its sign of zero; an fma feeding an add is never contracted.
__device__ __forceinline__ float2 prod2(float2 a, float2 b, float2 nz) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(nz.x), "f"(nz.y));
    return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "add.rn.f32x2 rd, ra, rb;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// One tap of the forward: the product rounded, then the sum rounded (bit-exact with the reference).
struct ExactTap {
    float2 nz;  // {-0, -0}, read at run time (see prod2)
    __device__ __forceinline__ float2 operator()(float2 acc, float2 w, float2 x) const {
        return add2(acc, prod2(w, x, nz));
    }
};

// d = a * b + c in each half, rounded on its own (the two halves of fmaf).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

// One tap as a fused multiply-add, acc + w * x rounded once: the adjoint's gather, and the forward's
// contracted mode (not bit-exact with the reference).
struct FmaTap {
    __device__ __forceinline__ float2 operator()(float2 acc, float2 w, float2 x) const { return fma2(w, x, acc); }
};

// Shared loads by 32-bit shared address.  Volatile keeps them behind the barrier that publishes the data.
__device__ __forceinline__ unsigned smem_addr(const void *p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ float lds1(unsigned a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ float2 lds2(unsigned a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ float4 lds4(unsigned a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ unsigned lds_u1(unsigned a) {
    unsigned v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 lds_u2(unsigned a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ int4 lds_i4(unsigned a) {
    int4 v;
    asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}

// 4 bytes from global to shared memory, asynchronously; zero (and no read) unless ok.
__device__ __forceinline__ void copy_or_zero(unsigned dst, const float *src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(ok ? 4 : 0) : "memory");
}

// Every thread of the cluster's CTAs; shared memory written before it is visible to the others after it.
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Shared address a as CTA `rank` of the cluster has it, and a load from there.
__device__ __forceinline__ unsigned cluster_addr(unsigned a, unsigned rank) {
    unsigned remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(a), "r"(rank));
    return remote;
}
__device__ __forceinline__ float cluster_lds1(unsigned remote) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}

// Smallest odd pitch (in float2) >= need.
__host__ __device__ inline int tile_pitch2(int need) { return need | 1; }

// A tile configuration: WX x WY region warps of Q column pairs per thread, times DS direction groups.
template <int WX, int WY, int Q, int DS>
struct TileShape {
    static_assert(Q == 4 || Q == 8, "the lane mapping and the run loop know Q = 4 and Q = 8");
    static constexpr int kRegion = 32 * WX * WY;  // threads of one direction group
    static constexpr int kThreads = kRegion * DS;
    static constexpr int kTileW = WX * 4 * Q;
    static constexpr int kTileH = WY * 16;
    // the exchange of a round: estimate * 1/var and 1/var of every group and pixel
    static constexpr size_t kXchBytes = DS > 1 ? sizeof(float) * 2 * DS * 2 * Q * kRegion : 0;
};

// Shared-memory geometry of a tile for radius R and Q column pairs per thread: tile_w + 2R columns
// of halo'd input plus Q spare columns, a margin no load reaches (the last column a run's window
// reads is tile_w + 2R - 1).
struct TileGeom {
    int R, pitch2, pairs, half;  // pairs: number of T rows; half: rows between the two halves of a pair
    __host__ __device__ static TileGeom make(int tile_w, int tile_h, int R, int Q) {
        TileGeom g;
        g.R = R;
        g.half = tile_h / 2;
        g.pitch2 = tile_pitch2(tile_w + 2 * R + Q);
        g.pairs = g.half + 2 * R;
        return g;
    }
    // rounded to 16 bytes: the exchange area follows
    __host__ __device__ size_t tile_bytes() const {
        return (sizeof(float2) * static_cast<size_t>(pitch2) * pairs + 15) & ~size_t(15);
    }
};

// Words of shared memory before the tile: the blob, then var/thr/rvar (padded to 16 bytes).
__host__ __device__ inline int table_words(int nk) { return (3 * nk + 3) & ~3; }

template <class Shape, int Q>
__host__ __device__ inline size_t sweep_smem(int blob_words, int nk, int R) {
    return sizeof(int) * (blob_words + table_words(nk)) + TileGeom::make(Shape::kTileW, Shape::kTileH, R, Q).tile_bytes() +
           Shape::kXchBytes;
}

// The first H = L % 4 taps of a run of L: straight-line code that loads the H + Q - 1 window columns and
// the H weights (one 16-byte group after the descriptor at `at`) and leaves the window of the next tap in
// win[0 .. Q - 2] and `at` behind the head.
template <int Q, int H, class Tap>
__device__ __forceinline__ void run_head(float2 (&acc)[Q], float2 (&win)[Q], unsigned src, unsigned &at, const Tap &tap) {
    float2 t[H + Q - 1];
    float w[4] = {};
    if constexpr (H == 1) {
        w[0] = lds1(at + 16);
    } else if constexpr (H == 2) {
        const float2 v = lds2(at + 16);
        w[0] = v.x, w[1] = v.y;
    } else if constexpr (H == 3) {
        const float4 v = lds4(at + 16);
        w[0] = v.x, w[1] = v.y, w[2] = v.z;
    }
#pragma unroll
    for (int i = 0; i < H + Q - 1; i++) t[i] = lds2(src + 8 * i);
#pragma unroll
    for (int j = 0; j < H; j++)
#pragma unroll
        for (int m = 0; m < Q; m++) acc[m] = tap(acc[m], make_float2(w[j], w[j]), t[j + m]);
#pragma unroll
    for (int i = 0; i < Q - 1; i++) win[i] = t[H + i];
    at += H > 0 ? 32 : 16;
}

// Four taps; the window slots have been rotated by 4 * P taps (Q = 8 alternates P = 0, 1).  src: column
// Q - 1 of the first of them.
template <int Q, int P, class Tap>
__device__ __forceinline__ void run_block(float2 (&acc)[Q], float2 (&win)[Q], unsigned src, unsigned wp, const Tap &tap) {
    const float4 v = lds4(wp);
    const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
        win[(4 * P + j + Q - 1) % Q] = lds2(src + 8 * j);
#pragma unroll
        for (int m = 0; m < Q; m++) acc[m] = tap(acc[m], make_float2(w[j], w[j]), win[(4 * P + j + m) % Q]);
    }
}

// acc[m] = tap(acc[m], w_j, T[.][col + m + j]) for j < L, tap by tap in order, for the thread's Q pixel
// pairs.  The run's descriptor is at `at`, its weights follow, the next run's descriptor follows them: {byte
// offset of the run's first column from the lane's pixel, L % 4, address of the run's end, byte offset of
// column L % 4 + Q - 1}.
template <int Q, class Tap>
__device__ __forceinline__ void conv_taps(float2 (&acc)[Q], unsigned lane_base, unsigned &at, const Tap &tap) {
    float2 win[Q];
    const int4 run = lds_i4(at);
    unsigned src = lane_base + run.x;
    const unsigned end = run.z;
    const int h = run.y;
    if (h < 2) {
        if (h == 0)
            run_head<Q, 0>(acc, win, src, at, tap);
        else
            run_head<Q, 1>(acc, win, src, at, tap);
    } else {
        if (h == 2)
            run_head<Q, 2>(acc, win, src, at, tap);
        else
            run_head<Q, 3>(acc, win, src, at, tap);
    }
    if (at == end) return;
    src = lane_base + run.w;
#pragma unroll 1
    while (true) {
        run_block<Q, 0>(acc, win, src, at, tap);
        at += 16;
        if constexpr (Q == 8) {
            if (at == end) break;
            run_block<Q, 1>(acc, win, src + 32, at, tap);
            at += 16;
        }
        if (at == end) break;
        src += 8 * Q;
    }
}

// Copies the forward blob to shared memory and resolves it for this tile: kernel table entries become
// shared addresses, run descriptors {dy, dx0, L % 4, L / 4} the offsets and addresses that conv_taps reads.
// Only the stream's bytes [from, to) are copied (a CTA that sweeps some directions).
template <int Q>
__device__ __forceinline__ void stage_blob(int *dst, const int *__restrict__ src, int words, int mask_word, int stream_word,
                                           int pitch2, int from = 0, int to = 1 << 30) {
    const int4 *s = reinterpret_cast<const int4 *>(src);
    int4 *d = reinterpret_cast<int4 *>(dst);
    const int m0 = mask_word >> 2, s0 = stream_word >> 2;
    const int stream = static_cast<int>(smem_addr(dst + stream_word));
    constexpr int kAhead = 4;  // groups and mask words loaded before the first is used
    const int n = min(words, stream_word + (to >> 2)) >> 2, step = blockDim.x, skip = from >> 4;
    for (int i0 = threadIdx.x; i0 < n - skip; i0 += kAhead * step) {
        int4 v[kAhead];
        int m[kAhead];
#pragma unroll
        for (int e = 0; e < kAhead; e++) {
            const int i = i0 + e * step + (i0 + e * step >= s0 ? skip : 0), j = i - s0;
            v[e] = i < n ? __ldg(s + i) : make_int4(0, 0, 0, 0);
            m[e] = i < n && j >= 0 ? __ldg(src + mask_word + (j >> 5)) >> (j & 31) : 0;
        }
#pragma unroll
        for (int e = 0; e < kAhead; e++) {
            const int i = i0 + e * step + (i0 + e * step >= s0 ? skip : 0), j = i - s0;
            int4 r = v[e];
            if (i < m0) {
                r = make_int4(stream + r.x, stream + r.y, stream + r.z, stream + r.w);
            } else if (m[e] & 1) {
                const int o = 8 * (r.x * pitch2 + r.y);
                r = make_int4(o, r.z, stream + 16 * (j + 1 + (r.z > 0) + r.w), o + 8 * (r.z + Q - 1));
            }
            if (i < n) d[i] = r;
        }
    }
}

// var, thr and rvar = 1/var (correctly rounded, the reference's 1.0f / var_d) into shared memory.
__device__ __forceinline__ void stage_tables(float *s_tab, const float *var, const float *thr, int nk) {
    for (int i = threadIdx.x; i < nk; i += blockDim.x) {
        s_tab[i] = var[i];
        s_tab[nk + i] = thr[i];
        s_tab[2 * nk + i] = __fdiv_rn(1.0f, var[i]);
    }
}

// Builds T for the output tile whose top-left output pixel is (x0, y0): input pixel (gy0 + j, gx0 + c) and
// (gy0 + j + TH/2, gx0 + c), gy0 = y0 + row_begin - R, gx0 = x0 - R.  Asynchronous 4-byte copies straight
// into the interleaved pairs (no alignment asked of the image, zeros where it ends): no load latency is
// waited for until tile_wait, and the kernel set is staged meanwhile (16 x 16 tiles: 22.4 us a tile, 24.0
// with plain loads; 128 x 64: 503 us, 508).  A lane keeps its column and walks down the rows, four rows of
// copies at a time: with few warps on an SM the copies' addresses, not the memory, are what takes time (97 x
// 64 in clusters 20.6 us with a row's pointers formed per copy, 18.9 us so; 1535 x 1021 691 and 683 us).
__device__ __forceinline__ void load_tile(float2 *s_tile, const ImageArgs &img, int x0, int y0, const TileGeom &g) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int gy0 = y0 + img.row_begin - g.R, gx0 = x0 - g.R;
    const ptrdiff_t down = static_cast<ptrdiff_t>(g.half) * img.in_pitch, next = static_cast<ptrdiff_t>(nwarps) * img.in_pitch;
    for (int c = lane; c < g.pitch2; c += 32) {
        const int gx = gx0 + c;
        const bool ok_x = gx >= 0 && gx < img.W;
        const int in_h = ok_x ? img.in_h : 0;
        int row = gy0 + warp;
        const float *src = img.in + static_cast<ptrdiff_t>(row) * img.in_pitch + static_cast<ptrdiff_t>(gx) * img.step;
        unsigned dst = smem_addr(s_tile + warp * g.pitch2 + c);
#pragma unroll 4
        for (int j = warp; j < g.pairs; j += nwarps) {
            const bool ok_a = static_cast<unsigned>(row) < static_cast<unsigned>(in_h);
            const bool ok_b = static_cast<unsigned>(row + g.half) < static_cast<unsigned>(in_h);
            copy_or_zero(dst, ok_a ? src : img.in, ok_a);
            copy_or_zero(dst + 4, ok_b ? src + down : img.in, ok_b);
            row += nwarps;
            src += next;
            dst += 8 * nwarps * g.pitch2;
        }
    }
}
// This thread's copies have landed (the barrier after it publishes everyone's).
__device__ __forceinline__ void tile_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Pixel i = 2m + h of a thread: column tx + m, row ty + h * TH/2.
template <int Q>
__device__ __forceinline__ float pick(const float2 (&v)[Q], int i) { return (i & 1) ? v[i >> 1].y : v[i >> 1].x; }

// Two warps share a direction of a cluster's tile (SweepSplit): the second one, its helper, convolves the scales
// from `first` on (the last one or two) while the other sweeps those before it, and hands the sums over in
// shared memory.  There is one warp to a scheduler otherwise, which waits for its own results most of the time
// (26,800 cycles for the slowest direction of 97 x 64, 6,000 of them packed arithmetic), and the largest scales
// are half of a direction's work.  Back to back in a graph, us: 97 x 64 18.9 -> 12.8 us, 128 x 128 23.6 -> 17.0, 150 x 120 27.2 -> 22.7; tapered
// set 25.0 -> 17.3, 32.9 -> 24.1, 41.9 -> 36.2 (with the exchange's loads ahead of its sums).
constexpr int kHelperScales = 2;
struct SweepSplit {
    int first;      // scale; S: no helper
    unsigned sums;  // shared address of the lane's first pair; a pair of the next column is kRegion pairs on
    unsigned pair;  // named barrier of the two warps
    unsigned stop;  // shared address of the number of the direction (+ 1) whose remaining scales nobody needs
};
// The first scale of direction d's helper: both warps' parts of the stream as equal as they get.
__device__ __forceinline__ int helper_first(unsigned kernel_table, int d, int S) {
    if (S < 2) return S;
    const unsigned at = kernel_table + 4 * d * S;
    const unsigned begin = lds_u1(at), end = lds_u1(at + 4 * S), last = lds_u1(at + 4 * (S - 1));
    if (S == 2) return 1;
    const unsigned before = lds_u1(at + 4 * (S - 2));
    return max(before - begin, end - before) < max(last - begin, end - last) ? S - 2 : S - 1;
}
__device__ __forceinline__ void pair_arrive(unsigned id) { asm volatile("barrier.cta.arrive %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void pair_wait(unsigned id) { asm volatile("barrier.cta.sync %0, 64;" ::"r"(id) : "memory"); }

// The ICI scale sweep of direction d for the thread's 2Q pixels (mask `valid`): per pixel the estimate
// of the last accepted scale (best) and that scale's index (4 bits per pixel in sidx, 8 pixels a word).
// The intersection [lo, hi] only shrinks, so once it is empty no later scale can be accepted: a stopped
// pixel needs no mask, its updates simply never accept again; a pixel outside the image starts with an
// empty intersection.  Scale 0 is always accepted (lo = -inf, hi = +inf before it), so the index is the
// count of accepted scales after it.  Warp-uniform scale loop; it ends when no pixel of the warp accepts.
template <int Q, bool Split, class Tap>
__device__ __forceinline__ void direction_sweep(int d, int S, unsigned valid, unsigned lane_base, unsigned kernel_table,
                                                unsigned thr_addr, const Tap &tap, float2 (&best)[Q],
                                                unsigned (&sidx)[Q / 4], const SweepSplit &split = {}) {
    [[maybe_unused]] bool waited = false;
    float lo[2 * Q], hi[2 * Q];
    unsigned next = kernel_table + 4 * d * S;
    unsigned thr_at = thr_addr + 4 * d * S;
    unsigned at = lds_u1(next);
#pragma unroll
    for (int i = 0; i < Q / 4; i++) sidx[i] = 0;
#pragma unroll 1
    for (int s = 0; s < S; s++) {
        float2 acc[Q];
#pragma unroll
        for (int m = 0; m < Q; m++) acc[m] = make_float2(0.0f, 0.0f);
        if (!Split || s < split.first) {
            next += 4;
            const unsigned end = lds_u1(next);
            if (at != end) {
#pragma unroll 1
                do conv_taps<Q>(acc, lane_base, at, tap);
                while (at != end);
            }
        } else {
            if (!waited) pair_wait(split.pair);
            waited = true;
#pragma unroll
            for (int m = 0; m < Q; m++) acc[m] = lds2(split.sums + 8 * 32 * ((s - split.first) * Q + m));
        }
        const float thr = lds1(thr_at);
        thr_at += 4;
        if (s == 0) {
#pragma unroll
            for (int m = 0; m < Q; m++) {
                const float2 lb = add2(acc[m], make_float2(-thr, -thr));  // conv - thr, exactly
                const float2 ub = add2(acc[m], make_float2(thr, thr));
                best[m] = acc[m];
                lo[2 * m] = (valid >> (2 * m)) & 1u ? fmaxf(-INFINITY, lb.x) : INFINITY;
                hi[2 * m] = (valid >> (2 * m)) & 1u ? fminf(INFINITY, ub.x) : -INFINITY;
                lo[2 * m + 1] = (valid >> (2 * m + 1)) & 1u ? fmaxf(-INFINITY, lb.y) : INFINITY;
                hi[2 * m + 1] = (valid >> (2 * m + 1)) & 1u ? fminf(INFINITY, ub.y) : -INFINITY;
            }
            continue;
        }
        unsigned was[Q / 4], changed = 0;
#pragma unroll
        for (int i = 0; i < Q / 4; i++) was[i] = sidx[i];
#pragma unroll
        for (int m = 0; m < Q; m++) {
            const float2 lb = add2(acc[m], make_float2(-thr, -thr));
            const float2 ub = add2(acc[m], make_float2(thr, thr));
            lo[2 * m] = fmaxf(lo[2 * m], lb.x);
            hi[2 * m] = fminf(hi[2 * m], ub.x);
            lo[2 * m + 1] = fmaxf(lo[2 * m + 1], lb.y);
            hi[2 * m + 1] = fminf(hi[2 * m + 1], ub.y);
            if (hi[2 * m] >= lo[2 * m]) {
                best[m].x = acc[m].x;
                sidx[m / 4] += 1u << (8 * (m % 4));
            }
            if (hi[2 * m + 1] >= lo[2 * m + 1]) {
                best[m].y = acc[m].y;
                sidx[m / 4] += 16u << (8 * (m % 4));
            }
        }
#pragma unroll
        for (int i = 0; i < Q / 4; i++) changed |= was[i] ^ sidx[i];
        if (!__any_sync(0xffffffffu, changed != 0)) break;  // every pixel of the warp has stopped
    }
    if constexpr (Split)
        if (!waited) {
            asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(split.stop), "r"(d + 1) : "memory");
            pair_wait(split.pair);
        }
}

// The helper's part: the sums of the scales from split.first on.  Between runs it looks whether the other warp has
// stopped before them (volatile: an ordinary shared load is hoisted out of the loop), so that a tile whose pixels all
// stop early ends early: one direction of scales 1 to 42, 33 x 17 flat 116 us without and 39 us so, 16 x 7 symmetric
// set 97 x 64 14.5 us either way.
template <int Q, class Tap>
__device__ __forceinline__ void helper_sweep(int d, int S, unsigned lane_base, unsigned kernel_table, const Tap &tap,
                                             const SweepSplit &split) {
    unsigned next = kernel_table + 4 * (d * S + split.first);
    unsigned at = lds_u1(next), to = split.sums;
#pragma unroll 1
    for (int s = split.first; s < S; s++) {
        float2 acc[Q];
#pragma unroll
        for (int m = 0; m < Q; m++) acc[m] = make_float2(0.0f, 0.0f);
        next += 4;
        const unsigned end = lds_u1(next);
        bool stopped = false;
        if (at != end) {
#pragma unroll 1
            do {
                unsigned word;
                asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(word) : "r"(split.stop) : "memory");
                conv_taps<Q>(acc, lane_base, at, tap);
                stopped = __any_sync(0xffffffffu, word == static_cast<unsigned>(d + 1));
            } while (at != end && !stopped);
        }
        if (stopped) break;
#pragma unroll
        for (int m = 0; m < Q; m++) {
            asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(to), "f"(acc[m].x), "f"(acc[m].y) : "memory");
            to += 8 * 32;
        }
    }
    pair_arrive(split.pair);
}

// The forward sweep of one tile (blob, tables and tile in shared memory, block-synchronised).
//
// DS = 1: every thread sweeps all directions of its pixels and sums num and den in registers.  DS > 1:
// DS groups of threads cover the same pixels and take the directions in rounds, group g direction
// round * DS + g; after each round the groups' estimates meet in shared memory (xch) and each group adds
// them, in direction order, to the num and den of its share of the pixels -- the same additions in the same
// order as DS = 1, so the results are equal bit for bit.  A tile then takes 1/DS of the time: images with
// fewer pixels than the chip has room for (148 SMs x 8,192 pixels) are cut into smaller tiles (97 x 64: 257
// us before, 36 us as 16 x 16 tiles of 8 groups; 512^2: 268 us before, 135 us as 64 x 32 tiles of 4).  It
// costs halo and a barrier per round: at 4096^2 the tiles of 2, 4, 8 and 16 groups take 7.3, 7.3, 7.8 and
// 8.3 ms against 6.84 ms.
//
// C > 1: the CTAs of a cluster share the tile in the same way, CTA `rank` with the directions
// round * DS * C + rank * DS + group; the estimates meet through distributed shared memory.
template <int WX, int WY, int Q, int DS, bool Fused, int C = 1>
__device__ __forceinline__ void sweep_tile(const ImageArgs &img, int x0, int y0, int D, int S, const TileGeom &g,
                                           const int *s_blob, const float *s_tab, const float2 *s_tile, float *s_xch,
                                           float neg_zero) {
    using Shape = TileShape<WX, WY, Q, DS>;
    static_assert(C == 1 || DS > 1, "a cluster's CTAs have the exchange of direction groups");
    constexpr int kGroups = DS * C;
    unsigned rank = 0;
    if constexpr (C > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    // first output row and column of a thread's pixels (see the thread mapping above), from its index: formed
    // again where results are written (`again` is opaque), so that the sweep does not carry them
    auto place = [&](int t, int *oy, int *ox) {
        const int rt = DS == 1 ? t : t % Shape::kRegion, warp = rt >> 5, lane = rt & 31;
        const int a = Q == 4 ? (lane >> 2) : (lane & 7), b = Q == 4 ? (lane & 3) : (lane >> 3);
        *oy = y0 + (warp / WX) * 8 + a;
        *ox = x0 + (warp % WX) * 4 * Q + Q * b;
    };
    auto again = [] {
        int t;
        asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
        return t;
    };
    // the group is the same in every lane of a warp: reduced, the compiler knows it warp-uniform, so the run
    // loops branch without reconvergence bookkeeping
    const int groups_warp = DS == 1 ? 0 : static_cast<int>(__reduce_max_sync(0xffffffffu, threadIdx.x / Shape::kRegion));
    const bool helper = C > 1 && groups_warp >= DS;
    const int group = helper ? groups_warp - DS : groups_warp;
    const int nk = D * S;
    unsigned valid = 0, lane_base;
    {
        int oy, ox;
        place(threadIdx.x, &oy, &ox);
#pragma unroll
        for (int i = 0; i < 2 * Q; i++)
            if (oy + g.half * (i & 1) < img.rows_out && ox + (i >> 1) < img.W) valid |= 1u << i;
        lane_base = smem_addr(s_tile + (oy - y0 + g.R) * g.pitch2 + ox - x0 + g.R);
    }
    const bool work = __any_sync(0xffffffffu, valid != 0);  // a warp outside the image only joins the barriers
    if (DS == 1 && !work) return;
    const unsigned kernel_table = smem_addr(s_blob);
    const unsigned thr_addr = smem_addr(s_tab + nk), rvar_addr = smem_addr(s_tab + 2 * nk);
    // opaque, so that the compiler keeps it in a register instead of reading it again in every run
    asm volatile("mov.b32 %0, %0;" : "+f"(neg_zero));
    const float2 nz = make_float2(neg_zero, neg_zero);

    auto stop_word = [&](int g) {
        return smem_addr(s_xch) + static_cast<unsigned>(Shape::kXchBytes) + 8 * DS * kHelperScales * Q * 32 + 4 * g;
    };
    // the pixels whose num and den this thread sums: all 2Q (DS = 1), else kOwn of them
    constexpr int kOwn = DS == 1 ? 2 * Q : (2 * Q >= kGroups ? 2 * Q / kGroups : 1);
    const int owner = static_cast<int>(rank) * DS + group;  // among all groups
    float2 num[Q], den[Q];
    float onum[kOwn], oden[kOwn];
    if constexpr (DS == 1) {
#pragma unroll
        for (int m = 0; m < Q; m++) num[m] = den[m] = make_float2(0.0f, 0.0f);
    } else {
#pragma unroll
        for (int i = 0; i < kOwn; i++) onum[i] = oden[i] = 0.0f;
    }

#pragma unroll 1
    for (int d0 = 0; d0 < D; d0 += kGroups) {
        const int d = d0 + owner;
        if (DS > 1 && d0 > 0) {  // the previous round's estimates have been added
            if constexpr (C > 1)
                cluster_barrier();
            else
                __syncthreads();
        }
        if (helper && d < D && work) {
            const SweepSplit split{helper_first(kernel_table, d, S),
                                   smem_addr(s_xch) + static_cast<unsigned>(Shape::kXchBytes) +
                                       8 * (group * kHelperScales * Q * 32 + threadIdx.x % 32),
                                   1u + group, stop_word(group)};
            if constexpr (Fused)
                helper_sweep<Q>(d, S, lane_base, kernel_table, FmaTap{}, split);
            else
                helper_sweep<Q>(d, S, lane_base, kernel_table, ExactTap{nz}, split);
        } else if (d < D && work) {
            float2 best[Q];
            unsigned sidx[Q / 4];
            SweepSplit split{};
            if constexpr (C > 1) {
                split.first = helper_first(kernel_table, d, S);
                split.sums = smem_addr(s_xch) + static_cast<unsigned>(Shape::kXchBytes) +
                             8 * (group * kHelperScales * Q * 32 + threadIdx.x % 32);
                split.pair = 1 + group;
                split.stop = stop_word(group);
            }
            if constexpr (Fused)
                direction_sweep<Q, (C > 1)>(d, S, valid, lane_base, kernel_table, thr_addr, FmaTap{}, best, sidx, split);
            else
                direction_sweep<Q, (C > 1)>(d, S, valid, lane_base, kernel_table, thr_addr, ExactTap{nz}, best, sidx, split);
            const unsigned rd = rvar_addr + 4 * d * S;
#pragma unroll
            for (int m = 0; m < Q; m++) {
                const unsigned bits = sidx[m / 4] >> (8 * (m % 4));
                const float2 r = make_float2(lds1(rd + 4 * (bits & 15)), lds1(rd + 4 * ((bits >> 4) & 15)));
                const float2 e = prod2(best[m], r, nz);
                if constexpr (DS == 1) {
                    num[m] = add2(num[m], e);
                    den[m] = add2(den[m], r);
                } else {
                    float *x = s_xch + (group * 2 * Q + 2 * m) * Shape::kRegion + threadIdx.x % Shape::kRegion;
                    x[0] = e.x;
                    x[Shape::kRegion] = e.y;
                    x += DS * 2 * Q * Shape::kRegion;
                    x[0] = r.x;
                    x[Shape::kRegion] = r.y;
                }
            }
            if (img.smap) {
                int oy, ox;
                place(again(), &oy, &ox);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    uint8_t *row = img.smap + (static_cast<size_t>(d) * img.rows_out + oy + g.half * h) * img.W + ox;
                    constexpr unsigned kRow = Q == 8 ? 0x5555u : 0x55u;  // this half's pixels in `valid`
                    if (((valid >> h) & kRow) == kRow && (reinterpret_cast<size_t>(row) & 3) == 0) {
                        // the index words hold four pixels of either row as bytes of 4 + 4 bits
#pragma unroll
                        for (int w = 0; w < Q / 4; w++)
                            reinterpret_cast<unsigned *>(row)[w] = (sidx[w] >> (4 * h)) & 0x0f0f0f0fu;
                    } else {
#pragma unroll
                        for (int m = 0; m < Q; m++)
                            if (valid & (1u << (2 * m + h)))
                                row[m] = static_cast<uint8_t>((sidx[m / 4] >> (8 * (m % 4) + 4 * h)) & 15);
                    }
                }
            }
        }
        if constexpr (DS > 1) {
            if constexpr (C > 1)
                cluster_barrier();
            else
                __syncthreads();
            if (owner * kOwn < 2 * Q && work && !helper) {
                const float *x = s_xch + owner * kOwn * Shape::kRegion + threadIdx.x % Shape::kRegion;
                // all loads before the first sum: one latency a round instead of one per group
                float nu[kGroups][kOwn], de[kGroups][kOwn];
#pragma unroll
                for (int e = 0; e < kGroups; e++)
#pragma unroll
                    for (int i = 0; i < kOwn; i++) {
                        const float *p = x + (e % DS * 2 * Q + i) * Shape::kRegion;
                        if constexpr (C > 1) {
                            const unsigned at = cluster_addr(smem_addr(p), e / DS);
                            nu[e][i] = cluster_lds1(at);
                            de[e][i] = cluster_lds1(at + sizeof(float) * DS * 2 * Q * Shape::kRegion);
                        } else {
                            nu[e][i] = p[0];
                            de[e][i] = p[DS * 2 * Q * Shape::kRegion];
                        }
                    }
#pragma unroll
                for (int e = 0; e < kGroups; e++)
                    if (d0 + e < D)
#pragma unroll
                        for (int i = 0; i < kOwn; i++) {
                            onum[i] = __fadd_rn(onum[i], nu[e][i]);
                            oden[i] = __fadd_rn(oden[i], de[e][i]);
                        }
            }
        }
    }
    if constexpr (C > 1) cluster_barrier();  // a CTA's shared memory stays until every other one has read it
    if (DS > 1 && (owner * kOwn >= 2 * Q || helper)) return;
    int oy, ox;
    place(again(), &oy, &ox);
#pragma unroll
    for (int j = 0; j < kOwn; j++) {
        const int i = DS == 1 ? j : owner * kOwn + j;
        if (!(valid & (1u << i))) continue;
        const float nu = DS == 1 ? pick<Q>(num, j) : onum[j], de = DS == 1 ? pick<Q>(den, j) : oden[j];
        const int y = oy + g.half * (i & 1), x = ox + (i >> 1);
        if (img.out)
            img.out[static_cast<size_t>(y) * img.out_pitch + static_cast<size_t>(x) * img.step] = __fdiv_rn(nu, de);
        if (img.rden) {
            const float r = __frcp_rn(de);
            img.rden[static_cast<size_t>(y) * img.W + x] = img.g ? __ldg(img.g + static_cast<size_t>(y) * img.g_pitch + x) * r : r;
        }
    }
}

// One CTA's work on the tile at (x0, y0) of img: stages the kernel set, the tables and the tile, and sweeps.
template <int WX, int WY, int Q, int DS>
struct SweepCta {
    using Shape = TileShape<WX, WY, Q, DS>;
    int *blob;
    float *tab;
    float2 *tile;
    float *xch;
    TileGeom g;
    __device__ __forceinline__ SweepCta(int *smem, int blob_words, int nk, int R)
        : blob(smem), g(TileGeom::make(Shape::kTileW, Shape::kTileH, R, Q)) {
        tab = reinterpret_cast<float *>(smem + blob_words);
        tile = reinterpret_cast<float2 *>(smem + blob_words + table_words(nk));
        xch = reinterpret_cast<float *>(reinterpret_cast<char *>(tile) + g.tile_bytes());
    }
};

}  // namespace lpaici
