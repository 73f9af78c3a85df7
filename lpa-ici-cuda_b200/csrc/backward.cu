// backward.cu -- adjoint of the LPA-ICI forward with the ICI selection held fixed.
//
// For L = sum_p g[p] * out[p] and the selected scale s*(d,p) of every direction and pixel frozen,
// out is linear in the input x:  out(p) = sum_d alpha_d(p) * sum_t h_{d,s*}(t) x(p + t - c), with
// alpha_d(p) = (1/v_{d,s*}) / den(p), den(p) = sum_d' 1/v_{d',s*}.  With the adjoint field of direction d
//     c_d(p) = g(p) / den(p) / v_{d, s*(d,p)},
//     dL/dx(q) = sum_d sum_s sum_t h'_{d,s}(t) [s*(d, q + t) = s] c_d(q + t)       (zero padding)
// where h' is h mirrored through its centre: for every direction and scale, a correlation of the field
// masked to the pixels that selected that scale.  Two passes:
//   A. selection: the forward's exact tile sweep recomputes s*(d,p) (one byte per direction and
//      pixel) and writes u = g * (1/den) beside it, into a transient workspace -- the forward stores
//      nothing for the adjoint (a kept state holds 1/den, and the gather forms the product itself);
//   B. gather: 128 x 64 output tiles (128 x 32 or 64 x 32 for kernels that leave no room).  Per direction
//      it reads s*(d,.) and u on the tile plus its R-pixel halo (from L2) and forms the field
//      c_d = u / v_{d,s*} in shared memory.
//      The kernels are telescoped, D_s = h'_s - h'_{s-1} (D_0 = h'_0, built by kernelset.cpp), which
//      turns the sum over scales into
//          sum_s D_s (*) (c_d [s* >= s]):
//      the field is zeroed in place where s* < s, scale after scale, and never rebuilt.  Two (or four)
//      groups of warps take every second (fourth) unit of each kernel over the same outputs.  Every output is
//      written once: no atomics, deterministic.
//
// Order of the sums.  The directions are cut into kGatherChunks chunks; each group sums every chunk from
// zero (its units in order), the chunks' sums are added in order, and the groups' totals are added in order.
// A tile is gathered by one CTA or by a cluster of kGatherChunks or half as many CTAs (the tiles after the last
// whole wave, gather_plan) that share the chunks
// and add the same sums in the same order through distributed shared memory, so the gradient does not depend on
// how many CTAs a tile gets (single images, plans and kept states agree bit for bit).
// No counterpart in the reference.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <vector>

#include "configs.h"
#include "tile_core.cuh"

namespace lpaici {

namespace {

// Gather tile geometry.  A lane owns output rows ty, ty + 1 (ty even) at Q = 16 consecutive columns; a warp
// covers 32 rows x 32 columns (lane l: row pair l & 15, column group l >> 4), WX x WY warps make a group,
// two or four groups a CTA (AdjointLayout::groups).
//
// Why row pairs one row apart: field row j meets output row y in kernel row j - y and output row y + 1 in
// kernel row j - y - 1, so one window of field values serves both output rows, and the packed FMA takes
// {D(dy, t), D(dy - 1, t)} times one broadcast value.  Against rows 8 apart with one weight and a pair of
// values per tap (the design before), that halves the shared loads, which the gather was limited by (29
// wavefronts a run of 5.7 taps against 8 x 5.7 packed FMAs at 16 outputs a lane), and the packed FMA itself
// issues faster: 2.0 to 2.2 cycles with one 64-bit operand reused, one broadcast and the accumulator,
// against 2.4 to 3.4 with three register pairs (measured in chains).  It costs the taps where only one of
// two neighbouring kernel rows has one: 18 % more for the 16 x 7 sets, 10 % for the tapered ones.  Sets with much
// more of them have units of single weights and windows of both field rows (single_unit): twice the shared loads, 3 %
// more for a packed FMA, twice the time before a unit's first tap, no padding (kernelset.cpp has the rule).
// Q = 16 spreads a run's descriptor, branches and window over 32 outputs.
// From kept state, 16 x 7 symmetric set: 1024^2 573 us before, 452 us now (300 us of it the units: 250 cycles
// a unit of 6.0 taps and 32 outputs a lane, 191 of them the packed FMAs; builds 44 us, masking 45 us); tapered
// set 964 and 685 us; 384 x 320 (15 tiles) 571 and 66 us.
constexpr int kGatherQ = 16;
constexpr int kGatherChunks = 8;
template <int WX, int WY, bool Single>
struct GatherShape {
    static constexpr int kTW = 32 * WX, kTH = 32 * WY;
    static constexpr int kGroups = AdjointLayout::groups(WX, WY, Single);
    static constexpr int kEntry = AdjointLayout::entry_words(kGroups);
    static constexpr int kRegion = 32 * WX * WY;
    static constexpr int kThreads = kGroups * kRegion;
    // Kernels in pieces have the smallest tile (build_adjoint_blob); elsewhere a piece is a kernel, and looking pieces up
    // would cost (64 directions of two scales, 2048^2 from kept state: 2,152 us with lookups, 2,119 us so).
    static constexpr bool kPieces = WX == 2;
};

// One image of the gather: pass A's outputs and the caller's buffers.
struct GatherImage {
    const float *g;        // cotangent, pitch g_pitch
    const uint8_t *smap;   // D x H x W selected scales (pass A)
    const float *rden;     // H x W, pitch W: 1 / den, den = sum_d 1/v_d (pass A); u = g * (1/den) when u_ready
    float *grad;           // result, pitch grad_pitch
    const float *rvar;     // 1 / v_k of this image (batched plans; one image: GatherArgs::rvar)
    int g_pitch, grad_pitch, W, H;
    int tiles_x;
    int u_ready;           // rden holds u = g * (1 / den) already (pass A)
};

struct GatherArgs {
    GatherImage single;          // the image of a one-image launch (images == null)
    const GatherImage *images;   // batched: per-image descriptors in device memory
    const int2 *items;           // batched: (image, tile) of every tile
    int D, S, R;
    const int *blob;       // mirrored kernels (lpaici_kernelset::adj_blob, AdjointLayout)
    int pieces;
    int block_bytes;       // shared memory for one piece's block
    int pitch, plane;      // field geometry (AdjointLayout)
    int cluster;           // CTAs per tile: 1, kGatherChunks / 2 or kGatherChunks
    int first_tile;        // this launch's tiles start here
    int rest_follows;      // a launch over the tiles after this one's follows
    float rvar[kMaxKernels];  // 1 / v_k of the one image
    // per direction: the field cells its kernels read, rows [x, y), columns [z, w)
    int4 drect[kMaxKernels];
    int first_piece[kMaxKernels + 1];  // per direction, and past the last one
};

// Shared memory: piece table | 1/v table | non-finite flags | two blocks | field | selected scales |
// the groups' sums over the chunks (touched once per chunk: in registers they would cost the run loop its own).
// The field is stored as two planes of even and odd rows (field row r: plane r & 1, row r >> 1): the 16 row
// pairs of a warp start on rows of one parity, so with an odd pitch its 32 scalar loads hit 32 banks.
struct GatherSmem {
    int rv, flag, block, field, smap, sums, total;  // byte offsets
    __host__ __device__ static GatherSmem make(int nk, int entry_words, int pieces, int block_bytes, int plane, int region, int groups) {
        GatherSmem m;
        m.rv = (4 * entry_words * (pieces + 1) + 15) & ~15;
        m.flag = m.rv + ((4 * nk + 15) & ~15);
        m.block = m.flag + 16;
        m.field = m.block + 2 * block_bytes;
        m.smap = m.field + 4 * 2 * plane;
        m.sums = m.smap + ((2 * plane + 15) & ~15);
        m.total = m.sums + static_cast<int>(sizeof(float2)) * kGatherQ * region * groups;
        return m;
    }
};

// The first H = L % 4 taps of a unit; the next tap's window is loaded already, src points at its first value.
template <int H>
__device__ __forceinline__ void gather_head(float2 (&acc)[kGatherQ], const float (&win)[kGatherQ], unsigned src, unsigned &at) {
    constexpr int Q = kGatherQ;
    float lead[H];  // the H columns before the window
    float2 w[H];
#pragma unroll
    for (int j = 0; j < H; j++) w[j] = lds2(at + 8 * j);
#pragma unroll
    for (int j = 0; j < H; j++) lead[j] = lds1(src + 4 * j - 4 * H);
#pragma unroll
    for (int j = 0; j < H; j++)
#pragma unroll
        for (int m = 0; m < Q; m++) {
            const float x = j + m < H ? lead[j + m < H ? j + m : 0] : win[j + m < H ? 0 : j + m - H];
            acc[m] = fma2(w[j], make_float2(x, x), acc[m]);
        }
    at += 8 * H;
}

// Four taps; the window slots have been rotated by 4 * P taps.
template <int P>
__device__ __forceinline__ void gather_block(float2 (&acc)[kGatherQ], float (&win)[kGatherQ], unsigned src, unsigned wp) {
    constexpr int Q = kGatherQ;
    float2 w[4];
#pragma unroll
    for (int j = 0; j < 4; j++) w[j] = lds2(wp + 8 * j);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        win[(4 * P + j + Q - 1) % Q] = lds1(src + 4 * j);
#pragma unroll
        for (int m = 0; m < Q; m++) {
            const float x = win[(4 * P + j + m) % Q];
            acc[m] = fma2(w[j], make_float2(x, x), acc[m]);
        }
    }
}

// acc[m] += {w0_t, w1_t} * field[m + t] over a unit of h + 4n taps whose L weight pairs are at [at, end); src: the
// field value of tap h.  The window is loaded before the dispatch on h: loaded in each head it costs register moves
// where the heads meet.
__device__ __forceinline__ void gather_unit(float2 (&acc)[kGatherQ], unsigned src, unsigned h, unsigned at, unsigned end) {
    float win[kGatherQ];
#pragma unroll
    for (int i = 0; i < kGatherQ - 1; i++) win[i] = lds1(src + 4 * i);
    if (h > 0) {
        if (h == 1)
            gather_head<1>(acc, win, src, at);
        else if (h == 2)
            gather_head<2>(acc, win, src, at);
        else
            gather_head<3>(acc, win, src, at);
    }
    if (at == end) return;
    src += 4 * (kGatherQ - 1);
#pragma unroll 1
    while (true) {
        gather_block<0>(acc, win, src, at);
        src += 16;
        at += 32;
        if (at == end) break;
        gather_block<1>(acc, win, src, at);
        src += 16;
        at += 32;
        if (at == end) break;
        gather_block<2>(acc, win, src, at);
        src += 16;
        at += 32;
        if (at == end) break;
        gather_block<3>(acc, win, src, at);
        src += 16;
        at += 32;
        if (at == end) break;
    }
}

// A unit of single weights (AdjointLayout::single): acc[m] += w_t * {field row r, field row r + 1}[m + t].  The window
// holds both rows; a and b: their values of tap h.
template <int H>
__device__ __forceinline__ void single_head(float2 (&acc)[kGatherQ], const float2 (&win)[kGatherQ], unsigned a, unsigned b,
                                            unsigned &at) {
    constexpr int Q = kGatherQ;
    float2 lead[H];
    float w[4] = {};
    const float2 v = lds2(at);
    w[0] = v.x, w[1] = v.y;
    if constexpr (H == 3) w[2] = lds1(at + 8);
#pragma unroll
    for (int j = 0; j < H; j++) lead[j] = make_float2(lds1(a + 4 * j - 4 * H), lds1(b + 4 * j - 4 * H));
#pragma unroll
    for (int j = 0; j < H; j++)
#pragma unroll
        for (int m = 0; m < Q; m++)
            acc[m] = fma2(make_float2(w[j], w[j]), j + m < H ? lead[j + m < H ? j + m : 0] : win[j + m < H ? 0 : j + m - H], acc[m]);
    at += H == 3 ? 16 : 8;
}
template <int P>
__device__ __forceinline__ void single_block(float2 (&acc)[kGatherQ], float2 (&win)[kGatherQ], unsigned a, unsigned b, unsigned wp) {
    constexpr int Q = kGatherQ;
    const float2 w01 = lds2(wp), w23 = lds2(wp + 8);
    const float w[4] = {w01.x, w01.y, w23.x, w23.y};
#pragma unroll
    for (int j = 0; j < 4; j++) {
        win[(4 * P + j + Q - 1) % Q] = make_float2(lds1(a + 4 * j), lds1(b + 4 * j));
#pragma unroll
        for (int m = 0; m < Q; m++) acc[m] = fma2(make_float2(w[j], w[j]), win[(4 * P + j + m) % Q], acc[m]);
    }
}
__device__ __forceinline__ void single_unit(float2 (&acc)[kGatherQ], unsigned a, unsigned b, unsigned h, unsigned at, unsigned end) {
    float2 win[kGatherQ];
#pragma unroll
    for (int i = 0; i < kGatherQ - 1; i++) win[i] = make_float2(lds1(a + 4 * i), lds1(b + 4 * i));
    if (h > 0) {
        if (h == 1)
            single_head<1>(acc, win, a, b, at);
        else if (h == 2)
            single_head<2>(acc, win, a, b, at);
        else
            single_head<3>(acc, win, a, b, at);
    }
    if (at == end) return;
    a += 4 * (kGatherQ - 1);
    b += 4 * (kGatherQ - 1);
#pragma unroll 1
    while (true) {
        single_block<0>(acc, win, a, b, at);
        at += 16;
        if (at == end) break;
        single_block<1>(acc, win, a + 16, b + 16, at);
        at += 16;
        if (at == end) break;
        single_block<2>(acc, win, a + 32, b + 32, at);
        at += 16;
        if (at == end) break;
        single_block<3>(acc, win, a + 48, b + 48, at);
        at += 16;
        if (at == end) break;
        a += 64;
        b += 64;
    }
}

// The same as gather_unit for a field with infinities or NaNs: the padding weights (-0, where only the other output row has
// a tap) are skipped, so that only the pixels whose kernels reach such a value see it.
__device__ __noinline__ void gather_run_skipping(float2 *acc, unsigned src, unsigned wp, int len) {
    for (int t = 0; t < len; t++) {
        const float2 w = lds2(wp + 8 * t);
        const bool first = __float_as_uint(w.x) != 0x80000000u, second = __float_as_uint(w.y) != 0x80000000u;
        for (int m = 0; m < kGatherQ; m++) {
            const float x = lds1(src + 4 * (t + m));
            if (first) acc[m].x = fmaf(w.x, x, acc[m].x);
            if (second) acc[m].y = fmaf(w.y, x, acc[m].y);
        }
    }
}

// Pieces I .. N - 1 of one row, 32 columns apart: selected scale and u of the lane's column, zero (and no read) unless
// first <= piece < past.  One predicate for both loads, no branch around them, offsets in the instructions.
template <bool UReady, int I, int N>
__device__ __forceinline__ void load_pieces(unsigned (&sc)[N], float (&u)[N], const uint8_t *map, const float *den, const float *g,
                                            int first, int past) {
    if constexpr (I < N) {
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tsetp.le.s32 p, %4, %6;\n\tsetp.gt.and.s32 q, %5, %6, p;\n\t"
            "mov.u32 %0, 0;\n\tmov.f32 %1, 0f00000000;\n\t"
            "@q ld.global.nc.u8 %0, [%2 + %7];\n\t@q ld.global.nc.f32 %1, [%3 + %8];\n\t}"
            : "=r"(sc[I]), "=f"(u[I])
            : "l"(map), "l"(den), "r"(first), "r"(past), "n"(I), "n"(32 * I), "n"(128 * I));
        if constexpr (!UReady) {
            float x;
            asm volatile(
                "{\n\t.reg .pred p, q;\n\tsetp.le.s32 p, %2, %4;\n\tsetp.gt.and.s32 q, %3, %4, p;\n\t"
                "mov.f32 %0, 0f00000000;\n\t@q ld.global.nc.f32 %0, [%1 + %5];\n\t}"
                : "=f"(x)
                : "l"(g), "r"(first), "r"(past), "n"(I), "n"(128 * I));
            u[I] = x * u[I];
        }
        load_pieces<UReady, I + 1, N>(sc, u, map, den, g, first, past);
    }
}

// s*(d, .) and c_d = u / v_{d, s*}, u = g / den (0 outside the image), for the field rows [dr.x, dr.y) and
// columns [dr.z, dr.w) that the direction's kernels reach; the other cells keep stale values that no
// correlation of this direction reads.  u is read again for every direction (from L2): kept in shared memory
// it would not leave room for 128 x 64 tiles.  A warp takes kRows rows of kAcross x 32 columns at a time, all
// loads in flight: between the barriers around it the build is bound by the loads' latency and the index
// arithmetic, not by the bytes.  Returns whether a value of this thread is infinite or NaN.
template <bool UReady, bool Inside>
__device__ __forceinline__ bool build_field(unsigned s_f, unsigned s_s, unsigned rv, const GatherImage &im,
                                            const uint8_t *map, const int4 dr, int gx0, int gy0, int pitch, int plane,
                                            int warp, int nwarps, int lane) {
    constexpr int kRows = 2, kAcross = 5;
    bool bad = false;
    for (int c0 = dr.z; c0 < dr.w; c0 += 32 * kAcross) {
        const int c = c0 + lane, gx = gx0 + c;
        // columns c + 32 i: stored for i < stored, read from the image for first <= i < past
        const int stored = (dr.w - c + 31) >> 5, first = gx >= 0 ? 0 : (-gx + 31) >> 5, past = min(stored, (im.W - gx + 31) >> 5);
        // of field row 0 (outside the image possibly: only rows and columns inside are read)
        const long long px0 = static_cast<long long>(gy0) * im.W + gx;
        const uint8_t *pm0 = map + px0;
        const float *pd0 = im.rden + px0, *pg0 = im.g + static_cast<long long>(gy0) * im.g_pitch + gx;
        for (int r0 = dr.x + warp; r0 < dr.y; r0 += kRows * nwarps) {
            float u[kRows][kAcross];
            unsigned sc[kRows][kAcross];
#pragma unroll
            for (int j = 0; j < kRows; j++) {
                const int r = r0 + j * nwarps;
                const bool ok = r < dr.y && (Inside || static_cast<unsigned>(gy0 + r) < static_cast<unsigned>(im.H));
                const long long px = static_cast<long long>(r) * im.W;
                load_pieces<UReady, 0>(sc[j], u[j], pm0 + px, pd0 + px, pg0 + static_cast<long long>(r) * im.g_pitch,
                                       Inside ? 0 : first, ok ? (Inside ? stored : past) : 0);
            }
#pragma unroll
            for (int j = 0; j < kRows; j++) {
                const int r = r0 + j * nwarps;
                if (r >= dr.y) break;
                const unsigned at = (r & 1) * plane + (r >> 1) * pitch + c;
                const unsigned pf = s_f + 4 * at, ps = s_s + at;
#pragma unroll
                for (int i = 0; i < kAcross; i++) {
                    const float v = u[j][i] * lds1(rv + 4 * sc[j][i]);
                    bad |= !(fabsf(v) <= FLT_MAX);
                    if (i < stored) {
                        asm volatile("st.shared.u8 [%0], %1;" ::"r"(ps + 32 * i), "r"(sc[j][i]) : "memory");
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(pf + 128 * i), "f"(v) : "memory");
                    }
                }
            }
        }
    }
    return bad;
}

// Masking zeroes the direction's field where s* = s - 1 (smaller scales are zero since their own pass): the cells of
// every 4-cell word from the rectangle's first cell to its last in each row plane, as one flat range over all threads.
// Only the excluded cells are stored to: reading and writing back whole words (16 bytes of 4 cells) costs 8
// shared-memory wavefronts a warp where these stores cost one or two each, although it can skip the cells a scale's
// kernel does not reach (1024^2: 471 us so, 464 us with stores alone).  The cells beside the rectangle in those rows
// and those outside this direction's region hold stale values, which no correlation reads.
struct MaskRange {
    int w0[2], w1[2];  // words [w0, w1) of the even and the odd plane
    __device__ __forceinline__ MaskRange(const int4 dr, int pitch, int plane) {
        const int e0 = (dr.x + 1) >> 1, e1 = (dr.y + 1) >> 1, o0 = dr.x >> 1, o1 = dr.y >> 1;
        w0[0] = (e0 * pitch + dr.z) >> 2;
        w1[0] = e1 > e0 ? ((e1 - 1) * pitch + dr.w + 3) >> 2 : w0[0];
        w0[1] = (plane + o0 * pitch + dr.z) >> 2;
        w1[1] = o1 > o0 ? (plane + (o1 - 1) * pitch + dr.w + 3) >> 2 : w0[1];
    }
};

// Zeroes the cells (16 bytes at f4) of a word of selected scales v that equal the byte `excluded` repeats: a byte's
// top bit stays exactly where it differs (scales are below 0x80).
template <int Offset>
__device__ __forceinline__ void mask_word(unsigned v, unsigned f4, unsigned excluded) {
    const unsigned keep = ((v ^ excluded) | 0x80808080u) - 0x01010101u;
    asm volatile(
        "{\n\t.reg .pred p0, p1, p2, p3;\n\t.reg .b32 t0, t1, t2, t3;\n\t"
        "and.b32 t0, %1, 0x80;\n\tand.b32 t1, %1, 0x8000;\n\tand.b32 t2, %1, 0x800000;\n\tand.b32 t3, %1, 0x80000000;\n\t"
        "setp.eq.u32 p0, t0, 0;\n\tsetp.eq.u32 p1, t1, 0;\n\tsetp.eq.u32 p2, t2, 0;\n\tsetp.eq.u32 p3, t3, 0;\n\t"
        "@p0 st.shared.b32 [%0 + %2], 0;\n\t@p1 st.shared.b32 [%0 + %2 + 4], 0;\n\t@p2 st.shared.b32 [%0 + %2 + 8], 0;\n\t"
        "@p3 st.shared.b32 [%0 + %2 + 12], 0;\n\t}" ::"r"(f4),
        "r"(keep), "n"(Offset)
        : "memory");
}

// A thread's words of both planes, held in registers over a direction's scales where the range has no more than
// kHeldWords a thread (sets of radius 31: 95 rows of 191 cells are 2,300 words a plane; 1024^2 464 us with the words
// read again for every scale, 452 us so).
constexpr int kHeldWords = 5;
template <int Threads>
struct HeldWords {
    unsigned v[2][kHeldWords];
    static __device__ __forceinline__ bool fits(const MaskRange &m) {
        return m.w1[0] - m.w0[0] <= kHeldWords * Threads && m.w1[1] - m.w0[1] <= kHeldWords * Threads;
    }
    __device__ __forceinline__ void load(const MaskRange &m, unsigned s_s, int tid) {
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int j = 0; j < kHeldWords; j++) {
                v[p][j] = 0xffffffffu;  // no scale
                const int w = m.w0[p] + tid + j * Threads;
                if (w < m.w1[p]) v[p][j] = lds_u1(s_s + 4 * w);
            }
    }
    __device__ __forceinline__ void mask(const MaskRange &m, unsigned s_f, int tid, unsigned excluded) const {
        static_assert(kHeldWords == 5, "one mask_word per word");
#pragma unroll
        for (int p = 0; p < 2; p++) {
            const unsigned f4 = s_f + 16 * (m.w0[p] + tid);
            mask_word<0>(v[p][0], f4, excluded);
            mask_word<16 * Threads>(v[p][1], f4, excluded);
            mask_word<32 * Threads>(v[p][2], f4, excluded);
            mask_word<48 * Threads>(v[p][3], f4, excluded);
            mask_word<64 * Threads>(v[p][4], f4, excluded);
        }
    }
};
// Ranges of more words: read again for every scale.
__device__ __forceinline__ void mask_read(const MaskRange &m, unsigned s_f, unsigned s_s, int tid, int nthreads, unsigned excluded) {
    for (int p = 0; p < 2; p++)
        for (int w = m.w0[p] + tid; w < m.w1[p]; w += nthreads) mask_word<0>(lds_u1(s_s + 4 * w), s_f + 16 * w, excluded);
}

// The float2 at shared address a of CTA `rank` of the cluster.
__device__ __forceinline__ float2 cluster_lds2(unsigned a, unsigned rank) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(cluster_addr(a, rank)) : "memory");
    return v;
}

template <int WX, int WY, bool Single>
__global__ void __launch_bounds__(GatherShape<WX, WY, Single>::kThreads, 1)
    lpaici_adjoint_gather_kernel(const __grid_constant__ GatherArgs a) {
    using Shape = GatherShape<WX, WY, Single>;
    constexpr int Q = kGatherQ, nthreads = Shape::kThreads, kGroups = Shape::kGroups, kEntry = Shape::kEntry;
    extern __shared__ __align__(16) int smem[];
    const int nk = a.D * a.S;
    const int pieces = Shape::kPieces ? a.pieces : nk;
    const GatherSmem lay = GatherSmem::make(nk, kEntry, pieces, a.block_bytes, a.plane, Shape::kRegion, kGroups);
    char *base = reinterpret_cast<char *>(smem);
    uint2 *s_tab = reinterpret_cast<uint2 *>(base);
    float *s_rv = reinterpret_cast<float *>(base + lay.rv);
    int *s_flag = reinterpret_cast<int *>(base + lay.flag);
    // the field of the current direction and s*(d, .) on the halo'd tile, as shared addresses (loads and stores
    // through pointers cost an address computation each)
    const unsigned s_f = smem_addr(base + lay.field), s_s = smem_addr(base + lay.smap);
    // the rest's CTAs may start once every CTA of this launch has (they depend on nothing of it)
    if (a.rest_follows) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int rank = a.cluster > 1 ? static_cast<int>(blockIdx.x % a.cluster) : 0;
    int tile = a.first_tile + blockIdx.x / a.cluster;
    GatherImage im;
    if (a.images) {
        const int2 it = a.items[tile];
        im = a.images[it.x];
        tile = it.y;
    } else {
        im = a.single;
    }
    const float *rvar_k = a.images ? im.rvar : a.rvar;
    const int x0 = (tile % im.tiles_x) * Shape::kTW, y0 = (tile / im.tiles_x) * Shape::kTH;
    const int gx0 = x0 - a.R, gy0 = y0 - a.R;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = nthreads >> 5;
    // the same in every lane of a warp: reduced, the compiler knows it warp-uniform
    const int group = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(tid / Shape::kRegion));
    const int gtid = tid % Shape::kRegion;
    const int gwarp = gtid >> 5;
    const int ty = (gwarp / WX) * 32 + 2 * (lane & 15), tx = (gwarp % WX) * 32 + (lane >> 4) * Q;
    const unsigned lane_base = s_f + 4 * ((ty >> 1) * a.pitch + tx);
    // from a cell to the one a row down, from the even and from the odd rows' plane
    [[maybe_unused]] const int to_odd = 4 * a.plane, to_even = 4 * (a.pitch - a.plane);
    const unsigned blocks = smem_addr(base + lay.block);

    for (int i = tid; i < kEntry / 2 * (pieces + 1); i += nthreads) s_tab[i] = __ldg(reinterpret_cast<const uint2 *>(a.blob) + i);
    for (int k = tid; k < nk; k += nthreads) s_rv[k] = rvar_k[k];
    if (tid < 2) s_flag[tid] = 0;
    __syncthreads();
    // piece q's block to shared memory, asynchronously, into block buffer q & 1
    auto stage = [&](int q) {
        const unsigned from = s_tab[kEntry / 2 * q].x & ~15u, bytes = (s_tab[kEntry / 2 * (q + 1)].x & ~15u) - from;
        const unsigned dst = blocks + (q & 1) * a.block_bytes;
        const char *src = reinterpret_cast<const char *>(a.blob) + from;
        for (unsigned o = 16 * tid; o < bytes; o += 16 * nthreads)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + o), "l"(src + o) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const int per_chunk = (a.D + kGatherChunks - 1) / kGatherChunks;
    const int chunks = kGatherChunks / a.cluster;  // of this CTA
    const int d_begin = min(a.D, rank * chunks * per_chunk), d_end = min(a.D, (rank + 1) * chunks * per_chunk);
    const auto first_piece = [&](int d) { return Shape::kPieces ? a.first_piece[d] : d * a.S; };
    const int q_end = first_piece(d_end);
    if (d_begin < d_end) stage(first_piece(d_begin));

    float2 acc[Q];
    // sums of this thread's outputs, pair i at [i * kRegion]: over all chunks (one CTA per tile), else the
    // sums of this CTA's first chunk
    constexpr int slot = Q * Shape::kRegion;  // float2 of one group's sums
    float2 *s_sum = reinterpret_cast<float2 *>(base + lay.sums) + group * slot + gtid;
#pragma unroll
    for (int i = 0; i < Q; i++) {
        acc[i] = make_float2(0.0f, 0.0f);
        s_sum[i * Shape::kRegion] = acc[i];
    }

    int d = d_begin;
#pragma unroll 1
    for (int c = 0; c < chunks; c++) {
        const int d_stop = min(d_end, d_begin + (c + 1) * per_chunk);
#pragma unroll 1
        for (; d < d_stop; d++) {
            __syncthreads();  // the previous direction's correlations are done with the field
            const uint8_t *map = im.smap + static_cast<size_t>(d) * im.H * im.W;
            const unsigned rv_d = smem_addr(s_rv + d * a.S);
            const int4 dr = a.drect[d];
            const bool inside = gx0 + dr.z >= 0 && gx0 + dr.w <= im.W && gy0 + dr.x >= 0 && gy0 + dr.y <= im.H;
            bool bad;
            if (im.u_ready)
                bad = inside ? build_field<true, true>(s_f, s_s, rv_d, im, map, dr, gx0, gy0, a.pitch, a.plane, warp, nwarps, lane)
                             : build_field<true, false>(s_f, s_s, rv_d, im, map, dr, gx0, gy0, a.pitch, a.plane, warp, nwarps, lane);
            else
                bad = build_field<false, false>(s_f, s_s, rv_d, im, map, dr, gx0, gy0, a.pitch, a.plane, warp, nwarps, lane);
            if (bad) s_flag[d & 1] = 1;
            HeldWords<nthreads> held;
            const int q_begin = first_piece(d), n = Shape::kPieces ? first_piece(d + 1) - q_begin : a.S;
#pragma unroll 1
            for (int i = 0; i < n; i++) {
                // (a scale of several pieces is masked again for each, which changes nothing)
                const int q = q_begin + i, s = Shape::kPieces ? static_cast<int>(s_tab[kEntry / 2 * q].x & 15u) : i;
                if (i > 0) __syncthreads();  // every correlation of the previous piece is done with the field
                if (q + 1 < q_end)
                    stage(q + 1);
                else
                    asm volatile("cp.async.commit_group;" ::: "memory");
                if (s > 0) {
                    const MaskRange range(dr, a.pitch, a.plane);
                    const unsigned excluded = 0x01010101u * static_cast<unsigned>(s - 1);
                    if (HeldWords<nthreads>::fits(range)) {
                        if (s == 1) held.load(range, s_s, tid);
                        held.mask(range, s_f, tid, excluded);
                    } else {
                        mask_read(range, s_f, s_s, tid, nthreads, excluded);
                    }
                }
                asm volatile("cp.async.wait_group 1;" ::: "memory");  // this piece's block has landed
                __syncthreads();
                const bool finite = s_flag[d & 1] == 0;
                if (i == 0 && tid == 0) s_flag[(d + 1) & 1] = 0;  // last read before this direction's first barrier
                const unsigned block = blocks + (q & 1) * a.block_bytes;
                // the group's units: one stream, the next unit behind the weights of the one before
                const unsigned ends = s_tab[kEntry / 2 * q].y;
                unsigned at, last;
                if constexpr (kGroups == 2) {
                    at = block + (group == 0 ? 0 : 8 * (ends & 0xffffu));
                    last = block + 8 * (group == 0 ? ends & 0xffffu : ends >> 16);
                } else {
                    const unsigned more = s_tab[kEntry / 2 * q + 1].x;
                    const unsigned e0 = ends & 0xffffu, e1 = ends >> 16, e2 = more & 0xffffu, e3 = more >> 16;
                    at = block + 8 * (group < 2 ? (group == 0 ? 0 : e0) : (group == 2 ? e1 : e2));
                    last = block + 8 * (group < 2 ? (group == 0 ? e0 : e1) : (group == 2 ? e2 : e3));
                }
                if constexpr (Single) {  // no padding taps: infinities and NaNs need no other loop
#pragma unroll 1
                    while (at != last) {
                        const uint2 u = lds_u2(at);
                        const unsigned h = u.y & 3u, end = at + (u.y & ~7u), row = lane_base + u.x;
                        single_unit(acc, row, row + ((u.y & 4u) ? to_even : to_odd), h, at + 8, end);
                        at = end;
                    }
                } else if (finite) {
#pragma unroll 1
                    while (at != last) {
                        const uint2 u = lds_u2(at);
                        const unsigned h = u.y & 3u, end = at + u.y - h;
                        gather_unit(acc, lane_base + u.x, h, at + 8, end);
                        at = end;
                    }
                } else {
                    float2 tmp[Q];
#pragma unroll
                    for (int i = 0; i < Q; i++) tmp[i] = acc[i];
#pragma unroll 1
                    while (at != last) {
                        const uint2 u = lds_u2(at);
                        gather_run_skipping(tmp, lane_base + u.x - 4 * (u.y & 3u), at + 8, (u.y - 8) / 8);
                        at += u.y & ~3u;
                    }
#pragma unroll
                    for (int i = 0; i < Q; i++) acc[i] = tmp[i];
                }
            }
        }
        if (a.cluster == 1 || c == 0) {
#pragma unroll
            for (int i = 0; i < Q; i++) {
                const float2 t = s_sum[i * Shape::kRegion];
                s_sum[i * Shape::kRegion] = make_float2(t.x + acc[i].x, t.y + acc[i].y);
                if (c + 1 < chunks) acc[i] = make_float2(0.0f, 0.0f);
            }
        }
    }
    __syncthreads();  // every sum is there, and the field is free
    if (a.cluster == 1) {
        if (group == 0) {
#pragma unroll
            for (int i = 0; i < Q; i++) {
                float2 t = s_sum[i * Shape::kRegion];
#pragma unroll
                for (int g = 1; g < kGroups; g++) {
                    const float2 other = s_sum[g * slot + i * Shape::kRegion];
                    t = make_float2(t.x + other.x, t.y + other.y);
                }
                acc[i] = t;
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int oy = y0 + ty + h;
                if (oy >= im.H) break;
                float *o = im.grad + static_cast<size_t>(oy) * im.grad_pitch + x0 + tx;
#pragma unroll
                for (int i = 0; i < Q; i++)
                    if (x0 + tx + i < im.W) o[i] = h == 0 ? acc[i].x : acc[i].y;
            }
        }
        return;
    }
    // a cluster: the second chunk's sums go over the field; every CTA adds its share of the tile's outputs
    // over all CTAs
    float2 *s_second = reinterpret_cast<float2 *>(smem);
    if (chunks == 2) {
#pragma unroll
        for (int i = 0; i < Q; i++) s_second[group * slot + i * Shape::kRegion + gtid] = acc[i];
    }
    cluster_barrier();
    const int share = slot / a.cluster;
    const unsigned part[2] = {smem_addr(base + lay.sums), smem_addr(s_second)};
    for (int e = rank * share + tid; e < (rank + 1) * share; e += nthreads) {
        float2 sum[kGroups];
#pragma unroll
        for (int g = 0; g < kGroups; g++) {
            sum[g] = make_float2(0.0f, 0.0f);
            for (int c = 0; c < kGatherChunks; c++) {
                const float2 v = cluster_lds2(part[c % chunks] + 8 * (g * slot + e), c / chunks);
                sum[g] = make_float2(sum[g].x + v.x, sum[g].y + v.y);
            }
        }
#pragma unroll
        for (int g = 1; g < kGroups; g++) sum[0] = make_float2(sum[0].x + sum[g].x, sum[0].y + sum[g].y);
        const int t = e % Shape::kRegion, m = e / Shape::kRegion, w = t >> 5, l = t & 31;
        const int ox = x0 + (w % WX) * 32 + (l >> 4) * Q + m, oy = y0 + (w / WX) * 32 + 2 * (l & 15);
        if (ox < im.W && oy < im.H) {
            float *o = im.grad + static_cast<size_t>(oy) * im.grad_pitch + ox;
            o[0] = sum[0].x;
            if (oy + 1 < im.H) o[im.grad_pitch] = sum[0].y;
        }
    }
    cluster_barrier();  // a CTA's shared memory stays until every other one has read it
    // what follows in the stream follows the launch before this one too
    if (blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <bool Single>
const void *gather_fn_of(const AdjointLayout &L) {
    return L.wx == 2   ? reinterpret_cast<const void *>(lpaici_adjoint_gather_kernel<2, 1, Single>)
           : L.wy == 1 ? reinterpret_cast<const void *>(lpaici_adjoint_gather_kernel<4, 1, Single>)
                       : reinterpret_cast<const void *>(lpaici_adjoint_gather_kernel<4, 2, Single>);
}
const void *gather_fn(const AdjointLayout &L) { return L.single ? gather_fn_of<true>(L) : gather_fn_of<false>(L); }

int gather_groups(const AdjointLayout &L) { return AdjointLayout::groups(L.wx, L.wy, L.single); }
int gather_threads(const AdjointLayout &L) { return gather_groups(L) * 32 * L.wx * L.wy; }

// How a launch's tiles are gathered: the first n_single by one CTA each, the others by clusters of `cluster`.
struct GatherPlan {
    long tiles = 0, n_single = 0;
    int cluster = 1;
};

int gather_launch(const AdjointLayout &L, const GatherArgs &args, const GatherPlan &plan, size_t smem, cudaStream_t stream) {
    GatherArgs ga = args;
    void *params[] = {&ga};
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(gather_threads(L));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    const long rest = plan.tiles - plan.n_single;
    if (plan.n_single > 0) {
        ga.cluster = 1;
        ga.first_tile = 0;
        ga.rest_follows = rest > 0 ? 1 : 0;
        cfg.gridDim = dim3(static_cast<unsigned>(plan.n_single));
        const cudaError_t e = cudaLaunchKernelExC(&cfg, gather_fn(L), params);
        if (e != cudaSuccess) return cuda_error(e, "adjoint gather launch");
    }
    if (rest > 0) {
        ga.cluster = plan.cluster;
        ga.first_tile = static_cast<int>(plan.n_single);
        ga.rest_follows = 0;
        cfg.gridDim = dim3(static_cast<unsigned>(rest * plan.cluster));
        cudaLaunchAttribute attr[2] = {};
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = static_cast<unsigned>(plan.cluster);
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = plan.n_single > 0 ? 2 : 1;
        const cudaError_t e = cudaLaunchKernelExC(&cfg, gather_fn(L), params);
        if (e != cudaSuccess) return cuda_error(e, "adjoint gather launch (clusters)");
    }
    return LPAICI_OK;
}

// Fills the geometry and the directions' rectangles of the field; smem receives the dynamic shared
// memory of one CTA per tile, checked against the device.
int gather_setup(const lpaici_kernelset *ks, const int *adj_blob, GatherArgs *ga, size_t *smem) {
    const AdjointLayout &L = ks->adj_layout;
    const int nk = ks->D * ks->S, tw = 32 * L.wx, th = 32 * L.wy;
    int dev = 0, max_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (L.limit_bytes > static_cast<size_t>(max_optin))
        return set_error(LPAICI_ERR_UNSUPPORTED, "adjoint tile needs %zu B of shared memory, device allows %d",
                         L.limit_bytes, max_optin);
    ga->D = ks->D;
    ga->S = ks->S;
    ga->R = ks->radius;
    ga->blob = adj_blob;
    ga->pieces = L.pieces;
    std::copy(L.first_piece.begin(), L.first_piece.end(), ga->first_piece);
    ga->block_bytes = L.block_bytes;
    ga->pitch = L.pitch;
    ga->plane = L.plane;
    const GatherSmem m = GatherSmem::make(nk, AdjointLayout::entry_words(gather_groups(L)), L.pieces, L.block_bytes, L.plane, 32 * L.wx * L.wy, gather_groups(L));
    *smem = m.total;
    if (*smem > static_cast<size_t>(max_optin))
        return set_error(LPAICI_ERR_UNSUPPORTED, "adjoint tile needs %zu B of shared memory, device allows %d", *smem,
                         max_optin);
    const int rows = th + 2 * ga->R;
    for (int d = 0; d < ks->D; d++) {
        // a lane reads rows ty + R + j for field rows j of its two output rows (ty + 1 < th) and columns
        // tx + R + dx + [0, Q) (tx + Q <= tile width): rows [R + dy_min, R + th + dy_max), columns
        // [R + dx_min, R + tile width + dx_max)
        int4 u = make_int4(0, 0, 0, 0);
        for (int s = 0; s < ks->S; s++) {
            const int *box = &L.box[4 * (static_cast<size_t>(d) * ks->S + s)];
            if (box[1] < box[0]) continue;
            const int4 r = make_int4(std::max(0, ga->R + box[0]), std::min(rows, ga->R + th + box[1]),
                                     std::max(0, ga->R + box[2]), std::min(ga->pitch, ga->R + tw + box[3]));
            u = u.y <= u.x ? r : make_int4(std::min(u.x, r.x), std::max(u.y, r.y), std::min(u.z, r.z), std::max(u.w, r.w));
        }
        ga->drect[d] = u;
    }
    return LPAICI_OK;
}

// CTAs per tile: one for whole waves of tiles, for the rest as many as shorten the launch.  A tile's time goes
// with its share of the directions, plus about 8.5 us for the cluster's exchange and staging; a cluster needs its
// CTAs free at once in one GPC: 33 clusters of four or 15 of eight run together on 148 SMs.  The tile's time is
// fitted to the symmetric (475 us), tapered (706 us) and 8 x 4 (74 us) sets.
// Measured (16 x 7 symmetric set, us for 1 / 4 / 8 CTAs per tile): 15 tiles 473 / 129 / 70, 32 tiles
// 475 / 130 / 201, 40 tiles 475 / 254 / 203, 128 tiles 475 / 505 / 599, 160 tiles 947 / 629 / 732.
int gather_plan(const lpaici_kernelset *ks, long tiles, GatherPlan *plan) {
    const AdjointLayout &L = ks->adj_layout;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    *plan = GatherPlan{tiles, tiles, 1};
    const double tile_us = ks->D * (1.8 + 1.27 * ks->S) + (L.single ? 0.037 * L.taps + 0.1 * L.units : 0.0354 * L.taps + 0.046 * L.units);
    double best = static_cast<double>((tiles + sms - 1) / sms);
    const GatherSmem m = GatherSmem::make(ks->D * ks->S, AdjointLayout::entry_words(gather_groups(L)), L.pieces, L.block_bytes, L.plane, 32 * L.wx * L.wy, gather_groups(L));
    for (const int c : {kGatherChunks / 2, kGatherChunks}) {
        // the second chunk's sums of half as many CTAs lie over everything before the first one's
        if (c < kGatherChunks && m.sums < m.total - m.sums) continue;
        if (ks->D < c || tiles * c > 0x7fffffffL) continue;
        const long slots = std::max(1, (sms - 4 - 3 * c) / c);
        for (const long waves : {0L, tiles / sms}) {
            const long rest = tiles - waves * sms;
            const double t = waves + (1.0 / c + 8.5 / tile_us) * static_cast<double>((rest + slots - 1) / slots);
            if (rest > 0 && t < best) {
                best = t;
                *plan = GatherPlan{tiles, waves * sms, c};
            }
        }
    }
    const cudaError_t e = allow_shared_memory(gather_fn(L));
    return e == cudaSuccess ? LPAICI_OK : cuda_error(e, "adjoint gather attributes");
}

long gather_tiles(const AdjointLayout &L, int width, int height, int *tiles_x) {
    *tiles_x = (width + 32 * L.wx - 1) / (32 * L.wx);
    return static_cast<long>(*tiles_x) * ((height + 32 * L.wy - 1) / (32 * L.wy));
}

}  // namespace

int gather_pass(const lpaici_kernelset *ks, const int *adj_blob, const uint8_t *smap, const float *rden,
                const float *d_grad_out, int gout_pitch, float *d_grad_in, int gin_pitch, int width, int height,
                float sigma, bool u_ready, cudaStream_t stream);

// The two passes over caller-provided storage (lpaici_backward, lpaici_backward_noalloc).
int adjoint_passes(const lpaici_kernelset *ks, const int *blob, const int *adj_blob, uint8_t *smap, float *rden,
                   const float *d_noisy, int noisy_pitch, const float *d_grad_out, int gout_pitch, float *d_grad_in,
                   int gin_pitch, int width, int height, float sigma, float gamma, cudaStream_t stream) {
    int tiles_x = 0;
    if (gather_tiles(ks->adj_layout, width, height, &tiles_x) > 0x7fffffffL)
        return set_error(LPAICI_ERR_UNSUPPORTED, "image too large: %d x %d", width, height);

    // A. selection
    ImageArgs img{};
    img.in = d_noisy;
    img.out = nullptr;
    img.smap = smap;
    img.rden = rden;
    img.g = d_grad_out;
    img.g_pitch = gout_pitch;
    img.W = width;
    img.in_h = height;
    img.in_pitch = noisy_pitch;
    img.out_pitch = width;
    img.row_begin = 0;
    img.rows_out = height;
    KernelTables tab;
    fill_tables(ks, nullptr, sigma, gamma, &tab);
    tab.blob = blob;
    int rc = launch_forward(img, tab, plan_for(ks, width, height), stream);
    if (rc != LPAICI_OK) return rc;
    // B. gather
    return gather_pass(ks, adj_blob, smap, rden, d_grad_out, gout_pitch, d_grad_in, gin_pitch, width, height, sigma,
                       true, stream);
}

// Pass B alone, from the s* planes and 1/den of the image (pass A's outputs or a kept state), or u = g / den
// in place of 1/den (u_ready).
int gather_pass(const lpaici_kernelset *ks, const int *adj_blob, const uint8_t *smap, const float *rden,
                const float *d_grad_out, int gout_pitch, float *d_grad_in, int gin_pitch, int width, int height,
                float sigma, bool u_ready, cudaStream_t stream) {
    GatherArgs ga{};
    size_t smem = 0;
    int rc = gather_setup(ks, adj_blob, &ga, &smem);
    if (rc != LPAICI_OK) return rc;
    int tiles_x = 0;
    const long tiles = gather_tiles(ks->adj_layout, width, height, &tiles_x);
    if (tiles > 0x7fffffffL) return set_error(LPAICI_ERR_UNSUPPORTED, "image too large: %d x %d", width, height);
    GatherPlan plan;
    rc = gather_plan(ks, tiles, &plan);
    if (rc != LPAICI_OK) return rc;
    KernelTables tab;
    fill_tables(ks, nullptr, sigma, 1.0f, &tab);
    ga.single = GatherImage{d_grad_out, smap, rden, d_grad_in, nullptr, gout_pitch, gin_pitch, width, height, tiles_x,
                            u_ready ? 1 : 0};
    for (int k = 0; k < ks->D * ks->S; k++) ga.rvar[k] = 1.0f / tab.var[k];
    return gather_launch(ks->adj_layout, ga, plan, smem, stream);
}

namespace {

// The adjoint's workspace comes from a stream-ordered memory pool owned by this library, one per
// device, that keeps freed memory for the next call (release threshold: never).  The device's default
// pool returns memory to the driver at every synchronisation, so a caller that synchronises between
// calls would map the workspace afresh each time (about 20 bytes per pixel: tens of ms at 8192^2).
constexpr int kMaxPoolDevices = 64;
std::mutex g_pool_lock;
cudaMemPool_t g_pools[kMaxPoolDevices];

int workspace_pool(cudaMemPool_t *out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_error(e, "cudaGetDevice");
    if (dev < 0 || dev >= kMaxPoolDevices)
        return set_error(LPAICI_ERR_UNSUPPORTED, "device %d beyond %d", dev, kMaxPoolDevices);
    std::lock_guard<std::mutex> hold(g_pool_lock);
    if (!g_pools[dev]) {
        int supported = 0;
        cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, dev);
        if (!supported)
            return set_error(LPAICI_ERR_UNSUPPORTED,
                             "device %d has no stream-ordered memory pools: use lpaici_backward_noalloc", dev);
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        e = cudaMemPoolCreate(&pool, &props);
        if (e != cudaSuccess) return cuda_error(e, "cudaMemPoolCreate(adjoint workspace)");
        uint64_t keep = ~uint64_t(0);
        e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            return cuda_error(e, "cudaMemPoolSetAttribute(adjoint workspace)");
        }
        g_pools[dev] = pool;
    }
    *out = g_pools[dev];
    return LPAICI_OK;
}

}  // namespace

int check_adjoint_params(const lpaici_kernelset *ks, float sigma, const float *gamma, const char *who) {
    if (!(sigma > 0.0f) || !std::isfinite(sigma) || (gamma && (!(*gamma > 0.0f) || !std::isfinite(*gamma))))
        return set_error(LPAICI_ERR_INVALID_ARG, "%s: sigma and gamma need finite positive numbers", who);
    if (ks->S > kMaxScales)
        return set_error(LPAICI_ERR_UNSUPPORTED, "%s: %d scales per direction; the adjoint supports at most %d", who,
                         ks->S, kMaxScales);
    return LPAICI_OK;
}

}  // namespace lpaici

using namespace lpaici;

extern "C" int lpaici_trim_workspace(void) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_error(e, "cudaGetDevice");
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> hold(g_pool_lock);
        if (dev >= 0 && dev < kMaxPoolDevices) pool = g_pools[dev];
    }
    if (!pool) return LPAICI_OK;
    e = cudaMemPoolTrimTo(pool, 0);
    return e == cudaSuccess ? LPAICI_OK : cuda_error(e, "cudaMemPoolTrimTo(adjoint workspace)");
}

extern "C" int lpaici_backward(const lpaici_kernelset *ks, const float *d_noisy, int noisy_pitch,
                               const float *d_grad_out, int gout_pitch, float *d_grad_in, int gin_pitch, int width,
                               int height, float sigma, float gamma, lpaici_stream_t stream_) {
    if (!ks || !d_noisy || !d_grad_out || !d_grad_in)
        return set_error(LPAICI_ERR_INVALID_ARG, "lpaici_backward: null argument");
    if (width <= 0 || height <= 0 || noisy_pitch < width || gout_pitch < width || gin_pitch < width)
        return set_error(LPAICI_ERR_INVALID_ARG, "lpaici_backward: bad size or pitch");
    int rc = check_adjoint_params(ks, sigma, &gamma, "lpaici_backward");
    if (rc != LPAICI_OK) return rc;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    const int *blob = nullptr, *adj = nullptr;
    rc = device_blob(ks, &blob);
    if (rc == LPAICI_OK) rc = device_adj_blob(ks, &adj);
    if (rc != LPAICI_OK) return rc;

    // transient workspace: D selection planes (bytes) and g/den (floats)
    cudaMemPool_t pool = nullptr;
    rc = workspace_pool(&pool);
    if (rc != LPAICI_OK) return rc;
    const size_t npx = static_cast<size_t>(width) * height;
    void *ws = nullptr;
    const size_t smap_bytes = (static_cast<size_t>(ks->D) * npx + 255) & ~size_t(255);
    cudaError_t e = cudaMallocFromPoolAsync(&ws, smap_bytes + sizeof(float) * npx, pool, stream);
    if (e != cudaSuccess) return cuda_error(e, "cudaMallocFromPoolAsync(adjoint workspace)");
    uint8_t *smap = static_cast<uint8_t *>(ws);
    float *rden = reinterpret_cast<float *>(static_cast<char *>(ws) + smap_bytes);
    rc = adjoint_passes(ks, blob, adj, smap, rden, d_noisy, noisy_pitch, d_grad_out, gout_pitch, d_grad_in, gin_pitch,
                        width, height, sigma, gamma, stream);
    cudaError_t ef = cudaFreeAsync(ws, stream);
    if (rc == LPAICI_OK && ef != cudaSuccess) rc = cuda_error(ef, "cudaFreeAsync(adjoint workspace)");
    return rc;
}

// ---------------------------------------------------------------------------------------------
// Batched adjoint plan.
// ---------------------------------------------------------------------------------------------
struct lpaici_backward_batch {
    int device = -1;
    lpaici_batch *select = nullptr;  // pass A: the forward batch plan (out = null, s* and g/den on)
    void *dev_mem = nullptr;         // s* planes | g/den maps | GatherImage[n] | 1/v tables | items
    GatherArgs ga{};
    size_t smem = 0;
    AdjointLayout layout;
    GatherPlan plan;
    bool use_graph = false;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
};

namespace {

int backward_batch_enqueue(lpaici_backward_batch *b, cudaStream_t stream) {
    int rc = batch_plan_enqueue(b->select, stream);
    if (rc != LPAICI_OK) return rc;
    return gather_launch(b->layout, b->ga, b->plan, b->smem, stream);
}

void backward_batch_free(lpaici_backward_batch *b) {
    if (!b) return;
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    batch_plan_free(b->select);
    if (b->dev_mem) cudaFree(b->dev_mem);
    delete b;
}

size_t align256(size_t n) { return (n + 255) & ~size_t(255); }

}  // namespace

extern "C" int lpaici_backward_batch_create(const lpaici_kernelset *ks, const lpaici_grad_image *images, int n,
                                            const lpaici_batch_options *opts, lpaici_stream_t stream_,
                                            lpaici_backward_batch **out) {
    if (!ks || !images || n <= 0 || !out)
        return set_error(LPAICI_ERR_INVALID_ARG, "lpaici_backward_batch_create: bad argument");
    *out = nullptr;
    for (int i = 0; i < n; i++) {
        const lpaici_grad_image &im = images[i];
        if (!im.noisy || !im.grad_out || !im.grad_in || im.width <= 0 || im.height <= 0 || im.noisy_pitch < im.width ||
            im.gout_pitch < im.width || im.gin_pitch < im.width)
            return set_error(LPAICI_ERR_INVALID_ARG, "adjoint batch image %d: bad pointer, size or pitch", i);
        const int rc = check_adjoint_params(ks, im.sigma, &im.gamma, "lpaici_backward_batch_create");
        if (rc != LPAICI_OK) return rc;
    }
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    const int *adj = nullptr;
    int rc = device_adj_blob(ks, &adj);
    if (rc != LPAICI_OK) return rc;
    auto *b = new lpaici_backward_batch();
    cudaGetDevice(&b->device);
    b->layout = ks->adj_layout;
    rc = gather_setup(ks, adj, &b->ga, &b->smem);
    if (rc != LPAICI_OK) {
        backward_batch_free(b);
        return rc;
    }

    // plan memory: per image s* planes and g/den, then the gather's descriptors, tables and items
    const int nk = ks->D * ks->S;
    std::vector<size_t> smap_off(n), rden_off(n);
    std::vector<int> tiles_x(n);
    size_t off = 0;
    long total_tiles = 0;
    for (int i = 0; i < n; i++) {
        const size_t npx = static_cast<size_t>(images[i].width) * images[i].height;
        smap_off[i] = off;
        off = align256(off + static_cast<size_t>(ks->D) * npx);
        rden_off[i] = off;
        off = align256(off + sizeof(float) * npx);
        total_tiles += gather_tiles(ks->adj_layout, images[i].width, images[i].height, &tiles_x[i]);
    }
    if (total_tiles > 0x7fffffffL) {
        backward_batch_free(b);
        return set_error(LPAICI_ERR_UNSUPPORTED, "adjoint batch too large: %ld tiles", total_tiles);
    }
    const size_t desc_off = off;
    off = align256(off + sizeof(GatherImage) * n);
    const size_t rvar_off = off;
    off = align256(off + sizeof(float) * static_cast<size_t>(n) * nk);
    const size_t item_off = off;
    off = align256(off + sizeof(int2) * static_cast<size_t>(total_tiles));
    cudaError_t e = cudaMalloc(&b->dev_mem, off);
    if (e != cudaSuccess) {
        backward_batch_free(b);
        return cuda_error(e, "cudaMalloc(adjoint batch plan)");
    }
    char *base = static_cast<char *>(b->dev_mem);
    std::vector<GatherImage> desc(n);
    std::vector<float> rvar(static_cast<size_t>(n) * nk);
    std::vector<int2> items;
    items.reserve(static_cast<size_t>(total_tiles));
    std::vector<BatchSpec> specs(n);
    for (int i = 0; i < n; i++) {
        const lpaici_grad_image &im = images[i];
        uint8_t *smap = reinterpret_cast<uint8_t *>(base + smap_off[i]);
        float *rden = reinterpret_cast<float *>(base + rden_off[i]);
        KernelTables tab;
        fill_tables(ks, nullptr, im.sigma, im.gamma, &tab);
        float *rv = rvar.data() + static_cast<size_t>(i) * nk;
        for (int k = 0; k < nk; k++) rv[k] = 1.0f / tab.var[k];
        desc[i] = GatherImage{im.grad_out, smap, rden, im.grad_in,
                              reinterpret_cast<const float *>(base + rvar_off) + static_cast<size_t>(i) * nk,
                              im.gout_pitch, im.gin_pitch, im.width, im.height, tiles_x[i], 1};
        int tx = 0;
        const long t = gather_tiles(ks->adj_layout, im.width, im.height, &tx);
        for (long j = 0; j < t; j++) items.push_back(make_int2(i, static_cast<int>(j)));
        specs[i] = BatchSpec{im.noisy, nullptr, smap, rden, im.width, im.height, im.noisy_pitch, im.width, im.sigma,
                             im.gamma, im.grad_out, im.gout_pitch};
    }
    e = cudaMemcpy(base + desc_off, desc.data(), sizeof(GatherImage) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(base + rvar_off, rvar.data(), sizeof(float) * rvar.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(base + item_off, items.data(), sizeof(int2) * items.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        backward_batch_free(b);
        return cuda_error(e, "cudaMemcpy(adjoint batch plan)");
    }
    b->ga.images = reinterpret_cast<const GatherImage *>(base + desc_off);
    b->ga.items = reinterpret_cast<const int2 *>(base + item_off);
    rc = gather_plan(ks, total_tiles, &b->plan);
    if (rc != LPAICI_OK) {
        backward_batch_free(b);
        return rc;
    }

    const int config = opts ? opts->tile_config : -1;
    rc = batch_plan_create(ks, specs.data(), n, config, false, stream, &b->select);
    if (rc != LPAICI_OK) {
        backward_batch_free(b);
        return rc;
    }
    b->use_graph = opts && opts->use_graph;
    if (b->use_graph) {
        cudaStream_t cap = nullptr;
        e = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            rc = backward_batch_enqueue(b, cap);
            const cudaError_t e2 = cudaStreamEndCapture(cap, &b->graph);
            if (rc == LPAICI_OK && e2 != cudaSuccess) rc = cuda_error(e2, "cudaStreamEndCapture");
            if (rc == LPAICI_OK) {
                e = cudaGraphInstantiate(&b->exec, b->graph, 0);
                if (e != cudaSuccess) rc = cuda_error(e, "cudaGraphInstantiate");
            }
        } else {
            rc = cuda_error(e, "graph capture");
        }
        if (cap) cudaStreamDestroy(cap);
        if (rc == LPAICI_OK) {
            e = cudaGraphUpload(b->exec, stream);
            if (e != cudaSuccess) rc = cuda_error(e, "cudaGraphUpload");
        }
        if (rc != LPAICI_OK) {
            backward_batch_free(b);
            return rc;
        }
    }
    *out = b;
    return LPAICI_OK;
}

extern "C" int lpaici_backward_batch_run(lpaici_backward_batch *b, lpaici_stream_t stream_) {
    if (!b) return set_error(LPAICI_ERR_INVALID_ARG, "lpaici_backward_batch_run: null plan");
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    int dev = -1;
    cudaGetDevice(&dev);
    if (dev != b->device)
        return set_error(LPAICI_ERR_INVALID_ARG, "adjoint batch planned on device %d, current device is %d", b->device,
                         dev);
    if (b->use_graph) {
        const cudaError_t e = cudaGraphLaunch(b->exec, stream);
        return e == cudaSuccess ? LPAICI_OK : cuda_error(e, "cudaGraphLaunch");
    }
    return backward_batch_enqueue(b, stream);
}

extern "C" int lpaici_backward_batch_destroy(lpaici_backward_batch *b) {
    if (b) {
        int cur = -1;
        cudaGetDevice(&cur);
        cudaSetDevice(b->device);
        cudaDeviceSynchronize();
        backward_batch_free(b);
        if (cur >= 0) cudaSetDevice(cur);
    }
    return LPAICI_OK;
}

// ---------------------------------------------------------------------------------------------
// Kept state: the forward stores what its adjoint needs, the adjoint runs the gather only.
// ---------------------------------------------------------------------------------------------
namespace {

size_t state_smap_bytes(const lpaici_kernelset *ks, int width, int height) {
    return (static_cast<size_t>(ks->D) * width * height + 255) & ~size_t(255);
}

int state_args(const lpaici_kernelset *ks, int width, int height, float sigma, const char *who) {
    if (!ks) return set_error(LPAICI_ERR_INVALID_ARG, "%s: null kernel set", who);
    if (width <= 0 || height <= 0) return set_error(LPAICI_ERR_INVALID_ARG, "%s: bad size %d x %d", who, width, height);
    return check_adjoint_params(ks, sigma, nullptr, who);
}

}  // namespace

extern "C" size_t lpaici_adjoint_state_bytes(const lpaici_kernelset *ks, int width, int height) {
    if (!ks || width <= 0 || height <= 0) return 0;
    return state_smap_bytes(ks, width, height) + sizeof(float) * static_cast<size_t>(width) * height;
}

extern "C" int lpaici_forward_state(const lpaici_kernelset *ks, const float *d_noisy, int noisy_pitch,
                                    float *d_denoised, int out_pitch, int width, int height, float sigma, float gamma,
                                    void *d_state, lpaici_stream_t stream_) {
    int rc = state_args(ks, width, height, sigma, "lpaici_forward_state");
    if (rc != LPAICI_OK) return rc;
    if (!d_noisy || !d_denoised || !d_state || noisy_pitch < width || out_pitch < width)
        return set_error(LPAICI_ERR_INVALID_ARG, "lpaici_forward_state: null pointer or bad pitch");
    rc = check_adjoint_params(ks, sigma, &gamma, "lpaici_forward_state");
    if (rc != LPAICI_OK) return rc;
    const int *blob = nullptr;
    rc = device_blob(ks, &blob);
    if (rc != LPAICI_OK) return rc;
    ImageArgs img{};
    img.in = d_noisy;
    img.out = d_denoised;
    img.smap = static_cast<uint8_t *>(d_state);
    img.rden = reinterpret_cast<float *>(static_cast<char *>(d_state) + state_smap_bytes(ks, width, height));
    img.W = width;
    img.in_h = height;
    img.in_pitch = noisy_pitch;
    img.out_pitch = out_pitch;
    img.row_begin = 0;
    img.rows_out = height;
    KernelTables tab;
    fill_tables(ks, nullptr, sigma, gamma, &tab);
    tab.blob = blob;
    return launch_forward(img, tab, plan_for(ks, width, height), reinterpret_cast<cudaStream_t>(stream_));
}

extern "C" int lpaici_backward_state(const lpaici_kernelset *ks, const void *d_state, const float *d_grad_out,
                                     int gout_pitch, float *d_grad_in, int gin_pitch, int width, int height, float sigma,
                                     lpaici_stream_t stream_) {
    int rc = state_args(ks, width, height, sigma, "lpaici_backward_state");
    if (rc != LPAICI_OK) return rc;
    if (!d_state || !d_grad_out || !d_grad_in || gout_pitch < width || gin_pitch < width)
        return set_error(LPAICI_ERR_INVALID_ARG, "lpaici_backward_state: null pointer or bad pitch");
    const int *adj = nullptr;
    rc = device_adj_blob(ks, &adj);
    if (rc != LPAICI_OK) return rc;
    const uint8_t *smap = static_cast<const uint8_t *>(d_state);
    const float *rden =
        reinterpret_cast<const float *>(static_cast<const char *>(d_state) + state_smap_bytes(ks, width, height));
    return gather_pass(ks, adj, smap, rden, d_grad_out, gout_pitch, d_grad_in, gin_pitch, width, height, sigma,
                       false, reinterpret_cast<cudaStream_t>(stream_));
}
