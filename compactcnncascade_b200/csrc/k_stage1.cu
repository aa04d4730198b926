// Stage-1 fully-convolutional net over every pyramid level, in two launches per frame.
//
// Reference: SIMD::ConvNeuralNetwork::Run (src/CNNObjectDetector/cnn_simd_cntk.cpp:640-963) with
// the plain CNNPP primitives (cnnpp_cplusplus.cpp): conv_4x4 (:92-157), lrelu_bn_max (:593-622),
// add/add2 (:916-950), conv_3x3 (:36-91), conv_5x4 (:158-187), lrelu_bn (:623-645),
// mulCN_add_tanhW (:646-672), mulC/mulC1_add (:952-984), tanhW (:673-690).
//
// front: one CTA of 128 threads per 32x16 tile of pooled L1 pixels of one level. The CTA resamples its
//        (67 x 35) input tile straight from the gray frame (the pyramid is never stored; a stored image is
//        read instead where the caller gives one; with the learned gate each warp resamples only the 7
//        rows of a strip of two pooled rows and runs on its own), runs the 4x4 conv + folded
//        BN/LReLU + 2x2 max for the 4 L1 maps and writes the 4 neighbour-map sums that L2 consumes
//        (S1 arena). Bound by the fp32 pipe (65 % busy with every SM full; independent chains of these packed
//        instructions alone reach 96 %, k_peak.cu) and the latency of the gray samples: 1.07 ms for the 83 levels
//        of a 3840x2160 frame at scale 1.05 (1.30 with 256-thread blocks and 25 % more instructions: the row
//        references once a tile instead of once a sample, both gray rows of a sample as one packed chain, two weights
//        a constant load), 36 us for the 13 of a 1080p frame (43.3).
// back:  one CTA per 32x16 tile of response pixels (128 threads with two pixel pairs a thread, 256 with
//        one). It takes the S1 tile (4 x 42 x 72) map by map through two shared-memory buffers
//        (asynchronous copies), computes the pooled L2 maps of each and the sums they complete on the
//        35 x 20 halo tile, then the 16 L3 maps (4w x 5h), the 52 hidden neurons and the output sum as far
//        as those reach. Bound by the fp32 pipe (69 % busy with every SM full): 1.36 ms for the 83 levels (1.64 when a
//        thread packed two vertical neighbours, whose operands had to be paired in registers, with two
//        reciprocal steps and twice the constant loads a pixel), 49 us for the 13 (58).
// Both kernels come in two register budgets, chosen per workload by the schedule (Stage1Sched).
// Packed f32x2 instructions run two identical chains of IEEE operations at once (two pixels, or
// two maps that read the same input), so every value still sees the reference's roundings.
// Every tile of every level is one block of the same grid; a block finds its level by binary
// search over the level descriptors (kernel parameters), so a frame is two launches per group of
// up to kParamLevels levels.
#include "kernels.h"
#include "resample.cuh"

namespace ccnn {

constexpr int kInW = 2 * kK1TileX + 3;  // 67
constexpr int kInH = 2 * kK1TileY + 3;  // 35
constexpr int kInWh = (kInW + 1) / 2;   // 34 columns of each parity

constexpr int kFrontThreads = 128;
constexpr int kStrips = kK1TileY / 2;  // a strip: two pooled rows, 32 columns
constexpr int kStripRows = 7;          // input rows of a strip

// One input sample of the front tile: row r, column c (tile coordinates) = value v. Row r is
// stored next to row r+2 as a packed pair (a thread computes two vertically adjacent pooled
// pixels, whose windows are 2 rows apart), and columns are split by parity so that the stride-2
// column walk of a warp is conflict-free.
struct FrontTile {
    float2 p[kInH - 2][2][kInWh];
    __device__ __forceinline__ void put(int r, int c, float v) {
        if (r < kInH - 2) p[r][c & 1][c >> 1].x = v;
        if (r >= 2) p[r - 2][c & 1][c >> 1].y = v;
    }
};

// Loads the (67 x 35) input tile of a front CTA from its level image. Rows that start 16-byte
// aligned with a pitch of whole float4 groups are read as 17 float4 per row (columns past the
// image width hold zeros or the caller's own padding; no stored pixel depends on them), other
// images one float at a time.
__device__ __forceinline__ void load_front_tile(FrontTile& T, const float* img, const LevelDesc& L, int ix0, int iy0) {
    if (L.img_vec) {
        constexpr int kV = (kInW + 3) / 4;  // 17
        for (int i = threadIdx.x; i < kInH * kV; i += blockDim.x) {
            const int r = i / kV, c4 = i - r * kV;
            const int x = ix0 + 4 * c4, y = iy0 + r;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (y < L.h && x < L.img_pitch) {
                const float4* src = reinterpret_cast<const float4*>(img + (long long)y * L.img_pitch + x);
                v = *src;
            }
            T.put(r, 4 * c4, v.x);
            T.put(r, 4 * c4 + 1, v.y);
            T.put(r, 4 * c4 + 2, v.z);
            if (4 * c4 + 3 < kInW) T.put(r, 4 * c4 + 3, v.w);
        }
    } else {
        for (int i = threadIdx.x; i < kInH * kInW; i += blockDim.x) {
            const int r = i / kInW, c = i - r * kInW;
            const int x = ix0 + c, y = iy0 + r;
            const float* src = img + (long long)y * L.img_pitch + x;
            T.put(r, c, (x < L.w && y < L.h) ? *src : 0.f);
        }
    }
}

// The input rows of one strip of a gated front tile, held as local rows 0..6, row r next to row r + 2
// (columns split by parity, as in FrontTile). Rows 4..6 are also the next strip's first three; each
// warp resamples its own copy, so no block barrier separates resampling and compute.
struct FrontStripRows {
    float2 p[kStripRows - 2][2][kInWh];
    __device__ __forceinline__ void put(int r, int c, float v) {
        if (r < kStripRows - 2) p[r][c & 1][c >> 1].x = v;
        if (r >= 2) p[r - 2][c & 1][c >> 1].y = v;
    }
};

// Where a level row is sampled: the gray row's offset (floats; 64 bits, a frame may have more than 2^32 pixels) and,
// for bilinear levels, the row weights (of the row and of the one below).
struct alignas(16) RowRef {
    size_t off;
    float2 cf;
};

// Two consecutive duplicated parameters by one 16-byte constant load.
struct Pair16 {
    f2_t a, b;
};
__device__ __forceinline__ Pair16 ld_pair(const float2* p) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return Pair16{v.x, v.y};
}

struct FrontSmem {
    union {
        FrontTile T;                               // the block's whole input tile (full scan, or a stored level image)
        FrontStripRows w[kFrontThreads / 32];      // each warp's own input rows (gated scan from the gray frame)
    };
    RowRef rows[kInH];                             // of the tile's rows, or kStripRows a warp
};

__device__ __forceinline__ RowRef row_ref(const GrayRef& G, const LevelDesc& L, int y) {
    RowRef r{};
    if (L.mode == 0) {
        r.off = (size_t)min(y, G.h - 1) * G.pitch;
        return r;
    }
    const AxisSample sy = sample_row(y, L.scly, G.h);
    uint32_t py = sy.idx;
    if (L.mode == 2 && py + 1 >= (uint32_t)G.h) py--;  // bilinear keeps a row below
    r.off = (size_t)py * G.pitch;
    r.cf = make_float2(sy.c, sy.f);
    return r;
}

// A level column: the gray column and, for bilinear levels, the column weights as pairs (both gray rows
// of a sample run packed).
struct ColRef {
    uint32_t x;
    f2_t c, f;
};
__device__ __forceinline__ ColRef col_ref(const GrayRef& G, const LevelDesc& L, int x) {
    ColRef r;
    if (L.mode == 0) {
        r.x = (uint32_t)min(x, G.w - 1);
        r.c = r.f = 0ull;
        return r;
    }
    const AxisSample sx = sample_col(x, L.sclx, G.w);
    r.x = sx.idx;
    r.c = f2_dup(sx.c);
    r.f = f2_dup(sx.f);
    return r;
}

// Level pixels straight from the gray frame, resampled the way the pyramid kernel writes them (copy,
// nearest neighbour, or bilinear on the 12-bit fixed-point steps; RunCPUDetect,
// cnn_detector_v3.cpp:2090-2104, with ImageResizer, image_resize.cpp:46-122, 393-541), so the level image
// is never stored. Samples past the level's last row or column read the frame's own last ones: no stored
// pooled pixel depends on them.
// kBilinear: (p0 * cx + p1 * fx) of the two gray rows as one packed chain, then top * cy + bot * fy.
template <bool kBilinear>
__device__ __forceinline__ float resample_px(const GrayRef& G, const RowRef& row, const ColRef& col, f2_t nz) {
    const float* p = G.p + (row.off + col.x);
    if (!kBilinear) return *p;
    const float* q = p + G.pitch;
    const f2_t l = f2_pack(*p, *q), r = f2_pack(p[1], q[1]);
    const f2_t h = f2_mul(f2_add(f2_mul(l, col.c, nz), f2_mul(r, col.f, nz)), f2_ld(row.cf), nz);
    return fadd(f2_lo(h), f2_hi(h));
}

// The whole (67 x 35) tile by the block (the full scan: every strip is computed, so no row is resampled
// twice): warp w takes rows w, w + 4, ... with the row's reference broadcast from shared memory, lane l
// columns l and l + 32 with theirs in registers; columns 64-66 follow, one sample a thread. `rows`: tile
// rows that lie in the level.
template <bool kBilinear>
__device__ __forceinline__ void resample_front_tile(FrontSmem& S, const GrayRef& G, const LevelDesc& L, int ix0, int rows, f2_t nz) {
    static_assert(kInW == 67 && 3 * kInH <= kFrontThreads, "64 + 3 columns, one edge sample a thread");
    constexpr int kWarps = kFrontThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const ColRef ca = col_ref(G, L, ix0 + lane), cb = col_ref(G, L, ix0 + lane + 32);
#pragma unroll 3
    for (int r = warp; r < rows; r += kWarps) {
        const RowRef row = S.rows[r];
        const float va = resample_px<kBilinear>(G, row, ca, nz), vb = resample_px<kBilinear>(G, row, cb, nz);
        S.T.put(r, lane, va);
        S.T.put(r, lane + 32, vb);
    }
    if (threadIdx.x < 3 * rows) {
        const int c = 64 + threadIdx.x % 3, r = threadIdx.x / 3;
        S.T.put(r, c, resample_px<kBilinear>(G, S.rows[r], col_ref(G, L, ix0 + c), nz));
    }
}

// One strip's 7 input rows (the gated scan, where warps run on their own): lane l takes columns l and
// l + 32; columns 64-66 of the rows follow, one sample a lane.
template <bool kBilinear>
__device__ __forceinline__ void resample_strip(FrontStripRows& R, const RowRef* rows, const GrayRef& G, const LevelDesc& L, int ix0, f2_t nz) {
    const int lane = threadIdx.x & 31;
    const ColRef ca = col_ref(G, L, ix0 + lane), cb = col_ref(G, L, ix0 + lane + 32);
#pragma unroll
    for (int r = 0; r < kStripRows; ++r) {
        const RowRef row = rows[r];
        const float va = resample_px<kBilinear>(G, row, ca, nz), vb = resample_px<kBilinear>(G, row, cb, nz);
        R.put(r, lane, va);
        R.put(r, lane + 32, vb);
    }
    if (lane < 3 * kStripRows) {
        const int c = 64 + lane % 3, r = lane / 3;
        R.put(r, c, resample_px<kBilinear>(G, rows[r], col_ref(G, L, ix0 + c), nz));
    }
}

// The learned gate inside a running stage-1 tile: whether any response pixel of [rx0, rx1] x [ry0, ry1]
// (clamped to the level's response map) has a likely cell of the level's octave within the margin of
// its window centre ((4x + 11.5) / s, (4y + 13.5) / s). The centre moves monotonically with x and y, so
// the rectangle's cells are those of its corners (the same rule as the gate's tile decisions). Only
// live response pixels can become candidates; everything else a gated tile computes is skipped.
__device__ __forceinline__ bool gate_gating(const GateCells& cells) { return cells.bits && *cells.ambiguous <= cells.amb_limit; }

__device__ __forceinline__ bool gate_live(const GateCells& cells, const LevelDesc& L, int rx0, int rx1, int ry0, int ry1) {
    rx0 = max(rx0, 0);
    ry0 = max(ry0, 0);
    rx1 = min(rx1, L.ow - 1);
    ry1 = min(ry1, L.oh - 1);
    if (rx0 > rx1 || ry0 > ry1) return false;
    const int px0 = (int)((4.f * rx0 + 11.5f) * L.inv_scale), px1 = (int)((4.f * rx1 + 11.5f) * L.inv_scale);
    const int py0 = (int)((4.f * ry0 + 13.5f) * L.inv_scale), py1 = (int)((4.f * ry1 + 13.5f) * L.inv_scale);
    const uint32_t* B = cells.bits + (long long)min(L.octave, kGK - 1) * cells.h16 * cells.wwords;
    const int m = cells.margin;
    return gate_any_bit(B, cells.wwords, gate_cell_lo(px0, m), gate_cell_hi(px1, m, cells.w16), gate_cell_lo(py0, m),
                        gate_cell_hi(py1, m, cells.h16));
}

// Front tile t of level L: its (67 x 35) level-image tile in shared memory (resampled from the gray
// frame G when kFromGray, by the block, or with the gate by each warp for the 7 rows of a strip; else read
// from the stored level images limg by the block), then the 4x4 conv + folded BN/LReLU + 2x2 max of the 4
// L1 maps for 32 x 16 pooled pixels, a warp a strip of 2 x 32 (two vertically adjacent pixels a thread), and
// the 4 neighbour-map sums written to the S1 arena.
// cells (the learned gate, optional; frames only, a stored image is always computed in full): a strip that feeds no
// live response pixel is not computed. S1 row y
// feeds pooled-L2 rows ceil((y - 3) / 2) .. y / 2 (a 3x3 conv at the 2x2 pool positions), and L2 row Y
// feeds response rows Y - 4 .. Y (the 4-wide, 5-tall L3 kernel); columns alike with the 4-wide kernel. The
// back kernel computes exactly the live pixels' inputs, so a skipped strip is never read for a value that
// is kept.
template <bool kFromGray>
__device__ __forceinline__ void front_tile(const Stage1W& W, FrontSmem& S, const LevelDesc& L, int t, const float* limg,
                                           const GrayRef& G, float* s1, const GateCells& cells) {
    constexpr int kWarps = kFrontThreads / 32;
    const int px0 = (t % L.k1_tiles_x) * kK1TileX;
    const int py0 = (t / L.k1_tiles_x) * kK1TileY;
    const int ix0 = 2 * px0, iy0 = 2 * py0;
    const int qx = threadIdx.x & (kK1TileX - 1);
    const int warp = threadIdx.x >> 5;
    const int strips = min(kStrips, (L.p1h - py0 + 1) >> 1);  // those with pooled rows inside the level
    const f2_t nz = f2_ld(W.negzero);
    // with the gate: whether strip s has a live pixel downstream
    auto strip_live = [&](int s) {
        const int ya = py0 + 2 * s, yb = ya + 1, xa = px0, xb = px0 + kK1TileX - 1;
        return gate_live(cells, L, ((xa - 3 + 1) >> 1) - 3, xb >> 1, ((ya - 3 + 1) >> 1) - 4, yb >> 1);
    };
    // the four L1 maps of strip s from its input rows In[r] = (row 4s + r, row 4s + r + 2), r = 0..4, and
    // their neighbour sums into the arena
    auto strip = [&](int s, const float2(*In)[2][kInWh]) {
        // pr[r][c] = (input row 4s + r, row 4s + r + 2) at column 2qx + c: the windows of both pixels
        f2_t pr[5][5];
#pragma unroll
        for (int r = 0; r < 5; ++r)
#pragma unroll
            for (int c = 0; c < 5; ++c) pr[r][c] = f2_ld(In[r][c & 1][qx + (c >> 1)]);

        // packed over the two pixels (lo = row 2s, hi = row 2s + 1)
        f2_t P[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            f2_t cv[4];
#pragma unroll
            for (int k = 0; k < 16; k += 2) {
                const Pair16 w = ld_pair(&W.k1d[m][k]);
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    const int dy = d >> 1, dx = d & 1;
                    const f2_t a = f2_mul(pr[dy + (k >> 2)][dx + (k & 3)], w.a, nz);
                    cv[d] = f2_add(k ? f2_add(cv[d], a) : a, f2_mul(pr[dy + (k >> 2)][dx + (k & 3) + 1], w.b, nz));
                }
            }
#pragma unroll
            for (int d = 0; d < 4; ++d) cv[d] = lrelu_bn2(cv[d], W.a1d[m], nz);
            P[m] = f2_max4(cv[0], cv[1], cv[2], cv[3]);
        }
        // neighbour-map sums consumed by L2 (add/add2 of the reference)
        const f2_t s01 = f2_add(P[0], P[1]);
        const f2_t o[4] = {s01, f2_add(s01, P[2]), f2_add(f2_add(P[1], P[2]), P[3]), f2_add(P[2], P[3])};
        const int gx = px0 + qx, gy = py0 + 2 * s;
        if (gx < L.p1w) {
            // a row holds its even columns, then its odd ones
            float* out = s1 + L.s1_off + (long long)gy * L.s1_pitch + ((gx & 1) ? L.s1_pitch >> 1 : 0) + (gx >> 1);
            const bool two = gy + 1 < L.p1h;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                out[0] = f2_lo(o[k]);
                if (two) out[L.s1_pitch] = f2_hi(o[k]);
                out += L.s1_plane;
            }
        }
    };
    if (kFromGray && gate_gating(cells)) {
        // with the gate every warp runs on its own: its strips' liveness, their 7 input rows, their two
        // pooled rows (the rows a live strip shares with a dead neighbour are not resampled twice over the
        // tile, and no warp waits for the block)
        RowRef* rows = &S.rows[warp * kStripRows];
        static_assert(kWarps * kStripRows <= kInH, "a row table a warp");
        const int lane = threadIdx.x & 31;
#pragma unroll 1
        for (int s = warp; s < strips; s += kWarps) {
            int lv = 0;
            if (lane == 0) lv = strip_live(s) ? 1 : 0;
            if (!__shfl_sync(0xffffffffu, lv, 0)) continue;  // no live response pixel downstream of this strip
            __syncwarp();
            if (lane < kStripRows) rows[lane] = row_ref(G, L, iy0 + 4 * s + lane);
            __syncwarp();
            if (L.mode == 2)
                resample_strip<true>(S.w[warp], rows, G, L, ix0, nz);
            else
                resample_strip<false>(S.w[warp], rows, G, L, ix0, nz);
            __syncwarp();
            strip(s, S.w[warp].p);
        }
        return;
    }
    if (kFromGray) {
        // the full scan: the block resamples the tile once
        if (threadIdx.x < kInH) S.rows[threadIdx.x] = row_ref(G, L, iy0 + threadIdx.x);
        __syncthreads();
        const int rows = 4 * strips + 3;
        if (L.mode == 2)
            resample_front_tile<true>(S, G, L, ix0, rows, nz);
        else
            resample_front_tile<false>(S, G, L, ix0, rows, nz);
    } else {
        load_front_tile(S.T, limg + L.img_off, L, ix0, iy0);
    }
    __syncthreads();
#pragma unroll 1
    for (int s = warp; s < strips; s += kWarps) strip(s, &S.T.p[4 * s]);
}


// kFromGray: level tiles resampled from the gray frame G (the detection path), else read from the
// stored level images limg (a caller's own level image)
template <bool kFromGray, int kMinBlocks>
__global__ void __launch_bounds__(kFrontThreads, kMinBlocks) stage1_front_kernel(const __grid_constant__ Stage1W W, const __grid_constant__ LevelTable LT,
                                                              const float* limg, const GrayRef G, float* s1, const uint8_t* front_on,
                                                              const GateCells cells, int* counts, int n_counts) {
    __shared__ FrontSmem S;
    chain_wait();
    if (blockIdx.x == 0)  // the back kernel's candidate counts start from zero
        for (int i = threadIdx.x; i < n_counts; i += kFrontThreads) counts[i] = 0;
    const int g = LT.first + blockIdx.x;
    if (front_on && !front_on[g]) return;  // gated off: no back tile reads this one
    const LevelDesc& L = LT.lv[find_level<&LevelDesc::k1_base>(LT, g)];
    front_tile<kFromGray>(W, S, L, g - L.k1_base, limg, G, s1, cells);
}

constexpr int kP2TW = kK2TileX + 3;   // 35 pooled L2 columns (halo 3)
constexpr int kP2TH = kK2TileY + 4;   // 20 pooled L2 rows (halo 4)
constexpr int kS1TW = 2 * kP2TW + 2;  // 72
constexpr int kS1TH = 2 * kP2TH + 2;  // 42
constexpr int kHalfX = kK2TileX / 2;  // 16: pixels x and x + 16 of a row run as a packed pair
constexpr int kS2P = kHalfX + 3;      // 19 pairs a row of pooled L2 pixels (columns 16-18 are in two pairs)

struct BackSmem {
    // two S1 maps of the tile (map k in s1[k & 1]), each row its even columns, then its odd ones: a warp's
    // 2x2-pooling windows read consecutive words
    float s1[2][kS1TH][2][kS1TW / 2];
    // the neighbour sums of the pooled L2 maps that this S1 map completes (at most three), column x next to
    // column x + 16: the taps of a thread's response pixels load as packed pairs
    float2 s2[3][kP2TH][kS2P];
};
constexpr int kP2Units = kS2P * kP2TH;  // 380 pairs of pooled L2 pixels of a tile

// Pooled L2 pair k of a tile: the 16 x 20 block first (a warp takes two rows of 16 pairs: no bank
// conflicts), then the 3 x 20 right edge.
__device__ __forceinline__ void p2_unit(int p, int* x, int* y) {
    if (p < kHalfX * kP2TH) {
        *x = p & (kHalfX - 1);
        *y = p / kHalfX;
    } else {
        const int q = p - kHalfX * kP2TH;
        *x = kHalfX + q % 3;
        *y = q / 3;
    }
}

// S1 map k of a back tile into shared memory by asynchronous 16-byte copies (cp.async through L2);
// columns past the plane pitch and rows past p1h are zero-filled (no valid response pixel depends on
// them).
template <int kThreads>
__device__ __forceinline__ void load_back_map_async(BackSmem& S, const float* s1, const LevelDesc& L, int sx0, int sy0, int k) {
    const float* base = s1 + L.s1_off + (long long)k * L.s1_plane;
    constexpr int kV = kS1TW / 8;  // 16-byte vectors of a row's columns of one parity
    const int half = L.s1_pitch >> 1;
    float* buf = &S.s1[k & 1][0][0][0];
    for (int i = threadIdx.x; i < kS1TH * 2 * kV; i += kThreads) {
        const int rr = i / (2 * kV), q = i - rr * (2 * kV);
        const int par = q >= kV ? 1 : 0, c4 = q - par * kV;
        const int x = (sx0 >> 1) + 4 * c4, y = sy0 + rr;
        const bool in = y < L.p1h && x < half;  // x and half are multiples of 4: the whole vector is in the row's half
        const float* src = in ? base + (long long)y * L.s1_pitch + par * half + x : base;
        const unsigned dst = (unsigned)__cvta_generic_to_shared(buf + rr * kS1TW + par * (kS1TW / 2) + 4 * c4);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ f2_t lrelu_bn_d(f2_t x, const float2* p, f2_t nz) {
    const Pair16 u = ld_pair(p), v = ld_pair(p + 2);
    const f2_t c = f2_add(x, u.a);
    return f2_add(f2_add(f2_mul(u.b, c, nz), f2_mul(v.a, f2_max0(c), nz)), v.b);
}

// Pooled L2 map m at the tile's pixel pair whose input is q: 3x3 conv + BN/LReLU at the four positions
// of the 2x2 window, then their max.
__device__ __forceinline__ f2_t pool_l2(const f2_t (*q)[4], const Stage1Back::L2Map& M, f2_t nz) {
    f2_t w[10];
#pragma unroll
    for (int k = 0; k < 10; k += 2) {
        const Pair16 u = ld_pair(&M.k[k]);
        w[k] = u.a;
        w[k + 1] = u.b;
    }
    f2_t acc[4];
#pragma unroll
    for (int d = 0; d < 4; ++d) acc[d] = f2_mul(q[d >> 1][d & 1], w[0], nz);
#pragma unroll
    for (int k = 1; k < 9; ++k)
#pragma unroll
        for (int d = 0; d < 4; ++d) acc[d] = f2_add(acc[d], f2_mul(q[(d >> 1) + k / 3][(d & 1) + k % 3], w[k], nz));
#pragma unroll
    for (int d = 0; d < 4; ++d) acc[d] = lrelu_bn_d(acc[d], M.a, nz);
    return f2_max4(acc[0], acc[1], acc[2], acc[3]);
}

// back: one CTA per 32 x 16 tile of response pixels, every operation packed over the pixels (x, x + 16)
// of a row, so that no operand has to be duplicated or paired in registers. kPairs pixel pairs a thread
// in C (256 / kPairs threads): two halve the constant loads a pixel, which share one queue with the
// shared-memory loads, and suit launches with many tiles a SM; one gives a tile twice the warps
// (back_pixel_pairs).
// The four S1 maps of the tile (42 x 72 each) pass through shared memory one after the other; for map k
//   A: the pooled L2 maps 2k and 2k + 1 on the 35 x 20 halo tile, and the neighbour sums whose three maps
//      are now known (the two partial sums a pixel still needs stay in registers);
//   C: the L3 maps (4w x 5h) of those sums, the hidden groups whose four L3 maps are now known and their
//      part of the output sum, all in registers, while S1 map k + 1 is copied (cp.async).
// Two S1 maps and three sums are ever held, 33 KB, so that registers alone limit the resident blocks.
// Back tile t of level L as above; g is its global back-tile index (the gate's tile index).
// The S1 arena may have been written earlier in the same launch (the persistent kernel): its copies go through L2
// (cp.async.cg), where those writes are.
// Warps (32 x 2 kPairs response pixels) and L2 rows that only pixels past the map's last row need are
// skipped. With the learned gate (cells), a warp without a live pixel writes the skip marker instead of
// computing, A computes only the rows live warps read (a warp's rows and the four after them), and
// every pixel that is not live is written as the skip marker: only live pixels can become candidates,
// and their inputs are exactly what runs (the front kernel skips the rest of S1).
template <int kPairs>
__device__ __forceinline__ void back_tile(const Stage1Back& D, BackSmem& S, const LevelDesc& L, int t, int g, const float* s1,
                                          float* resp, int* counts, float thr, const uint8_t* back_on,
                                          const GateCells& cells) {
    constexpr int kThreads = kK2TileX * kK2TileY / (2 * kPairs);
    constexpr int kWarps = kThreads / 32, kWarpRows = kK2TileY / kWarps;
    constexpr int kP2Passes = (kP2Units + kThreads - 1) / kThreads;
    const int ox0 = (t % L.k2_tiles_x) * kK2TileX;
    const int oy0 = (t / L.k2_tiles_x) * kK2TileY;
    if (back_on && !back_on[g]) {  // gated off: responses below any stage-1 threshold
        for (int i = threadIdx.x; i < kK2TileX * kK2TileY; i += kThreads) {
            const int gx = ox0 + (i & (kK2TileX - 1)), gy = oy0 + i / kK2TileX;
            if (gx < L.ow && gy < L.oh) resp[L.resp_off + (long long)gy * L.ow + gx] = -1e30f;
        }
        return;
    }
    const int sx0 = 2 * ox0, sy0 = 2 * oy0;
    load_back_map_async<kThreads>(S, s1, L, sx0, sy0, 0);
    load_back_map_async<kThreads>(S, s1, L, sx0, sy0, 1);
    const f2_t nz = f2_ld(D.negzero);
    const bool gating = gate_gating(cells);
    const int warp = threadIdx.x >> 5;
    __shared__ int s_live[kWarps];  // per warp: any live response pixel
    if (gating && (threadIdx.x & 31) == 0) {
        const int ry = oy0 + kWarpRows * warp;
        s_live[warp] = gate_live(cells, L, ox0, ox0 + kK2TileX - 1, ry, ry + kWarpRows - 1) ? 1 : 0;
    }
    // live warps: those with response rows inside the map (with the gate, with a live pixel in them)
    const int rows = min(kK2TileY, L.oh - oy0);
    uint32_t live = (1u << ((rows + kWarpRows - 1) / kWarpRows)) - 1u;
    const int xe = L.ow - ox0 + 3;  // pooled L2 columns from here on feed no response pixel of the map
    // L2 row y is read by warps ceil((y - kWarpRows - 3) / kWarpRows) .. y / kWarpRows
    auto need_row = [&](int y) {
        const int wlo = max(0, y - (kWarpRows + 3) + kWarpRows - 1) / kWarpRows, whi = min(kWarps - 1, y / kWarpRows);
        return ((live >> wlo) & ((1u << (whi - wlo + 1)) - 1u)) != 0u;
    };
    // the thread's response pixels: (x, x + 16) of rows y .. y + kPairs - 1
    const int x = threadIdx.x & (kHalfX - 1), y = (threadIdx.x / kHalfX) * kPairs;
    const f2_t half = f2_pack(0.5f, 0.5f);
    // A: the sums in the reference's order: s0 = P0 + P1, s1 = s0 + P2, s(2j) = (P(2j-1) + P(2j)) + P(2j+1),
    // s(2j+1) = (P(2j) + P(2j+1)) + P(2j+2), s7 = P6 + P7; ca and cb carry (P(2k) + P(2k+1)) and P(2k+1)
    // to the next map
    f2_t ca[kP2Passes], cb[kP2Passes];
    // C: hidden neuron n = 4*i + t reads L3 maps i..i+3: a[0]..a[3] is the window of the last four L3 maps;
    // the output sum runs over n in order
    static_assert(Stage1W::kConn == 4 && Stage1W::kGroups + 3 == Stage1W::kM3, "sliding window of four L3 maps");
    f2_t a[4][kPairs] = {}, out[kPairs] = {};
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
        if (k < 3) cp_async_wait<1>();
        else cp_async_wait<0>();
        __syncthreads();  // S1 map k is in shared memory for every thread, and the sums of map k - 1 are read
        if (k == 0 && gating) {
            uint32_t on = 0u;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) on |= (s_live[w] ? 1u : 0u) << w;
            live &= on;
        }
        const float(*T)[2][kS1TW / 2] = S.s1[k & 1];
#pragma unroll
        for (int kk = 0; kk < kP2Passes; ++kk) {
            const int p = threadIdx.x + kThreads * kk;
            int ux = 0, uy = 0;
            if (p < kP2Units) p2_unit(p, &ux, &uy);
            if (p < kP2Units && ux < xe && need_row(uy)) {
                f2_t q[4][4];
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        q[r][c] = f2_pack(T[2 * uy + r][c & 1][ux + (c >> 1)], T[2 * uy + r][c & 1][ux + kHalfX + (c >> 1)]);
                const f2_t A = pool_l2(q, D.l2[2 * k], nz), B = pool_l2(q, D.l2[2 * k + 1], nz);
                auto put = [&](int slot, f2_t v) { *reinterpret_cast<f2_t*>(&S.s2[slot][uy][ux]) = v; };
                const f2_t ab = f2_add(A, B);
                if (k == 0) {
                    put(0, ab);
                } else {
                    put(0, f2_add(ca[kk], A));
                    put(1, f2_add(f2_add(cb[kk], A), B));
                    if (k == 3) put(2, ab);
                }
                ca[kk] = ab;
                cb[kk] = B;
            }
        }
        __syncthreads();  // the sums are complete, and map k's buffer is free
        if (k < 2) load_back_map_async<kThreads>(S, s1, L, sx0, sy0, k + 2);
        if (!((live >> warp) & 1u)) continue;
        const int first = k == 0 ? 0 : 2 * k - 1, n_sums = k == 0 ? 1 : (k == 3 ? 3 : 2);
#pragma unroll 1
        for (int j = 0; j < n_sums; ++j) {
            // L3 maps (2s, 2s+1) of the pixel pairs from sum s; conv_5x4 keeps one partial sum per kernel
            // row, added in row order
            const int s = first + j;
            f2_t nm[2][kPairs];
            {
                f2_t acc[2][kPairs], v[kPairs][4];
#pragma unroll
                for (int p = 0; p < kPairs - 1; ++p)
#pragma unroll
                    for (int c = 0; c < 4; ++c) v[p][c] = f2_ld(S.s2[j][y + p][x + c]);
#pragma unroll
                for (int r = 0; r < 5; ++r) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) v[kPairs - 1][c] = f2_ld(S.s2[j][y + r + kPairs - 1][x + c]);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const Pair16 w01 = ld_pair(&D.l3[2 * s + e].k[4 * r]), w23 = ld_pair(&D.l3[2 * s + e].k[4 * r + 2]);
#pragma unroll
                        for (int p = 0; p < kPairs; ++p) {
                            f2_t rs = f2_mul(v[p][0], w01.a, nz);
                            rs = f2_add(rs, f2_mul(v[p][1], w01.b, nz));
                            rs = f2_add(rs, f2_mul(v[p][2], w23.a, nz));
                            rs = f2_add(rs, f2_mul(v[p][3], w23.b, nz));
                            acc[e][p] = (r == 0) ? rs : f2_add(acc[e][p], rs);
                        }
                    }
#pragma unroll
                    for (int p = 0; p < kPairs - 1; ++p)
#pragma unroll
                        for (int c = 0; c < 4; ++c) v[p][c] = v[p + 1][c];
                }
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int p = 0; p < kPairs; ++p) nm[e][p] = lrelu_bn_d(acc[e][p], D.l3[2 * s + e].a, nz);
            }
#pragma unroll 1
            for (int e = 0; e < 2; ++e) {
#pragma unroll
                for (int p = 0; p < kPairs; ++p) {
                    a[0][p] = a[1][p];
                    a[1][p] = a[2][p];
                    a[2][p] = a[3][p];
                    a[3][p] = nm[0][p];
                    nm[0][p] = nm[1][p];
                }
                const int i = 2 * s + e - 3;  // the hidden group that L3 map 2s + e completes
                if (i < 0) continue;
                const f2_t tw = f2_ld(D.htw[i]);
#pragma unroll
                for (int tt = 0; tt < Stage1W::kHS; ++tt) {
                    const int n = Stage1W::kHS * i + tt;
                    const Stage1Back::Neuron& N = D.hid[n];
                    const Pair16 bw = ld_pair(&N.b), w12 = ld_pair(&N.w[1]), w3o = ld_pair(&N.w[3]), bn = ld_pair(&D.hbn[tt].w);
#pragma unroll
                    for (int p = 0; p < kPairs; ++p) {
                        f2_t h = f2_add(bw.a, f2_mul(a[0][p], bw.b, nz));
                        h = f2_add(h, f2_mul(a[1][p], w12.a, nz));
                        h = f2_add(h, f2_mul(a[2][p], w12.b, nz));
                        h = f2_add(h, f2_mul(a[3][p], w3o.a, nz));
                        const f2_t v = tanh_half2(f2_mul(h, tw, nz), nz, half);
                        const f2_t hw = f2_mul(f2_add(f2_mul(bn.a, v, nz), bn.b), w3o.b, nz);
                        out[p] = (n == 0) ? hw : f2_add(hw, out[p]);
                    }
                }
            }
        }
    }
    const int gx = ox0 + x, gy = oy0 + y;
    const bool on = (live >> warp) & 1u;  // else the skip marker instead of the responses
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
        f2_t c = f2_mul(f2_add(out[p], f2_ld(D.ob)), f2_ld(D.otw), nz);
        c = tanh_rational2(c, nz);
        const f2_t r = D.half_out ? f2_add(f2_mul(half, c, nz), half) : f2_mul(f2_ld(D.af), c, nz);
        if (gy + p >= L.oh) break;
        const int at = (gy + p) * L.ow + gx;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int px = gx + h * kHalfX;
            if (px >= L.ow) break;
            float v = h == 0 ? f2_lo(r) : f2_hi(r);
            // only live pixels keep their response (a candidate needs a likely cell of its octave within
            // the margin of its window centre); the others may have read skipped inputs
            if (!on || (gating && !gate_live(cells, L, px, px, gy + p, gy + p))) v = -1e30f;
            resp[L.resp_off + at + h * kHalfX] = v;
            // candidates (response > treshold_1) are counted per scan chunk for the compaction
            if (counts && v > thr) atomicAdd(&counts[L.chunk_base + (at + h * kHalfX) / kCandChunk], 1);
        }
    }
}

template <int kPairs, int kMinBlocks>
__global__ void __launch_bounds__(256 / kPairs, kMinBlocks) stage1_back_kernel(const __grid_constant__ Stage1Back D, const __grid_constant__ LevelTable LT,
                                                             const float* s1, float* resp, int* counts, float thr, const uint8_t* back_on,
                                                             const GateCells cells) {
    __shared__ BackSmem S;
    const int g = LT.first + blockIdx.x;
    const LevelDesc& L = LT.lv[find_level<&LevelDesc::k2_base>(LT, g)];
    const int t = g - L.k2_base;
    chain_wait();
    back_tile<kPairs>(D, S, L, t, g, s1, resp, counts, thr, back_on, cells);
}

// The back kernel's parameters, derived from the packed weight block.
static Stage1Back make_back(const Stage1W& W) {
    Stage1Back D{};
    auto dup = [](float v) { return make_float2(v, v); };
    auto act = [&](float2* a, float b, float wa, float wb, float bn) {
        a[0] = dup(b);
        a[1] = dup(wa);
        a[2] = dup(wb);
        a[3] = dup(bn);
    };
    for (int m = 0; m < Stage1W::kM2; ++m) {
        for (int k = 0; k < Stage1W::kK2W * Stage1W::kK2H; ++k) D.l2[m].k[k] = dup((m & 1) ? W.k2p[m / 2][k].y : W.k2p[m / 2][k].x);
        act(D.l2[m].a, W.b2[m], W.w2a[m], W.w2b[m], W.bn2[m]);
    }
    for (int m = 0; m < Stage1W::kM3; ++m) {
        for (int k = 0; k < Stage1W::kK3W * Stage1W::kK3H; ++k) D.l3[m].k[k] = dup((m & 1) ? W.k3p[m / 2][k].y : W.k3p[m / 2][k].x);
        act(D.l3[m].a, W.b3[m], W.w3a[m], W.w3b[m], W.bn3[m]);
    }
    for (int n = 0; n < Stage1W::kHL; ++n) {
        D.hid[n].b = dup(W.hb[n]);
        for (int j = 0; j < Stage1W::kConn; ++j) D.hid[n].w[j] = dup((n & 1) ? W.hwp[n / 2][j].y : W.hwp[n / 2][j].x);
        D.hid[n].o = dup(W.ow[n]);
    }
    for (int i = 0; i < Stage1W::kGroups; ++i) D.htw[i] = dup(W.htw[i]);
    for (int t = 0; t < Stage1W::kHS; ++t) {
        D.hbn[t].w = dup(W.hbnw[t]);
        D.hbn[t].b = dup(W.hbnb[t]);
    }
    D.ob = dup(W.ob);
    D.otw = dup(W.otw);
    D.af = dup(W.af);
    D.negzero = W.negzero;
    D.half_out = W.af == 0.f ? 1 : 0;
    return D;
}

// Launches KERNEL once per group of at most kParamLevels levels; tiles(L) is a level's block count
// and base(L) its first global block.
template <class Launch, class Tiles>
static cudaError_t launch_grouped(const LevelDesc* levels, int n_levels, int LevelDesc::*base, Tiles tiles, Launch launch) {
    for (int g0 = 0; g0 < n_levels; g0 += kParamLevels) {
        LevelTable T;
        T.n = n_levels - g0 < kParamLevels ? n_levels - g0 : kParamLevels;
        for (int i = 0; i < T.n; ++i) T.lv[i] = levels[g0 + i];
        T.first = T.lv[0].*base;
        const LevelDesc& last = T.lv[T.n - 1];
        const int blocks = last.*base + tiles(last) - T.first;
        const cudaError_t e = blocks > 0 ? launch(T, blocks) : cudaSuccess;
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

cudaError_t launch_stage1_front(const Stage1W& W, const LevelDesc* levels, int n_levels, const float* limg, float* s1, cudaStream_t st,
                                const uint8_t* front_on, Stage1Sched sched, GrayRef gray, GateCells cells, int* counts, int n_counts) {
    return launch_grouped(
        levels, n_levels, &LevelDesc::k1_base, [](const LevelDesc& L) { return L.k1_tiles_x * ((L.p1h + kK1TileY - 1) / kK1TileY); },
        [&](const LevelTable& T, int blocks) {
            const bool six = sched.front_blocks_per_sm >= 4;
            const auto kernel = gray.p ? (six ? stage1_front_kernel<true, 6> : stage1_front_kernel<true, 5>)
                                       : (six ? stage1_front_kernel<false, 6> : stage1_front_kernel<false, 5>);
            const cudaError_t e = launch_chained(kernel, blocks, kFrontThreads, 0, st, W, T, limg, gray, s1, front_on, cells, counts, n_counts);
            n_counts = 0;  // by the first launch
            return e;
        });
}

cudaError_t launch_stage1_back(const Stage1W& W, const LevelDesc* levels, int n_levels, const float* s1, float* resp, cudaStream_t st,
                               int* counts, float thr, const uint8_t* back_on, GateCells cells, Stage1Sched sched) {
    const Stage1Back D = make_back(W);
    if (n_levels <= 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    return launch_grouped(
        levels, n_levels, &LevelDesc::k2_base, [](const LevelDesc& L) { return L.k2_tiles_x * ((L.oh + kK2TileY - 1) / kK2TileY); },
        [&](const LevelTable& T, int blocks) {
            const bool two_pairs = back_pixel_pairs(blocks, sms, back_on != nullptr) == 2;
            const auto kernel = two_pairs ? (sched.back_blocks_per_sm >= 4 ? stage1_back_kernel<2, 6> : stage1_back_kernel<2, 5>) : stage1_back_kernel<1, 3>;
            return launch_chained(kernel, blocks, two_pairs ? 128 : 256, 0, st, D, T, s1, resp, counts, thr, back_on, cells);
        });
}

cudaError_t launch_stage1(const Stage1W& W, const LevelDesc* levels, int n_levels, const float* limg, float* s1, float* resp,
                          cudaStream_t st, int* counts, float thr, const uint8_t* front_on, const uint8_t* back_on, GateCells cells,
                          Stage1Sched sched, GrayRef gray, int n_counts) {
    cudaError_t e = launch_stage1_front(W, levels, n_levels, limg, s1, st, front_on, sched, gray, cells, counts, n_counts);
    if (e != cudaSuccess) return e;
    return launch_stage1_back(W, levels, n_levels, s1, resp, st, counts, thr, back_on, cells, sched);
}

// ---------------- batched form: one persistent launch over B frames ----------------
//
// Every front tile and back tile of every level of every frame of a batch is one item of a device
// work queue (an atomic counter); a persistent grid takes items in queue order until none are left,
// claiming its next item while it works on the current one. Items of the back stage of frame f wait
// until every front item of frame f has finished (a counter per (frame, stage), polled with acquire
// loads by one thread, a bounded number of times); the diagonal queue order puts about one frame's
// worth of other items between a frame's front tiles and its back tiles, so the polls almost never
// wait. An item only waits on items queued before it, and a block holds at most the item it works on
// and the one it claimed after it, so every wait ends whatever the number of resident blocks. Front
// items resample their level tiles from the gray frames (written by the gray launch before); the S1
// planes are written earlier in the same launch and are read through L2 (ld.global.cg), never the
// read-only path.

void build_batch_queue(BatchQueue* q, int n_frames, int n_levels, int n_chunks, int front_items, int back_items, float thr) {
    q->n_frames = n_frames;
    q->n_levels = n_levels;
    q->n_chunks = n_chunks;
    q->thr = thr;
    q->stage_items[0] = front_items;
    q->stage_items[1] = back_items;
    q->wait_limit = 1 << 22;  // x 256 ns of sleep: about a second before the launch gives up
    int n = 0, first = 0;
    for (int t = 0; t < n_frames + kBatchStages - 1; ++t)
        for (int st = 0; st < kBatchStages; ++st) {
            const int f = t - st;
            if (f < 0 || f >= n_frames || q->stage_items[st] <= 0) continue;
            q->seg_stage[n] = st;
            q->seg_frame[n] = f;
            q->seg_first[n] = first;
            first += q->stage_items[st];
            ++n;
        }
    q->seg_first[n] = first;
    q->n_seg = n;
    q->total = first;
}

__device__ __forceinline__ int ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

constexpr int kBatchThreads = kFrontThreads;  // a front tile's block, and a back tile's with two pairs a thread
constexpr int kBatchSmem = (int)sizeof(BackSmem) > (int)sizeof(FrontSmem) ? (int)sizeof(BackSmem) : (int)sizeof(FrontSmem);

__global__ void __launch_bounds__(kBatchThreads, 5) stage1_batch_kernel(const __grid_constant__ Stage1W W, const __grid_constant__ Stage1Back D,
                                                              const __grid_constant__ BatchFrames F, const __grid_constant__ BatchQueue Q,
                                                              const LevelDesc* __restrict__ levels, int* __restrict__ sync,
                                                              int* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_item;
    __shared__ unsigned long long s_ready;  // bit 2f+s: stage s of frame f is known complete
    __shared__ int s_base[kBatchStages][kMaxBatchLevels];  // first front / back item of each level
    const int nl = Q.n_levels < kMaxBatchLevels ? Q.n_levels : kMaxBatchLevels;
    for (int l = threadIdx.x; l < nl; l += blockDim.x) {
        s_base[0][l] = levels[l].k1_base;
        s_base[1][l] = levels[l].k2_base;
    }
    if (threadIdx.x == 0) {
        s_ready = 0ull;
        s_item = atomicAdd(&sync[0], 1);
    }
    __syncthreads();
    int item = s_item;
    while (item < Q.total) {
        int next = 0;
        if (threadIdx.x == 0) next = atomicAdd(&sync[0], 1);  // the next item, claimed while this one runs
        int sg = 0;
        while (sg + 1 < Q.n_seg && Q.seg_first[sg + 1] <= item) ++sg;
        const int stage = Q.seg_stage[sg], f = Q.seg_frame[sg], g = item - Q.seg_first[sg];
        if (stage > 0) {
            const int dep = kBatchStages * f + stage - 1;
            if (!(s_ready & (1ull << dep))) {  // uniform: every thread reads the same word
                if (threadIdx.x == 0) {
                    const int need = Q.stage_items[stage - 1];
                    int polls = 0;
                    while (ld_acquire(&sync[1 + dep]) < need) {
                        if (++polls > Q.wait_limit || ld_acquire(err) != 0) {
                            atomicExch(err, 1);
                            break;
                        }
                        __nanosleep(256);
                    }
                    __threadfence();
                }
                __syncthreads();
                if (threadIdx.x == 0) s_ready |= 1ull << dep;
            }
        }
        // the level of the item: the last level whose first item is <= g
        int lo = 0, hi = nl - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (s_base[stage][mid] <= g) lo = mid; else hi = mid - 1;
        }
        const LevelDesc& L = levels[lo];
        if (stage == 0) {
            if (!F.front_on[f] || F.front_on[f][g])
                front_tile<true>(W, *reinterpret_cast<FrontSmem*>(smem_raw), L, g - L.k1_base, nullptr,
                                        GrayRef{F.gray[f], F.gpitch, F.gw, F.gh}, F.s1[f], F.cells[f]);
        } else {
            back_tile<2>(D, *reinterpret_cast<BackSmem*>(smem_raw), L, g - L.k2_base, g, F.s1[f], F.resp[f], F.counts[f], Q.thr,
                            F.back_on[f], F.cells[f]);
        }
        __syncthreads();  // every thread is done with the item (and with the shared memory)
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(&sync[1 + kBatchStages * f + stage], 1);
            s_item = next;
        }
        __syncthreads();
        item = s_item;
    }
}

// The candidate counts of every frame of a batch zeroed (blockIdx.x is the frame), before the
// persistent stage-1 launch counts into them.
__global__ void __launch_bounds__(256) counts_zero_batch_kernel(const __grid_constant__ BatchFrames F, int n_chunks) {
    int* c = F.counts[blockIdx.x];
    for (int i = threadIdx.x; i < n_chunks; i += blockDim.x) c[i] = 0;
}

cudaError_t launch_counts_zero_batch(const BatchFrames& F, int n_chunks, int n_frames, cudaStream_t st) {
    if (n_chunks <= 0 || n_frames <= 0) return cudaSuccess;
    counts_zero_batch_kernel<<<n_frames, 256, 0, st>>>(F, n_chunks);
    return cudaGetLastError();
}

// resident blocks per SM of the persistent kernel: twice the schedule's count (1-4, in units of 256
// threads), at most what fits
int stage1_batch_blocks_per_sm(int blocks_per_sm) {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, stage1_batch_kernel, kBatchThreads, kBatchSmem);
    if (blocks_per_sm >= 1 && 2 * blocks_per_sm < n) n = 2 * blocks_per_sm;
    return n > 0 ? n : 1;
}

cudaError_t launch_stage1_batch(const Stage1W& W, const BatchFrames& F, const BatchQueue& Q, const LevelDesc* d_levels, int* sync, int* err,
                                int grid, cudaStream_t st) {
    if (Q.total <= 0) return cudaSuccess;
    if (Q.n_levels > kMaxBatchLevels) return cudaErrorInvalidValue;
    const Stage1Back D = make_back(W);
    grid = grid < Q.total ? grid : Q.total;
    stage1_batch_kernel<<<grid, kBatchThreads, kBatchSmem, st>>>(W, D, F, Q, d_levels, sync, err);
    return cudaGetLastError();
}

// The back kernels' resident blocks need most of a SM's 228 KB as shared memory (33 KB each).
cudaError_t stage1_setup() {
    const auto prefer = [](const void* f) { return cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared); };
    cudaError_t e = prefer(reinterpret_cast<const void*>(stage1_back_kernel<1, 3>));
    if (e == cudaSuccess) e = prefer(reinterpret_cast<const void*>(stage1_back_kernel<2, 5>));
    if (e == cudaSuccess) e = prefer(reinterpret_cast<const void*>(stage1_back_kernel<2, 6>));
    return e;
}

}  // namespace ccnn
