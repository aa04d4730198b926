// Training of the learned gate (the network is described in gate.cu): positive-weighted binary
// cross-entropy over all cells, minimised with Adam. No reference counterpart.
//
// A step is three launches: forward + head (gate_forward_kernel), backward (gate_backward_kernel), and
// the sum of the blocks' gradients with Adam (gate_update_kernel). Only the pooled cells' gradient and
// the signs of a2 (a byte a pixel) pass between the first two; a1 is computed again from the features
// where it is needed (72 of a pixel's 1,872 multiply-adds, against 64 bytes of traffic a pixel). Both
// are persistent, a block of 128 threads a tile of 32 x 16 pixels at a time with its halo in shared
// memory, and keep their gradient sums in registers over all their tiles, so there are no atomics and
// every run gives the same bits. A step on 64 frames of 240 x 135 takes 0.28 ms on B200: 0.1 forward, 0.17
// backward, 0.009 update (3.1 ms when every map passed through memory, a weight gradient was one thread's walk
// over the pixels of a row band and the sums were atomics): 3.9 G multiply-adds, 0.11 ms at the fp32 pipe's rate.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "../../include/ccnn_gate.h"
#include "gate_net.cuh"

namespace ccnn {

void set_error(const std::string& msg);

namespace {

constexpr int kTT = 128;                   // threads: lane = column of the tile, warp = four of its rows
constexpr int kTW = 32, kTH = 16;          // tile
constexpr int kHW = kTW + 2, kHH = kTH + 2;  // with a halo of one (a1, gz2)
constexpr int kFW = kTW + 4, kFH = kTH + 4;  // with a halo of two (features)
constexpr int kFS = 37;                    // feature row stride
// Row stride and plane stride of the halo tiles. A warp reads either 32 columns of a row or (the weight
// gradients) 8 planes x 4 rows of a column: plane strides of 4 mod 32 and row strides of 3 mod 32 put
// both on 32 banks.
constexpr int kRS = 35, kPS = kHH * kRS + 14;
static_assert(kPS % 32 == 4 && kRS % 32 == 3 && kTT == 4 * 32 && kTH == 16, "bank layout");
constexpr int kHeadGrads = kGateParams - kW3;  // W3, b3; the loss follows
constexpr int kConvGrads = kW3;                // W1, b1, W2, b2

struct TrainShape {
    int n, w8, h8, tiles_x, tiles_y;
    long long tiles;
};

struct TrainTile {
    int fr, x0, y0;
};
__device__ __forceinline__ TrainTile train_tile(const TrainShape& s, long long t) {
    const int per = s.tiles_x * s.tiles_y;
    TrainTile r;
    r.fr = (int)(t / per);
    const int k = (int)(t - (long long)r.fr * per), ty = k / s.tiles_x;
    r.x0 = (k - ty * s.tiles_x) * kTW;
    r.y0 = ty * kTH;
    return r;
}

// The tile's features with a halo of two (zero outside the frame), loaded into registers a tile ahead so
// that their latency passes under the previous tile's arithmetic (packed in pairs), then put in place.
constexpr int kFPer = (kFW * kFH + kTT - 1) / kTT;
struct Features {
    __half2 v[kFPer / 2];
};
static_assert(kFPer % 2 == 0, "pairs");
__device__ __forceinline__ Features fetch_features(const __half* __restrict__ feat, const TrainShape& s, long long t) {
    const TrainTile T = train_tile(s, t);
    const __half* F = feat + (long long)T.fr * s.w8 * s.h8;
    __half h[kFPer];
#pragma unroll
    for (int j = 0; j < kFPer; ++j) {
        const int i = threadIdx.x + j * kTT, r = i / kFW, c = i - r * kFW;
        const int x = T.x0 - 2 + c, y = T.y0 - 2 + r;
        h[j] = (i < kFW * kFH && x >= 0 && x < s.w8 && y >= 0 && y < s.h8) ? F[(long long)y * s.w8 + x] : __float2half(0.f);
    }
    Features f;
#pragma unroll
    for (int j = 0; j < kFPer / 2; ++j) f.v[j] = __halves2half2(h[2 * j], h[2 * j + 1]);
    return f;
}
__device__ __forceinline__ void put_features(float* sf, const Features& f) {
#pragma unroll
    for (int j = 0; j < kFPer; ++j) {
        const int i = threadIdx.x + j * kTT, r = i / kFW;
        if (i < kFW * kFH) sf[r * kFS + (i - r * kFW)] = __half2float((j & 1) ? __high2half(f.v[j / 2]) : __low2half(f.v[j / 2]));
    }
}

// W1 as [tap][map]
__device__ __forceinline__ void load_w1(float (*w)[kGC], float* b, const float* __restrict__ P) {
    for (int i = threadIdx.x; i < kGC * 9; i += kTT) w[i % 9][i / 9] = P[kW1 + i];
    if (threadIdx.x < kGC) b[threadIdx.x] = P[kB1 + threadIdx.x];
}

// a1 (rounded to binary16, zero outside the frame) of the tile with a halo of one. Five pixels a thread,
// so that a weight is loaded once for five products.
__device__ __forceinline__ void compute_a1(float* a1, const float* sf, const float (*w)[kGC], const float* b, const TrainShape& s, const TrainTile& T) {
    constexpr int kPx = (kHW * kHH + kTT - 1) / kTT;
    int at[kPx];
    f2_t z[kPx][kGC / 2];
#pragma unroll
    for (int j = 0; j < kPx; ++j) {
        const int p = min((int)threadIdx.x + j * kTT, kHW * kHH - 1), r = p / kHW;
        at[j] = r * kFS + (p - r * kHW);
#pragma unroll
        for (int c = 0; c < kGC / 2; ++c) z[j][c] = f2_ld(reinterpret_cast<const float2*>(b)[c]);
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        f2_t wk[kGC / 2];
#pragma unroll
        for (int c = 0; c < kGC / 2; ++c) wk[c] = f2_ld(reinterpret_cast<const float2*>(w[k])[c]);
#pragma unroll
        for (int j = 0; j < kPx; ++j) {
            const f2_t v = f2_dup(sf[at[j] + (k / 3) * kFS + k % 3]);
#pragma unroll
            for (int c = 0; c < kGC / 2; ++c) z[j][c] = f2_fma(v, wk[c], z[j][c]);
        }
    }
#pragma unroll
    for (int j = 0; j < kPx; ++j) {
        const int p = threadIdx.x + j * kTT;
        if (p >= kHW * kHH) break;
        const int r = p / kHW, c = p - r * kHW;
        const int x = T.x0 - 1 + c, y = T.y0 - 1 + r;
        const bool in = x >= 0 && x < s.w8 && y >= 0 && y < s.h8;
#pragma unroll
        for (int m = 0; m < kGC; ++m) {
            const float v = (m & 1) ? f2_hi(z[j][m / 2]) : f2_lo(z[j][m / 2]);
            a1[m * kPS + r * kRS + c] = in ? __half2float(__float2half(lrelu(v))) : 0.f;
        }
    }
}

// A warp's four rows x 32 columns of a 3x3 convolution of 8 planes into 8: acc[row][plane pair] += in
// (halo tile) x w[plane][tap][8]; tap k reads halo position (row + k / 3, column + k % 3), or with kFlip
// (the transposed convolution) row + 2 - k / 3, column + 2 - k % 3. Packed over output planes; a weight
// load serves four pixels.
template <bool kFlip>
__device__ __forceinline__ void conv_rows(f2_t (*acc)[kGC / 2], const float* in, const float (*w)[9][kGC]) {
#pragma unroll 1
    for (int p = 0; p < kGC; ++p) {
        float v[6][3];
        const float* src = in + p * kPS + (threadIdx.x >> 5) * 4 * kRS + (threadIdx.x & 31);
#pragma unroll
        for (int r = 0; r < 6; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) v[r][c] = src[r * kRS + c];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const float4 wa = *reinterpret_cast<const float4*>(&w[p][k][0]), wb = *reinterpret_cast<const float4*>(&w[p][k][4]);
            const f2_t wk[4] = {f2_pack(wa.x, wa.y), f2_pack(wa.z, wa.w), f2_pack(wb.x, wb.y), f2_pack(wb.z, wb.w)};
            const int dr = kFlip ? 2 - k / 3 : k / 3, dc = kFlip ? 2 - k % 3 : k % 3;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const f2_t x = f2_dup(v[j + dr][dc]);
#pragma unroll
                for (int c = 0; c < kGC / 2; ++c) acc[j][c] = f2_fma(x, wk[c], acc[j][c]);
            }
        }
    }
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct ForwardSmem {
    float a1[kGC * kPS];
    float f[kFH * kFS];
    alignas(16) float w1[9][kGC];
    alignas(16) float b1[kGC];
    alignas(16) float w2[kGC][9][kGC];  // [input map][tap][map]
    alignas(16) float b2[kGC];
    float w3[kGK][kGC], b3[kGK];
    float red[kTT / 32][kHeadGrads + 1];
};

// Forward pass, loss, the head's gradients (part[block][kHeadGrads + 1], the loss last), and per pooled
// cell the gradient of its 8 averages (gq) and per pixel the signs of a2 (a bit a map). A lane pair's
// 2 x 4 pixels are two cells, one a lane.
// Bound by the fp32 pipe (652 multiply-adds a pixel, 58 % busy) and the latency between its barriers: 0.1 ms
// for 64 frames of 240 x 135.
__global__ void __launch_bounds__(kTT, 4) gate_forward_kernel(const float* __restrict__ P, const __half* __restrict__ feat,
                                                              const uint8_t* __restrict__ labels, const TrainShape s, float pos_weight,
                                                              float inv_cells, float4* __restrict__ gq, uint8_t* __restrict__ signs,
                                                              float* __restrict__ part) {
    __shared__ ForwardSmem S;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    load_w1(S.w1, S.b1, P);
    for (int i = threadIdx.x; i < kGC * kGC * 9; i += kTT) S.w2[(i / 9) % kGC][i % 9][i / (9 * kGC)] = P[kW2 + i];
    if (threadIdx.x < kGC) S.b2[threadIdx.x] = P[kB2 + threadIdx.x];
    if (threadIdx.x < kGK * kGC) S.w3[threadIdx.x / kGC][threadIdx.x % kGC] = P[kW3 + threadIdx.x];
    if (threadIdx.x < kGK) S.b3[threadIdx.x] = P[kB3 + threadIdx.x];
    const int w16 = s.w8 / 2, h16 = s.h8 / 2;
    const long long cells = (long long)w16 * h16;
    f2_t gw[kGK][kGC / 2];
    float gb[kGK], loss = 0.f;
#pragma unroll
    for (int k = 0; k < kGK; ++k) {
        gb[k] = 0.f;
#pragma unroll
        for (int c = 0; c < kGC / 2; ++c) gw[k][c] = 0ull;
    }
    Features next = fetch_features(feat, s, blockIdx.x);
    for (long long t = blockIdx.x; t < s.tiles; t += gridDim.x) {
        const TrainTile T = train_tile(s, t);
        put_features(S.f, next);
        __syncthreads();  // also: every warp is done with the previous tile's a1
        if (t + gridDim.x < s.tiles) next = fetch_features(feat, s, t + gridDim.x);
        // this lane's cell and its labels (a bit an octave)
        const int x = T.x0 + lane, y = T.y0 + 4 * warp;
        const int X = x >> 1, Y = (y >> 1) + (lane & 1);
        const bool live = X < w16 && Y < h16;
        const long long cell = (long long)Y * w16 + X;
        uint32_t lab = 0;
        if (live) {
            const uint8_t* lb = labels + (long long)T.fr * kGK * cells + cell;
#pragma unroll
            for (int k = 0; k < kGK; ++k) lab |= (uint32_t)(lb[k * cells] != 0) << k;
        }
        compute_a1(S.a1, S.f, S.w1, S.b1, s, T);
        __syncthreads();
        f2_t z[4][kGC / 2];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int c = 0; c < kGC / 2; ++c) z[j][c] = f2_ld(reinterpret_cast<const float2*>(S.b2)[c]);
        conv_rows<false>(z, S.a1, S.w2);
        // a2 (binary16), its signs, and the sums of rows (0, 1) and (2, 3)
        uint32_t sg[4] = {0u, 0u, 0u, 0u};
        float own[kGC];
#pragma unroll
        for (int c = 0; c < kGC; ++c) {
            float a[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                a[j] = __half2float(__float2half(lrelu((c & 1) ? f2_hi(z[j][c / 2]) : f2_lo(z[j][c / 2]))));
                sg[j] |= (a[j] > 0.f ? 1u : 0u) << c;
            }
            const float top = a[0] + a[1], bot = a[2] + a[3];
            // the even lane's cell takes both columns of the upper rows, the odd lane's of the lower ones
            const float other = __shfl_xor_sync(0xffffffffu, (lane & 1) ? top : bot, 1);
            own[c] = 0.25f * (((lane & 1) ? bot : top) + other);
        }
        if (x < s.w8) {
            uint8_t* o = signs + ((long long)T.fr * s.h8 + y) * s.w8 + x;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (y + j < s.h8) o[(long long)j * s.w8] = (uint8_t)sg[j];
        }
        if (live) {
            f2_t g8[kGC / 2], q2[kGC / 2];
#pragma unroll
            for (int c = 0; c < kGC / 2; ++c) {
                g8[c] = 0ull;
                q2[c] = f2_pack(own[2 * c], own[2 * c + 1]);
            }
#pragma unroll
            for (int k = 0; k < kGK; ++k) {
                float v = S.b3[k];
#pragma unroll
                for (int c = 0; c < kGC; ++c) v = fmaf(S.w3[k][c], own[c], v);
                const float p = 1.f / (1.f + expf(-v));
                const bool pos = (lab >> k) & 1u;
                // positive-weighted binary cross-entropy on the logit
                const float l = fminf(-logf(fmaxf(pos ? p : 1.f - p, 1e-7f)), 30.f);
                loss += (pos ? pos_weight * l : l) * inv_cells;
                const float g = (pos ? p * pos_weight - pos_weight : p) * inv_cells;
                gb[k] += g;
                const f2_t gg = f2_dup(g);
#pragma unroll
                for (int c = 0; c < kGC / 2; ++c) {
                    gw[k][c] = f2_fma(gg, q2[c], gw[k][c]);
                    g8[c] = f2_fma(gg, f2_pack(S.w3[k][2 * c], S.w3[k][2 * c + 1]), g8[c]);
                }
            }
            float4* o = gq + ((long long)T.fr * cells + cell) * 2;
            o[0] = make_float4(f2_lo(g8[0]), f2_hi(g8[0]), f2_lo(g8[1]), f2_hi(g8[1]));
            o[1] = make_float4(f2_lo(g8[2]), f2_hi(g8[2]), f2_lo(g8[3]), f2_hi(g8[3]));
        }
    }
#pragma unroll
    for (int k = 0; k < kGK; ++k) {
#pragma unroll
        for (int c = 0; c < kGC; ++c) {
            const float v = warp_sum((c & 1) ? f2_hi(gw[k][c / 2]) : f2_lo(gw[k][c / 2]));
            if (lane == 0) S.red[warp][k * kGC + c] = v;
        }
        const float v = warp_sum(gb[k]);
        if (lane == 0) S.red[warp][kGK * kGC + k] = v;
    }
    loss = warp_sum(loss);
    if (lane == 0) S.red[warp][kHeadGrads] = loss;
    __syncthreads();
    if (threadIdx.x <= kHeadGrads)
        part[(long long)blockIdx.x * (kHeadGrads + 1) + threadIdx.x] =
            (S.red[0][threadIdx.x] + S.red[1][threadIdx.x]) + (S.red[2][threadIdx.x] + S.red[3][threadIdx.x]);
}

struct BackwardSmem {
    float a1[kGC * kPS];
    float g[kGC * kPS];  // gz2 with its halo, then gz1; at the end the blocks' sums
    float f[kFH * kFS];
    alignas(16) float w1[9][kGC];
    alignas(16) float b1[kGC];
    alignas(16) float w2[kGC][9][kGC];  // [map][tap][input map]
};

// gz2 = d loss / d z2 of the tile and a halo of one from the cells' gradients and the signs of a2 (zero
// outside the frame and past its last whole cell); sum += those of the tile
__device__ __forceinline__ void load_gz2(float* g, float* sum, const float4* __restrict__ gq, const uint8_t* __restrict__ signs, const TrainShape& s,
                                         const TrainTile& T) {
    constexpr int kCW = kTW / 2 + 2, kCH = kTH / 2 + 2;
    const int w16 = s.w8 / 2, h16 = s.h8 / 2;
#pragma unroll
    for (int i = threadIdx.x; i < kCW * kCH; i += kTT) {
        const int r = i / kCW, c = i - r * kCW;
        const int X = T.x0 / 2 - 1 + c, Y = T.y0 / 2 - 1 + r;
        const bool in = X >= 0 && X < w16 && Y >= 0 && Y < h16;
        float q[kGC];
        uint32_t sg[4] = {0u, 0u, 0u, 0u};
        if (in) {
            const float4* src = gq + (((long long)T.fr * h16 + Y) * w16 + X) * 2;
            const float4 a = src[0], b = src[1];
            q[0] = 0.25f * a.x;
            q[1] = 0.25f * a.y;
            q[2] = 0.25f * a.z;
            q[3] = 0.25f * a.w;
            q[4] = 0.25f * b.x;
            q[5] = 0.25f * b.y;
            q[6] = 0.25f * b.z;
            q[7] = 0.25f * b.w;
            const uint8_t* m = signs + ((long long)T.fr * s.h8 + 2 * Y) * s.w8 + 2 * X;
            sg[0] = m[0];
            sg[1] = m[1];
            sg[2] = m[s.w8];
            sg[3] = m[s.w8 + 1];
        } else {
#pragma unroll
            for (int k = 0; k < kGC; ++k) q[k] = 0.f;
        }
        const bool core = c >= 1 && c <= kTW / 2 && r >= 1 && r <= kTH / 2;
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            const int hx = 2 * c - 1 + (d & 1), hy = 2 * r - 1 + (d >> 1);  // in the halo tile
            if (hx < 0 || hx >= kHW || hy < 0 || hy >= kHH) continue;
#pragma unroll
            for (int k = 0; k < kGC; ++k) {
                const float v = ((sg[d] >> k) & 1u) ? q[k] : 0.1f * q[k];
                g[k * kPS + hy * kRS + hx] = v;
                if (core) sum[k] += v;
            }
        }
    }
}

// The convolutions' gradients (part[block][kConvGrads]) from gz2: W2's (8 x 8 x 9 sums of gz2 x a1 over the
// pixels), gz1 by the transposed convolution, and W1's (8 x 9 sums of gz1 x f). For W2's a lane holds
// the 72 sums of one input map (lane % 8) over the rows lane / 8 of its warp's four; for W1's the 9 of one
// map. Bound by the fp32 pipe (1,296 multiply-adds a pixel, 58 % busy) and its five barriers a tile, with
// three blocks a SM (the 72 + 9 sums a thread): 0.17 ms for 64 frames of 240 x 135.
__global__ void __launch_bounds__(kTT, 3) gate_backward_kernel(const float* __restrict__ P, const __half* __restrict__ feat,
                                                               const float4* __restrict__ gq, const uint8_t* __restrict__ signs,
                                                               const TrainShape s, float* __restrict__ part) {
    __shared__ BackwardSmem S;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m8 = lane & 7, row = 4 * warp + (lane >> 3);
    load_w1(S.w1, S.b1, P);
    for (int i = threadIdx.x; i < kGC * kGC * 9; i += kTT) S.w2[i / (9 * kGC)][i % 9][(i / 9) % kGC] = P[kW2 + i];
    f2_t gw2[9][kGC / 2];  // of input map m8: [tap][map pair]
    float gw1[9], gb1 = 0.f, gb2[kGC];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        gw1[k] = 0.f;
#pragma unroll
        for (int c = 0; c < kGC / 2; ++c) gw2[k][c] = 0ull;
    }
#pragma unroll
    for (int c = 0; c < kGC; ++c) gb2[c] = 0.f;
    Features next = fetch_features(feat, s, blockIdx.x);
    for (long long t = blockIdx.x; t < s.tiles; t += gridDim.x) {
        const TrainTile T = train_tile(s, t);
        __syncthreads();  // every warp is done with the previous tile
        put_features(S.f, next);
        load_gz2(S.g, gb2, gq, signs, s, T);
        __syncthreads();
        if (t + gridDim.x < s.tiles) next = fetch_features(feat, s, t + gridDim.x);
        compute_a1(S.a1, S.f, S.w1, S.b1, s, T);
        __syncthreads();
        {
            const float* gs = S.g + (row + 1) * kRS + 1;
            const float* as = S.a1 + m8 * kPS + row * kRS;
            float w[3][3];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                w[r][1] = as[r * kRS];
                w[r][2] = as[r * kRS + 1];
            }
#pragma unroll 8
            for (int x = 0; x < kTW; ++x) {
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    w[r][0] = w[r][1];
                    w[r][1] = w[r][2];
                    w[r][2] = as[r * kRS + x + 2];
                }
                f2_t gv[kGC / 2];
#pragma unroll
                for (int c = 0; c < kGC / 2; ++c) gv[c] = f2_pack(gs[2 * c * kPS + x], gs[(2 * c + 1) * kPS + x]);
#pragma unroll
                for (int k = 0; k < 9; ++k) {
                    const f2_t v = f2_dup(w[k / 3][k % 3]);
#pragma unroll
                    for (int c = 0; c < kGC / 2; ++c) gw2[k][c] = f2_fma(v, gv[c], gw2[k][c]);
                }
            }
        }
        f2_t ga[4][kGC / 2];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int c = 0; c < kGC / 2; ++c) ga[j][c] = 0ull;
        conv_rows<true>(ga, S.g, S.w2);
        __syncthreads();  // gz2 is read; gz1 takes its place
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int o = (4 * warp + j + 1) * kRS + lane + 1;
            const bool in = T.x0 + lane < s.w8 && T.y0 + 4 * warp + j < s.h8;
#pragma unroll
            for (int c = 0; c < kGC; ++c) {
                const float v = (c & 1) ? f2_hi(ga[j][c / 2]) : f2_lo(ga[j][c / 2]);
                S.g[c * kPS + o] = in ? (S.a1[c * kPS + o] > 0.f ? v : 0.1f * v) : 0.f;
            }
        }
        __syncthreads();
        {
            const float* gs = S.g + m8 * kPS + (row + 1) * kRS + 1;
            const float* fs = S.f + (row + 1) * kFS + 1;
            float w[3][3];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                w[r][1] = fs[r * kFS];
                w[r][2] = fs[r * kFS + 1];
            }
#pragma unroll 8
            for (int x = 0; x < kTW; ++x) {
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    w[r][0] = w[r][1];
                    w[r][1] = w[r][2];
                    w[r][2] = fs[r * kFS + x + 2];
                }
                const float g = gs[x];
                gb1 += g;
#pragma unroll
                for (int k = 0; k < 9; ++k) gw1[k] = fmaf(g, w[k / 3][k % 3], gw1[k]);
            }
        }
    }
    // the four row lanes of a map, then the four warps
    __syncthreads();
    float* out = S.g + warp * kConvGrads;
    static_assert(4 * kConvGrads <= kGC * kPS, "the warps' sums fit the gradient tile");
    auto rows_sum = [](float v) {
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        return v + __shfl_xor_sync(0xffffffffu, v, 16);
    };
#pragma unroll
    for (int k = 0; k < 9; ++k) {
#pragma unroll
        for (int c = 0; c < kGC; ++c) {
            const float v = rows_sum((c & 1) ? f2_hi(gw2[k][c / 2]) : f2_lo(gw2[k][c / 2]));
            if (lane < kGC) out[kW2 + (c * kGC + lane) * 9 + k] = v;
        }
        const float v = rows_sum(gw1[k]);
        if (lane < kGC) out[kW1 + lane * 9 + k] = v;
    }
    gb1 = rows_sum(gb1);
    if (lane < kGC) out[kB1 + lane] = gb1;
#pragma unroll
    for (int c = 0; c < kGC; ++c) {
        const float v = warp_sum(gb2[c]);
        if (lane == 0) out[kB2 + c] = v;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kConvGrads; i += kTT)
        part[(long long)blockIdx.x * kConvGrads + i] = (S.g[i] + S.g[kConvGrads + i]) + (S.g[2 * kConvGrads + i] + S.g[3 * kConvGrads + i]);
}

// Sums the blocks' gradients (32 threads a parameter, in a fixed order) and the loss; with P also one
// Adam step.
__global__ void __launch_bounds__(1024) gate_update_kernel(const float* __restrict__ conv, int n_conv, const float* __restrict__ head, int n_head,
                                                           float* __restrict__ grad, float* __restrict__ loss, float* __restrict__ P,
                                                           float* __restrict__ m, float* __restrict__ v, float lr, float b1t, float b2t) {
    __shared__ float sum[32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (i < kConvGrads) {
        for (int b = warp; b < n_conv; b += 32) s += conv[(long long)b * kConvGrads + i];
    } else if (i <= kGateParams) {
        for (int b = warp; b < n_head; b += 32) s += head[(long long)b * (kHeadGrads + 1) + i - kConvGrads];
    }
    sum[warp][lane] = s;
    __syncthreads();
    const float total = warp_sum(sum[lane][warp]);  // parameter blockIdx.x * 32 + warp
    const int p = blockIdx.x * 32 + warp;
    if (lane || p > kGateParams) return;
    if (p == kGateParams) {
        *loss = total;
        return;
    }
    if (grad) grad[p] = total;
    if (!P) return;
    const float mi = 0.9f * m[p] + 0.1f * total, vi = 0.999f * v[p] + 0.001f * total * total;
    m[p] = mi;
    v[p] = vi;
    const float mh = mi / (1.f - b1t), vh = vi / (1.f - b2t);
    P[p] -= lr * mh / (sqrtf(vh) + 1e-8f);
}

// One stream-ordered allocation for everything a run needs (from the device's pool, which gives it back to
// the system at a later synchronisation, or hands it to the next run: cudaMalloc and cudaFree took 0.6 ms
// a run on B200, as long as the kernels of two steps).
struct TrainBuffers {
    char* base = nullptr;
    float4* gq = nullptr;
    uint8_t* signs = nullptr;
    float *conv = nullptr, *head = nullptr, *grad = nullptr, *P = nullptr, *m = nullptr, *v = nullptr, *loss = nullptr;
    int fwd_grid = 0, bwd_grid = 0;

    cudaError_t alloc(int n, int w8, int h8, size_t n_loss) {
        int dev = 0, sms = 0, fwd = 0, bwd = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        // the shared memory of all resident blocks
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gate_backward_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fwd, gate_forward_kernel, kTT, 0);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bwd, gate_backward_kernel, kTT, 0);
        if (e != cudaSuccess) return e;
        fwd_grid = sms * std::max(1, fwd);
        bwd_grid = sms * std::max(1, bwd);
        size_t at = 0;
        auto take = [&](size_t bytes) {
            const size_t o = at;
            at += (bytes + 255) / 256 * 256;
            return o;
        };
        const size_t px = (size_t)n * w8 * h8, cells = (size_t)n * (w8 / 2) * (h8 / 2);
        const size_t oq = take(cells * 2 * sizeof(float4)), os = take(px);
        const size_t oc = take(sizeof(float) * kConvGrads * bwd_grid), oh = take(sizeof(float) * (kHeadGrads + 1) * fwd_grid);
        const size_t og = take(sizeof(float) * kGateParams), op = take(sizeof(float) * kGateParams), om = take(sizeof(float) * 2 * kGateParams);
        const size_t ol = take(sizeof(float) * n_loss);
        e = cudaMallocAsync((void**)&base, at, nullptr);
        if (e != cudaSuccess) return e;
        gq = (float4*)(base + oq);
        signs = (uint8_t*)(base + os);
        conv = (float*)(base + oc);
        head = (float*)(base + oh);
        grad = (float*)(base + og);
        P = (float*)(base + op);
        m = (float*)(base + om);
        v = m + kGateParams;
        loss = (float*)(base + ol);
        return cudaSuccess;
    }
    ~TrainBuffers() {
        if (base) cudaFreeAsync(base, nullptr);
    }
};

// One forward + backward pass over n frames: the gradient and the loss (written, not added to); with
// `adam` the step that follows (its two bias corrections at `step`).
cudaError_t gate_pass(const float* P, const __half* f, const uint8_t* labels, int n, int w8, int h8, float pos_weight, TrainBuffers& B, float* loss,
                      bool adam, float lr, int step, cudaStream_t st) {
    const long long cells = (long long)(w8 / 2) * (h8 / 2);
    const float inv_cells = 1.f / (float)(n * cells * kGK);
    TrainShape s;
    s.n = n;
    s.w8 = w8;
    s.h8 = h8;
    s.tiles_x = (w8 + kTW - 1) / kTW;
    s.tiles_y = (h8 + kTH - 1) / kTH;
    s.tiles = (long long)n * s.tiles_x * s.tiles_y;
    const int gf = (int)std::min<long long>(s.tiles, B.fwd_grid), gb = (int)std::min<long long>(s.tiles, B.bwd_grid);
    gate_forward_kernel<<<gf, kTT, 0, st>>>(P, f, labels, s, pos_weight, inv_cells, B.gq, B.signs, B.head);
    gate_backward_kernel<<<gb, kTT, 0, st>>>(P, f, B.gq, B.signs, s, B.conv);
    gate_update_kernel<<<(kGateParams + 1 + 31) / 32, 1024, 0, st>>>(B.conv, gb, B.head, gf, adam ? nullptr : B.grad, loss, adam ? B.P : nullptr, B.m, B.v,
                                                                     lr, powf(0.9f, (float)step), powf(0.999f, (float)step));
    return cudaGetLastError();
}

}  // namespace

}  // namespace ccnn

using namespace ccnn;

extern "C" CCNN_API ccnn_status ccnn_gate_gradient(const float* d_params, const void* d_feat, const unsigned char* d_labels, int n, int w8, int h8,
                                                   float pos_weight, float* grad_out, float* loss_out) {
    if (!d_params || !d_feat || !d_labels || n <= 0 || w8 < 2 || h8 < 2 || !grad_out || !loss_out) {
        set_error("invalid arguments");
        return CCNN_ERR_INVALID_ARG;
    }
    TrainBuffers B;
    cudaError_t e = B.alloc(n, w8, h8, 1);
    if (e == cudaSuccess) e = gate_pass(d_params, (const __half*)d_feat, d_labels, n, w8, h8, pos_weight, B, B.loss, false, 0.f, 0, nullptr);
    if (e == cudaSuccess) e = cudaMemcpy(grad_out, B.grad, sizeof(float) * kGateParams, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(loss_out, B.loss, sizeof(float), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        set_error(std::string("gate gradient: ") + cudaGetErrorString(e));
        return CCNN_ERR_CUDA;
    }
    return CCNN_OK;
}

// Adam over mini-batches of `batch` frames taken in order, `epochs` times; params (host, fp32)
// are read as the start point and overwritten with the result; losses[e] = mean loss of epoch e. The
// host waits once a pass over the data (its steps' losses come back together).
extern "C" CCNN_API ccnn_status ccnn_gate_train(float* params, const void* d_feat, const unsigned char* d_labels, int n, int w8, int h8, int batch,
                                                int epochs, float lr, float pos_weight, float* losses) {
    if (!params || !d_feat || !d_labels || n <= 0 || batch <= 0 || epochs <= 0 || w8 < 2 || h8 < 2) {
        set_error("invalid arguments");
        return CCNN_ERR_INVALID_ARG;
    }
    batch = std::min(batch, n);
    const int nb = n / batch;
    TrainBuffers B;
    cudaError_t e = B.alloc(batch, w8, h8, nb);
    if (e == cudaSuccess) e = cudaMemcpy(B.P, params, sizeof(float) * kGateParams, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemsetAsync(B.m, 0, sizeof(float) * 2 * kGateParams, nullptr);
    const size_t fplane = (size_t)w8 * h8, lplane = (size_t)kGK * (w8 / 2) * (h8 / 2);
    std::vector<float> step_loss(nb);
    int step = 0;
    for (int ep = 0; ep < epochs && e == cudaSuccess; ++ep) {
        for (int b = 0; b < nb && e == cudaSuccess; ++b)
            e = gate_pass(B.P, (const __half*)d_feat + b * (size_t)batch * fplane, d_labels + b * (size_t)batch * lplane, batch, w8, h8, pos_weight, B,
                          B.loss + b, true, lr, ++step, nullptr);
        if (e == cudaSuccess) e = cudaMemcpy(step_loss.data(), B.loss, sizeof(float) * nb, cudaMemcpyDeviceToHost);
        double ep_loss = 0.0;
        for (const float l : step_loss) ep_loss += l;
        if (losses) losses[ep] = (float)(ep_loss / nb);
    }
    if (e == cudaSuccess) e = cudaMemcpy(params, B.P, sizeof(float) * kGateParams, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        set_error(std::string("gate training: ") + cudaGetErrorString(e));
        return CCNN_ERR_CUDA;
    }
    return CCNN_OK;
}
