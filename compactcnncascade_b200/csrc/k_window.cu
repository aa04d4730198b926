// Stage-2/3 window CNNs on the compacted stage-1 candidates.
//
// Reference: CNNDetector::CPUCheckDetect (src/CNNObjectDetector/cnn_detector_v3.cpp:1485-1818):
//   crop  x = int((px-6)/s), y = int((py-5)/s), w = int(36/s), h = int(38/s)  (:1492-1495)
//   retry window (mod 1) shrunk by 15 % (:1535-1542), clamped to the frame (:1553-1556)
//   nearest-neighbour resize to 49 x 51 (:1565), byte rounding uchar(v + 0.5) (image_proc.cpp:365),
//   histogram equalisation (image_proc.cpp:720-799),
//   stage 2 on columns 2..48 (UCharToFloat offset 2, image_proc.cpp:417-427),
//   stage 3 on the mirror of columns 0..46 (UCharToFloat_inv, image_proc.cpp:478-490),
//   4x4 response maps counted against treshold_2 / treshold_3 with the type_check early exits
//   (:1655-1706) and the accept rule (:1709-1725); score s0 + k1*max(-1.7159, m1) + k2*max(-1.7159, m2).
//
// Every candidate is evaluated speculatively: both nets on both the first and the retry window,
// as independent CTA work items. Which of them the reference would have reached (early exits,
// retry, drop_detect) is decided by the replay kernel, so the verdicts are the same while all
// items run in parallel.
//
// Bound by latency and barriers as much as by the fp32 pipe: an item is a chain of small layers. With L1 packed over
// pixels 11 columns apart (operands load as pairs; map pairs needed every input converted and duplicated), weights
// loaded once for four positions, the layers whose lanes read different maps taken off the constant bank, and the
// crop a row a warp, 32 gated 1920x1080 frames on B200 go from 1.64 to 1.50 ms and 16 monochrome 1280x720 ones from
// 0.88 to 0.79 ms.
//
// One CTA (256 threads) per work item, persistent over the item list. The networks run
// entirely in shared memory: L1 (6 maps, 44x48 -> pooled 22x24), neighbour sums, L2 (12 maps,
// 20x22 -> pooled 10x11), sums, L3 (24 maps, 7w x 8h -> 4x4), hidden layer and output neuron.
#include "kernels.h"
#include "resample.cuh"
#include "window_common.cuh"
#include "legacy_dev.cuh"

namespace ccnn {

constexpr int kWT = 256;
constexpr int kP1W = 22, kP1H = 24;   // pooled L1 of a 47x51 window
constexpr int kP2W = 10, kP2H = 11;   // pooled L2
constexpr int kOutN = 16;             // 4x4 response map

constexpr int kHalfW = kP1W / 2;      // 11: L1 pixels x and x + 11 of a row run as a packed pair
constexpr int kP1Pairs = kHalfW * kP1H;
constexpr int kInPairs = 2 * kHalfW + 3;  // 25 columns of a row of input pairs

constexpr int kMaxRest = 16;  // L1 pairs (CNTK) or pixels (legacy) past the whole passes

struct WindowSmem {
    uint8_t crop[kCropH][kCropW + 3];
    int hist[256];
    int lut[256];
    float s1[6][kP1H][kP1W + 1];
    union {
        // the network's input: column c next to column c + 22 (the windows of L1 pixels x and x + 11 load as packed
        // pairs), even columns, then odd ones (L1 steps by two); the row stride spreads a warp's rows over the banks
        float2 in[kCropH][2][15];
        struct {  // after L1
            float p2[12][kP2H][kP2W + 1];
            float s2[12][kP2H][kP2W + 1];
            float a3[24][kOutN];
        } l;
    } u;
    union {
        alignas(16) float2 k3[12][56];  // L3 taps of the network that runs
        float hbuf[84][kOutN];          // after L3
    } v;
    float out[kOutN];
    float2 l1rest[kMaxRest][6];  // pooled L1 maps of the partial pass's pixels
    int geo[4];
};
static_assert(kInPairs <= 30, "columns of an input row");
// six resident blocks a SM (a schedule knob's value): 228 KB, of which each block also takes its static 32 bytes and
// 1 KB, in steps of 128 bytes
static_assert(6 * ((sizeof(WindowSmem) + 32 + 1024 + 127) / 128 * 128) <= 228 * 1024, "six blocks a SM");

// mode: 0 = stage-2 view (columns 2..48), 1 = mirrored (46 - x), 2 = plain (columns 0..46)
__device__ __forceinline__ float win_in(const WindowSmem& S, int mode, int x, int y) {
    int c = mode == 0 ? x + kXOff : (mode == 1 ? (kWinW - 1) - x : x);
    return (float)S.crop[y][c];
}

// Two consecutive duplicated parameters by one 16-byte constant load.
__device__ __forceinline__ ulonglong2 ld_two(const float2* p) { return *reinterpret_cast<const ulonglong2*>(p); }

// One CNTK window network. W: its parameters as kernel parameters (warp-uniform constant loads); G: the same in
// global memory, for the layers whose lanes read different maps (their constant loads took a pass a map: L3's 56
// taps 90 cycles each): L3's taps are copied to shared memory while L1 and L2 run.
template <class NW>
__device__ void window_net(const NW& W, const NW* __restrict__ G, WindowSmem& S, int mode) {
    static_assert(NW::kM1 == 6 && NW::kM2 == 12 && NW::kM3 == 24 && NW::kK3W * NW::kK3H == 56 && NW::kHS % 2 == 0, "shared-memory layout");
    const f2_t nz = f2_ld(W.negzero);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < (int)sizeof(S.v.k3) / 16; i += kWT) {
        const unsigned dst = (unsigned)__cvta_generic_to_shared(reinterpret_cast<char*>(S.v.k3) + 16 * i);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(reinterpret_cast<const char*>(G->k3p) + 16 * i) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    if (lane < kInPairs)
        for (int y = warp; y < kCropH; y += kWT / 32)
            S.u.in[y][lane & 1][lane >> 1] = make_float2(win_in(S, mode, lane, y), win_in(S, mode, lane + 2 * kHalfW, y));
    __syncthreads();
    // L1: conv 4x4 + folded BN/LReLU + 2x2 max, then neighbour sums (add / add2), on the pixels x and x + 11 at
    // once. 256 pairs take a pass of every map a thread; the last 8 are split into (pair, map) units, one
    // warp a map, so that they take a sixth of a pass.
    constexpr int kRest = kP1Pairs - kWT;
    static_assert(kRest > 0 && kRest <= kMaxRest && NW::kM1 <= kWT / 32, "one full pass, the rest a warp a map");
    auto pooled = [&](const f2_t (&win)[5][5], int m) {
        f2_t c[4];
#pragma unroll
        for (int k = 0; k < 16; k += 2) {
            const ulonglong2 w = ld_two(&W.k1d[m][k]);
#pragma unroll
            for (int d = 0; d < 4; ++d) {
                const int dy = d >> 1, dx = d & 1;
                const f2_t a = f2_mul(win[dy + (k >> 2)][dx + (k & 3)], w.x, nz);
                c[d] = f2_add(k ? f2_add(c[d], a) : a, f2_mul(win[dy + (k >> 2)][dx + (k & 3) + 1], w.y, nz));
            }
        }
#pragma unroll
        for (int d = 0; d < 4; ++d) c[d] = lrelu_bn2(c[d], W.a1d[m], nz);
        return f2_max4(c[0], c[1], c[2], c[3]);
    };
    auto put = [&](int m, int x, int y, f2_t v) {
        S.s1[m][y][x] = f2_lo(v);
        S.s1[m][y][x + kHalfW] = f2_hi(v);
    };
    for (int p = threadIdx.x; p < kWT + 32 * NW::kM1; p += kWT) {
        const bool unit = p >= kWT;  // one map (warp-uniform) of a pair of the partial pass
        if (unit && lane >= kRest) continue;
        const int pair = unit ? kWT + lane : p;
        const int x = pair % kHalfW, y = pair / kHalfW;
        f2_t win[5][5];
#pragma unroll
        for (int r = 0; r < 5; ++r)
#pragma unroll
            for (int c = 0; c < 5; ++c) win[r][c] = f2_ld(S.u.in[2 * y + r][c & 1][x + (c >> 1)]);
        if (unit) {
            *reinterpret_cast<f2_t*>(&S.l1rest[lane][warp]) = pooled(win, warp);
            continue;
        }
        f2_t before = 0ull, last = pooled(win, 0);  // maps m - 2 and m - 1
#pragma unroll 1
        for (int m = 1; m < NW::kM1; ++m) {
            const f2_t v = pooled(win, m);
            const f2_t two = m == 1 ? last : f2_add(before, last);
            put(m - 1, x, y, f2_add(two, v));
            before = last;
            last = v;
        }
        put(NW::kM1 - 1, x, y, f2_add(before, last));
    }
    __syncthreads();
    if (threadIdx.x < kRest) {
        const int x = (kWT + threadIdx.x) % kHalfW, y = (kWT + threadIdx.x) / kHalfW;
        f2_t P[NW::kM1];
#pragma unroll
        for (int k = 0; k < NW::kM1; ++k) P[k] = f2_ld(S.l1rest[threadIdx.x][k]);
        put(0, x, y, f2_add(P[0], P[1]));
#pragma unroll
        for (int k = 1; k < NW::kM1 - 1; ++k) put(k, x, y, f2_add(f2_add(P[k - 1], P[k]), P[k + 1]));
        put(NW::kM1 - 1, x, y, f2_add(P[NW::kM1 - 2], P[NW::kM1 - 1]));
    }
    __syncthreads();
    // L2: map pair (2i, 2i+1) convolves sum map i; 3x3 + BN/LReLU + 2x2 max
    for (int it = threadIdx.x; it < kP2W * kP2H * NW::kM1; it += kWT) {
        const int i = it / (kP2W * kP2H);
        const int p = it - i * (kP2W * kP2H);
        const int x = p % kP2W, y = p / kP2W;
        f2_t q[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) q[r][c] = f2_dup(S.s1[i][2 * y + r][2 * x + c]);
        f2_t cv[4];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const f2_t w = f2_ld(W.k2p[i][k]);
#pragma unroll
            for (int d = 0; d < 4; ++d) {
                const f2_t a = f2_mul(q[(d >> 1) + k / 3][(d & 1) + k % 3], w, nz);
                cv[d] = k ? f2_add(cv[d], a) : a;
            }
        }
#pragma unroll
        for (int d = 0; d < 4; ++d) cv[d] = lrelu_bn2(cv[d], W.a2p[i], nz);
        const f2_t pm = f2_max4(cv[0], cv[1], cv[2], cv[3]);
        S.u.l.p2[2 * i][y][x] = f2_lo(pm);
        S.u.l.p2[2 * i + 1][y][x] = f2_hi(pm);
    }
    __syncthreads();
    for (int p = threadIdx.x; p < kP2W * kP2H; p += kWT) {
        const int x = p % kP2W, y = p / kP2W;
        constexpr int M = NW::kM2;
        S.u.l.s2[0][y][x] = fadd(S.u.l.p2[0][y][x], S.u.l.p2[1][y][x]);
        for (int k = 1; k < M - 1; ++k) S.u.l.s2[k][y][x] = fadd(fadd(S.u.l.p2[k - 1][y][x], S.u.l.p2[k][y][x]), S.u.l.p2[k + 1][y][x]);
        S.u.l.s2[M - 1][y][x] = fadd(S.u.l.p2[M - 2][y][x], S.u.l.p2[M - 1][y][x]);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    // L3: 7w x 8h conv summed in one left-to-right chain (conv_8x7), BN/LReLU, no pooling;
    // maps (2i, 2i+1) share the input: packed
    for (int it = threadIdx.x; it < (NW::kM3 / 2) * kOutN; it += kWT) {
        const int i = it / kOutN, o = it - i * kOutN;
        const int ox = o & 3, oy = o >> 2;
        f2_t acc = f2_mul(f2_dup(S.u.l.s2[i][oy][ox]), f2_ld(S.v.k3[i][0]), nz);
#pragma unroll
        for (int k = 1; k < NW::kK3W * NW::kK3H; ++k)
            acc = f2_add(acc, f2_mul(f2_dup(S.u.l.s2[i][oy + k / NW::kK3W][ox + k % NW::kK3W]), f2_ld(S.v.k3[i][k]), nz));
        const f2_t av = lrelu_bn2(acc, G->a3p[i], nz);
        S.u.l.a3[2 * i][o] = f2_lo(av);
        S.u.l.a3[2 * i + 1][o] = f2_hi(av);
    }
    __syncthreads();
    // hidden neurons n = HS*i + t read L3 maps i .. i+CONN-1; neurons (2q, 2q+1) share the
    // group, so they run as one packed pair
    for (int it = threadIdx.x; it < (NW::kHL / 2) * kOutN; it += kWT) {
        const int q = it / kOutN, o = it - q * kOutN;
        const int n = 2 * q;
        const int i = n / NW::kHS;
        f2_t s = f2_pack(__ldg(&G->hb[n]), __ldg(&G->hb[n + 1]));
#pragma unroll
        for (int j = 0; j < NW::kConn; ++j) s = f2_add(s, f2_mul(f2_dup(S.u.l.a3[i + j][o]), f2_ld(G->hwp[q][j]), nz));
        s = f2_mul(s, f2_dup(__ldg(&G->htw[i])), nz);
        const f2_t half = f2_pack(0.5f, 0.5f);
        const f2_t v = f2_add(f2_mul(half, tanh_rational2(s, nz), nz), half);
        const int t = n - i * NW::kHS;  // neurons n, n+1 are slots t, t+1 of group i
        const f2_t h = f2_add(f2_mul(f2_pack(__ldg(&G->hbnw[t]), __ldg(&G->hbnw[t + 1])), v, nz), f2_pack(__ldg(&G->hbnb[t]), __ldg(&G->hbnb[t + 1])));
        S.v.hbuf[n][o] = f2_lo(h);
        S.v.hbuf[n + 1][o] = f2_hi(h);
    }
    __syncthreads();
    if (threadIdx.x < kOutN) {
        const int o = threadIdx.x;
        float acc = fmul(S.v.hbuf[0][o], W.ow[0]);
        for (int n = 1; n < NW::kHL; ++n) acc = fadd(fmul(S.v.hbuf[n][o], W.ow[n]), acc);
        float c = fmul(fadd(acc, W.ob), W.otw);
        c = tanh_rational(c);
        S.out[o] = (W.af == 0.f) ? fadd(fmul(0.5f, c), 0.5f) : fmul(W.af, c);
    }
    __syncthreads();
}

// The legacy (format 1.0) stage-2/3 networks on the window in shared memory: the sums of neighbouring L1 maps
// (6 maps, 22x24 pooled) in S.s1, L2 (12 maps, 10x11) in S.u.l.p2 and their sums in S.u.l.s2, the L3 values of the
// 16 outputs in S.u.l.a3, fully connected hidden neurons in S.v.hbuf; the arithmetic of the standalone legacy
// forward pass (legacy_dev.cuh), map pairs packed, spread over the block. As in window_net, whole passes of
// L1 pixels take every map pair a thread and the pixels of the last, partial pass one pair a warp. The windows
// of a 640 x 480 frame took 81 us on B200 with one map a thread and the map sums made tap by tap, now 40.
__device__ void legacy_window_net(const LegacyNet& W, WindowSmem& S, int mode, f2_t nz) {
    constexpr int kP2 = kP2W * kP2H;
    constexpr int kM0 = 6;  // the most first-layer maps of a stage-2/3 network
    constexpr int kFull = (kP1W * kP1H / kWT) * kWT, kRest = kP1W * kP1H - kFull, kMP = kM0 / 2;
    static_assert(kRest > 0 && kRest <= kMaxRest && 32 * kMP <= kWT, "partial L1 pass must fit one warp per map pair");
    const int m0 = W.m0;
    const f2_t af = f2_dup(W.af);
    auto sums = [&](const float (&P)[kM0], int px) {
        const int x = px % kP1W, y = px / kP1W;
#pragma unroll
        for (int k = 0; k < kM0; ++k)
            if (k < m0) S.s1[k][y][x] = lg_neighbour_sum(P, k, m0);
    };
    for (int p = threadIdx.x; p < kFull + 32 * kMP; p += kWT) {
        const bool unit = p >= kFull;  // one map pair (warp-uniform) of a pixel of the partial pass
        if (unit && ((p - kFull) & 31) >= kRest) continue;
        const int px = unit ? kFull + ((p - kFull) & 31) : p;
        const int mp0 = unit ? (p - kFull) >> 5 : 0;
        const int x = px % kP1W, y = px / kP1W;
        f2_t win[5][5];
#pragma unroll
        for (int r = 0; r < 5; ++r)
#pragma unroll
            for (int c = 0; c < 5; ++c) win[r][c] = f2_dup(win_in(S, mode, 2 * x + c, 2 * y + r));
        float P[kM0];
#pragma unroll
        for (int mp = 0; mp < kMP; ++mp) {
            P[2 * mp] = P[2 * mp + 1] = 0.f;
            if (2 * mp >= m0 || (unit && mp != mp0)) continue;
            f2_t c[4];
#pragma unroll
            for (int t = 0; t < 16; ++t) {
                const f2_t w = f2_pack(__ldg(&W.k1[2 * mp][t]), __ldg(&W.k1[2 * mp + 1][t]));
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    const f2_t m = f2_mul(win[(d >> 1) + (t >> 2)][(d & 1) + (t & 3)], w, nz);
                    c[d] = t ? f2_add(c[d], m) : m;
                }
            }
            const f2_t v = lg_pool_tanh2(c, W.max_pool, lg_pool_pair(W, 0, mp), af, nz);
            P[2 * mp] = f2_lo(v);
            P[2 * mp + 1] = f2_hi(v);
            if (unit) {
                S.l1rest[px - kFull][mp] = make_float2(P[2 * mp], P[2 * mp + 1]);
            }
        }
        if (!unit) sums(P, px);
    }
    __syncthreads();
    if (threadIdx.x < kRest) {
        float P[kM0];
#pragma unroll
        for (int k = 0; k < kM0; ++k) P[k] = (k & 1) ? S.l1rest[threadIdx.x][k / 2].y : S.l1rest[threadIdx.x][k / 2].x;
        sums(P, kFull + threadIdx.x);
    }
    __syncthreads();
    for (int it = threadIdx.x; it < m0 * kP2; it += kWT) {
        const int i = it / kP2, p = it - i * kP2;
        const int x = p % kP2W, y = p / kP2W;
        f2_t q[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) q[r][c] = f2_dup(S.s1[i][2 * y + r][2 * x + c]);
        f2_t c[4];
#pragma unroll
        for (int t = 0; t < 9; ++t) {
            const f2_t w = f2_pack(__ldg(&W.k2[2 * i][t]), __ldg(&W.k2[2 * i + 1][t]));
#pragma unroll
            for (int d = 0; d < 4; ++d) {
                const f2_t m = f2_mul(q[(d >> 1) + t / 3][(d & 1) + t % 3], w, nz);
                c[d] = t ? f2_add(c[d], m) : m;
            }
        }
        const f2_t v = lg_pool_tanh2(c, W.max_pool, lg_pool_pair(W, 1, i), af, nz);
        S.u.l.p2[2 * i][y][x] = f2_lo(v);
        S.u.l.p2[2 * i + 1][y][x] = f2_hi(v);
    }
    __syncthreads();
    for (int it = threadIdx.x; it < W.m1 * kP2; it += kWT) {
        const int k = it / kP2, p = it - k * kP2;
        const int x = p % kP2W, y = p / kP2W;
        const float two = k ? fadd(S.u.l.p2[k - 1][y][x], S.u.l.p2[k][y][x]) : fadd(S.u.l.p2[0][y][x], S.u.l.p2[1][y][x]);
        S.u.l.s2[k][y][x] = (k == 0 || k == W.m1 - 1) ? two : fadd(two, S.u.l.p2[k + 1][y][x]);
    }
    __syncthreads();
    constexpr int kK3W = 7, kK3H = 8;  // the third-layer kernel of the stage-2/3 networks
    for (int it = threadIdx.x; it < (W.m2 >> 1) * kOutN; it += kWT) {
        const int i = it / kOutN, o = it - i * kOutN;
        const int ox = o & 3, oy = o >> 2;
        f2_t acc = 0ull;
#pragma unroll
        for (int t = 0; t < kK3W * kK3H; ++t) {
            const f2_t m = f2_mul(f2_dup(S.u.l.s2[i][oy + t / kK3W][ox + t % kK3W]), f2_pack(__ldg(&W.k3[2 * i][t]), __ldg(&W.k3[2 * i + 1][t])), nz);
            acc = t ? f2_add(acc, m) : m;
        }
        const f2_t v = lg_l3_finish2(W, lg_l3_pair(W, i), acc, nz);
        S.u.l.a3[2 * i][o] = f2_lo(v);
        S.u.l.a3[2 * i + 1][o] = f2_hi(v);
    }
    __syncthreads();
    if (W.full_connect) {
        for (int it = threadIdx.x; it < W.hl * kOutN; it += kWT) {
            const int n = it / kOutN, o = it - n * kOutN;
            S.v.hbuf[n][o] = lg_hidden_fc(W, n, [&](int j) { return S.u.l.a3[j][o]; });
        }
        __syncthreads();
    }
    if (threadIdx.x < kOutN) {
        const int o = threadIdx.x;
        float acc;
        if (W.full_connect) {
            acc = S.v.hbuf[0][o];
            for (int n = 1; n < W.hl; ++n) acc = fadd(acc, S.v.hbuf[n][o]);
        } else {
            acc = fadd(S.u.l.a3[1][o], S.u.l.a3[0][o]);
            for (int i = 1; i < W.m2 / 2; ++i) acc = fadd(acc, fadd(S.u.l.a3[2 * i + 1][o], S.u.l.a3[2 * i][o]));
        }
        S.out[o] = lg_finish(W, acc);
    }
    __syncthreads();
}

struct WinArgs {
    const float* gray;
    int gpitch, gw, gh;
    const Candidate* cands;
    const int* n_cand;
    const LevelDesc* levels;
    WinOut* out;
    CascadeConfig cfg;
    const WindowNets* nets;  // the CNTK networks in device memory too
    const LegacyNet* lg;  // legacy networks ([1] stage 2, [2] stage 3) instead of the CNTK ones, or null
    float2 negzero;       // (-0, -0), for the legacy networks (the CNTK ones carry their own)
};

// crop + byte rounding + (optional) equalisation of one window into S.crop
__device__ void prepare_window(const WinArgs& a, WindowSmem& S, const Candidate& cd, float inv_scale, int mod) {
    if (threadIdx.x == 0) window_geometry(cd, inv_scale, mod, a.gw, a.gh, a.cfg.pat_w, a.cfg.pat_h, S.geo);
    if (threadIdx.x < 256) S.hist[threadIdx.x] = 0;
    __syncthreads();
    const int rx = S.geo[0], ry = S.geo[1], rcols = S.geo[2], rrows = S.geo[3];
    const bool copy = (rcols == kCropW && rrows == kCropH);  // FastImageResize copies equal sizes
    const uint32_t sclx = fp_step(max(rcols, 1), kCropW), scly = fp_step(max(rrows, 1), kCropH);
    // a warp a row, a lane the columns lane and lane + 32. Every load of a thread's pixels is issued before the first
    // is used (the gray frame is read from L2, so the loads overlap instead of queueing one latency each);
    // the byte values stay in registers until the equalisation table is known
    constexpr int kRows = (kCropH + kWT / 32 - 1) / (kWT / 32);  // 7 rows a warp
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool two = lane + 32 < kCropW;
    // the clamps are memory guards only: valid candidates always sample inside the frame
    int gx[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int ix = min(lane + 32 * h, kCropW - 1);
        gx[h] = min(max(rx + (copy ? ix : (int)sample_col(ix, sclx, rcols).idx), 0), a.gw - 1);
    }
    float v[kRows][2];
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
        const int iy = min(warp + k * (kWT / 32), kCropH - 1);
        const int gy = min(max(ry + (copy ? iy : (int)sample_row(iy, scly, rrows).idx), 0), a.gh - 1);
        const float* row = a.gray + (size_t)gy * a.gpitch;
        v[k][0] = row[gx[0]];
        v[k][1] = two ? row[gx[1]] : 0.f;
    }
    const bool eq = a.cfg.equalize != 0;
    uint32_t u[(2 * kRows + 3) / 4];  // the bytes, four to a register
#pragma unroll
    for (int k = 0; k < (2 * kRows + 3) / 4; ++k) u[k] = 0u;
#pragma unroll
    for (int q = 0; q < 2 * kRows; ++q) {
        const int iy = warp + (q >> 1) * (kWT / 32), ix = lane + 32 * (q & 1);
        const uint32_t b = (uint8_t)__float2int_rz(fadd(v[q >> 1][q & 1], 0.5f));
        u[q >> 2] |= b << (8 * (q & 3));
        if (iy < kCropH && ix < kCropW) {
            if (eq)
                atomicAdd(&S.hist[b], 1);
            else
                S.crop[iy][ix] = (uint8_t)b;
        }
    }
    __syncthreads();
    if (!eq) return;
    // cumulative histogram (256 bins, one per thread): shuffle scan + warp totals
    {
        const int wid = warp;
        int c = S.hist[threadIdx.x];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y2 = __shfl_up_sync(0xffffffffu, c, o);
            if (lane >= o) c += y2;
        }
        __shared__ int wsum[8];
        if (lane == 31) wsum[wid] = c;
        __syncthreads();
        int add = 0;
        for (int w = 0; w < wid; ++w) add += wsum[w];
        S.lut[threadIdx.x] = c + add;  // cf_hist
        __syncthreads();
    }
    const float bmin = (float)S.lut[0], bmax = (float)S.lut[255];
    if (bmin != bmax) {
        const float delt = fdiv(255.f, fsub(bmax, bmin));
        const int lv = (int)fadd(fmul(fsub((float)S.lut[threadIdx.x], bmin), delt), 0.5f);
        __syncthreads();
        S.lut[threadIdx.x] = lv;
        __syncthreads();
    }
    // the equalised bytes (the reference leaves the window unchanged when every pixel is equal)
#pragma unroll
    for (int q = 0; q < 2 * kRows; ++q) {
        const int iy = warp + (q >> 1) * (kWT / 32), ix = lane + 32 * (q & 1);
        const uint32_t b = (u[q >> 2] >> (8 * (q & 3))) & 0xffu;
        if (iy < kCropH && ix < kCropW) S.crop[iy][ix] = (uint8_t)(bmin != bmax ? S.lut[b] : b);
    }
    __syncthreads();
}

// One work item = (candidate, window): window 0 is the first crop, window 1 the shrunken retry
// crop. Both windows of a candidate run in parallel (the retry is speculative: the verdict reads it
// only when window 0 is rejected, cnn_detector_v3.cpp:1806-1811); running it on demand instead
// would save the ~10 % of retries whose first window accepts but put the two windows of a rejected
// candidate one after the other, doubling the kernel's latency. Inside an item, stage 3 runs only
// when stage 2 does not end the check (the reference's early exits, cnn_detector_v3.cpp:1698-1706);
// otherwise its slot keeps (max -10, count 0), exactly what the reference leaves behind.
// One work item: window `mod` of candidate ci, stage 2 then (unless an early exit ends the check)
// stage 3, the (max, count) pair of each written to a.out.
template <bool kLegacy>
__device__ __forceinline__ void window_item(const WindowNets& N, const WinArgs& a, WindowSmem& S, int ci, int mod) {
    const CascadeConfig& C = a.cfg;
    const Candidate cd = a.cands[ci];
    const LevelDesc& L = a.levels[cd.level];
    const int mn = (C.adapt_min_neighbors && L.scale > 0.7f && C.min_neighbors > 1) ? C.min_neighbors - 1 : C.min_neighbors;
    prepare_window(a, S, cd, L.inv_scale, mod);
    WinOut r[2];
    r[1].max = -10.f;
    r[1].knn = 0;
    for (int stage = 0; stage < 2; ++stage) {
        if constexpr (kLegacy)
            legacy_window_net(a.lg[1 + stage], S, stage == 0 ? 0 : (C.reflection ? 1 : 2), f2_ld(a.negzero));
        else if (stage == 0)
            window_net(N.s2, &a.nets->s2, S, 0);
        else
            window_net(N.s3, &a.nets->s3, S, C.reflection ? 1 : 2);
        // every thread reduces the 16 responses itself (no extra barrier needed)
        const float thr = stage == 0 ? C.thr2 : C.thr3;
        float mx = -10.f;
        int kc = 0;
#pragma unroll
        for (int o = 0; o < kOutN; ++o) {
            const float d = S.out[o];
            mx = (mx < d) ? d : mx;  // MAX(max_score, d) (cnn_detector_v3.cpp:1667-1683)
            if (d > thr) kc++;
        }
        r[stage].max = mx;
        r[stage].knn = kc;
        if (stage == 0) {
            const bool stop = (C.type_check == 0 && kc >= mn) || (C.type_check > 0 && kc <= 0) || (C.type_check == 2 && kc < mn);
            if (stop) break;
        }
    }
    if (threadIdx.x == 0) {
        a.out[(size_t)ci * 4 + 2 * mod] = r[0];
        a.out[(size_t)ci * 4 + 2 * mod + 1] = r[1];
    }
    __syncthreads();
}

// kMinBlocks: the register budget (2 resident blocks a SM: up to 128 registers, no spills; 4: 64;
// 5: 48; 6: 40, more spilled), matched to the schedule's resident blocks
template <bool kLegacy, int kMinBlocks>
__global__ void __launch_bounds__(kWT, kMinBlocks) window_kernel(const __grid_constant__ WindowNets N, const WinArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WindowSmem& S = *reinterpret_cast<WindowSmem*>(smem_raw);
    chain_wait();
    const int n = *a.n_cand;
    const int per_cand = a.cfg.double_check ? 2 : 1;
    const int total = n * per_cand;
    for (int it = blockIdx.x; it < total; it += gridDim.x) {
        const int ci = it / per_cand;
        window_item<kLegacy>(N, a, S, ci, it - ci * per_cand);
    }
}

// The candidates of every frame of a batch as one persistent item list (frame by frame); the
// per-frame gray image, candidates and outputs come from B, the rest from `base`.
template <int kMinBlocks>
__global__ void __launch_bounds__(kWT, kMinBlocks) window_batch_kernel(const __grid_constant__ WindowNets N, const WinArgs base,
                                                              const __grid_constant__ WinBatch B) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WindowSmem& S = *reinterpret_cast<WindowSmem*>(smem_raw);
    __shared__ int s_pre[kMaxBatch + 1];
    if (threadIdx.x == 0) {
        s_pre[0] = 0;
        for (int f = 0; f < B.n_frames; ++f) s_pre[f + 1] = s_pre[f] + *B.ncand[f];
    }
    __syncthreads();
    const int per_cand = base.cfg.double_check ? 2 : 1;
    const int total = s_pre[B.n_frames] * per_cand;
    for (int it = blockIdx.x; it < total; it += gridDim.x) {
        const int c = it / per_cand;
        int f = 0;
        while (s_pre[f + 1] <= c) ++f;
        WinArgs a = base;
        a.gray = B.gray[f];
        a.cands = B.cands[f];
        a.n_cand = B.ncand[f];
        a.out = B.out[f];
        window_item<false>(N, a, S, c - s_pre[f], it - c * per_cand);
    }
}

int window_smem_bytes() { return (int)sizeof(WindowSmem); }

cudaError_t launch_window_batch(const WindowNets& N, const WindowNets* d_nets, const WinBatch& B, int gpitch, int gw, int gh, const LevelDesc* levels,
                                const CascadeConfig& cfg, int grid, cudaStream_t st, int ctas_per_sm) {
    WinArgs a{};
    a.gpitch = gpitch;
    a.gw = gw;
    a.gh = gh;
    a.levels = levels;
    a.cfg = cfg;
    a.lg = nullptr;
    a.nets = d_nets;
    if (ctas_per_sm <= 2)
        window_batch_kernel<2><<<grid, kWT, sizeof(WindowSmem), st>>>(N, a, B);
    else
        window_batch_kernel<4><<<grid, kWT, sizeof(WindowSmem), st>>>(N, a, B);
    return cudaGetLastError();
}

cudaError_t launch_window(const WindowNets& N, const WindowNets* d_nets, const float* gray, int gpitch, int gw, int gh, const Candidate* cands, const int* n_cand,
                          const LevelDesc* levels, WinOut* out, const CascadeConfig& cfg, int grid, cudaStream_t st, const LegacyNet* lg,
                          int ctas_per_sm) {
    static_assert(sizeof(WindowSmem) + 64 <= 48 * 1024, "window kernel shared memory must stay under the default 48 KB");
    WinArgs a;
    a.gray = gray;
    a.gpitch = gpitch;
    a.gw = gw;
    a.gh = gh;
    a.cands = cands;
    a.n_cand = n_cand;
    a.levels = levels;
    a.out = out;
    a.cfg = cfg;
    a.lg = lg;
    a.nets = d_nets;
    a.negzero = make_float2(-0.f, -0.f);
    const auto kernel = lg ? (ctas_per_sm <= 2 ? window_kernel<true, 2> : window_kernel<true, 4>)
                        : ctas_per_sm <= 2 ? window_kernel<false, 2>
                        : ctas_per_sm == 5 ? window_kernel<false, 5>
                        : ctas_per_sm >= 6 ? window_kernel<false, 6>
                                           : window_kernel<false, 4>;
    return launch_chained(kernel, grid, kWT, sizeof(WindowSmem), st, N, a);
}

// five or six resident window blocks need most of a SM's 228 KB as shared memory
cudaError_t window_setup() {
    cudaError_t e = cudaFuncSetAttribute(window_kernel<false, 5>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(window_kernel<false, 6>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    return e;
}

}  // namespace ccnn
