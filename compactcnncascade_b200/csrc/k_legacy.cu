// Legacy cascade networks (model format 1.0, `_new.bin`) on the device: the reader and the forward
// pass of SIMD::ConvNeuralNetwork in the reference's plain-C++ build (src/CNNObjectDetector/
// cnn_simd.cpp:40-336 and 551-874 with the CNNPP operations of cnnpp_cplusplus.cpp), reproduced
// operation for operation in IEEE single precision (the file is built with -fmad=false):
//   L1  conv 4x4 (conv_4x4 :92), tanh(c + bias) of the four positions of a 2x2 window, their max
//       or sum, tanh(w * pooled + b) * af                      (max_tanh_tanh :473, tanh_avr_tanh :411)
//   sums of neighbouring L1 maps (add :916, add2 :933), conv 3x3 (conv_3x3 :36), the same pooling
//   sums of neighbouring L2 maps, conv 5x6 or 7x8 (conv_6x5 :212, conv_8x7 :292), then either
//     two hidden neurons per L3 map (tanh_tanh_2tanh :692) summed over the maps, or
//     tanh_tanh (:778) and fully connected hidden neurons (mulC24_add_tanh :1003, or
//     mulC2_add / mulC1_add / tanh :968-1002, :868) summed over the neurons,
//   and the output tanh(sum + bias) * af (tanh :868).
// tanh is the reference's rational form sgn(c) (1 - 1 / (1 + |c| + c^2 + 1.41645 c^4)) (USE_FAST_TANH).
// Two kernels over all levels: L1 and L2 with the neighbouring-map sums, and L3 to the output. Maps
// (2i, 2i + 1) read the same input and run as packed pairs, each lane with the reference's roundings.
#include <cuda_runtime.h>

#include <cstring>
#include <fstream>
#include <iterator>
#include <string>
#include <vector>

#include "../../include/ccnn_inspect.h"
#include "kernels.h"
#include "legacy_dev.cuh"

namespace ccnn {

void set_error(const std::string& msg);

// ---- reader ----

namespace {
struct LgReader {
    const uint8_t* p;
    size_t n, off = 0;
    bool ok = true;
    template <class T>
    T get() {
        T v{};
        if (off + sizeof(T) > n) {
            ok = false;
            return v;
        }
        std::memcpy(&v, p + off, sizeof(T));
        off += sizeof(T);
        return v;
    }
};
}  // namespace

bool parse_legacy_model(const uint8_t* data, size_t n, LegacyNet* net, std::string* err) {
    LgReader r{data, n};
    std::memset(net, 0, sizeof(LegacyNet));
    const float version = r.get<float>();
    if (!r.ok || version != 1.0f) {
        *err = "not a legacy (format 1.0) model file";
        return false;
    }
    net->max_pool = r.get<uint8_t>() != 0 ? 1 : 0;
    net->min_w = r.get<int32_t>();
    net->min_h = r.get<int32_t>();
    const int layers = r.get<int32_t>();
    if (!r.ok || layers != 3) {
        *err = "this configuration of cnn models is not supported (3 convolution layers expected)";
        return false;
    }
    int maps[3];
    for (int& m : maps) m = r.get<int32_t>();
    net->m0 = maps[0];
    net->m1 = maps[1];
    net->m2 = maps[2];
    if (!r.ok || maps[0] < 2 || maps[0] > kLgMaxM0 || maps[1] != 2 * maps[0] || maps[2] != 2 * maps[1]) {
        *err = "legacy model: map counts must double from layer to layer, with at most 8 first-layer maps";
        return false;
    }
    int kw[3], kh[3];
    for (int l = 0; l < 3; ++l) {
        kw[l] = r.get<int32_t>();
        kh[l] = r.get<int32_t>();
        if (!r.ok || kw[l] <= 0 || kh[l] <= 0 || kw[l] * kh[l] > kLgMaxK3) {
            *err = "legacy model: malformed convolution layer";
            return false;
        }
        for (int m = 0; m < maps[l]; ++m)
            for (int k = 0; k < kw[l] * kh[l]; ++k) {
                const float v = r.get<float>();
                if (l == 0 && k < 16) net->k1[m][k] = v;
                if (l == 1 && k < 9) net->k2[m][k] = v;
                if (l == 2) net->k3[m][k] = v;
            }
    }
    net->k3w = kw[2];
    net->k3h = kh[2];
    net->af = r.get<float>();
    for (int l = 0; l < 3; ++l)
        for (int m = 0; m < maps[l]; ++m) {
            net->cb[l][m] = r.get<float>();
            net->sw[l][m] = r.get<float>();
            net->sb[l][m] = r.get<float>();
        }
    net->full_connect = r.get<uint8_t>() != 0 ? 1 : 0;
    net->hl = r.get<int32_t>();
    if (!r.ok) {
        *err = "legacy model: file is truncated";
        return false;
    }
    // the reference's own shape check (cnn_simd.cpp:267-276)
    if (kw[0] * kh[0] != 16 || kw[1] * kh[1] != 9 || (kw[2] * kh[2] != 30 && kw[2] * kh[2] != 56) || kw[0] != 4 || kw[1] != 3) {
        *err = "this configuration of cnn models is not supported (4x4, 3x3 and 5x6 or 7x8 kernels expected)";
        return false;
    }
    if (net->hl <= 0 || net->hl > kLgMaxHL || (!net->full_connect && net->hl != 2 * net->m2)) {
        *err = "legacy model: hidden layer size is not supported";
        return false;
    }
    if (!net->full_connect) {
        for (int i = 0; i < net->hl; ++i) net->hw[i] = r.get<float>();
    } else {
        for (int i = 0; i < net->hl; ++i)
            for (int j = 0; j < net->m2; ++j) net->hwfc[i][j] = r.get<float>();
    }
    for (int i = 0; i < net->hl; ++i) net->hb[i] = r.get<float>();
    for (int i = 0; i < net->hl; ++i) net->ow[i] = r.get<float>();
    net->ob = r.get<float>();
    if (!r.ok) {
        *err = "legacy model: file is truncated";
        return false;
    }
    return true;
}

bool load_legacy_model_file(const std::string& path, LegacyNet* net, std::string* err) {
    std::ifstream f(path, std::ios::binary);
    if (!f) {
        *err = "cannot open model file " + path;
        return false;
    }
    std::vector<uint8_t> bytes((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
    return parse_legacy_model(bytes.data(), bytes.size(), net, err);
}

// ---- forward pass ----

namespace {

constexpr int kLgT = 256;              // threads
constexpr int kLgTX = 32, kLgTY = 8;   // pooled L2 pixels, or responses, of a block
constexpr int kLgLevels = 32;          // levels a launch (its table travels as a kernel parameter)
constexpr int kLgP1X = 2 * kLgTX + 2, kLgP1Y = 2 * kLgTY + 2;  // pooled L1 pixels that a tile of L2 reads
constexpr int kLgP1S = kLgP1X + 1;                             // row stride of their sums

// The levels of one launch and each one's first block: `pool` for the L1 and L2 layers, `out` for the rest.
struct LgTable {
    int n;
    struct Level {
        LegacyLevel L;
        int p2w, p2h, ow, oh;
        int pool_base, pool_tx, out_base, out_tx;
    } lv[kLgLevels];
};

template <int LgTable::Level::* base>
__device__ __forceinline__ const LgTable::Level& lg_level(const LgTable& T, int block) {
    int i = 0;
    while (i + 1 < T.n && block >= T.lv[i + 1].*base) ++i;
    return T.lv[i];
}

// L1, the sums of neighbouring L1 maps, L2 and the sums of neighbouring L2 maps (which L3 reads) of one
// 32 x 8 tile of pooled L2 pixels; the L1 sums stay in shared memory. A thread computes every map of its
// pixel, two at a time (packed; an odd last map's partner is computed with zero weights and dropped). Bound by
// latency: a 640 x 480 frame's levels are about one block a SM.
__global__ void __launch_bounds__(kLgT) legacy_pool_kernel(const LegacyNet* __restrict__ N, const __grid_constant__ LgTable T, const f2_t nz) {
    __shared__ float s1[kLgMaxM0][kLgP1Y][kLgP1S];
    __shared__ float2 k1[kLgMaxM0 / 2][16], k2[kLgMaxM0][9];
    __shared__ LgPoolPair q1[kLgMaxM0 / 2], q2[kLgMaxM0];
    const int tid = threadIdx.x;
    chain_wait();
    const int m0 = N->m0, max_pool = N->max_pool;
    for (int i = tid; i < kLgMaxM0 / 2 * 16; i += kLgT) {
        const int p = i >> 4, t = i & 15;  // maps past m0 have zero weights
        k1[p][t] = make_float2(N->k1[2 * p][t], N->k1[2 * p + 1][t]);
    }
    for (int i = tid; i < m0 * 9; i += kLgT) k2[i / 9][i % 9] = make_float2(N->k2[2 * (i / 9)][i % 9], N->k2[2 * (i / 9) + 1][i % 9]);
    if (tid < kLgMaxM0 / 2) q1[tid] = lg_pool_pair(*N, 0, tid);
    if (tid < m0) q2[tid] = lg_pool_pair(*N, 1, tid);
    const f2_t af = f2_dup(N->af);
    const LgTable::Level& V = lg_level<&LgTable::Level::pool_base>(T, blockIdx.x);
    const int tile = blockIdx.x - V.pool_base, ty = tile / V.pool_tx;
    const int x0 = (tile - ty * V.pool_tx) * kLgTX, y0 = ty * kLgTY;
    // of the L1 pixels, those that a pooled L2 pixel of the level reads
    const int nx = min(kLgP1X, 2 * (V.p2w - x0) + 2), ny = min(kLgP1Y, 2 * (V.p2h - y0) + 2);
    __syncthreads();
    for (int it = tid; it < kLgP1X * ny; it += kLgT) {
        const int y = it / kLgP1X, x = it - y * kLgP1X;
        if (x >= nx) continue;
        const float* src = V.L.img + (size_t)(2 * (2 * y0 + y)) * V.L.pitch + 2 * (2 * x0 + x);
        f2_t win[5][5];
#pragma unroll
        for (int r = 0; r < 5; ++r)
#pragma unroll
            for (int c = 0; c < 5; ++c) win[r][c] = f2_dup(ld_chain(src + (size_t)r * V.L.pitch + c));
        float P[kLgMaxM0];
#pragma unroll
        for (int p = 0; p < kLgMaxM0 / 2; ++p) {
            P[2 * p] = P[2 * p + 1] = 0.f;
            if (2 * p >= m0) continue;
            f2_t c[4];
#pragma unroll
            for (int t = 0; t < 16; ++t) {
                const f2_t w = f2_ld(k1[p][t]);
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    const f2_t m = f2_mul(win[(d >> 1) + (t >> 2)][(d & 1) + (t & 3)], w, nz);
                    c[d] = t ? f2_add(c[d], m) : m;
                }
            }
            const f2_t v = lg_pool_tanh2(c, max_pool, q1[p], af, nz);
            P[2 * p] = f2_lo(v);
            P[2 * p + 1] = f2_hi(v);
        }
#pragma unroll
        for (int k = 0; k < kLgMaxM0; ++k)
            if (k < m0) s1[k][y][x] = lg_neighbour_sum(P, k, m0);
    }
    __syncthreads();
    const int lx = tid & (kLgTX - 1), ly = tid / kLgTX;
    if (x0 + lx >= V.p2w || y0 + ly >= V.p2h) return;
    float P[kLgMaxM1];
#pragma unroll
    for (int i = 0; i < kLgMaxM0; ++i) {
        P[2 * i] = P[2 * i + 1] = 0.f;
        if (i >= m0) continue;
        f2_t q[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) q[r][c] = f2_dup(s1[i][2 * ly + r][2 * lx + c]);
        f2_t c[4];
#pragma unroll
        for (int t = 0; t < 9; ++t) {
            const f2_t w = f2_ld(k2[i][t]);
#pragma unroll
            for (int d = 0; d < 4; ++d) {
                const f2_t m = f2_mul(q[(d >> 1) + t / 3][(d & 1) + t % 3], w, nz);
                c[d] = t ? f2_add(c[d], m) : m;
            }
        }
        const f2_t v = lg_pool_tanh2(c, max_pool, q2[i], af, nz);
        P[2 * i] = f2_lo(v);
        P[2 * i + 1] = f2_hi(v);
    }
    const size_t plane = (size_t)V.p2w * V.p2h;
    float* out = V.L.scratch + (size_t)(y0 + ly) * V.p2w + x0 + lx;
#pragma unroll
    for (int k = 0; k < kLgMaxM1; ++k)
        if (k < 2 * m0) out[k * plane] = lg_neighbour_sum(P, k, 2 * m0);
}

// L3 maps (2i, 2i + 1) of 32 x 8 responses, a lane a column, on the sums of map i: every input row is
// loaded once and continues the chains of the rows that it reaches (each output's taps stay in row-major
// order); the pair's weights are in registers. done(row, (c0, c1)) takes each result.
template <int KW, int KH, class Done>
__device__ __forceinline__ void lg_l3_rows(const LegacyNet& N, int i, const float* in, int pitch, int last, f2_t nz, Done done) {
    f2_t w[KH * KW];
#pragma unroll
    for (int t = 0; t < KH * KW; ++t) w[t] = f2_pack(__ldg(&N.k3[2 * i][t]), __ldg(&N.k3[2 * i + 1][t]));
    f2_t acc[kLgTY];
#pragma unroll
    for (int r = 0; r < kLgTY + KH - 1; ++r) {
        const float* row = in + (size_t)min(r, last) * pitch;  // rows past the map feed responses past it
        f2_t v[KW];
#pragma unroll
        for (int c = 0; c < KW; ++c) v[c] = f2_dup(ld_chain(row + c));
#pragma unroll
        for (int j = 0; j < kLgTY; ++j) {
            const int kr = r - j;
            if (kr < 0 || kr >= KH) continue;
#pragma unroll
            for (int c = 0; c < KW; ++c) {
                const f2_t m = f2_mul(v[c], w[kr * KW + c], nz);
                acc[j] = kr + c ? f2_add(acc[j], m) : m;
            }
            if (kr == KH - 1) done(j, acc[j]);
        }
    }
}

// L3 to the output of one 32 x 8 tile of responses: a warp takes every eighth map pair for the whole tile,
// then a thread a response sums what the pairs left in shared memory, in map (or neuron) order.
template <int KW, int KH>
__global__ void __launch_bounds__(kLgT) legacy_out_kernel(const LegacyNet* __restrict__ Np, const __grid_constant__ LgTable T, int* counts,
                                                          float thr, const f2_t nz) {
    __shared__ float vals[kLgMaxM2][kLgTY][kLgTX];  // L3 values, or without a fully connected layer each pair's sum
    chain_wait();
    const LegacyNet& N = *Np;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int it2 = N.m2 >> 1;
    const LgTable::Level& V = lg_level<&LgTable::Level::out_base>(T, blockIdx.x);
    const int tile = blockIdx.x - V.out_base, ty = tile / V.out_tx;
    const int x0 = (tile - ty * V.out_tx) * kLgTX, y0 = ty * kLgTY;
    const size_t plane = (size_t)V.p2w * V.p2h;
    const int sx = min(x0 + lane, V.ow - 1);  // columns past the map compute the last one again
    for (int i = warp; i < it2; i += kLgT / 32) {
        const LgL3Pair q = lg_l3_pair(N, i);
        const float* in = V.L.scratch + i * plane + (size_t)y0 * V.p2w + sx;
        auto done = [&](int j, f2_t c) {
            const f2_t v = lg_l3_finish2(N, q, c, nz);
            if (N.full_connect) {
                vals[2 * i][j][lane] = f2_lo(v);
                vals[2 * i + 1][j][lane] = f2_hi(v);
            } else {
                vals[i][j][lane] = fadd(f2_hi(v), f2_lo(v));
            }
        };
        if constexpr (KW > 0) {
            lg_l3_rows<KW, KH>(N, i, in, V.p2w, V.p2h - 1 - y0, nz, done);
        } else {
            // any other kernel shape of the format: one output after the other
            const int kw = N.k3w, kt = N.k3w * N.k3h;
            for (int j = 0; j < kLgTY && y0 + j < V.oh; ++j) {
                f2_t acc = 0ull;
                for (int t = 0; t < kt; ++t) {
                    const f2_t m = f2_mul(f2_dup(ld_chain(in + (size_t)(j + t / kw) * V.p2w + t % kw)), f2_pack(N.k3[2 * i][t], N.k3[2 * i + 1][t]), nz);
                    acc = t ? f2_add(acc, m) : m;
                }
                done(j, acc);
            }
        }
    }
    __syncthreads();
    const int x = x0 + lane, y = y0 + warp;
    if (x >= V.ow || y >= V.oh) return;
    float acc = 0.f;
    if (N.full_connect) {
        for (int n = 0; n < N.hl; ++n) {
            const float h = lg_hidden_fc(N, n, [&](int j) { return vals[j][warp][lane]; });
            acc = (n == 0) ? h : fadd(acc, h);
        }
    } else {
        acc = vals[0][warp][lane];
        for (int i = 1; i < it2; ++i) acc = fadd(acc, vals[i][warp][lane]);
    }
    const float r = lg_finish(N, acc);
    V.L.resp[(long long)y * V.ow + x] = r;
    // candidates (response > treshold_1) counted per scan chunk, as the CNTK stage-1 back kernel does
    if (counts && r > thr) atomicAdd(&counts[V.L.chunk_base + (y * V.ow + x) / kCandChunk], 1);
}

}  // namespace

// Two launches for up to kLgLevels levels. Before, every level took three (one thread a pooled pixel and map,
// or a response with all its maps, each tap summing three maps from memory): the 13 levels of a 640 x 480
// frame took 1.03 ms of kernels on B200, now 33 us (19 for L1 and L2, 14 for the rest).
cudaError_t launch_legacy_forward(const LegacyNet* d_net, const LegacyNet& h_net, const LegacyLevel* levels, int n_levels, cudaStream_t st, int* counts,
                                  float thr) {
    const f2_t nz = 0x8000000080000000ull;  // (-0, -0)
    for (int g0 = 0; g0 < n_levels; g0 += kLgLevels) {
        LgTable T;
        T.n = n_levels - g0 < kLgLevels ? n_levels - g0 : kLgLevels;
        int pool = 0, out = 0;
        for (int i = 0; i < T.n; ++i) {
            LgTable::Level& V = T.lv[i];
            V.L = levels[g0 + i];
            V.p2w = (((V.L.w - 3) >> 1) - 2) >> 1;
            V.p2h = (((V.L.h - 3) >> 1) - 2) >> 1;
            legacy_output_size(h_net, V.L.w, V.L.h, &V.ow, &V.oh);
            const bool any = V.ow > 0 && V.oh > 0;
            V.pool_tx = (V.p2w + kLgTX - 1) / kLgTX;
            V.pool_base = pool;
            if (any) pool += V.pool_tx * ((V.p2h + kLgTY - 1) / kLgTY);
            V.out_tx = (V.ow + kLgTX - 1) / kLgTX;
            V.out_base = out;
            if (any) out += V.out_tx * ((V.oh + kLgTY - 1) / kLgTY);
        }
        if (!pool) continue;
        cudaError_t e = launch_chained(legacy_pool_kernel, pool, kLgT, 0, st, d_net, T, nz);
        if (e != cudaSuccess) return e;
        const auto kernel = h_net.k3w == 5 && h_net.k3h == 6   ? legacy_out_kernel<5, 6>
                            : h_net.k3w == 7 && h_net.k3h == 8 ? legacy_out_kernel<7, 8>
                                                               : legacy_out_kernel<0, 0>;
        e = launch_chained(kernel, out, kLgT, 0, st, d_net, T, counts, thr, nz);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

size_t legacy_scratch_floats(const LegacyNet& n, int w, int h) {
    return (size_t)n.m1 * ((((w - 3) >> 1) - 2) >> 1) * ((((h - 3) >> 1) - 2) >> 1);
}

}  // namespace ccnn

using namespace ccnn;

extern "C" CCNN_API ccnn_status ccnn_legacy_model_info(const char* model_path, int* info, int n_info) {
    if (!model_path || !info || n_info < 10) {
        set_error("invalid arguments");
        return CCNN_ERR_INVALID_ARG;
    }
    LegacyNet net;
    std::string err;
    if (!load_legacy_model_file(model_path, &net, &err)) {
        set_error(err);
        return CCNN_ERR_MODEL;
    }
    const int v[10] = {net.max_pool, net.min_w, net.min_h, net.m0, net.m1, net.m2, net.k3w, net.k3h, net.full_connect, net.hl};
    for (int i = 0; i < 10; ++i) info[i] = v[i];
    return CCNN_OK;
}

extern "C" CCNN_API ccnn_status ccnn_legacy_net_forward(const char* model_path, const float* d_img, int cols, int rows, size_t step, float* d_resp,
                                                        int resp_cap, int* ow, int* oh, void* stream) {
    if (!model_path || !d_img || !d_resp || !ow || !oh || step % sizeof(float) || step < sizeof(float) * (size_t)cols) {
        set_error("invalid arguments");
        return CCNN_ERR_INVALID_ARG;
    }
    LegacyNet net;
    std::string err;
    if (!load_legacy_model_file(model_path, &net, &err)) {
        set_error(err);
        return CCNN_ERR_MODEL;
    }
    if (cols < net.min_w || rows < net.min_h) {
        set_error("image is smaller than the network's input");
        return CCNN_ERR_INVALID_ARG;
    }
    legacy_output_size(net, cols, rows, ow, oh);
    if ((long long)*ow * *oh > resp_cap) {
        set_error("response buffer too small");
        return CCNN_ERR_INVALID_ARG;
    }
    const cudaStream_t st = (cudaStream_t)stream;
    void* buf = nullptr;
    const size_t scratch = legacy_scratch_floats(net, cols, rows);
    cudaError_t e = cudaMallocAsync(&buf, sizeof(LegacyNet) + sizeof(float) * scratch, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(buf, &net, sizeof(LegacyNet), cudaMemcpyHostToDevice, st);
    const LegacyLevel L = {d_img, (int)(step / sizeof(float)), cols, rows, (float*)((char*)buf + sizeof(LegacyNet)), d_resp, 0};
    if (e == cudaSuccess) e = launch_legacy_forward((const LegacyNet*)buf, net, &L, 1, st, nullptr, 0.f);
    if (buf) {
        const cudaError_t f = cudaFreeAsync(buf, st);
        if (e == cudaSuccess) e = f;
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // `net` on the host stack was copied from
    if (e != cudaSuccess) {
        set_error(std::string("legacy forward: ") + cudaGetErrorString(e));
        return CCNN_ERR_CUDA;
    }
    return CCNN_OK;
}
