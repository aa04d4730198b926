// Device arithmetic of the legacy (format 1.0) networks, shared by the standalone forward pass
// and the stage-2/3 window kernel. Every operation is the reference's plain-C++ one
// (src/CNNObjectDetector/cnnpp_cplusplus.cpp), in the same order.
#pragma once

#include "ccnn_common.cuh"
#include "legacy.h"

namespace ccnn {

// A packed pair of maps' pooling parameters: convolution bias, pooling weight and bias.
struct LgPoolPair {
    float2 cb, sw, sb;
};
__device__ __forceinline__ LgPoolPair lg_pool_pair(const LegacyNet& N, int layer, int p) {
    LgPoolPair q;
    q.cb = make_float2(N.cb[layer][2 * p], N.cb[layer][2 * p + 1]);
    q.sw = make_float2(N.sw[layer][2 * p], N.sw[layer][2 * p + 1]);
    q.sb = make_float2(N.sb[layer][2 * p], N.sb[layer][2 * p + 1]);
    return q;
}

// tanh(c + b) of the four convolution outputs of a 2x2 window, their max or sum, then
// tanh(w * pooled + b) * af (max_tanh_tanh :473, tanh_avr_tanh :411), for a pair of maps. Rounded sums,
// products and reciprocals are monotone, so c -> tanh(c + b) is (every term of its denominator grows with
// |c|), and the max of the four tanh is the tanh of the max: one instead of four.
__device__ __forceinline__ f2_t lg_pool_tanh2(const f2_t c[4], int max_pool, const LgPoolPair& q, f2_t af, f2_t nz) {
    const f2_t cb = f2_ld(q.cb);
    f2_t p;
    if (max_pool) {
        p = tanh_rational2(f2_add(f2_max4(c[0], c[1], c[2], c[3]), cb), nz);
    } else {
        p = tanh_rational2(f2_add(c[0], cb), nz);
#pragma unroll
        for (int d = 1; d < 4; ++d) p = f2_add(p, tanh_rational2(f2_add(c[d], cb), nz));
    }
    return f2_mul(af, tanh_rational2(f2_add(f2_mul(f2_ld(q.sw), p, nz), f2_ld(q.sb)), nz), nz);
}

// neighbouring-map sum i of `count` pooled maps of one pixel, with the reference's additions: maps 0+1,
// (i-1)+i+(i+1), and (count-2)+(count-1) (add :916, add2 :933). `i` a constant after unrolling.
template <int kMax>
__device__ __forceinline__ float lg_neighbour_sum(const float (&p)[kMax], int i, int count) {
    if (i == 0) return fadd(p[0], p[1]);
    const float two = fadd(p[i - 1], p[i]);
    return (i + 1 >= kMax || i == count - 1) ? two : fadd(two, p[i + 1 < kMax ? i + 1 : i]);
}

// What an L3 map pair's activations need: convolution bias, pooling weight and bias, and of the two hidden
// neurons of each map (first and second, a lane a map) af * weight, bias and output weight.
struct LgL3Pair {
    f2_t cb, sw, sb, hw1, hb1, ow1, hw2, hb2, ow2;
};
__device__ __forceinline__ LgL3Pair lg_l3_pair(const LegacyNet& N, int i) {
    const int a = 2 * i, b = 2 * i + 1;
    LgL3Pair q;
    q.cb = f2_pack(N.cb[2][a], N.cb[2][b]);
    q.sw = f2_pack(N.sw[2][a], N.sw[2][b]);
    q.sb = f2_pack(N.sb[2][a], N.sb[2][b]);
    if (!N.full_connect) {
        q.hw1 = f2_pack(fmul(N.af, N.hw[2 * a]), fmul(N.af, N.hw[2 * b]));
        q.hb1 = f2_pack(N.hb[2 * a], N.hb[2 * b]);
        q.ow1 = f2_pack(N.ow[2 * a], N.ow[2 * b]);
        q.hw2 = f2_pack(fmul(N.af, N.hw[2 * a + 1]), fmul(N.af, N.hw[2 * b + 1]));
        q.hb2 = f2_pack(N.hb[2 * a + 1], N.hb[2 * b + 1]);
        q.ow2 = f2_pack(N.ow[2 * a + 1], N.ow[2 * b + 1]);
    }
    return q;
}

// An L3 map pair at one output from its convolution sums (conv_6x5 :212, conv_8x7 :292): tanh_tanh (:778)
// for a fully connected net, or tanh_tanh_2tanh (:692) with each map's two hidden neurons
__device__ __forceinline__ f2_t lg_l3_finish2(const LegacyNet& N, const LgL3Pair& q, f2_t c, f2_t nz) {
    const f2_t af = f2_dup(N.af);
    c = tanh_rational2(f2_add(c, q.cb), nz);
    c = tanh_rational2(f2_add(f2_mul(q.sw, c, nz), q.sb), nz);
    if (N.full_connect) return f2_mul(af, c, nz);
    const f2_t c1 = tanh_rational2(f2_add(f2_mul(q.hw1, c, nz), q.hb1), nz);
    const f2_t c2 = tanh_rational2(f2_add(f2_mul(q.hw2, c, nz), q.hb2), nz);
    return f2_mul(af, f2_add(f2_mul(q.ow1, c1, nz), f2_mul(q.ow2, c2, nz)), nz);
}

// fully connected hidden neuron n from the L3 values (val(j)): mulC24_add_tanh (:1003) for 24 maps, else
// mulC2_add / mulC1_add / tanh (:968-1002, :868), which leave out the output weight
template <class Val>
__device__ __forceinline__ float lg_hidden_fc(const LegacyNet& N, int n, Val val) {
    if (N.m2 == 24) {
        float s = N.hb[n];
#pragma unroll
        for (int j = 0; j < 24; ++j) s = fadd(s, fmul(val(j), N.hwfc[n][j]));
        return fmul(fmul(N.af, tanh_rational(s)), N.ow[n]);
    }
    float s = fadd(fmul(val(0), N.hwfc[n][0]), fmul(val(1), N.hwfc[n][1]));
    for (int j = 2; j < N.m2; ++j) s = fadd(fmul(val(j), N.hwfc[n][j]), s);
    return fmul(N.af, tanh_rational(fadd(s, N.hb[n])));
}

// the output neuron on the summed hidden values (tanh :868)
__device__ __forceinline__ float lg_finish(const LegacyNet& N, float acc) { return fmul(N.af, tanh_rational(fadd(acc, N.ob))); }

}  // namespace ccnn
