// Sequential cascade bookkeeping, sort and box clustering on the device (one CTA).
//
// Reference order (src/CNNObjectDetector/cnn_detector_v3.cpp):
//   for every level, smallest first (RunCheckDetectAsync :2041-2049):
//     scan candidates in raster order; with drop_detect each one is tested against the
//       detections gathered so far (DropDetection :1820-1840): the first earlier box that
//       overlaps it by > 0.5 appends a copy (this box, that box's score/knn) and drops it, a box
//       that contains its 70 % core drops it (:1928-1941);
//     then for the survivors in order (CPUCheckDetect :1485-1818): a survivor overlapping
//       (> 0.5) a box appended since the scan appends a copy instead of running stages 2/3
//       (:1507-1527); otherwise the stage-2/3 verdict (precomputed by the window kernel)
//       appends the detection.
//   reverse, std::sort by scale (:2746-2750), Merger(0.5), min_num_detect filter,
//   Merger(0.2, del) (:2753-2772), optional rescale for shrunken gray input (:2785-2806).
//
// The scan test of a level against the detections of earlier levels has no order dependence,
// so all warps run it in parallel (one warp per candidate, 32 earlier boxes per ballot).
// Every box a level appends has the geometry of one of that level's candidates, so the tests
// against boxes appended during the level (its own scan, then the survivors' pass) are candidate
// pairs: all warps evaluate them into bit matrices first, and warp 0 then replays the order-
// dependent decisions with one ballot over the bit words per candidate. Levels with more than
// kBitMax candidates take the direct route (warp 0 tests the appended boxes 32 at a time). The sort
// permutes (scale, index) keys. The first clustering pass runs per group of boxes that cannot
// interact (a warp a group, its boxes in the lanes), the second on bit matrices of its pair tests; lists too long
// for the shared scratch take one warp through the reference's loop. Without drop_detect no candidate depends on
// another, and the accepted ones are listed at once.
// Bound by the latency of its dependent steps (one block). On B200, SM cycles of a warm run, before and after the
// merges took their boxes into lanes, pair tests lost their divisions and doubles, scores were left to a pass after
// the loop, and the block went from 1,024 to 512 threads: a 1920x1080 frame (221 candidates, 67 boxes) 115 K -> 102 K,
// a 640x480 one 57 K -> 46 K, a 1280x720 one with facial analysis (83 candidates, no drop_detect) 101 K -> 42 K.
#include <climits>
#include <vector>

#include "kernels.h"
#include "replay.cuh"
#include "window_common.cuh"

namespace ccnn {

// most steps are short dependent chains that every warp walks through: 1,024 threads took 2-9 % longer
constexpr int kRT = 512;

// v = (a, a2, b, b2), the two boxes' edges on an axis, in ascending order. Edges of overlapping boxes that are not
// inside out take one min / max step.
__device__ __forceinline__ void sort4(int* v) {
    const int m1 = imax(v[0], v[2]), m2 = imin(v[1], v[3]);
    if (v[0] <= v[1] && v[2] <= v[3] && m1 <= m2) {
        const int lo = imin(v[0], v[2]), hi = imax(v[1], v[3]);
        v[0] = lo;
        v[1] = m1;
        v[2] = m2;
        v[3] = hi;
        return;
    }
    // any correct sort gives the same ascending values
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3 - i; ++j)
            if (v[j] > v[j + 1]) {
                int t = v[j];
                v[j] = v[j + 1];
                v[j + 1] = t;
            }
}

// Merger's pair test (cnn_detector_v3.cpp:2842-2881). Returns ratio > threshold and the data
// needed to apply the merge.
struct MergeTest {
    bool hit;
    bool s1_gt_s2;
    int X[4], Y[4];
};

__device__ __forceinline__ MergeTest merge_test(const Det& a, const Det& b, float threshold) {
    MergeTest t;
    t.hit = false;
    t.s1_gt_s2 = false;
    int X[4] = {a.x, a.x2, b.x, b.x2};
    int Y[4] = {a.y, a.y2, b.y, b.y2};
    if (X[0] >= X[3] || X[1] <= X[2] || Y[0] >= Y[3] || Y[1] <= Y[2]) return t;
    const int s1 = (X[1] - X[0]) * (Y[1] - Y[0]);
    const int s2 = (X[3] - X[2]) * (Y[3] - Y[2]);
    sort4(X);
    sort4(Y);
    const int sui = (X[3] - X[0]) * (Y[3] - Y[0]);
    const int sii = (X[2] - X[1]) * (Y[2] - Y[1]);
    const int CX1 = X[0] + ((X[3] - X[0]) >> 1);
    const int CY1 = Y[0] + ((Y[3] - Y[0]) >> 1);
    const int CX2 = X[1] + ((X[2] - X[1]) >> 1);
    const int CY2 = Y[1] + ((Y[2] - Y[1]) >> 1);
    const int thrC = imin(X[3] - X[0], X[2] - X[1]) >> 1;
    const bool centred = abs(CX1 - CX2) < thrC && abs(CY1 - CY2) < thrC;
    // r1 = si / S1, r2 = si / S2, r3 = si / su as the reference rounds them, compared without dividing:
    // min(r1, r2) > threshold is both > threshold, max(r1, r2) > 0.7 is either
    if (s1 > 0 && s1 < kQuotMax && s2 > 0 && s2 < kQuotMax && sui > 0 && sui < kQuotMax && sii >= 0 && sii < kQuotMax && threshold >= 0x1p-12f &&
        threshold <= 1.f) {
        const QuotBound bt = quot_bound(__float_as_uint(threshold)), b7 = quot_bound(0x3f333333u);  // 0.7f
        const bool over = centred && quot_gt_int(sii, sui, quot_bound(__float_as_uint(fmul(0.75f, threshold)))) &&
                          (quot_gt_int(sii, s1, b7) || quot_gt_int(sii, s2, b7));
        t.hit = over ? (1.f > threshold) : (quot_gt_int(sii, s1, bt) && quot_gt_int(sii, s2, bt));
        t.s1_gt_s2 = s1 > s2;
    } else {
        const float S1 = (float)s1, S2 = (float)s2, su = (float)sui, si = (float)sii;
        const float r1 = fdiv(si, S1), r2 = fdiv(si, S2), r3 = fdiv(si, su);
        float ratio = r1 > r2 ? r2 : r1;
        if (r3 > fmul(0.75f, threshold) && (r1 < r2 ? r2 : r1) > 0.7f && centred) ratio = 1.f;
        t.hit = ratio > threshold;
        t.s1_gt_s2 = S1 > S2;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        t.X[i] = X[i];
        t.Y[i] = Y[i];
    }
    return t;
}

// Merger(0.5), or with del Merger(0.2, del) (cnn_detector_v3.cpp:2814-2936), run by one warp. in[] is read-only; checked[] is scratch.
// clus (optional): cluster (output index) of every input box; src (optional): input index of
// every output box.
template <bool del>
__device__ int merger_warp(const Det* in, int n, uint8_t* checked, Det* out, int* clus = nullptr, int* src = nullptr) {
    constexpr float threshold = del ? 0.2f : 0.5f;  // a constant, so that the bounds of the pair test are too
    const int lane = threadIdx.x & 31;
    for (int k = lane; k < n; k += 32) checked[k] = 0;
    __syncwarp();
    int nout = 0;
    for (int i1 = 0; i1 < n; ++i1) {
        if (checked[i1]) continue;
        Det nmax = in[i1], nmin = in[i1];
        bool dropped = false;
        // bound by the latency of its loads: the next 32 boxes and their flags are loaded ahead (only flags of the
        // current ones change meanwhile). NMS of 2,000 boxes takes 7.1 ms on B200, 12.0 without
        bool live_next = i1 + 1 + lane < n && !checked[i1 + 1 + lane];
        Det e_next = in[imin(i1 + 1 + lane, n - 1)];
        for (int base = i1 + 1; base < n && !dropped; base += 32) {
            const int j = base + lane;
            bool live = live_next;
            const Det e = e_next;
            live_next = j + 32 < n && !checked[j + 32];
            e_next = in[imin(j + 32, n - 1)];
            if (del) {
                const MergeTest mt = merge_test(nmax, e, threshold);
                const bool pred = live && mt.hit;
                const unsigned mb = __ballot_sync(0xffffffffu, pred && !mt.s1_gt_s2);
                const int lim = mb ? __ffs(mb) - 1 : 32;
                if (pred && mt.s1_gt_s2 && lane < lim) checked[j] = 1;
                if (mb) dropped = true;
            } else {
                // the first lane (at or after `start`) whose box merges into the running cluster is
                // absorbed; every lane then re-tests against the grown cluster box. The absorbed
                // box is read by all lanes from shared memory (a broadcast), not shuffled.
                int start = 0;
                while (true) {
                    const MergeTest mt = merge_test(nmax, e, threshold);
                    const bool pred = live && lane >= start && mt.hit;
                    const unsigned m = __ballot_sync(0xffffffffu, pred);
                    if (!m) break;
                    const int f = __ffs(m) - 1;
                    const Det ef = in[base + f];
                    int X[4] = {nmax.x, nmax.x2, ef.x, ef.x2};
                    int Y[4] = {nmax.y, nmax.y2, ef.y, ef.y2};
                    sort4(X);
                    sort4(Y);
                    nmax.x = imin(nmax.x, X[0]);
                    nmax.y = imin(nmax.y, Y[0]);
                    nmax.x2 = imax(nmax.x2, X[3]);
                    nmax.y2 = imax(nmax.y2, Y[3]);
                    nmin.x = imax(nmin.x, X[1]);
                    nmin.y = imax(nmin.y, Y[1]);
                    nmin.x2 = imin(nmin.x2, X[2]);
                    nmin.y2 = imin(nmin.y2, Y[2]);
                    nmax.score = (nmax.score < ef.score) ? ef.score : nmax.score;
                    nmax.knn = imax(nmax.knn, ef.knn);
                    nmax.scale = (nmax.scale > ef.scale) ? ef.scale : nmax.scale;
                    nmax.num_detect++;
                    if (lane == f) {
                        checked[j] = 1;
                        live = false;
                        if (clus) clus[j] = nout;
                    }
                    start = f + 1;
                }
            }
            __syncwarp();
        }
        if (del && dropped) continue;
        if (lane == 0) {
            if (clus) clus[i1] = nout;
            if (src) src[nout] = i1;
        }
        Det r = nmax;
        r.x = (nmin.x + nmax.x) >> 1;
        r.y = (nmin.y + nmax.y) >> 1;
        r.x2 = (nmin.x2 + nmax.x2) >> 1;
        r.y2 = (nmin.y2 + nmax.y2) >> 1;
        r.w = r.x2 - r.x;
        r.h = r.y2 - r.y;
        if (lane == 0) out[nout] = r;
        nout++;
        __syncwarp();
    }
    return nout;
}

// ---- the first merge by independent groups ----
// Merger(0.5, false) grows a cluster box as the bounding box of the boxes it absorbed, and a box
// only merges into a cluster box it overlaps. Split the boxes into groups whose bounding boxes do not
// overlap each other (the overlap relation closed under bounding boxes): no cluster box of one group
// can then overlap a box of another, so each group runs the reference's loop on its own and the
// clusters, listed by their first box, come out in the order of the single loop.

// concurrent union-find in shared memory: parent[x] <= x, roots have parent[x] == x. Linking CASes
// the larger root onto the smaller and retries from the value found (the hooking of Jaiganesh and
// Burtscher's ECL-CC, SC'18); roots only ever move to a smaller index, so a compression write, even
// a late one, still points at an ancestor.
__device__ __forceinline__ int uf_root(volatile int* parent, int x) {
    int cur = parent[x];
    if (cur != x) {
        int prev = x, next;
        while (cur > (next = parent[cur])) {
            parent[prev] = next;
            prev = cur;
            cur = next;
        }
    }
    return cur;
}

__device__ __forceinline__ bool uf_hook(volatile int* parent, int a, int b) {
    int ra = uf_root(parent, a), rb = uf_root(parent, b);
    while (ra != rb) {
        if (ra < rb) {
            const int t = ra;
            ra = rb;
            rb = t;
        }
        const int old = atomicCAS(const_cast<int*>(parent + ra), ra, rb);
        if (old == ra) return true;
        ra = old;
    }
    return false;
}

// The reference's loop over the boxes of group r (parent[j] == r) by one warp, as merger_warp does
// for the whole list; seed_box[i1] / seed_of[j]: the merged box of the cluster that box i1 starts,
// the first box of the cluster that absorbed box j.
__device__ void merge_group_warp(const Det* in, int n, const int* parent, int r, uint8_t* checked, Det* seed_box, int* seed_of) {
    const int lane = threadIdx.x & 31;
    for (int cb = r & ~31; cb < n; cb += 32) {
        const int jj = cb + lane;
        unsigned mm = __ballot_sync(0xffffffffu, jj < n && jj >= r && parent[jj] == r);
        while (mm) {
            const int i1 = cb + __ffs(mm) - 1;
            mm &= mm - 1;
            if (checked[i1]) continue;
            Det nmax = in[i1], nmin = in[i1];
            for (int base = i1 + 1; base < n; base += 32) {
                const int j = base + lane;
                bool live = j < n && parent[j] == r && !checked[j];
                if (!__any_sync(0xffffffffu, live)) continue;
                const Det e = live ? in[j] : nmax;
                int start = 0;
                while (true) {
                    const MergeTest mt = merge_test(nmax, e, 0.5f);
                    const unsigned m = __ballot_sync(0xffffffffu, live && lane >= start && mt.hit);
                    if (!m) break;
                    const int f = __ffs(m) - 1;
                    const Det ef = in[base + f];
                    int X[4] = {nmax.x, nmax.x2, ef.x, ef.x2};
                    int Y[4] = {nmax.y, nmax.y2, ef.y, ef.y2};
                    sort4(X);
                    sort4(Y);
                    nmax.x = imin(nmax.x, X[0]);
                    nmax.y = imin(nmax.y, Y[0]);
                    nmax.x2 = imax(nmax.x2, X[3]);
                    nmax.y2 = imax(nmax.y2, Y[3]);
                    nmin.x = imax(nmin.x, X[1]);
                    nmin.y = imax(nmin.y, Y[1]);
                    nmin.x2 = imin(nmin.x2, X[2]);
                    nmin.y2 = imin(nmin.y2, Y[2]);
                    nmax.score = (nmax.score < ef.score) ? ef.score : nmax.score;
                    nmax.knn = imax(nmax.knn, ef.knn);
                    nmax.scale = (nmax.scale > ef.scale) ? ef.scale : nmax.scale;
                    nmax.num_detect++;
                    if (lane == f) {
                        checked[j] = 1;
                        live = false;
                        seed_of[j] = i1;
                    }
                    start = f + 1;
                }
                __syncwarp();
            }
            Det rr = nmax;
            rr.x = (nmin.x + nmax.x) >> 1;
            rr.y = (nmin.y + nmax.y) >> 1;
            rr.x2 = (nmin.x2 + nmax.x2) >> 1;
            rr.y2 = (nmin.y2 + nmax.y2) >> 1;
            rr.w = rr.x2 - rr.x;
            rr.h = rr.y2 - rr.y;
            if (lane == 0) {
                seed_of[i1] = i1;
                seed_box[i1] = rr;
            }
            __syncwarp();
        }
    }
}

// The same for a group of at most 32 boxes, lane k its k-th (idx: its index, -1 past the last): the boxes stay in
// registers, and a test of the running cluster covers all that are left (the boxes of a group are spread over
// the list, so merge_group_warp takes several tests for the same). The steps are one dependent chain, so where
// no box is inside out and the whole group's box is below 2^24 pixels the test is cut down to what depends on the
// growing cluster (`quick`).
__device__ void merge_group_lanes(const Det* in, int idx, Det* seed_box, int* seed_of) {
    const int lane = threadIdx.x & 31;
    constexpr unsigned kAll = 0xffffffffu;
    unsigned alive = __ballot_sync(kAll, idx >= 0);
    const Det e = in[imax(idx, 0)];  // a lane past the last repeats a box of the list
    const int gx0 = __reduce_min_sync(kAll, idx >= 0 ? e.x : INT_MAX), gx1 = __reduce_max_sync(kAll, idx >= 0 ? e.x2 : INT_MIN);
    const int gy0 = __reduce_min_sync(kAll, idx >= 0 ? e.y : INT_MAX), gy1 = __reduce_max_sync(kAll, idx >= 0 ? e.y2 : INT_MIN);
    const bool quick = __all_sync(kAll, idx < 0 || (e.x < e.x2 && e.y < e.y2)) && (long long)gx1 - gx0 < kQuotMax && (long long)gy1 - gy0 < kQuotMax &&
                       ((long long)gx1 - gx0) * ((long long)gy1 - gy0) < kQuotMax;
    constexpr QuotBound b5 = quot_bound(0x3f000000u), b375 = quot_bound(0x3ec00000u), b7 = quot_bound(0x3f333333u);  // 0.5, 0.75 * 0.5, 0.7
    const int s2 = quick ? (e.x2 - e.x) * (e.y2 - e.y) : 0;
    while (alive) {
        const int s = __ffs(alive) - 1;
        const int i1 = __shfl_sync(kAll, idx, s);
        Det nmax = in[i1], nmin = nmax;
        alive &= alive - 1;
        unsigned later = alive;  // those not yet passed by this cluster
        while (later) {
            bool hit;
            if (quick) {
                // merge_test of two boxes with edges in order
                const int x1 = imax(nmax.x, e.x), x2 = imin(nmax.x2, e.x2), x0 = imin(nmax.x, e.x), x3 = imax(nmax.x2, e.x2);
                const int y1 = imax(nmax.y, e.y), y2 = imin(nmax.y2, e.y2), y0 = imin(nmax.y, e.y), y3 = imax(nmax.y2, e.y2);
                const int s1 = (nmax.x2 - nmax.x) * (nmax.y2 - nmax.y);
                const int su = (x3 - x0) * (y3 - y0), si = (x2 - x1) * (y2 - y1);
                const int thr_c = imin(x3 - x0, x2 - x1) >> 1;
                const bool centred = abs((x0 + ((x3 - x0) >> 1)) - (x1 + ((x2 - x1) >> 1))) < thr_c &&
                                     abs((y0 + ((y3 - y0) >> 1)) - (y1 + ((y2 - y1) >> 1))) < thr_c;
                const bool over = centred & quot_gt_int(si, su, b375) & (quot_gt_int(si, s1, b7) | quot_gt_int(si, s2, b7));
                hit = (x1 < x2) & (y1 < y2) & (over | (quot_gt_int(si, s1, b5) & quot_gt_int(si, s2, b5)));
            } else {
                hit = merge_test(nmax, e, 0.5f).hit;
            }
            const unsigned m = __ballot_sync(kAll, hit) & later;
            if (!m) break;
            const int f = __ffs(m) - 1;
            const int jf = __shfl_sync(kAll, idx, f);
            const Det ef = in[jf];
            int X[4] = {nmax.x, nmax.x2, ef.x, ef.x2};
            int Y[4] = {nmax.y, nmax.y2, ef.y, ef.y2};
            sort4(X);
            sort4(Y);
            nmax.x = imin(nmax.x, X[0]);
            nmax.y = imin(nmax.y, Y[0]);
            nmax.x2 = imax(nmax.x2, X[3]);
            nmax.y2 = imax(nmax.y2, Y[3]);
            nmin.x = imax(nmin.x, X[1]);
            nmin.y = imax(nmin.y, Y[1]);
            nmin.x2 = imin(nmin.x2, X[2]);
            nmin.y2 = imin(nmin.y2, Y[2]);
            nmax.score = (nmax.score < ef.score) ? ef.score : nmax.score;
            nmax.knn = imax(nmax.knn, ef.knn);
            nmax.scale = (nmax.scale > ef.scale) ? ef.scale : nmax.scale;
            nmax.num_detect++;
            if (lane == f) seed_of[jf] = i1;
            alive &= ~(1u << f);
            later &= ~((2u << f) - 1u);
        }
        Det rr = nmax;
        rr.x = (nmin.x + nmax.x) >> 1;
        rr.y = (nmin.y + nmax.y) >> 1;
        rr.x2 = (nmin.x2 + nmax.x2) >> 1;
        rr.y2 = (nmin.y2 + nmax.y2) >> 1;
        rr.w = rr.x2 - rr.x;
        rr.h = rr.y2 - rr.y;
        if (lane == 0) {
            seed_of[i1] = i1;
            seed_box[i1] = rr;
        }
    }
    __syncwarp();
}

// Merger(0.5, false) of n <= kGroupMax sorted boxes by the whole block; returns the cluster count
// (every thread). out: the clusters in reference order; seed_box: n Det of scratch; clus (optional):
// cluster of every box; ws_a / ws_b: 4n / 3n ints of shared memory.
constexpr int kGroupMax = 512;
__device__ int first_merge_groups(const Det* in, int n, uint8_t* checked, Det* out, Det* seed_box, int* clus, int* ws_a, int* ws_b) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    volatile int* parent = ws_a;
    int* bx0 = ws_a + n;
    int* by0 = ws_a + 2 * n;
    int* bx1 = ws_a + 3 * n;
    int* by1 = ws_b;
    int* seed_of = ws_b + n;
    int* rank_of = ws_b + 2 * n;
    __shared__ int s_groups;
    __shared__ uint16_t s_member[kRT / 32][32];
    const bool one = n <= 32;  // a single warp's worth: no groups
    if (one && warp == 0) merge_group_lanes(in, lane < n ? lane : -1, seed_box, seed_of);
    for (int j = tid; j < n && !one; j += blockDim.x) {
        parent[j] = j;
        checked[j] = 0;
    }
    __syncthreads();
    // boxes that overlap or touch share a group
    for (int i = warp; i < n && !one; i += nwarps) {
        const Det bi = in[i];
        const int ax0 = imin(bi.x, bi.x2), ax1 = imax(bi.x, bi.x2), ay0 = imin(bi.y, bi.y2), ay1 = imax(bi.y, bi.y2);
        for (int j = i + 1 + lane; j < n; j += 32) {
            const Det bj = in[j];
            if (ax0 <= imax(bj.x, bj.x2) && imin(bj.x, bj.x2) <= ax1 && ay0 <= imax(bj.y, bj.y2) && imin(bj.y, bj.y2) <= ay1)
                uf_hook(parent, i, j);
        }
    }
    __syncthreads();
    // groups whose bounding boxes overlap or touch are joined until none do
    while (!one) {
        for (int j = tid; j < n; j += blockDim.x) {
            int v = parent[j];
            while (v != parent[v]) v = parent[v];
            parent[j] = v;  // only this thread writes parent[j] in this pass
            bx0[j] = by0[j] = INT_MAX;
            bx1[j] = by1[j] = INT_MIN;
        }
        __syncthreads();
        for (int j = tid; j < n; j += blockDim.x) {
            const Det b = in[j];
            const int g = parent[j];
            atomicMin(&bx0[g], imin(b.x, b.x2));
            atomicMin(&by0[g], imin(b.y, b.y2));
            atomicMax(&bx1[g], imax(b.x, b.x2));
            atomicMax(&by1[g], imax(b.y, b.y2));
        }
        __syncthreads();
        bool linked = false;
        for (int i = warp; i < n; i += nwarps) {
            if (parent[i] != i) continue;
            for (int j = i + 1 + lane; j < n; j += 32)
                if (parent[j] == j && bx0[i] <= bx1[j] && bx0[j] <= bx1[i] && by0[i] <= by1[j] && by0[j] <= by1[i])
                    linked |= uf_hook(parent, i, j);
        }
        if (!__syncthreads_or(linked)) break;
    }
    // a pass without links left every parent a root: group g = the root; warp w takes the groups
    // w, w + nwarps, ... in order of their roots
    int ord = 0;
    for (int cb = 0; cb < n && !one; cb += 32) {
        const int j = cb + lane;
        unsigned rm = __ballot_sync(0xffffffffu, j < n && parent[j] == j);
        while (rm) {
            const int g = cb + __ffs(rm) - 1;
            rm &= rm - 1;
            if (ord++ % nwarps != warp) continue;
            int members = 0;
            for (int mb = g & ~31; mb < n; mb += 32) {
                const int k = mb + lane;
                const bool in_g = k < n && parent[k] == g;
                const unsigned mm = __ballot_sync(0xffffffffu, in_g);
                const int pos = members + __popc(mm & ((1u << lane) - 1u));
                if (in_g && pos < 32) s_member[warp][pos] = (uint16_t)k;
                members += __popc(mm);
            }
            __syncwarp();
            if (members <= 32)
                merge_group_lanes(in, lane < members ? s_member[warp][lane] : -1, seed_box, seed_of);
            else
                merge_group_warp(in, n, const_cast<const int*>(ws_a), g, checked, seed_box, seed_of);
        }
    }
    __syncthreads();
    // clusters ranked by their first box
    if (warp == 0) {
        int w = 0;
        for (int cb = 0; cb < n; cb += 32) {
            const int j = cb + lane;
            const bool s = j < n && seed_of[j] == j;
            const unsigned m = __ballot_sync(0xffffffffu, s);
            if (s) rank_of[j] = w + __popc(m & ((1u << lane) - 1u));
            w += __popc(m);
        }
        if (lane == 0) s_groups = w;
    }
    __syncthreads();
    const int nM = s_groups;
    for (int j = tid; j < n; j += blockDim.x) {
        const int s = seed_of[j];
        if (s == j) out[rank_of[j]] = seed_box[j];
        if (clus) clus[j] = rank_of[s];
    }
    __syncthreads();
    return nM;
}

// Merger(0.2, true) of n <= 256 boxes by the whole block. With deletion a box never grows, so each
// pair test depends on the two boxes only: bit j of word w of row i (j = 32w + bit > i) is set in
// `take` when box i deletes box j (the test hits and box i is larger), in `drop` when box j deletes
// box i. The reference's loop then runs on bit sets in warp 0: a box not yet deleted deletes its live
// `take` boxes up to its first live `drop` box, and is itself dropped if there is one.
// take / drop: n * ceil(n / 32) words each. Returns the output count (every thread).
__device__ int second_merge_bits(const Det* in, int n, Det* out, int* src, uint32_t* take, uint32_t* drop) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int W = (n + 31) >> 5;
    __shared__ int s_out;
    for (int it = warp; it < n * W; it += nwarps) {
        const int i = it / W, w = it - i * W;
        const int j = 32 * w + lane;
        bool hit = false, gt = false;
        if (j > i && j < n) {
            const MergeTest mt = merge_test(in[i], in[j], 0.2f);
            hit = mt.hit;
            gt = mt.s1_gt_s2;
        }
        const uint32_t bt = __ballot_sync(0xffffffffu, hit && gt), bd = __ballot_sync(0xffffffffu, hit && !gt);
        if (lane == 0) {
            take[it] = bt;
            drop[it] = bd;
        }
    }
    __syncthreads();
    if (warp == 0) {
        uint32_t del = 0u;  // lane w < W: the deleted boxes of word w
        int nout = 0;
        for (int i = 0; i < n; ++i) {
            if ((__shfl_sync(0xffffffffu, del, i >> 5) >> (i & 31)) & 1u) continue;
            const uint32_t t = lane < W ? take[i * W + lane] & ~del : 0u;
            const uint32_t d = lane < W ? drop[i * W + lane] & ~del : 0u;
            const unsigned dm = __ballot_sync(0xffffffffu, d != 0u);
            if (dm) {
                const int wf = __ffs(dm) - 1;
                const uint32_t first = __shfl_sync(0xffffffffu, d, wf);
                if (lane < wf) del |= t;
                else if (lane == wf) del |= t & ((1u << (__ffs(first) - 1)) - 1u);
                continue;
            }
            del |= t;
            if (lane == 0) {
                const Det b = in[i];
                Det rr = b;
                rr.x = (b.x + b.x) >> 1;
                rr.y = (b.y + b.y) >> 1;
                rr.x2 = (b.x2 + b.x2) >> 1;
                rr.y2 = (b.y2 + b.y2) >> 1;
                rr.w = rr.x2 - rr.x;
                rr.h = rr.y2 - rr.y;
                out[nout] = rr;
                if (src) src[nout] = i;
            }
            nout++;
        }
        if (lane == 0) s_out = nout;
    }
    __syncthreads();
    return s_out;
}

constexpr int kMaxLevels = 1024;
// what the loop needs of a level: its scale and its candidates' pattern size
struct LevelRect {
    float scale, inv_scale;
    int w, h;
};
constexpr int kLevelSmem = 128;  // levels kept in shared memory (deeper pyramids make the rest from global)

constexpr int kBitMax = 256;              // candidates per level handled with bit matrices
constexpr int kBitWords = kBitMax / 32;
constexpr int kOwnVerdict = -kBitMax - 1;  // the candidate's own stage-2/3 verdict (or stage-1 score, detection disabled)

__device__ __forceinline__ void replay_body(const ReplayArgs& a) {
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ int s_lvl_start[kMaxLevels + 1];
    __shared__ int s_nD, s_nS;
    // bit j of word w of row i: drop_test(candidate i, box of candidate 32w + j) == 1 (A1) / == 2 (A2)
    __shared__ uint32_t s_a1[kBitMax * kBitWords], s_a2[kBitMax * kBitWords];
    __shared__ int s_didx[kBitMax];  // D index of the box a candidate appended, or -1
    __shared__ int s_src[kBitMax];   // where that box's score/knn come from
    __shared__ uint32_t s_S[kBitWords], s_T[kBitWords];  // candidate sets of the level (see below)
    __shared__ LevelRect s_lv[kLevelSmem];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const CascadeConfig& C = a.cfg;
    const int n = *a.n_cand;
    const int nl = a.n_levels;

    // working set in shared memory when it fits (121 bytes per candidate), else global scratch:
    //   region A: candidates, verdicts, scan results, survivors (40 B each); later the first merge
    //   region B: detections in reference order; later the second merge
    //   region C: reversed + sorted detections; region E: merge flags
    const bool fits = (long long)n * 121 + 64 <= kReplaySmemBytes;
    Candidate* cands;
    CandResult* res;
    int* first_dec;
    int* surv;
    Det *D, *R, *M, *F;
    uint8_t* checked;
    if (fits) {
        unsigned char* p = sm;
        cands = reinterpret_cast<Candidate*>(p);
        res = reinterpret_cast<CandResult*>(p + 16LL * n);
        first_dec = reinterpret_cast<int*>(p + 32LL * n);
        surv = reinterpret_cast<int*>(p + 36LL * n);
        M = reinterpret_cast<Det*>(p);
        D = reinterpret_cast<Det*>(p + 40LL * n);
        F = D;
        R = reinterpret_cast<Det*>(p + 80LL * n);
        checked = p + 120LL * n;
        for (int i = tid; i < n; i += kRT) cands[i] = a.cands[i];
    } else {
        cands = const_cast<Candidate*>(a.cands);
        res = a.results;
        first_dec = a.first_dec;
        surv = a.survivors;
        D = a.D;
        R = a.R;
        M = a.M;
        F = a.F;
        checked = a.checked;
    }
    // With drop_detect, the candidate-pair tests of every level (bit j of word w of candidate i's row:
    // drop_test(candidate i, box of candidate 32w + j of the same level) == 1 / == 2) are evaluated
    // for all levels at once before the level loop, where the rows (kBitWords words per candidate)
    // fit in shared memory beside the working set; the loop then only reads them.
    const bool pre_rows = fits && C.drop_detect && ((121LL * n + 15) & ~15LL) + 8LL * kBitWords * n <= kReplaySmemBytes;
    uint32_t* P1 = pre_rows ? reinterpret_cast<uint32_t*>(sm + ((121LL * n + 15) & ~15LL)) : nullptr;
    uint32_t* P2 = pre_rows ? P1 + (size_t)kBitWords * n : nullptr;
    for (int l = tid; l <= nl; l += kRT) s_lvl_start[l] = 0;
    auto load_level = [&](int l) {
        const float inv = a.levels[l].inv_scale;
        return LevelRect{a.levels[l].scale, inv, (int)((float)C.pat_w * inv), (int)((float)C.pat_h * inv)};
    };
    for (int l = tid; l < nl && l < kLevelSmem; l += kRT) s_lv[l] = load_level(l);
    auto level_rect = [&](int l) { return l < kLevelSmem ? s_lv[l] : load_level(l); };
    // the candidate's stage-1 pattern rectangle (new_rect, cnn_detector_v3.cpp:1497-1501); the pattern is the stage-1
    // network's smallest input. In the shared copy px and py are made the rectangle's corner below.
    auto cand_rect = [&](const Candidate& c, const LevelRect& L) {
        return make_det(fits ? c.px : (int)((float)c.px * L.inv_scale), fits ? c.py : (int)((float)c.py * L.inv_scale), L.w, L.h, 0.f, L.scale, 0);
    };
    __syncthreads();
    // verdicts and per-level candidate counts (candidates are grouped by level, smallest first)
    for (int i = tid; i < n; i += kRT) {
        const Candidate cd = cands[i];
        if (C.detect_enabled) {
            const CandResult r = verdict(a.win + (size_t)i * 4, cd, level_rect(cd.level).scale, C);
            if (fits) a.results[i] = r;  // kept for inspection
            res[i] = r;
            // facial analysis drops a window whose landmarks collapse (cnn_detector_v3.cpp:1750)
            res[i].pad = r.accepted && !(a.attr && a.attr[i].x);
        }
        if (fits) {
            const float inv = level_rect(cd.level).inv_scale;
            cands[i].px = (int)((float)cd.px * inv);
            cands[i].py = (int)((float)cd.py * inv);
        }
        atomicAdd(&s_lvl_start[nl - 1 - cd.level + 1], 1);
    }
    __syncthreads();
    if (tid == 0) {
        for (int k = 1; k <= nl; ++k) s_lvl_start[k] += s_lvl_start[k - 1];
        s_nD = 0;
    }
    __syncthreads();
    if (pre_rows) {
        // a warp a candidate row, one ballot a word
        for (int c = warp; c < n; c += kRT / 32) {
            const Candidate cd = cands[c];
            const int k = nl - 1 - cd.level;
            const int g = s_lvl_start[k], m = s_lvl_start[k + 1] - g, i = c - g;
            if (m > kBitMax) continue;
            const LevelRect L = level_rect(cd.level);
            const Det nr = cand_rect(cd, L);
            const Det ex = rect_shrink(nr, 0.7f);
            for (int w = 0; w < ((i + 31) >> 5); ++w) {
                const int j = 32 * w + lane;
                int t = 0;
                if (j < i) t = drop_test(nr, ex, cand_rect(cands[g + j], L));
                const uint32_t b1 = __ballot_sync(0xffffffffu, t == 1), b2 = __ballot_sync(0xffffffffu, t == 2);
                if (lane == 0) {
                    P1[(size_t)c * kBitWords + w] = b1;
                    P2[(size_t)c * kBitWords + w] = b2;
                }
            }
            // words at and past the candidate's own index stay 0
            if (lane < kBitWords && lane >= ((i + 31) >> 5)) {
                P1[(size_t)c * kBitWords + lane] = 0u;
                P2[(size_t)c * kBitWords + lane] = 0u;
            }
        }
        __syncthreads();
    }

    int nD = 0;
    if (!C.drop_detect) {
        // no candidate depends on another: the accepted ones in order
        for (int base = 0; base < n; base += kRT) {
            const int i = base + tid;
            const bool in = i < n && (!C.detect_enabled || res[i].pad);
            const uint32_t word = __ballot_sync(0xffffffffu, in);
            if (lane == 0) s_didx[warp] = __popc(word);
            __syncthreads();
            int dst = nD + __popc(word & ((1u << lane) - 1u));
            for (int w = 0; w < kRT / 32; ++w) {
                if (w < warp) dst += s_didx[w];
                nD += s_didx[w];
            }
            if (in) {
                const LevelRect L = level_rect(cands[i].level);
                const Det nr = cand_rect(cands[i], L);
                D[dst] = make_det(nr.x, nr.y, nr.w, nr.h, 0.f, L.scale, -1 - i);
            }
            __syncthreads();
        }
    }
    for (int k = 0; k < nl && C.drop_detect; ++k) {
        const int g = s_lvl_start[k], e = s_lvl_start[k + 1];
        if (g == e) continue;
        const int lev = nl - 1 - k;
        const LevelRect L = level_rect(lev);
        const float scale = L.scale;
        const int n_prefix = nD;

        // scan test against the detections of earlier levels, one warp per candidate
        for (int c = g + warp; c < e; c += kRT / 32) {
            const Det nr = cand_rect(cands[c], L);
            const Det ex = rect_shrink(nr, 0.7f);
            int code = -1;
            // 64 boxes a step, loaded together: a list too long for shared memory is read from L2, and with 32 a step the
            // block's 16 warps did not cover its latency (a 640x480 frame of 250 levels, 7,253 candidates and 1,562
            // boxes: 7.9 ms, 6.3 with 32 warps, 5.4 now)
            for (int base = 0; base < n_prefix && code < 0; base += 64) {
                const int k0 = imin(base + lane, n_prefix - 1), k1 = imin(base + 32 + lane, n_prefix - 1);
                const Det e0 = D[k0], e1 = D[k1];
                int t[2] = {drop_test(nr, ex, e0), 0};
                if (base + 32 < n_prefix) t[1] = drop_test(nr, ex, e1);
#pragma unroll
                for (int h = 1; h >= 0; --h) {
                    // lanes past the last box tested it again; the lane it belongs to comes first
                    const unsigned m = __ballot_sync(0xffffffffu, t[h] != 0);
                    if (!m) continue;
                    const int f = __ffs(m) - 1;
                    code = (base + 32 * h + f) * 2 + (__shfl_sync(0xffffffffu, t[h], f) - 1);
                }
            }
            if (lane == 0) first_dec[c] = code;
        }
        const int m = e - g;
        const int W = (m + 31) >> 5;
        // box of candidate i of the level (scores follow after the loop): where its score and knn come from
        auto emit_box = [&](int i) {
            const int src = s_src[i];
            const Det nr = cand_rect(cands[g + i], L);
            D[s_didx[i]] = make_det(nr.x, nr.y, nr.w, nr.h, 0.f, scale, src >= 0 ? src : (src > kOwnVerdict ? s_didx[-1 - src] : -1 - (g + i)));
        };
        if (pre_rows) {
            // the level's rows, evaluated before the loop (levels of up to 32 read them in warp 0)
            if (m > 32 && m <= kBitMax)
                for (int it = tid; it < m * W; it += kRT) {
                    const int i = it / W, w = it - i * W;
                    s_a1[it] = P1[(size_t)(g + i) * kBitWords + w];
                    s_a2[it] = P2[(size_t)(g + i) * kBitWords + w];
                }
        } else if (m <= kBitMax) {
            // candidate-pair tests of this level, one ballot per (row i, word w)
            for (int it = warp; it < m * W; it += kRT / 32) {
                const int i = it / W, w = it - i * W;
                const int j = 32 * w + lane;
                int t = 0;
                if (j < i) {
                    const Det nr = cand_rect(cands[g + i], L);
                    t = drop_test(nr, rect_shrink(nr, 0.7f), cand_rect(cands[g + j], L));
                }
                const uint32_t b1 = __ballot_sync(0xffffffffu, t == 1), b2 = __ballot_sync(0xffffffffu, t == 2);
                if (lane == 0) {
                    s_a1[i * W + w] = b1;
                    s_a2[i * W + w] = b2;
                }
            }
        }
        __syncthreads();
        // The order-dependent decisions of the level as fixed points over candidate sets (bit j of
        // word w = candidate 32w + j). Candidate i's decision depends only on candidates j < i, so
        // after t rounds the first t candidates are final, and a round that changes nothing has
        // reached the unique solution, which is the sequential one.
        //   S: boxes appended during the scan: the first decisive box of candidate i (earlier
        //      levels first, then S in order) has drop type 1;
        //   T: boxes appended by the survivors' pass: survivor i overlaps (> 0.5) a box of T
        //      (a copy), or its stage-2/3 verdict accepts it (or detection is disabled).
        const bool check = C.detect_enabled != 0;
        if (m <= 32) {
            // one word: warp 0 alone, candidate i = lane, its rows and decisions in registers;
            // a round is one ballot
            if (warp == 0) {
                const int i = lane;
                const bool valid = i < m;
                int code = -1, acc = 0;
                uint32_t r1 = 0u, r2 = 0u;
                if (valid) {
                    code = first_dec[g + i];
                    acc = C.detect_enabled ? res[g + i].pad : 1;
                    r1 = pre_rows ? P1[(size_t)(g + i) * kBitWords] : s_a1[i];
                    r2 = pre_rows ? P2[(size_t)(g + i) * kBitWords] : s_a2[i];
                }
                uint32_t S = 0u;
                for (int round = 0; round <= m; ++round) {
                    bool in = false;
                    if (valid) {
                        if (code >= 0) {
                            in = (code & 1) == 0;
                        } else {
                            const uint32_t hit = (r1 | r2) & S;
                            if (hit) in = ((r1 >> (__ffs(hit) - 1)) & 1u) != 0u;
                        }
                    }
                    const uint32_t nS = __ballot_sync(0xffffffffu, in);
                    if (nS == S) break;
                    S = nS;
                }
                // survivors: not decided by the scan
                const bool surv_i = valid && code < 0 && ((r1 | r2) & S) == 0u;
                uint32_t T = 0u;
                for (int round = 0; round <= m; ++round) {
                    const bool in = surv_i && (acc != 0 || (check && (r1 & T) != 0u));
                    const uint32_t nT = __ballot_sync(0xffffffffu, in);
                    if (nT == T) break;
                    T = nT;
                }
                // D index (scan appends in candidate order, then the survivors' appends) and the
                // source of each box's score/knn
                const int nScan = __popc(S);
                const uint32_t below = (1u << i) - 1u;
                if (valid && (((S | T) >> i) & 1u)) {
                    // the box of candidate j < i of the level that decided this one
                    const uint32_t by = (S >> i) & 1u ? (r1 | r2) & S : (check ? r1 & T : 0u);
                    const uint32_t before = by ? (by & (0u - by)) - 1u : 0u;  // candidates in front of j
                    int dst, src;
                    if ((S >> i) & 1u) {
                        dst = nD + __popc(S & below);
                        src = code >= 0 ? code >> 1 : nD + __popc(S & before);
                    } else {
                        dst = nD + nScan + __popc(T & below);
                        src = by ? nD + nScan + __popc(T & before) : -1 - (g + i);
                    }
                    const Det nr = cand_rect(cands[g + i], L);
                    D[dst] = make_det(nr.x, nr.y, nr.w, nr.h, 0.f, scale, src);
                }
                if (lane == 0) s_nD = nD + nScan + __popc(T);
            }
            __syncthreads();
            nD = s_nD;
            continue;
        }
        if (m <= kBitMax) {
            // several words: a thread a candidate (m <= 256: warps 0..7), block-wide rounds
            const bool thread_item = tid < m;
            const int i = tid;
            int code = -1, acc = 0;
            if (thread_item) {
                code = first_dec[g + i];
                acc = C.detect_enabled ? res[g + i].pad : 1;
            }
            if (tid < kBitWords) {
                s_S[tid] = 0u;
                s_T[tid] = 0u;
            }
            __syncthreads();
            bool inS = false;
            for (int round = 0; round <= m; ++round) {
                bool in = false;
                if (thread_item) {
                    if (code >= 0) {
                        in = (code & 1) == 0;
                    } else {
                        for (int w = 0; w < W; ++w) {
                            const uint32_t hit = (s_a1[i * W + w] | s_a2[i * W + w]) & s_S[w];
                            if (hit) {
                                in = (s_a1[i * W + w] >> (__ffs(hit) - 1)) & 1u;
                                break;
                            }
                        }
                    }
                }
                const uint32_t word = __ballot_sync(0xffffffffu, in);
                __syncthreads();  // every thread has read the previous round's S
                const bool changed = (lane == 0 && warp < W && s_S[warp] != word);
                if (lane == 0 && warp < W) s_S[warp] = word;
                inS = in;
                if (!__syncthreads_or(changed)) break;
            }
            // survivors: not decided by the scan
            bool surv_i = false;
            if (thread_item && code < 0) {
                surv_i = true;
                for (int w = 0; w < W; ++w)
                    if ((s_a1[i * W + w] | s_a2[i * W + w]) & s_S[w]) {
                        surv_i = false;
                        break;
                    }
            }
            for (int round = 0; round <= m; ++round) {
                bool in = false;
                if (surv_i) {
                    in = acc != 0;
                    if (check)
                        for (int w = 0; w < W && !in; ++w) in = (s_a1[i * W + w] & s_T[w]) != 0u;
                }
                const uint32_t word = __ballot_sync(0xffffffffu, in);
                __syncthreads();
                const bool changed = (lane == 0 && warp < W && s_T[warp] != word);
                if (lane == 0 && warp < W) s_T[warp] = word;
                if (!__syncthreads_or(changed)) break;
            }
            int nScan = 0, nSurv = 0;
            for (int w = 0; w < W; ++w) {
                nScan += __popc(s_S[w]);
                nSurv += __popc(s_T[w]);
            }
            if (thread_item) {
                const uint32_t below = (1u << (i & 31)) - 1u;
                int dst = -1, src = 0;
                if (inS) {
                    int r = 0;
                    for (int w = 0; w < (i >> 5); ++w) r += __popc(s_S[w]);
                    dst = nD + r + __popc(s_S[i >> 5] & below);
                    if (code >= 0) {
                        src = code >> 1;
                    } else {
                        for (int w = 0; w < W; ++w) {
                            const uint32_t hit = (s_a1[i * W + w] | s_a2[i * W + w]) & s_S[w];
                            if (hit) {
                                src = -1 - (32 * w + __ffs(hit) - 1);
                                break;
                            }
                        }
                    }
                } else if ((s_T[i >> 5] >> (i & 31)) & 1u) {
                    int r = 0;
                    for (int w = 0; w < (i >> 5); ++w) r += __popc(s_T[w]);
                    dst = nD + nScan + r + __popc(s_T[i >> 5] & below);
                    src = kOwnVerdict;
                    if (check)
                        for (int w = 0; w < W; ++w) {
                            const uint32_t hit = s_a1[i * W + w] & s_T[w];
                            if (hit) {
                                src = -1 - (32 * w + __ffs(hit) - 1);
                                break;
                            }
                        }
                }
                s_didx[i] = dst;
                s_src[i] = src;
            }
            __syncthreads();
            if (thread_item && s_didx[i] >= 0) emit_box(i);
            nD += nScan + nSurv;
            __syncthreads();
            continue;
        }
        if (warp == 0) {
            int nS = 0;
            for (int c = g; c < e; ++c) {
                const int code = first_dec[c];
                int k0 = -1, type = 0;
                Det nr;
                if (code >= 0) {
                    k0 = code >> 1;
                    type = (code & 1) + 1;
                } else if (nD > n_prefix) {
                    nr = cand_rect(cands[c], L);
                    const Det ex = rect_shrink(nr, 0.7f);
                    for (int base = n_prefix; base < nD; base += 32) {
                        const int kk = base + lane;
                        const int t = kk < nD ? drop_test(nr, ex, D[kk]) : 0;
                        const unsigned m = __ballot_sync(0xffffffffu, t != 0);
                        if (m) {
                            const int f = __ffs(m) - 1;
                            type = __shfl_sync(0xffffffffu, t, f);
                            k0 = base + f;
                            break;
                        }
                    }
                }
                if (k0 >= 0) {
                    if (type == 1) {
                        if (lane == 0) {
                            nr = cand_rect(cands[c], L);
                            D[nD] = make_det(nr.x, nr.y, nr.w, nr.h, 0.f, scale, k0);
                        }
                        nD++;
                        __syncwarp();
                    }
                    continue;
                }
                if (lane == 0) surv[nS] = c;
                nS++;
            }
            if (lane == 0) {
                s_nS = nS;
                s_nD = nD;
            }
        }
        __syncthreads();
        nD = s_nD;

        if (warp == 0) {
            const int nS = s_nS;
            const int rect_size = nD;
            for (int si = 0; si < nS; ++si) {
                const int c = surv[si];
                const Candidate cd = cands[c];
                const Det nr = cand_rect(cd, L);
                if (C.detect_enabled && nD > rect_size) {
                    int k0 = -1;
                    for (int base = rect_size; base < nD; base += 32) {
                        const int kk = base + lane;
                        const bool hit = kk < nD && rect_overlap(nr, D[kk]) > 0.5f;
                        const unsigned m = __ballot_sync(0xffffffffu, hit);
                        if (m) {
                            k0 = base + __ffs(m) - 1;
                            break;
                        }
                    }
                    if (k0 >= 0) {
                        if (lane == 0) D[nD] = make_det(nr.x, nr.y, nr.w, nr.h, 0.f, scale, k0);
                        nD++;
                        __syncwarp();
                        continue;
                    }
                }
                if (!C.detect_enabled || res[c].pad) {
                    if (lane == 0) D[nD] = make_det(nr.x, nr.y, nr.w, nr.h, 0.f, scale, -1 - c);
                    nD++;
                }
                __syncwarp();
            }
            if (lane == 0) s_nD = nD;
        }
        __syncthreads();
        nD = s_nD;
    }

    // scores and knn: a box's knn field holds the box it is a copy of, or -1 - its own candidate, so each copy chain
    // ends at a candidate (kept in num_detect until every chain has been read). Facial data travels with a
    // candidate's own accepted box, not with copies.
    for (int i = tid; i < nD; i += kRT) {
        int src = D[i].knn;
        if (a.fa_scratch) a.fa_scratch[i] = src < 0 && C.detect_enabled ? -1 - src : -1;
        while (src >= 0) src = D[src].knn;
        D[i].num_detect = -1 - src;
    }
    __syncthreads();
    for (int i = tid; i < nD; i += kRT) {
        const int c = D[i].num_detect;
        D[i].score = C.detect_enabled ? res[c].score : cands[c].score;
        D[i].knn = C.detect_enabled ? res[c].knn : 0;
        D[i].num_detect = 0;
    }
    __syncthreads();  // the keys below take the place of the candidates and verdicts
    // raw list (reference order) to global memory for inspection; the reversed list is sorted by
    // permuting (scale, index) keys (the first region is free once the levels are done)
    if (fits)
        for (int i = tid; i < nD; i += kRT) a.D[i] = D[i];
    ScaleKey* K = fits ? reinterpret_cast<ScaleKey*>(sm) : reinterpret_cast<ScaleKey*>(a.M);
    for (int i = tid; i < nD; i += kRT) K[i] = ScaleKey{D[nD - 1 - i].scale, i};
    __syncthreads();
    // n <= 16: insertion sort of a sorted list. The block-wide sort keeps its segment lists in the
    // bit-matrix words (free after the level loop) and its partitions' stop lists in the scan and
    // survivor scratch (also free).
    constexpr int kSortSegs = (kBitMax * kBitWords) / 3;
    if (nD > 16 && nD / 17 <= kSortSegs) {
        introsort_scale_desc_block(K, nD, reinterpret_cast<int*>(s_a1), reinterpret_cast<int*>(s_a2), kSortSegs, first_dec, surv);
    } else {
        if (nD > 16 && tid == 0) introsort_scale_desc(K, nD);
        __syncthreads();
    }
    for (int i = tid; i < nD; i += kRT) {
        R[i] = D[nD - 1 - K[i].idx];
        if (a.fa_scratch) a.fa_scratch[a.face_cap + i] = a.fa_scratch[nD - 1 - K[i].idx];
    }
    __syncthreads();

    // post-processing: the two merges by the whole block where their scratch fits in the bit-matrix
    // words (free after the level loop and the sort), else in warp 0
    __shared__ int s_nM;
    if (tid == 0) {
        *a.n_raw = nD;
        if (a.n_m_out) *a.n_m_out = 0;
    }
    int nF = 0;
    const Det* fin = R;
    int* fa = a.fa_scratch;
    const int cap = a.face_cap;
    int* clus = fa ? fa + 2 * cap : nullptr;     // cluster of every sorted box
    int* keepmap = fa ? fa + 3 * cap : nullptr;  // first-merge cluster of every kept box
    int* fsrc = fa ? fa + 4 * cap : nullptr;     // kept box of every final box
    uint32_t* ws_a = reinterpret_cast<uint32_t*>(s_a1);
    uint32_t* ws_b = reinterpret_cast<uint32_t*>(s_a2);
    if (nD > 0 && C.merger_detect) {
        int nM;
        if (nD <= kGroupMax) {
            // F is scratch here (the first box of every cluster's merged box) until the second merge
            nM = first_merge_groups(R, nD, checked, M, F, clus, reinterpret_cast<int*>(ws_a), reinterpret_cast<int*>(ws_b));
        } else {
            if (warp == 0) {
                const int k = merger_warp<false>(R, nD, checked, M, clus);
                if (lane == 0) s_nM = k;
            }
            __syncthreads();
            nM = s_nM;
        }
        if (keepmap)
            for (int k = tid; k < nM; k += kRT) keepmap[k] = k;
        __syncthreads();
        if (C.min_num_detect > 1) {
            // stable erase of clusters with fewer than min_num_detect merges
            if (warp == 0) {
                int w = 0;
                for (int base = 0; base < nM; base += 32) {
                    const int kk = base + lane;
                    const bool keep = kk < nM && M[kk].num_detect >= C.min_num_detect;
                    const Det v = kk < nM ? M[kk] : M[0];
                    const unsigned m = __ballot_sync(0xffffffffu, keep);
                    const int pos = w + __popc(m & ((1u << lane) - 1u));
                    __syncwarp();
                    if (keep) {
                        M[pos] = v;
                        if (keepmap) keepmap[pos] = kk;
                    }
                    __syncwarp();
                    w += __popc(m);
                }
                if (lane == 0) s_nM = w;
            }
            __syncthreads();
            nM = s_nM;
        }
        if (a.m_out) {
            for (int k = tid; k < nM; k += kRT) a.m_out[k] = M[k];
            if (tid == 0) *a.n_m_out = nM;
        }
        if (nM > 0) {
            if (nM <= kBitMax) {
                nF = second_merge_bits(M, nM, F, fsrc, ws_a, ws_b);
            } else {
                __syncthreads();
                if (warp == 0) {
                    const int k = merger_warp<true>(M, nM, checked, F, nullptr, fsrc);
                    if (lane == 0) s_nM = k;
                }
                __syncthreads();
                nF = s_nM;
            }
            fin = F;
        }
    } else if (nD > 0) {
        if (fa)
            for (int k = tid; k < nD; k += kRT) {
                clus[k] = k;
                keepmap[k] = k;
                fsrc[k] = k;
            }
        nF = nD;
        fin = R;
    }
    __syncthreads();
    for (int i = tid; i < nF && i < a.face_cap; i += kRT) {
        const Det d = fin[i];
        FaceOut f;
        if (C.rescale_output) {
            f.x = (int)((float)d.x * C.rescale);
            f.y = (int)((float)d.y * C.rescale);
            f.w = (int)((float)d.w * C.rescale);
            f.h = (int)((float)d.h * C.rescale);
        } else {
            f.x = d.x;
            f.y = d.y;
            f.w = d.w;
            f.h = d.h;
        }
        f.score = d.score;
        f.scale = d.scale;
        f.knn = d.knn;
        f.num_detect = d.num_detect;
        f.pad = 0;
        f.gender = f.smile = f.glasses = -1;
        a.faces[i] = f;
    }
    if (tid == 0) *a.n_faces = nF;
    if (a.fa_scratch) {
        // CompactCNNLibAPI_v2.cpp:296-319: each attribute is the element at size/2 of the merged box's facial
        // data sorted in descending order: a value v with #(> v) <= k < #(>= v). A warp a (face, attribute), a lane
        // a raw box, on the clusters and values gathered into shared memory (global where they don't fit).
        constexpr int kStage = kBitMax * kBitWords / 4;
        const int* rcand = a.fa_scratch + cap;
        int* st_cl = reinterpret_cast<int*>(s_a1);
        const bool staged = nD <= kStage;
        __syncthreads();  // the scratch's last users are done, and the faces are written
        auto cluster_of = [&](int r) { return rcand[r] >= 0 ? clus[r] : -1; };
        auto value_of = [&](int r, int q) {
            const int4 at = a.attr[rcand[r]];
            return q == 0 ? at.y : (q == 1 ? at.z : at.w);
        };
        for (int r = tid; r < nD && staged; r += kRT) {
            const int c = cluster_of(r);
            st_cl[4 * r] = c;
            for (int q = 0; q < 3; ++q) st_cl[4 * r + 1 + q] = c >= 0 ? value_of(r, q) : 0;
        }
        __syncthreads();
        auto cl = [&](int r) { return staged ? st_cl[4 * r] : cluster_of(r); };
        auto val = [&](int r, int q) { return staged ? st_cl[4 * r + 1 + q] : value_of(r, q); };
        for (int it = warp; it < 3 * imin(nF, cap); it += kRT / 32) {
            const int i = it / 3, q = it - 3 * i;
            const int c = keepmap[fsrc[i]];
            int size = 0;
            for (int r0 = 0; r0 < nD; r0 += 32) size += __popc(__ballot_sync(0xffffffffu, r0 + lane < nD && cl(r0 + lane) == c));
            const int k = size / 2;
            int out = -1;
            for (int r0 = 0; r0 < nD && size > 0; r0 += 32) {
                const int r = r0 + lane;
                const bool mine = r < nD && cl(r) == c;
                if (!__any_sync(0xffffffffu, mine)) continue;
                const int v = mine ? val(r, q) : 0;
                int gt = 0, ge = 0;
                for (int u = 0; u < nD; ++u) {
                    if (cl(u) != c) continue;
                    const int w = val(u, q);
                    gt += w > v;
                    ge += w >= v;
                }
                const unsigned ok = __ballot_sync(0xffffffffu, mine && gt <= k && k < ge);
                if (ok) {
                    out = __shfl_sync(0xffffffffu, v, __ffs(ok) - 1);
                    break;
                }
            }
            if (lane == 0) {
                FaceOut& f = a.faces[i];
                if (q == 0) f.gender = out;
                else if (q == 1) f.smile = out;
                else f.glasses = out;
            }
        }
    }
    if (a.host_faces) {
        // the result straight into the caller's page-locked memory, a warp's stores side by side (two copies
        // after the kernel took 5 us of a frame's latency)
        __syncthreads();
        constexpr int kWords = sizeof(FaceOut) / sizeof(int);
        const int words = imin(imin(nF, a.face_cap), a.host_cap) * kWords;
        for (int i = tid; i < words; i += kRT) reinterpret_cast<int*>(a.host_faces)[i] = reinterpret_cast<const int*>(a.faces)[i];
        if (tid == 0) *a.host_n_faces = nF;
    }
}

// Detect with the caller's detections in front (cnn_detector_v3.cpp:2753-2806), one warp: the
// priors pass the stable min_num_detect filter (the new clusters arrive filtered), then the
// whole list goes through Merger(0.2, del) and the optional rescale of a shrunken input frame.
__global__ void __launch_bounds__(32, 1) prior_merge_kernel(const Det* prior, int n_prior, const Det* clusters, const int* n_clusters,
                                                            const CascadeConfig C, Det* list, uint8_t* checked, Det* out, int* n_out) {
    const int lane = threadIdx.x;
    const int nc = *n_clusters;
    int n = 0;
    for (int base = 0; base < n_prior; base += 32) {  // stable erase of priors below min_num_detect
        const int k = base + lane;
        const bool keep = k < n_prior && (C.min_num_detect <= 1 || prior[k].num_detect >= C.min_num_detect);
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) list[n + __popc(m & ((1u << lane) - 1u))] = prior[k];
        n += __popc(m);
    }
    for (int k = lane; k < nc; k += 32) list[n + k] = clusters[k];
    n += nc;
    __syncwarp();
    const int nf = n > 0 ? merger_warp<true>(list, n, checked, list + n) : 0;
    for (int i = lane; i < nf; i += 32) {
        Det d = list[n + i];
        if (C.rescale_output) {
            d.x = (int)((float)d.x * C.rescale);
            d.y = (int)((float)d.y * C.rescale);
            d.w = (int)((float)d.w * C.rescale);
            d.h = (int)((float)d.h * C.rescale);
        }
        out[i] = d;
    }
    if (lane == 0) *n_out = nf;
}

// CNNDetector::NMS: Merger(detections, rect, 0.5) of the caller's boxes, one warp
__global__ void __launch_bounds__(32, 1) nms_kernel(const Det* in, int n, uint8_t* checked, Det* out, int* n_out) {
    const int nf = merger_warp<false>(in, n, checked, out);
    if (threadIdx.x == 0) *n_out = nf;
}

cudaError_t launch_prior_merge(const Det* prior, int n_prior, const Det* clusters, const int* n_clusters, const CascadeConfig& cfg, Det* scratch,
                               uint8_t* checked, Det* out, int* n_out, cudaStream_t st) {
    prior_merge_kernel<<<1, 32, 0, st>>>(prior, n_prior, clusters, n_clusters, cfg, scratch, checked, out, n_out);
    return cudaGetLastError();
}

cudaError_t launch_nms(const Det* in, int n, uint8_t* checked, Det* out, int* n_out, cudaStream_t st) {
    nms_kernel<<<1, 32, 0, st>>>(in, n, checked, out, n_out);
    return cudaGetLastError();
}

__global__ void __launch_bounds__(kRT, 1) replay_kernel(const ReplayArgs a) {
    chain_wait();
    replay_body(a);
}

// the frames of a batch: block f replays args[f]
__global__ void __launch_bounds__(kRT, 1) replay_batch_kernel(const ReplayArgs* __restrict__ args) {
    __shared__ ReplayArgs s_args;
    if (threadIdx.x == 0) s_args = args[blockIdx.x];
    __syncthreads();
    replay_body(s_args);
}

// The block-wide sort of n (scale, index) keys (device memory) and its permutation, for tests.
__global__ void __launch_bounds__(kRT, 1) sort_check_kernel(ScaleKey* K, int n, int* scratch, int* perm) {
    constexpr int kSegs = (kBitMax * kBitWords) / 3;
    __shared__ int seg_a[3 * kSegs], seg_b[3 * kSegs];
    if (n > 16 && n / 17 <= kSegs) {
        introsort_scale_desc_block(K, n, seg_a, seg_b, kSegs, scratch, scratch + n);
    } else {
        if (threadIdx.x == 0) {
            if (n > 16) introsort_scale_desc(K, n);
            else insertion_sort(K, 0, n);
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) perm[i] = K[i].idx;
}

cudaError_t sort_permutation_device(const float* scales, int n, int* perm) {
    std::vector<ScaleKey> k(n);
    for (int i = 0; i < n; ++i) k[i] = ScaleKey{scales[i], i};
    ScaleKey* d_k = nullptr;
    int *d_leaves = nullptr, *d_perm = nullptr;
    cudaError_t e = cudaMalloc(&d_k, sizeof(ScaleKey) * (n + 1));
    if (e == cudaSuccess) e = cudaMalloc(&d_leaves, sizeof(int) * (2 * n + 2));
    if (e == cudaSuccess) e = cudaMalloc(&d_perm, sizeof(int) * (n + 1));
    if (e == cudaSuccess && n > 0) e = cudaMemcpy(d_k, k.data(), sizeof(ScaleKey) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        sort_check_kernel<<<1, kRT>>>(d_k, n, d_leaves, d_perm);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && n > 0) e = cudaMemcpy(perm, d_perm, sizeof(int) * n, cudaMemcpyDeviceToHost);
    cudaFree(d_k);
    cudaFree(d_leaves);
    cudaFree(d_perm);
    return e;
}

cudaError_t replay_setup() {
    cudaError_t e = cudaFuncSetAttribute(replay_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kReplaySmemBytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(replay_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kReplaySmemBytes);
    return e;
}

cudaError_t launch_replay(const ReplayArgs& a, cudaStream_t st) {
    return launch_chained(replay_kernel, 1, kRT, kReplaySmemBytes, st, a);
}

cudaError_t launch_replay_batch(const ReplayArgs* d_args, int n_frames, cudaStream_t st) {
    replay_batch_kernel<<<n_frames, kRT, kReplaySmemBytes, st>>>(d_args);
    return cudaGetLastError();
}

}  // namespace ccnn
