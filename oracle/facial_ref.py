"""CPU restatement of facial analysis in float32 numpy (test infrastructure: a checker, never a product path).

The landmark network (cnn4landmarks_cntk.bin) follows SIMD::ConvNeuralNetwork of the reference
(src/CNNObjectDetector/cnn_simd_cntk.cpp: the reader :42-404, Run :640-963) over the CNNPP operations of
cnnpp_cplusplus.cpp (conv_4x4 :92, conv_3x3 :36, conv_11x10 :352, lrelu_bn_max :593, lrelu_bn :623,
mulCN_add_tanhW :646, mulC / mulC1_add :952-984, tanhW :673, add / add2 :916-950), each operation one float32
operation in the reference's order. The attributes of a face are those of CompactCNNLibAPI_v2.cpp:296-319 over the
boxes that Merger (cnn_detector_v3.cpp:2814-2936) joins.
"""
import struct

import numpy as np

F = np.float32


def load(path):
    with open(path, "rb") as f:
        b = f.read()
    o = [0]

    def rd(fmt):
        v = struct.unpack_from("<" + fmt, b, o[0])
        o[0] += struct.calcsize("<" + fmt)
        return v if len(v) > 1 else v[0]

    def floats(*shape):
        n = int(np.prod(shape))
        v = np.frombuffer(b, "<f4", n, o[0]).astype(F).reshape(shape)
        o[0] += 4 * n
        return v

    net = {"version": rd("f"), "max_pool": rd("B"), "min": rd("ii")}
    if rd("i") != 3:
        raise ValueError("three layers expected")
    maps = [rd("i") for _ in range(3)]
    net["k"] = []
    for m in maps:
        kw, kh = rd("ii")
        net["k"].append(floats(m, kh, kw))
    net["af"] = F(rd("f"))
    net["act"] = [floats(m, 5) for m in maps]  # bias, w1, w2, (unused), bn bias
    full, hl, conn, hs = rd("B"), rd("i"), rd("i"), rd("i")
    net["full"], net["hl"] = full, hl
    net["hw"] = floats(hl, maps[2] if full else conn)
    net["hb"], net["htw"], net["hbn"] = floats(hl), floats(hl // hs), floats(hs, 2)
    nout = rd("i")
    net["ow"], net["ob"], net["otw"] = floats(nout, hl), floats(nout), F(rd("f"))
    if o[0] != len(b):
        raise ValueError("unexpected model size")
    return net


def tanh_r(c):
    sgn = np.where(c < 0, F(-1), F(1)).astype(F)
    return sgn * (F(1) - F(1) / (((F(1) + np.abs(c)) + c * c) + (((F(1.41645) * c) * c) * c) * c))


def _conv(maps, k, start):
    """maps (n, h, w) with kernels k (n, kh, kw): taps in row-major order; start: from 0 (conv_11x10) or the first tap."""
    n, kh, kw = k.shape
    oh, ow = maps.shape[1] - kh + 1, maps.shape[2] - kw + 1
    acc = np.zeros((n, oh, ow), F) if start else None
    for t in range(kh * kw):
        r, c = divmod(t, kw)
        v = maps[:, r:r + oh, c:c + ow] * k[:, r, c][:, None, None]
        acc = v if acc is None else acc + v
    return acc


def _act(x, a):
    a = a[:, :, None, None]
    c = x + a[:, 0]
    return (a[:, 1] * c + a[:, 2] * np.maximum(c, F(0))) + a[:, 4]


def _pool(x):
    h, w = x.shape[1] // 2 * 2, x.shape[2] // 2 * 2
    return np.maximum(np.maximum(x[:, 0:h:2, 0:w:2], x[:, 0:h:2, 1:w:2]), np.maximum(x[:, 1:h:2, 0:w:2], x[:, 1:h:2, 1:w:2]))


def _sums(p):
    s = p[:-1] + p[1:]
    return np.concatenate([s[:1], s[:-1] + p[2:], s[-1:]])


def forward(net, img):
    """The 13 outputs for a 51 x 49 crop."""
    x = np.asarray(img, F)
    n = [k.shape[0] for k in net["k"]]
    p1 = _pool(_act(_conv(np.broadcast_to(x, (n[0],) + x.shape), net["k"][0], False), net["act"][0]))
    p2 = _pool(_act(_conv(np.repeat(_sums(p1), 2, 0), net["k"][1], False), net["act"][1]))
    a3 = _act(_conv(np.repeat(_sums(p2), 2, 0), net["k"][2], True), net["act"][2])[:, 0, 0]
    s = net["hb"].copy()
    for j in range(n[2]):
        s = s + a3[j] * net["hw"][:, j]
    v = F(0.5) * tanh_r(s * net["htw"][0]) + F(0.5)
    hid = net["hbn"][:, 0] * v + net["hbn"][:, 1]
    acc = hid[0] * net["ow"][:, 0]
    for t in range(1, net["hl"]):
        acc = hid[t] * net["ow"][:, t] + acc
    c = tanh_r((acc + net["ob"]) * net["otw"])
    return F(0.5) * c + F(0.5) if net["af"] == 0 else net["af"] * c


def analyse(net, crop, cols, rows):
    """(dropped, gender, smile, glasses) of a window of cols x rows gray pixels (cnn_detector_v3.cpp:1731-1764)."""
    v = forward(net, crop)
    zero = sum(int(v[2 * t] * F(cols)) < cols >> 1 and int(v[2 * t + 1] * F(rows)) < rows >> 1 for t in range(5))
    return (zero == 5,) + tuple(int(v[10 + q] + F(0.5)) for q in range(3))


def merger(boxes, thr, delete):
    """Merger over (x, y, x2, y2, score) boxes: the output boxes and the input boxes of each."""
    thr = F(thr)
    out, members, checked = [], [], [False] * len(boxes)
    for i, first in enumerate(boxes):
        if checked[i]:
            continue
        mx, mn, score, own, drop = list(first[:4]), list(first[:4]), first[4], [i], False
        for j in range(i + 1, len(boxes)):
            e = boxes[j]
            if checked[j] or mx[0] >= e[2] or mx[2] <= e[0] or mx[1] >= e[3] or mx[3] <= e[1]:
                continue
            s1, s2 = F((mx[2] - mx[0]) * (mx[3] - mx[1])), F((e[2] - e[0]) * (e[3] - e[1]))
            X, Y = sorted((mx[0], mx[2], e[0], e[2])), sorted((mx[1], mx[3], e[1], e[3]))
            su, si = F((X[3] - X[0]) * (Y[3] - Y[0])), F((X[2] - X[1]) * (Y[2] - Y[1]))
            r1, r2, r3 = si / s1, si / s2, si / su
            ratio, tc = min(r1, r2), min(X[3] - X[0], X[2] - X[1]) >> 1
            if r3 > F(0.75) * thr and max(r1, r2) > F(0.7) and abs(X[0] + ((X[3] - X[0]) >> 1) - X[1] - ((X[2] - X[1]) >> 1)) < tc and \
                    abs(Y[0] + ((Y[3] - Y[0]) >> 1) - Y[1] - ((Y[2] - Y[1]) >> 1)) < tc:
                ratio = F(1)
            if not ratio > thr:
                continue
            if delete:
                if s1 > s2:
                    checked[j] = True
                    continue
                drop = True
                break
            mx = [min(mx[0], X[0]), min(mx[1], Y[0]), max(mx[2], X[3]), max(mx[3], Y[3])]
            mn = [max(mn[0], X[1]), max(mn[1], Y[1]), min(mn[2], X[2]), min(mn[3], Y[2])]
            score = max(score, e[4])
            checked[j] = True
            own.append(j)
        if not drop:
            out.append(tuple((a + b) >> 1 for a, b in zip(mn, mx)) + (score,))
            members.append(own)
    return out, members


def faces(boxes, attributes):
    """boxes: (x, y, x2, y2, score) sorted by scale; attributes: (gender, smile, glasses) of each. The faces of the
    two merges, each attribute the element at size / 2 of its boxes' values in descending order."""
    clusters, members = merger(boxes, 0.5, False)
    final, kept = merger(clusters, 0.2, True)
    out = []
    for (x, y, x2, y2, score), own in zip(final, kept):
        values = [sorted((attributes[m][q] for m in members[own[0]]), reverse=True) for q in range(3)]
        out.append((x, y, x2 - x, y2 - y, score) + tuple(v[len(v) // 2] for v in values))
    return out
