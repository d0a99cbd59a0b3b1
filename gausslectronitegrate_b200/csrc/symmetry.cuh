// O_h orbit helpers on a rotationally symmetric grid (-e .. e on every axis),
// shared by the enumeration (enumerate.cu) and the sparse -> dense kernels
// (dense.cu).  Reference: minimum_octahedral_orbit_{eri,erida}_tensor_index
// (src/eri_integrals.c:240-291, src/erida_integrals.c:209-234) with the
// bias-shift loops of the enumerators and fill routines.
#pragma once
#include <limits.h>

#include "gli_internal.cuh"

namespace gli {

struct SymGrid {
    int e;   // extent: coordinates -e .. e
    int L;   // 2e + 1
    i64 N;   // L^3
    const int* omin = nullptr;  // enumeration: smallest linear index among each point's 48 O_h images
    const uint4* images = nullptr;  // ERI enumeration: the 48 images themselves, 16 bits each (N <= 65535), 6 uint4 a point
};

__device__ inline i64 lin3(const SymGrid& G, const int q[3]) {
    return ((i64)(q[0] + G.e) * G.L + (q[1] + G.e)) * G.L + (q[2] + G.e);
}

__device__ inline int absi(int v) { return v < 0 ? -v : v; }

// ERIDA: is (p0, p1) the smallest index of its orbit?  idx = lin(p0) N + lin(p1)
__device__ inline bool canonical_pair(const SymGrid& G, const int p[2][3], const int bias[3], i64 idx) {
    for (int bx = 0; bx <= absi(bias[0]); ++bx)
        for (int by = 0; by <= absi(bias[1]); ++by)
            for (int bz = 0; bz <= absi(bias[2]); ++bz) {
                const int sft[3] = {bx * bias[0], by * bias[1], bz * bias[2]};
                int q0[3], q1[3];
                for (int a = 0; a < 3; ++a) {
                    q0[a] = p[0][a] - sft[a];
                    q1[a] = p[1][a] - sft[a];
                }
                for (int g = 0; g < 48; ++g) {
                    int r0[3], r1[3];
                    oh_apply(g, q0, r0);
                    oh_apply(g, q1, r1);
                    i64 a = lin3(G, r0), b = lin3(G, r1);
                    if (a > b) { i64 t = a; a = b; b = t; }
                    if (a * G.N + b < idx) return false;
                }
            }
    return true;
}

// ERI: is (l0, l1, l2, l3) (linear point indices, l0 the leading one) the
// smallest index of its orbit?  An image's index leads with its smallest
// point.  omin rules a shifted copy out at once when no point of it has an image
// at l0 or below, and decides at once when one lies below; only copies with an
// image at l0 look at their images, read eight per load from the table.  The
// index pairs compare in 32 bits (N^2 < 2^32).
__device__ inline bool canonical_copy(const SymGrid& G, const int l[4], int sft) {  // (the copy moved by -sft)
    const uint32_t N = (uint32_t)G.N;
    const uint32_t ij = l[0] * N + l[1], kl = l[2] * N + l[3];
    int q[4], least = INT_MAX;
    for (int k = 0; k < 4; ++k) {
        q[k] = l[k] - sft;
        least = min(least, G.omin[q[k]]);
    }
    if (least != l[0]) return least > l[0];
    const uint32_t both = (uint32_t)l[0] * 0x10001u;
    for (int c = 0; c < 6; ++c) {
        uint4 im[4];
        for (int k = 0; k < 4; ++k) im[k] = __ldg(G.images + (i64)q[k] * 6 + c);
#pragma unroll
        for (int h = 0; h < 4; ++h) {  // two images of each point in a word
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) w[k] = h == 0 ? im[k].x : h == 1 ? im[k].y : h == 2 ? im[k].z : im[k].w;
            const uint32_t off = __vimin3_u16x2(__vimin3_u16x2(w[0], w[1], w[2]), w[3], w[3]) ^ both;
            if ((off & 0xffffu) && off >> 16) continue;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (u ? off >> 16 : off & 0xffffu) continue;
                uint32_t r[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) r[k] = u ? w[k] >> 16 : w[k] & 0xffffu;
                const uint32_t ab = min(r[0], r[1]) * N + max(r[0], r[1]);
                const uint32_t cd = min(r[2], r[3]) * N + max(r[2], r[3]);
                const uint32_t first = min(ab, cd), second = max(ab, cd);
                if (first < ij || (first == ij && second < kl)) return false;
            }
        }
    }
    return true;
}
// the shift of copy m (bit a: moved by the bias of axis a) as a linear index
__device__ __forceinline__ int copy_shift(const SymGrid& G, const int bias[3], int m) {
    return ((m & 1 ? bias[0] : 0) * G.L + (m & 2 ? bias[1] : 0)) * G.L + (m & 4 ? bias[2] : 0);
}
__device__ __forceinline__ bool copy_exists(const int bias[3], int m) {
    return !((m & 1 && !bias[0]) || (m & 2 && !bias[1]) || (m & 4 && !bias[2]));
}
__device__ inline bool canonical_quad(const SymGrid& G, const int l[4], const int bias[3]) {
    for (int m = 0; m < 8; ++m)
        if (copy_exists(bias, m) && !canonical_copy(G, l, copy_shift(G, bias, m))) return false;
    return true;
}

__device__ inline void point_of(const SymGrid& G, i64 lin, int p[3]) {
    p[2] = (int)(lin % G.L) - G.e;
    lin /= G.L;
    p[1] = (int)(lin % G.L) - G.e;
    p[0] = (int)(lin / G.L) - G.e;
}


// smallest index of the orbit of a pair / quadruple already translated so that
// each axis' doubled box centre is in {-1, 0, 1} (bias = that centre)
__device__ inline i64 orbit_min_pair(const SymGrid& G, const int p[2][3], const int bias[3]) {
    i64 best = INT64_MAX;
    for (int bx = 0; bx <= absi(bias[0]); ++bx)
        for (int by = 0; by <= absi(bias[1]); ++by)
            for (int bz = 0; bz <= absi(bias[2]); ++bz) {
                const int sft[3] = {bx * bias[0], by * bias[1], bz * bias[2]};
                int q0[3], q1[3];
                for (int a = 0; a < 3; ++a) {
                    q0[a] = p[0][a] - sft[a];
                    q1[a] = p[1][a] - sft[a];
                }
                for (int g = 0; g < 48; ++g) {
                    int r0[3], r1[3];
                    oh_apply(g, q0, r0);
                    oh_apply(g, q1, r1);
                    i64 a = lin3(G, r0), b = lin3(G, r1);
                    const i64 v = a <= b ? a * G.N + b : b * G.N + a;
                    if (v < best) best = v;
                }
            }
    return best;
}

__device__ inline i64 orbit_min_quad(const SymGrid& G, const int p[4][3], const int bias[3]) {
    const i64 N2 = G.N * G.N;
    i64 best = INT64_MAX;
    for (int bx = 0; bx <= absi(bias[0]); ++bx)
        for (int by = 0; by <= absi(bias[1]); ++by)
            for (int bz = 0; bz <= absi(bias[2]); ++bz) {
                const int sft[3] = {bx * bias[0], by * bias[1], bz * bias[2]};
                int q[4][3];
                for (int k = 0; k < 4; ++k)
                    for (int a = 0; a < 3; ++a) q[k][a] = p[k][a] - sft[a];
                for (int g = 0; g < 48; ++g) {
                    i64 l4[4];
                    for (int k = 0; k < 4; ++k) {
                        int r[3];
                        oh_apply(g, q[k], r);
                        l4[k] = lin3(G, r);
                    }
                    i64 ab = l4[0] <= l4[1] ? l4[0] * G.N + l4[1] : l4[1] * G.N + l4[0];
                    i64 cd = l4[2] <= l4[3] ? l4[2] * G.N + l4[3] : l4[3] * G.N + l4[2];
                    if (ab > cd) { i64 t = ab; ab = cd; cd = t; }
                    const i64 v = ab * N2 + cd;
                    if (v < best) best = v;
                }
            }
    return best;
}

// move the bounding-box centre of np points to the origin (reference
// src/eri_integrals.c:869-903: trans = (min+max)/2 truncating, bias = remainder)
template <int NP>
__device__ inline void centre_points(int p[NP][3], int bias[3]) {
    for (int a = 0; a < 3; ++a) {
        int lo = p[0][a], hi = p[0][a];
        for (int k = 1; k < NP; ++k) {
            lo = min(lo, p[k][a]);
            hi = max(hi, p[k][a]);
        }
        const int c = lo + hi;
        const int trans = c / 2;
        bias[a] = c - 2 * trans;
        for (int k = 0; k < NP; ++k) p[k][a] -= trans;
    }
}

}  // namespace gli
