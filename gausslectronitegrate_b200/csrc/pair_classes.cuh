// Contractions of a complete ERI tensor by pair classes.
//
// V[i j k l] depends on the point pair (i, j) only through its class: per axis
// the unordered pair of coordinates.  On a box of n0 x n1 x n2 points
// (a product of coordinate lists) the N^2 ordered pairs fall into F0 F1 F2
// classes, Fa = na (na + 1) / 2 (6^3 points: 9,261 classes of 46,656 ordered
// pairs; 7^3: 21,952 of 117,649), and V[c][k l] = V[c'][k l] as matrices in
// (k, l) for every pair of class c.  So every contraction over (k, l) is made
// once per class:
//   projection   Y[c] = B^T V[c] B                     (an M x M block per class)
//   apply        C[(i j)] = V[c] X_j for the pairs (i, j) of class c
// and V[c] itself holds one value per class c' of (k, l).
//
// The values come from the key table of the complete list (dense.cu): slot
// tetra_index of the sorted triple of axis keys.  An axis key joins the fields
// (|d|, s) and (|d'|, s') of the two pairs' coordinates, d = difference and
// s = sum: the unordered {|d|, |d'|} and |s - s'|.  s - s' has the parity of
// d + d', so |s - s'| / 2 (rounded down) tells the keys apart, and a grid of L
// points per axis has L (L + 1) / 2 L of them.  (With |s - s'| itself half of
// the keys never occur: at 7^3 the table takes 64 MB, and the values that a
// warp reads lie every other slot; now 10 MB, neighbours in one sector.)
#pragma once

#include "dmma.cuh"
#include "gli_internal.cuh"

namespace gli {

// axis keys of the key table
__host__ __device__ __forceinline__ int pair_axis_keys(int L) { return L * (L + 1) / 2 * L; }
__host__ __device__ __forceinline__ int pair_axis_key(int d01, int d23, int cc, int L) {
    int a = d01 < 0 ? -d01 : d01;
    int b = d23 < 0 ? -d23 : d23;
    if (a > b) { const int t = a; a = b; b = t; }
    const int c = cc < 0 ? -cc : cc;
    return (b * (b + 1) / 2 + a) * L + (c >> 1);
}

__host__ __device__ inline i64 tetra_index(i64 k1, i64 k2, i64 k3) {  // k1 <= k2 <= k3
    return k3 * (k3 + 1) * (k3 + 2) / 6 + k2 * (k2 + 1) / 2 + k1;
}
// the same in 32-bit arithmetic, for key tables of at most 2^29 slots (the
// only ones built): then k3 (k3 + 1) (k3 + 2) <= 6 * 2^29 < 2^32
__device__ __forceinline__ uint32_t tetra_index32(uint32_t k1, uint32_t k2, uint32_t k3) {
    return k3 * (k3 + 1) * (k3 + 2) / 6u + k2 * (k2 + 1) / 2u + k1;
}

constexpr int PAIR_MAX_AXIS = 16, PAIR_MAX_WARPS = 16;
constexpr int PAIR_MAX_TILES = 2;                                      // 16-row tiles per warp
constexpr int PAIR_MAX_POINTS = 16 * PAIR_MAX_WARPS * PAIR_MAX_TILES;  // 512

// A box of points, x-major: coordinate lists (ascending) per axis
struct PairBox {
    int L;        // points per axis of the class list's grid (key range)
    int n[3], F[3];
    int N, nyz;   // points; points of one x plane
    int F2, PS;   // F1 F2; plane stride: F2 values and a zero
    int S;        // k steps of 4 per x plane
    int classes;  // F0 F1 F2
    short c[3][PAIR_MAX_AXIS];
};

inline PairBox make_pair_box(int L, const std::vector<int> coords[3]) {
    PairBox b = {};
    b.L = L;
    for (int a = 0; a < 3; ++a) {
        b.n[a] = (int)coords[a].size();
        b.F[a] = b.n[a] * (b.n[a] + 1) / 2;
        for (int k = 0; k < b.n[a]; ++k) b.c[a][k] = (short)coords[a][k];
    }
    b.nyz = b.n[1] * b.n[2];
    b.N = b.n[0] * b.nyz;
    b.F2 = b.F[1] * b.F[2];
    b.PS = b.F2 + 1;
    b.S = (b.nyz + 3) / 4;
    b.classes = b.F[0] * b.F2;
    return b;
}

// field f = hi (hi + 1) / 2 + lo of an axis -> coordinate positions lo <= hi
__device__ __forceinline__ void pair_field(int f, int& lo, int& hi) {
    int h = 0;
    while ((h + 1) * (h + 2) / 2 <= f) ++h;
    hi = h;
    lo = f - h * (h + 1) / 2;
}

// class of the ordered pair of box points (i, j)
__device__ __forceinline__ int pair_class(const PairBox& b, int i, int j) {
    int f[3];
#pragma unroll
    for (int a = 2; a >= 0; --a) {
        const int n = b.n[a], x = a ? i % n : i, y = a ? j % n : j;
        i /= n;
        j /= n;
        const int lo = min(x, y), hi = max(x, y);
        f[a] = hi * (hi + 1) / 2 + lo;
    }
    return (f[0] * b.F[1] + f[1]) * b.F[2] + f[2];
}

// 8-byte asynchronous copy without the compiler's ordering of other memory
// accesses (the kernel's barriers and waits order it): between two k steps it
// must not hold back the next step's loads
__device__ __forceinline__ void pair_cp8(double* dst, const double* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src));
}

// Shared memory of k_pair_contract (the launch and the kernel agree on it)
struct PairSmem {
    int ldb;      // doubles per row of B: 4 or 12 mod 16, so that fragment reads have no bank conflicts
    int planes;   // doubles: two buffers of n0 planes (the epilogue's tiles reuse them)
    int brows;    // rows of B
    int map_ld;   // uint16 per row of the (y z) x (y z) maps
    int sum, part, rows;  // (SYM epilogue) Y, the warps' parts of it and the 8-row strips of Y they hold at a time
    size_t bytes;
    __host__ __device__ PairSmem(const PairBox& b, int warps, int nt) {
        ldb = 8 * nt + 4;
        planes = 2 * b.n[0] * b.PS;
        sum = b.PS;  // (past the next class's first plane)
        part = sum + 8 * nt * (8 * nt + 1);
        const int strip = warps * 64 * nt;
        if (planes < part + strip) planes = part + strip;
        rows = (planes - part) / strip < nt ? (planes - part) / strip : nt;
        brows = b.N + 4;
        map_ld = 4 * b.S;
        bytes = 8 * ((size_t)planes + (size_t)brows * ldb + 2 * 8 * (size_t)nt) + 6 * ((size_t)b.F2 + b.F[0] + b.F[1] + b.F[2]) +
                2 * ((size_t)2 * b.nyz + 1) * map_ld;
    }
};

// One class c per turn of a persistent block: A = V[c] B over the box's points,
// V[c] the N x N matrix of the class and B of at most 8 NT columns.
//
//   SYM   B is the basis (N x cols); V[c] is taken as U + U^T, U its upper
//         triangle with half the diagonal, so only U B is formed, and
//         Y = B^T (U B) gives B^T V B = Y + Y^T; out[c] holds its lower
//         triangle (r >= s, packed).
//   else  (apply) B holds the columns [state rows of j] of the ordered pairs
//         (i, j) of class c, states col0 .. col0 + cols of each:
//         out[(i N + j) N + k][state] = sum_l V[c][k l] x[j N + l][state].
//
// The k loop runs over the x planes of l.  V[c] restricted to l's plane needs
// one plane of values per x coordinate of k (F1 F2 each): they are copied from
// the key table with 8-byte cp.async into one of two buffers while the previous
// plane is contracted, one value per thread between two k steps (all copies
// ahead of the plane's first MMA left the tensor pipe idle behind them: 5.19
// against 4.88 ms at 343 points and 20 orbitals).  V fragments are read from
// there through a map (yz of k, yz of l) -> value, 16 bits each, the same for
// every plane; rows and columns outside the triangle (or the box) point at the
// plane's zero.  V is the right operand: an accumulator tile holds A^T, eight
// columns by eight rows k, and is as it stands the left operand of Y^T = A^T B
// (the values of one lane have k of equal parity), so the second contraction
// needs no trip of A through shared memory, and every warp takes part in it.
// The next class's keys are made under the last plane, its first plane's copies
// under that contraction.
// A tile's k steps that lie before all its rows in the diagonal plane are zero
// and left out (343 points: 4.43 to 4.26 ms).
// Bound: the FP64 tensor pipe, 50% busy (343 points, 20 orbitals), with the
// shared-memory pipe 59% busy (V fragments, and copies whose 32 values lie in
// about as many lines; contiguous copies in their place measured 4.03 ms).
// Measured on a B200, first two contractions: 216 points and 32 orbitals 0.98
// ms (a contraction per point pair, its slab staged from the key table: 5.25
// ms), 343 points and 20 orbitals 4.26 ms (23.7 ms; A through shared memory 4.88
// ms); the whole projection calls 9.9 to 3.5 ms and 28.0 to 6.4 ms, the apply at
// 5^3 points and 4 states 12.7 to 0.48 ms (0.16 ms of this kernel; 0.21 ms with
// four column tiles multiplied whatever the class's pairs).
//
// A warp owns up to two 16-row tiles (rows 16 (w + W t)) and keeps their
// accumulators over all planes, so each B fragment serves all its tiles.  The
// FP64 MMAs of four warps per scheduler hide each other's issue gaps and the
// map and value loads: two blocks of 8 warps on an SM, or one of 16 where the
// planes and B of one box take more than half of the shared memory.  (Two warps
// per scheduler with three tiles each kept the FP64 tensor pipe 39% busy; loads
// issued a step ahead gained nothing, 4.54 ms.)
template <int W, int NT, int TPW, bool SYM>
__global__ void __launch_bounds__(32 * W, W == 8 ? 2 : 1)
    k_pair_contract(const PairBox box, const double* __restrict__ table, const double* __restrict__ bsrc, int cols,
                    int ld, int col0, double* __restrict__ out) {
    extern __shared__ __align__(16) double sm[];
    constexpr int PAIR_WARPS = W, PAIR_THREADS = 32 * W;
    const PairSmem lay(box, W, NT);
    const int LDB = 8 * NT + 4;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane & 3, c8 = lane >> 2;
    const int N = box.N, nyz = box.nyz, PS = box.PS, F2 = box.F2, map_ld = lay.map_ld;
    double* planes = sm;
    double* B = sm + lay.planes;
    i64* csrc = reinterpret_cast<i64*>(B + lay.brows * LDB);  // (apply) source and destination of each column
    i64* cdst = csrc + 8 * NT;
    uint32_t* yz = reinterpret_cast<uint32_t*>(cdst + 8 * NT);  // (min, max, diagonal) of the y and z keys
    int* kx = reinterpret_cast<int*>(yz + F2);
    int* ky = kx + box.F[0];
    int* kz = ky + box.F[1];
    uint16_t* fields = reinterpret_cast<uint16_t*>(kz + box.F[2]);  // coordinate positions lo | hi << 8 of x, y, z fields
    uint16_t* fyz = fields + box.F[0] + box.F[1] + box.F[2];        // y field | z field << 8 of a plane's values
    uint16_t* map = fyz + F2;                                       // nyz rows: every l
    uint16_t* tmap = map + nyz * map_ld;                          // nyz rows: l >= k only
    uint16_t* zrow = tmap + nyz * map_ld;                         // a row of zeros
    // the maps, the fields, and B where every class has the same
    const int nfields = box.F[0] + box.F[1] + box.F[2];
    for (int g = tid; g < nfields; g += PAIR_THREADS) {
        const int a = g < box.F[0] ? 0 : g < box.F[0] + box.F[1] ? 1 : 2;
        int lo, hi;
        pair_field(g - (a > 0 ? box.F[0] : 0) - (a > 1 ? box.F[1] : 0), lo, hi);
        fields[g] = (uint16_t)(lo | hi << 8);
    }
    for (int e = tid; e < F2; e += PAIR_THREADS) fyz[e] = (uint16_t)(e / box.F[2] | e % box.F[2] << 8);
    for (int e = tid; e < nyz * map_ld; e += PAIR_THREADS) {
        const int k = e / map_ld, l = e - k * map_ld;
        int v = F2;
        if (l < nyz) {
            const int n2 = box.n[2], yk = k / n2, zk = k - yk * n2, yl = l / n2, zl = l - yl * n2;
            const int yh = max(yk, yl), zh = max(zk, zl);
            v = (yh * (yh + 1) / 2 + min(yk, yl)) * box.F[2] + zh * (zh + 1) / 2 + min(zk, zl);
        }
        map[e] = (uint16_t)v;
        tmap[e] = (uint16_t)(l >= k ? v : F2);
    }
    for (int e = tid; e < map_ld; e += PAIR_THREADS) zrow[e] = (uint16_t)F2;
    for (int e = tid; e < lay.brows * 8 * NT; e += PAIR_THREADS) {
        const int r = e / (8 * NT), c = e - r * (8 * NT);
        B[r * LDB + c] = SYM && r < N && c < cols ? bsrc[(i64)r * ld + c] : 0.0;
    }
    // this thread's rows: x plane and the offsets of its rows of the two maps
    const int tiles = (N + 15) / 16, mine = tiles > warp ? (tiles - warp + PAIR_WARPS - 1) / PAIR_WARPS : 0;
    int row_k[TPW][2], row_m[TPW][2];
#pragma unroll
    for (int t = 0; t < TPW; ++t)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = 16 * (warp + PAIR_WARPS * t) + 8 * i + c8;
            row_k[t][i] = r / nyz;
            row_m[t][i] = (r - row_k[t][i] * nyz) * map_ld + q;
        }

    __syncthreads();  // the fields

    // the axis keys of class cls with every field: bit 15 marks the y and z
    // fields of one coordinate
    auto keys = [&](int cls) {
        for (int g = tid; g < nfields; g += PAIR_THREADS) {
            const int a = g < box.F[0] ? 0 : g < box.F[0] + box.F[1] ? 1 : 2;
            const int f = a == 0 ? cls / F2 : a == 1 ? box.F[0] + cls / box.F[2] % box.F[1]
                                                     : box.F[0] + box.F[1] + cls % box.F[2];
            const int p1 = fields[f], p2 = fields[g], h1 = p1 >> 8, l1 = p1 & 255, h2 = p2 >> 8, l2 = p2 & 255;
            const int xl = box.c[a][l1], xh = box.c[a][h1], yl = box.c[a][l2], yh = box.c[a][h2];
            kx[g] = pair_axis_key(xh - xl, yh - yl, xh + xl - yh - yl, box.L) | (a && l2 == h2 ? 1 << 15 : 0);
        }
    };
    auto key_pairs = [&]() {
        for (int e = tid; e < F2; e += PAIR_THREADS) {
            const uint32_t f = fyz[e], y = ky[f & 255], z = kz[f >> 8];
            const uint32_t a = min(y & 0x7fffu, z & 0x7fffu), b = max(y & 0x7fffu, z & 0x7fffu);
            yz[e] = a | b << 15 | (y & z) >> 15 << 31;
        }
    };
    auto zeros = [&]() {
        for (int e = tid; e < 2 * box.n[0]; e += PAIR_THREADS) planes[e * PS + F2] = 0.0;
    };
    // copies the values of l's plane glx into its buffer, one value per
    // thread and call: value ge of the plane for k's x coordinate gk
    int glx = 0, gend = 0, gk = 0, ge = 0;
    uint32_t gx = 0;
    auto gen_wrap = [&]() {
        while (ge >= F2 && gk < gend) {
            ge -= F2;
            ++gk;
        }
        const int h = max(gk, glx);
        if (gk < gend) gx = kx[h * (h + 1) / 2 + min(gk, glx)];
    };
    auto gen_plane = [&](int lx) {
        glx = lx;
        gend = lx >= box.n[0] ? 0 : SYM ? lx + 1 : box.n[0];
        gk = 0;
        ge = tid;
        gen_wrap();
    };
    auto gen_one = [&]() {
        if (gk >= gend) return;
        const uint32_t v = yz[ge], a = v & 0x7fffu, b = v >> 15 & 0x7fffu;
        pair_cp8(planes + ((glx & 1) * box.n[0] + gk) * PS + ge,
                 table + tetra_index32(min(a, gx), max(a, min(b, gx)), max(b, gx)));
        ge += PAIR_THREADS;
        if (ge >= F2) gen_wrap();
    };
    auto gen_first = [&]() {
        gen_plane(0);
        while (gk < gend) gen_one();
        dm_commit();
    };
    if (SYM) {
        keys(blockIdx.x);
        zeros();
        __syncthreads();
        key_pairs();
        __syncthreads();
        gen_first();
    }

    for (int cls = blockIdx.x; cls < box.classes; cls += gridDim.x) {
        int lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
        if (!SYM) {
            const int f[3] = {cls / F2, box.F[0] + cls / box.F[2] % box.F[1], box.F[0] + box.F[1] + cls % box.F[2]};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const int p = fields[f[a]];
                lo[a] = p & 255;
                hi[a] = p >> 8;
            }
            __syncthreads();  // the previous class is done with the tables, the planes and B
            keys(cls);
            zeros();
            __syncthreads();
            key_pairs();
        }
        int axes = 0;  // (apply) axes on which the class's two coordinates differ
        if (!SYM) {
#pragma unroll
            for (int a = 0; a < 3; ++a) axes += lo[a] != hi[a];
        }
        // the ordered pair p of the class: bit per differing axis
        auto pair_points = [&](int p, int& i, int& j) {
            i = j = 0;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                bool flip = false;
                if (lo[a] != hi[a]) {
                    flip = p & 1;
                    p >>= 1;
                }
                i = i * box.n[a] + (flip ? hi[a] : lo[a]);
                j = j * box.n[a] + (flip ? lo[a] : hi[a]);
            }
        };
        const int bcols = SYM ? cols : cols << axes;
        for (int ct = 0; ct < bcols; ct += 8 * NT) {  // (SYM: one turn)
        if (!SYM) {
            if (tid < 8 * NT) {
                const int cc = ct + tid;
                i64 from = -1, to = -1;
                if (cc < bcols) {
                    int i, j;
                    pair_points(cc / cols, i, j);
                    from = (i64)j * N * ld + col0 + cc % cols;
                    to = ((i64)i * N + j) * N * cols + cc % cols;
                }
                csrc[tid] = from;
                cdst[tid] = to;
            }
            __syncthreads();
            for (int e = tid; e < 8 * NT * N; e += PAIR_THREADS) {
                const int r = e / (8 * NT), c = e - r * (8 * NT);
                const i64 from = csrc[c];
                dm_cp8(B + r * LDB + c, from >= 0 ? bsrc + from + (i64)r * ld : bsrc, from >= 0);
            }
        }
        double acc[TPW][2][NT][2];
#pragma unroll
        for (int t = 0; t < TPW; ++t)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < NT; ++j) acc[t][i][j][0] = acc[t][i][j][1] = 0.0;
        if (!SYM) gen_first();
        const int next = cls + gridDim.x;
        const int live = SYM ? NT : min(NT, (bcols - ct + 7) / 8);  // column tiles in use
        for (int lx = 0; lx < box.n[0]; ++lx) {
            double* buf = planes + (lx & 1) * box.n[0] * PS;
            dm_wait<0>();
            if (SYM)  // the diagonal k = l, halved by the thread that copied it
                for (int e = (unsigned)(tid + PAIR_THREADS * F2 - lx * F2) % PAIR_THREADS; e < F2; e += PAIR_THREADS)
                    if (yz[e] >> 31) buf[lx * PS + e] *= 0.5;
            __syncthreads();  // the plane has landed everywhere; the other buffer is consumed
            gen_plane(lx + 1);
            if (SYM && lx + 1 == box.n[0] && next < box.classes) keys(next);  // (every copy of this class is queued)
            // rows that meet this plane (offsets into the maps and the values)
            const int rows = SYM ? (lx + 1) * nyz : N, xmax = SYM ? lx + 1 : box.n[0];
            int mo[TPW][2], po[TPW][2];
            // first k step of a tile: below it, in the diagonal plane, l lies
            // before every row of the tile
            int from[TPW];
            int nact = 0;
#pragma unroll
            for (int t = 0; t < TPW; ++t) {
                const int below = 16 * (warp + PAIR_WARPS * t) - lx * nyz;
                from[t] = SYM && below > 0 ? below >> 2 : 0;
                if (16 * (warp + PAIR_WARPS * t) < rows) nact = t + 1;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int k = row_k[t][i];
                    const bool in = k < xmax;
                    mo[t][i] = in ? row_m[t][i] + (SYM && k == lx ? nyz * map_ld : 0) : 2 * nyz * map_ld + q;
                    po[t][i] = (lx & 1) * box.n[0] * PS + (in ? k * PS : 0);
                }
            }
            const int bo = lay.planes + (lx * nyz + q) * LDB + c8;
            auto steps = [&](auto active, auto columns, int st0, int st1) {
                constexpr int A = decltype(active)::value, J = decltype(columns)::value;
                auto step = [&](int st, bool last) {
                    // (past the plane's last point B is taken as zero, not only
                    // A: a state or orbital may hold infinities in the next plane)
                    const bool in = !last || 4 * st + q < nyz;
                    double bf[J];
#pragma unroll
                    for (int j = 0; j < J; ++j) bf[j] = in ? sm[bo + st * 4 * LDB + 8 * j] : 0.0;
#pragma unroll
                    for (int t = 0; t < A; ++t) {
                        const double a0 = sm[po[t][0] + map[mo[t][0] + 4 * st]], a1 = sm[po[t][1] + map[mo[t][1] + 4 * st]];
#pragma unroll
                        for (int j = 0; j < J; ++j) dm_mma(acc[t][0][j], bf[j], a0);
#pragma unroll
                        for (int j = 0; j < J; ++j) dm_mma(acc[t][1][j], bf[j], a1);
                    }
                };
#pragma unroll 2
                for (int st = st0; st < min(st1, box.S - 1); ++st) {
                    step(st, false);
                    gen_one();
                }
                if (st1 == box.S) step(box.S - 1, true);
            };
            auto planes_of = [&](auto active, int st0, int st1) {
                if constexpr (!SYM && NT > 1) {
                    if (live == 1) return steps(active, std::integral_constant<int, 1>{}, st0, st1);
                    if constexpr (NT > 2)
                        if (live == 2) return steps(active, std::integral_constant<int, 2>{}, st0, st1);
                }
                steps(active, std::integral_constant<int, NT>{}, st0, st1);
            };
            if constexpr (TPW >= 2)
                if (nact == 2) {
                    if (SYM) planes_of(std::integral_constant<int, 1>{}, from[0], from[1]);
                    planes_of(std::integral_constant<int, 2>{}, from[1], box.S);
                }
            if (nact == 1) planes_of(std::integral_constant<int, 1>{}, from[0], box.S);
            while (gk < gend) gen_one();
            dm_commit();
        }
        if constexpr (SYM) {
            // Y^T[s][r] = sum_k A[k][s] B[k][r]: an accumulator tile (s, k) is
            // itself the left operand of two MMAs over its k of equal parity; each
            // warp's rows give a part of Y^T, summed in shared memory
            __syncthreads();  // the planes are consumed, the next class's keys made
            if (next < box.classes) key_pairs();
            double* Y = sm + lay.sum;  // [s][8 NT + 1]
            double* part = sm + lay.part;
            for (int i0 = 0; i0 < NT; i0 += lay.rows) {
#pragma unroll
                for (int is = 0; is < NT; ++is) {
                    if (is < i0 || is >= i0 + lay.rows) continue;
                    double y[NT][2];
#pragma unroll
                    for (int j = 0; j < NT; ++j) y[j][0] = y[j][1] = 0.0;
#pragma unroll
                    for (int t = 0; t < TPW; ++t)
                        if (t < mine) {
#pragma unroll
                            for (int i = 0; i < 2; ++i)
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    const int k = 16 * (warp + PAIR_WARPS * t) + 8 * i + 2 * q + h;
#pragma unroll
                                    for (int j = 0; j < NT; ++j)
                                        dm_mma(y[j], acc[t][i][is][h], k < N ? B[k * LDB + 8 * j + c8] : 0.0);
                                }
                        }
                    double* p = part + (((is - i0) * PAIR_WARPS + warp) * 8 + c8) * 8 * NT + 2 * q;
#pragma unroll
                    for (int j = 0; j < NT; ++j) p[8 * j] = y[j][0], p[8 * j + 1] = y[j][1];
                }
                __syncthreads();
                // the next class's first plane: its copies land meanwhile
                if (i0 == 0 && next < box.classes) gen_first();
                const int n = min(lay.rows, NT - i0) * 64 * NT;
                for (int e = tid; e < n; e += PAIR_THREADS) {
                    const double* p = part + e / (64 * NT) * (PAIR_WARPS * 64 * NT) + e % (64 * NT);
                    double v = 0.0;
#pragma unroll
                    for (int w = 0; w < PAIR_WARPS; ++w) v += p[w * 64 * NT];
                    Y[(8 * i0 + e / (8 * NT)) * (8 * NT + 1) + e % (8 * NT)] = v;
                }
                __syncthreads();
            }
            double* o = out + (i64)cls * (cols * (cols + 1) / 2);
            for (int e = tid; e < 64 * NT * NT; e += PAIR_THREADS) {
                const int r = e / (8 * NT), c = e - r * (8 * NT);
                if (r < cols && c <= r) o[r * (r + 1) / 2 + c] = Y[r * (8 * NT + 1) + c] + Y[c * (8 * NT + 1) + r];
            }
            __syncthreads();  // Y is consumed
            zeros();
        } else {
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                if (j >= live) break;
                const i64 to = cdst[8 * j + c8];
                if (to < 0) continue;
#pragma unroll
                for (int t = 0; t < TPW; ++t)
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int k = 16 * (warp + PAIR_WARPS * t) + 8 * i + 2 * q + h;
                            if (k < N) out[to + (i64)k * cols] = acc[t][i][j][h];
                        }
            }
            __syncthreads();  // the planes are consumed before the next columns' first copy
        }
        }
    }
}

// the box fits the kernel: rows in the warps' tiles, 16-bit maps, shared memory
inline bool pair_box_fits(const PairBox& b, int nt) {
    return b.N <= PAIR_MAX_POINTS && b.F2 < 65535 && pair_axis_keys(b.L) < 32768 &&
           PairSmem(b, PAIR_MAX_WARPS, nt).bytes <= (size_t)227 * 1024;
}

template <int W, int NT, int TPW, bool SYM>
void pair_contract_launch(const PairBox& b, const double* table, const double* bsrc, int cols, int ld, int col0,
                          double* out, cudaStream_t s) {
    const size_t smem = PairSmem(b, W, NT).bytes;
    auto* kernel = k_pair_contract<W, NT, TPW, SYM>;
    GLI_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 1;
    GLI_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * W, smem));
    const i64 slots = (i64)context().num_sms * (per_sm > 0 ? per_sm : 1);
    const unsigned blocks = (unsigned)(b.classes < slots ? b.classes : slots);
    launch_kernel(kernel, dim3(blocks), dim3(32 * W), smem, s, b, table, bsrc, cols, ld, col0, out);
}

// A = V[c] B for every class c of the box; nt = column tiles of 8
template <bool SYM>
void pair_contract(const PairBox& b, int nt, const double* table, const double* bsrc, int cols, int ld, int col0,
                   double* out, cudaStream_t s) {
    auto go = [&](auto n) {
        constexpr int NT = decltype(n)::value;
        // two blocks of 8 warps where both fit an SM (228 KB with 1 KB a block)
        const bool two = b.N <= 256 && 2 * (PairSmem(b, 8, NT).bytes + 1024) <= (size_t)228 * 1024;
        if (two && b.N <= 128)
            pair_contract_launch<8, NT, 1, SYM>(b, table, bsrc, cols, ld, col0, out, s);
        else if (two)
            pair_contract_launch<8, NT, 2, SYM>(b, table, bsrc, cols, ld, col0, out, s);
        else if (b.N <= 256)
            pair_contract_launch<16, NT, 1, SYM>(b, table, bsrc, cols, ld, col0, out, s);
        else
            pair_contract_launch<16, NT, 2, SYM>(b, table, bsrc, cols, ld, col0, out, s);
    };
    if (nt <= 1)
        go(std::integral_constant<int, 1>{});
    else if (nt == 2)
        go(std::integral_constant<int, 2>{});
    else if (nt == 3)
        go(std::integral_constant<int, 3>{});
    else
        go(std::integral_constant<int, 4>{});
}

}  // namespace gli
