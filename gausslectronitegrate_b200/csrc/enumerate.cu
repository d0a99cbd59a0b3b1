// Symmetry-reduced class enumeration on the device, bit-exact with
// enumerate_symmetry_reduced_erida_indices (src/erida_integrals.c:300-410) and
// enumerate_symmetry_reduced_eri_indices (src/eri_integrals.c:382-526).
//
// A candidate tuple is kept when no element of its orbit -- the 48 O_h images
// of the tuple and of its bias-shifted copies (a doubled box centre of +-1 on an
// axis admits the copy moved by that centre), combined with the index
// permutations i<->j (and k<->l, (ij)<->(kl) for ERI) -- has a smaller
// linearised index.  Images are computed arithmetically from the signed
// permutation matrices, so no 48 x N permutation tables are built.
//
// Candidates are generated so that the flat candidate order equals ascending
// index order: a slot is i (ERIDA: partners j ascending) or (i, j, k) (ERI:
// partners l ascending), and slots ascend with the index.
//
// A filter skips most candidates before the orbit test.  A candidate's index
// leads with its first point i, and an image of the tuple whose smallest point
// index lies below i is a smaller index, so no point of a canonical tuple has
// an O_h image below i: with omin[p] the smallest index among the 48 images of
// point p (the unshifted copies are part of every orbit), a canonical tuple has
// omin[i] = i and omin[q] >= i for each other point q.
//
// ERIDA, live slots in closed form: a point that is the smallest of its images
// is (-a, -b, -c) with a >= b >= c >= 0, so the live slots are numbered by the
// tetrahedral index of (a, b, c), descending.  A warp takes one slot, a lane each
// of its 27 partners, and keeps the ballot of the survivors (k_erida_slots); a
// scan of their counts and a pass over the ballots write the list
// (k_erida_place).  The orbit test is arithmetic too: the copies' points compare
// by their sorted absolute coordinates, and where a point's image is the slot's
// point itself, six axis permutations give the smallest partner (the signs
// follow, or are free where a coordinate is zero).  33^3: 388 us for a thread per
// point of the grid over all 48 images, 5 us now; the 129^3 list 1.4 ms, now 0.16
// ms with its copy.
//
// ERI, live slots: at 7^3, 168,092 of the 40 million slots (i, j, k) hold a
// canonical class, and a thread per slot leaves most lanes of a warp idle
// beside one busy slot.  The slots that pass the filter are compacted first
// (k_enum_live; 3^3 skips it, k_enum_small); a warp then takes each live slot's partner candidates 32 at
// a time in ascending order, keeps the survivors (placed in order by its
// ballots) in shared memory and appends them to a scratch buffer, and a scan
// of the slots' counts and a copy place the runs (k_enum_slots_collect).  7^3:
// 25 ms with arithmetic images of every copy, 3.5 ms reading them from the table, 2.9
// ms testing two images at a time for one that leads with i.
//
// Fallbacks, when a slot's survivors exceed its buffer or the scratch buffer
// fills: two passes (count, scan, write) over the live slots (k_enum_slots).
// The thread-per-slot two passes (k_enum_erida, k_enum_eri) and the live-slot
// passes for ERIDA remain for the tests.  The output is sorted by construction
// on every path.
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>

#include "symmetry.cuh"

namespace gli {

// ---------------------------------------------------------------------------
// ERIDA: slot i; partner coordinates j_a = -i_a - 1 + t_a, t_a in {0,1,2}
// (doubled box centre t_a - 1), ascending in (t_x, t_y, t_z) = ascending j.
template <class Emit>
__device__ inline void erida_candidates(const SymGrid& G, i64 i, Emit&& emit) {
    if (G.omin[i] != (int)i) return;
    int p[2][3];
    point_of(G, i, p[0]);
    for (int tx = 0; tx < 3; ++tx) {
        const int jx = -p[0][0] - 1 + tx;
        if (jx < -G.e || jx > G.e || jx < p[0][0]) continue;
        for (int ty = 0; ty < 3; ++ty) {
            const int jy = -p[0][1] - 1 + ty;
            if (jy < -G.e || jy > G.e) continue;
            for (int tz = 0; tz < 3; ++tz) {
                const int jz = -p[0][2] - 1 + tz;
                if (jz < -G.e || jz > G.e) continue;
                p[1][0] = jx;
                p[1][1] = jy;
                p[1][2] = jz;
                const i64 j = lin3(G, p[1]);
                if (G.omin[j] < (int)i) continue;
                const int bias[3] = {tx - 1, ty - 1, tz - 1};
                const i64 idx = i * G.N + j;
                if (canonical_pair(G, p, bias, idx)) emit(idx);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// ERI: one thread per (i, j, k); admissible l coordinates per axis keep the
// doubled box centre min + max in {-1, 0, 1}.
constexpr int MAX_AXIS = 72;  // room for L <= 63

// ascending admissible partner coordinates l for fixed lo/hi of (i, j, k)
__device__ inline int axis_partners(int lo, int hi, int e, int lmin, signed char* s) {
    int n = 0;
    for (int d = -1; d <= 1; ++d) {  // l < lo: centre l + hi
        const int l = d - hi;
        if (l >= -e && l < lo && l >= lmin) s[n++] = (signed char)l;
    }
    if (lo + hi >= -1 && lo + hi <= 1)  // lo <= l <= hi: centre lo + hi
        for (int l = lo; l <= hi; ++l)
            if (l >= lmin) s[n++] = (signed char)l;
    for (int d = -1; d <= 1; ++d) {  // l > hi: centre lo + l
        const int l = d - lo;
        if (l > hi && l <= e && l >= lmin) s[n++] = (signed char)l;
    }
    return n;
}

// ERI slot t = (i N + j) N + k -> points, and a point's coordinates, in 32-bit
// arithmetic where the slots fit it (grids up to 11^3): 64-bit divisions took
// most of a small grid's walk
__device__ __forceinline__ void eri_slot_points(const SymGrid& G, i64 t, int& i, int& j, int& k) {
    const uint32_t N = (uint32_t)G.N;
    if (N <= 1625) {
        const uint32_t u = (uint32_t)t, ij = u / N;
        k = (int)(u - ij * N);
        i = (int)(ij / N);
        j = (int)(ij - i * N);
    } else {
        const uint32_t ij = (uint32_t)(t / N);  // (N^2 < 2^32)
        k = (int)(t - (i64)ij * N);
        i = (int)(ij / N);
        j = (int)(ij - i * N);
    }
}
__device__ __forceinline__ void point32(const SymGrid& G, int lin, int p[3]) {
    const int r = lin / G.L, x = r / G.L;
    p[2] = lin - r * G.L - G.e;
    p[1] = r - x * G.L - G.e;
    p[0] = x - G.e;
}

// ERI: slot t = (i, j, k)
template <class Emit>
__device__ inline void eri_candidates(const SymGrid& G, i64 t, Emit&& emit) {
    int i, j, k;
    eri_slot_points(G, t, i, j, k);
    if (G.omin[i] != i || G.omin[j] < i || G.omin[k] < i) return;
    int p[4][3];
    point32(G, i, p[0]);
    point32(G, j, p[1]);
    point32(G, k, p[2]);
    // reference x-ordering: i <= j, i <= k (and k <= l below) on the x coordinate
    if (p[0][0] <= p[1][0] && p[0][0] <= p[2][0]) {
        signed char sx[MAX_AXIS], sy[MAX_AXIS], sz[MAX_AXIS];
        int lo[3], hi[3];
        for (int a = 0; a < 3; ++a) {
            lo[a] = min(min(p[0][a], p[1][a]), p[2][a]);
            hi[a] = max(max(p[0][a], p[1][a]), p[2][a]);
        }
        const int nx = axis_partners(lo[0], hi[0], G.e, p[2][0], sx);
        const int ny = axis_partners(lo[1], hi[1], G.e, -G.e, sy);
        const int nz = axis_partners(lo[2], hi[2], G.e, -G.e, sz);
        const i64 base = t * G.N;
        for (int ax = 0; ax < nx; ++ax) {
            p[3][0] = sx[ax];
            const int bx = min(lo[0], p[3][0]) + max(hi[0], p[3][0]);
            for (int ay = 0; ay < ny; ++ay) {
                p[3][1] = sy[ay];
                const int by = min(lo[1], p[3][1]) + max(hi[1], p[3][1]);
                for (int az = 0; az < nz; ++az) {
                    p[3][2] = sz[az];
                    const i64 l = lin3(G, p[3]);
                    if (G.omin[l] < (int)i) continue;
                    const int bz = min(lo[2], p[3][2]) + max(hi[2], p[3][2]);
                    const int bias[3] = {bx, by, bz};
                    const int pts[4] = {i, j, k, (int)l};
                    if (canonical_quad(G, pts, bias)) emit(base + l);
                }
            }
        }
    }
}

template <int KIND, class Emit>
__device__ inline void slot_candidates(const SymGrid& G, i64 t, Emit&& emit) {
    if (KIND == 0)
        erida_candidates(G, t, emit);
    else
        eri_candidates(G, t, emit);
}

// status of the pass over the live slots
struct EnumStatus {
    unsigned long long used;  // scratch entries reserved
    uint64_t total;           // classes in the list (the scan of the runs)
    int overflow;             // 1: a slot's survivors exceeded its buffer; 2: the scratch buffer filled
};

// smallest linear index among the 48 O_h images of each grid point, and (images
// non-null: ERI) the images themselves, 16 bits each; eight lanes a point, six of
// them with eight images each.  Clears the status of the pass that follows.
__global__ void __launch_bounds__(256) k_orbit_min(SymGrid G, int* __restrict__ omin, uint4* __restrict__ images,
                                                   EnumStatus* __restrict__ st) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *st = EnumStatus{0ull, 0ull, 0};
    const i64 p = (i64)blockIdx.x * (blockDim.x >> 3) + (threadIdx.x >> 3);
    const int c = threadIdx.x & 7;
    int best = INT_MAX;
    if (p < G.N && c < 6) {
        int q[3];
        point32(G, (int)p, q);
        uint32_t w[4];
#pragma unroll
        for (int h = 0; h < 8; ++h) {
            int r[3];
            oh_apply(8 * c + h, q, r);
            const int l = ((r[0] + G.e) * G.L + r[1] + G.e) * G.L + r[2] + G.e;
            best = min(best, l);
            w[h >> 1] = h & 1 ? w[h >> 1] | (uint32_t)l << 16 : (uint32_t)l;
        }
        if (images) images[p * 6 + c] = make_uint4(w[0], w[1], w[2], w[3]);
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (p < G.N && c == 0) omin[p] = best;
}

// ---------------------------------------------------------------------------
// ERIDA: live slots in closed form

// live slot s (ascending linear index) of extent e -> (a, b, c): the tetrahedral
// index from the other end
__device__ __forceinline__ void erida_slot_point(i64 t, int& a, int& b, int& c) {
    a = (int)cbrt(6.0 * (double)t);
    while ((i64)(a + 1) * (a + 2) * (a + 3) / 6 <= t) ++a;
    while ((i64)a * (a + 1) * (a + 2) / 6 > t) --a;
    const i64 r = t - (i64)a * (a + 1) * (a + 2) / 6;
    b = (int)((sqrt(8.0 * (double)r + 1.0) - 1.0) * 0.5);
    while ((i64)(b + 1) * (b + 2) / 2 <= r) ++b;
    while ((i64)b * (b + 1) / 2 > r) --b;
    c = (int)(r - (i64)b * (b + 1) / 2);
}

// sorted absolute coordinates, largest first, 10 bits each: a larger key is a
// smaller smallest image
__device__ __forceinline__ uint32_t orbit_key(int x, int y, int z) {
    const int a = absi(x), b = absi(y), c = absi(z);
    const int hi = max(a, max(b, c)), lo = min(a, min(b, c));
    return (uint32_t)hi << 20 | (uint32_t)(a + b + c - hi - lo) << 10 | (uint32_t)lo;
}

// does some O_h element that takes q to (-a, -b, -c) take r below j?
__device__ __forceinline__ bool partner_below(const int q[3], const int r[3], int a, int b, int c, const int j[3]) {
    bool below = false;
#pragma unroll
    for (int perm = 0; perm < 6; ++perm) {
        const int a0 = perm < 2 ? 0 : perm < 4 ? 1 : 2;
        const int a1 = perm == 0 ? 1 : perm == 1 ? 2 : perm == 2 ? 0 : perm == 3 ? 2 : perm == 4 ? 0 : 1;
        const int a2 = 3 - a0 - a1;
        const bool maps = absi(q[a0]) == a && absi(q[a1]) == b && absi(q[a2]) == c;
        const int x = q[a0] == 0 ? -absi(r[a0]) : q[a0] > 0 ? -r[a0] : r[a0];
        const int y = q[a1] == 0 ? -absi(r[a1]) : q[a1] > 0 ? -r[a1] : r[a1];
        const int z = q[a2] == 0 ? -absi(r[a2]) : q[a2] > 0 ? -r[a2] : r[a2];
        below = below || (maps && (x < j[0] || (x == j[0] && (y < j[1] || (y == j[1] && z < j[2])))));
    }
    return below;
}

// a warp per live slot: masks[s] = ballot of its surviving partners (lane
// 9 tx + 3 ty + tz, ascending j), counts[s] their number
__global__ void __launch_bounds__(256) k_erida_slots(SymGrid G, i64 nlive, uint32_t* __restrict__ masks,
                                                     uint32_t* __restrict__ counts) {
    const i64 s = (i64)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (s >= nlive) return;
    const int lane = threadIdx.x & 31;
    int a, b, c;
    erida_slot_point(nlive - 1 - s, a, b, c);
    const uint32_t key = (uint32_t)a << 20 | (uint32_t)b << 10 | (uint32_t)c;
    const int tx = lane / 9, ty = lane / 3 % 3, tz = lane % 3;
    const int p[3] = {-a, -b, -c}, j[3] = {a - 1 + tx, b - 1 + ty, c - 1 + tz};
    bool keep = lane < 27 && j[0] >= p[0];
    for (int x = 0; x < 3; ++x) keep = keep && absi(j[x]) <= G.e;
    if (keep) {
        const int bias[3] = {tx - 1, ty - 1, tz - 1};
        for (int m = 0; m < 8 && keep; ++m) {
            if ((m & 1 && !bias[0]) || (m & 2 && !bias[1]) || (m & 4 && !bias[2])) continue;
            int q0[3], q1[3];
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                const int sft = m >> x & 1 ? bias[x] : 0;
                q0[x] = p[x] - sft;
                q1[x] = j[x] - sft;
            }
            const uint32_t k0 = orbit_key(q0[0], q0[1], q0[2]), k1 = orbit_key(q1[0], q1[1], q1[2]);
            keep = k0 <= key && k1 <= key;
            if (keep && k0 == key) keep = !partner_below(q0, q1, a, b, c, j);
            if (keep && k1 == key) keep = !partner_below(q1, q0, a, b, c, j);
        }
    }
    const unsigned ballot = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) {
        masks[s] = ballot;
        counts[s] = __popc(ballot);
    }
}

// the classes of slot s, a thread per slot, at dest[s]
__global__ void __launch_bounds__(256) k_erida_place(SymGrid G, i64 nlive, const uint32_t* __restrict__ masks,
                                                     const uint64_t* __restrict__ dest, int64_t* __restrict__ out) {
    const i64 s = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nlive) return;
    uint32_t m = masks[s];
    if (!m) return;
    int a, b, c;
    erida_slot_point(nlive - 1 - s, a, b, c);
    const int p[3] = {-a, -b, -c};
    const i64 base = lin3(G, p) * G.N;
    int64_t* o = out + dest[s];
    for (; m; m &= m - 1) {
        const int l = __ffs(m) - 1;
        const int j[3] = {a - 1 + l / 9, b - 1 + l / 3 % 3, c - 1 + l % 3};
        *o++ = base + lin3(G, j);
    }
}

// ---------------------------------------------------------------------------
// two passes: survivors per slot, then each slot's survivors at its offset
template <bool WRITE>
__global__ void k_enum_erida(SymGrid G, uint32_t* __restrict__ counts, const uint64_t* __restrict__ offsets,
                             int64_t* __restrict__ out) {
    const i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= G.N) return;
    if (WRITE) {
        uint64_t w = offsets[i];
        erida_candidates(G, i, [&](i64 idx) { out[w++] = idx; });
    } else {
        uint32_t c = 0;
        erida_candidates(G, i, [&](i64) { ++c; });
        counts[i] = c;
    }
}

template <bool WRITE>
__global__ void k_enum_eri(SymGrid G, uint32_t* __restrict__ counts, const uint64_t* __restrict__ offsets,
                           int64_t* __restrict__ out) {
    const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= G.N * G.N * G.N) return;
    if (WRITE) {
        uint64_t w = offsets[t];
        eri_candidates(G, t, [&](i64 idx) { out[w++] = idx; });
    } else {
        uint32_t c = 0;
        eri_candidates(G, t, [&](i64) { ++c; });
        counts[t] = c;
    }
}

// ---------------------------------------------------------------------------
// one pass over the live slots

// each slot's run from the scratch buffer to its place (dest: exclusive scan
// of the run lengths in slot order); one warp per run
__global__ void k_enum_place(const int64_t* __restrict__ scratch, const uint32_t* __restrict__ run_n,
                             const unsigned long long* __restrict__ run_off, const uint64_t* __restrict__ dest,
                             i64 runs, int64_t* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const i64 warps = (i64)gridDim.x * (blockDim.x >> 5);
    for (i64 r = (i64)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < runs; r += warps) {
        const uint32_t n = run_n[r];
        if (n == 0) continue;
        const int64_t* src = scratch + run_off[r];
        int64_t* dst = out + dest[r];
        for (uint32_t k = lane; k < n; k += 32) dst[k] = src[k];
    }
}

// scratch entries of ERI lists, which hold about N^4 / 3,900 classes at L = 7
// (and a falling fraction beyond): N^4 / 1024 with a floor; at most 2^26 entries
// (512 MB); a list that does not fit takes the two passes
static i64 enum_scratch(const SymGrid& G) {
    const double N = (double)G.N;
    return (i64)std::min(N * N * N * N / 1024 + (1 << 20), (double)((i64)1 << 26));
}

// the ERIDA list through the live slots in closed form
static i64 enumerate_erida(const SymGrid& G, int64_t** d_out, cudaStream_t s) {
    const i64 e = G.e, nlive = (e + 1) * (e + 2) * (e + 3) / 6;
    DevBuf<uint32_t> masks(nlive, s), counts(nlive, s);
    DevBuf<uint64_t> dest(nlive, s);
    k_erida_slots<<<(unsigned)((nlive + 7) / 8), 256, 0, s>>>(G, nlive, masks.p, counts.p);
    GLI_CHECK_LAUNCH();
    int64_t* out = nullptr;
    auto place = [&](i64 entries) {
        GLI_CUDA(cudaMallocAsync((void**)&out, std::max<i64>(entries, 1) * sizeof(int64_t), s));
        k_erida_place<<<(unsigned)((nlive + 255) / 256), 256, 0, s>>>(G, nlive, masks.p, dest.p, out);
        GLI_CHECK_LAUNCH();
    };
    // A slot has at most 27 partners: lists whose bound takes at most 32 MB
    // (191 points per axis) are placed before the host reads their length, which
    // saves a round trip in the middle (20 us of 33^3's 190).
    const i64 bound = 27 * nlive;
    i64 total = 0;
    if (bound <= ((i64)4 << 20)) {
        DevBuf<uint64_t> len(1, s);
        exclusive_scan_u32_dev(counts.p, dest.p, nlive, len.p, s);
        place(bound);
        uint64_t h = 0;
        GLI_CUDA(cudaMemcpyAsync(&h, len.p, sizeof(h), cudaMemcpyDeviceToHost, s));
        GLI_CUDA(cudaStreamSynchronize(s));
        total = (i64)h;
    } else {
        total = exclusive_scan_u32(counts.p, dest.p, nlive, s);
        place(total);
    }
    *d_out = out;
    return total;
}

// can slot t hold a canonical class: the omin filter (ERIDA: i canonical;
// ERI: also omin[j], omin[k] >= i) and for ERI the reference's x-ordering
// (i_x <= j_x, i_x <= k_x)
template <int KIND>
__device__ inline bool slot_live(const SymGrid& G, i64 t) {
    if (KIND == 0) return G.omin[t] == (int)t;
    int i, j, k;
    eri_slot_points(G, t, i, j, k);
    if (G.omin[i] != i || G.omin[j] < i || G.omin[k] < i) return false;
    // x coordinate: the leading digit of the x-major linear index
    const int x0 = i / (G.L * G.L) * (G.L * G.L);
    return x0 <= j && x0 <= k;
}

// WRITE = false: live slots per block of 256; WRITE = true: their ids at the
// block's offset, in order
template <int KIND, bool WRITE>
__global__ void __launch_bounds__(256) k_enum_live(SymGrid G, i64 slots, uint32_t* __restrict__ block_counts,
                                                   const uint64_t* __restrict__ block_offsets,
                                                   int64_t* __restrict__ slot_ids) {
    __shared__ uint32_t wsum[8];
    const i64 t = (i64)blockIdx.x * 256 + threadIdx.x;
    const bool live = t < slots && slot_live<KIND>(G, t);
    const unsigned b = __ballot_sync(0xffffffffu, live);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) wsum[warp] = __popc(b);
    __syncthreads();
    if (!WRITE) {
        if (threadIdx.x == 0) {
            uint32_t tot = 0;
            for (int w = 0; w < 8; ++w) tot += wsum[w];
            block_counts[blockIdx.x] = tot;
        }
        return;
    }
    uint32_t before = 0;
    for (int w = 0; w < warp; ++w) before += wsum[w];
    if (live) slot_ids[block_offsets[blockIdx.x] + before + __popc(b & ((1u << lane) - 1u))] = t;
}

// The 27 partner candidates j of live ERIDA slot i (lane c = 9 tx + 3 ty + tz,
// ascending j), emit(idx, rank) called by every lane after the ballot (idx < 0
// for a lane without a survivor).  Returns the slot's survivors.
template <class Emit>
__device__ inline uint32_t erida_slot_walk(const SymGrid& G, i64 i, int lane, Emit&& emit) {
    int p[2][3];
    point_of(G, i, p[0]);
    bool keep = false;
    i64 idx = 0;
    if (lane < 27) {
        const int tx = lane / 9, ty = (lane / 3) % 3, tz = lane % 3;
        p[1][0] = -p[0][0] - 1 + tx;
        p[1][1] = -p[0][1] - 1 + ty;
        p[1][2] = -p[0][2] - 1 + tz;
        bool in = p[1][0] >= p[0][0];
        for (int a = 0; a < 3; ++a) in = in && p[1][a] >= -G.e && p[1][a] <= G.e;
        if (in) {
            const i64 j = lin3(G, p[1]);
            if (G.omin[j] >= (int)i) {
                const int bias[3] = {tx - 1, ty - 1, tz - 1};
                idx = i * G.N + j;
                keep = canonical_pair(G, p, bias, idx);
            }
        }
    }
    const unsigned b = __ballot_sync(0xffffffffu, keep);
    emit(keep ? idx : (i64)-1, (uint32_t)__popc(b & ((1u << lane) - 1u)));
    return (uint32_t)__popc(b);
}

// The partner candidates l of live slot t (ascending), 32 at a time, one per
// lane; emit(idx, rank) is called by every lane after each group's ballot
// (rank: the place of the lane's survivor among the slot's survivors; idx < 0
// for a lane without one).  Returns the slot's survivors (the same in every
// lane).
template <class Emit>
__device__ inline uint32_t eri_slot_walk(const SymGrid& G, i64 t, int lane, Emit&& emit) {
    const i64 N = G.N;
    {
        int i, j, k;
        eri_slot_points(G, t, i, j, k);
        int p[4][3];
        point32(G, i, p[0]);
        point32(G, j, p[1]);
        point32(G, k, p[2]);
        signed char sx[MAX_AXIS], sy[MAX_AXIS], sz[MAX_AXIS];
        int lo[3], hi[3];
        for (int a = 0; a < 3; ++a) {
            lo[a] = min(min(p[0][a], p[1][a]), p[2][a]);
            hi[a] = max(max(p[0][a], p[1][a]), p[2][a]);
        }
        const int nx = axis_partners(lo[0], hi[0], G.e, p[2][0], sx);
        const int ny = axis_partners(lo[1], hi[1], G.e, -G.e, sy);
        const int nz = axis_partners(lo[2], hi[2], G.e, -G.e, sz);
        const int total = nx * ny * nz;  // the same in every lane
        const i64 base = t * N;
        uint32_t c = 0;
        for (int c0 = 0; c0 < total; c0 += 32) {
            const int cand = c0 + lane;
            bool keep = false;
            i64 idx = 0;
            if (cand < total) {
                const int az = cand % nz, r = cand / nz, ay = r % ny, ax = r / ny;
                p[3][0] = sx[ax];
                p[3][1] = sy[ay];
                p[3][2] = sz[az];
                const int l = ((p[3][0] + G.e) * G.L + p[3][1] + G.e) * G.L + p[3][2] + G.e;
                if (G.omin[l] >= i) {
                    const int bias[3] = {min(lo[0], p[3][0]) + max(hi[0], p[3][0]),
                                         min(lo[1], p[3][1]) + max(hi[1], p[3][1]),
                                         min(lo[2], p[3][2]) + max(hi[2], p[3][2])};
                    const int pts[4] = {i, j, k, l};
                    idx = base + l;
                    keep = canonical_quad(G, pts, bias);
                }
            }
            const unsigned b = __ballot_sync(0xffffffffu, keep);
            emit(keep ? idx : (i64)-1, c + __popc(b & ((1u << lane) - 1u)));
            c += __popc(b);
        }
        return c;
    }
}

template <int KIND, class Emit>
__device__ inline uint32_t slot_walk(const SymGrid& G, i64 t, int lane, Emit&& emit) {
    if (KIND == 0) return erida_slot_walk(G, t, lane, emit);
    return eri_slot_walk(G, t, lane, emit);
}

// one warp per live slot; WRITE = false: survivors per slot; WRITE = true:
// survivors at the slot's offset, in order
template <int KIND, bool WRITE>
__global__ void __launch_bounds__(256) k_enum_slots(SymGrid G, const int64_t* __restrict__ slot_ids, i64 nlive,
                                                    uint32_t* __restrict__ counts,
                                                    const uint64_t* __restrict__ offsets, int64_t* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const i64 warps = (i64)gridDim.x * (blockDim.x >> 5);
    for (i64 sl = (i64)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); sl < nlive; sl += warps) {
        const uint64_t w = WRITE ? offsets[sl] : 0;
        const uint32_t c = slot_walk<KIND>(G, slot_ids[sl], lane, [&](i64 idx, uint32_t rank) {
            if (WRITE && idx >= 0) out[w + rank] = idx;
        });
        if (!WRITE && lane == 0) counts[sl] = c;
    }
}

// one pass over the live slots: each warp keeps its slot's survivors in shared
// memory, then appends them to the scratch buffer (run_n, run_off per slot);
// a slot with more than ENUM_SLOT_CAP survivors or a full scratch buffer sets
// the overflow status
constexpr int ENUM_SLOT_CAP = 512;

template <int KIND>
__global__ void __launch_bounds__(256) k_enum_slots_collect(SymGrid G, const int64_t* __restrict__ slot_ids,
                                                            i64 nlive, int64_t* __restrict__ scratch,
                                                            unsigned long long cap, uint32_t* __restrict__ run_n,
                                                            unsigned long long* __restrict__ run_off,
                                                            EnumStatus* __restrict__ st) {
    __shared__ int64_t buf[8][ENUM_SLOT_CAP];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const i64 warps = (i64)gridDim.x * (blockDim.x >> 5);
    int64_t* mine = buf[warp];
    for (i64 sl = (i64)blockIdx.x * (blockDim.x >> 5) + warp; sl < nlive; sl += warps) {
        const uint32_t c = slot_walk<KIND>(G, slot_ids[sl], lane, [&](i64 idx, uint32_t rank) {
            if (idx >= 0 && rank < ENUM_SLOT_CAP) mine[rank] = idx;
        });
        __syncwarp();
        unsigned long long off = 0;
        if (c > 0 && c <= ENUM_SLOT_CAP && lane == 0) off = atomicAdd(&st->used, (unsigned long long)c);
        off = __shfl_sync(0xffffffffu, off, 0);
        const bool fits = c <= ENUM_SLOT_CAP && off + c <= cap;
        if (lane == 0) {
            run_n[sl] = fits ? c : 0u;
            run_off[sl] = off;
            if (!fits) atomicOr(&st->overflow, c > ENUM_SLOT_CAP ? 1 : 2);
        }
        if (fits)
            for (uint32_t q = lane; q < c; q += 32) scratch[off + q] = mine[q];
        __syncwarp();
    }
}

// ERI grids up to 3^3 (at most 27 partners a slot): a block per slot of the live
// leading points (those in closed form as for ERIDA: 4 of 27), without compacting
// the live slots and the host round trip for their number.  The few slots do not
// fill the GPU, so each is spread out: a warp takes four partners, eight lanes
// each, a lane per shifted copy.  Bound: instructions, 69% of the issue slots
// (3^3: 14 us; 23 us with every warp making the slot's points and partner lists
// for itself, 53 us with a warp per slot and a lane per partner, one chain of up
// to eight copies' images).
constexpr int ENUM_SMALL_L = 3;

__global__ void __launch_bounds__(256) k_enum_small(SymGrid G, i64 npoints, int64_t* __restrict__ scratch,
                                                    unsigned long long cap, uint32_t* __restrict__ run_n,
                                                    unsigned long long* __restrict__ run_off,
                                                    EnumStatus* __restrict__ st) {
    __shared__ unsigned kept;
    __shared__ int s_pts[3], s_lo[3], s_hi[3], s_n[3];  // the slot's points; per axis their box and the partners
    __shared__ signed char s_part[3][4];
    const int N = (int)G.N, N2 = N * N, sl = blockIdx.x, lane = threadIdx.x & 31;
    // the slot, made by the first warp, a lane per axis
    if (threadIdx.x < 32) {
        const int r = (int)npoints - 1 - sl / N2;  // the leading point's number, as erida_slot_point
        int a = 0, b = 0;
        while ((a + 1) * (a + 2) * (a + 3) / 6 <= r) ++a;
        const int rb = r - a * (a + 1) * (a + 2) / 6;
        while ((b + 1) * (b + 2) / 2 <= rb) ++b;
        const int p0[3] = {-a, -b, b * (b + 1) / 2 - rb};
        const int jk = sl % N2, i = (int)lin3(G, p0), j = jk / N, k = jk - j * N;
        const bool live = slot_live<1>(G, (i64)i * N2 + jk);
        if (lane < 3) {
            const int pw = lane == 0 ? G.L * G.L : lane == 1 ? G.L : 1;
            const int x = i / pw % G.L - G.e, y = j / pw % G.L - G.e, z = k / pw % G.L - G.e;
            const int lo = min(min(x, y), z), hi = max(max(x, y), z);
            s_pts[lane] = lane == 0 ? i : lane == 1 ? j : k;
            s_lo[lane] = lo;
            s_hi[lane] = hi;
            s_n[lane] = live ? axis_partners(lo, hi, G.e, lane ? -G.e : z, s_part[lane]) : 0;
        }
        if (lane == 0) kept = 0u;
    }
    __syncthreads();
    const int i = s_pts[0], nx = s_n[0], ny = s_n[1], nz = s_n[2], total = nx * ny * nz;  // (at most 27)
    if (!total) {
        if (threadIdx.x == 0) run_n[sl] = 0u;
        return;
    }
    const i64 t = (i64)i * N2 + sl % N2;
    auto partner = [&](int cand, int q[3]) {
        const int yz = cand / nz, x = yz / ny;
        q[0] = s_part[0][x];
        q[1] = s_part[1][yz - x * ny];
        q[2] = s_part[2][cand - yz * nz];
        return ((q[0] + G.e) * G.L + q[1] + G.e) * G.L + q[2] + G.e;
    };
    const int cand = threadIdx.x >> 3, m = lane & 7;
    int q[3];
    bool keep = false;
    if (cand < total) {
        const int l = partner(cand, q);
        if (G.omin[l] >= i) {
            int bias[3];
            for (int x = 0; x < 3; ++x) bias[x] = min(s_lo[x], q[x]) + max(s_hi[x], q[x]);
            const int pts[4] = {i, s_pts[1], s_pts[2], l};
            keep = !copy_exists(bias, m) || canonical_copy(G, pts, copy_shift(G, bias, m));
        }
    }
    const unsigned vote = __ballot_sync(0xffffffffu, keep) >> (lane & 24) & 0xffu;
    if (m == 0 && vote == 0xffu) atomicOr(&kept, 1u << cand);  // a partner survives in all its copies
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const unsigned list = kept, n = __popc(list);
    unsigned long long off = 0;
    if (n && lane == 0) off = atomicAdd(&st->used, (unsigned long long)n);
    off = __shfl_sync(0xffffffffu, off, 0);
    const bool fits = off + n <= cap;
    if (lane == 0) {
        run_n[sl] = fits ? n : 0u;
        run_off[sl] = off;
        if (!fits) atomicOr(&st->overflow, 2);
    }
    if (fits && list >> lane & 1u) scratch[off + __popc(list & ((1u << lane) - 1u))] = t * N + partner(lane, q);
}

// collect = false: the count and write passes over the live slots (the
// fallback of a slot with more survivors than a warp's buffer)
template <int KIND>
static i64 enumerate_live(const SymGrid& G, bool collect, EnumStatus* st, int64_t** d_out, int num_sms, cudaStream_t s) {
    const i64 slots = KIND == 0 ? G.N : G.N * G.N * G.N;
    int64_t* out = nullptr;
    // one pass: survivors kept per warp, appended to scratch, placed in slot
    // order; false when they do not fit.  Without slot ids (k_enum_small) the
    // list's length is bounded by 27 partners a slot, so it is placed before the
    // host reads the length (a round trip, 20 us).
    bool clear = true;  // (the status, by k_orbit_min)
    auto one_pass = [&](const int64_t* ids, i64 n, i64* total) {
        const unsigned grid = (unsigned)std::max<i64>(1, std::min<i64>((n + 7) / 8, (i64)num_sms * 16));
        const i64 cap = enum_scratch(G);
        DevBuf<int64_t> scratch(cap, s);
        DevBuf<uint32_t> run_n(n, s);
        DevBuf<unsigned long long> run_off(n, s);
        DevBuf<uint64_t> dest(n, s);
        if (!clear) GLI_CUDA(cudaMemsetAsync(st, 0, sizeof(EnumStatus), s));
        clear = false;
        auto place = [&](i64 entries) {
            GLI_CUDA(cudaMallocAsync((void**)&out, std::max<i64>(entries, 1) * sizeof(int64_t), s));
            k_enum_place<<<grid, 256, 0, s>>>(scratch.p, run_n.p, run_off.p, dest.p, n, out);
            GLI_CHECK_LAUNCH();
        };
        if (ids)
            k_enum_slots_collect<KIND><<<grid, 256, 0, s>>>(G, ids, n, scratch.p, (unsigned long long)cap, run_n.p,
                                                            run_off.p, st);
        else
            k_enum_small<<<(unsigned)n, 256, 0, s>>>(G, n / (G.N * G.N), scratch.p, (unsigned long long)cap, run_n.p,
                                                     run_off.p, st);
        GLI_CHECK_LAUNCH();
        exclusive_scan_u32_dev(run_n.p, dest.p, n, &st->total, s);
        if (!ids) place(27 * n);
        EnumStatus h;
        GLI_CUDA(cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, s));
        GLI_CUDA(cudaStreamSynchronize(s));
        if (h.overflow) {
            if (out) cudaFreeAsync(out, s);
            out = nullptr;
            return false;
        }
        *total = (i64)h.total;
        if (ids) place(*total);
        return true;
    };
    i64 total = 0;
    if (KIND == 1 && collect && G.L <= ENUM_SMALL_L &&
        one_pass(nullptr, (i64)(G.e + 1) * (G.e + 2) * (G.e + 3) / 6 * G.N * G.N, &total)) {
        *d_out = out;
        return total;
    }
    const i64 nb = (slots + 255) / 256;
    DevBuf<uint32_t> bc(nb, s);
    DevBuf<uint64_t> bo(nb, s);
    k_enum_live<KIND, false><<<(unsigned)nb, 256, 0, s>>>(G, slots, bc.p, nullptr, nullptr);
    GLI_CHECK_LAUNCH();
    const i64 nlive = exclusive_scan_u32(bc.p, bo.p, nb, s);
    if (nlive == 0) {
        GLI_CUDA(cudaMallocAsync((void**)&out, sizeof(int64_t), s));
        *d_out = out;
        return 0;
    }
    DevBuf<int64_t> ids(nlive, s);
    k_enum_live<KIND, true><<<(unsigned)nb, 256, 0, s>>>(G, slots, nullptr, bo.p, ids.p);
    GLI_CHECK_LAUNCH();
    if (collect && one_pass(ids.p, nlive, &total)) {
        *d_out = out;
        return total;
    }
    const unsigned grid = (unsigned)std::max<i64>(1, std::min<i64>((nlive + 7) / 8, (i64)num_sms * 16));
    DevBuf<uint32_t> counts(nlive, s);
    DevBuf<uint64_t> offsets(nlive, s);
    k_enum_slots<KIND, false><<<grid, 256, 0, s>>>(G, ids.p, nlive, counts.p, nullptr, nullptr);
    GLI_CHECK_LAUNCH();
    total = exclusive_scan_u32(counts.p, offsets.p, nlive, s);
    GLI_CUDA(cudaMallocAsync((void**)&out, (total > 0 ? total : 1) * sizeof(int64_t), s));
    k_enum_slots<KIND, true><<<grid, 256, 0, s>>>(G, ids.p, nlive, nullptr, offsets.p, out);
    GLI_CHECK_LAUNCH();
    *d_out = out;
    return total;
}

i64 enumerate_device(int kind, const GridDesc& g, int64_t** d_out, cudaStream_t s) {
    const i64 e = symmetric_extent(g);
    if (e < 0) fail(GLI_ERR_ARGUMENT, "specified grid is not rotationally symmetric");
    SymGrid G;
    G.e = (int)e;
    G.L = (int)(2 * e + 1);
    G.N = (i64)G.L * G.L * G.L;
    // (ERI: N^3 slots in blocks of 128, fewer than 2^31 blocks)
    if (kind == 1 && G.L > 17) fail(GLI_ERR_LIMIT, "ERI enumeration supports grids up to 17^3 (got %d^3)", G.L);
    if (kind == 0 && G.L > 1025) fail(GLI_ERR_LIMIT, "ERIDA enumeration supports grids up to 1025^3");
    const i64 slots = kind == 0 ? G.N : G.N * G.N * G.N;
    // For their tests, GLI_B200_ENUM_TWO_PASS selects the thread-per-slot two
    // passes, and the value "live" the count and write passes over the live
    // slots.
    const char* two = getenv("GLI_B200_ENUM_TWO_PASS");
    const bool live_two = two && strcmp(two, "live") == 0;
    if (kind == 0 && !two) return enumerate_erida(G, d_out, s);
    DevBuf<int> omin(G.N, s);
    DevBuf<uint4> images;
    if (kind == 1) images.alloc(6 * G.N, s);
    DevBuf<EnumStatus> st(1, s);
    k_orbit_min<<<(unsigned)((G.N + 31) / 32), 256, 0, s>>>(G, omin.p, images.p, st.p);
    GLI_CHECK_LAUNCH();
    G.omin = omin.p;
    G.images = images.p;
    if (!two || live_two) {
        const int sms = context().num_sms;
        if (kind == 1) return enumerate_live<1>(G, !live_two, st.p, d_out, sms, s);
        return enumerate_live<0>(G, false, st.p, d_out, sms, s);
    }
    DevBuf<uint32_t> counts(slots, s);
    DevBuf<uint64_t> offsets(slots, s);
    const unsigned blocks = (unsigned)((slots + 127) / 128);
    if (kind == 0)
        k_enum_erida<false><<<blocks, 128, 0, s>>>(G, counts.p, nullptr, nullptr);
    else
        k_enum_eri<false><<<blocks, 128, 0, s>>>(G, counts.p, nullptr, nullptr);
    GLI_CHECK_LAUNCH();
    const i64 total = exclusive_scan_u32(counts.p, offsets.p, slots, s);
    int64_t* out = nullptr;
    GLI_CUDA(cudaMallocAsync((void**)&out, (total > 0 ? total : 1) * sizeof(int64_t), s));
    if (kind == 0)
        k_enum_erida<true><<<blocks, 128, 0, s>>>(G, nullptr, offsets.p, out);
    else
        k_enum_eri<true><<<blocks, 128, 0, s>>>(G, nullptr, offsets.p, out);
    GLI_CHECK_LAUNCH();
    *d_out = out;
    return total;
}

}  // namespace gli
