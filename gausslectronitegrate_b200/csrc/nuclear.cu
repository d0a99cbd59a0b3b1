// Nuclear-attraction integrals, reference src/nuclear_integrals.c:16-24 (the
// Gaussian-nucleus kernel erf(r/w)/r, w = 1/3), :31-126 (single entry) and
// :133-266 (matrix).
//
// The reference evaluates, per orbital pair (i, j),
//   V_ij = sum_{x,y,z} Fx[x] Fy[y] Fz[z] sum_k Z_k g(|p - R_k|),
//   p_a = (i_a + j_a)/2 + m_a/6,
// one erf per (primitive point, nucleus).  Every primitive point lies on the
// 1/6 lattice, so the nuclear field is tabulated once on the lattice box that
// the grid's primitives cover,
//   Phi[u][v][t] = sum_k Z_k g(|(u,v,t)/6 + origin - R_k|),
// and the separable weights are contracted against it axis by axis:
//   A   H[kz][u][v]     = sum_t Wz[kz][t] Phi[u][v][t]      (GEMM)
//   B   H2[ky][kz][u]   = sum_v Wy[ky][v] H[kz][u][v]       (batched GEMM)
//   C   Vk[kx][ky,kz]   = sum_u Wx[kx][u] H2[ky][kz][u]     (GEMM)
// where an axis key is the unordered coordinate pair {i_a, j_a} (the factor
// depends on |i_a - j_a|, the position on i_a + j_a).  A final scatter writes
// the dense N x N matrix, V_ij = Vk[kx(i,j)][ky(i,j), kz(i,j)] (the sliced
// tensor-core contractions keep the (kz, ky) order of their batched stage B).
//
// Band.  A key's weights are nonzero on the 2 mmax + 1 positions around
// 3 (i_a + j_a) only (mmax: the outermost factor above tol; 99 of 237 positions
// on a 24-point axis at tol 1e-8).  Keys are therefore ordered by i_a + j_a, so
// that the 64 keys of a tile share most of their positions, and a tile's K loop
// covers just the positions that any of its keys reaches.  Keys whose factor is
// below tol throughout (|i_a - j_a| from 17 at tol 1e-8) are no keys at all:
// their matrix entries are zero.
//
// Batches.  Any number of instances (each its own grid and nuclei, all with
// the same coefficients and tol) run as one plan: one upload of every
// instance's descriptor, coordinates and nuclei; per pipeline one kernel builds
// every instance's weights, one tabulates every instance's field, three
// contract (every instance's tiles in one launch per stage) and one scatters
// every instance's matrix.  The autotuner chooses how many pipelines (streams)
// the instances of a chunk are dealt over.  (One launch per instance and stage,
// captured as a graph on each call, spent more on the capture, on launches under
// a wave and on their tails than it saved: 200 us of host time per call for one
// 13 x 16 x 11 instance.)  Forms: FP64 throughout (the drop-in), or mixed: the
// three contractions as int8-sliced products on the tensor cores (5 slices),
// field, weights and scatter in FP64, where the autotuner measures that faster.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <string>

#include "autotune.cuh"
#include "dmma.cuh"
#include "gli_internal.cuh"
#include "tc_gemm.cuh"

namespace gli {

// masks F at tol; reach[0] = largest |m|, reach[1] = largest s of an entry above tol
__global__ void k_mask_factors(double* __restrict__ F, i64 n, int nf, int nb, double tol, int* __restrict__ reach) {
    const i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    double v = F[e];
    if (!(fabs(v) > tol)) v = 0;
    F[e] = v;
    if (v != 0) {
        const int m = (int)(e % nf) - (nb - 1);
        atomicMax(&reach[0], m < 0 ? -m : m);
        atomicMax(&reach[1], (int)(e / nf));
    }
}

// device descriptor of one instance
struct NucInst {
    int n[3];          // axis lengths
    int coord_off[3];  // first coordinate of each axis in the packed coordinate list
    int U[3], u0[3];   // lattice extent and origin (units of 1/6) per axis
    int P[3];          // U rounded up to even: row pitches (16-byte rows)
    int nk[3];         // axis keys: pairs lo <= hi whose factor is not zero throughout
    int rk_off[3];     // n x n table: key of (i, j), NUC_DEAD where the factor is zero
    int key_off[3];    // lo | hi << 8 of each key
    int band;          // weights per key (2 mmax + 1); 0: the keys' order is not by position
    int nuc0, nnuc;    // nuclei in the packed nucleus arrays
    i64 N;             // grid points
    i64 w_off[3];      // weights of each axis in the packed W buffer (even)
    int ks_off[3];     // first position of each key in the packed start list
    i64 x_off;         // the field; the key-indexed matrix overwrites it (even)
    i64 h_off;         // the stage-A product H (even)
    i64 h2_off;        // the stage-B product H2 (even)
    double* out;       // N x N row-major
};

constexpr uint16_t NUC_DEAD = 0xffff;

// W[key][u] of every (instance, axis), u a lattice position (zeros up to the
// pitch), and the first position of each key.  grid (u blocks, key, 3 * instance)
__global__ void k_nuc_weights(const NucInst* __restrict__ inst, const double* __restrict__ F, int nf, int nb,
                              const int* __restrict__ coords, const uint16_t* __restrict__ tables,
                              double* __restrict__ W, int* __restrict__ kstart) {
    const NucInst& in = inst[blockIdx.z / 3];
    const int a = blockIdx.z % 3;
    const int key = blockIdx.y;
    if (key >= in.nk[a]) return;
    const int lohi = tables[in.key_off[a] + key], lo = lohi & 0xff, hi = lohi >> 8;
    const int xa = coords[in.coord_off[a] + lo], xb = coords[in.coord_off[a] + hi];
    const int s = xa > xb ? xa - xb : xb - xa;
    const int U = in.U[a], P = in.P[a];
    double* w = W + in.w_off[a] + (i64)key * P;
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < P; u += gridDim.x * blockDim.x) {
        const int m = u + in.u0[a] - 3 * (xa + xb);  // factor logical index
        double v = 0;
        if (u < U && m >= -(nb - 1) && m <= nb - 1) v = F[(i64)s * nf + m + (nb - 1)];
        w[u] = v;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        kstart[in.ks_off[a] + key] = 3 * (xa + xb) - 6 * coords[in.coord_off[a]];
}

// the Gaussian-nucleus field g(r) = erf(r / w) / r with w = 1/3 at squared
// distance r2; g(0) = 2 / (sqrt(pi) w).  For 3 r >= 6, erfc(3 r) <= 2.2e-17 is
// below a quarter ulp of 1: erf rounds to 1 and g = 1 / r
__device__ __forceinline__ double nuc_gaussian(double r2) {
    if (r2 >= 4.0) return rsqrt(r2);
    const double r = sqrt(r2);
    return r > 0 ? erf(3.0 * r) / r : 3.3851375012865379;  // 6 / sqrt(pi)
}

// Phi[u][v][t] (t fastest, pitches P) of every instance, position
// (u + u0x, v + u0y, t + u0z) / 6; grid (row blocks, instance), a warp fills
// whole (u, v) rows, up to eight cells per lane and turn: per nucleus the row's part of
// the squared distance is formed once and each cell costs two FP64
// multiply-adds and a reciprocal square root.  Bound: the issue slots (64% busy,
// the FP64 pipe 41%).  13 x 16 x 11 points and 5 nuclei, 171 x 189 x 159 cells:
// 45 us; the batch of eight, 24^3 to 8^3, 376 us (71%, 49%), 722 us with a thread
// per cell, its coordinates divided by 6 and its whole distance per nucleus.
constexpr int NUC_FIELD_MAX_T = 2048;  // z positions held in shared memory (axes of 256 points: 1531 + 2 mmax)
constexpr int NUC_FIELD_BLOCKS = 3;     // per SM
__global__ void __launch_bounds__(256, NUC_FIELD_BLOCKS) k_nuc_field(const NucInst* __restrict__ inst, const double* __restrict__ npos,
                                                   const double* __restrict__ ncharge, double* __restrict__ X) {
    __shared__ double zs[NUC_FIELD_MAX_T];
    const NucInst& in = inst[blockIdx.y];
    const int Py = in.P[1], Pz = in.P[2], lane = threadIdx.x & 31;
    const int rows = in.P[0] * Py, warps = gridDim.x * (blockDim.x >> 5);
    for (int t = threadIdx.x; t < Pz && t < NUC_FIELD_MAX_T; t += blockDim.x) zs[t] = (t + in.u0[2]) / 6.0;
    __syncthreads();
    for (int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); row < rows; row += warps) {
        const int u = row / Py, v = row - u * Py;
        const double px = (u + in.u0[0]) / 6.0, py = (v + in.u0[1]) / 6.0;
        double* phi = X + in.x_off + (i64)row * Pz;
        auto zs_at = [&](int t) { return t < NUC_FIELD_MAX_T ? zs[t < Pz ? t : 0] : (t + in.u0[2]) / 6.0; };
        auto cells = [&](auto count, int t0) {
            constexpr int C = decltype(count)::value;
            double pz[C], acc[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int t = t0 + 32 * c + lane;
                pz[c] = zs_at(t);
                acc[c] = 0.0;
            }
            for (int k = in.nuc0; k < in.nuc0 + in.nnuc; ++k) {
                const double dx = px - npos[3 * k], dy = py - npos[3 * k + 1], nz = npos[3 * k + 2], q = ncharge[k];
                const double r2 = dx * dx + dy * dy;
                // (a whole row that has no cell near the nucleus: g = 1 / r throughout)
                if (r2 >= 4.0 && !isnan(nz)) {
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        const double dz = pz[c] - nz;
                        acc[c] += q * rsqrt(r2 + dz * dz);
                    }
                } else {
#pragma unroll 1
                    for (int c = 0; c < C; ++c) {
                        const double dz = zs_at(t0 + 32 * c + lane) - nz, g = q * nuc_gaussian(r2 + dz * dz);
#pragma unroll
                        for (int e = 0; e < C; ++e)
                            if (e == c) acc[e] += g;
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int t = t0 + 32 * c + lane;
                if (t < Pz) phi[t] = acc[c];
            }
        };
        // the row's 32-cell pieces in turns of equal width, at most eight
        const int pieces = (Pz + 31) >> 5, turns = (pieces + 7) >> 3, width = (pieces + turns - 1) / turns;
        for (int t0 = 0; t0 < Pz; t0 += 32 * width) {
            switch (width) {
                case 8: cells(std::integral_constant<int, 8>{}, t0); break;
                case 7: cells(std::integral_constant<int, 7>{}, t0); break;
                case 6: cells(std::integral_constant<int, 6>{}, t0); break;
                case 5: cells(std::integral_constant<int, 5>{}, t0); break;
                case 4: cells(std::integral_constant<int, 4>{}, t0); break;
                default: cells(std::integral_constant<int, 3>{}, t0);
            }
        }
    }
}

// V[i][j] of every instance from its key-indexed block: Vk[kx][ky * nkz + kz]
// (zfast: the FP64 contractions) or Vk[kx][kz * nky + ky] (the sliced ones).
//
// zfast: item (iy, ix <= jx) writes the nz x (ny nz) sub-blocks of rows
// (ix, iy, .) and columns (jx, ., .) and of rows (jx, iy, .) and columns
// (ix, ., .), which hold the same values.  They lie in the ny lines
// ky = key(iy, jy) of the slice kx = key(ix, jx).  A few lines at a time are read
// (coalesced) and laid out in shared memory as the output's rows, each value
// at (lo, hi) and (hi, lo), then copied out row by row in 16-byte stores.
// Bound: HBM writes.  Batch of eight, 24^3 to 8^3 (2.67 GB): 868 us with a
// thread per column, 8-byte stores and every value gathered from its line in
// L1; 778 us gathering it from the line in shared memory; 934 us with two
// buffers filled by 8-byte cp.async (two copies per value).
constexpr int NUC_LINE_MAX_Z = 64;         // z axis of the shared-memory route
constexpr int NUC_ROWS_BYTES = 44 * 1024;  // output rows held at a time: five blocks on an SM

// lines (jy) held at a time, and the row pitch in doubles (6 mod 16: the values
// of neighbouring keys, on falling diagonals of the square, fall in different banks)
__host__ __device__ __forceinline__ int nuc_row_pitch(int group, int nz) { return (group * nz + 9) / 16 * 16 + 6; }
__host__ __device__ __forceinline__ int nuc_line_group(int ny, int nz) {
    int cap = NUC_ROWS_BYTES / (8 * nz * nz);
    while (cap > 1 && 8 * nz * nuc_row_pitch(cap, nz) > NUC_ROWS_BYTES) --cap;
    if (cap < 1) cap = 1;
    const int turns = (ny + cap - 1) / cap;
    return (ny + turns - 1) / turns;
}

__global__ void __launch_bounds__(256) k_nuc_scatter(const NucInst* __restrict__ inst, const double* __restrict__ X,
                                                     const uint16_t* __restrict__ tables, int zfast) {
    extern __shared__ __align__(16) double rows[];
    const NucInst& in = inst[blockIdx.y];
    const int nx = in.n[0], ny = in.n[1], nz = in.n[2], nky = in.nk[1], nkz = in.nk[2];
    const int nyz = ny * nz;
    const i64 N = in.N;
    const double* Vk = X + in.x_off;
    const uint16_t *rx = tables + in.rk_off[0], *ry = tables + in.rk_off[1], *rz = tables + in.rk_off[2];
    if (zfast && nz <= NUC_LINE_MAX_Z) {
        const int items = nx * (nx + 1) / 2 * ny;
        if ((int)blockIdx.x >= items) return;
        const int group = nuc_line_group(ny, nz), pitch = nuc_row_pitch(group, nz);
        const uint16_t* keys = tables + in.key_off[2];
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
        // (the entries of zero factors are never written below)
        for (int e = threadIdx.x; e < nz * pitch; e += blockDim.x) rows[e] = 0.0;
        for (int item = blockIdx.x; item < items; item += gridDim.x) {
            // (iy, ix <= jx): the sub-blocks (ix, iy, jx) and (jx, iy, ix) hold the same values
            const int iy = item % ny, xp = item / ny;
            int jx = (int)((sqrtf(8.0f * xp + 1.0f) - 1.0f) * 0.5f);
            while ((jx + 1) * (jx + 2) / 2 <= xp) ++jx;
            while (jx * (jx + 1) / 2 > xp) --jx;
            const int ix = xp - jx * (jx + 1) / 2;
            const int kx = rx[ix * nx + jx];
            const double* slice = Vk + (i64)kx * ((i64)nky * nkz);
            for (int j0 = 0; j0 < ny; j0 += group) {
                const int cnt = min(group, ny - j0), cols = cnt * nz;
                __syncthreads();  // the rows before are copied out
                for (int l = warp; l < cnt; l += warps) {
                    const int ky = kx == NUC_DEAD ? NUC_DEAD : ry[iy * ny + j0 + l];
                    const bool live = ky != NUC_DEAD;
                    const double* src = slice + (live ? (i64)ky * nkz : 0);
                    double* dst = rows + l * nz;
                    constexpr int V = 5;
                    for (int e0 = lane; e0 < nkz; e0 += 32 * V) {
                        double v[V];
                        int k[V];
#pragma unroll
                        for (int u = 0; u < V; ++u) {
                            const int e = e0 + 32 * u;
                            v[u] = live && e < nkz ? __ldg(src + e) : 0.0;
                            k[u] = e < nkz ? __ldg(keys + e) : 0;
                        }
#pragma unroll
                        for (int u = 0; u < V; ++u)
                            if (e0 + 32 * u < nkz) {
                                const int lo = k[u] & 0xff, hi = k[u] >> 8;
                                dst[lo * pitch + hi] = v[u];
                                dst[hi * pitch + lo] = v[u];
                            }
                    }
                }
                __syncthreads();
                double* const block0 = in.out + (i64)(ix * ny + iy) * nz * N + (i64)jx * nyz + (i64)j0 * nz;
                double* const block1 = in.out + (i64)(jx * ny + iy) * nz * N + (i64)ix * nyz + (i64)j0 * nz;
                const int nrows = ix == jx ? nz : 2 * nz;
                for (int r = warp; r < nrows; r += warps) {
                    const int iz = r < nz ? r : r - nz;
                    double* out = (r < nz ? block0 : block1) + (i64)iz * N;
                    const double* row = rows + iz * pitch;
                    // (pairs start on 16-byte boundaries: an odd start leaves its first entry alone)
                    const int odd = (int)(((uintptr_t)out >> 3) & 1);
                    if (odd) {
                        if (lane == 0) __stcs(out, row[0]);
                        for (int c = 1 + 2 * lane; c + 1 < cols; c += 64)
                            __stcs(reinterpret_cast<double2*>(out + c), make_double2(row[c], row[c + 1]));
                    } else {
                        for (int c = 2 * lane; c + 1 < cols; c += 64)
                            __stcs(reinterpret_cast<double2*>(out + c), *reinterpret_cast<const double2*>(row + c));
                    }
                    if (((cols - odd) & 1) && lane == 0 && cols > odd) __stcs(out + cols - 1, row[cols - 1]);
                }
            }
        }
        return;
    }
    // other layouts and long z axes: a thread per column, rows as (iy, iz) loops
    const i64 sy = zfast ? nkz : 1, sz = zfast ? 1 : nky;  // strides of ky and kz in a slice
    for (int pair = blockIdx.x; pair < nx * nx; pair += gridDim.x) {
        const int ix = pair / nx, jx = pair - ix * nx, kx = rx[ix * nx + jx];
        const double* slice = Vk + (i64)kx * ((i64)nky * nkz);
        double* block = in.out + (i64)ix * nyz * N + (i64)jx * nyz;
        for (int c = threadIdx.x; c < nyz; c += blockDim.x) {
            const int jy = c / nz, jz = c - jy * nz;
            double* col = block + c;
            for (int iy = 0; iy < ny; ++iy) {
                const int ky = kx == NUC_DEAD ? NUC_DEAD : ry[iy * ny + jy];
                double* out = col + (i64)iy * nz * N;
                for (int iz = 0; iz < nz; ++iz) {
                    const int kz = ky == NUC_DEAD ? NUC_DEAD : rz[iz * nz + jz];
                    out[(i64)iz * N] = kz == NUC_DEAD ? 0.0 : slice[ky * sy + kz * sz];
                }
            }
        }
    }
}

// One stage of the FP64 contractions over every instance of a pipeline:
// Y[m][n] = sum_k W[m][k] X[n][k], m a key of the stage's axis, n the rows of
//   A  X = Phi, n = (u, v) with pitch P1:   Y = H[kz][n]
//   B  X = H,   n = (kz, u) with pitch P0:  Y = H2[ky][n]
//   C  X = H2,  n = (ky, kz):               Y = Vk[kx][n]
// (row pitches make each stage's output the next one's rows as they are; the
// rows past an axis' extent hold finite values that no later K range reads).
// Blocks find their instance in `pre`, the tiles before each instance; the key
// tiles of one n tile are neighbours, so X comes from L2 after the first.  K
// runs over the positions from the tile's first key's to its last key's last
// one, both operands K-contiguous 16-byte copies, and an 8-key strip takes part
// only in the chunks it reaches.
//
// Bound: the FP64 tensor pipe, 75% busy on the batch of eight, 24^3 to 8^3,
// whose three stages take 381 + 348 + 345 us; 2.95 ms over full K ranges with
// 8-byte copies, a launch per instance.
template <int STAGE>
struct NucStageOp {
    static constexpr bool A_KMAJOR = false, B_KMAJOR = false;
    static constexpr int BN = DM_BN;
    // (short K ranges: a fourth block per SM covers the blocks' starts and ends
    // better than a third pipeline stage, 5% on each stage; 32-column tiles at
    // six blocks 4% slower)
    static constexpr int STAGES = 2, MIN_BLOCKS = 4;
    static constexpr int SKIP = SKIP_M;
    static constexpr int AXIS = 2 - STAGE;
    const NucInst* inst;
    const int* pre;  // ni + 1 tile counts
    int ni;
    const double* W;
    const int* kstart;
    double* Xb;  // packed buffers
    double* Hb;
    double* H2b;
    struct Block {
        int mvalid, nvalid, nk;
        int k0, kend;
        int pitch;
        int first, last;  // positions that strip (lane & 7) reaches
        i64 ldy;
        const double* a;
        const double* b;
        double* y;
    };
    struct AState {
        const uint16_t* live;
    };
    struct BState {};
    __device__ bool begin(Block& b) const {
        // the instance: the last one whose tiles start at or before this block
        int lo = 0, hi = ni;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(&pre[mid]) <= (int)blockIdx.x) lo = mid;
            else hi = mid;
        }
        const NucInst& in = inst[lo];
        const int t = (int)blockIdx.x - __ldg(&pre[lo]);
        const int M = in.nk[AXIS], mt = (M + DM_BM - 1) / DM_BM;
        const int m0 = t % mt * DM_BM, n0 = t / mt * BN;
        const int rows = STAGE == 0 ? in.P[0] * in.P[1] : STAGE == 1 ? in.nk[2] * in.P[0] : in.nk[1] * in.nk[2];
        b.mvalid = min(DM_BM, M - m0);
        b.nvalid = min(BN, rows - n0);
        b.pitch = in.P[AXIS];
        b.kend = in.U[AXIS];
        // the positions that each 8-key strip reaches (its first key's first to
        // its last key's last), a strip per lane; empty strips reach none
        const int strip = threadIdx.x & 7, r0 = 8 * strip;
        b.first = 0;
        b.last = r0 < b.mvalid ? b.kend - 1 : -1;
        if (in.band && r0 < b.mvalid) {
            const int* ks = kstart + in.ks_off[AXIS] + m0;
            b.first = __ldg(&ks[r0]);
            b.last = min(b.kend, __ldg(&ks[min(r0 + 7, b.mvalid - 1)]) + in.band) - 1;
        }
        b.k0 = __shfl_sync(0xffffffffu, b.first, 0) & ~3;
        b.kend = __reduce_max_sync(0xffffffffu, b.last) + 1;
        b.nk = (b.kend - b.k0 + DM_BK - 1) / DM_BK;
        b.ldy = rows;
        const double* x = STAGE == 0 ? Xb + in.x_off : STAGE == 1 ? Hb + in.h_off : H2b + in.h2_off;
        double* y = STAGE == 0 ? Hb + in.h_off : STAGE == 1 ? H2b + in.h2_off : Xb + in.x_off;
        b.a = W + in.w_off[AXIS] + (i64)m0 * b.pitch + b.k0;
        b.b = x + (i64)n0 * b.pitch + b.k0;
        b.y = y + (i64)m0 * b.ldy + n0;
        return true;
    }
    __device__ void live_chunks(const Block& b, int, int& first, int& last) const {
        first = (b.first - b.k0) / DM_BK;  // (thread t asks for strip t)
        last = b.last < b.first ? -1 : (b.last - b.k0) / DM_BK;
    }
    __device__ void a_init(const Block&, AState&) const {}
    __device__ void b_init(const Block&, BState&) const {}
    __device__ void a_issue(const Block& b, AState& st, int kc, double* tile) const {
        const unsigned live = st.live[dm_run_entry(kc)];
#pragma unroll
        for (int q = 0; q < DM_BM / 16; ++q) {
            if (!dm_live(live, q)) continue;
            const int r = dm_pair_row(threadIdx.x, q), k = dm_pair_k(threadIdx.x), kk = kc * DM_BK + k;
            const int bytes = r < b.mvalid ? dm_pair_bytes(b.k0 + kk, b.kend) : 0;
            dm_cp16(tile + dm_rowmajor_at(r, k), bytes ? b.a + r * b.pitch + kk : b.a, bytes);
        }
    }
    __device__ void b_issue(const Block& b, BState&, int kc, double* tile) const {
#pragma unroll
        for (int q = 0; q < BN / 16; ++q) {
            const int r = dm_pair_row(threadIdx.x, q), k = dm_pair_k(threadIdx.x), kk = kc * DM_BK + k;
            const int bytes = r < b.nvalid ? dm_pair_bytes(b.k0 + kk, b.kend) : 0;
            dm_cp16(tile + dm_rowmajor_at(r, k), bytes ? b.b + r * b.pitch + kk : b.b, bytes);
        }
    }
    __device__ void store(const Block& b, int m, int n, double v0, double v1) const {
        if (m >= b.mvalid) return;
        double* y = b.y + m * b.ldy + n;
        if (n + 1 < b.nvalid && !(b.ldy & 1)) {
            *reinterpret_cast<double2*>(y) = make_double2(v0, v1);
        } else {
            if (n < b.nvalid) y[0] = v0;
            if (n + 1 < b.nvalid) y[1] = v1;
        }
    }
};

// tiles of a shared-B batched product: batch b, B row block j of nbt
__global__ void k_shared_b_tiles(int batches, int nbt, int nrows, int bn, int* __restrict__ tb, int* __restrict__ tc,
                                 int* __restrict__ tn, int* __restrict__ tbb) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= batches * nbt) return;
    const int b = t / nbt, j = t % nbt;
    tb[t] = b;
    tc[t] = b * nrows + j * bn;
    tn[t] = min(bn, nrows - j * bn);
    tbb[t] = j;
}

// rows r = b * rows + i of a batched dense matrix, each batch padded to whole
// 128-row tiles
struct BatchedRows {
    const double* src;
    i64 ld;
    int rows, blocks;
    __device__ RowBase row(i64 r) const { return {src + r * ld}; }
    __device__ double at(const RowBase& c, int k) const { return c.p[k]; }
    __device__ i64 dest(i64 r) const { return (r / rows) * blocks * TC_BM + r % rows; }
    __device__ i64 source(i64 d, i64 total) const {
        const i64 b = d / ((i64)blocks * TC_BM), i = d % ((i64)blocks * TC_BM);
        return (i < rows && b * rows + i < total) ? b * rows + i : -1;
    }
    __device__ bool valid(i64) const { return true; }
};

// host copy of an instance
struct NucHost {
    NucInst d;
};

// doubles of an instance's packed buffers (even): the field and, later, the
// key-indexed matrix in one; the two intermediate products
static i64 nuc_even(i64 n) { return (n + 1) & ~(i64)1; }
static i64 nuc_x_size(const NucInst& in) {
    return nuc_even(std::max((i64)in.P[0] * in.P[1] * in.P[2], (i64)in.nk[0] * in.nk[1] * in.nk[2]));
}
static i64 nuc_h_size(const NucInst& in) { return nuc_even((i64)in.nk[2] * in.P[0] * in.P[1]); }
static i64 nuc_h2_size(const NucInst& in) { return nuc_even((i64)in.nk[1] * in.nk[2] * in.P[0]); }

static void nuc_contract_mixed(const NucInst& in, const double* W, double* X, double* Hb, double* H2b, int* err,
                               cudaStream_t s) {
    constexpr int S = MIXED_SLICES, BN = tile_n(MIXED_SLICES);
    const int* U = in.U;
    const int* P = in.P;
    const double* Phi = X + in.x_off;
    double *Vk = X + in.x_off, *H = Hb + in.h_off, *H2 = H2b + in.h2_off;
    const int* nk = in.nk;
    const i64 UxUy = (i64)P[0] * P[1], nzy = (i64)nk[2] * nk[1];
    const double* Wx = W + in.w_off[0];
    const double* Wy = W + in.w_off[1];
    const double* Wz = W + in.w_off[2];
    {   // A: rows (u v) of the field against the z keys
        TiledSlices As, Bs;
        const i64 mb = (UxUy + TC_BM - 1) / TC_BM, nbt = (nk[2] + BN - 1) / BN;
        As.alloc(mb, TC_BM, U[2], S, s);
        slice_tiled(DenseRows{Phi, P[2]}, UxUy, U[2], As, s);
        Bs.alloc(nbt, BN, U[2], S, s);
        slice_tiled(DenseRows{Wz, P[2]}, nk[2], U[2], Bs, s);
        TileWork w;
        w.a_rows = (int)UxUy;
        w.a_blocks = (int)mb;
        w.n_total = nk[2];
        w.C = H;
        w.rs = 1;
        w.cs = UxUy;
        tc_gemm_tiled(As.view(), Bs.view(), w, (int)nbt, err, s);
    }
    {   // B: batch kz, rows u of H[kz] (K = v) against the y keys (shared by every batch)
        TiledSlices As, Bs;
        const int mb = (P[0] + TC_BM - 1) / TC_BM, nbt = (nk[1] + BN - 1) / BN;
        As.alloc((i64)nk[2] * mb, TC_BM, U[1], S, s);
        slice_tiled(BatchedRows{H, P[1], P[0], mb}, (i64)nk[2] * P[0], U[1], As, s);
        Bs.alloc(nbt, BN, U[1], S, s);
        slice_tiled(DenseRows{Wy, P[1]}, nk[1], U[1], Bs, s);
        const int ntiles = nk[2] * nbt;
        DevBuf<int> tiles(4 * (i64)ntiles, s);
        k_shared_b_tiles<<<(ntiles + 255) / 256, 256, 0, s>>>(nk[2], nbt, nk[1], BN, tiles.p, tiles.p + ntiles,
                                                              tiles.p + 2 * ntiles, tiles.p + 3 * ntiles);
        GLI_CHECK_LAUNCH();
        TileWork w;
        w.a_rows = P[0];
        w.a_blocks = mb;
        w.a_batched = 1;
        w.tile_batch = tiles.p;
        w.tile_col0 = tiles.p + ntiles;
        w.tile_ncols = tiles.p + 2 * ntiles;
        w.tile_bblock = tiles.p + 3 * ntiles;
        w.C = H2;
        w.rs = 1;
        w.cs = P[0];
        tc_gemm_tiled(As.view(), Bs.view(), w, ntiles, err, s);
    }
    {   // C: rows (kz ky) of H2 (K = u) against the x keys
        TiledSlices As, Bs;
        const i64 mb = (nzy + TC_BM - 1) / TC_BM, nbt = (nk[0] + BN - 1) / BN;
        As.alloc(mb, TC_BM, U[0], S, s);
        slice_tiled(DenseRows{H2, P[0]}, nzy, U[0], As, s);
        Bs.alloc(nbt, BN, U[0], S, s);
        slice_tiled(DenseRows{Wx, P[0]}, nk[0], U[0], Bs, s);
        TileWork w;
        w.a_rows = (int)nzy;
        w.a_blocks = (int)mb;
        w.n_total = nk[0];
        w.C = Vk;
        w.rs = 1;
        w.cs = nzy;
        tc_gemm_tiled(As.view(), Bs.view(), w, (int)nbt, err, s);
    }
}

// streams of the per-instance contractions (per thread and device)
struct StreamRing {
    int device = -1;
    std::vector<cudaStream_t> streams;
    std::vector<cudaEvent_t> events;
    void ensure(int dev, int n) {
        if (device != dev) {
            streams.clear();
            events.clear();
            device = dev;
        }
        while ((int)streams.size() < n) {
            cudaStream_t st;
            cudaEvent_t ev;
            GLI_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
            GLI_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
            streams.push_back(st);
            events.push_back(ev);
        }
    }
};
static thread_local StreamRing t_ring;
static thread_local cudaEvent_t t_fork = nullptr;
static thread_local int t_fork_dev = -1;

// streams and the fork event exist before any capture starts
static void ensure_streams(int device, int n) {
    if (t_fork_dev != device) {
        GLI_CUDA(cudaEventCreateWithFlags(&t_fork, cudaEventDisableTiming));
        t_fork_dev = device;
    }
    t_ring.ensure(device, n);
}

static_assert(8 * NUC_LINE_MAX_Z * ((NUC_LINE_MAX_Z + 9) / 16 * 16 + 6) <= NUC_ROWS_BYTES, "a line of the longest z axis fits");

// kernel attributes: shared memory above the 48 KB default
static void nuc_prepare() {
    GLI_CUDA(cudaFuncSetAttribute(k_nuc_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, NUC_ROWS_BYTES));
}

// Queues one chunk of instances, dealt over `pipes` pipelines (largest first,
// round robin; one pipeline: stream s itself, else forked streams): per
// pipeline the weights, the field, the three contractions (int8-sliced
// tensor-core products per instance when `sliced`, else one FP64 tensor-core
// launch per stage) and the scatter.
static void run_chunk(const std::vector<NucHost>& hosts, const double* F, int nf, int nb, const int* coords,
                      const double* npos, const double* ncharge, const uint16_t* tables, bool sliced, int pipes, int num_sms,
                      int* err, cudaStream_t s) {
    const int ni = (int)hosts.size();
    pipes = std::min(pipes, ni);
    std::vector<int> order(ni);
    for (int k = 0; k < ni; ++k) order[k] = k;
    std::sort(order.begin(), order.end(), [&](int a, int b) { return hosts[a].d.N > hosts[b].d.N; });
    // descriptors pipeline by pipeline, then the tiles before each instance per stage
    const size_t dbytes = ni * sizeof(NucInst);
    std::vector<char> up(dbytes + 3 * (size_t)(ni + pipes) * sizeof(int));
    NucInst* desc = reinterpret_cast<NucInst*>(up.data());
    int* pre = reinterpret_cast<int*>(up.data() + dbytes);
    std::vector<int> first(pipes + 1, 0);
    i64 w_total = 0, x_total = 0, h_total = 0, h2_total = 0, ks_total = 0;
    int at = 0;
    for (int p = 0; p < pipes; ++p) {
        first[p] = at;
        for (int k = p; k < ni; k += pipes) desc[at++] = hosts[order[k]].d;
        const int cnt = at - first[p];
        for (int st = 0; st < 3; ++st) {
            int* pr = pre + st * (ni + pipes) + first[p] + p;
            i64 t = 0;
            for (int k = 0; k <= cnt; ++k) {
                if (t >= ((i64)1 << 31)) fail(GLI_ERR_LIMIT, "too many nuclear contraction tiles in one chunk");
                pr[k] = (int)t;
                if (k == cnt) break;
                const NucInst& in = desc[first[p] + k];
                const i64 rows = st == 0 ? (i64)in.P[0] * in.P[1] : st == 1 ? (i64)in.nk[2] * in.P[0] : (i64)in.nk[1] * in.nk[2];
                t += (i64)((in.nk[2 - st] + DM_BM - 1) / DM_BM) * ((rows + DM_BN - 1) / DM_BN);
            }
        }
    }
    first[pipes] = at;
    for (const NucHost& h : hosts) {
        for (int a = 0; a < 3; ++a) {
            w_total = std::max(w_total, h.d.w_off[a] + (i64)h.d.nk[a] * h.d.P[a]);
            ks_total = std::max<i64>(ks_total, h.d.ks_off[a] + h.d.nk[a]);
        }
        x_total = std::max(x_total, h.d.x_off + nuc_x_size(h.d));
        h_total = std::max(h_total, h.d.h_off + nuc_h_size(h.d));
        h2_total = std::max(h2_total, h.d.h2_off + nuc_h2_size(h.d));
    }
    DevBuf<char> d_up(up.size(), s);
    DevBuf<double> W(w_total, s), X(x_total, s), H(h_total, s), H2(h2_total, s);
    DevBuf<int> ks(ks_total, s);
    GLI_CUDA(cudaMemcpyAsync(d_up.p, up.data(), up.size(), cudaMemcpyHostToDevice, s));
    const NucInst* d_inst = reinterpret_cast<const NucInst*>(d_up.p);
    const int* d_pre = reinterpret_cast<const int*>(d_up.p + dbytes);
    if (pipes > 1) {
        GLI_CUDA(cudaEventRecord(t_fork, s));
        for (int p = 0; p < pipes; ++p) GLI_CUDA(cudaStreamWaitEvent(t_ring.streams[p], t_fork, 0));
    }
    for (int p = 0; p < pipes; ++p) {
        cudaStream_t st = pipes > 1 ? t_ring.streams[p] : s;
        const int i0 = first[p], cnt = first[p + 1] - i0;
        const NucInst* di = d_inst + i0;
        int max_nk = 1, max_p = 1;
        i64 max_rows = 1, max_items = 1;
        int lines = 0;
        for (int k = i0; k < i0 + cnt; ++k) {
            const NucInst& in = desc[k];
            for (int a = 0; a < 3; ++a) {
                max_nk = std::max(max_nk, in.nk[a]);
                max_p = std::max(max_p, in.P[a]);
            }
            max_rows = std::max(max_rows, (i64)in.P[0] * in.P[1]);
            const bool by_lines = !sliced && in.n[2] <= NUC_LINE_MAX_Z;
            max_items = std::max(max_items, by_lines ? (i64)in.n[0] * (in.n[0] + 1) / 2 * in.n[1] : (i64)in.n[0] * in.n[0]);
            if (by_lines) {
                lines = std::max(lines, 8 * in.n[2] * nuc_row_pitch(nuc_line_group(in.n[1], in.n[2]), in.n[2]));
            }
        }
        k_nuc_weights<<<dim3((unsigned)((max_p + 127) / 128), (unsigned)max_nk, (unsigned)(3 * cnt)), 128, 0, st>>>(
            di, F, nf, nb, coords, tables, W.p, ks.p);
        GLI_CHECK_LAUNCH();
        const unsigned fb = (unsigned)std::min<i64>((max_rows + 7) / 8, std::max<i64>(1, (i64)num_sms * NUC_FIELD_BLOCKS));
        k_nuc_field<<<dim3(fb, (unsigned)cnt), 256, 0, st>>>(di, npos, ncharge, X.p);
        GLI_CHECK_LAUNCH();
        if (sliced) {
            for (int k = i0; k < i0 + cnt; ++k) nuc_contract_mixed(desc[k], W.p, X.p, H.p, H2.p, err, st);
        } else {
            const int* pr[3];
            for (int q = 0; q < 3; ++q) pr[q] = d_pre + q * (ni + pipes) + i0 + p;
            const int* h_pr = pre + i0 + p;
            auto total = [&](int q) { return dim3((unsigned)h_pr[q * (ni + pipes) + cnt]); };
            dmma_launch(NucStageOp<0>{di, pr[0], cnt, W.p, ks.p, X.p, H.p, H2.p}, total(0), st);
            dmma_launch(NucStageOp<1>{di, pr[1], cnt, W.p, ks.p, X.p, H.p, H2.p}, total(1), st);
            dmma_launch(NucStageOp<2>{di, pr[2], cnt, W.p, ks.p, X.p, H.p, H2.p}, total(2), st);
        }
        k_nuc_scatter<<<dim3((unsigned)std::min<i64>(max_items, (i64)num_sms * 8), (unsigned)cnt), 256, lines, st>>>(
            di, X.p, tables, sliced ? 0 : 1);
        GLI_CHECK_LAUNCH();
    }
    if (pipes > 1)
        for (int p = 0; p < pipes; ++p) {
            GLI_CUDA(cudaEventRecord(t_ring.events[p], t_ring.streams[p]));
            GLI_CUDA(cudaStreamWaitEvent(s, t_ring.events[p], 0));
        }
}

static thread_local NuclearBatchStats t_nuc_stats;
const NuclearBatchStats& last_nuclear_stats() { return t_nuc_stats; }

void nuclear_batch_device(const double* h_coeffs, i64 nb, const std::vector<NuclearJob>& jobs, double tol, int form,
                          cudaStream_t s) {
    if (form != FORM_FP64 && form != FORM_MIXED)
        fail(GLI_ERR_ARGUMENT, "form %d is not a nuclear evaluation form (0 = FP64, 1 = mixed)", form);
    if (!(tol >= 0)) fail(GLI_ERR_ARGUMENT, "tol must be non-negative");
    if (jobs.empty()) return;
    NuclearBatchStats stats;
    // factor shifts needed: 0 .. max |i_a - j_a| over every instance
    i64 L = 1;
    i64 total_nuclei = 0, total_coords = 0;
    for (const NuclearJob& j : jobs) {
        if (j.nn <= 0 || !j.nuclei) fail(GLI_ERR_ARGUMENT, "every instance needs at least one nucleus");
        if (j.nn > 4096) fail(GLI_ERR_LIMIT, "at most 4096 nuclei per instance (got %d)", j.nn);
        if (!j.d_out) fail(GLI_ERR_ARGUMENT, "an instance has no output buffer");
        for (int a = 0; a < 3; ++a) {
            if (j.axes[a].empty() || j.axes[a].size() > 256)
                fail(GLI_ERR_LIMIT, "axis %d has %zu points (1..256)", a, j.axes[a].size());
            L = std::max(L, (i64)j.axes[a].back() - j.axes[a].front() + 1);
            total_coords += (i64)j.axes[a].size();
        }
        total_nuclei += j.nn;
    }
    const int nf = (int)(2 * nb - 1);
    // (a factor of shift s holds exp(-(3 s + i - j)^2 / 4), |i - j| < nb: zero in
    // FP64 from 3 s - nb = 55 on, so larger shifts need no rows)
    L = std::min<i64>(L, (nb + 55) / 3 + 2);
    DevBuf<double> b(nb, s), F(L * nf, s);
    GLI_CUDA(cudaMemcpyAsync(b.p, h_coeffs, nb * sizeof(double), cudaMemcpyHostToDevice, s));
    factors_device(b.p, (int)nb, (int)L, F.p, s);
    DevBuf<int> reach(2, s);
    GLI_CUDA(cudaMemsetAsync(reach.p, 0xff, 2 * sizeof(int), s));
    k_mask_factors<<<(unsigned)((L * nf + 255) / 256), 256, 0, s>>>(F.p, L * nf, nf, (int)nb, tol, reach.p);
    GLI_CHECK_LAUNCH();
    int h_reach[2] = {-1, -1};
    GLI_CUDA(cudaMemcpyAsync(h_reach, reach.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
    GLI_CUDA(cudaStreamSynchronize(s));
    const int h_mmax = h_reach[0], h_smax = h_reach[1];
    // an entry between two points further apart on an axis than any factor
    // reaches is zero: nothing to tabulate (the lattice box of the points grows
    // with the cube of their distance)
    bool dead = jobs.size() == 1 && jobs[0].far_only;
    if (dead) {
        i64 gap = 0;
        for (const auto& list : jobs[0].axes) gap = std::max(gap, (i64)list.back() - list.front());
        dead = gap > h_smax;
    }
    if (h_mmax < 0 || dead) {  // every factor below tol
        for (const NuclearJob& j : jobs) {
            const i64 N = (i64)j.axes[0].size() * j.axes[1].size() * j.axes[2].size();
            GLI_CUDA(cudaMemsetAsync(j.d_out, 0, N * N * sizeof(double), s));
        }
        t_nuc_stats = stats;
        return;
    }
    // host plan and one packed upload: descriptors, coordinates, nuclei
    const i64 ni = (i64)jobs.size();
    std::vector<NucHost> hosts(ni);
    std::vector<int> coords;
    coords.reserve(total_coords);
    std::vector<double> nuc((size_t)(4 * total_nuclei));  // positions, then charges
    i64 nuc_at = 0;
    // key tables, one per axis length (and gap of a two-point list)
    std::vector<uint16_t> tables;
    struct AxisTable {
        int rk_off, key_off, nk;
    };
    std::map<std::pair<int, int>, AxisTable> axis_tables;
    auto axis_table = [&](const std::vector<int>& list) {
        const int n = (int)list.size();
        const bool run = list.back() - list.front() == n - 1;
        const std::pair<int, int> id{n, run ? 1 : n == 2 ? list[1] - list[0] : -(int)axis_tables.size() - 1};
        auto it = axis_tables.find(id);
        if (it != axis_tables.end()) return it->second;
        AxisTable t{(int)tables.size(), 0, 0};
        tables.resize(tables.size() + (size_t)n * n, NUC_DEAD);
        std::vector<uint16_t> keys;
        for (int sum = 0; sum <= 2 * (n - 1); ++sum)
            for (int lo = std::max(0, sum - (n - 1)); 2 * lo <= sum; ++lo) {
                const int hi = sum - lo;
                if (list[hi] - list[lo] > h_smax) continue;
                tables[t.rk_off + lo * n + hi] = tables[t.rk_off + hi * n + lo] = (uint16_t)keys.size();
                keys.push_back((uint16_t)(lo | hi << 8));
            }
        t.key_off = (int)tables.size();
        t.nk = (int)keys.size();
        tables.insert(tables.end(), keys.begin(), keys.end());
        axis_tables[id] = t;
        return t;
    };
    for (i64 k = 0; k < ni; ++k) {
        const NuclearJob& j = jobs[k];
        NucInst& in = hosts[k].d;
        in.band = 2 * h_mmax + 1;
        for (int a = 0; a < 3; ++a) {
            in.n[a] = (int)j.axes[a].size();
            in.coord_off[a] = (int)coords.size();
            coords.insert(coords.end(), j.axes[a].begin(), j.axes[a].end());
            in.u0[a] = 6 * j.axes[a].front() - h_mmax;
            in.U[a] = 6 * (j.axes[a].back() - j.axes[a].front()) + 2 * h_mmax + 1;
            in.P[a] = (int)nuc_even(in.U[a]);
            const AxisTable t = axis_table(j.axes[a]);
            in.nk[a] = t.nk;
            in.rk_off[a] = t.rk_off;
            in.key_off[a] = t.key_off;
            // the keys' order (by the sum of their positions in the list) is by
            // coordinate sum where the list is a run or holds at most two points
            const int span = j.axes[a].back() - j.axes[a].front();
            if (in.n[a] > 2 && span != in.n[a] - 1) in.band = 0;
        }
        in.N = (i64)in.n[0] * in.n[1] * in.n[2];
        in.nuc0 = (int)nuc_at;
        in.nnuc = j.nn;
        for (int q = 0; q < j.nn; ++q, ++nuc_at) {
            for (int a = 0; a < 3; ++a) nuc[(size_t)(3 * nuc_at + a)] = j.nuclei[q].pos[a];
            nuc[(size_t)(3 * total_nuclei + nuc_at)] = (double)j.nuclei[q].charge;
        }
        in.out = j.d_out;
        if ((i64)in.nk[2] * in.nk[1] > ((i64)65535 * TC_BM))
            fail(GLI_ERR_LIMIT, "instance %lld: too many key pairs", (long long)k);
    }
    // chunks: instances whose packed buffers stay under a memory budget (and
    // the weights kernel's grid limit: 3 x instances <= 65535)
    const i64 budget = (i64)6 << 30;  // bytes of packed buffers per chunk
    std::vector<std::pair<i64, i64>> chunks;
    {
        i64 start = 0, bytes = 0;
        for (i64 k = 0; k < ni; ++k) {
            const NucInst& in = hosts[k].d;
            const i64 sz = 8 * ((i64)in.nk[0] * in.P[0] + (i64)in.nk[1] * in.P[1] + (i64)in.nk[2] * in.P[2] +
                                nuc_x_size(in) + nuc_h_size(in) + nuc_h2_size(in));
            if (k > start && (bytes + sz > budget || k - start >= 16384)) {
                chunks.push_back({start, k});
                start = k;
                bytes = 0;
            }
            bytes += sz;
        }
        chunks.push_back({start, ni});
    }
    // one upload: nuclei, coordinates, key tables
    const size_t nbytes = nuc.size() * sizeof(double), cbytes = coords.size() * sizeof(int);
    std::vector<char> up(nbytes + cbytes + tables.size() * sizeof(uint16_t));
    memcpy(up.data(), nuc.data(), nbytes);
    memcpy(up.data() + nbytes, coords.data(), cbytes);
    memcpy(up.data() + nbytes + cbytes, tables.data(), tables.size() * sizeof(uint16_t));
    DevBuf<char> d_up(up.size(), s);
    GLI_CUDA(cudaMemcpyAsync(d_up.p, up.data(), up.size(), cudaMemcpyHostToDevice, s));
    const double* d_npos = reinterpret_cast<const double*>(d_up.p);
    const double* d_nq = d_npos + 3 * total_nuclei;
    const int* d_coords = reinterpret_cast<const int*>(d_up.p + nbytes);
    const uint16_t* d_tables = reinterpret_cast<const uint16_t*>(d_up.p + nbytes + cbytes);
    DevBuf<int> err;
    if (form == FORM_MIXED) {
        err.alloc(1, s);
        err.zero();
    }
    // offsets within the chunk's packed buffers
    for (auto& c : chunks) {
        i64 w = 0, x = 0, h = 0, h2 = 0;
        int ks = 0;
        for (i64 k = c.first; k < c.second; ++k) {
            NucInst& in = hosts[k].d;
            for (int a = 0; a < 3; ++a) {
                in.w_off[a] = w;
                w += (i64)in.nk[a] * in.P[a];
                in.ks_off[a] = ks;
                ks += in.nk[a];
            }
            in.x_off = x;
            in.h_off = h;
            in.h2_off = h2;
            x += nuc_x_size(in);
            h += nuc_h_size(in);
            h2 += nuc_h2_size(in);
        }
    }

    const Context& ctx = context();
    ensure_streams(ctx.device, 8);
    nuc_prepare();
    for (size_t c = 0; c < chunks.size(); ++c) {
        const std::vector<NucHost> part(hosts.begin() + chunks[c].first, hosts.begin() + chunks[c].second);
        // pipelines and, in the mixed form, the contraction path: chosen by
        // timing the first chunk of a batch of this shape (cached per shape
        // key).  Candidate c: c % 16 pipelines, c >= 16 the int8-sliced
        // tensor-core contractions (mixed form only; they pay only where the
        // GEMMs are large enough to carry the slicing passes)
        char key[160];
        snprintf(key, sizeof(key), "nuclear form=%d dev=%d inst=%zu maxN=%lld", form, ctx.device, part.size(),
                 (long long)std::max_element(part.begin(), part.end(), [](const NucHost& a, const NucHost& b) {
                     return a.d.N < b.d.N;
                 })->d.N);
        auto run = [&](int cand) {
            const bool sliced = cand >= 16;
            const int nstreams = cand % 16;
            run_chunk(part, F.p, nf, (int)nb, d_coords, d_npos, d_nq, d_tables, sliced, nstreams, ctx.num_sms, err.p, s);
        };
        std::vector<int> cands = part.size() == 1 ? std::vector<int>{1} : std::vector<int>{1, 2, 4, 8};
        if (form == FORM_MIXED)
            for (size_t k = 0, n0 = cands.size(); k < n0; ++k) cands.push_back(16 + cands[k]);
        const int choice = autotune().choose(key, cands, [&](int cand) {
            cudaEvent_t e0, e1;
            GLI_CUDA(cudaEventCreate(&e0));
            GLI_CUDA(cudaEventCreate(&e1));
            GLI_CUDA(cudaEventRecord(e0, s));
            run(cand);
            GLI_CUDA(cudaEventRecord(e1, s));
            GLI_CUDA(cudaEventSynchronize(e1));
            float ms = 0;
            cudaEventElapsedTime(&ms, e0, e1);
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            return (double)ms;
        });
        stats.streams = choice % 16;
        run(choice);
        stats.chunks += 1;
    }
    int h_err = 0;
    if (err.p) GLI_CUDA(cudaMemcpyAsync(&h_err, err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    GLI_CUDA(cudaStreamSynchronize(s));
    if (h_err) fail(GLI_ERR_INTERNAL, "tensor-core stage: an mbarrier wait expired (code %d)", h_err);
    stats.instances = ni;
    t_nuc_stats = stats;
}

void nuclear_matrix_device(const double* h_coeffs, i64 nb, const std::vector<int> axes[3],
                           const struct atomic_nucleus* nuclei, int nn, double tol, double* d_out, cudaStream_t s,
                           bool far_only) {
    if (nn <= 0) fail(GLI_ERR_ARGUMENT, "at least one nucleus is required");
    std::vector<NuclearJob> jobs(1);
    for (int a = 0; a < 3; ++a) jobs[0].axes[a] = axes[a];
    jobs[0].nuclei = nuclei;
    jobs[0].nn = nn;
    jobs[0].d_out = d_out;
    jobs[0].far_only = far_only;
    nuclear_batch_device(h_coeffs, nb, jobs, tol, FORM_FP64, s);
}

}  // namespace gli
