// FP64 tensor-core tiles: mma.sync.m8n8k4.f64 over operand tiles that the
// caller gathers into shared memory with 8-byte cp.async copies.
//
// A block (4 warps) computes a 64 x BN tile of C = A B (BN = 32, 64 or 80,
// chosen per Op) over K in chunks of 16, three chunks in flight (two for an Op
// that declares STAGES = 2, so that four blocks fit on an SM; cp.async groups,
// the waits are the hardware's own group waits, no flag spins).  Warp w owns every other 8-row and 8-column strip (rows
// 16 i + 8 (w & 1), columns 16 j + 8 (w >> 1)) as 4 x BN/16 m8n8 accumulators,
// so that a partly filled tile loads the four warps (and their tensor pipes)
// alike; per k-step of 4 it reads 4 A and BN/16 B fragments (one double each)
// for 4 BN/16 MMAs of 256 FMAs.  BN = 80 serves 65..80 and 129..160 columns in
// one and two column tiles (129 keys: 2 tiles instead of 3, measured 20%
// faster on the stage A shape).
//
// The operand sources are arbitrary: an Op class says, per tile element, where
// the double comes from (a strided matrix, a lattice-table gather, a gather
// through an index map) and where the results go.  Each operand tile is kept
// in shared memory in one of two layouts, chosen so that the thread mapping
// that coalesces the global reads also writes shared memory without bank
// conflicts, and so that the fragment reads (row = lane / 4, k = lane % 4) are
// conflict-free in both:
//   K-major  [k][row], rows + 4 doubles per k (rows are the unit-stride direction)
//   row-major [row][k], 20 doubles per row    (k is the unit-stride direction)
// (rows + 4 and 20 are 4 mod 16 doubles, so the 16 (row, k) pairs of a half
// warp's fragment read fall in distinct bank pairs.)
// Fragment layouts of m8n8k4 (PTX ISA, mma .f64 m8n8k4): A row = lane/4,
// k = lane%4; B k = lane%4, column = lane/4; C row = lane/4, columns
// 2 (lane%4) + {0, 1}.
#pragma once

#include <cooperative_groups.h>

#include <atomic>
#include <type_traits>

#include "gli_internal.cuh"

namespace gli {

constexpr int DM_BM = 64, DM_BN = 64, DM_BK = 16, DM_STAGES = 3, DM_THREADS = 128;
constexpr int DM_LDK = DM_BK + 4;          // row-major tile: doubles per row
constexpr int DM_LDR = DM_BM + 4;          // K-major 64-row tile: doubles per k
constexpr int DM_TILE_A = DM_BM * DM_LDK;  // doubles of the A tile (>= DM_BK * DM_LDR)
static_assert(DM_TILE_A >= DM_BK * DM_LDR, "operand tile too small for the K-major layout");

// doubles of a B tile of BN rows, and the shared memory of a launch
__host__ __device__ constexpr int dm_tile_b(int bn) { return bn * DM_LDK; }
__host__ __device__ constexpr int dm_smem(int bn, int stages = DM_STAGES) {
    return stages * (DM_TILE_A + dm_tile_b(bn)) * (int)sizeof(double);
}

// pipeline stages of an Op: Op::STAGES where it declares one, else DM_STAGES
template <class Op, class = void>
struct dm_stages_of {
    static constexpr int value = DM_STAGES;
};
template <class Op>
struct dm_stages_of<Op, std::void_t<decltype(Op::STAGES)>> {
    static constexpr int value = Op::STAGES;
};

// Thread tid's q-th element of a rows x 16 operand tile:
//   K-major (64 rows):  row = tid & 63,          k = (tid >> 6) + 2 q,  q < 8
//   row-major:          row = (tid >> 4) + 8 q,  k = tid & 15,          q < rows / 8
constexpr int DM_ELEMS = DM_BM * DM_BK / DM_THREADS;  // 8: the 64-row tiles

__device__ __forceinline__ int dm_kmajor_row(int tid) { return tid & 63; }
__device__ __forceinline__ int dm_kmajor_k(int tid, int q) { return (tid >> 6) + 2 * q; }
__device__ __forceinline__ int dm_rowmajor_row(int tid, int q) { return (tid >> 4) + 8 * q; }
__device__ __forceinline__ int dm_rowmajor_k(int tid) { return tid & 15; }
__device__ __forceinline__ int dm_kmajor_at(int row, int k) { return k * DM_LDR + row; }
__device__ __forceinline__ int dm_rowmajor_at(int row, int k) { return row * DM_LDK + k; }

// 8-byte asynchronous copy global -> shared; src-size 0 writes zeros (src must
// still be a valid address)
__device__ __forceinline__ void dm_cp8(double* dst, const double* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(valid ? 8 : 0)
                 : "memory");
}
// 16-byte copy of two consecutive doubles; bytes (0, 8 or 16) are read, the
// rest of the 16 written as zeros (src 16-byte aligned, valid even for 0)
__device__ __forceinline__ void dm_cp16(double* dst, const double* src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
// row-major tiles whose rows are contiguous in K: thread tid's q-th pair of
// elements (q < rows / 16) is row (tid >> 3) + 16 q, k = 2 (tid & 7) and k + 1
__device__ __forceinline__ int dm_pair_row(int tid, int q) { return (tid >> 3) + 16 * q; }
__device__ __forceinline__ int dm_pair_k(int tid) { return (tid & 7) * 2; }
// bytes of the pair (k, k + 1) that lie before the end of the K range
__device__ __forceinline__ int dm_pair_bytes(int k, int kend) { return k + 1 < kend ? 16 : (k < kend ? 8 : 0); }
__device__ __forceinline__ void dm_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void dm_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ void dm_mma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

template <bool KMAJOR>
__device__ __forceinline__ double dm_frag(const double* s, int row0, int k0, int lane) {
    return KMAJOR ? s[dm_kmajor_at(row0 + (lane >> 2), k0 + (lane & 3))]
                  : s[dm_rowmajor_at(row0 + (lane >> 2), k0 + (lane & 3))];
}

// Op interface (all device, const):
//   static constexpr bool A_KMAJOR, B_KMAJOR;  static constexpr int BN (32, 64
//   or 80; K-major B tiles have 64 rows); optionally STAGES (2 or 3)
//   struct Block { int mvalid, nvalid, nk; ... };       the block's work item
//   struct AState; struct BState;                       per-thread cached row data
//   bool begin(Block&)                                  false: nothing to do (uniform)
//   void a_init(const Block&, AState&), b_init(...)
//   void a_issue(const Block&, AState&, int kc, double* tile)   cp.async of chunk kc
//   void b_issue(const Block&, BState&, int kc, double* tile)   (chunks issued in order)
//   void store(const Block&, int m, int n, double v_n, double v_n1)   C[m][n], C[m][n+1]
//
// Op::a_landed(const Block&, AState&, int kc, double* tile) (optional, when
// the Op declares A_LANDED): called by each thread once its own copies of
// chunk kc have landed and before the block's barrier, to adjust the elements
// it copied (in place, in shared memory)
template <class Op, class = void>
struct dm_a_landed {
    static constexpr bool value = false;
};
template <class Op>
struct dm_a_landed<Op, std::void_t<decltype(Op::A_LANDED)>> {
    static constexpr bool value = Op::A_LANDED;
};

// Skipped strips (an Op that declares SKIP): rows (SKIP_M) or columns (SKIP_N)
// whose operand is zero outside a run of K -- lattice weights, nonzero around
// their key's position -- take part only in the chunks of their 8-row
// strip's run.  Op::live_chunks(blk, strip, first, last) gives the chunks
// [first, last] of a strip (empty: last < first).  Per chunk and strip parity
// (a warp's strips are the even or the odd ones) the live strips [lo, hi) are
// found in shared memory before the main loop (lo | hi << 8; dead strips between
// live ones count as live).  The main loop branches to code made for that run:
// a predicate per strip is turned into predicated MMAs, which take the tensor
// pipe's time whether they execute or not (ERIDA 129^3 stage A: 206 us
// predicated).  The operand's state gets the runs of the strips that the thread
// copies (`live`, row-major tiles copied in pairs: its row dm_pair_row(tid, q)
// lies in strip q of its parity), so that skipped strips are not copied either.
// A skipped MMA would have added products with exact zeros.
constexpr int SKIP_M = 1, SKIP_N = 2, DM_MAX_CHUNKS = 256;
template <class Op, class = void>
struct dm_skip_of {
    static constexpr int value = 0;
};
template <class Op>
struct dm_skip_of<Op, std::void_t<decltype(Op::SKIP)>> {
    static constexpr int value = Op::SKIP;
};

// The runs of at most DM_MAX_CHUNKS chunks are held (4,096 positions, the
// lattice limit of the class lists).  A longer K range (nuclear matrices: the two
// points of an axis may lie any distance apart) shares the last entry among the
// chunks from it on: a strip is live there if it is live in any of them.
__host__ __device__ __forceinline__ int dm_run_entry(int kc) { return kc < DM_MAX_CHUNKS ? kc : DM_MAX_CHUNKS - 1; }
// a strip's chunks [first, last] as entries, first | last << 16 (first > last: empty)
__host__ __device__ __forceinline__ int dm_strip_run(int first, int last) {
    return last < first ? 1 : dm_run_entry(first) | dm_run_entry(last) << 16;
}
// the live strips of parity g at an entry
template <int STRIPS>
__host__ __device__ __forceinline__ uint16_t dm_live_run(const int* run, int g, int entry) {
    int lo = STRIPS / 2, hi = 0;
#pragma unroll
    for (int t = 0; t < STRIPS / 2; ++t) {
        const int r = run[2 * t + g];
        if ((r & 0xffff) <= entry && entry <= r >> 16) {
            if (lo > t) lo = t;
            hi = t + 1;
        }
    }
    return (uint16_t)(hi > lo ? lo | hi << 8 : 0);
}

template <class Op>
__device__ __forceinline__ void dm_build_masks(const Op& op, const typename Op::Block& blk,
                                               uint16_t (&live)[2][DM_MAX_CHUNKS]) {
    constexpr int STRIPS = (dm_skip_of<Op>::value == SKIP_M ? DM_BM : Op::BN) / 8;
    __shared__ int run[STRIPS];
    for (int t = threadIdx.x; t < STRIPS; t += DM_THREADS) {
        int first, last;
        op.live_chunks(blk, t, first, last);
        run[t] = dm_strip_run(first, last);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < min(blk.nk, DM_MAX_CHUNKS); e += DM_THREADS)
#pragma unroll
        for (int g = 0; g < 2; ++g) live[g][e] = dm_live_run<STRIPS>(run, g, e);
    __syncthreads();
}
__device__ __forceinline__ bool dm_live(unsigned run, int strip) {
    return strip >= (int)(run & 0xffu) && strip < (int)(run >> 8);
}

// f(LO, HI) for the run [lo, hi) of N strips
template <int LO, int N, class F>
__device__ __forceinline__ void dm_run_from(int hi, F&& f) {
    using std::integral_constant;
    static_assert(N <= 5, "five strips per warp");
    switch (hi - LO) {
        case 1: f(integral_constant<int, LO>{}, integral_constant<int, LO + 1>{}); break;
        case 2: if constexpr (LO + 2 <= N) f(integral_constant<int, LO>{}, integral_constant<int, LO + 2>{}); break;
        case 3: if constexpr (LO + 3 <= N) f(integral_constant<int, LO>{}, integral_constant<int, LO + 3>{}); break;
        case 4: if constexpr (LO + 4 <= N) f(integral_constant<int, LO>{}, integral_constant<int, LO + 4>{}); break;
        case 5: if constexpr (LO + 5 <= N) f(integral_constant<int, LO>{}, integral_constant<int, LO + 5>{}); break;
    }
}
template <int N, class F>
__device__ __forceinline__ void dm_run(unsigned run, F&& f) {
    const int hi = run >> 8;
    switch (run & 0xffu) {
        case 0: dm_run_from<0, N>(hi, f); break;
        case 1: if constexpr (N > 1) dm_run_from<1, N>(hi, f); break;
        case 2: if constexpr (N > 2) dm_run_from<2, N>(hi, f); break;
        case 3: if constexpr (N > 3) dm_run_from<3, N>(hi, f); break;
        case 4: if constexpr (N > 4) dm_run_from<4, N>(hi, f); break;
    }
}

// The k loop of one block; FULL: every m8n8 tile of the warp's quadrant holds
// data, so the MMAs run unpredicated (a runtime predicate per MMA costs about
// a fifth of the tensor-pipe throughput).
template <class Op, bool FULL>
__device__ __forceinline__ void dm_mainloop(const Op& op, const typename Op::Block& blk, typename Op::AState& as,
                                            typename Op::BState& bs, double* smem, int wm, int wn, int mt, int nt,
                                            const uint16_t* live, double (&acc)[4][Op::BN / 16][2]) {
    constexpr int SKIP = dm_skip_of<Op>::value;
    constexpr int NJ = Op::BN / 16, STAGE = DM_TILE_A + dm_tile_b(Op::BN), NS = dm_stages_of<Op>::value;
    const int lane = threadIdx.x & 31;
    const int nk = blk.nk;
    for (int kc = 0; kc < nk; ++kc) {
        dm_wait<NS - 2>();  // chunk kc has landed (this thread's copies)
        if constexpr (dm_a_landed<Op>::value) op.a_landed(blk, as, kc, smem + (kc % NS) * STAGE);
        __syncthreads();    // ... everyone's; and chunk kc - 1 is consumed
        const int nx = kc + NS - 1;
        if (nx < nk) {
            const int st = nx % NS;
            op.a_issue(blk, as, nx, smem + st * STAGE);
            op.b_issue(blk, bs, nx, smem + st * STAGE + DM_TILE_A);
        }
        dm_commit();
        const double* a_s = smem + (kc % NS) * STAGE;
        const double* b_s = a_s + DM_TILE_A;
        if constexpr (SKIP != 0) {
            // (strips past the tile's rows or columns hold zeros: no run covers
            // them alone, and their results are not stored)
            dm_run<SKIP == SKIP_M ? 4 : NJ>(live[dm_run_entry(kc)], [&](auto lo, auto hi) {
                constexpr int LO = decltype(lo)::value, HI = decltype(hi)::value;
                constexpr int I0 = SKIP == SKIP_M ? LO : 0, I1 = SKIP == SKIP_M ? HI : 4;
                constexpr int J0 = SKIP == SKIP_M ? 0 : LO, J1 = SKIP == SKIP_M ? NJ : HI;
#pragma unroll
                for (int k0 = 0; k0 < DM_BK; k0 += 4) {
                    double af[4], bf[NJ];
#pragma unroll
                    for (int i = I0; i < I1; ++i) af[i] = dm_frag<Op::A_KMAJOR>(a_s, wm + 16 * i, k0, lane);
#pragma unroll
                    for (int j = J0; j < J1; ++j) bf[j] = dm_frag<Op::B_KMAJOR>(b_s, wn + 16 * j, k0, lane);
#pragma unroll
                    for (int i = I0; i < I1; ++i)
#pragma unroll
                        for (int j = J0; j < J1; ++j) dm_mma(acc[i][j], af[i], bf[j]);
                }
            });
            continue;
        }
#pragma unroll
        for (int k0 = 0; k0 < DM_BK; k0 += 4) {
            double af[4], bf[NJ];
#pragma unroll
            for (int i = 0; i < 4; ++i) af[i] = dm_frag<Op::A_KMAJOR>(a_s, wm + 16 * i, k0, lane);
#pragma unroll
            for (int j = 0; j < NJ; ++j) bf[j] = dm_frag<Op::B_KMAJOR>(b_s, wn + 16 * j, k0, lane);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j)
                    if (FULL || (i < mt && j < nt)) dm_mma(acc[i][j], af[i], bf[j]);
        }
    }
}

// blocks per SM a launch is compiled for: Op::MIN_BLOCKS where declared, else 3
template <class Op, class = void>
struct dm_blocks_of {
    static constexpr int value = 3;
};
template <class Op>
struct dm_blocks_of<Op, std::void_t<decltype(Op::MIN_BLOCKS)>> {
    static constexpr int value = Op::MIN_BLOCKS;
};

// Split K inside a thread-block cluster (CLUSTER = true): the launch's
// gridDim.z chunks of K form one cluster of gridDim.z (<= 8) blocks; each
// block leaves its partial tile in its own shared memory, and after a cluster
// barrier every block sums its share of the tile's rows over the cluster's
// blocks through distributed shared memory, in the order of their ranks (the
// same order on every run), and stores it.  Op::begin gives the same answer to
// every block of a cluster (its parts differ in their K range only, which may
// be empty), so that all of them or none reach the cluster barriers.
constexpr int DM_RED_LD = 2;  // doubles of padding per reduction-tile row

template <class Op, bool CLUSTER>
__device__ __forceinline__ void dm_cluster_reduce(const Op& op, const typename Op::Block& blk,
                                                  double* smem, int wm, int wn, int mt, int nt,
                                                  const double (&acc)[4][Op::BN / 16][2]) {
    constexpr int NJ = Op::BN / 16, LD = Op::BN + DM_RED_LD;
    namespace cg = cooperative_groups;
    const int lane = threadIdx.x & 31;
    __syncthreads();  // every warp is done with the operand tiles
    // this block's partial tile, zeros where it has none
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const bool has = i < mt && j < nt;
            double* d = smem + (wm + 16 * i + (lane >> 2)) * LD + wn + 16 * j + 2 * (lane & 3);
            d[0] = has ? acc[i][j][0] : 0.0;
            d[1] = has ? acc[i][j][1] : 0.0;
        }
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    const int P = (int)cl.num_blocks(), r = (int)cl.block_rank();
    {
        // block r sums rows [r0, r1) of the tile: per column pair, the P
        // partial pairs are loaded first (16-byte distributed shared-memory
        // loads, all in flight together) and then added in rank order
        constexpr int PAIRS = Op::BN / 2;
        const int r0 = (DM_BM * r) / P, r1 = (DM_BM * (r + 1)) / P;
        const double2* part[8];
#pragma unroll
        for (int q = 0; q < 8; ++q)
            part[q] = reinterpret_cast<const double2*>(cl.map_shared_rank(smem, q < P ? q : 0));
        // (neighbouring threads read neighbouring pairs of a row: taking rows
        // instead, for Ops whose output is contiguous that way, spreads the remote
        // reads and measured slower, ERIDA 33^3 stage B 23.5 against 18.6 us)
        for (int e = r0 * PAIRS + threadIdx.x; e < r1 * PAIRS; e += blockDim.x) {
            const int row = e / PAIRS, c = 2 * (e % PAIRS);
            const int off = (row * LD + c) / 2;  // LD and c are even: 16-byte aligned pairs
            double2 v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (q < P) v[q] = part[q][off];
            double v0 = v[0].x, v1 = v[0].y;
#pragma unroll
            for (int q = 1; q < 8; ++q)
                if (q < P) {
                    v0 += v[q].x;
                    v1 += v[q].y;
                }
            op.store(blk, row, c, v0, v1);
        }
    }
    cl.sync();  // no block leaves while another still reads its tile
}

template <class Op, bool CLUSTER = false>
__global__ void __launch_bounds__(DM_THREADS, dm_blocks_of<Op>::value) k_dmma(const Op op) {
    constexpr int NJ = Op::BN / 16, STAGE = DM_TILE_A + dm_tile_b(Op::BN), NS = dm_stages_of<Op>::value;
    static_assert(Op::BN == 64 || ((Op::BN == 80 || Op::BN == 32) && !Op::B_KMAJOR),
                  "column tiles of 64, or 32 and 80 read row-major");
    static_assert(NS >= 2 && NS <= 3, "two or three stages");
    static_assert(!CLUSTER || DM_BM * (Op::BN + DM_RED_LD) <= NS * STAGE, "reduction tile exceeds the operand ring");
    extern __shared__ __align__(16) double dm_smem[];
    typename Op::Block blk;
    if (!op.begin(blk)) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = (warp & 1) * 8, wn = (warp >> 1) * 8;
    typename Op::AState as;
    typename Op::BState bs;
    op.a_init(blk, as);
    op.b_init(blk, bs);
    const uint16_t* live = nullptr;
    if constexpr (dm_skip_of<Op>::value != 0) {
        __shared__ uint16_t s_live[2][DM_MAX_CHUNKS];
        dm_build_masks(op, blk, s_live);
        live = s_live[dm_skip_of<Op>::value == SKIP_M ? warp & 1 : warp >> 1];
        // (this thread copies rows (tid >> 3) + 16 q of the skipped operand: strips of one parity)
        if constexpr (dm_skip_of<Op>::value == SKIP_M) as.live = s_live[threadIdx.x >> 6 & 1];
        else bs.live = s_live[threadIdx.x >> 6 & 1];
    }
#pragma unroll
    for (int st = 0; st < NS - 1; ++st) {
        if (st < blk.nk) {
            op.a_issue(blk, as, st, dm_smem + st * STAGE);
            op.b_issue(blk, bs, st, dm_smem + st * STAGE + DM_TILE_A);
        }
        dm_commit();
    }
    // m8 / n8 tiles of this warp's quadrant that hold rows / columns (warp-uniform)
    const int mt = min(4, max(0, (blk.mvalid - wm + 15) >> 4));
    const int nt = min(NJ, max(0, (blk.nvalid - wn + 15) >> 4));
    double acc[4][NJ][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    if (dm_skip_of<Op>::value != 0 || (mt == 4 && nt == NJ))
        dm_mainloop<Op, true>(op, blk, as, bs, dm_smem, wm, wn, mt, nt, live, acc);
    else if constexpr (dm_skip_of<Op>::value == 0)
        dm_mainloop<Op, false>(op, blk, as, bs, dm_smem, wm, wn, mt, nt, live, acc);
    dm_wait<0>();
    if constexpr (CLUSTER) {
        dm_cluster_reduce<Op, CLUSTER>(op, blk, dm_smem, wm, wn, mt, nt, acc);
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
            if (i < mt && j < nt)
                op.store(blk, wm + 16 * i + (lane >> 2), wn + 16 * j + 2 * (lane & 3), acc[i][j][0], acc[i][j][1]);
}

// (three blocks per SM: 3 x 60 or 69 KB of shared memory, at most 170 registers)

// shared memory above the 48 KB default: set once per device and Op type,
// outside any graph capture (cudaFuncSetAttribute is not a stream operation)
template <class Op, bool CLUSTER = false>
void dmma_prepare() {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    GLI_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = dev < 64 ? (uint64_t)1 << dev : 0;
    if (bit && (done.load() & bit)) return;
    GLI_CUDA(cudaFuncSetAttribute(k_dmma<Op, CLUSTER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  dm_smem(Op::BN, dm_stages_of<Op>::value)));
    done.fetch_or(bit);
}

// one launch of k_dmma<Op> on grid `grid`
template <class Op>
void dmma_launch(const Op& op, dim3 grid, cudaStream_t s) {
    if (grid.x == 0 || grid.y == 0 || grid.z == 0) return;
    dmma_prepare<Op>();
    launch_kernel(k_dmma<Op>, grid, dim3(DM_THREADS), dm_smem(Op::BN, dm_stages_of<Op>::value), s, op);
}

// the same with K split over grid.z (2..8) blocks that sum their partial tiles
// in a cluster
template <class Op>
void dmma_launch_cluster(const Op& op, dim3 grid, cudaStream_t s) {
    if (grid.x == 0 || grid.y == 0 || grid.z == 0) return;
    if (grid.z == 1) return dmma_launch(op, grid, s);
    if (grid.z > 8) fail(GLI_ERR_INTERNAL, "cluster split of %u parts", grid.z);
    dmma_prepare<Op, true>();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(DM_THREADS);
    cfg.dynamicSmemBytes = dm_smem(Op::BN, dm_stages_of<Op>::value);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = grid.z;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GLI_CUDA(cudaLaunchKernelEx(&cfg, k_dmma<Op, true>, op));
    count_launch();
}

}  // namespace gli
