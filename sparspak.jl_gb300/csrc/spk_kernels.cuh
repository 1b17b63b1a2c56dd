// Device kernels of the supernodal LU engine (sm_103a).
//
// Storage.  Consecutive supernodes that form a path of the elimination tree
// (each one's parent is the next) are grouped into a *front*, allowing a
// little padding (structural zeros that stay exactly zero).  A front F owns
// columns f..f+nf-1 and has m off-diagonal rows R_F (global, permuted,
// ascending: the rows of its last supernode below the front).  Its part of
// the factor is
//   Lf: (nf+m) x nf column-major, ld = nf+m: rows 0..nf-1 are the front's own
//       columns (unit-lower L11 below the diagonal, U11 on and above it),
//       rows nf.. are L21;
//   Uf: m x nf column-major (U12 transposed: column k holds U row f+k).
// Without padding this is a permutation of the reference's lnz/unz storage
// (src/SparseMethod/SpkSparseBase.jl:253-284); with padding it holds it.
//
// Pivoting.  Every supernode of the reference partition (a *piece* of a
// front, at most 32 columns) factors its own diagonal block with row
// interchanges restricted to that block, applied to the U rows to its right
// only, exactly as _lufactor! does (src/SparseMethod/SpkLUFactor.jl:229-241).
//
// Schedule.  Fronts are processed by elimination-tree level.  Inside a
// level, piece step s runs a panel kernel (triangular solves of piece s)
// and a trailing kernel (rank-w update of the rest of each front, which
// also factors the next piece's diagonal block); then one kernel forms each
// front's Schur complement L21*U12 and scatter-adds it into the ancestor
// fronts.  Kernel boundaries are the only synchronisation.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "spk_umma.cuh"

namespace spk {

typedef long long ll;

struct DFront {
    ll loff;       // Lf offset in the factor array
    ll uoff;       // Uf offset
    ll rows_off;   // R_F offset in rows[]
    ll runid_off;  // offset of the per-row run ids in runid[]
    int f;         // first column (0-based, permuted)
    int nf;        // columns
    int m;         // off-diagonal rows
    int ld;        // nf + m
    int piece0;    // first supernode (0-based) of the front
    int npieces;
    int run0;      // first run of the front in run_*[]
    int block0;    // first block of the front (in the plan's block arrays)
    int nblocks;
    int sq;        // update-row tiles (128 rows) holding the rows that fronts of the next level own (schur_part_tile)
};

// A run is a maximal stretch of R_F lying in the columns of one ancestor
// front G; rel[] gives, for every row of R_F from the run's start on, its
// position in G's row list (G's columns, then R_G).
struct Sched {
    const DFront* fronts;
    const int* xsuper;     // 0-based first column of each supernode, [nsuper+1]
    const int* rows;       // concatenated R_F
    const int* runid;      // run index (absolute) per row of each R_F
    const int* run_tgt;    // target front of each run
    const int* run_start;  // first row (local to R_F) of each run
    const ll* run_rel;     // offset in rel[] of the run's first row
    const int* rel;
    const int* blk_c0;     // front-local first column of each block
    const int* blk_c1;     // front-local end column of each block
    const int* blk_p0;     // first supernode (0-based) of each block
    const int* blk_np;     // supernodes in the block
    const ll* blk_inv2;    // offset in inv2[] of the block's Minv (then Uinv), bw x bw each
    const ll* blk_lpack;   // byte offset of the block's packed L panel (FP32 tensor-core fronts), -1 if none
    const ll* blk_upack;   // byte offset of the block's packed U panel, -1 if none
    // 1: the symmetric form for SPD matrices (POTRF-like: no interchanges;
    // only the lower part of every update is formed, SYRK-like; the U side,
    // U = D L^T, is written from the L panel; LU storage otherwise)
    int sym;
};

// One launch = a list of fronts and the prefix sum of their tile counts.
struct Launch {
    const int* front_ids;
    const int* prefix;     // [count+1]
    int count;
};

__device__ __forceinline__ void locate(const Launch& L, int bid, int& fid, int& tile) {
    int lo = 0, hi = L.count - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (L.prefix[mid] <= bid) lo = mid; else hi = mid - 1;
    }
    fid = L.front_ids[lo];
    tile = bid - L.prefix[lo];
}

__host__ __device__ __forceinline__ int cdiv(int a, int b) { return (a + b - 1) / b; }

// Programmatic dependent launch, for kernels that form a dependent chain:
// griddep_launch lets the next kernel of the stream launch once every CTA of
// this one has started; griddep_wait blocks until the previous kernel has
// completed and its writes are visible (immediately when there is no such
// dependency).  A kernel issues the loads that do not depend on its
// predecessor before waiting.
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename T> __device__ __forceinline__ T tabs(T x) { return x < T(0) ? -x : x; }

// Widest supernode handled.  The reference's splitting rule
// (src/SparseSpdMethod/SpkSymFct.jl:432-460) caps pieces near maxblocksize
// but lets the last piece of a long chain reach about 1.5x that (46 for 30).
constexpr int MAXW = 64;

// ---------------------------------------------------------------------------
// Blocks.  The pieces of a front are processed in *blocks* of consecutive
// pieces (at most BlockMax<T> columns).  A block step is: the block LU
// (k_block_lu_f32, k_block_lu_f64, k_block_lu_small) with exactly the reference's in-piece
// pivoting, then the block's two panels (k_block_panel), then the trailing
// update of the front (k_block_trail).  After the factorisation
// k_block_inv forms, per block, the two operators the triangular solves
// apply: Minv = inv(L_B) P_B and Uinv = inv(U_B) (below).
// ---------------------------------------------------------------------------
template <typename T> struct BlockMax;
template <> struct BlockMax<float> { static constexpr int value = 128; };
template <> struct BlockMax<double> { static constexpr int value = 64; };


// Order-preserving pivot key of |x| for a candidate row (larger key = larger
// |x|, all candidates above non-candidates), with the ggetrf! rules: a NaN
// never wins, except on the diagonal row k, where nothing can displace it.
__device__ __forceinline__ unsigned long long pivot_key(float x, bool cand, bool diag) {
    if (!cand) return 0ull;
    unsigned b = __float_as_uint(x) & 0x7fffffffu;
    if (b > 0x7f800000u) return diag ? ~0ull : 1ull;   // NaN
    return (unsigned long long)b + 2ull;
}
__device__ __forceinline__ unsigned long long pivot_key(double x, bool cand, bool diag) {
    if (!cand) return 0ull;
    unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
    if (b > 0x7ff0000000000000ull) return diag ? ~0ull : 1ull;
    return b + 2ull;
}

// First lane holding the largest key (the reference's first strict maximum).
__device__ __forceinline__ int warp_first_max(unsigned long long key) {
    const unsigned FULL = 0xffffffffu;
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mh = __reduce_max_sync(FULL, hi);
    const unsigned ml = __reduce_max_sync(FULL, hi == mh ? lo : 0u);
    const unsigned ballot = __ballot_sync(FULL, hi == mh && lo == ml);
    return __ffs(ballot) - 1;
}

// 32-bit pivot key of a float (same order as pivot_key).
__device__ __forceinline__ unsigned pivot_key32(float x, bool cand, bool diag) {
    if (!cand) return 0u;
    const unsigned b = __float_as_uint(x) & 0x7fffffffu;
    if (b > 0x7f800000u) return diag ? 0xffffffffu : 1u;
    return b + 2u;
}

// 16-byte loads of N entries (N * sizeof(T) a multiple of 16) from shared memory.
template <int N, typename T>
__device__ __forceinline__ void sm_load(const T* p, T* v) {
    constexpr int E = 16 / sizeof(T);
#pragma unroll
    for (int q = 0; q < N / E; ++q) {
        if constexpr (sizeof(T) == 4) {
            const float4 t = *reinterpret_cast<const float4*>(p + q * E);
            v[q * E] = t.x; v[q * E + 1] = t.y; v[q * E + 2] = t.z; v[q * E + 3] = t.w;
        } else {
            const double2 t = *reinterpret_cast<const double2*>(p + q * E);
            v[q * E] = t.x; v[q * E + 1] = t.y;
        }
    }
}

// Correctly rounded reciprocal (the value of T(1) / x).
__device__ __forceinline__ float rcp_rn(float x) { return __frcp_rn(x); }
__device__ __forceinline__ double rcp_rn(double x) { return __drcp_rn(x); }

__device__ __forceinline__ float rcp_approx(float x) {   // normal x whose reciprocal is normal
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Scaling factor 1 / pivot of the FP32 block LU: the hardware reciprocal
// (within 2 ulp; the FP32 factor is refined in FP64); FP64 keeps the
// correctly rounded one, and so do the FP32 pivots whose reciprocal is not
// normal (__fdividef would give 0 above 2^126).  In a column's chain
// __fdividef costs 140 cycles where the bare instruction takes 20 (measured in
// a loop of one warp).
__device__ __forceinline__ float lu_recip(float x) {
    const float a = fabsf(x);
    return a >= 1.1754944e-38f && a <= 8.5070592e37f ? rcp_approx(x) : rcp_rn(x);
}
__device__ __forceinline__ double lu_recip(double x) { return rcp_rn(x); }

// The pivot lane of a column (first strict maximum of |x| among the
// candidates, pivot_key's rules): one 32-bit reduction for FP32, two for FP64.
__device__ __forceinline__ int warp_pivot_lane(float x, bool cand, bool diag) {
    unsigned key = 0u;
    if (cand) {
        const unsigned b = __float_as_uint(x) & 0x7fffffffu;
        key = b > 0x7f800000u ? (diag ? 0xffffffffu : 1u) : b + 2u;
    }
    const unsigned m = __reduce_max_sync(0xffffffffu, key);
    return __ffs(__ballot_sync(0xffffffffu, key == m)) - 1;
}
__device__ __forceinline__ int warp_pivot_lane(double x, bool cand, bool diag) {
    return warp_first_max(pivot_key(x, cand, diag));
}

// r[k] for a runtime k without indexing a register array dynamically: a
// tree of selects (depth log2 W instead of a W-long chain); W a power of 2.
template <int W, typename T>
__device__ __forceinline__ T pickw(const T (&r)[W], int k) {
    if constexpr (W == 1) {
        return r[0];
    } else {
        T h[W / 2];
#pragma unroll
        for (int i = 0; i < W / 2; ++i) h[i] = (k & (W / 2)) ? r[i + W / 2] : r[i];
        return pickw<W / 2>(h, k);
    }
}

// One right-looking LU sweep over the columns [0, ncols) of a register block
// held one row per lane (rows/columns below 32).  For column k in piece
// [a, b): pivot = first strict maximum among rows [k, b) (ggetrf!), whole
// rows interchanged over columns [a, 32) (the piece's columns, then
// _luswap! of its U rows), column k scaled below the diagonal (ggetrf!
// scaling, and the L-panel trsm 'r','u','n','n' for rows past the piece),
// rank-1 update of rows and columns after k (ggetrf!, the U-panel trsm
// 'r','l','t','u' and the block-local update).  `nrows` rows take part;
// W (a power of 2, at most 32) bounds the columns held.
template <typename T, int W>
__device__ bool warp_lu_sweep(T (&r)[W], int nrows, int ncols, const int* q0, int* piv, bool sym) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    bool sing = false;
    int pc = 0;
    // a rolled loop (the unrolled form's code outgrows the instruction cache),
    // r[k] picked by a tree of selects
#pragma unroll 1
    for (int k = 0; k < ncols; ++k) {
        while (q0[pc + 1] <= k) ++pc;
        const int a = q0[pc], b = q0[pc + 1];
        const T rk0 = pickw<W>(r, k);
        const int kp = warp_pivot_lane(rk0, sym ? lane == k : (lane >= k && lane < b), lane == k);
        if (lane == 0) piv[k] = kp - a;
        const T pv = __shfl_sync(FULL, rk0, kp);
        if (pv != T(0)) {
            if (kp != k) {
#pragma unroll
                for (int j = 0; j < W; ++j) {
                    const T vk = __shfl_sync(FULL, r[j], k), vp = __shfl_sync(FULL, r[j], kp);
                    if (j >= a) {
                        if (lane == k) r[j] = vp;
                        else if (lane == kp) r[j] = vk;
                    }
                }
            }
            const T inv = lu_recip(pv);
            if (lane > k && lane < nrows) {
#pragma unroll
                for (int j = 0; j < W; ++j)
                    if (j == k) r[j] *= inv;
            }
        } else {
            sing = true;
        }
        const T lk = pickw<W>(r, k);
        const bool upd = lane > k && lane < nrows;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            const T u = __shfl_sync(FULL, r[j], k);
            if (upd && j > k) r[j] -= lk * u;
        }
    }
    return sing;
}

// A whole block of at most W <= 32 columns factored by one warp in registers
// (a lane per row) as one right-looking sweep over its columns.  For column
// k in piece [a, b): the pivot is the first strict maximum among rows [k, b)
// (ggetrf!), the interchange acts on whole rows over columns [a, bw) (the
// piece's own columns, then _luswap! of its U rows), column k is scaled
// below the diagonal (ggetrf! scaling for rows in the piece, the L-panel
// trsm 'r','u','n','n' for rows below it) and the rank-1 update covers rows
// and columns after k (ggetrf!, the U-panel trsm 'r','l','t','u' and the
// block-local update).  Columns left of the piece are never interchanged.
// No row moves during the sweep: a lane keeps the position its row has
// reached, and the block is put in order when it is written back: entry j
// of lane's row belongs at row (j >= p0 ? pos : lane).  Unrolled, so that
// only the columns after k are touched (in FP64 a multiply-add takes a warp
// 64 cycles).  Lanes bw .. nrow - 1 may hold rows below the block: the sweep
// turns them into their L21 rows.  piv: local pivot rows; gm[i]: the row now
// at position i; pa[i]: the first row of the piece of position i.
template <typename T, int W>
__device__ __forceinline__ bool warp_block_lu(T (&r)[W], int bw, int nrow, const int* q0, int* piv, int* gm, int* pa, bool sym,
                                              int& pos, int& p0) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    p0 = 0;
    int p1 = 0;   // the piece of row (and column) `lane`
    if (lane < bw) {
        int pc = 0;
        while (q0[pc + 1] <= lane) ++pc;
        p0 = q0[pc];
        p1 = q0[pc + 1];
    }
    pos = lane;
    bool act = lane < nrow, sing = false;
#pragma unroll
    for (int k = 0; k < W; ++k)
        if (k < bw) {
            const T c = r[k];
            const int ce = __shfl_sync(FULL, p1, k);
            const bool diag = pos == k, cand = act && (sym ? diag : pos < ce);
            T rc, rn = T(1);   // every candidate's reciprocal, beside the search; rn for the rows below the block
            if constexpr (sizeof(T) == 4) {
                rc = rcp_approx(c);
                if (nrow > bw) rn = rcp_rn(cand ? c : T(1));
            } else {
                rc = rn = lu_recip(cand ? c : T(1));
            }
            unsigned m;
            if constexpr (sizeof(T) == 4) {
                const unsigned key = pivot_key32(c, cand, diag);
                m = __ballot_sync(FULL, key == __reduce_max_sync(FULL, key));
            } else {
                const unsigned long long key = pivot_key(c, cand, diag);
                const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
                const unsigned mh = __reduce_max_sync(FULL, hi);
                m = __ballot_sync(FULL, hi == mh);
                if (m & (m - 1)) {
                    const unsigned ml = __reduce_max_sync(FULL, hi == mh ? lo : 0u);
                    m = __ballot_sync(FULL, hi == mh && lo == ml);
                }
            }
            if (m & (m - 1)) {   // equal values: the first position
                const bool tied = (m >> lane) & 1u;
                const unsigned p = __reduce_min_sync(FULL, tied ? (unsigned)pos : 0xffffffffu);
                m = __ballot_sync(FULL, tied && (unsigned)pos == p);
            }
            const int kl = 31 - __clz(m);
            const T pv = __shfl_sync(FULL, c, kl);
            T inv = __shfl_sync(FULL, rc, kl);
            const int pp = __shfl_sync(FULL, pos, kl);
            if constexpr (sizeof(T) == 4) {
                if (!(tabs(pv) >= 1.1754944e-38f && tabs(pv) <= 8.5070592e37f)) inv = lu_recip(pv);
            }
            if (pv == T(0)) {   // no scaling
                inv = T(1);
                sing = true;
            }
            if (nrow > bw) {   // below the block 1 / U(k, k) correctly rounded, as the panels take it
                const T r21 = __shfl_sync(FULL, rn, kl);
                if (lane >= bw) inv = r21;
            }
            if (pos == k) pos = pp;
            if (lane == kl) {
                pos = k;
                act = false;
                piv[k] = pp - p0;
            }
            const T l = c * inv;
            if (act) r[k] = l;
#pragma unroll
            for (int j = k + 1; j < W; ++j) {
                const T u = __shfl_sync(FULL, r[j], kl);
                if (act) r[j] -= l * u;
            }
        }
    if (lane < bw) {
        gm[pos] = lane;
        pa[lane] = p0;
    }
    __syncwarp();
    return sing;
}

// Blocks of at most 32 columns: one warp per block, four blocks per CTA (the
// launch holds one block per front).
template <typename T>
__global__ void __launch_bounds__(128) k_block_lu_small(T* fac, int* ipiv, int* info, Sched S, Launch L, int step) {
    __shared__ int sq[4][33];
    __shared__ int spiv[4][32], sgm[4][32], spa[4][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int idx = blockIdx.x * 4 + warp;
    if (idx >= L.count) return;
    const DFront F = S.fronts[L.front_ids[idx]];
    const int blk = F.block0 + step;
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk], bw = c1 - c0;
    const int p0 = S.blk_p0[blk], np = S.blk_np[blk];
    int* q0 = sq[warp];
    int* piv = spiv[warp];
    for (int k = lane; k <= np; k += 32) q0[k] = S.xsuper[p0 + k] - F.f - c0;
    T* blkp = fac + F.loff + (ll)c0 * F.ld + c0;   // block (i, j) at blkp[j * ld + i]
    T r[32];
#pragma unroll
    for (int j = 0; j < 32; ++j)   // symmetric form: the upper triangle mirrors the lower one
        r[j] = lane < bw && j < bw ? ((S.sym && lane < j) ? blkp[(ll)lane * F.ld + j] : blkp[(ll)j * F.ld + lane]) : T(0);
    __syncwarp();
    int pos, pa0;
    const bool sing = warp_block_lu<T, 32>(r, bw, bw, q0, piv, sgm[warp], spa[warp], S.sym != 0, pos, pa0);
    bool zero = false;   // this row's pivot
    if (lane < bw) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (j < bw) {
                blkp[(ll)j * F.ld + (j >= pa0 ? pos : lane)] = r[j];
                zero |= j == pos && r[j] == T(0);
            }
        ipiv[F.f + c0 + lane] = piv[lane];
    }
    if (sing) {   // uniform across the warp: the first piece with a zero pivot
        const unsigned first = __reduce_min_sync(0xffffffffu, zero ? (unsigned)pos : 0xffffffffu);
        if (lane == 0 && first != 0xffffffffu) {
            int pc = 0;
            while (q0[pc + 1] <= (int)first) ++pc;
            atomicMin(info, p0 + pc + 1);
        }
    }
}

// Row sources of a block's interchanges: applying, piece by piece, the
// swaps k <-> a + ipiv[k] of the piece [a, b) to a vector v gives
// v'[R] = v[gmap[R]]; pa[R] = first row of R's piece.  One thread per piece.
__device__ __forceinline__ void block_gather_map(const int* ipiv_blk, const int* q0, int np, int* gmap, int* pa) {
    for (int pc = threadIdx.x; pc < np; pc += blockDim.x) {
        const int a = q0[pc], b = q0[pc + 1];
        for (int i = a; i < b; ++i) {
            gmap[i] = i;
            pa[i] = a;
        }
        for (int k = a; k < b; ++k) {
            const int kp = a + ipiv_blk[k];
            const int t = gmap[k];
            gmap[k] = gmap[kp];
            gmap[kp] = t;
        }
    }
}


// ---------------------------------------------------------------------------
// FP32 block LU by a whole CTA (blocks of 33..128 columns; one CTA per
// front), in groups of at most 32 columns: consecutive whole pieces that
// fit, or a slice of a wider piece.  The block is in shared memory.  Per
// group [a, b):
//   1. warps 0..3 factor the group's rows and columns in registers
//      (lu_sweep): exactly ggetrf!'s pivots, a lane per row, eight columns
//      per warp; no row ever moves, a lane records the position its row has
//      reached;
//   2. a thread per later row solves its L21 entries (trsm 'r','u','n','n')
//      and a thread per later column its U12 entries (_luswap! as a gather
//      of source rows, trsm 'l','l','t','u');
//   3. the rest of the block takes the rank-w update.  The next group's
//      diagonal block is updated first, by eight warps, so that warps 0..3
//      factor it while the others do the rest and write out what is final
//      (look-ahead).
// What bounds it is the latency of step 1 (per column a reduction, a vote,
// the shuffles of the winner's reciprocal and of the next column's entry, a
// multiply-add), so everything else is kept off that chain: the reciprocal
// of every candidate is formed beside the reduction, the warp that owns a
// column only publishes its multipliers and goes on, and the warps of the
// later columns follow two columns behind.  One block of 120 columns alone
// on the GPU: 29 us when every pivot is on the diagonal, 37 us with searches
// (60 us in the form before it, whose owner warp of each four columns also moved
// rows and updated 128 of them per column).
// ---------------------------------------------------------------------------
constexpr int LU_THREADS = 512, LU_G = 32, LU_W = 8;   // group, columns per warp of a sweep
constexpr int LU_LSW = LU_G + 4;   // entries per staged row of a group: 16-byte rows, 4 words apart in the bank cycle

typedef unsigned long long f2;     // two floats, the first in the low half
__device__ __forceinline__ f2 f2_pack(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float f2_lo(f2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float f2_hi(f2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// A sweep's outputs in shared memory.
struct LuSweep {
    float* lu;    // L and U by position: entry (i, j) at lu + i * LU_LSW + j (up to 64 rows)
    float* lt;    // the first w rows transposed: entry (i, j) at lt + j * LU_LSW + i
    float* ex;    // exchange: multipliers of column k by row (ex + k * 64)
    float* rd;    // per column, the reciprocal of its pivot (1 for a zero pivot: no scaling)
    int* piv;     // per column, row | position << 8 of the pivot (position before the interchange)
    int* lsrc;    // original row now at each position
    int* at;      // position of each original row
    int* bad;     // set when the group has to be repeated by a more general form
    int* zero;    // least column with a zero pivot (LU_GENERAL), counted from the block's first: the group's is a
    int a;
};

// Called by warps q = 0 .. cdiv(w, 8) - 1; A is only read, so that a group can
// be repeated.  RPL: rows per lane (at most 32 RPL rows).  cend: in lane k,
// the end of the candidate positions of column k (its piece's end; k + 1 in
// the symmetric form, where the diagonal row is the only candidate).
//   LU_DIAG: the diagonal row is taken as every column's pivot and each
//     candidate is checked against it beside the chain; *bad is set when one is
//     larger.  Nothing of the chain waits for a search then: a column is two
//     shuffles and a multiply-add.
//   LU_SEARCH: a reduction and a vote find the pivot, the first position among
//     equal ones.
//   LU_GENERAL: the same with zero pivots (no scaling), NaN (never wins, except
//     on the diagonal) and reciprocals outside the normal range, for which the
//     other two set *bad.
// A 120-column block with pivots of the one kind throughout: 29, 37 (equal values
// or not) and 63 us.
constexpr int LU_DIAG = 0, LU_SEARCH = 1, LU_GENERAL = 2;
template <int MODE, int RPL>
__device__ __forceinline__ void lu_sweep(const float* A, int lda, int nrow, int w, int cend, const LuSweep& O, int q) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, nq = cdiv(w, LU_W);
    f2 P[RPL][LU_W / 2];
    int pos[RPL];
    bool act[RPL], bad = false;
#pragma unroll
    for (int s = 0; s < RPL; ++s) {
        const int r = lane + 32 * s;
        pos[s] = r;
        act[s] = r < nrow;
#pragma unroll
        for (int i = 0; i < LU_W / 2; ++i) {
            const int j = q * LU_W + 2 * i;
            P[s][i] = f2_pack(r < nrow && j < w ? A[j * lda + r] : 0.0f, r < nrow && j + 1 < w ? A[(j + 1) * lda + r] : 0.0f);
        }
    }
    // rank-1 update of pairs i0 .. with the row in lane kl, slot ks
    auto update = [&](int i0, int kl, int ks, const float (&l)[RPL]) {
        f2 nl[RPL];
#pragma unroll
        for (int s = 0; s < RPL; ++s) nl[s] = f2_pack(-l[s], -l[s]);
#pragma unroll
        for (int i = 0; i < LU_W / 2; ++i)
            if (i >= i0) {
                const f2 v = RPL == 2 && ks ? P[RPL - 1][i] : P[0][i];
                const f2 u = f2_pack(__shfl_sync(FULL, f2_lo(v), kl), __shfl_sync(FULL, f2_hi(v), kl));
#pragma unroll
                for (int s = 0; s < RPL; ++s)
                    if (act[s]) P[s][i] = f2_fma(nl[s], u, P[s][i]);
            }
    };
    // row r (lane kl, slot ks) goes to position k
    auto place = [&](int k, int kl, int ks, int pp) {
#pragma unroll
        for (int s = 0; s < RPL; ++s) {
            if (MODE != LU_DIAG && pos[s] == k) pos[s] = pp;
            if (lane == kl && s == ks) {
                pos[s] = k;
                act[s] = false;
            }
        }
    };
#pragma unroll 1
    for (int o = 0; o < q; ++o)   // follow the warps of the earlier columns, two columns at a time
#pragma unroll
        for (int t = 0; t < LU_W; t += 2) {
            const int k = o * LU_W + t;
            asm volatile("bar.sync %0, %1;" ::"r"(4 + t / 2), "r"(32 * (nq - o)) : "memory");
            float l[2][RPL];
            int pv[2] = {0, 0};
#pragma unroll
            for (int c = 0; c < 2; ++c) {
#pragma unroll
                for (int s = 0; s < RPL; ++s) l[c][s] = O.ex[(k + c) * 64 + lane + 32 * s];
                if (MODE != LU_DIAG) pv[c] = O.piv[k + c];
            }
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int kr = MODE != LU_DIAG ? pv[c] & 255 : k + c;
                place(k + c, kr & 31, kr >> 5, pv[c] >> 8);
                update(0, kr & 31, kr >> 5, l[c]);
            }
        }
#pragma unroll
    for (int t = 0; t < LU_W; ++t) {
        const int k = q * LU_W + t;
        if (k >= w) break;
        float c[RPL], r[RPL], l[RPL];
        const int ce = __shfl_sync(FULL, cend, k);
#pragma unroll
        for (int s = 0; s < RPL; ++s) {
            c[s] = (t & 1) ? f2_hi(P[s][t / 2]) : f2_lo(P[s][t / 2]);
            r[s] = rcp_approx(c[s]);
        }
        int kl = k, ks = 0, pp = k;
        float inv;
        if constexpr (MODE != LU_DIAG) {
            unsigned key[RPL], best = 0u, m = 0u, dup = 0u;
#pragma unroll
            for (int s = 0; s < RPL; ++s) {
                const bool cand = act[s] && pos[s] < ce;
                if (MODE == LU_GENERAL) key[s] = pivot_key32(c[s], cand, pos[s] == k);
                else key[s] = cand ? __float_as_uint(c[s]) & 0x7fffffffu : 0u;   // NaN above infinity: caught below
                best = max(best, key[s]);
            }
            const unsigned mx = __reduce_max_sync(FULL, best);
#pragma unroll
            for (int s = 0; s < RPL; ++s) {
                const unsigned b = __ballot_sync(FULL, key[s] == mx);
                dup |= (b & (b - 1)) | (b ? m : 0u);
                if (b) ks = s;
                m |= b;
            }
            kl = 31 - __clz(m);
            if (dup && mx) {   // equal values: the first position
                unsigned p = 0xffffffffu;
#pragma unroll
                for (int s = 0; s < RPL; ++s)
                    if (key[s] == mx) p = min(p, (unsigned)pos[s]);
                p = __reduce_min_sync(FULL, p);
#pragma unroll
                for (int s = 0; s < RPL; ++s) {
                    const unsigned b = __ballot_sync(FULL, key[s] == mx && (unsigned)pos[s] == p);
                    if (b) {
                        ks = s;
                        kl = 31 - __clz(b);
                    }
                }
            }
            if constexpr (MODE == LU_GENERAL) {
                const float pv = __shfl_sync(FULL, RPL == 2 && ks ? c[RPL - 1] : c[0], kl);
                inv = pv != 0.0f ? lu_recip(pv) : 1.0f;
                if (pv == 0.0f && lane == 0) atomicMin(O.zero, O.a + k);
            } else {
                bad |= mx - 0x00800000u > 0x7e000000u - 0x00800000u;
                inv = __shfl_sync(FULL, RPL == 2 && ks ? r[RPL - 1] : r[0], kl);
            }
            pp = __shfl_sync(FULL, RPL == 2 && ks ? pos[RPL - 1] : pos[0], kl);
        } else {
            inv = __shfl_sync(FULL, r[0], k);
            const unsigned d = __float_as_uint(__shfl_sync(FULL, c[0], k)) & 0x7fffffffu;
            bad |= d - 0x00800000u > 0x7e000000u - 0x00800000u;
#pragma unroll
            for (int s = 0; s < RPL; ++s)   // a tie keeps the diagonal row, the first candidate; NaN counts as larger
                bad |= act[s] && pos[s] < ce && (__float_as_uint(c[s]) & 0x7fffffffu) > d;
        }
        place(k, kl, ks, pp);
#pragma unroll
        for (int s = 0; s < RPL; ++s) {
            l[s] = c[s] * inv;
            O.ex[k * 64 + lane + 32 * s] = l[s];
            if (lane == kl && s == ks) {
                O.piv[k] = (kl + 32 * ks) | pp << 8;
                O.rd[k] = inv;
            }
        }
        if ((t & 1) && q + 1 < nq) asm volatile("bar.arrive %0, %1;" ::"r"(4 + t / 2), "r"(32 * (nq - q)) : "memory");
        if (!(t & 1)) {
            const float v = f2_hi(RPL == 2 && ks ? P[RPL - 1][t / 2] : P[0][t / 2]);
            const float u = __shfl_sync(FULL, v, kl);
#pragma unroll
            for (int s = 0; s < RPL; ++s)
                if (act[s]) P[s][t / 2] = f2_pack(l[s], fmaf(-l[s], u, f2_hi(P[s][t / 2])));
        } else {
#pragma unroll
            for (int s = 0; s < RPL; ++s)
                if (act[s]) P[s][t / 2] = f2_pack(f2_lo(P[s][t / 2]), l[s]);
        }
        update(t / 2 + 1, kl, ks, l);
    }
    if (q == nq - 1)   // the last warp knows every row's final position
#pragma unroll
        for (int s = 0; s < RPL; ++s)
            if (lane + 32 * s < nrow) {
                O.at[lane + 32 * s] = pos[s];
                O.lsrc[pos[s]] = lane + 32 * s;
            }
    if (bad) *O.bad = 1;
    asm volatile("bar.sync 12, %0;" ::"r"(32 * nq) : "memory");
#pragma unroll
    for (int s = 0; s < RPL; ++s)
        if (lane + 32 * s < nrow) {
            const int i = O.at[lane + 32 * s];
            ulonglong2* d = reinterpret_cast<ulonglong2*>(O.lu + i * LU_LSW + q * LU_W);
            d[0] = make_ulonglong2(P[s][0], P[s][1]);
            d[1] = make_ulonglong2(P[s][2], P[s][3]);
            if (i < LU_G)
#pragma unroll
                for (int j = 0; j < LU_W; ++j)
                    O.lt[(q * LU_W + j) * LU_LSW + i] = (j & 1) ? f2_hi(P[s][j / 2]) : f2_lo(P[s][j / 2]);
        }
}

struct LuSmem {   // offsets in floats
    static constexpr int BM = 128, LD = BM + 1, SLB = BM + 4;   // a slab's last row is read up to 28 entries past its end
    static constexpr int a = 0;                          // A(i, j) at a + j * LD + i
    static constexpr int lu = (BM * LD + 3) / 4 * 4;     // LuSweep::lu
    static constexpr int lt = lu + 2 * LU_G * LU_LSW;    // LuSweep::lt
    static constexpr int ex = lt + LU_G * LU_LSW;        // LuSweep::ex
    static constexpr int sl = ex + LU_G * 2 * LU_G;      // L21 by column: sl + k * SLB + row - b
    static constexpr int su = sl + LU_G * SLB;           // U12 by row: su + k * SLB + column - b
    static constexpr int bytes = (su + LU_G * SLB + 32) * 4;
};

// A(i, j) -= sum_k sl[k][i] su[k][j], one warp: rows r0 + lane + 32 m (m < M,
// below r1) and columns [4 c, 4 c + 4) below q1 (relative to the slabs).
// Lanes run along the rows, so that every access is free of bank conflicts.
template <int M>
__device__ __forceinline__ void lu_rank_tile(float* A, const float* sl, const float* su, int w, int r0, int r1, int c, int q1) {
    constexpr int LD = LuSmem::LD, SLB = LuSmem::SLB;
    const int lane = threadIdx.x & 31;
    f2 acc[M][2];
#pragma unroll
    for (int m = 0; m < M; ++m) acc[m][0] = acc[m][1] = 0ull;
    const float* x = sl + r0 + lane;
    const float* y = su + 4 * c;
#pragma unroll 4
    for (int k = 0; k < w; ++k) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(y + k * SLB);   // past r1 (q1): read, never stored
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const float xm = x[k * SLB + 32 * m];
            const f2 xx = f2_pack(xm, xm);
            acc[m][0] = f2_fma(xx, v.x, acc[m][0]);
            acc[m][1] = f2_fma(xx, v.y, acc[m][1]);
        }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int i = r0 + lane + 32 * m;
        const float d[4] = {f2_lo(acc[m][0]), f2_hi(acc[m][0]), f2_lo(acc[m][1]), f2_hi(acc[m][1])};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i < r1 && 4 * c + j < q1) A[(4 * c + j) * LD + i] -= d[j];
    }
}
// Rows [r0, r1) (at most 128), one quad of columns.
__device__ __forceinline__ void lu_rank_quad(float* A, const float* sl, const float* su, int w, int r0, int r1, int c, int q1) {
    const int m = cdiv(r1 - r0, 32);
    if (m == 1) lu_rank_tile<1>(A, sl, su, w, r0, r1, c, q1);
    else if (m == 2) lu_rank_tile<2>(A, sl, su, w, r0, r1, c, q1);
    else if (m >= 3) {
        lu_rank_tile<3>(A, sl, su, w, r0, r1, c, q1);
        if (m > 3) lu_rank_tile<1>(A, sl, su, w, r0 + 96, r1, c, q1);
    }
}

__global__ void __launch_bounds__(LU_THREADS, 1) k_block_lu_f32(float* fac, int* ipiv, int* info, int* bmap, Sched S,
                                                                Launch L, int step) {
    using SM = LuSmem;
    constexpr int BM = SM::BM, LD = SM::LD, SLB = SM::SLB, NW = LU_THREADS / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* sm = reinterpret_cast<float*>(smem_raw);
    float *A = sm + SM::a, *lu = sm + SM::lu, *sl = sm + SM::sl, *su = sm + SM::su;
    __shared__ int cpa[BM], cpb[BM];          // piece of each column
    __shared__ int gs[BM + 1], ge[BM];        // groups: first column, end of the rows that take part
    __shared__ __align__(16) float srd[LU_G];   // reciprocals of the group's pivots
    __shared__ __align__(16) int lsrc[2 * LU_G];
    __shared__ int spv[LU_G], sat[2 * LU_G], sbad;
    __shared__ int spiv[BM], gmap[BM];        // gmap: row sources of the block's interchanges
    __shared__ int szero, ngrp;
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    const int blk = F.block0 + step;
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk], bw = c1 - c0;
    const int p0 = S.blk_p0[blk], np = S.blk_np[blk];
    const int tid = threadIdx.x, wp = tid >> 5, lane = tid & 31;
    const bool sym = S.sym != 0;
    float* blkp = fac + F.loff + (ll)c0 * F.ld + c0;   // block (i, j) at blkp[j * ld + i]
    {
        float v[BM / NW][4];
#pragma unroll
        for (int q = 0; q < BM / NW; ++q)
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int C = wp + q * NW, R = lane + 32 * s;
                v[q][s] = (C < bw && R < bw && (!sym || R >= C)) ? blkp[(ll)C * F.ld + R] : 0.0f;
            }
        for (int pc = tid; pc < np; pc += LU_THREADS) {
            const int a = S.xsuper[p0 + pc] - F.f - c0, b = S.xsuper[p0 + pc + 1] - F.f - c0;
            for (int k = a; k < b; ++k) {
                cpa[k] = a;
                cpb[k] = b;
            }
        }
        if (tid < BM) gmap[tid] = tid;
        if (tid == 0) {
            szero = INT_MAX;
            sbad = 0;
        }
#pragma unroll
        for (int q = 0; q < BM / NW; ++q)
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int C = wp + q * NW, R = lane + 32 * s;
                if (C < bw && R < bw && (!sym || R >= C)) {
                    A[C * LD + R] = v[q][s];
                    if (sym) A[R * LD + C] = v[q][s];   // symmetric form: the upper triangle mirrors the lower one
                }
            }
    }
    __syncthreads();
    if (tid == 0) {   // groups: whole pieces up to LU_G columns, or LU_G-column slices of a wider piece
        int n = 0, a = 0;
        while (a < bw) {
            int b = a, e;
            while (b < bw && cpb[b] - a <= LU_G) b = cpb[b];
            e = b;
            if (b == a) {
                e = cpb[a];
                b = a + LU_G;
            }
            gs[n] = a;
            ge[n++] = e;
            a = b;
        }
        gs[n] = bw;
        ngrp = n;
    }
    LuSweep O{lu, sm + SM::lt, sm + SM::ex, srd, spv, lsrc, sat, &sbad, &szero, 0};
    // part 1 of group [a, b), rows to e (warps 0..3)
    auto sweep = [&](int a, int b, int e, int mode) {
        const int w = b - a, nrow = e - a;
        O.a = a;
        if (wp >= cdiv(w, LU_W)) return;
        const int cend = lane < w ? (sym ? lane + 1 : cpb[a + lane] - a) : 0;
        const float* D = A + a * LD + a;
        if (nrow <= 32) {
            if (mode == LU_DIAG) lu_sweep<LU_DIAG, 1>(D, LD, nrow, w, cend, O, wp);
            else if (mode == LU_SEARCH) lu_sweep<LU_SEARCH, 1>(D, LD, nrow, w, cend, O, wp);
            else lu_sweep<LU_GENERAL, 1>(D, LD, nrow, w, cend, O, wp);
        } else {
            if (mode != LU_GENERAL) lu_sweep<LU_SEARCH, 2>(D, LD, nrow, w, cend, O, wp);
            else lu_sweep<LU_GENERAL, 2>(D, LD, nrow, w, cend, O, wp);
        }
    };
    __syncthreads();
    const int ng = ngrp;
    int mode = LU_DIAG;   // a group that needs a more general form starts the next ones with it
    if (wp < 4) sweep(gs[0], gs[1], ge[0], mode);
    __syncthreads();
    int done = 0;   // columns [0, done) and their rows are written out
#pragma unroll 1
    for (int g = 0; g < ng; ++g) {
        const int a = gs[g], b = gs[g + 1], w = b - a, e = ge[g], nrow = e - a;
        const bool moved = e > b || cpa[a] < a;
        for (int again = sbad; again; again = sbad) {   // (the symmetric form has nothing to search)
            mode = mode == LU_DIAG && !sym && nrow <= 32 ? LU_SEARCH : LU_GENERAL;
            __syncthreads();
            if (tid == 0) sbad = 0;
            __syncthreads();
            if (wp < 4) sweep(a, b, e, mode);
            __syncthreads();
        }
        if (moved) {
            // a slice of a wide piece: its interchanges move whole rows, over
            // the columns right of the group and those of the piece left of it
            const int left = a - cpa[a], nc = left + (bw - b);
            for (int c = wp; c < nc; c += NW) {
                float* col = A + (c < left ? cpa[a] + c : b + c - left) * LD + a;
                const int lim = c < left ? cpb[a] - a : nrow;   // left: the rows of this piece only
                const float v0 = lane < lim ? col[lsrc[lane]] : 0.0f, v1 = lane + 32 < lim ? col[lsrc[lane + 32]] : 0.0f;
                __syncwarp();
                if (lane < lim) col[lane] = v0;
                if (lane + 32 < lim) col[lane + 32] = v1;
            }
            __syncthreads();
        }
        // part 2: warps 0, 2, 4 (.. by 32) the rows below, warps 1, 3, 5 the columns right
        const int nr = bw - b;
        if (wp < 2 * cdiv(nr, 32)) {
            const int x = (wp >> 1) * 32 + lane;
            // Both are x := x T^-1 with the rows of T in order: T = U for a
            // row of L21 (entries scaled by 1 / U(k, k)), T = L^T for a
            // column of U12 (unit diagonal), so they share their code.
            const bool isU = wp & 1;
            float* line = isU ? A + (b + x) * LD + a : A + a * LD + b + x;   // entry k at line[k * ls]
            const int ls = isU ? 1 : LD;
            float* out = (isU ? su : sl) + x;
            const float* T = isU ? O.lt : lu;
            if (x < nr && !isU && b + x < e) {   // a row of the sliced piece: its multipliers are known
                for (int k = 0; k < w; ++k) {
                    const float v = lu[(b + x - a) * LU_LSW + k];
                    line[k * ls] = v;
                    out[k * SLB] = v;
                }
            } else if (x < nr) {
                const bool gather = isU && !moved;   // the interchanges of whole pieces, as a gather
                f2 y[LU_G / 2];
#pragma unroll
                for (int k = 0; k < LU_G; k += 4) {
                    const int4 src = gather ? *reinterpret_cast<const int4*>(lsrc + k) : make_int4(k, k + 1, k + 2, k + 3);
                    y[k / 2] = f2_pack(k < w ? line[src.x * ls] : 0.0f, k + 1 < w ? line[src.y * ls] : 0.0f);
                    y[k / 2 + 1] = f2_pack(k + 2 < w ? line[src.z * ls] : 0.0f, k + 3 < w ? line[src.w * ls] : 0.0f);
                }
#pragma unroll
                for (int k = 0; k < LU_G; ++k) {   // past w: zeros, times whatever is there, never stored
                    const float v = (k & 1 ? f2_hi(y[k / 2]) : f2_lo(y[k / 2])) * (isU ? 1.0f : srd[k]);
                    const f2 nv = f2_pack(-v, -v);
                    const ulonglong2* tr = reinterpret_cast<const ulonglong2*>(T + k * LU_LSW);
                    if (!(k & 1)) y[k / 2] = f2_pack(v, f2_hi(y[k / 2]) - v * T[k * LU_LSW + k + 1]);
                    else y[k / 2] = f2_pack(f2_lo(y[k / 2]), v);
#pragma unroll
                    for (int q = (k / 2 + 1) / 2; q < LU_G / 4; ++q) {
                        const ulonglong2 u = tr[q];
                        if (2 * q > k / 2) y[2 * q] = f2_fma(nv, u.x, y[2 * q]);
                        y[2 * q + 1] = f2_fma(nv, u.y, y[2 * q + 1]);
                    }
                }
#pragma unroll
                for (int k = 0; k < LU_G; ++k)
                    if (k < w) {
                        const float v = k & 1 ? f2_hi(y[k / 2]) : f2_lo(y[k / 2]);
                        line[k * ls] = v;
                        out[k * SLB] = v;
                    }
            }
        } else if (wp >= 8) {
            // the group's own part of the factor (the multipliers left of a
            // row's piece are never interchanged), pivots and row sources
            for (int j = wp - 8; j < w; j += NW - 8)
                if (lane < w) {
                    const int i = lane;
                    const int s = i <= j || a + j >= cpa[a + i] ? i : sat[i];
                    A[(a + j) * LD + a + i] = lu[s * LU_LSW + j];
                }
            if (wp == 13 && lane < w) spiv[a + lane] = a + (spv[lane] >> 8) - cpa[a + lane];
            if (wp >= 14) {   // row sources: composed over the slices of a wide piece
                const int i = tid - (LU_THREADS - 64);
                const int v = i < nrow ? gmap[a + lsrc[i]] : 0;
                asm volatile("bar.sync 3, 64;" ::: "memory");
                if (i < nrow) gmap[a + i] = v;
            }
        }
        __syncthreads();
        if (g + 1 == ng) break;
        // part 3, the next group's diagonal block first
        // (its rows rounded up to 32, its columns to 4)
        const int b2 = gs[g + 2], e2 = ge[g + 1], rn = min(cdiv(e2 - b, 32) * 32, nr), cn = cdiv(b2 - b, 4);
        float* D = A + b * LD + b;
        if (wp < 8) {
            for (int c = wp; c < cn; c += 8) lu_rank_quad(D, sl, su, w, 0, rn, c, nr);
            asm volatile("bar.sync 1, 256;" ::: "memory");
        }
        if (wp < 4) {
            sweep(b, b2, e2, mode);
        } else {
            for (int c = wp - 4; c < cdiv(nr, 4); c += NW - 4) lu_rank_quad(D, sl, su, w, c < cn ? rn : 0, nr, c, nr);
            if (e == b) {   // whole pieces: their columns, and their rows right of them, are final
                for (int C = done + wp - 4; C < bw; C += NW - 4)
                    for (int R = done + lane; R < (C < b ? bw : b); R += 32) blkp[(ll)C * F.ld + R] = A[C * LD + R];
            }
        }
        if (e == b) done = b;
        __syncthreads();
    }
    for (int C = done + wp; C < bw; C += NW)
        for (int R = done + lane; R < bw; R += 32) blkp[(ll)C * F.ld + R] = A[C * LD + R];
    if (tid < bw) {
        ipiv[F.f + c0 + tid] = spiv[tid];
        bmap[F.f + c0 + tid] = gmap[tid] | (cpa[tid] << 8);
    }
    if (tid == 0 && szero != INT_MAX) {
        int p = 0;
        while (S.xsuper[p0 + p + 1] - F.f - c0 <= szero) ++p;
        atomicMin(info, p0 + p + 1);   // first singular piece of the block
    }
}

// Block LU by pieces, for blocks whose pieces are all at most 32 columns
// wide (the supernode partition's maxblocksize, 30 by default).  The
// block is staged in shared memory; for each piece [a, b) in turn:
//   (1) one warp factors the piece's diagonal block in registers
//       (warp_lu_sweep: ggetrf!, pivots among the piece's rows);
//   (2) a thread per column right of the piece applies the piece's
//       interchanges and solves U12 := inv(L11) P A12 (_luswap!, trsm
//       'l','l','n','u'), and a thread per row below it solves
//       L21 := A21 inv(U11) (trsm 'r','u','n','n');
//   (3) the rest of the block takes the rank-w update A22 -= L21 U12 (gemm),
//       a warp per four columns with its lanes on the rows.
// Only the w rows of the piece are on the sequential path of (1); the rows
// below are solved in parallel afterwards, which is where this form gains
// over forms whose owner warp sweeps all rows of the block for every column.
// Outputs: the factored block, ipiv, the row
// sources of the interchanges (bmap) and the first singular piece.
constexpr int PC_THREADS = 512;
template <typename T> struct PcLu {
    static constexpr int BM = BlockMax<T>::value;
    static constexpr int LDS = BM + 1;   // column stride of the staged block (conflict-free rows and columns)
    static constexpr size_t smem = sizeof(T) * ((size_t)BM * LDS + (size_t)32 * BM + 32);
};

template <typename T>
__global__ void __launch_bounds__(PC_THREADS, 1) k_block_lu_pc(T* fac, int* ipiv, int* info, int* bmap, Sched S,
                                                                Launch L, int step) {
    constexpr int BM = BlockMax<T>::value, LDS = PcLu<T>::LDS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* sA = reinterpret_cast<T*>(smem_raw);   // A(i, j) at sA[j * LDS + i]
    T* sU = sA + BM * LDS;                    // U(a + k, b + c) of the current piece at sU[k * BM + c]
    T* srv = sU + 32 * BM;                    // 1 / U(a + k, a + k)
    __shared__ int q0[BM + 1], spiv[BM], sgm[32], sgmap[BM], sq[2];
    __shared__ int szero;
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    const int blk = F.block0 + step;
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk], bw = c1 - c0;
    const int p0 = S.blk_p0[blk], np = S.blk_np[blk];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const bool sym = S.sym != 0;
    for (int k = tid; k <= np; k += PC_THREADS) q0[k] = S.xsuper[p0 + k] - F.f - c0;
    if (tid == 0) szero = INT_MAX;
    T* blkp = fac + F.loff + (ll)c0 * F.ld + c0;   // block (i, j) at blkp[j * ld + i]
    for (int e = tid; e < bw * bw; e += PC_THREADS) {
        const int C = e / bw, R = e - C * bw;
        // symmetric form: the upper triangle mirrors the lower one
        sA[C * LDS + R] = (sym && R < C) ? blkp[(ll)R * F.ld + C] : blkp[(ll)C * F.ld + R];
    }
    __syncthreads();
#pragma unroll 1
    for (int pc = 0; pc < np; ++pc) {
        const int a = q0[pc], b = q0[pc + 1], wd = b - a, nr = bw - b;
        if (w == 0) {   // (1) the piece's diagonal block
            if (lane == 0) {
                sq[0] = 0;
                sq[1] = wd;
            }
            T r[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = (lane < wd && j < wd) ? sA[(a + j) * LDS + a + lane] : T(0);
            __syncwarp();
            const bool sing = warp_lu_sweep<T, 32>(r, wd, wd, sq, spiv + a, sym);
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (lane < wd && j < wd) sA[(a + j) * LDS + a + lane] = r[j];
            const T d = pickw<32>(r, lane);
            if (lane < wd) srv[lane] = d != T(0) ? T(1) / d : T(1);
            if (sing) {   // uniform in the warp
                const unsigned z = __ballot_sync(0xffffffffu, lane < wd && d == T(0));
                if (lane == 0 && z) szero = min(szero, a + __ffs(z) - 1);
            }
            __syncwarp();
            // the row now at position i of the piece came from row sgm[i]
            int g = lane;
            for (int k = 0; k < wd; ++k) {
                const int kp = spiv[a + k];
                const int vk = __shfl_sync(0xffffffffu, g, k), vp = __shfl_sync(0xffffffffu, g, kp);
                g = lane == k ? vp : (lane == kp ? vk : g);
            }
            if (lane < wd) sgm[lane] = g;
        }
        __syncthreads();
        // (2) U12 columns (threads 0..) and L21 rows (threads 256..) inside the block
        if (tid < nr) {
            const int j = b + tid;
            T y[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) y[i] = i < wd ? sA[j * LDS + a + sgm[i]] : T(0);
#pragma unroll
            for (int k = 0; k < 32; ++k)
                if (k < wd) {
#pragma unroll
                    for (int i = k + 1; i < 32; ++i)
                        if (i < wd) y[i] -= sA[(a + k) * LDS + a + i] * y[k];
                }
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (i < wd) {
                    sA[j * LDS + a + i] = y[i];
                    sU[i * BM + tid] = y[i];
                }
        } else if (tid >= PC_THREADS / 2 && tid - PC_THREADS / 2 < nr) {
            const int rr = b + tid - PC_THREADS / 2;
            T x[32];
#pragma unroll
            for (int k = 0; k < 32; ++k) x[k] = k < wd ? sA[(a + k) * LDS + rr] : T(0);
#pragma unroll
            for (int k = 0; k < 32; ++k)
                if (k < wd) {
                    x[k] *= srv[k];
#pragma unroll
                    for (int jj = k + 1; jj < 32; ++jj)
                        if (jj < wd) x[jj] -= x[k] * sA[(a + jj) * LDS + a + k];
                }
#pragma unroll
            for (int k = 0; k < 32; ++k)
                if (k < wd) sA[(a + k) * LDS + rr] = x[k];
        }
        __syncthreads();
        // (3) A22 -= L21 U12: warp per four columns, lane + 32 q on the rows
        if (nr > 0) {
            const int ncg = cdiv(nr, 4);
            for (int cg = w; cg < ncg; cg += PC_THREADS / 32) {
                const int j0 = 4 * cg;
                T acc[4][4];
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[q][c] = T(0);
                for (int k = 0; k < wd; ++k) {
                    T l[4], u[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) l[q] = lane + 32 * q < nr ? sA[(a + k) * LDS + b + lane + 32 * q] : T(0);
#pragma unroll
                    for (int c = 0; c < 4; ++c) u[c] = sU[k * BM + j0 + c];
#pragma unroll
                    for (int q = 0; q < 4; ++q)
#pragma unroll
                        for (int c = 0; c < 4; ++c) acc[q][c] += l[q] * u[c];
                }
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (j0 + c < nr)
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (lane + 32 * q < nr) sA[(b + j0 + c) * LDS + b + lane + 32 * q] -= acc[q][c];
            }
        }
        __syncthreads();
    }
    for (int e = tid; e < bw * bw; e += PC_THREADS) {
        const int C = e / bw, R = e - C * bw;
        blkp[(ll)C * F.ld + R] = sA[C * LDS + R];
    }
    for (int c = tid; c < bw; c += PC_THREADS) ipiv[F.f + c0 + c] = spiv[c];
    // Row sources of the block's interchanges (block_gather_map), a warp per
    // piece: lane i tracks gmap[a + i] through the piece's swaps.
    for (int pc = w; pc < np; pc += PC_THREADS / 32) {
        const int a = q0[pc], b = q0[pc + 1];
        int g = a + lane;
        for (int k = a; k < b; ++k) {
            const int kp = a + spiv[k];
            const int vk = __shfl_sync(0xffffffffu, g, k - a), vp = __shfl_sync(0xffffffffu, g, kp - a);
            g = lane == k - a ? vp : (lane == kp - a ? vk : g);
        }
        if (lane < b - a) bmap[F.f + c0 + a + lane] = g | (a << 8);
    }
    (void)sgmap;
    if (tid == 0 && szero != INT_MAX) {
        int p = 0;
        while (q0[p + 1] <= szero) ++p;
        atomicMin(info, p0 + p + 1);   // first singular piece of the block
    }
}

// ---------------------------------------------------------------------------
// Panel sweeps on register lines.  A line (a row of X or a column of Y) of
// a block of width bw <= W is held by 4 consecutive lanes, lane q of the
// group owning entries [q*CQ, q*CQ + CQ), CQ = W / 4.  Column by column the
// owner of entry k scales it (rows) and shuffles it to its group, and every
// lane updates its entries with a row of U or a column of L read from
// shared memory (the triangles are staged with zeros outside the strict
// part, so the updates need no predicates).
//   rows: X := X inv(U_B), U_B the block's upper triangle with its diagonal:
//         sU by rows, zero on and below the diagonal, rd[k] = 1/U(k,k);
//   cols: Y := inv(L_B) Y, L_B the block's unit lower triangle: sL by
//         columns, zero on and above the diagonal.
// A staged row (column) is SLD(W) entries: the four lanes' chunks of CQ
// entries each start 16 bytes apart in the bank cycle (chunk q at
// q * (CQ + SK)), so their 16-byte loads do not collide; one more 16-byte
// unit per row puts consecutive rows 20 words apart in the 32-bank cycle, so
// that the staging copies of 8 rows x 4 entries per warp hit 32 banks.
// ---------------------------------------------------------------------------
template <typename T> struct Skew { static constexpr int value = 16 / sizeof(T); };
template <typename T, int W> struct SLD { static constexpr int value = W + 5 * Skew<T>::value; };
template <typename T, int W>
__device__ __forceinline__ int sidx(int k, int j) {   // entry j of staged row / column k
    constexpr int CQ = W / 4, SK = Skew<T>::value;
    return k * SLD<T, W>::value + (j / CQ) * (CQ + SK) + (j % CQ);
}

template <typename T, int W>
__device__ __forceinline__ void sweep_rows(T (&x)[W / 4], const T* sU, const T* rd, int bw) {
    constexpr int CQ = W / 4;
    const int lane = threadIdx.x & 31, q = lane & 3, base = lane & ~3;
#pragma unroll 1
    for (int kq = 0; kq * CQ < bw; ++kq) {
#pragma unroll
        for (int kk = 0; kk < CQ; ++kk) {
            const int k = kq * CQ + kk;
            if (k >= bw) break;
            if (q == kq) x[kk] *= rd[k];
            const T xk = __shfl_sync(0xffffffffu, x[kk], base | kq);
            const T* u = sU + k * SLD<T, W>::value + q * (CQ + Skew<T>::value);
#pragma unroll
            for (int jj = 0; jj < CQ; ++jj) x[jj] -= xk * u[jj];
        }
    }
}

template <typename T, int W>
__device__ __forceinline__ void sweep_cols(T (&y)[W / 4], const T* sL, int bw) {
    constexpr int CQ = W / 4;
    const int lane = threadIdx.x & 31, q = lane & 3, base = lane & ~3;
#pragma unroll 1
    for (int kq = 0; kq * CQ < bw; ++kq) {
#pragma unroll
        for (int kk = 0; kk < CQ; ++kk) {
            const int k = kq * CQ + kk;
            if (k >= bw) break;
            const T yk = __shfl_sync(0xffffffffu, y[kk], base | kq);
            const T* l = sL + k * SLD<T, W>::value + q * (CQ + Skew<T>::value);
#pragma unroll
            for (int ii = 0; ii < CQ; ++ii) y[ii] -= l[ii] * yk;
        }
    }
}

// The same sweeps for W = 128 with four lines per lane: the 16 lanes of a
// half-warp share four lines, lane c holding entries [8c, 8c + 8) of each,
// so that a staged row (column) read from shared memory serves four lines
// (two 16-byte loads per lane and step instead of eight; the staged layout
// sidx<float, 128> puts the eight chunks of a quarter-warp in distinct bank
// quads).  The owner of entry k shuffles its four values to the half-warp.
__device__ __forceinline__ void sweep_rows4(float (&x)[4][8], const float* sU, const float* rd, int bw, int kc_end) {
    // Steps past bw are no-ops (zero staged rows, rd = 0, zero entries), so
    // whole chunks of 8 run unguarded; the next step's row and rd are loaded
    // one step ahead, and the update of the next step's pivot entry comes
    // first.  Chunks [0, kc_end) only.
    const int lane = threadIdx.x & 31, c = lane & 15, base = lane & 16;
    const int nk = min(cdiv(bw, 8), kc_end);
    float4 n0 = *reinterpret_cast<const float4*>(sU + sidx<float, 128>(0, 8 * c));
    float4 n1 = *reinterpret_cast<const float4*>(sU + sidx<float, 128>(0, 8 * c) + 4);
    float nr = rd[0];
#pragma unroll 1
    for (int kc = 0; kc < nk; ++kc) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            const int k = kc * 8 + kk;
            const float4 u0 = n0, u1 = n1;
            const float r = nr;
            const int kn = k + 1 < 128 ? k + 1 : k;
            n0 = *reinterpret_cast<const float4*>(sU + sidx<float, 128>(kn, 8 * c));
            n1 = *reinterpret_cast<const float4*>(sU + sidx<float, 128>(kn, 8 * c) + 4);
            nr = rd[kn];
            float xk[4];
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                if (c == kc) x[l][kk] *= r;
                xk[l] = __shfl_sync(0xffffffffu, x[l][kk], base | kc);
            }
            const float uv[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
            const int jn = (kk + 1) & 7;
#pragma unroll
            for (int l = 0; l < 4; ++l) x[l][jn] -= xk[l] * uv[jn];
#pragma unroll
            for (int l = 0; l < 4; ++l)
#pragma unroll
                for (int jj = 0; jj < 8; ++jj)
                    if (jj != jn) x[l][jj] -= xk[l] * uv[jj];
        }
    }
}

__device__ __forceinline__ void sweep_cols4(float (&y)[4][8], const float* sL, int bw, int kc_end) {
    const int lane = threadIdx.x & 31, c = lane & 15, base = lane & 16;
    const int nk = min(cdiv(bw, 8), kc_end);
    float4 n0 = *reinterpret_cast<const float4*>(sL + sidx<float, 128>(0, 8 * c));
    float4 n1 = *reinterpret_cast<const float4*>(sL + sidx<float, 128>(0, 8 * c) + 4);
#pragma unroll 1
    for (int kc = 0; kc < nk; ++kc) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            const int k = kc * 8 + kk;
            const float4 l0 = n0, l1 = n1;
            const int kn = k + 1 < 128 ? k + 1 : k;
            n0 = *reinterpret_cast<const float4*>(sL + sidx<float, 128>(kn, 8 * c));
            n1 = *reinterpret_cast<const float4*>(sL + sidx<float, 128>(kn, 8 * c) + 4);
            float yk[4];
#pragma unroll
            for (int l = 0; l < 4; ++l) yk[l] = __shfl_sync(0xffffffffu, y[l][kk], base | kc);
            const float lv[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
            const int jn = (kk + 1) & 7;
#pragma unroll
            for (int l = 0; l < 4; ++l) y[l][jn] -= lv[jn] * yk[l];
#pragma unroll
            for (int l = 0; l < 4; ++l)
#pragma unroll
                for (int ii = 0; ii < 8; ++ii)
                    if (ii != jn) y[l][ii] -= lv[ii] * yk[l];
        }
    }
}

// Second phase of the 128-wide sweeps: from step 64 on only entries 64..127
// are still updated, so lane c of a half-warp takes entries [64 + 4c,
// 64 + 4c + 4) of the same four lines (moved there from lane 8 + c / 2),
// four per lane instead of eight.  Entries below 64 are final after the
// first phase and stay with their lanes.
__device__ __forceinline__ void sweep_to_hi(const float (&x)[4][8], float (&x2)[4][4]) {
    const int lane = threadIdx.x & 31, c = lane & 15, src = (lane & 16) | (8 + (c >> 1));
#pragma unroll
    for (int l = 0; l < 4; ++l)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float v0 = __shfl_sync(0xffffffffu, x[l][q], src), v1 = __shfl_sync(0xffffffffu, x[l][4 + q], src);
            x2[l][q] = (c & 1) ? v1 : v0;
        }
}

__device__ __forceinline__ void sweep_rows4_hi(float (&x)[4][4], const float* sU, const float* rd, int bw) {
    const int lane = threadIdx.x & 31, c = lane & 15, base = lane & 16;
    const int nk = min(cdiv(bw - 64, 4), 8);   // steps 64..95
    float4 n0 = *reinterpret_cast<const float4*>(sU + sidx<float, 128>(64, 64 + 4 * c));
    float nr = rd[64];
#pragma unroll 1
    for (int kc = 0; kc < nk; ++kc) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const int k = 64 + kc * 4 + kk;
            const float4 u0 = n0;
            const float r = nr;
            const int kn = k + 1 < 128 ? k + 1 : k;
            n0 = *reinterpret_cast<const float4*>(sU + sidx<float, 128>(kn, 64 + 4 * c));
            nr = rd[kn];
            float xk[4];
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                if (c == kc) x[l][kk] *= r;
                xk[l] = __shfl_sync(0xffffffffu, x[l][kk], base | kc);
            }
            const float uv[4] = {u0.x, u0.y, u0.z, u0.w};
            const int jn = (kk + 1) & 3;
#pragma unroll
            for (int l = 0; l < 4; ++l) x[l][jn] -= xk[l] * uv[jn];
#pragma unroll
            for (int l = 0; l < 4; ++l)
#pragma unroll
                for (int jj = 0; jj < 4; ++jj)
                    if (jj != jn) x[l][jj] -= xk[l] * uv[jj];
        }
    }
}

__device__ __forceinline__ void sweep_cols4_hi(float (&y)[4][4], const float* sL, int bw) {
    const int lane = threadIdx.x & 31, c = lane & 15, base = lane & 16;
    const int nk = min(cdiv(bw - 64, 4), 8);   // steps 64..95
    float4 n0 = *reinterpret_cast<const float4*>(sL + sidx<float, 128>(64, 64 + 4 * c));
#pragma unroll 1
    for (int kc = 0; kc < nk; ++kc) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const int k = 64 + kc * 4 + kk;
            const float4 l0 = n0;
            const int kn = k + 1 < 128 ? k + 1 : k;
            n0 = *reinterpret_cast<const float4*>(sL + sidx<float, 128>(kn, 64 + 4 * c));
            float yk[4];
#pragma unroll
            for (int l = 0; l < 4; ++l) yk[l] = __shfl_sync(0xffffffffu, y[l][kk], base | kc);
            const float lv[4] = {l0.x, l0.y, l0.z, l0.w};
            const int jn = (kk + 1) & 3;
#pragma unroll
            for (int l = 0; l < 4; ++l) y[l][jn] -= lv[jn] * yk[l];
#pragma unroll
            for (int l = 0; l < 4; ++l)
#pragma unroll
                for (int ii = 0; ii < 4; ++ii)
                    if (ii != jn) y[l][ii] -= lv[ii] * yk[l];
        }
    }
}

// Third phase, from step 96 on: entries 96..127, lane c taking [96 + 2c,
// 96 + 2c + 2) (moved from lane 8 + c / 2 of the second phase).
__device__ __forceinline__ void sweep_to_top(const float (&x2)[4][4], float (&x3)[4][2]) {
    const int lane = threadIdx.x & 31, c = lane & 15, src = (lane & 16) | (8 + (c >> 1));
#pragma unroll
    for (int l = 0; l < 4; ++l)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float v0 = __shfl_sync(0xffffffffu, x2[l][q], src), v1 = __shfl_sync(0xffffffffu, x2[l][2 + q], src);
            x3[l][q] = (c & 1) ? v1 : v0;
        }
}

template <bool ROWS>
__device__ __forceinline__ void sweep_top(float (&x)[4][2], const float* sT, const float* rd, int bw) {
    const int lane = threadIdx.x & 31, c = lane & 15, base = lane & 16;
    const int nk = cdiv(bw - 96, 2);
    float2 n0 = *reinterpret_cast<const float2*>(sT + sidx<float, 128>(96, 96 + 2 * c));
    float nr = ROWS ? rd[96] : 0.f;
#pragma unroll 1
    for (int kc = 0; kc < nk; ++kc) {
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            const int k = 96 + kc * 2 + kk;
            const float2 u0 = n0;
            const float r = nr;
            const int kn = k + 1 < 128 ? k + 1 : k;
            n0 = *reinterpret_cast<const float2*>(sT + sidx<float, 128>(kn, 96 + 2 * c));
            if (ROWS) nr = rd[kn];
            float xk[4];
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                if (ROWS && c == kc) x[l][kk] *= r;
                xk[l] = __shfl_sync(0xffffffffu, x[l][kk], base | kc);
            }
            const float uv[2] = {u0.x, u0.y};
            const int jn = (kk + 1) & 1;
#pragma unroll
            for (int l = 0; l < 4; ++l) x[l][jn] -= xk[l] * uv[jn];
#pragma unroll
            for (int l = 0; l < 4; ++l) x[l][kk] -= xk[l] * uv[kk];
        }
    }
}

// Asynchronous element copy global -> shared (cp.async, 4 or 8 bytes); a
// copy with valid = false writes zero and reads nothing.
template <typename T>
__device__ __forceinline__ void cp_elem(T* dst, const T* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(T) == 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(valid ? 4 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(valid ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// sU and rd from the factored block (column-major at blkp, leading dimension
// ld); the triangle is copied asynchronously (the caller waits with
// cp_wait_all and a barrier before using it).
// Staging order: a warp copies 8 consecutive rows k x 4 consecutive entries
// j (global: 4 columns, 32 contiguous bytes each; shared: 32 distinct banks).
template <int W>
__device__ __forceinline__ void stage_coords(int e, int& k, int& j) {
    const int sub = e & 31, b = e >> 5;
    k = (b % (W / 8)) * 8 + (sub & 7);
    j = (b / (W / 8)) * 4 + (sub >> 3);
}

template <typename T, int W>
__device__ __forceinline__ void stage_upper(T* sU, T* rd, const T* blkp, ll ld, int bw) {
    for (int e = threadIdx.x; e < W * W; e += blockDim.x) {
        int k, j;
        stage_coords<W>(e, k, j);
        const bool v = j > k && j < bw;
        cp_elem(&sU[sidx<T, W>(k, j)], v ? blkp + (ll)j * ld + k : blkp, v);
    }
    for (int k = threadIdx.x; k < W; k += blockDim.x) rd[k] = k < bw ? T(1) / blkp[(ll)k * ld + k] : T(0);
    cp_wait_all();
}

// sL from the factored block with the rows of each piece, in the columns
// left of the piece, put in the piece's pivoted order: the interchanges of
// all pieces then act once, as a gather by gmap, before the sweep (the
// reference applies a piece's interchanges when the forward elimination
// reaches it; moving them ahead of the earlier pieces' updates permutes
// those updates' rows the same way).
template <typename T, int W>
__device__ __forceinline__ void stage_lower(T* sL, const T* blkp, ll ld, int bw, const int* gmap, const int* pa) {
    for (int e = threadIdx.x; e < W * W; e += blockDim.x) {
        int k, i;
        stage_coords<W>(e, k, i);
        const bool v = i > k && i < bw;
        cp_elem(&sL[sidx<T, W>(k, i)], v ? blkp + (ll)k * ld + (k < pa[i] ? gmap[i] : i) : blkp, v);
    }
    cp_wait_all();
}

// Packed copy of one panel line for the tensor-core updates (FP32 fronts
// with a pack): the line's entries k < nch * KCH, held CQ per lane from
// q * CQ, split into TF32 hi / lo at tile `t`, line `i` of the block's pack.
template <int CQ>
__device__ __forceinline__ void pack_line(unsigned char* base, int t, int i, int q, int nch, const float (&v)[CQ]) {
#pragma unroll
    for (int g = 0; g < CQ / 4; ++g) {
        const int k = q * CQ + 4 * g;
        if (k < nch * umma::KCH) {
            unsigned char* dst = base + ((ll)t * nch + k / umma::KCH) * umma::PCHUNK + umma::packed_offset(i, k % umma::KCH);
            uint32_t h[4], l[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                h[e] = umma::tf32_rna(v[4 * g + e]);
                l[e] = umma::tf32_rna(v[4 * g + e] - __uint_as_float(h[e]));
            }
            *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<uint4*>(dst + umma::OPB) = make_uint4(l[0], l[1], l[2], l[3]);
        }
    }
}

// BF16 form of pack_line: the line's entries times `scale` (a power of two)
// as BF16 at tile `t`, line `i` of the block's BF16 pack.
template <int CQ>
__device__ __forceinline__ void pack_line16(unsigned char* base, int t, int i, int q, int nch, const float (&v)[CQ],
                                            float scale) {
#pragma unroll
    for (int g = 0; g < CQ / 4; ++g) {
        const int k = q * CQ + 4 * g;
        if (k < nch * umma::KCH) {
            unsigned char* dst =
                base + ((ll)t * nch + k / umma::KCH) * umma::PCHUNK16 + umma::packed_offset16(i, k % umma::KCH);
            *reinterpret_cast<uint2*>(dst) = make_uint2(umma::pack_bf16x2(v[4 * g] * scale, v[4 * g + 1] * scale),
                                                        umma::pack_bf16x2(v[4 * g + 2] * scale, v[4 * g + 3] * scale));
        }
    }
}

// Per-block exponent of the BF16 panel scaling: e = floor(E / 2), E the
// binary exponent of the largest |diagonal entry of U_B|; the L panel is
// packed times 2^e and the U panel times 2^-e, so L U^T is unchanged and both
// scaled panels are about 2^(E/2) in size.  Every CTA of the block's panel
// launch computes the same e from the final diagonal block (all threads
// call; contains a barrier).
__device__ __forceinline__ int block_scale_exp(const float* blkp, int ld, int bw, int* smax) {
    if (threadIdx.x == 0) *smax = 0;
    __syncthreads();
    if ((int)threadIdx.x < bw) atomicMax(smax, __float_as_int(fabsf(blkp[(ll)threadIdx.x * ld + threadIdx.x])));
    __syncthreads();
    const int E = ((*smax >> 23) & 255) - 127;
    return E >> 1;
}

// The panels of a block of more than 64 columns in FP32 (W = 128), four
// lines per lane (sweep_rows4 / sweep_cols4): lane c of half-warp h holds
// entries [8c, 8c + 8) of the tile's lines 4h .. 4h + 3.  Same tiles,
// operations and outputs as the generic form in k_block_panel; the row
// sources of the block's interchanges (gmap | pa << 8 per block column) come
// from k_block_lu_f32 through bmap.  The 64 lines of the tile pass through a
// shared-memory copy sX (line li, entry j at li * PT_LD + j) so that the
// global loads, stores and packed writes are coalesced: a warp moves 8 rows
// x 4 columns of a column-major array (32-byte runs), and the packed writes
// of 8 lines x 4 entries form 512 contiguous bytes.
constexpr int PT_LD = 132;   // 16-byte rows, 4 words apart in the bank cycle
constexpr int PT_LINES = 64;  // lines per CTA (4 * PT_LINES threads)
constexpr int PT_SMEM = PT_LINES * PT_LD * 4;

// Element e of a PT_LINES-line x 128-entry tile: a warp copies 8
// consecutive entries x 4 lines when `entries_fast`, else 8 lines x 4
// entries.
__device__ __forceinline__ void tile_coords(int e, bool entries_fast, int& li, int& j) {
    const int sub = e & 31, b = e >> 5;
    if (entries_fast) {
        j = (b % 16) * 8 + (sub & 7);
        li = (b / 16) * 4 + (sub >> 3);
    } else {
        li = (b % (PT_LINES / 8)) * 8 + (sub & 7);
        j = (b / (PT_LINES / 8)) * 4 + (sub >> 3);
    }
}

// Packed copy of the tile's lines [0, nl) from sX; line li goes to pack tile
// t(li), line i(li) (computed by `where`).
template <typename Where>
__device__ __forceinline__ void pack_tile(unsigned char* base, const float* sX, int nl, int nch, Where where) {
    for (int item = threadIdx.x; item < PT_LINES * 32; item += blockDim.x) {   // 8 lines x 32 groups of 4 entries
        const int g = (item >> 3) & 31, li = (item >> 8) * 8 + (item & 7);
        if (li >= nl || 4 * g >= nch * umma::KCH) continue;
        int t, i;
        where(li, t, i);
        const int k = 4 * g;
        const float4 v = *reinterpret_cast<const float4*>(sX + li * PT_LD + k);
        const float vv[4] = {v.x, v.y, v.z, v.w};
        uint32_t hh[4], ll_[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            hh[e] = umma::tf32_rna(vv[e]);
            ll_[e] = umma::tf32_rna(vv[e] - __uint_as_float(hh[e]));
        }
        unsigned char* dst = base + ((ll)t * nch + k / umma::KCH) * umma::PCHUNK + umma::packed_offset(i, k % umma::KCH);
        *reinterpret_cast<uint4*>(dst) = make_uint4(hh[0], hh[1], hh[2], hh[3]);
        *reinterpret_cast<uint4*>(dst + umma::OPB) = make_uint4(ll_[0], ll_[1], ll_[2], ll_[3]);
    }
}

// BF16 form of pack_tile: entries times `scale`, one BF16 part per chunk.
template <typename Where>
__device__ __forceinline__ void pack_tile16(unsigned char* base, const float* sX, int nl, int nch, float scale,
                                            Where where) {
    for (int item = threadIdx.x; item < PT_LINES * 32; item += blockDim.x) {
        const int g = (item >> 3) & 31, li = (item >> 8) * 8 + (item & 7);
        if (li >= nl || 4 * g >= nch * umma::KCH) continue;
        int t, i;
        where(li, t, i);
        const int k = 4 * g;
        const float4 v = *reinterpret_cast<const float4*>(sX + li * PT_LD + k);
        unsigned char* dst =
            base + ((ll)t * nch + k / umma::KCH) * umma::PCHUNK16 + umma::packed_offset16(i, k % umma::KCH);
        *reinterpret_cast<uint2*>(dst) =
            make_uint2(umma::pack_bf16x2(v.x * scale, v.y * scale), umma::pack_bf16x2(v.z * scale, v.w * scale));
    }
}

__device__ __forceinline__ void block_panel128(float* fac, const int* bmap, const Sched& S, const DFront& F, int blk,
                                               int tile, unsigned char* pack, float* sT, float* sX, float* rd,
                                               int* gmap, int* pa, int bf16, int* smax, float* sd) {
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk], bw = c1 - c0;
    const int tid = threadIdx.x, c = tid & 15, line0 = (tid >> 4) * 4;
    const int nL = cdiv(F.ld - c1, PT_LINES), nUa = cdiv(F.nf - c1, PT_LINES);
    const float* blkp = fac + F.loff + (ll)c0 * F.ld + c0;
    const int nch = cdiv(bw, umma::KCH);
    const int n1 = cdiv(F.nf - c1, umma::TM);
    if (tile < nL) {
        const int rb0 = c1 + tile * PT_LINES, nl = min(PT_LINES, F.ld - rb0);
        float* xb = fac + F.loff + (ll)c0 * F.ld + rb0;   // line li, entry j at xb[j * ld + li]
        for (int e = tid; e < PT_LINES * 128; e += PT_LINES * 4) {
            int li, j;
            tile_coords(e, false, li, j);
            const bool v = li < nl && j < bw;
            cp_elem(&sX[li * PT_LD + j], v ? xb + (ll)j * F.ld + li : xb, v);
        }
        if (S.sym && tid < bw) sd[tid] = blkp[(ll)tid * F.ld + tid];   // U(j, j) for the U side
        stage_upper<float, 128>(sT, rd, blkp, F.ld, bw);   // waits for all copies
        __syncthreads();
        float x[4][8];
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const float4 a0 = *reinterpret_cast<const float4*>(sX + (line0 + l) * PT_LD + 8 * c);
            const float4 a1 = *reinterpret_cast<const float4*>(sX + (line0 + l) * PT_LD + 8 * c + 4);
            x[l][0] = a0.x; x[l][1] = a0.y; x[l][2] = a0.z; x[l][3] = a0.w;
            x[l][4] = a1.x; x[l][5] = a1.y; x[l][6] = a1.z; x[l][7] = a1.w;
        }
        sweep_rows4(x, sT, rd, bw, 8);   // steps 0..63
        float x2[4][4];
        sweep_to_hi(x, x2);
        sweep_rows4_hi(x2, sT, rd, bw);  // steps 64..95
        float x3[4][2];
        sweep_to_top(x2, x3);
        sweep_top<true>(x3, sT, rd, bw);  // steps 96..
#pragma unroll
        for (int l = 0; l < 4; ++l) {   // entries 0..63, 64..95, 96..127 from the three phases
            float* dst = sX + (line0 + l) * PT_LD;
            if (c < 8) {
                *reinterpret_cast<float4*>(dst + 8 * c) = make_float4(x[l][0], x[l][1], x[l][2], x[l][3]);
                *reinterpret_cast<float4*>(dst + 8 * c + 4) = make_float4(x[l][4], x[l][5], x[l][6], x[l][7]);
                *reinterpret_cast<float4*>(dst + 64 + 4 * c) = make_float4(x2[l][0], x2[l][1], x2[l][2], x2[l][3]);
            }
            *reinterpret_cast<float2*>(dst + 96 + 2 * c) = make_float2(x3[l][0], x3[l][1]);
        }
        __syncthreads();
        for (int e = tid; e < PT_LINES * 128; e += PT_LINES * 4) {
            int li, j;
            tile_coords(e, false, li, j);
            if (li < nl && j < bw) xb[(ll)j * F.ld + li] = sX[li * PT_LD + j];
        }
        const ll off = S.blk_lpack[blk];
        auto whereL = [&](int li, int& t, int& i) {
            const int r = rb0 + li;
            t = r < F.nf ? (r - c1) / umma::TM : n1 + (r - F.nf) / umma::TM;
            i = r < F.nf ? (r - c1) % umma::TM : (r - F.nf) % umma::TM;
        };
        const int e = (off >= 0 && bf16) ? block_scale_exp(blkp, F.ld, bw, smax) : 0;
        if (off >= 0 && bf16) pack_tile16(pack + (off >> 2), sX, nl, nch, umma::exp2i(e), whereL);
        else if (off >= 0) pack_tile(pack + off, sX, nl, nch, whereL);
        if (S.sym) {   // the U side: U(c0 + j, r) = U(j, j) L(r, c0 + j), stored and packed
            __syncthreads();   // the L pack has read the tile
            for (int q = tid; q < PT_LINES * 128; q += PT_LINES * 4) {
                int li, j;
                tile_coords(q, true, li, j);
                if (li < nl && j < bw) sX[li * PT_LD + j] *= sd[j];
            }
            __syncthreads();
            for (int q = tid; q < PT_LINES * 128; q += PT_LINES * 4) {   // rows r < nf: column r of Lf
                int li, j;
                tile_coords(q, true, li, j);
                const int r = rb0 + li;
                if (li < nl && j < bw && r < F.nf) fac[F.loff + (ll)r * F.ld + c0 + j] = sX[li * PT_LD + j];
            }
            for (int q = tid; q < PT_LINES * 128; q += PT_LINES * 4) {   // rows r >= nf: U12 in Uf
                int li, j;
                tile_coords(q, false, li, j);
                const int r = rb0 + li;
                if (li < nl && j < bw && r >= F.nf) fac[F.uoff + (ll)(c0 + j) * F.m + (r - F.nf)] = sX[li * PT_LD + j];
            }
            const ll offu = S.blk_upack[blk];
            if (offu >= 0 && bf16) pack_tile16(pack + (offu >> 2), sX, nl, nch, umma::exp2i(-e), whereL);
            else if (offu >= 0) pack_tile(pack + offu, sX, nl, nch, whereL);
        }
    } else {
        if (tid < bw) {   // the block's row sources, from k_block_lu_f32
            const int v = bmap[F.f + c0 + tid];
            gmap[tid] = v & 255;
            pa[tid] = v >> 8;
        }
        __syncthreads();
        const bool inner = tile < nL + nUa;
        const int cb0 = inner ? c1 + (tile - nL) * PT_LINES : (tile - nL - nUa) * PT_LINES;
        const int nl = min(PT_LINES, (inner ? F.nf : F.m) - cb0);
        // line li, block row R at yb[li * ls + R * rs]
        float* yb = inner ? fac + F.loff + (ll)cb0 * F.ld + c0 : fac + F.uoff + (ll)c0 * F.m + cb0;
        const ll ls = inner ? (ll)F.ld : 1, rs = inner ? 1 : (ll)F.m;
        for (int e = tid; e < PT_LINES * 128; e += PT_LINES * 4) {
            int li, R;
            tile_coords(e, inner, li, R);
            const bool v = li < nl && R < bw;
            cp_elem(&sX[li * PT_LD + R], v ? yb + li * ls + (ll)gmap[R] * rs : yb, v);
        }
        stage_lower<float, 128>(sT, blkp, F.ld, bw, gmap, pa);   // waits for all copies
        __syncthreads();
        float y[4][8];
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const float4 a0 = *reinterpret_cast<const float4*>(sX + (line0 + l) * PT_LD + 8 * c);
            const float4 a1 = *reinterpret_cast<const float4*>(sX + (line0 + l) * PT_LD + 8 * c + 4);
            y[l][0] = a0.x; y[l][1] = a0.y; y[l][2] = a0.z; y[l][3] = a0.w;
            y[l][4] = a1.x; y[l][5] = a1.y; y[l][6] = a1.z; y[l][7] = a1.w;
        }
        sweep_cols4(y, sT, bw, 8);
        float y2[4][4];
        sweep_to_hi(y, y2);
        sweep_cols4_hi(y2, sT, bw);
        float y3[4][2];
        sweep_to_top(y2, y3);
        sweep_top<false>(y3, sT, nullptr, bw);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            float* dst = sX + (line0 + l) * PT_LD;
            if (c < 8) {
                *reinterpret_cast<float4*>(dst + 8 * c) = make_float4(y[l][0], y[l][1], y[l][2], y[l][3]);
                *reinterpret_cast<float4*>(dst + 8 * c + 4) = make_float4(y[l][4], y[l][5], y[l][6], y[l][7]);
                *reinterpret_cast<float4*>(dst + 64 + 4 * c) = make_float4(y2[l][0], y2[l][1], y2[l][2], y2[l][3]);
            }
            *reinterpret_cast<float2*>(dst + 96 + 2 * c) = make_float2(y3[l][0], y3[l][1]);
        }
        __syncthreads();
        for (int e = tid; e < PT_LINES * 128; e += PT_LINES * 4) {
            int li, R;
            tile_coords(e, inner, li, R);
            if (li < nl && R < bw) yb[li * ls + (ll)R * rs] = sX[li * PT_LD + R];
        }
        const ll off = S.blk_upack[blk];
        auto whereU = [&](int li, int& t, int& i) {
            const int col = cb0 + li;
            t = inner ? (col - c1) / umma::TM : n1 + col / umma::TM;
            i = inner ? (col - c1) % umma::TM : col % umma::TM;
        };
        if (off >= 0 && bf16) {
            const float scale = umma::exp2i(-block_scale_exp(blkp, F.ld, bw, smax));
            pack_tile16(pack + (off >> 2), sX, nl, nch, scale, whereU);
        } else if (off >= 0) {
            pack_tile(pack + off, sX, nl, nch, whereU);
        }
    }
}

// Panels of block `step` (block width bw <= W): 64-row tiles of the L panel
// below the block, X := X inv(U_B) (the reference's trsm 'r','u','n','n' of
// every piece, with the earlier pieces' updates X_p -= X_<p U_<p,p), and
// 64-column tiles of the U panel to its right, inside the front (Lf) and in
// U12 (Uf): Y := inv(L_B) P_B Y (_luswap! and trsm 'r','l','t','u' of every
// piece, with Y_p -= L_p,<p Y_<p).  One line per 4 lanes (W = 32, 64); FP32
// blocks wider than 64 columns take block_panel128 (four lines per 16
// lanes, PT_LINES-line tiles).  For FP32 fronts with a pack (blk_lpack >= 0)
// the lines are also written, split into TF32 hi / lo, to the packed tiles
// that the tensor-core updates read: rows of the L panel tiled from c1
// ([c1, nf)) and from nf ([nf, ld)), columns of the U panel from c1
// ([c1, nf)) and from 0 (U12).
// Dynamic shared memory: W * SLD(W) T's (plus the line tile of
// block_panel128).
// Panel tiles of one launch part: 0 every tile; 1 the near ones (the first
// two line tiles of the rows below the block and of the front columns right
// of it: the lines the next block's diagonal region is updated from); 2 the
// others.  Tiles of 64 lines: L rows first (nL tiles), then front columns
// (nUa), then U12 columns.
__host__ __device__ __forceinline__ int panel_tile(int part, int tile, int nL, int nUa, bool sym) {
    if (part == 0) return tile;
    const int aL = min(2, nL), aU = sym ? 0 : min(2, nUa);
    if (part == 1) return tile < aL ? tile : nL + (tile - aL);
    return tile < nL - aL ? aL + tile : nL + aU + (tile - (nL - aL));
}

// FP64 panels.  A double multiply-add takes a warp 64 cycles and an SM 19 per
// warp, so the panels are bound by how many there are and how many SMs share
// them: a line (row of X, column of Y) is held by eight lanes, lane q entries
// q, q + 8, .. (cyclic, so that step k touches only the entries after it: 288
// instead of 1024 multiply-adds per 64-step sweep), and a CTA of four warps
// takes 16 lines (64 before), four times as many CTAs for the few fronts near
// the root.  rows: X := X inv(U_B), entry k scaled by 1 / U(k, k) at its step
// (rows of U_B over their diagonal would spare that multiplication, but overflow
// where columns of A differ by more than the exponent range, and round once
// more); cols: Y := inv(L_B) P_B Y.
// 48^3 convection-diffusion: 18.0 -> 10.0 ms for all panels (FP64-bound: 5.6 ms
// at the full rate, without the scaling; 9.8 with the rows over their diagonal).
constexpr int PD_LINES = 16, PD_LANES = 8;
template <int W>
__device__ __forceinline__ void sweep_f64(double (&x)[W / PD_LANES], const double* sT, const double* rd, int bw) {   // rd null: cols
    constexpr int CQ = W / PD_LANES;
    const int lane = threadIdx.x & 31, q = lane & (PD_LANES - 1), base = lane & ~(PD_LANES - 1);
#pragma unroll
    for (int k = 0; k < W; ++k)
        if (k < bw) {
            if (rd && q == k % PD_LANES) x[k / PD_LANES] *= rd[k];
            if (k == bw - 1) break;
            const double xk = __shfl_sync(0xffffffffu, x[k / PD_LANES], base | (k % PD_LANES));
            const double* t = sT + k * (W + 1) + q;
#pragma unroll
            for (int jj = (k + 1) / PD_LANES; jj < CQ; ++jj) x[jj] -= xk * t[jj * PD_LANES];   // zero up to the diagonal
        }
}

// The largest exponent field of the finite entries of every U row (L column)
// over the lines of a CTA into every second entry of rexp, from which the
// slices of the tensor-core updates take their scaling along the block.  (An
// infinity's would leave nothing of the columns beside it.)
template <int CQ>
__device__ __forceinline__ void oz_row_max(const double (&y)[CQ], bool ok, int bw, int* smx, int* rexp) {
    const int lane = threadIdx.x & 31, q = lane & (PD_LANES - 1);
    if ((int)threadIdx.x < PD_LANES * CQ) smx[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < CQ; ++i) {
        int e = ok ? (__double2hiint(y[i]) >> 20) & 0x7ff : 0;
        e = e == 0x7ff ? 0 : e;
        e = max(e, __shfl_xor_sync(0xffffffffu, e, 8));
        e = max(e, __shfl_xor_sync(0xffffffffu, e, 16));
        if (lane < PD_LANES && e > 0) atomicMax(&smx[i * PD_LANES + q], e);
    }
    __syncthreads();
    if ((int)threadIdx.x < bw && smx[threadIdx.x] > 0) atomicMax(&rexp[2 * threadIdx.x], smx[threadIdx.x]);
}

template <int W>
__global__ void __launch_bounds__(128) k_block_panel_f64(double* fac, const int* ipiv, Sched S, Launch L, int step, int* rexp) {
    constexpr int CQ = W / PD_LANES, LD = W + 1;   // staged row k at k * LD
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sT = reinterpret_cast<double*>(smem_raw);
    __shared__ double sd[W], rd[W];   // U(k, k) and its reciprocal
    __shared__ int q0[W + 1], gmap[W], pa[W], smx[W];
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    const int blk = F.block0 + step;
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk], bw = c1 - c0;
    const int p0 = S.blk_p0[blk], np = S.blk_np[blk];
    const int tid = threadIdx.x, line = tid / PD_LANES, q = tid & (PD_LANES - 1);
    const int nL = cdiv(F.ld - c1, PD_LINES), nUa = cdiv(F.nf - c1, PD_LINES);
    const double* blkp = fac + F.loff + (ll)c0 * F.ld + c0;
    double x[CQ];
    if (tile < nL) {
        const int r = c1 + tile * PD_LINES + line;
        const bool ok = r < F.ld;
        double* xp = fac + F.loff + (ll)c0 * F.ld + r;   // row r, block column j at xp[j * ld]
#pragma unroll
        for (int jj = 0; jj < CQ; ++jj) {   // in flight while the triangle is staged
            const int j = jj * PD_LANES + q;
            x[jj] = (ok && j < bw) ? xp[(ll)j * F.ld] : 0.0;
        }
        if (tid < bw) {
            const double d = blkp[(ll)tid * F.ld + tid];
            sd[tid] = d;
            rd[tid] = 1.0 / d;
        }
        __syncthreads();
        for (int e = tid; e < W * W; e += 128) {
            const int k = e % W, j = e / W;   // contiguous in k
            sT[k * LD + j] = j > k && j < bw ? blkp[(ll)j * F.ld + k] : 0.0;
        }
        __syncthreads();
        sweep_f64<W>(x, sT, rd, bw);
#pragma unroll
        for (int jj = 0; jj < CQ; ++jj) {
            const int j = jj * PD_LANES + q;
            if (ok && j < bw) xp[(ll)j * F.ld] = x[jj];
        }
        if (S.blk_upack[blk] >= 0) oz_row_max<CQ>(x, ok, bw, smx, rexp + 2 * (F.f + c0) + 1);
        if (S.sym) {   // symmetric form: the U side, U(c0 + j, r) = U(j, j) L(r, c0 + j)
#pragma unroll
            for (int jj = 0; jj < CQ; ++jj) {
                const int j = jj * PD_LANES + q;
                if (j < bw) x[jj] *= sd[j];
                if (ok && j < bw) {
                    if (r < F.nf) fac[F.loff + (ll)r * F.ld + c0 + j] = x[jj];
                    else fac[F.uoff + (ll)(c0 + j) * F.m + (r - F.nf)] = x[jj];
                }
            }
            if (S.blk_upack[blk] >= 0) oz_row_max<CQ>(x, ok, bw, smx, rexp + 2 * (F.f + c0));
        }
    } else {
        for (int k = tid; k <= np; k += 128) q0[k] = S.xsuper[p0 + k] - F.f - c0;
        __syncthreads();
        block_gather_map(ipiv + F.f + c0, q0, np, gmap, pa);
        __syncthreads();
        const bool inner = tile < nL + nUa;
        const int col = inner ? c1 + (tile - nL) * PD_LINES + line : (tile - nL - nUa) * PD_LINES + line;
        const bool ok = inner ? col < F.nf : col < F.m;
        // block row k of this column at cp[k * stride]
        double* cp = inner ? fac + F.loff + (ll)col * F.ld + c0 : fac + F.uoff + (ll)c0 * F.m + col;
        const ll stride = inner ? 1 : (ll)F.m;
#pragma unroll
        for (int jj = 0; jj < CQ; ++jj) {   // in flight while the triangle is staged
            const int k = jj * PD_LANES + q;
            x[jj] = (ok && k < bw) ? cp[(ll)gmap[k] * stride] : 0.0;
        }
        for (int e = tid; e < W * W; e += 128) {   // rows left of a piece in its pivoted order, as stage_lower
            const int i = e % W, k = e / W;
            sT[k * LD + i] = i > k && i < bw ? blkp[(ll)k * F.ld + (k < pa[i] ? gmap[i] : i)] : 0.0;
        }
        __syncthreads();
        sweep_f64<W>(x, sT, nullptr, bw);
#pragma unroll
        for (int jj = 0; jj < CQ; ++jj) {
            const int k = jj * PD_LANES + q;
            if (ok && k < bw) cp[(ll)k * stride] = x[jj];
        }
        if (S.blk_upack[blk] >= 0) oz_row_max<CQ>(x, ok, bw, smx, rexp + 2 * (F.f + c0));
    }
}

// ---------------------------------------------------------------------------
// FP64 block LU by a whole CTA (blocks of 33..64 columns; one CTA per front),
// in the groups of k_block_lu_f32.  What bounds it is the number of double
// multiply-adds (64 cycles each for a warp, 19 for an SM): every step touches
// only rows and columns that are left, spread over the SM's four quarters:
// a group's rows and columns in four warps of eight columns each (a lane per
// row; the reciprocals of all candidates, 350 cycles, beside the search), its
// L21 rows and U12 columns eight lanes per line as in the panels, the
// rank-w update over all warps.  The form before it updated every row of the
// block in every step: all block LUs of the 48^3 convection-diffusion system
// 15.8 -> 13.3 ms, of the 256 x 256 diffusion system 2.0 -> 1.8 ms.
// ---------------------------------------------------------------------------
constexpr int LU64_THREADS = 256;
struct Lu64Smem {   // offsets in doubles
    static constexpr int BM = 64, LD = BM + 1, LT = LU_G + 1;
    static constexpr int a = 0;                       // A(i, j) at a + j * LD + i
    static constexpr int ex = a + BM * LD + 1;        // multipliers of the group's column k by row: ex + k * BM + row
    static constexpr int t = ex + LU_G * BM;          // the group's triangles: U, row k at t + k * LT
    static constexpr int l = t + LU_G * LT;           // L11, column k at l + k * LT
    static constexpr int bytes = (l + LU_G * LT) * 8;
};

// Part 1 of a group, by warps q = 0 .. cdiv(w, 8) - 1: rows [0, nrow) (up to
// 32 RPL) and columns [0, w) at A(i, j) = A[j * LD + i], in place (rows in
// their final positions: entry (i, j) of original row r at position (j >=
// left[r] ? at[r] : r), left[r] the first column (of the group) of r's piece).
// piv: row | position << 8 of each column's pivot; at: positions; rd: pivot
// reciprocals (1 for a zero pivot).
template <int RPL>
__device__ __forceinline__ void lu64_sweep(double* A, int nrow, int w, int cend, const int* left, double* ex, double* rd,
                                           int* piv, int* at, int* zero, bool sym, int q) {
    constexpr int LD = Lu64Smem::LD, BM = Lu64Smem::BM;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, nq = cdiv(w, LU_W);
    double P[RPL][LU_W];
    int pos[RPL];
    bool act[RPL];
#pragma unroll
    for (int s = 0; s < RPL; ++s) {
        const int r = lane + 32 * s;
        pos[s] = r;
        act[s] = r < nrow;
#pragma unroll
        for (int j = 0; j < LU_W; ++j) P[s][j] = r < nrow && q * LU_W + j < w ? A[(q * LU_W + j) * LD + r] : 0.0;
    }
    auto place = [&](int k, int kr, int pp) {
#pragma unroll
        for (int s = 0; s < RPL; ++s) {
            if (pos[s] == k) pos[s] = pp;
            if (lane + 32 * s == kr) {
                pos[s] = k;
                act[s] = false;
            }
        }
    };
#pragma unroll 1
    for (int o = 0; o < q; ++o)   // follow the warps of the earlier columns
#pragma unroll 1
        for (int t = 0; t < LU_W; ++t) {
            const int k = o * LU_W + t;
            asm volatile("bar.sync %0, %1;" ::"r"(4 + t), "r"(32 * (nq - o)) : "memory");
            double l[RPL];
#pragma unroll
            for (int s = 0; s < RPL; ++s) l[s] = ex[k * BM + lane + 32 * s];
            const int pv = piv[k], kr = pv & 255;
            place(k, kr, pv >> 8);
#pragma unroll
            for (int j = 0; j < LU_W; ++j) {
                const double u = __shfl_sync(FULL, RPL == 2 && kr >= 32 ? P[RPL - 1][j] : P[0][j], kr & 31);
#pragma unroll
                for (int s = 0; s < RPL; ++s)
                    if (act[s]) P[s][j] -= l[s] * u;
            }
        }
#pragma unroll
    for (int t = 0; t < LU_W; ++t) {
        const int k = q * LU_W + t;
        if (k >= w) break;
        const int ce = __shfl_sync(FULL, cend, k);
        double rc[RPL];
        unsigned long long key[RPL], best = 0ull;
#pragma unroll
        for (int s = 0; s < RPL; ++s) {
            const bool diag = pos[s] == k, cand = act[s] && (sym ? diag : pos[s] < ce);
            rc[s] = rcp_rn(cand ? P[s][t] : 1.0);
            key[s] = pivot_key(P[s][t], cand, diag);
            best = key[s] > best ? key[s] : best;
        }
        const unsigned mh = __reduce_max_sync(FULL, (unsigned)(best >> 32));
        const unsigned ml = __reduce_max_sync(FULL, (unsigned)(best >> 32) == mh ? (unsigned)best : 0u);
        const unsigned long long mx = ((unsigned long long)mh << 32) | ml;
        unsigned p = 0xffffffffu;   // the first position that holds it
#pragma unroll
        for (int s = 0; s < RPL; ++s)
            if (key[s] == mx && (unsigned)pos[s] < p) p = (unsigned)pos[s];
        const unsigned pp = __reduce_min_sync(FULL, p);
        int kr = 0;
#pragma unroll
        for (int s = 0; s < RPL; ++s) {
            const unsigned b = __ballot_sync(FULL, act[s] && (unsigned)pos[s] == pp);
            if (b) kr = 31 - __clz(b) + 32 * s;
        }
        const bool hi = RPL == 2 && kr >= 32;
        const double pv = __shfl_sync(FULL, hi ? P[RPL - 1][t] : P[0][t], kr & 31);
        double inv = __shfl_sync(FULL, hi ? rc[RPL - 1] : rc[0], kr & 31);
        if (pv == 0.0) {   // no scaling
            inv = 1.0;
            if (lane == 0) atomicMin(zero, k);
        }
        place(k, kr, (int)pp);
        double l[RPL];
#pragma unroll
        for (int s = 0; s < RPL; ++s) {
            l[s] = P[s][t] * inv;
            ex[k * BM + lane + 32 * s] = l[s];
            if (act[s]) P[s][t] = l[s];
        }
        if (lane == 0) {
            piv[k] = kr | (int)pp << 8;
            rd[k] = inv;
        }
        if (q + 1 < nq) asm volatile("bar.arrive %0, %1;" ::"r"(4 + t), "r"(32 * (nq - q)) : "memory");
#pragma unroll
        for (int j = t + 1; j < LU_W; ++j) {
            const double u = __shfl_sync(FULL, hi ? P[RPL - 1][j] : P[0][j], kr & 31);
#pragma unroll
            for (int s = 0; s < RPL; ++s)
                if (act[s]) P[s][j] -= l[s] * u;
        }
    }
    if (q == nq - 1)
#pragma unroll
        for (int s = 0; s < RPL; ++s)
            if (lane + 32 * s < nrow) at[lane + 32 * s] = pos[s];
    asm volatile("bar.sync 12, %0;" ::"r"(32 * nq) : "memory");   // (and every warp has read its columns)
#pragma unroll
    for (int s = 0; s < RPL; ++s) {
        const int r = lane + 32 * s;
        if (r < nrow)
#pragma unroll
            for (int j = 0; j < LU_W; ++j)
                if (q * LU_W + j < w) A[(q * LU_W + j) * LD + (q * LU_W + j >= left[r] ? at[r] : r)] = P[s][j];
    }
}

__global__ void __launch_bounds__(LU64_THREADS) k_block_lu_f64(double* fac, int* ipiv, int* info, Sched S, Launch L, int step) {
    using SM = Lu64Smem;
    constexpr int BM = SM::BM, LD = SM::LD, LT = SM::LT, NW = LU64_THREADS / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sm = reinterpret_cast<double*>(smem_raw);
    double *A = sm + SM::a, *ex = sm + SM::ex, *sT = sm + SM::t, *sL = sm + SM::l;
    __shared__ double srd[LU_G];
    __shared__ int cpa[BM], cpb[BM], spiv[BM];            // piece of each column, local pivot rows
    __shared__ int spv[LU_G], sat[BM], slsrc[BM], sleft[BM], szero, zpiece;
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    const int blk = F.block0 + step;
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk], bw = c1 - c0;
    const int p0 = S.blk_p0[blk], np = S.blk_np[blk];
    const int tid = threadIdx.x, wp = tid >> 5, lane = tid & 31;
    const bool sym = S.sym != 0;
    double* blkp = fac + F.loff + (ll)c0 * F.ld + c0;   // block (i, j) at blkp[j * ld + i]
#pragma unroll
    for (int x = 0; x < BM / NW; ++x)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int C = wp + x * NW, R = lane + 32 * s;
            if (C < bw && R < bw && (!sym || R >= C)) {
                const double v = blkp[(ll)C * F.ld + R];
                A[C * LD + R] = v;
                if (sym) A[R * LD + C] = v;   // symmetric form: the upper triangle mirrors the lower one
            }
        }
    for (int pc = tid; pc < np; pc += LU64_THREADS) {
        const int a = S.xsuper[p0 + pc] - F.f - c0, b = S.xsuper[p0 + pc + 1] - F.f - c0;
        for (int k = a; k < b; ++k) {
            cpa[k] = a;
            cpb[k] = b;
        }
    }
    if (tid == 0) zpiece = INT_MAX;
    __syncthreads();
    for (int a = 0; a < bw;) {
        // group [a, b): whole pieces of up to 32 columns, or a slice of a wider one; rows to e
        int b = a;
        while (b < bw && cpb[b] - a <= LU_G) b = cpb[b];
        int e = b;
        if (b == a) {
            e = cpb[a];
            b = a + LU_G;
        }
        const int w = b - a, nrow = e - a, nr = bw - b;
        if (tid < nrow) sleft[tid] = max(cpa[a + tid] - a, 0);
        if (tid == 0) szero = LU_G;
        __syncthreads();
        if (wp < cdiv(w, LU_W)) {
            const int cend = lane < w ? cpb[a + lane] - a : 0;
            if (nrow <= 32) lu64_sweep<1>(A + a * LD + a, nrow, w, cend, sleft, ex, srd, spv, sat, &szero, sym, wp);
            else lu64_sweep<2>(A + a * LD + a, nrow, w, cend, sleft, ex, srd, spv, sat, &szero, sym, wp);
        }
        __syncthreads();
        if (tid < nrow) slsrc[sat[tid]] = tid;
        if (tid < w) spiv[a + tid] = a + (spv[tid] >> 8) - cpa[a + tid];
        if (tid == 0 && szero < LU_G) zpiece = min(zpiece, a + szero);
        __syncthreads();
        // the interchanges over the columns right of the group, and over those of
        // the first piece left of it when that is a slice (its rows only)
        const int nleft = a - cpa[a];
        for (int c = wp; c < nleft + nr; c += NW) {
            double* col = A + (c < nleft ? cpa[a] + c : b + c - nleft) * LD + a;
            const int lim = c < nleft ? cpb[a] - a : nrow;
            const double v0 = lane < lim ? col[slsrc[lane]] : 0.0, v1 = lane + 32 < lim ? col[slsrc[lane + 32]] : 0.0;
            __syncwarp();
            if (lane < lim) col[lane] = v0;
            if (lane + 32 < lim) col[lane + 32] = v1;
        }
        if (nr > 0) {
            // U11 by rows, L11 by columns (as the rows eliminated: original rows' multipliers)
            for (int t = tid; t < w * LU_G; t += LU64_THREADS) {
                const int k = t / LU_G, j = t % LU_G;
                sT[k * LT + j] = j > k && j < w ? A[(a + j) * LD + a + k] : 0.0;
                sL[k * LT + j] = j > k && j < w ? ex[k * BM + slsrc[j]] : 0.0;
            }
            __syncthreads();
            // L21 rows below e (warps 0 .. 3) and U12 columns (4 .. 7), eight lanes per line
            const bool isU = wp >= 4;
            const int q = lane & (PD_LANES - 1);
            for (int x = (wp & 3) * 4 + lane / PD_LANES; x < cdiv(nr, 16) * 16; x += 16) {
                const bool ok = x < nr && (isU || b + x >= e);
                double* line = isU ? A + (b + min(x, nr - 1)) * LD + a : A + a * LD + b + min(x, nr - 1);
                const int ls = isU ? 1 : LD;
                double y[LU_G / PD_LANES];
#pragma unroll
                for (int jj = 0; jj < LU_G / PD_LANES; ++jj) {
                    const int j = jj * PD_LANES + q;
                    y[jj] = ok && j < w ? line[j * ls] : 0.0;
                }
                if (isU) sweep_f64<LU_G>(y, sL, nullptr, w);
                else sweep_f64<LU_G>(y, sT, srd, w);
#pragma unroll
                for (int jj = 0; jj < LU_G / PD_LANES; ++jj) {
                    const int j = jj * PD_LANES + q;
                    if (ok && j < w) line[j * ls] = y[jj];
                }
            }
            // a sliced piece's own later rows: their multipliers came out of the sweep in place
            __syncthreads();
            // A22 -= L21 U12: a lane per row, four columns per warp and pass
            for (int cq = wp; cq < cdiv(nr, 4); cq += NW)
                for (int r = b + lane; r < b + cdiv(nr, 32) * 32; r += 32) {
                    const bool ok = r < bw;
                    double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
                    for (int k = 0; k < w; ++k) {
                        const double lv = ok ? A[(a + k) * LD + r] : 0.0;
#pragma unroll
                        for (int j = 0; j < 4; ++j) acc[j] += lv * A[min(b + 4 * cq + j, bw - 1) * LD + a + k];
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (ok && b + 4 * cq + j < bw) A[(b + 4 * cq + j) * LD + r] -= acc[j];
                }
            __syncthreads();
        }
        a = b;
    }
    __syncthreads();
#pragma unroll
    for (int x = 0; x < BM / NW; ++x)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int C = wp + x * NW, R = lane + 32 * s;
            if (C < bw && R < bw) blkp[(ll)C * F.ld + R] = A[C * LD + R];
        }
    if (tid < bw) ipiv[F.f + c0 + tid] = spiv[tid];
    if (tid == 0 && zpiece != INT_MAX) {
        int p = 0;
        while (S.xsuper[p0 + p + 1] - F.f - c0 <= zpiece) ++p;
        atomicMin(info, p0 + p + 1);   // first singular piece of the block
    }
}

template <typename T, int W>
__global__ void __launch_bounds__(256) k_block_panel(T* fac, const int* ipiv, const int* bmap, Sched S, Launch L,
                                                      int step, unsigned char* pack, int bf16, int part) {
    constexpr int CQ = W / 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* sT = reinterpret_cast<T*>(smem_raw);
    __shared__ T rd[W];
    __shared__ int q0[W + 1], gmap[W], pa[W];
    __shared__ int smax;
    __shared__ T sdg[W];   // symmetric form: U(j, j) of the block
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    const int blk = F.block0 + step;
    {
        const int c1 = S.blk_c1[blk];
        tile = panel_tile(part, tile, cdiv(F.ld - c1, 64), cdiv(F.nf - c1, 64), S.sym != 0);
    }
    if constexpr (std::is_same<T, float>::value && W == 128) {
        block_panel128(fac, bmap, S, F, blk, tile, pack, sT, sT + 128 * SLD<float, 128>::value, rd, gmap, pa, bf16,
                       &smax, sdg);
        return;
    }
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk], bw = c1 - c0;
    const int p0 = S.blk_p0[blk], np = S.blk_np[blk];
    const int tid = threadIdx.x, line = tid >> 2, q = tid & 3;
    const int nL = cdiv(F.ld - c1, 64), nUa = cdiv(F.nf - c1, 64);
    const T* blkp = fac + F.loff + (ll)c0 * F.ld + c0;
    if (tile < nL) {
        const int r = c1 + tile * 64 + line;
        const bool ok = r < F.ld;
        T* xp = fac + F.loff + (ll)c0 * F.ld + r;   // row r, block column j at xp[j * ld]
        T x[CQ];
#pragma unroll
        for (int jj = 0; jj < CQ; ++jj) {   // in flight while the triangle is staged
            const int j = q * CQ + jj;
            x[jj] = (ok && j < bw) ? xp[(ll)j * F.ld] : T(0);
        }
        if (S.sym && tid < bw) sdg[tid] = blkp[(ll)tid * F.ld + tid];   // U(j, j) for the U side
        stage_upper<T, W>(sT, rd, blkp, F.ld, bw);
        __syncthreads();
        sweep_rows<T, W>(x, sT, rd, bw);
#pragma unroll
        for (int jj = 0; jj < CQ; ++jj) {
            const int j = q * CQ + jj;
            if (ok && j < bw) xp[(ll)j * F.ld] = x[jj];
        }
        T u[CQ];   // symmetric form: the U side, U(c0 + j, r) = U(j, j) L(r, c0 + j)
#pragma unroll
        for (int jj = 0; jj < CQ; ++jj) {
            const int j = q * CQ + jj;
            u[jj] = (S.sym && j < bw) ? x[jj] * sdg[j] : T(0);
            if (S.sym && ok && j < bw) {
                if (r < F.nf) fac[F.loff + (ll)r * F.ld + c0 + j] = u[jj];
                else fac[F.uoff + (ll)(c0 + j) * F.m + (r - F.nf)] = u[jj];
            }
        }
        if constexpr (std::is_same<T, float>::value) {
            const ll off = S.blk_lpack[blk];
            const int e = (off >= 0 && bf16) ? block_scale_exp(blkp, F.ld, bw, &smax) : 0;
            if (off >= 0 && ok) {
                const int n1 = cdiv(F.nf - c1, umma::TM);
                const int t = r < F.nf ? (r - c1) / umma::TM : n1 + (r - F.nf) / umma::TM;
                const int i = r < F.nf ? (r - c1) % umma::TM : (r - F.nf) % umma::TM;
                if (bf16) pack_line16<CQ>(pack + (off >> 2), t, i, q, cdiv(bw, umma::KCH), x, umma::exp2i(e));
                else pack_line<CQ>(pack + off, t, i, q, cdiv(bw, umma::KCH), x);
                const ll offu = S.blk_upack[blk];   // symmetric form: the U side's pack, same tiles
                if (S.sym && offu >= 0) {
                    if (bf16) pack_line16<CQ>(pack + (offu >> 2), t, i, q, cdiv(bw, umma::KCH), u, umma::exp2i(-e));
                    else pack_line<CQ>(pack + offu, t, i, q, cdiv(bw, umma::KCH), u);
                }
            }
        }
    } else {
        for (int k = tid; k <= np; k += 256) q0[k] = S.xsuper[p0 + k] - F.f - c0;
        __syncthreads();
        block_gather_map(ipiv + F.f + c0, q0, np, gmap, pa);
        __syncthreads();
        const bool inner = tile < nL + nUa;
        const int col = inner ? c1 + (tile - nL) * 64 + line : (tile - nL - nUa) * 64 + line;
        const bool ok = inner ? col < F.nf : col < F.m;
        // block row k of this column at cp[k * stride]
        T* cp = inner ? fac + F.loff + (ll)col * F.ld + c0 : fac + F.uoff + (ll)c0 * F.m + col;
        const ll stride = inner ? 1 : (ll)F.m;
        T y[CQ];
#pragma unroll
        for (int ii = 0; ii < CQ; ++ii) {   // in flight while the triangle is staged
            const int R = q * CQ + ii;
            y[ii] = (ok && R < bw) ? cp[(ll)gmap[R] * stride] : T(0);
        }
        stage_lower<T, W>(sT, blkp, F.ld, bw, gmap, pa);
        __syncthreads();
        sweep_cols<T, W>(y, sT, bw);
#pragma unroll
        for (int ii = 0; ii < CQ; ++ii) {
            const int R = q * CQ + ii;
            if (ok && R < bw) cp[(ll)R * stride] = y[ii];
        }
        if constexpr (std::is_same<T, float>::value) {
            const ll off = S.blk_upack[blk];
            const float scale = (off >= 0 && bf16) ? umma::exp2i(-block_scale_exp(blkp, F.ld, bw, &smax)) : 1.0f;
            if (off >= 0 && ok) {
                const int n1 = cdiv(F.nf - c1, umma::TM);
                const int t = inner ? (col - c1) / umma::TM : n1 + col / umma::TM;
                const int i = inner ? (col - c1) % umma::TM : col % umma::TM;
                if (bf16) pack_line16<CQ>(pack + (off >> 2), t, i, q, cdiv(bw, umma::KCH), y, scale);
                else pack_line<CQ>(pack + off, t, i, q, cdiv(bw, umma::KCH), y);
            }
        }
    }
}

// After the factorisation: the whole-block solve operators of every block,
//   Minv = inv(L_B) P_B  (the forward steps of all its pieces, in order)
//   Uinv = inv(U_B)      (the backward steps, pieces reversed)
// written column-major (bw x bw, Minv then Uinv) at inv2[blk_inv2[blk]], so
// that a triangular-solve step of a block is one product.  They are the
// panel sweeps applied to the identity: column j of Minv is the U-panel
// sweep of e_j, row i of Uinv the L-panel sweep of e_i.  This kernel takes
// the blocks of more than 32 columns (W = 64, 128); `entries` lists the
// work, entry = blk * 4 + kind * 2 + tile (kind 0 Minv, 1 Uinv; 64 lines per
// tile).  Dynamic shared memory: W * SLD(W) T's.  Narrower blocks:
// k_block_inv_small.
template <typename T, int W>
__global__ void __launch_bounds__(256) k_block_inv(const T* fac, const int* ipiv, T* inv2, Sched S,
                                                    const int* blk_front, const int* entries) {
    constexpr int CQ = W / 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ T rd[W];
    __shared__ int q0[W + 1], gmap[W], pa[W];
    static_assert(W > 32, "blocks of at most 32 columns: k_block_inv_small");
    const int e = entries[blockIdx.x];
    const int blk = e >> 2, kind = (e >> 1) & 1, l0 = (e & 1) * 64;
    const DFront F = S.fronts[blk_front[blk]];
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk], bw = c1 - c0;
    const int p0 = S.blk_p0[blk], np = S.blk_np[blk];
    const T* blkp = fac + F.loff + (ll)c0 * F.ld + c0;
    T* sL = reinterpret_cast<T*>(smem_raw);
    T* sU = sL;   // one kind per entry
    const int tid = threadIdx.x, line = tid >> 2, q = tid & 3;
    if (kind != 1) {
        for (int k = tid; k <= np; k += 256) q0[k] = S.xsuper[p0 + k] - F.f - c0;
        __syncthreads();
        block_gather_map(ipiv + F.f + c0, q0, np, gmap, pa);
        __syncthreads();
        stage_lower<T, W>(sL, blkp, F.ld, bw, gmap, pa);
    }
    if (kind != 0) stage_upper<T, W>(sU, rd, blkp, F.ld, bw);
    __syncthreads();
    const bool doM = kind == 0;
    const int idx = l0 + line;
    if (__all_sync(0xffffffffu, idx >= bw)) return;   // the whole warp is past the block
    T v[CQ];
    T* out = inv2 + S.blk_inv2[blk];
    if (doM) {
#pragma unroll
        for (int ii = 0; ii < CQ; ++ii) {
            const int R = q * CQ + ii;
            v[ii] = (R < bw && gmap[R] == idx) ? T(1) : T(0);
        }
        sweep_cols<T, W>(v, sL, bw);
        if (idx < bw) {
#pragma unroll
            for (int ii = 0; ii < CQ; ++ii) {
                const int R = q * CQ + ii;
                if (R < bw) out[(ll)idx * bw + R] = v[ii];
            }
        }
    } else {
#pragma unroll
        for (int jj = 0; jj < CQ; ++jj) v[jj] = (q * CQ + jj == idx) ? T(1) : T(0);
        sweep_rows<T, W>(v, sU, rd, bw);
        if (idx < bw) {
#pragma unroll
            for (int jj = 0; jj < CQ; ++jj) {
                const int j = q * CQ + jj;
                if (j < bw) out[(ll)bw * bw + (ll)j * bw + idx] = v[jj];
            }
        }
    }
}

// The same operators for blocks of at most W <= 32 columns, a warp per
// block, four per CTA (launches by width class W = 4, 8, 16, 32): the block
// in shared memory, lane j forms column j of Minv (P e_j through the
// forward steps of the pieces, the multipliers of row i left of its piece
// taken from its source row, as stage_lower stages them), lane i row i of
// Uinv (e_i through the backward steps, scaled by 1 / U(j, j)).  The
// operations of the sweeps k_block_inv applies, in the same order, without
// a CTA per block for blocks of a few columns.
constexpr int BI_WARPS = 4;
template <typename T, int W>
__global__ void __launch_bounds__(32 * BI_WARPS) k_block_inv_small(const T* fac, const int* ipiv, T* inv2, Sched S,
                                                                    const int* blk_front, const int* entries,
                                                                    int count) {
    constexpr int LD = W + 1;
    __shared__ T sD[BI_WARPS][W * LD];   // D(r, c) at [c * LD + r]
    __shared__ T srd[BI_WARPS][W];
    __shared__ int sq[BI_WARPS][W + 1], sgm[BI_WARPS][W], spa[BI_WARPS][W];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int idx = blockIdx.x * BI_WARPS + warp;
    if (idx >= count) return;   // whole warp; no CTA barrier below
    const int blk = entries[idx];
    const DFront F = S.fronts[blk_front[blk]];
    const int c0 = S.blk_c0[blk], bw = S.blk_c1[blk] - c0;
    const int p0 = S.blk_p0[blk], np = S.blk_np[blk];
    const T* blkp = fac + F.loff + (ll)c0 * F.ld + c0;
    T* D = sD[warp];
    T* rd = srd[warp];
    int* q0 = sq[warp];
    int* gm = sgm[warp];
    int* pa = spa[warp];
    for (int k = lane; k <= np; k += 32) q0[k] = S.xsuper[p0 + k] - F.f - c0;
    for (int j = 0; j < bw; ++j)
        if (lane < bw) D[j * LD + lane] = blkp[(ll)j * F.ld + lane];
    if (lane < bw) rd[lane] = T(1) / blkp[(ll)lane * F.ld + lane];
    __syncwarp();
    const int* ipb = ipiv + F.f + c0;
    for (int pc = lane; pc < np; pc += 32) {   // block_gather_map, a lane per piece
        const int a = q0[pc], b = q0[pc + 1];
        for (int i = a; i < b; ++i) {
            gm[i] = i;
            pa[i] = a;
        }
        for (int k = a; k < b; ++k) {
            const int kp = a + ipb[k];
            const int t = gm[k];
            gm[k] = gm[kp];
            gm[kp] = t;
        }
    }
    __syncwarp();
    T* out = inv2 + S.blk_inv2[blk];
    {   // Minv(:, lane)
        T y[W];
#pragma unroll
        for (int i = 0; i < W; ++i) y[i] = (lane < bw && i < bw && gm[i] == lane) ? T(1) : T(0);
#pragma unroll
        for (int i = 1; i < W; ++i)
            if (i < bw) {
                const int gi = gm[i], ai = pa[i];
#pragma unroll
                for (int k = 0; k < i; ++k) y[i] -= D[k * LD + (k < ai ? gi : i)] * y[k];
            }
        if (lane < bw)
#pragma unroll
            for (int i = 0; i < W; ++i)
                if (i < bw) out[(ll)lane * bw + i] = y[i];
    }
    {   // Uinv(lane, :)
        T x[W];
#pragma unroll
        for (int j = 0; j < W; ++j) x[j] = (j == lane && lane < bw) ? T(1) : T(0);
#pragma unroll
        for (int j = 0; j < W; ++j)
            if (j < bw) {
#pragma unroll
                for (int k = 0; k < j; ++k) x[j] -= x[k] * D[j * LD + k];
                x[j] *= rd[j];
            }
        if (lane < bw)
#pragma unroll
            for (int j = 0; j < W; ++j)
                if (j < bw) out[(ll)bw * bw + (ll)j * bw + lane] = x[j];
    }
}

// ---------------------------------------------------------------------------
// 64 x 64 register-tiled block product, 256 threads, 4 x 4 outputs each.
// sA[k][i] (k < kc, i < 64), sB[k][j]; thread (tx, ty) owns rows tx+16a and
// columns ty+16b when rows_fast, else rows ty+16a and columns tx+16b.
// ---------------------------------------------------------------------------
constexpr int TT = 64;
constexpr int KC = 32;

// Symmetric form: the tiles (i, j) of an nr x nc tile grid with i >= j
// (the lower part and the diagonal tiles), column by column: column j holds
// nr - j tiles.  Tile number t -> (i, j).
__host__ __device__ __forceinline__ void lower_tile(int t, int nr, int& i, int& j) {
    j = 0;
    while (t >= nr - j) {
        t -= nr - j;
        ++j;
    }
    i = j + t;
}
__host__ __device__ __forceinline__ int lower_tiles(int nr, int nc) {
    int n = 0;
    for (int j = 0; j < nc && j < nr; ++j) n += nr - j;
    return n;
}
// The same for groups of w adjacent tile columns (wide tiles): group j
// covers columns w j .. w j + w - 1 and rows w j .. nr - 1.
__host__ __device__ __forceinline__ void lower_tile_w(int t, int nr, int w, int& i, int& j) {
    j = 0;
    while (t >= nr - w * j) {
        t -= nr - w * j;
        ++j;
    }
    i = w * j + t;
}
__host__ __device__ __forceinline__ int lower_tiles_w(int nr, int w) {
    int n = 0;
    for (int j = 0; w * j < nr; ++j) n += nr - w * j;
    return n;
}

// The Schur complement tiles of a tensor-core front in two parts: the near
// part (1) holds every tile with an entry whose target front - the owner of
// the smaller of its row and column, rows sorted ascending - is factored at
// the next level, i.e. a row tile or a column below q (the first q row
// tiles hold every row such a front owns); the far part (2) the others,
// whose targets are factored two or more levels up.  Tiles of the whole
// update (part 0): t = g n2 + rt, column group g of nh tiles and row tile
// rt; in the SPD form the lower tiles of group g (rows nh g .. n2 - 1) in
// that order, where the near part is the groups below cdiv(q, nh).
__host__ __device__ __forceinline__ int schur_part_count(int part, int n2, int nh, int q, bool sym) {
    const int ng = cdiv(n2, nh);
    q = min(q, n2);
    const int gq = min(cdiv(q, nh), ng);
    const int all = sym ? lower_tiles_w(n2, nh) : ng * n2;
    int far;
    if (sym) {
        int near = 0;
        for (int j = 0; j < gq; ++j) near += n2 - nh * j;
        far = all - near;
    } else {
        far = (ng - gq) * (n2 - q);
    }
    return part == 0 ? all : part == 1 ? all - far : far;
}
__host__ __device__ __forceinline__ int schur_part_tile(int part, int e, int n2, int nh, int q, bool sym) {
    if (part == 0) return e;
    q = min(q, n2);
    const int gq = min(cdiv(q, nh), cdiv(n2, nh));
    if (sym) return part == 1 ? e : schur_part_count(1, n2, nh, q, true) + e;
    if (part == 1) {
        if (e < gq * n2) return e;
        e -= gq * n2;
        return (gq + e / q) * n2 + e % q;
    }
    return (gq + e / (n2 - q)) * n2 + q + e % (n2 - q);
}

template <typename T, bool rows_fast>
__device__ __forceinline__ void mma_tile(const T* sA, const T* sB, int kc, T acc[4][4]) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int ri = rows_fast ? tx : ty, ci = rows_fast ? ty : tx;
#pragma unroll 4
    for (int k = 0; k < kc; ++k) {
        T a[4], b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) { a[q] = sA[k * TT + ri + 16 * q]; b[q] = sB[k * TT + ci + 16 * q]; }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] += a[i] * b[j];
    }
}

// Trailing update after block `step`: A[R, C] -= L[R, block] * U[block, C]
// over the front minus its Schur-complement block.  L tiles: rows in
// [c1, nf+m), columns in [c1, nf) (stored in Lf).  U tiles: rows in [c1, nf),
// columns in U12 (stored in Uf).
template <typename T>
__global__ void __launch_bounds__(256) k_block_trail(T* fac, Sched S, Launch L, int step) {
    __shared__ T sA[KC * TT];
    __shared__ T sB[KC * TT];
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    const int blk = F.block0 + step;
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk];
    const int tid = threadIdx.x;
    const int nrL = cdiv(F.ld - c1, TT), ncL = cdiv(F.nf - c1, TT);
    const bool isL = S.sym || tile < nrL * ncL;   // the symmetric form: lower L tiles only
    int r0, col0, nr, nc;
    if (isL) {
        int ti = tile % nrL, tj = tile / nrL;
        if (S.sym) lower_tile(tile, nrL, ti, tj);
        r0 = c1 + ti * TT;
        col0 = c1 + tj * TT;
        nr = min(TT, F.ld - r0);
        nc = min(TT, F.nf - col0);
    } else {
        const int t2 = tile - nrL * ncL, nrU = cdiv(F.nf - c1, TT);
        r0 = c1 + (t2 % nrU) * TT;
        col0 = (t2 / nrU) * TT;            // U12 column index
        nr = min(TT, F.nf - r0);
        nc = min(TT, F.m - col0);
    }
    T acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = T(0);
    for (int k0 = c0; k0 < c1; k0 += KC) {
        const int kc = min(KC, c1 - k0);
        for (int e = tid; e < kc * TT; e += 256) {
            int i = e % TT, k = e / TT;
            sA[k * TT + i] = (i < nr) ? fac[F.loff + (ll)(k0 + k) * F.ld + r0 + i] : T(0);
        }
        if (isL) {
            for (int e = tid; e < kc * TT; e += 256) {
                int k = e % kc, j = e / kc;
                sB[k * TT + j] = (j < nc) ? fac[F.loff + (ll)(col0 + j) * F.ld + k0 + k] : T(0);
            }
        } else {
            for (int e = tid; e < kc * TT; e += 256) {
                int j = e % TT, k = e / TT;
                sB[k * TT + j] = (j < nc) ? fac[F.uoff + (ll)(k0 + k) * F.m + col0 + j] : T(0);
            }
        }
        __syncthreads();
        if (isL) mma_tile<T, true>(sA, sB, kc, acc);
        else mma_tile<T, false>(sA, sB, kc, acc);
        __syncthreads();
    }
    const int tx = tid & 15, ty = tid >> 4;
    // the 16 entries are loaded before any is stored (distinct addresses the
    // compiler cannot prove distinct)
    T old[4][4];
    ll addr[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int r = isL ? tx + 16 * a : ty + 16 * a, c = isL ? ty + 16 * b : tx + 16 * b;
            const bool in = r < nr && c < nc;
            addr[a][b] = !in ? -1 : isL ? F.loff + (ll)(col0 + c) * F.ld + r0 + r : F.uoff + (ll)(r0 + r) * F.m + col0 + c;
            old[a][b] = in ? fac[addr[a][b]] : T(0);
        }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (addr[a][b] >= 0) fac[addr[a][b]] = old[a][b] - acc[a][b];
}

// Scatter target of one row or column x of a Schur complement tile: the
// front G of R_F[x] (its run), and x's position in G.
struct ScatterRow {
    ll rel0;     // offset in rel[] of R_F[0] for the run of this row / column
    ll loff, uoff;
    int ld, nf, m, pos;
};

template <typename T>
__device__ __forceinline__ ScatterRow scatter_row(const Sched& S, const DFront& F, int x) {
    ScatterRow e{};
    e.pos = -1;
    if (x < F.m) {
        const int g = S.runid[F.runid_off + x];
        const DFront G = S.fronts[S.run_tgt[g]];
        e.rel0 = S.run_rel[g] - S.run_start[g];
        e.loff = G.loff;
        e.uoff = G.uoff;
        e.ld = G.ld;
        e.nf = G.nf;
        e.m = G.m;
        e.pos = S.rel[e.rel0 + x];
    }
    return e;
}

// Small fronts (one block of at most 32 columns, m <= LF_M) factored whole
// by one warp each, four per CTA: the block LU of k_block_lu_small, then
// the L21 rows (x := x U^-1, a lane per row), the U12 columns (interchanges
// of the block, then u := L^-1 u, a lane per column), both in the entry
// order of the panel sweeps, and the Schur complement L21 U12 (k in order)
// scatter-subtracted into the ancestors like k_schur.  Replaces, for these
// fronts, k_block_lu_small + k_block_panel + k_schur (three launches whose
// CTAs would be mostly idle on fronts this small).  Each launch holds fronts
// of one width class W (block width <= W, W = 4, 8, 16 or 32), so that the
// unrolled register loops and the shared memory are sized to the class.
constexpr int LF_M = 32, LF_WARPS = 4;
constexpr int LF_CLASSES = 4;   // W = 4 << class
__host__ __device__ constexpr int leaf_class(int bw) { return bw <= 4 ? 0 : bw <= 8 ? 1 : bw <= 16 ? 2 : 3; }
template <typename T, int W> struct LeafSmem {
    static constexpr int LD = W + 1;
    static constexpr size_t warp_bytes = (((size_t)(W + 2 * LF_M) * LD + W) * sizeof(T) + LF_M * sizeof(ScatterRow) +
                                          (W + 1 + 3 * W) * sizeof(int) + 15) / 16 * 16;
    static constexpr size_t bytes = LF_WARPS * warp_bytes;
};

// A load of factor data that other CTAs of the same launch may have updated
// (COH: at L2, bypassing the SM's L1, which is not coherent across SMs).
template <bool COH, typename T>
__device__ __forceinline__ T ld_fac(const T* p) {
    if constexpr (COH) return __ldcg(p);
    else return *p;
}

// One small front (block width <= W) factored whole by the calling warp;
// `base` is the warp's slice of LeafSmem<T, W>.
template <typename T, bool COH, int W>
__device__ __forceinline__ void leaf_front(T* fac, int* ipiv, int* info, const Sched& S, const DFront& F,
                                           unsigned char* base) {
    constexpr int LD = LeafSmem<T, W>::LD;
    const int lane = threadIdx.x & 31;
    ScatterRow* tab = reinterpret_cast<ScatterRow*>(base);
    T* sD = reinterpret_cast<T*>(tab + LF_M);          // diagonal block, D(i, j) at sD[j * LD + i]
    T* sL = sD + W * LD;                               // L21 rows, L21(r, k) at sL[r * LD + k]
    T* sV = sL + LF_M * LD;                            // U12 columns, U12(k, c) at sV[c * LD + k]
    T* srv = sV + LF_M * LD;                           // 1 / U(k, k)
    int* q0 = reinterpret_cast<int*>(srv + W);
    int* piv = q0 + W + 1;
    int* gm = piv + W;
    int* pam = gm + W;
    const int blk = F.block0, bw = F.nf, m = F.m;
    const int p0 = S.blk_p0[blk], np = S.blk_np[blk];
    const bool sym = S.sym != 0;
    for (int k = lane; k <= np; k += 32) q0[k] = S.xsuper[p0 + k] - F.f;
    // the block, with the rows below it where a warp holds both
    const bool fit = bw + m <= 32;
    const int nrow = fit ? bw + m : bw;
    T r0[W];
#pragma unroll
    for (int j = 0; j < W; ++j)   // symmetric form: the upper triangle mirrors the lower one
        r0[j] = lane < nrow && j < bw ? ((sym && lane < j) ? ld_fac<COH>(fac + F.loff + (ll)lane * F.ld + j)
                                                           : ld_fac<COH>(fac + F.loff + (ll)j * F.ld + lane))
                                      : T(0);
    for (int x = lane; x < m; x += 32) tab[x] = scatter_row<T>(S, F, x);
    __syncwarp();
    // block LU (ggetrf! pivots inside each piece; none in the symmetric form)
    int pos, pa0;
    const bool sing = warp_block_lu<T, W>(r0, bw, nrow, q0, piv, gm, pam, sym, pos, pa0);
    if (lane < nrow) {
#pragma unroll
        for (int j = 0; j < W; ++j)
            if (j < bw) {
                const int i = lane >= bw || j < pa0 ? lane : pos;
                fac[F.loff + (ll)j * F.ld + i] = r0[j];
                if (lane < bw) sD[j * LD + i] = r0[j];
                else sL[(lane - bw) * LD + j] = r0[j];
            }
    }
    __syncwarp();
    if (lane < bw) {
        ipiv[F.f + lane] = piv[lane];
        srv[lane] = fit ? T(1) : rcp_rn(sD[lane * LD + lane]);   // as the panel's 1 / U(k, k)
    }
    if (lane == 0 && sing) {
        for (int pc = 0; pc < np; ++pc) {
            bool z = false;
            for (int k = q0[pc]; k < q0[pc + 1]; ++k) z |= sD[k * LD + k] == T(0);
            if (z) { atomicMin(info, p0 + pc + 1); break; }
        }
    }
    __syncwarp();
    // L21 rows (m <= 32: a lane per row): x := x U^-1 (left-looking: entry j
    // gets k = 0, 1, .. then its scaling)
    const int r = lane;
    if (!fit && r < m) {
        T x[W];
#pragma unroll
        for (int k = 0; k < W; ++k) x[k] = k < bw ? ld_fac<COH>(fac + F.loff + (ll)k * F.ld + bw + r) : T(0);
#pragma unroll
        for (int j = 0; j < W; ++j)
            if (j < bw) {
#pragma unroll
                for (int k = 0; k < j; ++k) x[j] -= x[k] * sD[j * LD + k];
                x[j] *= srv[j];
            }
#pragma unroll
        for (int k = 0; k < W; ++k)
            if (k < bw) {
                fac[F.loff + (ll)k * F.ld + bw + r] = x[k];
                sL[r * LD + k] = x[k];
            }
    }
    // U12 columns, a lane per column c: y := inv(L) P y (symmetric form:
    // y_k = U(k, k) L21(c, k), from this lane's own L21 row)
    const int c = lane;
    T y[W];
    if (sym) {
#pragma unroll
        for (int k = 0; k < W; ++k) y[k] = (c < m && k < bw) ? sD[k * LD + k] * sL[c * LD + k] : T(0);
    } else {
#pragma unroll
        for (int k = 0; k < W; ++k) y[k] = (c < m && k < bw) ? ld_fac<COH>(fac + F.uoff + (ll)gm[k] * m + c) : T(0);
#pragma unroll
        for (int i = 0; i < W; ++i)
            if (i < bw) {
#pragma unroll
                for (int k = 0; k < i; ++k) {
                    const T l = k < pam[i] ? sD[k * LD + gm[i]] : sD[k * LD + i];
                    y[i] -= l * y[k];
                }
            }
    }
    if (c < m)
#pragma unroll
        for (int k = 0; k < W; ++k)
            if (k < bw) {
                fac[F.uoff + (ll)k * m + c] = y[k];
                sV[c * LD + k] = y[k];
            }
    __syncwarp();
    // Schur complement, entries (rr, cc) over the lanes, rows fastest: every
    // lane works whatever m is, and the adds to a column of an ancestor are
    // contiguous
    for (int e = lane; e < m * m; e += 32) {
        const int cc = e / m, rr = e - cc * m;
        if (sym && rr < cc) continue;   // the symmetric form forms the lower part only
        T acc = T(0);
#pragma unroll
        for (int k = 0; k < W; ++k)
            if (k < bw) acc += sL[rr * LD + k] * sV[cc * LD + k];
        if (rr >= cc) {   // L entry of the front of R_F[cc]
            const ScatterRow& Cc = tab[cc];
            const int p = S.rel[Cc.rel0 + rr];
            if (Cc.pos >= 0 && p >= 0) atomicAdd(&fac[Cc.loff + (ll)Cc.pos * Cc.ld + p], -acc);
        } else {          // entry of the front of R_F[rr]
            const ScatterRow& R = tab[rr];
            const int p = S.rel[R.rel0 + cc];
            if (R.pos >= 0 && p >= 0) {
                const ll addr = p < R.nf ? R.loff + (ll)p * R.ld + R.pos : R.uoff + (ll)R.pos * R.m + (p - R.nf);
                atomicAdd(&fac[addr], -acc);
            }
        }
    }
}

template <typename T, int W>
__global__ void __launch_bounds__(32 * LF_WARPS) k_leaf_factor(T* fac, int* ipiv, int* info, Sched S, Launch L) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5;
    unsigned char* base = smem_raw + (size_t)warp * LeafSmem<T, W>::warp_bytes;
    const int idx = blockIdx.x * LF_WARPS + warp;
    if (idx >= L.count) return;   // whole warp; the kernel has no CTA barrier
    leaf_front<T, false, W>(fac, ipiv, info, S, S.fronts[L.front_ids[idx]], base);
}

// Small fronts of every width class in one launch, for levels with few of
// them: lists ids[i] (class i % LF_CLASSES) hold the fronts up to the running
// count end[i].
constexpr int LEAF_LISTS = 2 * LF_CLASSES;
struct LeafSet {
    const int* ids[LEAF_LISTS];
    int end[LEAF_LISTS];
};
__device__ __forceinline__ int leaf_of(const LeafSet& L, int idx, int& list) {
    int first = 0, front = -1;
    list = LEAF_LISTS;
#pragma unroll
    for (int i = 0; i < LEAF_LISTS; ++i) {
        if (list == LEAF_LISTS && idx < L.end[i]) {
            list = i;
            front = L.ids[i][idx - first];
        }
        first = L.end[i];
    }
    return front;
}
template <typename T>
__global__ void __launch_bounds__(32 * LF_WARPS) k_leaf_factor_set(T* fac, int* ipiv, int* info, Sched S, LeafSet L,
                                                                   unsigned warp_bytes) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5;
    unsigned char* base = smem_raw + (size_t)warp * warp_bytes;
    int list;
    const int fid = leaf_of(L, blockIdx.x * LF_WARPS + warp, list);
    if (fid < 0) return;   // whole warp; the kernel has no CTA barrier
    const DFront F = S.fronts[fid];
    switch (list % LF_CLASSES) {
    case 0: leaf_front<T, false, 4>(fac, ipiv, info, S, F, base); break;
    case 1: leaf_front<T, false, 8>(fac, ipiv, info, S, F, base); break;
    case 2: leaf_front<T, false, 16>(fac, ipiv, info, S, F, base); break;
    default: leaf_front<T, false, 32>(fac, ipiv, info, S, F, base); break;
    }
}

// The bottom subtrees of small fronts (every front of the subtree factored
// whole, as by k_leaf_factor) in one persistent launch: a merged work queue
// in level order.  A warp takes the next front (atomic counter `next`),
// waits until the front's children have signalled (deps[front] == 0; a
// bounded spin of `budget` polls, after which it records a timeout in *err
// and goes on, so that the launch always ends), factors it, makes its writes
// visible (fence) and signals its parent (qparent[position], -1 when the
// parent is factored by the level launches).  A front's children come
// earlier in the queue, so every front waited on is held by a running warp.
// `stall` (a queue position, or -1) makes that position's wait one that
// nothing ends, so that the timeout path can be tested.  Shared memory is
// sized for the widest class.
template <typename T>
__global__ void __launch_bounds__(32 * LF_WARPS) k_leaf_queue(T* fac, int* ipiv, int* info, Sched S, const int* order,
                                                              const int* qparent, int nq, int* next, int* deps,
                                                              unsigned budget, int stall, int* err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char* base = smem_raw + (size_t)warp * LeafSmem<T, 32>::warp_bytes;
    for (;;) {
        int pos = 0;
        if (lane == 0) pos = atomicAdd(next, 1);
        pos = __shfl_sync(0xffffffffu, pos, 0);
        if (pos >= nq) break;
        const int fid = order[pos];
        if (lane == 0) {
            const int done = pos == stall ? -1 : 0;   // deps never falls below 0
            unsigned it = 0;
            while (*reinterpret_cast<volatile int*>(deps + fid) > done) {
                if (++it >= budget) {
                    atomicExch(err, 1);
                    break;
                }
                if (it > 32) __nanosleep(64);
            }
            __threadfence();
        }
        __syncwarp();
        const DFront F = S.fronts[fid];
        switch (leaf_class(F.nf)) {
        case 0: leaf_front<T, true, 4>(fac, ipiv, info, S, F, base); break;
        case 1: leaf_front<T, true, 8>(fac, ipiv, info, S, F, base); break;
        case 2: leaf_front<T, true, 16>(fac, ipiv, info, S, F, base); break;
        default: leaf_front<T, true, 32>(fac, ipiv, info, S, F, base); break;
        }
        __threadfence();
        __syncwarp();
        if (lane == 0 && qparent[pos] >= 0) atomicSub(deps + qparent[pos], 1);
    }
}

// Schur complement of every front in the launch: C = L21 * U12 (m x m,
// inner dimension nf), scatter-subtracted into the ancestors.  An entry
// (r, c) of C belongs to the front of column R_F[c] when r >= c (an L
// entry) and to the front of row R_F[r] when r < c (a U entry); both are
// the front of R_F[min(r, c)], whose run gives the positions.
template <typename T>
__global__ void __launch_bounds__(256) k_schur(T* fac, Sched S, Launch L) {
    __shared__ T sA[KC * TT];
    __shared__ T sB[KC * TT];
    __shared__ ScatterRow tab[2][TT];   // [0] tile columns, [1] tile rows
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    const int tid = threadIdx.x;
    const int nt = cdiv(F.m, TT);
    int ti = tile % nt, tj = tile / nt;
    if (S.sym) lower_tile(tile, nt, ti, tj);   // the symmetric form: lower tiles only
    const int r0 = ti * TT, c0 = tj * TT;
    const int nr = min(TT, F.m - r0), nc = min(TT, F.m - c0);
    if (tid < 2 * TT) tab[tid / TT][tid % TT] = scatter_row<T>(S, F, (tid < TT ? c0 : r0) + tid % TT);   // published by the first barrier below
    T acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = T(0);
    for (int k0 = 0; k0 < F.nf; k0 += KC) {
        const int kc = min(KC, F.nf - k0);
        for (int e = tid; e < kc * TT; e += 256) {
            int i = e % TT, k = e / TT;
            sA[k * TT + i] = (i < nr) ? fac[F.loff + (ll)(k0 + k) * F.ld + F.nf + r0 + i] : T(0);
            sB[k * TT + i] = (i < nc) ? fac[F.uoff + (ll)(k0 + k) * F.m + c0 + i] : T(0);
        }
        __syncthreads();
        mma_tile<T, true>(sA, sB, kc, acc);
        __syncthreads();
    }
    // scatter through the tile's target tables: one rel[] load per entry,
    // the 16 loads of a thread in flight together, then its 16 scatter-adds
    const int tx = tid & 15, ty = tid >> 4;
    int pos[4][4];
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int ic = ty + 16 * b, ir = tx + 16 * a, c = c0 + ic, r = r0 + ir;
            pos[a][b] = -1;
            if (ic < nc && ir < nr && (r >= c || !S.sym))
                pos[a][b] = r >= c ? S.rel[tab[0][ic].rel0 + r] : S.rel[tab[1][ir].rel0 + c];
        }
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int ic = ty + 16 * b, ir = tx + 16 * a, c = c0 + ic, r = r0 + ir;
            const int p = pos[a][b];
            if (p < 0) continue;
            if (r >= c) {   // L entry of the front of R_F[c]
                const ScatterRow& Cc = tab[0][ic];
                if (Cc.pos >= 0) atomicAdd(&fac[Cc.loff + (ll)Cc.pos * Cc.ld + p], -acc[a][b]);
            } else {        // entry of the front of R_F[r]
                const ScatterRow& R = tab[1][ir];
                if (R.pos >= 0) {
                    const ll addr = p < R.nf ? R.loff + (ll)p * R.ld + R.pos : R.uoff + (ll)R.pos * R.m + (p - R.nf);
                    atomicAdd(&fac[addr], -acc[a][b]);
                }
            }
        }
}

// ---------------------------------------------------------------------------
// Rank updates of the FP32 fronts on the tensor cores (3xTF32), from the
// panels packed by k_block_panel.  Tiles are 128 x 128; the rows of a
// front are tiled in two regions, [c1, nf) from c1 (n1 tiles) and [nf, ld)
// from nf (n2 tiles), the columns likewise ([c1, nf) of the front, then the
// U12 columns), so that the packed tiles of every block line up with the
// Schur complement's.
//   TRAIL (block `step`): A = L panel row tile rt, B = U panel column tile
//     ct, K = the block's columns; tiles (rt < n1 + n2, ct < n1) update Lf,
//     tiles (rt < n1, n1 <= ct) update U12 in Uf.
//   SCHUR: A = L21 row tile, B = U12 column tile, K = all blocks' columns;
//     the product is scattered into the ancestors like k_schur.
// A launch covers local tiles tile_base.. of each front in its list (the
// trailing update is launched as tile 0, which holds the next block's
// diagonal block, and tiles 1.., so that the next block LU can start before
// the rest of the update is done).  SCHUR launches of part 1 / 2 cover the
// near / far tiles of each front (schur_part_tile), part 0 all of them.
// Persistent: CTA b takes tiles b, b + gridDim.x, ...  Warp 0 lane 0 issues
// the bulk copies, warp 1 lane 0 the MMAs, and the TC_EPI epilogue warps
// (from warp 4; warp w reads TMEM lanes 32 (w % 4).. and the 32 accumulator
// columns 32 ((w - 4) / 4)..) drain the accumulator.
// ---------------------------------------------------------------------------

constexpr int TC_TRAIL = 0, TC_SCHUR = 1;
constexpr int TC_EPI = 16, TC_THREADS = 32 * (4 + TC_EPI);

struct TcTile {
    DFront F;
    int rt, ct, n1, n2, nchunks;
    int nh;   // 128-column tiles of the (wide) tile that exist: ct .. ct + nh - 1
};

template <int MODE, int NH = 1>
__device__ __forceinline__ TcTile tc_decode(const Sched& S, const Launch& L, int step, int tile, int tile_base,
                                           int part) {
    TcTile T;
    int fid, t;
    locate(L, tile, fid, t);
    t += tile_base;
    T.F = S.fronts[fid];
    const int n2 = cdiv(T.F.m, umma::TM);
    T.n2 = n2;
    if (MODE == TC_TRAIL) {
        const int blk = T.F.block0 + step;
        const int c1 = S.blk_c1[blk], bw = c1 - S.blk_c0[blk];
        const int n1 = cdiv(T.F.nf - c1, umma::TM);
        T.n1 = n1;
        if (S.sym) {   // lower tiles of the front columns only
            lower_tile(t, n1 + n2, T.rt, T.ct);
        } else if (t < (n1 + n2) * n1) {
            T.rt = t % (n1 + n2);
            T.ct = t / (n1 + n2);
        } else {
            const int t2 = t - (n1 + n2) * n1;
            T.rt = t2 % n1;
            T.ct = n1 + t2 / n1;
        }
        T.nchunks = cdiv(bw, umma::KCH);
        T.nh = 1;
    } else {
        T.n1 = 0;
        t = schur_part_tile(part, t, n2, NH, T.F.sq, S.sym != 0);
        int g;
        if (S.sym) {
            lower_tile_w(t, n2, NH, T.rt, g);
        } else {
            T.rt = t % n2;
            g = t / n2;
        }
        T.ct = NH * g;
        T.nh = min(NH, n2 - T.ct);
        if (S.sym) T.nh = min(T.nh, T.rt - T.ct + 1);   // no tile above the diagonal
        int nc = 0;
        for (int b = 0; b < T.F.nblocks; ++b) {
            const int blk = T.F.block0 + b;
            nc += cdiv(S.blk_c1[blk] - S.blk_c0[blk], umma::KCH);
        }
        T.nchunks = nc;
    }
    return T;
}

// The K loop of one tile as a sequence of pipeline stages: (block, first
// chunk, chunks).  TRAIL: the chunks of block `step`; SCHUR: those of every
// block of the front in turn.  A stage holds one chunk (TF32: hi + lo of A
// and of B) or, in the BF16 form, up to umma::BF_GROUP consecutive chunks of
// one block.  The copy and the MMA threads walk the same sequence.
template <int MODE, bool BF>
struct ChunkWalk {
    static constexpr int G = BF ? umma::BF_GROUP : 1;
    int b, c, nb, left;   // current block, its next chunk, its chunks; chunks of the tile left
    __device__ __forceinline__ ChunkWalk(const Sched& S, const TcTile& T, int step) {
        b = MODE == TC_TRAIL ? T.F.block0 + step : T.F.block0;
        c = 0;
        nb = cdiv(S.blk_c1[b] - S.blk_c0[b], umma::KCH);
        left = T.nchunks;
    }
    // Next stage: block, first chunk, number of chunks; false when done.
    __device__ __forceinline__ bool next(const Sched& S, int& blk, int& c0, int& kc) {
        if (left <= 0) return false;
        while (c == nb) {   // SCHUR: the next block of the front
            ++b;
            c = 0;
            nb = cdiv(S.blk_c1[b] - S.blk_c0[b], umma::KCH);
        }
        blk = b;
        c0 = c;
        kc = min(G, nb - c);
        c += kc;
        left -= kc;
        return true;
    }
};

template <int MODE, bool BF, int NH = 1>
__global__ void __launch_bounds__(TC_THREADS, 1) k_tc_update(float* fac, const unsigned char* pack, Sched S, Launch L,
                                                              int step, int ntiles, int tile_base, int part, int* err) {
    static_assert(MODE == TC_SCHUR || NH == 1, "wide tiles are for the Schur complements");
    using G = umma::PGeo<NH>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ ScatterRow tab[NH + 1][umma::TM];   // SCHUR: [h] columns of tile h, [NH] tile rows
    __shared__ int dead;
    const umma::PCtx cx = umma::pctx_of<NH>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < G::NST; ++s) {
            umma::mbar_init(&cx.full[s], 1);
            umma::mbar_init(&cx.empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            umma::mbar_init(&cx.tfull[b], 1);
            umma::mbar_init(&cx.tempty[b], 32 * TC_EPI);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        dead = 0;
    }
    if (warp == 1) umma::tmem_alloc(cx.tmem_slot, G::TMEM_COLS);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = *cx.tmem_slot;
    volatile int* vdead = &dead;
    // bytes of one chunk of one operand; B tile h of a stage at BOFF + h * BSTEP
    constexpr uint32_t CB = BF ? umma::PCHUNK16 : umma::PCHUNK;
    constexpr uint32_t BOFF = 2 * umma::OPB, BSTEP = 2 * umma::OPB;
    constexpr uint32_t ACC_COLS = NH * umma::TN;

    if (warp == 0) {
        if (lane == 0) {   // bulk copies
            int s = 0;
            uint32_t ph = 0;
            for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
                const TcTile T = tc_decode<MODE, NH>(S, L, step, tile, tile_base, part);
                ChunkWalk<MODE, BF> w(S, T, step);
                int b, c, kc;
                while (w.next(S, b, c, kc)) {
                    const int nch = w.nb;
                    const int n1b = MODE == TC_TRAIL ? T.n1 : cdiv(T.F.nf - S.blk_c1[b], umma::TM);
                    const int ra = MODE == TC_TRAIL ? T.rt : n1b + T.rt;
                    const int rb = MODE == TC_TRAIL ? T.ct : n1b + T.ct;
                    const ll lp = BF ? (S.blk_lpack[b] >> 2) : S.blk_lpack[b];
                    const ll up = BF ? (S.blk_upack[b] >> 2) : S.blk_upack[b];
                    const unsigned char* pa = pack + lp + ((ll)ra * nch + c) * CB;
                    umma::wait_bounded(&cx.empty[s], ph ^ 1, vdead, err);
                    umma::arrive_expect_tx(&cx.full[s], (1 + T.nh) * kc * CB);
                    const uint32_t dst = umma::saddr(cx.stage + s * G::STAGE);
                    umma::bulk_g2s(dst, pa, kc * CB, &cx.full[s]);
                    for (int h = 0; h < T.nh; ++h) {
                        const unsigned char* pb = pack + up + ((ll)(rb + h) * nch + c) * CB;
                        umma::bulk_g2s(dst + BOFF + h * BSTEP, pb, kc * CB, &cx.full[s]);
                    }
                    if (++s == G::NST) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {   // MMAs
            constexpr uint32_t IDESC = BF ? umma::idesc_bf16(umma::TM, umma::TN) : umma::idesc_tf32(umma::TM, umma::TN);
            int s = 0;
            uint32_t ph = 0;
            int acc = 0;
            uint32_t aph = 0;
            for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
                const TcTile T = tc_decode<MODE, NH>(S, L, step, tile, tile_base, part);
                umma::wait_bounded(&cx.tempty[acc], aph ^ 1, vdead, err);
                umma::fence_after();
                ChunkWalk<MODE, BF> w(S, T, step);
                int b, c, kc;
                bool first = true;
                while (w.next(S, b, c, kc)) {
                    umma::wait_bounded(&cx.full[s], ph, vdead, err);
                    umma::fence_after();
                    const uint32_t a0 = umma::saddr(cx.stage + s * G::STAGE);
                    for (int h = 0; h < T.nh; ++h) {
                        const uint32_t d = tmem + acc * ACC_COLS + h * umma::TN;
                        const uint32_t b0 = a0 + BOFF + h * BSTEP;
                        if constexpr (BF) {
                            for (int j = 0; j < kc; ++j) {   // one K = 16 product per chunk
                                const uint64_t da = umma::desc_kmajor(a0 + j * CB, 128, umma::SBO16);
                                const uint64_t db = umma::desc_kmajor(b0 + j * CB, 128, umma::SBO16);
                                umma::mma_bf16(d, da, db, IDESC, (first && j == 0) ? 0u : 1u);
                            }
                        } else {
                            const uint32_t a_hi = a0, a_lo = a0 + umma::OPB;
                            const uint32_t b_hi = b0, b_lo = b0 + umma::OPB;
#pragma unroll
                            for (int kk = 0; kk < umma::KCH / 8; ++kk) {
                                const uint32_t o = kk * 256;
                                const uint64_t dah = umma::desc_kmajor(a_hi + o, 128, umma::SBO);
                                const uint64_t dal = umma::desc_kmajor(a_lo + o, 128, umma::SBO);
                                const uint64_t dbh = umma::desc_kmajor(b_hi + o, 128, umma::SBO);
                                const uint64_t dbl = umma::desc_kmajor(b_lo + o, 128, umma::SBO);
                                umma::mma_tf32(d, dah, dbh, IDESC, (first && kk == 0) ? 0u : 1u);
                                umma::mma_tf32(d, dah, dbl, IDESC, 1u);
                                umma::mma_tf32(d, dal, dbh, IDESC, 1u);
                            }
                        }
                    }
                    first = false;
                    umma::commit(&cx.empty[s]);
                    if (++s == G::NST) { s = 0; ph ^= 1; }
                }
                umma::commit(&cx.tfull[acc]);
                if (++acc == 2) { acc = 0; aph ^= 1; }
            }
        }
    } else if (warp >= 4) {   // epilogue: thread = one TMEM lane (tile row), 32 columns of each tile
        const int q4 = warp & 3, i = 32 * q4 + lane, cg = (warp - 4) >> 2, et = threadIdx.x - 128;
        int acc = 0;
        uint32_t aph = 0;
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            const TcTile T = tc_decode<MODE, NH>(S, L, step, tile, tile_base, part);
            const DFront& F = T.F;
            if (MODE == TC_SCHUR) {
                asm volatile("bar.sync 1, %0;" ::"n"(32 * TC_EPI) : "memory");   // previous tile's scatter done
                for (int e = et; e < (T.nh + 1) * umma::TM; e += 32 * TC_EPI) {
                    const int side = e / umma::TM, rows = side == T.nh;
                    const int x = (rows ? T.rt : T.ct + side) * umma::TM + (e % umma::TM);
                    tab[rows ? NH : side][e % umma::TM] = scatter_row<float>(S, F, x);
                }
                asm volatile("bar.sync 1, %0;" ::"n"(32 * TC_EPI) : "memory");
            }
            umma::wait_bounded(&cx.tfull[acc], aph, vdead, err);
            umma::fence_after();
            const uint32_t taddr = tmem + acc * ACC_COLS + ((uint32_t)(32 * q4) << 16);
            if (MODE == TC_TRAIL) {
                const int c1 = S.blk_c1[F.block0 + step];
                const bool rL = T.rt < T.n1;   // row region [c1, nf) else [nf, ld)
                const int row = rL ? c1 + T.rt * umma::TM + i : F.nf + (T.rt - T.n1) * umma::TM + i;
                const bool rok = rL ? row < F.nf : row < F.ld;
                const bool cL = T.ct < T.n1;   // column region: front columns [c1, nf) else U12
                const int col0 = cL ? c1 + T.ct * umma::TN : (T.ct - T.n1) * umma::TN;
                const int ncol = cL ? F.nf - col0 : F.m - col0;
                {
                    const int h = cg;
                    float v[32];
                    umma::tmem_ld32(taddr + h * 32, v);
                    if (rok) {
                        // all 32 loads before any store: the compiler cannot tell that the
                        // entries are distinct, and would otherwise serialise the round trips
                        float* dst = cL ? fac + F.loff + (ll)(col0 + h * 32) * F.ld + row
                                        : fac + F.uoff + (ll)row * F.m + col0 + h * 32;
                        const ll step_j = cL ? (ll)F.ld : 1;
#pragma unroll
                        for (int half = 0; half < 2; ++half) {   // 16 loads in flight, no spills
                            float old[16];
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const int jj = 16 * half + j;
                                old[j] = (h * 32 + jj < ncol) ? dst[(ll)jj * step_j] : 0.0f;
                            }
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const int jj = 16 * half + j;
                                if (h * 32 + jj < ncol) dst[(ll)jj * step_j] = old[j] - v[jj];
                            }
                        }
                    }
                }
            } else {
                const int r = T.rt * umma::TM + i;
                const ScatterRow& R = tab[NH][i];
                for (int th = 0; th < T.nh; ++th) {
                    const int c0 = (T.ct + th) * umma::TN;
                    const int h = cg;
                    float v[32];
                    umma::tmem_ld32(taddr + th * umma::TN + h * 32, v);
                    if (r < F.m) {
                        // positions of 16 entries first (their rel[] loads in flight
                        // together), then the 16 scatter-adds
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
                            int pos[16];
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const int jj = 16 * half + j, c = c0 + h * 32 + jj;
                                pos[j] = -1;
                                if (c < F.m && (r >= c || !S.sym))
                                    pos[j] = r >= c ? S.rel[tab[th][h * 32 + jj].rel0 + r] : S.rel[R.rel0 + c];
                            }
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const int jj = 16 * half + j, c = c0 + h * 32 + jj;
                                if (c >= F.m || pos[j] < 0) continue;
                                if (r >= c) {   // L entry of the front of R_F[c]
                                    const ScatterRow& Cc = tab[th][h * 32 + jj];
                                    if (Cc.pos >= 0) atomicAdd(&fac[Cc.loff + (ll)Cc.pos * Cc.ld + pos[j]], -v[jj]);
                                } else if (R.pos >= 0) {   // entry of the front of R_F[r]
                                    const int pc = pos[j];
                                    const ll addr = pc < R.nf ? R.loff + (ll)pc * R.ld + R.pos
                                                              : R.uoff + (ll)R.pos * R.m + (pc - R.nf);
                                    atomicAdd(&fac[addr], -v[jj]);
                                }
                            }
                        }
                    }
                }
            }
            umma::fence_before();
            umma::arrive(&cx.tempty[acc]);
            if (++acc == 2) { acc = 0; aph ^= 1; }
        }
    }
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    if (warp == 1) umma::tmem_dealloc(tmem, G::TMEM_COLS);
}

// ---------------------------------------------------------------------------
// FP64 rank updates on the tensor cores by exact integer slices (the error-
// free transformation of Ozaki, Ogita, Oishi and Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numerical Algorithms 59, 2012).
//   The FP64 units of this GPU do 1.7 multiply-adds per cycle and SM, the
// BF16 tensor pipe 4096.  Every line of a block's panels (a row of L, a
// column of U; 64 entries at most) is written as OZ_D = 8 signed base-256
// digits of a 62-bit fixed-point number relative to the line's largest entry:
// entries down to 2^-9 of it are held exactly, digits are exact BF16 values
// and a product of two slices over 64 columns is an exact FP32 integer
// (below 2^20, and below 2^23 for the up to eight pairs of one weight).  The
// 36 pairs of weight 0 .. 7 are summed per weight in tensor memory, joined as
// 64-bit integers in the epilogue and added to the FP64 target with one
// rounding per 64 columns.  The dropped pairs are below 2^-61 of the product
// of the two largest entries, so the error is that of a handful of FP64
// roundings where the multiply-add loop makes 64 (4096 x 4096 entries of
// 64-term sums of uniform [-1, 1] values against 128-bit sums: largest error
// 8.7e-16, of the loop 6.2e-15).
//   Rows and columns may differ in size by any power of two: each line has its
// exponent, and along the block column k of L is scaled by 2^t, row k of U by
// 2^-t, t half of what separates the exponents of the largest entries of the
// two.  That alone is not enough.  With M_i and N_j the largest scaled entries of
// a row of L and a column of U the error of entry (i, j) is about 2^-59 M_i N_j;
// where the entries of a line lie far apart (a column of A that is large, and
// zero in some rows of the block), the entry can be far smaller.  So
//   - index i (row i of L, column i of U) is marked where M_i N_i is more than
//     2^OZ_SPREAD times its largest product L(i, k) U(k, i).  Between indices
//     without a mark the error is below the rounding errors that the
//     multiply-add loop makes on the two diagonal entries, and no scaling of A's
//     rows or columns changes that (M_i N_i and the products change alike);
//   - an entry of a marked index that came out, and left its target, below
//     2^-OZ_TIGHT M_i N_j is formed again as a plain FP64 sum over the stored
//     factor, other entries below 2^-OZ_LOOSE.
// Errors of 64-term sums of 256 x 256 entries in units of 2^-53 (|target| +
// sum |L||U|), of the multiply-add loop, the slices with this rule and without
// it: uniform entries 3.7, 0.9, 0.9; one U column 2^40 larger in half of its
// rows 4.1, 4.1, 11,000; one L column 8.0, 4.6, 5,600.  Tighter than 2^-8 gains
// nothing over the loop, 2^-10 leaves 20.  Fronts of Laplacians, convection-
// diffusion and 2-D diffusion have no marked index (M_i N_i is at most 2^3 of
// the largest product; 2^8 with t from the U rows alone); 2^-8 for them too
// would form 1% of their entries again, nearly all in tiles beside the diagonal
// whose indices are far apart in a separator (48^3 convection-diffusion: 50.5 ms
// for the factorisation instead of 35.4; none at all 34.0).  With one column of
// that system scaled by 2^40 it takes 42 ms, with its rows scaled by random
// powers of two up to 2^30 159 ms (multiply-add loop: 164, 165).
//   Entries of a line that holds an infinity or a NaN, and those whose scale
// leaves the exponent range, are formed again too.
//   Tiles of 128 x 32: eight weights of 32 columns are 256 TMEM columns,
// double-buffered.  Digit i of L meets digits 0 .. 7 - i of U in one MMA of
// 32 (8 - i) columns, whose products are weights i .. 7: eight MMAs per 16
// columns where one per pair was 36, of 95 cycles each up to 64 columns.  The
// weights are joined and rounded by integer instructions (oz_join).  What
// bounds it now is latency: a tile's chain of copies (160 KB), accumulator
// loads, joins and target accesses (issue slots 37 to 41% busy in the Schur
// form, no pipe above 43%, ALU first).  48^3 convection-diffusion, rank updates:
// 131 -> 17.9 ms (16.5 without the second sums; 23.5 with an MMA per pair and
// FP64 joins, before there were any).  Two groups of epilogue warps on alternate
// tiles, and eight warps with twice the registers, were 4 and 10% slower.
// ---------------------------------------------------------------------------
constexpr int OZ_D = 8, OZ_N = 32;                       // digits, tile columns
constexpr int OZ_SLICE = umma::PCHUNK16;                 // one slice of a 128-line tile and 16 columns, 4 KB
constexpr int OZ_CHUNK = OZ_D * OZ_SLICE;                // 32 KB
constexpr int OZ_SUB = OZ_SLICE / 4;                     // 32 of its lines, 1 KB
constexpr int OZ_STAGE = OZ_CHUNK + OZ_D * OZ_SUB;       // A chunk, B chunk: 40 KB
constexpr int OZ_NST = 5;
constexpr int OZ_EXPS = (umma::TM + OZ_N) * 4;           // exponents of a tile's rows and columns for one block
constexpr int OZ_ERING = 8;                              // more than the blocks the copies can run ahead
constexpr int OZ_SMEM = OZ_NST * OZ_STAGE + OZ_ERING * OZ_EXPS + 2048;
constexpr int OZ_BAD = 1 << 28;                          // exponent of a line with a NaN or an infinity
constexpr int OZ_ZERO = -(1 << 20);                      // of a line of zeros
constexpr int OZ_SPREAD = 4;                             // lines marked: bits between M_i N_i and their largest common product
constexpr int OZ_TIGHT = 8, OZ_LOOSE = 16;               // entries formed again: bits below M_i N_j, of a marked line and of others
constexpr int OZ_FEW = 256;                              // of a tile's at most by eight lanes each

// Bytes of one side of a block's pack: T tiles of 128 lines, nch chunks of 16
// columns, then the lines' exponents.
__host__ __device__ __forceinline__ ll oz_side_bytes(int T, int nch) { return (ll)T * ((ll)nch * OZ_CHUNK + 512); }
__device__ __forceinline__ int* oz_exps(unsigned char* side, int T, int nch) {
    return reinterpret_cast<int*>(side + (ll)T * nch * OZ_CHUNK);
}

// Tiles of 128 rows x 32 columns, row by row.  TRAIL: (n1 + n2) x c1 on the
// front columns, then n1 x c2 on U12; the symmetric form the tiles with an
// entry on or below the diagonal of the front columns.  SCHUR: n2 x c2.
__host__ __device__ __forceinline__ int oz_lower(int n, int c) {   // rows rt hold min(4 (rt + 1), c) tiles
    const int full = c / 4 < n ? c / 4 : n;
    return 2 * full * (full + 1) + (n - full) * c;
}
__host__ __device__ __forceinline__ int oz_trail_tiles(int n1, int n2, int c1, int c2, bool sym) {
    return sym ? oz_lower(n1 + n2, c1) : (n1 + n2) * c1 + n1 * c2;
}
__host__ __device__ __forceinline__ int oz_schur_tiles(int n2, int c2, bool sym) { return sym ? oz_lower(n2, c2) : n2 * c2; }
// The trailing tiles that hold the next block's diagonal block (its 64 columns).
__host__ __device__ __forceinline__ int oz_near(int c1) { return c1 < 2 ? c1 : 2; }
__host__ __device__ __forceinline__ void oz_lower_tile(int t, int c, int& rt, int& ct) {
    rt = 0;
    for (;;) {
        const int k = 4 * (rt + 1) < c ? 4 * (rt + 1) : c;
        if (t < k) break;
        t -= k;
        ++rt;
    }
    ct = t;
}

// The slices of a block's L and U panels: a CTA per 64 lines of both sides, four
// threads per line (16 columns each).  A line's exponent is stored with its mark
// in the lowest bit.
constexpr int OZ_PLINES = 64;
__global__ void __launch_bounds__(8 * OZ_PLINES) k_oz_pack(const double* fac, const int* rexp, unsigned char* pack, Sched S, Launch L,
                                                           int step) {
    __shared__ int sE[2][4][OZ_PLINES], sB[4][OZ_PLINES], sS[64];
    __shared__ short sX[64][OZ_PLINES];   // exponents of the U lines' entries
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    const int blk = F.block0 + step;
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk], bw = c1 - c0, nch = cdiv(bw, umma::KCH);
    const int n1 = cdiv(F.nf - c1, umma::TM), T = n1 + cdiv(F.m, umma::TM);
    const bool isU = threadIdx.x >= 4 * OZ_PLINES;
    const int x0 = threadIdx.x % OZ_PLINES, part = (threadIdx.x / OZ_PLINES) & 3;
    const int t = tile / 2, line = (tile & 1) * OZ_PLINES + x0;
    const int idx = t < n1 ? c1 + t * umma::TM + line : F.nf + (t - n1) * umma::TM + line;
    const bool ok = idx < (t < n1 ? F.nf : F.ld);
    // entry k of the line at p[k * ps]
    const double* p = !isU ? fac + F.loff + (ll)c0 * F.ld + idx
                           : idx < F.nf ? fac + F.loff + (ll)idx * F.ld + c0 : fac + F.uoff + (ll)c0 * F.m + (idx - F.nf);
    const ll ps = !isU ? F.ld : idx < F.nf ? 1 : F.m;
    const int k0 = part * 16;
    long long x[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = ok && k0 + k < bw ? __double_as_longlong(p[(k0 + k) * ps]) : 0ll;
    if (threadIdx.x < 64) {   // a column of L (row of U) without a normal entry scales the other out of the way
        const int k = threadIdx.x, fu = k < bw ? rexp[2 * (F.f + c0 + k)] : 0, fl = k < bw ? rexp[2 * (F.f + c0 + k) + 1] : 0;
        sS[k] = fu && fl ? (fu - fl) >> 1 : fu ? fu + 2000 : fl ? -(fl + 2000) : 0;
    }
    __syncthreads();
    int E = OZ_ZERO;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const int ex = (int)((x[k] >> 52) & 0x7ff), sh = isU ? -sS[k0 + k] : sS[k0 + k];
        if (ex == 0x7ff) E = OZ_BAD;
        else if ((x[k] << 1) != 0) E = max(E, (ex ? ex : 1) - 1022 + sh);   // |x| 2^sh < 2^E
        if (isU) sX[k0 + k][x0] = (x[k] << 1) != 0 ? (short)ex : (short)-30000;
    }
    sE[isU][part][x0] = E;
    __syncthreads();
    E = max(max(sE[isU][0][x0], sE[isU][1][x0]), max(sE[isU][2][x0], sE[isU][3][x0]));
    if (!isU) {   // the line's largest product L(i, k) U(k, i) is below 2^B
        int B = OZ_ZERO;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int ex = (x[k] << 1) != 0 ? (int)((x[k] >> 52) & 0x7ff) : -30000;
            B = max(B, ex + sX[k0 + k][x0] - 2 * 1022);
        }
        sB[part][x0] = B;
    }
    __syncthreads();
    unsigned char* side = pack + (isU ? S.blk_upack[blk] : S.blk_lpack[blk]);
    if (part == 0) {
        const int O = isU ? 0 : 1;
        const int other = max(max(sE[O][0][x0], sE[O][1][x0]), max(sE[O][2][x0], sE[O][3][x0]));
        const int B = max(max(sB[0][x0], sB[1][x0]), max(sB[2][x0], sB[3][x0]));
        const bool mark = (E != OZ_ZERO || other != OZ_ZERO) && E + other - B > OZ_SPREAD;
        oz_exps(side, T, nch)[t * umma::TM + line] = 2 * E + (mark ? 1 : 0);
    }
#pragma unroll
    for (int g = 0; g < 2; ++g) {   // eight columns: one 16-byte unit per slice
        const int kg = k0 + 8 * g;
        if (kg >= nch * umma::KCH) break;
        long long q[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const long long b = x[8 * g + e];
            const int ex = (int)((b >> 52) & 0x7ff), sh = isU ? -sS[kg + e] : sS[kg + e];
            const long long m = (b & 0xfffffffffffffll) | (ex ? 1ll << 52 : 0ll);
            const int s = (ex ? ex : 1) - 1075 + sh + 62 - E;   // |x| 2^(sh + 62 - E) = m 2^s, s <= 9
            long long v = 0;
            if (E != OZ_BAD && E != OZ_ZERO && s >= 0) v = m << s;
            else if (E != OZ_BAD && E != OZ_ZERO && s > -54) v = (m + (1ll << (-s - 1))) >> -s;
            q[e] = b < 0 ? -v : v;
        }
        // L: slices of 128 lines; U: of 32 lines, so that a tile's eight slices are contiguous
        unsigned char* dst = side + ((ll)t * nch + kg / umma::KCH) * OZ_CHUNK +
                             (isU ? (line / OZ_N) * (OZ_D * OZ_SUB) : 0) +
                             umma::packed_offset16(isU ? line % OZ_N : line, kg % umma::KCH);
        const int ds = isU ? OZ_SUB : OZ_SLICE;
#pragma unroll
        for (int d = OZ_D - 1; d >= 0; --d) {
            unsigned w[4];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int c = (int)(signed char)(q[e] & 0xff);
                q[e] = (q[e] - c) >> 8;
                const unsigned h = __float_as_uint((float)c) >> 16;   // exact in BF16
                w[e / 2] = (e & 1) ? w[e / 2] | h << 16 : h;
            }
            *reinterpret_cast<uint4*>(dst + d * ds) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

struct OzTile {
    DFront F;
    int p0 = 0, p1 = 0;  // tiles of the launch in this front: a CTA's next tile is mostly in the same one
    int t0;              // its first local tile
    int rt, ct;          // 128-row tile, 32-column tile (of its region)
    int n1, n2, c1, c2;  // TRAIL: row tiles of [c1, nf) and [nf, ld), column tiles of [c1, nf) and U12
    int b0, nb;          // blocks
    int fc1;             // TRAIL: end column of the block
};
// part: TRAIL 1 the near tiles, 2 the others.
template <int MODE>
__device__ __forceinline__ void oz_decode(OzTile& T, const Sched& S, const Launch& L, int step, int tile, int part) {
    if (tile < T.p0 || tile >= T.p1) {
        int lo = 0, hi = L.count - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (L.prefix[mid] <= tile) lo = mid; else hi = mid - 1;
        }
        T.F = S.fronts[L.front_ids[lo]];
        T.p0 = L.prefix[lo];
        T.p1 = L.prefix[lo + 1];
        T.n2 = cdiv(T.F.m, umma::TM);
        T.c2 = cdiv(T.F.m, OZ_N);
        T.t0 = 0;
        if (MODE == TC_TRAIL) {
            T.fc1 = S.blk_c1[T.F.block0 + step];
            T.n1 = cdiv(T.F.nf - T.fc1, umma::TM);
            T.c1 = cdiv(T.F.nf - T.fc1, OZ_N);
            T.b0 = T.F.block0 + step;
            T.nb = 1;
            if (part == 2) T.t0 = oz_near(T.c1);
        } else {
            T.n1 = T.c1 = T.fc1 = 0;
            T.b0 = T.F.block0;
            T.nb = T.F.nblocks;
        }
    }
    const int t = tile - T.p0 + T.t0;
    if (MODE == TC_TRAIL) {
        const int nL = (T.n1 + T.n2) * T.c1;
        if (S.sym) oz_lower_tile(t, T.c1, T.rt, T.ct);
        else if (t < nL) {
            T.rt = t / T.c1;
            T.ct = t % T.c1;
        } else {
            T.rt = (t - nL) / T.c2;
            T.ct = T.c1 + (t - nL) % T.c2;
        }
    } else if (S.sym) {
        oz_lower_tile(t, T.c2, T.rt, T.ct);
    } else {
        T.rt = t / T.c2;
        T.ct = t % T.c2;
    }
}
// Pack tiles of block b for the tile: row tile ra, column tile rb and its quarter sub.
template <int MODE>
__device__ __forceinline__ void oz_lines(const Sched& S, const OzTile& T, int b, int& ra, int& rb, int& sub, int& nt) {
    const int n1 = MODE == TC_TRAIL ? T.n1 : cdiv(T.F.nf - S.blk_c1[b], umma::TM);
    nt = n1 + T.n2;
    if (MODE == TC_TRAIL) {
        ra = T.rt;
        rb = T.ct < T.c1 ? T.ct / 4 : n1 + (T.ct - T.c1) / 4;
        sub = T.ct < T.c1 ? T.ct % 4 : (T.ct - T.c1) % 4;
    } else {
        ra = n1 + T.rt;
        rb = n1 + T.ct / 4;
        sub = T.ct % 4;
    }
}

// The product from its weights (0 .. 4 joined in units of 2^E, 5 .. 7 of
// 2^(E - 24); 76 bits at most), rounded once to nearest; SIGN flips it.  By
// integer instructions: a conversion or an addition in FP64 costs a quarter of
// the SM 64 cycles and more, and the form with both takes four of them.  z:
// the product is below 2^(E + 54 - z), not below half of that.
__device__ __forceinline__ double oz_join(const int (&n)[OZ_D], int E, long long SIGN, int& z) {
    // |weight w| <= 2^20 (w + 1)
    const long long hi = ((long long)(n[0] * 256 + n[1]) << 24) + ((long long)n[2] << 16) + (n[3] * 256 + n[4]);
    const long long lo = ((long long)n[5] << 16) + (n[6] * 256 + n[7]);
    // 96 bits, units of 2^(E - 10) and 2^(E - 42): below 2^63 of the former
    const long long top = (hi << 10) + (lo >> 14);
    const unsigned frac = (unsigned)lo << 18;
    const long long neg = top >> 63;
    const unsigned long long a = (unsigned long long)(top ^ neg) + (neg && frac == 0);
    const unsigned fr = (frac ^ (unsigned)neg) - (unsigned)neg;
    z = __clzll((long long)a);
    if (z > 43) {   // small after cancellation, or zero
        const double v = fma((double)lo, __longlong_as_double((long long)(E - 24 + 1023) << 52),
                             (double)hi * __longlong_as_double((long long)(E + 1023) << 52));
        return SIGN ? -v : v;
    }
    unsigned w2 = (unsigned)(a >> 32), w1 = (unsigned)a, w0 = fr;
    if (z >= 32) {
        w2 = w1;
        w1 = w0;
        w0 = 0;
    }
    w2 = __funnelshift_l(w1, w2, z);   // the leading 64 bits; ties away from zero
    w1 = __funnelshift_l(w0, w1, z);
    const unsigned long long m = (((unsigned long long)w2 << 32 | w1) >> 11) + ((w1 >> 10) & 1u);
    return __longlong_as_double((((long long)(E + 1075 - z) << 52) + (long long)m) ^ (neg & (long long)(1ull << 63)) ^ SIGN);
}

// Sum of L(row, k) U(k, col) over k = c0, c0 + step, .. below c1 of a front,
// plain FP64 (front-local row; col of the front, or nf + the U12 column).
__device__ __forceinline__ double oz_sum(const double* fac, const DFront& F, int row, int col, int c0, int c1, int step) {
    const bool in = col < F.nf;
    const double *l = fac + F.loff + row, *u = in ? fac + F.loff + (ll)col * F.ld : fac + F.uoff + (col - F.nf);
    const ll us = in ? 1 : F.m;
    double s = 0.0;
#pragma unroll 8
    for (int k = c0; k < c1; k += step) s += l[(ll)k * F.ld] * u[k * us];
    return s;
}
__device__ __forceinline__ bool oz_below(double v, int lim) {   // |v| < 2^lim
    return ((__double2hiint(v) >> 20) & 0x7ff) - 1023 < lim;
}
// SCHUR: offset of entry (r, c)'s target, -1 if it has none.  (Rc, Rr: the
// scatter rows of c and r.)
__device__ __forceinline__ ll oz_target(const int* rel, const ScatterRow& Rc, const ScatterRow& Rr, int r, int c) {
    const ScatterRow& R = r >= c ? Rc : Rr;
    const int p = rel[R.rel0 + (r >= c ? r : c)];
    if (p < 0 || R.pos < 0) return -1;
    if (r >= c) return R.loff + (ll)R.pos * R.ld + p;   // L entry of the front of R_F[c]
    return p < R.nf ? R.loff + (ll)p * R.ld + R.pos : R.uoff + (ll)R.pos * R.m + (p - R.nf);   // of the front of R_F[r]
}
// A warp's entries to form again (place + j with bit j of fix), those of a
// column together.
__device__ __noinline__ void oz_push(unsigned short* again, int* n, int place, unsigned fix) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, total = __reduce_add_sync(FULL, __popc(fix));
    if (total == 0) return;
    int at = 0;
    if (lane == 0) at = atomicAdd(n, total);
    at = __shfl_sync(FULL, at, 0);
#pragma unroll 1
    for (int j = 0; j < 8; ++j) {
        const unsigned m = __ballot_sync(FULL, (fix >> j) & 1u);
        if ((fix >> j) & 1u) again[at + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(place + j);
        at += __popc(m);
    }
}

template <int MODE>
__global__ void __launch_bounds__(TC_THREADS, 1) k_oz_update(double* fac, unsigned char* pack, Sched S, Launch L, int step,
                                                             int ntiles, int part, int* err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ ScatterRow tab[umma::TM + OZ_N];   // SCHUR: tile rows, then tile columns
    __shared__ unsigned short again[umma::TM * OZ_N];   // the tile's entries to form again: row * OZ_N + column
    __shared__ int nagain[3];                           // their number, of this tile, the next and the last but one
    __shared__ int dead;
    unsigned char* stage = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* exps = stage + OZ_NST * OZ_STAGE;
    uint64_t* full = reinterpret_cast<uint64_t*>(exps + OZ_ERING * OZ_EXPS);
    uint64_t *empty = full + OZ_NST, *tfull = empty + OZ_NST, *tempty = tfull + 2, *efull = tempty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(efull + OZ_ERING);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < OZ_NST; ++s) {
            umma::mbar_init(&full[s], 1);
            umma::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < OZ_ERING; ++b) umma::mbar_init(&efull[b], 1);
        for (int b = 0; b < 2; ++b) {
            umma::mbar_init(&tfull[b], 1);
            umma::mbar_init(&tempty[b], 32 * TC_EPI);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        dead = 0;
        nagain[0] = nagain[1] = nagain[2] = 0;
    }
    if (warp == 1) umma::tmem_alloc(tmem_slot, 512);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = *tmem_slot;
    volatile int* vdead = &dead;

    if (warp == 0) {
        if (lane == 0) {   // bulk copies
            int s = 0, u = 0;
            uint32_t ph = 0;
            OzTile T;
            for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
                oz_decode<MODE>(T, S, L, step, tile, part);
                for (int b = T.b0; b < T.b0 + T.nb; ++b) {
                    int ra, rb, sub, nt;
                    oz_lines<MODE>(S, T, b, ra, rb, sub, nt);
                    const int nch = cdiv(S.blk_c1[b] - S.blk_c0[b], umma::KCH);
                    unsigned char *sa = pack + S.blk_lpack[b], *sb = pack + S.blk_upack[b];
                    const unsigned char* pa = sa + (ll)ra * nch * OZ_CHUNK;
                    const unsigned char* pb = sb + (ll)rb * nch * OZ_CHUNK + sub * (OZ_D * OZ_SUB);
                    for (int c = 0; c < nch; ++c) {
                        umma::wait_bounded(&empty[s], ph ^ 1, vdead, err);
                        if (c == 0) {
                            // the exponents: a free stage means that at most OZ_NST chunks, and the two
                            // blocks whose accumulators are in use, are ahead of the epilogue
                            const uint32_t e = umma::saddr(exps + (u % OZ_ERING) * OZ_EXPS);
                            umma::arrive_expect_tx(&efull[u % OZ_ERING], OZ_EXPS);
                            umma::bulk_g2s(e, oz_exps(sa, nt, nch) + ra * umma::TM, umma::TM * 4, &efull[u % OZ_ERING]);
                            umma::bulk_g2s(e + umma::TM * 4, oz_exps(sb, nt, nch) + rb * umma::TM + sub * OZ_N, OZ_N * 4,
                                           &efull[u % OZ_ERING]);
                            ++u;
                        }
                        umma::arrive_expect_tx(&full[s], OZ_STAGE);
                        const uint32_t dst = umma::saddr(stage + s * OZ_STAGE);
                        umma::bulk_g2s(dst, pa + (ll)c * OZ_CHUNK, OZ_CHUNK, &full[s]);
                        umma::bulk_g2s(dst + OZ_CHUNK, pb + (ll)c * OZ_CHUNK, OZ_D * OZ_SUB, &full[s]);
                        if (++s == OZ_NST) { s = 0; ph ^= 1; }
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {   // MMAs
            int s = 0, acc = 0;
            uint32_t ph = 0, aph = 0;
            OzTile T;
            for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
                oz_decode<MODE>(T, S, L, step, tile, part);
                for (int b = T.b0; b < T.b0 + T.nb; ++b) {
                    const int nch = cdiv(S.blk_c1[b] - S.blk_c0[b], umma::KCH);
                    umma::wait_bounded(&tempty[acc], aph ^ 1, vdead, err);
                    umma::fence_after();
                    for (int c = 0; c < nch; ++c) {
                        umma::wait_bounded(&full[s], ph, vdead, err);
                        umma::fence_after();
                        const uint32_t a0 = umma::saddr(stage + s * OZ_STAGE), b0 = a0 + OZ_CHUNK;
                        const uint64_t da = umma::desc_kmajor(a0, 128, umma::SBO16), db = umma::desc_kmajor(b0, 128, umma::SBO16);
                        const uint32_t d0 = tmem + acc * (OZ_D * OZ_N);
                        // digit i of L with digits 0 .. 7 - i of U, whose lines follow one another: weights
                        // i .. 7 (descriptors hold addresses in 16-byte units)
#pragma unroll
                        for (int i = 0; i < OZ_D; ++i)
                            umma::mma_bf16(d0 + i * OZ_N, da + i * (OZ_SLICE >> 4), db,
                                           umma::idesc_bf16(umma::TM, (OZ_D - i) * OZ_N), c > 0 || i > 0 ? 1u : 0u);
                        umma::commit(&empty[s]);
                        if (++s == OZ_NST) { s = 0; ph ^= 1; }
                    }
                    umma::commit(&tfull[acc]);
                    if (++acc == 2) { acc = 0; aph ^= 1; }
                }
            }
        }
    } else if (warp >= 4) {   // epilogue: thread = one TMEM lane (tile row), 8 of the tile's columns
        const int q4 = warp & 3, i = 32 * q4 + lane, cg = (warp - 4) >> 2, et = threadIdx.x - 128;
        int acc = 0, u = 0, turn = 0;   // turn: of nagain
        uint32_t aph = 0;
        OzTile T;
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            oz_decode<MODE>(T, S, L, step, tile, part);
            const DFront& F = T.F;
            if (MODE == TC_SCHUR) {
                asm volatile("bar.sync 1, %0;" ::"n"(32 * TC_EPI) : "memory");   // previous tile's scatter done
                if (et < umma::TM) tab[et] = scatter_row<double>(S, F, T.rt * umma::TM + et);
                else if (et < umma::TM + OZ_N) tab[et] = scatter_row<double>(S, F, T.ct * OZ_N + et - umma::TM);
                asm volatile("bar.sync 1, %0;" ::"n"(32 * TC_EPI) : "memory");
            }
            // front-local row and columns of the product (columns past nf: U12)
            int row, rend, col0, cend;
            if (MODE == TC_TRAIL) {
                const int c1 = T.fc1;
                row = T.rt < T.n1 ? c1 + T.rt * umma::TM + i : F.nf + (T.rt - T.n1) * umma::TM + i;
                rend = T.rt < T.n1 ? F.nf : F.ld;
                col0 = T.ct < T.c1 ? c1 + T.ct * OZ_N : F.nf + (T.ct - T.c1) * OZ_N;
                cend = T.ct < T.c1 ? F.nf : F.ld;
            } else {
                row = F.nf + T.rt * umma::TM + i;
                col0 = F.nf + T.ct * OZ_N;
                rend = cend = F.ld;
            }
            col0 += cg * 8;
            const bool rok = row < rend;
            // TRAIL: the targets' old values while the products are formed (and all loads before any store: distinct
            // entries the compiler cannot tell apart)
            const bool cL = MODE == TC_TRAIL && col0 < F.nf;
            double* dst = cL ? fac + F.loff + (ll)col0 * F.ld + row : fac + F.uoff + (ll)row * F.m + (col0 - F.nf);
            const ll sj = cL ? (ll)F.ld : 1;
            double sum[8];   // SCHUR: the product; TRAIL: the target minus the product
#pragma unroll
            for (int j = 0; j < 8; ++j) sum[j] = MODE == TC_TRAIL && rok && col0 + j < cend ? dst[j * sj] : 0.0;
            constexpr long long SIGN = MODE == TC_TRAIL ? (long long)(1ull << 63) : 0ll;
            unsigned low = 0;            // columns whose product came out low (or could not be formed) in some block
            int lim = -(1 << 30);        // and the largest 2^lim that it was below
            for (int b = T.b0; b < T.b0 + T.nb; ++b) {
                const int* ev = reinterpret_cast<const int*>(exps + (u % OZ_ERING) * OZ_EXPS);
                umma::wait_bounded(&efull[u % OZ_ERING], (u / OZ_ERING) & 1, vdead, err);
                ++u;
                const int ei = ev[i];   // exponent, and the mark in the lowest bit
                const int* fj = ev + umma::TM + cg * 8;
                umma::wait_bounded(&tfull[acc], aph, vdead, err);
                umma::fence_after();
                const uint32_t taddr = tmem + acc * (OZ_D * OZ_N) + cg * 8 + ((uint32_t)(32 * q4) << 16);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float v[OZ_D][4];
                    umma::tmem_ld8x4<OZ_N>(taddr + 4 * h, v);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        int n[OZ_D];
#pragma unroll
                        for (int w = 0; w < OZ_D; ++w) n[w] = __float2int_rn(v[w][j]);
                        const int fe = fj[4 * h + j], W = (ei >> 1) + (fe >> 1);   // M_i N_j < 2^W
                        double& s = sum[4 * h + j];
                        if (W - 68 > -1022 && W < 1004) {
                            int z;
                            s += oz_join(n, W - 44, SIGN, z);
                            const int guard = (ei | fe) & 1 ? OZ_TIGHT : OZ_LOOSE;
                            if (z >= 10 + guard) {
                                low |= 1u << (4 * h + j);
                                lim = max(lim, W - guard);
                            }
                        } else if (W > OZ_ZERO / 2) {   // (a line of zeros adds nothing)
                            low |= 1u << (4 * h + j);
                            lim = 1 << 20;
                        }
                    }
                    __syncwarp();   // the next load is warp-wide
                }
                umma::fence_before();
                umma::arrive(&tempty[acc]);
                if (++acc == 2) { acc = 0; aph ^= 1; }
            }
            if (__any_sync(0xffffffffu, low != 0)) {   // low: becomes the entries left out here and formed again below
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const bool there = rok && col0 + j < cend && (MODE == TC_TRAIL || row >= col0 + j || !S.sym);
                    if (!there || !oz_below(sum[j], lim)) low &= ~(1u << j);
                }
                oz_push(again, &nagain[turn], i * OZ_N + cg * 8, low);
            }
            if (MODE == TC_TRAIL) {
                if (rok)
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (col0 + j < cend && !((low >> j) & 1u)) dst[j * sj] = sum[j];
            } else if (rok) {
                const int r = row - F.nf, c0 = col0 - F.nf;
                const ScatterRow& R = tab[i];
                int pos[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int c = c0 + j;
                    pos[j] = -1;
                    if (c < F.m && (r >= c || !S.sym) && !((low >> j) & 1u)) pos[j] = r >= c ? S.rel[tab[umma::TM + cg * 8 + j].rel0 + r] : S.rel[R.rel0 + c];
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int c = c0 + j;
                    if (c >= F.m || pos[j] < 0) continue;
                    if (r >= c) {   // L entry of the front of R_F[c]
                        const ScatterRow& Cc = tab[umma::TM + cg * 8 + j];
                        if (Cc.pos >= 0) atomicAdd(&fac[Cc.loff + (ll)Cc.pos * Cc.ld + pos[j]], -sum[j]);
                    } else if (R.pos >= 0) {   // entry of the front of R_F[r]
                        const int pc = pos[j];
                        const ll addr = pc < R.nf ? R.loff + (ll)pc * R.ld + R.pos : R.uoff + (ll)R.pos * R.m + (pc - R.nf);
                        atomicAdd(&fac[addr], -sum[j]);
                    }
                }
            }
            // The entries to form again: eight lanes for each, along k, where they are few (their loads are what takes
            // time), else a lane (the multiply-adds do; neighbours share a column)
            if (et == 0) nagain[turn == 2 ? 0 : turn + 1] = 0;   // of the last but one tile, read by all before the last one's barrier
            asm volatile("bar.sync 2, %0;" ::"n"(32 * TC_EPI) : "memory");
            const int n = nagain[turn];
            turn = turn == 2 ? 0 : turn + 1;
            if (n > 0) {
                const int k0 = S.blk_c0[T.b0], k1 = S.blk_c1[T.b0 + T.nb - 1], row0 = row - i, c0 = col0 - cg * 8;
                const int along = n <= OZ_FEW ? 8 : 1, q = lane & (along - 1);
                for (int e0 = (warp - 4) * (32 / along); e0 < n; e0 += TC_EPI * 32 / along) {
                    const int e = e0 + lane / along;
                    const bool ok = e < n;
                    const int at = ok ? again[e] : 0, r = row0 + at / OZ_N, c = c0 + at % OZ_N;
                    double* d = fac + (c < F.nf ? F.loff + (ll)c * F.ld + r : F.uoff + (ll)r * F.m + (c - F.nf));
                    const double old = MODE == TC_TRAIL && ok ? *d : 0.0;
                    double s = ok ? oz_sum(fac, F, r, c, k0 + q, k1, along) : 0.0;
                    if (along == 8)
#pragma unroll
                        for (int off = 4; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
                    if (!ok || q != 0) continue;
                    if (MODE == TC_TRAIL) {
                        *d = old - s;
                    } else {
                        const ll t = oz_target(S.rel, tab[umma::TM + at % OZ_N], tab[at / OZ_N], r - F.nf, c - F.nf);
                        if (t >= 0) atomicAdd(&fac[t], -s);
                    }
                }
                asm volatile("bar.sync 2, %0;" ::"n"(32 * TC_EPI) : "memory");   // `again` is free
            }
            __syncwarp();
        }
    }
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    if (warp == 1) umma::tmem_dealloc(tmem, 512);
}

// Warp reduce-scatter: N (a power of 2, at most 32) values per lane, summed
// over the 32 lanes; each step keeps the half of the values picked by a
// lane bit and adds the partner's copy of it, and once one value is left
// the remaining lane bits are summed by a butterfly (N/2 + N/4 + ... + the
// rest shuffles instead of 5 N).  Lane l ends with the sum of value
// l * N / 32.
template <int N, int OFF, typename T>
__device__ __forceinline__ void rs_halve(T* v, int lane) {
    const bool hi = (lane & OFF) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        const T keep = hi ? v[i + N / 2] : v[i];
        const T send = hi ? v[i] : v[i + N / 2];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, OFF);
    }
}
template <int N, int OFF, typename T>
__device__ __forceinline__ void rs_rec(T* v, int lane) {
    if constexpr (OFF > 0) {
        if constexpr (N > 1) {
            rs_halve<N, OFF>(v, lane);
            rs_rec<N / 2, OFF / 2>(v, lane);
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], OFF);
            rs_rec<1, OFF / 2>(v, lane);
        }
    }
}
template <int N, typename T>
__device__ __forceinline__ T warp_reduce_scatter(T (&v)[N]) {
    static_assert(N >= 1 && N <= 32 && (N & (N - 1)) == 0, "a power of 2, at most 32 values");
    rs_rec<N, 16>(v, threadIdx.x & 31);
    return v[0];
}

// ---------------------------------------------------------------------------
// Triangular solves.  Right-hand sides are column-major n x nrhs (ld = n),
// nrhs <= 16 per launch.
// ---------------------------------------------------------------------------
constexpr int TS = 128;
constexpr int MAXRHS = 16;

// Forward step for block `step`, tiled as (128 rows below the block) x (32
// columns of the block): a tile computes its 32 values of y_B = Minv b_B
// (the interchanges and unit-lower solves of the block's pieces, the
// reference's _lulsolve!, SpkLUFactor.jl:297-321), the first row tile stores
// them, and every tile subtracts L[rows, chunk] y_chunk from its rows with
// atomics (column chunks and sibling fronts share rows).  b is the running
// right-hand side, y receives the block's values.
constexpr int SC = 32;   // block columns per solve tile
template <typename T>
__global__ void __launch_bounds__(TS) k_fwd(const T* fac, const T* inv2, T* b, T* y, int n, int nrhs, Sched S,
                                            Launch L, int step) {
    constexpr int BM = BlockMax<T>::value;
    __shared__ T sm[BM * SC];   // Minv[:, chunk], sm[k * SC + j]
    __shared__ T sb[BM * MAXRHS];
    __shared__ T sp[4 * SC * MAXRHS];
    __shared__ T sy[SC * MAXRHS];
    griddep_launch();
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    const int blk = F.block0 + step;
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk], bw = c1 - c0;
    const int ncc = cdiv(bw, SC), cc = tile % ncc, rt = tile / ncc;
    const int j0 = cc * SC, nj = min(SC, bw - j0);
    const T* Mi = inv2 + S.blk_inv2[blk];
    const int tid = threadIdx.x;
    // Factor data (complete before the solve) first: the chunk of Minv into
    // shared memory, this thread's row of L[:, chunk] into registers.
    for (int e = tid; e < bw * SC; e += TS) {
        const int k = e / SC, j = e % SC;
        cp_elem(&sm[e], Mi + (ll)k * bw + j0 + min(j, nj - 1), j < nj);
    }
    const int row = c1 + rt * TS + tid;
    const bool has_row = row < F.ld;
    T lv[SC];
    int grow = 0;
    {
        const T* lcol = fac + F.loff + (ll)(c0 + j0) * F.ld + (has_row ? row : c1);
#pragma unroll
        for (int j = 0; j < SC; ++j) lv[j] = (has_row && j < nj) ? lcol[(ll)j * F.ld] : T(0);
        if (has_row) grow = row < F.nf ? F.f + row : S.rows[F.rows_off + row - F.nf];
    }
    griddep_wait();
    for (int e = tid; e < bw * nrhs; e += TS) {
        int k = e % bw, r = e / bw;
        sb[r * BM + k] = b[(ll)r * n + F.f + c0 + k];
    }
    cp_wait_all();
    __syncthreads();
    {   // y_chunk = Minv[j0:j0+nj, :] b_B : 32 columns x 4 partial sums over k
        const int j = tid & 31, kq = tid >> 5;
        T acc[MAXRHS];
#pragma unroll
        for (int r = 0; r < MAXRHS; ++r) acc[r] = T(0);
#pragma unroll 8
        for (int k = kq; k < bw; k += 4) {
            const T mk = sm[k * SC + j];
#pragma unroll
            for (int r = 0; r < MAXRHS; ++r)
                if (r < nrhs) acc[r] += mk * sb[r * BM + k];
        }
#pragma unroll
        for (int r = 0; r < MAXRHS; ++r)
            if (r < nrhs) sp[(kq * MAXRHS + r) * SC + j] = acc[r];
    }
    __syncthreads();
    for (int e = tid; e < SC * nrhs; e += TS) {
        int j = e % SC, r = e / SC;
        sy[r * SC + j] = sp[(0 * MAXRHS + r) * SC + j] + sp[(1 * MAXRHS + r) * SC + j] +
                         sp[(2 * MAXRHS + r) * SC + j] + sp[(3 * MAXRHS + r) * SC + j];
    }
    __syncthreads();
    if (rt == 0)
        for (int e = tid; e < nj * nrhs; e += TS) {
            int j = e % nj, r = e / nj;
            y[(ll)r * n + F.f + c0 + j0 + j] = sy[r * SC + j];
        }
    if (has_row) {
#pragma unroll
        for (int r = 0; r < MAXRHS; ++r) {
            if (r >= nrhs) break;
            T acc = T(0);
#pragma unroll
            for (int j = 0; j < SC; ++j) acc += lv[j] * sy[r * SC + j];
            atomicAdd(&b[(ll)r * n + grow], -acc);
        }
    }
}

// First right-hand side of this CTA's groups of RG (grid y).  A single
// right-hand side has no groups: its one pass starts without a barrier, which
// would hold back the factor loads (backward solves of a 48^3 step 3.1 ms, with
// a barrier 3.6).
template <int RG>
__device__ __forceinline__ unsigned group0() { return RG == 1 ? 0u : blockIdx.y * RG; }

// Products y[F.f + k] -= dot(line k, x[R_F]) over the lines of a front's
// off-diagonal part (U12 rows for the backward solve, L21 columns for the
// transposed one; line k at base + k * stride, F.m values, contiguous).  A
// CTA (256 threads) takes a tile of U12_ROWS lines x U12_COLS positions of
// R_F: it gathers x at those positions into shared memory (four right-hand
// sides at a time), then each warp streams four lines against it, the four
// lines' loads interleaved so that 16 are in flight per lane; partial sums go
// to y with atomics.  The tile count of a front is
// cdiv(F.nf, U12_ROWS) * cdiv(F.m, U12_COLS), enough CTAs to keep HBM busy
// on the wide fronts near the root.
constexpr int U12_ROWS = 32, U12_COLS = 512;
template <typename T, int RG>
__device__ __forceinline__ void front_line_dots(const T* base, ll stride, T* y, const T* x, int n, int nrhs,
                                                const DFront& F, const int* rows, int tile) {
    __shared__ T sx[U12_COLS * RG];   // sx[c * RG + r]
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int ncc = cdiv(F.m, U12_COLS);
    const int i0 = (tile / ncc) * U12_ROWS + wid, c0 = (tile % ncc) * U12_COLS;
    const int nc = min(U12_COLS, F.m - c0);
    for (int r0 = group0<RG>(); r0 < nrhs; r0 += gridDim.y * RG) {
        const int nr = min(RG, nrhs - r0);
        if (RG > 1 || r0 > 0) __syncthreads();
        for (int c = threadIdx.x; c < nc; c += 256) {
            const int g = rows[c0 + c];
#pragma unroll
            for (int r = 0; r < RG; ++r) sx[c * RG + r] = r < nr ? x[(ll)(r0 + r) * n + g] : T(0);
        }
        __syncthreads();
        T acc[4][RG];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int r = 0; r < RG; ++r) acc[a][r] = T(0);
        const T* u[4];
        bool live[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            live[a] = i0 + 8 * a < F.nf;
            u[a] = base + (ll)(live[a] ? i0 + 8 * a : 0) * stride + c0;
        }
#pragma unroll 4
        for (int c = lane; c < nc; c += 32) {
            T uv[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) uv[a] = live[a] ? u[a][c] : T(0);
            T xv[RG];
#pragma unroll
            for (int r = 0; r < RG; ++r) xv[r] = sx[c * RG + r];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int r = 0; r < RG; ++r) acc[a][r] += uv[a] * xv[r];
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
#pragma unroll
            for (int r = 0; r < RG; ++r) {
                T v = acc[a][r];
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
                if (lane == 0 && live[a] && r < nr) atomicAdd(&y[(ll)(r0 + r) * n + F.f + i0 + 8 * a], -v);
            }
        }
    }
}

// Backward, part 1: y[F's columns] -= U12 * x[R_F] (U12 row i contiguous in Uf).
template <typename T, int RG>
__global__ void __launch_bounds__(256) k_bwd_u12(const T* fac, T* y, const T* x, int n, int nrhs, Sched S, Launch L) {
    griddep_launch();
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    griddep_wait();
    front_line_dots<T, RG>(fac + F.uoff, F.m, y, x, n, nrhs, F, S.rows + F.rows_off, tile);
}

// Backward, part 2, for the block `step`-th from the last, tiled as (128
// rows above the block) x (32 block columns): x_chunk = Uinv[chunk, :] c_B
// (the upper solves of the block's pieces, the reference's _luusolve!,
// SpkLUFactor.jl:350-375), stored by the first row tile, then the rows
// above get U[rows, chunk] x_chunk subtracted (atomics across chunks).
template <typename T>
__global__ void __launch_bounds__(TS) k_bwd(const T* fac, const T* inv2, T* y, T* x, int n, int nrhs, Sched S,
                                            Launch L, int step) {
    constexpr int BM = BlockMax<T>::value;
    __shared__ T sm[BM * SC];   // Uinv[:, chunk], sm[k * SC + j] (rows k >= j0)
    __shared__ T sc[BM * MAXRHS];
    __shared__ T sp[4 * SC * MAXRHS];
    __shared__ T sx[SC * MAXRHS];
    griddep_launch();
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    const int blk = F.block0 + F.nblocks - 1 - step;
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk], bw = c1 - c0;
    const int ncc = cdiv(bw, SC), cc = tile % ncc, rt = tile / ncc;
    const int j0 = cc * SC, nj = min(SC, bw - j0);
    const T* Ui = inv2 + S.blk_inv2[blk] + (ll)bw * bw;
    const int tid = threadIdx.x;
    // Factor data first: the chunk of Uinv, this thread's row of U[:, chunk].
    for (int e = j0 * SC + tid; e < bw * SC; e += TS) {
        const int k = e / SC, j = e % SC;
        cp_elem(&sm[e], Ui + (ll)k * bw + j0 + min(j, nj - 1), j < nj);
    }
    const int row = rt * TS + tid;
    const bool has_row = row < c0;
    T uv[SC];
    {
        const T* ucol = fac + F.loff + (ll)(c0 + j0) * F.ld + (has_row ? row : 0);
#pragma unroll
        for (int j = 0; j < SC; ++j) uv[j] = (has_row && j < nj) ? ucol[(ll)j * F.ld] : T(0);
    }
    griddep_wait();
    for (int e = tid; e < bw * nrhs; e += TS) {
        int k = e % bw, r = e / bw;
        sc[r * BM + k] = y[(ll)r * n + F.f + c0 + k];
    }
    cp_wait_all();
    __syncthreads();
    {   // x_chunk = Uinv[j0:j0+nj, :] c_B (upper: k >= j)
        const int j = tid & 31, kq = tid >> 5;
        T acc[MAXRHS];
#pragma unroll
        for (int r = 0; r < MAXRHS; ++r) acc[r] = T(0);
        if (j < nj) {
            const int kstart = j0 + j;
#pragma unroll 8
            for (int k = kstart + kq; k < bw; k += 4) {
                const T uk = sm[k * SC + j];
#pragma unroll
                for (int r = 0; r < MAXRHS; ++r)
                    if (r < nrhs) acc[r] += uk * sc[r * BM + k];
            }
        }
#pragma unroll
        for (int r = 0; r < MAXRHS; ++r)
            if (r < nrhs) sp[(kq * MAXRHS + r) * SC + j] = acc[r];
    }
    __syncthreads();
    for (int e = tid; e < SC * nrhs; e += TS) {
        int j = e % SC, r = e / SC;
        sx[r * SC + j] = sp[(0 * MAXRHS + r) * SC + j] + sp[(1 * MAXRHS + r) * SC + j] +
                         sp[(2 * MAXRHS + r) * SC + j] + sp[(3 * MAXRHS + r) * SC + j];
    }
    __syncthreads();
    if (rt == 0)
        for (int e = tid; e < nj * nrhs; e += TS) {
            int j = e % nj, r = e / nj;
            x[(ll)r * n + F.f + c0 + j0 + j] = sx[r * SC + j];
        }
    if (has_row) {
#pragma unroll
        for (int r = 0; r < MAXRHS; ++r) {
            if (r >= nrhs) break;
            T acc = T(0);
#pragma unroll
            for (int j = 0; j < SC; ++j) acc += uv[j] * sx[r * SC + j];
            atomicAdd(&y[(ll)r * n + F.f + row], -acc);
        }
    }
}

// ---------------------------------------------------------------------------
// Solves of a front with many blocks by a cluster of NC CTAs (16 where the
// GPU can hold such clusters, else FC = 8), all its block steps in one
// launch.  Step t handles block t (forward) or block nb-1-t
// (backward); CTA rank (t mod FC) owns step t: it holds that block's
// right-hand side in shared memory, receives the updates of the earlier
// steps there, and computes the step's solution (Minv b_B forward, Uinv c_B
// backward).  The solution is published in the owner's shared memory; every
// CTA reads it through distributed shared memory and subtracts its product
// with the block's column of the factor (L below the block forward, U above
// it backward) from the blocks it owns.  The operator of an owned step and
// the block linking it to the previous step are prefetched into shared
// memory while the earlier steps run.  One cluster barrier phase per step,
// split: a CTA arrives as soon as it has read the step's solution (the
// owner of the next step after publishing it), so that only the next
// owner's work is on the chain.  Same operations as k_fwd / k_bwd per step
// inside the front; forward, the R_F rows get L21 y_F afterwards from
// k_fwd_l21 (all the GPU's SMs).  Right-hand sides RG at a time.  Fronts
// with at least FC_MINB and at most FC * FC_OWN blocks take this path (the
// plan decides).
// ---------------------------------------------------------------------------
constexpr int FC = 8, FC_MINB = 4, FC_OWN = 16, FC_THREADS = 1024;

// The grid's second dimension takes groups of RG right-hand sides, here and in
// the products between fronts below (rhs_groups on the host).
//
// Vectors of a block for RG right-hand sides (4, or 1 for a single one):
// entry (k, r) at k * RG + r.
template <int RG, typename T>
__device__ __forceinline__ void rg_get(const T* p, T (&v)[RG]) {
    if constexpr (RG == 1) v[0] = p[0];
    else sm_load<RG>(p, v);
}

template <typename T, int RG>
struct FcSmem {
    static constexpr int BM = BlockMax<T>::value, CS = FC_THREADS / BM;
    static constexpr int LDT = BM + 1;   // transposed form: rows of the prefetched blocks, an odd stride
    static constexpr size_t ypub = 0, ycur = ypub + BM * RG, own = ycur + BM * RG,
                            part = own + (size_t)FC_OWN * BM * RG, preA = part + (size_t)CS * BM * RG,
                            preM = preA + (size_t)BM * LDT, total = preM + (size_t)BM * LDT;   // in T's
    static constexpr size_t bytes = total * sizeof(T);
};

// v[i * RG + r] -= sum_j A(i, j) w[j * RG + r], i < nrow, j < ncol,
// with A(i, j) = a[i * si + j * sj] (a block of the factor in global memory, or
// its prefetched copy in shared memory).  Thread (i, cs) takes columns
// cs, cs + CS, ...; all its loads are issued before the first use.
template <typename T, int RG>
__device__ __forceinline__ void fc_tile_update(const T* a, ll si, ll sj, int nrow, int ncol, T* v, const T* w, T* part) {
    constexpr int BM = BlockMax<T>::value, CS = FC_THREADS / BM, NJ = BM / CS;
    const int i = threadIdx.x % BM, cs = threadIdx.x / BM;
    T av[NJ];
#pragma unroll
    for (int q = 0; q < NJ; ++q) {
        const int j = cs + q * CS;
        av[q] = (i < nrow && j < ncol) ? a[i * si + j * sj] : T(0);
    }
    T acc[RG];
#pragma unroll
    for (int r = 0; r < RG; ++r) acc[r] = T(0);
#pragma unroll
    for (int q = 0; q < NJ; ++q) {
        T wv[RG];
        rg_get<RG>(w + (cs + q * CS) * RG, wv);
#pragma unroll
        for (int r = 0; r < RG; ++r) acc[r] += av[q] * wv[r];
    }
#pragma unroll
    for (int r = 0; r < RG; ++r) part[(cs * BM + i) * RG + r] = acc[r];
    __syncthreads();
    for (int e = threadIdx.x; e < nrow * RG; e += FC_THREADS) {
        T sum = T(0);
#pragma unroll
        for (int c = 0; c < CS; ++c) sum += part[c * BM * RG + e];
        v[e] -= sum;
    }
    __syncthreads();
}

// The same for the transposed solves' blocks in global memory, A(i, j) =
// a[i * ld + j]: a warp takes rows i, its lanes run along j, so that the loads
// are contiguous; the sums over the lanes by a warp reduce-scatter.
template <typename T, int RG>
__device__ __forceinline__ void fc_tile_update_t(const T* a, ll ld, int nrow, int ncol, T* v, const T* w) {
    constexpr int BM = BlockMax<T>::value, NW = FC_THREADS / 32, NI = BM / NW, NJ = BM / 32;
    const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T av[NI][NJ];
#pragma unroll
    for (int s = 0; s < NI; ++s)
#pragma unroll
        for (int q = 0; q < NJ; ++q) {
            const int i = wp + s * NW, j = lane + 32 * q;
            av[s][q] = (i < nrow && j < ncol) ? a[i * ld + j] : T(0);
        }
    T acc[NI * RG];
#pragma unroll
    for (int e = 0; e < NI * RG; ++e) acc[e] = T(0);
#pragma unroll
    for (int q = 0; q < NJ; ++q) {
        T wv[RG];
        rg_get<RG>(w + (lane + 32 * q) * RG, wv);
#pragma unroll
        for (int s = 0; s < NI; ++s)
#pragma unroll
            for (int r = 0; r < RG; ++r) acc[s * RG + r] += av[s][q] * wv[r];
    }
    const T sum = warp_reduce_scatter<NI * RG>(acc);   // lane l: value l * NI * RG / 32
    constexpr int per = 32 / (NI * RG);
    const int e = lane / per, i = wp + (e / RG) * NW;
    if (lane % per == 0 && i < nrow) v[i * RG + e % RG] -= sum;
    __syncthreads();
}

// out[j * RG + r] = sum_k op(j, k) v[k * RG + r] for the block's solve
// operator (forward Minv, backward Uinv, TRI: zero for k < j; transposed:
// Uinv^T, Minv^T); op(j, k) at m[j * sj + k * sk].
template <typename T, bool TRI, int RG>
__device__ __forceinline__ void fc_block_solve(const T* m, int sj, int sk, int bw, const T* v, T* out, T* part, int nr) {
    constexpr int BM = BlockMax<T>::value, CS = FC_THREADS / BM;
    const int j = threadIdx.x % BM, cs = threadIdx.x / BM;
    T acc[RG];
#pragma unroll
    for (int r = 0; r < RG; ++r) acc[r] = T(0);
    if (j < bw) {
#pragma unroll 4
        for (int k = (TRI ? j : 0) + cs; k < bw; k += CS) {
            const T mv = m[j * sj + k * sk];
            T vv[RG];
            rg_get<RG>(v + k * RG, vv);
#pragma unroll
            for (int r = 0; r < RG; ++r) acc[r] += mv * vv[r];
        }
    }
#pragma unroll
    for (int r = 0; r < RG; ++r) part[(cs * BM + j) * RG + r] = acc[r];
    __syncthreads();
    for (int e = threadIdx.x; e < BM * RG; e += FC_THREADS) {
        const int jj = e / RG, r = e % RG;
        T sum = T(0);
        if (jj < bw && r < nr)
#pragma unroll
            for (int c = 0; c < CS; ++c) sum += part[c * BM * RG + e];
        out[e] = sum;
    }
    __syncthreads();
}

template <typename T, bool FWD, int NC, int RG, bool TRANS = false>
__global__ void __cluster_dims__(NC, 1, 1) __launch_bounds__(FC_THREADS, 1)
    k_front_solve(const T* fac, const T* inv2, T* in, T* out, int n, int nrhs, Sched S, Launch L) {
    constexpr int FC = NC;   // CTAs of the cluster
    namespace cg = cooperative_groups;
    constexpr int BM = BlockMax<T>::value;
    using SM = FcSmem<T, RG>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* sm = reinterpret_cast<T*>(smem_raw);
    T* ypub = sm + SM::ypub;
    T* ycur = sm + SM::ycur;
    T* own = sm + SM::own;
    T* part = sm + SM::part;
    T* preA = sm + SM::preA;   // A(block of step st, block of step st - 1), [j * BM + i]
    T* preM = sm + SM::preM;   // solve operator of step st, [k * BM + j]
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const DFront F = S.fronts[L.front_ids[blockIdx.x / FC]];
    const int nb = F.nblocks, tid = threadIdx.x;
    auto blk_of = [&](int step) { return F.block0 + (FWD ? step : nb - 1 - step); };
    // A(i, j) of the update of block bs by block bt: L or U (row i of bs, column
    // j of bt) at a[j * ld + i]; transposed, (row j of bt, column i of bs) at a[i * ld + j]
    auto a_of = [&](int bs, int bt) {
        return TRANS ? fac + F.loff + (ll)S.blk_c0[bs] * F.ld + S.blk_c0[bt] : fac + F.loff + (ll)S.blk_c0[bt] * F.ld + S.blk_c0[bs];
    };
    // strides of the prefetched copies: element (i, j) at i * PI + j * PJ
    constexpr int PI = TRANS ? SM::LDT : 1, PJ = TRANS ? 1 : BM;
    // The factor data of owned step st (its operator, and the block linking
    // it to step st - 1) is copied asynchronously while other steps run.
    auto prefetch = [&](int st) {
        if (st >= nb) return;
        const int bs = blk_of(st), bw = S.blk_c1[bs] - S.blk_c0[bs];
        // forward Minv, backward Uinv; transposed, Uinv^T and Minv^T: the
        // contiguous index is k there, the row of the untransposed operator
        const T* Mi = inv2 + S.blk_inv2[bs] + (FWD != TRANS ? 0 : (ll)bw * bw);
        for (int e = tid; e < BM * BM; e += FC_THREADS) {
            const int x = e % BM, y = e / BM;
            const bool v = x < bw && y < bw;
            cp_elem(&preM[TRANS ? y * PI + x : y * PJ + x], v ? Mi + (ll)y * bw + x : Mi, v);
        }
        if (st > 0) {
            const int bt = blk_of(st - 1), ncol = S.blk_c1[bt] - S.blk_c0[bt];
            const T* a = a_of(bs, bt);
            for (int e = tid; e < BM * BM; e += FC_THREADS) {
                const int x = e % BM, y = e / BM;   // x contiguous: row i, transposed column j
                const bool v = x < (TRANS ? ncol : bw) && y < (TRANS ? bw : ncol);
                cp_elem(&preA[TRANS ? y * PI + x : y * PJ + x], v ? a + (ll)y * F.ld + x : a, v);
            }
        }
    };
    for (int r0 = group0<RG>(); r0 < nrhs; r0 += gridDim.y * RG) {
        const int nr = min(RG, nrhs - r0);
        prefetch(rank);
        for (int st = rank, o = 0; st < nb; st += FC, ++o) {   // the owned blocks' right-hand sides
            const int blk = blk_of(st), c0 = S.blk_c0[blk], bw = S.blk_c1[blk] - c0;
            T* v = own + (size_t)o * BM * RG;
            for (int e = tid; e < BM * RG; e += FC_THREADS) {
                const int k = e / RG, r = e % RG;
                v[e] = (k < bw && r < nr) ? in[(ll)(r0 + r) * n + F.f + c0 + k] : T(0);
            }
        }
        __syncthreads();
        auto solve_step = [&](int st) {   // owner: publish the solution of step st
            const int blk = blk_of(st), bw = S.blk_c1[blk] - S.blk_c0[blk];
            fc_block_solve<T, !FWD && !TRANS, RG>(preM, PI, PJ, bw, own + (size_t)(st / FC) * BM * RG, ypub, part, nr);
        };
        auto finish_step = [&](int st) {   // owner, after the barrier arrival: output and next prefetch
            const int blk = blk_of(st), c0 = S.blk_c0[blk], bw = S.blk_c1[blk] - c0;
            for (int e = tid; e < bw * nr; e += FC_THREADS) {
                const int j = e % bw, r = e / bw;
                out[(ll)(r0 + r) * n + F.f + c0 + j] = ypub[j * RG + r];
            }
            prefetch(st + FC);   // preM / preA are free again
        };
        if (rank == 0) {
            cp_wait_all();
            __syncthreads();
            solve_step(0);
        }
        cl.barrier_arrive();
        if (rank == 0) finish_step(0);
        for (int t = 0; t < nb; ++t) {
            cl.barrier_wait();
            const T* src = cl.map_shared_rank(ypub, t % FC);
            for (int e = tid; e < BM * RG; e += FC_THREADS) ycur[e] = src[e];
            __syncthreads();
            const int bt = blk_of(t), ncol = S.blk_c1[bt] - S.blk_c0[bt];
            const bool next = t + 1 < nb && (t + 1) % FC == rank;
            if (next) {   // the next step's block first, from its prefetched copy: it is on the chain
                cp_wait_all();
                __syncthreads();
                const int bs = blk_of(t + 1);
                fc_tile_update<T, RG>(preA, PI, PJ, S.blk_c1[bs] - S.blk_c0[bs], ncol,
                                  own + (size_t)((t + 1) / FC) * BM * RG, ycur, part);
                solve_step(t + 1);
            }
            cl.barrier_arrive();
            if (next) finish_step(t + 1);
            for (int st = rank, o = 0; st < nb; st += FC, ++o)
                if (st > t && !(next && st == t + 1)) {
                    const int bs = blk_of(st);
                    T* v = own + (size_t)o * BM * RG;
                    const int nrow = S.blk_c1[bs] - S.blk_c0[bs];
                    if constexpr (TRANS) fc_tile_update_t<T, RG>(a_of(bs, bt), F.ld, nrow, ncol, v, ycur);
                    else fc_tile_update<T, RG>(a_of(bs, bt), 1, F.ld, nrow, ncol, v, ycur, part);
                }
            __syncthreads();
        }
        cl.barrier_wait();   // every CTA has read every published solution
        cp_wait_all();   // no copy outlives the group
        __syncthreads();
    }
}

// Solves of small fronts (one block of at most 32 columns, m <= LEAF_M), one
// warp per front, eight fronts per CTA: the whole front in one pass.
//   forward:  y_F = Minv b_F; b[R_F] -= L21 y_F (atomics, the rows are
//             shared with sibling fronts);
//   backward: c_F = y_F - U12 x[R_F]; x_F = Uinv c_F.
// Each launch holds fronts of one width class W (block width <= W, the
// classes of k_leaf_factor).  Lane j holds column j of the front; the
// front's right-hand side values are exchanged by shuffles.  Every factor
// load of a pass (a lane's column of the operator, its row of L21, its part
// of U12 for 32 rows) is issued before the first use, so that a pass waits
// for one memory round trip, not one per column.  U12 x[R_F]: for W <= 8 a
// lane per row accumulates all W columns and the warp reduces once at the
// end; wider fronts keep a lane per column and shuffle x.  Same operations as
// k_fwd / k_bwd_u12 / k_bwd.
constexpr int LEAF_M = 128;

// RG: right-hand sides per pass (1 for a single one, else 4).  TRANS, the
// transposed solves: forward Uinv^T and U12^T in the places of Minv and L21,
// backward L21^T and Minv^T in those of U12 and Uinv; only the addresses
// differ (L21 column k and U12 row k are both contiguous).
template <typename T, bool FWD, int W, int RG, bool TRANS>
__device__ __forceinline__ void solve_leaf_front(const T* fac, const T* inv2, T* in, T* out, const T* xs, int n, int nrhs,
                                                 const Sched& S, const DFront& F) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int blk = F.block0, bw = F.nf;
    const T* Mi = inv2 + S.blk_inv2[blk] + (FWD != TRANS ? 0 : (ll)bw * bw);
    // entry i of line k of the front's off-diagonal part
    auto pan = [&](int k, int i) {
        if constexpr (FWD != TRANS) return fac[F.loff + (ll)k * F.ld + F.nf + i];
        else return fac[F.uoff + (ll)k * F.m + i];
    };
    const int* rows = S.rows + F.rows_off;
    griddep_wait();
    for (int r0 = 0; r0 < nrhs; r0 += RG) {
        const int nr = min(RG, nrhs - r0);
        // narrow fronts: the loads that do not depend on the solve first (the
        // operator column, forward this lane's L21 row among the first 32
        // rows), so that a front waits for fewer round trips; wider ones
        // keep them where they are used (registers)
        constexpr bool EARLY = W <= 8;
        T mv[W];   // op(lane, k), op(j, k) at Mi[k * bw + j] (TRANS: Mi[j * bw + k])
        auto load_mv = [&] {
#pragma unroll
            for (int k = 0; k < W; ++k)
                mv[k] = (k < bw && lane < bw && (FWD || TRANS || k >= lane)) ? Mi[TRANS ? (ll)lane * bw + k : (ll)k * bw + lane] : T(0);
        };
        if constexpr (EARLY) load_mv();
        T lv0[FWD && EARLY ? W : 1];
        if constexpr (FWD && EARLY) {
#pragma unroll
            for (int k = 0; k < W; ++k) lv0[k] = (k < bw && lane < F.m) ? pan(k, lane) : T(0);
        }
        T v[RG];
#pragma unroll
        for (int r = 0; r < RG; ++r) v[r] = (lane < bw && r < nr) ? in[(ll)(r0 + r) * n + F.f + lane] : T(0);
        if constexpr (!FWD) {   // c_F = y_F - U12 x[R_F] (U12 row j contiguous in Uf)
            T acc[RG];
#pragma unroll
            for (int r = 0; r < RG; ++r) acc[r] = T(0);
            if constexpr (W <= 8) {
                T pw[W][RG];   // lane: its rows' share of every column's sum
#pragma unroll
                for (int j = 0; j < W; ++j)
#pragma unroll
                    for (int r = 0; r < RG; ++r) pw[j][r] = T(0);
                for (int i0 = 0; i0 < F.m; i0 += 32) {
                    const int il = i0 + lane;
                    const bool ok = il < F.m;
                    const int g = ok ? rows[il] : 0;
                    T uv[W], xv[RG];
#pragma unroll
                    for (int j = 0; j < W; ++j) uv[j] = (ok && j < bw) ? pan(j, il) : T(0);
#pragma unroll
                    for (int r = 0; r < RG; ++r) xv[r] = (ok && r < nr) ? xs[(ll)(r0 + r) * n + g] : T(0);
#pragma unroll
                    for (int j = 0; j < W; ++j)
#pragma unroll
                        for (int r = 0; r < RG; ++r) pw[j][r] += uv[j] * xv[r];
                }
                constexpr int NV = W * RG;   // value j * RG + r
                T flat[NV];
#pragma unroll
                for (int j = 0; j < W; ++j)
#pragma unroll
                    for (int r = 0; r < RG; ++r) flat[j * RG + r] = pw[j][r];
                const T t = warp_reduce_scatter<NV>(flat);   // lane l: value l * NV / 32
#pragma unroll
                for (int r = 0; r < RG; ++r) {
                    const T vr = __shfl_sync(FULL, t, ((lane * RG + r) * 32 / NV) & 31);
                    if (lane < bw) acc[r] = vr;
                }
            } else {
                const T* u = fac + (FWD != TRANS ? F.loff + (ll)lane * F.ld + F.nf : F.uoff + (ll)lane * F.m);
                for (int i0 = 0; i0 < F.m; i0 += 32) {
                    // lane l: x at row R_F[i0 + l]; lane j: U12(j, i0 ..)
                    const int il = i0 + lane;
                    T xv[RG];
                    const int g = il < F.m ? rows[il] : 0;
#pragma unroll
                    for (int r = 0; r < RG; ++r) xv[r] = (il < F.m && r < nr) ? xs[(ll)(r0 + r) * n + g] : T(0);
                    T uv[32];
#pragma unroll
                    for (int q = 0; q < 32; ++q) uv[q] = (lane < bw && i0 + q < F.m) ? u[i0 + q] : T(0);
#pragma unroll
                    for (int q = 0; q < 32; ++q) {
                        if (i0 + q < F.m) {   // uniform
#pragma unroll
                            for (int r = 0; r < RG; ++r) acc[r] += uv[q] * __shfl_sync(FULL, xv[r], q);
                        }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < RG; ++r) v[r] -= acc[r];
        }
        if constexpr (!EARLY) load_mv();
        T y[RG];   // lane j: sum_k op(j, k) v_k
#pragma unroll
        for (int r = 0; r < RG; ++r) y[r] = T(0);
#pragma unroll
        for (int k = 0; k < W; ++k) {
            if (k < bw) {   // uniform
#pragma unroll
                for (int r = 0; r < RG; ++r) y[r] += mv[k] * __shfl_sync(FULL, v[r], k);
            }
        }
        if (lane < bw)
#pragma unroll
            for (int r = 0; r < RG; ++r)
                if (r < nr) out[(ll)(r0 + r) * n + F.f + lane] = y[r];
        if constexpr (FWD) {   // b[R_F] -= L21 y_F (L21 column k contiguous in Lf)
            for (int i0 = 0; i0 < F.m; i0 += 32) {
                const int i = i0 + lane;
                T lv[W];   // this lane's row of L21 (the first chunk's came in early)
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    if constexpr (EARLY) {
                        if (i0 == 0) { lv[k] = lv0[k]; continue; }
                    }
                    lv[k] = (k < bw && i < F.m) ? pan(k, i) : T(0);
                }
                T acc[RG];
#pragma unroll
                for (int r = 0; r < RG; ++r) acc[r] = T(0);
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    if (k < bw) {   // uniform
#pragma unroll
                        for (int r = 0; r < RG; ++r) acc[r] += lv[k] * __shfl_sync(FULL, y[r], k);
                    }
                }
                if (i < F.m)
#pragma unroll
                    for (int r = 0; r < RG; ++r)
                        if (r < nr) atomicAdd(&in[(ll)(r0 + r) * n + rows[i]], -acc[r]);
            }
        }
    }
}

template <typename T, bool FWD, int W, int RG, bool TRANS = false>
__global__ void __launch_bounds__(256) k_solve_leaf(const T* fac, const T* inv2, T* in, T* out, const T* xs, int n,
                                                     int nrhs, Sched S, Launch L) {
    griddep_launch();
    const int idx = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (idx >= L.count) return;   // whole warp
    const DFront F = S.fronts[L.front_ids[idx]];
    solve_leaf_front<T, FWD, W, RG, TRANS>(fac, inv2, in, out, xs, n, nrhs, S, F);
}

// Every width class in one launch, for levels with few of these fronts.
template <typename T, bool FWD, int RG, bool TRANS = false>
__global__ void __launch_bounds__(256) k_solve_leaf_set(const T* fac, const T* inv2, T* in, T* out, const T* xs, int n,
                                                         int nrhs, Sched S, LeafSet L) {
    griddep_launch();
    int list;
    const int fid = leaf_of(L, blockIdx.x * 8 + (threadIdx.x >> 5), list);
    if (fid < 0) return;   // whole warp
    const DFront F = S.fronts[fid];
    switch (list % LF_CLASSES) {
    case 0: solve_leaf_front<T, FWD, 4, RG, TRANS>(fac, inv2, in, out, xs, n, nrhs, S, F); break;
    case 1: solve_leaf_front<T, FWD, 8, RG, TRANS>(fac, inv2, in, out, xs, n, nrhs, S, F); break;
    case 2: solve_leaf_front<T, FWD, 16, RG, TRANS>(fac, inv2, in, out, xs, n, nrhs, S, F); break;
    default: solve_leaf_front<T, FWD, 32, RG, TRANS>(fac, inv2, in, out, xs, n, nrhs, S, F); break;
    }
}

// Forward, after k_front_solve: b[R_F] -= L21 y_F for the fronts it solved.
// Tiles of 256 R_F rows x 128 front columns; a thread takes one row
// (L21 column k contiguous in Lf), y_F of the tile's columns in shared
// memory, partial sums added to b with atomics.
constexpr int L21_ROWS = 256, L21_COLS = 64;   // 64 columns: twice the CTAs and loads in flight of 128
// TRANS: U12^T in the place of L21 (the transposed solves).
template <typename T, int RG, bool TRANS = false>
__global__ void __launch_bounds__(256) k_fwd_l21(const T* fac, T* b, const T* y, int n, int nrhs, Sched S, Launch L) {
    __shared__ T sy[L21_COLS * RG];
    griddep_launch();
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    const int nrt = cdiv(F.m, L21_ROWS), i0 = (tile % nrt) * L21_ROWS, k0 = (tile / nrt) * L21_COLS;
    const int nk = min(L21_COLS, F.nf - k0), i = i0 + threadIdx.x;
    const bool ok = i < F.m;
    const int grow = ok ? S.rows[F.rows_off + i] : 0;
    const ll sk = TRANS ? F.m : F.ld;
    const T* a = fac + (TRANS ? F.uoff : F.loff + F.nf) + k0 * sk + (ok ? i : 0);
    griddep_wait();
    for (int r0 = group0<RG>(); r0 < nrhs; r0 += gridDim.y * RG) {
        const int nr = min(RG, nrhs - r0);
        if (RG > 1 || r0 > 0) __syncthreads();
        for (int e = threadIdx.x; e < L21_COLS * RG; e += blockDim.x) {
            const int k = e % L21_COLS, r = e / L21_COLS;
            sy[e] = (k < nk && r < nr) ? y[(ll)(r0 + r) * n + F.f + k0 + k] : T(0);
        }
        __syncthreads();
        T acc[RG];
#pragma unroll
        for (int r = 0; r < RG; ++r) acc[r] = T(0);
        if (ok) {
#pragma unroll 16
            for (int k = 0; k < nk; ++k) {
                const T av = a[k * sk];
#pragma unroll
                for (int r = 0; r < RG; ++r) acc[r] += av * sy[r * L21_COLS + k];
            }
#pragma unroll
            for (int r = 0; r < RG; ++r)
                if (r < nr) atomicAdd(&b[(ll)(r0 + r) * n + grow], -acc[r]);
        }
    }
}

// A root front (no rows below it) of more blocks than a cluster solves well
// in one launch is solved in chunks of consecutive blocks, a cluster launch
// each; between two of them every SM takes part in the rectangular product
// that links them: out[f + r] -= sum_c A(r, c) in[f + c] over rows
// [r0, r1) and columns [c0, c1) of the front (A(r, c) = fac[loff + c ld +
// r]; forward the L rows below the chunk, backward the U rows above it).
// Tiles of L21_ROWS rows x L21_COLS columns, atomics as k_fwd_l21.
constexpr int FC_CHUNK = 16;   // blocks per chunk at most
template <typename T, int RG>
__global__ void __launch_bounds__(256) k_front_gemv(const T* fac, T* out, const T* in, int n, int nrhs, ll loff, int ld,
                                                    int f, int r0, int r1, int c0, int c1) {
    __shared__ T sv[L21_COLS * RG];
    const int nrt = cdiv(r1 - r0, L21_ROWS);
    const int i0 = r0 + (int)(blockIdx.x % nrt) * L21_ROWS, k0 = c0 + (int)(blockIdx.x / nrt) * L21_COLS;
    const int nk = min(L21_COLS, c1 - k0), i = i0 + threadIdx.x;
    const bool ok = i < r1;
    const T* a = fac + loff + (ll)k0 * ld + (ok ? i : 0);
    for (int q0 = group0<RG>(); q0 < nrhs; q0 += gridDim.y * RG) {
        const int nr = min(RG, nrhs - q0);
        if (RG > 1 || q0 > 0) __syncthreads();
        for (int e = threadIdx.x; e < L21_COLS * RG; e += blockDim.x) {
            const int k = e % L21_COLS, r = e / L21_COLS;
            sv[e] = (k < nk && r < nr) ? in[(ll)(q0 + r) * n + f + k0 + k] : T(0);
        }
        __syncthreads();
        T acc[RG];
#pragma unroll
        for (int r = 0; r < RG; ++r) acc[r] = T(0);
        if (ok) {
#pragma unroll 16
            for (int k = 0; k < nk; ++k) {
                const T av = a[(ll)k * ld];
#pragma unroll
                for (int r = 0; r < RG; ++r) acc[r] += av * sv[r * L21_COLS + k];
            }
#pragma unroll
            for (int r = 0; r < RG; ++r)
                if (r < nr) atomicAdd(&out[(ll)(q0 + r) * n + f + i], -acc[r]);
        }
    }
}

// The transposed product: out[f + r] -= sum_c A(c, r) in[f + c] (line r is
// contiguous).  Tiles of GT_ROWS lines, a warp per four of them, lanes along
// the columns; a line's sum is one warp's, so no atomics.
constexpr int GT_ROWS = 32;
template <typename T, int RG>
__global__ void __launch_bounds__(256) k_front_gemv_t(const T* fac, T* out, const T* in, int n, int nrhs, ll loff, int ld, int f,
                                                      int r0, int r1, int c0, int c1) {
    const int lane = threadIdx.x & 31, i0 = r0 + (int)blockIdx.x * GT_ROWS + (int)(threadIdx.x >> 5) * 4;
    for (int q0 = group0<RG>(); q0 < nrhs; q0 += gridDim.y * RG) {
        T acc[4 * RG];
#pragma unroll
        for (int e = 0; e < 4 * RG; ++e) acc[e] = T(0);
#pragma unroll 4
        for (int c = c0 + lane; c < c1; c += 32) {
            T av[4], x[RG];
#pragma unroll
            for (int s = 0; s < 4; ++s) av[s] = i0 + s < r1 ? fac[loff + (ll)(i0 + s) * ld + c] : T(0);
#pragma unroll
            for (int r = 0; r < RG; ++r) x[r] = q0 + r < nrhs ? in[(ll)(q0 + r) * n + f + c] : T(0);
#pragma unroll
            for (int s = 0; s < 4; ++s)
#pragma unroll
                for (int r = 0; r < RG; ++r) acc[s * RG + r] += av[s] * x[r];
        }
        const T sum = warp_reduce_scatter<4 * RG>(acc);   // lane l: value l * 4 RG / 32
        constexpr int per = 32 / (4 * RG);
        const int e = lane / per, i = i0 + e / RG, r = q0 + e % RG;
        if (lane % per == 0 && i < r1 && r < nrhs) out[(ll)r * n + f + i] -= sum;
    }
}

// ---------------------------------------------------------------------------
// Transposed solves, A^T x = b with the same factors (no reference kernel:
// the reference's `transposetriangularsolve` is commented out,
// SpkSparseSpdSolver.jl:384).  With A~ = L U factored block by block, the
// forward operator is E_N ... E_1 (E_B: y_B = Minv_B b_B, b_below -=
// L_below,B y_B) and the backward one G_1 ... G_N (G_B: x_B = Uinv_B (y_B -
// U_B,right x_right)); A~^T = (G-chain)^T (E-chain)^T reversed:
//   pass 1, blocks in order (children first): z_B = Uinv_B^T c_B, then the
//     columns right of the block (front columns and U12, through R_F) get
//     U_B,right^T z_B subtracted;
//   pass 2, fronts top-down: the front's columns get L21^T x[R_F]
//     subtracted, then blocks in reverse: x_B = Minv_B^T z_B, and the
//     front's earlier columns get L_B,earlier^T x_B subtracted.
// The launch lists are those of the plain solves: small fronts and fronts of
// many blocks by k_solve_leaf and k_front_solve in their TRANS forms, the
// others by the kernels below, with the tiles of k_fwd / k_bwd_u12 / k_bwd.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(TS) k_tfwd(const T* fac, const T* inv2, T* b, T* z, int n, int nrhs, Sched S,
                                             Launch L, int step) {
    constexpr int BM = BlockMax<T>::value;
    __shared__ T sb[BM * MAXRHS];
    __shared__ T sp[4 * SC * MAXRHS];
    __shared__ T sz[SC * MAXRHS];
    griddep_launch();
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    const int blk = F.block0 + step;
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk], bw = c1 - c0;
    const int ncc = cdiv(bw, SC), cc = tile % ncc, rt = tile / ncc;
    const int j0 = cc * SC, nj = min(SC, bw - j0);
    const T* Ui = inv2 + S.blk_inv2[blk] + (ll)bw * bw;   // Uinv(k, j) at Ui[j * bw + k], zero for k > j
    griddep_wait();
    const int tid = threadIdx.x;
    for (int e = tid; e < bw * nrhs; e += TS) {
        int k = e % bw, r = e / bw;
        sb[r * BM + k] = b[(ll)r * n + F.f + c0 + k];
    }
    __syncthreads();
    {   // z_chunk = (Uinv^T)[j0:j0+nj, :] c_B : 32 columns x 4 partial sums over k <= j
        const int j = tid & 31, kq = tid >> 5;
        T acc[MAXRHS];
#pragma unroll
        for (int r = 0; r < MAXRHS; ++r) acc[r] = T(0);
        if (j < nj) {
            const T* ucol = Ui + (ll)(j0 + j) * bw;
#pragma unroll 8
            for (int k = kq; k <= j0 + j; k += 4) {
                const T uk = ucol[k];
#pragma unroll
                for (int r = 0; r < MAXRHS; ++r)
                    if (r < nrhs) acc[r] += uk * sb[r * BM + k];
            }
        }
#pragma unroll
        for (int r = 0; r < MAXRHS; ++r)
            if (r < nrhs) sp[(kq * MAXRHS + r) * SC + j] = acc[r];
    }
    __syncthreads();
    for (int e = tid; e < SC * nrhs; e += TS) {
        int j = e % SC, r = e / SC;
        sz[r * SC + j] = sp[(0 * MAXRHS + r) * SC + j] + sp[(1 * MAXRHS + r) * SC + j] +
                         sp[(2 * MAXRHS + r) * SC + j] + sp[(3 * MAXRHS + r) * SC + j];
    }
    __syncthreads();
    if (rt == 0)
        for (int e = tid; e < nj * nrhs; e += TS) {
            int j = e % nj, r = e / nj;
            z[(ll)r * n + F.f + c0 + j0 + j] = sz[r * SC + j];
        }
    const int col = c1 + rt * TS + tid;   // a column right of the block: front column (< nf) or U12 column
    if (col < F.ld) {
        T uv[SC];
        int gcol;
        if (col < F.nf) {
            gcol = F.f + col;
            const T* u = fac + F.loff + (ll)col * F.ld + c0 + j0;      // U(c0 + j0 + jj, col), contiguous
#pragma unroll
            for (int jj = 0; jj < SC; ++jj) uv[jj] = jj < nj ? u[jj] : T(0);
        } else {
            const int uc = col - F.nf;
            gcol = S.rows[F.rows_off + uc];
            const T* u = fac + F.uoff + (ll)(c0 + j0) * F.m + uc;       // U12(c0 + j0 + jj, uc)
#pragma unroll
            for (int jj = 0; jj < SC; ++jj) uv[jj] = jj < nj ? u[(ll)jj * F.m] : T(0);
        }
#pragma unroll
        for (int r = 0; r < MAXRHS; ++r) {
            if (r >= nrhs) break;
            T acc = T(0);
#pragma unroll
            for (int jj = 0; jj < SC; ++jj) acc += uv[jj] * sz[r * SC + jj];
            atomicAdd(&b[(ll)r * n + gcol], -acc);
        }
    }
}

// Pass 2, per front: z[F's columns] -= L21^T x[R_F] (L21 column k contiguous in Lf).
template <typename T, int RG>
__global__ void __launch_bounds__(256) k_tbwd_l21(const T* fac, T* z, const T* x, int n, int nrhs, Sched S, Launch L) {
    griddep_launch();
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    griddep_wait();
    front_line_dots<T, RG>(fac + F.loff + F.nf, F.ld, z, x, n, nrhs, F, S.rows + F.rows_off, tile);
}

// Pass 2, block `step`-th from the last: x_chunk = (Minv^T)[chunk, :] z_B,
// stored by the first tile, then the front's columns before the block get
// L[block rows, column]^T x_chunk subtracted (atomics across chunks).
template <typename T>
__global__ void __launch_bounds__(TS) k_tbwd(const T* fac, const T* inv2, T* z, T* x, int n, int nrhs, Sched S,
                                             Launch L, int step) {
    constexpr int BM = BlockMax<T>::value;
    __shared__ T sc[BM * MAXRHS];
    __shared__ T sp[4 * SC * MAXRHS];
    __shared__ T sx[SC * MAXRHS];
    griddep_launch();
    int fid, tile;
    locate(L, blockIdx.x, fid, tile);
    const DFront F = S.fronts[fid];
    const int blk = F.block0 + F.nblocks - 1 - step;
    const int c0 = S.blk_c0[blk], c1 = S.blk_c1[blk], bw = c1 - c0;
    const int ncc = cdiv(bw, SC), cc = tile % ncc, rt = tile / ncc;
    const int j0 = cc * SC, nj = min(SC, bw - j0);
    const T* Mi = inv2 + S.blk_inv2[blk];   // Minv(k, j) at Mi[j * bw + k]
    griddep_wait();
    const int tid = threadIdx.x;
    for (int e = tid; e < bw * nrhs; e += TS) {
        int k = e % bw, r = e / bw;
        sc[r * BM + k] = z[(ll)r * n + F.f + c0 + k];
    }
    __syncthreads();
    {
        const int j = tid & 31, kq = tid >> 5;
        T acc[MAXRHS];
#pragma unroll
        for (int r = 0; r < MAXRHS; ++r) acc[r] = T(0);
        if (j < nj) {
            const T* mcol = Mi + (ll)(j0 + j) * bw;
#pragma unroll 8
            for (int k = kq; k < bw; k += 4) {
                const T mk = mcol[k];
#pragma unroll
                for (int r = 0; r < MAXRHS; ++r)
                    if (r < nrhs) acc[r] += mk * sc[r * BM + k];
            }
        }
#pragma unroll
        for (int r = 0; r < MAXRHS; ++r)
            if (r < nrhs) sp[(kq * MAXRHS + r) * SC + j] = acc[r];
    }
    __syncthreads();
    for (int e = tid; e < SC * nrhs; e += TS) {
        int j = e % SC, r = e / SC;
        sx[r * SC + j] = sp[(0 * MAXRHS + r) * SC + j] + sp[(1 * MAXRHS + r) * SC + j] +
                         sp[(2 * MAXRHS + r) * SC + j] + sp[(3 * MAXRHS + r) * SC + j];
    }
    __syncthreads();
    if (rt == 0)
        for (int e = tid; e < nj * nrhs; e += TS) {
            int j = e % nj, r = e / nj;
            x[(ll)r * n + F.f + c0 + j0 + j] = sx[r * SC + j];
        }
    const int col = rt * TS + tid;   // a front column before the block
    if (col < c0) {
        T lv[SC];
        const T* l = fac + F.loff + (ll)col * F.ld + c0 + j0;   // L(c0 + j0 + jj, col), contiguous
#pragma unroll
        for (int jj = 0; jj < SC; ++jj) lv[jj] = jj < nj ? l[jj] : T(0);
#pragma unroll
        for (int r = 0; r < MAXRHS; ++r) {
            if (r >= nrhs) break;
            T acc = T(0);
#pragma unroll
            for (int jj = 0; jj < SC; ++jj) acc += lv[jj] * sx[r * SC + jj];
            atomicAdd(&z[(ll)r * n + F.f + col], -acc);
        }
    }
}

// dA (on A's pattern, CSC order) = -sum_r lambda_r x_r^T: the gradient of a
// loss of x = A^{-1} b with respect to A's stored entries, given the adjoint
// lambda = A^{-T} dloss/dx.
__global__ void k_grad_pattern(const int* __restrict__ row, const int* __restrict__ colof, const double* __restrict__ lam,
                               const double* __restrict__ x, ll ld, int nrhs, double* __restrict__ dA, ll nnz) {
    for (ll k = (ll)blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += (ll)gridDim.x * blockDim.x) {
        const int i = row[k], j = colof[k];
        double s = 0.0;
        for (int r = 0; r < nrhs; ++r) s += lam[(ll)r * ld + i] * x[(ll)r * ld + j];
        dA[k] = -s;
    }
}

// ---------------------------------------------------------------------------
// Assembly, permutation, residual.
// ---------------------------------------------------------------------------

// Zero-initialised factor storage += A's values at their slots (_inmatrix!).
// A's values in CSR order (aval in CSC order, src the CSC index of each CSR
// position), so that the residuals read each row's values contiguously.
__global__ void __launch_bounds__(256) k_gather_csr(const double* __restrict__ aval, const ll* __restrict__ src,
                                                    double* __restrict__ acsr, ll nnz) {
    for (ll k = blockIdx.x * (ll)blockDim.x + threadIdx.x; k < nnz; k += (ll)gridDim.x * blockDim.x)
        acsr[k] = aval[src[k]];
}

template <typename T>
__global__ void k_scatter_values(const double* __restrict__ aval, const ll* __restrict__ slot, T* fac, ll nnz) {
    ll k = (ll)blockIdx.x * blockDim.x + threadIdx.x;
    ll stride = (ll)gridDim.x * blockDim.x;
    for (; k < nnz; k += stride) atomicAdd(&fac[slot[k]], (T)aval[k]);
}

// out[i + r*n] = in[perm[i] + r*ldin]: rhs into permuted order (and precision).
template <typename Tin, typename Tout>
__global__ void k_permute(const Tin* __restrict__ in, ll ldin, Tout* __restrict__ out, ll ldout, const int* __restrict__ perm,
                          int n, int nrhs) {
    ll t = (ll)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (ll)n * nrhs) return;
    int i = (int)(t % n), r = (int)(t / n);
    out[(ll)r * ldout + i] = (Tout)in[(ll)r * ldin + perm[i]];
}

// x[j] (+)= xp[invp[j]]: solution back to original order.
template <typename Tin>
__global__ void k_unpermute(const Tin* __restrict__ xp, ll ldp, double* __restrict__ x, ll ldx, const int* __restrict__ invp,
                            int n, int nrhs, int accumulate) {
    ll t = (ll)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (ll)n * nrhs) return;
    int j = (int)(t % n), r = (int)(t / n);
    double v = (double)xp[(ll)r * ldp + invp[j]];
    if (accumulate) x[(ll)r * ldx + j] += v; else x[(ll)r * ldx + j] = v;
}

// Sums of the squares of r and b for RES_RG right-hand sides over a CTA
// (256 threads), one atomic per sum and CTA.
constexpr int RES_RG = 4;
__device__ __forceinline__ void residual_sums(double (&rr)[RES_RG], double (&bb)[RES_RG], int r0, int nr,
                                              double* __restrict__ sums) {
    __shared__ double part[8][2 * RES_RG];
#pragma unroll
    for (int q = 0; q < RES_RG; ++q)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            rr[q] += __shfl_down_sync(0xffffffffu, rr[q], off);
            bb[q] += __shfl_down_sync(0xffffffffu, bb[q], off);
        }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int q = 0; q < RES_RG; ++q) {
            part[w][2 * q] = rr[q];
            part[w][2 * q + 1] = bb[q];
        }
    __syncthreads();
    if (threadIdx.x < 2 * nr) {
        double t = 0.0;
        for (int v = 0; v < (int)(blockDim.x >> 5); ++v) t += part[v][threadIdx.x];
        atomicAdd(&sums[2 * r0 + threadIdx.x], t);
    }
    __syncthreads();
}

// r = b - A x in FP64 with A in row order (values gathered from CSC order
// through src), or r = b - A^T x with A^T's rows = A's CSC columns (src
// null); the squares of r and b are accumulated per right-hand side.  A
// thread takes a row for RES_RG right-hand sides at a time.
__global__ void __launch_bounds__(256) k_residual(const double* __restrict__ aval, const int* __restrict__ rowptr,
                                                  const int* __restrict__ col, const ll* __restrict__ src,
                                                  const double* __restrict__ x, ll ldx, const double* __restrict__ b,
                                                  ll ldb, double* __restrict__ r, int n, int nrhs,
                                                  double* __restrict__ sums) {
    for (int r0 = 0; r0 < nrhs; r0 += RES_RG) {
        const int nr = min(RES_RG, nrhs - r0);
        double rr[RES_RG], bb[RES_RG];
#pragma unroll
        for (int q = 0; q < RES_RG; ++q) rr[q] = bb[q] = 0.0;
        // grid-stride over the rows: one partial sum per CTA and right-hand side
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
            double s[RES_RG];
#pragma unroll
            for (int q = 0; q < RES_RG; ++q) s[q] = 0.0;
            for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) {
                const double a = aval[src ? src[k] : k];
                const int c = col[k];
#pragma unroll
                for (int q = 0; q < RES_RG; ++q)
                    if (q < nr) s[q] += a * x[(ll)(r0 + q) * ldx + c];
            }
#pragma unroll
            for (int q = 0; q < RES_RG; ++q)
                if (q < nr) {
                    const double bi = b[(ll)(r0 + q) * ldb + i], ri = bi - s[q];
                    r[(ll)(r0 + q) * n + i] = ri;
                    rr[q] += ri * ri;
                    bb[q] += bi * bi;
                }
        }
        residual_sums(rr, bb, r0, nr, sums);
    }
}

// ---------------------------------------------------------------------------
// GMRES-IR (refinement whose correction equation A d = r is solved by GMRES
// in FP64, preconditioned on the right by the low-precision LU).  Vectors are
// n x nrhs column-major (ld n); a basis is an array of such blocks, vector j
// at V + j * n * nrhs.  Every right-hand side has its own Krylov space.
// ---------------------------------------------------------------------------

// w = A z (FP64, rows of A; values in CSR order, or gathered from CSC order
// through src).
__global__ void __launch_bounds__(256) k_gm_spmv(const double* __restrict__ aval, const int* __restrict__ rowptr,
                                                 const int* __restrict__ col, const ll* __restrict__ src,
                                                 const double* __restrict__ z, double* __restrict__ w, int n, int nrhs) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        for (int r0 = 0; r0 < nrhs; r0 += RES_RG) {
            double acc[RES_RG] = {0.0, 0.0, 0.0, 0.0};
            for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) {
                const double a = aval[src ? src[k] : k];
                const int c = col[k];
#pragma unroll
                for (int q = 0; q < RES_RG; ++q)
                    if (r0 + q < nrhs) acc[q] += a * z[(ll)(r0 + q) * n + c];
            }
#pragma unroll
            for (int q = 0; q < RES_RG; ++q)
                if (r0 + q < nrhs) w[(ll)(r0 + q) * n + i] = acc[q];
        }
    }
}

constexpr int GM_MAXRHS = 16;

// out[j * nrhs + r] += <V_j[:, r], w[:, r]> for the basis vectors j = blockIdx.y
// (w may be V itself with nv = 1: squared norms).
__global__ void __launch_bounds__(256) k_gm_dots(const double* __restrict__ V, const double* __restrict__ w, int n,
                                                 int nrhs, double* __restrict__ out) {
    __shared__ double part[8][GM_MAXRHS];
    const int j = blockIdx.y;
    const double* v = V + (ll)j * n * nrhs;
    double acc[GM_MAXRHS];
#pragma unroll
    for (int r = 0; r < GM_MAXRHS; ++r) acc[r] = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
#pragma unroll
        for (int r = 0; r < GM_MAXRHS; ++r)
            if (r < nrhs) acc[r] += v[(ll)r * n + i] * w[(ll)r * n + i];
    const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < GM_MAXRHS; ++r) {
        double t = acc[r];
        for (int off = 16; off > 0; off >>= 1) t += __shfl_down_sync(0xffffffffu, t, off);
        if (lane == 0) part[wp][r] = t;
    }
    __syncthreads();
    if ((int)threadIdx.x < nrhs) {
        double t = 0.0;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += part[q][threadIdx.x];
        atomicAdd(&out[(ll)j * nrhs + threadIdx.x], t);
    }
}

// w[:, r] += sign * sum_{j < nv} c[j * nrhs + r] V_j[:, r]  (w has leading dimension ldw).
__global__ void __launch_bounds__(256) k_gm_axpy(const double* __restrict__ V, const double* __restrict__ c,
                                                 double* __restrict__ w, ll ldw, int n, int nrhs, int nv, double sign) {
    const ll tot = (ll)n * nrhs;
    for (ll e = (ll)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (ll)gridDim.x * blockDim.x) {
        const int r = (int)(e / n);
        const int i = (int)(e - (ll)r * n);
        double t = 0.0;
        for (int j = 0; j < nv; ++j) t += c[(ll)j * nrhs + r] * V[(ll)j * tot + e];
        w[(ll)r * ldw + i] += sign * t;
    }
}

// v[:, r] = w[:, r] / sqrt(nrm2[r]) (zero where the norm is zero).
__global__ void __launch_bounds__(256) k_gm_scale(const double* __restrict__ w, const double* __restrict__ nrm2,
                                                  double* __restrict__ v, int n, int nrhs) {
    const ll tot = (ll)n * nrhs;
    for (ll e = (ll)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (ll)gridDim.x * blockDim.x) {
        const double s = nrm2[e / n];
        v[e] = s > 0.0 ? w[e] / sqrt(s) : 0.0;
    }
}

// Norms only: sums[2r] += ||b_r - A x_r||^2 and sums[2r+1] += ||b_r||^2, with
// no residual vector written (used where no work space may be allocated).
__global__ void __launch_bounds__(256) k_residual_norms(const double* __restrict__ aval, const int* __restrict__ rowptr,
                                                        const int* __restrict__ col, const ll* __restrict__ src,
                                                        const double* __restrict__ x, ll ldx,
                                                        const double* __restrict__ b, ll ldb, int n, int nrhs,
                                                        double* __restrict__ sums) {
    for (int r0 = 0; r0 < nrhs; r0 += RES_RG) {
        const int nr = min(RES_RG, nrhs - r0);
        double rr[RES_RG], bb[RES_RG];
#pragma unroll
        for (int q = 0; q < RES_RG; ++q) rr[q] = bb[q] = 0.0;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
            double s[RES_RG];
#pragma unroll
            for (int q = 0; q < RES_RG; ++q) s[q] = 0.0;
            for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) {
                const double a = aval[src ? src[k] : k];
                const int c = col[k];
#pragma unroll
                for (int q = 0; q < RES_RG; ++q)
                    if (q < nr) s[q] += a * x[(ll)(r0 + q) * ldx + c];
            }
#pragma unroll
            for (int q = 0; q < RES_RG; ++q)
                if (q < nr) {
                    const double bi = b[(ll)(r0 + q) * ldb + i], ri = bi - s[q];
                    rr[q] += ri * ri;
                    bb[q] += bi * bi;
                }
        }
        residual_sums(rr, bb, r0, nr, sums);
    }
}

}  // namespace spk

