// Tile machinery shared by the substitution kernels (solve.cu) and the
// triangle inversion (tri.cu): small GEMMs of 32- or 64-row factor tiles
// with 32- or 40-column right operands, both staged in shared memory by
// asynchronous copies, 128 threads per CTA.
#pragma once
#include "kernels.cuh"
#include "cplx.cuh"
#include "async_copy.cuh"
#include "mma_f64.cuh"

namespace gm {

constexpr int SNB = 32;   // pivot block (= factorisation block)
constexpr int NT = 128;   // threads per CTA
// Template parameters of the kernels:
//   RT (output rows per tile, 64 or 32): 64-row tiles reuse each staged
//      right-hand-side row over more factor rows; 32-row tiles halve the
//      accumulators and the factor tile, so more CTAs fit on an SM -- the
//      better trade on the small fronts of the lower tree levels;
//   B (right-hand sides per CTA = 8 B): every slice re-stages the front's
//      factor tiles, so wider slices read the factors fewer times.

// Tile rows are padded by SPAD elements: the complex128 tile product reads
// 8 x 4 fragments (4 pivots x 8 rows), which a stride of RT + 2 spreads over
// distinct shared-memory banks.
constexpr int SPAD = 2;

template <class C, int RT, int B>
struct SolveSmem {
    C L[SNB][RT + SPAD];       // factor tile, [pivot q][row]
    C Y[SNB][8 * B + SPAD];    // right operand, [pivot q][rhs]
};

// Below, M'(i, c) is the element of the forward (L') or backward (U') factor:
// F[i + c f] for M x = b, F[c + i f] for M^T x = b.
//
// The staging helpers below issue asynchronous copies (every load of the
// tile in flight at once, no register round trip); the tile is complete
// after staged_sync().
//
// L[q][row] = M'(i0 + row, c0 + q) for row < rows, q < qb.  Entries
// outside are left as they are: the products read only q < qb, and rows >= rows
// (or right-hand sides >= rn) only feed accumulators that are never stored,
// so partial tiles stage only what they use.
// (lt = 0 .. nt - 1: the participating threads)
template <class C, bool TRANS, int RT, int KQ = SNB>
__device__ __forceinline__ void stage_factor_p(C (*L)[RT + SPAD], const C *F, int f, int i0, int rows, int c0, int qb,
                                               int lt, int nt) {
    if (!TRANS) {
        for (int t = lt; t < RT * qb; t += nt) {
            const int row = t % RT, q = t / RT;
            if (row < rows) cp_async_elem(&L[q][row], F + (i0 + row) + (size_t)(c0 + q) * f);
        }
    } else {
        for (int t = lt; t < KQ * rows; t += nt) {
            const int q = t % KQ, row = t / KQ;
            if (q < qb) cp_async_elem(&L[q][row], F + (c0 + q) + (size_t)(i0 + row) * f);
        }
    }
}

// L[q][p] = entry (p, q0 + q) of the inverse diagonal-block operator of
// pivot block k0, p < rows, q < qb:
//   FWD && !TRANS: L^-1        FWD && TRANS: (U^-1)^T
//   !FWD && !TRANS: U^-1       !FWD && TRANS: (L^-1)^T
// The stored block holds L^-1 strictly below the diagonal (unit diagonal
// implied) and U^-1 on and above it.
template <class C, bool FWD, bool TRANS, int RT, int KQ = SNB>
__device__ __forceinline__ void stage_dinv_p(C (*L)[RT + SPAD], const C *F, int f, int k0, int rows, int q0, int qb,
                                             int lt, int nt) {
    constexpr int IN = TRANS ? KQ : SNB;   // the index along the stored columns runs fastest
    for (int t = lt; t < IN * (TRANS ? rows : qb); t += nt) {
        const int p = TRANS ? t / IN : t % IN, q = TRANS ? t % IN : t / IN;
        if (TRANS ? q >= qb : p >= rows) continue;
        const bool lower_src = FWD != TRANS;         // L^-1 (or its transpose) wanted
        const int r = TRANS ? q0 + q : p, c = TRANS ? p : q0 + q;  // position in the stored block
        const bool stored = lower_src ? r > c : r <= c;
        if (stored) {
            cp_async_elem(&L[q][p], F + (k0 + r) + (size_t)(k0 + c) * f);
        } else {
            using RR = decltype(L[0][0].x);
            L[q][p] = (lower_src && r == c) ? mk(RR(1), RR(0)) : czero<C>();
        }
    }
}

// Per-thread accumulators of an RT x 8B complex output tile (128 threads,
// lt = 0 .. 127), in the layout of the tile product that fills them.
template <class C, int RT, int B>
struct TileAcc;

// complex64: CUDA-core FMAs; thread (tr, tc) = (lt / 8, lt % 8) owns rows
// tr + 16 i and columns tc + 8 j
template <int RT, int B>
struct TileAcc<float2, RT, B> {
    static constexpr int NR = RT / 16, NC = B;
    float2 v[NR][NC];
    __device__ __forceinline__ static int row(int i, int lt) { return lt / 8 + 16 * i; }
    __device__ __forceinline__ static int col(int j, int lt) { return lt % 8 + 8 * j; }
};

// complex128: FP64 matrix instructions (mma.sync m8n8k4 f64) on 8 x 8
// blocks; warp w owns row blocks w + 4 i, lane l row 8 (w + 4 i) + l / 4 of
// them and columns 8 c + 2 (l % 4) + {0, 1} of every column block c
template <int RT, int B>
struct TileAcc<double2, RT, B> {
    static constexpr int NR = RT / 32, NC = 2 * B;
    double2 v[NR][NC];
    __device__ __forceinline__ static int row(int i, int lt) { return 8 * ((lt >> 5) + 4 * i) + ((lt & 31) >> 2); }
    __device__ __forceinline__ static int col(int j, int lt) { return 8 * (j >> 1) + 2 * (lt & 3) + (j & 1); }
};

template <class C, int RT, int B>
__device__ __forceinline__ void zero_acc(TileAcc<C, RT, B> &acc) {
#pragma unroll
    for (int i = 0; i < TileAcc<C, RT, B>::NR; ++i)
#pragma unroll
        for (int j = 0; j < TileAcc<C, RT, B>::NC; ++j) acc.v[i][j] = czero<C>();
}

// f(row, col, value) for the thread's accumulators with row < rows, col < rn
template <class C, int RT, int B, class F>
__device__ __forceinline__ void for_acc(TileAcc<C, RT, B> &acc, int rows, int rn, int lt, F f) {
    using A = TileAcc<C, RT, B>;
#pragma unroll
    for (int i = 0; i < A::NR; ++i) {
        const int row = A::row(i, lt);
        if (row >= rows) continue;
#pragma unroll
        for (int j = 0; j < A::NC; ++j) {
            const int col = A::col(j, lt);
            if (col < rn) f(row, col, acc.v[i][j]);
        }
    }
}

// acc += L'[rows x qb] Y[qb x rn]: L[q][row] holds operator entry (row, q),
// Y[q][col] the right operand.  Rows >= `rows` and columns >= rn of the
// tile only feed accumulators that are never stored; row and column groups
// that lie entirely outside are skipped warp-uniformly, so small fronts and
// short slices do not pay for the full tile.
//
// complex64: each thread accumulates its 16-row-strided rows x 8-column-
// strided columns with CUDA-core FMAs, one pivot q at a time
template <int RT, int B>
__device__ __forceinline__ void tile_mma_p(const float2 (*L)[RT + SPAD], const float2 (*Y)[8 * B + SPAD], int qb,
                                           TileAcc<float2, RT, B> &acc, int rows, int rn, int lt) {
    constexpr int A = RT / 16;
    const int tr = lt / 8, tc = lt % 8;
    const int wrow = (lt >> 5) * 4;   // a warp owns rows 4w .. 4w + 3 of each 16-row group
    const int na = rows <= wrow ? 0 : min(A, (rows - wrow + 15) / 16);
    const int nb = min(B, (rn + 7) / 8);
    if (na == 0) return;   // warp-uniform: this warp owns no row of the tile
#pragma unroll 2
    for (int q = 0; q < qb; ++q) {
        float2 l[A], y[B];
#pragma unroll
        for (int a = 0; a < A; ++a) l[a] = a < na ? L[q][tr + 16 * a] : czero<float2>();
#pragma unroll
        for (int b = 0; b < B; ++b) y[b] = b < nb ? Y[q][tc + 8 * b] : czero<float2>();
#pragma unroll
        for (int a = 0; a < A; ++a) {
            if (a >= na) break;
#pragma unroll
            for (int b = 0; b < B; ++b)
                if (b < nb) cfma(acc.v[a][b], l[a], y[b]);
        }
    }
}

// complex128: per 4 pivots and per 8 x 8 block, four FP64 matrix
// instructions (Re += Ar Br - Ai Bi, Im += Ar Bi + Ai Br); a lane loads one
// complex entry of each left and right fragment.  Pivots q >= qb enter as
// zeros.
template <int RT, int B>
__device__ __forceinline__ void tile_mma_p(const double2 (*L)[RT + SPAD], const double2 (*Y)[8 * B + SPAD], int qb,
                                           TileAcc<double2, RT, B> &acc, int rows, int rn, int lt) {
    constexpr int NRB = RT / 32;
    const int w = lt >> 5, lane = lt & 31;
    const int nb = min(B, (rn + 7) / 8);
    for (int k0 = 0; k0 < qb; k0 += 4) {
        const int kk = k0 + (lane & 3);
        const bool kin = kk < qb;
        double2 bf[B];
#pragma unroll
        for (int b = 0; b < B; ++b) bf[b] = kin && b < nb ? Y[kk][8 * b + (lane >> 2)] : czero<double2>();
#pragma unroll
        for (int i = 0; i < NRB; ++i) {
            const int rb = w + 4 * i;   // row block: rows 8 rb .. 8 rb + 7
            if (8 * rb >= rows) break;   // warp-uniform
            const double2 af = kin ? L[kk][8 * rb + (lane >> 2)] : czero<double2>();
#pragma unroll
            for (int b = 0; b < B; ++b) {
                if (b >= nb) break;
                cmma_884(af, bf[b], acc.v[i][2 * b], acc.v[i][2 * b + 1]);
            }
        }
    }
}

// 32 x 32 output tile of the small-front kernels in 8 x 8 blocks, dealt to
// the four warps by columns (warp w: block column w, every row block) or, in
// slices of at most 16 columns, by rows.  By rows alone a front of 6 pivots
// kept one warp busy and one of 20 three -- and always the same ones, so that
// one of the SM's four schedulers carried the level.
// (NB8: blocks per warp kept, at least 2 for the slices dealt by rows)
template <class C, int NB8 = 4>
struct BlockTile {
    static constexpr int N = NB8;
    C v[N][2];   // this lane's two entries of the warp's blocks
    bool bycol;
    int w, lane;
    // (by rows: the first row block goes to another warp in every front)
    __device__ __forceinline__ BlockTile(int rn, int turn) {
        lane = threadIdx.x & 31;
        bycol = rn > 16;
        w = (threadIdx.x >> 5) + (bycol ? 0 : turn) & 3;
        zero();
    }
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i][0] = v[i][1] = czero<C>();
    }
    __device__ __forceinline__ int row(int i) const { return 8 * (bycol ? i : w) + (lane >> 2); }
    __device__ __forceinline__ int col(int i, int e) const {
        return 8 * (bycol ? w : i) + (sizeof(C) == 16 ? 2 * (lane & 3) + e : (lane & 3) + 4 * e);
    }
    // f(row, col, value) over the lane's entries with row < rows, col < rn
    template <class F>
    __device__ __forceinline__ void each(int rows, int rn, F f) {
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (row(i) < rows && col(i, e) < rn) f(row(i), col(i, e), v[i][e]);
    }
};

// acc += L'[rows x qb] Y[qb x rn], operands as tile_mma_p.  TRI: 0 a full
// operator; TRI_LOWER / TRI_UPPER a triangular one (the diagonal-block
// inverses), whose column q has no entries above / below row q: row blocks that
// column q does not reach are skipped for that q.
constexpr int TRI_LOWER = 1, TRI_UPPER = 2;
template <int TRI, int LW, int N>
__device__ __forceinline__ void block_mma(const double2 (*L)[LW], const double2 (*Y)[32 + SPAD], int qb,
                                          BlockTile<double2, N> &acc, int rows, int rn) {
    const int g = acc.lane >> 2, w = acc.w;
    const int n = acc.bycol ? (rows + 7) / 8 : (rn + 7) / 8;   // blocks of this warp
    if (8 * w >= (acc.bycol ? rn : rows)) return;              // warp-uniform
    for (int k0 = 0; k0 < qb; k0 += 4) {
        const int kk = k0 + (acc.lane & 3);
        const bool kin = kk < qb;
        if (acc.bycol) {
            const double2 b = kin ? Y[kk][8 * w + g] : czero<double2>();
#pragma unroll
            for (int i = 0; i < N; ++i) {
                if (i >= n || (TRI == TRI_UPPER && 8 * i > k0 + 3)) break;
                if (TRI == TRI_LOWER && 8 * i + 7 < k0) continue;
                cmma_884(kin ? L[kk][8 * i + g] : czero<double2>(), b, acc.v[i][0], acc.v[i][1]);
            }
        } else {
            if ((TRI == TRI_UPPER && 8 * w > k0 + 3) || (TRI == TRI_LOWER && 8 * w + 7 < k0)) continue;
            const double2 a = kin ? L[kk][8 * w + g] : czero<double2>();
#pragma unroll
            for (int i = 0; i < N; ++i) {
                if (i >= n) break;
                cmma_884(a, kin ? Y[kk][8 * i + g] : czero<double2>(), acc.v[i][0], acc.v[i][1]);
            }
        }
    }
}
template <int TRI, int LW, int N>
__device__ __forceinline__ void block_mma(const float2 (*L)[LW], const float2 (*Y)[32 + SPAD], int qb,
                                          BlockTile<float2, N> &acc, int rows, int rn) {
    const int g = acc.lane >> 2, kq = acc.lane & 3, w = acc.w;
    const int n = acc.bycol ? (rows + 7) / 8 : (rn + 7) / 8;
    if (8 * w >= (acc.bycol ? rn : rows)) return;
    if (acc.bycol) {
#pragma unroll 2
        for (int k = 0; k < qb; ++k) {
            const float2 y0 = Y[k][8 * w + kq], y1 = Y[k][8 * w + kq + 4];
#pragma unroll
            for (int i = 0; i < N; ++i) {
                if (i >= n || (TRI == TRI_UPPER && 8 * i > k)) break;
                if (TRI == TRI_LOWER && 8 * i + 7 < k) continue;
                const float2 l = L[k][8 * i + g];
                cfma(acc.v[i][0], l, y0);
                cfma(acc.v[i][1], l, y1);
            }
        }
    } else {
        for (int k = 0; k < qb; ++k) {
            if ((TRI == TRI_UPPER && 8 * w > k) || (TRI == TRI_LOWER && 8 * w + 7 < k)) continue;
            const float2 l = L[k][8 * w + g];
#pragma unroll
            for (int i = 0; i < N; ++i) {
                if (i >= n) break;
                cfma(acc.v[i][0], l, Y[k][8 * i + kq]);
                cfma(acc.v[i][1], l, Y[k][8 * i + kq + 4]);
            }
        }
    }
}

// Y[q][r] = row_ptr(q)[r] for q < qb, r < rn (entries outside: as above)
template <class C, int TC, class RowPtr>
__device__ __forceinline__ void stage_rows_p(C (*Y)[TC + SPAD], RowPtr row_ptr, int qb, int rn, int lt, int nt) {
    for (int t = lt; t < qb * TC; t += nt) {
        const int q = t / TC, r = t % TC;
        if (r < rn) cp_async_elem(&Y[q][r], row_ptr(q) + r);
    }
}

}  // namespace gm
