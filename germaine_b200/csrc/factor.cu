// K2-K4: numeric multifrontal LU of one elimination-tree level, batched
// over every front of the level and every frequency (the replacement of
// umfpack_zi_numeric, src/AC/forward_shot_AC.c:61).
//
// Fronts live in HBM as dense column-major nfront x nfront complex blocks
// (one block per node per frequency).  A level is processed by
//   K2 gather   -- each front's pivot rows and columns pull their children's
//                  contribution blocks (extend-add by inverse maps:
//                  deterministic, no atomics),
//   K3 diag     -- adds the operator entries owned by the front (first block),
//                  then per NB-wide pivot block: LU of the diagonal block with
//                  threshold partial pivoting inside the block (static
//                  pivots as the last resort) and the inverses of its two
//                  triangles, factored once per front (the first block by
//                  k_diag, each later one by the first CTA of the preceding
//                  K4),
//   K3 panels   -- L21 = A21 U11^-1 and U12 = L11^-1 P A12 as products with
//                  those inverses (FP64 matrix instructions in complex128),
//   K4 update   -- rank-NB Schur update of the pivot rows and columns still
//                  to come, 64x64 or 32x32 tiles.
// K3/K4 alternate ceil(max_piv/NB) times per level.  After the last step a
// front holds L (unit lower) and U in its first npiv rows/columns -- except
// that each NB x NB diagonal block holds the INVERSES of its two triangles
// (what the substitution multiplies by) -- and its Schur complement (the
// contribution block) in the trailing block.  With row exchanges, the rows
// of a block's diagonal block and U part are in pivot order, its rows'
// multipliers of earlier blocks in equation order, and the block's
// permutation is in FactorArgs::pivsrc.
//
// Two fused kernels leave the same layout:
//   k_factor_front  fronts that fit shared memory whole (the lower levels):
//                   extend-add, entries, LU and Schur complement in one CTA;
//   k_factor_mid    on request (GM_MID_MAX_PIV): fronts with at most NB pivots
//                   and at most 256 rows above those: after K2, one CTA
//                   factorises the pivot columns and applies the Schur update
//                   to the contribution block once, in place of K3 / K4 and the
//                   contribution GEMM.
// The remaining (upper) levels take the blocked K2-K4 sequence.
#include <algorithm>
#include <cstdlib>
#include <type_traits>
#include "kernels.cuh"
#include "cplx.cuh"
#include "async_copy.cuh"
#include "mma_f64.cuh"

namespace gm {

constexpr int NB = 32;       // pivot block width
constexpr int TILE = 64;     // panel and Schur-update tile
constexpr int kTileFill = kGemmTileFill;

constexpr int GATHER_COLS = 4;   // front columns per CTA of the extend-add gather
constexpr int TSTR = TILE + 2;   // padded row stride of staged 64-wide tiles (conflict-free 8 x 4 fragments)

// TL x TL complex output tile (TL 64 or 32) of a 256-thread CTA, in the layout
// of the product that fills it: complex64 with CUDA-core FMAs, thread t owning
// rows t % 16 + 16 i and columns t / 16 + 16 j (v[i][j]); complex128 on FP64
// matrix instructions (mma.sync m8n8k4 f64) on 8 x 8 blocks, lane l holding
// row 8 rb + l / 4 and columns 8 cb + 2 (l % 4) + j of each block its warp w
// owns: for TL = 64 row blocks w % 4 and w % 4 + 4 of column blocks 4 (w / 4)
// .. 4 (w / 4) + 3 (v[4 rbi + cbi], so a tile with few rows still keeps six of
// the eight warps busy), for TL = 32 row block w % 4 of column blocks
// 2 (w / 4) and 2 (w / 4) + 1 (v[cbi]).
template <class C, bool MMA, int TL>
struct TileCC;
template <class C, int TL>
struct TileCC<C, false, TL> {   // CUDA-core FMAs (complex64, or complex128 where short K suits them better)
    static constexpr int NI = TL / 16, NJ = TL / 16;
    C v[NI][NJ];
    __device__ __forceinline__ static int row(int i, int, int t) { return t % 16 + 16 * i; }
    __device__ __forceinline__ static int col(int, int j, int t) { return t / 16 + 16 * j; }
};
template <int TL>
struct TileCC<double2, true, TL> {   // FP64 matrix instructions
    static constexpr int NRB = TL / 32, NCB = TL / 16, NI = NRB * NCB, NJ = 2;
    double2 v[NI][NJ];
    __device__ __forceinline__ static int row(int i, int, int t) {
        return 8 * ((t >> 5) % 4 + 4 * (i / NCB)) + ((t & 31) >> 2);
    }
    __device__ __forceinline__ static int col(int i, int j, int t) {
        return 8 * (NCB * ((t >> 5) / 4) + i % NCB) + 2 * (t & 3) + j;
    }
};

// f(row, col, value) over the thread's entries of the tile
template <class C, bool MMA, int TL, class F>
__device__ __forceinline__ void for_tile(TileCC<C, MMA, TL> &acc, int t, F f) {
    using T = TileCC<C, MMA, TL>;
#pragma unroll
    for (int i = 0; i < T::NI; ++i)
#pragma unroll
        for (int j = 0; j < T::NJ; ++j) f(T::row(i, j, t), T::col(i, j, t), acc.v[i][j]);
}

// acc += A B (NEG: acc -= A B) over k < kb, A(r, k) = As[k * ak + r * ar]
// for rows r < mrows, B(k, c) = Bs[k * bk + c * bc] for columns c < ncols
// (entries outside read as zero)
template <bool NEG, class C, int TL>
__device__ __forceinline__ void mma_tile(const C *As, int ak, int ar, const C *Bs, int bk, int bc, int kb, int mrows,
                                         int ncols, TileCC<C, false, TL> &acc, int t) {
    constexpr int NT = TL / 16;
    const int tx = t % 16, ty = t / 16;
    for (int k = 0; k < kb; ++k) {
        C lv[NT], uv[NT];
#pragma unroll
        for (int i = 0; i < NT; ++i)
            lv[i] = tx + 16 * i < mrows ? As[(size_t)k * ak + (size_t)(tx + 16 * i) * ar] : czero<C>();
#pragma unroll
        for (int j = 0; j < NT; ++j)
            uv[j] = ty + 16 * j < ncols ? Bs[(size_t)k * bk + (size_t)(ty + 16 * j) * bc] : czero<C>();
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                if (NEG) cfms(acc.v[i][j], lv[i], uv[j]);
                else cfma(acc.v[i][j], lv[i], uv[j]);
            }
    }
}

template <bool NEG, int TL>
__device__ __forceinline__ void mma_tile(const double2 *As, int ak, int ar, const double2 *Bs, int bk, int bc, int kb,
                                         int mrows, int ncols, TileCC<double2, true, TL> &acc, int t) {
    using T = TileCC<double2, true, TL>;
    const int w = t >> 5, lane = t & 31, g = lane >> 2;
    const int rb0 = w % 4, cb0 = T::NCB * (w / 4);
    if (8 * rb0 >= mrows || 8 * cb0 >= ncols) return;   // warp-uniform: none of this warp's blocks is used
    for (int k0 = 0; k0 < kb; k0 += 4) {
        const int kk = k0 + (lane & 3);
        const bool kin = kk < kb;
        double2 bf[T::NCB];
#pragma unroll
        for (int ci = 0; ci < T::NCB; ++ci) {
            const int c = 8 * (cb0 + ci) + g;
            bf[ci] = kin && c < ncols ? Bs[(size_t)kk * bk + (size_t)c * bc] : czero<double2>();
        }
#pragma unroll
        for (int ri = 0; ri < T::NRB; ++ri) {
            const int rb = rb0 + 4 * ri;
            if (8 * rb >= mrows) break;   // warp-uniform
            const int r = 8 * rb + g;
            double2 af = kin && r < mrows ? As[(size_t)kk * ak + (size_t)r * ar] : czero<double2>();
            if (NEG) af = make_double2(-af.x, -af.y);
#pragma unroll
            for (int ci = 0; ci < T::NCB; ++ci) {
                if (8 * (cb0 + ci) >= ncols) break;   // warp-uniform
                cmma_884(af, bf[ci], acc.v[T::NCB * ri + ci][0], acc.v[T::NCB * ri + ci][1]);
            }
        }
    }
}

// (pivots: only the pivot rows and columns, the contribution-block kernel
// gathers the rest itself)
template <class R>
__global__ void k_front_gather(FactorArgs<R> a, int lvl_first, int pivots) {
    using C = cplx<R>;
    const NodeDesc d = a.s.desc[lvl_first + blockIdx.y];
    const int f = d.nfront;
    const int rows = pivots && blockIdx.x * GATHER_COLS >= (unsigned)d.npiv ? d.npiv : f;   // of this CTA's columns
    const int j = blockIdx.x * GATHER_COLS + (threadIdx.x >> 5);   // one warp per front column
    if (j >= f) return;   // warp-uniform (no barrier below)
    C *base = reinterpret_cast<C *>(a.front) + (size_t)blockIdx.z * a.s.front_total;
    C *F = base + d.front_off;
    const int *inv = a.s.inv + d.inv_off;
    const int b0 = d.child0 >= 0 ? inv[j] : -1;
    const int b1 = d.child1 >= 0 ? inv[f + j] : -1;
    const C *cb0 = b0 >= 0 ? base + d.cb0 + (size_t)b0 * d.ld0 : nullptr;
    const C *cb1 = b1 >= 0 ? base + d.cb1 + (size_t)b1 * d.ld1 : nullptr;
    for (int i = threadIdx.x & 31; i < rows; i += 32) {
        C v = czero<C>();
        if (cb0) { const int r = inv[i]; if (r >= 0) v = cadd(v, cb0[r]); }
        if (cb1) { const int r = inv[f + i]; if (r >= 0) v = cadd(v, cb1[r]); }
        F[i + (size_t)j * f] = v;
    }
}

// the operator entries owned by the front, added into it by one CTA
// (positions are distinct)
template <class R>
__device__ __forceinline__ void add_entries(const FactorArgs<R> &a, const NodeDesc &nd, int z) {
    using C = cplx<R>;
    C *F = reinterpret_cast<C *>(a.front) + (size_t)z * a.s.front_total;
    const double2 *A = a.A + (size_t)z * 9 * a.s.n;
    const int64_t e1 = nd.ent_first + nd.ent_count;
    for (int64_t e = nd.ent_first + threadIdx.x; e < e1; e += blockDim.x) {
        C &d = F[a.ent_dst[e]];
        d = cadd(d, cconv<C>(A[a.ent_src[e]]));
    }
}

// Static pivoting: a pivot of magnitude below pivtol (or NaN) is replaced by
// itself scaled to magnitude pivtol (pivtol when it is zero) and counted.
// The test compares squares, so the common case takes no square root; where
// pivtol^2 underflows to zero every square would pass, and magnitudes are
// compared (a caller that tests the square first has to come here then).
template <class R>
__device__ __forceinline__ cplx<R> static_pivot(cplx<R> piv, R pivtol, int &npert) {
    const R m2 = cabs2(piv), tol2 = pivtol * pivtol;
    const bool small = tol2 > R(0) ? !(m2 >= tol2) : !(sqrt(m2) >= pivtol);   // also catches NaN
    if (small) {
        const R mag = sqrt(m2);
        if (mag > R(0)) {
            const R sc = pivtol / mag;
            piv = mk(piv.x * sc, piv.y * sc);
        } else {
            piv = mk(pivtol, R(0));
        }
        ++npert;
    }
    return piv;
}

// LU of the kb x kb diagonal block at (k0, k0) of the front F (leading
// dimension f), with threshold row exchanges inside the block or without
// (PIV), a pivot that stays tiny replaced as static_pivot does; the inverses
// of its two triangles are written back in its place (all that the panel
// products and the substitution use): L^-1 in the strict lower part (unit
// diagonal implied), U^-1 in the upper part with the diagonal.
//
// Both inverses are built during the elimination, in place, by 8-pivot
// panels q.  With the panel's own triangles L_q, U_q, the block rows / columns
// it meets change as
//   row q     X_qc := L_q^-1 X_qc (c < q),   U_qc = L_q^-1 D_qc,  Z_qc := -U_q^-1 U_qc (c > q)
//   column q  Z_rq := Z_rq U_q^-1 (r < q),   L_rq = D_rq U_q^-1,  X_rq := -L_rq L_q^-1 (r > q)
//   others    T_rc -= a_r b_c with a = Z_rq or L_rq, b = X_qc or U_qc, except r < q and c < q
// (X the finished part of L^-1 below, Z that of U^-1 above the diagonal; one
// array holds D, X and Z).  Per panel:
//   1. warp 0 factors it with a row per lane and its 8 columns in registers:
//      the pivot row goes round by shuffles, so a pivot costs no block
//      barrier, and its reciprocal is formed while the search (one warp
//      reduction) is still out;
//   2. warp 0 solves with L_q for the 24 other columns and the identity (b),
//      warp 1 with U_q for the 24 other rows and the identity (a), a column /
//      row per lane;
//   3. all warps form the 16 products a_r b_c on 8 x 8 blocks.
// Row exchanges: position p goes to the row of largest |D(r, p)| among those
// left when the row there has |D(p, p)|^2 < pivtau2 |D(r, p)|^2; whole rows of
// the array trade places (a few per front).
// The block's permutation goes to pivsrc[vars[k0 + q]] (q: pivot position,
// value: block row in equation order); columns right of the block are
// exchanged when the U panel is staged, columns left of it (earlier blocks'
// multipliers) stay in equation order -- the forward substitution gathers the
// block's rows at the same point of the elimination.
//
// The block is the serial part of every pivot step of the upper levels.
// Pivot by pivot over all 256 threads (two barriers and ~155 dependent
// instructions each) k_diag took 31 us for 32 complex128 pivots alone on an
// SM; so it takes 21 us (24.5k cycles after the loads: four panels of 4250,
// the triangle solves 520 each, the products 1400 each), and an update launch
// of a top level, which ends in one, 22.5 us instead of 48.  The CTA has DIAG_THREADS threads; sm is shared scratch of
// DIAG_SCRATCH complex values.
constexpr int PW8 = 8;       // panel width
constexpr int DSTR = NB + 1;
constexpr int ASTR = PW8 + 4, BSTR = NB + 2;   // strides of conflict-free 8 x 4 / 4 x 8 fragments
constexpr int DIAG_SCRATCH = NB * DSTR + NB * ASTR + PW8 * BSTR + NB;
constexpr int DIAG_THREADS = 256;

// leading bits of a non-negative value: ordered as the value is
__device__ __forceinline__ int lead_bits(double v) { return __double2hiint(v); }
__device__ __forceinline__ int lead_bits(float v) { return __float_as_int(v); }
__device__ __forceinline__ double from_lead(int b, double) { return __hiloint2double(b, 0); }
__device__ __forceinline__ float from_lead(int b, float) { return __int_as_float(b); }

// acc (this lane's two entries of an 8 x 8 block: row l / 4, columns
// 2 (l % 4) + {0, 1}) -= A B, A(r, j) = Ab[r * sa + j], B(j, c) = Bb[j * sb + c], j < 8
__device__ __forceinline__ void block8_sub(const double2 *Ab, int sa, const double2 *Bb, int sb, double2 *acc, int lane) {
    const int g = lane >> 2, kq = lane & 3;
#pragma unroll
    for (int j = 0; j < PW8; j += 4) {
        const double2 v = Ab[g * sa + j + kq];
        cmma_884(make_double2(-v.x, -v.y), Bb[(j + kq) * sb + g], acc[0], acc[1]);
    }
}
__device__ __forceinline__ void block8_sub(const float2 *Ab, int sa, const float2 *Bb, int sb, float2 *acc, int lane) {
    const int g = lane >> 2, kq = lane & 3;
#pragma unroll
    for (int j = 0; j < PW8; ++j) {
        const float2 v = Ab[g * sa + j];
        cfms(acc[0], v, Bb[j * sb + 2 * kq]);
        cfms(acc[1], v, Bb[j * sb + 2 * kq + 1]);
    }
}

// The lane whose row takes the pivot's place by the threshold rule: the largest
// m2 = |entry|^2 of the column (the lowest lane among equals) when piv2 =
// |pivot|^2 is below pivtau2 times that, else -1; the same in every lane.
// key: lead_bits(m2), -1 where the lane has no candidate.  The chain of the
// pivots carries one warp reduction over the keys.  In complex128 it sees half
// of the bits: rows can only be exchanged if the leading bits of piv2 pivreach
// (below piv2 / pivtau2 by more than it is rounded; formed while the reduction
// is out) do not lead its result, and behind that the remaining bits decide.
__device__ __forceinline__ int exchange_lane(const FactorArgs<double> &a, double m2, int key, double piv2) {
    constexpr unsigned ALL = 0xffffffffu;
    const int top = __reduce_max_sync(ALL, key);
    if (lead_bits(piv2 * a.pivreach) > top) return -1;
    const unsigned lo = key == top ? (unsigned)__double2loint(m2) : 0u;
    const unsigned l = __reduce_max_sync(ALL, lo);
    const int arg = __ffs(__ballot_sync(ALL, key == top && lo == l)) - 1;
    return piv2 < a.pivtau2 * __hiloint2double(top, (int)l) ? arg : -1;
}
__device__ __forceinline__ int exchange_lane(const FactorArgs<float> &a, float, int key, float piv2) {
    const int top = __reduce_max_sync(0xffffffffu, key);
    if (!(piv2 < (float)a.pivtau2 * from_lead(top, 0.f))) return -1;
    return __ffs(__ballot_sync(0xffffffffu, key == top)) - 1;
}

template <class R, bool PIV>
__device__ void factor_diag_block(const FactorArgs<R> &a, cplx<R> *F, int f, int k0, int kb, cplx<R> *sm,
                                  unsigned char *src, const int *vars) {
    using C = cplx<R>;
    constexpr unsigned ALL = 0xffffffffu;
    C *T = sm;                                // [NB][DSTR]
    C *Ab = T + NB * DSTR;                    // [NB][ASTR]
    C *Bb = Ab + NB * ASTR;                   // [PW8][BSTR]
    C *rd = Bb + PW8 * BSTR;                  // [NB] reciprocal pivots
    __shared__ int rowat[NB];                 // block row (equation order) at pivot position q
    const R pivtol = (R)(a.pivscale * __longlong_as_double((long long)*a.amax)), tol2 = pivtol * pivtol;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid < NB) {
        rowat[tid] = tid;
        rd[tid] = czero<C>();
    }
    for (int t = tid; t < NB * NB; t += DIAG_THREADS) {   // rows and columns beyond kb: zero throughout
        const int r = t % NB, c = t / NB;
        T[r * DSTR + c] = r < kb && c < kb ? F[(k0 + r) + (size_t)(k0 + c) * f] : czero<C>();
    }
    __syncthreads();
    int np = 0, nsw = 0;      // pivots perturbed / exchanged (warp 0: the same in every lane)
#pragma unroll 1
    for (int q = 0; q * PW8 < kb; ++q) {
        const int p0 = q * PW8, pw = min(PW8, kb - p0);
        C *Tq = T + p0 * DSTR + p0;   // the panel's own 8 x 8 block
        if (warp == 0) {   // 1. the panel: x[i] = this row's entry in column p + i
            C x[PW8];
            C *own = T + lane * DSTR;
#pragma unroll
            for (int i = 0; i < PW8; ++i) x[i] = own[p0 + i];
            // pivots j0 .. j1 - 1 of the panel, W of its columns still live (no
            // divergent branch: each costs the chain)
            auto pivots = [&](auto width, int j0, int j1) {
                constexpr int W = decltype(width)::value;
#pragma unroll 1
                for (int j = j0; j < j1; ++j) {
                    const int p = p0 + j;
                    C pr[W];   // the pivot row
#pragma unroll
                    for (int i = 0; i < W; ++i) pr[i] = mk(__shfl_sync(ALL, x[i].x, p), __shfl_sync(ALL, x[i].y, p));
                    C rp = crcp(pr[0]);
                    if (PIV) {
                        const R m2 = cabs2(x[0]);
                        const int key = lane >= p && lane < kb ? lead_bits(m2) : -1;
                        const int arg = exchange_lane(a, m2, key, cabs2(pr[0]));
                        if (arg > p) {   // rows p and arg trade places
                            __syncwarp();   // the multipliers that other lanes stored (shuffles order no memory)
                            const int from = lane == p ? arg : lane == arg ? p : lane;
#pragma unroll
                            for (int i = 0; i < W; ++i) {
                                pr[i] = mk(__shfl_sync(ALL, x[i].x, arg), __shfl_sync(ALL, x[i].y, arg));
                                x[i] = mk(__shfl_sync(ALL, x[i].x, from), __shfl_sync(ALL, x[i].y, from));
                            }
                            const C u = T[p * DSTR + lane], v = T[arg * DSTR + lane];
                            T[p * DSTR + lane] = v;
                            T[arg * DSTR + lane] = u;
                            if (lane == 0) {
                                const int t = rowat[p];
                                rowat[p] = rowat[arg];
                                rowat[arg] = t;
                            }
                            __syncwarp();
                            rp = crcp(pr[0]);
                            ++nsw;
                        }
                    }
                    C piv = pr[0];
                    if (!(cabs2(piv) >= tol2) || !(tol2 > R(0))) {   // rare, off the chain: rp is formed already
                        piv = static_pivot<R>(piv, pivtol, np);
                        rp = crcp(piv);
                    }
                    const C l = lane > p ? cmul(x[0], rp) : czero<C>();   // rows p and above are final
                    own[p] = lane > p ? l : lane == p ? piv : x[0];
                    if (lane == p) rd[p] = rp;
#pragma unroll
                    for (int i = 1; i < W; ++i) {
                        C v = x[i];
                        cfms(v, l, pr[i]);
                        x[i - 1] = v;
                    }
                    x[W - 1] = czero<C>();
                }
            };
            pivots(std::integral_constant<int, PW8>(), 0, min(pw, PW8 / 2));
            pivots(std::integral_constant<int, PW8 / 2>(), PW8 / 2, pw);
        }
        __syncthreads();
        // 2. the panel's triangles applied to its rows and columns (rows and
        // columns beyond kb hold zeros: no cases for a short last panel)
        const int ql = lane - p0;   // 0 .. 7: this lane takes a column / row of the identity
        const bool mid = ql >= 0 && ql < PW8;
        if (warp == 0) {   // b: columns `lane` of the panel's rows
            C v[PW8];
#pragma unroll
            for (int j = 0; j < PW8; ++j)
                v[j] = mid ? mk(R(j == ql && j < pw), R(0)) : T[(p0 + j) * DSTR + lane];
#pragma unroll
            for (int i = 0; i + 1 < PW8; ++i)
#pragma unroll
                for (int j = i + 1; j < PW8; ++j) cfms(v[j], Tq[j * DSTR + i], v[i]);
#pragma unroll
            for (int j = 0; j < PW8; ++j) Bb[j * BSTR + lane] = v[j];
        } else if (warp == 1) {   // a: rows `lane` of the panel's columns
            C v[PW8];
#pragma unroll
            for (int j = 0; j < PW8; ++j)
                v[j] = mid ? mk(R(j == ql && j < pw), R(0)) : T[lane * DSTR + p0 + j];
            if (ql < PW8) {   // (rows below hold their multipliers already)
#pragma unroll
                for (int i = 0; i < PW8; ++i) {
                    v[i] = cmul(v[i], rd[p0 + i]);
#pragma unroll
                    for (int j = i + 1; j < PW8; ++j) cfms(v[j], v[i], Tq[i * DSTR + j]);
                }
            }
#pragma unroll
            for (int j = 0; j < PW8; ++j) Ab[lane * ASTR + j] = v[j];
        }
        __syncthreads();
        // 3. 8 x 8 blocks (bi, bj) of the array, two per warp
        const int g = lane >> 2, kq = lane & 3;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int bi = warp & 3, bj = (warp >> 2) + 2 * e;
            if (bi < q && bj < q) continue;
            C *d = T + (8 * bi + g) * DSTR + 8 * bj + 2 * kq;
            const C *ar = Ab + (8 * bi + g) * ASTR + 2 * kq, *bc = Bb + g * BSTR + 8 * bj + 2 * kq;
            C v[2];
            if (bi == q && bj == q) {   // L_q^-1 below, U_q^-1 on and above the diagonal
                v[0] = g > 2 * kq ? bc[0] : ar[0];
                v[1] = g > 2 * kq + 1 ? bc[1] : ar[1];
            } else if (bi == q && bj < q) {
                v[0] = bc[0];
                v[1] = bc[1];
            } else if (bi < q && bj == q) {
                v[0] = ar[0];
                v[1] = ar[1];
            } else {   // T - a b, the panel's own rows and columns starting from zero
                v[0] = v[1] = czero<C>();
                if (bi != q && bj != q) {
                    v[0] = d[0];
                    v[1] = d[1];
                }
                block8_sub(Ab + 8 * bi * ASTR, ASTR, Bb + 8 * bj, BSTR, v, lane);
            }
            d[0] = v[0];
            d[1] = v[1];
        }
        __syncthreads();
    }
    for (int t = tid; t < NB * NB; t += DIAG_THREADS) {
        const int r = t % NB, c = t / NB;
        if (r < kb && c < kb) F[(k0 + r) + (size_t)(k0 + c) * f] = T[r * DSTR + c];
    }
    if (PIV && tid < kb) src[vars[k0 + tid]] = (unsigned char)rowat[tid];
    if (tid == 0) {
        if (np) atomicAdd(a.npert, (unsigned long long)np);
        if (PIV && nsw) atomicAdd(a.nswap, (unsigned long long)nsw);
    }
}

// the diagonal block (k0, kb) of the front in matrix z, with row exchanges
// when piv (the level's fronts have more than NB pivots)
template <class R>
__device__ __forceinline__ void diag_block(const FactorArgs<R> &a, cplx<R> *F, const NodeDesc &d, int z, int k0, int kb,
                                           cplx<R> *sm, bool piv) {
    if (piv) {
        factor_diag_block<R, true>(a, F, d.nfront, k0, kb, sm, a.pivsrc + (size_t)z * a.s.n, a.s.vars + d.var_off);
    } else {
        factor_diag_block<R, false>(a, F, d.nfront, k0, kb, sm, nullptr, nullptr);
    }
}

// K2 + K3a: the front's operator entries, then its first diagonal block (the
// later ones are factored by the first CTA of the preceding trailing update)
template <class R>
__global__ void __launch_bounds__(DIAG_THREADS) k_diag(FactorArgs<R> a, int lvl_first, int piv) {
    using C = cplx<R>;
    const NodeDesc d = a.s.desc[lvl_first + blockIdx.x];
    if (d.npiv <= 0) return;
    C *F = reinterpret_cast<C *>(a.front) + (size_t)blockIdx.y * a.s.front_total + d.front_off;
    add_entries(a, d, blockIdx.y);
    __syncthreads();   // the entries are visible to the CTA
    extern __shared__ __align__(16) unsigned char smem_raw[];
    diag_block<R>(a, F, d, blockIdx.y, 0, min(NB, d.npiv), reinterpret_cast<C *>(smem_raw), piv != 0);
}

// K3b: the L and U panels of pivot block k0 as products with the inverted
// triangles of its (already factored) diagonal block: L21 = A21 U11^-1 and
// U12 = L11^-1 A12, one 64-row (L) or 64-column (U) slice per CTA, 256
// threads.  Both are formed with kb rows of output (the L slice as its
// transpose U11^-T A21^T), so all eight warps of the matrix-instruction
// tile layout hold work.  Each CTA reads and writes only its own slice;
// the diagonal block is read-only here.
template <class R>
__global__ void __launch_bounds__(256) k_panel_mm(FactorArgs<R> a, int lvl_first, int k0, int ntmax, int piv) {
    using C = cplx<R>;
    const NodeDesc d = a.s.desc[lvl_first + blockIdx.y];
    const int s = d.npiv;
    if (k0 >= s) return;
    const int f = d.nfront;
    const int kb = min(NB, s - k0);
    const int i0 = k0 + kb;
    const bool upper = blockIdx.x >= (unsigned)ntmax;
    const int x0 = i0 + (upper ? blockIdx.x - ntmax : blockIdx.x) * TILE;   // first row (L) / column (U)
    if (x0 >= f) return;
    const int nx = min(TILE, f - x0);
    C *F = reinterpret_cast<C *>(a.front) + (size_t)blockIdx.z * a.s.front_total + d.front_off;

    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *Is = reinterpret_cast<C *>(smem_raw);   // [NB][TSTR]: Is[k * TSTR + r] = triangle-inverse factor (r, k)
    C *Ps = Is + NB * TSTR;                    // [NB][TSTR]: Ps[k * TSTR + x] = panel entry (k, x)
    const C *Dg = F + k0 + (size_t)k0 * f;    // the inverted diagonal block
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
        const int r = t % NB, k = t / NB;      // Is(r, k): U^-T (r, k) = U^-1 (k, r), or L^-1 (r, k)
        if (r < kb && k < kb) {
            if (upper) {
                if (k < r) cp_async_elem(Is + k * TSTR + r, Dg + r + (size_t)k * f);
                else Is[k * TSTR + r] = k == r ? mk(R(1), R(0)) : czero<C>();
            } else {
                if (k <= r) cp_async_elem(Is + k * TSTR + r, Dg + k + (size_t)r * f);
                else Is[k * TSTR + r] = czero<C>();
            }
        }
    }
    __shared__ unsigned char rsrc[NB];   // U slice: block row of pivot position k (row exchanges)
    if (upper) {
        if (threadIdx.x < NB)
            rsrc[threadIdx.x] = piv && threadIdx.x < kb
                                    ? a.pivsrc[(size_t)blockIdx.z * a.s.n + a.s.vars[d.var_off + k0 + threadIdx.x]]
                                    : (unsigned char)threadIdx.x;
        __syncthreads();
    }
    for (int t = threadIdx.x; t < NB * TILE; t += blockDim.x) {
        if (upper) {   // A12 columns: contiguous along the pivot index; rows in pivot order
            const int x = t / NB, k = t % NB;
            if (k < kb && x < nx) cp_async_elem(Ps + k * TSTR + x, F + (k0 + rsrc[k]) + (size_t)(x0 + x) * f);
        } else {       // A21 rows: contiguous along the row index
            const int x = t % TILE, k = t / TILE;
            if (k < kb && x < nx) cp_async_elem(Ps + k * TSTR + x, F + (x0 + x) + (size_t)(k0 + k) * f);
        }
    }
    staged_sync();
    TileCC<C, sizeof(R) == 8, TILE> acc;
    for_tile(acc, threadIdx.x, [](int, int, C &v) { v = czero<C>(); });
    mma_tile<false>(Is, TSTR, 1, Ps, TSTR, 1, kb, kb, nx, acc, threadIdx.x);
    for_tile(acc, threadIdx.x, [&](int k, int x, C &v) {
        if (k < kb && x < nx) {
            if (upper) F[(k0 + k) + (size_t)(x0 + x) * f] = v;
            else F[(x0 + x) + (size_t)(k0 + k) * f] = v;
        }
    });
}

// acc -= A B over k < K for one TL x TL tile (A: column-major rows 0 .. mrows
// of K columns, B: columns 0 .. ncols of K rows), 256 threads.  K runs in
// chunks of GKC staged through shared memory by asynchronous copies, two
// buffers: the next chunk's loads are in flight while the current one is
// multiplied.  Entries outside mrows and ncols are not staged (they only feed
// accumulators that are never stored).  sm: GEMM_SMEM<TL> complex values.
constexpr int GKC = 16;
template <int TL>
constexpr int GEMM_SMEM = 4 * GKC * (TL + 2);

template <class C, bool MMA, int TL>
__device__ __forceinline__ void gemm_chunks(const C *A, int lda, const C *B, int ldb, int K, int mrows, int ncols,
                                            TileCC<C, MMA, TL> &acc, C *sm) {
    constexpr int SS = TL + 2;   // padded stride of the staged operands
    C *As = sm;                  // [2][GKC][SS]: As[c * SS + r]
    C *Bs = As + 2 * GKC * SS;   // [2][GKC][SS]: Bs[c * SS + col]
    auto stage = [&](int buf, int k0) {
        const int kb = min(GKC, K - k0);
        C *Ab = As + buf * GKC * SS, *Bb = Bs + buf * GKC * SS;
        for (int t = threadIdx.x; t < GKC * TL; t += 256) {
            const int r = t % TL, c = t / TL;
            if (c < kb && r < mrows) cp_async_elem(Ab + c * SS + r, A + (size_t)r + (size_t)(k0 + c) * lda);
            const int col = t / GKC, cc = t % GKC;   // B: contiguous along k
            if (cc < kb && col < ncols) cp_async_elem(Bb + cc * SS + col, B + (size_t)(k0 + cc) + (size_t)col * ldb);
        }
        async_commit();
    };
    const int nk = (K + GKC - 1) / GKC;
    if (nk > 0) stage(0, 0);
    for (int kc = 0; kc < nk; ++kc) {
        async_wait_group<0>();   // chunk kc has landed
        __syncthreads();         // and every warp is past chunk kc - 1
        if (kc + 1 < nk) stage((kc + 1) & 1, (kc + 1) * GKC);
        mma_tile<true>(As + (kc & 1) * GKC * SS, SS, 1, Bs + (kc & 1) * GKC * SS, SS, 1, min(GKC, K - kc * GKC), mrows,
                       ncols, acc, threadIdx.x);
    }
}

// Trailing update C -= L U of the pivots k0 .. k0 + kw - 1 on TL x TL tiles,
// 256 threads, over the trailing rows and columns from k0 + kw on of which one
// at least is a pivot before `lim`.  The contribution block (rows and columns
// >= npiv) receives all pivot steps at once in one K = npiv GEMM at the end of
// the level (launch_contribution), and the pivots from `lim` on their outer
// block's at once: with every 32-pivot step applied to all of them, a front's
// pivot rows and columns went through global memory once per step (64 KB read
// and written per 4.3 us of products in a 64 x 64 tile).  So fronts of many
// pivots take them in outer blocks of kOuter: the inner steps update the outer
// block's own rows and columns, one kw = kOuter step the rest.
// The first CTA takes the next diagonal block alone, updates and factors it
// (it starts first, so this overlaps the tiles); the others take tile
// blockIdx.x - 1 without that block.
//
// Tile size: a 64 x 64 x 32 complex128 product keeps one SM's FP64 pipe busy
// for 4.3 us, a 32 x 32 one for 1.1 us, so where the level's 64-row tiles do
// not fill the chip twice (kTileFill CTAs) the smaller ones shorten the step:
// one 241 x 141 matrix, contribution GEMMs of the top levels 22-39 -> 11-15 us,
// updates without a diagonal block behind them 19 -> 11 us.
// (complex64 keeps one block: its products are short against the steps there.
// 2060 x 1060, one matrix, levels 11-15: 18.9 -> 17.8 ms in blocks of 128, 17.9
// in 64, 18.2 in 256.)
template <class R>
constexpr int kOuter = sizeof(R) == 8 ? 128 : 1 << 20;
static_assert(DIAG_THREADS == 256, "k_update's first CTA factors the next diagonal block");
template <class R, int TL>
__global__ void __launch_bounds__(256) k_update(FactorArgs<R> a, int lvl_first, int k0, int kw, int lim, int ntmax,
                                                int piv) {
    using C = cplx<R>;
    const NodeDesc d = a.s.desc[lvl_first + blockIdx.y];
    if (k0 >= d.npiv) return;
    const int f = d.nfront, s = min(d.npiv, lim);
    const int i0 = min(d.npiv, k0 + kw), m = f - i0;
    const int nt = (m + TL - 1) / TL;
    C *F = reinterpret_cast<C *>(a.front) + (size_t)blockIdx.z * a.s.front_total + d.front_off;
    const bool next = blockIdx.x == 0;   // the next diagonal block
    const int ti = next ? 0 : (blockIdx.x - 1) / ntmax, tj = next ? 0 : (blockIdx.x - 1) % ntmax;
    if (ti >= nt || tj >= nt) return;
    if (i0 + ti * TL >= s && i0 + tj * TL >= s) return;   // no pivot before lim
    const int nd = min(NB, s - i0);                        // size of the next diagonal block
    const bool first = !next && ti == 0 && tj == 0;        // the tile that holds it
    if (first && TL <= NB && nd == NB) return;
    if (next && nd <= 0) return;

    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *sm = reinterpret_cast<C *>(smem_raw);
    const int r0 = i0 + ti * TL, c0 = i0 + tj * TL;
    // a tile whose columns all lie from lim on needs only its rows before it
    // (and the other way round): the product is cut to them
    const int mrows = next ? nd : c0 >= s ? min(TL, s - r0) : min(TL, f - r0);
    const int ncols = next ? nd : r0 >= s ? min(TL, s - c0) : min(TL, f - c0);
    // the tile's current values go into the accumulators while the first
    // operands land (read after the products, their latency was exposed)
    TileCC<C, sizeof(R) == 8, TL> acc;
    auto mine = [&](int rr, int cc) {
        return rr < mrows && cc < ncols && (r0 + rr < s || c0 + cc < s) && !(first && rr < nd && cc < nd);
    };
    for_tile(acc, threadIdx.x, [&](int rr, int cc, C &v) {
        v = mine(rr, cc) ? F[(r0 + rr) + (size_t)(c0 + cc) * f] : czero<C>();
    });
    gemm_chunks(F + r0 + (size_t)k0 * f, f, F + k0 + (size_t)c0 * f, f, i0 - k0, mrows, ncols, acc, sm);
    for_tile(acc, threadIdx.x, [&](int rr, int cc, C &v) {
        if (mine(rr, cc)) F[(r0 + rr) + (size_t)(c0 + cc) * f] = v;
    });
    if (next) {
        __syncthreads();   // the block's global writes are visible; the staged operands are free
        diag_block<R>(a, F, d, blockIdx.z, i0, nd, sm, piv != 0);
    }
}

// Contribution blocks of a level, C = (children's contribution blocks) - L21
// U12 with all of the front's pivots (TL x TL tiles, 256 threads): tiles[t] =
// (level position, tile row, tile column, matrix).  The extend-add of the
// block happens here, into the accumulators: gathered by a kernel of its own
// the block went through global memory twice more (841 x 227, 10 matrices,
// levels 5-8: 4.19 -> 3.73 ms; 2060 x 1060, one matrix, factorisation 37.4 ->
// 35.8 ms).
template <class R, int TL>
__global__ void __launch_bounds__(256, 2) k_contribution(FactorArgs<R> a, int lvl_first, const int4 *__restrict__ tiles) {
    using C = cplx<R>;
    const int4 tl = tiles[blockIdx.x];
    const NodeDesc d = a.s.desc[lvl_first + tl.x];
    const int f = d.nfront, s = d.npiv;
    const int r0 = s + tl.y * TL, c0 = s + tl.z * TL;   // first row / column of the tile
    const int mrows = min(TL, f - r0), ncols = min(TL, f - c0);
    C *base = reinterpret_cast<C *>(a.front) + (size_t)tl.w * a.s.front_total;
    C *F = base + d.front_off;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int map[2][2][TL];   // children's positions of the tile's rows / columns
    for (int t = threadIdx.x; t < 4 * TL; t += 256) {
        const int ch = t / (2 * TL), rc = t / TL % 2, i = t % TL;
        int v = -1;
        if ((ch ? d.child1 : d.child0) >= 0 && i < (rc ? ncols : mrows)) v = a.s.inv[d.inv_off + ch * f + (rc ? c0 : r0) + i];
        map[ch][rc][i] = v;
    }
    __syncthreads();
    const C *cb0 = base + d.cb0, *cb1 = base + d.cb1;
    TileCC<C, sizeof(R) == 8, TL> acc;
    for_tile(acc, threadIdx.x, [&](int rr, int cc, C &v) {
        v = czero<C>();
        const int i0 = map[0][0][rr], j0 = map[0][1][cc], i1 = map[1][0][rr], j1 = map[1][1][cc];
        if (i0 >= 0 && j0 >= 0) v = cb0[i0 + (size_t)j0 * d.ld0];
        if (i1 >= 0 && j1 >= 0) v = cadd(v, cb1[i1 + (size_t)j1 * d.ld1]);
    });
    gemm_chunks(F + r0, f, F + (size_t)c0 * f, f, s, mrows, ncols, acc, reinterpret_cast<C *>(smem_raw));
    for_tile(acc, threadIdx.x, [&](int rr, int cc, C &v) {
        if (rr < mrows && cc < ncols) F[(r0 + rr) + (size_t)(c0 + cc) * f] = v;
    });
}

template <class R, int TL>
static void launch_contribution_tl(const FactorArgs<R> &a, const LevelInfo &L, const int4 *d_tiles, int ntiles,
                                   cudaStream_t st) {
    const size_t smem = GEMM_SMEM<TL> * sizeof(cplx<R>);
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(k_contribution<R, TL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        attr = true;
    }
    (k_contribution<R, TL><<<ntiles, 256, smem, st>>>(a, L.first, d_tiles), note_launch());
}

template <class R>
void launch_contribution(const FactorArgs<R> &a, const LevelInfo &L, const int4 *d_tiles, int ntiles, int tile,
                         cudaStream_t st) {
    if (ntiles <= 0) return;
    if (tile == 32) launch_contribution_tl<R, 32>(a, L, d_tiles, ntiles, st);
    else launch_contribution_tl<R, 64>(a, L, d_tiles, ntiles, st);
}

template void launch_contribution<double>(const FactorArgs<double> &, const LevelInfo &, const int4 *, int, int,
                                          cudaStream_t);
template void launch_contribution<float>(const FactorArgs<float> &, const LevelInfo &, const int4 *, int, int,
                                         cudaStream_t);

// one trailing update of a level's fronts over TL x TL tiles
template <class R, int TL>
static void launch_update_tl(const FactorArgs<R> &a, int first, int count, int mmax, int k0, int kw, int lim, int piv,
                             cudaStream_t st) {
    const size_t smem = std::max<size_t>(GEMM_SMEM<TL>, DIAG_SCRATCH) * sizeof(cplx<R>);
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(k_update<R, TL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        attr = true;
    }
    const int nt = (mmax + TL - 1) / TL;
    (k_update<R, TL><<<dim3(nt * nt + 1, count, a.nf), 256, smem, st>>>(a, first, k0, kw, lim, nt, piv), note_launch());
}
template <class R>
static void launch_update(const FactorArgs<R> &a, const LevelInfo &L, int mmax, int k0, int kw, int lim, int piv,
                          cudaStream_t st) {
    const int64_t nt = (mmax + TILE - 1) / TILE;
    for_level_pieces(L, [&](int first, int count) {
        if (nt * nt * L.count * a.nf < kTileFill) launch_update_tl<R, 32>(a, first, count, mmax, k0, kw, lim, piv, st);
        else launch_update_tl<R, 64>(a, first, count, mmax, k0, kw, lim, piv, st);
    });
}

template <class R>
void launch_factor_level(const FactorArgs<R> &a, const LevelInfo &L, bool whole_gather, cudaStream_t st) {
    using C = cplx<R>;
    if (L.count == 0) return;
    for_level_pieces(L, [&](int first, int count) {
        (k_front_gather<R><<<dim3((L.max_front + GATHER_COLS - 1) / GATHER_COLS, count, a.nf), 32 * GATHER_COLS, 0,
                             st>>>(a, first, !whole_gather),
         note_launch());
    });
    const size_t smem = 2 * NB * TSTR * sizeof(C);
    static bool attr_set = false;
    if (!attr_set) {
        cudaFuncSetAttribute(k_panel_mm<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        attr_set = true;
    }
    const int piv = a.pivsrc && a.pivtau2 > 0;   // row exchanges (every level of this route)
    for_level_pieces(L, [&](int first, int count) {
        (k_diag<R><<<dim3(count, a.nf), DIAG_THREADS, DIAG_SCRATCH * sizeof(C), st>>>(a, first, piv), note_launch());
    });
    for (int k0 = 0; k0 < L.max_piv; k0 += NB) {
        const int mmax = L.max_front - k0 - 1;   // largest trailing size (kb >= 1)
        const int ntmax = mmax > 0 ? (mmax + TILE - 1) / TILE : 0;
        if (ntmax > 0)
            for_level_pieces(L, [&](int first, int count) {
                (k_panel_mm<R><<<dim3(2 * ntmax, count, a.nf), 256, smem, st>>>(a, first, k0, ntmax, piv), note_launch());
            });
        // the trailing tiles only update pivot rows and columns still to
        // come (and factor the next diagonal block): after the level's last
        // pivot block there is nothing left for them
        const int lim = (k0 / kOuter<R> + 1) * kOuter<R>;   // end of the outer block
        if (ntmax > 0 && std::min(L.max_piv, lim) > k0 + NB) launch_update<R>(a, L, mmax, k0, NB, lim, piv, st);
        if (ntmax > 0 && k0 + NB == lim && L.max_piv > lim)
            launch_update<R>(a, L, L.max_front - lim, lim - kOuter<R>, kOuter<R>, L.max_piv, piv, st);
    }
}

template void launch_factor_level<double>(const FactorArgs<double> &, const LevelInfo &, bool, cudaStream_t);
template void launch_factor_level<float>(const FactorArgs<float> &, const LevelInfo &, bool, cudaStream_t);

// ---------------------------------------------------------------------
// Fronts that fit shared memory whole (the lower levels of the tree): one CTA
// assembles and factorises a front -- extend-add of the children's
// contribution blocks, the operator entries, LU of the npiv pivot columns,
// the inverses of both pivot triangles and the Schur complement of the
// contribution block -- and writes it back once, in one launch per level and
// size class instead of the gather / diagonal / panel / update / contribution
// GEMM sequence.  The result has the layout the blocked path leaves.
//
// The front is held in 8 x 8 blocks, the pivots padded to a multiple of 8 by
// decoupled unit pivots: S[i + j ld], pivot k at position k, ring variable i
// at i - npiv + sp.  Per 8-pivot panel q the three steps of
// factor_diag_block, over the whole front:
//   1. one warp factors the panel's pivot rows (a row per lane, up to 32 below
//      the panel's first; row exchanges inside them when PIV);
//   2. a thread per column solves with L_q (b), a thread per row with U_q (a);
//      the ring parts are final (U12 and L21) and stay in S, the pivot parts
//      and the panel's triangle inverses go to Bb and Ab;
//   3. the warps form T - a b on 8 x 8 blocks (FP64 matrix instructions in
//      complex128): the trailing front, the finished rows and columns of the
//      inverses, the panel's own inverse rows and columns.  The panels' warp
//      takes the next one's pivot blocks and goes on with its step 1 beside
//      the others.
// So a front costs three barriers per 8 pivots and the inverses no pass of
// their own.  (Before: one barrier per pivot or two per 4 pivots, then one
// thread per inverse column chaining up to 435 multiply-adds, and from 80 rows
// on the gathered front passed through global memory twice more.  841 x 227,
// 10 matrices, complex128, levels 0-4: 3.87, 0.73, 1.03, 1.47, 1.04 ms then;
// 2.58, 0.57, 0.59, 0.83, 0.92 ms now.  complex64: 2.90, 0.63, 0.67, 0.69,
// 0.93 -> 1.85, 0.38, 0.36, 0.56, 0.73 ms.)
//
// What bounds it: the pivots' latency chain (about 420 cycles each, 3 to 8
// fronts per SM side by side), then the shared-memory traffic of the 8 x 8
// blocks (16-byte elements, 128 B a cycle).  Fronts are launched largest
// first in classes of like size, so a class's shared memory, and with it the
// fronts per SM, follows its own largest front.  (The substitution keeps the
// dissection's order: neighbouring fronts share rows of x in L2.)
// ---------------------------------------------------------------------
constexpr size_t FRONT_SMEM = 226 << 10;   // largest dynamic shared memory of a CTA (1 KB left for static)

__host__ __device__ constexpr int front_sp(int s) { return (s + PW8 - 1) / PW8 * PW8; }
__host__ __device__ constexpr int front_fp(int f, int s) { return f - s + front_sp(s); }
// column stride: whole blocks of rows (zero below the front), odd (conflict-free blocks)
__host__ __device__ constexpr int front_ld(int fp) { return (fp + PW8 - 1) / PW8 * PW8 + 1; }
// elements: S, Ab [8][sp + 2], Bb [sp][12], rd [sp]
static size_t front_words(int fp, int sp) { return (size_t)front_ld(fp) * fp + 8 * (sp + 2) + 12 * (size_t)sp + sp; }

// Right operand of a column of 8 x 8 blocks, held by the warp: B(k, c) =
// pb[k + c bc] for k < 8, c < nc; sub() subtracts A B from this lane's two
// entries of a block (row l / 4, columns 2 (l % 4) + {0, 1}); pa points at the
// lane's part of A (left()), A's pivots being ak apart.
template <class C>
struct BlockCol;
template <>
struct BlockCol<double2> {
    double by[2], nx[2], ny[2];   // b and -b: the matrix instructions take no negated operands
    __device__ __forceinline__ static int left(int ak, int lane) { return (lane >> 2) + (lane & 3) * ak; }
    __device__ __forceinline__ void load(const double2 *pb, int bc, int nc, int lane) {
        const int g = lane >> 2, kq = lane & 3;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const double2 w = g < nc ? pb[4 * h + kq + g * bc] : czero<double2>();
            by[h] = w.y; nx[h] = -w.x; ny[h] = -w.y;
        }
    }
    __device__ __forceinline__ void sub(const double2 *pa, int ak, double2 &a0, double2 &a1) const {
        const double2 v0 = pa[0], v1 = pa[4 * ak];
        dmma_884(v0.x, nx[0], a0.x, a1.x);   // Re -= Ar Br - Ai Bi
        dmma_884(v0.x, ny[0], a0.y, a1.y);   // Im -= Ar Bi + Ai Br
        dmma_884(v0.y, by[0], a0.x, a1.x);
        dmma_884(v0.y, nx[0], a0.y, a1.y);
        dmma_884(v1.x, nx[1], a0.x, a1.x);
        dmma_884(v1.x, ny[1], a0.y, a1.y);
        dmma_884(v1.y, by[1], a0.x, a1.x);
        dmma_884(v1.y, nx[1], a0.y, a1.y);
    }
};
template <>
struct BlockCol<float2> {
    float2 b[2][PW8];
    __device__ __forceinline__ static int left(int, int lane) { return lane >> 2; }
    __device__ __forceinline__ void load(const float2 *pb, int bc, int nc, int lane) {
        const int c = 2 * (lane & 3);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < PW8; ++k) b[h][k] = c + h < nc ? pb[k + (c + h) * bc] : czero<float2>();
    }
    __device__ __forceinline__ void sub(const float2 *pa, int ak, float2 &a0, float2 &a1) const {
#pragma unroll
        for (int k = 0; k < PW8; ++k) {
            const float2 v = pa[k * ak];
            cfms(a0, v, b[0][k]);
            cfms(a1, v, b[1][k]);
        }
    }
};

template <class R, int NTH, bool PIV>
__global__ void __launch_bounds__(NTH, NTH == 128 ? (sizeof(R) == 8 ? 5 : 8) : NTH == 256 ? (sizeof(R) == 8 ? 2 : 3) : 1) k_factor_front(FactorArgs<R> a, int lvl_first) {
    using C = cplx<R>;
    constexpr unsigned ALL = 0xffffffffu;
    constexpr int NW = NTH / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int rowat[PIV ? NB : 1];      // PIV: front row at pivot position k (npiv <= NB)
    __shared__ int pm[NTH == 128 ? 64 : NTH == 256 ? 96 : 128];   // a child's ring positions here
    __shared__ int swaps[PW8 + 1];           // the panel's row exchanges: count, then p | arg << 16
    const NodeDesc d = a.s.fdesc[lvl_first + blockIdx.x];
    const int f = d.nfront, s = d.npiv, sp = front_sp(s), fp = front_fp(f, s), ld = front_ld(fp);
    const int nb = (fp + PW8 - 1) / PW8, npb = sp / PW8;
    C *S = reinterpret_cast<C *>(smem_raw);
    C *Ab = S + (size_t)ld * fp;             // [PW8][sp + 2]: Ab[k * (sp + 2) + r], pivot rows r
    C *Bb = Ab + PW8 * (sp + 2);             // [sp][12]: Bb[c * 12 + k], pivot columns c
    C *rd = Bb + 12 * sp;                    // reciprocal pivots
    const int sa = sp + 2;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // wi 0 factors the panels: another of the CTA's first four warps in every
    // CTA, so that the panels of the fronts on an SM meet all its schedulers
    // (all on the first one they took twice as long)
    const int wi = (warp + NW - ((blockIdx.x + blockIdx.y) & 3)) % NW;
    const size_t fz = blockIdx.y;
    C *base = reinterpret_cast<C *>(a.front) + fz * a.s.front_total;
    C *F = base + d.front_off;

    // the operator entries owned by the front (positions are distinct): the
    // first NE per thread are requested before anything else
    constexpr int NE = NTH == 128 ? 2 : 1;
    const double2 *A = a.A + fz * 9 * (size_t)a.s.n;
    double2 ev[NE];
    int ep[NE];
#pragma unroll
    for (int x = 0; x < NE; ++x) {
        const int e = tid + x * NTH;
        ep[x] = e < d.ent_count ? (int)(a.ent_dst[d.ent_first + e] - d.front_off) : -1;
        ev[x] = ep[x] >= 0 ? A[a.ent_src[d.ent_first + e]] : make_double2(0.0, 0.0);
    }
    auto add_entry = [&](int q, const double2 &v) {
        int i = q % f, j = q / f;
        if (i >= s) i += sp - s;
        if (j >= s) j += sp - s;
        C &t = S[i + j * ld];
        t = cadd(t, cconv<C>(v));
    };
    // extend-add: zeros, then each child's contribution block read once down
    // its columns (GB of them in flight per warp) and added at its rows'
    // positions here (pm: the inverse of the extend-add map)
    constexpr int NR = NTH == 128 ? 2 : NTH == 256 ? 3 : 4;   // rows per lane (launch condition)
    constexpr int GB = NTH == 128 ? 4 : 2;
    {
        const int pad = sp - s;
        for (int t = tid; t < ld * fp; t += NTH) S[t] = czero<C>();
#pragma unroll 1
        for (int ch = 0; ch < 2; ++ch) {
            if ((ch ? d.child1 : d.child0) < 0) continue;   // CTA-uniform
            const int *inv = a.s.inv + d.inv_off + (ch ? f : 0);
            const int ldc = ch ? d.ld1 : d.ld0;
            const C *cb = base + (ch ? d.cb1 : d.cb0);
            for (int i = tid; i < f; i += NTH) {
                const int r = inv[i];
                if (r >= 0) pm[r] = i < s ? i : i + pad;
            }
            const int m = ch ? d.ring1 : d.ring0;   // the child's ring, which lies in this front whole
            __syncthreads();
#pragma unroll 1
            for (int j = warp; j < m; j += GB * NW) {
                C v[GB][NR];
#pragma unroll
                for (int w = 0; w < GB; ++w)
#pragma unroll
                    for (int u = 0; u < NR; ++u) {
                        const int jw = j + w * NW, i = lane + 32 * u;
                        v[w][u] = jw < m && i < m ? cb[i + (size_t)jw * ldc] : czero<C>();
                    }
#pragma unroll
                for (int w = 0; w < GB; ++w)
#pragma unroll
                    for (int u = 0; u < NR; ++u) {
                        const int jw = j + w * NW, i = lane + 32 * u;
                        if (jw < m && i < m) {
                            C &t = S[pm[i] + pm[jw] * ld];
                            t = cadd(t, v[w][u]);
                        }
                    }
            }
            __syncthreads();
        }
        if (PIV && tid < NB) rowat[tid] = tid;
        for (int k = tid; k < sp; k += NTH) rd[k] = mk(R(1), R(0));
        __syncthreads();
        if (tid < pad) S[(s + tid) * (ld + 1)] = mk(R(1), R(0));   // decoupled unit pivots
#pragma unroll
        for (int x = 0; x < NE; ++x)
            if (ep[x] >= 0) add_entry(ep[x], ev[x]);
        for (int e = tid + NE * NTH; e < d.ent_count; e += NTH)
            add_entry((int)(a.ent_dst[d.ent_first + e] - d.front_off), A[a.ent_src[d.ent_first + e]]);
        __syncthreads();
    }

    const R pivtol = (R)(a.pivscale * __longlong_as_double((long long)*a.amax)), tol2 = pivtol * pivtol;
    int np = 0, nsw = 0;   // the panels' warp: the same in every lane
    // 1. the panel at p0 (one warp): lane l holds pivot row p0 + l in registers,
    // x[i] its entry in column p + i
    auto panel = [&](int p0) {
        C *own = S + p0 + lane;
        const bool in = p0 + lane < sp;
        C x[PW8];
#pragma unroll
        for (int i = 0; i < PW8; ++i) x[i] = in ? own[(p0 + i) * ld] : czero<C>();
        int nx = 0;
        const int pw = min(PW8, s - p0);
#pragma unroll 1
        for (int j = 0; j < pw; ++j) {
            const int p = p0 + j;
            C piv = mk(__shfl_sync(ALL, x[0].x, j), __shfl_sync(ALL, x[0].y, j));
            C rp = crcp(piv);
            if (PIV) {
                const R m2 = cabs2(x[0]);
                const int key = lane >= j && p0 + lane < s ? lead_bits(m2) : -1;
                const int arg = exchange_lane(a, m2, key, cabs2(piv));
                if (arg > j) {   // rows p and p0 + arg trade places: the panel's columns here, the others in step 2
                    __syncwarp();   // the multipliers that other lanes stored (shuffles order no memory)
                    const int from = lane == j ? arg : lane == arg ? j : lane;
#pragma unroll
                    for (int i = 0; i < PW8; ++i)
                        x[i] = mk(__shfl_sync(ALL, x[i].x, from), __shfl_sync(ALL, x[i].y, from));
                    piv = mk(__shfl_sync(ALL, x[0].x, j), __shfl_sync(ALL, x[0].y, j));
                    if (lane < j) {   // the multipliers stored so far
                        C *c = S + (p0 + lane) * ld;
                        const C t = c[p];
                        c[p] = c[p0 + arg];
                        c[p0 + arg] = t;
                    }
                    if (lane == 0) {
                        const int t = rowat[p];
                        rowat[p] = rowat[p0 + arg];
                        rowat[p0 + arg] = t;
                        swaps[1 + nx] = p | (p0 + arg) << 16;
                    }
                    __syncwarp();
                    ++nx;
                    rp = crcp(piv);
                }
            }
            if (!(cabs2(piv) >= tol2) || !(tol2 > R(0))) {   // rare, off the chain: rp is formed already
                piv = static_pivot<R>(piv, pivtol, np);
                rp = crcp(piv);
            }
            const C l = lane > j ? cmul(x[0], rp) : czero<C>();   // rows p and above are final
            if (in) own[p * ld] = lane > j ? l : lane == j ? piv : x[0];
            if (lane == j) rd[p] = rp;
#pragma unroll
            for (int i = 1; i < PW8; ++i) {   // less the pivot row's entry, from its lane
                const C v = mk(__shfl_sync(ALL, x[i].x, j), __shfl_sync(ALL, x[i].y, j));
                cfms(x[i], l, v);
                x[i - 1] = x[i];
            }
            x[PW8 - 1] = czero<C>();
        }
        if (PIV && lane == 0) swaps[0] = nx;
        nsw += nx;
    };
    // 3. blocks bi0 .. bi1 - 1 of block column bj in step q: T - a b, or its
    // special forms on the panel's row and column and the finished parts of
    // the inverses
    const int g = lane >> 2, kq = lane & 3;
    auto column = [&](int q, int bj, int bi0, int bi1) {
        const bool rj = bj >= npb;   // ring columns
        if (rj) bi0 = max(bi0, q + 1);                  // (U12 above is final)
        else if (bj < q) bi0 = max(bi0, q), bi1 = min(bi1, npb);
        else if (bj == q) bi1 = min(bi1, npb);          // (L21 is final)
        if (bi0 >= bi1) return;
        const int c = 8 * bj + 2 * kq, nc = fp - 8 * bj;
        const bool in0 = c < fp, in1 = c + 1 < fp;
        BlockCol<C> b;
        b.load(rj ? S + q * PW8 + 8 * bj * ld : Bb + 8 * bj * 12, rj ? ld : 12, nc, lane);
        const C *paA = Ab + BlockCol<C>::left(sa, lane), *paS = S + q * PW8 * ld + BlockCol<C>::left(ld, lane);
        C *t = S + 8 * bi0 + g + c * ld;
#pragma unroll 1
        for (int bi = bi0; bi < bi1; ++bi, t += PW8) {
            C a0 = czero<C>(), a1 = czero<C>();
            if (bi <= q && bj <= q) {   // X's row q, L_q^-1; Z's column q, U_q^-1 (bi == q or bj == q)
                const bool x0 = bi == q && (bj < q || g > 2 * kq), x1 = bi == q && (bj < q || g > 2 * kq + 1);
                a0 = x0 ? Bb[c * 12 + g] : Ab[2 * kq * sa + 8 * bi + g];
                a1 = x1 ? Bb[(c + 1) * 12 + g] : Ab[(2 * kq + 1) * sa + 8 * bi + g];
            } else {
                if (bi != q && bj != q) {
                    if (in0) a0 = t[0];
                    if (in1) a1 = t[ld];
                }
                const bool ri = bi >= npb;
                b.sub((ri ? paS : paA) + 8 * bi, ri ? ld : sa, a0, a1);
            }
            if (in0) t[0] = a0;
            if (in1) t[ld] = a1;
        }
    };

    // q = -1: the first panel alone
    const int nseg = 1 + (nb - npb + 3) / 4;   // pieces of a block column: its pivot rows, four blocks of ring rows each
#pragma unroll 1
    for (int q = npb > 0 ? -1 : 0; q < npb; ++q) {
        const int p0 = q * PW8, p1 = p0 + PW8;
        if (q >= 0) {
            __syncthreads();
            // 2. a and b (the panel's own rows and columns take the identity)
            const C *Tq = S + p0 + p0 * ld;
            constexpr int HALF = NTH / 2;
            if (tid < HALF) {
                for (int r = tid; r < fp; r += HALF) {
                    C v[PW8];
                    const int ql = r - p0;
#pragma unroll
                    for (int j = 0; j < PW8; ++j)
                        v[j] = ql >= 0 && ql < PW8 ? mk(R(j == ql), R(0)) : S[r + (p0 + j) * ld];
                    if (!(r >= p1 && r < min(sp, p0 + 32))) {   // (the panel's lanes hold their multipliers already)
#pragma unroll
                        for (int i = 0; i < PW8; ++i) {
                            v[i] = cmul(v[i], rd[p0 + i]);
#pragma unroll
                            for (int j = i + 1; j < PW8; ++j) cfms(v[j], v[i], Tq[i + j * ld]);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < PW8; ++j) {
                        if (r < sp) Ab[j * sa + r] = v[j];
                        else S[r + (p0 + j) * ld] = v[j];
                    }
                }
            } else {
                const int nx = PIV ? swaps[0] : 0;
                for (int c = tid - HALF; c < fp; c += HALF) {
                    C v[PW8];
                    const int ql = c - p0;
                    const bool mid = ql >= 0 && ql < PW8;
                    C *col = S + c * ld;
                    if (PIV && !mid)
                        for (int x = 0; x < nx; ++x) {
                            const int w = swaps[1 + x], u = w & 0xffff, z = w >> 16;
                            const C t = col[u];
                            col[u] = col[z];
                            col[z] = t;
                        }
#pragma unroll
                    for (int j = 0; j < PW8; ++j) v[j] = mid ? mk(R(j == ql), R(0)) : col[p0 + j];
#pragma unroll
                    for (int i = 0; i + 1 < PW8; ++i)
#pragma unroll
                        for (int j = i + 1; j < PW8; ++j) cfms(v[j], Tq[j + i * ld], v[i]);
#pragma unroll
                    for (int j = 0; j < PW8; ++j) {
                        if (c < sp) Bb[c * 12 + j] = v[j];
                        else col[p0 + j] = v[j];
                    }
                }
            }
            __syncthreads();
        }
        const bool more = q + 1 < npb, ahead = more && wi == 0;   // one warp goes on with the next panel
        if (q >= 0) {
            const int e1 = ahead ? 0 : nb * nseg, step = ahead ? 1 : more ? NW - 1 : NW;
#pragma unroll 1
            for (int e = ahead ? -1 : more ? wi - 1 : wi; e < e1; e += step) {
                int bj = q + 1, b0 = q + 1, b1 = npb;   // ahead: the next panel's pivot blocks
                if (!ahead) {
                    const int seg = e % nseg;
                    bj = nb - 1 - e / nseg;
                    b0 = seg ? npb + 4 * (seg - 1) : 0;
                    b1 = seg ? min(nb, b0 + 4) : more && bj == q + 1 ? q + 1 : npb;
                }
                column(q, bj, b0, b1);
            }
        }
        if (ahead) {
            __syncwarp();
            panel(p1);
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int j = warp; j < f; j += GB * NW) {
        C v[GB][NR];
#pragma unroll
        for (int w = 0; w < GB; ++w)
#pragma unroll
            for (int u = 0; u < NR; ++u) {
                const int jw = j + w * NW, i = lane + 32 * u;
                if (jw < f && i < f) v[w][u] = S[(i < s ? i : i + sp - s) + (jw < s ? jw : jw + sp - s) * ld];
            }
#pragma unroll
        for (int w = 0; w < GB; ++w)
#pragma unroll
            for (int u = 0; u < NR; ++u) {
                const int jw = j + w * NW, i = lane + 32 * u;
                if (jw < f && i < f) F[i + (size_t)jw * f] = v[w][u];
            }
    }
    if (PIV && tid < s) a.pivsrc[fz * (size_t)a.s.n + a.s.vars[d.var_off + tid]] = (unsigned char)rowat[tid];
    if (wi == 0 && lane == 0) {
        if (np) atomicAdd(a.npert, (unsigned long long)np);
        if (PIV && nsw) atomicAdd(a.nswap, (unsigned long long)nsw);
    }
}

// Levels whose fronts take static pivots: those of at most 100 KB.  (The
// larger fronts' levels exchange rows; the line is the one the exchanges were
// measured with: with them on the levels above it the direct solves' worst
// residual on the 841 x 227 operators fell from 3.1e-11 to 1.5e-11, on the
// lower levels a replay finds nothing more to gain.)
template <class R>
static bool static_pivot_level(const LevelInfo &L) {
    const int f = L.max_front;
    return L.count > 0 && f <= 128 && ((size_t)(f + 1) * f + f) * sizeof(cplx<R>) <= (size_t)100 << 10;
}

// Row exchanges happen on every other level
template <class R>
bool level_pivots(const LevelInfo &L) {
    return L.count > 0 && !static_pivot_level<R>(L);
}
template bool level_pivots<double>(const LevelInfo &);
template bool level_pivots<float>(const LevelInfo &);

template <class R>
bool front_factor_level(const LevelInfo &L) {
    return L.count > 0 && (size_t)L.front_words * sizeof(cplx<R>) <= FRONT_SMEM &&
           L.max_front + PW8 - 1 <= 128 && (L.max_piv <= NB || static_pivot_level<R>(L));
}

// Size classes of a level whose nodes are ordered by front size, largest
// first: a class is closed where the next front's shared memory lets more
// fronts share an SM, once it holds kMinClass fronts.
constexpr int kMinClass = 1024;
std::vector<FrontClass> front_classes(const NodeDesc *desc, int count, size_t csize) {
    std::vector<FrontClass> out;
    auto fit = [](size_t bytes) { return (int)std::min<size_t>(16, (FRONT_SMEM + 1024) / (bytes + 1024)); };
    for (int t = 0; t < count; ++t) {
        const int f = desc[t].nfront, s = desc[t].npiv;
        const size_t bytes = front_words(front_fp(f, s), front_sp(s)) * csize;
        if (out.empty() || (out.back().count >= kMinClass && fit(bytes) > fit(out.back().smem)))
            out.push_back(FrontClass{t, 0, 0, 0});
        FrontClass &c = out.back();
        ++c.count;
        c.max_rows = std::max(c.max_rows, front_ld(front_fp(f, s)) - 1);
        c.smem = std::max(c.smem, bytes);
    }
    return out;
}

template <class R, int NTH, bool PIV>
static void launch_front_class(const FactorArgs<R> &a, const LevelInfo &L, const FrontClass &c, cudaStream_t st) {
    static bool attr_set = false;
    if (!attr_set) {
        cudaFuncSetAttribute(k_factor_front<R, NTH, PIV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FRONT_SMEM);
        attr_set = true;
    }
    (k_factor_front<R, NTH, PIV><<<dim3(c.count, a.nf), NTH, c.smem, st>>>(a, L.first + c.first), note_launch());
}

// Threads per front: 128 up to 64 rows (several fronts per SM hide each
// other's chains), 256 up to 96 and 512 up to 128, where one or two fronts
// fill the SM.
template <class R>
void launch_factor_front(const FactorArgs<R> &a, const LevelInfo &L, cudaStream_t st) {
    const bool piv = level_pivots<R>(L) && a.pivsrc && a.pivtau2 > 0;
    for (const FrontClass &c : L.classes) {
        if (piv) {
            if (c.max_rows <= 64) launch_front_class<R, 128, true>(a, L, c, st);
            else if (c.max_rows <= 96) launch_front_class<R, 256, true>(a, L, c, st);
            else launch_front_class<R, 512, true>(a, L, c, st);
        } else {
            if (c.max_rows <= 64) launch_front_class<R, 128, false>(a, L, c, st);
            else if (c.max_rows <= 96) launch_front_class<R, 256, false>(a, L, c, st);
            else launch_front_class<R, 512, false>(a, L, c, st);
        }
    }
}

template bool front_factor_level<double>(const LevelInfo &);
template bool front_factor_level<float>(const LevelInfo &);
template void launch_factor_front<double>(const FactorArgs<double> &, const LevelInfo &, cudaStream_t);
template void launch_factor_front<float>(const FactorArgs<float> &, const LevelInfo &, cudaStream_t);
int64_t front_words_of(int f, int s) { return (int64_t)front_words(front_fp(f, s), front_sp(s)); }

// Grid-stride max of |A| with one atomicMax per warp.  Non-negative doubles
// order like their bit patterns read as unsigned integers.
__global__ void __launch_bounds__(256) k_amax(const double2 *A, size_t cnt, unsigned long long *out) {
    double m = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += (size_t)gridDim.x * blockDim.x) {
        const double2 v = A[i];
        const double a = hypot(v.x, v.y);
        m = (a > m || a != a) ? a : m;   // a NaN entry makes the maximum NaN (reported by the host)
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double q = __shfl_xor_sync(0xffffffffu, m, o);
        m = (q > m || q != q) ? q : m;
    }
    if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

void launch_amax(const double2 *A, size_t cnt, unsigned long long *out, cudaStream_t st) {
    note_launch();
    k_amax<<<148 * 8, 256, 0, st>>>(A, cnt, out);
}

__global__ void k_pack_split(double2 *dst, const double *re, const double *im, size_t cnt) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = make_double2(re[i], im[i]);
}

void launch_pack_split(double2 *dst, const double *re, const double *im, size_t cnt, cudaStream_t st) {
    note_launch();
    k_pack_split<<<148 * 8, 256, 0, st>>>(dst, re, im, cnt);
}

}  // namespace gm


namespace gm {

// ---------------------------------------------------------------------
// Mid-level fronts: at most NB pivots and at most MID_FT rows, but too
// large for the whole-front kernel.  Taken on request only (GM_MID_MAX_PIV,
// engine.cpp).  After the extend-add
// gather and the operator entries (K2), one CTA per front and frequency
//   1. factorises the pivot columns (f x s) right-looking with each thread
//      holding one front row in registers: per pivot, warp 0 picks the
//      pivot row by the threshold rule (mid_select_pivot: rows keep their
//      threads and trade pivot positions), and the row's owner replaces a
//      pivot that stays tiny as static_pivot does and publishes the row and
//      the pivot's reciprocal in shared memory: one barrier per pivot, and
//      no shared-memory traffic for the update itself;
//   2. solves L11 U12 = P A12 with each thread holding one column of U12;
//   3. inverts the pivot block's two triangles;
//   4. writes L, U and the inverses back (the layout the blocked path
//      leaves);
//   5. applies the rank-s Schur update to the contribution block,
//      64 x 64 tiles of 4 x 4 complex per thread, each tile's old values
//      loaded into the accumulators first.
// This replaces the K3 / K4 steps and the level's contribution GEMM.
// Shared memory: P[i + c * (f + 1)] the pivot columns, then
// U[r + j * (s | 1)] the U12 rows (odd strides: conflict-free 16-byte
// accesses).
// ---------------------------------------------------------------------
constexpr int MID_FT = 256;   // threads per CTA, also the largest front handled

// Warp 0 of k_factor_mid (which holds every pivot row): pivot position kp
// goes to the row of largest |x[kp]| among the rows at positions >= kp when
// the row there has |x[kp]|^2 < tau2 times that (c2: this lane's
// |x[kp]|^2, pos: the pivot position of this lane's row; the two rows swap
// positions).  Only scalars: the caller's row stays in registers.
template <class R>
__device__ __forceinline__ void mid_select_pivot(R c2, int &pos, int kp, int s, R tau2, int &nsw) {
    const int lane = threadIdx.x & 31;
    R m2 = pos >= kp && pos < s ? c2 : R(-1);
    int arg = lane;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const R om = __shfl_xor_sync(0xffffffffu, m2, o);
        const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
        if (om > m2 || (om == m2 && oa < arg)) {
            m2 = om;
            arg = oa;
        }
    }
    m2 = __shfl_sync(0xffffffffu, m2, 0);     // lane 0's result for all (NaN entries
    arg = __shfl_sync(0xffffffffu, arg, 0);   // could leave the lanes disagreeing)
    const int cur = __ffs(__ballot_sync(0xffffffffu, pos == kp)) - 1;   // the lane at position kp
    const R d2 = __shfl_sync(0xffffffffu, c2, cur);
    if (arg != cur && d2 < tau2 * m2) {   // warp-uniform
        const int pa = __shfl_sync(0xffffffffu, pos, arg);
        if (lane == cur) pos = pa;
        if (lane == arg) pos = kp;
        ++nsw;
    }
}

template <class R>
__global__ void __launch_bounds__(MID_FT) k_factor_mid(FactorArgs<R> a, int lvl_first) {
    using C = cplx<R>;
    constexpr int NPR = NB;   // entries of a pivot row in registers
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ C Dinv[NB][NB + 1];
    __shared__ C urow[2][NPR];   // pivot row k at columns k .. s-1, alternating buffers
    __shared__ C rd[NPR];        // reciprocal pivots
    __shared__ int perm[NB];     // front row at pivot position q (row exchanges)
    __shared__ int npert;
    const NodeDesc d = a.s.desc[lvl_first + blockIdx.x];
    const int f = d.nfront, s = d.npiv, m = f - s;
    if (s == 0) return;   // the gathered front is already the contribution block
    add_entries(a, d, blockIdx.y);
    __syncthreads();   // the entries are visible to the CTA
    const int ldp = f + 1, ldu = s | 1;
    C *P = reinterpret_cast<C *>(smem_raw);
    C *U = P + (size_t)ldp * s;
    const int tid = threadIdx.x;
    C *F = reinterpret_cast<C *>(a.front) + (size_t)blockIdx.y * a.s.front_total + d.front_off;
    const R pivtol = (R)(a.pivscale * __longlong_as_double((long long)*a.amax));
    if (tid == 0) npert = 0;

    for (int t = tid; t < s * m; t += MID_FT) {   // A12, down each column, landing during step 1
        const int j = t / s, r = t - j * s;
        cp_async_elem(U + r + j * ldu, F + r + (size_t)(s + j) * f);
    }

    // 1. pivot columns, one row per thread.  Iteration k applies pivot k
    // and publishes pivot k + 1: the row at pivot position k + 1 and the
    // reciprocal.  Rows stay with their threads; pos is the pivot position
    // of the thread's row (its own index but for exchanged pivot rows).
    // With row exchanges (piv), warp 0 -- which holds every pivot row,
    // s <= 32 -- first gives position k + 1 to the row r of largest
    // |x_r[k+1]| among those at positions > k when the row there has
    // |x[k+1]|^2 < pivtau2 |x_r[k+1]|^2 (the two rows swap positions); the
    // rows go to shared memory at their positions afterwards.
    const bool own = tid < f;
    const bool piv = a.pivsrc != nullptr && a.pivtau2 > 0;
    C x[NPR];
#pragma unroll
    for (int j = 0; j < NPR; ++j) x[j] = (own && j < s) ? F[tid + (size_t)j * f] : czero<C>();
    int np = 0, nsw = 0, pos = tid;
    if (piv && tid < 32) mid_select_pivot<R>(cabs2(x[0]), pos, 0, s, (R)a.pivtau2, nsw);
    if (pos == 0) {
        x[0] = static_pivot<R>(x[0], pivtol, np);
        rd[0] = crcp(x[0]);
#pragma unroll
        for (int j = 0; j < NPR; ++j)
            if (j < s) urow[0][j] = x[j];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NPR; ++k) {
        if (k >= s) continue;   // s is the same for the whole CTA
        if (own && pos > k) {
            const C l = cmul(x[k], rd[k]);
            x[k] = l;
#pragma unroll
            for (int j = k + 1; j < NPR; ++j)
                if (j < s) cfms(x[j], l, urow[k & 1][j]);
        }
        const int k1 = k + 1 < NPR ? k + 1 : NPR - 1;   // pivot published by this iteration
        if (k + 1 < NPR && k + 1 < s) {
            if (piv && tid < 32) mid_select_pivot<R>(cabs2(x[k1]), pos, k1, s, (R)a.pivtau2, nsw);
            if (pos == k1 && own) {   // the row at the next pivot position
                x[k1] = static_pivot<R>(x[k1], pivtol, np);
                rd[k1] = crcp(x[k1]);
#pragma unroll
                for (int j = k1; j < NPR; ++j)
                    if (j < s) urow[k1 & 1][j] = x[j];
            }
        }
        __syncthreads();
    }
    if (own) {
#pragma unroll
        for (int j = 0; j < NPR; ++j)
            if (j < s) P[pos + j * ldp] = x[j];
        if (pos < s) perm[pos] = tid;
    }
    if (np) atomicAdd(&npert, np);
    if (tid == 0 && nsw) atomicAdd(a.nswap, (unsigned long long)nsw);
    staged_sync();
    if (piv && tid < s) a.pivsrc[(size_t)blockIdx.y * a.s.n + a.s.vars[d.var_off + tid]] = (unsigned char)perm[tid];

    // 2. U12 = L11^-1 A12, one column per thread of warps 2 .. 7, while
    // warps 0 and 1 invert the pivot block's triangles (3.)
    for (int j = tid - 64; j >= 0 && j < m; j += MID_FT - 64) {
        C u[NPR];   // A12's rows in pivot order
#pragma unroll
        for (int r = 0; r < NPR; ++r) u[r] = r < s ? U[(piv ? perm[r] : r) + j * ldu] : czero<C>();
#pragma unroll
        for (int k = 0; k + 1 < NPR; ++k) {
            if (k + 1 < s) {
                const C uk = u[k];
#pragma unroll
                for (int r = k + 1; r < NPR; ++r)
                    if (r < s) cfms(u[r], P[r + k * ldp], uk);
            }
        }
#pragma unroll
        for (int r = 0; r < NPR; ++r)
            if (r < s) U[r + j * ldu] = u[r];
    }

    // 3. inverses of the pivot block's triangles: L^-1 strictly below the
    // diagonal (unit diagonal implied), U^-1 on and above it
    if (tid < s) {
        const int c = tid;
        for (int r = c + 1; r < s; ++r) {
            C acc = P[r + c * ldp];
            for (int q = c + 1; q < r; ++q) cfma(acc, P[r + q * ldp], Dinv[q][c]);
            Dinv[r][c] = mk(-acc.x, -acc.y);
        }
    } else if (tid >= 32 && tid < 32 + s) {
        const int c = tid - 32;
        Dinv[c][c] = rd[c];
        for (int r = c - 1; r >= 0; --r) {
            C acc = czero<C>();
            for (int q = r + 1; q <= c; ++q) cfma(acc, P[r + q * ldp], Dinv[q][c]);
            Dinv[r][c] = cmul(mk(-acc.x, -acc.y), rd[r]);
        }
    }
    __syncthreads();

    // 4. write back: pivot columns (inverses in the pivot block), U12
    for (int t = tid; t < f * s; t += MID_FT) {
        const int c = t / f, i = t - c * f;
        F[t] = i < s ? Dinv[i][c] : P[i + c * ldp];
    }
    for (int t = tid; t < s * m; t += MID_FT) {
        const int j = t / s, r = t - j * s;
        F[r + (size_t)(s + j) * f] = U[r + j * ldu];
    }
    if (tid == 0 && npert) atomicAdd(a.npert, (unsigned long long)npert);

    // 5. contribution block -= L21 U12, 64 x 64 tiles, each tile's old
    // values loaded into the accumulators first
    for (int i0 = 0; i0 < m; i0 += 64)
        for (int j0 = 0; j0 < m; j0 += 64) {
            TileCC<C, sizeof(R) == 8, 64> acc;
            for_tile(acc, tid, [&](int rr, int cc, C &v) {
                const int i = i0 + rr, j = j0 + cc;
                v = (i < m && j < m) ? F[s + i + (size_t)(s + j) * f] : czero<C>();
            });
            mma_tile<true>(P + s + i0, ldp, 1, U + (size_t)j0 * ldu, 1, ldu, s, min(64, m - i0), min(64, m - j0), acc,
                        tid);
            for_tile(acc, tid, [&](int rr, int cc, C &v) {
                const int i = i0 + rr, j = j0 + cc;
                if (i < m && j < m) F[s + i + (size_t)(s + j) * f] = v;
            });
        }
}

constexpr size_t MID_FACTOR_SMEM = 200 << 10;

template <class R>
bool mid_factor_level(const LevelInfo &L) {
    return L.count > 0 && L.max_piv <= NB && L.max_front <= MID_FT &&
           (size_t)L.mid_words * sizeof(cplx<R>) <= MID_FACTOR_SMEM;
}

template <class R>
static void launch_mid(const FactorArgs<R> &a, const LevelInfo &L, cudaStream_t st) {
    static bool attr_set = false;
    if (!attr_set) {
        cudaFuncSetAttribute(k_factor_mid<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MID_FACTOR_SMEM);
        attr_set = true;
    }
    (k_factor_mid<R><<<dim3(L.count, a.nf), MID_FT, (size_t)L.mid_words * sizeof(cplx<R>), st>>>(a, L.first),
     note_launch());
}

template <class R>
void launch_factor_mid(const FactorArgs<R> &a, const LevelInfo &L, cudaStream_t st) {
    for_level_pieces(L, [&](int first, int count) {
        (k_front_gather<R><<<dim3((L.max_front + GATHER_COLS - 1) / GATHER_COLS, count, a.nf), 32 * GATHER_COLS, 0,
                             st>>>(a, first, 0),
         note_launch());
    });
    launch_mid<R>(a, L, st);
}

template bool mid_factor_level<double>(const LevelInfo &);
template bool mid_factor_level<float>(const LevelInfo &);
template void launch_factor_mid<double>(const FactorArgs<double> &, const LevelInfo &, cudaStream_t);
template void launch_factor_mid<float>(const FactorArgs<float> &, const LevelInfo &, cudaStream_t);

}  // namespace gm
