// K5: multi-right-hand-side forward/backward substitution through the
// multifrontal factors (the replacement of one umfpack_zi_solve call per
// shot, src/AC/forward_shot_AC.c:88, by one block solve over every shot of
// every frequency).
//
// Right-hand sides / solutions are [nf][n][ldr] complex, right-hand side
// fastest.  Work units are (front, frequency, slice of 32 or 40 right-hand
// sides).  The factorisation stores the inverse of every pivot triangle (of
// the 32 x 32 diagonal block of the fronts with at most 32 pivots, of the
// whole triangle above that, tri.cu), so every step below is a small GEMM:
// 128 threads fill an RT-row x 8B-right-hand-side output tile, operands
// staged in shared memory (solve_tile.cuh).
//
// x holds the right-hand side, then the solution; the workspace w holds each
// front's update vector for its parent (its ring rows).  Per
// elimination-tree level, fronts of at most 32 pivots take one fused kernel
// per pass (k_fwd_small, k_bwd_small), the others
//   forward  (leaves -> root)
//     k_fwd_rhs   the children's update vectors added into x at the pivots;
//     k_fwd_tri   y = L^-1 x_piv into the pivot workspace, 32-row tiles;
//     k_fwd_ring  w_ring = (children's update vectors at the ring rows)
//                 - L_ring,piv * y over RT-row tiles of the ring;
//   backward (root -> leaves)
//     k_bwd_ring  t = y - U_piv,ring * x_ring (x_ring = final values of the
//                 ancestors' variables) in the pivot workspace;
//     k_bwd_tri   x_piv = U^-1 t, 32-row tiles.
// trans = 1 solves M^T x = b with the same factors: M^T = U^T L^T, the
// forward pass runs with U^T and the backward pass with L^T; only the
// factor indexing and which stored inverse is used change.
#include <algorithm>
#include <cstdlib>

#include "solve_tile.cuh"

namespace gm {

// false when right-hand sides r0 .. r0 + rn - 1 are zero throughout node v's
// subtree (forward-pass pruning mask; no mask: always true)
template <class R>
__device__ __forceinline__ bool live(const SolveArgs<R> &a, int v, int r0, int rn) {
    if (!a.mask) return true;
    const unsigned char *m = a.mask + (size_t)v * a.mask_nch;
    for (int g = r0 >> 5; g <= (r0 + rn - 1) >> 5; ++g)
        if (m[g]) return true;
    return false;
}

// false when right-hand side `col` is zero throughout node v's subtree
template <class R>
__device__ __forceinline__ bool col_live(const SolveArgs<R> &a, int v, int col) {
    return !a.mask || a.mask[(size_t)v * a.mask_nch + (col >> 5)];
}

// The columns r of a slice in which child v's update vector was formed.  The
// small-front levels form 32-column slices, pruned one by one; a wider slice
// of a level above can cover a live and a pruned one, whose columns hold
// what an earlier solve left there.
template <int TC>
struct LiveCols {
    static_assert(TC <= 40, "a slice meets at most two 32-column groups");
    int lo = 0, n = TC;
    template <class R>
    __device__ __forceinline__ LiveCols(const SolveArgs<R> &a, int v, int r0, int rn) {
        if (TC % 32 == 0 || v < 0 || !a.mask || (r0 & 31) + rn <= 32) return;
        const unsigned char *m = a.mask + (size_t)v * a.mask_nch + (r0 >> 5);
        const int cut = 32 - (r0 & 31);
        lo = m[0] ? 0 : cut;
        n = (m[1] ? rn : cut) - lo;
    }
    __device__ __forceinline__ bool has(int r) const { return TC % 32 == 0 || (unsigned)(r - lo) < (unsigned)n; }
};

// matrix handled by this CTA: blockIdx.z indexes the launch's matrix list
template <class R>
__device__ __forceinline__ size_t solve_matrix(const SolveArgs<R> &a) {
    return a.fmap ? (size_t)a.fmap[blockIdx.z] : (size_t)blockIdx.z;
}
// slot of x and of the workspace w used by this CTA
template <class R>
__device__ __forceinline__ size_t solve_slot(const SolveArgs<R> &a) {
    return a.xmap ? (size_t)a.xmap[blockIdx.z] : solve_matrix(a);
}

template <class R>
struct Ctx {
    using C = cplx<R>;
    int node, f, s, rn;
    const C *F;
    const int *vars;
    C *X;   // this slice of x; pivot rows are solved in place here
    C *W;   // this node's update vector: ring row i (front position s + i)
};

template <class R, int TC>
__device__ __forceinline__ Ctx<R> make_ctx(const SolveArgs<R> &a, int lvl_first, int chunk, int pos = -1,
                                           const NodeDesc *desc = nullptr) {
    using C = cplx<R>;
    Ctx<R> c;
    const NodeDesc d = (desc ? desc : a.s.desc)[lvl_first + (pos < 0 ? (int)blockIdx.y : pos)];
    c.node = d.node;
    c.f = d.nfront;
    c.s = d.npiv;
    const int r0 = chunk * TC;
    c.rn = min(TC, a.nrhs - r0);
    const size_t fz = solve_matrix(a), xz = solve_slot(a);
    c.F = reinterpret_cast<const C *>(a.front) + fz * a.s.front_total + d.front_off;
    c.vars = a.s.vars + d.var_off;
    c.X = reinterpret_cast<C *>(a.x) + xz * (size_t)a.s.n * a.ldr + r0;
    c.W = reinterpret_cast<C *>(a.w) + xz * (size_t)a.s.rhs_total * a.ldr + r0 + (size_t)d.rhs_off * a.ldr;
    return c;
}

// Right-hand sides that x does not hold (implicit spikes, or the caller's FP64
// b): the entry of a row and column of this slice.  Copied into x first, b
// went through memory twice more, and in complex64 the spikes were written,
// converted and the solution added to a cleared x (841 x 227, 100 right-hand
// sides: 10 matrices in complex64 63.0 -> 60.7 ms a call, the gradient of 3
// matrices, dense adjoint sources in FP64, 13.4 -> 13.0 ms).
template <class R>
struct OuterRhs {
    using C = cplx<R>;
    const int *spike_k;
    const double2 *b;
    C amp;
    __device__ __forceinline__ OuterRhs(const SolveArgs<R> &a, int r0) {
        const size_t f = solve_matrix(a);
        spike_k = a.spike_k ? a.spike_k + r0 : nullptr;
        b = a.b ? a.b + f * (size_t)a.s.n * a.ldr + r0 : nullptr;
        amp = spike_k ? cconv<C>(a.spike_amp[f]) : czero<C>();
    }
    __device__ __forceinline__ bool given() const { return spike_k || b; }
    __device__ __forceinline__ C at(int row, int r, size_t ldr) const {
        if (b) return cconv<C>(b[(size_t)row * ldr + r]);
        return spike_k[r] == row ? amp : czero<C>();
    }
};

// The pivot rows of this front's slice of x receive the children's update
// vectors (W0, W1: NULL for a child that is absent or pruned); where x does
// not hold the right-hand sides they become b + the updates, x not being read
// (it is not cleared before the solve).
template <class R>
__device__ __forceinline__ void pivot_rhs(const SolveArgs<R> &a, const Ctx<R> &c, const int *inv, const cplx<R> *W0,
                                          const cplx<R> *W1, int r0, size_t ldr) {
    using C = cplx<R>;
    const OuterRhs<R> outer(a, r0);
    if (!(W0 || W1 || outer.given())) return;   // CTA-uniform
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = warp; i < c.s; i += NT / 32) {
        const int q0 = W0 ? inv[i] : -1, q1 = W1 ? inv[c.f + i] : -1;
        if (!outer.given() && q0 < 0 && q1 < 0) continue;
        const int row = c.vars[i];
        for (int r = lane; r < c.rn; r += 32) {
            C v = czero<C>();
            if (q0 >= 0) v = cadd(v, W0[(size_t)q0 * ldr + r]);
            if (q1 >= 0) v = cadd(v, W1[(size_t)q1 * ldr + r]);
            C &x = c.X[(size_t)row * ldr + r];
            x = cadd(outer.given() ? outer.at(row, r, ldr) : x, v);
        }
    }
    __syncthreads();
}

// ---- fronts of the levels with more than 32 pivots ----
// The factorisation leaves the full inverses of both pivot triangles there
// (tri.cu), so the pivot rows are products too, over as many CTAs as they
// have 32-row tiles, and no CTA walks a chain of 32-pivot blocks: in one
// CTA per front and slice that chain was the longest part of every upper
// level (1030 pivots, one matrix, 100 right-hand sides: 2.8 ms for the
// forward and 2.6 ms for the backward pivot rows of two such fronts).
// y goes to the separate pivot workspace a.y, since every tile reads all the
// rows above (below) it.

// Product of rows i0 .. i0 + rows of a factor with the right operand rows
// row_ptr(k), k = k0 .. k1 - 1, accumulated in chunks of PKC pivots staged PST
// deep: the next chunks' copies are in flight while one is multiplied.  TRI:
// i0 is a multiple of 32 and the chunks inside i0 .. i0 + 31 belong to the
// diagonal block's stored inverse (of the forward or the backward operator).
// Two 16-pivot chunks take the shared memory of one 32-pivot tile, so six
// CTAs still fit an SM; measured at 841 x 227 (10 x 100), backward levels
// 7-10 (52-113 pivots): 1.11 ms unpiped in 32-pivot tiles, 1.27 ms with two
// 32-pivot chunks (three CTAs per SM), 1.03 ms so; three or four chunks in
// flight 1.16 and 1.28 ms.
constexpr int PKC = 16, PST = 2;

template <class C, int RT, int B>
struct PipeStage {
    C L[PKC][RT + SPAD];       // factor tile, [pivot q][row]
    C Y[PKC][8 * B + SPAD];    // right operand, [pivot q][rhs]
};

template <class R, bool TRANS, bool FWD, bool TRI, int RT, int B, class RowPtr>
__device__ __forceinline__ void pipe_product(PipeStage<cplx<R>, RT, B> *st, const cplx<R> *F, int f, int i0, int rows,
                                             int k0, int k1, RowPtr row_ptr, int rn, TileAcc<cplx<R>, RT, B> &acc) {
    using C = cplx<R>;
    const int nc = (k1 - k0 + PKC - 1) / PKC;
    auto stage = [&](int j) {
        if (j < nc) {
            PipeStage<C, RT, B> &sm = st[j % PST];
            const int q0 = k0 + j * PKC, qb = min(PKC, k1 - q0);
            if (TRI && q0 >= i0 && q0 < i0 + SNB)
                stage_dinv_p<C, FWD, TRANS, RT, PKC>(sm.L, F, f, i0, rows, q0 - i0, qb, threadIdx.x, NT);
            else
                stage_factor_p<C, TRANS, RT, PKC>(sm.L, F, f, i0, rows, q0, qb, threadIdx.x, NT);
            stage_rows_p<C, 8 * B>(sm.Y, [&](int q) { return row_ptr(q0 + q); }, qb, rn, threadIdx.x, NT);
        }
        async_commit();
    };
#pragma unroll
    for (int j = 0; j < PST - 1; ++j) stage(j);
    for (int j = 0; j < nc; ++j) {
        async_wait_group<PST - 2>();   // chunk j has landed
        __syncthreads();               // and every warp is past chunk j - 1
        stage(j + PST - 1);
        const PipeStage<C, RT, B> &sm = st[j % PST];
        tile_mma_p<RT, B>(sm.L, sm.Y, min(PKC, k1 - k0 - j * PKC), acc, rows, rn, threadIdx.x);
    }
}

// rows of this front in the pivot workspace, this slice's columns
template <class R, int TC>
__device__ __forceinline__ cplx<R> *pivot_work(const SolveArgs<R> &a, int node, int chunk) {
    return reinterpret_cast<cplx<R> *>(a.y) + (solve_slot(a) * (size_t)a.s.y_total + (size_t)a.s.y_off[node]) * a.ldr +
           chunk * TC;
}

// Forward pass, right-hand sides: the children's update vectors (gathered by
// the extend-add inverse maps) are added into x at this front's pivots, one
// 32-pivot block x slice per CTA; for M x = b with row exchanges the block's
// rows are left in pivot order (prow[q]: the block row at pivot position q).
// blockIdx.x = chunk + nchunk * block
template <class R, bool TRANS, int B>
__global__ void __launch_bounds__(NT) k_fwd_rhs(SolveArgs<R> a, int lvl_first, int nchunk) {
    using C = cplx<R>;
    constexpr int TC = 8 * B, NE = SNB * TC / NT;
    const int chunk = blockIdx.x % nchunk, k0 = blockIdx.x / nchunk * SNB;
    const Ctx<R> c = make_ctx<R, TC>(a, lvl_first, chunk);
    if (c.rn <= 0 || k0 >= c.s) return;
    const int r0 = chunk * TC;
    if (!live(a, c.node, r0, c.rn)) return;   // y and the update vector are zero
    const int *inv = a.s.inv + a.s.inv_off[c.node];
    const C *Wall = reinterpret_cast<const C *>(a.w) + solve_slot(a) * (size_t)a.s.rhs_total * a.ldr + r0;
    const int c0 = a.s.child0[c.node], c1 = a.s.child1[c.node];
    const C *W0 = c0 >= 0 && live(a, c0, r0, c.rn) ? Wall + (size_t)a.s.rhs_off[c0] * a.ldr : nullptr;
    const C *W1 = c1 >= 0 && live(a, c1, r0, c.rn) ? Wall + (size_t)a.s.rhs_off[c1] * a.ldr : nullptr;
    const LiveCols<TC> l0(a, c0, r0, c.rn), l1(a, c1, r0, c.rn);
    const size_t ldr = a.ldr;
    const OuterRhs<R> outer(a, r0);
    const bool pv = !TRANS && a.pivsrc;
    if (!(W0 || W1 || outer.given() || pv)) return;   // CTA-uniform: x holds the block's right-hand sides already
    const unsigned char *psrc = pv ? a.pivsrc + solve_matrix(a) * (size_t)a.s.n : nullptr;
    const int kb = min(SNB, c.s - k0);
    C v[NE];   // all of the block's rows are read before any is written
#pragma unroll
    for (int e = 0; e < NE; ++e) {
        const int t = threadIdx.x + NT * e, q = t / TC, r = t % TC;
        v[e] = czero<C>();
        if (q < kb && r < c.rn) {
            const int p = k0 + (pv ? psrc[c.vars[k0 + q]] : q);
            const int row = c.vars[p];
            const int q0 = W0 ? inv[p] : -1, q1 = W1 ? inv[c.f + p] : -1;
            v[e] = outer.given() ? outer.at(row, r, ldr) : c.X[(size_t)row * ldr + r];
            C g = czero<C>();
            if (q0 >= 0 && l0.has(r)) g = cadd(g, W0[(size_t)q0 * ldr + r]);
            if (q1 >= 0 && l1.has(r)) g = cadd(g, W1[(size_t)q1 * ldr + r]);
            v[e] = cadd(v[e], g);
        }
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < NE; ++e) {
        const int t = threadIdx.x + NT * e, q = t / TC, r = t % TC;
        if (q < kb && r < c.rn) c.X[(size_t)c.vars[k0 + q] * ldr + r] = v[e];
    }
}

// Forward pass, pivot part: y = (inverse of the forward triangle) x[pivots],
// one 32-row tile x slice per CTA; zero where the pruned pass skips the
// front.  blockIdx.x = chunk + nchunk * tile
template <class R, bool TRANS, int B>
__global__ void __launch_bounds__(NT) k_fwd_tri(SolveArgs<R> a, int lvl_first, int nchunk) {
    using C = cplx<R>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto *st = reinterpret_cast<PipeStage<C, SNB, B> *>(smem_raw);
    constexpr int TC = 8 * B;
    const int chunk = blockIdx.x % nchunk, i0 = blockIdx.x / nchunk * SNB;
    const Ctx<R> c = make_ctx<R, TC>(a, lvl_first, chunk);
    if (c.rn <= 0 || i0 >= c.s) return;
    const int rows = min(SNB, c.s - i0);
    const size_t ldr = a.ldr;
    C *Y = pivot_work<R, TC>(a, c.node, chunk);
    TileAcc<C, SNB, B> acc;
    zero_acc(acc);
    if (live(a, c.node, chunk * TC, c.rn))
        pipe_product<R, TRANS, true, true, SNB, B>(st, c.F, c.f, i0, rows, 0, i0 + rows,
                                                   [&](int k) { return c.X + (size_t)c.vars[k] * ldr; }, c.rn, acc);
    for_acc(acc, rows, c.rn, threadIdx.x, [&](int row, int r, const C &v) { Y[(size_t)(i0 + row) * ldr + r] = v; });
}

// Forward pass, ring part: update vector = children's update vectors at the
// ring rows - L'(ring, pivots) y, RT-row tiles of the ring over many CTAs;
// blockIdx.x = chunk + nchunk * tile
template <class R, bool TRANS, int RT, int B>
__global__ void __launch_bounds__(NT) k_fwd_ring(SolveArgs<R> a, int lvl_first, int nchunk) {
    using C = cplx<R>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto *st = reinterpret_cast<PipeStage<C, RT, B> *>(smem_raw);
    constexpr int TC = 8 * B;
    const int chunk = blockIdx.x % nchunk, tile = blockIdx.x / nchunk;
    const Ctx<R> c = make_ctx<R, TC>(a, lvl_first, chunk);
    const int i0 = c.s + tile * RT;
    if (c.rn <= 0 || i0 >= c.f) return;
    if (!live(a, c.node, chunk * TC, c.rn)) return;   // the update vector is zero (never read)
    const int rows = min(RT, c.f - i0);
    const size_t ldr = a.ldr;
    const C *Y = pivot_work<R, TC>(a, c.node, chunk);
    // the accumulators start from minus the children's update vectors, whose
    // loads then overlap the first chunk's copies
    const int *inv = a.s.inv + a.s.inv_off[c.node];
    const C *Wall = reinterpret_cast<const C *>(a.w) + solve_slot(a) * a.s.rhs_total * a.ldr + chunk * TC;
    const int c0 = a.s.child0[c.node], c1 = a.s.child1[c.node];
    const C *W0 = c0 >= 0 && live(a, c0, chunk * TC, c.rn) ? Wall + (size_t)a.s.rhs_off[c0] * a.ldr : nullptr;
    const C *W1 = c1 >= 0 && live(a, c1, chunk * TC, c.rn) ? Wall + (size_t)a.s.rhs_off[c1] * a.ldr : nullptr;
    const LiveCols<TC> l0(a, c0, chunk * TC, c.rn), l1(a, c1, chunk * TC, c.rn);
    TileAcc<C, RT, B> acc;
    zero_acc(acc);
    for_acc(acc, rows, c.rn, threadIdx.x, [&](int row, int r, C &v) {
        const int i = i0 + row;
        const int q0 = W0 ? inv[i] : -1, q1 = W1 ? inv[c.f + i] : -1;
        if (q0 >= 0 && l0.has(r)) v = csub(v, W0[(size_t)q0 * ldr + r]);
        if (q1 >= 0 && l1.has(r)) v = csub(v, W1[(size_t)q1 * ldr + r]);
    });
    pipe_product<R, TRANS, true, false, RT, B>(st, c.F, c.f, i0, rows, 0, c.s,
                                               [&](int k) { return Y + (size_t)k * ldr; }, c.rn, acc);
    for_acc(acc, rows, c.rn, threadIdx.x, [&](int row, int r, const C &v) {
        c.W[(size_t)(i0 + row - c.s) * ldr + r] = csub(czero<C>(), v);
    });
}

// Backward pass, ring part: t = y - U'(pivots, ring) x[ring] (final values
// of the ancestors' variables) in the pivot workspace; blockIdx.x = chunk +
// nchunk * tile
template <class R, bool TRANS, int RT, int B>
__global__ void __launch_bounds__(NT) k_bwd_ring(SolveArgs<R> a, int lvl_first, int nchunk) {
    using C = cplx<R>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto *st = reinterpret_cast<PipeStage<C, RT, B> *>(smem_raw);
    constexpr int TC = 8 * B;
    const int chunk = blockIdx.x % nchunk, tile = blockIdx.x / nchunk;
    const Ctx<R> c = make_ctx<R, TC>(a, lvl_first, chunk);
    const int i0 = tile * RT;
    if (c.rn <= 0 || i0 >= c.s || c.f == c.s) return;
    const int rows = min(RT, c.s - i0);
    const size_t ldr = a.ldr;
    C *Y = pivot_work<R, TC>(a, c.node, chunk);
    TileAcc<C, RT, B> acc;   // starts from -y: its loads overlap the first chunk's copies
    zero_acc(acc);
    for_acc(acc, rows, c.rn, threadIdx.x,
            [&](int row, int r, C &v) { v = csub(v, Y[(size_t)(i0 + row) * ldr + r]); });
    pipe_product<R, TRANS, false, false, RT, B>(st, c.F, c.f, i0, rows, c.s, c.f,
                                                [&](int k) { return c.X + (size_t)c.vars[k] * ldr; }, c.rn, acc);
    for_acc(acc, rows, c.rn, threadIdx.x,
            [&](int row, int r, const C &v) { Y[(size_t)(i0 + row) * ldr + r] = csub(czero<C>(), v); });
}

// Backward pass, pivot part: x[pivots] = (inverse of the backward triangle)
// t, one 32-row tile x slice per CTA; for M^T x = b with row exchanges the
// result comes out in pivot order and is scattered to equation order within
// its block (prow[q]: the block row at pivot position q).
template <class R, bool TRANS, int B>
__global__ void __launch_bounds__(NT) k_bwd_tri(SolveArgs<R> a, int lvl_first, int nchunk) {
    using C = cplx<R>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto *st = reinterpret_cast<PipeStage<C, SNB, B> *>(smem_raw);
    constexpr int TC = 8 * B;
    const int chunk = blockIdx.x % nchunk, i0 = blockIdx.x / nchunk * SNB;
    const Ctx<R> c = make_ctx<R, TC>(a, lvl_first, chunk);
    if (c.rn <= 0 || i0 >= c.s) return;
    const int rows = min(SNB, c.s - i0);
    const size_t ldr = a.ldr;
    const C *Y = pivot_work<R, TC>(a, c.node, chunk);
    const bool pv = TRANS && a.pivsrc;
    const unsigned char *psrc = pv ? a.pivsrc + solve_matrix(a) * (size_t)a.s.n : nullptr;
    TileAcc<C, SNB, B> acc;
    zero_acc(acc);
    pipe_product<R, TRANS, false, true, SNB, B>(st, c.F, c.f, i0, rows, i0, c.s,
                                                [&](int k) { return Y + (size_t)k * ldr; }, c.rn, acc);
    for_acc(acc, rows, c.rn, threadIdx.x, [&](int row, int r, const C &v) {
        const int p = i0 + (pv ? psrc[c.vars[i0 + row]] : row);
        c.X[(size_t)c.vars[p] * ldr + r] = v;
    });
}

// (The small-front kernels are held to 80 registers, six CTAs per SM: they
// stall on global loads first, so more resident warps pay.  Measured at
// 841 x 227, 10 matrices x 100 right-hand sides, complex64 forward levels 0-6:
// 18.0 -> 14.4 ms over three passes against the unbounded 118 registers.)
//
// P8: the largest pivot count of the launch's fronts in blocks of 8 (1 .. 4);
// the operand tiles and accumulators follow it.  These kernels wait for global
// loads most of the time, so what counts is how many fronts an SM holds: six
// with 80 registers, eight with 64, ten with 51.  Measured at 841 x 227 (10
// matrices x 100 right-hand sides), backward levels 0-4, complex128:
// 2.78, 0.83, 0.83, 0.57, 0.39 ms with one kernel of 32 pivot rows dealt to
// the warps by rows; 2.64, 0.76, 0.75, 0.52, 0.35 dealt by columns;
// 2.47, 0.57, 0.57, 0.43, 0.30 in these sizes, a level's fronts grouped by
// theirs.
template <class C, int P8>
struct FwdSmall {
    C L[8 * P8][SNB + SPAD];    // factor rows, [pivot][row]
    C Y[8 * P8][32 + SPAD];     // pivot rows, [pivot][rhs]
};
template <class C, int P8>
struct BwdSmall {
    C L[SNB][8 * P8 + SPAD];    // factor tile, [column][pivot row]
    C Y[SNB][32 + SPAD];        // right operand, [column][rhs]
};
template <class R, int P8>
constexpr int small_ctas(bool fwd) {
    return sizeof(R) == 8 ? (P8 == 4 ? 6 : P8 == 3 ? 7 : P8 == 2 || fwd ? 8 : 10) : P8 == 4 ? 9 : fwd ? 12 : 10;
}

// Forward pass of a whole front whose pivots fit one 32-pivot block (the
// small fronts of the lower levels): the children's update vectors are added
// into x at the pivots, y = Dinv x_piv is formed in shared memory and written
// back to x, and the update vector w = (children's update vectors at the
// ring rows) - L'(ring, pivots) y follows tile by tile with y kept in shared
// memory -- k_fwd_tri and k_fwd_ring in one CTA, y read once.
// wofs >= 0: the CTA's (front position, slice) is work[wofs + blockIdx.x],
// the live pairs of a pruned pass; wofs < 0: (blockIdx.y, blockIdx.x).
template <class R, bool TRANS, int P8>
__global__ void __launch_bounds__(NT, small_ctas<R, P8>(true)) k_fwd_small(SolveArgs<R> a, int lvl_first, int wofs) {
    using C = cplx<R>;
    constexpr int RT = 32, B = 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FwdSmall<C, P8> &sm = *reinterpret_cast<FwdSmall<C, P8> *>(smem_raw);
    constexpr int TC = 8 * B;
    const int2 wk = wofs >= 0 ? a.work[wofs + blockIdx.x] : make_int2((int)blockIdx.y, (int)blockIdx.x);
    const Ctx<R> c = make_ctx<R, TC>(a, lvl_first, wk.y, wk.x, wofs >= 0 ? a.s.desc : a.s.sdesc);
    if (c.rn <= 0) return;
    const int r0 = wk.y * TC;
    if (!live(a, c.node, r0, c.rn)) return;   // y and the update vector are zero
    const int *inv = a.s.inv + a.s.inv_off[c.node];
    const size_t xz = solve_slot(a);
    const C *Wall = reinterpret_cast<const C *>(a.w) + xz * (size_t)a.s.rhs_total * a.ldr + r0;
    const int c0 = a.s.child0[c.node], c1 = a.s.child1[c.node];
    const C *W0 = c0 >= 0 && live(a, c0, r0, c.rn) ? Wall + (size_t)a.s.rhs_off[c0] * a.ldr : nullptr;
    const C *W1 = c1 >= 0 && live(a, c1, r0, c.rn) ? Wall + (size_t)a.s.rhs_off[c1] * a.ldr : nullptr;
    const size_t ldr = a.ldr;
    const int s = c.s;   // <= SNB (launch condition)

    pivot_rhs(a, c, inv, W0, W1, r0, ldr);
    // M x = b with row exchanges: the pivot rows' right-hand sides are taken
    // in pivot order (prow[q]: the front row at pivot position q)
    __shared__ unsigned char prow[SNB];
    const bool pv = !TRANS && a.pivsrc;
    if (pv) {
        if (threadIdx.x < s) prow[threadIdx.x] = a.pivsrc[solve_matrix(a) * (size_t)a.s.n + c.vars[threadIdx.x]];
        __syncthreads();
    }
    BlockTile<C> acc(c.rn, wk.x);
    if (s > 0) {
        stage_dinv_p<C, true, TRANS, RT>(sm.L, c.F, c.f, 0, s, 0, s, threadIdx.x, NT);
        stage_rows_p<C, TC>(sm.Y, [&](int q) { return c.X + (size_t)c.vars[pv ? prow[q] : q] * ldr; }, s, c.rn, threadIdx.x, NT);
        staged_sync();
        block_mma<TRI_LOWER>(sm.L, sm.Y, s, acc, s, c.rn);   // y = Dinv x_piv
        __syncthreads();
        acc.each(s, c.rn, [&](int row, int col, const C &v) { sm.Y[row][col] = v; });
        __syncthreads();
        for (int t = threadIdx.x; t < s * TC; t += NT) {
            const int q = t / TC, r = t % TC;
            if (r < c.rn) c.X[(size_t)c.vars[q] * ldr + r] = sm.Y[q][r];
        }
    }
    // w over the ring rows, 32-row tiles, y staying in sm.Y
    for (int i0 = s; i0 < c.f; i0 += RT) {
        const int rows = min(RT, c.f - i0);
        stage_factor_p<C, TRANS, RT, 8 * P8>(sm.L, c.F, c.f, i0, rows, 0, s, threadIdx.x, NT);
        staged_sync();
        acc.zero();
        block_mma<0>(sm.L, sm.Y, s, acc, rows, c.rn);
        acc.each(rows, c.rn, [&](int row, int r, const C &v) {
            const int i = i0 + row;
            const int q0 = W0 ? inv[i] : -1, q1 = W1 ? inv[c.f + i] : -1;
            C g = czero<C>();
            if (q0 >= 0) g = cadd(g, W0[(size_t)q0 * ldr + r]);
            if (q1 >= 0) g = cadd(g, W1[(size_t)q1 * ldr + r]);
            c.W[(size_t)(i - s) * ldr + r] = csub(g, v);
        });
        __syncthreads();   // sm.L is staged again for the next tile
    }
}

// Backward pass of a whole front whose pivots fit one 32-pivot block (the
// small fronts of the lower levels): t = y - U'(pivots, ring) x[ring] with
// the product accumulated in registers over 32-column ring blocks, t placed
// in shared memory, then x_piv = Dinv t -- k_bwd_ring and k_bwd_tri in one
// CTA, without writing t to x in between.
template <class R, bool TRANS, int P8>
__global__ void __launch_bounds__(NT, small_ctas<R, P8>(false)) k_bwd_small(SolveArgs<R> a, int lvl_first) {
    using C = cplx<R>;
    constexpr int RT = 8 * P8, B = 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BwdSmall<C, P8> &sm = *reinterpret_cast<BwdSmall<C, P8> *>(smem_raw);
    constexpr int TC = 8 * B;
    const Ctx<R> c = make_ctx<R, TC>(a, lvl_first, blockIdx.x, -1, a.s.sdesc);
    if (c.rn <= 0 || c.s == 0) return;
    const size_t ldr = a.ldr;
    const int s = c.s;   // <= SNB (launch condition)
    // M^T x = b with row exchanges: the result comes out in pivot order and
    // is scattered to equation order (prow[q]: the front row at pivot
    // position q; read after the staged_sync below)
    __shared__ unsigned char prow[SNB];
    const bool pv = TRANS && a.pivsrc;
    if (pv && threadIdx.x < s) prow[threadIdx.x] = a.pivsrc[solve_matrix(a) * (size_t)a.s.n + c.vars[threadIdx.x]];
    BlockTile<C, (P8 < 2 ? 2 : P8)> acc(c.rn, blockIdx.y);
    for (int j0 = s; j0 < c.f; j0 += SNB) {
        const int jb = min(SNB, c.f - j0);
        stage_factor_p<C, TRANS, RT, SNB>(sm.L, c.F, c.f, 0, s, j0, jb, threadIdx.x, NT);
        stage_rows_p<C, TC>(sm.Y, [&](int q) { return c.X + (size_t)c.vars[j0 + q] * ldr; }, jb, c.rn, threadIdx.x, NT);
        staged_sync();
        block_mma<0>(sm.L, sm.Y, jb, acc, s, c.rn);
        __syncthreads();
    }
    // t = y - acc in sm.Y (row q of the next product's right operand = pivot
    // q); y = 0 where the pruned forward pass skipped the front (its rows of
    // x are not cleared when x does not hold the right-hand sides)
    if ((a.spike_k || a.b) && a.mask) {   // y = 0 in the right-hand sides the pruned forward pass skipped
        for (int t = threadIdx.x; t < s * TC; t += NT) {
            const int q = t / TC, r = t % TC;
            if (r >= c.rn) continue;
            if (col_live(a, c.node, blockIdx.x * TC + r)) cp_async_elem(&sm.Y[q][r], c.X + (size_t)c.vars[q] * ldr + r);
            else sm.Y[q][r] = czero<C>();
        }
    } else {
        stage_rows_p<C, TC>(sm.Y, [&](int q) { return c.X + (size_t)c.vars[q] * ldr; }, s, c.rn, threadIdx.x, NT);
    }
    stage_dinv_p<C, false, TRANS, RT>(sm.L, c.F, c.f, 0, s, 0, s, threadIdx.x, NT);
    staged_sync();
    acc.each(s, c.rn, [&](int row, int col, const C &v) { sm.Y[row][col] = csub(sm.Y[row][col], v); });
    __syncthreads();
    acc.zero();
    block_mma<TRI_UPPER>(sm.L, sm.Y, s, acc, s, c.rn);   // x_piv = Dinv t
    acc.each(s, c.rn,
             [&](int row, int col, const C &v) { c.X[(size_t)c.vars[pv ? prow[row] : row] * ldr + col] = v; });
}

template <class R, int RT, int B>
static size_t pipe_smem() { return PST * sizeof(PipeStage<cplx<R>, RT, B>); }

template <class K>
static void set_smem(K kernel, size_t bytes) {
    cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <class R, int P8>
static void set_small_attrs() {
    set_smem(k_fwd_small<R, false, P8>, sizeof(FwdSmall<cplx<R>, P8>));
    set_smem(k_fwd_small<R, true, P8>, sizeof(FwdSmall<cplx<R>, P8>));
    set_smem(k_bwd_small<R, false, P8>, sizeof(BwdSmall<cplx<R>, P8>));
    set_smem(k_bwd_small<R, true, P8>, sizeof(BwdSmall<cplx<R>, P8>));
}

template <class R, int RT, int B>
static void set_attrs() {
    static bool done = false;
    if (done) return;
    const size_t sm = pipe_smem<R, RT, B>();
    set_smem(k_fwd_ring<R, false, RT, B>, sm);
    set_smem(k_fwd_ring<R, true, RT, B>, sm);
    set_smem(k_bwd_ring<R, false, RT, B>, sm);
    set_smem(k_bwd_ring<R, true, RT, B>, sm);
    if (RT == 32 && B == 4) {
        set_small_attrs<R, 1>();
        set_small_attrs<R, 2>();
        set_small_attrs<R, 3>();
        set_small_attrs<R, 4>();
    }
    if (RT == 32) {
        set_smem(k_fwd_tri<R, false, B>, sm);
        set_smem(k_fwd_tri<R, true, B>, sm);
        set_smem(k_bwd_tri<R, false, B>, sm);
        set_smem(k_bwd_tri<R, true, B>, sm);
        set_smem(k_fwd_rhs<R, false, B>, 0);
        set_smem(k_fwd_rhs<R, true, B>, 0);
    }
    done = true;
}

static int env_int(const char *name) {
    const char *v = std::getenv(name);
    return v ? std::atoi(v) : 0;
}

// Tile height of the levels with more than 32 pivots: 32 rows.  64-row tiles
// read each right operand half as often, but leave too few CTAs on the top
// levels and hold fewer per SM.  Backward pass, 32 / 64 rows: 2060 x 1060, one
// matrix, 100 right-hand sides 8.44 / 8.90 ms; 841 x 227, 10 matrices 6.25 /
// 6.28 ms, in complex64 (four passes) 19.0 / 18.8 ms.  (64 rows on levels of at
// most four fronts only: 8.55, 6.25 and 19.1 ms.)  GM_SOLVE_RT=64 forces 64;
// gm_autotune times both.
static int level_rt() {
    static const int forced = env_int("GM_SOLVE_RT");
    return forced == 64 ? 64 : 32;
}

// Right-hand-side slice width (8 B) of the same levels.  With 100 right-hand
// sides 32 / 40 columns: 841 x 227, 10 matrices, both passes 7.14 / 7.34 ms
// (one substitution), in complex64 38.6 / 38.7 ms (four); the wider slices
// read the factors less often and are kept in complex64.  GM_SOLVE_B=4 / 5
// forces 32 / 40.
template <class R>
static int slice_b(int nrhs) {
    static const int forced = env_int("GM_SOLVE_B");
    if (forced == 4 || forced == 5) return forced;
    return (sizeof(R) == 4 && nrhs > 32) ? 5 : 4;
}

template <class R>
static int solve_nfz(const SolveArgs<R> &a) { return a.fmap ? a.nfz : a.nf; }

// the live (front, slice) pairs of a pruned forward pass
template <class R, int P8>
static void forward_small_work(const SolveArgs<R> &a, const LevelInfo &L, cudaStream_t st) {
    const int wofs = a.work_off[L.index];
    const int nlive = a.work_off[L.index + 1] - wofs;
    if (nlive == 0) return;
    const size_t smem = sizeof(FwdSmall<cplx<R>, P8>);
    dim3 g(nlive, 1, solve_nfz(a));
    if (a.trans) (k_fwd_small<R, true, P8><<<g, NT, smem, st>>>(a, L.first, wofs), note_launch());
    else (k_fwd_small<R, false, P8><<<g, NT, smem, st>>>(a, L.first, wofs), note_launch());
}

// one group of a level's fronts
template <class R, int P8>
static void small_group(bool fwd, const SolveArgs<R> &a, const LevelInfo &L, const PivGroup &G, cudaStream_t st) {
    for (int c0 = 0; c0 < G.count; c0 += kMaxGridY) {
        const int first = L.first + G.first + c0;
        dim3 g((a.nrhs + 31) / 32, std::min(kMaxGridY, G.count - c0), solve_nfz(a));
        if (fwd) {
            const size_t smem = sizeof(FwdSmall<cplx<R>, P8>);
            if (a.trans) (k_fwd_small<R, true, P8><<<g, NT, smem, st>>>(a, first, -1), note_launch());
            else (k_fwd_small<R, false, P8><<<g, NT, smem, st>>>(a, first, -1), note_launch());
        } else {
            const size_t smem = sizeof(BwdSmall<cplx<R>, P8>);
            if (a.trans) (k_bwd_small<R, true, P8><<<g, NT, smem, st>>>(a, first), note_launch());
            else (k_bwd_small<R, false, P8><<<g, NT, smem, st>>>(a, first), note_launch());
        }
    }
}

template <class R>
static void small_level(bool fwd, const SolveArgs<R> &a, const LevelInfo &L, cudaStream_t st) {
    set_attrs<R, 32, 4>();
    if (fwd && a.work) {
        if (L.max_piv <= 8) forward_small_work<R, 1>(a, L, st);
        else if (L.max_piv <= 16) forward_small_work<R, 2>(a, L, st);
        else if (L.max_piv <= 24) forward_small_work<R, 3>(a, L, st);
        else forward_small_work<R, 4>(a, L, st);
        return;
    }
    for (const PivGroup &G : L.groups) {
        if (G.p8 == 1) small_group<R, 1>(fwd, a, L, G, st);
        else if (G.p8 == 2) small_group<R, 2>(fwd, a, L, G, st);
        else if (G.p8 == 3) small_group<R, 3>(fwd, a, L, G, st);
        else small_group<R, 4>(fwd, a, L, G, st);
    }
}

// Levels with at most 32 pivots per front take the fused small-front kernels
// in 32-column slices whatever the tile height and slice width; the others the
// four kernels above, RT being the tile height of their ring parts.
template <class R, int RT, int B>
static void forward_level(const SolveArgs<R> &a, const LevelInfo &L, cudaStream_t st) {
    set_attrs<R, 32, B>();
    set_attrs<R, RT, B>();
    const int nchunk = (a.nrhs + 8 * B - 1) / (8 * B);
    if (L.max_piv <= SNB) {   // one pivot block per front: fused pivot + ring kernel
        small_level<R>(true, a, L, st);
        return;
    }
    const int nblk = (L.max_piv + SNB - 1) / SNB;
    for_level_pieces(L, [&](int first, int count) {
        dim3 g(nchunk * nblk, count, solve_nfz(a));
        if (a.trans) {
            (k_fwd_rhs<R, true, B><<<g, NT, 0, st>>>(a, first, nchunk), note_launch());
            (k_fwd_tri<R, true, B><<<g, NT, pipe_smem<R, 32, B>(), st>>>(a, first, nchunk), note_launch());
        } else {
            (k_fwd_rhs<R, false, B><<<g, NT, 0, st>>>(a, first, nchunk), note_launch());
            (k_fwd_tri<R, false, B><<<g, NT, pipe_smem<R, 32, B>(), st>>>(a, first, nchunk), note_launch());
        }
        if (L.max_ring > 0) {
            const size_t smr = pipe_smem<R, RT, B>();
            dim3 g2(nchunk * ((L.max_ring + RT - 1) / RT), count, solve_nfz(a));
            if (a.trans) (k_fwd_ring<R, true, RT, B><<<g2, NT, smr, st>>>(a, first, nchunk), note_launch());
            else (k_fwd_ring<R, false, RT, B><<<g2, NT, smr, st>>>(a, first, nchunk), note_launch());
        }
    });
}

template <class R, int RT, int B>
static void backward_level(const SolveArgs<R> &a, const LevelInfo &L, cudaStream_t st) {
    set_attrs<R, 32, B>();
    set_attrs<R, RT, B>();
    const int nchunk = (a.nrhs + 8 * B - 1) / (8 * B);
    if (L.max_piv <= SNB) {   // one pivot block per front: fused ring + pivot kernel
        small_level<R>(false, a, L, st);
        return;
    }
    const int nblk = (L.max_piv + SNB - 1) / SNB;
    for_level_pieces(L, [&](int first, int count) {
        if (L.max_ring > 0) {
            const size_t smr = pipe_smem<R, RT, B>();
            dim3 g1(nchunk * ((L.max_piv + RT - 1) / RT), count, solve_nfz(a));
            if (a.trans) (k_bwd_ring<R, true, RT, B><<<g1, NT, smr, st>>>(a, first, nchunk), note_launch());
            else (k_bwd_ring<R, false, RT, B><<<g1, NT, smr, st>>>(a, first, nchunk), note_launch());
        }
        dim3 g2(nchunk * nblk, count, solve_nfz(a));
        if (a.trans) (k_bwd_tri<R, true, B><<<g2, NT, pipe_smem<R, 32, B>(), st>>>(a, first, nchunk), note_launch());
        else (k_bwd_tri<R, false, B><<<g2, NT, pipe_smem<R, 32, B>(), st>>>(a, first, nchunk), note_launch());
    });
}

template <class R, int B>
static void level_pass(bool fwd, int rt, const SolveArgs<R> &a, const LevelInfo &L, cudaStream_t st) {
    if (rt == 32) {
        if (fwd) forward_level<R, 32, B>(a, L, st);
        else backward_level<R, 32, B>(a, L, st);
    } else {
        if (fwd) forward_level<R, 64, B>(a, L, st);
        else backward_level<R, 64, B>(a, L, st);
    }
}

// The level's tile height and slice width: the autotuned choice when the
// engine holds one (a.lvl_cfg, per level: forward rt, forward B, backward
// rt, backward B; 0 = the default rule), else the default rules above.
template <class R>
static void dispatch(bool fwd, const SolveArgs<R> &a_in, const LevelInfo &L, cudaStream_t st) {
    if (L.count == 0 || solve_nfz(a_in) <= 0) return;
    SolveArgs<R> a = a_in;
    if (!level_pivots<R>(L)) a.pivsrc = nullptr;   // no row exchanges on this level
    const int *c = a.lvl_cfg ? a.lvl_cfg + 4 * L.index + (fwd ? 0 : 2) : nullptr;
    const int rt = c && c[0] ? c[0] : level_rt(), b = c && c[1] ? c[1] : slice_b<R>(a.nrhs);
    if (b == 5) level_pass<R, 5>(fwd, rt, a, L, st);
    else level_pass<R, 4>(fwd, rt, a, L, st);
}

template <class R>
void launch_solve_forward_level(const SolveArgs<R> &a, const LevelInfo &L, cudaStream_t st) {
    dispatch<R>(true, a, L, st);
}

template <class R>
void launch_solve_backward_level(const SolveArgs<R> &a, const LevelInfo &L, cudaStream_t st) {
    dispatch<R>(false, a, L, st);
}

// Sets the shared-memory attribute of every substitution kernel variant,
// which also loads each kernel (CUDA loads modules and functions lazily, on
// first use, and a load takes device memory): a caller that must not
// allocate once solving has begun calls this beforehand.
void preload_solve_kernels() {
    set_attrs<double, 32, 4>();
    set_attrs<double, 64, 4>();
    set_attrs<double, 32, 5>();
    set_attrs<double, 64, 5>();
    set_attrs<float, 32, 4>();
    set_attrs<float, 64, 4>();
    set_attrs<float, 32, 5>();
    set_attrs<float, 64, 5>();
}

int solve_slice_width(int nrhs, bool fp64) { return 8 * (fp64 ? slice_b<double>(nrhs) : slice_b<float>(nrhs)); }
int solve_level_rt() { return level_rt(); }

template void launch_solve_forward_level<double>(const SolveArgs<double> &, const LevelInfo &, cudaStream_t);
template void launch_solve_forward_level<float>(const SolveArgs<float> &, const LevelInfo &, cudaStream_t);
template void launch_solve_backward_level<double>(const SolveArgs<double> &, const LevelInfo &, cudaStream_t);
template void launch_solve_backward_level<float>(const SolveArgs<float> &, const LevelInfo &, cudaStream_t);

}  // namespace gm
