// Full inverses of the pivot triangles of the fronts with more than 32
// pivots, from the 32 x 32 diagonal-block inverses the factorisation leaves,
// so that the substitution forms a front's pivot rows as one product.
//
// In place, by doubling: with the diagonal blocks of size h inverted, a pair
// of them gives the inverse of the 2h block,
//   [ L11      ]^-1   [       X11           ]
//   [ L21  L22 ]    = [ -X22 (L21 X11)  X22 ],   U alike with the upper part,
// as two products through a scratch matrix (T = L21 X11, X21 = -X22 T), so a
// front of s pivots takes 2 ceil(log2(s / 32)) launches.  L21's rows are
// taken through the blocks' row exchanges (FactorArgs::pivsrc): X is left in
// pivot order on both sides.
//
// Nothing in the factorisation reads a level's pivot triangles once the
// level is eliminated, so these launches run on their own stream beside the
// levels above: the work is s^3 / 3 complex multiply-adds per triangle pair,
// small against the fronts' Schur updates, and the upper levels leave most of
// the chip idle.  Accuracy, against inverses of the 32 x 32 blocks only: direct
// residuals within a factor of two either way over the 2-11 Hz, 5-25 Hz SH and
// 100-400 MHz georadar operators (multifrontal replay in double precision); on
// the device 841 x 227, 9 / 10 / 11 Hz 1.3e-12 -> 1.5e-12, 1.2e-11 -> 1.7e-11
// (the worst), 4.3e-13 -> 3.6e-13.  The fields are no further from a 64-bit
// solution.
#include "solve_tile.cuh"

namespace gm {

constexpr int TRB = 4;   // 32-column right operands

// One 32 x 32 output tile per CTA.  blockIdx.x = triangle (0: L, 1: U) + 2 *
// (tile + (h / 32)^2 * pair); PHASE 0 forms T, PHASE 1 the inverse's block.
template <class R, int PHASE>
__global__ void __launch_bounds__(NT) k_tri_inverse(FactorArgs<R> a, int lvl_first, int h, cplx<R> *scratch,
                                                    int64_t scratch_total, const int64_t *scratch_off) {
    using C = cplx<R>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto *st = reinterpret_cast<SolveSmem<C, SNB, TRB> *>(smem_raw);
    const int node = a.s.lvl_nodes[lvl_first + blockIdx.y];
    const int f = a.s.nfront[node], s = a.s.npiv[node];
    const int nb = h / SNB;
    const bool upper = blockIdx.x & 1;
    const int tile = (blockIdx.x >> 1) % (nb * nb), pair = (blockIdx.x >> 1) / (nb * nb);
    const int k0 = pair * 2 * h, mid = k0 + h, end = min(s, mid + h);
    if (mid >= s) return;
    // rows / columns of the output tile: L fills rows mid.. x columns k0..mid,
    // U rows k0..mid x columns mid..
    const int r0 = (upper ? k0 : mid) + tile % nb * SNB, c0 = (upper ? mid : k0) + tile / nb * SNB;
    if (r0 >= end || c0 >= end) return;
    const int rows = min(SNB, (upper ? mid : end) - r0), cols = min(SNB, (upper ? end : mid) - c0);
    const C *F = reinterpret_cast<const C *>(a.front) + (size_t)blockIdx.z * a.s.front_total + a.s.front_off[node];
    C *T = scratch + (size_t)blockIdx.z * scratch_total + scratch_off[node];   // [s][s], leading dimension s

    // inner range: T = L21 X11 (inner c0 .. mid), U12 Z22 (mid .. c0 + cols);
    // X21 = -X22 T (mid .. r0 + rows), Z12 = -Z11 T (r0 .. mid)
    const int q_lo = PHASE == 0 ? (upper ? mid : c0) : (upper ? r0 : mid);
    const int q_hi = PHASE == 0 ? (upper ? c0 + cols : mid) : (upper ? mid : r0 + rows);

    // equation rows of the tile's pivot rows (L21 of an earlier block)
    __shared__ int prow[SNB];
    if (PHASE == 0) {
        if (threadIdx.x < rows) {
            int p = threadIdx.x;
            if (!upper && a.pivsrc)
                p = a.pivsrc[(size_t)blockIdx.z * a.s.n + a.s.vars[a.s.var_off[node] + r0 + threadIdx.x]];
            prow[threadIdx.x] = r0 + p;
        }
        __syncthreads();
    }
    // entry (i, j) of the inverse's triangle inside a diagonal block: stored,
    // the implied unit diagonal of L^-1, or zero
    auto stage_tri = [&](C *dst, int i, int j) {
        if (upper ? i <= j : i > j) cp_async_elem(dst, F + i + (size_t)j * f);
        else *dst = !upper && i == j ? mk(R(1), R(0)) : czero<C>();
    };
    auto stage = [&](int buf, int q0) {
        const int qb = min(SNB, q_hi - q0);
        for (int t = threadIdx.x; t < SNB * qb; t += NT) {   // left operand, columns of the front
            const int row = t % SNB, q = t / SNB;
            if (row >= rows) continue;
            C *dst = &st[buf].L[q][row];
            if (PHASE == 0) cp_async_elem(dst, F + prow[row] + (size_t)(q0 + q) * f);
            else if (q0 == r0) stage_tri(dst, r0 + row, q0 + q);
            else cp_async_elem(dst, F + (r0 + row) + (size_t)(q0 + q) * f);
        }
        for (int t = threadIdx.x; t < SNB * cols; t += NT) {   // right operand, down its columns
            const int q = t % SNB, col = t / SNB;
            if (q >= qb) continue;
            C *dst = &st[buf].Y[q][col];
            if (PHASE == 1) cp_async_elem(dst, T + (q0 + q) + (size_t)(c0 + col) * s);
            else if (q0 == c0) stage_tri(dst, q0 + q, c0 + col);
            else cp_async_elem(dst, F + (q0 + q) + (size_t)(c0 + col) * f);
        }
        async_commit();
    };
    TileAcc<C, SNB, TRB> acc;
    zero_acc(acc);
    stage(0, q_lo);
    int buf = 0;
    for (int q0 = q_lo; q0 < q_hi; q0 += SNB, buf ^= 1) {
        if (q0 + SNB < q_hi) {
            stage(buf ^ 1, q0 + SNB);
            async_wait_group<1>();
        } else {
            async_wait_group<0>();
        }
        __syncthreads();
        tile_mma_p<SNB, TRB>(st[buf].L, st[buf].Y, min(SNB, q_hi - q0), acc, rows, cols, threadIdx.x);
        __syncthreads();
    }
    C *out = PHASE == 0 ? T : const_cast<C *>(F);
    const size_t ld = PHASE == 0 ? s : f;
    for_acc(acc, rows, cols, threadIdx.x, [&](int row, int col, const C &v) {
        out[(r0 + row) + (size_t)(c0 + col) * ld] = PHASE == 0 ? v : csub(czero<C>(), v);
    });
}

template <class R>
void launch_tri_inverse(const FactorArgs<R> &a, const LevelInfo &L, void *scratch, int64_t scratch_total,
                        const int64_t *scratch_off, cudaStream_t st) {
    using C = cplx<R>;
    if (L.count == 0 || L.max_piv <= SNB) return;
    const size_t smem = 2 * sizeof(SolveSmem<C, SNB, TRB>);
    static bool attr_set = false;
    if (!attr_set) {
        cudaFuncSetAttribute(k_tri_inverse<R, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(k_tri_inverse<R, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        attr_set = true;
    }
    FactorArgs<R> b = a;
    if (!level_pivots<R>(L) || !(a.pivtau2 > 0)) b.pivsrc = nullptr;   // no row exchanges on this level
    for (int h = SNB; h < L.max_piv; h *= 2) {
        const int nb = h / SNB, npair = (L.max_piv - h + 2 * h - 1) / (2 * h);
        for_level_pieces(L, [&](int first, int count) {
            const dim3 g(2 * nb * nb * npair, count, a.nf);
            C *t = reinterpret_cast<C *>(scratch);
            (k_tri_inverse<R, 0><<<g, NT, smem, st>>>(b, first, h, t, scratch_total, scratch_off), note_launch());
            (k_tri_inverse<R, 1><<<g, NT, smem, st>>>(b, first, h, t, scratch_total, scratch_off), note_launch());
        });
    }
}

template void launch_tri_inverse<double>(const FactorArgs<double> &, const LevelInfo &, void *, int64_t,
                                         const int64_t *, cudaStream_t);
template void launch_tri_inverse<float>(const FactorArgs<float> &, const LevelInfo &, void *, int64_t,
                                        const int64_t *, cudaStream_t);

}  // namespace gm
