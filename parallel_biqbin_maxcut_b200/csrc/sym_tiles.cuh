// FP64 matrices of one 512-thread CTA as 8 x 8 tiles (n <= 128), on the FP64
// tensor instruction (mma.sync m8n8k4 f64; sm_100a has no tcgen05 form for
// FP64).
//
// A symmetric matrix of T = ceil(n / 8) tile rows is stored as its lower
// tiles (I >= J), tile (I, J) at 64 (I (I + 1) / 2 + J) doubles; one whose two
// triangles differ in the last bit as all of them, (I, J) at 64 (I T + J).  A
// tile is row-major with the halves of rows 2, 3, 6 and 7 exchanged (column q
// of row r at q ^ (r & 2) * 2).
// Lane l of a warp holds row l >> 2, columns 2 (l & 3) and + 1 of a tile: the
// accumulator layout of the instruction.  The same two values are also the A
// and the B operand of the two k = 4 steps of an 8 x 8 x 8 product when the
// first step takes the even and the second the odd columns, so a product
// X Y^T of two tiles needs one 16-byte load a lane and operand, without
// shuffles; with the permutation these loads and the accumulators' stores
// touch every bank once.
#pragma once
#include "bqb_common.cuh"

namespace bqb {

constexpr int ST_NMAX = 128;
constexpr int ST_THREADS = 512;

// The CTA's dynamic shared memory (every kernel's own name for it is the
// same array); the routines below take offsets in doubles into it, so their
// accesses stay shared-memory accesses.
extern __shared__ __align__(16) double st_smem[];

__host__ __device__ __forceinline__ int st_tiles(int n) { return (n + 7) >> 3; }
__host__ __device__ __forceinline__ int st_packed(int T) { return 64 * (T * (T + 1) / 2); }
__device__ __forceinline__ int st_index(int I, int J) { return I * (I + 1) / 2 + J; }

// Tile row and column of packed index t.
__device__ __forceinline__ void st_decode(int t, int* I, int* J)
{
    int i = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    if ((i + 1) * (i + 2) / 2 <= t) ++i;
    if (i * (i + 1) / 2 > t) --i;
    *I = i;
    *J = t - i * (i + 1) / 2;
}

// Offset of column q of row r inside a tile (or of row r of a row buffer), and
// of the pair p of columns 2p and 2p + 1.
__device__ __forceinline__ int st_elem(int r, int q) { return r * 8 + (q ^ ((r & 2) << 1)); }
__device__ __forceinline__ int st_pair(int r, int p) { return st_elem(r, 2 * p); }

__device__ __forceinline__ double2 st_ld(const double* p) { return *reinterpret_cast<const double2*>(p); }
__device__ __forceinline__ void st_st(double* p, double a, double b)
{
    *reinterpret_cast<double2*>(p) = make_double2(a, b);
}

// c += a b^T over four columns.
__device__ __forceinline__ void st_mma1(double& c0, double& c1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}

// c += a b^T over the eight columns of two tiles held as pairs.
__device__ __forceinline__ void st_mma(double& c0, double& c1, const double2& a, const double2& b)
{
    st_mma1(c0, c1, a.x, b.x);
    st_mma1(c0, c1, a.y, b.y);
}

// c += a b^T, the two steps in separate accumulators (a shorter chain).
__device__ __forceinline__ void st_mma_split(double2& c, const double2& a, const double2& b)
{
    double2 h = make_double2(0.0, 0.0);
    st_mma1(c.x, c.y, a.x, b.x);
    st_mma1(h.x, h.y, a.y, b.y);
    c.x += h.x;
    c.y += h.y;
}

// This lane's places in a tile for products whose operands come from memory:
// columns c and c + 4 of its row (o, o + d), and of its row of the transpose.
struct StOp {
    int o, d, to;
    __device__ __forceinline__ StOp()
    {
        const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
        o = st_elem(r, c);
        d = (r & 2) ? -4 : 4;
        to = st_elem(c, r);   // (the second element is four rows on)
    }
};

// Named barriers of the eliminations (two of each kind of hand-over, by the
// parity of the panel: one side may be a panel ahead of the other).
enum StBar : int {
    ST_BAR_L = 1,   // + parity: the chain warp is done with a panel's diagonal block
    ST_BAR_P = 3,   // + parity: the tiles the chain warp needs after a panel
    ST_BAR_U = 5    // the update warps among themselves: a panel's operands
};
__device__ __forceinline__ void st_bar_sync(int id, int threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void st_bar_arrive(int id, int threads)
{
    __threadfence_block();
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Doubles of the eliminations' buffers.  st_inverse (T < 16): two W buffers of
// 8 T rows x 8, two sets of the chain warp's results and two pairs of tiles
// for it; st_posdef: V (8 T rows x 8), two tiles of L^{-1} and two pairs.
constexpr int ST_SET = 64 + 64 + 64 + 8;   // multipliers, row operand, block, reciprocals
__host__ __device__ __forceinline__ int st_buffers(int T)
{
    return T < 16 ? 2 * 64 * T + 2 * ST_SET + 256 : 64 * T + 384;
}

// Place of a warp in the order in which tile rows T - 1, T - 2, ... 1 are given
// out: the twelve warps of schedulers 1, 2 and 3 back and forth (equal sums
// of row lengths), then warps 4, 8 and 12 beside the chain warp.
__device__ __forceinline__ int st_row_order(int warp)
{
    const int q = warp >> 2, sch = warp & 3;
    if (sch == 0) return 11 + q;
    return 3 * q + ((q & 1) ? 3 - sch : sch - 1);
}

// ---- the inverse --------------------------------------------------------------

// Eliminate a panel's eight columns from its tile t of another row (the steps
// of the sweep, in order): step j with the column u = t(:, j) before it takes
// t(:, q) -= u w_j(q) (q != j) and t(:, j) = u inv_j.  Keeps -u and u inv of this
// lane's columns c and c + 4 (operands of the other tiles).  mult: the panel's
// w_j by rows, inv: its reciprocals (shared memory).
__device__ __forceinline__ void st_eliminate(double2& t, const double* mult, const double* inv, double2& nu, double2& w)
{
    const int lane = threadIdx.x & 31, c = lane & 3, row0 = lane & ~3;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const double u = __shfl_sync(0xffffffffu, (j & 1) ? t.y : t.x, row0 + (j >> 1));
        const double2 m = st_ld(mult + 8 * j + 2 * c);
        const double ui = u * inv[j];
        t.x = 2 * c == j ? ui : fma(-u, m.x, t.x);
        t.y = 2 * c + 1 == j ? ui : fma(-u, m.y, t.y);
        if (c == (j & 3)) {
            if (j < 4) {
                nu.x = -u;
                w.x = ui;
            } else {
                nu.y = -u;
                w.y = ui;
            }
        }
    }
}

// The sweep's eight steps on the panel's own diagonal block d (one warp): step
// j with the column u = d(:, j), inv = 1 / d_jj as the square of its reciprocal
// square root: d(i, q) -= u_i (u_q inv) (i, q != j), row and column j = u inv,
// d_jj = -inv.  Every lane computes the next pivot for itself, so the chain is
// a reciprocal square root, two products and an FMA a step.  set: the results
// for the other warps: the multipliers u_q inv by steps, the operand of the
// panel's own row (its row i starts at step i with the multipliers and takes
// the later steps: 0 before, 1 at and -u_i after step i), the block, the
// reciprocals.  False on a non-positive pivot, in every lane.  ALONE: the first
// n steps of a matrix's only tile, with nothing left in set.
template <bool ALONE = false>
__device__ __forceinline__ bool st_diagonal(double2& d, double* set, int n = 8)
{
    const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
    const int row0 = lane & ~3;
    constexpr unsigned ALL = 0xffffffffu;
    bool pd = true;
    double2 po = make_double2(0.0, 0.0);
    double p = __shfl_sync(ALL, d.x, 0);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (ALONE && j >= n) break;
        const int h = j >> 1;
        const double dj = (j & 1) ? d.y : d.x;
        double e = 0.0, pn = 1.0;
        if (j < 7) {
            e = __shfl_sync(ALL, dj, 4 * (j + 1) + h);                                        // d[j+1][j]
            pn = __shfl_sync(ALL, ((j + 1) & 1) ? d.y : d.x, 4 * (j + 1) + ((j + 1) >> 1));   // d[j+1][j+1]
        }
        const double dr = __shfl_sync(ALL, dj, row0 + h);        // d[r][j]
        const double d0 = __shfl_sync(ALL, dj, 8 * c + h);       // d[2c][j]
        const double d1 = __shfl_sync(ALL, dj, 8 * c + 4 + h);   // d[2c+1][j]
        pd = pd && p > 0.0;
        const double rq = rsqrt(p);
        const double inv = rq * rq;
        const double we = e * inv;
        p = fma(-e, we, pn);
        const double w0 = d0 * inv, w1 = d1 * inv, dv = dr * inv;
        const double a0 = fma(-dr, w0, d.x), a1 = fma(-dr, w1, d.y);
        d.x = 2 * c == j ? (r == j ? -inv : dv) : (r == j ? w0 : a0);
        d.y = 2 * c + 1 == j ? (r == j ? -inv : dv) : (r == j ? w1 : a1);
        if (ALONE) continue;
        if (r == j) st_st(set + 8 * j + 2 * c, w0, w1);
        if (c == (j & 3)) {
            const double v = r == j ? 1.0 : (r < j ? -dr : 0.0);
            if (j < 4) po.x = v;
            else po.y = v;
        }
        if (lane == 0) set[192 + j] = inv;
    }
    if (ALONE) return pd;
    const StOp op;
    set[64 + op.o] = po.x;
    set[64 + op.o + op.d] = po.y;
    st_st(set + 128 + st_pair(r, c), d.x, d.y);
    return pd;
}

// Inverse of a symmetric positive definite matrix A (n <= 8 T rows, T < 16) by
// the symmetric Gauss-Jordan sweep without pivoting.  Entry by entry this is
// the sweep by single columns k,
//   A_ij -= c_i (c_j / d)  (i, j != k; c = A(:, k) and d = A_kk before the step),
//   A_ik = A_ki = c_i / d, A_kk = -1 / d,  1 / d = rsqrt(d)^2,
// each product and FMA in that order (both triangles are kept: their entries
// round differently in the last bit), so the result is the same bits as the
// step-by-step form.  Eight steps at a time: the diagonal block and the
// panel's column tiles take the steps one after another; every other tile
// (I, J) takes them as A_IJ += (-U_I) W_J^T, U_I and W_J the columns c and c / d of
// the panel's tiles, whose k order on the tensor instruction is the steps'
// order (the instruction rounds after every k, in ascending order).
//
// Roles.  The chain warp (warp 0) goes from diagonal block to diagonal block:
// the block's steps, then its own copy of the next tile row's elimination and
// the next block, from two tiles that the update warps leave it a panel ahead.
// Update warp of tile row I: with the panel's multipliers it eliminates its
// column tile (keeping U_I, sharing W_I), then updates its other tiles, its U_I
// (or the panel's own row operand) being one operand of all of them.  A row's
// tiles are indexed by their column, so nothing is searched for.  The rows go
// to the warps of schedulers 1, 2 and 3 first: an FP64 instruction of the
// chain waits up to 16 cycles for a tensor instruction on its own scheduler
// (eight pivots take 1000 cycles alone, 2200 beside three rows).
// A panel takes 2000 cycles for T = 1 .. 5 (the chain), 2650 at T = 8, 4400 at
// T = 13 (the update warps: 1100 for their column tile, 2900 for the other
// tiles, against 1660 of tensor issue); the single-column sweep took 8 x 1340.
//
// `fill(I, J, r, c)` gives A's pair (row r, columns 2c and 2c + 1 of tile
// (I, J)); `store(I, J, v0, v1)` takes the inverse's pairs.
// buf: st_buffers(T) doubles of shared memory; flag: one shared int.  All
// threads of the CTA call it; false (in all) on a non-positive pivot.
template <class Fill, class Store>
__device__ __forceinline__ bool st_inverse(int T, double* buf, int* flag, Fill fill, Store store)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = lane >> 2, c = lane & 3;
    const int pr = st_pair(r, c);
    const StOp op;
    const int NU = 32 * T, NC = NU + 32;   // threads at the barriers
    double* const sets = buf + 128 * T;
    double* const Pb = sets + 2 * ST_SET;   // + 128: odd panels; tiles (K + 1, K) and (K + 1, K + 1)
    if (threadIdx.x == 0) *flag = 0;
    __syncthreads();
    int failed = 0;   // (the chain warp's)
    if (warp == 0) {
        st_bar_sync(ST_BAR_P + 1, NC);
        double2 d = st_ld(Pb + 128 + 64 + pr);
        for (int K = 0; K < T; ++K) {
            double* set = sets + ST_SET * (K & 1);
            const bool pd = st_diagonal(d, set);
            failed = pd ? 0 : 1;
            if (lane == 0 && !pd) *flag = K + 1;   // (the panel: an update warp may be one behind)
            st_bar_arrive(ST_BAR_L + (K & 1), NC);
            if (K + 1 == T) break;
            st_bar_sync(ST_BAR_P + (K & 1), NC);
            if (!pd) break;
            double2 t = st_ld(Pb + 128 * (K & 1) + pr), nu, w;
            d = st_ld(Pb + 128 * (K & 1) + 64 + pr);
            __syncwarp();
            st_eliminate(t, set, set + 192, nu, w);
            st_mma(d.x, d.y, nu, w);
        }
    } else if (const int I = st_row_order(warp); I < T) {
        double2 m[15];
#pragma unroll
        for (int J = 0; J < 15; ++J) {
            m[J] = make_double2(0.0, 0.0);
            if (J < T) m[J] = fill(I, J, r, c);
        }
        double2 nx = m[0];   // tile (I, K) when panel K comes
        if (I == 0) st_st(Pb + 128 + 64 + pr, nx.x, nx.y);
        st_bar_arrive(ST_BAR_P + 1, NC);
        if (I == 1) {
            st_st(Pb + pr, nx.x, nx.y);
            st_st(Pb + 64 + pr, m[1].x, m[1].y);
        }
        if (T > 1) st_bar_arrive(ST_BAR_P, NC);
        for (int K = 0; K < T; ++K) {
            const double* set = sets + ST_SET * (K & 1);
            double* Wk = buf + ((K & 1) ? 64 * T : 0);
            st_bar_sync(ST_BAR_L + (K & 1), NC);
            const int bad = *(volatile int*)flag;
            if (bad && bad <= K + 1) break;
            const bool own = I == K;
            double2 a = make_double2(0.0, 0.0);
            if (own) {
                nx = st_ld(set + 128 + pr);
                a = make_double2(set[64 + op.o], set[64 + op.o + op.d]);
            } else {
                double2 w = a;
                st_eliminate(nx, set, set + 192, a, w);
                Wk[64 * I + op.o] = w.x;
                Wk[64 * I + op.o + op.d] = w.y;
            }
            st_bar_sync(ST_BAR_U, NU);
            // the other tiles, four at a time: their operands, their first
            // steps, their second steps
            const double2 done = nx;
#pragma unroll
            for (int g = 0; g < 15; g += 4) {
                if (g >= T) break;
                double2 b[4];
#pragma unroll
                for (int q = 0; q < 4 && g + q < 15; ++q) {
                    b[q] = make_double2(Wk[64 * (g + q) + op.o], Wk[64 * (g + q) + op.o + op.d]);
                    m[g + q].x = own ? 0.0 : m[g + q].x;
                    m[g + q].y = own ? 0.0 : m[g + q].y;
                }
#pragma unroll
                for (int q = 0; q < 4 && g + q < 15; ++q)
                    if (g + q < T && g + q != K) st_mma1(m[g + q].x, m[g + q].y, a.x, b[q].x);
#pragma unroll
                for (int q = 0; q < 4 && g + q < 15; ++q)
                    if (g + q < T && g + q != K) st_mma1(m[g + q].x, m[g + q].y, a.y, b[q].y);
#pragma unroll
                for (int q = 0; q < 4 && g + q < 15; ++q) {
                    // (component by component: a select of structures would put
                    // the tiles in local memory)
                    const bool is_k = g + q == K, is_n = g + q == K + 1;
                    m[g + q].x = is_k ? done.x : m[g + q].x;
                    m[g + q].y = is_k ? done.y : m[g + q].y;
                    nx.x = is_n ? m[g + q].x : nx.x;
                    nx.y = is_n ? m[g + q].y : nx.y;
                    if (g + q == K + 2 && I == K + 2) {
                        st_st(Pb + 128 * ((K + 1) & 1) + pr, nx.x, nx.y);
                        st_st(Pb + 128 * ((K + 1) & 1) + 64 + pr, m[g + q].x, m[g + q].y);
                    }
                }
            }
            if (K + 2 < T) st_bar_arrive(ST_BAR_P + ((K + 1) & 1), NC);
        }
#pragma unroll
        for (int J = 0; J < 15; ++J)
            if (J < T) store(I, J, -m[J].x, -m[J].y);
    }
    // (the flag itself may be reset by the next elimination's first thread
    // before every thread here has read it)
    return __syncthreads_or(failed) == 0;
}

// ---- positive definite or not ----------------------------------------------------

// y = L^{-1} for the Cholesky factor L of the 8 x 8 tile d (one warp, both in
// the accumulators' layout); false on a non-positive pivot, in every lane.
// Step j: column j of D and row j of Y go to the lanes by shuffles while the
// pivot's reciprocal square root is computed, and every lane computes the next
// pivot for itself, so the chain is eight times a reciprocal square root, a
// product and an FMA (69 + 8 + 8 cycles) and no shuffle is in it.  WITH_L: L
// itself, too.  ALONE: the first n steps of a matrix's only tile.
template <bool WITH_L = false, bool ALONE = false>
__device__ __forceinline__ bool st_chol_inv(double2 d, double2& y, double2* l = nullptr, int n = 8)
{
    const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
    const int row0 = lane & ~3;
    constexpr unsigned ALL = 0xffffffffu;
    y = make_double2(r == 2 * c ? 1.0 : 0.0, r == 2 * c + 1 ? 1.0 : 0.0);
    bool pd = true;
    double p = __shfl_sync(ALL, d.x, 0);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (ALONE && j >= n) break;
        const int h = j >> 1;
        const double dj = (j & 1) ? d.y : d.x;
        double e = 0.0, pn = 1.0;
        if (j < 7) {
            e = __shfl_sync(ALL, dj, 4 * (j + 1) + h);                                        // D[j+1][j]
            pn = __shfl_sync(ALL, ((j + 1) & 1) ? d.y : d.x, 4 * (j + 1) + ((j + 1) >> 1));   // D[j+1][j+1]
        }
        const double dr = __shfl_sync(ALL, dj, row0 + h);        // D[r][j]
        const double d0 = __shfl_sync(ALL, dj, 8 * c + h);       // D[2c][j]
        const double d1 = __shfl_sync(ALL, dj, 8 * c + 4 + h);   // D[2c+1][j]
        const double y0 = __shfl_sync(ALL, y.x, 4 * j + c);      // Y[j][2c]
        const double y1 = __shfl_sync(ALL, y.y, 4 * j + c);
        pd = pd && p > 0.0;
        const double rs = rsqrt(p);
        const double le = e * rs;
        p = fma(-le, le, pn);
        const double lr = r > j ? dr * rs : 0.0;
        if (WITH_L) {
            const double lj = r >= j ? dr * rs : 0.0;
            l->x = 2 * c == j ? lj : l->x;
            l->y = 2 * c + 1 == j ? lj : l->y;
        }
        d.x = fma(-lr, d0 * rs, d.x);
        d.y = fma(-lr, d1 * rs, d.y);
        const double w0 = y0 * rs, w1 = y1 * rs;
        y.x = r == j ? w0 : fma(-lr, w0, y.x);
        y.y = r == j ? w1 : fma(-lr, w1, y.y);
    }
    return pd;
}

// Is the symmetric matrix A (n <= 8 T rows) positive definite: the trailing
// updates of a Cholesky factorisation, for the pivots.  For panel K of eight
// columns with diagonal block D = L L^T and columns C: V = C L^{-T}, and the
// tiles right of it take A_IJ -= V_I V_J^T.  Roles as in st_inverse: the chain
// warp inverts the diagonal blocks' factors, the update warps hold the lower
// tile rows (negated, so that their update is one tensor instruction with the
// same operand twice), the long ones first.
//
// `fill(I, J, r, c)` gives -A's pair (row r, columns 2c and 2c + 1 of tile
// (I, J)), I >= J.  buf, flag, result as for st_inverse.  FACTOR: `store(I, J,
// v)` takes the factor's pairs (tiles I >= J) as they come, also in front of a
// non-positive pivot; without it nothing is stored.
struct StNoStore {
    __device__ void operator()(int, int, const double2&) const {}
};
template <bool FACTOR = false, class Fill, class Store = StNoStore>
__device__ __forceinline__ bool st_posdef(int T, double* buf, int* flag, Fill fill, Store store = {})
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = lane >> 2, c = lane & 3;
    const int pr = st_pair(r, c);
    const int nu = T > 1 ? T - 1 : 1;       // update warps (tile rows 1 .. T - 1)
    const int NU = 32 * nu, NC = NU + 32;   // threads at the barriers
    double* V = buf;
    double* Lb = V + 64 * T;       // + 64: odd panels
    double* Pb = Lb + 128;         // + 128: odd panels; tiles (K + 1, K) and (K + 1, K + 1)
    if (threadIdx.x == 0) *flag = 0;
    __syncthreads();
    int failed = 0;   // (the chain warp's)
    if (warp == 0) {
        st_bar_sync(ST_BAR_P + 1, NC);
        double2 d = st_ld(Pb + 128 + 64 + pr);
        for (int K = 0; K < T; ++K) {
            double2 y, l = make_double2(0.0, 0.0);
            const bool pd = st_chol_inv<FACTOR>(d, y, &l);
            if (FACTOR) store(K, K, l);
            failed = pd ? 0 : 1;
            if (lane == 0 && !pd) *flag = K + 1;   // (the panel: an update warp may be one behind)
            st_st(Lb + 64 * (K & 1) + pr, y.x, y.y);
            st_bar_arrive(ST_BAR_L + (K & 1), NC);
            if (K + 1 == T) break;
            st_bar_sync(ST_BAR_P + (K & 1), NC);
            if (!pd) break;
            // V_{K+1} = C L^{-T}, D_{K+1} -= V_{K+1} V_{K+1}^T
            const double2 cc = st_ld(Pb + 128 * (K & 1) + pr);
            d = st_ld(Pb + 128 * (K & 1) + 64 + pr);
            double2 v = make_double2(0.0, 0.0);
            st_mma_split(v, cc, y);
            st_mma_split(d, make_double2(-v.x, -v.y), v);
        }
    } else if (const int k = st_row_order(warp); k < nu) {
        const int I = T - 1 - k;         // (0 only for T = 1)
        double2 m[15], dg;
        double2 nx = make_double2(0.0, 0.0);   // A's tile (I, K) when panel K comes
        dg = nx;
#pragma unroll
        for (int J = 0; J < 15; ++J) {
            m[J] = nx;
            if (J < I) m[J] = fill(I, J, r, c);
        }
        if (I > 0) dg = fill(I, I, r, c);
        if (k == nu - 1) {
            const double2 x = fill(0, 0, r, c);
            st_st(Pb + 128 + 64 + pr, -x.x, -x.y);
        }
        st_bar_arrive(ST_BAR_P + 1, NC);
        nx = make_double2(-m[0].x, -m[0].y);
        if (I == 1) {
            st_st(Pb + pr, nx.x, nx.y);
            st_st(Pb + 64 + pr, -dg.x, -dg.y);
        }
        if (T > 1) st_bar_arrive(ST_BAR_P, NC);
        bool stopped = false;
        for (int K = 0; K + 1 < T; ++K) {
            st_bar_sync(ST_BAR_L + (K & 1), NC);
            const int bad = *(volatile int*)flag;
            if (bad && bad <= K + 1) {
                stopped = true;
                break;
            }
            double2 v = make_double2(0.0, 0.0);
            if (I > K) {
                st_mma_split(v, nx, st_ld(Lb + 64 * (K & 1) + pr));
                st_st(V + 64 * I + pr, v.x, v.y);
                if (FACTOR) store(I, K, v);
            }
            st_bar_sync(ST_BAR_U, NU);
            // the update, four tiles at a time: their operands, their first
            // steps, their second steps
            const int N = K + 1;
            if (I >= N) {
#pragma unroll
                for (int g = 0; g < 15; g += 4) {
                    if (g >= I) break;
                    if (g + 3 < N) continue;
                    double2 b[4];
#pragma unroll
                    for (int q = 0; q < 4 && g + q < 15; ++q) b[q] = st_ld(V + 64 * (g + q) + pr);
#pragma unroll
                    for (int q = 0; q < 4 && g + q < 15; ++q)
                        if (g + q < I) st_mma1(m[g + q].x, m[g + q].y, v.x, b[q].x);
#pragma unroll
                    for (int q = 0; q < 4 && g + q < 15; ++q)
                        if (g + q < I) st_mma1(m[g + q].x, m[g + q].y, v.y, b[q].y);
#pragma unroll
                    for (int q = 0; q < 4 && g + q < 15; ++q)
                        if (g + q == N) nx = make_double2(-m[g + q].x, -m[g + q].y);
                }
                st_mma(dg.x, dg.y, v, v);
                if (I == N + 1) {
                    st_st(Pb + 128 * (N & 1) + pr, nx.x, nx.y);
                    st_st(Pb + 128 * (N & 1) + 64 + pr, -dg.x, -dg.y);
                }
            }
            if (N + 1 < T) st_bar_arrive(ST_BAR_P + (N & 1), NC);
            st_bar_sync(ST_BAR_U, NU);   // (V is written again)
        }
        // the last panel has no update; its announcement is taken
        if (!stopped) st_bar_sync(ST_BAR_L + ((T - 1) & 1), NC);
    }
    return __syncthreads_or(failed) == 0;
}

// ---- matrices of one tile (n <= 8) ---------------------------------------------
//
// One warp takes the n steps, without roles and their hand-overs and without the
// padding's steps, which a bound of a few vertices would spend most of its time
// in: n = 1, 2, 4, 8 took 105, 106, 143, 144 us with st_inverse and st_posdef (73,
// 82, 144, 196 with single columns) and take 57, 57, 73, 82.  The same bits.

// As st_inverse.
template <class Fill, class Store>
__device__ __forceinline__ bool st_inverse_one(int n, Fill fill, Store store)
{
    const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
    __syncthreads();
    bool pd = true;
    if (threadIdx.x < 32) {
        double2 d = fill(0, 0, r, c);
        pd = st_diagonal<true>(d, nullptr, n);
        store(0, 0, r < n ? -d.x : d.x, r < n ? -d.y : d.y);   // (the identity outside)
    }
    return __syncthreads_and(pd) != 0;
}

// As st_posdef (nothing is stored).
template <class Fill>
__device__ __forceinline__ bool st_posdef_one(int n, Fill fill)
{
    const int lane = threadIdx.x & 31;
    __syncthreads();
    bool pd = true;
    if (threadIdx.x < 32) {
        const double2 d = fill(0, 0, lane >> 2, lane & 3);
        double2 y;
        pd = st_chol_inv<false, true>(make_double2(-d.x, -d.y), y, nullptr, n);
    }
    return __syncthreads_and(pd) != 0;
}

// The Cholesky factor of the n x n matrix A (column-major, n <= 128, lower
// triangle read and written; the upper one is left alone) by the CTA; false, in
// all threads, on a non-positive pivot (then the lower triangle is partly
// written).  buf: st_buffers(ceil(n / 8)) + 1 doubles of shared memory, 16-byte
// aligned.  n = 100: 22 us; a column, a barrier and a rank-1 update at a time
// (cta_potrf_lower) 98.
static __device__ __noinline__ bool st_potrf(double* A, int n, double* buf)
{
    const int T = st_tiles(n), lane = threadIdx.x & 31;
    return st_posdef<true>(
        T, buf, reinterpret_cast<int*>(buf + st_buffers(T)),
        [=](int I, int J, int r, int c) {
            const int i = 8 * I + r, j = 8 * J + 2 * c;
            double2 v = make_double2(i == j ? 1.0 : 0.0, i == j + 1 ? 1.0 : 0.0);
            if (i < n && j < n) v.x = A[i >= j ? i + j * n : j + i * n];
            if (i < n && j + 1 < n) v.y = A[i >= j + 1 ? i + (j + 1) * n : j + 1 + i * n];
            return make_double2(-v.x, -v.y);
        },
        [=](int I, int J, const double2& v) {
            const int i = 8 * I + (lane >> 2), j = 8 * J + 2 * (lane & 3);
            if (i < n && j <= i) A[i + j * n] = v.x;
            if (i < n && j + 1 <= i) A[i + (j + 1) * n] = v.y;
        });
}

}  // namespace bqb
