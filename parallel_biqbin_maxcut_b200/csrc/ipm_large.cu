// The basic SDP interior-point method (src/ipm_mc_pk.c:28-359) for n above
// the one-CTA limit (IPM_REG_NMAX = 128): ONE cooperative launch
// per call.  Every CTA (one per SM at most) runs the whole predictor-
// corrector loop; the phases of an iteration (the inverses, the solves, the
// two products, the line searches' positive-definiteness tests, the step)
// are separated by a grid barrier, and every decision (a failed pivot, the
// line-search step, the stopping test) is taken by every CTA from the same
// data with the same arithmetic, so all CTAs follow one control path with no
// host round trip.
//
// Inverses (Zi = inv(Z), F = inv(Zi .* X)) use a blocked symmetric
// Gauss-Jordan sweep on panels of CB = 32 columns.  For panel K with
// D = A_KK = Ld Ld^T and the panel columns C = A(:, K): V = C Ld^{-T},
// A_ij -= V_i V_j^T (i, j outside K), A_iK = W_i = V_i Ld^{-1} (= C_i D^{-1}),
// A_KK = -D^{-1}; after the last panel A = -inv(A).  The Cholesky pivots are
// the Schur complements of A: a non-positive one means "not positive
// definite".  The line searches' tests run the trailing part of the sweep
// only (a blocked right-looking Cholesky).  The Schur update goes through
// Ld, not the explicit D^{-1}: at n = 343 with couplings of 1e5, M reaches a
// condition number of 1e11 at the last iteration, and C D^{-1} C^T then
// turned a pivot of the positive definite M negative.
//
// A sweep holds the lower tiles only (row-major, 32 x 32; the diagonal tiles
// whole); the final phase of a full sweep writes both triangles.
//
// One grid barrier per panel: every CTA factors the 32 x 32 panel block
// itself (the same arithmetic in every CTA, hence the same decision), and
// the owner of a 32 x 32 tile of A computes the V rows it needs itself.  The
// writes of panel K's own row and column blocks (W and -D^{-1}) would race
// with the other CTAs' reads of the panel columns, so they are deferred:
// panel K leaves W_K and D^{-1}_K in side buffers, and in the next phase the
// owner of each tile in row or column block K writes them before its own
// update, while readers of the panel columns take them from the buffers.
//
// What bounds a phase is its latency (n = 343, cycles): the barrier 3000, one
// round trip to L2 1600 (the panel block, and the CTA's first tile and its panel
// columns, are loaded together, from addresses worked out before the barrier),
// the panel block's chain of 32 pivots on one warp 6000, a tile 4000.  A call at
// n = 343 takes 3.8 ms, at n = 150 1.7 (with rank-1 panel factors by rows, scalar
// tiles and all tiles of both triangles 10.2 and 4.1).  All products go through
// the FP64 tensor instruction as X Y^T of 8 x 8 tiles in its accumulators' layout
// (a lane's pair of columns is also its operand of the two k = 4 steps); V comes
// from L by tile columns, each solve with a diagonal tile's inverse.
//
// Each solve with M is the product with F = inv(M) followed by one step of
// iterative refinement with M = Zi .* X (x <- x + F (b - M x)).
//
// The grid barrier is a growing counter in global memory; every wait is
// bounded (2 s), after which the barrier sets an error word, no CTA waits any
// more, every loop ends, and the call reports status IPM_SYNC (a fatal error on
// the host).
#include <math.h>

#include <map>
#include <mutex>
#include <vector>

#include "bqb_common.cuh"
#include "internal.h"
#include "ipm.cuh"
#include "sym_tiles.cuh"

namespace bqb {

double* ipm_stats_device();

namespace {

constexpr int CB = 32;          // panel and tile width
constexpr int CT = 256;         // threads per CTA
constexpr int CW = CT / 32;     // warps per CTA
// Shared-memory rows of 40 doubles: the pairs of a fragment (eight rows, four
// pairs each) then meet every bank once.
constexpr int LD = CB + 8;
static_assert(CT == CW * 32 && CB == 32 && CW == 8, "a CTA's eight warps hold two of a tile's 16 fragments each");
constexpr unsigned long long BAR_TIMEOUT_NS = 2000000000ull;

struct CoopArgs {
    const double* L;     // n x n, read only
    double* Xbase;       // output matrix (X = Xbase + (*xslot) n^2)
    const int* xslot;
    double* out;         // phi, iterations, status, <L,X>
    double* stats;       // IPM work counters (may be null)
    double *Zi, *F, *M, *T, *T2, *dX, *dX1;   // n x n each (T, T2: the line searches' trial matrices)
    double *Wb, *Db;                     // 2 x (n x CB), 2 x (CB x CB)
    double *y, *zd, *dy, *dy1, *dy2, *r, *t;
    double* part;        // gridDim.x x 4 partial sums
    unsigned* bar;       // [0] arrivals, [2] error
    unsigned long long* prof;   // (may be null) CTA 0's nanoseconds per part, COOP_PROF_* slots
    double* yout;        // (may be null) y of the last iterate
    int n;
};

// Parts of the time CTA 0 spends in a call (bqb_ipm_coop_profile).
enum CoopProf : int {
    COOP_PROF_BARRIER,   // waiting at grid barriers
    COOP_PROF_FACTOR,    // the panel factorisations (every CTA factors each panel block), its loads and the first tile's included
    COOP_PROF_TILES,     // the sweeps' tile updates
    COOP_PROF_GEMM,      // the two symmetric products
    COOP_PROF_TOTAL,     // the whole call
    COOP_PROF_BARRIERS,  // count of grid barriers
    COOP_PROF_PHASES,    // count of sweep phases
    COOP_PROF_PF_LOAD,   // the part of them until the panel block has come (trial 0's)
    COOP_PROF_WORDS = 8
};

// Trial sweeps a line-search round runs together (each with its own panel
// factor in shared memory).
constexpr int NTRIAL = 4;

using Block = double[CB][LD];

// Shared memory: a trial's panel factor (L, the inverses Y of its diagonal tiles,
// G = L^{-T}), the tile step's V_I, V_J in two sets; the products' two sets of four operands and their
// transposes' scratch.
struct Smem {
    Block b[3 * NTRIAL + 4];
    double red[CW * 4];
    double tot[4];
    // what the sweeps use of the call's arguments: an acquire empties L1, and
    // with it whatever a function keeps in local memory
    double* A[NTRIAL];
    double *Wb, *Db;
    unsigned* bar;
    unsigned epoch;   // grid barriers passed
    int ok;
    int pd[NTRIAL];
    __device__ Block& Y(int t) { return b[2 * t]; }
    __device__ Block& G(int t) { return b[2 * t + 1]; }
    __device__ Block& L(int t) { return b[2 * NTRIAL + t]; }
    __device__ Block& V(int set, int side) { return b[3 * NTRIAL + 2 * set + side]; }
};

// This lane's fragment of 8 x 8 tile (I, J) of a block: row lane / 4, columns
// 2 (lane % 4) and + 1.
__device__ __forceinline__ double2 frag(const Block& m, int I, int J)
{
    const int lane = threadIdx.x & 31;
    return *reinterpret_cast<const double2*>(&m[8 * I + (lane >> 2)][8 * J + 2 * (lane & 3)]);
}
__device__ __forceinline__ void put(Block& m, int I, int J, const double2& v)
{
    const int lane = threadIdx.x & 31;
    *reinterpret_cast<double2*>(&m[8 * I + (lane >> 2)][8 * J + 2 * (lane & 3)]) = v;
}
// ... and the transposed tile at (J, I).
__device__ __forceinline__ void put_t(Block& m, int I, int J, const double2& v)
{
    const int lane = threadIdx.x & 31, r = 8 * J + 2 * (lane & 3), c = 8 * I + (lane >> 2);
    m[r][c] = v.x;
    m[r + 1][c] = v.y;
}
__device__ __forceinline__ void mma(double2& c, const double2& a, const double2& b) { st_mma(c.x, c.y, a, b); }
__device__ __forceinline__ double2 neg(const double2& a) { return make_double2(-a.x, -a.y); }

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid barrier with a bounded wait: one counter that only grows, a CTA
// waiting until all have added to it as often as itself.  Returns false once
// any CTA has given up (then nothing waits any more).  The fences around the
// arrival make every write before the barrier visible to every read after it.
__device__ bool grid_sync(unsigned* bar, Smem& sm, unsigned long long* prof = nullptr)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned long long tb = prof && blockIdx.x == 0 ? global_ns() : 0ull;
        const unsigned target = (sm.epoch += 1) * gridDim.x;
        int ok = 1;
        __threadfence();
        asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        unsigned long long t0 = 0ull;
        for (unsigned spin = 1;; ++spin) {
            unsigned v;
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if ((int)(v - target) >= 0) break;
            if ((spin & 255u) == 0u) {
                const unsigned long long now = global_ns();
                if (!t0) t0 = now;
                if (*(volatile unsigned*)(bar + 2) != 0u) {
                    ok = 0;
                    break;
                }
                if (now - t0 > BAR_TIMEOUT_NS) {
                    atomicExch(bar + 2, 1u);
                    ok = 0;
                    break;
                }
            }
        }
        __threadfence();
        sm.ok = ok;
        if (prof && blockIdx.x == 0) {
            prof[COOP_PROF_BARRIER] += global_ns() - tb;
            prof[COOP_PROF_BARRIERS] += 1;
        }
    }
    __syncthreads();
    return sm.ok != 0;
}

// The sums over all entries (the starting point's, the step's) are taken
// over a fixed partition into as many parts as give a thread four entries (at
// most VCTA), a block of CT threads each; a CTA of a smaller grid takes
// several parts in turn.  The totals are then the same bits for any grid.
constexpr int VCTA = 148;
__device__ __forceinline__ int sum_parts(int n)
{
    const long long p = ((long long)n * n + 4 * CT - 1) / (4 * CT);
    return p < VCTA ? (int)p : VCTA;
}

// Block-reduce four partial sums into part[v * 4 + k] (the CTA's part v).
__device__ void block_partials(double a, double b, double c, double d, Smem& sm, double* part, int v)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    a = warp_sum(a);
    b = warp_sum(b);
    c = warp_sum(c);
    d = warp_sum(d);
    if (lane == 0) {
        sm.red[w * 4 + 0] = a;
        sm.red[w * 4 + 1] = b;
        sm.red[w * 4 + 2] = c;
        sm.red[w * 4 + 3] = d;
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        double s = 0.0;
        for (int q = 0; q < CW; ++q) s += sm.red[q * 4 + threadIdx.x];
        part[v * 4 + threadIdx.x] = s;
    }
    __syncthreads();   // sm.red is reused by the CTA's next part
}

// The totals of the partial sums (after a barrier), a warp each, in a fixed
// order: the same value in every CTA.
__device__ void grid_totals(const double* part, int parts, Smem& sm)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    static_assert(VCTA <= 5 * 32, "a lane's five parts");
    if (w < 4) {
        double v[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) v[q] = lane + 32 * q < parts ? __ldcg(part + (lane + 32 * q) * 4 + w) : 0.0;
        const double s = warp_sum((((v[0] + v[1]) + v[2]) + v[3]) + v[4]);
        if (lane == 0) sm.tot[w] = s;
    }
    __syncthreads();
}

// ---- the panel sweep ---------------------------------------------------------

// Named barrier by which trial t's chain warp hands tile columns up to K of
// the factor to its helper (K = 1, 2, 3; 64 threads).
__device__ __forceinline__ int hand_over(int t, int K) { return 3 * t + K; }
static_assert(3 * NTRIAL < 16, "named barriers");

// a y^T (y = L^{-1}: x with x L^T = a).
__device__ __forceinline__ double2 solve_t(const double2& a, const double2& y)
{
    double2 x = make_double2(0.0, 0.0);
    mma(x, a, y);
    return x;
}

// The panel block D = A[K, K] (b x b, padded to 32 x 32 with the identity), its
// lower tiles, by one warp; a: this lane's first pair.
struct PanelTiles {
    double2 d[4][4];
};
__device__ __forceinline__ void panel_load(const double* a, unsigned n, int b, PanelTiles& f)
{
    const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
#pragma unroll
    for (int I = 0; I < 4; ++I)
#pragma unroll
        for (int J = 0; J <= I; ++J) {
            const double* x = a + 8 * I * n + 8 * J;
            if (b == CB) {
                f.d[I][J] = make_double2(__ldcg(x), __ldcg(x + 1));
            } else {
                const int p = 8 * I + r, q = 8 * J + 2 * c;
                f.d[I][J].x = p < b && q < b ? __ldcg(x) : (p == q ? 1.0 : 0.0);
                f.d[I][J].y = p < b && q + 1 < b ? __ldcg(x + 1) : (p == q + 1 ? 1.0 : 0.0);
            }
        }
}

// Its Cholesky factor L (tiles below the diagonal, in sm.L(t)) and the inverses
// Y of L's diagonal tiles (sm.Y(t)), as a factorisation of 4 x 4 tiles: a tile's
// eight pivots are st_chol_inv's chain (1000 cycles), the column below them and
// the trailing tiles are tensor products in registers.  5100 cycles; the 32
// steps of a rank-1 update by rows, and the substitution for the inverse after
// them, took 20000.  sm.pd[t] = 0 on a non-positive pivot (then the results are
// garbage).  helped: panel_help follows on another warp.
__device__ __forceinline__ void panel_chain(PanelTiles& f, int t, bool helped, Smem& sm)
{
    double2 (&d)[4][4] = f.d;
    Block& yb = sm.Y(t);
    Block& lo = sm.L(t);
    bool pd = true;
#pragma unroll
    for (int K = 0; K < 4; ++K) {
        double2 y;
        const bool ok = st_chol_inv(d[K][K], y);
        pd = pd && ok;
        put(yb, K, K, y);
#pragma unroll
        for (int I = K + 1; I < 4; ++I) {
            d[I][K] = solve_t(d[I][K], y);
            put(lo, I, K, d[I][K]);
        }
        if (K > 0 && helped) st_bar_arrive(hand_over(t, K), 64);
#pragma unroll
        for (int I = K + 1; I < 4; ++I)
#pragma unroll
            for (int J = K + 1; J <= I; ++J) mma(d[I][J], neg(d[I][K]), d[J][K]);
    }
    if ((threadIdx.x & 31) == 0) sm.pd[t] = pd ? 1 : 0;
}

// The helper, for a full sweep: G = L^{-T} (upper tiles), column K when the
// chain has tile column K: G_JK = -(sum_{J <= m < K} G_Jm L_Km^T) L_KK^{-T}.
__device__ __forceinline__ void panel_help(int t, Smem& sm)
{
    const Block& yb = sm.Y(t);
    Block& g = sm.G(t);
    const Block& lo = sm.L(t);
    double2 gt[4][4];   // upper tiles
#pragma unroll
    for (int K = 0; K < 4; ++K) {
        if (K > 0) st_bar_sync(hand_over(t, K), 64);
        if (K == 0) continue;
#pragma unroll
        for (int k = K == 1 ? 0 : K; k <= K; ++k) {
            const double2 y = frag(yb, k, k);
            put_t(g, k, k, y);
            __syncwarp();
            gt[k][k] = frag(g, k, k);
#pragma unroll
            for (int J = 0; J < k; ++J) {
                double2 x = make_double2(0.0, 0.0);
#pragma unroll
                for (int m = J; m < k; ++m) mma(x, gt[J][m], frag(lo, k, m));
                gt[J][k] = solve_t(neg(x), y);
                put(g, J, k, gt[J][k]);
            }
        }
    }
}

// A CTA's tile of a phase, as it comes from memory: its entries (this warp's two
// fragments: tile row warp / 2, tile columns 2 (warp & 1) and + 1), and of the
// panel's columns a strip of eight rows (strip warp & 3 of the tile's rows, or
// from warp 4 on of its columns' rows).
struct TileLoad {
    double2 c[4];
    double2 a[2];
};

// Which tile of A the phase gives the CTA, and what is to be done with it.
struct TileJob {
    double* A;
    int I, J;
    bool full;    // a full sweep's tile: also the previous panel's fix, W, D^{-1}
    int trial;    // whose panel factor
};

// Where a thread's values of a tile come from, worked out before the grid
// barrier (the index arithmetic took as long as the round trip to L2).
struct TileAddr {
    const double* c;   // the strip's pairs: columns 8 u + 2 (lane % 4) and + 1, cn of them in range, cs apart
    const double* a;   // the entries: columns 8 e and + 1, an in range, as apart
    unsigned cs, as;
    int cn, an;
};

__device__ __forceinline__ TileAddr tile_addr(const TileJob& q, int n, int K, int k0, int b, const double* Wprev,
                                              const double* Dprev)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int I = q.I, J = q.J;
    const bool upd = I != K && J != K;
    const bool fixI = q.full && K > 0 && I == K - 1, fixJ = q.full && K > 0 && J == K - 1;
    const unsigned un = n;
    TileAddr t;
    {
        // rows of the lower triangle, columns of it, or the previous panel's W
        const int B = w >= 4 ? J : I;
        const bool from_w = w >= 4 ? fixJ : fixI;
        const unsigned r = 8 * (w & 3) + (lane >> 2), i = B * CB + r, p = 2 * (lane & 3);
        t.cs = from_w ? CB : B < K ? un : 1u;
        t.c = from_w ? Wprev + ((k0 + p) * CB + r) : q.A + (B < K ? (k0 + p) * un + i : i * un + k0 + p);
        t.cn = upd && (int)i < n && (w < 4 || J != I) ? b - (int)p : 0;
    }
    {
        const unsigned i = I * CB + 8 * (w >> 1) + (lane >> 2), j = J * CB + 16 * (w & 1) + 2 * (lane & 3);
        const unsigned kp0 = (K - 1) * CB;
        t.as = fixI && !fixJ ? CB : 1u;
        t.a = fixI && fixJ ? Dprev + ((i - kp0) * CB + (j - kp0))
              : fixJ       ? Wprev + (i * CB + (j - kp0))
              : fixI       ? Wprev + (j * CB + (i - kp0))
                           : q.A + (i * un + j);
        t.an = (upd || fixI || fixJ) && (int)i < n ? n - (int)j : 0;
    }
    return t;
}

// Issue the loads (of nothing that the phase writes).
__device__ __forceinline__ void tile_load(const TileAddr& s, TileLoad& t)
{
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        t.c[u].x = 8 * u < s.cn ? __ldcg(s.c + 8 * u * s.cs) : 0.0;
        t.c[u].y = 8 * u + 1 < s.cn ? __ldcg(s.c + (8 * u + 1) * s.cs) : 0.0;
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        t.a[e].x = 8 * e < s.an ? __ldcg(s.a + 8 * e * s.as) : 0.0;
        t.a[e].y = 8 * e + 1 < s.an ? __ldcg(s.a + (8 * e + 1) * s.as) : 0.0;
    }
}

// The tile's step, from its loads: the pending fix of panel K - 1 (tiles in
// its row or column block), the update (I, J != K), and for a full sweep W_K
// of row block I (diagonal tiles) and D^{-1}_K (tile (K, K)).  One barrier,
// after the V strips (a warp each), and none without an update: the CTA's next
// update uses the other set, and its barrier is behind this one's reads.
__device__ __forceinline__ void tile_step(const TileJob& q, int n, int K, TileLoad& t, double* Wcur, double* Dcur,
                                          int set, Smem& sm)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int I = q.I, J = q.J;
    const int ta = w >> 1, tb = 2 * (w & 1);
    const bool upd = I != K && J != K;
    const bool fixI = q.full && K > 0 && I == K - 1, fixJ = q.full && K > 0 && J == K - 1;
    const Block& G = sm.G(q.trial);
    const int i = I * CB + 8 * ta + (lane >> 2);
    if (fixI && fixJ) {
        t.a[0] = neg(t.a[0]);
        t.a[1] = neg(t.a[1]);
    }
    if (upd) {
        // V L^T = C, tile column by tile column
        if (w < 4 || J != I) {
            const Block& L = sm.L(q.trial);
            const Block& Y = sm.Y(q.trial);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                double2 x = t.c[u];
#pragma unroll
                for (int p = 0; p < u; ++p) mma(x, neg(t.c[p]), frag(L, u, p));
                t.c[u] = solve_t(x, frag(Y, u, u));
                put(sm.V(set, w >> 2), w & 3, u, t.c[u]);
            }
        }
        __syncthreads();
        const Block& V = sm.V(set, 0);
        const Block& VJ = sm.V(set, J != I ? 1 : 0);
        // (summed apart and subtracted once: 32 roundings at A's size a panel
        // instead of one made the line searches of problems with couplings of
        // 2e5 fail)
        double2 x[2] = {};
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const double2 v = frag(V, ta, p);
            mma(x[0], v, frag(VJ, tb, p));
            mma(x[1], v, frag(VJ, tb + 1, p));
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) t.a[e] = make_double2(t.a[e].x - x[e].x, t.a[e].y - x[e].y);
    }
    if (upd || fixI || fixJ) {
        const int j = J * CB + 8 * tb + 2 * (lane & 3);
        double* o = q.A + ((unsigned)i * (unsigned)n + (unsigned)j);
        if (i < n) {
            if (j < n) o[0] = t.a[0].x;
            if (j + 1 < n) o[1] = t.a[0].y;
            if (j + 8 < n) o[8] = t.a[1].x;
            if (j + 9 < n) o[9] = t.a[1].y;
        }
    }
    if (q.full && upd && I == J) {
        // W = V Li = V G^T
        const Block& V = sm.V(set, 0);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            double2 x = make_double2(0.0, 0.0);
#pragma unroll
            for (int p = 0; p < 4; ++p)
                if (p >= tb + e) mma(x, frag(V, ta, p), frag(G, tb + e, p));
            if (i < n) {
                double* o = Wcur + (size_t)i * CB + 8 * (tb + e) + 2 * (lane & 3);
                o[0] = x.x;
                o[1] = x.y;
            }
        }
    }
    if (q.full && I == K && J == K) {
        // D^{-1} = Li^T Li = G G^T
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            double2 x = make_double2(0.0, 0.0);
#pragma unroll
            for (int p = 0; p < 4; ++p)
                if (p >= ta && p >= tb + e) mma(x, frag(G, ta, p), frag(G, tb + e, p));
            double* o = Dcur + (8 * ta + (lane >> 2)) * CB + 8 * (tb + e) + 2 * (lane & 3);
            o[0] = x.x;
            o[1] = x.y;
        }
    }
}

// The final phase of a full sweep: the fix of the last panel's row and
// column blocks, and A = -A, both triangles; with Xm, also Mout = A .* Xm (both
// triangles) and Fout's lower tiles the same.  No grid barrier.
__device__ void sweep_final(double* A, const CoopArgs& a, Smem& sm, const double* Xm, double* Mout, double* Fout)
{
    const int n = a.n;
    const int T = (n + CB - 1) / CB;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double* Wl = a.Wb + (size_t)((T + 1) & 1) * n * CB;
    const double* Dl = a.Db + (size_t)((T + 1) & 1) * CB * CB;
    const int kp0 = (T - 1) * CB;
    for (int q = blockIdx.x; q < T * (T + 1) / 2; q += gridDim.x) {
        int I, J;
        st_decode(q, &I, &J);
        const bool fixI = I == T - 1, fixJ = J == T - 1;
        Block& z = sm.V(0, 0);
        Block& m = sm.V(0, 1);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = w + CW * k;
            const int i = I * CB + r, j = J * CB + lane;
            if (i >= n || j >= n) continue;
            double v;
            if (fixI && fixJ) v = -__ldcg(Dl + (i - kp0) * CB + (j - kp0));
            else if (fixI) v = __ldcg(Wl + (size_t)j * CB + (i - kp0));
            else v = __ldcg(A + (size_t)i * n + j);
            const size_t ij = (size_t)i * n + j;
            A[ij] = -v;
            z[r][lane] = -v;
            if (Xm) {
                const double x = -v * Xm[ij];
                Mout[ij] = x;
                Fout[ij] = x;
                m[r][lane] = x;
            }
        }
        if (I == J) continue;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = w + CW * k;
            const int i = J * CB + r, j = I * CB + lane;
            if (i >= n || j >= n) continue;
            A[(size_t)i * n + j] = z[lane][r];
            if (Xm) Mout[(size_t)i * n + j] = m[lane][r];
        }
    }
}

// The panel sweep of A (n x n, lower tiles).  FULL: A becomes inv(A) (both
// triangles); otherwise only the trailing updates run, for the pivots.  With
// Xm (FULL only), the final phase also writes Mout = Fout = inv(A) .* Xm (the
// next inverse's input), saving a phase.  Sweeps run together: nt matrices,
// at most one of them full.  state[t] becomes 1 (positive definite) or -1 (a
// non-positive pivot); every CTA takes the same decisions.
struct TrialSet {
    double* A[NTRIAL];
    int full[NTRIAL];
    int state[NTRIAL];
    int nt;
    const double* Xm = nullptr;   // (of the full one)
    double *Mout = nullptr, *Fout = nullptr;
};

// In each phase every running trial's panel block is factored by its own
// warp (warp t for trial t) and the lower tiles of all running trials are
// spread over the CTAs; a trial drops out at its first non-positive pivot, a
// trailing sweep is done at its last panel's factorisation, a full sweep
// after its final phase.  Returns false when a barrier gave up.  The last
// phase has no barrier when no full sweep runs on (the caller's next fill
// goes to other matrices or follows a barrier).
__device__ __noinline__ bool msweep(TrialSet& ts, const CoopArgs& a, Smem& sm)
{
    const int n = a.n;
    const int T = (n + CB - 1) / CB;
    unsigned long long* const prof = a.prof;
    const bool rec = prof && blockIdx.x == 0 && threadIdx.x == 0;
    const int nt = ts.nt;
    unsigned run = (1u << nt) - 1u, fullm = 0u, passed = 0u;   // bit t: trial t
#pragma unroll
    for (int t = 0; t < NTRIAL; ++t) {
        if (t >= nt) continue;
        if (ts.full[t]) fullm |= 1u << t;
        if (threadIdx.x == 0) sm.A[t] = ts.A[t];
    }
    if (threadIdx.x == 0) {
        sm.Wb = a.Wb;
        sm.Db = a.Db;
    }
    __syncthreads();
    auto done = [&](bool alive) {
#pragma unroll
        for (int t = 0; t < NTRIAL; ++t)
            if (t < nt) ts.state[t] = (run >> t & 1u) ? 0 : (passed >> t & 1u) ? 1 : -1;
        return alive;
    };
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, wt = w & (NTRIAL - 1);   // (a warp's trial)
    // what a phase loads and works on, set up before the barrier in front of it
    int total = 0;
    const double* wpanel = nullptr;
    TileJob cur;
    TileAddr addr;
    int k0 = 0, b = 0;
    // tiles of a running trial in phase K
    auto tiles = [&](int K, int t) {
        const int tt = (run >> t & 1u) ? ((fullm >> t & 1u) ? T : T - K - 1) : 0;
        return tt * (tt + 1) / 2;
    };
    auto job = [&](int K, unsigned started, int q) {
        TileJob j;
        int t = 0, r = q;
#pragma unroll
        for (int u = 0; u < NTRIAL - 1; ++u) {
            const int tt = (started >> u & 1u) ? ((fullm >> u & 1u) ? T : T - K - 1) : 0, c = tt * (tt + 1) / 2;
            if (t == u && r >= c) {
                r -= c;
                ++t;
            }
        }
        j.trial = t;
        j.A = sm.A[t];
        j.full = (fullm >> t & 1u) != 0u;
        st_decode(r, &j.I, &j.J);
        if (!j.full) {
            j.I += K + 1;
            j.J += K + 1;
        }
        return j;
    };
    auto wd = [&](int K) { return sm.Wb + (K & 1 ? (unsigned)n * CB : 0u); };
    auto dd = [&](int K) { return sm.Db + (K & 1 ? CB * CB : 0); };
    auto setup = [&](int K) {
        k0 = K * CB;
        b = n - k0 < CB ? n - k0 : CB;
        total = 0;
#pragma unroll
        for (int t = 0; t < NTRIAL; ++t) total += tiles(K, t);
        if (run >> wt & 1u)
            wpanel = sm.A[wt] + ((unsigned)(k0 + (lane >> 2)) * (unsigned)n + (unsigned)(k0 + 2 * (lane & 3)));
        if ((int)blockIdx.x < total) {
            cur = job(K, run, blockIdx.x);
            addr = tile_addr(cur, n, K, k0, b, wd(K + 1), dd(K + 1));
        }
    };
    setup(0);
    for (int K = 0; K < T; ++K) {
        unsigned long long tp = rec ? global_ns() : 0ull;
        const unsigned started = run;
        const bool wrun = (run >> wt & 1u) != 0u, wfull = (fullm >> wt & 1u) != 0u;
        // the panel blocks and the CTA's first tile, in one round trip
        PanelTiles pf;
        if (wrun && w < NTRIAL) panel_load(wpanel, n, b, pf);
        TileLoad load;
        int q = blockIdx.x;
        if (q < total) tile_load(addr, load);
        if (rec && wrun) {   // (a use of the last pair, so that the clock is read after it)
            *(volatile double*)sm.red = pf.d[3][3].y;
            prof[COOP_PROF_PF_LOAD] += global_ns() - tp;
        }
        if (wrun && w < NTRIAL) panel_chain(pf, wt, wfull, sm);
        if (wrun && w >= NTRIAL && wfull) panel_help(wt, sm);
        __syncthreads();
#pragma unroll
        for (int t = 0; t < NTRIAL; ++t) {
            if (!(started >> t & 1u)) continue;
            if (!sm.pd[t]) {
                run &= ~(1u << t);
            } else if (!(fullm >> t & 1u) && K == T - 1) {
                run &= ~(1u << t);
                passed |= 1u << t;
            }
        }
        if (rec) {
            const unsigned long long tn = global_ns();
            prof[COOP_PROF_FACTOR] += tn - tp;
            prof[COOP_PROF_PHASES] += 1;
            tp = tn;
        }
        if (!run) return done(true);
        int set = 0;
        while (q < total) {
            q += gridDim.x;
            const TileJob now = cur;
            TileLoad here = load;
            if (q < total) {
                cur = job(K, started, q);
                tile_load(tile_addr(cur, n, K, k0, b, wd(K + 1), dd(K + 1)), load);
            }
            if (!(run >> now.trial & 1u)) continue;
            tile_step(now, n, K, here, wd(K), dd(K), set, sm);
            if (now.I != K && now.J != K) set ^= 1;   // (a tile with a barrier)
        }
        if (prof) __syncthreads();
        if (rec) prof[COOP_PROF_TILES] += global_ns() - tp;
        if (K + 1 < T) setup(K + 1);
        if (!grid_sync(sm.bar, sm, prof)) return done(false);
    }
    const unsigned fin = run & fullm;   // (at most one)
    if (fin) {
        sweep_final(sm.A[__ffs(fin) - 1], a, sm, ts.Xm, ts.Mout, ts.Fout);
        if (!grid_sync(sm.bar, sm, prof)) return done(false);
        run &= ~fin;
        passed |= fin;
    }
    return done(true);
}

// One full sweep: 1 (positive definite), 0 (a non-positive pivot) or -1 (a
// barrier gave up).
__device__ int sweep(double* A, const CoopArgs& a, Smem& sm, const double* Xm = nullptr, double* Mout = nullptr,
                     double* Fout = nullptr)
{
    TrialSet ts;
#pragma unroll
    for (int t = 0; t < NTRIAL; ++t) {
        ts.A[t] = A;
        ts.full[t] = 1;
    }
    ts.nt = 1;
    ts.Xm = Xm;
    ts.Mout = Mout;
    ts.Fout = Fout;
    if (!msweep(ts, a, sm)) return -1;
    return ts.state[0] == 1 ? 1 : 0;
}

// The lower tiles of a sweep's matrix: f(i, j) for i, j < n, by the grid in
// strips of eight rows.
template <class F>
__device__ __forceinline__ void lower_fill(int n, F f)
{
    const int T = (n + CB - 1) / CB;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int u = blockIdx.x; u < 2 * T * (T + 1); u += gridDim.x) {
        int I, J;
        st_decode(u >> 2, &I, &J);
        const int i = I * CB + CW * (u & 3) + w, j = J * CB + lane;
        if (i < n && j < n) f(i, j);
    }
}

// ---- products ------------------------------------------------------------------

// A thread's four entries of a block: rows warp + 8 j, column lane.
__device__ __forceinline__ void block_store(Block& m, int j, double v) { m[(threadIdx.x >> 5) + CW * j][threadIdx.x & 31] = v; }

// out = sym(Zi (Diag(-a) X + Diag(-b) Y) + e1 E1 + e2 E2) (b, Y, E2 may be
// null; the row scales enter negated, -(a_k X_kc) being exactly
// (-a_k) X_kc; X, Y, E1, E2 symmetric): the owner of the tile pair (I, J),
// (J, I) forms both products on the tensor instruction (a warp E tiles of
// P_IJ and their mirrors of P_JI) and writes the symmetric part.  k in chunks
// of 32 through two sets of shared-memory operands, the next chunk's loads in
// flight during a chunk's products.  E = 1: a CTA takes half of a pair's rows
// of I, for grids of as many CTAs as halves (at n = 343 the 66 pairs would leave
// half of the chip idle); the sums are the same.
template <int E>
__device__ __noinline__ void gemm_sym_e(const double* Zi, const double* av, const double* X, const double* bv,
                                        const double* Y, double e1, const double* E1, double e2, const double* E2,
                                        int n, double* out, Smem& sm)
{
    const int T = (n + CB - 1) / CB;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int r = lane >> 2, c = lane & 3;
    constexpr int UNITS = E == 2 ? 1 : 2;
    for (int u = blockIdx.x; u < UNITS * (T * (T + 1) / 2); u += gridDim.x) {
        int I, J;
        st_decode(u / UNITS, &I, &J);
        const int hh = u % UNITS;
        const int ta = E == 2 ? w >> 1 : 2 * hh + (w >> 2), tb = E == 2 ? 2 * (w & 1) : w & 3;
        const bool off = I != J;
        double z[2][4], x[2][4], y[2][4], sa, sb;
        auto load = [&](int k0) {
            const int k = k0 + lane;
            sa = k < n ? -av[k] : 0.0;
            sb = bv && k < n ? -bv[k] : 0.0;
#pragma unroll
            for (int side = 0; side < 2; ++side)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int i = (side ? J : I) * CB + w + CW * j;
                    const bool in = i < n && k < n && (side ? off : !(E == 1 && off && (j >> 1) != hh));
                    const size_t o = (size_t)i * n + k;
                    z[side][j] = in ? __ldcg(Zi + o) : 0.0;
                    x[side][j] = in ? __ldcg(X + o) : 0.0;
                    y[side][j] = bv && in ? __ldcg(Y + o) : 0.0;
                }
        };
        auto store = [&](int set) {
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                if (side && !off) continue;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    double h = sa * x[side][j];
                    if (bv) h = fma(sb, y[side][j], h);
                    block_store(sm.b[4 * set + side], j, z[side][j]);
                    block_store(sm.b[4 * set + 2 + side], j, h);
                }
            }
        };
        double2 p[E] = {}, pt[E] = {};   // P_IJ (ta, tb + e), P_JI (tb + e, ta)
        load(0);
        store(0);
        __syncthreads();
        int set = 0;
        for (int k0 = 0; k0 < n; k0 += CB, set ^= 1) {
            const bool more = k0 + CB < n;
            if (more) load(k0 + CB);
            const Block& zi = sm.b[4 * set];
            const Block& zj = sm.b[4 * set + (off ? 1 : 0)];
            const Block& hi = sm.b[4 * set + 2];
            const Block& hj = sm.b[4 * set + 2 + (off ? 1 : 0)];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double2 f = frag(zi, ta, q), g = frag(hi, ta, q);
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    mma(p[e], f, frag(hj, tb + e, q));
                    mma(pt[e], frag(zj, tb + e, q), g);
                }
            }
            if (more) store(set ^ 1);
            __syncthreads();
        }
        double* scratch = &sm.V(0, 0)[0][0] + 64 * w;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            // P_JI's tile transposed through the warp's scratch
            scratch[st_elem(2 * c, r)] = pt[e].x;
            scratch[st_elem(2 * c + 1, r)] = pt[e].y;
            __syncwarp();
            const double2 m = st_ld(scratch + st_pair(r, c));
            __syncwarp();
            const int i = I * CB + 8 * ta + r;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int j = J * CB + 8 * (tb + e) + 2 * c + k;
                if (i >= n || j >= n) continue;
                const size_t ij = (size_t)i * n + j, ji = (size_t)j * n + i;
                double vij = (k ? p[e].y : p[e].x) + e1 * E1[ij];
                double vji = (k ? m.y : m.x) + e1 * E1[ij];
                if (E2) {
                    vij += e2 * E2[ij];
                    vji += e2 * E2[ij];
                }
                const double v = i == j ? vij : 0.5 * (vij + vji);
                out[ij] = v;
                if (off) out[ji] = v;
            }
        }
    }
}

__device__ __forceinline__ void gemm_sym(const double* Zi, const double* av, const double* X, const double* bv,
                                         const double* Y, double e1, const double* E1, double e2, const double* E2,
                                         int n, double* out, Smem& sm)
{
    const int T = (n + CB - 1) / CB;
    if (T * (T + 1) <= (int)gridDim.x) gemm_sym_e<1>(Zi, av, X, bv, Y, e1, E1, e2, E2, n, out, sm);
    else gemm_sym_e<2>(Zi, av, X, bv, Y, e1, E1, e2, E2, n, out, sm);
}

// sum_c a(c) b(c) over a row, by a warp: the lanes' loads of 12 steps are in
// flight together (three steps at a time took a round trip to L2 each).
template <class FA, class FB>
__device__ __forceinline__ double row_dot(int n, FA fa, FB fb)
{
    const int lane = threadIdx.x & 31;
    double acc = 0.0;
    for (int c0 = lane; c0 < n; c0 += 32 * 12) {
        double x[12], y[12];
#pragma unroll
        for (int q = 0; q < 12; ++q) {
            const int c = c0 + 32 * q;
            x[q] = c < n ? fa(c) : 0.0;
            y[q] = c < n ? fb(c) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 12; ++q) acc = fma(x[q], y[q], acc);
    }
    return warp_sum(acc);
}

// One warp per row i (the grid's warps in turn): out_i = sum_c F(c, i) v_c
// (F symmetric; v null: v = -e).
__device__ void warp_rows_matvec(const double* F, int n, const double* v, double* out)
{
    const int lane = threadIdx.x & 31;
    const int nw = gridDim.x * CW;
    for (int i = blockIdx.x * CW + (threadIdx.x >> 5); i < n; i += nw) {
        const double* col = F + (size_t)i * n;
        const double acc = row_dot(n, [=](int c) { return __ldcg(col + c); }, [=](int c) { return v ? __ldcg(v + c) : -1.0; });
        if (lane == 0) out[i] = acc;
    }
}

// r_i = b_i - sum_c M(c, i) x_c (b null: -1)
__device__ void warp_rows_resid(const double* M, int n, const double* b, const double* x, double* r)
{
    const int lane = threadIdx.x & 31;
    const int nw = gridDim.x * CW;
    for (int i = blockIdx.x * CW + (threadIdx.x >> 5); i < n; i += nw) {
        const double* col = M + (size_t)i * n;
        const double acc = row_dot(n, [=](int c) { return __ldcg(col + c); }, [=](int c) { return __ldcg(x + c); });
        if (lane == 0) r[i] = (b ? b[i] : -1.0) - acc;
    }
}

// t = F r; x += t (row i of both by the same warp)
__device__ void warp_rows_refine(const double* F, int n, const double* r, double* t, double* x)
{
    const int lane = threadIdx.x & 31;
    const int nw = gridDim.x * CW;
    for (int i = blockIdx.x * CW + (threadIdx.x >> 5); i < n; i += nw) {
        const double* col = F + (size_t)i * n;
        const double acc = row_dot(n, [=](int c) { return __ldcg(col + c); }, [=](int c) { return __ldcg(r + c); });
        if (lane == 0) {
            t[i] = acc;
            x[i] = x[i] + acc;
        }
    }
}

// rhs_i = mu Zi_ii - sum_c Zi_ic dX1_ic dy1_c (columns i by symmetry)
__device__ void warp_rows_rhs(const double* Zi, const double* dX1, const double* dy1, double mu, int n, double* rhs)
{
    const int lane = threadIdx.x & 31;
    const int nw = gridDim.x * CW;
    for (int i = blockIdx.x * CW + (threadIdx.x >> 5); i < n; i += nw) {
        const size_t o = (size_t)i * n;
        const double acc = row_dot(n, [=](int c) { return __ldcg(Zi + o + c) * __ldcg(dX1 + o + c); },
                                   [=](int c) { return __ldcg(dy1 + c); });
        if (lane == 0) rhs[i] = mu * Zi[o + i] - acc;
    }
}

// x = M^{-1} b (b null: -e): x = F b, then one refinement step.  Three
// phases; returns false when a barrier gave up.
__device__ bool solve(const CoopArgs& a, const double* F, const double* b, double* x, Smem& sm)
{
    warp_rows_matvec(F, a.n, b, x);
    if (!grid_sync(a.bar, sm, a.prof)) return false;
    warp_rows_resid(a.M, a.n, b, x, a.r);
    if (!grid_sync(a.bar, sm, a.prof)) return false;
    warp_rows_refine(F, a.n, a.r, a.t, x);
    return grid_sync(a.bar, sm, a.prof);
}

__global__ void __launch_bounds__(CT, 1) ipm_coop_kernel(const __grid_constant__ CoopArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
    const int n = a.n;
    const size_t nn = (size_t)n * n;
    const size_t gtid = (size_t)blockIdx.x * CT + threadIdx.x, gstride = (size_t)gridDim.x * CT;
    const double* __restrict__ L = a.L;
    double* X = a.Xbase + (a.xslot ? (size_t)(*a.xslot) * nn : 0);
    const unsigned long long t_call = a.prof && blockIdx.x == 0 ? global_ns() : 0ull;
    if (threadIdx.x == 0) {
        sm.epoch = 0u;
        sm.bar = a.bar;
    }

    // ---- initial point (src/ipm_mc_pk.c:65-99): y_c = sum_r |L_rc| + 1.1,
    // zd = y - diag(L), X = I; psi = trace(L), mu = sum(zd) / 2n, phi = sum(y)
    const int parts = sum_parts(n);
    const size_t vstride = (size_t)parts * CT;
    for (int v = blockIdx.x; v < parts; v += gridDim.x) {
        double s0 = 0.0, s1 = 0.0, s2 = 0.0;
        for (int c = v * CW + (threadIdx.x >> 5); c < n; c += parts * CW) {
            const double* Lc = L + (size_t)c * n;
            const double acc = row_dot(n, [=](int q) { return fabs(Lc[q]); }, [](int) { return 1.0; });
            if ((threadIdx.x & 31) == 0) {
                const double yc = acc + 1.1;
                const double zc = yc - Lc[c];
                a.y[c] = yc;
                a.zd[c] = zc;
                s0 += Lc[c];
                s1 += zc;
                s2 += yc;
            }
        }
        block_partials(s0, s1, s2, 0.0, sm, a.part, v);
    }
    for (size_t e = gtid; e < nn; e += gstride) X[e] = (e % n == e / n) ? 1.0 : 0.0;
    bool alive = grid_sync(a.bar, sm, a.prof);
    grid_totals(a.part, parts, sm);
    double psi = sm.tot[0];
    double mu = sm.tot[1] / (2.0 * n);
    double phi = sm.tot[2];
    double gap = fabs(phi - psi);
    int iter = 0, ls_total = 0, status = IPM_OK;
    // When the dual line search's first trial (ad = 1) passes, its full sweep
    // leaves inv(Z) of the new point in Zi (the same matrix, with the same
    // arithmetic, as this iteration's own sweep would), and the next
    // iteration only forms M = F = Zi .* X.
    double* const Zi = a.Zi;
    double* const F = a.F;
    bool have_zi = false;

    while (alive && gap > 1e-2) {
        if (++iter > IPM_MAX_ITERS) {
            status = IPM_MAXITER;
            break;
        }
        int pd = 1;
        if (!have_zi) {
            // Zi = inv(Z), Z = Diag(zd) - L off the diagonal
            lower_fill(n, [&](int i, int j) {
                Zi[(size_t)i * n + j] = i == j ? a.zd[i] : -L[i + (size_t)j * n];
            });
            if (!(alive = grid_sync(a.bar, sm, a.prof))) break;
            // (its last phase also writes M = Zi .* X and F = M)
            pd = sweep(Zi, a, sm, X, a.M, F);
            if (pd < 0) {
                alive = false;
                break;
            }
            if (!pd) {
                status = IPM_Z_NOT_PD;
                break;
            }
        } else {
            for (size_t e = gtid; e < nn; e += gstride) {
                const double m = Zi[e] * X[e];
                a.M[e] = m;
                F[e] = m;
            }
            if (!(alive = grid_sync(a.bar, sm, a.prof))) break;
        }
        have_zi = false;
        // F = inv(M); dy1 = F (-e)
        pd = sweep(F, a, sm);
        if (pd < 0) {
            alive = false;
            break;
        }
        if (!pd) {
            status = IPM_M_NOT_PD;
            break;
        }
        if (!(alive = solve(a, F, nullptr, a.dy1, sm))) break;
        // dX1 = sym(Zi (-Diag(dy1) X) - X)
        unsigned long long tg = a.prof && blockIdx.x == 0 ? global_ns() : 0ull;
        gemm_sym(Zi, a.dy1, X, nullptr, nullptr, -1.0, X, 0.0, nullptr, n, a.dX1, sm);
        if (a.prof) __syncthreads();
        if (a.prof && blockIdx.x == 0 && threadIdx.x == 0) a.prof[COOP_PROF_GEMM] += global_ns() - tg;
        if (!(alive = grid_sync(a.bar, sm, a.prof))) break;
        // corrector: rhs = mu diag(Zi) - (Zi .* dX1) dy1; dy2 = F rhs
        warp_rows_rhs(Zi, a.dX1, a.dy1, mu, n, a.dy);
        if (!(alive = grid_sync(a.bar, sm, a.prof))) break;
        if (!(alive = solve(a, F, a.dy, a.dy2, sm))) break;
        // dX = sym(Zi (-Diag(dy2) X - Diag(dy1) dX1) + mu Zi + dX1)
        tg = a.prof && blockIdx.x == 0 ? global_ns() : 0ull;
        gemm_sym(Zi, a.dy2, X, a.dy1, a.dX1, 1.0, a.dX1, mu, Zi, n, a.dX, sm);
        if (a.prof) __syncthreads();
        if (a.prof && blockIdx.x == 0 && threadIdx.x == 0) a.prof[COOP_PROF_GEMM] += global_ns() - tg;
        if (!(alive = grid_sync(a.bar, sm, a.prof))) break;

        // line searches (src/ipm_mc_pk.c:281-309): the primal search
        // (X + ap dX positive definite) and the dual search (Z + ad Diag(dy)
        // positive definite) each try 1, 0.8, 0.64, ... and keep the first
        // step that passes.  Here a round sweeps the next two trials of each
        // unfinished search together (primal in T, T2; dual in Zi, F, all free
        // by now); every trial's pivots are those of its own sweep, so the
        // steps kept are the one-at-a-time searches' steps.  The dual's first
        // trial (ad = 1, the step itself when it passes) is a full sweep whose
        // inverse starts the next iteration.
        double ap = 1.0, ad = 1.0;   // the next trial step of each search
        int pi = 0, di = 0;          // its trial index
        int pres = 0, dres = 0;      // 1 found, -1 gave up
        double ap_ok = 1.0, ad_ok = 1.0;
        int rounds = 0;
        while (pres == 0 || dres == 0) {
            // a CTA may still read the last round's panel blocks
            if (rounds++ > 0 && !(alive = grid_sync(a.bar, sm, a.prof))) break;
            TrialSet ts;
            double alpha[NTRIAL];
            int dual[NTRIAL];
            ts.nt = 0;
            auto add = [&](double* buf, double al, bool du, bool full) {
                ts.A[ts.nt] = buf;
                ts.full[ts.nt] = full ? 1 : 0;
                alpha[ts.nt] = al;
                dual[ts.nt] = du ? 1 : 0;
                ++ts.nt;
            };
            const int np0 = ts.nt;
            if (pres == 0) {
                add(a.T, ap, false, false);
                if (pi + 1 < IPM_MAX_TRIALS) add(a.T2, ap * 0.8, false, false);
            }
            const int nd0 = ts.nt;
            if (dres == 0) {
                add(Zi, ad, true, di == 0);
                if (di + 1 < IPM_MAX_TRIALS) add(F, ad * 0.8, true, false);
            }
            // (dy_i = dy1_i + dy2_i)
            lower_fill(n, [&](int i, int j) {
                const size_t e = (size_t)i * n + j;
                for (int t = 0; t < ts.nt; ++t)
                    ts.A[t][e] = dual[t] ? (i == j ? fma(alpha[t], a.dy1[i] + a.dy2[i], a.zd[i]) : -L[i + (size_t)j * n])
                                         : fma(alpha[t], a.dX[e], X[e]);
            });
            if (!(alive = grid_sync(a.bar, sm, a.prof))) break;
            if (!(alive = msweep(ts, a, sm))) break;
            // each search: the first of its trials that passed, in order
            auto decide = [&](int t0, int t1, int& res, int& idx, double& step, double& ok_step) {
                for (int t = t0; t < t1; ++t) {
                    if (ts.state[t] == 1) {
                        res = 1;
                        ok_step = alpha[t];
                        ls_total += idx + (t - t0) + 1;
                        return t - t0;
                    }
                }
                idx += t1 - t0;
                step = alpha[t1 - 1] * 0.8;
                if (idx >= IPM_MAX_TRIALS) res = -1;
                return -1;
            };
            if (pres == 0) decide(np0, nd0, pres, pi, ap, ap_ok);
            if (dres == 0) {
                const bool first = di == 0;
                if (decide(nd0, ts.nt, dres, di, ad, ad_ok) == 0 && first) have_zi = true;
            }
            if (pres < 0 || dres < 0) break;
        }
        if (!alive) break;
        if (pres < 0 || dres < 0) {
            status = IPM_LINESEARCH;
            break;
        }
        ap = ap_ok;
        ad = ad_ok;
        if (ap < 1.0) ap *= 0.95;
        if (ad < 1.0) ad *= 0.95;

        // update (src/ipm_mc_pk.c:313-334): X += ap dX, y += ad dy,
        // zd += ad dy (dy = dy1 + dy2), and the sums zx = <Z, X>, lx = <L, X>,
        // sum(y) of the new point.  The diagonal of X goes with the vectors
        // (the thread that moves zd_i also moves X_ii).
        for (int v = blockIdx.x; v < parts; v += gridDim.x) {
            const size_t vt = (size_t)v * CT + threadIdx.x;
            double zx = 0.0, lx = 0.0, ys = 0.0;
            int i = (int)(vt % n), j = (int)(vt / n);
            const int di = (int)(vstride % n), dj = (int)(vstride / n);
            for (size_t e = vt; e < nn; e += vstride, i += di, j += dj) {
                if (i >= n) {
                    i -= n;
                    ++j;
                }
                if (i == j) continue;
                const double xv = fma(ap, a.dX[e], X[e]);
                X[e] = xv;
                const double lv = L[e];
                lx = fma(lv, xv, lx);
                zx = fma(-lv, xv, zx);
            }
            for (size_t c = vt; c < (size_t)n; c += vstride) {
                const size_t e = c * n + c;
                const double xv = fma(ap, a.dX[e], X[e]);
                X[e] = xv;
                const double dyc = a.dy1[c] + a.dy2[c];
                const double yv = fma(ad, dyc, a.y[c]);
                const double zv = fma(ad, dyc, a.zd[c]);
                a.y[c] = yv;
                a.zd[c] = zv;
                lx = fma(L[e], xv, lx);
                zx = fma(zv, xv, zx);
                ys += yv;
            }
            block_partials(zx, lx, ys, 0.0, sm, a.part, v);
        }
        if (!(alive = grid_sync(a.bar, sm, a.prof))) break;
        grid_totals(a.part, parts, sm);
        mu = sm.tot[0] / (2.0 * n);
        if (ap + ad > 1.6) mu *= 0.5;
        if (ap + ad > 1.9) mu *= 0.2;
        phi = sm.tot[2];
        psi = sm.tot[1];
        gap = fabs(phi - psi);
        // (the partials are rewritten only after the next iteration's
        // barriers, so no barrier is needed here)
    }
    if (!alive) status = IPM_SYNC;
    // (y's last writes came before the update's barrier)
    if (a.yout)
        for (size_t c = gtid; c < (size_t)n; c += gstride) a.yout[c] = a.y[c];
    if (a.prof && blockIdx.x == 0 && threadIdx.x == 0) a.prof[COOP_PROF_TOTAL] += global_ns() - t_call;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out[0] = phi;
        a.out[1] = (double)iter;
        a.out[2] = (double)status;
        a.out[3] = psi;
        if (a.stats) {
            const double n3 = (double)n * n * n;
            atomicAdd(&a.stats[0], iter * n3);
            atomicAdd(&a.stats[1], 1.0);
            atomicAdd(&a.stats[2], (double)iter);
            atomicAdd(&a.stats[3], (double)ls_total);
        }
    }
}

struct CoopConfig {
    int grid = 0;
    size_t smem = 0;
};

// Per-part timing of CTA 0 (off unless bqb_ipm_coop_profile_enable(1)).
std::atomic<int> g_coop_prof_on{0};
DevBuf<unsigned long long> g_coop_prof;
std::mutex g_coop_prof_mu;

unsigned long long* coop_prof_device()
{
    if (!g_coop_prof_on.load()) return nullptr;
    std::lock_guard<std::mutex> lock(g_coop_prof_mu);
    if (!g_coop_prof.p) {
        g_coop_prof.ensure(COOP_PROF_WORDS);
        BQB_CUDA(cudaMemset(g_coop_prof.p, 0, COOP_PROF_WORDS * sizeof(unsigned long long)));
    }
    return g_coop_prof.p;
}

// The per-size schedule: the grid (CTAs) to use for T = ceil(n / 32) tiles
// per dimension, filled by the autotuner (bqb_ipm_autotune) or set by hand
// (bqb_ipm_schedule_set); sizes without an entry use coop_config's rule.
std::mutex g_sched_mu;
std::map<int, int> g_sched;

}  // namespace

// Engines bounding nodes above IPM_REG_NMAX right now (node.cu counts them):
// each multi-CTA IPM launch then takes its share of the co-resident CTAs, so
// the IPMs of concurrent engines run side by side instead of one after
// another.  The IPM's result does not depend on its grid.
std::atomic<int> g_large_share{0};

namespace {

// CTAs for T tiles per dimension: one for half a pair of 32 x 32 tiles, at most
// max_blocks.  A call alone is faster with the whole chip (the line searches sweep
// up to four matrices, and fills and products have more parts than tiles), by
// 38 of 1557 us at n = 136, 58 of 1917 at 160, 56 of 2429 at 224, 35 of 2853 at 288,
// nothing from 321 on; but a cooperative launch waits until all its CTAs find a
// free SM, so beside other engines' one-CTA kernels the whole chip loses: eight
// nodes of n = 130 on four engines take 59 ms so and 89 with it, of n = 200 53.8
// and 54.7.
int coop_default_grid(int T, int max_blocks)
{
    return T * (T + 1) < max_blocks ? T * (T + 1) : max_blocks;
}

// Grid size for n: the schedule's entry for its tile count, else the default; at
// most as many as can be co-resident (one per SM at this register count),
// divided by the number of engines bounding large nodes at the time.
CoopConfig coop_config(int n)
{
    static int max_blocks = -1;
    static std::atomic<int> ready{0};
    CoopConfig c;
    c.smem = sizeof(Smem);
    BQB_SMEM_LIMIT(ipm_coop_kernel, c.smem);   // per device (cached)
    if (!ready.load()) {
        int per_sm = 0;
        BQB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ipm_coop_kernel, CT, c.smem));
        max_blocks = per_sm * rt().num_sms;
        ready.store(1);
    }
    const int T = (n + CB - 1) / CB;
    int g = coop_default_grid(T, max_blocks);
    {
        std::lock_guard<std::mutex> lock(g_sched_mu);
        auto it = g_sched.find(T);
        if (it != g_sched.end()) g = it->second;
    }
    const int share = g_large_share.load();
    const int cap = share > 1 ? max_blocks / share : max_blocks;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    c.grid = g;
    return c;
}

}  // namespace

size_t ipm_large_ws_doubles(int n)
{
    const size_t nn = (size_t)n * n;
    return 7 * nn + 2 * (size_t)n * CB + 2 * (size_t)CB * CB + 8 * (size_t)n + 4 * 1024 + 16;
}

// ipm_mc_pk for n > IPM_REG_NMAX: one cooperative launch on stream s, no
// host synchronisation.  xslot (optional, device): write X into
// Xbase + (*xslot) * n * n.  Results in dout[0..3] (phi, iterations, status,
// psi); status IPM_SYNC when a grid barrier gave up waiting.
void ipm_large(DevBuf<double>& wsbuf, const double* L, double* Xbase, int n, double* dout, cudaStream_t s,
               const int* xslot, double* yout)
{
    const size_t nn = (size_t)n * n;
    double* p = wsbuf.ensure(ipm_large_ws_doubles(n));
    CoopArgs a;
    a.L = L;
    a.Xbase = Xbase;
    a.xslot = xslot;
    a.out = dout;
    a.stats = ipm_stats_device();
    a.prof = coop_prof_device();
    a.yout = yout;
    a.n = n;
    a.Zi = p;
    a.F = a.Zi + nn;
    a.M = a.F + nn;
    a.T = a.M + nn;
    a.T2 = a.T + nn;
    a.dX = a.T2 + nn;
    a.dX1 = a.dX + nn;
    a.Wb = a.dX1 + nn;
    a.Db = a.Wb + 2 * (size_t)n * CB;
    a.y = a.Db + 2 * (size_t)CB * CB;
    a.zd = a.y + n;
    a.dy = a.zd + n;
    a.dy1 = a.dy + n;
    a.dy2 = a.dy1 + n;
    a.r = a.dy2 + n;
    a.t = a.r + n;
    a.part = a.t + n;
    a.bar = reinterpret_cast<unsigned*>(a.part + 4 * 1024);
    const CoopConfig c = coop_config(n);
    BQB_CUDA(cudaMemsetAsync(a.bar, 0, 4 * sizeof(unsigned), s));
    void* args[] = {&a};
    BQB_CUDA(cudaLaunchCooperativeKernel((const void*)ipm_coop_kernel, dim3(c.grid), dim3(CT), args, c.smem, s));
    BQB_COUNT_LAUNCH();
    check_launch("ipm_large");
}

}  // namespace bqb

using namespace bqb;

// Use `grid` CTAs for the multi-CTA IPM of every n with the same tile count
// as n (grid <= 0 removes the entry).  No reference counterpart.
BQB_API void bqb_ipm_schedule_set(int n, int grid)
{
    if (n <= 0) return;
    const int T = (n + CB - 1) / CB;
    std::lock_guard<std::mutex> lock(g_sched_mu);
    if (grid > 0) g_sched[T] = grid;
    else g_sched.erase(T);
}

// Autotune the multi-CTA IPM's grid for size n (> 128): time `reps` calls (at
// least three) for each candidate (the default grid, T^2 CTAs, T = ceil(n / 32), a
// half, a quarter and an eighth of that, and the SM count) on a seeded problem of
// that size (the Laplacian of a random +-1 graph, as the B&B's subproblems are),
// keep the one with the fastest call in the schedule.  best_grid / best_ms (may
// be null) receive the choice and that time.  Calls are timed alone: beside other
// engines a smaller grid may be better (coop_default_grid).  Returns 0, 1 for n <=
// 128.  No reference counterpart.
BQB_API int bqb_ipm_autotune(int n, int reps, int* best_grid, double* best_ms)
{
    if (n <= 128) return 1;
    if (reps < 3) reps = 3;
    Runtime& R = rt();
    cudaStream_t s = R.stream;
    const size_t nn = (size_t)n * n;
    std::vector<double> L(nn, 0.0);
    unsigned long long z = 0x5eedull + (unsigned long long)n;
    auto next = [&]() {
        z += 0x9E3779B97F4A7C15ull;
        unsigned long long x = z;
        x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
        x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
        return x ^ (x >> 31);
    };
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < i; ++j) {
            const unsigned long long r = next();
            if (r & 1) continue;                       // edge with probability 1/2
            const double w = (r & 2) ? 1.0 : -1.0;     // weight +-1
            L[i + (size_t)j * n] = L[j + (size_t)i * n] = -w;
            L[i + (size_t)i * n] += w;
            L[j + (size_t)j * n] += w;
        }
    for (double& v : L) v *= 0.25;
    DevBuf<double> dL, dX, ws, out;
    BQB_CUDA(cudaMemcpy(dL.ensure(nn), L.data(), nn * sizeof(double), cudaMemcpyHostToDevice));
    dX.ensure(nn);
    out.ensure(4);
    const int T = (n + CB - 1) / CB;
    const int def = coop_default_grid(T, R.num_sms);
    std::vector<int> cand = {def, T * T, (T * T + 1) / 2, (T * T + 3) / 4, (T * T + 7) / 8, R.num_sms};
    cudaEvent_t e0, e1;
    BQB_CUDA(cudaEventCreate(&e0));
    BQB_CUDA(cudaEventCreate(&e1));
    int bg = def;
    double bms = 1e300;
    for (int g : cand) {
        if (g < 1) continue;
        bqb_ipm_schedule_set(n, g);
        ipm_large(ws, dL.p, dX.p, n, out.p, s, nullptr);   // warm-up
        float ms = 1e30f;
        for (int r = 0; r < reps; ++r) {
            float t = 0.f;
            BQB_CUDA(cudaEventRecord(e0, s));
            ipm_large(ws, dL.p, dX.p, n, out.p, s, nullptr);
            BQB_CUDA(cudaEventRecord(e1, s));
            BQB_CUDA(cudaEventSynchronize(e1));
            BQB_CUDA(cudaEventElapsedTime(&t, e0, e1));
            ms = t < ms ? t : ms;
        }
        double h[4];
        BQB_CUDA(cudaMemcpy(h, out.p, sizeof h, cudaMemcpyDeviceToHost));
        if ((int)h[2] == IPM_OK && ms < bms) {
            bms = ms;
            bg = g;
        }
    }
    BQB_CUDA(cudaEventDestroy(e0));
    BQB_CUDA(cudaEventDestroy(e1));
    // (DevBuf does not free: the tuning problem's buffers go here)
    for (double* q : {dL.p, dX.p, ws.p, out.p})
        if (q) BQB_CUDA(cudaFree(q));
    bqb_ipm_schedule_set(n, bg);   // the fastest candidate stays in the schedule
    if (best_grid) *best_grid = bg;
    if (best_ms) *best_ms = bms;
    return 0;
}

// Time the multi-CTA IPM spends per part (its CTA 0, summed over calls since
// the last reset): enable (on != 0) or disable the timing; out[8] = {barrier
// waits, panel factorisations, tile updates, products, whole calls (ms),
// grid barriers, sweep phases, the part of the panel factorisations until the
// panel block has come (ms)};
// reset != 0 zeroes after reading.  For
// profiling; no reference counterpart.
BQB_API void bqb_ipm_coop_profile_enable(int on) { g_coop_prof_on.store(on != 0); }

BQB_API void bqb_ipm_coop_profile(double* out, int reset)
{
    unsigned long long h[COOP_PROF_WORDS] = {};
    std::lock_guard<std::mutex> lock(g_coop_prof_mu);
    if (g_coop_prof.p) {
        BQB_CUDA(cudaMemcpy(h, g_coop_prof.p, sizeof h, cudaMemcpyDeviceToHost));
        if (reset) BQB_CUDA(cudaMemset(g_coop_prof.p, 0, sizeof h));
    }
    for (int i = 0; i < COOP_PROF_WORDS; ++i)
        out[i] = (i < COOP_PROF_BARRIERS || i == COOP_PROF_PF_LOAD) ? 1e-6 * (double)h[i] : (double)h[i];
}
