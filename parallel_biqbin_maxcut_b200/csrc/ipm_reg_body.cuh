// IPM body for n <= 128 (one CTA of IPM_THREADS threads per problem), shared
// by the IPM kernels (ipm.cu) and the fused node kernel (nodek.cu) so both run
// the same arithmetic.
#pragma once
#include <math.h>

#include "ipm.cuh"
#include "reg_linalg.cuh"
#include "sym_tiles.cuh"

namespace bqb {

// ---------------------------------------------------------------------------
// The matrices are 8 x 8 tiles on the SM (sym_tiles.cuh): X and dX1 / dX
// symmetric, Zi = inv(Z) with both triangles.  An iteration is at most two
// inverses, two products and the line searches' factorisations:
//  * inverses: st_inverse, eight columns a panel (n > 120, where its sixteen
//    tile rows and the chain warp would need a warp more than the CTA has:
//    the sweep by single columns, rm_spd_inverse);
//  * both solves with M = Zi .* X are products with F = inv(M);
//  * products on the tensor instruction, both of a pair of tiles (I, J), (J, I)
//    in one warp, which symmetrises them;
//  * line searches need only "positive definite or not": st_posdef.  The dual
//    search's first trial (step 1) is an inverse: when it passes, it is the
//    next iteration's Zi.
// Every sum keeps the order of the step-by-step method it replaced (single
// columns, a CTA barrier, a reciprocal square root and a rank-1 update of a
// padded 128 x 128 matrix each), so results are the same bits: products run
// over ascending k from zero, row sums over lanes and then a shuffle tree.
// An iteration, before and now: 84 -> 38 us at n = 24, 202 -> 82 at n = 60,
// 365 -> 182 at n = 100, 461 -> 248 at n = 120; n = 121 .. 128, whose inverses
// stay the single-column sweep, 483 -> 354.  What bounds it now is the
// eliminations' chain from one diagonal block to the next: at n = 100 the two
// inverses and the searches' trials are two thirds of the time.
//
// Shared memory (doubles, from st_smem): red[ST_RED], the vectors y, zd, dy,
// dy1, rhs (8 T each), the eliminations' buffers (also the products' scratch
// for transposes), X, Zi, then dX1 / dX and F while they fit in
// `smem_doubles`; the ones that do not are in the problem's scratch (on a
// B200 F from n = 89 on, dX1 / dX from n = 105 on).
// ---------------------------------------------------------------------------
constexpr int ST_RED = 80;
constexpr int IPM_VECS = 5;

__host__ __device__ inline int ipm_st_base_doubles(int T) { return ST_RED + IPM_VECS * 8 * T + st_buffers(T); }

// Doubles of shared memory for n: the fixed part, X and Zi, then dX and F when
// they fit in `limit`.
__host__ __device__ inline size_t ipm_st_smem_doubles(int n, size_t limit)
{
    const int T = st_tiles(n);
    size_t d = ipm_st_base_doubles(T) + (size_t)st_packed(T) + 64 * (size_t)T * T;
    if (d + st_packed(T) <= limit) {
        d += st_packed(T);
        if (d + 64 * (size_t)T * T <= limit) d += 64 * (size_t)T * T;
    }
    return d;
}

// The same for problems of up to n (a smaller one may place more).
__host__ __device__ inline size_t ipm_st_smem_doubles_upto(int n, size_t limit)
{
    size_t d = 0;
    for (int T = st_tiles(n); T > 0; --T) {
        const size_t t = ipm_st_smem_doubles(8 * T, limit);
        d = t > d ? t : d;
    }
    return d;
}

// Scratch doubles a problem of size n may need (dX and F).
__host__ __device__ inline size_t ipm_st_ws_doubles(int n)
{
    const size_t T = st_tiles(n);
    return (size_t)st_packed((int)T) + 64 * T * T;
}

// The arrays of one problem.  The ones that are always in shared memory are
// named from st_smem wherever they are used (shared-memory accesses instead
// of generic ones).
struct IpmSt {
    int n, T;
    double* Q;   // dX1, then dX (symmetric tiles)
    double* F;   // inv(M), column-major with 8 T rows
    const double* L;
    __device__ double* red() const { return st_smem; }
    __device__ double* y() const { return st_smem + ST_RED; }
    __device__ double* zd() const { return st_smem + ST_RED + 8 * T; }
    __device__ double* dy() const { return st_smem + ST_RED + 16 * T; }
    __device__ double* dy1() const { return st_smem + ST_RED + 24 * T; }
    __device__ double* rhs() const { return st_smem + ST_RED + 32 * T; }
    __device__ double* buf() const { return st_smem + ST_RED + 8 * IPM_VECS * T; }
    __device__ double* X() const { return buf() + st_buffers(T); }
    __device__ double* Zi() const { return X() + st_packed(T); }
    __device__ int* flag() const { return reinterpret_cast<int*>(st_smem + ST_RED - 2); }
    // entry (i, j) of a symmetric and of a whole tile matrix
    __device__ static int sym(int i, int j)
    {
        const int a = i > j ? i : j, b = i > j ? j : i;
        return 64 * st_index(a >> 3, b >> 3) + st_elem(a & 7, b & 7);
    }
    __device__ int all(int i, int j) const { return 64 * ((i >> 3) * T + (j >> 3)) + st_elem(i & 7, j & 7); }
};

// This lane's pair of -L at tile (I, J) with the diagonal of Z + al Diag(dy);
// the identity outside n x n.
__device__ __forceinline__ double2 ipm_st_z(const IpmSt& s, double al, int I, int J, int r, int c)
{
    const int n = s.n, i = 8 * I + r, j = 8 * J + 2 * c;
    double2 v = make_double2(i == j ? 1.0 : 0.0, i == j + 1 ? 1.0 : 0.0);
    if (i < n && j < n) v.x = i == j ? fma(al, s.dy()[i], s.zd()[i]) : -s.L[i + (size_t)j * n];
    if (i < n && j + 1 < n) v.y = i == j + 1 ? fma(al, s.dy()[i], s.zd()[i]) : -s.L[i + (size_t)(j + 1) * n];
    return v;
}

// Zi = inv(Z + al Diag(dy)) (not inlined, nor the others here: the tiles in
// registers then have the whole register budget).  ONE: of one tile.
template <bool ONE>
static __device__ __noinline__ bool ipm_st_inv_z(const IpmSt& s, double al)
{
    const int T = s.T, lane = threadIdx.x & 31;
    double* Zi = s.Zi();
    auto fill = [&](int I, int J, int r, int c) { return ipm_st_z(s, al, I, J, r, c); };
    auto store = [&](int I, int J, double a, double b) {
        st_st(Zi + 64 * (I * T + J) + st_pair(lane >> 2, lane & 3), a, b);
    };
    if constexpr (ONE) return st_inverse_one(s.n, fill, store);
    if (T < 16) return st_inverse(T, s.buf(), s.flag(), fill, store);
    RegMat R;
    const int n = s.n;
    rm_fill(R, n, [&](int r, int c) { return r == c ? fma(al, s.dy()[r], s.zd()[r]) : -s.L[r + (size_t)c * n]; });
    const bool pd = rm_spd_inverse(R, n, s.buf());
    if (pd) {
#pragma unroll
        for (int b = 0; b < 8; ++b)
#pragma unroll
            for (int a = 0; a < 4; ++a) Zi[s.all(rm_row(a), rm_col(b))] = R.m[a][b];   // (0 outside n x n)
    }
    __syncthreads();
    return pd;
}

// F = inv(Zi .* X)
template <bool ONE>
static __device__ __noinline__ bool ipm_st_inv_m(const IpmSt& s)
{
    const int T = s.T, n = s.n, lane = threadIdx.x & 31;
    const double* X = s.X();
    const double* Zi = s.Zi();
    double* F = s.F;
    auto fill = [&](int I, int J, int r, int c) {
        const int i = 8 * I + r, j = 8 * J + 2 * c;
        const double2 z = st_ld(Zi + 64 * (I * T + J) + st_pair(r, c));
        double2 v = make_double2(i == j ? 1.0 : 0.0, i == j + 1 ? 1.0 : 0.0);
        if (i < n && j < n) v.x = z.x * X[IpmSt::sym(i, j)];
        if (i < n && j + 1 < n) v.y = z.y * X[IpmSt::sym(i, j + 1)];
        return v;
    };
    auto store = [&](int I, int J, double a, double b) {
        double* f = F + 8 * I + (lane >> 2) + (size_t)(8 * J + 2 * (lane & 3)) * (8 * T);
        f[0] = a;
        f[8 * T] = b;
    };
    if constexpr (ONE) return st_inverse_one(n, fill, store);
    if (T < 16) return st_inverse(T, s.buf(), s.flag(), fill, store);
    RegMat R;
    rm_fill(R, n, [&](int r, int c) { return Zi[s.all(r, c)] * X[IpmSt::sym(r, c)]; });
    const bool pd = rm_spd_inverse(R, n, s.buf());
    if (pd) rm_store(R, F, 8 * T);
    __syncthreads();
    return pd;
}

// X + al dX (Z + al Diag(dy) with dual) positive definite?
template <bool ONE>
static __device__ __noinline__ bool ipm_st_trial(const IpmSt& s, bool dual, double al)
{
    const double* X = s.X();
    const double* Q = s.Q;
    auto fill = [&](int I, int J, int r, int c) {
        double2 v;
        if (dual) {
            v = ipm_st_z(s, al, I, J, r, c);
        } else {
            const int o = 64 * st_index(I, J) + st_pair(r, c);
            const double2 x = st_ld(X + o), d = st_ld(Q + o);
            v = make_double2(fma(al, d.x, x.x), fma(al, d.y, x.y));
            if (I == J && 8 * I + r >= s.n) v = make_double2(r == 2 * c ? 1.0 : 0.0, r == 2 * c + 1 ? 1.0 : 0.0);
        }
        return make_double2(-v.x, -v.y);
    };
    if constexpr (ONE) return st_posdef_one(s.n, fill);
    return st_posdef(s.T, s.buf(), s.flag(), fill);
}

// out = F v, one warp per row, reading F's column (v null: v = -e); four rows
// at a time for their loads.
static __device__ __noinline__ void ipm_st_apply(const IpmSt& s, const double* v, double* out)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = s.n, ld = 8 * s.T;
    constexpr int nw = ST_THREADS / 32;
    for (int r0 = warp; r0 < n; r0 += 4 * nw) {
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        for (int c = lane; c < n; c += 32) {
            const double x = v ? v[c] : -1.0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = r0 + q * nw;
                acc[q] = fma(r < n ? s.F[c + (size_t)r * ld] : 0.0, x, acc[q]);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            acc[q] = warp_sum(acc[q]);
            if (lane == 0 && r0 + q * nw < n) out[r0 + q * nw] = acc[q];
        }
    }
    __syncthreads();
}

// P = Zi H, H = -Diag(d2) X (+ -Diag(d1) Y with WITH_Y), for all tiles; the
// warp of lower tile (I, J) has P_IJ and P_JI and hands P_ij and P_ji to epi(i,
// j, o, P_ij, P_ji) (o: the offset of (i, j) in a symmetric tile matrix), in
// squares of G x G tiles.  Sums over ascending k from zero.
template <int G, bool WITH_Y, class Epi>
__device__ __forceinline__ void ipm_st_product_g(const IpmSt& s, const double* d2, const double* Y, const double* d1,
                                                 Epi epi)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r = lane >> 2, c = lane & 3;
    const int T = s.T;
    const double* Zi = s.Zi();
    const double* X = s.X();
    double* scratch = s.buf() + 64 * warp;
    const StOp op;
    const int nb = (T + G - 1) / G;
    for (int b = warp; b < nb * (nb + 1) / 2; b += ST_THREADS / 32) {
        int BI, BJ;
        st_decode(b, &BI, &BJ);
        const int I0 = G * BI, J0 = G * BJ;
        const int ni = min(G, T - I0);
        const bool off = BI != BJ;
        double2 lo[G][G] = {}, up[G][G] = {};   // P_IJ and P_JI
        for (int K = 0; K < T; ++K) {
            double2 zi[G], zj[G], hi[G], hj[G];
            const double s0 = -d2[8 * K + c], s1 = -d2[8 * K + c + 4];
            double e0 = 0.0, e1 = 0.0;
            if (WITH_Y) {
                e0 = -d1[8 * K + c];
                e1 = -d1[8 * K + c + 4];
            }
            const int tk = 64 * st_index(K, 0) + op.to;
            auto load = [&](int A, double2& z, double2& h) {
                const int oz = 64 * (A * T + K) + op.o;
                z = make_double2(Zi[oz], Zi[oz + op.d]);
                const bool low = K <= A;
                const int o = low ? 64 * (st_index(A, 0) + K) + op.o : tk + 64 * A;
                const int o2 = o + (low ? op.d : 32);
                h = make_double2(s0 * X[o], s1 * X[o2]);
                if (WITH_Y) {
                    h.x = h.x + e0 * Y[o];
                    h.y = h.y + e1 * Y[o2];
                }
            };
#pragma unroll
            for (int a = 0; a < G; ++a) load(a < ni ? I0 + a : I0, zi[a], hi[a]);
            if (off) {
#pragma unroll
                for (int a = 0; a < G; ++a) load(J0 + a, zj[a], hj[a]);   // (a full square of columns)
            } else {
#pragma unroll
                for (int a = 0; a < G; ++a) {
                    zj[a] = zi[a];
                    hj[a] = hi[a];
                }
            }
#pragma unroll
            for (int a = 0; a < G; ++a)
#pragma unroll
                for (int e = 0; e < G; ++e) {
                    if (a >= ni || (!off && e > a)) continue;
                    st_mma(lo[a][e].x, lo[a][e].y, zi[a], hj[e]);
                    if (off || e < a) st_mma(up[a][e].x, up[a][e].y, zj[e], hi[a]);
                }
        }
#pragma unroll
        for (int a = 0; a < G; ++a)
#pragma unroll
            for (int e = 0; e < G; ++e) {
                if (a >= ni || (!off && e > a)) continue;
                // P_JI transposed through the warp's scratch
                const bool diagonal = !off && e == a;
                double2 t = diagonal ? lo[a][e] : up[a][e];
                scratch[st_elem(2 * c, r)] = t.x;
                scratch[st_elem(2 * c + 1, r)] = t.y;
                __syncwarp();
                t = st_ld(scratch + st_pair(r, c));
                __syncwarp();
                const int I = I0 + a, J = J0 + e;
                const int i = 8 * I + r, j = 8 * J + 2 * c;
                const int o = 64 * st_index(I, J) + st_pair(r, c);
                epi(i, j, o, lo[a][e].x, t.x);
                epi(i, j + 1, o + 1, lo[a][e].y, t.y);
            }
    }
    __syncthreads();
}

// The square's size: large squares load fewer operands a product, small ones
// keep more warps busy.
template <bool WITH_Y, class Epi>
__device__ __forceinline__ void ipm_st_product(const IpmSt& s, const double* d2, const double* Y, const double* d1,
                                               Epi epi)
{
    if (s.T < 5) ipm_st_product_g<1, WITH_Y>(s, d2, Y, d1, epi);
    else ipm_st_product_g<2, WITH_Y>(s, d2, Y, d1, epi);
}

// dX1 = sym(Zi (-Diag(dy1) X) - X) into Q
static __device__ __noinline__ void ipm_st_predictor(const IpmSt& s)
{
    double* Q = s.Q;
    const double* X = s.X();
    ipm_st_product<false>(s, s.dy1(), nullptr, nullptr, [=](int i, int j, int o, double p, double pt) {
        const double x = X[o];
        const double v = p - x;
        Q[o] = i == j ? v : 0.5 * ((pt - x) + v);
    });
}

// dX = sym(Zi (-Diag(dy2) X - Diag(dy1) dX1) + mu Zi + dX1) into `out`
static __device__ __noinline__ void ipm_st_corrector(const IpmSt& s, double mu, double* out)
{
    const double* Q = s.Q;
    const double* Zi = s.Zi();
    ipm_st_product<true>(s, s.dy(), Q, s.dy1(), [=](int i, int j, int o, double p, double pt) {
        const double q = Q[o];
        const double v = q + (p + mu * Zi[s.all(i, j)]);
        out[o] = i == j ? v : 0.5 * ((q + (pt + mu * Zi[s.all(j, i)])) + v);
    });
}

// stats (optional, device): the work counters [iterations n^3, problems,
// iterations, line-search trials] are added there.  smem_doubles: the CTA's
// dynamic shared memory (st_smem).  ONE: for n <= 8 only, by one warp's
// eliminations.
template <bool ONE = false>
__device__ inline void ipm_body_reg(const IpmDesc& d, int smem_doubles, double* stats)
{
    const int tid = threadIdx.x;
    constexpr int nt = ST_THREADS, nw = nt / 32;
    const int lane = tid & 31, warp = tid >> 5;
    const int r = lane >> 2, c = lane & 3;
    const int n = d.n;
    const int T = st_tiles(n), rows = 8 * T, ntiles = T * (T + 1) / 2;
    const int packed = st_packed(T), whole = 64 * T * T;
    const size_t nn = (size_t)n * n;
    const double* __restrict__ L = d.L;
    IpmSt s;
    s.n = n;
    s.T = T;
    s.L = L;
    {
        int used = ipm_st_base_doubles(T) + packed + whole;
        double* room = s.Zi() + whole;
        double* ws = d.ws;
        if (used + packed <= smem_doubles) {
            s.Q = room;
            room += packed;
            used += packed;
        } else {
            s.Q = ws;
            ws += packed;
        }
        s.F = used + whole <= smem_doubles ? room : ws;
    }
    double* const red = s.red();
    double* const y = s.y();
    double* const zd = s.zd();
    double* const dy = s.dy();
    double* const dy1 = s.dy1();
    double* const rhs = s.rhs();
    double* const X = s.X();
    double* const Zi = s.Zi();

    // ---- initial point (src/ipm_mc_pk.c:65-99): y_c = sum_r |L_rc| + 1.1, r in
    // order, from a copy in shared memory (X's and Zi's place) ----
    {
        const int ld = n | 1;
        double* const st = X;
        for (int j = warp; j < n; j += nw)
            for (int i = lane; i < n; i += 32) st[i + j * ld] = L[i + (size_t)j * n];
        __syncthreads();
        for (int q = tid; q < rows; q += nt) {
            double acc = 0.0;
            if (q < n)
                for (int i = 0; i < n; ++i) acc += fabs(st[i + q * ld]);
            y[q] = q < n ? acc + 1.1 : 0.0;
            zd[q] = q < n ? (acc + 1.1) - st[q + q * ld] : 0.0;
            dy[q] = dy1[q] = rhs[q] = 0.0;
        }
        __syncthreads();
    }
    for (int t = warp; t < ntiles; t += nw) {
        int I, J;
        st_decode(t, &I, &J);
        st_st(X + 64 * t + st_pair(r, c), I == J && r == 2 * c ? 1.0 : 0.0, I == J && r == 2 * c + 1 ? 1.0 : 0.0);
    }
    double a0 = 0.0, b0 = 0.0, p0 = 0.0;
    for (int i = tid; i < n; i += nt) {
        a0 += L[i + (size_t)i * n];
        b0 += zd[i];
        p0 += y[i];
    }
    double psi = block_sum(a0, red);
    double mu = block_sum(b0, red) / (2.0 * n);
    double phi = block_sum(p0, red);
    double gap = fabs(phi - psi);
    int iter = 0, ls_total = 0;
    int status = IPM_OK;
    bool have_zi = false;

    while (gap > 1e-2) {
        if (++iter > IPM_MAX_ITERS) { status = IPM_MAXITER; break; }

        // ---- Zi = inv(Z), Z = Diag(zd) - L off the diagonal ----
        if (!have_zi && !ipm_st_inv_z<ONE>(s, 0.0)) { status = IPM_Z_NOT_PD; break; }
        have_zi = false;
        // ---- F = inv(M), M = Zi .* X; dy1 = M \ (-e) (a non-positive pivot of
        // M is where the reference's dposv fails) ----
        if (!ipm_st_inv_m<ONE>(s)) { status = IPM_M_NOT_PD; break; }
        ipm_st_apply(s, nullptr, dy1);

        // ---- dX1 = sym(Zi (-Diag(dy1) X) - X) ----
        ipm_st_predictor(s);

        // ---- corrector rhs = mu diag(Zi) - (Zi .* dX1) dy1; dy2 = F rhs ----
        for (int q = warp; q < n; q += nw) {
            double acc = 0.0;
            for (int e = lane; e < n; e += 32) acc = fma(Zi[s.all(q, e)] * s.Q[IpmSt::sym(q, e)], dy1[e], acc);
            acc = warp_sum(acc);
            if (lane == 0) rhs[q] = mu * Zi[s.all(q, q)] - acc;
        }
        __syncthreads();
        ipm_st_apply(s, rhs, dy);

        // ---- dX = sym(Zi (-Diag(dy2) X - Diag(dy1) dX1) + mu Zi + dX1), over F,
        // which is done with; dy = dy1 + dy2 ----
        {
            double* const out = s.F;
            ipm_st_corrector(s, mu, out);
            for (int e = 2 * tid; e < packed; e += 2 * nt) *(double2*)(s.Q + e) = *(const double2*)(out + e);
        }
        for (int i = tid; i < n; i += nt) dy[i] = dy1[i] + dy[i];
        __syncthreads();

        // ---- primal line search: X + ap dX positive definite (the reference's chol) ----
        double ap = 1.0;
        int trials = 0;
        bool ok = false;
        while (true) {
            if (ipm_st_trial<ONE>(s, false, ap)) { ok = true; break; }
            if (++trials >= IPM_MAX_TRIALS) break;
            ap *= 0.8;
        }
        ls_total += trials + 1;
        if (!ok) { status = IPM_LINESEARCH; break; }
        if (ap < 1.0) ap *= 0.95;

        // ---- dual line search: Z + ad Diag(dy) positive definite ----
        double ad = 1.0;
        trials = 0;
        ok = false;
        while (true) {
            if (trials == 0 ? ipm_st_inv_z<ONE>(s, ad) : ipm_st_trial<ONE>(s, true, ad)) { ok = true; break; }
            if (++trials >= IPM_MAX_TRIALS) break;
            ad *= 0.8;
        }
        ls_total += trials + 1;
        if (!ok) { status = IPM_LINESEARCH; break; }
        have_zi = trials == 0;
        if (ad < 1.0) ad *= 0.95;

        // ---- update (src/ipm_mc_pk.c:313-334) ----
        double zx = 0.0, lx = 0.0;
        for (int j = warp; j < n; j += nw) {
            for (int i = lane; i < n; i += 32) {
                const int o = IpmSt::sym(i, j);
                const double xv = fma(ap, s.Q[o], X[o]);
                const double lv = L[i + (size_t)j * n];
                lx = fma(lv, xv, lx);
                if (i != j) zx = fma(-lv, xv, zx);
            }
        }
        __syncthreads();
        for (int e = 2 * tid; e < packed; e += 2 * nt) {
            const double2 x = st_ld(X + e), q = *(const double2*)(s.Q + e);
            st_st(X + e, fma(ap, q.x, x.x), fma(ap, q.y, x.y));
        }
        __syncthreads();
        double ysum = 0.0;
        for (int i = tid; i < n; i += nt) {
            const double yi = fma(ad, dy[i], y[i]);
            const double zi = fma(ad, dy[i], zd[i]);
            y[i] = yi;
            zd[i] = zi;
            ysum += yi;
            zx = fma(zi, X[IpmSt::sym(i, i)], zx);
        }
        zx = block_sum(zx, red);
        lx = block_sum(lx, red);
        ysum = block_sum(ysum, red);
        mu = zx / (2.0 * n);
        if (ap + ad > 1.6) mu *= 0.5;
        if (ap + ad > 1.9) mu *= 0.2;
        phi = ysum;
        psi = lx;
        gap = fabs(phi - psi);
    }

    // X, both triangles
    double* out = d.X + (d.xslot ? (size_t)(*d.xslot) * nn : 0);
    for (int j = warp; j < n; j += nw)
        for (int i = lane; i < n; i += 32) out[i + (size_t)j * n] = X[IpmSt::sym(i, j)];
    if (d.yout)
        for (int i = tid; i < n; i += nt) d.yout[i] = y[i];
    if (tid == 0) {
        d.out[0] = phi;
        d.out[1] = (double)iter;
        d.out[2] = (double)status;
        d.out[3] = psi;
        const double n3 = (double)n * n * n;
        if (stats) {
            atomicAdd(&stats[0], iter * n3);
            atomicAdd(&stats[1], 1.0);
            atomicAdd(&stats[2], (double)iter);
            atomicAdd(&stats[3], (double)ls_total);
        }
    }
}

}  // namespace bqb
