// Streaming top-T replay of the triangle separation (src/cutting_planes.c:
// 70-116) by one CTA, shared by the separation kernels (trisep.cu) and the
// fused node kernel (nodek.cu).
//
// The reference scans the violated cuts in order; the first T fill its list,
// each later one replaces the first-found minimum of the list when it is
// strictly larger.  Which slot a cut ends in depends on the whole history of
// replacements, so the history is replayed; replacing a heap's top one cut at
// a time took 1.5 us a replacement (28,000 of them, 43 ms, at n = 343 with T =
// 5000).  Here a chunk of up to TR_THREADS candidates goes in at once, from two
// facts about the sequence of replacements:
//  * candidate x is taken iff fewer than T of the candidates before it are
//    >= x: in the list L at the chunk's start, #{L >= x} + #{earlier in the
//    chunk, >= x} < T;
//  * the list's minimum never falls, and what a replacement removes was in the
//    list before it, so the t-th replacement of a chunk removes the t-th
//    smallest of L and the chunk's taken candidates together.
// So a chunk is a merge sort of its candidates (which counts the earlier larger
// ones on the way), a merge with the sorted list, and pointer jumping along
// "took the slot of" within the chunk.  Equal values leave in the order of their
// slots, and all of them are in the list before the first one leaves (a cut
// equal to the minimum is not taken): the list is kept in the order of (value,
// slot), and where a taken candidate equals another value of the union the slots
// are found run by run in ascending order instead, a run's from the
// replacements before it.  A whole separation at n = 343, T = 5000 takes 1.6 ms
// instead of 46; what bounds the replay is the chunk's chain of CTA barriers
// and the read of the candidates by one SM.
#pragma once
#include "trisep.cuh"

namespace bqb {

constexpr int TR_THREADS = 512;   // threads of the CTA, and candidates of a chunk

// Shared memory of the replay for lists of T cuts.
__host__ __device__ inline size_t tr_smem_bytes(int T)
{
    // two lists (value, slot, candidate) and the chunk's arrays
    return 2 * (size_t)T * 16 + (size_t)TR_THREADS * (8 + 4 + 2 * (8 + 4) + 4 + 4 + 8 + 4 + 4) + 256;
}

// Replay heap: the list's minimum by (value, slot) at the top.
__device__ __forceinline__ bool tr_heap_less(const double* hv, const int* hs, int a, int b)
{
    return hv[a] < hv[b] || (hv[a] == hv[b] && hs[a] < hs[b]);
}

__device__ inline void tr_heap_down(double* hv, int* hs, int T, int i)
{
    while (true) {
        const int l = 2 * i + 1, r = l + 1;
        int m = i;
        if (l < T && tr_heap_less(hv, hs, l, m)) m = l;
        if (r < T && tr_heap_less(hv, hs, r, m)) m = r;
        if (m == i) return;
        const double tv = hv[i];
        hv[i] = hv[m];
        hv[m] = tv;
        const int ts = hs[i];
        hs[i] = hs[m];
        hs[m] = ts;
        i = m;
    }
}

// One warp, one replacement at a time (V > T > 0).  hv: T doubles, then T
// ints, of shared memory.
__device__ inline void tr_replay_warp(const TriCand* __restrict__ cand, long long V, int T, TriCand* __restrict__ list,
                                      double* hv)
{
    const int lane = threadIdx.x & 31;
    int* hs = (int*)(hv + T);
    for (int q = lane; q < T; q += 32) {
        const TriCand c = cand[q];
        list[q] = c;
        hv[q] = c.value;
        hs[q] = q;
    }
    __syncwarp();
    if (lane == 0)
        for (int q = T / 2 - 1; q >= 0; --q) tr_heap_down(hv, hs, T, q);
    __syncwarp();
    for (long long base = T; base < V; base += 32) {
        const long long idx = base + lane;
        const double v = idx < V ? cand[idx].value : -INFINITY;
        double thr = hv[0];
        unsigned mask = __ballot_sync(0xffffffffu, v > thr);
        while (mask) {
            const int l = __ffs(mask) - 1;
            const double vl = __shfl_sync(0xffffffffu, v, l);
            __syncwarp();
            if (lane == 0) {
                const int slot = hs[0];
                list[slot] = cand[base + l];
                hv[0] = vl;
                tr_heap_down(hv, hs, T, 0);
            }
            __syncwarp();
            thr = hv[0];
            mask = __ballot_sync(0xffffffffu, lane > l && v > thr);
        }
    }
}

// First position in the ascending a[0..n) whose value is >= x (GE) or > x.
template <bool GE, class V>
__device__ __forceinline__ int tr_bound(const V* a, int n, V x)
{
    int lo = 0;
    for (int len = n; len > 0;) {
        const int half = len >> 1;
        const V v = a[lo + half];
        const bool right = GE ? v < x : v <= x;
        lo = right ? lo + half + 1 : lo;
        len = right ? len - half - 1 : half;
    }
    return lo;
}

// Exclusive prefix of v over the CTA's threads; *total = the sum.  ws: 17 ints.
__device__ __forceinline__ int tr_prefix(int v, int* ws, int* total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
    }
    if (lane == 31) ws[warp] = s;
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < TR_THREADS / 32; ++w) {
        const int x = ws[w];
        before += w < warp ? x : 0;
        all += x;
    }
    __syncthreads();
    *total = all;
    return before + s - v;
}

// The replay, by a CTA of TR_THREADS threads (V > T > 0): list[slot] for every
// slot.  sm: tr_smem_bytes(T) bytes of shared memory.
__device__ inline void tr_replay_cta(const TriCand* __restrict__ cand, long long V, int T,
                                     TriCand* __restrict__ list, double* sm)
{
    constexpr int S = TR_THREADS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double* lv = sm;                      // the sorted list: values,
    double* lw = lv + T;                  // (the other list's)
    double* xv = lw + T;                  // the chunk in arrival order
    double* mv = xv + S;                  // merge sort, 2 x S
    double* ev = mv + 2 * S;              // taken values, ascending (S)
    int* ls = (int*)(ev + S);             // slots,
    int* li = ls + T;                     // candidates
    int* lt = li + T;
    int* lj = lt + T;
    int* xi = lj + T;                     // candidates of the chunk
    int* mp = xi + S;                     // arrival positions, 2 x S
    int* ep = mp + 2 * S;                 // equal values: a taken one's slot
    int* tk = ep + S;                     // by arrival position: rank among the taken, or -1
    int* rf = tk + S;                     // replacement t: a slot, or -1 - the replacement it follows
    int* rg = rf + S;
    int* ws = rg + S;                     // 17 + flags

    // the first T cuts, sorted (merge passes; payload: slot)
    for (int q = tid; q < T; q += S) {
        lv[q] = cand[q].value;
        ls[q] = q;
    }
    __syncthreads();
    for (int w = 1; w < T; w <<= 1) {
        for (int q = tid; q < T; q += S) {
            const int b = q & ~(2 * w - 1), m = min(b + w, T), e = min(b + 2 * w, T);
            const double x = lv[q];
            const int to = q < m ? q + tr_bound<true>(lv + m, e - m, x) : b + (q - m) + tr_bound<false>(lv + b, m - b, x);
            lw[to] = x;
            lt[to] = ls[q];
        }
        __syncthreads();
        double* t = lv;
        lv = lw;
        lw = t;
        int* s = ls;
        ls = lt;
        lt = s;
    }
    for (int q = tid; q < T; q += S) li[q] = ls[q];
    __syncthreads();

    long long pos = T;
    while (pos < V) {
        // up to S candidates above the list's minimum, in order
        const double thr = lv[0];
        int n = 0;
        while (pos < V && n <= S / 2) {
            constexpr int R = 8;
            double v[R];
            unsigned m[R];
            const long long base = pos + (long long)warp * (32 * R);
            int mine = 0;
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const long long idx = base + 32 * k + lane;
                v[k] = idx < V ? cand[idx].value : -INFINITY;
            }
#pragma unroll
            for (int k = 0; k < R; ++k) {
                m[k] = __ballot_sync(0xffffffffu, v[k] > thr);
                mine += __popc(m[k]);
            }
            int total;
            int at = n + tr_prefix(lane == 0 ? mine : 0, ws, &total);
            at = __shfl_sync(0xffffffffu, at, 0);
            if (tid == 0) ws[20] = 0x7fffffff;
            __syncthreads();
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const int p = at + __popc(m[k] & ((1u << lane) - 1u));
                if (m[k] >> lane & 1) {
                    if (p < S) {
                        xv[p] = v[k];
                        xi[p] = (int)(base + 32 * k + lane);
                    } else if (p == S) {
                        ws[20] = (int)(base + 32 * k + lane - pos);   // the first one left for the next chunk
                    }
                }
                at += __popc(m[k]);
            }
            __syncthreads();
            const int cut = ws[20];
            n += total;
            __syncthreads();
            if (n > S) {
                n = S;
                pos += cut;
                break;
            }
            pos += 32 * R * (S / 32);
        }
        if (n == 0) continue;
        // merge sort of the chunk; c: earlier candidates >= this one
        if (tid < n) {
            mv[tid] = xv[tid];
            mp[tid] = tid;
        }
        tk[tid] = 0;
        __syncthreads();
        int cur = 0;
        for (int w = 1; w < n; w <<= 1) {
            const double* a = mv + cur * S;
            const int* ap = mp + cur * S;
            if (tid < n) {
                const int b = tid & ~(2 * w - 1), m = min(b + w, n), e = min(b + 2 * w, n);
                const double x = a[tid];
                int to;
                if (tid < m) {
                    to = tid + tr_bound<true>(a + m, e - m, x);
                } else {
                    const int le = tr_bound<false>(a + b, m - b, x);
                    to = b + (tid - m) + le;
                    // earlier ones >= x: those above, and the equal ones
                    int ge = m - b - le;
                    for (int q = b + le - 1; q >= b && a[q] == x; --q) ++ge;
                    tk[ap[tid]] += ge;
                }
                mv[(cur ^ 1) * S + to] = x;
                mp[(cur ^ 1) * S + to] = ap[tid];
            }
            __syncthreads();
            cur ^= 1;
        }
        const double* sv = mv + cur * S;   // ascending
        const int* sp = mp + cur * S;
        // taken?
        bool take = false;
        int below = 0;   // list values < x
        if (tid < n) {
            below = tr_bound<true>(lv, T, xv[tid]);
            take = (T - below) + tk[tid] < T;
        }
        int e;
        const int rank = tr_prefix(take ? 1 : 0, ws, &e);   // which replacement (arrival order)
        __syncthreads();
        tk[tid] = take ? rank : -1;
        __syncthreads();
        const bool staken = tid < n && tk[sp[tid < n ? tid : 0]] >= 0;
        int dummy;
        const int before = tr_prefix(staken ? 1 : 0, ws, &dummy);
        if (e == 0) continue;
        // the taken ones in ascending order: place u = before; below: list values
        // smaller than it
        int event = -1, id = 0;
        double x = 0.0;
        bool equal = false;
        if (staken) {
            const int a = sp[tid];
            x = sv[tid];
            event = tk[a];
            id = xi[a];
            below = tr_bound<true>(lv, T, x);
            equal = below < T && lv[below] == x;
            ev[before] = x;
        }
        __syncthreads();
        if (staken) equal = equal || (before + 1 < e && ev[before + 1] == x);
        if (!__syncthreads_or(equal)) {
            // places in the union
            for (int q = tid; q < T; q += S) {
                const double y = lv[q];
                const int p = q + tr_bound<true>(ev, e, y);
                if (p < e) {
                    rf[p] = ls[q];
                } else {
                    lw[p - e] = y;
                    lt[p - e] = ls[q];
                    lj[p - e] = li[q];
                }
            }
            const int place = below + before;
            if (staken) {
                if (place < e) {
                    rf[place] = -1 - event;
                } else {
                    lw[place - e] = x;
                    lj[place - e] = id;
                }
            }
            __syncthreads();
            // replacement t takes the slot of what it removed (chains of up to S: at
            // most ten doublings)
            bool more = true;
            for (int jump = 1; more && jump <= 2 * S; jump <<= 1) {
                bool open = false;
                if (tid < e) {
                    const int r = rf[tid];
                    const int s = r < 0 ? rf[-1 - r] : r;
                    rg[tid] = s;
                    open = s < 0;
                }
                more = __syncthreads_or(open) != 0;
                int* t = rf;
                rf = rg;
                rg = t;
            }
            if (staken && place >= e) lt[place - e] = rf[event];
        } else {
            // (what the chunk's arrays held is in registers)
            int* const cb = (int*)mv;   // by place u: list values smaller,
            int* const ce = cb + S;     // smaller or equal,
            int* const ue = ce + S;     // the end of its run of equal taken ones,
            int* const ci = xi;         // its candidate;
            int* const fs = mp;         // slots and candidates, a run by slots
            int* const fi = mp + S;
            if (staken) {
                cb[before] = below;
                ce[before] = tr_bound<false>(lv, T, x);
                ue[before] = tr_bound<false>(ev, e, x);
                rg[before] = event;
                ci[before] = id;
            }
            // rf[t]: the slot that replacement t takes; first the list's values that
            // no taken one equals
            if (tid < T && tid < e) {
                const double y = lv[tid];
                const int u = tr_bound<true>(ev, e, y);
                if (tid + u < e && !(u < e && ev[u] == y)) rf[tid + u] = ls[tid];
            }
            __syncthreads();
            if (warp == 0) {
                for (int u0 = 0; u0 < e;) {
                    const int u1 = ue[u0], a = cb[u0], b = ce[u0];
                    for (int u = u0 + lane; u < u1; u += 32) ep[u] = rf[rg[u]];
                    __syncwarp();
                    for (int u = u0 + lane; u < u1; u += 32) {
                        int r = u0;
                        for (int w = u0; w < u1; ++w) r += ep[w] < ep[u] ? 1 : 0;
                        fs[r] = ep[u];
                        fi[r] = ci[u];
                    }
                    __syncwarp();
                    for (int u = u0 + lane; u < u1; u += 32) {
                        const int p = a + u + tr_bound<true>(ls + a, b - a, fs[u]);
                        if (p < e) rf[p] = fs[u];
                    }
                    for (int q = a + lane; q < b && q + u0 < e; q += 32) {
                        const int p = q + u0 + tr_bound<true>(fs + u0, u1 - u0, ls[q]);
                        if (p < e) rf[p] = ls[q];
                    }
                    __syncwarp();
                    u0 = u1;
                }
            }
            __syncthreads();
            for (int q = tid; q < T; q += S) {
                const double y = lv[q];
                int u = tr_bound<true>(ev, e, y);
                if (u < e && ev[u] == y) u += tr_bound<true>(fs + u, ue[u] - u, ls[q]);
                const int p = q + u - e;
                if (p >= 0) {
                    lw[p] = y;
                    lt[p] = ls[q];
                    lj[p] = li[q];
                }
            }
            if (tid < e) {
                const int a = cb[tid], p = a + tid + tr_bound<true>(ls + a, ce[tid] - a, fs[tid]) - e;
                if (p >= 0) {
                    lw[p] = ev[tid];
                    lt[p] = fs[tid];
                    lj[p] = fi[tid];
                }
            }
        }
        __syncthreads();
        double* t = lv;
        lv = lw;
        lw = t;
        int* u = ls;
        ls = lt;
        lt = u;
        u = li;
        li = lj;
        lj = u;
    }
    for (int q = tid; q < T; q += S) list[ls[q]] = cand[li[q]];
    __syncthreads();
}

}  // namespace bqb
