// k-nearest-neighbour ball radii (fBall2) of every point of a tree, among the
// tree's own points, self included (smDensityInit/smBallSearch,
// smooth1.c:41-243).  Only the k-th smallest squared distance is kept: the
// density gather needs fBall2 alone, and that value does not depend on how
// equal distances are ordered.
//
// One warp per leaf of 32 query points, one query per lane (several warps
// while there are few leaves).  Each lane keeps its nearest squared distances
// in shared memory (value i of lane l at i*32+l, so every access is
// bank-conflict free): an unsorted buffer cut back by counting for k from 24
// to 128, a max-heap of k otherwise.  The warp first scans its own leaf, then
// climbs to the root visiting each sibling subtree depth-first (the search
// order of smBallSearch, smooth1.c:89-127), entering a node when any lane's
// bound reaches its box.  The last five
// levels of a subtree are tested one leaf per lane against the query leaf's
// box and the warp's largest bound; at a leaf only candidates within that
// bound of the query box are compacted and tested.
#include <cfloat>

#include <mutex>

#include "internal.h"

namespace skid {

namespace {

constexpr int KNN_WARPS = 4;

struct KnnLane {
    float3 q;       // query
    float thr;      // current k-th smallest (heap top)
    float *heap;    // this lane's heap base (stride 32)
};

__device__ __forceinline__ void heap_replace_top(float *heap, int k, float d)
{
    int i = 0;
    for (;;) {
        int c = 2 * i + 1;
        if (c >= k) break;
        float vc = heap[c * 32];
        if (c + 1 < k) {
            float vr = heap[(c + 1) * 32];
            if (vr > vc) { vc = vr; ++c; }
        }
        if (vc <= d) break;
        heap[i * 32] = vc;
        i = c;
    }
    heap[i * 32] = d;
}

// Process one leaf: candidates staged in shared memory, every lane tests all
// of them.  With a query box (filter), lane j first drops candidate j when
// its distance to the box is at least the warp's largest heap bound tmax:
// no lane can take it; the survivors are compacted in order.
__device__ __forceinline__ void knn_leaf(const TreeView &t, int node, float4 blo, float4 bhi,
                                         KnnLane &ln, int k, float3 L, float3 hL, bool per,
                                         float4 *cand, int lane, bool filter, float4 qlo,
                                         float4 qhi, float tmax)
{
    int leaf = node - t.leafBase;
    if (leaf >= t.nLeaf) return;
    int base = leaf * SKID_LEAF;
    int cnt = min(SKID_LEAF, t.n - base);
    float4 c4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    bool rel = lane < cnt;
    if (rel) {
        c4 = t.pos[base + lane];
        if (filter) rel = box_lb(make_float3(c4.x, c4.y, c4.z), qlo, qhi, L, per) < tmax;
    }
    const unsigned R = __ballot_sync(SKID_FULL, rel);
    cnt = __popc(R);
    __syncwarp();
    if (rel) cand[__popc(R & ((1u << lane) - 1u))] = c4;
    __syncwarp();
    int cx = img_class(ln.q.x, blo.x, bhi.x, hL.x);
    int cy = img_class(ln.q.y, blo.y, bhi.y, hL.y);
    int cz = img_class(ln.q.z, blo.z, bhi.z, hL.z);
    bool mixed = (cx == 2) | (cy == 2) | (cz == 2);
    if (__any_sync(SKID_FULL, mixed)) {
        for (int j = 0; j < cnt; ++j) {
            float4 c = cand[j];
            float dx = img_dx(ln.q.x, c.x, L.x, hL.x);
            float dy = img_dx(ln.q.y, c.y, L.y, hL.y);
            float dz = img_dx(ln.q.z, c.z, L.z, hL.z);
            float d2 = d2of(dx, dy, dz);
            if (d2 < ln.thr) {
                heap_replace_top(ln.heap, k, d2);
                ln.thr = ln.heap[0];
            }
        }
        return;
    }
    float sx = cx == 0 ? ln.q.x : (cx < 0 ? fsub(ln.q.x, L.x) : fadd(ln.q.x, L.x));
    float sy = cy == 0 ? ln.q.y : (cy < 0 ? fsub(ln.q.y, L.y) : fadd(ln.q.y, L.y));
    float sz = cz == 0 ? ln.q.z : (cz < 0 ? fsub(ln.q.z, L.z) : fadd(ln.q.z, L.z));
#pragma unroll 4
    for (int j = 0; j < cnt; ++j) {
        float4 c = cand[j];
        float d2 = d2of(fsub(sx, c.x), fsub(sy, c.y), fsub(sz, c.z));
        if (d2 < ln.thr) {
            heap_replace_top(ln.heap, k, d2);
            ln.thr = ln.heap[0];
        }
    }
}

__device__ __forceinline__ float warp_max(float v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(SKID_FULL, v, o));
    return v;
}

// ---- k from KB_MINK to KB_MAXK: unsorted buffers ----
//
// The heaps' sift-down runs for the whole warp whenever any lane takes a
// candidate, some 50k of 79k instructions for 32 queries at k = 64.  Here a
// lane appends what lies below its bound to a buffer of cap values in shared
// memory (value i of lane l at i * 32 + l) and, when some lane's is nearly
// full, all lanes cut theirs back at once: a threshold that leaves k values or
// somewhat more is found by counting (a guess from the counts and the 3/2
// power law of squared distances, usually one or two counts), the rest
// dropped, and the threshold is the lane's new bound.  The k-th smallest is
// found exactly at the end.  Candidates are tested two to a packed FP32
// operation, and where no periodic image can be nearer (nearly every leaf of
// a query away from the box's faces) the bounds are exact and cheap.
//
// At 2^20 points, k = 64: 82k instructions a leaf to 52k, 4.04 ms to 3.34; the
// call with its tree, 2^18 points: k = 128 3.81 to 2.78 ms, 32 1.24 to 1.05, 24
// 1.06 to 0.94, 16 0.83 to 0.84 (so the heaps keep small k; above 128 the
// buffers would leave too few warps an SM).  Bound by instruction issue at
// half the slots: 13 warps an SM, each a chain.  Room for 48 or 96 values
// beyond k, and cutting closer or less, were slower.  Counting distances into
// radial bins instead, with a second walk to pick from the k-th one's, took
// 62k instructions and had a longer tail: no faster.
constexpr int KB_MINK = 24, KB_MAXK = 128;
constexpr int KB_SLACK = 64;         // values a buffer holds beyond k
constexpr int KB_STEP = 8;           // candidates tested between checks for room
// Counts at guessed values, and all counts before the values themselves are
// asked (few lanes are left by then where distances differ; sooner costs 6 %).
constexpr int KB_GUESSES = 6, KB_TIGHTEN = 10;

struct KnnBuf {
    float *b;        // this lane's values, stride 32
    int n;           // values held
    float thr;       // at or above the k-th smallest so far; new values lie below
};

// Values at or below T (entries past a lane's last are infinite).
__device__ __forceinline__ int kb_count(const KnnBuf &B, int m, float T)
{
    // non-negative floats order as their bit patterns: the sign of the
    // difference to the pattern after T's is the comparison
    const int after = __float_as_int(T) + 1;
    const int *b = reinterpret_cast<const int *>(B.b);
    unsigned c = 0;
#pragma unroll 16
    for (int i = 0; i < m; ++i) c += (unsigned)(b[i * 32] - after) >> 31;
    return (int)c;
}

// A value summed or maximised over the S lanes that share a query.
template <int S>
__device__ __forceinline__ int kb_sum(int v)
{
#pragma unroll
    for (int o = 1; o < S; o <<= 1) v += __shfl_xor_sync(SKID_FULL, v, o);
    return v;
}

template <int S>
__device__ __forceinline__ float kb_max(float v)
{
#pragma unroll
    for (int o = 1; o < S; o <<= 1) v = fmaxf(v, __shfl_xor_sync(SKID_FULL, v, o));
    return v;
}

// The largest value (0 without any).
__device__ __forceinline__ float kb_largest(const KnnBuf &B, int m)
{
    float v = 0.0f;
#pragma unroll 8
    for (int i = 0; i < m; ++i) {
        const float x = B.b[i * 32];
        v = x < INFINITY ? fmaxf(v, x) : v;
    }
    return v;
}

// The least value's pattern above l, and the largest up to h.
__device__ __noinline__ int2 kb_span(const float *values, int m, int l, int h)
{
    const int *b = reinterpret_cast<const int *>(values);
    int2 v = make_int2(0x7f800000, 0);
#pragma unroll 8
    for (int i = 0; i < m; ++i) {
        const int x = b[i * 32];
        v.x = x > l ? min(v.x, x) : v.x;
        v.y = x <= h ? max(v.y, x) : v.y;
    }
    return v;
}

// The k-th smallest of the values that S lanes hold together (each its own
// buffer), between lo (fewer than k values at or below it; -1: none are) and hi
// (k or more): guesses from the counts, of which lo's is cl and hi's near ch,
// then bisection of the bit patterns, then (it >= KB_TIGHTEN) of those between
// the least and the largest value left: where many distances are equal but for
// rounding (a lattice, a shell of it at the k-th) no count is k and the values
// are a few patterns apart.  200,000 points of a lattice, k = 128: 2.53 to 2.06
// ms.  Lanes that are done have no use for it.
template <int S>
__device__ __forceinline__ float kb_kth(const KnnBuf &B, int m, int k, int lo, float hi, int cl, int ch,
                                        bool done, int it = 0)
{
    int l = lo, h = __float_as_int(hi);
    bool largest = false;
    for (; __any_sync(SKID_FULL, !done); ++it) {
        if (!done && h - l <= 1) done = true;      // h is the answer
        if (it == KB_TIGHTEN) {
            int2 v = kb_span(B.b, m, l, h);
#pragma unroll
            for (int o = 1; o < S; o <<= 1) {
                v.x = min(v.x, __shfl_xor_sync(SKID_FULL, v.x, o));
                v.y = max(v.y, __shfl_xor_sync(SKID_FULL, v.y, o));
            }
            if (!done) {
                l = v.x - 1;
                h = v.y;
                done = h - l <= 1;
            }
        }
        int mid = l + (h - l) / 2;
        if (it < KB_GUESSES) {
            const float a = l < 0 ? 0.0f : __int_as_float(l), b = __int_as_float(h);
            float t = (k + 0.0f - cl) / fmaxf((float)(ch - cl), 1.0f);
            if (cl == 0) t = exp2f(0.6666667f * log2f(t));
            const int g = __float_as_int(fmaf(b - a, fminf(fmaxf(t, 0.02f), 0.98f), a));
            if (g > l && g < h) mid = g;
        }
        const int c = kb_sum<S>(kb_count(B, m, __int_as_float(mid)));
        if (!done) {
            if (c < k) {
                l = mid;
                cl = c;
            } else {
                h = mid;
                ch = c;
                if (c == k) done = largest = true;
            }
        }
    }
    // a lane that stopped at exactly k values takes the largest of them
    const float T = __int_as_float(h);
    if (!__any_sync(SKID_FULL, largest)) return T;
    float v = 0.0f;
#pragma unroll 8
    for (int i = 0; i < m; ++i) {
        const float x = B.b[i * 32];
        v = x <= T ? fmaxf(v, x) : v;
    }
    v = kb_max<S>(v);
    return largest ? v : T;
}

// Cut every lane's buffer back, to `most` values at most.  At least k of those
// at or below the lane's bound stay, or all where there are fewer (a bound
// that another warp found: SHARED).
template <bool SHARED>
__device__ __noinline__ KnnBuf kb_cut(KnnBuf B, int k, int most)
{
    const int m = __reduce_max_sync(SKID_FULL, B.n);
    float hi = B.thr;
    if (__any_sync(SKID_FULL, B.thr == FLT_MAX)) hi = fminf(hi, kb_largest(B, m));
    float lo = 0.0f, T = hi;
    int cl = 0, ch = SHARED ? kb_count(B, m, hi) : B.n;
    // lanes with little to drop keep what they have (at or below the bound)
    bool done = ch <= k + (most - k) / 4;
    const bool skip = done;
    const float aim = k + 0.15f * (most - k);
    for (int it = 0; it < KB_GUESSES && __any_sync(SKID_FULL, !done); ++it) {
        float t = (aim - cl) / fmaxf((float)(ch - cl), 1.0f);
        if (cl == 0) t = exp2f(0.6666667f * log2f(t));
        const float mid = fmaf(hi - lo, fminf(fmaxf(t, 0.02f), 0.98f), lo);
        const int c = kb_count(B, m, mid);
        if (!done) {
            if (c < k) {
                lo = mid;
                cl = c;
            } else {
                hi = T = mid;
                ch = c;
                done = c <= most;
            }
        }
    }
    // ties or an uneven spread: the exact k-th value, and of its copies only
    // as many as make k
    const bool tight = !done && (SHARED || B.n >= k);
    int room = 0x7fffffff;
    if (__any_sync(SKID_FULL, tight)) {
        const float e = kb_kth<1>(B, m, k, cl == 0 ? -1 : __float_as_int(lo), hi, cl, ch, !tight, KB_TIGHTEN);
        int below = 0;
#pragma unroll 8
        for (int i = 0; i < m; ++i) below += B.b[i * 32] < e;
        if (tight) {
            T = e;
            room = k - below;
        }
    }
    if (skip && !SHARED) T = FLT_MAX;
    int o = 0;
    if (__any_sync(SKID_FULL, tight)) {
        for (int i = 0; i < m; ++i) {
            const float x = B.b[i * 32];
            bool keep = x <= T;
            if (keep && x == T) keep = room-- > 0;
            if (keep) B.b[o++ * 32] = x;
        }
    } else {
#pragma unroll 8
        for (int i = 0; i < m; ++i) {
            const float x = B.b[i * 32];
            if (x <= T) B.b[o++ * 32] = x;
        }
    }
    for (int i = __reduce_min_sync(SKID_FULL, o); i < m; ++i)
        if (i >= o) B.b[i * 32] = INFINITY;
    B.n = o;
    if (!skip) B.thr = fminf(B.thr, T);
    return B;
}

// S warps (a block) share a query leaf: of the leaves under a node warp w takes
// every S-th from w, with buffers of its own; a bound that one finds, at or above
// the k-th smallest of all, serves all of them through shared memory.
template <int S>
__global__ void __launch_bounds__(S * 32)
knn_buffer_kernel(TreeView t, int k, int cap, float3 L, float3 hL, bool per, int logLeafBase,
                  int subShift, float zero_arg, float *__restrict__ ball2, int *work)
{
    extern __shared__ float4 smem4[];
    __shared__ unsigned thr_s[32];
    __shared__ int n_s[S][32];
    __shared__ int leaf_s;
    const int lane = threadIdx.x & 31, w = S > 1 ? threadIdx.x >> 5 : 0;
    // candidates by component, then the lanes' buffers
    float *cx = reinterpret_cast<float *>(smem4) + w * 3 * SKID_LEAF;
    float *cy = cx + SKID_LEAF, *cz = cy + SKID_LEAF;
    float *bufs = reinterpret_cast<float *>(smem4) + S * 3 * SKID_LEAF;
    const int rootLo = t.leafBase >> subShift;
    const int most = k + (cap - k) / 2;
    const f32x2 zero = pack2(zero_arg, zero_arg);
    // of 32 leaves from a multiple of 32, this warp's
    const unsigned mine = (S == 1 ? ~0u : S == 2 ? 0x55555555u : S == 4 ? 0x11111111u : 0x01010101u) << w;
    KnnBuf B;
    B.b = bufs + (size_t)w * cap * 32 + lane;
    for (;;) {
        int leaf = 0;
        if (S == 1) {
            if (lane == 0) leaf = atomicAdd(work, 1);
            leaf = __shfl_sync(SKID_FULL, leaf, 0);
        } else {
            __syncthreads();
            if (threadIdx.x == 0) leaf_s = atomicAdd(work, 1);
            if (w == 0) thr_s[lane] = __float_as_uint(FLT_MAX);
            __syncthreads();
            leaf = leaf_s;
        }
        if (leaf >= t.nLeaf) break;
        const int base = leaf * SKID_LEAF, qi = base + lane;
        const bool valid = qi < t.n;
        const float4 qp = t.pos[valid ? qi : base];
        const float3 q = make_float3(qp.x, qp.y, qp.z);
        const f32x2 nqx = pack2(-q.x, -q.x), nqy = pack2(-q.y, -q.y), nqz = pack2(-q.z, -q.z);
        B.n = 0;
        B.thr = FLT_MAX;
        for (int i = 0; i < cap; ++i) B.b[i * 32] = INFINITY;
        const int own = t.leafBase + leaf;
        const float4 qlo = t.lo[own], qhi = t.hi[own];   // the queries' box
        auto tmax = [&]() {
            return __uint_as_float(__reduce_max_sync(SKID_FULL, __float_as_uint(B.thr)));
        };
        auto room = [&]() {
            if (!__any_sync(SKID_FULL, B.n > cap - KB_STEP)) return;
            B = kb_cut<(S > 1)>(B, k, most);
            if (S > 1) B.thr = fminf(B.thr, __uint_as_float(atomicMin(&thr_s[lane], __float_as_uint(B.thr))));
        };
        // lane j keeps candidate j while it may lie below some lane's bound
        auto leaf_values = [&](int node, bool direct, bool all) {
            const int cb = (node - t.leafBase) * SKID_LEAF;
            float4 c4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (S > 1) B.thr = fminf(B.thr, __uint_as_float(*(volatile unsigned *)&thr_s[lane]));
            const float tm = all ? INFINITY : tmax();
            bool rel = cb + lane < t.n;
            if (rel) {
                c4 = t.pos[cb + lane];
                if (!all)
                    rel = (direct ? gap2(xyz(c4), xyz(c4), qlo, qhi)
                                  : box_lb(xyz(c4), qlo, qhi, L, per)) < tm;
            }
            const unsigned R = __ballot_sync(SKID_FULL, rel);
            const int nR = __popc(R);
            const int rank = __popc(R & ((1u << lane) - 1u));
            // survivors in order, then entries no query can take
            const int slot = rel ? rank : nR + lane - rank;
            __syncwarp();
            cx[slot] = rel ? c4.x : INFINITY;
            cy[slot] = c4.y;
            cz[slot] = c4.z;
            __syncwarp();
            for (int j0 = 0; j0 < nR; j0 += KB_STEP) {
                room();
                if (direct) {
#pragma unroll
                    for (int j = 0; j < KB_STEP; j += 4) {
                        const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(cx + j0 + j);
                        const ulonglong2 Y = *reinterpret_cast<const ulonglong2 *>(cy + j0 + j);
                        const ulonglong2 Z = *reinterpret_cast<const ulonglong2 *>(cz + j0 + j);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const f32x2 dx = add2(h ? X.y : X.x, nqx), dy = add2(h ? Y.y : Y.x, nqy),
                                        dz = add2(h ? Z.y : Z.x, nqz);
                            const float2 d = unpack2(add2(add2(sq2(dx, zero), sq2(dy, zero)), sq2(dz, zero)));
                            if (d.x < B.thr) B.b[B.n++ * 32] = d.x;
                            if (d.y < B.thr) B.b[B.n++ * 32] = d.y;
                        }
                    }
                } else {
                    for (int j = j0; j < min(nR, j0 + KB_STEP); ++j) {
                        const float d2 = d2of(img_dx(q.x, cx[j], L.x, hL.x), img_dx(q.y, cy[j], L.y, hL.y),
                                              img_dx(q.z, cz[j], L.z, hL.z));
                        if (d2 < B.thr) B.b[B.n++ * 32] = d2;
                    }
                }
            }
        };
        if (S == 1 || leaf % S == w) leaf_values(own, boxes_direct(qlo, qhi, qlo, qhi, hL), true);
        int cell = own;
        while (cell > 1) {
            int cp = cell ^ 1;
            const int end = next_node(cp);
            for (;;) {
                const float4 blo = t.lo[cp], bhi = t.hi[cp];
                const bool direct = boxes_direct(qlo, qhi, blo, bhi, hL);
                if (cp >= rootLo) {
                    // a subtree of at most 2^subShift leaves: one lane per
                    // leaf against the queries' box, then the leaves below
                    // the largest bound with the exact bounds
                    const int sh = logLeafBase - (31 - __clz(cp));
                    const int first = cp << sh;
                    float dist = INFINITY;
                    if (lane < (1 << sh) && first + lane - t.leafBase < t.nLeaf &&
                        (S == 1 || (((mine << (S - (first & (S - 1)))) | (mine >> (first & (S - 1)))) >> lane & 1u))) {
                        const float4 l = t.lo[first + lane], h = t.hi[first + lane];
                        dist = direct ? gap2(xyz(qlo), xyz(qhi), l, h) : boxbox_lb(qlo, qhi, l, h, L, per);
                    }
                    for (;;) {
                        // the nearest leaf left, while it may hold something:
                        // bounds fall sooner than in curve order (a call at
                        // 2^20 points, k = 64, 3.42 to 3.23 ms; at 131,071,
                        // k = 128, 1.64 to 1.51)
                        const unsigned near = __reduce_min_sync(SKID_FULL, __float_as_uint(dist));
                        if (!(__uint_as_float(near) < tmax())) break;
                        const int at = __ffs(__ballot_sync(SKID_FULL, __float_as_uint(dist) == near)) - 1;
                        if (lane == at) dist = INFINITY;
                        const int node = first + at;
                        const float4 l = t.lo[node], h = t.hi[node];
                        const bool dl = direct || boxes_direct(qlo, qhi, l, h, hL);
                        const bool want = (dl ? gap2(q, q, l, h) : box_lb(q, l, h, L, per)) < B.thr;
                        if (!__any_sync(SKID_FULL, want)) continue;
                        leaf_values(node, dl, false);
                    }
                } else {
                    const bool want = (direct ? gap2(q, q, blo, bhi) : box_lb(q, blo, bhi, L, per)) < B.thr;
                    if (__any_sync(SKID_FULL, want)) { cp <<= 1; continue; }
                }
                cp = next_node(cp);
                if (cp == end) break;
            }
            cell >>= 1;
        }
        // the k-th smallest of what is left (the last bound is at or above
        // it); of S buffers a query, S lanes look at one each
        int n = B.n, query = lane;
        float hi = B.thr;
        if (S > 1) {
            n_s[w][lane] = B.n;
            __syncthreads();
            const int part = lane & (S - 1);
            query = w * (32 / S) + lane / S;
            n = n_s[part][query];
            hi = __uint_as_float(thr_s[query]);
            B.b = bufs + (size_t)part * cap * 32 + query;
        }
        const int m = __reduce_max_sync(SKID_FULL, n), all = kb_sum<S>(n);
        if (__any_sync(SKID_FULL, hi == FLT_MAX)) hi = fminf(hi, kb_max<S>(kb_largest(B, m)));
        const float r = kb_kth<S>(B, m, k, -1, hi, 0, all, all < k);
        if (base + query < t.n && (lane & (S - 1)) == 0) ball2[base + query] = all >= k ? r : FLT_MAX;
        if (S > 1) B.b = bufs + (size_t)w * cap * 32 + lane;
    }
}

template <int S>
cudaError_t launch_buffers(const Tree &t, int k, float3 L, float3 hL, bool per, int logLeafBase, int subShift,
                           float *ball2_sorted, int *d_work, cudaStream_t st)
{
    const int cap = k + KB_SLACK;
    const size_t smem = S * (3 * SKID_LEAF + (size_t)cap * 32) * sizeof(float);
    static std::mutex attr_mu;
    static bool attr_done[SKID_MAX_DEVICES] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e) return e;
    if (dev < 0 || dev >= SKID_MAX_DEVICES) return cudaErrorInvalidDevice;
    {
        // the most any k asks for
        std::lock_guard<std::mutex> lk(attr_mu);
        if (!attr_done[dev]) {
            e = cudaFuncSetAttribute(knn_buffer_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(S * (3 * SKID_LEAF + (KB_MAXK + KB_SLACK) * 32) * sizeof(float)));
            if (e) return e;
            attr_done[dev] = true;
        }
    }
    int perSM = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, knn_buffer_kernel<S>, S * 32, smem);
    if (e) return e;
    if (perSM < 1) return cudaErrorInvalidConfiguration;
    const int blocks = num_sms() * perSM < t.nLeaf ? num_sms() * perSM : t.nLeaf;
    if ((e = cudaMemsetAsync(d_work, 0, sizeof(int), st))) return e;
    knn_buffer_kernel<S><<<blocks, S * 32, smem, st>>>(t.view(), k, cap, L, hL, per, logLeafBase, subShift, 0.0f,
                                                       ball2_sorted, d_work); skid::note_launch();
    return cudaGetLastError();
}

// ---- any k: heaps ----

// Heaps live in shared memory after the candidate buffers, or -- for k too
// large for one warp's heaps to fit -- in global scratch (gheap, one slab per
// resident warp).
__global__ void __launch_bounds__(KNN_WARPS * 32, 6)
knn_kernel(TreeView t, int k, float3 L, float3 hL, bool per, int logLeafBase, int subShift,
           float *__restrict__ ball2, int *work, float *gheap)
{
    extern __shared__ float4 smem4[];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int nw = blockDim.x >> 5;
    float4 *cand = smem4 + w * SKID_LEAF;
    float *heaps = gheap ? gheap + (size_t)blockIdx.x * nw * k * 32
                         : reinterpret_cast<float *>(smem4 + nw * SKID_LEAF);
    const int rootLo = t.leafBase >> subShift;
    KnnLane ln;
    ln.heap = heaps + (size_t)w * k * 32 + lane;
    for (;;) {
        int leaf = 0;
        if (lane == 0) leaf = atomicAdd(work, 1);
        leaf = __shfl_sync(SKID_FULL, leaf, 0);
        if (leaf >= t.nLeaf) break;
        int base = leaf * SKID_LEAF;
        int qi = base + lane;
        bool valid = qi < t.n;
        float4 qp = t.pos[valid ? qi : base];
        ln.q = make_float3(qp.x, qp.y, qp.z);
        for (int i = 0; i < k; ++i) ln.heap[i * 32] = FLT_MAX;
        ln.thr = FLT_MAX;
        int own = t.leafBase + leaf;
        const float4 qlo = t.lo[own], qhi = t.hi[own];   // the queries' box
        knn_leaf(t, own, qlo, qhi, ln, k, L, hL, per, cand, lane, false, qlo, qhi, FLT_MAX);
        int cell = own;
        while (cell > 1) {
            int cp = cell ^ 1;
            int end = next_node(cp);
            for (;;) {
                if (cp >= rootLo) {
                    // a subtree of at most 2^subShift leaves: one lane per
                    // leaf against the queries' box and the largest bound,
                    // then each passing leaf in order with the exact bounds
                    const int sh = logLeafBase - (31 - __clz(cp));
                    const int first = cp << sh;
                    float tmax = warp_max(ln.thr);
                    bool pass = false;
                    if (lane < (1 << sh) && first + lane - t.leafBase < t.nLeaf)
                        pass = boxbox_lb(qlo, qhi, t.lo[first + lane], t.hi[first + lane], L, per) < tmax;
                    for (unsigned lm = __ballot_sync(SKID_FULL, pass); lm; lm &= lm - 1) {
                        const int node = first + __ffs(lm) - 1;
                        float4 blo = t.lo[node], bhi = t.hi[node];
                        bool want = box_lb(ln.q, blo, bhi, L, per) < ln.thr;
                        if (!__any_sync(SKID_FULL, want)) continue;
                        knn_leaf(t, node, blo, bhi, ln, k, L, hL, per, cand, lane, true, qlo, qhi,
                                 warp_max(ln.thr));
                    }
                } else {
                    float4 blo = t.lo[cp], bhi = t.hi[cp];
                    bool want = box_lb(ln.q, blo, bhi, L, per) < ln.thr;
                    if (__any_sync(SKID_FULL, want)) { cp <<= 1; continue; }
                }
                cp = next_node(cp);
                if (cp == end) break;
            }
            cell >>= 1;
        }
        if (valid) ball2[qi] = ln.thr;
    }
}

}  // namespace

cudaError_t knn_ball2(const Tree &t, int k, float3 L, bool per, float *ball2_sorted, int *d_work,
                      DBuf<float> &gheap, cudaStream_t st)
{
    if (t.n <= 0) return cudaSuccess;
    float3 hL = make_float3(0.5f * L.x, 0.5f * L.y, 0.5f * L.z);
    int logLeafBase = 0;
    while ((2 << logLeafBase) <= t.leafBase) ++logLeafBase;
    const int subShift = logLeafBase < 5 ? logLeafBase : 5;
    if (k >= KB_MINK && k <= KB_MAXK) {
        // Warps that share a leaf cost more in all (each collects k values
        // before it has a bound: about the factor S on a full chip), and pay
        // while the chip is not full.  k = 32, a call's time with S = 1 / 2 /
        // 4 / 8: 5,003 points 0.58 / 0.45 / 0.44 / 0.36 ms, 20,000 0.61 /
        // 0.57 / 0.51 / 0.59, 40,000 0.59 / 0.65 / 0.71 / 0.89; k = 128,
        // 20,000 points 1.07 / 1.13 / 1.32 / 1.70.
        const size_t smem = (3 * SKID_LEAF + (size_t)(k + KB_SLACK) * 32) * sizeof(float);
        int perSM = 0;
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, knn_buffer_kernel<1>, 32, smem);
        if (e) return e;
        const int slots = num_sms() * perSM;
        auto launch = t.nLeaf * 8 <= slots       ? launch_buffers<8>
                      : t.nLeaf * 4 <= slots     ? launch_buffers<4>
                      : t.nLeaf * 8 <= slots * 3 ? launch_buffers<2>
                                                 : launch_buffers<1>;
        return launch(t, k, L, hL, per, logLeafBase, subShift, ball2_sorted, d_work, st);
    }
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    size_t heapBytes = (size_t)k * 32 * sizeof(float);
    size_t candBytes = SKID_LEAF * sizeof(float4);
    int nw = KNN_WARPS;
    while (nw > 1 && (size_t)nw * (candBytes + heapBytes) > (size_t)optin) nw >>= 1;
    bool global = (size_t)nw * (candBytes + heapBytes) > (size_t)optin;
    size_t smem = (size_t)nw * candBytes + (global ? 0 : (size_t)nw * heapBytes);
    // The attribute belongs to the device and is only an upper bound: raise it
    // to the opt-in maximum once per device (contexts on other threads launch
    // with other k).
    static std::mutex attr_mu;
    static bool attr_done[SKID_MAX_DEVICES] = {};
    if (dev < 0 || dev >= SKID_MAX_DEVICES) return cudaErrorInvalidDevice;
    cudaError_t e = cudaSuccess;
    {
        std::lock_guard<std::mutex> lk(attr_mu);
        if (!attr_done[dev]) {
            cudaFuncAttributes fa;
            e = cudaFuncGetAttributes(&fa, knn_kernel);
            if (!e)
                e = cudaFuncSetAttribute(knn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         optin - (int)fa.sharedSizeBytes);
            if (!e) attr_done[dev] = true;
        }
    }
    if (e) return e;
    int perSM = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, knn_kernel, nw * 32, smem);
    if (e) return e;
    if (perSM < 1) return cudaErrorInvalidConfiguration;
    int blocks = num_sms() * perSM;
    int need = (t.nLeaf + nw - 1) / nw;
    if (blocks > need) blocks = need;
    float *gh = nullptr;
    if (global) {
        if ((e = dalloc(gheap, (size_t)blocks * nw * k * 32))) return e;
        gh = gheap.p;
    }
    if ((e = cudaMemsetAsync(d_work, 0, sizeof(int), st))) return e;
    knn_kernel<<<blocks, nw * 32, smem, st>>>(t.view(), k, L, hL, per, logLeafBase, subShift,
                                              ball2_sorted, d_work, gh); skid::note_launch();
    return cudaGetLastError();
}

}  // namespace skid
