// Device tree build: Hilbert- (or Morton-) sorted points bucketed into leaves of one warp
// (32 points) under an implicit complete binary tree (heap numbering of
// kd.h:6-15).  Replaces the reference's median-split kd build
// (kdBuildTree/kdBuildMoveTree, kd.c:225-552): any tree gives the same search
// results; this one is built with one sort and one up-pass.
//
// Node records (float4 pairs):
//   lo/hi   : tight box of the points below; lo.w = max ball2 below
//   blo/bhi : box of the balls below (x -/+ sqrt(ball2)), scatterer trees only
#include <cfloat>

#include "internal.h"

namespace skid {

namespace {

constexpr int BBOX_THREADS = 256;

__global__ void __launch_bounds__(BBOX_THREADS)
bbox_kernel(const float4 *__restrict__ p, int n, unsigned *box)
{
    float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4 q = p[i];
        mn[0] = fminf(mn[0], q.x); mx[0] = fmaxf(mx[0], q.x);
        mn[1] = fminf(mn[1], q.y); mx[1] = fmaxf(mx[1], q.y);
        mn[2] = fminf(mn[2], q.z); mx[2] = fmaxf(mx[2], q.z);
    }
    // one set of atomics a block: a set a warp, six addresses for all of
    // them, took 15 us at 100,000 points, this 2.7
    __shared__ unsigned smn[3][BBOX_THREADS / 32], smx[3][BBOX_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const unsigned a = __reduce_min_sync(SKID_FULL, f2ord(mn[d])), b = __reduce_max_sync(SKID_FULL, f2ord(mx[d]));
        if (lane == 0) {
            smn[d][w] = a;
            smx[d][w] = b;
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        unsigned a = smn[lane][0], b = smx[lane][0];
        for (int i = 1; i < BBOX_THREADS / 32; ++i) {
            a = min(a, smn[lane][i]);
            b = max(b, smx[lane][i]);
        }
        atomicMin(&box[lane], a);
        atomicMax(&box[3 + lane], b);
    }
}

__global__ void curve_kernel(const float4 *__restrict__ p, int n, const unsigned *box, int hil,
                             uint64_t *keys, uint32_t *vals)
{
    float3 lo = make_float3(ord2f(box[0]), ord2f(box[1]), ord2f(box[2]));
    float3 hi = make_float3(ord2f(box[3]), ord2f(box[4]), ord2f(box[5]));
    float ext = fmaxf(fmaxf(hi.x - lo.x, hi.y - lo.y), fmaxf(hi.z - lo.z, 1e-30f));
    float s = 2097151.0f / ext;
    float3 inv = make_float3(s, s, s);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4 q = p[i];
        keys[i] = curve63(make_float3(q.x, q.y, q.z), lo, inv, hil != 0);
        vals[i] = (uint32_t)i;
    }
}

__global__ void gather_sorted(const float4 *__restrict__ p, const uint32_t *__restrict__ perm,
                              int n, float4 *out, uint32_t *perm_out)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t j = perm[i];
        out[i] = p[j];
        perm_out[i] = j;
    }
}

// A node's box and ball box.
struct NodeBox {
    float3 lo, hi, blo, bhi;
    float b2;        // largest ball2
};

__device__ __forceinline__ float warp_min(float v) { return ord2f(__reduce_min_sync(SKID_FULL, f2ord(v))); }
__device__ __forceinline__ float warp_max(float v) { return ord2f(__reduce_max_sync(SKID_FULL, f2ord(v))); }

// One block per 32 leaves: each warp bounds leaves of one point per lane,
// then one warp combines the 32 boxes up five levels.  The block that is the
// last to finish below a node five levels further up combines those 32 in
// turn, to the root.  ball2 (sorted order) builds ball boxes when given; aux
// (sorted order, x = ball2, w = live-copy mask bits) is the alternative source
// for refits.
//
// A chain of latencies bounds it: a thread per leaf reading its 32 points one
// after the other, then an atomic and a fence per level, took 28.6 us a pass at
// 100,000 points and 30 to 50 at 2^20; this 9.7 and 12 to 24.
constexpr int UP_WARPS = 8;

__global__ void __launch_bounds__(UP_WARPS * 32)
upward_kernel(const float4 *__restrict__ pos, const float *__restrict__ ball2,
              const float4 *__restrict__ aux, int ballw, int n_host, const int *d_n, int leafBase,
              float4 *lo, float4 *hi, float4 *blo, float4 *bhi, int *flag, int *d_dirty)
{
    __shared__ NodeBox leaf_s[32];
    if (d_dirty && !*d_dirty) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int first = blockIdx.x * 32;
    const int n = d_n ? *d_n : n_host;
    // max ball2 (lo.w) needs ball data; ball boxes also need allocated arrays
    const bool hasb = (ball2 != nullptr) || (aux != nullptr) || ballw;
    const bool balls = hasb && blo != nullptr && bhi != nullptr;
    auto store = [&](int node, const NodeBox &x) {
        lo[node] = make_float4(x.lo.x, x.lo.y, x.lo.z, x.b2);
        hi[node] = make_float4(x.hi.x, x.hi.y, x.hi.z, 0.0f);
        if (balls) {
            blo[node] = make_float4(x.blo.x, x.blo.y, x.blo.z, 0.0f);
            bhi[node] = make_float4(x.bhi.x, x.bhi.y, x.bhi.z, 0.0f);
        }
    };
    const float3 top = make_float3(FLT_MAX, FLT_MAX, FLT_MAX), bottom = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
    const int leaves = min(32, leafBase - first);
#pragma unroll
    for (int r = 0; r < 32 / UP_WARPS; ++r) {
        const int l = r * UP_WARPS + w, i = (first + l) * SKID_LEAF + lane;
        NodeBox x;
        x.lo = x.blo = top;
        x.hi = x.bhi = bottom;
        x.b2 = -FLT_MAX;
        if (l < leaves && i < n) {
            const float4 q = pos[i];
            float b2 = 0.0f;
            bool live = true;
            if (ballw) {
                b2 = q.w;
            } else if (aux) {
                const float4 a = aux[i];
                b2 = a.x;
                live = __float_as_uint(a.w) != 0u;
            } else if (ball2) {
                b2 = ball2[i];
            }
            if (live) {
                x.lo = make_float3(fminf(FLT_MAX, q.x), fminf(FLT_MAX, q.y), fminf(FLT_MAX, q.z));
                x.hi = make_float3(fmaxf(-FLT_MAX, q.x), fmaxf(-FLT_MAX, q.y), fmaxf(-FLT_MAX, q.z));
                if (hasb) x.b2 = fmaxf(-FLT_MAX, b2);
                if (balls) {
                    // ball radius rounded up so the box contains every d2 < b2 point
                    float rad = sqrtf(b2) * (1.0f + 1e-6f) + 1e-30f;
                    rad += 4.8e-7f * (fabsf(q.x) + fabsf(q.y) + fabsf(q.z) + rad);
                    x.blo = make_float3(fminf(FLT_MAX, q.x - rad), fminf(FLT_MAX, q.y - rad), fminf(FLT_MAX, q.z - rad));
                    x.bhi = make_float3(fmaxf(-FLT_MAX, q.x + rad), fmaxf(-FLT_MAX, q.y + rad), fmaxf(-FLT_MAX, q.z + rad));
                }
            }
        }
        x.lo = make_float3(warp_min(x.lo.x), warp_min(x.lo.y), warp_min(x.lo.z));
        x.hi = make_float3(warp_max(x.hi.x), warp_max(x.hi.y), warp_max(x.hi.z));
        if (hasb) x.b2 = warp_max(x.b2);
        if (balls) {
            x.blo = make_float3(warp_min(x.blo.x), warp_min(x.blo.y), warp_min(x.blo.z));
            x.bhi = make_float3(warp_max(x.bhi.x), warp_max(x.bhi.y), warp_max(x.bhi.z));
        }
        if (lane == 0) leaf_s[l] = x;
    }
    __syncthreads();
    if (w != 0) return;
    NodeBox x = leaf_s[lane];
    if (lane < leaves) store(leafBase + first + lane, x);
    // lane i holds the box of node first_node + i, of 2^levels nodes
    int node = leafBase + first, levels = 0;
    while (levels < 5 && (1 << levels) < leaves) ++levels;
    for (;;) {
        for (int d = 0; d < levels; ++d) {
            const int o = 1 << d;
            x.lo = make_float3(fminf(x.lo.x, __shfl_xor_sync(SKID_FULL, x.lo.x, o)),
                               fminf(x.lo.y, __shfl_xor_sync(SKID_FULL, x.lo.y, o)),
                               fminf(x.lo.z, __shfl_xor_sync(SKID_FULL, x.lo.z, o)));
            x.hi = make_float3(fmaxf(x.hi.x, __shfl_xor_sync(SKID_FULL, x.hi.x, o)),
                               fmaxf(x.hi.y, __shfl_xor_sync(SKID_FULL, x.hi.y, o)),
                               fmaxf(x.hi.z, __shfl_xor_sync(SKID_FULL, x.hi.z, o)));
            x.b2 = fmaxf(x.b2, __shfl_xor_sync(SKID_FULL, x.b2, o));
            if (balls) {
                x.blo = make_float3(fminf(x.blo.x, __shfl_xor_sync(SKID_FULL, x.blo.x, o)),
                                    fminf(x.blo.y, __shfl_xor_sync(SKID_FULL, x.blo.y, o)),
                                    fminf(x.blo.z, __shfl_xor_sync(SKID_FULL, x.blo.z, o)));
                x.bhi = make_float3(fmaxf(x.bhi.x, __shfl_xor_sync(SKID_FULL, x.bhi.x, o)),
                                    fmaxf(x.bhi.y, __shfl_xor_sync(SKID_FULL, x.bhi.y, o)),
                                    fmaxf(x.bhi.z, __shfl_xor_sync(SKID_FULL, x.bhi.z, o)));
            }
            node >>= 1;
            if (lane < (1 << levels) && (lane & (2 * o - 1)) == 0) store(node + (lane >> (d + 1)), x);
        }
        if (node == 1) {
            // the root is finished after every block has read d_dirty
            if (d_dirty && lane == 0) *d_dirty = 0;
            return;
        }
        // node is finished; so is all below its ancestor `levels` up once as
        // many blocks have come by as that has descendants here
        levels = min(5, 31 - __clz(node));
        const int up = node >> levels;
        int old = 0;
        __syncwarp();
        if (lane == 0) {
            __threadfence();
            old = atomicAdd(&flag[up], 1);
        }
        if (__shfl_sync(SKID_FULL, old, 0) != (1 << levels) - 1) return;
        if (lane == 0) flag[up] = 0;   // for the next refit
        __threadfence();
        node = up << levels;
        x.lo = x.blo = top;
        x.hi = x.bhi = bottom;
        x.b2 = -FLT_MAX;
        if (lane < (1 << levels)) {
            const float4 a = __ldcg(&lo[node + lane]), b = __ldcg(&hi[node + lane]);
            x.lo = xyz(a);
            x.b2 = a.w;
            x.hi = xyz(b);
            if (balls) {
                x.blo = xyz(__ldcg(&blo[node + lane]));
                x.bhi = xyz(__ldcg(&bhi[node + lane]));
            }
        }
    }
}

}  // namespace

cudaError_t bbox_of(const float4 *pts, int n, unsigned *d_box6, cudaStream_t st)
{
    // order-preserving bit patterns: the three minima start at all ones, the
    // three maxima at zero (set on the device, no host memory involved)
    cudaError_t e = cudaMemsetAsync(d_box6, 0xff, 3 * sizeof(unsigned), st);
    if (!e) e = cudaMemsetAsync(d_box6 + 3, 0, 3 * sizeof(unsigned), st);
    if (e) return e;
    int blocks = min((n + 255) / 256, num_sms() * 4);
    if (blocks < 1) blocks = 1;
    bbox_kernel<<<blocks, 256, 0, st>>>(pts, n, d_box6); skid::note_launch();
    return cudaGetLastError();
}

static int leaf_base_for(int n)
{
    int nLeaf = (n + SKID_LEAF - 1) / SKID_LEAF;
    int p = 1;
    while (p < nLeaf) p <<= 1;
    return p;
}

cudaError_t tree_build(Tree &t, const float4 *pts, int n, bool balls, SortScratch &s,
                       cudaStream_t st, bool hil)
{
    cudaError_t e;
    t.n = n;
    t.nLeaf = (n + SKID_LEAF - 1) / SKID_LEAF;
    t.leafBase = leaf_base_for(n);
    size_t nodes = 2 * (size_t)t.leafBase;
    if ((e = dalloc(t.pos, n)) || (e = dalloc(t.perm, n)) || (e = dalloc(t.lo, nodes)) ||
        (e = dalloc(t.hi, nodes)) || (e = dalloc(t.flag, nodes)))
        return e;
    t.flag_clear = false;
    if (balls) {
        if ((e = dalloc(t.blo, nodes)) || (e = dalloc(t.bhi, nodes))) return e;
    }
    if (n > 0) {
        int blocks = min((n + 255) / 256, num_sms() * 8);
        if ((e = curve_order(pts, n, s, st, hil))) return e;
        gather_sorted<<<blocks, 256, 0, st>>>(pts, s.v0.p, n, t.pos.p, t.perm.p); skid::note_launch();
    }
    return tree_refit(t, nullptr, nullptr, nullptr, st);
}

cudaError_t curve_order(const float4 *pts, int n, SortScratch &s, cudaStream_t st, bool hil)
{
    cudaError_t e;
    if (n <= 0) return cudaSuccess;
    if ((e = dalloc(s.k0, n)) || (e = dalloc(s.k1, n)) || (e = dalloc(s.v0, n)) ||
        (e = dalloc(s.v1, n)) || (e = dalloc(s.box, 8)))
        return e;
    unsigned *dbox = s.box.p;
    if ((e = bbox_of(pts, n, dbox, st))) return e;
    int blocks = min((n + 255) / 256, num_sms() * 8);
    curve_kernel<<<blocks, 256, 0, st>>>(pts, n, dbox, hil ? 1 : 0, s.k0.p, s.v0.p); skid::note_launch();
    return radix_sort(s, n, 63, st);
}

cudaError_t tree_refit(Tree &t, const float4 *pos, const float4 *aux, const int *d_n,
                       cudaStream_t st, bool ballw, int *d_dirty)
{
    cudaError_t e = cudaSuccess;
    // arrival flags start zero (allocation) and every launch leaves them zero
    if (!t.flag_clear) {
        if ((e = cudaMemsetAsync(t.flag.p, 0, 2 * (size_t)t.leafBase * sizeof(int), st))) return e;
        t.flag_clear = true;
    }
    const int threads = UP_WARPS * 32, blocks = (t.leafBase + 31) / 32;
    bool nb = t.blo.n < 2 * (size_t)t.leafBase || t.bhi.n < 2 * (size_t)t.leafBase;
    upward_kernel<<<blocks, threads, 0, st>>>(pos ? pos : t.pos.p, nullptr, aux, ballw ? 1 : 0,
                                              t.n, d_n, t.leafBase, t.lo.p, t.hi.p,
                                              nb ? nullptr : t.blo.p, nb ? nullptr : t.bhi.p,
                                              t.flag.p, d_dirty); skid::note_launch();
    return cudaGetLastError();
}

cudaError_t tree_shape(Tree &t, int n, bool balls)
{
    cudaError_t e;
    t.n = n;
    t.nLeaf = (n + SKID_LEAF - 1) / SKID_LEAF;
    t.leafBase = leaf_base_for(n);
    size_t nodes = 2 * (size_t)t.leafBase;
    if ((e = dalloc(t.lo, nodes)) || (e = dalloc(t.hi, nodes)) || (e = dalloc(t.flag, nodes)))
        return e;
    t.flag_clear = false;
    if (balls && ((e = dalloc(t.blo, nodes)) || (e = dalloc(t.bhi, nodes)))) return e;
    return cudaSuccess;
}

}  // namespace skid
