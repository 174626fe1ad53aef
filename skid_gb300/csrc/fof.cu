// Friends-of-friends (kdFoF, kd.c:802-917) as a lock-free union-find.
//
// Edge rule: particles i and j are friends when d2(i->j) < tau^2 or
// d2(j->i) < tau^2 (float, no FMA, periodic image of the query; the
// reference tests the dequeued particle's frame, kd.c:869-876).  Groups are
// the connected components, numbered by ascending smallest member iOrder.
//
// The reference floods breadth-first and takes whole "contained" cells at
// once (INTERCONT, kd.h:217-335, kd.c:888-897), which matters because the
// moved particles of a group sit inside a ball of radius ~fCvg.  Here a node
// whose box diagonal is below tau is a clique; a pre-pass links each clique
// to its children's first points, and a query skips a clique subtree as soon
// as it is already in that clique's component.  Each pair is linked from its
// lower slot, so a query skips every subtree below its own leaf.
#include <cfloat>

#include "ctx.h"

namespace skid {

namespace {

constexpr int F_WARPS = 4;
constexpr int UF_SPIN_LIMIT = 1 << 22;

__device__ __forceinline__ int uf_find(int *par, int x)
{
    for (int it = 0; it < UF_SPIN_LIMIT; ++it) {
        int p = __ldcg(&par[x]);
        if (p == x) return x;
        int gp = __ldcg(&par[p]);
        if (gp != p) par[x] = gp;   // path halving; gp is an ancestor of x
        x = gp;
    }
    return x;
}

__device__ __forceinline__ void uf_union(int *par, int a, int b, unsigned *status)
{
    for (int it = 0; it < UF_SPIN_LIMIT; ++it) {
        a = uf_find(par, a);
        b = uf_find(par, b);
        if (a == b) return;
        if (a > b) { int t = a; a = b; b = t; }
        int old = atomicCAS(&par[b], b, a);
        if (old == b) return;
        b = old;
    }
    set_status(status, ST_TIMEOUT);
}

__device__ __forceinline__ int first_slot(int node, int leafBase)
{
    while (node < leafBase) node <<= 1;
    return (node - leafBase) * SKID_LEAF;
}

__global__ void uf_init(int *par, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        par[i] = i;
}

// Mark cliques (hi.w = 1) and pre-link them.
__global__ void clique_kernel(float4 *lo, float4 *hi, int leafBase, int n, float tau2, int *par,
                              unsigned *status)
{
    for (int node = blockIdx.x * blockDim.x + threadIdx.x + 1; node < 2 * leafBase;
         node += gridDim.x * blockDim.x) {
        float4 l = lo[node], h = hi[node];
        float dx = h.x - l.x, dy = h.y - l.y, dz = h.z - l.z;
        bool empty = !(dx >= 0.0f);
        float diag2 = dx * dx + dy * dy + dz * dz;
        bool clique = !empty && diag2 * (1.0f + 1e-5f) < tau2;
        h.w = clique ? 1.0f : 0.0f;
        hi[node] = h;
        if (!clique) continue;
        if (node >= leafBase) {
            // plain stores: of a leaf's slots only the first is seen by any
            // other node here (32 unions took this kernel 54 us at 2^20 points, this 7)
            int b = (node - leafBase) * SKID_LEAF, e = min(b + SKID_LEAF, n);
            for (int j = b + 1; j < e; ++j) par[j] = b;
        } else {
            int a = first_slot(2 * node, leafBase), c = first_slot(2 * node + 1, leafBase);
            if (a < n && c < n) uf_union(par, a, c, status);
        }
    }
}

// One warp per leaf of queries; each pair is linked from its lower slot, so
// subtrees wholly below the query leaf are skipped.  The last 2^subShift
// leaves under a node are tested one per lane against the query leaf's box;
// at a visited leaf, only candidates above the first query slot within tau
// of the query box are compacted and tested.  A clique node (box diagonal
// below tau) is skipped by a lane already in its component.
//
// Most friends found are in one component already, and asking the forest for
// both of a pair is two chains of dependent loads, which is what bounded the
// kernel.  So pairs are first tested alone (two to a packed FP32 operation;
// boxes no image can bring nearer are bounded without images), each candidate
// some lane found looks its root up once, and a lane joins only components
// that differ from its own root and from the one it joined last -- a root once
// found stays in its component, so an old one may cost a union but misses
// none.  2^20 points at half the mean spacing: 2.40 to 1.05 ms.
__global__ void __launch_bounds__(F_WARPS * 32, 8)
link_kernel(TreeView t, float tau2, float3 L, float3 hL, bool per, int subShift, float zero_arg, int *par,
            int *work, unsigned *status)
{
    __shared__ __align__(16) float cand[F_WARPS][3][SKID_LEAF];
    __shared__ int cslot[F_WARPS][SKID_LEAF];
    __shared__ int croot[F_WARPS][SKID_LEAF];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float (*cs)[SKID_LEAF] = cand[w];
    const int rootLo = t.leafBase >> subShift;
    const int logLeafBase = 31 - __clz(t.leafBase);
    const f32x2 zero = pack2(zero_arg, zero_arg), ntau2 = pack2(-tau2, -tau2);
    for (;;) {
        int leaf = 0;
        if (lane == 0) leaf = atomicAdd(work, 1);
        leaf = __shfl_sync(SKID_FULL, leaf, 0);
        if (leaf >= t.nLeaf) break;
        int base = leaf * SKID_LEAF;
        int qi = base + lane;
        bool valid = qi < t.n;
        float4 qp = t.pos[valid ? qi : base];
        float3 q = make_float3(qp.x, qp.y, qp.z);
        const int own = t.leafBase + leaf;
        const float4 qlo = t.lo[own], qhi = t.hi[own];
        const f32x2 nqx = pack2(-q.x, -q.x), nqy = pack2(-q.y, -q.y), nqz = pack2(-q.z, -q.z);
        int root = valid ? uf_find(par, qi) : -1;   // a root this query had
        int joined = -1;                            // and one it was joined to
        // lane is outside the component of a clique's first point
        auto apart = [&](int node) {
            const int rf = uf_find(par, first_slot(node, t.leafBase));
            if (rf == root) return false;
            root = uf_find(par, qi);
            return rf != root;
        };
        int cp = 1;
        for (;;) {
            // the last leaf under cp (its subtree is skipped when below ours)
            const int last = ((cp + 1) << (logLeafBase - (31 - __clz(cp)))) - 1;
            if (last >= own) {
                const float4 nlo = t.lo[cp], nhi = t.hi[cp];
                const bool dnode = boxes_direct(qlo, qhi, nlo, nhi, hL);
                if (cp >= rootLo) {
                    const int first = cp << subShift;
                    bool pass = false;
                    if (lane < (1 << subShift) && first + lane >= own &&
                        first + lane - t.leafBase < t.nLeaf) {
                        const float4 l = t.lo[first + lane], h = t.hi[first + lane];
                        pass = (dnode ? gap2(xyz(qlo), xyz(qhi), l, h) : boxbox_lb(qlo, qhi, l, h, L, per)) < tau2;
                    }
                    for (unsigned lm = __ballot_sync(SKID_FULL, pass); lm; lm &= lm - 1) {
                        const int node = first + __ffs(lm) - 1;
                        float4 blo = t.lo[node], bhi = t.hi[node];
                        const bool direct = dnode || boxes_direct(qlo, qhi, blo, bhi, hL);
                        bool want = valid && (direct ? gap2(q, q, blo, bhi) : box_lb(q, blo, bhi, L, per)) < tau2;
                        if (bhi.w != 0.0f && want) want = apart(node);
                        if (!__any_sync(SKID_FULL, want)) continue;
                        const int cb = (node - t.leafBase) * SKID_LEAF;
                        const int cnt = min(SKID_LEAF, t.n - cb);
                        bool rel = false;
                        float4 c4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        if (lane < cnt && cb + lane > base) {
                            c4 = t.pos[cb + lane];
                            rel = (direct ? gap2(xyz(c4), xyz(c4), qlo, qhi)
                                          : box_lb(xyz(c4), qlo, qhi, L, per)) < tau2;
                        }
                        const unsigned R = __ballot_sync(SKID_FULL, rel);
                        if (R == 0) continue;
                        const int nR = __popc(R);
                        const int rank = __popc(R & ((1u << lane) - 1u));
                        const int slot = rel ? rank : nR + lane - rank;
                        __syncwarp();
                        cs[0][slot] = rel ? c4.x : INFINITY;
                        cs[1][slot] = c4.y;
                        cs[2][slot] = c4.z;
                        cslot[w][slot] = cb + lane;
                        __syncwarp();
                        // friends, a bit per candidate
                        unsigned m = 0;
                        if (direct) {
                            for (int j = (nR - 1) & ~3; j >= 0; j -= 4) {
                                const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(&cs[0][j]);
                                const ulonglong2 Y = *reinterpret_cast<const ulonglong2 *>(&cs[1][j]);
                                const ulonglong2 Z = *reinterpret_cast<const ulonglong2 *>(&cs[2][j]);
#pragma unroll
                                for (int h = 1; h >= 0; --h) {
                                    const f32x2 dx = add2(h ? X.y : X.x, nqx), dy = add2(h ? Y.y : Y.x, nqy),
                                                dz = add2(h ? Z.y : Z.x, nqz);
                                    const float2 d = unpack2(
                                        add2(add2(add2(sq2(dx, zero), sq2(dy, zero)), sq2(dz, zero)), ntau2));
                                    m = __funnelshift_l(__float_as_uint(d.y), m, 1);
                                    m = __funnelshift_l(__float_as_uint(d.x), m, 1);
                                }
                            }
                        } else if (want) {
                            for (int j = 0; j < nR; ++j) {
                                const float3 c = make_float3(cs[0][j], cs[1][j], cs[2][j]);
                                float d1 = d2of(img_dx(q.x, c.x, L.x, hL.x), img_dx(q.y, c.y, L.y, hL.y),
                                                img_dx(q.z, c.z, L.z, hL.z));
                                float d2v = d2of(img_dx(c.x, q.x, L.x, hL.x), img_dx(c.y, q.y, L.y, hL.y),
                                                 img_dx(c.z, q.z, L.z, hL.z));
                                m |= (unsigned)(fminf(d1, d2v) < tau2) << j;
                            }
                        }
                        if (!want) m = 0;
                        // a pair is linked from its lower slot
                        if (node == own)
                            for (unsigned x = m; x; x &= x - 1) {
                                const int j = __ffs(x) - 1;
                                if (cslot[w][j] <= qi) m ^= 1u << j;
                            }
                        const unsigned any = __reduce_or_sync(SKID_FULL, m);
                        if (!any) continue;
                        if ((any >> lane) & 1u) croot[w][lane] = uf_find(par, cslot[w][lane]);
                        __syncwarp();
                        for (; m; m &= m - 1) {
                            const int j = __ffs(m) - 1;
                            const int r = croot[w][j];
                            if (r == root || r == joined) continue;
                            uf_union(par, qi, cslot[w][j], status);
                            joined = r;
                            root = uf_find(par, qi);
                        }
                    }
                } else {
                    bool want = valid && (dnode ? gap2(q, q, nlo, nhi) : box_lb(q, nlo, nhi, L, per)) < tau2;
                    if (nhi.w != 0.0f && want) want = apart(cp);
                    if (__any_sync(SKID_FULL, want)) { cp <<= 1; continue; }
                }
            }
            cp = next_node(cp);
            if (cp == 1) break;
        }
    }
}

// The root of x without path halving.
__device__ __forceinline__ int uf_root(const int *par, int x)
{
    for (int it = 0; it < UF_SPIN_LIMIT; ++it) {
        const int p = __ldcg(&par[x]);
        if (p == x) return x;
        x = p;
    }
    return x;
}

// label -> smallest member iOrder per root.  A thread writes its own slot
// only: halving other slots' paths here could put an ancestor read earlier
// over a root already written there, and what follows takes par for roots.
__global__ void root_min_iorder(int *par, int n, const uint32_t *__restrict__ perm,
                                const int *__restrict__ mio, int *__restrict__ minio)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int r = uf_root(par, i);
        par[i] = r;
        atomicMin(&minio[r], mio[perm[i]]);
    }
}

__global__ void mark_roots(const int *__restrict__ par, const int *__restrict__ minio, int n,
                           int *__restrict__ flag)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (par[i] == i) flag[minio[i]] = 1;
}

__global__ void write_groups(const int *__restrict__ par, const int *__restrict__ minio,
                             const int *__restrict__ rank, int n, const uint32_t *__restrict__ perm,
                             const int *__restrict__ mio, int *__restrict__ grp)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int r = par[i];
        grp[mio[perm[i]]] = rank[minio[r]] + 1;
    }
}

__global__ void fill_int(int *p, int v, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = v;
}

}  // namespace

// FoF over np points (float4) whose iOrders are mio[perm-index]; writes
// group ids (1..) to grp[iOrder] and the group count to *d_ng.  Scratch:
// par[np], minio[np], flag/rank over the iOrder space [niorder].
cudaError_t fof_run(Tree &t, const float4 *pts, int np, const int *mio, int niorder, float tau,
                    float3 L, bool per, SortScratch &ss, DBuf<int> &par, DBuf<int> &minio,
                    DBuf<int> &flag, int *grp, int *d_ng, int *d_work, unsigned *d_status,
                    cudaStream_t st)
{
    cudaError_t e;
    if (np <= 0) return cudaMemsetAsync(d_ng, 0, sizeof(int), st);
    if ((e = tree_build(t, pts, np, false, ss, st))) return e;
    if ((e = dalloc(par, np)) || (e = dalloc(minio, np)) || (e = dalloc(flag, 2 * (size_t)niorder)))
        return e;
    float tau2 = tau * tau;
    float3 hL = make_float3(0.5f * L.x, 0.5f * L.y, 0.5f * L.z);
    uf_init<<<grid_for(np), 256, 0, st>>>(par.p, np); skid::note_launch();
    clique_kernel<<<grid_for(2 * t.leafBase), 256, 0, st>>>(t.lo.p, t.hi.p, t.leafBase, np, tau2,
                                                           par.p, d_status); skid::note_launch();
    if ((e = cudaMemsetAsync(d_work, 0, sizeof(int), st))) return e;
    int perSM = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, link_kernel, F_WARPS * 32, 0);
    if (perSM < 1) perSM = 1;
    int blocks = num_sms() * perSM;
    int need = (t.nLeaf + F_WARPS - 1) / F_WARPS;
    if (blocks > need) blocks = need;
    int subShift = 0;
    while (subShift < 5 && (2 << subShift) <= t.leafBase) ++subShift;
    link_kernel<<<blocks, F_WARPS * 32, 0, st>>>(t.view(), tau2, L, hL, per, subShift, 0.0f, par.p, d_work,
                                                 d_status); skid::note_launch();
    fill_int<<<grid_for(np), 256, 0, st>>>(minio.p, 0x7fffffff, np); skid::note_launch();
    root_min_iorder<<<grid_for(np), 256, 0, st>>>(par.p, np, t.perm.p, mio, minio.p); skid::note_launch();
    int *fl = flag.p, *rank = flag.p + niorder;
    if ((e = cudaMemsetAsync(fl, 0, niorder * sizeof(int), st))) return e;
    mark_roots<<<grid_for(np), 256, 0, st>>>(par.p, minio.p, np, fl); skid::note_launch();
    if ((e = scan_exclusive(fl, rank, niorder, d_ng, ss, st))) return e;
    write_groups<<<grid_for(np), 256, 0, st>>>(par.p, minio.p, rank, np, t.perm.p, mio, grp); skid::note_launch();
    return cudaGetLastError();
}

}  // namespace skid
