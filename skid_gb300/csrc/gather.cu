// Gather kernels over the scatterer tree.
//
// density_gather: the reference scatters each pair (i, j in NN(i)) to both
// ends (smooth1.c:248-263).  Here each particle gathers both halves itself:
//   rho_i = sum_j 1/2 m_j W(d2(i->j), b_i) [d2 < b_i]     (its own neighbours)
//         + sum_k 1/2 m_k W(d2(k->i), b_k) [d2 < b_k]     (balls that hold it)
// with W the M4 spline of h^2 = b/4.  Each distance is taken in the frame the
// reference uses for that half (the query of the ball).  Deterministic order,
// Kahan-compensated FP32 sums.
//
// field_move: the move step.  The reference has every live scatterer copy
// gather the active movers inside its ball and add m/(pi h^5) F(q)(x_c - y)
// to them (smAccDensity/smBallGather, smooth1.c:338-508), then moves each
// mover by fStep along -a/|a| (kdMoveParticles, kd.c:702-732).  Here each
// mover walks the scatterer tree (ball boxes) and sums the copies whose ball
// holds it, then moves itself in the same kernel; a copy is the scatterer's
// periodic image nearest the mover, x_c = fl(x + sL), and must be live.  The
// warp keeps the least density of the scatterers that reached a mover (the
// floor of the cut, smooth1.c:460-461).
#include <cfloat>

#include "internal.h"

namespace skid {

namespace {

constexpr int G_WARPS = 4;

// Field kernel build tunables: unroll of the candidate test loop, and the
// minimum resident blocks per SM passed to __launch_bounds__ (caps registers).
#ifndef SKID_FIELD_UNROLL
#define SKID_FIELD_UNROLL 4
#endif
#ifndef SKID_FIELD_MINB
#define SKID_FIELD_MINB 9
#endif
constexpr int FIELD_UNROLL = SKID_FIELD_UNROLL;
// Boxes of consecutive movers a node is tested against: every mover's own
// point up to 16 per warp, halves of the warp above.  A warp whose movers lie
// on both sides of a gap in the order would otherwise reach for everything
// between them; those warps set the time of a step with few active movers.
// Field time of the 2^21 box 36.6 to 34.2 ms, of 150k mixed species 9.3 to 7.9.
constexpr int FNB(int G) { return G <= 16 ? G : 2; }
// Warps a split one-mover-per-warp step aims for (at most FIELD_SPLIT_CAP).
constexpr int FIELD_SPLIT_ITEMS = 8192;
static_assert(FIELD_SPLIT_ITEMS <= FIELD_SPLIT_CAP, "split buffers too small");

__device__ __forceinline__ float w_m4(float r2)
{
    float q = sqrtf(r2);
    float rs = 2.0f - q;
    return r2 < 1.0f ? 1.0f - 0.75f * rs * r2 : 0.25f * rs * rs * rs;
}

__device__ __forceinline__ void kahan_add(float &s, float &c, float x)
{
    float y = x - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
}

__device__ __forceinline__ float shifted(float x, int s, float L)
{
    return s == 0 ? x : (s < 0 ? fsub(x, L) : fadd(x, L));
}

// One warp per leaf of queries.  The walk descends a node while some lane's
// ball reaches its box or some ball below may hold the lane (box distance
// below max(b_i, max ball2 below)); the last 2^subShift leaves of a subtree
// are tested one per lane against the query leaf's box.  At a visited leaf,
// lane j keeps candidate j if its distance to the query box is below
// max(its ball, the largest query ball) -- the only candidates that can
// enter either half -- and the survivors, compacted in order, are summed.
//
// Instruction issue bounds it.  Where no periodic image can be nearer (nearly
// every leaf of a query away from the box's faces) the box bounds are exact
// and cheap, and one distance serves both halves; there the survivors are
// first tested, two to a packed FP32 operation, into a bit for each half, and
// each lane then runs the kernel terms of its own hits only, in the same
// order: 2^20 points 1.98 to 1.52 ms, the sums unchanged.
__global__ void __launch_bounds__(G_WARPS * 32)
density_kernel(TreeView t, const float *__restrict__ ball2, float3 L, float3 hL, bool per,
               int subShift, float zero_arg, float *__restrict__ rho, int *work)
{
    // survivors: x, y, z, -fBall2; and (fBall2, 1/h^2, 1/(2 pi h^3), mass)
    __shared__ __align__(16) float cand_s[G_WARPS][4][SKID_LEAF];
    __shared__ float4 caux[G_WARPS][SKID_LEAF];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float (*cs)[SKID_LEAF] = cand_s[w];
    const int rootLo = t.leafBase >> subShift;
    const f32x2 zero = pack2(zero_arg, zero_arg);
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
        float bi = ball2[valid ? qi : base];
        float ih2i = 4.0f / bi;
        float fni = 0.5f * (float)M_1_PI * sqrtf(ih2i) * ih2i;
        // the query leaf's box (its points) and largest ball
        const float4 qlo = t.lo[t.leafBase + leaf], qhi = t.hi[t.leafBase + leaf];
        float s = 0.0f, c = 0.0f;
        // the two halves' terms of a candidate at slot j
        auto own_half = [&](float4 aj, float d) { kahan_add(s, c, aj.w * fni * w_m4(d * ih2i)); };
        auto other_half = [&](float4 aj, float d) { kahan_add(s, c, aj.w * aj.z * w_m4(d * aj.y)); };
        int cp = 1;
        for (;;) {
            const float4 nlo = t.lo[cp], nhi = t.hi[cp];
            const bool dnode = boxes_direct(qlo, qhi, nlo, nhi, hL);
            if (cp >= rootLo) {
                const int first = cp << subShift;
                bool pass = false;
                if (lane < (1 << subShift)) {
                    float4 bl = t.lo[first + lane], bh = t.hi[first + lane];
                    pass = (dnode ? gap2(xyz(qlo), xyz(qhi), bl, bh) : boxbox_lb(qlo, qhi, bl, bh, L, per)) <
                           fmaxf(qlo.w, bl.w);
                }
                for (unsigned lm = __ballot_sync(SKID_FULL, pass); lm; lm &= lm - 1) {
                    const int node = first + __ffs(lm) - 1;
                    const int lf = node - t.leafBase;
                    if (lf >= t.nLeaf) break;
                    float4 blo = t.lo[node], bhi = t.hi[node];
                    const bool direct = dnode || boxes_direct(qlo, qhi, blo, bhi, hL);
                    bool want =
                        (direct ? gap2(q, q, blo, bhi) : box_lb(q, blo, bhi, L, per)) < fmaxf(bi, blo.w);
                    if (!__any_sync(SKID_FULL, want)) continue;
                    int cb = lf * SKID_LEAF;
                    int cnt = min(SKID_LEAF, t.n - cb);
                    bool rel = false;
                    float4 cj4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    float bj = 0.0f;
                    if (lane < cnt) {
                        cj4 = t.pos[cb + lane];
                        bj = ball2[cb + lane];
                        rel = (direct ? gap2(xyz(cj4), xyz(cj4), qlo, qhi)
                                      : box_lb(xyz(cj4), qlo, qhi, L, per)) < fmaxf(bj, qlo.w);
                    }
                    const unsigned R = __ballot_sync(SKID_FULL, rel);
                    if (R == 0) continue;
                    const int nR = __popc(R);
                    const int rank = __popc(R & ((1u << lane) - 1u));
                    // survivors in reverse order of rank, so that the first
                    // hit is the highest bit; above them entries without hits
                    const int slot = rel ? nR - 1 - rank : nR + lane - rank;
                    __syncwarp();
                    cs[0][slot] = rel ? cj4.x : INFINITY;
                    cs[1][slot] = cj4.y;
                    cs[2][slot] = cj4.z;
                    cs[3][slot] = -bj;
                    if (rel) {
                        float ih2 = 4.0f / bj;
                        caux[w][slot] = make_float4(bj, ih2, 0.5f * (float)M_1_PI * sqrtf(ih2) * ih2, cj4.w);
                    }
                    __syncwarp();
                    if (direct) {
                        const f32x2 nqx = pack2(-q.x, -q.x), nqy = pack2(-q.y, -q.y), nqz = pack2(-q.z, -q.z);
                        const f32x2 nbi = pack2(-bi, -bi);
                        unsigned own = 0, oth = 0;
                        for (int j = (nR - 1) & ~3; j >= 0; j -= 4) {
                            const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(&cs[0][j]);
                            const ulonglong2 Y = *reinterpret_cast<const ulonglong2 *>(&cs[1][j]);
                            const ulonglong2 Z = *reinterpret_cast<const ulonglong2 *>(&cs[2][j]);
                            const ulonglong2 B = *reinterpret_cast<const ulonglong2 *>(&cs[3][j]);
#pragma unroll
                            for (int h = 1; h >= 0; --h) {
                                const f32x2 dx = add2(h ? X.y : X.x, nqx), dy = add2(h ? Y.y : Y.x, nqy),
                                            dz = add2(h ? Z.y : Z.x, nqz);
                                const f32x2 d = add2(add2(sq2(dx, zero), sq2(dy, zero)), sq2(dz, zero));
                                const float2 a = unpack2(add2(d, nbi)), b = unpack2(add2(d, h ? B.y : B.x));
                                own = __funnelshift_l(__float_as_uint(a.y), own, 1);
                                own = __funnelshift_l(__float_as_uint(a.x), own, 1);
                                oth = __funnelshift_l(__float_as_uint(b.y), oth, 1);
                                oth = __funnelshift_l(__float_as_uint(b.x), oth, 1);
                            }
                        }
                        for (unsigned m = own | oth; m;) {
                            const int j = 31 - __clz(m);
                            m ^= 1u << j;
                            const float4 aj = caux[w][j];
                            const float d = d2of(fsub(q.x, cs[0][j]), fsub(q.y, cs[1][j]), fsub(q.z, cs[2][j]));
                            if ((own >> j) & 1u) own_half(aj, d);
                            if ((oth >> j) & 1u) other_half(aj, d);
                        }
                        continue;
                    }
                    if (!want) continue;
                    int cx = img_class(q.x, blo.x, bhi.x, hL.x);
                    int cy = img_class(q.y, blo.y, bhi.y, hL.y);
                    int cz = img_class(q.z, blo.z, bhi.z, hL.z);
                    bool mixed = (cx == 2) | (cy == 2) | (cz == 2);
                    bool noshift = (cx == 0) & (cy == 0) & (cz == 0);
                    float sx = shifted(q.x, cx, L.x), sy = shifted(q.y, cy, L.y), sz = shifted(q.z, cz, L.z);
                    for (int j = nR - 1; j >= 0; --j) {
                        const float3 cj = make_float3(cs[0][j], cs[1][j], cs[2][j]);
                        float4 aj = caux[w][j];
                        float dik, dki;
                        if (mixed) {
                            dik = d2of(img_dx(q.x, cj.x, L.x, hL.x), img_dx(q.y, cj.y, L.y, hL.y),
                                       img_dx(q.z, cj.z, L.z, hL.z));
                            dki = d2of(img_dx(cj.x, q.x, L.x, hL.x), img_dx(cj.y, q.y, L.y, hL.y),
                                       img_dx(cj.z, q.z, L.z, hL.z));
                        } else {
                            dik = d2of(fsub(sx, cj.x), fsub(sy, cj.y), fsub(sz, cj.z));
                            if (noshift) {
                                dki = dik;
                            } else {
                                dki = d2of(fsub(shifted(cj.x, -cx, L.x), q.x),
                                           fsub(shifted(cj.y, -cy, L.y), q.y),
                                           fsub(shifted(cj.z, -cz, L.z), q.z));
                            }
                        }
                        if (dik < bi) own_half(aj, dik);
                        if (dki < aj.x) other_half(aj, dki);
                    }
                }
            } else {
                bool want = (dnode ? gap2(q, q, nlo, nhi) : box_lb(q, nlo, nhi, L, per)) < fmaxf(bi, nlo.w);
                if (__any_sync(SKID_FULL, want)) { cp <<= 1; continue; }
            }
            cp = next_node(cp);
            if (cp == 1) break;
        }
        if (valid) rho[qi] = s;
    }
}

// Movers per warp G: 64, 32, 16, 8, 4 or 1; with G <= 32, 32/G lanes per
// mover, and with G = 64 two movers per lane.  More movers per warp share
// the tree walk and the leaf staging among more of them while the active
// movers are dense; fewer keep the union of their neighbourhoods small when
// they are sparse.  At a visited leaf the candidates whose ball reaches the
// movers' box are compacted in order; a mover's lanes test every (32/G)-th
// of them (one cheap pass that sets a hit mask), then run the field terms for
// their hits only, and are combined with a fixed xor-butterfly, so sums are
// deterministic for a given G.
//
// Instruction issue bounds it at 32 movers per warp (85 % of the issue slots
// at full activity of the 2^21 box), latency at few.  There (L = 1) the exact
// tests run two candidates to a packed FP32 operation with the decision read
// from a sign bit, and the prefilter is the exact test's own expression of the
// gaps.  At every G the leaves under a node are walked from registers, the
// next leaf's copies loaded while one is worked on, and the reciprocal root
// is the flushing one behind a floor.  Field time of the 2^21 box per run 42.2
// to 36.6 ms (a full-activity step 1.89 to 1.58 ms), the 150k mixed-species
// run 10.75 to 9.3 ms, 5k particles 1.60 to 1.40 ms.  Nine blocks an SM (56
// registers): 12 spill (41.5 ms), 10 took 40.1, 8 37.2.
template <int G, bool STATS>
__global__ void __launch_bounds__(G_WARPS * 32, G > 32 ? 8 : SKID_FIELD_MINB)
field_kernel(FieldArgs a)
{
    constexpr int MPL = G > 32 ? G / 32 : 1;   // movers per lane
    constexpr int L = G >= 32 ? 1 : 32 / G;    // lanes per mover
    constexpr int NB = FNB(G);                 // boxes the walk tests nodes against
    // a leaf's survivors by component: x, y, z, -fBall2 (four at a time go
    // into packed operands), and their (1/h^2, m/(pi h^5))
    __shared__ __align__(16) float cand_s[G_WARPS][4][SKID_LEAF];
    __shared__ float2 ccoef_s[G_WARPS][SKID_LEAF];
    __shared__ float4 box_s[G_WARPS][2 * NB];
    __shared__ unsigned floor_s[G_WARPS][32];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float (*cs)[SKID_LEAF] = cand_s[w];
    float2 *cc = ccoef_s[w];
    const int nA = *a.d_nA;
    const int nC = *a.d_nC;
    // One mover per warp and few movers: each mover's walk is split over S
    // warps (about FIELD_SPLIT_ITEMS warps in all); all walk the inner nodes,
    // and of each 32 leaves under a node, part p takes every S-th from p.
    int S = 1;
    if (G == 1 && a.part_acc && a.logLeafBase >= 5) {
        const int t = FIELD_SPLIT_ITEMS / (nA > 0 ? nA : 1);
        S = t >= 16 ? 16 : t >= 8 ? 8 : t >= 4 ? 4 : t >= 2 ? 2 : 1;
    }
    const int nItems = G == 1 ? nA * S : (nA + G - 1) / G;
    const int sub = lane % L;
    unsigned long long st_nodes = 0, st_leaves = 0, st_tests = 0, st_hits = 0;
    floor_s[w][lane] = 0xffffffffu;
    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(a.d_work, 1);
        item = __shfl_sync(SKID_FULL, item, 0);
        if (item >= nItems) break;
        int part = 0;
        if (G == 1) {
            part = item % S;
            item /= S;
        }
        int slot[MPL], mi[MPL];
        bool valid[MPL];
        float4 yp[MPL];
        float3 y[MPL];
        // bounding box of the warp's movers, for the per-leaf candidate prefilter
        float3 wlo = make_float3(FLT_MAX, FLT_MAX, FLT_MAX);
        float3 whi = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
#pragma unroll
        for (int k = 0; k < MPL; ++k) {
            slot[k] = item * G + k * 32 + lane / L;
            valid[k] = slot[k] < nA;
            mi[k] = a.act[valid[k] ? slot[k] : item * G];
            yp[k] = a.mpos[mi[k]];
            y[k] = make_float3(yp[k].x, yp[k].y, yp[k].z);
            if (valid[k]) {
                wlo = make_float3(fminf(wlo.x, y[k].x), fminf(wlo.y, y[k].y), fminf(wlo.z, y[k].z));
                whi = make_float3(fmaxf(whi.x, y[k].x), fmaxf(whi.y, y[k].y), fmaxf(whi.z, y[k].z));
            }
        }
        auto join = [&](int o) {
            wlo.x = fminf(wlo.x, __shfl_xor_sync(SKID_FULL, wlo.x, o));
            wlo.y = fminf(wlo.y, __shfl_xor_sync(SKID_FULL, wlo.y, o));
            wlo.z = fminf(wlo.z, __shfl_xor_sync(SKID_FULL, wlo.z, o));
            whi.x = fmaxf(whi.x, __shfl_xor_sync(SKID_FULL, whi.x, o));
            whi.y = fmaxf(whi.y, __shfl_xor_sync(SKID_FULL, whi.y, o));
            whi.z = fmaxf(whi.z, __shfl_xor_sync(SKID_FULL, whi.z, o));
        };
        // the boxes of the warp's NB runs of consecutive movers, then the
        // box of them all
#pragma unroll
        for (int o = L; o < 32 / NB; o <<= 1) join(o);
        if (NB > 1) {
            __syncwarp();
            if (lane % (32 / NB) == 0) {
                box_s[w][2 * (lane / (32 / NB))] = make_float4(wlo.x, wlo.y, wlo.z, 0.0f);
                box_s[w][2 * (lane / (32 / NB)) + 1] = make_float4(whi.x, whi.y, whi.z, 0.0f);
            }
            __syncwarp();
        }
#pragma unroll
        for (int o = 32 / NB; o < 32; o <<= 1) join(o);
        float ax[MPL], ay[MPL], az[MPL];
#pragma unroll
        for (int k = 0; k < MPL; ++k) ax[k] = ay[k] = az[k] = 0.0f;
        // Depth-first walk by ball boxes in strides of five levels, aligned
        // so the last stride ends at the leaves: a visited node has each lane
        // test one of its 32 descendants five levels down against the movers'
        // box, and those that pass are visited in order (so leaves come in
        // depth-first order).  A visited inner node is entered only if some
        // mover lies in its ball box (up to 16 movers per warp the nodes are
        // tested against each one, and passing says so already).  Stack level l (its
        // first node and the descendants still to visit) is held by lane l.
        auto reach = [&](int node) {
            const float4 bl = a.blo[node], bh = a.bhi[node];
            if (NB == 1)
                return bl.x <= whi.x && bh.x >= wlo.x && bl.y <= whi.y && bh.y >= wlo.y &&
                       bl.z <= whi.z && bh.z >= wlo.z;
            bool hit = false;
#pragma unroll
            for (int q = 0; q < NB; ++q) {
                const float4 l = box_s[w][2 * q], h = box_s[w][2 * q + 1];
                hit = hit || (bl.x <= h.x && bh.x >= l.x && bl.y <= h.y && bh.y >= l.y &&
                              bl.z <= h.z && bh.z >= l.z);
            }
            return hit;
        };
        // one of this lane's movers lies in the box
        auto inside = [&](float4 blo, float4 bhi) {
            bool in = false;
#pragma unroll
            for (int k = 0; k < MPL; ++k)
                in = in || (valid[k] && y[k].x >= blo.x && y[k].x <= bhi.x && y[k].y >= blo.y &&
                            y[k].y <= bhi.y && y[k].z >= blo.z && y[k].z <= bhi.z);
            return in;
        };
        // the copy of this lane in a leaf (an empty ball past the end)
        auto load_copy = [&](int lf) {
            const int i = lf * SKID_LEAF + lane;
            return i < nC ? a.cpos[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        };
        // One term of the field: the value (smooth1.c:450-458) only has to be
        // accurate, not bit-exact: FMA and the approximate reciprocal square
        // root (q = r2 / sqrt(r2), 1/q).  At r2 = 0 the floor under the root
        // gives q = 0, and 1/q is not used.
        auto add_term = [&](int k, int j) {
            const float dx = cs[0][j] - y[k].x, dy = cs[1][j] - y[k].y, dz = cs[2][j] - y[k].z;
            const float2 cf = cc[j];
            const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)) * cf.x;
            float iq;
            asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(iq) : "f"(fmaxf(r2, 1e-37f)));
            const float q = r2 * iq;
            float F = r2 < 1.0f ? __fmaf_rn(2.25f, q, -3.0f)
                                : __fmaf_rn(-0.75f, q, 3.0f) - 3.0f * iq;
            F *= cf.y;
            ax[k] = __fmaf_rn(dx, F, ax[k]);
            ay[k] = __fmaf_rn(dy, F, ay[k]);
            az[k] = __fmaf_rn(dz, F, az[k]);
        };
        // A visited leaf: c4 is this lane's copy.
        auto leaf_terms = [&](int lf, float4 c4) {
            const int cb = lf * SKID_LEAF;
            // a leaf box that overlaps the movers' often holds none of them
            if (G > NB) {
                float4 blo = a.blo[a.leafBase + lf], bhi = a.bhi[a.leafBase + lf];
                if (!__any_sync(SKID_FULL, inside(blo, bhi))) return;
            }
            if (STATS) ++st_leaves;
            // prefilter: lane j keeps candidate j if its ball reaches the
            // movers' box; the exact test below decides, so this only skips
            // candidates that cannot hit (per-axis gaps to the box, zero
            // inside).  An empty ball is rejected.
            const float gx = fmaxf(fmaxf(wlo.x - c4.x, c4.x - whi.x), 0.0f);
            const float gy = fmaxf(fmaxf(wlo.y - c4.y, c4.y - whi.y), 0.0f);
            const float gz = fmaxf(fmaxf(wlo.z - c4.z, c4.z - whi.z), 0.0f);
            bool rel;
            if (L == 1) {
                // float subtraction, product and sum are monotonic, so the
                // exact test's d2 of a mover in the box is never below the
                // same expression of the gaps
                rel = d2of(gx, gy, gz) < c4.w;
            } else {
                // radius from the approximate reciprocal square root, widened
                // to cover its error; which survivors there are decides the
                // lane that sums each, so this form is kept to the last bit
                float r = c4.w * rsqrtf(c4.w) * (1.0f + 4e-6f) +
                          1e-6f * (fabsf(c4.x) + fabsf(c4.y) + fabsf(c4.z)) + 1e-30f;
                rel = __fmaf_rn(gz, gz, __fmaf_rn(gy, gy, gx * gx)) <= r * r;
            }
            const unsigned R = __ballot_sync(SKID_FULL, rel);
            if (R == 0) return;
            const int nR = __popc(R);
            const int rank = __popc(R & ((1u << lane) - 1u));
            unsigned hitany = 0;
            int slot_r;
            if (L == 1) {
                // Survivors go into slots in reverse order of rank, the rest
                // as entries no mover is inside above them: with a hit's bit
                // at its slot, the highest set bit is the first hit.
                slot_r = rel ? nR - 1 - rank : nR + lane - rank;
                __syncwarp();
                cs[0][slot_r] = c4.x;
                cs[1][slot_r] = c4.y;
                cs[2][slot_r] = c4.z;
                cs[3][slot_r] = rel ? -c4.w : INFINITY;
                if (rel) {
                    float4 co = a.ccoef[cb + lane];
                    cc[slot_r] = make_float2(co.x, co.y);
                }
                __syncwarp();
                if (STATS) st_tests += MPL * nR;
#pragma unroll
                for (int k = 0; k < MPL; ++k) {
                    const f32x2 nyx = pack2(-y[k].x, -y[k].x), nyy = pack2(-y[k].y, -y[k].y),
                                nyz = pack2(-y[k].z, -y[k].z);
                    // smBallGather's test d2 < fBall2 (smooth1.c:365-369),
                    // from the copy, two copies an operation: the sign of
                    // d2 - fBall2 is shifted in
                    const f32x2 zero = pack2(a.zero, a.zero);
                    unsigned m = 0;
                    for (int t = (nR - 1) & ~3; t >= 0; t -= 4) {
                        const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(&cs[0][t]);
                        const ulonglong2 Y = *reinterpret_cast<const ulonglong2 *>(&cs[1][t]);
                        const ulonglong2 Z = *reinterpret_cast<const ulonglong2 *>(&cs[2][t]);
                        const ulonglong2 W = *reinterpret_cast<const ulonglong2 *>(&cs[3][t]);
                        f32x2 dx = add2(X.y, nyx), dy = add2(Y.y, nyy), dz = add2(Z.y, nyz);
                        float2 d = unpack2(add2(add2(add2(sq2(dx, zero), sq2(dy, zero)), sq2(dz, zero)), W.y));
                        m = __funnelshift_l(__float_as_uint(d.y), m, 1);
                        m = __funnelshift_l(__float_as_uint(d.x), m, 1);
                        dx = add2(X.x, nyx), dy = add2(Y.x, nyy), dz = add2(Z.x, nyz);
                        d = unpack2(add2(add2(add2(sq2(dx, zero), sq2(dy, zero)), sq2(dz, zero)), W.x));
                        m = __funnelshift_l(__float_as_uint(d.y), m, 1);
                        m = __funnelshift_l(__float_as_uint(d.x), m, 1);
                    }
                    if (!valid[k]) m = 0;
                    hitany |= m;
                    if (STATS) st_hits += __popc(m);
                    while (m) {
                        const int j = 31 - __clz(m);
                        m ^= 1u << j;
                        add_term(k, j);
                    }
                }
            } else {
                slot_r = rank;
                __syncwarp();
                if (rel) {
                    cs[0][rank] = c4.x;
                    cs[1][rank] = c4.y;
                    cs[2][rank] = c4.z;
                    cs[3][rank] = -c4.w;
                    float4 co = a.ccoef[cb + lane];
                    cc[rank] = make_float2(co.x, co.y);
                }
                __syncwarp();
                if (STATS) st_tests += (nR - sub + L - 1) / L;
                // a mover's L lanes take every L-th survivor
                unsigned m = 0;
                if (valid[0]) {
#pragma unroll FIELD_UNROLL
                    for (int t = sub; t < nR; t += L) {
                        float d2 = d2of(fsub(cs[0][t], y[0].x), fsub(cs[1][t], y[0].y),
                                        fsub(cs[2][t], y[0].z));
                        m |= (unsigned)(d2 < -cs[3][t]) << t;
                    }
                }
                hitany = m;
                if (STATS) st_hits += __popc(m);
                for (; m; m &= m - 1) add_term(0, __ffs(m) - 1);
            }
            // copies that reached a mover: their density enters the floor of
            // the cut (smooth1.c:460-461), the lane's least one in shared
            // memory (a register more in this loop costs more than it)
            unsigned any = __reduce_or_sync(SKID_FULL, hitany);
            if (rel && ((any >> slot_r) & 1u)) {
                floor_s[w][lane] = min(floor_s[w][lane], f2ord(a.ccoef[cb + lane].z));
                if (a.touched) a.touched[cb + lane] = 1;
            }
        };
        // The leaves that pass under one node, in order; the next one's
        // copies are loaded while one is worked on.
        auto visit_leaves = [&](int lf0, unsigned m) {
            if (!m) return;
            int lf = lf0 + __ffs(m) - 1;
            float4 next = load_copy(lf);
            for (;;) {
                const float4 c4 = next;
                const int cur = lf;
                m &= m - 1;
                if (m) {
                    lf = lf0 + __ffs(m) - 1;
                    next = load_copy(lf);
                }
                leaf_terms(cur, c4);
                if (!m) break;
            }
        };
        unsigned smask;
        int sfirst;
        const int d0 = a.logLeafBase % 5;
        {
            sfirst = 1 << d0;
            smask = __ballot_sync(SKID_FULL, lane < (1 << d0) && reach(sfirst + lane));
        }
        int sp = 0;
        if (sfirst == a.leafBase) {   // at most 16 leaves: they are the first level
            visit_leaves(0, smask);
            sp = -1;
        }
        while (sp >= 0) {
            const unsigned m = __shfl_sync(SKID_FULL, smask, sp);
            if (!m) { --sp; continue; }
            const int node = __shfl_sync(SKID_FULL, sfirst, sp) + __ffs(m) - 1;
            if (lane == sp) smask = m & (m - 1);
            if (STATS) ++st_nodes;
            if (G > NB) {
                float4 blo = a.blo[node], bhi = a.bhi[node];
                if (!__any_sync(SKID_FULL, inside(blo, bhi))) continue;
            }
            const int cf = node << 5;
            unsigned cm = __ballot_sync(SKID_FULL, reach(cf + lane));
            if (cf >= a.leafBase) {
                if (G == 1 && S > 1)
                    cm &= (S == 2 ? 0x55555555u : S == 4 ? 0x11111111u
                           : S == 8 ? 0x01010101u : 0x00010001u) << part;
                visit_leaves(cf - a.leafBase, cm);
            } else if (cm) {
                ++sp;
                if (lane == sp) { smask = cm; sfirst = cf; }
            }
        }
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) {
            ax[0] = fadd(ax[0], __shfl_xor_sync(SKID_FULL, ax[0], o));
            ay[0] = fadd(ay[0], __shfl_xor_sync(SKID_FULL, ay[0], o));
            az[0] = fadd(az[0], __shfl_xor_sync(SKID_FULL, az[0], o));
        }
        if (sub != 0) continue;
#pragma unroll
        for (int k = 0; k < MPL; ++k) {
            if (!valid[k]) continue;
            float fx = ax[k], fy = ay[k], fz = az[k];
            if (G == 1 && S > 1) {
                // the last of the mover's S parts sums them in part order
                float *pa = a.part_acc + 3 * ((size_t)slot[k] * S + part);
                pa[0] = fx;
                pa[1] = fy;
                pa[2] = fz;
                __threadfence();
                if (atomicAdd(&a.part_cnt[slot[k]], 1) != S - 1) continue;
                __threadfence();
                fx = fy = fz = 0.0f;
                for (int p = 0; p < S; ++p) {
                    const float *q = a.part_acc + 3 * ((size_t)slot[k] * S + p);
                    fx = fadd(fx, __ldcg(q));
                    fy = fadd(fy, __ldcg(q + 1));
                    fz = fadd(fz, __ldcg(q + 2));
                }
                a.part_cnt[slot[k]] = 0;
            }
            if (a.acc_out) {
                a.acc_out[3 * (size_t)slot[k] + 0] = fx;
                a.acc_out[3 * (size_t)slot[k] + 1] = fy;
                a.acc_out[3 * (size_t)slot[k] + 2] = fz;
            }
            if (a.fStep > 0.0f) {
                // kdMoveParticles (kd.c:711-728)
                float3 yk = y[k];
                float s2 = d2of(fx, fy, fz);
                float ai = sqrtf(s2);
                ai = ai > 0.0f ? __fdiv_rn(a.fStep, ai) : 0.0f;
                yk.x = fsub(yk.x, fmul(ai, fx));
                yk.y = fsub(yk.y, fmul(ai, fy));
                yk.z = fsub(yk.z, fmul(ai, fz));
                if (yk.x > a.wrapHi.x) yk.x = fsub(yk.x, a.period.x);
                if (yk.x <= a.wrapLo.x) yk.x = fadd(yk.x, a.period.x);
                if (yk.y > a.wrapHi.y) yk.y = fsub(yk.y, a.period.y);
                if (yk.y <= a.wrapLo.y) yk.y = fadd(yk.y, a.period.y);
                if (yk.z > a.wrapHi.z) yk.z = fsub(yk.z, a.period.z);
                if (yk.z <= a.wrapLo.z) yk.z = fadd(yk.z, a.period.z);
                a.mpos[mi[k]] = make_float4(yk.x, yk.y, yk.z, yp[k].w);
            }
        }
    }
    if (a.floor) {
        const unsigned least = __reduce_min_sync(SKID_FULL, floor_s[w][lane]);
        if (lane == 0 && least < *(volatile unsigned *)a.floor) atomicMin(a.floor, least);
    }
    if (STATS && a.stats) {
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            st_tests += __shfl_xor_sync(SKID_FULL, st_tests, o);
            st_hits += __shfl_xor_sync(SKID_FULL, st_hits, o);
        }
        if (lane == 0) {
            atomicAdd(&a.stats[0], st_nodes);
            atomicAdd(&a.stats[1], st_leaves);
            atomicAdd(&a.stats[2], st_tests);
            atomicAdd(&a.stats[3], st_hits);
        }
    }
}

}  // namespace

cudaError_t density_gather(const Tree &t, const float *ball2_sorted, float3 L, bool per,
                           float *rho_sorted, int *d_work, cudaStream_t st)
{
    if (t.n <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(d_work, 0, sizeof(int), st);
    if (e) return e;
    int perSM = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, density_kernel, G_WARPS * 32, 0);
    if (perSM < 1) perSM = 1;
    int blocks = num_sms() * perSM;
    int need = (t.nLeaf + G_WARPS - 1) / G_WARPS;
    if (blocks > need) blocks = need;
    float3 hL = make_float3(0.5f * L.x, 0.5f * L.y, 0.5f * L.z);
    int subShift = 0;
    while (subShift < 5 && (2 << subShift) <= t.leafBase) ++subShift;
    density_kernel<<<blocks, G_WARPS * 32, 0, st>>>(t.view(), ball2_sorted, L, hL, per, subShift, 0.0f,
                                                    rho_sorted, d_work); skid::note_launch();
    return cudaGetLastError();
}

template <int G, bool STATS>
static cudaError_t launch_field_t(const FieldArgs &a, int max_movers, cudaStream_t st)
{
    int perSM = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, field_kernel<G, STATS>, G_WARPS * 32, 0);
    if (perSM < 1) perSM = 1;
    int blocks = num_sms() * perSM;
    int need = ((max_movers + G - 1) / G + G_WARPS - 1) / G_WARPS;
    if (blocks > need) blocks = need;
    if (blocks < 1) blocks = 1;
    field_kernel<G, STATS><<<blocks, G_WARPS * 32, 0, st>>>(a); skid::note_launch();
    return cudaGetLastError();
}

// Work counters compiled in only when asked for (they cost registers).
template <int G>
static cudaError_t launch_field(const FieldArgs &a, int max_movers, cudaStream_t st)
{
    return a.stats ? launch_field_t<G, true>(a, max_movers, st) : launch_field_t<G, false>(a, max_movers, st);
}

// The move alone (kdMoveParticles, kd.c:702-732) from a field written by
// field_kernel with fStep = 0: the unfused form, a separate gradient pass.
__global__ void move_kernel(FieldArgs a, const float *__restrict__ acc, float fStep, int cap)
{
    const int nA = *a.d_nA;
    for (int slot = blockIdx.x * blockDim.x + threadIdx.x; slot < nA && slot < cap;
         slot += gridDim.x * blockDim.x) {
        int mi = a.act[slot];
        if (mi < 0 || mi >= cap) {
            set_status(a.d_status, ST_BADSTATE);
            continue;
        }
        float4 yp = a.mpos[mi];
        float3 y = make_float3(yp.x, yp.y, yp.z);
        float ax = acc[3 * (size_t)slot], ay = acc[3 * (size_t)slot + 1], az = acc[3 * (size_t)slot + 2];
        float s = d2of(ax, ay, az);
        float ai = sqrtf(s);
        ai = ai > 0.0f ? __fdiv_rn(fStep, ai) : 0.0f;
        y.x = fsub(y.x, fmul(ai, ax));
        y.y = fsub(y.y, fmul(ai, ay));
        y.z = fsub(y.z, fmul(ai, az));
        if (y.x > a.wrapHi.x) y.x = fsub(y.x, a.period.x);
        if (y.x <= a.wrapLo.x) y.x = fadd(y.x, a.period.x);
        if (y.y > a.wrapHi.y) y.y = fsub(y.y, a.period.y);
        if (y.y <= a.wrapLo.y) y.y = fadd(y.y, a.period.y);
        if (y.z > a.wrapHi.z) y.z = fsub(y.z, a.period.z);
        if (y.z <= a.wrapLo.z) y.z = fadd(y.z, a.period.z);
        a.mpos[mi] = make_float4(y.x, y.y, y.z, yp.w);
    }
}

cudaError_t move_movers(const FieldArgs &a, const float *acc, float fStep, int max_movers,
                        cudaStream_t st)
{
    if (max_movers <= 0) return cudaSuccess;
    move_kernel<<<grid_for(max_movers), 256, 0, st>>>(a, acc, fStep, max_movers); note_launch();
    return cudaGetLastError();
}

cudaError_t field_move(const FieldArgs &a, int max_movers, cudaStream_t st)
{
    if (max_movers <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(a.d_work, 0, sizeof(int), st);
    if (e) return e;
    switch (a.G) {
    case 64: return launch_field<64>(a, max_movers, st);
    case 1: return launch_field<1>(a, max_movers, st);
    case 4: return launch_field<4>(a, max_movers, st);
    case 8: return launch_field<8>(a, max_movers, st);
    case 16: return launch_field<16>(a, max_movers, st);
    default: return launch_field<32>(a, max_movers, st);
    }
}

}  // namespace skid
