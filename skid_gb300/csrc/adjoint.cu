// Adjoint (reverse-mode) kernels of the SPH density and of the group
// potential energy with respect to particle positions.  No reference
// counterpart: the reference evaluates these quantities (smooth1.c:132-276,
// grav.c:8-60) but never differentiates them.
//
// Density.  With the neighbour sets of skid_density held fixed,
//   L = sum_i w_i rho_i = sum_i sum_{j in B(i)} P_ij W(r_ij, h_i),
//   P_ij = (w_i m_j + w_j m_i) / 2,  h_i^2 = fBall2_i / 4,
// B(i) the ball of i (self included), W the M4 kernel (1/(pi h^3)) f(q).
// Differentiating each term in r_ij and in h_i (h_i = |x_i - x_K(i)|/2,
// K(i) the k-th neighbour, the one at distance^2 == fBall2_i):
//   dW/dr = (1/(pi h^5)) F(q) r,         F = f'(q)/q = -3 + 9q/4 (q<1),
//                                                      -3(2-q)^2/(4q) (q<2)
//   dW/dh = -(1/(pi h^4)) g(q),          g = 3f + q f' = 3 - 15q^2/2 + 9q^3/2 (q<1),
//                                                        3(2-q)^2 (1-q)/2 (q<2)
// so dL/dx_p gets  P F(q)/(pi h^5) (x_p - x_j)  for every pair it is an end
// of (in the frame and with the h of the ball that holds the pair), and
// H_i (x_i - x_K)/(4 h_i) at i, minus the same at K(i), with
// H_i = sum_{j in B(i)} P_ij dW/dh (r_ij, h_i).  F is the reference's move
// field profile (smooth1.c:447-459); the move field itself is minus the
// gradient of the density field rho_f(y) = sum_j m_j W(|y - x_j|, h_j) at the
// mover, i.e. the query-position adjoint with a unit cotangent, which the
// move kernel computes.
//
// Two ways to find the pairs: walk the scatterer tree again (the same walk
// as the density gather; each particle gathers both halves and needs atomics
// only for the h term of its k-th neighbour), or gather every ball's list
// once into memory (n x (k + slack) indices) and scatter from the lists.
//
// Potential energy of a group g (the pair potential of kdCellPot, grav.c:8-36,
// grav.h:11-31, on member coordinates relative to the group's reference
// point as in kdUnbind, kd.c:1338-1352):
//   E_g = -1/2 sum_{i != j} G m_i m_j psi(r_ij, eps_i + eps_j)
//   dE_g/dx_i = -G m_i sum_{j != i} m_j (psi'(r_ij)/r_ij) (x_i - x_j)
// psi'/r follows from differentiating the spline polynomials (Hernquist &
// Katz 1989): (2/e)^3 (-4/3 + 6u^2/5 - u^3/2) for u = 2r/e < 1,
// 1/(15 r^3) + (2/e)^3 (-8/3 + 3u - 6u^2/5 + u^3/6) for u < 2, -1/r^3 beyond;
// Plummer -(r^2 + e^2/4)^(-3/2).  Pair sums are FP32; the per-group energy
// total is FP64.
#include <algorithm>
#include <cfloat>
#include <vector>

#include "ctx.h"

namespace skid {

namespace {

constexpr int A_WARPS = 4;
constexpr float INV_PI = 0.318309886183790671538f;

__device__ __forceinline__ float img_shift(float x, int s, float L)
{
    return s == 0 ? x : (s < 0 ? fsub(x, L) : fadd(x, L));
}

// F(q) = f'(q)/q of the M4 kernel, from q^2.
__device__ __forceinline__ float kern_F(float q2)
{
    float q = sqrtf(q2);
    if (q2 < 1.0f) return -3.0f + 2.25f * q;
    float t = 2.0f - q;
    return -0.75f * t * t / q;
}

// g(q) = 3 f(q) + q f'(q), from q^2.
__device__ __forceinline__ float kern_g(float q2)
{
    float q = sqrtf(q2);
    if (q2 < 1.0f) return 3.0f - 7.5f * q2 + 4.5f * q2 * q;
    float t = 2.0f - q;
    return 1.5f * t * t * (1.0f - q);
}

__device__ __forceinline__ void add3(float *g, float s, float x, float y, float z)
{
    g[0] += s * x;
    g[1] += s * y;
    g[2] += s * z;
}

__device__ __forceinline__ void atomic_add3(float *g, float x, float y, float z)
{
    atomicAdd(g, x);
    atomicAdd(g + 1, y);
    atomicAdd(g + 2, z);
}

// Per-particle constants of its own ball: 1/(pi h^5), -1/(pi h^4), 1/(4h).
struct Ball {
    float b, ih2, c5, c4, q4;
};

__device__ __forceinline__ Ball ball_of(float b)
{
    Ball r;
    r.b = b;
    r.ih2 = 4.0f / b;
    float ih = sqrtf(r.ih2);
    r.c4 = -INV_PI * r.ih2 * r.ih2;
    r.c5 = INV_PI * r.ih2 * r.ih2 * ih;
    r.q4 = 0.25f * ih;
    return r;
}

// The h term of particle i once H_i is complete: +c (x_i - x_K) at i, -c at K.
__device__ __forceinline__ void h_term(float *gi, float *grad, int K, float H, const Ball &bi,
                                       float kx, float ky, float kz)
{
    float c = H * bi.q4;
    add3(gi, c, kx, ky, kz);
    atomic_add3(grad + 3 * (size_t)K, -c * kx, -c * ky, -c * kz);
}

__global__ void __launch_bounds__(A_WARPS * 32)
density_adjoint_walk(TreeView t, const float *__restrict__ ball2, const float *__restrict__ wsort,
                     float3 L, float3 hL, bool per, int subShift, float *__restrict__ grad,
                     int *work, unsigned *status)
{
    __shared__ float4 cpos[A_WARPS][SKID_LEAF];
    __shared__ float4 caux[A_WARPS][SKID_LEAF];   // fBall2, 1/h^2, 1/(pi h^5), w
    __shared__ int cslot[A_WARPS][SKID_LEAF];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int rootLo = t.leafBase >> subShift;
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
        Ball bi = ball_of(ball2[valid ? qi : base]);
        float wi = wsort[valid ? qi : base], mi = qp.w;
        // the query leaf's box (its points) and largest ball
        const float4 qlo = t.lo[t.leafBase + leaf], qhi = t.hi[t.leafBase + leaf];
        float g[3] = {0.0f, 0.0f, 0.0f};
        float H = 0.0f;
        int K = -1;
        float kx = 0.0f, ky = 0.0f, kz = 0.0f;
        int cp = 1;
        for (;;) {
            if (cp >= rootLo) {
                // the subtree's leaves one per lane against the query box, then
                // each passing leaf in order; at a leaf only candidates whose
                // distance to the query box is below max(their ball, the
                // largest query ball) can enter either half
                const int first = cp << subShift;
                bool pass = false;
                if (lane < (1 << subShift) && first + lane - t.leafBase < t.nLeaf) {
                    float4 bl = t.lo[first + lane];
                    pass = boxbox_lb(qlo, qhi, bl, t.hi[first + lane], L, per) < fmaxf(qlo.w, bl.w);
                }
                for (unsigned lm = __ballot_sync(SKID_FULL, pass); lm; lm &= lm - 1) {
                    const int node = first + __ffs(lm) - 1;
                    float4 blo = t.lo[node], bhi = t.hi[node];
                    bool want = box_lb(q, blo, bhi, L, per) < fmaxf(bi.b, blo.w);
                    if (!__any_sync(SKID_FULL, want)) continue;
                    const int cb = (node - t.leafBase) * SKID_LEAF;
                    const int cnt = min(SKID_LEAF, t.n - cb);
                    bool rel = false;
                    float4 c4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    float b = 0.0f;
                    if (lane < cnt) {
                        c4 = t.pos[cb + lane];
                        b = ball2[cb + lane];
                        rel = box_lb(make_float3(c4.x, c4.y, c4.z), qlo, qhi, L, per) < fmaxf(b, qlo.w);
                    }
                    const unsigned R = __ballot_sync(SKID_FULL, rel);
                    const int nR = __popc(R);
                    __syncwarp();
                    if (rel) {
                        const int k = __popc(R & ((1u << lane) - 1u));
                        float ih2 = 4.0f / b;
                        cpos[w][k] = c4;
                        caux[w][k] = make_float4(b, ih2, INV_PI * ih2 * ih2 * sqrtf(ih2), wsort[cb + lane]);
                        cslot[w][k] = cb + lane;
                    }
                    __syncwarp();
                    if (!want) continue;
                    int cx = img_class(q.x, blo.x, bhi.x, hL.x);
                    int cy = img_class(q.y, blo.y, bhi.y, hL.y);
                    int cz = img_class(q.z, blo.z, bhi.z, hL.z);
                    bool slow = (cx == 2) | (cy == 2) | (cz == 2);
                    float sx = img_shift(q.x, cx, L.x), sy = img_shift(q.y, cy, L.y),
                          sz = img_shift(q.z, cz, L.z);
                    for (int j = 0; j < nR; ++j) {
                        float4 cj = cpos[w][j];
                        float4 aj = caux[w][j];
                        // (ax, ay, az): x_i - x_j in i's frame; (bx, by, bz): in j's frame
                        float ax, ay, az, bx, by, bz;
                        if (slow) {
                            ax = img_dx(q.x, cj.x, L.x, hL.x);
                            ay = img_dx(q.y, cj.y, L.y, hL.y);
                            az = img_dx(q.z, cj.z, L.z, hL.z);
                            bx = -img_dx(cj.x, q.x, L.x, hL.x);
                            by = -img_dx(cj.y, q.y, L.y, hL.y);
                            bz = -img_dx(cj.z, q.z, L.z, hL.z);
                        } else {
                            ax = fsub(sx, cj.x);
                            ay = fsub(sy, cj.y);
                            az = fsub(sz, cj.z);
                            bx = -fsub(img_shift(cj.x, -cx, L.x), q.x);
                            by = -fsub(img_shift(cj.y, -cy, L.y), q.y);
                            bz = -fsub(img_shift(cj.z, -cz, L.z), q.z);
                        }
                        float dik = d2of(ax, ay, az);
                        float dki = d2of(bx, by, bz);
                        float P = 0.5f * (wi * cj.w + aj.w * mi);
                        if (dik < bi.b) {
                            float q2 = dik * bi.ih2;
                            add3(g, P * bi.c5 * kern_F(q2), ax, ay, az);
                            H += P * bi.c4 * kern_g(q2);
                        }
                        const int sj = cslot[w][j];
                        if (dik == bi.b && sj != qi) {
                            K = sj;
                            kx = ax; ky = ay; kz = az;
                        }
                        if (dki < aj.x) add3(g, P * aj.z * kern_F(dki * aj.y), bx, by, bz);
                    }
                }
            } else {
                float4 blo = t.lo[cp], bhi = t.hi[cp];
                bool want = box_lb(q, blo, bhi, L, per) < fmaxf(bi.b, blo.w);
                if (__any_sync(SKID_FULL, want)) { cp <<= 1; continue; }
            }
            cp = next_node(cp);
            if (cp == 1) break;
        }
        if (valid) {
            if (K >= 0) h_term(g, grad, K, H, bi, kx, ky, kz);
            else set_status(status, ST_BADSTATE);
            atomic_add3(grad + 3 * (size_t)qi, g[0], g[1], g[2]);
        }
    }
}

// Gather every ball's members (distance^2 <= fBall2, the kNN set with its
// ties) into rows of `cap` sorted-order indices, each in sorted order.
//
// Instruction issue bounds it.  The walk goes as in the density gather: the
// last 2^subShift leaves of a subtree one per lane against the query leaf's
// box, then a leaf's particles one per lane against that box and the largest
// ball of the query leaf.  Where no periodic image can be nearer the survivors
// are tested two to a packed FP32 operation into a mask per lane, from which
// the lane writes its members: 100,000 points, k = 64, 539 to 235 us.
__global__ void __launch_bounds__(A_WARPS * 32)
ball_lists(TreeView t, const float *__restrict__ ball2, float3 L, float3 hL, bool per, int subShift,
           float zero_arg, int cap, int *__restrict__ nbr, int *__restrict__ ncnt, int *work,
           unsigned *status)
{
    __shared__ __align__(16) float cand_s[A_WARPS][3][SKID_LEAF];
    __shared__ int slot_s[A_WARPS][SKID_LEAF];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float (*cs)[SKID_LEAF] = cand_s[w];
    const int rootLo = t.leafBase >> subShift;
    const f32x2 zero = pack2(zero_arg, zero_arg), neg1 = pack2(-1.0f, -1.0f);
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
        float bi = valid ? ball2[qi] : -1.0f;
        // the query leaf's box and its largest ball
        const float4 qlo = t.lo[t.leafBase + leaf], qhi = t.hi[t.leafBase + leaf];
        const float bmax = __uint_as_float(__reduce_max_sync(SKID_FULL, __float_as_uint(fmaxf(bi, 0.0f))));
        const f32x2 nqx = pack2(-q.x, -q.x), nqy = pack2(-q.y, -q.y), nqz = pack2(-q.z, -q.z);
        const f32x2 b2 = pack2(bi, bi);
        int c = 0;
        int *row = nbr + (size_t)(valid ? qi : 0) * cap;
        int cp = 1;
        for (;;) {
            const float4 nlo = t.lo[cp], nhi = t.hi[cp];
            const bool dnode = !per || boxes_direct(qlo, qhi, nlo, nhi, hL);
            if (cp < rootLo) {
                if ((dnode ? gap2(xyz(qlo), xyz(qhi), nlo, nhi) : boxbox_lb(qlo, qhi, nlo, nhi, L, per)) <= bmax) {
                    cp <<= 1;
                    continue;
                }
            } else {
                const int first = cp << subShift;
                bool pass = false;
                if (lane < (1 << subShift) && first + lane - t.leafBase < t.nLeaf) {
                    const float4 bl = t.lo[first + lane], bh = t.hi[first + lane];
                    pass = (dnode ? gap2(xyz(qlo), xyz(qhi), bl, bh) : boxbox_lb(qlo, qhi, bl, bh, L, per)) <= bmax;
                }
                for (unsigned lm = __ballot_sync(SKID_FULL, pass); lm; lm &= lm - 1) {
                    const int node = first + __ffs(lm) - 1;
                    const float4 blo = t.lo[node], bhi = t.hi[node];
                    const bool direct = dnode || boxes_direct(qlo, qhi, blo, bhi, hL);
                    const bool want = (direct ? gap2(q, q, blo, bhi) : box_lb(q, blo, bhi, L, per)) <= bi;
                    if (!__any_sync(SKID_FULL, want)) continue;
                    const int cb = (node - t.leafBase) * SKID_LEAF;
                    bool rel = false;
                    float4 cj = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (cb + lane < t.n) {
                        cj = t.pos[cb + lane];
                        rel = (direct ? gap2(xyz(cj), xyz(cj), qlo, qhi) : box_lb(xyz(cj), qlo, qhi, L, per)) <= bmax;
                    }
                    const unsigned R = __ballot_sync(SKID_FULL, rel);
                    if (R == 0) continue;
                    const int nR = __popc(R);
                    const int rank = __popc(R & ((1u << lane) - 1u));
                    // survivors in reverse order of rank, so that the first
                    // member is the highest bit; above them no members
                    const int slot = rel ? nR - 1 - rank : nR + lane - rank;
                    __syncwarp();
                    cs[0][slot] = rel ? cj.x : INFINITY;
                    cs[1][slot] = cj.y;
                    cs[2][slot] = cj.z;
                    slot_s[w][slot] = cb + lane;
                    __syncwarp();
                    unsigned in = 0;
                    if (direct) {
                        unsigned out = 0;
                        for (int j = (nR - 1) & ~3; j >= 0; j -= 4) {
                            const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(&cs[0][j]);
                            const ulonglong2 Y = *reinterpret_cast<const ulonglong2 *>(&cs[1][j]);
                            const ulonglong2 Z = *reinterpret_cast<const ulonglong2 *>(&cs[2][j]);
#pragma unroll
                            for (int h = 1; h >= 0; --h) {
                                const f32x2 dx = add2(h ? X.y : X.x, nqx), dy = add2(h ? Y.y : Y.x, nqy),
                                            dz = add2(h ? Z.y : Z.x, nqz);
                                const f32x2 d = add2(add2(sq2(dx, zero), sq2(dy, zero)), sq2(dz, zero));
                                const float2 a = unpack2(fma2(d, neg1, b2));   // negative: outside
                                out = __funnelshift_l(__float_as_uint(a.y), out, 1);
                                out = __funnelshift_l(__float_as_uint(a.x), out, 1);
                            }
                        }
                        in = ~out & (nR < 32 ? (1u << nR) - 1u : ~0u);
                    } else if (want) {
                        for (int j = 0; j < nR; ++j) {
                            const float d = d2of(img_dx(q.x, cs[0][j], L.x, hL.x), img_dx(q.y, cs[1][j], L.y, hL.y),
                                                 img_dx(q.z, cs[2][j], L.z, hL.z));
                            if (d <= bi) in |= 1u << j;
                        }
                    }
                    for (; in; ++c) {
                        const int j = 31 - __clz(in);
                        in ^= 1u << j;
                        if (c < cap) row[c] = slot_s[w][j];
                    }
                }
            }
            cp = next_node(cp);
            if (cp == 1) break;
        }
        if (valid) {
            if (c > cap) set_status(status, ST_OVERFLOW);
            ncnt[qi] = min(c, cap);
        }
    }
}

// Scatter form over the stored lists: each (i, j in B(i)) once, both ends.
__global__ void density_adjoint_lists(const float4 *__restrict__ pos, const float *__restrict__ ball2,
                                      const float *__restrict__ wsort, int n, float3 L, float3 hL,
                                      bool per, int cap, const int *__restrict__ nbr,
                                      const int *__restrict__ ncnt, float *__restrict__ grad,
                                      unsigned *status)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4 pi = pos[i];
        Ball bi = ball_of(ball2[i]);
        float wi = wsort[i];
        float g[3] = {0.0f, 0.0f, 0.0f};
        float H = 0.0f;
        int K = -1;
        float kx = 0.0f, ky = 0.0f, kz = 0.0f;
        const int *row = nbr + (size_t)i * cap;
        int c = ncnt[i];
        for (int k = 0; k < c; ++k) {
            int j = row[k];
            float4 pj = pos[j];
            float ax, ay, az;
            if (per) {
                ax = img_dx(pi.x, pj.x, L.x, hL.x);
                ay = img_dx(pi.y, pj.y, L.y, hL.y);
                az = img_dx(pi.z, pj.z, L.z, hL.z);
            } else {
                ax = fsub(pi.x, pj.x);
                ay = fsub(pi.y, pj.y);
                az = fsub(pi.z, pj.z);
            }
            float d = d2of(ax, ay, az);
            if (d == bi.b && j != i) {
                K = j;
                kx = ax; ky = ay; kz = az;
            }
            if (!(d < bi.b)) continue;
            float P = 0.5f * (wi * pj.w + wsort[j] * pi.w);
            float q2 = d * bi.ih2;
            float s = P * bi.c5 * kern_F(q2);
            add3(g, s, ax, ay, az);
            if (j != i) atomic_add3(grad + 3 * (size_t)j, -s * ax, -s * ay, -s * az);
            H += P * bi.c4 * kern_g(q2);
        }
        if (K >= 0) h_term(g, grad, K, H, bi, kx, ky, kz);
        else set_status(status, ST_BADSTATE);
        atomic_add3(grad + 3 * (size_t)i, g[0], g[1], g[2]);
    }
}

__global__ void gather_w(const int *__restrict__ sidx, const float *__restrict__ w_io, int n,
                         float *__restrict__ w_sorted)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        w_sorted[i] = w_io[sidx[i]];
}

__global__ void scatter_grad(const int *__restrict__ sidx, const float *__restrict__ g_sorted, int n,
                             float *__restrict__ g_io)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int o = sidx[i];
        g_io[3 * (size_t)o] = g_sorted[3 * (size_t)i];
        g_io[3 * (size_t)o + 1] = g_sorted[3 * (size_t)i + 1];
        g_io[3 * (size_t)o + 2] = g_sorted[3 * (size_t)i + 2];
    }
}

// ---- group potential energy ----

// psi(r, e) as kdCellPot evaluates it (grav.h:11-31) and psi'(r)/r.
// Beyond the softening (r >= 2h, certain once d2 clears (2h)^2 by the margin
// below) and for Plummer softening, psi comes from the hardware reciprocal
// square root (2 ulp).
__device__ __forceinline__ void pair_psi(float d2, float twoh, int plummer, float &psi, float &gr)
{
    if (plummer || d2 >= twoh * twoh * 1.000001f) {
        float t = rsqrtf(plummer ? d2 + 0.25f * twoh * twoh : d2);
        psi = t;
        gr = -t * t * t;
        return;
    }
    float r = sqrtf(d2);
    if (r < twoh) {
        float dih = 2.0f / twoh;
        float u = r * dih;
        float u2 = u * u;
        float d3 = dih * dih * dih;
        if (u < 1.0f) {
            psi = dih * (1.4f - (2.0f / 3.0f) * u2 + 0.3f * u2 * u2 - 0.1f * u2 * u2 * u);
            gr = d3 * (-4.0f / 3.0f + 1.2f * u2 - 0.5f * u2 * u);
        } else {
            psi = -(1.0f / 15.0f) / r +
                  dih * (1.6f - (4.0f / 3.0f) * u2 + u2 * u - 0.3f * u2 * u2 + (1.0f / 30.0f) * u2 * u2 * u);
            gr = (1.0f / 15.0f) / (d2 * r) + d3 * (-8.0f / 3.0f + 3.0f * u - 1.2f * u2 + (1.0f / 6.0f) * u2 * u);
        }
        return;
    }
    psi = 1.0f / r;
    gr = -psi / d2;
}

__device__ __forceinline__ float wrap_rel(float d, float h)
{
    if (d > h) d = fsub(d, fmul(2.0f, h));
    if (d <= -h) d = fadd(d, fmul(2.0f, h));
    return d;
}

// The pair sums of the selected groups, split into items of PA_TILE rows by
// up to `chunk` columns of one group.  FP32 issue bounds it: per pair 16 FP32
// operations with the gradient, 10 without, and a reciprocal square root.  A
// thread carries two rows in packed FP32 operands (half the issue slots), a
// column read from shared memory serving both; tile pairs whose boxes are
// further apart than the softening run without any test.  Columns are split
// as well as rows because a group's rows alone leave the GPU idle: 24 groups
// of up to 35k members (140k rows, 2.9e9 pairs) gave 14 warps an SM and
// items of 35k columns, 9.9 ms a call with or without the gradient.  Now 2.5
// and 1.75 ms.  A row's sums over each chunk (the potential's Kahan-compensated)
// go to memory, and pa_finish adds them in FP64 in chunk order, rounding to
// float once at the end: the sums do not depend on the order in which blocks
// run.  (The last block to finish a tile's chunks adding them here, a fence
// and a count per item, cost 8 % at short chunks.)
constexpr int PA_TILE = 128;
constexpr int PA_THREADS = PA_TILE / 2;
// Columns per item: 1024 once the pairs make PA_FILL items of that length for
// every SM, halved below until they do, at least 128.  A long walk over columns
// saves partial sums, and leaves SMs idle at the end.  A call's time without /
// with the gradient at 128, 256, 512, 1024 columns (chosen: *), ms:
//   one group of 8,660           .15 / .21*    .16 / .22     .17 / .22     .25 / .30
//   one group of 17,000          .36 / .47*    .39 / .51     .47 / .58     .70 / .85
//   20 groups of up to 19,700    .72 / 1.03    .70 / .93*    .79 / 1.04    .84 / 1.07
//   8 groups of 17,000          1.64 / 2.36   1.56 / 2.18   1.69 / 2.33*  1.94 / 2.43
//   300 groups of 3,000         2.51 / 3.43   2.30 / 3.11   2.25 / 3.00   2.27 / 2.97*
//   4,000 groups of 1,000       5.85 / 9.55   5.23 / 8.75   4.87 / 8.26   4.36 / 7.58*
// A group has at most PA_MAX_CHUNKS (longer ones from 131,072 members on), which
// bounds the memory of its rows' partial sums (20 B each with the gradient, 8 B
// without); 64 took 0.43 / 0.54 for the group of 17,000.
constexpr int PA_CHUNK = 1024, PA_CHUNK_MIN = 128, PA_MAX_CHUNKS = 128;
constexpr long long PA_FILL = 128;
// From PA_SORT_PAIRS pairs an SM (4e8 on 152) where a row meets PA_SORT_COLS
// columns or more, and from PA_SORT_ANY (2e9) in any case, the members are
// packed in Hilbert order: a warp takes the softened pair factor (divides, a
// root) whenever any of its pairs lies inside the softening, and with members
// in file order some pair of 64 does in 40-50 % of the steps of a halo whose
// pairs are 2-3 % inside it; in Hilbert order in 12-20 %, and in a group of
// many tiles most pairs of tiles are beyond the softening as a whole; for 0.1 ms
// of sorting and more with a million rows.  File order / Hilbert order without
// the gradient, ms:
//   one group of 17,000 (2.9e8 pairs)    .35 / .43    20 of up to 19,700 (8.7e8)  .79 / .70
//   8 of 8,660 (6e8)                     .68 / .63    one of 35,000 (1.2e9)      1.21 / .89
//   300 of up to 6,600 (9.3e8)           .78 / .85    8 of 17,000 (2.3e9)        2.22 / 1.70
//   1,000 of up to 4,900 (1.8e9)        1.43 / 1.50   300 of 3,000 (2.7e9)       2.75 / 2.20
constexpr double PA_SORT_PAIRS = 2.6e6, PA_SORT_COLS = 4000.0, PA_SORT_ANY = 1.3e7;
// Rows with this many chunks on average have them added by PA_PARTS warps.
// One / four: one group of 8,660 (68 chunks) with the gradient .228 / .211 ms,
// 150 groups of 1,000 (8) .472 / .492, 4,000 of 1,000 (1) 7.57 / 7.94.
constexpr int PA_PARTS = 4, PA_PARTS_MIN = 16;

struct PotSlot {
    long long item0;            // items of the slots before this one
    long long row0;             // rows of the slots before this one
    long long tile0;            // row tiles of the slots before this one
    long long part0;            // partial sums of the slots before this one
    int g, n, chunk, nchunk;
    float v;
};

struct PotAdjArgs {
    const PotSlot *slots;
    int nslot;
    long long nitems, nrows;
    const int *gstart, *members;
    const float4 *pos4, *vel4;  // (x, y, z, m), (vx, vy, vz, soft)
    const skid_group *rec;
    float3 hP;
    float G;
    int plummer;
    const uint32_t *perm;       // packed row -> row in member order (null: the same)
    float4 *rm;                 // packed rows: position relative to the group's rel, mass
    float *re;                  // packed rows: softening
    int *rio;                   // packed rows: iOrder
    float4 *tlo, *thi;          // per row tile: its box; tlo.w: its largest softening
    long long ntile;
    float2 *pphi;               // per slot, chunk and row: sum_j m_j psi and its compensation,
    float *pgx, *pgy, *pgz;     // (gradient) sum_j m_j psi'/r (x_i - x_j)
    double *eblock;             // per block of pa_finish: its rows' energy
    double *E;                  // per slot (zeroed)
    int *done;                  // such blocks finished per slot (zeroed)
    float *grad;                // 3n by iOrder (zeroed) or null
};

// The slot holding item, row or tile k: the last one that starts at or before
// it by that running sum.
__device__ __forceinline__ int pa_slot(const PotAdjArgs &a, long long k, long long PotSlot::*start)
{
    int lo = 0, hi = a.nslot - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (a.slots[mid].*start <= k) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The same for a whole warp and one k, 32 slots at a time: each step of the
// search is a load that the next one waits for, the most of a call on many
// small groups.
__device__ __forceinline__ int pa_slot_warp(const PotAdjArgs &a, long long k, long long PotSlot::*start)
{
    const int lane = threadIdx.x & 31;
    int lo = 0, count = a.nslot;
    while (count > 1) {
        const int step = (count + 31) / 32;
        const bool before = lane * step < count && (lane == 0 || a.slots[lo + lane * step].*start <= k);
        const int j = 31 - __clz(__ballot_sync(SKID_FULL, before));
        lo += j * step;
        count = min(step, count - j * step);
    }
    return lo;
}

__device__ __forceinline__ float3 pa_rel(const PotAdjArgs &a, const PotSlot &S, float4 p)
{
    const float *rel = a.rec[S.g].rel;
    return make_float3(wrap_rel(fsub(p.x, rel[0]), a.hP.x), wrap_rel(fsub(p.y, rel[1]), a.hP.y),
                       wrap_rel(fsub(p.z, rel[2]), a.hP.z));
}

// The largest |coordinate| of any row (order-preserving bits, zeroed before).
__global__ void pa_extent(PotAdjArgs a, unsigned *ext)
{
    float m = 0.0f;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < a.nrows;
         k += (long long)gridDim.x * blockDim.x) {
        const PotSlot S = a.slots[pa_slot(a, k, &PotSlot::row0)];
        const float3 r = pa_rel(a, S, a.pos4[a.members[a.gstart[S.g] + (int)(k - S.row0)]]);
        m = fmaxf(m, fmaxf(fabsf(r.x), fmaxf(fabsf(r.y), fabsf(r.z))));
    }
    const unsigned u = __reduce_max_sync(SKID_FULL, __float_as_uint(m));
    if ((threadIdx.x & 31) == 0) atomicMax(ext, u);
}

// Sort keys: the slot, then the Hilbert index of the relative position on a
// 2^13 grid.
constexpr int PA_KEY_BITS = 39;

__global__ void pa_keys(PotAdjArgs a, const unsigned *ext, uint64_t *keys, uint32_t *vals)
{
    const float R = fmaxf(__uint_as_float(*ext), 1e-30f), sc = 4095.5f / R;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < a.nrows;
         k += (long long)gridDim.x * blockDim.x) {
        const int s = pa_slot(a, k, &PotSlot::row0);
        const PotSlot S = a.slots[s];
        const float3 r = pa_rel(a, S, a.pos4[a.members[a.gstart[S.g] + (int)(k - S.row0)]]);
        auto cell = [&](float x) {
            return (uint32_t)fminf(fmaxf((x + R) * sc, 0.0f), 8191.0f);
        };
        keys[k] = ((uint64_t)s << PA_KEY_BITS) | hilbert3<13>(cell(r.x), cell(r.y), cell(r.z));
        vals[k] = (uint32_t)k;
    }
}

// Pack the rows, a warp to each tile of PA_TILE, and the tile's box and largest
// softening with them (one launch: a call on a small group is launches).
__global__ void pa_pack(PotAdjArgs a)
{
    const int lane = threadIdx.x & 31;
    const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long t = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5); t < a.ntile;
         t += nw) {
        const PotSlot S = a.slots[pa_slot_warp(a, t, &PotSlot::tile0)];
        float4 lo = make_float4(FLT_MAX, FLT_MAX, FLT_MAX, 0.0f);
        float4 hi = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, 0.0f);
        const int i0 = (int)(t - S.tile0) * PA_TILE + lane, gs = a.gstart[S.g];
#pragma unroll
        for (int q = 0; q < PA_TILE / 32; ++q) {
            const int i = i0 + 32 * q;
            if (i >= S.n) continue;
            const long long k = S.row0 + i;
            const int io = a.members[gs + (a.perm ? (int)(a.perm[k] - S.row0) : i)];
            const float4 p = a.pos4[io];
            const float e = a.vel4[io].w;
            const float3 r = pa_rel(a, S, p);
            a.rm[k] = make_float4(r.x, r.y, r.z, p.w);
            a.re[k] = e;
            a.rio[k] = io;
            lo.x = fminf(lo.x, r.x); lo.y = fminf(lo.y, r.y); lo.z = fminf(lo.z, r.z);
            hi.x = fmaxf(hi.x, r.x); hi.y = fmaxf(hi.y, r.y); hi.z = fmaxf(hi.z, r.z);
            lo.w = fmaxf(lo.w, e);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            lo.x = fminf(lo.x, __shfl_xor_sync(SKID_FULL, lo.x, o));
            lo.y = fminf(lo.y, __shfl_xor_sync(SKID_FULL, lo.y, o));
            lo.z = fminf(lo.z, __shfl_xor_sync(SKID_FULL, lo.z, o));
            hi.x = fmaxf(hi.x, __shfl_xor_sync(SKID_FULL, hi.x, o));
            hi.y = fmaxf(hi.y, __shfl_xor_sync(SKID_FULL, hi.y, o));
            hi.z = fmaxf(hi.z, __shfl_xor_sync(SKID_FULL, hi.z, o));
            lo.w = fmaxf(lo.w, __shfl_xor_sync(SKID_FULL, lo.w, o));
        }
        if (lane == 0) {
            a.tlo[t] = lo;
            a.thi[t] = hi;
        }
    }
}

// A thread's two rows, packed: position, the Kahan-compensated sum_j m_j psi
// and sum_j m_j psi'/r (x_i - x_j).
struct PaRows {
    f32x2 x, y, z;
    f32x2 phi, phic, gx, gy, gz;
};

__device__ __forceinline__ float rsqrt_ftz(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Both rows' term for one column, given psi (and psi'/r) of each.
template <bool GRAD>
__device__ __forceinline__ void pa_add(PaRows &w, f32x2 dx, f32x2 dy, f32x2 dz, f32x2 m, f32x2 psi,
                                       f32x2 gr)
{
    const f32x2 y = fma2(m, psi, w.phic);       // phic holds minus the compensation
    const f32x2 tt = add2(w.phi, y);
    w.phic = sub2(y, sub2(tt, w.phi));
    w.phi = tt;
    if (GRAD) {
        const f32x2 c = mul2(m, gr);
        w.gx = fma2(c, dx, w.gx);
        w.gy = fma2(c, dy, w.gy);
        w.gz = fma2(c, dz, w.gz);
    }
}

// A column in shared memory: (-x, -x, -y, -y), (-z, -z, m, m), both halves of
// the packed operands.
struct PaCol {
    ulonglong2 xy, zm;
};

// The sum of a tile's rows' values in row order, warps first: thread t holds
// row t (and, Q = 2, row t + PA_TILE / 2).
template <int Q>
__device__ __forceinline__ double pa_tile_sum(const double (&v)[Q])
{
    __shared__ double red[PA_TILE / 32];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        double x = v[q];
#pragma unroll
        for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(SKID_FULL, x, o);
        if ((threadIdx.x & 31) == 0) red[(threadIdx.x >> 5) + q * (PA_TILE / 32 / Q)] = x;
    }
    __syncthreads();
    double t = red[0];
    for (int k = 1; k < PA_TILE / 32; ++k) t += red[k];
    return t;
}

// A row's gradient by iOrder from its sums v over all columns, and its share
// -1/2 G m phi of the energy.
template <bool GRAD>
__device__ __forceinline__ double pa_row_out(const PotAdjArgs &a, const PotSlot &S, float m, int io,
                                             const double *v)
{
    if (GRAD) {
        const float c = -a.G * m * S.v;
        float *o = a.grad + 3 * (size_t)io;
#pragma unroll
        for (int d = 0; d < 3; ++d) o[d] = c * (float)v[d + 1];
    }
    return -0.5 * (double)a.G * (double)m * (double)(float)v[0];
}

// ONE: every group of the call is one tile (and one chunk), and its energy and
// gradient are written here: no pa_finish, the most of a call on small groups
// being launches (100 groups of 50: 0.076 / 0.094 ms a call without / with the
// gradient, 0.071 / 0.086 so).
template <bool GRAD, bool ONE>
__global__ void __launch_bounds__(PA_THREADS) potential_adjoint_kernel(PotAdjArgs a)
{
    __shared__ PaCol sc[PA_TILE];
    __shared__ float ss[PA_TILE];
    const int tid = threadIdx.x;
    for (long long it = blockIdx.x; it < a.nitems; it += gridDim.x) {
        const int slot = pa_slot_warp(a, it, &PotSlot::item0);
        const PotSlot S = a.slots[slot];
        const int tile = (int)(it - S.item0) / S.nchunk, ch = (int)(it - S.item0) - tile * S.nchunk;
        const int n = S.n;
        const float4 *rm = a.rm + S.row0;
        const float *re = a.re + S.row0;
        const int i0 = tile * PA_TILE + tid, i1 = i0 + PA_THREADS;
        const float4 alo = a.tlo[S.tile0 + tile], ahi = a.thi[S.tile0 + tile];
        // rows past the end repeat the last member and are not stored
        const float4 q0 = rm[min(i0, n - 1)], q1 = rm[min(i1, n - 1)];
        const float e0 = re[min(i0, n - 1)], e1 = re[min(i1, n - 1)];
        PaRows w;
        w.x = pack2(q0.x, q1.x);
        w.y = pack2(q0.y, q1.y);
        w.z = pack2(q0.z, q1.z);
        w.phi = w.phic = w.gx = w.gy = w.gz = 0ull;
        const int c0 = ch * S.chunk, c1 = min(n, c0 + S.chunk);
        for (int jb = c0; jb < c1; jb += PA_TILE) {
            const int cnt = min(PA_TILE, c1 - jb);
            const float4 blo = a.tlo[S.tile0 + jb / PA_TILE], bhi = a.thi[S.tile0 + jb / PA_TILE];
            __syncthreads();
            for (int c = tid; c < cnt; c += PA_THREADS) {
                const float4 r = rm[jb + c];
                PaCol o;
                o.xy = make_ulonglong2(pack2(-r.x, -r.x), pack2(-r.y, -r.y));
                o.zm = make_ulonglong2(pack2(-r.z, -r.z), pack2(r.w, r.w));
                sc[c] = o;
                ss[c] = re[jb + c];
            }
            __syncthreads();
            // far is at or above every pair's (2h)^2 (1 + 1e-6) in the tile
            // pair (infinite for Plummer softening): beyond it pair_psi is
            // the hardware 1/r, taken without forming the pair's softening
            float far = INFINITY;
            if (!a.plummer) far = fmaxf((alo.w + blo.w) * (alo.w + blo.w) * 1.000001f, 1e-30f);
            // the squared gap between the tiles' boxes: float subtraction,
            // product and sum are monotonic, so no pair's d2 is below it
            const float gx = fmaxf(fmaxf(blo.x - ahi.x, alo.x - bhi.x), 0.0f);
            const float gy = fmaxf(fmaxf(blo.y - ahi.y, alo.y - bhi.y), 0.0f);
            const float gz = fmaxf(fmaxf(blo.z - ahi.z, alo.z - bhi.z), 0.0f);
            if (__fmaf_rn(gz, gz, __fmaf_rn(gx, gx, gy * gy)) >= far) {
                // every pair beyond the softening
#pragma unroll 4
                for (int c = 0; c < cnt; ++c) {
                    const PaCol o = sc[c];
                    const f32x2 dx = add2(w.x, o.xy.x), dy = add2(w.y, o.xy.y), dz = add2(w.z, o.zm.x);
                    const float2 d2 = unpack2(fma2(dz, dz, fma2(dx, dx, mul2(dy, dy))));
                    const f32x2 psi = pack2(rsqrt_ftz(d2.x), rsqrt_ftz(d2.y));
                    f32x2 gr = 0ull;
                    if (GRAD) gr = mul2(mul2(psi, psi), mul2(psi, 0xbf800000bf800000ull));
                    pa_add<GRAD>(w, dx, dy, dz, o.zm.y, psi, gr);
                }
            } else {
                // a step without any pair inside the softening takes the same
                // form (a member with itself, at d2 = 0, is inside)
                const int s0 = i0 - jb, s1 = i1 - jb;   // the rows' own columns, if here
#pragma unroll 2
                for (int c = 0; c < cnt; ++c) {
                    const PaCol o = sc[c];
                    const f32x2 dx = add2(w.x, o.xy.x), dy = add2(w.y, o.xy.y), dz = add2(w.z, o.zm.x);
                    const float2 d2 = unpack2(fma2(dz, dz, fma2(dx, dx, mul2(dy, dy))));
                    f32x2 psi = pack2(rsqrt_ftz(d2.x), rsqrt_ftz(d2.y)), gr = 0ull;
                    if (GRAD) gr = mul2(mul2(psi, psi), mul2(psi, 0xbf800000bf800000ull));
                    if (!(d2.x >= far && d2.y >= far)) {
                        float2 p = unpack2(psi), q = unpack2(gr);
                        if (!(d2.x >= far)) pair_psi(d2.x, e0 + ss[c], a.plummer, p.x, q.x);
                        if (!(d2.y >= far)) pair_psi(d2.y, e1 + ss[c], a.plummer, p.y, q.y);
                        // no pair of a member with itself
                        if (c == s0) p.x = q.x = 0.0f;
                        if (c == s1) p.y = q.y = 0.0f;
                        psi = pack2(p.x, p.y);
                        gr = pack2(q.x, q.y);
                    }
                    pa_add<GRAD>(w, dx, dy, dz, o.zm.y, psi, gr);
                }
            }
        }
        const float2 phi = unpack2(w.phi), phic = unpack2(w.phic);
        const float2 hx = unpack2(w.gx), hy = unpack2(w.gy), hz = unpack2(w.gz);
        if (ONE) {
            double e[2] = {};
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int i = q ? i1 : i0;
                if (i >= n) continue;
                const double v[4] = {q ? (double)phi.y + (double)phic.y : (double)phi.x + (double)phic.x,
                                     q ? hx.y : hx.x, q ? hy.y : hy.x, q ? hz.y : hz.x};
                e[q] = pa_row_out<GRAD>(a, S, q ? q1.w : q0.w, a.rio[S.row0 + i], v);
            }
            const double sum = pa_tile_sum(e);
            if (tid == 0) a.E[slot] = sum;
            continue;
        }
        const size_t first = S.part0 + (size_t)ch * n;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int i = q ? i1 : i0;
            if (i >= n) continue;
            a.pphi[first + i] = q ? make_float2(phi.y, phic.y) : make_float2(phi.x, phic.x);
            if (GRAD) {
                a.pgx[first + i] = q ? hx.y : hx.x;
                a.pgy[first + i] = q ? hy.y : hy.x;
                a.pgz[first + i] = q ? hz.y : hz.x;
            }
        }
    }
}

// A block takes a row tile's rows (with PARTS = 4 a quarter of them, a warp to
// each quarter of the chunks): their sums over all chunks, their gradient by
// iOrder, and their energy -1/2 G sum_i m_i phi_i in FP64; the block that is
// the last to finish of a slot's adds the blocks' energies.  A chain of
// latencies bounds it; four parts shorten it where there are many chunks, and
// cost a second wave of blocks where there are few (PA_PARTS).
template <bool GRAD, int PARTS>
__global__ void __launch_bounds__(PA_TILE) pa_finish(PotAdjArgs a)
{
    constexpr int NA = 4, ROWS = PA_TILE / PARTS;
    __shared__ double sums[PARTS][GRAD ? NA : 1][ROWS];
    __shared__ int last;
    const int tid = threadIdx.x, row = tid % ROWS, part = tid / ROWS;
    for (long long b = blockIdx.x; b < a.ntile * PARTS; b += gridDim.x) {
        const int slot = pa_slot_warp(a, b / PARTS, &PotSlot::tile0);
        const PotSlot S = a.slots[slot];
        const int i = (int)(b - S.tile0 * PARTS) * ROWS + row;
        const bool in = i < S.n;
        float m = 0.0f;
        int io = 0;
        if (in && part == 0) {
            m = a.rm[S.row0 + i].w;
            io = a.rio[S.row0 + i];
        }
        double v[NA] = {};
        if (in) {
            const int c1 = (int)((long long)S.nchunk * (part + 1) / PARTS);
#pragma unroll 8
            for (int c = (int)((long long)S.nchunk * part / PARTS); c < c1; ++c) {
                const size_t o = S.part0 + (size_t)c * S.n + i;
                const float2 p = a.pphi[o];
                v[0] += (double)p.x + (double)p.y;
                if (GRAD) {
                    v[1] += (double)a.pgx[o];
                    v[2] += (double)a.pgy[o];
                    v[3] += (double)a.pgz[o];
                }
            }
        }
        if (PARTS > 1) {
            __syncthreads();
            for (int d = 0; d < (GRAD ? NA : 1); ++d) sums[part][d][row] = v[d];
            __syncthreads();
            if (part == 0)
                for (int k = 1; k < PARTS; ++k)
                    for (int d = 0; d < (GRAD ? NA : 1); ++d) v[d] += sums[k][d][row];
        }
        double mine[1] = {in && part == 0 ? pa_row_out<GRAD>(a, S, m, io, v) : 0.0};
        double e = pa_tile_sum(mine);
        const int nb = (S.n + PA_TILE - 1) / PA_TILE * PARTS;
        if (nb > 1) {
            if (tid == 0) {
                a.eblock[b] = e;
                __threadfence();
                last = atomicAdd(a.done + slot, 1) == nb - 1;
            }
            __syncthreads();
            if (!last) continue;
            __threadfence();
            mine[0] = 0.0;
            for (int k = tid; k < nb; k += PA_TILE) mine[0] += __ldcg(&a.eblock[S.tile0 * PARTS + k]);
            e = pa_tile_sum(mine);
        }
        if (tid == 0) a.E[slot] = e;
    }
}

}  // namespace

cudaError_t density_adjoint(const Tree &t, const float *ball2_sorted, const int *sidx, const float *w_io,
                            int n_io, float3 L, bool per, int mode, int k, AdjointState &A,
                            int *d_work, unsigned *d_status, cudaStream_t st)
{
    cudaError_t e;
    int ns = t.n;
    size_t m = ns > 0 ? ns : 1;
    if ((e = dalloc(A.w, m)) || (e = dalloc(A.g, 3 * m)) || (e = dalloc(A.out, 3 * (size_t)(n_io > 0 ? n_io : 1))))
        return e;
    if ((e = cudaMemsetAsync(A.g.p, 0, 3 * m * sizeof(float), st))) return e;
    if ((e = cudaMemsetAsync(A.out.p, 0, 3 * (size_t)(n_io > 0 ? n_io : 1) * sizeof(float), st))) return e;
    if (ns <= 0) return cudaSuccess;
    gather_w<<<grid_for(ns), 256, 0, st>>>(sidx, w_io, ns, A.w.p); note_launch();
    float3 hL = make_float3(0.5f * L.x, 0.5f * L.y, 0.5f * L.z);
    int need = (t.nLeaf + A_WARPS - 1) / A_WARPS;
    int subShift = 0;
    while (subShift < 5 && (2 << subShift) <= t.leafBase) ++subShift;
    if (mode == 2) {
        // store the lists only while they take at most a quarter of the free memory
        size_t fr = 0, tot = 0;
        size_t bytes = m * (size_t)(k + 16 + 1) * sizeof(int);
        mode = (A.lists || (cudaMemGetInfo(&fr, &tot) == cudaSuccess && bytes <= fr / 4)) ? 1 : 0;
    }
    if (mode == 0) {
        if ((e = cudaMemsetAsync(d_work, 0, sizeof(int), st))) return e;
        int perSM = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, density_adjoint_walk, A_WARPS * 32, 0);
        int blocks = num_sms() * (perSM > 0 ? perSM : 1);
        if (blocks > need) blocks = need;
        density_adjoint_walk<<<blocks, A_WARPS * 32, 0, st>>>(t.view(), ball2_sorted, A.w.p, L, hL, per,
                                                             subShift, A.g.p, d_work, d_status); note_launch();
    } else {
        if (!A.lists) {
            A.cap = k + 16;
            if ((e = dalloc(A.nbr, m * (size_t)A.cap)) || (e = dalloc(A.ncnt, m))) return e;
            if ((e = cudaMemsetAsync(d_work, 0, sizeof(int), st))) return e;
            int perSM = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, ball_lists, A_WARPS * 32, 0);
            int blocks = num_sms() * (perSM > 0 ? perSM : 1);
            if (blocks > need) blocks = need;
            ball_lists<<<blocks, A_WARPS * 32, 0, st>>>(t.view(), ball2_sorted, L, hL, per, subShift, 0.0f, A.cap,
                                                       A.nbr.p, A.ncnt.p, d_work, d_status); note_launch();
            A.lists = true;
        }
        density_adjoint_lists<<<grid_for(ns, 128), 128, 0, st>>>(t.pos.p, ball2_sorted, A.w.p, ns, L, hL,
                                                                per, A.cap, A.nbr.p, A.ncnt.p, A.g.p,
                                                                d_status); note_launch();
    }
    scatter_grad<<<grid_for(ns), 256, 0, st>>>(sidx, A.g.p, ns, A.out.p); note_launch();
    return cudaGetLastError();
}

cudaError_t potential_adjoint(const GroupState &G, const float4 *pos4, const float4 *vel4, int n,
                              float3 period, float Gc, int plummer, int nSel, const int *h_sel,
                              const float *h_v, bool want_grad, AdjointState &A, SortScratch &ss,
                              cudaStream_t st)
{
    cudaError_t e;
    std::vector<int> counts(G.nGroup);
    if ((e = cudaMemcpyAsync(counts.data(), G.count.p, G.nGroup * sizeof(int), cudaMemcpyDeviceToHost, st)))
        return e;
    if ((e = cudaStreamSynchronize(st))) return e;
    // items and rows per selected group: columns split into chunks of a
    // length chosen by the pairs there are
    double pairs = 0.0;
    for (int s = 0; s < nSel; ++s) pairs += (double)counts[h_sel[s]] * (double)counts[h_sel[s]];
    int chunk = PA_CHUNK;
    while (chunk > PA_CHUNK_MIN && pairs < (double)(PA_FILL * num_sms()) * PA_TILE * chunk) chunk >>= 1;
    std::vector<PotSlot> slots(nSel);
    long long nitems = 0, nrows = 0, ntile = 0, npart = 0;
    bool one = true;            // every group one tile of one chunk
    for (int s = 0; s < nSel; ++s) {
        const int c = counts[h_sel[s]];
        PotSlot &S = slots[s];
        S.item0 = nitems;
        S.row0 = nrows;
        S.tile0 = ntile;
        S.part0 = npart;
        S.g = h_sel[s];
        S.n = c;
        S.chunk = std::max(chunk, ((c + PA_MAX_CHUNKS - 1) / PA_MAX_CHUNKS + PA_TILE - 1) / PA_TILE * PA_TILE);
        S.nchunk = (c + S.chunk - 1) / S.chunk;
        S.v = h_v ? h_v[s] : 0.0f;
        nitems += (long long)((c + PA_TILE - 1) / PA_TILE) * S.nchunk;
        nrows += c;
        ntile += (c + PA_TILE - 1) / PA_TILE;
        npart += (long long)c * S.nchunk;
        one = one && c <= std::min(PA_TILE, S.chunk);
    }
    // energies, then the counts of finished blocks, cleared together
    const size_t nE = nSel > 0 ? nSel : 1, nclear = nE + (nE + 1) / 2;
    // one buffer for all of a call's scratch, the same with and without the
    // gradient: allocations cost as much as a small call, and the torch wrapper
    // makes a context per pass and asks for the energies first
    size_t bytes = 0;
    auto take = [&](size_t b) {
        const size_t at = bytes;
        bytes += (b + 255) / 256 * 256;
        return at;
    };
    const size_t oE = take(nclear * sizeof(double)), oslots = take(nSel * sizeof(PotSlot)),
                 orm = take(nrows * sizeof(float4)), ore = take(nrows * sizeof(float)),
                 orio = take(nrows * sizeof(int)), obox = take(2 * ntile * sizeof(float4)),
                 oeb = take(PA_PARTS * ntile * sizeof(double)),
                 opart = take(one ? 0 : 5 * npart * sizeof(float));
    if ((e = dalloc(A.ws, bytes)) || (e = dalloc(A.out, 3 * (size_t)(n > 0 ? n : 1)))) return e;
    unsigned char *ws = A.ws.p;
    PotSlot *d_slots = reinterpret_cast<PotSlot *>(ws + oslots);
    float *part = reinterpret_cast<float *>(ws + opart);
    A.E = reinterpret_cast<double *>(ws + oE);
    if (nSel) {
        if ((e = cudaMemcpyAsync(d_slots, slots.data(), nSel * sizeof(PotSlot), cudaMemcpyHostToDevice, st)))
            return e;
        if ((e = cudaMemsetAsync(A.E, 0, nclear * sizeof(double), st))) return e;
    }
    if (want_grad && (e = cudaMemsetAsync(A.out.p, 0, 3 * (size_t)(n > 0 ? n : 1) * sizeof(float), st))) return e;
    if (!nitems) return cudaSuccess;
    PotAdjArgs a;
    a.slots = d_slots;
    a.nslot = nSel;
    a.nitems = nitems;
    a.nrows = nrows;
    a.gstart = G.start.p;
    a.members = G.members.p;
    a.pos4 = pos4;
    a.vel4 = vel4;
    a.rec = G.rec.p;
    a.hP = make_float3((float)(0.5 * (double)period.x), (float)(0.5 * (double)period.y),
                       (float)(0.5 * (double)period.z));
    a.G = Gc;
    a.plummer = plummer;
    a.perm = nullptr;
    a.rm = reinterpret_cast<float4 *>(ws + orm);
    a.re = reinterpret_cast<float *>(ws + ore);
    a.rio = reinterpret_cast<int *>(ws + orio);
    a.tlo = reinterpret_cast<float4 *>(ws + obox);
    a.thi = a.tlo + ntile;
    a.ntile = ntile;
    a.pphi = reinterpret_cast<float2 *>(part);
    a.pgx = part + 2 * npart;
    a.pgy = a.pgx + npart;
    a.pgz = a.pgy + npart;
    a.eblock = reinterpret_cast<double *>(ws + oeb);
    a.E = A.E;
    a.done = reinterpret_cast<int *>(A.E + nE);
    a.grad = want_grad ? A.out.p : nullptr;
    const long long most = (long long)num_sms() * 32;
    const int rgrid = grid_for((int)(nrows < (1 << 30) ? nrows : 1 << 30));
    const double perSM = pairs / num_sms();
    if ((perSM >= PA_SORT_ANY || (perSM >= PA_SORT_PAIRS && pairs >= PA_SORT_COLS * nrows)) &&
        nrows < (1ll << 31)) {
        int sbits = 0;
        while ((1ll << sbits) < nSel) ++sbits;
        if ((e = dalloc(ss.k0, (size_t)nrows)) || (e = dalloc(ss.k1, (size_t)nrows)) ||
            (e = dalloc(ss.v0, (size_t)nrows)) || (e = dalloc(ss.v1, (size_t)nrows)) ||
            (e = dalloc(ss.box, 8)) || (e = cudaMemsetAsync(ss.box.p, 0, sizeof(unsigned), st)))
            return e;
        pa_extent<<<rgrid, 256, 0, st>>>(a, ss.box.p); note_launch();
        pa_keys<<<rgrid, 256, 0, st>>>(a, ss.box.p, ss.k0.p, ss.v0.p); note_launch();
        if ((e = radix_sort(ss, (int)nrows, PA_KEY_BITS + sbits, st))) return e;
        a.perm = ss.v0.p;
    }
    pa_pack<<<grid_for((int)(ntile < (1 << 25) ? ntile * 32 : 1 << 30), 128), 128, 0, st>>>(a); note_launch();
    const int blocks = (int)(nitems < most ? nitems : most);
    if (one) {
        if (want_grad) potential_adjoint_kernel<true, true><<<blocks, PA_THREADS, 0, st>>>(a);
        else potential_adjoint_kernel<false, true><<<blocks, PA_THREADS, 0, st>>>(a);
        note_launch();
        return cudaGetLastError();
    }
    const bool parts = npart >= PA_PARTS_MIN * nrows;
    const int fblocks = (int)std::min(most, ntile * (parts ? PA_PARTS : 1));
    if (want_grad) {
        potential_adjoint_kernel<true, false><<<blocks, PA_THREADS, 0, st>>>(a); note_launch();
        if (parts) pa_finish<true, PA_PARTS><<<fblocks, PA_TILE, 0, st>>>(a);
        else pa_finish<true, 1><<<fblocks, PA_TILE, 0, st>>>(a);
    } else {
        potential_adjoint_kernel<false, false><<<blocks, PA_THREADS, 0, st>>>(a); note_launch();
        if (parts) pa_finish<false, PA_PARTS><<<fblocks, PA_TILE, 0, st>>>(a);
        else pa_finish<false, 1><<<fblocks, PA_TILE, 0, st>>>(a);
    }
    note_launch();
    return cudaGetLastError();
}

}  // namespace skid
