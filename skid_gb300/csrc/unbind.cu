// Gravitational unbinding of every group in one pass (kdUnbind,
// kd.c:1299-1466; kdCellPot/kdSubPot/kdAddScoopPot, grav.c:8-135; the
// Hernquist-Katz spline SPLINE_POT, grav.h:11-31).
//
// Per group g (members in ascending iOrder, positions relative to rel and
// wrapped with half periods, kd.c:1341-1355):
//   pot_i = sum_{j != i} G m_j psi(r_ij, eps_i + eps_j)            (kdCellPot)
//         + sum_{ungrouped k within fScoop of the centre} G m_k psi  (scoop; the
//           reference applies it for every input type, kd.c:1379-1384)
//   then repeatedly: E_i = 1/2 |a (v_i - vcm) + aH (r_i - rcm)|^2 - pot_i (1+z);
//   if max E < 0 stop, else remove the first member with the largest E,
//   update rcm/vcm (FP64), swap it with the last member, and for pure dark
//   or pure star input subtract its potential from the others (kdSubPot).
//
// Potentials are accumulated in 64-bit fixed point (term * 2^S rounded to an
// integer).  The reference adds float terms into a double, which is exact
// for realistic groups, so when kdSubPot later subtracts the same terms the
// remainder is exact -- in particular a group's last member ends with
// potential exactly 0 (or its scoop part) and is unbound with E = 1/2 dv^2 >= 0.
// Integer sums reproduce that exactly and in any order.
//
// Kernels, each taking every group in one launch (the removal in two):
//  - scoop lists: one warp per group walks the tree of ungrouped particles;
//  - potentials: work items are the upper-triangle tile pairs (I <= J) of
//    every group, largest groups first; each pair's psi is evaluated once and
//    added to both ends (the terms are exact integers, so the sums do not
//    depend on the order);
//  - removal: two persistent kernels take groups largest first, each from a
//    queue: one those above `tw` members, the whole block on a group (BS
//    threads, block-wide arg-max with first-index ties), the other the smaller
//    ones, a warp each (warp shuffles only, no block barriers), beside it.
// (tw, BS) is picked by timing the candidates on the first call (autotune),
// or fixed through the context's options.  A per-group mode (one potential
// and one removal launch per group, the reference's serial loop on the GPU)
// serves as the unbatched comparison.
#include <algorithm>
#include <cfloat>
#include <vector>

#include <cooperative_groups.h>

#include "ctx.h"

namespace cg = cooperative_groups;

namespace skid {

namespace {

constexpr int POT_TILE = 128;   // power of two
// Every removal decision is the reference's: each pass computes FP32 energies
// with an error bound, and only members within twice the bound of the
// largest or smallest energy are evaluated exactly (the reference's FP64
// expression rounded to float, kd.c:1396-1399), so the arg-max and arg-min,
// ties included, are those of the reference's loop.  Warps use the plain FP32
// form with a per-member bound up to this size; blocks and larger groups the
// staged a v + aH r form with one bound per pass (GB300's FP64 rate is a small
// fraction of its FP32 rate, so FP64 is kept to the few candidates).
constexpr int EXACT_E_MAX = 1024;

// The reference's pair factor, bit for bit.  grav.c:25-30 forms it as a float
// assigned from FP64 arithmetic (gcc, no contraction): Plummer
// 1.0/sqrt(d2 + 0.25*twoh*twoh); spline SPLINE_POT (grav.h:11-31) with
// r = sqrt(d2) in FP64, the polynomials evaluated left to right, and 1/r
// beyond the softening.  The FP64 forms below spell every operation out with
// round-to-nearest intrinsics so the compiler cannot fuse them.
__device__ __noinline__ float ref_dir_fp64(float d2f, float twohf, int plummer)
{
    const double r2 = (double)d2f, twoh = (double)twohf;
    if (plummer)
        return (float)__ddiv_rn(1.0, __dsqrt_rn(__dadd_rn(r2, __dmul_rn(__dmul_rn(0.25, twoh), twoh))));
    const double r = __dsqrt_rn(r2);
    if (r < twoh) {
        const double dih = __ddiv_rn(2.0, twoh);
        const double u = __dmul_rn(r, dih);
        if (u < 1.0) {
            // dih*(7/5 - 2/3*u*u + 3/10*u*u*u*u - 1/10*u*u*u*u*u)
            const double a = __dmul_rn(__dmul_rn(2.0 / 3.0, u), u);
            const double b = __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(3.0 / 10.0, u), u), u), u);
            const double c =
                __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(1.0 / 10.0, u), u), u), u), u);
            return (float)__dmul_rn(dih, __dsub_rn(__dadd_rn(__dsub_rn(7.0 / 5.0, a), b), c));
        }
        // -1/15*dir + dih*(8/5 - 4/3*u*u + u*u*u - 3/10*u*u*u*u + 1/30*u*u*u*u*u)
        const double dir = __ddiv_rn(1.0, r);
        const double a = __dmul_rn(__dmul_rn(4.0 / 3.0, u), u);
        const double b = __dmul_rn(__dmul_rn(u, u), u);
        const double c = __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(3.0 / 10.0, u), u), u), u);
        const double e =
            __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(1.0 / 30.0, u), u), u), u), u);
        const double poly = __dadd_rn(__dsub_rn(__dadd_rn(__dsub_rn(8.0 / 5.0, a), b), c), e);
        return (float)__dadd_rn(__dmul_rn(-1.0 / 15.0, dir), __dmul_rn(dih, poly));
    }
    return (float)__ddiv_rn(1.0, r);
}

// 1/r beyond the softening as the reference rounds it: float(1.0/sqrt(d2)),
// two correctly rounded FP64 operations then a rounding to float.  That float
// is the one nearest the real 1/sqrt(d2) unless 1/sqrt(d2) lies within about
// 2^-52 (relative) of a midpoint between floats.  Here 1/sqrt(d2) is formed
// as the unevaluated float pair y + d, within 2^-43 of it: y the hardware
// reciprocal square root (within 2^-22) and d = y r / 2 one Newton
// correction, whose residual r = 1 - x y^2 comes from the error-free product
// x y = ph + pl (pl by a fused multiply-add) as fma(-pl, y, fma(-ph, y, 1)),
// each fused step rounding only the small result.  The float s nearest
// y + d is returned unless y + d lies within 2^-17 ulp(s) of a midpoint
// (|(y + d) - s|, exact by Dekker's fast two-sum, at or above
// (1/2 - 2^-17) ulp), or s is a power of two; those few pairs in a hundred
// thousand take the FP64 expression itself.
__device__ __forceinline__ float ref_rsqrt(float x)
{
    if (!(x >= 1e-30f && x <= 1e30f)) return ref_dir_fp64(x, 0.0f, 0);
    const float y = rsqrtf(x);
    const float ph = __fmul_rn(x, y);
    const float pl = __fmaf_rn(x, y, -ph);
    const float r = __fmaf_rn(-pl, y, __fmaf_rn(-ph, y, 1.0f));
    const float d = __fmul_rn(__fmul_rn(0.5f, y), r);
    const float s = __fadd_rn(y, d);
    const float e = __fsub_rn(d, __fsub_rn(s, y));
    const unsigned sb = __float_as_uint(s);
    // (1/2 - 2^-17) ulp(s): exponent of ulp/4, mantissa 2 - 2^-15
    const float near = __uint_as_float(((sb & 0x7f800000u) - (25u << 23)) | 0x7fff00u);
    if ((sb & 0x7fffffu) == 0u || fabsf(e) >= near) return ref_dir_fp64(x, 0.0f, 0);
    return s;
}

// Float-float numbers (an unevaluated sum h + l, |l| <= ulp(h) / 2) with
// round-to-nearest intrinsics throughout, so no step is contracted.  Every
// operation is within about 2^-46 (relative) of the real result.
struct ffl {
    float h, l;
};

__device__ __forceinline__ ffl ff_norm(float s, float e)
{
    const float h = __fadd_rn(s, e);
    return {h, __fsub_rn(e, __fsub_rn(h, s))};
}

__device__ __forceinline__ ffl ff_add(ffl a, ffl b)
{
    const float s = __fadd_rn(a.h, b.h);
    const float v = __fsub_rn(s, a.h);
    float e = __fadd_rn(__fsub_rn(a.h, __fsub_rn(s, v)), __fsub_rn(b.h, v));
    e = __fadd_rn(e, __fadd_rn(a.l, b.l));
    return ff_norm(s, e);
}

__device__ __forceinline__ ffl ff_mul(ffl a, ffl b)
{
    const float p = __fmul_rn(a.h, b.h);
    float e = __fmaf_rn(a.h, b.h, -p);
    e = __fmaf_rn(a.h, b.l, e);
    e = __fmaf_rn(a.l, b.h, e);
    return ff_norm(p, e);
}

// A double constant as the nearest float pair (within 2^-48 of it).
#define SKID_FFC(x) ffl{(float)(x), (float)((x) - (double)(float)(x))}

// The spline branch of the reference's pair factor (grav.h:11-31 as
// grav.c:25-30 evaluates it, r < 2h) without FP64: the same real-number
// expression in float-float arithmetic, within about 2^-37 (relative) of
// its real value -- the one polynomial with cancellation has terms up to 16
// times its value -- while the reference's FP64 evaluation is within about
// 2^-45.  Both therefore round to the same float unless the value lies
// within 2^-32 (relative) of a midpoint between floats, or r is that close
// to 2h or u = 2r/(2h) to 1 (where the reference's own rounding could take
// the other branch).  Those inputs, tiny ones and powers of two return
// false, and the caller takes the FP64 expression.
__device__ __forceinline__ bool ref_spline_ff(float d2, float twoh, float &out)
{
    if (!(d2 >= 1e-30f && twoh >= 1e-30f && twoh <= 1e30f)) return false;
    // r = sqrt(d2): the correctly rounded root plus one Newton correction
    // (d2 - s^2 is exact by a fused multiply-add)
    const float s = __fsqrt_rn(d2);
    const ffl r = ff_norm(s, __fdiv_rn(__fmaf_rn(-s, s, d2), __fmul_rn(2.0f, s)));
    // the branch r < 2h, decided only when r is clear of 2h
    const float dr = ff_add(r, ffl{-twoh, 0.0f}).h;
    if (fabsf(dr) <= 0x1p-40f * twoh) return false;
    if (dr >= 0.0f) return false;   // 1/r beyond the softening: not this branch
    // dih = 2/(2h), the quotient plus its remainder (exact by a fused multiply-add)
    const float q = __fdiv_rn(2.0f, twoh);
    const ffl dih = ff_norm(q, __fdiv_rn(__fmaf_rn(-q, twoh, 2.0f), twoh));
    const ffl u = ff_mul(r, dih);
    const float du = __fadd_rn(__fsub_rn(u.h, 1.0f), u.l);
    if (fabsf(du) <= 0x1p-38f) return false;
    const ffl u2 = ff_mul(u, u);
    const ffl u4 = ff_mul(u2, u2);
    const ffl u5 = ff_mul(u4, u);
    ffl v;
    if (du < 0.0f) {
        // dih*(7/5 - 2/3 u^2 + 3/10 u^4 - 1/10 u^5)
        ffl p = ff_add(SKID_FFC(7.0 / 5.0), ff_mul(SKID_FFC(-2.0 / 3.0), u2));
        p = ff_add(p, ff_mul(SKID_FFC(3.0 / 10.0), u4));
        p = ff_add(p, ff_mul(SKID_FFC(-1.0 / 10.0), u5));
        v = ff_mul(dih, p);
    } else {
        // -1/15 / r + dih*(8/5 - 4/3 u^2 + u^3 - 3/10 u^4 + 1/30 u^5)
        const ffl u3 = ff_mul(u2, u);
        ffl p = ff_add(SKID_FFC(8.0 / 5.0), ff_mul(SKID_FFC(-4.0 / 3.0), u2));
        p = ff_add(p, u3);
        p = ff_add(p, ff_mul(SKID_FFC(-3.0 / 10.0), u4));
        p = ff_add(p, ff_mul(SKID_FFC(1.0 / 30.0), u5));
        // 1/r: the rounded reciprocal and its residual 1 - r y
        const float y = __frcp_rn(r.h);
        const float t = __fmaf_rn(-r.l, y, __fmaf_rn(-r.h, y, 1.0f));
        const ffl dir = ff_norm(y, __fmul_rn(y, t));
        v = ff_add(ff_mul(dih, p), ff_mul(SKID_FFC(-1.0 / 15.0), dir));
    }
    // the float nearest v, kept unless v is within 2^-9 ulp of a midpoint
    const float f = __fadd_rn(v.h, v.l);
    const float e = __fadd_rn(__fsub_rn(v.h, f), v.l);
    const unsigned fb = __float_as_uint(f);
    if (!(f >= 1e-30f && f <= 1e30f) || (fb & 0x7fffffu) == 0u) return false;
    // (1/2 - 2^-9) ulp(f): exponent of ulp/4, mantissa 2 - 2^-7
    const float near = __uint_as_float(((fb & 0x7f800000u) - (25u << 23)) | 0x7f0000u);
    if (fabsf(e) >= near) return false;
    out = f;
    return true;
}
#undef SKID_FFC

// The pair factor of every potential term, added (potentials, scoop) and
// subtracted (removal) alike, equal to the reference's float dir.  Beyond
// the softening (r >= 2h, certain once d2 clears (2h)^2 by the margin below)
// it is ref_rsqrt; inside, the float-float spline where it decides the
// rounding, else (and for Plummer softening) the FP64 form.
__device__ __forceinline__ float pair_dir(float d2, float twoh, int plummer)
{
    if (!plummer && d2 >= twoh * twoh * 1.000001f) return ref_rsqrt(d2);
    float v;
    if (!plummer && ref_spline_ff(d2, twoh, v)) return v;
    return ref_dir_fp64(d2, twoh, plummer);
}

// The same, kept out of line where it is seldom reached.
__device__ __noinline__ float pair_dir_call(float d2, float twoh) { return pair_dir(d2, twoh, 0); }

__device__ __forceinline__ float wrap_h(float d, float h)
{
    // kd.c:1345-1350: if (dx > hx) dx -= 2*hx; if (dx <= -hx) dx += 2*hx
    if (d > h) d = fsub(d, fmul(2.0f, h));
    if (d <= -h) d = fadd(d, fmul(2.0f, h));
    return d;
}

// float -> int64 with round-half-to-even, bit-identical to __float2ll_rn for
// finite |f| < 2^63, on the integer units: the mantissa shifted by the
// exponent.  (GB300 runs the 64-bit conversion instructions on its FP64
// path, which made them the bottleneck of the potential sums.)
__device__ __forceinline__ long long f2ll_rn(float f)
{
    const unsigned b = __float_as_uint(f);
    const int e = (int)((b >> 23) & 0xffu);
    if (e == 0) return 0;                              // zero or denormal (< 0.5)
    const unsigned long long m = (b & 0x7fffffu) | 0x800000u;
    const int sh = e - 150;                            // |f| = m * 2^sh
    unsigned long long q;
    if (sh > 39) {
        q = 0x7fffffffffffffffull;                     // |f| >= 2^63: saturate
    } else if (sh >= 0) {
        q = m << sh;
    } else if (sh > -25) {
        const int r = -sh;                             // 1..24
        const unsigned long long rem = m & ((1ull << r) - 1ull);
        const unsigned long long half = 1ull << (r - 1);
        q = m >> r;
        q += (rem > half) || (rem == half && (q & 1ull));
    } else {
        q = 0;                                         // |f| < 0.5
    }
    return (b >> 31) ? -(long long)q : (long long)q;
}

// int64 -> float within two roundings (relative error <= 2^-23), on the
// FP32 and integer units: |p| in three 22-bit chunks, each exact as a float
// (2^23 + x - 2^23), recombined by two fused multiply-adds.
__device__ __forceinline__ float ll2f_approx(long long p)
{
    const unsigned long long a = p < 0 ? (unsigned long long)(-p) : (unsigned long long)p;
    const float c0 = __uint_as_float(0x4B000000u | (unsigned)(a & 0x3fffffull)) - 8388608.0f;
    const float c1 = __uint_as_float(0x4B000000u | (unsigned)((a >> 22) & 0x3fffffull)) - 8388608.0f;
    const float c2 = __uint_as_float(0x4B000000u | (unsigned)((a >> 44) & 0x3fffffull)) - 8388608.0f;
    const float f = __fmaf_rn(c2, 17592186044416.0f, __fmaf_rn(c1, 4194304.0f, c0));   // 2^44, 2^22
    return p < 0 ? -f : f;
}

// int64 -> float within three roundings (relative error below 2^-22), from
// the two 32-bit halves of |p| and one fused multiply-add: the FP32 energies
// of large groups only.
__device__ __forceinline__ float ll2f_fast(long long p)
{
    const unsigned long long a = p < 0 ? (unsigned long long)(-p) : (unsigned long long)p;
    const float f = __fmaf_rn(__uint2float_rn((unsigned)(a >> 32)), 4294967296.0f,
                              __uint2float_rn((unsigned)a));
    return p < 0 ? -f : f;
}

// Fixed-point quantum of a float term (scale = 2^S, exact multiply), equal to
// __float2ll_rn(t * scale).  Terms are non-negative: below 2^23 adding 2^23
// rounds to the nearest integer (ties to even) in the float adder, at or above
// it the float is already an integer, its mantissa shifted by the exponent.
__device__ __forceinline__ long long fx(float t, float scale)
{
    const float f = t * scale;
    if (f < 8388608.0f) {
        if (!(f >= 0.0f)) return f2ll_rn(f);          // negative or NaN: general form
        return (long long)(__float_as_uint(f + 8388608.0f) - 0x4B000000u);
    }
    const unsigned b = __float_as_uint(f);
    const int sh = (int)(b >> 23) - 150;              // 0 .. for f >= 2^23
    if (sh > 39) return f2ll_rn(f);                   // beyond 2^63: saturates
    return (long long)(((unsigned long long)((b & 0x7fffffu) | 0x800000u)) << sh);
}

__global__ void prep_members(const int *__restrict__ members, const int *__restrict__ gof, int n,
                             const float4 *__restrict__ pos4, const float4 *__restrict__ vel4,
                             const skid_group *__restrict__ rec, float3 hP,
                             float4 *__restrict__ qr, float4 *__restrict__ qv)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        int io = members[k];
        int g = gof[k];
        float4 p = pos4[io];
        const float *rel = rec[g].rel;
        qr[k] = make_float4(wrap_h(fsub(p.x, rel[0]), hP.x), wrap_h(fsub(p.y, rel[1]), hP.y),
                            wrap_h(fsub(p.z, rel[2]), hP.z), p.w);
        qv[k] = vel4[io];
    }
}

// Scoop: ungrouped particles within fScoop of each group's centre, a warp per
// group.  pass 0 counts, pass 1 fills (offsets from an exclusive scan), in the
// order of the sorted particles.
//
// The walk is one chain of dependent loads: with a thread per group the
// slowest lane's whole walk, its leaves' particles one by one.  A warp tests
// the last 2^subShift leaves of a subtree one per lane, then a leaf's
// particles one per lane, and counts with ballots: 300 groups over
// 400,000 particles 650 to 27 us, both passes.
constexpr int SCOOP_THREADS = 128;

__global__ void __launch_bounds__(SCOOP_THREADS)
scoop_kernel(TreeView t, const float *__restrict__ usoft, const skid_group *__restrict__ rec,
             const int *__restrict__ gcount, int ng, int nmax, float fBall2, float3 L, float3 hL,
             bool per, int subShift, int pass, int *__restrict__ cnt, const int *__restrict__ off,
             float4 *__restrict__ list, float *__restrict__ lsoft)
{
    const int lane = threadIdx.x & 31;
    const int rootLo = t.leafBase >> subShift;
    // every entry is written, group 0 (the ungrouped particles) with 0: the
    // counts are scanned into offsets as a whole
    const int nwarps = gridDim.x * (SCOOP_THREADS / 32);
    for (int g = (blockIdx.x * SCOOP_THREADS + threadIdx.x) >> 5; g < ng; g += nwarps) {
        int c = 0;
        const int n = gcount[g];
        if (g > 0 && n > 0 && n < nmax && t.n > 0) {
            const float *cen = rec[g].rCenter;
            const float *rel = rec[g].rel;
            const float3 q = make_float3(cen[0], cen[1], cen[2]);
            const int o = pass ? off[g] : 0;
            int cp = 1;
            for (;;) {
                if (cp < rootLo) {
                    if (box_lb(q, t.lo[cp], t.hi[cp], L, per) < fBall2) { cp <<= 1; continue; }
                } else {
                    const int leaf = (cp << subShift) + lane;
                    const bool near = lane < (1 << subShift) && leaf - t.leafBase < t.nLeaf &&
                                      box_lb(q, t.lo[leaf], t.hi[leaf], L, per) < fBall2;
                    for (unsigned lm = __ballot_sync(SKID_FULL, near); lm; lm &= lm - 1) {
                        const int j = ((cp << subShift) + __ffs(lm) - 1 - t.leafBase) * SKID_LEAF + lane;
                        float4 p;
                        bool in = false;
                        if (j < t.n) {
                            p = t.pos[j];
                            in = d2of(img_dx(q.x, p.x, L.x, hL.x), img_dx(q.y, p.y, L.y, hL.y),
                                      img_dx(q.z, p.z, L.z, hL.z)) < fBall2;
                        }
                        const unsigned m = __ballot_sync(SKID_FULL, in);
                        if (pass && in) {
                            // grav.c:103-111
                            float nx = fsub(p.x, rel[0]), ny = fsub(p.y, rel[1]), nz = fsub(p.z, rel[2]);
                            if (nx > hL.x) nx = fsub(nx, L.x);
                            if (nx <= -hL.x) nx = fadd(nx, L.x);
                            if (ny > hL.y) ny = fsub(ny, L.y);
                            if (ny <= -hL.y) ny = fadd(ny, L.y);
                            if (nz > hL.z) nz = fsub(nz, L.z);
                            if (nz <= -hL.z) nz = fadd(nz, L.z);
                            const int k = o + c + __popc(m & ((1u << lane) - 1u));
                            list[k] = make_float4(nx, ny, nz, p.w);
                            lsoft[k] = usoft[j];
                        }
                        c += __popc(m);
                    }
                }
                cp = next_node(cp);
                if (cp == 1) break;
            }
        }
        if (!pass && lane == 0) cnt[g] = c;
    }
}


// ---- scheduling order: valid groups by descending size ----

__global__ void sched_keys(const int *__restrict__ gcount, int ng, int nmax, uint64_t *keys,
                           uint32_t *vals)
{
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += gridDim.x * blockDim.x) {
        int n = gcount[g];
        bool ok = g > 0 && n > 0 && n < nmax;
        keys[g] = ok ? (uint64_t)(0x7fffffff - n) : 0xffffffffull;
        vals[g] = (uint32_t)g;
    }
}

// cnt[0] = valid groups, cnt[1] = groups above tw members
__global__ void sched_counts(const int *__restrict__ gcount, int ng, int nmax, int tw, int *cnt)
{
    int v = 0, b = 0;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += gridDim.x * blockDim.x) {
        int n = gcount[g];
        if (g > 0 && n > 0 && n < nmax) {
            ++v;
            b += n > tw;
        }
    }
    for (int o = 16; o; o >>= 1) {
        v += __shfl_xor_sync(SKID_FULL, v, o);
        b += __shfl_xor_sync(SKID_FULL, b, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(cnt, v);
        atomicAdd(cnt + 1, b);
    }
}

// ---- potentials ----

// out[0]: groups taken by clusters, the largest ones above `floor` members
// but at most kmax of them; out[2]: the largest valid group's size (order is
// largest first)
__global__ void cluster_groups(const uint32_t *__restrict__ order, const int *d_nvalid,
                               const int *__restrict__ gcount, int floor, int kmax, int *out)
{
    if (threadIdx.x != 0) return;
    const int nv = *d_nvalid;
    int k = 0;
    while (k < nv && k < kmax && gcount[order[k]] > floor) ++k;
    out[0] = k;
    out[2] = nv > 0 ? gcount[order[0]] : 0;
}

__global__ void pot_nitems(const uint32_t *__restrict__ order, const int *d_nvalid,
                           const int *__restrict__ gcount, int ng, int *__restrict__ ni)
{
    int nv = *d_nvalid;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < ng; k += gridDim.x * blockDim.x) {
        int c = 0;
        if (k < nv) {
            int nt = (gcount[order[k]] + POT_TILE - 1) / POT_TILE;
            c = nt * (nt + 1) / 2;
        }
        ni[k] = c;
    }
}

// A group's tile pairs, row by row, a warp per group (a thread writing a large
// group's in turn took 27 us at 300 groups, this 10).
__global__ void pot_fill(const uint32_t *__restrict__ order, const int *d_nvalid,
                         const int *__restrict__ gcount, const int *__restrict__ ioff,
                         int2 *__restrict__ items)
{
    const int nv = *d_nvalid, lane = threadIdx.x & 31;
    for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < nv; k += (gridDim.x * blockDim.x) >> 5) {
        const int g = order[k];
        const int nt = (gcount[g] + POT_TILE - 1) / POT_TILE;
        int o = ioff[k];
        for (int I = 0; I < nt; ++I) {
            for (int J = I + lane; J < nt; J += 32) items[o + J - I] = make_int2(g, (I << 16) | J);
            o += nt - I;
        }
    }
}

// One tile pair (I, J) of one group per block iteration, POT_TILE / 2
// threads with two rows each (t and t + POT_TILE / 2).  Off-diagonal items
// take every (i in I, j in J); diagonal items every i < j in the tile, plus
// the scoop terms of the tile's rows (kdAddScoopPot, grav.c:112-127).  At
// rotation step k thread t pairs its rows with column (t + k) mod T: the
// lanes of a warp touch distinct columns, so each warp keeps its own column
// accumulators (plain adds, a warp barrier per step), summed at the end.
// Columns carry G m 2^S, so a term is one multiply from its quantum.
//
// Instruction issue bounds it.  Off the diagonal a thread's two rows go
// through packed FP32 operations together, and one test sends the pairs whose
// rounding or range is not plain (inside the softening, next to a rounding
// boundary, tiny terms) to pot_pair: 300 groups of 400,000 particles 1.41 to
// 1.15 ms, the groups of a 2^21-particle run 7.7 to 5.7.  Two columns a step
// for more independent work took 1.9 and 6.1.
//
// Where such pairs are many, the packed operations come on top of pot_pair's:
// when POT_SLOW of a tile pair's first POT_PROBE steps have one, its other
// steps leave them out.  400,000 particles in one clump, most steps with a pair
// inside the softening, 893 to 790 ms (769 without any packed operations); with
// POT_SLOW 4 the 300 groups take 1.17 ms, 8 and 12 1.11.
constexpr int POT_THREADS = POT_TILE / 2;
constexpr int POT_PROBE = 16, POT_SLOW = 8;

struct PotRow {
    float4 r;     // position, G m 2^S
    float e;      // softening
    bool v;       // a member of the tile
};

// ref_rsqrt's decision: the float s nearest y + d, off by e, is certain.
__device__ __forceinline__ bool rsqrt_decided(float s, float e)
{
    const unsigned sb = __float_as_uint(s);
    return (sb & 0x7fffffu) != 0u && fabsf(e) < __uint_as_float((sb & 0x7f800000u) - (25u << 23) + 0x7fff00u);
}

__device__ __forceinline__ float rsqrt_ftz(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// fx of a term from 2^23 to 2^63: its mantissa shifted.
__device__ __forceinline__ bool fx_large(float f)
{
    return __float_as_uint(f) - (150u << 23) < (40u << 23);
}

__device__ __forceinline__ long long fx_shift(float f)
{
    const unsigned b = __float_as_uint(f);
    return (long long)((unsigned long long)((b & 0x7fffffu) | 0x800000u) << ((b >> 23) - 150u));
}

// The terms of row a and column j (tr: on a, tc: on j).  far is at or above
// every pair's (2h)^2 (1 + 1e-6) in the tile pair (infinite for Plummer
// softening): beyond it pair_dir is 1/r, taken without forming the pair's
// softening, with the same value.
__device__ __forceinline__ void pot_pair(const PotRow &a, float4 rj, float ej, int plummer,
                                         float far, long long &tr, long long &tc)
{
    float d2 = d2of(fsub(a.r.x, rj.x), fsub(a.r.y, rj.y), fsub(a.r.z, rj.z));
    float dir = d2 >= far ? ref_rsqrt(d2) : pair_dir(d2, fadd(a.e, ej), plummer);
    tr = fx(fmul(rj.w, dir), 1.0f);
    // equal masses (all-dark runs): both ends get the same term
    tc = rj.w == a.r.w ? tr : fx(fmul(a.r.w, dir), 1.0f);
}

__global__ void __launch_bounds__(POT_THREADS)
pot_sym_kernel(const int2 *__restrict__ items, const int *d_nitems, int nitems_host,
               const int *__restrict__ gstart, const int *__restrict__ gcount,
               const float4 *__restrict__ qr, const float4 *__restrict__ qv,
               const int *__restrict__ soff, const int *__restrict__ scnt,
               const float4 *__restrict__ slist, const float *__restrict__ ssoft, float G,
               int plummer, float scale, float zero_arg, long long *__restrict__ pot)
{
    constexpr int T = POT_TILE, H = POT_TILE / 2, NW = POT_THREADS / 32;
    __shared__ float4 sr[T];
    __shared__ float ss[T];
    __shared__ long long acc_w[NW][T];
    __shared__ float emax_w[2][NW];
    const int t = threadIdx.x, wid = t >> 5;
    const int nitems = nitems_host >= 0 ? nitems_host : *d_nitems;
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
        int2 w = items[it];
        int g = w.x, I = w.y >> 16, J = w.y & 0xffff;
        int s = gstart[g], n = gcount[g];
        PotRow ra, rb;
        {
            const int ia = I * T + t, ib = ia + H;
            ra.v = ia < n;
            rb.v = ib < n;
            float4 q = ra.v ? qr[s + ia] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            ra.r = make_float4(q.x, q.y, q.z, fmul(G, q.w) * scale);
            ra.e = ra.v ? qv[s + ia].w : 0.0f;
            q = rb.v ? qr[s + ib] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            rb.r = make_float4(q.x, q.y, q.z, fmul(G, q.w) * scale);
            rb.e = rb.v ? qv[s + ib].w : 0.0f;
        }
        int j0 = J * T;
        int nj = min(T, n - j0);
        __syncthreads();
        for (int c = t; c < T; c += POT_THREADS) {
            if (c < nj) {
                float4 q = qr[s + j0 + c];
                sr[c] = make_float4(q.x, q.y, q.z, fmul(G, q.w) * scale);
                ss[c] = qv[s + j0 + c].w;
            }
#pragma unroll
            for (int k = 0; k < NW; ++k) acc_w[k][c] = 0;
        }
        __syncthreads();
        // the far bound: (largest row softening + largest column softening)^2,
        // above every pair's own (softenings are non-negative, so their bit
        // patterns order like their values)
        float far = INFINITY;
        if (!plummer) {
            float er = fmaxf(ra.v ? ra.e : 0.0f, rb.v ? rb.e : 0.0f), ec = 0.0f;
            for (int c = t; c < nj; c += POT_THREADS) ec = fmaxf(ec, ss[c]);
            er = __uint_as_float(__reduce_max_sync(SKID_FULL, __float_as_uint(er)));
            ec = __uint_as_float(__reduce_max_sync(SKID_FULL, __float_as_uint(ec)));
            if ((t & 31) == 0) {
                emax_w[0][wid] = er;
                emax_w[1][wid] = ec;
            }
            __syncthreads();
            er = emax_w[0][0];
            ec = emax_w[1][0];
#pragma unroll
            for (int k = 1; k < NW; ++k) {
                er = fmaxf(er, emax_w[0][k]);
                ec = fmaxf(ec, emax_w[1][k]);
            }
            const float twoh = er + ec;
            far = twoh * twoh * 1.000001f;
        }
        long long acca = 0, accb = 0;
        if (I != J) {
            // every row is a member: only a group's last tile is ragged
            const f32x2 rx = pack2(ra.r.x, rb.r.x), ry = pack2(ra.r.y, rb.r.y), rz = pack2(ra.r.z, rb.r.z);
            const f32x2 rw = pack2(ra.r.w, rb.r.w);
            const f32x2 zero = pack2(zero_arg, zero_arg), one = pack2(1.0f, 1.0f), half = pack2(0.5f, 0.5f),
                        neg1 = pack2(-1.0f, -1.0f);
            const float least = fmaxf(far, 1e-30f);
            // pot_pair of both rows at once, where every decision is plain:
            // ref_rsqrt's steps, and the terms' mantissas shifted
            auto both = [&](float4 rj, long long &col) {
                const f32x2 dx = sub2(rx, pack2(rj.x, rj.x)), dy = sub2(ry, pack2(rj.y, rj.y)),
                            dz = sub2(rz, pack2(rj.z, rj.z));
                const f32x2 x = add2(add2(sq2(dx, zero), sq2(dy, zero)), sq2(dz, zero));
                const float2 d2 = unpack2(x);
                const f32x2 y = pack2(rsqrt_ftz(d2.x), rsqrt_ftz(d2.y)), ny = mul2(y, neg1);
                const f32x2 nph = mul2(x, ny), pl = fma2(x, y, nph);
                const f32x2 r = fma2(pl, ny, fma2(nph, y, one));
                const f32x2 d = mul2(mul2(half, y), r), s2 = add2(y, d);
                const float2 e = unpack2(fma2(add2(s2, ny), neg1, d)), dir = unpack2(s2);
                const float2 f = unpack2(mul2(pack2(rj.w, rj.w), s2));
                if (!(fminf(d2.x, d2.y) >= least && fmaxf(d2.x, d2.y) <= 1e30f &&
                      rsqrt_decided(dir.x, e.x) && rsqrt_decided(dir.y, e.y) && fx_large(f.x) &&
                      fx_large(f.y)))
                    return false;
                const long long ta = fx_shift(f.x), tb = fx_shift(f.y);
                acca += ta;
                accb += tb;
                if (rj.w == ra.r.w && rj.w == rb.r.w) {
                    col = ta + tb;
                } else {
                    const float2 c = unpack2(mul2(rw, s2));
                    col = fx(c.x, 1.0f) + fx(c.y, 1.0f);
                }
                return true;
            };
            bool packed = true;
            unsigned slow = 0;           // steps with a pair that was not
            int k = 0;
#pragma unroll 1
            for (int end = POT_PROBE;; end = T) {
#pragma unroll 1
                for (; k < end; ++k) {
                    const int jl = (t + k) & (T - 1);
                    if (jl < nj) {
                        const float4 rj = sr[jl];
                        long long col;
                        if (!(packed && both(rj, col))) {
                            long long tr, tc;
                            slow |= 1u << (k & 31);
                            pot_pair(ra, rj, ss[jl], plummer, far, tr, tc);
                            acca += tr;
                            col = tc;
                            pot_pair(rb, rj, ss[jl], plummer, far, tr, tc);
                            accb += tr;
                            col += tc;
                        }
                        acc_w[wid][jl] += col;
                    }
                    __syncwarp();
                }
                if (end == T) break;
                packed = __popc(__reduce_or_sync(SKID_FULL, slow)) < POT_SLOW;
            }
        } else {
            // offset (column - row) mod T in 1..T/2 for row t (k = 1..H),
            // 1..T/2-1 for row t + H (k = H+1..T-1): each pair once
            for (int k = 1; k < T; ++k) {
                const int jl = (t + k) & (T - 1);
                const PotRow &a = k <= H ? ra : rb;
                if (jl < nj && a.v) {
                    long long tr, tc;
                    pot_pair(a, sr[jl], ss[jl], plummer, far, tr, tc);
                    if (k <= H) acca += tr; else accb += tr;
                    acc_w[wid][jl] += tc;
                }
                __syncwarp();
            }
            int so = soff[g], sc = scnt[g];
            for (int jb = 0; jb < sc; jb += T) {
                __syncthreads();
                for (int c = t; c < T; c += POT_THREADS)
                    if (jb + c < sc) {
                        float4 q = slist[so + jb + c];
                        sr[c] = make_float4(q.x, q.y, q.z, fmul(G, q.w) * scale);
                        ss[c] = ssoft[so + jb + c];
                    }
                __syncthreads();
                int cnt = min(T, sc - jb);
                for (int k = 0; k < cnt; ++k) {
                    const float4 rj = sr[k];
                    const float ej = ss[k];
                    // kdAddScoopPot's pair: d2 from the scoop particle
                    float d2a = d2of(fsub(rj.x, ra.r.x), fsub(rj.y, ra.r.y), fsub(rj.z, ra.r.z));
                    float d2b = d2of(fsub(rj.x, rb.r.x), fsub(rj.y, rb.r.y), fsub(rj.z, rb.r.z));
                    if (ra.v) acca += fx(fmul(rj.w, pair_dir(d2a, fadd(ej, ra.e), plummer)), 1.0f);
                    if (rb.v) accb += fx(fmul(rj.w, pair_dir(d2b, fadd(ej, rb.e), plummer)), 1.0f);
                }
            }
        }
        __syncthreads();
        if (ra.v) atomicAdd((unsigned long long *)&pot[s + I * T + t], (unsigned long long)acca);
        if (rb.v) atomicAdd((unsigned long long *)&pot[s + I * T + t + H], (unsigned long long)accb);
        for (int c = t; c < nj; c += POT_THREADS) {
            long long cs = 0;
#pragma unroll
            for (int k = 0; k < NW; ++k) cs += acc_w[k][c];
            if (cs) atomicAdd((unsigned long long *)&pot[s + j0 + c], (unsigned long long)cs);
        }
    }
}

// ---- removal ----

struct ArgRed {
    float v;
    int i;
};

__device__ __forceinline__ ArgRed warp_argmax(ArgRed a)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        float v = __shfl_xor_sync(SKID_FULL, a.v, o);
        int i = __shfl_xor_sync(SKID_FULL, a.i, o);
        if (v > a.v || (v == a.v && i < a.i)) { a.v = v; a.i = i; }
    }
    return a;
}

__device__ __forceinline__ ArgRed warp_argmin(ArgRed a)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        float v = __shfl_xor_sync(SKID_FULL, a.v, o);
        int i = __shfl_xor_sync(SKID_FULL, a.i, o);
        if (v < a.v || (v == a.v && i < a.i)) { a.v = v; a.i = i; }
    }
    return a;
}

// A thread's two largest (a, then b) or two smallest energies, the first
// index kept on ties (members are visited in increasing index).
__device__ __forceinline__ void keep_top2(ArgRed &a, ArgRed &b, float E, int i)
{
    if (E > a.v) { b = a; a.v = E; a.i = i; }
    else if (E > b.v) { b.v = E; b.i = i; }
}

__device__ __forceinline__ void keep_bot2(ArgRed &a, ArgRed &b, float E, int i)
{
    if (E < a.v) { b = a; a.v = E; a.i = i; }
    else if (E < b.v) { b.v = E; b.i = i; }
}

struct RemoveArgs {
    const int *gstart, *gcount;
    int ng, nmax;
    float4 *qr, *qv;
    float4 *qa, *qw;                // block groups' member state beyond shared memory (BlockGroup)
    int lcap;                       // members a block holds in shared memory
    int *qid;
    long long *pot;
    skid_group *rec;
    int *grp;
    int *d_unbound;
    float G, fShift, fCosmo, opz;   // a, a*H(a), 1+z
    float z;
    float scale, inv_scale;         // 2^S, 2^-S
    float3 hP;
    int plummer, subpot, nounbind;
    const uint32_t *order;          // valid groups, largest first
    const int *d_cnt;               // [valid groups, groups above tw]
    int *d_queue, *d_wqueue;        // next group for a block, for a warp
    const int *d_ccnt;              // groups taken by clusters (the largest, a prefix of order)
    int *d_cqueue;
    int qcap;                       // members per block slice a cluster can hold
    int single;                     // > 0: process only this group (per-group mode)
};

// E_i of kd.c:1392-1400: exact form (the reference's FP64 expression with
// each operation rounded as gcc rounds it, no fused multiply-adds, then
// rounded to float) or FP32 form.  Exact form:
//   dv_j = (float)(a * ((double)v_j - vcm_j) + aH * ((double)r_j - rcm_j))
//   dv2  = dv_0^2 + dv_1^2 + dv_2^2                      (float)
//   E    = (float)(0.5 * dv2 - pot * (1.0 + z))
__device__ __forceinline__ float exact_energy(const RemoveArgs &A, float4 r, float4 v, long long p,
                                              const double *dcm, double inv_d, double opz_d)
{
    const double fs = A.fShift, fc = A.fCosmo;
    const float dv0 = (float)__dadd_rn(__dmul_rn(fs, __dsub_rn((double)v.x, dcm[3])),
                                       __dmul_rn(fc, __dsub_rn((double)r.x, dcm[0])));
    const float dv1 = (float)__dadd_rn(__dmul_rn(fs, __dsub_rn((double)v.y, dcm[4])),
                                       __dmul_rn(fc, __dsub_rn((double)r.y, dcm[1])));
    const float dv2 = (float)__dadd_rn(__dmul_rn(fs, __dsub_rn((double)v.z, dcm[5])),
                                       __dmul_rn(fc, __dsub_rn((double)r.z, dcm[2])));
    const float dd = fadd(fadd(fmul(dv0, dv0), fmul(dv1, dv1)), fmul(dv2, dv2));
    // pot * 2^-S is exact (a power-of-two scale of an integer below 2^53)
    return (float)__dsub_rn(__dmul_rn(0.5, (double)dd), __dmul_rn(__dmul_rn((double)p, inv_d), opz_d));
}

__device__ __forceinline__ float member_energy(bool exact, const RemoveArgs &A, float4 r, float4 v,
                                               long long p, const double *dcm, const float *scm,
                                               double inv_d, double opz_d)
{
    if (exact) return exact_energy(A, r, v, p, dcm, inv_d, opz_d);
    float dv0 = A.fShift * (v.x - scm[3]) + A.fCosmo * (r.x - scm[0]);
    float dv1 = A.fShift * (v.y - scm[4]) + A.fCosmo * (r.y - scm[1]);
    float dv2 = A.fShift * (v.z - scm[5]) + A.fCosmo * (r.z - scm[2]);
    float dd = fadd(fadd(fmul(dv0, dv0), fmul(dv1, dv1)), fmul(dv2, dv2));
    return 0.5f * dd - (ll2f_approx(p) * A.inv_scale) * A.opz;
}

// Bound on |FP32 energy - exact energy|: each of them is within a few
// roundings of the real value of the same expression, so 2^-19 of the sum of
// the magnitudes that enter it (velocity and position terms before their
// cancellation, the kinetic term, the potential term) bounds the difference.
__device__ __forceinline__ float energy_err(const RemoveArgs &A, float4 r, float4 v, long long p,
                                            const float *scm, float e32)
{
    const float a = fabsf(A.fShift), c = fabsf(A.fCosmo);
    float s = 0.0f, k = 0.0f;
    const float vv[3] = {v.x, v.y, v.z}, rr[3] = {r.x, r.y, r.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        float mag = a * (fabsf(vv[d]) + fabsf(scm[3 + d])) + c * (fabsf(rr[d]) + fabsf(scm[d]));
        float dv = A.fShift * (vv[d] - scm[3 + d]) + A.fCosmo * (rr[d] - scm[d]);
        s += mag * (2.0f * fabsf(dv) + mag);
        k += dv * dv;
    }
    float pe = fabsf(ll2f_approx(p) * A.inv_scale * A.opz);
    return 1.9073486e-06f * (s + k + pe + fabsf(e32)) + 1e-30f;   // 2^-19
}

// kdSubPot (grav.c:44-59) of the removed particle rs on member (r, v).
__device__ __forceinline__ long long sub_pot(const RemoveArgs &A, float4 rs, float es, float4 r,
                                             float4 v, long long p)
{
    float d2 = d2of(fsub(rs.x, r.x), fsub(rs.y, r.y), fsub(rs.z, r.z));
    float dir = pair_dir(d2, fadd(es, v.w), A.plummer);
    return p - fx(fmul(fmul(A.G, rs.w) * A.scale, dir), 1.0f);
}

// centre of mass after removing (r, v): kd.c:1424-1431,
//   dMass -= m;  rcm_j += m/dMass * (rcm_j - r_j);  vcm_j likewise,
// each FP64 operation rounded separately as the reference's are.
__device__ __forceinline__ void rcm_update(double &mass, double *dcm, float4 r, float4 v)
{
    mass = __dsub_rn(mass, (double)r.w);
    const double f = __ddiv_rn((double)r.w, mass);
    const float x[6] = {r.x, r.y, r.z, v.x, v.y, v.z};
#pragma unroll
    for (int d = 0; d < 6; ++d)
        dcm[d] = __dadd_rn(dcm[d], __dmul_rn(f, __dsub_rn(dcm[d], (double)x[d])));
}

__device__ __forceinline__ void write_record(const RemoveArgs &A, int g, int n, double mass,
                                             const double *dcm, float4 rb, int nrem)
{
    skid_group r = A.rec[g];
    r.nMembers = n;
    r.fMass = (float)mass;
    r.vcm[0] = (float)dcm[3];
    r.vcm[1] = (float)dcm[4];
    r.vcm[2] = (float)dcm[5];
    float hx = A.hP.x;   // kd.c:1452-1456 wraps every axis with hx
    r.rBound[0] = wrap_h(fadd(rb.x, r.rel[0]), hx);
    r.rBound[1] = wrap_h(fadd(rb.y, r.rel[1]), hx);
    r.rBound[2] = wrap_h(fadd(rb.z, r.rel[2]), hx);
    A.rec[g] = r;
    if (nrem) atomicAdd(A.d_unbound, nrem);
}

// A small group, one warp: every lane keeps the FP64 centre itself (the same
// values on every lane), lane 0 writes.
__device__ void warp_group(const RemoveArgs &A, int g)
{
    const int lane = threadIdx.x & 31;
    const int s = A.gstart[g], n0 = A.gcount[g];
    float4 *qr = A.qr + s;
    float4 *qv = A.qv + s;
    int *qid = A.qid + s;
    long long *pot = A.pot + s;
    double m = 0.0, dcm[6] = {0, 0, 0, 0, 0, 0};
    for (int i = lane; i < n0; i += 32) {
        float4 r = qr[i], v = qv[i];
        m += r.w;
        dcm[0] += fmul(r.w, r.x); dcm[1] += fmul(r.w, r.y); dcm[2] += fmul(r.w, r.z);
        dcm[3] += fmul(r.w, v.x); dcm[4] += fmul(r.w, v.y); dcm[5] += fmul(r.w, v.z);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        m += __shfl_xor_sync(SKID_FULL, m, o);
        for (int d = 0; d < 6; ++d) dcm[d] += __shfl_xor_sync(SKID_FULL, dcm[d], o);
    }
    float scm[6];
    for (int d = 0; d < 6; ++d) {
        dcm[d] /= m;
        scm[d] = (float)dcm[d];
    }
    const bool exact = n0 <= EXACT_E_MAX;
    const double opz_d = 1.0 + (double)A.z, inv_d = 1.0 / (double)A.scale;
    int n = n0, nrem = 0, imin = 0;
    bool have = false;
    float4 rs = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float es = 0.0f;
    for (;;) {
        ArgRed mx{-FLT_MAX, 0x7fffffff}, mn{FLT_MAX, 0x7fffffff};
        ArgRed mx2 = mx, mn2 = mn;
        // FP32 energies with error bounds
        float dmax = 0.0f;
        for (int i = lane; i < n; i += 32) {
            float4 r = qr[i], v = qv[i];
            long long p = pot[i];
            if (have && A.subpot) {
                p = sub_pot(A, rs, es, r, v, p);
                pot[i] = p;
            }
            float E = member_energy(false, A, r, v, p, dcm, scm, inv_d, opz_d);
            keep_top2(mx, mx2, E, i);
            keep_bot2(mn, mn2, E, i);
            if (exact) dmax = fmaxf(dmax, energy_err(A, r, v, p, scm, E));
        }
        float hi = 0.0f, lo = 0.0f;
        const ArgRed t1 = mx, b1 = mn;
        // members again, in the same order with the same FP32 energies: the
        // candidates on the asked sides exactly (FP64, as the reference)
        auto rescan = [&](bool scan_hi, bool scan_lo) {
            for (int i = lane; i < n; i += 32) {
                float4 r = qr[i], v = qv[i];
                long long p = pot[i];
                float E = member_energy(false, A, r, v, p, dcm, scm, inv_d, opz_d);
                const bool ch = scan_hi && E >= hi, cl = scan_lo && E <= lo;
                if (ch || cl) {
                    float X = member_energy(true, A, r, v, p, dcm, scm, inv_d, opz_d);
                    if (ch && X > mx.v) { mx.v = X; mx.i = i; }
                    if (cl && X < mn.v) { mn.v = X; mn.i = i; }
                }
            }
        };
        if (exact) {
            // only members whose FP32 energy is within twice the error bound
            // of the extremes can be the exact arg-max / arg-min
            float emax = mx.v, emin = mn.v;
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                emax = fmaxf(emax, __shfl_xor_sync(SKID_FULL, emax, o));
                emin = fminf(emin, __shfl_xor_sync(SKID_FULL, emin, o));
                dmax = fmaxf(dmax, __shfl_xor_sync(SKID_FULL, dmax, o));
            }
            hi = emax - 2.0f * dmax;
            lo = emin + 2.0f * dmax;
            // One candidate alone is the exact arg-max (every other member's
            // exact energy is below emax - dmax, and its own at least that),
            // and the sign of its exact energy is known when its FP32 energy
            // is at least the bound, or below minus the bound: the usual pass
            // needs no FP64 energy.  Otherwise the candidates are evaluated
            // exactly -- usually just the lane's own extreme, else its
            // members again.
            const unsigned chi = __ballot_sync(SKID_FULL, t1.v >= hi);
            const bool one = chi != 0 && (chi & (chi - 1)) == 0 && !__any_sync(SKID_FULL, mx2.v >= hi);
            if (one && emax >= dmax) {
                mx.v = emax;
                mx.i = __shfl_sync(SKID_FULL, t1.i, __ffs(chi) - 1);
            } else if (one && emax < -dmax) {
                mx.v = emax;
            } else {
                mx = ArgRed{-FLT_MAX, 0x7fffffff};
                if (t1.i < n && t1.v >= hi && mx2.v < hi) {
                    mx.v = member_energy(true, A, qr[t1.i], qv[t1.i], pot[t1.i], dcm, scm, inv_d, opz_d);
                    mx.i = t1.i;
                }
                if (mx2.v >= hi) rescan(true, false);
                mx = warp_argmax(mx);
            }
        } else {
            mx = warp_argmax(mx);
        }
        if (!(mx.v >= 0.0f) || A.nounbind || n == 0) {
            // the group's most bound member (kd.c:1389-1409: fTotMin starts
            // at 1), needed only once the removals stop
            if (exact) {
                mn = ArgRed{FLT_MAX, 0x7fffffff};
                if (b1.i < n && b1.v <= lo && mn2.v > lo) {
                    mn.v = member_energy(true, A, qr[b1.i], qv[b1.i], pot[b1.i], dcm, scm, inv_d, opz_d);
                    mn.i = b1.i;
                }
                if (mn2.v <= lo) rescan(false, true);
            }
            mn = warp_argmin(mn);
            imin = mn.v < 1.0f ? mn.i : 0;
            break;
        }
        const int ib = mx.i;
        __syncwarp();
        float4 r = qr[ib], v = qv[ib];
        __syncwarp();   // every lane has read the removed member before lane 0 swaps it away
        if (lane == 0) A.grp[qid[ib]] = 0;
        ++nrem;
        const int nn = n - 1;
        if (nn == 0) {
            m = 0.0;
            dcm[3] = dcm[4] = dcm[5] = 0.0;
            n = 0;
            break;
        }
        rcm_update(m, dcm, r, v);
        for (int d = 0; d < 6; ++d) scm[d] = (float)dcm[d];
        if (lane == 0) {
            // swap with the last member (kd.c:1435-1440)
            float4 rl = qr[nn], vl = qv[nn];
            int il = qid[nn], ir = qid[ib];
            long long pl = pot[nn], pb = pot[ib];
            qr[ib] = rl; qv[ib] = vl; qid[ib] = il; pot[ib] = pl;
            qr[nn] = r; qv[nn] = v; qid[nn] = ir; pot[nn] = pb;
        }
        __syncwarp();
        rs = r;
        es = v.w;
        have = true;
        n = nn;
    }
    __syncwarp();
    if (lane == 0) write_record(A, g, n, m, dcm, qr[imin], nrem);
    __syncwarp();
}

// Members near an extreme are evaluated exactly one by one, each with the terms
// of all members removed since potentials were last brought up to date (a unit
// of work per 32 of them, latency, takes some UNIT_COST times as long as one
// term does in bulk).  When these have cost as much as bringing every member up
// to date would, or there are more than CAND_MAX of them, that is done instead:
// exact ties come back pass after pass.  6,000 members with 600 fast ones, by
// threes at one place each 5.2 ms, by thirties 15 (25 with a block to each
// candidate and no limit but CAND_MAX, 19 with that at 8; 10 where every pass
// was exact, which takes 5 for 600 places against 1.5).  Where candidates are
// few neither limit matters: CAND_MAX 8, 32 and 128 and UNIT_COST 10 to 2000
// time alike within 1 % on the groups of 20,000- to 400,000-particle catalogues.
constexpr int CAND_MAX = 32;
constexpr float UNIT_COST = 50.0f;

template <int BS>
struct BlockShared {
    ArgRed smax[BS / 32], smin[BS / 32];
    float4 s_r;
    float s_eps;
    float s_cm[6];
    int s_n, s_go, s_have, s_imin, s_item;
    double d_cm[6], d_mass;
    double part[BS / 32][7];
    float ext[BS / 32][4];      // per-warp partials: FP32 energy max, min, error-bound terms
    float s_w[3];               // a vcm + aH rcm (the members' FP32 energies)
    float s_mW;                 // max_j |a vcm_j| + |aH rcm_j|
    float s_mg;                 // max over members and axes of |a v_j| + |aH r_j|
    float gpart[8][4];          // a cluster's blocks' partials, gathered (rank order)
    ArgRed gmx[8], gmn[8];
    // block_group, by parity of the pass: per-warp largest and second largest
    // energy, largest kinetic term (ordered bits), the largest's slot and state
    unsigned wbest[2][BS / 32], wnext[2][BS / 32], wkin[2][BS / 32];
    int wi[2][BS / 32];
    float4 wa[2][BS / 32], wb[2][BS / 32];
    float pub_w[2][3], pub_mW[2], pub_mass[2];   // W, its magnitude and the group's mass
    int ncand;
    int spent;                  // candidates' terms (per 32) since potentials were brought up to date
    ArgRed cand[CAND_MAX];
    unsigned long long candq[CAND_MAX];
};

// max_j |a c_j| + |aH c_{j-3}| of a centre (rcm, vcm)
__device__ __forceinline__ float centre_mag(const RemoveArgs &A, const double *dcm)
{
    float m = 0.0f;
#pragma unroll
    for (int d = 0; d < 3; ++d)
        m = fmaxf(m, fabsf(A.fShift * (float)dcm[3 + d]) + fabsf(A.fCosmo * (float)dcm[d]));
    return m * 1.0000002f;
}

// A large group, the whole block.
//
// A group's removals are a serial chain -- one pass over its members per
// removed member -- and the largest groups' chains set the time of the whole
// unbinding, so a pass is made short:
//  - Between the few exact decisions a member's potential is kept only as a
//    compensated float that each removal changes by the hardware 1/r: about
//    25 issue slots a member instead of about 170 for the reference's pair
//    factor in fixed point, and no 64-bit arithmetic.  The exact potential of
//    a member is its stored one less the terms of the members removed since
//    (they lie behind the live ones, slots [n, nfl)); it is formed only for
//    the members an exact decision needs, or for every member at once (flush)
//    when those are many.
//  - Members sit in shared memory (32 B each, the first A.lcap of them; the
//    rest in global memory), two to a record so that a thread takes both in
//    packed FP32 operations.
//  - One barrier carries the warps' two largest energies, the largest's state
//    and the largest kinetic term, from which every warp forms the same
//    decision and the next centre to one float step; the block's last warp
//    (the keeper) meanwhile brings the FP64 centre and the records in global
//    memory up to date behind the pass that follows.
// Removal at 2^21 (271 groups above 1024 members, the largest of 10,024, up to
// 1,092 removed from one of 9,620) 4.65 ms, 10.4 with the exact terms every
// pass, members in L2 and three barriers; 300 groups of up to 6.6k 2.2 to 0.66;
// 5k particles 1.51 to 0.63.  A pass over 600 members takes 3300 cycles, over
// 3700 3700.  What was
// measured and left out: members in packed records in global memory too, the
// next record loaded ahead, and velocities instead of w in the records (so
// that the keeper reads none) were each no faster.
template <int BS>
struct BlockGroup {
    static constexpr int NW = BS / 32;
    static constexpr int BC = BS - 32;   // threads that carry members
    const RemoveArgs &A;
    BlockShared<BS> &S;
    float4 *qr, *qv;
    int *qid;
    long long *pot;
    float *sm;                       // records in shared memory
    // state in global memory, by slot: (u, v, w, x), (y, z) and, all that a
    // pass writes, (p, c): whole sectors, where a member's 32 bytes in two
    // float4s had two sectors written for four bytes each.  Without a
    // potential to take off a pass reads no y and z.
    float4 *gux;
    float2 *gyz, *gpc;
    int cap;                         // slots in shared memory
    int tid, lane, w;
    int n, nfl;                      // live members; slots below nfl have potentials as of then
    float epot;
    bool force;                      // exact potentials every pass

    // Slot i (thread i % BC, its k-th member) lies in half k & 1 of record
    // (k >> 1) BC + i % BC: x x' y y' | z z' p p' | u u' v v' | w w' c c', with
    // p = -(potential energy), c its compensation, (u, v, w) = a v + aH r.  The
    // four quarters of the records are arrays of their own, so that a warp's
    // 16-byte accesses are contiguous.
    static __device__ __forceinline__ int word(int i)
    {
        const int k = i / BC, t = i - k * BC;
        return (((k >> 1) * BC + t) << 2) + (k & 1);
    }
    // (x, y, z, p) and (u, v, w, c) of a slot
    __device__ __forceinline__ void gget(int i, float4 &a, float4 &b, bool yz = true) const
    {
        const float4 r = gux[i];
        const float2 p = gpc[i], v = yz ? gyz[i] : make_float2(0.0f, 0.0f);
        a = make_float4(r.w, v.x, v.y, p.x);
        b = make_float4(r.x, r.y, r.z, p.y);
    }
    __device__ __forceinline__ void get(int i, float4 &a, float4 &b) const
    {
        if (i < cap) {
            const float *q = sm + word(i);
            const int c2 = 2 * cap;
            a = make_float4(q[0], q[2], q[c2], q[c2 + 2]);
            b = make_float4(q[2 * c2], q[2 * c2 + 2], q[3 * c2], q[3 * c2 + 2]);
        } else {
            gget(i, a, b);
        }
    }
    __device__ __forceinline__ void put(int i, float4 a, float4 b) const
    {
        if (i < cap) {
            float *q = sm + word(i);
            const int c2 = 2 * cap;
            q[0] = a.x; q[2] = a.y; q[c2] = a.z; q[c2 + 2] = a.w;
            q[2 * c2] = b.x; q[2 * c2 + 2] = b.y; q[3 * c2] = b.z; q[3 * c2 + 2] = b.w;
        } else {
            gux[i] = make_float4(b.x, b.y, b.z, a.x);
            gyz[i] = make_float2(a.y, a.z);
            gpc[i] = make_float2(a.w, b.w);
        }
    }

    // FP32 filter energy E = 1/2 |w - W|^2 + p, each operation rounded as
    // written (the packed form's too), so every evaluation of a member gives
    // the same value.
    static __device__ __forceinline__ float energy(float4 a, float4 b, float wx, float wy, float wz,
                                                   float &dd)
    {
        const float dx = __fsub_rn(b.x, wx), dy = __fsub_rn(b.y, wy), dz = __fsub_rn(b.z, wz);
        dd = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
        return __fmaf_rn(0.5f, dd, a.w);
    }

    // Exact fixed-point terms of the removed members in slots [from, nfl), a
    // stride apart, on a member (kdSubPot, grav.c:44-59).
    __device__ __forceinline__ long long pending(float4 r, float soft, int from, int stride) const
    {
        long long q = 0;
        for (int e = from; e < nfl; e += stride) {
            const float4 rs = qr[e];
            const float d2 = d2of(fsub(rs.x, r.x), fsub(rs.y, r.y), fsub(rs.z, r.z));
            q += fx(fmul(fmul(A.G, rs.w) * A.scale, pair_dir(d2, fadd(qv[e].w, soft), A.plummer)), 1.0f);
        }
        return q;
    }

    // The exact arg-max (or arg-min), first member on ties, among the members
    // whose FP32 energy against (wx, wy, wz) reaches lim.  Called by the whole
    // block, on a copy of the view (so that the caller's stays in registers),
    // with the published FP64 centre current; *flushed says whether every
    // member's potential is now exact.
    template <bool MAX>
    static __device__ __noinline__ ArgRed decide(BlockGroup B, float wx, float wy, float wz, float lim,
                                                 bool *flushed)
    {
        return B.template decide_in<MAX>(wx, wy, wz, lim, flushed);
    }

    template <bool MAX>
    __device__ __forceinline__ ArgRed decide_in(float wx, float wy, float wz, float lim, bool *flushed)
    {
        *flushed = false;
        const double inv_d = 1.0 / (double)A.scale, opz_d = 1.0 + (double)A.z;
        double dcm[6];
        for (int d = 0; d < 6; ++d) dcm[d] = S.d_cm[d];
        __syncthreads();
        if (tid == 0) S.ncand = 0;
        if (tid < CAND_MAX) S.candq[tid] = 0;
        __syncthreads();
        for (int i = tid; i < n; i += BS) {
            float4 a, b;
            float dd;
            get(i, a, b);
            const float E = energy(a, b, wx, wy, wz, dd);
            if (MAX ? E >= lim : E <= lim) {
                const int k = atomicAdd(&S.ncand, 1);
                if (k < CAND_MAX) S.cand[k].i = i;
            }
        }
        __syncthreads();
        const int nc = S.ncand;
        ArgRed best{MAX ? -FLT_MAX : FLT_MAX, 0x7fffffff};
        auto better = [&](ArgRed x) {
            return MAX ? x.v > best.v || (x.v == best.v && x.i < best.i)
                       : x.v < best.v || (x.v == best.v && x.i < best.i);
        };
        // (a warp for each 32 removed members of a candidate; in bulk, each thread
        // all of them in turn for its members)
        const int m = A.subpot ? nfl - n : 0, mw = (m + 31) / 32, units = nc * mw, spent = S.spent + units;
        if (nc <= CAND_MAX && !force && (m == 0 || spent * UNIT_COST <= (float)max(n, BS) * (float)m)) {
            for (int u = w; u < units; u += NW) {
                const int k = u / mw, i = S.cand[k].i, e = n + (u - k * mw) * 32 + lane;
                long long q = e < nfl ? pending(qr[i], qv[i].w, e, nfl) : 0;
#pragma unroll
                for (int o = 16; o; o >>= 1) q += __shfl_xor_sync(SKID_FULL, q, o);
                if (lane == 0) atomicAdd(&S.candq[k], (unsigned long long)q);
            }
            __syncthreads();
            if (tid < nc) {
                const int i = S.cand[tid].i;
                S.cand[tid].v =
                    exact_energy(A, qr[i], qv[i], pot[i] - (long long)S.candq[tid], dcm, inv_d, opz_d);
            }
            __syncthreads();
            for (int k = 0; k < nc; ++k)
                if (better(S.cand[k])) best = S.cand[k];
            if (tid == 0) S.spent = spent;
            __syncthreads();
            return best;
        }
        for (int i = tid; i < n; i += BS) {
            float4 a, b;
            float dd;
            get(i, a, b);
            const float E = energy(a, b, wx, wy, wz, dd);
            const float4 r = qr[i], v = qv[i];
            const long long p = pot[i] - (A.subpot ? pending(r, v.w, n, 1) : 0);
            pot[i] = p;
            a.w = -(ll2f_approx(p) * epot);
            b.w = 0.0f;
            put(i, a, b);
            if (force || (MAX ? E >= lim : E <= lim)) {
                const ArgRed x{exact_energy(A, r, v, p, dcm, inv_d, opz_d), i};
                if (better(x)) best = x;
            }
        }
        *flushed = true;
        if (tid == 0) S.spent = 0;
        best = MAX ? warp_argmax(best) : warp_argmin(best);
        if (lane == 0) S.smax[w] = best;
        __syncthreads();
        best = S.smax[0];
        for (int k = 1; k < NW; ++k)
            if (better(S.smax[k])) best = S.smax[k];
        __syncthreads();
        return best;
    }
};

template <int BS>
__device__ void block_group(const RemoveArgs &A, int g, BlockShared<BS> &S, float4 *dyn)
{
    using BG = BlockGroup<BS>;
    constexpr int NW = BG::NW, BC = BG::BC;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const bool keeper = w == NW - 1;
    const int s = A.gstart[g], n0 = A.gcount[g];
    float4 *qr = A.qr + s, *qv = A.qv + s;
    int *qid = A.qid + s;
    long long *pot = A.pot + s;
    // slots in shared memory: whole records of a row of BC threads
    const int cap = A.lcap / (2 * BC) * (2 * BC);
    float *sm = reinterpret_cast<float *>(dyn);
    float4 *gux = A.qa + s;
    float2 *gyz = reinterpret_cast<float2 *>(A.qw + s), *gpc = gyz + n0;
    int n = n0, nfl = n0;
    bool force = false;
    const float epot = A.inv_scale * A.opz;
    auto view = [&]() {
        return BG{A, S, qr, qv, qid, pot, sm, gux, gyz, gpc, cap, tid, lane, w, n, nfl, epot, force};
    };
    double m = 0.0, c[6] = {0, 0, 0, 0, 0, 0};
    for (int i = tid; i < n0; i += BS) {
        float4 r = qr[i], v = qv[i];
        m += r.w;
        c[0] += fmul(r.w, r.x); c[1] += fmul(r.w, r.y); c[2] += fmul(r.w, r.z);
        c[3] += fmul(r.w, v.x); c[4] += fmul(r.w, v.y); c[5] += fmul(r.w, v.z);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        m += __shfl_xor_sync(SKID_FULL, m, o);
        for (int d = 0; d < 6; ++d) c[d] += __shfl_xor_sync(SKID_FULL, c[d], o);
    }
    __syncthreads();
    if (lane == 0) {
        S.part[w][0] = m;
        for (int d = 0; d < 6; ++d) S.part[w][1 + d] = c[d];
    }
    // Every member's state: FP32 filter energies E_i = 1/2 |w_i - W|^2 + p_i,
    // with w_i = a v_i + aH r_i fixed per member and W = a vcm + aH rcm per
    // pass; their error bound needs the largest |a v_j| + |aH r_j| and the
    // largest |p|.
    float mg = 0.0f, gpe = 0.0f;
    float emax = -FLT_MAX, emin = FLT_MAX, mmax = -FLT_MAX, mmin = FLT_MAX;
    bool odd = !(A.G >= 0.0f) || !(A.opz >= 0.0f);
    {
        const BG B = view();
        for (int i = tid; i < n0; i += BS) {
            const float4 r = qr[i], v = qv[i];
            const float p = -(ll2f_approx(pot[i]) * epot);
            B.put(i, make_float4(r.x, r.y, r.z, p),
                  make_float4(__fmaf_rn(A.fShift, v.x, A.fCosmo * r.x),
                              __fmaf_rn(A.fShift, v.y, A.fCosmo * r.y),
                              __fmaf_rn(A.fShift, v.z, A.fCosmo * r.z), 0.0f));
            mg = fmaxf(mg, fabsf(A.fShift * v.x) + fabsf(A.fCosmo * r.x));
            mg = fmaxf(mg, fabsf(A.fShift * v.y) + fabsf(A.fCosmo * r.y));
            mg = fmaxf(mg, fabsf(A.fShift * v.z) + fabsf(A.fCosmo * r.z));
            gpe = fmaxf(gpe, fabsf(p));
            emax = fmaxf(emax, v.w);
            emin = fminf(emin, v.w);
            mmax = fmaxf(mmax, r.w);
            mmin = fminf(mmin, r.w);
            // the bound takes every removed term as part of the first
            // potential, which a negative mass, G or softening would break
            odd = odd || !(r.w >= 0.0f) || !(v.w >= 0.0f);
        }
    }
    mg = __uint_as_float(__reduce_max_sync(SKID_FULL, __float_as_uint(mg)));
    gpe = __uint_as_float(__reduce_max_sync(SKID_FULL, __float_as_uint(gpe)));
    emax = ord2f(__reduce_max_sync(SKID_FULL, f2ord(emax)));
    emin = ord2f(__reduce_min_sync(SKID_FULL, f2ord(emin)));
    mmax = ord2f(__reduce_max_sync(SKID_FULL, f2ord(mmax)));
    mmin = ord2f(__reduce_min_sync(SKID_FULL, f2ord(mmin)));
    odd = __any_sync(SKID_FULL, odd);
    if (lane == 0) {
        S.wa[0][w] = make_float4(mg, gpe, emax, emin);
        S.wb[0][w] = make_float4(mmax, mmin, 0.0f, 0.0f);
        S.wi[0][w] = odd;
    }
    __syncthreads();
    for (int k = 0; k < NW; ++k) {
        const float4 x = S.wa[0][k], y = S.wb[0][k];
        mg = fmaxf(mg, x.x);
        gpe = fmaxf(gpe, x.y);
        emax = fmaxf(emax, x.z);
        emin = fminf(emin, x.w);
        mmax = fmaxf(mmax, y.x);
        mmin = fminf(mmin, y.y);
        force = force || S.wi[0][k];
    }
    mg *= 1.0000002f;
    // one mass and one softening: a pass reads no record from global memory
    const bool uniform = mmin == mmax && emin == emax;
    if (tid == 0) {
        // warp partials in warp order: the same sums on every run
        double t[7] = {0, 0, 0, 0, 0, 0, 0};
        for (int k = 0; k < NW; ++k)
            for (int d = 0; d < 7; ++d) t[d] += S.part[k][d];
        S.d_mass = t[0];
        for (int d = 0; d < 6; ++d) S.d_cm[d] = t[1 + d] / t[0];
        for (int d = 0; d < 3; ++d)
            S.pub_w[0][d] = (float)((double)A.fShift * S.d_cm[3 + d] + (double)A.fCosmo * S.d_cm[d]);
        S.pub_mW[0] = centre_mag(A, S.d_cm);
        S.pub_mass[0] = (float)t[0];
        S.s_imin = 0;
        S.spent = 0;
    }
    __syncthreads();
    int nrem = 0, par = 0;           // the same on every thread
    int ib = 0;                      // the last removed member's slot, and its state
    float4 ra = make_float4(0.0f, 0.0f, 0.0f, 0.0f), rb = ra;
    float gms = 0.0f, es = 0.0f;     // its G m (1+z) and softening
    float f = 0.0f;                  // its m / (mass left)
    float wx = S.pub_w[0][0], wy = S.pub_w[0][1], wz = S.pub_w[0][2];
    // The keeper: FP64 centre (kd.c:1424-1431, a lane per component) and, with
    // uniform members, the records' swap with the last member (kd.c:1435-1440)
    // for the member removed last; n is the slot it goes to.
    auto keep = [&]() {
        const float4 r = qr[ib], v = qv[ib];
        const int qb = qid[ib];
        const float4 rl = qr[n], vl = qv[n];
        const int ql = qid[n];
        const long long pl = pot[n];
        // a known mass lets the division run while the records arrive
        const double dm = (double)(uniform ? mmax : r.w);
        const double mm = __dsub_rn(S.d_mass, dm);
        const double fd = __ddiv_rn(dm, mm);
        const int d = lane < 6 ? lane : 0;
        const double x =
            (double)(d == 0 ? r.x : d == 1 ? r.y : d == 2 ? r.z : d == 3 ? v.x : d == 4 ? v.y : v.z);
        const double o = S.d_cm[d];
        const double cn = __dadd_rn(o, __dmul_rn(fd, __dsub_rn(o, x)));
        const double vd = __shfl_sync(SKID_FULL, cn, (d % 3) + 3);
        const double rd = __shfl_sync(SKID_FULL, cn, d % 3);
        const float W = (float)((double)A.fShift * vd + (double)A.fCosmo * rd);
        const float mag = (fabsf(A.fShift * (float)vd) + fabsf(A.fCosmo * (float)rd)) * 1.0000002f;
        const float mW = __uint_as_float(__reduce_max_sync(SKID_FULL, __float_as_uint(mag)));
        __syncwarp();
        if (lane < 6) S.d_cm[lane] = cn;
        if (lane < 3) S.pub_w[par][lane] = W;
        if (lane == 0) {
            S.d_mass = mm;
            S.pub_mass[par] = (float)mm;
            S.pub_mW[par] = mW;
            if (uniform) {
                A.grp[qb] = 0;
                qr[ib] = rl; qv[ib] = vl; qid[ib] = ql; pot[ib] = pl;
                qr[n] = r; qv[n] = v; qid[n] = qb;
            }
        }
    };
    for (;;) {
        const bool sub = nrem > 0 && A.subpot;
        // after a member that held much of the mass the float step is not
        // good enough: the pass waits for the FP64 centre
        const bool late = f <= 0.25f;
        if (!late) {
            if (keeper) keep();
            __syncthreads();
            wx = S.pub_w[par][0];
            wy = S.pub_w[par][1];
            wz = S.pub_w[par][2];
            f = 0.0f;
        }
        // beyond far every member's pair with the removed one is 1/r
        const float far = A.plummer ? INFINITY : fmaxf((es + emax) * (es + emax) * 1.000001f, 1e-30f);
        float m1 = -FLT_MAX, m2 = -FLT_MAX, ddmx = 0.0f;
        int i1 = 0x7fffffff;
        if (!keeper) {
            // the pair factor of the removed member for one nearer than far
            auto near_dir = [&](float dx, float dy, float dz, int i) {
                const float e = uniform ? emax : qv[i].w;
                if (A.plummer) {
                    const float t = es + e;
                    return rsqrtf(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)) + 0.25f * t * t);
                }
                return pair_dir_call(d2of(dx, dy, dz), fadd(es, e));
            };
            auto track = [&](float E, float dd, int i) {
                m2 = fmaxf(m2, fminf(m1, E));
                if (E > m1) i1 = i;
                m1 = fmaxf(m1, E);
                ddmx = fmaxf(ddmx, dd);
            };
            auto single = [&](int i, float4 &a, float4 &b) {
                if (sub) {
                    const float dx = a.x - ra.x, dy = a.y - ra.y, dz = a.z - ra.z;
                    const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx));
                    float dir;
                    if (d2 >= far) asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(dir) : "f"(d2));
                    else dir = near_dir(dx, dy, dz, i);
                    const float y = __fmaf_rn(gms, dir, b.w), t = __fadd_rn(a.w, y);
                    b.w = __fsub_rn(y, __fsub_rn(t, a.w));
                    a.w = t;
                }
                float dd;
                const float E = BG::energy(a, b, wx, wy, wz, dd);
                track(E, dd, i);
            };
            const int ns = min(n, cap);
            int i = tid;
            {
                const f32x2 nrx = pack2(-ra.x, -ra.x), nry = pack2(-ra.y, -ra.y), nrz = pack2(-ra.z, -ra.z);
                const f32x2 nwx = pack2(-wx, -wx), nwy = pack2(-wy, -wy), nwz = pack2(-wz, -wz);
                const f32x2 gm2 = pack2(gms, gms), half2 = pack2(0.5f, 0.5f);
                ulonglong2 *q0 = reinterpret_cast<ulonglong2 *>(sm) + tid;
                const int h = cap >> 1;
                ulonglong2 *q1 = q0 + h, *q2 = q1 + h, *q3 = q2 + h;
#pragma unroll 2
                for (; i + BC < ns; i += 2 * BC, q0 += BC, q1 += BC, q2 += BC, q3 += BC) {
                    const ulonglong2 r0 = *q0, r1 = *q1, r2 = *q2, r3 = *q3;
                    f32x2 P = r1.y;
                    if (sub) {
                        const f32x2 dx = add2(r0.x, nrx), dy = add2(r0.y, nry), dz = add2(r1.x, nrz);
                        const float2 d2 = unpack2(fma2(dz, dz, fma2(dy, dy, mul2(dx, dx))));
                        float2 dir;
                        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(dir.x) : "f"(d2.x));
                        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(dir.y) : "f"(d2.y));
                        if (!(fminf(d2.x, d2.y) >= far)) {
                            const float2 X = unpack2(dx), Y = unpack2(dy), Z = unpack2(dz);
                            if (!(d2.x >= far)) dir.x = near_dir(X.x, Y.x, Z.x, i);
                            if (!(d2.y >= far)) dir.y = near_dir(X.y, Y.y, Z.y, i + BC);
                        }
                        // p + G m (1+z) dir, compensated
                        const f32x2 y = fma2(gm2, pack2(dir.x, dir.y), r3.y);
                        const f32x2 t = add2(P, y);
                        q3->y = sub2(y, sub2(t, P));
                        q1->y = t;
                        P = t;
                    }
                    const f32x2 ux = add2(r2.x, nwx), uy = add2(r2.y, nwy), uz = add2(r3.x, nwz);
                    const f32x2 dd2 = fma2(uz, uz, fma2(uy, uy, mul2(ux, ux)));
                    const float2 E = unpack2(fma2(half2, dd2, P)), dd = unpack2(dd2);
                    track(E.x, dd.x, i);
                    track(E.y, dd.y, i + BC);
                }
            }
            const BG B = view();
            if (i < ns) {
                float4 a, b;
                B.get(i, a, b);
                single(i, a, b);
                if (sub) B.put(i, a, b);
                i += BC;
            }
            // a thread's first slot past the shared ones has its own column
            if (i < cap) i += (cap - i + BC - 1) / BC * BC;
            constexpr int RG = 4;    // loads in flight
            for (; i < n; i += RG * BC) {
                float4 a[RG], b[RG];
#pragma unroll
                for (int k = 0; k < RG; ++k)
                    if (i + k * BC < n) B.gget(i + k * BC, a[k], b[k], sub);
#pragma unroll
                for (int k = 0; k < RG; ++k) {
                    if (i + k * BC >= n) break;
                    single(i + k * BC, a[k], b[k]);
                    if (sub) gpc[i + k * BC] = make_float2(a[k].w, b[k].w);
                }
            }
            // the warp's largest energy and its member, and its second largest
            const unsigned u = f2ord(m1), best = __reduce_max_sync(SKID_FULL, u);
            const int fl = __ffs(__ballot_sync(SKID_FULL, u == best)) - 1;
            const unsigned next = __reduce_max_sync(SKID_FULL, lane == fl ? f2ord(m2) : u);
            const unsigned kin = __reduce_max_sync(SKID_FULL, __float_as_uint(ddmx));
            if (lane == fl) {
                S.wbest[par][w] = best;
                S.wnext[par][w] = next;
                S.wkin[par][w] = kin;
                S.wi[par][w] = i1;
                if (i1 < n) {
                    float4 a, b;
                    B.get(i1, a, b);
                    S.wa[par][w] = a;
                    S.wb[par][w] = b;
                }
            }
        } else if (nrem > 0 && late) {
            keep();
        }
        __syncthreads();
        // Published for every removal so far.
        const float pwx = S.pub_w[par][0], pwy = S.pub_w[par][1], pwz = S.pub_w[par][2];
        const float mW = S.pub_mW[par], mass = S.pub_mass[par];
        float gmax, gnext, gdd;
        int kw;
        {
            const bool in = lane < NW - 1;
            const unsigned u = in ? S.wbest[par][lane] : 0u;
            const unsigned best = __reduce_max_sync(SKID_FULL, u);
            kw = __ffs(__ballot_sync(SKID_FULL, in && u == best)) - 1;
            const unsigned x = in ? S.wnext[par][lane] : 0u;
            const unsigned next = __reduce_max_sync(SKID_FULL, lane == kw ? x : u);
            gdd = __uint_as_float(__reduce_max_sync(SKID_FULL, in ? S.wkin[par][lane] : 0u));
            gmax = ord2f(best);
            gnext = ord2f(next);
        }
        // Bound on |E_i(FP32) - E_i(reference)|.  With C at or above every
        // |a v_j| + |aH r_j| of a member plus the centre's: w_i - W is within
        // 2^-23 C + 2^-23 |dv| of the reference's dv in each component (w_i's
        // two roundings 2^-23 of a member's magnitude; W, one float step from
        // the published rounding of the FP64 centre, 2^-23 of the centre's and
        // 2^-22 f C; the subtraction's and the reference's own rounding 2^-24
        // |dv| each), so 1/2 |dv|^2 is within 2^-23 (1.7321 C sqrt(dd) +
        // 3.25 dd) (both sides' sums of squares 3 x 2^-24 x dd / 2 included).
        // p starts within 2^-22 of the potential's energy; a removed term is
        // within 10 x 2^-24 of the exact one (hardware root 2^-22.9, squared
        // distance 2.8, products 2, the exact term's two float roundings 2,
        // the sum's 1) besides its rounding to the fixed-point quantum, and
        // together the terms are no more than the first potential; the
        // compensated sum adds 2 x 2^-24: in all 2^-20 of the group's largest.
        // Both energies' last rounding: 2^-24 (dd + 2 |p|).  Twice all that:
        const float C = (mg + mW) * (1.0f + 4.0f * f);
        const float bnd = 2.0f * (1.1920929e-07f * (1.7320509f * C * sqrtf(gdd) + 3.75f * gdd) +
                                  1e-12f * C * C + 1.1e-06f * gpe + (float)nrem * epot) +
                          1e-30f;
        // Only members within twice the bound of the extremes can be the
        // exact arg-max or arg-min.  One candidate alone is the exact arg-max
        // (every other member's exact energy is below gmax - bnd, its own at
        // least that), and the sign of its exact energy is known when
        // gmax >= bnd or gmax < -bnd: the usual pass evaluates no FP64 energy.
        const float hi = gmax - 2.0f * bnd;
        bool go;
        if (A.nounbind || n == 0) {
            go = false;
        } else if (!force && gnext < hi && gmax >= bnd) {
            go = true;
            ib = S.wi[par][kw];
            ra = S.wa[par][kw];
            rb = S.wb[par][kw];
        } else if (!force && gnext < hi && gmax < -bnd) {
            go = false;
        } else {
            bool flushed;
            const ArgRed x = BG::template decide<true>(view(), wx, wy, wz, hi, &flushed);
            if (flushed) nfl = n;
            go = x.v >= 0.0f;   // kd.c:1389-1409: fTotBig starts at -1
            if (go) {
                ib = x.i;
                view().get(ib, ra, rb);
                __syncthreads();     // before the slot is overwritten
            }
        }
        if (!go) {
            // the group's most bound member (fTotMin starts at 1), needed
            // only once the removals stop
            float gmin = FLT_MAX;
            {
                const BG B = view();
                for (int k = tid; k < n; k += BS) {
                    float4 a, b;
                    float dd;
                    B.get(k, a, b);
                    gmin = fminf(gmin, BG::energy(a, b, wx, wy, wz, dd));
                }
            }
            gmin = ord2f(__reduce_min_sync(SKID_FULL, f2ord(gmin)));
            if (lane == 0) S.ext[w][0] = gmin;
            __syncthreads();
            for (int k = 0; k < NW; ++k) gmin = fminf(gmin, S.ext[k][0]);
            bool flushed;
            const ArgRed x =
                BG::template decide<false>(view(), wx, wy, wz, gmin + 2.0f * bnd, &flushed);
            if (tid == 0) S.s_imin = x.v < 1.0f ? x.i : 0;
            break;
        }
        // Remove member ib: the last member takes its slot.
        const float ms = uniform ? mmax : qr[ib].w;
        es = uniform ? emax : qv[ib].w;
        gms = fmul(A.G, ms) * A.opz;
        ++nrem;
        --n;
        if (n == 0) {
            if (tid == 0) {
                A.grp[qid[ib]] = 0;
                S.d_mass = 0.0;
                for (int d = 3; d < 6; ++d) S.d_cm[d] = 0.0;
            }
            break;
        }
        // the centre without it, one float step from the published one
        f = __fdividef(ms, mass - ms);
        wx = __fmaf_rn(f, pwx - rb.x, pwx);
        wy = __fmaf_rn(f, pwy - rb.y, pwy);
        wz = __fmaf_rn(f, pwz - rb.z, pwz);
        if (!uniform) {
            // masses and softenings are read from the records during a pass:
            // they move before it
            __syncthreads();
            if (tid == 0) {
                const float4 r = qr[ib], v = qv[ib], rl = qr[n], vl = qv[n];
                const int qb = qid[ib], ql = qid[n];
                A.grp[qb] = 0;
                qr[ib] = rl; qv[ib] = vl; qid[ib] = ql; pot[ib] = pot[n];
                qr[n] = r; qv[n] = v; qid[n] = qb;
            }
            __syncthreads();
            if (keeper) ib = n;      // where its record is now
        }
        if (!keeper) {
            // its owner moves the state before it comes to the slot
            if (ib % BC == tid && ib != n) {
                const BG B = view();
                float4 a, b;
                B.get(n, a, b);
                B.put(ib, a, b);
            }
        }
        par ^= 1;
    }
    __syncthreads();
    if (tid == 0) {
        double dcm[6];
        for (int d = 0; d < 6; ++d) dcm[d] = S.d_cm[d];
        write_record(A, g, n, S.d_mass, dcm, qr[S.s_imin], nrem);
    }
    __syncthreads();
}

// ---- the largest groups: one thread-block cluster each ----
//
// One of the largest groups can be shared by the CS blocks of one cluster.
// Block c holds slots [c Q, (c+1) Q) of the members (Q = ceil(n0 / CS)) in
// shared memory: relative position and mass, the staged w = a v + aH r with
// the softening, and the fixed-point potential, so every pass reads on-chip
// memory instead of L2.  A removal takes three cluster barriers:
//   1. each block's FP32 extremes and error-bound terms are gathered from
//      all blocks' shared memory (distributed shared memory) and combined in
//      rank order, so every block holds the same candidate thresholds;
//   2. likewise the blocks' exact arg-max and arg-min (first index on ties)
//      give every block the same decision; each reads the removed member from
//      its owner block and updates its FP64 centre;
//   3. once all have read it, the owner of the freed slot copies the last
//      member into it (swap with the last, kd.c:1435-1440).
// Velocities, positions and ids in global memory are swapped the same way:
// velocities are read only for the exact energies of the few candidates and
// for the removed member.
struct ClusterShared {
    float part[4];          // block FP32 max, min, max dd, max |pe|
    ArgRed pmax, pmin;      // block exact arg-max, arg-min
    double psum[7];         // block FP64 sums: mass, m r, m v
    float pmg;              // block max |a v_j| + |aH r_j|
    int item;
};

template <int BS, int CS>
__device__ void cluster_group(const RemoveArgs &A, int g, BlockShared<BS> &S, ClusterShared &C,
                              float4 *dyn, cg::cluster_group &cl)
{
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int rank = (int)cl.block_rank();
    const int s = A.gstart[g], n0 = A.gcount[g];
    const int Q = (n0 + CS - 1) / CS;
    const int lo = rank * Q, hi = min(lo + Q, n0);
    float4 *s_r = dyn, *s_w = dyn + A.qcap;
    long long *s_p = reinterpret_cast<long long *>(dyn + 2 * A.qcap);
    float4 *qr = A.qr + s, *qv = A.qv + s;
    int *qid = A.qid + s;
    const long long *pot = A.pot + s;
    // the slice into shared memory, its FP64 sums and member magnitudes
    double m = 0.0, c[6] = {0, 0, 0, 0, 0, 0};
    float mg = 0.0f;
    for (int i = lo + tid; i < hi; i += BS) {
        const float4 r = qr[i], v = qv[i];
        s_r[i - lo] = r;
        s_w[i - lo] = make_float4(__fmaf_rn(A.fShift, v.x, A.fCosmo * r.x),
                                  __fmaf_rn(A.fShift, v.y, A.fCosmo * r.y),
                                  __fmaf_rn(A.fShift, v.z, A.fCosmo * r.z), v.w);
        s_p[i - lo] = pot[i];
        m += r.w;
        c[0] += fmul(r.w, r.x); c[1] += fmul(r.w, r.y); c[2] += fmul(r.w, r.z);
        c[3] += fmul(r.w, v.x); c[4] += fmul(r.w, v.y); c[5] += fmul(r.w, v.z);
        mg = fmaxf(mg, fabsf(A.fShift * v.x) + fabsf(A.fCosmo * r.x));
        mg = fmaxf(mg, fabsf(A.fShift * v.y) + fabsf(A.fCosmo * r.y));
        mg = fmaxf(mg, fabsf(A.fShift * v.z) + fabsf(A.fCosmo * r.z));
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        m += __shfl_xor_sync(SKID_FULL, m, o);
        for (int d = 0; d < 6; ++d) c[d] += __shfl_xor_sync(SKID_FULL, c[d], o);
    }
    mg = __uint_as_float(__reduce_max_sync(SKID_FULL, __float_as_uint(mg)));
    if (lane == 0) {
        S.part[w][0] = m;
        for (int d = 0; d < 6; ++d) S.part[w][1 + d] = c[d];
        S.ext[w][0] = mg;
    }
    __syncthreads();
    if (tid == 0) {
        double t[7] = {0, 0, 0, 0, 0, 0, 0};
        float tm = 0.0f;
        for (int k = 0; k < BS / 32; ++k) {
            for (int d = 0; d < 7; ++d) t[d] += S.part[k][d];
            tm = fmaxf(tm, S.ext[k][0]);
        }
        for (int d = 0; d < 7; ++d) C.psum[d] = t[d];
        C.pmg = tm;
    }
    cl.sync();
    if (tid == 0) {
        // every block combines the partials in rank order: the same values
        double t[7] = {0, 0, 0, 0, 0, 0, 0};
        float tm = 0.0f;
        for (int b = 0; b < CS; ++b) {
            const ClusterShared *rc = cl.map_shared_rank(&C, b);
            for (int d = 0; d < 7; ++d) t[d] += rc->psum[d];
            tm = fmaxf(tm, rc->pmg);
        }
        S.d_mass = t[0];
        for (int d = 0; d < 6; ++d) {
            S.d_cm[d] = t[1 + d] / t[0];
            S.s_cm[d] = (float)S.d_cm[d];
        }
        for (int d = 0; d < 3; ++d)
            S.s_w[d] = (float)((double)A.fShift * S.d_cm[3 + d] + (double)A.fCosmo * S.d_cm[d]);
        S.s_mg = tm * 1.0000002f;
        S.s_mW = centre_mag(A, S.d_cm);
        S.s_n = n0;
        S.s_have = 0;
        S.s_go = 1;
    }
    cl.sync();   // every block has read the sums before any overwrites them
    int nrem = 0;
    const double opz_d = 1.0 + (double)A.z, inv_d = 1.0 / (double)A.scale;
    const float epot = A.inv_scale * A.opz;
    for (;;) {
        const int n = S.s_n;
        const bool sub = S.s_have != 0 && A.subpot;
        const float4 rs = S.s_r;
        const float es = S.s_eps;
        double dcm[6];
        for (int d = 0; d < 6; ++d) dcm[d] = S.d_cm[d];
        const float wx = S.s_w[0], wy = S.s_w[1], wz = S.s_w[2];
        const float gms = fmul(A.G, rs.w) * A.scale;
        ArgRed mx{-FLT_MAX, 0x7fffffff}, mn{FLT_MAX, 0x7fffffff};
        ArgRed mx2 = mx, mn2 = mn;
        float ddmx = 0.0f, pemx = 0.0f;
        const int e = min(hi, n);
        for (int i = lo + tid; i < e; i += BS) {
            const float4 r = s_r[i - lo], wv = s_w[i - lo];
            long long p = s_p[i - lo];
            if (sub) {
                // kdSubPot (grav.c:44-59): the term the potentials added
                const float d2 = d2of(fsub(rs.x, r.x), fsub(rs.y, r.y), fsub(rs.z, r.z));
                p -= fx(fmul(gms, pair_dir(d2, fadd(es, wv.w), A.plummer)), 1.0f);
                s_p[i - lo] = p;
            }
            const float dx = wv.x - wx, dy = wv.y - wy, dz = wv.z - wz;
            const float dd = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx));
            const float pe = ll2f_fast(p) * epot;
            const float E = 0.5f * dd - pe;
            keep_top2(mx, mx2, E, i);
            keep_bot2(mn, mn2, E, i);
            ddmx = fmaxf(ddmx, dd);
            pemx = fmaxf(pemx, fabsf(pe));
        }
        // 1. the FP32 extremes and bound terms over the whole group
        {
            float a0 = mx.v, a1 = mn.v, a2 = ddmx, a3 = pemx;
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                a0 = fmaxf(a0, __shfl_xor_sync(SKID_FULL, a0, o));
                a1 = fminf(a1, __shfl_xor_sync(SKID_FULL, a1, o));
                a2 = fmaxf(a2, __shfl_xor_sync(SKID_FULL, a2, o));
                a3 = fmaxf(a3, __shfl_xor_sync(SKID_FULL, a3, o));
            }
            if (lane == 0) {
                S.ext[w][0] = a0;
                S.ext[w][1] = a1;
                S.ext[w][2] = a2;
                S.ext[w][3] = a3;
            }
            __syncthreads();
            if (tid == 0) {
                float b0 = -FLT_MAX, b1 = FLT_MAX, b2 = 0.0f, b3 = 0.0f;
                for (int k = 0; k < BS / 32; ++k) {
                    b0 = fmaxf(b0, S.ext[k][0]);
                    b1 = fminf(b1, S.ext[k][1]);
                    b2 = fmaxf(b2, S.ext[k][2]);
                    b3 = fmaxf(b3, S.ext[k][3]);
                }
                C.part[0] = b0;
                C.part[1] = b1;
                C.part[2] = b2;
                C.part[3] = b3;
            }
        }
        cl.sync();
        if (tid < CS) {
            // thread b fetches block b's partials from its shared memory
            const ClusterShared *rc = cl.map_shared_rank(&C, tid);
            for (int d = 0; d < 4; ++d) S.gpart[tid][d] = rc->part[d];
        }
        __syncthreads();
        float gmax = -FLT_MAX, gmin = FLT_MAX, gdd = 0.0f, gpe = 0.0f;
        for (int b = 0; b < CS; ++b) {
            gmax = fmaxf(gmax, S.gpart[b][0]);
            gmin = fminf(gmin, S.gpart[b][1]);
            gdd = fmaxf(gdd, S.gpart[b][2]);
            gpe = fmaxf(gpe, S.gpart[b][3]);
        }
        // the staged path's bound (block_group, groups above 1024 members)
        const float Cm = S.s_mg + S.s_mW;
        const float bound =
            1.9073486e-06f * (Cm * (1.7320509f * sqrtf(gdd) + 3.0f * Cm) + 1.5f * gdd + 2.0f * gpe) +
            1e-30f;
        const float hiE = gmax - 2.0f * bound, loE = gmin + 2.0f * bound;
        const ArgRed t1 = mx, b1 = mn;
        mx = ArgRed{-FLT_MAX, 0x7fffffff};
        mn = ArgRed{FLT_MAX, 0x7fffffff};
        if (t1.i < e && t1.v >= hiE && mx2.v < hiE) {
            mx.v = exact_energy(A, s_r[t1.i - lo], qv[t1.i], s_p[t1.i - lo], dcm, inv_d, opz_d);
            mx.i = t1.i;
        }
        if (b1.i < e && b1.v <= loE && mn2.v > loE) {
            mn.v = exact_energy(A, s_r[b1.i - lo], qv[b1.i], s_p[b1.i - lo], dcm, inv_d, opz_d);
            mn.i = b1.i;
        }
        const bool scan_hi = mx2.v >= hiE, scan_lo = mn2.v <= loE;
        if (scan_hi || scan_lo) {
            for (int i = lo + tid; i < e; i += BS) {
                const float4 wv = s_w[i - lo];
                const long long p = s_p[i - lo];
                const float dx = wv.x - wx, dy = wv.y - wy, dz = wv.z - wz;
                const float E =
                    0.5f * __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)) - ll2f_fast(p) * epot;
                const bool ch = scan_hi && E >= hiE, clo = scan_lo && E <= loE;
                if (ch || clo) {
                    const float X = exact_energy(A, s_r[i - lo], qv[i], p, dcm, inv_d, opz_d);
                    if (ch && X > mx.v) { mx.v = X; mx.i = i; }
                    if (clo && X < mn.v) { mn.v = X; mn.i = i; }
                }
            }
        }
        // 2. the exact arg-max and arg-min over the whole group
        mx = warp_argmax(mx);
        mn = warp_argmin(mn);
        if (lane == 0) { S.smax[w] = mx; S.smin[w] = mn; }
        __syncthreads();
        if (tid == 0) {
            ArgRed a = S.smax[0], b = S.smin[0];
            for (int k = 1; k < BS / 32; ++k) {
                const ArgRed x = S.smax[k], y = S.smin[k];
                if (x.v > a.v || (x.v == a.v && x.i < a.i)) a = x;
                if (y.v < b.v || (y.v == b.v && y.i < b.i)) b = y;
            }
            C.pmax = a;
            C.pmin = b;
        }
        cl.sync();
        if (tid < CS) {
            const ClusterShared *rc = cl.map_shared_rank(&C, tid);
            S.gmx[tid] = rc->pmax;
            S.gmn[tid] = rc->pmin;
        }
        __syncthreads();
        if (tid == 0) {
            ArgRed a = S.gmx[0], b = S.gmn[0];
            for (int k = 1; k < CS; ++k) {
                const ArgRed x = S.gmx[k], y = S.gmn[k];
                if (x.v > a.v || (x.v == a.v && x.i < a.i)) a = x;
                if (y.v < b.v || (y.v == b.v && y.i < b.i)) b = y;
            }
            // kd.c:1389-1409: fTotBig starts at -1, fTotMin at 1
            S.s_imin = b.v < 1.0f ? b.i : 0;
            if (!(a.v >= 0.0f) || A.nounbind || n == 0) {
                S.s_go = 0;
            } else {
                const int ib = a.i;
                const int ob = ib / Q;
                const float4 r = cl.map_shared_rank(s_r, ob)[ib - ob * Q];
                const float4 wv = cl.map_shared_rank(s_w, ob)[ib - ob * Q];
                const float4 v = qv[ib];
                if (rank == 0) A.grp[qid[ib]] = 0;
                ++nrem;
                const int nn = n - 1;
                if (nn == 0) {
                    S.d_mass = 0.0;
                    for (int d = 3; d < 6; ++d) S.d_cm[d] = 0.0;
                    S.s_go = 0;
                } else {
                    double mm = S.d_mass;
                    for (int d = 0; d < 6; ++d) dcm[d] = S.d_cm[d];
                    rcm_update(mm, dcm, r, v);
                    S.d_mass = mm;
                    for (int d = 0; d < 6; ++d) {
                        S.d_cm[d] = dcm[d];
                        S.s_cm[d] = (float)dcm[d];
                    }
                    for (int d = 0; d < 3; ++d)
                        S.s_w[d] = (float)((double)A.fShift * dcm[3 + d] + (double)A.fCosmo * dcm[d]);
                    S.s_mW = centre_mag(A, dcm);
                    S.s_r = r;
                    S.s_eps = wv.w;
                    S.s_have = 1;
                }
                S.s_n = nn;
                S.s_item = ib;
            }
        }
        // 3. every block has read the removed member (and rank 0 its id)
        // before its slot is overwritten
        cl.sync();
        if (tid == 0 && S.s_go) {
            const int ib = S.s_item;
            const int nn = S.s_n;
            if (ib / Q == rank && ib != nn) {
                const int on = nn / Q;
                s_r[ib - lo] = cl.map_shared_rank(s_r, on)[nn - on * Q];
                s_w[ib - lo] = cl.map_shared_rank(s_w, on)[nn - on * Q];
                s_p[ib - lo] = cl.map_shared_rank(s_p, on)[nn - on * Q];
                const float4 rl = qr[nn], vl = qv[nn], rb = qr[ib], vb = qv[ib];
                const int il = qid[nn], ir = qid[ib];
                qr[ib] = rl; qv[ib] = vl; qid[ib] = il;
                qr[nn] = rb; qv[nn] = vb; qid[nn] = ir;
            }
        }
        __syncthreads();
        if (!S.s_go) break;
    }
    if (rank == 0 && tid == 0) {
        double dcm[6];
        for (int d = 0; d < 6; ++d) dcm[d] = S.d_cm[d];
        write_record(A, g, S.s_n, S.d_mass, dcm, qr[S.s_imin], nrem);
    }
    cl.sync();   // no block leaves while another may still read its shared memory
}

// Persistent removal of the groups above tw members, a block each (the
// largest on clusters of CS blocks first, when launched so), largest first.
// With A.single > 0 one block processes just that group.  The kernel of the
// other groups may start once every block here has (remove_launch).
template <int BS, int CS>
__global__ void __launch_bounds__(BS) remove_kernel(const __grid_constant__ RemoveArgs A)
{
    __shared__ BlockShared<BS> S;
    __shared__ int s_item;
    extern __shared__ float4 dyn[];
    asm volatile("griddepcontrol.launch_dependents;");
    if (A.single > 0) {
        block_group<BS>(A, A.single, S, dyn);
        return;
    }
    int first = 0;
    if constexpr (CS > 1) {
        // launched as clusters of CS blocks: the largest groups first, one
        // cluster each, then every block goes on alone
        __shared__ ClusterShared C;
        cg::cluster_group cl = cg::this_cluster();
        const int nclu = *A.d_ccnt;
        for (;;) {
            if (cl.block_rank() == 0 && threadIdx.x == 0) C.item = atomicAdd(A.d_cqueue, 1);
            cl.sync();
            const int item = cl.map_shared_rank(&C, 0)->item;
            cl.sync();
            if (item >= nclu) break;
            cluster_group<BS, CS>(A, (int)A.order[item], S, C, dyn, cl);
        }
        first = nclu;
    }
    const int nbig = A.d_cnt[1];
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(A.d_queue, 1);
        __syncthreads();
        const int item = first + s_item;
        __syncthreads();
        if (item >= nbig) break;
        block_group<BS>(A, (int)A.order[item], S, dyn);
    }
}

// Persistent removal of the groups of up to tw members, a warp each.
//
// Latency bounds it (one chain of passes a group), so warps in flight decide,
// and it is a kernel of its own for that: 90 registers, 20 warps an SM, where
// the block form takes 184 (128 and spills at 512 threads).  In one kernel
// with the block form 20,000 groups of 100 members took 2.13 ms, 5,000 of 300
// 1.28 and 3,000 of 1,000 5.32; on their own 1.39, 0.53 and 2.41.
constexpr int RW_THREADS = 128;

__global__ void __launch_bounds__(RW_THREADS) remove_warps_kernel(const __grid_constant__ RemoveArgs A)
{
    const int lane = threadIdx.x & 31;
    const int nvalid = A.d_cnt[0], nbig = A.d_cnt[1];
    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(A.d_wqueue, 1);
        item = nbig + __shfl_sync(SKID_FULL, item, 0);
        if (item >= nvalid) break;
        warp_group(A, (int)A.order[item]);
    }
    // the blocks' kernel, if it is still running, ends before this one does (one
    // block sees to it: blocks that wait keep their SMs from other streams)
    if (blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Raise a removal kernel's shared-memory limit to all it can have, once per
// device (the attribute is only an upper bound; contexts on other threads
// launch with other sizes).
template <int BS, int CS>
cudaError_t remove_smem_limit(int *dyn_max)
{
    static std::mutex mu;
    static int most[SKID_MAX_DEVICES] = {};
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e) return e;
    if (dev < 0 || dev >= SKID_MAX_DEVICES) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(mu);
    if (!most[dev]) {
        cudaFuncAttributes fa;
        if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) ||
            (e = cudaFuncGetAttributes(&fa, remove_kernel<BS, CS>)))
            return e;
        const int d = optin - (int)fa.sharedSizeBytes;
        if ((e = cudaFuncSetAttribute(remove_kernel<BS, CS>, cudaFuncAttributeMaxDynamicSharedMemorySize, d)))
            return e;
        most[dev] = d;
    }
    *dyn_max = most[dev];
    return cudaSuccess;
}

// Shared memory a block of a plain removal launch takes: 32 B for each member
// of the largest group, up to LCAP_KB.  One block an SM for every other group
// then, and still the fastest: at 220 / 110 / 48 KB a group of 10,000 members
// over 2,000 of 1,300 takes 2.26 / 2.81 / 3.18 ms, over 300 of 3,000 2.09 /
// 2.78 / 3.13.
#ifndef SKID_LCAP_KB
#define SKID_LCAP_KB 220
#endif
constexpr int LCAP_BYTES = SKID_LCAP_KB * 1024;
constexpr int LMEMBER = 2 * (int)sizeof(float4);

template <int BS>
cudaError_t launch_remove(RemoveArgs A, int nlargest, int single, cudaStream_t st)
{
    int most = 0, perSM = 0;
    cudaError_t e = remove_smem_limit<BS, 1>(&most);
    if (e) return e;
    if (most > LCAP_BYTES) most = LCAP_BYTES;
    constexpr int row = 2 * BlockGroup<BS>::BC;
    const long long want = ((long long)nlargest + row - 1) / row * row * LMEMBER;
    A.lcap = (int)(want < most ? want : most) / LMEMBER;
    const size_t smem = (size_t)A.lcap * LMEMBER;
    int blocks = 1;
    if (!single) {
        if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, remove_kernel<BS, 1>, BS, smem)))
            return e;
        blocks = num_sms() * (perSM > 0 ? perSM : 1);
    }
    remove_kernel<BS, 1><<<blocks, BS, smem, st>>>(A); note_launch();
    return cudaGetLastError();
}

// Cluster launch: as many clusters of CS blocks as fit at once, each block
// with A.qcap members' worth of dynamic shared memory.
template <int BS, int CS>
cudaError_t launch_remove_clusters(RemoveArgs A, cudaStream_t st)
{
    const size_t smem = (size_t)A.qcap * (2 * sizeof(float4) + sizeof(long long));
    int most = 0;
    cudaError_t e = remove_smem_limit<BS, CS>(&most);
    if (e) return e;
    if (smem > (size_t)most) return cudaErrorInvalidValue;
    A.lcap = (int)smem / LMEMBER;   // the same memory, once the blocks go on alone
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(BS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(CS, 1, 1);
    int nclusters = 0;
    if ((e = cudaOccupancyMaxActiveClusters(&nclusters, remove_kernel<BS, CS>, &cfg))) return e;
    if (nclusters < 1) return cudaErrorInvalidConfiguration;
    cfg.gridDim = dim3(CS * nclusters, 1, 1);
    e = cudaLaunchKernelEx(&cfg, remove_kernel<BS, CS>, A);
    note_launch();
    return e ? e : cudaGetLastError();
}

// cs: 1 (no clusters), 4 or 8; nlargest: the members of the largest group a
// block will take; single: one block for A.single alone
cudaError_t remove_blocks(const RemoveArgs &A, int bs, int cs, int nlargest, bool single, cudaStream_t st)
{
    if (cs == 4 || cs == 8) {
        switch (bs) {
        case 512: return cs == 8 ? launch_remove_clusters<512, 8>(A, st) : launch_remove_clusters<512, 4>(A, st);
        case 1024: return cs == 8 ? launch_remove_clusters<1024, 8>(A, st) : launch_remove_clusters<1024, 4>(A, st);
        default: return cs == 8 ? launch_remove_clusters<256, 8>(A, st) : launch_remove_clusters<256, 4>(A, st);
        }
    }
    switch (bs) {
    case 128: return launch_remove<128>(A, nlargest, single, st);
    case 512: return launch_remove<512>(A, nlargest, single, st);
    case 1024: return launch_remove<1024>(A, nlargest, single, st);
    default: return launch_remove<256>(A, nlargest, single, st);
    }
}

// All nvalid groups: those above tw members by blocks (none where the largest
// has nlargest <= tw), the others by warps, on the SMs that the blocks leave:
// the second launch is a dependent one that starts when every block of the
// first has started (its inputs are older than both), so that a group that
// takes long does not hold up the small ones.
cudaError_t remove_launch(const RemoveArgs &A, int tw, int bs, int cs, int nvalid, int nlargest, cudaStream_t st)
{
    cudaError_t e;
    const bool blocks = nlargest > tw;
    if (blocks && (e = remove_blocks(A, bs, cs, nlargest, false, st))) return e;
    int perSM = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, remove_warps_kernel, RW_THREADS, 0))) return e;
    constexpr int W = RW_THREADS / 32;
    const int need = (nvalid + W - 1) / W, most = num_sms() * (perSM > 0 ? perSM : 1);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.blockDim = dim3(RW_THREADS, 1, 1);
    cfg.gridDim = dim3(need < most ? need : most, 1, 1);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = blocks ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, remove_warps_kernel, A); note_launch();
    return e ? e : cudaGetLastError();
}

}  // namespace

// Candidate removal schedules (tw, BS) for the autotuner.
static const int kTW[] = {0, 32, 128, 256, 512, 1024};
static const int kBS[] = {256, 512, 1024};

cudaError_t unbind_run(GroupState &G, const int *gof, int nslots, const float4 *pos4,
                       const float4 *vel4, Tree &ut, const UnbindParams &P, int *grp,
                       int *d_unbound, SortScratch &ss, UnbindScratch &U, cudaStream_t st)
{
    cudaError_t e;
    int ng = G.nGroup;
    if ((e = dalloc(U.qr, nslots)) || (e = dalloc(U.qv, nslots)) || (e = dalloc(U.qw, nslots)) || (e = dalloc(U.qa, nslots)) ||
        (e = dalloc(U.qid, nslots)) ||
        (e = dalloc(U.pot, nslots)) || (e = dalloc(U.scnt, ng)) || (e = dalloc(U.soff, ng + 1)) ||
        (e = dalloc(U.nt, ng)) || (e = dalloc(U.toff, ng + 1)) || (e = dalloc(U.cnt, 16)) ||
        (e = dalloc(U.order, ng)))
        return e;
    float3 hP = make_float3((float)(0.5 * (double)P.period.x), (float)(0.5 * (double)P.period.y),
                            (float)(0.5 * (double)P.period.z));
    auto prep = [&]() -> cudaError_t {
        prep_members<<<grid_for(nslots), 256, 0, st>>>(G.members.p, gof, nslots, pos4, vel4, G.rec.p,
                                                       hP, U.qr.p, U.qv.p); note_launch();
        return cudaMemcpyAsync(U.qid.p, G.members.p, nslots * sizeof(int), cudaMemcpyDeviceToDevice, st);
    };
    if ((e = prep())) return e;
    // scoop lists
    float fBall2 = P.fScoop * P.fScoop;
    float3 hL = make_float3(0.5f * P.period.x, 0.5f * P.period.y, 0.5f * P.period.z);
    int subShift = 0;
    while (subShift < 5 && (2 << subShift) <= ut.leafBase) ++subShift;
    const int scoopBlocks = grid_for(ng, SCOOP_THREADS / 32);
    scoop_kernel<<<scoopBlocks, SCOOP_THREADS, 0, st>>>(ut.view(), U.usoft.p, G.rec.p, G.count.p, ng, P.nmax,
                                                        fBall2, P.period, hL, P.per, subShift, 0, U.scnt.p,
                                                        nullptr, nullptr, nullptr); note_launch();
    if ((e = scan_exclusive(U.scnt.p, U.soff.p, ng, U.cnt.p, ss, st))) return e;
    int nscoop = 0;
    if ((e = cudaMemcpyAsync(&nscoop, U.cnt.p, sizeof(int), cudaMemcpyDeviceToHost, st))) return e;
    if ((e = cudaStreamSynchronize(st))) return e;
    if ((e = dalloc(U.slist, nscoop > 0 ? nscoop : 1)) || (e = dalloc(U.ssoft, nscoop > 0 ? nscoop : 1)))
        return e;
    if (nscoop > 0)
        scoop_kernel<<<scoopBlocks, SCOOP_THREADS, 0, st>>>(ut.view(), U.usoft.p, G.rec.p, G.count.p, ng, P.nmax,
                                                            fBall2, P.period, hL, P.per, subShift, 1, U.scnt.p,
                                                            U.soff.p, U.slist.p, U.ssoft.p); note_launch();
    // groups by descending size
    if ((e = dalloc(ss.k0, ng)) || (e = dalloc(ss.v0, ng)) || (e = dalloc(ss.k1, ng)) ||
        (e = dalloc(ss.v1, ng)))
        return e;
    sched_keys<<<grid_for(ng), 256, 0, st>>>(G.count.p, ng, P.nmax, ss.k0.p, ss.v0.p); note_launch();
    if ((e = radix_sort(ss, ng, 32, st))) return e;
    if ((e = cudaMemcpyAsync(U.order.p, ss.v0.p, ng * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st)))
        return e;
    if ((e = cudaMemsetAsync(U.cnt.p + 2, 0, 2 * sizeof(int), st))) return e;
    sched_counts<<<grid_for(ng), 256, 0, st>>>(G.count.p, ng, P.nmax, 1 << 30, U.cnt.p + 2); note_launch();
    // potential items, largest groups first
    pot_nitems<<<grid_for(ng), 256, 0, st>>>(U.order.p, U.cnt.p + 2, G.count.p, ng, U.nt.p); note_launch();
    if ((e = scan_exclusive(U.nt.p, U.toff.p, ng, U.cnt.p + 1, ss, st))) return e;
    // clustered groups: the largest ones above clu_min members, at most as
    // many as keep half the SMs busy with clusters of 4 blocks; and the
    // largest group's size, which sizes the blocks' shared-memory slices
    const int clu_min = P.clu_min > P.tw && P.clu_min > 1024 ? P.clu_min : 0;
    const int clu_kmax = num_sms() / 8 > 1 ? num_sms() / 8 : 1;
    if ((e = cudaMemsetAsync(U.cnt.p + 8, 0, 4 * sizeof(int), st))) return e;
    cluster_groups<<<1, 32, 0, st>>>(U.order.p, U.cnt.p + 2, G.count.p, clu_min,
                                     clu_min > 0 ? clu_kmax : 0, U.cnt.p + 9); note_launch();
    int hc[11] = {0};
    if ((e = cudaMemcpyAsync(hc, U.cnt.p + 1, 11 * sizeof(int), cudaMemcpyDeviceToHost, st))) return e;
    if ((e = cudaStreamSynchronize(st))) return e;
    const int nitems = hc[0], nvalid = hc[1], nclu = hc[8], nlargest = hc[10];
    // cluster size: 4 blocks while a quarter of the largest group fits in
    // about 200 KB of shared memory (40 B per member), else 8, else none
    int cs = 1, qcap = 0;
    if (clu_min > 0 && nclu > 0) {
        const int per = (int)(2 * sizeof(float4) + sizeof(long long));
        const int q4 = (nlargest + 3) / 4, q8 = (nlargest + 7) / 8;
        if ((size_t)q4 * per <= 200u * 1024u) { cs = 4; qcap = q4; }
        else if ((size_t)q8 * per <= 200u * 1024u) { cs = 8; qcap = q8; }
    }
    if ((e = dalloc(U.items, nitems > 0 ? nitems : 1))) return e;
    if (nitems > 0)
        pot_fill<<<grid_for(nvalid, 8), 256, 0, st>>>(U.order.p, U.cnt.p + 2, G.count.p, U.toff.p,
                                                   U.items.p); note_launch();

    RemoveArgs A;
    A.gstart = G.start.p;
    A.gcount = G.count.p;
    A.ng = ng;
    A.nmax = P.nmax;
    A.qr = U.qr.p;
    A.qv = U.qv.p;
    A.qa = U.qa.p;
    A.qw = U.qw.p;
    A.lcap = 0;
    A.qid = U.qid.p;
    A.pot = U.pot.p;
    A.rec = G.rec.p;
    A.grp = grp;
    A.d_unbound = d_unbound;
    A.G = P.G;
    A.fShift = P.a;
    A.fCosmo = P.aH;
    A.opz = P.opz;
    A.z = P.z;
    A.scale = P.scale;
    A.inv_scale = 1.0f / P.scale;
    A.hP = hP;
    A.plummer = P.plummer;
    A.subpot = P.subpot;
    A.nounbind = P.nounbind;
    A.order = U.order.p;
    A.d_cnt = U.cnt.p + 4;
    A.d_queue = U.cnt.p + 6;
    A.d_wqueue = U.cnt.p + 7;
    A.d_ccnt = U.cnt.p + 9;
    A.d_cqueue = U.cnt.p + 10;
    A.qcap = qcap;
    A.single = 0;

    const int potBlocks = nitems < num_sms() * 32 ? (nitems > 0 ? nitems : 1) : num_sms() * 32;
    auto potentials = [&]() -> cudaError_t {
        cudaError_t e2 = cudaMemsetAsync(U.pot.p, 0, nslots * sizeof(long long), st);
        if (e2 || nitems <= 0) return e2;
        pot_sym_kernel<<<potBlocks, POT_THREADS, 0, st>>>(U.items.p, U.cnt.p + 1, -1, G.start.p, G.count.p,
                                                       U.qr.p, U.qv.p, U.soff.p, U.scnt.p, U.slist.p,
                                                       U.ssoft.p, P.G, P.plummer, P.scale, 0.0f, U.pot.p); note_launch();
        return cudaGetLastError();
    };
    auto removal = [&](int tw, int bs, int ucs) -> cudaError_t {
        cudaError_t e2;
        if ((e2 = cudaMemsetAsync(U.cnt.p + 4, 0, 4 * sizeof(int), st))) return e2;
        if ((e2 = cudaMemsetAsync(U.cnt.p + 10, 0, sizeof(int), st))) return e2;
        sched_counts<<<grid_for(ng), 256, 0, st>>>(G.count.p, ng, P.nmax, tw, U.cnt.p + 4); note_launch();
        if ((e2 = cudaMemsetAsync(d_unbound, 0, sizeof(int), st))) return e2;
        if (nvalid <= 0) return cudaSuccess;
        return remove_launch(A, tw, bs, bs >= 256 ? ucs : 1, nvalid, nlargest, st);
    };

    if (P.per_group) {
        // the reference's serial loop on the GPU: two launches per group
        std::vector<uint32_t> order(ng);
        std::vector<int> ioff(ng + 1);
        if ((e = cudaMemcpyAsync(order.data(), U.order.p, ng * sizeof(uint32_t), cudaMemcpyDeviceToHost, st)) ||
            (e = cudaMemcpyAsync(ioff.data(), U.toff.p, ng * sizeof(int), cudaMemcpyDeviceToHost, st)) ||
            (e = cudaStreamSynchronize(st)))
            return e;
        ioff[nvalid] = nitems;
        if ((e = cudaMemsetAsync(U.pot.p, 0, nslots * sizeof(long long), st))) return e;
        if ((e = cudaMemsetAsync(d_unbound, 0, sizeof(int), st))) return e;
        for (int k = 0; k < nvalid; ++k) {
            int cnt = ioff[k + 1] - ioff[k];
            pot_sym_kernel<<<cnt < num_sms() * 32 ? cnt : num_sms() * 32, POT_THREADS, 0, st>>>(
                U.items.p + ioff[k], nullptr, cnt, G.start.p, G.count.p, U.qr.p, U.qv.p, U.soff.p,
                U.scnt.p, U.slist.p, U.ssoft.p, P.G, P.plummer, P.scale, 0.0f, U.pot.p); note_launch();
            RemoveArgs A1 = A;
            A1.single = (int)order[k];
            if ((e = remove_blocks(A1, 256, 1, nlargest, true, st))) return e;
        }
        return cudaGetLastError();
    }

    cudaEvent_t t0 = nullptr, t1 = nullptr, t2 = nullptr;
    cudaEventCreate(&t0);
    cudaEventCreate(&t1);
    cudaEventCreate(&t2);
    cudaEventRecord(t0, st);
    if ((e = potentials())) return e;
    cudaEventRecord(t1, st);
    int tw = P.tw, bs = P.bs;
    if ((tw < 0 || bs < 0) && U.tuned_bs > 0) {
        if (tw < 0) tw = U.tuned_tw;
        if (bs < 0) bs = U.tuned_bs;
    }
    if (tw < 0 || bs < 0) {
        // autotune: time every candidate removal schedule on these groups,
        // restoring the inputs between runs, then keep the fastest
        if ((e = dalloc(U.pot_save, nslots)) || (e = dalloc(U.rec_save, ng)) ||
            (e = dalloc(U.grp_save, P.n > 0 ? P.n : 1)))
            return e;
        if ((e = cudaMemcpyAsync(U.pot_save.p, U.pot.p, nslots * sizeof(long long), cudaMemcpyDeviceToDevice, st)) ||
            (e = cudaMemcpyAsync(U.rec_save.p, G.rec.p, ng * sizeof(skid_group), cudaMemcpyDeviceToDevice, st)) ||
            (e = cudaMemcpyAsync(U.grp_save.p, grp, P.n * sizeof(int), cudaMemcpyDeviceToDevice, st)))
            return e;
        cudaEvent_t e0, e1;
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        float best = FLT_MAX;
        int btw = 32, bbs = 256;
        for (int a : kTW) {
            if (P.tw >= 0 && a != P.tw) continue;
            for (int b : kBS) {
                if (P.bs >= 0 && b != P.bs) continue;
                if ((e = cudaMemcpyAsync(U.pot.p, U.pot_save.p, nslots * sizeof(long long), cudaMemcpyDeviceToDevice, st)) ||
                    (e = cudaMemcpyAsync(G.rec.p, U.rec_save.p, ng * sizeof(skid_group), cudaMemcpyDeviceToDevice, st)) ||
                    (e = cudaMemcpyAsync(grp, U.grp_save.p, P.n * sizeof(int), cudaMemcpyDeviceToDevice, st)) ||
                    (e = prep()))
                    break;
                cudaEventRecord(e0, st);
                if ((e = removal(a, b, 1))) break;
                cudaEventRecord(e1, st);
                if ((e = cudaEventSynchronize(e1))) break;
                float ms = 0.0f;
                cudaEventElapsedTime(&ms, e0, e1);
                U.tune_ms[U.ntune < 32 ? U.ntune : 31] = ms;
                ++U.ntune;
                U.ntune_now = 1;
                if (ms < best) { best = ms; btw = a; bbs = b; }
            }
            if (e) break;
        }
        // then the best schedule with the largest groups on thread-block
        // clusters, kept only if it is faster
        int bcs = 1;
        if (!e && cs > 1 && bbs >= 256) {
            if (!(e = cudaMemcpyAsync(U.pot.p, U.pot_save.p, nslots * sizeof(long long), cudaMemcpyDeviceToDevice, st)) &&
                !(e = cudaMemcpyAsync(G.rec.p, U.rec_save.p, ng * sizeof(skid_group), cudaMemcpyDeviceToDevice, st)) &&
                !(e = cudaMemcpyAsync(grp, U.grp_save.p, P.n * sizeof(int), cudaMemcpyDeviceToDevice, st)) &&
                !(e = prep())) {
                cudaEventRecord(e0, st);
                e = removal(btw, bbs, cs);
                cudaEventRecord(e1, st);
                if (!e) e = cudaEventSynchronize(e1);
                float ms = 0.0f;
                if (!e) cudaEventElapsedTime(&ms, e0, e1);
                U.tune_ms[U.ntune < 32 ? U.ntune : 31] = ms;
                ++U.ntune;
                if (!e && ms < best) bcs = cs;
            }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        if (e) return e;
        U.tuned_tw = btw;
        U.tuned_bs = bbs;
        U.tuned_cs = bcs > 1 ? 1 : 0;
        tw = btw;
        bs = bbs;
        if ((e = cudaMemcpyAsync(U.pot.p, U.pot_save.p, nslots * sizeof(long long), cudaMemcpyDeviceToDevice, st)) ||
            (e = cudaMemcpyAsync(G.rec.p, U.rec_save.p, ng * sizeof(skid_group), cudaMemcpyDeviceToDevice, st)) ||
            (e = cudaMemcpyAsync(grp, U.grp_save.p, P.n * sizeof(int), cudaMemcpyDeviceToDevice, st)) ||
            (e = prep()))
            return e;
    }
    // clusters: as the tuner chose for a tuned schedule; with a fixed one,
    // whenever there are groups for them and the caller set the threshold
    const bool tuned_sched = P.tw < 0 || P.bs < 0;
    const int ucs = cs > 1 && (tuned_sched ? U.tuned_cs == 1 : !P.clu_auto) ? cs : 1;
    U.used_tw = tw;
    U.used_bs = bs;
    U.used_cs = ucs;
    U.used_nclu = ucs > 1 ? nclu : 0;
    if (U.ntune) cudaEventRecord(t1, st);   // tuning ran in between: time the final removal only
    e = removal(tw, bs, ucs);
    cudaEventRecord(t2, st);
    if (!e) e = cudaEventSynchronize(t2);
    float a = 0.0f, b = 0.0f;
    if (!e && !U.ntune_now) cudaEventElapsedTime(&a, t0, t1);
    if (!e) cudaEventElapsedTime(&b, t1, t2);
    if (!U.ntune_now) U.pot_ms = a;
    U.remove_ms = b;
    U.ntune_now = 0;
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    cudaEventDestroy(t2);
    return e;
}

}  // namespace skid

// ---- numerics check of the pair factor ----

namespace {

__global__ void pair_factor_kernel(const float *__restrict__ d2, const float *__restrict__ twoh, int n,
                                   int plummer, int mode, float *__restrict__ out)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float v = __int_as_float(0x7fc00000);   // NaN: the float-float form declined
        if (mode == SKID_PAIR_FP64) v = skid::ref_dir_fp64(d2[i], twoh[i], plummer);
        else if (mode == SKID_PAIR_SPLINE_FF) skid::ref_spline_ff(d2[i], twoh[i], v);
        else v = skid::pair_dir(d2[i], twoh[i], plummer);
        out[i] = v;
    }
}

}  // namespace

extern "C" int skid_pair_factor(int n, const float *d2, const float *twoh, int plummer, int mode,
                                float *out)
{
    if (n < 0 || (n > 0 && (!d2 || !twoh || !out))) return SKID_EINVAL;
    if (mode != SKID_PAIR_USED && mode != SKID_PAIR_FP64 && mode != SKID_PAIR_SPLINE_FF)
        return SKID_EINVAL;
    if (n == 0) return 0;
    float *dv = nullptr;
    const size_t bytes = (size_t)n * sizeof(float);
    {
        std::lock_guard<std::recursive_mutex> lk(skid::device_mutex());
        if (cudaMalloc((void **)&dv, 3 * bytes)) {
            cudaGetLastError();
            return SKID_ENOMEM;
        }
    }
    cudaError_t e = cudaMemcpy(dv, d2, bytes, cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(dv + n, twoh, bytes, cudaMemcpyHostToDevice);
    if (!e) {
        const int blocks = (int)std::min<long long>(((long long)n + 255) / 256, 65536);
        pair_factor_kernel<<<blocks, 256>>>(dv, dv + n, n, plummer, mode, dv + 2 * (size_t)n);
        skid::note_launch();
        e = cudaGetLastError();
    }
    if (!e) e = cudaMemcpy(out, dv + 2 * (size_t)n, bytes, cudaMemcpyDeviceToHost);
    {
        std::lock_guard<std::recursive_mutex> lk(skid::device_mutex());
        cudaFree(dv);
    }
    if (e) {
        cudaGetLastError();
        return SKID_ECUDA;
    }
    return 0;
}
