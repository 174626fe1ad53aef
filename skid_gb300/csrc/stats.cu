// Per-group statistics of the .stat table (kdOutStats, kd.c:1703-1839) on the
// device, after too-small removal.
//
// The reference takes each group's members relative to its density centre
// (wrapped with half periods), sorts them by radius with qsort, and walks
// them outwards keeping running float sums: total, gas and star mass, the
// largest G M(<r)/r outside twice the softening, the radius where the
// enclosed mass first exceeds half, and the velocity dispersion about vcm
// with the Hubble flow.  Here:
//   1. one thread per particle forms the key (group << 32 | radius^2 bits;
//      radius^2 >= 0, so its bits order like its value) -- ungrouped
//      particles get the largest key;
//   2. a stable radix sort of (key, iOrder) puts every group's members in
//      radius order, ties in iOrder order;
//   3. one thread per sorted slot marks where each group's run starts;
//   4. one warp (for a few members, one thread) per group walks its run
//      outwards with the reference's own float and double operations, each
//      rounded as gcc rounds it, so the running sums and the maximum /
//      half-mass decisions are the reference's (the sums are inherently
//      sequential: each depends on the float rounding of the previous one).
#include <cfloat>

#include "ctx.h"

using namespace skid;

namespace {

__device__ __forceinline__ float stat_wrap(float d, float h)
{
    // kd.c:1741-1746: if (dx > hx) dx -= 2*hx; if (dx <= -hx) dx += 2*hx
    if (d > h) d = fsub(d, fmul(2.0f, h));
    if (d <= -h) d = fadd(d, fmul(2.0f, h));
    return d;
}

__device__ __forceinline__ float3 stat_rel(float4 p, const skid_group &g, float3 h)
{
    return make_float3(stat_wrap(fsub(p.x, g.rCenter[0]), h.x),
                       stat_wrap(fsub(p.y, g.rCenter[1]), h.y),
                       stat_wrap(fsub(p.z, g.rCenter[2]), h.z));
}

__global__ void stat_keys(const float4 *__restrict__ pos4, const int *__restrict__ grp, int n,
                          const skid_group *__restrict__ rec, float3 h, uint64_t *__restrict__ keys,
                          uint32_t *__restrict__ vals)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int g = grp[i];
        uint64_t k = ~0ull;
        if (g > 0) {
            const float3 r = stat_rel(pos4[i], rec[g], h);
            // kd.c:1756-1760: radius2 = 0.0; radius2 += r_k * r_k (float)
            const float r2 = fadd(fadd(fmul(r.x, r.x), fmul(r.y, r.y)), fmul(r.z, r.z));
            k = ((uint64_t)(unsigned)g << 32) | __float_as_uint(r2);
        }
        keys[i] = k;
        vals[i] = (uint32_t)i;
    }
}

__global__ void stat_starts(const uint64_t *__restrict__ keys, int n, int *__restrict__ start)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const uint64_t k = keys[p];
        if (k == ~0ull) continue;
        const unsigned g = (unsigned)(k >> 32);
        if (p == 0 || (unsigned)(keys[p - 1] >> 32) != g) start[g] = p;
    }
}

struct StatArgs {
    const uint64_t *keys;
    const uint32_t *vals;
    const int *start;
    const skid_group *rec;
    const float4 *pos4, *vel4;
    const float *temp, *rho;
    int nGroup, nGas, nDark;
    float3 h;
    float G, fExp, fExpHub, fDensMin, fTempMax;
    skid_stat *out;
    int small;                  // groups of up to so many members take a thread
};

// The running float sums of one group are a serial chain: each add waits for
// the last one's rounding (4 cycles), so a group of n members takes at least
// 3 n dependent adds (the three dispersion terms).  Everything else can be
// done 32 members at a time.  One warp takes a group: its lanes load and
// prepare 32 members at once (the next 32 are loaded meanwhile), lanes 0-3
// then run the four chains -- total, gas and star mass, dispersion -- side by
// side from shared memory, and the maximum and half-mass rules, which depend
// on the running total only, are resolved by ballots in member order.  With
// one thread per group (every load, divide and root in the one chain) the 150k
// mixed-species snapshot took 19.5 ms, its largest group of some 14k members
// setting the time; now about 0.36 ms.
//
// Where there are ST_MANY groups an SM, those of up to ST_THREAD_MAX members
// take a thread each after all: their FP64 roots and divides (a member's
// circular velocity, five more a group) use as many issue slots for one group
// as for 32.  A warp / a thread a group, ms a call: 3,000 groups of 8 .13 / .13,
// of 30 .14 / .18; 10,000 of 8 .18 / .14, of 30 .21 / .20; 40,000 of 5 .37 /
// .20, of 16 .42 / .28, of 30 .47 / .35.
constexpr int ST_THREAD_MAX = 32, ST_MANY = 64;
constexpr int ST_WARPS = 2;
constexpr int ST_ROW = 97;   // 3 adds for each of 32 members, one word of padding

struct StatMember {
    int io;
    float r2;
    float4 p, v;
    bool gas;
};

__device__ __forceinline__ void stat_load(const StatArgs &A, int s, int n, int j, StatMember &q)
{
    q.io = 0;
    q.r2 = 0.0f;
    q.p = q.v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    q.gas = false;
    if (j >= n) return;
    q.io = (int)A.vals[s + j];
    q.r2 = __uint_as_float((unsigned)A.keys[s + j]);
    q.p = A.pos4[q.io];
    q.v = A.vel4[q.io];
    q.gas = q.io < A.nGas && A.rho[q.io] >= A.fDensMin && A.temp[q.io] <= A.fTempMax;
}

// dv = fExp*(v - vcm) + fExpHub*r (float, kd.c:1792-1796), squared.
__device__ __forceinline__ float stat_dv2(const StatArgs &A, float v, float vcm, float r)
{
    const float dv = fadd(fmul(A.fExp, fsub(v, vcm)), fmul(A.fExpHub, r));
    return fmul(dv, dv);
}

// What follows the walk (kd.c:1798-1803); r2 is the outermost member's.
__device__ __forceinline__ void stat_store(const StatArgs &A, int g, int n, float fTot, float fGas,
                                           float fStar, float fVc, float fmVc, float fRVmax, float fRh,
                                           float r2, float fVd)
{
    const float flVc = (float)__ddiv_rn((double)fmul(A.G, fTot), __dsqrt_rn((double)r2));
    if (fVc == 0.0f) {
        fVc = flVc;
        fRVmax = (float)__dsqrt_rn((double)r2);
    }
    fVd = (float)__dsqrt_rn(__ddiv_rn((double)fVd, __dmul_rn(3.0, (double)n)));
    skid_stat o;
    o.nMembers = n;
    o.fTotMass = fTot;
    o.fGasMass = fGas;
    o.fStarMass = fStar;
    o.fVcirc2Max = fVc;
    o.fVcirc2Half = fmVc;
    o.fVcirc2Outer = flVc;
    o.fRVmax = fRVmax;
    o.fRHalf = fRh;
    o.fROuter2 = r2;
    o.fVdisp = fVd;
    A.out[g] = o;
}

// A group without members.
__device__ __forceinline__ void stat_none(const StatArgs &A, int g, int n)
{
    skid_stat o = {};
    o.nMembers = n;
    A.out[g] = o;
}

// A group on one thread, member by member.
__device__ void stat_thread(const StatArgs &A, int g)
{
    const skid_group rg = A.rec[g];
    const int n = rg.nMembers, s = A.start[g];
    if (n <= 0) return stat_none(A, g, n);
    // kd.c:1766-1767: fHalfMass += 0.5*fMass (FP64 sum rounded to float)
    float fHalf = 0.0f;
    for (int j = 0; j < n; ++j)
        fHalf = (float)__dadd_rn((double)fHalf, __dmul_rn(0.5, (double)A.pos4[A.vals[s + j]].w));
    float fTot = 0.0f, fGas = 0.0f, fStar = 0.0f, fVc = 0.0f, fmVc = 0.0f, fVd = 0.0f;
    float fRVmax = 0.0f, fRh = 0.0f;
    StatMember q, nx;
    stat_load(A, s, n, 0, nx);
    for (int j = 0; j < n; ++j) {
        q = nx;
        stat_load(A, s, n, j + 1, nx);
        fTot = fadd(fTot, q.p.w);
        // kd.c:1774-1778: r2 > 4.0*soft*soft && G*fTot/sqrt(r2) > fVcirc
        // (FP64 comparisons); fRVmax = sqrt(r2), fVcirc = G*fTot/fRVmax (float)
        const double d2 = (double)q.r2;
        const float gm = fmul(A.G, fTot);
        if (d2 > __dmul_rn(__dmul_rn(4.0, (double)q.v.w), (double)q.v.w) &&
            __ddiv_rn((double)gm, __dsqrt_rn(d2)) > (double)fVc) {
            fRVmax = (float)__dsqrt_rn(d2);
            fVc = __fdiv_rn(gm, fRVmax);
        }
        if (q.gas) fGas = fadd(fGas, q.p.w);
        if (q.io >= A.nGas + A.nDark) fStar = fadd(fStar, q.p.w);
        if (fTot > fHalf && fmVc == 0.0f) {
            fRh = (float)__dsqrt_rn(d2);
            fmVc = __fdiv_rn(gm, fRh);
        }
        const float3 r = stat_rel(q.p, rg, A.h);
        fVd = fadd(fVd, stat_dv2(A, q.v.x, rg.vcm[0], r.x));
        fVd = fadd(fVd, stat_dv2(A, q.v.y, rg.vcm[1], r.y));
        fVd = fadd(fVd, stat_dv2(A, q.v.z, rg.vcm[2], r.z));
    }
    stat_store(A, g, n, fTot, fGas, fStar, fVc, fmVc, fRVmax, fRh, q.r2, fVd);
}

__global__ void stat_small_groups(StatArgs A)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (g < A.nGroup && A.rec[g].nMembers <= A.small) stat_thread(A, g);
}

__global__ void __launch_bounds__(ST_WARPS * 32) stat_groups(StatArgs A)
{
    __shared__ float term_s[ST_WARPS][4][ST_ROW];
    __shared__ float tot_s[ST_WARPS][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = blockIdx.x * ST_WARPS + w + 1;
    if (g >= A.nGroup) return;
    float (*term)[ST_ROW] = term_s[w];
    float *tot = tot_s[w];
    const skid_group rg = A.rec[g];
    const int n = rg.nMembers, s = A.start[g];
    if (A.small && n <= A.small) return;
    if (n <= 0) {
        if (lane == 0) stat_none(A, g, n);
        return;
    }
    // kd.c:1766-1767: fHalfMass += 0.5*fMass (FP64 sum rounded to float).  The
    // sum of two floats rounded to double and then to float is the float sum,
    // and 0.5 m is exact in float unless it is subnormal.
    float fHalf = 0.0f;
    {
        float mn = lane < n ? A.pos4[A.vals[s + lane]].w : 0.0f;
        for (int j0 = 0; j0 < n; j0 += 32) {
            const float m = mn;
            mn = j0 + 32 + lane < n ? A.pos4[A.vals[s + j0 + 32 + lane]].w : 0.0f;
            const bool odd = __any_sync(SKID_FULL, m != 0.0f && fabsf(m) < 1e-36f);
            __syncwarp();
            term[0][lane] = odd ? m : 0.5f * m;
            __syncwarp();
            if (lane == 0) {
                if (odd) {
                    for (int j = 0; j < 32; ++j)
                        fHalf = (float)__dadd_rn((double)fHalf, __dmul_rn(0.5, (double)term[0][j]));
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) fHalf = fadd(fHalf, term[0][j]);
                }
            }
        }
        fHalf = __shfl_sync(SKID_FULL, fHalf, 0);
    }
    float sum = 0.0f;   // lanes 0-3: total, gas, star mass, dispersion
    float fVc = 0.0f, fmVc = 0.0f, fRVmax = 0.0f, fRh = 0.0f;
    StatMember q, nx;
    stat_load(A, s, n, lane, nx);
    for (int j0 = 0; j0 < n; j0 += 32) {
        q = nx;
        stat_load(A, s, n, j0 + 32 + lane, nx);
        const bool in = j0 + lane < n;
        const bool star = in && q.io >= A.nGas + A.nDark;
        const float m = q.p.w;
        __syncwarp();
        // a chain's three adds a member: (m, 0, 0) for the masses -- adding
        // +0 changes no running sum, which starts at +0 and so is never -0 --
        // and the three squared velocity components for the dispersion
        term[0][3 * lane] = m;
        term[1][3 * lane] = in && q.gas ? m : 0.0f;
        term[2][3 * lane] = star ? m : 0.0f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            term[k][3 * lane + 1] = 0.0f;
            term[k][3 * lane + 2] = 0.0f;
        }
        const float3 r = stat_rel(q.p, rg, A.h);
        const float vv[3] = {q.v.x, q.v.y, q.v.z}, rr[3] = {r.x, r.y, r.z};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float d = stat_dv2(A, vv[k], rg.vcm[k], rr[k]);
            term[3][3 * lane + k] = in ? d : 0.0f;
        }
        __syncwarp();
        if (lane < 4) {
            const float *t = term[lane];
#pragma unroll 4
            for (int j = 0; j < 32; j += 4) {
                float x[12];
#pragma unroll
                for (int k = 0; k < 12; ++k) x[k] = t[3 * j + k];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    sum = fadd(sum, x[3 * k]);
                    if (lane == 0) tot[j + k] = sum;
                    sum = fadd(sum, x[3 * k + 1]);
                    sum = fadd(sum, x[3 * k + 2]);
                }
            }
        }
        __syncwarp();
        const float gm = fmul(A.G, tot[lane]);
        // kd.c:1774-1778: r2 > 4.0*soft*soft && G*fTot/sqrt(r2) > fVcirc
        // (FP64 comparisons); fRVmax = sqrt(r2), fVcirc = G*fTot/fRVmax (float).
        // The float estimate (within 1e-6) clears most members of the FP64
        // divide; those that may exceed the running maximum are taken in order.
        const double d2 = (double)q.r2;
        const float est = gm * rsqrtf(q.r2);
        const bool may = in && !(est > 1e-30f && est * 1.00001f < fVc) &&
                         d2 > __dmul_rn(__dmul_rn(4.0, (double)q.v.w), (double)q.v.w);
        if (__any_sync(SKID_FULL, may)) {
            double x = 0.0;
            float y = 0.0f, rv = 0.0f;
            if (may) {
                const double root = __dsqrt_rn(d2);
                x = __ddiv_rn((double)gm, root);
                rv = (float)root;
                y = __fdiv_rn(gm, rv);
            }
            for (int cur = 0; cur < 32;) {
                const unsigned b = __ballot_sync(SKID_FULL, may && lane >= cur && x > (double)fVc);
                if (!b) break;
                const int l = __ffs(b) - 1;
                fVc = __shfl_sync(SKID_FULL, y, l);
                fRVmax = __shfl_sync(SKID_FULL, rv, l);
                cur = l + 1;
            }
        }
        // the first radius that encloses more than half the mass
        for (int cur = 0; cur < 32 && fmVc == 0.0f;) {
            const unsigned b = __ballot_sync(SKID_FULL, in && lane >= cur && tot[lane] > fHalf);
            if (!b) break;
            const int l = __ffs(b) - 1;
            fRh = (float)__dsqrt_rn((double)__shfl_sync(SKID_FULL, q.r2, l));
            fmVc = __fdiv_rn(__shfl_sync(SKID_FULL, gm, l), fRh);
            cur = l + 1;
        }
    }
    const float r2 = __shfl_sync(SKID_FULL, q.r2, (n - 1) & 31);
    const float fTot = __shfl_sync(SKID_FULL, sum, 0);
    const float fGas = __shfl_sync(SKID_FULL, sum, 1);
    const float fStar = __shfl_sync(SKID_FULL, sum, 2);
    const float fVd = __shfl_sync(SKID_FULL, sum, 3);
    if (lane == 0) stat_store(A, g, n, fTot, fGas, fStar, fVc, fmVc, fRVmax, fRh, r2, fVd);
}

int bits_for_groups(int ng)
{
    int b = 1;
    while (b < 31 && (1 << b) <= ng) ++b;
    return b;
}

}  // namespace

extern "C" int skid_group_stats(skid_ctx *ctx, float G, float fExp, float fExpHub, float fDensMin,
                                float fTempMax, skid_stat *stats)
{
    if (!ctx || !stats) return SKID_EINVAL;
    if (ctx->stage < STAGE_FINAL) return ctx->fail(SKID_ESTATE);
    const int n = ctx->n, ng = ctx->G.nGroup;
    cudaStream_t st = ctx->st;
    SortScratch &ss = ctx->ss;
    if (dalloc(ss.k0, n) || dalloc(ss.k1, n) || dalloc(ss.v0, n) || dalloc(ss.v1, n) ||
        dalloc(ctx->stat_start, ng > 0 ? ng : 1) || dalloc(ctx->stat_out, ng > 0 ? ng : 1))
        return ctx->fail(SKID_ENOMEM);
    if (ng <= 1) return 0;
    const float3 h = make_float3((float)(0.5 * (double)ctx->L.x), (float)(0.5 * (double)ctx->L.y),
                                 (float)(0.5 * (double)ctx->L.z));
    if (n > 0) {
        stat_keys<<<grid_for(n), 256, 0, st>>>(ctx->pos4.p, ctx->grp.p, n, ctx->G.rec.p, h,
                                               ss.k0.p, ss.v0.p); note_launch();
        CK(radix_sort(ss, n, 32 + bits_for_groups(ng), st));
        CK(cudaMemsetAsync(ctx->stat_start.p, 0, ng * sizeof(int), st));
        stat_starts<<<grid_for(n), 256, 0, st>>>(ss.k0.p, n, ctx->stat_start.p); note_launch();
    }
    StatArgs A;
    A.keys = ss.k0.p;
    A.vals = ss.v0.p;
    A.start = ctx->stat_start.p;
    A.rec = ctx->G.rec.p;
    A.pos4 = ctx->pos4.p;
    A.vel4 = ctx->vel4.p;
    A.temp = ctx->temp.p;
    A.rho = ctx->rho_final.p;
    A.nGroup = ng;
    A.nGas = ctx->nGas;
    A.nDark = ctx->nDark;
    A.h = h;
    A.G = G;
    A.fExp = fExp;
    A.fExpHub = fExpHub;
    A.fDensMin = fDensMin;
    A.fTempMax = fTempMax;
    A.out = ctx->stat_out.p;
    A.small = ng - 1 >= ST_MANY * num_sms() ? ST_THREAD_MAX : 0;
    if (A.small) {
        stat_small_groups<<<(ng - 1 + 63) / 64, 64, 0, st>>>(A); note_launch();
    }
    stat_groups<<<(ng - 1 + ST_WARPS - 1) / ST_WARPS, ST_WARPS * 32, 0, st>>>(A); note_launch();
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(stats, ctx->stat_out.p, ng * sizeof(skid_stat), cudaMemcpyDeviceToHost, st));
    return ctx->sync_check();
}
