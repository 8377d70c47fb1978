/* topgrid.cu -- the top level of the hierarchical sum on the device: the support-following grow, the
 * shadow-tier flood fill and the dilation (driver/sumkey.h:20-461).
 *
 * Points of the top grid (step st) are identified by the reference's mixed-radix key
 * 1 c_0 ... c_{D-1} in base W = 2(K/st)+1, c_i = k_i/st + K/st (driver/sumkey.h:7-18): numeric order is
 * lexicographic order in k, and an axis step is +-P[j].
 *
 * One device hash table holds every evaluated point of the grow with a 32-bit claim word: SEEN for a
 * point already evaluated, else the best claim of this frontier's candidates, stored as
 * 0xFFFFFFFE - id so that atomicMax keeps the lowest candidate id (the reference's parallel claims,
 * driver/sumkey.h:288-374).  The winners, compacted in id order, are the next frontier: exactly the
 * not-yet-seen neighbours of the kept points in (kept point, axis, sign) order.
 *
 * A frontier's values never leave the device.  The running sum a of |f w| whose threshold eps a decides what is
 * kept is a sequence of rounded additions in point order, and it is replayed exactly in parallel (seq_sum): while
 * a stays in one binade with unit u every addition adds RN(x/u) units, so a chunk's additions are one integer sum;
 * the element that leaves the binade, or that lies half-way between units, is added by itself.  The sums
 * that decide nothing (S, the shells, the dropped weight, the round column) are double-double in a fixed order.
 * The host waits once per frontier, for the next one's size.  Waits, launches and the host's sums bound the grow
 * before (three waits and about 19 operations a frontier, 17 bytes a point to the host), launches now: d = 5, h = 1.5
 * (10 frontiers, 8816 points) 2.1 -> 0.66 ms; d = 8, h = 1 (17 frontiers, 4.06e6 points) 37 -> 3.5 ms.
 *
 * After the grow the table's claim words, all SEEN by then, serve the tiers (the index of a kept point) and the
 * dilation (the merged flags of a cell): every neighbour of a kept point was a candidate and is in the table.
 * (A table of its own, sized for four cells a kept point, overflowed at D = 11 and was probed from end to end before
 * it was enlarged: 26.4 s at h = 1, eps = 1e-8, 3.3 ms with the tiers now.)  The dilation's cells are the marked slots'
 * keys, sorted with a stable LSD radix sort (8-bit digits), the
 * reference's summation order.  Every probe loop is bounded by the table size and reports overflow instead of
 * spinning. */
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "sqb_rt.h"
#include "sqdd.cuh"

#define TG_T 256                 /* threads per CTA of the compaction kernels */
#define GT 1024                  /* threads of the one-CTA kernels */
#define GS_TILE 2048             /* points per tile of a larger frontier's sums */
#define SEEN 0xFFFFFFFFu
#define CLAIM(id) (0xFFFFFFFEu - (unsigned)(id))

static thread_local char terr[512];   /* the state of this file is per host thread, like the runtime's */
#define TCK(x) do { cudaError_t e_ = (x); if(e_ != cudaSuccess){                                    \
    snprintf(terr, sizeof terr, "%s at %s:%d: %s", #x, __FILE__, __LINE__, cudaGetErrorString(e_));   \
    cudaGetLastError();              /* reported here: not the next call's error */                  \
    return (int)e_; } } while(0)
extern "C" const char *sqb_top_error(void){ return terr; }

typedef unsigned long long u64;

__device__ __forceinline__ u64 hslot(u64 y, u64 mask){
    return ((y*0x9E3779B97F4A7C15ULL) >> 21) & mask;
}
/* slot of key y, inserting it if absent (*isnew = 1); -1 if the table is full */
__device__ long h_insert(u64 *key, u64 mask, u64 y, int *isnew){
    u64 i = hslot(y, mask);
    for(u64 p = 0; p <= mask; p++){
        u64 c = key[i];
        if(c == y){ *isnew = 0; return (long)i; }
        if(c == 0){
            u64 o = atomicCAS(&key[i], 0ULL, y);
            if(o == 0){ *isnew = 1; return (long)i; }
            if(o == y){ *isnew = 0; return (long)i; }
        }
        i = (i + 1) & mask;
    }
    return -1;
}
__device__ long h_find(const u64 *key, u64 mask, u64 y){
    u64 i = hslot(y, mask);
    for(u64 p = 0; p <= mask; p++){
        u64 c = key[i];
        if(c == y) return (long)i;
        if(c == 0) return -1;
        i = (i + 1) & mask;
    }
    return -1;
}

/* sh: log2 of the step */
struct geom_t { int D, K, st, sh, W; u64 P[SQB_MAXD]; };

/* a point of this file's lists as three words (the lists are 4-byte aligned; byte 11 is the flags) */
struct pt3 { unsigned w[3]; };
__device__ __forceinline__ pt3 ld_pt(const sqb_pt_t *p){ const unsigned *q = (const unsigned*)p; return {{q[0], q[1], q[2]}}; }
__device__ __forceinline__ void st_pt(sqb_pt_t *p, const pt3 &x){ unsigned *q = (unsigned*)p; q[0] = x.w[0]; q[1] = x.w[1]; q[2] = x.w[2]; }
__device__ __forceinline__ int pt_byte(const pt3 &x, int d){
    const unsigned w = d < 4 ? x.w[0] : d < 8 ? x.w[1] : x.w[2];
    return (int)(signed char)(w >> (8*(d & 3)));
}
__device__ __forceinline__ void pt_add(pt3 &x, int d, int v){            /* k[d] += v (no overflow of the byte) */
    const unsigned b = ((unsigned)v & 0xffu) << (8*(d & 3));
    if(d < 4) x.w[0] = __vadd4(x.w[0], b); else if(d < 8) x.w[1] = __vadd4(x.w[1], b); else x.w[2] = __vadd4(x.w[2], b);
}
__device__ __forceinline__ void pt_flag(pt3 &x, int f){ x.w[2] = (x.w[2] & 0x00ffffffu) | ((unsigned)(f & 0xff) << 24); }
/* max |k_d| */
__device__ __forceinline__ int pt_max(const pt3 &x){
    unsigned m = __vmaxu4(__vabs4(x.w[0]), __vmaxu4(__vabs4(x.w[1]), __vabs4(x.w[2] & 0x00ffffffu)));
    m = __vmaxu4(m, m >> 16);
    return (int)max(m & 0xffu, (m >> 8) & 0xffu);
}
__device__ __forceinline__ u64 key_pt(const geom_t &g, const pt3 &x){
    u64 y = 1;
    for(int i = 0; i < g.D; i++) y = y*g.W + (u64)((pt_byte(x, i) + g.K) >> g.sh);
    return y;
}
/* x = q n + r, in 32 bits where they do */
__device__ __forceinline__ void split(long x, int n, long *q, int *r){
    if(x <= 0xFFFFFFFFL){ const unsigned y = (unsigned)x/(unsigned)n; *q = y; *r = (int)((unsigned)x - y*(unsigned)n); }
    else { *q = x/n; *r = (int)(x - *q*n); }
}

/* the grow's counters and sums, in device memory and, after each wait, in pinned host memory */
struct gacc_t {
    double a, thr, eps, pw;                 /* running sum of |f w|, its threshold eps a, the weight step^D */
    double S[2], x1[2], x2[2], dr[2], gs[2], u[2];   /* sum f w; outer shells; dropped weight; its signed sum; round column */
    u64 ngs, nq, unres;                     /* points below the threshold; fallback and unresolved points */
    u64 nk, nn, nkeep;                      /* this frontier's kept points, the next frontier, kept so far */
    u64 nrun, seen, steps;                  /* the next frontier if one cluster takes it, else 0; points and frontiers so far */
    u64 m, ncell, err;                      /* kept after the final threshold; dilated cells; full-table inserts */
    u64 nz, punres;                         /* the zero probe: any value not 0; its unresolved points */
};

/* a barrier over the cluster that also orders its global memory accesses; the CTA's rank in the cluster */
__device__ __forceinline__ void cl_sync(){ asm volatile("barrier.cluster.arrive;\n\tbarrier.cluster.wait;" ::: "memory"); }
__device__ __forceinline__ int cl_rank(){ unsigned r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return (int)r; }

/* ------------------------------------- block sums and scans ------------------------------------------ */
__device__ __forceinline__ sqdd dd_shfl(const sqdd &a, int off){
    return sqdd(__shfl_down_sync(0xffffffffu, a.hi, off), __shfl_down_sync(0xffffffffu, a.lo, off));
}
template<int T> __device__ u64 block_sum(u64 x, u64 *sh){
    for(int off = 16; off; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
    if((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
    __syncthreads();
    u64 s = 0;
    for(int w = 0; w < T/32; w++) s += sh[w];
    __syncthreads();
    return s;
}
/* exclusive scan of x over the CTA, every partial sum cut off at cap; *total the CTA's sum */
template<int T> __device__ u64 block_scan(u64 x, u64 cap, u64 *total, u64 *sh){
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    u64 inc = x < cap ? x : cap;
    for(int off = 1; off < 32; off <<= 1){
        const u64 y = __shfl_up_sync(0xffffffffu, inc, off);
        if(l >= off){ inc += y; inc = inc < cap ? inc : cap; }
    }
    u64 ex = __shfl_up_sync(0xffffffffu, inc, 1);
    if(l == 0) ex = 0;
    if(l == 31) sh[w] = inc;
    __syncthreads();
    if(w == 0){
        u64 z = l < T/32 ? sh[l] : 0;
        for(int off = 1; off < 32; off <<= 1){
            const u64 y = __shfl_up_sync(0xffffffffu, z, off);
            if(l >= off){ z += y; z = z < cap ? z : cap; }
        }
        if(l < T/32) sh[l] = z;
    }
    __syncthreads();
    if(w > 0){ ex += sh[w - 1]; ex = ex < cap ? ex : cap; }
    *total = sh[T/32 - 1];
    __syncthreads();
    return ex;
}
template<int T> __device__ unsigned block_min(unsigned x, unsigned *sh){
    x = __reduce_min_sync(0xffffffffu, x);
    if((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
    __syncthreads();
    unsigned m = 0xFFFFFFFFu;
    for(int w = 0; w < T/32; w++) m = min(m, sh[w]);
    __syncthreads();
    return m;
}

/* NQ double-double sums and NC counts over the CTA at once, in a fixed order, the results in every thread: the warps'
 * trees interleave, then warp q adds the warps' parts of sum q */
template<int T, int NQ, int NC> struct sums_sh { double h[NQ][T/32], l[NQ][T/32]; u64 c[NC][T/32]; };
template<int T, int NQ, int NC> __device__ void block_sums(sqdd (&x)[NQ], u64 (&c)[NC], sums_sh<T, NQ, NC> &sh){
    static_assert(NQ + NC <= T/32, "a warp for each sum");
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    /* a sum that is zero in the whole warp (the shells, the round column mostly) has no tree */
#pragma unroll
    for(int q = 0; q < NQ; q++)
        if(__any_sync(0xffffffffu, x[q].hi != 0)) for(int off = 16; off; off >>= 1) x[q] = x[q] + dd_shfl(x[q], off);
#pragma unroll
    for(int q = 0; q < NC; q++)
        if(__any_sync(0xffffffffu, c[q] != 0)) for(int off = 16; off; off >>= 1) c[q] += __shfl_down_sync(0xffffffffu, c[q], off);
    if(l == 0){
#pragma unroll
        for(int q = 0; q < NQ; q++){ sh.h[q][w] = x[q].hi; sh.l[q][w] = x[q].lo; }
#pragma unroll
        for(int q = 0; q < NC; q++) sh.c[q][w] = c[q];
    }
    __syncthreads();
    if(w < NQ){
        sqdd y = l < T/32 ? sqdd(sh.h[w][l], sh.l[w][l]) : sqdd(0.0);
        for(int off = 16; off; off >>= 1) y = y + dd_shfl(y, off);
        if(l == 0){ sh.h[w][0] = y.hi; sh.l[w][0] = y.lo; }
    } else if(w < NQ + NC){
        u64 y = l < T/32 ? sh.c[w - NQ][l] : 0;
        for(int off = 16; off; off >>= 1) y += __shfl_down_sync(0xffffffffu, y, off);
        if(l == 0) sh.c[w - NQ][0] = y;
    }
    __syncthreads();
#pragma unroll
    for(int q = 0; q < NQ; q++) x[q] = sqdd(sh.h[q][0], sh.l[q][0]);
#pragma unroll
    for(int q = 0; q < NC; q++) c[q] = sh.c[q][0];
    __syncthreads();
}

/* ------------------------------ a sequential rounded sum, in parallel --------------------------------- */
/* For x >= 0 and a in [2^e, 2^(e+1)), u = 2^(e-52): RN(a + x) = a + u RN(x/u) as long as the result stays in the
 * binade and x/u is not half-way between two integers (there the parity of a/u decides).  So over the elements
 * up to the first that breaks this, the rounded additions in order are one sum of integers. */
#define SQ_ONE53 (1ULL << 53)
#define SQ_ODD (1ULL << 63)      /* the element, or an element of the tile, has to be added by itself */
__device__ __forceinline__ bool seq_binade(double a, double *inv, double *u){
    const int ex = (__double2hiint(a) >> 20) & 0x7ff;
    if(!(a > 0) || ex < 100 || ex > 1900) return false;
    *u = __hiloint2double((ex - 52) << 20, 0);
    *inv = __hiloint2double((2046 - (ex - 52)) << 20, 0);
    return true;
}
/* x in units of u: RN(x/u), or SQ_ODD */
__device__ __forceinline__ u64 seq_units(double x, double inv){
    const double t = __dmul_rn(x, inv), r = rint(t);
    return !(t < 0x1p53) || fabs(__dsub_rn(t, r)) == 0.5 ? SQ_ODD : (u64)r;
}
template<int T> struct seq_sh { u64 s[T/32]; unsigned m[T/32]; u64 pre; };
/* a after the additions of |v[i]| pw, i0 <= i < i1, one after another (called by all T threads) */
template<int T> __device__ double seq_sum(double a, const double *v, double pw, long i0, long i1, seq_sh<T> &sh){
    long i = i0;
    while(i < i1){
        if(!(a < INFINITY)) return a;                       /* infinite, and so it stays */
        double inv = 0, u = 0;
        const bool ok = seq_binade(a, &inv, &u);
        const u64 A0 = ok ? (u64)__dmul_rn(a, inv) : 0, room = ok ? SQ_ONE53 - A0 : SQ_ONE53;
        u64 q[4], s = 0;
#pragma unroll
        for(int e = 0; e < 4; e++){
            const long j = i + threadIdx.x*4L + e;
            const double w = j < i1 ? __dmul_rn(fabs(v[j]), pw) : 0.0;
            q[e] = ok ? seq_units(w, inv) : (w == 0 ? 0 : SQ_ODD);   /* outside the range only zeros pass */
            s += q[e] < room ? q[e] : room; s = s < room ? s : room;
        }
        u64 total, pre = block_scan<T>(s, room, &total, sh.s);
        unsigned first = 0xFFFFFFFFu; u64 at = 0;
#pragma unroll
        for(int e = 0; e < 4; e++){
            if(first == 0xFFFFFFFFu && (q[e] == SQ_ODD || pre + q[e] >= room)){ first = threadIdx.x*4u + e; at = pre; }
            if(first == 0xFFFFFFFFu) pre += q[e];
        }
        const unsigned f = block_min<T>(first, sh.m);
        if(f == 0xFFFFFFFFu){
            if(ok) a = __dmul_rn((double)(A0 + total), u);
            i += 4L*T;
            continue;
        }
        if(first == f) sh.pre = at;
        __syncthreads();
        if(ok) a = __dmul_rn((double)(A0 + sh.pre), u);
        a = __dadd_rn(a, __dmul_rn(fabs(v[i + f]), pw));
        i += f + 1;
        __syncthreads();
    }
    return a;
}

/* --------------------------------- ordered compaction ------------------------------------------------- */
/* An Op has bool pred(long i) and void emit(long i, u64 rank); with DROP, the |weight(i)| of an element that is left
 * out adds to the grow's dropped weight, and with DROP = 2 its weight(i) to the signed sum and its number to the
 * count as well (the frontiers' points; the final threshold has |f| alone and adds to the dropped weight only,
 * driver/sumkey.h:399-401).  The number of elements is read on the device (*np + nadd); the grid covers
 * the host's bound on it.  Counting and emitting are two launches; a CTA finds its offset by adding the counts
 * before it itself, up to OFFS_CTAS CTAs, above that from a scan of the counts. */
#define OFFS_CTAS 1024
struct drop_t { double dr[2], gs[2]; u64 n; };
struct cnt_t { const u64 *np; long mul, max; };          /* min(*np mul, max) elements (np NULL: max) */
__device__ __forceinline__ long cnt_of(const cnt_t &c){
    if(!c.np) return c.max;
    const long n = (long)*c.np*c.mul;
    return n < c.max ? n : c.max;
}
template<class Op, int I>
__global__ void __launch_bounds__(TG_T) k_count(const __grid_constant__ Op op, cnt_t cn, unsigned *bcnt, drop_t *drop){
    __shared__ u64 ws[TG_T/32];
    __shared__ sums_sh<TG_T, 2, 2> wd;
    const long n = cnt_of(cn), b0 = blockIdx.x*(long)(TG_T*I);
    u64 c = 0;
    if(b0 < n){
        sqdd d[2]; u64 m[2] = {0, 0};                  /* dropped weight and signed sum; their number, the count */
        for(int j = 0; j < I; j++){
            const long i = b0 + j*TG_T + threadIdx.x;
            if(i >= n) break;
            if(op.pred(i)) c++;
            else if constexpr(Op::DROP){
                const double w = op.weight(i);
                d[0] = sqdd_add_d(d[0], fabs(w)); d[1] = sqdd_add_d(d[1], w); m[0]++;
            }
        }
        if constexpr(Op::DROP){
            m[1] = c;
            block_sums<TG_T, 2, 2>(d, m, wd);
            c = m[1];
            if(threadIdx.x == 0) drop[blockIdx.x] = {{d[0].hi, d[0].lo}, {d[1].hi, d[1].lo}, m[0]};
        } else c = block_sum<TG_T>(c, ws);
    } else if(Op::DROP && threadIdx.x == 0) drop[blockIdx.x] = {{0, 0}, {0, 0}, 0};
    if(threadIdx.x == 0) bcnt[blockIdx.x] = (unsigned)c;
}
/* a CTA: exclusive scan of nb counts; the total into *tot.  CTA c scans the c-th nb counts */
__global__ void __launch_bounds__(GT) k_scan(const unsigned *bcnt, long nb, u64 *boff, u64 *tot){
    __shared__ u64 sh[GT/32];
    u64 carry = 0;
    bcnt += blockIdx.x*nb; boff += blockIdx.x*nb;
    for(long b = 0; b < nb; b += 4*GT){
        const long j = b + threadIdx.x*4L;
        unsigned c[4]; u64 s = 0, t;
#pragma unroll
        for(int e = 0; e < 4; e++){ c[e] = j + e < nb ? bcnt[j + e] : 0; s += c[e]; }
        u64 x = carry + block_scan<GT>(s, ~0ULL, &t, sh);
#pragma unroll
        for(int e = 0; e < 4; e++){ if(j + e < nb) boff[j + e] = x; x += c[e]; }
        carry += t;
    }
    if(threadIdx.x == 0 && tot) tot[blockIdx.x] = carry;
}
/* everything a CTA of an emitting kernel needs: counts, their scan (or NULL), and where the total goes */
struct emit_t { const unsigned *bcnt; const u64 *boff; long nb; u64 *tot; drop_t *drop; gacc_t *acc, *host; };
__device__ __forceinline__ void dd_into(double *dst, const sqdd &x){
    const sqdd z = sqdd(dst[0], dst[1]) + x;
    dst[0] = z.hi; dst[1] = z.lo;
}
/* the grow's record to pinned host memory (one warp) */
__device__ __forceinline__ void publish(const gacc_t *acc, gacc_t *host){
    const u64 *s = (const u64*)acc; u64 *d = (u64*)host;
    for(unsigned w = threadIdx.x; w < sizeof(gacc_t)/8; w += 32) d[w] = s[w];
}
/* one cluster takes a frontier of up to CL_MAX points, a thread up to 64 of its candidates */
#define CL 8                     /* CTAs of the one-cluster kernels, and their threads */
#define CT 512
#define CL_MAX ((long)CL*CT)     /* points of a frontier that one cluster takes: one per thread.  With four per thread
                                    the whole sum of d = 5, h = 1 (16 frontiers up to 12,000 points) took 1.76 ms, with one
                                    1.40, without the cluster 1.67 */
static __host__ __device__ __forceinline__ bool one_cluster(long n, int D2){ return n <= CL_MAX && n*D2 <= 64L*CL*CT; }
__device__ __forceinline__ void next_frontier(gacc_t *acc, u64 nn, int D2){
    acc->nn = nn; acc->seen += nn; acc->steps++; acc->nrun = one_cluster((long)nn, D2) ? nn : 0;
}
template<class Op, int I>
__global__ void __launch_bounds__(TG_T) k_emit(const __grid_constant__ Op op, cnt_t cn, emit_t e){
    __shared__ u64 ws[TG_T/32];
    __shared__ sums_sh<TG_T, 2, 1> wd;
    const long n = cnt_of(cn), b0 = blockIdx.x*(long)(TG_T*I);
    const bool last = blockIdx.x == gridDim.x - 1;
    if(b0 >= n && !last) return;
    u64 r;
    if(e.boff) r = e.boff[blockIdx.x];
    else {
        u64 s = 0;
        for(long j = threadIdx.x; j < (long)blockIdx.x; j += TG_T) s += e.bcnt[j];
        r = block_sum<TG_T>(s, ws);
    }
    for(int j = 0; j < I; j++){                     /* TG_T consecutive elements at a time keep the order */
        const long i = b0 + j*TG_T + threadIdx.x;
        if(b0 + j*TG_T >= n) break;
        const int p = i < n && op.pred(i);
        u64 t;
        const u64 x = block_scan<TG_T>((u64)p, ~0ULL, &t, ws);
        if(p) op.emit(i, r + x);
        r += t;
    }
    if(!last) return;
    if constexpr(Op::DROP){
        sqdd d[2]; u64 m[1] = {0};
        for(long j = threadIdx.x; j < e.nb; j += TG_T){
            const drop_t &p = e.drop[j];
            d[0] = d[0] + sqdd(p.dr[0], p.dr[1]); d[1] = d[1] + sqdd(p.gs[0], p.gs[1]); m[0] += p.n;
        }
        block_sums<TG_T, 2, 1>(d, m, wd);
        if(threadIdx.x == 0){
            dd_into(e.acc->dr, d[0]);
            if(Op::DROP == 2){ dd_into(e.acc->gs, d[1]); e.acc->ngs += m[0]; }
        }
    }
    if(threadIdx.x == 0){
        *e.tot = r;
        if(Op::DROP) e.acc->nkeep = op.base + r;
        if(e.host) next_frontier(e.acc, r, op.D2);         /* the winners */
        __threadfence();
    }
    __syncthreads();
    if(e.host && threadIdx.x < 32) publish(e.acc, e.host);
}

/* a grid that covers n items, at most 1184 CTAs of 256 */
static unsigned grid256(long n){ const long w = (n + 255)/256; return (unsigned)(w < 1 ? 1 : w < 1184 ? w : 1184); }
struct Scratch { unsigned *bcnt; u64 *boff; drop_t *drop; long nbcap; };
static thread_local Scratch SC;
static thread_local cudaStream_t TS;
/* stream-ordered allocation from the device's memory pool: no device-wide synchronisation, and the pool
 * keeps freed memory for the next integral (the runtime sets its release threshold) */
#define DMALLOC(p, n) cudaMallocAsync((void**)(p), (n), TS)
#define DFREE(p) cudaFreeAsync((p), TS)
static thread_local u64 TL;    /* kernels launched by this file */
extern "C" unsigned long long sqb_top_launches(void){ return TL; }
extern "C" void sqb_dev_count_copy(unsigned long long h2d, unsigned long long d2h);

/* device memory of one function: released on every return, an error's included, unless it is handed on (keep) */
template<class T> struct Tmp {
    T *p = NULL;
    Tmp(){}
    Tmp(const Tmp &) = delete;
    Tmp &operator=(const Tmp &) = delete;
    ~Tmp(){ drop(); }
    int get(long n){ TCK(DMALLOC(&p, n*sizeof(T))); return 0; }
    T *keep(){ T *q = p; p = NULL; return q; }
    void drop(){ if(p) DFREE(p); p = NULL; }
};
/* a held pointer replaced */
template<class T> static void hold(T *&dst, T *p){ if(dst) DFREE(dst); dst = p; }

static int scratch(long nb){
    if(nb <= SC.nbcap) return 0;
    long c = 1024; while(c < nb) c <<= 1;
    Tmp<unsigned> a; Tmp<u64> b; Tmp<drop_t> d;
    if(a.get(c) || b.get(c) || d.get(c)) return -1;
    hold(SC.bcnt, a.keep()); hold(SC.boff, b.keep()); hold(SC.drop, d.keep());
    SC.nbcap = c;
    return 0;
}
template<class Op, int I>
static int compact_i(const Op &op, cnt_t cn, u64 *tot, gacc_t *acc, gacc_t *host){
    const long nb = (cn.max + TG_T*I - 1)/(TG_T*I);
    if(scratch(nb)) return -1;
    k_count<Op, I><<<(unsigned)nb, TG_T, 0, TS>>>(op, cn, SC.bcnt, SC.drop);
    const bool scan = nb > OFFS_CTAS;
    if(scan){ k_scan<<<1, GT, 0, TS>>>(SC.bcnt, nb, SC.boff, NULL); TL++; }
    emit_t e = {SC.bcnt, scan ? SC.boff : NULL, nb, tot, SC.drop, acc, host};
    k_emit<Op, I><<<(unsigned)nb, TG_T, 0, TS>>>(op, cn, e);
    TL += 2;
    TCK(cudaGetLastError());
    return 0;
}
/* one element per thread while that fills the device in one round, else eight */
template<class Op>
static int compact(const Op &op, cnt_t cn, u64 *tot, gacc_t *acc, gacc_t *host){
    return cn.max <= 1L << 18 ? compact_i<Op, 1>(op, cn, tot, acc, host) : compact_i<Op, 8>(op, cn, tot, acc, host);
}

/* --------------------------------------------- grow --------------------------------------------- */
struct gpart_t { u64 q; double f[4][2]; u64 nq, unres; };    /* one tile of a frontier's sums */
struct clpart_t { gpart_t s; drop_t d; double a; u64 nk, nw; };                /* one of its CTAs' sums and counts */
struct Grow {
    geom_t g;
    u64 *key; unsigned *word; u64 mask; long nseen;   /* seen table */
    sqb_pt_t *fr, *nx; unsigned char *frsk, *nxsk; long nfr, frcap;         /* frontier, next */
    sqb_pt_t *keep; double *kv; u64 *kk; long nkeep, keepcap;               /* kept so far: points, values, keys */
    long *kj; long kjcap;                                                  /* this frontier's kept */
    long *qs; long qscap;                                                  /* slot per candidate */
    gpart_t *part; long partcap; clpart_t *cpart;                          /* sums per tile; per CTA of a cluster */
    gacc_t *acc, *host;                                                    /* device record; its pinned copy */
    sqb_pt_t *probe;                                                       /* the zero probe's points */
    int gs, abskip, nfrs;
};
static thread_local Grow GR;

__global__ void k_rehash(const u64 *ok, const unsigned *ow, long ocap, u64 *key, unsigned *word, u64 mask, gacc_t *acc){
    for(long i = blockIdx.x*(long)blockDim.x + threadIdx.x; i < ocap; i += (long)gridDim.x*blockDim.x){
        if(!ok[i]) continue;
        int nw; long q = h_insert(key, mask, ok[i], &nw);
        if(q < 0){ atomicAdd(&acc->err, 1ULL); continue; }
        word[q] = ow[i];
    }
}
/* keep the seen table at most 60% full after extra more keys */
static int table_room(long extra){
    long cap = (long)GR.mask + 1;
    if((double)(GR.nseen + extra) <= 0.6*cap) return 0;
    long nc = cap; while((double)(GR.nseen + extra) > 0.6*nc) nc <<= 1;
    Tmp<u64> k2; Tmp<unsigned> w2;
    if(k2.get(nc) || w2.get(nc)) return -1;
    TCK(cudaMemsetAsync(k2.p, 0, nc*sizeof(u64), TS)); TCK(cudaMemsetAsync(w2.p, 0, nc*sizeof(unsigned), TS));
    k_rehash<<<1184, 256, 0, TS>>>(GR.key, GR.word, cap, k2.p, w2.p, (u64)(nc - 1), GR.acc); TL++;
    TCK(cudaGetLastError());
    hold(GR.key, k2.keep()); hold(GR.word, w2.keep()); GR.mask = (u64)(nc - 1);
    return 0;
}
/* device array of at least n elements, keeping the first keep elements */
template<class T> static int devbuf(T **p, long *cap, long n, long keep){
    if(n <= *cap && *p) return 0;
    long c = 1L << 16; while(c < n) c <<= 1;
    Tmp<T> q;
    if(q.get(c)) return -1;
    if(*p && keep > 0) TCK(cudaMemcpyAsync(q.p, *p, keep*sizeof(T), cudaMemcpyDeviceToDevice, TS));
    hold(*p, q.keep()); *cap = c;
    return 0;
}
/* frontier buffers for n points, the current frontier kept */
static int frontier_room(long n){
    if(n <= GR.frcap && GR.fr) return 0;
    long c = 1L << 16; while(c < n) c <<= 1;
    Tmp<sqb_pt_t> a, b; Tmp<unsigned char> s1, s2;
    if(a.get(c) || b.get(c) || s1.get(c) || s2.get(c)) return -1;
    if(GR.fr){
        TCK(cudaMemcpyAsync(a.p, GR.fr, GR.nfr*sizeof(sqb_pt_t), cudaMemcpyDeviceToDevice, TS));
        TCK(cudaMemcpyAsync(s1.p, GR.frsk, GR.nfr, cudaMemcpyDeviceToDevice, TS));
    }
    hold(GR.fr, a.keep()); hold(GR.nx, b.keep()); hold(GR.frsk, s1.keep()); hold(GR.nxsk, s2.keep()); GR.frcap = c;
    return 0;
}

/* z = 0 into the table and the frontier, the record cleared, and the zero probe's nodes (driver/sum.c:346-359): z = 0
 * and NPROBE nodes from a fixed hash */
#define NPROBE 4096
__global__ void k_seed(const __grid_constant__ geom_t g, u64 *key, unsigned *word, u64 mask, u64 y0, sqb_pt_t *fr, unsigned char *frsk, gacc_t *acc,
                       double eps, double pw, sqb_pt_t *probe){
    const int j = blockIdx.x*blockDim.x + threadIdx.x;
    if(j == 0){
        gacc_t z = {}; z.eps = eps; z.pw = pw; z.nrun = z.seen = 1;
        int nw; const long q = h_insert(key, mask, y0, &nw);
        if(q < 0) z.err = 1; else word[q] = SEEN;
        for(int i = 0; i < SQB_MAXD; i++) fr[0].k[i] = 0;
        frsk[0] = 0;
        *acc = z;
    }
    if(j > NPROBE) return;
    sqb_pt_t p;
    for(int i = 0; i < SQB_MAXD; i++) p.k[i] = 0;
    u64 y = 0x9E3779B97F4A7C15ULL*(u64)(j + 1);
    const int h = g.K/g.st; const u64 W = 2*h + 1;
    if(j) for(int d = 0; d < g.D; d++){ y ^= y >> 29; y *= 0xBF58476D1CE4E5B9ULL; y ^= y >> 32; p.k[d] = (signed char)(((int)(y % W) - h)*g.st); }
    probe[j] = p;
}
__global__ void __launch_bounds__(GT) k_probe_check(const double *v, const unsigned char *stt, gacc_t *acc){
    __shared__ u64 sh[GT/32];
    u64 nz = 0, un = 0;
    for(int j = threadIdx.x; j <= NPROBE; j += GT){ nz += v[j] != 0; un += (stt[j] & SQB_UNRES) != 0; }
    nz = block_sum<GT>(nz, sh); un = block_sum<GT>(un, sh);
    if(threadIdx.x == 0){ acc->nz = nz; acc->punres = un; }
}

/* a new grow at step st with threshold eps times the running sum; the frontier is z = 0.  *probe, *nprobe: the zero
 * probe's nodes, for the caller to evaluate and hand to sqb_grow_probe */
extern "C" int sqb_grow_begin(int D, int K, int st, int W, const unsigned long long *P, int gs, int abskip, double eps, double pw,
                              void *stream, const sqb_pt_t **probe, long *nprobe){
    TS = (cudaStream_t)stream;
    memset(&GR.g, 0, sizeof GR.g);
    GR.g.D = D; GR.g.K = K; GR.g.st = st; GR.g.W = W; for(int i = 0; i < D; i++) GR.g.P[i] = P[i];
    while((1 << GR.g.sh) < st) GR.g.sh++;
    GR.gs = gs; GR.abskip = abskip; GR.nseen = 1; GR.nkeep = 0; GR.nfr = 0; GR.nfrs = 0;
    const long cap = 1L << 20;
    Tmp<u64> key; Tmp<unsigned> word;
    if(key.get(cap) || word.get(cap)) return -1;
    hold(GR.key, key.keep()); hold(GR.word, word.keep());
    TCK(cudaMemsetAsync(GR.key, 0, cap*sizeof(u64), TS)); TCK(cudaMemsetAsync(GR.word, 0, cap*sizeof(unsigned), TS));
    GR.mask = (u64)(cap - 1);
    if(!GR.acc) TCK(DMALLOC(&GR.acc, sizeof(gacc_t)));
    if(!GR.host) TCK(cudaMallocHost(&GR.host, sizeof(gacc_t)));
    if(!GR.cpart) TCK(DMALLOC(&GR.cpart, CL*sizeof(clpart_t)));
    if(!GR.probe) TCK(DMALLOC(&GR.probe, (NPROBE + 1)*sizeof(sqb_pt_t)));
    if(frontier_room(1)) return -1;
    u64 y0 = 1; for(int i = 0; i < D; i++) y0 = y0*W + (u64)(K/st);
    k_seed<<<(NPROBE + 256)/256, 256, 0, TS>>>(GR.g, GR.key, GR.word, GR.mask, y0, GR.fr, GR.frsk, GR.acc, eps, pw, GR.probe); TL++;
    TCK(cudaGetLastError());
    GR.nfr = 1;
    *probe = GR.probe; *nprobe = NPROBE + 1;
    return 0;
}
extern "C" int sqb_grow_probe(const double *v_dev, const unsigned char *stt_dev){
    k_probe_check<<<1, GT, 0, TS>>>(v_dev, stt_dev, GR.acc); TL++;
    TCK(cudaGetLastError());
    return 0;
}
extern "C" long sqb_grow_frontier(const sqb_pt_t **pts, const unsigned char **skip){
    *pts = GR.fr; *skip = GR.gs ? GR.frsk : NULL; return GR.nfr;
}

/* a frontier point's part of the sums: S, the two outer shells, the round column; fallback and unresolved points */
__device__ __forceinline__ void fsum_add(sqdd (&f)[4], u64 &nq, u64 &unres, const geom_t &g, const sqb_pt_t *fr, const double *v,
                                         const unsigned char *stt, const double *uu, double pw, long i){
    const double x = __dmul_rn(v[i], pw), w = fabs(x);
    f[0] = sqdd_add_d(f[0], x);
    const int mx = pt_max(ld_pt(fr + i));     /* driver/sumkey.h:236-238 */
    if(mx == g.K) f[1] = sqdd_add_d(f[1], w); else if(mx == g.K - g.st) f[2] = sqdd_add_d(f[2], w);
    const unsigned char s = stt[i];
    if(s & SQB_FALLBACK){ nq++; f[3] = sqdd_add_d(f[3], uu[i]); }
    if(s & SQB_UNRES) unres++;
}
/* per tile of GS_TILE points: the sums, and the running sum's additions in units of its binade */
__global__ void __launch_bounds__(TG_T) k_gs_tiles(const __grid_constant__ geom_t g, const sqb_pt_t *fr, const double *v, const unsigned char *stt,
                                                   const double *uu, long n, const gacc_t *acc, gpart_t *part){
    __shared__ sums_sh<TG_T, 4, 4> sh;
    const double pw = acc->pw; double inv = 0, u;
    const bool ok = seq_binade(acc->a, &inv, &u);
    sqdd f[4]; u64 c[4] = {0, 0, 0, 0};
    for(int j = 0; j < GS_TILE/TG_T; j++){
        const long i = blockIdx.x*(long)GS_TILE + j*TG_T + threadIdx.x;
        if(i >= n) break;
        fsum_add(f, c[0], c[1], g, fr, v, stt, uu, pw, i);
        const u64 x = ok ? seq_units(__dmul_rn(fabs(v[i]), pw), inv) : SQ_ODD;
        /* GS_TILE = 2^11 terms below 2^42 cannot overflow the tile's sum (nor would 2^52: what the sums may not pass is
         * tested where they are added up); a tile with a larger one goes element by element */
        if(x == SQ_ODD || x >= SQ_ONE53 >> 11) c[2] = 1; else c[3] += x;
    }
    block_sums<TG_T, 4, 4>(f, c, sh);
    if(threadIdx.x == 0) part[blockIdx.x] = gpart_t{c[2] ? SQ_ODD : c[3], {{f[0].hi, f[0].lo}, {f[1].hi, f[1].lo}, {f[2].hi, f[2].lo},
                                                    {f[3].hi, f[3].lo}}, c[0], c[1]};
}
/* one CTA: the tiles' sums in order, the running sum and its threshold */
__global__ void __launch_bounds__(GT) k_gs_total(const double *v, long n, gacc_t *acc, const gpart_t *part, long nb){
    __shared__ sums_sh<GT, 4, 2> ss;
    __shared__ u64 ws[GT/32];
    __shared__ unsigned wm[GT/32];
    __shared__ seq_sh<GT> sh;
    __shared__ u64 pre_;
    sqdd f[4]; u64 c[2] = {0, 0};
    for(long j = threadIdx.x; j < nb; j += GT){
        const gpart_t &p = part[j];
#pragma unroll
        for(int q = 0; q < 4; q++) f[q] = f[q] + sqdd(p.f[q][0], p.f[q][1]);
        c[0] += p.nq; c[1] += p.unres;
    }
    block_sums<GT, 4, 2>(f, c, ss);
    const double pw = acc->pw, a0 = acc->a;
    double a = a0, inv = 0, u = 0;
    const bool ok = seq_binade(a0, &inv, &u);
    long tb = 0;
    while(tb < nb){
        double i2, u2;
        if(!ok || !seq_binade(a, &i2, &u2) || u2 != u){ a = seq_sum<GT>(a, v, pw, tb*GS_TILE, n, sh); break; }
        const u64 A0 = (u64)__dmul_rn(a, inv), room = SQ_ONE53 - A0;
        const long b = tb + threadIdx.x;
        const u64 q = b < nb ? part[b].q : 0;
        u64 total, pre = block_scan<GT>(q, room, &total, ws);
        const bool stop = q == SQ_ODD || pre + q >= room;
        const unsigned fb = block_min<GT>(stop ? threadIdx.x : 0xFFFFFFFFu, wm);
        if(fb == 0xFFFFFFFFu){ a = __dmul_rn((double)(A0 + total), u); tb += GT; continue; }
        if(threadIdx.x == fb) pre_ = pre;
        __syncthreads();
        a = __dmul_rn((double)(A0 + pre_), u);
        const long i0 = (tb + fb)*GS_TILE, i1 = i0 + GS_TILE;
        a = seq_sum<GT>(a, v, pw, i0, i1 < n ? i1 : n, sh);
        tb += fb + 1;
        __syncthreads();
    }
    if(threadIdx.x == 0){
        dd_into(acc->S, f[0]); dd_into(acc->x1, f[1]); dd_into(acc->x2, f[2]); dd_into(acc->u, f[3]);
        acc->nq += c[0]; acc->unres += c[1];
        acc->a = a; acc->thr = __dmul_rn(acc->eps, a);
    }
}

struct KeepOp {                  /* kept frontier points and their keys appended to the keep list, their index to kj */
    enum { DROP = 2, D2 = 0 };
    geom_t g; const sqb_pt_t *fr; const double *v; const unsigned char *stt; const gacc_t *acc; int abskip;
    sqb_pt_t *keep; double *kv; u64 *kk; long *kj; u64 base;
    __device__ bool pred(long i) const { return fabs(v[i]) >= acc->thr; }
    __device__ double weight(long i) const { return __dmul_rn(v[i], acc->pw); }
    __device__ void emit(long i, u64 r) const { put(i, base + r, r); }
    __device__ void put(long i, u64 at, u64 r) const {
        pt3 p = ld_pt(fr + i);
        kk[at] = key_pt(g, p);
        pt_flag(p, abskip && !(stt[i] & SQB_NEAR));
        st_pt(keep + at, p); kv[at] = fabs(v[i]); kj[r] = i;
    }
};
/* candidate id = (kept point j of this frontier, axis, sign): its slot in the table, and its claim; keep, kk: the
 * frontier's part of the keep list */
__device__ __forceinline__ void claim_one(const geom_t &g, const sqb_pt_t *keep, const u64 *kk, u64 *key, unsigned *word, u64 mask,
                                          long *qs, gacc_t *acc, long id){
    long j; int c;
    split(id, 2*g.D, &j, &c);
    const int d = c >> 1, sg = (c & 1) ? 1 : -1, kx = keep[j].k[d] + g.st*sg;
    if(kx > g.K || kx < -g.K){ qs[id] = -1; return; }
    int nw; const long q = h_insert(key, mask, kk[j] + (sg > 0 ? g.P[d] : (u64)0 - g.P[d]), &nw);
    qs[id] = q;
    if(q < 0) atomicAdd(&acc->err, 1ULL); else atomicMax(&word[q], CLAIM(id));
}
__global__ void k_claim(const __grid_constant__ geom_t g, const sqb_pt_t *keep, const u64 *kk, u64 *key, unsigned *word, u64 mask, long *qs, gacc_t *acc){
    const long nc = (long)acc->nk*2*g.D;
    for(long id = blockIdx.x*(long)blockDim.x + threadIdx.x; id < nc; id += (long)gridDim.x*blockDim.x)
        claim_one(g, keep, kk, key, word, mask, qs, acc, id);
}
struct WinOp {                   /* winners in id order become the next frontier */
    enum { DROP = 0 };
    const sqb_pt_t *fr; const long *kj; const long *qs; unsigned *word; const unsigned char *frsk; const unsigned char *stt;
    sqb_pt_t *nx; unsigned char *nxsk; int D2, st, gs; u64 base;
    __device__ bool pred(long id) const { const long q = qs[id]; return q >= 0 && word[q] == CLAIM(id); }
    __device__ void emit(long id, u64 r) const {
        long j; int c;
        split(id, D2, &j, &c);
        const long pi = kj[j];
        pt3 p = ld_pt(fr + pi);
        int fl = 0;
        if(gs){ const int pg = pt_byte(p, SQB_PFLAG);
            fl = !frsk[pi] ? ((stt[pi] & SQB_NEAR) ? 0 : 1) : (pg < gs ? pg + 1 : 0);
            nxsk[r] = fl > 0; }
        pt_add(p, c >> 1, (c & 1) ? st : -st);
        pt_flag(p, fl);
        st_pt(nx + r, p);
        word[qs[id]] = SEEN;
    }
};

/* A frontier of up to CL_MAX points in one cluster: sums, threshold, kept points, claims and the next frontier, with
 * a cluster barrier between the steps.  Latency bounds a frontier of this size; as seven launches (sums, kept points in
 * one CTA, claims, winners counted and emitted) the same steps
 * took 0.66 ms for the grow of d = 5, h = 1.5 (10 frontiers, 8816 points); 0.59 with this.  CTA r takes the r-th eighth of the points
 * and of the candidates, a thread a run of consecutive ones, so that one scan per CTA ranks them. */
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(CT)
k_frontier(const __grid_constant__ KeepOp ko, const __grid_constant__ WinOp wo, const double *uu, u64 *key, u64 mask, long *qs, gacc_t *acc, gacc_t *host, clpart_t *part){
    __shared__ sums_sh<CT, 4, 4> ss;
    __shared__ sums_sh<CT, 2, 1> sd;
    __shared__ u64 ws[CT/32];
    __shared__ seq_sh<CT> sh;
    const geom_t &g = ko.g;
    const int r = cl_rank(), t = threadIdx.x, D2 = 2*g.D;
    const long n = (long)acc->nrun; const u64 base = acc->nkeep;
    if(n == 0) return;                                         /* the chain has ended, or its next frontier is larger */
    const double pw = acc->pw, a0 = acc->a;
    double inv = 0, u = 0;
    const bool ok = seq_binade(a0, &inv, &u);
    /* the sums */
    const int E = (int)((n + CL*CT - 1)/(CL*CT));              /* points per thread: 1 */
    const long i0 = ((long)r*CT + t)*E;
    {
        sqdd f[4]; u64 c[4] = {0, 0, 0, 0};
        for(int e = 0; e < E && i0 + e < n; e++){
            fsum_add(f, c[0], c[1], g, ko.fr, ko.v, ko.stt, uu, pw, i0 + e);
            const u64 x = ok ? seq_units(__dmul_rn(fabs(ko.v[i0 + e]), pw), inv) : SQ_ODD;
            if(x == SQ_ODD || x >= SQ_ONE53 >> 11) c[2] = 1; else c[3] += x;
        }
        block_sums<CT, 4, 4>(f, c, ss);
        if(t == 0) part[r].s = gpart_t{c[2] ? SQ_ODD : c[3], {{f[0].hi, f[0].lo}, {f[1].hi, f[1].lo}, {f[2].hi, f[2].lo}, {f[3].hi, f[3].lo}}, c[0], c[1]};
    }
    cl_sync();
    /* the running sum: one sum of integers if it stays in its binade (every thread has all it takes), else element by
     * element in CTA 0 */
    double a;
    {
        const u64 A0 = ok ? (u64)__dmul_rn(a0, inv) : 0, room = ok ? SQ_ONE53 - A0 : 0;
        u64 tot = 0; bool odd = !ok;
        for(int q = 0; q < CL; q++){ const u64 x = __ldcg(&part[q].s.q); odd = odd || x == SQ_ODD || tot + x >= room; tot += x; }
        if(!odd) a = __dmul_rn((double)(A0 + tot), u);
        else {
            if(r == 0){ a = seq_sum<CT>(a0, ko.v, pw, 0, n, sh); if(t == 0) part[0].a = a; }
            cl_sync();
            a = __ldcg(&part[0].a);
        }
    }
    const double thr = __dmul_rn(acc->eps, a);
    /* the kept points */
    unsigned km = 0; u64 tot, rank;
    {
        sqdd d[2]; u64 c[1] = {0};
        for(int e = 0; e < E && i0 + e < n; e++){
            const double v = ko.v[i0 + e];
            if(fabs(v) >= thr) km |= 1u << e;
            else { const double w = __dmul_rn(v, pw); d[0] = sqdd_add_d(d[0], fabs(w)); d[1] = sqdd_add_d(d[1], w); c[0]++; }
        }
        block_sums<CT, 2, 1>(d, c, sd);
        rank = block_scan<CT>((u64)__popc(km), ~0ULL, &tot, ws);
        if(t == 0){ part[r].d = {{d[0].hi, d[0].lo}, {d[1].hi, d[1].lo}, c[0]}; part[r].nk = tot; }
    }
    cl_sync();
    u64 nk = 0;
    for(int q = 0; q < CL; q++){ const u64 x = __ldcg(&part[q].nk); if(q < r) rank += x; nk += x; }
    for(unsigned b = km; b; b &= b - 1, rank++) ko.put(i0 + __ffs(b) - 1, base + rank, rank);
    if(r == CL - 1 && t < 7*32){
        /* the CTAs' parts into the record: warp w adds sum w, the last one the counts */
        const int w = t >> 5, l = t & 31;
        if(w < 6){
            const double *p = w < 4 ? part[l & 7].s.f[w] : w == 4 ? part[l & 7].d.dr : part[l & 7].d.gs;
            sqdd y = l < CL ? sqdd(__ldcg(p), __ldcg(p + 1)) : sqdd(0.0);
            for(int off = CL/2; off; off >>= 1) y = y + dd_shfl(y, off);
            double *dst[6] = {acc->S, acc->x1, acc->x2, acc->u, acc->dr, acc->gs};
            if(l == 0) dd_into(dst[w], y);
        } else if(l == 0){
            u64 x = 0, y = 0, z = 0;
            for(int q = 0; q < CL; q++){ x += __ldcg(&part[q].s.nq); y += __ldcg(&part[q].s.unres); z += __ldcg(&part[q].d.n); }
            acc->nq += x; acc->unres += y; acc->ngs += z;
        }
    }
    cl_sync();
    /* the claims */
    const long nc = (long)nk*D2;
    for(long id = (long)r*CT + t; id < nc; id += CL*CT) claim_one(g, ko.keep + base, ko.kk + base, key, wo.word, mask, qs, acc, id);
    if(r == 0 && t == 0){ acc->a = a; acc->thr = thr; acc->nk = nk; acc->nkeep = base + nk; }
    cl_sync();
    /* the winners */
    const long m = (nc + CL*CT - 1)/(CL*CT), id0 = ((long)r*CT + t)*m;
    u64 wm = 0;                                               /* m <= 64 */
    for(long e = 0; e < m && id0 + e < nc; e++) if(wo.pred(id0 + e)) wm |= 1ULL << e;
    rank = block_scan<CT>((u64)__popcll(wm), ~0ULL, &tot, ws);
    if(t == 0) part[r].nw = tot;
    cl_sync();
    u64 nn = 0;
    for(int q = 0; q < CL; q++){ const u64 x = __ldcg(&part[q].nw); if(q < r) rank += x; nn += x; }
    for(u64 b = wm; b; b &= b - 1) wo.emit(id0 + __ffsll((long long)b) - 1, rank++);
    if(r == 0 && t < 32){
        if(t == 0) next_frontier(acc, nn, D2);
        __syncwarp();
        publish(acc, host);
    }
}

/* the lists' part of the launch arguments, for the frontier in fr and its successor in nx */
static void frontier_ops(KeepOp *ko, WinOp *wo, sqb_pt_t *fr, sqb_pt_t *nx, unsigned char *frsk, unsigned char *nxsk, const double *v_dev,
                         const unsigned char *stt_dev){
    ko->g = GR.g; ko->fr = fr; ko->v = v_dev; ko->stt = stt_dev; ko->acc = GR.acc; ko->abskip = GR.abskip;
    ko->keep = GR.keep; ko->kv = GR.kv; ko->kk = GR.kk; ko->kj = GR.kj; ko->base = (u64)GR.nkeep;
    wo->fr = fr; wo->kj = GR.kj; wo->qs = GR.qs; wo->word = GR.word; wo->frsk = frsk; wo->stt = stt_dev;
    wo->nx = nx; wo->nxsk = nxsk; wo->D2 = 2*GR.g.D; wo->st = GR.g.st; wo->gs = GR.gs; wo->base = 0;
}
/* room for the points of n more frontier points and nc more candidates */
static int keep_room(long n){
    long kc = GR.keepcap, vc = GR.keepcap, yc = GR.keepcap;
    if(devbuf(&GR.keep, &kc, GR.nkeep + n, GR.nkeep) || devbuf(&GR.kv, &vc, GR.nkeep + n, GR.nkeep) ||
       devbuf(&GR.kk, &yc, GR.nkeep + n, GR.nkeep)) return -1;
    GR.keepcap = kc;
    return devbuf(&GR.kj, &GR.kjcap, n, 0);
}
static int cand_room(long nc, long frontiers){
    if(table_room(nc*frontiers)) return -1;
    if(devbuf(&GR.qs, &GR.qscap, nc, 0)) return -1;
    return frontier_room(nc);
}
/* after the host's wait: the counts, and err */
static int grow_counts(void){
    sqb_dev_count_copy(0, sizeof(gacc_t));
    GR.nkeep = (long)GR.host->nkeep; GR.nseen = (long)GR.host->seen; GR.nfr = (long)GR.host->nn;
    const int done = (int)((long)GR.host->steps - GR.nfrs);
    GR.nfrs = (int)GR.host->steps;
    if(done & 1){ sqb_pt_t *t = GR.fr; GR.fr = GR.nx; GR.nx = t; unsigned char *q = GR.frsk; GR.frsk = GR.nxsk; GR.nxsk = q; }
    if(GR.host->err){ snprintf(terr, sizeof terr, "grow: hash table overflow"); return -1; }
    return 0;
}
/* Frontiers that one cluster takes run in a chain: their sizes stay on the device (acc->nrun), the host queues the
 * evaluation and the step of SQB_GROW_CHAIN of them and waits once.  A frontier that turns out larger, or empty, ends the
 * chain: nrun is 0, and what is queued behind it does nothing.  (With the fallback inside the axis form's kernel, two launches a frontier and a
 * wait for four of them: whole sum of d = 5, h = 1.5, ten frontiers, 0.66 -> 0.56 ms.) */
extern "C" int sqb_grow_chain(long *nmax, const unsigned long long **np){
    const int D2 = 2*GR.g.D;
    *nmax = CL_MAX; *np = (const unsigned long long*)((char*)GR.acc + offsetof(gacc_t, nrun));
    if(!one_cluster(GR.nfr, D2)) return 0;
    if(keep_room(SQB_GROW_CHAIN*CL_MAX) || cand_room(CL_MAX*D2, SQB_GROW_CHAIN)) return -1;
    return SQB_GROW_CHAIN;
}
extern "C" void sqb_grow_link(int s, const sqb_pt_t **pts, const unsigned char **skip){
    *pts = s & 1 ? GR.nx : GR.fr; *skip = !GR.gs ? NULL : s & 1 ? GR.nxsk : GR.frsk;
}
extern "C" int sqb_grow_step(int s, const double *v_dev, const unsigned char *stt_dev, const double *uu_dev){
    KeepOp ko; WinOp wo;
    if(s & 1) frontier_ops(&ko, &wo, GR.nx, GR.fr, GR.nxsk, GR.frsk, v_dev, stt_dev);
    else frontier_ops(&ko, &wo, GR.fr, GR.nx, GR.frsk, GR.nxsk, v_dev, stt_dev);
    k_frontier<<<CL, CT, 0, TS>>>(ko, wo, uu_dev, GR.key, GR.mask, GR.qs, GR.acc, GR.host, GR.cpart); TL++;
    TCK(cudaGetLastError());
    return 0;
}
extern "C" int sqb_grow_wait(void){
    TCK(cudaStreamSynchronize(TS));
    return grow_counts();
}
/* a larger frontier: its evaluation (device arrays) in; its sums and kept points added, the next frontier built.  The host
 * waits once, for the next frontier's size; a frontier with more than 2^22 possible candidates also waits for its
 * kept count, so that the table and the candidate list grow by what is needed and not by that bound */
extern "C" int sqb_grow_expand(const double *v_dev, const unsigned char *stt_dev, const double *uu_dev){
    const long n = GR.nfr; const int D2 = 2*GR.g.D;
    if(keep_room(n)) return -1;
    KeepOp ko; WinOp wo;
    frontier_ops(&ko, &wo, GR.fr, GR.nx, GR.frsk, GR.nxsk, v_dev, stt_dev);
    const long nb = (n + GS_TILE - 1)/GS_TILE;
    if(devbuf(&GR.part, &GR.partcap, nb, 0)) return -1;
    k_gs_tiles<<<(unsigned)nb, TG_T, 0, TS>>>(GR.g, GR.fr, v_dev, stt_dev, uu_dev, n, GR.acc, GR.part);
    k_gs_total<<<1, GT, 0, TS>>>(v_dev, n, GR.acc, GR.part, nb);
    TL += 2;
    if(compact(ko, cnt_t{NULL, 1, n}, &GR.acc->nk, GR.acc, NULL)) return -1;
    long nk = n;
    if(n*D2 > 1L << 22){
        TCK(cudaMemcpyAsync(GR.host, GR.acc, sizeof(gacc_t), cudaMemcpyDeviceToHost, TS));
        TCK(cudaStreamSynchronize(TS));
        sqb_dev_count_copy(0, sizeof(gacc_t));
        nk = (long)GR.host->nk;
    }
    const long nc = nk*D2;
    if(nc >= 0xFFFFFFF0L){ snprintf(terr, sizeof terr, "grow: %ld candidates exceed the 32-bit claim ids", nc); return -1; }
    if(cand_room(nc > 0 ? nc : 1, 1)) return -1;
    frontier_ops(&ko, &wo, GR.fr, GR.nx, GR.frsk, GR.nxsk, v_dev, stt_dev);      /* the lists may have moved */
    if(nc){
        k_claim<<<grid256(nc), 256, 0, TS>>>(GR.g, GR.keep + GR.nkeep, GR.kk + GR.nkeep, GR.key, GR.word, GR.mask, GR.qs, GR.acc); TL++;
        TCK(cudaGetLastError());
    }
    if(compact(wo, cnt_t{&GR.acc->nk, D2, nc > 0 ? nc : 1}, &GR.acc->nn, GR.acc, GR.host)) return -1;
    TCK(cudaStreamSynchronize(TS));
    return grow_counts();
}

/* the running sum on its own (checks): a + |v[0]| pw + |v[1]| pw + ..., each addition rounded, for n values on the
 * device, through the small frontiers' route (tiles = 0) or the tiles' */
__global__ void __launch_bounds__(GT) k_seq_check(const double *v, long n, gacc_t *acc){
    __shared__ seq_sh<GT> sh;
    const double a = seq_sum(acc->a, v, acc->pw, 0, n, sh);
    if(threadIdx.x == 0) acc->a = a;
}
extern "C" int sqb_running_sum(const double *v_dev, long n, double a, double pw, int tiles, void *stream, double *out){
    TS = (cudaStream_t)stream;
    const long nb = (n + GS_TILE - 1)/GS_TILE;
    gacc_t h; memset(&h, 0, sizeof h); h.a = a; h.pw = pw;
    const size_t pb = (size_t)(n + 1)*(sizeof(sqb_pt_t) + 1);
    Tmp<gacc_t> acc_; Tmp<gpart_t> part_; Tmp<char> pts_;
    if(acc_.get(1) || part_.get(nb + 1) || pts_.get((long)pb)) return -1;
    gacc_t *const acc = acc_.p; gpart_t *const part = part_.p; char *const pts = pts_.p;
    TCK(cudaMemcpyAsync(acc, &h, sizeof h, cudaMemcpyHostToDevice, TS));
    TCK(cudaMemsetAsync(pts, 0, pb, TS));
    geom_t g; memset(&g, 0, sizeof g); g.D = 1; g.K = 1; g.st = 1; g.W = 3;
    if(!tiles) k_seq_check<<<1, GT, 0, TS>>>(v_dev, n, acc);
    else if(n > 0){
        k_gs_tiles<<<(unsigned)nb, TG_T, 0, TS>>>(g, (const sqb_pt_t*)pts, v_dev, (const unsigned char*)pts + (n + 1)*sizeof(sqb_pt_t), v_dev, n, acc, part);
        k_gs_total<<<1, GT, 0, TS>>>(v_dev, n, acc, part, nb);
    }
    TCK(cudaGetLastError());
    TCK(cudaMemcpyAsync(&h, acc, sizeof h, cudaMemcpyDeviceToHost, TS));
    TCK(cudaStreamSynchronize(TS));
    *out = h.a;
    return 0;
}

/* the zero probe's answer (valid after the first frontier's expansion) */
extern "C" int sqb_grow_probe_zero(long *unres){ *unres = (long)GR.host->punres; return GR.host->nz == 0; }

struct RethOp {
    enum { DROP = 1, D2 = 0 };
    const sqb_pt_t *keep; const double *kv; const u64 *kk; const gacc_t *acc; sqb_pt_t *out; double *okv; u64 *okk; u64 base;
    __device__ bool pred(long i) const { return kv[i] >= acc->thr; }
    __device__ double weight(long i) const { return __dmul_rn(kv[i], acc->pw); }
    __device__ void emit(long i, u64 r) const { st_pt(out + r, ld_pt(keep + i)); okv[r] = kv[i]; okk[r] = kk[i]; }
};

/* shadow tiers: breadth-first from z = 0 through kept points with |f| >= 10 thr (tier 1) and 100 thr (tier 2)
 * (driver/sumkey.h:402-444), both at once: a point of tier t raises a neighbour to the highest tier up to t
 * whose bound the neighbour's value meets, and a raised point goes (again) into the next step's list */
__global__ void k_index(const u64 *kk, const u64 *key, unsigned *word, u64 mask, gacc_t *acc){
    const long m = (long)acc->m;
    for(long i = blockIdx.x*(long)blockDim.x + threadIdx.x; i < m; i += (long)gridDim.x*blockDim.x){
        const long q = h_find(key, mask, kk[i]);
        if(q < 0){ atomicAdd(&acc->err, 1ULL); continue; }
        word[q] = (unsigned)i;
    }
}
__device__ __forceinline__ unsigned tier_of(double f, double thr){ return (f >= 10*thr) + (f >= 100*thr); }
__device__ __forceinline__ void tier_seed(const geom_t &g, const u64 *key, const unsigned *word, u64 mask, const double *kv, double thr,
                                          unsigned *tr, long *cu, u64 *cnt){
    u64 y = 1; for(int i = 0; i < g.D; i++) y = y*g.W + (u64)(g.K >> g.sh);
    const long q = h_find(key, mask, y);
    cnt[0] = cnt[1] = cnt[2] = 0;
    if(q < 0 || word[q] == SEEN) return;
    const long i = word[q];
    const unsigned t = tier_of(kv[i], thr);
    if(t){ tr[i] = t; cu[0] = i; cnt[0] = 1; }
}
__global__ void k_tier_seed(const __grid_constant__ geom_t g, const u64 *key, const unsigned *word, u64 mask, const double *kv, const gacc_t *acc,
                            unsigned *tr, long *cu, u64 *cnt){
    tier_seed(g, key, word, mask, kv, acc->thr, tr, cu, cnt);
}
__device__ __forceinline__ void tier_edge(const geom_t &g, const sqb_pt_t *keep, const u64 *kk, const u64 *key, const unsigned *word,
                                          u64 mask, const double *kv, double thr, unsigned *tr, const long *cu, long x, long *nw, u64 *nnw){
    long p; int c;
    split(x, 2*g.D, &p, &c);
    const long i = __ldcg(cu + p);
    const int d = c >> 1, sg = (c & 1) ? 1 : -1, kx = keep[i].k[d] + g.st*sg;
    if(kx > g.K || kx < -g.K) return;
    const long q = h_find(key, mask, kk[i] + (sg > 0 ? g.P[d] : (u64)0 - g.P[d]));
    if(q < 0 || word[q] == SEEN) return;
    const long j = word[q];
    const unsigned t = min(*(volatile unsigned*)&tr[i], tier_of(kv[j], thr));
    if(t && *(volatile unsigned*)&tr[j] < t && atomicMax(&tr[j], t) < t) nw[atomicAdd(nnw, 1ULL)] = j;
}
__global__ void k_tier_step(const __grid_constant__ geom_t g, const sqb_pt_t *keep, const u64 *kk, const u64 *key, const unsigned *word, u64 mask, const double *kv,
                            const gacc_t *acc, unsigned *tr, const long *cu, long *nw, u64 *cnt, int s){
    const int D2 = 2*g.D;
    const long nc = (long)cnt[s % 3]*D2;      /* this step's list, written by the step (or seed) before */
    if(blockIdx.x == 0 && threadIdx.x == 0) cnt[(s + 2) % 3] = 0;
    for(long x = blockIdx.x*(long)blockDim.x + threadIdx.x; x < nc; x += (long)gridDim.x*blockDim.x)
        tier_edge(g, keep, kk, key, word, mask, kv, acc->thr, tr, cu, x, nw, &cnt[(s + 1) % 3]);
}
/* what a long way round leaves after the steps the host launched: one CTA, step after step to the end (every step
 * raises at least one point, at most twice) */
__global__ void __launch_bounds__(GT) k_tier_rest(const __grid_constant__ geom_t g, const sqb_pt_t *keep, const u64 *kk, const u64 *key, const unsigned *word, u64 mask,
                                                  const double *kv, const gacc_t *acc, unsigned *tr, long *cu, long *nw, u64 *cnt, int s){
    const int D2 = 2*g.D;
    const long bound = 2*(long)acc->m + 1;
    for(long it = 0; it < bound; it++, s++){
        const long nc = (long)*(volatile u64*)&cnt[s % 3]*D2;
        if(nc == 0) break;
        if(threadIdx.x == 0) cnt[(s + 2) % 3] = 0;
        __syncthreads();
        for(long x = threadIdx.x; x < nc; x += GT)
            tier_edge(g, keep, kk, key, word, mask, kv, acc->thr, tr, cu, x, nw, &cnt[(s + 1) % 3]);
        __threadfence();
        __syncthreads();
        long *t = cu; cu = nw; nw = t;
    }
}
/* the whole flood of a kept list of up to TIER_CL points in one cluster, the index and the flags included: a step costs a
 * barrier instead of a launch.  With the bitmap below, final threshold to cells of d = 5, h = 1.5 (3783 kept): 0.24 -> 0.12
 * ms; of 47,579 kept points one cluster is the slower one (0.43 against 0.35 ms) */
#define TIER_CL (1L << 14)
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(CT)
k_tiers(const __grid_constant__ geom_t g, sqb_pt_t *keep, const u64 *kk, const u64 *key, unsigned *word, u64 mask, const double *kv, gacc_t *acc, unsigned *tr,
        long *cu, long *nw, u64 *cnt){
    const long m = (long)acc->m; const int D2 = 2*g.D, r = cl_rank();
    const double thr = acc->thr;
    const long x0 = (long)r*CT + threadIdx.x;
    for(long i = x0; i < m; i += CL*CT){
        const long q = h_find(key, mask, kk[i]);
        tr[i] = 0;
        if(q < 0) atomicAdd(&acc->err, 1ULL); else word[q] = (unsigned)i;
    }
    cl_sync();
    if(x0 == 0) tier_seed(g, key, word, mask, kv, thr, tr, cu, cnt);
    cl_sync();
    const long bound = 2*m + 1;                 /* every step raises at least one point, each at most twice */
    for(long s = 0; s < bound; s++){
        const long nc = (long)__ldcg(&cnt[s % 3])*D2;
        if(nc == 0) break;
        if(x0 == 0) cnt[(s + 2) % 3] = 0;
        for(long x = x0; x < nc; x += CL*CT)
            tier_edge(g, keep, kk, key, word, mask, kv, thr, tr, cu, x, nw, &cnt[(s + 1) % 3]);
        cl_sync();
        long *y = cu; cu = nw; nw = y;
    }
    for(long i = x0; i < m; i += CL*CT)
        keep[i].k[SQB_PFLAG] = (signed char)((keep[i].k[SQB_PFLAG] & 1) | (__ldcg(&tr[i]) << 1));
}
__global__ void k_tier_apply(sqb_pt_t *keep, const unsigned *tr, const gacc_t *acc){
    const long m = (long)acc->m;
    for(long i = blockIdx.x*(long)blockDim.x + threadIdx.x; i < m; i += (long)gridDim.x*blockDim.x)
        keep[i].k[SQB_PFLAG] = (signed char)((keep[i].k[SQB_PFLAG] & 1) | (tr[i] << 1));
}

/* the final threshold (eps times the whole sum) and the tiers; the kept list stays on the device, its length there
 * too (GR.nkeep bounds it until a wait) */
extern "C" int sqb_grow_finish(int tiers){
    const long n = GR.nkeep;
    {
        Tmp<sqb_pt_t> out; Tmp<double> okv; Tmp<u64> okk;
        if(out.get(n ? n : 1) || okv.get(n ? n : 1) || okk.get(n ? n : 1)) return -1;
        if(n){
            RethOp ro; ro.keep = GR.keep; ro.kv = GR.kv; ro.kk = GR.kk; ro.acc = GR.acc; ro.out = out.p; ro.okv = okv.p; ro.okk = okk.p; ro.base = 0;
            if(compact(ro, cnt_t{NULL, 1, n}, &GR.acc->m, GR.acc, NULL)) return -1;
        }
        hold(GR.keep, out.keep()); hold(GR.kv, okv.keep()); hold(GR.kk, okk.keep()); GR.keepcap = n ? n : 1;
    }
    if(!tiers || !n) return 0;
    Tmp<unsigned> tr_; Tmp<long> cu_, nw_; Tmp<u64> cnt_;
    if(tr_.get(n) || cu_.get(2*n) || nw_.get(2*n) || cnt_.get(3)) return -1;
    unsigned *const tr = tr_.p; long *cu = cu_.p, *nw = nw_.p; u64 *const cnt = cnt_.p;
    if(n <= TIER_CL){
        k_tiers<<<CL, CT, 0, TS>>>(GR.g, GR.keep, GR.kk, GR.key, GR.word, GR.mask, GR.kv, GR.acc, tr, cu, nw, cnt); TL++;
        TCK(cudaGetLastError());
        return 0;
    }
    TCK(cudaMemsetAsync(tr, 0, n*sizeof(unsigned), TS));
    k_index<<<grid256(n), 256, 0, TS>>>(GR.kk, GR.key, GR.word, GR.mask, GR.acc);
    k_tier_seed<<<1, 1, 0, TS>>>(GR.g, GR.key, GR.word, GR.mask, GR.kv, GR.acc, tr, cu, cnt);
    TL += 2;
    /* the points lie within as many steps of z = 0 as the grow had frontiers; a way through the larger values
     * alone may be longer, and the rest kernel walks it */
    int s = 0;
    for(; s < GR.nfrs; s++){
        k_tier_step<<<grid256(n), 256, 0, TS>>>(GR.g, GR.keep, GR.kk, GR.key, GR.word, GR.mask, GR.kv, GR.acc, tr, cu, nw, cnt, s); TL++;
        long *x = cu; cu = nw; nw = x;
    }
    k_tier_rest<<<1, GT, 0, TS>>>(GR.g, GR.keep, GR.kk, GR.key, GR.word, GR.mask, GR.kv, GR.acc, tr, cu, nw, cnt, s);
    k_tier_apply<<<grid256(n), 256, 0, TS>>>(GR.keep, tr, GR.acc);
    TL += 2;
    TCK(cudaGetLastError());
    return 0;
}
/* waits and reads the record: the grow's sums (S, a, x1, x2, dropped weight, signed sum below the threshold) and counts */
extern "C" int sqb_grow_sums(sqb_grow_sums_t *r){
    TCK(cudaMemcpyAsync(GR.host, GR.acc, sizeof(gacc_t), cudaMemcpyDeviceToHost, TS));
    TCK(cudaStreamSynchronize(TS));
    sqb_dev_count_copy(0, sizeof(gacc_t));
    const gacc_t &h = *GR.host;
    if(h.err){ snprintf(terr, sizeof terr, "grow: %llu table lookups failed", h.err); return -1; }
    r->S = h.S[0] + h.S[1]; r->a = h.a; r->x1 = h.x1[0] + h.x1[1]; r->x2 = h.x2[0] + h.x2[1]; r->drop = h.dr[0] + h.dr[1];
    r->gshs = h.gs[0] + h.gs[1]; r->gshn = (long)h.ngs; r->u = h.u[0] + h.u[1]; r->nq = (long)h.nq; r->unres = (long)h.unres;
    r->kept = (long)h.m; r->cells = (long)h.ncell; r->seen = (long)h.seen; r->frontiers = (long)h.steps;
    GR.nkeep = (long)h.m;
    return 0;
}

/* ------------------------------------------- dilation -------------------------------------------- */
/* every kept cell and its in-box axis neighbours marked in the seen table, which holds them all: bit 3 present,
 * bit 0 some cell does not skip (the skip bits' AND), bits 1 and 2 the tier's maximum in unary (driver/sumkey.h:41-44) */
__global__ void k_dil_mark(const __grid_constant__ geom_t g, const sqb_pt_t *cur, const u64 *kk, const u64 *key, unsigned *word, u64 mask, gacc_t *acc, unsigned *bm, u64 base){
    const int C = 2*g.D + 1;
    const long n = (long)acc->m*C;
    for(long x = blockIdx.x*(long)blockDim.x + threadIdx.x; x < n; x += (long)gridDim.x*blockDim.x){
        long q0; int c;
        split(x, C, &q0, &c);
        const signed char *k = cur[q0].k; const int fl = k[SQB_PFLAG];
        u64 y = kk[q0];
        if(c > 0){
            const int j = (c - 1) >> 1, sg = ((c - 1) & 1) ? 1 : -1, kx = k[j] + g.st*sg;
            if(kx > g.K || kx < -g.K) continue;
            y = sg > 0 ? y + g.P[j] : y - g.P[j];
        }
        const long q = h_find(key, mask, y);
        if(q < 0){ atomicAdd(&acc->err, 1ULL); continue; }
        const unsigned b = 8u | ((fl & 1) ? 0 : 1) | (((fl >> 1) & 3) >= 1 ? 2 : 0) | (((fl >> 1) & 3) >= 2 ? 4 : 0);
        if((*(volatile unsigned*)&word[q] & b) == b) continue;
        if(!(atomicOr(&word[q], b) & 8u) && bm) atomicOr(&bm[(y - base) >> 5], 1u << ((y - base) & 31));
    }
}
/* a grid of up to BM_BITS keys (W^D) in a bitmap: its set bits in order are the sorted cells, without a sort */
#define BM_BITS (1ULL << 29)
template<int I>
__global__ void __launch_bounds__(TG_T) k_bm_count(const uint4 *bm, long n4, unsigned *bcnt){
    __shared__ u64 ws[TG_T/32];
    u64 c = 0;
    for(int j = 0; j < I; j++){
        const long i = (blockIdx.x*(long)TG_T + threadIdx.x)*I + j;
        if(i < n4){ const uint4 x = bm[i]; c += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w); }
    }
    c = block_sum<TG_T>(c, ws);
    if(threadIdx.x == 0) bcnt[blockIdx.x] = (unsigned)c;
}
template<int I>
__global__ void __launch_bounds__(TG_T) k_bm_emit(const uint4 *bm, long n4, emit_t e, u64 base, u64 *out){
    __shared__ u64 ws[TG_T/32];
    u64 r;
    if(e.boff) r = e.boff[blockIdx.x];
    else {
        u64 s = 0;
        for(long j = threadIdx.x; j < (long)blockIdx.x; j += TG_T) s += e.bcnt[j];
        r = block_sum<TG_T>(s, ws);
    }
    const long i0 = (blockIdx.x*(long)TG_T + threadIdx.x)*I;
    u64 c = 0, t;
    for(int j = 0; j < I; j++) if(i0 + j < n4){ const uint4 x = bm[i0 + j]; c += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w); }
    u64 o = r + block_scan<TG_T>(c, ~0ULL, &t, ws);
    if(c) for(int j = 0; j < I; j++) if(i0 + j < n4){
        const uint4 x = bm[i0 + j];
        const unsigned w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for(int q = 0; q < 4; q++) for(unsigned b = w[q]; b; b &= b - 1) out[o++] = base + (u64)(i0 + j)*128 + q*32 + __ffs(b) - 1;
    }
    if(blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *e.tot = r + t;
}
template<int I> static int bm_order(const unsigned *bm, u64 bits, u64 base, u64 *out, u64 *tot){
    const long n4 = (long)((bits + 127)/128), nb = (n4 + TG_T*I - 1)/(TG_T*I);
    if(scratch(nb)) return -1;
    k_bm_count<I><<<(unsigned)nb, TG_T, 0, TS>>>((const uint4*)bm, n4, SC.bcnt);
    const bool scan = nb > OFFS_CTAS;
    if(scan){ k_scan<<<1, GT, 0, TS>>>(SC.bcnt, nb, SC.boff, NULL); TL++; }
    emit_t e = {SC.bcnt, scan ? SC.boff : NULL, nb, tot, NULL, NULL, NULL};
    k_bm_emit<I><<<(unsigned)nb, TG_T, 0, TS>>>((const uint4*)bm, n4, e, base, out);
    TL += 2;
    TCK(cudaGetLastError());
    return 0;
}
struct SlotOp {
    enum { DROP = 0, D2 = 0 };
    const u64 *key; const unsigned *word; u64 *out; u64 base;
    __device__ bool pred(long i) const { return word[i] != 0; }
    __device__ void emit(long i, u64 r) const { out[r] = key[i]; }
};
__global__ void k_dil_decode(const __grid_constant__ geom_t g, const u64 *U, const u64 *key, const unsigned *word, u64 mask, sqb_pt_t *out, const gacc_t *acc){
    const long m = (long)acc->ncell;
    for(long j = blockIdx.x*(long)blockDim.x + threadIdx.x; j < m; j += (long)gridDim.x*blockDim.x){
        u64 y = U[j]; sqb_pt_t p;
        for(int i = 0; i < SQB_MAXD; i++) p.k[i] = 0;
        for(int i = g.D - 1; i >= 0; i--){ p.k[i] = (signed char)((int)(y % g.W)*g.st - g.K); y /= g.W; }
        const long q = h_find(key, mask, U[j]);
        if(q >= 0){ const unsigned b = word[q]; p.k[SQB_PFLAG] = (signed char)(((b & 1) ? 0 : 1) | ((b & 4) ? 4 : (b & 2))); }
        out[j] = p;
    }
}

/* stable LSD radix sort of n 64-bit keys, nbits significant, 8-bit digits; result in *a (a, b swapped) */
#define RS_T 256
#define RS_I 16
#define RS_TILE (RS_T*RS_I)
__global__ void __launch_bounds__(RS_T) k_rs_hist(const u64 *a, cnt_t cn, int sh, unsigned *hist, long nblk){
    __shared__ unsigned h[256];
    const long n = cnt_of(cn);
    h[threadIdx.x] = 0; __syncthreads();
    const long t0 = blockIdx.x*(long)RS_TILE;
    for(int j = 0; j < RS_I; j++){ long i = t0 + j*RS_T + threadIdx.x; if(i < n) atomicAdd(&h[(a[i] >> sh) & 255], 1u); }
    __syncthreads();
    hist[(long)threadIdx.x*nblk + blockIdx.x] = h[threadIdx.x];
}
/* off: the counts' offsets within their digit, tot: the digits' counts.  One CTA that scanned all 256 nblk counts took 208 us
 * a pass for 4e6 keys, five times the scatter; a CTA per digit takes 5 */
__global__ void __launch_bounds__(RS_T) k_rs_scatter(const u64 *a, u64 *b, cnt_t cn, int sh, const u64 *off, const u64 *tot, long nblk){
    __shared__ u64 base[256], ws[RS_T/32];
    u64 all;
    __shared__ unsigned wc[RS_T/32][256];
    const long n = cnt_of(cn);
    static_assert(RS_T == 256, "a thread per digit");
    base[threadIdx.x] = off[(long)threadIdx.x*nblk + blockIdx.x] + block_scan<RS_T>(tot[threadIdx.x], ~0ULL, &all, ws);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const long t0 = blockIdx.x*(long)RS_TILE;
    for(int j = 0; j < RS_I; j++){
        if(t0 + j*RS_T >= n) break;
        for(int q = 0; q < RS_T/32; q++) wc[q][threadIdx.x] = 0;
        __syncthreads();
        const long i = t0 + j*RS_T + threadIdx.x;
        const bool in = i < n;
        const u64 x = in ? a[i] : 0;
        const unsigned dg = in ? (unsigned)((x >> sh) & 255) : 256u + l;   /* out-of-range lanes never match */
        const unsigned peers = __match_any_sync(0xffffffffu, dg);
        const unsigned lt = peers & ((1u << l) - 1);
        if(in && lt == 0) wc[w][dg] = __popc(peers);
        __syncthreads();
        if(in){
            u64 o = base[dg] + __popc(lt);
            for(int q = 0; q < w; q++) o += wc[q][dg];
            b[o] = x;
        }
        __syncthreads();
        unsigned s = 0; for(int q = 0; q < RS_T/32; q++) s += wc[q][threadIdx.x];
        base[threadIdx.x] += s;
        __syncthreads();
    }
}
static int radix_sort(u64 **a, u64 **b, cnt_t cn, int nbits){
    if(cn.max <= 1) return 0;
    const long nblk = (cn.max + RS_TILE - 1)/RS_TILE;
    Tmp<unsigned> hist_; Tmp<u64> off_;
    if(hist_.get(256*nblk) || off_.get(256*(nblk + 1))) return -1;
    unsigned *const hist = hist_.p; u64 *const off = off_.p;
    for(int sh = 0; sh < nbits; sh += 8){
        k_rs_hist<<<(unsigned)nblk, RS_T, 0, TS>>>(*a, cn, sh, hist, nblk);
        k_scan<<<256, GT, 0, TS>>>(hist, nblk, off, off + 256*nblk);
        k_rs_scatter<<<(unsigned)nblk, RS_T, 0, TS>>>(*a, *b, cn, sh, off, off + 256*nblk, nblk);
        TL += 3;
        TCK(cudaGetLastError());
        u64 *t = *a; *a = *b; *b = t;
    }
    return 0;
}
extern "C" int sqb_radix_sort_u64(unsigned long long *keys_dev, long n, int nbits, void *stream){
    TS = (cudaStream_t)stream;
    Tmp<u64> tmp;
    if(tmp.get(n ? n : 1)) return -1;
    u64 *b = tmp.p, *a = keys_dev;
    if(radix_sort(&a, &b, cnt_t{NULL, 1, n}, nbits)) return -1;
    if(a != keys_dev) TCK(cudaMemcpyAsync(keys_dev, a, n*sizeof(u64), cudaMemcpyDeviceToDevice, TS));
    TCK(cudaStreamSynchronize(TS));
    return 0;
}

/* the kept list (from sqb_grow_finish) and its axis neighbours at the top step, sorted, flags merged; *out is a device
 * list owned by the caller (sqb_dev_free), its length in sqb_grow_sums' record */
extern "C" int sqb_grow_dilate(int nbits, sqb_pt_t **out){
    *out = NULL;
    if(!GR.nkeep) return 0;
    const long cap = (long)GR.mask + 1, n = GR.nseen;
    Tmp<u64> U_, T_; Tmp<sqb_pt_t> o; Tmp<char> bm_;
    if(U_.get(n) || T_.get(n) || o.get(n)) return -1;
    u64 *U = U_.p, *T = T_.p;
    /* the keys are base ... 2 base - 1, base = W^D.  In key order by a bitmap where the grid is small (D = 5: every
     * lattice up to W = 55; 83,362 cells of 31^5: 33 us), else by a sort (about 60 us a pass of eight bits for 4e6 cells) */
    const u64 base = GR.g.P[0]*(u64)GR.g.W;
    unsigned *bm = NULL;
    const size_t bmb = (size_t)((base + 127)/128)*16;
    if(base <= BM_BITS){
        if(bm_.get((long)bmb)) return -1;
        bm = (unsigned*)bm_.p;
        TCK(cudaMemsetAsync(bm, 0, bmb, TS));
    }
    TCK(cudaMemsetAsync(GR.word, 0, cap*sizeof(unsigned), TS));
    k_dil_mark<<<grid256(GR.nkeep*(2*GR.g.D + 1)), 256, 0, TS>>>(GR.g, GR.keep, GR.kk, GR.key, GR.word, GR.mask, GR.acc, bm, base); TL++;
    if(bm){
        if(base <= 1ULL << 25 ? bm_order<1>(bm, base, base, U, &GR.acc->ncell) : bm_order<8>(bm, base, base, U, &GR.acc->ncell)) return -1;
    } else {
        SlotOp so; so.key = GR.key; so.word = GR.word; so.out = U; so.base = 0;
        if(compact(so, cnt_t{NULL, 1, cap}, &GR.acc->ncell, GR.acc, NULL)) return -1;
        if(radix_sort(&U, &T, cnt_t{&GR.acc->ncell, 1, n}, nbits)) return -1;
    }
    k_dil_decode<<<grid256(n), 256, 0, TS>>>(GR.g, U, GR.key, GR.word, GR.mask, o.p, GR.acc); TL++;
    TCK(cudaGetLastError());
    *out = o.keep();
    return 0;
}

/* the kept list after sqb_grow_finish (tiers in the flag byte), on the device; its length after a wait (sqb_grow_sums) */
extern "C" void sqb_grow_kept(const sqb_pt_t **keep, long *m){ *keep = GR.keep; *m = GR.nkeep; }

/* top = 0 keeps no list; the kept list is released with the table */
extern "C" void sqb_grow_end(void){
    hold(GR.key, (u64*)NULL); hold(GR.word, (unsigned*)NULL);
    hold(GR.keep, (sqb_pt_t*)NULL); hold(GR.kv, (double*)NULL); hold(GR.kk, (u64*)NULL);
    GR.nkeep = GR.keepcap = 0;
}
