/* sqkern.cuh -- the evaluation kernels, instantiated once per graph by the generated translation
 * unit (kgen output included after this header, then SQ_GRAPH(...) below).
 *
 * One thread per lattice point.  A point is a node (k given) or child b of a cell (k_d - st*bit_d(b),
 * in the order of prep() in the reference, driver/sum.c:405-408; children below the box, k_d < -K,
 * are not points).  The per-coordinate tables X[k+K] (the integration variable, s = e^{kh}) and
 * Wt[k+K] (its weight factor s*h) sit in shared memory; the weight is accumulated in coordinate order
 * as lattice_node() does (driver/lattice.c:30-34), so it rounds identically.
 *
 * FP64 pass (sqb_k_f64): f and the |.| sum in double.  Raw mode returns f*w and ab*w (the reference's
 * GPU plug-in contract, driver/gpu_kernel.h:22-36).  Test mode applies the reference's per-point tests
 * (finish(), driver/eval.c:33-53): skipped points keep f*w; otherwise the bound ab*w*16*eps/DDSLACK sets
 * the near flag and, above ABSERR, queues the point for the double-double pass.
 * DD pass (sqb_k_dd): the queued points (or all of them) in double-double, with qvalue()'s round
 * column and unresolved-point rule (driver/eval.c:25-30). */
#pragma once
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include "sqdd.cuh"
#include "sqb_internal.h"
#include "sqscale.cuh"
#include "sqorbit.cuh"

#ifndef SQG_NS
#define SQG_NS(n) sqg_##n                    /* the graph's namespace (sqgf_<name> in the contracted unit) */
#endif
#define SQ_TABLE static __constant__ const
#define SQ_FUNC __device__
#ifndef SQ_FUNC_K
#define SQ_FUNC_K __device__                    /* FP64 class: point functions (pt_, vp_, helpers); a graph's
                                                   unit may define it __forceinline__ */
#endif
#define SQ_CHUNK __device__ __forceinline__      /* FP64: chunk arguments stay in registers */
#define SQ_CHUNK_DD __device__ __noinline__     /* double-double: real calls bound the compile */
#define RABS(x) sq_rabs(x)
#define SQ_EXP(x) sq_exp(x)
#define SQ_LOG(x) sq_log(x)
#define SQ_AXIS_FORM                             /* the axis form of the integrands that have one is compiled */

#ifndef SQB_BLOCK
#define SQB_BLOCK 128
#endif
#ifndef SQB_MINB
#define SQB_MINB 1            /* FP64 kernel: resident blocks per SM the register allocation must allow */
#endif
#ifndef SQB_LEVEL_KERNEL
#ifdef SQB_FMA_TU
#define SQB_LEVEL_KERNEL 1    /* the contracted unit: a level kernel beside the general one, both calling the point
                                 function (sqb_fcall); the exact unit keeps one kernel with the function inlined */
#else
#define SQB_LEVEL_KERNEL 0
#endif
#endif
#ifndef SQB_SWEEPS
#define SQB_SWEEPS 1          /* level kernel: 2 = two sweeps over a batch's tiles, the children of cells that skip
                                 the |.| sums first, then the others, so that the CTAs on an SM run one form of a
                                 point function at a time (a large integrand's two forms do not fit the
                                 instruction caches together); the reduce kernel then sums every tile */
#endif
#ifndef SQB_FUSE
#define SQB_FUSE 1            /* FP64 kernel: level mode (tile sums in shared memory) compiled in; a kernel
                                 that spills its registers is built without it, keeping L1 for its stack */
#endif
#define SQB_QEPS 4.93e-32   /* double-double epsilon of the fallback's error model (driver/common.h:8) */
#ifndef SQB_TABLE_GLOBAL
#define SQB_TABLE_GLOBAL 0    /* FP64 pass: 1 = the lattice tables read through the read-only data cache instead of
                                 from the CTA's shared-memory copy */
#endif
#if SQB_TABLE_GLOBAL
#define SQB_TAB(p, j) __ldg((p) + (j))
#else
#define SQB_TAB(p, j) (p)[j]
#endif

/* The per-integral fields of a launch (sqb_inst_t) sit in shared memory: every thread of a CTA works on
 * one integral at a time.  A launch over one batch (ninst = 0) has one record, made from its own fields;
 * a multi-instance launch (ninst >= 1) has one per integral, with their tables side by side. */
__device__ __forceinline__ void sqb_inst_of(const sqb_eval_t &a, sqb_inst_t *I){
    I->pts = a.pts; I->n = a.n; I->child0 = 0; I->st = a.st; I->K = a.K; I->toff = 0; I->fused = 1;
    I->last = a.last; I->pw = a.pw; I->thr = a.thr; I->abserr = a.abserr; I->near_thr = a.near_thr;
    I->X = a.X; I->Wt = a.Wt; I->U = a.U; I->Ud = a.Ud;
}
/* the instance of global child index i (ninst >= 1): the last one whose range starts at or before i */
__device__ __forceinline__ int sqb_inst_at(const sqb_eval_t &a, long i){
    int k = 0;
    for(int q = 1; q < a.ninst; q++) if(a.inst[q].child0 <= i) k = q;
    return k;
}
/* the nodes or cells of a launch over one batch */
__device__ __forceinline__ long sqb_count(const sqb_eval_t &a){ return a.np ? (long)*a.np : a.n; }
/* shared-memory words of the tables of a launch: 2(2K+1) per integral */
__host__ __device__ __forceinline__ int sqb_table_words(const sqb_eval_t &a){
    if(a.ninst <= 0) return 2*(2*a.K + 1);
    int w = 0;
    for(int q = 0; q < a.ninst; q++) w += 2*(2*a.inst[q].K + 1);
    return w;
}

/* coordinates and weight of point il of integral I (ig: its index in the launch, the same for one batch);
 * returns 0 for a child below the box, a child the predictor leaves out or, under a symmetry fold, a child
 * that is not the minimum of its orbit (driver/sum.c:405-416), else the point's multiplicity (the orbit
 * size; 1 without a fold) */
template<int D, bool ORB = true, int LV = 0>
__device__ __forceinline__ int sqb_point(const sqb_eval_t &a, const sqb_inst_t &I, const double *sX, const double *sW,
                                         long il, long ig, long *cell, double *sf, double *w, int *ko = NULL){
    long c; int b;
    const bool cells = LV || a.cells;           /* the level kernel: cells of int8 coordinates */
    if(cells){ c = il >> D; b = (int)(il & ((1L << D) - 1)); } else { c = il; b = 0; }
    *cell = c;
    if(!LV && a.sfin){
#pragma unroll
        for(int d = 0; d < D; d++) sf[d] = a.sfin[ig*D + d];
        *w = 1.0;
        return 1;
    }
    double ww = 1.0; bool in = true;
    int kk[D];
    const int K = I.K, st = I.st;
    if(LV || a.esize == 1){
        const signed char *p = (const signed char*)I.pts + c*(long)a.stride;
#pragma unroll
        for(int d = 0; d < D; d++){
            int kd = p[d] - (((b >> d) & 1) ? st : 0);
            kk[d] = kd;
            if(kd < -K){ in = false; kd = -K; }
            if(ko) ko[d] = kd;
            sf[d] = SQB_TAB(sX, kd + K); ww = ww*SQB_TAB(sW, kd + K);
        }
    } else {
        const short *p = (const short*)I.pts + c*(long)a.stride;
#pragma unroll
        for(int d = 0; d < D; d++){
            int kd = p[d] - (((b >> d) & 1) ? st : 0);
            kk[d] = kd;
            if(kd < -K){ in = false; kd = -K; }
            if(ko) ko[d] = kd;
            sf[d] = SQB_TAB(sX, kd + K); ww = ww*SQB_TAB(sW, kd + K);
        }
    }
    *w = ww;
    if(!in) return 0;
    if(a.cfl && (a.cfl[ig] & 1)) return 0;          /* left out by the predictor */
    if constexpr(!ORB) return 1;               /* list mode: the select pass has the orbit weight */
    return cells && a.sym.n > 1 ? sqb_orbit<D>(a.sym, kk) : 1;
}

template<int D>
__device__ __forceinline__ int sqb_skip(const sqb_eval_t &a, const sqb_inst_t &I, long c){
    if(a.skip) return a.skip[c];
    if(a.flag_at >= 0 && a.abskip){
        int fl = a.esize == 1 ? ((const signed char*)I.pts)[c*(long)a.stride + a.flag_at]
                              : ((const short*)I.pts)[c*(long)a.stride + a.flag_at];
        return fl & 1;
    }
    return 0;
}

/* the launch's tables into shared memory (X then the weight factor Wt = X H when a batch has no Wt) and
 * the integral records: one batch (ninst = 0) fills sI[0] */
__device__ __forceinline__ void sqb_tables(const sqb_eval_t &a, double *sm, sqb_inst_t *sI){
    if(a.ninst <= 0){
        const int nt = 2*a.K + 1;
        for(int j = threadIdx.x; j < nt; j += blockDim.x){ sm[j] = a.X[j]; sm[nt + j] = a.Wt ? a.Wt[j] : a.X[j]*a.H; }
        if(threadIdx.x == 0) sqb_inst_of(a, &sI[0]);
    } else {
        for(int q = 0; q < a.ninst; q++){
            const sqb_inst_t &I = a.inst[q];
            const int nt = 2*I.K + 1;
            for(int j = threadIdx.x; j < nt; j += blockDim.x){ sm[I.toff + j] = I.X[j]; sm[I.toff + nt + j] = I.Wt[j]; }
        }
        if(threadIdx.x < a.ninst) sI[threadIdx.x] = a.inst[threadIdx.x];
    }
    __syncthreads();
}

/* the per-point tests of finish() (driver/eval.c:33-53) on the FP64 value fw = f w and |.| sum abw = ab w
 * of point i: skipped points keep fw; otherwise the bound abw 16 eps / DDSLACK sets the near flag and,
 * above ABSERR, queues the point for the double-double pass (value 0 until then).  Writes v[i] and
 * stt[i]; returns the value */
__device__ __forceinline__ double sqb_point_test(const sqb_eval_t &a, const sqb_inst_t &I, long i, int sk, bool noab,
                                                 double fw, double abw, bool *fallback){
    unsigned char s = SQB_PRESENT | (sk ? SQB_SKIPPED : 0);
    double v;
    *fallback = false;
    if(noab) v = isfinite(fw) ? fw : 0.0;
    else {
        double bnd = abw*16*DBL_EPSILON;
        if(a.ddslack != 1.0) bnd = bnd/a.ddslack;      /* x/1 = x: the default divides nothing */
        if(!(bnd <= I.near_thr)) s |= SQB_NEAR;
        if(!(bnd <= I.abserr)){
            s |= SQB_FALLBACK; v = 0.0; *fallback = true;
            const unsigned long long q = atomicAdd(a.nfb, 1ULL);
            if((long)q < a.fbcap) a.fb[q] = i;
        } else v = isfinite(fw) ? fw : 0.0;
    }
    a.v[i] = v; a.stt[i] = s;
    return v;
}

/* the tile's sums in level mode: thread t's running sums sit in shared memory (column t), out of the
 * registers that the integrand needs; at the tile's end warp 0 adds the columns in a fixed order */
#if SQB_FUSE
static_assert(SQB_BLOCK == SQB_TILE_THREADS, "the tile sums have one column per thread of the FP64 kernel's block");
#endif

__device__ __forceinline__ void sqb_acc_dd(double (*x)[SQB_BLOCK], int t, double y){
    const sqdd z = sqdd_add_d(sqdd(x[0][t], x[1][t]), y);
    x[0][t] = z.hi; x[1][t] = z.lo;
}

/* warp 0: the tile's sums in a fixed order (lane l adds columns l, l+32, l+64, l+96, then a shuffle
 * tree), written to part[tile]; the block's threads have synchronised before */
__device__ __forceinline__ void sqb_tile_flush(const sqb_eval_t &a, sqb_tile_acc &ta, long tile){
    if(threadIdx.x >= 32) return;
    const int l = threadIdx.x;
    sqdd S, b1, b2; double A = 0, dr = 0; unsigned ne = 0, nsk = 0, keep = 0;
    for(int q = l; q < SQB_BLOCK; q += 32){
        S = S + sqdd(ta.S[0][q], ta.S[1][q]); b1 = b1 + sqdd(ta.b1[0][q], ta.b1[1][q]); b2 = b2 + sqdd(ta.b2[0][q], ta.b2[1][q]);
        A += ta.A[q]; dr += ta.dr[q]; ne += ta.ne[q]; nsk += ta.nsk[q]; keep += ta.keep[q];
    }
    sqdd Ad(A), dd(dr);
    for(int off = 16; off; off >>= 1){
        S = S + sqdd(__shfl_down_sync(0xffffffffu, S.hi, off), __shfl_down_sync(0xffffffffu, S.lo, off));
        Ad = Ad + sqdd(__shfl_down_sync(0xffffffffu, Ad.hi, off), __shfl_down_sync(0xffffffffu, Ad.lo, off));
        dd = dd + sqdd(__shfl_down_sync(0xffffffffu, dd.hi, off), __shfl_down_sync(0xffffffffu, dd.lo, off));
        b1 = b1 + sqdd(__shfl_down_sync(0xffffffffu, b1.hi, off), __shfl_down_sync(0xffffffffu, b1.lo, off));
        b2 = b2 + sqdd(__shfl_down_sync(0xffffffffu, b2.hi, off), __shfl_down_sync(0xffffffffu, b2.lo, off));
        ne += __shfl_down_sync(0xffffffffu, ne, off); nsk += __shfl_down_sync(0xffffffffu, nsk, off);
        keep += __shfl_down_sync(0xffffffffu, keep, off);
    }
    if(l == 0){
        sqb_part_t p;
        p.S[0] = S.hi; p.S[1] = S.lo; p.A[0] = Ad.hi; p.A[1] = Ad.lo; p.drop[0] = dd.hi; p.drop[1] = dd.lo;
        p.b1[0] = b1.hi; p.b1[1] = b1.lo; p.b2[0] = b2.hi; p.b2[1] = b2.lo; p.u[0] = 0; p.u[1] = 0;
        p.ne = ne; p.nq = 0; p.unres = 0; p.skipped = nsk;
        a.part[tile] = p; a.tkeep[tile] = keep;
    }
}

/* The point function as a real call (contracted unit): its two forms (without and with the |.| sums) are
 * compiled as functions apart from the callers' loop state, so that the level kernel and the general one
 * share them instead of each inlining both (measured on the B200: as fast as the inlined function in the
 * level kernel). */
template<int D> struct sqb_pt { double s[D]; };
struct sqb_fab { double f, ab; };
template<class F, int D, int AB>
__device__ __noinline__ sqb_fab sqb_fcall(const sqb_pt<D> p){
    double sf[D];
#pragma unroll
    for(int d = 0; d < D; d++) sf[d] = p.s[d];
    sqb_fab r; r.ab = 0; r.f = F::template f<double, AB>(sf, &r.ab);
    return r;
}

/* ------------------------------------- the axis form --------------------------------------------------
 * An integrand that is a scan over its axes (kgen.axis_plan: class template KA) reads its functions of one
 * coordinate from a table over (axis, k) instead of evaluating them at every point: NU columns and the
 * reciprocals of the NR columns it divides by.  Entries in FP64: u then r, and in the lattice's table (PAD) the variable
 * and a word of padding if need be, so that the level kernel reads an entry by 16-byte loads; in double-double: (hi, lo)
 * of every column, then r. */
template<class R> struct sqb_axrow;
template<int SM> __device__ __forceinline__ double sqb_axld(const double *e){ if constexpr(SM) return *e; else return __ldg(e); }
template<> struct sqb_axrow<double> {
    static __device__ __forceinline__ void put(double *e, int c, double x){ e[c] = x; }
    template<int SM> static __device__ __forceinline__ double get(const double *e, int c){ return sqb_axld<SM>(e + c); }
    enum { W = 1 };
};
template<> struct sqb_axrow<sqdd> {
    static __device__ __forceinline__ void put(double *e, int c, const sqdd &x){ e[2*c] = x.hi; e[2*c + 1] = x.lo; }
    template<int SM> static __device__ __forceinline__ sqdd get(const double *e, int c){
        return sqdd(sqb_axld<SM>(e + 2*c), sqb_axld<SM>(e + 2*c + 1)); }
    enum { W = 2 };
};
template<class A, class R, int PAD = 0> struct sqb_axw {
    enum { E = A::NU*sqb_axrow<R>::W + A::NR, N = PAD && sqb_axrow<R>::W == 1 ? (E + 2)/2*2 : E };
};

/* entry j = axis (2K+1) + k + K of the table T over the variables X */
template<class A, class R, int PAD = 0>
__device__ __forceinline__ void sqb_axentry(const double *X, int nt, int j, double *T){
    R u[A::NU > 0 ? A::NU : 1];
    A::axis(j/nt, R(X[j % nt]), u);
    double *e = T + (long)j*sqb_axw<A, R, PAD>::N;
    if(PAD && sqb_axrow<R>::W == 1) e[sqb_axw<A, R>::E] = X[j % nt];
#pragma unroll
    for(int c = 0; c < A::NU; c++) sqb_axrow<R>::put(e, c, u[c]);
#pragma unroll
    for(int n = 0; n < A::NR; n++) e[A::NU*sqb_axrow<R>::W + n] = sqdd_rcp(u[A::rc(n)]);
}
/* the tables of one lattice, FP64 at T and double-double at Td: one thread per entry, the double-double ones (the
 * longer chains) in the first CTAs */
template<class A, class Ad, int D>
__global__ void __launch_bounds__(32) sqb_k_axis(const double *X, int K, double *T, double *Td){
    const int nt = 2*K + 1, n = D*nt, h = (n + 31)/32;
    const int j = (blockIdx.x % h)*32 + threadIdx.x;
    if(j >= n) return;
    if((int)blockIdx.x < h) sqb_axentry<Ad, sqdd, 1>(X, nt, j, Td);
    else sqb_axentry<A, double, 1>(X, nt, j, T);
}
/* one step of the scan from table entry e (SM: in shared memory) */
template<class A, class R, int SM = 0>
__device__ __forceinline__ void sqb_axstep(typename A::st &S, double si, const double *e){
    R u[A::NU > 0 ? A::NU : 1]; double r[A::NR > 0 ? A::NR : 1];
#pragma unroll
    for(int c = 0; c < A::NU; c++) u[c] = sqb_axrow<R>::template get<SM>(e, c);
#pragma unroll
    for(int n = 0; n < A::NR; n++) r[n] = sqb_axld<SM>(e + A::NU*sqb_axrow<R>::W + n);
    A::step(S, R(si), u, r);
}
/* the integrand at one point k (inside the box) from its table */
template<class A, class R, int D, int SM = 0>
__device__ __forceinline__ R sqb_axeval(const double *T, int K, const double *sf, const int *k, R *ab){
    typename A::st S;
    A::init(S);
    const int nt = 2*K + 1;
#pragma unroll
    for(int d = 0; d < D; d++) sqb_axstep<A, R, SM>(S, sf[d], T + (d*nt + k[d] + K)*(int)sqb_axw<A, R, !SM>::N);
    return A::fin(S, ab);
}
/* one step by the 16-byte loads of a padded entry, its quotients' tests put off (sqdd_flag) */
template<class A>
__device__ __forceinline__ void sqb_axstep_wide(typename A::st &S, const double *e, unsigned *bad){
    constexpr int E = sqb_axw<A, double, 1>::E;
    double x[E + 2];
#pragma unroll
    for(int c = 0; c <= E; c += 2){ const double2 y = __ldg((const double2*)(e + c)); x[c] = y.x; x[c + 1] = y.y; }
    A::template step<0>(S, x[E], x, x + A::NU, bad);
}
/* the point of cell w (a packed point) whose lower bits are low, with every quotient tested */
template<class A, int D>
__device__ __noinline__ sqb_fab sqb_ax_redo(const double *U, int K, int st, int w0, int w1, int w2, int low){
    constexpr int EW = sqb_axw<A, double, 1>::N;
    const int w[3] = {w0, w1, w2};
    typename A::st S;
    A::init(S);
#pragma unroll 1
    for(int d = 0; d < D; d++){
        const int k = (int)(signed char)(w[d >> 2] >> (8*(d & 3))) - (((low >> d) & 1) ? st : 0);
        const double *e = U + (d*(2*K + 1) + k + K)*EW;
        sqb_axstep<A, double>(S, e[sqb_axw<A, double>::E], e);
    }
    sqb_fab r; r.ab = 0; r.f = A::fin(S, &r.ab);
    return r;
}

/* The FP64 pass.  The CTAs take tiles of consecutive points in turn: tile b, b + gridDim.x, ... of one
 * batch, or, in a multi-instance launch, the next tile of the device counter queue (the tile's integral
 * from its position); SQB_TILE points per tile in level mode and in multi-instance launches, SQB_BLOCK
 * otherwise.  In a tile, thread t evaluates points t, t + SQB_BLOCK, ... (consecutive threads, consecutive
 * points).
 * In level mode (a.part) each CTA also sums the tiles of its integrals that it is asked to (sqb_inst_t
 * fused): the children that need no fallback add v*pw and the rest into the thread's column of shared
 * memory; a tile with a fallback point is flagged (a.tfb = 2), and the reduce kernel adds those points after the
 * double-double pass; a tile of an integral that the reduce kernel sums is only flagged (a.tfb = 1).
 * LV = 1 is the level kernel: the same pass compiled for level batches alone (cells of int8 coordinates,
 * tiles from the device queue, no list, no plain-form output), which leaves the other modes' code out of
 * the kernel that runs almost every point (measured 3-4 % faster on the three-loop graphs); with
 * SQB_SWEEPS = 2 it takes every tile twice, first for the children of cells that skip the |.| sums, then
 * for the others.  LV = 0 runs every other launch. */
template<class F, int D, int LV = 0>
__global__ void __launch_bounds__(SQB_BLOCK, SQB_MINB) sqb_k_f64(const __grid_constant__ sqb_eval_t a){
    extern __shared__ double sqb_sm[];
    __shared__ sqb_inst_t sI[SQB_MAXINST];
    __shared__ long s_tile;
    __shared__ int s_k;
#if SQB_FUSE
    /* the tile sums' columns follow the tables in dynamic shared memory (level launches only) */
    sqb_tile_acc &ta = *(sqb_tile_acc*)(sqb_sm + sqb_table_words(a));
    const bool lvl = LV || a.part != NULL;
#else
    const bool lvl = false;
#endif
    constexpr int NSW = LV ? SQB_SWEEPS : 1;
    sqb_tables(a, sqb_sm, sI);
    const bool multi = LV || a.ninst > 0;
    const bool list = !LV && a.sel;
    const long n1 = multi ? 0 : sqb_count(a) << (a.cells ? D : 0);  /* one batch: its points */
    const long tl = (lvl || multi) ? SQB_TILE : SQB_BLOCK;          /* other modes: one point per thread per step */
    const long nsel = list ? (long)*a.nsel : 0;                     /* list mode (one integral, queue): its entries */
    const long ntiles = list ? (nsel + tl - 1)/tl : multi ? a.ntile : (n1 + tl - 1)/tl;
    const int t = threadIdx.x;
    long q = blockIdx.x;                                            /* the work item: sweep*ntiles + tile */
    if(multi){ if(t == 0) s_tile = (long)atomicAdd(a.queue, 1ULL); __syncthreads(); q = s_tile; }
    while(q < NSW*ntiles){
        const int sweep = NSW > 1 ? (int)(q/ntiles) : 0;
        const long tile = NSW > 1 ? q - sweep*ntiles : q;
        int k = 0;
        if(multi){ if(t == 0) s_k = sqb_inst_at(a, tile*tl); __syncthreads(); k = s_k; }
        const sqb_inst_t &I = sI[k];
#if SQB_TABLE_GLOBAL
        const double *sX = I.X, *sW = I.Wt;
#else
        const double *sX = sqb_sm + I.toff, *sW = sX + (2*I.K + 1);
#endif
        const long base = multi ? tile*tl - I.child0 : tile*tl;     /* the tile's first point in its integral */
        const long n = multi ? ((LV || a.cells) ? (I.n << D) : I.n) : n1;
        const long off = multi ? I.child0 : 0;                       /* global index = local index + off */
#if SQB_FUSE
        const bool tsum = lvl && I.fused && !list && NSW == 1;
        if(tsum){
            ta.S[0][t] = ta.S[1][t] = ta.A[t] = ta.dr[t] = ta.b1[0][t] = ta.b1[1][t] = ta.b2[0][t] = ta.b2[1][t] = 0;
            ta.ne[t] = ta.nsk[t] = ta.keep[t] = 0;
            if(t == 0) ta.fb = 0;
            __syncthreads();
        }
#else
        const bool tsum = false;
#endif
        for(int j = 0; j < tl/SQB_BLOCK; j++){
            long il, i; int mw;
            long c; double sf[D], w;
            if(list){
                const long e_ = tile*tl + (long)j*SQB_BLOCK + t;
                if(e_ >= nsel) break;
                const unsigned long long e = a.sel[e_];
                il = i = (long)(e & ((1ULL << SQB_SEL_SHIFT) - 1));
                sqb_point<D, false, LV>(a, I, sX, sW, il, i, &c, sf, &w);
                mw = (int)(e >> SQB_SEL_SHIFT);
            } else {
                il = base + (long)j*SQB_BLOCK + t; i = il + off;
                if(il >= n) break;
                /* two sweeps: this child only in its cell's sweep (0: skips the |.| sums, 1: the others) */
                if(NSW > 1 && (sqb_skip<D>(a, I, il >> D) ? 0 : 1) != sweep) continue;
                mw = sqb_point<D, true, LV>(a, I, sX, sW, il, i, &c, sf, &w);
            }
            if(!mw){
                a.v[i] = 0;
                if(!LV && a.raw) a.ab[i] = 0; else a.stt[i] = 0;
                continue;
            }
            const int sk = sqb_skip<D>(a, I, c);
            const bool noab = sk && !a.abcheck;
            double ab = 0, f;
#if SQB_LEVEL_KERNEL
            {
                sqb_pt<D> p;
#pragma unroll
                for(int d = 0; d < D; d++) p.s[d] = sf[d];
                const sqb_fab r = noab ? sqb_fcall<F, D, 0>(p) : sqb_fcall<F, D, 1>(p);
                f = r.f; ab = r.ab;
            }
#else
            if(noab) f = F::template f<double, 0>(sf, &ab);
            else     f = F::template f<double, 1>(sf, &ab);
#endif
            const double fw = f*w;
            if(!LV && a.raw){ a.v[i] = fw; a.ab[i] = ab*w; continue; }
            bool fallback;
            const double v = sqb_point_test(a, I, i, sk, noab, fw, ab*w, &fallback);
#if SQB_FUSE
            if(tsum){
                if(fallback){ ta.fb = 1; continue; }
                /* a folded point stands for its orbit: (mw v) pw and mw |v| (driver/sum.c:734-745) */
                const double m = (double)mw, vp = (m*v)*I.pw, av = fabs(v);
                sqb_acc_dd(ta.S, t, vp); ta.A[t] += m*av; ta.ne[t]++; ta.nsk[t] += sk ? 1 : 0;
                if(I.last){
                    const int te = a.cfl ? (a.cfl[i] >> 1) & 3
                                         : (((const signed char*)I.pts)[c*(long)a.stride + a.flag_at] >> 1) & 3;
                    if(te >= 1) sqb_acc_dd(ta.b1, t, vp);
                    if(te >= 2) sqb_acc_dd(ta.b2, t, vp);
                } else if(av >= I.thr) ta.keep[t] += mw;
                else ta.dr[t] += (m*av)*I.pw;
            }
#else
            (void)fallback;
#endif
        }
#if SQB_FUSE
        if(tsum){
            __syncthreads();
            sqb_tile_flush(a, ta, tile);
            if(t == 0) a.tfb[tile] = ta.fb ? 2 : 0;
            __syncthreads();
        } else
#endif
        if(multi && a.tfb && !list && t == 0) a.tfb[tile] = 1;       /* summed by the reduce kernel */
        if(multi){
            __syncthreads();                                          /* every thread has read s_tile, s_k */
            if(t == 0) s_tile = (long)atomicAdd(a.queue, 1ULL);
            __syncthreads();
            q = s_tile;
        } else q += gridDim.x;
    }
}

/* qvalue() (driver/eval.c:25-30) on a point's double-double value and |.| sum: the value, the round column's e^2 and the
 * status s with the unresolved bit */
__device__ __forceinline__ double sqb_dd_value(double vqd, double abqd, double w, double abserr, int dropunres, double *u, unsigned char *s){
    const double ee = abqd*w*SQB_QEPS;
    *u = !(ee*16 <= abserr) ? (isfinite(ee) ? ee*ee : 0.0) : 0.0;
    double v = isfinite(vqd) ? vqd*w : 0.0;
    if(!(ee <= fabs(v))){ *s |= SQB_UNRES; if(dropunres) v = 0.0; }
    return v;
}

/* The axis form's kernel for launches outside the level batches: one batch of nodes or cells, tested or raw.  SM = 0 reads
 * the table at a.U; SM = 1 (the plug-in's launches, which have no table) fills one in shared memory per CTA first,
 * which pays from SQB_AX_RAW points on (sqb_ax_points).  DDI = 1: a point that needs the fallback is recomputed in
 * double-double at once, by its own thread (a.inl: a small launch, whose time is latency; the queue and the second
 * kernel would only add to it). */
template<class F, int D, int SM, int DDI>
__global__ void __launch_bounds__(SQB_BLOCK) sqb_k_ax(const __grid_constant__ sqb_eval_t a){
    extern __shared__ double sqb_sm[];
    __shared__ sqb_inst_t sI[SQB_MAXINST];
    using A0 = typename F::template AX<double, 0>;
    using A1 = typename F::template AX<double, 1>;
    const long n = sqb_count(a) << (a.cells ? D : 0);
    if(blockIdx.x*(long)SQB_BLOCK >= n) return;
    sqb_tables(a, sqb_sm, sI);
    const sqb_inst_t &I = sI[0];
    const int nt = 2*a.K + 1;
    const double *sX = sqb_sm, *sW = sqb_sm + nt;
    double *T = sqb_sm + 2*nt;
    if constexpr(SM){
        for(int j = threadIdx.x; j < D*nt; j += SQB_BLOCK) sqb_axentry<A0, double>(sX, nt, j, T);
        __syncthreads();
    }
    const double *U = SM ? T : a.U;
    for(long i = blockIdx.x*(long)SQB_BLOCK + threadIdx.x; i < n; i += (long)gridDim.x*SQB_BLOCK){
        long c; double sf[D], w; int kk[D];
        if(!sqb_point<D>(a, I, sX, sW, i, i, &c, sf, &w, kk)){
            a.v[i] = 0;
            if(a.raw) a.ab[i] = 0; else a.stt[i] = 0;
            continue;
        }
        const int sk = sqb_skip<D>(a, I, c);
        const bool noab = sk && !a.abcheck;
        double ab = 0, f;
        if(noab) f = sqb_axeval<A0, double, D, SM>(U, a.K, sf, kk, &ab);
        else     f = sqb_axeval<A1, double, D, SM>(U, a.K, sf, kk, &ab);
        const double fw = f*w;
        if(a.raw){ a.v[i] = fw; a.ab[i] = ab*w; continue; }
        if constexpr(DDI){
            /* sqb_point_test with the fallback in place of the queue */
            unsigned char s = SQB_PRESENT | (sk ? SQB_SKIPPED : 0);
            double v = isfinite(fw) ? fw : 0.0;
            if(!noab){
                double bnd = ab*w*16*DBL_EPSILON;
                if(a.ddslack != 1.0) bnd = bnd/a.ddslack;
                if(!(bnd <= I.near_thr)) s |= SQB_NEAR;
                if(!(bnd <= I.abserr)){
                    s |= SQB_FALLBACK;
                    sqdd abq;
                    const sqdd vq = sqb_axeval<typename F::template AX<sqdd, 1>, sqdd, D>(a.Ud, a.K, sf, kk, &abq);
                    double u;
                    v = sqb_dd_value(vq.value(), abq.value(), w, I.abserr, a.dropunres, &u, &s);
                    a.uu[i] = u;
                }
            }
            a.v[i] = v; a.stt[i] = s;
        } else {
            bool fallback;
            sqb_point_test(a, I, i, sk, noab, fw, ab*w, &fallback);
        }
    }
}

/* The axis form's level kernel (sqb_axis_launch).  The general kernel is bound by the FP64 pipe with the
 * integrand's exponentials and logarithms (syn_d8: 25 a point, 710 FP64 instructions); here one exponential a
 * point is left.  A thread takes the eight children of a cell that agree in
 * the first D - 3 axes: it scans those axes once, then the last three as a binary tree, so that a child costs
 * under two and a half steps of the scan instead of D.  Thread t of a tile takes groups t, t + SQB_BLOCK, ... in
 * order of (cell, first axes): a warp's writes for one choice of the last axes are 2^(D-3) consecutive
 * children.  A group's sums stay in registers and are added to the thread's column in shared memory.  Every child's
 * value is the general kernel's bit for bit; the tile sums add the same values in another fixed order.
 * Measured on the B200, whole last level against the general kernel: syn_d8 at h = 0.7 (1.18e9 children) 125.4 -> 12.6 ms,
 * syn_d11 at h = 2 (9.2e8) 93.6 -> 9.5 ms, syn_d5 at h = 1 (2.7e6) 0.40 -> 0.11 ms; this kernel 8.5 ps a child of syn_d8.
 * What bounds it is the number of instructions, two thirds of them not FP64, and the code's size (46 KB; 52 KB ran 5 %
 * longer, 137 KB 2.8 times as long where both forms of the leaf run).  In batches of 2^25 children, syn_d8 at h = 0.7: the
 * quotients' tests put off to one per child (sqdd_flag), wide table loads and rolled tile sums took 13.6 -> 11.9 ms, a warp per sum at the tile's end
 * instead of every thread for all of them 11.9 -> 11.4, groups counted in 32 bits 11.3 -> 11.25.  Five CTAs an SM
 * (96 registers, 24 bytes spilled); six 0.2 ms more, seven the same as six.  Sharing the step along axis D - 3 between
 * two turns of the loop took 11.8, the first axes' loop rolled 11.8. */
#define SQB_AXG 8
#ifndef SQB_AX_MINB
#define SQB_AX_MINB 5
#endif
/* an integral's fields: of the launch's arguments (one integral: constant memory, no registers), or read once per tile (in
 * shared memory every store to global memory would have them read again) */
struct sqb_ax_in { const double *U, *sX, *sW; int K, st; bool tsum; double pw, thr, abserr, near_thr, slack; };

template<class F, int D, int AB, int LAST>
__device__ __forceinline__ void sqb_ax_group(const sqb_eval_t &a, const sqb_ax_in &I, const int *w3, const int *k, int low, int sk, int tier, long i0,
                                             sqb_tile_acc &ta, bool &fb){
    using A = typename F::template AX<double, AB>;
    constexpr int M = D - 3, EW = sqb_axw<A, double, 1>::N;
    const int K = I.K, st = I.st, nt = 2*K + 1;
    /* the axes along which the lower child lies below the box; its coordinate is clamped, and the children with such a
     * bit are no points */
    int out = 0;
#pragma unroll
    for(int d = 0; d < D; d++) out |= (k[d] - st < -K) << d;
    typename A::st S0;
    A::init(S0);
    double w0 = 1.0; unsigned bad0 = 0;
#pragma unroll
    for(int d = 0; d < M; d++){
        const int kd = max(k[d] + K - ((low >> d) & 1)*st, 0);
        sqb_axstep_wide<A>(S0, I.U + (d*nt + kd)*EW, &bad0);
        w0 = w0*I.sW[kd];
    }
    const bool keepv = !LAST || !I.tsum;         /* the last level's summed tiles need no values but the fallback's, which the
                                                    double-double pass writes: 9.7 -> 9.5 ms of syn_d11's last level at h = 2 */
    double *const v = a.v + i0; unsigned char *const stt = a.stt + i0;
    const unsigned char s0 = SQB_PRESENT | (sk ? SQB_SKIPPED : 0);
    /* the group's sums: S as (hi, running error), |v|, the dropped weight; its children added and kept */
    double S = 0, Se = 0, Ag = 0, dr = 0; unsigned added = 0, kept = 0;
    int kx[3], dx[3];                                          /* the last axes' upper entries and the steps to the lower */
#pragma unroll
    for(int q = 0; q < 3; q++){ kx[q] = k[M + q] + K; dx[q] = min(kx[q], st); }
    /* rolled, for the code's size */
#pragma unroll 1
    for(int h = 0; h < 4; h++){
        typename A::st S1 = S0; double w1 = w0; unsigned bad1 = bad0;
#pragma unroll
        for(int q = 0; q < 2; q++){
            const int kd = kx[q] - ((h >> q) & 1)*dx[q];
            sqb_axstep_wide<A>(S1, I.U + ((M + q)*nt + kd)*EW, &bad1);
            w1 = w1*I.sW[kd];
        }
        double fw[2], abw[2];
#pragma unroll
        for(int b = 0; b < 2; b++){
            const int kd = b ? kx[2] - dx[2] : kx[2];
            typename A::st S2 = S1; unsigned bad = bad1;
            sqb_axstep_wide<A>(S2, I.U + ((D - 1)*nt + kd)*EW, &bad);
            const double w = w1*I.sW[kd];
            double ab = 0, f = A::template fin<0>(S2, &ab, &bad);
            if(sqdd_bad(bad)){
                const int lo = low | (h + 4*b) << M;
                if(!(lo & out)){
                    const sqb_fab r = sqb_ax_redo<A, D>(I.U, K, st, w3[0], w3[1], w3[2], lo);
                    f = r.f; ab = r.ab;
                }
            }
            fw[b] = f*w; abw[b] = ab*w;
        }
#pragma unroll
        for(int b = 0; b < 2; b++){
            const int o = (h + 4*b) << M;
            if((low | o) & out){ if(keepv) v[o] = 0; stt[o] = 0; continue; }
            /* finish()'s tests, as sqb_point_test */
            unsigned char s = s0; bool fallback = false;
            double x = isfinite(fw[b]) ? fw[b] : 0.0;
            if(AB){
                double bnd = abw[b]*16*DBL_EPSILON;
                if(I.slack != 1.0) bnd = bnd/I.slack;              /* x/1 = x: the default divides nothing */
                if(!(bnd <= I.near_thr)) s |= SQB_NEAR;
                if(!(bnd <= I.abserr)){
                    s |= SQB_FALLBACK; x = 0.0; fallback = true;
                    const unsigned long long q = atomicAdd(a.nfb, 1ULL);
                    if((long)q < a.fbcap) a.fb[q] = i0 + o;
                }
            }
            if(keepv) v[o] = x;
            stt[o] = s;
            if(!I.tsum) continue;
            if(fallback){ fb = true; continue; }
            const double vp = x*I.pw, av = fabs(x);
            const sqdd z = sqdd_two_sum(S, vp);
            S = z.hi; Se = SQ_ADD(Se, z.lo); Ag += av; added++;
            if(!LAST){ if(av >= I.thr) kept++; else dr += av*I.pw; }
        }
    }
    if(!I.tsum) return;
    /* into the thread's column; a cell's children share its shadow tier */
    const int t = threadIdx.x;
    const auto add = [&](double (*c)[SQB_TILE_THREADS]){        /* (hi, running error) again, normalised at the tile's end */
        const sqdd y = sqdd_two_sum(c[0][t], S);
        c[0][t] = y.hi; c[1][t] = SQ_ADD(c[1][t], SQ_ADD(y.lo, Se)); };
    add(ta.S);
    ta.A[t] += Ag; ta.ne[t] += added; ta.nsk[t] += sk ? added : 0;
    if(LAST){ if(tier >= 1) add(ta.b1); if(tier >= 2) add(ta.b2); }
    else { ta.dr[t] += dr; ta.keep[t] += kept; }
}

template<class F, int D, int LAST, int MULTI>
__global__ void __launch_bounds__(SQB_BLOCK, SQB_AX_MINB) sqb_k_lvax(const __grid_constant__ sqb_eval_t a){
    extern __shared__ double sqb_sm[];
    __shared__ sqb_inst_t sI[SQB_MAXINST];
    __shared__ long s_item;
    constexpr int M = D - 3;
    sqb_tile_acc &ta = *(sqb_tile_acc*)(sqb_sm + sqb_table_words(a));      /* the tile sums' columns follow the tables */
    sqb_tables(a, sqb_sm, sI);
    const int t = threadIdx.x, sub = a.sub > 1 ? a.sub : 1;
    const int gper = SQB_TILE/SQB_AXG/sub;                     /* groups per work item */
    for(;;){
        __syncthreads();                                       /* every thread has read s_item and the columns */
        if(t == 0) s_item = (long)atomicAdd(a.queue, 1ULL);
        __syncthreads();
        const long item = s_item;
        if(item >= a.ntile*sub) break;
        const long tile = item/sub;
        const sqb_inst_t &I = MULTI ? sI[sqb_inst_at(a, tile*SQB_TILE)] : a.inst[0];
        const double *sX = sqb_sm + I.toff, *sW = sX + (2*I.K + 1);
        const bool tsum = I.fused != 0;
        const sqb_ax_in in = {I.U, sX, sW, I.K, I.st, tsum, I.pw, I.thr, I.abserr, I.near_thr, a.ddslack};
        const int *const pts = (const int*)I.pts;
        const long ncell = I.n, child0 = I.child0;
        const long g0 = (tile*SQB_TILE - child0)/SQB_AXG + (item - tile*sub)*gper, c0 = g0 >> M;
        /* the item's first cell and, from there on, the groups in 32 bits */
        const int f0 = (int)(g0 & ((1 << M) - 1)), left = (int)min(ncell - c0, (long)SQB_TILE);
        const int *const src0 = pts + c0*3;
        const long at0 = (c0 << D) + child0;
        bool fbt = false;
        if(tsum){
            ta.S[0][t] = ta.S[1][t] = ta.A[t] = ta.dr[t] = ta.b1[0][t] = ta.b1[1][t] = ta.b2[0][t] = ta.b2[1][t] = 0;
            ta.ne[t] = ta.nsk[t] = ta.keep[t] = 0;
        }
        for(int j = t; j < gper; j += SQB_BLOCK){
            const int c = (f0 + j) >> M;
            if(c >= left) break;
            const int low = (f0 + j) & ((1 << M) - 1);
            const int *src = src0 + c*3;
            const int w3[3] = {src[0], src[1], src[2]};
            int k[D];
#pragma unroll
            for(int d = 0; d < D; d++) k[d] = (int)(signed char)(w3[d >> 2] >> (8*(d & 3)));
            const int fl = w3[2] >> 24;
            const int sk = a.abskip && (fl & 1);
            const long i0 = at0 + (((long)c << D) + low);
            if(sk && !a.abcheck) sqb_ax_group<F, D, 0, LAST>(a, in, w3, k, low, sk, (fl >> 1) & 3, i0, ta, fbt);
            else                 sqb_ax_group<F, D, 1, LAST>(a, in, w3, k, low, sk, (fl >> 1) & 3, i0, ta, fbt);
        }
        const int fb = __syncthreads_or(tsum && fbt);
        if(!tsum){ if(t == 0) a.tfb[tile] = 1; continue; }             /* summed by the reduce kernel */
        /* warp q sums the columns of the q-th sum and count; small code, which matters here (32 children a thread and tile) */
        const int q = t >> 5, l = t & 31;
        sqb_part_t &P = a.part[tile];
        {
            const double *hi = q == 0 ? ta.S[0] : q == 1 ? ta.A : q == 2 ? (LAST ? ta.b1[0] : ta.dr) : ta.b2[0];
            const double *lo = q == 0 ? ta.S[1] : q == 2 ? ta.b1[1] : ta.b2[1];
            const bool one = q == 1 || (!LAST && q == 2);          /* |v| and the dropped weight: plain sums */
            sqdd z;
#pragma unroll 1
            for(int c = l; c < SQB_BLOCK; c += 32) z = z + sqdd_two_sum(hi[c], one ? 0.0 : lo[c]);
#pragma unroll 1
            for(int off = 16; off; off >>= 1) z = z + sqdd(__shfl_down_sync(0xffffffffu, z.hi, off), __shfl_down_sync(0xffffffffu, z.lo, off));
            if(l == 0){
                double *dst = q == 0 ? P.S : q == 1 ? P.A : q == 2 ? (LAST ? P.b1 : P.drop) : P.b2;
                dst[0] = z.hi; dst[1] = z.lo;
            }
        }
        if(q < 3){
            const unsigned *col = q == 0 ? ta.ne : q == 1 ? ta.nsk : ta.keep;
            const unsigned n = __reduce_add_sync(0xffffffffu, col[l] + col[l + 32] + col[l + 64] + col[l + 96]);
            if(l == 0){
                if(q == 0) P.ne = n; else if(q == 1) P.skipped = n; else a.tkeep[tile] = n;
            }
        } else if(l == 0){
            double *none = LAST ? P.drop : P.b1;
            none[0] = none[1] = P.u[0] = P.u[1] = 0; P.nq = 0; P.unres = 0; a.tfb[tile] = fb ? 2 : 0;
        }
    }
}
static_assert(SQB_BLOCK == 128, "the tile sums of sqb_k_lvax: four warps");

template<class F, int D>
__global__ void __launch_bounds__(SQB_BLOCK) sqb_k_dd(const __grid_constant__ sqb_dd_t a){
    extern __shared__ double sqb_sm[];
    __shared__ sqb_inst_t sI[SQB_MAXINST];
    const sqb_eval_t &e = a.e;
    const bool multi = e.ninst > 0;
    long n;
    if(a.all) n = multi ? e.ntile*SQB_TILE : sqb_count(e) << (e.cells ? D : 0);
    else { n = (long)*a.nlist; if(n > a.listcap) n = a.listcap; }
    if(blockIdx.x*(long)blockDim.x >= n) return;      /* the grid is for a full queue: most queues are short */
    sqb_tables(e, sqb_sm, sI);
    for(long j = blockIdx.x*(long)blockDim.x + threadIdx.x; j < n; j += (long)gridDim.x*blockDim.x){
        const long i = a.all ? j : a.list[j];
        const int k = multi ? sqb_inst_at(e, i) : 0;
        const sqb_inst_t &I = sI[k];
        const double *sX = sqb_sm + I.toff, *sW = sX + (2*I.K + 1);
        const long il = i - I.child0;
        if(multi && il >= (e.cells ? (I.n << D) : I.n)) continue;    /* a tile's padding: no point */
        long c; double sf[D], w;
        using A = typename F::template AX<sqdd, 1>;
        [[maybe_unused]] int kk[D];
        if(!sqb_point<D>(e, I, sX, sW, il, i, &c, sf, &w, A::NU > 0 ? kk : NULL)){ e.v[i] = 0; e.stt[i] = 0; a.uu[i] = 0; continue; }
        sqdd abq, vq;
        bool tab = false;
        if constexpr(A::NU > 0) if(I.Ud){ tab = true; vq = sqb_axeval<A, sqdd, D>(I.Ud, I.K, sf, kk, &abq); }
        if(!tab){
            sqdd sq[D];
#pragma unroll
            for(int d = 0; d < D; d++) sq[d] = sqdd(sf[d]);
            vq = F::template f<sqdd, 1>(sq, &abq);
        }
        if(e.raw){ const long o = i*e.raw; e.v[o] = vq.hi; e.vlo[o] = vq.lo; e.ab[o] = abq.hi; e.ablo[o] = abq.lo; continue; }
        const double vqd = vq.value(), abqd = abq.value();
        unsigned char s;
        if(a.all){
            /* the all-double-double form: the near flag from the double-double |.| sum */
            s = SQB_PRESENT | SQB_FALLBACK | (sqb_skip<D>(e, I, c) ? SQB_SKIPPED : 0);
            if(!(abqd*w*16*DBL_EPSILON/e.ddslack <= I.near_thr)) s |= SQB_NEAR;
        } else s = e.stt[i];
        double u;
        const double v = sqb_dd_value(vqd, abqd, w, I.abserr, a.dropunres, &u, &s);
        e.v[i] = v; e.stt[i] = s; a.uu[i] = u;
    }
}

/* A graph whose point function is a flat sum of independent forest nodes (kgen.split_plan: g3_lbl) can
 * run the FP64 pass of a level batch as NP passes and a final one.  Pass P evaluates the nodes of group P
 * at every point and adds their contributions to the point's running (tot, tota) in tt[i], ta[i]; the
 * final pass applies f_'s own arithmetic to them and the tests of finish().  The operations and their
 * order are those of the single function, so the values are the same; each pass's code is a fraction of
 * the whole, which fits the instruction caches (the single kernel of g3_lbl waits on instruction fetch). */
template<class F, int D, int P>
__global__ void __launch_bounds__(SQB_BLOCK) sqb_k_part(const sqb_eval_t a, double *tt, double *ta){
    extern __shared__ double sqb_sm[];
    __shared__ sqb_inst_t sI[1];
    sqb_tables(a, sqb_sm, sI);                       /* one batch (ninst = 0) */
    const sqb_inst_t &I = sI[0];
    const double *sX = sqb_sm, *sW = sqb_sm + (2*a.K + 1);
    const long n = a.cells ? (a.n << D) : a.n;
    for(long i = blockIdx.x*(long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x*blockDim.x){
        long c; double sf[D], w;
        if(!sqb_point<D>(a, I, sX, sW, i, i, &c, sf, &w)) continue;
        const int sk = sqb_skip<D>(a, I, c);
        double T = P ? tt[i] : 0.0, A = P ? ta[i] : 0.0;
        if(sk && !a.abcheck) F::template part<P, 0>(sf, &T, &A);
        else                 F::template part<P, 1>(sf, &T, &A);
        tt[i] = T; ta[i] = A;
    }
}

template<class F, int D>
__global__ void __launch_bounds__(SQB_BLOCK) sqb_k_fin(const sqb_eval_t a, const double *tt, const double *ta){
    extern __shared__ double sqb_sm[];
    __shared__ sqb_inst_t sI[1];
    sqb_tables(a, sqb_sm, sI);                       /* one batch (ninst = 0) */
    const sqb_inst_t &I = sI[0];
    const double *sX = sqb_sm, *sW = sqb_sm + (2*a.K + 1);
    const long n = a.cells ? (a.n << D) : a.n;
    for(long i = blockIdx.x*(long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x*blockDim.x){
        long c; double sf[D], w;
        if(!sqb_point<D>(a, I, sX, sW, i, i, &c, sf, &w)){ a.v[i] = 0; a.stt[i] = 0; continue; }
        const int sk = sqb_skip<D>(a, I, c);
        const bool noab = sk && !a.abcheck;
        double ab = 0, f;
        if(noab) f = F::template fin<0>(sf, tt[i], ta[i], &ab);
        else     f = F::template fin<1>(sf, tt[i], ta[i], &ab);
        bool fallback;
        sqb_point_test(a, I, i, sk, noab, f*w, ab*w, &fallback);
    }
}

/* launch pass P (P < NP) or the final pass (P == NP) */
template<class F, int D, int NP>
static void sqb_split_launch(int P, const sqb_eval_t *a, double *tt, double *ta, int grid, int block, size_t smem, cudaStream_t st){
    static_assert(NP >= 1 && NP <= 16, "at most sixteen passes have launchers");
#define SQB_PASS_(Q) if constexpr((Q) < NP) if(P == (Q)){ sqb_k_part<F, D, (Q) < NP ? (Q) : 0><<<grid, block, smem, st>>>(*a, tt, ta); return; }
    SQB_PASS_(0) SQB_PASS_(1) SQB_PASS_(2) SQB_PASS_(3) SQB_PASS_(4) SQB_PASS_(5) SQB_PASS_(6) SQB_PASS_(7)
    SQB_PASS_(8) SQB_PASS_(9) SQB_PASS_(10) SQB_PASS_(11) SQB_PASS_(12) SQB_PASS_(13) SQB_PASS_(14) SQB_PASS_(15)
#undef SQB_PASS_
    sqb_k_fin<F, D><<<grid, block, smem, st>>>(*a, tt, ta);
}
template<class K_>
static int sqb_attr_of(K_ kernel, int block, size_t smem, sqb_kattr_t *o){
    cudaFuncAttributes fa; int nb = 0;
    if(cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) return 0;
    if(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, block, smem) != cudaSuccess) return 0;
    o->regs = fa.numRegs; o->local_bytes = (int)fa.localSizeBytes; o->max_threads = fa.maxThreadsPerBlock;
    o->blocks_per_sm = nb; o->fused = 0; o->sweeps = 1; return 1;
}
/* an FP64 (or dd) kernel's attributes; lv: the level kernel, which sums level tiles itself unless it sweeps
 * twice */
template<class K_>
static int sqb_f64_attr(K_ kernel, int lv, int block, size_t smem, sqb_kattr_t *o){
    if(!sqb_attr_of(kernel, block, smem, o)) return 0;
    o->fused = SQB_FUSE && !(lv && SQB_SWEEPS > 1);
    o->sweeps = lv ? SQB_SWEEPS : 1;
    return 1;
}
template<class F, int D, int NP>
static int sqb_split_attr(int P, int block, size_t smem, sqb_kattr_t *o){
    static_assert(NP >= 1 && NP <= 16, "at most sixteen passes have launchers");
#define SQB_PASS_(Q) if constexpr((Q) < NP) if(P == (Q)) return sqb_attr_of(sqb_k_part<F, D, (Q) < NP ? (Q) : 0>, block, smem, o);
    SQB_PASS_(0) SQB_PASS_(1) SQB_PASS_(2) SQB_PASS_(3) SQB_PASS_(4) SQB_PASS_(5) SQB_PASS_(6) SQB_PASS_(7)
    SQB_PASS_(8) SQB_PASS_(9) SQB_PASS_(10) SQB_PASS_(11) SQB_PASS_(12) SQB_PASS_(13) SQB_PASS_(14) SQB_PASS_(15)
#undef SQB_PASS_
    return sqb_attr_of(sqb_k_fin<F, D>, block, smem, o);
}

/* the axis form's launchers, empty for an integrand without one */
template<class R, int AB> struct sqb_noaxis { enum { NU = 0, NR = 0 }; };
template<class F, int D>
static bool sqb_ax_level(const sqb_eval_t *a, int grid, int block, size_t smem, cudaStream_t st){
    if constexpr(F::template AX<double, 0>::NU > 0) if(sqb_axis_launch(a)){
        if(a->ninst == 1){
            if(a->inst[0].last) sqb_k_lvax<F, D, 1, 0><<<grid, block, smem, st>>>(*a);
            else sqb_k_lvax<F, D, 0, 0><<<grid, block, smem, st>>>(*a);
        } else if(a->inst[0].last) sqb_k_lvax<F, D, 1, 1><<<grid, block, smem, st>>>(*a);      /* the same level of every integral */
        else sqb_k_lvax<F, D, 0, 1><<<grid, block, smem, st>>>(*a);
        return true;
    }
    return false;
}
/* a raw launch of the plug-in fills a table per CTA from this many points on and if it fits, beside the lattice
 * tables and the kernel's own sI, in the 48 KB that need no opt-in (static and dynamic together): syn_d8 up to K = 115,
 * syn_d11 to 85, syn_d5 at every K.  Measured per launch, K = 44: 131,072 children of syn_d5, d8, d11 13.3, 16.5,
 * 21.0 us -> 10.0, 12.3, 14.4; 65,536 the same either way; 4.1e6 of d8 and d11 390 and 457 us -> 114 and 120 */
#define SQB_AX_RAW (1L << 17)
#define SQB_AX_ROOM (48*1024 - SQB_MAXINST*sizeof(sqb_inst_t))
template<class F, int D>
static bool sqb_ax_points(const sqb_eval_t *a, int grid, int block, size_t smem, cudaStream_t st){
    if constexpr(F::template AX<double, 0>::NU > 0){
        if(a->ninst > 0 || a->sfin || a->sel || a->part || a->sym.n > 1 || a->cfl) return false;
        if(a->inl){ sqb_k_ax<F, D, 0, 1><<<grid, block, smem, st>>>(*a); return true; }
        if(a->U){ sqb_k_ax<F, D, 0, 0><<<grid, block, smem, st>>>(*a); return true; }
        const size_t sm = smem + (size_t)D*(2*a->K + 1)*sqb_axw<typename F::template AX<double, 0>, double>::N*sizeof(double);
        if(a->raw && (a->cells ? a->n << D : a->n) >= SQB_AX_RAW && sm <= SQB_AX_ROOM){
            sqb_k_ax<F, D, 1, 0><<<grid, block, sm, st>>>(*a); return true; }
    }
    return false;
}
template<class F, int D>
static bool sqb_ax_attr(int block, size_t smem, sqb_kattr_t *o, int *ok){
    if constexpr(F::template AX<double, 0>::NU > 0){
        *ok = sqb_attr_of(sqb_k_lvax<F, D, 1, 0>, block, smem, o);
        o->fused = 1; o->sweeps = 1;
        return true;
    }
    return false;
}
/* SQB_ATTR_REST: a build's level kernel and its axis form's kernels, loaded by asking for their attributes; their number */
template<class K_>
static int sqb_load(K_ kernel){ cudaFuncAttributes fa; return cudaFuncGetAttributes(&fa, kernel) == cudaSuccess; }
template<class F, int D, int LV>
static int sqb_load_rest(){
    int n = 0;
    if constexpr(LV > 0) n += sqb_load(sqb_k_f64<F, D, LV>);
    if constexpr(F::template AX<double, 0>::NU > 0)
        n += sqb_load(sqb_k_lvax<F, D, 0, 0>) + sqb_load(sqb_k_lvax<F, D, 1, 0>) + sqb_load(sqb_k_lvax<F, D, 0, 1>) +
             sqb_load(sqb_k_lvax<F, D, 1, 1>) + sqb_load(sqb_k_ax<F, D, 0, 0>) + sqb_load(sqb_k_ax<F, D, 0, 1>) + sqb_load(sqb_k_ax<F, D, 1, 0>) +
             sqb_load(sqb_k_axis<typename F::template AX<double, 0>, typename F::template AX<sqdd, 1>, D>);
    return n;
}
template<class F, int D>
static void sqb_ax_table(const double *X, int K, double *T, double *Td, cudaStream_t st){
    if constexpr(F::template AX<double, 0>::NU > 0)
        sqb_k_axis<typename F::template AX<double, 0>, typename F::template AX<sqdd, 1>, D><<<2*((D*(2*K + 1) + 31)/32), 32, 0, st>>>(X, K, T, Td);
}
template<class F, class R> struct sqb_ax_words { enum { N = F::template AX<R, 0>::NU > 0 ? (int)sqb_axw<typename F::template AX<R, 0>, R, 1>::N : 0 }; };

/* the scaling test (sqb_scale_t): one thread per (direction, q); P::pt is the graph's raw double-double
 * point function (pt_<name> of the QREAL half, SQ_AB = 1 as the reference's default) */
template<class P>
__global__ void __launch_bounds__(SQB_BLOCK) sqb_k_scale(const sqb_scale_t a){
    for(long j = blockIdx.x*(long)blockDim.x + threadIdx.x; j < 3*a.ndir; j += (long)gridDim.x*blockDim.x)
        a.g[j] = sqb_scale_value<P>(a, j);
}

/* SQ_GRAPH(name, volkov, L, D, weight, n, fixed): the generated file ends with it, after namespace
 * SQG_NS(name) with the class template K<Real, SQ_AB> holding f_<name>.
 *
 * Every graph has two translation units.  The first (compiled with -fmad=false) holds the FP64 kernel
 * whose roundings are those of the source, the double-double kernel and the registry entry SQB_<name>.
 * The second (SQB_FMA_TU, compiled with -fmad=true, namespace sqgf_<name> so that no symbol is shared)
 * holds only the FP64 kernel with multiplies and adds contracted into fused multiply-adds, exported as
 * SQB_<name>_f64fma and SQB_<name>_attrfma; the registry entry refers to them weakly. */
/* the split form's point functions (SQ_GRAPH_SPLIT): pass P and the final pass in FP64 */
#define SQ_SPLIT_F(NAME)                                                                           \
namespace SQG_NS(NAME) {                                                                           \
struct FS {                                                                                        \
    template<int P, int AB> static __device__ __forceinline__ void part(const double *sf, double *T, double *A){ \
        K<double, AB>::template fpart_##NAME<P>(sf, T, A); }                                       \
    template<int AB> static __device__ __forceinline__ double fin(const double *sf, double T, double A, double *ab){ \
        return K<double, AB>::ffin_##NAME(sf, T, A, ab); }                                         \
};                                                                                                 \
}
/* an integrand without the axis form */
#define SQ_NOAXIS(NAME) namespace SQG_NS(NAME) { template<class R, int AB> using KA = sqb_noaxis<R, AB>; }
#define SQ_GRAPH(NAME, VOLKOV, L, D, W, NP, FIX) SQ_NOAXIS(NAME) SQ_GRAPH_AXIS(NAME, VOLKOV, L, D, W, NP, FIX)
#if defined(SQB_FMA_TU)
#define SQ_SCALE(NAME)
#define SQ_GRAPH_AXIS(NAME, VOLKOV, L, D, W, NP, FIX)                                               \
namespace SQG_NS(NAME) {                                                                           \
struct F {                                                                                         \
    template<class R, int AB> using AX = KA<R, AB>;                                                \
    template<class R, int AB> static __device__ __forceinline__ R f(const R *sf, R *ab){           \
        return K<R, AB>::f_##NAME(sf, ab); }                                                       \
};                                                                                                 \
}                                                                                                  \
extern "C" void SQB_##NAME##_axisfma(const double *X, int K, double *T, double *Td, void *st){     \
    sqb_ax_table<SQG_NS(NAME)::F, D>(X, K, T, Td, (cudaStream_t)st); }                              \
extern "C" void SQB_##NAME##_f64fma(const sqb_eval_t *a, int grid, int block, size_t smem, void *st){ \
    if(sqb_ax_level<SQG_NS(NAME)::F, D>(a, grid, block, smem, (cudaStream_t)st)) return;            \
    if(sqb_ax_points<SQG_NS(NAME)::F, D>(a, grid, block, smem, (cudaStream_t)st)) return;           \
    if(sqb_level_launch(a)) sqb_k_f64<SQG_NS(NAME)::F, D, 1><<<grid, block, smem, (cudaStream_t)st>>>(*a); \
    else sqb_k_f64<SQG_NS(NAME)::F, D, 0><<<grid, block, smem, (cudaStream_t)st>>>(*a); }           \
extern "C" int SQB_##NAME##_attrfma(int lv, int block, size_t smem, sqb_kattr_t *o){               \
    if(lv == SQB_ATTR_REST) return sqb_load_rest<SQG_NS(NAME)::F, D, 1>();                          \
    int ok; if(lv && sqb_ax_attr<SQG_NS(NAME)::F, D>(block, smem, o, &ok)) return ok;               \
    return lv ? sqb_f64_attr(sqb_k_f64<SQG_NS(NAME)::F, D, 1>, 1, block, smem, o)                  \
              : sqb_f64_attr(sqb_k_f64<SQG_NS(NAME)::F, D, 0>, 0, block, smem, o); }
#define SQ_GRAPH_SPLIT(NAME, VOLKOV, L, D, W, NP, FIX, NPARTS)                                      \
SQ_GRAPH(NAME, VOLKOV, L, D, W, NP, FIX)                                                           \
SQ_SPLIT_F(NAME)                                                                                   \
extern "C" void SQB_##NAME##_splitfma(int P, const sqb_eval_t *a, double *tt, double *ta, int grid, int block, \
                                      size_t smem, void *st){                                      \
    sqb_split_launch<SQG_NS(NAME)::FS, D, NPARTS>(P, a, tt, ta, grid, block, smem, (cudaStream_t)st); } \
extern "C" int SQB_##NAME##_splitattrfma(int P, int block, size_t smem, sqb_kattr_t *o){          \
    return sqb_split_attr<SQG_NS(NAME)::FS, D, NPARTS>(P, block, smem, o); }
#else
/* SQ_SCALE(name) follows SQ_GRAPH for a graph with a raw point function: its scaling-test launcher */
#define SQ_SCALE(NAME)                                                                              \
namespace SQG_NS(NAME) {                                                                           \
struct PT {                                                                                        \
    static __device__ __forceinline__ sqdd pt(const sqdd *x, sqdd Vx, sqdd *ab){                   \
        return KD<sqdd, 1>::pt_##NAME(x, Vx, ab); }                                                \
};                                                                                                 \
}                                                                                                  \
extern "C" void SQB_##NAME##_scale(const sqb_scale_t *a, int grid, int block, void *st){           \
    sqb_k_scale<SQG_NS(NAME)::PT><<<grid, block, 0, (cudaStream_t)st>>>(*a); }
#define SQ_GRAPH_CORE(NAME, D)                                                                      \
extern "C" void SQB_##NAME##_f64fma(const sqb_eval_t *, int, int, size_t, void *) __attribute__((weak)); \
extern "C" void SQB_##NAME##_axisfma(const double *, int, double *, double *, void *) __attribute__((weak)); \
extern "C" void SQB_##NAME##_scale(const sqb_scale_t *, int, int, void *) __attribute__((weak));   \
extern "C" int SQB_##NAME##_attrfma(int, int, size_t, sqb_kattr_t *) __attribute__((weak));        \
namespace SQG_NS(NAME) {                                                                           \
struct F {                                                                                         \
    template<class R, int AB> using AX = KA<R, AB>;                                                \
    template<class R, int AB> static __device__ __forceinline__ R f(const R *sf, R *ab){           \
        return K<R, AB>::f_##NAME(sf, ab); }                                                       \
};                                                                                                 \
template<> __device__ __forceinline__ sqdd F::f<sqdd, 1>(const sqdd *sf, sqdd *ab){                \
    return KD<sqdd, 1>::f_##NAME(sf, ab); }                                                        \
static void f64(const sqb_eval_t *a, int grid, int block, size_t smem, void *st){                  \
    if(sqb_ax_level<F, D>(a, grid, block, smem, (cudaStream_t)st)) return;                         \
    if(sqb_ax_points<F, D>(a, grid, block, smem, (cudaStream_t)st)) return;                        \
    if(SQB_LEVEL_KERNEL && sqb_level_launch(a))                                                    \
        sqb_k_f64<F, D, SQB_LEVEL_KERNEL><<<grid, block, smem, (cudaStream_t)st>>>(*a);            \
    else sqb_k_f64<F, D, 0><<<grid, block, smem, (cudaStream_t)st>>>(*a); }                        \
static void dd(const sqb_dd_t *a, int grid, int block, size_t smem, void *st){                     \
    sqb_k_dd<F, D><<<grid, block, smem, (cudaStream_t)st>>>(*a); }                                 \
static void axis(int fma, const double *X, int K, double *T, double *Td, void *st){                \
    if(fma && SQB_##NAME##_axisfma) SQB_##NAME##_axisfma(X, K, T, Td, st);                         \
    else sqb_ax_table<F, D>(X, K, T, Td, (cudaStream_t)st); }                                      \
static int attr(int which, int block, size_t smem, sqb_kattr_t *o){                                \
    const int lv = which & (SQB_ATTR_LEVEL | SQB_ATTR_REST); which &= ~lv;                         \
    if(which == 2) return SQB_##NAME##_attrfma ? SQB_##NAME##_attrfma(lv, block, smem, o) : 0;      \
    if(which == 1) return sqb_f64_attr(sqb_k_dd<F, D>, 0, block, smem, o);                         \
    if(lv == SQB_ATTR_REST) return sqb_load_rest<F, D, SQB_LEVEL_KERNEL>();                         \
    int ok; if(lv && sqb_ax_attr<F, D>(block, smem, o, &ok)) return ok;                             \
    return SQB_LEVEL_KERNEL && lv ? sqb_f64_attr(sqb_k_f64<F, D, SQB_LEVEL_KERNEL>, 1, block, smem, o) \
                                  : sqb_f64_attr(sqb_k_f64<F, D, 0>, 0, block, smem, o); }         \
}
#define SQ_AXIS_ENTRY(NAME) sqb_ax_words<SQG_NS(NAME)::F, double>::N ? SQG_NS(NAME)::axis : NULL,    \
    {sqb_ax_words<SQG_NS(NAME)::F, double>::N, sqb_ax_words<SQG_NS(NAME)::F, sqdd>::N}
#define SQ_GRAPH_AXIS(NAME, VOLKOV, L, D, W, NP, FIX)                                               \
SQ_GRAPH_CORE(NAME, D)                                                                             \
extern "C" const sqb_graph_t SQB_##NAME = {#NAME, VOLKOV, L, D, W, NP, FIX, 0,                     \
    SQG_NS(NAME)::f64, SQG_NS(NAME)::dd, SQG_NS(NAME)::attr, SQB_##NAME##_f64fma, 0, NULL, NULL,     \
    SQB_##NAME##_scale, SQ_AXIS_ENTRY(NAME)};
#define SQ_GRAPH_SPLIT(NAME, VOLKOV, L, D, W, NP, FIX, NPARTS)                                      \
SQ_NOAXIS(NAME)                                                                                    \
SQ_GRAPH_CORE(NAME, D)                                                                             \
SQ_SPLIT_F(NAME)                                                                                   \
extern "C" void SQB_##NAME##_splitfma(int, const sqb_eval_t *, double *, double *, int, int, size_t, void *) \
    __attribute__((weak));                                                                         \
extern "C" int SQB_##NAME##_splitattrfma(int, int, size_t, sqb_kattr_t *) __attribute__((weak));   \
namespace SQG_NS(NAME) {                                                                           \
static void split(int P, int fma, const sqb_eval_t *a, double *tt, double *ta, int grid, int block, size_t smem, \
                  void *st){                                                                       \
    if(fma && SQB_##NAME##_splitfma) SQB_##NAME##_splitfma(P, a, tt, ta, grid, block, smem, st);    \
    else sqb_split_launch<FS, D, NPARTS>(P, a, tt, ta, grid, block, smem, (cudaStream_t)st); }     \
static int split_attr(int P, int fma, int block, size_t smem, sqb_kattr_t *o){                     \
    if(fma && SQB_##NAME##_splitattrfma) return SQB_##NAME##_splitattrfma(P, block, smem, o);       \
    return sqb_split_attr<FS, D, NPARTS>(P, block, smem, o); }                                      \
}                                                                                                  \
extern "C" const sqb_graph_t SQB_##NAME = {#NAME, VOLKOV, L, D, W, NP, FIX, 0,                     \
    SQG_NS(NAME)::f64, SQG_NS(NAME)::dd, SQG_NS(NAME)::attr, SQB_##NAME##_f64fma, NPARTS,           \
    SQG_NS(NAME)::split, SQG_NS(NAME)::split_attr, SQB_##NAME##_scale, NULL, {0, 0}};
#endif
