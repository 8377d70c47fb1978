/* runtime.cu -- the device layer: device state, node-batch evaluation with the precision fallback, the
 * device-resident refinement level (evaluate, fall back, reduce, keep), and the reference's GPU plug-in
 * ABI (the plain form, driver/gpu.h:12-22).
 *
 * A refinement level (driver/sum.c:652-799) is run on the device in batches of cells:
 *   1. sqb_k_f64 (per graph): every child in FP64 with the per-point tests; points whose |.| bound is
 *      above ABSERR are queued;
 *   2. sqb_k_dd (per graph): the queued points in double-double (qvalue semantics);
 *   3. sqb_k_reduce: per tile of children (in cell order, b ascending), compensated double-double sums of
 *      v*pw, |v|, the dropped weight, the shadow-tier sums and the round column, plus counters and the
 *      number of kept children;
 *   4. sqb_k_finish: exclusive scan of the tiles' kept counts and the tiles' sums added in
 *      a fixed order into the level accumulator, so that a run is reproducible;
 *   5. sqb_k_scatter: the kept children written, in order, to the next level's cell list with their
 *      flags (skip bit, shadow tier; driver/sum.c:741-745).
 * Nothing goes back to the host until the level ends: the host reads the accumulator once per level. */
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <math.h>
#include <omp.h>
#include "sqb_rt.h"
#include "sqdd.cuh"
#include "sqorbit.cuh"
#include <atomic>
#include <vector>
#include "sincfeyn_b200.h"

extern "C" const sqb_graph_t *const SQB_ALL[];
extern "C" const int SQB_NALL;

/* Every piece of state below is per host thread (thread_local): each thread that calls the chosen form
 * has its own stream, events, buffers and error text, so several integrals can run concurrently from
 * a pool of threads (batch.cpp).  The plain form (gpu_setup ... gpu_wait) stays single-threaded, as the
 * reference's driver calls it (driver/eval.c:104-107). */
static thread_local char g_err[512];
#define CKR(x) do { cudaError_t e_ = (x); if(e_ != cudaSuccess){                                    \
    snprintf(g_err, sizeof g_err, "%s at %s:%d: %s", #x, __FILE__, __LINE__, cudaGetErrorString(e_)); \
    cudaGetLastError();              /* reported here: not the next call's error */                  \
    return (int)e_; } } while(0)

extern "C" const char *sqb_last_error(void){ return g_err; }
extern "C" void sqb_set_error_msg(const char *msg);        /* the text sqb_error() returns (engine.cpp) */

extern "C" const sqb_graph_t *sqb_find_graph(const char *name){
    for(int i = 0; i < SQB_NALL; i++) if(!strcmp(SQB_ALL[i]->name, name) || !strcmp(SQB_ALL[i]->volkov, name)) return SQB_ALL[i];
    return NULL;
}
extern "C" int sqb_ngraphs(void){ return SQB_NALL; }
extern "C" const sqb_graph_t *sqb_graph_at(int i){ return i >= 0 && i < SQB_NALL ? SQB_ALL[i] : NULL; }

/* ------------------------------------------------------------------------------------------------ */
#define RT 256                    /* threads per reduce / scatter CTA */
#define RPT 16                    /* children per thread (scatter: consecutive; reduce: RT apart) */
#define RTILE (RT*RPT)
#define FT 256                    /* tiles per CTA of the finish kernel, one per thread */

typedef sqb_part_t part_t;
static_assert(RTILE == SQB_TILE, "the reduce kernel's tiles are the FP64 kernel's");

/* one integral of a multi-instance level batch, for the tail kernels: its children are the launch's
 * [child0, child0 + n); its kept children go to next (cap cells), its sums to acc, its first kept slot to
 * *base */
typedef struct {
    const signed char *cells; long n, child0;
    int st, last; double pw, thr;
    sqb_pt_t *next; long cap;
    sqb_acc_t *acc; unsigned long long *base;
} lvi_t;
typedef struct {
    const signed char *cells;     /* device pt_t list (12 bytes per cell) */
    long n;                       /* children in this batch */
    int D, st, last, abskip;
    double pw, thr;
    const double *v, *uu;
    const unsigned char *stt;
    sqb_sym_t sym;                /* the symmetry fold (sym.n <= 1: off) */
    const unsigned char *cfl;     /* the predictor's per-child tiers at the last level (NULL: the parent's) */
    int ninst;                    /* > 0: a multi-instance batch, the integrals in inst (the fields above that
                                     describe one batch unused); 0: one batch */
    lvi_t inst[SQB_MAXINST];
    const unsigned char *cw;      /* list mode: every child's orbit weight from the select pass (0: not evaluated) */
} lvl_t;

/* the finish kernel's sums of FT tiles: S, |v|, drop, b1, b2, u; evaluated, fallback, unresolved, skipped, kept */
struct fpart_t { double x[6][2]; unsigned long long c[5]; };

struct Dev {
    int on, dev, nsm;
    cudaEvent_t t0, t1; void *flush; size_t flushn;
    unsigned long long launches;   /* kernels of this library launched so far */
    cudaEvent_t kev[3*256]; int nkev, kevn;   /* kernel timing: (FP64 start, FP64 end / dd start, dd end) per pass */
    double f64_ms, dd_ms; long f64_n;
    char info[256];
    cudaStream_t s;
    cudaEvent_t e0, e1;
    double *X, *Wt; int tabcap, K;
    double *axb; long axcap; const double *U, *Ud;   /* axis tables of the current lattice and graph (NULL: none) */
    long cap;                      /* points per batch */
    double *v, *uu; unsigned char *stt, *cfl, *cw; long *fb; unsigned long long *nfb;
    unsigned long long *sel, *nsel;   /* list mode: the children to evaluate and their number */
    long nbcap; part_t *bp; unsigned *bkeep; unsigned long long *boff; unsigned char *tfb;
    fpart_t *fp; unsigned long long *coff; unsigned *fcnt;   /* per FT tiles: sums, kept before them; CTAs done per integral */
    long ttcap; double *tt, *ta;   /* split FP64 pass: running sums per point */
    sqb_acc_t *acc; unsigned long long *base;
    sqb_acc_t *accm; unsigned long long *basem, *queue;   /* multi-instance levels: per integral, tile queue */
};
static thread_local Dev G;
static int KTIME;                  /* sqb_kernel_timing(): all threads */
static std::atomic<unsigned long long> H2D, D2H;   /* bytes copied by the chosen form's calls, all threads */

/* the timed passes so far: their events are read once the stream has passed them (the callers that wait
 * on the stream anyway), so timing adds no synchronisation between a level's batches */
static void ktime_collect(void){
    if(!G.nkev) return;
    cudaEventSynchronize(G.kev[3*G.nkev - 1]);
    for(int i = 0; i < G.nkev; i++){
        float x = 0, y = 0;
        cudaEventElapsedTime(&x, G.kev[3*i], G.kev[3*i + 1]); cudaEventElapsedTime(&y, G.kev[3*i + 1], G.kev[3*i + 2]);
        G.f64_ms += x; G.dd_ms += y; G.f64_n++;
    }
    G.nkev = 0;
}
/* the event triple of the next timed pass (NULL: timing off or no events) */
static cudaEvent_t *ktime_slot(void){
    if(!KTIME) return NULL;
    const int cap = (int)(sizeof G.kev/sizeof G.kev[0])/3;
    if(G.nkev == cap) ktime_collect();
    if(G.nkev >= G.kevn){
        for(int j = 0; j < 3; j++) if(cudaEventCreate(&G.kev[3*G.nkev + j]) != cudaSuccess) return NULL;
        G.kevn = G.nkev + 1;
    }
    return &G.kev[3*G.nkev++];
}

extern "C" int sqb_dev_init(int device){
    if(G.on) return 0;
    int nd = 0; CKR(cudaGetDeviceCount(&nd));
    if(nd == 0){ snprintf(g_err, sizeof g_err, "no CUDA device"); return -1; }
    if(device < 0 || device >= nd) device = 0;
    CKR(cudaSetDevice(device));
    cudaDeviceProp p; CKR(cudaGetDeviceProperties(&p, device));
    G.dev = device; G.nsm = p.multiProcessorCount;
    snprintf(G.info, sizeof G.info, "%s (sm_%d%d, %d SMs)", p.name, p.major, p.minor, p.multiProcessorCount);
    CKR(cudaStreamCreateWithFlags(&G.s, cudaStreamNonBlocking));
    /* the cell lists and the grow's tables come from the device's stream-ordered pool, which keeps
     * freed memory for the next integral instead of returning it (no cudaFree synchronisation) */
    { cudaMemPool_t pool; CKR(cudaDeviceGetDefaultMemPool(&pool, device));
      unsigned long long keep = ~0ULL; CKR(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep)); }
    CKR(cudaEventCreate(&G.e0)); CKR(cudaEventCreate(&G.e1));
    CKR(cudaEventCreate(&G.t0)); CKR(cudaEventCreate(&G.t1));
    CKR(cudaMalloc(&G.acc, sizeof(sqb_acc_t)));
    CKR(cudaMalloc(&G.base, sizeof(unsigned long long)));
    CKR(cudaMalloc(&G.nfb, sizeof(unsigned long long)));
    CKR(cudaMalloc(&G.accm, SQB_MAXINST*sizeof(sqb_acc_t)));
    CKR(cudaMalloc(&G.basem, SQB_MAXINST*sizeof(unsigned long long)));
    CKR(cudaMalloc(&G.queue, sizeof(unsigned long long)));
    CKR(cudaMalloc(&G.nsel, sizeof(unsigned long long)));
    CKR(cudaMalloc(&G.fcnt, SQB_MAXINST*sizeof(unsigned)));
    CKR(cudaMemsetAsync(G.fcnt, 0, SQB_MAXINST*sizeof(unsigned), G.s));      /* every finish leaves it 0 */
    G.on = 1;
    return 0;
}
extern "C" const char *sqb_dev_info(void){ return G.on ? G.info : "off"; }

extern "C" int sqb_dev_tables(const double *X, const double *Wt, int K){
    int nt = 2*K + 1;
    if(nt > G.tabcap){
        if(G.X){ cudaFree(G.X); cudaFree(G.Wt); }
        CKR(cudaMalloc(&G.X, nt*sizeof(double))); CKR(cudaMalloc(&G.Wt, nt*sizeof(double)));
        G.tabcap = nt;
    }
    CKR(cudaMemcpy(G.X, X, nt*sizeof(double), cudaMemcpyHostToDevice));
    CKR(cudaMemcpy(G.Wt, Wt, nt*sizeof(double), cudaMemcpyHostToDevice));
    H2D += 2*nt*sizeof(double);
    G.K = K; G.U = G.Ud = NULL;
    return 0;
}

/* doubles of a graph's two axis tables over a lattice (0: the integrand has no axis form); FP64 first */
static long axis_words(const sqb_graph_t *g, int K, int which){ return g->axis ? (long)g->D*(2*K + 1)*g->axw[which] : 0; }
extern "C" long sqb_dev_axis_words(const sqb_graph_t *g, int K){ return axis_words(g, K, 0) + axis_words(g, K, 1); }
/* fills the tables of the lattice X (device) for the FP64 build fma at T (device), on the thread's stream */
extern "C" int sqb_dev_axis_fill(const sqb_graph_t *g, int fma, const double *X, int K, double *T){
    if(!g->axis) return 0;
    g->axis(fma, X, K, T, T + axis_words(g, K, 0), G.s);
    CKR(cudaGetLastError());
    G.launches++;
    return 0;
}
/* the axis tables of graph g on the thread's current lattice (sqb_dev_tables), used by the evaluations that
 * follow until the lattice changes */
extern "C" int sqb_dev_axis(const sqb_graph_t *g, int fma){
    G.U = G.Ud = NULL;
    const long n = sqb_dev_axis_words(g, G.K);
    if(!n) return 0;
    if(n > G.axcap){
        if(G.axb) cudaFree(G.axb);
        G.axb = NULL; G.axcap = 0;
        long c = 1L << 13; while(c < n) c <<= 1;
        CKR(cudaMalloc(&G.axb, c*sizeof(double)));
        G.axcap = c;
    }
    if(sqb_dev_axis_fill(g, fma, G.X, G.K, G.axb)) return -1;
    G.U = G.axb; G.Ud = G.axb + axis_words(g, G.K, 0);
    return 0;
}

static void free_points(void){
    void *p[] = {G.v, G.uu, G.stt, G.cfl, G.cw, G.fb, G.sel, G.bp, G.bkeep, G.boff, G.tfb, G.fp, G.coff};
    for(void *q : p) if(q) cudaFree(q);
    G.v = G.uu = NULL; G.stt = G.cfl = G.cw = G.tfb = NULL; G.fb = NULL; G.sel = G.boff = G.coff = NULL;
    G.bp = NULL; G.bkeep = NULL; G.fp = NULL; G.cap = G.nbcap = 0;
}
static int alloc_points(long c){
    CKR(cudaMalloc(&G.v, c*sizeof(double))); CKR(cudaMalloc(&G.uu, c*sizeof(double)));
    CKR(cudaMalloc(&G.stt, c)); CKR(cudaMalloc(&G.cfl, c)); CKR(cudaMalloc(&G.cw, c)); CKR(cudaMalloc(&G.fb, c*sizeof(long)));
    CKR(cudaMalloc(&G.sel, c*sizeof(unsigned long long)));
    const long nb = (c + RTILE - 1)/RTILE;
    CKR(cudaMalloc(&G.bp, nb*sizeof(part_t))); CKR(cudaMalloc(&G.bkeep, nb*sizeof(unsigned))); CKR(cudaMalloc(&G.tfb, nb));
    CKR(cudaMalloc(&G.boff, nb*sizeof(unsigned long long)));
    const long nf = nb/FT + SQB_MAXINST + 1;
    CKR(cudaMalloc(&G.fp, nf*sizeof(fpart_t))); CKR(cudaMalloc(&G.coff, nf*sizeof(unsigned long long)));
    G.cap = c; G.nbcap = nb;
    return 0;
}
/* room for n points; without it none is left */
static int reserve_points(long n){
    if(n <= G.cap) return 0;
    long c = 1L << 16; while(c < n) c <<= 1;
    free_points();
    if(!alloc_points(c)) return 0;
    free_points();
    cudaGetLastError();
    return -1;
}
/* children per batch unless the caller says: each batch costs about 80 us beside its children (the tails of its kernels, the
 * double-double pass's longest chain), and 35 bytes a child are held (alloc_points).  syn_d8 at h = 0.7 with 2^24, 2^25, 2^26,
 * 2^27: 19.7, 16.6, 15.3, 14.7 ms; 2.35 GB at 2^26.  2^25 for the split pass, which holds its running sums as well; for a
 * thread that finds no room for more; and for one of more than sixteen workers of a batch, so that together they take no
 * more than the most workers (32) do with the lower size: 37.6 GB, which their cell lists, and an integral run again
 * alone beside the workers' buffers, leave. */
#define CHILDREN (1L << 26)
#define CHILDREN_LOW (1L << 25)
#define CHILDREN_SHARE (1.0/16)
extern "C" double sqb_mem_share(void);
extern "C" long sqb_share_children(double share){ return share >= CHILDREN_SHARE ? CHILDREN : CHILDREN_LOW; }
/* whether the FP64 pass sums a level's tiles itself: where a batch gives every one of the cap resident CTAs two tiles or more.
 * One answer for the whole level, a last short batch included: the two ways round |v| differently, and a level's sums
 * do not depend on the size of its batches (a thread short of memory runs smaller ones) */
static bool fuses(long ncell, long ncb, int D, long cap){ return ((ncell < ncb ? ncell : ncb) << D) >= 2*SQB_TILE*cap; }
/* children per launch of a group's round: a launch takes the batches of as many of its integrals as fit (eight of the lower
 * size, four of the full one; a batch is never split, so that every integral keeps the batches it has alone) */
#define GROUP_CHILDREN (SQB_MAXINST*CHILDREN_LOW)
static long batch_children(const sqb_graph_t *g, const sqb_level_t *L){
    return L->max_children > 0 ? L->max_children : L->t.split && g->nparts > 0 ? CHILDREN_LOW : sqb_share_children(sqb_mem_share());
}

/* the FP64 kernel to run: the contracted one (which 2) when asked for and built, else the exact one */
static inline int f64_which(const sqb_graph_t *g, int fma){ return fma && g->f64_fma ? 2 : 0; }
static inline void launch_f64(const sqb_graph_t *g, int which, const sqb_eval_t *a, int grid, size_t smem, cudaStream_t s){
    if(which == 2) g->f64_fma(a, grid, 128, smem, s); else g->f64(a, grid, 128, smem, s);
}

/* resident CTAs of a graph's kernel on the whole device (which | SQB_ATTR_LEVEL: its level kernel); *fused:
 * the kernel sums level tiles itself; *sweeps: the level kernel's passes over a batch's tiles */
static long grid_cap(const sqb_graph_t *g, int which, size_t smem, int *fused = NULL, int *sweeps = NULL){
    sqb_kattr_t at; memset(&at, 0, sizeof at); int per = 2;
    const int ok = g->attr(which, 128, smem, &at);
    if(ok && at.blocks_per_sm > 0) per = at.blocks_per_sm;
    if(fused) *fused = ok && at.fused;
    if(sweeps) *sweeps = ok && at.sweeps > 1 ? at.sweeps : 1;
    return (long)G.nsm*per;
}

static int grid_for(const sqb_graph_t *g, int which, long npts, size_t smem){
    sqb_kattr_t at; int per = 2;
    long want = (npts + 127)/128;
    if(want <= 4*G.nsm) return want < 1 ? 1 : (int)want;     /* two waves at most whatever the kernel: no occupancy query, which
                                                                costs a small launch a tenth of its time */
    if(g->attr(which, 128, smem, &at) && at.blocks_per_sm > 0) per = at.blocks_per_sm;
    const long full = (long)G.nsm*per;
    return (int)(want < full ? want : full);
}

static void fill_eval(sqb_eval_t *a, const sqb_test_t *t){
    a->X = G.X; a->Wt = G.Wt; a->K = G.K; a->H = 0; a->raw = 0; a->U = G.U; a->Ud = G.Ud;
    a->abskip = t->abskip; a->abcheck = t->abcheck;
    a->abserr = t->abserr; a->near_thr = t->nearf*t->abserr; a->ddslack = t->ddslack;
    a->v = G.v; a->ab = NULL; a->stt = G.stt; a->fb = G.fb; a->nfb = G.nfb; a->fbcap = G.cap;
}

/* work items per tile of an axis-form level launch whose tiles the reduce kernel sums: 1024 children each */
#define SQB_SUB 4

/* whether a batch's FP64 pass runs in passes (the graph has them, they are asked for, a level batch) */
static inline bool use_split(const sqb_graph_t *g, const sqb_eval_t *a, const sqb_test_t *t){
    return t->split && g->nparts > 0 && a->cells && !t->alldd;
}

/* FP64 pass (or the all-dd pass) and the fallback pass for one batch already described by a */
/* dynamic shared memory of a launch: the tables of its integral(s), 2(2K+1) doubles each */
static size_t table_bytes(const sqb_eval_t *a){
    if(a->ninst <= 0) return 2*(2*(size_t)a->K + 1)*sizeof(double);
    size_t w = 0;
    for(int q = 0; q < a->ninst; q++) w += 2*(2*(size_t)a->inst[q].K + 1);
    return w*sizeof(double);
}

/* SQB_TILE_SUMS (environment, read once): 1 (default) = a level batch's FP64 kernel sums the tiles that
 * need no fallback itself; 0 = the reduce kernel sums every tile */
static int tile_sums(void){
    static int v = -1;
    if(v < 0){ const char *e = getenv("SQB_TILE_SUMS"); v = e && *e ? atoi(e) != 0 : 1; }
    return v;
}

static int eval_batch(const sqb_graph_t *g, sqb_eval_t *a, const sqb_test_t *t, long npts){
    /* the tables, then (level launches) the FP64 kernel's tile-sum columns */
    size_t smem = table_bytes(a) + (a->part ? sizeof(sqb_tile_acc) : 0);
    sqb_dd_t d; memset(&d, 0, sizeof d);
    d.e = *a; d.dropunres = t->dropunres; d.uu = G.uu;
    if(t->alldd){
        d.all = 1;
        g->dd(&d, grid_for(g, 1, npts, smem), 128, smem, G.s);
        CKR(cudaGetLastError());
        G.launches++;
        return 0;
    }
    cudaEvent_t *ev = ktime_slot();
    if(ev) CKR(cudaEventRecord(ev[0], G.s));
    if(g->axis && !use_split(g, a, t) && sqb_axis_inline(a, npts)){
        const int w = f64_which(g, t->fma);
        a->inl = 1; a->dropunres = t->dropunres; a->uu = G.uu;
        launch_f64(g, w, a, grid_for(g, w, npts, smem), smem, G.s);
        CKR(cudaGetLastError());
        G.launches++;
        if(ev){ CKR(cudaEventRecord(ev[1], G.s)); CKR(cudaEventRecord(ev[2], G.s)); }
        return 0;
    }
    CKR(cudaMemsetAsync(G.nfb, 0, sizeof(unsigned long long), G.s));
    if(use_split(g, a, t)){
        if(npts > G.ttcap){
            if(G.tt){ cudaFree(G.tt); cudaFree(G.ta); }
            long c = 1L << 16; while(c < npts) c <<= 1;
            CKR(cudaMalloc(&G.tt, c*sizeof(double))); CKR(cudaMalloc(&G.ta, c*sizeof(double)));
            G.ttcap = c;
        }
        for(int P = 0; P <= g->nparts; P++){
            sqb_kattr_t at; memset(&at, 0, sizeof at); int per = 2;
            if(g->split_attr(P, t->fma, 128, smem, &at) && at.blocks_per_sm > 0) per = at.blocks_per_sm;
            long want = (npts + 127)/128, full = (long)G.nsm*per;
            g->split(P, t->fma, a, G.tt, G.ta, (int)(want < full ? want : full), 128, smem, G.s);
            CKR(cudaGetLastError());
        }
        G.launches += g->nparts;
    } else {
        const int w = f64_which(g, t->fma);
        if(a->ninst > 0){
            CKR(cudaMemsetAsync(a->queue, 0, sizeof(unsigned long long), G.s));
            int sw = 1;
            const long cap = grid_cap(g, w | (sqb_level_launch(a) ? SQB_ATTR_LEVEL : 0), smem, NULL, &sw);
            const long items = sqb_axis_launch(a) && a->sub > 1 ? a->ntile*a->sub : a->ntile*sw;   /* the level kernel may
                                                                                  take every tile twice */
            launch_f64(g, w, a, (int)(items < cap ? items : cap), smem, G.s);
        } else launch_f64(g, w, a, grid_for(g, w, npts, smem), smem, G.s);
        CKR(cudaGetLastError());
    }
    if(ev) CKR(cudaEventRecord(ev[1], G.s));
    d.list = G.fb; d.nlist = G.nfb; d.listcap = G.cap; d.all = 0;
    /* the queue length is known only on the device: a persistent grid reads it */
    g->dd(&d, grid_for(g, 1, 1L << 30, smem), 128, smem, G.s);
    CKR(cudaGetLastError());
    G.launches += 2;
    if(ev) CKR(cudaEventRecord(ev[2], G.s));
    return 0;
}

/* n device-resident nodes (pt_t, flags ignored; np: their number on the device, at most n, or NULL; skip per node on the
 * device or NULL) evaluated with the tests and the fallback; the values, status and round column stay on the device until the next evaluation.  Queued on the
 * thread's stream, no wait */
extern "C" int sqb_dev_eval_resident(const sqb_graph_t *g, const sqb_pt_t *pts, long n, const unsigned long long *np,
                                     const unsigned char *skip, const sqb_test_t *t, const double **v_dev, const unsigned char **stt_dev, const double **uu_dev){
    *v_dev = *uu_dev = NULL; *stt_dev = NULL;
    if(n <= 0) return 0;
    if(reserve_points(n)) return -1;
    sqb_eval_t a; memset(&a, 0, sizeof a); fill_eval(&a, t);
    a.pts = pts; a.n = n; a.esize = 1; a.stride = SQB_MAXD; a.flag_at = -1; a.cells = 0; a.st = 0; a.skip = skip; a.np = np;
    if(eval_batch(g, &a, t, n)) return -1;
    *v_dev = G.v; *stt_dev = G.stt; *uu_dev = G.uu;
    return 0;
}
extern "C" void *sqb_dev_stream(void){ return (void*)G.s; }

/* Load the device code of a graph's kernels now (NULL: every graph).  CUDA loads a kernel's code on
 * its first launch by default (lazy loading); for this library's large per-graph kernels that first
 * launch costs up to a second, so a caller that times integrals, or wants the cost at start-up,
 * preloads.  Returns the number of kernels loaded, or -1. */
extern "C" int sqb_preload(const char *graph){
    if(sqb_dev_init(0)) return -1;
    int n = 0;
    for(int i = 0; i < SQB_NALL; i++){
        const sqb_graph_t *g = SQB_ALL[i];
        if(graph && strcmp(graph, g->name)) continue;
        sqb_kattr_t at;
        for(int which = 0; which < 3; which++) if(g->attr(which, 128, 4096, &at)) n++;
        for(int which = 0; which < 3; which += 2) n += g->attr(which | SQB_ATTR_REST, 128, 4096, &at);
        for(int P = 0; P <= g->nparts && g->nparts > 0; P++)
            for(int fma = 0; fma < 2; fma++) if(g->split_attr(P, fma, 128, 4096, &at)) n++;
    }
    return n;
}
/* instrumentation: kernels launched so far; with ktime on, the FP64 and double-double kernels of every
 * evaluation pass are bracketed by events, read when the host next waits on the stream, and their times
 * summed */
extern "C" unsigned long long sqb_launch_count(void){ return G.launches; }
extern "C" void sqb_kernel_timing(int on){ KTIME = on; }
extern "C" void sqb_kernel_times(double *f64_ms, double *dd_ms, long *f64_launches, int reset){
    ktime_collect();
    *f64_ms = G.f64_ms; *dd_ms = G.dd_ms; *f64_launches = G.f64_n;
    if(reset){ G.f64_ms = G.dd_ms = 0; G.f64_n = 0; }
}

/* ---------------------------------------- level reduce ------------------------------------------ */
__device__ __forceinline__ sqdd shfl_dd(const sqdd &a, int off){
    return sqdd(__shfl_down_sync(0xffffffffu, a.hi, off), __shfl_down_sync(0xffffffffu, a.lo, off));
}
/* the integral of tile b of a batch (one batch: the batch itself, with child0 = 0) */
__device__ __forceinline__ lvi_t lvl_inst(const lvl_t &a, long b, int *index = NULL){
    lvi_t v;
    if(index) *index = 0;
    if(a.ninst <= 0){
        v.cells = a.cells; v.n = a.n; v.child0 = 0; v.st = a.st; v.last = a.last; v.pw = a.pw; v.thr = a.thr;
        v.next = NULL; v.cap = 0; v.acc = NULL; v.base = NULL;
        return v;
    }
    int k = 0;
    for(int q = 1; q < a.ninst; q++) if(a.inst[q].child0 <= b*(long)RTILE) k = q;
    if(index) *index = k;
    return a.inst[k];
}
/* the finish kernel's slot of tile b (of integral k, whose first tile is tb): FT tiles each, no slot shared by two
 * integrals */
__device__ __forceinline__ long fin_slot(long tb, int k, long b){ return tb/FT + k + (b - tb)/FT; }
/* child il's coordinates k_d - st bit_d(b) (driver/sum.c:407) */
__device__ __forceinline__ void child_of(const lvl_t &a, const lvi_t &L, long il, int *k){
    const long c = il >> a.D; const int b = (int)(il & ((1L << a.D) - 1));
    const signed char *p = L.cells + c*SQB_MAXD;
    for(int d = 0; d < a.D; d++) k[d] = p[d] - (((b >> d) & 1) ? L.st : 0);
}
/* child b of cell p as the three words of its pt_t, flag byte fl, in bytes four at a time: bit d of b spread to byte d
 * (the product puts bit j of its four-bit factor at bit 8 j) times the step, subtracted per byte; a kept child lies in the
 * box, so no byte overflows.  Bytes from D on are 0.  Cells that the caller does not keep 4-byte aligned are
 * read byte by byte */
__device__ __forceinline__ void child_words(const signed char *p, int D, int st, int b, signed char fl, unsigned *w){
    if(((size_t)p & 3) == 0){ w[0] = ((const unsigned*)p)[0]; w[1] = ((const unsigned*)p)[1]; w[2] = ((const unsigned*)p)[2]; }
    else for(int q = 0; q < 3; q++) w[q] = (unsigned char)p[4*q] | (unsigned)(unsigned char)p[4*q + 1] << 8 |
                                           (unsigned)(unsigned char)p[4*q + 2] << 16 | (unsigned)(unsigned char)p[4*q + 3] << 24;
#pragma unroll
    for(int q = 0; q < 3; q++){
        const unsigned sub = ((((unsigned)b >> (4*q)) & 15u)*0x00204081u & 0x01010101u)*(unsigned)st;
        const int nb = D - 4*q;                                    /* axes in this word */
        const unsigned keep = nb >= 4 ? 0xffffffffu : nb <= 0 ? 0u : (1u << (8*nb)) - 1;
        w[q] = __vsub4(w[q], sub) & keep;
    }
    w[2] = (w[2] & 0x00ffffffu) | ((unsigned)(unsigned char)fl << 24);
}
/* a present child's multiplicity: its orbit size under a fold, else 1 */
__device__ __forceinline__ int child_weight(const lvl_t &a, const lvi_t &L, long il){
    if(a.cw) return a.cw[il];
    if(a.sym.n <= 1) return 1;
    int k[SQB_MAXD];
    child_of(a, L, il, k);
    return sqb_orbit_n(a.sym, k, a.D);
}

__device__ __forceinline__ int parent_tier(const lvl_t &a, const lvi_t &L, long i, long il){
    if(a.cfl) return (a.cfl[i] >> 1) & 3;
    const long c = il >> a.D;
    return (L.cells[c*SQB_MAXD + SQB_PFLAG] >> 1) & 3;
}

/* one child's part of a tile's sums */
struct rsum_t { sqdd S, b1, b2; double A, dr, uu; unsigned ne, nq, nu, nsk, keep; };
__device__ __forceinline__ void rsum_add(rsum_t &x, const lvl_t &a, const lvi_t &L, long i, unsigned char s, double v, double u){
    /* a folded point stands for its orbit: (mw v) pw and mw |v| (driver/sum.c:734-745) */
    const long il = i - L.child0;
    const int mw = child_weight(a, L, il);
    const double m = (double)mw, vp = (m*v)*L.pw, av = fabs(v);
    x.S = sqdd_add_d(x.S, vp); x.A += m*av; x.ne++;
    x.nsk += (s & SQB_SKIPPED) ? 1 : 0;
    if(s & SQB_FALLBACK){ x.nq++; x.uu += u; }
    if(s & SQB_UNRES) x.nu++;
    if(L.last){
        const int te = parent_tier(a, L, i, il);
        if(te >= 1) x.b1 = sqdd_add_d(x.b1, vp);
        if(te >= 2) x.b2 = sqdd_add_d(x.b2, vp);
    } else if(av >= L.thr) x.keep += mw;
    else x.dr += (m*av)*L.pw;
}
/* per tile of RTILE children: S = sum v*pw and the shadow-tier sums in double-double per thread (they
 * can cancel), sum |v|, the dropped weight and the round column (non-negative) in double per thread,
 * then double-double across threads in a fixed tree; the order is fixed, so a run is reproducible.  tfb[tile] says
 * what the FP64 pass left: 0 = nothing; 2 = the tile's fallback points, to be added to its sums (a thread finds them
 * among sixteen consecutive children by one load of their statuses); 1 (or no tfb) = the whole tile, thread t taking
 * children t, t + RT, t + 2 RT, ... (each warp reads 256 contiguous bytes of v per step). */
__global__ void __launch_bounds__(RT) sqb_k_reduce(const __grid_constant__ lvl_t a, part_t *bp, unsigned *bkeep,
                                                   const unsigned char *tfb){
    const int mode = tfb ? tfb[blockIdx.x] : 1;
    if(mode == 0) return;
    const lvi_t L = lvl_inst(a, blockIdx.x);
    rsum_t rs; rs.A = rs.dr = rs.uu = 0; rs.ne = rs.nq = rs.nu = rs.nsk = rs.keep = 0;
    if(mode == 2){
        const long t0 = blockIdx.x*(long)RTILE + threadIdx.x*(long)RPT;
        const uint4 q = *(const uint4*)(a.stt + t0);
        const unsigned w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll 1
        for(int h = 0; h < 4; h++)
            for(unsigned b = w[h] & (SQB_FALLBACK*0x01010101u); b; b &= b - 1){
                const int j = 4*h + ((__ffs(b) - 1) >> 3);
                const long i = t0 + j;
                if(i - L.child0 < L.n) rsum_add(rs, a, L, i, a.stt[i], a.v[i], a.uu[i]);
            }
    } else {
        const long t0 = blockIdx.x*(long)RTILE + threadIdx.x;
        /* four children's loads at a time, in flight together (a load per child left each waiting for the one before) */
#pragma unroll 1
        for(int j0 = 0; j0 < RPT; j0 += 4){
            unsigned char st_[4]; double v_[4], u_[4];
#pragma unroll
            for(int j = 0; j < 4; j++){
                const long i = t0 + (long)(j0 + j)*RT;
                const bool in = i - L.child0 < L.n;
                st_[j] = in ? a.stt[i] : 0; v_[j] = in ? a.v[i] : 0.0;
            }
#pragma unroll
            for(int j = 0; j < 4; j++) u_[j] = (st_[j] & SQB_FALLBACK) ? a.uu[t0 + (long)(j0 + j)*RT] : 0.0;
#pragma unroll
            for(int j = 0; j < 4; j++) if(st_[j] & SQB_PRESENT) rsum_add(rs, a, L, t0 + (long)(j0 + j)*RT, st_[j], v_[j], u_[j]);
        }
    }
    sqdd S = rs.S, b1 = rs.b1, b2 = rs.b2;
    unsigned ne = rs.ne, nq = rs.nq, nu = rs.nu, nsk = rs.nsk, keep = rs.keep;
    const double A = rs.A, dr = rs.dr, uu = rs.uu;
    sqdd Ad(A), dd(dr), ud(uu);
    if(__any_sync(0xffffffffu, ne))                    /* a warp without a child to add has zeros */
    for(int off = 16; off; off >>= 1){
        S = S + shfl_dd(S, off); Ad = Ad + shfl_dd(Ad, off); dd = dd + shfl_dd(dd, off);
        b1 = b1 + shfl_dd(b1, off); b2 = b2 + shfl_dd(b2, off); ud = ud + shfl_dd(ud, off);
        ne += __shfl_down_sync(0xffffffffu, ne, off); nq += __shfl_down_sync(0xffffffffu, nq, off);
        nu += __shfl_down_sync(0xffffffffu, nu, off); nsk += __shfl_down_sync(0xffffffffu, nsk, off);
        keep += __shfl_down_sync(0xffffffffu, keep, off);
    }
    __shared__ double wd[RT/32][12];
    __shared__ unsigned wc[RT/32][5];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if(l == 0){
        wd[w][0] = S.hi; wd[w][1] = S.lo; wd[w][2] = Ad.hi; wd[w][3] = Ad.lo; wd[w][4] = dd.hi; wd[w][5] = dd.lo;
        wd[w][6] = b1.hi; wd[w][7] = b1.lo; wd[w][8] = b2.hi; wd[w][9] = b2.lo; wd[w][10] = ud.hi; wd[w][11] = ud.lo;
        wc[w][0] = ne; wc[w][1] = nq; wc[w][2] = nu; wc[w][3] = nsk; wc[w][4] = keep;
    }
    __syncthreads();
    if(w == 0){
        const int nw = RT/32;
        sqdd x[6]; unsigned c[5];
        for(int q = 0; q < 6; q++) x[q] = l < nw ? sqdd(wd[l][2*q], wd[l][2*q + 1]) : sqdd(0.0);
        for(int q = 0; q < 5; q++) c[q] = l < nw ? wc[l][q] : 0;
        for(int off = nw/2; off; off >>= 1){
            for(int q = 0; q < 6; q++) x[q] = x[q] + shfl_dd(x[q], off);
            for(int q = 0; q < 5; q++) c[q] += __shfl_down_sync(0xffffffffu, c[q], off);
        }
        if(l == 0){
            part_t p;
            p.S[0] = x[0].hi; p.S[1] = x[0].lo; p.A[0] = x[1].hi; p.A[1] = x[1].lo; p.drop[0] = x[2].hi; p.drop[1] = x[2].lo;
            p.b1[0] = x[3].hi; p.b1[1] = x[3].lo; p.b2[0] = x[4].hi; p.b2[1] = x[4].lo; p.u[0] = x[5].hi; p.u[1] = x[5].lo;
            p.ne = c[0]; p.nq = c[1]; p.unres = c[2]; p.skipped = c[3];
            if(mode == 2){
                const part_t o = bp[blockIdx.x];
                const sqdd z[6] = {x[0] + sqdd(o.S[0], o.S[1]), x[1] + sqdd(o.A[0], o.A[1]), x[2] + sqdd(o.drop[0], o.drop[1]),
                                   x[3] + sqdd(o.b1[0], o.b1[1]), x[4] + sqdd(o.b2[0], o.b2[1]), x[5] + sqdd(o.u[0], o.u[1])};
                p.S[0] = z[0].hi; p.S[1] = z[0].lo; p.A[0] = z[1].hi; p.A[1] = z[1].lo; p.drop[0] = z[2].hi; p.drop[1] = z[2].lo;
                p.b1[0] = z[3].hi; p.b1[1] = z[3].lo; p.b2[0] = z[4].hi; p.b2[1] = z[4].lo; p.u[0] = z[5].hi; p.u[1] = z[5].lo;
                p.ne += o.ne; p.nq += o.nq; p.unres += o.unres; p.skipped += o.skipped;
                c[4] += bkeep[blockIdx.x];
            }
            bp[blockIdx.x] = p; bkeep[blockIdx.x] = c[4];
        }
    }
}

/* the tiles' offsets (exclusive scan of their kept counts) and the batch's sums, in a fixed order, added into the level
 * accumulator; *base = this batch's first slot in the next list.  One CTA per FT tiles of an integral (blockIdx.y: the
 * integral of a multi-instance batch, with its own accumulator and base), a tile per thread; the CTA that is
 * done last adds the CTAs' sums and scans their kept counts (a tile's offset is boff[tile] after coff[its CTA]).  Latency
 * bounds it: one CTA of 1024 threads, a run of consecutive tiles each, took 79 us for the 8192 tiles of a full batch,
 * and the reduce kernel 52 us with a fallback point or more in a third of them; together 30 us now (syn_d8, h = 0.7). */
__device__ __forceinline__ unsigned long long scan256(unsigned long long v, unsigned long long *ws, unsigned long long *total){
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    unsigned long long inc = v;
    for(int off = 1; off < 32; off <<= 1){ const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, off); if(l >= off) inc += y; }
    if(l == 31) ws[w] = inc;
    __syncthreads();
    unsigned long long o = inc - v, t = 0;
    for(int q = 0; q < FT/32; q++){ if(q < w) o += ws[q]; t += ws[q]; }
    __syncthreads();
    *total = t;
    return o;
}
/* the CTA's six sums and four counts, in warp w's lane 0 (sum w of x in warp w < 6, the counts in warp 6) */
__device__ __forceinline__ void fin_sums(sqdd (&x)[6], unsigned long long (&c)[4], double (*wd)[12], unsigned long long (*wc)[4]){
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    for(int off = 16; off; off >>= 1){
#pragma unroll
        for(int q = 0; q < 6; q++) x[q] = x[q] + shfl_dd(x[q], off);
#pragma unroll
        for(int q = 0; q < 4; q++) c[q] += __shfl_down_sync(0xffffffffu, c[q], off);
    }
    if(l == 0){
#pragma unroll
        for(int q = 0; q < 6; q++){ wd[w][2*q] = x[q].hi; wd[w][2*q + 1] = x[q].lo; }
#pragma unroll
        for(int q = 0; q < 4; q++) wc[w][q] = c[q];
    }
    __syncthreads();
    if(w < 6){
        sqdd y = l < FT/32 ? sqdd(wd[l][2*w], wd[l][2*w + 1]) : sqdd(0.0);
        for(int off = FT/64; off; off >>= 1) y = y + shfl_dd(y, off);
        x[0] = y;
    } else if(w == 6) for(int q = 0; q < 4; q++){ c[q] = 0; for(int j = 0; j < FT/32; j++) c[q] += wc[j][q]; }
}
__global__ void __launch_bounds__(FT) sqb_k_finish(const __grid_constant__ lvl_t a, const part_t *bp, const unsigned *bkeep,
                                                   long nb, unsigned long long *boff, sqb_acc_t *acc, unsigned long long *base,
                                                   fpart_t *fp, unsigned long long *coff, unsigned *fcnt){
    __shared__ double wd[FT/32][12];
    __shared__ unsigned long long wc[FT/32][4], ws[FT/32];
    __shared__ int last_;
    const int t = threadIdx.x, w = t >> 5, l = t & 31, k = blockIdx.y;
    long tb = 0;
    if(a.ninst > 0){
        const lvi_t &L = a.inst[k];
        tb = L.child0/RTILE; nb = (L.n + RTILE - 1)/RTILE; acc = L.acc; base = L.base;
    }
    const long nch = (nb + FT - 1)/FT, ch = blockIdx.x, j = ch*FT + t;
    if(ch >= nch) return;
    const long slot0 = fin_slot(tb, k, tb);
    sqdd x[6]; unsigned long long c[4] = {0, 0, 0, 0}, kp = 0, total;
    if(j < nb){
        const part_t &p = bp[tb + j];
        x[0] = sqdd(p.S[0], p.S[1]); x[1] = sqdd(p.A[0], p.A[1]); x[2] = sqdd(p.drop[0], p.drop[1]);
        x[3] = sqdd(p.b1[0], p.b1[1]); x[4] = sqdd(p.b2[0], p.b2[1]); x[5] = sqdd(p.u[0], p.u[1]);
        c[0] = p.ne; c[1] = p.nq; c[2] = p.unres; c[3] = p.skipped; kp = bkeep[tb + j];
    }
    const unsigned long long o = scan256(kp, ws, &total);
    if(j < nb) boff[tb + j] = o;
    fin_sums(x, c, wd, wc);
    if(nch > 1){
        fpart_t &f = fp[slot0 + ch];
        if(l == 0 && w < 6){ f.x[w][0] = x[0].hi; f.x[w][1] = x[0].lo; }
        if(t == 192){ for(int q = 0; q < 4; q++) f.c[q] = c[q]; f.c[4] = total; }
        __threadfence();
        __syncthreads();
        if(t == 0) last_ = atomicAdd(&fcnt[k], 1u) == (unsigned)nch - 1;
        __syncthreads();
        if(!last_) return;
        __threadfence();
        for(int q = 0; q < 6; q++) x[q] = sqdd(0.0);
        for(int q = 0; q < 4; q++) c[q] = 0;
        unsigned long long sum = 0;
        for(long b = 0; b < nch; b += FT){
            unsigned long long kc = 0;
            if(b + t < nch){
                const fpart_t &g = fp[slot0 + b + t];
#pragma unroll
                for(int q = 0; q < 6; q++) x[q] = x[q] + sqdd(__ldcg(&g.x[q][0]), __ldcg(&g.x[q][1]));
#pragma unroll
                for(int q = 0; q < 4; q++) c[q] += __ldcg(&g.c[q]);
                kc = __ldcg(&g.c[4]);
            }
            const unsigned long long oc = scan256(kc, ws, &total);
            if(b + t < nch) coff[slot0 + b + t] = sum + oc;
            sum += total;
        }
        total = sum;
        fin_sums(x, c, wd, wc);
        if(t == 0) fcnt[k] = 0;
    } else if(t == 0) coff[slot0] = 0;
    double *dst[6] = {acc->S, acc->A, acc->drop, acc->b1, acc->b2, acc->u};
    if(l == 0 && w < 6){ const sqdd z = sqdd(dst[w][0], dst[w][1]) + x[0]; dst[w][0] = z.hi; dst[w][1] = z.lo; }
    if(t == 192){
        acc->ne += c[0]; acc->nq += c[1]; acc->unres += c[2]; acc->skipped += c[3];
        *base = acc->keep; acc->keep += total;
    }
}

__global__ void __launch_bounds__(RT) sqb_k_scatter(const __grid_constant__ lvl_t a, const unsigned long long *boff,
                                                    const unsigned long long *coff, const unsigned long long *base, sqb_pt_t *next,
                                                    long cap, unsigned long long *overflow){
    int ki;
    const lvi_t L = lvl_inst(a, blockIdx.x, &ki);
    const long slot = fin_slot(L.child0/RTILE, ki, blockIdx.x);
    if(a.ninst > 0){ base = L.base; next = L.next; cap = L.cap; overflow = &L.acc->overflow; }
    const long t0 = blockIdx.x*(long)RTILE + threadIdx.x*(long)RPT;
    unsigned mask = 0; int cnt = 0;
    /* the thread's sixteen statuses in one load and its values in eight, before anything depends on them (the arrays
     * hold whole tiles, and a tile starts at a multiple of RTILE: the vectors are aligned and in bounds) */
    static_assert(RPT == 16, "one 16-byte load of statuses per thread");
    {
        union { uint4 q; unsigned char c[RPT]; } sv;
        double2 vv[RPT/2];
        sv.q = *(const uint4*)(a.stt + t0);
#pragma unroll
        for(int j = 0; j < RPT/2; j++) vv[j] = *(const double2*)(a.v + t0 + 2*j);
#pragma unroll
        for(int j = 0; j < RPT; j++)
            if(t0 + j - L.child0 < L.n && (sv.c[j] & SQB_PRESENT) && fabs(j & 1 ? vv[j/2].y : vv[j/2].x) >= L.thr) mask |= 1u << j;
    }
    if(!a.cw && a.sym.n <= 1) cnt = __popc(mask);
    else for(unsigned b = mask; b; b &= b - 1) cnt += child_weight(a, L, t0 + __ffs(b) - 1 - L.child0);
    /* block exclusive scan of cnt */
    __shared__ int ws[RT/32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    int x = cnt;
    for(int off = 1; off < 32; off <<= 1){ int y = __shfl_up_sync(0xffffffffu, x, off); if(l >= off) x += y; }
    if(l == 31) ws[w] = x;
    __syncthreads();
    if(threadIdx.x == 0){ int s = 0; for(int j = 0; j < RT/32; j++){ int y = ws[j]; ws[j] = s; s += y; } }
    __syncthreads();
    unsigned long long o = *base + coff[slot] + boff[blockIdx.x] + (unsigned long long)(ws[w] + x - cnt);
    const double thr10 = 10*L.thr, thr100 = 100*L.thr;
    for(unsigned b = mask; b; b &= b - 1){
        const long i = t0 + __ffs(b) - 1, il = i - L.child0;
        const long c = il >> a.D;
        const signed char *p = L.cells + c*SQB_MAXD;
        const unsigned char s = a.stt[i];
        const double av = fabs(a.v[i]);
        const int te = (p[SQB_PFLAG] >> 1) & 3, tv = (av >= thr10) + (av >= thr100);
        const int psk = (s & SQB_SKIPPED) ? 1 : 0, nr = (s & SQB_NEAR) ? 1 : 0;
        const signed char fl = (signed char)((a.abskip && (psk || !nr)) | ((te < tv ? te : tv) << 1));
        if(a.sym.n <= 1){
            if((long)o >= cap) atomicAdd(overflow, 1ULL);
            else {
                unsigned w3[3];
                child_words(p, a.D, L.st, (int)(il & ((1L << a.D) - 1)), fl, w3);
                unsigned *dst = (unsigned*)(next + o);
                dst[0] = w3[0]; dst[1] = w3[1]; dst[2] = w3[2];
            }
            o++;
            continue;
        }
        int k[SQB_MAXD];
        child_of(a, L, il, k);
        /* the child, then the other members of its orbit in group order, each once
         * (symorbit(), driver/sum.c:38-46), all with the child's flags (driver/sum.c:741-744) */
        for(int e = 0; e < a.sym.n; e++){
            if(!sqb_image_new(a.sym, k, a.D, e)) continue;
            if((long)o >= cap){ atomicAdd(overflow, 1ULL); o++; continue; }
            union { signed char k[SQB_MAXD]; int w[3]; } q;
            q.w[0] = q.w[1] = q.w[2] = 0;
            int im[SQB_MAXD];
            sqb_image(a.sym, k, a.D, e, im);
            for(int d = 0; d < a.D; d++) q.k[d] = (signed char)im[d];
            q.k[SQB_PFLAG] = fl;
            int *dst = (int*)(next + o);
            dst[0] = q.w[0]; dst[1] = q.w[1]; dst[2] = q.w[2];
            o++;
        }
    }
}

/* list mode: the children of one level batch to evaluate -- in the box, not left out by the predictor and,
 * under a fold, the minimum of their orbit (driver/sum.c:405-416) -- appended to sel as child index | orbit
 * weight << SQB_SEL_SHIFT, in no particular order (each child's value and status go to its own slot, and
 * the reduce kernel sums them in child order).  The other children get value 0 and no status; cw holds
 * every child's weight (0: not evaluated) for the reduce and scatter kernels. */
__global__ void __launch_bounds__(RT) sqb_k_select(const __grid_constant__ lvl_t a, int K, unsigned long long *sel,
                                                   unsigned long long *nsel, double *v, unsigned char *stt,
                                                   unsigned char *cw){
    const lvi_t L = lvl_inst(a, 0);
    const int lane = threadIdx.x & 31;
    for(long b0 = blockIdx.x*(long)RT; b0 < a.n; b0 += (long)gridDim.x*RT){     /* the same trips for a warp */
        const long i = b0 + threadIdx.x;
        int mw = 0;
        if(i < a.n){
            int k[SQB_MAXD]; bool in = true;
            child_of(a, L, i, k);
            for(int d = 0; d < a.D; d++) in = in && k[d] >= -K;
            if(in && !(a.cfl && (a.cfl[i] & 1))) mw = a.sym.n > 1 ? sqb_orbit_n(a.sym, k, a.D) : 1;
            cw[i] = (unsigned char)mw;
            if(!mw){ v[i] = 0; stt[i] = 0; }
        }
        const unsigned m = __ballot_sync(0xffffffffu, mw > 0);
        unsigned long long base = 0;
        if(lane == 0 && m) base = atomicAdd(nsel, (unsigned long long)__popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if(mw > 0) sel[base + __popc(m & ((1u << lane) - 1))] = (unsigned long long)i | ((unsigned long long)mw << SQB_SEL_SHIFT);
    }
}

extern "C" int sqb_dev_level(const sqb_level_t *L, sqb_acc_t *acc, long *next_n, double *ms){
    const sqb_graph_t *g = L->g; const int D = g->D;
    long maxch = batch_children(g, L), ncb;
again:
    if(maxch < (1L << D)) maxch = 1L << D;
    ncb = maxch >> D;
    /* full batches hold whole rounds of tiles: the FP64 kernel's cap resident CTAs take tiles b, b + cap,
     * ..., so with a multiple of cap tiles every CTA takes the same number and none idles while others
     * finish one more */
    {
        int can0 = 0;
        const long cap0 = grid_cap(g, f64_which(g, L->t.fma) | SQB_ATTR_LEVEL, 2*(2*G.K + 1)*sizeof(double), &can0);
        const long round = (cap0*SQB_TILE) >> D;            /* cells per round (SQB_TILE >= 2^D) */
        if(!L->t.alldd && can0 && round > 0 && ncb >= 2*round) ncb = (ncb/round)*round;
    }
    /* a small level reserves the lower size, so that the next ones find it */
    const long low = CHILDREN_LOW >> D, need = L->ncell > low ? L->ncell : low;
    if(reserve_points((need < ncb ? need : ncb) << D)){
        if(L->max_children > 0 || maxch <= CHILDREN_LOW) return -1;
        maxch = CHILDREN_LOW;
        goto again;
    }
    /* the predictor runs at the last level when its table holds values (driver/sum.c:385) */
    bool pon = false;
    if(L->last && L->predict > 0 && L->vt && L->vt->tab){
        long vn = 0, full = 0;
        if(sqb_vtab_counts(L->vt, &vn, &full, G.s)){ snprintf(g_err, sizeof g_err, "%s", sqb_vtab_error()); return -1; }
        pon = vn > 0;
    }
    CKR(cudaMemsetAsync(G.acc, 0, sizeof(sqb_acc_t), G.s));
    CKR(cudaEventRecord(G.e0, G.s));
    for(long c0 = 0; c0 < L->ncell; c0 += ncb){
        const long nc = L->ncell - c0 < ncb ? L->ncell - c0 : ncb, nch = nc << D;
        const sqb_pt_t *cells = L->cells + c0;
        sqb_eval_t a; memset(&a, 0, sizeof a); fill_eval(&a, &L->t);
        a.pts = cells; a.n = nc; a.esize = 1; a.stride = SQB_MAXD; a.flag_at = SQB_PFLAG; a.cells = 1; a.st = L->st;
        if(L->sym && L->sym->n > 1){
            bool ok = L->sym->n <= SQB_SYMG;
            for(int e = 0; ok && e < L->sym->n; e++) for(int i = 0; i < D; i++) ok = ok && L->sym->g[e][i] >= 0 && L->sym->g[e][i] < D;
            if(!ok){ snprintf(g_err, sizeof g_err, "symmetry group: %d elements or an axis outside 0..%d", L->sym->n, D - 1); return -1; }
            a.sym = *L->sym;
        }
        /* level mode: the FP64 pass sums the tiles without fallback points (the all-dd form has no FP64
         * pass: the reduce kernel sums every tile) */
        /* the FP64 pass as a persistent grid taking tiles from the device queue (one integral: ninst = 1);
         * under a fold or the predictor it walks the list of children to evaluate (list mode), and the
         * reduce kernel sums every tile */
        const bool queue = !L->t.alldd && !use_split(g, &a, &L->t);
        /* list mode pays where the orbit test is costly or many children are left out: a group of order
         * 4 or more, or the predictor (measured on four-loop VP integrals: order 8, 1.5x faster; order 2,
         * 16 % slower than testing in place) */
        const bool listm = queue && (a.sym.n >= 4 || pon);
        /* the kernel that runs: the level kernel for a queue batch outside list mode */
        int can = 0;
        const long cap = grid_cap(g, f64_which(g, L->t.fma) | (queue && !listm ? SQB_ATTR_LEVEL : 0),
                                  2*(2*G.K + 1)*sizeof(double), &can);
        const bool fused = tile_sums() && !L->t.alldd && can && !use_split(g, &a, &L->t) && !listm && fuses(L->ncell, ncb, D, cap);
        /* the predictor at the last level: which children to leave out, and their tiers */
        if(pon){
            if(sqb_vtab_predict(L->vt, cells, nc, D, L->st, G.K, L->thr, L->predict, L->esok, L->sym, G.cfl,
                                &G.acc->pskip, G.nsm, G.s)){ snprintf(g_err, sizeof g_err, "%s", sqb_vtab_error()); return -1; }
            G.launches++;
            a.cfl = G.cfl;
        }
        if(fused){ a.part = G.bp; a.tkeep = G.bkeep; a.tfb = G.tfb; a.pw = L->pw; a.thr = L->thr; a.last = L->last; }
        if(queue){
            a.part = G.bp; a.tkeep = G.bkeep; a.tfb = G.tfb;     /* every tile summed or flagged for the reduce */
            a.ninst = 1; a.ntile = (nch + SQB_TILE - 1)/SQB_TILE; a.queue = G.queue;
            sqb_inst_t &I = a.inst[0];
            I.pts = cells; I.n = nc; I.child0 = 0; I.st = L->st; I.K = G.K; I.toff = 0; I.fused = fused;
            I.last = L->last; I.pw = L->pw; I.thr = L->thr; I.abserr = L->t.abserr; I.near_thr = L->t.nearf*L->t.abserr;
            I.X = G.X; I.Wt = G.Wt; I.U = G.U; I.Ud = G.Ud;
            a.sub = fused ? 1 : SQB_SUB;
        }
        lvl_t r; memset(&r, 0, sizeof r);
        r.cells = (const signed char*)cells; r.n = nch; r.D = D; r.st = L->st; r.last = L->last;
        r.abskip = L->t.abskip; r.pw = L->pw; r.thr = L->thr; r.v = G.v; r.uu = G.uu; r.stt = G.stt;
        r.sym = a.sym; r.cfl = a.cfl;
        const long nb = (nch + RTILE - 1)/RTILE;
        if(listm){
            CKR(cudaMemsetAsync(G.nsel, 0, sizeof(unsigned long long), G.s));
            CKR(cudaMemsetAsync(G.tfb, 1, nb, G.s));
            const long want = (nch + RT - 1)/RT, full = (long)G.nsm*8;
            sqb_k_select<<<(unsigned)(want < full ? want : full), RT, 0, G.s>>>(r, G.K, G.sel, G.nsel, G.v, G.stt, G.cw);
            CKR(cudaGetLastError());
            G.launches++;
            a.sel = G.sel; a.nsel = G.nsel;
            r.cw = G.cw;
        }
        if(eval_batch(g, &a, &L->t, nch)) return -1;
        /* the level before the last stores its values for the predictor */
        if(L->vput && L->vt){
            if(sqb_vtab_put_children(L->vt, cells, nch, D, L->st, G.v, G.stt, L->sym, G.s)){
                snprintf(g_err, sizeof g_err, "%s", sqb_vtab_error()); return -1; }
            G.launches++;
        }
        sqb_k_reduce<<<(unsigned)nb, RT, 0, G.s>>>(r, G.bp, G.bkeep, fused || queue ? G.tfb : NULL);
        CKR(cudaGetLastError());
        sqb_k_finish<<<(unsigned)((nb + FT - 1)/FT), FT, 0, G.s>>>(r, G.bp, G.bkeep, nb, G.boff, G.acc, G.base, G.fp, G.coff, G.fcnt);
        CKR(cudaGetLastError());
        G.launches += 2;
        if(!L->last){
            sqb_k_scatter<<<(unsigned)nb, RT, 0, G.s>>>(r, G.boff, G.coff, G.base, L->next, L->next_cap, &G.acc->overflow);
            CKR(cudaGetLastError());
            G.launches++;
        }
    }
    CKR(cudaEventRecord(G.e1, G.s));
    sqb_acc_t h;
    CKR(cudaMemcpyAsync(&h, G.acc, sizeof h, cudaMemcpyDeviceToHost, G.s));
    CKR(cudaStreamSynchronize(G.s));
    D2H += sizeof h;
    float t = 0; cudaEventElapsedTime(&t, G.e0, G.e1); if(ms) *ms = t;
    double *src[6] = {h.S, h.A, h.drop, h.b1, h.b2, h.u}, *dst[6] = {acc->S, acc->A, acc->drop, acc->b1, acc->b2, acc->u};
    for(int q = 0; q < 6; q++){ sqdd x = sqdd(dst[q][0], dst[q][1]) + sqdd(src[q][0], src[q][1]); dst[q][0] = x.hi; dst[q][1] = x.lo; }
    acc->ne += h.ne; acc->nq += h.nq; acc->unres += h.unres; acc->skipped += h.skipped; acc->keep += h.keep; acc->overflow += h.overflow;
    acc->pskip += h.pskip;
    *next_n = (long)h.keep;
    return 0;
}

/* an integral's axis tables: they follow X and Wt (sqb_level_t) when the graph has the axis form */
static const double *level_axis(const sqb_level_t &L, int dd){
    if(!L.X || !L.g->axis) return NULL;
    return L.X + 2*(2*L.K + 1) + (dd ? axis_words(L.g, L.K, 0) : 0);
}

/* A level of several integrals of one graph at once (see sqb_rt.h).  Each integral keeps the batches,
 * tiles and fused/unfused choice that sqb_dev_level would give it alone; round r launches batch r of every
 * integral that has one, its children numbered integral after integral from tile boundaries, in as few launches of up
 * to GROUP_CHILDREN as hold them. */
extern "C" int sqb_dev_level_multi(const sqb_level_t *Ls, int n, sqb_acc_t *accs, long *next_n, double *ms){
    if(n <= 0) return 0;
    bool one_by_one = n == 1 || n > SQB_MAXINST;
    const sqb_graph_t *g = Ls[0].g; const int D = g->D;
    for(int k = 0; k < n && !one_by_one; k++){
        const sqb_level_t &L = Ls[k];
        one_by_one = L.g != g || L.t.alldd || L.t.split || L.predict > 0 || L.vput || L.st != Ls[0].st ||
                     L.last != Ls[0].last || !L.X || !L.Wt || L.K < 1 || L.K > 127 || L.t.fma != Ls[0].t.fma ||
                     L.t.split != Ls[0].t.split || L.t.abskip != Ls[0].t.abskip || L.t.abcheck != Ls[0].t.abcheck ||
                     L.t.dropunres != Ls[0].t.dropunres || L.t.ddslack != Ls[0].t.ddslack ||
                     ((L.sym && L.sym->n > 1) != (Ls[0].sym && Ls[0].sym->n > 1)) ||
                     (L.sym && Ls[0].sym && L.sym->n > 1 && memcmp(L.sym, Ls[0].sym, sizeof(sqb_sym_t)));
    }
    if(one_by_one){
one_by_one:
        /* each integral on its own tables: the thread's current ones are lent the integral's device copy */
        double tot = 0; int rc = 0;
        double *sx = G.X, *sw = G.Wt; const int sk = G.K; const double *su = G.U, *sd = G.Ud;
        for(int k = 0; k < n && !rc; k++){
            if(Ls[k].X){
                G.X = (double*)Ls[k].X; G.Wt = (double*)Ls[k].Wt; G.K = Ls[k].K;
                G.U = level_axis(Ls[k], 0); G.Ud = level_axis(Ls[k], 1);
            }
            double m = 0;
            rc = sqb_dev_level(&Ls[k], &accs[k], &next_n[k], &m);
            tot += m;
            G.X = sx; G.Wt = sw; G.K = sk; G.U = su; G.Ud = sd;
        }
        if(ms) *ms = tot;
        return rc;
    }
    const sqb_level_t &L0 = Ls[0];
    if(L0.sym && L0.sym->n > 1){
        bool ok = L0.sym->n <= SQB_SYMG;
        for(int e = 0; ok && e < L0.sym->n; e++) for(int i = 0; i < D; i++) ok = ok && L0.sym->g[e][i] >= 0 && L0.sym->g[e][i] < D;
        if(!ok){ snprintf(g_err, sizeof g_err, "symmetry group: %d elements or an axis outside 0..%d", L0.sym->n, D - 1); return -1; }
    }
    /* per integral: cells per batch and the number of batches, as sqb_dev_level chooses them */
    long ncb[SQB_MAXINST], nbat[SQB_MAXINST], capk[SQB_MAXINST]; int cank[SQB_MAXINST]; long rounds = 0;
    const int which = f64_which(g, L0.t.fma);
    for(int k = 0; k < n; k++){
        const sqb_level_t &L = Ls[k];
        long maxch = batch_children(g, &L);
        if(maxch < (1L << D)) maxch = 1L << D;
        long c = maxch >> D;
        const size_t sm1 = 2*(2*(size_t)L.K + 1)*sizeof(double);
        int can0 = 0;
        const long cap0 = grid_cap(g, which | SQB_ATTR_LEVEL, sm1, &can0);
        const long round = (cap0*SQB_TILE) >> D;
        if(can0 && round > 0 && c >= 2*round) c = (c/round)*round;
        ncb[k] = c; capk[k] = cap0; cank[k] = can0;
        nbat[k] = (L.ncell + c - 1)/c;
        if(nbat[k] > rounds) rounds = nbat[k];
    }
    /* the children of integral k's batch r, from a tile boundary; the largest launch's children */
    const auto batch_tiles = [&](int k, long r){
        const long nc = Ls[k].ncell - r*ncb[k] < ncb[k] ? Ls[k].ncell - r*ncb[k] : ncb[k];
        return ((nc << D) + SQB_TILE - 1)/SQB_TILE*SQB_TILE;
    };
    long maxtot = 0;
    for(long r = 0; r < rounds; r++){
        long tot = 0;
        for(int k = 0; k < n; k++) if(r < nbat[k]){
            const long b = batch_tiles(k, r);
            if(tot > 0 && tot + b > GROUP_CHILDREN) tot = 0;
            tot += b;
            if(tot > maxtot) maxtot = tot;
        }
    }
    if(reserve_points(maxtot)) goto one_by_one;                /* no room for all at once */
    CKR(cudaMemsetAsync(G.accm, 0, n*sizeof(sqb_acc_t), G.s));
    CKR(cudaEventRecord(G.e0, G.s));
    for(long r = 0; r < rounds; r++) for(int k0 = 0; k0 < n;){
        sqb_eval_t a; memset(&a, 0, sizeof a); fill_eval(&a, &L0.t);
        a.esize = 1; a.stride = SQB_MAXD; a.flag_at = SQB_PFLAG; a.cells = 1;
        if(L0.sym && L0.sym->n > 1) a.sym = *L0.sym;
        a.part = G.bp; a.tkeep = G.bkeep; a.tfb = G.tfb; a.queue = G.queue;
        lvl_t rl; memset(&rl, 0, sizeof rl);
        rl.D = D; rl.abskip = L0.t.abskip; rl.v = G.v; rl.uu = G.uu; rl.stt = G.stt; rl.sym = a.sym;
        long child0 = 0; int m = 0, toff = 0, last = 0;
        a.sub = SQB_SUB;
        /* the round's integrals in order, as many as a launch takes */
        for(; k0 < n; k0++){
            const int k = k0;
            if(r >= nbat[k]) continue;
            if(m > 0 && child0 + batch_tiles(k, r) > GROUP_CHILDREN) break;
            const sqb_level_t &L = Ls[k];
            const long c0 = r*ncb[k], nc = L.ncell - c0 < ncb[k] ? L.ncell - c0 : ncb[k], nch = nc << D;
            sqb_inst_t &I = a.inst[m];
            I.pts = L.cells + c0; I.n = nc; I.child0 = child0; I.st = L.st; I.K = L.K; I.toff = toff;
            I.fused = tile_sums() && cank[k] && fuses(L.ncell, ncb[k], D, capk[k]);
            I.last = L.last; I.pw = L.pw; I.thr = L.thr; I.abserr = L.t.abserr; I.near_thr = L.t.nearf*L.t.abserr;
            I.X = L.X; I.Wt = L.Wt; I.U = level_axis(L, 0); I.Ud = level_axis(L, 1);
            if(I.fused) a.sub = 1;
            lvi_t &V = rl.inst[m];
            V.cells = (const signed char*)(L.cells + c0); V.n = nch; V.child0 = child0; V.st = L.st; V.last = L.last;
            V.pw = L.pw; V.thr = L.thr; V.next = L.next; V.cap = L.next_cap; V.acc = G.accm + k; V.base = G.basem + k;
            last = L.last;
            toff += 2*(2*L.K + 1);
            child0 += (nch + SQB_TILE - 1)/SQB_TILE*SQB_TILE;
            m++;
        }
        if(!m) break;
        a.ninst = m; a.ntile = child0/SQB_TILE; rl.ninst = m;
        /* the per-point thresholds of the first integral stand in the launch's own fields (unused by the
         * kernels in a multi-instance launch) */
        if(eval_batch(g, &a, &Ls[0].t, child0)) return -1;
        sqb_k_reduce<<<(unsigned)a.ntile, RT, 0, G.s>>>(rl, G.bp, G.bkeep, G.tfb);
        CKR(cudaGetLastError());
        sqb_k_finish<<<dim3((unsigned)((a.ntile + FT - 1)/FT), (unsigned)m), FT, 0, G.s>>>(rl, G.bp, G.bkeep, 0, G.boff, NULL, NULL, G.fp, G.coff, G.fcnt);
        CKR(cudaGetLastError());
        G.launches += 2;
        if(!last){
            sqb_k_scatter<<<(unsigned)a.ntile, RT, 0, G.s>>>(rl, G.boff, G.coff, NULL, NULL, 0, NULL);
            CKR(cudaGetLastError());
            G.launches++;
        }
    }
    CKR(cudaEventRecord(G.e1, G.s));
    sqb_acc_t h[SQB_MAXINST];
    CKR(cudaMemcpyAsync(h, G.accm, n*sizeof(sqb_acc_t), cudaMemcpyDeviceToHost, G.s));
    CKR(cudaStreamSynchronize(G.s));
    D2H += n*sizeof(sqb_acc_t);
    float t = 0; cudaEventElapsedTime(&t, G.e0, G.e1); if(ms) *ms = t;
    for(int k = 0; k < n; k++){
        sqb_acc_t *acc = &accs[k];
        double *src[6] = {h[k].S, h[k].A, h[k].drop, h[k].b1, h[k].b2, h[k].u}, *dst[6] = {acc->S, acc->A, acc->drop, acc->b1, acc->b2, acc->u};
        for(int q = 0; q < 6; q++){ sqdd x = sqdd(dst[q][0], dst[q][1]) + sqdd(src[q][0], src[q][1]); dst[q][0] = x.hi; dst[q][1] = x.lo; }
        acc->ne += h[k].ne; acc->nq += h[k].nq; acc->unres += h[k].unres; acc->skipped += h[k].skipped;
        acc->keep += h[k].keep; acc->overflow += h[k].overflow; acc->pskip += h[k].pskip;
        next_n[k] = (long)h[k].keep;
    }
    return 0;
}

extern "C" void *sqb_dev_alloc(size_t bytes){ void *p = NULL; if(cudaMallocAsync(&p, bytes ? bytes : 16, G.s) != cudaSuccess){ cudaGetLastError(); return NULL; } return p; }
extern "C" void sqb_dev_free(void *p){ if(p) cudaFreeAsync(p, G.s); }
extern "C" int sqb_dev_upload(void *dst, const void *src, size_t bytes){
    CKR(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, G.s)); CKR(cudaStreamSynchronize(G.s)); H2D += bytes; return 0; }
extern "C" int sqb_dev_download(void *dst, const void *src, size_t bytes){
    CKR(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, G.s)); CKR(cudaStreamSynchronize(G.s)); D2H += bytes; return 0; }
extern "C" void sqb_dev_count_copy(unsigned long long h2d, unsigned long long d2h){ H2D += h2d; D2H += d2h; }

/* measurement helpers: bytes copied between host and device so far; events on the library's stream
 * around a region of work (device milliseconds); an L2 flush (a memset larger than L2) on that stream */
extern "C" void sqb_copy_bytes(unsigned long long *h2d, unsigned long long *d2h){ *h2d = H2D.load(); *d2h = D2H.load(); }
extern "C" int sqb_timer_start(void){ if(sqb_dev_init(0)) return -1; CKR(cudaEventRecord(G.t0, G.s)); return 0; }
extern "C" double sqb_timer_stop(void){
    if(cudaEventRecord(G.t1, G.s) != cudaSuccess || cudaEventSynchronize(G.t1) != cudaSuccess) return -1;
    float t = 0; cudaEventElapsedTime(&t, G.t0, G.t1); return t;
}
extern "C" int sqb_l2_flush(size_t bytes){
    if(sqb_dev_init(0)) return -1;
    if(bytes > G.flushn){ if(G.flush) cudaFree(G.flush); G.flush = NULL; CKR(cudaMalloc(&G.flush, bytes)); G.flushn = bytes; }
    CKR(cudaMemsetAsync(G.flush, G.launches & 255, bytes, G.s));
    return 0;
}
extern "C" size_t sqb_dev_free_bytes(void){ size_t f = 0, t = 0; cudaMemGetInfo(&f, &t); return f; }
extern "C" size_t sqb_dev_total_bytes(void){ size_t f = 0, t = 0; cudaMemGetInfo(&f, &t); return t; }

/* ------------------------------ plain form: the reference's GPU plug-in ABI ---------------------- */
/* Same contract as driver/gpu.cu:1-103: two slots, each with its own stream, event and pinned buffers;
 * gpu_submit* pack the coordinates (here to int8: |k| <= 127, driver/sq.h:117), copy, launch and copy
 * back f*w and |.|*w; gpu_wait waits for the slot.  SINCQED_GPU=0 turns the GPU off, SINCQED_GPU=d
 * picks device d-1.  CUDA errors print and exit(3), as the reference does. */
#define CKX(x) do { cudaError_t e_ = (x); if(e_ != cudaSuccess){ fprintf(stderr, "CUDA error %s at %s:%d: %s\n", #x, __FILE__, __LINE__, cudaGetErrorString(e_)); exit(3); } } while(0)

typedef struct { cudaStream_t st; cudaEvent_t ev; long cap, n; signed char *hK, *dK; unsigned char *hS, *dS; double *hF, *hA, *dF, *dA; } pslot_t;
static pslot_t PS[2];
static int PON = -1, PD, PK; static double PH;
static const sqb_graph_t *PCUR;
static double *PEX; static int PEXN;

static int plain_init(void){
    if(PON >= 0) return PON;
    const char *e = getenv("SINCQED_GPU"); PON = 0;
    if(e && !strcmp(e, "0")) return 0;
    int nd = 0; if(cudaGetDeviceCount(&nd) != cudaSuccess || nd == 0){ cudaGetLastError(); return 0; }
    int dev = e && atoi(e) > 0 ? atoi(e) - 1 : 0; if(dev >= nd) dev = 0;
    if(sqb_dev_init(dev)){ fprintf(stderr, "gpu: %s\n", g_err); exit(3); }
    for(int b = 0; b < 2; b++){ CKX(cudaStreamCreateWithFlags(&PS[b].st, cudaStreamNonBlocking)); CKX(cudaEventCreateWithFlags(&PS[b].ev, cudaEventDisableTiming)); }
    return PON = 1;
}
static void plain_reserve(pslot_t *s, long n){
    if(n <= s->cap) return;
    if(s->cap){ cudaFreeHost(s->hK); cudaFree(s->dK); cudaFreeHost(s->hS); cudaFree(s->dS); cudaFreeHost(s->hF); cudaFree(s->dF); cudaFreeHost(s->hA); cudaFree(s->dA); }
    long c = 1L << 16; while(c < n) c <<= 1; s->cap = c;
    CKX(cudaMallocHost(&s->hK, c*SQB_MAXD)); CKX(cudaMalloc(&s->dK, c*SQB_MAXD));
    CKX(cudaMallocHost(&s->hS, c)); CKX(cudaMalloc(&s->dS, c));
    CKX(cudaMallocHost(&s->hF, c*sizeof(double))); CKX(cudaMalloc(&s->dF, c*sizeof(double)));
    CKX(cudaMallocHost(&s->hA, c*sizeof(double))); CKX(cudaMalloc(&s->dA, c*sizeof(double)));
}

extern "C" const char *gpu_info(void){ return PON == 1 ? G.info : "off"; }

extern "C" int gpu_setup(const char *name, int D, const double *EX, int K, double H){
    PCUR = NULL;
    if(!plain_init()) return 0;
    const sqb_graph_t *g = sqb_find_graph(name);
    if(!g || strcmp(g->name, name)) return 0;
    if(g->D != D){ fprintf(stderr, "gpu: %s has D=%d, expected %d\n", name, g->D, D); exit(3); }
    PCUR = g; PD = D; PK = K; PH = H;
    CKX(cudaDeviceSynchronize());
    if(PEXN < 2*K + 1){ if(PEX) CKX(cudaFree(PEX)); PEXN = 2*K + 1; CKX(cudaMalloc(&PEX, PEXN*sizeof(double))); }
    CKX(cudaMemcpy(PEX, EX, (2*K + 1)*sizeof(double), cudaMemcpyHostToDevice));
    return 1;
}

static void plain_launch(pslot_t *s, long npts, long nrows, int cells, int st, int has_skip){
    sqb_eval_t a; memset(&a, 0, sizeof a);
    a.pts = s->dK; a.n = nrows; a.esize = 1; a.stride = PD; a.flag_at = -1; a.cells = cells; a.st = st;
    a.X = PEX; a.Wt = NULL; a.K = PK; a.H = PH; a.raw = 1; a.skip = has_skip ? s->dS : NULL;
    a.v = s->dF; a.ab = s->dA;
    size_t smem = 2*(2*PK + 1)*sizeof(double);
    PCUR->f64(&a, grid_for(PCUR, 0, npts, smem), 128, smem, s->st);
    CKX(cudaGetLastError());
}

extern "C" void gpu_submit(int slot, long n, const int *k, int stride, const unsigned char *skip){
    pslot_t *s = &PS[slot]; plain_reserve(s, n); s->n = n;
    if(n <= 0) return;
    signed char *hk = s->hK; const int D = PD;
    #pragma omp parallel for schedule(static)
    for(long i = 0; i < n; i++) for(int d = 0; d < D; d++) hk[i*D + d] = (signed char)k[i*stride + d];
    CKX(cudaMemcpyAsync(s->dK, hk, n*D, cudaMemcpyHostToDevice, s->st));
    if(skip){ memcpy(s->hS, skip, n); CKX(cudaMemcpyAsync(s->dS, s->hS, n, cudaMemcpyHostToDevice, s->st)); }
    plain_launch(s, n, n, 0, 0, skip != NULL);
    CKX(cudaMemcpyAsync(s->hF, s->dF, n*sizeof(double), cudaMemcpyDeviceToHost, s->st));
    CKX(cudaMemcpyAsync(s->hA, s->dA, n*sizeof(double), cudaMemcpyDeviceToHost, s->st));
    CKX(cudaEventRecord(s->ev, s->st));
}

extern "C" void gpu_submit_cells(int slot, long nc, const int *cells, int stride, const unsigned char *skip, int st){
    pslot_t *s = &PS[slot]; const long n = nc << PD; plain_reserve(s, n); s->n = n;
    if(nc <= 0) return;
    signed char *hk = s->hK; const int D = PD;
    #pragma omp parallel for schedule(static)
    for(long c = 0; c < nc; c++) for(int d = 0; d < D; d++) hk[c*D + d] = (signed char)cells[c*stride + d];
    CKX(cudaMemcpyAsync(s->dK, hk, nc*D, cudaMemcpyHostToDevice, s->st));
    if(skip){ memcpy(s->hS, skip, nc); CKX(cudaMemcpyAsync(s->dS, s->hS, nc, cudaMemcpyHostToDevice, s->st)); }
    plain_launch(s, n, nc, 1, st, skip != NULL);
    CKX(cudaMemcpyAsync(s->hF, s->dF, n*sizeof(double), cudaMemcpyDeviceToHost, s->st));
    CKX(cudaMemcpyAsync(s->hA, s->dA, n*sizeof(double), cudaMemcpyDeviceToHost, s->st));
    CKX(cudaEventRecord(s->ev, s->st));
}

extern "C" void gpu_wait(int slot, const double **fw, const double **abw){
    pslot_t *s = &PS[slot];
    if(s->n > 0) CKX(cudaEventSynchronize(s->ev));
    *fw = s->hF; *abw = s->hA;
}

/* the reference's per-graph launcher (sq_gpu_launch_t, driver/gpu.h:18-19) on device buffers: int16
 * coordinates, stride D, n points (cells: n = nc << D).  It has no return value, and the caller's own CUDA runtime
 * does not see this library's errors: a launch that fails prints and exits, as the rest of the plain form */
extern "C" void sqb_gg_launch(const sqb_graph_t *g, void *st, long n, const short *k, const unsigned char *skip,
                              const double *EX, int K, double H, double *of, double *oab, int cmode, int cst){
    if(n <= 0) return;
    if(!G.on && sqb_dev_init(0)){ fprintf(stderr, "gpu: %s\n", g_err); exit(3); }
    sqb_eval_t a; memset(&a, 0, sizeof a);
    a.pts = k; a.n = cmode ? (n >> g->D) : n; a.esize = 2; a.stride = g->D; a.flag_at = -1; a.cells = cmode; a.st = cst;
    a.X = EX; a.Wt = NULL; a.K = K; a.H = H; a.raw = 1; a.skip = skip; a.v = of; a.ab = oab;
    size_t smem = 2*(2*K + 1)*sizeof(double);
    const int grid = grid_for(g, 0, n, smem);
    cudaGetLastError();                                 /* an earlier call's error is not this launch's */
    g->f64(&a, grid, 128, smem, st);
    CKX(cudaGetLastError());
}

/* GG_<graph>'s launcher with the FP64 build chosen (0 as written, 2 contracted) */
extern "C" int sqb_plugin_launch(const char *graph, int form, cudaStream_t st, long n, const short *k, const unsigned char *skip,
                                 const double *EX, int K, double H, double *of, double *oab, int cmode, int cst){
    const sqb_graph_t *g = sqb_find_graph(graph);
    if(!g || (form != 0 && form != 2) || (form == 2 && !g->f64_fma) || K < 0 || K > 127){
        snprintf(g_err, sizeof g_err, "sqb_plugin_launch: no graph %s with FP64 build %d (or K %d outside 0..127)", graph, form, K);
        sqb_set_error_msg(g_err);
        return -1;
    }
    if(n <= 0) return 0;
    if(sqb_dev_init(0)){ sqb_set_error_msg(g_err); return -1; }
    sqb_eval_t a; memset(&a, 0, sizeof a);
    a.pts = k; a.n = cmode ? (n >> g->D) : n; a.esize = 2; a.stride = g->D; a.flag_at = -1; a.cells = cmode; a.st = cst;
    a.X = EX; a.Wt = NULL; a.K = K; a.H = H; a.raw = 1; a.skip = skip; a.v = of; a.ab = oab;
    const size_t smem = 2*(2*K + 1)*sizeof(double);
    launch_f64(g, form, &a, grid_for(g, form, n, smem), smem, st);
    const cudaError_t e = cudaGetLastError();
    if(e != cudaSuccess){
        snprintf(g_err, sizeof g_err, "sqb_plugin_launch: %s", cudaGetErrorString(e)); sqb_set_error_msg(g_err); return (int)e; }
    G.launches++;
    return 0;
}

/* Copies of a caller's pageable arrays through the thread's pinned buffers, two halves of PIN_HALF bytes in turn: the host
 * fills or empties one half (four threads for a large piece) while the device copies the other.  The driver's own staging
 * of pageable memory took about 170 us of the 342 of 20,001 points of syn_d11 in double-double (1.8 MB in, 0.6 out); 175 in all now.
 * pin_to_device returns with the last pieces still under way on the stream, pin_to_host when everything has arrived. */
#define PIN_HALF (512UL << 10)
struct Pin {
    char *p; cudaEvent_t ev[2];
    ~Pin(){ if(p) cudaFreeHost(p); for(cudaEvent_t e : ev) if(e) cudaEventDestroy(e); }      /* given back when the thread ends */
};
static thread_local Pin P = {NULL, {NULL, NULL}};
static int pin_room(void){
    for(cudaEvent_t &e : P.ev) if(!e) CKR(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    if(!P.p) CKR(cudaMallocHost(&P.p, 2*PIN_HALF));
    return 0;
}
static void piece_copy(char *dst, const char *src, size_t n){
    if(n < (128UL << 10)){ memcpy(dst, src, n); return; }
    const size_t q = (n/4 + 63)/64*64;
    #pragma omp parallel for num_threads(4) schedule(static, 1)
    for(int j = 0; j < 4; j++){ const size_t o = j*q; if(o < n) memcpy(dst + o, src + o, n - o < q ? n - o : q); }
}
static int pin_to_device(void *dst, const void *src, size_t n){
    for(size_t o = 0; o < n; o += PIN_HALF){
        const int h = (o/PIN_HALF) & 1; const size_t m = n - o < PIN_HALF ? n - o : PIN_HALF;
        CKR(cudaEventSynchronize(P.ev[h]));                /* the half's last copy (a new event is complete) */
        piece_copy(P.p + h*PIN_HALF, (const char*)src + o, m);
        CKR(cudaMemcpyAsync((char*)dst + o, P.p + h*PIN_HALF, m, cudaMemcpyHostToDevice, G.s));
        CKR(cudaEventRecord(P.ev[h], G.s));
    }
    return 0;
}
static int pin_to_host(void *dst, const void *src, size_t n){
    const size_t np = (n + PIN_HALF - 1)/PIN_HALF;
    for(size_t p = 0; p <= np; p++){
        if(p < np){                                         /* the half's earlier use has ended: on the stream, or below */
            const size_t o = p*PIN_HALF, m = n - o < PIN_HALF ? n - o : PIN_HALF;
            CKR(cudaMemcpyAsync(P.p + (p & 1)*PIN_HALF, (const char*)src + o, m, cudaMemcpyDeviceToHost, G.s));
            CKR(cudaEventRecord(P.ev[p & 1], G.s));
        }
        if(p > 0){
            const size_t o = (p - 1)*PIN_HALF, m = n - o < PIN_HALF ? n - o : PIN_HALF;
            CKR(cudaEventSynchronize(P.ev[(p - 1) & 1]));
            piece_copy((char*)dst + o, P.p + ((p - 1) & 1)*PIN_HALF, m);
        }
    }
    return 0;
}

/* pointwise evaluation (parity checks): n points given by their variables, FP64 (SQ_AB = ab) or
 * double-double; f, abs_ hold n values (FP64) or n (hi, lo) pairs (double-double) */
extern "C" int sqb_eval_points_impl(const sqb_graph_t *g, long n, const double *sf, int prec, int ab, double *f, double *abs_){
    if(n <= 0) return 0;
    const int D = g->D;
    /* one stream-ordered block (no device-wide synchronisation, so other threads' work runs on): sf[n D], the values and
     * the |.| sums (n each, or n pairs), skip[n] */
    const bool dd = !(prec == 0 || prec == 2);
    const int w = dd ? 1 : f64_which(g, prec == 2);
    if(prec == 2 && w != 2){ snprintf(g_err, sizeof g_err, "%s: no contracted FP64 kernel in this library", g->name); return -1; }
    const size_t nv = (dd ? 2 : 1)*(size_t)n, nd = (size_t)n*D + 2*nv, nin = (size_t)n*D*sizeof(double), nout = nv*sizeof(double);
    if(pin_room()) return -1;
    struct Block { char *p = NULL; ~Block(){ if(p) cudaFreeAsync(p, G.s); } } blk;       /* released on every return */
    CKR(cudaMallocAsync((void**)&blk.p, nd*sizeof(double) + (size_t)n, G.s));
    double *dsf = (double*)blk.p, *dv = dsf + (size_t)n*D, *dab = dv + nv;
    unsigned char *dsk = (unsigned char*)(dab + nv);
    const bool small = nin <= PIN_HALF && 2*nout <= PIN_HALF;       /* one piece each way */
    if(small){
        memcpy(P.p, sf, nin);
        CKR(cudaMemcpyAsync(dsf, P.p, nin, cudaMemcpyHostToDevice, G.s));
    } else if(pin_to_device(dsf, sf, nin)) return -1;
    if(!ab) CKR(cudaMemsetAsync(dsk, 1, n, G.s));
    sqb_eval_t a; memset(&a, 0, sizeof a);
    a.pts = NULL; a.n = n; a.esize = 1; a.stride = D; a.flag_at = -1; a.cells = 0;
    /* no lattice: the one-entry tables are loaded and not used */
    a.X = dsf; a.Wt = dsf; a.K = 0; a.raw = 1; a.skip = ab ? NULL : dsk; a.v = dv; a.ab = dab; a.sfin = dsf;
    const size_t smem = 2*sizeof(double);
    if(!dd) launch_f64(g, w, &a, grid_for(g, w, n, smem), smem, G.s);
    else {                                           /* raw = 2: (hi, lo) pairs, as the caller's arrays hold them */
        a.raw = 2; a.vlo = dv + 1; a.ablo = dab + 1;
        sqb_dd_t d; memset(&d, 0, sizeof d); d.e = a; d.all = 1;
        g->dd(&d, grid_for(g, 1, n, smem), 128, smem, G.s);
    }
    CKR(cudaGetLastError());
    if(small){
        CKR(cudaMemcpyAsync(P.p + PIN_HALF, dv, 2*nout, cudaMemcpyDeviceToHost, G.s));
        CKR(cudaStreamSynchronize(G.s));
        memcpy(f, P.p + PIN_HALF, nout); memcpy(abs_, P.p + PIN_HALF + nout, nout);
        return 0;
    }
    return pin_to_host(f, dv, nout) || pin_to_host(abs_, dab, nout) ? -1 : 0;
}

/* the scaling test's device part: a->g[3 ndir] for the directions of a, with the factor table xs
 * (3 x (2E+1), host); the values come back to g_host.  Returns 0, 1 if the graph has no raw point
 * function, or -1 */
extern "C" int sqb_dev_scale(const sqb_graph_t *g, sqb_scale_t *a, const double *xs, double *g_host){
    if(!g->scale) return 1;
    const size_t nxs = 3*(size_t)(2*a->E + 1), ng = 3*(size_t)a->ndir;
    double *blk = NULL;
    CKR(cudaMallocAsync((void**)&blk, (nxs + ng)*sizeof(double), G.s));
    a->xs = blk; a->g = blk + nxs;
    CKR(cudaMemcpyAsync(blk, xs, nxs*sizeof(double), cudaMemcpyHostToDevice, G.s));
    long want = ((long)ng + 127)/128, full = (long)G.nsm*4;
    g->scale(a, (int)(want < full ? want : full), 128, G.s);
    CKR(cudaGetLastError());
    G.launches++;
    CKR(cudaMemcpyAsync(g_host, a->g, ng*sizeof(double), cudaMemcpyDeviceToHost, G.s));
    CKR(cudaStreamSynchronize(G.s));
    cudaFreeAsync(blk, G.s);
    return 0;
}

/* FP64 peak probe: independent chains of fused multiply-adds (8 per thread, unrolled) or of adds, on
 * every SM; flops = 2 per FMA, 1 per add.  The measured rate is the denominator of the evaluation
 * kernels' roofline (the device has no vendor FP64 figure in this environment). */
template<int FMA>
__global__ void __launch_bounds__(256) sqb_k_fp64_probe(double *out, long iters, double a, double b){
    double x[8];
#pragma unroll
    for(int j = 0; j < 8; j++) x[j] = threadIdx.x*1e-9 + j;
    for(long i = 0; i < iters; i++){
#pragma unroll
        for(int j = 0; j < 8; j++) x[j] = FMA ? __fma_rn(x[j], a, b) : __dadd_rn(x[j], b);
    }
    double s = 0;
#pragma unroll
    for(int j = 0; j < 8; j++) s += x[j];
    if(s == 1.2345) out[0] = s;      /* keeps the chains alive */
}
/* returns the rate in TFLOP/s (fma = 1: FMA, 2 flops each; fma = 0: adds) */
extern "C" double sqb_probe_fp64(int fma, long iters){
    if(sqb_dev_init(0)) return -1;
    double *o; if(cudaMalloc(&o, sizeof(double)) != cudaSuccess) return -1;
    int per = 0;
    if(fma) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, sqb_k_fp64_probe<1>, 256, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, sqb_k_fp64_probe<0>, 256, 0);
    const int grid = G.nsm*(per > 0 ? per : 4);
    float best = 1e30f;
    for(int r = 0; r < 4; r++){
        cudaEventRecord(G.e0, G.s);
        if(fma) sqb_k_fp64_probe<1><<<grid, 256, 0, G.s>>>(o, iters, 0.999999, 1e-7);
        else sqb_k_fp64_probe<0><<<grid, 256, 0, G.s>>>(o, iters, 0.999999, 1e-7);
        cudaEventRecord(G.e1, G.s);
        cudaEventSynchronize(G.e1);
        float t = 0; cudaEventElapsedTime(&t, G.e0, G.e1);
        if(r && t < best) best = t;
    }
    cudaFree(o);
    const double ops = (double)grid*256*8*(double)iters*(fma ? 2 : 1);
    return ops/(best*1e-3)/1e12;
}

/* The reduce / finish / scatter sequence of one level batch on buffers the caller names (used by the
 * allocation-free entry point, noalloc.cu): v, uu, stt per child; bp, bkeep, boff per tile; acc and
 * base the accumulator and this batch's first kept slot. */
extern "C" int sqb_level_tail(const void *cells, long nchildren, int D, int st, int last, int abskip, double pw, double thr,
                              const double *v, const double *uu, const unsigned char *stt,
                              void *bp, unsigned *bkeep, unsigned long long *boff, sqb_acc_t *acc, unsigned long long *base,
                              void *fin, void *next, long next_cap, void *stream){
    /* fin: SQB_FIN_BYTES, zeroed before the first use: the finish kernel's counter, its offsets and its sums, of at most
     * FT tiles */
    if((nchildren + RTILE - 1)/RTILE > FT){ snprintf(g_err, sizeof g_err, "level tail: more than %d tiles", FT); return -1; }
    static_assert(sizeof(fpart_t) + 32 <= SQB_FIN_BYTES, "the caller's room for the finish kernel");
    unsigned *fcnt = (unsigned*)fin; unsigned long long *coff = (unsigned long long*)fin + 1; fpart_t *fp = (fpart_t*)((char*)fin + 32);
    lvl_t r; memset(&r, 0, sizeof r);        /* no symmetry fold here (r.sym.n = 0) */
    r.cells = (const signed char*)cells; r.n = nchildren; r.D = D; r.st = st; r.last = last;
    r.abskip = abskip; r.pw = pw; r.thr = thr; r.v = v; r.uu = uu; r.stt = stt;
    const long nb = (nchildren + RTILE - 1)/RTILE;
    cudaStream_t s = (cudaStream_t)stream;
    sqb_k_reduce<<<(unsigned)nb, RT, 0, s>>>(r, (part_t*)bp, bkeep, NULL);
    CKR(cudaGetLastError());
    sqb_k_finish<<<1, FT, 0, s>>>(r, (const part_t*)bp, bkeep, nb, boff, acc, base, fp, coff, fcnt);
    CKR(cudaGetLastError());
    if(!last){
        sqb_k_scatter<<<(unsigned)nb, RT, 0, s>>>(r, boff, coff, base, (sqb_pt_t*)next, next_cap, &acc->overflow);
        CKR(cudaGetLastError());
    }
    return 0;
}
/* bytes of one tile partial (sizing of caller-provided tile buffers) and children per tile */
extern "C" size_t sqb_level_tile_bytes(void){ return sizeof(part_t); }
extern "C" long sqb_level_tile_children(void){ return RTILE; }
