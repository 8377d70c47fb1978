"""The grow's device memory when an allocation fails (CPU, against a stand-in for the CUDA runtime that counts
allocations and refuses the n-th): whichever allocation of a grow, its final threshold, its tiers and its dilation is
refused, the call returns an error, nothing is released twice, and after sqb_grow_end only the buffers that the thread
keeps for its next grow are held; the next grow on the thread runs, and does not meet the reported error again as the
runtime's last one.  Kernels do not run: the stand-in launches nothing,
and the sizes that the host would read back are set by the test."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, 'sincfeyn_b200', 'csrc')
NVCC = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
pytestmark = pytest.mark.skipif(not os.path.exists(NVCC), reason='no nvcc')

FAKE = r'''
#include <stdlib.h>
#include <string.h>
#define MAX 4096
void *fake_live[MAX]; int fake_nlive, fake_count, fake_fail, fake_twice, fake_last;
int fake_is_live(void *p){ for(int i = 0; i < fake_nlive; i++) if(fake_live[i] == p) return 1; return 0; }
int cudaMallocAsync(void **p, size_t n, void *s){
    if(++fake_count == fake_fail) return fake_last = 2;
    *p = calloc(1, n); fake_live[fake_nlive++] = *p; return 0; }
int cudaFreeAsync(void *p, void *s){
    for(int i = 0; i < fake_nlive; i++) if(fake_live[i] == p){ free(p); fake_live[i] = fake_live[--fake_nlive]; return 0; }
    fake_twice++; return 1; }
int cudaMallocHost(void **p, size_t n){ *p = calloc(1, n); return 0; }
int cudaHostAlloc(void **p, size_t n, unsigned f){ *p = calloc(1, n); return 0; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *st){ memmove(d, s, n); return 0; }
int cudaMemsetAsync(void *d, int v, size_t n, void *st){ memset(d, v, n); return 0; }
int cudaStreamSynchronize(void *s){ return 0; }
int cudaGetLastError(void){ const int e = fake_last; fake_last = 0; return e; }
const char *cudaGetErrorString(int e){ return e == 2 ? "out of memory" : "error"; }
int cudaLaunchKernel(){ return 0; }
int cudaLaunchKernelExC(){ return 0; }
unsigned __cudaPushCallConfiguration(){ return 0; }
int __cudaPopCallConfiguration(){ return 0; }
static void *handle;
void **__cudaRegisterFatBinary(void *f){ return &handle; }
void __cudaRegisterFatBinaryEnd(void **h){}
void __cudaUnregisterFatBinary(void **h){}
void __cudaRegisterFunction(){}
void __cudaRegisterVar(){}
char __cudaInitModule(void **h){ return 1; }
int __cudaGetKernel(void **k, const void *f){ *k = (void*)f; return 0; }
int __cudaLaunchKernel(){ return 0; }
void sqb_dev_count_copy(unsigned long long a, unsigned long long b){}
'''

HARNESS = r'''
#include "topgrid.cu"
extern "C" { extern void *fake_live[]; extern int fake_nlive, fake_count, fake_fail, fake_twice, fake_last; int fake_is_live(void *p); }
/* one grow with a frontier of n points, kept kept points and a grid of W^5 nodes; 0, or where it failed */
extern "C" int grow_once(long n, long kept, int W){
    u64 P[SQB_MAXD] = {0}; u64 y = 1;
    for(int i = 4; i >= 0; i--){ P[i] = y; y *= W; }
    const sqb_pt_t *pts; long np; sqb_pt_t *out = NULL; sqb_grow_sums_t s;
    int rc = 0;
    if(sqb_grow_begin(5, (W - 1)/2*2, 2, W, P, 0, 1, 1e-9, 32.0, NULL, &pts, &np)) rc = 1;
    long nmax; const u64 *cnt;
    if(!rc && sqb_grow_chain(&nmax, &cnt) < 0) rc = 2;
    if(!rc){ GR.nfr = n; if(sqb_grow_expand(NULL, NULL, NULL)) rc = 3; }
    if(!rc){ GR.nkeep = kept; GR.nseen = 2*kept; if(sqb_grow_finish(1)) rc = 4; }
    if(!rc && sqb_grow_dilate(40, &out)) rc = 5;
    if(!rc && sqb_grow_sums(&s)) rc = 6;
    if(out) cudaFreeAsync(out, NULL);
    sqb_grow_end();
    return rc;
}
/* pointers the thread holds; -1 if one of them has been released, or if memory is held that none of them names */
extern "C" int held(void){
    void *p[] = {GR.key, GR.word, GR.fr, GR.nx, GR.frsk, GR.nxsk, GR.keep, GR.kv, GR.kk, GR.kj, GR.qs, GR.part, GR.cpart, GR.acc, GR.probe,
                 SC.bcnt, SC.boff, SC.drop};
    int n = 0;
    for(void *q : p) if(q){ if(!fake_is_live(q)) return -1; n++; }
    return n == fake_nlive ? n : -1;
}
extern "C" int sort_once(void){
    static u64 keys[5000];
    return sqb_radix_sort_u64(keys, 5000, 24, NULL);
}
extern "C" void reset(void){          /* as a new thread */
    GR = Grow(); SC = Scratch(); fake_nlive = fake_count = fake_fail = fake_twice = fake_last = 0;
}
'''


@pytest.fixture(scope='module')
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp('topgrid')
    (d / 'fake.c').write_text(FAKE)
    (d / 'harness.cu').write_text(HARNESS)
    subprocess.run(['gcc', '-w', '-std=gnu11', '-fPIC', '-c', str(d / 'fake.c'), '-o', str(d / 'fake.o')], check=True)
    subprocess.run([NVCC, '-gencode', 'arch=compute_100a,code=sm_100a', '-O1', '-std=c++17', '-cudart', 'none', '-shared', '-Xlinker', '-Bsymbolic', '-Xcompiler', '-fPIC',
                    '-diag-suppress', '177,550', '-I' + CSRC, '-I' + os.path.join(ROOT, 'include'), '-o', str(d / 'topgrid.so'),
                    str(d / 'harness.cu'), str(d / 'fake.o')], check=True)
    L = C.CDLL(str(d / 'topgrid.so'))
    L.grow_once.argtypes = [C.c_long, C.c_long, C.c_int]
    return L


def var(L, name):
    return C.c_int.in_dll(L, 'fake_' + name)


# a grown table and lists; a kept list for one cluster and a longer one; the dilation by bitmap (33^5) and by sort (57^5)
@pytest.mark.parametrize('n,kept,W', [(65000, 20000, 33), (65000, 20000, 57), (6000, 3000, 33)])
def test_a_refused_allocation_leaves_nothing_behind(lib, n, kept, W):
    lib.reset()
    assert lib.grow_once(n, kept, W) == 0 and var(lib, 'twice').value == 0
    total, keeps = var(lib, 'count').value, lib.held()
    assert total > 15 and keeps > 0
    for i in range(1, total + 1):
        lib.reset()
        var(lib, 'fail').value = i
        assert lib.grow_once(n, kept, W) != 0, i
        assert var(lib, 'twice').value == 0 and lib.held() >= 0, (i, 'of', total)
        assert lib.grow_once(n, kept, W) == 0 and var(lib, 'twice').value == 0 and lib.held() == keeps, (i, 'of', total)


def test_a_refused_allocation_of_the_sort(lib):
    for i in (1, 2, 3):
        lib.reset()
        var(lib, 'fail').value = i
        assert lib.sort_once() != 0 and var(lib, 'nlive').value == 0 and var(lib, 'twice').value == 0
