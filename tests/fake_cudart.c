/* A CUDA runtime on host memory, for tests of the library's host code where no
 * device is at hand: preloaded before libcudart, it serves the calls that
 * libmset_b200.so makes.  Device memory is host memory in a table, kernels are
 * logged and do nothing, copies and clears really happen and are checked
 * against the table: one that leaves a live allocation is counted (fake_bad)
 * and left out.  A captured graph replays the checks of what it holds, so one
 * that was captured on memory freed since shows up too.  The controls and the
 * log are the fake_* functions. */
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

typedef int cudaError_t;
typedef struct {
    unsigned x, y, z;
} dim3;
enum { kOk = 0, kInvalid = 1, kNoMem = 2 };

/* ---- memory ---------------------------------------------------------------- */
#define MAXA 4096
static struct {
    char *p;
    size_t n;
    int live;
} g_mem[MAXA];
static int g_count, g_bad;
static size_t g_deny;
static cudaError_t g_last;

static cudaError_t err(cudaError_t e) {
    if (e) g_last = e;
    return e;
}
int fake_bad(void) { return g_bad; }
int fake_allocs(void) { return g_count; }
void *fake_alloc(int i) { return g_mem[i].p; }
size_t fake_alloc_bytes(int i) { return g_mem[i].live ? g_mem[i].n : 0; }
/* allocations of exactly this size fail (0: none) */
void fake_deny(size_t bytes) { g_deny = bytes; }

cudaError_t cudaMalloc(void **p, size_t n) {
    *p = NULL;
    if ((g_deny && n == g_deny) || g_count == MAXA) return err(kNoMem);
    g_mem[g_count].p = calloc(1, n ? n : 1); /* never handed back: a stale pointer stays recognisable */
    g_mem[g_count].n = n;
    g_mem[g_count].live = 1;
    *p = g_mem[g_count++].p;
    return kOk;
}
cudaError_t cudaFree(void *p) {
    for (int i = 0; i < g_count; ++i)
        if (p && g_mem[i].p == p && g_mem[i].live) {
            g_mem[i].live = 0;
            return kOk;
        }
    return p ? err(kInvalid) : kOk;
}
/* 1: [p, p + n) inside a live allocation */
static int inside(const void *p, size_t n) {
    const char *c = p;
    for (int i = 0; i < g_count; ++i)
        if (g_mem[i].live && c >= g_mem[i].p && c + n <= g_mem[i].p + g_mem[i].n) return 1;
    return 0;
}
/* ---- launches, copies and clears, recorded while a stream captures ----------- */
typedef struct {
    int kind; /* 0 kernel, 1 clear, 2 copy */
    const char *name;
    void *dst;
    const void *src;
    size_t n;
    int value, dir;
    dim3 grid, block;
    size_t arg_bytes;
    char arg[1024]; /* the first argument's bytes, for the kernels of fake_watch */
} Op;
typedef struct {
    Op *op;
    int n, cap;
} List;
static List *g_capture;

static List g_log;
static void append(List *l, const Op *o) {
    if (l->n == l->cap) l->op = realloc(l->op, sizeof(Op) * (size_t)(l->cap = l->cap ? 2 * l->cap : 64));
    l->op[l->n++] = *o;
}
static cudaError_t perform(const Op *o) {
    if (o->kind == 0) {
        append(&g_log, o);
        return kOk;
    }
    const int dev_dst = o->kind == 1 || o->dir == 1 || o->dir == 3, dev_src = o->kind == 2 && (o->dir == 2 || o->dir == 3);
    if (o->n == 0) return kOk;
    if ((dev_dst && !inside(o->dst, o->n)) || (dev_src && !inside(o->src, o->n))) {
        ++g_bad;
        return kOk;
    }
    if (o->kind == 1) memset(o->dst, o->value, o->n);
    else memcpy(o->dst, o->src, o->n);
    return kOk;
}
static cudaError_t submit(const Op *o) {
    if (g_capture) {
        append(g_capture, o);
        return kOk;
    }
    return perform(o);
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, void *st) {
    Op o = {.kind = 1, .dst = p, .value = v, .n = n};
    (void)st;
    return submit(&o);
}
cudaError_t cudaMemset(void *p, int v, size_t n) { return cudaMemsetAsync(p, v, n, NULL); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, int dir, void *st) {
    Op o = {.kind = 2, .dst = d, .src = s, .n = n, .dir = dir};
    (void)st;
    return submit(&o);
}

/* kernels whose first argument is kept: part of the name, bytes of it */
static char g_watch[64];
static size_t g_watch_bytes;
void fake_watch(const char *part, size_t bytes) {
    snprintf(g_watch, sizeof g_watch, "%s", part);
    g_watch_bytes = bytes < 1024 ? bytes : 1024;
}
int fake_launches(void) { return g_log.n; }
const char *fake_name(int i) { return g_log.op[i].name; }
const void *fake_arg(int i) { return g_log.op[i].arg_bytes ? g_log.op[i].arg : NULL; }
int fake_blocks(int i) { return (int)(g_log.op[i].grid.x * g_log.op[i].grid.y * g_log.op[i].grid.z); }
void fake_clear_log(void) { g_log.n = 0; }

#define MAXF 8192
static struct {
    const void *host;
    char *name;
} g_fun[MAXF];
static int g_funs;
void **__cudaRegisterFatBinary(void *f) {
    (void)f;
    static void *h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterFunction(void **h, const char *host, char *dev, const char *name, int lim, void *a, void *b, void *c,
                            void *d, int *e) {
    (void)h, (void)dev, (void)lim, (void)a, (void)b, (void)c, (void)d, (void)e;
    if (g_funs < MAXF) {
        g_fun[g_funs].host = host;
        g_fun[g_funs++].name = strdup(name);
    }
}
void __cudaRegisterVar(void **h, char *v, char *d, const char *n, int e, size_t s, int c, int g) {
    (void)h, (void)v, (void)d, (void)n, (void)e, (void)s, (void)c, (void)g;
}
static const char *name_of(const void *f) {
    for (int i = 0; i < g_funs; ++i)
        if (g_fun[i].host == f) return g_fun[i].name;
    return "?";
}
static cudaError_t launch(const void *f, dim3 g, dim3 b, void **args) {
    Op o = {.kind = 0, .name = name_of(f), .grid = g, .block = b};
    if (g_watch_bytes && strstr(o.name, g_watch)) memcpy(o.arg, args[0], o.arg_bytes = g_watch_bytes);
    return submit(&o);
}
static dim3 g_pg, g_pb;
static size_t g_ps;
static void *g_pst;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void *st) {
    g_pg = g, g_pb = b, g_ps = s, g_pst = st;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
    *g = g_pg, *b = g_pb, *s = g_ps, *(void **)st = g_pst;
    return kOk;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **args, size_t s, void *st) {
    (void)s, (void)st;
    return launch(f, g, b, args);
}
typedef struct {
    dim3 grid, block;
} Cfg; /* the leading members of cudaLaunchConfig_t */
cudaError_t cudaLaunchKernelExC(const Cfg *c, const void *f, void **args) { return launch(f, c->grid, c->block, args); }

/* ---- graphs ------------------------------------------------------------------- */
cudaError_t cudaStreamBeginCapture(void *st, int mode) {
    (void)st, (void)mode;
    g_capture = calloc(1, sizeof *g_capture);
    return kOk;
}
cudaError_t cudaStreamEndCapture(void *st, void **g) {
    (void)st;
    *g = g_capture;
    g_capture = NULL;
    return kOk;
}
cudaError_t cudaGraphInstantiate(void **x, void *g, unsigned long long f) {
    (void)f;
    *x = g;
    return kOk;
}
cudaError_t cudaGraphLaunch(void *x, void *st) {
    (void)st;
    const List *l = x;
    for (int i = 0; i < l->n; ++i) perform(&l->op[i]);
    return kOk;
}
cudaError_t cudaGraphDestroy(void *g) { return (void)g, kOk; }
cudaError_t cudaGraphExecDestroy(void *g) { return (void)g, kOk; }

/* ---- device, streams, events ----------------------------------------------------- */
/* clusters of more than 8 CTAs: how many the device holds at once; below 0 the
 * query fails */
static int g_clusters = 8;
void fake_clusters(int n) { g_clusters = n; }
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *f, const void *c) {
    (void)f, (void)c;
    *n = g_clusters;
    return g_clusters < 0 ? err(912 /* cudaErrorInvalidClusterSize */) : kOk;
}
cudaError_t cudaFuncSetAttribute(const void *f, int a, int v) { return (void)f, (void)a, (void)v, kOk; }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, kOk; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, kOk; }
cudaError_t cudaSetDevice(int d) { return (void)d, kOk; }
cudaError_t cudaDeviceGetAttribute(int *v, int a, int d) { return (void)a, (void)d, *v = 148, kOk; }
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = g_last;
    g_last = kOk;
    return e;
}
const char *cudaGetErrorString(cudaError_t e) { return (void)e, "error of the host-memory runtime"; }
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { return (void)s, *p = NULL, err(kInvalid); }
cudaError_t cudaGetDriverEntryPoint(const char *n, void **f, unsigned long long l, void *r) {
    return (void)n, (void)l, (void)r, *f = NULL, err(kInvalid);
}
static int g_handle;
cudaError_t cudaStreamCreateWithFlags(void **s, unsigned f) { return (void)f, *s = &g_handle, kOk; }
cudaError_t cudaStreamDestroy(void *s) { return (void)s, kOk; }
cudaError_t cudaStreamSynchronize(void *s) { return (void)s, kOk; }
cudaError_t cudaStreamWaitEvent(void *s, void *e, unsigned f) { return (void)s, (void)e, (void)f, kOk; }
cudaError_t cudaEventCreate(void **e) { return *e = &g_handle, kOk; }
cudaError_t cudaEventCreateWithFlags(void **e, unsigned f) { return (void)f, *e = &g_handle, kOk; }
cudaError_t cudaEventDestroy(void *e) { return (void)e, kOk; }
cudaError_t cudaEventRecord(void *e, void *s) { return (void)e, (void)s, kOk; }
cudaError_t cudaEventSynchronize(void *e) { return (void)e, kOk; }
cudaError_t cudaEventElapsedTime(float *ms, void *a, void *b) { return (void)a, (void)b, *ms = 1.0f, kOk; }
